"""FP64 products of more rows (columns) than one grid dimension holds tiles of:
65535 tiles are 1.05 M rows of 16 and 2.1 M of 32, the tiles that few columns
take.  Bound as for every product: 2 (c K + 8) eps of sum |a| |b|, c = 4 complex."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cplx,M,N,K", [
    (True, 1048560, 5, 17), (True, 1048561, 5, 17), (True, 5, 1048561, 17), (False, 1048577, 16, 33),
    (False, 2097121, 32, 4), (True, 2097121, 17, 2), (False, 17, 2097121, 4),
])
def test_tall_and_wide_products(cplx, M, N, K):
    from renormalizer_b200._native import Engine
    g = torch.Generator(device="cuda").manual_seed(M + N)
    r = lambda *s: torch.randn(s, dtype=torch.float64, device="cuda", generator=g)
    f = lambda *s: torch.complex(r(*s), r(*s)) if cplx else r(*s)
    A, B = f(M, K), f(K, N)
    C = Engine.get(0).matmul(A, B)
    bound = 4 * (4 * K + 8) * np.finfo(float).eps * (A.abs() @ B.abs())
    assert bool(((C - A @ B).abs() <= bound).all())
