"""The tiles and K splits of the FP64 GEMM against plain torch.

Each shape sits at an edge of one of the kernel's paths: 16 / 32 / 64 tiles,
one tile and one row or column past it, K shorter than a chunk, at a chunk
and one past it, and K long enough that a cluster of 2, 4 or 8 CTAs shares
it.  Every entry is a sum of c K products (c = 4 complex, 1 real), so both
sides are within (c K + 8) eps of the exact value relative to
sum |a| |b|; the tolerance is twice that.  A grouped matvec rounds like the
single one whatever paths its problems take, so those agree bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (16, 16, 15), (17, 15, 16), (16, 33, 17), (32, 32, 128), (31, 65, 257), (40, 50, 4096),
          (64, 320, 1500), (65, 63, 1023), (256, 640, 2048), (640, 64, 256), (1280, 1280, 48), (2049, 320, 64)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("ta", [False, True])
@pytest.mark.parametrize("types", ["cc", "rc", "cr", "rr"])
def test_gemm_tiles(shape, ta, types):
    from renormalizer_b200._native import Engine
    M, N, K = shape
    g = torch.Generator(device="cuda").manual_seed(M + 7 * N + 31 * K)

    def rnd(s, cplx):
        r = lambda: torch.randn(s, dtype=torch.float64, device="cuda", generator=g)
        return torch.complex(r(), r()) if cplx else r()

    A = rnd((K, M) if ta else (M, K), types[0] == "c")
    B = rnd((N, K) if ta else (K, N), types[1] == "c")
    A, B = (A.transpose(0, 1), B.transpose(0, 1)) if ta else (A, B)
    C = Engine.get(0).matmul(A, B, conj_a=ta)
    a = A.conj().resolve_conj() if ta else A
    dt = torch.complex128 if "c" in types else torch.float64
    ref = a.to(dt) @ B.to(dt)
    bound = 4 * (4 * K + 8) * np.finfo(float).eps * (A.abs() @ B.abs())
    assert bool(((C - ref).abs() <= bound).all())


def test_grouped_matvec_of_mixed_paths_is_each_ones_own():
    from renormalizer_b200.hop_expr import HeffOperator, apply_grouped
    g = torch.Generator(device="cuda").manual_seed(3)
    r = lambda *s: torch.randn(s, dtype=torch.float64, device="cuda", generator=g)
    c = lambda *s: torch.complex(r(*s), r(*s))
    ops, xs = [], []
    for ml, mr, d1, d2, w in ((1, 2, 2, 3, 2), (40, 33, 2, 10, 5), (97, 130, 3, 4, 5), (200, 16, 2, 2, 4)):
        L, R, W1, W2 = c(ml, w, ml), c(mr, w, mr), r(w, d1, d1, w), r(w, d2, d2, w)
        ops.append(HeffOperator(L, R, [W1, W2], (ml, d1, d2, mr), prec="fp64"))
        xs.append(c(ml, d1, d2, mr))
    for y, op, x in zip(apply_grouped(ops, xs), ops, xs):
        assert torch.equal(y, op.apply(x))
