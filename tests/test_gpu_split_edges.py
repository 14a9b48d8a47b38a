"""Packing and output edges of the split-precision path.

Packing: a 32 x 64 block whose values all lie well inside FP32's range is
rounded to its BF16 pairs in integer operations, any other block by the
conversion instructions.  The same rows packed beside an ordinary row and
beside a row of 1e-25 take one and the other; the products have to agree bit
by bit (equal pairs, equal products), halfway cases and zeros included.

Outputs: matvec shapes whose runs and tiles end inside a 16-column run, a
32-byte store or a 256-column tile, against FP64.  The bound is the split
chain's: 4 GEMMs of relative error 5e-5 (a 17-bit pair, lo * lo dropped, FP32
accumulation), grown with sqrt(K / 256) for the longest contraction."""
import numpy as np
import pytest
import torch

from oracle import reno_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 63, 64, 65, 129])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("view", ["rows", "columns", "conj"])
def test_integer_packing_rounds_as_the_conversions(k, cplx, view):
    from renormalizer_b200._native import Engine
    rng = np.random.default_rng(k)
    m = 31

    def draw():
        x = rng.standard_normal((m, k)) * 10.0 ** rng.uniform(-15, 3, (m, k))
        x[rng.random((m, k)) < 0.1] = 0.0
        ties = np.ldexp(1.0 + rng.integers(0, 128, (m, k)) / 128.0 + 1.0 / 256.0, 3)  # halfway between two BF16 numbers
        x = np.where(rng.random((m, k)) < 0.1, ties, x)
        return np.where(rng.random((m, k)) < 0.05, np.nextafter(ties, 0.0), x)

    a = draw() + 1j * draw() if cplx else draw()
    b = torch.from_numpy(rng.standard_normal((k, 40))).cuda()
    eng, got = Engine.get(0), []
    for last in (1.0, 1e-25):
        dev = torch.from_numpy(np.concatenate([a, np.full((1, k), last)])).cuda()
        if view == "columns":
            dev = dev.t().contiguous().t()
        got.append(eng.matmul(dev, b, conj_a=view == "conj", prec="bf16x3")[:m].cpu().numpy())
    np.testing.assert_array_equal(got[0], got[1])


@pytest.mark.parametrize("prec,tol", [("bf16x3", 5e-5), ("tf32x3", 5e-6)])
@pytest.mark.parametrize("cplx", [True, False])
@pytest.mark.parametrize("ml,mr,d1,d2,wl,wm,wr", [
    (3, 136, 10, 6, 3, 5, 4),     # runs of 10 and 6; 136 = 128 + 8 columns, complex ones past a tile
    (5, 192, 16, 16, 2, 3, 2),    # a tile half of whose columns lie past the operand
    (4, 129, 16, 3, 2, 2, 3),     # odd row lengths: no 32-byte aligned run
    (2, 17, 5, 16, 3, 4, 1),
    (1, 1, 2, 2, 1, 2, 1),
])
def test_fused_matvec_output_edges(prec, tol, cplx, ml, mr, d1, d2, wl, wm, wr):
    from renormalizer_b200.hop_expr import HeffOperator
    rng = np.random.default_rng(ml * 1000 + mr)

    def t(*shape):
        x = rng.standard_normal(shape)
        return x + 1j * rng.standard_normal(shape) if cplx else x

    L, R, psi = t(ml, wl, ml), t(mr, wr, mr), t(ml, d1, d2, mr)
    w1, w2 = rng.standard_normal((wl, d1, d1, wm)), rng.standard_normal((wm, d2, d2, wr))
    op = HeffOperator(L, R, [w1, w2], psi.shape, prec=prec)
    y = op(torch.from_numpy(psi).cuda()).cpu().numpy()
    ref = O.hop(L, [w1, w2], R, psi)
    scale = max(1.0, np.sqrt(max(2 * ml, 2 * wr * mr, wl * d1, wm * d2) / 256.0))
    assert np.abs(y - ref).max() < 4 * tol * scale * np.abs(ref).max()
