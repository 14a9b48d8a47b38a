"""Every instance of the MPO stage kernel, at the limits of its tile widths,
against torch's einsum.

A tile holds 32, 64 or 128 columns of Q = w d rows, the widest of which two
stages fit 112 KB: complex 64 up to Q = 46 and 32 up to 90, real 128 up to 46, 64
up to 90 and 32 up to 170.  Also six output rows, fewer than the kernel's
eight warps, and a stage beyond the limit (the GEMM's).  Each output is a
contraction of at most K = ml w + w d + mr w products per level, so 1e-12 of
max|y| holds like for every FP64 matvec."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cplx", [True, False])
@pytest.mark.parametrize("sparse", [True, False])
@pytest.mark.parametrize("ml,mr,w,d", [(600, 300, 3, 2), (256, 129, 23, 2), (256, 129, 47, 1), (160, 129, 10, 9),
                                       (160, 129, 13, 7), (128, 129, 8, 16), (128, 97, 10, 17), (128, 97, 9, 19)])
def test_one_site(ml, mr, w, d, sparse, cplx):
    from renormalizer_b200.hop_expr import HeffOperator
    assert ml * w * d * mr >= 1 << 20  # the kernel's smallest T1
    g = torch.Generator(device="cuda").manual_seed(ml + w + d)
    r = lambda *s: torch.randn(s, dtype=torch.float64, device="cuda", generator=g)
    f = lambda *s: torch.complex(r(*s), r(*s)) if cplx else r(*s)
    L, R, psi, W = f(ml, w, ml), f(mr, w, mr), f(ml, d, mr), r(w, d, d, w)
    if sparse:
        W = W * (torch.rand(W.shape, device="cuda", generator=g) < 0.03)
    y = HeffOperator(L, R, [W], psi.shape, prec="fp64")(psi)
    t = torch.einsum("abc,cek->abek", L, psi)
    t = torch.einsum("abek,bdef->adfk", t, W.to(psi.dtype))
    ref = torch.einsum("adfk,lfk->adl", t, R)
    assert float((y - ref).abs().max()) <= 1e-12 * max(float(ref.abs().max()), 1e-300)
