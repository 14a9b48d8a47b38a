"""The MPO stage kernel (matvecs and environment updates with a million
elements or more of the first intermediate) against torch's einsum.

Sparse, dense and all-zero MPO tensors, complex and real operands, even and
odd column counts (copies of two real elements or of one), the last tile
full and of one column, more rows than warps and fewer.  Each output is a
contraction of at most K = ml wl + wl d + wr d + mr wr products per level, so
1e-12 of max|y| holds like for every FP64 matvec.  Where psi holds an infinity
or NaN the result has to be non-finite exactly where the full contraction's
is."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
HOP = {1: "abc,bdef,lfk,cek->adl", 2: "abc,bdef,fghj,ljk,cehk->adgl"}


def _hop(L, Ws, R, psi):
    dt = psi.dtype
    t = torch.einsum("abc,c...->ab...", L, psi)
    t = torch.einsum("abe...,bdef->adf...", t, Ws[0].to(dt))
    if len(Ws) == 1:
        return torch.einsum("adfk,lfk->adl", t, R)
    t = torch.einsum("adfhk,fghj->adgjk", t, Ws[1].to(dt))
    return torch.einsum("adgjk,ljk->adgl", t, R)


def _case(nsite, ml, mr, w, d, kind, cplx, seed=1):
    g = torch.Generator(device="cuda").manual_seed(seed + ml + mr)
    r = lambda *s: torch.randn(s, dtype=torch.float64, device="cuda", generator=g)
    f = lambda *s: torch.complex(r(*s), r(*s)) if cplx else r(*s)
    Ws = []
    for _ in range(nsite):
        W = r(w, d, d, w)
        if kind == "sparse":
            W = W * (torch.rand(W.shape, device="cuda", generator=g) < 0.03)
        elif kind == "zero":
            W = W * 0.0
        Ws.append(W.contiguous())
    return f(ml, w, ml), Ws, f(mr, w, mr), f(ml, *([d] * nsite), mr)


@pytest.mark.parametrize("cplx", [True, False])
@pytest.mark.parametrize("kind", ["sparse", "dense", "zero"])
@pytest.mark.parametrize("nsite,ml,mr,w,d", [(1, 160, 129, 5, 16), (1, 190, 161, 4, 10), (2, 65, 31, 5, 16),
                                             (2, 128, 65, 3, 8), (2, 300, 97, 3, 2)])
def test_matvec(nsite, ml, mr, w, d, kind, cplx):
    from renormalizer_b200.hop_expr import HeffOperator
    L, Ws, R, psi = _case(nsite, ml, mr, w, d, kind, cplx)
    assert ml * w * psi[0].numel() >= 1 << 20 or d == 2
    y = HeffOperator(L, R, Ws, psi.shape, prec="fp64")(psi)
    ref = _hop(L, Ws, R, psi)
    assert float((y - ref).abs().max()) <= 1e-12 * max(float(ref.abs().max()), 1e-300)


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("cplx", [True, False])
def test_nonfinite_reaches_what_the_full_contraction_says(bad, cplx):
    from renormalizer_b200.hop_expr import HeffOperator
    L, Ws, R, psi = _case(2, 65, 31, 5, 16, "sparse", cplx)
    psi[3, 2, 7, 30] = bad
    y = HeffOperator(L, R, Ws, psi.shape, prec="fp64")(psi)
    # every product of the row meets the entry: a zero times it is a NaN, so nothing of y stays finite
    assert not bool(torch.isfinite(torch.view_as_real(y) if cplx else y).any())


@pytest.mark.parametrize("domain", ["L", "R"])
def test_environment_update(domain):
    from renormalizer_b200 import contract_one_site
    L, Ws, R, psi = _case(1, 160, 129, 5, 16, "sparse", True)
    E, W = (L, Ws[0]) if domain == "L" else (R, Ws[0])
    out = contract_one_site(E, psi, W, domain, prec="fp64")
    Wc = W.to(psi.dtype)
    if domain == "L":
        t = torch.einsum("abc,ceh->abeh", E, psi)
        t = torch.einsum("abeh,bdeg->adgh", t, Wc)
        ref = torch.einsum("adf,adgh->fgh", psi.conj(), t)
    else:
        t = torch.einsum("abc,hec->abeh", E, psi)
        t = torch.einsum("abeh,gdeb->adgh", t, Wc)
        ref = torch.einsum("fda,adgh->fgh", psi.conj(), t)
    assert float((out - ref).abs().max()) <= 1e-12 * float(ref.abs().max())


def test_grouped_is_each_ones_own():
    from renormalizer_b200.hop_expr import HeffOperator, apply_grouped
    ops, xs = [], []
    for ml, mr in ((65, 31), (4, 5), (90, 40)):
        L, Ws, R, psi = _case(2, ml, mr, 5, 16, "sparse", True)
        ops.append(HeffOperator(L, R, Ws, psi.shape, prec="fp64"))
        xs.append(psi)
    for y, op, x in zip(apply_grouped(ops, xs), ops, xs):
        assert torch.equal(y, op.apply(x))
