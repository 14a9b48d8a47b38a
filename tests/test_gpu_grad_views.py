"""Gradients of the effective-Hamiltonian matvec where the operands of its
contractions change between being read in place and being copied: extents of one
(a stride that does not matter), ragged sizes, real and complex operands mixed.
Reference: torch's own derivative of the plain contraction on the CPU.  Bound:
chains of FP64 sums of at most 2000 terms, 1e-12 of the largest entry."""
import pytest
import torch

pytestmark = pytest.mark.gpu

EINSUM = ["abc,lbk,ck->al", "abc,bdef,lfk,cek->adl", "abc,bdef,fghj,ljk,cehk->adgl"]


@pytest.mark.parametrize("cplx", [(True, True), (False, True), (True, False), (False, False)])
@pytest.mark.parametrize("nsite,ml,mr,d1,d2,wl,wm,wr", [
    (0, 1, 1, 1, 1, 1, 1, 1), (0, 7, 7, 1, 1, 3, 1, 3), (0, 1, 9, 1, 1, 2, 1, 2),
    (1, 1, 1, 1, 1, 1, 1, 1), (1, 1, 17, 4, 1, 1, 1, 3), (1, 13, 1, 3, 1, 3, 1, 1), (1, 9, 11, 1, 1, 2, 1, 4),
    (1, 8, 16, 5, 1, 1, 1, 1),
    (2, 1, 1, 1, 1, 1, 1, 1), (2, 1, 12, 2, 3, 1, 4, 2), (2, 11, 1, 3, 2, 2, 4, 1), (2, 9, 8, 1, 4, 2, 1, 3),
    (2, 7, 9, 3, 1, 2, 3, 1),
])
def test_gradients_of_every_operand(nsite, ml, mr, d1, d2, wl, wm, wr, cplx):
    from renormalizer_b200.autodiff import heff
    g = torch.Generator().manual_seed(ml * 100 + mr + nsite)
    env_c, psi_c = cplx

    def t(shape, c):
        return torch.randn(shape, dtype=torch.complex128 if c else torch.float64, generator=g)

    if nsite == 0:
        wr = wl
        Ws, ps = [], (ml, mr)
    elif nsite == 1:
        Ws, ps = [t((wl, d1, d1, wr), False)], (ml, d1, mr)
    else:
        Ws, ps = [t((wl, d1, d1, wm), False), t((wm, d2, d2, wr), False)], (ml, d1, d2, mr)
    cpu = [t((ml, wl, ml), env_c)] + Ws + [t((mr, wr, mr), env_c), t(ps, psi_c)]
    gy = t(ps, env_c or psi_c)

    ref = [x.clone().requires_grad_(True) for x in cpu]
    ctype = torch.complex128 if env_c or psi_c else torch.float64
    y = torch.einsum(EINSUM[nsite], *[x.to(ctype) for x in ref])
    y.backward(gy)

    dev = [x.cuda().requires_grad_(True) for x in cpu]
    out = heff(dev[-1], dev[0], dev[1:-2], dev[-2])
    out.backward(gy.cuda())
    for a, b in zip(dev, ref):
        assert a.grad.shape == b.grad.shape and a.grad.dtype == b.grad.dtype
        assert float((a.grad.cpu() - b.grad).abs().max()) <= 1e-12 * max(float(b.grad.abs().max()), 1e-300)
