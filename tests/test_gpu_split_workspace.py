"""The split-precision chains in a workspace from a caller's own pool: the
planes' stores are chosen by address, so a workspace aligned to 16 bytes only
(a sector and a half from the last boundary, what the tensor maps ask for)
gives the bits of an aligned one.  Row pitches of whole and of half sectors,
runs that fill a store and runs that do not."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("cplx", [True, False])
@pytest.mark.parametrize("nsite,ml,mr,d1,d2,wl,wm,wr", [
    (2, 6, 136, 16, 16, 2, 3, 2), (2, 5, 40, 16, 8, 3, 3, 3), (2, 4, 20, 24, 5, 5, 1, 2), (1, 9, 48, 16, 1, 3, 1, 3),
    (1, 12, 33, 8, 1, 5, 1, 1),
])
def test_workspace_at_sixteen_bytes(nsite, ml, mr, d1, d2, wl, wm, wr, cplx, prec):
    from renormalizer_b200._native import Engine, HeffDesc, load_library
    lib, eng = load_library(), Engine.get(0)
    g = torch.Generator(device="cuda").manual_seed(ml * 100 + mr)
    r = lambda *s: torch.randn(s, dtype=torch.float64, device="cuda", generator=g)
    f = lambda *s: torch.complex(r(*s), r(*s)) if cplx else r(*s)
    L, R, psi = f(ml, wl, ml), f(mr, wr, mr), f(*((ml, d1, d2, mr) if nsite == 2 else (ml, d1, mr)))
    W1 = r(wl, d1, d1, wm if nsite == 2 else wr)
    W2 = r(wm, d2, d2, wr) if nsite == 2 else None
    d = HeffDesc(nsite=nsite, ml=ml, mr=mr, wl=wl, wm=wm, wr=wr, d1=d1, d2=d2, psi_dtype=int(cplx),
                 env_dtype=int(cplx), mpo_dtype=0, prec=prec)
    n = ctypes.c_size_t()
    assert lib.reno_heff_workspace_bytes(ctypes.byref(d), ctypes.byref(n)) == 0
    pool = torch.zeros(n.value + 512, dtype=torch.uint8, device="cuda")
    assert pool.data_ptr() % 256 == 0
    ys = []
    for off in (0, 16, 32, 48):
        y = torch.empty_like(psi)
        st = lib.reno_heff_apply(eng.ctx, ctypes.byref(d), _p(L), _p(W1), _p(W2), _p(R), _p(psi), _p(y),
                                 ctypes.c_void_p(pool.data_ptr() + off), n.value)
        assert st == 0, lib.reno_last_error(eng.ctx)
        torch.cuda.synchronize()
        ys.append(y)
    assert bool((ys[0] != 0).any())
    for y in ys[1:]:
        assert torch.equal(y, ys[0])
