"""reno_lanczos_expm after an error: the start vector is the caller's only
copy, so a call that ends for want of Krylov vectors (after convergence
tests that formed approximations) leaves it bit for bit, and the second call
with more vectors gives what one call with enough of them gives."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _problem():
    from renormalizer_b200._native import HeffDesc
    m = 40
    g = torch.Generator(device="cuda").manual_seed(2)
    A = torch.randn(m, m, dtype=torch.float64, device="cuda", generator=g)
    L = ((A + A.T) * 10).to(torch.complex128).reshape(m, 1, m).contiguous()
    R = torch.ones((1, 1, 1), dtype=torch.complex128, device="cuda")
    psi = torch.complex(torch.randn(m, dtype=torch.float64, device="cuda", generator=g),
                        torch.randn(m, dtype=torch.float64, device="cuda", generator=g))
    d = HeffDesc(nsite=0, ml=m, mr=1, wl=1, wm=1, wr=1, d1=1, d2=1, psi_dtype=1, env_dtype=1, mpo_dtype=0, prec=0)
    return d, L, R, psi


def _call(d, L, R, psi, out, kmax, dt):
    from renormalizer_b200._native import Engine, load_library
    lib, eng = load_library(), Engine.get(0)
    n = ctypes.c_size_t()
    assert lib.reno_lanczos_workspace_bytes(ctypes.byref(d), kmax, ctypes.byref(n)) == 0
    ws = torch.empty(n.value, dtype=torch.uint8, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    k = ctypes.c_int32(0)
    head = (eng.ctx, ctypes.byref(d), p(L), None, None, p(R), 0.0, dt)
    tail = (kmax, ctypes.byref(k), p(ws), n.value)
    if out is None:
        st = lib.reno_lanczos_expm(*head, p(psi), *tail)
    else:
        st = lib.reno_lanczos_expm_to(*head, p(psi), p(out), *tail)
    torch.cuda.synchronize()
    return st, k.value


@pytest.mark.parametrize("kmax", [7, 8, 9, 12])
def test_start_vector_survives_too_few_vectors(kmax):
    from renormalizer_b200._native import RENO_ERR_WORKSPACE
    d, L, R, psi = _problem()
    start, ref = psi.clone(), torch.empty_like(psi)
    assert _call(d, L, R, psi, ref, 60, -1.0)[0] == 0 and torch.equal(psi, start)
    assert _call(d, L, R, psi, None, kmax, -1.0)[0] == RENO_ERR_WORKSPACE
    assert torch.equal(psi, start)
    out = torch.empty_like(psi)
    assert _call(d, L, R, psi, out, kmax, -1.0)[0] == RENO_ERR_WORKSPACE and torch.equal(psi, start)
    assert _call(d, L, R, psi, None, 60, -1.0)[0] == 0
    assert torch.equal(psi, ref)


def test_in_place_equals_separate_output():
    """an exponential that converges at a test (a small step) and one that exhausts its space"""
    for dt in (-1e-3, -1.0):
        d, L, R, psi = _problem()
        out = torch.empty_like(psi)
        st, k = _call(d, L, R, psi, out, 60, dt)
        assert st == 0
        assert _call(d, L, R, psi, None, 60, dt) == (0, k) and torch.equal(psi, out)
