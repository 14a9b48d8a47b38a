"""Exponentials that need more Krylov vectors than one workspace holds go on in
a larger one: bit for bit the result and the count of a call with enough
vectors, without a second matvec for any vector."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _problem(prec="fp64"):
    from renormalizer_b200.hop_expr import HeffOperator
    g = torch.Generator(device="cuda").manual_seed(5)
    c = lambda *s: torch.complex(*torch.randn((2,) + s, dtype=torch.float64, device="cuda", generator=g))
    L, R = c(20, 3, 20), c(17, 3, 17)
    W = [torch.randn(3, 4, 4, 3, dtype=torch.float64, device="cuda", generator=g) for _ in range(2)]
    op = HeffOperator((L + L.transpose(0, 2).conj()) / 2, (R + R.transpose(0, 2).conj()) / 2,
                      [w + w.transpose(1, 2) for w in W], (20, 4, 4, 17), prec=prec)
    v = c(20 * 16 * 17)
    return op, v / torch.linalg.vector_norm(v)


@pytest.mark.parametrize("prec", ["fp64", "bf16x3"])
@pytest.mark.parametrize("block", [1, 5, 7, 50])
def test_resumed_equals_one_call(block, prec):
    from renormalizer_b200._native import launch_count
    from renormalizer_b200.krylov import expm_krylov
    op, v = _problem(prec)
    dt = -0.07j  # 50 .. 200 vectors
    runs = []
    for b in (400, block):
        torch.cuda.synchronize()
        n0, m0 = launch_count(), op.engine.launches
        y, k = expm_krylov(op, dt, v, b)
        runs.append((y, k, launch_count() - n0, op.engine.launches - m0))
    (y1, k1, l1, m1), (y2, k2, l2, m2) = runs
    assert 50 < k1 < 400 and k1 == k2 == m1 == m2 and torch.equal(y1, y2)
    # each call transposes (and, in split precision, packs) the constant operands once more: at most 8 launches
    assert l2 <= l1 + 8 * (k1 // block)


def test_resume_through_the_c_entry():
    from renormalizer_b200._native import RENO_ERR_INVALID, RENO_ERR_WORKSPACE, ptr
    op, v = _problem()
    lib, ctx, d = op.engine.lib, op.engine.ctx, op.desc
    d.psi_dtype = 1
    head = (ctx, ctypes.byref(d), ptr(op.L), ptr(op.W[0]), ptr(op.W[1]), ptr(op.R), 0.0, -0.07)

    def space(kmax):
        n = ctypes.c_size_t()
        assert lib.reno_lanczos_workspace_bytes(ctypes.byref(d), kmax, ctypes.byref(n)) == 0
        return torch.empty(n.value, dtype=torch.uint8, device="cuda")

    k, ref, psi = ctypes.c_int32(-1), torch.empty_like(v), v.clone()
    big, small, mid = space(400), space(9), space(30)
    assert lib.reno_lanczos_expm_to(*head, ptr(v), ptr(ref), 400, ctypes.byref(k), ptr(big), big.numel()) == 0
    kref = k.value
    assert lib.reno_lanczos_expm(*head, ptr(psi), 9, ctypes.byref(k), ptr(small), small.numel()) == RENO_ERR_WORKSPACE
    assert k.value == 9 and torch.equal(psi, v)
    for kmax, prev in ((9, small), (5, small)):  # no more vectors than before
        assert lib.reno_lanczos_expm_resume(*head, ptr(psi), kmax, 9, ptr(prev), ctypes.byref(k), ptr(mid),
                                            mid.numel()) == RENO_ERR_INVALID
    st = lib.reno_lanczos_expm_resume(*head, ptr(psi), 30, 9, ptr(small), ctypes.byref(k), ptr(mid), 1000)
    assert st == RENO_ERR_WORKSPACE and k.value == 0
    assert lib.reno_lanczos_expm_resume(*head, ptr(psi), 30, 9, ptr(small), ctypes.byref(k), ptr(mid),
                                        mid.numel()) == RENO_ERR_WORKSPACE and k.value == 30
    assert lib.reno_lanczos_expm_resume(*head, ptr(psi), 400, 30, ptr(mid), ctypes.byref(k), ptr(big),
                                        big.numel()) == 0
    assert k.value == kref and torch.equal(psi, ref)
