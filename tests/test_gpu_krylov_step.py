"""One Lanczos step (RENO_VOP_STEP) and the convergence check
(RENO_VOP_CHECK) against plain torch, at the edges of the cluster kernel:
fewer elements than CTAs, one per thread and one over, the longest vector a
cluster holds and the first that takes the separate operations.

Every scalar is a sum of at most 2 n products, so it is within
(2 n + 16) eps of the exact value relative to the sum of their magnitudes;
the vector entries follow by one division.  A batch must give each item the
bits of its own call."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def _state(n, cplx, j, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(s, dtype=torch.float64, device="cuda", generator=g)
    f = lambda *s: torch.complex(r(*s), r(*s)) if cplx else r(*s)
    V = f(4, n)
    V = V / torch.linalg.vector_norm(V, dim=1, keepdim=True)
    ab = torch.zeros(8, dtype=torch.float64, device="cuda")
    if j:
        ab[2 * j - 1] = 0.7
    return V.contiguous(), f(n), ab


def _item(V, w, ab, j):
    n = V.shape[1]
    return (n, 1 if V.is_complex() else 0, j, V[j], V[j - 1] if j else None, w, ab, None, n)


@pytest.mark.parametrize("cplx,n", [(True, 1), (True, 7), (True, 4096), (True, 4097), (True, 65536), (True, 65537),
                                    (False, 3), (False, 8 * 512 + 1), (False, 131072), (False, 131073)])
@pytest.mark.parametrize("j", [0, 2])
def test_step(n, cplx, j):
    from renormalizer_b200._native import Engine, VOP_STEP
    eng = Engine.get(0)
    V, w0, ab = _state(n, cplx, j, n + j)
    V1, ab1 = V.clone(), ab.clone()
    eng.vec_grouped(VOP_STEP, [_item(V1, w0.clone(), ab1, j)])
    tol = (2 * n + 16) * EPS
    alpha = torch.vdot(w0, V[j]).real
    w = w0 - alpha * V[j] - (0.7 * V[j - 1] if j else 0)
    beta = torch.linalg.vector_norm(w)
    assert abs(float(ab1[2 * j] - alpha)) <= tol * float((w0.abs() * V[j].abs()).sum())
    # an error of alpha moves w by it times v, and beta by at most as much
    da = tol * float((w0.abs() * V[j].abs()).sum())
    scale = float(w0.abs().max() + abs(alpha) * V[j].abs().max() + 0.7 * V[j - 1].abs().max() * bool(j))
    slack = da * float(V[j].abs().max()) + 8 * EPS * scale
    db = da + tol * float(beta)
    assert abs(float(ab1[2 * j + 1] - beta)) <= db
    got, ref = V1[j + 1], w / beta
    assert float((got - ref).abs().max()) <= (slack + db * float(ref.abs().max())) / float(beta) + 4 * EPS
    rows = [i for i in range(4) if i != j + 1]
    assert torch.equal(V1[rows], V[rows])


def test_step_batch_is_each_ones_own():
    from renormalizer_b200._native import Engine, VOP_STEP
    eng = Engine.get(0)
    sizes = [(3, True), (5000, True), (65536, True), (70000, True), (777, False), (140000, False)]
    sts = [_state(n, c, 1, n) for n, c in sizes]
    one = [(V.clone(), w.clone(), ab.clone()) for V, w, ab in sts]
    for V, w, ab in one:
        eng.vec_grouped(VOP_STEP, [_item(V, w, ab, 1)])
    eng.vec_grouped(VOP_STEP, [_item(V, w, ab, 1) for V, w, ab in sts])
    for (V, _, ab), (U, _, ac) in zip(sts, one):
        assert torch.equal(V, U) and torch.equal(ab, ac)


@pytest.mark.parametrize("n,cplx,k", [(1, True, 3), (1000, True, 5), (300001, True, 7), (4097, False, 9)])
def test_check(n, cplx, k):
    from renormalizer_b200._native import Engine, VOP_CHECK
    eng = Engine.get(0)
    g = torch.Generator(device="cuda").manual_seed(n)
    r = lambda *s: torch.randn(s, dtype=torch.float64, device="cuda", generator=g)
    V = torch.complex(r(k, n), r(k, n)) if cplx else r(k, n)
    for last, close in ((1e-9, 1.0), (1e-2, 0.0)):
        c = r(2 * k)
        c[2 * (k - 2):] = last
        if not cplx:
            c[1::2] = 0.0
        coef = torch.cat([c, c[: 2 * (k - 2)]]).contiguous()
        out, flag = torch.empty_like(V[0]), torch.full((1,), -1.0, dtype=torch.float64, device="cuda")
        eng.vec_grouped(VOP_CHECK, [(n, int(cplx), k, V, None, out, flag, coef, n)], 1e-5, 1e-7)
        cc = torch.complex(c[0::2], c[1::2]) if cplx else c[0::2]
        assert float((out - cc @ V).abs().max()) <= 4 * k * EPS * float((cc.abs() @ V.abs()).max())
        # 1e-9 of a few Gaussians is far inside atol, 1e-2 of them far outside for at least one element
        assert float(flag) == close
