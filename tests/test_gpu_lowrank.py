"""The truncation through a block's numerical range (heev.LowRankOptions)
against the dense device eigensolver's route and against torch's SVD.

Blocks sit at the route's edges: the smallest order it takes and one below,
the kept side the smaller, the larger and an equal one, real and complex, one
block that takes it beside one that does not, a spectrum that passes the
probe but not the checks (redone by the dense path) and a flat one (never
tried).  The singular values leave a factor 10 at the cut, at 1e-2 of the
largest: with a backward error of b = 1e-13 lambda_1 (the checks' 2e-14 plus
n eps) the kept space turns by at most 2 b / (0.99e-4 lambda_1) = 2e-9, so the
truncated coefficient moves by less than 1e-2 2e-9 sqrt(keep) < 1e-9 of its
norm, and the kept sigma by less than that squared; 1e-12 of sigma_1 for them
is rounding of the products."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

svd_qn = importlib.import_module("renormalizer_b200.svd_qn")
heev = importlib.import_module("renormalizer_b200.heev")


def _block(m, n, spectrum, keep, cplx, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(s, dtype=torch.float64, device="cuda", generator=g)
    f = lambda *s: torch.complex(r(*s), r(*s)) if cplx else r(*s)
    k = min(m, n)
    j = torch.arange(k, dtype=torch.float64, device="cuda")
    if spectrum == "decay":    # 1 .. 1e-2 over the kept, 1e-3 and 12 more decades over the next 3 keep / 2
        s = torch.where(j < keep, 10.0 ** (-2.0 * j / keep), 10.0 ** (-3.0 - 12.0 * (j - keep) / (1.5 * keep)))
    elif spectrum == "shelf":  # falls like the above, then stays at 1e-5
        s = torch.where(j < keep, 10.0 ** (-2.0 * j / keep), torch.full_like(j, 1e-5))
        s[8:keep] *= 0.5
    else:
        s = 1.0 + 0.5 * torch.cos(j)
        s, _ = torch.sort(s, descending=True)
        s[keep:] *= 0.1
    U, _ = torch.linalg.qr(f(m, k))
    V, _ = torch.linalg.qr(f(n, k))
    return (U * s) @ V.mH


def _truncate(X, keep, keep_left):
    m, n = X.shape
    return svd_qn.svd_truncate(X, np.zeros((m, 1), int), np.zeros((n, 1), int), np.array([0]), keep_left,
                               lambda s: min(keep, len(s)), kcap=keep)


# m, n, keep, spectrum, calls, missed (None: the kept values fall too slowly over the probe's columns for it to say)
CASES = [
    (480, 500, 32, "decay", 1, 0), (479, 500, 32, "decay", 0, 0), (480, 480, 32, "decay", 1, 0),
    (900, 600, 64, "decay", None, None), (600, 1111, 64, "decay", None, None), (700, 640, 32, "shelf", 1, 1),
    (640, 640, 32, "flat", 0, 0)]


@pytest.mark.parametrize("cplx", [True, False])
@pytest.mark.parametrize("keep_left", [True, False])
@pytest.mark.parametrize("m,n,keep,spectrum,calls,missed", CASES)
def test_lowrank_truncation(m, n, keep, spectrum, calls, missed, keep_left, cplx):
    X = _block(m, n, spectrum, keep, cplx, seed=m + n)
    c0, m0, f0 = heev.lowrank_opts.calls, heev.lowrank_opts.missed, heev.heev_opts.fallbacks
    res = _truncate(X, keep, keep_left)
    if calls is not None:
        assert (heev.lowrank_opts.calls - c0, heev.lowrank_opts.missed - m0) == (calls, missed)
    assert heev.heev_opts.fallbacks == f0
    U, S, Vh = torch.linalg.svd(X, full_matrices=False)
    ref = (U[:, :keep] * S[:keep]) @ Vh[:keep]
    assert float(torch.linalg.vector_norm(res.left @ res.right - ref)) <= 1e-9 * float(torch.linalg.vector_norm(ref))
    assert np.abs(res.sigma - S[:keep].cpu().numpy()).max() <= 1e-12 * float(S[0])
    kept = res.left if keep_left else res.right.mH
    eye = torch.eye(keep, dtype=kept.dtype, device="cuda")
    assert float((kept.mH @ kept - eye).abs().max()) <= 1e-12


def test_lowrank_beside_dense_block():
    """two sectors, only one of them large enough"""
    A, B = _block(700, 640, "decay", 32, True, 1), _block(300, 330, "decay", 32, True, 2)
    X = torch.zeros((1000, 970), dtype=A.dtype, device="cuda")
    X[:700, :640], X[700:, 640:] = A, 0.7 * B
    ql, qr = np.repeat([0, 1], [700, 300]).reshape(-1, 1), np.repeat([1, 0], [640, 330]).reshape(-1, 1)
    c0 = heev.lowrank_opts.calls
    # both blocks' 32 kept values: the next ones are a factor 10 below the last of either
    res = svd_qn.svd_truncate(X, ql, qr, np.array([1]), True, lambda s: 64, kcap=64)
    assert heev.lowrank_opts.calls - c0 == 1
    ref = torch.zeros_like(X)
    for r, c in ((slice(0, 700), slice(0, 640)), (slice(700, 1000), slice(640, 970))):
        U, S, Vh = torch.linalg.svd(X[r, c], full_matrices=False)
        ref[r, c] = (U[:, :32] * S[:32]) @ Vh[:32]
    assert float(torch.linalg.vector_norm(res.left @ res.right - ref)) <= 1e-9 * float(torch.linalg.vector_norm(ref))
