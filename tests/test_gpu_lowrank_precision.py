"""The range route against the dense route on the same blocks: truncated
coefficients no further from torch's SVD, on the spectra of sweeps (a
decade every keep / 5 to keep / 7 values), a power law, a steep head before
a slow tail and one large value far ahead of the rest; and missed blocks of a batch in one dense call.

Both routes end in an eigenproblem with rounding at eps lambda_1, whose mixing
of kept and discarded vectors is the error; the range route adds nothing of
that size, so the two errors agree up to the scatter of rounding between two
orders of summation, for which 5 % are allowed."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

svd_qn = importlib.import_module("renormalizer_b200.svd_qn")
heev = importlib.import_module("renormalizer_b200.heev")


def _block(m, n, spectrum, keep, cplx, seed, digits=3.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(s, dtype=torch.float64, device="cuda", generator=g)
    f = lambda *s: torch.complex(r(*s), r(*s)) if cplx else r(*s)
    k = min(m, n)
    j = torch.arange(k, dtype=torch.float64, device="cuda")
    if spectrum == "exponential":
        s = 10.0 ** (-digits * j / keep)
        return (f(m, k) * s) @ f(k, n) / np.sqrt(m * n)
    if spectrum == "power":
        s = 1.0 / (1.0 + j) ** 2
    elif spectrum == "head":
        s = torch.where(j < 30, 10.0 ** (-j / 10.0), 1e-3 / (1.0 + (j - 30)) ** 1.5)
    else:  # one value, then eight decades lower
        s = torch.where(j < 1, torch.ones_like(j), 1e-8 * 10.0 ** (-3.0 * j / keep))
    U, _ = torch.linalg.qr(f(m, k))
    V, _ = torch.linalg.qr(f(n, k))
    return (U * s) @ V.mH


def _truncate(X, keep, keep_left):
    m, n = X.shape
    return svd_qn.svd_truncate(X, np.zeros((m, 1), int), np.zeros((n, 1), int), np.array([0]), keep_left,
                               lambda s: min(keep, len(s)), kcap=keep)


@pytest.mark.parametrize("m,n,spectrum,keep,cplx,keep_left,digits", [
    (1540, 1196, "exponential", 110, False, True, 3.54), (798, 1440, "exponential", 96, True, False, 3.31),
    (981, 747, "exponential", 108, True, True, 3.69), (972, 840, "exponential", 105, False, False, 2.88),
    (1196, 1540, "exponential", 110, False, False, 3.54), (600, 620, "exponential", 62, True, True, 2.54),
    (640, 700, "power", 32, True, True, 0), (800, 800, "head", 64, False, False, 0), (700, 640, "one", 40, True, False, 0),
])
def test_no_further_from_64_bits_than_the_dense_route(m, n, spectrum, keep, cplx, keep_left, digits):
    X = _block(m, n, spectrum, keep, cplx, m + n, digits)
    U, S, Vh = torch.linalg.svd(X, full_matrices=False)
    ref = (U[:, :keep] * S[:keep]) @ Vh[:keep]
    err = []
    ratio = heev.lowrank_opts.min_ratio
    for r in (ratio, 1e9):
        heev.lowrank_opts.min_ratio = r
        try:
            res = _truncate(X, keep, keep_left)
        finally:
            heev.lowrank_opts.min_ratio = ratio
        err.append(float(torch.linalg.vector_norm(res.left @ res.right - ref)))
    assert err[0] <= 1.05 * err[1] + 1e-15 * float(S[0])


def test_missed_blocks_share_one_dense_call(monkeypatch):
    """three truncations whose block passes the probe and misses the check"""
    calls = []
    orig = heev.heev_top_batched
    monkeypatch.setattr(heev, "heev_top_batched", lambda eng, Gs, kts: (calls.append([G.shape[0] for G in Gs]),
                                                                       orig(eng, Gs, kts))[1])
    keep, args, refs = 32, [], []
    for seed in (1, 2, 3):
        g = torch.Generator(device="cuda").manual_seed(seed)
        j = torch.arange(640, dtype=torch.float64, device="cuda")
        s = torch.where(j < keep, 10.0 ** (-2.0 * j / keep), torch.full_like(j, 1e-5))
        s[8:keep] *= 0.5
        c = lambda a, b: torch.complex(*torch.randn((2, a, b), dtype=torch.float64, device="cuda", generator=g))
        X = (torch.linalg.qr(c(700, 640))[0] * s) @ torch.linalg.qr(c(640, 640))[0].mH
        args.append(dict(coef=X, qnbigl=np.zeros((700, 1), int), qnbigr=np.zeros((640, 1), int), qntot=np.array([0]),
                         keep_left=True, m_trunc_fn=lambda s: keep, kcap=keep))
        U, S, Vh = torch.linalg.svd(X, full_matrices=False)
        refs.append((U[:, :keep] * S[:keep]) @ Vh[:keep])
    c0, m0 = heev.lowrank_opts.calls, heev.lowrank_opts.missed
    got = svd_qn.svd_truncate_batch(args)
    assert (heev.lowrank_opts.calls - c0, heev.lowrank_opts.missed - m0) == (3, 3)
    assert calls == [[640] * 3]
    for res, ref in zip(got, refs):
        assert float(torch.linalg.vector_norm(res.left @ res.right - ref)) <= 1e-9 * float(torch.linalg.vector_norm(ref))


@pytest.mark.parametrize("other,tried", [(640, 0), (520, 0), (500, 1)])
def test_range_route_beside_a_dense_block(other, tried):
    """a block beside one that the probe refuses: left to the dense reduction that runs anyway, unless that
    one is of less than 0.8 the order; the same in a batch with another truncation whose blocks both qualify"""
    keep, n = 32, 640
    A = _block(n, n, "exponential", keep, True, 5)
    g = torch.Generator(device="cuda").manual_seed(9)
    F = torch.complex(*torch.randn((2, other, other), dtype=torch.float64, device="cuda", generator=g)) / other
    X = torch.zeros((n + other, n + other), dtype=A.dtype, device="cuda")
    X[:n, :n], X[n:, n:] = A, F
    Y = torch.zeros((2 * n, 2 * n), dtype=A.dtype, device="cuda")
    Y[:n, :n], Y[n:, n:] = A, 0.5 * A
    job = lambda Z, k: dict(coef=Z, qnbigl=np.repeat([0, 1], [n, k]).reshape(-1, 1),
                            qnbigr=np.repeat([1, 0], [n, k]).reshape(-1, 1), qntot=np.array([1]), keep_left=True,
                            m_trunc_fn=lambda s: 2 * keep, kcap=2 * keep)
    c0 = heev.lowrank_opts.calls
    alone = svd_qn.svd_truncate(**job(X, other))
    assert heev.lowrank_opts.calls - c0 == tried
    both = svd_qn.svd_truncate_batch([job(Y, n), job(X, other)])
    assert heev.lowrank_opts.calls - c0 == 2 * tried + 2
    ref = alone.left @ alone.right
    assert float(torch.linalg.vector_norm(both[1].left @ both[1].right - ref)) <= 1e-12 * float(torch.linalg.vector_norm(ref))
