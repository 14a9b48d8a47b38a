"""Eigenvalues far below the norm, where the reduction is exact (diagonal
matrices, 2 x 2 blocks on the diagonal): bisection finds each to 2 ulp of its own
size down to 1e-43 of the norm, with a count that sees couplings and exact
zeros there.  Bound: 2 ulp of the bracket, one of its middle and one of the reference: 4 ulp."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def _top(G, kt):
    from renormalizer_b200._native import Engine
    from renormalizer_b200.heev import heev_top
    return heev_top(Engine.get(0), torch.from_numpy(G.astype(complex)).cuda(), kt)[0].cpu().numpy()


@pytest.mark.parametrize("n", [2, 9, 64, 130, 300, 430])
@pytest.mark.parametrize("scale", [1.0, 3e-60, 7e80])
def test_graded_diagonal(n, scale):
    d = scale * 10.0 ** np.linspace(0, -43, n)
    w = _top(np.diag(np.random.default_rng(n).permutation(d)), n)
    assert np.all(np.abs(w - d) <= 4 * EPS * d)


@pytest.mark.parametrize("n", [1, 3, 33])
def test_graded_pairs_and_zeros(n):
    """blocks s [[1, t], [t, 1]] with eigenvalues s (1 +- t), s over 30 decades, and as many zeros"""
    s, t = 10.0 ** np.linspace(0, -30, n), 0.25
    G = np.zeros((4 * n, 4 * n))
    for i, x in enumerate(s):
        G[2 * i:2 * i + 2, 2 * i:2 * i + 2] = [[x, t * x], [t * x, x]]
    ref = np.sort(np.concatenate([s * (1 + t), s * (1 - t)]))[::-1]
    w = _top(G, 4 * n)
    assert np.all(np.abs(w[:2 * n] - ref) <= 4 * EPS * ref)
    assert np.all(np.abs(w[2 * n:]) <= 1e-50)
