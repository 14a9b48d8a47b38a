"""The eigensolver's stages at the sizes where they change form: one element,
one row per CTA, a CTA without rows, the sizes around one, two and three rows per
warp, the largest matrix of an 8- and of a 16-CTA cluster and the first beyond each, one
and two reflector blocks, split and repeated spectra, and mixed batches.

Bounds, relative to max |lambda|: the reduction and the bisection are backward
stable, with errors of a few n ulps (n <= 425: 1e-13), residuals and orthogonality
ten times that, as the solver's own acceptance test."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(G, kt, w, K, chk):
    from renormalizer_b200.heev import accepted
    assert accepted(chk.cpu().numpy()), chk.cpu().numpy()
    n = G.shape[0]
    ref = np.linalg.eigvalsh(G.cpu().numpy())[::-1][:kt]
    scale = max(float(np.abs(np.linalg.eigvalsh(G.cpu().numpy())).max()), 1e-300)
    assert np.abs(w.cpu().numpy() - ref).max() <= 1e-13 * scale
    Kc = K.to(torch.complex128).cpu().numpy()
    Gc = G.cpu().numpy()
    assert np.abs(Gc @ Kc - Kc * w.cpu().numpy()).max() <= 1e-12 * scale
    assert np.abs(Kc.conj().T @ Kc - np.eye(kt)).max() <= 1e-12
    assert K.shape == (n, kt)


def _gram(n, rng, kind):
    if kind == "generic":
        x = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
        g = x @ x.conj().T
    elif kind == "split":      # decoupled blocks, zero off-diagonals of T
        g = np.diag(rng.integers(1, 5, n).astype(float)).astype(complex)
        g[: n // 2, : n // 2] += np.ones((n // 2, n // 2))
    elif kind == "graded":     # twelve decades
        q = np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))[0]
        g = (q * 10.0 ** np.linspace(0, -12, n)) @ q.conj().T
        g = 0.5 * (g + g.conj().T)
    else:                      # far from 1 in size
        x = rng.standard_normal((n, n))
        g = (x @ x.T) * 1e-140
    return torch.from_numpy(np.ascontiguousarray(g)).cuda()


@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 9, 63, 64, 65, 66, 120, 121, 128, 129, 240, 241, 256, 257, 400, 424, 425])
def test_sizes(n):
    from renormalizer_b200._native import Engine
    from renormalizer_b200.heev import heev_top
    rng = np.random.default_rng(n)
    G = _gram(n, rng, "generic")
    for kt in {1, max(1, n // 3), n}:
        w, K, chk = heev_top(Engine.get(0), G, kt)
        _check(G, kt, w, K, chk)


@pytest.mark.parametrize("n", [10, 65, 130, 300])
def test_repeated_eigenvalues_of_a_split_matrix(n):
    """T falls apart into blocks (couplings of 0 and of rounding size) with
    eigenvalues of multiplicity ~n/4.  Every eigenvalue is found as often as
    it occurs; vectors of one T block in another's eigenvalue are what the acceptance
    test is for (it sends such a block to the dense solver)."""
    from renormalizer_b200._native import Engine
    from renormalizer_b200.heev import accepted, heev_top
    G = _gram(n, np.random.default_rng(n), "split")
    kt = max(1, n // 4)
    w, K, chk = heev_top(Engine.get(0), G, kt)
    ref = np.linalg.eigvalsh(G.cpu().numpy())[::-1]
    assert np.abs(w.cpu().numpy() - ref[:kt]).max() <= 1e-13 * np.abs(ref).max()
    if accepted(chk.cpu().numpy()):
        _check(G, kt, w, K, chk)


@pytest.mark.parametrize("kind", ["graded", "small"])
@pytest.mark.parametrize("n", [10, 65, 130, 300])
def test_spectra(n, kind):
    from renormalizer_b200._native import Engine
    from renormalizer_b200.heev import heev_top
    G = _gram(n, np.random.default_rng(n), kind)
    kt = max(1, n // 4)
    _check(G, kt, *heev_top(Engine.get(0), G, kt))


def test_batch_of_all_reductions():
    """one batch whose matrices take the 8-CTA cluster, the 16-CTA cluster and
    the grid; results equal those of single calls"""
    from renormalizer_b200._native import Engine
    from renormalizer_b200.heev import heev_top, heev_top_batched
    rng = np.random.default_rng(5)
    ns, eng = [5, 256, 300, 424, 1, 500, 64], Engine.get(0)
    Gs = [_gram(n, rng, "generic") for n in ns]
    kts = [max(1, n // 5) for n in ns]
    for G, kt, (w, K, chk) in zip(Gs, kts, heev_top_batched(eng, Gs, kts)):
        _check(G, kt, w, K, chk)


def test_many_small_matrices_equal_single_calls():
    """more small matrices than 8-CTA clusters fit: one CTA each, bit for bit the
    results of single calls (a larger one among them stays on its cluster)"""
    from renormalizer_b200._native import Engine
    from renormalizer_b200.heev import heev_top, heev_top_batched
    rng = np.random.default_rng(11)
    ns, eng = [1, 2, 5, 8, 13, 16, 17, 30, 31, 32, 33, 40, 48, 50, 60, 63, 64, 64, 65, 3], Engine.get(0)
    Gs = [_gram(n, rng, "generic") for n in ns]
    kts = [max(1, n // 2) for n in ns]
    for G, kt, (w, K, chk) in zip(Gs, kts, heev_top_batched(eng, Gs, kts)):
        _check(G, kt, w, K, chk)
        w1, _, _ = heev_top(eng, G, kt)
        assert torch.equal(w, w1)
