"""The panel kernels of the batched QR at the edges of their ranges, against
LAPACK (SciPy) entry by entry: rows per lane 2 / 4 / 8 / 16 / 32 full and one
row over, panels of 32 and of 16 columns, a last panel of one column, the
shared-memory kernel past the register panels, and a batch whose matrices
fill very different shares of the panel.  Gaussian matrices have condition
numbers far below 1 / (eps m), so Householder QR reproduces Q and R to a small
multiple of m eps: 1e-12 m as in the general QR test."""
import numpy as np
import pytest
import scipy.linalg as sla
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cplx", [True, False])
@pytest.mark.parametrize("shapes", [
    [(33, 33)], [(512, 65)], [(513, 31)], [(1024, 33)], [(1025, 64)], [(2048, 33)], [(2049, 17)], [(4096, 33)],
    [(4097, 20)], [(8193, 9)], [(2050, 40), (3, 40), (31, 31), (700, 1)],
])
def test_qr_panels(shapes, cplx):
    from renormalizer_b200._native import Engine
    rng = np.random.default_rng(sum(m + 3 * k for m, k in shapes) + cplx)
    hs = [rng.standard_normal(s) + (1j * rng.standard_normal(s) if cplx else 0) for s in shapes]
    Qs, Rs = Engine.get(0).qr_blocks([torch.from_numpy(h).cuda() for h in hs])
    for h, Q, R in zip(hs, Qs, Rs):
        q, r = sla.qr(h, mode="economic")
        tol = 1e-12 * max(h.shape)
        assert np.abs(Q.cpu().numpy() - q).max() < tol
        assert np.abs(R.cpu().numpy() - r).max() < tol * np.abs(h).max()
