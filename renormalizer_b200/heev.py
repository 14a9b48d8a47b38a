"""Leading eigenpairs of the truncation's Hermitian Gram blocks on the device.

The QN-blocked truncation (svd_qn.py:12-49 with mp.py:693-778 in the
reference, which takes LAPACK gesdd of every block) diagonalises each block's
Gram matrix.  Under a fixed cap k only the leading k + 64 eigenvectors of a
block are used, and cuSOLVER's dense eigensolver spends most of its time in a
tridiagonal reduction kernel (about 25 ms of a 37 ms call on a 2048^2 complex
block).  ``heev_top_batched`` runs the whole eigensolver in libreno_b200
instead, for all QN blocks of a bond at once:

* reno_heev_top_batched: Householder reduction to a real tridiagonal T in one
  cooperative launch shared by the blocks (one grid barrier per column), the kt largest
  eigenvalues of T by Sturm-count multisection and their eigenvectors by
  inverse iteration;
* Householder QR of the kt tridiagonal eigenvectors, largest eigenvalue
  first (inverse iteration leaves vectors of eigenvalues closer than the
  rounding level non-orthogonal, or nearly parallel);
* the residual max ||T z - rho z|| / max |lambda| and the reduction's
  status word, returned as a device tensor so that the caller reads them with
  the singular values it already brings to the host;
* reno_heev_backtransform_batched: K = Q Z in blocks of 64 reflectors (compact WY
  form, three FP64 GEMMs per block).

The caller falls back to cuSOLVER for a block whose check fails.
"""
from __future__ import annotations

import math
import os

import numpy as np
import torch

from ._native import HEEV_MAX_BATCH, Engine, HeevProblem


class HeevOptions:
    """``enabled``: use the device eigensolver for Gram blocks of order at
    least ``min_n`` (default: every block; cuSOLVER only redoes a block whose
    checks fail); ``tol``: the largest accepted residual relative to
    max |lambda|.  RENO_HEEV="0" / "1" overrides ``enabled``."""

    def __init__(self, enabled=True, min_n=1, tol=1e-12):
        env = os.environ.get("RENO_HEEV")
        self.enabled = enabled if env is None else env not in ("0", "")
        self.min_n = min_n
        self.tol = tol
        self.calls = 0
        self.fallbacks = 0


heev_opts = HeevOptions()
def heev_top(eng: Engine, G: torch.Tensor, kt: int):
    """The kt largest eigenpairs of the Hermitian matrix G (n x n, float64 or
    complex128, on the device), descending: (w (kt,), K (n, kt) complex128,
    check) with check = [status, 0, relative residual] on the device (accept
    when status == 0 and residual <= tol).  One matrix of heev_top_batched."""
    return heev_top_batched(eng, [G], [kt])[0]


def accepted(check_host) -> bool:
    status, fails, res = check_host
    return status == 0 and fails == 0 and res <= heev_opts.tol


_WSB = {}


def _batched_ws(eng: Engine, nbytes: int) -> torch.Tensor:
    ws = _WSB.get(eng.device)
    if ws is None or ws.numel() < nbytes:
        ws = torch.empty(max(nbytes, 1 << 20), dtype=torch.uint8, device=f"cuda:{eng.device}")
        _WSB[eng.device] = ws
    return ws


def _vp(t):
    import ctypes
    return ctypes.c_void_p(t.data_ptr())


def heev_top_batched(eng: Engine, Gs, kts):
    """heev_top for several Hermitian matrices at once (the QN blocks of one
    bond): one batched reduction launch, then per matrix the kt largest
    eigenvalues (Sturm bisection) and inverse-iteration vectors, ordered
    descending and orthonormalised together by Householder QR
    (reno_qr_blocks) -- which, unlike a Cholesky-based orthonormalisation,
    cannot fail when vectors of a tight cluster come out nearly parallel --
    then the back-transformation.  Returns per matrix (w (kt,) descending,
    K (n, kt) complex128, check) with check = [status, 0, residual] on the
    device; the residual is max_j ||T z_j - rho_j z_j|| / max |w| with rho_j
    the Rayleigh quotient of the orthonormalised z_j."""
    out = []
    for i0 in range(0, len(Gs), HEEV_MAX_BATCH):
        out += _heev_chunk(eng, Gs[i0:i0 + HEEV_MAX_BATCH], kts[i0:i0 + HEEV_MAX_BATCH])
    return out


def _heev_chunk(eng, Gs, kts):
    dev = Gs[0].device
    heev_opts.calls += len(Gs)
    mats, probs = [], []
    for G, kt in zip(Gs, kts):
        n = G.shape[0]
        A = G.to(torch.complex128).contiguous().clone()
        d = torch.empty(n, dtype=torch.float64, device=dev)
        e = torch.empty(max(n - 1, 1), dtype=torch.float64, device=dev)
        tau = torch.empty(max(n - 1, 1), dtype=torch.complex128, device=dev)
        w = torch.empty(kt, dtype=torch.float64, device=dev)
        Z = torch.empty((n, kt), dtype=torch.float64, device=dev)
        mats.append((n, kt, A, d, e, tau, w, Z))
        probs.append(HeevProblem(n, kt, _vp(A), _vp(d), _vp(e), _vp(tau), _vp(w), _vp(Z), None))
    ws = _batched_ws(eng, eng.heev_batched_bytes(probs))
    status = torch.zeros(len(Gs), dtype=torch.int32, device=dev)
    eng.heev_batched(probs, status, ws, "top")
    Qs, _ = eng.qr_blocks([Z.flip(1).contiguous() for (_, _, _, _, _, _, _, Z) in mats])
    Ks, checks = [], []
    for i, ((n, kt, A, d, e, tau, w, Z), Q) in enumerate(zip(mats, Qs)):
        TQ = d[:, None] * Q
        if n > 1:
            TQ[:-1] += e[:n - 1, None] * Q[1:]
            TQ[1:] += e[:n - 1, None] * Q[:-1]
        rho = (Q * TQ).sum(dim=0)
        scale = torch.clamp(w.abs().max(), min=torch.finfo(torch.float64).tiny)
        res = torch.nan_to_num((TQ - Q * rho).abs().max() / scale, nan=float("inf"))
        K = Q.to(torch.complex128).contiguous()
        probs[i].k = _vp(K)
        Ks.append(K)
        checks.append(torch.stack([status[i].to(torch.float64), torch.zeros((), dtype=torch.float64, device=dev),
                                   res]))
    eng.heev_batched(probs, status, ws, "back")
    return [(torch.flip(m[6], dims=[0]), K, chk) for m, K, chk in zip(mats, Ks, checks)]


class LowRankOptions:
    """Leading eigenpairs of a Gram matrix G = M^H M from its numerical range.

    The Gram matrix of a coefficient whose singular values decay over the
    kept ones has few eigenvalues above its own rounding errors (8 decades of
    sigma are 16 of lambda), while forming it and reducing all of its n
    columns to a tridiagonal matrix costs the same however few they are.  For
    orders n >= ``min_n`` and n >= ``min_ratio`` r the range is found first
    (Halko, Martinsson, Tropp, SIAM Rev. 53, 2011): Q1 = orth(M^H Omega) with
    r >= kt + ``oversample`` seeded Gaussian columns Omega, Q = orth(M^H (M Q1)),
    B = M Q, T = B^H B.  T goes through the device eigensolver, and with its
    eigenvectors S the wanted ones are K = Q S and the projected block M K = B S,
    so G itself is never formed.

    The order of the passes is for precision.  From orth(M^H (M Omega)), what
    rounding adds to the small columns of the second product leaves some 2e-15
    of G outside Q, and truncated coefficients came out up to 1.24 times further from
    64 bits than the dense route's (30 blocks of 480 to 2048 rows, mean
    1.05).  Rounding of M^H Omega hides singular values below eps sigma_1 instead of
    eigenvalues below eps lambda_1, M^H M maps each column of Q1 to its
    own size, and the ratio is 1.000 or less on all of those blocks.

    The range is kept only where it carries all of G to G's own rounding
    level: the trace that is missing, ||M - B Q^H||_F^2 <= ``tol`` sqrt(n)
    ||M||_F^2, bounds every eigenvalue left out because G is positive semidefinite.
    It is estimated without cancellation from ``check`` Gaussian vectors w, for
    which ||M w - B (Q^H w)||^2 has that mean and falls to a tenth of it once in 1e12
    times.  The host reads it twice, for Q1 (which leaves up to ten times
    more, hence 64 limits) and for Q, both before the eigenproblem, and a block that
    misses goes to the dense path with the others of its call.

    r comes from a sketch of ``probe`` columns, whose R factor's diagonal
    falls like the eigenvalues: the slope of its logarithm extrapolated to
    rounding level, at least kt + oversample and at most n / min_ratio.  Where
    that upper limit is below 0.7 of the extrapolation the block is not tried.
    Nor is it where a dense block of 0.8 its order or more belongs to the same
    truncation and r > n^2 / 10240: the dense reduction, a chain of columns, takes
    little longer for two blocks than for one (1.2 / 3.7 / 16 / 82 ms at n = 1024 /
    1440 / 2048 / 3584, which grows like n^3), while the range alone costs 5.3
    / 6.2 / 10.4 / 30.7 ms at r = n / 5 and grows like n r.

    Kept sides of two complex 2048^2 blocks, 320 vectors each: 48.7 ms by the
    dense path, 13.4 / 21.3 / 28.3 through 416 / 608 / 800 columns; two of 600
    rows, 128 vectors: 5.7 ms, 4.6 through 224 columns.  A probe that says no costs 0.2
    to 0.5 ms, 4 % of a block of 480 rows and 1 % of one of 2048."""

    def __init__(self, min_n=480, min_ratio=2.5, oversample=32, probe=32, tol=1e-16, check=32):
        self.min_n, self.min_ratio, self.oversample = min_n, min_ratio, oversample
        self.probe, self.tol, self.check = probe, tol, check
        self.calls = 0
        self.missed = 0


lowrank_opts = LowRankOptions()


def _range_columns(n: int, kt: int, diag=None) -> int:
    """Columns of the range sketch for kt eigenpairs of order n, given the
    diagonal of its probe's R factor; 0 = dense path."""
    least = (kt + lowrank_opts.oversample + 31) // 32 * 32
    most = int(n / lowrank_opts.min_ratio) // 32 * 32
    if n < lowrank_opts.min_n:
        return 0
    if least > most or diag is None:
        return least if least <= most else 0
    eps = np.finfo(np.float64).eps
    if not (diag[0] > 0 and np.all(np.isfinite(diag))):
        return 0
    j = np.arange(4, len(diag))
    slope = -np.polyfit(j, np.log(np.maximum(diag[4:] / diag[0], eps * eps)), 1)[0]
    need = -math.log(eps) / slope if slope > 0 else math.inf
    if most < 0.7 * need:
        return 0
    return min(most, max(least, (int(need) + 31) // 32 * 32))


def lowrank_top_batched(eng: Engine, Ms, kts, calls):
    """The kts[i] largest eigenpairs of each Gram matrix G = M^H M through its
    numerical range (LowRankOptions).  Ms: (matrix, adjoint) pairs, M the
    matrix or, with adjoint, its conjugate transpose; calls: which truncation
    each entry belongs to.  Returns per entry
    (w, K, check, M K) -- w, K and check like heev_top_batched -- or None where
    the dense path is to be taken."""
    out = [None] * len(Ms)
    size = lambda i: Ms[i][0].shape[0 if Ms[i][1] else 1]
    long = lambda i: Ms[i][0].shape[1 if Ms[i][1] else 0]
    idx = [i for i, kt in enumerate(kts) if _range_columns(size(i), kt)]
    if not idx:
        return out

    def fwd(i, v):  # M v
        X, adj = Ms[i]
        return eng.matmul(X.transpose(0, 1), v, conj_a=True) if adj else eng.matmul(X, v)

    def back(i, v):  # M^H v
        X, adj = Ms[i]
        return eng.matmul(X, v) if adj else eng.matmul(X.transpose(0, 1), v, conj_a=True)

    dev, norm = Ms[0][0].device, torch.linalg.vector_norm

    def gaussian(rows, cols, seed):  # seeded by its shape alone: a block's result does not depend on the batch it is in
        gen = torch.Generator(device=dev).manual_seed(seed)
        return torch.randn((rows, cols), dtype=torch.float64, device=dev, generator=gen)

    def orth(mats):
        return dict(zip(idx, _qr_by_type(eng, [mats[i] for i in idx])[0]))

    def keep(bad):  # drops the blocks whose (device) flag is set
        for i, b in zip(list(idx), torch.stack([bad[i] for i in idx]).cpu().tolist()):
            if b:
                idx.remove(i)
                lowrank_opts.missed += 1

    Y = [back(i, fwd(i, gaussian(size(i), lowrank_opts.probe, 0x5EED))) for i in idx]
    diag = torch.stack([torch.diagonal(R).abs() for R in _qr_by_type(eng, Y)[1]]).cpu().numpy()
    rs = {i: _range_columns(size(i), kts[i], d) for i, d in zip(idx, diag)}
    beside = {}  # the largest block of each truncation that the probe sends to the dense path
    for i, c in enumerate(calls):
        if not rs.get(i):
            beside[c] = max(beside.get(c, 0), size(i))
    idx = [i for i in idx if rs[i] and (size(i) > 1.25 * beside.get(calls[i], 0) or 10240 * rs[i] <= size(i) ** 2)]
    lowrank_opts.calls += len(idx)
    if not idx:
        return out
    W = {i: gaussian(size(i), lowrank_opts.check, 0x5EED + 2) for i in idx}
    MW = {i: fwd(i, W[i]) for i in idx}
    limit = {i: lowrank_opts.tol * math.sqrt(size(i)) for i in idx}
    full = {i: norm(Ms[i][0]) ** 2 for i in idx}

    def missing(i):  # of the trace, relative
        x = MW[i] - eng.matmul(B[i], eng.matmul(Q[i].transpose(0, 1), W[i], conj_a=True))
        return norm(x) ** 2 / (lowrank_opts.check * full[i])

    Q = orth({i: back(i, gaussian(long(i), rs[i], 0x5EED + 1)) for i in idx})
    B = {i: fwd(i, Q[i]) for i in idx}
    keep({i: ~(missing(i) <= 64 * limit[i]) for i in idx})
    if not idx:
        return out
    Q = orth({i: back(i, B[i]) for i in idx})
    B = {i: fwd(i, Q[i]) for i in idx}
    T = {i: eng.matmul(B[i].transpose(0, 1), B[i], conj_a=True) for i in idx}
    keep({i: ~(missing(i) <= limit[i]) for i in idx})
    for i, (w, S, chk) in zip(idx, heev_top_batched(eng, [T[i] for i in idx], [kts[i] for i in idx])):
        S = S if Q[i].is_complex() else S.real.contiguous()
        out[i] = (w, eng.matmul(Q[i], S), chk, eng.matmul(B[i], S))
    return out


def _qr_by_type(eng: Engine, mats):
    """Engine.qr_blocks for matrices of both types"""
    Qs, Rs = [None] * len(mats), [None] * len(mats)
    for cplx in (False, True):
        idx = [i for i, m in enumerate(mats) if m.is_complex() == cplx]
        if idx:
            q, r = eng.qr_blocks([mats[i] for i in idx])
            for i, a, b in zip(idx, q, r):
                Qs[i], Rs[i] = a, b
    return Qs, Rs
