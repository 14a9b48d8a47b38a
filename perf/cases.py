"""Timed workloads of the sweep engine, through its public entry points.

Each case is one call (or one whole step) that a program built on the engine
makes, with the operators, bond dimensions and data types it makes it with:
effective-Hamiltonian matvecs, environment updates, Lanczos exponentials of
one problem and of many in lockstep, gradients of a matvec, truncations and
canonicalising QRs of quantum-number blocked tensors, and a TDVP step.

``listed()`` names the workloads, ``draw()`` samples the same ranges,
``prepare()`` makes a case's inputs from a seed, ``run()`` makes the call,
``work()`` counts what the call cannot do without and ``exact()`` gives the
same result in plain double-precision torch.  Results that are defined only
up to the phase of singular vectors are returned as the products that do not
depend on it.
"""
import math

import numpy as np
import torch

from renormalizer_b200 import (CompressConfig, CompressCriteria, EvolveConfig, EvolveMethod, HolsteinModel, Mol, Mpo,
                               Mps, Phonon, Quantity, SpectralDensityFunction, SpinBosonModel, contract_one_site,
                               expm_krylov, heff_autograd, svd_qn)
from renormalizer_b200.hop_expr import HeffOperator, apply_grouped
from renormalizer_b200.krylov import expm_krylov_batch
from renormalizer_b200.svd_qn import svd_truncate

DEV = "cuda"
EINSUM = {0: "abc,lbk,ck->al", 1: "abc,bdef,lfk,cek->adl"}


def listed():
    return [
        # one-site matvec of a 10-level Holstein mode at M = 32 (the 10-molecule chain run with TDVP-PS): the smallest
        # contraction a sweep makes, thousands of times per trajectory
        {"name": "matvec1_m32", "kind": "matvec", "model": "holstein1", "nlev": 10, "site": 1, "nsite": 1, "ml": 32,
         "mr": 32, "prec": "fp64"},
        # two-site matvec of a phonon-phonon bond at ragged bond dimensions just under the cap, FP64 engine
        {"name": "matvec2_m251_fp64", "kind": "matvec", "model": "holstein2", "nlev": 16, "site": 1, "nsite": 2,
         "ml": 251, "mr": 243, "prec": "fp64"},
        # real two-site matvec of the spin-boson ground-state search (Davidson), M = 256
        {"name": "matvec2_dmrg_m256", "kind": "matvec", "model": "spinboson", "nlev": 8, "site": 7, "nsite": 2,
         "ml": 256, "mr": 256, "prec": "fp64"},
        # the largest contraction of the 96-site two-mode chain, split precision: its default engine
        {"name": "matvec2_m256_bf16x3", "kind": "matvec", "model": "holstein2", "nlev": 16, "site": 1, "nsite": 2,
         "ml": 256, "mr": 256, "prec": "bf16x3"},
        # environment update after a site has moved, M = 256 (every site of every sweep)
        {"name": "env_m256", "kind": "env", "model": "holstein2", "nlev": 16, "site": 1, "domain": "R", "m_in": 256,
         "m_out": 256, "prec": "fp64"},
        # gradients of a one-site matvec with respect to all of its operands (coupling gradients through TDVP, M = 64)
        {"name": "grad1_m64", "kind": "grad", "model": "holstein1", "nlev": 10, "site": 1, "nsite": 1, "ml": 64,
         "mr": 64, "prec": "fp64"},
        # local two-site exponential of a time step in split precision at a bond that has not reached the cap
        {"name": "expm2_m192_bf16x3", "kind": "expm", "model": "holstein2", "nlev": 16, "site": 1, "nsite": 2,
         "ml": 192, "mr": 192, "prec": "bf16x3", "dt": 0.025},
        # the pending two-site exponentials of 64 static-disorder realisations in lockstep, uneven small bonds
        {"name": "expm_batch64", "kind": "batch", "count": 64, "nlev": 10, "m_max": 14, "dt": 0.05},
        # two-site truncation in the middle of a growing trajectory
        {"name": "trunc_m48", "kind": "trunc", "d1": 10, "d2": 10, "ml": 48, "mr": 45, "keep": 48, "digits": 3.0,
         "left": True, "cplx": True},
        # two-site truncation back to M = 256 with 16-level modes: the largest factorisation of a step
        {"name": "trunc_m256", "kind": "trunc", "d1": 16, "d2": 16, "ml": 256, "mr": 256, "keep": 256, "digits": 3.5,
         "left": False, "cplx": True},
        # canonicalising QR of a one-site tensor at M = 256
        {"name": "qr_m256", "kind": "qr", "d": 16, "ml": 256, "mr": 256, "system": "L", "cplx": True},
        # a whole TDVP-PS step and its observables: 10 molecules with one 10-level mode, M = 32
        {"name": "evolve_ps_m32", "kind": "evolve", "nmol": 10, "nlev": 10, "m": 32, "dt": 0.05},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["matvec", "matvec", "matvec", "env", "grad", "expm", "expm", "batch", "trunc", "trunc", "qr",
                       "evolve"])
    if kind == "evolve":
        return {"kind": kind, "nmol": rng.randint(4, 10), "nlev": rng.randint(4, 10), "m": _log(rng, 8, 32),
                "dt": round(rng.uniform(0.02, 0.05), 4)}
    if kind == "batch":
        return {"kind": kind, "count": _log(rng, 6, 64), "nlev": rng.randint(4, 10), "m_max": rng.randint(3, 14),
                "dt": 0.05}
    if kind == "trunc":
        d1, d2, ml, mr = rng.randint(2, 16), rng.randint(2, 16), _log(rng, 24, 256), _log(rng, 24, 256)
        # cut where a user cuts: the discarded weight sits at 1e-5 .. 1e-8 of the norm squared
        return {"kind": kind, "d1": d1, "d2": d2, "ml": ml, "mr": mr,
                "keep": min(max(ml, mr), ml * d1 // 2, mr * d2 // 2), "digits": round(rng.uniform(2.5, 3.75), 2),
                "left": rng.random() < 0.5, "cplx": rng.random() < 0.75}
    if kind == "qr":
        d = rng.randint(2, 16)
        ml = _log(rng, 16, 256)
        return {"kind": kind, "d": d, "ml": ml, "mr": max(4, min(256, int(ml * rng.uniform(0.5, 1.5)))),
                "system": rng.choice("LR"), "cplx": rng.random() < 0.75}
    model = rng.choice(["holstein1", "holstein2", "spinboson"])
    c = {"kind": kind, "model": model, "nlev": rng.randint(4, 16) if model != "spinboson" else rng.randint(4, 8)}
    c["site"] = rng.randint(0, {"holstein1": 1, "holstein2": 2, "spinboson": 0}[model]) if model != "spinboson" \
        else rng.randint(6, 9)
    if kind == "env":
        m = _log(rng, 16, 256)
        c.update(domain=rng.choice("LR"), m_in=m, m_out=max(4, min(256, int(m * rng.uniform(0.5, 1.5)))),
                 prec=rng.choice(["fp64", "fp64", "bf16x3"]))
        return c
    big = {"matvec": 256, "grad": 96, "expm": 160}[kind]
    m = _log(rng, 16, big)
    c.update(nsite=rng.choice([1, 1, 2]) if kind == "grad" else rng.choice([0, 1, 2, 2]), ml=m,
             mr=max(4, min(big, int(m * rng.uniform(0.6, 1.4)))),
             prec="fp64" if kind == "grad" else rng.choice(["fp64", "fp64", "bf16x3", "tf32x3"]))
    if kind == "expm":
        c["dt"] = round(rng.uniform(0.02, 0.05), 4)
    return c


# ---------------------------------------------------------------- operators
def _model(case, disorder=None):
    nlev = case["nlev"]
    if case.get("model") == "spinboson":
        w, c2 = SpectralDensityFunction(0.5, Quantity(10.0)).Wang1(16)
        ph = [Phonon.simple_phonon(Quantity(wi), Quantity(np.sqrt(ci) / wi ** 2), nlev) for wi, ci in zip(w, c2)]
        return SpinBosonModel(Quantity(0.0), Quantity(1.0), ph)
    modes = [(1.0, 1.0), (0.5, 0.7)][: 2 if case.get("model") == "holstein2" else 1]
    ph = [Phonon.simple_phonon(Quantity(w), Quantity(np.sqrt(2.0) * g / np.sqrt(w)), nlev) for w, g in modes]
    nmol = case.get("nmol", 6)
    if disorder is None:
        return HolsteinModel([Mol(Quantity(0), ph)] * nmol, Quantity(1.0), 3)
    eps, hop = disorder.normal(0.0, 0.5, nmol), 1.0 + disorder.normal(0.0, 0.1, nmol - 1)
    J = np.zeros((nmol, nmol))
    for i in range(nmol - 1):
        J[i, i + 1] = J[i + 1, i] = hop[i]
    return HolsteinModel([Mol(Quantity(float(e)), ph) for e in eps], J, 3)


def _first_site(case):
    """chain index of the case's first active site: the middle molecule's
    ``site``-th, or the ``site``-th mode of the spin-boson chain"""
    per = {"holstein1": 2, "holstein2": 3}.get(case.get("model", "holstein1"))
    return case["site"] if case.get("model") == "spinboson" else 3 * per + case["site"]


def _randn(g, shape, cplx):
    r = lambda: torch.randn(shape, dtype=torch.float64, device=DEV, generator=g)
    return torch.complex(r(), r()) if cplx else r()


def _isometry(g, l, d, r, left, cplx):
    """a random canonical site tensor (l, d, r)"""
    a = _randn(g, (l * d, r) if left else (r * d, l), cplx)
    q, _ = torch.linalg.qr(a)
    return q.reshape(l, d, r) if left else q.reshape(r, d, l).permute(2, 1, 0).contiguous()


def _pair(expr, *ts):
    dt = torch.complex128 if any(t.is_complex() for t in ts) else torch.float64
    return torch.einsum(expr, *[t.to(dt) for t in ts])


def _env_step(E, A, W, left):
    """the environment E of one side taken over the site A with MPO tensor W"""
    if left:
        t = _pair("abc,ceh->abeh", E, A)
        t = _pair("abeh,bdeg->adgh", t, W)
        return _pair("adf,adgh->fgh", A.conj(), t)
    t = _pair("abc,hec->abeh", E, A)
    t = _pair("abeh,gdeb->adgh", t, W)
    return _pair("fda,adgh->fgh", A.conj(), t)


def _environment(g, mpo, dims, upto, m, left, cplx):
    """the left (right) environment of the sites before (after) ``upto`` of a
    random canonical state whose bonds grow to ``m``"""
    n = len(dims)
    order = range(upto) if left else range(n - 1, upto, -1)
    bond, E = 1, torch.ones((1, 1, 1), dtype=torch.complex128 if cplx else torch.float64, device=DEV)
    order = list(order)
    # growth from the boundary, at least to m at the last site
    for i in order:
        nxt = min(m, bond * dims[i])
        A = _isometry(g, bond, dims[i], nxt, True, cplx) if left else _isometry(g, nxt, dims[i], bond, False, cplx)
        E = _env_step(E, A, mpo[i], left)
        bond = nxt
    return E.contiguous()


def _local_problem(case, g, model=None):
    """L, W.., R and a normalised random coefficient of the case's sites"""
    model = model or _model(case)
    mpo = Mpo(model)
    cplx = case.get("model") != "spinboson" or case["kind"] == "expm"
    dims = model.pbond_list
    i0, ns = _first_site(case), case["nsite"]
    L = _environment(g, mpo, dims, i0, case["ml"], True, cplx)
    R = _environment(g, mpo, dims, i0 + ns - 1, case["mr"], False, cplx)
    Ws = [mpo[i] for i in range(i0, i0 + ns)]
    shape = (L.shape[0],) + tuple(dims[i0:i0 + ns]) + (R.shape[0],)
    psi = _randn(g, shape, cplx)
    return L, Ws, R, psi / torch.linalg.vector_norm(psi)


# ---------------------------------------------------------------- blocked tensors
def _labels(g, n):
    """quantum numbers 0 / 1 of a bond, about half each, in no order"""
    ones = n // 2
    p = torch.randperm(n, generator=torch.Generator().manual_seed(int(torch.randint(1 << 30, (1,), device=DEV,
                                                                                    generator=g).item())))
    return (p.numpy() < ones).astype(int).reshape(n, 1)


def _blocked(g, ql, qr, decay, cplx):
    """a (rows, cols) coefficient with exciton number 1: each block with
    singular values falling by ``decay`` digits per unit of its index"""
    rows, cols = len(ql), len(qr)
    X = torch.zeros((rows, cols), dtype=torch.complex128 if cplx else torch.float64, device=DEV)
    for q, scale in ((0, 1.0), (1, 0.6)):
        r = torch.from_numpy(np.flatnonzero(ql[:, 0] == q)).to(DEV)
        c = torch.from_numpy(np.flatnonzero(qr[:, 0] == 1 - q)).to(DEV)
        k = min(len(r), len(c))
        s = scale * 10.0 ** (-decay * torch.arange(k, dtype=torch.float64, device=DEV))
        B = (_randn(g, (len(r), k), cplx) * s) @ _randn(g, (k, len(c)), cplx)
        X[r[:, None], c[None, :]] = B / math.sqrt(len(r) * len(c))
    return X / torch.linalg.vector_norm(X)


def _blocks(ql, qr):
    """(rows, columns) of every block in the order the factorisations visit them"""
    for q in set(tuple(int(v) for v in x) for x in ql):
        r, c = np.flatnonzero(ql[:, 0] == q[0]), np.flatnonzero(qr[:, 0] == 1 - q[0])
        if len(r) and len(c):
            yield torch.from_numpy(r).to(DEV), torch.from_numpy(c).to(DEV)


# ---------------------------------------------------------------- cases
def prepare(case, seed):
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    kind = case["kind"]
    s = {"case": case}
    if kind in ("matvec", "expm"):
        L, Ws, R, psi = _local_problem(case, g)
        s.update(L=L, Ws=Ws, R=R, psi=psi, op=HeffOperator(L, R, Ws, psi.shape, prec=case["prec"]))
    elif kind == "grad":
        L, Ws, R, psi = _local_problem(case, g)
        s.update(leaves=[t.clone().requires_grad_(True) for t in [psi, L] + Ws + [R]],
                 gy=_randn(g, psi.shape, psi.is_complex()))
    elif kind == "env":
        model = _model(case)
        mpo = Mpo(model)
        cplx = case["model"] != "spinboson"
        i, left = _first_site(case), case["domain"] == "L"
        E = _environment(g, mpo, model.pbond_list, i, case["m_in"], left, cplx)
        d, m_in = model.pbond_list[i], E.shape[0]
        m_out = min(case["m_out"], m_in * d)
        A = _isometry(g, m_in, d, m_out, True, cplx) if left else _isometry(g, m_out, d, m_in, False, cplx)
        s.update(E=E, A=A, W=mpo[i])
    elif kind == "batch":
        rng = np.random.default_rng(int(seed))
        sizes = np.random.default_rng(case["count"])
        probs = []
        models = [_model(case, rng) for _ in range(4)]
        for b in range(case["count"]):
            # bonds as a 1e-8 threshold leaves them over the first steps: a few states, now and then many
            bond = lambda: 1 + int((case["m_max"] - 1) * sizes.random() ** 3)
            c = dict(case, model="holstein1", site=int(sizes.integers(0, 2)), nsite=2, ml=bond(), mr=bond())
            probs.append(_local_problem(c, g, models[b % 4]))
        s.update(probs=probs, ops=[HeffOperator(L, R, Ws, psi.shape, prec="fp64") for L, Ws, R, psi in probs])
    elif kind == "trunc":
        ml, mr, d1, d2 = case["ml"], case["mr"], case["d1"], case["d2"]
        ql = np.repeat(_labels(g, ml)[:, None, :], d1, axis=1)
        qr = np.repeat(_labels(g, mr)[None, :, :], d2, axis=0)
        # the kept half of each block spans ``digits`` decades
        X = _blocked(g, ql.reshape(-1, 1), qr.reshape(-1, 1), 2.0 * case["digits"] / case["keep"], case["cplx"])
        s.update(coef=X.reshape(ml, d1, d2, mr), ql=ql, qr=qr)
    elif kind == "qr":
        ml, mr, d = case["ml"], case["mr"], case["d"]
        lab_l, lab_r = _labels(g, ml), _labels(g, mr)
        if case["system"] == "L":
            ql, qr = np.repeat(lab_l[:, None, :], d, axis=1), lab_r
        else:
            ql, qr = lab_l, np.repeat(lab_r[None, :, :], d, axis=0)
        k = min(ml, mr)
        X = _blocked(g, ql.reshape(-1, 1), qr.reshape(-1, 1), 2.0 / k, case["cplx"])
        s.update(coef=X.reshape(ml, d, mr), ql=ql, qr=qr)
    else:
        model = _model(case)
        np.random.seed(int(seed) % (1 << 31))
        rng = np.random.default_rng(int(seed))
        cond = {model.e_dofs[0]: 1}
        for v in model.v_dofs:  # coherent phonon states
            a = rng.uniform(0.1, 0.6)
            amp = np.array([a ** k / math.sqrt(math.factorial(k)) for k in range(case["nlev"])])
            cond[v] = amp / np.linalg.norm(amp)
        mps = Mps.hartree_product_state(model, cond)
        mps.compress_config = CompressConfig(CompressCriteria.fixed, max_bonddim=case["m"])
        mps = mps.expand_bond_dimension(coef=0.05)
        mps.evolve_config = EvolveConfig(EvolveMethod.tdvp_ps)
        s.update(mps=mps, mpo=Mpo(model))
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "matvec":
        return s["op"](s["psi"])
    if kind == "expm":
        y, n = expm_krylov(s["op"], -0.5j * case["dt"], s["psi"].reshape(-1))
        return {"psi": y, "vectors": n}
    if kind == "env":
        return contract_one_site(s["E"], s["A"], s["W"], case["domain"], prec=case["prec"])
    if kind == "grad":
        psi, L, *Ws, R = s["leaves"]
        y = heff_autograd(psi, L, Ws, R, prec=case["prec"])
        return [y.detach()] + list(torch.autograd.grad(y, s["leaves"], s["gy"]))
    if kind == "batch":
        ops = s["ops"]
        res = expm_krylov_batch(lambda idx, xs: apply_grouped([ops[i] for i in idx], xs), -0.5j * case["dt"],
                                [p[3].reshape(-1) for p in s["probs"]])
        return {"psi": torch.cat([y for y, _ in res]), "vectors": np.array([n for _, n in res])}
    if kind == "trunc":
        res = svd_truncate(s["coef"], s["ql"], s["qr"], np.array([1]), case["left"],
                           lambda sig: min(case["keep"], len(sig)), kcap=case["keep"])
        return {"coef": res.left @ res.right, "sigma": res.sigma, "qn": res.qn}
    if kind == "qr":
        u, qnl, v, qnr = svd_qn(s["coef"], s["ql"], s["qr"], np.array([1]), QR=True, system=case["system"],
                                full_matrices=False)
        return {"u": u, "qnl": np.array(qnl), "v": v, "qnr": np.array(qnr)}
    new = s["mps"].evolve(s["mpo"], case["dt"])
    rdm = new.calc_1site_rdm()
    return {"e": new.e_occupations, "ph": new.ph_occupations, "energy": new.expectation(s["mpo"]),
            "rdm": [rdm[i] for i in sorted(rdm)]}


# ---------------------------------------------------------------- what a call cannot do without
def _shape(case):
    """(ml, mr, wl, wm, wr, d1, d2) of a local problem"""
    if case.get("model") == "spinboson":
        return case["ml"], case["mr"], 3, 3, 3, case["nlev"], case["nlev"]
    per = 3 if case["model"] == "holstein2" else 2
    d = lambda i: 2 if i % per == 0 else case["nlev"]
    w = lambda i: 4 if i % per == 0 else 5
    i, ns = case["site"], case["nsite"]
    return case["ml"], case["mr"], w(i), w(i + 1), w(i + ns), d(i), d(i + 1)


def _matvec_work(case):
    ml, mr, wl, wm, wr, d1, d2 = _shape(case)
    cplx = case["model"] != "spinboson" or case["kind"] == "expm"
    c1, c2, b = (8, 4, 16) if cplx else (2, 2, 8)
    if case["nsite"] == 2:
        f = c1 * (ml * wl * ml * d1 * d2 * mr + ml * d1 * d2 * wr * mr * mr) + \
            c2 * (ml * d1 * wm * wl * d1 * d2 * mr + ml * d1 * d2 * wr * wm * d2 * mr)
        n = ml * d1 * d2 * mr
    elif case["nsite"] == 1:
        f = c1 * (ml * wl * ml * d1 * mr + ml * d1 * wr * mr * mr) + c2 * ml * d1 * wr * wl * d1 * mr
        n = ml * d1 * mr
    else:
        f = c1 * (ml * wl * ml * mr + ml * wl * mr * mr)
        n = ml * mr
    return f, b * (ml * wl * ml + mr * wr * mr + 2 * n), b * n


def work(case):
    kind = case["kind"]
    if kind == "matvec":
        f, b, _ = _matvec_work(case)
    elif kind == "expm":
        f, b, _ = _matvec_work(case)
        f *= 7  # Krylov vectors of a usual step
    elif kind == "grad":
        f, b, n = _matvec_work(case)
        f, b = 4 * f, 2 * b + n
    elif kind == "env":
        c = dict(case, kind="matvec", nsite=1, ml=case["m_in"], mr=case["m_out"])
        mi, mo, wl, _, wr, d, _ = _shape(c)
        c1, c2, e = (8, 4, 16) if case["model"] != "spinboson" else (2, 2, 8)
        f = c1 * (mi * wl * mi * d * mo + mi * d * wr * mo * mo) + c2 * mi * d * wr * wl * d * mo
        b = e * (mi * wl * mi + mo * wr * mo + mi * d * mo)
    elif kind == "batch":
        m = 1 + (case["m_max"] - 1) / 4.0
        c = dict(case, kind="matvec", model="holstein1", site=0, nsite=2, ml=m, mr=m)
        f, b, _ = _matvec_work(c)
        f, b = 7 * case["count"] * f, case["count"] * b
    elif kind == "trunc":
        m, n, k = case["ml"] * case["d1"], case["mr"] * case["d2"], case["keep"]
        c = 8 if case["cplx"] else 2
        f = c * m * n * k + c * m * n * k / 2  # two halves of the rows and columns, both factors of the kept k
        b = (16 if case["cplx"] else 8) * (m * n + (m + n) * k)
    elif kind == "qr":
        rows, k = max(case["ml"], case["mr"]) * case["d"], min(case["ml"], case["mr"])
        f = (8 if case["cplx"] else 2) * rows * k * k / 2  # two blocks of half the rows and columns, Q formed
        b = (16 if case["cplx"] else 8) * (2 * rows * k + k * k)
    else:
        c = {"kind": "matvec", "model": "holstein1", "nlev": case["nlev"], "site": 1, "nsite": 1, "ml": case["m"],
             "mr": case["m"]}
        f1, _, n = _matvec_work(c)
        f = 2 * 2 * case["nmol"] * 8 * f1
        b = 2 * 2 * case["nmol"] * 4 * n
    return {"bytes": float(b), "flops": float(f)}


# ---------------------------------------------------------------- the same in plain double precision
def _hop(L, Ws, R, psi):
    t = _pair("abc,c...->ab...", L, psi)
    if len(Ws) == 0:
        return _pair("abk,lbk->al", t, R)
    t = _pair("abe...,bdef->adf...", t, Ws[0])
    if len(Ws) == 1:
        return _pair("adfk,lfk->adl", t, R)
    t = _pair("adfhk,fghj->adgjk", t, Ws[1])
    return _pair("adgjk,ljk->adgl", t, R)


def _lanczos(hop, dt, v):
    """exp(dt H) v with the documented stopping rule: successive results at
    even steps past the third agree within rtol 1e-5 / atol 1e-8"""
    nrm = torch.linalg.vector_norm(v)
    V, al, be, prev = [v / nrm], [], [], None
    for j in range(v.numel()):
        w = hop(V[j])
        a = torch.vdot(V[j], w).real
        al.append(float(a))
        w = w - a * V[j] - (be[-1] * V[j - 1] if j else 0.0)
        b = float(torch.linalg.vector_norm(w))
        last = j == v.numel() - 1 or b < 100 * v.numel() * np.finfo(float).eps
        if last or (j > 3 and j % 2 == 0):
            T = np.diag(al) + np.diag(be, 1) + np.diag(be, -1)
            ev, U = np.linalg.eigh(T)
            c = U @ (float(nrm) * np.exp(dt * ev) * U[0])
            new = sum(complex(x) * y for x, y in zip(c, V))
            if last or (prev is not None and torch.allclose(prev, new, rtol=1e-5, atol=1e-8)):
                return new
            prev = new
        be.append(b)
        V.append(w / b)


def exact(case, seed):
    kind = case["kind"]
    if kind == "evolve":
        return None
    s = prepare(case, seed)
    if kind == "matvec":
        return _hop(s["L"], s["Ws"], s["R"], s["psi"])
    if kind == "expm":
        f = lambda x: _hop(s["L"], s["Ws"], s["R"], x.reshape(s["psi"].shape)).reshape(-1)
        return {"psi": _lanczos(f, -0.5j * case["dt"], s["psi"].reshape(-1).to(torch.complex128)), "vectors": None}
    if kind == "env":
        return _env_step(s["E"], s["A"], s["W"], case["domain"] == "L")
    if kind == "grad":
        psi, L, *Ws, R = s["leaves"]
        y = _hop(L, Ws, R, psi)
        return [y.detach()] + list(torch.autograd.grad(y, s["leaves"], s["gy"]))
    if kind == "batch":
        out = [_lanczos(lambda x, p=p: _hop(p[0], p[1], p[2], x.reshape(p[3].shape)).reshape(-1), -0.5j * case["dt"],
                        p[3].reshape(-1)) for p in s["probs"]]
        return {"psi": torch.cat(out), "vectors": None}
    ql, qr = s["ql"].reshape(-1, 1), s["qr"].reshape(-1, 1)
    X = s["coef"].reshape(len(ql), len(qr))
    if kind == "trunc":
        parts, sig, own = [], [], []
        for b, (r, c) in enumerate(_blocks(ql, qr)):
            U, S, Vh = torch.linalg.svd(X[r[:, None], c[None, :]], full_matrices=False)
            parts.append((r, c, U, S, Vh))
            sig.append(S)
            own += [b] * len(S)
        sig = torch.cat(sig).cpu().numpy()
        order = np.argsort(-sig, kind="stable")[: case["keep"]]
        out = torch.zeros_like(X)
        for b, (r, c, U, S, Vh) in enumerate(parts):
            k = int(np.sum(np.array(own)[order] == b))
            out[r[:, None], c[None, :]] = (U[:, :k] * S[:k]) @ Vh[:k]
        return {"coef": out, "sigma": sig[order], "qn": None}
    us, vs = [], []
    for r, c in _blocks(ql, qr):
        B = X[r[:, None], c[None, :]]
        if case["system"] == "L":
            Q, T = torch.linalg.qr(B)
        else:
            # RQ from the QR of the reversed conjugate transpose
            q, t = torch.linalg.qr(B.flip([0, 1]).mH.resolve_conj().contiguous())
            Q, T = t.mH.flip([0, 1]), q.mH.flip([0, 1])
        u = torch.zeros((X.shape[0], Q.shape[1]), dtype=X.dtype, device=X.device)
        v = torch.zeros((X.shape[1], Q.shape[1]), dtype=X.dtype, device=X.device)
        u[r], v[c] = Q, T.transpose(0, 1)
        us.append(u)
        vs.append(v)
    return {"u": torch.cat(us, 1), "qnl": None, "v": torch.cat(vs, 1), "qnr": None}
