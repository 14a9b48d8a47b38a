"""The one-call exponential of a HeffOperator and the lockstep exponentials'
address tables against the generic driver (which serves any callable).

Both run the same kernels on the same vectors and differ only in where the
small coefficients are formed, so results agree to rounding (1e-12 of a unit
vector) and counts exactly: 0 / 1 / 2 sites, FP64 and split chains (whose
constant operands stay packed between the matvecs), fewer dimensions than
Krylov vectors, a start vector in an invariant subspace, and a vector budget
that is too small, where the generic driver takes over."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _problem(nsite, ml, mr, d, seed, prec="fp64", scale=1.0):
    from renormalizer_b200.hop_expr import HeffOperator
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(s, dtype=torch.float64, device="cuda", generator=g)
    c = lambda *s: torch.complex(r(*s), r(*s))
    herm = lambda t: ((t + t.transpose(0, 2).conj()) * 0.5).contiguous()
    sym = lambda t: ((t + t.transpose(1, 2)) * 0.5).contiguous()
    L, R = herm(c(ml, 3, ml)), herm(c(mr, 3, mr)) * scale
    Ws = [sym(r(3, d, d, 3)) for _ in range(nsite)]
    shape = (ml,) + (d,) * nsite + (mr,)
    psi = c(*shape)
    return HeffOperator(L, R, Ws, shape, prec=prec), psi / torch.linalg.vector_norm(psi)


@pytest.mark.parametrize("nsite,ml,mr,d,prec", [(0, 1, 2, 1, "fp64"), (0, 9, 14, 1, "fp64"), (1, 1, 1, 2, "fp64"),
                                                (1, 31, 17, 5, "fp64"), (2, 20, 33, 4, "fp64"),
                                                (1, 40, 24, 6, "bf16x3"), (2, 24, 20, 3, "tf32x3"),
                                                (2, 70, 66, 16, "bf16x3")])
@pytest.mark.parametrize("block", [50, 7, 3])
def test_native_matches_generic(nsite, ml, mr, d, prec, block):
    from renormalizer_b200.krylov import expm_krylov
    op, psi = _problem(nsite, ml, mr, d, 5, prec)
    dt = -0.3j / (ml + mr)
    x0 = psi.reshape(-1).clone()
    ref, k = expm_krylov(lambda x: op.apply(x), dt, x0, block)
    got, kn = expm_krylov(op, dt, x0, block)
    assert kn == k and torch.equal(x0, psi.reshape(-1))
    assert float((got - ref).abs().max()) <= 1e-12


def test_native_breakdown_and_bad_start():
    from renormalizer_b200.hop_expr import HeffOperator
    from renormalizer_b200.krylov import expm_krylov
    m = 30
    L = torch.diag(torch.arange(1.0, m + 1, dtype=torch.float64)).to(torch.complex128).reshape(m, 1, m).cuda()
    op = HeffOperator(L.contiguous(), torch.ones((1, 1, 1), dtype=torch.complex128, device="cuda"), [], (m, 1))
    v = torch.zeros(m, dtype=torch.complex128, device="cuda")
    v[[3, 11, 20]] = torch.tensor([1.0, 0.5j, -0.25], dtype=torch.complex128, device="cuda")
    ref, k = expm_krylov(lambda x: op.apply(x), -0.1j, v)
    got, kn = expm_krylov(op, -0.1j, v)
    assert kn == k == 3 and float((got - ref).abs().max()) <= 1e-12
    for bad, exc in ((0.0, AssertionError), (float("nan"), AssertionError), (float("inf"), FloatingPointError)):
        w = torch.full_like(v, 0.0)
        w[4] = bad
        for f in (op, lambda x: op.apply(x)):
            with pytest.raises(exc):
                expm_krylov(f, -0.1j, w)


def test_lockstep_tables_match_each_ones_own():
    from renormalizer_b200.hop_expr import apply_grouped
    from renormalizer_b200.krylov import expm_krylov, expm_krylov_batch
    probs = [_problem(2, ml, mr, 3, 7 + ml, scale=s) for ml, mr, s in ((1, 1, 1), (4, 3, 1), (13, 6, 3), (1, 2, 0.01),
                                                                     (30, 21, 1))]
    ops, dt = [p[0] for p in probs], -0.02j
    own = [expm_krylov(lambda x, op=op: op.apply(x), dt, p.reshape(-1)) for op, p in probs]
    cut = expm_krylov_batch(lambda i, xs: apply_grouped([ops[k] for k in i], xs), dt, [p.reshape(-1) for _, p in probs], 4)

    def swapped(i, xs):  # a caller that replaces an entry of the list it was given
        xs[0] = xs[0].clone()
        return list(apply_grouped([ops[k] for k in i], xs))

    lists = expm_krylov_batch(swapped, dt, [p.reshape(-1) for _, p in probs])
    for (a, k), (b, kb), (c, kc) in zip(own, cut, lists):
        assert k == kb == kc and torch.equal(a, b) and torch.equal(a, c)
