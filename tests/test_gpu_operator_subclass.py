"""The exponential of an operator class that a program derives from
HeffOperator: its own ``__call__`` or ``apply`` is what is exponentiated,
like any callable's."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["__call__", "apply"])
def test_overridden_operator_is_used(method):
    from renormalizer_b200.hop_expr import HeffOperator
    from renormalizer_b200.krylov import expm_krylov

    def shifted(self, psi, *args, **kw):
        y = getattr(HeffOperator, method)(self, psi, *args, **kw)
        return y + 0.5 * psi.reshape(y.shape)

    Shifted = type("Shifted", (HeffOperator,), {method: shifted})
    g = torch.Generator(device="cuda").manual_seed(7)
    c = lambda *s: torch.complex(*torch.randn((2,) + s, dtype=torch.float64, device="cuda", generator=g))
    L, R = c(6, 2, 6), c(5, 2, 5)
    W = torch.randn(2, 3, 3, 2, dtype=torch.float64, device="cuda", generator=g)
    args = ((L + L.transpose(0, 2).conj()) / 2, (R + R.transpose(0, 2).conj()) / 2, [W + W.transpose(1, 2)], (6, 3, 5))
    op, v = Shifted(*args, prec="fp64"), c(90)
    ref, k = expm_krylov(lambda x: op(x), -0.02j, v)
    got, kn = expm_krylov(op, -0.02j, v)
    assert kn == k and float((got - ref).abs().max()) <= 1e-12 * float(torch.linalg.vector_norm(v))
    plain, _ = expm_krylov(HeffOperator(*args, prec="fp64"), -0.02j, v)
    assert float((got - plain).abs().max()) > 1e-3
