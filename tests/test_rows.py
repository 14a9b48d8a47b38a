"""The vector lists of lockstep exponentials when a caller replaces entries by
views of the same memory: a lazy conjugate, a negation, a transpose or a part
has the address of the vector it stands for and another meaning."""
import numpy as np
import pytest
import torch


def _rows(shapes, device="cpu"):
    from renormalizer_b200.hop_expr import Rows
    sizes = [int(np.prod(s)) for s in shapes]
    g = torch.Generator().manual_seed(1)
    flat = torch.complex(*torch.randn((2, sum(sizes)), dtype=torch.float64, generator=g)).to(device)
    ptrs = np.uint64(flat.data_ptr()) + (16 * (np.cumsum(sizes) - sizes)).astype(np.uint64)
    return Rows([t.view(s) for t, s in zip(flat.split(sizes), shapes)], ptrs, sizes)


VIEWS = {
    "conj": lambda t: t.conj(),
    "neg": lambda t: torch._neg_view(t),
    "transpose": lambda t: t.transpose(0, 1),
    "part": lambda t: t[:2],
    "real": lambda t: torch.view_as_real(t),
    "copy": lambda t: t.clone(),
}


@pytest.mark.parametrize("view", sorted(VIEWS))
def test_views_of_the_same_memory_are_noticed(view):
    rows = _rows([(4, 3), (5, 2)])
    assert rows.intact()
    rows[0] = rows[0].reshape(-1).view(4, 3)  # the same vector
    assert rows.intact()
    rows[1] = VIEWS[view](rows[1])
    assert not rows.intact()
    rows = _rows([(4, 3), (5, 2)])
    del rows[1]
    assert not rows.intact()


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["arguments", "results"])
@pytest.mark.parametrize("view", ["conj", "neg", "transpose"])
def test_lockstep_reads_replaced_entries(view, where):
    """replaced entries give what the same entries in a plain list (which is
    looked at tensor by tensor) give: the same result, or the refusal of a lazy
    conjugate as an operator's argument"""
    from renormalizer_b200.hop_expr import HeffOperator, apply_grouped
    from renormalizer_b200.krylov import expm_krylov_batch
    g = torch.Generator(device="cuda").manual_seed(3)
    c = lambda *s: torch.complex(*torch.randn((2,) + s, dtype=torch.float64, device="cuda", generator=g))
    ops, vs = [], []
    for m in (5, 4):
        L, R = c(m, 2, m), c(m, 2, m)
        W = torch.randn(2, 3, 3, 2, dtype=torch.float64, device="cuda", generator=g)
        ops.append(HeffOperator((L + L.transpose(0, 2).conj()) / 2, (R + R.transpose(0, 2).conj()) / 2,
                                [W + W.transpose(1, 2)], (m, 3, m), prec="fp64"))
        vs.append(c(m * 3 * m))

    def apply(plain):
        def group(idx, xs):
            if where == "arguments":
                xs = list(xs) if plain else xs
                for i in range(len(xs)):
                    x = xs[i].view(ops[idx[i]].cshape)
                    xs[i] = VIEWS[view](x) if view != "transpose" else x.transpose(0, 2)
                return list(apply_grouped([ops[i] for i in idx], xs))
            ys = apply_grouped([ops[i] for i in idx], xs)
            ys = list(ys) if plain else ys
            for i in range(len(ys)):
                ys[i] = VIEWS[view](ys[i]) if view != "transpose" else ys[i].transpose(0, 2)
            return ys
        return group

    dts = [-0.01j, -0.02j]
    if where == "arguments" and view != "transpose":
        for plain in (True, False):
            with pytest.raises(AssertionError):
                expm_krylov_batch(apply(plain), dts, vs)
        return
    for (a, ka), (b, kb) in zip(expm_krylov_batch(apply(True), dts, vs), expm_krylov_batch(apply(False), dts, vs)):
        assert ka == kb and torch.equal(a, b)
