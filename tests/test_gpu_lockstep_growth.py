"""Lockstep exponentials of which a few need more Krylov vectors than the rows
first taken: those move to a buffer of their own, the finished ones' memory
goes, and every result is its own exponential's, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _problems(sizes, ranges):
    g = torch.Generator(device="cuda").manual_seed(4)
    ds, vs = [], []
    for n, r in zip(sizes, ranges):
        ds.append(r * torch.rand(n, dtype=torch.float64, device="cuda", generator=g))
        v = torch.complex(*torch.randn((2, n), dtype=torch.float64, device="cuda", generator=g))
        vs.append(v / torch.linalg.vector_norm(v))
    return ds, vs


@pytest.mark.parametrize("block", [2, 5, 8, 50])
def test_results_across_growth(block):
    from renormalizer_b200.krylov import expm_krylov, expm_krylov_batch
    ds, vs = _problems([300, 7, 1000, 1, 64, 501, 20], [40.0, 5.0, 1.0, 3.0, 90.0, 20.0, 200.0])
    got = expm_krylov_batch(lambda idx, xs: [ds[i] * x for i, x in zip(idx, xs)], -0.5j, vs, block)
    counts = []
    for d, v, (y, k) in zip(ds, vs, got):
        ref, kr = expm_krylov(lambda x: d * x, -0.5j, v, block)
        assert k == kr and torch.equal(y, ref)
        counts.append(k)
    assert max(counts) > 24 and counts[2] == 7  # one of them past several growths of 8, one before the first


def test_only_unfinished_problems_grow():
    from renormalizer_b200.krylov import expm_krylov_batch
    N = 1 << 20
    ds, vs = _problems([N, 64], [0.1, 90.0])
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    (_, k0), (_, k1) = expm_krylov_batch(lambda idx, xs: [ds[i] * x for i, x in zip(idx, xs)], -0.5j, vs, 8)
    assert k0 == 7 and k1 > 24
    # 8 rows, the combination, its copy, an image and its conversions: 13 vectors; 24 when all grow
    assert torch.cuda.max_memory_allocated() - before <= 14 * 16 * N
