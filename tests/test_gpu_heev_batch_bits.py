"""A matrix's eigenpairs do not depend on what else is in the call: batches
large enough that the inverse iteration leaves shared memory give, bit for bit, the
values and vectors of single calls, which stay in it (the reduction on
clusters, the tile of every product and the panels of these QRs depend on each matrix alone)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,kt", [([424] * 19, 424), ([400, 20, 1, 65, 130] * 6, 400)])
def test_batch_is_each_ones_own(ns, kt):
    from renormalizer_b200._native import Engine
    from renormalizer_b200.heev import heev_top, heev_top_batched
    eng = Engine.get(0)
    g = torch.Generator(device="cuda").manual_seed(len(ns))
    Gs = []
    for n in ns:
        x = torch.complex(*torch.randn((2, n, n), dtype=torch.float64, device="cuda", generator=g))
        x = x * 10.0 ** (-6.0 * torch.arange(n, device="cuda", dtype=torch.float64) / n)
        Gs.append(x.mH @ x)
    # turns of the shared-memory form in the batch: more than four per SM, so it takes the other
    lanes = (227 * 1024 // 8 - 2 * max(ns)) // (5 * max(ns))
    assert -(-min(kt, max(ns)) // lanes) * len(ns) > 4 * torch.cuda.get_device_properties(0).multi_processor_count
    kts = [min(kt, n) for n in ns]
    for G, k, (w, K, _) in zip(Gs, kts, heev_top_batched(eng, Gs, kts)):
        w1, K1, _ = heev_top(eng, G, k)
        assert torch.equal(w, w1) and torch.equal(K, K1)
