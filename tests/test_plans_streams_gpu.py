"""Batched plans in flight on several streams at once, their tiles cut into many parts:
each launch's CTAs wait for one another, so every launch has to be resident as a
whole beside the others. Same bits as one plan at a time, no wait runs out."""
import pytest
import torch

import skgemm
from tests.test_batch_gpu import Item

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [128, 64])
@pytest.mark.parametrize("graph", [True, False])
def test_plans_on_several_streams_at_once(cuda, tile, graph):
    S, G = skgemm.OP_SYRK_PACKED, skgemm.OP_GEMM_PACKED
    sets = [[Item(S, 10 * i, 64, 64, 60000 + 16 * i), Item(G, 10 * i + 1, 100, 60, 30000),
             Item(S, 10 * i + 2, 130, 130, 20000)] for i in range(3)]
    plans = [skgemm.Plan([it.item() for it in s], tile=tile, tune=False, graph=graph)
             for s in sets]
    streams = [torch.cuda.Stream() for _ in plans]
    want = []
    for p, s in zip(plans, sets):
        p.run()
        torch.cuda.synchronize()
        want.append([it.dD.clone() for it in s])
    torch.cuda.synchronize()
    for _ in range(40):
        for p, st in zip(plans, streams):
            p.run(stream=st)
    for p, st in zip(plans, streams):
        p.status(stream=st)
    for s, w in zip(sets, want):
        for it, d in zip(s, w):
            assert torch.equal(it.dD, d)
            it.check(sample=200 if it.op == S else 0)
