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


@pytest.mark.parametrize("tile", [128, 64])
@pytest.mark.parametrize("grid", [1, 3, 4, 5, 6, 9, 40])
@pytest.mark.parametrize("tiles", [1, 3])
def test_tiles_around_the_shared_fixup_line(cuda, tile, grid, tiles):
    """Tiles cut into fewer parts than the shared fix-up takes, just as many, and more,
    alone and beside shorter ones (the group is launched with or without it)."""
    S, G = skgemm.OP_SYRK_PACKED, skgemm.OP_GEMM_PACKED
    items = [Item(G, 77, 40, 50, 6400)] + [Item(S, 80 + i, 30, 30, 900 + 16 * i)
                                           for i in range(tiles - 1)]
    p = skgemm.Plan([it.item() for it in items], tile=tile, grid=grid, tune=False, graph=False)
    p.run()
    p.status()
    for it in items:
        it.check()
