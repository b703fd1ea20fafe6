"""Rounds of the batch kernel end by the clock: their length changes when pixels are compacted, never
what they are -- one step a round, rounds longer than any pixel, and the default give the same maps."""
from decimal import Decimal

import numpy as np
import pytest

from fractura_b200 import batch as fb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arith", ["ref_cpu", "fast"])
def test_round_lengths_give_the_same_maps(arith):
    import torch
    # bounded and escaping pixels of the three formulas, more pixels than one block's slots
    tiles = [fb.Tile(cx=Decimal(cx), cy=Decimal(cy), width=Decimal(w), W=61, H=47, max_iter=3000, fractal_type=ft,
                     gen_n=3, gen_kr=0.25, gen_ki=0.1, strict_glitch=False, rebase=arith == "fast")
             for ft, cx, cy, w in ((0, "-0.75", "0.1", "0.4"), (1, "-1.7", "-0.03", "0.2"), (4, "0.1", "0.6", "0.8"))]
    b = fb.prepare_batch(tiles, arith=arith, bla_form="accurate")
    maps = []
    for cfg in (fb.BatchConfig(), fb.BatchConfig(quantum=1, blocks_per_sm=1), fb.BatchConfig(quantum=1 << 20)):
        for out in b.tiles_out:
            out["kmap"].fill_(-7)
        b.render(cfg)
        torch.cuda.synchronize()
        maps.append([(o["kmap"].cpu().numpy().copy(), o["iter"].cpu().numpy().copy()) for o in b.tiles_out])
    for other in maps[1:]:
        for (k0, i0), (k1, i1) in zip(maps[0], other):
            assert np.array_equal(k0, k1) and np.array_equal(i0.view(np.uint32), i1.view(np.uint32))
    assert all((k != -7).all() for k, _ in maps[0]) and any((k == -1).any() for k, _ in maps[0])
