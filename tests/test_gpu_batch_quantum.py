"""A short quantum is a number of loop steps: rounds of 1, 5 and 16 steps pause every pixel at the same
states in every run, so the work counters repeat (those of pixels that end in a cycle too), and the
maps are those of the default rounds."""
import ctypes as C
from decimal import Decimal

import numpy as np
import pytest

from fractura_b200 import batch as fb
from fractura_b200 import high_precision as hp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quantum", [1, 5, 16])
def test_short_rounds_repeat(quantum):
    import torch
    hp.clear_reference_orbit_cache()
    # a reference with a periodic tail, bounded pixels of a Multibrot, and a direct second stage
    tiles = [fb.Tile(cx=Decimal(cx), cy=Decimal(cy), width=Decimal(w), W=29, H=23, max_iter=mi, fractal_type=ft, gen_n=3,
                     gen_kr=0.25, gen_ki=0.1, strict_glitch=False, rebase=rebase)
             for ft, cx, cy, w, mi, rebase in ((0, "-0.1226", "0.7449", "1e-13", 2500, True), (0, "-0.1226", "0.7449", "0.2", 2500, False),
                                               (4, "0.1", "0.6", "0.8", 2000, True), (4, "0.1", "0.6", "0.8", 2000, False))]
    b = fb.prepare_batch(tiles, arith="ref_cuda", bla_form="accurate")
    work = [torch.zeros((t.H, t.W, 4), dtype=torch.int32, device="cuda") for t in tiles]
    for slot, q in enumerate(b.order):
        b.desc_host[slot].counters = C.c_void_p(work[q].data_ptr())
    b.desc_dev = torch.from_numpy(np.frombuffer(bytes(b.desc_host), dtype=np.uint8).copy()).cuda()
    runs = []
    for cfg in [fb.BatchConfig()] + [fb.BatchConfig(quantum=quantum, blocks_per_sm=s) for s in (1, 2, 1)]:
        b.render(cfg)
        torch.cuda.synchronize()
        runs.append(([(o["kmap"].cpu().numpy().copy(), o["iter"].cpu().numpy().view(np.uint32).copy()) for o in b.tiles_out],
                     [w.cpu().numpy().copy() for w in work]))
    assert any((k == -1).any() for k, _ in runs[0][0])
    for maps, _ in runs[1:]:
        assert all(np.array_equal(x, y) for p, q in zip(runs[0][0], maps) for x, y in zip(p, q))
    for _, counts in runs[2:]:
        assert all(np.array_equal(x, y) for x, y in zip(runs[1][1], counts))
