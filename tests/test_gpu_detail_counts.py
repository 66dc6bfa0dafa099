"""The pair diagnostics (GPU) count list entries only: both walks evaluate the
same (pixel, entry) pairs whatever the number of entries of a group."""
import numpy as np
import pytest

import splatfield_b200 as sf
from splatfield_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 33, 64, 3001])
@pytest.mark.parametrize("order", [sf.ORDER_SORTED, sf.ORDER_IN_RASTER])
def test_both_walks_evaluate_the_same_pairs(ctx, n, order):
    """A culled pair's power is above power_max at every pixel of the block, so
    the culled walk leaves out no evaluated pair."""
    attr, sh = synth.scene_uniform(n, 1, 13)
    attr = attr.reshape(11, n).copy()
    attr[0:3] *= 0.3
    attr[10] = 1.0
    splats, size = sf.Splats(attr.reshape(-1), sh), (200, 150)
    cam = sf.look_at((0.0, 0.0, -2.0), (0.0, 0.0, 0.0))
    got = []
    for cull in (0, 1):
        scratch = sf.RenderScratch(n, size)
        scratch.set_tuning(raster_cull=cull, raster_detail=1, raster_order=order)
        splats.render_with(scratch, cam, size)
        got.append(scratch.stats())
    assert got[0]["exp_evaluated"] == got[1]["exp_evaluated"] >= got[0]["contributing"] > 0
    assert got[0]["contributing"] == got[1]["contributing"]
    assert got[0]["pairs_processed"] >= got[1]["pairs_processed"]
