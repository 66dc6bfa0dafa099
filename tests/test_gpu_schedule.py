"""The rasterizer's longest-first block schedule (GPU), against the CPU oracle."""
import numpy as np
import pytest

import splatfield_b200 as sf
from splatfield_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(16, 16), (129, 97), (640, 33), (512, 512)])
def test_longest_first_schedule_draws_every_tile(ctx, oracle_mod, w, h):
    """Tile counts around multiples of 32 with empty tiles: a frame that
    follows a covered one on the same scratch overwrites every pixel (the
    schedule's list of empty tiles holds each of them once, and no other)."""
    O = oracle_mod
    n = 200
    attr, sh = synth.scene_uniform(n, 1, 9)
    wide = attr.reshape(11, n).copy()
    wide[7:10] = 1.0
    wide[10] = 8.0
    pos, tgt = (0.3, -0.2, -3.0), (0.0, 0.0, 0.0)
    cam_o, cam = O.look_at(pos, tgt), sf.look_at(pos, tgt)
    want = O.rasterize(O.prepare(cam_o, w, h, attr, sh, 1), 0)["bitmap"][:, :w]
    cover, splats = sf.Splats(wide.reshape(-1), sh), sf.Splats(attr, sh)
    scratch = sf.RenderScratch(n, (w, h))
    scratch.set_tuning(raster_schedule=sf.SCHEDULE_LONGEST)
    for _ in range(20):
        cover.render_with(scratch, cam, (w, h))
        np.testing.assert_array_equal(splats.render_with(scratch, cam, (w, h)).read()[:, :w], want)
