"""Binned lists (GPU) at the splat counts where the build's chunks change (128
and 512 splats a chunk on 148 SMs), of small splats and of few large ones,
against the CPU oracle."""
import numpy as np
import pytest

import splatfield_b200 as sf
from splatfield_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,grow", [(1, 5.0), (127, 5.0), (129, 4.0), (600, 3.0), (128 * 148 - 1, 0.0),
                                    (128 * 148 + 1, 0.0), (512 * 148 - 31, 0.0), (512 * 148 + 1, 0.0)])
def test_lists_equal_the_oracle(ctx, oracle_mod, n, grow):
    w, h = 333, 217
    attr, sh = synth.scene_uniform(n, 1, 21)
    attr = attr.reshape(11, n).copy()
    attr[7:10] += grow
    attr[10] = np.abs(attr[10])
    pos, tgt = (0.1, 0.2, -2.5), (0.0, 0.0, 0.0)
    scratch = sf.RenderScratch(n, (w, h))
    ti = sf.Splats(attr.reshape(-1), sh).prepare_isects(scratch, sf.look_at(pos, tgt), (w, h))
    want = oracle_mod.prepare(oracle_mod.look_at(pos, tgt), w, h, attr.reshape(-1), sh, 1)
    assert ti.num_visible == want["num_visible"] > 0
    np.testing.assert_array_equal(ti.tile_ids().read(), want["tile_ids"])
    np.testing.assert_array_equal(ti.gaussian_ids().read(), want["gaussian_ids"])
