"""Projection on either side of the size at which its blocks change, with a
last block that is full, nearly empty or nearly full."""
import numpy as np
import pytest

import splatfield_b200 as sf
from splatfield_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 16])
@pytest.mark.parametrize("n", [(1 << 18) - 1, 1 << 18, (1 << 18) + 1, (1 << 18) + 127])
def test_lists_equal_the_oracle(ctx, oracle_mod, n, k):
    w, h = 208, 144
    attr, sh = synth.scene_uniform(n, k, 17)
    pos, tgt = (0.1, 0.2, -2.5), (0.0, 0.0, 0.0)
    scratch = sf.RenderScratch(n, (w, h))
    ti = sf.Splats(attr, sh).prepare_isects(scratch, sf.look_at(pos, tgt), (w, h))
    want = oracle_mod.prepare(oracle_mod.look_at(pos, tgt), w, h, attr, sh, k)
    assert ti.num_visible == want["num_visible"]
    np.testing.assert_array_equal(ti.tile_ids().read(), want["tile_ids"])
    np.testing.assert_array_equal(ti.gaussian_ids().read(), want["gaussian_ids"])
