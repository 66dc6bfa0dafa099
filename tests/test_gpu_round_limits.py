"""Rounds past the intersection limit (GPU) are refused whatever the form of
their lists."""
import pytest

import splatfield_b200 as sf
from splatfield_b200 import synth
from splatfield_b200._lib import SF_ERR_CAPACITY

pytestmark = pytest.mark.gpu


def test_whole_lists_past_the_limit_are_refused(ctx):
    """820k splats that each cover 1600 tiles: 1.3e9 pairs, of which the nearest
    few thousand a tile saturate every pixel. The round takes other splats
    afterwards."""
    n, size = 820_000, (640, 640)
    attr, sh = synth.scene_uniform(n, 1, seed=7)
    a = attr.reshape(11, n).copy()
    a[0:3] *= 0.05
    a[7:10] = 1.0
    a[10] = 4.0
    cam = sf.look_at((0.0, 0.0, -3.0), (0.0, 0.0, 0.0))
    beta = sf.BetaState.from_host(*synth.beta_posterior(n, seed=3))
    small, wide = sf.Splats(attr, sh), sf.Splats(a.reshape(-1), sh)
    rnd = sf.Round(n, [size])
    # Room for far more than the heads: whole lists of a scene that has them.
    a[7:10] = -3.0
    rnd.set_tuning(raster_order=sf.ORDER_IN_RASTER)
    rnd.eig(sf.Splats(a.reshape(-1), sh), beta, [cam])
    assert rnd.responsibility(0)[2] > 1 << 23
    rnd.set_tuning(raster_order=sf.ORDER_SORTED)
    for _ in range(2):
        with pytest.raises(sf.SplatfieldError) as e:
            rnd.eig(wide, beta, [cam])
        assert e.value.code == SF_ERR_CAPACITY
    with pytest.raises(sf.SplatfieldError) as e:
        wide.prepare_isects(sf.RenderScratch(n, size), cam, size)
    assert e.value.code == SF_ERR_CAPACITY
    assert rnd.eig(small, beta, [cam])[0] > 0.0
