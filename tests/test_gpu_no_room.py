"""A scratch asked for an image that does not fit the GPU (GPU): an error each
time, and the next size works."""
import numpy as np
import pytest

import splatfield_b200 as sf
from splatfield_b200 import synth
from splatfield_b200._lib import SF_ERR_NOMEM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["prepare_isects", "render_with", "render_float"])
def test_image_past_the_memory(ctx, call):
    """A 1.1 TB image behind 4.3 GB of tile starts, which are given back."""
    n, size, huge = 3000, (160, 120), (1 << 19, 1 << 19)
    splats, cam = sf.Splats(*synth.scene_uniform(n, 1, seed=5)), sf.look_at((0.0, 0.0, -3.0), (0.0, 0.0, 0.0))
    want = splats.render_with(sf.RenderScratch(n, size), cam, size).read()
    scratch = sf.RenderScratch(n, size)
    for _ in range(2):
        for _ in range(2):
            with pytest.raises(sf.SplatfieldError) as e:
                getattr(splats, call)(scratch, cam, huge)
            assert e.value.code == SF_ERR_NOMEM
        np.testing.assert_array_equal(splats.render_with(scratch, cam, size).read(), want)
