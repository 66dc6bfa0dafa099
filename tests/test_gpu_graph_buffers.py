"""A captured frame (GPU) goes with its scratch's buffers: a scratch resized by
another call and back draws into the buffers it has now."""
import numpy as np
import pytest

import splatfield_b200 as sf
from splatfield_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frames", [1, 3])
def test_frame_after_its_scratch_was_resized_and_back(ctx, frames):
    n, size, other = 5000, (160, 120), (333, 217)
    splats = sf.Splats(*synth.scene_uniform(n, 1, seed=3))
    cams = synth.sphere_cameras(frames, 3.0, 4, sf.look_at)
    scratch, held = sf.RenderScratch(n, size), []

    def draw(s):
        if frames > 1:
            return splats.render_frames_to_host(s, cams, size)
        return [splats.render_with(s, cams[0], size).read()]

    for words in (1, 200, 40_000, 300_000):
        want = draw(sf.RenderScratch(n, size))
        for got, w in zip(draw(scratch), want):
            np.testing.assert_array_equal(got, w)
        splats.prepare_isects(scratch, cams[0], other)
        # Takes a freed block, so that the buffers do not come back in order.
        held.append(sf.DeviceBuffer.from_array(np.zeros(words, np.uint32)))
        splats.prepare_isects(scratch, cams[0], size)
    for got, w in zip(draw(scratch), want):
        np.testing.assert_array_equal(got, w)
