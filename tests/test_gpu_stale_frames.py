"""Lists of a frame whose scratch has since been drawn to in vain, resized or
drawn to without sorted lists (GPU) are refused."""
import numpy as np
import pytest

import splatfield_b200 as sf
from splatfield_b200 import synth
from splatfield_b200._lib import SF_ERR_CAPACITY

pytestmark = pytest.mark.gpu

N, SIZE = 820_000, (640, 640)
CAM = sf.look_at((0.0, 0.0, -3.0), (0.0, 0.0, 0.0))


def small_and_wide():
    """A scene, and one of 1.3e9 pairs in the same view."""
    attr, sh = synth.scene_uniform(N, 1, seed=7)
    a = attr.reshape(11, N).copy()
    a[0:3] *= 0.05
    a[7:10] = 1.0
    a[10] = 4.0
    return sf.Splats(attr, sh), sf.Splats(a.reshape(-1), sh)


def refused(call):
    with pytest.raises(sf.SplatfieldError):
        call()


@pytest.mark.parametrize("draw", ["prepare", "frame", "path"])
@pytest.mark.parametrize("build", [sf.ISECTS_BINNED, sf.ISECTS_DEPTH_SORTED])
def test_after_a_refused_frame(ctx, draw, build):
    small, wide = small_and_wide()
    scratch, acc = sf.RenderScratch(N, SIZE), sf.Accumulators(N)
    scratch.set_tuning(isect_build=build)
    small.render_forward(scratch, CAM, SIZE)
    isects = small.prepare_isects(scratch, CAM, SIZE)
    small.accumulate_prepared(scratch, isects, SIZE, acc)
    want = acc.bits.read()
    with pytest.raises(sf.SplatfieldError) as e:
        if draw == "prepare":
            wide.prepare_isects(scratch, CAM, SIZE)
        elif draw == "frame":
            wide.render_with(scratch, CAM, SIZE)
        else:
            wide.render_frames(scratch, [CAM] * 2, SIZE)
    assert e.value.code == SF_ERR_CAPACITY
    refused(lambda: small.accumulate_prepared(scratch, isects, SIZE, acc))
    refused(lambda: small.finalize_rgb(scratch, isects, SIZE))
    refused(lambda: small.render_backward(scratch, CAM, SIZE, np.zeros((*SIZE[::-1], 4), np.float32)))
    small.accumulate_prepared(scratch, small.prepare_isects(scratch, CAM, SIZE), SIZE, acc)
    np.testing.assert_array_equal(acc.bits.read(), want)


def test_after_the_lists_were_freed_or_left_out(ctx):
    n, size = 5000, (160, 120)
    splats = sf.Splats(*synth.scene_uniform(n, 1, seed=7))
    scratch, acc = sf.RenderScratch(n, size), sf.Accumulators(n)
    isects = splats.prepare_isects(scratch, CAM, size)
    scratch.reserve(2 * scratch.capacity())
    refused(lambda: splats.accumulate_prepared(scratch, isects, size, acc))
    isects = splats.prepare_isects(scratch, CAM, size)
    splats.accumulate_prepared(scratch, isects, size, acc)
    scratch.set_tuning(raster_order=sf.ORDER_IN_RASTER)
    splats.render_with(scratch, CAM, size)
    refused(lambda: splats.accumulate_prepared(scratch, isects, size, acc))
    refused(lambda: splats.finalize_rgb(scratch, isects, size))
