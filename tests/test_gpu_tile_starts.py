"""Tile starts of the binned build (GPU) around the scan's 4096-count steps and
its 4-count loads, and chunk counts around one chunk of splats."""
import numpy as np
import pytest

import splatfield_b200 as sf
from splatfield_b200 import _lib as L
from splatfield_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 511, 513, 20_000])
@pytest.mark.parametrize("w,h", [(16, 16), (48, 17), (1040, 1008), (1024, 1024), (1056, 1024), (2064, 1024)])
def test_tile_starts_are_the_prefix_of_the_lists(ctx, oracle_mod, w, h, n):
    attr, sh = synth.scene_uniform(n, 1, 31)
    pos, tgt = (0.1, 0.0, -2.5), (0.0, 0.0, 0.0)
    cam = sf.look_at(pos, tgt)
    scratch = sf.RenderScratch(n, (w, h))
    splats = sf.Splats(attr, sh)
    tiles = ((w + 15) // 16) * ((h + 15) // 16)
    ti = splats.prepare_isects(scratch, cam, (w, h))
    start = scratch.read(L.READ_TILE_START, tiles + 1)
    want = oracle_mod.prepare(oracle_mod.look_at(pos, tgt), w, h, attr, sh, 1)
    assert ti.num_isects == want["tile_ids"].size == start[-1]
    np.testing.assert_array_equal(start[:-1], np.searchsorted(want["tile_ids"], np.arange(tiles)))
    np.testing.assert_array_equal(ti.gaussian_ids().read(), want["gaussian_ids"])


def test_frame_past_the_capacity_is_drawn_again_whole(ctx, oracle_mod):
    """Starts cut at the capacity: a frame whose pairs outgrow it comes out
    whole after the growth, in the graph and on a camera path."""
    n, w, h = 3000, 320, 240
    attr, sh = synth.scene_uniform(n, 1, 5)
    big = attr.reshape(11, n).copy()
    big[7:10] += 3.0
    pos, tgt = (0.1, 0.0, -2.5), (0.0, 0.0, 0.0)
    cam = sf.look_at(pos, tgt)
    small, splats = sf.Splats(attr, sh), sf.Splats(big.reshape(-1), sh)
    want = oracle_mod.rasterize(oracle_mod.prepare(oracle_mod.look_at(pos, tgt), w, h, big.reshape(-1), sh, 1), 0)
    scratch = sf.RenderScratch(n, (w, h))
    small.render_with(scratch, cam, (w, h))
    got = splats.render_frames_to_host(scratch, [cam] * 5, (w, h))
    for img in got:
        np.testing.assert_array_equal(img, want["bitmap"][:, :w])


def test_prepare_past_the_capacity_places_again(ctx, oracle_mod):
    """The placement runs before the host knows the total: lists that outgrow
    the capacity of an earlier frame are placed again after the growth."""
    n, w, h = 6000, 640, 480
    attr, sh = synth.scene_uniform(n, 1, 5)
    big = attr.reshape(11, n).copy()
    big[7:10] += 4.0
    pos, tgt = (0.1, 0.0, -2.5), (0.0, 0.0, 0.0)
    cam = sf.look_at(pos, tgt)
    small, splats = sf.Splats(attr, sh), sf.Splats(big.reshape(-1), sh)
    want = oracle_mod.prepare(oracle_mod.look_at(pos, tgt), w, h, big.reshape(-1), sh, 1)
    scratch = sf.RenderScratch(n, (w, h))
    small.prepare_isects(scratch, cam, (w, h))
    before = scratch.capacity()
    assert want["gaussian_ids"].size > before
    ti = splats.prepare_isects(scratch, cam, (w, h))
    assert scratch.capacity() > before
    np.testing.assert_array_equal(ti.gaussian_ids().read(), want["gaussian_ids"])
    np.testing.assert_array_equal(ti.tile_ids().read(), want["tile_ids"])
