"""The tile walks at the sizes and shapes where their culls, warp sums and
flushes could go wrong (GPU), against the CPU oracle or the u32 lift."""
import numpy as np
import pytest

import splatfield_b200 as sf
from splatfield_b200 import synth

pytestmark = pytest.mark.gpu


def thin_scene(n, seed, long_scale):
    """Splats of one long axis (log-scale `long_scale`) and two short ones."""
    rng = np.random.default_rng(seed)
    attr = np.zeros((11, n), np.float32)
    attr[0:3] = rng.uniform(-1.0, 1.0, (3, n))
    q = rng.standard_normal((4, n))
    attr[3:7] = q / np.linalg.norm(q, axis=0)
    attr[7] = long_scale
    attr[8:10] = -5.0
    attr[10] = rng.standard_normal(n)
    sh = (0.5 * rng.standard_normal((3, n))).astype(np.float32)
    return attr.reshape(-1), sh.reshape(-1)


@pytest.mark.parametrize("cull", [0, 1])
@pytest.mark.parametrize("long_scale", [-5.0, 0.0, 1.5, 3.0, 4.0, 45.0])
@pytest.mark.parametrize("w,h", [(129, 97), (640, 33)])
def test_thin_splats_match_oracle(ctx, oracle_mod, w, h, long_scale, cull):
    """Needles from a pixel to far past the image (and of infinite extent,
    log-scale 45): the per-warp cull skips no pair that the oracle composites."""
    O = oracle_mod
    n = 300
    attr, sh = thin_scene(n, 7, long_scale)
    pos, tgt = (0.3, -0.2, -3.0), (0.0, 0.0, 0.0)
    cam_o, cam = O.look_at(pos, tgt), sf.look_at(pos, tgt)
    want = O.prepare(cam_o, w, h, attr, sh, 1)
    splats = sf.Splats(attr, sh)
    scratch = sf.RenderScratch(n, (w, h))
    scratch.set_tuning(raster_cull=cull)
    got = splats.render_with(scratch, cam, (w, h)).read()
    np.testing.assert_array_equal(got[:, :w], O.rasterize(want, 0)["bitmap"][:, :w])
    acc = sf.Accumulators(n)
    splats.render_responsibility(scratch, acc, cam, (w, h))
    np.testing.assert_array_equal(acc.bits.read(), O.rasterize(want, 1, scale=acc.scale)["resp"])


@pytest.mark.parametrize("split", [1, 2, 4])
@pytest.mark.parametrize("n", [1, 33, 700, 6000])
@pytest.mark.parametrize("masked", [False, True])
def test_real_responsibilities_match_u32_lift(ctx, n, split, masked):
    """The adjoint responsibilities bound the u32 words of the same view as
    truncation allows (each pixel loses less than one unit; f32 sums of a few
    hundred positive terms drift by less than 1e-5), at list lengths around
    the chunk and group sizes and at masks that cut through pixel blocks."""
    sizes = [(16, 16), (37, 61), (130, 18)]
    attr, sh = synth.scene_uniform(n, 1, 23)
    splats = sf.Splats(attr, sh)
    cams = synth.sphere_cameras(len(sizes), 2.5, 3, sf.look_at)
    masks = [sf.Mask.from_bytes(s, synth.ellipse_mask(s[0], s[1], 60 + v)) for v, s in enumerate(sizes)]
    rnd = sf.Round(n, sizes)
    rnd.set_tuning(lanes=2, raster_split=split)
    rnd.evidence_adjoint(splats, None, cams, masks if masked else None)
    for v, s in enumerate(sizes):
        scratch, acc = sf.RenderScratch(n, s), sf.Accumulators(n)
        isects = splats.prepare_isects(scratch, cams[v], s)
        splats.accumulate_prepared(scratch, isects, s, acc, masks[v] if masked else None)
        pixels = 256.0 * scratch.read(sf._lib.READ_TILE_COUNTS, n).astype(np.float64)
        got = [x.read().astype(np.float64) * acc.scale for x in rnd.adjoint_responsibility(v)]
        want = [acc.fg.read(), acc.bg.read()] if masked else [acc.bits.read(), np.zeros(n)]
        for g, u in zip(got, want):
            diff = g - u.astype(np.float64)
            assert np.all(diff >= -1e-5 * g - 1.0) and np.all(diff <= 1e-5 * g + pixels + 1.0)
