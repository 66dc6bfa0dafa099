"""Captured rounds and frames (GPU) follow the handles of each call: a handle
made where a freed one lay has other device buffers."""
import numpy as np
import pytest

import splatfield_b200 as sf
from splatfield_b200 import synth

pytestmark = pytest.mark.gpu

N, SIZE = 4000, (120, 90)


def scene(seed):
    return sf.Splats(*synth.scene_uniform(N, 1, seed=seed))


@pytest.mark.parametrize("form", ["responsibility", "evidence"])
def test_round_after_its_handles_were_freed(ctx, form):
    cams = synth.sphere_cameras(2, 3.0, 4, sf.look_at)
    rnd = sf.Round(N, [SIZE] * 2)
    held = []  # keeps freed device blocks from coming back in the same order
    for seed in range(6):
        splats, beta = scene(seed), sf.BetaState.from_host(*synth.beta_posterior(N, seed=seed))
        masks = [sf.Mask.from_bytes(SIZE, synth.ellipse_mask(*SIZE, seed + v)) for v in range(2)]
        if form == "responsibility":
            eig = rnd.eig(splats, beta, cams)
        else:
            eig = rnd.evidence(splats, beta, cams, masks)
        for v in range(2):
            scratch, acc = sf.RenderScratch(N, SIZE), sf.Accumulators(N)
            isects = splats.prepare_isects(scratch, cams[v], SIZE)
            splats.accumulate_prepared(scratch, isects, SIZE, acc, masks[v] if form == "evidence" else None)
            if form == "responsibility":
                np.testing.assert_array_equal(rnd.responsibility(v)[0].read(), acc.bits.read())
            else:
                for got, want in zip(rnd.evidence_words(v), (acc.fg, acc.bg)):
                    np.testing.assert_array_equal(got.read(), want.read())
            assert eig[v] == beta.eig(acc)
        del splats, beta, masks, scratch, acc, isects
        held.append(sf.DeviceBuffer.from_array(np.zeros(N, np.uint32)))


def test_frames_after_their_splats_were_freed(ctx):
    cam = sf.look_at((0.3, 0.2, -3.0), (0.0, 0.0, 0.0))
    scratch, held = sf.RenderScratch(N, SIZE), []
    for seed in range(6):
        splats = scene(seed)
        want = splats.render_with(sf.RenderScratch(N, SIZE), cam, SIZE).read()
        np.testing.assert_array_equal(splats.render_with(scratch, cam, SIZE).read(), want)
        del splats
        held.append(sf.DeviceBuffer.from_array(np.zeros(N, np.uint32)))
