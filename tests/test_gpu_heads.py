"""Depth-limited lists of a round (GPU): views of many splats whose heads
suffice, whose tails are wanted everywhere, whose depths are all equal, and
whose lists outgrow the capacity give the words of the plain per-view path,
which sorts whole lists."""
import numpy as np
import pytest

import splatfield_b200 as sf
from splatfield_b200 import synth

pytestmark = pytest.mark.gpu

N = 650_000  # heads are taken from 640k splats and 1024 tiles on


def scene(kind):
    attr, sh = synth.scene_clustered(N, 1, seed=17) if kind != "flat" else synth.scene_uniform(N, 1, seed=17)
    a = attr.reshape(11, N).copy()
    if kind == "faint":
        # Opacities just above the cull: no pixel saturates early, so every
        # tile walks far past its head.
        a[10] = -2.9
    if kind == "flat":
        # One depth for all: every limit takes the whole list.
        a[2] = 0.0
    if kind == "big":
        a[7:10] += 0.8
    return a.reshape(-1), sh


@pytest.mark.parametrize("kind", ["clustered", "faint", "flat", "big"])
@pytest.mark.parametrize("form,split", [("responsibility", 1), ("evidence", 2), ("adjoint", 4)])
def test_round_words_match_whole_lists(ctx, kind, form, split):
    attr, sh = scene(kind)
    splats = sf.Splats(attr, sh)
    sizes = [(512, 512), (523, 511), (96, 64)]  # the last one takes whole lists
    if kind == "flat":
        cams = [sf.look_at((0.0, 0.0, -3.0), (0.0, 0.0, 0.0)) for _ in sizes]
    else:
        cams = synth.sphere_cameras(len(sizes), 3.5, 4, sf.look_at)
    masks = [sf.Mask.from_bytes(s, synth.ellipse_mask(s[0], s[1], 80 + v)) for v, s in enumerate(sizes)]
    a, b = synth.beta_posterior(N, seed=3)
    beta = sf.BetaState.from_host(a, b)
    rnd = sf.Round(N, sizes)
    rnd.set_tuning(lanes=2, raster_split=split)
    for _ in range(2):
        if form == "responsibility":
            eig = rnd.eig(splats, beta, cams)
        elif form == "evidence":
            eig = rnd.evidence(splats, beta, cams, masks)
        else:
            eig = rnd.evidence_adjoint(splats, beta, cams, masks)
    for v, s in enumerate(sizes):
        scratch, acc = sf.RenderScratch(N, s), sf.Accumulators(N)
        if form == "adjoint":
            fg, bg = splats.render_feature_adjoint(scratch, cams[v], s, masks[v])
            for got, want in zip(rnd.adjoint_responsibility(v), (fg, bg)):
                # f32 sums of the same terms in another order.
                np.testing.assert_allclose(got.read(), want.read(), rtol=1e-5, atol=1e-6)
            assert abs(eig[v] - beta.eig_real(fg, bg)) <= 1e-5 * abs(eig[v])
            continue
        isects = splats.prepare_isects(scratch, cams[v], s)
        splats.accumulate_prepared(scratch, isects, s, acc, masks[v] if form == "evidence" else None)
        if form == "responsibility":
            words, _, total, visible = rnd.responsibility(v)
            np.testing.assert_array_equal(words.read(), acc.bits.read())
            assert (total, visible) == (isects.num_isects, isects.num_visible)
        else:
            for got, want in zip(rnd.evidence_words(v), (acc.fg, acc.bg)):
                np.testing.assert_array_equal(got.read(), want.read())
        assert eig[v] == beta.eig(acc)
