"""Depth-limited lists of a round (GPU) whose heads, or whose heads and tails,
outgrow the lists' capacity: the round grows it and gives the words of the plain
per-view path, from its first call on. Each scene is made for one of the two
(and the large one for the kernels' shared memory past 10240 tiles)."""
import numpy as np
import pytest

import splatfield_b200 as sf
from splatfield_b200 import synth

pytestmark = pytest.mark.gpu


def scene(kind):
    n = {"heads": 700_000, "tails": 6_000_000, "tiles": 6_300_000}[kind]
    attr, sh = synth.scene_uniform(n, 1, seed=23)
    a = attr.reshape(11, n).copy()
    if kind == "heads":
        # One depth for all: heads are whole lists, 21M pairs.
        a[2] = 0.0
        a[7:10] += 1.3
    if kind == "tails":
        # Faint splats of a pixel or two: heads of 2.1M pairs, past which 702
        # of the 1056 tiles want their tails, 4.7M pairs (oracle).
        a[7:10] -= 2.0
        a[10] = -2.9
    if kind == "tiles":
        a[7:10] -= 0.7
    return a.reshape(-1), sh


@pytest.mark.parametrize("kind,size", [("heads", (512, 512)), ("tails", (520, 512)), ("tiles", (1792, 1648))])
@pytest.mark.parametrize("form", ["responsibility", "evidence", "adjoint"])
def test_first_rounds_match_whole_lists(ctx, capfd, kind, size, form):
    attr, sh = scene(kind)
    n = attr.size // 11
    splats, cam = sf.Splats(attr, sh), sf.look_at((0.0, 0.0, -3.0), (0.0, 0.0, 0.0))
    mask = sf.Mask.from_bytes(size, synth.ellipse_mask(size[0], size[1], 80))
    beta = sf.BetaState.from_host(*synth.beta_posterior(n, seed=3))
    scratch, acc = sf.RenderScratch(n, size), sf.Accumulators(n)
    if form == "adjoint":
        fg, bg = (x.read() for x in splats.render_feature_adjoint(scratch, cam, size, mask))
        want_eig = beta.eig_real(*splats.render_feature_adjoint(scratch, cam, size, mask))
    else:
        isects = splats.prepare_isects(scratch, cam, size)
        splats.accumulate_prepared(scratch, isects, size, acc, mask if form == "evidence" else None)
        want_eig = beta.eig(acc)
    rnd = sf.Round(n, [size])
    capfd.readouterr()
    for call in range(3):
        if form == "responsibility":
            eig = rnd.eig(splats, beta, [cam])[0]
            words, _, total, visible = rnd.responsibility(0)
            np.testing.assert_array_equal(words.read(), acc.bits.read())
            assert (total, visible) == (isects.num_isects, isects.num_visible)
        elif form == "evidence":
            eig = rnd.evidence(splats, beta, [cam], [mask])[0]
            for got, want in zip(rnd.evidence_words(0), (acc.fg, acc.bg)):
                np.testing.assert_array_equal(got.read(), want.read())
        else:
            eig = rnd.evidence_adjoint(splats, beta, [cam], [mask])[0]
            for got, want in zip(rnd.adjoint_responsibility(0), (fg, bg)):
                # f32 sums of the same terms in another order.
                np.testing.assert_allclose(got.read(), want, rtol=1e-5, atol=1e-6)
            assert abs(eig - want_eig) <= 1e-5 * abs(want_eig)
        if form != "adjoint":
            assert eig == want_eig
        grown = capfd.readouterr().err.count("capacity grown")
        # Once per cause, and only in the first call ("tails": its whole lists,
        # taken from the second call on, fit the grown lists).
        assert grown == (1 if call == 0 and kind != "tiles" else 0)
