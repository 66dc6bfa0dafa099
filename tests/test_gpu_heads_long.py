"""Rounds whose heads or whole lists are long (GPU): which form and sort each
call captures, and the per-view path's words in every call."""
import numpy as np
import pytest

import splatfield_b200 as sf
from splatfield_b200 import synth
from splatfield_b200._lib import lib

pytestmark = pytest.mark.gpu

SIZE = (512, 512)


def patch_scene(n, edge):
    """Nine splats of ten in a slab of `edge` in front of the camera, faint and
    of a pixel or two; the others anywhere."""
    attr, sh = synth.scene_uniform(n, 1, seed=29)
    a = attr.reshape(11, n).copy()
    m = 9 * n // 10
    a[0:2, :m] *= 0.5 * edge
    a[2, :m] *= 0.2
    a[7:10] -= 2.0
    a[10] = -2.9
    return a, sh


def run(a, sh, calls, size=SIZE):
    """Kernel launches of each call, whose words it checks."""
    n = a.shape[1]
    splats, cam = sf.Splats(a.reshape(-1), sh), sf.look_at((0.0, 0.0, -3.0), (0.0, 0.0, 0.0))
    scratch, acc = sf.RenderScratch(n, size), sf.Accumulators(n)
    splats.render_responsibility(scratch, acc, cam, size)
    want = acc.bits.read()
    rnd, launched = sf.Round(n, [size]), []
    for _ in range(calls):
        before = lib().sf_kernel_launches()
        rnd.eig(splats, None, [cam])
        launched.append(lib().sf_kernel_launches() - before)
        np.testing.assert_array_equal(rnd.responsibility(0)[0].read(), want)
    return launched


def test_whole_lists_after_heads_take_the_segmented_sort_at_once(ctx):
    """Heads leave 36 tiles open, 16 of them with lists of 27000 to 41700 entries
    (oracle): the second call takes whole lists, with the seven launches of
    their segmented sort."""
    first, second, third = run(*patch_scene(1_000_000, 0.4), 3)
    assert first != second == third


@pytest.mark.parametrize("order", [1, -1])
def test_heads_of_splats_stored_in_depth_order(ctx, order):
    """15.4M pairs, some 15000 a tile. Heads cut by the farthest or the nearest
    splats alone would hold most of the list (past the 2^22 pairs that a round
    of 1024 tiles has room for at first) or leave most tiles open. No call
    grows the room or falls back to whole lists."""
    n = 3_000_000
    attr, sh = synth.scene_uniform(n, 1, seed=17)
    a = attr.reshape(11, n).copy()
    a[0:2] *= 0.6
    a[2] = np.sort(a[2])[::order]
    assert len(set(run(a, sh, 6))) == 1
