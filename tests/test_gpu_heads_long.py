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


FAINT = sf.look_at((20.0, 0.0, -3.0), (20.0, 0.0, 0.0))


def two_scenes():
    """650k splats whose heads suffice and, beside them in view of FAINT alone,
    300k that leave some 36 tiles open."""
    attr, sh = synth.scene_clustered(650_000, 1, seed=17)
    faint, sh2 = patch_scene(300_000, 0.4)
    faint[0] += 20.0
    a = np.concatenate([attr.reshape(11, -1), faint], axis=1)
    return sf.Splats(a.reshape(-1), np.concatenate([sh.reshape(3, -1), sh2.reshape(3, -1)], axis=1).reshape(-1))


def rounds(splats, cams_of, calls):
    n, launched = splats.n, []
    rnd = sf.Round(n, [SIZE] * 3)
    for k in range(calls):
        before = lib().sf_kernel_launches()
        rnd.eig(splats, None, cams_of(k))
        launched.append(lib().sf_kernel_launches() - before)
        v = k % 3
        if k > 6:
            continue
        scratch, acc = sf.RenderScratch(n, SIZE), sf.Accumulators(n)
        splats.render_responsibility(scratch, acc, cams_of(k)[v], SIZE)
        np.testing.assert_array_equal(rnd.responsibility(v)[0].read(), acc.bits.read())
    return launched


def test_a_passing_faint_view_leaves_its_slot_on_heads(ctx):
    """The faint camera is in another slot each round."""
    near = [sf.look_at((0.2 * j, 0.1, -3.5), (0.0, 0.0, 0.0)) for j in range(3)]
    launched = rounds(two_scenes(), lambda k: [FAINT if j == k % 3 else near[j] for j in range(3)], 6)
    assert len(set(launched)) == 1


def test_a_lasting_faint_view_takes_whole_lists_for_some_rounds(ctx):
    """From the second round of the same cameras on, for 64 rounds, then heads
    are tried once and 128 rounds follow."""
    near = [sf.look_at((0.2 * j, 0.1, -3.5), (0.0, 0.0, 0.0)) for j in range(3)]
    launched = rounds(two_scenes(), lambda k: [near[0], FAINT, near[2]], 2 + 64 + 1 + 128 + 1)
    heads, whole = launched[0], launched[2]
    assert heads > whole
    assert launched == [heads] * 2 + [whole] * 64 + [heads] + [whole] * 128 + [heads]
