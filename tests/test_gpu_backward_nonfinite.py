"""A non-finite dL/d(rgba) at one pixel (GPU) spoils the adjoints of the splats
that the pixel composites and of no others."""
import numpy as np
import pytest

import splatfield_b200 as sf

pytestmark = pytest.mark.gpu

POS, TGT = (0.2, -0.1, -2.6), (0.0, 0.0, 0.0)


def scene(n, k, seed):
    rng = np.random.default_rng(seed)
    a = np.zeros((11, n))
    a[0:2] = rng.uniform(-0.7, 0.7, (2, n))
    a[2] = rng.uniform(-0.4, 0.6, n)
    q = rng.normal(size=(4, n))
    a[3:7] = q / np.linalg.norm(q, axis=0)
    a[7:10] = rng.normal(-2.9, 0.35, (3, n))
    a[10] = rng.normal(0.0, 1.2, n)
    sh = rng.normal(0, 0.3, (k, 3, n))
    return a.astype(np.float32).reshape(-1), sh.astype(np.float32).reshape(-1)


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-12))


@pytest.mark.parametrize("covered", [True, False])
@pytest.mark.parametrize("channel", [0, 1, 2, 3])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_other_splats_keep_finite_gradients(ctx, oracle_mod, covered, channel, bad):
    """The pixel's own splats come from a one-hot gradient at it; the others'
    gradients agree with the FP64 adjoint of the same dL with the pixel's set
    to zero (relative L2 below 5e-3, as for finite gradients)."""
    n, k, w, h = 700, 4, 96, 80
    attr, sh = scene(n, k, 5)
    rng = np.random.default_rng(6)
    splats, scratch = sf.Splats(attr, sh), sf.RenderScratch(n, (w, h))
    cam = sf.look_at(POS, TGT)
    alpha = splats.render_forward(scratch, cam, (w, h)).read()[..., 3]
    # A covered pixel amid others; or one that nothing covers, beside covered
    # ones of its 8x4 block.
    blocks = alpha.reshape(h // 4, 4, w // 8, 8)
    if covered:
        y, x = np.unravel_index(np.argmax(alpha), alpha.shape)
    else:
        part = (blocks == 0).any(axis=(1, 3)) & (blocks > 0).any(axis=(1, 3))
        by, bx = np.argwhere(part)[0]
        iy, ix = np.argwhere(blocks[by, :, bx, :] == 0)[0]
        y, x = 4 * by + iy, 8 * bx + ix
    hot = np.zeros((h, w, 4), np.float32)
    hot[y, x, 0] = 1.0
    seen = (splats.render_backward(scratch, cam, (w, h), hot)[1][0, 0] != 0.0)
    assert seen.any() == covered and not seen.all()

    dl = rng.normal(size=(h, w, 4)).astype(np.float32)
    dl[y, x] = 0.0
    ref_attr, ref_sh = oracle_mod.render64_backward(oracle_mod.look_at(POS, TGT), w, h, attr.astype(np.float64),
                                                    sh.astype(np.float64), k, dl.astype(np.float64))
    dl[y, x, channel] = bad
    splats.render_forward(scratch, cam, (w, h))
    d_attr, d_sh = splats.render_backward(scratch, cam, (w, h), dl)[:2]
    ref_attr, ref_sh = ref_attr.reshape(11, n), ref_sh.reshape(k, 3, n)
    assert np.isfinite(d_attr[:, ~seen]).all() and np.isfinite(d_sh[..., ~seen]).all()
    assert rel_l2(d_sh[..., ~seen], ref_sh[..., ~seen]) < 5e-3
    for sl in (slice(0, 3), slice(3, 7), slice(7, 10), slice(10, 11)):
        assert rel_l2(d_attr[sl][:, ~seen], ref_attr[sl][:, ~seen]) < 5e-3
    if covered and channel < 3:
        assert not np.isfinite(d_sh[:, channel, seen]).any()
