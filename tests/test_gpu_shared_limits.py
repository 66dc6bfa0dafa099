"""Shared-memory limits of kernels whose launches differ in size (GPU): calls
of one size leave the larger calls of other threads, and of the same captured
graph, alone."""
import threading

import numpy as np
import pytest
import torch

import splatfield_b200 as sf
from splatfield_b200 import synth

pytestmark = pytest.mark.gpu


def test_sorts_of_different_widths_from_several_threads(ctx):
    """From 2^20 keys on, the histogram's table follows the sorted bits."""
    n = 1 << 20
    keys = np.random.default_rng(3).integers(0, 1 << 32, n).astype(np.uint32)
    dk = sf.DeviceBuffer.from_array(keys)
    dv = sf.DeviceBuffer.from_array(np.arange(n, dtype=np.uint32))
    widths = (8, 32, 8, 32)
    errors, last = [], {}
    start = threading.Barrier(len(widths))

    def work(bits):
        try:
            stream, scratch = torch.cuda.Stream(), sf.RadixScratch(n)
            start.wait()
            for _ in range(400):
                for _ in range(4):
                    out = scratch.argsort(dk, dv, n, bits, stream=stream, sync=False)
                scratch.status(stream)
            last[bits] = (out[0].read(stream), out[1].read(stream))
        except Exception as e:  # noqa: BLE001
            errors.append((bits, e))

    threads = [threading.Thread(target=work, args=(b,)) for b in widths]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for bits, (k, v) in last.items():
        order = np.argsort(keys & np.uint32((1 << bits) - 1), kind="stable")
        np.testing.assert_array_equal(v, order.astype(np.uint32))
        np.testing.assert_array_equal(k, keys[order])


@pytest.mark.parametrize("build", [sf.ISECTS_BINNED, sf.ISECTS_DEPTH_SORTED])
def test_round_of_mixed_sizes_in_one_graph(ctx, build):
    """A large view's kernels recorded before a small one's; the depth-sorted
    round's 32-bit sort before its tile-id sort."""
    n, sizes = 1 << 20, [(720, 720), (512, 512), (64, 64)]
    attr, sh = synth.scene_clustered(n, 1, seed=5)
    splats = sf.Splats(attr, sh)
    cams = synth.sphere_cameras(len(sizes), 3.5, 4, sf.look_at)
    rnd = sf.Round(n, sizes)
    rnd.set_tuning(lanes=1, isect_build=build)
    beta = sf.BetaState.from_host(*synth.beta_posterior(n, seed=3))
    rnd.eig(splats, beta, cams)
    for v, s in enumerate(sizes):
        scratch, acc = sf.RenderScratch(n, s), sf.Accumulators(n)
        splats.render_responsibility(scratch, acc, cams[v], s)
        np.testing.assert_array_equal(rnd.responsibility(v)[0].read(), acc.bits.read())
