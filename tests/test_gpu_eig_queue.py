"""The EIG's per-warp queues (GPU): splat counts around a warp's group and a
block, weights from none to all, against the CPU oracle's sums."""
import numpy as np
import pytest

import splatfield_b200 as sf
from splatfield_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 129, 256, 1025, 40_000, 400_003])
@pytest.mark.parametrize("share", [0.0, 0.05, 0.5, 1.0])
def test_eig_sums_the_weighted_splats(ctx, oracle_mod, n, share):
    """LUT terms are the oracle's f32 values and FP64 terms agree to about
    1e-12 nats; both are added in f64, so n terms of at most a few nats differ
    by the order of the sum and by their own error: below 1e-9 relative plus
    n * 1e-11."""
    rng = np.random.default_rng(n)
    a, b = synth.beta_posterior(n, seed=n)
    words = (rng.integers(1, 1 << 24, n) * (rng.random(n) < share)).astype(np.uint32)
    acc = sf.Accumulators(n)
    acc.write_bits(words)
    acc.set_scale(float(1 << 20))
    beta = sf.BetaState.from_host(a, b)
    for mode in (sf.EIG_LUT_F32, sf.EIG_FP64):
        want = oracle_mod.eig(a, b, words, acc.scale, mode)
        got = beta.eig(acc, mode)
        assert abs(got - want) <= 1e-9 * abs(want) + 1e-11 * n
        real = sf.DeviceBuffer.from_array((words / np.float32(acc.scale)).astype(np.float32))
        got_real = beta.eig_real(real, None, mode)
        assert abs(got_real - want) <= 1e-9 * abs(want) + 1e-11 * n
