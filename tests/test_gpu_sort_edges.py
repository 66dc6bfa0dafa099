"""Radix sort at its partition edges and digit distributions (GPU), against
numpy's stable argsort."""
import numpy as np
import pytest

import splatfield_b200 as sf

pytestmark = pytest.mark.gpu

# Around the 4096- and 8192-key partitions, the wide histogram's start (2^20)
# and the wide pass's (2^21).
SIZES = [2, 31, 33, 4095, 4096, 4097, 12289, (1 << 20) - 1, 1 << 20, (1 << 21) - 1, (1 << 21) + 8191]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("dist", ["random", "equal", "runs", "two"])
@pytest.mark.parametrize("digit_bits,bits", [(8, 32), (8, 13), (4, 32), (5, 31), (7, 20)])
def test_argsort_matches_numpy(ctx, n, dist, digit_bits, bits):
    if n > 100_000 and (digit_bits, bits) not in ((8, 32), (8, 13), (4, 32)):
        pytest.skip("covered at the smaller sizes")
    rng = np.random.default_rng(n)
    keys = {"random": lambda: rng.integers(0, 1 << 32, n), "equal": lambda: np.full(n, 0xA5A5A5A5),
            "runs": lambda: np.sort(rng.integers(0, 1 << 12, n)), "two": lambda: rng.integers(0, 2, n) * 0xFFFFFFFF}
    keys = keys[dist]().astype(np.uint32)
    vals = rng.integers(0, 1 << 32, n).astype(np.uint32)
    scratch = sf.RadixScratch(n)
    scratch.set_digit_bits(digit_bits)
    k, v = scratch.argsort(sf.DeviceBuffer.from_array(keys), sf.DeviceBuffer.from_array(vals), n, bits)
    order = np.argsort(keys & np.uint32((1 << bits) - 1), kind="stable")
    np.testing.assert_array_equal(k.read(), keys[order])
    np.testing.assert_array_equal(v.read(), vals[order])
