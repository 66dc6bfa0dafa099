"""Error words of many sort and scan scratches of one context: those in its
page and those past it report their own timeouts only, and slots are reused
clean."""
import numpy as np
import pytest

import splatfield_b200 as sf
from splatfield_b200._lib import SF_ERR_TIMEOUT, SF_OK, lib

pytestmark = pytest.mark.gpu

N = 20_011  # five scan partitions


def test_each_scratch_reports_its_own_timeout(ctx):
    counts = np.random.default_rng(7).integers(0, 50, N).astype(np.uint32)
    want = (np.cumsum(counts.astype(np.uint64)) - counts).astype(np.uint32)
    dc, out = sf.DeviceBuffer.from_array(counts), sf.DeviceBuffer.empty(N)
    scans = [sf.ScanScratch(N) for _ in range(70)]  # a page has 64 words
    bad = (0, 63, 64, 69)
    assert lib().sf_debug_lookback(16, 1) == SF_OK
    try:
        for i in bad:
            sf.exclusive_scan_gather(None, dc, out, N, scans[i], sync=False)
        sf.DeviceBuffer.from_array(counts).read()
    finally:
        assert lib().sf_debug_lookback(0, 0) == SF_OK
    for i, s in enumerate(scans):
        if i in bad:
            with pytest.raises(sf.SplatfieldError) as e:
                s.status()
            assert e.value.code == SF_ERR_TIMEOUT
        s.status()
    for i in bad:
        scans[i].close()
        scans[i] = sf.ScanScratch(N)
    for s in scans:
        sf.exclusive_scan_gather(None, dc, out, N, s)
    np.testing.assert_array_equal(out.read(), want)
