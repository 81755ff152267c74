"""The FP32 MAC on a per-bin phasor table against the FP64 oracle: every width
of a segment tile (1 to 10) and the first two past it, DM counts at the edges of
a thread's and a block's share, channels at the edge of a staged chunk, both
delay roundings, and a table larger than the phasors it serves. Tolerances as
for the FP32 plans (tests/test_fdd_gpu.py)."""
import numpy as np
import pytest

import dedisp_tests_b200 as dd
from oracle import pyoracle as po
from tests.test_fdd_gpu import FP32_MAX_ABS, FP32_REL_L2, _delays, _errs, _input, _oracle_x, _plan

pytestmark = pytest.mark.gpu

NFFT = 4096


@pytest.mark.parametrize("nseg,ndm,nchans,dm_max,rounding", [
    (1, 1, 32, 60.0, False), (1, 33, 128, 60.0, True), (1, 1025, 64, 60.0, False), (2, 130, 129, 60.0, True),
    (3, 63, 32, 60.0, False), (4, 64, 32, 60.0, False), (5, 127, 160, 60.0, False), (6, 128, 32, 60.0, True),
    (7, 7, 32, 60.0, False), (8, 257, 32, 60.0, False), (9, 129, 32, 60.0, False), (10, 520, 32, 60.0, False),
    (11, 66, 32, 60.0, False), (23, 20, 32, 60.0, False), (12, 3, 32, 600.0, False)])
def test_segments_and_trials(nseg, ndm, nchans, dm_max, rounding):
    dms = np.linspace(0, dm_max, ndm).astype(np.float32) if ndm > 1 else np.array([dm_max], np.float32)
    probe_in, params = _input(nchans, 16, 1)
    p = _plan(params, dms, segmented=1, segment_nfft=NFFT, round_delays=rounding)
    md = p.get_max_delay()
    nsamps = nseg * (NFFT - md) - 37  # the last segment is not full
    inp, params = _input(nchans, nsamps, 17 + nseg)
    nout = nsamps - md
    out = np.zeros((ndm, nout), np.float32)
    p.execute(nsamps, inp, 8, out, 32)
    x = _oracle_x(inp, nsamps, params, 8)
    ref = po.fdd_timeseries(x, _delays(params), np.ones(nchans, np.int32), dms, nout, round_delays=int(rounding))
    rel, mx = _errs(out, ref)
    assert rel < FP32_REL_L2 and mx < FP32_MAX_ABS, (rel, mx)


def test_longest_series():
    """N = 16384 x 394, the longest whole series that FP32 plans take (8
    channels, delays of a few samples; 200 KB of phasor tables). Tolerance as
    above: the MAC sums 8 products, the transforms lose log2(N) / 2 roundings
    each way and the direct sums of 197 terms sqrt(197) of one pass, about
    1.5e-6 relative L2."""
    nchans, q = 8, 394
    nsamps = 16384 * q - 700
    inp, params = _input(nchans, nsamps, 91)
    dms = np.linspace(0, 40, 3, dtype=np.float32)
    p = _plan(params, dms, segmented=0, timeseries=True, precision=0)
    nout = nsamps - p.get_max_delay()
    out = np.zeros((len(dms), nout), np.float32)
    p.execute(nsamps, inp, 8, out, 32)
    x = _oracle_x(inp, nsamps, params, 8)
    ref = po.fdd_timeseries(x, _delays(params), np.ones(nchans, np.int32), dms, nout)
    rel, mx = _errs(out, ref)
    print(f"rel-L2 {rel:.3e} max-abs {mx:.3e}")
    assert rel < FP32_REL_L2 and mx < FP32_MAX_ABS, (rel, mx)
