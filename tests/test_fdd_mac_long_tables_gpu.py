"""The FP32 table MAC where the table is long for the DMs and segments it serves:
warps that only build entries and stage channels, and both sides of the rule
that leaves such shapes to the tiled kernel. Against the FP64 oracle, tolerances
as for the FP32 plans."""
import numpy as np
import pytest

from oracle import pyoracle as po
from tests.test_fdd_gpu import FP32_MAX_ABS, FP32_REL_L2, _delays, _errs, _input, _oracle_x, _plan

pytestmark = pytest.mark.gpu

NFFT = 16384


@pytest.mark.parametrize("delay,nseg,ndm,nchans", [
    (9000, 1, 1, 32), (9000, 1, 33, 64), (9000, 4, 20, 160), (5000, 2, 64, 96), (5000, 4, 100, 32),
    (5000, 7, 64, 224), (5000, 7, 64, 64), (12000, 9, 30, 128), (12000, 13, 64, 224), (12000, 3, 5, 32)])
def test_long_tables(delay, nseg, ndm, nchans):
    _, params = _input(nchans, NFFT, 1)
    top = 10.0
    for _ in range(60):  # the DM whose largest delay is `delay`
        p = _plan(params, np.array([top], np.float32), segmented=1, segment_nfft=NFFT)
        if p.get_max_delay() >= delay:
            break
        top *= min(1.5, max(1.0001, delay / max(1, p.get_max_delay())))
    dms = np.linspace(0, top, ndm).astype(np.float32) if ndm > 1 else np.array([top], np.float32)
    p = _plan(params, dms, segmented=1, segment_nfft=NFFT)
    md = p.get_max_delay()
    assert delay <= md < delay * 1.01
    nsamps = max(nseg * (NFFT - md) - 37, md + 1000)
    inp, params = _input(nchans, nsamps, 5 + nseg)
    nout = nsamps - md
    out = np.zeros((ndm, nout), np.float32)
    p.execute(nsamps, inp, 8, out, 32)
    x = _oracle_x(inp, nsamps, params, 8)
    ref = po.fdd_timeseries(x, _delays(params), np.ones(nchans, np.int32), dms, nout)
    rel, mx = _errs(out, ref)
    assert rel < FP32_REL_L2 and mx < FP32_MAX_ABS, (rel, mx)
