"""Every radix and pass order of the N = 16384 Q transforms, forward and
inverse, through whole-series time-series plans against the FP64 oracle.

Q <= 16 is one pass in registers; 18 and 144 are two; 270 is three; 17 is a
direct sum of staged elements, 34 a direct sum after a register pass, 289 two
direct sums, 306 both with a buffer swap between them. Odd trial lengths put
every second output row on an odd float.

Tolerance: the FP32 transforms lose about log2(N) / 2 roundings of 2^-24 in
the relative L2 norm each way (12 x 6e-8 = 7e-7 at N = 2^23 for both), the
direct sums of 17 terms sqrt(17) more of one pass: 2e-6 relative L2 and 2e-5
of the largest value, as for the other lengths.
"""
import numpy as np
import pytest

from oracle import pyoracle as po
from tests.test_fdd_gpu import _delays, _errs, _input, _oracle_x, _plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q", [6, 7, 9, 10, 11, 12, 14, 15, 17, 18, 34, 144, 270, 289, 306])
def test_time_series_every_radix(q):
    nchans = 8
    nsamps = 16384 * q - 700 - q % 2
    inp, params = _input(nchans, nsamps, 300 + q)
    dms = np.linspace(0, 40, 3, dtype=np.float32)
    p = _plan(params, dms, segmented=0, timeseries=True, precision=0)
    nout = nsamps - p.get_max_delay()
    nout -= 1 - nout % 2
    out = np.zeros((len(dms), nsamps - p.get_max_delay()), np.float32)
    p.execute(nsamps, inp, 8, out, 32)
    x = _oracle_x(inp, nsamps, params, 8)
    ref = po.fdd_timeseries(x, _delays(params), np.ones(nchans, np.int32), dms, nout)
    rel, mx = _errs(out[:, :nout], ref)
    print(f"Q = {q}: rel-L2 {rel:.3e} max-abs {mx:.3e}")
    assert rel < 2e-6 and mx < 2e-5, (q, rel, mx)
