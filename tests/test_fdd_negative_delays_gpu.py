"""FP32 Fourier-domain plans whose channel delays are negative (a band below zero
frequency, which plans accept): their phasors come from the twiddle tables, the
per-bin table holds delays from 0 on and is read without a check of the index.
Spectra against the FP64 oracle, tolerances as for the FP32 plans."""
import numpy as np
import pytest

from oracle import pyoracle as po
from tests.test_fdd_gpu import FP32_MAX_ABS, FP32_REL_L2, _delays, _errs, _input, _oracle_x, _plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsamps", [4000, 16384 * 3 - 200])
def test_band_below_zero(nsamps):
    nchans = 64
    inp, _ = _input(nchans, nsamps, 7)
    params = (nchans, 250e-6, -1581.8, -1.5625)
    delays = _delays(params)
    assert delays[1] < 0 and np.all(np.diff(delays) < 0)
    dms = np.linspace(0, 200, 40, dtype=np.float32)
    p = _plan(params, dms, segmented=0, precision=0)
    assert p.get_max_delay() == 0
    out = np.zeros((len(dms), p.output_row_length(nsamps)), np.float32)
    p.execute(nsamps, inp, 8, out, 32)
    x = _oracle_x(inp, nsamps, params, 8)
    ref = po.fdd_spectrum(x, delays, np.ones(nchans, np.int32), dms, out.shape[1])
    rel, mx = _errs(out, ref)
    assert rel < FP32_REL_L2 and mx < FP32_MAX_ABS, (rel, mx)
    # segments: every delay wraps inside its segment; it has to run, not match
    p = _plan(params, dms, segmented=1, segment_nfft=1024, precision=0)
    out = np.zeros((len(dms), nsamps), np.float32)
    p.execute(nsamps, inp, 8, out, 32)
    assert np.isfinite(out).all() and np.abs(out).max() > 0
