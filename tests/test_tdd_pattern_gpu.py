"""Time-domain plans on the shared channel-group sums: bit-exact against the CPU
oracle where the kernel can go wrong -- trial blocks of 32 and channel groups
of 8 with remainders, the 256-channel flush of the 8-bit lanes, every period
(chosen by the call's size), gulps, a thinned and an unsorted list, and DM steps
from many trials per pattern to trials taken in rounds or row by row."""
import numpy as np
import pytest

import dedisp_tests_b200 as dd
from dedisp_tests_b200 import synthetic as sy
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

FINE = (64e-6, 1300.0, -0.078125)   # dt, f0, df: wide spans per trial
COARSE = (250e-6, 1500.0, -0.5)


@pytest.mark.parametrize("nbits", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("setup,nchans,ndm,dm_lo,dm_hi,nout,gulp", [
    (COARSE, 64, 1, 40.0, 40.0, 700, 0),          # one trial, a few short tiles
    (COARSE, 32, 31, 0.0, 30.0, 2049, 0),         # trials fill most of one block
    (COARSE, 288, 33, 0.0, 60.0, 4100, 1500),     # one trial past a block, gulps
    (COARSE, 1056, 65, 0.0, 100.0, 9000, 0),      # several flushes and periods
    (COARSE, 1024, 700, 0.0, 80.0, 25000, 0),     # enough blocks for the longest period
    (FINE, 512, 64, 1000.0, 1060.0, 5000, 0),     # spans of tens of samples
    (FINE, 512, 64, 1000.0, 1400.0, 5000, 0),     # hundreds: trials in rounds
    (FINE, 512, 40, 0.0, 2000.0, 5000, 0),        # wider than a ring's half
])
def test_bit_exact(nbits, setup, nchans, ndm, dm_lo, dm_hi, nout, gulp):
    dt, f0, df = setup
    rng = np.random.default_rng(nchans + ndm + nbits)
    dms = np.linspace(dm_lo, dm_hi, ndm).astype(np.float32)
    if ndm % 2:
        dms[:-1] = rng.permutation(dms[:-1])  # the last DM sets the output length
    km = np.ones(nchans, np.int32)
    km[3::29] = 0                              # active channels: no multiple of 8
    p = dd.TDDPlan(nchans, dt, f0, df)
    p.set_dm_list(dms)
    p.set_killmask(km)
    if gulp:
        p.set_gulp_size(gulp)
    nsamps = nout + p.get_max_delay()
    top = (1 << nbits) - 1
    vals = rng.integers(0, top + 1, (nsamps, nchans)).astype(np.uint32)
    vals[nsamps // 2:, : nchans // 2] = top    # saturated lanes
    packed = sy.pack(vals, nbits)
    delays = po.delay_table(nchans, np.float32(dt), np.float32(f0), np.float32(df))
    for out_nbits, dtype in ((32, np.float32), (8, np.uint8)):
        out = np.zeros((ndm, nout), dtype)
        p.execute(nsamps, packed, nbits, out, out_nbits)
        ref = po.tdd(packed, nsamps, packed.shape[1], nbits, nchans, delays, km, dms, out_nbits, nout)
        assert np.array_equal(out.view(np.uint8), ref.view(np.uint8)), out_nbits


def test_saturated_bytes_all_channels():
    """All samples at their maximum over 513 groups: every 16-bit lane reaches
    256 x 255 before a flush, and the 32-bit sums 4104 x 255."""
    nchans, nout = 4104, 1100
    p = dd.TDDPlan(nchans, 250e-6, 1500.0, -0.02)
    dms = np.linspace(0, 30, 34).astype(np.float32)
    p.set_dm_list(dms)
    nsamps = nout + p.get_max_delay()
    packed = np.full((nsamps, nchans), 255, np.uint8)
    out = np.zeros((len(dms), nout), np.float32)
    p.execute(nsamps, packed, 8, out, 32)
    delays = po.delay_table(nchans, np.float32(250e-6), np.float32(1500.0), np.float32(-0.02))
    ref = po.tdd(packed, nsamps, nchans, 8, nchans, delays, np.ones(nchans, np.int32), dms, 32, nout)
    assert np.array_equal(out.view(np.uint32), ref.view(np.uint32))


def test_scarce_memory_takes_the_row_form():
    """16-bit strided rows are twice the packed ones: with device memory for
    1.4 times the packed rows only, a call gives what it gives with room."""
    import torch
    dt, f0, df = FINE
    nchans, nout = 4096, 4096
    dms = np.linspace(1480, 1500, 64).astype(np.float32)
    p = dd.TDDPlan(nchans, dt, f0, df)
    p.set_dm_list(dms)
    nsamps = nout + p.get_max_delay()
    x = torch.randint(0, 256, (nsamps, 2 * nchans), dtype=torch.uint8, device="cuda")
    y = [torch.zeros((len(dms), nout), dtype=torch.float32, device="cuda") for _ in range(2)]
    p.execute(nsamps, x, 16, y[0], 32, dd.DEDISP_DEVICE_POINTERS)
    p.close()
    p = dd.TDDPlan(nchans, dt, f0, df)
    p.set_dm_list(dms)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    target = int(1.4 * (nchans + 1) * nsamps * 2)
    free = torch.cuda.mem_get_info()[0]
    block = torch.empty(free - target, dtype=torch.uint8, device="cuda")
    try:
        p.execute(nsamps, x, 16, y[1], 32, dd.DEDISP_DEVICE_POINTERS)
    finally:
        del block
        torch.cuda.empty_cache()
    assert torch.equal(y[0].view(torch.int32), y[1].view(torch.int32))
