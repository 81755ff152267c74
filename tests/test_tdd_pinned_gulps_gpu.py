"""Calls from pinned host buffers: gulps where the copies and kernels of neighbouring
gulps overlap, one gulp where the input copy binds and each gulp would copy its
overlap rows again (few trials, long delays). Outputs equal the device-buffer
call's, bit for bit, in every kernel form."""
import numpy as np
import pytest

import dedisp_tests_b200 as dd

pytestmark = pytest.mark.gpu

PARAMS = (1024, 250e-6, 1581.8, -0.390625)


@pytest.mark.parametrize("nbits,ndm,dm_max,nout,mask,several", [
    (8, 8, 400.0, 50000, 1, False),
    (8, 512, 400.0, 50000, 1, True),
    (8, 511, 100.0, 50001, 1, True),
    (2, 512, 400.0, 70001, 1, True),
    (16, 512, 200.0, 30000, 1, True),
    (32, 128, 100.0, 30000, 1, True),
    (8, 128, 100.0, 30000, 3, True),    # a general mask: the plain kernel
])
def test_gulps(nbits, ndm, dm_max, nout, mask, several):
    import torch
    dms = np.linspace(0, dm_max, ndm).astype(np.float32)
    if ndm % 2:
        dms[:-1] = np.random.default_rng(1).permutation(dms[:-1])
    p = dd.TDDPlan(*PARAMS)
    p.set_dm_list(dms)
    p.set_killmask(np.full(PARAMS[0], mask, np.int32))
    n = nout + p.get_max_delay()
    x = torch.randint(0, 256, (n, PARAMS[0] * nbits // 8), dtype=torch.uint8).pin_memory()
    y = torch.zeros((ndm, nout), dtype=torch.float32).pin_memory()
    want = torch.zeros((ndm, nout), dtype=torch.float32, device="cuda")
    p.execute(n, x.cuda(), nbits, want, 32, dd.DEDISP_DEVICE_POINTERS)
    want = want.cpu()
    for _ in range(3):
        y.zero_()
        p.execute(n, x, nbits, y, 32)
        assert torch.equal(y.view(torch.int32), want.view(torch.int32))
        # a row build and a kernel per gulp, the last one's by groups of trials
        assert (p.get_timing()["launches"] > 4) == several
