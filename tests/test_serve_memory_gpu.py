"""The streaming server holds its device memory from start() on, whatever the
gulps' lengths, and stays inside its budget: where the shared-sum tables of its
TDD plans would exceed it, they run row by row. Outputs equal a plan's."""
import numpy as np
import pytest

import dedisp_tests_b200 as dd
from tests.test_pattern_memory_gpu import FINE, PARAMS, free_bytes

pytestmark = pytest.mark.gpu

MAX_GULP = 6000
GULPS = (300, 6000, 1500, 2900)


def serve(budget):
    """(bytes held, device bytes taken by the gulps, outputs, rows)"""
    import torch
    s = dd.StreamServer(*PARAMS, in_nbits=8, max_gulp=MAX_GULP, tdd_workers=1, hbm_budget=budget)
    beam = s.add_beam(FINE, 0)
    held = s.start()
    rng = np.random.default_rng(4)
    rows = [rng.integers(0, 256, (n, PARAMS[0]), dtype=np.uint8) for n in GULPS]
    outs = [torch.zeros((len(FINE), n), dtype=torch.float32, device="cuda") for n in GULPS]
    before = free_bytes()
    for r, y in zip(rows, outs):
        s.submit(beam, r, r.shape[0], y)
    s.drain()
    taken = before - free_bytes()
    md = s.max_delay(beam)
    s.close()
    return held, taken, torch.cat(outs, 1), np.concatenate([np.zeros((md, PARAMS[0]), np.uint8)] + rows)


def test_gulps_allocate_nothing_and_budget_drops_the_tables():
    import torch
    held, taken, out, series = serve(0)
    assert taken == 0
    p = dd.TDDPlan(*PARAMS)
    p.set_dm_list(FINE)
    x = torch.from_numpy(series).cuda()
    want = torch.zeros_like(out)
    p.execute(series.shape[0], x, 8, want, 32, dd.DEDISP_DEVICE_POINTERS)
    p.close()
    assert torch.equal(out.view(torch.int32), want.view(torch.int32))
    # a budget just below what it took: the same results without the tables
    held2, taken2, out2, _ = serve(held - 1)
    assert held2 < held and taken2 == 0
    assert torch.equal(out2.view(torch.int32), want.view(torch.int32))
