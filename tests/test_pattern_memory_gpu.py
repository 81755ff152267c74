"""Device memory of the shared-sum tables: given back when the lists take another
kernel, and held tables count as room when they are built again."""
import numpy as np
import pytest

import dedisp_tests_b200 as dd

pytestmark = pytest.mark.gpu

PARAMS = (4096, 64e-6, 1500.0, -0.078125)
FINE = np.linspace(0, 150, 3000).astype(np.float32)      # tables of tens of MB
COARSE = np.linspace(0, 150, 12).astype(np.float32)
NOUT = 2000


def free_bytes():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def beams(*lists):
    import torch
    q = dd.TDDPlan(*PARAMS)
    res = []
    for dms in lists:
        q.set_dm_list(dms)
        n = NOUT + q.get_max_delay()
        x = torch.zeros((n, PARAMS[0]), dtype=torch.uint8, device="cuda")
        y = torch.zeros((len(dms), NOUT), dtype=torch.float32, device="cuda")
        res.append((x, PARAMS[0], n, dms, y, NOUT * 4))
    return res


def test_batch_gives_tables_back():
    fine, coarse = beams(FINE, COARSE)
    b = dd.Batch(*PARAMS)
    b.set_beams([coarse])
    b.execute(0, use_graph=False)
    b.sync(0)
    assert b.get_form()[0] == "rows"
    before = free_bytes()
    b.set_beams([fine])
    held = before - free_bytes()
    assert held > 8 << 20
    b.set_beams([coarse])
    assert before - free_bytes() < held // 2
    b.set_beams([fine, coarse])     # one beam declines for all: nothing is kept
    b.execute(0, use_graph=False)
    b.sync(0)
    assert b.get_form()[0] == "rows"


def test_batch_counts_held_tables_as_room():
    import torch
    fine, = beams(FINE)
    b = dd.Batch(*PARAMS)
    before = free_bytes()
    b.set_beams([fine])
    tables = before - free_bytes()
    b.execute(0, use_graph=False)
    b.sync(0)
    assert b.get_form()[0] == "shared"
    torch.cuda.empty_cache()
    # less than four times the tables free, but more than three times
    block = torch.empty(free_bytes() - int(3.3 * tables), dtype=torch.uint8, device="cuda")
    try:
        b.set_beams([fine])
        b.execute(0, use_graph=False)
        b.sync(0)
        assert b.get_form()[0] == "shared"
    finally:
        del block
        torch.cuda.empty_cache()


def test_plan_gives_tables_back():
    fine, coarse = beams(FINE, COARSE)
    p = dd.TDDPlan(*PARAMS)

    def run(beam, tries=1):
        p.set_dm_list(beam[3])
        for _ in range(tries):
            p.execute(beam[2], beam[0], 8, beam[4], 32, dd.DEDISP_DEVICE_POINTERS)
            if p.get_form()[0] == "shared":
                break
        return p.get_form()[0]

    p.set_tile_variant(6)             # a row-by-row variant: the buffers, no tables
    assert run(fine) == "rows"
    before = free_bytes()
    p.set_tile_variant(5)             # the default one
    assert run(fine, 64) == "shared"
    held = before - free_bytes()
    assert held > 8 << 20
    assert run(coarse, 2) == "rows"   # this list takes no tables (known at its second call)
    assert before - free_bytes() < held // 2
    assert run(fine, 64) == "shared"
    p.set_tile_variant(6)             # nor does this variant
    assert run(fine) == "rows"
    assert before - free_bytes() < held // 2
