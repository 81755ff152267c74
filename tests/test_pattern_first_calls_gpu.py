"""When a plan builds the shared-sum tables: at once for a call that earns them, at
the second one on the same list, mask, range and width for a small one, never
while ranges alternate in small calls; and a captured graph of a small call
stays valid when the plan's later calls take the tables. Outputs are exact in
every form."""
import numpy as np
import pytest

import dedisp_tests_b200 as dd
from tests.test_tdd_forms_gpu import NCH, PARAMS, fine_list, oracle, same, series

pytestmark = pytest.mark.gpu


def plan(dms):
    p = dd.TDDPlan(*PARAMS)
    p.set_dm_list(dms)
    return p


@pytest.mark.parametrize("nbits,nout,forms", [
    (8, 3000, ["rows", "shared", "shared"]),
    (16, 3000, ["rows", "shared", "shared"]),
    (2, 30000, ["shared", "shared"]),
])
def test_calls_on_one_list(nbits, nout, forms):
    dms = fine_list(320)
    p = plan(dms)
    packed = series(nbits, nout + p.get_max_delay(), 21)
    want = oracle(packed, nbits, dms, nout)
    for form in forms:
        out = np.zeros((len(dms), nout), np.float32)
        p.execute(packed.shape[0], packed, nbits, out, 32)
        assert p.get_form()[0] == form
        assert same(out, want)


def test_alternating_ranges_and_widths():
    dms, nout, n = fine_list(320), 3000, 96
    p = plan(dms)
    inputs = {nb: series(nb, nout + p.get_max_delay(), nb) for nb in (4, 8)}
    for first, nb in ((0, 8), (96, 8), (0, 4), (33, 8), (0, 8)):
        packed = inputs[nb]
        out = np.zeros((n, nout), np.float32)
        p.execute_guru(packed.shape[0], packed, nb, packed.shape[1], out, 32, nout * 4, first, n)
        assert p.get_form()[0] == "rows"
        assert same(out, oracle(packed, nb, dms[first:first + n], nout))


@pytest.mark.parametrize("warm", [1, 3])
def test_captured_call_outlives_the_change_of_form(warm):
    import torch
    dms, nout = fine_list(320), 2100   # rows of both forms differ in length
    p = plan(dms)
    packed = series(8, nout + p.get_max_delay(), 5)
    want = oracle(packed, 8, dms, nout)
    x = torch.from_numpy(packed).cuda()
    y = torch.zeros((len(dms), nout), dtype=torch.float32, device="cuda")
    z = torch.zeros_like(y)
    s = torch.cuda.Stream()
    p.set_stream(s.cuda_stream)
    flags = dd.DEDISP_DEVICE_POINTERS | dd.DEDISP_ASYNC

    def run(out):
        p.execute(packed.shape[0], x, 8, out, 32, flags)

    torch.cuda.synchronize()
    for _ in range(warm):
        run(y)
    s.synchronize()
    captured = p.get_form()[0]
    assert captured == ("rows" if warm == 1 else "shared")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s, capture_error_mode="thread_local"):
        run(y)
    assert p.get_form()[0] == captured
    for _ in range(2):
        run(z)
    s.synchronize()
    assert p.get_form()[0] == "shared"
    assert same(z.cpu().numpy(), want)
    y.zero_()
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    assert same(y.cpu().numpy(), want)
    del g
    p.set_stream(0)


def test_more_plans_than_status_words():
    """Plans take a status word each from one page of 1024; those past it, and
    those that take a word given back, give the same results."""
    dms, nout = fine_list(8), 300
    packed = series(8, nout + plan(dms).get_max_delay(), 9)
    want = oracle(packed, 8, dms, nout)

    def run(p):
        out = np.zeros((len(dms), nout), np.float32)
        p.execute(packed.shape[0], packed, 8, out, 32)
        assert same(out, want)

    plans = [plan(dms) for _ in range(1030)]
    for p in plans:
        run(p)
    for p in plans[1000:]:
        run(p)
    for p in plans[:20]:
        p.close()
    run(plan(dms))
    for p in plans[20:]:
        p.close()
