"""Which time-domain kernel ran, and that its output is exact: DM lists that the
shared channel-group sums take at every width, period (4, 8 and 16 words per
lane) and number of rounds (1, 2 and 4; a group whose trials would need 8 does
not fit the row ring), in plans and in batches, and calls that other forms take.

The lists are fine steps (few delay patterns per block of 32 trials) followed by
one block of coarse ones, whose low-frequency groups take their trials in
rounds; the period follows from the number of tiles."""
import numpy as np
import pytest

import dedisp_tests_b200 as dd
from dedisp_tests_b200 import synthetic as sy
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

PARAMS = (256, 250e-6, 1500.0, -1.0)
NCH = PARAMS[0]


def fine_list(n, coarse=None, step=0.02):
    d = np.arange(n) * step
    if coarse:
        d = np.concatenate([d, d[-1] + np.arange(1, 33) * coarse])
    return d.astype(np.float32)


def series(nbits, nsamps, seed):
    rng = np.random.default_rng(seed)
    vals = rng.integers(0, 1 << nbits, (nsamps, NCH)).astype(np.uint32)
    vals[nsamps // 2:, : NCH // 3] = (1 << nbits) - 1
    return sy.pack(vals, nbits)


def oracle(packed, nbits, dms, nout, km=None):
    delays = po.delay_table(NCH, *[np.float32(x) for x in PARAMS[1:]])
    km = np.ones(NCH, np.int32) if km is None else km
    return po.tdd(packed, packed.shape[0], packed.shape[1], nbits, NCH, delays, km, dms, 32, nout)


def same(a, b):
    return np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("nbits,nfine,coarse,nout,form", [
    (1, 320, None, 2500, ("shared", 4, 1)),
    (2, 320, 10.0, 9000, ("shared", 8, 4)),
    (4, 672, 5.0, 9000, ("shared", 16, 4)),
    (8, 320, 10.0, 2500, ("shared", 4, 4)),
    (8, 320, 2.0, 9000, ("shared", 8, 2)),
    (8, 640, 2.0, 40000, ("shared", 16, 4)),
    (16, 320, 2.0, 2500, ("shared", 4, 2)),
    (16, 672, 5.0, 9000, ("shared", 8, 4)),
    (16, 640, 2.0, 20000, ("shared", 16, 4)),
    (8, 64, 10.0, 3000, ("rows", 0, 0)),      # too many patterns
    (32, 64, None, 1000, ("rows", 0, 0)),     # no shared sums at this width
])
def test_plan_form(nbits, nfine, coarse, nout, form):
    dms = fine_list(nfine, coarse)
    p = dd.TDDPlan(*PARAMS)
    p.set_dm_list(dms)
    packed = series(nbits, nout + p.get_max_delay(), nbits + nfine)
    want = oracle(packed, nbits, dms, nout)
    assert p.get_form() == (None, 0, 0)
    for _ in range(64):
        out = np.zeros((len(dms), nout), np.float32)
        p.execute(packed.shape[0], packed, nbits, out, 32)
        assert same(out, want)
        if p.get_form() == form:
            break
    assert p.get_form() == form


def test_plain_form():
    dms = fine_list(40)
    p = dd.TDDPlan(*PARAMS)
    p.set_dm_list(dms)
    p.set_killmask(np.full(NCH, 2, np.int32))
    packed = series(8, 900 + p.get_max_delay(), 1)
    out = np.zeros((len(dms), 900), np.float32)
    p.execute(packed.shape[0], packed, 8, out, 32)
    assert p.get_form() == ("plain", 0, 0)
    assert same(out, oracle(packed, 8, dms, 900, np.full(NCH, 2, np.int32)))


def make_batch(nbits, lists, nouts, seed=1, extra=0):
    """A batch of one beam per list on device buffers: (batch, packed inputs,
    outputs, beam tuples); `extra` more floats per output row."""
    import torch
    b = dd.Batch(*PARAMS, in_nbits=nbits, out_nbits=32)
    q = dd.TDDPlan(*PARAMS)
    ins, outs, beams = [], [], []
    for i, (dms, nout) in enumerate(zip(lists, nouts)):
        q.set_dm_list(dms)
        packed = series(nbits, nout + q.get_max_delay(), seed + i)
        x = torch.from_numpy(packed).cuda()
        y = torch.full((len(dms), nout + extra), -7.0, dtype=torch.float32, device="cuda")
        ins.append(packed)
        outs.append(y)
        beams.append((x, packed.shape[1], packed.shape[0], dms, y, y.shape[1] * 4))
    b.set_beams(beams)
    return b, ins, outs, beams


@pytest.mark.parametrize("nbits,nouts,lane_words", [
    (1, (2500, 700), 4), (2, (5000, 12000), 8), (4, (14000, 30000), 16),
    (8, (2500, 700), 4), (8, (5000, 12000), 8), (8, (14000, 30000), 16),
    (16, (2500, 700), 4), (16, (9000, 30000), 8), (16, (14000, 30000), 16),
])
def test_batch_form(nbits, nouts, lane_words):
    """Beams of ragged sizes on the persistent shared-sum kernel, direct and as
    a graph; nothing is written past a row."""
    lists = [fine_list(320, 5.0), fine_list(75)]
    b, ins, outs, _ = make_batch(nbits, lists, nouts, extra=3)
    for graph in (False, True, True):
        for y in outs:
            y.fill_(-7.0)
        b.execute(0, use_graph=graph)
        b.sync(0)
        name, words, rounds = b.get_form()
        assert (name, words) == ("shared", lane_words) and rounds > 1
        for packed, dms, nout, y in zip(ins, lists, nouts, outs):
            a = y.cpu().numpy()
            assert same(np.ascontiguousarray(a[:, :nout]), oracle(packed, nbits, dms, nout))
            assert np.all(a[:, nout:] == -7.0)
    b.close()


def test_delays_past_the_tables_sums():
    """Delays of 2^25 samples and more: the tables' sizes would pass 32 bits, so
    such lists run row by row (or plain) without asking for them."""
    import torch
    nch, nout = 32, 300
    params = (nch, 1e-6, 400.0, -1.0)
    p = dd.TDDPlan(*params)
    p.set_dm_list(np.array([1000.0], np.float32))
    dm = 1000.0 * 2.0 ** 25.1 / p.get_max_delay()
    dms = np.linspace(dm * (1 - 1e-6), dm, 40).astype(np.float32)
    p.set_dm_list(dms)
    md = p.get_max_delay()
    assert md > 1 << 25
    n = nout + md
    x = torch.randint(0, 2, (n, nch), dtype=torch.uint8, device="cuda")
    words = (x.to(torch.int32) << torch.arange(nch, device="cuda", dtype=torch.int32)).sum(1, dtype=torch.int64)
    packed = (words & 0xFFFFFFFF).to(torch.uint32).view(torch.uint8)
    out = torch.zeros((len(dms), nout), dtype=torch.float32, device="cuda")
    for _ in range(2):
        p.execute(n, packed, 1, out, 32, dd.DEDISP_DEVICE_POINTERS)
        assert p.get_form()[0] in ("rows", "plain")
    delays = po.delay_table(nch, *[np.float32(v) for v in params[1:]])
    got = out.cpu().numpy()
    xs = x.cpu().numpy()
    scale = np.float32(3.0 * 1024.0 / 255.0 / 16.0)
    for i in (0, 17, 39):
        d = np.rint((dms[i] * delays[:nch]).astype(np.float32)).astype(np.int64)
        want = sum(xs[k:k + nout, c].astype(np.float32) for c, k in enumerate(d))
        want = (want / np.float32(nch)).astype(np.float32) * scale
        assert np.array_equal(got[i], want), i


def test_batch_set_again_while_it_runs():
    """New beams and a new mask right behind an execute on a stream of its own:
    the lists and tables that its kernels still read are written after it."""
    import torch
    s = torch.cuda.Stream()
    lists, nouts = [fine_list(640, 5.0), fine_list(320)], (40000, 30000)
    b, ins, outs, beams = make_batch(8, lists, nouts, seed=3)
    other, nout2 = [fine_list(96, step=0.05)], 5000
    b2, ins2, outs2, beams2 = make_batch(8, other, [nout2], seed=9)
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        for graph in (False, True):
            for y in outs + outs2:
                y.zero_()
            b.set_beams(beams)
            s.synchronize()
            b.execute(s.cuda_stream, use_graph=graph)
            first = b.get_form()[0]
            b.set_beams(beams2)
            b.execute(s.cuda_stream, use_graph=graph)
            km = np.ones(NCH, np.int32)
            km[::3] = 0
            b.set_killmask(km)
            b.set_killmask(None)
            b.sync(s.cuda_stream)
            assert first == "shared" and b.get_form()[0] == "shared"
            for packed, dms, y in zip(ins, lists, outs):
                assert same(y[:, :2000].contiguous().cpu().numpy(),
                            np.ascontiguousarray(oracle(packed, 8, dms, 2000)))
            assert same(outs2[0].cpu().numpy(), oracle(ins2[0], 8, other[0], nout2))
    b.close()
