"""A batch stays inside a caller's workspace: the scratch is checked against the
layout of every execute, so that beams or masks set later, which may change the
kernel and with it the rows' size, take a form that fits or are refused. The
bytes behind the workspace must keep their value."""
import numpy as np
import pytest

import dedisp_tests_b200 as dd
from tests.test_tdd_forms_gpu import NCH, fine_list, make_batch, oracle, same

pytestmark = pytest.mark.gpu

GUARD = 64 << 20


class Workspace:
    def __init__(self, nbytes):
        import torch
        self.n = nbytes
        self.buf = torch.full((nbytes + GUARD,), 0xA5, dtype=torch.uint8, device="cuda")

    def intact(self):
        return bool((self.buf[self.n:] == 0xA5).all())


def check(b, ins, outs, lists, nbits, km=None):
    b.execute(0, use_graph=False)
    b.sync(0)
    for packed, dms, y in zip(ins, lists, outs):
        assert same(y.cpu().numpy(), oracle(packed, nbits, dms, y.shape[1], km))


@pytest.mark.parametrize("nbits", [8, 16])
def test_beams_set_after_the_workspace(nbits):
    """Sized for beams that run row by row; then a list that the shared sums
    would take in rows of twice the size (16 bits), with and without room."""
    fine = fine_list(320, 5.0)
    coarse = np.array([0.0, fine[-1]], np.float32)
    b, ins, outs, beams = make_batch(nbits, [coarse], [2500])
    ws = Workspace(b.workspace_size())
    b.set_workspace(ws.buf, ws.n)
    check(b, ins, outs, [coarse], nbits)
    assert b.get_form()[0] == "rows" and ws.intact()
    b2, ins2, outs2, beams2 = make_batch(nbits, [fine], [2500])
    b.set_beams(beams2)
    check(b, ins2, outs2, [fine], nbits)
    assert ws.intact()
    if b.workspace_size() > ws.n:
        assert b.get_form()[0] == "rows"
    assert nbits == 8 or b.workspace_size() > ws.n
    big = Workspace(b.workspace_size())
    b.set_workspace(big.buf, big.n)
    check(b, ins2, outs2, [fine], nbits)
    assert b.get_form()[0] == "shared" and big.intact() and ws.intact()
    # fewer channels change the decision too: still inside
    km = np.ones(NCH, np.int32)
    km[1:] = 0
    b.set_killmask(km)
    check(b, ins2, outs2, [fine], nbits, km)
    assert big.intact()


def test_longer_beams_are_refused():
    dms = fine_list(64)
    b, ins, outs, _ = make_batch(8, [dms], [700])
    ws = Workspace(b.workspace_size())
    b.set_workspace(ws.buf, ws.n)
    check(b, ins, outs, [dms], 8)
    b2, ins2, outs2, beams2 = make_batch(8, [dms], [30000])
    b.set_beams(beams2)
    with pytest.raises(dd.DedispError) as ei:
        b.execute(0, use_graph=False)
    assert ei.value.code == dd.ERROR_NAMES.index("DEDISP_MEM_ALLOC_FAILED")
    assert ws.intact()
    with pytest.raises(dd.DedispError):
        b.set_workspace(ws.buf, ws.n)
    b.set_workspace(None, 0)
    check(b, ins2, outs2, [dms], 8)
    assert ws.intact()


@pytest.mark.parametrize("nbits,nout,shapes", [
    (8, 2816, [(5, 16), (5, 0)]),   # just past a 2560-sample tile: longer rows than the shared sums'
    (2, 2700, [(1, 8), (1, 0)]),
    (16, 200, [(0, 24), (0, 16), (0, 0)]),  # packed rows of 448-sample blocks
])
def test_workspace_holds_every_shape(nbits, nout, shapes):
    """The default variant has two layouts, shared sums (0 channels per stage)
    and row by row (any other count): the workspace holds both."""
    lists = [fine_list(64, step=0.4)] if nbits == 8 else [fine_list(40)]
    b, ins, outs, _ = make_batch(nbits, lists, [nout])
    ws = Workspace(b.workspace_size())
    b.set_workspace(ws.buf, ws.n)
    for shape in shapes:
        b.set_shape(*shape)
        check(b, ins, outs, lists, nbits)
        assert b.get_form()[0] == ("rows" if shape[1] else "shared"), shape
        assert ws.intact(), shape
    b.autotune()
    check(b, ins, outs, lists, nbits)
    assert ws.intact()
