"""Expiry of the shared-sum kernel's bounded waits, in a plan and in a batch: with
the expiry test on and a limit of 1 ms its building warps wait on a barrier that
nothing arrives on, the staging and summing warps run into the limit behind them,
and the call reports DEDISP_INTERNAL_GPU_ERROR. The same plan and batch then give
exact results: registers, tensor memory and barriers were given back."""
import numpy as np
import pytest

import dedisp_tests_b200 as dd
from tests.test_tdd_forms_gpu import PARAMS, fine_list, make_batch, oracle, same, series
from tests.test_wait_expiry_gpu import INTERNAL, _Expiry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbits,nfine,coarse,nout", [
    (2, 320, None, 2500), (8, 320, 2.0, 2500), (8, 320, 2.0, 9000), (8, 640, 2.0, 40000), (16, 320, 2.0, 2500)])
def test_plan_expiry_then_recovers(nbits, nfine, coarse, nout):
    dms = fine_list(nfine, coarse)
    p = dd.TDDPlan(*PARAMS)
    p.set_dm_list(dms)
    packed = series(nbits, nout + p.get_max_delay(), 3)
    out = np.zeros((len(dms), nout), np.float32)
    for _ in range(64):
        p.execute(packed.shape[0], packed, nbits, out, 32)
        if p.get_form()[0] == "shared":
            break
    with _Expiry():
        with pytest.raises(dd.DedispError) as ei:
            p.execute(packed.shape[0], packed, nbits, out, 32)
    assert ei.value.detail == INTERNAL, ei.value
    assert p.get_form()[0] == "shared"
    out[:] = 0
    p.execute(packed.shape[0], packed, nbits, out, 32)
    assert p.get_form()[0] == "shared"
    assert same(out, oracle(packed, nbits, dms, nout))


@pytest.mark.parametrize("nbits", [2, 8, 16])
def test_batch_expiry_then_recovers(nbits):
    lists, nouts = [fine_list(320, 2.0), fine_list(75)], (2500, 700)
    b, ins, outs, _ = make_batch(nbits, lists, nouts)
    with _Expiry():
        b.execute(0, use_graph=False)
        with pytest.raises(dd.DedispError) as ei:
            b.sync(0)
    assert ei.value.code == INTERNAL, ei.value
    assert b.get_form()[0] == "shared"
    b.execute(0, use_graph=False)
    b.sync(0)
    for packed, dms, nout, y in zip(ins, lists, nouts, outs):
        assert same(y.cpu().numpy(), oracle(packed, nbits, dms, nout))
    b.close()
