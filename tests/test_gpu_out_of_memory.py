"""A call that runs out of device memory on the way returns DTK_ERR_OOM and can
be made again: the adjoint on a handle whose transpose it builds on the first
call, with each of its allocations refused in turn (dtk_set_failing_allocation,
on the host).  The repeated call gives the bits of an undisturbed one."""
import numpy as np
import pytest
import torch

import datatransferkit_gb300 as dtk
from datatransferkit_gb300 import _capi
from datatransferkit_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu
OOM = 4


@pytest.fixture
def restore():
    yield
    assert _capi.lib().dtk_set_failing_allocation(0) == 0


@pytest.mark.parametrize("coords", [False, True])
def test_adjoint_after_a_refused_allocation(coords, restore):
    L = _capi.lib()
    src = torch.from_numpy(syn.uniform_points(4000, 71)).cuda()
    tgt = torch.from_numpy(syn.uniform_points(2500, 72)).cuda()
    vals = torch.from_numpy(syn.smooth_field(src.cpu().numpy())).cuda()
    cot = torch.from_numpy(np.random.default_rng(1).standard_normal(len(tgt))).cuda()

    def operator():
        return dtk.MovingLeastSquaresOperator(None, src, tgt, dtk.Wendland(2),
                                              dtk.MultivariatePolynomialBasis(dtk.Linear, 3), k=12, keep_points=True)

    def adjoint(op):
        gv = torch.full((len(src),), np.nan, dtype=torch.float64, device="cuda")
        gc = torch.full((len(src), 3), np.nan, dtype=torch.float64, device="cuda")
        st = L.dtk_mls_apply_adjoint(op._h, cot.data_ptr(), len(tgt), vals.data_ptr(), gv.data_ptr(),
                                     gc.data_ptr() if coords else None, None)
        return st, gv, gc

    st, gv0, gc0 = adjoint(operator())
    assert st == 0
    refused = 0
    for nth in range(1, 100):
        op = operator()
        assert L.dtk_set_failing_allocation(nth) == 0
        st, gv, gc = adjoint(op)
        assert L.dtk_set_failing_allocation(0) == 0
        if st == 0:
            break
        refused += 1
        assert st == OOM
        for _ in range(2):
            st, gv, gc = adjoint(op)
            assert st == 0
            assert torch.equal(gv, gv0) and (not coords or torch.equal(gc, gc0))
    assert refused >= 6 and st == 0


def test_failing_allocation_range():
    assert _capi.lib().dtk_set_failing_allocation(-1) == 1


@pytest.mark.parametrize("what", ["fp64", "mixed", "radius", "batch", "nearest", "host"])
def test_calls_after_a_refused_allocation(what, restore):
    """Every allocation of a call refused in turn: DTK_ERR_OOM, and the same call
    made right after it gives an undisturbed one's bits."""
    L = _capi.lib()
    src = torch.from_numpy(syn.uniform_points(30000, 73)).cuda()
    tgt = torch.from_numpy(syn.uniform_points(20000, 74)).cuda()
    vals = torch.from_numpy(syn.smooth_field(src.cpu().numpy())).cuda()
    basis, rbf = dtk.MultivariatePolynomialBasis(dtk.Linear, 3), dtk.Wendland(2)
    pinned = [t.cpu().pin_memory() for t in (src, tgt, vals)]

    def call():
        out = torch.full((len(tgt),), np.nan, dtype=torch.float64, device="cuda")
        if what == "host":
            host = out.cpu().pin_memory()
            dtk.MovingLeastSquaresOperator.transfer_host(None, *pinned, host, rbf, basis, k=8)
            return host
        if what == "batch":
            op = dtk.MovingLeastSquaresBatch([dict(source_points=src, target_points=tgt, rbf=rbf, basis=basis, k=8)])
        elif what == "nearest":
            op = dtk.NearestNeighborOperator(None, src, tgt)
        else:
            rows = dict(radius=0.06) if what == "radius" else dict(k=8)
            op = dtk.MovingLeastSquaresOperator(None, src, tgt, rbf, basis,
                                                precision="mixed" if what == "mixed" else "fp64", **rows)
        op.apply(vals, out)
        return out

    want = call()
    refused = 0
    for nth in range(1, 400):
        assert L.dtk_set_failing_allocation(nth) == 0
        try:
            got = call()
        except dtk.DTKError as e:
            assert e.status == OOM
            refused += 1
            got = call()
        else:
            assert L.dtk_set_failing_allocation(0) == 0
            assert torch.equal(got, want)
            break
        assert torch.equal(got, want)
    else:
        raise AssertionError("the call never ran out of allocations to refuse")
    assert refused >= 20
