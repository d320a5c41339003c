"""Fields of several components over the range of FP64: a mixed operator's
coefficients are FP32, its sums are not.  Row lengths with and without a kernel
of their own, one to five components, the operator and its saved copy, against
the oracle's FP64 sums of the same coefficients: 1e-14 of sum_j |c_j v_j|, for
FP64 sums of up to 32 terms."""
import numpy as np
import pytest
import torch

import datatransferkit_gb300 as dtk
from datatransferkit_gb300 import synthetic as syn
from oracle import cpu

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("k", [8, 16, 20, 32])
@pytest.mark.parametrize("scale", [1e-250, 1e-40, 1e-30, 1.0, 1e40, 1e300])
def test_components_keep_the_range_of_fp64(precision, k, scale):
    src, tgt = syn.uniform_points(3000, 61), syn.uniform_points(301, 62)
    basis = dtk.MultivariatePolynomialBasis(dtk.Linear, 3)
    op = dtk.MovingLeastSquaresOperator(None, dev(src), dev(tgt), dtk.Wendland(2), basis, k=k, precision=precision)
    off, idx, coeff = (t.cpu().numpy() for t in op.csr())
    coeff = coeff.astype(np.float64)
    for n_comp in (1, 3, 5):
        vals = scale * np.random.default_rng(n_comp).standard_normal((len(src), n_comp))
        ref = np.stack([cpu.apply(off, idx, coeff, vals[:, c]) for c in range(n_comp)], 1)
        mag = np.stack([cpu.apply(off, idx, np.abs(coeff), np.abs(vals[:, c])) for c in range(n_comp)], 1)
        for o in (op, dtk.MovingLeastSquaresOperator.from_bytes(op.to_bytes())):
            out = torch.full((len(tgt), n_comp), np.nan, dtype=torch.float64, device="cuda")
            o.apply(dev(vals), out)
            assert np.all(np.abs(out.cpu().numpy() - ref) <= 1e-14 * mag)


@pytest.mark.parametrize("k", [8, 16, 20, 32])
@pytest.mark.parametrize("field", [1e-250, 1e-60, 1e-40, 1e-30, 1e-20, 1.0, 1e30, 3e38, 1e40, 1e300, "bump", "patch"])
def test_one_component_of_a_mixed_operator(k, field):
    """A field of rank 1, summed in double-float where FP32's range allows it: 2^-40
    of sum_j |c_j v_j|, as in tests/test_gpu_apply_rows.py, at every scale."""
    src, tgt = syn.uniform_points(3000, 63), syn.uniform_points(301, 64)
    basis = dtk.MultivariatePolynomialBasis(dtk.Linear, 3)
    rbf = dtk.Wendland(2)
    op = dtk.MovingLeastSquaresOperator(None, dev(src), dev(tgt), rbf, basis, k=k, precision="mixed")
    off, idx, coeff = (t.cpu().numpy() for t in op.csr())
    coeff = coeff.astype(np.float64)
    r2 = ((src - 0.5) ** 2).sum(1)
    if field == "bump":
        vals = np.exp(-600.0 * r2)  # 1 to 1e-195 over the cloud
    elif field == "patch":
        vals = np.where(r2 < 0.04, 1e-45, 0.0) + np.where(src[:, 0] > 0.8, 1.0, 0.0)
    else:
        vals = field * np.random.default_rng(7).standard_normal(len(src))
    ref, mag = cpu.apply(off, idx, coeff, vals), cpu.apply(off, idx, np.abs(coeff), np.abs(vals))
    outs = []
    for o in (op, dtk.MovingLeastSquaresOperator.from_bytes(op.to_bytes())):
        y = torch.full((len(tgt),), np.nan, dtype=torch.float64, device="cuda")
        o.apply(dev(vals), y)
        outs.append(y.cpu().numpy())
    host = torch.full((len(tgt),), np.nan, dtype=torch.float64).pin_memory()
    dtk.MovingLeastSquaresOperator.transfer_host(None, torch.from_numpy(src).pin_memory(),
                                                 torch.from_numpy(tgt).pin_memory(),
                                                 torch.from_numpy(vals).pin_memory(), host, rbf, basis, k=k,
                                                 precision="mixed")
    outs.append(host.numpy())
    for y in outs:
        assert np.all(np.abs(y - ref) <= 2.0 ** -40 * mag)
        assert np.array_equal(y, outs[0]) or k == 20
