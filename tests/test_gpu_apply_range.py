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
