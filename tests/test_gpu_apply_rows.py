"""The apply over uniform rows at the edges of its groups: a lane's rows for
every row length it takes, last groups that are partly empty, one to five
components (passes of up to four), strided fields, and a saved operator (by
index).  Against the oracle's FP64 sums of the same coefficients: 1e-14 of
sum_j |c_j v_j| for FP64 sums of up to 32 terms, 2^-40 for double-floats."""
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
@pytest.mark.parametrize("k", [4, 8, 16, 32])
@pytest.mark.parametrize("n_tgt", [1, 3, 31, 257])
def test_rows_and_components(precision, k, n_tgt):
    src, tgt = syn.uniform_points(3000, 51), syn.uniform_points(n_tgt, 52)
    basis = dtk.MultivariatePolynomialBasis(dtk.Quadratic if k >= 16 else dtk.Linear, 3)
    op = dtk.MovingLeastSquaresOperator(None, dev(src), dev(tgt), dtk.Wendland(2), basis, k=k, precision=precision)
    off, idx, coeff = (t.cpu().numpy() for t in op.csr())
    coeff = coeff.astype(np.float64)
    tol = 1e-14 if precision == "fp64" else 2.0 ** -40
    for n_comp in (1, 2, 3, 4, 5):
        vals = np.random.default_rng(n_comp).standard_normal((len(src), n_comp))
        ref = np.stack([cpu.apply(off, idx, coeff, vals[:, c]) for c in range(n_comp)], 1)
        mag = np.stack([cpu.apply(off, idx, np.abs(coeff), np.abs(vals[:, c])) for c in range(n_comp)], 1)
        for o in (op, dtk.MovingLeastSquaresOperator.from_bytes(op.to_bytes())):
            for v in (dev(vals), dev(vals.T.copy()).t()):
                out = torch.full((n_comp, n_tgt), np.nan, dtype=torch.float64, device="cuda").t()
                o.apply(v, out)
                assert np.all(np.abs(out.cpu().numpy() - ref) <= tol * mag + 1e-300)
        y = torch.full((n_tgt,), np.nan, dtype=torch.float64, device="cuda")
        op.apply(dev(vals[:, 0]), y)
        assert np.all(np.abs(y.cpu().numpy() - ref[:, 0]) <= tol * mag[:, 0] + 1e-300)
