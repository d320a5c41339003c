"""Which neighbour of a row carries the radius' gradient: the last of largest
distance, where the distances are the square roots.  On a grid the squares of
equal distances differ by a rounding that the square root takes away, and the
rows of a radius search are not sorted, so the choice moves a gradient from one
source to another.  Against the oracle, with the bounds of
tests/test_gpu_adjoint.py."""
import numpy as np
import pytest
import torch

import datatransferkit_gb300 as dtk
from oracle import cpu
from tests.test_fixed_jacobi_structured_cpu import rotation

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("radius", [0.9, 1.7])
def test_ties_of_the_square_root(radius):
    i = np.arange(9.0)
    src = np.stack(np.meshgrid(i, i, i, indexing="ij"), -1).reshape(-1, 3)
    j = np.arange(8.0) + 0.5
    tgt = np.stack(np.meshgrid(j, j, j, indexing="ij"), -1).reshape(-1, 3)
    src, tgt = src @ rotation(), tgt @ rotation()
    rng = np.random.default_rng(9)
    vals, cot = rng.standard_normal(len(src)), rng.standard_normal(len(tgt))
    op = dtk.MovingLeastSquaresOperator(None, dev(src), dev(tgt), dtk.Wendland(2),
                                        dtk.MultivariatePolynomialBasis(dtk.Linear, 3), radius=radius,
                                        keep_points=True)
    _, gc = op.apply_adjoint(dev(cot), dev(vals), coords=True)
    off, idx, _ = (t.cpu().numpy() for t in op.csr())
    # the rows this is about: several largest distances that are not several largest squares
    x = src[idx] - np.repeat(tgt, np.diff(off), axis=0)
    d2 = (x[:, 0] * x[:, 0] + x[:, 1] * x[:, 1]) + x[:, 2] * x[:, 2]
    differ = 0
    for t in range(len(tgt)):
        row = d2[off[t]:off[t + 1]]
        differ += len(row) > 0 and np.nonzero(np.sqrt(row) == np.sqrt(row.max()))[0][-1] != np.nonzero(row == row.max())[0][-1]
    assert differ > 10
    want = cpu.coord_grad(src, tgt, off, idx, 1, 1, vals, cot)
    assert np.abs(gc.cpu().numpy() - want).max() <= 1e-8 * np.abs(want).max()
