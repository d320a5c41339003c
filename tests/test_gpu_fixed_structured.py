"""The FP64 setup on structured grids: moment matrices with (nearly) equal
diagonal entries through the single operator (both layouts of the fixed-point
kernel), radius rows and a batch, against the oracle.  The bound per row is that
of tests/test_gpu_fixed_setup.py: 1e-12, or 100 times the distance between the
oracle and its multiply-add-contracted build."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import datatransferkit_gb300 as dtk
from oracle import cpu
from tests.test_fixed_jacobi_structured_cpu import rotation

BASIS = dtk.MultivariatePolynomialBasis(dtk.Linear, 3)


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def grid(kind, n, spacing=2.0):
    i = np.arange(n + 1.0)
    src = np.stack(np.meshgrid(i, i, i, indexing="ij"), -1).reshape(-1, 3) * spacing
    j = np.arange(float(n)) + 0.5
    tgt = np.stack(np.meshgrid(j, j, j, indexing="ij"), -1).reshape(-1, 3) * spacing
    if kind == "shifted":
        return src + 0.1, tgt + 0.1
    if kind == "rotated":
        return src @ rotation(), tgt @ rotation()
    return src + kind * np.random.default_rng(6).standard_normal(src.shape), tgt


def check(src, tgt, rbf, op):
    off, idx, coeff = (t.cpu().numpy() for t in op.csr())
    ref = cpu.mls_coefficients(src, tgt, off, idx, rbf.id, 1)[0]
    other = cpu.mls_coefficients(src, tgt, off, idx, rbf.id, 1, contract=True)[0]
    r, c, o = (a.reshape(len(tgt), -1) for a in (ref, coeff, other))
    size = np.abs(r).max(1)
    spread = (np.abs(o - r).max(1) / size).max()
    assert (np.abs(c - r).max(1) / size).max() <= max(1e-12, 100 * spread)
    assert np.abs(c.sum(1) - 1).max() <= 1e-12


@pytest.mark.parametrize("kind", ["shifted", "rotated", 1e-14, 1e-12, 1e-9])
@pytest.mark.parametrize("n", [8, 36])  # two lanes a matrix, one
@pytest.mark.parametrize("rbf", [dtk.Wendland(0), dtk.Wendland(2)])
def test_grid_cells(kind, n, rbf):
    src, tgt = grid(kind, n)
    check(src, tgt, rbf, dtk.MovingLeastSquaresOperator(None, dev(src), dev(tgt), rbf, BASIS, k=8))


@pytest.mark.parametrize("kind", ["shifted", "rotated", 1e-12])
def test_grid_cells_radius_and_batch(kind):
    rbf = dtk.Wendland(0)
    src, tgt = grid(kind, 8)
    # the eight corners lie at sqrt(3), the next points at 3.3
    check(src, tgt, rbf, dtk.MovingLeastSquaresOperator(None, dev(src), dev(tgt), rbf, BASIS, radius=2.0))
    problems = [dict(source_points=dev(src), target_points=dev(tgt), rbf=rbf, basis=BASIS, k=8)]
    check(src, tgt, rbf, dtk.MovingLeastSquaresBatch(problems))
