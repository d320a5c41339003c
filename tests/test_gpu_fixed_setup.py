"""The FP64 setup with the fixed-point Jacobi (csrc/dtk_setup_fixed.cu) at the
edges of its tiles: 16 or 32 targets a warp (two lanes a matrix below about
39k targets, one above: the same bits), partial warps, rows that are handed
back to the FP64 kernel in between."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import datatransferkit_gb300 as dtk
from datatransferkit_gb300 import synthetic as syn
from oracle import cpu

BASES = {0: dtk.Constant, 1: dtk.Linear, 2: dtk.Quadratic}


def coefficients(src, tgt, basis, rbf, k):
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    op = dtk.MovingLeastSquaresOperator(None, to(src), to(tgt), rbf, dtk.MultivariatePolynomialBasis(BASES[basis], 3), k=k)
    off, idx, coeff = op.csr()
    return off.cpu().numpy(), idx.cpu().numpy(), coeff.cpu().numpy(), op


def check(src, tgt, basis, rbf, k):
    off, idx, coeff, op = coefficients(src, tgt, basis, rbf, k)
    ref = cpu.mls_coefficients(src, tgt, off, idx, rbf.id, basis)[0]
    other = cpu.mls_coefficients(src, tgt, off, idx, rbf.id, basis, contract=True)[0]
    row = int(off[1]) if len(tgt) else 1
    r, c, o = (a.reshape(-1, row) for a in (ref, coeff, other))
    size = np.abs(r).max(1)
    spread = (np.abs(o - r).max(1) / size).max()
    assert (np.abs(c - r).max(1) / size).max() <= max(1e-12, 100 * spread)
    return coeff, op


@pytest.mark.parametrize("basis, rbf, k", [(2, dtk.Wendland(2), 20), (1, dtk.Wendland(0), 8), (0, dtk.Wu(4), 5)])
@pytest.mark.parametrize("n_tgt", [1, 15, 16, 17, 31, 32, 33, 500])
def test_partial_warps(n_tgt, basis, rbf, k):
    check(syn.uniform_points(3000, 31), syn.uniform_points(n_tgt, 32), basis, rbf, k)


@pytest.mark.parametrize("basis, k", [(2, 32), (1, 8), (2, 15)])  # (15: V in larger units)
def test_both_layouts_give_the_same_bits(basis, k):
    src, tgt = syn.uniform_points(20000, 33), syn.uniform_points(40001, 34)
    whole = coefficients(src, tgt, basis, dtk.Wendland(4), k)[2].reshape(-1, k)  # one lane a matrix
    some = coefficients(src, tgt[:777], basis, dtk.Wendland(4), k)[2].reshape(-1, k)  # two
    assert np.array_equal(whole[:777], some)


def test_rows_handed_back_among_others():
    """Targets whose neighbours lie in one plane (a zero column) between targets in a volume."""
    src = syn.uniform_points(4000, 35)
    plane = syn.uniform_points(2000, 36)
    plane[:, 2] = 0.0
    plane[:, :2] += 5.0
    tgt = np.concatenate([syn.uniform_points(300, 37), plane[:300] + [1e-3, 0, 0]])
    tgt = tgt[np.random.default_rng(1).permutation(len(tgt))]
    _, op = check(np.concatenate([src, plane]), tgt, 2, dtk.Wendland(2), 32)
    assert op.underdetermined == 300
