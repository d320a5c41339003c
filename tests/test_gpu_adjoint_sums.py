"""The order and the rounding of the adjoint's sums over a source's entries: one
fused multiply-add an entry, ascending in (target, place in the row), so that
the result is that of the same sums on the CPU (computed here with twice FP64's
precision between the roundings, which is what a fused multiply-add rounds
once).  This needs a stable sort of the entries by source: entry counts on both
sides of the sort's paths (16384 and 128 * 4096 pairs)."""
from fractions import Fraction

import numpy as np
import pytest
import torch

import datatransferkit_gb300 as dtk
from datatransferkit_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def fused_sums(off, idx, coeff, cot, sources):
    """grad_values of the given sources, each sum rounded once an entry."""
    rows = np.repeat(np.arange(len(off) - 1), np.diff(off))
    out = []
    for s in sources:
        acc = 0.0
        for e in np.nonzero(idx == s)[0]:
            acc = float(Fraction(float(coeff[e])) * Fraction(float(cot[rows[e]])) + Fraction(acc))
        out.append(acc)
    return np.array(out)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n_tgt, k", [(2048, 8), (2049, 8), (128 * 4096 // 16, 16), (128 * 4096 // 16 + 1, 16),
                                      (3000, 10)])
def test_one_fused_multiply_add_an_entry_in_order(precision, n_tgt, k):
    src, tgt = syn.uniform_points(500, 81), syn.uniform_points(n_tgt, 82)  # (few sources: long sums)
    vals, cot = syn.smooth_field(src), np.random.default_rng(2).standard_normal(n_tgt)
    op = dtk.MovingLeastSquaresOperator(None, dev(src), dev(tgt), dtk.Wendland(2),
                                        dtk.MultivariatePolynomialBasis(dtk.Linear, 3), k=k, precision=precision,
                                        keep_points=True)
    off, idx, coeff = (t.cpu().numpy() for t in op.csr())
    some = np.random.default_rng(3).choice(len(src), 12, replace=False)
    want = fused_sums(off, idx, coeff, cot, some)
    for coords in (False, True):
        gv, _ = op.apply_adjoint(dev(cot), dev(vals), coords=coords)
        assert np.array_equal(gv.cpu().numpy()[some], want)


def test_rows_of_a_radius():
    src, tgt = syn.uniform_points(500, 83), syn.uniform_points(400, 84)
    vals, cot = syn.smooth_field(src), np.random.default_rng(4).standard_normal(len(tgt))
    op = dtk.MovingLeastSquaresOperator(None, dev(src), dev(tgt), dtk.Wendland(2),
                                        dtk.MultivariatePolynomialBasis(dtk.Linear, 3), radius=0.3, keep_points=True)
    off, idx, coeff = (t.cpu().numpy() for t in op.csr())
    want = fused_sums(off, idx, coeff, cot, range(12))
    for coords in (False, True):
        gv, _ = op.apply_adjoint(dev(cot), dev(vals), coords=coords)
        assert np.array_equal(gv.cpu().numpy()[:12], want)


@pytest.mark.parametrize("n_src", [704 * 700 + 1, 704 * 700 + 703])  # the larger blocks, a partial last one
def test_many_sources(n_src):
    src, tgt = syn.uniform_points(n_src, 85), syn.uniform_points(60000, 86)
    cot = np.random.default_rng(5).standard_normal(len(tgt))
    op = dtk.MovingLeastSquaresOperator(None, dev(src), dev(tgt), dtk.Wendland(2),
                                        dtk.MultivariatePolynomialBasis(dtk.Linear, 3), k=8)
    off, idx, coeff = (t.cpu().numpy() for t in op.csr())
    some = [0, 703, 704, n_src - 1, *np.unique(idx)[:: 30000]]
    gv, _ = op.apply_adjoint(dev(cot))
    assert np.array_equal(gv.cpu().numpy()[some], fused_sums(off, idx, coeff, cot, some))
