"""The FP64 sums over uniform rows: the same bits from a field of any layout, by
index or on a sorted copy, with one row or several a group of lanes, and from a
saved operator (which has indices only, and rows of any length: 64 and 128 here).
Against the oracle's FP64 sums: 1e-14 of sum_j |c_j v_j| for up to 32 terms, 4e-14
for up to 128."""
import struct

import numpy as np
import pytest
import torch

import datatransferkit_gb300 as dtk
from datatransferkit_gb300 import synthetic as syn
from oracle import cpu

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def product(n_src, off, idx, coeff):
    """The bytes of a saved operator (layout: csrc/dtk_io.cu)."""
    head = b"DTKMLS01" + struct.pack("<IIqqqiiiid", 1, int(coeff.dtype == np.float32), n_src, len(off) - 1, len(idx),
                                     1, 1, 0, int(coeff.dtype == np.float32), 0.0)
    body = head + off.astype("<i4").tobytes() + idx.astype("<i4").tobytes() + coeff.tobytes()
    h = 1469598103934665603
    for w in np.frombuffer(body + b"\0" * (-len(body) % 8), "<u8").tolist():
        h = ((h ^ w) * 1099511628211) & (2 ** 64 - 1)
    return body + struct.pack("<Q", h)


def fields(vals):
    """The same field in several layouts."""
    n, c = vals.shape
    wide = np.zeros((n, c + 2))
    wide[:, 1:1 + c] = vals
    yield dev(vals)
    yield dev(vals.T).t()
    yield dev(wide)[:, 1:1 + c]


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("row", [4, 8, 16, 32, 64, 128])
@pytest.mark.parametrize("n_tgt", [1, 7, 257, 100001])
def test_row_lengths_components_and_layouts(dtype, row, n_tgt):
    rng = np.random.default_rng(row + n_tgt)
    n_src = 5000
    idx = rng.integers(0, n_src, n_tgt * row)
    coeff = rng.standard_normal(n_tgt * row).astype(dtype)
    coeff[::97] = 0.0
    if dtype == np.float32:
        coeff[1::89] = np.float32(1e-41)  # subnormal
    off = np.arange(n_tgt + 1) * row
    op = dtk.MovingLeastSquaresOperator.from_bytes(product(n_src, off, idx, coeff))
    tol = 1e-14 if row <= 32 else 4e-14
    for n_comp in (1, 2, 3, 4, 5, 7, 9):
        vals = rng.standard_normal((n_src, n_comp))
        g = vals[idx].reshape(n_tgt, row, n_comp)
        c = coeff.astype(np.float64).reshape(n_tgt, row, 1)
        ref, mag = (c * g).sum(1), np.abs(c * g).sum(1)
        first = None
        for v in fields(vals):
            out = torch.full((n_tgt, n_comp), np.nan, dtype=torch.float64, device="cuda")
            op.apply(v, out)
            first = out if first is None else first
            assert torch.equal(out, first)
            part = torch.full((n_comp, n_tgt), np.nan, dtype=torch.float64, device="cuda").t()
            op.apply(v, part)
            assert torch.equal(part, first)
        assert np.all(np.abs(first.cpu().numpy() - ref) <= tol * mag)
        # one component of it, as a field of one component, and (FP64) of rank 1
        one = torch.empty((n_tgt, 1), dtype=torch.float64, device="cuda")
        op.apply(dev(vals[:, :1]), one)
        assert torch.equal(one[:, 0], first[:, 0])
        if dtype == np.float64:
            y = torch.empty(n_tgt, dtype=torch.float64, device="cuda")
            op.apply(dev(vals[:, 0]), y)
            assert torch.equal(y, first[:, 0])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n_src, n_tgt, k", [(3000, 2000, 32), (200000, 150000, 8), (2000000, 1000000, 32),
                                             (2000000, 2000000, 16)])  # the last two on a sorted copy
def test_saved_operator_gives_the_same_bits(precision, n_src, n_tgt, k):
    src, tgt = syn.uniform_points(n_src, 87), syn.uniform_points(n_tgt, 88)
    op = dtk.MovingLeastSquaresOperator(None, dev(src), dev(tgt), dtk.Wendland(2),
                                        dtk.MultivariatePolynomialBasis(dtk.Linear, 3), k=k, precision=precision)
    saved = dtk.MovingLeastSquaresOperator.from_bytes(op.to_bytes())
    for n_comp in (1, 2, 3, 5):
        vals = dev(np.random.default_rng(n_comp).standard_normal((n_src, n_comp)))
        a, b = (torch.full((n_tgt, n_comp), np.nan, dtype=torch.float64, device="cuda") for _ in range(2))
        op.apply(vals, a)
        saved.apply(vals, b)
        assert torch.equal(a, b) and bool(torch.isfinite(a).all())
