"""The fixed-point Jacobi (csrc/dtk_fixed.cuh, built for the host) on moment
matrices whose diagonal entries are nearly or exactly equal, as structured grids
give them: the rotation has to stay orthogonal when the difference of two
diagonal entries and the pivot are both a few units of the last place.  The
bound is that of tests/test_fixed_jacobi_cpu.py: ten times the distance between
the oracle and its multiply-add-contracted build, or 1e-12."""
import numpy as np
import pytest

from oracle import cpu
from tests.test_fixed_jacobi_cpu import both_oracles, fixed, moments_of  # noqa: F401


def rotation():
    q, _ = np.linalg.qr(np.random.default_rng(5).standard_normal((3, 3)))
    return q


@pytest.mark.parametrize("basis, k, rbf", [(1, 8, 0), (1, 8, 1), (2, 32, 1), (2, 20, 2)])
@pytest.mark.parametrize("spacing", [2.0, 1.0, 0.1])
@pytest.mark.parametrize("grid", ["plain", "shifted", "rotated", 1e-14, 1e-12, 1e-9])
def test_grids_with_targets_at_the_cell_centres(fixed, grid, spacing, basis, k, rbf):  # noqa: F811
    i = np.arange(9.0)
    src = np.stack(np.meshgrid(i, i, i, indexing="ij"), -1).reshape(-1, 3) * spacing
    j = np.arange(8.0) + 0.5
    tgt = np.stack(np.meshgrid(j, j, j, indexing="ij"), -1).reshape(-1, 3) * spacing
    if grid == "shifted":
        src, tgt = src + 0.1, tgt + 0.1
    elif grid == "rotated":
        src, tgt = src @ rotation(), tgt @ rotation()
    elif grid != "plain":
        src = src + grid * np.random.default_rng(6).standard_normal(src.shape)
    off, idx, _ = cpu.knn(src, tgt, k)
    m = cpu.BASIS_SIZE[basis]
    moments = moments_of(src, tgt, idx, k, rbf, basis)
    # (32 of a grid's points leave some quadratic moments singular: not the form's)
    full = np.zeros((len(tgt), m, m))
    full[(slice(None), *np.triu_indices(m))] = moments
    full += np.triu(full, 1).transpose(0, 2, 1)
    d = 1 / np.sqrt(np.einsum("nii->ni", full))
    well = np.linalg.cond(full * d[:, :, None] * d[:, None, :]) < 1e4
    ref, other = both_oracles(src, tgt, off, idx, rbf, basis)
    got, back = fixed(moments, m)
    deg = np.array([0, 1, 1, 1, 2, 2, 2, 2, 2, 2])[:m]
    size = np.abs(ref * spacing ** deg).max(1)
    err = np.abs((got - ref) * spacing ** deg).max(1) / size
    spread = np.abs((other - ref) * spacing ** deg).max(1) / size
    keep = ~back & well
    assert keep[well].all()
    if keep.any():
        assert err[keep].max() <= max(1e-12, 10 * spread[keep].max())
    assert keep.any() or basis == 2


@pytest.mark.parametrize("m", [4, 10])
@pytest.mark.parametrize("c", [1.0, 1e4, 1e-3])
@pytest.mark.parametrize("p", [8, 24, 32, 40, 44, 48, 50, 52, 54, 56, 58, 60])
def test_near_multiples_of_the_identity(fixed, p, c, m):  # noqa: F811
    rng = np.random.default_rng(p)
    s = rng.uniform(-1, 1, (200, m, m))
    s = (s + s.transpose(0, 2, 1)) / 2
    a = c * (np.eye(m) + 2.0 ** -p * s)
    # (and with equal diagonal entries: a turn of 45 degrees)
    a[::2, np.arange(m), np.arange(m)] = c
    got, back = fixed(a[(slice(None), *np.triu_indices(m))], m)
    assert not back.any()
    ref = np.linalg.inv(a)[:, 0]
    # the stop is absolute, DBL_EPSILON over all entries: what it leaves moves row 0 by up to that over c^2
    assert np.abs(got - ref).max() * c <= 1e-12 + 4 * 2.220446049250313e-16 / c
