"""The fixed-point Jacobi of the FP64 setup (csrc/dtk_fixed.cuh), built for the
host (tests/cpp/fixed_jacobi.cpp), against the oracle: row 0 of the
pseudo-inverse of the same moment matrices.  The bound per row is the largest
row distance between the oracle and its multiply-add-contracted build, ten
times over, or 1e-12: the form rounds no more coarsely than FP64 does."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from datatransferkit_gb300 import synthetic as syn
from oracle import cpu

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def fixed(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    lib = tmp_path_factory.mktemp("fixed") / "libfixed.so"
    cmd = [gxx, "-std=c++17", "-O2", "-ffp-contract=off", "-Wno-unknown-pragmas", "-shared", "-fPIC", "-I",
           str(ROOT / "datatransferkit_gb300" / "csrc"), str(ROOT / "tests" / "cpp" / "fixed_jacobi.cpp"),
           "-o", str(lib)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    f = C.CDLL(str(lib)).fixed_row0
    f.restype = None

    def run(moments, m, cap=224):
        moments = np.ascontiguousarray(moments)
        out = np.zeros((len(moments), m))
        back = np.zeros(len(moments), np.int32)
        f(C.c_int(m), C.c_long(len(moments)), moments.ctypes.data_as(C.c_void_p), C.c_int(cap),
          out.ctypes.data_as(C.c_void_p), back.ctypes.data_as(C.c_void_p))
        return out, back.astype(bool)

    return run


def moments_of(src, tgt, idx, k, rbf, basis):
    """(n, m (m + 1) / 2) upper triangles of P^T Phi P, the reference's radius rule."""
    x = src[idx.reshape(-1, k)] - tgt[:, None]
    d = np.sqrt((x[..., 0] * x[..., 0] + x[..., 1] * x[..., 1]) + x[..., 2] * x[..., 2])
    phi = cpu.rbf(rbf, (d / (1.1 * d.max(1))[:, None]).ravel()).reshape(d.shape)
    m = cpu.BASIS_SIZE[basis]
    P = cpu.basis(basis, x.reshape(-1, 3)).reshape(len(tgt), k, m)
    A = np.einsum("nka,nk,nkc->nac", P, phi, P)
    return A[(slice(None), *np.triu_indices(m))]


def both_oracles(src, tgt, off, idx, rbf, basis):
    return [cpu.mls_coefficients(src, tgt, off, idx, rbf, basis, want_row0=True, contract=c)[2] for c in (False, True)]


@pytest.mark.parametrize("n, scale, basis, k, rbf", [
    (1000, 1.0, 1, 8, 0), (1000, 1.0, 2, 20, 1), (10000, 1.0, 2, 20, 1), (100000, 1.0, 2, 32, 2),
    (100000, 1.0, 1, 16, 4), (5000, 1e3, 2, 32, 1), (5000, 3e-2, 2, 32, 3), (5000, 10.0, 2, 32, 2), (5000, 1e3, 1, 12, 5)])
def test_row0_matches_the_oracle(fixed, n, scale, basis, k, rbf):
    src, tgt = scale * syn.uniform_points(n, 11), scale * syn.uniform_points(2000, 12)
    off, idx, _ = cpu.knn(src, tgt, k)
    ref, other = both_oracles(src, tgt, off, idx, rbf, basis)
    got, back = fixed(moments_of(src, tgt, idx, k, rbf, basis), cpu.BASIS_SIZE[basis])
    # row 0 of the pseudo-inverse in the basis' own scale: entry j times h^degree
    h = scale * (k / n) ** (1 / 3)
    deg = np.array([0, 1, 1, 1, 2, 2, 2, 2, 2, 2])[:ref.shape[1]]
    size = np.abs(ref * h ** deg).max(1)
    err = np.abs((got - ref) * h ** deg).max(1) / size
    spread = np.abs((other - ref) * h ** deg).max(1) / size
    keep = ~back
    assert keep.mean() > 0.9, "most matrices of a well-posed cloud are taken"
    assert err[keep].max() <= max(1e-12, 10 * spread.max())
    assert np.sqrt(np.mean(err[keep] ** 2)) <= max(1e-12, 10 * np.sqrt(np.mean(spread ** 2)))


def test_what_the_form_does_not_hold_is_handed_back(fixed):
    eye = np.eye(4)
    up = np.triu_indices(4)
    bad = []
    for value in (0.0, -1.0, np.nan, np.inf, 1e-300, 1e300):  # a diagonal entry
        a = eye.copy()
        a[2, 2] = value
        bad.append(a[up])
    a = np.ones((4, 4))  # singular
    bad.append(a[up])
    a = eye.copy()
    a[1, 1] = 3e-16  # at the truncation threshold
    bad.append(a[up])
    a = eye.copy()
    a[0, 1] = 5.0  # not bounded by the diagonal: indefinite
    bad.append(a[up])
    _, back = fixed(np.array(bad), 4)
    assert back.all()
    row, back = fixed(np.array([eye[up], (4.0 * eye)[up]]), 4)
    assert not back.any()
    assert np.array_equal(row, [[1, 0, 0, 0], [0.25, 0, 0, 0]])


def test_more_rotations_than_the_cap_are_handed_back(fixed):
    src, tgt = syn.uniform_points(2000, 3), syn.uniform_points(50, 4)
    off, idx, _ = cpu.knn(src, tgt, 32)
    _, back = fixed(moments_of(src, tgt, idx, 32, 1, 2), 10, cap=40)
    assert back.all()


def test_rows_far_below_row_0_s_scale(fixed):
    # half as many neighbours again as the basis has: V outgrows its first unit
    src, tgt = syn.uniform_points(10000, 13), syn.uniform_points(10000, 14)
    off, idx, _ = cpu.knn(src, tgt, 15)
    got, back = fixed(moments_of(src, tgt, idx, 15, 2, 2), 10)
    assert not back.any()
    ref, other = both_oracles(src, tgt, off, idx, 2, 2)
    deg = np.array([0, 1, 1, 1, 2, 2, 2, 2, 2, 2])
    h = (15 / 10000) ** (1 / 3)
    size = np.abs(ref * h ** deg).max(1)
    err = np.abs((got - ref) * h ** deg).max(1) / size
    spread = np.abs((other - ref) * h ** deg).max(1) / size
    assert err.max() <= max(1e-12, 10 * spread.max())
    assert np.sqrt(np.mean(err ** 2)) <= max(1e-12, 10 * np.sqrt(np.mean(spread ** 2)))
