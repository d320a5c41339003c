"""The tests that hand a moment matrix back before its Jacobi because it will be
truncated (csrc/dtk_fixed.cuh and dtk_setup_fixed.cu, built for the host or
restated): they answer yes only where the smallest eigenvalue is below the
threshold, twice DBL_EPSILON, and do so for matrices well below it."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from datatransferkit_gb300 import synthetic as syn
from oracle import cpu
from tests.test_fixed_jacobi_cpu import moments_of

ROOT = Path(__file__).resolve().parents[1]
THRESHOLD = 2.0 ** -51


@pytest.fixture(scope="module")
def truncates(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    lib = tmp_path_factory.mktemp("fixed") / "libtruncates.so"
    cmd = [gxx, "-std=c++17", "-O2", "-ffp-contract=off", "-Wno-unknown-pragmas", "-shared", "-fPIC", "-I",
           str(ROOT / "datatransferkit_gb300" / "csrc"), str(ROOT / "tests" / "cpp" / "fixed_truncates.cpp"),
           "-o", str(lib)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    f = C.CDLL(str(lib)).fixed_truncates
    f.restype = None

    def run(moments, m):
        moments = np.ascontiguousarray(moments)
        out = np.zeros(len(moments), np.int32)
        f(C.c_int(m), C.c_long(len(moments)), moments.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p))
        return out

    return run


def smallest_eigenvalues(moments, m):
    """From the inverse, whose largest eigenvalue loses nothing to the matrix' range."""
    a = np.zeros((len(moments), m, m))
    a[(slice(None), *np.triu_indices(m))] = moments
    a += np.triu(a, 1).transpose(0, 2, 1)
    return 1 / np.linalg.eigvalsh(np.linalg.inv(a))[:, -1]


@pytest.mark.parametrize("basis, k, rbf, scales", [(2, 32, 1, np.geomspace(2e-3, 1.0, 14)),
                                                   (2, 20, 2, np.geomspace(2e-3, 1.0, 14)),
                                                   (1, 12, 0, np.geomspace(1e-8, 1e-4, 10))])
def test_only_what_truncates(truncates, basis, k, rbf, scales):
    m = cpu.BASIS_SIZE[basis]
    seen = set()
    for scale in scales:
        src, tgt = scale * syn.uniform_points(3000, 21), scale * syn.uniform_points(400, 22)
        _, idx, _ = cpu.knn(src, tgt, k)
        moments = moments_of(src, tgt, idx, k, rbf, basis)
        smallest = smallest_eigenvalues(moments, m)
        said = truncates(moments, m)
        assert (smallest[said == 1] < THRESHOLD).all()
        # a diagonal entry bounds the smallest eigenvalue: far enough below, the test has to say so
        diag = moments[:, [i * m - i * (i - 1) // 2 for i in range(m)]]
        assert (said[diag.min(1) < THRESHOLD / 2] != 0).all()
        seen |= set(said.tolist())
    assert {0, 1} <= seen


def test_the_size_of_a_row_bounds_its_least_diagonal_moment():
    # min over the axes of sum phi x^2 (x^2 y^2) <= len a max over q of phi(q) q^p (1.1 dmax)^p, a = 1/3 (1/9)
    q = np.linspace(0.0, 1.0, 200001)[:-1]
    for rbf in range(6):  # the positive functions
        phi = cpu.rbf(rbf, q)
        assert (phi * q ** 2).max() * 1.1 ** 2 / 3 < 0.125
        assert (phi * q ** 4).max() * 1.1 ** 4 / 9 < 0.0125
