"""The search of 32 queries a warp at the row lengths that take it from larger target
sets on: 13 to 16 from 1.5M, 29 to 32 from 3.9M.  As tests/test_gpu_knn_batches.py:
rows are bit-exact; of the targets that make the size, the first, the last and 20,000
others are compared."""
import numpy as np
import pytest

from tests.test_gpu_knn_batches import check

pytestmark = pytest.mark.gpu

N_16, N_32 = 1_600_003, 4_000_037


@pytest.mark.parametrize("k, n, n_src", [(13, N_16, 13), (16, N_16, 33), (16, N_16, 200000), (29, N_32, 40),
                                         (32, N_32, 32), (32, N_32, 300001)])
def test_row_lengths_and_source_counts(k, n, n_src):
    rng = np.random.default_rng(k + n_src)
    check(rng.random((n_src, 3)), rng.random((n, 3)) * 1.2 - 0.1, k, left=k == 16)


@pytest.mark.parametrize("k, n", [(16, N_16), (32, N_32)])
@pytest.mark.parametrize("cloud", ["ties", "duplicates", "clusters"])
def test_clouds(cloud, k, n):
    rng = np.random.default_rng(8)
    tgt = rng.random((n, 3))
    if cloud == "ties":
        g = np.arange(30.0)
        src = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
        tgt = rng.integers(0, 59, (n, 3)) * 0.5
    elif cloud == "duplicates":
        src = np.repeat(rng.random((3000, 3)), 7, axis=0)
    else:
        src = rng.random((50, 3))[rng.integers(0, 50, 100000)] + 1e-3 * rng.standard_normal((100000, 3))
    check(src, tgt, k)
