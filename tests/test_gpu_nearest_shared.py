"""The nearest search where many sources lie in one Morton cell, on both sides of
its rule (1500 queries for each leaf of the fullest cell, four fifths of the
nodes in such cells): graded coordinates, and clusters far smaller than a cell.
Indices are bit-exact."""
import numpy as np
import pytest
import torch

import datatransferkit_gb300 as dtk
from oracle import cpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cloud", ["graded", "clusters", "points"])
@pytest.mark.parametrize("n_src", [40000, 300000])
@pytest.mark.parametrize("n_tgt", [30001, 130003])
def test_crowded_cells(cloud, n_src, n_tgt):
    rng = np.random.default_rng(n_src + n_tgt)
    if cloud == "graded":
        src, tgt = rng.random((n_src, 3)) ** 4, rng.random((n_tgt, 3)) ** 4
    else:
        centres = rng.random((40, 3))
        spread = 1e-5 if cloud == "clusters" else 0.0  # (0: exact duplicates by the thousand)
        src = centres[rng.integers(0, 40, n_src)] + spread * rng.standard_normal((n_src, 3))
        tgt = centres[rng.integers(0, 40, n_tgt)] + 1e-4 * rng.standard_normal((n_tgt, 3))
    _, idx = dtk.knn_search(torch.from_numpy(src).cuda(), torch.from_numpy(tgt).cuda(), 1)
    some = np.unique(np.concatenate([np.arange(64), rng.integers(0, n_tgt, 3000)]))
    assert np.array_equal(idx.cpu().numpy()[some], cpu.knn(src, tgt[some], 1)[1])
