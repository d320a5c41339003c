"""The search of 32 queries a warp (from 6 batches a resident warp on for rows up to
16, 24 above): row lengths at the edges of its two column sizes, source
clouds of one leaf and of a row's length, a partial last batch, ties and
duplicates, clusters that it leaves to the general kernel, squares outside
FP32's range, strided points.  Rows are bit-exact; of the targets that make the
size, the first, the last and 20,000 others are compared."""
import numpy as np
import pytest
import torch

import datatransferkit_gb300 as dtk
from oracle import cpu

pytestmark = pytest.mark.gpu

N_SHORT, N_LONG = 1_000_003, 2_000_005


def check(src, tgt, k, left=False):
    s, t = torch.from_numpy(src).cuda(), torch.from_numpy(tgt).cuda()
    if left:
        s, t = s.t().contiguous().t(), t.t().contiguous().t()
    off, idx = dtk.knn_search(s, t, k)
    row = min(k, len(src))
    assert off.cpu().numpy()[-1] == row * len(tgt)
    sample = np.unique(np.concatenate([np.arange(64), np.arange(len(tgt) - 64, len(tgt)),
                                       np.random.default_rng(1).integers(0, len(tgt), 20000)]))
    got = idx.view(-1, row)[torch.from_numpy(sample).cuda()].cpu().numpy()
    assert np.array_equal(got.ravel(), cpu.knn(src, tgt[sample], k)[1])


@pytest.mark.parametrize("k,n_src,left", [(2, 2, False), (4, 20, False), (16, 33, True), (8, 3000, False),
                                          (16, 200000, False), (17, 16, True), (17, 40, False), (20, 150000, True),
                                          (32, 32, False), (32, 300001, False)])
def test_row_lengths_and_source_counts(k, n_src, left):
    rng = np.random.default_rng(k + n_src)
    check(rng.random((n_src, 3)), rng.random((N_SHORT if k <= 16 else N_LONG, 3)) * 1.2 - 0.1, k, left)


@pytest.mark.parametrize("k,n", [(6, N_SHORT), (24, N_LONG)])
@pytest.mark.parametrize("cloud", ["ties", "duplicates", "clusters", "far", "tiny", "huge"])
def test_clouds(cloud, k, n):
    rng = np.random.default_rng(7)
    tgt = rng.random((n, 3))
    if cloud == "ties":
        g = np.arange(30.0)
        src = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
        tgt = rng.integers(0, 59, (n, 3)) * 0.5
    elif cloud == "duplicates":
        src = np.repeat(rng.random((3000, 3)), 7, axis=0)
    elif cloud == "clusters":
        src = rng.random((50, 3))[rng.integers(0, 50, 100000)] + 1e-3 * rng.standard_normal((100000, 3))
    elif cloud == "far":
        src = rng.random((20000, 3)) - 4.0
    elif cloud == "tiny":
        src, tgt = rng.random((2000, 3)) * 1e-20, tgt * 1e-20
    else:
        src, tgt = rng.random((200, 3)) * 1e24, tgt * 1e24
    check(src, tgt, k)
