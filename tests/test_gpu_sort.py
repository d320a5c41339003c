"""The point sort at the edges of its paths (one block, an even number of pairs a
thread of 1024 up to 16, tiles of 4096 pairs with summed or scanned histograms): a
search over n sources and n targets visits every point of both sorted orders,
so a lost, doubled or misplaced pair changes its rows.  Rows are bit-exact."""
import numpy as np
import pytest
import torch

import datatransferkit_gb300 as dtk
from datatransferkit_gb300 import synthetic as syn
from oracle import cpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 33, 2048, 2049, 4097, 6144, 6145, 8193, 10241, 12289, 14337, 16384, 16385,
                                128 * 4096, 128 * 4096 + 1])
def test_sorted_orders_at_path_edges(n):
    src, tgt = syn.uniform_points(n, 31), syn.uniform_points(n, 32)
    src[n // 2:] = src[: n - n // 2]  # equal keys: a stable order is part of the result
    off, idx = dtk.knn_search(torch.from_numpy(src).cuda(), torch.from_numpy(tgt).cuda(), 4)
    o2, i2, _ = cpu.knn(src, tgt, 4)
    assert np.array_equal(off.cpu().numpy(), o2) and np.array_equal(idx.cpu().numpy(), i2)
