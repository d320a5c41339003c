"""The one-query-a-lane nearest search (k = 1 from three queries a resident warp
on) at the edges of its range: source counts around one leaf, a partial last
warp, exact ties and duplicates (the FP64 pass), scales whose squares leave
FP32's range, targets far outside, strided points.  Indices are bit-exact."""
import numpy as np
import pytest
import torch

import datatransferkit_gb300 as dtk
from oracle import cpu

pytestmark = pytest.mark.gpu

N_TGT = 40003


def check(src, tgt, left=False):
    s, t = torch.from_numpy(src).cuda(), torch.from_numpy(tgt).cuda()
    if left:
        s, t = s.t().contiguous().t(), t.t().contiguous().t()
    _, idx = dtk.knn_search(s, t, 1)
    assert np.array_equal(idx.cpu().numpy(), cpu.knn(src, tgt, 1)[1])


@pytest.mark.parametrize("n_src", [1, 2, 31, 32, 33, 257, 5000, 60001])
@pytest.mark.parametrize("left", [False, True])
def test_source_counts(n_src, left):
    rng = np.random.default_rng(n_src)
    check(rng.random((n_src, 3)), rng.random((N_TGT, 3)) * 1.5 - 0.25, left)


@pytest.mark.parametrize("scale", [1e-24, 1e-12, 1.0, 1e12, 1e25])
def test_scales(scale):
    rng = np.random.default_rng(3)
    check((rng.random((300, 3)) - 0.5) * scale, (rng.random((N_TGT, 3)) - 0.5) * scale)


@pytest.mark.parametrize("spread", [0.0, 1e-15, 1e-8])
def test_ties_and_near_ties(spread):
    rng = np.random.default_rng(4)
    g = np.stack(np.meshgrid(*[np.arange(10.0)] * 3, indexing="ij"), -1).reshape(-1, 3)
    src = np.concatenate([g, g + spread * rng.standard_normal(g.shape)])
    check(src, rng.integers(0, 19, (N_TGT, 3)) * 0.5)


def test_far_targets_and_offset():
    rng = np.random.default_rng(5)
    src = rng.random((4000, 3)) + 1e6
    check(src, rng.random((N_TGT, 3)) * 50 + (1e6 - 25))
