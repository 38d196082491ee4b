"""Leaf index ranges of sorted samples whose last warp is partial, whose runs
of one leaf end inside and at the ends of a warp, and that take more than one
round of the grid: loss and gradient, which hold every leaf's range, against
the fp64 oracle (tolerances as in test_cdf_gpu.py)."""
import numpy as np
import pytest

import cdf_oracle
from test_cdf_gpu import gpu_loss_grad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 33, 1000, 1024, 4097, 1_300_001])
@pytest.mark.parametrize("leaves", [1, 7, 1024])
def test_leaf_ranges(ctx, torch_cuda, n, leaves):
    rng = np.random.default_rng(n + leaves)
    keys = np.sort(rng.integers(0, 1 << 40, n))
    keys[-1] = keys[0] + (1 << 40)
    lo, sc = float(keys[0]), 1.0 / float(1 << 40)
    # The root line leaves both ends to clamping.
    p = np.concatenate([[1.1, -0.05], np.tile([0.8, 0.1], leaves)]).astype(np.float32)
    l_gpu, g_gpu = gpu_loss_grad(ctx, torch_cuda, keys, leaves, p, lo, sc)
    l_cpu, g_cpu = cdf_oracle.loss_grad(keys, leaves, p, lo, sc)
    assert abs(l_gpu - l_cpu) <= 1e-9 + 1e-6 * abs(l_cpu)
    np.testing.assert_allclose(g_gpu, g_cpu, rtol=1e-4, atol=1e-7)
