"""Queued fragments with an empty build side and probe tuples: nothing joins,
whatever their tables' memory held before (here, earlier tables that held the
probed keys).  Few items, so that clears and probes run at the same time."""
import numpy as np
import pytest

import pyg

pytestmark = pytest.mark.gpu


def test_empty_builds_join_nothing(ctx, torch_cuda):
    torch = torch_cuda
    n, frags = 4096, 48
    keys = [torch.randperm(n, device="cuda") + 17 * i for i in range(frags)]
    R = [torch.stack([k, k], 1).contiguous() for k in keys]
    full = ctx.fragments([(r, n, r, n) for r in R])
    empty = ctx.fragments([(r, 0, r, n - i) for i, r in enumerate(R)])
    mixed = ctx.fragments([(r, 0 if i % 2 else n, r, n) for i, r in enumerate(R)])
    sums = np.array([2 * int(k.sum()) for k in keys])
    odd = np.arange(frags) % 2 == 1
    for _ in range(4):
        for fr, want in ((full, np.zeros(frags, bool)), (empty, np.ones(frags, bool)), (mixed, odd)):
            b = ctx.batch_create(fr)
            try:
                for _ in range(3):
                    rc, c, s, _ = ctx.batch_run(b, frags)
                    assert rc == 0
                    assert np.array_equal(c, np.where(want, 0, n)) and np.array_equal(s, np.where(want, 0, sums))
            finally:
                ctx.batch_free(b)
