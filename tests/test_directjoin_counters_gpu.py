"""The direct join's counters come from the last CTA of its probe: one CTA, as
many as the grid holds and one tile more, the build's flags (repeated keys, a
side list past its 1024 entries) as well as the sums, and calls one after
another, each with its own ticket.  Whole numbers, so results are identical."""
import numpy as np
import pytest

import pyg
from util import I64, dev_rel, struct

pytestmark = pytest.mark.gpu
MIN64 = -(1 << 63)


@pytest.mark.parametrize("nR", [6145, 1 << 16])
@pytest.mark.parametrize("nS", [0, 1, 1024, 1025, 148 * 8 * 1024, 148 * 8 * 1024 + 1])
@pytest.mark.parametrize("extra", ["none", "dup", "side", "side_full"])
def test_counters_of_consecutive_joins(ctx, torch_cuda, nR, nS, extra):
    rng = np.random.default_rng(nR + nS)
    k = rng.permutation(2 * nR)[:nR].astype(np.int64)
    f = rng.integers(0, 2 * nR, nS)
    if extra == "dup":
        k[-1] = k[0]
    if extra.startswith("side"):
        k[: 1024 if extra == "side" else 1025] = MIN64
        f[::9] = MIN64
    p, v = rng.integers(-(1 << 50), 1 << 50, nR), rng.integers(-(1 << 30), 1 << 30, nS)
    u, inv, cnt = np.unique(k, return_inverse=True, return_counts=True)
    ps = np.zeros(len(u), dtype=np.int64)
    np.add.at(ps, inv, p)
    at = np.minimum(np.searchsorted(u, f), len(u) - 1)
    hit = u[at] == f
    at, vv = at[hit], v[hit]
    want = (int(cnt[at].sum()), [int(ps[at].sum()), int((cnt[at] * vv).sum())])
    R, S = dev_rel(torch_cuda, struct([k, p], [I64, I64]), [I64, I64]), dev_rel(torch_cuda, struct([f, v], [I64, I64]), [I64, I64])
    for _ in range(3):
        got = ctx.hashjoin_agg(R, [0], S, [0], [(0, 1), (1, 1)], pyg.JOIN_DIRECT, 0, 0.5)
        if nS == 0:
            assert got[0] == 0
        else:
            assert (got[0], [int(x) for x in got[1]]) == want
