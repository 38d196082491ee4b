"""The one-launch join of small build sides: sizes around its limit and around
one CTA's and all CTAs' tuples, misses, the INT64_MIN marker on both sides, and
repeated build keys (which the general path answers)."""
import numpy as np
import pytest

import pyg
from util import I64, dev_rel, struct

pytestmark = pytest.mark.gpu
MIN64 = -(1 << 63)


@pytest.mark.parametrize("nR", [1, 255, 1024, 1025, 6143, 6144, 6145])
@pytest.mark.parametrize("nS", [1, 1023, 1025, 148 * 1024 + 1, 148 * 4096 + 17])
@pytest.mark.parametrize("extra", ["none", "marker", "dup"])
def test_small_join(ctx, torch_cuda, nR, nS, extra):
    rng = np.random.default_rng(nR + nS)
    k = rng.permutation(2 * nR)[:nR].astype(np.int64) * 3 - nR
    f = rng.integers(-nR - 5, 6 * nR, nS)
    if extra == "marker":
        k[: min(nR, 3)] = MIN64
        f[::7] = MIN64
    if extra == "dup":
        k[-1] = k[0]
    p, v = rng.integers(-(1 << 50), 1 << 50, nR), rng.integers(-(1 << 50), 1 << 50, nS)
    u, inv, cnt = np.unique(k, return_inverse=True, return_counts=True)
    ps = np.zeros(len(u), dtype=np.int64)
    np.add.at(ps, inv, p)
    at = np.minimum(np.searchsorted(u, f), len(u) - 1)
    hit = u[at] == f
    at, vv = at[hit], v[hit]
    want = (int(cnt[at].sum()), [int(ps[at].sum()), int((cnt[at] * vv).sum())])
    R, S = struct([k, p], [I64, I64]), struct([f, v], [I64, I64])
    got = ctx.hashjoin_agg(dev_rel(torch_cuda, R, [I64, I64]), [0], dev_rel(torch_cuda, S, [I64, I64]), [0],
                           [(0, 1), (1, 1)])
    assert got == want
