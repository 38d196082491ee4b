"""The shared-memory group-by fold where its pieces meet: sums that carry
between their 32-bit halves and are negative, the empty markers of the
tables as keys, frequent keys held in registers, packed and 16-byte
partitions, (int32, int32) keys, and group estimates far below the truth.
Expected values: NumPy over the same tuples, modulo 2^64."""
import numpy as np
import pytest

import pyg
from util import I32, I64, alloc, dev_rel, from_device, struct

pytestmark = pytest.mark.gpu
MIN64, MIN32 = -(1 << 63), -(1 << 31)


def expect(keys, vals):
    """(unique rows of keys in order, sums, counts); keys (n, k) int64."""
    u, inv, cnt = np.unique(keys, axis=0, return_inverse=True, return_counts=True)
    s = np.zeros(len(u), dtype=np.uint64)
    np.add.at(s, inv.reshape(-1), vals.astype(np.uint64))
    return u, s.view(np.int64), cnt


VALUES = {
    "small": lambda r, n: r.integers(0, 1 << 20, n),
    "signed": lambda r, n: r.integers(-(1 << 40), 1 << 40, n),
    "wide": lambda r, n: r.integers(MIN64, (1 << 63) - 1, n, dtype=np.int64, endpoint=True),
    "carry": lambda r, n: np.full(n, 0xFFFFFFFF, dtype=np.int64),
}


@pytest.mark.parametrize("vals", sorted(VALUES))
@pytest.mark.parametrize("groups,hint", [(12, 12), (60, 64), (900, 900), (5000, 5000), (5000, 10), (70000, 4000)])
@pytest.mark.parametrize("low", [0, MIN64])  # key frames: from 0, and from INT64_MIN (the tables' marker)
def test_fold_int64(ctx, torch_cuda, vals, groups, hint, low):
    rng = np.random.default_rng(groups + hint)
    n = 300_007
    ids = rng.integers(0, groups, n)
    ids[rng.random(n) < 0.4] = groups // 2  # one frequent key
    k = ids + np.int64(low)
    v = VALUES[vals](rng, n)
    A = struct([k, v], [I64, I64])
    out = alloc(torch_cuda, 24 * (groups + 1))
    rc, g = ctx.groupby(dev_rel(torch_cuda, A, [I64, I64]), [0], 3, 1, True, hint, out, groups + 1)
    u, s, c = expect(k[:, None], v)
    assert rc == 0 and g == len(u)
    got = from_device(torch_cuda, out, g, np.dtype([("k", np.int64), ("s", np.int64), ("c", np.int64)]))
    assert np.array_equal(got["k"], u[:, 0]) and np.array_equal(got["s"], s) and np.array_equal(got["c"], c)


@pytest.mark.parametrize("groups,hint", [(40, 64), (2000, 2000), (20000, 20000), (20000, 100)])
@pytest.mark.parametrize("n", [1000, 300_007, (1 << 22) + 3])
def test_fold_int32_pair(ctx, torch_cuda, groups, hint, n):
    rng = np.random.default_rng(groups + n)
    ids = rng.integers(0, groups, n)
    a = (ids // 7 - groups // 14).astype(np.int32)
    b = (ids % 7 - 3).astype(np.int32)
    a[:2], b[:2] = (MIN32, 0), (0, MIN32)  # the marker as a key word, and its mirror image
    v = rng.integers(-1000, 1 << 34, n)
    A = struct([a, b, v], [I32, I32, I64])
    out = alloc(torch_cuda, 24 * (groups + 2))
    rc, g = ctx.groupby(dev_rel(torch_cuda, A, [I32, I32, I64]), [0, 1], 3, 2, True, hint, out, groups + 2)
    u, s, c = expect(np.stack([a, b], 1).astype(np.int64), v)
    assert rc == 0 and g == len(u)
    got = from_device(torch_cuda, out, g, np.dtype([("a", np.int32), ("b", np.int32), ("s", np.int64), ("c", np.int64)]))
    assert np.array_equal(got["a"], u[:, 0]) and np.array_equal(got["b"], u[:, 1])
    assert np.array_equal(got["s"], s) and np.array_equal(got["c"], c)


def test_fold_sampled_single_pass_skew(ctx, torch_cuda):
    """2^25 tuples and more sample their layout, also with one pass; ids that
    the strided sample misjudges overflow their region and are redone."""
    torch = torch_cuda
    n, G = (1 << 25) + 4096, 6000
    ids = torch.arange(n, device="cuda") % G
    ids[::7] = 17
    ids[: n // 3] = torch.arange(n // 3, device="cuda") // 64 % G  # runs: a strided sample sees few of each
    A = torch.stack([ids, torch.full_like(ids, 3)], 1).contiguous()
    out = torch.empty(G, 3, dtype=torch.int64, device="cuda")
    rc, g = ctx.groupby(pyg.Rel(A, n, [I64, I64]), [0], 3, 1, True, G, out, G)
    cnt = torch.bincount(ids, minlength=G)
    assert rc == 0 and g == G
    assert bool((out[:, 0] == torch.arange(G, device="cuda")).all())
    assert bool((out[:, 2] == cnt).all()) and bool((out[:, 1] == cnt * 3).all())
