"""The materialising sort-merge join at its edges: tiles of 1024 probe items,
build ranges that fit shared memory and that do not, repeated keys on either
side, int64 extremes, projections of the key, one column and several (row
gather), and outputs cut at their capacity.  Expected rows by NumPy: ordered
by key, probe row, build row."""
import numpy as np
import pytest

import pyg
from util import I32, I64, alloc, dev_rel, from_device, struct

pytestmark = pytest.mark.gpu


def expect(R, S, proj):
    ro, so = np.argsort(R["c0"], kind="stable"), np.argsort(S["c0"], kind="stable")
    rk, sk = R["c0"][ro], S["c0"][so]
    lo, hi = np.searchsorted(rk, sk, "left"), np.searchsorted(rk, sk, "right")
    c = hi - lo
    s = np.repeat(so, c)
    first = np.repeat(lo - (np.cumsum(c) - c), c)
    r = ro[first + np.arange(c.sum())]
    return [(S if side else R)[f"c{col}"][s if side else r] for side, col in proj]


def check(ctx, torch, R, S, rt, st, proj, cap=None, kind=pyg.MPSM_SAMPLED):
    want = expect(R, S, proj)
    n = len(want[0])
    cap = n if cap is None else cap
    dt = np.dtype([(f"p{i}", w.dtype) for i, w in enumerate(want)])
    out = alloc(torch, max(cap, 1) * dt.itemsize + 64)
    rc, got = ctx.mpsm_join_materialize(dev_rel(torch, R, rt), 0, dev_rel(torch, S, st), 0, proj,
                                        ctx.mpsm_opts(kind, 64, 0.05, 64), out, cap)
    assert got == n and (rc == 0) == (n <= cap)
    m = min(n, cap)
    rows = from_device(torch, out, m, dt)
    for i, w in enumerate(want):
        assert np.array_equal(rows[f"p{i}"], w[:m])
    assert not out[m * dt.itemsize:].any()  # nothing past the rows


def keys(kind, rng, n, m):
    if kind == "pk":
        return rng.permutation(n).astype(np.int64), rng.integers(-5, n + 5, m)
    if kind == "dups":
        return rng.integers(0, max(n // 3, 1), n), rng.integers(0, max(n // 3, 1), m)
    if kind == "sparse":  # few probe keys over a wide build range: the range does not fit a tile
        return rng.permutation(n).astype(np.int64) * 1000, rng.integers(0, n, m) * 1000
    if kind == "hot":  # one key with many rows on both sides
        k, f = rng.integers(0, n, n), rng.integers(0, n, m)
        k[: min(n, 700)] = 3
        f[: min(m, 90)] = 3
        return k, f
    ends = np.array([-(1 << 63), (1 << 63) - 1, 0, -1], dtype=np.int64)
    return rng.choice(ends, n), rng.choice(ends, min(m, 60))


@pytest.mark.parametrize("kind", ["pk", "dups", "sparse", "hot", "ends"])
@pytest.mark.parametrize("n,m", [(1, 1), (50, 1023), (50, 2047), (4096, 2049), (4097, 4097), (60000, 9000)])
def test_rows(ctx, torch_cuda, kind, n, m):
    rng = np.random.default_rng(n + m)
    if kind == "ends":
        n = min(n, 300)
    k, f = keys(kind, rng, n, m)
    R = struct([k, np.arange(n) * 7], [I64, I64])
    S = struct([f, rng.integers(0, 1 << 40, len(f))], [I64, I64])
    check(ctx, torch_cuda, R, S, [I64, I64], [I64, I64], [(0, 1), (1, 1)])
    check(ctx, torch_cuda, R, S, [I64, I64], [I64, I64], [(1, 0), (0, 0), (1, 1)], kind=pyg.MPSM_LEARNED)


@pytest.mark.parametrize("cap", [0, 1, 2500, 5999])
def test_rows_cut_at_capacity(ctx, torch_cuda, cap):
    rng = np.random.default_rng(cap)
    R = struct([rng.permutation(5000).astype(np.int64), np.arange(5000)], [I64, I64])
    S = struct([rng.integers(0, 5000, 6000), np.arange(6000)], [I64, I64])
    check(ctx, torch_cuda, R, S, [I64, I64], [I64, I64], [(0, 1), (1, 1)], cap=cap)


def test_rows_several_columns(ctx, torch_cuda):
    """Two value columns per side: the items carry row numbers; int32 keys."""
    rng = np.random.default_rng(8)
    n, m = 6000, 9000
    R = struct([rng.integers(-2000, 2000, n).astype(np.int32), np.arange(n, dtype=np.int32), np.arange(n) * 3],
               [I32, I32, I64])
    S = struct([rng.integers(-2500, 2500, m).astype(np.int32), np.arange(m) * 5, np.arange(m, dtype=np.int32)],
               [I32, I64, I32])
    proj = [(0, 2), (1, 1), (0, 1), (1, 2), (0, 0)]
    check(ctx, torch_cuda, R, S, [I32, I32, I64], [I32, I64, I32], proj)
