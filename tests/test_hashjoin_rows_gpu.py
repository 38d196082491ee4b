"""The materialising probe of 16-byte tuples (one row per probe tuple at
most): tile edges, keys that miss, the INT64_MIN marker on both sides, repeated
build keys (which take the general probe), payloads of either width and
projections other than {build payload, probe value}."""
import numpy as np
import pytest

import pyg
from util import I32, I64, alloc, dev_rel, from_device, struct

pytestmark = pytest.mark.gpu
MIN64 = -(1 << 63)


def rows_of(ctx, torch, R, rt, S, st, proj, dtype):
    ht = ctx.hashjoin_build(dev_rel(torch, R, rt), [0], [1], pyg.HT_MATERIALIZE, 0.5)
    out = alloc(torch, (4 * len(S) + 64) * dtype.itemsize)
    rc, n = ctx.hashjoin_probe_materialize(ht, dev_rel(torch, S, st), [0], proj, out, 4 * len(S) + 64)
    ht.free()
    assert rc == 0
    return np.sort(from_device(torch, out, n, dtype))


def expect(R, S, proj, dtype):
    by = {}
    for i, k in enumerate(R["c0"].tolist()):
        by.setdefault(k, []).append(i)
    rows = [tuple((S[j] if side else R[i])[f"c{c}"] for side, c in proj)
            for j, k in enumerate(S["c0"].tolist()) for i in by.get(k, [])]
    return np.sort(np.array(rows, dtype=dtype))


@pytest.mark.parametrize("m", [1, 255, 1023, 1024, 1025, 9001])
@pytest.mark.parametrize("extra", ["none", "marker", "dups"])
def test_rows(ctx, torch_cuda, m, extra):
    rng = np.random.default_rng(m)
    n = 3000
    k = rng.permutation(n).astype(np.int64) - 500
    f = rng.integers(-700, n, m)
    if extra == "marker":
        k[:3] = MIN64
        f[: max(1, m // 50)] = MIN64
    if extra == "dups":
        k[:3] = k[10]
    R, S = struct([k, k * 7 + 1], [I64, I64]), struct([f, np.arange(m, dtype=np.int64)], [I64, I64])
    dt = np.dtype([("a", np.int64), ("b", np.int64)])
    assert np.array_equal(rows_of(ctx, torch_cuda, R, [I64, I64], S, [I64, I64], [(0, 1), (1, 1)], dt),
                          expect(R, S, [(0, 1), (1, 1)], dt))


def test_rows_other_projections(ctx, torch_cuda):
    rng = np.random.default_rng(5)
    n, m = 2000, 5003
    k = rng.permutation(n).astype(np.int64)
    R = struct([k, np.arange(n, dtype=np.int32) - 900, np.arange(n, dtype=np.int32)], [I64, I32, I32])
    S = struct([rng.integers(0, n + 200, m), np.arange(m, dtype=np.int32), -np.arange(m, dtype=np.int32)],
               [I64, I32, I32])
    proj = [(1, 2), (0, 1), (1, 0), (1, 1)]
    dt = np.dtype([("a", np.int32), ("b", np.int32), ("c", np.int64), ("d", np.int32)])
    assert np.array_equal(rows_of(ctx, torch_cuda, R, [I64, I32, I32], S, [I64, I32, I32], proj, dt),
                          expect(R, S, proj, dt))
