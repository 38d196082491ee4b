"""General hash tables of 16-byte tuples: small relations take a thread per
tuple (up to 2048 per SM), larger ones four tuples per thread."""
import time

import numpy as np
import pytest

import pyg
from util import I64

pytestmark = pytest.mark.gpu
BOTH = [(0, 1), (1, 1)]
KEMPTY = -(1 << 63)


def wrap(x):
    return (int(x) + (1 << 63)) % (1 << 64) - (1 << 63)


def limit(torch):
    return torch.cuda.get_device_properties(0).multi_processor_count * 2048


@pytest.mark.parametrize("nS", [1, 31, 32, 255, 256, 257, 1025, 70_001, "limit", "limit+1"])
@pytest.mark.parametrize("nR", [1, 300, "limit", "limit+1"])
@pytest.mark.parametrize("markers", [0, 3])
def test_rows_of_small_relations(ctx, torch_cuda, nR, nS, markers):
    torch = torch_cuda
    nR, nS = (limit(torch) + x.endswith("+1") if isinstance(x, str) else x for x in (nR, nS))
    rng = np.random.default_rng(nR + nS)
    k = rng.permutation(nR).astype(np.int64) * 5 + 1
    if markers and nR > markers:
        k[:1] = KEMPTY
    f = np.where(rng.random(nS) < 0.7, k[rng.integers(0, nR, nS)], 2)
    f[: min(markers, nS)] = KEMPTY
    R = torch.from_numpy(np.stack([k, k ^ 77], 1)).cuda()
    S = torch.from_numpy(np.stack([f, np.arange(nS)], 1)).cuda()
    Rr, Sr = pyg.Rel(R, nR, [I64, I64]), pyg.Rel(S, nS, [I64, I64])
    hit = np.isin(f, k)
    want = np.stack([f[hit] ^ 77, np.arange(nS)[hit]], 1)
    rows = torch.empty(max(1, nS), 2, dtype=torch.int64, device="cuda")
    ht = ctx.hashjoin_build(Rr, [0], [1], pyg.HT_MATERIALIZE, 0.5)
    rc, c = ctx.hashjoin_probe_materialize(ht, Sr, [0], BOTH, rows, nS)
    ht.free()
    got = rows[:c].cpu().numpy()
    assert rc == 0 and c == len(want) and np.array_equal(got[np.argsort(got[:, 1])], want)
    ht = ctx.hashjoin_build(Rr, [0], [1], pyg.HT_AGGREGATE, 0.5)
    count, sums = ctx.hashjoin_probe_agg(ht, Sr, [0], BOTH)
    ht.free()
    assert count == len(want) and [wrap(x) for x in sums] == [wrap(v) for v in want.sum(0)]


def test_rows_of_a_small_join_take_no_longer_than_by_the_general_kernels(ctx, torch_cuda):
    """5000 x 70000 random keys, eight of them.  24-byte tuples take the
    general kernels, one tuple per thread."""
    torch = torch_cuda
    nR, nS = 5000, 70_000
    total = {2: 0.0, 3: 0.0}
    rows = torch.empty(nS, 2, dtype=torch.int64, device="cuda")
    for seed in range(8):
        gen = torch.Generator(device="cuda").manual_seed(seed)
        k = torch.unique(torch.randint(-(1 << 62), 1 << 62, (nR + 9,), device="cuda", generator=gen))
        k = k[torch.randperm(k.numel(), device="cuda", generator=gen)[:nR]]
        f = k[torch.randint(0, nR, (nS,), device="cuda", generator=gen)]
        for cols in (2, 3):
            R, S = (pyg.Rel(torch.stack([x] * cols, 1).contiguous(), len(x), [I64] * cols) for x in (k, f))
            times = []
            for _ in range(20):
                torch.cuda.synchronize()
                t = time.perf_counter()
                ht = ctx.hashjoin_build(R, [0], [1], pyg.HT_MATERIALIZE, 0.5)
                rc, c = ctx.hashjoin_probe_materialize(ht, S, [0], BOTH, rows, nS)
                times.append(time.perf_counter() - t)
                ht.free()
                assert rc == 0 and c == nS
            total[cols] += min(times)
    assert total[2] < 1.06 * total[3], total
