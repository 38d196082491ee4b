"""The partition passes at the edges of their tiles: one tuple to a few past
a tile of either pass, small tiles for small relations, one and two passes,
and keys of which none, some or all share one bin (the combined ranking).
Checked through the radix join against closed forms: unique build keys with
payload 7 x key, every probe key present."""
import numpy as np
import pytest

import pyg
from util import I64, dev_rel, struct

pytestmark = pytest.mark.gpu


def relations(nR, nS, hot, base, seed):
    rng = np.random.default_rng(seed)
    k = rng.permutation(nR).astype(np.int64) + base
    fk = k[rng.integers(0, nR, nS)]
    if hot:
        fk[rng.random(nS) < hot] = k[0]
    v = rng.integers(0, 1000, nS)
    return struct([k, k * 7], [I64, I64]), struct([fk, v], [I64, I64]), int((fk * 7).sum()), int(v.sum())


@pytest.mark.parametrize("bits", [1, 7, 9, 10, 13])
@pytest.mark.parametrize("hot", [0.0, 0.3, 1.0])
@pytest.mark.parametrize("nS", [1, 1023, 1025, 7937, 296 * 1024 - 1, 296 * 7936 + 5])
def test_tile_edges(ctx, torch_cuda, bits, hot, nS):
    R, S, sb, sp = relations(5000, nS, hot, 1, nS + bits)
    got = ctx.hashjoin_agg(dev_rel(torch_cuda, R, [I64, I64]), [0], dev_rel(torch_cuda, S, [I64, I64]), [0],
                           [(0, 1), (1, 1)], pyg.JOIN_RADIX, bits)
    assert got == (nS, [sb, sp])


@pytest.mark.parametrize("bits", [9, 12])
@pytest.mark.parametrize("nS", [2401, 300001])
def test_unpacked_tile_edges(ctx, torch_cuda, bits, nS):
    """Probe values spread over 2^40 do not fit a packed frame: 16-byte
    intermediates on the probe side."""
    R, S, sb, _ = relations(5000, nS, 0.0, 1, nS)
    S["c1"] = np.arange(nS, dtype=np.int64) << 20
    got = ctx.hashjoin_agg(dev_rel(torch_cuda, R, [I64, I64]), [0], dev_rel(torch_cuda, S, [I64, I64]), [0],
                           [(0, 1), (1, 1)], pyg.JOIN_RADIX, bits)
    assert got == (nS, [sb, int(S["c1"].sum())])


@pytest.mark.parametrize("dup", [False, True])
def test_items_beyond_the_device_list(ctx, torch_cuda, dup):
    """Two partitions cut into many chunks on both sides need more work items
    than the device forms: the host does."""
    n = 2_000_003
    R, S, sb, sp = relations(n, n, 0.0, 5, 11)
    if dup:  # one build key twice
        R["c0"][7] = R["c0"][8]
        hit = S["c0"] == R["c0"][8]
        lost = S["c0"] == R["c1"][7] // 7
        sb = int((S["c0"][~lost] * 7).sum() + hit.sum() * int(R["c1"][7]))
        sp = int(S["c1"][~lost].sum() + S["c1"][hit].sum())
        n += int(hit.sum()) - int(lost.sum())
    got = ctx.hashjoin_agg(dev_rel(torch_cuda, R, [I64, I64]), [0], dev_rel(torch_cuda, S, [I64, I64]), [0],
                           [(0, 1), (1, 1)], pyg.JOIN_RADIX, 1)
    assert got == (n, [sb, sp])
