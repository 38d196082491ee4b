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
