"""Packed words keep 32-bit key offsets, and the offset 2^32 - 1 marks a free
table slot, so a key there must leave the packed form.  An exact frame never
gives that offset to a key; a frame taken from a sample does when one of the
tuples between the samples lies 2^32 - 1 above its base: the relation is then
redone, and the key is a group, or an unmatched probe key, like any other."""
import pytest

import pyg
from util import I64

pytestmark = pytest.mark.gpu
N, G = 1 << 25, 4000  # sampled layouts begin at 2^25 tuples
# Sampled keys span [0, G - 1]; the frame is centred on them.
BASE = -((0xFFFFFFFE - (G - 1)) // 2)
MARKER = BASE + 0xFFFFFFFF
ROWS = [12_345_677, N - 2]  # rows that the sample of one in 256 does not read


def relation(torch, key, row):
    gen = torch.Generator(device="cuda").manual_seed(row)
    A = torch.empty(N, 2, dtype=torch.int64, device="cuda")
    A[:, 0] = torch.randint(0, G, (N,), device="cuda", generator=gen)
    A[:, 1] = torch.randint(0, 1000, (N,), device="cuda", generator=gen)
    A[row, 0] = key
    return A


@pytest.mark.parametrize("row", ROWS)
@pytest.mark.parametrize("key", [MARKER - 1, MARKER, MARKER + 1, BASE, BASE - 1])
def test_groupby_key_at_the_marker(ctx, torch_cuda, key, row):
    torch = torch_cuda
    A = relation(torch, key, row)
    ids = A[:, 0].clone()
    ids[row] = G
    cnt = torch.bincount(ids, minlength=G + 1)
    tot = torch.zeros(G + 1, dtype=torch.int64, device="cuda").index_add_(0, ids, A[:, 1])
    keys = torch.arange(G + 1, device="cuda")
    keys[G] = key
    order = torch.argsort(keys)
    out = torch.empty(G + 1, 3, dtype=torch.int64, device="cuda")
    rc, g = ctx.groupby(pyg.Rel(A, N, [I64, I64]), [0], 3, 1, True, G + 1, out, G + 1)
    assert rc == 0 and g == G + 1
    assert torch.equal(out, torch.stack([keys, tot, cnt], 1)[order])


@pytest.mark.parametrize("row", ROWS)
@pytest.mark.parametrize("bits", [7, 12])  # one pass, two passes
@pytest.mark.parametrize("key", [MARKER - 1, MARKER, MARKER + 1])
def test_probe_key_at_the_marker(ctx, torch_cuda, key, bits, row):
    torch = torch_cuda
    S = relation(torch, key, row)
    k = torch.arange(G, device="cuda")
    R = torch.stack([k, k * 7], 1).contiguous()
    hit = S[:, 0] != key
    want = (N - 1, [int((S[hit, 0] * 7).sum()), int(S[hit, 1].sum())])
    got = ctx.hashjoin_agg(pyg.Rel(R, G, [I64, I64]), [0], pyg.Rel(S, N, [I64, I64]), [0], [(0, 1), (1, 1)],
                           pyg.JOIN_RADIX, bits)
    assert (got[0], [int(x) for x in got[1]]) == want
