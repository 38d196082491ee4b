"""Layouts taken from a sample of the rows: keys that repeat with the row
number must reach the sample like any others, so that no region overflows and
the relation is partitioned once."""
import pytest

import pyg
from util import I64

pytestmark = pytest.mark.gpu
N = 1 << 25  # sampled layouts begin here


@pytest.mark.parametrize("period,bits", [(1 << 16, 7), (1 << 12, 7), (50_000, 7), (257, 7),
                                         (1 << 16, 9), (1 << 12, 9),    # one pass
                                         (1 << 20, 12), (257, 12)])     # two passes
def test_keys_periodic_in_the_row_number(ctx, torch_cuda, period, bits):
    torch = torch_cuda
    k = torch.arange(period, device="cuda")
    R = torch.stack([k, k * 7], 1).contiguous()
    S = torch.empty(N, 2, dtype=torch.int64, device="cuda")
    S[:, 0] = torch.arange(N, device="cuda") % period
    S[:, 1] = 1
    (got, sums), st = ctx.hashjoin_agg(pyg.Rel(R, period, [I64, I64]), [0], pyg.Rel(S, N, [I64, I64]), [0],
                                       [(0, 1), (1, 1)], pyg.JOIN_RADIX, bits, stats=True)
    assert got == N and [int(x) for x in sums] == [int((S[:, 0] * 7).sum()), N]
    assert st.histogram_tuples < N // 4 and st.overflow_tuples == 0
