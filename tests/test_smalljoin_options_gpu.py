"""Load factors of the one-launch join of small build sides: those of a table
are taken, one that no table accepts is refused as it is for larger builds."""
import pytest

import pyg
from util import I64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4096, 6144, 8192])
@pytest.mark.parametrize("lf", [0.0, 0.1, 0.5, 0.95, 4.0])
def test_load_factor(ctx, torch_cuda, n, lf):
    torch = torch_cuda
    k = torch.arange(n, device="cuda")
    R = torch.stack([k, k * 3], 1).contiguous()
    rel = pyg.Rel(R, n, [I64, I64])
    args = (rel, [0], rel, [0], [(0, 1), (1, 1)], pyg.JOIN_DIRECT, 0, lf)
    if lf > 1:
        with pytest.raises(pyg.PygError) as e:
            ctx.hashjoin_agg(*args)
        assert e.value.code == pyg.PYG_ERR_ARG
    else:
        got, sums = ctx.hashjoin_agg(*args)
        assert got == n and [int(x) for x in sums] == [3 * n * (n - 1) // 2] * 2
