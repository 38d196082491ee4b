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


@pytest.mark.parametrize("n", [1, 63, 64, 65, 3583, 3584, 3585, 6143, 6144])
@pytest.mark.parametrize("kind", ["dense", "random", "high", "marker"])
def test_slot_counts(ctx, torch_cuda, n, kind):
    """Four slots per build tuple, at least 256 and at most 14336; chains that
    wrap around the table's end; probes that miss."""
    torch = torch_cuda
    gen = torch.Generator(device="cuda").manual_seed(n)
    i = torch.randperm(n, device="cuda", generator=gen)
    k = {"dense": i, "random": torch.randint(-(1 << 62), 1 << 62, (n,), device="cuda", generator=gen) * 2, "high": i << 32,
         "marker": i - (1 << 63)}[kind]
    m = 50_001
    f = k[torch.randint(0, n, (m,), device="cuda", generator=gen)]
    miss = torch.rand(m, device="cuda", generator=gen) < 0.5
    f = torch.where(miss, f + (1 if kind == "random" else 1 << 20), f)
    v = torch.arange(m, device="cuda")
    R, S = torch.stack([k, k * 3], 1).contiguous(), torch.stack([f, v], 1).contiguous()
    got, sums = ctx.hashjoin_agg(pyg.Rel(R, n, [I64, I64]), [0], pyg.Rel(S, m, [I64, I64]), [0], [(0, 1), (1, 1)],
                                 pyg.JOIN_DIRECT)
    hit = torch.isin(f, k)
    assert torch.unique(k).numel() == n
    assert got == int(hit.sum()) and [int(x) for x in sums] == [int((f[hit] * 3).sum()), int(v[hit].sum())]
