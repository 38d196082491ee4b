"""Narrow key ranges far from zero, where neighbouring int64 keys are one
double: the learned model has no scale then (or a coarse one) and must still
give ordered bins, a usable distinct estimate and the right join."""
import numpy as np
import pytest

import pyg
from test_cdf_gpu import model_bin_splitters, model_bins, splitters, train
from util import I64

pytestmark = pytest.mark.gpu
MIN64, MAX64 = -(1 << 63), (1 << 63) - 1
BASES = [MIN64, MAX64 - 4999, 1 << 60, -(1 << 62) - 3]


@pytest.mark.parametrize("base", BASES)
@pytest.mark.parametrize("width", [2, 100, 5000])
def test_bins_and_splitters(ctx, torch_cuda, base, width):
    rng = np.random.default_rng(width)
    keys = base + rng.integers(0, width, 20_000)
    keys[:2] = base, base + width - 1
    m = train(ctx, torch_cuda, keys, leaves=64, epochs=2)
    try:
        probe = np.unique(np.concatenate([keys, np.array([MIN64, base, base + width - 1, MAX64, 0])]))
        sp = model_bin_splitters(ctx, m, 7)
        got = model_bins(ctx, torch_cuda, m, 7, probe)
        assert np.all(np.diff(sp) >= 0) and np.array_equal(got, np.searchsorted(sp, probe, side="right"))
        assert np.all(np.diff(splitters(ctx, m, 50)) >= 0)
    finally:
        pyg.lib().pyg_cdf_free(ctx.h, m)


@pytest.mark.parametrize("base", BASES)
@pytest.mark.parametrize("width", [100, 5000])
def test_groupby_without_an_estimate(ctx, torch_cuda, base, width):
    torch = torch_cuda
    n = (1 << 20) + 7
    ids = torch.randint(0, width, (n,), device="cuda")
    A = torch.stack([ids + base, torch.ones_like(ids)], 1).contiguous()
    out = torch.empty(width, 3, dtype=torch.int64, device="cuda")
    rc, g = ctx.groupby(pyg.Rel(A, n, [I64, I64]), [0], 3, 1, True, 0, out, width)
    assert rc == 0 and g == width
    assert torch.equal(out[:, 0], torch.arange(width, device="cuda") + base)
    assert torch.equal(out[:, 2], torch.bincount(ids, minlength=width)) and torch.equal(out[:, 1], out[:, 2])


@pytest.mark.parametrize("base", BASES)
@pytest.mark.parametrize("width", [100, 5000])
def test_learned_merge_join(ctx, torch_cuda, base, width):
    torch = torch_cuda
    n = 300_000
    k = torch.randperm(width, device="cuda")
    R = torch.stack([k + base, k], 1).contiguous()
    f = torch.randint(0, width + 50, (n,), device="cuda")
    f = torch.where(f >= width, 0, f) if base > MAX64 - (1 << 20) else f
    S = torch.stack([f + base, torch.arange(n, device="cuda")], 1).contiguous()
    hit = f < width
    got, sums, _ = ctx.mpsm_join_agg(pyg.Rel(R, width, [I64, I64]), 0, pyg.Rel(S, n, [I64, I64]), 0, [(0, 1), (1, 1)],
                                     ctx.mpsm_opts(pyg.MPSM_LEARNED))
    assert got == int(hit.sum())
    assert [int(x) for x in sums] == [int(f[hit].sum()), int(torch.arange(n, device="cuda")[hit].sum())]
