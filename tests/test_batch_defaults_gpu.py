"""The default plan of a batch: smaller work items for little work, and large
fragments with many probes as their own joins."""
import time

import pytest

import pyg

pytestmark = pytest.mark.gpu


def fragments(torch, sizes, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    pairs, want = [], []
    for nb, np_ in sizes:
        k = torch.unique(torch.randint(0, 1 << 31, (nb + nb // 2 + 64,), device="cuda", generator=gen))
        k = k[torch.randperm(k.numel(), device="cuda", generator=gen)[:nb]]
        i = torch.randint(0, nb, (np_,), device="cuda", generator=gen)
        pairs.append((torch.stack([k, k], 1).contiguous(), nb,
                      torch.stack([k[i], torch.arange(np_, device="cuda")], 1).contiguous(), np_))
        want.append((np_, int(k[i].sum()) + np_ * (np_ - 1) // 2))
    return pairs, want


def best_run(ctx, torch, pairs, want, tuning=None):
    b = ctx.batch_create(ctx.fragments(pairs), tuning)
    times = []
    try:
        for _ in range(10):
            torch.cuda.synchronize()
            t = time.perf_counter()
            rc, c, s, _ = ctx.batch_run(b, len(pairs))
            times.append(time.perf_counter() - t)
            assert rc == 0 and [(int(x), int(y)) for x, y in zip(c, s)] == want
    finally:
        ctx.batch_free(b)
    return min(times)


@pytest.mark.parametrize("sizes", [[(1, 1)], [(511, 513)], [(512, 512), (513, 1)], [(4000, 40_000)],
                                   [(1023 + 64 * i, 2047 * (i + 1)) for i in range(40)],
                                   [(20_000, 150_000 + i) for i in range(90)]])
def test_items_of_every_grain(ctx, torch_cuda, sizes):
    pairs, want = fragments(torch_cuda, sizes, len(sizes))
    best_run(ctx, torch_cuda, pairs, want)


@pytest.mark.parametrize("sizes", [[(4000, 40_000)], [(20_000, 200_000)] * 2, [(9000, 20_000)] * 16])
def test_little_work_is_spread_over_the_chip(ctx, torch_cuda, sizes):
    """Items of 4096 tuples and 256 threads took 1.7 to 2 times as long as
    with 512 threads, smaller ones take 0.6."""
    pairs, want = fragments(torch_cuda, sizes, 3)
    default = best_run(ctx, torch_cuda, pairs, want)
    assert default < 1.1 * best_run(ctx, torch_cuda, pairs, want, pyg.pyg_tuning(512, 2, 0.5, 4096, 0))


def test_large_fragments_with_probes_run_on_their_own(ctx, torch_cuda):
    """Random keys: 1.26 to 1.42 times the time when queued."""
    sizes = [((1 << 20) + 100_000 * i, ((1 << 20) + 100_000 * i) * (1 + i % 3)) for i in range(10)]
    pairs, want = fragments(torch_cuda, sizes, 4)
    default = best_run(ctx, torch_cuda, pairs, want)
    assert default < 1.1 * best_run(ctx, torch_cuda, pairs, want, pyg.pyg_tuning(256, 4, 0.5, 4096, 1 << 20))
