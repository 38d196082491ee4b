"""A batch's queued tables stay within 2^26 slots: the smallest fragments are
queued, the others run as their own joins and share one table."""
import pytest

import pyg

pytestmark = pytest.mark.gpu
SLOTS = 1 << 26


def test_queued_tables_are_bounded(ctx, torch_cuda):
    torch = torch_cuda
    gen = torch.Generator(device="cuda").manual_seed(3)
    pairs, want = [], []
    for i in range(40):
        nb, np_ = (1 << 20) + 512 * ((7 * i) % 40), 3000 + i
        k = torch.randperm(nb, device="cuda", generator=gen) + i
        R = torch.stack([k, k * 3], 1).contiguous()
        f = torch.randint(0, 2 * nb, (np_,), device="cuda", generator=gen)
        S = torch.stack([f, torch.arange(np_, device="cuda")], 1).contiguous()
        hit = (f >= i) & (f < nb + i)
        pairs.append((R, nb, S, np_))
        want.append((int(hit.sum()), int((f[hit] * 3 + S[hit, 1]).sum())))
    b = ctx.batch_create(ctx.fragments(pairs))
    try:
        for _ in range(2):
            rc, c, s, lat = ctx.batch_run(b, len(pairs))
            assert rc == 0 and [(int(x), int(y)) for x, y in zip(c, s)] == want and (lat > 0).all()
        order = sorted(range(len(pairs)), key=lambda i: pairs[i][1])
        slots, queued = 0, 0
        for i in order:
            slots += 2 * pairs[i][1] + 64
            queued += slots <= SLOTS
        assert 0 < queued < len(pairs)
        # The stall hook takes queued fragments only (the batch is not run after it).
        got = [pyg.lib().pyg_batch_inject_stall(ctx.h, b, i) for i in order]
        assert got == [pyg.PYG_OK] * queued + [pyg.PYG_ERR_ARG] * (len(pairs) - queued)
    finally:
        ctx.batch_free(b)


def test_tuner_tries_the_default_threshold(ctx, torch_cuda):
    """Builds just above 2^20 with few probes: every smaller threshold sends
    each fragment to a join of its own, whose clear of a table for one
    fragment at a time is most of the run."""
    torch = torch_cuda
    pairs = []
    for i in range(24):
        nb, np_ = (1 << 20) + 1 + i, 1024
        k = torch.randperm(nb, device="cuda")
        R = torch.stack([k, k], 1).contiguous()
        pairs.append((R, nb, R[:np_].clone(), np_))
    t = ctx.autotune(ctx.fragments(pairs), None)
    assert t.large_build == 0
