"""Queued fragments over several waves of tables (2^20 slots each), with empty
sides, repeated build keys, the INT64_MIN marker and fragments larger than a
wave; default tuning."""
import numpy as np
import pytest

import pyg

pytestmark = pytest.mark.gpu


def test_batch_over_several_waves(ctx, torch_cuda):
    torch = torch_cuda
    rng = np.random.default_rng(3)
    pairs, want, keep = [], [], []
    for i in range(30):
        nb = int(2 ** rng.uniform(4, 20)) if i else 700_001  # the first one fills a wave by itself
        np_ = nb * int(rng.integers(1, 5))
        if i == 7:
            np_ = 0
        if i == 8:
            nb = 0
        k = rng.permutation(max(nb, 1))[:nb].astype(np.int64) + 10
        if nb and i % 5 == 1:
            k[: nb // 3] = k[nb // 2]  # one key many times
        if nb and i % 5 == 2:
            k[0] = -(1 << 63)
        f = k[rng.integers(0, nb, np_)] if nb else rng.integers(0, 99, np_)
        f = np.where(rng.random(np_) < 0.2, f + 10 * nb + 7, f)
        p, v = rng.integers(0, 1000, nb), rng.integers(0, 1000, np_)
        u, inv, cnt = np.unique(k, return_inverse=True, return_counts=True)
        psum = np.bincount(inv, weights=p, minlength=len(u)).astype(np.int64) if nb else np.zeros(0, np.int64)
        at = np.searchsorted(u, f)
        ok = at < len(u)
        ok[ok] = u[at[ok]] == f[ok]
        at, vv = at[ok], v[ok]
        want.append((int(cnt[at].sum()), int((psum[at] + cnt[at] * vv).sum())))
        R = torch.from_numpy(np.stack([k, p], 1).astype(np.int64)).cuda()
        S = torch.from_numpy(np.stack([f, v], 1).astype(np.int64)).cuda()
        keep += [R, S]
        pairs.append((R, nb, S, np_))
    b = ctx.batch_create(ctx.fragments(pairs))
    try:
        for _ in range(2):
            rc, c, s, _ = ctx.batch_run(b, len(pairs))
            assert rc == 0 and [(int(x), int(y)) for x, y in zip(c, s)] == want
    finally:
        ctx.batch_free(b)
