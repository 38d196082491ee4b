"""Contexts of their own on several host threads: calls whose kernels need
different amounts of shared memory must not disturb one another."""
import threading

import pytest

import pyg
from util import I64

pytestmark = pytest.mark.gpu


def run(torch, bodies, rounds):
    """bodies: functions of a context; each on its own thread and context."""
    errors = []
    start = threading.Barrier(len(bodies))

    def work(body):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                ctx = pyg.Ctx(0)
                try:
                    start.wait()
                    for _ in range(rounds):
                        body(ctx)
                finally:
                    ctx.close()
        except BaseException as e:  # noqa: B902
            errors.append(e)

    threads = [threading.Thread(target=work, args=(b,)) for b in bodies]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def join(rel, n, bits):
    def body(ctx):
        got, sums = ctx.hashjoin_agg(rel, [0], rel, [0], [(0, 1), (1, 1)], pyg.JOIN_RADIX, bits)
        assert got == n and [int(x) for x in sums] == [3 * n * (n - 1) // 2] * 2
    return body


def mpsm(rel, n, kind):
    def body(ctx):
        got, sums, _ = ctx.mpsm_join_agg(rel, 0, rel, 0, [(0, 1), (1, 1)], ctx.mpsm_opts(kind))
        assert got == n and [int(x) for x in sums] == [3 * n * (n - 1) // 2] * 2
    return body


def partition(torch, rel, n, fanout):
    out = torch.empty(n, 2, dtype=torch.int64, device="cuda")

    def body(ctx):
        assert ctx.partition(rel, 0, pyg.SPLIT_EXACTRANGE, fanout, out, 0, n - 1)[-1] == n
    return body


def relation(torch, n):
    k = torch.arange(n, device="cuda")
    return pyg.Rel(torch.stack([k, k * 3], 1).contiguous(), n, [I64, I64])


def test_radix_bits(torch_cuda):
    n = 20_000
    rel = relation(torch_cuda, n)
    torch_cuda.cuda.synchronize()
    run(torch_cuda, [join(rel, n, b) for b in (2, 9, 14, 16)], 150)


def test_range_counts(torch_cuda):
    small, large = 3_000, 40_000_000
    a, b = relation(torch_cuda, small), relation(torch_cuda, large)
    torch_cuda.cuda.synchronize()
    run(torch_cuda, [mpsm(a, small, pyg.MPSM_SAMPLED), mpsm(b, large, pyg.MPSM_SAMPLED)], 30)


def test_fanouts(torch_cuda):
    n = 50_000
    rel = relation(torch_cuda, n)
    torch_cuda.cuda.synchronize()
    run(torch_cuda, [partition(torch_cuda, rel, n, f) for f in (2, 64, 4096)], 150)


def test_operators_side_by_side(torch_cuda):
    torch = torch_cuda
    n, G = 300_000, 5000
    rel = relation(torch, n)
    ids = torch.arange(n, device="cuda") % G
    A = pyg.Rel(torch.stack([ids, ids], 1).contiguous(), n, [I64, I64])
    perm = torch.randperm(n, device="cuda")
    P = pyg.Rel(torch.stack([perm, perm * 3], 1).contiguous(), n, [I64, I64])
    want_rows = torch.stack([torch.arange(n, device="cuda") * 3] * 2, 1)
    R = torch.stack([torch.arange(2000, device="cuda")] * 2, 1).contiguous()

    def groupby(ctx):
        out = torch.empty(G, 3, dtype=torch.int64, device="cuda")
        rc, g = ctx.groupby(A, [0], 3, 1, True, G, out, G)
        assert rc == 0 and g == G and torch.equal(out[:, 2], torch.bincount(ids, minlength=G))

    def sort(ctx):
        out = torch.empty(n, 2, dtype=torch.int64, device="cuda")
        ctx.sort(P, 0, out)
        assert torch.equal(out[:, 0], torch.arange(n, device="cuda"))

    def rows(ctx):
        out = torch.empty(n, 2, dtype=torch.int64, device="cuda")
        rc, c = ctx.mpsm_join_materialize(P, 0, rel, 0, [(0, 1), (1, 1)], ctx.mpsm_opts(), out, n)
        assert rc == 0 and c == n and torch.equal(out, want_rows)

    def direct(ctx):
        for algo in (pyg.JOIN_DIRECT, pyg.JOIN_RADIX):
            got, _ = ctx.hashjoin_agg(P, [0], rel, [0], [(0, 1), (1, 1)], algo)
            assert got == n

    def batch(ctx):
        b = ctx.batch_create(ctx.fragments([(R, 2000, R, 2000)] * 8))
        rc, c, _, _ = ctx.batch_run(b, 8)
        ctx.batch_free(b)
        assert rc == 0 and (c == 2000).all()

    torch.cuda.synchronize()
    run(torch, [groupby, sort, rows, direct, batch], 40)
