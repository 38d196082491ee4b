"""A look-back wait that gives up: the tile before never publishes its counts
(a host-side hook), the waits end after their limit, every later pass and
every kernel that would take row numbers from the unfinished order does
nothing, the call reports PYG_ERR_TIMEOUT, and the same call then answers."""
import numpy as np
import pytest

import pyg
from util import I32, I64, alloc, dev_rel, from_device, struct

pytestmark = pytest.mark.gpu
SORT, MERGE = 0, 1
N = 200_003


def data():
    rng = np.random.default_rng(5)
    return rng.permutation(N).astype(np.int64) - N // 2


def sort16(ctx, torch):
    k = data()
    A = struct([k, np.arange(N)], [I64, I64])
    out = alloc(torch, A.nbytes)
    ctx.sort(dev_rel(torch, A, [I64, I64]), 0, out)
    assert np.array_equal(from_device(torch, out, N, A.dtype), A[np.argsort(k)])


def sort_gathered(ctx, torch):
    k = data().astype(np.int32)
    A = struct([np.arange(N), k], [I64, I32])
    out = alloc(torch, A.nbytes)
    ctx.sort(dev_rel(torch, A, [I64, I32]), 1, out)
    assert np.array_equal(from_device(torch, out, N, A.dtype), A[np.argsort(k)])


def sortlimit(ctx, torch):
    k = data()
    A = struct([k, np.arange(N)], [I64, I64])
    out = alloc(torch, A.nbytes)
    rc, got = ctx.sortlimit(dev_rel(torch, A, [I64, I64]), [0], True, N - 3, out, N)
    pyg.check(rc)
    assert got == N - 3 and np.array_equal(from_device(torch, out, got, A.dtype), A[np.argsort(k)][: N - 3])


def groups(ctx, torch):
    k = data()
    A = struct([k, k * 3], [I64, I64])
    out = alloc(torch, 24 * N)
    rc, g = ctx.groupby(dev_rel(torch, A, [I64, I64]), [0], 3, 1, True, N, out, N)
    assert rc == 0 and g == N
    t = from_device(torch, out, N, np.dtype([("k", np.int64), ("s", np.int64), ("c", np.int64)]))
    k = np.sort(k)
    assert np.array_equal(t["k"], k) and np.array_equal(t["s"], 3 * k) and (t["c"] == 1).all()


def merge(ctx, torch, cols):
    """cols: projected build columns (more than one besides the key: rows are gathered)."""
    k = data()
    types = [I64] * (1 + max(cols))
    R = struct([k] + [k * (c + 1) for c in range(1, len(types))], types)
    S = struct([k[::-1].copy(), np.arange(N)], [I64, I64])
    out = alloc(torch, 8 * (len(cols) + 1) * N)
    rc, got = ctx.mpsm_join_materialize(dev_rel(torch, R, types), 0, dev_rel(torch, S, [I64, I64]), 0,
                                        [(0, c) for c in cols] + [(1, 1)], ctx.mpsm_opts(), out, N)
    assert rc == 0 and got == N
    t = from_device(torch, out, N, np.dtype([(f"c{i}", np.int64) for i in range(len(cols) + 1)]))
    for i, c in enumerate(cols):
        assert np.array_equal(t[f"c{i}"], np.sort(k) * (c + 1))
    assert np.array_equal(t[f"c{len(cols)}"], np.argsort(k[::-1]))


def merge_values(ctx, torch):
    merge(ctx, torch, [1])


def merge_rows(ctx, torch):
    merge(ctx, torch, [1, 2])


def splitters(ctx, torch):
    import ctypes as C

    k = data()
    sp = np.zeros(N - 1, dtype=np.int64)
    pyg.check(pyg.lib().pyg_sampled_splitters(ctx.h, torch.from_numpy(k).cuda().data_ptr(), N, N,
                                              sp.ctypes.data_as(C.POINTER(C.c_int64))))
    assert np.array_equal(sp, np.sort(k)[1:])


@pytest.mark.parametrize("where,call", [(SORT, sort16), (SORT, sort_gathered), (SORT, sortlimit), (SORT, groups),
                                        (SORT, merge_values), (SORT, merge_rows), (MERGE, merge_values),
                                        (MERGE, merge_rows), (SORT, splitters)])
def test_stalled_look_back(ctx, torch_cuda, where, call):
    call(ctx, torch_cuda)
    pyg.check(pyg.lib().pyg_inject_stall(ctx.h, where))
    with pytest.raises(pyg.PygError) as e:
        call(ctx, torch_cuda)
    assert e.value.code == pyg.PYG_ERR_TIMEOUT
    call(ctx, torch_cuda)


def test_unknown_place_is_refused(ctx):
    assert pyg.lib().pyg_inject_stall(ctx.h, 2) == pyg.PYG_ERR_ARG
