"""The one-sweep radix sort at the sizes where its paths meet: the
single-CTA network (up to 4096 elements), one tile, whole tiles and ragged
last tiles, and at key ranges that take 0 to 8 digit passes (both parities,
so both buffers end up holding the result).  Expected order: NumPy's stable
argsort."""
import numpy as np
import pytest

import pyg
from util import I32, I64, alloc, dev_rel, from_device, struct

pytestmark = pytest.mark.gpu

# Key generators by name: (rng, n) -> int64 keys.
KEYS = {
    "one": lambda r, n: np.full(n, -7, dtype=np.int64),
    "two": lambda r, n: r.integers(-1, 1, n),
    "byte": lambda r, n: r.integers(1000, 1256, n),
    "bits9": lambda r, n: r.integers(-256, 256, n),
    "bits24": lambda r, n: r.integers(-(1 << 23), 1 << 23, n),
    "bits40": lambda r, n: r.integers(-(1 << 39), 1 << 39, n),
    "full": lambda r, n: r.integers(-(1 << 63), (1 << 63) - 1, n, dtype=np.int64, endpoint=True),
    "ends": lambda r, n: r.choice(np.array([-(1 << 63), (1 << 63) - 1, 0], dtype=np.int64), n),
    "skew": lambda r, n: np.where(r.random(n) < 0.9, 5, r.integers(0, 1 << 20, n)),
    "sorted": lambda r, n: np.arange(n, dtype=np.int64) // 3,
}


@pytest.mark.parametrize("n", [2, 63, 4095, 4096, 4097, 8192, 50021, (1 << 18) + 1])
@pytest.mark.parametrize("kind", sorted(KEYS))
def test_sort_sweep(ctx, torch_cuda, n, kind):
    rng = np.random.default_rng(n)
    k = KEYS[kind](rng, n)
    order = np.argsort(k, kind="stable")
    for col in (0, 1):  # the key in either column; the other holds the row
        cols = [k, np.arange(n, dtype=np.int64)]
        A = struct(cols if col == 0 else cols[::-1], [I64, I64])
        out = alloc(torch_cuda, A.nbytes)
        ctx.sort(dev_rel(torch_cuda, A, [I64, I64]), col, out)
        assert np.array_equal(from_device(torch_cuda, out, n, A.dtype), A[order])


@pytest.mark.parametrize("n", [4096, 4097, 70001])
def test_sort_sweep_rows_gathered(ctx, torch_cuda, n):
    """Layouts that are not two int64 columns sort (key, row) items."""
    rng = np.random.default_rng(n)
    A = struct([rng.integers(-(1 << 31), 1 << 31, n).astype(np.int32), np.arange(n, dtype=np.int64)], [I32, I64])
    out = alloc(torch_cuda, A.nbytes)
    ctx.sort(dev_rel(torch_cuda, A, [I32, I64]), 0, out)
    assert np.array_equal(from_device(torch_cuda, out, n, A.dtype), A[np.argsort(A["c0"], kind="stable")])


@pytest.mark.parametrize("n", [3000, 4097, 100003])
def test_sample_keys_sorted(ctx, torch_cuda, n):
    """Bare 8-byte keys: the sampled splitters are quantiles of the sorted sample."""
    import ctypes as C

    rng = np.random.default_rng(n)
    k = rng.integers(-(1 << 40), 1 << 40, n)
    d = torch_cuda.from_numpy(k).cuda()
    fan = n  # splitter j is then sorted key j
    sp = np.zeros(fan - 1, dtype=np.int64)
    pyg.check(pyg.lib().pyg_sampled_splitters(ctx.h, d.data_ptr(), n, fan, sp.ctypes.data_as(C.POINTER(C.c_int64))))
    assert np.array_equal(sp, np.sort(k)[1:])


@pytest.mark.parametrize("limit", [1, 5000, 60000, 80000])
@pytest.mark.parametrize("asc", [True, False])
def test_sortlimit_ties_in_input_order(ctx, torch_cuda, limit, asc):
    rng = np.random.default_rng(limit)
    n = 80000
    A = struct([rng.integers(-50, 50, n), np.arange(n, dtype=np.int64)], [I64, I64])
    out = alloc(torch_cuda, A.nbytes)
    rc, got = ctx.sortlimit(dev_rel(torch_cuda, A, [I64, I64]), [0], asc, limit, out, n)
    assert rc == 0 and got == limit
    order = np.argsort(A["c0"] if asc else -A["c0"], kind="stable")[:limit]
    assert np.array_equal(from_device(torch_cuda, out, limit, A.dtype), A[order])
