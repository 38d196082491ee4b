"""Keys that share their low bits: digits start above these, so such keys take
as many launches as the same keys without the shared bits, at every shift;
and small sorts of keys that are in order already."""
import numpy as np
import pytest

from util import I64, alloc, dev_rel, from_device, struct

pytestmark = pytest.mark.gpu


def sort(ctx, torch, k):
    """Sorts by k, checks the result and returns the launches it took."""
    A = struct([k, np.arange(len(k))], [I64, I64])
    out = alloc(torch, A.nbytes)
    rel = dev_rel(torch, A, [I64, I64])
    before = ctx.launches()
    ctx.sort(rel, 0, out)
    took = ctx.launches() - before
    assert np.array_equal(from_device(torch, out, len(k), A.dtype), A[np.argsort(k, kind="stable")])
    return took


@pytest.mark.parametrize("n", [5000, 300_007])
@pytest.mark.parametrize("bits,shift", [(1, 63), (1, 62), (8, 56), (8, 3), (16, 32), (9, 55), (20, 20), (63, 1)])
@pytest.mark.parametrize("low", [0, 5])  # the shared low bits: zeros, or a constant
def test_shared_low_bits(ctx, torch_cuda, n, bits, shift, low):
    rng = np.random.default_rng(n + bits)
    x = rng.integers(-(1 << (bits - 1)), 1 << (bits - 1), n)
    x[:2] = -(1 << (bits - 1)), (1 << (bits - 1)) - 1
    if low >> shift:
        low &= 1
    assert sort(ctx, torch_cuda, (x << shift) | low) == sort(ctx, torch_cuda, x)


@pytest.mark.parametrize("n", [2, 63, 64, 65, 1000, 4096])
@pytest.mark.parametrize("kind", ["equal", "ordered", "last", "first", "largest"])
def test_small_sorts_in_order(ctx, torch_cuda, n, kind):
    k = np.arange(n, dtype=np.int64) // 3 - 5
    if kind == "equal":
        k[:] = 9
    elif kind == "last":
        k[-1] = -(1 << 63)
    elif kind == "first":
        k[0] = (1 << 63) - 1
    elif kind == "largest":
        k[:] = (1 << 63) - 1
    sort(ctx, torch_cuda, k)
