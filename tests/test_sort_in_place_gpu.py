"""Sorting into the relation's own buffer, or one that overlaps it, at no, one,
two, three and eight digit passes and below the single-CTA limit."""
import numpy as np
import pytest

import pyg
from util import I32, I64, alloc, from_device, struct

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1000, 300_007])
@pytest.mark.parametrize("bits", [0, 7, 15, 23, 63])
@pytest.mark.parametrize("shift", [0, 64])  # bytes between the buffers' starts
@pytest.mark.parametrize("types", [(I64, I64), (I32, I64)])
def test_sort_in_place(ctx, torch_cuda, n, bits, shift, types):
    rng = np.random.default_rng(n + bits)
    k = rng.integers(0, 1 << min(bits, 31 if types[0] == I32 else 63), n)
    A = struct([k, np.arange(n)], list(types))
    buf = alloc(torch_cuda, A.nbytes + shift)
    raw = A.view(np.uint8).reshape(-1)
    buf[: raw.size].copy_(torch_cuda.from_numpy(raw))
    offs = [A.dtype.fields[c][1] for c in ("c0", "c1")]
    rel = pyg.Rel(buf, n, list(types), tuple_bytes=A.dtype.itemsize, offsets=offs)
    out = buf[shift:]
    ctx.sort(rel, 0, out)
    assert np.array_equal(from_device(torch_cuda, out, n, A.dtype), A[np.argsort(k, kind="stable")])
