"""Calls whose faster route needs more device memory than there is fall back
to the one that needs less, and a call that cannot run at all reports
PYG_ERR_OOM once.  Each case runs in a process of its own that first takes
all device memory but a stated rest."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HEAD = """
import sys
sys.path.insert(0, sys.argv[1] + "/pythia-core_b200")
import torch, pyg
I32, I64 = pyg.INT32, pyg.INT64
ctx = pyg.Ctx(0)
def leave(mib):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    return torch.empty(free - (mib << 20), dtype=torch.uint8, device="cuda")
def small_join():  # loads the kernels and proves the context
    k = torch.arange(10000, device="cuda")
    R = torch.stack([k, k], 1).contiguous()
    for algo in (pyg.JOIN_DIRECT, pyg.JOIN_RADIX):
        n, _ = ctx.hashjoin_agg(pyg.Rel(R, 10000, [I64, I64]), [0], pyg.Rel(R, 10000, [I64, I64]), [0], [(0, 1), (1, 1)],
                                algo)
        assert n == 10000
small_join()
"""

# One sampled pass over 2^28 wide tuples: 4.0 GiB of exact regions, 4.8 GiB
# with a sample's slack.
JOIN = HEAD + """
n, m = 1 << 28, 5000
S = torch.empty(n, 2, dtype=torch.int64, device="cuda")
S[:, 0] = torch.randint(0, m, (n,), device="cuda")
S[:, 1] = 1
S[::1000, 1] = 1 << 40
sums = [int(S[:, 0].sum()) * 7, int(S[:, 1].sum())]
k = torch.arange(m, device="cuda")
R = torch.stack([k, k * 7], 1).contiguous()
hog = leave(4500)
got, s = ctx.hashjoin_agg(pyg.Rel(R, m, [I64, I64]), [0], pyg.Rel(S, n, [I64, I64]), [0], [(0, 1), (1, 1)],
                          pyg.JOIN_RADIX, 7)
assert got == n and [int(x) for x in s] == sums
small_join()
"""

# (int32, int32) keys: no room for partitions of the 4 GiB input.
GROUPBY = HEAD + """
n, g = 1 << 28, 5000
A = torch.empty(n, 2, dtype=torch.int64, device="cuda")
ids = torch.randint(0, g, (n,), dtype=torch.int32, device="cuda")
P = A.view(torch.int32).view(n, 4)
P[:, 0] = ids
P[:, 1] = 3
A[:, 1] = 2
cnt = torch.bincount(ids, minlength=g).cpu()
del ids
out = torch.empty(g, 3, dtype=torch.int64, device="cuda")
hog = leave(1200)
rc, got = ctx.groupby(pyg.Rel(A, n, [I32, I32, I64]), [0, 1], 3, 2, True, g, out, g)
assert rc == 0 and got == g
out = out.cpu()
assert torch.equal(out[:, 0], torch.arange(g) | (3 << 32))
assert torch.equal(out[:, 2], cnt) and torch.equal(out[:, 1], cnt * 2)
small_join()
"""

# 24 fragments whose tables would take 1.1 GiB together.
BATCH = HEAD + """
pairs = []
for i in range(24):
    nb = 1200000 + i
    k = torch.randperm(nb, device="cuda")
    R = torch.stack([k, k], 1).contiguous()
    pairs.append((R, nb, R[: 5000 + i].clone(), 5000 + i))
want = [(n, 2 * int(S[:, 0].sum())) for _, _, S, n in pairs]
hog = leave(700)
b = ctx.batch_create(ctx.fragments(pairs))
for _ in range(2):
    rc, c, s, _ = ctx.batch_run(b, len(pairs))
    assert rc == 0 and [(int(x), int(y)) for x, y in zip(c, s)] == want
ctx.batch_free(b)
small_join()
"""

# Two buffers of 2 GiB do not fit: an error, after which the context works.
SORT = HEAD + """
n = 1 << 27
A = torch.randint(-(1 << 62), 1 << 62, (n, 2), device="cuda")
out = torch.empty_like(A)
hog = leave(1000)
try:
    ctx.sort(pyg.Rel(A, n, [I64, I64]), 0, out)
    raise SystemExit("the sort was expected to run out of memory")
except pyg.PygError as e:
    assert e.code == pyg.PYG_ERR_OOM, e.code
small_join()
"""


@pytest.mark.parametrize("script", [JOIN, GROUPBY, BATCH, SORT], ids=["join", "groupby", "batch", "sort"])
def test_little_memory(torch_cuda, script):
    torch_cuda.cuda.empty_cache()
    r = subprocess.run([sys.executable, "-c", script, ROOT], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
