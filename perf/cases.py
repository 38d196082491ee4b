"""Performance cases of the join / aggregation engine.

Each case is one call (or one short pipeline) that a plan makes of the
engine, through the public Python binding of the C ABI, on device-resident
relations: the small and the large join, grouped aggregation over few and
many keys, ordering, the sort-merge join, and a batch of query fragments.
Inputs are synthetic and seeded, made with torch on the GPU: primary keys
are a random permutation of 1..n with payload key * 7 and foreign keys are
Zipf over them, as in the benchmark and the tests.

  listed()             the named cases
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  inputs and handles a program holds before the call
  run(state)           one pass through the public entry points
  work(case)           bytes the pass cannot do without
  exact(case, seed)    the same outputs by plain torch
"""
import os
import random
import sys

import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "pythia-core_b200"))

import pyg  # noqa: E402

I32, I64 = pyg.INT32, pyg.INT64
VMAX = 1 << 20  # payloads and values are uniform in [0, 2^20)

# Ranges, per operation (tuples; G = groups):
#   join       build 2^10..2^27, probe 2x..32x the build, at most 2^30;
#              keys uniform or Zipf 0.5..1.25 over the build keys
#   join_rows  build 2^14..2^22, probe 2x..16x, 50..100 % of the probe
#              tuples match; rows materialised, then ordered by row number
#   groupby    2^20..2^28 tuples, G 2^4..2^20, int64 or (int32, int32) keys,
#              uniform or Zipf(1.0) ids, group count known to the plan or not
#   sort       2^16..2^26 tuples, keys of 16..63 bits
#   mpsm       build 2^18..2^26, probe 2x..8x, theta 0..1.5, sampled or
#              learned splitters, sum sink
#   mpsm_rows  build 2^16..2^22, probe 2x..8x, theta 0..1.0, rows out
#   batch      16..128 fragments, builds log-uniform in 2^10..2^20, probes
#              4x..32x the build, uniform or Zipf(1.0)


def listed():
    return [
        # A dimension lookup inside a small query: launches and the host
        # round trip are most of its time.
        {"name": "join_small", "op": "join", "build": 4096, "probe": 65536, "theta": 0.0},
        # The plain PK-FK join + sum of the benchmark's small configuration.
        {"name": "join_pkfk", "op": "join", "build": 1 << 20, "probe": 1 << 24, "theta": 0.0},
        # A mid-size fact table with skewed foreign keys, ragged sizes.
        {"name": "join_zipf", "op": "join", "build": 10_000_019, "probe": 150_000_001, "theta": 0.75},
        # The benchmark's headline join.
        {"name": "join_large", "op": "join", "build": 1 << 27, "probe": 1 << 30, "theta": 0.0},
        # hashjoin -> sort: joined rows delivered in probe-row order.
        {"name": "join_rows", "op": "join_rows", "build": 1_000_003, "probe": 8_000_009, "match": 0.9},
        # Aggregation by a status or category column.
        {"name": "groupby_few", "op": "groupby", "tuples": 1 << 28, "groups": 16, "key": "int64", "theta": 0.0,
         "known": True},
        # Aggregation by an entity id with a few very active entities.
        {"name": "groupby_zipf", "op": "groupby", "tuples": 1 << 27, "groups": 1 << 16, "key": "int64", "theta": 1.0,
         "known": True},
        # Aggregation by a composite (int32, int32) key.
        {"name": "groupby_composite", "op": "groupby", "tuples": 40_000_003, "groups": 1 << 16, "key": "int32x2",
         "theta": 0.0, "known": True},
        # ORDER BY an int64 column.
        {"name": "sort", "op": "sort", "tuples": 20_000_003, "key_bits": 40},
        # The sort-merge join with learned range splitters on skewed keys.
        {"name": "mpsm_sum", "op": "mpsm", "build": 1 << 26, "probe": 1 << 28, "theta": 1.0, "splitter": "learned"},
        # The sort-merge join delivering its rows in key order.
        {"name": "mpsm_rows", "op": "mpsm_rows", "build": 1_000_003, "probe": 6_000_011, "theta": 0.5,
         "splitter": "sampled"},
        # A concurrent workload of many joins of uneven size.
        {"name": "batch", "op": "batch", "fragments": 96, "min_log2": 10, "max_log2": 20, "theta": 0.0, "mix": 1},
    ]


def draw(rng):
    def size(lo, hi):
        return int(2 ** rng.uniform(lo, hi)) | 1

    op = rng.choice(["join", "join", "join_rows", "groupby", "groupby", "sort", "mpsm", "mpsm_rows", "batch"])
    if op == "join":
        b = size(10, 26)
        return {"op": op, "build": b, "probe": min(1 << 29, int(b * 2 ** rng.uniform(1, 5))),
                "theta": rng.choice([0.0, 0.5, 0.75, 1.0, 1.25])}
    if op == "join_rows":
        b = size(14, 22)
        return {"op": op, "build": b, "probe": int(b * 2 ** rng.uniform(1, 4)),
                "match": round(rng.uniform(0.5, 1.0), 3)}
    if op == "groupby":
        return {"op": op, "tuples": size(20, 28), "groups": int(2 ** rng.uniform(4, 20)),
                "key": rng.choice(["int64", "int64", "int32x2"]), "theta": rng.choice([0.0, 0.0, 1.0]),
                "known": rng.random() < 0.75}
    if op == "sort":
        return {"op": op, "tuples": size(16, 26), "key_bits": rng.randint(16, 63)}
    if op == "mpsm":
        b = size(18, 26)
        return {"op": op, "build": b, "probe": int(b * 2 ** rng.uniform(1, 3)) if b < 1 << 25 else 2 * b,
                "theta": rng.choice([0.0, 0.5, 1.0, 1.5]), "splitter": rng.choice(["sampled", "learned"])}
    if op == "mpsm_rows":
        b = size(16, 22)
        return {"op": op, "build": b, "probe": int(b * 2 ** rng.uniform(1, 3)),
                "theta": rng.choice([0.0, 0.5, 1.0]), "splitter": rng.choice(["sampled", "learned"])}
    return {"op": op, "fragments": rng.randint(16, 128), "min_log2": 10, "max_log2": rng.randint(15, 20),
            "theta": rng.choice([0.0, 1.0]), "mix": rng.randrange(1 << 20)}


# ---------------------------------------------------------------------------
# Inputs (torch only).


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFFFFFF)


def _ranks(n, size, theta, gen):
    """n ranks in [0, size), uniform or Zipf(theta) by inversion of the continuous CDF."""
    if theta == 0:
        return torch.randint(0, size, (n,), device="cuda", generator=gen)
    u = torch.rand(n, device="cuda", dtype=torch.float64, generator=gen)
    if theta == 1:
        x = torch.exp(u.mul_(torch.log(torch.tensor(size + 1.0, dtype=torch.float64)).item()))
    else:
        e = 1.0 - theta
        x = u.mul_((size + 1.0) ** e - 1.0).add_(1.0).pow_(1.0 / e)
    return x.sub_(1.0).long().clamp_(0, size - 1)


def _build(n, gen):
    """n (key, key * 7) tuples, keys a permutation of 1..n; and the keys."""
    keys = torch.randperm(n, device="cuda", generator=gen).add_(1)
    R = torch.empty(n, 2, dtype=torch.int64, device="cuda")
    R[:, 0] = keys
    torch.mul(keys, 7, out=R[:, 1])
    return R, keys


def _probe(n, keys, theta, gen, row_numbers=False, match=1.0):
    """n (fk, value) tuples; a share 1 - match of the fks has no build key
    (the same number of tuples for every seed)."""
    S = torch.empty(n, 2, dtype=torch.int64, device="cuda")
    nk = keys.numel()
    step = 1 << 26
    for i in range(0, n, step):
        m = min(step, n - i)
        fk = keys[_ranks(m, nk, theta, gen)]
        S[i:i + m, 0] = fk
        if row_numbers:
            S[i:i + m, 1] = torch.arange(i, i + m, device="cuda")
        else:
            S[i:i + m, 1] = torch.randint(0, VMAX, (m,), device="cuda", generator=gen)
    if match < 1.0:
        S[torch.randperm(n, device="cuda", generator=gen)[int(n * match):], 0] += nk
    return S


def _fragment_sizes(case):
    r = random.Random(case["mix"])
    out = []
    for _ in range(case["fragments"]):
        b = int(2 ** r.uniform(case["min_log2"], case["max_log2"]))
        out.append((b, b * r.randint(4, 32)))
    return out


def _inputs(case, seed):
    g = _generator(seed)
    op = case["op"]
    if op in ("join", "join_rows", "mpsm", "mpsm_rows"):
        R, keys = _build(case["build"], g)
        S = _probe(case["probe"], keys, case.get("theta", 0.0), g, row_numbers=op == "join_rows",
                   match=case.get("match", 1.0))
        return R, S
    if op == "groupby":
        n, G = case["tuples"], case["groups"]
        A = torch.empty(n, 2, dtype=torch.int64, device="cuda")
        ids = torch.randperm(G, device="cuda", generator=g)
        k_of = ids[_ranks(n, G, case["theta"], g)]
        k_of[torch.randperm(n, device="cuda", generator=g)[:G]] = ids  # every group has a tuple
        step = 1 << 26
        for i in range(0, n, step):
            m = min(step, n - i)
            k = k_of[i:i + m]
            if case["key"] == "int32x2":
                pair = A.view(torch.int32).view(n, 4)
                pair[i:i + m, 0] = (k >> 8).to(torch.int32)
                pair[i:i + m, 1] = (k & 255).to(torch.int32)
            else:
                A[i:i + m, 0] = k
            A[i:i + m, 1] = torch.randint(0, VMAX, (m,), device="cuda", generator=g)
        return (A,)
    if op == "sort":
        n, h = case["tuples"], 1 << (case["key_bits"] - 1)
        A = torch.empty(n, 2, dtype=torch.int64, device="cuda")
        A[:, 0] = torch.randint(-h, h, (n,), device="cuda", generator=g)
        A[:, 1] = torch.arange(n, device="cuda")
        return (A,)
    pairs = []
    for nb, np_ in _fragment_sizes(case):
        R, keys = _build(nb, g)
        pairs.append((R, _probe(np_, keys, case["theta"], g)))
    return tuple(pairs)


# ---------------------------------------------------------------------------

_CTX = None


def _ctx():
    """The program's context: created once and kept."""
    global _CTX
    if _CTX is None:
        _CTX = pyg.Ctx(0)
    return _CTX


class _Batch:
    """A planned batch; freed with the state that holds it."""

    def __init__(self, ctx, frags):
        self.ctx, self.h = ctx, ctx.batch_create(frags)

    def __del__(self):
        self.ctx.batch_free(self.h)


SPLITTERS = {"sampled": pyg.MPSM_SAMPLED, "learned": pyg.MPSM_LEARNED}
BOTH = [(0, 1), (1, 1)]  # B$1, P$1


def prepare(case, seed):
    ctx = _ctx()
    op = case["op"]
    data = _inputs(case, seed)
    s = {"op": op, "ctx": ctx, "case": case}
    if op == "batch":
        s["data"] = data
        s["n"] = len(data)
        s["batch"] = _Batch(ctx, ctx.fragments([(R, R.shape[0], S, S.shape[0]) for R, S in data]))
        return s
    types = [I32, I32, I64] if case.get("key") == "int32x2" else [I64, I64]
    rels = [pyg.Rel(t, t.shape[0], types) for t in data]
    if op in ("join", "join_rows", "mpsm", "mpsm_rows"):
        s["R"], s["S"] = rels
        n = rels[1].ntuples
        if op in ("join_rows", "mpsm_rows"):
            s["rows"] = torch.empty(n, 2, dtype=torch.int64, device="cuda")
        if op == "join_rows":
            s["sorted"] = torch.empty(n, 2, dtype=torch.int64, device="cuda")
        if op in ("mpsm", "mpsm_rows"):
            s["opts"] = ctx.mpsm_opts(SPLITTERS[case["splitter"]], 1024, 0.01, 1024)
        return s
    s["A"] = rels[0]
    if op == "groupby":
        s["groups"] = case["groups"]
        s["known"] = case["groups"] if case["known"] else 0
        s["out"] = torch.empty(case["groups"], 3, dtype=torch.int64, device="cuda")
        s["keys"] = [0, 1] if case["key"] == "int32x2" else [0]
    else:
        s["out"] = torch.empty_like(data[0])
    return s


def run(s):
    ctx, op = s["ctx"], s["op"]
    if op == "join":
        count, sums = ctx.hashjoin_agg(s["R"], [0], s["S"], [0], BOTH)
        return {"count": count, "sums": sums}
    if op == "join_rows":
        ht = ctx.hashjoin_build(s["R"], [0], [1], pyg.HT_MATERIALIZE, 0.5)
        _, count = ctx.hashjoin_probe_materialize(ht, s["S"], [0], BOTH, s["rows"], s["S"].ntuples)
        ht.free()
        ctx.sort(pyg.Rel(s["rows"], count, [I64, I64]), 1, s["sorted"])
        return {"count": count, "rows": s["sorted"][:count]}
    if op == "groupby":
        _, n = ctx.groupby(s["A"], s["keys"], pyg.AGG_SUM | pyg.AGG_COUNT, len(s["keys"]), True, s["known"], s["out"],
                           s["groups"])
        return {"groups": n, "table": s["out"][:n]}
    if op == "sort":
        ctx.sort(s["A"], 0, s["out"])
        return s["out"]
    if op == "mpsm":
        count, sums, _ = ctx.mpsm_join_agg(s["R"], 0, s["S"], 0, BOTH, s["opts"])
        return {"count": count, "sums": sums}
    if op == "mpsm_rows":
        _, count = ctx.mpsm_join_materialize(s["R"], 0, s["S"], 0, BOTH, s["opts"], s["rows"], s["S"].ntuples)
        return {"count": count, "rows": s["rows"][:count]}
    _, counts, sums, _ = ctx.batch_run(s["batch"].h, s["n"])
    return {"counts": counts, "sums": sums}


def work(case):
    op = case["op"]
    if op == "groupby":
        b = 16 * case["tuples"] + 24 * case["groups"]
    elif op == "sort":
        b = 32 * case["tuples"]
    elif op == "batch":
        b = sum(16 * (nb + np_) for nb, np_ in _fragment_sizes(case))
    else:
        b = 16 * (case["build"] + case["probe"])
        if op in ("join_rows", "mpsm_rows"):
            b += 16 * int(case["probe"] * case.get("match", 1.0))
    return {"bytes": float(b), "flops": 0.0}


def exact(case, seed):
    op = case["op"]
    data = _inputs(case, seed)
    if op in ("join", "mpsm"):
        S = data[1]
        return {"count": S.shape[0], "sums": [int(S[:, 0].sum().item()) * 7, int(S[:, 1].sum().item())]}
    if op == "join_rows":
        nk, S = data[0].shape[0], data[1]
        S = S[S[:, 0] <= nk]
        return {"count": S.shape[0], "rows": torch.stack([S[:, 0] * 7, S[:, 1]], 1)}
    if op == "groupby":
        (A,) = data
        if case["key"] == "int32x2":
            pair = A.view(torch.int32).view(-1, 4)
            ids = (pair[:, 0].long() << 8) | pair[:, 1].long()
        else:
            ids = A[:, 0]
        G = case["groups"]
        cnt = torch.bincount(ids, minlength=G)
        tot = torch.zeros(G, dtype=torch.int64, device="cuda").index_add_(0, ids, A[:, 1])
        k = torch.nonzero(cnt).view(-1)
        first = k
        if case["key"] == "int32x2":  # the two int32 key columns read as one int64 word
            first = ((k & 255) << 32) | (k >> 8)
        return {"groups": k.numel(), "table": torch.stack([first, tot[k], cnt[k]], 1)}
    if op == "sort":
        (A,) = data
        return A[torch.sort(A[:, 0], stable=True)[1]]
    if op == "mpsm_rows":
        S = data[1]
        S = S[torch.sort(S[:, 0], stable=True)[1]]
        return {"count": S.shape[0], "rows": torch.stack([S[:, 0] * 7, S[:, 1]], 1)}
    sums = [int((S[:, 0] * 7 + S[:, 1]).sum().item()) for _, S in data]
    return {"counts": torch.tensor([S.shape[0] for _, S in data]), "sums": torch.tensor(sums)}
