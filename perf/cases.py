"""The work this library's users have it do, as measurable cases.

Each case is one pass of calls on one table, table set or wide table, through
the package's public classes, at sizes of the library's own workloads (the
2^20-key test scale, the 2^28-key table, the resize stream, the 4096-table
rounds, the 64-tenant serving steps) and of request traffic below them.
Passes that change a table come in pairs of batches, the second undoing what
the first did to the key set, so a state can be used again and every pass
does the same work.

Every output is a whole number (values, hit bits, counts), so there is no
rounding to bound and no exact().
"""
import math

import numpy as np
import torch

import databases_gpu_gb300 as dg
from databases_gpu_gb300.table import DyCuckooSet, DyCuckooWide
from databases_gpu_gb300.workloads import ResizeStream, perm32, splitmix64

M32 = 0xFFFFFFFF
NEW = 1 << 29    # indices of keys that a pass inserts and removes again
MISS = 1 << 30   # indices of keys that are never inserted
SLICE = 1 << 25  # keys generated and loaded at a time


def listed():
    return [
        # a service looking up one small request in a resident table: latency
        dict(name="find_request", kind="find", key_bytes=4, keys=1 << 20, load=0.85, n=1000,
             hit=0.5, zipf=False),
        # bulk lookups in a table far beyond the L2 (the headline workload)
        dict(name="find_large", kind="find", key_bytes=4, keys=1 << 28, load=0.90, n=1 << 26,
             hit=1.0, zipf=False),
        # 64-bit keys, skewed popularity, mostly absent keys, a ragged batch
        dict(name="find_u64_zipf", kind="find", key_bytes=8, keys=1 << 26, load=0.85, n=12345677,
             hit=0.1, zipf=True),
        # the reference's own test sequence at its scale: insert, find, erase, find again
        dict(name="cycle_small", kind="cycle", key_bytes=4, keys=1 << 20, load=0.85, n=1 << 19,
             dup=0.0),
        # a large resident table taking in and dropping a batch, some keys repeated
        dict(name="cycle_large", kind="cycle", key_bytes=4, keys=1 << 27, load=0.85, n=20000003,
             dup=0.02),
        # one client's mixed request on its own table: latency
        dict(name="mixed_request", kind="mixed", key_bytes=8, value_bytes=4, keys=1 << 18, n=4096,
             zipf=False),
        # mixed bulk updates, keys drawn with replacement
        dict(name="mixed_bulk", kind="mixed", key_bytes=4, value_bytes=4, keys=1 << 27, n=1 << 24,
             zipf=False),
        # a table growing and shrinking under mixed traffic, resizing on the way
        dict(name="resize_stream", kind="stream", batch=1 << 22, batches=3, start=1 << 20),
        # one round of work for 4096 independent tables
        dict(name="set_round", kind="set", key_bytes=4, value_bytes=4, tables=4096, lo=8, hi=20,
             ops_lo=4, ops_hi=16, requests=0),
        # one step of a serving loop over 64 tenants: coalesced requests
        dict(name="set_step", kind="set", key_bytes=8, value_bytes=4, tables=64, lo=16, hi=24,
             ops_lo=5, ops_hi=16, requests=42),
        # records wider than a slot: look up, add, remove
        dict(name="wide_records", kind="wide", key_bytes=4, keys=1 << 24, value_bytes=32, n=3000001),
        # a caller with host arrays: insert, find and erase through host memory
        dict(name="host_calls", kind="host", key_bytes=4, keys=1 << 22, n=1000003),
    ]


def _log(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm, odd as often as even."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["find", "find", "cycle", "cycle", "mixed", "mixed", "mixed", "stream", "set",
                       "set", "wide", "host"])
    kb = rng.choice([4, 8])
    if kind == "find":
        keys = _log(rng, 1 << 12, 1 << (28 if kb == 4 else 26))
        return dict(kind=kind, key_bytes=kb, keys=keys, load=round(rng.uniform(0.5, 0.9), 2),
                    n=_log(rng, 32, 1 << (26 if kb == 4 else 25)),
                    hit=rng.choice([0.1, 0.5, 1.0]), zipf=rng.random() < 0.5)
    if kind == "cycle":
        keys = _log(rng, 1 << 12, 1 << (27 if kb == 4 else 25))
        return dict(kind=kind, key_bytes=kb, keys=keys, load=round(rng.uniform(0.5, 0.88), 2),
                    n=max(32, min(_log(rng, 32, 1 << 24), keys // 2)),
                    dup=rng.choice([0.0, 0.02, 0.1]))
    if kind == "mixed":
        keys = _log(rng, 1 << 12, 1 << (27 if kb == 4 else 25))
        return dict(kind=kind, key_bytes=kb, value_bytes=4 if kb == 4 else rng.choice([4, 8]),
                    keys=keys, n=_log(rng, 32, 1 << 23), zipf=rng.random() < 0.25)
    if kind == "stream":
        batch = _log(rng, 1 << 16, 1 << 22)
        return dict(kind=kind, batch=batch, batches=3, start=batch // 4)
    if kind == "set":
        if rng.random() < 0.5:
            return dict(kind=kind, key_bytes=4, value_bytes=4, tables=_log(rng, 129, 2048), lo=8,
                        hi=rng.choice([16, 18, 20]), ops_lo=4, ops_hi=rng.choice([10, 13, 16]),
                        requests=0)
        return dict(kind=kind, key_bytes=8, value_bytes=rng.choice([4, 8]),
                    tables=_log(rng, 16, 128), lo=14, hi=rng.choice([18, 20, 22]), ops_lo=5,
                    ops_hi=rng.choice([12, 16]), requests=_log(rng, 2, 60))
    if kind == "wide":
        keys = _log(rng, 1 << 14, 1 << 24)
        return dict(kind=kind, key_bytes=kb, keys=keys, value_bytes=4 * _log(rng, 3, 32),
                    n=max(32, min(_log(rng, 256, 1 << 22), keys // 2)))
    keys = _log(rng, 1 << 14, 1 << 24)
    return dict(kind=kind, key_bytes=4, keys=keys, n=max(32, min(_log(rng, 256, 1 << 22), keys // 2)))


# ---- inputs ------------------------------------------------------------------
def _keys(kb, j, seed):
    """Key of index j (int64 tensor below 2^31): distinct, never 0."""
    if kb == 8:
        return splitmix64(j, seed)
    # perm32 sends one number to 0; the indices start just above it
    shift = (0x5BD1E996 + (seed * 7919) % (1 << 30)) & M32
    k = perm32((j + shift) & M32)
    return (k - ((k >> 31) << 32)).to(torch.int32)


def _vals(vb, j, seed):
    v = (j * 0x9E3779B1 + seed * 40503 + 1) & 0x7FFFFFFF
    return v.to(torch.int32) if vb == 4 else v * 0x100000001


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _pick(n, N, zipf, g):
    """n indices in [0, N), uniform or by Zipf(0.99) popularity."""
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    if not zipf:
        return (u * N).long().clamp_(0, N - 1)
    a = 0.01
    return (torch.pow(1.0 + u * (float(N) ** a - 1.0), 1.0 / a).long() - 1).clamp_(0, N - 1)


def _load(table, kb, vb, N, seed):
    for lo in range(0, N, SLICE):
        j = torch.arange(lo, min(N, lo + SLICE), dtype=torch.int64, device="cuda")
        table.insert(_keys(kb, j, seed), _vals(vb, j, seed), unique=True, new_keys=True)


def _outputs(n, vb):
    return (torch.zeros(n, dtype=torch.int32 if vb == 4 else torch.int64, device="cuda"),
            torch.zeros((n + 31) // 32, dtype=torch.int32, device="cuda"))


def _prepare_find(c, seed):
    g, kb, N, n = _gen(seed), c["key_bytes"], c["keys"], c["n"]
    t = dg.DyCuckoo(int(N / c["load"]), key_bytes=kb, auto_resize=False)
    _load(t, kb, kb, N, seed)
    j = _pick(n, N, c["zipf"], g)
    if c["hit"] < 1.0:
        miss = torch.rand(n, generator=g, device="cuda") >= c["hit"]
        j = torch.where(miss, j + MISS, j)
    return dict(t=t, q=_keys(kb, j, seed), out=_outputs(n, kb))


def _repeated(j, dup, g):
    """j with a share of its entries repeating other entries."""
    if dup <= 0.0:
        return j
    at = torch.rand(j.numel(), generator=g, device="cuda") < dup
    return torch.where(at, j[_pick(j.numel(), j.numel(), False, g)], j)


def _prepare_cycle(c, seed):
    """The table holds keys - n keys; a pass takes in n more, as a batch in
    random order, and drops them again."""
    g, kb, N, n = _gen(seed), c["key_bytes"], c["keys"], c["n"]
    t = dg.DyCuckoo(int(N / c["load"]), key_bytes=kb, auto_resize=False)
    _load(t, kb, kb, N - n, seed)
    new = _repeated(torch.randperm(n, generator=g, device="cuda") + NEW, c["dup"], g)
    # finds: half of them among the new keys, half never inserted
    miss = torch.rand(2 * n, generator=g, device="cuda") < 0.5
    f = _pick(2 * n, n, False, g)
    f = torch.where(miss, f + MISS, f + NEW)
    gone = _repeated(torch.randperm(n, generator=g, device="cuda") + NEW, c["dup"], g)
    rest = torch.arange(n, dtype=torch.int64, device="cuda") + NEW
    return dict(t=t, ins=_keys(kb, new, seed), val=_vals(kb, new + seed, seed),
                q=_keys(kb, f, seed), gone=_keys(kb, gone, seed), rest=_keys(kb, rest, seed),
                f1=_outputs(2 * n, kb), f2=_outputs(2 * n, kb), eb=_outputs(n, kb)[1],
                dup=c["dup"] > 0.0)


def _mixed_ops(n, mix, new_share, N, zipf, g):
    """Ops and indices of a batch and of the batch that undoes it: finds (half
    of absent keys), inserts (a share of them new keys, the rest updates),
    erases of present keys; in the second batch a new key is erased and an
    erased one inserted."""
    u = torch.rand(n, generator=g, device="cuda")
    op = torch.where(u < mix[0], 0, torch.where(u < mix[0] + mix[1], 1, 2))
    j = _pick(n, N, zipf, g) if not torch.is_tensor(N) else \
        (torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * N).long()
    r = torch.rand(n, generator=g, device="cuda")
    fresh = (op == 1) & (r < new_share)
    idx = torch.where((op == 0) & (r < 0.5), j + MISS, torch.where(fresh, j + NEW, j))
    back = torch.where(op == 0, 0, torch.where(fresh, 2, 1))
    return idx, op.to(torch.uint8), back.to(torch.uint8)


def _prepare_mixed(c, seed):
    g, kb, vb, N, n = _gen(seed), c["key_bytes"], c["value_bytes"], c["keys"], c["n"]
    t = dg.DyCuckoo(N, key_bytes=kb, value_bytes=vb)
    _load(t, kb, vb, N, seed)
    idx, op, back = _mixed_ops(n, (0.5, 0.3), 0.5, N, c["zipf"], g)
    return dict(t=t, keys=_keys(kb, idx, seed), ops=(op, back),
                vals=(_vals(vb, idx + 3, seed + 1), _vals(vb, idx + 5, seed + 2)),
                out=(_outputs(n, vb), _outputs(n, vb)))


class _Ring(ResizeStream):
    """The resize stream with its key window on a ring: after the last batch
    the window is where it began, so the batches can run again."""
    ring = 0

    def key(self, idx):
        return splitmix64(torch.where(idx < (1 << 40), idx % self.ring, idx), self.seed)


def _prepare_stream(c, seed):
    B, g, S = c["batch"], c["batches"], c["start"]
    peak = S + int(0.44 * B) * g
    w = _Ring(B, g, g, S, peak, dup=0.05, seed=seed)
    # every pass inserts this many new keys and erases as many
    ins, fnd = int(round(0.6 * B)), int(round(0.3 * B))
    w.ring = g * (B - ins - fnd) + (peak - S) + g * int(round(0.1 * B))
    t = dg.DyCuckoo(S, key_bytes=8, value_bytes=8, upper_load=0.90, lower_load=0.35,
                    min_downsize_capacity=0, max_evictions=256)
    k, v = w.preload()
    t.insert(k, v)
    batches = [w.next() for _ in range(len(w))]
    return dict(t=t, batches=[(b.ops, b.keys, b.vals) for b in batches],
                out=[_outputs(B, 8) for _ in batches])


def _prepare_set(c, seed):
    g, kb, vb, nt = _gen(seed), c["key_bytes"], c["value_bytes"], c["tables"]
    rng = np.random.default_rng(seed)
    # the set and its sizes are the user's program's; requests differ by seed
    sizes = np.round(2.0 ** np.random.default_rng(10327).uniform(c["lo"], c["hi"], nt)).astype(np.int64)
    if c["requests"]:  # requests of log-uniform size to tenants by Zipf(0.9)
        p = np.arange(1, nt + 1) ** -0.9
        cnt = np.zeros(nt, np.int64)
        who = np.random.default_rng(7).choice(nt, size=c["requests"], p=p / p.sum())
        np.add.at(cnt, who, np.round(2.0 ** np.random.default_rng(8).uniform(
            c["ops_lo"], c["ops_hi"], c["requests"])).astype(np.int64))
    else:
        cnt = np.round(2.0 ** np.random.default_rng(9).uniform(c["ops_lo"], c["ops_hi"], nt)).astype(np.int64)
    s = DyCuckooSet(sizes, key_bytes=kb, value_bytes=vb)

    def offsets(counts):
        off = np.zeros(nt + 1, np.uint32)
        off[1:] = np.cumsum(counts)
        return off, torch.from_numpy(off.view(np.int32)).cuda()

    def table_of(counts):
        return torch.repeat_interleave(torch.arange(nt, device="cuda"),
                                       torch.from_numpy(counts).cuda())

    def keys(tid, j):
        if kb == 8:
            return splitmix64(j + (tid << 32), seed)
        # the 32-bit keys of a table: its own shift of the same sequence
        return _keys(4, (j + tid * 0x1357B) & (2 * MISS - 1), seed)

    if nt <= 128:  # tenants: each loads its own table
        for t in range(nt):
            m = s.table(t)
            for lo in range(0, int(sizes[t]), SLICE):
                j = torch.arange(lo, min(int(sizes[t]), lo + SLICE), device="cuda")
                m.insert(keys(torch.full_like(j, t), j), _vals(vb, j, seed), unique=True,
                         new_keys=True)
    else:  # many small tables: slices of whole tables, all inserts, through the set
        lo = 0
        while lo < nt:
            hi = lo + 1
            while hi < nt and sizes[lo:hi + 1].sum() <= SLICE:
                hi += 1
            part = np.zeros(nt, np.int64)
            part[lo:hi] = sizes[lo:hi]
            h, d = offsets(part)
            tid = table_of(part)
            j = torch.arange(tid.numel(), device="cuda") - d.long()[tid]
            s.apply(d, torch.ones(tid.numel(), dtype=torch.uint8, device="cuda"), keys(tid, j),
                    _vals(vb, j, seed), h_offsets=h)
            lo = hi
    h, d = offsets(cnt)
    tid = table_of(cnt)
    size = torch.from_numpy(sizes).cuda()[tid]
    idx, op, back = _mixed_ops(tid.numel(), (0.7, 0.2), 0.5, size, False, g)
    n = tid.numel()
    return dict(s=s, h=h, d=d, keys=keys(tid, idx), ops=(op, back),
                vals=(_vals(vb, idx + 3, seed + 1), _vals(vb, idx + 5, seed + 2)),
                out=(_outputs(n, vb), _outputs(n, vb)))


def _prepare_wide(c, seed):
    g, kb, N, n, vb = _gen(seed), c["key_bytes"], c["keys"], c["n"], c["value_bytes"]
    w = DyCuckooWide(int(N / 0.85), vb, key_bytes=kb, auto_resize=False)

    def rows(j):
        return (j[:, None] * 31 + torch.arange(vb // 4, device="cuda") + seed).to(torch.int32)

    for lo in range(0, N - n, 1 << 22):
        j = torch.arange(lo, min(N - n, lo + (1 << 22)), dtype=torch.int64, device="cuda")
        w.insert(_keys(kb, j, seed), rows(j), unique=True)
    new = torch.randperm(n, generator=g, device="cuda") + NEW
    r = torch.rand(n, generator=g, device="cuda")
    old = _pick(n, N - n, False, g)
    q = torch.where(r < 0.5, old, torch.where(r < 0.75, new, old + MISS))
    # half updates of present keys, half new keys
    ins = torch.where(r < 0.5, old, new)
    return dict(w=w, q=_keys(kb, q, seed), ins=_keys(kb, ins, seed), val=rows(ins + 7),
                gone=_keys(kb, new, seed))


def _prepare_host(c, seed):
    g, N, n = _gen(seed), c["keys"], c["n"]
    t = dg.DyCuckoo(int(N / 0.85), auto_resize=False)
    _load(t, 4, 4, N - n, seed)
    new = torch.randperm(n, generator=g, device="cuda") + NEW
    r = torch.rand(2 * n, generator=g, device="cuda")
    f = _pick(2 * n, n, False, g)
    q = torch.where(r < 0.5, f + NEW, f + MISS)

    def host(x):
        return x.cpu().pin_memory().numpy()

    return dict(t=t, ins=host(_keys(4, new, seed)), val=host(_vals(4, new, seed)),
                q=host(_keys(4, q, seed)), out=host(_outputs(2 * n, 4)[0]),
                bits=host(_outputs(2 * n, 4)[1]), eb=host(_outputs(n, 4)[1]))


def prepare(case, seed):
    return dict(_PREPARE[case["kind"]](case, seed), kind=case["kind"])


_PREPARE = {"find": _prepare_find, "cycle": _prepare_cycle, "mixed": _prepare_mixed,
            "stream": _prepare_stream, "set": _prepare_set, "wide": _prepare_wide,
            "host": _prepare_host}


# ---- passes ------------------------------------------------------------------
def _run_find(s):
    return s["t"].find(s["q"], out=s["out"][0], hit_bits=s["out"][1])


def _run_cycle(s):
    t = s["t"]
    st = t.insert(s["ins"], s["val"])
    a = t.find(s["q"], out=s["f1"][0], hit_bits=s["f1"][1])
    n1 = t.erase(s["gone"], erased_bits=s["eb"])
    # repeats in the erase batch leave some of the new keys: a second erase takes them
    n2 = t.erase(s["rest"]) if s["dup"] else 0
    b = t.find(s["q"], out=s["f2"][0], hit_bits=s["f2"][1])
    return [st["inserted"], st["updated"], st["superseded"], a, n1, s["eb"], n2, b]


def _run_mixed(s):
    t = s["t"]
    got = []
    for ops, vals, out in zip(s["ops"], s["vals"], s["out"]):
        t.apply(ops, s["keys"], vals, out=out[0], bits=out[1])
        got += [out, t.size]
    return got


def _run_stream(s):
    t = s["t"]
    got = []
    for (ops, keys, vals), out in zip(s["batches"], s["out"]):
        t.apply(ops, keys, vals, out=out[0], bits=out[1])
        got += [out, t.size]
    return got


def _run_set(s):
    got = []
    for ops, vals, out in zip(s["ops"], s["vals"], s["out"]):
        s["s"].apply(s["d"], ops, s["keys"], vals, out=out[0], bits=out[1], h_offsets=s["h"],
                     graph=True)
        got += [out, s["s"].sizes()[0].astype(np.int64)]
    return got


def _run_wide(s):
    w = s["w"]
    st = w.insert(s["ins"], s["val"])
    v, bits = w.find(s["q"])
    n, gv, gb = w.erase(s["gone"])
    return [st["inserted"], st["updated"], v, bits, n, gv, gb]


def _run_host(s):
    t = s["t"]
    t.insert_host(s["ins"], s["val"])
    t.find_host(s["q"], s["out"], s["bits"])
    n = t.erase_host(s["ins"], s["eb"])
    return [s["out"], s["bits"], n, s["eb"]]


_RUN = {"find": _run_find, "cycle": _run_cycle, "mixed": _run_mixed, "stream": _run_stream,
        "set": _run_set, "wide": _run_wide, "host": _run_host}


def run(state):
    return _RUN[state["kind"]](state)


# ---- work --------------------------------------------------------------------
def work(case):
    """Bytes of a pass: the batch arrays read and written once, and for every
    op the one 32-byte sector of the table that holds its key's slot, written
    back too where the op changes it (a table's sectors at most once a batch
    and direction). No floating-point work."""
    k = case["kind"]

    def probe(n, slots, slot_bytes, write=0.0):
        return min(32.0 * n, slots * slot_bytes) + min(32.0 * n * write, slots * slot_bytes)

    if k == "find":
        n, kb, S = case["n"], case["key_bytes"], case["keys"] / case["load"]
        return {"bytes": n * (2 * kb + 0.125) + probe(n, S, 2 * kb), "flops": 0}
    if k == "cycle":
        n, kb, S = case["n"], case["key_bytes"], case["keys"] / case["load"]
        b = n * 2 * kb + probe(n, S, 2 * kb, 1.0)                       # insert
        b += n * (kb + 0.125) + probe(n, S, 2 * kb, 1.0)                # erase
        b += (n * kb + probe(n, S, 2 * kb)) if case["dup"] else 0       # erase of the rest
        b += 2 * (2 * n * (2 * kb + 0.125) + probe(2 * n, S, 2 * kb))   # two finds
        return {"bytes": b, "flops": 0}
    if k in ("mixed", "stream", "set"):
        if k == "stream":
            n, kb, vb, S, passes = case["batch"], 8, 8, case["start"] * 2, 2 * case["batches"]
        elif k == "mixed":
            n, kb, vb, S, passes = case["n"], case["key_bytes"], case["value_bytes"], case["keys"] / 0.7, 2
        else:
            kb, vb, passes = case["key_bytes"], case["value_bytes"], 2
            mean = lambda lo, hi: (2.0 ** hi - 2.0 ** lo) / ((hi - lo) * math.log(2.0))  # noqa: E731
            n = mean(case["ops_lo"], case["ops_hi"]) * (case["requests"] or case["tables"])
            S = mean(case["lo"], case["hi"]) * case["tables"] / 0.7
        slot = 8 if kb == 4 else 16
        return {"bytes": passes * (n * (1 + kb + 2 * vb + 0.125) + probe(n, S, slot, 0.4)), "flops": 0}
    if k == "wide":
        n, kb, vb, S = case["n"], case["key_bytes"], case["value_bytes"], case["keys"] / 0.85
        slot = 8 if kb == 4 else 16
        b = n * (kb + 2 * vb) + probe(n, S, slot, 0.5)                  # insert: row in, row stored
        b += n * (kb + 2 * vb + 0.125) + probe(n, S, slot)              # find: row read and returned
        b += n * (kb + 2 * vb + 0.125) + probe(n, S, slot, 0.5)         # erase returns the rows
        return {"bytes": b, "flops": 0}
    n, S = case["n"], case["keys"] / 0.85
    b = n * 8 + probe(n, S, 8, 1.0) + 2 * n * 8.125 + probe(2 * n, S, 8) + n * 4.125 + \
        probe(n, S, 8, 1.0)
    return {"bytes": b, "flops": 0}
