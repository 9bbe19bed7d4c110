"""The work that a program has this library do, as measurable cases.

Every case goes through the package's public operators (HashJoin,
HashAggregate, StarPipeline, Server, parquet_decode_chunk) with device-resident
Arrow columns, as an engine hands its batches over; the Parquet case starts
from host bytes, as a scan does. Join and group order is not defined, so a
pass lays its output out by probe row or by group key, as a program that
collects the rows does: a scatter of the output columns.

Inputs are made with torch and numpy from the seed alone. Sizes follow the
benchmark's workloads (bench.py, workloads.py) and the TPC-H shapes of the
tests (Q1's two-column grouping, Q18's grouping by order).
"""
import importlib
import math

import numpy as np
import torch

kb = importlib.import_module("krishiv-engine_b200")
W = importlib.import_module("krishiv-engine_b200.workloads")

BATCH = 8192  # rows of an Arrow batch of the engine's streams
_SPARSE = 0x9E3779B97F4A7C15 - (1 << 64)  # odd: multiplication by it permutes the 64-bit integers
_shared = {}


def listed():
    return [
        # The smallest calls: a lookup-sized table probed by two engine batches. Launches, waits
        # and host work are all there is.
        {"name": "join_small", "op": "join", "type": "inner", "build": 1_000, "probe": 10_000, "keys": "dense",
         "dup": 1.0, "nulls": 0.0, "batch": BATCH},
        # The plain equi-join of the benchmark: 1M permuted keys, 10M probe rows, half of them match.
        {"name": "join_inner", "op": "join", "type": "inner", "build": 1_000_000, "probe": 10_000_000, "keys": "dense",
         "dup": 1.0, "nulls": 0.0, "batch": 0},
        # A left outer join on surrogate keys spread over 64 bits, half the build keys repeated,
        # NULL keys on both sides, ragged sizes.
        {"name": "join_outer", "op": "join", "type": "left_outer", "build": 3_000_017, "probe": 24_000_011,
         "keys": "sparse", "dup": 1.5, "nulls": 0.01, "batch": 0},
        # An IN / EXISTS subquery on a two-column key (int64, int32).
        {"name": "join_semi", "op": "join", "type": "left_semi", "build": 2_000_003, "probe": 16_000_057,
         "keys": "pair", "dup": 1.2, "nulls": 0.0, "batch": 0},
        # A dashboard query: few rows, pushed as the engine's 8192-row batches.
        {"name": "agg_small", "op": "agg", "rows": 100_003, "groups": 1_000, "dist": "uniform", "keys": 1,
         "nulls": 0.0, "batch": BATCH, "set": "sum"},
        # TPC-H Q1 at scale factor 1: lineitem grouped by two columns into a handful of groups.
        {"name": "agg_q1", "op": "agg", "rows": 6_001_215, "groups": 6, "dist": "uniform", "keys": 2, "nulls": 0.0,
         "batch": 0, "set": "q1"},
        # TPC-H Q18's subquery at scale factor 1: lineitem grouped by order, 4 rows a group.
        {"name": "agg_q18", "op": "agg", "rows": 6_001_215, "groups": 1_500_000, "dist": "uniform", "keys": 1,
         "nulls": 0.0, "batch": 0, "set": "sum"},
        # The benchmark's aggregate: 100M rows, Zipf(1.1) keys, NULLs, 15 aggregates.
        {"name": "agg_zipf", "op": "agg", "rows": 100_000_000, "groups": 1_000_000, "dist": "zipf", "keys": 1,
         "nulls": 0.02, "batch": 0, "set": "full"},
        # The benchmark's headline: the star join with runtime filters over 300M fact rows.
        {"name": "star", "op": "star", "fact": 300_000_000, "dim_a": 20_000_000, "dim_b": 1_000_000},
        # The partitioned join under a device budget that makes it spill, at a tenth of the benchmark's size.
        {"name": "grace", "op": "grace", "build": 50_000_000, "probe": 200_000_000, "budget": 2_400_000_000},
        # The request server: a mix of join + aggregate requests of very different sizes, admitted at once.
        {"name": "serve", "op": "serve", "requests": 24, "largest": 1_000_000},
        # A row group's two column chunks off the storage: Snappy, a dictionary key with a runtime filter, a float.
        {"name": "parquet", "op": "parquet", "rows": 2_000_003, "entries": 100_000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["join", "join", "join", "agg", "agg", "agg", "star", "grace", "serve", "parquet"])
    if op == "join":
        build = _log(rng, 1_000, 5_000_000)
        probe = int(build * rng.uniform(1.0, 12.0))
        return {"op": op, "type": rng.choice(["inner", "left_outer", "left_semi"]), "build": build, "probe": probe,
                "keys": rng.choice(["dense", "sparse", "pair"]), "dup": rng.choice([1.0, 1.0, round(rng.uniform(1.1, 3.0), 2)]),
                "nulls": rng.choice([0.0, 0.01]), "batch": rng.choice([0, BATCH]) if probe < 400_000 else 0}
    if op == "agg":
        rows = _log(rng, 20_000, 100_000_000)
        return {"op": op, "rows": rows, "groups": min(rows, _log(rng, 4, 2_000_000)), "dist": rng.choice(["uniform", "zipf"]),
                "keys": rng.choice([1, 1, 2]), "nulls": rng.choice([0.0, 0.02]),
                "batch": rng.choice([0, BATCH]) if rows < 400_000 else 0, "set": rng.choice(["sum", "q1", "full"])}
    if op == "star":
        fact = _log(rng, 1_000_000, 300_000_000)
        return {"op": op, "fact": fact, "dim_a": max(1_000, fact // rng.randint(10, 60)),
                "dim_b": max(500, fact // rng.randint(200, 600))}
    if op == "grace":
        build = _log(rng, 5_000_000, 50_000_000)
        return {"op": op, "build": build, "probe": int(build * rng.uniform(2.0, 4.0)), "budget": 48 * build}
    if op == "serve":
        return {"op": op, "requests": rng.randint(8, 32), "largest": _log(rng, 20_000, 1_000_000)}
    return {"op": op, "rows": _log(rng, 50_000, 4_000_000), "entries": _log(rng, 500, 150_000)}


# ---- shared by the cases ----------------------------------------------------------------------
def _rt():
    """The program's one runtime, on a torch stream of its own."""
    if "rt" not in _shared:
        _shared["rt"] = kb.Runtime.on_torch_stream(0)
    return _shared["rt"]


def _decimal():
    """The Arrow type decimal64(15, 2), as the package's own aggregate workload declares it."""
    if "dec" not in _shared:
        _shared["dec"] = W.agg(_rt(), scale=1e-5)[1][3]
    return _shared["dec"]


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _ints(g, lo, hi, n, dtype=torch.int64):
    return torch.randint(lo, hi, (n,), dtype=dtype, device="cuda", generator=g)


def _valid(g, n, nulls):
    """A validity mask with the given share of NULLs and its Arrow bitmap."""
    if nulls <= 0:
        return None, None
    mask = torch.rand(n, device="cuda", generator=g) >= nulls
    bits = torch.zeros((n + 63) // 64 * 64, dtype=torch.uint8, device="cuda")
    bits[:n] = mask
    weights = torch.tensor([1, 2, 4, 8, 16, 32, 64, 128], dtype=torch.uint8, device="cuda")
    return mask, (bits.view(-1, 8) * weights).sum(1, dtype=torch.uint8)


def _batches(cols, n, batch):
    """The columns as DeviceBatches of `batch` rows (0: one batch); bitmaps are cut at whole bytes."""
    step = batch or max(n, 1)
    out = []
    for r0 in range(0, n, step):
        m = min(step, n - r0)
        out.append(kb.DeviceBatch([(c[0], c[1][r0:r0 + m], None if c[2] is None else c[2][r0 // 8:(r0 + m + 7) // 8])
                                   + tuple(c[3:]) for c in cols]))
    return out


# ---- joins --------------------------------------------------------------------------------------
def _join_inputs(case, seed):
    g = _generator(seed)
    nb, n = case["build"], case["probe"]
    distinct = max(1, int(nb / case["dup"]))
    ids = torch.randperm(nb, device="cuda", generator=g) if case["dup"] == 1.0 else _ints(g, 0, distinct, nb)
    pid = _ints(g, 0, 2 * distinct, n)

    def keys(i):
        if case["keys"] == "dense":
            return [i]
        wide = i * _SPARSE
        return [wide] if case["keys"] == "sparse" else [wide, (i % 1000).to(torch.int32)]
    v = _ints(g, -(1 << 62), 1 << 62, nb)
    return keys(ids), _valid(g, nb, case["nulls"]), v, keys(pid), _valid(g, n, case["nulls"])


class _Join:
    def __init__(self, case, seed):
        rt = _rt()
        bk, (_, bv), v, pk, (_, pv) = _join_inputs(case, seed)
        n = case["probe"]
        self.case, self.rt, self.n = case, rt, n
        nk = len(bk)
        build = [("k%d" % i, k, bv if i == 0 else None) for i, k in enumerate(bk)] + [("v", v, None)]
        probe = [("k%d" % i, k, pv if i == 0 else None) for i, k in enumerate(pk)] + \
            [("row", torch.arange(n, device="cuda"), None)]
        self.build = _batches(build, case["build"], case["batch"])
        self.probe = _batches(probe, n, case["batch"])
        semi = case["type"] == "left_semi"
        self.spec = kb.join_spec(case["type"], probe_keys=range(nk), build_keys=range(nk), probe_out=list(range(nk + 1)),
                                 build_out=[] if semi else [nk], build_rows_hint=case["build"])
        self.row, self.value = nk, nk + 1

    def run(self):
        case = self.case
        j = kb.HashJoin(self.rt, self.spec)
        for b in self.build:
            j.build_push_device(b)
        j.build_finish()
        if case["type"] == "left_semi":
            out = torch.zeros(self.n, dtype=torch.bool, device="cuda")
        else:
            out = torch.zeros(self.n, dtype=torch.int64, device="cuda")
        rows = 0
        for p in self.probe:
            r = j.probe_device(p)
            rows += r.rows
            if not r.rows:
                continue
            at = r.columns[self.row]
            if case["type"] == "left_semi":
                out[at] = True
            elif case["dup"] == 1.0:
                out[at] = r.columns[self.value]
            else:
                out.scatter_add_(0, at, r.columns[self.value])
        return {"by_row": out, "rows": rows}


def _join_work(case):
    nb, n = case["build"], case["probe"]
    key = 12 if case["keys"] == "pair" else 8
    fan = {"inner": 0.5 * case["dup"], "left_outer": 0.5 + 0.5 * case["dup"], "left_semi": 0.5}[case["type"]]
    width = key + 8 + (0 if case["type"] == "left_semi" else 8)
    return {"bytes": nb * (key + 8) + n * (key + 8) + n * fan * width, "flops": 0}


# ---- grouped aggregates -----------------------------------------------------------------------------
_SETS = {
    "sum": [("sum", "dec"), ("count_star", None)],
    "q1": [("sum", "q"), ("sum", "dec"), ("sum", "f"), ("avg", "q"), ("avg", "dec"), ("avg", "f"), ("count_star", None)],
    "full": [(f, c) for c in ("dec", "f", "q") for f in ("sum", "count", "min", "max", "avg")],
}


def _agg_inputs(case, seed):
    g = _generator(seed)
    n, groups = case["rows"], case["groups"]
    if case["dist"] == "zipf":
        cdf = torch.cumsum(torch.arange(1, groups + 1, device="cuda", dtype=torch.float64) ** -1.1, 0)
        u = torch.rand(n, dtype=torch.float64, device="cuda", generator=g) * cdf[-1]
        k = torch.randperm(groups, device="cuda", generator=g)[torch.searchsorted(cdf, u).clamp_(max=groups - 1)]
        del u
    else:
        k = _ints(g, 0, groups, n)
    used = {c for _, c in _SETS[case["set"]]}
    cols = {"dec": _ints(g, 100, 10_000_001, n)}
    if "f" in used:
        cols["f"] = torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
    if "q" in used:
        cols["q"] = _ints(g, 1, 51, n, torch.int32)
    return k, {c: (t, _valid(g, n, case["nulls"])) for c, t in cols.items() if c in used}


class _Agg:
    def __init__(self, case, seed):
        self.rt, self.groups = _rt(), case["groups"]
        k, cols = _agg_inputs(case, seed)
        self.split = max(1, int(math.sqrt(self.groups))) if case["keys"] == 2 else 0
        keys = [("k", k, None)]
        if self.split:
            keys = [("k0", (k // self.split).to(torch.int32), None), ("k1", (k % self.split).to(torch.int32), None)]
        at = {c: len(keys) + i for i, c in enumerate(cols)}
        batch = keys + [(c, t, bits) + ((_decimal(),) if c == "dec" else ()) for c, (t, (_, bits)) in cols.items()]
        self.batches = _batches(batch, case["rows"], case["batch"])
        self.nkeys = len(keys)
        self.spec = kb.agg_spec(0 if self.nkeys == 1 else (0, 1),
                                [(f, 0 if c is None else at[c]) for f, c in _SETS[case["set"]]],
                                expected_groups=self.groups)

    def run(self):
        a = kb.HashAggregate(self.rt, self.spec)
        for b in self.batches:
            a.push_device(b)
        a.finish()
        r = a.result_device()
        key = r.columns[0]
        if self.split:
            key = key.long() * self.split + r.columns[1]
        out = {}
        for i in range(self.nkeys, len(r.columns)):
            c = r.columns[i]
            c = c if c.shape[0] == r.rows else c.view(r.rows, -1)  # decimal128: two words a value
            o = torch.zeros((self.groups,) + tuple(c.shape[1:]), dtype=c.dtype, device="cuda")
            o[key] = c
            out["%02d" % (i - self.nkeys)] = o
        return out


def _agg_exact(case, seed):
    """The float64 outputs from exact integer sums (the values are multiples of 2^-53, or whole numbers)."""
    k, cols = _agg_inputs(case, seed)
    groups = case["groups"]

    def total(t):
        return torch.zeros(groups, dtype=torch.int64, device="cuda").index_add_(0, k, t)
    out, memo = {}, {}
    for i, (f, c) in enumerate(_SETS[case["set"]]):
        name = "%02d" % i
        out[name] = None
        if c is None or c == "dec" or f == "count" or (c == "q" and f != "avg"):
            continue
        t, (mask, _) = cols[c]
        if c not in memo:
            ok = torch.ones_like(t, dtype=torch.bool) if mask is None else mask
            count = total(ok.long())
            if c == "f":
                m = torch.where(ok, (t * float(1 << 53)).long(), 0)
                s = (total(m >> 27).double() * float(1 << 27) + total(m & ((1 << 27) - 1)).double()) / float(1 << 53)
            else:
                s = total(torch.where(ok, t.long(), 0)).double()
            memo[c] = ok, count, s
        ok, count, s = memo[c]
        if f == "sum":
            v = s
        elif f == "avg":
            v = s / count.clamp(min=1)
        else:
            start = torch.full((groups,), 2.0 if f == "min" else -1.0, dtype=torch.float64, device="cuda")
            v = start.scatter_reduce(0, k, torch.where(ok, t, start[0]), "amin" if f == "min" else "amax")
        out[name] = torch.where(count > 0, v, 0.0)
    return out if any(v is not None for v in out.values()) else None


def _agg_work(case):
    used = [c for c in ("dec", "f", "q") if c in {x for _, x in _SETS[case["set"]]}]
    width = {"dec": 8, "f": 8, "q": 4}
    outs = sum(16 if f in ("sum", "avg") and c == "dec" else 4 if f in ("min", "max") and c == "q" else 8
               for f, c in _SETS[case["set"]])
    row = 8 + sum(width[c] + (0.125 if case["nulls"] else 0) for c in used)
    return {"bytes": case["rows"] * row + case["groups"] * (8 + outs), "flops": 0}


# ---- the star query -----------------------------------------------------------------------------------
def _star_inputs(case, seed):
    g = _generator(seed)
    nf, na, nb = case["fact"], case["dim_a"], case["dim_b"]
    fact = {"fk_a": _ints(g, 0, na, nf), "fk_b": _ints(g, 0, nb, nf), "price": _ints(g, 1_000, 10_000_001, nf),
            "discount": torch.rand(nf, dtype=torch.float64, device="cuda", generator=g).mul_(0.1)}
    dims = [{"key": torch.randperm(n, device="cuda", generator=g), "pred": _ints(g, 0, 20, n, torch.int32),
             "attr": _ints(g, 0, 25, n, torch.int32)} for n in (na, nb)]
    return fact, dims


class _Star:
    def __init__(self, case, seed):
        fact, dims = _star_inputs(case, seed)
        self.fact = kb.DeviceBatch([(c, t, None) for c, t in fact.items()])
        self.dims = [kb.DeviceBatch([(c, t, None) for c, t in d.items()]) for d in dims]
        self.pipe = kb.StarPipeline(_rt(), kb.star_spec(W.PRED_VALUE, W.PRED_VALUE))

    def run(self):
        p = self.pipe
        p.reset()
        p.build_device(*self.dims)
        p.probe_device(self.fact)
        r = p.result()
        attr, total = (np.asarray(r.column(i)) for i in (0, 1))
        order = np.argsort(attr)
        return {"attr": attr[order], "sum": total[order], "joined": p.counters()["joined_rows"]}


def _star_exact(case, seed):
    fact, (a, b) = _star_inputs(case, seed)
    group = torch.full((case["dim_a"],), -1, dtype=torch.int64, device="cuda")
    group[a["key"]] = torch.where(a["pred"] == W.PRED_VALUE, a["attr"].long(), -1)
    keep_b = torch.zeros(case["dim_b"], dtype=torch.bool, device="cuda")
    keep_b[b["key"]] = b["pred"] == W.PRED_VALUE
    at = group[fact["fk_a"]]
    hit = ((at >= 0) & keep_b[fact["fk_b"]]).nonzero().view(-1)
    at = at[hit]
    value = fact["price"][hit].double() * (1.0 - fact["discount"][hit])
    have = torch.bincount(at, minlength=25)
    total = torch.zeros(25, dtype=torch.float64, device="cuda").index_add_(0, at, value)
    return {"attr": None, "sum": total[have > 0], "joined": None}


def _star_work(case):
    # per fact row both foreign keys; price and discount of the rows that join (5% of 5%); the dimensions
    return {"bytes": case["fact"] * 16.0 + case["fact"] * 0.0025 * 16 + (case["dim_a"] + case["dim_b"]) * 16.0, "flops": 0}


# ---- the partitioned join ---------------------------------------------------------------------------------
_GRACE_BATCH = 32 << 20


def _grace_inputs(case, seed):
    g = _generator(seed)
    nb, n = case["build"], case["probe"]
    domain = 2 * nb
    build = [("k", _ints(g, 0, domain, nb), _valid(g, nb, 0.01)[1]), ("p1", _ints(g, -(1 << 62), 1 << 62, nb), None),
             ("p2", _ints(g, -(1 << 62), 1 << 62, nb), None)]
    heavy = _ints(g, 0, domain, 100)
    k = _ints(g, 0, domain, n)
    hot = torch.rand(n, device="cuda", generator=g) < 0.1
    k[hot] = heavy[_ints(g, 0, 100, int(hot.sum()))]
    return build, [("k", k, _valid(g, n, 0.01)[1]), ("row", torch.arange(n, device="cuda"), None)]


class _Grace:
    def __init__(self, case, seed):
        build, probe = _grace_inputs(case, seed)
        self.n, self.budget = case["probe"], case["budget"]
        self.build = _batches(build, case["build"], _GRACE_BATCH)
        self.probe = _batches(probe, case["probe"], _GRACE_BATCH)
        self.spec = kb.join_spec("left_outer", probe_out=[0, 1], build_out=[1, 2], build_rows_hint=case["build"],
                                 max_output_rows=64 << 20)

    def run(self):
        j = kb.HashJoin(_rt(), self.spec, partitioned=True, device_budget=self.budget)
        for b in self.build:
            j.build_push_device(b)
        j.build_finish()
        out = torch.zeros(self.n, dtype=torch.int64, device="cuda")
        rows = 0

        def collect(results):
            nonlocal rows
            for r in results:
                rows += r.rows
                if r.rows:
                    out.scatter_add_(0, r.columns[1], r.columns[2])
        for p in self.probe:
            collect(j.probe_device_all(p))
        collect(j.finish_device())
        return {"by_row": out, "rows": rows}


def _grace_work(case):
    # 24 B a build row, 16 B a probe row, 32 B an output row (about 1.1 output rows per probe row)
    return {"bytes": 24.0 * case["build"] + 16.0 * case["probe"] + 35.0 * case["probe"], "flops": 0}


# ---- the request server -----------------------------------------------------------------------------------
def _serve_sizes(case):
    """(build rows, groups, match ratio) of each request; spread evenly over the logarithm, so that every seed has
    the same amount of work."""
    n = case["requests"]
    out = []
    for i in range(n):
        nb = int(round(math.exp(math.log(1_000) + (math.log(case["largest"]) - math.log(1_000)) * i / max(1, n - 1))))
        groups = min(nb, int(10 * 10 ** (4.0 * ((i * 7) % n) / n)))
        out.append((nb, groups, 0.1 + 0.9 * ((i * 5) % n) / n))
    return out


def _serve_inputs(case, seed):
    g = _generator(seed)
    base, out = 0, []
    for nb, groups, match in _serve_sizes(case):
        k = torch.randperm(nb, device="cuda", generator=g)
        grp = _ints(g, base, base + groups, nb)  # group values of different tables do not meet
        n = 10 * nb
        pk = torch.where(torch.rand(n, device="cuda", generator=g) < match, _ints(g, 0, nb, n),
                         _ints(g, 1 << 40, 1 << 41, n))
        out.append((k, grp, pk, _ints(g, -1_000_000_000, 1_000_000_001, n)))
        base += groups
    return out, base


class _Serve:
    def __init__(self, case, seed):
        inputs, self.groups = _serve_inputs(case, seed)
        self.server = kb.Server(_rt())
        self.tables, self.probes = [], []
        for k, grp, pk, x in inputs:
            self.tables.append(self.server.add_table(kb.DeviceBatch([("k", k, None), ("g", grp, None)])))
            self.probes.append(kb.DeviceBatch([("k", pk, None), ("x", x, None)]))

    def run(self):
        s = self.server
        for t, p in zip(self.tables, self.probes):
            s.submit(t, p)
        done = []
        while len(done) < len(self.probes):
            s.step(wait=True)
            while (r := s.poll()) is not None:
                done.append(r[2])
        done = [r for r in done if r is not None and r.rows]
        at, total, count = (torch.cat([r.columns[i] for r in done]) for i in range(3))
        out = {}
        for name, c in (("sum", total), ("count", count)):
            o = torch.zeros(self.groups, dtype=torch.int64, device="cuda")
            o[at] = c
            out[name] = o
        return out


def _serve_work(case):
    return {"bytes": sum(160.0 * nb + 24.0 * groups for nb, groups, _ in _serve_sizes(case)), "flops": 0}


# ---- Parquet column chunks -----------------------------------------------------------------------------------
_PAGE_ROWS = 20_000  # the row limit of a data page of the common writers


def _varint(v):
    out = bytearray()
    while v >= 0x80:
        out.append(v & 0x7F | 0x80)
        v >>= 7
    out.append(v)
    return bytes(out)


def _i32(field_delta, v):
    return bytes([field_delta << 4 | 5]) + _varint(v << 1)  # compact protocol, zigzag of v >= 0


def _page(kind, plain, body, values, encoding):
    """A page: its Thrift header (data page v1 or dictionary page) and its compressed body."""
    head = _i32(1, kind) + _i32(1, plain) + _i32(1, len(body))
    inner = _i32(1, values) + _i32(1, encoding)
    if kind == 0:
        inner += _i32(1, 3) + _i32(1, 3)  # RLE definition and repetition levels
    return head + bytes([(2 if kind == 0 else 4) << 4 | 12]) + inner + b"\0\0" + body


def _snappy_literals(data):
    """Snappy of bytes that do not compress: one literal per 64 KiB block."""
    out = [_varint(len(data))]
    for o in range(0, len(data), 65536):
        part = data[o:o + 65536]
        out += [b"\xf4", (len(part) - 1).to_bytes(2, "little"), part]
    return b"".join(out)


def _snappy_small_ints(values):
    """Snappy of int64 values below 2^24: each value's three low bytes as a literal, the zero bytes as a reference
    to those of the value before; 64 KiB blocks start afresh."""
    raw = values.astype("<i8").view(np.uint8).reshape(-1, 8)
    out = [_varint(raw.size)]
    for o in range(0, len(raw), 8192):
        b = raw[o:o + 8192]
        out.append(bytes([7 << 2]) + b[0].tobytes())
        e = np.empty((len(b) - 1, 6), dtype=np.uint8)
        e[:, 0] = 2 << 2
        e[:, 1:4] = b[1:, :3]
        e[:, 4], e[:, 5] = 0x05, 8
        out.append(e.tobytes())
    return b"".join(out)


def _levels(valid):
    """Definition levels, RLE / bit-packed hybrid: runs of all-valid groups of 8 as RLE, the rest bit-packed."""
    groups = np.packbits(valid, bitorder="little")
    full = groups == 255
    edges = np.concatenate([[0], np.flatnonzero(np.diff(full)) + 1, [len(groups)]])
    out = bytearray()
    for a, b in zip(edges[:-1], edges[1:]):
        if full[a]:
            out += _varint(int(b - a) * 8 << 1) + b"\1"
            continue
        for c in range(a, b, 63):
            part = groups[c:min(b, c + 63)]
            out += bytes([len(part) << 1 | 1]) + part.tobytes()
    return len(out).to_bytes(4, "little") + bytes(out)


def _indices(idx, width):
    """Dictionary indices: bit-packed runs of up to 504 values."""
    padded = np.zeros((len(idx) + 503) // 504 * 504, dtype=np.uint32)
    padded[:len(idx)] = idx
    bits = (padded[:, None] >> np.arange(width, dtype=np.uint32) & 1).astype(np.uint8)
    packed = np.packbits(bits.reshape(-1), bitorder="little").reshape(-1, 63 * width)
    runs = np.concatenate([np.full((len(packed), 1), 63 << 1 | 1, dtype=np.uint8), packed], axis=1).reshape(-1)
    return bytes([width]) + runs.tobytes()


def _parquet_inputs(case, seed):
    rng = np.random.default_rng(seed)
    n, entries = case["rows"], case["entries"]
    return rng, rng.permutation(entries).astype(np.int64), rng.integers(0, entries, n), rng.random(n) >= 0.02, rng.random(n)


class _Parquet:
    def __init__(self, case, seed):
        rng, dictionary, idx, valid, x = _parquet_inputs(case, seed)
        n, entries = case["rows"], case["entries"]
        width = max(1, (entries - 1).bit_length())
        keys = [_page(2, entries * 8, _snappy_small_ints(dictionary), entries, 0)]
        floats = []
        for r0 in range(0, n, _PAGE_ROWS):
            r1 = min(n, r0 + _PAGE_ROWS)
            v = valid[r0:r1]
            plain = _levels(v) + _indices(idx[r0:r1][v], width)
            keys.append(_page(0, len(plain), _snappy_literals(plain), r1 - r0, 8))
            level = _varint((r1 - r0) << 1) + b"\1"
            plain = len(level).to_bytes(4, "little") + level + x[r0:r1].tobytes()
            floats.append(_page(0, len(plain), _snappy_literals(plain), r1 - r0, 0))
        self.rt, self.n = _rt(), n
        self.chunks = []
        for parts in (keys, floats):
            data = np.frombuffer(b"".join(parts), dtype=np.uint8)
            host = torch.empty(data.size, dtype=torch.uint8, pin_memory=True)
            host.numpy()[:] = data
            self.chunks.append(host)
        wanted = rng.choice(entries, max(1, entries // 20), replace=False).astype(np.int64)
        self.filter = kb.KeyFilter.build_device(self.rt, kb.DeviceBatch([("k", torch.from_numpy(wanted).cuda(), None)]), 0)

    def run(self):
        k, info = kb.parquet_decode_chunk(self.rt, self.chunks[0].numpy(), kb.PQ_INT64, kb.PQ_SNAPPY, 1, self.n, "l", "k",
                                          self.filter)
        x, _ = kb.parquet_decode_chunk(self.rt, self.chunks[1].numpy(), kb.PQ_DOUBLE, kb.PQ_SNAPPY, 1, self.n, "g", "x")
        # the columns share the results' memory, which goes with them: a program that keeps the rows copies them
        return {"k": k.columns[0].clone(), "k_valid": k.valid[0].clone(), "pass": k.columns[1].clone(),
                "x": x.columns[0].clone(), "passing": info["passing_rows"]}


def _parquet_exact(case, seed):
    x = _parquet_inputs(case, seed)[4]
    return {"k": None, "k_valid": None, "pass": None, "x": x, "passing": None}


def _parquet_work(case):
    n, entries = case["rows"], case["entries"]
    width = max(1, (entries - 1).bit_length())
    encoded = n * (width / 8 + 8 + 0.06) + entries * 6.0
    return {"bytes": encoded + n * 16.25, "flops": 0}


# ---- the measured functions --------------------------------------------------------------------------------
_OPS = {"join": (_Join, _join_work, None), "agg": (_Agg, _agg_work, _agg_exact), "star": (_Star, _star_work, _star_exact),
        "grace": (_Grace, _grace_work, None), "serve": (_Serve, _serve_work, None),
        "parquet": (_Parquet, _parquet_work, _parquet_exact)}


def prepare(case, seed):
    _rt()
    return _OPS[case["op"]][0](case, seed)


def run(state):
    return state.run()


def work(case):
    return _OPS[case["op"]][1](case)


def exact(case, seed):
    f = _OPS[case["op"]][2]
    return f(case, seed) if f else None
