"""Timing cases of the engine's main path: one function call per query, through
the public entry points (``Database.sql``, ``falcondb_b200.ops`` and
``falcondb_b200.serving``), over the range of sizes, types and options in which
the queries are used.

Data follows ``falcondb_b200/workloads.py``: ``score`` float64 uniform [0, 100),
``salary`` int64 uniform [30000, 200000], 12 ``dept`` labels, build keys a
permutation with probe keys matching about half the time, Zipf(1.1) group keys.
Everything is drawn on the GPU from the seed alone.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import falcondb_b200 as F
from falcondb_b200 import ops, serving as S, workloads as W

DEV = "cuda"
SCATTER = 7919          # build and probe keys * 7919 + 3: too wide for a direct-addressed join table
MIX = -7046029254386353131  # odd 64-bit multiplier: int64 ids spread over the whole range


# ----------------------------------------------------------------------------- the cases
def listed():
    return [
        # A dashboard tile over a small table: four aggregates, latency only.
        {"name": "agg_10k", "kind": "aggregate", "n": 10_000, "where": "one", "nulls": False},
        # The same report over a third of a 100M-row month, with NULL scores and
        # a WHERE of two comparisons; a ragged row count.
        {"name": "agg_nulls_33m", "kind": "aggregate", "n": 33_333_331, "where": "two", "nulls": True},
        # The filter -> GROUP BY dept configuration (1M rows) as SQL text, the
        # result read on the host.
        {"name": "sql_group_1m", "kind": "sql", "n": 1_000_000, "query": "group"},
        # SELECT id, score WHERE two comparisons LIMIT m (nine in ten of the rows
        # that pass): mask, row list, two gathers.
        {"name": "rows_40m", "kind": "rows", "n": 40_000_000, "where": "two", "keep": 0.25},
        # The scan + top-k configuration's ORDER BY score DESC LIMIT 10.
        {"name": "topk_100m", "kind": "topk", "n": 100_000_000, "k": 10, "dtype": "f64", "desc": True,
         "nulls": False},
        # The join configuration: 1M-row build side kept resident, 100M probes.
        {"name": "join_inner_100m", "kind": "join", "n": 100_000_000, "build": 1_000_000, "keys": "dense",
         "type": "inner", "with_build": False},
        # A join of a query: both sides new, ids scattered, so the table hashes;
        # build and probe in one pass.
        {"name": "join_left_50m", "kind": "join", "n": 50_000_017, "build": 3_000_000, "keys": "scattered",
         "type": "left", "with_build": True},
        # The Zipf GROUP BY configuration: 100M rows of a resident table, 10M keys.
        {"name": "groupby_zipf_100m", "kind": "groupby", "n": 100_000_000, "domain": 10_000_000, "zipf": True,
         "keys": "dense", "nulls": False},
        # GROUP BY a 64-bit id (spread over the whole range), groups in id order.
        {"name": "groupby_ids_20m", "kind": "groupby", "n": 20_000_003, "domain": 1_000_000, "zipf": False,
         "keys": "scattered", "nulls": False},
        # 64 GROUP BY queries over log-uniform slices of one table, one graph.
        {"name": "batch_64", "kind": "batch", "n": 4_000_000, "queries": 64, "domain": 2_000, "zipf": True},
        # ORDER BY score DESC without LIMIT at the full-sort benchmark's size.
        {"name": "sort_100m", "kind": "sort", "n": 100_000_000, "op": "order", "dtype": "f64", "desc": True,
         "nulls": False},
        # 256 requests of the four serving templates at once: the request loop
        # under a backlog.
        {"name": "serve_256", "kind": "serve", "n": 20_000_000, "queries": 256},
    ]


def _log_int(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["aggregate", "sql", "rows", "topk", "join", "groupby", "groupby", "batch", "sort", "serve"])
    if kind == "aggregate":
        return {"kind": kind, "n": _log_int(rng, 10_000, 100_000_000), "where": rng.choice(["none", "one", "two"]),
                "nulls": rng.random() < 0.4}
    if kind == "sql":
        return {"kind": kind, "n": _log_int(rng, 10_000, 4_000_000), "query": rng.choice(sorted(SQL))}
    if kind == "rows":
        return {"kind": kind, "n": _log_int(rng, 100_000, 60_000_000), "where": rng.choice(["one", "two"]),
                "keep": round(rng.uniform(0.02, 0.9), 3)}
    if kind == "topk":
        return {"kind": kind, "n": _log_int(rng, 100_000, 100_000_000), "k": rng.choice([1, 10, 10, 25, 100]),
                "dtype": rng.choice(["f64", "i64"]), "desc": rng.random() < 0.6, "nulls": rng.random() < 0.25}
    if kind == "join":
        n = _log_int(rng, 1_000_000, 100_000_000)
        return {"kind": kind, "n": n, "build": _log_int(rng, 10_000, 4_000_000),
                "keys": rng.choice(["dense", "scattered"]), "type": rng.choice(["inner", "left", "semi", "anti"]),
                "with_build": rng.random() < 0.5}
    if kind == "groupby":
        n = _log_int(rng, 500_000, 60_000_000)
        return {"kind": kind, "n": n, "domain": _log_int(rng, 1_000, min(10_000_000, n // 4)),
                "zipf": rng.random() < 0.5, "keys": rng.choice(["dense", "scattered"]), "nulls": rng.random() < 0.2}
    if kind == "batch":
        return {"kind": kind, "n": _log_int(rng, 300_000, 5_000_000), "queries": rng.randint(16, 64),
                "domain": _log_int(rng, 200, 20_000), "zipf": rng.random() < 0.5}
    if kind == "sort":
        return {"kind": kind, "n": _log_int(rng, 100_000, 80_000_000), "op": rng.choice(["order", "order", "distinct"]),
                "dtype": rng.choice(["f64", "i64"]), "desc": rng.random() < 0.5, "nulls": rng.random() < 0.25}
    return {"kind": kind, "n": _log_int(rng, 1_000_000, 20_000_000), "queries": rng.randint(64, 256)}


# ----------------------------------------------------------------------------- data
def _gen(seed, *part):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(np.random.SeedSequence([seed, *part]).generate_state(1)[0]))
    return g


def _uniform(n, seed, part, scale=1.0):
    return torch.rand(n, dtype=torch.float64, device=DEV, generator=_gen(seed, part)).mul_(scale)


def _ints(lo, hi, n, seed, part):
    return torch.randint(lo, hi, (n,), dtype=torch.int64, device=DEV, generator=_gen(seed, part))


def _score(n, seed):
    return _uniform(n, seed, 3, 100.0)


def _salary(n, seed):
    return _ints(30_000, 200_001, n, seed, 4)


def _valid(n, seed, part, share=0.95):
    """Rows that hold a value, and the same as validity words (LSB first)."""
    ok = torch.rand(n, device=DEV, generator=_gen(seed, part)) < share
    words = torch.zeros((n + 63) // 64, dtype=torch.int64, device=DEV)
    padded = torch.nn.functional.pad(ok, (0, words.numel() * 64 - n)).view(-1, 64)
    for b in range(64):
        words |= padded[:, b].to(torch.int64) << b
    return ok, words


def _ranks(n, domain, zipf, seed):
    """n draws from 0..domain-1, uniform or Zipf(1.1), the ranks shuffled."""
    if not zipf:
        return _ints(0, domain, n, seed, 11)
    # Whole-number weights: their running sums, and so the draws, repeat exactly.
    weight = torch.arange(1, domain + 1, dtype=torch.float64, device=DEV).pow_(-1.1).mul_(2.0 ** 45).long()
    cdf = weight.cumsum(0)
    r = torch.searchsorted(cdf, _ints(0, int(cdf[-1]), n, seed, 11), right=True)
    return torch.randperm(domain, device=DEV, generator=_gen(seed, 12))[r]


_db = []


def _database():
    if not _db:
        _db.append(F.Database(0))
    return _db[0]


class State:
    """Inputs and handles of one case; drops its tables and handles with itself."""

    def __init__(self, case):
        self.case = case
        self.db = _database()
        self.tables = []
        self.server = None

    def table(self, name, cols):
        """A resident table from device tensors (their copies are the table's)."""
        name = f"{name}_{id(self)}"
        torch.cuda.synchronize()
        self.db.create_table_from_pointers(
            name, [(c, F.FLOAT64 if t.dtype == torch.float64 else F.INT64, t.data_ptr()) for c, t in cols.items()],
            len(next(iter(cols.values()))))
        self.db.synchronize()
        self.tables.append(name)
        return name

    def __del__(self):
        if self.server is not None:
            self.server.stop()
        for t in self.tables:
            self.db.drop_table(t)


# ----------------------------------------------------------------------------- aggregates
AGGS = [(F.AGG_COUNT_STAR, 0), (F.AGG_SUM, 0), (F.AGG_AVG, 1), (F.AGG_MAX, 0)]


def _where(kind, x=50.0, y=150_000):
    if kind == "none":
        return []
    one = [ops.cmp(0, F.GT, x)]
    return one if kind == "one" else one + [ops.cmp(1, F.LT, y), ops.AND()]


def _aggregate_prepare(s, n, where, nulls, seed):
    s.score, s.salary = _score(n, seed), _salary(n, seed)
    s.ok = None
    s.cols = [s.score, s.salary]
    if nulls:
        s.ok, words = _valid(n, seed, 5)
        s.cols[0] = (s.score, words)
    s.prog = _where(where)


def _aggregate_run(s):
    out = ops.aggregate(s.db, s.cols, s.case["n"], s.prog, AGGS)
    return {"f": out.view(torch.float64).view(-1, 4)[:, 0], "i": out.view(torch.int64).view(-1, 4)[:, 1:3]}


def _aggregate_exact(s):
    ok = torch.ones_like(s.score, dtype=torch.bool) if s.ok is None else s.ok
    keep = torch.ones_like(ok)
    if s.case["where"] != "none":
        keep = ok & (s.score > 50.0)
    if s.case["where"] == "two":
        keep &= s.salary < 150_000
    v, w = s.score[keep & ok], s.salary[keep]
    return {"f": torch.stack([v.new_zeros(()), v.sum(), w.sum().double() / w.numel(), v.max()]), "i": None}


# ----------------------------------------------------------------------------- SQL text
SQL = {
    "group": "SELECT dept, COUNT(*), SUM(score), AVG(salary) FROM {t} WHERE score > 50 GROUP BY dept ORDER BY dept",
    "aggregate": "SELECT COUNT(*), SUM(score), AVG(salary), MAX(score) FROM {t} WHERE score > 50 AND salary < 150000",
    "sum": "SELECT SUM(score) FROM {t}",
    "topk": "SELECT id, score FROM {t} ORDER BY score DESC LIMIT 10",
}


def _sql_prepare(s, n, query, seed):
    s.host = W.table_t(n, seed=seed)
    name = f"t_{id(s)}"
    s.db.create_table(name, s.host)
    s.db.synchronize()
    s.tables.append(name)
    s.text = SQL[query].format(t=name)


def _sql_run(s):
    r = s.db.sql(s.text)
    cols = [r.column(j) for j in range(len(r.columns))]
    return [np.array([int(v[1:]) for v in c]) if isinstance(c, list) else c for c in cols]


def _sql_exact(s):
    t = s.host
    score, salary, q = t["score"], t["salary"], s.case["query"]
    if q == "group":
        keep = score > 50
        code = t["dept"].codes[keep]
        cnt = np.bincount(code, minlength=12)
        s0 = np.bincount(code, weights=score[keep], minlength=12)
        s2 = np.bincount(code, weights=salary[keep].astype(np.float64), minlength=12)
        return [None, None, s0, s2 / cnt]
    if q == "aggregate":
        keep = (score > 50) & (salary < 150_000)
        return [None, np.array([score[keep].sum()]), np.array([salary[keep].mean()]), np.array([score[keep].max()])]
    if q == "sum":
        return [np.array([score.sum()])]
    return [None, np.sort(score)[::-1][:10].copy()]


# ----------------------------------------------------------------------------- SELECT rows WHERE LIMIT
def _rows_prepare(s, n, where, keep, seed):
    s.score, s.salary = _score(n, seed), _salary(n, seed)
    s.id = torch.arange(n, dtype=torch.int64, device=DEV)
    side = math.sqrt(keep) if where == "two" else keep
    s.x, s.y = 100.0 * (1.0 - side), int(30_000 + 170_000 * side)
    s.prog = _where(where, s.x, s.y)
    s.cols = [s.score, s.salary] if where == "two" else [s.score]
    s.limit = int(0.9 * keep * n)


def _rows_run(s):
    n = s.case["n"]
    mask = ops.filter_mask(s.db, s.cols, n, s.prog)
    rows, count = ops.compact(s.db, mask, n)
    m = min(s.limit, int(count.item()))
    return {"count": count, "id": ops.gather(s.db, s.id, rows, m)[0], "score": ops.gather(s.db, s.score, rows, m)[0]}


def _rows_exact(s):
    keep = s.score > s.x
    if s.case["where"] == "two":
        keep &= s.salary < s.y
    return {"count": None, "id": None, "score": s.score[keep][:s.limit]}


# ----------------------------------------------------------------------------- top-k and full sort
def _order_prepare(s, n, dtype, nulls, seed):
    col = _score(n, seed) if dtype == "f64" else _salary(n, seed)
    s.col = (col, _valid(n, seed, 5)[1]) if nulls else col
    s.rows = torch.zeros(n, dtype=torch.int32, device=DEV)


def _topk_run(s):
    return ops.topk(s.db, s.col, s.case["n"], s.case["k"], s.case["desc"])


def _sort_run(s):
    n = s.case["n"]
    if s.case["op"] == "order":
        return ops.sort(s.db, s.col, n, s.case["desc"], rows=s.rows)
    return ops.distinct(s.db, s.col, n, rows=s.rows)  # rows past the count stay as they are


# ----------------------------------------------------------------------------- join
JOIN = {"inner": F.JOIN_INNER, "left": F.JOIN_LEFT, "semi": F.JOIN_SEMI, "anti": F.JOIN_ANTI}


def _join_prepare(s, n, build, keys, with_build, seed):
    s.bkey = torch.randperm(build, device=DEV, generator=_gen(seed, 1))
    s.payload = _ints(0, 1_000_000, build, seed, 2)
    s.pkey = _ints(0, 2 * build, n, seed, 3)
    if keys == "scattered":
        s.bkey, s.pkey = s.bkey * SCATTER + 3, s.pkey.mul_(SCATTER).add_(3)
    s.value = _uniform(n, seed, 4) if s.case["type"] in ("semi", "anti") else None
    s.join = None if with_build else ops.HashTable(s.db, s.bkey, s.payload, build)


def _join_run(s):
    c = s.case
    h = s.join or ops.HashTable(s.db, s.bkey, s.payload, c["build"])
    out = h.probe_agg(s.pkey, c["n"], JOIN[c["type"]], value=s.value)
    if s.join is None:
        h.free()
    ints = out.view(torch.int64)
    return {"count": ints[0], "sum_payload": ints[1], "sum_value": out.view(torch.float64)[2], "payload_rows": ints[3]}


def _join_exact(s):
    total = 0.0
    if s.value is not None:
        key = s.pkey if s.case["keys"] == "dense" else (s.pkey - 3) // SCATTER
        total = s.value[(key < s.case["build"]) == (s.case["type"] == "semi")].sum()
    return {"count": None, "sum_payload": None, "sum_value": total, "payload_rows": None}


# ----------------------------------------------------------------------------- int64-key GROUP BY
def _group_columns(rec):
    """The columns of fdb_group_i64 records (40 bytes each)."""
    ints, floats = rec.view(torch.int64).view(-1, 5), rec.view(torch.float64).view(-1, 5)
    return {"key": ints[:, 0], "count": ints[:, 1], "sum": floats[:, 2], "min": floats[:, 3], "max": floats[:, 4]}


def _groupby_prepare(s, n, domain, zipf, keys, nulls, seed):
    key, v = _ranks(n, domain, zipf, seed), _uniform(n, seed, 13)
    s.cap = domain + 1
    s.ok = None
    if keys == "dense":  # resident table: its zone maps bound the keys
        name = s.table("g", {"key": key, "v": v})
        s.key, s.v = s.db.column(name, "key"), s.db.column(name, "v")
    else:
        s.key, s.v = key.mul_(MIX), v
    if nulls:
        s.ok, words = _valid(n, seed, 5)
        s.v = (v, words)
    s.out = torch.zeros(40 * s.cap, dtype=torch.uint8, device=DEV)  # records past the group count stay zero
    s.ordered = torch.zeros_like(s.out) if keys == "scattered" else s.out
    s.ngroups = torch.empty(1, dtype=torch.int64, device=DEV)


def _groupby_run(s):
    n = s.case["n"]
    ops.group_by_i64(s.db, s.key, s.v, n, capacity=s.cap, out=s.out, ngroups=s.ngroups)
    if s.case["keys"] == "scattered":  # ORDER BY key; a direct-addressed table gives its groups in key order
        m = int(s.ngroups.item())
        rec = s.out.view(torch.int64).view(-1, 5)[:m]
        order = ops.sort(s.db, rec[:, 0].contiguous(), m, False)
        torch.index_select(rec, 0, order, out=s.ordered.view(torch.int64).view(-1, 5)[:m])
    return {"groups": s.ngroups, **_group_columns(s.ordered)}


def _group_exact(key, v, ok):
    """Per key in ascending order: SUM, MIN, MAX of v (NULL values left out)."""
    keys, inv = torch.unique(key, return_inverse=True)
    m = keys.numel()
    if ok is not None:
        inv, v = inv[ok], v[ok]
    total = torch.zeros(m, dtype=torch.float64, device=DEV).index_add_(0, inv, v)
    lo = torch.full((m,), math.inf, dtype=torch.float64, device=DEV).scatter_reduce_(0, inv, v, "amin")
    hi = torch.full((m,), -math.inf, dtype=torch.float64, device=DEV).scatter_reduce_(0, inv, v, "amax")
    empty = torch.isinf(lo)
    lo[empty] = math.nan
    hi[empty] = math.nan
    return keys, total, lo, hi


def _groupby_exact(s, seed):
    c = s.case
    key = _ranks(c["n"], c["domain"], c["zipf"], seed)
    if c["keys"] == "scattered":
        key.mul_(MIX)
    _, *cols = _group_exact(key, _uniform(c["n"], seed, 13), s.ok)
    cols = [torch.nn.functional.pad(x, (0, s.cap - x.numel())) for x in cols]
    return {"groups": None, "key": None, "count": None, **dict(zip(("sum", "min", "max"), cols))}


# ----------------------------------------------------------------------------- batched GROUP BY
def _slices(case, seed):
    """(first row, rows) of the batch's queries: log-uniform slices of the table."""
    r = np.random.default_rng([seed, 21])
    n = case["n"]
    rows = np.exp(r.uniform(math.log(min(10_000, n // 8)), math.log(n), case["queries"])).astype(np.int64)
    return [(int(r.integers(0, n - m + 1)), int(m)) for m in rows]


def _batch_prepare(s, n, domain, zipf, seed):
    s.key, s.v = _ranks(n, domain, zipf, seed), _uniform(n, seed, 13)
    s.slices = _slices(s.case, seed)
    s.batch = ops.GroupByBatch(s.db, [(s.key[a:a + m], s.v[a:a + m], m) for a, m in s.slices],
                               capacity=[domain + 1] * len(s.slices))


def _batch_run(s):
    """Every query's groups in key order, padded to the largest possible group
    count with key INT64_MAX (the other fields of padding are zero)."""
    s.batch.run()
    rec = torch.stack([g for g, _ in s.batch.outs])
    count = torch.cat([c for _, c in s.batch.outs])
    ints = rec.view(torch.int64).view(len(s.slices), -1, 5)
    live = torch.arange(ints.shape[1], device=DEV) < count[:, None]
    key, order = torch.where(live, ints[:, :, 0], torch.iinfo(torch.int64).max).sort(dim=1)
    live = live.gather(1, order)
    ints = torch.where(live[:, :, None], ints.gather(1, order[:, :, None].expand(-1, -1, 5)), 0)
    floats = ints.view(torch.float64)
    return {"key": key, "count": ints[:, :, 1], "sum": floats[:, :, 2], "min": floats[:, :, 3],
            "max": floats[:, :, 4]}


def _batch_exact(s):
    width = s.case["domain"] + 1
    out = {k: torch.zeros(len(s.slices), width, dtype=torch.float64, device=DEV) for k in ("sum", "min", "max")}
    for i, (a, m) in enumerate(s.slices):
        keys, *cols = _group_exact(s.key[a:a + m], s.v[a:a + m], None)
        for k, c in zip(("sum", "min", "max"), cols):
            out[k][i, :keys.numel()] = c
    return {"key": None, "count": None, **out}


# ----------------------------------------------------------------------------- serving
def _serve_prepare(s, n, queries, seed):
    s.score, s.salary = _score(n, seed), _salary(n, seed)
    s.dept = torch.randint(0, 12, (n,), dtype=torch.int32, device=DEV, generator=_gen(seed, 2))
    build = max(1_000, n // 20)
    s.bkey = torch.randperm(build, device=DEV, generator=_gen(seed, 6))
    s.payload = _ints(0, 1_000_000, build, seed, 7)
    s.pkey, s.pval = _ints(0, 2 * build, n, seed, 8), _uniform(n, seed, 9)
    s.join = ops.HashTable(s.db, s.bkey, s.payload, build)
    r = np.random.default_rng([seed, 22])
    s.qs = []
    for i in range(queries):
        kind = i % 4
        m, x = int(n * 10 ** (-3 * r.random())), float(100 * r.random())
        if kind == S.SERVE_COUNT:
            q = S.count_query(s.score.data_ptr(), m, x)
        elif kind == S.SERVE_GROUP:
            q = S.group_query(s.score.data_ptr(), s.dept.data_ptr(), s.salary.data_ptr(), 12, m, x)
        elif kind == S.SERVE_JOIN:
            q = S.join_query(s.pkey.data_ptr(), s.pval.data_ptr(), s.join._h.value, m, x)
        else:
            q = S.topk_query(s.score.data_ptr(), m, x, k=10)
        s.qs.append(q)
    torch.cuda.synchronize()
    s.server = S.Server(s.db, max_batch=128, slots=2)


def _serve_run(s):
    tickets = [s.server.submit(q) for q in s.qs]
    res = [s.server.wait(t) for t in tickets]
    kinds = [q.kind for q in s.qs]
    groups = [r for r, k in zip(res, kinds) if k == S.SERVE_GROUP]
    return {"count": np.array([r.count for r, k in zip(res, kinds) if k != S.SERVE_GROUP], dtype=np.int64),
            "payload": np.array([r.sum_payload for r, k in zip(res, kinds) if k == S.SERVE_JOIN], dtype=np.int64),
            "rows": np.array([r.rows[:10] for r, k in zip(res, kinds) if k == S.SERVE_TOPK], dtype=np.int64),
            "group_count": np.array([r.group_count[:12] for r in groups], dtype=np.int64),
            "group_score": np.array([r.group_sum0[:12] for r in groups], dtype=np.float64),
            "group_salary": np.array([r.group_sum2[:12] for r in groups], dtype=np.int64)}


def _serve_exact(s):
    sums = []
    for q in s.qs:
        if q.kind == S.SERVE_GROUP:
            keep = s.score[:q.nrows] > q.threshold
            sums.append(torch.zeros(12, dtype=torch.float64, device=DEV).index_add_(
                0, s.dept[:q.nrows][keep].long(), s.score[:q.nrows][keep]))
    return {"count": None, "payload": None, "rows": None, "group_count": None, "group_salary": None,
            "group_score": torch.stack(sums) if sums else torch.zeros(0, dtype=torch.float64)}


# ----------------------------------------------------------------------------- entry points
def prepare(case, seed):
    s, c = State(case), case
    if c["kind"] == "aggregate":
        _aggregate_prepare(s, c["n"], c["where"], c["nulls"], seed)
    elif c["kind"] == "sql":
        _sql_prepare(s, c["n"], c["query"], seed)
    elif c["kind"] == "rows":
        _rows_prepare(s, c["n"], c["where"], c["keep"], seed)
    elif c["kind"] in ("topk", "sort"):
        _order_prepare(s, c["n"], c["dtype"], c["nulls"], seed)
    elif c["kind"] == "join":
        _join_prepare(s, c["n"], c["build"], c["keys"], c["with_build"], seed)
    elif c["kind"] == "groupby":
        _groupby_prepare(s, c["n"], c["domain"], c["zipf"], c["keys"], c["nulls"], seed)
    elif c["kind"] == "batch":
        _batch_prepare(s, c["n"], c["domain"], c["zipf"], seed)
    else:
        _serve_prepare(s, c["n"], c["queries"], seed)
    return s


_RUN = {"aggregate": _aggregate_run, "sql": _sql_run, "rows": _rows_run, "topk": _topk_run, "sort": _sort_run,
        "join": _join_run, "groupby": _groupby_run, "batch": _batch_run, "serve": _serve_run}


def run(state):
    return _RUN[state.case["kind"]](state)


def exact(case, seed):
    if case["kind"] in ("topk", "sort"):
        return None  # row numbers
    s = prepare(case, seed)
    if case["kind"] == "groupby":
        return _groupby_exact(s, seed)
    return {"aggregate": _aggregate_exact, "sql": _sql_exact, "rows": _rows_exact, "join": _join_exact,
            "batch": _batch_exact, "serve": _serve_exact}[case["kind"]](s)


def work(case):
    """Input columns read once, results written once."""
    c, n = case, case["n"]
    if c["kind"] == "aggregate":
        b = 16 * n + (n // 8 if c["nulls"] else 0) + 4 * 32
    elif c["kind"] == "sql":
        b = {"group": 20, "aggregate": 16, "sum": 8, "topk": 8}[c["query"]] * n
    elif c["kind"] == "rows":
        m = int(n * c["keep"])
        b = (16 if c["where"] == "two" else 8) * n + 2 * 16 * m
    elif c["kind"] == "topk":
        b = 8 * n + (n // 8 if c["nulls"] else 0) + 4 * c["k"]
    elif c["kind"] == "sort":
        b = 8 * n + (n // 8 if c["nulls"] else 0) + 4 * n
    elif c["kind"] == "join":
        b = 8 * n + (8 * n if c["type"] in ("semi", "anti") else 0) + 16 * c["build"]
    elif c["kind"] == "groupby":
        b = 16 * n + (n // 8 if c["nulls"] else 0) + 40 * min(n, c["domain"])
    elif c["kind"] == "batch":
        b = sum(16 * m + 40 * min(m, c["domain"]) for _, m in _slices(c, 0))
    else:
        b = (8 + 8 + 4 + 8 + 8) * n  # each column of the tables read once
    return {"bytes": b, "flops": 0}
