"""The performance cases of pageflow_b200: the work that a program built on it
has it do, each through the package's public entry points.

  join       JoinAggregate.run: the fused partition -> join -> group-by
  partition  tqpkernels.partition_sort of one tick, narrowed by host_out
  hashjoin   tqpkernels.join_unique_hash, then both sides' columns gathered
  semi       tqpkernels.join_semi_anti with or without a residual comparison
  keyed      KeyedPass1 over a table's ticks, their runs merged (both passes of
             a keyed GROUP BY)
  slab       DenseAggregationSlab over a table's ticks
  encode     encode_pages_device: output columns compressed on the device
  paged      PagedScan over compressed pages in pinned host memory, its kept
             rows joined and grouped
  batch      BatchJoinAggregate: many uneven joins in one persistent launch
  serve      serve.Server over resident dimension tables

A case is a dict of plain values.  listed() gives the named ones, draw(rng)
one more of the same ranges, prepare(case, seed) what a program holds before
the call, run(state) one pass, work(case) the bytes a pass cannot do without,
exact(case, seed) the results by plain torch in 64 bits.

A case's sizes hold for every seed: the seed orders the rows and draws the
values, and how many rows match, are kept or form a group is the case's.
"""
import dataclasses
import math

import numpy as np
import torch

from pageflow_b200 import datagen, paged, serve, tqpkernels
from pageflow_b200.aggregation_slab import DenseAggregationSlab
from pageflow_b200.batch import BatchJoinAggregate, Instance
from pageflow_b200.gather import index_select_many
from pageflow_b200.join_aggregate import JoinAggregate
from pageflow_b200.keyed_aggregate import KeyedPass1
from pageflow_b200.sorted_run_merge import merge_sorted_unique_runs_inplace

DEVICE = "cuda"


def listed():
    return [
        # the small workload (250 thousand x 1 million rows, 25 groups): one
        # morsel's join, where launches and waits count
        {"name": "join_small", "kind": "join", "n_build": 250_000, "n_probe": 1_000_000,
         "groups": 25, "disc": True},
        # a mid-sized join of odd sizes, one value column and no discount
        {"name": "join_ragged", "kind": "join", "n_build": 3_000_017, "n_probe": 20_000_003,
         "groups": 100_003, "disc": False},
        # the scale workload: 150M x 600M rows, 1.5M groups
        {"name": "join_scale", "kind": "join", "n_build": 150_000_000, "n_probe": 600_000_000,
         "groups": 1_500_000, "disc": True},
        # one 128 MiB-key tick partitioned with columns of three widths
        {"name": "partition_tick", "kind": "partition", "rows": 16_777_213, "B": 8, "sel": 1.0,
         "select_first": False},
        # one bucket pair's inner join and the gather of its output columns
        {"name": "hashjoin_gather", "kind": "hashjoin", "n_build": 1_500_000, "n_probe": 6_000_000,
         "keys": 1},
        # EXISTS with a <> residual (op 1) on odd sizes
        {"name": "semi_residual", "kind": "semi", "n_build": 400_003, "n_probe": 2_500_001, "op": 1,
         "anti": False},
        # a two-column GROUP BY over four ticks: pass 1 a tick, runs merged
        {"name": "keyed_ticks", "kind": "keyed", "rows": 4_000_000, "ticks": 4, "groups": 250_000,
         "B": 8, "float": False},
        # a dense group-by over four ticks into 1.5M direct-addressed groups
        {"name": "slab_ticks", "kind": "slab", "rows": 4_000_000, "ticks": 4,
         "capacity": 1_500_000},
        # three result columns compressed into pages on the device
        {"name": "encode_pages", "kind": "encode", "rows": 8_000_000, "page_rows": 131_072},
        # compressed pages decoded on arrival, filtered, joined and grouped
        {"name": "paged_join", "kind": "paged", "rows": 16_000_000, "n_build": 1_000_000,
         "groups": 1000},
        # 48 instances of the batching workload, replayed as a graph
        {"name": "batch_48", "kind": "batch", "instances": 48, "max_build": 4_000_000},
        # a burst of mixed requests against the resident tables
        {"name": "serve_burst", "kind": "serve", "requests": 32, "fact_rows": 100_000_000,
         "max_keys": 2_000_000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["join", "join", "partition", "hashjoin", "semi", "keyed", "slab", "encode",
                       "paged", "batch", "serve"])
    if kind == "join":
        nb = _log(rng, 20_000, 20_000_000)
        return {"kind": kind, "n_build": nb, "n_probe": nb * rng.randint(2, 10) + rng.randint(0, 99),
                "groups": _log(rng, 5, nb // 20), "disc": rng.random() < 0.6}
    if kind == "partition":
        sel = rng.choice([1.0, round(rng.uniform(0.05, 0.95), 3)])
        return {"kind": kind, "rows": _log(rng, 100_000, 30_000_000), "B": rng.choice([2, 4, 8]),
                "sel": sel, "select_first": sel < 0.25}
    if kind == "hashjoin":
        nb = _log(rng, 20_000, 6_000_000)
        return {"kind": kind, "n_build": nb, "n_probe": nb * rng.randint(1, 6) + rng.randint(0, 99),
                "keys": rng.choice([1, 2])}
    if kind == "semi":
        nb = _log(rng, 20_000, 6_000_000)
        return {"kind": kind, "n_build": nb, "n_probe": nb * rng.randint(1, 6) + rng.randint(0, 99),
                "op": rng.randint(0, 5), "anti": rng.random() < 0.5}
    if kind == "keyed":
        rows = _log(rng, 300_000, 6_000_000)
        return {"kind": kind, "rows": rows, "ticks": rng.randint(1, 4),
                "groups": _log(rng, 4, rows // 4), "B": rng.choice([1, 8, 16]),
                "float": rng.random() < 0.5}
    if kind == "slab":
        return {"kind": kind, "rows": _log(rng, 200_000, 6_000_000), "ticks": rng.randint(1, 5),
                "capacity": _log(rng, 8, 3_000_000)}
    if kind == "encode":
        return {"kind": kind, "rows": _log(rng, 200_000, 12_000_000),
                "page_rows": rng.choice([16_384, 65_536, 131_072])}
    if kind == "paged":
        rows = _log(rng, 1_000_000, 16_000_000)
        return {"kind": kind, "rows": rows, "n_build": _log(rng, 50_000, 1_000_000),
                "groups": _log(rng, 10, 500)}
    if kind == "batch":
        return {"kind": kind, "instances": rng.randint(8, 48),
                "max_build": _log(rng, 50_000, 4_000_000)}
    return {"kind": kind, "requests": rng.randint(4, 32), "fact_rows": _log(rng, 10_000_000, 100_000_000),
            "max_keys": _log(rng, 200_000, 2_000_000)}


def _order(g, n):
    return torch.randperm(n, generator=g, device=DEVICE)


def _rng(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


def _ints(g, lo, hi, n, dtype=torch.int64):
    return torch.randint(lo, hi, (n,), generator=g, device=DEVICE, dtype=dtype)


# ---- join ---------------------------------------------------------------------

def _join_inputs(c, seed):
    """Unique build keys 1..n permuted; a tenth of the foreign keys miss."""
    g = _rng(seed)
    nb, np_ = c["n_build"], c["n_probe"]
    key = _order(g, nb) + 1
    group = ((key + seed) % c["groups"]).to(torch.int32)
    fk = _ints(g, 1, nb + max(1, nb // 9) + 1, np_)
    price = _ints(g, 90_000, 10_500_001, np_)
    disc = _ints(g, 0, 11, np_) if c["disc"] else None
    return key, group, fk, price, disc


def _join_prepare(c, seed):
    cols = _join_inputs(c, seed)
    # a fixed launch configuration, so that two programs run the same launches
    plan = JoinAggregate(c["n_build"], c["n_probe"], 0, c["groups"], DEVICE, autotune=False)
    return plan, cols


def _join_run(state):
    plan, cols = state
    return plan.run(*cols)


def _grouped(group_of, value, groups):
    """(occupied groups, int64 sums, counts) of rows with group_of >= 0."""
    hit = group_of >= 0
    gid = group_of[hit]
    sums = torch.zeros(groups, dtype=torch.int64, device=DEVICE).index_add_(0, gid, value[hit])
    counts = torch.bincount(gid, minlength=groups)
    keys = torch.nonzero(counts).flatten()
    return keys, sums[keys], counts[keys]


def _group_of(key, group, fk):
    order = torch.argsort(key)
    at = torch.searchsorted(key[order], fk).clamp_(max=key.numel() - 1)
    row = order[at]
    return torch.where(key[row] == fk, group[row].to(torch.int64), -1)


def _join_exact(c, seed):
    if c["n_probe"] > 250_000_000:
        return None
    key, group, fk, price, disc = _join_inputs(c, seed)
    value = price * 100 if disc is None else price * (100 - disc)
    return _grouped(_group_of(key, group, fk), value, c["groups"])


# ---- partition ------------------------------------------------------------------

def _partition_prepare(c, seed):
    g = _rng(seed)
    n = c["rows"]
    row = _order(g, n)
    cols = [row % (n // 4) + 1, _ints(g, 90_000, 10_500_001, n),
            _ints(g, 8035, 10592, n, torch.int32), _ints(g, 0, 3, n, torch.int8)]
    mask, kept = None, n
    if c["sel"] < 1.0:
        mask = row * 2_654_435_761 % 1_000_003 < int(c["sel"] * 1_000_003)
        kept = int(mask.sum())
    host = torch.empty(c["B"] + 5, dtype=torch.int64, pin_memory=True)
    return c, cols, mask, kept, host


def _partition_run(state):
    c, cols, mask, kept, host = state
    outs = tqpkernels.partition_sort(cols, [0] * len(cols), 0, mask, kept, 0, c["B"],
                                     c["select_first"], host)
    counts = host[:c["B"]].tolist()
    buckets = []
    for t in outs:
        unit = 512 // math.gcd(t.element_size(), 512)   # buckets start on 512-byte units
        at = 0
        for n in counts:
            buckets.append(t[at:at + n])
            at += -(-n // unit) * unit
    return buckets


# ---- join cores ----------------------------------------------------------------

def _hashjoin_prepare(c, seed):
    g = _rng(seed)
    nb, np_ = c["n_build"], c["n_probe"]
    build = [_order(g, nb) + 1]
    probe = [_order(g, np_) * 1_000_003 % (nb + nb // 9) + 1]   # a tenth misses
    if c["keys"] == 2:   # (order, line)-like pairs
        build = [(build[0] >> 2), (build[0] & 3)]
        probe = [(probe[0] >> 2), (probe[0] & 3)]
    bcols = [_ints(g, 0, 1 << 40, nb), _ints(g, 0, 25, nb, torch.int32)]
    pcols = [_ints(g, 90_000, 10_500_001, np_), _ints(g, 8035, 10592, np_, torch.int32)]
    return build, probe, bcols, pcols, torch.empty(2, dtype=torch.int64, pin_memory=True)


def _hashjoin_run(state):
    build, probe, bcols, pcols, host = state
    b, p = tqpkernels.join_unique_hash(build, probe, host)
    n = int(host[0])
    b, p = b[:n], p[:n]
    return [b, p, index_select_many(bcols, b), index_select_many(pcols, p)]


def _semi_prepare(c, seed):
    g = _rng(seed)
    nb, np_ = c["n_build"], c["n_probe"]
    # two build rows a key, half of the probe keys without one
    b, p = _order(g, nb), _order(g, np_)
    build, probe = b // 2 + 1, p * 1_000_003 % nb + 1
    bval, pval = b * 7919 % 1009 + seed % 100, p * 104_729 % 1009 + seed % 100
    return c, build, probe, bval, pval, torch.empty(2, dtype=torch.int64, pin_memory=True)


def _semi_run(state):
    c, build, probe, bval, pval, host = state
    rows = tqpkernels.join_semi_anti(build, probe, bval if c["op"] else None,
                                     pval if c["op"] else None, c["op"], c["anti"], host)
    return rows[:int(host[0])]


# ---- keyed aggregation ----------------------------------------------------------

KEYED_AGGS = [("sum", 2), ("count", None), ("avg", 2), ("min", 3), ("max", 3)]
KEYED_OPS = ["amax", "amax", "sum", "sum", "sum", "amin", "amax"]


def _keyed_inputs(c, seed):
    g = _rng(seed)
    ticks = []
    for _ in range(c["ticks"]):
        n = c["rows"]
        price = _ints(g, 90_000, 10_500_001, n)
        group = _order(g, n) % c["groups"]
        ticks.append({0: (group >> 2) + 1, 1: (group & 3).to(torch.int32),
                      2: price.to(torch.float64) / 100 if c["float"] else price,
                      3: _ints(g, 8035, 10592, n)})
    return ticks


def _keyed_prepare(c, seed):
    ticks = _keyed_inputs(c, seed)
    room = c["groups"]
    kinds = [torch.int64, torch.int32, torch.float64 if c["float"] else torch.int64, torch.int64,
             (torch.float64, 2), torch.int64, torch.int64]
    bufs = [torch.empty((room, k[1]), dtype=k[0], device=DEVICE) if isinstance(k, tuple)
            else torch.empty(room, dtype=k, device=DEVICE) for k in kinds]
    return c, ticks, KeyedPass1([0, 1], KEYED_AGGS), torch.empty(room, dtype=torch.int64,
                                                               device=DEVICE), bufs


def _keyed_run(state):
    c, ticks, pass1, key_buf, bufs = state
    m, buckets = 0, []
    for t in ticks:
        out, bk = pass1.pass1(t, c["B"])
        cols = [v.to(b.dtype) for v, b in zip(out[1:], bufs)]
        m = merge_sorted_unique_runs_inplace(key_buf, bufs, m, out[0], cols, KEYED_OPS)
        if bk is not None:
            buckets += [bk[0], bk[2]]
    return [key_buf[:m]] + [b[:m] for b in bufs] + buckets


def _keyed_exact(c, seed):
    ticks = _keyed_inputs(c, seed)
    col = [torch.cat([t[i] for t in ticks]) for i in range(4)]
    # the grouping hash: each key word times a coefficient of the seeded generator
    g = torch.Generator(device=DEVICE).manual_seed(2029)
    co = [torch.randint(2, 10_000_000, (1,), dtype=torch.int64, device=DEVICE, generator=g)
          for _ in range(2)]
    h, at = torch.unique(col[0] * co[0] + col[1].to(torch.int64) * co[1], return_inverse=True)
    n = h.numel()

    def total(v):
        return torch.zeros(n, dtype=v.dtype, device=DEVICE).index_add_(0, at, v)

    def most(v, op):
        return torch.zeros(n, dtype=v.dtype, device=DEVICE).scatter_reduce_(
            0, at, v, op, include_self=False)

    count = torch.bincount(at, minlength=n)
    s = total(col[2])
    return [h, most(col[0], "amax"), most(col[1].to(torch.int64), "amax"), s, count,
            torch.stack([s.to(torch.float64), count.to(torch.float64)], dim=1),
            most(col[3], "amin"), most(col[3], "amax")]


# ---- dense slab ------------------------------------------------------------------

SLAB_SPECS = [(torch.int64, ()), (torch.float64, ()), (torch.int64, ()), (torch.int32, ())]
SLAB_OPS = ["sum", "sum", "sum", "amax"]


def _slab_inputs(c, seed):
    g = _rng(seed)
    ticks = []
    for _ in range(c["ticks"]):
        n = c["rows"]
        price = _ints(g, 90_000, 10_500_001, n)
        ticks.append((_order(g, n) * c["capacity"] // n + 1,
                      [price, price.to(torch.float64) / 100,
                       torch.ones(n, dtype=torch.int64, device=DEVICE),
                       _ints(g, 8035, 10592, n, torch.int32)]))
    return ticks


def _slab_prepare(c, seed):
    return c, _slab_inputs(c, seed)


def _slab_run(state):
    c, ticks = state
    slab = DenseAggregationSlab(1, c["capacity"], torch.int64, SLAB_SPECS, SLAB_OPS, DEVICE)
    for keys, values in ticks:
        slab.add(keys, values)
    return slab.finish()


def _slab_exact(c, seed):
    ticks = _slab_inputs(c, seed)
    at = torch.cat([t[0] for t in ticks]) - 1
    v = [torch.cat([t[1][i] for t in ticks]) for i in range(4)]
    n = c["capacity"]
    full = [torch.zeros(n, dtype=x.dtype, device=DEVICE).index_add_(0, at, x) for x in v[:3]]
    full.append(torch.zeros(n, dtype=torch.int64, device=DEVICE).scatter_reduce_(
        0, at, v[3].to(torch.int64), "amax", include_self=False))
    keys = torch.nonzero(torch.bincount(at, minlength=n)).flatten()
    return keys + 1, [x[keys] for x in full]


# ---- pages -------------------------------------------------------------------------

def _encode_prepare(c, seed):
    g = _rng(seed)
    n = c["rows"]
    # dates ascend inside a run of 1M rows; their steps are the same for every
    # seed (a page's bytes depend on them), the first day is not
    run = torch.arange(n, device=DEVICE) // 1_000_000
    date = torch.sort(run * 4096 + _ints(_rng(7), 0, 2500, n))[0] - run * 4096
    cols = [_ints(g, 1, 200_000_001, n), (date + 8035 + seed % 57).to(torch.int32),
            _ints(g, 1, 51, n)]
    rows = list(range(0, n, c["page_rows"])) + [n]
    return cols, rows


def _encode_run(state):
    cols, rows = state
    out = []
    for col in cols:
        pages, offsets = paged.encode_pages_device(col, rows)
        out += [pages, torch.tensor(offsets)]
    return out


def _paged_inputs(c, seed):
    spec = paged.PagedSpec(seed, c["rows"], c["n_build"], 0.8, 131_072, 9000, 9384)
    g = _rng(seed)
    key = _order(g, c["n_build"]) + 1
    return spec, key, _ints(g, 0, c["groups"], c["n_build"], torch.int32)


def _paged_prepare(c, seed):
    spec, key, group = _paged_inputs(c, seed)
    table = paged.PagedTable.generate(spec)
    scan = paged.PagedScan(table, "date", spec.date_lo, spec.date_hi, "fk",
                           capacity_rows=c["rows"] // 3)
    return c, scan, key, group


def _paged_run(state):
    c, scan, key, group = state
    parts = scan.run()
    stats = parts.read_stats()
    n = stats["rows"]
    # a bucket's rows come in no fixed order: the join's groups are the result
    plan = JoinAggregate(c["n_build"], n, 0, c["groups"], DEVICE, autotune=False)
    keys, sums, counts = plan.run(key, group, parts.columns["fk"][:n], parts.columns["price"][:n])
    return keys, sums, counts, parts.bucket_offsets, n


# ---- batch and serve ------------------------------------------------------------------

def _batch_specs(c):
    return datagen.batch_workload(c["instances"], build_range=(1_000, c["max_build"]),
                                  group_range=(4, 1_000_000))


def _batch_prepare(c, seed):
    specs = [dataclasses.replace(s, seed=seed * 1_000_003 + s.index) for s in _batch_specs(c)]
    insts = [Instance(*datagen.gen_batch_instance(s, DEVICE), 0, s.n_groups) for s in specs]
    batch = BatchJoinAggregate(insts, DEVICE)
    return batch, batch.graph()


def _batch_run(state):
    batch, graph = state
    graph.replay()
    return [batch.slab(i) for i in range(len(batch.instances))]


def _serve_spec(c, seed):
    keys = serve._logspace_int(c["max_keys"] / 2000, c["max_keys"], 8)
    groups = tuple(min(g, k) for g, k in zip((16, 100, 1000, 2000, 5000, 10_000, 15_000, 20_000),
                                             keys))
    return serve.ServeSpec(seed, c["max_keys"], keys, groups, c["fact_rows"], 0.8, 100_000,
                           c["fact_rows"], 0.01, 0.50, c["fact_rows"] * 20 + (1 << 30))


def _serve_prepare(c, seed):
    spec = _serve_spec(c, seed)
    device = torch.device(DEVICE, torch.cuda.current_device())
    dims, fact = serve.Dimensions(spec, device), serve.FactPool(spec, device)
    server = serve.Server(dims, fact, spec.budget_bytes, device, pinned_bytes=1 << 28)
    requests = serve.make_requests(spec, c["requests"], seed=4)
    # a request's groups go to its own place in one table of results
    ends = np.cumsum([spec.dim_groups[r.dim] for r in requests])
    return server, requests, ends


def _serve_run(state):
    server, requests, ends = state
    done = server.run(requests).requests
    out = np.zeros((3, ends[-1]), np.int64)
    for r, end in zip(done, ends):
        at = end - server.dims.spec.dim_groups[r.dim]
        for k in range(3):
            out[k, at:at + r.n_groups_out] = r.result[k]
    return out


_PREPARE = {"join": _join_prepare, "partition": _partition_prepare, "hashjoin": _hashjoin_prepare,
            "semi": _semi_prepare, "keyed": _keyed_prepare, "slab": _slab_prepare,
            "encode": _encode_prepare, "paged": _paged_prepare, "batch": _batch_prepare,
            "serve": _serve_prepare}
_RUN = {"join": _join_run, "partition": _partition_run, "hashjoin": _hashjoin_run,
        "semi": _semi_run, "keyed": _keyed_run, "slab": _slab_run, "encode": _encode_run,
        "paged": _paged_run, "batch": _batch_run, "serve": _serve_run}
_EXACT = {"join": _join_exact, "keyed": _keyed_exact, "slab": _slab_exact}


def prepare(case, seed):
    return case["kind"], _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state[0]](state[1])


def exact(case, seed):
    """None for row orders, pages and request streams: whole numbers whose
    order and bytes are the result."""
    f = _EXACT.get(case["kind"])
    return None if f is None else f(case, seed)


def work(case):
    c, kind = case, case["kind"]
    if kind == "join":
        b = 12 * c["n_build"] + (24 if c["disc"] else 16) * c["n_probe"] + 24 * c["groups"]
    elif kind == "partition":
        kept = c["sel"] * c["rows"]
        b = 21 * c["rows"] + 29 * kept + (c["rows"] if c["sel"] < 1 else 0)
    elif kind == "hashjoin":
        hit = 0.9 * c["n_probe"]
        b = 8 * c["keys"] * (c["n_build"] + c["n_probe"]) + 12 * c["n_build"] \
            + 12 * c["n_probe"] + (16 + 24) * hit
    elif kind == "semi":
        b = (16 if c["op"] else 8) * (c["n_build"] + c["n_probe"]) + 4 * c["n_probe"]
    elif kind == "keyed":
        groups = min(c["groups"], c["rows"])
        b = c["ticks"] * 28 * c["rows"] + 68 * groups
    elif kind == "slab":
        b = c["ticks"] * 36 * c["rows"] + 29 * c["capacity"]
    elif kind == "encode":
        # 8 + 4 + 8 bytes a row read, pages of about 28, 8 and 6 bits written
        b = 26 * c["rows"]
    elif kind == "paged":
        # pages of about 8 bytes a row, 15% of the rows kept
        b = 8 * c["rows"] + 0.15 * 32 * c["rows"] + 12 * c["n_build"]
    elif kind == "batch":
        b = sum(12 * s.n_build + 16 * s.n_probe + 16 * s.n_groups for s in _batch_specs(c))
    else:
        spec = _serve_spec(c, 4)
        # a date every row, key and value of the quarter that passes
        b = sum(r.n_rows * (4 + 16 * 0.25) for r in serve.make_requests(spec, c["requests"], seed=4))
    return {"bytes": float(b), "flops": 0.0}
