"""The hash route of the keyed (GROUP BY) aggregation's pass 1 on the sm_100a
kernels: the mirror of PageFlow's ``KeyedAggregate.pass1`` (operators/
aggregate.py:1511-1563) for aggregates over plain columns.

One chunk's rows are reduced to one row per group:

  hash      each row's grouping hash, the linear hash of its key columns'
            packed words with the deterministic coefficients of
            ``_make_key_coeffs`` (:529-548; pf_group_hash)
  groups    the unique hashes ascending, one representative of every key
            column per group, and each aggregate's partial (pf_unique_reduce:
            radix sort of the hashes, segment reduction; a key column travels
            as its packed words)
  buckets   with B > 1, each group's bucket (``_bucket_ids``) and the groups
            per bucket, on the host and on the device (pf_hash_buckets)

A chunk whose rows share groups (two a group or more) takes hash and groups
in one read of its rows (pf_keyed_pass1_read, _emit: a place of a hash table
holds every accumulator of its group); one of mostly single rows, or of
columns that the table does not hold (floats' min and max, two-dimensional or
narrow values), the steps above.  After a chunk of integer columns whose groups
were too many for the table, the object's next seven take the steps without the
attempt.  A float64 SUM is exact to its own rounding in the one read, and added
as a segmented tree by the steps.

Aggregates: ``('sum', col)``, ``('count', None)`` (every row) or
``('count', col)`` (the rows whose value is not the null -64), ``('min',
col)``, ``('max', col)`` (folded from 0, as the reference's partial is) and
``('avg', col)`` (its state: [sum of every row, count of the non-null
ones]), each as the reference's pass 1 computes it.  SUM of an
integer column is exact in int64 (the reference sums through a float64
bincount, :395-398, which equals it while every partial stays below 2^53).
"""
from __future__ import annotations

import ctypes
import os
from typing import Dict, List, Sequence, Tuple

import torch

from . import _native
from ._native import check, lib, ptr, stream_of
from .sorted_run_merge import reduce_tick_slice

NULL = -64   # the reference's null value (constants.null)
COEFF_BASE_SEED = int(os.environ.get('TQP_HASH_SEED', '2029')) & 0x7FFF_FFFF_FFFF_FFFF


def packed_width(col: torch.Tensor) -> int:
    """int64 words of a (N, W) tensor's rows (_packed_width, :477-479)."""
    return (col.shape[1] * col.element_size() + 7) // 8


def make_key_coeffs(key_tensors: Sequence[torch.Tensor], device) -> List[torch.Tensor]:
    """The reference's coefficients: a local generator on the device seeded
    with the base seed, one randint(2, 10_000_000) vector per packed key
    column (_make_key_coeffs, :529-548)."""
    g = torch.Generator(device=device)
    g.manual_seed(COEFF_BASE_SEED)
    return [torch.randint(2, 10_000_000, (packed_width(c),), dtype=torch.int64, device=device,
                          generator=g) for c in key_tensors]


def _as_2d(col: torch.Tensor) -> torch.Tensor:
    return col.unsqueeze(1) if col.dim() < 2 else col


def group_hash(key_tensors: Sequence[torch.Tensor], coeffs: Sequence[torch.Tensor]) -> torch.Tensor:
    """Each row's grouping hash (_hash_key_columns, :551-564), one launch."""
    keys = [_as_2d(k).contiguous() for k in key_tensors]
    n = keys[0].shape[0]
    dev = keys[0].device
    out = torch.empty(n, dtype=torch.int64, device=dev)
    coeffs = [c.contiguous() for c in coeffs]
    cols = (ctypes.c_void_p * len(keys))(*[ptr(k) for k in keys])
    rb = (ctypes.c_int * len(keys))(*[k.shape[1] * k.element_size() for k in keys])
    cf = (ctypes.c_void_p * len(keys))(*[ptr(c) for c in coeffs])
    check(lib().pf_group_hash(cols, rb, cf, len(keys), n, ptr(out), stream_of(dev)), "group_hash")
    return out


def hash_buckets(hashes: torch.Tensor, B: int):
    """(bucket int32, counts on the host, counts on the device)."""
    n = hashes.numel()
    dev = hashes.device
    bucket = torch.empty(n, dtype=torch.int32, device=dev)
    counts = torch.empty(B, dtype=torch.int64, device=dev)
    check(lib().pf_hash_buckets(ptr(hashes), n, B, ptr(bucket), ptr(counts), stream_of(dev)),
          "hash_buckets")
    return bucket, counts.tolist(), counts


def _pack_words(col: torch.Tensor) -> torch.Tensor:
    """A (N, W) tensor's rows as int64 words, zero-padded (_pack_as_int64)."""
    n, w = col.shape
    rb = w * col.element_size()
    raw = col.contiguous().view(torch.uint8).reshape(n, rb)
    tb = (rb + 7) // 8 * 8
    if tb == rb:
        return raw.view(torch.int64)
    buf = torch.zeros(n, tb, dtype=torch.uint8, device=col.device)
    buf[:, :rb] = raw
    return buf.view(torch.int64)


def _unpack_words(words: torch.Tensor, like: torch.Tensor) -> torch.Tensor:
    n = words.shape[0]
    rb = like.shape[1] * like.element_size()
    raw = words.contiguous().view(torch.uint8).reshape(n, -1)[:, :rb].contiguous()
    return raw.view(like.dtype).reshape(n, like.shape[1])


# accumulators, column kinds and outputs of pf_keyed_pass1_read and _emit
(_KA_WORD, _KA_COUNT, _KA_NULLS, _KA_SUM_I, _KA_SUM_F, _KA_MIN, _KA_MAX, _KA_SUM_ERR) = range(8)
_KK = {torch.int64: 0, torch.int32: 1, torch.float64: 2, torch.float32: 3}
(_KO_WORD, _KO_I64, _KO_I32, _KO_F64, _KO_F32, _KO_I64_MAX0, _KO_I32_MAX0, _KO_COUNT, _KO_AVG_I,
 _KO_AVG_F) = range(10)
_MAX_ACCS, _MAX_OUTS, _MAX_KEYS, _MAX_B = 15, 40, 8, 4096
_MAX_EXPECT = 1 << 24
# chunks that go straight to the general route after one whose groups were too many
# for the one-read route's table: the attempt costs 4M rows of as many groups 210 of
# 1440 us, which a table's other chunks, mostly alike, need not pay
_GENERAL_CHUNKS = 7


class KeyedPass1:
    """Pass 1 of a keyed aggregation over plain columns: ``key_ids`` group
    the rows (``emitted_ids``, default all of them, are carried out as key
    representatives); ``aggs`` is a list of (op, column id or None)."""

    def __init__(self, key_ids: Sequence[int], aggs: Sequence[Tuple[str, int]],
                 emitted_ids: Sequence[int] | None = None):
        self.key_ids = list(key_ids)
        self.emitted = list(self.key_ids if emitted_ids is None else emitted_ids)
        self.aggs = list(aggs)
        for op, _ in self.aggs:
            if op not in ('sum', 'count', 'min', 'max', 'avg'):
                raise NotImplementedError(f"KeyedPass1: aggregate {op!r}")
        self._coeffs = None
        self._laid = None   # (column types and widths, _layout's answer for them)
        self._general = 0   # chunks left that take the general route unasked

    def pass1(self, columns: Dict[int, torch.Tensor], B: int = 1):
        """``[hash] + keys + values`` of one chunk (hash ascending, unique),
        and the buckets (None at B = 1 or with no group, else (bucket,
        counts, counts_t)), as KeyedAggregate.pass1 returns them."""
        keys = [_as_2d(columns[k]) for k in self.key_ids]
        if self._coeffs is None:
            self._coeffs = make_key_coeffs(keys, keys[0].device)
        out, general = None, self._general
        if general > 0:
            self._general = general - 1
        else:
            try:
                out = self._one_read(columns, keys, B)
            except torch.OutOfMemoryError:
                # no room for its table (3 GB for 16M groups of eight accumulators):
                # the general route works a column at a time
                pass
        if out is not None:
            return out
        out = self._hash_and_sort(columns, keys)
        buckets = None
        if B > 1 and out[0].numel() > 0:
            buckets = hash_buckets(out[0], B)
        return out, buckets

    def _layout(self, keys, cols):
        """What pf_keyed_pass1_read does for columns of these types and widths:
        its accumulators and outputs without their pointers, which column each
        accumulator reads, and each result column's dtype and width; None when
        it does not take them."""
        accs, source, where = [], [], {}

        def acc(op, cid=None, kind=0, row_bytes=0, word=0):
            at = where.get((op, cid, word))
            if at is None:
                at = where[(op, cid, word)] = len(accs)
                accs.append(_native.KeyedAcc(op, kind, row_bytes, word, None))
                source.append(None if cid is None else (op == _KA_WORD, cid))
            return at

        def summed(cid, kind, fp):
            s = acc(_KA_SUM_F if fp else _KA_SUM_I, cid, kind)
            if cols[cid].dtype == torch.float64:
                acc(_KA_SUM_ERR, None, kind, 0, s)   # its rounding errors
            return s

        outs, dest, results = [], [], []

        def out(*fields):
            outs.append(_native.KeyedOut(*fields, None))
            dest.append(len(results))

        for e in self.emitted:
            k = keys[e]
            rb = k.shape[1] * k.element_size()
            for w in range(packed_width(k)):
                out(_KO_WORD, acc(_KA_WORD, e, 0, rb, w), 0, 0, rb, w)
            results.append((k.dtype, k.shape[1]))
        for op, cid in self.aggs:
            v = None if cid is None else cols[cid]
            fp = v is not None and v.dtype.is_floating_point
            kind = 0 if v is None else _KK[v.dtype]
            if op == 'count':
                c = acc(_KA_COUNT)
                if v is None:
                    out(_KO_I64, c, 0, 0, 0, 0)
                else:
                    out(_KO_COUNT, c, acc(_KA_NULLS, cid, kind), 0, 0, 0)
                results.append((torch.int64, 1))
            elif op == 'avg':
                s = summed(cid, kind, fp)
                out(_KO_AVG_F if fp else _KO_AVG_I, s, acc(_KA_COUNT), acc(_KA_NULLS, cid, kind),
                    0, 0)
                results.append((torch.float64, 2))
            elif op == 'sum':
                s = summed(cid, kind, fp)
                out({torch.float64: _KO_F64, torch.float32: _KO_F32}.get(v.dtype, _KO_I64), s, 0,
                    0, 0, 0)
                results.append((v.dtype if fp else torch.int64, 1))
            elif fp:
                return None
            else:
                wide = v.dtype == torch.int64
                m = acc(_KA_MIN if op == 'min' else _KA_MAX, cid, kind)
                # MAX folds into a zeroed partial (operator_utils.py:365-369)
                out((_KO_I64 if wide else _KO_I32) if op == 'min' else
                    (_KO_I64_MAX0 if wide else _KO_I32_MAX0), m, 0, 0, 0, 0)
                results.append((v.dtype, 1))
        if len(accs) > _MAX_ACCS or len(outs) > _MAX_OUTS:
            return None
        return (bytes((_native.KeyedAcc * max(1, len(accs)))(*accs)), source,
                bytes((_native.KeyedOut * max(1, len(outs)))(*outs)), dest, results)

    def _layout_of(self, keys, cols):
        """_layout's answer, kept for the last types and widths (it depends on
        nothing else); another thread may keep its own meanwhile."""
        sig = (tuple((k.dtype, k.shape[1]) for k in keys),
               tuple(v.dtype for v in cols.values()))
        laid = self._laid
        if laid is None or laid[0] != sig:
            laid = self._laid = (sig, self._layout(dict(zip(self.key_ids, keys)), cols))
        return laid[1]

    def _one_read(self, columns, keys, B=1):
        """pass1 by pf_keyed_pass1_read, or None when a column's type or shape or
        the number of groups is not its."""
        n, dev = keys[0].shape[0], keys[0].device
        if (n == 0 or dev.type != 'cuda' or len(keys) > _MAX_KEYS or not 1 <= B <= _MAX_B
                or B & (B - 1) or not set(self.emitted) <= set(self.key_ids)
                or any(k.dim() != 2 or k.shape[0] != n or k.shape[1] == 0 or k.device != dev
                       for k in keys)):
            return None
        cols = {cid: columns[cid] for _, cid in self.aggs if cid is not None}
        if any(v.dim() != 1 or v.shape[0] != n or v.device != dev or v.dtype not in _KK
               for v in cols.values()):
            return None
        lay = self._layout_of(keys, cols)
        if lay is None:
            return None
        acc_bytes, source, out_bytes, dest, results = lay
        L = lib()
        nk, na, no = len(keys), len(source), len(dest)
        keys = [k.contiguous() for k in keys]
        held = {True: dict(zip(self.key_ids, keys)),
                False: {cid: v.contiguous() for cid, v in cols.items()}}
        coeffs = [c.contiguous() for c in self._coeffs]
        accs = (_native.KeyedAcc * max(1, na)).from_buffer_copy(acc_bytes)
        for a, src in zip(accs, source):
            if src is not None:
                a.src = held[src[0]][src[1]].data_ptr()
        kcols = (ctypes.c_void_p * nk)(*[k.data_ptr() for k in keys])
        kbytes = (ctypes.c_int * nk)(*[k.shape[1] * k.element_size() for k in keys])
        kcoeffs = (ctypes.c_void_p * nk)(*[c.data_ptr() for c in coeffs])
        groups, crowded = ctypes.c_int64(), ctypes.c_int64()
        expect = 0
        with torch.cuda.device(dev):
            st = stream_of(dev)
            while True:
                ws_bytes = L.pf_keyed_pass1_workspace(n, na, expect)
                ws = _native.workspace(ws_bytes, dev)
                check(L.pf_keyed_pass1_read(kcols, kbytes, kcoeffs, nk, n, accs, na, expect,
                                            ws.data_ptr(), ws_bytes, st), "keyed_pass1")
                # the outputs are made while the rows are read
                room = L.pf_keyed_pass1_groups(n, na, expect)
                res = [torch.empty((room, w) if w > 1 else room, dtype=dt, device=dev)
                       for dt, w in results]
                outs = (_native.KeyedOut * max(1, no)).from_buffer_copy(out_bytes)
                for o, i in zip(outs, dest):
                    o.dst = res[i].data_ptr()
                h = torch.empty(room, dtype=torch.int64, device=dev)
                bucket = counts = None
                host_counts = (ctypes.c_int64 * B)()
                if B > 1:
                    bucket = torch.empty(room, dtype=torch.int32, device=dev)
                    counts = torch.empty(B, dtype=torch.int64, device=dev)
                sort_ws = None
                while True:
                    check(L.pf_keyed_pass1_emit(
                        n, accs, na, expect, outs, no, h.data_ptr(), B, ptr(bucket), ptr(counts),
                        host_counts, ctypes.byref(groups), ctypes.byref(crowded), ws.data_ptr(),
                        ws_bytes, ptr(sort_ws), crowded.value, st), "keyed_pass1")
                    if not crowded.value:
                        break
                    sort_ws = _native.workspace(crowded.value, dev)
                g = groups.value
                if g >= 0:
                    break
                # more groups than the table holds, about -g: once more into
                # one for them, unless most rows are a group of their own (the
                # general route is as fast then, at a smaller workspace)
                if expect or -g > 2 * n // 3 or -g > _MAX_EXPECT:
                    # (float sums are rounded otherwise there: a chunk's own groups
                    # decide, not those of another)
                    if not any(v.dtype.is_floating_point for v in cols.values()):
                        self._general = _GENERAL_CHUNKS
                    return None
                expect = -g
                ws = res = outs = h = bucket = counts = None   # before the larger ones
        buckets = (bucket[:g], list(host_counts), counts) if B > 1 and g > 0 else None
        return [h[:g]] + [t[:g] for t in res], buckets

    def _hash_and_sort(self, columns, keys):
        """pass1's columns by the grouping hash of every row, a radix sort
        and a segmented reduction a column (pf_group_hash, pf_unique_reduce)."""
        h = group_hash(keys, self._coeffs)
        vals, ops, post, at = [], [], [], {}

        def column(name, make, op):
            """The value column `name`'s place, made once: AVG(x)'s sum is
            SUM(x)'s."""
            if name not in at:
                at[name] = len(vals)
                vals.append(make())
                ops.append(op)
            return at[name]

        emitted = [_as_2d(columns[k]) for k in self.emitted]
        for e in emitted:
            vals.append(_pack_words(e))
            ops.append('amax')   # every row of a group holds the same key
        n = h.numel()

        def summed(cid):
            v = columns[cid]
            # integer sums in int64, as the reference's result
            return v if v.dtype in (torch.float32, torch.float64) else v.to(torch.int64)

        def non_null(cid):
            # COUNT(x) counts the rows whose x is not the null value
            # (operator_utils.py:384-385); COUNT(*) every row
            return (columns[cid] != NULL).to(torch.int64)

        def ranged(cid):
            v = columns[cid]
            return v if v.dtype in (torch.float32, torch.float64, torch.int64, torch.int32) \
                else v.to(torch.int64)

        for op, cid in self.aggs:
            if op == 'count':
                j = (column('rows', lambda: torch.ones(n, dtype=torch.int64, device=h.device),
                            'sum') if cid is None else
                     column(('non_null', cid), lambda: non_null(cid), 'sum'))
                post.append(('count', j, None))
            elif op == 'avg':
                # the state [SUM(x), COUNT(x)] (aggregate.py:249-250, 323-336):
                # the sum over every row, the count over the non-null ones
                post.append(('avg', column(('sum', cid), lambda: summed(cid), 'sum'),
                             column(('non_null', cid), lambda: non_null(cid), 'sum')))
            elif op == 'sum':
                post.append((op, column(('sum', cid), lambda: summed(cid), 'sum'), None))
            else:
                post.append((op, column((op, cid), lambda: ranged(cid),
                                        {'min': 'amin', 'max': 'amax'}[op]), None))
        u, red = reduce_tick_slice(h, vals, ops)
        key_reps = []
        for i, e in enumerate(emitted):
            rep = _unpack_words(red[i], e)
            key_reps.append(rep.squeeze(1) if rep.shape[1] == 1 else rep)
        agg_vals = []
        for op, j, j2 in post:
            if op == 'avg':
                agg_vals.append(torch.stack([red[j].to(torch.float64),
                                             red[j2].to(torch.float64)], dim=1))
            elif op == 'max':
                # MAX folds into a zeroed partial (a scatter_reduce into zeros
                # that includes them, operator_utils.py:365-369), so a group
                # whose values are all negative has the partial 0
                agg_vals.append(torch.clamp_min(red[j], 0))
            else:
                agg_vals.append(red[j])
        return [u] + key_reps + agg_vals
