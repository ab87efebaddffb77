// The batched join -> group-by: many independent instances of uneven size in
// one persistent launch fed by a device work queue.
//
// Layout (the workspace, laid out by pf_batch_prepare):
//   header       epoch, work counters, item totals, error word
//   descriptors  per instance: its columns, table region, slab, item ranges
//   remaining    per instance: build items not yet done
//   checks       per instance: a run's matched rows and what its packed sums
//                are checked by
//   flags        per instance: how its runs go (below), kept from run to run
//   tables       per instance: a compact table (compact.cuh) where its groups
//                leave an entry room, else 2 x build rows 16-byte slots {key,
//                group | tag}; a region holds either
//   packed       per instance and group: {count, sum} in one word
//   slabs        per instance, n_groups (sum, count) int64 pairs
//
// Work items, instance by instance: its build rows in items of BITEM rows,
// then its probe rows in items of `pitem` rows (so the tables in use at any
// time are those of the few instances in flight, which stay in L2).  A block
// takes the next item from the counter; a probe item waits (bounded) until
// its instance's build items are all done.  Those items were taken before it,
// by blocks that are running, so the wait always ends.  The compact tables
// are cleared by each run (22 bytes a build row written); a 16-byte slot is
// free for this run when its tag is below the run's epoch, and the claim is an
// atomicMax of the tag.
//
// What bounds it: L2's rate of requests.  A probe row costs one table sector and
// one RED, where 16-byte slots half full took two or three dependent reads and a
// group's (sum, count) pair two REDs: 48 instances (29M build, 290M probe rows,
// FKs of Zipf 0, 0.8 and 1.2) 8.7 -> 5.2 ms, 8 of up to 50K rows 285 -> 90 us.
// One instance of 2M x 20M rows and 20 groups 548 -> 260 us.  Its value and 1 go into the
// group's packed word, or, for the groups a block meets often (skewed keys),
// through a cache in shared memory flushed into the slab at the item's end.
// The values are offset by 2^(b - 1) to take negative ones, b bits each.  What
// the packed words hold is checked after the run, instance by instance, as in
// join_direct.cu: every offset value in [0, 2^b), the words' counts add up to
// the rows put into them, and the sum of the values is bounded, or else some
// sum may have left its field.  k_batch_sums adds the packed words to the slab
// and decides; an instance that fails, or whose hashes crowd its compact table,
// is run again in the same call (k_batch<true>: two words a group, 16-byte
// slots) and goes that way in later runs of the batch from the start.
#include <algorithm>
#include <map>
#include <mutex>
#include <type_traits>
#include <vector>

#include "agg.cuh"
#include "compact.cuh"

namespace pf {
namespace {

constexpr int BT2 = 256;
#ifndef PF_BATCH_BV
#define PF_BATCH_BV 2
#endif
#ifndef PF_BATCH_MINB
#define PF_BATCH_MINB 4
#endif
// probe rows a thread takes at a time, at four blocks a SM (62 registers): 48
// instances 5.1 ms, 1 row at five blocks 5.6, at six 5.5
constexpr int BV = PF_BATCH_BV;
constexpr size_t BATCH_SMEM = sizeof(OwnSums);
constexpr int BATCH_MAX_Q = 23;     // 256 MiB tables, 0.4 full at most
constexpr double BATCH_LOAD = 0.4;
constexpr int SUM_CHUNK = 4096;     // groups a block of k_batch_sums adds up at a time

constexpr int BITEM = 4096;
// Probe rows of an item: more rows an item, fewer of its barriers, flushes and
// waits; fewer, and a small batch still has items for every block (8 instances
// of up to 50K build rows, 1M probe rows: 140 us at 16384, 94 at 4096; 24 of up
// to 400K, 20M rows: 623 and 809).
long long probe_item(unsigned long long probe_rows) {
  return probe_rows <= 2000000 ? 4096 : probe_rows <= 5000000 ? 8192 : 16384;
}
constexpr unsigned WAIT_LIMIT = 1u << 24;  // polls of a probe item's wait (x ~0.5 us)

struct Desc {
  const long long* bkey;
  const int* bgrp;
  long long nb;
  const long long* pfk;
  const long long* pval;
  long long np;
  long long gmin, ng;
  unsigned long long toff;   // first slot of the table region
  unsigned long long tcap;   // 16-byte slots
  unsigned long long soff;   // first (sum, count) pair of the slab
  long long item0;           // first work item (its build items, then its probe items)
  long long nbi;             // build items
  long long pitem;           // probe rows of an item
  long long chunk0;          // first chunk of k_batch_sums
  unsigned long long region; // slots of the table region
  int q, gbits, dbits;       // compact table (q = 0: none)
  int sbits, vbits;          // packed word: bits of the sum, of an offset value
};

// How an instance's runs go: bits of its flags word.
constexpr unsigned WIDE_SUMS = 1, WIDE_TABLE = 2, REDO = 4;

struct Check {
  unsigned long long matched;  // probe rows that found their build row
  unsigned long long rows;     // rows put into packed words
  unsigned long long high;     // their offset values >> 20, added up
  unsigned long long counts;   // the packed words' counts, added up
  unsigned bad_value, crowded;
};

struct Header {
  unsigned epoch;
  unsigned n_redo;
  unsigned long long counter, counter2;  // items of the first pass, of the second
  unsigned chunks_done, pad;
  long long n_build_items, n_items, n_chunks;
  int n_inst;
  int pad2;
  unsigned long long error;
};

struct Slot {
  unsigned long long key;
  unsigned long long tagged;  // (tag << 32) | group offset
};

struct Sizes {
  unsigned long long table_slots, cleared_slots, slab_pairs, items, chunks;
  long long pitem;
};

struct Layout {
  Header* header;
  Desc* desc;
  unsigned* remaining;
  Check* check;
  unsigned* flags;
  int* imap;  // work item -> instance
  int* cmap;  // chunk of groups -> instance
  Slot* tables;
  unsigned long long* packed;
  unsigned long long* slabs;
};

Layout layout(char* base, int n, const Sizes& z, size_t* used) {
  Arena a(base, ~(size_t)0);
  Layout l{};
  l.header = a.take<Header>(1);
  l.desc = a.take<Desc>(std::max(n, 1));
  l.remaining = a.take<unsigned>(std::max(n, 1));
  l.check = a.take<Check>(std::max(n, 1));
  l.flags = a.take<unsigned>(std::max(n, 1));
  l.imap = a.take<int>(std::max<unsigned long long>(z.items, 1));
  l.cmap = a.take<int>(std::max<unsigned long long>(z.chunks, 1));
  l.tables = a.take<Slot>(std::max<unsigned long long>(z.table_slots, 1));
  l.packed = a.take<unsigned long long>(std::max<unsigned long long>(z.slab_pairs, 1));
  l.slabs = a.take<unsigned long long>(2 * std::max<unsigned long long>(z.slab_pairs, 1));
  if (used) *used = a.used;
  return l;
}

// An instance's compact table (q = 0: none) and the slots of its region.
unsigned long long table_of(long long nb, long long ng, int* q, int* gbits, int* dbits,
                            unsigned long long* tcap) {
  *q = 0;
  *tcap = 0;
  if (nb < 1) return 0;
  // 16-byte slots: a quarter full to 64 MiB (a sector of two in ten full), half
  // full past it
  *tcap = (64LL * nb <= (64LL << 20) ? 4ULL : 2ULL) * (unsigned long long)nb;
  ct_size(nb, std::max<long long>(ng, 1), BATCH_MAX_Q, BATCH_LOAD, BATCH_LOAD, q, gbits, dbits);
  const unsigned long long least = 2ULL * (unsigned long long)nb;
  // groups numbered far past the rows would need a table far larger than them
  if (*q && (2ULL << *q) > 4 * least + 256) *q = 0;
  if (!*q) return *tcap;
  *tcap = least;  // only where the compact table fails
  return std::max(least, 2ULL << *q);
}

Sizes totals(const pf_batch_instance* in, int n) {
  Sizes z{};
  unsigned long long probes = 0;
  for (int i = 0; i < n; ++i)
    if (in[i].n_build > 0) probes += (unsigned long long)std::max<int64_t>(in[i].n_probe, 0);
  z.pitem = probe_item(probes);
  for (int i = 0; i < n; ++i) {
    const long long nb = std::max<int64_t>(in[i].n_build, 0);
    const long long np = nb > 0 ? std::max<int64_t>(in[i].n_probe, 0) : 0;
    const long long ng = std::max<int64_t>(in[i].n_groups, 0);
    int q, gbits, dbits;
    unsigned long long tcap;
    const unsigned long long slots = table_of(nb, ng, &q, &gbits, &dbits, &tcap);
    z.table_slots += slots;
    if (q) z.cleared_slots += slots;
    z.slab_pairs += (unsigned long long)ng;
    z.items += (unsigned long long)((nb + BITEM - 1) / BITEM + (np + z.pitem - 1) / z.pitem);
    z.chunks += (unsigned long long)((ng + SUM_CHUNK - 1) / SUM_CHUNK);
  }
  return z;
}

// Run start: bump the epoch, zero the counters, the error word, the checks, the
// sums and the compact tables, and set every instance's remaining build items.
__global__ void __launch_bounds__(BT2) k_batch_reset(Header* h, const Desc* d,
                                                     unsigned* remaining, Check* check, int n,
                                                     Slot* tables,
                                                     unsigned long long cleared_slots,
                                                     unsigned long long* packed,
                                                     unsigned long long* slabs,
                                                     unsigned long long pairs) {
  const unsigned long long tid = (unsigned long long)blockIdx.x * BT2 + threadIdx.x;
  const unsigned long long stride = (unsigned long long)gridDim.x * BT2;
  if (tid == 0) {
    h->epoch += 1;
    h->n_redo = 0;
    h->counter = h->counter2 = 0;
    h->chunks_done = 0;
    h->error = 0;
  }
  for (unsigned long long i = tid; i < (unsigned long long)n; i += stride) {
    remaining[i] = (unsigned)d[i].nbi;
    check[i] = Check{0, 0, 0, 0, 0, 0};
  }
  const ulonglong2 zero = make_ulonglong2(0ULL, 0ULL);
  ulonglong2* t = reinterpret_cast<ulonglong2*>(tables);
  for (unsigned long long i = tid; i < cleared_slots; i += stride) t[i] = zero;
  ulonglong2* s = reinterpret_cast<ulonglong2*>(slabs);
  for (unsigned long long i = tid; i < pairs; i += stride) {
    s[i] = zero;
    packed[i] = 0;
  }
}

// A wide table's slots lie two a sector; a key's home sector.
__device__ __forceinline__ unsigned first_sector(uint64_t h, unsigned long long cap) {
  return (unsigned)(((h >> 32) * (cap >> 1)) >> 32);
}

// One build row into a table of 16-byte slots.
__device__ __forceinline__ bool wide_insert(const Desc& D, Slot* tables, unsigned epoch,
                                            unsigned long long key, uint32_t goff) {
  unsigned p = 2 * first_sector(mix64(key), D.tcap);
  for (unsigned long long left = D.tcap; left > 0; --left) {
    Slot* sl = tables + D.toff + p;
    unsigned* tag = reinterpret_cast<unsigned*>(&sl->tagged) + 1;
    if (atomicMax(tag, epoch) < epoch) {
      *reinterpret_cast<ulonglong2*>(sl) =
          make_ulonglong2(key, ((unsigned long long)epoch << 32) | goff);
      return true;
    }
    if (++p == D.tcap) p = 0;
  }
  return false;
}

// A key in a table of 16-byte slots, x its home sector p: -2 not there, -1
// there without a group, else the group.
__device__ __forceinline__ long long wide_lookup(const Desc& D, const Slot* tables,
                                                 unsigned epoch, unsigned long long key,
                                                 unsigned p, CtBucket x) {
  for (unsigned long long probes = 0; probes < D.tcap >> 1; ++probes) {
#pragma unroll
    for (int j = 0; j < 4; j += 2) {
      if ((uint32_t)(x.e[j + 1] >> 32) != epoch) return -2;
      if (x.e[j] == key) {
        const uint32_t go = (uint32_t)x.e[j + 1];
        return go == 0xffffffffu ? -1 : (long long)go;
      }
    }
    if (++p == D.tcap >> 1) p = 0;
    x = ct_load(reinterpret_cast<const unsigned long long*>(tables + D.toff + 2ULL * p));
  }
  return -2;
}

struct BatchArgs {
  Header* h;
  const Desc* d;
  const int* imap;
  unsigned* remaining;
  Check* check;
  const unsigned* flags;
  Slot* tables;
  unsigned long long* packed;
  unsigned long long* slabs;
  unsigned long long* stats;
};

// The probe rows [lo, hi) of an instance, BV rows a thread a step: every value
// and home sector (or slot) loaded before the first is looked at, the next
// step's keys on their way (48 instances 5170 -> 5077 us).
// PACK: a row's value and 1 in one packed word, else in the slab's two.
template <bool COMPACT, bool PACK>
__device__ __forceinline__ void probe_rows(const Desc& D, const BatchArgs& a, unsigned epoch,
                                           Own& own, long long lo, long long hi,
                                           unsigned& matched, unsigned& rows,
                                           unsigned long long& high, bool& outside) {
  unsigned long long* slab = a.slabs + 2 * D.soff;
  unsigned long long* packed = a.packed + D.soff;
  const CompactTable t{reinterpret_cast<unsigned long long*>(a.tables + D.toff), D.q, D.gbits,
                       D.dbits};
  // D lies in memory that the compiler must take for changed by every atomic
  const long long* pfk = (const long long*)D.pfk;
  const long long* pval = (const long long*)D.pval;
  __builtin_assume(__isGlobal(pfk));
  __builtin_assume(__isGlobal(pval));
  const int vbits = D.vbits;
  const unsigned long long one = 1ULL << D.sbits;
  const unsigned long long bias = 1ULL << (vbits - 1);
  unsigned long long next[BV];
#pragma unroll
  for (int k = 0; k < BV; ++k) {
    const long long i = lo + k * BT2 + threadIdx.x;
    next[k] = i < hi ? (unsigned long long)__ldcs(pfk + i) : 0ULL;
  }
  auto step = [&](long long i0, auto first) {
    unsigned long long key[BV], hash[BV];
    long long value[BV], g[BV];
    bool live[BV];
#pragma unroll
    for (int k = 0; k < BV; ++k) {
      const long long i = i0 + k * BT2 + threadIdx.x;
      live[k] = i < hi;
      key[k] = next[k];
      const long long j = i + BT2 * BV;
      next[k] = j < hi ? (unsigned long long)__ldcs(pfk + j) : 0ULL;
    }
#pragma unroll
    for (int k = 0; k < BV; ++k) {
      const long long i = i0 + k * BT2 + threadIdx.x;
      value[k] = live[k] ? __ldcs(pval + i) : 0;
    }
    if (COMPACT) {
      CtBucket b[BV];
#pragma unroll
      for (int k = 0; k < BV; ++k) {
        hash[k] = ct_hash((long long)key[k]);
        b[k] = ct_load(ct_home(t, hash[k]));
      }
#pragma unroll
      for (int k = 0; k < BV; ++k) {
        g[k] = -2;
        if (!live[k]) continue;
        bool more;
        const unsigned long long want = ct_want(t, hash[k]);
        unsigned long long e = ct_among(t, b[k], want, &more);
        if (more) e = ct_walk(t, hash[k], want);
        if (e != CT_EMPTY) g[k] = ct_group(t, e);
      }
    } else {
      CtBucket x[BV];
#pragma unroll
      for (int k = 0; k < BV; ++k) {
        hash[k] = first_sector(mix64(key[k]), D.tcap);
        x[k] = ct_load(
            reinterpret_cast<const unsigned long long*>(a.tables + D.toff + 2ULL * hash[k]));
      }
#pragma unroll
      for (int k = 0; k < BV; ++k)
        g[k] = live[k] ? wide_lookup(D, a.tables, epoch, key[k], (unsigned)hash[k], x[k]) : -2;
    }
    // a block's first rows of an instance, before its hot groups have cells: a warp's
    // rows of a group in one add (592 blocks' 512 rows each queued up on the group of the
    // most frequent key: 2M x 20M rows of 150K groups, Zipf 1.5 and 2.0 keys, 407 and
    // 494 us, so 317 and 320)
    const bool together = first.value && own.look && !own.small;
#pragma unroll
    for (int k = 0; k < BV; ++k) {
      matched += g[k] >= -1;
      const bool add = g[k] >= 0 && !own.add((unsigned)g[k], value[k], first.value);
      if (!together && !add) continue;
      unsigned long long v = (unsigned long long)value[k];
      if (PACK) {
        v += bias;
        if (add) {
          outside |= v >> vbits != 0;
          high += v >> 20;
          ++rows;
        }
        v += one;
      }
      const unsigned n = together ? warp_group_sum(add ? (int)g[k] : -1, v) : 1u;
      if (!n) continue;
      if (PACK) {
        red_add(&packed[g[k]], v);
      } else {
        red_add(&slab[2 * (unsigned long long)g[k]], v);
        red_add(&slab[2 * (unsigned long long)g[k] + 1], (unsigned long long)n);
      }
    }
  };
  step(lo, std::true_type{});
  own.after_first();
  for (long long i0 = lo + BT2 * BV; i0 < hi; i0 += BT2 * BV) step(i0, std::false_type{});
  own.flush(slab);
}

// SECOND: the instances to be run again, two words a group, 16-byte slots.
template <bool SECOND>
__global__ void __launch_bounds__(BT2, PF_BATCH_MINB) k_batch(BatchArgs a) {
  Header* h = a.h;
  if (SECOND && h->n_redo == 0) return;
  __shared__ long long item_s;
  __shared__ int ok_s;
  __shared__ unsigned long long red[3][BT2 / 32];
  __shared__ unsigned outside_s;
  const unsigned epoch = h->epoch;
  const long long ni = h->n_items;
  unsigned long long bad_group = 0, overflow = 0;
  extern __shared__ __align__(16) unsigned char batch_smem[];
  OwnSums& S = *reinterpret_cast<OwnSums*>(batch_smem);
  own_init(S);
  // Items are taken in increasing order and an item waits only for items
  // before it, so the smallest unfinished item is always some block's
  // current item with nothing left to wait for: the launch progresses.
  unsigned long long* counter = SECOND ? &h->counter2 : &h->counter;
  while (true) {
    if (threadIdx.x == 0) item_s = (long long)atomicAdd(counter, 1ULL);
    __syncthreads();
    const long long it = item_s;
    __syncthreads();  // every thread has read item_s
    if (it >= ni) break;
    const int inst = a.imap[it];
    const unsigned flags = a.flags[inst];
    if (SECOND && !(flags & REDO)) continue;
    // the instance's descriptor in registers for the item (read through a
    // reference, every store to the tables or slabs would reload it)
    const Desc D = a.d[inst];
    const bool compact = !SECOND && D.q > 0 && !(flags & WIDE_TABLE);
    const long long local = it - D.item0;
    if (local < D.nbi) {
      const CompactTable t{reinterpret_cast<unsigned long long*>(a.tables + D.toff), D.q,
                           D.gbits, D.dbits};
      const long long lo = local * BITEM, hi = min(D.nb, lo + BITEM);
      for (long long i = lo + threadIdx.x; i < hi; i += BT2) {
        const long long key = __ldcs(D.bkey + i), g = (long long)__ldcs(D.bgrp + i) - D.gmin;
        const bool in = g >= 0 && g < D.ng;
        if (!SECOND) bad_group += !in;
        if (compact) {
          if (!ct_insert(t, key, in ? g : -1)) a.check[inst].crowded = 1;
        } else {
          overflow += !wide_insert(D, a.tables, epoch, (unsigned long long)key,
                                   in ? (uint32_t)g : 0xffffffffu);
        }
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        __threadfence();
        atomicSub(&a.remaining[inst], 1u);
      }
    } else {
      if (threadIdx.x == 0) {
        unsigned polls = 0;
        while (ld_acquire_u32(&a.remaining[inst]) != 0 && polls < WAIT_LIMIT) {
          __nanosleep(256);
          ++polls;
        }
        ok_s = polls < WAIT_LIMIT;
        if (!ok_s) atomicOr(&h->error, 1ULL);
        outside_s = 0;
        __threadfence();
      }
      __syncthreads();
      if (!ok_s) continue;
      Own own(S);
      own.begin(inst, D.ng);
      const long long lo = (local - D.nbi) * D.pitem, hi = min(D.np, lo + D.pitem);
      unsigned matched = 0, rows = 0;
      unsigned long long high = 0;
      bool outside = false;
      const bool pack = !SECOND && !(flags & WIDE_SUMS);
      if (compact && pack)
        probe_rows<true, true>(D, a, epoch, own, lo, hi, matched, rows, high, outside);
      else if (compact)
        probe_rows<true, false>(D, a, epoch, own, lo, hi, matched, rows, high, outside);
      else if (pack)
        probe_rows<false, true>(D, a, epoch, own, lo, hi, matched, rows, high, outside);
      else
        probe_rows<false, false>(D, a, epoch, own, lo, hi, matched, rows, high, outside);
      // the item's counts, one atomic each
      unsigned long long m = __reduce_add_sync(FULL, matched), r = __reduce_add_sync(FULL, rows);
      for (int o = 16; o; o >>= 1) high += __shfl_xor_sync(FULL, high, o);
      if (outside) outside_s = 1;
      if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = m;
        red[1][threadIdx.x >> 5] = r;
        red[2][threadIdx.x >> 5] = high;
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        for (int w = 1; w < BT2 / 32; ++w) {
          m += red[0][w];
          r += red[1][w];
          high += red[2][w];
        }
        Check* c = a.check + inst;
        if (m) atomicAdd(&c->matched, m);
        if (r) atomicAdd(&c->rows, r);
        if (high) atomicAdd(&c->high, high);
        if (outside_s) c->bad_value = 1;
      }
    }
  }
  if (bad_group) atomicAdd(&a.stats[2], bad_group);
  if (overflow) atomicAdd(&a.stats[3], overflow);
}

// The packed words added to the slabs; the last block decides which instances
// are run again and how, and readies them (their tables and sums are cleared
// by k_batch_again).
__global__ void __launch_bounds__(BT2) k_batch_sums(BatchArgs a, const int* __restrict__ cmap,
                                                    unsigned* flags) {
  Header* h = a.h;
  __shared__ unsigned long long red[BT2 / 32];
  __shared__ int last_s;
  for (long long c = blockIdx.x; c < h->n_chunks; c += gridDim.x) {
    const int inst = cmap[c];
    const Desc& D = a.d[inst];
    const long long g0 = (c - D.chunk0) * SUM_CHUNK, g1 = min(D.ng, g0 + SUM_CHUNK);
    const unsigned long long smask = (1ULL << D.sbits) - 1;
    const unsigned long long bias = 1ULL << (D.vbits - 1);
    ulonglong2* slab = reinterpret_cast<ulonglong2*>(a.slabs) + D.soff;
    unsigned long long total = 0;
    for (long long g = g0 + threadIdx.x; g < g1; g += BT2) {
      const unsigned long long x = a.packed[D.soff + g];
      if (!x) continue;
      const unsigned long long n = x >> D.sbits;
      ulonglong2 v = slab[g];
      v.x += (x & smask) - n * bias;
      v.y += n;
      slab[g] = v;
      total += n;
    }
    for (int o = 16; o; o >>= 1) total += __shfl_xor_sync(FULL, total, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = total;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < BT2 / 32; ++w) total += red[w];
      if (total) atomicAdd(&a.check[inst].counts, total);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last_s = atomicAdd(&h->chunks_done, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last_s) return;
  unsigned redo = 0;
  for (int i = threadIdx.x; i < h->n_inst; i += BT2) {
    Check* c = a.check + i;
    const unsigned f = flags[i] & ~REDO;
    unsigned add = 0;
    if (*(volatile unsigned*)&c->crowded) add |= WIDE_TABLE | REDO;
    const unsigned long long rows = *(volatile unsigned long long*)&c->rows;
    if (!(f & WIDE_SUMS) &&
        (*(volatile unsigned*)&c->bad_value ||
         *(volatile unsigned long long*)&c->counts != rows ||
         *(volatile unsigned long long*)&c->high + rows >= 1ULL << 43))
      add |= WIDE_SUMS | REDO;
    flags[i] = f | add;
    if (add & REDO) {
      ++redo;
      a.remaining[i] = (unsigned)a.d[i].nbi;
      c->matched = 0;
    }
  }
  if (redo) atomicAdd(&h->n_redo, redo);
}

// The tables and sums of the instances to be run again, cleared.
__global__ void __launch_bounds__(BT2) k_batch_again(BatchArgs a) {
  if (a.h->n_redo == 0) return;
  const unsigned long long tid = (unsigned long long)blockIdx.x * BT2 + threadIdx.x;
  const unsigned long long stride = (unsigned long long)gridDim.x * BT2;
  const ulonglong2 zero = make_ulonglong2(0ULL, 0ULL);
  for (int i = 0; i < a.h->n_inst; ++i) {
    if (!(a.flags[i] & REDO)) continue;
    const Desc& D = a.d[i];
    ulonglong2* t = reinterpret_cast<ulonglong2*>(a.tables + D.toff);
    for (unsigned long long k = tid; k < D.region; k += stride) t[k] = zero;
    ulonglong2* s = reinterpret_cast<ulonglong2*>(a.slabs) + D.soff;
    for (unsigned long long k = tid; k < (unsigned long long)D.ng; k += stride) s[k] = zero;
  }
}

// The run's end: the instances' matched rows added up, the error word.
__global__ void __launch_bounds__(BT2) k_batch_end(BatchArgs a) {
  __shared__ unsigned long long red[BT2 / 32];
  unsigned long long m = 0;
  for (int i = threadIdx.x; i < a.h->n_inst; i += BT2) m += a.check[i].matched;
  for (int o = 16; o; o >>= 1) m += __shfl_xor_sync(FULL, m, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int w = 1; w < BT2 / 32; ++w) m += red[w];
  a.stats[0] = m;
  if (a.h->error) a.stats[1] |= a.h->error;
}

// What pf_batch_run and pf_batch_slab need of a prepared workspace, kept on
// the host (keyed by the workspace's address) so that a run touches no host
// copy of device memory and can be captured.
struct HostPlan {
  int n = 0;
  Sizes sizes{};
  std::vector<unsigned long long> slab_off;
};

std::mutex g_plans_mu;
std::map<void*, HostPlan> g_plans;

bool find_plan(void* ws, HostPlan* out) {
  std::lock_guard<std::mutex> lock(g_plans_mu);
  auto it = g_plans.find(ws);
  if (it == g_plans.end()) return false;
  *out = it->second;
  return true;
}

// A persistent grid: every block resident at once.
template <bool SECOND>
int batch_grid(int* grid) {
  int per_sm = 0;
  if (int rc = opt_in_smem((const void*)k_batch<SECOND>, BATCH_SMEM)) return rc;
  PF_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch<SECOND>, BT2,
                                                        BATCH_SMEM));
  *grid = std::max(1, per_sm) * sm_count();
  return PF_OK;
}

}  // namespace
}  // namespace pf

using namespace pf;

extern "C" size_t pf_batch_workspace(const pf_batch_instance* in, int n) {
  size_t used = 0;
  layout(nullptr, n, totals(in, n), &used);
  return used + 256;
}

extern "C" int pf_batch_prepare(const pf_batch_instance* in, int n, void* workspace,
                                size_t workspace_bytes, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (n < 1) return fail(PF_EINVAL, "batch: at least one instance");
  const Sizes z = totals(in, n);
  const unsigned long long ts = z.table_slots, items = z.items;
  size_t used = 0;
  Layout l = layout((char*)workspace, n, z, &used);
  if (!workspace || used > workspace_bytes || ((uintptr_t)workspace & 255))
    return fail(PF_ENOSPACE,
                "batch: workspace of %zu bytes at %p, %zu needed on a 256-byte boundary",
                workspace_bytes, workspace, used);
  std::vector<Desc> d(n);
  // the regions of compact tables first: a run clears them in one piece
  unsigned long long toff = 0, wide_off = z.cleared_slots, soff = 0;
  long long bi = 0, pi = 0, chunks = 0;
  for (int i = 0; i < n; ++i) {
    const pf_batch_instance& x = in[i];
    if (x.n_build < 0 || x.n_probe < 0 || x.n_groups < 0 || x.n_groups > 0xfffffffeLL)
      return fail(PF_EINVAL, "batch: instance %d has bad sizes", i);
    if ((x.n_build > 0 && (!x.build_key || !x.build_group)) ||
        (x.n_probe > 0 && (!x.probe_fk || !x.probe_value)))
      return fail(PF_EINVAL, "batch: instance %d has a null column", i);
    Desc& D = d[i];
    D.bkey = (const long long*)x.build_key;
    D.bgrp = x.build_group;
    D.nb = x.n_build;
    D.pfk = (const long long*)x.probe_fk;
    D.pval = (const long long*)x.probe_value;
    // no build rows or no groups: nothing can match or be aggregated
    D.np = (x.n_build > 0) ? x.n_probe : 0;
    D.gmin = x.group_min;
    D.ng = x.n_groups;
    D.region = table_of(x.n_build, x.n_groups, &D.q, &D.gbits, &D.dbits, &D.tcap);
    unsigned long long& at = D.q ? toff : wide_off;
    D.toff = at;
    at += D.region;
    if (2ULL * (unsigned long long)x.n_build > 0xffffffffULL) return fail(PF_EINVAL, "batch: instance %d is over 2^31 build rows", i);
    // the packed word: the count's field for 16 times the mean rows a group (or
    // for all rows), a value's bits what a group of four times the mean leaves,
    // 40 at most (the offset counts in every sum)
    const int mean = bits_of((unsigned long long)(D.np / std::max<long long>(x.n_groups, 1)));
    const int cbits = std::min(bits_of((unsigned long long)D.np), mean + 4);
    D.sbits = std::min(64 - cbits, 62);
    D.vbits = std::max(8, std::min(D.sbits - mean - 2, 40));
    D.soff = soff;
    D.item0 = bi + pi;
    D.nbi = (D.nb + BITEM - 1) / BITEM;
    D.pitem = z.pitem;
    D.chunk0 = chunks;
    chunks += (x.n_groups + SUM_CHUNK - 1) / SUM_CHUNK;
    soff += (unsigned long long)x.n_groups;
    bi += (D.nb + BITEM - 1) / BITEM;
    pi += (D.np + z.pitem - 1) / z.pitem;
  }
  Header hh{};
  hh.epoch = 0;
  hh.counter = 0;
  hh.n_build_items = bi;
  hh.n_items = bi + pi;
  hh.n_chunks = chunks;
  hh.n_inst = n;
  if ((unsigned long long)(bi + pi) != items)
    return fail(PF_EINVAL, "batch: %lld work items, %llu planned", bi + pi, items);
  std::vector<int> imap((size_t)std::max<unsigned long long>(items, 1), 0);
  for (int i = 0; i < n; ++i) {
    const long long nit = d[i].nbi + (d[i].np + z.pitem - 1) / z.pitem;
    for (long long k = 0; k < nit; ++k) imap[(size_t)(d[i].item0 + k)] = i;
  }
  std::vector<int> cmap((size_t)std::max<unsigned long long>(z.chunks, 1), 0);
  for (int i = 0; i < n; ++i)
    for (long long k = 0; k < (d[i].ng + SUM_CHUNK - 1) / SUM_CHUNK; ++k)
      cmap[(size_t)(d[i].chunk0 + k)] = i;
  PF_CUDA(cudaMemcpyAsync(l.cmap, cmap.data(), sizeof(int) * cmap.size(), cudaMemcpyHostToDevice,
                          st));
  PF_CUDA(cudaMemsetAsync(l.flags, 0, sizeof(unsigned) * n, st));
  PF_CUDA(cudaMemcpyAsync(l.imap, imap.data(), sizeof(int) * imap.size(), cudaMemcpyHostToDevice,
                          st));
  PF_CUDA(cudaMemcpyAsync(l.desc, d.data(), sizeof(Desc) * n, cudaMemcpyHostToDevice, st));
  PF_CUDA(cudaMemcpyAsync(l.header, &hh, sizeof(Header), cudaMemcpyHostToDevice, st));
  // (each run clears the compact tables)
  PF_CUDA(cudaMemsetAsync(l.tables + z.cleared_slots, 0, sizeof(Slot) * (ts - z.cleared_slots),
                          st));
  if (int rc = wait_stream(st)) return rc;  // the host copies above read d, hh and the maps
  HostPlan hp;
  hp.n = n;
  hp.sizes = z;
  hp.slab_off.resize(n);
  for (int i = 0; i < n; ++i) hp.slab_off[i] = d[i].soff;
  {
    std::lock_guard<std::mutex> lock(g_plans_mu);
    g_plans[workspace] = std::move(hp);
  }
  return ok();
}

extern "C" int pf_batch_run(void* workspace, int64_t* stats, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  HostPlan hp;
  if (!find_plan(workspace, &hp)) return fail(PF_EINVAL, "batch: workspace was not prepared");
  if (!stats) return fail(PF_EINVAL, "batch: null stats");
  Layout l = layout((char*)workspace, hp.n, hp.sizes, nullptr);
  int grid = 0, grid2 = 0;
  if (int rc = batch_grid<false>(&grid)) return rc;
  if (int rc = batch_grid<true>(&grid2)) return rc;
  const BatchArgs a{l.header,   l.desc,   l.imap,  l.remaining, l.check,
                    l.flags,    l.tables, l.packed, l.slabs,    (unsigned long long*)stats};
  const int sms = sm_count();
  PF_CUDA(cudaMemsetAsync(stats, 0, 4 * sizeof(int64_t), st));
  {
    PF_KERNEL("k_batch_reset", st);
    const long long words = (long long)std::max(hp.sizes.slab_pairs, hp.sizes.cleared_slots);
    k_batch_reset<<<(unsigned)std::max<long long>(
                        1, std::min<long long>((words + BT2 - 1) / BT2, sms * 8LL)),
                    BT2, 0, st>>>(l.header, l.desc, l.remaining, l.check, hp.n, l.tables,
                                  hp.sizes.cleared_slots, l.packed, l.slabs,
                                  hp.sizes.slab_pairs);
  }
  PF_LAUNCH("k_batch_reset");
  {
    PF_KERNEL("k_batch", st);
    k_batch<false><<<grid, BT2, BATCH_SMEM, st>>>(a);
  }
  PF_LAUNCH("k_batch");
  {
    PF_KERNEL("k_batch_sums", st);
    k_batch_sums<<<(unsigned)std::max<long long>(
                       1, std::min<long long>((long long)hp.sizes.chunks, sms * 4LL)),
                   BT2, 0, st>>>(a, l.cmap, l.flags);
  }
  PF_LAUNCH("k_batch_sums");
  {
    PF_KERNEL("k_batch_again", st);
    k_batch_again<<<sms * 4, BT2, 0, st>>>(a);
  }
  PF_LAUNCH("k_batch_again");
  {
    PF_KERNEL("k_batch", st);
    k_batch<true><<<grid2, BT2, BATCH_SMEM, st>>>(a);
  }
  PF_LAUNCH("k_batch");
  {
    PF_KERNEL("k_batch_end", st);
    k_batch_end<<<1, BT2, 0, st>>>(a);
  }
  PF_LAUNCH("k_batch_end");
  return ok();
}

extern "C" int64_t* pf_batch_slab(void* workspace, int i) {
  HostPlan hp;
  if (!find_plan(workspace, &hp) || i < 0 || i >= hp.n) return nullptr;
  Layout l = layout((char*)workspace, hp.n, hp.sizes, nullptr);
  return (int64_t*)(l.slabs + 2 * hp.slab_off[i]);
}
