// The fused join -> group-by without a radix pass, for builds whose hash table
// fits L2: the build rows go into one table, each probe row is read once, its
// group looked up and its value added, and the groups are written out.
//
//   k_dj_init    the table emptied, the sums zeroed
//   k_dj_build   each build row into the table
//   k_dj_probe   each probe row hashed and looked up, its value and 1 added to
//                its group
//   k_dj_finish  the sums and counts, and the occupied groups ascending
//
// The radix path (join_aggregate.cu) moves a build row through two passes and
// a probe row through 24 + 16 + 16 + 16 + 16 bytes, over 20 launches and two
// waits; here a probe row is 24 bytes read, one 32-byte sector of the table
// and one RED.  What bounds it: L2's rate of requests (about 0.2 T/s reached
// for a random read and a RED a row; the figures are at dj_table).
//
// The table is compact.cuh's; a build whose hashes crowd it raises the overflow
// word and the caller takes the radix path.
//
// The sums.  Up to DJ_SMALL groups: a block adds into shared memory (as many
// copies of a group as fit, a lane its own, so a warp's lanes meet on no
// address), flushed once into one of DJ_REPS copies in global memory.  More
// groups: count and sum in one 64-bit word {count, sum}, one RED a row instead
// of two, s bits of sum.  That is exact or known not to be: group g's word gives
// the count C_g + floor(S_g / 2^s) modulo 2^(64 - s).  Values of [0, 2^v) alone go
// into words, v chosen so that all of them add up to less than 2^63: what the
// sums carry into the counts is then less than a wrapped count takes away, and the
// counts add up to the rows put into the words, counted by themselves, only if no
// field was left.  (A matched row whose build row has no group in the range is in
// none.)  Where they do not, the call runs again with two words a group.
// Other values go into a pair {sum, count} of the group, and so do the groups that a
// block meets often (skewed keys or groups), collected in shared memory, so that
// they neither queue up on one address nor fill a count's field.  Up to 64K groups
// have several copies of their words, so that four groups' words of a sector do not
// queue up (18M rows into 5000 groups: 488 -> 354 us).
#include <algorithm>
#include <climits>

#include "compact.cuh"

namespace pf {
namespace {

constexpr int DT = 256;
#ifndef PF_DJ_R
#define PF_DJ_R 2
#endif
#ifndef PF_DJ_MINB
#define PF_DJ_MINB 5
#endif
// probe rows a thread takes at a time, at five blocks a SM (48 registers):
// 20M rows against 3M, 203 us; at six blocks (40, spills) 265, 1 row 208-222,
// 3 rows 207, 4 rows 215-274
constexpr int DR = PF_DJ_R;
constexpr int FG = 4;                  // groups a thread of k_dj_finish takes
constexpr int FTILE = DT * FG;
constexpr int DJ_SMALL = 2048;         // groups summed in shared memory
constexpr int DJ_REPS = 8;             // global copies of their sums
constexpr int DJ_SPREAD = 1 << 17;     // words that a few groups' sums are spread over
constexpr int DJ_MAX_REPS = 32;
// A block's cache of its hot groups.  In the block's first DJ_LOOK steps (4096
// rows) a group that comes again before another one of its `seen` entry gets a
// cell, which one of a share of 0.1% or more soon does and one of 100K equal ones
// hardly ever; the cells stay in use where DJ_HITS threads found theirs by then (a
// share of 0.2% in all), else the other steps do without.  3M x 20M rows into 100K
// groups, the radix path's time after it: equal ones 350 us (600), one of 1% 358
// (614), one of 10% 385 (917), Zipf 1.0 594 (1379); with a cache taken into use by
// the first 512 rows alone and emptied into the packed words, whose counts it then
// overfilled, so that the call ran twice: 350, 1065, 798 and 1251.
constexpr int DJ_CACHE = 1024;
constexpr int DJ_LOOK = 8;
constexpr int DJ_HITS = 8;

struct DjHead {
  unsigned overflow;            // a build row found no entry
  unsigned pairs;               // packed sums: some are in the groups' pairs
  unsigned gave_up;             // k_dj_finish: a wait on another tile ran out
  unsigned ticket, done;        // its tiles taken and done
  unsigned pad;
  unsigned long long rows;      // rows put into packed words
  unsigned long long counts;    // the groups' counts added up
  long long groups;             // occupied groups
};

struct DjArgs {
  const long long* bkey;
  const int* bgrp;
  long long nb;
  const long long* fk;
  const long long* price;
  const long long* disc;
  long long scale, np;
  CompactTable table;
  long long gmin, G;
  unsigned long long* slab;     // the groups' pairs [preps][2 * G]
  unsigned long long* packed;   // and packed words [reps][G]
  int sbits, vbits;             // packed: bits of the sum, of a value
  int reps, preps;              // copies, a block's own by its number
  int copies;                   // small: copies of a group in shared memory, log2
  unsigned long long* stats;
  DjHead* head;
  unsigned long long* tiles;    // k_dj_finish: each tile's state
  int ntiles;
};

enum { SUM_SMALL, SUM_PACKED, SUM_WIDE };

__global__ void __launch_bounds__(DT) k_dj_init(DjArgs a, long long slab_words) {
  const long long t = (long long)blockIdx.x * DT + threadIdx.x, step = (long long)gridDim.x * DT;
  const long long words = 4LL << a.table.q;
  ulonglong2* tab = reinterpret_cast<ulonglong2*>(a.table.e);
  for (long long i = t; i < words / 2; i += step) tab[i] = make_ulonglong2(CT_EMPTY, CT_EMPTY);
  for (long long i = t; i < slab_words; i += step) a.slab[i] = 0;
  for (long long i = t; i < a.ntiles; i += step) a.tiles[i] = 0;
  if (t < 4) a.stats[t] = 0;
  if (t == 0) *a.head = DjHead{};
}

// (3M rows 55 us; 86 with the bucket read before the claim. Two or four rows a
// thread claiming together measured no faster.)
__global__ void __launch_bounds__(DT) k_dj_build(DjArgs a) {
  unsigned bad = 0;
  for (long long i = (long long)blockIdx.x * DT + threadIdx.x; i < a.nb;
       i += (long long)gridDim.x * DT) {
    const long long key = __ldcs(a.bkey + i), g = (long long)__ldcs(a.bgrp + i) - a.gmin;
    const bool in = g >= 0 && g < a.G;
    bad += !in;
    if (!ct_insert(a.table, key, in ? g : -1)) a.head->overflow = 1;
  }
  for (int o = 16; o; o >>= 1) bad += __shfl_xor_sync(FULL, bad, o);
  if ((threadIdx.x & 31) == 0 && bad) atomicAdd(&a.stats[2], (unsigned long long)bad);
}

__device__ __forceinline__ void add_shared(unsigned* lo, unsigned* hi, unsigned* cnt, unsigned s,
                                           long long v) {
  const unsigned l = (unsigned)(unsigned long long)v, h = (unsigned)((unsigned long long)v >> 32);
  const unsigned old = atomicAdd(&lo[s], l);
  const unsigned hc = h + (old + l < old ? 1u : 0u);
  if (hc) atomicAdd(&hi[s], hc);
  atomicAdd(&cnt[s], 1u);
}

template <int MODE, bool DISC>
__global__ void __launch_bounds__(DT, PF_DJ_MINB) k_dj_probe(DjArgs a) {
  extern __shared__ __align__(16) unsigned dj_smem[];
  if (a.head->overflow) return;
  const int tid = threadIdx.x, lane = tid & 31;
  const int cells = MODE == SUM_SMALL ? (int)a.G << a.copies : DJ_CACHE;
  unsigned* lo = dj_smem;
  unsigned* hi = lo + cells;
  unsigned* cnt = hi + cells;
  int* tag = reinterpret_cast<int*>(cnt + cells);  // the cache's groups
  unsigned short* seen = reinterpret_cast<unsigned short*>(tag + cells);
  for (int i = tid; i < cells; i += DT) {
    lo[i] = hi[i] = cnt[i] = 0;
    if (MODE != SUM_SMALL) {
      tag[i] = -1;
      seen[i] = 0;
    }
  }
  __syncthreads();
  const unsigned copy = lane & ((1u << a.copies) - 1);
  const unsigned long long G = (unsigned long long)a.G;
  unsigned long long* pairs = a.slab + 2 * G * (unsigned)(blockIdx.x % a.preps);
  unsigned long long* packed = a.packed + G * (unsigned)(blockIdx.x % a.reps);
  unsigned matched = 0, rows = 0;
  int hits = 0, steps = 0;
  bool paired = false, look = MODE != SUM_SMALL, cached = false;
  const long long tile = (long long)DT * DR;
  // a block's first step, before its hot groups have cells, would overfill a hot
  // group's count: its rows go into pairs where they are an eighth at most
  int vbits = a.np >= DJ_LOOK * (long long)gridDim.x * tile ? 0 : a.vbits;
  for (long long t0 = (long long)blockIdx.x * tile; t0 < a.np; t0 += (long long)gridDim.x * tile) {
    unsigned long long h[DR], want[DR];
    long long v[DR];
    CtBucket k[DR];
    bool live[DR];
#pragma unroll
    for (int r = 0; r < DR; ++r) {
      const long long i = t0 + r * DT + tid;
      live[r] = i < a.np;
      h[r] = live[r] ? (unsigned long long)__ldcs(a.fk + i) : 0ULL;
    }
#pragma unroll
    for (int r = 0; r < DR; ++r) {
      const long long i = t0 + r * DT + tid;
      v[r] = live[r] ? __ldcs(a.price + i) : 0;
    }
    if (DISC) {
      long long d[DR];
#pragma unroll
      for (int r = 0; r < DR; ++r) {
        const long long i = t0 + r * DT + tid;
        d[r] = live[r] ? __ldcs(a.disc + i) : 0;
      }
#pragma unroll
      for (int r = 0; r < DR; ++r)
        v[r] = (long long)((unsigned long long)v[r] * (unsigned long long)(a.scale - d[r]));
    }
#pragma unroll
    for (int r = 0; r < DR; ++r) {
      h[r] = ct_hash((long long)h[r]);
      want[r] = ct_want(a.table, h[r]);
      k[r] = ct_load(ct_home(a.table, h[r]));
    }
#pragma unroll
    for (int r = 0; r < DR; ++r) {
      if (!live[r]) continue;
      bool more;
      unsigned long long e = ct_among(a.table, k[r], want[r], &more);
      if (more) e = ct_walk(a.table, h[r], want[r]);
      if (e == CT_EMPTY) continue;
      const long long grp = ct_group(a.table, e);
      ++matched;
      if (grp < 0) continue;
      const unsigned g = (unsigned)grp;
      if (MODE == SUM_SMALL) {
        add_shared(lo, hi, cnt, g << a.copies | copy, v[r]);
        continue;
      }
      if (look || cached) {
        const unsigned mixed = g * 0x9E3779B1u, c = mixed >> 22;  // of DJ_CACHE = 1024
        const int t = *(volatile int*)&tag[c];
        if (t == (int)g) {
          add_shared(lo, hi, cnt, c, v[r]);
          ++hits;
          continue;
        }
        if (look) {
          volatile unsigned short* last = &seen[c];
          const unsigned short me = (unsigned short)(mixed >> 6);
          if (*last != me) *last = me;
          else if (t == -1) atomicCAS(&tag[c], -1, (int)g);
        }
      }
      if (MODE == SUM_PACKED && (unsigned long long)v[r] >> vbits == 0) {
        ++rows;
        red_add(&packed[g], (1ULL << a.sbits) + (unsigned long long)v[r]);
      } else {
        paired = true;
        red_add(&pairs[2 * (unsigned long long)g], (unsigned long long)v[r]);
        red_add(&pairs[2 * (unsigned long long)g + 1], 1ULL);
      }
    }
    vbits = a.vbits;
    if (MODE != SUM_SMALL && ++steps == DJ_LOOK) {
      look = false;
      cached = __syncthreads_count(hits > 0) >= DJ_HITS;
    }
  }
  __syncthreads();
  if (MODE == SUM_SMALL) {
    unsigned long long* rep = a.slab + 2ULL * (blockIdx.x % DJ_REPS) * (unsigned long long)a.G;
    for (int g = tid; g < (int)a.G; g += DT) {
      unsigned long long s = 0, c = 0;
      for (int j = 0; j < 1 << a.copies; ++j) {
        const int x = g << a.copies | ((j + tid) & ((1 << a.copies) - 1));
        s += (unsigned long long)hi[x] << 32 | lo[x];
        c += cnt[x];
      }
      if (c) {
        atomicAdd(&rep[2 * g], s);
        atomicAdd(&rep[2 * g + 1], c);
      }
    }
  } else {
    for (int i = tid; i < cells; i += DT) {
      const int g = tag[i];
      if (g < 0) continue;
      const unsigned long long s = (unsigned long long)hi[i] << 32 | lo[i], c = cnt[i];
      if (!c) continue;
      paired = true;
      red_add(&pairs[2 * (unsigned long long)g], s);
      red_add(&pairs[2 * (unsigned long long)g + 1], c);
    }
  }
  // the block's counts, one atomic each
  __shared__ unsigned long long red[2][DT / 32];
  unsigned long long m = matched, in = rows;
  for (int o = 16; o; o >>= 1) {
    m += __shfl_xor_sync(FULL, m, o);
    if (MODE == SUM_PACKED) in += __shfl_xor_sync(FULL, in, o);
  }
  if (lane == 0) {
    red[0][tid >> 5] = m;
    red[1][tid >> 5] = in;
  }
  if (MODE == SUM_PACKED && paired) a.head->pairs = 1;
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < DT / 32; ++w) {
      m += red[0][w];
      in += red[1][w];
    }
    if (m) atomicAdd(&a.stats[0], m);
    if (MODE == SUM_PACKED && in) atomicAdd(&a.head->rows, in);
  }
}

struct DjOut {
  long long* sum;     // [G] dense
  long long* count;
  long long* keys;    // occupied groups (null: not wanted)
  long long* sums;
  long long* counts;
  DjHead* host;
};

// Up to DJ_SMALL groups: one block adds up the copies and compacts.
__global__ void __launch_bounds__(1024) k_dj_finish_small(DjArgs a, DjOut o) {
  __shared__ int wsum[32];
  constexpr int PER = DJ_SMALL / 1024;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  unsigned long long s[PER], c[PER];
  int mine = 0;
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int g = tid * PER + k;
    s[k] = c[k] = 0;
    if (g >= a.G) continue;
    ulonglong2 x[DJ_REPS];
#pragma unroll
    for (int r = 0; r < DJ_REPS; ++r)
      x[r] = reinterpret_cast<const ulonglong2*>(a.slab)[(long long)r * a.G + g];
#pragma unroll
    for (int r = 0; r < DJ_REPS; ++r) {
      s[k] += x[r].x;
      c[k] += x[r].y;
    }
    o.sum[g] = (long long)s[k];
    o.count[g] = (long long)c[k];
    mine += c[k] > 0;
  }
  int incl = mine;
  for (int d = 1; d < 32; d <<= 1) {
    const int y = __shfl_up_sync(FULL, incl, d);
    if (lane >= d) incl += y;
  }
  if (lane == 31) wsum[w] = incl;
  __syncthreads();
  int at = incl - mine, tot = 0;
  for (int q = 0; q < 32; ++q) {
    at += q < w ? wsum[q] : 0;
    tot += wsum[q];
  }
  if (o.keys) {
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      if (!c[k]) continue;
      o.keys[at] = a.gmin + tid * PER + k;
      o.sums[at] = (long long)s[k];
      o.counts[at] = (long long)c[k];
      ++at;
    }
  }
  if (tid == 0) {
    DjHead h = *a.head;
    h.groups = tot;
    *o.host = h;
  }
}

// A tile's state: 0, or its occupied groups with TILE_OWN, or all groups' up
// to its end with TILE_ALL.
constexpr unsigned long long TILE_OWN = 1ULL << 62, TILE_ALL = 2ULL << 62,
                             TILE_VALUE = (1ULL << 62) - 1;
constexpr int DJ_POLLS = 1 << 22;

__device__ __forceinline__ unsigned long long ld_state(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_state(unsigned long long* p, unsigned long long v) {
  asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// One pass over the groups, a tile of FTILE a block, its sums and counts held
// in registers; a tile's first output is the sum of the tiles before it, looked
// up 32 at a time from the nearest back (tiles are taken in order, so the ones
// before are at work or done; a wait is bounded).  The last tile done tells the
// host.
template <bool PACKED>
__global__ void __launch_bounds__(DT) k_dj_finish(DjArgs a, DjOut o) {
  __shared__ int wsum[DT / 32];
  __shared__ unsigned long long csum[DT / 32];
  __shared__ int tile_s;
  __shared__ long long before_s;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  if (tid == 0) tile_s = (int)atomicAdd(&a.head->ticket, 1u);
  __syncthreads();
  const int t = tile_s;
  if (t >= a.ntiles) return;
  const long long g0 = (long long)t * FTILE + (long long)tid * FG;
  const unsigned long long smask = PACKED ? (1ULL << a.sbits) - 1 : 0;
  unsigned long long s[FG], c[FG], total = 0;
  int mine = 0;
#pragma unroll
  for (int k = 0; k < FG; ++k) s[k] = c[k] = 0;
  if (PACKED) {
    for (int r = 0; r < a.reps; ++r) {
#pragma unroll
      for (int k = 0; k < FG; ++k)
        if (g0 + k < a.G) s[k] += a.packed[(long long)r * a.G + g0 + k];
    }
#pragma unroll
    for (int k = 0; k < FG; ++k) {
      c[k] = s[k] >> a.sbits;
      s[k] &= smask;
      total += c[k];
    }
  }
  if (!PACKED || a.head->pairs) {
    for (int r = 0; r < a.preps; ++r) {
#pragma unroll
      for (int k = 0; k < FG; ++k) {
        if (g0 + k >= a.G) continue;
        const ulonglong2 x =
            reinterpret_cast<const ulonglong2*>(a.slab)[(long long)r * a.G + g0 + k];
        s[k] += x.x;
        c[k] += x.y;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < FG; ++k) {
    if (g0 + k >= a.G) continue;
    mine += c[k] > 0;
    o.sum[g0 + k] = (long long)s[k];
    o.count[g0 + k] = (long long)c[k];
  }
  int incl = mine;
  for (int d = 1; d < 32; d <<= 1) {
    const int y = __shfl_up_sync(FULL, incl, d);
    if (lane >= d) incl += y;
  }
  if (PACKED)
    for (int d = 16; d; d >>= 1) total += __shfl_xor_sync(FULL, total, d);
  if (lane == 31) wsum[w] = incl;
  if (lane == 0) csum[w] = total;
  __syncthreads();
  int at = incl - mine, tot = 0;
#pragma unroll
  for (int q = 0; q < DT / 32; ++q) {
    at += q < w ? wsum[q] : 0;
    tot += wsum[q];
  }
  if (w == 0) {
    long long before = 0;
    if (lane == 0 && t > 0) st_state(&a.tiles[t], TILE_OWN | (unsigned long long)tot);
    bool ok = true;
    for (int end = t; end > 0 && ok;) {
      const int q = end - 1 - lane;  // lane 0 the nearest
      unsigned long long x = q >= 0 ? 0 : TILE_ALL;
      for (int polls = 0; q >= 0 && polls < DJ_POLLS; ++polls) {
        x = ld_state(&a.tiles[q]);
        if (x) break;
      }
      ok = __all_sync(FULL, x != 0);
      const unsigned all = __ballot_sync(FULL, (x & TILE_ALL) != 0);
      const int stop = all ? __ffs(all) - 1 : 31;
      long long add = lane <= stop ? (long long)(x & TILE_VALUE) : 0;
      for (int d = 16; d; d >>= 1) add += __shfl_xor_sync(FULL, add, d);
      before += add;
      if (all) break;
      end -= 32;
    }
    if (lane == 0) {
      if (!ok) a.head->gave_up = 1;
      st_state(&a.tiles[t], TILE_ALL | (unsigned long long)(before + tot));
      before_s = before;
      if (PACKED) {
        for (int q = 1; q < DT / 32; ++q) total += csum[q];
        if (total) atomicAdd(&a.head->counts, total);
      }
    }
  }
  __syncthreads();
  long long j = before_s + at;
  if (o.keys) {
#pragma unroll
    for (int k = 0; k < FG; ++k) {
      if (!c[k]) continue;
      o.keys[j] = a.gmin + g0 + k;
      o.sums[j] = (long long)s[k];
      o.counts[j] = (long long)c[k];
      ++j;
    }
  }
  if (tid != 0) return;
  if (t == a.ntiles - 1) a.head->groups = before_s + tot;
  __threadfence();
  if (atomicAdd(&a.head->done, 1u) == (unsigned)a.ntiles - 1) {
    __threadfence();
    volatile DjHead* h = a.head;
    o.host->overflow = h->overflow;
    o.host->gave_up = h->gave_up;
    o.host->rows = h->rows;
    o.host->counts = h->counts;
    o.host->groups = h->groups;
  }
}

struct DjLayout {
  DjHead* head;
  unsigned long long* table;
  unsigned long long* slab;
  unsigned long long* tiles;
  int q, gbits, dbits, ntiles, reps, preps;
};

// The table's bits for nb build rows and groups of g bits, or q = 0.
//
// At most 0.3 full, or 0.4 from 64 MiB on, where the next size up leaves L2
// (3M x 18M rows: 306 us in 64 MiB, 351 in 128).
// How large: up to 128 MiB, a little over L2. Against the radix path, 8 M x 40M
// and more rows lose (9M x 45M in 256 MiB 1.33 against 1.14 ms); 5.9M x 47M
// rows take 1.02 against 1.08, 4.5M x 13.5M 0.42 against 0.50, 1M x 5M 0.15
// against 0.29, 250K x 1M 0.07 against 0.17 to 0.35.
constexpr int DJ_MAX_Q = 22;
constexpr double DJ_LOAD = 0.3, DJ_LOAD_TOP = 0.4;
void dj_table(long long nb, long long G, int* q, int* gbits, int* dbits) {
  ct_size(nb, G, DJ_MAX_Q, DJ_LOAD, DJ_LOAD_TOP, q, gbits, dbits);
}

DjLayout dj_layout(Arena& a, long long nb, long long G) {
  DjLayout l{};
  dj_table(nb, G, &l.q, &l.gbits, &l.dbits);
  l.head = a.take<DjHead>(1);
  l.table = a.take<unsigned long long>(l.q ? (size_t)4 << l.q : 1);
  l.reps = G <= DJ_SMALL ? DJ_REPS
                         : (int)std::max<long long>(1, std::min<long long>(DJ_MAX_REPS, DJ_SPREAD / G));
  // the packed form's copies of the words, and half as many of the pairs
  l.preps = std::max(1, l.reps / 2);
  const long long words = std::max(2LL * l.reps, 2LL * l.preps + l.reps) * G;
  l.slab = a.take<unsigned long long>((size_t)std::max<long long>(words, 1));
  l.ntiles = G <= DJ_SMALL ? 0 : (int)((G + FTILE - 1) / FTILE);
  l.tiles = a.take<unsigned long long>((size_t)l.ntiles + 1);
  return l;
}

DjHead* pinned_dj_head() {
  thread_local DjHead* buf = nullptr;
  if (!buf && cudaHostAlloc((void**)&buf, sizeof(DjHead),
                            cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
    cudaGetLastError();
    buf = nullptr;
  }
  return buf;
}

template <int MODE>
int dj_probe(const DjArgs& a, cudaStream_t st) {
  const size_t smem = MODE == SUM_SMALL ? (size_t)3 * 4 * (a.G << a.copies) : 18 * DJ_CACHE;
  auto kern = a.disc ? k_dj_probe<MODE, true> : k_dj_probe<MODE, false>;
  if (int rc = opt_in_smem((const void*)kern, smem)) return rc;
  int per_sm = 0;
  PF_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, DT, smem));
  const unsigned g = (unsigned)std::max<long long>(
      1, std::min<long long>((a.np + DT * DR - 1) / (DT * DR),
                             (long long)sm_count() * std::max(1, per_sm)));
  {
    PF_KERNEL("k_dj_probe", st);
    kern<<<g, DT, smem, st>>>(a);
  }
  PF_LAUNCH("k_dj_probe");
  return PF_OK;
}

}  // namespace
}  // namespace pf

using namespace pf;

extern "C" int pf_join_direct_fits(int64_t n_build, int64_t n_probe, int64_t n_groups) {
  if (n_build < 1 || n_probe < 1 || n_groups < 1 || n_groups > (1 << 28)) return 0;
  int q, gbits, dbits;
  dj_table(n_build, n_groups, &q, &gbits, &dbits);
  return q > 0;
}

extern "C" size_t pf_join_direct_workspace(int64_t n_build, int64_t n_groups) {
  Arena a(nullptr, 0);
  dj_layout(a, n_build, n_groups);
  return a.used + 256;
}

extern "C" int pf_join_direct(const int64_t* build_key, const int32_t* build_group,
                              int64_t n_build, const int64_t* probe_fk,
                              const int64_t* probe_price, const int64_t* probe_disc,
                              int64_t scale, int64_t n_probe, int64_t group_min,
                              int64_t n_groups, int64_t* sum_out, int64_t* count_out,
                              int64_t* stats_out, int64_t* keys_out, int64_t* sums_out,
                              int64_t* counts_out, int64_t* n_out, int* done, void* workspace,
                              size_t workspace_bytes, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (!pf_join_direct_fits(n_build, n_probe, n_groups))
    return fail(PF_EINVAL, "join_direct: %lld build rows and %lld groups do not fit its table",
                (long long)n_build, (long long)n_groups);
  if (n_probe >= (1LL << 40)) return fail(PF_EINVAL, "join_direct: at most 2^40 probe rows");
  if (!build_key || !build_group || !probe_fk || !probe_price || !sum_out || !count_out ||
      !stats_out || !done || (keys_out && (!sums_out || !counts_out || !n_out)))
    return fail(PF_EINVAL, "join_direct: null pointer");
  Arena ar(workspace, workspace_bytes);
  const DjLayout l = dj_layout(ar, n_build, n_groups);
  if (!workspace || !ar.fits())
    return fail(PF_ENOSPACE, "join_direct: workspace of %zu bytes, %zu needed", workspace_bytes,
                ar.used);
  DjHead* host = pinned_dj_head();
  DjHead* host_dev = nullptr;
  if (!host) return fail(PF_ECUDA, "join_direct: no pinned result words");
  if (int rc = host_alias(host, (void**)&host_dev)) return rc;
  DjArgs a{};
  a.bkey = (const long long*)build_key;
  a.bgrp = build_group;
  a.nb = n_build;
  a.fk = (const long long*)probe_fk;
  a.price = (const long long*)probe_price;
  a.disc = (const long long*)probe_disc;
  a.scale = scale;
  a.np = n_probe;
  a.table = CompactTable{l.table, l.q, l.gbits, l.dbits};
  a.gmin = group_min;
  a.G = n_groups;
  a.slab = l.slab;
  a.stats = (unsigned long long*)stats_out;
  a.head = l.head;
  a.tiles = l.tiles;
  a.ntiles = l.ntiles;
  const bool small = n_groups <= DJ_SMALL;
  // packed: the count's field for a 256th of the rows (a larger group is hot), for
  // 2^17 and for 16 times the mean of a group (or for all rows), where that leaves a
  // mean group's sum 31 bits a value: else the check would fail on ordinary values,
  // and the call run twice
  const int all = bits_of((unsigned long long)n_probe);
  const int mean = bits_of((unsigned long long)(n_probe / n_groups));
  a.sbits = 64 - std::min(all, std::max(mean + 4, std::min(std::max(17, all - 8), 33 - mean)));
  const bool pack = a.sbits - mean >= 31;
  a.vbits = std::min(a.sbits - mean - 2, 63 - all);
  while (a.copies < 5 && (n_groups << (a.copies + 1)) <= DJ_SMALL) ++a.copies;
  DjOut o{(long long*)sum_out, (long long*)count_out, (long long*)keys_out, (long long*)sums_out,
          (long long*)counts_out, host_dev};
  const int sms = sm_count();
  *done = 0;
  for (int attempt = small || pack ? 0 : 1; attempt < 2; ++attempt) {
    const bool packed = !small && attempt == 0;
    a.reps = packed ? l.reps : 1;
    a.preps = packed ? l.preps : l.reps;
    a.packed = l.slab + 2LL * a.preps * n_groups;
    const long long words = (2LL * a.preps + (packed ? l.reps : 0)) * n_groups;
    {
      const long long work = (4LL << a.table.q) / 2 + words;
      PF_KERNEL("k_dj_init", st);
      k_dj_init<<<(unsigned)std::max<long long>(
                      1, std::min<long long>((work + DT * 4 - 1) / (DT * 4), sms * 8LL)),
                  DT, 0, st>>>(a, words);
    }
    PF_LAUNCH("k_dj_init");
    {
      PF_KERNEL("k_dj_build", st);
      k_dj_build<<<(unsigned)std::min<long long>((n_build + DT - 1) / DT, sms * 8LL),
                   DT, 0, st>>>(a);
    }
    PF_LAUNCH("k_dj_build");
    if (int rc = small    ? dj_probe<SUM_SMALL>(a, st)
                 : packed ? dj_probe<SUM_PACKED>(a, st)
                          : dj_probe<SUM_WIDE>(a, st))
      return rc;
    {
      PF_KERNEL("k_dj_finish", st);
      if (small) k_dj_finish_small<<<1, 1024, 0, st>>>(a, o);
      else if (packed) k_dj_finish<true><<<a.ntiles, DT, 0, st>>>(a, o);
      else k_dj_finish<false><<<a.ntiles, DT, 0, st>>>(a, o);
    }
    PF_LAUNCH("k_dj_finish");
    if (int rc = wait_stream(st)) return rc;
    if (host->gave_up) return fail(PF_EDEVICE, "join_direct: a device wait gave up");
    if (host->overflow) return ok();  // *done = 0
    if (!packed || host->counts == host->rows) {
      *done = 1;
      if (n_out) *n_out = host->groups;
      return ok();
    }
  }
  return ok();
}
