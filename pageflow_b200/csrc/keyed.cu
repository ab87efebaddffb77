// Pass 1 of a keyed aggregation in one read of its rows (PageFlow's
// KeyedAggregate.pass1, operators/aggregate.py:1511-1563): the grouping hash of
// each row's key columns, a row per distinct hash in an open-addressing table
// whose slots hold every accumulator of the group, and the groups written out
// ascending by hash.
//
//   k_kp_init     the keys emptied, the accumulators at their start
//   k_kp_insert   each row hashed, its group found or claimed, its values
//                 folded in; a block first folds into a table of its own in
//                 shared memory while that pays (few or hot groups: thousands
//                 of rows on one address would queue up in L2), flushed at the
//                 end.  A group's place is looked for four keys (one 32-byte
//                 sector) at a time.  Sums and counts are one RED each; a max,
//                 a min or a key word is compared with the group's first and
//                 only a better one costs an atomic
//   k_kp_collect  groups per bucket of the hash's range, k_kp_scan their
//                 offsets and number
//   k_kp_place    the groups' (hash, place) by bucket
//   k_kp_emit     a warp a bucket: the bucket's groups ranked in shared
//                 memory and written out, the results' types made on the way
//   k_kp_buckets  the groups' partition buckets
// The first four are queued by pf_keyed_pass1_read, the rest by
// pf_keyed_pass1_emit, which waits once, so that a caller makes its outputs
// while the rows are read.
//
// What bounds it: random L2 sectors, a group's keys and its compared
// accumulators, and a RED a sum or count.  The general route it replaces
// where the groups fit (pf_group_hash, five or six radix passes of (hash, row)
// pairs, then a gather and a segmented reduction a value column, some of the
// columns made for it by elementwise kernels) moved about 700 bytes a row.
//
// The first table is at most KP_TABLE_BYTES, half of L2; with more groups the
// launch stops early (first_step, or a probe that finds KP_WALK full sectors),
// what it met tells how many there are, and the caller reads the rows again
// into a table for them, or takes the general route where most rows are a
// group of their own.  4M rows, two key columns, five aggregates, the pass
// through KeyedPass1 against the general route: 4 groups 0.30 against 1.38 ms,
// 1000 0.37 against 0.94, 100K 0.34 against 1.05, 900K (a second table) 0.63
// against 1.10; 4M, by the general route after a failed attempt, 1.43 against
// 1.23.  k_kp_insert takes 0.18 ms of it at 250K groups.
#include <algorithm>
#include <climits>
#include <cmath>

#include "common.cuh"

namespace pf {
namespace {

constexpr int KT = 256;
#ifndef PF_KP_R
#define PF_KP_R 2
#endif
#ifndef PF_KP_MINB
#define PF_KP_MINB 4
#endif
// rows a thread takes at a time, at four blocks a SM: 4M rows into 250K groups
// take 184 us at 2 rows, 300 at 4 (spills), 197 at 1 with six blocks
constexpr int KR = PF_KP_R;
constexpr int KP_MAX_KEYS = 8;
constexpr int KP_MAX_ACC = 15;
constexpr int KP_MAX_OUT = 40;
constexpr long long KP_EMPTY = LLONG_MIN;  // a group of this hash has the slot after the last
// Sectors of keys a probe looks at: in a table two thirds full, the fullest one made, a
// place that far from home is as good as never needed (16 sectors, three quarters
// full, gave up tables that fitted: 20,000 rows of as many groups took 670 us, by
// the general route after all, now 159; 300,000 in one run of two 690, now 211).
constexpr int KP_WALK = 64;
constexpr size_t KP_TABLE_BYTES = (size_t)64 << 20;
constexpr size_t KP_CACHE_BYTES = 36 << 10;
constexpr int KP_CACHE_WALK = 12;
constexpr int KP_REPEATS = 8;      // of a block's first 256 rows, groups met twice
constexpr int KP_BUCKET = 512;     // groups of a bucket the warp ranks, at most
constexpr int KP_MAX_B = 4096;     // partition buckets, at most

struct KeyCols {
  const unsigned char* col[KP_MAX_KEYS];
  const long long* coeff[KP_MAX_KEYS];
  int rb[KP_MAX_KEYS];
  int words[KP_MAX_KEYS];
  int path[KP_MAX_KEYS];  // 0: whole aligned words, 1: one aligned 4-byte row, 2: bytes
  int n;
};

// How a row's value for an accumulator is read.
enum { H_I64, H_I32, H_F64, H_F32, H_WORD8, H_WORD4, H_WORD, H_ONE };

// The accumulators as the table holds them: first the `ncmp` that keep the
// largest value (key words, maxima, and minima of the values' complements),
// then, to `nplain`, the sums and counts, then the `nerr` float64 sums whose adds'
// errors are kept, and the errors in their order.
struct Accs {
  int ncmp, nplain, nerr, n;
  const unsigned char* src[KP_MAX_ACC];
  int how[KP_MAX_ACC];
  int rb[KP_MAX_ACC];          // key words: the rows' bytes, the word
  int word[KP_MAX_ACC];
  long long flip[KP_MAX_ACC];  // -1: the value's complement
  int nulls[KP_MAX_ACC];       // 1, 2: 1 for the null as an integer, a float
  int is_float[KP_MAX_ACC];
};

struct KpHead {
  long long lo, hi;      // the hashes' range
  long long groups;
  long long max_bucket;
  long long placed, claimed;  // rows folded in; of them, groups' first
  long long seen;        // the same of the first step alone, 32 bits each
  int full;              // a probe gave up: too many groups for the table
};

struct KpArgs {
  KeyCols key;
  Accs acc;
  long long n;
  long long* keys;             // [cap + 4]: cap for KP_EMPTY's own group
  long long* accs;             // [cap + 1][W]
  unsigned long long cap;      // a power of two
  int W;                       // accumulator words a group, whole sectors
  int cache;                   // slots of a block's own table (a power of two)
  KpHead* head;
};

// Word w of a row of rb bytes, zero-padded (_pack_as_int64).
__device__ __forceinline__ unsigned long long row_word(const unsigned char* col, long long i,
                                                       int rb, int w, int path) {
  const unsigned char* row = col + i * rb;
  if (path == 0) return __ldcs(reinterpret_cast<const unsigned long long*>(row) + w);
  if (path == 1) return (unsigned long long)__ldcs(reinterpret_cast<const unsigned*>(row));
  unsigned long long v = 0;
  const int b0 = 8 * w, b1 = min(rb, b0 + 8);
  for (int b = b0; b < b1; ++b) v |= (unsigned long long)row[b] << (8 * (b - b0));
  return v;
}

// The start of accumulator k: the least value, 0 or 0.0.
__device__ __forceinline__ long long acc_start(const Accs& c, int k) {
  return k < c.ncmp ? LLONG_MIN : 0;
}

__global__ void __launch_bounds__(KT) k_kp_init(KpArgs a, int* __restrict__ hist, int nbuckets) {
  const long long words = (long long)(a.cap + 1) * a.W;
  const long long t = (long long)blockIdx.x * KT + threadIdx.x, step = (long long)gridDim.x * KT;
  // a thread writes the words of one accumulator: step is a multiple of W
  const long long x = acc_start(a.acc, (int)(t % a.W));
  for (long long i = t; i < words; i += step) a.accs[i] = x;
  for (long long i = t; i < (long long)a.cap + 4; i += step) a.keys[i] = KP_EMPTY;
  for (long long b = t; b < nbuckets; b += step) hist[b] = 0;
  if (t == 0) *a.head = KpHead{LLONG_MAX, LLONG_MIN, 0, 0, 0, 0, 0, 0};
}

// 32 bytes in one load (keys and accumulators lie on 32-byte sectors).  Stale
// words do no harm: a free mark is settled by the claim, and a smaller
// largest value costs an atomic that changes nothing.
struct Sector {
  long long w[4];
};
__device__ __forceinline__ Sector ld_sector(const long long* p) {
  Sector s;
  asm volatile("ld.global.L1::no_allocate.v4.b64 {%0, %1, %2, %3}, [%4];"
               : "=l"(s.w[0]), "=l"(s.w[1]), "=l"(s.w[2]), "=l"(s.w[3])
               : "l"(p)
               : "memory");
  return s;
}

// The first of the four keys that hash h is looked for at.
__device__ __forceinline__ unsigned long long kp_home(long long h, unsigned long long cap) {
  return mix64((uint64_t)h) & (cap - 4);
}

// Hash h among four keys (s: as loaded from place `at`): its place, claimed
// when a key is free, or -1 when all four are other hashes'.  Keys fill a
// sector in order and never leave, so two rows of a new hash meet at the
// same claim.
__device__ __forceinline__ int kp_among(const KpArgs& a, long long h, unsigned long long at,
                                        const Sector& s, unsigned& claims) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    long long x = s.w[j];
    if (x == KP_EMPTY) {
      x = (long long)atomicCAS((unsigned long long*)&a.keys[at + j], (unsigned long long)KP_EMPTY,
                               (unsigned long long)h);
      if (x == KP_EMPTY) {
        ++claims;
        return (int)at + j;
      }
    }
    if (x == h) return (int)at + j;
  }
  return -1;
}

// The place of hash h, or -1.
__device__ __forceinline__ int kp_place_of(const KpArgs& a, long long h, unsigned& claims) {
  if (h == KP_EMPTY) {
    a.keys[a.cap] = 0;  // in use
    return (int)a.cap;
  }
  unsigned long long at = kp_home(h, a.cap);
  for (int k = 0; k < KP_WALK; ++k) {
    const int g = kp_among(a, h, at, ld_sector(a.keys + at), claims);
    if (g >= 0) return g;
    at = (at + 4) & (a.cap - 1);
  }
  return -1;
}

// What s = x + v, rounded, leaves out (Knuth's two-sum; NaN where s is no number).
__device__ __forceinline__ double sum_error(double x, double v) {
  const double s = __dadd_rn(x, v), w = __dsub_rn(s, x);
  return __dadd_rn(__dsub_rn(x, __dsub_rn(s, w)), __dsub_rn(v, w));
}

// A value added to a sum or count of the global table.
__device__ __forceinline__ void add_to(long long* p, int is_float, long long v) {
  if (is_float) red_add(reinterpret_cast<double*>(p), __longlong_as_double(v));
  else if (v) red_add(reinterpret_cast<unsigned long long*>(p), (unsigned long long)v);
}

// A float64 value, and its own error e, added to a sum whose errors are at p[nerr].
// Rows come in any order and one by one, where the general route adds a warp's
// rows of a group as a tree first: what each add rounds away, which its answer
// shows, is collected beside the sum and given back at the end.  4M rows of prices
// in 250K, 1000 and 4 groups, the mean error of a sum: without 7.8e-11, 1.2e-7 and
// 2.6e-5, by the general route 4.6e-11, 5.1e-8 and 2.5e-4, with 3.1e-11, 7.6e-9 and
// 2.8e-6 (the sum's own rounding); the pass 330, 312 and 319 us without, 362, 361
// and 272 with (the general route 1097, 1002 and 1662).
__device__ __forceinline__ void add_with_error(long long* p, int nerr, double x, double e) {
  e += sum_error(fetch_add(reinterpret_cast<double*>(p), x), x);
  if (e != 0) red_add(reinterpret_cast<double*>(p + nerr), e);
}

// The same in a block's own table.  A 64-bit add on shared memory is a
// compare-and-swap loop, so integer sums add their halves with the carry that
// the low half's old value shows.
__device__ __forceinline__ void add_to_shared(long long* p, int is_float, long long v) {
  if (is_float) {
    atomicAdd(reinterpret_cast<double*>(p), __longlong_as_double(v));
    return;
  }
  if (!v) return;
  unsigned* u = reinterpret_cast<unsigned*>(p);
  const unsigned l = (unsigned)(unsigned long long)v;
  const unsigned old = l ? atomicAdd(u, l) : 0u;
  const unsigned hi = (unsigned)((unsigned long long)v >> 32) + (l && old + l < old ? 1u : 0u);
  if (hi) atomicAdd(u + 1, hi);
}

// A float64 sum's rows with their errors (every lane of the warp; at < 0: none): the
// lanes of a group add theirs up as a tree, so that a group of many lanes does
// not queue up on the loop of its add (the pass over 4M rows of 4 groups: 272 us; a
// lane each 423).
__device__ __forceinline__ void add_group_to_shared(long long* own, int na, int k, int nerr,
                                                    int at, double x) {
  const int lane = threadIdx.x & 31;
  unsigned peers = __match_any_sync(FULL, at < 0 ? -1 - lane : at);
  const bool first = (peers & lanemask_lt()) == 0;
  unsigned rank = __popc(peers & lanemask_lt());
  double e = 0;
  peers &= ~1u << lane;  // those above
  while (__any_sync(FULL, peers)) {
    const int next = peers ? __ffs(peers) - 1 : lane;
    const double y = __shfl_sync(FULL, x, next), f = __shfl_sync(FULL, e, next);
    if (peers) {
      e += f + sum_error(x, y);
      x = __dadd_rn(x, y);
    }
    // every other one has been taken
    peers &= __ballot_sync(FULL, (rank & 1) == 0);
    rank >>= 1;
  }
  if (at < 0 || !first) return;
  double* sum = reinterpret_cast<double*>(own + at * na + k);
  e += sum_error(atomicAdd(sum, x), x);
  if (e != 0) atomicAdd(sum + nerr, e);
}

// KR rows' values for accumulator k (rows i0, i0 + KT, ..; at < 0: none), as
// the bits its fold takes.
__device__ __forceinline__ void acc_values(const Accs& c, int k, long long i0,
                                           const int (&at)[KR], long long (&v)[KR]) {
  const unsigned char* src = c.src[k];
#pragma unroll
  for (int r = 0; r < KR; ++r) v[r] = 1;
#define KP_LOAD(expr)                 \
  _Pragma("unroll") for (int r = 0; r < KR; ++r) { \
    const long long i = i0 + r * KT;  \
    if (at[r] >= 0) v[r] = (expr);    \
  }                                   \
  break
  switch (c.how[k]) {
    case H_I64:
    case H_F64: KP_LOAD(__ldcs(reinterpret_cast<const long long*>(src) + i));
    case H_I32: KP_LOAD((long long)__ldcs(reinterpret_cast<const int*>(src) + i));
    case H_F32:
      KP_LOAD(__double_as_longlong((double)__ldcs(reinterpret_cast<const float*>(src) + i)));
    case H_WORD8: KP_LOAD((long long)row_word(src, i, c.rb[k], c.word[k], 0));
    case H_WORD4: KP_LOAD((long long)row_word(src, i, 4, 0, 1));
    case H_WORD: KP_LOAD((long long)row_word(src, i, c.rb[k], c.word[k], 2));
    default: break;
  }
#undef KP_LOAD
  if (const int nulls = c.nulls[k]) {
#pragma unroll
    for (int r = 0; r < KR; ++r)
      v[r] = nulls == 1 ? v[r] == -64 : __longlong_as_double(v[r]) == -64.0;
  }
  const long long flip = c.flip[k];
#pragma unroll
  for (int r = 0; r < KR; ++r) v[r] ^= flip;
}

// KR rows' grouping hashes, a thread's every KT-th from i0 on.
__device__ __forceinline__ void kp_hashes(const KpArgs& a, long long i0, const bool (&live)[KR],
                                          long long (&h)[KR]) {
#pragma unroll
  for (int r = 0; r < KR; ++r) h[r] = 0;
  for (int c = 0; c < a.key.n; ++c) {
    for (int w = 0; w < a.key.words[c]; ++w) {
      const unsigned long long co = (unsigned long long)a.key.coeff[c][w];
      unsigned long long x[KR];
#pragma unroll
      for (int r = 0; r < KR; ++r)
        x[r] = live[r] ? row_word(a.key.col[c], i0 + r * KT, a.key.rb[c], w, a.key.path[c]) : 0ULL;
#pragma unroll
      for (int r = 0; r < KR; ++r) h[r] = (long long)((unsigned long long)h[r] + x[r] * co);
    }
  }
}

// Hash h's place in the block's own table, or -1; *met: it was there before.
__device__ __forceinline__ int own_place(long long* own_key, int slots, long long h, bool* met) {
  unsigned s = (unsigned)(mix64((uint64_t)h) >> 40) & (unsigned)(slots - 1);
  for (int k = 0; k < KP_CACHE_WALK; ++k) {
    long long x = *(volatile long long*)&own_key[s];
    *met = x == h;
    if (x == KP_EMPTY)
      x = (long long)atomicCAS((unsigned long long*)&own_key[s], (unsigned long long)KP_EMPTY,
                               (unsigned long long)h);
    if (x == KP_EMPTY || x == h) return (int)s;
    s = (s + 1) & (unsigned)(slots - 1);
  }
  *met = false;
  return -1;
}

// After a block's first step its last warp adds the block's rows and claims
// to the launch's and looks whether the groups will fit: rows drawn alike from
// U groups claim (1 - exp(-z)) / z of the first P, z = P / U.  Past the share
// that a U of two thirds of the table would give, the launch stops, and what
// it met tells the caller how many groups to expect (4M rows of 2M groups: the
// attempt took 0.6 ms until the table was full).
struct FirstStep {
  unsigned placed, claims, warps;
};
__device__ __forceinline__ void first_step(const KpArgs& a, FirstStep& f, unsigned placed,
                                           unsigned claims) {
  placed = __reduce_add_sync(FULL, placed);
  claims = __reduce_add_sync(FULL, claims);
  if ((threadIdx.x & 31) != 0) return;
  atomicAdd(&f.placed, placed);
  atomicAdd(&f.claims, claims);
  __threadfence_block();
  if (atomicAdd(&f.warps, 1u) != KT / 32 - 1) return;
  // both counts in one word, so that they are of the same blocks (a step is
  // at most some 300K rows)
  const unsigned long long mine = (unsigned long long)*(volatile unsigned*)&f.placed << 32 |
                                  *(volatile unsigned*)&f.claims;
  const unsigned long long all = atomicAdd((unsigned long long*)&a.head->seen, mine) + mine;
  const unsigned long long P = all >> 32, C = all & 0xffffffffu;
  if (P < 16384) return;
  const float z = 1.5f * (float)P / (float)a.cap;
  if ((float)C > (float)P * ((1.0f - expf(-z)) / z + 0.005f)) a.head->full = 1;
}

// The block's rows folded in, KR a thread a step.  OWN: through the block's
// own table, by a warp while one row in eight finds its group there (looked
// at every eight steps).
template <bool OWN, bool ERRS>
__device__ __forceinline__ void kp_rows(const KpArgs& a, long long* own_key, long long* own_acc,
                                        long long from, long long to, long long& lo,
                                        long long& hi, unsigned& placed, unsigned& claims) {
  const int tid = threadIdx.x, W = a.W, na = a.acc.n, ncmp = a.acc.ncmp;
  const long long tile = (long long)KT * KR;
  bool own = OWN;
  int hits = 0, steps = 0;
  for (long long t0 = from; t0 < to; t0 += (long long)gridDim.x * tile) {
    if (__any_sync(FULL, *(volatile int*)&a.head->full)) break;  // the warp stays together
    const long long i0 = t0 + tid;
    long long h[KR];
    bool live[KR];
#pragma unroll
    for (int r = 0; r < KR; ++r) live[r] = i0 + r * KT < a.n;
    kp_hashes(a, i0, live, h);
    // each row's group (-1: none), in the block's table (bit r of in_own) or
    // in the global one
    int at[KR];
    unsigned in_own = 0;
#pragma unroll
    for (int r = 0; r < KR; ++r) {
      at[r] = -1;
      if (!live[r]) continue;
      lo = min(lo, h[r]);
      hi = max(hi, h[r]);
      if (OWN && own && h[r] != KP_EMPTY) {
        bool met;
        at[r] = own_place(own_key, a.cache, h[r], &met);
        hits += met;
        if (at[r] >= 0) in_own |= 1u << r;
      }
    }
    {
      // the usual case first: a group met before, in its first sector
      Sector sec[KR];
      int home[KR];
#pragma unroll
      for (int r = 0; r < KR; ++r) {
        home[r] = (int)kp_home(h[r], a.cap);
        if (live[r] && at[r] < 0) sec[r] = ld_sector(a.keys + home[r]);
      }
      bool more = false;
#pragma unroll
      for (int r = 0; r < KR; ++r) {
        if (!live[r] || at[r] >= 0) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (sec[r].w[j] == h[r]) at[r] = home[r] + j;
        if (h[r] == KP_EMPTY) at[r] = -1;
        more |= at[r] < 0;
      }
      if (more) {
#pragma unroll 1
        for (int q = 0; q < KR; ++q) {
          long long hq = 0;
          bool need = false;
#pragma unroll
          for (int r = 0; r < KR; ++r)
            if (r == q) {
              hq = h[r];
              need = live[r] && at[r] < 0;
            }
          if (!need) continue;
          const int g = kp_place_of(a, hq, claims);
          if (g < 0) a.head->full = 1;
#pragma unroll
          for (int r = 0; r < KR; ++r)
            if (r == q) at[r] = g;
        }
      }
    }
#pragma unroll
    for (int r = 0; r < KR; ++r) placed += at[r] >= 0;
    // the largest values, a sector of the groups' at a time
    for (int w0 = 0; w0 < ncmp; w0 += 4) {
      Sector sec[KR];
#pragma unroll
      for (int r = 0; r < KR; ++r)
        if (at[r] >= 0 && !(OWN && (in_own >> r & 1)))
          sec[r] = ld_sector(a.accs + (long long)at[r] * W + w0);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int k = w0 + j;
        if (k >= ncmp) break;
        long long v[KR];
        acc_values(a.acc, k, i0, at, v);
#pragma unroll
        for (int r = 0; r < KR; ++r) {
          if (at[r] < 0) continue;
          if (OWN && (in_own >> r & 1)) {
            long long* p = own_acc + at[r] * na + k;
            if (v[r] > *(volatile long long*)p) atomicMax(p, v[r]);
          } else if (v[r] > sec[r].w[j]) {
            red_max(a.accs + (long long)at[r] * W + k, v[r]);
          }
        }
      }
    }
    for (int k = ncmp; k < (ERRS ? a.acc.nplain : na); ++k) {
      long long v[KR];
      acc_values(a.acc, k, i0, at, v);
      const int is_float = a.acc.is_float[k];
#pragma unroll
      for (int r = 0; r < KR; ++r) {
        if (at[r] < 0) continue;
        if (OWN && (in_own >> r & 1)) add_to_shared(own_acc + at[r] * na + k, is_float, v[r]);
        else add_to(a.accs + (long long)at[r] * W + k, is_float, v[r]);
      }
    }
    for (int k = a.acc.nplain; ERRS && k < a.acc.nplain + a.acc.nerr; ++k) {
      const double* src = reinterpret_cast<const double*>(a.acc.src[k]);
      double v[KR];
#pragma unroll
      for (int r = 0; r < KR; ++r) v[r] = at[r] >= 0 ? __ldcs(src + i0 + r * KT) : 0.0;
#pragma unroll
      for (int r = 0; r < KR; ++r) {
        const bool in = OWN && (in_own >> r & 1);
        if (OWN) add_group_to_shared(own_acc, na, k, a.acc.nerr, in ? at[r] : -1, v[r]);
        if (!in && at[r] >= 0)
          add_with_error(a.accs + (long long)at[r] * W + k, a.acc.nerr, v[r], 0.0);
      }
    }
    if (OWN && own && (++steps & 7) == 0) {
      own = __reduce_add_sync(FULL, (unsigned)hits) >= 8u * KR * 32 / 8;
      hits = 0;
    }
  }
}

// ERRS: there are float64 sums whose errors are kept (3% of the others' time).
template <bool ERRS>
__global__ void __launch_bounds__(KT, PF_KP_MINB) k_kp_insert(KpArgs a) {
  extern __shared__ __align__(16) long long own_smem[];
  __shared__ long long red[2][KT / 32];
  __shared__ FirstStep first, total;
  const int tid = threadIdx.x, lane = tid & 31, W = a.W, na = a.acc.n, ncmp = a.acc.ncmp;
  long long* own_key = own_smem;              // [a.cache]
  long long* own_acc = own_smem + a.cache;    // [a.cache][na]
  for (int s = tid; s < a.cache; s += KT) own_key[s] = KP_EMPTY;
  if (tid == 0) first = total = FirstStep{0, 0, 0};
  __syncthreads();
  long long lo = LLONG_MAX, hi = LLONG_MIN;
  const long long tile = (long long)KT * KR;
  // the block's own table is used when its first KT rows meet some groups
  // twice (few or hot groups); else its claims and flush cost more than they
  // save
  bool own;
  {
    const long long i = (long long)blockIdx.x * tile + tid;
    bool live[KR], met = false;
    long long h[KR];
#pragma unroll
    for (int r = 0; r < KR; ++r) live[r] = r == 0 && i < a.n;
    kp_hashes(a, i, live, h);
    int at = -1;
    if (live[0] && h[0] != KP_EMPTY) at = own_place(own_key, a.cache, h[0], &met);
    // a claim that another row of the group won counts as a meeting too
    const int rows = __syncthreads_count(at >= 0);
    int claimed = 0;
    for (int s = tid; s < a.cache; s += KT) claimed += own_key[s] != KP_EMPTY;
    for (int o = 16; o; o >>= 1) claimed += __shfl_xor_sync(FULL, claimed, o);
    if (lane == 0) red[0][tid >> 5] = claimed;
    __syncthreads();
    for (int q = 0; q < KT / 32; ++q) claimed = q ? claimed + (int)red[0][q] : (int)red[0][0];
    own = rows - claimed >= KP_REPEATS;
    __syncthreads();
  }
  if (own)
    for (int s = tid; s < a.cache; s += KT)
      for (int k = 0; k < na; ++k) own_acc[s * na + k] = acc_start(a.acc, k);
  __syncthreads();
  unsigned placed = 0, claims = 0;  // a thread's, below 2^32 (at most 2^40 rows)
  const long long from = (long long)blockIdx.x * tile, step = (long long)gridDim.x * tile;
  if (own) {
    kp_rows<true, ERRS>(a, own_key, own_acc, from, a.n, lo, hi, placed, claims);
  } else {
    const bool look = a.cap < (unsigned long long)(a.n + a.n / 2 + 1);
#pragma unroll 1
    for (int part = look ? 0 : 1; part < 2; ++part) {
      const long long f = part && look ? from + step : from;
      kp_rows<false, ERRS>(a, own_key, own_acc, f, part ? a.n : min(a.n, from + step), lo, hi, placed,
                     claims);
      if (part == 0) {
        first_step(a, first, placed, claims);
        __syncthreads();
      }
    }
  }
  __syncthreads();
  // the block's own groups into the global table
  for (int s = tid; own && s < a.cache; s += KT) {
    const long long x = own_key[s];
    if (x == KP_EMPTY) continue;
    const int g = kp_place_of(a, x, claims);
    if (g < 0) {
      a.head->full = 1;
      continue;
    }
    long long* p = a.accs + (long long)g * W;
    const int nplain = ERRS ? a.acc.nplain : na, nerr = ERRS ? a.acc.nerr : 0;
    for (int k = 0; k < nplain + nerr; ++k) {
      const long long v = own_acc[s * na + k];
      if (k < ncmp) red_max(p + k, v);
      else if (!ERRS || k < nplain) add_to(p + k, a.acc.is_float[k], v);
      else add_with_error(p + k, nerr, __longlong_as_double(v),
                          __longlong_as_double(own_acc[s * na + k + nerr]));
    }
  }
  for (int o = 16; o; o >>= 1) {
    lo = min(lo, __shfl_xor_sync(FULL, lo, o));
    hi = max(hi, __shfl_xor_sync(FULL, hi, o));
  }
  placed = __reduce_add_sync(FULL, placed);
  claims = __reduce_add_sync(FULL, claims);
  if (lane == 0) {
    red[0][tid >> 5] = lo;
    red[1][tid >> 5] = hi;
    atomicAdd(&total.placed, placed);
    atomicAdd(&total.claims, claims);
  }
  __syncthreads();
  if (tid == 0) {
    for (int q = 0; q < KT / 32; ++q) {
      lo = min(lo, red[0][q]);
      hi = max(hi, red[1][q]);
    }
    if (lo <= hi) {
      atomicMin(&a.head->lo, lo);
      atomicMax(&a.head->hi, hi);
    }
    // what the caller's next attempt is sized by
    atomicAdd((unsigned long long*)&a.head->placed, (unsigned long long)total.placed);
    atomicAdd((unsigned long long*)&a.head->claimed, (unsigned long long)total.claims);
  }
}

// The bucket of a hash: the top log2(buckets) bits (three at least) of its place in
// the hashes' range, the range taken up to a power of two.
__device__ __forceinline__ unsigned kp_bucket(long long h, long long lo, long long hi,
                                              int log_buckets) {
  const unsigned long long r = (unsigned long long)hi - (unsigned long long)lo;
  const int up = r ? __clzll((long long)r) : 63;
  return (unsigned)((((unsigned long long)h - (unsigned long long)lo) << up) >>
                    (64 - log_buckets));
}

// Place s's hash, and whether a group holds it.
__device__ __forceinline__ bool kp_used(const KpArgs& a, unsigned long long s, long long* h) {
  const long long x = a.keys[s];
  *h = s == a.cap ? KP_EMPTY : x;
  return x != KP_EMPTY;
}

__global__ void __launch_bounds__(KT) k_kp_collect(KpArgs a, int log_buckets,
                                                   int* __restrict__ hist) {
  if (a.head->full) return;
  const long long lo = a.head->lo, hi = a.head->hi;
  for (unsigned long long s = (unsigned long long)blockIdx.x * KT + threadIdx.x; s <= a.cap;
       s += (unsigned long long)gridDim.x * KT) {
    long long h;
    if (kp_used(a, s, &h)) atomicAdd(&hist[kp_bucket(h, lo, hi, log_buckets)], 1);
  }
}

// One block: hist -> each bucket's first place (first[b]) and its cursor (the
// same, in hist); the groups, the fullest bucket.
__global__ void __launch_bounds__(1024) k_kp_scan(int* __restrict__ hist, int nbuckets,
                                                  int* __restrict__ first, KpHead* head) {
  __shared__ int wsum[32];
  __shared__ int wmax[32];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  int base = 0, most = 0;
  for (int b0 = 0; b0 < nbuckets; b0 += 4096) {
    const int b = b0 + tid * 4;
    int x[4], s = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      x[k] = b + k < nbuckets ? hist[b + k] : 0;
      s += x[k];
      most = max(most, x[k]);
    }
    int incl = s;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    int pre = base, tot = 0;
    for (int q = 0; q < 32; ++q) {
      pre += q < w ? wsum[q] : 0;
      tot += wsum[q];
    }
    int at = pre + incl - s;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (b + k < nbuckets) {
        first[b + k] = at;
        hist[b + k] = at;
      }
      at += x[k];
    }
    base += tot;
    __syncthreads();
  }
  most = (int)__reduce_max_sync(FULL, (unsigned)most);
  if (lane == 0) wmax[w] = most;
  __syncthreads();
  if (tid == 0) {
    for (int q = 0; q < 32; ++q) most = max(most, wmax[q]);
    first[nbuckets] = base;
    KpHead r = *head;
    r.groups = base;
    r.max_bucket = most;
    *head = r;
  }
}

struct KpList {
  long long* hash;
  long long* slot;
};

__global__ void __launch_bounds__(KT) k_kp_place(KpArgs a, int log_buckets,
                                                 int* __restrict__ cursor, KpList l,
                                                 KpHead* host) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *host = *a.head;
  if (a.head->full) return;
  const long long lo = a.head->lo, hi = a.head->hi;
  for (unsigned long long s = (unsigned long long)blockIdx.x * KT + threadIdx.x; s <= a.cap;
       s += (unsigned long long)gridDim.x * KT) {
    long long h;
    if (!kp_used(a, s, &h)) continue;
    const int at = atomicAdd(&cursor[kp_bucket(h, lo, hi, log_buckets)], 1);
    l.hash[at] = h;
    l.slot[at] = (long long)s;
  }
}

struct Outs {
  unsigned char* dst[KP_MAX_OUT];
  int op[KP_MAX_OUT];
  int acc[KP_MAX_OUT];
  int flip[KP_MAX_OUT];  // the accumulator holds its value's complement
  int err[KP_MAX_OUT];   // the accumulator of a float64 sum's errors, or -1
  int acc2[KP_MAX_OUT];
  int acc3[KP_MAX_OUT];
  int rb[KP_MAX_OUT];
  int word[KP_MAX_OUT];
  int n;
};

// A group's results at output row j.
__device__ __forceinline__ void put_group(const KpArgs& a, const Outs& o, long long j,
                                          long long slot) {
  const long long* acc = a.accs + slot * a.W;
  for (int q = 0; q < o.n; ++q) {
    long long x = o.flip[q] ? ~acc[o.acc[q]] : acc[o.acc[q]];
    if (o.err[q] >= 0) {
      const double s = __longlong_as_double(x);
      if (isfinite(s)) x = __double_as_longlong(s + __longlong_as_double(acc[o.err[q]]));
    }
    switch (o.op[q]) {
      case PF_KO_WORD: {
        unsigned char* d = o.dst[q] + j * o.rb[q] + 8 * o.word[q];
        const int nb = min(8, o.rb[q] - 8 * o.word[q]);
        if (nb == 8 && ((uintptr_t)d & 7) == 0) *reinterpret_cast<long long*>(d) = x;
        else if (nb == 4 && ((uintptr_t)d & 3) == 0) *reinterpret_cast<int*>(d) = (int)x;
        else
          for (int b = 0; b < nb; ++b) d[b] = (unsigned char)((unsigned long long)x >> (8 * b));
        break;
      }
      case PF_KO_I32: reinterpret_cast<int*>(o.dst[q])[j] = (int)x; break;
      case PF_KO_I32_MAX0: reinterpret_cast<int*>(o.dst[q])[j] = (int)max(x, 0LL); break;
      case PF_KO_I64_MAX0: reinterpret_cast<long long*>(o.dst[q])[j] = max(x, 0LL); break;
      case PF_KO_F32:
        reinterpret_cast<float*>(o.dst[q])[j] = (float)__longlong_as_double(x);
        break;
      case PF_KO_COUNT:
        reinterpret_cast<long long*>(o.dst[q])[j] = x - acc[o.acc2[q]];
        break;
      case PF_KO_AVG_I:
      case PF_KO_AVG_F: {
        double* d = reinterpret_cast<double*>(o.dst[q]) + 2 * j;
        d[0] = o.op[q] == PF_KO_AVG_F ? __longlong_as_double(x) : (double)x;
        d[1] = (double)(acc[o.acc2[q]] - acc[o.acc3[q]]);
        break;
      }
      default: reinterpret_cast<long long*>(o.dst[q])[j] = x; break;
    }
  }
}

// A warp a bucket of at most KP_BUCKET groups: each group's rank among them
// is the number of smaller hashes.
__global__ void __launch_bounds__(KT) k_kp_emit(KpArgs a, Outs o, KpList l,
                                                const int* __restrict__ first, int nbuckets,
                                                long long* __restrict__ hash_out) {
  __shared__ long long hs[KT / 32][KP_BUCKET];
  // crowded buckets: the host sorts the groups instead
  if (a.head->full || a.head->max_bucket > KP_BUCKET) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (long long b = (long long)blockIdx.x * (KT / 32) + w; b < nbuckets;
       b += (long long)gridDim.x * (KT / 32)) {
    const int f = first[b], n = first[b + 1] - f;
    __syncwarp();
    for (int e = lane; e < n; e += 32) hs[w][e] = l.hash[f + e];
    __syncwarp();
    for (int e = lane; e < n; e += 32) {
      const long long h = hs[w][e];
      int rank = 0;
      for (int q = 0; q < n; ++q) rank += hs[w][q] < h;
      hash_out[f + rank] = h;
      put_group(a, o, f + rank, l.slot[f + e]);
    }
  }
}

// The groups already in order (l sorted by hash).
__global__ void __launch_bounds__(KT) k_kp_emit_sorted(KpArgs a, Outs o, const long long* hash,
                                                       const long long* slot, long long n,
                                                       long long* __restrict__ hash_out) {
  for (long long j = (long long)blockIdx.x * KT + threadIdx.x; j < n;
       j += (long long)gridDim.x * KT) {
    hash_out[j] = hash[j];
    put_group(a, o, j, slot[j]);
  }
}

// The partition buckets of the groups' hashes and the groups per bucket.
__global__ void __launch_bounds__(KT) k_kp_buckets(const KpHead* head,
                                                   const long long* __restrict__ hash, int logB,
                                                   int* __restrict__ bucket,
                                                   long long* __restrict__ counts) {
  extern __shared__ int hc[];
  if (head->full) return;  // (crowded hashes: counted again once they are out)
  const int B = 1 << logB;
  for (int b = threadIdx.x; b < B; b += KT) hc[b] = 0;
  __syncthreads();
  const long long n = head->groups;
  for (long long i = (long long)blockIdx.x * KT + threadIdx.x; i < n;
       i += (long long)gridDim.x * KT) {
    const int b = bucket_of_hash(mix64((uint64_t)hash[i]), logB);
    bucket[i] = b;
    atomicAdd(&hc[b], 1);
  }
  __syncthreads();
  for (int b = threadIdx.x; b < B; b += KT)
    if (hc[b]) atomicAdd((unsigned long long*)&counts[b], (unsigned long long)hc[b]);
}

struct KpLayout {
  KpHead* head;
  long long* keys;
  long long* accs;
  int* hist;
  int* first;
  KpList list;
  unsigned long long cap;
  int W, log_buckets;
};

// Places for n rows of naccs accumulators: a power of two of at least 3 n / 2, the
// table of at most KP_TABLE_BYTES; with an expected number of groups, at
// least half more than them.
unsigned long long kp_places(long long n, int naccs, long long expect) {
  const int W = (std::max(naccs, 1) + 3) / 4 * 4;
  if (expect > 0)
    return pow2_at_least((uint64_t)std::max<long long>(1024, expect + expect / 2 + 1));
  unsigned long long most = 1024;
  while (most * 2 * (W + 1) * 8 <= KP_TABLE_BYTES) most *= 2;
  return std::min<unsigned long long>(
      most, std::max<unsigned long long>(1024, pow2_at_least((uint64_t)(n + n / 2 + 1))));
}

// The groups U of n rows of which the first `placed` held `claimed` of them:
// claimed = U (1 - exp(-placed / U)), each row's group drawn alike (bisected).
long long kp_estimate(long long placed, long long claimed, long long n) {
  if (claimed <= 0 || placed <= 0) return n;
  double lo = (double)claimed, hi = (double)std::max(n, claimed);
  for (int k = 0; k < 60; ++k) {
    const double u = 0.5 * (lo + hi);
    if (u * -std::expm1(-(double)placed / u) < (double)claimed) lo = u;
    else hi = u;
  }
  return (long long)hi;
}

KpLayout kp_layout(Arena& a, long long n, int naccs, long long expect) {
  KpLayout l{};
  l.W = (std::max(naccs, 1) + 3) / 4 * 4;
  l.cap = kp_places(n, naccs, expect);
  l.log_buckets = log2_exact(l.cap) - 7;  // about 128 places a bucket
  l.head = a.take<KpHead>(1);
  l.keys = a.take<long long>((size_t)l.cap + 4);
  l.accs = a.take<long long>((size_t)(l.cap + 1) * l.W);
  l.hist = a.take<int>((size_t)1 << l.log_buckets);
  l.first = a.take<int>(((size_t)1 << l.log_buckets) + 1);
  l.list.hash = a.take<long long>((size_t)l.cap + 1);
  l.list.slot = a.take<long long>((size_t)l.cap + 1);
  return l;
}

int row_path(const void* p, int rb) {
  const uintptr_t x = (uintptr_t)p;
  return rb % 8 == 0 && x % 8 == 0 ? 0 : rb == 4 && x % 4 == 0 ? 1 : 2;
}

// A host thread's pinned result words (kept).
struct KpHost {
  KpHead head;
  long long counts[KP_MAX_B];
};
KpHost* pinned_host() {
  thread_local KpHost* buf = nullptr;
  if (!buf && cudaHostAlloc((void**)&buf, sizeof(KpHost),
                            cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
    cudaGetLastError();
    buf = nullptr;
  }
  return buf;
}

unsigned kp_grid(long long work, int per_block, int blocks_a_sm) {
  return (unsigned)std::max<long long>(
      1, std::min<long long>((work + per_block - 1) / per_block,
                             (long long)sm_count() * blocks_a_sm));
}

// The accumulator that holds accumulator k's errors, or -1.
int err_of(const pf_keyed_acc* accs, int n, int k) {
  for (int q = 0; q < n; ++q)
    if (accs[q].op == PF_KA_SUM_ERR && accs[q].word == k) return q;
  return -1;
}

// The place of each of the caller's accumulators among the table's (Accs).
void place_accs(const pf_keyed_acc* accs, int n, int* place, Accs* out) {
  int at = 0;
  for (int k = 0; k < n; ++k)
    if (accs[k].op == PF_KA_WORD || accs[k].op == PF_KA_MIN || accs[k].op == PF_KA_MAX)
      place[k] = at++;
  out->ncmp = at;
  for (int k = 0; k < n; ++k)
    if (accs[k].op >= PF_KA_COUNT && accs[k].op <= PF_KA_SUM_F && err_of(accs, n, k) < 0)
      place[k] = at++;
  out->nplain = at;
  for (int k = 0; k < n; ++k)
    if (accs[k].op == PF_KA_SUM_F && err_of(accs, n, k) >= 0) place[k] = at++;
  out->nerr = at - out->nplain;
  for (int k = 0; k < n; ++k)
    if (accs[k].op == PF_KA_SUM_ERR) place[k] = place[accs[k].word] + out->nerr;
}

int fill_accs(const pf_keyed_acc* accs, int naccs, int* place, Accs* out) {
  for (int k0 = 0; k0 < naccs; ++k0) {
    const pf_keyed_acc& c = accs[k0];
    if (c.op < PF_KA_WORD || c.op > PF_KA_SUM_ERR || c.kind < PF_KK_I64 || c.kind > PF_KK_F32)
      return fail(PF_EINVAL, "keyed_pass1: accumulator %d: op %d of kind %d", k0, c.op, c.kind);
    const bool f = c.kind == PF_KK_F64 || c.kind == PF_KK_F32;
    const bool of_ints = c.op == PF_KA_SUM_I || c.op == PF_KA_MIN || c.op == PF_KA_MAX;
    if ((of_ints && f) || (c.op == PF_KA_SUM_F && !f) ||
        (c.op == PF_KA_SUM_ERR &&
         (c.word < 0 || c.word >= naccs || accs[c.word].op != PF_KA_SUM_F ||
          accs[c.word].kind != PF_KK_F64 || err_of(accs, naccs, c.word) != k0)))
      return fail(PF_EINVAL, "keyed_pass1: accumulator %d: op %d of kind %d", k0, c.op, c.kind);
    const bool no_column = c.op == PF_KA_COUNT || c.op == PF_KA_SUM_ERR;
    if (!no_column && !c.src)
      return fail(PF_EINVAL, "keyed_pass1: accumulator %d has a null column", k0);
    const int es = c.kind == PF_KK_I64 || c.kind == PF_KK_F64 ? 8 : 4;
    if (c.op == PF_KA_WORD) {
      if (c.row_bytes < 1 || c.word < 0 || 8 * c.word >= c.row_bytes)
        return fail(PF_EINVAL, "keyed_pass1: accumulator %d: word %d of %d bytes", k0, c.word,
                    c.row_bytes);
    } else if (!no_column && ((uintptr_t)c.src % es) != 0) {
      return fail(PF_EINVAL, "keyed_pass1: accumulator %d: a misaligned column", k0);
    }
  }
  place_accs(accs, naccs, place, out);
  for (int k0 = 0; k0 < naccs; ++k0) {
    const pf_keyed_acc& c = accs[k0];
    const int k = place[k0];
    const bool f = c.kind == PF_KK_F64 || c.kind == PF_KK_F32;
    static const int how_of[] = {H_I64, H_I32, H_F64, H_F32};
    const int path = c.op == PF_KA_WORD ? row_path(c.src, c.row_bytes) : 0;
    out->how[k] = c.op == PF_KA_COUNT  ? H_ONE
                  : c.op == PF_KA_WORD ? (path == 0 ? H_WORD8 : path == 1 ? H_WORD4 : H_WORD)
                                       : how_of[c.kind];
    out->src[k] = (const unsigned char*)c.src;
    out->rb[k] = c.row_bytes;
    out->word[k] = c.word;
    out->flip[k] = c.op == PF_KA_MIN ? -1 : 0;
    out->nulls[k] = c.op != PF_KA_NULLS ? 0 : f ? 2 : 1;
    out->is_float[k] = c.op == PF_KA_SUM_F;
  }
  out->n = naccs;
  return PF_OK;
}

int fill_outs(const pf_keyed_out* outs, int nouts, const pf_keyed_acc* accs, int naccs,
              const int* place, Outs* out) {
  for (int q = 0; q < nouts; ++q) {
    const pf_keyed_out& c = outs[q];
    if (!c.dst || c.op < PF_KO_WORD || c.op > PF_KO_AVG_F || c.acc < 0 || c.acc >= naccs ||
        c.acc2 < 0 || c.acc2 >= naccs || c.acc3 < 0 || c.acc3 >= naccs ||
        (c.op == PF_KO_WORD && (c.row_bytes < 1 || c.word < 0 || 8 * c.word >= c.row_bytes)))
      return fail(PF_EINVAL, "keyed_pass1: output %d", q);
    out->dst[q] = (unsigned char*)c.dst;
    out->op[q] = c.op;
    out->acc[q] = place[c.acc];
    out->flip[q] = accs[c.acc].op == PF_KA_MIN;
    const int err = err_of(accs, naccs, c.acc);
    out->err[q] = err < 0 ? -1 : place[err];
    out->acc2[q] = place[c.acc2];
    out->acc3[q] = place[c.acc3];
    out->rb[q] = c.row_bytes;
    out->word[q] = c.word;
  }
  out->n = nouts;
  return PF_OK;
}

}  // namespace
}  // namespace pf

using namespace pf;

extern "C" size_t pf_keyed_pass1_workspace(int64_t n, int naccs, int64_t expect) {
  Arena a(nullptr, 0);
  kp_layout(a, n, std::max(0, std::min(naccs, KP_MAX_ACC)), expect);
  return a.used + 256;
}

extern "C" int64_t pf_keyed_pass1_groups(int64_t n, int naccs, int64_t expect) {
  return std::min<int64_t>(
      n, (int64_t)kp_places(n, std::max(0, std::min(naccs, KP_MAX_ACC)), expect) + 1);
}

namespace {
// The call's arguments checked and laid out: what both halves share.
struct KpCall {
  KpArgs x;
  KpLayout l;
  int place[KP_MAX_ACC];
};
int kp_call(int64_t n, const pf_keyed_acc* accs, int naccs, int64_t expect, void* workspace,
            size_t workspace_bytes, KpCall* c) {
  if (naccs < 0 || naccs > KP_MAX_ACC)
    return fail(PF_EINVAL, "keyed_pass1: at most %d accumulators", KP_MAX_ACC);
  if (n < 0 || n > (1LL << 40) || expect < 0 || expect > (1LL << 28))
    return fail(PF_EINVAL, "keyed_pass1: bad rows or groups");
  c->x = KpArgs{};
  c->x.n = n;
  if (int rc = fill_accs(accs, naccs, c->place, &c->x.acc)) return rc;
  Arena ar(workspace, workspace_bytes);
  c->l = kp_layout(ar, n, naccs, expect);
  if (!workspace || !ar.fits())
    return fail(PF_ENOSPACE, "keyed_pass1: workspace of %zu bytes, %zu needed", workspace_bytes,
                ar.used);
  c->x.keys = c->l.keys;
  c->x.accs = c->l.accs;
  c->x.cap = c->l.cap;
  c->x.W = c->l.W;
  c->x.head = c->l.head;
  return PF_OK;
}
}  // namespace

extern "C" int pf_keyed_pass1_read(const void* const* key_cols, const int* row_bytes,
                                   const int64_t* const* coeffs, int ncols, int64_t n,
                                   const pf_keyed_acc* accs, int naccs, int64_t expect,
                                   void* workspace, size_t workspace_bytes, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (ncols < 1 || ncols > KP_MAX_KEYS)
    return fail(PF_EINVAL, "keyed_pass1: 1 to %d key columns", KP_MAX_KEYS);
  KpCall c;
  if (int rc = kp_call(n, accs, naccs, expect, workspace, workspace_bytes, &c)) return rc;
  if (n == 0) return ok();
  KpArgs& x = c.x;
  const KpLayout& l = c.l;
  x.key.n = ncols;
  for (int k = 0; k < ncols; ++k) {
    if (row_bytes[k] < 1 || !key_cols[k] || !coeffs[k])
      return fail(PF_EINVAL, "keyed_pass1: key column %d is null or has no bytes", k);
    x.key.col[k] = (const unsigned char*)key_cols[k];
    x.key.coeff[k] = (const long long*)coeffs[k];
    x.key.rb[k] = row_bytes[k];
    x.key.words[k] = (row_bytes[k] + 7) / 8;
    x.key.path[k] = row_path(key_cols[k], row_bytes[k]);
  }
  x.cache = 1;
  while ((size_t)x.cache * 2 * (1 + naccs) * 8 <= KP_CACHE_BYTES) x.cache *= 2;
  const size_t smem = (size_t)x.cache * (1 + naccs) * 8;
  const int nbuckets = 1 << l.log_buckets;
  {
    // a multiple of three blocks of 256 threads: whole groups of 4, 8, 12 or
    // 16 words a step
    PF_KERNEL("k_kp_init", st);
    k_kp_init<<<(unsigned)(sm_count() * 2 * 3), KT, 0, st>>>(x, l.hist, nbuckets);
  }
  PF_LAUNCH("k_kp_init");
  auto insert = x.acc.nerr ? k_kp_insert<true> : k_kp_insert<false>;
  if (int rc = opt_in_smem((const void*)insert, smem)) return rc;
  {
    PF_KERNEL("k_kp_insert", st);
    insert<<<kp_grid(n, KT * KR, PF_KP_MINB), KT, smem, st>>>(x);
  }
  PF_LAUNCH("k_kp_insert");
  {
    PF_KERNEL("k_kp_collect", st);
    k_kp_collect<<<kp_grid((long long)l.cap + 1, KT, 16), KT, 0, st>>>(x, l.log_buckets, l.hist);
  }
  PF_LAUNCH("k_kp_collect");
  {
    PF_KERNEL("k_kp_scan", st);
    k_kp_scan<<<1, 1024, 0, st>>>(l.hist, nbuckets, l.first, l.head);
  }
  PF_LAUNCH("k_kp_scan");
  return ok();
}

extern "C" int pf_keyed_pass1_emit(int64_t n, const pf_keyed_acc* accs, int naccs, int64_t expect,
                                   const pf_keyed_out* outs, int nouts, int64_t* hash_out, int B,
                                   int32_t* bucket_out, int64_t* counts_out,
                                   int64_t* host_counts, int64_t* n_groups, int64_t* crowded,
                                   void* workspace, size_t workspace_bytes, void* sort_workspace,
                                   size_t sort_workspace_bytes, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (nouts < 0 || nouts > KP_MAX_OUT || !n_groups || !crowded)
    return fail(PF_EINVAL, "keyed_pass1: at most %d outputs", KP_MAX_OUT);
  if (B < 1 || B > KP_MAX_B || (B & (B - 1)))
    return fail(PF_EINVAL, "keyed_pass1: B must be a power of two <= %d", KP_MAX_B);
  if (B > 1 && (!bucket_out || !counts_out || !host_counts))
    return fail(PF_EINVAL, "keyed_pass1: null buckets");
  KpCall c;
  if (int rc = kp_call(n, accs, naccs, expect, workspace, workspace_bytes, &c)) return rc;
  const bool sorted = *crowded != 0;  // the second call, with room for the sort
  *n_groups = 0;
  *crowded = 0;
  if (n == 0) return ok();
  if (!hash_out) return fail(PF_EINVAL, "keyed_pass1: null output");
  Outs o{};
  if (int rc = fill_outs(outs, nouts, accs, naccs, c.place, &o)) return rc;
  const KpArgs& x = c.x;
  const KpLayout& l = c.l;
  KpHost* host = pinned_host();
  KpHost* host_dev = nullptr;
  if (!host) return fail(PF_ECUDA, "keyed_pass1: no pinned result words");
  if (int rc = host_alias(host, (void**)&host_dev)) return rc;
  const int nbuckets = 1 << l.log_buckets, logB = log2_exact((uint64_t)B);
  cudaEvent_t ev;
  if (!sorted) {
    {
      PF_KERNEL("k_kp_place", st);
      k_kp_place<<<kp_grid((long long)l.cap + 1, KT, 16), KT, 0, st>>>(
          x, l.log_buckets, l.hist, l.list, &host_dev->head);
    }
    PF_LAUNCH("k_kp_place");
    if (B == 1)
      if (int rc = record_event(st, &ev)) return rc;
    {
      PF_KERNEL("k_kp_emit", st);
      k_kp_emit<<<kp_grid(nbuckets, KT / 32, 32), KT, 0, st>>>(x, o, l.list, l.first, nbuckets,
                                                              (long long*)hash_out);
    }
    PF_LAUNCH("k_kp_emit");
  } else {
    // hashes crowded into a few buckets of their range: the radix sort
    PF_CUDA(cudaMemcpyAsync(&host->head, l.head, sizeof(KpHead), cudaMemcpyDeviceToHost, st));
    if (int rc = wait_stream(st)) return rc;
    const long long groups = host->head.groups;
    Arena ea(sort_workspace, sort_workspace_bytes);
    long long* hs = ea.take<long long>((size_t)groups);
    long long* sl = ea.take<long long>((size_t)groups);
    const size_t sort_bytes = pf_sort_pairs_workspace(groups);
    unsigned char* sort_ws = ea.take<unsigned char>(sort_bytes);
    if (!sort_workspace || !ea.fits())
      return fail(PF_ENOSPACE, "keyed_pass1: sort workspace of %zu bytes, %zu needed",
                  sort_workspace_bytes, ea.used);
    if (int rc = pf_sort_pairs((const int64_t*)l.list.hash, (const int64_t*)l.list.slot, groups,
                               (int64_t*)hs, (int64_t*)sl, sort_ws, sort_bytes, stream))
      return rc;
    {
      PF_KERNEL("k_kp_emit", st);
      k_kp_emit_sorted<<<kp_grid(groups, KT, 16), KT, 0, st>>>(x, o, hs, sl, groups,
                                                              (long long*)hash_out);
    }
    PF_LAUNCH("k_kp_emit");
    if (B == 1)
      if (int rc = record_event(st, &ev)) return rc;
  }
  if (B > 1) {
    PF_CUDA(cudaMemsetAsync(counts_out, 0, sizeof(long long) * B, st));
    {
      PF_KERNEL("k_kp_buckets", st);
      k_kp_buckets<<<kp_grid((long long)l.cap, KT * 4, 4), KT, sizeof(int) * B, st>>>(
          l.head, (const long long*)hash_out, logB, bucket_out, (long long*)counts_out);
    }
    PF_LAUNCH("k_kp_buckets");
    PF_CUDA(cudaMemcpyAsync(host->counts, counts_out, sizeof(long long) * B,
                            cudaMemcpyDeviceToHost, st));
    if (int rc = record_event(st, &ev)) return rc;
  }
  if (int rc = wait_event(ev)) return rc;
  const KpHead head = host->head;
  if (!sorted && !head.full && head.max_bucket > KP_BUCKET) {
    *crowded = (int64_t)(pf_sort_pairs_workspace(head.groups) +
                         2 * ((size_t)head.groups * 8 + 256) + 512);
    return ok();
  }
  if (B > 1 && !head.full)
    for (int b = 0; b < B; ++b) host_counts[b] = host->counts[b];
  *n_groups = head.full ? -std::max(1LL, kp_estimate(head.placed, head.claimed, n)) : head.groups;
  return ok();
}
