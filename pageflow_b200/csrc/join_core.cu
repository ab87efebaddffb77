// The join cores, sm_100a replacements of tqpkernels.join_unique_hash,
// join_semi_anti and join_expand (reference operators/kernels/join_core.cu,
// wrapper operators/join_core.py):
//
//   unique hash  inner join on a build tuple (1-2 int64 keys) proven unique:
//                a table of 4-byte slots (the build row in the low r bits, r
//                the bit width of n_build; the tuple hash's bits above them as
//                a fingerprint) in buckets of one 32-byte sector; each probe
//                row's partner; the matched probe rows compacted in order
//   semi / anti  a set of the build keys (INT64_MIN marks an empty slot), with
//                an optional per-key min / max of one build column answering
//                a residual comparison; the kept probe rows compacted in order
//   expand       the pairs of the sort/search probe: each probe row's run of
//                equal build keys, in probe-row order
//
// Slots come from the tuple hash's bits just below its top nine (the radix
// bucket's bits, B <= 512, are shared by a bucket's keys).  Every kernel
// bounds its probe loop by the table's size.  Each call queues its kernels,
// writes its row count into the caller's pinned host_out through the device
// alias, and waits for that count once.
#include <climits>
#include <mutex>

#include "scan.cuh"

namespace pf {
namespace {

constexpr int T = 256;
constexpr unsigned EMPTY_SLOT = ~0u;
constexpr long long EMPTY_KEY = LLONG_MIN;

__device__ __forceinline__ uint64_t tuple_hash(long long k0, long long k1, bool two) {
  uint64_t h = mix64((uint64_t)k0);
  if (two) h = mix64(h ^ (mix64((uint64_t)k1) + 0x9e3779b97f4a7c15ULL + (h << 6) + (h >> 2)));
  return h;
}

// The home slot of a key in the semi / anti set: the multiply-shift of the bits
// right below its hash's top nine.
__device__ __forceinline__ unsigned long long set_home(uint64_t key, unsigned long long slots) {
  return __umul64hi(mix64(key) << 9, slots);
}

// ---- unique hash -------------------------------------------------------------
//
// A slot holds (hash << r) | row, rmask = 2^r - 1 with n_build <= rmask: a
// row never fills its r bits, so no entry is all ones (EMPTY_SLOT).  The home
// bucket is the multiply-shift of the hash's bits below its top nine onto
// [0, buckets), which leans on the high bits; the fingerprint takes the low
// ones.  A row leaves a bucket only when its eight slots are taken, so a bucket
// with a free one ends a lookup.
//
// A random read costs about the same whatever its size up to a sector: with
// linear probing a lookup read two slots and a build key (6M against 1.5M rows:
// 98 us), now a bucket and a build key (61 us).

struct UhTable {
  unsigned* slot;              // [8 * buckets]
  unsigned long long buckets;
  unsigned rmask;
  int rbits;
};

__device__ __forceinline__ unsigned long long uh_home(uint64_t h, unsigned long long buckets) {
  return __umul64hi(h << 9, buckets);
}

__device__ __forceinline__ unsigned long long uh_next(unsigned long long b,
                                                      unsigned long long buckets) {
  return b + 1 == buckets ? 0 : b + 1;
}

// Claims a slot without reading it first, from one that the fingerprint picks
// on (1.2 claims a row at 0.3 full; 1.5M rows 33 -> 24 us).
template <bool TWO>
__global__ void __launch_bounds__(T) k_uh_build(const long long* __restrict__ b0,
                                                const long long* __restrict__ b1, long long n,
                                                UhTable t) {
  const long long i = (long long)blockIdx.x * T + threadIdx.x;
  if (i >= n) return;
  const uint64_t h = tuple_hash(b0[i], TWO ? b1[i] : 0, TWO);
  const unsigned entry = ((unsigned)h << t.rbits) | (unsigned)i;
  unsigned long long b = uh_home(h, t.buckets);
  for (unsigned long long probes = 0; probes < t.buckets; ++probes) {
    for (unsigned k = 0; k < 8; ++k)
      if (atomicCAS(&t.slot[8 * b + (((unsigned)h + k) & 7)], EMPTY_SLOT, entry) == EMPTY_SLOT)
        return;
    b = uh_next(b, t.buckets);
  }
}

struct UhBucket {
  unsigned e[8];
};
__device__ __forceinline__ UhBucket uh_load(const unsigned* p) {
  UhBucket b;
  asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(b.e[0]), "=r"(b.e[1]), "=r"(b.e[2]), "=r"(b.e[3]), "=r"(b.e[4]),
                 "=r"(b.e[5]), "=r"(b.e[6]), "=r"(b.e[7])
               : "l"(p));
  return b;
}

// The slots of a bucket that hold the fingerprint, and whether one is free.
__device__ __forceinline__ unsigned uh_match(const UhBucket& b, unsigned fp, unsigned fmask,
                                             bool* open) {
  unsigned m = 0;
  *open = false;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    if (b.e[k] == EMPTY_SLOT) *open = true;
    else if ((b.e[k] & fmask) == fp) m |= 1u << k;
  }
  return m;
}

constexpr int UH_U = 2;  // probe rows a thread resolves together (6M: 61 us; 1 or 4: 70)
static_assert(CITEMS % UH_U == 0, "probe batches tile a thread's rows");

// Probe CB rows a block: partner[i] (build row or -1), the block's matches.
// UH_U rows at a time: their home buckets loaded together, then their first
// candidates' keys; a row that those do not settle walks from its home bucket.
template <bool TWO>
__global__ void __launch_bounds__(CT) k_uh_probe(const long long* __restrict__ b0,
                                                 const long long* __restrict__ b1,
                                                 const long long* __restrict__ p0,
                                                 const long long* __restrict__ p1, long long n,
                                                 UhTable t, int* __restrict__ partner,
                                                 long long* __restrict__ bcnt) {
  const unsigned fmask = ~t.rmask;
  const long long base = (long long)blockIdx.x * CB;
  int c = 0;
  for (int kk = 0; kk < CITEMS; kk += UH_U) {
    long long k0[UH_U], k1[UH_U];
    unsigned fp[UH_U];
    unsigned long long home[UH_U];
    UhBucket bu[UH_U];
    int cand[UH_U];
    bool settled[UH_U];
#pragma unroll
    for (int u = 0; u < UH_U; ++u) {
      const long long i = base + (kk + u) * CT + threadIdx.x;
      k0[u] = i < n ? __ldcs(p0 + i) : 0;
      k1[u] = TWO && i < n ? __ldcs(p1 + i) : 0;
    }
#pragma unroll
    for (int u = 0; u < UH_U; ++u) {
      const uint64_t h = tuple_hash(k0[u], k1[u], TWO);
      fp[u] = (unsigned)h << t.rbits;
      home[u] = uh_home(h, t.buckets);
      if (base + (kk + u) * CT + threadIdx.x < n) bu[u] = uh_load(t.slot + 8 * home[u]);
    }
    // the first candidate (-1: none), and whether a miss of it settles the row
#pragma unroll
    for (int u = 0; u < UH_U; ++u) {
      cand[u] = -1;
      settled[u] = true;
      if (base + (kk + u) * CT + threadIdx.x >= n) continue;
      bool open;
      const unsigned m = uh_match(bu[u], fp[u], fmask, &open);
      unsigned e = 0;
#pragma unroll
      for (int k = 7; k >= 0; --k)
        if (m >> k & 1) e = bu[u].e[k];
      if (m) cand[u] = (int)(e & t.rmask);
      settled[u] = open && (m & (m - 1)) == 0;
    }
    long long c0[UH_U], c1[UH_U];
#pragma unroll
    for (int u = 0; u < UH_U; ++u) {
      c0[u] = cand[u] >= 0 ? b0[cand[u]] : 0;
      c1[u] = TWO && cand[u] >= 0 ? b1[cand[u]] : 0;
    }
#pragma unroll
    for (int u = 0; u < UH_U; ++u) {
      const long long i = base + (kk + u) * CT + threadIdx.x;
      int r = cand[u] >= 0 && c0[u] == k0[u] && (!TWO || c1[u] == k1[u]) ? cand[u] : -1;
      if (r < 0 && !settled[u]) {
        // another slot of its fingerprint, or a full bucket
        unsigned long long b = home[u];
        for (unsigned long long probes = 0; probes < t.buckets && r < 0; ++probes) {
          bool open = false;
          for (int k = 0; k < 8 && r < 0; ++k) {
            const unsigned e = t.slot[8 * b + k];
            if (e == EMPTY_SLOT) {
              open = true;
              continue;
            }
            if ((e & fmask) != fp[u]) continue;
            const int row = (int)(e & t.rmask);
            if (b0[row] == k0[u] && (!TWO || b1[row] == k1[u])) r = row;
          }
          if (open) break;
          b = uh_next(b, t.buckets);
        }
      }
      if (i < n) {
        partner[i] = r;
        c += r >= 0;
      }
    }
  }
  __shared__ int red[CT / 32];
  for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(FULL, c, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    int s = 0;
    for (int q = 0; q < CT / 32; ++q) s += red[q];
    bcnt[blockIdx.x] = s;
  }
}

// The matched probe rows of each block, in order, from the block's offset.
__global__ void __launch_bounds__(CT) k_uh_emit(const int* __restrict__ partner, long long n,
                                                const long long* __restrict__ boff,
                                                long long* __restrict__ build_idx,
                                                long long* __restrict__ probe_idx) {
  __shared__ int wsum[CT / 32];
  const long long base = (long long)blockIdx.x * CB + (long long)threadIdx.x * CITEMS;
  bool keep[CITEMS];
  int part[CITEMS], rank[CITEMS];
  if (base + CITEMS <= n) {
    const int4* v = reinterpret_cast<const int4*>(partner + base);
#pragma unroll
    for (int q = 0; q < CITEMS / 4; ++q) {
      const int4 x = v[q];
      part[4 * q] = x.x;
      part[4 * q + 1] = x.y;
      part[4 * q + 2] = x.z;
      part[4 * q + 3] = x.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < CITEMS; ++k) part[k] = base + k < n ? partner[base + k] : -1;
  }
#pragma unroll
  for (int k = 0; k < CITEMS; ++k) keep[k] = part[k] >= 0;
  __shared__ unsigned short rows[CB];
  __shared__ int sp[CB];
  const int tot = block_ranks(keep, rank, wsum);
#pragma unroll
  for (int k = 0; k < CITEMS; ++k) {
    if (keep[k]) {
      rows[rank[k]] = (unsigned short)(threadIdx.x * CITEMS + k);
      sp[rank[k]] = part[k];
    }
  }
  __syncthreads();
  const long long o = boff[blockIdx.x], b0 = (long long)blockIdx.x * CB;
  for (int e = threadIdx.x; e < tot; e += CT) {
    build_idx[o + e] = sp[e];
    probe_idx[o + e] = b0 + rows[e];
  }
}

// ---- semi / anti ----------------------------------------------------------------

// A slot is W words: the key, the minimum or maximum (W 2) or both and one
// unused (W 4, a 32-byte sector), so that one random read answers a probe row
// (a != residual with the three in arrays of their own: 20M rows against 6M 1180
// us, so 895; build and reset for 400K rows 33 us, so 23).

template <int W>
__device__ __forceinline__ void set_load(const long long* slot, long long (&x)[4]) {
  if (W == 4)
    asm volatile("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(x[0]), "=l"(x[1]), "=l"(x[2]), "=l"(x[3])
                 : "l"(slot));
  else if (W == 2)
    asm volatile("ld.global.v2.b64 {%0, %1}, [%2];" : "=l"(x[0]), "=l"(x[1]) : "l"(slot));
  else
    asm volatile("ld.global.b64 %0, [%1];" : "=l"(x[0]) : "l"(slot));
}

// The empty set, 16 bytes at a time.  least: word 1 is a maximum (W 2), else a
// minimum.
template <int W>
__global__ void __launch_bounds__(T) k_set_reset(longlong2* table, long long pairs, bool least) {
  for (long long i = (long long)blockIdx.x * T + threadIdx.x; i < pairs;
       i += (long long)gridDim.x * T)
    table[i] = W == 4 && (i & 1) ? make_longlong2(LLONG_MIN, 0)
               : W == 1          ? make_longlong2(EMPTY_KEY, EMPTY_KEY)
                                 : make_longlong2(EMPTY_KEY, least ? LLONG_MIN : LLONG_MAX);
}

template <int W>
__global__ void __launch_bounds__(T) k_set_build(const long long* __restrict__ key,
                                                 const long long* __restrict__ val, long long n,
                                                 long long* table, unsigned long long slots,
                                                 bool least, long long* bad) {
  const long long i = (long long)blockIdx.x * T + threadIdx.x;
  if (i >= n) return;
  const long long k = key[i];
  if (k == EMPTY_KEY) {
    *bad = 1;
    return;
  }
  unsigned long long s = set_home((uint64_t)k, slots);
  long long x[4];
  bool in = false;
  for (unsigned long long probes = 0; probes < slots; ++probes) {
    set_load<W>(table + W * s, x);
    if (x[0] == EMPTY_KEY)
      x[0] = (long long)atomicCAS((unsigned long long*)&table[W * s],
                                  (unsigned long long)EMPTY_KEY, (unsigned long long)k);
    if (x[0] == EMPTY_KEY || x[0] == k) {
      in = true;
      break;
    }
    s = s + 1 == slots ? 0 : s + 1;
  }
  if (!in) {
    *bad = 2;  // the set is full: there are more slots than rows
    return;
  }
  if (W == 1) return;
  const long long v = val[i];
  if ((W == 4 || !least) && v < x[1]) atomicMin(&table[W * s + 1], v);
  if (W == 2 && least && v > x[1]) atomicMax(&table[W * s + 1], v);
  if (W == 4 && v > x[2]) atomicMax(&table[W * s + 2], v);
}

constexpr int SA_U = 2;
static_assert(CITEMS % SA_U == 0, "probe batches tile a thread's rows");

// SA_U rows a thread at a time, their slots loaded together (2.5M rows: 29.8
// us; 1 row 32.4, 4 rows 42.4, blocks of 512 or 1024 31.7 and 30.4).
template <int W>
__global__ void __launch_bounds__(CT) k_set_probe(const long long* __restrict__ key,
                                                  const long long* __restrict__ val, long long n,
                                                  const long long* __restrict__ table,
                                                  unsigned long long slots, int op, bool anti,
                                                  unsigned char* __restrict__ keep,
                                                  long long* __restrict__ bcnt) {
  const long long base = (long long)blockIdx.x * CB;
  int c = 0;
  for (int kk = 0; kk < CITEMS; kk += SA_U) {
    long long k[SA_U], v[SA_U], x[SA_U][4];
    unsigned long long s[SA_U];
#pragma unroll
    for (int u = 0; u < SA_U; ++u) {
      const long long i = base + (kk + u) * CT + threadIdx.x;
      k[u] = i < n ? __ldcs(key + i) : EMPTY_KEY;
      v[u] = W > 1 && i < n ? __ldcs(val + i) : 0;
    }
#pragma unroll
    for (int u = 0; u < SA_U; ++u) {
      s[u] = set_home((uint64_t)k[u], slots);
      set_load<W>(table + W * s[u], x[u]);
    }
#pragma unroll
    for (int u = 0; u < SA_U; ++u) {
      // the key's slot, or an empty one
      for (unsigned long long probes = 1;
           probes < slots && x[u][0] != k[u] && x[u][0] != EMPTY_KEY; ++probes) {
        s[u] = s[u] + 1 == slots ? 0 : s[u] + 1;
        set_load<W>(table + W * s[u], x[u]);
      }
      const long long i = base + (kk + u) * CT + threadIdx.x;
      if (i >= n) continue;
      bool hit = x[u][0] == k[u] && k[u] != EMPTY_KEY;
      if (W > 1 && hit) {
        switch (op) {
          case PF_OP_NE: hit = x[u][1] != v[u] || x[u][W == 4 ? 2 : 1] != v[u]; break;
          case PF_OP_LT: hit = x[u][1] < v[u]; break;
          case PF_OP_LE: hit = x[u][1] <= v[u]; break;
          case PF_OP_GT: hit = x[u][1] > v[u]; break;
          default: hit = x[u][1] >= v[u]; break;
        }
      }
      const bool kp = hit != anti;
      keep[i] = kp;
      c += kp;
    }
  }
  __shared__ int red[CT / 32];
  for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(FULL, c, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int q = 0; q < CT / 32; ++q) t += red[q];
    bcnt[blockIdx.x] = t;
  }
}

__global__ void __launch_bounds__(CT) k_keep_emit(const unsigned char* __restrict__ keep,
                                                  long long n, const long long* __restrict__ boff,
                                                  long long* __restrict__ out) {
  __shared__ int wsum[CT / 32];
  const long long base = (long long)blockIdx.x * CB + (long long)threadIdx.x * CITEMS;
  bool kp[CITEMS];
  int rank[CITEMS];
  if (base + CITEMS <= n) {
    const uint4 x = *reinterpret_cast<const uint4*>(keep + base);
    const unsigned w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int k = 0; k < CITEMS; ++k) kp[k] = ((w[k / 4] >> (8 * (k % 4))) & 0xffu) != 0;
  } else {
#pragma unroll
    for (int k = 0; k < CITEMS; ++k) kp[k] = base + k < n && keep[base + k];
  }
  __shared__ unsigned short rows[CB];
  const int tot = block_compact(kp, rank, rows, wsum);
  const long long o = boff[blockIdx.x], b0 = (long long)blockIdx.x * CB;
  for (int e = threadIdx.x; e < tot; e += CT) out[o + e] = b0 + rows[e];
}

// ---- expand ---------------------------------------------------------------------

constexpr int EITEMS = 8;

// Thread t covers pairs [t*EITEMS, t*EITEMS + EITEMS): one binary search for
// the probe row of its first pair, then a walk.
__global__ void __launch_bounds__(T) k_expand(const long long* __restrict__ sorted_ids,
                                              const long long* __restrict__ start,
                                              const long long* __restrict__ len,
                                              const long long* __restrict__ incl, long long m,
                                              long long n_pairs, long long* __restrict__ cs,
                                              long long* __restrict__ cr) {
  const long long k0 = ((long long)blockIdx.x * T + threadIdx.x) * EITEMS;
  if (k0 >= n_pairs) return;
  long long lo = 0, hi = m - 1;  // first i with incl[i] > k0
  while (lo < hi) {
    const long long mid = (lo + hi) >> 1;
    if (incl[mid] <= k0) lo = mid + 1;
    else hi = mid;
  }
  long long i = lo;
  long long end = incl[i];
  for (int e = 0; e < EITEMS; ++e) {
    const long long k = k0 + e;
    if (k >= n_pairs) break;
    while (end <= k && i + 1 < m) end = incl[++i];
    const long long first = end - len[i];
    cs[k] = sorted_ids[start[i] + (k - first)];
    cr[k] = i;
  }
}

struct UhLayout {
  UhTable table;
  int* partner;
  long long* bcnt;
  long long* total;
};

UhLayout uh_layout(Arena& a, long long nb, long long np) {
  UhLayout l{};
  l.table.buckets = (unsigned long long)std::max<long long>(2 * nb / 8, 1);
  int r = 1;
  while (r < 31 && (1LL << r) - 1 < nb) ++r;  // nb <= 2^r - 1 (nb < 2^31)
  l.table.rbits = r;
  l.table.rmask = (1u << r) - 1;
  l.table.slot = a.take<unsigned>(8 * l.table.buckets);
  l.partner = a.take<int>(std::max<long long>(np, 1));
  l.bcnt = a.take<long long>((np + CB - 1) / CB + 1);
  l.total = a.take<long long>(1);
  return l;
}

// The scratch holds a table half full.  One 0.3 full is faster while L2 holds it
// (a lookup that leaves its bucket holds up its warp; 1.5M x 6M rows: build and
// probe 24 + 61 us, half full 35 + 85); it lies in the probe row output, which
// nothing writes before the last lookup is done, where that is large enough,
// aligned and none of the inputs.
constexpr long long UH_ROOMY = (64LL << 20) / 32;  // buckets

void uh_roomy(UhLayout& l, const int64_t* b0, const int64_t* b1, long long nb,
              const int64_t* p0, const int64_t* p1, long long np, int64_t* probe_idx) {
  const long long room = (nb * 10 / 3 + 7) / 8;
  if (room > UH_ROOMY || room * 32 > np * 8 || ((uintptr_t)probe_idx & 31)) return;
  auto apart = [&](const int64_t* x, long long n) {
    return !x || x + n <= probe_idx || probe_idx + np <= x;
  };
  if (!apart(b0, nb) || !apart(b1, nb) || !apart(p0, np) || !apart(p1, np)) return;
  l.table.slot = (unsigned*)probe_idx;
  l.table.buckets = (unsigned long long)std::max<long long>(room, 1);
}

// Queues the table's reset, build and probe, and the scan of the probe
// blocks' match counts (the total also into *count, a device address).
int uh_queue(const UhLayout& l, const int64_t* build0, const int64_t* build1, int64_t nb,
             const int64_t* probe0, const int64_t* probe1, int64_t np, int nkeys,
             long long* count, cudaStream_t st) {
  PF_CUDA(cudaMemsetAsync(l.table.slot, 0xff, 8 * l.table.buckets * sizeof(unsigned), st));
  const unsigned nblk = blocks_for(np, CB);
  const long long* b0 = (const long long*)build0;
  const long long* b1 = (const long long*)(nkeys == 2 ? build1 : build0);
  const long long* p0 = (const long long*)probe0;
  const long long* p1 = (const long long*)(nkeys == 2 ? probe1 : probe0);
  if (nkeys == 2) {
    {
      PF_KERNEL("k_uh_build", st);
      k_uh_build<true><<<blocks_for(nb, T), T, 0, st>>>(b0, b1, nb, l.table);
    }
    {
      PF_KERNEL("k_uh_probe", st);
      k_uh_probe<true><<<nblk, CT, 0, st>>>(b0, b1, p0, p1, np, l.table, l.partner, l.bcnt);
    }
  } else {
    {
      PF_KERNEL("k_uh_build", st);
      k_uh_build<false><<<blocks_for(nb, T), T, 0, st>>>(b0, b1, nb, l.table);
    }
    {
      PF_KERNEL("k_uh_probe", st);
      k_uh_probe<false><<<nblk, CT, 0, st>>>(b0, b1, p0, p1, np, l.table, l.partner, l.bcnt);
    }
  }
  PF_LAUNCH("k_uh_build/k_uh_probe");
  {
    PF_KERNEL("k_scan_counts", st);
    k_scan_counts<<<1, 1024, 0, st>>>(l.bcnt, nblk, l.total, count);
  }
  PF_LAUNCH("k_scan_counts");
  return PF_OK;
}

int uh_emit(const UhLayout& l, int64_t np, int64_t* build_idx, int64_t* probe_idx,
            cudaStream_t st) {
  {
    PF_KERNEL("k_uh_emit", st);
    k_uh_emit<<<blocks_for(np, CB), CT, 0, st>>>(l.partner, np, l.bcnt, (long long*)build_idx,
                                                 (long long*)probe_idx);
  }
  PF_LAUNCH("k_uh_emit");
  return PF_OK;
}

constexpr unsigned long long SA_SLOTS = 1ULL << 26;  // 2 GiB

struct SaLayout {
  long long* table;
  int words;                 // a slot's (1, 2, 4)
  unsigned long long slots;
  unsigned char* keep;
  long long* bcnt;
  long long* total;
};

SaLayout sa_layout(Arena& a, long long nb, long long np, int op) {
  SaLayout l{};
  l.slots = pow2_at_least((uint64_t)std::max<long long>(2 * nb, 2));
  l.words = op == PF_OP_NONE ? 1 : op == PF_OP_NE ? 4 : 2;
  // a slot of a sector where three words would do: at most two thirds full in
  // the same bytes once those matter
  if (l.words == 4 && l.slots > SA_SLOTS) l.slots = l.slots / 4 * 3;
  l.table = a.take<long long>(l.words * l.slots);
  l.keep = a.take<unsigned char>(std::max<long long>(np, 1));
  l.bcnt = a.take<long long>((np + CB - 1) / CB + 1);
  l.total = a.take<long long>(1);
  return l;
}

template <int W>
int sa_queue(const SaLayout& l, const int64_t* bk, long long nb, const int64_t* pk, long long np,
             const int64_t* bv, const int64_t* pv, int op, bool anti, long long* bad,
             cudaStream_t st) {
  const bool least = op == PF_OP_GT || op == PF_OP_GE;
  {
    PF_KERNEL("k_set_reset", st);
    const uint64_t pairs = W * l.slots / 2;  // an even number of slots
    k_set_reset<W><<<(unsigned)std::min<uint64_t>((pairs + T - 1) / T, 8192), T, 0, st>>>(
        (longlong2*)l.table, (long long)pairs, least);
  }
  PF_LAUNCH("k_set_reset");
  {
    PF_KERNEL("k_set_build", st);
    k_set_build<W><<<blocks_for(nb, T), T, 0, st>>>((const long long*)bk, (const long long*)bv,
                                                    nb, l.table, l.slots, least, bad);
  }
  PF_LAUNCH("k_set_build");
  {
    PF_KERNEL("k_set_probe", st);
    k_set_probe<W><<<blocks_for(np, CB), CT, 0, st>>>((const long long*)pk, (const long long*)pv,
                                                      np, l.table, l.slots, op, anti, l.keep,
                                                      l.bcnt);
  }
  PF_LAUNCH("k_set_probe");
  return PF_OK;
}

}  // namespace
}  // namespace pf

using namespace pf;

extern "C" size_t pf_join_unique_hash_workspace(int64_t n_build, int64_t n_probe) {
  Arena a(nullptr, 0);
  uh_layout(a, n_build, n_probe);
  return a.used + 256;
}

extern "C" int pf_join_unique_hash(const int64_t* build0, const int64_t* build1, int64_t n_build,
                                   const int64_t* probe0, const int64_t* probe1, int64_t n_probe,
                                   int nkeys, int64_t* build_idx, int64_t* probe_idx,
                                   int64_t* host_out, void* workspace, size_t workspace_bytes,
                                   void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (nkeys != 1 && nkeys != 2) return fail(PF_EINVAL, "join_unique_hash: one or two keys, got %d", nkeys);
  if (n_build < 1 || n_probe < 1)
    return fail(PF_EINVAL, "join_unique_hash: unique hash needs rows on both sides");
  if (n_build > PF_JOIN_MAX_ROWS || n_probe > PF_JOIN_MAX_ROWS)
    return fail(PF_EINVAL, "join_unique_hash: a call takes at most %lld rows a side",
                (long long)PF_JOIN_MAX_ROWS);
  if (!build0 || !probe0 || (nkeys == 2 && (!build1 || !probe1)) || !build_idx || !probe_idx)
    return fail(PF_EINVAL, "join_unique_hash: null column");
  Arena a(workspace, workspace_bytes);
  UhLayout l = uh_layout(a, n_build, n_probe);
  if (!workspace || !a.fits())
    return fail(PF_ENOSPACE, "join_unique_hash: workspace of %zu bytes, %zu needed",
                workspace_bytes, a.used);
  uh_roomy(l, build0, nkeys == 2 ? build1 : nullptr, n_build, probe0,
           nkeys == 2 ? probe1 : nullptr, n_probe, probe_idx);
  long long* host_dev = nullptr;
  if (int rc = host_alias(host_out, (void**)&host_dev)) return rc;
  host_out[1] = 0;
  if (int rc = uh_queue(l, build0, build1, n_build, probe0, probe1, n_probe, nkeys, host_dev, st))
    return rc;
  cudaEvent_t ev;
  if (int rc = record_event(st, &ev)) return rc;
  if (int rc = uh_emit(l, n_probe, build_idx, probe_idx, st)) return rc;
  if (int rc = wait_event(ev)) return rc;
  return ok();
}

extern "C" size_t pf_join_semi_anti_workspace(int64_t n_build, int64_t n_probe, int op) {
  Arena a(nullptr, 0);
  sa_layout(a, n_build, n_probe, op);
  return a.used + 256;
}

extern "C" int pf_join_semi_anti(const int64_t* build_key, int64_t n_build,
                                 const int64_t* probe_key, int64_t n_probe,
                                 const int64_t* build_val, const int64_t* probe_val, int op,
                                 int anti, int64_t* out, int64_t* host_out, void* workspace,
                                 size_t workspace_bytes, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (n_build < 1 || n_probe < 1)
    return fail(PF_EINVAL, "join_semi_anti: semi/anti needs rows on both sides");
  if (n_probe > PF_JOIN_MAX_ROWS || n_build > PF_JOIN_MAX_ROWS)
    return fail(PF_EINVAL, "join_semi_anti: a call takes at most %lld rows a side",
                (long long)PF_JOIN_MAX_ROWS);
  if (op < PF_OP_NONE || op > PF_OP_GE) return fail(PF_EINVAL, "join_semi_anti: unknown residual operator %d", op);
  if (op != PF_OP_NONE && (!build_val || !probe_val))
    return fail(PF_EINVAL, "join_semi_anti: a residual needs both value columns");
  Arena a(workspace, workspace_bytes);
  SaLayout l = sa_layout(a, n_build, n_probe, op);
  if (!workspace || !a.fits())
    return fail(PF_ENOSPACE, "join_semi_anti: workspace of %zu bytes, %zu needed", workspace_bytes,
                a.used);
  long long* host_dev = nullptr;
  if (int rc = host_alias(host_out, (void**)&host_dev)) return rc;
  host_out[0] = 0;
  host_out[1] = 0;  // the build sets it through the alias
  auto queue = l.words == 1 ? sa_queue<1> : l.words == 2 ? sa_queue<2> : sa_queue<4>;
  if (int rc = queue(l, build_key, n_build, probe_key, n_probe, build_val, probe_val, op,
                     anti != 0, host_dev + 1, st))
    return rc;
  const unsigned nblk = blocks_for(n_probe, CB);
  {
    PF_KERNEL("k_scan_counts", st);
    k_scan_counts<<<1, 1024, 0, st>>>(l.bcnt, nblk, l.total, host_dev);
  }
  PF_LAUNCH("k_scan_counts");
  cudaEvent_t ev;
  if (int rc = record_event(st, &ev)) return rc;
  {
    PF_KERNEL("k_keep_emit", st);
    k_keep_emit<<<nblk, CT, 0, st>>>(l.keep, n_probe, l.bcnt, (long long*)out);
  }
  PF_LAUNCH("k_keep_emit");
  if (int rc = wait_event(ev)) return rc;
  if (host_out[1] == 2) return fail(PF_EDEVICE, "join_semi_anti: the key set overflowed");
  return ok();
}

extern "C" size_t pf_join_expand_workspace(int64_t m) {
  Arena a(nullptr, 0);
  a.take<long long>(std::max<int64_t>(m, 1));           // incl
  a.take<long long>(1);                                 // total
  a.take<long long>(scan_scratch_elems(std::max<int64_t>(m, 1)));
  return a.used + 256;
}

namespace {
struct ExLayout {
  long long* incl;
  long long* total;
  long long* scratch;
};
ExLayout ex_layout(Arena& a, int64_t m) {
  ExLayout l{};
  l.incl = a.take<long long>(std::max<int64_t>(m, 1));
  l.total = a.take<long long>(1);
  l.scratch = a.take<long long>(scan_scratch_elems(std::max<int64_t>(m, 1)));
  return l;
}
}  // namespace

extern "C" int pf_join_expand_prepare(const int64_t* len, int64_t m, int64_t* host_out,
                                      void* workspace, size_t workspace_bytes, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (m < 0 || m > PF_JOIN_MAX_ROWS)
    return fail(PF_EINVAL, "join_expand: at most %lld probe rows", (long long)PF_JOIN_MAX_ROWS);
  Arena a(workspace, workspace_bytes);
  ExLayout l = ex_layout(a, m);
  if (!workspace || !a.fits())
    return fail(PF_ENOSPACE, "join_expand: workspace of %zu bytes, %zu needed", workspace_bytes,
                a.used);
  long long* host_dev = nullptr;
  if (int rc = host_alias(host_out, (void**)&host_dev)) return rc;
  if (m == 0) {
    host_out[0] = 0;
    return ok();
  }
  if (int rc = scan_i64((const long long*)len, l.incl, m, true, l.total, l.scratch, st)) return rc;
  {
    PF_KERNEL("k_copy_i64", st);
    k_copy_i64<<<1, 32, 0, st>>>(l.total, host_dev, 1);
  }
  PF_LAUNCH("k_copy_i64");
  if (int rc = wait_stream(st)) return rc;
  return ok();
}

extern "C" int pf_join_expand(const int64_t* sorted_ids, const int64_t* start, const int64_t* len,
                              int64_t m, int64_t n_pairs, int64_t* cs, int64_t* cr,
                              void* workspace, size_t workspace_bytes, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (n_pairs <= 0 || m <= 0) return ok();
  Arena a(workspace, workspace_bytes);
  ExLayout l = ex_layout(a, m);
  if (!workspace || !a.fits())
    return fail(PF_ENOSPACE, "join_expand: workspace of %zu bytes, %zu needed", workspace_bytes,
                a.used);
  const long long threads = (n_pairs + EITEMS - 1) / EITEMS;
  {
    PF_KERNEL("k_expand", st);
    k_expand<<<blocks_for(threads, T), T, 0, st>>>((const long long*)sorted_ids,
                                                   (const long long*)start, (const long long*)len,
                                                   l.incl, m, n_pairs, (long long*)cs,
                                                   (long long*)cr);
  }
  PF_LAUNCH("k_expand");
  return ok();
}

// ---- unique hash join on static scratch (allocates nothing) -------------------
//
// pf_join_unique_hash with its scratch (hash table, per-row partners, per-block
// counts) in one file-scope device array instead of a caller's workspace, and
// its match count left on the device instead of a host wait.  The first call
// on a device, with that device current, looks the array's address up once
// (cudaGetSymbolAddress, which also loads this module on that device); later
// calls reuse it.  The array is shared: calls that overlap on one device, from
// two streams or two host threads, race on it.

namespace pf {
namespace {

__device__ __align__(256) unsigned char g_uh_static_scratch[PF_UH_STATIC_SCRATCH_BYTES];

constexpr int MAX_DEVICES = 64;
std::mutex g_uh_static_mu;
void* g_uh_static_ptr[MAX_DEVICES];

// This device's address of g_uh_static_scratch (looked up on first use).
int uh_static_scratch(void** out) {
  int dev = 0;
  PF_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= MAX_DEVICES)
    return fail(PF_EDEVICE, "join_unique_hash_static: device %d out of range", dev);
  std::lock_guard<std::mutex> lock(g_uh_static_mu);
  if (!g_uh_static_ptr[dev]) {
    void* p = nullptr;
    const cudaError_t rc = cudaGetSymbolAddress(&p, g_uh_static_scratch);
    if (rc != cudaSuccess || !p)
      return fail(PF_ECUDA, "join_unique_hash_static: cudaGetSymbolAddress: %s",
                  cudaGetErrorString(rc));
    g_uh_static_ptr[dev] = p;
  }
  *out = g_uh_static_ptr[dev];
  return PF_OK;
}

}  // namespace
}  // namespace pf

extern "C" int pf_join_unique_hash_static(const int64_t* build0, const int64_t* build1,
                                          int64_t n_build, const int64_t* probe0,
                                          const int64_t* probe1, int64_t n_probe, int nkeys,
                                          int64_t* build_idx, int64_t* probe_idx,
                                          int64_t* match_count, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (nkeys != 1 && nkeys != 2)
    return fail(PF_EINVAL, "join_unique_hash_static: one or two keys, got %d", nkeys);
  if (n_build < 1 || n_probe < 1)
    return fail(PF_EINVAL, "join_unique_hash_static: unique hash needs rows on both sides");
  if (!build0 || !probe0 || (nkeys == 2 && (!build1 || !probe1)) || !build_idx || !probe_idx ||
      !match_count)
    return fail(PF_EINVAL, "join_unique_hash_static: null pointer");
  // the sizes must fit the fixed scratch (checked before anything is queued)
  if (n_build > PF_JOIN_MAX_ROWS || n_probe > PF_JOIN_MAX_ROWS)
    return fail(PF_EINVAL, "join_unique_hash_static: at most %lld rows a side",
                (long long)PF_JOIN_MAX_ROWS);
  Arena need(nullptr, 0);
  uh_layout(need, n_build, n_probe);
  if (need.used > (size_t)PF_UH_STATIC_SCRATCH_BYTES)
    return fail(PF_EINVAL,
                "join_unique_hash_static: %lld build x %lld probe rows need %zu bytes of "
                "scratch, the static scratch holds %zu (e.g. up to 524288 build with "
                "1048576 probe rows); use pf_join_unique_hash",
                (long long)n_build, (long long)n_probe, need.used,
                (size_t)PF_UH_STATIC_SCRATCH_BYTES);
  void* scratch = nullptr;
  if (int rc = uh_static_scratch(&scratch)) return rc;
  Arena a(scratch, PF_UH_STATIC_SCRATCH_BYTES);
  UhLayout l = uh_layout(a, n_build, n_probe);
  // the table starts empty (all ones) every call; partners, block counts and
  // the total are written in full before they are read
  if (int rc = uh_queue(l, build0, build1, n_build, probe0, probe1, n_probe, nkeys,
                        (long long*)match_count, st))
    return rc;
  if (int rc = uh_emit(l, n_probe, build_idx, probe_idx, st)) return rc;
  return ok();
}
