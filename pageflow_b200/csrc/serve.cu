// Serving: join -> date filter -> group-by requests against resident
// dimension tables, folded into persistent launches.
//
// A dimension table's hash table is built once (pf_dim_build) and stays in
// HBM across requests.  After a 256-byte head it has a compact table
// (compact.cuh) at most a quarter full, or, where the groups' numbers leave an
// entry no room or the keys' hashes crowd it, 16-byte slots {key, OCCUPIED |
// group}, at most half full, linear probing from the key's mix64; the head says
// which.  Probes run in later launches only.
//
// pf_serve_run runs one launch over a list of requests, each a range of its
// probe rows [row_begin, row_end) and, for a request's last launch, its
// finish.  Work items, request by request in the order given:
//   probe items   PROBE_ROWS rows each: keep date in [lo, hi), look the FK up,
//                 add (value, 1) into the block's own sums (agg.cuh) or the
//                 request's (sum, count) slab
//   count items   (finish) GROUP_CHUNK groups each: occupied groups, after
//                 the request's probe items of this launch are done
//   emit items    (finish) the chunk's occupied groups in ascending order at
//                 the chunk's offset, after the count items are done; the
//                 last one writes the group count and sets the request's
//                 pinned done word to 1 + groups (~0 if a wait gave up)
// A block takes the next item from one counter; a finish item waits
// (bounded) for items of its own request that were taken before it by
// blocks that are running, so every wait ends.  The host sees a request
// complete through its done word while the launch goes on with others.
#include <algorithm>
#include <climits>
#include <cstring>
#include <map>

#include "agg.cuh"
#include "compact.cuh"

namespace pf {
namespace {

constexpr int ST = 256;
constexpr int DV = 8;  // dates a lane reads at a time
constexpr long long PROBE_ROWS = 16384;  // at most 65536: a list's offsets are 16 bits
constexpr long long GROUP_CHUNK = 16384;
constexpr long long MAX_CHUNKS = 256;  // groups <= 4M a request
constexpr unsigned WAIT_LIMIT = 1u << 22;
constexpr int MAX_REQUESTS = 8192;  // a launch's requests (their first items sit in smem)
constexpr unsigned long long OCCUPIED = 1ULL << 63;
constexpr unsigned long long NO_GROUP = 0xffffffffULL;

struct DimSlot {
  unsigned long long key;
  unsigned long long val;  // OCCUPIED | group (NO_GROUP: outside [0, n_groups))
};

__device__ __forceinline__ unsigned long long dim_first_slot(uint64_t h, int logcap) {
  return h >> (64 - logcap);
}

// A dimension table's first 256 bytes.
struct DimHead {
  int compact;  // 1: a compact table, 0: 16-byte slots
  int q, gbits, dbits;
  int logcap;   // 16-byte slots, log2
  int crowded;  // the compact table took not every key
  int pad[58];
};
static_assert(sizeof(DimHead) == 256, "the slots start on a 256-byte boundary");

// The table as a lookup takes it.
struct DimTable {
  const unsigned long long* slots;
  int compact, q, gbits, dbits, logcap;
};

__global__ void k_dim_head(DimHead* h, DimHead v) {
  if (threadIdx.x == 0) *h = v;
}

__device__ __forceinline__ bool wide_dim_insert(DimSlot* table, int logcap,
                                                unsigned long long key, unsigned long long v) {
  const unsigned long long mask = (1ULL << logcap) - 1;
  unsigned long long s = dim_first_slot(mix64(key), logcap);
  for (unsigned long long probes = 0; probes <= mask; ++probes) {
    if (atomicCAS(&table[s].val, 0ULL, v) == 0ULL) {
      table[s].key = key;
      return true;
    }
    s = (s + 1) & mask;
  }
  return false;
}

// AGAIN: 16-byte slots, where the compact table (cleared by k_dim_clear) did
// not take every key.
template <bool AGAIN>
__global__ void __launch_bounds__(256) k_dim_build(const long long* __restrict__ keys,
                                                   const int* __restrict__ groups, long long n,
                                                   long long n_groups, DimHead* head,
                                                   unsigned long long* __restrict__ stats) {
  const DimHead h = *head;
  if (AGAIN && !h.crowded) return;
  unsigned long long* slots = reinterpret_cast<unsigned long long*>(head + 1);
  const CompactTable t{slots, h.q, h.gbits, h.dbits};
  unsigned long long bad = 0, overflow = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const long long key = keys[i];
    const int g = groups[i];
    const bool in = g >= 0 && (long long)g < n_groups;
    if (!AGAIN) bad += !in;
    if (!AGAIN && h.compact) {
      if (!ct_insert(t, key, in ? g : -1)) head->crowded = 1;
    } else {
      overflow += !wide_dim_insert(reinterpret_cast<DimSlot*>(slots), h.logcap,
                                   (unsigned long long)key,
                                   OCCUPIED | (in ? (unsigned long long)(unsigned)g : NO_GROUP));
    }
  }
  if (bad) atomicAdd(&stats[0], bad);
  if (overflow) atomicAdd(&stats[1], overflow);
}

__global__ void __launch_bounds__(256) k_dim_clear(DimHead* head) {
  if (!head->crowded) return;
  const unsigned long long words = 2ULL << head->logcap;
  unsigned long long* slots = reinterpret_cast<unsigned long long*>(head + 1);
  for (unsigned long long i = (unsigned long long)blockIdx.x * 256 + threadIdx.x; i < words;
       i += (unsigned long long)gridDim.x * 256)
    slots[i] = 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) head->compact = 0;
}

struct SReq {
  const long long* fk;
  const int* date;
  const long long* value;
  long long r0, r1;
  const DimHead* table;
  long long ng;
  unsigned long long* slab;
  long long* okeys;
  long long* osums;
  long long* ocounts;
  long long* on;
  unsigned long long* done;  // device alias of the pinned done word, or null
  long long item0, npi, nch;  // first item; probe items; finish chunks (0: no finish)
  int lo, hi;
};

struct SCounters {
  unsigned probe_left, count_left, emit_left, pad;
};

struct SHead {
  unsigned long long counter;
  long long n_items;
  int n_req;
  int pad;
  unsigned long long error;
};

// The request of item `it`: the last request whose first item is <= it
// (first[] holds every request's first item, in shared memory).
__device__ __forceinline__ int request_of(const int* first, int n, long long it) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (first[mid] <= it) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ void set_done(unsigned long long* done, unsigned long long v) {
  asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(done), "l"(v) : "memory");
}

// Thread 0 waits (bounded) until *left is zero; false when it gave up, after
// raising the error word and marking the request's done word failed (~0).
__device__ bool wait_zero(const unsigned* left, SHead* h, unsigned long long* done) {
  unsigned polls = 0;
  while (ld_acquire_u32(left) != 0 && polls < WAIT_LIMIT) {
    __nanosleep(200);
    ++polls;
  }
  if (polls >= WAIT_LIMIT) {
    atomicOr(&h->error, 1ULL);
    if (done) set_done(done, ~0ULL);
    return false;
  }
  __threadfence();
  return true;
}

__device__ __forceinline__ long long block_sum(long long v, long long* red) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  long long t = 0;
  for (int q = 0; q < ST / 32; ++q) t += red[q];
  return t;
}

// A key's group in the dimension table: -2 not there, -1 there without a group.
__device__ __forceinline__ long long dim_lookup(const DimTable& t, unsigned long long key) {
  if (t.compact) {
    const CompactTable c{const_cast<unsigned long long*>(t.slots), t.q, t.gbits, t.dbits};
    bool more;
    const unsigned long long hash = ct_hash((long long)key), want = ct_want(c, hash);
    unsigned long long e = ct_among(c, ct_load(ct_home(c, hash)), want, &more);
    if (more) e = ct_walk(c, hash, want);
    return e == CT_EMPTY ? -2 : ct_group(c, e);
  }
  const unsigned long long mask = (1ULL << t.logcap) - 1;
  unsigned long long s = dim_first_slot(mix64(key), t.logcap);
  for (unsigned long long probes = 0; probes <= mask; ++probes) {
    const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(t.slots + 2 * s);
    if (x.y == 0) return -2;
    if (x.x == key) {
      const unsigned long long go = x.y & ~OCCUPIED;
      return go == NO_GROUP ? -1 : (long long)go;
    }
    s = (s + 1) & mask;
  }
  return -2;
}

// Probe rows [lo, hi) of a request.  A warp reads its dates, DV a lane and the
// next step's while this one runs, and keeps the offsets of the rows that pass
// in its own list: a quarter of them pass, and warps that look up and add with
// a quarter of their lanes were the whole time (487M rows: 4350 us, so 3200, and 2850
// once its adds no longer fetched what they replaced).
// It takes 32 off the list's end while that has them (at the item's end, and
// where the block has yet to see the request's groups, whatever is there):
// key and value, then the home sector, then the sums.  (Three takes in flight
// at a time, or two rows a lane: no faster.)
__device__ __forceinline__ void serve_rows(const SReq& R, const DimTable& t, Own& own,
                                           unsigned short* list, long long lo, long long hi,
                                           unsigned& kept, unsigned& matched) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1;
  const int rows = (int)(hi - lo);
  const int steps = (rows + ST * DV - 1) / (ST * DV);
  const int* date = R.date + lo;
  const long long* fk = R.fk + lo;
  const long long* val = R.value + lo;
  unsigned long long* slab = R.slab;
  __builtin_assume(__isGlobal(date));
  __builtin_assume(__isGlobal(fk));
  __builtin_assume(__isGlobal(val));
  __builtin_assume(__isGlobal(t.slots));
  const int dlo = R.lo, dhi = R.hi;
  int n = 0;
  int dt[DV];
  int at = warp * 32 * DV + lane;
#pragma unroll
  for (int k = 0; k < DV; ++k) dt[k] = at + 32 * k < rows ? __ldcs(date + at + 32 * k) : INT_MIN;
  for (int s = 0; s < steps; ++s) {
#pragma unroll
    for (int k = 0; k < DV; ++k) {
      const bool keep = at + 32 * k < rows && dt[k] >= dlo && dt[k] < dhi;
      const unsigned m = __ballot_sync(FULL, keep);
      if (keep) list[n + __popc(m & below)] = (unsigned short)(at + 32 * k);
      n += __popc(m);
      kept += keep;
    }
    at += ST * DV;
#pragma unroll
    for (int k = 0; k < DV; ++k)
      dt[k] = at + 32 * k < rows ? __ldcs(date + at + 32 * k) : INT_MIN;
    __syncwarp();
    const int least = s == steps - 1 || (s == 0 && own.look) ? 1 : 32;
    while (n >= least) {
      const int take = min(n, 32);
      n -= take;
      if (lane < take) {
        const int i = list[n + lane];
        const unsigned long long key = (unsigned long long)__ldcs(fk + i);
        const long long value = __ldcs(val + i);
        const long long g = dim_lookup(t, key);
        matched += g >= -1;
        if (g >= 0 && !own.add((unsigned)g, value, s == 0)) {
          red_add(&slab[2 * (unsigned long long)g], (unsigned long long)value);
          red_add(&slab[2 * (unsigned long long)g + 1], 1ULL);
        }
      }
      __syncwarp();
    }
    if (s == 0) own.after_first();
  }
  own.flush(slab);
}

__global__ void __launch_bounds__(ST, 4) k_serve(SHead* h,
                                                 const SReq* __restrict__ reqs,
                                                 SCounters* cnt, long long* chunk_counts,
                                                 unsigned long long* stats) {
  extern __shared__ __align__(16) unsigned char serve_smem[];
  OwnSums& S = *reinterpret_cast<OwnSums*>(serve_smem);
  int* first_item = reinterpret_cast<int*>(serve_smem + sizeof(OwnSums));
  __shared__ unsigned short lists[ST / 32][32 * (DV + 1)];
  own_init(S);
  __shared__ long long item_s;
  __shared__ int ok_s;
  __shared__ long long red[ST / 32];
  __shared__ int wpre[ST / 32];
  const long long ni = h->n_items;
  const int n = h->n_req;
  for (int i = threadIdx.x; i < n; i += ST) first_item[i] = (int)reqs[i].item0;
  unsigned long long matched = 0, kept = 0;
  // Items are taken in increasing order and an item waits only for items
  // before it, so the smallest unfinished item is always some block's
  // current item with nothing left to wait for: the launch progresses.
  if (threadIdx.x == 0) item_s = (long long)atomicAdd(&h->counter, 1ULL);
  while (true) {
    __syncthreads();
    const long long it = item_s;
    if (it >= ni) break;
    const int q = request_of(first_item, n, it);
    const SReq& R = reqs[q];
    const long long local = it - R.item0;
    if (local < R.npi) {
      // ---- probe rows
      const long long lo = R.r0 + local * PROBE_ROWS, hi = min(R.r1, lo + PROBE_ROWS);
      const DimTable t{reinterpret_cast<const unsigned long long*>(R.table + 1),
                       R.table->compact, R.table->q, R.table->gbits, R.table->dbits,
                       R.table->logcap};
      unsigned kp = 0, ma = 0;
      Own own(S);
      own.begin(q, R.ng);
      serve_rows(R, t, own, lists[threadIdx.x >> 5], lo, hi, kp, ma);
      kept += kp;
      matched += ma;
      __syncthreads();
      if (threadIdx.x == 0) {
        __threadfence();
        atomicSub(&cnt[q].probe_left, 1u);
      }
    } else if (local < R.npi + R.nch) {
      // ---- count a chunk's occupied groups
      const long long c = local - R.npi;
      if (threadIdx.x == 0) ok_s = wait_zero(&cnt[q].probe_left, h, R.done);
      __syncthreads();
      if (!ok_s) {
        if (threadIdx.x == 0) item_s = (long long)atomicAdd(&h->counter, 1ULL);
        continue;
      }
      const long long g0 = c * GROUP_CHUNK, g1 = min(R.ng, g0 + GROUP_CHUNK);
      long long occ = 0;
      for (long long g = g0 + threadIdx.x; g < g1; g += ST) occ += __ldcg(&R.slab[2 * g + 1]) != 0;
      occ = block_sum(occ, red);
      if (threadIdx.x == 0) {
        chunk_counts[(long long)q * MAX_CHUNKS + c] = occ;
        __threadfence();
        atomicSub(&cnt[q].count_left, 1u);
      }
    } else {
      // ---- emit a chunk's occupied groups, ascending
      const long long c = local - R.npi - R.nch;
      if (threadIdx.x == 0) ok_s = wait_zero(&cnt[q].count_left, h, R.done);
      __syncthreads();
      if (!ok_s) {
        if (threadIdx.x == 0) item_s = (long long)atomicAdd(&h->counter, 1ULL);
        continue;
      }
      const long long* cc = chunk_counts + (long long)q * MAX_CHUNKS;
      long long base = 0, total = 0;
      for (long long k = 0; k < R.nch; ++k) {
        const long long v = __ldcg(&cc[k]);
        if (k < c) base += v;
        total += v;
      }
      const long long g0 = c * GROUP_CHUNK, g1 = min(R.ng, g0 + GROUP_CHUNK);
      const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
      for (long long t0 = g0; t0 < g1; t0 += ST) {
        const long long g = t0 + threadIdx.x;
        unsigned long long s = 0, k = 0;
        if (g < g1) {
          s = __ldcg(&R.slab[2 * g]);
          k = __ldcg(&R.slab[2 * g + 1]);
        }
        const bool occ = k != 0;
        const unsigned bal = __ballot_sync(FULL, occ);
        __syncthreads();
        if (lane == 0) wpre[w] = __popc(bal);
        __syncthreads();
        int before = 0, tile = 0;
        for (int qw = 0; qw < ST / 32; ++qw) {
          if (qw < w) before += wpre[qw];
          tile += wpre[qw];
        }
        if (occ) {
          const long long o = base + before + __popc(bal & ((1u << lane) - 1));
          R.okeys[o] = g;
          R.osums[o] = (long long)s;
          R.ocounts[o] = (long long)k;
        }
        base += tile;
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        __threadfence_system();  // the outputs may be host memory
        if (atomicSub(&cnt[q].emit_left, 1u) == 1u) {
          *R.on = total;
          __threadfence_system();
          if (R.done) set_done(R.done, (unsigned long long)(total + 1));
        }
      }
    }
    __syncthreads();  // every thread has read item_s
    if (threadIdx.x == 0) item_s = (long long)atomicAdd(&h->counter, 1ULL);
  }
  for (int o = 16; o; o >>= 1) {
    matched += __shfl_xor_sync(FULL, matched, o);
    kept += __shfl_xor_sync(FULL, kept, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (matched) atomicAdd(&stats[0], matched);
    if (kept) atomicAdd(&stats[2], kept);
  }
}

__global__ void k_serve_error(const SHead* h, unsigned long long* stats) {
  if (threadIdx.x == 0 && h->error) stats[1] |= h->error;
}

// Slabs to be cleared in one launch: 32 of them in 2 us.  A launch each, and an
// array view for each pointer, kept a burst's first rows waiting for 2.5 ms.
constexpr int CLEAR_SLABS = 128;
struct ClearList {
  ulonglong2* slab[CLEAR_SLABS];
  long long ng[CLEAR_SLABS];
};

__global__ void __launch_bounds__(256) k_serve_clear(const __grid_constant__ ClearList c) {
  ulonglong2* slab = c.slab[blockIdx.y];
  const long long ng = c.ng[blockIdx.y];
  for (long long g = (long long)blockIdx.x * 256 + threadIdx.x; g < ng; g += 256LL * gridDim.x)
    slab[g] = make_ulonglong2(0, 0);
}

struct ServeLayout {
  SHead* head;
  SReq* reqs;
  SCounters* cnt;
  long long* chunks;
};

ServeLayout serve_layout(Arena& a, int n) {
  ServeLayout l{};
  l.head = a.take<SHead>(1);
  l.reqs = a.take<SReq>(std::max(n, 1));
  l.cnt = a.take<SCounters>(std::max(n, 1));
  l.chunks = a.take<long long>((size_t)std::max(n, 1) * MAX_CHUNKS);
  return l;
}

// The host image of a launch's header, requests and counters is written into
// pinned staging (one per device and host thread) and copied in one piece;
// the staging is reused once the previous copy out of it has completed.
struct Staging {
  char* buf = nullptr;
  size_t cap = 0;
  cudaEvent_t ev = nullptr;
  bool pending = false;
};

int staging_for(size_t bytes, Staging** out) {
  int dev = 0;
  PF_CUDA(cudaGetDevice(&dev));
  thread_local std::map<int, Staging> stages;
  Staging& s = stages[dev];
  if (!s.ev) PF_CUDA(cudaEventCreateWithFlags(&s.ev, cudaEventDisableTiming));
  if (s.pending) {
    if (int rc = wait_event(s.ev)) return rc;
    s.pending = false;
  }
  if (s.cap < bytes) {
    if (s.buf) PF_CUDA(cudaFreeHost(s.buf));
    s.buf = nullptr;
    s.cap = 0;
    const size_t want = std::max<size_t>(bytes * 2, 1 << 16);
    PF_CUDA(cudaHostAlloc((void**)&s.buf, want, cudaHostAllocDefault));
    s.cap = want;
  }
  *out = &s;
  return PF_OK;
}

int serve_grid(int* grid, size_t smem) {
  int per_sm = 0;
  if (int rc = opt_in_smem((const void*)k_serve, smem)) return rc;
  PF_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_serve, ST, smem));
  *grid = std::max(1, per_sm) * sm_count();
  return PF_OK;
}

}  // namespace
}  // namespace pf

using namespace pf;

namespace {
// 16-byte slots of a table, log2: at least twice the keys, and 256 (64 buckets).
int dim_logcap(int64_t n_keys) {
  return std::max(8, log2_exact(pow2_at_least((uint64_t)std::max<int64_t>(2 * n_keys, 2))));
}
}  // namespace

extern "C" size_t pf_dim_table_bytes(int64_t n_keys) {
  return sizeof(DimHead) + (sizeof(DimSlot) << dim_logcap(n_keys));
}

extern "C" int pf_dim_build(const int64_t* keys, const int32_t* groups, int64_t n_keys,
                            int64_t n_groups, void* table, size_t table_bytes, int64_t* stats,
                            void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (n_keys < 1 || n_groups < 1 || n_groups >= (int64_t)NO_GROUP)
    return fail(PF_EINVAL, "dim_build: bad sizes");
  if (!keys || !groups || !table || !stats) return fail(PF_EINVAL, "dim_build: null pointer");
  const size_t need = pf_dim_table_bytes(n_keys);
  if (table_bytes < need)
    return fail(PF_ENOSPACE, "dim_build: table of %zu bytes, %zu needed", table_bytes, need);
  // the same bytes as a compact table: four entries for two slots
  DimHead hd{};
  hd.logcap = dim_logcap(n_keys);
  hd.q = hd.logcap - 1;
  hd.gbits = bits_of((unsigned long long)n_groups + 1);
  // its loads are 32 bytes
  hd.compact = hd.gbits < 32 && hd.q - hd.gbits >= 3 && ((uintptr_t)table & 31) == 0;
  hd.dbits = hd.compact ? std::min(6, hd.q - hd.gbits) : 0;
  DimHead* head = (DimHead*)table;
  PF_CUDA(cudaMemsetAsync(table, 0, need, st));
  PF_CUDA(cudaMemsetAsync(stats, 0, 2 * sizeof(int64_t), st));
  {
    PF_KERNEL("k_dim_head", st);
    k_dim_head<<<1, 32, 0, st>>>(head, hd);
  }
  PF_LAUNCH("k_dim_head");
  const unsigned grid = (unsigned)std::max<long long>(
      1, std::min<long long>((n_keys + 255) / 256, (long long)sm_count() * 16));
  {
    PF_KERNEL("k_dim_build", st);
    k_dim_build<false><<<grid, 256, 0, st>>>((const long long*)keys, groups, n_keys, n_groups,
                                             head, (unsigned long long*)stats);
  }
  PF_LAUNCH("k_dim_build");
  if (hd.compact) {
    {
      PF_KERNEL("k_dim_clear", st);
      k_dim_clear<<<sm_count() * 4, 256, 0, st>>>(head);
    }
    PF_LAUNCH("k_dim_clear");
    PF_KERNEL("k_dim_build", st);
    k_dim_build<true><<<grid, 256, 0, st>>>((const long long*)keys, groups, n_keys, n_groups,
                                            head, (unsigned long long*)stats);
  }
  PF_LAUNCH("k_dim_build");
  return ok();
}

extern "C" size_t pf_serve_workspace(int max_requests) {
  Arena a(nullptr, 0);
  serve_layout(a, max_requests);
  return a.used + 256;
}

extern "C" int pf_serve_clear(int64_t* const* slabs, const int64_t* n_groups, int n,
                              void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (n < 1 || !slabs || !n_groups) return fail(PF_EINVAL, "serve_clear: bad arguments");
  for (int i = 0; i < n; ++i)
    if (!slabs[i] || ((uintptr_t)slabs[i] & 15) || n_groups[i] < 1)
      return fail(PF_EINVAL, "serve_clear: slab %d: null, not on 16 bytes or empty", i);
  for (int i0 = 0; i0 < n; i0 += CLEAR_SLABS) {
    ClearList c{};
    const int m = std::min(n - i0, CLEAR_SLABS);
    long long most = 0;
    for (int i = 0; i < m; ++i) {
      c.slab[i] = (ulonglong2*)slabs[i0 + i];
      c.ng[i] = n_groups[i0 + i];
      most = std::max(most, c.ng[i]);
    }
    const unsigned gx = (unsigned)std::min<long long>((most + 1023) / 1024, sm_count());
    {
      PF_KERNEL("k_serve_clear", st);
      k_serve_clear<<<dim3(gx, m), 256, 0, st>>>(c);
    }
    PF_LAUNCH("k_serve_clear");
  }
  return ok();
}

extern "C" int pf_serve_run(const pf_serve_request* reqs, int n, void* workspace,
                            size_t workspace_bytes, int64_t* stats, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (n < 1 || n > MAX_REQUESTS)
    return fail(PF_EINVAL, "serve_run: 1 to %d requests a launch, got %d", MAX_REQUESTS, n);
  if (!stats) return fail(PF_EINVAL, "serve_run: null stats");
  Arena a(workspace, workspace_bytes);
  ServeLayout l = serve_layout(a, n);
  if (!workspace || !a.fits())
    return fail(PF_ENOSPACE, "serve_run: workspace of %zu bytes, %zu needed", workspace_bytes,
                a.used);
  // one host image of header, requests and counters, copied in one piece
  const size_t off_r = (char*)l.reqs - (char*)l.head, off_c = (char*)l.cnt - (char*)l.head;
  const size_t bytes = off_c + sizeof(SCounters) * n;
  Staging* stg = nullptr;
  if (int rc = staging_for(bytes, &stg)) return rc;
  char* img = stg->buf;
  std::memset(img, 0, bytes);
  SHead* H = (SHead*)img;
  SReq* D = (SReq*)(img + off_r);
  SCounters* C = (SCounters*)(img + off_c);
  long long items = 0;
  for (int i = 0; i < n; ++i) {
    const pf_serve_request& x = reqs[i];
    if (!x.table || x.n_keys < 1 || x.n_groups < 1 || x.n_groups > GROUP_CHUNK * MAX_CHUNKS)
      return fail(PF_EINVAL, "serve_run: request %d: bad table or groups (at most %lld)", i,
                  (long long)(GROUP_CHUNK * MAX_CHUNKS));
    if (x.row_begin < 0 || x.row_end < x.row_begin)
      return fail(PF_EINVAL, "serve_run: request %d: bad row range", i);
    if (x.row_end > x.row_begin && (!x.fk || !x.date || !x.value))
      return fail(PF_EINVAL, "serve_run: request %d: null column", i);
    if (!x.slab || (x.finish && (!x.out_keys || !x.out_sums || !x.out_counts || !x.out_n)))
      return fail(PF_EINVAL, "serve_run: request %d: null output", i);
    SReq& R = D[i];
    R.fk = (const long long*)x.fk;
    R.date = x.date;
    R.value = (const long long*)x.value;
    R.r0 = x.row_begin;
    R.r1 = x.row_end;
    R.table = (const DimHead*)x.table;
    R.ng = x.n_groups;
    R.slab = (unsigned long long*)x.slab;
    R.okeys = (long long*)x.out_keys;
    R.osums = (long long*)x.out_sums;
    R.ocounts = (long long*)x.out_counts;
    R.on = (long long*)x.out_n;
    R.done = nullptr;
    if (x.finish && x.done) {
      if (int rc = host_alias((void*)x.done, (void**)&R.done)) return rc;
    }
    R.lo = x.date_lo;
    R.hi = x.date_hi;
    if (items > INT_MAX / 2) return fail(PF_EINVAL, "serve_run: too many work items");
    R.item0 = items;
    R.npi = (x.row_end - x.row_begin + PROBE_ROWS - 1) / PROBE_ROWS;
    R.nch = x.finish ? (x.n_groups + GROUP_CHUNK - 1) / GROUP_CHUNK : 0;
    items += R.npi + 2 * R.nch;
    C[i].probe_left = (unsigned)R.npi;
    C[i].count_left = (unsigned)R.nch;
    C[i].emit_left = (unsigned)R.nch;
  }
  H->counter = 0;
  H->n_items = items;
  H->n_req = n;
  H->error = 0;
  int grid = 0;
  if (int rc = serve_grid(&grid, sizeof(OwnSums) + sizeof(int) * n)) return rc;
  PF_CUDA(cudaMemcpyAsync(l.head, img, bytes, cudaMemcpyHostToDevice, st));
  PF_CUDA(cudaEventRecord(stg->ev, st));
  stg->pending = true;
  {
    PF_KERNEL("k_serve", st);
    k_serve<<<grid, ST, sizeof(OwnSums) + sizeof(int) * n, st>>>(l.head, l.reqs, l.cnt, l.chunks,
                                                (unsigned long long*)stats);
  }
  PF_LAUNCH("k_serve");
  {
    PF_KERNEL("k_serve_error", st);
    k_serve_error<<<1, 32, 0, st>>>(l.head, (unsigned long long*)stats);
  }
  PF_LAUNCH("k_serve_error");
  return ok();
}
