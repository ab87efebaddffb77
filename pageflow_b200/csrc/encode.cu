// Output-side encoding on the device: partitioned columns written as PFC1
// pages (codec.h) without leaving the GPU, so partitioned intermediates can
// be kept or spilled compressed (the reference compresses its partitioned
// outputs region by region through nvCOMP on the way out:
// IO/codec/region_producer.py, IO/codec/batched_compress.py:27-59).
//
// The pages are byte for byte the ones the host encoder (codec.cu) writes for
// the same values: the same four candidate schemes sized the same way, the
// same choice (the smallest; RAW, FOR, DELTA, RLE in that order on a tie),
// the same block tables, bits and padding.
//
// A page is cut into parts of whole mini-blocks (at most EPARTS a page) and a
// warp takes a part, so a column of a few dozen pages still fills the chip
// (one block a page, the earlier split, kept 62 of 148 SMs busy and paid five
// block barriers a mini-block and range: 8M int64 rows took 400 us to plan
// and 190 us to write where their bytes need 15 us):
//
//   k_enc_plan    a warp a part: each mini-block's value and delta range by
//                 one warp reduction, the words its FOR and DELTA streams
//                 take and the run starts in it, summed over the part
//   k_enc_choose  a block a page: the parts' sums; with few enough runs the
//                 runs themselves (each warp knows its parts' first run) and
//                 the RLE sizes; the choice and the page's bytes
//   k_enc_offsets the pages' byte offsets (one block)
//   k_enc_write   a warp a part: FOR, DELTA and RAW pages. A mini-block's
//                 terms are staged in shared memory and each lane gathers
//                 whole output words from them (no atomics, one coalesced
//                 write); the stream position is the sum of the parts before
//   k_enc_rle     a block a page: RLE pages, whose streams are a few
//                 mini-blocks
//
// The caller's one wait is for the offsets, while the pages are written.
// 8M int64 rows in 131072-row pages, B200: plan 400 -> 21 us, write 190 -> 32; three
// columns of 8M rows (20 bytes a row) through the Python call 1850 -> 430 us a pass.
#include <algorithm>
#include <climits>

#include "codec.h"
#include "common.cuh"

namespace pf {
namespace {

constexpr int WT = 256;       // threads of the part kernels: a warp a part
constexpr int ET = 1024;      // threads of the page kernels
constexpr int EPARTS = 128;   // parts a page is cut into, at most
constexpr unsigned E_HOST_PAGES = 4096;  // offsets a thread's pinned buffer holds

struct PageMeta {
  long long bytes;   // the page's size
  int scheme;
  int rle_vs;        // RLE: the runs' values as FOR or DELTA
  int nruns;
  int pad;
};

__device__ __forceinline__ unsigned bit_width64(unsigned long long r) {
  return r ? 64u - (unsigned)__clzll((long long)r) : 0u;
}

// A part's share of its page's plan.
struct PartPlan {
  long long wfor, wdelta;  // words of its mini-blocks as FOR and as DELTA
  long long runs;          // run starts in it
};

struct Range {
  long long lo, hi;
};
__device__ __forceinline__ void range_add(Range& r, long long x) {
  r.lo = min(r.lo, x);
  r.hi = max(r.hi, x);
}
// The warp's range (an empty one is 0 to 0).
__device__ __forceinline__ Range warp_range(Range r) {
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    r.lo = min(r.lo, __shfl_xor_sync(FULL, r.lo, o));
    r.hi = max(r.hi, __shfl_xor_sync(FULL, r.hi, o));
  }
  if (r.lo > r.hi) r.lo = r.hi = 0;
  return r;
}
__device__ __forceinline__ unsigned width_of(const Range& r) {
  return bit_width64((unsigned long long)r.hi - (unsigned long long)r.lo);
}

// The parts of a page of n rows at `parts` parts a page: part w holds
// mini-blocks [w * per, min(nblk, (w + 1) * per)).
__device__ __forceinline__ long long blocks_of(long long n) {
  return (n + PFC_BLOCK - 1) / PFC_BLOCK;
}
__device__ __forceinline__ long long part_blocks(long long n, int parts) {
  return (blocks_of(n) + parts - 1) / parts;
}

__device__ __forceinline__ long long words_of(unsigned bw, int cnt) {
  return ((long long)bw * cnt + 31) / 32;
}

__device__ __forceinline__ long long align16(long long x) { return (x + 15) / 16 * 16; }

// A stream's bytes from its words: header, block table, words and three
// words of padding, to a 16-byte boundary.
__device__ __forceinline__ long long stream_bytes(long long nblk, long long words) {
  return align16(16 + 32 * nblk + 4 * (words + 3));
}

constexpr int EU = 8;  // rows a lane loads before it looks at them

// One warp over a mini-block of cnt values (get(j) its j-th): the range of
// its values, of its differences after the first, and the run starts in it
// (prev: the value before the mini-block, first: there is none).
template <typename Get>
__device__ __forceinline__ void scan_block(int cnt, Get get, long long prev, bool first,
                                           Range& rv, Range& rd, int& runs) {
  const int lane = threadIdx.x & 31;
  rv = rd = Range{LLONG_MAX, LLONG_MIN};
  int starts = 0;
  for (int i0 = 0; i0 < cnt; i0 += 32 * EU) {
    long long v[EU];
#pragma unroll
    for (int u = 0; u < EU; ++u) {
      const int j = i0 + u * 32 + lane;
      v[u] = j < cnt ? get(j) : 0;
    }
#pragma unroll
    for (int u = 0; u < EU; ++u) {
      const int j = i0 + u * 32 + lane;
      long long before = __shfl_up_sync(FULL, v[u], 1);
      if (lane == 0) before = prev;
      prev = __shfl_sync(FULL, v[u], 31);
      if (j < cnt) {
        range_add(rv, v[u]);
        if (j > 0)
          range_add(rd, (long long)((unsigned long long)v[u] - (unsigned long long)before));
        starts += (first && j == 0) || v[u] != before;
      }
    }
  }
  rv = warp_range(rv);
  rd = warp_range(rd);
  runs = __reduce_add_sync(FULL, starts);
}

template <typename V>
__global__ void __launch_bounds__(WT) k_enc_plan(const V* __restrict__ col,
                                                 const long long* __restrict__ rows, int npages,
                                                 int parts, PartPlan* __restrict__ plan) {
  const long long t = ((long long)blockIdx.x * WT + threadIdx.x) >> 5;
  if (t >= (long long)npages * parts) return;
  const int p = (int)(t / parts), w = (int)(t - (long long)p * parts);
  const long long p0 = rows[p], n = rows[p + 1] - p0;
  const long long per = part_blocks(n, parts), k1 = min(blocks_of(n), (w + 1) * per);
  const V* v = col + p0;
  PartPlan s{0, 0, 0};
  for (long long k = w * per; k < k1; ++k) {
    const long long b0 = k * PFC_BLOCK;
    const int cnt = (int)min((long long)PFC_BLOCK, n - b0);
    Range rv, rd;
    int runs;
    scan_block(cnt, [&](int j) { return (long long)v[b0 + j]; },
               b0 > 0 ? (long long)v[b0 - 1] : 0, b0 == 0, rv, rd, runs);
    s.wfor += words_of(width_of(rv), cnt);
    s.wdelta += words_of(width_of(rd), cnt);
    s.runs += runs;
  }
  if ((threadIdx.x & 31) == 0) plan[t] = s;
}

// A page's runs: their values and exclusive ends.
struct Runs {
  long long rv[PFC_RLE_MAX_RUNS];
  long long re[PFC_RLE_MAX_RUNS];
  long long first[EPARTS + 1];  // each part's first run, then the runs of the page
  long long words[3][PFC_RLE_MAX_RUNS / PFC_BLOCK];
  unsigned stage[2 * PFC_BLOCK];  // a mini-block's words
  Range range;
  int cnt;
};

// The run values and ends of a page of at most PFC_RLE_MAX_RUNS runs (R.first
// filled): each warp walks its parts and writes the starts it meets.
template <typename V>
__device__ void page_runs(const V* __restrict__ v, long long n, int parts, Runs& R) {
  // 4 bytes a row: 16 rows a lane in flight (a page's block is one SM's, and
  // waits on these loads), 8-byte rows 8
  constexpr int RU = 64 / (int)sizeof(V);
  const int lane = threadIdx.x & 31;
  const long long per = part_blocks(n, parts) * PFC_BLOCK;
  for (int w = threadIdx.x >> 5; w < parts; w += ET / 32) {
    const long long j0 = w * per, j1 = min(n, j0 + per);
    if (j0 >= n) break;
    long long r = R.first[w];
    if (R.first[w + 1] == r) continue;  // no run starts in it
    V prev = j0 > 0 ? v[j0 - 1] : (V)0;
    for (long long i0 = j0; i0 < j1; i0 += 32 * RU) {
      V x[RU];
#pragma unroll
      for (int u = 0; u < RU; ++u) {
        const long long j = i0 + u * 32 + lane;
        x[u] = j < j1 ? v[j] : (V)0;
      }
#pragma unroll
      for (int u = 0; u < RU; ++u) {
        const long long j = i0 + u * 32 + lane;
        V before = __shfl_up_sync(FULL, x[u], 1);
        if (lane == 0) before = prev;
        prev = __shfl_sync(FULL, x[u], 31);
        const bool start = j < j1 && (j == 0 || x[u] != before);
        const unsigned m = __ballot_sync(FULL, start);
        if (start) {
          const long long at = r + __popc(m & lanemask_lt());
          R.rv[at] = x[u];
          if (at > 0) R.re[at - 1] = j;
        }
        r += __popc(m);
      }
    }
  }
  if (threadIdx.x == 0 && n > 0) R.re[R.first[parts] - 1] = n;
  __syncthreads();
}

// The parts' first runs (one warp; parts <= EPARTS) and the sums of both
// word counts, into R.first and *wfor, *wdelta (lane 0 holds them).
__device__ __forceinline__ void part_sums(const PartPlan* __restrict__ plan, int parts, Runs& R,
                                          long long* wfor, long long* wdelta) {
  const int lane = threadIdx.x & 31;
  long long run = 0, a = 0, b = 0;
  for (int w0 = 0; w0 < parts; w0 += 32) {
    const bool in = w0 + lane < parts;
    const PartPlan x = in ? plan[w0 + lane] : PartPlan{0, 0, 0};
    long long incl = x.runs;
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += y;
    }
    if (in) R.first[w0 + lane] = run + incl - x.runs;
    run += __shfl_sync(FULL, incl, 31);
    a += x.wfor;
    b += x.wdelta;
  }
  for (int o = 16; o; o >>= 1) {
    a += __shfl_xor_sync(FULL, a, o);
    b += __shfl_xor_sync(FULL, b, o);
  }
  if (lane == 0) R.first[parts] = run;
  *wfor = a;
  *wdelta = b;
}

template <typename V>
__global__ void __launch_bounds__(ET) k_enc_choose(const V* __restrict__ col,
                                                   const long long* __restrict__ rows, int parts,
                                                   const PartPlan* __restrict__ plan,
                                                   PageMeta* __restrict__ meta) {
  extern __shared__ __align__(16) unsigned char enc_smem[];
  Runs& R = *reinterpret_cast<Runs*>(enc_smem);
  const int p = blockIdx.x, esize = (int)sizeof(V);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long p0 = rows[p], n = rows[p + 1] - p0;
  long long wfor = 0, wdelta = 0;
  if (w == 0) part_sums(plan + (long long)p * parts, parts, R, &wfor, &wdelta);
  __syncthreads();
  const long long nr = R.first[parts];
  const bool rle = n > 0 && nr <= PFC_RLE_MAX_RUNS;
  const int nrb = rle ? (int)blocks_of(nr) : 0;
  if (rle) {
    page_runs(col + p0, n, parts, R);
    // a warp a mini-block of the run values and one of the run ends
    for (int t = w; t < 2 * nrb; t += ET / 32) {
      const int k = t >> 1;
      const int cnt = (int)min((long long)PFC_BLOCK, nr - (long long)k * PFC_BLOCK);
      const long long* src = ((t & 1) ? R.re : R.rv) + k * PFC_BLOCK;
      Range rv, rd;
      int runs;
      scan_block(cnt, [&](int j) { return src[j]; }, 0, true, rv, rd, runs);
      if (lane == 0) {
        if (t & 1) {
          R.words[2][k] = words_of(width_of(rd), cnt);
        } else {
          R.words[0][k] = words_of(width_of(rv), cnt);
          R.words[1][k] = words_of(width_of(rd), cnt);
        }
      }
    }
    __syncthreads();
  }
  if (threadIdx.x != 0) return;
  const long long raw = (long long)esize * n + 16;
  const long long s_for = stream_bytes(blocks_of(n), wfor);
  const long long s_delta = stream_bytes(blocks_of(n), wdelta);
  long long s_rle = LLONG_MAX;
  int rle_vs = PFC_FOR;
  if (rle) {
    long long a = 0, b = 0, e = 0;
    for (int k = 0; k < nrb; ++k) {
      a += R.words[0][k];
      b += R.words[1][k];
      e += R.words[2][k];
    }
    a = stream_bytes(nrb, a);
    b = stream_bytes(nrb, b);
    rle_vs = b < a ? PFC_DELTA : PFC_FOR;
    s_rle = min(a, b) + stream_bytes(nrb, e);
  }
  int scheme = PFC_RAW;
  long long best = raw;
  if (s_for < best) { best = s_for; scheme = PFC_FOR; }
  if (s_delta < best) { best = s_delta; scheme = PFC_DELTA; }
  if (s_rle < best) { best = s_rle; scheme = PFC_RLE; }
  // the page: 64-byte header, then the chosen streams
  long long bytes = 64;
  if (scheme == PFC_RAW) bytes += align16((long long)esize * n);
  else if (scheme == PFC_RLE) bytes = align16(bytes + s_rle);
  else bytes += best;
  meta[p] = PageMeta{align16(bytes), scheme, rle_vs, (int)min(nr, (long long)INT_MAX), 0};
}

// One block: offs[p] = the bytes of the pages before p (offs[npages] all of
// them), to the host's buffer too when it has one.
__global__ void __launch_bounds__(ET) k_enc_offsets(const PageMeta* __restrict__ meta, int npages,
                                                    long long* __restrict__ offs,
                                                    long long* host) {
  __shared__ long long wsum[32];
  __shared__ long long base;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x == 0) base = 0;
  __syncthreads();
  for (int q = 0; q <= npages; q += ET) {
    const int p = q + threadIdx.x;
    const long long x = p < npages ? meta[p].bytes : 0;
    long long incl = x;
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    long long pre = base, tot = 0;
    for (int i = 0; i < 32; ++i) {
      pre += i < w ? wsum[i] : 0;
      tot += wsum[i];
    }
    if (p <= npages) {
      offs[p] = pre + incl - x;
      if (host) host[p] = pre + incl - x;
    }
    __syncthreads();
    if (threadIdx.x == 0) base += tot;
    __syncthreads();
  }
}

// Word w of a mini-block's packed bits: the terms whose bw-bit fields meet
// bits [32w, 32w + 32), gathered from the staged differences to the minimum.
template <typename D>
__device__ __forceinline__ unsigned gather_word(const D* d, int cnt, unsigned bw, unsigned w) {
  const unsigned bit0 = w * 32;
  unsigned j = bit0 / bw;
  unsigned sh = bit0 - j * bw;           // bits of term j before this word
  unsigned out = (unsigned)((unsigned long long)d[j] >> sh);
  unsigned have = bw - sh;               // bits filled so far
  while (have < 32 && ++j < (unsigned)cnt) {
    out |= (unsigned)((unsigned long long)d[j] << have);
    have += bw;
  }
  return out;
}

__device__ __forceinline__ void write_header(unsigned char* page, const PageMeta& pm, int esize,
                                             long long n, long long s1) {
  PfcPage h;
  unsigned* hw = reinterpret_cast<unsigned*>(&h);
  for (int i = 0; i < (int)(sizeof(PfcPage) / 4); ++i) hw[i] = 0;
  h.magic = PFC_MAGIC;
  h.scheme = (uint8_t)pm.scheme;
  h.esize = (uint8_t)esize;
  h.n = (uint32_t)n;
  h.nruns = pm.scheme == PFC_RLE ? (uint32_t)pm.nruns : 0u;
  h.s0 = 64;
  h.s1 = pm.scheme == PFC_RLE ? (uint32_t)s1 : 0u;
  h.bytes = (uint32_t)pm.bytes;
  *reinterpret_cast<PfcPage*>(page) = h;
}

// One warp writes mini-block k of a stream at `out`: its words from word
// woff of the stream on, and its table entry; returns its words.  stage: the
// warp's 2 * PFC_BLOCK words of shared memory.
template <typename Get>
__device__ __forceinline__ long long write_block(unsigned char* out, long long nblk, long long k,
                                                 int cnt, int scheme, Get get, long long woff,
                                                 unsigned* stage) {
  const int lane = threadIdx.x & 31;
  PfcBlock* table = reinterpret_cast<PfcBlock*>(out + 16);
  unsigned* words = reinterpret_cast<unsigned*>(out + 16 + 32 * nblk) + woff;
  const bool delta = scheme == PFC_DELTA;
  Range r{LLONG_MAX, LLONG_MIN};
  long long prev = 0, first = 0;
  unsigned long long* s64 = reinterpret_cast<unsigned long long*>(stage);
  __syncwarp();
  for (int i0 = 0; i0 < cnt; i0 += 32 * EU) {
    long long v[EU];
#pragma unroll
    for (int u = 0; u < EU; ++u) {
      const int j = i0 + u * 32 + lane;
      v[u] = j < cnt ? get(j) : 0;
    }
    if (i0 == 0) first = __shfl_sync(FULL, v[0], 0);
#pragma unroll
    for (int u = 0; u < EU; ++u) {
      const int j = i0 + u * 32 + lane;
      long long t = v[u];
      if (delta) {
        long long before = __shfl_up_sync(FULL, v[u], 1);
        if (lane == 0) before = prev;
        prev = __shfl_sync(FULL, v[u], 31);
        t = (long long)((unsigned long long)v[u] - (unsigned long long)before);
      }
      if (j < cnt) {
        if (!delta || j > 0) range_add(r, t);
        s64[j] = (unsigned long long)t;
      }
    }
  }
  r = warp_range(r);
  const unsigned bw = width_of(r);
  const long long nw = words_of(bw, cnt);
  // the terms as differences to the minimum (a DELTA block's first is 0), 32
  // bits each when they fit
  __syncwarp();
  if (bw > 32) {
    for (int j = lane; j < cnt; j += 32)
      s64[j] = delta && j == 0 ? 0ULL : s64[j] - (unsigned long long)r.lo;
    __syncwarp();
    for (unsigned w = lane; w < nw; w += 32) words[w] = gather_word(s64, cnt, bw, w);
  } else if (bw) {
    // packed in place, front to back: term j's 4 bytes never pass the 8-byte
    // terms still to be read
    for (int j0 = 0; j0 < cnt; j0 += 32) {
      const int j = j0 + lane;
      const unsigned x = j < cnt ? (unsigned)(s64[j] - (unsigned long long)r.lo) : 0u;
      __syncwarp();
      if (j < cnt) stage[j] = delta && j == 0 ? 0u : x;
      __syncwarp();
    }
    for (unsigned w = lane; w < nw; w += 32) words[w] = gather_word(stage, cnt, bw, w);
  }
  if (lane == 0) {
    PfcBlock b;
    b.base = r.lo;
    b.first = delta ? first : 0;
    b.word_off = (uint32_t)woff;
    b.bw = bw;
    b.pad[0] = b.pad[1] = 0;
    table[k] = b;
  }
  return nw;
}

// A stream's header, and its padding: three zero words, then zeros to the
// 16-byte end (threads t of nt).
__device__ __forceinline__ void write_frame(unsigned char* out, long long n, int scheme,
                                            long long words, int t, int nt) {
  const long long nblk = blocks_of(n);
  if (t == 0) {
    PfcStream sh{(uint32_t)scheme, (uint32_t)n, (uint32_t)nblk, 0};
    *reinterpret_cast<PfcStream*>(out) = sh;
  }
  const long long end = stream_bytes(nblk, words);
  for (long long b = 16 + 32 * nblk + 4 * words + t; b < end; b += nt) out[b] = 0;
}

template <typename V>
__global__ void __launch_bounds__(WT) k_enc_write(const V* __restrict__ col,
                                                  const long long* __restrict__ rows, int npages,
                                                  int parts, const PartPlan* __restrict__ plan,
                                                  const PageMeta* __restrict__ meta,
                                                  const long long* __restrict__ offs,
                                                  long long capacity,
                                                  unsigned char* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char enc_smem[];
  if (offs[npages] > capacity) return;  // the host returns the error
  const long long t = ((long long)blockIdx.x * WT + threadIdx.x) >> 5;
  if (t >= (long long)npages * parts) return;
  const int lane = threadIdx.x & 31;
  const int p = (int)(t / parts), w = (int)(t - (long long)p * parts);
  const PageMeta pm = meta[p];
  if (pm.scheme == PFC_RLE) return;  // k_enc_rle's
  const long long p0 = rows[p], n = rows[p + 1] - p0;
  const long long nblk = blocks_of(n), per = part_blocks(n, parts);
  const long long k0 = w * per, k1 = min(nblk, k0 + per);
  const V* v = col + p0;
  unsigned char* page = out + offs[p];
  if (w == 0 && lane == 0) write_header(page, pm, (int)sizeof(V), n, 0);
  if (pm.scheme == PFC_RAW) {
    V* dst = reinterpret_cast<V*>(page + 64);
    for (long long i = k0 * PFC_BLOCK + lane; i < min(n, k1 * PFC_BLOCK); i += 32) dst[i] = v[i];
    if (w == 0)
      for (long long b = 64 + (long long)sizeof(V) * n + lane; b < pm.bytes; b += 32) page[b] = 0;
    return;
  }
  // the words of the parts before this one, and of the page
  long long before = 0, total = 0;
  for (int q = lane; q < parts; q += 32) {
    const PartPlan& x = plan[(long long)p * parts + q];
    const long long c = pm.scheme == PFC_DELTA ? x.wdelta : x.wfor;
    before += q < w ? c : 0;
    total += c;
  }
  for (int o = 16; o; o >>= 1) {
    before += __shfl_xor_sync(FULL, before, o);
    total += __shfl_xor_sync(FULL, total, o);
  }
  unsigned* stage = reinterpret_cast<unsigned*>(enc_smem) + (threadIdx.x >> 5) * 2 * PFC_BLOCK;
  if (w == 0) write_frame(page + 64, n, pm.scheme, total, lane, 32);
  for (long long k = k0; k < k1; ++k) {
    const long long b0 = k * PFC_BLOCK;
    const int cnt = (int)min((long long)PFC_BLOCK, n - b0);
    before += write_block(page + 64, nblk, k, cnt, pm.scheme,
                          [&](int j) { return (long long)v[b0 + j]; }, before, stage);
  }
}

// One warp writes a whole stream of n values (the runs' of an RLE page) and
// returns its bytes.
__device__ long long write_runs_stream(unsigned char* out, long long n, int scheme,
                                       const long long* src, unsigned* stage) {
  long long woff = 0;
  const long long nblk = blocks_of(n);
  for (long long k = 0; k < nblk; ++k) {
    const int cnt = (int)min((long long)PFC_BLOCK, n - k * PFC_BLOCK);
    const long long* b = src + k * PFC_BLOCK;
    woff += write_block(out, nblk, k, cnt, scheme, [&](int j) { return b[j]; }, woff, stage);
  }
  write_frame(out, n, scheme, woff, threadIdx.x & 31, 32);
  return stream_bytes(nblk, woff);
}

template <typename V>
__global__ void __launch_bounds__(ET) k_enc_rle(const V* __restrict__ col,
                                                const long long* __restrict__ rows, int npages,
                                                int parts, const PartPlan* __restrict__ plan,
                                                const PageMeta* __restrict__ meta,
                                                const long long* __restrict__ offs,
                                                long long capacity,
                                                unsigned char* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char enc_smem[];
  Runs& R = *reinterpret_cast<Runs*>(enc_smem);
  const int p = blockIdx.x;
  const PageMeta pm = meta[p];
  if (pm.scheme != PFC_RLE || offs[npages] > capacity) return;
  const long long p0 = rows[p], n = rows[p + 1] - p0;
  long long wfor, wdelta;
  if (threadIdx.x < 32) part_sums(plan + (long long)p * parts, parts, R, &wfor, &wdelta);
  __syncthreads();
  page_runs(col + p0, n, parts, R);
  if (threadIdx.x >= 32) return;
  unsigned char* page = out + offs[p];
  const long long nr = pm.nruns;
  const long long s1 = 64 + write_runs_stream(page + 64, nr, pm.rle_vs, R.rv, R.stage);
  __syncwarp();
  const long long end = s1 + write_runs_stream(page + s1, nr, PFC_DELTA, R.re, R.stage);
  for (long long b = end + threadIdx.x; b < pm.bytes; b += 32) page[b] = 0;
  if (threadIdx.x == 0) write_header(page, pm, (int)sizeof(V), n, s1);
}

struct EncLayout {
  PageMeta* meta;
  PartPlan* plan;
  long long* rows;
  long long* offs;
};
EncLayout enc_layout(Arena& a, int npages) {
  EncLayout l{};
  l.meta = a.take<PageMeta>((size_t)npages);
  l.plan = a.take<PartPlan>((size_t)npages * EPARTS);
  l.rows = a.take<long long>((size_t)npages + 1);
  l.offs = a.take<long long>((size_t)npages + 1);
  return l;
}


// A thread's pinned words for the offsets of a call (kept; null when there
// is none).
long long* pinned_offsets() {
  thread_local long long* buf = nullptr;
  if (!buf && cudaHostAlloc((void**)&buf, (E_HOST_PAGES + 1) * sizeof(long long),
                            cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
    cudaGetLastError();
    buf = nullptr;
  }
  return buf;
}

template <typename V>
int encode_pages(const void* values, const int64_t* page_rows, int npages, void* out,
                 int64_t capacity, int64_t* page_offsets, const EncLayout& l, cudaStream_t st) {
  const V* col = (const V*)values;
  long long most = 1;
  for (int p = 0; p < npages; ++p)
    most = std::max<long long>(most, (page_rows[p + 1] - page_rows[p] + PFC_BLOCK - 1) / PFC_BLOCK);
  const int parts = (int)std::min<long long>(EPARTS, most);
  // a mini-block of 8-byte terms a warp; the page kernels hold a page's runs
  const size_t wsm = (size_t)(WT / 32) * 2 * PFC_BLOCK * sizeof(unsigned);
  if (int rc = opt_in_smem((const void*)k_enc_choose<V>, sizeof(Runs))) return rc;
  if (int rc = opt_in_smem((const void*)k_enc_rle<V>, sizeof(Runs))) return rc;
  if (int rc = opt_in_smem((const void*)k_enc_write<V>, wsm)) return rc;
  // pageable source: the copy takes the data before it returns
  PF_CUDA(cudaMemcpyAsync(l.rows, page_rows, ((size_t)npages + 1) * sizeof(long long),
                          cudaMemcpyHostToDevice, st));
  const unsigned g = blocks_for((long long)npages * parts, WT / 32);
  {
    PF_KERNEL("k_enc_plan", st);
    k_enc_plan<V><<<g, WT, 0, st>>>(col, l.rows, npages, parts, l.plan);
  }
  PF_LAUNCH("k_enc_plan");
  {
    PF_KERNEL("k_enc_choose", st);
    k_enc_choose<V><<<npages, ET, sizeof(Runs), st>>>(col, l.rows, parts, l.plan, l.meta);
  }
  PF_LAUNCH("k_enc_choose");
  long long* host = npages <= (int)E_HOST_PAGES ? pinned_offsets() : nullptr;
  long long* host_dev = nullptr;
  if (host)
    if (int rc = host_alias(host, (void**)&host_dev)) return rc;
  {
    PF_KERNEL("k_enc_offsets", st);
    k_enc_offsets<<<1, ET, 0, st>>>(l.meta, npages, l.offs, host_dev);
  }
  PF_LAUNCH("k_enc_offsets");
  cudaEvent_t ev;
  if (int rc = record_event(st, &ev)) return rc;
  {
    PF_KERNEL("k_enc_write", st);
    k_enc_write<V><<<g, WT, wsm, st>>>(col, l.rows, npages, parts, l.plan, l.meta, l.offs,
                                       capacity, (unsigned char*)out);
  }
  PF_LAUNCH("k_enc_write");
  {
    PF_KERNEL("k_enc_rle", st);
    k_enc_rle<V><<<npages, ET, sizeof(Runs), st>>>(col, l.rows, npages, parts, l.plan, l.meta,
                                                  l.offs, capacity, (unsigned char*)out);
  }
  PF_LAUNCH("k_enc_rle");
  if (host) {
    if (int rc = wait_event(ev)) return rc;
    for (int p = 0; p <= npages; ++p) page_offsets[p] = host[p];
  } else {
    PF_CUDA(cudaMemcpyAsync(page_offsets, l.offs, ((size_t)npages + 1) * sizeof(long long),
                            cudaMemcpyDeviceToHost, st));
    if (int rc = wait_stream(st)) return rc;
  }
  if (page_offsets[npages] > capacity)
    return fail(PF_ENOSPACE, "encode_pages: %lld bytes of pages, capacity %lld",
                (long long)page_offsets[npages], (long long)capacity);
  return ok();
}

}  // namespace
}  // namespace pf

using namespace pf;

extern "C" size_t pf_encode_pages_workspace(int npages) {
  Arena a(nullptr, 0);
  enc_layout(a, std::max(1, npages));
  return a.used + 256;
}

extern "C" int pf_encode_pages(const void* values, int esize, const int64_t* page_rows,
                               int npages, void* out, int64_t capacity, int64_t* page_offsets,
                               void* workspace, size_t workspace_bytes, void* stream) {
  cudaStream_t st = (cudaStream_t)stream;
  if (esize != 4 && esize != 8) return fail(PF_EINVAL, "encode_pages: esize 4 or 8");
  if (npages < 1 || !page_rows || !page_offsets)
    return fail(PF_EINVAL, "encode_pages: at least one page and its rows");
  for (int p = 0; p < npages; ++p) {
    const long long n = page_rows[p + 1] - page_rows[p];
    if (page_rows[p] < 0 || n < 0 || n > (1LL << 30))
      return fail(PF_EINVAL, "encode_pages: page %d has %lld rows (0 to 2^30)", p, n);
  }
  Arena ar(workspace, workspace_bytes);
  EncLayout l = enc_layout(ar, npages);
  if (!workspace || !ar.fits())
    return fail(PF_ENOSPACE, "encode_pages: workspace of %zu bytes, %zu needed", workspace_bytes,
                ar.used);
  return esize == 8 ? encode_pages<long long>(values, page_rows, npages, out, capacity,
                                              page_offsets, l, st)
                    : encode_pages<int>(values, page_rows, npages, out, capacity, page_offsets, l,
                                        st);
}
