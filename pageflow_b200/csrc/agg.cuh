// Device helpers shared by the persistent kernels (batch.cu, serve.cu): an
// acquire load for their bounded waits, and a block's own (sum, count) cells in
// shared memory.
#pragma once

#include "common.cuh"

namespace pf {

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Where a warp has a group in four lanes or more: the words x of the lanes of the same
// group (every lane of the warp; g < 0: none) added up into the group's first lane; how
// many they are, 0 in the others.  Else each lane's own.
__device__ __forceinline__ unsigned warp_group_sum(int g, unsigned long long& x) {
  const int lane = threadIdx.x & 31;
  const unsigned all = __match_any_sync(FULL, g);
  if (!__any_sync(FULL, g >= 0 && __popc(all) >= 4)) return g >= 0;
  unsigned rank = __popc(all & lanemask_lt()), above = g < 0 ? 0u : all & ~1u << lane;
  const unsigned n = g < 0 || rank ? 0u : (unsigned)__popc(all);
  while (__any_sync(FULL, above)) {
    const unsigned long long y = __shfl_sync(FULL, x, above ? __ffs(above) - 1 : lane);
    if (above) x += y;
    above &= __ballot_sync(FULL, (rank & 1) == 0);  // every other one has been taken
    rank >>= 1;
  }
  return n;
}

// The block's own sums: lo, hi and count of OWN_CELLS cells.  A source of few
// groups has all of them there, as many copies of each as fit, a lane its own
// (a warp's lanes then meet on no address).  Else, where the source's first
// rows show groups again, its hot groups: one is let in when it comes again
// before another group of its `seen` entry (so one row in about a thousand or
// more; a group that frequent would queue up on its address in L2, which takes
// a RED every 14 clocks, while groups met once an item would fill the cells),
// OWN_COPIES copies of each.  The cells are flushed into the (sum, count) slab
// at an item's end; the hot groups' places stay for the block's next item of
// the same source.  (48 batch instances: 512 groups of 2 copies 5.6 ms, 256 of 4 5.8,
// and twice the time with 54 KB of cells, whose blocks leave no L1.  Serving:
// 2048 cells no faster, 4096 a tenth slower.)
constexpr int OWN_CELLS = 1024;
constexpr int OWN_SMALL = 512;
constexpr int OWN_HOT_LOG = 9, OWN_HOT = 1 << OWN_HOT_LOG, OWN_COPIES = 2;
constexpr int OWN_SEEN_LOG = 10;
constexpr int OWN_REPEATS = 16;  // of a source's first rows in a block, groups met again
static_assert(OWN_HOT * OWN_COPIES <= OWN_CELLS && OWN_SMALL <= OWN_CELLS, "cells");

struct OwnSums {
  unsigned lo[OWN_CELLS], hi[OWN_CELLS], cnt[OWN_CELLS];
  int tag[OWN_HOT];
  int seen[1 << OWN_SEEN_LOG];
  int source;  // whose hot groups the tags are
  int cached;  // whether it has any
};

// Every thread of the block; a barrier follows before the first use.
__device__ __forceinline__ void own_init(OwnSums& S) {
  for (int i = threadIdx.x; i < OWN_CELLS; i += blockDim.x) S.lo[i] = S.hi[i] = S.cnt[i] = 0;
  for (int i = threadIdx.x; i < 1 << OWN_SEEN_LOG; i += blockDim.x) S.seen[i] = -1;
  if (threadIdx.x == 0) S.source = -1;
}

// A thread's view of the cells for one item.
struct Own {
  OwnSums& S;
  int ng;        // small: the groups
  bool small;
  bool look;     // the source's first rows in this block: watch for repeats
  bool cached;
  int lcopies;
  unsigned copy;
  int repeats;

  __device__ __forceinline__ explicit Own(OwnSums& s) : S(s) {}

  // Every thread, at an item's start, after a barrier since the last item.
  __device__ __forceinline__ void begin(int source, long long groups) {
    small = groups <= OWN_SMALL;
    ng = small ? (int)groups : 0;
    lcopies = 0;
    if (small)
      while (lcopies < 5 && (ng << (lcopies + 1)) <= OWN_CELLS) ++lcopies;
    copy = threadIdx.x & ((1u << lcopies) - 1);
    repeats = 0;
    look = S.source != source;
    cached = !look && S.cached;
    if (look) {
      for (int i = threadIdx.x; i < OWN_HOT; i += blockDim.x) S.tag[i] = -1;
      __syncthreads();  // every thread has read S.source
      if (threadIdx.x == 0) {
        S.source = source;
        S.cached = 0;
      }
      __syncthreads();
    }
  }

  __device__ __forceinline__ void add_cell(unsigned c, long long v) {
    const unsigned l = (unsigned)(unsigned long long)v;
    const unsigned hw = (unsigned)((unsigned long long)v >> 32);
    const unsigned old = atomicAdd(&S.lo[c], l);
    const unsigned hc = hw + (old + l < old ? 1u : 0u);
    if (hc) atomicAdd(&S.hi[c], hc);
    atomicAdd(&S.cnt[c], 1u);
  }

  // One row of group g into the cells; false: the caller adds it to the slab.
  // first: of the item's first step.
  __device__ __forceinline__ bool add(unsigned g, long long v, bool first) {
    if (small) {
      add_cell(g << lcopies | copy, v);
      return true;
    }
    if (!cached && !(look && first)) return false;
    const unsigned mixed = g * 0x9E3779B1u;
    volatile int* seen = &S.seen[mixed >> (32 - OWN_SEEN_LOG)];
    if (!cached) {
      repeats += *seen == (int)g;
      *seen = (int)g;
      return false;
    }
    unsigned slot = mixed >> (32 - OWN_HOT_LOG);
    const int t0 = *(volatile int*)&S.tag[slot], t1 = *(volatile int*)&S.tag[slot ^ 1];
    if (t1 == (int)g) slot ^= 1;
    if (t0 == (int)g || t1 == (int)g) {
      add_cell(slot * OWN_COPIES + (threadIdx.x & (OWN_COPIES - 1)), v);
      return true;
    }
    if (*seen == (int)g) {
      if (t0 == -1) atomicCAS(&S.tag[slot], -1, (int)g);
      else if (t1 == -1) atomicCAS(&S.tag[slot ^ 1], -1, (int)g);
    } else {
      *seen = (int)g;
    }
    return false;
  }

  // Every thread, after the item's first step.
  __device__ __forceinline__ void after_first() {
    if (!look || small) return;
    cached = __syncthreads_count(repeats > 0) >= OWN_REPEATS;
    if (threadIdx.x == 0) S.cached = cached;
  }

  // Every thread, at the item's end: the cells into the slab, and emptied.
  __device__ __forceinline__ void flush(unsigned long long* slab) {
    __syncthreads();
    const int cells = small ? ng : cached ? OWN_HOT : 0;
    const int per = small ? 1 << lcopies : OWN_COPIES;
    for (int i = threadIdx.x; i < cells; i += blockDim.x) {
      const long long g = small ? i : (long long)(unsigned)S.tag[i];
      if (!small && S.tag[i] == -1) continue;
      unsigned long long sum = 0, n = 0;
      for (int j = 0; j < per; ++j) {
        const int c = i * per + ((j + (int)threadIdx.x) & (per - 1));
        sum += (unsigned long long)S.hi[c] << 32 | S.lo[c];
        n += S.cnt[c];
        S.lo[c] = S.hi[c] = S.cnt[c] = 0;
      }
      if (!n) continue;
      red_add(&slab[2 * g], sum);
      red_add(&slab[2 * g + 1], n);
    }
    __syncthreads();
  }
};

}  // namespace pf
