// A hash table of 8-byte entries over unique int64 keys with a small group
// number each, shared by the joins that keep one in L2 or HBM (join_direct.cu,
// batch.cu, serve.cu).
//
// 2^q buckets of four entries, a bucket one 32-byte sector.  A key's hash is a
// bijection of it, so its top q bits (the home bucket) and the 64 - q others
// (the remainder, held in the entry) are the key itself.  An entry is
// {remainder, distance of its bucket from home, group + 1}; a lookup compares
// whole remainders, never a fingerprint.  A row leaves a bucket only when it is
// full, so a bucket with a free entry ends a lookup.  A row that finds no entry
// within the distance field's reach is not in the table: the builder is told.
// (The hash is mix64's bits rotated: rows of one radix bucket, whose top bits
// agree, spread over the table.)
//
// How full it may be: a lookup that leaves its home bucket holds up its warp
// for a round trip, so a table 0.72 full (a bucket in three full) took 553 us
// for 3M x 18M rows where one of 0.36 takes 306.
#pragma once

#include "common.cuh"

namespace pf {

constexpr unsigned long long CT_EMPTY = 0;  // an entry's group field counts from 1

struct CompactTable {
  unsigned long long* e;  // [4 << q]
  int q, gbits, dbits;
};

__device__ __forceinline__ unsigned long long ct_hash(long long key) {
  const unsigned long long h = mix64((uint64_t)key);
  return h << 21 | h >> 43;
}

struct CtBucket {
  unsigned long long e[4];
};
__device__ __forceinline__ CtBucket ct_load(const unsigned long long* p) {
  CtBucket b;
  asm volatile("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];"
               : "=l"(b.e[0]), "=l"(b.e[1]), "=l"(b.e[2]), "=l"(b.e[3])
               : "l"(p)
               : "memory");
  return b;
}

// The home bucket of a hash, and its remainder at its place in an entry.
__device__ __forceinline__ const unsigned long long* ct_home(const CompactTable& t,
                                                             unsigned long long h) {
  return t.e + 4 * (h >> (64 - t.q));
}
__device__ __forceinline__ unsigned long long ct_want(const CompactTable& t,
                                                      unsigned long long h) {
  return (h << t.q >> t.q) << (t.dbits + t.gbits);
}

// Claims an entry for a key of group g (g < 0: none; its rows match without a
// group), without reading it first, from the one the hash picks, and the next
// ones while they are taken: 1.2 claims a row in a table at most 0.4 full (4M
// claims of 64 MiB take 39 us, a read and a claim of the same entry 84).  False:
// no entry within reach.
__device__ __forceinline__ bool ct_insert(const CompactTable& t, long long key, long long g) {
  const unsigned long long h = ct_hash(key), mask = (1ULL << t.q) - 1;
  const unsigned long long group = g >= 0 ? (unsigned long long)g + 1 : (1ULL << t.gbits) - 1;
  const unsigned long long e = ct_want(t, h) | group, home = h >> (64 - t.q);
  for (int k = 0; k < 4 << t.dbits; ++k) {
    const unsigned d = (unsigned)k >> 2;
    if (atomicCAS(t.e + 4 * ((home + d) & mask) + ((h + (unsigned)k) & 3), CT_EMPTY,
                  e + ((unsigned long long)d << t.gbits)) == CT_EMPTY)
      return true;
  }
  return false;
}

// A remainder and distance among a bucket's entries: the entry (CT_EMPTY:
// none); *more: the lookup goes on in the next bucket.  An entry's low word is
// not zero (its group field), so the low words show a free one.
__device__ __forceinline__ unsigned long long ct_among(const CompactTable& t, const CtBucket& b,
                                                       unsigned long long want, bool* more) {
  const unsigned long long keep = ~((1ULL << t.gbits) - 1);
  unsigned long long r = CT_EMPTY;
  unsigned least = ~0u;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const unsigned low = (unsigned)b.e[j];
    if (((b.e[j] ^ want) & keep) == 0 && low) r = b.e[j];
    least = min(least, low);
  }
  *more = r == CT_EMPTY && least;
  return r;
}

// The lookup past the home bucket.
__device__ __forceinline__ unsigned long long ct_walk(const CompactTable& t,
                                                      unsigned long long h,
                                                      unsigned long long want) {
  const unsigned long long mask = (1ULL << t.q) - 1;
  unsigned long long b = h >> (64 - t.q), r = CT_EMPTY;
  bool more = true;
  for (int d = 1; d < 1 << t.dbits && more; ++d) {
    b = (b + 1) & mask;
    want += 1ULL << t.gbits;
    r = ct_among(t, ct_load(t.e + 4 * b), want, &more);
  }
  return r;
}

// The group of an entry, or -1 where it has none.
__device__ __forceinline__ long long ct_group(const CompactTable& t, unsigned long long e) {
  const unsigned g = (unsigned)(e & ((1ULL << t.gbits) - 1));
  return g == (1u << t.gbits) - 1u ? -1 : (long long)g - 1;
}

inline int bits_of(unsigned long long x) { return x ? 64 - __builtin_clzll(x) : 0; }

// The table for n rows and G groups: the smallest of at most 2^max_q buckets,
// at most `load` full (`load_top` from 2^(max_q - 1) buckets on), whose entry
// has three bits of distance left (a table that empty has no run of seven full
// buckets); false when there is none.
inline bool ct_size(long long n, long long G, int max_q, double load, double load_top, int* q,
                    int* gbits, int* dbits) {
  *gbits = bits_of((unsigned long long)G + 1);  // 1 to G, and all ones for no group
  for (*q = 6; *q <= max_q; ++*q) {
    const double full = (double)n / (double)(4LL << *q);
    const int room = *q - *gbits;
    if (full <= (*q < max_q - 1 ? load : load_top) && room >= 3) {
      *dbits = room < 6 ? room : 6;
      return true;
    }
  }
  *q = 0;
  return false;
}

}  // namespace pf
