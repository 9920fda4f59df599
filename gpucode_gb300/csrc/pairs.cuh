/*
 * pairs.cuh -- the native engine's pair list (pairs.cu): each pair of
 * neighbouring spheres once, with its history record.
 */
#pragma once

#include <cuda_runtime.h>

#include "dem_internal.h"

namespace dem {

/* a slot without a pair: the pair arrays were full (reported as an overflow) */
constexpr int kNoPair = (int)0x80000000;

/* bytes of one pair's result in a mixed step (mixed.cu) */
constexpr size_t kPairOut32 = 48;

/* A mixed pair's record in rec[]: the spring and the largest overlap in FP64 (32
 * bytes, one sector, at 32 p) and, after cap of these, the overlap, plastic
 * radius, plastic offset and load stage (16 bytes, at 16 p).  The FP32 copy of
 * the spring that MixedRec has beside them is its truncation (d2f): 16 bytes a
 * pair and direction less to move. */
constexpr size_t kPairRec32 = 48;

/* The pair arrays (device pointers), twice: ctl[0] is the current set,
 * ctl[1 + set] the number of pairs in it; ctl[3] counts the wall slots in use
 * (mixed.cu), ctl[4] the list entries that found no pair.  off: first
 * pair of each sphere (n + 1; the pairs after off[n] are one-sided).  eidx: per
 * neighbour slot, the pair's index, ~index where the slot's sphere is the
 * pair's second one.  sides: the records and flags a pair has, 1 (mixed, in two
 * parts) or 2 (FP64, one as each sphere sees it: record sides * p + side). */
struct PairSet {
  int2* pair[2];
  int* off[2];
  ContactRec* rec[2];
  unsigned char* brg[2];
  int* eidx;
  int* ctl;
  int cap, sides;
};

/* the control word in one load: (current set, pairs of set 0, of set 1, wall slots) */
__device__ __forceinline__ int4 pair_ctl(const PairSet& ps) { return *reinterpret_cast<const int4*>(ps.ctl); }

/* pairs a set-up's arrays hold: half the slots, and a reserve for entries that
 * have no mirror image */
inline long long pair_capacity(long long n, long long slots) {
  const long long half = (slots + 1) / 2 + n / 8 + 64;
  const long long most = 0x7ffffff0ll;
  const long long c = half < slots ? half : slots;
  return c < most ? c : most;
}

/* neighbour lists: level/slot-major slots, their counts, and the tables that
 * find a sphere's slots */
struct NeborLists {
  const int *nebor, *num, *nidx, *plevel, *npars, *nneb;
};

/* condense fresh neighbour lists into the set that is not current; owned: the
 * higher-indexed partners of each list (neighbor_find); scratch (n + 64 ints) is
 * free to use */
dem_status pair_build(const PairSet& ps, const NeborLists& nl, int n, const int* owned, void* scratch, int* err,
                      cudaStream_t s);
/* the same counts of lists that come from elsewhere */
dem_status pair_owned(const NeborLists& nl, int n, int* owned, cudaStream_t s);
/* link the slots of the pairs' second spheres, and fill the pairs' records and
 * flags from the current set's; src[q]: sphere q's position before the rebuild
 * (NULL: unchanged) */
dem_status pair_carry(const PairSet& ps, const NeborLists& nl, int n, const int* src, int* err, cudaStream_t s);
/* make it the current set */
dem_status pair_flip(const PairSet& ps, cudaStream_t s);

/* out[set][i] = sum of in[0 .. i) for i <= n, set = the one that is not
 * current (build.cu); scratch: a scan tile's total per 2048 entries */
dem_status exclusive_scan(const int* in, int n, int* out0, int* out1, const int* ctl, void* scratch, cudaStream_t s);

}  // namespace dem
