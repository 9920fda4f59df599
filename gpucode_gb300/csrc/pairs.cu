/*
 * pairs.cu -- the pair list of the native engine and its history.
 *
 * The reference keeps a contact's history twice, once in each sphere's slots,
 * and evaluates every contact twice (kernel.cu:463-546).  The two evaluations
 * mirror one another: the normal, the relative velocity and the tangential
 * spring change sign, everything else is the same.  The engine therefore works
 * on pairs: at every rebuild the neighbour lists (level/slot-major, the
 * reference's, kept for the API) are condensed into
 *   pair[p] = (i, j), the pairs each sphere owns one after another in list
 *             order (off[i] .. off[i + 1]).  Mixed precision keeps one history
 *             record and one bridge flag per pair, as sphere i sees j; FP64 keeps
 *             the two the reference keeps, which differ in last bits because
 *             its overlap subtracts the own radius first;
 *   eidx[s]   per used neighbour slot: its pair's index, complemented (~p) in
 *             the slots of the sphere that does not own the pair.
 * A sphere owns its pairs with higher-indexed partners.  A list entry of a
 * lower-indexed partner that does not list the sphere itself (possible only
 * where a list overflowed, or where the two searches decide a pair at the
 * cut-off differently) becomes a one-sided pair after all others, so that it
 * acts on its own sphere alone, as in the reference.
 *
 * A step then runs one thread per pair (FP64: per pair and side) over
 * consecutive records and one thread per sphere over its pairs' results
 * (mixed.cu, step64.cu): a warp's lanes all hold a pair, and in mixed precision
 * the law evaluations and the history traffic are half those of a thread per
 * sphere that walks its own slots.
 *
 * The pair arrays exist twice; the rebuild reads set `cur` and writes the
 * other, so no history is copied aside first.  ctl[0] says which set is
 * current, ctl[1 + set] how many pairs it holds: every kernel reads them as
 * one 16-byte word.
 */
#include <cuda_runtime.h>

#include "dem_device.cuh"
#include "pairs.cuh"

namespace dem {
namespace {

inline int grid_for(long long n, int block) { return n <= 0 ? 1 : (int)((n + block - 1) / block); }

/* a pointer of one of the two sets (a dynamic index into the parameter would
 * go through local memory) */
template <class T>
__device__ __forceinline__ T* pick(T* const (&v)[2], int k) {
  return k ? v[1] : v[0];
}

/* sphere q's slots: first, stride */
__device__ __forceinline__ long long first_slot(const NeborLists& nl, int q, long long& stride) {
  const int L = nl.plevel[q];
  stride = nl.npars[L];
  return slot_base(L, nl.npars, nl.nneb) + nl.nidx[q];
}

/* the pairs each sphere owns, of lists that no search has just counted */
__global__ void k_owned(NeborLists nl, int n, int* __restrict__ owned) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  long long stride;
  const long long base = first_slot(nl, q, stride);
  const int nn = nl.num[q];
  int m = 0;
  for (int k = 0; k < nn; k++) m += nl.nebor[base + k * stride] >= q;
  owned[q] = m;
}

/* list entries a sphere's thread has in flight */
constexpr int kSlotBatch = 4;

/* the pairs and their owners' slots, from the scanned counts (the set that is
 * not current).  Pairs past the arrays' capacity are dropped and reported
 * like a slot overflow. */
__global__ void k_pair_fill(PairSet ps, NeborLists nl, int n, int* __restrict__ err) {
  const int q = reversed_block_thread();
  if (q >= n) return;
  const int nx = 1 - ps.ctl[0];
  const int* __restrict__ off = pick(ps.off, nx);
  int2* __restrict__ pair = pick(ps.pair, nx);
  if (q == 0) {
    const int total = off[n];
    ps.ctl[1 + nx] = min(total, ps.cap);
    if (total > ps.cap) atomicOr(err, 1);
  }
  long long stride;
  const long long base = first_slot(nl, q, stride);
  const int nn = nl.num[q];
  int p = off[q];
  for (int k0 = 0; k0 < nn; k0 += kSlotBatch) {
    int j[kSlotBatch];
#pragma unroll
    for (int t = 0; t < kSlotBatch; t++) j[t] = k0 + t < nn ? nl.nebor[base + (k0 + t) * stride] : -1;
#pragma unroll
    for (int t = 0; t < kSlotBatch; t++) {
      if (j[t] < q) continue;
      if (p < ps.cap) pair[p] = make_int2(q, j[t]);
      ps.eidx[base + (k0 + t) * stride] = p < ps.cap ? p : kNoPair;
      p++;
    }
  }
}

/* a record in two 256-bit accesses */
union RecWords {
  ContactRec r;
  float f[16];
  __device__ __forceinline__ RecWords() {}
};
__device__ __forceinline__ ContactRec read_rec(const ContactRec* p) {
  RecWords w;
  const float* q = reinterpret_cast<const float*>(p);
#pragma unroll
  for (int h = 0; h < 2; h++) {
    float* f = w.f + 8 * h;
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]), "=f"(f[4]), "=f"(f[5]), "=f"(f[6]), "=f"(f[7])
        : "l"(q + 8 * h));
  }
  return w.r;
}
__device__ __forceinline__ void write_rec(ContactRec* p, const ContactRec& r) {
  RecWords w;
  w.r = r;
  float* q = reinterpret_cast<float*>(p);
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const float* f = w.f + 8 * h;
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(q + 8 * h), "f"(f[0]), "f"(f[1]), "f"(f[2]),
                 "f"(f[3]), "f"(f[4]), "f"(f[5]), "f"(f[6]), "f"(f[7])
                 : "memory");
  }
}

/* HstryCopyG (kernel.cu:869-911) for one new pair: the record and bridge flag
 * of the same two spheres' old pair, or zero.  The old pair is looked for among
 * the few owned by the lower of its spheres' old positions, then by the
 * other's, then among the one-sided ones. */
__device__ __forceinline__ void carry_pair(const PairSet& ps, int cur, int n, int p, int2 ij, const int* src) {
  const int* __restrict__ off = pick(ps.off, cur);
  const int2* __restrict__ old = pick(ps.pair, cur);
  const int Pold = ps.ctl[1 + cur];
  const int oi = src ? src[ij.x] : ij.x, oj = src ? src[ij.y] : ij.y;
  const int a = min(oi, oj), b = max(oi, oj);
  int hit = -1;
  for (int t = off[a], e = min(off[a + 1], Pold); t < e && hit < 0; t++)
    if (old[t].y == b) hit = t;
  if (hit < 0) {
    for (int t = off[b], e = min(off[b + 1], Pold); t < e && hit < 0; t++)
      if (old[t].y == a) hit = t;
    for (int t = off[n]; t < Pold && hit < 0; t++)
      if (old[t].x == b && old[t].y == a) hit = t;
  }
  const bool turned = hit >= 0 && old[hit].x != oi;
  if (ps.sides == 1) {
    const float4* from = reinterpret_cast<const float4*>(pick(ps.rec, cur));
    float4* to = reinterpret_cast<float4*>(pick(ps.rec, 1 - cur));
    float4 a4 = make_float4(0.f, 0.f, 0.f, 0.f), b4 = a4, law = a4;
    unsigned char brg = 0;
    if (hit >= 0) {
      get2(from + 2 * (size_t)hit, a4, b4);
      law = from[2 * (size_t)ps.cap + hit];
      brg = pick(ps.brg, cur)[hit];
      if (turned) { /* the spring as the other sphere sees it: the signs of three doubles */
        a4.y = __uint_as_float(__float_as_uint(a4.y) ^ 0x80000000u);
        a4.w = __uint_as_float(__float_as_uint(a4.w) ^ 0x80000000u);
        b4.y = __uint_as_float(__float_as_uint(b4.y) ^ 0x80000000u);
      }
    }
    put2(to + 2 * (size_t)p, a4, b4);
    to[2 * (size_t)ps.cap + p] = law;
    pick(ps.brg, 1 - cur)[p] = brg;
    return;
  }
  for (int side = 0; side < 2; side++) {
    ContactRec r;
    unsigned char brg = 0;
    if (hit >= 0) {
      const long long from = 2LL * hit + (turned ? 1 - side : side);
      r = read_rec(pick(ps.rec, cur) + from);
      brg = pick(ps.brg, cur)[from];
    } else {
      r.dx = r.dy = r.dz = r.nDsp = r.nDsp_mx = r.plstRad = r.plstDfm = 0.0;
      r.stage = 0;
    }
    write_rec(pick(ps.rec, 1 - cur) + 2LL * p + side, r);
    pick(ps.brg, 1 - cur)[2LL * p + side] = brg;
  }
}

/* The links from the slots of the pairs' second spheres: a thread per sphere
 * looks for itself among the few pairs of each lower-indexed partner, which lie
 * together.  (Looking for the pair's first sphere in the second one's list, a
 * thread per pair, read a sector per entry of lists that lie apart.) */
__device__ __forceinline__ void link_slots(const PairSet& ps, const NeborLists& nl, int n, int q, int cur) {
  int lost = 0;
  if (q < n) {
    const int* __restrict__ off = pick(ps.off, 1 - cur);
    const int2* __restrict__ pair = pick(ps.pair, 1 - cur);
    long long stride;
    const long long base = first_slot(nl, q, stride);
    const int nn = nl.num[q];
    for (int k0 = 0; k0 < nn; k0 += kSlotBatch) {
      int j[kSlotBatch], at[kSlotBatch], end[kSlotBatch];
#pragma unroll
      for (int t = 0; t < kSlotBatch; t++) j[t] = k0 + t < nn ? nl.nebor[base + (k0 + t) * stride] : n;
#pragma unroll
      for (int t = 0; t < kSlotBatch; t++) {
        at[t] = j[t] < q ? off[j[t]] : 0;
        end[t] = j[t] < q ? min(off[j[t] + 1], ps.cap) : 0;
      }
#pragma unroll
      for (int t = 0; t < kSlotBatch; t++) {
        if (j[t] >= q) continue;
        int p = at[t];
        while (p < end[t] && pair[p].y != q) p++;
        const bool hit = p < end[t];
        ps.eidx[base + (k0 + t) * stride] = hit ? ~p : kNoPair;
        lost += !hit;
      }
    }
  }
  lost = __reduce_add_sync(0xffffffffu, lost);
  if ((threadIdx.x & 31) == 0 && lost) atomicAdd(ps.ctl + 4, lost);
}

/* One thread per new pair: its history; the first link_blocks blocks link the
 * slots meanwhile.  Bound by the scattered reads of the old pair and its record:
 * 53.5 us cold on the packed wet bed, 69 as one pass per pair with plain copies. */
__global__ void __launch_bounds__(256) k_carry(PairSet ps, NeborLists nl, int n, const int* __restrict__ src,
                                               int link_blocks) {
  const int cur = ps.ctl[0];
  if (blockIdx.x < link_blocks) {
    link_slots(ps, nl, n, (link_blocks - 1 - blockIdx.x) * blockDim.x + threadIdx.x, cur);
    return;
  }
  const int P = ps.ctl[2 - cur];
  const int2* __restrict__ pair = pick(ps.pair, 1 - cur);
  const int step = (gridDim.x - link_blocks) * blockDim.x;
  for (int p = (blockIdx.x - link_blocks) * blockDim.x + threadIdx.x; p < P; p += step)
    carry_pair(ps, cur, n, p, pair[p], src);
}

/* One-sided pairs for the slots that found none: nothing to do on a set of
 * lists that mirror one another. */
__global__ void k_one_sided(PairSet ps, NeborLists nl, int n, const int* __restrict__ src,
                            int* __restrict__ err) {
  if (ps.ctl[4] == 0) return;
  const int cur = ps.ctl[0];
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    long long stride;
    const long long base = first_slot(nl, q, stride);
    const int nn = nl.num[q];
    for (int k = 0; k < nn; k++) {
      const long long s = base + k * stride;
      if (ps.eidx[s] != kNoPair || nl.nebor[s] >= q) continue;
      const int p = atomicAdd(ps.ctl + 2 - cur, 1);
      if (p >= ps.cap) {
        atomicSub(ps.ctl + 2 - cur, 1);
        atomicOr(err, 1);
        continue;
      }
      const int2 ij = make_int2(q, nl.nebor[s]);
      pick(ps.pair, 1 - cur)[p] = ij;
      ps.eidx[s] = p;
      carry_pair(ps, cur, n, p, ij, src);
    }
  }
}

__global__ void k_flip(int* ctl) {
  ctl[0] = 1 - ctl[0];
  ctl[4] = 0;
}

}  // namespace

dem_status pair_owned(const NeborLists& nl, int n, int* owned, cudaStream_t s) {
  k_owned<<<grid_for(n, 128), 128, 0, s>>>(nl, n, owned);
  return cuda_check(cudaGetLastError(), "pair count launch");
}

dem_status pair_build(const PairSet& ps, const NeborLists& nl, int n, const int* owned, void* scratch, int* err,
                      cudaStream_t s) {
  dem_status st = exclusive_scan(owned, n, ps.off[0], ps.off[1], ps.ctl, scratch, s);
  if (st != DEM_OK) return st;
  k_pair_fill<<<grid_for(n, 128), 128, 0, s>>>(ps, nl, n, err);
  return cuda_check(cudaGetLastError(), "pair list launch");
}

dem_status pair_carry(const PairSet& ps, const NeborLists& nl, int n, const int* src, int* err, cudaStream_t s) {
  const long long most = 6LL * n; /* beyond it the grid strides */
  const int link = grid_for(n, 256);
  k_carry<<<link + grid_for(most < ps.cap ? most : ps.cap, 256), 256, 0, s>>>(ps, nl, n, src, link);
  k_one_sided<<<grid_for(n < 152 * 1024 ? n : 152 * 1024, 256), 256, 0, s>>>(ps, nl, n, src, err);
  return cuda_check(cudaGetLastError(), "history carry launch");
}

dem_status pair_flip(const PairSet& ps, cudaStream_t s) {
  k_flip<<<1, 1, 0, s>>>(ps.ctl);
  return cuda_check(cudaGetLastError(), "pair set launch");
}

}  // namespace dem
