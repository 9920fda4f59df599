/*
 * mixed.cu -- the FP32-force / FP64-state step kernels (sm_103a).
 *
 * Two launches per time step: k_pair_mixed, one thread per pair of the pair
 * list (pairs.cu) -- contact law and capillary bridge, the pair's history --
 * with the listed walls as its first blocks; and k_body_mixed, one thread per
 * sphere -- gravity, the sum of its pairs' and walls' results, the integrator.
 * Together the reference's VarInit + PPForceCalcG + CirPWInterG + UpdateSystemG
 * (kernel.cu:413-606, 958-1023).
 *
 * Why two: a thread per sphere that walks its own slots evaluates every pair
 * twice, moves its history twice, keeps 18 of 32 lanes busy (lists of 2 to 30
 * entries) and chains index -> shadow -> record -> law per slot.  On the packed
 * 200k wet bed that one kernel took 114 us; the pair kernel takes 27 us (25 of
 * 32 lanes, half the evaluations, 68 + 13 MB of DRAM traffic at 56 % occupancy;
 * bound by issue, 65 %) and the sphere kernel 32 us (bound by the gather of the
 * pairs' results), 61 against 116 us a chained step; 2M spheres 520 against 912
 * us, 5,000 dry spheres 15 against 43 us (a graph of several steps among it).
 *
 * Why this shape on GB300: FP64 arithmetic runs at ~0.6 T op/s (1/58 of
 * FP32) and FP64 pow at ~6 G/s, so the reference's all-FP64 pair math is
 * bound by FP64 issue.  Here:
 *  - neighbours are read from FP32 "shadow" copies of last step's state
 *    (double-buffered: step t reads buffer t%2, writes the other), written by
 *    the integrator;
 *  - positions are shadowed as hi + lo float pairs of (x + offset), where the
 *    offset puts every coordinate in the binade [2^k, 2^(k+1)): hi_i - hi_j
 *    is then exact (Sterbenz), and the overlap d - (ri + rj) is computed as
 *    (d^2 - S^2) / (d + S) with d^2 - S^2 accumulated from exact products
 *    (FMA two-products + two-sums), so the overlap keeps ~1e-7 relative
 *    accuracy without FP64 operations even though d and S agree to 1e-4;
 *  - pair forces are FP32, summed per particle with Kahan compensation in
 *    the reference's neighbour order;
 *  - FP64 stays for the state (integrator) and for the tangential spring of
 *    the contact history, which is advanced by FP64 additions of FP32
 *    increments (projection correction, length-preserving rescale written as
 *    a small difference, v_t dt) so its accumulation error is relative to
 *    the increment, not to the spring;
 *  - contact records are 48 bytes (a sector and half a one) read and written only
 *    for contacts, streamed past L2's reusable lines; bridge flags are one byte a
 *    pair; a pair's two spheres get one evaluation, mirrored by its signs.
 */
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "capnet.cuh"
#include "dem_device.cuh"
#include "engine.h"

namespace dem {

struct MixedState {
  /* the FP32 shadows, two float4 to a sphere so that what is read together is
   * one 32-byte sector: the position's high parts and radius, the low parts;
   * the velocity and bridge count, the spin */
  float4 *place[2], *motion[2];
  float4* force;
  float4* wall_out; /* the step's wall results, two per wall slot */
  int* wall_entry;  /* the listed wall slots (slot w of sphere q: w * n + q) */
  double3 off;
  float coarse_tol;
  int bin_exp;    /* FP64 biased exponent of the binade [2^k, 2^(k+1)) */
  float base;     /* 2^k: the offset coordinate of the domain's origin */
  float lo_scale; /* 2^(k-52): the weight of the last significand bit */
};

namespace {

inline int grid_for(long long n, int block) { return n <= 0 ? 1 : (int)((n + block - 1) / block); }

constexpr float kPiF = 3.1415926f;

/* contact-law constants in FP32 */
struct Law32 {
  float emod, pois, sfrc, ydsp, yforce, ystiff;
  float rot_eps, dsmx_eps;
  float kt;      /* 16 (1 - pois) emod / (4 - 2 pois): slip-distance denominator */
  float dmp;     /* sqrt(dmpn product) */
  int hertz_le;  /* p-p: <=, wall: < */
  int damp_on;
};

struct MixArgs {
  const float4 *place_in, *motion_in;
  const int* body_order; /* the sphere kernel's blocks, levels side by side (NULL: in reverse) */
  float4 *place_out, *motion_out;
  double3 *pos, *vel, *angv;
  const double* rad;
  double* pmove;
  const int *num_nebor, *plevel, *nidx, *npars, *nneb;
  PairSet ps;
  float4* pair_out; /* two float4s per pair, then what bridges and rolling add (k_pair_mixed) */
  float4* wall_out; /* the same per wall slot */
  const int* wall_entry; /* the listed wall slots, ctl[3] of them */
  unsigned wall_blocks;
  const int *wlist, *nwall;
  ContactRec* wrec;
  float4* force_out;
  int *flag, *err;
  unsigned long long* counters;
  const CylinderBC* cyl;
  int n, force_cap;
  double3 off;
  float3 offf;    /* the offset rounded to FP32 */
  float wall_tol; /* bound on the error of the FP32 wall gap from the shadow */
  int bin_exp;
  float lo_scale;
  double dt, move_limit; /* 0.3 * SearchGap */
  float dtf, rfrc;
  float lqd_vol, lqd_layer, lqd_gapmn, lqd_st;
  Law32 pp, pw;
  /* batched systems (NULL for one system): system of each particle id (its
   * cylinder is cyl[system]) and whether the system is wet */
  const int *sys_of_id, *sys_wet;
  /* learned capillary closure (NET variant only) */
  const int* id;
  const CapNetSmem* capw;
  unsigned long long theta_seed;
  float theta_max;
  /* a step chained on the device: the rebuild request word; when it is set
   * the step does nothing (it runs again after the rebuild).  NULL otherwise */
  const int* gate;
  /* the liquid model in FP32 (liquid.cuh): mode 0 the reference's, 1 per-contact
   * volumes (fraction lq_vmin + lq_vspan u of the smaller sphere) and angles */
  int lq_mode;
  float lq_vmin, lq_vspan, lq_theta_max;
  unsigned long long lq_seed;
};

__device__ __forceinline__ float3 f3(float x, float y, float z) { return make_float3(x, y, z); }
__device__ __forceinline__ float3 operator+(float3 a, float3 b) { return f3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ float3 operator-(float3 a, float3 b) { return f3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float3 operator*(float3 a, float s) { return f3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ float3 operator*(float s, float3 a) { return f3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ float dotf(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float lenf(float3 a) { return sqrtf(dotf(a, a)); }
__device__ __forceinline__ float3 crossf(float3 a, float3 b) {
  return f3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}

/* Kahan-compensated running sum */
struct KSum {
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float v) {
    const float y = v - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
  }
};
struct KSum3 {
  KSum x, y, z;
  __device__ __forceinline__ void add(float3 v) { x.add(v.x); y.add(v.y); z.add(v.z); }
};
/* error-free transforms (Knuth two-sum, FMA two-product) */
__device__ __forceinline__ float two_sum(float a, float b, float& err) {
  const float s = a + b;
  const float bb = s - a;
  err = (a - (s - bb)) + (b - bb);
  return s;
}

/* The overlap of spheres i and j from their shadows, exactly enough for a
 * contact law: with a = hi_i - hi_j (exact: both in one binade) and
 * b = lo_i - lo_j, d^2 - S^2 is accumulated from error-free pieces (FMA
 * two-products, Knuth two-sums) and the overlap is (d^2 - S^2) / (d + S), so
 * it keeps ~1e-7 relative accuracy although d and S agree to ~1e-4.  Returns
 * the gap (negative: overlap); u is the unit vector from j to i, rj j's radius. */
__device__ __forceinline__ float exact_gap(float4 hi, float4 lo, float4 hj, float4 lj, float ax, float ay, float az,
                                           float3& u, float& rj) {
  rj = hj.w + lj.w;
  const float bx = lo.x - lj.x, by = lo.y - lj.y, bz = lo.z - lj.z;
  const float px = ax * ax, py = ay * ay, pz = az * az;
  const float ex = fmaf(ax, ax, -px), ey = fmaf(ay, ay, -py), ez = fmaf(az, az, -pz);
  float t1, t2, es;
  const float s1 = two_sum(px, py, t1);
  const float s2 = two_sum(s1, pz, t2);
  const float slo = (lo.w + lj.w);
  const float Sh = two_sum(hi.w, hj.w, es);
  const float Sl = es + slo;
  const float qq2 = Sh * Sh, eq = fmaf(Sh, Sh, -qq2);
  const float s3 = s2 - qq2;
  const float small = (t1 + t2) + (ex + ey + ez - eq) + 2.0f * (ax * bx + ay * by + az * bz) -
                      2.0f * Sh * Sl + (bx * bx + by * by + bz * bz) - Sl * Sl;
  const float D = s3 + small;
  const float dx = ax + bx, dy = ay + by, dz = az + bz;
  const float dist = sqrtf(dx * dx + dy * dy + dz * dz);
  const float inv = __frcp_rn(dist);
  u = make_float3(dx * inv, dy * inv, dz * inv);
  return __fdividef(D, dist + (Sh + Sl));
}

/* the elasto-plastic normal law, damping and tangential spring of
 * kernel.cu:89-228 / :236-359 in FP32: the normal force fN, the damping fD
 * (both along u) and the friction fT.  The spring is advanced
 * as an FP64 update by a small FP32 increment (three FP64 adds per contact);
 * the maximum overlap stays an FP64 field. */
__device__ __forceinline__ void law32_forces(const Law32& c, float ijRad, float nrm, float3 u, float3 cpv, MixedRec& r,
                                      float dt, float& fN_out, float& fD_out, float3& fT_out) {
  const float plstDfm0 = r.plstDfm, nDsp0 = r.nDsp, nDspMx0 = d2f(r.nDsp_mx);
  float plstRad = r.plstRad, plstDfm = plstDfm0;
  int st;
  if (nrm < plstDfm0) st = 1;
  else if (nrm >= plstDfm0 && nrm < nDsp0) st = 3;
  else if (nrm >= nDsp0 && nrm < nDspMx0) st = 4;
  else st = 2;
  float fN = 0.f;
  const float k43 = 4.0f / 3.0f * c.emod;
  const float sq = sqrtf(ijRad * nrm);
  if (st == 2) {
    const bool elastic = c.hertz_le ? (nrm <= c.ydsp * ijRad) : (nrm < c.ydsp * ijRad);
    if (elastic) {
      fN = k43 * sq * nrm;
      plstRad = ijRad;
      plstDfm = 0.f;
    } else {
      fN = c.yforce * ijRad * ijRad + c.ystiff * ijRad * (nrm - c.ydsp * ijRad);
      plstRad = ijRad * (k43 * sq * nrm) / fN;
      const float t = cbrtf(fN / (k43 * sqrtf(ijRad)));
      plstDfm = nrm - t * t;
    }
    r.nDsp_mx = f2d(nrm);
  } else if (st != 1) {
    const float t = nrm - plstDfm0;
    fN = k43 * sqrtf(plstRad) * (t * sqrtf(t));
  }
  const float vn = dotf(cpv, u);
  const float fD = c.damp_on ? -2.0f * c.dmp * c.emod * sq * vn : 0.f;
  const float3 vt = cpv - vn * u;

  /* spring: d_new = rescale(project(d)) + v_t dt.  With cq = u.d the
   * projection is d - u cq, of length^2 |d|^2 - cq^2, so the rescale factor
   * minus one is cq^2 / ((|d| + |p|) |p|): every term of the increment is
   * small, and its FP32 error is relative to the increment, not the spring. */
  const float3 d = f3(r.fx, r.fy, r.fz);
  const float cq = dotf(u, d);
  const float3 corr = f3(-u.x * cq, -u.y * cq, -u.z * cq);
  const float ld = lenf(d);
  const float lp = lenf(d + corr);
  float3 inc;
  if (lp > c.rot_eps) {
    const float sm1 = __fdividef(cq * cq, (ld + lp) * lp);
    inc = corr * (1.0f + sm1) + d * sm1 + vt * dt;
  } else {
    inc = corr + vt * dt;
  }
  double nx = r.dx + f2d(inc.x), ny = r.dy + f2d(inc.y), nz = r.dz + f2d(inc.z);
  float3 dn = f3(d2f(nx), d2f(ny), d2f(nz));
  const float dsmx = __fdividef(3.0f * c.sfrc * fN, c.kt * sq);
  float ratio = 1.0f;
  float ldn = lenf(dn);
  if (ldn < dsmx) {
    if (dsmx > c.dsmx_eps) {
      /* the approximate quotient may round above 1 just below the slip limit */
      const float t = fmaxf(0.0f, 1.0f - __fdividef(ldn, dsmx));
      ratio = 1.0f - t * sqrtf(t);
    }
  } else {
    const float f = (ldn > c.dsmx_eps) ? __fdividef(dsmx, ldn) : dsmx;
    const double fd = f2d(f);
    nx *= fd;
    ny *= fd;
    nz *= fd;
    dn = f3(d2f(nx), d2f(ny), d2f(nz));
    ldn = lenf(dn);
  }
  r.dx = nx;
  r.dy = ny;
  r.dz = nz;
  r.fx = dn.x;
  r.fy = dn.y;
  r.fz = dn.z;
  float3 fT = f3(0.f, 0.f, 0.f);
  if (ldn < dsmx) {
    if (ldn > 1.0e-10f) fT = dn * __fdividef(-c.sfrc * fN * ratio, ldn);
  } else {
    const float lvt = lenf(vt);
    if (lvt > 1.0e-10f) fT = vt * __fdividef(-c.sfrc * fN * ratio, lvt);
  }
  fN_out = fN;
  fD_out = fD;
  fT_out = fT;
  r.nDsp = nrm;
  r.plstRad = plstRad;
  r.plstDfm = plstDfm;
  r.stage = st;
}

/* the same with the force, moment and rolling moment on a sphere of radius iRad */
__device__ __forceinline__ void law32(const Law32& c, float ijRad, float nrm, float3 u, float3 cpv, MixedRec& r,
                                      float iRad, float rfrc, float dt, float3& dF, float3& dM, float& dR) {
  float fN, fD;
  float3 fT;
  law32_forces(c, ijRad, nrm, u, cpv, r, dt, fN, fD, fT);
  dF = (fN + fD) * u + fT;
  const float arm = iRad - nrm * 0.5f;
  dM = crossf(u * (-arm), fT);
  dR = 0.5f * (rfrc + rfrc) * fN * iRad;
}

/* a bridge's force magnitude and rupture distance under the context's liquid
 * model: V the pair's bridge volume (reduced, unscaled), th its contact angle
 * (per-contact model only).  The reference's model is kernel.cu:65-81 and
 * :518 in FP32 (the normalised regression: capnet.cuh) */
__device__ __forceinline__ float bridge_force32(const MixArgs& a, float S, float V, float th, float effR) {
  const float s = fmaxf(a.lqd_gapmn, S);
  const float fs = a.lq_mode ? willett32(s, 8.0f * V, th) : cap_formula32(s, 8.0f * V);
  return 2.0f * kPiF * effR * a.lqd_st * fs;
}
__device__ __forceinline__ float bridge_rupture32(const MixArgs& a, float V, float th) {
  return a.lq_mode ? rupture32(V, th) : 0.99f * exp2f(0.33f * __log2f(V));
}

/* get2 and put2 (dem_device.cuh), streaming */
__device__ __forceinline__ void get2cs(const float4* p, float4& a, float4& b) {
  asm volatile("ld.global.cs.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
      : "l"(p) : "memory");
}
__device__ __forceinline__ void put2cs(float4* p, float4 a, float4 b) {
  asm volatile("st.global.cs.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(a.x), "f"(a.y), "f"(a.z),
               "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
               : "memory");
}

/* A contact record is read once and written once per step: streaming
 * (evict-first) loads and stores keep it from displacing the partners'
 * shadows, which a warp's neighbours read again, from L1 (114.6 vs 118.5 us
 * on the packed 200k bed, the same bits) */
__device__ __forceinline__ MixedRec load_rec(const ContactRec* p) {
  const float4* q = reinterpret_cast<const float4*>(p);
  MixedRec r;
  float4* o = reinterpret_cast<float4*>(&r);
  get2cs(q, o[0], o[1]);
  get2cs(q + 2, o[2], o[3]);
  return r;
}
__device__ __forceinline__ void store_rec(ContactRec* p, const MixedRec& r) {
  float4* q = reinterpret_cast<float4*>(p);
  const float4* o = reinterpret_cast<const float4*>(&r);
  put2cs(q, o[0], o[1]);
  put2cs(q + 2, o[2], o[3]);
}

/* read-only global loads (inputs of the step: never written by this launch) */
template <class T>
__device__ __forceinline__ T ro(const T* p) {
  return __ldg(p);
}
/* pull a line into L2 ahead of its use (no register is held meanwhile) */
__device__ __forceinline__ void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

__device__ __forceinline__ void warp_add(unsigned long long* ctr, unsigned v) {
  v = __reduce_add_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(ctr, (unsigned long long)v);
}

/* One bridge of a warp's pairs waiting for the learned closure (16 bytes in
 * shared memory); after the network has run, sep and vol hold its two outputs
 * (normalised force, rupture distance). */
struct __align__(16) CapEntry {
  float sep, vol, theta, ratio; /* raw features */
};
/* resident blocks per SM the network variant is built for: 8 (64 registers, some
 * spills) 114.4 us a closure step on the packed 200k bed, 7 114.6, 6 116.7, 5 122.6, 9
 * 118.6 */
#ifndef DEM_NET_BLOCKS
#define DEM_NET_BLOCKS 8
#endif
constexpr int kNetBlocks = DEM_NET_BLOCKS;
constexpr int kWarps = 4;                  /* warps per block of the step kernels */
constexpr size_t kCapSmem = ((sizeof(CapNetSmem) + 15) / 16) * 16 + sizeof(CapEntry) * 32 * kWarps;

__device__ __forceinline__ uint32_t cap_pair(const CapNetSmem& w, const CapEntry& e, int t) {
  return cap_pair(w, e.sep, e.vol, e.theta, e.ratio, t);
}

/* Run this warp's queued bridges (at most 32) through the network in 16-row
 * BF16 tensor-core tiles.  All 32 lanes call it. */
__device__ __forceinline__ void cap_run_queue(const CapNetSmem& w, CapEntry* qw, int qn) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  __syncwarp();
  for (int t0 = 0; t0 < qn; t0 += 16) {
    const int r0 = t0 + g, r1 = r0 + 8;
    uint32_t xa = 0u, xb = 0u;
    if (t < 2) {
      if (r0 < qn) xa = cap_pair(w, qw[r0], t);
      if (r1 < qn) xb = cap_pair(w, qw[r1], t);
    }
    float o[4];
    cap_tile16(w, xa, xb, o);
    __syncwarp();
    if (t == 0) {
      if (r0 < qn) {
        qw[r0].sep = o[0] * w.y_std[0] + w.y_mean[0];
        qw[r0].vol = o[1] * w.y_std[1] + w.y_mean[1];
      }
      if (r1 < qn) {
        qw[r1].sep = o[2] * w.y_std[0] + w.y_mean[0];
        qw[r1].vol = o[3] * w.y_std[1] + w.y_mean[1];
      }
    }
    __syncwarp();
  }
}

/* pair p's record (pairs.cuh) */
__device__ __forceinline__ MixedRec load_pair_rec(const float4* base, int cap, int p) {
  MixedRec r;
  float4* o = reinterpret_cast<float4*>(&r);
  get2cs(base + 2 * (size_t)p, o[0], o[1]);
  const float4 w = __ldcs(base + 2 * (size_t)cap + p);
  r.fx = d2f(r.dx);
  r.fy = d2f(r.dy);
  r.fz = d2f(r.dz);
  r.nDsp = w.x;
  r.plstRad = w.y;
  r.plstDfm = w.z;
  r.stage = __float_as_int(w.w);
  r.pad = 0;
  return r;
}
__device__ __forceinline__ void store_pair_rec(float4* base, int cap, int p, const MixedRec& r) {
  const float4* o = reinterpret_cast<const float4*>(&r);
  put2cs(base + 2 * (size_t)p, o[0], o[1]);
  __stcs(base + 2 * (size_t)cap + p, make_float4(r.nDsp, r.plstRad, r.plstDfm, __int_as_float(r.stage)));
}

/* One entry of the wall list (sphere q's wall slot w) against its cylinder, the
 * distance in FP64 (CirPWInterG, kernel.cu:958-1023).  The result: the force
 * and the normal force, the moment and the overlap (0: no contact).  Listed walls are evaluated from a compact
 * list (k_wall_entries), one thread each, because a listed sphere is one in
 * six and a touching one in fifteen, spread over almost every warp of a thread
 * per sphere, and the exact distance is two FP64 roots and three divisions. */
__device__ __forceinline__ void wall_entry(const MixArgs& a, int e) {
  const int w = e / a.n, q = e - w * a.n;
  float4 hi, lo;
  get2(a.place_in + 2 * q, hi, lo);
  const float ri = hi.w + lo.w;
  const CylinderBC cy = a.cyl[a.sys_of_id ? a.sys_of_id[ro(a.id + q)] : 0];
  const int kind = a.wlist[3 * q + w];
  float4 f = make_float4(0.f, 0.f, 0.f, 0.f), t = f;
  /* A wall the sphere certainly does not touch costs no FP64 work: a coarse
   * gap from the shadow (hi part of x + offset, truncated to the binade) is
   * within wall_tol of the exact one -- 5 binade ulps for the flat walls, 11
   * for the curved one, bounded by 16 -- so only spheres within wall_tol of a
   * wall take the reference's geometry. */
  float gc;
  if (kind == 2) {
    const float cxo = d2f(cy.cir.x) + a.offf.x, cyo = d2f(cy.cir.y) + a.offf.y;
    const float dx = hi.x - cxo, dy = hi.y - cyo;
    gc = fabsf(sqrtf(dx * dx + dy * dy) - d2f(cy.R)) - ri;
  } else {
    gc = fabsf(hi.z - (d2f(kind == 0 ? cy.Tw : cy.Bw) + a.offf.z)) - ri;
  }
  if (gc <= a.wall_tol) {
    const double3 p = a.pos[q];
    const double rid = a.rad[q];
    double3 jp;
    if (kind == 2) {
      const double ddx = cy.cir.x - p.x, ddy = cy.cir.y - p.y;
      const double dist = sqrt(ddx * ddx + ddy * ddy);
      jp = make_double3(cy.R * ((p.x - cy.cir.x) / dist) + cy.cir.x, cy.R * ((p.y - cy.cir.y) / dist) + cy.cir.y,
                        p.z);
    } else {
      jp = make_double3(p.x, p.y, kind == 0 ? cy.Tw : cy.Bw);
    }
    const double3 d = make_double3(p.x - jp.x, p.y - jp.y, p.z - jp.z);
    const double len = sqrt(d.x * d.x + d.y * d.y + d.z * d.z);
    const float gapw = (float)(len - rid);
    if (gapw < 0.f) {
      const float il = (float)(1.0 / len);
      const float3 u = f3((float)d.x * il, (float)d.y * il, (float)d.z * il);
      float4 vi4, wi4;
      get2(a.motion_in + 2 * q, vi4, wi4);
      /* the top wall's velocity carries over to the walls after it in the
       * list, as the reference's jVel does (kernel.cu:987-1020) */
      double jv = 0.0;
      for (int k = 0; k <= w; k++)
        if (a.wlist[3 * q + k] == 0) jv = cy.topv;
      const float3 cpv = (f3(vi4.x, vi4.y, vi4.z) - f3(0.f, 0.f, (float)jv)) - crossf(f3(wi4.x, wi4.y, wi4.z) * ri, u);
      ContactRec* rp = a.wrec + (long long)w * a.n + q;
      MixedRec rc = load_rec(rp);
      float fN, fD;
      float3 fT;
      law32_forces(a.pw, ri, -gapw, u, cpv, rc, a.dtf, fN, fD, fT);
      store_rec(rp, rc);
      const float3 F = (fN + fD) * u + fT, M = crossf(u * (-(ri - -gapw * 0.5f)), fT);
      f = make_float4(F.x, F.y, F.z, fN);
      t = make_float4(M.x, M.y, M.z, -gapw);
    }
  }
  a.wall_out[2 * (size_t)e] = f;
  a.wall_out[2 * (size_t)e + 1] = t;
}

/* resident blocks per SM the pair kernel is built for: 10 (48 registers, no
 * spills) 60.9 us a step on the packed 200k bed, 9 62.1, 8 62.8; 2M spheres 573,
 * 585, 598 us (there it moves 1.42 GB in 267 us, 78 % of the copy rate) */
#ifndef DEM_PAIR_BLOCKS
#define DEM_PAIR_BLOCKS 10
#endif

/* One thread per pair of the list: overlap, contact law, capillary bridge, the
 * pair's history.  What it leaves for the two spheres (k_body_mixed) is what
 * each would have computed for itself, in pieces that are the same for both
 * but for their sign: the normal u and the overlap (0: no contact; the sign bit
 * says that a bridge acts), the friction fT and the normal force with damping,
 * and, where a bridge acts or the material rolls, fN and the bridge's force:
 * u c_i and u c_j for the two spheres (formula), or u c_i times the network's
 * output, d for the first sphere and c_j for the second.  Which of the two is
 * the sign bit of fN, which is never negative: the outputs take any value.
 * Without rolling and network only c_i and c_j are left: 8 bytes a pair. */
template <bool WET, bool NET>
__global__ void __launch_bounds__(128, NET ? kNetBlocks : DEM_PAIR_BLOCKS) k_pair_mixed(const __grid_constant__ MixArgs a) {
  const int4 ct = pair_ctl(a.ps);
  if (a.gate && *a.gate) return;
  if (blockIdx.x < a.wall_blocks) { /* the first blocks take the wall list */
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < ct.w; k += a.wall_blocks * blockDim.x)
      wall_entry(a, a.wall_entry[k]);
    return;
  }
  extern __shared__ __align__(16) unsigned char dsm[];
  const CapNetSmem* capw = reinterpret_cast<const CapNetSmem*>(dsm);
  CapEntry* qw = reinterpret_cast<CapEntry*>(dsm + ((sizeof(CapNetSmem) + 15) / 16) * 16) + (threadIdx.x >> 5) * 32;
  const int P = ct.x ? ct.z : ct.y;
  const int2* __restrict__ pair = ct.x ? a.ps.pair[1] : a.ps.pair[0];
  float4* const rec = reinterpret_cast<float4*>(ct.x ? a.ps.rec[1] : a.ps.rec[0]);
  unsigned char* const brg = ct.x ? a.ps.brg[1] : a.ps.brg[0];
  if (NET) {
    cap_stage(a.capw, reinterpret_cast<CapNetSmem*>(dsm));
    __syncthreads();
  }
  unsigned nmlp = 0, nfall = 0;
  const int lane = threadIdx.x & 31;
  const int step = (gridDim.x - a.wall_blocks) * blockDim.x;
  const int first = (blockIdx.x - a.wall_blocks) * blockDim.x + threadIdx.x;
  /* NET: whole warps go round together */
  const int last = NET ? (P + 31) / 32 * 32 : P;
  for (int p = first; p < last; p += step) {
    const bool act = !NET || p < P;
    bool want = false; /* NET: this lane's bridge goes to the network */
    bool form = false, wet = false;
    int bprev = 0;
    float gap = 0.f, fN = 0.f, nrm = 0.f, s_n = 0.f, ci = 0.f, cj = 0.f, d = 0.f;
    float3 fT = f3(0.f, 0.f, 0.f), u = f3(0.f, 0.f, 0.f);
    CapEntry ent, ent_j;
    bool want_j = false;
    if (act) {
      const int2 ij = ro(pair + p);
      const int i = ij.x, j = ij.y;
      float4 hi, lo, hj, lj;
      get2(a.place_in + 2 * i, hi, lo);
      get2(a.place_in + 2 * j, hj, lj);
      float4 vi, vj, wi, wj;
      get2(a.motion_in + 2 * i, vi, wi);
      get2(a.motion_in + 2 * j, vj, wj);
      if (WET) bprev = brg[p];
      const float ax = hi.x - hj.x, ay = hi.y - hj.y, az = hi.z - hj.z; /* exact */
      const float ri = hi.w + lo.w;
      float rj;
      gap = exact_gap(hi, lo, hj, lj, ax, ay, az, u, rj);
      if (gap < 0.f) {
        MixedRec rc = load_pair_rec(rec, a.ps.cap, p);
        const float3 cpv = f3(vi.x - vj.x, vi.y - vj.y, vi.z - vj.z) -
                           crossf(f3(wi.x, wi.y, wi.z) * ri + f3(wj.x, wj.y, wj.z) * rj, u);
        float fD;
        nrm = -gap;
        law32_forces(a.pp, ri * rj / (ri + rj), nrm, u, cpv, rc, a.dtf, fN, fD, fT);
        store_pair_rec(rec, a.ps.cap, p, rc);
        s_n = fN + fD;
      }
      if (WET && (!a.sys_wet || a.sys_wet[a.sys_of_id[ro(a.id + i)]])) {
        form = gap < 2.0f * a.lqd_layer * (ri + rj);
        if (form || bprev) {
          /* the pair's bridge volume and contact angle: the reference's split of
           * both spheres' liquid, or the per-contact model's.  Each sphere adds
           * the partner's share (and angle) to its own, rounded first: vol_j and
           * th_j are what the second sphere gets, mostly the same bits. */
          float vol, vol_j, th_i = 0.f, th_j = 0.f;
          int id_i = 0, id_j = 0;
          if (NET || a.lq_mode) {
            id_i = ro(a.id + i);
            id_j = ro(a.id + j);
            /* the mean contact angle, the own angle rounded first */
            const float tm = a.lq_mode ? a.lq_theta_max : a.theta_max;
            const float xi = a.lq_mode ? cap_theta32(id_i, a.lq_seed, 1.0f) : cap_theta(id_i, a.theta_seed, 1.0f);
            const float xj = a.lq_mode ? cap_theta32(id_j, a.lq_seed, 1.0f) : cap_theta(id_j, a.theta_seed, 1.0f);
            th_i = 0.5f * fmaf(tm, xj, __fmul_rn(tm, xi));
            th_j = 0.5f * fmaf(tm, xi, __fmul_rn(tm, xj));
          }
          if (a.lq_mode == 0) {
            const int inl = max(__float_as_int(vi.w), 12), jnl = max(__float_as_int(vj.w), 12);
            const float ti = 2.0f * ri, tj = 2.0f * rj;
            const float mi = ti * ti * ti, mj = tj * tj * tj;
            const float qi = __fdividef(1.0f, (float)inl), qj = __fdividef(1.0f, (float)jnl);
            const float xi = a.lqd_vol * mi, xj = a.lqd_vol * mj;
            vol = fmaf(xj, qj, __fmul_rn(xi, qi));
            vol_j = fmaf(xi, qi, __fmul_rn(xj, qj));
          } else {
            vol = vol_j = pair_bridge_volume32(id_i, id_j, a.lq_seed, a.lq_vmin, a.lq_vspan, fminf(ri, rj));
          }
          const float lq_th_i = a.lq_mode ? th_i : 0.f, lq_th_j = a.lq_mode ? th_j : 0.f;
          const float effR = 2.0f * ri * rj / (ri + rj);
          if (NET) {
            ent = CapEntry{fmaxf(a.lqd_gapmn, fmaxf(gap, 0.f)), 8.0f * vol, th_i,
                           __fdividef(fminf(ri, rj), fmaxf(ri, rj))};
            want = cap_in_hull(*capw, ent.sep, ent.vol, ent.theta, ent.ratio);
            /* the second sphere's features, where their BF16 roundings differ */
            ent_j = ent;
            ent_j.vol = 8.0f * vol_j;
            ent_j.theta = th_j;
            want_j = want && (cap_pair(*capw, ent, 0) != cap_pair(*capw, ent_j, 0) ||
                              cap_pair(*capw, ent, 1) != cap_pair(*capw, ent_j, 1));
          }
          if (!NET || !want) {
            const int b = form ? 1 : (gap > bridge_rupture32(a, vol, lq_th_i) ? 0 : 1);
            if (b != bprev) brg[p] = (unsigned char)b;
            if (b) {
              const float sep = gap < 0.f ? 0.f : gap;
              ci = -bridge_force32(a, sep, vol, lq_th_i, effR);
              cj = vol_j == vol && lq_th_j == lq_th_i ? ci : -bridge_force32(a, sep, vol_j, lq_th_j, effR);
              wet = true;
            }
            if (NET) nfall++;
          } else {
            ci = -2.0f * kPiF * effR * a.lqd_st;
          }
        }
      }
    }
    if (NET) {
      const unsigned m = __ballot_sync(0xffffffffu, want);
      const unsigned mj = __ballot_sync(0xffffffffu, want_j);
      const unsigned below = (1u << lane) - 1u;
      const int at = __popc(m & below);
      if (want) qw[at] = ent;
      if (m) cap_run_queue(*capw, qw, __popc(m));
      if (want) {
        d = cj = qw[at].sep;
        const int b = form ? 1 : (gap > qw[at].vol ? 0 : 1);
        if (b != bprev) brg[p] = (unsigned char)b;
        wet = b != 0;
        nmlp++;
      }
      if (mj) {
        __syncwarp();
        const int atj = __popc(mj & below);
        if (want_j) qw[atj] = ent_j;
        cap_run_queue(*capw, qw, __popc(mj));
        if (want_j) cj = qw[atj].sep;
      }
      __syncwarp(); /* the queue is read before the next round fills it */
    }
    if (act) {
      float4* o = a.pair_out + 2 * (size_t)p;
      put2(o, make_float4(u.x, u.y, u.z, __uint_as_float(__float_as_uint(nrm) | (wet ? 0x80000000u : 0u))),
           make_float4(fT.x, fT.y, fT.z, s_n));
      float4* more = a.pair_out + 2 * (size_t)a.ps.cap;
      if (NET || a.rfrc != 0.f) {
        if (wet || nrm > 0.f)
          more[p] = make_float4(__uint_as_float(__float_as_uint(fN) | (want ? 0x80000000u : 0u)), ci, cj, d);
      } else if (wet) {
        reinterpret_cast<float2*>(more)[p] = make_float2(ci, cj);
      }
    }
  }
  if (NET && a.counters) {
    /* counted once per sphere, as every sphere feels its bridges */
    warp_add(&a.counters[5], 2u * nmlp);
    warp_add(&a.counters[6], 2u * nfall);
  }
}

/* resident blocks per SM the sphere kernel is built for, and the pair results
 * a sphere has in flight: 6 and 3, 62.1 us a step on the packed 200k bed and 585
 * on 2M spheres; 2 in flight 62.8 and 610, 5 blocks with 4 67.0 and 588 (7 with 2 and
 * 8 with 1 were 3 % slower still).  The indexes of the next results are read while
 * the present ones are on their way (690 to 664 us on 2M spheres when this came
 * in).  On 2M spheres it moves 1.49 GB in 288 us, 76 % of the copy rate. */
#ifndef DEM_BODY_BLOCKS
#define DEM_BODY_BLOCKS 6
#endif
#ifndef DEM_BODY_BATCH
#define DEM_BODY_BATCH 3
#endif
constexpr int kBodyBatch = DEM_BODY_BATCH, kNetBatch = 2;

/* a pair's vector as the slot's sphere sees it: the second sphere's (e < 0)
 * points the other way.  Sign bits, not a product, so that no contraction
 * touches it. */
__device__ __forceinline__ float3 turned(float4 v, int e) {
  const unsigned m = (unsigned)e & 0x80000000u;
  return f3(__uint_as_float(__float_as_uint(v.x) ^ m), __uint_as_float(__float_as_uint(v.y) ^ m),
            __uint_as_float(__float_as_uint(v.z) ^ m));
}

/* the network's bridges of a warp's spheres that wait to be added: direction
 * times reach, the network's output, and the same sphere's entry before */
constexpr int kCapQ = 128;
struct NetQueue {
  float4 f[kCapQ];
  short before[kCapQ];
};

/* One thread per sphere: gravity, its pairs' results summed in neighbour order
 * with Kahan compensation, the <= 3 cylinder-wall contacts (CirPWInterG,
 * kernel.cu:958-1023), the integrator (UpdateSystemG, kernel.cu:563-606), the
 * next step's shadows and the counters. */
template <bool WET, bool NET>
__global__ void __launch_bounds__(128, DEM_BODY_BLOCKS) k_body_mixed(MixArgs a) {
  if (a.gate && *a.gate) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.flag = -1; /* held back (chain.cu) */
    return;
  }
  const int q = a.body_order ? ro(a.body_order + blockIdx.x) * blockDim.x + threadIdx.x
                             : reversed_block_thread(); /* the spheres with the most pairs first */
  const bool live = q < a.n;
  const int qq = live ? q : a.n - 1;
  __shared__ unsigned sums[5];
  if (threadIdx.x < 5) sums[threadIdx.x] = 0u;
  __syncthreads();
  /* the integrator's FP64 state and the wall count are needed only after the
   * pairs: start bringing them in now */
  prefetch_l2(a.pos + qq);
  prefetch_l2(a.vel + qq);
  prefetch_l2(a.angv + qq);
  prefetch_l2(a.pmove + qq);
  prefetch_l2(a.nwall + qq);
  const int L = ro(a.plevel + qq);
  const int nn = live ? ro(a.num_nebor + qq) : 0;
  const long long stride = ro(a.npars + L);
  const long long base = slot_base(L, a.npars, a.nneb) + ro(a.nidx + qq);
  const float4 wi4 = ro(a.motion_in + 2 * qq + 1);
  float4 hi, lo;
  get2(a.place_in + 2 * qq, hi, lo);
  const float ri = hi.w + lo.w, twor = 2.0f * ri;
  const float mass_f = __fmul_rn(__fmul_rn(twor, twor), twor);
  KSum3 F, M;
  KSum R;
  F.z.add(-mass_f); /* gravity, m = (2r)^3 */
  int wet = 0;
  unsigned ncont = 0, nbr = 0;
  if (NET) {
    /* The network's bridges join the sum a warp's queue at a time, the newest
     * first, once more than kCapQ - 32 wait: the order in which a kernel that
     * queues them while it walks the slots adds them.  A sphere's entries are
     * chained (read again from the results: 127.5 us a step, so 118). */
    __shared__ NetQueue waiting[NET ? 4 : 1];
    NetQueue& wq = waiting[NET ? threadIdx.x >> 5 : 0];
    const unsigned below = (1u << (threadIdx.x & 31)) - 1u;
    const int nloop = __reduce_max_sync(0xffffffffu, nn);
    int queued = 0, last = -1; /* this sphere's newest entry */
    auto flush = [&]() {
      for (; last >= 0; last = wq.before[last]) {
        const float4 v = wq.f[last];
        F.add(f3(v.x, v.y, v.z) * v.w);
      }
      queued = 0;
      __syncwarp(); /* read before the next entries overwrite them */
    };
    int en[kNetBatch];
#pragma unroll
    for (int t = 0; t < kNetBatch; t++) en[t] = t < nn ? ro(a.ps.eidx + base + (long long)t * stride) : kNoPair;
    for (int k0 = 0; k0 < nloop; k0 += kNetBatch) {
      int e[kNetBatch];
      float4 nu[kNetBatch], ft[kNetBatch], br[kNetBatch];
#pragma unroll
      for (int t = 0; t < kNetBatch; t++) {
        e[t] = en[t];
        nu[t] = make_float4(0.f, 0.f, 0.f, 0.f);
        ft[t] = br[t] = nu[t];
        if (e[t] != kNoPair) {
          const int p = e[t] < 0 ? ~e[t] : e[t];
          get2(a.pair_out + 2 * (size_t)p, nu[t], ft[t]);
          br[t] = a.pair_out[2 * (size_t)a.ps.cap + p];
        }
      }
#pragma unroll
      for (int t = 0; t < kNetBatch; t++)
        en[t] = k0 + kNetBatch + t < nn ? ro(a.ps.eidx + base + (long long)(k0 + kNetBatch + t) * stride) : kNoPair;
#pragma unroll
      for (int t = 0; t < kNetBatch; t++) {
        const unsigned nb = __float_as_uint(nu[t].w);
        const float nrm = fabsf(nu[t].w);
        const float3 u = turned(nu[t], e[t]);
        bool net = false;
        if (nrm > 0.f) {
          const float3 fT = turned(ft[t], e[t]);
          F.add(ft[t].w * u + fT);
          const float arm = ri - nrm * 0.5f;
          M.add(crossf(u * (-arm), fT));
          if (a.rfrc != 0.f) R.add(0.5f * (a.rfrc + a.rfrc) * fabsf(br[t].x) * ri);
          ncont++;
        }
        if (nb >> 31) {
          net = __float_as_uint(br[t].x) >> 31 != 0u; /* the network's, not the formula's */
          if (!net) F.add(u * (e[t] < 0 ? br[t].z : br[t].y));
          wet++;
          if (!(nrm > 0.f)) nbr++;
        }
        const unsigned m = __ballot_sync(0xffffffffu, net);
        if (net) {
          const int at = queued + __popc(m & below);
          const float3 v = u * br[t].y;
          wq.f[at] = make_float4(v.x, v.y, v.z, e[t] < 0 ? br[t].z : br[t].w);
          wq.before[at] = (short)last;
          last = at;
        }
        queued += __popc(m);
        if (queued > kCapQ - 32) flush();
      }
    }
    flush();
  }
  int en[kBodyBatch];
#pragma unroll
  for (int t = 0; !NET && t < kBodyBatch; t++) en[t] = t < nn ? ro(a.ps.eidx + base + (long long)t * stride) : kNoPair;
  for (int k0 = 0; !NET && k0 < nn; k0 += kBodyBatch) {
    int e[kBodyBatch];
    float4 nu[kBodyBatch], ft[kBodyBatch], br[kBodyBatch];
#pragma unroll
    for (int t = 0; t < kBodyBatch; t++)
      e[t] = en[t];
#pragma unroll
    for (int t = 0; t < kBodyBatch; t++) {
      nu[t] = make_float4(0.f, 0.f, 0.f, 0.f);
      ft[t] = br[t] = nu[t];
      if (e[t] != kNoPair) {
        const int p = e[t] < 0 ? ~e[t] : e[t];
        get2(a.pair_out + 2 * (size_t)p, nu[t], ft[t]);
        const float4* more = a.pair_out + 2 * (size_t)a.ps.cap;
        if (a.rfrc != 0.f) {
          br[t] = more[p];
        } else if (WET) {
          const float2 c = reinterpret_cast<const float2*>(more)[p];
          br[t].y = c.x;
          br[t].z = c.y;
        }
      }
    }
#pragma unroll
    for (int t = 0; t < kBodyBatch; t++)
      en[t] = k0 + kBodyBatch + t < nn ? ro(a.ps.eidx + base + (long long)(k0 + kBodyBatch + t) * stride) : kNoPair;
#pragma unroll
    for (int t = 0; t < kBodyBatch; t++) {
      const unsigned nb = __float_as_uint(nu[t].w);
      if (nb == 0u) continue; /* neither contact nor bridge (or no pair) */
      const float nrm = fabsf(nu[t].w);
      const float3 u = turned(nu[t], e[t]);
      if (nrm > 0.f) {
        const float3 fT = turned(ft[t], e[t]);
        F.add(ft[t].w * u + fT);
        const float arm = ri - nrm * 0.5f;
        M.add(crossf(u * (-arm), fT));
        if (a.rfrc != 0.f) R.add(0.5f * (a.rfrc + a.rfrc) * br[t].x * ri);
        ncont++;
      }
      if (WET && (nb >> 31)) {
        F.add(u * (e[t] < 0 ? br[t].z : br[t].y));
        wet++;
        if (!(nrm > 0.f)) nbr++;
      }
    }
  }
  unsigned nwc = 0;
  const int nw = live ? a.nwall[qq] : 0;
  for (int w = 0; w < nw; w++) {
    const float4* r = a.wall_out + 2 * ((size_t)w * a.n + qq);
    const float4 t = r[1], f = r[0];
    if (!(t.w > 0.f)) continue;
    F.add(f3(f.x, f.y, f.z));
    M.add(f3(t.x, t.y, t.z));
    R.add(0.5f * (a.rfrc + a.rfrc) * f.w * ri);
    nwc++;
  }

  /* integrator (UpdateSystemG) in FP64 with FP32 increments */
  bool flagged = false;
  if (live) {
    /* 13 FP64 operations per particle: v += dv (3), x += v dt (3), path
     * length (1), spin (3), binade shift of the shadow (3); every conversion
     * goes through the integer pipe */
    const float fx = F.x.s - F.x.c, fy = F.y.s - F.y.c, fz = F.z.s - F.z.c;
    const float inv_m = a.dtf / mass_f;
    double3 p = a.pos[q], v = a.vel[q];
    v.x += f2d(fx * inv_m);
    v.y += f2d(fy * inv_m);
    v.z += f2d(fz * inv_m);
    p.x = fma(v.x, a.dt, p.x);
    p.y = fma(v.y, a.dt, p.y);
    p.z = fma(v.z, a.dt, p.z);
    const float vxf = d2f(v.x), vyf = d2f(v.y), vzf = d2f(v.z);
    const double pm = a.pmove[q] + f2d(sqrtf(vxf * vxf + vyf * vyf + vzf * vzf) * a.dtf);
    const float inert = 0.1f * mass_f * twor * twor;
    const float inv_i = a.dtf / inert;
    double3 w = a.angv[q];
    /* spin: w += M dt / I, then the rolling-resistance damping
     * w *= 1 - min(1, Mr dt / I / |w|), folded into one increment */
    const float dwx = (M.x.s - M.x.c) * inv_i, dwy = (M.y.s - M.y.c) * inv_i, dwz = (M.z.s - M.z.c) * inv_i;
    const float rm = (R.s - R.c) * inv_i;
    const float wx1 = wi4.x + dwx, wy1 = wi4.y + dwy, wz1 = wi4.z + dwz;
    const float wl = sqrtf(wx1 * wx1 + wy1 * wy1 + wz1 * wz1);
    float ix = dwx, iy = dwy, iz = dwz;
    if (wl > 1.0e-7f) {
      const float f = fminf(1.0f, rm / wl);
      ix -= wx1 * f;
      iy -= wy1 * f;
      iz -= wz1 * f;
    }
    w.x += f2d(ix);
    w.y += f2d(iy);
    w.z += f2d(iz);
    a.vel[q] = v;
    a.pos[q] = p;
    a.angv[q] = w;
    a.pmove[q] = pm;
    flagged = pm > a.move_limit;
    if (!(isfinite(fx) && isfinite(fy) && isfinite(fz))) atomicOr(a.err, 2);
    /* next step's shadows */
    float4 ph, pl;
    split_hi_lo(p.x + a.off.x, a.bin_exp, a.lo_scale, ph.x, pl.x);
    split_hi_lo(p.y + a.off.y, a.bin_exp, a.lo_scale, ph.y, pl.y);
    split_hi_lo(p.z + a.off.z, a.bin_exp, a.lo_scale, ph.z, pl.z);
    ph.w = hi.w;
    pl.w = lo.w;
    put2(a.place_out + 2 * q, ph, pl);
    put2(a.motion_out + 2 * q, make_float4(vxf, vyf, vzf, __int_as_float(wet)),
         make_float4(d2f(w.x), d2f(w.y), d2f(w.z), 0.f));
    a.force_out[q] = make_float4(fx, fy, fz, 0.f);
  }
  const unsigned fm = __ballot_sync(0xffffffffu, flagged);
  if ((threadIdx.x & 31) == 0 && fm) atomicAdd(a.flag, __popc(fm));
  if (a.counters) {
    /* a block's counts go out together, by its last warp: an atomic per warp
     * on four words of one sector would queue up behind one another, and a
     * barrier would hold the finished warps' places */
    const unsigned c[4] = {(unsigned)nn, ncont, nbr, nwc};
    unsigned mine = 0;
#pragma unroll
    for (int t = 0; t < 4; t++) {
      const unsigned v = __reduce_add_sync(0xffffffffu, c[t]);
      if ((threadIdx.x & 31) == t) mine = v;
    }
    if ((threadIdx.x & 31) < 4) atomicAdd(&sums[threadIdx.x & 31], mine);
    __threadfence_block();
    __syncwarp();
    unsigned done = 0;
    if ((threadIdx.x & 31) == 0) done = atomicAdd(&sums[4], 1u);
    done = __shfl_sync(0xffffffffu, done, 0);
    if (done == blockDim.x / 32 - 1 && (threadIdx.x & 31) < 4) {
      const unsigned v = atomicAdd(&sums[threadIdx.x & 31], 0u);
      if (v) atomicAdd(&a.counters[threadIdx.x & 31], (unsigned long long)v);
    }
  }
}

/* the listed wall slots, compact (their order does not matter: each writes its
 * own slot's result) */
__global__ void k_wall_entries(const int* __restrict__ nwall, int n, int* __restrict__ entry, int* __restrict__ count) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  const int nw = q < n ? nwall[q] : 0;
  const int lane = threadIdx.x & 31;
  int incl = nw;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  const int total = __shfl_sync(0xffffffffu, incl, 31);
  if (total == 0) return;
  int at = 0;
  if (lane == 0) at = atomicAdd(count, total);
  at = __shfl_sync(0xffffffffu, at, 0) + incl - nw;
  for (int w = 0; w < nw; w++) entry[at + w] = w * n + q;
}

/* CirPWInterG's wall motion (kernel.cu:966-969): every cylinder's top wall
 * moves by topv dt before any particle meets it this step (not in a chained
 * step that waits for a rebuild: it moves them when it runs again) */
__global__ void k_move_walls(CylinderBC* cyl, int n_cyl, double dt, const int* gate) {
  if (gate && *gate) return;
  for (int k = threadIdx.x; k < n_cyl; k += blockDim.x) cyl[k].Tw = cyl[k].Tw + cyl[k].topv * dt;
}

__global__ void k_shadows(int n, const double3* __restrict__ pos, const double3* __restrict__ vel,
                          const double3* __restrict__ angv, const double* __restrict__ rad, const int* __restrict__ lqd,
                          ShadowOut sh) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < n) write_shadow(sh, q, pos[q], vel[q], angv[q], rad[q], lqd[q]);
}

/* A state import without a rebuild in one pass: the caller-order arrays
 * gathered into cell order (k_import), the bridge counts of the last step
 * taken from the shadow (k_lqd_from_shadow) and the shadow rewritten from the
 * new state (k_shadows) -- the same values as those three launches */
__global__ void k_import_shadows(int n, const int* __restrict__ id, const double3* __restrict__ hp,
                                 const double3* __restrict__ hv, const double3* __restrict__ hw, int has_v, int has_w,
                                 double3* __restrict__ pos, double3* __restrict__ vel, double3* __restrict__ angv,
                                 const double* __restrict__ rad, int* __restrict__ lqd, ShadowOut sh) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const int i = id[q];
  const double3 p = hp[i];
  const double3 v = has_v ? hv[i] : make_double3(0.0, 0.0, 0.0);
  const double3 w = has_w ? hw[i] : make_double3(0.0, 0.0, 0.0);
  pos[q] = p;
  vel[q] = v;
  angv[q] = w;
  const int lq = __float_as_int(sh.motion[2 * q].w);
  lqd[q] = lq;
  write_shadow(sh, q, p, v, w, rad[q], lq);
}

/* the same import from mapped host arrays read in caller order.  A block
 * walks slices of kImportThreads particles (slice, slice + gridDim.x, ...):
 * the caller's three arrays of a slice are read over the host link into
 * registers, staged in shared memory, and each thread scatters its particle
 * to cell position inv[i] (state, bridge count and shadows) -- while the next
 * slice's reads are already in flight, so the link stays busy during the
 * scatter.  16-byte reads where a slice starts 16-byte aligned (a slice of
 * 256 double3 is 6144 bytes, so all slices share the array's alignment),
 * else 8-byte reads. */
constexpr int kImportThreads = 256;
constexpr int kSliceDoubles = 3 * kImportThreads;
/* resident import blocks per SM: 4 (or 8) read the 14.4 MB state of the
 * packed 200k bed in 79 us, 2 in 84 us; one slice per block (the whole grid
 * in one wave, reads then scatters) took 89 us */
#ifndef DEM_IMPORT_BLOCKS
#define DEM_IMPORT_BLOCKS 4
#endif
constexpr int kImportBlocksPerSM = DEM_IMPORT_BLOCKS;

/* this thread's part of one slice of one array: doubles [2t, 2t+1] and
 * [2(t+256), 2(t+256)+1] (aligned), or t, t+256, t+512 (unaligned) */
struct SliceRegs {
  double2 a, b;
};

__device__ __forceinline__ void slice_fetch(const double3* __restrict__ h, int n, long long slice, bool al,
                                            SliceRegs& r) {
  const long long i0 = slice * kImportThreads;
  const int nd = 3 * (int)min((long long)kImportThreads, n - i0);
  const double* src = reinterpret_cast<const double*>(h + i0);
  const int t = threadIdx.x;
  if (al) {
    const int e0 = 2 * t, e1 = 2 * (t + kImportThreads);
    r.a = e0 + 1 < nd ? *reinterpret_cast<const double2*>(src + e0)
                      : make_double2(e0 < nd ? src[e0] : 0.0, 0.0);
    r.b = e1 + 1 < nd ? *reinterpret_cast<const double2*>(src + e1)
                      : make_double2(e1 < nd ? src[e1] : 0.0, 0.0);
  } else {
    r.a.x = t < nd ? src[t] : 0.0;
    r.a.y = t + kImportThreads < nd ? src[t + kImportThreads] : 0.0;
    r.b.x = t + 2 * kImportThreads < nd ? src[t + 2 * kImportThreads] : 0.0;
    r.b.y = 0.0;
  }
}

__device__ __forceinline__ void slice_put(const SliceRegs& r, bool al, double* sm) {
  const int t = threadIdx.x;
  if (al) {
    const int e0 = 2 * t, e1 = 2 * (t + kImportThreads);
    sm[e0] = r.a.x;
    sm[e0 + 1] = r.a.y;
    if (e1 < kSliceDoubles) {
      sm[e1] = r.b.x;
      sm[e1 + 1] = r.b.y;
    }
  } else {
    sm[t] = r.a.x;
    sm[t + kImportThreads] = r.a.y;
    sm[t + 2 * kImportThreads] = r.b.x;
  }
}

__global__ void __launch_bounds__(kImportThreads) k_import_shadows_mapped(
    int n, const int* __restrict__ inv, const double3* __restrict__ hp, const double3* __restrict__ hv,
    const double3* __restrict__ hw, double3* __restrict__ pos, double3* __restrict__ vel, double3* __restrict__ angv,
    const double* __restrict__ rad, int* __restrict__ lqd, ShadowOut sh) {
  __shared__ double sp[kSliceDoubles], sv[kSliceDoubles], sw[kSliceDoubles];
  const long long nsl = ((long long)n + kImportThreads - 1) / kImportThreads;
  const bool ap = (reinterpret_cast<size_t>(hp) & 15) == 0;
  const bool av = hv && (reinterpret_cast<size_t>(hv) & 15) == 0;
  const bool aw = hw && (reinterpret_cast<size_t>(hw) & 15) == 0;
  SliceRegs rp{}, rv{}, rw{};
  long long slice = blockIdx.x;
  if (slice < nsl) {
    slice_fetch(hp, n, slice, ap, rp);
    if (hv) slice_fetch(hv, n, slice, av, rv);
    if (hw) slice_fetch(hw, n, slice, aw, rw);
  }
  for (; slice < nsl; slice += gridDim.x) {
    slice_put(rp, ap, sp);
    if (hv) slice_put(rv, av, sv);
    if (hw) slice_put(rw, aw, sw);
    __syncthreads();
    const long long next = slice + gridDim.x;
    if (next < nsl) {
      slice_fetch(hp, n, next, ap, rp);
      if (hv) slice_fetch(hv, n, next, av, rv);
      if (hw) slice_fetch(hw, n, next, aw, rw);
    }
    const long long ii = slice * kImportThreads + threadIdx.x;
    if (ii < n) {
      const int i = (int)ii;
      const int t3 = 3 * threadIdx.x;
      const int q = inv[i];
      const double3 p = make_double3(sp[t3], sp[t3 + 1], sp[t3 + 2]);
      const double3 v = hv ? make_double3(sv[t3], sv[t3 + 1], sv[t3 + 2]) : make_double3(0.0, 0.0, 0.0);
      const double3 w = hw ? make_double3(sw[t3], sw[t3 + 1], sw[t3 + 2]) : make_double3(0.0, 0.0, 0.0);
      pos[q] = p;
      vel[q] = v;
      angv[q] = w;
      const int lq = __float_as_int(sh.motion[2 * q].w);
      lqd[q] = lq;
      write_shadow(sh, q, p, v, w, rad[q], lq);
    }
    __syncthreads();
  }
}

__global__ void k_force_out(int n, const float4* __restrict__ f, double3* __restrict__ force, double3* __restrict__ mom) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const float4 v = f[q];
  force[q] = make_double3(v.x, v.y, v.z);
  mom[q] = make_double3(0.0, 0.0, 0.0);
}

__global__ void k_lqd_from_shadow(int n, const float4* __restrict__ vs, int* __restrict__ lqd) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  lqd[q] = __float_as_int(vs[2 * q].w);
}

Law32 make_law(const calParaPP& c, bool pp, double dmp_sq, int stage) {
  Law32 l;
  l.emod = (float)c.emod;
  l.pois = (float)c.pois;
  l.sfrc = (float)c.sfrc;
  l.ydsp = (float)c.ydsp_t;
  l.yforce = (float)c.yforce_t;
  l.ystiff = (float)c.ystiff_t;
  l.rot_eps = pp ? 1.0e-7f : 1.0e-10f;
  l.dsmx_eps = pp ? 1.0e-7f : 1.0e-10f;
  l.kt = (float)(16.0 * (1.0 - c.pois) * c.emod / (4.0 - 2.0 * c.pois));
  l.dmp = (float)std::sqrt(dmp_sq);
  l.hertz_le = pp ? 1 : 0;
  l.damp_on = pp ? (stage == 1) : (stage == 1 || stage == 7);
  return l;
}


/* ---- the reference's entry points in mixed precision ----
 * PpInterCalc and CirPWCalc (kernel.cu:413-552, :958-1023) on the reference's
 * own layouts -- spheres in the caller's order, level/slot-major lists, FP64
 * SoA histories -- with the fused step's FP32 laws: a pair's overlap from the
 * FP64 positions as (d^2 - S^2) / (d + S) with d^2 - S^2 in FP64 (eight FP64
 * operations, no FP64 square root, division or pow), the contact law and
 * the bridge in FP32, the sums in Kahan FP32 added to the FP64 force arrays.
 * The histories keep the spring and the peak overlap in FP64, as the fused
 * step does; the re-derived fields are written back as FP64 copies of FP32
 * values. */
struct RefArrays {
  const double3 *pos, *vel, *angv;
  const double* rad;
  const int *nebor, *plevel, *npars, *nneb, *nidx, *num_nebor, *lqd_old;
  int* lqd;
  HistSoA h;
  double3 *force, *mom;
  double* rmom;
  /* walls */
  const CylinderBC* cyl;
  const int *nwall, *wlist;
  size_t pitch;
  int np;
};

__device__ __forceinline__ float3 d2f3(double3 v) { return f3(d2f(v.x), d2f(v.y), d2f(v.z)); }

__device__ __forceinline__ MixedRec soa_load(const HistSoA& h, long long s) {
  MixedRec r;
  const double3 d = h.dispt[s];
  r.dx = d.x;
  r.dy = d.y;
  r.dz = d.z;
  r.nDsp_mx = h.nDsp_mx[s];
  r.fx = d2f(d.x);
  r.fy = d2f(d.y);
  r.fz = d2f(d.z);
  r.nDsp = d2f(h.nDsp[s]);
  r.plstRad = d2f(h.plstRad[s]);
  r.plstDfm = d2f(h.plstDfm[s]);
  r.stage = h.stage[s];
  r.pad = 0;
  return r;
}
__device__ __forceinline__ void soa_store(const HistSoA& h, long long s, const MixedRec& r) {
  h.dispt[s] = make_double3(r.dx, r.dy, r.dz);
  h.nDsp_mx[s] = r.nDsp_mx;
  h.nDsp[s] = f2d(r.nDsp);
  h.plstRad[s] = f2d(r.plstRad);
  h.plstDfm[s] = f2d(r.plstDfm);
  h.stage[s] = r.stage;
}

/* adds sums to an FP64 triple */
__device__ __forceinline__ double3 add_sum(double3 v, const KSum3& s) {
  return make_double3(v.x + f2d(s.x.s - s.x.c), v.y + f2d(s.y.s - s.y.c), v.z + f2d(s.z.s - s.z.c));
}

/* A sphere as its partners read it: position and radius in one 32-byte sector,
 * velocity, spin (FP32) and bridge count in the next, where the caller's five
 * arrays are seven sectors a partner */
struct __align__(32) RefBody {
  double x, y, z, r;
  float vx, vy, vz, wx;
  float wy, wz;
  int nl, pad;
};
static_assert(sizeof(RefBody) == 64, "two sectors a sphere");
constexpr size_t kRefBody = sizeof(RefBody);

__device__ __forceinline__ RefBody ref_body(const RefArrays& r, int i, bool wet) {
  const double3 p = r.pos[i], v = r.vel[i], w = r.angv[i];
  RefBody b;
  b.x = p.x;
  b.y = p.y;
  b.z = p.z;
  b.r = r.rad[i];
  b.vx = d2f(v.x);
  b.vy = d2f(v.y);
  b.vz = d2f(v.z);
  b.wx = d2f(w.x);
  b.wy = d2f(w.y);
  b.wz = d2f(w.z);
  b.nl = wet ? max(r.lqd_old[i], 12) : 12;
  b.pad = 0;
  return b;
}
__global__ void k_ref_bodies(RefArrays r, int n, int wet, RefBody* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = ref_body(r, i, wet != 0);
}
/* sphere i, packed or (no scratch to pack into) from the caller's arrays */
__device__ __forceinline__ RefBody load_body(const RefArrays& r, const RefBody* pk, int i, bool wet) {
  return pk ? pk[i] : ref_body(r, i, wet);
}

/* PPForceCalcG on the reference's layouts.  Bound by latency: a thread per
 * sphere chained index -> partner -> history -> law per slot with 16 of 32
 * lanes at work (249 us cold on the packed wet bed of 200,000).  Now a warp
 * walks its 32 spheres' lists row by row (the caller's arrays are contiguous
 * along a row; the next row's indexes are in flight), keeps the slots that
 * touch or are wet as one dense list, and takes contacts and bridges from it
 * with all lanes; the sums then go by sphere, in slot order, so every result
 * keeps its bits (174 us).  A list of 64 leaves the L1 to the partners' records
 * (96: no better, 128: 25 us slower); 24 warps of 80 registers an SM
 * run the bed in two waves (20: three waves, 28: spills, both slower). */
constexpr int kRefCap = 64, kRefBlocks = 24;
static_assert(kRefCap >= 32 && kRefCap <= 256, "a row has to fit; entries are numbered in a byte");
struct RefWarp {
  float4 u[kRefCap];  /* normal, gap */
  float4 f[kRefCap];  /* tangential force, normal and damping force */
  float n[kRefCap];   /* normal force */
  int j[kRefCap];     /* partner, then the bridge force */
  unsigned row[kRefCap]; /* lanes with an entry, by row */
  unsigned short slot[kRefCap];
  unsigned char owner[kRefCap], flags[kRefCap]; /* flags: 1 touches, 2 forms a bridge, 4 wet, 8 was wet */
  unsigned char contact[kRefCap];
};
__global__ void __launch_bounds__(32, kRefBlocks)
    k_pp_ref_mixed(MixArgs a, RefArrays r, const RefBody* __restrict__ pk) {
  __shared__ RefWarp sm;
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x;
  const unsigned below = (1u << lane) - 1u;
  const int i = reversed_block_thread();
  const bool live = i < a.n;
  const int ii = live ? i : a.n - 1;
  const int first = i - lane;
  const bool wet_on = a.force_cap == 1;
  const int L = r.plevel[ii];
  const int stride = r.npars[L];
  const long long base = slot_base(L, r.npars, r.nneb) + r.nidx[ii];
  const int nn = live ? r.num_nebor[ii] : 0;
  const int rows = __reduce_max_sync(FULL, nn);
  const double3 ip = r.pos[ii];
  const double ird = r.rad[ii];
  const float ri0 = d2f(ird);
  KSum3 F, M;
  KSum R;
  int wet = 0;
  int k = 0;
  int jn, bn; /* the next row */
  auto fetch = [&]() {
    const long long s = base + (long long)k * stride;
    jn = k < nn ? r.nebor[s] : ii;
    bn = wet_on && k < nn ? r.h.lqdBrg[s] : 0;
  };
  fetch();
  while (k < rows) {
    int ne = 0, nc = 0, nr = 0;
    const int kc = k;
    do {
      const int j = jn, bprev = bn;
      const bool in = k < nn;
      double4 q;
      if (pk) {
        q = *reinterpret_cast<const double4*>(pk + j);
      } else {
        const double3 p = r.pos[j];
        q = make_double4(p.x, p.y, p.z, r.rad[j]);
      }
      k++;
      fetch();
      const double dx = ip.x - q.x, dy = ip.y - q.y, dz = ip.z - q.z;
      const double d2 = dx * dx + dy * dy + dz * dz;
      const double S = ird + q.w;
      const double D = d2 - S * S;
      const float dist = sqrtf(d2f(d2));
      const float gap = __fdividef(d2f(D), dist + d2f(S));
      const bool touch = in && (wet_on || D < 0.0) && gap < 0.f;
      const bool form = in && wet_on && gap < 2.0f * a.lqd_layer * (ri0 + d2f(q.w));
      const bool keep = touch || form || bprev != 0;
      const unsigned mk = __ballot_sync(FULL, keep), mc = __ballot_sync(FULL, touch);
      if (keep) {
        const int e = ne + __popc(mk & below);
        const float inv = __frcp_rn(dist);
        sm.u[e] = make_float4(d2f(dx) * inv, d2f(dy) * inv, d2f(dz) * inv, gap);
        sm.j[e] = j;
        sm.slot[e] = (unsigned short)(k - 1 - kc);
        sm.owner[e] = (unsigned char)lane;
        sm.flags[e] = (unsigned char)((touch ? 1 : 0) | (form ? 2 : 0) | (bprev != 0 ? 8 : 0));
        if (touch) sm.contact[nc + __popc(mc & below)] = (unsigned char)e;
      }
      if (mk) {
        if (lane == 0) sm.row[nr] = mk;
        nr++;
      }
      ne += __popc(mk);
      nc += __popc(mc);
    } while (k < rows && ne <= kRefCap - 32 && k - kc < 65535);
    __syncwarp();
    for (int t0 = 0; t0 < nc; t0 += 32) {
      const int t = t0 + lane;
      const int e = sm.contact[min(t, nc - 1)], o = sm.owner[e];
      const long long bo = __shfl_sync(FULL, base, o);
      const int so = __shfl_sync(FULL, stride, o);
      if (t >= nc) continue;
      const long long s = bo + (long long)(kc + sm.slot[e]) * so;
      MixedRec rc = soa_load(r.h, s);
      const RefBody bi = load_body(r, pk, first + o, wet_on), bj = load_body(r, pk, sm.j[e], wet_on);
      const float ri = d2f(bi.r), rj = d2f(bj.r);
      const float4 ug = sm.u[e];
      const float3 u = f3(ug.x, ug.y, ug.z);
      /* the own spin's part rounded first */
      const float3 spin = f3(fmaf(bj.wx, rj, __fmul_rn(bi.wx, ri)), fmaf(bj.wy, rj, __fmul_rn(bi.wy, ri)),
                             fmaf(bj.wz, rj, __fmul_rn(bi.wz, ri)));
      const float3 cpv = (f3(bi.vx, bi.vy, bi.vz) - f3(bj.vx, bj.vy, bj.vz)) -
                         crossf(spin, u);
      float fN, fD;
      float3 fT;
      law32_forces(a.pp, ri * rj / (ri + rj), -ug.w, u, cpv, rc, a.dtf, fN, fD, fT);
      soa_store(r.h, s, rc);
      sm.f[e] = make_float4(fT.x, fT.y, fT.z, fN + fD);
      sm.n[e] = fN;
    }
    __syncwarp();
    if (wet_on)
      for (int t0 = 0; t0 < ne; t0 += 32) {
        const int e = min(t0 + lane, ne - 1), o = sm.owner[e];
        const long long bo = __shfl_sync(FULL, base, o);
        const int so = __shfl_sync(FULL, stride, o);
        if (t0 + lane >= ne) continue;
        const int j = sm.j[e];
        const float ri = d2f(pk ? pk[first + o].r : r.rad[first + o]), rj = d2f(pk ? pk[j].r : r.rad[j]);
        const int nli = pk ? pk[first + o].nl : max(r.lqd_old[first + o], 12);
        const int nlj = pk ? pk[j].nl : max(r.lqd_old[j], 12);
        const float gap = sm.u[e].w;
        const float ti = 2.0f * ri, tj = 2.0f * rj;
        const float qi = __fdividef(1.0f, (float)nli), qj = __fdividef(1.0f, (float)nlj);
        /* the partner's share joins the own one, rounded first */
        const float ijVol = fmaf(a.lqd_vol * (tj * tj * tj), qj, __fmul_rn(a.lqd_vol * (ti * ti * ti), qi));
        const int fl = sm.flags[e], bprev = (fl & 8) ? 1 : 0;
        int b = (fl & 2) ? 1 : bprev;
        if (!(fl & 2) && gap > bridge_rupture32(a, ijVol, 0.f)) b = 0;
        if (b != bprev) r.h.lqdBrg[bo + (long long)(kc + sm.slot[e]) * so] = b;
        if (b == 1) {
          sm.j[e] = __float_as_int(bridge_force32(a, gap < 0.f ? 0.f : gap, ijVol, 0.f, 2.0f * ri * rj / (ri + rj)));
          sm.flags[e] = (unsigned char)(fl | 4);
        }
      }
    __syncwarp();
    int e0 = 0;
    for (int t = 0; t < nr; t++) {
      const unsigned mk = sm.row[t];
      const int e = e0 + __popc(mk & below);
      e0 += __popc(mk);
      if (!((mk >> lane) & 1)) continue;
      const int fl = sm.flags[e];
      const float4 ug = sm.u[e];
      const float3 u = f3(ug.x, ug.y, ug.z);
      if (fl & 1) {
        const float4 f = sm.f[e];
        const float3 fT = f3(f.x, f.y, f.z);
        const float arm = ri0 - -ug.w * 0.5f;
        F.add(f.w * u + fT);
        M.add(crossf(u * (-arm), fT));
        R.add(0.5f * (a.rfrc + a.rfrc) * sm.n[e] * ri0);
      }
      if (fl & 4) {
        F.add(u * (-__int_as_float(sm.j[e])));
        wet++;
      }
    }
    __syncwarp();
  }
  if (!live) return;
  double3 f = add_sum(r.force[i], F);
  const double t = 2.0 * r.rad[i];
  f.z = f.z - t * t * t; /* gravity, m = (2r)^3 */
  r.force[i] = f;
  r.mom[i] = add_sum(r.mom[i], M);
  r.rmom[i] = r.rmom[i] + f2d(R.s - R.c);
  if (wet_on) r.lqd[i] = r.lqd[i] + wet;
}

/* The gap of a wall the sphere certainly does not touch, from FP32 copies of
 * the coordinates: within tol of the exact one (a few FP32 ulps of the largest
 * coordinate involved, taken 8x), so such a wall costs no FP64 work.  Any
 * other kind of wall exerts nothing. */
__device__ __forceinline__ bool wall_apart(const CylinderBC& cy, int kind, float px, float py, float pz, float ri) {
  if (kind == 0 || kind == 1) {
    const float wz = d2f(kind == 0 ? cy.Tw : cy.Bw);
    return fabsf(pz - wz) - ri > 1e-6f * (fabsf(pz) + fabsf(wz) + ri);
  }
  if (kind != 2) return true;
  const float cx = d2f(cy.cir.x), cyy = d2f(cy.cir.y), R = d2f(cy.R);
  const float dx = px - cx, dy = py - cyy;
  return fabsf(sqrtf(dx * dx + dy * dy) - R) - ri >
         1e-6f * (fabsf(px) + fabsf(py) + fabsf(cx) + fabsf(cyy) + R + ri);
}

/* CirPWInterG on the reference's wall lists (row i of pitch bytes) and wall
 * histories (slot a * NP + i); the wall point in FP64 as the fused step
 * takes it, the law in FP32.  The top wall has moved before this launch.
 * Few spheres touch a wall, and those lie together: a block of kRefWallThreads
 * sifts kRefWallEach times as many, 32 at a time from all over the bed, and
 * works on the rest as one dense list (31 us cold on 200,000 spheres; 42 as a
 * thread per sphere, with 3 of 32 lanes in the law). */
constexpr int kRefWallThreads = 128, kRefWallEach = 3;
__global__ void __launch_bounds__(kRefWallThreads) k_wall_ref_mixed(MixArgs a, RefArrays r) {
  __shared__ int list[kRefWallThreads * kRefWallEach];
  __shared__ int listed;
  if (threadIdx.x == 0) listed = 0;
  __syncthreads();
  const CylinderBC cy = *r.cyl;
#pragma unroll
  for (int e = 0; e < kRefWallEach; e++) {
    const int i = ((e * (kRefWallThreads / 32) + (threadIdx.x >> 5)) * gridDim.x + blockIdx.x) * 32 + (threadIdx.x & 31);
    const int nw = i < a.n ? r.nwall[i] : 0;
    if (nw <= 0) continue;
    const double3 p = r.pos[i];
    const float px = d2f(p.x), py = d2f(p.y), pz = d2f(p.z), ri = d2f(r.rad[i]);
    const int* row = reinterpret_cast<const int*>(reinterpret_cast<const char*>(r.wlist) + (size_t)i * r.pitch);
    bool near = false;
    for (int w = 0; w < nw; w++) near = near || !wall_apart(cy, row[w], px, py, pz, ri);
    if (near) list[atomicAdd(&listed, 1)] = i;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < listed; t += kRefWallThreads) {
    const int i = list[t];
    const int nw = r.nwall[i];
    const double3 p = r.pos[i];
    const double rid = r.rad[i];
    const float ri = d2f(rid);
    const float3 iv = d2f3(r.vel[i]), iw = d2f3(r.angv[i]);
    const int* row = reinterpret_cast<const int*>(reinterpret_cast<const char*>(r.wlist) + (size_t)i * r.pitch);
    KSum3 F, M;
    KSum R;
    float3 jv = f3(0.f, 0.f, 0.f); /* persists across walls (kernel.cu:980) */
    const float pxf = d2f(p.x), pyf = d2f(p.y), pzf = d2f(p.z);
    for (int w = 0; w < nw; w++) {
      const int kind = row[w];
      if (kind == 0) jv = f3(0.f, 0.f, d2f(cy.topv));
      if (wall_apart(cy, kind, pxf, pyf, pzf, ri)) continue;
      double3 jp = make_double3(p.x, p.y, kind == 0 ? cy.Tw : cy.Bw);
      if (kind == 2) {
        const double ddx = cy.cir.x - p.x, ddy = cy.cir.y - p.y;
        const double dist = sqrt(ddx * ddx + ddy * ddy);
        jp = make_double3(cy.R * ((p.x - cy.cir.x) / dist) + cy.cir.x, cy.R * ((p.y - cy.cir.y) / dist) + cy.cir.y,
                          p.z);
      }
      const double3 d = make_double3(p.x - jp.x, p.y - jp.y, p.z - jp.z);
      const double len = sqrt(d.x * d.x + d.y * d.y + d.z * d.z);
      const float gapw = d2f(len - rid);
      if (gapw >= 0.f) continue;
      const float il = __frcp_rn(d2f(len));
      const float3 u = f3(d2f(d.x) * il, d2f(d.y) * il, d2f(d.z) * il);
      const float3 cpv = (iv - jv) - crossf(iw * ri, u);
      const long long s = (long long)w * r.np + i;
      MixedRec rc = soa_load(r.h, s);
      float3 dF, dM;
      float dR;
      law32(a.pw, ri, -gapw, u, cpv, rc, ri, a.rfrc, a.dtf, dF, dM, dR);
      soa_store(r.h, s, rc);
      F.add(dF);
      M.add(dM);
      R.add(dR);
    }
    r.force[i] = add_sum(r.force[i], F);
    r.mom[i] = add_sum(r.mom[i], M);
    r.rmom[i] = r.rmom[i] + f2d(R.s - R.c);
  }
}

/* UpdateSystemG (kernel.cu:563-606) for the reference entry points' mixed
 * mode: the increments in FP32, as the fused step's integrator takes them,
 * added to the FP64 state (no FP64 division or square root) */
__global__ void k_update_ref_mixed(const double* __restrict__ rad, double3* __restrict__ pos,
                                   double3* __restrict__ vel, double3* __restrict__ angv,
                                   const double3* __restrict__ force, const double3* __restrict__ mom,
                                   double* __restrict__ rmom, int* __restrict__ flag, double* __restrict__ pmove,
                                   int n, double dt, float dtf, double move_limit) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  bool flagged = false;
  if (i < n) {
    const float t = 2.0f * d2f(rad[i]);
    const float mass = t * t * t;
    const float inv_m = dtf / mass;
    const double3 f = force[i];
    double3 v = vel[i];
    v.x += f2d(d2f(f.x) * inv_m);
    v.y += f2d(d2f(f.y) * inv_m);
    v.z += f2d(d2f(f.z) * inv_m);
    vel[i] = v;
    double3 p = pos[i];
    p.x = fma(v.x, dt, p.x);
    p.y = fma(v.y, dt, p.y);
    p.z = fma(v.z, dt, p.z);
    pos[i] = p;
    const float vx = d2f(v.x), vy = d2f(v.y), vz = d2f(v.z);
    const double pm = pmove[i] + f2d(sqrtf(vx * vx + vy * vy + vz * vz) * dtf);
    pmove[i] = pm;
    const float inv_i = dtf / (0.1f * mass * t * t);
    const double3 m = mom[i];
    const float dwx = d2f(m.x) * inv_i, dwy = d2f(m.y) * inv_i, dwz = d2f(m.z) * inv_i;
    const float rm = d2f(rmom[i]) * inv_i;
    rmom[i] = f2d(rm);
    double3 w = angv[i];
    const float wx1 = d2f(w.x) + dwx, wy1 = d2f(w.y) + dwy, wz1 = d2f(w.z) + dwz;
    const float wl = sqrtf(wx1 * wx1 + wy1 * wy1 + wz1 * wz1);
    float ix = dwx, iy = dwy, iz = dwz;
    if (wl > 1.0e-7f) {
      const float s = fminf(1.0f, rm / wl);
      ix -= wx1 * s;
      iy -= wy1 * s;
      iz -= wz1 * s;
    }
    w.x += f2d(ix);
    w.y += f2d(iy);
    w.z += f2d(iz);
    angv[i] = w;
    flagged = pm > move_limit;
  }
  const unsigned fm = __ballot_sync(0xffffffffu, flagged);
  if ((threadIdx.x & 31) == 0 && fm) atomicAdd(flag, __popc(fm));
}

MixArgs ref_args(const DevConsts& k, int n, int force_cap, int stage) {
  MixArgs a;
  std::memset(&a, 0, sizeof(a));
  a.n = n;
  a.force_cap = force_cap;
  a.dt = k.prm.dt;
  a.dtf = (float)k.prm.dt;
  a.rfrc = (float)k.mat[0].rfrc;
  a.lqd_vol = (float)k.lqd.vol;
  a.lqd_layer = (float)k.lqd.layer;
  a.lqd_gapmn = (float)k.lqd.gapmn;
  a.lqd_st = (float)k.lqd.stension;
  a.pp = make_law(k.cal, true, k.mat[0].dmpn * k.mat[0].dmpn, stage);
  a.pw = make_law(k.pwcal, false, k.mat[0].dmpn * k.mat[1].dmpn, stage);
  a.lq_mode = 0;
  return a;
}
}  // namespace

dem_status mixed_create(dem_ctx* c) {
  MixedState* m = new MixedState();
  std::memset(m, 0, sizeof(*m));
  c->mx = m;
  const size_t N = (size_t)c->n;
  float4** bufs[5] = {&m->place[0], &m->place[1], &m->motion[0], &m->motion[1], &m->force};
  for (float4** b : bufs) {
    void* p = nullptr;
    const size_t bytes = sizeof(float4) * N * (b == &m->force ? 1 : 2);
    dem_status st = cuda_alloc(&p, bytes);
    if (st != DEM_OK) return st;
    cudaMemset(p, 0, bytes);
    c->allocs.push_back(p);
    *b = (float4*)p;
  }
  {
    void *o = nullptr, *e = nullptr;
    dem_status st = cuda_alloc(&o, sizeof(float4) * 6 * N);
    if (st != DEM_OK) return st;
    c->allocs.push_back(o);
    m->wall_out = (float4*)o;
    st = cuda_alloc(&e, sizeof(int) * 3 * N);
    if (st != DEM_OK) return st;
    c->allocs.push_back(e);
    m->wall_entry = (int*)e;
  }
  /* offset putting every coordinate of the domain in [2^k, 2^(k+1)) */
  const PARAMETER& prm = c->s.prm;
  double ext = std::max(prm.EndPoint.x - prm.Origin.x,
                        std::max(prm.EndPoint.y - prm.Origin.y, prm.EndPoint.z - prm.Origin.z));
  int k2 = (int)std::ceil(std::log2(std::max(ext, 1.0) * 1.0001));
  const double base = std::ldexp(1.0, k2);
  m->off = make_double3(base - prm.Origin.x, base - prm.Origin.y, base - prm.Origin.z);
  /* the hi-part-only overlap estimate is off by at most |lo_i - lo_j| per
   * axis, below two ulps of the binade: four ulps is a safe candidate margin */
  m->coarse_tol = (float)(4.0 * std::ldexp(1.0, k2 - 23));
  m->bin_exp = 1023 + k2;
  m->base = (float)base;
  m->lo_scale = (float)std::ldexp(1.0, k2 - 52);
  return DEM_OK;
}

void mixed_destroy(dem_ctx* c) {
  delete c->mx;
  c->mx = nullptr;
}

int mixed_block_size(const dem_ctx* c) {
  /* the option (a multiple of 32 up to 128), else 128 */
  const int ob = c->opt.block_size;
  return (ob >= 32 && ob <= 32 * kWarps && ob % 32 == 0) ? ob : 32 * kWarps;
}

ShadowOut mixed_shadow_out(const dem_ctx* c, int which) {
  const MixedState* m = c->mx;
  return ShadowOut{m->place[which], m->motion[which], m->off, m->bin_exp, m->lo_scale};
}
const float4* mixed_motion(const dem_ctx* c, int which) { return c->mx->motion[which]; }

dem_status mixed_shadows(dem_ctx* c, int which, cudaStream_t s) {
  EngineBufs& b = c->b;
  k_shadows<<<grid_for(c->n, 256), 256, 0, s>>>(c->n, b.pos, b.vel, b.angv, b.rad, b.lqd, mixed_shadow_out(c, which));
  return cuda_check(cudaGetLastError(), "mixed_shadows launch");
}

dem_status mixed_import(dem_ctx* c, int which, int has_v, int has_w, cudaStream_t s) {
  EngineBufs& b = c->b;
  k_import_shadows<<<grid_for(c->n, 256), 256, 0, s>>>(c->n, b.id, b.tmp_pos, b.tmp_vel, b.tmp_angv, has_v, has_w,
                                                        b.pos, b.vel, b.angv, b.rad, b.lqd, mixed_shadow_out(c, which));
  return cuda_check(cudaGetLastError(), "mixed_import launch");
}

dem_status mixed_import_mapped(dem_ctx* c, int which, const int* inv, const double3* hp, const double3* hv,
                               const double3* hw, cudaStream_t s) {
  EngineBufs& b = c->b;
  /* a few resident blocks per SM, each walking several slices */
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 152;
  }
  const long long nsl = ((long long)c->n + kImportThreads - 1) / kImportThreads;
  const int grid = (int)std::min<long long>(nsl, (long long)kImportBlocksPerSM * sms);
  k_import_shadows_mapped<<<grid, kImportThreads, 0, s>>>(c->n, inv, hp, hv, hw, b.pos, b.vel, b.angv, b.rad, b.lqd,
                                                         mixed_shadow_out(c, which));
  return cuda_check(cudaGetLastError(), "mixed_import_mapped launch");
}

Prefilter mixed_prefilter(dem_ctx* c, int which) {
  /* |(hi_i - hi_j) - (x_i - x_j)| <= one binade ulp per axis (the lo parts are
   * below half an ulp each): sqrt(3) ulps, plus FP32 rounding of the distance
   * and of the cut-off (~3e-7 relative, distances < 4 reduced units) */
  return Prefilter{c->mx->place[which], 0.5f * c->mx->coarse_tol + 2.0e-6f, c->mx->base, 0.25f * c->mx->coarse_tol,
                   c->radii_bounded};
}

const char* mixed_step_kernel_name(const dem_ctx* c) {
  const bool wet = c->s.force_cap == 1;
  const bool net = wet && c->opt.capillary == DEM_CAP_MLP;
  return net ? "k_pair_mixed<1,1> + k_body_mixed<1,1>" : wet ? "k_pair_mixed<1,0> + k_body_mixed<1,0>"
                                                             : "k_pair_mixed<0,0> + k_body_mixed<0,0>";
}

dem_status mixed_step(dem_ctx* c, int which, cudaStream_t s) {
  MixedState* m = c->mx;
  EngineBufs& b = c->b;
  MixArgs a;
  std::memset(&a, 0, sizeof(a));
  a.place_in = m->place[which];
  a.motion_in = m->motion[which];
  a.place_out = m->place[1 - which];
  a.motion_out = m->motion[1 - which];
  a.pos = b.pos; a.vel = b.vel; a.angv = b.angv; a.rad = b.rad; a.pmove = b.pmove;
  a.num_nebor = b.num_nebor; a.plevel = b.plevel; a.nidx = b.nidx; a.npars = b.npars; a.nneb = b.nneb;
  a.body_order = c->body_order;
  a.ps = b.ps; a.pair_out = reinterpret_cast<float4*>(b.pair_out);
  a.wall_out = m->wall_out; a.wall_entry = m->wall_entry;
  a.wlist = b.wlist; a.nwall = b.nwall; a.wrec = b.wrec;
  a.force_out = m->force; a.flag = c->step_flag ? c->step_flag : b.flag; a.err = b.err; a.counters = b.counters; a.cyl = b.cyl;
  a.sys_of_id = b.sys_of_id; a.sys_wet = b.sys_wet;
  a.n = c->n;
  a.force_cap = c->s.force_cap;
  a.off = m->off;
  a.offf = make_float3((float)m->off.x, (float)m->off.y, (float)m->off.z);
  a.wall_tol = 4.0f * m->coarse_tol; /* 16 binade ulps */
  a.bin_exp = m->bin_exp;
  a.lo_scale = m->lo_scale;
  a.dt = c->s.prm.dt;
  a.dtf = (float)c->s.prm.dt;
  a.move_limit = 0.3 * c->s.prm.SearchGap;
  a.rfrc = (float)c->s.mat[0].rfrc;
  a.lqd_vol = (float)c->s.lqd.vol;
  a.lqd_layer = (float)c->s.lqd.layer;
  a.lqd_gapmn = (float)c->s.lqd.gapmn;
  a.lqd_st = (float)c->s.lqd.stension;
  a.pp = make_law(c->s.cal, true, c->s.mat[0].dmpn * c->s.mat[0].dmpn, c->s.load_stage);
  calParaPP pw;
  std::memcpy(&pw, &c->s.pwcal, sizeof(pw));
  a.pw = make_law(pw, false, c->s.mat[0].dmpn * c->s.mat[1].dmpn, c->s.load_stage);
  a.id = b.id;
  a.capw = reinterpret_cast<const CapNetSmem*>(c->cap_w);
  a.theta_seed = c->theta_seed;
  a.theta_max = c->theta_max;
  a.gate = c->step_gate;
  a.lq_mode = c->lm.mode;
  a.lq_vmin = (float)c->lm.vol_min;
  a.lq_vspan = (float)(c->lm.vol_max - c->lm.vol_min);
  a.lq_theta_max = c->lm.theta_max;
  a.lq_seed = c->lm.seed;
  const bool net = c->s.force_cap == 1 && c->opt.capillary == DEM_CAP_MLP;
  if (net && !c->cap_w) return fail(DEM_ERR_STATE, "DEM_CAP_MLP: no network installed (dem_set_capnet)");
  const bool wet = c->s.force_cap == 1;
  const int bs = mixed_block_size(c);
  /* The pair count is known on the device only: the grid covers six pairs a
   * sphere (a packed bed lists 4.3) and strides beyond; the closure's blocks
   * stage its weights once, so they are as many as stay resident. */
  const long long most = std::min<long long>(c->b.ps.cap, 6LL * c->n);
  const int g = grid_for(c->n, bs);
  int gp = grid_for(most, bs);
  if (net) gp = std::min(gp, 152 * kNetBlocks * (32 * kWarps / bs));
  if (c->moving_walls) {
    k_move_walls<<<1, 32, 0, s>>>(b.cyl, b.n_sys > 0 ? b.n_sys : 1, c->s.prm.dt, c->step_gate);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_check(e, "mixed_step wall motion");
  }
  a.wall_blocks = (unsigned)grid_for(c->n / 4 + 1, bs); /* a packed bed lists one sphere in six */
  gp += (int)a.wall_blocks;
  if (net) k_pair_mixed<true, true><<<gp, bs, kCapSmem, s>>>(a);
  else if (wet) k_pair_mixed<true, false><<<gp, bs, 0, s>>>(a);
  else k_pair_mixed<false, false><<<gp, bs, 0, s>>>(a);
  if (net) k_body_mixed<true, true><<<g, bs, 0, s>>>(a);
  else if (wet) k_body_mixed<true, false><<<g, bs, 0, s>>>(a);
  else k_body_mixed<false, false><<<g, bs, 0, s>>>(a);
  return cuda_check(cudaGetLastError(), "mixed_step launch");
}

dem_status mixed_wall_entries(dem_ctx* c, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(c->b.ps.ctl + 3, 0, sizeof(int), s);
  if (e != cudaSuccess) return cuda_check(e, "wall entries");
  k_wall_entries<<<grid_for(c->n, 256), 256, 0, s>>>(c->b.nwall, c->n, c->mx->wall_entry, c->b.ps.ctl + 3);
  return cuda_check(cudaGetLastError(), "wall entries launch");
}

dem_status mixed_bridge_counts(dem_ctx* c, int which, cudaStream_t s) {
  k_lqd_from_shadow<<<grid_for(c->n, 256), 256, 0, s>>>(c->n, c->mx->motion[which], c->b.lqd);
  return cuda_check(cudaGetLastError(), "mixed_bridge_counts launch");
}

const float4* mixed_force_shadow(const dem_ctx* c) { return c->mx ? c->mx->force : nullptr; }

dem_status mixed_force_to_master(dem_ctx* c, cudaStream_t s) {
  k_force_out<<<grid_for(c->n, 256), 256, 0, s>>>(c->n, c->mx->force, c->b.force, c->b.mom);
  /* the bridge counts of the last step live in the shadow the next step reads */
  k_lqd_from_shadow<<<grid_for(c->n, 256), 256, 0, s>>>(c->n, c->mx->motion[c->parity], c->b.lqd);
  return cuda_check(cudaGetLastError(), "mixed_force_to_master launch");
}

size_t ref_mixed_scratch(int n) { return kRefBody * (size_t)n; }

dem_status pp_force_ref_mixed(const double3* pos, const double3* vel, const double3* angvel, const double* rad,
                              const int* nebor, const int* plevel, const int* level_npars, const int* level_nnebors,
                              const int* nebor_idx, HistSoA h, const int* num_nebor, int* lqd, const int* lqd_old,
                              double3* force, double3* mom, double* rmom, int n, int force_cap, int stage,
                              const DevConsts& k, void* bodies, cudaStream_t s) {
  if (n <= 0) return DEM_OK;
  RefArrays r;
  std::memset(&r, 0, sizeof(r));
  r.pos = pos; r.vel = vel; r.angv = angvel; r.rad = rad;
  r.nebor = nebor; r.plevel = plevel; r.npars = level_npars; r.nneb = level_nnebors; r.nidx = nebor_idx;
  r.num_nebor = num_nebor; r.lqd_old = lqd_old; r.lqd = lqd; r.h = h;
  r.force = force; r.mom = mom; r.rmom = rmom;
  RefBody* pk = static_cast<RefBody*>(bodies);
  if (pk) k_ref_bodies<<<grid_for(n, 128), 128, 0, s>>>(r, n, force_cap == 1, pk);
  k_pp_ref_mixed<<<grid_for(n, 32), 32, 0, s>>>(ref_args(k, n, force_cap, stage), r, pk);
  return cuda_check(cudaGetLastError(), "pp_force_ref_mixed launch");
}

dem_status wall_force_ref_mixed(const double3* pos, const double3* vel, const double3* angvel, double3* force,
                                double3* mom, double* rmom, const double* rad, CylinderBC* cyl, HistSoA h,
                                const int* nwall, const int* wlist, size_t pitch, int n, int NP, int stage,
                                const DevConsts& k, cudaStream_t s) {
  if (n <= 0) return DEM_OK;
  RefArrays r;
  std::memset(&r, 0, sizeof(r));
  r.pos = pos; r.vel = vel; r.angv = angvel; r.rad = rad; r.h = h;
  r.force = force; r.mom = mom; r.rmom = rmom;
  r.cyl = cyl; r.nwall = nwall; r.wlist = wlist; r.pitch = pitch; r.np = NP;
  k_move_walls<<<1, 32, 0, s>>>(cyl, 1, k.prm.dt, nullptr);
  k_wall_ref_mixed<<<grid_for(n, kRefWallThreads * kRefWallEach), kRefWallThreads, 0, s>>>(ref_args(k, n, 0, stage), r);
  return cuda_check(cudaGetLastError(), "wall_force_ref_mixed launch");
}

dem_status update_ref_mixed(const double* rad, double3* pos, double3* vel, double3* angvel, const double3* force,
                            const double3* mom, double* rmom, int* flag, double* pmove, int n, const DevConsts& k,
                            cudaStream_t s) {
  if (n <= 0) return DEM_OK;
  k_update_ref_mixed<<<grid_for(n, 256), 256, 0, s>>>(rad, pos, vel, angvel, force, mom, rmom, flag, pmove, n,
                                                     k.prm.dt, (float)k.prm.dt, 0.3 * k.prm.SearchGap);
  return cuda_check(cudaGetLastError(), "update_ref_mixed launch");
}

}  // namespace dem
