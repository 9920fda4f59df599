/*
 * dem_device.cuh -- device math of the DEM engine, FP64 reference-formula path.
 *
 * The contact laws here restate the reference's kernel.cu formulas with the
 * same operand order and parenthesisation, so that, compiled with
 * -fmad=false, their results differ from a CPU FP64 evaluation only by the
 * last-ulp differences of pow/log/exp between CUDA and the host libm.
 */
#pragma once

#include <cuda_runtime.h>

#include "dem_internal.h"
#include "liquid.cuh"
#include "pairs.cuh"

namespace dem {

/* heydem.h:15 */
constexpr double kPiRef = 3.1415926;

/* ---- double3 algebra in the reference's evaluation order (double_math.h) ---- */
__device__ __forceinline__ double3 d3(double x, double y, double z) { return make_double3(x, y, z); }
__device__ __forceinline__ double3 add3(double3 a, double3 b) { return d3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ double3 sub3(double3 a, double3 b) { return d3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ double3 mul3(double3 a, double s) { return d3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ double3 smul3(double s, double3 a) { return d3(s * a.x, s * a.y, s * a.z); }
__device__ __forceinline__ double3 div3(double3 a, double s) { return d3(a.x / s, a.y / s, a.z / s); }
__device__ __forceinline__ double dot3(double3 a, double3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ double len3(double3 a) { return sqrt(dot3(a, a)); }
__device__ __forceinline__ double3 cross3(double3 a, double3 b) {
  return d3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}

/* The reference's pow with the exponents 1.5, 3 and 5 as products of sqrt and
 * x (IEEE sqrt and products, no contraction in the FP64 files): x^1.5 and x^3
 * land within 1.3 ulp of the exact power and x^5 within 2.6 ulp (three
 * roundings), against 2 ulp for CUDA's pow and 0.52 for the CPU oracle's --
 * relative differences of a few 1e-16, far inside the 1e-12 lockstep bound --
 * for a few FP64 instructions instead of some tens: on GB300 the FP64 laws are
 * bound by FP64 issue.  pow5 only scales the integrator's spin increments. */
__device__ __forceinline__ double pow1_5(double x) { return x * sqrt(x); }
__device__ __forceinline__ double cube(double x) { return x * x * x; }
__device__ __forceinline__ double pow5(double x) {
  const double x2 = x * x;
  return x2 * x2 * x;
}

/* This thread's particle with the blocks taken in reverse.  Particles sit in
 * level-major cell order, so the largest spheres -- the most neighbours, the
 * longest loops -- come last; the GPU starts blocks roughly in index order,
 * and in index order their blocks would run in the grid's tail.  Taken first,
 * they overlap the many light blocks instead (each particle's work is its
 * own, so the results are the same bits). */
__device__ __forceinline__ int reversed_block_thread() {
  return (int)((gridDim.x - 1 - blockIdx.x) * blockDim.x + threadIdx.x);
}

/* ---- FP32 <-> FP64 through the integer pipe ----
 * On GB300 FP64 conversions issue on the scarce FP64 pipe; these move the bits
 * with integer operations instead.  d2f truncates the mantissa (error below one
 * FP32 ulp) and flushes results below the FP32 normal range to zero; f2d is
 * exact for normal floats.  Infinities and NaNs stay non-finite. */
__device__ __forceinline__ float d2f(double x) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  const unsigned sign = (unsigned)(u >> 32) & 0x80000000u;
  const int e = (int)((u >> 52) & 0x7ff);
  const int fe = e - 1023 + 127;
  if (fe <= 0) return __uint_as_float(sign);
  if (fe >= 255) return __uint_as_float(sign | 0x7f800000u | (e == 0x7ff && (u & 0xfffffffffffffull) ? 1u : 0u));
  return __uint_as_float(sign | ((unsigned)fe << 23) | (unsigned)((u >> 29) & 0x7fffffu));
}
__device__ __forceinline__ double f2d(float f) {
  const unsigned b = __float_as_uint(f);
  const unsigned e = (b >> 23) & 0xffu;
  const unsigned long long sign = (unsigned long long)(b & 0x80000000u) << 32;
  if (e == 0) return __longlong_as_double((long long)sign);
  const unsigned long long de = (e == 255) ? 0x7ffull : (unsigned long long)(e - 127 + 1023);
  return __longlong_as_double((long long)(sign | (de << 52) | ((unsigned long long)(b & 0x7fffffu) << 29)));
}

/* ---- cell hash (kernel.cu:617-641) ---- */
/* floor(d / cs) for a cell size cs, as the FP64 quotient gives it: from FP32
 * unless that quotient is within its error (two truncations and a rounding,
 * below 4e-7 of it) of an integer -- an FP64 division is ten instructions of a
 * pipe that takes 17 cycles each (hashing 200,000 spheres 16.1 -> 5.9 us) */
__device__ __forceinline__ int cell_along(double d, double cs) {
  const float t = d2f(d) / d2f(cs), f = floorf(t), tol = 4.0e-7f * t;
  if (t - f > tol && f + 1.0f - t > tol) return (int)f;
  return (int)floor(d / cs);
}
__device__ __forceinline__ int3 grid_pos(double3 p, int lvl, const LevelView& lv, double3 origin) {
  const double cs = lv.cell_size[lvl];
  const int3 g = lv.grid_size[lvl];
  int3 r;
  r.x = max(0, min(cell_along(p.x - origin.x, cs), g.x));
  r.y = max(0, min(cell_along(p.y - origin.y, cs), g.y));
  r.z = max(0, min(cell_along(p.z - origin.z, cs), g.z));
  return r;
}
__device__ __forceinline__ int grid_hash(int3 g, int lvl, const LevelView& lv) {
  const int3 s = lv.grid_size[lvl];
  return (g.z * s.y * s.x) + (g.y * s.x) + g.x;
}

/* first slot of level L's block in a level/slot-major list: the sum over the
 * lower levels of slots x particles (kernel.cu:443-454); reads levels < L only */
__device__ __forceinline__ long long slot_base(int L, const int* npars, const int* nneb) {
  long long b = 0;
  for (int l = 0; l < L; l++) b += (long long)nneb[l] * npars[l];
  return b;
}

/* ---- history record (the fields of one contact slot) ---- */
struct HistRec {
  double3 dispt;
  double nDsp, nDsp_mx, plstRad, plstDfm;
  int stage;
};

/* history access, reference SoA layout */
struct HistSoAAcc {
  HistSoA h;
  __device__ __forceinline__ long long at(long long slot) const { return slot; } /* a slot's record */
  __device__ __forceinline__ HistRec load(long long i) const {
    HistRec r;
    r.dispt = h.dispt[i];
    r.nDsp = h.nDsp[i];
    r.nDsp_mx = h.nDsp_mx[i];
    r.plstRad = h.plstRad[i];
    r.plstDfm = h.plstDfm[i];
    r.stage = h.stage[i];
    return r;
  }
  __device__ __forceinline__ void store(long long i, const HistRec& r) const {
    h.dispt[i] = r.dispt;
    h.nDsp[i] = r.nDsp;
    h.nDsp_mx[i] = r.nDsp_mx;
    h.plstRad[i] = r.plstRad;
    h.plstDfm[i] = r.plstDfm;
    h.stage[i] = r.stage;
  }
  __device__ __forceinline__ int brg(long long i) const { return h.lqdBrg[i]; }
  __device__ __forceinline__ void set_brg(long long i, int v) const { h.lqdBrg[i] = v; }
};

/* history access, the engine's 64-byte records + one bridge byte per slot */
struct HistAoSAcc {
  ContactRec* rec;
  unsigned char* brgf;
  __device__ __forceinline__ HistRec load(long long i) const {
    const double2* p = reinterpret_cast<const double2*>(rec + i);
    const double2 a = p[0], b = p[1], c = p[2];
    const double2 d = p[3];
    HistRec r;
    r.dispt = make_double3(a.x, a.y, b.x);
    r.nDsp = b.y;
    r.nDsp_mx = c.x;
    r.plstRad = c.y;
    r.plstDfm = d.x;
    r.stage = __double_as_longlong(d.y) & 0xffffffff;
    return r;
  }
  __device__ __forceinline__ void store(long long i, const HistRec& r) const {
    double2* p = reinterpret_cast<double2*>(rec + i);
    p[0] = make_double2(r.dispt.x, r.dispt.y);
    p[1] = make_double2(r.dispt.z, r.nDsp);
    p[2] = make_double2(r.nDsp_mx, r.plstRad);
    p[3] = make_double2(r.plstDfm, __longlong_as_double((long long)(unsigned)r.stage));
  }
  __device__ __forceinline__ int brg(long long i) const { return brgf ? brgf[i] : 0; }
  __device__ __forceinline__ void set_brg(long long i, int v) const {
    if (brgf) brgf[i] = (unsigned char)v;
  }
};

/* history access, the engine's pair list with a record and a flag a side */
struct HistPairAcc {
  PairSet ps;
  __device__ __forceinline__ HistAoSAcc set() const {
    return pair_ctl(ps).x ? HistAoSAcc{ps.rec[1], ps.brg[1]} : HistAoSAcc{ps.rec[0], ps.brg[0]};
  }
  __device__ __forceinline__ long long at(long long slot) const {
    const int e = ps.eidx[slot];
    return e == kNoPair ? -1 : e < 0 ? 2LL * ~e + 1 : 2LL * e;
  }
  __device__ __forceinline__ HistRec load(long long i) const { return set().load(i); }
  __device__ __forceinline__ void store(long long i, const HistRec& r) const { set().store(i, r); }
  __device__ __forceinline__ int brg(long long i) const { return set().brg(i); }
  __device__ __forceinline__ void set_brg(long long i, int v) const { set().set_brg(i, v); }
};

/* The constants of the p-p law (ContactForceD, kernel.cu:89-228) or the wall law
 * (PWcontactD, kernel.cu:236-359): products and quotients of the material alone,
 * taken once on the host by the same operations in the same order (IEEE, so the
 * same values), not by every thread -- a root, two divisions and a dozen
 * products of some 350 FP64 instructions a contact. */
struct LawK64 {
  double k43;             /* 4/3 E* */
  double ydsp_t, yforce_t, ystiff_t;
  double damp;            /* -2 sqrt(dmpn product) E* */
  double sfrc3, nsfrc;    /* 3 mu, -mu */
  double kt;              /* 16 (1 - nu) E* / (4 - 2 nu) */
  double roll;            /* 0.5 (rfrc + rfrc) */
  double dt;
  double film;            /* 2 x the liquid layer */
  double eps;             /* spring rotation, slip-ratio and rescale guard: 1e-7 (p-p) / 1e-10 (wall) */
  int hertz_le;           /* p-p: nrm <= ydsp*R; wall: nrm < ydsp*R */
  int damp_on;            /* p-p: stage == 1; wall: stage == 1 || 7 */
};

/* elasto-plastic Hertz normal force + damping + tangential spring with slip
 * + rolling resistance, FP64, the reference's operand order.
 *
 * The reference's pow(x, 0.5) and pow(x, 2.0) are taken as sqrt(x) and x * x:
 * the correctly rounded square root and product, which is what a correctly
 * rounded pow returns for these exponents (the CPU oracle's glibc pow, within
 * its 0.52-ulp bound; CUDA's pow carries up to 2 ulp); pow(x, 1.5) as pow1_5.
 * The exponent 2/3 (plastic loading only) stays pow.  On
 * GB300 the law is bound by FP64 issue, where each pow is some tens of FP64
 * instructions. */
__device__ __forceinline__ void contact_law64(const LawK64& c, double ijRad, double nrm, double3 u, double3 cpv,
                                              HistRec& h, double iRad, double3& dF, double3& dM, double& dR) {
  /* pow(ijRad * nrm, 0.5) (twice in the reference's law) and the damping's
   * sqrt(ijRad * nrm): one value */
  const double sq = sqrt(ijRad * nrm);
  double fN = 0.0;
  int st;
  if (nrm < h.plstDfm) st = 1;
  else if (nrm >= h.plstDfm && nrm < h.nDsp) st = 3;
  else if (nrm >= h.nDsp && nrm < h.nDsp_mx) st = 4;
  else st = 2;
  h.stage = st;
  if (st == 1) {
    fN = 0.0;
  } else if (st == 2) {
    bool elastic = c.hertz_le ? (nrm <= c.ydsp_t * ijRad) : (nrm < (c.ydsp_t * ijRad));
    if (elastic) {
      fN = c.k43 * sq * nrm;
      h.plstRad = ijRad;
      h.plstDfm = 0.0;
    } else {
      fN = c.yforce_t * (ijRad * ijRad) + c.ystiff_t * ijRad * (nrm - c.ydsp_t * ijRad);
      h.plstRad = ijRad * (c.k43 * sq * nrm) / fN;
      h.plstDfm = nrm - pow((fN / (c.k43 * sqrt(ijRad))), 2.0 / 3.0);
    }
    h.nDsp_mx = nrm;
  } else {
    fN = c.k43 * sqrt(h.plstRad) * pow1_5(nrm - h.plstDfm);
  }
  h.nDsp = nrm;

  const double vn = dot3(cpv, u);
  double fD = 0.0;
  if (c.damp_on) fD = c.damp * sq * vn;

  const double3 vt = sub3(cpv, smul3(vn, u));
  const double3 old = h.dispt;
  double3 dT = cross3(smul3(-1.0, u), cross3(u, old));
  if (len3(dT) > c.eps)
    dT = add3(div3(mul3(dT, len3(old)), len3(dT)), mul3(vt, c.dt));
  else
    dT = add3(dT, mul3(vt, c.dt));

  const double dsmx = c.sfrc3 * fN / (c.kt * sq);
  double ratio = 1.0;
  if (len3(dT) < dsmx) {
    if (dsmx > c.eps) ratio = 1.0 - pow1_5(1.0 - len3(dT) / dsmx);
  } else {
    ratio = 1.0;
    if (len3(dT) > c.eps) dT = div3(smul3(dsmx, dT), len3(dT));
    else dT = smul3(dsmx, dT);
  }
  h.dispt = dT;

  double3 fT = d3(0.0, 0.0, 0.0);
  if (len3(dT) < dsmx) {
    if (len3(dT) > 1.0e-10) fT = div3(smul3(c.nsfrc * fN * ratio, dT), len3(dT));
  } else {
    if (len3(vt) > 1.0e-10) fT = div3(smul3(c.nsfrc * fN * ratio, vt), len3(vt));
  }
  dF = add3(smul3(fN + fD, u), fT);
  const double arm = iRad - nrm / 2.0;
  dM = cross3(smul3(-arm, u), fT);
  dR = c.roll * fN * iRad;
}

/* capillary bridge force, kernel.cu:65-81 (the closed-form fit of Willett et
 * al. 2000 at zero contact angle, the reference's coefficients); pow(x, 0.5),
 * pow(x, 2.0) and pow(x, 3.0) as sqrt(x), x * x and cube(x) (contact_law64) */
__device__ __forceinline__ double fcap64(double Splus, double ijVol, double effectR, const LIQUID& L) {
  Splus = max(L.gapmn, Splus);
  Splus = Splus / sqrt(ijVol);
  const double lv = log(ijVol);
  const double lv2 = lv * lv, lv3 = cube(lv);
  const double f1 = -0.44507 - 0.1119 * lv - 0.012101 * lv2 - 0.0005 * lv3;
  const double f2 = 1.9222 - 0.0668 * lv - 0.0013375 * lv2;
  const double f3 = 1.268 + 0.198 * lv + 0.02232 * lv2 + 0.0008585 * lv3;
  const double f4 = -0.010703 + 0.03345 * lv + 0.0018574 * lv2;
  const double ls = log(Splus);
  return 2 * kPiRef * effectR * L.stension * exp(f1 - f2 * exp(f3 * ls + f4 * (ls * ls)));
}

/* Two float4 of one 32-byte sector in one 256-bit access (p a multiple of 32
 * bytes): the pair kernel's gathers are bound by the L1's wavefronts, and
 * scattered lanes cost one per sector and instruction.  Shadows, records and
 * results in this form: 70.6 us a step on the packed 200k bed, 608 on 2M spheres;
 * as single float4 of separate arrays 75.1 and 664. */
__device__ __forceinline__ void get2(const float4* p, float4& a, float4& b) {
  asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
      : "l"(p));
}
__device__ __forceinline__ void put2(float4* p, float4 a, float4 b) {
  asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w),
               "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
               : "memory");
}

/* hi/lo split of a coordinate already shifted into the binade [2^k, 2^(k+1)):
 * hi keeps the top 24 significand bits (exponent fixed), lo the remaining 29
 * bits as an exact integer times 2^(k-52), rounded to 24 bits.  Integer and
 * conversion units only; a value outside the binade takes the FP64 route. */
__device__ __forceinline__ void split_hi_lo(double xo, int dexp, float lo_scale, float& hi, float& lo) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(xo);
  if ((int)((u >> 52) & 0x7ff) == dexp && !(u >> 63)) {
    hi = __uint_as_float(((unsigned)(dexp - 1023 + 127) << 23) | (unsigned)((u >> 29) & 0x7fffffu));
    lo = __uint2float_rn((unsigned)(u & 0x1fffffffull)) * lo_scale;
  } else {
    hi = (float)xo;
    lo = (float)(xo - (double)hi);
  }
}

/* the FP32 shadows of a mixed step, two float4 to a sphere: the position's high
 * parts and radius, the low parts; the velocity and bridge count, the spin */
struct ShadowOut {
  float4 *place, *motion;
  double3 off;
  int bin_exp;
  float lo_scale;
};
__device__ __forceinline__ void write_shadow(const ShadowOut& sh, int q, double3 p, double3 v, double3 w, double r,
                                             int lqd) {
  float4 ph, pl;
  split_hi_lo(p.x + sh.off.x, sh.bin_exp, sh.lo_scale, ph.x, pl.x);
  split_hi_lo(p.y + sh.off.y, sh.bin_exp, sh.lo_scale, ph.y, pl.y);
  split_hi_lo(p.z + sh.off.z, sh.bin_exp, sh.lo_scale, ph.z, pl.z);
  ph.w = (float)r;
  pl.w = (float)(r - (double)ph.w);
  put2(sh.place + 2 * q, ph, pl);
  put2(sh.motion + 2 * q, make_float4(d2f(v.x), d2f(v.y), d2f(v.z), __int_as_float(lqd)),
       make_float4(d2f(w.x), d2f(w.y), d2f(w.z), 0.f));
}

}  // namespace dem
