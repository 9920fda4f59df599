/*
 * step64.cu -- FP64 per-step kernels with the reference's formulas (sm_103a).
 *
 * The validation path: p-p contact + capillary (PPForceCalcG, kernel.cu:413-552),
 * cylinder-wall contact (CirPWInterG, kernel.cu:958-1023) and the integrator
 * (UpdateSystemG, kernel.cu:563-606), on the reference's layouts.  Compiled
 * with -fmad=false so every + and * rounds as the CPU oracle's do; the
 * remaining differences are the last-ulp differences of pow/log/exp.
 *
 * Used by the reference-compatible entry points (PpInterCalc, CirPWCalc,
 * UpdateSystem, VarInit) and by the native engine's DEM_PREC_FP64 mode, which
 * runs them on cell-sorted buffers.  On GB300 these are bound by FP64
 * transcendental issue (about 6 Gpow/s per GPU); the fast path is mixed.cu.
 */
#include <cuda_runtime.h>

#include <cmath>

#include "dem_device.cuh"
#include "pairs.cuh"

namespace dem {

namespace {

inline int grid_for(long long n, int block) { return n <= 0 ? 1 : (int)((n + block - 1) / block); }

/* VarInit (Allocation.cpp:308-317) in one pass */
__global__ void k_var_init(double3* __restrict__ force, double3* __restrict__ mom, double* __restrict__ rmom,
                           int* __restrict__ lqd, int* __restrict__ lqd_old, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  lqd_old[i] = lqd[i];
  lqd[i] = 0;
  force[i] = make_double3(0.0, 0.0, 0.0);
  mom[i] = make_double3(0.0, 0.0, 0.0);
  rmom[i] = 0.0;
}

template <class H> struct Acc;
template <> struct Acc<HistSoA> { using T = HistSoAAcc; static T make(HistSoA h) { return T{h}; } };
template <> struct Acc<HistAoS> { using T = HistAoSAcc; static T make(HistAoS h) { return T{h.rec, h.brg}; } };
template <> struct Acc<PairSet> { using T = HistPairAcc; static T make(PairSet h) { return T{h}; } };

/* host: the law's constants, each by the operations the formulas prescribe */
LawK64 make_law64(const calParaPP& c, bool pp, double dmpn_product, int stage, double rfrc, double dt, double layer) {
  LawK64 l;
  l.k43 = 4.0 / 3.0 * c.emod;
  l.ydsp_t = c.ydsp_t;
  l.yforce_t = c.yforce_t;
  l.ystiff_t = c.ystiff_t;
  const double damp = -2.0 * std::sqrt(dmpn_product);
  l.damp = damp * c.emod;
  l.sfrc3 = 3.0 * c.sfrc;
  const double num = 16.0 * (1 - c.pois) * c.emod;
  l.kt = num / (4.0 - 2.0 * c.pois);
  l.nsfrc = -1.0 * c.sfrc;
  l.roll = 0.5 * (rfrc + rfrc);
  l.dt = dt;
  l.film = 2 * layer;
  l.eps = pp ? 1.0e-7 : 1.0e-10;
  l.hertz_le = pp ? 1 : 0;
  l.damp_on = pp ? stage == 1 : (stage == 1 || stage == 7);
  return l;
}

/* ---- p-p contact + capillary (PPForceCalcG, kernel.cu:413-552) ----
 * A warp takes 32 spheres and puts their neighbour slots end to end; kChunk of
 * them at a time go through four phases, every lane taking the next item
 * whichever sphere owns it: the distance of every entry, with the contacts and
 * the bridges listed; the contact law over the listed contacts; the capillary
 * force over the listed bridges; and every sphere's own sums, in neighbour
 * order.  Each entry's operations and each sphere's order of sums are the
 * reference's, so the results are those of a thread per sphere, bit for bit.
 *
 * FP64 issue bounds it (an FP64 instruction occupies the pipe for 17 cycles
 * whatever lanes are active), and a thread per sphere kept 15 of 32 lanes: the
 * warp waits for its longest list, and executes the law and the bridge wherever
 * one lane needs them.  The packed 200k bed's contacts and bridges on the
 * reference's layouts: 2787 -> 1353 us (whole steps there 3.34 -> 1.62 ms, of
 * the FP64 engine 2.63 -> 1.60).  A warp of that bed has 277 entries: steps with
 * chunks of 320, one warp a block, took 1618 us, of 256 1688, of 384 (fewer warps
 * resident) 1712, of 128 in blocks of four warps 2027.
 *
 * The unit normal, the partner's liquid and the rupture distance are evaluated
 * only where the reference's formulas use them: a contact or a bridge needs the
 * normal, a bridge's force the volume, and the rupture test can change only a
 * bridge that exists beyond the film distance. */
constexpr int kChunk = 320;
constexpr int kPpWarps = 1;

struct PpWarp {
  double ux[kChunk], uy[kChunk], uz[kChunk]; /* unit normal, then the bridge's force */
  double gap[kChunk];
  double ijr[kChunk];                                     /* r_i r_j / (r_i + r_j) */
  long long rec[kChunk]; /* the entry's history record */
  int j[kChunk];
  double out[7][kChunk]; /* dF, dM, dR */
  unsigned char owner[kChunk], flags[kChunk];
  unsigned short contact[kChunk], bridge[kChunk];
};
constexpr size_t kPpSmem = kPpWarps * sizeof(PpWarp);
static_assert(kPpSmem <= 48 * 1024, "above 48 KB a launch needs the attribute that allows it");

/* the lane whose slots hold entry p: the number of lanes whose inclusive slot
 * count is <= p.  Every lane of the warp calls it. */
__device__ __forceinline__ int entry_owner(int incl, int p) {
  int o = 0;
#pragma unroll
  for (int b = 16; b > 0; b >>= 1) {
    const int v = __shfl_sync(0xffffffffu, incl, o + b - 1);
    if (v <= p) o += b;
  }
  return min(o, 31);
}

/* counters[0]: neighbour entries visited, [1]: contacts, [2]: wet non-contact
 * bridges, [3]: wall contacts */
template <class HA>
__global__ void __launch_bounds__(32 * kPpWarps) k_pp_force64(
    const double3* __restrict__ pos, const double3* __restrict__ vel, const double3* __restrict__ angvel,
    const double* __restrict__ rad, const int* __restrict__ nebor, const int* __restrict__ plevel,
    const int* __restrict__ level_npars, const int* __restrict__ level_nnebors,
    const int* __restrict__ nebor_idx, HA h, const int* __restrict__ num_nebor, int* __restrict__ lqd,
    double3* __restrict__ force, double3* __restrict__ mom, double* __restrict__ rmom, int n, int force_cap,
    LawK64 law, DevConsts k, unsigned long long* __restrict__ counters, const int* __restrict__ id, LiquidModel lm,
    const double* __restrict__ pvol) {
  extern __shared__ __align__(16) unsigned char dsm[];
  constexpr unsigned FULL = 0xffffffffu;
  PpWarp& sm = reinterpret_cast<PpWarp*>(dsm)[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  /* blocks in reverse: in cell order the largest spheres, with the most
   * pairs, come last (in the reference's order this is only another schedule) */
  const int i = reversed_block_thread();
  const bool live = i < n;
  const int ii = live ? i : n - 1;
  const int first = i - lane; /* the warp's first sphere */
  const bool ref_liquid = force_cap == 1 && lm.mode == 0;
  const int L = plevel[ii];
  const int stride = level_npars[L];
  const long long base = slot_base(L, level_npars, level_nnebors) + nebor_idx[ii];
  const int nn = live ? num_nebor[ii] : 0;
  int incl = nn;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += t;
  }
  const int excl = incl - nn;
  const int total = __shfl_sync(FULL, incl, 31);
  double3 F = force[ii], M = mom[ii];
  double R = rmom[ii];
  F.z = F.z - cube(2.0 * rad[ii]); /* gravity, m = (2r)^3 */
  int wet = lqd[ii], ncontact = 0, nbridge = 0;
  for (int c0 = 0; c0 < total; c0 += kChunk) {
    const int cend = min(total, c0 + kChunk);
    /* distances; contacts and bridges listed */
    int nc = 0, nb = 0;
    for (int p0 = c0; p0 < cend; p0 += 32) {
      const int p = p0 + lane, e = p - c0;
      const int o = entry_owner(incl, p);
      const int eo = __shfl_sync(FULL, excl, o);
      const long long bo = __shfl_sync(FULL, base, o);
      const int so = __shfl_sync(FULL, stride, o);
      bool touch = false, bridge = false;
      if (p < cend) {
        const long long s = bo + (long long)(p - eo) * so;
        const long long rec = h.at(s);
        const int j = nebor[s], io = first + o;
        const double3 d = sub3(pos[io], pos[j]);
        const double ir = rad[io], jr = rad[j];
        const double dl = len3(d);
        const double gap = dl - ir - jr;
        touch = gap < 0.0 && rec >= 0;
        int fl = touch ? 1 : 0;
        if (force_cap == 1 && rec >= 0) {
          /* an existing bridge, or one forming this step */
          const bool film = gap < law.film * (ir + jr);
          bridge = film || h.brg(rec) != 0;
          if (film) fl |= 2;
        }
        if (touch || bridge) { /* both use the normal and the reduced radius */
          const double3 u = div3(d, dl);
          sm.ux[e] = u.x;
          sm.uy[e] = u.y;
          sm.uz[e] = u.z;
          sm.ijr[e] = ir * jr / (ir + jr);
        }
        sm.gap[e] = gap;
        sm.rec[e] = rec;
        sm.j[e] = j;
        sm.owner[e] = (unsigned char)o;
        sm.flags[e] = (unsigned char)fl;
      }
      const unsigned mc = __ballot_sync(FULL, touch), mb = __ballot_sync(FULL, bridge);
      if (touch) sm.contact[nc + __popc(mc & below)] = (unsigned short)e;
      if (bridge) sm.bridge[nb + __popc(mb & below)] = (unsigned short)e;
      nc += __popc(mc);
      nb += __popc(mb);
    }
    __syncwarp();
    /* the contact law */
    for (int t = lane; t < nc; t += 32) {
      const int e = sm.contact[t];
      const int io = first + sm.owner[e], j = sm.j[e];
      const double ir = rad[io], jr = rad[j];
      const double3 u = d3(sm.ux[e], sm.uy[e], sm.uz[e]);
      const double3 cpv =
          sub3(sub3(vel[io], vel[j]), cross3(add3(mul3(angvel[io], ir), mul3(angvel[j], jr)), u));
      const double ijRad = sm.ijr[e];
      HistRec rec = h.load(sm.rec[e]);
      double3 dF, dM;
      double dR;
      contact_law64(law, ijRad, -sm.gap[e], u, cpv, rec, ir, dF, dM, dR);
      h.store(sm.rec[e], rec);
      sm.out[0][e] = dF.x;
      sm.out[1][e] = dF.y;
      sm.out[2][e] = dF.z;
      sm.out[3][e] = dM.x;
      sm.out[4][e] = dM.y;
      sm.out[5][e] = dM.z;
      sm.out[6][e] = dR;
    }
    __syncwarp(); /* the normals have been read: a bridge's force takes their place */
    for (int t = lane; t < nb; t += 32) {
      const int e = sm.bridge[t];
      const int io = first + sm.owner[e], j = sm.j[e];
      const double gap = sm.gap[e];
      const bool film = (sm.flags[e] & 2) != 0;
      const int brg0 = h.brg(sm.rec[e]);
      int brg = film ? 1 : brg0;
      const double Splus = gap < 0 ? 0.0 : gap;
      const double effR = 2 * sm.ijr[e]; /* 2 r_i r_j / (r_i + r_j), exactly */
      double fcap = 0.0;
      if (ref_liquid) {
        double ijVol = pvol[io] + pvol[j];
        if (!film && gap > 0.99 * pow(ijVol, 0.33)) brg = 0;
        if (brg == 1) {
          ijVol = ijVol * 8.0;
          fcap = fcap64(Splus, ijVol, effR, k.lqd);
        }
      } else {
        /* per-contact volume and contact angle (liquid.cuh) */
        const int idi = id ? id[io] : io, idj = id ? id[j] : j;
        const double th = 0.5 * ((double)cap_theta(idi, lm.seed, lm.theta_max) +
                                 (double)cap_theta(idj, lm.seed, lm.theta_max));
        const double V = pair_bridge_volume(lm, idi, idj, min(rad[io], rad[j]));
        if (!film && gap > rupture64(V, th)) brg = 0;
        if (brg == 1) fcap = 2 * kPiRef * effR * k.lqd.stension * willett64(max(k.lqd.gapmn, Splus), 8.0 * V, th);
      }
      if (brg != brg0) h.set_brg(sm.rec[e], brg);
      if (brg == 1) {
        const double3 fc = smul3(-1.0 * fcap, d3(sm.ux[e], sm.uy[e], sm.uz[e]));
        sm.ux[e] = fc.x;
        sm.uy[e] = fc.y;
        sm.uz[e] = fc.z;
        sm.flags[e] |= 4;
      }
    }
    __syncwarp();
    /* every sphere's entries of the chunk, in neighbour order */
    for (int p = max(excl, c0); p < min(incl, cend); p++) {
      const int e = p - c0, fl = sm.flags[e];
      if (fl & 1) {
        F = add3(F, d3(sm.out[0][e], sm.out[1][e], sm.out[2][e]));
        M = add3(M, d3(sm.out[3][e], sm.out[4][e], sm.out[5][e]));
        R = R + sm.out[6][e];
        ncontact++;
      }
      if (fl & 4) {
        F = add3(F, d3(sm.ux[e], sm.uy[e], sm.uz[e]));
        wet = wet + 1;
        if (!(fl & 1)) nbridge++;
      }
    }
    __syncwarp();
  }
  if (live) {
    force[i] = F;
    mom[i] = M;
    rmom[i] = R;
    lqd[i] = wet;
  }
  if (counters) {
    const unsigned c[3] = {(unsigned)nn, (unsigned)ncontact, (unsigned)nbridge};
#pragma unroll
    for (int t = 0; t < 3; t++) {
      const unsigned v = __reduce_add_sync(FULL, c[t]);
      if (lane == 0 && v) atomicAdd(&counters[t], (unsigned long long)v);
    }
  }
}

/* CirPWInterG (kernel.cu:958-1023).  The reference's particle-0 thread moves
 * the top wall while other threads read it; here a one-thread launch moves it
 * first and every particle sees the moved wall. */
/* each sphere's share of liquid, vol (2r)^3 / max(bridges last step, 12)
 * (kernel.cu:429-434, :511-518): a per-sphere value the reference recomputes for
 * every neighbour entry; computed once here by the same operations */
__global__ void k_liquid_share(const double* __restrict__ rad, const int* __restrict__ lqd_old,
                               double* __restrict__ pvol, int n, DevConsts k) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int nl = lqd_old[i];
  if (nl < 12) nl = 12;
  pvol[i] = k.lqd.vol * cube(rad[i] * 2) / nl;
}

__global__ void k_move_top_wall(CylinderBC* cyl, double dt) {
  if (blockIdx.x == 0 && threadIdx.x == 0) cyl->Tw = cyl->Tw + cyl->topv * dt;
}

/* One listed sphere in six lists a wall and one in fifteen touches it, those lie
 * together, and an FP64 instruction costs a warp the same for one lane as for 32.
 * So a block sifts kWallEach times as many spheres as it has threads, 32 at a time
 * from all over the bed, by an FP32 gap (a wall farther than its error bound adds
 * nothing), and takes those left as one dense list, a sphere's walls in order.
 * A thread per sphere: 135 us on the packed 200k bed, with 3.4 of 32 lanes active;
 * a block's own spheres compacted per wall slot 50, waiting at barriers; this 38. */
constexpr int kWallThreads = 128, kWallEach = 3;
template <class HA>
__global__ void __launch_bounds__(kWallThreads) k_wall_force64(
    const double3* __restrict__ pos, const double3* __restrict__ vel, const double3* __restrict__ angvel,
    double3* __restrict__ force, double3* __restrict__ mom, double* __restrict__ rmom,
    const double* __restrict__ rad, const CylinderBC* __restrict__ cyl, HA h,
    const int* __restrict__ nwall, const int* __restrict__ wlist, size_t pitch, int n, int NP, LawK64 law,
    unsigned long long* __restrict__ counters) {
  __shared__ int list[kWallThreads * kWallEach];
  __shared__ int listed;
  if (threadIdx.x == 0) listed = 0;
  __syncthreads();
  const CylinderBC c = *cyl;
  /* the gap from FP32 copies is within tol of the exact one: a few FP32 ulps of
   * the largest coordinate involved, taken 8x */
  auto near = [&](int w, float px, float py, float pz, float ri) {
    float gc, tol;
    if (w == 0 || w == 1) {
      const float wz = d2f(w == 0 ? c.Tw : c.Bw);
      gc = fabsf(pz - wz) - ri;
      tol = 1e-6f * (fabsf(pz) + fabsf(wz) + ri);
    } else if (w == 2) {
      const float cx = d2f(c.cir.x), cy = d2f(c.cir.y), Rf = d2f(c.R);
      const float dx = px - cx, dy = py - cy;
      gc = fabsf(sqrtf(dx * dx + dy * dy) - Rf) - ri;
      tol = 1e-6f * (fabsf(px) + fabsf(py) + fabsf(cx) + fabsf(cy) + Rf + ri);
    } else {
      return false;
    }
    return !(gc > tol);
  };
#pragma unroll
  for (int e = 0; e < kWallEach; e++) {
    const int i = ((e * (kWallThreads / 32) + (threadIdx.x >> 5)) * gridDim.x + blockIdx.x) * 32 + (threadIdx.x & 31);
    const int nw = i < n ? nwall[i] : 0;
    if (nw <= 0) continue;
    const double3 p = pos[i];
    const float px = d2f(p.x), py = d2f(p.y), pz = d2f(p.z), ri = d2f(rad[i]);
    const int* row = (const int*)((const char*)wlist + (size_t)i * pitch);
    bool any = false;
    for (int a = 0; a < nw; a++) any = any || near(row[a], px, py, pz, ri);
    if (any) list[atomicAdd(&listed, 1)] = i;
  }
  __syncthreads();
  int nc = 0;
  for (int t = threadIdx.x; t < listed; t += kWallThreads) {
    const int q = list[t];
    const int nw = nwall[q];
    const int* rq = (const int*)((const char*)wlist + (size_t)q * pitch);
    const double3 ip = pos[q];
    const double ir = rad[q];
    const float px = d2f(ip.x), py = d2f(ip.y), pz = d2f(ip.z), rf = d2f(ir);
    double3 jv = make_double3(0.0, 0.0, 0.0); /* persists across walls (kernel.cu:980) */
    for (int a = 0; a < nw; a++) {
      const int w = rq[a];
      if (w == 0) jv.z = c.topv;
      if (!near(w, px, py, pz, rf)) continue;
      double3 jp;
      if (w == 2) {
        /* the reference's pow(pow(dx, 2) + pow(dy, 2), 0.5) (kernel.cu:1009) as the
         * correctly rounded squares and square root it denotes: CUDA's pow has up
         * to 2 ulp of error, and the wall overlap r - |p - jp| amplifies an error
         * of dist by R / overlap (~10^4 here) */
        const double ddx = c.cir.x - ip.x, ddy = c.cir.y - ip.y;
        const double dist = sqrt(ddx * ddx + ddy * ddy);
        const double cs = (ip.x - c.cir.x) / dist;
        const double sn = (ip.y - c.cir.y) / dist;
        jp = make_double3(c.R * cs + c.cir.x, c.R * sn + c.cir.y, ip.z);
      } else {
        jp = make_double3(ip.x, ip.y, w == 0 ? c.Tw : c.Bw);
      }
      const double3 d = sub3(ip, jp);
      const double len = len3(d);
      const double gap = len - ir;
      if (!(gap < 0.0)) continue;
      const double3 u = div3(d, len);
      const double3 cpv = sub3(sub3(vel[q], jv), cross3(mul3(angvel[q], ir), u));
      const long long ine = (long long)a * NP + q;
      HistRec rec = h.load(ine);
      double3 dF, dM;
      double dR;
      contact_law64(law, ir, -gap, u, cpv, rec, ir, dF, dM, dR);
      h.store(ine, rec);
      force[q] = add3(force[q], dF);
      mom[q] = add3(mom[q], dM);
      rmom[q] = rmom[q] + dR;
      nc++;
    }
  }
  if (counters && nc) atomicAdd(&counters[3], (unsigned long long)nc);
}

/* UpdateSystemG (kernel.cu:563-606) */
__global__ void k_update64(const double* __restrict__ rad, double3* __restrict__ pos, double3* __restrict__ vel,
                           double3* __restrict__ angvel, const double3* __restrict__ force,
                           const double3* __restrict__ mom, double* __restrict__ rmom, int* __restrict__ flag,
                           double* __restrict__ pmove, int n, double dt, double search_gap) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double r = rad[i];
  const double mass = cube(2.0 * r);
  double3 v = vel[i];
  const double3 f = force[i];
  v.x = v.x + f.x * dt / mass;
  v.y = v.y + f.y * dt / mass;
  v.z = v.z + f.z * dt / mass;
  vel[i] = v;
  pos[i] = add3(pos[i], mul3(v, dt));
  const double pm = pmove[i] + len3(v) * dt;
  pmove[i] = pm;
  const double inert = 0.1 * pow5(2.0 * r);
  double3 w = angvel[i];
  const double3 m = mom[i];
  w.x = w.x + m.x * dt / inert;
  w.y = w.y + m.y * dt / inert;
  w.z = w.z + m.z * dt / inert;
  const double rm = rmom[i] * dt / inert;
  rmom[i] = rm;
  const double wl = len3(w);
  if (wl > 1.0e-7) {
    const double s = rm / wl;
    w = mul3(w, (1.0 - (s < 1.0 ? s : 1.0)));
  }
  angvel[i] = w;
  if (pm > (0.3 * search_gap)) atomicAdd(flag, 1);
}

}  // namespace

dem_status var_init(double3* force, double3* mom, double* rmom, int* lqd, int* lqd_old, int n,
                    cudaStream_t stream) {
  if (n <= 0) return DEM_OK;
  k_var_init<<<grid_for(n, 256), 256, 0, stream>>>(force, mom, rmom, lqd, lqd_old, n);
  return cuda_check(cudaGetLastError(), "var_init launch");
}

template <class H>
dem_status pp_force64(const double3* pos, const double3* vel, const double3* angvel, const double* rad,
                      const int* nebor, const int* plevel, const int* level_npars, const int* level_nnebors,
                      const int* nebor_idx, H h, const int* num_nebor, int* lqd, const int* lqd_old,
                      double3* force, double3* mom, double* rmom, int n, int force_cap, int stage,
                      const DevConsts& k, unsigned long long* counters, double* pvol, cudaStream_t stream,
                      const int* id, LiquidModel lm) {
  if (n <= 0) return DEM_OK;
  using HA = typename Acc<H>::T;
  if (force_cap == 1 && lm.mode == 0) {
    if (!pvol) return fail(DEM_ERR_ARG, "pp_force64: the liquid shares need an n-double scratch array");
    k_liquid_share<<<grid_for(n, 256), 256, 0, stream>>>(rad, lqd_old, pvol, n, k);
  }
  const LawK64 law = make_law64(k.cal, true, k.mat[0].dmpn * k.mat[0].dmpn, stage, k.mat[0].rfrc, k.prm.dt,
                                k.lqd.layer);
  k_pp_force64<HA><<<grid_for(n, 32 * kPpWarps), 32 * kPpWarps, kPpSmem, stream>>>(
      pos, vel, angvel, rad, nebor, plevel, level_npars, level_nnebors, nebor_idx, Acc<H>::make(h), num_nebor, lqd,
      force, mom, rmom, n, force_cap, law, k, counters, id, lm, pvol);
  return cuda_check(cudaGetLastError(), "pp_force64 launch");
}

template <class H>
dem_status wall_force64(const double3* pos, const double3* vel, const double3* angvel, double3* force,
                        double3* mom, double* rmom, const double* rad, CylinderBC* cyl, H h,
                        const int* nwall, const int* wlist, size_t pitch, int n, int NP, int stage,
                        const DevConsts& k, unsigned long long* counters, bool move_wall,
                        cudaStream_t stream) {
  if (n <= 0) return DEM_OK;
  using HA = typename Acc<H>::T;
  if (move_wall) k_move_top_wall<<<1, 32, 0, stream>>>(cyl, k.prm.dt);
  const LawK64 law = make_law64(k.pwcal, false, k.mat[0].dmpn * k.mat[1].dmpn, stage, k.mat[0].rfrc, k.prm.dt,
                                k.lqd.layer);
  k_wall_force64<HA><<<grid_for(n, kWallThreads * kWallEach), kWallThreads, 0, stream>>>(
      pos, vel, angvel, force, mom, rmom, rad, cyl, Acc<H>::make(h), nwall, wlist, pitch, n, NP, law, counters);
  return cuda_check(cudaGetLastError(), "wall_force64 launch");
}

template dem_status pp_force64<HistSoA>(const double3*, const double3*, const double3*, const double*, const int*,
                                        const int*, const int*, const int*, const int*, HistSoA, const int*, int*,
                                        const int*, double3*, double3*, double*, int, int, int, const DevConsts&,
                                        unsigned long long*, double*, cudaStream_t, const int*, LiquidModel);
template dem_status pp_force64<PairSet>(const double3*, const double3*, const double3*, const double*, const int*,
                                        const int*, const int*, const int*, const int*, PairSet, const int*, int*,
                                        const int*, double3*, double3*, double*, int, int, int, const DevConsts&,
                                        unsigned long long*, double*, cudaStream_t, const int*, LiquidModel);
template dem_status wall_force64<HistSoA>(const double3*, const double3*, const double3*, double3*, double3*,
                                          double*, const double*, CylinderBC*, HistSoA, const int*, const int*,
                                          size_t, int, int, int, const DevConsts&, unsigned long long*, bool,
                                          cudaStream_t);
template dem_status wall_force64<HistAoS>(const double3*, const double3*, const double3*, double3*, double3*,
                                          double*, const double*, CylinderBC*, HistAoS, const int*, const int*,
                                          size_t, int, int, int, const DevConsts&, unsigned long long*, bool,
                                          cudaStream_t);

dem_status update64(const double* rad, double3* pos, double3* vel, double3* angvel, const double3* force,
                    const double3* mom, double* rmom, int* flag, double* pmove, int n, const DevConsts& k,
                    cudaStream_t stream) {
  if (n <= 0) return DEM_OK;
  k_update64<<<grid_for(n, 256), 256, 0, stream>>>(rad, pos, vel, angvel, force, mom, rmom, flag, pmove, n,
                                                  k.prm.dt, k.prm.SearchGap);
  return cuda_check(cudaGetLastError(), "update64 launch");
}

}  // namespace dem
