/*
 * engine.h -- the native engine's context (dem_ctx), shared by engine.cu and mixed.cu.
 *
 * Device memory layout (N particles, S neighbour slots, C cells):
 *  - particle state in cell order (reorder = 1) or caller order: pos, vel,
 *    angv (FP64 double3), rad, pmove (FP64), lqd (bridge count of the last
 *    step), id (caller id), plevel, nidx (rank inside the level: the slot
 *    column), plus tmp_* copies used while permuting;
 *  - neighbour lists: nebor[S] level/slot-major (slot(q,k) = base[L] +
 *    k*npars[L] + nidx[q], coalesced across consecutive particles for a fixed
 *    k), num_nebor[N]; wall lists wlist[N][3], nwall[N];
 *  - the pair list (pairs.cuh): every pair of neighbours once, with its record (48
 *    bytes in mixed precision, two of 64 in FP64) and bridge bytes, in two sets that
 *    a rebuild alternates between
 *    (fixed pointers, so a rebuild can sit inside a CUDA graph); each slot's
 *    pair index; the pairs' results of the running step;
 *  - 3N wall records (slot (a, q) at a*N + q), with *_old copies a rebuild
 *    writes first and carries over from;
 *  - mixed precision: FP32 shadow state read by neighbours, double-buffered
 *    per step (see mixed.cu).
 */
#pragma once

#include <cuda_runtime.h>

#include <utility>
#include <vector>

#include "dem_internal.h"
#include "pairs.cuh"

namespace dem {

struct MixedState; /* mixed.cu */

/* device-side step chaining (chain.cu): the device-launchable graphs of 1, 2, 4
 * and 8 steps and of a rebuild, per shadow parity, the countdown of the running chain,
 * and the move flags of a graph's steps but the last */
constexpr int kChainSizes = 4, kChainMost = 1 << (kChainSizes - 1);
struct StepCtl {
  int left;
  int flag[kChainMost - 1];
  cudaGraphExec_t step[kChainSizes][2], rebuild[2];
};

struct EngineBufs {
  /* particle state */
  double3 *pos, *vel, *angv;
  double *rad, *pmove;
  int *lqd, *lqd_old, *id, *plevel, *nidx;
  int* inv; /* inv[id[q]] = q: the cell position of each caller index, renewed at every rebuild */
  double3 *tmp_pos, *tmp_vel, *tmp_angv;
  double3* tmp_out; /* 2 N: staging of exported arrays beside the three above */
  double* tmp_rad;
  int *tmp_lqd, *tmp_id, *tmp_plevel;
  double3 *force, *mom;
  double* rmom;
  /* lists */
  int *nebor, *num_nebor, *wlist, *nwall;
  int *wlist_old, *nwall_old;
  /* the pair list with its history, and each pair's result of the running
   * step (mixed.cu / step64.cu) */
  PairSet ps;
  void* pair_out;
  /* wall history */
  ContactRec *wrec, *wrec_old;
  /* sort */
  int *sorted_hash, *sorted_src, *cell_start, *cell_end;
  int* cell_off; /* every cell's offset in sorted order, and the total (C + 1) */
  void* scratch;
  /* level tables */
  double* cell_size;
  int3* grid_size;
  int *ncell_idx, *npars, *nneb;
  double* level_size;
  CylinderBC* cyl; /* one cylinder, or one per system when systems are batched */
  /* batched systems (NULL for one system): system of each particle id, and
   * whether each system is wet */
  int *sys_of_id, *sys_wet;
  int n_sys;
  /* control words: flag (rebuild count from the integrator), need (host
   * request), err (error bits), counters (u64[8]) */
  int *flag, *need, *err;
  unsigned long long* counters;
};

}  // namespace dem

struct dem_ctx {
  dem_setup s;
  dem_options opt;
  int n;
  long long slots;
  cudaStream_t stream;
  /* host transfers: the copy stream and its events (xev[0]: the upload's
   * copies done; xev[1..5]: an export array gathered; xev[6]: the export's
   * copies done) */
  cudaStream_t xfer;
  cudaEvent_t xev[7];
  dem::DevConsts k;
  dem::LevelView lv;
  int lstart[DEM_MAX_LEVELS];
  dem::EngineBufs b;
  std::vector<void*> allocs;
  long long iter;
  long long rebuilds_host;
  double ctime;
  dem::MixedState* mx;
  /* CUDA graphs of opt.graph_steps steps, one per starting shadow parity, and
   * of one step (the remainder of a dem_step call) */
  cudaGraphExec_t graph_exec[2];
  cudaGraphExec_t graph_one[2];
  int parity; /* mixed: which shadow buffer the next step reads */
  int rebuild_due; /* the rebuild request on the device is known to be set */
  int radii_bounded; /* every radius is at most its level's size: the neighbour search may skip far rows */
  int moving_walls; /* a cylinder's top wall moves (topv != 0): moved before every step's wall contacts */
  /* device-side step chaining (mixed precision): 0 not built yet, 1 built (its
   * graphs anew if they were dropped since), -1 unavailable (the conditional-node
   * graphs run instead); the graphs (instantiated for device launch) and a
   * host-instantiated one-step graph without the countdown for dem_step(1)
   * (launched from the host, a device-launch graph starts ~5 us later); the control
   * block on the device; and, while a chained step is captured, the rebuild request
   * word that gates its kernels (NULL otherwise) */
  int chain_state;
  cudaGraphExec_t chain_step[dem::kChainSizes][2], chain_rebuild[2];
  cudaGraphExec_t chain_single_host[2];
  dem::StepCtl* chain_ctl;
  const int* step_gate; /* capture of a chain graph: the word that holds a step back, */
  int* body_order;      /* the sphere kernel's blocks, levels side by side (NULL: one level, or a small bed) */
  int* step_flag;       /* and its move flag (NULL: b.flag) */
  /* dem_profile_kernels: when set, the rebuild and the step record an event
   * after each of their kernels (NULL otherwise, and always during capture) */
  std::vector<std::pair<const char*, cudaEvent_t>>* marks;
  /* dem_e2e_parts: when set, six timing events the host-facing calls record
   * at their boundaries (upload start, upload copies done, import queued,
   * step queued, export start, export copies done); NULL otherwise */
  cudaEvent_t* trace;
  /* learned capillary closure (DEM_CAP_MLP): the staged network on the device
   * (NULL until dem_set_capnet) and the particles' contact angles */
  void* cap_w;
  float theta_max;
  unsigned long long theta_seed;
  /* the liquid-bridge model (dem_set_liquid_model; mode 0: the reference's) */
  dem::LiquidModel lm;
};

namespace dem {

/* engine.cu: wait for the context's steps and destroy its captured graphs; the
 * next dem_step captures them again, with the configuration of then */
void drop_graphs(dem_ctx* c);

/* mixed.cu */
dem_status mixed_create(dem_ctx* c);
void mixed_destroy(dem_ctx* c);
/* regenerate shadow buffer `which` from the FP64 master state */
struct ShadowOut;
/* threads per block of the step kernels */
int mixed_block_size(const dem_ctx* c);
/* Spheres from which the sphere kernel takes the levels side by side: about where
 * the pairs' results (40 bytes each, 4.3 pairs a sphere on a packed bed) and the
 * spheres' own state outgrow the L2.  Packed beds, us a step with and without:
 * 300,000 spheres 94.1 and 85.5, 500,000 143.9 and 143.9, 600,000 171.7 and 175.5,
 * 1,000,000 269.7 and 288.4, 2,000,000 520.2 and 569.9.  600,000 spheres with
 * other lists: dry 148.5 and 151.7, spread apart (3.2 pairs a sphere, no contacts)
 * wet 105.5 and 107.5, dry 97.4 and 97.5; without any pair 56.5 and 55.6. */
constexpr int kSideBySide = 600000;
ShadowOut mixed_shadow_out(const dem_ctx* c, int which);
const float4* mixed_motion(const dem_ctx* c, int which);
dem_status mixed_shadows(dem_ctx* c, int which, cudaStream_t s);
/* the last step's bridge counts to the master array */
dem_status mixed_bridge_counts(dem_ctx* c, int which, cudaStream_t s);
/* the neighbour build's FP32 prefilter over shadow buffer `which` */
Prefilter mixed_prefilter(dem_ctx* c, int which);
/* one step (pair kernel, sphere kernel) reading shadows `which`, writing shadows 1 - which */
dem_status mixed_step(dem_ctx* c, int which, cudaStream_t s);
/* a state import without a rebuild request: the host arrays already in the
 * tmp buffers, gathered into cell order with the shadow buffer `which`
 * rewritten, in one launch */
dem_status mixed_import(dem_ctx* c, int which, int has_v, int has_w, cudaStream_t s);
/* the same from mapped host arrays in caller order (hv, hw may be NULL: zero);
 * inv[i] is caller index i's cell position */
dem_status mixed_import_mapped(dem_ctx* c, int which, const int* inv, const double3* hp, const double3* hv,
                               const double3* hw, cudaStream_t s);
/* the names of the kernels mixed_step launches */
const char* mixed_step_kernel_name(const dem_ctx* c);
/* the compact list of the wall slots in use, from fresh wall lists */
dem_status mixed_wall_entries(dem_ctx* c, cudaStream_t s);
/* copy the last step's bridge counts from the shadow `which` to the master */
/* download the last step's force totals into the FP64 force array */
dem_status mixed_force_to_master(dem_ctx* c, cudaStream_t s);
/* the last step's forces, FP32, cell order (x, y, z, unused) */
const float4* mixed_force_shadow(const dem_ctx* c);

/* chain.cu: the chaining kernel after a step (tail-launches the rebuild and
 * the next step), the countdown, and the reset of the rebuild request */
dem_status chain_launch_tail(StepCtl* ctl, int* flag, int* need, int* err, int parity, int size, bool single,
                             cudaStream_t s);
dem_status chain_set_left(StepCtl* ctl, int nsteps, cudaStream_t s);
dem_status chain_clear_request(int* flag, int* need, cudaStream_t s);

}  // namespace dem
