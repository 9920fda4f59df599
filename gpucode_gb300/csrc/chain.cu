/*
 * chain.cu -- step chaining on the device for the mixed-precision engine.
 *
 * The reference decides on the host, before every step, whether the
 * neighbour lists must be rebuilt (main.cpp:467-470: a device-to-host read of
 * the move flag each step).  A CUDA-graph conditional node keeps that
 * decision on the device but costs about 11 us per step on the GB300 even
 * when the rebuild does not run -- an eighth of a 200k-sphere step.  Here the
 * steps launch one another from the device instead (device graph launch):
 *
 *   step graph S[G][p] = ([wall motion] -> [pair kernel] -> [sphere kernel]) x G
 *                        -> [k_chain]                              G = 1, 2, 4, 8
 *   rebuild graph R[p] = [k_clear_request] -> [the rebuild]
 *
 * (p: the parity of the first step's shadows.)  Every kernel of a step first
 * reads one word and does nothing if it is set: the rebuild request (need) in a
 * graph's first step, the move flag of the step before in the others.  A step
 * held back raises its own flag to -1, so that the rest of the graph is held
 * back too.  k_chain finds the first flag set.  If the graph's first step was
 * held back, it tail-launches R[p] and then the same graph again, so the step
 * runs on rebuilt lists.  Otherwise it counts the steps done and, while some are
 * left, tail-launches the largest graph that does not run too far, after R of its
 * parity if the last step done moved a sphere too far; the last step of a chain
 * leaves that request in need for the next call, which rebuilds before its
 * first step: the reference's order, the rebuild at the start of the step after
 * the flag.  A tail launch starts when the launching graph has completed, and
 * work queued on the stream after the host's launch waits for the whole chain.
 * A graph's end and the next one's start cost 4 to 6 us, a quarter of a step of
 * 5,000 spheres, which is why a graph holds several steps: one a graph 19.7 us a
 * step there and 70.6 on the packed 200k bed, up to two 16.6 and 66.3, four 16.4
 * and 64.1, eight 15.1 and 63.8, sixteen 14.9 and 63.3.  The kernels of a step
 * held back take 4 us, so more than eight would give back what they gain at the
 * first rebuild.
 *
 * For a one-step call the host launches a host-instantiated copy of S[1] without
 * the countdown: launched from the host, a graph instantiated for device launch
 * starts ~5 us later, and a kernel of the host copy tail-launches the device
 * graphs all the same: R and, as the rest of a chain of one step, S[1] (a chain of
 * many steps started from that copy measured ~1.5 us per step slower, so longer
 * calls launch the device copy).
 *
 * need and the flags are written only by k_chain and k_clear_request (need also
 * by the host between launches) and, its own flag, by a step's sphere kernel, so
 * every block of a kernel reads the same value in its word.
 *
 * This unit is compiled with relocatable device code (device-side
 * cudaGraphLaunch needs the device runtime); the step kernel is not, so its
 * register allocation is unchanged.
 */
#include "engine.h"

namespace dem {
namespace {

/* a tail launch that fails ends the chain early: error bit 8, which
 * dem_sync reports */
__device__ void tail(cudaGraphExec_t g, int* err) {
  if (cudaGraphLaunch(g, cudaStreamGraphTailLaunch) != cudaSuccess) atomicOr(err, 8);
}

/* the largest graph of at most `left` steps */
__device__ cudaGraphExec_t next_graph(const StepCtl* ctl, int left, int p) {
  int g = 0;
  while (g + 1 < kChainSizes && (2 << g) <= left) g++;
  return ctl->step[g][p];
}

__global__ void k_chain(StepCtl* ctl, int* flag, int* need, int* err, int p, int size, int single) {
  const int G = 1 << size;
  int done = G;
  bool moved = false;
  for (int s = 0; s < G; s++) {
    int* w = s == G - 1 ? flag : ctl->flag + s;
    const int f = *w;
    *w = 0;
    if (f > 0) {
      done = s + 1;
      moved = true;
    } else if (f < 0 && s == 0) {
      done = 0;
    }
  }
  if (done == 0) {
    /* the first step was held back: rebuild, then the same steps */
    if (single) ctl->left = 1;
    tail(ctl->rebuild[p], err);
    tail(ctl->step[size][p], err);
    return;
  }
  /* the countdown always moves, so the chain ends after `left` steps */
  const int left = single ? 0 : ctl->left - done;
  const int q = (p + done) & 1;
  if (!single) ctl->left = left;
  if (left <= 0) {
    if (moved) *need = 1;
    return;
  }
  if (moved) tail(ctl->rebuild[q], err);
  tail(next_graph(ctl, left, q), err);
}

__global__ void k_set_left(StepCtl* ctl, int n) { ctl->left = n; }

__global__ void k_clear_request(int* flag, int* need) {
  *flag = 0;
  *need = 0;
}

}  // namespace

dem_status chain_launch_tail(StepCtl* ctl, int* flag, int* need, int* err, int parity, int size, bool single,
                             cudaStream_t s) {
  k_chain<<<1, 1, 0, s>>>(ctl, flag, need, err, parity, size, single ? 1 : 0);
  return cuda_check(cudaGetLastError(), "step chain launch");
}

dem_status chain_set_left(StepCtl* ctl, int nsteps, cudaStream_t s) {
  k_set_left<<<1, 1, 0, s>>>(ctl, nsteps);
  return cuda_check(cudaGetLastError(), "step chain count");
}

dem_status chain_clear_request(int* flag, int* need, cudaStream_t s) {
  k_clear_request<<<1, 1, 0, s>>>(flag, need);
  return cuda_check(cudaGetLastError(), "rebuild request reset");
}

}  // namespace dem
