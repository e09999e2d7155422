// Decides on the device which kernel runs the chains of a launch, where neither is the faster one for every state.
//
// A scheduled kernel (cemc_sched.cu, cemc_schedt.cu) takes a time that does not depend on what is accepted; the
// speculative forms (cemc_mc.cu) commit a round up to the first trial that an accepted one touches, so they are the
// faster ones for chains that accept little, the more so the fewer trials touch one another by chance.  And trials
// of swaps that share a slot of a species' site list run one after the other in the scheduled kernel, accepted or
// not, which dilute species make frequent.  What decides, the acceptance so far and the composition, is in device
// memory, where a captured launch finds it anew at each replay.  Both kernels leave the same bits.
//
// One block looks at all chains (the slowest chain of a launch sets its time) and marks the status word of every
// chain that has trials; the two kernels follow on the stream, and each leaves the chains marked for the other.
// The decision cannot be taken by the two kernels themselves: the first one's chains change the counters.
#include "cemc_device.cuh"
#include "cemc_route.h"

namespace cemc {

__global__ void route_kernel(RunArgs a, int n_sym, bool swaps, Route q) {
  bool hot = false, warm = false, over_hot = false, over_warm = false, over = false;
  auto idle = [&](int c) { return a.chain_trials && a.chain_trials[c] <= a.chunk_offset; };
  for (int c = threadIdx.x; c < a.n_chains; c += blockDim.x) {
    if (idle(c)) continue;
    if (a.accum) {
      const cemc_accum *ac = a.accum + (a.accum_slot ? a.accum_slot[c] : c);
      const bool known = ac->n_samples >= kRouteKnown;
      hot |= known && (double)ac->n_accept >= q.hot * (double)ac->n_samples;
      warm |= known && (double)ac->n_accept >= q.warm * (double)ac->n_samples;
    }
    double share = 0.0;  // probability that two trials draw the same list slot of a species
    if (swaps) {
      int present = 0;
      for (int s = 0; s < n_sym; ++s) {
        const int n = a.trk_count[(size_t)c * n_sym + s];
        present += n > 0;
        share += n > 0 ? 1.0 / (double)n : 0.0;
      }
      share *= 4.0 / (double)(present * present);  // each species is one of a trial's two with 2 / present
    }
    over_hot |= share > q.share_hot;
    over_warm |= share > q.share_warm;
    over |= share > q.share;
  }
  hot = __syncthreads_or(hot);
  warm = __syncthreads_or(warm);
  over_hot = __syncthreads_or(over_hot);
  over_warm = __syncthreads_or(over_warm);
  over = __syncthreads_or(over);
  const int32_t mark =
      (hot && !over_hot) || (warm && !over_warm) || !over ? kRouteScheduled : kRouteSpeculative;
  for (int c = threadIdx.x; c < a.n_chains; c += blockDim.x)
    if (!idle(c)) a.status[c] = mark;
}

cudaError_t launch_route(const DevGeo &g, const RunArgs &a, bool swaps, const Route &q, cudaStream_t st) {
  route_kernel<<<1, 256, 0, st>>>(a, g.n_sym, swaps, q);
  return cudaGetLastError();
}

}  // namespace cemc
