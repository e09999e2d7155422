// Which of two kernels runs a launch's chains, decided on the device (cemc_route.cu).
#pragma once
#include <cuda_runtime.h>

#include "cemc_launch.h"

namespace cemc {

// Marks in a chain's status word between the decision and the chain's launch (RunArgs::route).
constexpr int32_t kRouteScheduled = -1, kRouteSpeculative = -2;

// Calls of fewer trials a chain go to the speculative form undecided: the decision and the launch that finds
// nothing to do cost about 5 us.
constexpr uint64_t kRouteTrials = 2048;
// Trials in a chain's running sums from which its acceptance counts as known.
constexpr uint64_t kRouteKnown = 1024;

// The chains of a launch take the scheduled kernel when no chain's trials share a list slot with a probability above
// `share`, or `share_warm` if the hottest chain accepts at least `warm` of its trials, or `share_hot` if it
// accepts `hot`.  (Flips have no list slots: probability 0; a negative bound is never met.)
struct Route {
  double hot, share_hot, warm, share_warm, share;
};

cudaError_t launch_route(const DevGeo &g, const RunArgs &a, bool swaps, const Route &q, cudaStream_t st);

}  // namespace cemc
