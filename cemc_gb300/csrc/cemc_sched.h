// Shared-memory layout of the scheduled flip kernel (cemc_sched.cu), computed identically on the
// host (to size the launch) and on the device.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "cemc_launch.h"
#include "cemc_spin.h"

namespace cemc {

constexpr int kSchedMaxThreads = 768;
constexpr int kSchedMaxCap = 64;       // trials per tick (four per evaluating warp)
constexpr int kSchedHelpers = 8;       // planner, follower, cutter, scanner, two summing and two fetching warps
constexpr int kSchedWords = 8;         // words of 32 trials a dependency mask spans: a trial's own and those before
constexpr int kSchedQueue = 256;       // hash hits between the lookups and the follower
constexpr int kSchedCuts = 32;         // booking rounds between the cutter and the scanner
constexpr int kSchedRecs = 64;         // booking records between the scanner and the summing warps
constexpr uint32_t kSchedNone = 0xffffffffu;  // published in place of the booked trials: the launch stops

struct SchedLayout {
  size_t cf, eci, w, coef, acc, sp_eci, sp_terms, sp_lane, misc, pub, cfsum, cuts, recs;
  size_t draws, uni, rows, prev, mask, r_acc, r_de, r_x, r_ds, heads, lists, queue, occ;
  size_t total;
};

// Rings: `ring_bits` for the trials in flight, `row_bits` for the neighbour rows of the unexecuted ones.
__host__ __device__ inline SchedLayout sched_layout(const DevGeo &g, int n_cl, int n_masks, int rsize, int cap,
                                                    int ring_bits, int row_bits, int head_bits) {
  SchedLayout L;
  size_t o = 0;
  const size_t K = (size_t)g.n_eci, RG = (size_t)1 << ring_bits;
  auto put = [&](size_t &at, size_t bytes) {
    at = o;
    o = align16(o + bytes);
  };
  put(L.cf, 8 * K);
  put(L.eci, 8 * K);
  put(L.w, 8 * K);
  put(L.coef, (size_t)rsize * K);
  put(L.acc, 8 * (size_t)(2 * (2 + 3 * CEMC_MAX_BF) * 32));  // [2 halves][14][32] at the end of the launch
  put(L.sp_eci, 32 * (size_t)n_cl);
  put(L.sp_terms, 16 * (size_t)n_masks);
  put(L.sp_lane, 4 * (9 + 8));
  put(L.misc, 4 * 16);
  put(L.pub, 4 * 2 * 16);
  put(L.cfsum, 8 * 10);  // committed changes of the cluster ECIs, then of the singlet
  put(L.cuts, 8 * (size_t)kSchedCuts);
  put(L.recs, 24 * (size_t)kSchedRecs);
  put(L.draws, 16 * RG);
  put(L.uni, 8 * RG);
  put(L.rows, 2 * ((size_t)1 << row_bits) * (size_t)g.cp16);
  put(L.prev, 4 * RG);
  put(L.mask, 4 * (size_t)kSchedWords * RG);  // [kSchedWords][RG]
  put(L.r_acc, RG);
  put(L.r_de, (size_t)rsize * RG);
  put(L.r_x, (size_t)rsize * RG);
  put(L.r_ds, RG);
  put(L.heads, 4 * ((size_t)1 << head_bits));
  put(L.lists, 2 * 2 * (size_t)cap);  // this tick's and the next one's
  put(L.queue, 2 * 2 * (size_t)kSchedQueue);
  put(L.occ, (size_t)g.n_sites);
  L.total = o;
  return L;
}

cudaError_t launch_sched(const DevGeo &g, const RunArgs &a, int precision, size_t smem, cudaStream_t st,
                         const SpinDev &sd);

}  // namespace cemc
