// Shared-memory layout of the scheduled table kernel (cemc_schedt.cu), computed identically on the host
// (to size the launch) and on the device.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "cemc_launch.h"

namespace cemc {

constexpr int kTickCap = 24;       // evaluating warps at most, one trial each per tick
constexpr int kTickHelpers = 6;    // planner, cutter, scanner, two summing warps, fetcher
// Two builds of the swaps: up to 16 evaluating warps with 80 registers a thread, up to 24 with 64.
constexpr int kTickWarps = 16;
constexpr int kTickRing = 256;     // trials in flight
constexpr int kTickWords = 2;      // words of 32 trials a trial's mask spans: its own and the one before
constexpr int kTickCuts = 32;      // booking rounds between the cutter and the scanner
constexpr int kTickRecs = 64;      // booking records between the scanner and the summing warps
constexpr int kTickBits = 14;      // log2 of the bits that mark the list slots in use (swaps)

struct TickLayout {
  size_t coef, bf, gstart, ftab, geos, sfx, acc, misc, pub, cuts, recs, draws, sites, rows, prev, mask, state, r_de, r_x,
      r_ds, r_dx, heads, lists, used, sp, occ;
  size_t sp_row, row_words;
  size_t total;
};

__host__ __device__ inline TickLayout tick_layout(const DevGeo &g, int swap, int rsize, int row_bits,
                                                  int head_bits) {
  TickLayout L;
  size_t o = 0;
  auto put = [&](size_t &at, size_t bytes) {
    at = o;
    o = align16(o + bytes);
  };
  const size_t RG = kTickRing, nb = (size_t)(swap ? 0 : g.n_bf);
  L.sp_row = align16((size_t)g.n_cols + 1);
  L.row_words = (size_t)g.cpad * (swap ? 2 : 1);
  put(L.coef, (size_t)rsize * g.n_eci);
  put(L.bf, (size_t)rsize * g.n_bf * g.n_sym);
  put(L.gstart, 4 * (CEMC_MAX_GROUPS + 1));
  put(L.ftab, (size_t)rsize * g.tab_len);
  put(L.geos, 16 * (size_t)g.n_geo);
  put(L.sfx, 8 * (size_t)(g.n_sym * g.n_sym));
  put(L.acc, 8 * (size_t)((2 + 3 * CEMC_MAX_BF) * 32));  // running sums [14][32]
  put(L.misc, 4 * 48);
  put(L.pub, 4 * 2 * 8);
  put(L.cuts, 8 * (size_t)kTickCuts);
  put(L.recs, (8 * (1 + CEMC_MAX_BF) + 8) * (size_t)kTickRecs);
  put(L.draws, 32 * RG);
  put(L.sites, 8 * RG);
  put(L.rows, 4 * (L.row_words << row_bits));  // of the trials listed and not finished
  put(L.prev, 4 * 2 * RG);
  put(L.mask, 4 * (size_t)kTickWords * RG);
  put(L.state, 2 * RG);
  put(L.r_de, (size_t)rsize * RG);
  put(L.r_x, (size_t)rsize * RG);
  put(L.r_ds, (size_t)rsize * RG * nb);
  put(L.r_dx, (size_t)rsize * RG * nb);
  put(L.heads, 4 * ((size_t)1 << head_bits));
  put(L.lists, 4 * 2 * kTickCap);
  put(L.used, swap ? ((size_t)1 << kTickBits) / 8 : 0);
  put(L.sp, (swap ? 2 : 1) * L.sp_row * kTickCap);
  put(L.occ, (size_t)g.n_sites);
  L.total = o;
  return L;
}

cudaError_t launch_tick(const DevGeo &g, const RunArgs &a, int move, int precision, size_t smem, cudaStream_t st);

}  // namespace cemc
