// Full correlation-function recompute of a periodic box by bit planes (cemc_boxcf.cu).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "cemc_device.cuh"

namespace cemc {

constexpr int kBoxMaxL = 64;        // a row of sites along z is one word of up to 64 bits
constexpr int kBoxMaxCounts = 4096;  // counters per chain (shared memory)

// Tables of the recompute, built with the geometry.  The clusters of a periodic box fall into orbits
// under lattice translation: every sub-cluster of every site is one instance of an orbit, and all
// instances of an orbit sum over the cells to the same number, so one is evaluated and counted as often as
// it occurs.  Orbits whose instances carry the same terms form a pattern; per pattern the kernel counts
// species tuples (or, for a +1/-1 basis, odd products) over all its orbits and cells as exact integers.
// A pattern's orbits are cut into jobs of about kBoxJob per basis site, one warp each.
constexpr int kBoxJob = 8;
struct BoxCf {
  int ok;
  int pm1;         // +1/-1 basis: one counter per pattern (products equal to -1), else n_sym^points
  int n_jobs, n_ents, n_counts;
  int hx;          // largest |x offset| of an entry, in cells
  const int2 *job;           // [n_jobs] {points, first counter of the pattern}
  const int4 *ent;           // [n_ents] orbits by (job, basis site of the first point): offsets of points 1..3,
                             // packed (dx + 128) | (dy + 128) << 8 | (dz mod L) << 16 | basis << 24
  const int32_t *ent_start;  // [n_jobs * box_nb + 1]
  const int32_t *k_start;    // [n_eci + 1] ranges of k_count / k_w of each ECI
  const int32_t *k_count;    // counter
  const double *k_w;         // its weight in the ECI's sum over all sites
  const double *k_const;     // [n_eci] constant part of that sum
};

// CTAs per chain (a thread-block cluster) and shared memory of a launch; 0 CTAs: does not fit.
int boxcf_ctas(const DevGeo &g, const BoxCf &c, int n_chains, int n_sms, size_t max_smem, size_t *smem);
cudaError_t launch_boxcf(const DevGeo &g, const BoxCf &c, int n_chains, int ctas, size_t smem, const int8_t *occ,
                         const double *eci, double *cf, double *energy, cudaStream_t st);

}  // namespace cemc
