// Table form of the trial energy change, shared by the speculative (cemc_mc.cu) and the scheduled
// (cemc_schedt.cu) kernels.
#pragma once
#include "cemc_device.cuh"

namespace cemc {

// Entry `idx` of a chain's pattern tables, F(old, new, member species), in FP64.
__device__ inline double table_entry(const DevGeo &g, const double *eci, int idx) {
  const int S = g.n_sym;
  int p = 0;
  while (p + 1 < g.n_pat && g.pat_info[p + 1].y <= idx) ++p;
  const int4 pi = g.pat_info[p];
  int stride = 1;
  for (int j = 0; j < pi.x; ++j) stride *= S;
  const int li = idx - pi.y, on = li / stride, tup = li - on * stride;
  const int old_s = on / S, new_s = on - old_s * S;
  double v = 0.0;
  for (int t = pi.z; t < pi.w; ++t) {
    const int pk = g.pat_terms[t];
    const int k = pk & 0xff, dr = (pk >> 8) & 15;
    double prod = g.bf[dr * S + new_s] - g.bf[dr * S + old_s];
    int tt = tup;
    for (int j = 0; j < pi.x; ++j) {
      const int sj = tt % S;
      tt /= S;
      prod *= g.bf[((pk >> (12 + 4 * j)) & 15) * S + sj];
    }
    v += eci[k] * (double)g.n_sites * g.eci_w[k] * prod;
  }
  return v;
}

// Fixed-point quanta of a chain's tables (fx_quanta; one warp): `n` entries at most make up an energy change, and with
// `singlets` (flips) the singlets' change.  NaN counts as infinite.
template <typename R>
__device__ inline double table_quanta(const DevGeo &g, const R *ftab, const double *eci, int n, bool singlets, int lane) {
  const int S = g.n_sym;
  double most = 0.0, alone = 0.0, least = HUGE_VAL;
  for (int i = lane; i < g.tab_len; i += 32) most = fmax(most, isnan((double)ftab[i]) ? HUGE_VAL : fabs((double)ftab[i]));
  for (int k = lane; k < g.n_eci; k += 32) {
    const int kind = g.eci_kind[k];
    if (kind == 0 || (kind == 1 && !singlets)) continue;
    const double c = kind == 2 ? fabs(eci[k] * (double)g.n_sites * g.eci_w[k]) : fabs(eci[k]);
    if (c > 0.0) least = fmin(least, c);
    if (kind == 1) {
      const double *bf = g.bf + g.eci_dec[k] * S;
      double d = 0.0;
      for (int s = 0; s < S * S; ++s) d = fmax(d, fabs(bf[s % S] - bf[s / S]));
      alone += isnan(c) ? HUGE_VAL : c * d;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    most = fmax(most, __shfl_xor_sync(kFull, most, o));
    least = fmin(least, __shfl_xor_sync(kFull, least, o));
  }
  return fx_quanta<kFxTableLow>((double)n * most + warp_sum(alone), least);
}

// Energy change of one flip (or, TWO, of a swap's two flips) from the pattern
// tables: one lookup per cluster geometry, F[off + on * S^m + s1 + S s2 + S^2 s3]
// with on = old * S + new and the member species s_j of the geometry's columns.
// Geometries [lo, hi) are those of the changed site's translation group, packed as
// {c1 | c2 << 8 | c3 << 16, off, S^m, 0}.  Lane l adds geometries lo + l, lo + l + 32, .. in this order, then a butterfly.
//
// T is the entries' type, float or double; table_sum_fx() is the same for entries in fixed point (FP64 launches).
// (Four lookups in flight at a time, with the geometries in shared memory or in registers, measured slower:
// ladder 34.1 -> 35.1 and 43 ms, the loop is bound by its shared-memory wavefronts and instructions.)
template <typename T, bool TWO>
__device__ __forceinline__ T table_sum(int S, const uint4 *geos, const T *F, const int8_t *spa, const int8_t *spb,
                                       int on_a, int on_b, int lo, int hi, int lane) {
  const int S2 = S * S;
  T sum = (T)0;
  for (int i = lo + lane; i < hi; i += 32) {
    const uint4 e = geos[i];
    const int c1 = e.x & 0xff, c2 = (e.x >> 8) & 0xff, c3 = (e.x >> 16) & 0xff;
    sum += F[e.y + on_a * e.z + spa[c1] + S * spa[c2] + S2 * spa[c3]];
    if (TWO) sum += F[e.y + on_b * e.z + spb[c1] + S * spb[c2] + S2 * spb[c3]];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(kFull, sum, o);
  return sum;
}

// table_sum() of entries in fixed point, their low parts in an array of their own; the sum's low part is not carried.
// The low parts' lookups cost swaps 5 to 12 % (4 chains of 16384 sites, 6,000 swaps, with the high parts alone, about 50
// bits of the largest entry, / with both: 78 columns 2.01 / 2.25 ms, 86 columns 1.53 / 1.62 ms).  Flips of 4 x 1000 HCP
// sites, 10 sweeps: 3.38 ms by FP64 additions and the booker of then, 2.19 high parts alone, 2.04 both and fx_value().
template <bool TWO>
__device__ __forceinline__ FxNum table_sum_fx(int S, const uint4 *geos, const long long *F, const uint32_t *low,
                                              const int8_t *spa, const int8_t *spb, int on_a, int on_b, int lo, int hi,
                                              int lane) {
  const int S2 = S * S;
  FxNum sum{0, 0u};
  for (int i = lo + lane; i < hi; i += 32) {
    const uint4 e = geos[i];
    const int c1 = e.x & 0xff, c2 = (e.x >> 8) & 0xff, c3 = (e.x >> 16) & 0xff;
    const uint32_t at = e.y + on_a * e.z + spa[c1] + S * spa[c2] + S2 * spa[c3];
    sum.hi += F[at];
    sum.lo += low[at];
    if (TWO) {
      const uint32_t bt = e.y + on_b * e.z + spb[c1] + S * spb[c2] + S2 * spb[c3];
      sum.hi += F[bt];
      sum.lo += low[bt];
    }
  }
  sum.hi += (long long)(sum.lo >> kFxTableLow);
  sum.lo = __reduce_add_sync(kFull, sum.lo & ((1u << kFxTableLow) - 1u));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum.hi += __shfl_xor_sync(kFull, sum.hi, o);
  return sum;
}

}  // namespace cemc
