// Scheduled table kernel: unconstrained flips and swaps of any basis by the table form, one trial per
// warp, executed out of order.
//
// The chain is that of mc_kernel (cemc_mc.cu) and of the reference's _mc_step loop
// (cemc/mcmc/montecarlo.py:970-1038 over CEUpdater::calculate, cpp/src/ce_updater.cpp:313-406), and like the
// scheduled flip kernel (cemc_sched.cu) this one runs trials that do not touch one another in any order,
// with one barrier per tick and no trial committed before those it has to see.  A swap's sites are read from
// the species' site lists, so they are known only once the earlier trials on the same two list slots have
// run; therefore trials are listed one tick before they run, and which of them touch is found by the
// evaluation itself, whose gather of a row passes by every site that matters:
//
//   planner   at tick r makes the list of tick r + 1: trials of list r - 1 that were put off, then the next
//             trials of the stream (up to the first that shares a list slot with a listed, unfinished one:
//             its sites are not known yet); enters their sites into a hash of chains and copies their
//             neighbour rows into shared memory (cp.async)
//   evaluate  one listed trial per warp: species of the rows' sites, and in the same pass whether a site's
//             bucket holds a recent trial.  An earlier trial on one of those sites that had not run before
//             this tick puts the trial off; otherwise it is evaluated, tested and committed at once
//   cutter, scanner, summers, fetcher: as in cemc_sched.cu (the running sums are taken in the rounds of the
//             speculative form, so they are the same bit for bit)
//
// In a tick the earlier of two trials that touch runs and the later is put off, so occupations and list
// slots have one writer and no reader.  mc_kernel needs two SMs per chain (a cluster pair), conflict tables in
// device memory for large cells (atomics and a fence a round) and two dependent global loads of the site
// lists per trial, and evaluates conflicting trials again.
//
// Bound: the latency of one warp's evaluation (sites, species and bucket heads, hits, table lookups, test)
// and the barrier that waits for the slowest: 1.7 warp instructions a cycle, shared-memory wavefronts at 40 %
// of their rate.  A tick takes 7,000 to 9,000 cycles for 15 to 23 trials.  Half-warps with two trials per
// warp (twice the instructions per warp) took twice as long per tick; geometries of 8 bytes, both rows'
// species side by side, or separate loops for one, two and three members were slower than the plain loop.
// 48 x 131072-site binary ladder, one sweep: 34.1 -> 29.8 ms, on half the SMs; 64 uneven ternary chains, one sweep: 19.5
// -> 13.7 ms a step, which is the longest chain's (55,296 sites), 7.2 -> 4.8 ms where the steps of three such batches
// overlap; 32 ternary flip chains of 4000 sites 4.42 -> 3.78 ms.  Where it is not the faster one: cemc_route.h.
#include <cuda_runtime.h>

#include <type_traits>

#include "cemc_device.cuh"
#include "cemc_launch.h"
#include "cemc_schedt.h"
#include "cemc_table.cuh"

namespace cemc {

namespace {

__device__ __forceinline__ void tk_cp_async16(void *dst, const void *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void tk_cp_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Ring entry of a trial.  Flips: a = site, b = species word, grp = its translation group.  Swaps: a, b = list
// slots, grp = first species | second species << 8.
struct __align__(16) TickDraw {
  int32_t a, b;
  uint32_t grp, ua, ub, pad0, pad1, pad2;
};
// A booking round (up to 32 trials) on its way from the scanner to the summing warps.
template <typename A>
struct __align__(8) TickRec {
  A eoff, dsum[CEMC_MAX_BF];  // energy, and singlet changes of the launch, before it
  uint32_t x;                 // its first trial
  int32_t kh;                 // its trials
};
// state of a trial: bits 0..7 tick it ran in (never 0), 8 accepted, 9..12 new species of a flip
__device__ __forceinline__ uint32_t tick_tag(uint32_t r) { return r % 255u + 1u; }

enum { kTkDrawn = 0, kTkLow, kTkCut, kTkScanned, kTkBooked, kTkCuts, kTkRecs, kTkWords = 8 };
constexpr uint32_t kTickStop = 0xffffffffu;

}  // namespace

template <typename R, int MOVE, int WARPS>
__global__ void __launch_bounds__(32 * (WARPS + kTickHelpers), 1) tick_kernel(DevGeo g, RunArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr bool SWAP = MOVE == CEMC_MOVE_SWAP;
  constexpr int NR = SWAP ? 2 : 1;  // sites of a trial
  constexpr int NBF = SWAP ? 0 : CEMC_MAX_BF;
  constexpr bool FX = sizeof(R) == 8;
  const int CW = a.part;  // at most 32
  const TickLayout L = tick_layout(g, SWAP, (int)sizeof(R), a.row_bits, a.head_bits);
  constexpr uint32_t RG = kTickRing, rmask = RG - 1u, emask = 2u * RG - 1u;
  const uint32_t rowm = (1u << a.row_bits) - 1u, hmask = (1u << a.head_bits) - 1u;
  const int chain = blockIdx.x;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int N = g.n_sites, n_eci = g.n_eci, n_cols = g.n_cols, cpad = g.cpad, S = g.n_sym, n_bf = g.n_bf;
  const int role = warp - a.warps;  // helpers: 0 planner, 1 cutter, 2 scanner, 3 and 4 summers, 5 fetcher

  constexpr bool DF = (sizeof(R) == 4);
  using A = typename std::conditional<DF, df64, double>::type;
  constexpr int NACC = 2 + 3 * CEMC_MAX_BF;
  R *coef_s = reinterpret_cast<R *>(smem + L.coef);
  R *bf_s = reinterpret_cast<R *>(smem + L.bf);
  int32_t *gstart_s = reinterpret_cast<int32_t *>(smem + L.gstart);
  R *ftab = reinterpret_cast<R *>(smem + L.ftab);
  long long *ftab_fx = reinterpret_cast<long long *>(smem + L.ftab);
  uint32_t *ftab_low = reinterpret_cast<uint32_t *>(smem + L.total);  // low parts (a.fx_low), then sfx's
  uint4 *geos_s = reinterpret_cast<uint4 *>(smem + L.geos);
  long long *sfx_s = reinterpret_cast<long long *>(smem + L.sfx);  // [old * S + new] energy of the singlets' change
  A *lacc0 = reinterpret_cast<A *>(smem + L.acc);
  // misc: [0..2) n_acc, [2] species present, [3] status, [4] fault, [6..8) list lengths, [8..16) present ids,
  //       [16..24) site-list starts, [24..32) site-list counts
  int32_t *misc = reinterpret_cast<int32_t *>(smem + L.misc);
  uint64_t *n_acc_s = reinterpret_cast<uint64_t *>(misc);
  volatile int32_t *fault_s = misc + 4;
  volatile uint32_t *pub = reinterpret_cast<volatile uint32_t *>(smem + L.pub);
  uint2 *cuts = reinterpret_cast<uint2 *>(smem + L.cuts);
  TickRec<A> *recs = reinterpret_cast<TickRec<A> *>(smem + L.recs);
  TickDraw *draws = reinterpret_cast<TickDraw *>(smem + L.draws);
  int32_t *sites = reinterpret_cast<int32_t *>(smem + L.sites);       // [RG][2]
  int32_t *rows = reinterpret_cast<int32_t *>(smem + L.rows);         // [1 << row_bits][NR][cpad]
  volatile uint32_t *prev = reinterpret_cast<volatile uint32_t *>(smem + L.prev);  // entry 2 x + w: site w of trial x
  uint32_t *mask = reinterpret_cast<uint32_t *>(smem + L.mask);       // [kTickWords][RG]
  volatile uint16_t *state = reinterpret_cast<volatile uint16_t *>(smem + L.state);
  R *r_de = reinterpret_cast<R *>(smem + L.r_de);
  R *r_x = reinterpret_cast<R *>(smem + L.r_x);    // energy change of the round up to the trial
  R *r_ds = reinterpret_cast<R *>(smem + L.r_ds);  // [n_bf][RG] singlet change of the trial
  R *r_dx = reinterpret_cast<R *>(smem + L.r_dx);  // [n_bf][RG] of the round up to the trial
  uint32_t *heads = reinterpret_cast<uint32_t *>(smem + L.heads);
  uint32_t *lists = reinterpret_cast<uint32_t *>(smem + L.lists);  // [2][kTickCap]
  uint32_t *used = reinterpret_cast<uint32_t *>(smem + L.used);    // bits of list slots in use
  int8_t *occ = reinterpret_cast<int8_t *>(smem + L.occ);
  int32_t *trk = SWAP ? a.trk + (size_t)chain * N : nullptr, *loc = SWAP ? a.loc + (size_t)chain * N : nullptr;

  // A chain with no trials in this launch (an empty serving slot) leaves its state untouched.
  if (a.chain_trials && a.chain_trials[chain] <= a.chunk_offset) return;
  if (a.route && a.status[chain] != a.route) return;  // left to the other kernel

  // ---- prologue ---------------------------------------------------------------
  for (int k = tid; k < n_eci; k += blockDim.x) {
    const int kind = g.eci_kind[k];
    const double e = a.eci[(size_t)chain * n_eci + k];
    coef_s[k] = (R)(kind == 2 ? e * (double)N * g.eci_w[k] : (kind == 1 ? e : 0.0));
  }
  for (int i = tid; i < n_bf * S; i += blockDim.x) bf_s[i] = (R)g.bf[i];
  for (int q = tid; q <= g.n_groups; q += blockDim.x) gstart_s[q] = g.geo_start[q];
  for (int i = tid; i < g.n_geo; i += blockDim.x) geos_s[i] = g.geo_list[i];
  for (int i = tid; i < g.tab_len; i += blockDim.x) ftab[i] = (R)table_entry(g, a.eci + (size_t)chain * n_eci, i);
  for (int i = tid; i < NACC * 32; i += blockDim.x) lacc0[i] = acc_from<A>(0.0);
  for (uint32_t i = tid; i <= hmask; i += blockDim.x) heads[i] = 0u;
  for (int i = tid; i < 2 * kTkWords; i += blockDim.x) pub[i] = i % kTkWords >= kTkCuts ? 0u : RG;
  if (SWAP)
    for (int i = tid; i < (1 << kTickBits) / 32; i += blockDim.x) used[i] = 0u;
  {
    const int8_t *src = a.occ + (size_t)chain * N;
    if ((((uintptr_t)src | (uintptr_t)N) & 15) == 0) {
      for (int i = tid; i < N / 16; i += blockDim.x)
        reinterpret_cast<uint4 *>(occ)[i] = reinterpret_cast<const uint4 *>(src)[i];
    } else {
      for (int i = tid; i < N; i += blockDim.x) occ[i] = src[i];
    }
  }
  if (tid < NR * kTickCap)  // an absent member of a smaller cluster reads species 0
    (reinterpret_cast<int8_t *>(smem + L.sp) + L.sp_row * tid)[n_cols] = 0;
  if (tid == 0) {
    *n_acc_s = 0;
    misc[3] = 0;
    *fault_s = 0;
    misc[6] = misc[7] = 0;
    if (SWAP) {
      int np = 0;
      for (int s = 0; s < S; ++s) {
        const int cnt = a.trk_count[(size_t)chain * S + s];
        misc[16 + s] = a.trk_start[(size_t)chain * S + s];
        misc[24 + s] = cnt;
        if (cnt > 0) misc[8 + np++] = s;
      }
      misc[2] = np;
      if (np < 2) misc[3] = CEMC_ERR_STATE;
    }
  }
  const double kT = a.kT[chain];
  const float inv_kT = (float)(1.0 / kT);
  const uint32_t key = a.chain_key ? a.chain_key[chain] : (uint32_t)chain;
  uint64_t my_trials = a.n_trials;
  if (a.chain_trials) {
    const uint64_t total = a.chain_trials[chain];
    my_trials = total <= a.chunk_offset ? 0 : (total - a.chunk_offset < a.n_trials ? total - a.chunk_offset : a.n_trials);
  }
  const uint64_t t_first = a.trial[chain];
  // trials are numbered x = t - t_first + RG here: 0 is before every trial the hash can hold
  const uint32_t x_end = RG + (uint32_t)my_trials;
  const uint32_t r_max = 8u * (uint32_t)my_trials + 65536u;
  const int acc_row = a.accum_slot ? a.accum_slot[chain] : chain;
  const double e_ref = a.accum ? a.accum[acc_row].e_ref : 0.0;
  __syncthreads();
  if (misc[3] != 0) {
    if (tid == 0 && a.status) a.status[chain] = misc[3];
    return;
  }
  double fx_scale = 0.0, fx_inv = 0.0;  // FP64: table entries are multiples of fx_inv (0: they are FP64)
  float fx_kT = 0.f;
  if constexpr (FX) {
    if (a.fx_low)
      fx_scale = table_quanta(g, ftab, a.eci + (size_t)chain * n_eci, (SWAP ? 2 : 1) * g.n_geo, !SWAP, lane);
    __syncthreads();
    if (fx_scale != 0.0) {
      fx_inv = 1.0 / fx_scale;
      fx_kT = (float)(fx_inv / kT);
      for (int i = tid; i < g.tab_len; i += blockDim.x) {
        const FxNum f = fx_of<kFxTableLow>((double)ftab[i], fx_scale);
        ftab_fx[i] = f.hi;
        ftab_low[i] = f.lo;
      }
      for (int s = tid; s < S * S; s += blockDim.x) {
        double v = 0.0;
        for (int b = 0; b < n_bf; ++b)
          if (g.singlet_eci[b] >= 0) v += coef_s[g.singlet_eci[b]] * (bf_s[b * S + s % S] - bf_s[b * S + s / S]);
        const FxNum f = fx_of<kFxTableLow>(v, fx_scale);
        sfx_s[s] = f.hi;
        ftab_low[g.tab_len + s] = f.lo;
      }
    }
    __syncthreads();
  }

  if (role < 0) {
    // ---- evaluating warps -------------------------------------------------------
    const int n_chunks = (n_cols + 31) / 32;
    int8_t *sp_a = reinterpret_cast<int8_t *>(smem + L.sp) + NR * L.sp_row * warp, *sp_b = sp_a + L.sp_row;
    for (uint32_t r = 1;; ++r) {
      const int n = misc[6 + (r & 1)];
      if (warp < n) {
        const uint32_t x = lists[(r & 1) * kTickCap + warp], slot = x & rmask;
        // oldest trial that may not have run, or that a booking round can reach; entries of one batch (16
        // trials) can be out of order in a chain, hence the margin
        const uint32_t low = min(pub[((r & 1) ^ 1) * kTkWords + kTkLow], x - (uint32_t)(CW - 1)), elow = 2u * (low - 16u);
        const TickDraw d = draws[slot];
        const int sa = sites[2 * slot], sb = SWAP ? sites[2 * slot + 1] : -1;
        const int oa = SWAP ? (int)(d.grp & 255u) : (int)occ[sa];
        int na;
        if (SWAP) {
          na = (int)(d.grp >> 8);
        } else {
          const int k = (int)cemc_below((uint32_t)d.b, (uint32_t)(S - 1));
          na = k + (k >= oa);
        }
        const int32_t *row = rows + (size_t)(x & rowm) * NR * cpad;
        uint32_t hit = 0;  // bit 4 w + j: column lane + 32 j of row w; bit 8 + w: the site itself (lane 0)
#pragma unroll
        for (int w = 0; w < NR; ++w) {
          // a row's sites first, then their species and bucket heads
          int ns[4];
          int8_t sv[4];
          uint32_t hv[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (j < n_chunks) ns[j] = row[w * cpad + min(lane + 32 * j, n_cols - 1)];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (j < n_chunks) {
              sv[j] = occ[ns[j]];
              hv[j] = heads[(uint32_t)ns[j] & hmask];
            }
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (lane + 32 * j < n_cols) {
              // site b's neighbours see site a already changed
              (w ? sp_b : sp_a)[lane + 32 * j] = w && ns[j] == sa ? (int8_t)na : sv[j];
              hit |= (hv[j] >= elow ? 1u : 0u) << (4 * w + j);
            }
        }
        if (lane == 0) {
#pragma unroll
          for (int w = 0; w < NR; ++w) {
            const uint32_t hd = heads[(uint32_t)(w ? sb : sa) & hmask], own = 2u * x + (uint32_t)w;
            if ((hd == own ? prev[own & emask] : hd) >= elow) hit |= 256u << w;
          }
        }
        bool off = false;  // put off: an earlier trial on one of these sites has not run
        if (__any_sync(kFull, hit != 0)) {
          const uint32_t now = tick_tag(r);
          while (hit) {
            const int j = __ffs(hit) - 1;
            hit &= hit - 1;
            const int s = j < 8 ? row[(j >> 2) * cpad + lane + 32 * (j & 3)] : (j == 8 ? sa : sb);
            uint32_t e = *(volatile uint32_t *)&heads[(uint32_t)s & hmask];
            while (e >= elow) {
              const uint32_t y = e >> 1;
              if (y < x && sites[e & emask] == s) {
                const uint32_t k = (x >> 5) - (y >> 5);
                if (k < (uint32_t)kTickWords) atomicOr(&mask[k * RG + slot], 1u << (y & 31u));
                const uint32_t ran = state[y & rmask] & 255u;
                off |= ran == 0u || ran == now;
              }
              e = prev[e & emask];
            }
          }
          off = __any_sync(kFull, off);
        }
        __syncwarp();
        if (!off) {
          int ga = 0, gb = 0;
          if (g.n_groups > 1) {
            ga = SWAP ? (int)g.site_group[sa] : (int)d.grp;
            if (SWAP) gb = g.site_group[sb];
          }
          // energy change by `sum`, table_sum or table_sum_fx (the swap's two sites in one pass, unless their groups
          // differ: `add` of two)
          auto change = [&](auto sum, auto add) {
            const int on_a = oa * S + na, on_b = na * S + oa;
            if constexpr (!SWAP)
              return sum(std::false_type{}, sp_a, sp_a, on_a, 0, gstart_s[ga], gstart_s[ga + 1]);
            else if (ga == gb)
              return sum(std::true_type{}, sp_a, sp_b, on_a, on_b, gstart_s[ga], gstart_s[ga + 1]);
            return add(sum(std::false_type{}, sp_a, sp_a, on_a, 0, gstart_s[ga], gstart_s[ga + 1]),
                       sum(std::false_type{}, sp_b, sp_b, on_b, 0, gstart_s[gb], gstart_s[gb + 1]));
          };
          R de;
          FxNum de_fx{0, 0u};  // the energy change in units of fx_inv
          if (FX && fx_scale != 0.0) {
            FxNum f = change(
                [&](auto two, const int8_t *pa, const int8_t *pb, int on_a, int on_b, int lo, int hi) {
                  return table_sum_fx<two.value>(S, geos_s, ftab_fx, ftab_low, pa, pb, on_a, on_b, lo, hi, lane);
                },
                [](FxNum x, FxNum y) { return FxNum{x.hi + y.hi, x.lo + y.lo}; });
            if (!SWAP) f = FxNum{f.hi + sfx_s[oa * S + na], f.lo + ftab_low[g.tab_len + oa * S + na]};
            de_fx = fx_carry<kFxTableLow>(f.hi, (int)f.lo);
            de = (R)fx_value<kFxTableLow>(de_fx, fx_inv);
          } else {
            de = change(
                [&](auto two, const int8_t *pa, const int8_t *pb, int on_a, int on_b, int lo, int hi) {
                  return table_sum<R, two.value>(S, geos_s, ftab, pa, pb, on_a, on_b, lo, hi, lane);
                },
                [](R x, R y) { return x + y; });
            if (!SWAP)
              for (int b = 0; b < n_bf; ++b)
                if (g.singlet_eci[b] >= 0)
                  de += coef_s[g.singlet_eci[b]] * (bf_s[b * S + na] - bf_s[b * S + oa]);
          }
          if (lane == 0) {
            const int acc = FX && fx_scale != 0.0 ? metropolis_fx(de_fx, (double)de, d.ua, d.ub, kT, fx_kT)
                                                  : metropolis<R>(de, d.ua, d.ub, kT, inv_kT);
            if (acc) {
              occ[sa] = (int8_t)na;
              if (SWAP) {
                occ[sb] = (int8_t)oa;
                *(volatile int32_t *)(trk + d.a) = sb;
                *(volatile int32_t *)(trk + d.b) = sa;
                loc[sb] = d.a - misc[16 + oa];
                loc[sa] = d.b - misc[16 + na];
              }
            }
            r_de[slot] = de;
            if (!SWAP)
              for (int b = 0; b < n_bf; ++b) r_ds[b * RG + slot] = bf_s[b * S + na] - bf_s[b * S + oa];
            __threadfence_block();  // the cutter may see the state in this tick
            state[slot] = (uint16_t)(tick_tag(r) | ((uint32_t)acc << 8) | ((uint32_t)(SWAP ? 0 : na) << 9));
          }
          __syncwarp();
        }
      }
      __syncthreads();
      if (pub[(r & 1) * kTkWords + kTkBooked] >= x_end) break;  // all booked, or stopped (kTickStop)
    }
  } else if (role == 0) {
    // ---- planner ------------------------------------------------------------------
    const int cap = a.warps;  // trials per tick
    uint32_t next = RG;  // first trial that was never listed
    for (uint32_t r = 1;; ++r) {
      const volatile uint32_t *pp = pub + ((r & 1) ^ 1) * kTkWords;
      const uint32_t drawn = pp[kTkDrawn];
      uint32_t *list = lists + ((r + 1) & 1) * kTickCap;             // list r - 1, becomes list r + 1
      const uint32_t *running = lists + (r & 1) * kTickCap;          // list r
      const int n_old = misc[6 + ((r + 1) & 1)], n_run = misc[6 + (r & 1)];
      // trials of list r - 1 that were put off
      const uint32_t xo = lane < n_old ? list[lane] : 0u;
      const bool again = lane < n_old && (state[xo & rmask] & 255u) == 0u;
      const unsigned am = __ballot_sync(kFull, again);
      const int n_again = __popc(am);
      __syncwarp();
      if (again) list[__popc(am & ((1u << lane) - 1u))] = xo;
      __syncwarp();
      const uint32_t first_run = n_run > 0 ? running[0] : next, first_again = n_again > 0 ? list[0] : next;
      const uint32_t low = min(first_run, first_again);  // oldest trial that may not have run
      // list slots of the unfinished listed trials: of list r, of those put off, of those listed below
      constexpr uint32_t um = (1u << kTickBits) - 1u;
      int32_t held[6] = {-1, -1, -1, -1, -1, -1};
      if (SWAP) {
        if (lane < n_run) {
          const TickDraw &q = draws[running[lane] & rmask];
          held[0] = q.a;
          held[1] = q.b;
        }
        if (lane < n_again) {
          const TickDraw &q = draws[list[lane] & rmask];
          held[2] = q.a;
          held[3] = q.b;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (held[q] >= 0) atomicOr(&used[((uint32_t)held[q] & um) >> 5], 1u << (held[q] & 31));
        __syncwarp();
      }
      // the next trials of the stream, sixteen at a time: lane i and lane 16 + i work on trial next + i
      int n_list = n_again;
      TickDraw d2[2];
      int s2[2];
      bool can2[2];
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const uint32_t x = next + 16u * p + (uint32_t)(lane & 15);
        can2[p] = 16 * p + (lane & 15) < cap - n_again && x < drawn && x - low <= rowm;
        d2[p] = draws[x & rmask];
        s2[p] = -1;  // the lane's site: the first below lane 16, the second above
        if (SWAP) {
          if (can2[p]) s2[p] = *(volatile int32_t *)(trk + (lane < 16 ? d2[p].a : d2[p].b));
        } else if (can2[p] && lane < 16) {
          s2[p] = d2[p].a;
        }
      }
      bool stopped = false;  // a trial's sites are not known yet: no later one is listed before it
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const uint32_t x = next + (uint32_t)(lane & 15), slot = x & rmask;
        bool can = can2[p] && !stopped;
        const int s = s2[p];
        const int32_t my = lane < 16 ? d2[p].a : d2[p].b;  // the lane's list slot (swaps)
        if (SWAP) {
          bool maybe = false;
          if (can) maybe = (atomicOr(&used[((uint32_t)my & um) >> 5], 1u << (my & 31)) >> (my & 31)) & 1u;
          if (__any_sync(kFull, maybe)) {
            // some slots share a bit: compare them one by one
            bool same = false;
            for (int i = 0; i < 32; ++i) {
#pragma unroll
              for (int q = 0; q < 6; ++q) same |= my == __shfl_sync(kFull, held[q], i);
              const int32_t qm = __shfl_sync(kFull, can ? my : -1, i);
              same |= (i & 15) < (lane & 15) && my == qm;
            }
            unsigned bad = __ballot_sync(kFull, can && same);
            bad = (bad | (bad >> 16)) & 0xffffu;
            if (bad) {
              if ((lane & 15) >= __ffs(bad) - 1) can = false;
              stopped = true;
            }
          }
          if (p == 0 && can) held[4] = my;
        }
        const int n_new = __popc(__ballot_sync(kFull, can && lane < 16));
        if (n_new < 16) stopped = true;
        if (can && lane < 16) list[n_list + lane] = x;
        if (can && (SWAP || lane < 16)) sites[2 * slot + (lane >> 4)] = s;
        // neighbour rows (a flip's row is copied by its two lanes)
        const int site0 = SWAP ? s : __shfl_sync(kFull, s, lane & 15);
        if (can) {
          const int32_t *src = g.table + (size_t)site0 * cpad;
          int32_t *dst = rows + ((size_t)(x & rowm) * NR + (SWAP ? (lane >> 4) : 0)) * cpad;
          for (int q = SWAP ? 0 : 4 * (lane >> 4); q < cpad; q += SWAP ? 4 : 8) tk_cp_async16(dst + q, src + q);
        }
        // sites into the hash: first sites, then second ones, each in trial order
        __syncwarp();
#pragma unroll
        for (int w = 0; w < NR; ++w) {
          const bool mine = can && (lane >> 4) == w;
          const uint32_t e = 2u * x + (uint32_t)w, bucket = mine ? ((uint32_t)s & hmask) : 0u;
          const uint32_t old = mine ? heads[bucket] : 0u;
          if (mine) prev[e & emask] = old;
          __threadfence_block();  // an evaluation that sees the new head sees its chain
          __syncwarp();
          if (mine) heads[bucket] = e;
          __syncwarp();
          if (__any_sync(kFull, mine && *(volatile uint32_t *)&heads[bucket] != e)) {
            // two of these trials share a bucket: chain them in trial order
            const unsigned sm = __match_any_sync(kFull, mine ? bucket : 0x80000000u + lane);
            const unsigned before = sm & ((1u << lane) - 1u);
            if (mine) prev[e & emask] = before ? e - 2u * (uint32_t)(lane - (31 - __clz(before))) : old;
            __threadfence_block();
            __syncwarp();
            if (mine && (sm >> lane) == 1u) heads[bucket] = e;
            __syncwarp();
          }
        }
        next += (uint32_t)n_new;
        n_list += n_new;
      }
      if (SWAP) {
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (held[q] >= 0) used[((uint32_t)held[q] & um) >> 5] = 0u;
#pragma unroll
        for (int p = 0; p < 2; ++p)
          if (can2[p]) used[((uint32_t)(lane < 16 ? d2[p].a : d2[p].b) & um) >> 5] = 0u;
      }
      tk_cp_wait_all();
      if (lane == 0) {
        misc[6 + ((r + 1) & 1)] = n_list;
        pub[(r & 1) * kTkWords + kTkLow] = low;
      }
      __syncthreads();
      if (pub[(r & 1) * kTkWords + kTkBooked] >= x_end) break;
    }
  } else if (role == 1) {
    // ---- cutter: finished trials in trial order, in rounds of up to `part` --------------------------
    uint32_t x0 = RG, n_cuts = 0;
    for (uint32_t r = 1;; ++r) {
      const uint32_t drawn = pub[((r & 1) ^ 1) * kTkWords + kTkDrawn];
      const uint32_t full = n_cuts + kTickCuts / 2;  // two ticks of rounds fit the buffer
      while (n_cuts < full && x0 < x_end) {
        // the round at x0: finished trials, up to the first one an accepted trial of the round touches; a
        // round lies in two words of trials
        const int nv = (int)min((uint32_t)CW, x_end - x0);
        const uint32_t w0 = x0 & ~31u;
        uint32_t acc[2], fin[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const uint32_t x = w0 + 32u * q + lane, st = state[x & rmask];
          const bool in = x >= x0 && x < drawn;
          fin[q] = __ballot_sync(kFull, in && (st & 255u) != 0u);
          acc[q] = __ballot_sync(kFull, in && (st & 255u) != 0u && (st & 256u));
        }
        // a trial may finish in this very tick: its mask is complete before its state says so (the evaluator's
        // fence), and is read after it here
        __threadfence_block();
        const volatile uint32_t *vmask = mask;
        int done_n = 32, cut = 32;  // trials finished from x0 on, without a gap; first trial touched
#pragma unroll
        for (int q = 1; q >= 0; --q) {
          const uint32_t x = w0 + 32u * q + lane;
          uint32_t on = vmask[x & rmask] & acc[q];
          if (q == 1) on |= vmask[RG + (x & rmask)] & acc[0];
          const unsigned hit = __ballot_sync(kFull, x >= x0 && x < drawn && on != 0);
          const unsigned gap = __ballot_sync(kFull, x >= x0) & ~fin[q];
          if (hit) cut = (int)(w0 + 32u * q + __ffs(hit) - 1 - x0);
          if (gap) done_n = (int)(w0 + 32u * q + __ffs(gap) - 1 - x0);
        }
        const int ks = min(cut, nv);
        if (ks > done_n) break;  // the rest of the round is not finished
        if (lane == 0) cuts[n_cuts & (kTickCuts - 1)] = make_uint2(x0, (uint32_t)ks);
        ++n_cuts;
        x0 += (uint32_t)ks;
      }
      if (lane == 0) {
        pub[(r & 1) * kTkWords + kTkCut] = x0;
        pub[(r & 1) * kTkWords + kTkCuts] = n_cuts;
      }
      __syncthreads();
      if (pub[(r & 1) * kTkWords + kTkBooked] >= x_end) break;
    }
  } else if (role == 2) {
    // ---- scanner: energy and singlet changes of each round up to every trial ------------------------
    A eoff = acc_from<A>(a.energy[chain] - e_ref), dsum[CEMC_MAX_BF];  // before the round
#pragma unroll
    for (int b = 0; b < CEMC_MAX_BF; ++b) dsum[b] = acc_from<A>(0.0);
    uint64_t n_acc = 0;
    uint32_t n_recs = 0, n_cuts = 0;
    for (uint32_t r = 1;; ++r) {
      const volatile uint32_t *pp = pub + ((r & 1) ^ 1) * kTkWords;
      const uint32_t cuts_n = pp[kTkCuts], scanned = pp[kTkCut];
      for (; n_cuts < cuts_n; ++n_cuts) {
        const uint2 cq = cuts[n_cuts & (kTickCuts - 1)];
        const int kh = (int)cq.y;
        const uint32_t slot = (cq.x + (uint32_t)lane) & rmask;
        const bool acc = lane < kh && (state[slot] & 256u);
        const unsigned am = __ballot_sync(kFull, acc);
        n_acc += (uint64_t)__popc(am);
        if (lane == 0) {
          TickRec<A> rec;
          rec.eoff = eoff;
#pragma unroll
          for (int b = 0; b < CEMC_MAX_BF; ++b) rec.dsum[b] = dsum[b];
          rec.x = cq.x;
          rec.kh = kh;
          recs[n_recs & (kTickRecs - 1)] = rec;
        }
        ++n_recs;
        if (!a.accum) continue;
        R xs = acc ? r_de[slot] : (R)0, ds[NBF > 0 ? NBF : 1];
#pragma unroll
        for (int b = 0; b < NBF; ++b) ds[b] = (acc && b < n_bf) ? r_ds[b * RG + slot] : (R)0;
        if (am) {
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const R nx = __shfl_up_sync(kFull, xs, o);
            R nd[NBF > 0 ? NBF : 1];
#pragma unroll
            for (int b = 0; b < NBF; ++b)
              if (b < n_bf) nd[b] = __shfl_up_sync(kFull, ds[b], o);
            if (lane >= o) {
              xs += nx;
#pragma unroll
              for (int b = 0; b < NBF; ++b)
                if (b < n_bf) ds[b] += nd[b];
            }
          }
        }
        if (lane < kh) {
          r_x[slot] = xs;
#pragma unroll
          for (int b = 0; b < NBF; ++b)
            if (b < n_bf) r_dx[b * RG + slot] = ds[b];
        }
        if (am) {
          eoff = acc_add_x(eoff, __shfl_sync(kFull, xs, kh - 1));
#pragma unroll
          for (int b = 0; b < NBF; ++b)
            if (b < n_bf) dsum[b] = acc_add_x(dsum[b], __shfl_sync(kFull, ds[b], kh - 1));
        }
      }
      if (lane == 0) {
        pub[(r & 1) * kTkWords + kTkScanned] = scanned;
        pub[(r & 1) * kTkWords + kTkRecs] = n_recs;
      }
      __syncthreads();
      if (pub[(r & 1) * kTkWords + kTkBooked] >= x_end) break;
    }
    if (lane == 0) *n_acc_s = n_acc;
  } else if (role == 3 || role == 4) {
    // ---- summers: role 3 the energy and its square, role 4 the singlets' sums; lane j takes trial j ---
    const bool first = role == 3;
    const A inv_n = acc_from<A>(1.0 / (double)N);
    A s_start[CEMC_MAX_BF];
#pragma unroll
    for (int b = 0; b < CEMC_MAX_BF; ++b)
      s_start[b] = acc_from<A>((b < n_bf && g.singlet_eci[b] >= 0) ? a.cf[(size_t)chain * n_eci + g.singlet_eci[b]] : 0.0);
    A *l = lacc0 + lane;  // [NACC][32]
    uint32_t done = 0, x_booked = RG;
    for (uint32_t r = 1;; ++r) {
      const volatile uint32_t *pp = pub + ((r & 1) ^ 1) * kTkWords;
      const uint32_t n = pp[kTkRecs];
      x_booked = pp[kTkScanned];
      for (; done < n; ++done) {
        const TickRec<A> *q = &recs[done & (kTickRecs - 1)];
        const uint32_t slot = (q->x + (uint32_t)lane) & rmask;
        if (lane >= q->kh) continue;
        if (a.trace_acc && first) {
          const size_t idx = (size_t)chain * a.n_trials + (size_t)(q->x + (uint32_t)lane - RG);
          const uint32_t st = state[slot];
          a.trace_site[2 * idx] = sites[2 * slot];
          a.trace_site[2 * idx + 1] = SWAP ? sites[2 * slot + 1] : (int32_t)((st >> 9) & 15u);
          a.trace_acc[idx] = (int8_t)((st >> 8) & 1u);
          a.trace_de[idx] = (double)r_de[slot];
        }
        if (!a.accum) continue;
        const A ve = acc_add_x(q->eoff, r_x[slot]);
        if (first) {
          l[0] = acc_add(l[0], ve);
          l[32] = acc_add(l[32], acc_mul(ve, ve));
        } else {
#pragma unroll
          for (int b = 0; b < CEMC_MAX_BF; ++b)
            if (b < n_bf) {
              const R ds = SWAP ? (R)0 : r_dx[(SWAP ? 0 : b) * RG + slot];
              const A vs = acc_add(s_start[b], acc_mul(acc_add_x(q->dsum[b], ds), inv_n));
              A *p = l + (2 + b) * 32;
              p[0] = acc_add(p[0], vs);
              p[CEMC_MAX_BF * 32] = acc_add(p[CEMC_MAX_BF * 32], acc_mul(vs, vs));
              p[2 * CEMC_MAX_BF * 32] = acc_add(p[2 * CEMC_MAX_BF * 32], acc_mul(vs, ve));
            }
        }
      }
      __syncwarp();
      if (first && lane == 0) {
        // the oldest trial that has not run is always free to run, so a launch that takes many more ticks
        // than trials has a fault: all warps stop at this barrier
        const bool fault = r > r_max;
        pub[(r & 1) * kTkWords + kTkBooked] = fault ? kTickStop : x_booked;
        if (fault) *fault_s = 1;
      }
      __syncthreads();
      if (pub[(r & 1) * kTkWords + kTkBooked] >= x_end) break;
    }
  } else {
    // ---- fetcher: draws as far ahead as the ring allows ---------------------------------------------
    uint32_t fill = RG;
    for (uint32_t r = 1;; ++r) {
      const volatile uint32_t *pp = pub + ((r & 1) ^ 1) * kTkWords;
      // the predecessors a round can reach (and the 16 of the hash's margin) stay in the ring while a trial is
      // unfinished
      const uint32_t want = min(min(x_end, pp[kTkBooked] + RG - (uint32_t)CW - 16u), fill + 64u);
      for (uint32_t x = fill + lane; x < want; x += 32) {
        const uint32_t slot = x & rmask;
        const uint64_t t = t_first + (uint64_t)(x - RG);
        const cemc_u32x4 w0 = cemc_trial_draw(a.seed, key, t, 0);
        TickDraw d;
        if (SWAP) {
          const cemc_u32x4 w1 = cemc_trial_draw(a.seed, key, t, 1);
          const int np = misc[2];
          const int ia = (int)cemc_below(w0.v[0], (uint32_t)np);
          int ib = (int)cemc_below(w0.v[1], (uint32_t)(np - 1));
          ib += (ib >= ia);
          const int A_ = misc[8 + ia], B_ = misc[8 + ib];
          // the list slots do not change (swaps keep every species count), only the sites in them
          d.a = misc[16 + A_] + (int)cemc_below(w0.v[2], (uint32_t)misc[24 + A_]);
          d.b = misc[16 + B_] + (int)cemc_below(w0.v[3], (uint32_t)misc[24 + B_]);
          d.grp = (uint32_t)A_ | ((uint32_t)B_ << 8);
          d.ua = w1.v[0];
          d.ub = w1.v[1];
        } else {
          // the flipped site: uniform over the movable sites (all sites without a background)
          d.a = g.n_movable == N ? (int)cemc_below(w0.v[0], (uint32_t)N)
                                 : g.movable[cemc_below(w0.v[0], (uint32_t)g.n_movable)];
          d.b = (int32_t)w0.v[1];
          d.grp = g.n_groups > 1 ? (uint32_t)g.site_group[d.a] : 0u;
          d.ua = w0.v[2];
          d.ub = w0.v[3];
        }
        d.pad0 = d.pad1 = d.pad2 = 0;
        draws[slot] = d;
        state[slot] = 0;
#pragma unroll
        for (int k = 0; k < kTickWords; ++k) mask[k * RG + slot] = 0u;
      }
      if (want > fill && want <= x_end) fill = want;
      if (lane == 0) pub[(r & 1) * kTkWords + kTkDrawn] = fill;
      __syncthreads();
      if (pub[(r & 1) * kTkWords + kTkBooked] >= x_end) break;
    }
  }
  __syncthreads();
  if (*fault_s) {  // only the site lists hold moves of this launch (a host that goes on rebuilds them)
    if (tid == 0 && a.status) a.status[chain] = CEMC_ERR_INTERNAL;
    return;
  }

  // ---- epilogue: the call ends with a full recompute of correlation functions and energy -------------
  if (a.accum && tid < NACC) {
    double sum_v = 0.0;
    for (int l = 0; l < 32; ++l) sum_v += acc_to(lacc0[tid * 32 + l]);
    const int b = tid < 2 ? 0 : (tid - 2) % CEMC_MAX_BF;
    if (tid < 2 || b < n_bf) {
      double *sums = &a.accum[acc_row].sum_e;  // sum_e, sum_e2, sum_s[], sum_s2[], sum_se[] in NACC order
      sums[tid] += sum_v;
    }
  }
  {
    int8_t *dst = a.occ + (size_t)chain * N;
    if ((((uintptr_t)dst | (uintptr_t)N) & 15) == 0) {
      for (int i = tid; i < N / 16; i += blockDim.x)
        reinterpret_cast<uint4 *>(dst)[i] = reinterpret_cast<const uint4 *>(occ)[i];
    } else {
      for (int i = tid; i < N; i += blockDim.x) dst[i] = occ[i];
    }
  }
  if (tid == 0) {
    a.trial[chain] = t_first + my_trials;
    if (a.accum) {
      cemc_accum *ac = a.accum + acc_row;
      ac->n_samples += my_trials;
      ac->n_accept += *n_acc_s;
    }
    if (a.status) a.status[chain] = 0;
  }
}

template <typename R>
static cudaError_t launch_tick_r(const DevGeo &g, const RunArgs &a, int move, size_t smem, cudaStream_t st) {
  if (a.warps > (move == CEMC_MOVE_SWAP ? kTickCap : kTickWarps)) return cudaErrorInvalidConfiguration;
  auto k = move != CEMC_MOVE_SWAP ? tick_kernel<R, CEMC_MOVE_FLIP, kTickWarps>
           : a.warps <= kTickWarps ? tick_kernel<R, CEMC_MOVE_SWAP, kTickWarps>
                                   : tick_kernel<R, CEMC_MOVE_SWAP, kTickCap>;
  cudaError_t e = allow_smem(k, g);
  if (e != cudaSuccess) return e;
  k<<<a.n_chains, 32 * (a.warps + kTickHelpers), smem, st>>>(g, a);
  return cudaGetLastError();
}

cudaError_t launch_tick(const DevGeo &g, const RunArgs &a, int move, int precision, size_t smem, cudaStream_t st) {
  return precision == CEMC_PREC_F32 ? launch_tick_r<float>(g, a, move, smem, st)
                                    : launch_tick_r<double>(g, a, move, smem, st);
}

}  // namespace cemc
