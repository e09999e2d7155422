// Scheduled flip kernel: unconstrained single-site flips in the binary +1/-1 basis, four trials per
// warp (the quarter-warp spin form), executed out of order.
//
// The chain is that of mc_kernel (cemc_mc.cu) and of the reference's _mc_step loop
// (cemc/mcmc/montecarlo.py:970-1038 over CEUpdater::calculate, cpp/src/ce_updater.cpp:313-406): trial t
// draws its site and uniform from the counter-based stream.  A flip's site does not depend on the
// chain's state, so which trials touch one another is known before any of them is evaluated: trial t
// has to see trial t' < t only when t' flips t's site or one of its neighbour columns.  mc_kernel
// speculates (evaluates a round of trials against one state, stamps the neighbourhoods of the accepted
// ones, commits the prefix before the first conflict and evaluates the rest again); this kernel
// schedules instead.  Helper warps find, for every trial, which of the trials shortly before it it has
// to see (a mask over up to 255 of them); per tick the evaluating warps get trials that wait for none
// that is not finished, so the trials of one tick never touch one another: they run in any order, write
// accepted flips straight into the occupation and meet one barrier.  No stamps, no commit phase, no
// trial evaluated twice, and the cost does not depend on the acceptance.
//
// Per tick, all warps between the same two barriers (trials move through the stages in batches):
//   fetchers  draws of upcoming trials and their neighbour rows (cp.async into a ring)
//   planner   the next tick's list: the oldest trials of the window that wait for nothing; and enters the
//             sites of the next batch into a hash of chains (head per bucket, `prev` per trial)
//   evaluate  the list of this tick; and looks the row of each trial posted a tick ago up in the hash:
//             buckets with a recent trial are queued
//   follower  the chains of those buckets: earlier trials on a site of the row set bits of the mask
//   cutter    takes finished trials in trial order, in booking rounds
//   scanner   scans the energy changes of the rounds cut a tick ago
//   summers   add the rounds scanned a tick ago to the running sums
// The sums are taken in the rounds of the speculative forms (up to `part` trials, cut before the first
// trial whose site an accepted trial of the round touched, which the masks tell), so they are the same
// bit for bit, whatever kernel ran the launch.
//
// Bound: instruction issue.  150 warp instructions a trial, a third each for the evaluation, the lookups
// and the helpers, at 2.0 of 4 a cycle; shared-memory wavefronts are at 40 % of their rate.  A tick takes
// about 4,500 cycles for 58 trials (82 cycles a trial; mc_kernel's rounds: 3,500 for 22 to 30 commits).
// Headline batch (64 chains x 16384 sites, 10 sweeps): 12.4 ms in mc_kernel's quarter-warp form, 6.4 ms here.  Small cells
// of chains that accept little, and more of them than SMs, are faster there: see the rule in cemc_abi.cu, cemc_route.h.
#include <cuda_runtime.h>

#include <type_traits>

#include "cemc_device.cuh"
#include "cemc_launch.h"
#include "cemc_sched.h"
#include "cemc_spin.h"

namespace cemc {

namespace {

__device__ __forceinline__ void sq_cp_async16(void *dst, const void *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void sq_cp_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

template <typename A>
__device__ __forceinline__ A acc_from_int(int v);  // exact below 2^24
template <>
__device__ __forceinline__ double acc_from_int<double>(int v) { return (double)v; }
template <>
__device__ __forceinline__ df64 acc_from_int<df64>(int v) { return df64{(float)v, 0.f}; }

// Ring entry of a trial: site and the acceptance test's parts (metropolis_parts); the uniform's words
// are kept apart, for the exact test.
struct __align__(16) SchedDraw {
  int32_t site;
  uint32_t lnu, mu, pad;
};
// A booking round (or its second half) on its way from the cutter to the summing warps.
template <typename A>
struct __align__(8) SchedRec {
  A eoff;            // energy before it
  int32_t dsum;      // singlet change of the launch before it
  uint32_t x;        // its first trial
  int32_t kh, half;  // its trials; half 1 = trials 32 .. 63 of a round
};

// Counters published at the end of each tick for the next one (double-buffered by tick parity):
// trials whose rows have landed (per fetcher), posted, with a complete mask, cut into rounds, scanned,
// booked; rounds cut and records made.
enum { kPubLanded = 0, kPubLanded1, kPubPosted, kPubMasked, kPubCut, kPubScanned, kPubBooked, kPubCuts, kPubRecs,
       kPubWords = 16 };

// First trial the mask of trial x can hold.
__device__ __forceinline__ uint32_t sched_low(uint32_t x) { return ((x >> 5) - (uint32_t)(kSchedWords - 1)) << 5; }

constexpr int kRegTerms = 9;  // multi-site terms a lane keeps in registers (the rest are read from shared memory)

}  // namespace

template <typename R>
__global__ void __launch_bounds__(kSchedMaxThreads, 1) sched_kernel(DevGeo g, RunArgs a, SpinDev sd) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int E = a.warps, CAP = 4 * E;
  const int CW = a.part, NB = CW > 32 ? 2 : 1;
  const SchedLayout L =
      sched_layout(g, sd.n_cl, sd.n_masks, (int)sizeof(R), CAP, a.ring_bits, a.row_bits, a.head_bits);
  const uint32_t RG = 1u << a.ring_bits, rmask = RG - 1u, hmask = (1u << a.head_bits) - 1u;
  const uint32_t RR = 1u << a.row_bits, rowm = RR - 1u;
  const int chain = blockIdx.x;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int N = g.n_sites, n_eci = g.n_eci, cp16 = g.cp16, n_cols = g.n_cols;
  const bool evaluator = warp < E;
  const int role = warp - E;  // helpers: 0 planner, 1 follower, 2 cutter, 3 scanner, 4 and 5 summers, 6 and 7 fetchers

  constexpr bool DF = (sizeof(R) == 4);
  using A = typename std::conditional<DF, df64, double>::type;
  constexpr int NACC = 2 + 3 * CEMC_MAX_BF;
  double *cf_s = reinterpret_cast<double *>(smem + L.cf);
  double *eci_s = reinterpret_cast<double *>(smem + L.eci);
  double *w_s = reinterpret_cast<double *>(smem + L.w);
  R *coef_s = reinterpret_cast<R *>(smem + L.coef);
  A *lacc0 = reinterpret_cast<A *>(smem + L.acc);
  SpinEci *sp_eci = reinterpret_cast<SpinEci *>(smem + L.sp_eci);
  uint4 *sp_terms = reinterpret_cast<uint4 *>(smem + L.sp_terms);  // {mask lo, mask hi, field shift, 0}
  int32_t *sp_term0 = reinterpret_cast<int32_t *>(smem + L.sp_lane);  // [9]
  uint64_t *n_acc_s = reinterpret_cast<uint64_t *>(smem + L.misc);  // accepted trials of the launch
  uint32_t *list_n = reinterpret_cast<uint32_t *>(smem + L.misc) + 2;   // [2] trials of the lists
  uint32_t *queue_n = reinterpret_cast<uint32_t *>(smem + L.misc) + 4;  // [2] entries of the queues
  volatile uint32_t *fault_s = reinterpret_cast<volatile uint32_t *>(smem + L.misc) + 6;
  volatile uint32_t *pub = reinterpret_cast<volatile uint32_t *>(smem + L.pub);
  unsigned long long *cfsum = reinterpret_cast<unsigned long long *>(smem + L.cfsum);
  SchedDraw *draws = reinterpret_cast<SchedDraw *>(smem + L.draws);
  uint2 *uni = reinterpret_cast<uint2 *>(smem + L.uni);
  uint16_t *rows = reinterpret_cast<uint16_t *>(smem + L.rows);
  volatile uint32_t *prev = reinterpret_cast<volatile uint32_t *>(smem + L.prev);
  uint32_t *mask = reinterpret_cast<uint32_t *>(smem + L.mask);  // word k: trials of the k-th word before the trial's own
  uint8_t *r_acc = reinterpret_cast<uint8_t *>(smem + L.r_acc);    // bit 0 accepted, 1 new species, 2 finished
  R *r_de = reinterpret_cast<R *>(smem + L.r_de);
  R *r_x = reinterpret_cast<R *>(smem + L.r_x);                    // energy change of the round up to the trial
  int8_t *r_ds = reinterpret_cast<int8_t *>(smem + L.r_ds);        // singlet change of the round up to the trial
  uint2 *cuts = reinterpret_cast<uint2 *>(smem + L.cuts);          // booking rounds: first trial, trials
  SchedRec<A> *recs = reinterpret_cast<SchedRec<A> *>(smem + L.recs);
  uint32_t *heads = reinterpret_cast<uint32_t *>(smem + L.heads);
  uint16_t *lists = reinterpret_cast<uint16_t *>(smem + L.lists);
  uint16_t *queue = reinterpret_cast<uint16_t *>(smem + L.queue);  // [2][kSchedQueue]
  int8_t *occ = reinterpret_cast<int8_t *>(smem + L.occ);
  const uint32_t xorv = (uint32_t)(sd.minus_id ^ 1);  // spin bit = occ ^ xorv (1 = the -1 species)

  // A chain with no trials in this launch (an empty serving slot) leaves its state untouched.
  if (a.chain_trials && a.chain_trials[chain] <= a.chunk_offset) return;
  if (a.route && a.status[chain] != a.route) return;  // left to the other kernel

  // ---- prologue ---------------------------------------------------------------
  for (int k = tid; k < n_eci; k += blockDim.x) {
    const int kind = g.eci_kind[k];
    const double e = a.eci[(size_t)chain * n_eci + k];
    cf_s[k] = a.cf[(size_t)chain * n_eci + k];
    eci_s[k] = e;
    w_s[k] = (kind == 2) ? g.eci_w[k] : 0.0;
    coef_s[k] = (R)(kind == 2 ? e * (double)N * g.eci_w[k] : (kind == 1 ? e : 0.0));
  }
  for (int k = tid; k < sd.n_cl; k += blockDim.x) sp_eci[k] = sd.eci[k];
  for (int i = tid; i < 9; i += blockDim.x) sp_term0[i] = sd.qtr_lane_term[i];
  for (int i = tid; i < 10; i += blockDim.x) cfsum[i] = 0ull;
  for (int i = tid; i < 2 * NACC * 32; i += blockDim.x) lacc0[i] = acc_from<A>(0.0);
  for (uint32_t i = tid; i <= hmask; i += blockDim.x) heads[i] = 0u;
  for (int i = tid; i < 2 * kPubWords; i += blockDim.x) pub[i] = i % kPubWords >= kPubCuts ? 0u : RG;
  {
    const int8_t *src = a.occ + (size_t)chain * N;
    if ((((uintptr_t)src | (uintptr_t)N) & 15) == 0) {
      for (int i = tid; i < N / 16; i += blockDim.x)
        reinterpret_cast<uint4 *>(occ)[i] = reinterpret_cast<const uint4 *>(src)[i];
    } else {
      for (int i = tid; i < N; i += blockDim.x) occ[i] = src[i];
    }
  }
  if (tid == 0) {
    *n_acc_s = 0;
    list_n[0] = list_n[1] = queue_n[0] = queue_n[1] = 0;
    *fault_s = 0;
  }
  // odd-term counts travel in one byte per multi-site cluster ECI: ECI el is byte rank(el)
  unsigned multi = 0;
  for (int k = 0; k < sd.n_cl; ++k) multi |= (sd.eci[k].n_multi > 0 ? 1u : 0u) << k;
  for (int t = tid; t < sd.n_masks; t += blockDim.x) {
    int l = 0;
    while (sd.qtr_lane_term[l + 1] <= t) ++l;
    const int k = sd.qtr_lane_first[l] + sd.qtr_shift[t] / 6;
    sp_terms[t] = make_uint4(sd.masks[t].x, sd.masks[t].y, 8u * (uint32_t)__popc(multi & ((1u << k) - 1u)), 0u);
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

  // Earlier trials on the site of column c of trial x's row (64: its own site): bits of its mask.
  auto follow = [&](uint32_t x, int c) {
    const uint32_t me = x & rmask, low = sched_low(x);
    const int s = c < 64 ? (int)rows[(size_t)(x & rowm) * cp16 + c] : draws[me].site;
    uint32_t y = c < 64 ? *(volatile uint32_t *)&heads[(uint32_t)s & hmask] : prev[me];
    while (y >= low) {  // trials of this bucket, latest first
      if (y < x && draws[y & rmask].site == s) atomicOr(&mask[((x >> 5) - (y >> 5)) * RG + me], 1u << (y & 31u));
      y = prev[y & rmask];
    }
  };

  if (evaluator) {
    // ---- evaluating warps: lane group h = lane / 8 takes entry 4 warp + h of the tick's list --------
    const int h = lane >> 3, hl = lane & 7;
    SpinEci se{};
    R coef = (R)0;
    if (hl < sd.n_cl) {
      se = sp_eci[hl];
      coef = coef_s[se.eci];
    }
    const int p_all = se.n_pairs + se.n_multi;
    const bool is_multi = (multi >> hl) & 1u;
    const int fshift = 8 * __popc(multi & ((1u << hl) - 1u));
    const bool wide = __popc(multi) > 4;
    const int t_lo = sp_term0[hl], t_hi = sp_term0[hl + 1];
    uint32_t mx[kRegTerms], my[kRegTerms], ms[kRegTerms];
#pragma unroll
    for (int i = 0; i < kRegTerms; ++i) {
      uint4 m = make_uint4(0u, 0u, 0u, 0u);
      if (t_lo + i < t_hi) m = sp_terms[t_lo + i];
      mx[i] = m.x;
      my[i] = m.y;
      ms[i] = m.z;
    }
    const R sing = sd.singlet_eci >= 0 ? coef_s[sd.singlet_eci] : (R)0;
    constexpr bool FX = sizeof(R) == 8;  // FP64: energy changes in fixed point (fx_quanta)
    double fx_inv = 0.0;                 // their quantum, 0: FP64 arithmetic
    float fx_kT = 0.f;
    FxNum coef_fx{0, 0u}, sing_fx{0, 0u};
    if constexpr (FX) {
      // |P| is at most the ECI's terms, the spin change 2
      const double most = warp_sum(lane < 8 ? 2.0 * fabs((double)coef) * (double)p_all : 0.0) + 2.0 * fabs((double)sing);
      double least = lane < 8 && (double)coef != 0.0 ? fabs((double)coef) : HUGE_VAL;  // smallest nonzero coefficient
      if ((double)sing != 0.0) least = fmin(least, fabs((double)sing));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) least = fmin(least, __shfl_xor_sync(kFull, least, o));
      const double scale = fx_quanta<kFxLow>(most, least);
      if (scale != 0.0) {
        fx_inv = 1.0 / scale;
        fx_kT = (float)(fx_inv / kT);
        coef_fx = fx_of<kFxLow>((double)coef, scale);
        sing_fx = fx_of<kFxLow>((double)sing, scale);
      }
    }
    const bool cols = 8 * hl < cp16;  // this lane's eight columns 8 hl .. 8 hl + 7 of a row
    const unsigned real = cols ? (1u << min(8, max(0, n_cols - 8 * hl))) - 1u : 0u;  // without the padding
    long long cf_acc = 0;
    int s_acc = 0;
    uint32_t looked = RG;
    for (uint32_t r = 1;; ++r) {
      const volatile uint32_t *pp = pub + ((r & 1) ^ 1) * kPubWords;
      const int n = (int)list_n[r & 1];
      // lookups: which sites of the row of trial x are in a bucket with a trial a mask can hold
      const uint32_t posted = pp[kPubPosted];
      const uint32_t x = looked + (uint32_t)(4 * warp + h);
      const bool look = x < posted;
      if (__any_sync(kFull, look)) {
        const uint32_t xs = look ? x : looked;
        const uint32_t low = sched_low(x);
        uint32_t hit = 0;
        uint4 q = make_uint4(0u, 0u, 0u, 0u);
        if (cols) q = *reinterpret_cast<const uint4 *>(rows + (size_t)(xs & rowm) * cp16 + 8 * hl);
        const uint32_t w4[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint32_t s = (w4[j >> 1] >> (16 * (j & 1))) & 0xffffu;
          hit |= (heads[s & hmask] >= low ? 1u : 0u) << j;
        }
        hit = look ? hit & real : 0u;
        if (look && hl == 0 && prev[x & rmask] >= low) hit |= 256u;  // trials before it in its own bucket
        while (hit) {
          const int j = __ffs(hit) - 1;
          hit &= hit - 1;
          const int c = j < 8 ? 8 * hl + j : 64;
          const uint32_t at = atomicAdd(&queue_n[r & 1], 1u);
          if (at < (uint32_t)kSchedQueue) queue[(r & 1) * kSchedQueue + at] = (uint16_t)((x - looked) | ((uint32_t)c << 8));
          else follow(x, c);
        }
      }
      looked = posted;
      if (4 * warp < n) {
        const uint16_t *list = lists + (size_t)(r & 1) * CAP;
        const int e = 4 * warp + h;
        const bool has = e < n;
        const uint32_t slot = list[has ? e : 4 * warp];
        uint4 q = make_uint4(0u, 0u, 0u, 0u);
        if (cols) q = *reinterpret_cast<const uint4 *>(rows + (size_t)(slot & rowm) * cp16 + 8 * hl);
        const uint4 dr = *reinterpret_cast<const uint4 *>(&draws[slot]);
        const uint32_t w4[4] = {q.x, q.y, q.z, q.w};
        uint32_t bits = 0;  // this lane's eight columns, then the spin words of the row's 64
#pragma unroll
        for (int j = 0; j < 8; ++j) bits |= (uint32_t)occ[(w4[j >> 1] >> (16 * (j & 1))) & 0xffffu] << j;
        const int sa = (int)dr.x;
        const int oa = occ[sa];
        bits <<= 8 * (hl & 3);
        bits |= __shfl_xor_sync(kFull, bits, 1);
        bits |= __shfl_xor_sync(kFull, bits, 2);
        const uint32_t other = __shfl_xor_sync(kFull, bits, 4);
        uint32_t wl = hl < 4 ? bits : other, wh = hl < 4 ? other : bits;
        if (xorv) {  // bits beyond the columns are in no mask
          wl = ~wl;
          wh = ~wh;
        }
        uint64_t odd64 = 0;
        uint32_t odd32 = 0;
        if (!wide) {
#pragma unroll
          for (int i = 0; i < kRegTerms; ++i)
            odd32 += (uint32_t)(__popc((wl & mx[i]) ^ (wh & my[i])) & 1) << ms[i];
          for (int t = t_lo + kRegTerms; t < t_hi; ++t) {
            const uint4 m = sp_terms[t];
            odd32 += (uint32_t)(__popc((wl & m.x) ^ (wh & m.y)) & 1) << m.z;
          }
#pragma unroll
          for (int o = 1; o < 8; o <<= 1) odd32 += __shfl_xor_sync(kFull, odd32, o);
          odd64 = odd32;
        } else {
#pragma unroll
          for (int i = 0; i < kRegTerms; ++i)
            odd64 += (uint64_t)(__popc((wl & mx[i]) ^ (wh & my[i])) & 1) << ms[i];
          for (int t = t_lo + kRegTerms; t < t_hi; ++t) {
            const uint4 m = sp_terms[t];
            odd64 += (uint64_t)(__popc((wl & m.x) ^ (wh & m.y)) & 1) << m.z;
          }
#pragma unroll
          for (int o = 1; o < 8; o <<= 1) odd64 += __shfl_xor_sync(kFull, odd64, o);
        }
        const int my_odd = is_multi ? (int)((odd64 >> fshift) & 255u) : 0;
        const int P = p_all - 2 * (__popc(wl & se.pair_lo) + __popc(wh & se.pair_hi) + my_odd);
        const int delta = ((uint32_t)oa ^ xorv) ? 2 : -2;
        R de;
        FxNum de_fx{0, 0u};
        if (FX && fx_inv != 0.0) {
          de_fx = fx_sum<8>(fx_mul(coef_fx, P), sing_fx, delta);
          de = (R)fx_value<kFxLow>(de_fx, fx_inv);
        } else {
          R sum = coef * (R)P;
#pragma unroll
          for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(kFull, sum, o);
          if (sd.singlet_eci >= 0) sum += sing;
          de = (R)delta * sum;
        }
        int acc = 0;
        if (hl == 0 && has) {
          const float lnu = __uint_as_float(dr.y), mu = __uint_as_float(dr.z);
          acc = FX && fx_inv != 0.0 ? metropolis_pre_fx(de_fx, (double)de, lnu, mu, &uni[slot].x, kT, fx_kT)
                                    : metropolis_pre<R>(de, lnu, mu, &uni[slot].x, kT, inv_kT);
          const int na = oa ^ 1;
          if (acc) occ[sa] = (int8_t)na;
          r_acc[slot] = (uint8_t)(acc | (na << 1) | 4);
          r_de[slot] = de;
        }
        acc = __shfl_sync(kFull, acc, lane & 24);
        cf_acc += acc ? (long long)(delta * P) : 0ll;
        s_acc += (hl == 0 && acc) ? delta : 0;
      }
      __syncthreads();
      if (pub[(r & 1) * kPubWords + kPubBooked] >= x_end) break;  // all booked, or stopped (kSchedNone)
    }
    if (hl < sd.n_cl && cf_acc) atomicAdd(&cfsum[hl], (unsigned long long)cf_acc);
    if (hl == 0 && s_acc) atomicAdd(&cfsum[8], (unsigned long long)(long long)s_acc);
  } else if (role == 0) {
    // ---- planner --------------------------------------------------------------------------------
    uint32_t wait[kSchedWords];  // trials of the window's words that no list holds yet
#pragma unroll
    for (int w = 0; w < kSchedWords; ++w) wait[w] = kFull;
    uint32_t b = RG >> 5;  // the window's first word
    uint32_t posted = RG;
    for (uint32_t r = 1;; ++r) {
      const volatile uint32_t *pp = pub + ((r & 1) ^ 1) * kPubWords;
      const uint32_t masked = pp[kPubMasked];
      const uint32_t landed = min(pp[kPubLanded], pp[kPubLanded1]);
      // the next tick's list, in trial order: trials whose mask holds no trial without a list, other
      // than those of the lists up to this tick (finished by its end)
      uint16_t *list = lists + (size_t)((r + 1) & 1) * CAP;
      uint32_t taken[kSchedWords];
      int total = 0;
#pragma unroll
      for (int w = 0; w < kSchedWords; ++w) {
        taken[w] = 0;
        const uint32_t x = 32u * (b + w) + (uint32_t)lane;
        if (32u * (b + w) < masked && total < CAP && wait[w]) {
          uint32_t on = 0;
#pragma unroll
          for (int k = 0; k <= w; ++k) on |= mask[k * RG + (x & rmask)] & wait[w - k];
          const bool ready = x < masked && ((wait[w] >> lane) & 1u) && on == 0;
          const int at = total + __popc(__ballot_sync(kFull, ready) & ((1u << lane) - 1u));
          const bool take = ready && at < CAP;
          taken[w] = __ballot_sync(kFull, take);
          if (take) list[at] = (uint16_t)(x & rmask);
          total += __popc(taken[w]);
        }
      }
      if (lane == 0) list_n[(r + 1) & 1] = (uint32_t)total;
#pragma unroll
      for (int w = 0; w < kSchedWords; ++w) wait[w] &= ~taken[w];
      while (wait[0] == 0) {
#pragma unroll
        for (int w = 0; w + 1 < kSchedWords; ++w) wait[w] = wait[w + 1];
        wait[kSchedWords - 1] = kFull;
        ++b;
      }
      // the next batch into the hash: no further than the window will reach when its masks are there
      const uint32_t hi = min(min(posted + (uint32_t)CAP, landed), 32u * (b + kSchedWords) + 3u * (uint32_t)CAP);
      for (uint32_t x0 = posted; x0 < hi; x0 += 32) {
        const uint32_t x = x0 + lane, slot = x & rmask;
        const bool mine = x < hi;
        const uint32_t bucket = mine ? ((uint32_t)draws[slot].site & hmask) : 0u;
        volatile uint32_t *hd = heads + bucket;
        if (mine) prev[slot] = *hd;
        __threadfence_block();  // a lookup that sees the new head sees its chain
        __syncwarp();
        const uint32_t old = mine ? prev[slot] : 0u;
        if (mine) *hd = x;
        __syncwarp();
        if (__any_sync(kFull, mine && *hd != x)) {
          // two of these trials share a bucket: chain them in trial order
          const unsigned same = __match_any_sync(kFull, mine ? bucket : 0x80000000u + lane);
          const unsigned before = same & ((1u << lane) - 1u);
          if (mine) prev[slot] = before ? x0 + (31u - (uint32_t)__clz(before)) : old;
          __threadfence_block();
          __syncwarp();
          if (mine && (same >> lane) == 1u) *hd = x;
          __syncwarp();
        }
      }
      if (hi > posted) posted = hi;
      if (lane == 0) pub[(r & 1) * kPubWords + kPubPosted] = posted;
      __syncthreads();
      if (pub[(r & 1) * kPubWords + kPubBooked] >= x_end) break;
    }
  } else if (role == 1) {
    // ---- follower: the buckets the lookups queued a tick ago ------------------------------------------
    uint32_t posted_1 = RG, posted_2 = RG, posted_3 = RG;  // posted by the end of ticks r - 1, r - 2, r - 3
    for (uint32_t r = 1;; ++r) {
      posted_3 = posted_2;
      posted_2 = posted_1;
      posted_1 = pub[((r & 1) ^ 1) * kPubWords + kPubPosted];
      const uint32_t q = (r & 1) ^ 1, n = min(queue_n[q], (uint32_t)kSchedQueue);
      for (uint32_t i = lane; i < n; i += 32) {  // of the trials posted in tick r - 2
        const uint32_t e = queue[q * kSchedQueue + i];
        follow(posted_3 + (e & 255u), (int)(e >> 8));
      }
      __syncwarp();
      if (lane == 0) {
        queue_n[q] = 0;
        pub[(r & 1) * kPubWords + kPubMasked] = posted_2;
      }
      __syncthreads();
      if (pub[(r & 1) * kPubWords + kPubBooked] >= x_end) break;
    }
  } else if (role == 2) {
    // ---- cutter: finished trials in trial order, in rounds of up to `part` --------------------------
    uint32_t x0 = RG, n_cuts = 0;
    for (uint32_t r = 1;; ++r) {
      const uint32_t masked = pub[((r & 1) ^ 1) * kPubWords + kPubMasked];
      const uint32_t full = n_cuts + kSchedCuts / 2;  // two ticks of rounds fit the buffer
      while (n_cuts < full && x0 < x_end) {
        // the round at x0: finished trials, up to the first one an accepted trial of the round touches;
        // a round lies in two words of trials, or (more than 32 trials) in three
        const int nv = (int)min((uint32_t)CW, x_end - x0);
        const uint32_t w0 = x0 & ~31u;
        uint32_t acc[3], fin[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          acc[q] = fin[q] = 0;
          if (q == 2 && NB == 1) continue;
          const uint32_t ra = r_acc[(w0 + 32u * q + lane) & rmask];
          const unsigned in = __ballot_sync(kFull, w0 + 32u * q + lane >= x0 && w0 + 32u * q + lane < masked);
          fin[q] = __ballot_sync(kFull, ra & 4u) & in;
          acc[q] = __ballot_sync(kFull, (ra & 5u) == 5u) & in;
        }
        int done_n = 64, cut = 64;  // trials finished from x0 on, without a gap; first trial touched
#pragma unroll
        for (int q = 2; q >= 0; --q) {
          if (q == 2 && NB == 1) continue;
          const uint32_t x = w0 + 32u * q + lane, slot = x & rmask;
          uint32_t on = 0;
#pragma unroll
          for (int k = 0; k <= q; ++k) on |= mask[k * RG + slot] & acc[q - k];
          const unsigned hit = __ballot_sync(kFull, x >= x0 && x < masked && on != 0);
          const unsigned gap = __ballot_sync(kFull, x >= x0) & ~fin[q];
          if (hit) cut = (int)(w0 + 32u * q + __ffs(hit) - 1 - x0);
          if (gap) done_n = (int)(w0 + 32u * q + __ffs(gap) - 1 - x0);
        }
        const int ks = min(cut, nv);
        if (ks > done_n) break;  // the rest of the round is not finished
        if (lane == 0) cuts[n_cuts & (kSchedCuts - 1)] = make_uint2(x0, (uint32_t)ks);
        ++n_cuts;
        x0 += (uint32_t)ks;
      }
      if (lane == 0) {
        pub[(r & 1) * kPubWords + kPubCut] = x0;
        pub[(r & 1) * kPubWords + kPubCuts] = n_cuts;
      }
      __syncthreads();
      if (pub[(r & 1) * kPubWords + kPubBooked] >= x_end) break;
    }
  } else if (role == 3) {
    // ---- scanner: energy and singlet changes of each round up to every trial ------------------------
    A eoff[2];  // energy relative to e_ref as the bookers of a round's two halves carry it
    eoff[0] = eoff[1] = acc_from<A>(a.energy[chain] - e_ref);
    int32_t dsum = 0;
    uint64_t n_acc = 0;
    uint32_t n_recs = 0, n_cuts = 0;
    for (uint32_t r = 1;; ++r) {
      const volatile uint32_t *pp = pub + ((r & 1) ^ 1) * kPubWords;
      const uint32_t cuts_n = pp[kPubCuts], scanned = pp[kPubCut];
      for (; n_cuts < cuts_n; ++n_cuts) {
        const uint2 cq = cuts[n_cuts & (kSchedCuts - 1)];
        const uint32_t x0 = cq.x;
        const int ks = (int)cq.y;
        const int kh[2] = {ks < 32 ? ks : 32, ks < 32 ? 0 : ks - 32};
        R tot[2] = {(R)0, (R)0}, xv[2] = {(R)0, (R)0};  // totals of the halves by the scan, as their own booker adds them
        int dh[2] = {0, 0};
        unsigned am[2] = {0u, 0u};
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          if (q == 1 && NB == 1) continue;
          const uint32_t slot = (x0 + (uint32_t)(lane + 32 * q)) & rmask;
          const uint32_t ra = r_acc[slot];
          const R de = r_de[slot];
          const bool acc = lane < kh[q] && (ra & 1u);
          am[q] = __ballot_sync(kFull, acc);
          // the site held -1 (spin bit of its old species): its spin change is +2
          const unsigned um = __ballot_sync(kFull, acc && ((((ra >> 1) & 1u) ^ 1u ^ xorv) != 0u));
          const unsigned le = kFull >> (31 - lane);
          R x = acc ? de : (R)0;
          xv[q] = x;
          if (am[q]) {
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
              const R nx = __shfl_up_sync(kFull, x, o);
              if (lane >= o) x += nx;
            }
          }
          if (lane < kh[q]) {
            r_x[slot] = x;
            // singlet changes are +-2: their prefix sums are exact from two population counts
            r_ds[slot] = (int8_t)(2 * (2 * __popc(um & le) - __popc(am[q] & le)));
          }
          tot[q] = __shfl_sync(kFull, x, (kh[q] + 31) & 31);
          dh[q] = 2 * (2 * __popc(um) - __popc(am[q]));
          n_acc += (uint64_t)__popc(am[q]);
        }
        if (lane == 0) recs[n_recs & (kSchedRecs - 1)] = SchedRec<A>{eoff[0], dsum, x0, kh[0], 0};
        ++n_recs;
        if (am[0]) eoff[0] = acc_add_x(eoff[0], tot[0]);
        if (NB > 1) {
          // each half's booker carries the other half's total as a plain sum over its trials
          if (am[0]) eoff[1] = acc_add_x(eoff[1], warp_sum(xv[0]));
          if (kh[1] > 0) {
            if (lane == 0) recs[n_recs & (kSchedRecs - 1)] = SchedRec<A>{eoff[1], dsum + dh[0], x0 + 32u, kh[1], 1};
            ++n_recs;
            if (am[1]) {
              eoff[0] = acc_add_x(eoff[0], warp_sum(xv[1]));
              eoff[1] = acc_add_x(eoff[1], tot[1]);
            }
          }
        }
        dsum += dh[0] + dh[1];
      }
      if (lane == 0) {
        pub[(r & 1) * kPubWords + kPubScanned] = scanned;
        pub[(r & 1) * kPubWords + kPubRecs] = n_recs;
      }
      __syncthreads();
      if (pub[(r & 1) * kPubWords + kPubBooked] >= x_end) break;
    }
    if (lane == 0) *n_acc_s = n_acc;
  } else if (role == 4 || role == 5) {
    // ---- summers: role 4 the energy and its square, role 5 the singlet's sums; lane j takes trial j ----
    const bool first = role == 4;
    const A s_start = acc_from<A>(g.singlet_eci[0] >= 0 ? a.cf[(size_t)chain * n_eci + g.singlet_eci[0]] : 0.0);
    const A inv_n = acc_from<A>(1.0 / (double)N);
    A l0[2], l1[2], l2[2];
    l0[0] = l0[1] = l1[0] = l1[1] = l2[0] = l2[1] = acc_from<A>(0.0);
    uint32_t done = 0, x_booked = RG;
    auto add = [&](const SchedRec<A> &q, A &c0, A &c1, A &c2) {
      if (lane >= q.kh) return;
      const uint32_t slot = (q.x + (uint32_t)lane) & rmask;
      const A ve = acc_add_x(q.eoff, r_x[slot]);
      if (first) {
        c0 = acc_add(c0, ve);
        c1 = acc_add(c1, acc_mul(ve, ve));
      } else {
        const A vs = acc_add(s_start, acc_mul(acc_from_int<A>(q.dsum + (int)r_ds[slot]), inv_n));
        c0 = acc_add(c0, vs);
        c1 = acc_add(c1, acc_mul(vs, vs));
        c2 = acc_add(c2, acc_mul(vs, ve));
      }
    };
    for (uint32_t r = 1;; ++r) {
      const volatile uint32_t *pp = pub + ((r & 1) ^ 1) * kPubWords;
      const uint32_t n = pp[kPubRecs];
      x_booked = pp[kPubScanned];
      for (; done < n; ++done) {
        const SchedRec<A> q = recs[done & (kSchedRecs - 1)];
        if (a.trace_acc && first) {
          for (int j = lane; j < q.kh; j += 32) {
            const uint32_t slot = (q.x + (uint32_t)j) & rmask;
            const size_t idx = (size_t)chain * a.n_trials + (size_t)(q.x + (uint32_t)j - RG);
            a.trace_site[2 * idx] = draws[slot].site;
            a.trace_site[2 * idx + 1] = (int32_t)((r_acc[slot] >> 1) & 1u);
            a.trace_acc[idx] = (int8_t)(r_acc[slot] & 1u);
            a.trace_de[idx] = (double)r_de[slot];
          }
        }
        if (a.accum) {
          if (q.half == 0) add(q, l0[0], l1[0], l2[0]);
          else add(q, l0[1], l1[1], l2[1]);
        }
      }
      if (first && lane == 0) {
        // the oldest waiting trial is always ready, so a launch that takes many more ticks than trials
        // has a fault: all warps stop at this barrier
        const bool fault = r > r_max;
        pub[(r & 1) * kPubWords + kPubBooked] = fault ? kSchedNone : x_booked;
        if (fault) *fault_s = 1;
      }
      __syncthreads();
      if (pub[(r & 1) * kPubWords + kPubBooked] >= x_end) break;
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      A *lacc = lacc0 + q * NACC * 32 + lane;
      if (first) {
        lacc[0] = l0[q];
        lacc[32] = l1[q];
      } else {
        lacc[32 * 2] = l0[q];
        lacc[32 * (2 + CEMC_MAX_BF)] = l1[q];
        lacc[32 * (2 + 2 * CEMC_MAX_BF)] = l2[q];
      }
    }
  } else {
    // ---- fetchers: draws and neighbour rows as far ahead as the rings allow --------------------------
    const int fq = role - 6;
    uint32_t fill = RG;
    for (uint32_t r = 1;; ++r) {
      const volatile uint32_t *pp = pub + ((r & 1) ^ 1) * kPubWords;
      const uint32_t want = min(min(x_end, pp[kPubBooked] + RG), min(pp[kPubCut] + RR, fill + (uint32_t)CAP));
      for (uint32_t x = fill + (uint32_t)(32 * fq + lane); x < want; x += 64) {
        const uint32_t slot = x & rmask;
        const uint64_t t = t_first + (uint64_t)(x - RG);
        const cemc_u32x4 w0 = cemc_trial_draw(a.seed, key, t, 0);
        // the flipped site: uniform over the movable sites (all sites without a background)
        const int site = g.n_movable == N ? (int)cemc_below(w0.v[0], (uint32_t)N)
                                          : g.movable[cemc_below(w0.v[0], (uint32_t)g.n_movable)];
        const uint16_t *src = g.table16 + (size_t)site * cp16;
        uint16_t *dst = rows + (size_t)(x & rowm) * cp16;
        for (int q = 0; q < cp16; q += 8) sq_cp_async16(dst + q, src + q);
        float lnu, mu;
        metropolis_parts(w0.v[2], lnu, mu);
        SchedDraw d;
        d.site = site;
        d.lnu = __float_as_uint(lnu);
        d.mu = __float_as_uint(mu);
        d.pad = 0;
        draws[slot] = d;
        uni[slot] = make_uint2(w0.v[2], w0.v[3]);
        r_acc[slot] = 0;
#pragma unroll
        for (int k = 0; k < kSchedWords; ++k) mask[k * RG + slot] = 0u;
      }
      sq_cp_wait_all();
      if (want > fill) fill = want;
      if (lane == 0) pub[(r & 1) * kPubWords + kPubLanded + fq] = fill;
      __syncthreads();
      if (pub[(r & 1) * kPubWords + kPubBooked] >= x_end) break;
    }
  }
  __syncthreads();
  if (*fault_s) {  // the chain's state is not written
    if (tid == 0 && a.status) a.status[chain] = CEMC_ERR_INTERNAL;
    return;
  }

  // ---- epilogue -----------------------------------------------------------------
  for (int k = tid; k < n_eci; k += blockDim.x) {
    const int kind = g.eci_kind[k];
    long long c = 0;
    for (int q = 0; q < sd.n_cl; ++q)
      if (sp_eci[q].eci == k) c = (long long)cfsum[q];
    if (k == sd.singlet_eci) c = (long long)cfsum[8];
    const double d = (double)c;
    if (kind == 2) cf_s[k] = cf_s[k] + d * w_s[k];
    else if (kind == 1) cf_s[k] = cf_s[k] + d / (double)N;
  }
  if (a.accum && tid < NACC) {
    double sum_v = 0.0;
    for (int q = 0; q < NB; ++q)
      for (int l = 0; l < 32; ++l) sum_v += acc_to(lacc0[(q * NACC + tid) * 32 + l]);
    const int b = tid < 2 ? 0 : (tid - 2) % CEMC_MAX_BF;
    if (tid < 2 || b < g.n_bf) {
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
  __syncthreads();
  for (int k = tid; k < n_eci; k += blockDim.x) a.cf[(size_t)chain * n_eci + k] = cf_s[k];
  if (tid == 0) {
    // energy = N * eci . cf in sorted-name order (ce_updater.cpp:236-242)
    double e = 0.0;
    for (int k = 0; k < n_eci; ++k) e += eci_s[k] * cf_s[k];
    a.energy[chain] = e * (double)(unsigned)N;
    a.trial[chain] = t_first + my_trials;
    if (a.accum) {
      cemc_accum *ac = a.accum + acc_row;
      ac->n_samples += my_trials;
      ac->n_accept += *n_acc_s;
    }
    if (a.status) a.status[chain] = 0;
  }
}

cudaError_t launch_sched(const DevGeo &g, const RunArgs &a, int precision, size_t smem, cudaStream_t st,
                         const SpinDev &sd) {
  const unsigned threads = (unsigned)((a.warps + kSchedHelpers) * 32);
  if (threads > kSchedMaxThreads || !g.table16 || !sd.qtr_ok) return cudaErrorInvalidConfiguration;
  auto k = precision == CEMC_PREC_F32 ? sched_kernel<float> : sched_kernel<double>;
  cudaError_t e = allow_smem(k, g);
  if (e != cudaSuccess) return e;
  k<<<a.n_chains, threads, smem, st>>>(g, a, sd);
  return cudaGetLastError();
}

}  // namespace cemc
