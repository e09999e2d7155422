// C ABI of libcemc_gb300.so (declared in include/cemc_gb300.h).
//
// Host-side work here: validating descriptors, packing a geometry's cluster
// terms into the per-lane chunks the kernels walk, sizing shared memory and
// launching.  No entry point throws; failures return a status code and leave a
// message for cemc_last_error().
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <array>
#include <map>
#include <mutex>
#include <tuple>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "cemc_boxcf.h"
#include "cemc_field.h"
#include "cemc_kernels.h"
#include "cemc_route.h"
#include "cemc_sched.h"
#include "cemc_schedt.h"
#include "cemc_spin.h"

namespace {

thread_local std::string g_err;

int fail(int code, const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  g_err = buf;
  return code;
}

int cuda_fail(cudaError_t e, const char *what) {
  return fail(CEMC_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

}  // namespace

struct cemc_geometry {
  cemc::DevGeo g;
  cemc::SpinDev spin{};  // tables of the binary spin-basis kernel (spin_ok)
  bool spin_ok = false;
  cemc::FieldDev field{};  // tables of the local-field kernel (field_ok)
  bool field_ok = false;
  cemc::BoxCf box{};  // tables of the bit-plane recompute (box.ok)
  void *dev = nullptr;  // one device allocation holding every table
  size_t dev_bytes = 0;  // its size
  int max_smem = 0;     // opt-in shared memory per block of the current device
  int n_sms = 0;        // multiprocessors of the current device
  // resident cluster pairs per launch configuration (warps, move, precision, spin, smem)
  mutable std::mutex mu;
  mutable std::map<std::tuple<int, int, int, int, size_t>, int> pairs;
};

extern "C" int cemc_last_error(char *buf, size_t len) {
  if (!buf || len == 0) return CEMC_ERR_ARG;
  snprintf(buf, len, "%s", g_err.c_str());
  return CEMC_OK;
}

extern "C" int cemc_version(int32_t *major, int32_t *minor, int32_t *sm) {
  if (major) *major = 1;
  if (minor) *minor = 0;
  if (sm) *sm = 103;
  return CEMC_OK;
}

extern "C" int cemc_geometry_create(const cemc_geometry_desc *d, cemc_geometry **out) {
  if (!d || !out) return fail(CEMC_ERR_ARG, "null descriptor or output");
  *out = nullptr;
  const int N = d->n_sites, C = d->n_cols, S = d->n_sym, B = d->n_bf, K = d->n_eci, T = d->n_terms;
  if (N <= 0 || C <= 0 || K <= 0 || T < 0) return fail(CEMC_ERR_ARG, "empty geometry");
  if (C > CEMC_MAX_COLS) return fail(CEMC_ERR_LIMIT, "%d neighbour columns exceed the limit %d", C, CEMC_MAX_COLS);
  if (B < 1 || B > CEMC_MAX_BF || S != B + 1 || S > 8)
    return fail(CEMC_ERR_LIMIT, "unsupported species count %d", S);
  if (K > CEMC_MAX_ECI) return fail(CEMC_ERR_LIMIT, "%d ECIs exceed the limit %d", K, CEMC_MAX_ECI);
  if (!d->table || !d->bf || !d->eci_kind || !d->eci_dec || !d->eci_weight || !d->eci_full_weight ||
      (T > 0 && (!d->term_eci || !d->term_ref || !d->term_size || !d->term_nb)))
    return fail(CEMC_ERR_ARG, "null table pointer");
  const int one_idx = C * B;
  if (one_idx + 1 + B >= (1 << cemc::kRefBits)) return fail(CEMC_ERR_LIMIT, "neighbour table too wide");
  for (size_t i = 0; i < (size_t)N * C; ++i)
    if (d->table[i] < 0 || d->table[i] >= N) return fail(CEMC_ERR_ARG, "table entry %zu out of range", i);
  // Movable (non-background) sites: ascending, in range; every other site is background.
  std::vector<int32_t> movable;
  std::vector<int8_t> site_active(N, 1);
  if (d->movable && d->n_movable < N) {
    if (d->n_movable < 2) return fail(CEMC_ERR_ARG, "fewer than two movable sites");
    movable.assign(d->movable, d->movable + d->n_movable);
    std::fill(site_active.begin(), site_active.end(), 0);
    for (int i = 0; i < d->n_movable; ++i) {
      if (movable[i] < 0 || movable[i] >= N || (i > 0 && movable[i] <= movable[i - 1]))
        return fail(CEMC_ERR_ARG, "movable sites must be ascending site indices");
      site_active[movable[i]] = 1;
    }
  }
  const int n_movable = movable.empty() ? N : (int)movable.size();
  if (movable.empty()) movable.assign(1, 0);
  int singlet[CEMC_MAX_BF];
  for (int b = 0; b < CEMC_MAX_BF; ++b) singlet[b] = 0;
  for (int k = 0; k < K; ++k) {
    if (d->eci_kind[k] < 0 || d->eci_kind[k] > 2) return fail(CEMC_ERR_ARG, "bad ECI kind");
    if (d->eci_kind[k] == 1) {
      if (d->eci_dec[k] < 0 || d->eci_dec[k] >= B) return fail(CEMC_ERR_ARG, "bad singlet decoration");
      singlet[d->eci_dec[k]] = k;
    }
  }
  // Translation-symmetry groups: each owns a contiguous, ECI-sorted range of
  // terms; a one-group geometry is group 0 with every term.
  const int G = d->n_groups > 1 ? d->n_groups : 1;
  if (G > CEMC_MAX_GROUPS) return fail(CEMC_ERR_LIMIT, "%d translation groups exceed the limit %d", G, CEMC_MAX_GROUPS);
  std::vector<int32_t> gterm(G + 1, 0);
  std::vector<double> gscale(G, 1.0);
  std::vector<int8_t> sgroup(N, 0);
  gterm[G] = T;
  if (G > 1) {
    if (!d->site_group || !d->group_terms || !d->group_scale) return fail(CEMC_ERR_ARG, "null group table");
    for (int q = 0; q <= G; ++q) gterm[q] = d->group_terms[q];
    if (gterm[0] != 0 || gterm[G] != T) return fail(CEMC_ERR_ARG, "group term ranges must cover the terms");
    for (int q = 0; q < G; ++q) {
      if (gterm[q + 1] < gterm[q]) return fail(CEMC_ERR_ARG, "group term ranges must ascend");
      gscale[q] = d->group_scale[q];
      if (!(gscale[q] > 0.0) || !std::isfinite(gscale[q])) return fail(CEMC_ERR_ARG, "bad group scale");
    }
    for (int i = 0; i < N; ++i) {
      if (!site_active[i]) continue;
      const int q = d->site_group[i];
      if (q < 0 || q >= G) return fail(CEMC_ERR_ARG, "site %d has no translation group", i);
      sgroup[i] = (int8_t)q;
    }
  }
  bool equal_groups = true;
  for (int q = 0; q < G; ++q) equal_groups = equal_groups && gscale[q] == 1.0;
  for (int t = 0; t < T; ++t) {
    const int k = d->term_eci[t];
    const bool group_start = std::find(gterm.begin(), gterm.end(), t) != gterm.end();
    if (k < 0 || k >= K || d->eci_kind[k] != 2) return fail(CEMC_ERR_ARG, "term %d has a bad ECI", t);
    if (t > 0 && !group_start && k < d->term_eci[t - 1]) return fail(CEMC_ERR_ARG, "terms are not sorted by ECI");
    if (d->term_size[t] < 2 || d->term_size[t] > 4) return fail(CEMC_ERR_ARG, "term %d has a bad size", t);
    if (d->term_ref[t] < 0 || d->term_ref[t] >= B) return fail(CEMC_ERR_ARG, "term %d has a bad decoration", t);
    for (int j = 0; j < d->term_size[t] - 1; ++j)
      if (d->term_nb[3 * t + j] < 0 || d->term_nb[3 * t + j] >= one_idx)
        return fail(CEMC_ERR_ARG, "term %d has a bad member", t);
  }

  // Lane chunks, per group: [G][33] bounds, [G][32] first ECI, [G][2K] lane range per ECI.
  std::vector<int32_t> lane_term(33 * (size_t)G), first(32 * (size_t)G, 0), eci_lane(2 * (size_t)K * G);
  int n_slots = 1;
  std::vector<uint16_t> terms(4 * (size_t)std::max(T, 1), 0);
  for (int q = 0; q < G; ++q) {
    const int t0 = gterm[q], Tg = gterm[q + 1] - gterm[q];
    int32_t *lt = lane_term.data() + 33 * q, *fi = first.data() + 32 * q, *el = eci_lane.data() + 2 * (size_t)K * q;
    for (int l = 0; l <= 32; ++l) lt[l] = t0 + (int32_t)(((long long)l * Tg) / 32);
    for (int k = 0; k < K; ++k) {
      el[2 * k] = 0;
      el[2 * k + 1] = -1;
    }
    std::vector<int> lo_seen(K, 33), hi_seen(K, -1);
    for (int l = 0; l < 32; ++l) {
      const int lo = lt[l], hi = lt[l + 1];
      // a lane without terms (fewer than 32) between two lanes of an ECI is read as that ECI's slot 0
      if (lo < t0 + Tg) fi[l] = d->term_eci[lo];
      if (lo >= hi) continue;
      n_slots = std::max(n_slots, d->term_eci[hi - 1] - fi[l] + 1);
      for (int i = lo; i < hi; ++i) {
        const int k = d->term_eci[i];
        lo_seen[k] = std::min(lo_seen[k], l);
        hi_seen[k] = std::max(hi_seen[k], l);
      }
    }
    for (int k = 0; k < K; ++k)
      if (hi_seen[k] >= 0) {
        el[2 * k] = lo_seen[k];
        el[2 * k + 1] = hi_seen[k];
      }
    for (int l = 0; l < 32; ++l)
      for (int i = lt[l]; i < lt[l + 1]; ++i) {
        const int slot = d->term_eci[i] - fi[l];
        terms[4 * i] = (uint16_t)((one_idx + 1 + d->term_ref[i]) | (slot << cemc::kRefBits));
        for (int j = 0; j < 3; ++j)
          terms[4 * i + 1 + j] = (uint16_t)(j < d->term_size[i] - 1 ? d->term_nb[3 * i + j] : one_idx);
      }
  }
  if (n_slots > cemc::kMaxSlots) return fail(CEMC_ERR_LIMIT, "a lane chunk spans %d ECIs", n_slots);
  std::vector<uint8_t> fterms(8 * (size_t)std::max(T, 1), 0);
  for (int i = 0; i < T; ++i) {
    for (int j = 0; j < 3; ++j) {
      const bool has = j < d->term_size[i] - 1;
      fterms[8 * i + j] = (uint8_t)(has ? d->term_nb[3 * i + j] / B : 0);
      fterms[8 * i + 3 + j] = (uint8_t)(has ? d->term_nb[3 * i + j] % B : 0);
    }
    fterms[8 * i + 6] = (uint8_t)d->term_ref[i];
    fterms[8 * i + 7] = (uint8_t)d->term_size[i];
  }
  // Term range of each (group, ECI): fterm_off[q * (K + 1) + k].
  std::vector<int32_t> fterm_off((size_t)G * (K + 1), 0);
  for (int q = 0; q < G; ++q) {
    int t = gterm[q];
    for (int k = 0; k < K; ++k) {
      fterm_off[(size_t)q * (K + 1) + k] = t;
      while (t < gterm[q + 1] && d->term_eci[t] == k) ++t;
    }
    fterm_off[(size_t)q * (K + 1) + K] = gterm[q + 1];
  }
  // Table form of the trial energy change: the terms grouped by cluster geometry
  // (the ordered member columns of a sub-cluster with the changed site as
  // reference); geometries whose terms carry the same (ECI, decorations) list
  // share a pattern, and each chain's kernel tabulates per pattern
  // F(old, new, member species) = sum over its terms of coef * (bf[d_ref][new] -
  // bf[d_ref][old]) * prod bf[d_j][s_j], so a flip costs one lookup per geometry.
  // With several translation groups each group has its own geometry range
  // (geo_start) and the groups share patterns; the table stores group 0's
  // weights, so it needs equal group sizes.
  std::vector<uint32_t> geo_list;  // per geometry: {packed columns, F offset, stride S^m, 0}
  std::vector<int32_t> pat_info;   // per pattern: {m, F offset, first term, end term}
  std::vector<int32_t> pat_terms;  // k | d_ref << 8 | d1 << 12 | d2 << 16 | d3 << 20
  std::vector<int32_t> geo_start(G + 1, 0);
  int n_geo = 0, n_pat = 0, tab_len = 0;
  bool table_ok = C < 255 && S <= 8 && equal_groups;
  std::map<std::vector<std::array<int, 5>>, int> pats;
  for (int q = 0; q < G && table_ok; ++q) {
    geo_start[q] = (int)(geo_list.size() / 4);
    std::map<std::vector<int>, std::vector<std::array<int, 5>>> geos;  // member columns -> terms
    std::vector<std::vector<int>> geo_order;
    for (int t = gterm[q]; t < gterm[q + 1]; ++t) {
      const int m = d->term_size[t] - 1;
      std::vector<int> cols(m);
      std::array<int, 5> term{d->term_eci[t], d->term_ref[t], 0, 0, 0};
      for (int j = 0; j < m; ++j) {
        cols[j] = d->term_nb[3 * t + j] / B;
        term[2 + j] = d->term_nb[3 * t + j] % B;
      }
      auto it = geos.find(cols);
      if (it == geos.end()) {
        geo_order.push_back(cols);
        it = geos.emplace(cols, std::vector<std::array<int, 5>>{}).first;
      }
      it->second.push_back(term);
    }
    for (const auto &cols : geo_order) {
      std::vector<std::array<int, 5>> sig = geos[cols];
      std::sort(sig.begin(), sig.end());
      const int m = (int)cols.size();
      auto it = pats.find(sig);
      if (it == pats.end()) {
        int stride = 1;
        for (int j = 0; j < m; ++j) stride *= S;
        const int id = (int)pats.size();
        it = pats.emplace(sig, id).first;
        pat_info.insert(pat_info.end(), {m, tab_len, (int)pat_terms.size(), 0});
        for (const auto &tm : sig)
          pat_terms.push_back(tm[0] | (tm[1] << 8) | (tm[2] << 12) | (tm[3] << 16) | (tm[4] << 20));
        pat_info[4 * id + 3] = (int)pat_terms.size();
        tab_len += S * S * stride;
      }
      const int id = it->second;
      uint32_t packed = 0;
      for (int j = 0; j < 3; ++j) packed |= (uint32_t)(j < m ? cols[j] : C) << (8 * j);  // column C: species 0
      int stride = 1;
      for (int j = 0; j < m; ++j) stride *= S;
      geo_list.insert(geo_list.end(), {packed, (uint32_t)pat_info[4 * id + 1], (uint32_t)stride, 0u});
    }
  }
  n_geo = (int)(geo_list.size() / 4);
  n_pat = (int)pats.size();
  geo_start[G] = n_geo;
  if (tab_len > cemc::kMaxTable || n_geo > cemc::kMaxGeo) table_ok = false;
  if (geo_list.empty()) geo_list.assign(4, 0u);
  if (pat_info.empty()) pat_info.assign(4, 0);
  if (pat_terms.empty()) pat_terms.assign(1, 0);

  // The trial kernel's conflict test needs a symmetric neighbour relation:
  // j in row(i) <=> i in row(j).
  {
    std::vector<int32_t> sorted_rows(d->table, d->table + (size_t)N * C);
    for (int i = 0; i < N; ++i) std::sort(sorted_rows.begin() + (size_t)i * C, sorted_rows.begin() + (size_t)(i + 1) * C);
    for (int i = 0; i < N; ++i)
      for (int c = 0; c < C; ++c) {
        const int j = d->table[(size_t)i * C + c];
        auto b = sorted_rows.begin() + (size_t)j * C, e = b + C;
        if (!std::binary_search(b, e, i))
          return fail(CEMC_ERR_ARG, "neighbour relation is not symmetric (site %d in row %d but not back)", j, i);
      }
  }
  const int cpad = (C + 3) & ~3;
  std::vector<int32_t> table_pad((size_t)N * cpad);
  for (int i = 0; i < N; ++i)
    for (int c = 0; c < cpad; ++c) table_pad[(size_t)i * cpad + c] = d->table[(size_t)i * C + (c < C ? c : 0)];
  // the rows in 16 bits for the scheduled kernel (spin basis only: its rows are one cp.async ring entry)
  const int cp16 = (C + 7) & ~7;
  const bool has16 = N <= 65536 && B == 1 && G == 1 && C <= CEMC_SPIN_MAX_COLS;
  std::vector<uint16_t> table16(has16 ? (size_t)N * cp16 : 1);
  for (int i = 0; has16 && i < N; ++i)
    for (int c = 0; c < cp16; ++c) table16[(size_t)i * cp16 + c] = (uint16_t)d->table[(size_t)i * C + (c < C ? c : 0)];
  std::vector<int32_t> table_cm((size_t)N * C);
  for (int i = 0; i < N; ++i)
    for (int c = 0; c < C; ++c) table_cm[(size_t)c * N + i] = d->table[(size_t)i * C + c];
  std::vector<double> w(d->eci_weight, d->eci_weight + K), fw(d->eci_full_weight, d->eci_full_weight + K);

  // Binary spin basis (values +1 / -1): pair terms of a cluster ECI folded into
  // one shell mask; the other terms sorted by ECI and cut into 32 lane ranges.
  std::vector<cemc::SpinEci> spin_eci;
  std::vector<uint32_t> spin_masks;  // (lo, hi) pairs
  std::vector<int> spin_mask_cl;     // cluster-ECI slot of each mask
  std::vector<uint8_t> spin_shift;
  std::vector<int32_t> spin_lane_term(33, 0), spin_lane_first(32, 0);
  std::vector<int32_t> half_lane_term(17, 0), half_lane_first(16, 0);  // the same terms over 16 lanes
  std::vector<uint8_t> half_shift;
  int minus_id = -1, singlet_eci = -1;
  bool spin_ok = (B == 1 && S == 2 && C <= CEMC_SPIN_MAX_COLS && G == 1);
  if (spin_ok) {
    if (d->bf[0] == 1.0 && d->bf[1] == -1.0)
      minus_id = 1;
    else if (d->bf[0] == -1.0 && d->bf[1] == 1.0)
      minus_id = 0;
    else
      spin_ok = false;
  }
  for (int k = 0; spin_ok && k < K; ++k) {
    if (d->eci_kind[k] == 1) singlet_eci = k;
    if (d->eci_kind[k] != 2) continue;
    cemc::SpinEci e{};
    e.eci = k;
    uint64_t pairs = 0;
    for (int t = fterm_off[k]; t < fterm_off[k + 1]; ++t) {
      uint64_t m = 0;
      for (int j = 0; j < d->term_size[t] - 1; ++j) m |= (uint64_t)1 << (d->term_nb[3 * t + j]);
      if (d->term_size[t] == 2 && !(pairs & m)) {
        pairs |= m;
        e.n_pairs++;
      } else {
        spin_masks.push_back((uint32_t)m);
        spin_masks.push_back((uint32_t)(m >> 32));
        spin_mask_cl.push_back((int)spin_eci.size());
        e.n_multi++;
      }
    }
    e.pair_lo = (uint32_t)pairs;
    e.pair_hi = (uint32_t)(pairs >> 32);
    spin_eci.push_back(e);
  }
  if (spin_ok && (spin_eci.empty() || spin_eci.size() > CEMC_SPIN_MAX_CL)) spin_ok = false;
  const int n_masks = (int)spin_mask_cl.size();
  if (spin_ok) {
    const int q = (n_masks + 31) / 32;
    for (int l = 0; l <= 32; ++l) spin_lane_term[l] = std::min(l * q, n_masks);
    spin_shift.assign(std::max(n_masks, 1), 0);
    for (int l = 0; l < 32 && spin_ok; ++l) {
      const int lo = spin_lane_term[l], hi = spin_lane_term[l + 1];
      if (lo >= hi) continue;
      spin_lane_first[l] = spin_mask_cl[lo];
      for (int t = lo; t < hi; ++t) {
        const int sl = spin_mask_cl[t] - spin_lane_first[l];
        if (sl > 4 || hi - lo > 63) spin_ok = false;  // 5 six-bit counters per lane
        spin_shift[t] = (uint8_t)(6 * sl);
      }
    }
  }
  // Half-warp form (two flips per warp): cluster ECIs on lanes 0..15, the
  // multi-site terms cut into 16 lane ranges with the same 6-bit counters.
  bool half_ok = spin_ok && spin_eci.size() <= 16;
  if (half_ok) {
    const int q = (n_masks + 15) / 16;
    for (int l = 0; l <= 16; ++l) half_lane_term[l] = std::min(l * q, n_masks);
    half_shift.assign(std::max(n_masks, 1), 0);
    for (int l = 0; l < 16 && half_ok; ++l) {
      const int lo = half_lane_term[l], hi = half_lane_term[l + 1];
      if (lo >= hi) continue;
      half_lane_first[l] = spin_mask_cl[lo];
      for (int t = lo; t < hi; ++t) {
        const int sl = spin_mask_cl[t] - half_lane_first[l];
        if (sl > 4 || hi - lo > 63) half_ok = false;
        half_shift[t] = (uint8_t)(6 * sl);
      }
    }
  }
  // Local-field form (single-site flips in the spin basis, cemc_field.h): one
  // count field per cluster ECI, packed into at most two words per site, and
  // the update list of a changed site j, derived from site 0's neighbourhood
  // and verified to hold at every site (a periodic supercell of one
  // translation group); rows must list distinct sites other than the site.
  bool field_ok = spin_ok && n_movable == N && N <= cemc::kFieldMaxSites &&
                  (int)spin_eci.size() <= cemc::kFieldMaxCl;
  int field_pw = 1;
  std::vector<int32_t> f_slot_eci, f_ustart(C + 1, 0);
  std::vector<uint32_t> f_meta, f_cnt, f_pairinc, f_upd;
  if (field_ok) {
    const int ncl = (int)spin_eci.size();
    std::vector<int> fword(ncl, 0), fshift(ncl, 0);
    int word = 0, used = 0;
    for (int q = 0; q < ncl && field_ok; ++q) {
      const int Kq = spin_eci[q].n_pairs + spin_eci[q].n_multi;
      int bits = 1;
      while ((1 << bits) <= Kq) ++bits;
      if (Kq > 255) field_ok = false;
      if (used + bits > 32) {
        ++word;
        used = 0;
      }
      if (word > 1) field_ok = false;
      fword[q] = word;
      fshift[q] = used;
      used += bits;
      f_slot_eci.push_back(spin_eci[q].eci);
      f_meta.push_back((uint32_t)Kq | ((uint32_t)fshift[q] << 8) | ((uint32_t)word << 13) | ((uint32_t)bits << 16));
    }
    field_pw = word + 1;
    auto add_inc = [&](int q, uint32_t *w) { w[fword[q]] += 1u << fshift[q]; };
    // (site, column) keys of every row, sorted by site: the column of a site in a row
    std::vector<uint64_t> keys(field_ok ? (size_t)N * C : 0);
    for (int i = 0; i < N && field_ok; ++i) {
      uint64_t *k = keys.data() + (size_t)i * C;
      for (int c = 0; c < C; ++c) {
        const int s = d->table[(size_t)i * C + c];
        if (s == i) field_ok = false;
        k[c] = ((uint64_t)(uint32_t)s << 8) | (uint64_t)c;
      }
      std::sort(k, k + C);
      for (int c = 1; c < C; ++c)
        if ((k[c] >> 8) == (k[c - 1] >> 8)) field_ok = false;
    }
    auto col_of = [&](int i, int x) -> int {
      const uint64_t *b = keys.data() + (size_t)i * C, *e = b + C;
      const uint64_t *p = std::lower_bound(b, e, (uint64_t)(uint32_t)x << 8);
      return (p != e && (*p >> 8) == (uint64_t)(uint32_t)x) ? (int)(*p & 255u) : -1;
    };
    std::vector<int> inv(C, -1);  // row_{row_j[c]}[inv[c]] = j
    for (int c = 0; c < C && field_ok; ++c) {
      inv[c] = col_of(d->table[c], 0);
      if (inv[c] < 0) field_ok = false;
    }
    std::vector<std::array<int, 3>> cmap;  // (c, c2, c3): row_j[c3] = row_{row_j[c]}[c2]
    if (field_ok) {
      for (int q = 0; q < ncl; ++q) {  // count entries: pair shells, then multi-site terms
        uint32_t w[2] = {0, 0};
        add_inc(q, w);
        f_cnt.insert(f_cnt.end(), {spin_eci[q].pair_lo, spin_eci[q].pair_hi, w[0], w[1]});
      }
      for (int t = 0; t < n_masks; ++t) {
        uint32_t w[2] = {0, 0};
        add_inc(spin_mask_cl[t], w);
        f_cnt.insert(f_cnt.end(), {spin_masks[2 * t], spin_masks[2 * t + 1], w[0], w[1]});
      }
      for (int c = 0; c < C && field_ok; ++c) {
        f_ustart[c] = (int32_t)(f_upd.size() / 4);
        const int i = d->table[c];  // the target row_0[c]
        const int cp = inv[c];      // site 0 seen from the target
        const uint64_t bit = (uint64_t)1 << cp;
        uint32_t pinc[2] = {0, 0};
        for (int q = 0; q < ncl; ++q)
          if ((((uint64_t)spin_eci[q].pair_hi << 32) | spin_eci[q].pair_lo) & bit) add_inc(q, pinc);
        f_pairinc.insert(f_pairinc.end(), {pinc[0], pinc[1]});
        // Terms at the target through site 0, by cluster slot: those with one other member
        // are counted together (one mask; the count of -1 products is a popcount), the
        // others (and repeated single members) toggle one by one with their parity.
        std::vector<uint64_t> single(ncl, 0);
        std::vector<uint64_t> multi;
        std::vector<int> multi_q;
        for (int t = 0; t < n_masks && field_ok; ++t) {
          const uint64_t m = ((uint64_t)spin_masks[2 * t + 1] << 32) | spin_masks[2 * t];
          if (!(m & bit)) continue;
          uint64_t others = m & ~bit, mj = 0;
          while (others) {
            const int c2 = __builtin_ctzll(others);
            others &= others - 1;
            const int c3 = col_of(0, d->table[(size_t)i * C + c2]);
            if (c3 < 0) {
              field_ok = false;
              break;
            }
            mj |= (uint64_t)1 << c3;
            cmap.push_back({c, c2, c3});
          }
          const int q = spin_mask_cl[t];
          if (__builtin_popcountll(mj) == 1 && !(single[q] & mj)) {
            single[q] |= mj;
          } else {
            multi.push_back(mj);
            multi_q.push_back(q);
          }
        }
        // entry {mask lo, mask hi, field increment, word | kind << 1 | members << 8}
        for (int q = 0; q < ncl && field_ok; ++q)
          if (single[q])
            f_upd.insert(f_upd.end(), {(uint32_t)single[q], (uint32_t)(single[q] >> 32), 1u << fshift[q],
                                       (uint32_t)fword[q] | 2u | ((uint32_t)__builtin_popcountll(single[q]) << 8)});
        for (size_t e = 0; e < multi.size() && field_ok; ++e) {
          const int q = multi_q[e];
          f_upd.insert(f_upd.end(), {(uint32_t)multi[e], (uint32_t)(multi[e] >> 32), 1u << fshift[q],
                                     (uint32_t)fword[q]});
        }
      }
      f_ustart[C] = (int32_t)(f_upd.size() / 4);
      std::sort(cmap.begin(), cmap.end());
      cmap.erase(std::unique(cmap.begin(), cmap.end()), cmap.end());
    }
    for (int j = 1; j < N && field_ok; ++j) {
      const int32_t *rj = d->table + (size_t)j * C;
      for (int c = 0; c < C; ++c)
        if (col_of(rj[c], j) != inv[c]) field_ok = false;
      for (const auto &m : cmap)
        if (col_of(j, d->table[(size_t)rj[m[0]] * C + m[1]]) != m[2]) field_ok = false;
    }
  }
  if (!field_ok) {
    f_slot_eci.assign(1, 0);
    f_meta.assign(1, 0u);
    f_cnt.assign(4, 0u);
    f_pairinc.assign(2 * (size_t)C, 0u);
    f_ustart.assign(C + 1, 0);
    f_upd.assign(4, 0u);
  }
  if (f_upd.empty()) f_upd.assign(4, 0u);
  // Quarter-warp form (four flips per warp): cluster ECIs on lanes 0..7, the multi-site terms cut
  // into 8 lane ranges with the same 6-bit counters; a trial's odd-term count of one cluster ECI
  // is summed in an 8-bit field of one warp reduction, so no ECI may have more than 255 terms.
  std::vector<int32_t> qtr_lane_term(9, 0), qtr_lane_first(8, 0);
  std::vector<uint8_t> qtr_shift;
  bool qtr_ok = spin_ok && spin_eci.size() <= 8;
  for (const auto &e : spin_eci) qtr_ok = qtr_ok && e.n_multi <= 255;
  if (qtr_ok) {
    const int q = (n_masks + 7) / 8;
    for (int l = 0; l <= 8; ++l) qtr_lane_term[l] = std::min(l * q, n_masks);
    qtr_shift.assign(std::max(n_masks, 1), 0);
    for (int l = 0; l < 8 && qtr_ok; ++l) {
      const int lo = qtr_lane_term[l], hi = qtr_lane_term[l + 1];
      if (lo >= hi) continue;
      qtr_lane_first[l] = spin_mask_cl[lo];
      for (int t = lo; t < hi; ++t) {
        const int sl = spin_mask_cl[t] - qtr_lane_first[l];
        if (sl > 4 || hi - lo > 63) qtr_ok = false;
        qtr_shift[t] = (uint8_t)(6 * sl);
      }
    }
  }
  if (qtr_shift.empty()) qtr_shift.assign(1, 0);
  if (half_shift.empty()) half_shift.assign(1, 0);
  if (spin_eci.empty()) spin_eci.push_back(cemc::SpinEci{});
  if (spin_masks.empty()) spin_masks.assign(2, 0u);
  if (spin_shift.empty()) spin_shift.assign(1, 0);

  // Periodic box of cells (DevGeo::box_L): sites ((x * L + y) * L + z) * nb + b, and at every
  // site the table holds the same (cell offset, basis site) per (b, column) as at cell 0.  Tried
  // for one translation group without background sites, for each basis count nb <= 8 with N / nb
  // a cube; every entry of the table and the multiply-high divisions are checked.
  int box_L = 0, box_nb = 0;
  uint32_t box_mnb = 0, box_mL = 0;
  std::vector<uint32_t> box_off;
  auto umulhi = [](uint32_t a, uint32_t m) { return (uint32_t)(((uint64_t)a * m) >> 32); };
  auto magic = [](uint32_t dv) { return (uint32_t)((((uint64_t)1 << 32) + dv - 1) / dv); };  // ceil(2^32 / dv)
  for (int nb = 1; nb <= 8 && box_L == 0 && G == 1 && n_movable == N; ++nb) {
    if (N % nb) continue;
    const int cells = N / nb;
    const int L = (int)std::lround(std::cbrt((double)cells));
    if ((long long)L * L * L != cells || L > 255) continue;
    auto decode = [&](int site, int &x, int &y, int &z) {
      int c = site / nb;
      z = c % L;
      c /= L;
      y = c % L;
      x = c / L;
      return site % nb;
    };
    auto near = [&](int v) { return 2 * v > L ? v - L : v; };  // minimal image in (-L/2, L/2]
    std::vector<uint32_t> off((size_t)nb * C);
    for (int b = 0; b < nb; ++b)
      for (int c = 0; c < C; ++c) {
        int x, y, z;
        const int bb = decode(d->table[(size_t)b * C + c], x, y, z);
        off[(size_t)b * C + c] = (uint32_t)(near(x) + 128) | ((uint32_t)(near(y) + 128) << 8) |
                                 ((uint32_t)(near(z) + 128) << 16) | ((uint32_t)bb << 24);
      }
    bool ok = true;
    for (int site = 0; site < N && ok; ++site) {
      int x, y, z;
      const int b = decode(site, x, y, z);
      for (int c = 0; c < C; ++c) {
        const uint32_t o = off[(size_t)b * C + c];
        int nx = x + (int)(o & 255u) - 128, ny = y + (int)((o >> 8) & 255u) - 128, nz = z + (int)((o >> 16) & 255u) - 128;
        nx += nx < 0 ? L : 0;
        nx -= nx >= L ? L : 0;
        ny += ny < 0 ? L : 0;
        ny -= ny >= L ? L : 0;
        nz += nz < 0 ? L : 0;
        nz -= nz >= L ? L : 0;
        if (((nx * L + ny) * L + nz) * nb + (int)(o >> 24) != d->table[(size_t)site * C + c]) {
          ok = false;
          break;
        }
      }
    }
    const uint32_t mnb = nb > 1 ? magic((uint32_t)nb) : 0u, mL = L > 1 ? magic((uint32_t)L) : 0u;
    for (uint32_t v = 0; ok && nb > 1 && v < (uint32_t)N; ++v) ok = umulhi(v, mnb) == v / (uint32_t)nb;
    for (uint32_t v = 0; ok && L > 1 && v < (uint32_t)cells; ++v) ok = umulhi(v, mL) == v / (uint32_t)L;
    if (ok) {
      box_L = L;
      box_nb = nb;
      box_mnb = mnb;
      box_mL = mL;
      box_off.swap(off);
    }
  }
  if (box_off.empty()) box_off.assign(1, 0u);

  // Bit-plane recompute of a periodic box (cemc_boxcf.h): the sub-clusters of every basis site grouped into
  // orbits under lattice translation, orbits with the same terms into patterns.
  std::vector<int32_t> bx_job, bx_ent, bx_ent_start, bx_k_start(K + 1, 0), bx_k_count;
  std::vector<double> bx_k_w, bx_k_const(K, 0.0);
  int bx_n_counts = 0, bx_hx = 0;
  const bool bx_pm1 = B == 1 && ((d->bf[0] == 1.0 && d->bf[1] == -1.0) || (d->bf[0] == -1.0 && d->bf[1] == 1.0));
  bool bx_ok = box_L > 0 && box_L <= cemc::kBoxMaxL && S <= 3;
  if (bx_ok) {
    using Point = std::array<int, 4>;                          // x, y, z (mod L), basis site
    using Term = std::array<int, 5>;                           // ECI, decoration of each point
    const int L = box_L;
    std::map<std::vector<int>, std::vector<Term>> geos;        // member columns -> terms (own decoration first)
    for (int t = 0; t < T; ++t) {
      std::vector<int> cols;
      Term tm{d->term_eci[t], d->term_ref[t], 0, 0, 0};
      for (int j = 0; j < d->term_size[t] - 1; ++j) {
        cols.push_back(d->term_nb[3 * t + j] / B);
        tm[2 + j] = d->term_nb[3 * t + j] % B;
      }
      geos[cols].push_back(tm);
    }
    std::map<std::vector<Point>, std::map<Term, int>> orbits;  // points, the first in cell 0 -> terms and counts
    for (int b = 0; b < box_nb; ++b)
      for (const auto &ge : geos) {
        std::vector<Point> pts{{0, 0, 0, b}};
        for (int col : ge.first) {
          const uint32_t o = box_off[(size_t)b * C + col];
          pts.push_back({(int)(o & 255u) - 128, (int)((o >> 8) & 255u) - 128, (int)((o >> 16) & 255u) - 128, (int)(o >> 24)});
        }
        const int n = (int)pts.size();
        std::vector<Point> best;
        std::vector<int> order;  // order[i]: position in pts of the i-th canonical point
        for (int from = 0; from < n; ++from) {
          std::vector<std::pair<Point, int>> list;
          for (int i = 0; i < n; ++i) {
            Point p = pts[i];
            for (int q = 0; q < 3; ++q) p[q] = ((p[q] - pts[from][q]) % L + L) % L;
            list.push_back({p, i});
          }
          std::sort(list.begin(), list.end());
          std::vector<Point> key;
          for (const auto &e : list) key.push_back(e.first);
          if (best.empty() || key < best) {
            best = key;
            order.clear();
            for (const auto &e : list) order.push_back(e.second);
          }
        }
        auto &terms = orbits[best];
        for (const Term &tm : ge.second) {
          Term c{tm[0], 0, 0, 0, 0};
          if (!bx_pm1)
            for (int i = 0; i < n; ++i) c[1 + i] = tm[1 + order[i]];
          terms[c] += 1;
        }
      }
    std::map<std::pair<int, std::map<Term, int>>, int> pats;
    std::vector<int> pat_first, pat_orbits;                // first counter, orbits
    std::vector<std::vector<std::array<int, 4>>> pat_ents; // basis site, offsets
    auto near_l = [&](int v) { return 2 * v > box_L ? v - box_L : v; };
    auto pack_point = [&](const Point &p) {
      const int x = near_l(p[0]), y = near_l(p[1]);
      bx_hx = std::max(bx_hx, std::abs(x));
      return (int)((uint32_t)(x + 128) | ((uint32_t)(y + 128) << 8) | ((uint32_t)p[2] << 16) | ((uint32_t)p[3] << 24));
    };
    for (const auto &ob : orbits) {
      const int n = (int)ob.first.size();
      const auto key = std::make_pair(n, ob.second);
      auto it = pats.find(key);
      if (it == pats.end()) {
        it = pats.emplace(key, (int)pats.size()).first;
        int tuples = 1;
        for (int i = 0; i < n && !bx_pm1; ++i) tuples *= S;
        pat_first.push_back(bx_n_counts);
        bx_n_counts += tuples;
        pat_orbits.push_back(0);
        pat_ents.push_back({});
      }
      pat_orbits[it->second] += 1;
      std::array<int, 4> e{ob.first[0][3], 0, 0, 0};
      for (int i = 1; i < n; ++i) e[i] = pack_point(ob.first[i]);
      pat_ents[it->second].push_back(e);
    }
    // jobs: the orbits of a pattern, by basis site of their first point, kBoxJob of each at a time
    bx_ent_start.assign(1, 0);
    for (const auto &pt : pats) {
      std::vector<std::vector<std::array<int, 4>>> by_b(box_nb);
      size_t most = 0;
      for (const auto &e : pat_ents[pt.second]) by_b[e[0]].push_back(e);
      for (const auto &v : by_b) most = std::max(most, v.size());
      for (size_t at = 0; at < most; at += cemc::kBoxJob) {
        bx_job.insert(bx_job.end(), {pt.first.first, pat_first[pt.second]});
        for (const auto &v : by_b) {
          for (size_t i = at; i < std::min(v.size(), at + cemc::kBoxJob); ++i)
            bx_ent.insert(bx_ent.end(), {v[i][1], v[i][2], v[i][3], 0});
          bx_ent_start.push_back((int32_t)(bx_ent.size() / 4));
        }
      }
    }
    // each ECI's sum over all sites as a weighted sum of counters
    const double cells = (double)(N / box_nb);
    std::vector<std::map<int, double>> w(K);
    for (const auto &pt : pats) {
      const int n = pt.first.first, id = pt.second, c0 = pat_first[id];
      for (const auto &tm : pt.first.second) {
        const int k = tm.first[0];
        const double mult = (double)tm.second;
        if (bx_pm1) {
          w[k][c0] -= 2.0 * mult;
          bx_k_const[k] += mult * cells * pat_orbits[id];
          continue;
        }
        int tuples = 1;
        for (int i = 0; i < n; ++i) tuples *= S;
        for (int q = 0; q < tuples; ++q) {
          double v = mult;
          for (int i = 0, r = q; i < n; ++i, r /= S) v *= d->bf[tm.first[1 + i] * S + r % S];
          w[k][c0 + q] += v;
        }
      }
    }
    for (int k = 0; k < K; ++k) {
      for (const auto &e : w[k]) {
        bx_k_count.push_back(e.first);
        bx_k_w.push_back(e.second);
      }
      bx_k_start[k + 1] = (int32_t)bx_k_count.size();
    }
    bx_ok = !bx_job.empty() && bx_n_counts <= cemc::kBoxMaxCounts;
  }
  const int bx_n_jobs = (int)(bx_job.size() / 2), bx_n_ents = (int)(bx_ent.size() / 4);
  if (bx_job.empty()) bx_job.assign(2, 0);
  if (bx_ent.empty()) bx_ent.assign(4, 0);
  if (bx_ent_start.empty()) bx_ent_start.assign(1, 0);
  if (bx_k_count.empty()) bx_k_count.assign(1, 0);
  if (bx_k_w.empty()) bx_k_w.assign(1, 0.0);

  // One device allocation for all tables.
  struct Part {
    const void *src;
    size_t bytes;
    size_t off;
  };
  std::vector<Part> parts = {
      {table_pad.data(), sizeof(int32_t) * N * cpad, 0}, {table_cm.data(), sizeof(int32_t) * N * C, 0},
      {terms.data(), terms.size() * 2, 0},         {lane_term.data(), lane_term.size() * 4, 0},
      {first.data(), first.size() * 4, 0},         {eci_lane.data(), eci_lane.size() * 4, 0},
      {d->eci_kind, sizeof(int32_t) * K, 0},       {d->eci_dec, sizeof(int32_t) * K, 0},
      {w.data(), sizeof(double) * K, 0},           {fw.data(), sizeof(double) * K, 0},
      {d->bf, sizeof(double) * B * S, 0},          {fterms.data(), fterms.size(), 0},
      {fterm_off.data(), fterm_off.size() * 4, 0},
      {spin_eci.data(), spin_eci.size() * sizeof(cemc::SpinEci), 0},
      {spin_masks.data(), spin_masks.size() * 4, 0},
      {spin_shift.data(), spin_shift.size(), 0},
      {spin_lane_term.data(), 33 * 4, 0},
      {spin_lane_first.data(), 32 * 4, 0},
      {half_shift.data(), half_shift.size(), 0},
      {half_lane_term.data(), 17 * 4, 0},
      {half_lane_first.data(), 16 * 4, 0},
      {geo_list.data(), geo_list.size() * 4, 0},
      {pat_info.data(), pat_info.size() * 4, 0},
      {pat_terms.data(), pat_terms.size() * 4, 0},
      {movable.data(), movable.size() * 4, 0},
      {site_active.data(), site_active.size(), 0},
      {sgroup.data(), sgroup.size(), 0},
      {geo_start.data(), geo_start.size() * 4, 0},
      {gscale.data(), gscale.size() * 8, 0},
      {f_slot_eci.data(), f_slot_eci.size() * 4, 0},
      {f_meta.data(), f_meta.size() * 4, 0},
      {f_cnt.data(), f_cnt.size() * 4, 0},
      {f_pairinc.data(), f_pairinc.size() * 4, 0},
      {f_ustart.data(), f_ustart.size() * 4, 0},
      {f_upd.data(), f_upd.size() * 4, 0},
      {box_off.data(), box_off.size() * 4, 0},
      {qtr_shift.data(), qtr_shift.size(), 0},
      {qtr_lane_term.data(), 9 * 4, 0},
      {qtr_lane_first.data(), 8 * 4, 0},
      {table16.data(), table16.size() * 2, 0},
      {bx_job.data(), bx_job.size() * 4, 0},
      {bx_ent.data(), bx_ent.size() * 4, 0},
      {bx_ent_start.data(), bx_ent_start.size() * 4, 0},
      {bx_k_start.data(), bx_k_start.size() * 4, 0},
      {bx_k_count.data(), bx_k_count.size() * 4, 0},
      {bx_k_w.data(), bx_k_w.size() * 8, 0},
      {bx_k_const.data(), bx_k_const.size() * 8, 0},
  };
  size_t total = 0;
  for (auto &p : parts) {
    p.off = total;
    total = align_up(total + p.bytes, 256);
  }
  cemc_geometry *geo = new cemc_geometry();
  geo->dev_bytes = total;
  cudaError_t e = cudaMalloc(&geo->dev, total);
  if (e != cudaSuccess) {
    delete geo;
    return cuda_fail(e, "cudaMalloc(geometry tables)");
  }
  std::vector<unsigned char> host(total, 0);
  for (auto &p : parts) memcpy(host.data() + p.off, p.src, p.bytes);
  e = cudaMemcpy(geo->dev, host.data(), total, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(geo->dev);
    delete geo;
    return cuda_fail(e, "cudaMemcpy(geometry tables)");
  }
  unsigned char *base = static_cast<unsigned char *>(geo->dev);
  cemc::DevGeo &g = geo->g;
  g.n_sites = N;
  g.n_cols = C;
  g.n_sym = S;
  g.n_bf = B;
  g.n_eci = K;
  g.n_terms = T;
  g.vals_len = one_idx + 1 + B;
  g.one_idx = one_idx;
  g.n_slots = n_slots;
  g.cpad = cpad;
  g.table = reinterpret_cast<const int32_t *>(base + parts[0].off);
  g.table16 = has16 ? reinterpret_cast<const uint16_t *>(base + parts[39].off) : nullptr;
  g.cp16 = cp16;
  g.table_cm = reinterpret_cast<const int32_t *>(base + parts[1].off);
  g.terms = reinterpret_cast<const uint16_t *>(base + parts[2].off);
  g.lane_term = reinterpret_cast<const int32_t *>(base + parts[3].off);
  g.lane_first_eci = reinterpret_cast<const int32_t *>(base + parts[4].off);
  g.eci_lane = reinterpret_cast<const int32_t *>(base + parts[5].off);
  g.eci_kind = reinterpret_cast<const int32_t *>(base + parts[6].off);
  g.eci_dec = reinterpret_cast<const int32_t *>(base + parts[7].off);
  g.eci_w = reinterpret_cast<const double *>(base + parts[8].off);
  g.eci_fw = reinterpret_cast<const double *>(base + parts[9].off);
  g.bf = reinterpret_cast<const double *>(base + parts[10].off);
  g.fterms = reinterpret_cast<const uint8_t *>(base + parts[11].off);
  g.fterm_off = reinterpret_cast<const int32_t *>(base + parts[12].off);
  for (int b = 0; b < CEMC_MAX_BF; ++b) g.singlet_eci[b] = singlet[b];
  g.table_ok = table_ok ? 1 : 0;
  g.n_geo = n_geo;
  g.n_pat = n_pat;
  g.tab_len = tab_len;
  g.geo_list = reinterpret_cast<const uint4 *>(base + parts[21].off);
  g.pat_info = reinterpret_cast<const int4 *>(base + parts[22].off);
  g.pat_terms = reinterpret_cast<const int32_t *>(base + parts[23].off);
  g.n_movable = n_movable;
  g.movable = reinterpret_cast<const int32_t *>(base + parts[24].off);
  g.site_active = n_movable == N ? nullptr : reinterpret_cast<const int8_t *>(base + parts[25].off);
  g.n_groups = G;
  g.site_group = reinterpret_cast<const int8_t *>(base + parts[26].off);
  g.geo_start = reinterpret_cast<const int32_t *>(base + parts[27].off);
  g.group_scale = reinterpret_cast<const double *>(base + parts[28].off);
  g.box_L = box_L;
  g.box_nb = box_nb;
  g.box_mnb = box_mnb;
  g.box_mL = box_mL;
  g.box_off = reinterpret_cast<const uint32_t *>(base + parts[35].off);
  g.pm1_minus = -1;
  if (B == 1 && S == 2) {
    if (d->bf[0] == 1.0 && d->bf[1] == -1.0) g.pm1_minus = 1;
    else if (d->bf[0] == -1.0 && d->bf[1] == 1.0) g.pm1_minus = 0;
  }
  geo->box.ok = bx_ok ? 1 : 0;
  geo->box.pm1 = bx_pm1 ? 1 : 0;
  geo->box.n_jobs = bx_n_jobs;
  geo->box.n_ents = bx_n_ents;
  geo->box.n_counts = bx_n_counts;
  geo->box.hx = bx_hx;
  geo->box.job = reinterpret_cast<const int2 *>(base + parts[40].off);
  geo->box.ent = reinterpret_cast<const int4 *>(base + parts[41].off);
  geo->box.ent_start = reinterpret_cast<const int32_t *>(base + parts[42].off);
  geo->box.k_start = reinterpret_cast<const int32_t *>(base + parts[43].off);
  geo->box.k_count = reinterpret_cast<const int32_t *>(base + parts[44].off);
  geo->box.k_w = reinterpret_cast<const double *>(base + parts[45].off);
  geo->box.k_const = reinterpret_cast<const double *>(base + parts[46].off);
  geo->spin_ok = spin_ok;
  geo->spin.n_cl = spin_ok ? (int)spin_eci.size() : 0;
  geo->spin.n_masks = spin_ok ? n_masks : 0;
  geo->spin.minus_id = minus_id;
  geo->spin.singlet_eci = singlet_eci;
  geo->spin.eci = reinterpret_cast<const cemc::SpinEci *>(base + parts[13].off);
  geo->spin.masks = reinterpret_cast<const uint2 *>(base + parts[14].off);
  geo->spin.shift = reinterpret_cast<const uint8_t *>(base + parts[15].off);
  geo->spin.lane_term = reinterpret_cast<const int32_t *>(base + parts[16].off);
  geo->spin.lane_first = reinterpret_cast<const int32_t *>(base + parts[17].off);
  geo->spin.qtr_ok = qtr_ok ? 1 : 0;
  geo->spin.qtr_shift = reinterpret_cast<const uint8_t *>(base + parts[36].off);
  geo->spin.qtr_lane_term = reinterpret_cast<const int32_t *>(base + parts[37].off);
  geo->spin.qtr_lane_first = reinterpret_cast<const int32_t *>(base + parts[38].off);
  geo->spin.half_ok = half_ok ? 1 : 0;
  geo->spin.half_shift = reinterpret_cast<const uint8_t *>(base + parts[18].off);
  geo->spin.half_lane_term = reinterpret_cast<const int32_t *>(base + parts[19].off);
  geo->spin.half_lane_first = reinterpret_cast<const int32_t *>(base + parts[20].off);
  geo->field_ok = field_ok;
  geo->field.n_cl = field_ok ? (int)f_slot_eci.size() : 0;
  geo->field.pw = field_pw;
  geo->field.n_cnt = field_ok ? (int)(f_cnt.size() / 4) : 0;
  geo->field.n_upd = field_ok ? (int)f_ustart[C] : 0;
  geo->field.minus_id = minus_id;
  geo->field.singlet_eci = singlet_eci;
  geo->field.slot_eci = reinterpret_cast<const int32_t *>(base + parts[29].off);
  geo->field.slot_meta = reinterpret_cast<const uint32_t *>(base + parts[30].off);
  geo->field.cnt = reinterpret_cast<const uint4 *>(base + parts[31].off);
  geo->field.pairinc = reinterpret_cast<const uint2 *>(base + parts[32].off);
  geo->field.ustart = reinterpret_cast<const int32_t *>(base + parts[33].off);
  geo->field.upd = reinterpret_cast<const uint4 *>(base + parts[34].off);
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&geo->max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  geo->g.max_smem = geo->max_smem;
  cudaDeviceGetAttribute(&geo->n_sms, cudaDevAttrMultiProcessorCount, dev);
  *out = geo;
  return CEMC_OK;
}

extern "C" int cemc_geometry_destroy(cemc_geometry *geo) {
  if (!geo) return CEMC_OK;
  cudaError_t e = cudaFree(geo->dev);
  delete geo;
  if (e != cudaSuccess) return cuda_fail(e, "cudaFree(geometry tables)");
  return CEMC_OK;
}

extern "C" size_t cemc_geometry_device_bytes(const cemc_geometry *geo) { return geo ? geo->dev_bytes : 0; }

extern "C" size_t cemc_stamp_words(const cemc_geometry *geo, int32_t n_chains) {
  if (!geo || n_chains <= 0) return 0;
  int bits = 5;
  while ((1 << bits) < geo->g.n_sites) ++bits;
  return 2 * ((size_t)1 << bits) * (size_t)n_chains;
}

namespace {

// Full recompute: by bit planes in a periodic box, else term by term through the neighbour table.
cudaError_t recompute(const cemc_geometry *geo, int n_chains, const int8_t *occ, const double *eci, double *cf,
                      double *energy, double *scratch, void *stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  size_t smem = 0;
  const int ctas = cemc::boxcf_ctas(geo->g, geo->box, n_chains, geo->n_sms, (size_t)geo->max_smem, &smem);
  if (ctas) return cemc::launch_boxcf(geo->g, geo->box, n_chains, ctas, smem, occ, eci, cf, energy, st);
  return cemc::launch_recompute(geo->g, n_chains, occ, eci, cf, energy, scratch, st);
}

// A scheduled kernel for a launch: not at all, for all of its calls, or for those whose chains' state on the device
// favours it (cemc_route.h).
struct Scheduled {
  enum { kNo = 0, kRouted, kAlways } how = kNo;
  cemc::RunArgs args;
  cemc::Route route{};
  size_t smem = 0;
};

// The scheduled flip kernel for this geometry in booking rounds of `part` trials, instead of the speculative launch
// `a` with `smem` bytes and `beside` chains of other launches next to it.
//
// Trials that touch one another cannot share a tick: with n_movable / (n_cols + 1) neighbourhoods in the
// cell, about a third of that many trials can run at once, so small cells take fewer evaluating warps and
// the smallest stay with the speculative forms, whose rounds they fill.  Measured (FCC, pairs to the 4th
// shell; ms, half-warp form / here with 8 / 12 / 16 evaluating warps, FP32):
//   2048 sites, 37 neighbourhoods   3.57 / 2.84 / 2.95 / 3.00     864 sites, 16: 4.87 / 6.1 and more
//   4000 sites, 73                  4.79 / 2.80 / 2.56 / 2.62
//   16384 sites, 298                5.36 / 3.20 / 2.69 / 2.61     55296 sites, 1005: 8.63 / 6.44 / 5.26 / 4.86
//
// Rounds of chains that accept little are committed nearly whole, while a tick takes its time whatever is
// accepted, so small cells take this kernel from an acceptance on.  Speculative time over time here, 64 chains,
// FP32, by the trials of a round and the acceptance:
//                           0.005  0.08   0.12   0.20   0.28   0.51   0.63   0.70   0.85
//   37 neighbourhoods   8    0.91          0.96                               1.12   1.17
//                      16    0.62   0.69   0.72   0.80   0.85   1.03   1.12   1.14   1.23
//                      18    0.49   0.55   0.59   0.67   0.70   0.87   0.95   0.99   1.08
//                      32    0.38   0.50   0.57   0.72   0.81   1.09   1.21   1.28   1.40
//   53                  8    1.20          1.24                               1.38   1.39
//                      16    0.85   0.92   0.96   1.03   1.09   1.25   1.34   1.36   1.43
//                      32    0.52   0.65   0.72   0.88   0.97   1.28   1.39   1.46   1.58
//   72                 16    1.06   1.14   1.16   1.24   1.27   1.41   1.47   1.49   1.55
//                      32    0.67   0.79   0.86   0.98   1.09   1.38   1.51   1.54   1.67
//   125                16    1.36   1.44          1.50   1.53   1.60   1.64   1.64   1.65
//                      32    0.90   1.00   1.07   1.15   1.26   1.48   1.56   1.61   1.70
//   159                32    1.05   1.15          1.31   1.35   1.54   1.62
//   1005               32    1.22   1.49          1.59   1.64   1.89   2.06
//         64, FP32 / FP64    0.85 / 0.82  1.04 / 0.90  1.16 / 0.96  1.22 / 1.00 (acceptance 0.005, 0.08, 0.24, 0.28)
//
// One chain takes an SM here.  Two or three CTAs of the speculative forms share one where the cell is small, so with
// more chains than SMs they are the faster ones, but for wide rounds above 48 neighbourhoods: 200 hot chains, ms,
// rounds of 8 / 16 / 32 trials, there and here: 2048 sites 1.96 2.96 / 2.12 2.86 / 2.82 2.85, 2916 2.09 2.65 / 2.07
// 2.46 / 2.70 2.42, 4000 2.06 2.30 / 1.88 2.04 / 2.37 2.00; 6912 (one CTA an SM) 3.99 2.30 / 3.11 1.87 / 2.97 1.74.
void fit_sched(const cemc_geometry *geo, int precision, int part, size_t smem, int beside, Scheduled &s) {
  const cemc::DevGeo &g = geo->g;
  const int rsize = precision == CEMC_PREC_F32 ? 4 : 8;
  const int room = g.n_movable / (g.n_cols + 1);
  if (room < 32) return;
  cemc::RunArgs &a = s.args;
  if ((int64_t)a.n_chains + beside > geo->n_sms && room < 150 && (part < 32 || room < 48)) {
    const auto key = std::make_tuple(a.warps, (int)CEMC_MOVE_FLIP, precision, -a.tpw, smem);
    std::lock_guard<std::mutex> lock(geo->mu);
    auto it = geo->pairs.find(key);
    if (it == geo->pairs.end()) it = geo->pairs.emplace(key, cemc::spin_flip_blocks(g, a, precision, smem)).first;
    if (it->second > 1) return;
  }
  a.warps = room < 64 ? 8 : (room < 128 ? 12 : 16);
  a.part = part;
  int exact = 5;
  while ((1 << exact) < g.n_sites) ++exact;
  // rows of 512 trials cover the eight or so ticks between a row's fetch and the end of its trial; 256
  // (which stalls 12 and 16 warps) where the hash would be left with fewer than 2^13 buckets
  for (int rows = 9; rows >= 8 && !s.how; --rows)
    for (int hb = exact; hb >= (rows == 9 ? std::min(exact, 13) : 8) && !s.how; --hb) {
      a.row_bits = rows;
      a.ring_bits = rows + 1;  // a mask's 255 trials before the oldest unfinished one stay in the ring
      a.head_bits = hb;
      s.smem = cemc::sched_layout(g, geo->spin.n_cl, geo->spin.n_masks, rsize, 4 * a.warps, a.ring_bits, a.row_bits,
                                  a.head_bits).total;
      if (s.smem <= (size_t)geo->max_smem) s.how = Scheduled::kRouted;
    }
  if (!s.how) return;
  double hot;
  if (part <= 8) hot = room < 48 ? 0.3 : 0.0;
  else if (part <= 16) hot = room < 48 ? 0.5 : room < 70 ? 0.2 : 0.0;
  else if (part <= 32) hot = room < 48 ? 0.7 : room < 64 ? 0.4 : room < 100 ? 0.25 : room < 150 ? 0.15 : 0.0;
  else hot = room < 48 ? 0.7 : room < 64 ? 0.4 : 0.3;
  if (hot == 0.0) s.how = Scheduled::kAlways;
  s.route = {hot, 0.0, 1.0, -1.0, -1.0};
}

// The scheduled table kernel for this geometry in booking rounds of `part` trials, instead of the speculative launch
// in sc.args, with `beside` chains of other launches next to it.
//
// `room` is the number of neighbourhoods of a move's sites in the cell; about a third of it can run at once.
// Measured (800 K, ms; speculative form in the default or its best explicit width / here with 8 / 16 / 24 trials a
// tick; FP32 unless said):
//   swaps   78 columns: 1372 sites, room 4   4.07 / 4.92 / 5.83 / 7.10     4000, 12   5.93 / 4.44 / 4.90 / 6.17
//                       16384, 51            4.30 / 2.83 / 2.39 / 2.64     55296, 174 6.03 / 5.55 / 4.27 / 4.24
//           86 columns: 131072, 376         10.25 / 15.9 / 10.0 / 9.08
//           54 columns: 4000, 18             3.89 / 3.72 / 3.88 / 4.53     16384, 74  4.85 / 3.81 / 3.12 / 3.24
//           42 columns: 4000, 23             3.65 / 3.41 / 3.37 / 3.95     16384, 95  4.59 / 3.72 / 2.98 / 3.04
//           18 columns: 1000, 13             2.13 / 2.39 / 2.60            4000, 52   1.98 / 2.18 / 1.92 / 2.03
//   flips   78 columns: 4000, 50             3.53 / 3.56 / 2.97 (FP64 3.83 / 4.32 / 4.08)
//           54 columns: 4000, 72             1.94 / 2.28 / 1.75            16384, 297 1.72 / 2.64 / 1.84
//           42 columns: 4000, 93             1.46 / 1.95 / 1.42            16384, 381 1.58 / 2.57 / 1.77
//           18 columns: 1000, 52             0.96 / 1.22 / 1.05            3528, 185  1.24 / 1.77 / 1.25
// A flip's rows and draws are as cheap ahead in the speculative form, so flips gain only where the evaluation
// is long, and in FP64 the booking of their singlets (FP64 scans) takes what they gain.  A CTA pair's round of 32 flips
// beats one SM's ticks in large cells (55296 sites, 54 columns: 2.02 / 2.21).
//
// What a tick costs does not depend on what is accepted, but for trials that share a list slot, which run one after
// the other; see cemc_route.h.  Speculative time over time here by acceptance and by the atoms of the solutes
// (`share`: probability that two trials share a slot); three species, 78 columns, the lower one of the default shape
// and of 16 warps, which are CTA pairs unless said:
//   4000 sites, lists in shared memory    equal parts  0.33: 0.80   0.57: 1.01   0.73: 1.14   0.82: 1.20
//               two solutes, 256 and 64 atoms each (share 0.0036, 0.014), acceptance 0.85, 0.92: 1.08, 0.88
//   6912                                  equal parts  0.34: 0.91   0.57: 1.19   0.73: 1.33   0.82: 1.41
//   16384, lists in device memory         equal parts  0.37: 1.29   0.58: 1.46   0.73: 1.60   0.82: 1.66
//               one solute, 512, 256, 64, 4 atoms (share 0.0010, 0.0018, 0.0071, 0.11), acceptance 0.24: 1.05, 0.96,
//                                                     0.71, 0.37;  0.82: 2.10, 1.93, 1.55, 1.16
//               two solutes, 512, 64, 16 (share 0.0018, 0.014, 0.056), acceptance 0.54, 0.84, 0.95: 1.37, 1.26, 1.06
//   55296                                 equal parts  0.46: 1.12   0.61: 1.25   0.74: 1.37   0.82: 1.43
//               one solute, 512, 64, 16, 2 (share 0.0009, 0.0070, 0.028, 0.22), acceptance 0.33: 0.92, 0.72, 0.57,
//                                                     0.41;  0.82: 1.29, 1.18, 1.04, 0.98
//   16384, 86 columns, two species, hot, one solute of 256, 32, 2 (share 0.0040, 0.031, 0.50): pairs 2.02, 1.50, 1.47;
//               one CTA of 16 warps 1.28, 0.86, 0.80, of 8 warps 1.32, 0.78, 0.66
// Flips, one CTA of 16 warps / the default shape (pairs from 5324 sites): 78 columns 4000 sites 0.003: 0.71 / 0.72,
// 0.59: 1.01 / 1.04, 0.85: 1.15 / 1.14; 86 columns 6912 sites 0.07: 0.77 / 0.60, 0.67: 0.97 / 1.40, 0.84: 1.03 / 1.64;
// pairs of 16384 sites, 188 neighbourhoods, 0.67: 1.17, 0.84: 1.32; 55296 sites, conflict tables of one CTA in device
// memory, 0.24: 1.09 / 0.85, 0.85: 1.18 / 0.99.  Rounds of 8: 1.03 to 1.6, whatever is accepted.
// Chains on most SMs slow down the smallest swap cells' 8 trials a tick (4000 sites, 78 columns, rounds of 8:
// 2.42 / 2.37 with 64 chains, 2.49 / 2.76 with 152).
void fit_tick(const cemc_geometry *geo, int precision, int move, int part, int beside, Scheduled &sc) {
  const cemc::DevGeo &g = geo->g;
  cemc::RunArgs &s = sc.args;
  const bool swap = move == CEMC_MOVE_SWAP;
  const int room = g.n_movable / ((swap ? 4 : 1) * (g.n_cols + 1));
  const bool wide = g.n_cols >= 48;
  if (part > 32 || (swap ? room < (wide ? 10 : 40) : (precision != CEMC_PREC_F32 || !wide || room < 40))) return;
  if (swap && room < 16 && 2 * ((int64_t)s.n_chains + beside) > geo->n_sms) return;
  const bool always = !swap && s.cl == 1 && (s.gstamp || part <= 8);
  if (!swap && !always && room > (s.cl == 2 ? 200 : 128)) return;
  const bool far_lists = !s.trk_smem;
  s.part = part;
  s.warps = swap && room < 20 ? 8 : (swap && room >= 150 ? cemc::kTickCap : cemc::kTickWarps);
  int exact = 5;
  while ((1 << exact) < g.n_sites) ++exact;
  for (; s.fx_low >= 0 && !sc.how; --s.fx_low)
    for (int rb = 7; rb >= 6 && !sc.how; --rb)
      for (int hb = std::min(exact, 14); hb >= std::min(exact, 11) && !sc.how; --hb) {
        s.row_bits = rb;
        s.head_bits = hb;
        sc.smem = cemc::tick_layout(g, swap, precision == CEMC_PREC_F32 ? 4 : 8, rb, hb).total +
                  (s.fx_low ? cemc::fx_low_bytes(g) : 0);
        if (sc.smem <= (size_t)geo->max_smem) sc.how = always ? Scheduled::kAlways : Scheduled::kRouted;
      }
  ++s.fx_low;  // as it was when the shape was found
  if (!swap) sc.route = {s.cl == 2 ? 0.6 : 0.8, 0.0, 1.0, -1.0, -1.0};
  else if (far_lists && s.cl == 2) sc.route = {0.7, room < 100 ? 1e9 : 0.06, 0.5, 0.008, 0.0008};
  else if (far_lists) sc.route = {0.7, 0.01, 0.5, 0.004, 0.0008};
  else sc.route = {0.6, 0.005, 1.0, -1.0, -1.0};
}

}  // namespace

// The choice between kernels that a call leaves to the device: taken in the call, alone, or taken before it.
enum class Decision { kHere, kOnly, kBefore };

static int run(const cemc_geometry *geo, cemc_run_desc *r, void *stream, Decision decision) {
  if (!geo || !r) return fail(CEMC_ERR_ARG, "null geometry or run descriptor");
  const cemc::DevGeo &g = geo->g;
  if (r->n_chains <= 0) return fail(CEMC_ERR_ARG, "no chains");
  if (r->move != CEMC_MOVE_FLIP && r->move != CEMC_MOVE_SWAP) return fail(CEMC_ERR_ARG, "unknown move type");
  if (r->precision != CEMC_PREC_F32 && r->precision != CEMC_PREC_F64) return fail(CEMC_ERR_ARG, "unknown precision");
  if (!r->occ || !r->cf || !r->energy || !r->eci || !r->kT || !r->trial)
    return fail(CEMC_ERR_ARG, "null chain state pointer");
  if (r->move == CEMC_MOVE_SWAP && (!r->trk || !r->loc || !r->trk_start || !r->trk_count))
    return fail(CEMC_ERR_ARG, "swap moves need the per-species site lists");
  if ((r->trace_site || r->trace_acc || r->trace_de) && !(r->trace_site && r->trace_acc && r->trace_de))
    return fail(CEMC_ERR_ARG, "trace buffers must be given together");
  if (r->n_chains > 65535 * 32) return fail(CEMC_ERR_LIMIT, "too many chains in one launch");
  r->kernel_used = CEMC_KERNEL_AUTO;  // nothing launched yet
  r->scheduled = 0;
  if (r->n_trials == 0) return CEMC_OK;
  if (r->kernel < CEMC_KERNEL_AUTO || r->kernel > CEMC_KERNEL_SPIN_QUARTER)
    return fail(CEMC_ERR_ARG, "unknown kernel %d", (int)r->kernel);
  if (r->cluster < 0 || r->cluster > 2) return fail(CEMC_ERR_ARG, "cluster must be 0 (auto), 1 or 2");
  // waste recycling runs its own build of the generic form, one CTA per chain
  const bool recycle = r->recycle_waste != 0;
  if (recycle && r->kernel != CEMC_KERNEL_AUTO && r->kernel != CEMC_KERNEL_GENERIC)
    return fail(CEMC_ERR_ARG, "waste recycling runs the generic kernel form");
  if (recycle && r->cluster == 2) return fail(CEMC_ERR_ARG, "waste recycling runs one CTA per chain");
  if ((r->site_allow || r->frozen || r->accept_first) && r->cluster == 2)
    return fail(CEMC_ERR_ARG, "move constraints and first-move acceptance run one CTA per chain");
  const bool want_spin = r->kernel == CEMC_KERNEL_SPIN || r->kernel == CEMC_KERNEL_SPIN_HALFWARP ||
                         r->kernel == CEMC_KERNEL_SPIN_QUARTER;
  if (want_spin && !geo->spin_ok)
    return fail(CEMC_ERR_ARG, "the spin-basis kernel needs two species with basis values +1/-1, <= 64 columns and "
                              "one translation-symmetry group");
  const bool use_spin = want_spin || (r->kernel == CEMC_KERNEL_AUTO && geo->spin_ok && !recycle);
  if (r->kernel == CEMC_KERNEL_TABLE && !g.table_ok)
    return fail(CEMC_ERR_LIMIT, "the table kernel needs translation groups of equal size and pattern tables of at "
                                "most %d entries", cemc::kMaxTable);
  // move constraints are checked (and redrawn) by the one-trial-per-warp forms
  const bool constrained = r->site_allow != nullptr || r->frozen != nullptr || r->accept_first != 0 || recycle;
  if (r->max_attempts < 0) return fail(CEMC_ERR_ARG, "max_attempts must be >= 0");
  const bool half_ok = use_spin && geo->spin.half_ok && r->move == CEMC_MOVE_FLIP && !constrained;
  if (r->kernel == CEMC_KERNEL_SPIN_QUARTER &&
      !(use_spin && geo->spin.qtr_ok && r->move == CEMC_MOVE_FLIP && !constrained && r->cluster != 2))
    return fail(CEMC_ERR_ARG, "the quarter-warp spin kernel runs unconstrained single-site flips with at most 8 "
                              "cluster ECIs, one CTA per chain");
  if (r->kernel == CEMC_KERNEL_SPIN_HALFWARP && !half_ok)
    return fail(CEMC_ERR_ARG, "the half-warp spin kernel runs unconstrained single-site flips with at most 16 "
                              "cluster ECIs");
  // Local-field form: unconstrained single-site flips of a geometry with field tables, one CTA
  // per chain, when asked for (its state fits in shared memory, with the conflict table in the
  // caller's stamp buffer when it does not fit beside the counts).
  const bool field_possible = geo->field_ok && r->move == CEMC_MOVE_FLIP && !constrained && r->cluster != 2;
  if (r->kernel == CEMC_KERNEL_FIELD && !field_possible)
    return fail(CEMC_ERR_ARG, "the local-field kernel runs unconstrained single-site flips of a periodic binary "
                              "+1/-1 geometry of one translation group without background sites, one CTA per chain");
  if (field_possible && r->kernel == CEMC_KERNEL_FIELD) {
    const cemc::FieldDev &fd = geo->field;
    cemc::RunArgs fa{};
    fa.n_chains = r->n_chains;
    fa.warps = r->warps > 0 ? std::min(r->warps, cemc::kFieldMaxWarps) : 16;
    fa.cl = 1;
    fa.tpw = 1;
    fa.ring_bits = cemc::field_ring_bits(cemc::field_round(fa.warps));
    fa.occ_smem = 1;
    int bits = 5;
    while ((1 << bits) < g.n_sites) ++bits;
    fa.stamp_bits = bits;
    const int rs = r->precision == CEMC_PREC_F32 ? 4 : 8;
    size_t smem = cemc::field_layout(g, fd.n_cl, fd.pw, fd.n_cnt, fd.n_upd, rs, fa.ring_bits, false).total;
    if (smem > (size_t)geo->max_smem && r->stamps && r->stamp_words >= cemc_stamp_words(geo, r->n_chains)) {
      fa.gstamp = r->stamps;
      smem = cemc::field_layout(g, fd.n_cl, fd.pw, fd.n_cnt, fd.n_upd, rs, fa.ring_bits, true).total;
    }
    if (smem <= (size_t)geo->max_smem) {
      if (decision == Decision::kOnly) return CEMC_OK;
      fa.seed = r->seed;
      fa.occ = r->occ;
      fa.cf = r->cf;
      fa.energy = r->energy;
      fa.eci = r->eci;
      fa.kT = r->kT;
      fa.trial = r->trial;
      fa.accum = r->accum;
      fa.trace_site = r->trace_site;
      fa.trace_acc = r->trace_acc;
      fa.trace_de = r->trace_de;
      fa.status = r->status;
      fa.chain_key = r->chain_key;
      fa.accum_slot = r->accum_slot;
      fa.chain_trials = r->chain_trials;
      const uint64_t max_chunk = (uint64_t)1 << 25;  // round numbers fit the 26 upper bits of a stamp
      if (r->n_trials > max_chunk && r->trace_acc)
        return fail(CEMC_ERR_LIMIT, "traced runs are limited to %llu trials per call", (unsigned long long)max_chunk);
      for (uint64_t done = 0; done < r->n_trials;) {
        const uint64_t n = std::min(max_chunk, r->n_trials - done);
        fa.n_trials = n;
        fa.chunk_offset = done;
        cudaError_t e = cemc::launch_field(g, fa, fd, r->precision, smem, static_cast<cudaStream_t>(stream));
        if (e != cudaSuccess) return cuda_fail(e, "local-field Monte Carlo kernel launch");
        done += n;
      }
      r->kernel_used = CEMC_KERNEL_FIELD;
      return CEMC_OK;
    }
    if (r->kernel == CEMC_KERNEL_FIELD)
      return fail(CEMC_ERR_LIMIT, "the local-field kernel needs %zu bytes of shared memory (limit %d); pass a stamp "
                                  "buffer or use another kernel", smem, geo->max_smem);
  }
  // two trials per warp: asked for, or chosen when eligible and no CTA pair was asked for
  // (a CTA pair takes the half-warp form only when that form is asked for explicitly)
  int tpw = r->kernel == CEMC_KERNEL_SPIN_QUARTER ? 4 :
                  (r->kernel == CEMC_KERNEL_SPIN_HALFWARP || (r->kernel == CEMC_KERNEL_AUTO && half_ok &&
                                                                r->cluster != 2)) ? 2 : 1;
  // Default round width: 16 evaluating warps, fewer where most trials of a
  // round would conflict.  A changed site reaches about n_cols sites, so with
  // n_movable / (2 n_cols sites-per-move) trials a round about half the round
  // commits (a 2048-site swap chain: 9 trials, about 4 commits a round); a
  // wider round only adds latency.  The same cap decides whether a chain may
  // take a CTA pair (twice the trials per round) when none is asked for.
  int warps = r->warps;
  int round_cap = 0;  // 0: the caller chose the width
  if (warps <= 0) {
    const int per_move = r->move == CEMC_MOVE_SWAP ? 2 : 1;
    round_cap = std::max(4, g.n_movable / (2 * g.n_cols * per_move));
    warps = std::max(2, std::min(16, round_cap / tpw));
  }
  // The automatic choice takes the quarter-warp form for a round of the same width where half the warps cost
  // less than their longer evaluation (one chain of 256 sites, half / quarter, ms: FP32 8 trials 1.58 / 1.59,
  // 16 0.90 / 0.88, 32 0.59 / 0.53; FP64 4 trials 3.25 / 3.23, 8 1.74 / 1.67, 16 1.02 / 0.91, 32 0.69 / 0.56).
  if (r->kernel == CEMC_KERNEL_AUTO && tpw == 2 && geo->spin.qtr_ok) {
    const int trials = 2 * std::min(warps, cemc::max_eval_warps(1, 2));
    if (trials % 4 == 0 && trials >= (r->precision == CEMC_PREC_F32 ? 16 : 8)) {
      tpw = 4;
      warps = trials / 4;
    }
  }
  const int rsize = r->precision == CEMC_PREC_F32 ? 4 : 8;
  cemc::RunArgs a{};
  a.n_chains = r->n_chains;
  a.warps = warps;
  a.seed = r->seed;
  a.occ = r->occ;
  a.cf = r->cf;
  a.energy = r->energy;
  a.eci = r->eci;
  a.kT = r->kT;
  a.trial = r->trial;
  a.accum = r->accum;
  a.trk = r->trk;
  a.loc = r->loc;
  a.trk_start = r->trk_start;
  a.trk_count = r->trk_count;
  a.trace_site = r->trace_site;
  a.trace_acc = r->trace_acc;
  a.trace_de = r->trace_de;
  a.status = r->status;
  a.chain_key = r->chain_key;
  a.accum_slot = r->accum_slot;
  a.chain_trials = r->chain_trials;
  a.site_allow = r->site_allow;
  a.frozen = r->frozen;
  a.max_attempts = r->max_attempts > 0 ? r->max_attempts : 10000;
  a.accept_first = r->accept_first != 0;
  a.cons = constrained ? 1 : 0;
  a.tpw = tpw;
  const int n_cl = use_spin ? geo->spin.n_cl : 0, n_masks = use_spin ? geo->spin.n_masks : 0;
  // Evaluation forms to try, in order: spin, or table then generic (AUTO), or the one asked for.
  std::vector<int> forms;
  if (recycle)
    forms = {cemc::kFormRecycle};
  else if (use_spin)
    forms = {cemc::kFormSpin};
  else if (r->kernel == CEMC_KERNEL_TABLE && r->n_chains > 65535)
    return fail(CEMC_ERR_LIMIT, "the table kernel ends with a recompute of at most 65535 chains per call");
  else if (r->kernel == CEMC_KERNEL_TABLE)
    forms = {cemc::kFormTable};
  else if (r->kernel == CEMC_KERNEL_GENERIC)
    forms = {cemc::kFormGeneric};
  else if (g.table_ok && r->n_chains <= 65535)
    forms = {cemc::kFormTable, cemc::kFormGeneric};
  else
    forms = {cemc::kFormGeneric};
  // Shared memory: the occupation, then (swaps) the site lists, then exact
  // stamp tables (one entry per site) are preferred; fall back in that order.
  const size_t budget = (size_t)geo->max_smem;
  int exact_bits = 0;
  while ((1 << exact_bits) < g.n_sites) ++exact_bits;
  if (exact_bits < 5) exact_bits = 5;
  const int is_swap = r->move == CEMC_MOVE_SWAP;
  struct Choice {
    int occ, trk, min_bits, global;
  };
  // exact tables in a caller buffer come before hashed shared-memory ones (hashing only costs speed)
  const bool gbuf = r->stamps && r->stamp_words >= cemc_stamp_words(geo, r->n_chains);
  std::vector<Choice> choices = {{1, is_swap, exact_bits, 0}, {1, 0, exact_bits, 0}};
  if (gbuf) choices.insert(choices.end(), {{1, is_swap, exact_bits, 1}, {1, 0, exact_bits, 1}});
  choices.insert(choices.end(), {{1, 0, 12, 0}, {0, 0, 12, 0}});
  if (gbuf) choices.push_back({0, 0, exact_bits, 1});
  choices.push_back({0, 0, 5, 0});
  int form = forms[0];
  auto fit = [&](int cl, cemc::McLayout &L, cemc::RunArgs &x) {
    const int w = std::min(warps, cemc::max_eval_warps(cl, tpw));
    const int rb = cemc::ring_bits_for(cemc::round_trials(cl, w, tpw));
    for (const Choice &ch : choices) {
      for (int bits = exact_bits; bits >= std::min(ch.min_bits, exact_bits); --bits) {
        L = cemc::mc_layout(g, w, r->move, rsize, ch.occ, ch.trk, bits, n_cl, n_masks, rb, form, tpw, ch.global);
        if (L.total <= budget) {
          x.occ_smem = ch.occ;
          x.trk_smem = ch.trk;
          x.stamp_bits = bits;
          x.gstamp = ch.global ? r->stamps : nullptr;
          x.ring_bits = rb;
          x.cl = cl;
          x.warps = w;
          return true;
        }
      }
    }
    return false;
  };
  // Resident cluster pairs of this configuration (cached per geometry).
  auto resident_pairs = [&](const cemc::McLayout &L, const cemc::RunArgs &x) {
    const auto key = std::make_tuple(x.warps, (int)r->move, (int)r->precision, form, L.total);
    std::lock_guard<std::mutex> lock(geo->mu);
    auto it = geo->pairs.find(key);
    if (it != geo->pairs.end()) return it->second;
    const int n = cemc::max_active_clusters(g, x, r->move, r->precision, L.total, form);
    geo->pairs[key] = n;
    return n;
  };
  cemc::McLayout L{};
  bool found = false;
  for (size_t fi = 0; fi < forms.size() && !found; ++fi) {
    form = forms[fi];
    if (r->cluster == 2 || (tpw == 1 && r->cluster == 0 && !constrained && 2 * r->n_chains <= geo->n_sms &&
                            (round_cap == 0 || round_cap >= 2 * warps))) {
      cemc::RunArgs x = a;
      cemc::McLayout L2{};
      if (fit(2, L2, x)) {
        const int n = resident_pairs(L2, x);
        if (r->cluster == 2 && n < 1) return fail(CEMC_ERR_LIMIT, "no CTA pair of this size fits on the device");
        if (r->cluster == 2 || n >= r->n_chains) {
          a = x;
          L = L2;
          found = true;
        }
      } else if (r->cluster == 2 && fi + 1 == forms.size()) {
        return fail(CEMC_ERR_LIMIT, "shared memory of a CTA pair exceeds %zu bytes; use fewer warps", budget);
      }
    }
    if (!found && r->cluster != 2) found = fit(1, L, a);
  }
  if (!found) return fail(CEMC_ERR_LIMIT, "shared memory exceeds %zu bytes; use fewer warps", budget);
  // Scheduled kernels.  They book in the rounds this launch shape would have had with exact conflict tables, so a
  // shape that would hash them stays.
  // FP64 table entries in fixed point where there is room for their low parts, in both kernels or in none.
  if (form == cemc::kFormTable && r->precision == CEMC_PREC_F64) a.fx_low = L.total + cemc::fx_low_bytes(g) <= budget;
  Scheduled sch;
  sch.args = a;
  const bool exact = a.gstamp || a.stamp_bits == exact_bits;
  const int beside = std::max(0, r->beside);
  const bool flips = form == cemc::kFormSpin && r->move == CEMC_MOVE_FLIP;  // else the table form's moves
  if (flips && geo->spin.qtr_ok && g.table16 && !constrained && exact && r->cluster != 2 &&
      (r->kernel == CEMC_KERNEL_AUTO || r->kernel == CEMC_KERNEL_SPIN_QUARTER))
    fit_sched(geo, r->precision, cemc::round_trials(1, a.warps, a.tpw), L.total, beside, sch);
  else if (form == cemc::kFormTable && !constrained && exact)
    fit_tick(geo, r->precision, r->move, cemc::round_trials(a.cl, a.warps, a.tpw), beside, sch);
  if (sch.how == Scheduled::kRouted && (!r->status || r->n_trials < cemc::kRouteTrials)) sch.how = Scheduled::kNo;
  // The table form leaves correlation functions to a full recompute at the end of the call.
  double *rscratch = nullptr;
  if (form == cemc::kFormTable) {
    const size_t need = cemc::recompute_blocks(g) * (size_t)r->n_chains * (size_t)g.n_eci;
    if (r->scratch && r->scratch_doubles < need)
      return fail(CEMC_ERR_ARG, "the table kernel's final recompute needs a scratch buffer of %zu doubles, the run "
                                "descriptor gives %llu", need, (unsigned long long)r->scratch_doubles);
    if (r->scratch) {
      rscratch = r->scratch;
    } else if (need <= cemc::kNoAllocScratchDoubles) {
      cudaError_t err = cudaSuccess;
      rscratch = cemc::noalloc_scratch(&err);
      if (!rscratch) return cuda_fail(err, "cudaGetSymbolAddress(recompute scratch)");
    } else {
      return fail(CEMC_ERR_LIMIT, "the table kernel needs a recompute scratch of %zu doubles (run desc scratch)", need);
    }
  }
  // Rounds are numbered in the upper 26 bits of the stamp marks: split very long runs.
  const uint64_t max_chunk = (uint64_t)1 << 25;
  if (r->n_trials > max_chunk && r->trace_acc)
    return fail(CEMC_ERR_LIMIT, "traced runs are limited to %llu trials per call", (unsigned long long)max_chunk);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (sch.how) a.fx_low = sch.args.fx_low;
  const size_t mc_smem = L.total + (a.fx_low ? cemc::fx_low_bytes(g) : 0);
  if (sch.how == Scheduled::kRouted) {
    sch.args.route = cemc::kRouteScheduled;
    a.route = cemc::kRouteSpeculative;
  }
  for (uint64_t done = 0; done < r->n_trials;) {
    const uint64_t n = std::min(max_chunk, r->n_trials - done);
    a.n_trials = sch.args.n_trials = n;
    a.chunk_offset = sch.args.chunk_offset = done;
    cudaError_t e;
    if (sch.how == Scheduled::kRouted && (decision != Decision::kBefore || done > 0)) {
      e = cemc::launch_route(g, a, is_swap, sch.route, st);
      if (e != cudaSuccess) return cuda_fail(e, "route kernel launch");
    }
    if (decision == Decision::kOnly) return CEMC_OK;
    if (sch.how) {
      e = flips ? cemc::launch_sched(g, sch.args, r->precision, sch.smem, st, geo->spin)
                : cemc::launch_tick(g, sch.args, r->move, r->precision, sch.smem, st);
      if (e != cudaSuccess) return cuda_fail(e, "scheduled Monte Carlo kernel launch");
    }
    if (sch.how != Scheduled::kAlways) {
      e = cemc::launch_mc(g, a, r->move, r->precision, mc_smem, st, form, use_spin ? &geo->spin : nullptr);
      if (e != cudaSuccess) return cuda_fail(e, "Monte Carlo kernel launch");
    }
    done += n;
    if (form == cemc::kFormTable) {  // after every launch: the next one's sums start from cf and energy
      e = recompute(geo, r->n_chains, r->occ, r->eci, r->cf, r->energy, rscratch, stream);
      if (e != cudaSuccess) return cuda_fail(e, "recompute after the table kernel");
    }
  }
  r->scheduled = sch.how == Scheduled::kAlways ? 1 : sch.how == Scheduled::kRouted ? 2 : 0;
  r->kernel_used = form == cemc::kFormTable ? CEMC_KERNEL_TABLE
                  : (form == cemc::kFormGeneric || form == cemc::kFormRecycle) ? CEMC_KERNEL_GENERIC
                  : (a.tpw == 4 || sch.how == Scheduled::kAlways ? CEMC_KERNEL_SPIN_QUARTER : a.tpw == 2 ? CEMC_KERNEL_SPIN_HALFWARP : CEMC_KERNEL_SPIN);
  return CEMC_OK;
}

extern "C" int cemc_run(const cemc_geometry *geo, cemc_run_desc *r, void *stream) {
  return run(geo, r, stream, Decision::kHere);
}

extern "C" int cemc_decide(const cemc_geometry *geo, cemc_run_desc *r, void *stream) {
  return run(geo, r, stream, Decision::kOnly);
}

extern "C" int cemc_run_decided(const cemc_geometry *geo, cemc_run_desc *r, void *stream) {
  return run(geo, r, stream, Decision::kBefore);
}

extern "C" size_t cemc_recompute_scratch_doubles(const cemc_geometry *geo, int32_t n_chains) {
  if (!geo || n_chains <= 0) return 0;
  return cemc::recompute_blocks(geo->g) * (size_t)n_chains * (size_t)geo->g.n_eci;
}

extern "C" int cemc_recompute(const cemc_geometry *geo, int32_t n_chains, const int8_t *occ, const double *eci,
                              double *cf, double *energy, double *scratch, void *stream) {
  if (!geo || n_chains <= 0 || !occ || !eci || !cf || !energy || !scratch)
    return fail(CEMC_ERR_ARG, "bad recompute arguments");
  if (n_chains > 65535) return fail(CEMC_ERR_LIMIT, "too many chains in one recompute");
  cudaError_t e = recompute(geo, n_chains, occ, eci, cf, energy, scratch, stream);
  if (e != cudaSuccess) return cuda_fail(e, "recompute kernel launch");
  return CEMC_OK;
}

extern "C" int cemc_recompute_noalloc(const cemc_geometry *geo, int32_t n_chains, const int8_t *occ,
                                      const double *eci, double *cf, double *energy, void *stream) {
  if (!geo || n_chains <= 0 || !occ || !eci || !cf || !energy)
    return fail(CEMC_ERR_ARG, "bad recompute_noalloc arguments");
  if (n_chains > 65535) return fail(CEMC_ERR_LIMIT, "too many chains in one recompute");
  const size_t need = cemc::recompute_blocks(geo->g) * (size_t)n_chains * (size_t)geo->g.n_eci;
  if (need > cemc::kNoAllocScratchDoubles)
    return fail(CEMC_ERR_LIMIT,
                "recompute_noalloc needs %zu scratch doubles but its fixed array holds %zu "
                "(reduce n_chains or call cemc_recompute with a caller buffer)",
                need, cemc::kNoAllocScratchDoubles);
  cudaError_t err = cudaSuccess;
  double *scratch = cemc::noalloc_scratch(&err);
  if (!scratch) return cuda_fail(err, "cudaGetSymbolAddress(recompute_noalloc scratch)");
  // Each scratch entry the second kernel reads is written by the first kernel
  // of the same call, so nothing has to be cleared between calls.
  cudaError_t e = recompute(geo, n_chains, occ, eci, cf, energy, scratch, stream);
  if (e != cudaSuccess) return cuda_fail(e, "recompute_noalloc kernel launch");
  return CEMC_OK;
}

extern "C" int cemc_energy(const cemc_geometry *geo, int32_t n_chains, const double *eci, const double *cf,
                           double *energy, void *stream) {
  if (!geo || n_chains <= 0 || !eci || !cf || !energy) return fail(CEMC_ERR_ARG, "bad energy arguments");
  cudaError_t e = cemc::launch_energy(geo->g, n_chains, eci, cf, energy, static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return cuda_fail(e, "energy kernel launch");
  return CEMC_OK;
}

extern "C" int cemc_apply_changes(const cemc_geometry *geo, int8_t *occ, double *cf, double *energy,
                                  const double *eci, int32_t n_changes, const int32_t *sites, const int8_t *old_sym,
                                  const int8_t *new_sym, int32_t *status, void *stream) {
  if (!geo || !occ || !cf || !energy || !eci || n_changes < 0 || (n_changes > 0 && (!sites || !old_sym || !new_sym)))
    return fail(CEMC_ERR_ARG, "bad apply_changes arguments");
  if (cemc::warp_kernel_smem(geo->g) > (size_t)geo->max_smem) return fail(CEMC_ERR_LIMIT, "tables too large");
  cudaError_t e = cemc::launch_apply(geo->g, occ, cf, energy, eci, n_changes, sites, old_sym, new_sym, status,
                                     static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return cuda_fail(e, "apply_changes kernel launch");
  return CEMC_OK;
}

extern "C" int cemc_calculate(const cemc_geometry *geo, int8_t *occ, double *cf, double *energy, const double *eci,
                              int32_t n_changes, const int32_t *sites, const int8_t *old_sym, const int8_t *new_sym,
                              double *out, void *stream) {
  if (!geo || !occ || !cf || !energy || !eci || !out || n_changes < 0 || n_changes > CEMC_CALC_CHANGES ||
      (n_changes > 0 && (!sites || !old_sym || !new_sym)))
    return fail(CEMC_ERR_ARG, "bad calculate arguments");
  const cemc::DevGeo &g = geo->g;
  if (cemc::warp_kernel_smem(g) > (size_t)geo->max_smem) return fail(CEMC_ERR_LIMIT, "tables too large");
  cemc::ChangeArgs ch{};
  ch.n = n_changes;
  for (int i = 0; i < n_changes; ++i) {
    if (sites[i] < 0 || sites[i] >= g.n_sites) return fail(CEMC_ERR_ARG, "site out of range");
    if (new_sym[i] < 0 || new_sym[i] >= g.n_sym) return fail(CEMC_ERR_ARG, "bad species");
    ch.site[i] = sites[i];
    ch.old_sym[i] = old_sym[i];
    ch.new_sym[i] = new_sym[i];
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e = cemc::launch_calculate(g, occ, cf, energy, eci, ch, out, st);
  if (e != cudaSuccess) return cuda_fail(e, "calculate kernel launch");
  e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return cuda_fail(e, "calculate");
  return CEMC_OK;
}

extern "C" int cemc_revert(const cemc_geometry *geo, int8_t *occ, double *cf, double *energy, const double *snap_cf,
                           const double *snap_energy, int32_t n_sites, const int32_t *sites, const int8_t *sym,
                           void *stream) {
  if (!geo || !occ || !cf || !energy || !snap_cf || !snap_energy || n_sites < 0 || n_sites > CEMC_CALC_CHANGES ||
      (n_sites > 0 && (!sites || !sym)))
    return fail(CEMC_ERR_ARG, "bad revert arguments");
  const cemc::DevGeo &g = geo->g;
  cemc::ChangeArgs ch{};
  ch.n = n_sites;
  for (int i = 0; i < n_sites; ++i) {
    if (sites[i] < 0 || sites[i] >= g.n_sites) return fail(CEMC_ERR_ARG, "site out of range");
    ch.site[i] = sites[i];
    ch.new_sym[i] = sym[i];
  }
  cudaError_t e = cemc::launch_revert(g.n_eci, occ, cf, energy, snap_cf, snap_energy, ch,
                                      static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return cuda_fail(e, "revert kernel launch");
  return CEMC_OK;
}

extern "C" int cemc_read(double *dst, const double *src, size_t count, void *stream) {
  if (count > 0 && (!dst || !src)) return fail(CEMC_ERR_ARG, "bad read arguments");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemcpyAsync(dst, src, 8 * count, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return cuda_fail(e, "read");
  return CEMC_OK;
}

extern "C" int cemc_delta_e(const cemc_geometry *geo, const int8_t *occ, const double *eci, int32_t move,
                            int32_t site_a, int32_t site_b, int32_t new_a, double *de_out, double *dcf_out,
                            void *stream) {
  if (!geo || !occ || !eci || !de_out || !dcf_out) return fail(CEMC_ERR_ARG, "bad delta_e arguments");
  const cemc::DevGeo &g = geo->g;
  if (site_a < 0 || site_a >= g.n_sites) return fail(CEMC_ERR_ARG, "site out of range");
  if (move == CEMC_MOVE_SWAP && (site_b < 0 || site_b >= g.n_sites || site_b == site_a))
    return fail(CEMC_ERR_ARG, "bad swap partner");
  if (move == CEMC_MOVE_FLIP && (new_a < 0 || new_a >= g.n_sym)) return fail(CEMC_ERR_ARG, "bad species");
  cudaError_t e = cemc::launch_delta(g, occ, eci, move, site_a, site_b, new_a, de_out, dcf_out,
                                     static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return cuda_fail(e, "delta_e kernel launch");
  return CEMC_OK;
}

extern "C" int cemc_pt_exchange(int32_t n_replicas, int32_t direction, uint64_t seed, uint64_t round,
                                const double *energy, double *kT, int32_t *replica_of, int32_t *position_of,
                                int32_t *n_accept, void *stream) {
  if (n_replicas < 1 || !energy || !kT || !replica_of || (direction != 0 && direction != 1))
    return fail(CEMC_ERR_ARG, "bad replica-exchange arguments");
  cudaError_t e = cemc::launch_pt(n_replicas, direction, seed, round, energy, kT, replica_of, position_of, n_accept,
                                  static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return cuda_fail(e, "replica-exchange kernel launch");
  return CEMC_OK;
}
