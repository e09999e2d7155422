// Full correlation-function recompute of a periodic box of cells (ce_calculator.py:169-177, CLEASE's
// CorrFunction; DevGeo::box_L) by bit planes.
//
// Sites are numbered ((x L + y) L + z) nb + b, so for each species and basis site b a row (x, y) is one
// word of L bits, bit z = cell z.  A neighbour at cell offset (dx, dy, dz) and basis site b' of all L sites
// of a row is row (x + dx, y + dy) of plane b' rotated by dz: one shared-memory load and one funnel shift
// serve L sites.  A product of +1/-1 spins is the parity of its members' bits (XOR, population count); other
// bases count, per pattern of clusters, how often each tuple of species occurs (AND, population count), and
// the ECIs' sums are dot products of those integers with precomputed basis products.  Clusters that are
// lattice translations of one another are evaluated once (BoxCf).
//
// A chain is one thread-block cluster of 1..8 CTAs, each with a slab of x rows (and the halo its offsets
// reach) in shared memory; the counters are added up in the first CTA, which writes the correlation
// functions and the energy.  All sums over sites are integers, so the result does not depend on the split.
//
// Bound: instruction issue (+1/-1: about 12 instructions per row and cluster member) and, for species
// tuples, the population count's quarter rate; for a few chains, the latency of one CTA's stages.
// 48 chains x 131072 sites, binary, 86 columns: 960 us by recompute_partial (cemc_cf.cu), 52 us here (121
// GB/s of occupations; their 6.3 MB alone take 1 us).  32 x 13500, ternary, 3416 terms: 11,050 us (FP64
// products) and 78 us; one binary cell of 256 sites 9 us.  recompute_partial, which stages a byte per site and
// column and multiplies term by term, stays for cells that are no such box.
#include <cuda_runtime.h>

#include <type_traits>

#include "cemc_boxcf.h"
#include "cemc_launch.h"

namespace cemc {

namespace {

constexpr int kBoxThreads = 512;

struct BoxLayout {
  size_t ent, ent_start, job, rows, counts, cf, eci, planes, total;
};
__host__ __device__ inline BoxLayout box_layout(const DevGeo &g, const BoxCf &c, int ctas, int slab) {
  BoxLayout L;
  size_t o = 0;
  L.ent = o;
  o = align16(o + 16 * (size_t)c.n_ents);
  L.ent_start = o;
  o = align16(o + 4 * ((size_t)c.n_jobs * g.box_nb + 1));
  L.job = o;
  o = align16(o + 8 * (size_t)c.n_jobs);
  L.rows = o;  // basis site, x in the slab and y of the CTA's rows
  o = align16(o + 4 * (size_t)((g.box_L + ctas - 1) / ctas) * g.box_L * g.box_nb);
  L.counts = o;
  o = align16(o + 4 * (size_t)c.n_counts + 4 * (size_t)g.n_sym);  // pattern counters, then sites per species
  L.cf = o;
  o = align16(o + 8 * (size_t)g.n_eci);
  L.eci = o;
  o = align16(o + 8 * (size_t)g.n_eci);
  L.planes = o;
  o = align16(o + 8 * (size_t)(c.pm1 ? 1 : g.n_sym - 1) * g.box_nb * slab * g.box_L);
  L.total = o;
  return L;
}
// x rows a CTA holds: its own and the halo, or all of them.
__host__ __device__ inline int box_slab(int L, int ctas, int hx) {
  const int nx = (L + ctas - 1) / ctas;
  return nx + 2 * hx >= L ? L : nx + 2 * hx;
}

__device__ __forceinline__ unsigned box_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ void box_cluster_barrier() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

}  // namespace

// S: 0 for a +1/-1 basis (parities), else the number of species.  WIDE: rows of 33..64 bits.
template <int S, bool WIDE>
__global__ void __launch_bounds__(kBoxThreads) boxcf_kernel(DevGeo g, BoxCf c, int ctas, const int8_t *occ_all,
                                                            const double *eci, double *cf, double *energy) {
  extern __shared__ __align__(16) unsigned char smem[];
  using Word = typename std::conditional<WIDE, uint64_t, uint32_t>::type;
  constexpr int NP = S == 0 ? 1 : S - 1;  // planes: the -1 species, or species 1 .. S - 1
  const int L = g.box_L, nb = g.box_nb, N = g.n_sites, tid = threadIdx.x, lane = tid & 31;
  const int rank = ctas > 1 ? (int)box_rank() : 0, chain = blockIdx.x / ctas;
  const int per = (L + ctas - 1) / ctas, x0 = rank * per, nx = max(0, min(L - x0, per));
  const int slab = box_slab(L, ctas, c.hx);
  const bool whole = slab == L;
  const int xs = whole ? 0 : x0 - c.hx;  // the slab's first x
  const BoxLayout lay = box_layout(g, c, ctas, slab);
  uint32_t *counts = reinterpret_cast<uint32_t *>(smem + lay.counts);
  uint32_t *species = counts + c.n_counts;
  double *cf_s = reinterpret_cast<double *>(smem + lay.cf);
  uint64_t *planes = reinterpret_cast<uint64_t *>(smem + lay.planes);  // [NP][nb][slab][L]
  const int8_t *occ = occ_all + (size_t)chain * N;

  int4 *ent = reinterpret_cast<int4 *>(smem + lay.ent);
  int32_t *ent_start = reinterpret_cast<int32_t *>(smem + lay.ent_start);
  int2 *jobs = reinterpret_cast<int2 *>(smem + lay.job);
  uint32_t *rowinfo = reinterpret_cast<uint32_t *>(smem + lay.rows);
  double *eci_s = reinterpret_cast<double *>(smem + lay.eci);
  const int rows = nx * L * nb, pstride = nb * slab * L;
  for (int i = tid; i < c.n_counts + g.n_sym; i += blockDim.x) counts[i] = 0u;
  for (int i = tid; i < c.n_ents; i += blockDim.x) ent[i] = c.ent[i];
  for (int i = tid; i <= c.n_jobs * nb; i += blockDim.x) ent_start[i] = c.ent_start[i];
  for (int i = tid; i < c.n_jobs; i += blockDim.x) jobs[i] = c.job[i];
  for (int i = tid; i < g.n_eci; i += blockDim.x) eci_s[i] = eci[(size_t)chain * g.n_eci + i];
  for (int i = tid; i < rows; i += blockDim.x) {
    const int b = i / (nx * L), r = i - b * nx * L;
    rowinfo[i] = (uint32_t)(r % L) | ((uint32_t)(r / L + (x0 - xs)) << 8) | ((uint32_t)b << 16);
  }
  // planes: one warp per (x, y) row, lane = z; rows of up to 32 bits are stored twice over, so that a
  // rotation is one funnel shift.  Four rows' sites are loaded before the first is packed.
  const bool quads = nb == 4 && (reinterpret_cast<uintptr_t>(occ) & 3) == 0;
  const int nw = blockDim.x >> 5;
  auto put_plane = [&](int b, int q, const uint64_t(&w)[NP]) {
    if (lane < NP) {
      uint64_t m = w[0];
#pragma unroll
      for (int p = 1; p < NP; ++p) m = lane == p ? w[p] : m;
      planes[lane * pstride + b * slab * L + q] = WIDE ? m : (m | (m << L));
    }
  };
  auto row_of = [&](int q) {
    const int xl = q / L, x = (xs + xl + 2 * L) % L;
    return occ + (size_t)(x * L + (q - xl * L)) * L * nb;
  };
  if (!WIDE && quads) {
    for (int q0 = tid >> 5; q0 < slab * L; q0 += 4 * nw) {
      uint32_t v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int q = q0 + i * nw;
        v[i] = q < slab * L && lane < L ? reinterpret_cast<const uint32_t *>(row_of(q))[lane] : 0xffffffffu;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int q = q0 + i * nw;
        if (q < slab * L) {
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            uint64_t w[NP];
#pragma unroll
            for (int p = 0; p < NP; ++p)
              w[p] = __ballot_sync(kFull, (int)(int8_t)(v[i] >> (8 * b)) == (S == 0 ? g.pm1_minus : p + 1));
            put_plane(b, q, w);
          }
        }
      }
    }
  } else {
    for (int q = tid >> 5; q < slab * L; q += nw) {
      const int8_t *row = row_of(q);
      for (int b = 0; b < nb; ++b) {
        uint64_t w[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) w[p] = 0;
        for (int z0 = 0; z0 < L; z0 += 32) {
          const int z = z0 + lane;
          const int v = z < L ? row[z * nb + b] : -1;
#pragma unroll
          for (int p = 0; p < NP; ++p)
            w[p] |= (uint64_t)__ballot_sync(kFull, v == (S == 0 ? g.pm1_minus : p + 1)) << z0;
        }
        put_plane(b, q, w);
      }
    }
  }
  if (ctas > 1) box_cluster_barrier();  // the first CTA's counters are zero before any remote add
  else __syncthreads();

  const Word full = (Word)(L == (WIDE ? 64 : 32) ? ~(Word)0 : (((Word)1 << L) - 1));
  auto rot = [&](uint64_t d, int s) -> Word {  // bit z of the result: bit (z + s) mod L of the row
    if constexpr (WIDE) return (d >> s) | ((d << 1) << (L - 1 - s));
    else return __funnelshift_r((uint32_t)d, (uint32_t)(d >> 32), s);
  };
  auto pop = [](Word w) -> uint32_t {
    if constexpr (WIDE) return (uint32_t)__popcll(w);
    else return (uint32_t)__popc(w);
  };
  // index of the row at packed offset o from (xl, y)
  auto at = [&](uint32_t o, int xl, int y) -> int {
    int xx = xl + (int)(o & 255u) - 128, yy = y + (int)((o >> 8) & 255u) - 128;
    if (whole) {
      xx += xx < 0 ? L : 0;
      xx -= xx >= L ? L : 0;
    }
    yy += yy < 0 ? L : 0;
    yy -= yy >= L ? L : 0;
    return ((int)(o >> 24) * slab + xx) * L + yy;
  };
  auto total = [&](uint32_t v, uint32_t *to) {
    v = __reduce_add_sync(kFull, v);
    if (lane == 0 && v) atomicAdd(to, v);
  };
  // sites per species
  {
    uint32_t n[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) n[p] = 0;
    for (int i = tid; i < rows; i += blockDim.x) {
      const uint32_t ri = rowinfo[i];
      const int own = ((int)(ri >> 16) * slab + (int)((ri >> 8) & 255u)) * L + (int)(ri & 255u);
#pragma unroll
      for (int p = 0; p < NP; ++p) n[p] += pop((Word)planes[p * pstride + own] & full);
    }
#pragma unroll
    for (int p = 0; p < NP; ++p) total(n[p], &species[p]);
  }
  // tasks: a job's orbits over a share of the rows, enough of them to keep every warp busy
  const int shares = max(1, min((rows + 31) / 32, (2 * nw + c.n_jobs - 1) / c.n_jobs));
  const int share = (((rows + shares - 1) / shares) + 31) & ~31;
  for (int task = tid >> 5; task < c.n_jobs * shares; task += nw) {
    const int q = task % c.n_jobs, i0 = task / c.n_jobs * share, i1 = min(rows, i0 + share);
    const int2 job = jobs[q];
    const int pts = job.x;
    uint32_t *to = counts + job.y;
    if constexpr (S == 0) {
      uint32_t odd = 0;
      for (int i = i0 + lane; i < i1; i += 32) {
        const uint32_t ri = rowinfo[i];
        const int b = (int)(ri >> 16), xl = (int)((ri >> 8) & 255u), y = (int)(ri & 255u);
        const Word me = rot(planes[(b * slab + xl) * L + y], 0);
        const int e0 = ent_start[q * nb + b], e1 = ent_start[q * nb + b + 1];
        if (pts == 2) {
#pragma unroll 4
          for (int e = e0; e < e1; ++e) {
            const uint32_t o1 = (uint32_t)ent[e].x;
            odd += pop((me ^ rot(planes[at(o1, xl, y)], (int)(o1 >> 16) & 255)) & full);
          }
        } else {
#pragma unroll 2
          for (int e = e0; e < e1; ++e) {
            const int4 o = ent[e];
            Word w = me ^ rot(planes[at((uint32_t)o.x, xl, y)], (o.x >> 16) & 255) ^
                     rot(planes[at((uint32_t)o.y, xl, y)], (o.y >> 16) & 255);
            if (pts > 3) w ^= rot(planes[at((uint32_t)o.z, xl, y)], (o.z >> 16) & 255);
            odd += pop(w & full);
          }
        }
      }
      total(odd, to);
    } else {
      // all species' words of a point from its planes (the first species is where no plane is set)
      auto words = [&](int idx, int s, Word(&w)[S]) {
        Word any = 0;
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          w[p + 1] = rot(planes[p * pstride + idx], s) & full;
          any |= w[p + 1];
        }
        w[0] = full & ~any;
      };
      const int first = pts == 4 ? S : 1;  // four points: one pass per species of the first
      for (int f = 0; f < first; ++f) {
        uint32_t n[S * S * S];
#pragma unroll
        for (int t = 0; t < S * S * S; ++t) n[t] = 0;
        for (int i = i0 + lane; i < i1; i += 32) {
          const uint32_t ri = rowinfo[i];
          const int b = (int)(ri >> 16), xl = (int)((ri >> 8) & 255u), y = (int)(ri & 255u);
          Word me[S];
          words((b * slab + xl) * L + y, 0, me);
          const int e1 = ent_start[q * nb + b + 1];
          for (int e = ent_start[q * nb + b]; e < e1; ++e) {
            const int4 o = ent[e];
            Word w1[S];
            words(at((uint32_t)o.x, xl, y), (o.x >> 16) & 255, w1);
            if (pts == 2) {
#pragma unroll
              for (int u = 0; u < S; ++u)
#pragma unroll
                for (int v = 0; v < S; ++v) n[u + S * v] += pop(me[u] & w1[v]);
            } else {
              Word w2[S];
              words(at((uint32_t)o.y, xl, y), (o.y >> 16) & 255, w2);
              if (pts == 3) {
#pragma unroll
                for (int u = 0; u < S; ++u)
#pragma unroll
                  for (int v = 0; v < S; ++v) {
                    const Word uv = me[u] & w1[v];
#pragma unroll
                    for (int w = 0; w < S; ++w) n[u + S * (v + S * w)] += pop(uv & w2[w]);
                  }
              } else {
                Word w3[S], mf = me[0];
                words(at((uint32_t)o.z, xl, y), (o.z >> 16) & 255, w3);
#pragma unroll
                for (int u = 1; u < S; ++u) mf = f == u ? me[u] : mf;
#pragma unroll
                for (int u = 0; u < S; ++u)
#pragma unroll
                  for (int v = 0; v < S; ++v) {
                    const Word uv = mf & w1[u] & w2[v];
#pragma unroll
                    for (int w = 0; w < S; ++w) n[u + S * (v + S * w)] += pop(uv & w3[w]);
                  }
              }
            }
          }
        }
        // tuple (s0, s1, ..) at s0 + S s1 + ..; four points: f + S (tuple of points 1 .. 3)
        if (pts == 2) {
#pragma unroll
          for (int t = 0; t < S * S; ++t) total(n[t], &to[t]);
        } else {
#pragma unroll
          for (int t = 0; t < S * S * S; ++t) total(n[t], &to[pts == 4 ? f + S * t : t]);
        }
      }
    }
  }
  __syncthreads();
  if (ctas > 1) {
    if (rank != 0) {
      const uint32_t a = (uint32_t)__cvta_generic_to_shared(counts);
      uint32_t r;
      asm volatile("mapa.shared::cluster.u32 %0, %1, 0;\n" : "=r"(r) : "r"(a));
      for (int i = tid; i < c.n_counts + g.n_sym; i += blockDim.x)
        asm volatile("red.shared::cluster.add.u32 [%0], %1;\n" ::"r"(r + 4u * (uint32_t)i), "r"(counts[i]) : "memory");
    }
    box_cluster_barrier();
    if (rank != 0) return;
  }
  for (int k = tid; k < g.n_eci; k += blockDim.x) {
    const int kind = g.eci_kind[k];
    double v = 1.0;
    if (kind == 1) {
      if constexpr (S == 0) {
        v = (double)(N - 2 * (int)species[0]) / (double)N;
      } else {
        const double *bf = g.bf + g.eci_dec[k] * g.n_sym;
        uint32_t rest = (uint32_t)N;
        double s = 0.0;
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          s += (double)species[p] * bf[p + 1];
          rest -= species[p];
        }
        v = (s + (double)rest * bf[0]) / (double)N;
      }
    } else if (kind == 2) {
      double s = c.k_const[k];
      for (int i = c.k_start[k]; i < c.k_start[k + 1]; ++i) s += (double)counts[c.k_count[i]] * c.k_w[i];
      v = s * g.eci_fw[k];
    }
    cf_s[k] = v;
    cf[(size_t)chain * g.n_eci + k] = v;
  }
  __syncthreads();
  if (tid == 0) {
    // N * sum(eci * cf) in sorted-name order (ce_updater.cpp:236-242)
    double e = 0.0;
    for (int k = 0; k < g.n_eci; ++k) e += eci_s[k] * cf_s[k];
    energy[chain] = e * (double)(unsigned)N;
  }
}

int boxcf_ctas(const DevGeo &g, const BoxCf &c, int n_chains, int n_sms, size_t max_smem, size_t *smem) {
  if (!c.ok) return 0;
  // as many CTAs per chain as fill the GPU up to three times, each with at least 64 rows
  int ctas = 1;
  while (ctas < 8 && (long long)n_chains * ctas * 2 <= 3LL * n_sms &&
         g.box_L / (2 * ctas) * g.box_L * g.box_nb >= 64)
    ctas *= 2;
  for (; ctas <= 8; ctas *= 2) {  // more CTAs, smaller slabs
    *smem = box_layout(g, c, ctas, box_slab(g.box_L, ctas, c.hx)).total;
    if (*smem <= max_smem) return ctas;
  }
  return 0;
}

template <int S, bool WIDE>
static cudaError_t launch_box_t(const DevGeo &g, const BoxCf &c, int n_chains, int ctas, size_t smem, const int8_t *occ,
                                const double *eci, double *cf, double *energy, cudaStream_t st) {
  auto k = boxcf_kernel<S, WIDE>;
  cudaError_t e = allow_smem(k, g);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(n_chains * ctas));
  cfg.blockDim = dim3(kBoxThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ctas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ctas > 1 ? 1 : 0;
  e = cudaLaunchKernelEx(&cfg, k, g, c, ctas, occ, eci, cf, energy);
  return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t launch_boxcf(const DevGeo &g, const BoxCf &c, int n_chains, int ctas, size_t smem, const int8_t *occ,
                         const double *eci, double *cf, double *energy, cudaStream_t st) {
  const bool wide = g.box_L > 32;
  if (c.pm1)
    return wide ? launch_box_t<0, true>(g, c, n_chains, ctas, smem, occ, eci, cf, energy, st)
                : launch_box_t<0, false>(g, c, n_chains, ctas, smem, occ, eci, cf, energy, st);
  if (g.n_sym == 2)
    return wide ? launch_box_t<2, true>(g, c, n_chains, ctas, smem, occ, eci, cf, energy, st)
                : launch_box_t<2, false>(g, c, n_chains, ctas, smem, occ, eci, cf, energy, st);
  if (g.n_sym == 3)
    return wide ? launch_box_t<3, true>(g, c, n_chains, ctas, smem, occ, eci, cf, energy, st)
                : launch_box_t<3, false>(g, c, n_chains, ctas, smem, occ, eci, cf, energy, st);
  return cudaErrorInvalidValue;
}

}  // namespace cemc
