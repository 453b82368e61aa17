// FP64 products with the spin matrix x (n x N, entries +-1):
//   theta = b + x W (log-amplitudes, tanh theta), O v and O^T v.
//
// All three are sums of +- the same numbers.  GB300 issues two FP64 operations per
// clock and SM against 128 integer ones, so the sums are formed in 64-bit integers: a
// column of W (or V, or v t over the samples of a chunk) is rounded to a multiple of
// 2^-B of its largest entry's power of two, B = 62 - log2(terms) (55 for 100 terms),
// where FP64 would round every partial sum to 53 bits; the integer sum is exact, and one
// fused multiply-add brings it back.  A column whose largest entry is not finite or is
// near the ends of the exponent range takes the same tables in FP64.
//
// Four entries have sixteen signed sums: a table of those, made once for all the rows
// that use it, turns four additions into one lookup and one addition.
//   theta, O v: the table holds sums over four sites of W (or V) for a tile of 32
//     hidden units; every sample looks up its N / 4 entries;
//   O^T v: it holds sums over four samples of v t for a tile of 32 hidden units;
//     every site looks up its entry.
// Lanes are hidden units, so a lookup reads 256 consecutive bytes of shared memory
// at an address that the warp shares.
//
// log_cosh: sum_j log_cosh(theta_j) = sum |theta| + log prod (1 + e^(-2|theta|)) / 2
// over a lane's hidden units: a product per hidden unit instead of a log1p; tanh shares
// the exponential (expm1, so that it keeps its relative precision near 0).
//
// O^T v is bound by the issue of the lookups (six instructions each), theta and O v by
// the barriers around a tile's tables.  Measured (GB300, kernel time; before = tables of
// eight sums in FP64, whose additions kept the FP64 pipe at 65 to 75 %):
//   O^T v, n = 4,096, N = 100, M = 200 / 400: 90 / 174 -> 20 / 32 us;
//   O v, the same sizes: 104 / 189 -> 34 / 50 us;
//   the forward pass of a small gradient (n = 1,008, N = M = 16): 9 us (74 us without
//   tables).
// Error of theta against extended precision, N = 100, weights 0.05 x normal: rms 3.6e-17
// (FP64 additions 1.7e-16); O^T v 9.7e-15 (3.8e-14).
#include "signsum.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "units_f64.cuh"

namespace vmck {

namespace cg = cooperative_groups;

namespace {

constexpr int SR_THREADS = 256, SR_WARPS = SR_THREADS / 32;
constexpr int SS_TAB = 16 * 32;  // entries per group of four
constexpr int SR_HELD = 4;       // groups of a warp held in registers
constexpr int SR_BLOCK = 26;     // groups per table block: two CTAs' tables in an SM
constexpr int64_t SR_INDEX_MAX = 32 * 1024;  // bytes of sign indices per CTA
constexpr int SR_SITES_MAX = 16384;
constexpr int SR_FOLD = 512;  // hidden units of a lane between two logarithms of log psi

// acc + the table's entry number `byte` (a byte of four, moved to bits 8 to 11: the
// entries are 256 bytes apart)
template <typename T, int K>
__device__ __forceinline__ T entry(const T *tab, uint32_t four) {
  static_assert(sizeof(T) * 32 == 256, "one table row");
  constexpr uint32_t pick = 0x4404u | K << 4;  // {0, 0, byte K, 0}; operand 2 is 0
  return *reinterpret_cast<const T *>(reinterpret_cast<const char *>(tab) +
                                      __byte_perm(four, 0u, pick));
}

// entry i: signs by the bits of i (bit q set: minus w_q)
template <typename T>
__device__ __forceinline__ void fill_table(T *tab, T w0, T w1, T w2, T w3) {
  const T p = w0 + w1, m = w0 - w1, s = w2 + w3, d = w2 - w3;
  const T ps = p + s, ms = m + s, pd = p + d, md = m + d;
  const T p_s = p - s, m_s = m - s, p_d = p - d, m_d = m - d;
  tab[0 * 32] = ps;
  tab[1 * 32] = -m_s;
  tab[2 * 32] = ms;
  tab[3 * 32] = -p_s;
  tab[4 * 32] = p_d;
  tab[5 * 32] = -md;
  tab[6 * 32] = m_d;
  tab[7 * 32] = -pd;
  tab[8 * 32] = pd;
  tab[9 * 32] = -m_d;
  tab[10 * 32] = md;
  tab[11 * 32] = -p_d;
  tab[12 * 32] = p_s;
  tab[13 * 32] = -ms;
  tab[14 * 32] = m_s;
  tab[15 * 32] = -ps;
}

enum RowsOut { ROWS_LOGPSI = 0, ROWS_DOT = 1, ROWS_THETA = 2 };

// A cluster takes SR_WARPS * SPW samples; its CTAs share the tiles of 32 hidden units
// (a table serves all of the cluster's samples) and the first adds their sums.  Per
// tile: the tables (4 KB per four sites, `block` groups of sites at a time), then each
// warp its SPW samples.
//   ROWS_LOGPSI: out = logpsi, optional theta_out / tanh_out;
//   ROWS_DOT: out = sum_j t_sj theta_sj + x . a;
//   ROWS_THETA: theta_out and q_out = q_units(theta).
template <RowsOut OUT, int SPW>
__global__ void __launch_bounds__(SR_THREADS, 2) signed_rows_kernel(
    const double *__restrict__ params, const int8_t *__restrict__ x, int N, int M, int64_t n,
    int block, const double *__restrict__ t, double *__restrict__ out,
    double *__restrict__ theta_out, double *__restrict__ tanh_out, u64 *__restrict__ q_out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ uint32_t largest[SR_WARPS][32];
  __shared__ double sum[2 * SR_WARPS * SPW];  // sums, their low parts
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), ranks = (int)cluster.num_blocks();
  const int G = (N + 3) >> 2, G4 = (G + 3) & ~3, bits = sum_bits(N);
  double *tab = reinterpret_cast<double *>(smem_raw);
  uint8_t *index = reinterpret_cast<uint8_t *>(tab + (size_t)block * SS_TAB);  // [sample][G4]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t s0 = (int64_t)(blockIdx.x / ranks) * (SR_WARPS * SPW);
  const double *W = params + M, *a = W + (int64_t)N * M;
  const bool words = (N & 3) == 0 && ((uintptr_t)x & 3) == 0;
#pragma unroll 4
  for (int e = tid; e < SR_WARPS * SPW * G4; e += SR_THREADS) {
    const int s = e / G4, i = 4 * (e - s * G4);
    uint32_t m = 0u;
    if (s0 + s < n && i < N) {
      const int8_t *xe = x + (s0 + s) * N + i;
      if (words) {  // the four sign bits, moved to bits 28 to 31 by the product
        m = ((*reinterpret_cast<const uint32_t *>(xe) & 0x80808080u) >> 7) * 0x10204080u >> 28;
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) m |= (uint32_t)(i + q < N && xe[q] < 0) << q;
      }
    }
    index[e] = (uint8_t)m;
  }
  const uint8_t *mine = index + (size_t)warp * SPW * G4;
  const int64_t sw = s0 + warp * SPW;  // this warp's first sample
  double acc[SPW], prod[SPW];
  int units = 0;  // this lane's hidden units in prod
#pragma unroll
  for (int s = 0; s < SPW; ++s) {
    acc[s] = 0.0;
    prod[s] = 1.0;
  }
  auto load = [&](int g, int j, double (&w)[4]) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      w[q] = j < M && 4 * g + q < N ? __ldg(W + (int64_t)(4 * g + q) * M + j) : 0.0;
  };
  double held[SR_HELD][4];  // this warp's first groups, a tile ahead
#pragma unroll
  for (int k = 0; k < SR_HELD; ++k) load(warp + SR_WARPS * k, rank * 32 + lane, held[k]);
  for (int j0 = rank * 32; j0 < M; j0 += ranks * 32) {
    const int j = j0 + lane;
    const bool in = j < M;
    const double bj = in ? params[j] : 0.0;
    units += in;
    uint32_t size = 0u;
#pragma unroll
    for (int k = 0; k < SR_HELD; ++k)
#pragma unroll
      for (int q = 0; q < 4; ++q) size = max(size, size_word(held[k][q]));
    for (int g = warp + SR_WARPS * SR_HELD; g < G; g += SR_WARPS) {
      double w[4];
      load(g, j, w);
#pragma unroll
      for (int q = 0; q < 4; ++q) size = max(size, size_word(w[q]));
    }
    largest[warp][lane] = size;
    __syncthreads();  // also: the last tile's lookups are done, the indices are written
#pragma unroll
    for (int w = 0; w < SR_WARPS; ++w) size = max(size, largest[w][lane]);
    const int e = size >> 20;
    // the same in every warp
    const bool whole = __all_sync(0xffffffffu, size == 0u || exponent_fits(e));
    auto sums = [&](auto *table, auto (&v)[SPW], const auto &convert) {
#pragma unroll
      for (int s = 0; s < SPW; ++s) v[s] = 0;
      for (int gb = 0; gb < G; gb += block) {
        const int ge = min(gb + block, G);
        if (gb > 0) __syncthreads();  // the last block's lookups are done
        auto fill = [&](int g, const double (&w)[4]) {
          fill_table(table + (size_t)(g - gb) * SS_TAB + lane, convert(w[0]), convert(w[1]),
                     convert(w[2]), convert(w[3]));
        };
        int g = gb + warp;
        if (gb == 0) {
#pragma unroll
          for (int k = 0; k < SR_HELD; ++k, g += SR_WARPS) {
            if (g < ge) fill(g, held[k]);
            load(warp + SR_WARPS * k, j + ranks * 32, held[k]);
          }
        }
        for (; g < ge; g += SR_WARPS) {
          double w[4];
          load(g, j, w);
          fill(g, w);
        }
        __syncthreads();
        for (int g0 = gb; g0 < ge; g0 += 4) {
          uint32_t four[SPW];  // the indices of four groups
#pragma unroll
          for (int s = 0; s < SPW; ++s)
            four[s] = *reinterpret_cast<const uint32_t *>(mine + s * G4 + g0);
          const auto *tg = table + (size_t)(g0 - gb) * SS_TAB + lane;
          auto add = [&](auto k) {
            if (g0 + k.value < ge)
#pragma unroll
              for (int s = 0; s < SPW; ++s)
                v[s] += entry<std::remove_reference_t<decltype(v[0])>, k.value>(
                    tg + k.value * SS_TAB, four[s]);
          };
          add(std::integral_constant<int, 0>{});
          add(std::integral_constant<int, 1>{});
          add(std::integral_constant<int, 2>{});
          add(std::integral_constant<int, 3>{});
        }
      }
    };
    double th[SPW], ts[SPW];
    if (OUT == ROWS_DOT)
#pragma unroll
      for (int s = 0; s < SPW; ++s) ts[s] = in && sw + s < n ? __ldg(t + (sw + s) * M + j) : 0.0;
    if (whole) {
      long long v[SPW];
      sums(reinterpret_cast<long long *>(tab), v, [&](double w) { return to_units(w, e, bits); });
      const double unit = size == 0u ? 0.0 : unit_of(e, bits);
#pragma unroll
      for (int s = 0; s < SPW; ++s) th[s] = fma((double)v[s], unit, bj);
    } else {
      sums(tab, th, [](double w) { return w; });
#pragma unroll
      for (int s = 0; s < SPW; ++s) th[s] += bj;
    }
#pragma unroll
    for (int s = 0; s < SPW; ++s) {
      const int64_t row = sw + s;
      if (!in || row >= n) continue;
      if (OUT == ROWS_THETA) {
        theta_out[row * M + j] = th[s];
        q_out[row * M + j] = q_units(th[s]);
        continue;
      }
      if (OUT == ROWS_DOT) {
        acc[s] = fma(ts[s], th[s], acc[s]);
        continue;
      }
      const double v = fabs(th[s]);
      acc[s] += v;
      if (tanh_out) {
        const double e1 = expm1(-2.0 * v);  // e^(-2|theta|) - 1
        prod[s] = fma(prod[s], e1 + 1.0, prod[s]);
        tanh_out[row * M + j] = copysign(-e1 / (2.0 + e1), th[s]);
      } else {
        prod[s] = fma(prod[s], exp(-2.0 * v), prod[s]);
      }
      if (theta_out) theta_out[row * M + j] = th[s];
    }
    // 1 + e^(-2|theta|) is up to 2: without this, prod leaves the double range at 1,024 units
    // of a lane (M = 65,536).  A lane comes here from M = 32,705 on.
    if (OUT == ROWS_LOGPSI && units == SR_FOLD) {
#pragma unroll
      for (int s = 0; s < SPW; ++s) {
        acc[s] += log(ldexp(prod[s], -SR_FOLD));
        prod[s] = 1.0;
      }
      units = 0;
    }
  }
  if constexpr (OUT != ROWS_THETA) {
    // log psi is a sum of hundreds that its callers subtract from another: its last
    // additions are kept with their errors
    double low[SPW];
#pragma unroll
    for (int s = 0; s < SPW; ++s) {
      low[s] = 0.0;  // prod is at most 2^units; log 2 taken out exactly
      if (OUT == ROWS_LOGPSI) acc[s] = two_sum(acc[s], log(ldexp(prod[s], -units)), low[s]);
    }
    if (rank == 0)
      for (int i = lane; i < N; i += 32) {
        const double ai = __ldg(a + i);
#pragma unroll
        for (int s = 0; s < SPW; ++s)
          if (sw + s < n) {
            const double v = x[(sw + s) * N + i] < 0 ? -ai : ai;
            acc[s] = OUT == ROWS_LOGPSI ? two_sum(acc[s], v, low[s]) : acc[s] + v;
          }
      }
#pragma unroll
    for (int s = 0; s < SPW; ++s) {
      if (OUT == ROWS_LOGPSI) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const double v = __shfl_xor_sync(0xffffffffu, acc[s], o);
          low[s] += __shfl_xor_sync(0xffffffffu, low[s], o);
          acc[s] = two_sum(acc[s], v, low[s]);
        }
      } else {
        acc[s] = warp_sum(acc[s]);
      }
      if (lane == 0) {
        sum[warp * SPW + s] = acc[s];
        sum[SR_WARPS * SPW + warp * SPW + s] = low[s];
      }
    }
    if (ranks > 1) cluster.sync();
    else __syncthreads();
    if (rank == 0 && tid < SR_WARPS * SPW && s0 + tid < n) {
      double v = sum[tid], l = sum[SR_WARPS * SPW + tid];
      for (int r = 1; r < ranks; ++r) {
        const double *other = cluster.map_shared_rank(sum, r);
        v = two_sum(v, other[tid], l);
        l += other[SR_WARPS * SPW + tid];
      }
      out[s0 + tid] = v + l;
    }
    if (ranks > 1) cluster.sync();  // the others' sums stay until they are read
  }
}

template <RowsOut OUT, int SPW>
int launch_rows_as(cudaStream_t st, int ranks, const double *params, const int8_t *x, int N, int M,
                   int64_t n, const double *t, double *out, double *theta, double *tanh_out,
                   u64 *q) {
  const int G = (N + 3) / 4, G4 = (G + 3) & ~3;
  // equal blocks of whole fours (an index word holds four groups)
  const int blocks = G <= SR_BLOCK ? 1 : (G + 23) / 24;
  const int block = blocks == 1 ? G : ((G + blocks - 1) / blocks + 3) & ~3;
  const size_t smem = (size_t)block * SS_TAB * 8 + (size_t)SR_WARPS * SPW * G4;
  if (smem > 40 * 1024)
    VMCK_CUDA(cudaFuncSetAttribute(signed_rows_kernel<OUT, SPW>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t grid = (n + SR_WARPS * SPW - 1) / (SR_WARPS * SPW) * ranks;
  VMCK_REQUIRE(grid < (1ll << 31), "too many rows");
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ranks;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(SR_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = ranks > 1;
  VMCK_CUDA(cudaLaunchKernelEx(&cfg, signed_rows_kernel<OUT, SPW>, params, x, N, M, n, block, t,
                               out, theta, tanh_out, q));
  return check_launch("rows of signed sums");
}

// Clusters of two: they halve the tables per sample (n = 4,096, N = 100, M = 200 / 400:
// 34 / 50 us; single CTAs 37 / 65, clusters of four 39 / 57, whose last tiles leave CTAs
// idle).  Samples per warp: more of them share a table (about 200 instructions per four
// sites against 6 per sample), fewer fill the SMs; eight while that leaves a CTA per SM
// (half as many samples each: 50 / 75 us).
template <RowsOut OUT>
int launch_rows(cudaStream_t st, const double *params, const int8_t *x, int N, int M, int64_t n,
                const double *t, double *out, double *theta, double *tanh_out, u64 *q) {
  const int ranks = M > 32 ? 2 : 1;
  const int64_t full = (int64_t)sm_count() * SR_WARPS / ranks;
  // (very many sites: fewer samples' index bytes, one per four sites)
  const int64_t per = SR_WARPS * ((N + 15) / 16 * 4);
  if (n >= 8 * full && 8 * per <= SR_INDEX_MAX)
    return launch_rows_as<OUT, 8>(st, ranks, params, x, N, M, n, t, out, theta, tanh_out, q);
  if (n >= 4 * full && 4 * per <= SR_INDEX_MAX)
    return launch_rows_as<OUT, 4>(st, ranks, params, x, N, M, n, t, out, theta, tanh_out, q);
  if (n >= 2 * full && 2 * per <= SR_INDEX_MAX)
    return launch_rows_as<OUT, 2>(st, ranks, params, x, N, M, n, t, out, theta, tanh_out, q);
  return launch_rows_as<OUT, 1>(st, ranks, params, x, N, M, n, t, out, theta, tanh_out, q);
}

// ------------------------------------------------------------ O^T v
// C_ij = sum_s x_si (v_s t_sj) for i <= N, j <= M with x_sN = 1 and t_sM = 1: the
// kernel part, the hidden bias (i = N) and the visible bias (j = M) at once.  A CTA
// takes 32 hidden units, 8 IT sites and a chunk of samples, 32 samples at a time:
// warp g makes the table of samples 4 g .. 4 g + 3, then each warp adds to its
// sites i = 8 q + warp.  Two buffers, one barrier per 32 samples.  The unit of a column
// follows the largest |v| and |t| of at most OV_SPAN samples, which are read once more
// for that; longer chunks add their spans in FP64.
constexpr int OV_THREADS = 256, OV_WARPS = OV_THREADS / 32, OV_STEP = 4 * OV_WARPS, OV_SPAN = 256;
constexpr size_t OV_SMEM = 2 * OV_WARPS * SS_TAB * 8;  // two buffers of tables

// One span's sums for the warp's sites; T = long long or double.
template <int IT, typename T, typename Convert>
__device__ __forceinline__ void ot_v_span(const double *__restrict__ t,
                                          const int8_t *__restrict__ x, int N, int M, int64_t s0,
                                          int64_t s1, int i0, int sites, int cnt,
                                          const double *__restrict__ v, T *tab,
                                          uint2 (*index)[OV_WARPS * IT], T (&acc)[IT],
                                          const Convert &convert) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int j = blockIdx.x * 32 + lane;
#pragma unroll
  for (int q = 0; q < IT; ++q) acc[q] = 0;
  double p[4];  // this warp's products, a step ahead
  auto load = [&](int64_t sb) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int64_t s = sb + 4 * warp + k;
      p[k] = s < s1 && j <= M ? __ldg(v + s) : 0.0;
      if (s < s1 && j < M) p[k] *= __ldg(t + s * M + j);
    }
  };
  load(s0);
  int buf = 0;
  for (int64_t sb = s0; sb < s1; sb += OV_STEP, buf ^= 1) {
    T *tb = tab + buf * OV_WARPS * SS_TAB;
    fill_table(tb + warp * SS_TAB + lane, convert(p[0]), convert(p[1]), convert(p[2]),
               convert(p[3]));
    // a site's bytes of the eight groups, four groups per thread
    for (int e = tid; e < 2 * sites; e += OV_THREADS) {
      const int half = e >= sites, i = i0 + e - half * sites;
      const int64_t s = sb + 16 * half;
      uint32_t word = 0u;
      if (i < N)
#pragma unroll
        for (int k = 0; k < 16; ++k)
          word |= (uint32_t)(s + k < s1 && x[(s + k) * N + i] < 0) << (8 * (k >> 2) + (k & 3));
      (half ? index[buf][i - i0].y : index[buf][i - i0].x) = word;
    }
    __syncthreads();  // the other buffer's readers are past it: they wrote this one
    load(sb + OV_STEP);
#pragma unroll
    for (int q = 0; q < IT; ++q) {
      if (q < cnt) {
        const uint2 word = index[buf][OV_WARPS * q + warp];
        const T *e = tb + lane;
        const T a = entry<T, 0>(e, word.x) + entry<T, 1>(e + SS_TAB, word.x);
        const T b = entry<T, 2>(e + 2 * SS_TAB, word.x) + entry<T, 3>(e + 3 * SS_TAB, word.x);
        const T c = entry<T, 0>(e + 4 * SS_TAB, word.y) + entry<T, 1>(e + 5 * SS_TAB, word.y);
        const T d = entry<T, 2>(e + 6 * SS_TAB, word.y) + entry<T, 3>(e + 7 * SS_TAB, word.y);
        acc[q] += (a + b) + (c + d);
      }
    }
  }
  __syncthreads();  // before the next span writes the first buffer
}

template <int IT>
__global__ void __launch_bounds__(OV_THREADS, 3) ot_v_f64_kernel(
    const double *__restrict__ t, const int8_t *__restrict__ x, int N, int M, int64_t n,
    int64_t chunk, const double *__restrict__ v, double *__restrict__ ws) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *tab = reinterpret_cast<double *>(smem_raw);
  __shared__ uint2 index[2][OV_WARPS * IT];
  __shared__ uint32_t largest[2][OV_WARPS][32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int j = blockIdx.x * 32 + lane, i0 = blockIdx.y * (OV_WARPS * IT);
  const int64_t s0 = (int64_t)blockIdx.z * chunk, s1 = s0 + chunk < n ? s0 + chunk : n;
  const int sites = min(OV_WARPS * IT, N + 1 - i0);
  const int cnt = (sites - warp + OV_WARPS - 1) / OV_WARPS;  // sites of this warp
  const int bits = sum_bits(chunk < OV_SPAN ? chunk : OV_SPAN);
  const int64_t P = (int64_t)M + (int64_t)N * M + N;
  double *part = ws + (int64_t)blockIdx.z * P;
  for (int64_t sb = s0; sb < s1; sb += OV_SPAN) {
    const int64_t se = sb + OV_SPAN < s1 ? sb + OV_SPAN : s1;
    uint32_t st = 0u, sv = 0u;
#pragma unroll 8
    for (int64_t s = sb + warp; s < se; s += OV_WARPS)
      if (j < M) st = max(st, size_word(__ldg(t + s * M + j)));
    if (j >= M) st = 1023u << 20;  // ones
    for (int64_t s = sb + tid; s < se; s += OV_THREADS) sv = max(sv, size_word(__ldg(v + s)));
    largest[0][warp][lane] = st;
    largest[1][warp][lane] = __reduce_max_sync(0xffffffffu, sv);
    __syncthreads();
#pragma unroll
    for (int w = 0; w < OV_WARPS; ++w) {
      st = max(st, largest[0][w][lane]);
      sv = max(sv, largest[1][w][lane]);
    }
    const int et = st >> 20, ev = sv >> 20;
    const bool zero = st == 0u || sv == 0u;
    const int e = zero ? 1023 : ev + et - 1021;  // |v t| < 2^(e - 1022), also when rounded
    // the same in every warp; an entry below 2^-1022 or a factor that is not finite
    // takes the FP64 form
    const bool whole =
        __all_sync(0xffffffffu, (zero || (exponent_fits(e) && et >= 1 && ev >= 1)) &&
                                    et < 2047 && ev < 2047);
    double sum[IT];
    if (whole) {
      long long acc[IT];
      ot_v_span<IT>(t, x, N, M, sb, se, i0, sites, cnt, v, reinterpret_cast<long long *>(tab),
                    index, acc, [&](double p) { return to_units(p, e, bits); });
      const double unit = zero ? 0.0 : unit_of(e, bits);
#pragma unroll
      for (int q = 0; q < IT; ++q) sum[q] = (double)acc[q] * unit;
    } else {
      ot_v_span<IT>(t, x, N, M, sb, se, i0, sites, cnt, v, tab, index, sum,
                    [](double p) { return p; });
    }
    if (j > M) continue;
#pragma unroll
    for (int q = 0; q < IT; ++q) {
      if (q < cnt) {
        const int i = i0 + OV_WARPS * q + warp;
        if (i == N && j == M) continue;
        double *o = part + (i == N ? j : j < M ? M + (int64_t)i * M + j : M + (int64_t)N * M + i);
        *o = sb == s0 ? sum[q] : *o + sum[q];
      }
    }
  }
}

// sites per warp by N + 1 (a CTA holds OV_WARPS IT)
int ot_v_it(int N) { return N + 1 <= 32 ? 4 : (N + 1 <= 64 ? 8 : 16); }
int64_t ot_v_site_tiles(int N) {
  const int per = OV_WARPS * ot_v_it(N);
  return ((int64_t)N + per) / per;
}

int64_t ot_v_chunk(int N, int M, int64_t n) {
  const int64_t tiles = ((int64_t)M + 32) / 32 * ot_v_site_tiles(N);
  // about three CTAs for each of 152 SMs, at least 32 samples each
  const int64_t want = std::max<int64_t>(1, std::min<int64_t>((n + 31) / 32, 456 / tiles));
  return ((n + want - 1) / want + OV_STEP - 1) / OV_STEP * OV_STEP;
}

template <int IT>
int launch_ot_v(cudaStream_t st, dim3 grid, const double *t, const int8_t *x, int N, int M,
                int64_t n, int64_t chunk, const double *v, double *ws) {
  VMCK_CUDA(cudaFuncSetAttribute(ot_v_f64_kernel<IT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)OV_SMEM));
  ot_v_f64_kernel<IT><<<grid, OV_THREADS, OV_SMEM, st>>>(t, x, N, M, n, chunk, v, ws);
  return check_launch("rbm_ot_v partial");
}

}  // namespace

// (an index byte per four sites of eight samples in shared memory)
bool signed_rows_fit(int N) { return N <= SR_SITES_MAX; }

int logpsi_f64(cudaStream_t st, const double *params, int N, int M, const int8_t *x, int64_t n,
               double *logpsi, double *theta, double *tanh_out) {
  return launch_rows<ROWS_LOGPSI>(st, params, x, N, M, n, nullptr, logpsi, theta, tanh_out,
                                  nullptr);
}

int o_v_f64(cudaStream_t st, const double *t, const int8_t *x, int N, int M, int64_t n,
            const double *v, double *out) {
  return launch_rows<ROWS_DOT>(st, v, x, N, M, n, t, out, nullptr, nullptr, nullptr);
}

int theta_q_f64(cudaStream_t st, const double *params, int N, int M, const int8_t *x, int64_t n,
                double *theta, u64 *q) {
  return launch_rows<ROWS_THETA>(st, params, x, N, M, n, nullptr, nullptr, theta, nullptr, q);
}

int ot_v_f64_chunks(int N, int M, int64_t n) {
  const int64_t c = ot_v_chunk(N, M, n);
  return (int)((n + c - 1) / c);
}

int ot_v_f64(cudaStream_t st, const double *t, const int8_t *x, int N, int M, int64_t n,
             const double *v, double *ws) {
  const int64_t chunk = ot_v_chunk(N, M, n);
  const dim3 grid((unsigned)((M + 32) / 32), (unsigned)ot_v_site_tiles(N),
                  (unsigned)ot_v_f64_chunks(N, M, n));
  VMCK_REQUIRE(grid.y <= 65535 && grid.z <= 65535, "rbm_ot_v: too many tiles");
  switch (ot_v_it(N)) {
    case 4: return launch_ot_v<4>(st, grid, t, x, N, M, n, chunk, v, ws);
    case 8: return launch_ot_v<8>(st, grid, t, x, N, M, n, chunk, v, ws);
    default: return launch_ot_v<16>(st, grid, t, x, N, M, n, chunk, v, ws);
  }
}

}  // namespace vmck
