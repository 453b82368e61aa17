// FP64 products with the spin matrix x (n x N, entries +-1):
//   theta = b + x W (log-amplitudes, tanh theta), O v and O^T v.
//
// All three are sums of +- the same numbers, and GB300 issues two FP64 operations
// per clock and SM, so the additions bound them.  Four entries have only eight
// signed sums up to an overall sign: a table of those eight, made once for all the
// rows that use it, turns four additions into one lookup and one addition.
//   theta, O v: the table holds sums over four sites of W (or V) for a tile of 32
//     hidden units; every sample looks up its N / 4 entries;
//   O^T v: it holds sums over four samples of v t for a tile of 32 hidden units;
//     every site looks up its entry.
// Lanes are hidden units, so a lookup reads 256 consecutive bytes of shared memory
// at an address that the warp shares.
//
// log_cosh: sum_j log_cosh(theta_j) = sum |theta| + log prod (1 + e^(-2|theta|))
// - M log 2: a product per hidden unit instead of a log1p; tanh shares the
// exponential (expm1, so that it keeps its relative precision near 0).
//
// Measured (GB300, kernel time; before = 64 x 64 tiles of one addition per entry,
// a CTA per 64 samples or per 1,024 samples and tile):
//   O^T v, n = 4,096, N = 100, M = 200: 1,540 -> 90 us;
//   O v, the same sizes: 403 -> 104 us;
//   the forward pass of a small gradient (n = 1,008, N = M = 16): 74 -> 9 us.
#include "signsum.cuh"

#include <algorithm>

namespace vmck {

namespace {

constexpr int SR_THREADS = 256, SR_WARPS = SR_THREADS / 32;
constexpr int SR_TAB = 8 * 32;  // doubles per group of four sites
constexpr size_t SS_SMEM_MAX = 200 * 1024;

// Signs of four spins as a table index: the three relative to the first in bits
// 0-2, the first itself in bit 7.
__device__ __forceinline__ uint32_t sign_index(bool m0, bool m1, bool m2, bool m3) {
  return (uint32_t)(m0 != m1) | (uint32_t)(m0 != m2) << 1 | (uint32_t)(m0 != m3) << 2 |
         (uint32_t)m0 << 7;
}

// +- the table's entry: byte's low bits choose it, bit 7 negates
__device__ __forceinline__ double lookup(const double *tab, uint32_t byte) {
  const double v = tab[(byte & 7u) * 32];
  return __hiloint2double(__double2hiint(v) ^ (int)((byte & 0x80u) << 24), __double2loint(v));
}

__device__ __forceinline__ void fill_table(double *tab, double w0, double w1, double w2,
                                           double w3) {
  const double p = w0 + w1, m = w0 - w1, s = w2 + w3, d = w2 - w3;
  tab[0 * 32] = p + s;
  tab[1 * 32] = m + s;
  tab[2 * 32] = p - d;  // w2 -, w3 +
  tab[3 * 32] = m - d;
  tab[4 * 32] = p + d;  // w2 +, w3 -
  tab[5 * 32] = m + d;
  tab[6 * 32] = p - s;
  tab[7 * 32] = m - s;
}

enum RowsOut { ROWS_LOGPSI = 0, ROWS_DOT = 1 };

// A CTA takes SR_WARPS * SPW samples through all hidden units, 32 at a time: the
// tables of the tile (2 KB per four sites), then each warp its SPW samples.
//   ROWS_LOGPSI: out = logpsi, optional theta_out / tanh_out;
//   ROWS_DOT: out = sum_j t_sj theta_sj + x . a.
template <RowsOut OUT, int SPW>
__global__ void __launch_bounds__(SR_THREADS) signed_rows_kernel(
    const double *__restrict__ params, const int8_t *__restrict__ x, int N, int M, int64_t n,
    const double *__restrict__ t, double *__restrict__ out, double *__restrict__ theta_out,
    double *__restrict__ tanh_out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int G = (N + 3) >> 2, G4 = (G + 3) & ~3;
  double *tab = reinterpret_cast<double *>(smem_raw);
  uint8_t *index = reinterpret_cast<uint8_t *>(tab + (size_t)G * SR_TAB);  // [sample][G4]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t s0 = (int64_t)blockIdx.x * (SR_WARPS * SPW);
  const double *W = params + M, *a = W + (int64_t)N * M;
  for (int e = tid; e < SR_WARPS * SPW * G4; e += SR_THREADS) {
    const int s = e / G4, i = 4 * (e - s * G4);
    bool m[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) m[q] = s0 + s < n && i + q < N && x[(s0 + s) * N + i + q] < 0;
    index[e] = (uint8_t)sign_index(m[0], m[1], m[2], m[3]);
  }
  const uint8_t *mine = index + (size_t)warp * SPW * G4;
  const int64_t sw = s0 + warp * SPW;  // this warp's first sample
  double acc[SPW], prod[SPW];
#pragma unroll
  for (int s = 0; s < SPW; ++s) {
    acc[s] = 0.0;
    prod[s] = 1.0;
  }
  for (int j0 = 0; j0 < M; j0 += 32) {
    const int j = j0 + lane;
    const bool in = j < M;
    __syncthreads();  // the last tile's lookups are done; the indices are written
    for (int g = warp; g < G; g += SR_WARPS) {
      double w[4];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        w[q] = in && 4 * g + q < N ? W[(int64_t)(4 * g + q) * M + j] : 0.0;
      fill_table(tab + (size_t)g * SR_TAB + lane, w[0], w[1], w[2], w[3]);
    }
    __syncthreads();
    double th[SPW];
    const double bj = in ? params[j] : 0.0;
#pragma unroll
    for (int s = 0; s < SPW; ++s) th[s] = bj;
    for (int g0 = 0; g0 < G; g0 += 4) {
      uint32_t four[SPW];  // the indices of four groups
#pragma unroll
      for (int s = 0; s < SPW; ++s)
        four[s] = *reinterpret_cast<const uint32_t *>(mine + s * G4 + g0);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (g0 + k < G) {
          const double *tg = tab + (size_t)(g0 + k) * SR_TAB + lane;
#pragma unroll
          for (int s = 0; s < SPW; ++s) th[s] += lookup(tg, (four[s] >> (8 * k)) & 0xffu);
        }
      }
    }
#pragma unroll
    for (int s = 0; s < SPW; ++s) {
      const int64_t row = sw + s;
      if (!in || row >= n) continue;
      if (OUT == ROWS_DOT) {
        acc[s] = fma(t[row * M + j], th[s], acc[s]);
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
  }
#pragma unroll
  for (int s = 0; s < SPW; ++s) {
    const int64_t row = sw + s;
    if (row >= n) break;  // uniform over the warp
    double v = acc[s];
    // at most 2^(M / 32) per lane
    if (OUT == ROWS_LOGPSI) v += log(prod[s]);
    for (int i = lane; i < N; i += 32) v += (x[row * N + i] < 0 ? -a[i] : a[i]);
    v = warp_sum(v);
    if (lane == 0) out[row] = OUT == ROWS_LOGPSI ? v - M * 0.69314718055994530942 : v;
  }
}

size_t rows_smem(int N, int spw) {
  const int G = (N + 3) / 4, G4 = (G + 3) & ~3;
  return (size_t)G * SR_TAB * 8 + (size_t)SR_WARPS * spw * G4;
}

int sm_count() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

template <RowsOut OUT, int SPW>
int launch_rows_as(cudaStream_t st, const double *params, const int8_t *x, int N, int M, int64_t n,
                   const double *t, double *out, double *theta, double *tanh_out) {
  const size_t smem = rows_smem(N, SPW);
  VMCK_CUDA(cudaFuncSetAttribute(signed_rows_kernel<OUT, SPW>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t grid = (n + SR_WARPS * SPW - 1) / (SR_WARPS * SPW);
  VMCK_REQUIRE(grid < (1ll << 31), "too many rows");
  signed_rows_kernel<OUT, SPW><<<(unsigned)grid, SR_THREADS, smem, st>>>(params, x, N, M, n, t, out,
                                                                         theta, tanh_out);
  return check_launch(OUT == ROWS_LOGPSI ? "rbm_logpsi" : "rbm_o_v");
}

// Samples per warp: more of them share a table (its 12 additions per four sites
// against one per sample), fewer fill the SMs; eight while that leaves two CTAs
// per SM.
template <RowsOut OUT>
int launch_rows(cudaStream_t st, const double *params, const int8_t *x, int N, int M, int64_t n,
                const double *t, double *out, double *theta, double *tanh_out) {
  const int64_t two = 2 * (int64_t)sm_count() * SR_WARPS;
  if (n >= 8 * two)
    return launch_rows_as<OUT, 8>(st, params, x, N, M, n, t, out, theta, tanh_out);
  if (n >= 4 * two)
    return launch_rows_as<OUT, 4>(st, params, x, N, M, n, t, out, theta, tanh_out);
  if (n >= two)
    return launch_rows_as<OUT, 2>(st, params, x, N, M, n, t, out, theta, tanh_out);
  return launch_rows_as<OUT, 1>(st, params, x, N, M, n, t, out, theta, tanh_out);
}

// ------------------------------------------------------------ O^T v
// C_ij = sum_s x_si (v_s t_sj) for i <= N, j <= M with x_sN = 1 and t_sM = 1: the
// kernel part, the hidden bias (i = N) and the visible bias (j = M) at once.  A CTA
// takes 32 hidden units, 4 IT sites and a chunk of samples, 16 samples at a time:
// warp g makes the table of samples 4 g .. 4 g + 3, then each warp adds to its
// sites i = 4 q + warp.  Two buffers, one barrier per 16 samples.
constexpr int OV_THREADS = 128, OV_STEP = 16;

template <int IT>
__global__ void __launch_bounds__(OV_THREADS) ot_v_f64_kernel(
    const double *__restrict__ t, const int8_t *__restrict__ x, int N, int M, int64_t n,
    int64_t chunk, const double *__restrict__ v, double *__restrict__ ws) {
  __shared__ double tab[2][4][8 * 32];
  __shared__ uint32_t index[2][4 * IT];  // the four groups' bytes of a site
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int j = blockIdx.x * 32 + lane, i0 = blockIdx.y * (4 * IT);
  const int64_t s0 = (int64_t)blockIdx.z * chunk, s1 = s0 + chunk < n ? s0 + chunk : n;
  const int sites = min(4 * IT, N + 1 - i0);
  const int cnt = (sites - warp + 3) >> 2;  // sites of this warp
  double acc[IT];
#pragma unroll
  for (int q = 0; q < IT; ++q) acc[q] = 0.0;
  int buf = 0;
  for (int64_t sb = s0; sb < s1; sb += OV_STEP, buf ^= 1) {
    double w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int64_t s = sb + 4 * warp + k;
      w[k] = 0.0;
      if (s < s1 && j <= M) w[k] = j < M ? v[s] * t[s * M + j] : v[s];
    }
    fill_table(&tab[buf][warp][lane], w[0], w[1], w[2], w[3]);
    for (int e = tid; e < sites; e += OV_THREADS) {
      const int i = i0 + e;
      uint32_t word = 0u;
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        bool m[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int64_t s = sb + 4 * g + k;
          m[k] = i < N && s < s1 && x[s * N + i] < 0;
        }
        word |= sign_index(m[0], m[1], m[2], m[3]) << (8 * g);
      }
      index[buf][e] = word;
    }
    __syncthreads();  // the other buffer's readers are past it: they wrote this one
#pragma unroll
    for (int q = 0; q < IT; ++q) {
      if (q < cnt) {
        const uint32_t word = index[buf][4 * q + warp];
#pragma unroll
        for (int g = 0; g < 4; ++g)
          acc[q] += lookup(&tab[buf][g][lane], (word >> (8 * g)) & 0xffu);
      }
    }
  }
  if (j > M) return;
  const int64_t P = (int64_t)M + (int64_t)N * M + N;
  double *part = ws + (int64_t)blockIdx.z * P;
#pragma unroll
  for (int q = 0; q < IT; ++q) {
    if (q < cnt) {
      const int i = i0 + 4 * q + warp;
      if (i < N)
        part[j < M ? M + (int64_t)i * M + j : M + (int64_t)N * M + i] = acc[q];
      else if (j < M)
        part[j] = acc[q];
    }
  }
}

// sites per warp by N + 1 (a CTA holds 4 IT)
int ot_v_it(int N) { return N + 1 <= 32 ? 8 : (N + 1 <= 64 ? 16 : 32); }

int64_t ot_v_chunk(int N, int M, int64_t n) {
  const int64_t tiles = ((int64_t)M + 32) / 32 * ((N + 4 * ot_v_it(N)) / (4 * ot_v_it(N)));
  // about four CTAs for each of 152 SMs, at least 32 samples each
  const int64_t want = std::max<int64_t>(1, std::min<int64_t>((n + 31) / 32, 608 / tiles));
  return ((n + want - 1) / want + OV_STEP - 1) / OV_STEP * OV_STEP;
}

}  // namespace

bool signed_rows_fit(int N) { return rows_smem(N, 8) <= SS_SMEM_MAX; }

int logpsi_f64(cudaStream_t st, const double *params, int N, int M, const int8_t *x, int64_t n,
               double *logpsi, double *theta, double *tanh_out) {
  return launch_rows<ROWS_LOGPSI>(st, params, x, N, M, n, nullptr, logpsi, theta, tanh_out);
}

int o_v_f64(cudaStream_t st, const double *t, const int8_t *x, int N, int M, int64_t n,
            const double *v, double *out) {
  return launch_rows<ROWS_DOT>(st, v, x, N, M, n, t, out, nullptr, nullptr);
}

int ot_v_f64_chunks(int N, int M, int64_t n) {
  const int64_t c = ot_v_chunk(N, M, n);
  return (int)((n + c - 1) / c);
}

int ot_v_f64(cudaStream_t st, const double *t, const int8_t *x, int N, int M, int64_t n,
             const double *v, double *ws) {
  const int64_t chunk = ot_v_chunk(N, M, n);
  const int it = ot_v_it(N);
  const dim3 grid((unsigned)((M + 32) / 32), (unsigned)((N + 4 * it) / (4 * it)),
                  (unsigned)ot_v_f64_chunks(N, M, n));
  VMCK_REQUIRE(grid.y <= 65535 && grid.z <= 65535, "rbm_ot_v: too many tiles");
  if (it == 8)
    ot_v_f64_kernel<8><<<grid, OV_THREADS, 0, st>>>(t, x, N, M, n, chunk, v, ws);
  else if (it == 16)
    ot_v_f64_kernel<16><<<grid, OV_THREADS, 0, st>>>(t, x, N, M, n, chunk, v, ws);
  else
    ot_v_f64_kernel<32><<<grid, OV_THREADS, 0, st>>>(t, x, N, M, n, chunk, v, ws);
  return check_launch("rbm_ot_v partial");
}

}  // namespace vmck
