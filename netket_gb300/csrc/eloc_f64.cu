// FP64 local energies of the RBM from tables of flip factors.
//
// A connected element that changes theta_j by delta_j multiplies the amplitude
// by prod_j cosh(theta_j + delta_j) / cosh(theta_j).  With rho_j = exp(-2 theta_j)
//   cosh(theta + delta) / cosh(theta) = e^delta (1 + rho e^(-2 delta)) / (1 + rho):
// only sums of positive terms, so every factor keeps its relative precision (a
// few ulp) whatever theta and delta are.  prod_j (1 + rho_j) belongs to the
// sample and prod_j e^delta_j to the flipped sites; what is left per hidden unit
// is one fused multiply-add and one product.  A spin flip changes theta_j by
// -+2 W_ij, so e^(-2 delta) comes from two tables, exp(4 W) and exp(-4 W), made
// once per call (N M exponentials for n N M factors).
//
// What bounds it: GB300 issues two FP64 operations per clock and SM.  A one-site
// flip costs 2 of them per hidden unit and a two-site one 3, where
// log_cosh(theta') - log_cosh(theta), with its exp and log1p, cost about 60 and
// kept the FP64 pipe at 86 % (ncu).
//
// A product leaves the double range only where the ratio, or a partial product
// of it, does; such an element is formed again as the difference of log_cosh sums
// (slow_log_ratio), which is also the path of a non-finite parameter.
#include <algorithm>

#include "common.cuh"
#include "localop.cuh"

namespace vmck {

constexpr int EF_THREADS = 128, EF_WARPS = EF_THREADS / 32;
constexpr int EF_SAMPLES = 4;  // Ising: samples per CTA
// a product outside this range (it holds no denormals) is formed again in the
// log domain
constexpr double EF_TINY = 1e-290, EF_HUGE = 1e290;

// Tables of the call: up[i, j] = exp(-4 W_ij) and down[i, j] = exp(4 W_ij), the
// factor e^(-2 delta) of turning spin i up (x = -1 -> 1) and down, for i < N and
// ones in row N (a site left alone); rup[i] = exp(2 (sum_j W_ij + a_i)) and rdown
// its inverse, the factors of a flip that do not depend on theta.
struct FlipTables {
  const double *up, *down;    // (N + 1) x M
  const double *rup, *rdown;  // N
};

__host__ __device__ inline int64_t flip_table_len(int N, int M) {
  return 2 * ((int64_t)(N + 1) * M + N);
}

__host__ __device__ inline FlipTables flip_tables(const double *ws, int N, int M) {
  const int64_t w = (int64_t)(N + 1) * M;
  return FlipTables{ws, ws + w, ws + 2 * w, ws + 2 * w + N};
}

// one block per row of the tables
__global__ void __launch_bounds__(256) flip_tables_kernel(const double *__restrict__ params, int N,
                                                          int M, double *__restrict__ ws) {
  __shared__ double red[8];
  const int64_t w = (int64_t)(N + 1) * M;
  const int i = blockIdx.x;
  const double *row = params + M + (int64_t)i * M;
  double sum = 0.0;
  for (int j = threadIdx.x; j < M; j += blockDim.x) {
    const double v = i < N ? row[j] : 0.0;
    ws[(int64_t)i * M + j] = exp(-4.0 * v);
    ws[w + (int64_t)i * M + j] = exp(4.0 * v);
    sum += v;
  }
  sum = block_sum(sum, red);
  if (threadIdx.x == 0 && i < N) {
    const double v = 2.0 * (sum + params[M + (int64_t)N * M + i]);
    ws[2 * w + i] = exp(v);
    ws[2 * w + N + i] = exp(-v);
  }
}

// x * W without a conversion of x: the sign bit of W flipped where x = -1
__device__ __forceinline__ double signed_by(double w, int x) {
  return __hiloint2double(__double2hiint(w) ^ (x & 0x80000000), __double2loint(w));
}

// theta of the samples xs[s * ldx + i], s < S, for one hidden unit
template <int S>
__device__ __forceinline__ void thetas(const double *__restrict__ params, int N, int M,
                                       const int8_t *xs, int ldx, int j, double (&th)[S]) {
  const double b = params[j];
#pragma unroll
  for (int s = 0; s < S; ++s) th[s] = b;
  const double *W = params + M + j;
#pragma unroll 4
  for (int i = 0; i < N; ++i) {
    const double w = __ldg(W + (int64_t)i * M);
#pragma unroll
    for (int s = 0; s < S; ++s) th[s] += signed_by(w, (int)xs[s * ldx + i]);
  }
}

// Log-ratio of one element as the difference of log_cosh sums, by the warp, from
// scratch (theta is not kept): sites site[q] with change d[q].
__device__ __noinline__ double slow_log_ratio(const double *__restrict__ params, int N, int M,
                                              const int8_t *xs, const int *site, const int *d,
                                              int ns) {
  const int lane = threadIdx.x & 31;
  const double *W = params + M, *a = W + (int64_t)N * M;
  double s = 0.0;
  for (int j = lane; j < M; j += 32) {
    double th[1];
    thetas<1>(params, N, M, xs, 0, j, th);
    double t = th[0];
    for (int q = 0; q < ns; ++q) t += (double)d[q] * W[(int64_t)site[q] * M + j];
    s += log_cosh(t) - log_cosh(th[0]);
  }
  s = warp_sum(s);
  for (int q = 0; q < ns; ++q) s += (double)d[q] * a[site[q]];
  return s;
}

__device__ __forceinline__ bool in_range(double v) { return v > EF_TINY && v < EF_HUGE; }

// Products over the warp of four values per lane: the value of element e =
// lane / 8 on every lane of its group, in six multiplies per lane where four
// full butterflies take twenty.
__device__ __forceinline__ double warp_prod4(const double (&v)[4]) {
  const int lane = threadIdx.x & 31;
  const bool h = lane & 16, g = lane & 8;
  const double a = (h ? v[2] : v[0]) * __shfl_xor_sync(0xffffffffu, h ? v[0] : v[2], 16);
  const double b = (h ? v[3] : v[1]) * __shfl_xor_sync(0xffffffffu, h ? v[1] : v[3], 16);
  double r = (g ? b : a) * __shfl_xor_sync(0xffffffffu, g ? a : b, 8);
  r *= __shfl_xor_sync(0xffffffffu, r, 4);
  r *= __shfl_xor_sync(0xffffffffu, r, 2);
  r *= __shfl_xor_sync(0xffffffffu, r, 1);
  return r;
}

// Product of 1 / (1 + rho_j) over the hidden units j = lane, lane + 32, ...
__device__ __forceinline__ double lane_norm(const double *rho, int M) {
  double v = 1.0;
  for (int j = threadIdx.x & 31; j < M; j += 32) v = fma(v, rho[j], v);
  return 1.0 / v;
}

// ------------------------------------------------------------ Ising
// One CTA takes EF_SAMPLES samples: theta of the four in one pass over W, rho in
// shared memory, then each warp takes sites k = warp, warp + 4, ...: one read of
// the two table rows serves the flip of site k in all four samples, whose
// products are reduced together (warp_prod4).  Lane group e accumulates sample
// e's sum.  FP64 work per sample: N M additions for theta, 2 N M operations for
// the flips.  N = 256, M = 256, n = 2,048: 1.14 ms; one
// log_cosh per hidden unit and flip (eloc_ising_kernel<double>) 20.1 ms.
__global__ void __launch_bounds__(EF_THREADS) eloc_ising_f64_kernel(
    const double *__restrict__ params, int N, int M, const int8_t *__restrict__ x, int64_t n,
    const int32_t *__restrict__ edges, int n_edges, double h, double J, FlipTables tab,
    double *__restrict__ eloc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *rho = reinterpret_cast<double *>(smem_raw);  // [sample][M]
  int8_t *xs = reinterpret_cast<int8_t *>(rho + (size_t)EF_SAMPLES * M);
  __shared__ double red[EF_WARPS][EF_SAMPLES];
  __shared__ double norm[EF_SAMPLES][32];
  __shared__ int diag[EF_SAMPLES];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, mine = lane >> 3;
  for (int64_t b0 = (int64_t)blockIdx.x * EF_SAMPLES; b0 < n;
       b0 += (int64_t)gridDim.x * EF_SAMPLES) {
    // the last CTA's missing samples repeat sample n - 1; their results are not stored
    for (int e = tid; e < EF_SAMPLES * N; e += EF_THREADS) {
      const int s = e / N, i = e - s * N;
      const int64_t b = b0 + s < n ? b0 + s : n - 1;
      xs[e] = x[b * N + i];
    }
    if (tid < EF_SAMPLES) diag[tid] = 0;
    __syncthreads();
    for (int e = tid; e < EF_SAMPLES * n_edges; e += EF_THREADS) {
      const int s = e / n_edges, q = e - s * n_edges;
      const int same = xs[s * N + edges[2 * q]] == xs[s * N + edges[2 * q + 1]] ? 1 : -1;
      atomicAdd(&diag[s], same);  // integers: the order does not matter
    }
    double acc = 0.0;
    if (h != 0.0) {
      for (int j = tid; j < M; j += EF_THREADS) {
        double th[EF_SAMPLES];
        thetas<EF_SAMPLES>(params, N, M, xs, N, j, th);
#pragma unroll
        for (int s = 0; s < EF_SAMPLES; ++s) rho[s * M + j] = exp(-2.0 * th[s]);
      }
      __syncthreads();
      static_assert(EF_WARPS == EF_SAMPLES, "one warp per sample's norms");
      norm[warp][lane] = lane_norm(rho + warp * M, M);
      __syncthreads();
      for (int k = warp; k < N; k += EF_WARPS) {
        bool up[EF_SAMPLES];
        double f[EF_SAMPLES];
#pragma unroll
        for (int s = 0; s < EF_SAMPLES; ++s) {
          up[s] = xs[s * N + k] < 0;
          f[s] = norm[s][lane];
        }
        const double *eu = tab.up + (int64_t)k * M, *ed = tab.down + (int64_t)k * M;
#pragma unroll 2
        for (int j = lane; j < M; j += 32) {
          const double u = __ldg(eu + j), d = __ldg(ed + j);
#pragma unroll
          for (int s = 0; s < EF_SAMPLES; ++s) f[s] *= fma(rho[s * M + j], up[s] ? u : d, 1.0);
        }
        bool ok = true;
#pragma unroll
        for (int s = 0; s < EF_SAMPLES; ++s) ok &= in_range(f[s]);
        const double r = warp_prod4(f);
        const double v = r * (xs[mine * N + k] < 0 ? tab.rup[k] : tab.rdown[k]);
        ok &= in_range(r) && in_range(v);
        if (__all_sync(0xffffffffu, ok)) {
          acc += v;
        } else {
#pragma unroll 1
          for (int s = 0; s < EF_SAMPLES; ++s) {
            const int d = -2 * xs[s * N + k];
            const double lr = slow_log_ratio(params, N, M, xs + s * N, &k, &d, 1);
            if (mine == s) acc += exp(lr);
          }
        }
      }
    }
    if ((lane & 7) == 0) red[warp][mine] = acc;
    __syncthreads();
    if (tid < EF_SAMPLES && b0 + tid < n) {
      double s = 0.0;
#pragma unroll
      for (int w = 0; w < EF_WARPS; ++w) s += red[w][tid];
      eloc[b0 + tid] = (h != 0.0 ? -h * s : 0.0) + J * (double)diag[tid];
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------ LocalOperator
// One CTA per sample: theta and rho of the sample, the connected elements
// enumerated in shared memory (local_conn_enumerate), then each warp takes groups
// of four elements: NS table rows each (a site that the element leaves alone
// reads the row of ones), four products reduced together.  Elements of two sites
// cost 3 FP64 operations per hidden unit.  10 x 10 Heisenberg, M = 200, n =
// 4,096 (about 100 elements a sample): 1.02 ms; eloc_local_kernel<double> 14.4 ms.
template <int NS>
__global__ void __launch_bounds__(EF_THREADS) eloc_local_f64_kernel(
    const double *__restrict__ params, int N, int M, const int8_t *__restrict__ x, int64_t n,
    vmck_local_op op, FlipTables tab, double *__restrict__ eloc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  LocalConnShared sh = local_conn_shared_layout(smem_raw, op);
  double *rho = reinterpret_cast<double *>(sh.end);
  __shared__ double red[32], norm[32];
  const Grp g = cta_grp();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, mine = lane >> 3;
  const int S = op.max_sites;
  const int64_t ones = (int64_t)N * M, down = tab.down - tab.up;
  for (int64_t b = blockIdx.x; b < n; b += gridDim.x) {
    for (int i = tid; i < N; i += EF_THREADS) sh.xs[i] = x[b * N + i];
    __syncthreads();
    for (int j = tid; j < M; j += EF_THREADS) {
      double th[1];
      thetas<1>(params, N, M, sh.xs, 0, j, th);
      rho[j] = exp(-2.0 * th[0]);
    }
    const int kept = local_conn_enumerate(op, sh, g, true);  // its barriers order rho
    if (warp == 0) norm[lane] = lane_norm(rho, M);
    __syncthreads();
    double acc = 0.0;
    for (int k0 = 4 * warp; k0 < kept; k0 += 4 * EF_WARPS) {
      const double *row[4][NS];
      double fix[4], f[4];
      int same = 0;  // bit e: element e leaves the configuration as it is (ratio 1)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        f[e] = norm[lane];
        fix[e] = 1.0;
#pragma unroll
        for (int q = 0; q < NS; ++q) row[e][q] = tab.up + ones;
        same |= 1 << e;
        const int k = k0 + e;
        const int t = k < kept ? sh.slot_term[k] : -1;
        if (t < 0) continue;
        const int8_t *xpv =
            op.x_prime + (((int64_t)t * op.max_rows + sh.row[t]) * op.max_conns +
                          sh.slot_col[k]) * S;
        const int sz = op.acting_size[t];
#pragma unroll
        for (int q = 0; q < NS; ++q) {
          if (q < sz) {
            const int st = op.acting_on[t * S + q];
            const int d = (int)xpv[q] - (int)sh.xs[st];
            if (d != 0) {
              row[e][q] = tab.up + (int64_t)st * M + (d > 0 ? 0 : down);
              fix[e] *= d > 0 ? tab.rup[st] : tab.rdown[st];
              same &= ~(1 << e);
            }
          }
        }
      }
#pragma unroll(NS <= 2 ? 2 : 1)
      for (int j = lane; j < M; j += 32) {
        const double r = rho[j];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          double u = __ldg(row[e][0] + j);
#pragma unroll
          for (int q = 1; q < NS; ++q) u *= __ldg(row[e][q] + j);
          f[e] *= fma(r, u, 1.0);
        }
      }
      bool ok = true;
#pragma unroll
      for (int e = 0; e < 4; ++e) ok &= in_range(f[e]);
      const double r = warp_prod4(f);
      double v = r * (mine == 0 ? fix[0] : mine == 1 ? fix[1] : mine == 2 ? fix[2] : fix[3]);
      ok &= in_range(r) && in_range(v);
      if ((same >> mine) & 1) v = 1.0;
      if (__all_sync(0xffffffffu, ok)) {
        if (k0 + mine < kept) acc += sh.slot_mel[k0 + mine] * v;
      } else {
#pragma unroll 1
        for (int e = 0; e < 4 && k0 + e < kept; ++e) {
          const int k = k0 + e, t = sh.slot_term[k];
          int site[4], d[4], ns = 0;
          if (t >= 0) {
            const int8_t *xpv =
                op.x_prime + (((int64_t)t * op.max_rows + sh.row[t]) * op.max_conns +
                              sh.slot_col[k]) * S;
            for (int q = 0; q < op.acting_size[t]; ++q) {
              const int st = op.acting_on[t * S + q];
              const int dv = (int)xpv[q] - (int)sh.xs[st];
              if (dv != 0) {
                site[ns] = st;
                d[ns++] = dv;
              }
            }
          }
          const double w = ns ? exp(slow_log_ratio(params, N, M, sh.xs, site, d, ns)) : 1.0;
          if (mine == e) acc += sh.slot_mel[k] * w;
        }
      }
    }
    // one lane of each group carries its sums
    acc = (lane & 7) == 0 ? acc : 0.0;
    const double e = block_sum(acc, red);
    if (tid == 0) eloc[b] = e;
    __syncthreads();
  }
}

static int sm_count() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

static int launch_flip_tables(cudaStream_t st, const double *params, int N, int M, double *ws) {
  flip_tables_kernel<<<N + 1, 256, 0, st>>>(params, N, M, ws);
  return check_launch("flip tables");
}

template <int NS>
static int launch_local(cudaStream_t st, const double *params, int N, int M, const int8_t *x,
                        int64_t n, const vmck_local_op &op, const FlipTables &tab, double *eloc,
                        size_t smem) {
  if (smem > 48 * 1024)
    VMCK_CUDA(cudaFuncSetAttribute(eloc_local_f64_kernel<NS>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t grid = std::min<int64_t>(n, (int64_t)sm_count() * 32);
  eloc_local_f64_kernel<NS><<<(unsigned)grid, EF_THREADS, smem, st>>>(params, N, M, x, n, op, tab,
                                                                      eloc);
  return check_launch("rbm_eloc_local_f64");
}

}  // namespace vmck

using namespace vmck;

extern "C" int64_t vmck_rbm_eloc_f64_workspace_size(int32_t N, int32_t M) {
  return flip_table_len(N, M);
}

extern "C" int vmck_rbm_eloc_ising_f64(vmck_stream s, const double *params, int32_t N, int32_t M,
                                       const int8_t *x, int64_t n, const int32_t *edges,
                                       int32_t n_edges, double h, double J, double *eloc,
                                       double *workspace, int64_t workspace_len) {
  VMCK_REQUIRE(params && x && eloc && workspace && N > 0 && M > 0 && n >= 0,
               "rbm_eloc_ising_f64 arguments");
  VMCK_REQUIRE(n_edges == 0 || edges, "edges");
  VMCK_REQUIRE(workspace_len >= flip_table_len(N, M), "rbm_eloc_ising_f64 workspace too small");
  if (n == 0) return VMCK_OK;
  cudaStream_t st = as_stream(s);
  const size_t smem = (size_t)EF_SAMPLES * M * 8 + align16((size_t)EF_SAMPLES * N);
  if (smem > 200 * 1024)  // four samples' rho do not fit: one log_cosh per hidden unit
    return vmck_rbm_eloc_ising(s, VMCK_F64, params, N, M, x, n, edges, n_edges, h, J, eloc,
                               nullptr);
  int rc;
  if (h != 0.0 && (rc = launch_flip_tables(st, params, N, M, workspace))) return rc;
  if (smem > 48 * 1024)
    VMCK_CUDA(cudaFuncSetAttribute(eloc_ising_f64_kernel,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t grid = std::min<int64_t>((n + EF_SAMPLES - 1) / EF_SAMPLES,
                                         (int64_t)sm_count() * 32);
  eloc_ising_f64_kernel<<<(unsigned)grid, EF_THREADS, smem, st>>>(
      params, N, M, x, n, edges, n_edges, h, J, flip_tables(workspace, N, M), eloc);
  return check_launch("rbm_eloc_ising_f64");
}

extern "C" int vmck_rbm_eloc_local_f64(vmck_stream s, const double *params, int32_t N, int32_t M,
                                       const int8_t *x, int64_t n, const vmck_local_op *op,
                                       double *eloc, double *workspace, int64_t workspace_len) {
  VMCK_REQUIRE(params && x && eloc && op && workspace && N > 0 && M > 0 && n >= 0,
               "rbm_eloc_local_f64 arguments");
  int rc = validate_local_op(*op);
  if (rc) return rc;
  VMCK_REQUIRE(op->n_sites == N, "operator and model sizes differ");
  VMCK_REQUIRE(workspace_len >= flip_table_len(N, M), "rbm_eloc_local_f64 workspace too small");
  if (n == 0) return VMCK_OK;
  cudaStream_t st = as_stream(s);
  const size_t smem = local_conn_shared_bytes(*op) + (size_t)M * 8 + 16;
  // the limit of vmck_rbm_eloc_local, whose kernel keeps two vectors
  VMCK_REQUIRE(smem + (size_t)M * 8 <= 200 * 1024,
               "operator / M too large for the fused local-energy kernel");
  if ((rc = launch_flip_tables(st, params, N, M, workspace))) return rc;
  const FlipTables tab = flip_tables(workspace, N, M);
  if (op->max_sites <= 1) return launch_local<1>(st, params, N, M, x, n, *op, tab, eloc, smem);
  if (op->max_sites == 2) return launch_local<2>(st, params, N, M, x, n, *op, tab, eloc, smem);
  return launch_local<4>(st, params, N, M, x, n, *op, tab, eloc, smem);
}
