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
// What bounds it: GB300 issues two FP64 operations per clock and SM, and 128 integer
// ones.  So the factors of one- and two-site flips, divided by 1 + rho, are formed in
// 64-bit fixed point: p + q u with p = 1 / (1 + rho) and q = 1 - p in units of 2^-63
// and u = e^(-2 delta) < 8 in units of 2^-60, and so is their product over a lane's
// hidden units, in units of 2^-(63 - S) where 2^S bounds it (S from the sums of |4 W|
// of the row, at most 8): about 24 integer instructions where FP64 takes two operations
// of 16 clocks per warp.  A factor is off by 2^-60 (2^-56 for two sites), a product by
// less than a unit without a preferred sign (times_factor): below FP64's roundings while the
// lane's product is about 1, as it is for weights of either sign.  It can fall to 2^-S,
// where a unit is 2^-(63 - 2 S) of it: 2^-47 at S = 8, eight hidden units that all pull one
// way.  A lane's product is scaled anew every eight (four, two) factors, as its bound asks,
// and the lanes' products meet as 64-bit floating-point numbers in integer registers.
// Error of an energy, rms (one log_cosh per hidden unit and flip before), N = 16 .. 100, M =
// 16 .. 256: weights of 0.01 to 0.1 7e-17 to 6e-16 (2e-16 to 1.4e-15); all weights of one
// sign, 0.05 to 0.25, hidden biases of -3, 0 and 3 at most 1.5e-15 (6.7e-15).  Rows with an
// entry |W| >= 0.52, and samples whose theta is not finite, take the FP64 form.  theta and q
// come from integer sums too (theta_q_f64).
//
// A product leaves the double range only where the ratio, or a partial product
// of it, does; such an element is formed again as the difference of log_cosh sums
// (slow_log_ratio), which is also the path of a non-finite parameter.
#include <algorithm>

#include "common.cuh"
#include "localop.cuh"
#include "signsum.cuh"

namespace vmck {

constexpr int EF_THREADS = 128, EF_WARPS = EF_THREADS / 32;  // LocalOperator
constexpr int EF_S_MAX = 8;
constexpr int EF_DIRECT = 12;
// Samples whose theta and q (16 bytes per hidden unit) are kept at once: 512 MB at most
__host__ __device__ inline int64_t ef_chunk(int M, int64_t n) {
  const int64_t most = M <= 2048 ? 16384 : (1ll << 25) / M;
  return n < most ? n : (most > 0 ? most : 1);
}

// Tables of the call: up[i, j] = exp(-4 W_ij) and down[i, j] = exp(4 W_ij), the
// factor e^(-2 delta) of turning spin i up (x = -1 -> 1) and down, for i < N and
// ones in row N (a site left alone); rup[i] = exp(2 (sum_j W_ij + a_i)) and rdown
// its inverse, the factors of a flip that do not depend on theta.  uup and udown hold
// up and down in units of 2^-60.  bound[i] = {S8, S4, S2, -}: a lane's product of 8 (4,
// 2) factors of a flip of site i, divided by 1 + rho, is within 2^-S and 2^S; 255 where
// an entry has no fixed-point form.  theta and q hold a chunk of samples.
struct FlipTables {
  const double *up, *down;    // (N + 1) x M
  const double *rup, *rdown;  // N
  const u64 *uup, *udown;     // (N + 1) x M
  const uchar4 *bound;        // N + 1
  double *theta;              // samples x M
  u64 *q;                     // samples x M (q_units)
};

__host__ __device__ inline int64_t flip_table_len(int N, int M, int64_t n) {
  return 4 * (int64_t)(N + 1) * M + 2 * N + (N + 2) / 2 + 2 * ef_chunk(M, n) * M;
}

// n: samples of a chunk
__host__ __device__ inline FlipTables flip_tables(double *ws, int N, int M, int64_t n) {
  const int64_t w = (int64_t)(N + 1) * M;
  double *bound = ws + 4 * w + 2 * N, *theta = bound + (N + 2) / 2;
  return FlipTables{ws,
                    ws + w,
                    ws + 4 * w,
                    ws + 4 * w + N,
                    reinterpret_cast<const u64 *>(ws + 2 * w),
                    reinterpret_cast<const u64 *>(ws + 3 * w),
                    reinterpret_cast<const uchar4 *>(bound),
                    theta,
                    reinterpret_cast<u64 *>(theta + n * M)};
}

// one block per row of the tables; 256 threads: warp c of a pass holds the c-th of the
// eight factors that a lane multiplies
__global__ void __launch_bounds__(256) flip_tables_kernel(const double *__restrict__ params, int N,
                                                          int M, double *__restrict__ ws) {
  __shared__ float size[8][32];
  __shared__ uint32_t largest[8];
  __shared__ long long part[2][8];
  const int64_t w = (int64_t)(N + 1) * M;
  const FlipTables tab = flip_tables(ws, N, M, 0);
  const int i = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double *row = params + M + (int64_t)i * M;
  uint32_t most = 0u;  // size of the row's largest entry
  float s8 = 0.0f, s4 = 0.0f, s2 = 0.0f;
  bool fits = true;
  for (int j0 = 0; j0 < M; j0 += 256) {
    const int j = j0 + threadIdx.x;
    const double v = i < N && j < M ? row[j] : 0.0;
    if (j < M) {
      const double u = exp(-4.0 * v), d = exp(4.0 * v);
      ws[(int64_t)i * M + j] = u;
      ws[w + (int64_t)i * M + j] = d;
      fits &= u < 8.0 && d < 8.0;
      const_cast<u64 *>(tab.uup)[(int64_t)i * M + j] = __double2ull_rn(u * 0x1p60);
      const_cast<u64 *>(tab.udown)[(int64_t)i * M + j] = __double2ull_rn(d * 0x1p60);
      most = max(most, size_word(v));
    }
    size[warp][lane] = 5.7708f * fabsf((float)v);  // 4 |W| log2 e, rounded up
    __syncthreads();
    if (warp == 0) {
      float a[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        a[c] = size[2 * c][lane] + size[2 * c + 1][lane];
        s2 = fmaxf(s2, a[c]);
      }
      s4 = fmaxf(s4, fmaxf(a[0] + a[1], a[2] + a[3]));
      s8 = fmaxf(s8, (a[0] + a[1]) + (a[2] + a[3]));
    }
    __syncthreads();
  }
  most = __reduce_max_sync(0xffffffffu, most);
  if (lane == 0) largest[warp] = most;
  fits = __syncthreads_and(fits);
  if (warp == 0) {
    // (a small margin for the rounding of the sums)
    auto level = [&](float s) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s = fmaxf(s, __shfl_xor_sync(0xffffffffu, s, o));
      return fits && s < 200.0f ? (unsigned char)ceilf(s + 0.01f) : (unsigned char)255;
    };
    uchar4 b = make_uchar4(level(s8), level(s4), level(s2), 0);
    if (i == N) b = make_uchar4(0, 0, 0, 0);
    if (lane == 0) const_cast<uchar4 *>(tab.bound)[i] = b;
  }
  if (i == N) return;
  // The row's sum can be far beyond the log-ratios that it is part of (entries of one sign),
  // and its exponential takes its absolute error.  Where it may be (up to 1 the exponential's
  // own rounding is more): an integer sum as in signed_rows_kernel, and one of what its
  // roundings leave (half a unit up in a tie, M times with one sign).
#pragma unroll
  for (int k = 0; k < 8; ++k) most = max(most, largest[k]);
  const int e = most >> 20, bits = sum_bits(M);
  const bool whole = exponent_fits(e) && (double)M * __hiloint2double((int)most, 0) > 1.0;
  const double unit = unit_of(e, bits);
  long long units[2] = {0, 0};
  double plain = 0.0;
  for (int j = threadIdx.x; j < M; j += 256) {
    if (whole) {
      const long long q = to_units(row[j], e, bits);
      units[0] += q;
      units[1] += to_units(fma((double)q, -unit, row[j]), e - bits, bits);
    } else {
      plain += row[j];
    }
  }
  if (whole) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int k = 0; k < 2; ++k) units[k] += __shfl_xor_sync(0xffffffffu, units[k], o);
  } else {
    units[0] = __double_as_longlong(warp_sum(plain));
  }
  if (lane < 2) part[lane][warp] = lane ? units[1] : units[0];
  __syncthreads();
  if (threadIdx.x > 0) return;
  double sum = 0.0, low = 0.0;  // the second: what the first leaves
  const double a = params[M + (int64_t)N * M + i];
  if (whole) {
    for (int k = 1; k < 8; ++k) {
      units[0] += part[0][k];
      units[1] += part[1][k];
    }
    sum = (double)units[0];
    low = (double)(units[0] - (long long)sum) * unit + (double)units[1] * unit_of(e - bits, bits);
    sum = two_sum(sum * unit, a, low);
  } else {
    for (int k = 0; k < 8; ++k) sum += __longlong_as_double(part[0][k]);
    sum += a;
  }
  const double up = exp(2.0 * sum), down = exp(-2.0 * sum);
  ws[4 * w + i] = fma(up, 2.0 * low, up);
  ws[4 * w + N + i] = fma(down, -2.0 * low, down);
}

// x * W without a conversion of x: the sign bit of W flipped where x = -1
__device__ __forceinline__ double signed_by(double w, int x) {
  return __hiloint2double(__double2hiint(w) ^ (x & 0x80000000), __double2loint(w));
}

// theta of the sample xs[i * ldx] for one hidden unit
__device__ __forceinline__ double theta_of(const double *__restrict__ params, int N, int M,
                                           const int8_t *xs, int ldx, int j) {
  double th = params[j];
  const double *W = params + M + j;
#pragma unroll 4
  for (int i = 0; i < N; ++i) th += signed_by(__ldg(W + (int64_t)i * M), (int)xs[i * ldx]);
  return th;
}

// Log-ratio of one element as the difference of log_cosh sums, by the warp, from
// scratch (theta is not kept): sites site[q] with change d[q].
__device__ __noinline__ double slow_log_ratio(const double *__restrict__ params, int N, int M,
                                              const int8_t *xs, int ldx, const int *site,
                                              const int *d, int ns) {
  const int lane = threadIdx.x & 31;
  const double *W = params + M, *a = W + (int64_t)N * M;
  double s = 0.0;
  for (int j = lane; j < M; j += 32) {
    const double th = theta_of(params, N, M, xs, ldx, j);
    double t = th;
    for (int q = 0; q < ns; ++q) t += (double)d[q] * W[(int64_t)site[q] * M + j];
    s += log_cosh(t) - log_cosh(th);
  }
  s = warp_sum(s);
  for (int q = 0; q < ns; ++q) s += (double)d[q] * a[site[q]];
  return s;
}

// 2^-962 <= v < 2^963 (about 1e-290 to 1e290), by the exponent
// (a product outside, or not positive, is formed again in the log domain)
__device__ __forceinline__ bool in_range(double v) {
  return (uint32_t)__double2hiint(v) - 0x03d00000u < 0x7c200000u - 0x03d00000u;
}

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

__device__ __forceinline__ UFloat warp_prod4(const UFloat (&v)[4]) {
  const int lane = threadIdx.x & 31;
  const bool h = lane & 16, g = lane & 8;
  const UFloat a = (h ? v[2] : v[0]) * shfl_xor(h ? v[0] : v[2], 16);
  const UFloat b = (h ? v[3] : v[1]) * shfl_xor(h ? v[1] : v[3], 16);
  UFloat r = (g ? b : a) * shfl_xor(g ? a : b, 8);
  r = r * shfl_xor(r, 4);
  r = r * shfl_xor(r, 2);
  return r * shfl_xor(r, 1);
}
// false where it is outside in_range
__device__ __forceinline__ bool to_double(UFloat v, double &d) {
  const double m = __ull2double_rn(v.m);
  d = __hiloint2double(__double2hiint(m) + (v.e << 20), __double2loint(m));
  return v.e > -1000 && v.e < 890;
}

// e^(-2 theta), and NaN for an infinite theta: its sample's products then take the log_cosh
// route, where the ratio is a difference of infinities.
__device__ __forceinline__ double rho_of(double theta) {
  return exp(-2.0 * theta) + (theta - theta);
}

// Product of 1 / (1 + rho_j) over the hidden units j = lane, lane + 32, ...
__device__ __forceinline__ double lane_norm(const double *rho, int M) {
  double v = 1.0;
  for (int j = threadIdx.x & 31; j < M; j += 32) v = fma(v, rho[j], v);
  return 1.0 / v;
}

// p + q u in units of 2^-(B - 1) for u in units of 2^-B: p = (p_offset(lane) - q) >> (64 -
// B), rounded.  q u is rounded for two sites; for one, whose units are finer, it is
// truncated and every second lane adds the unit that two of them lose.
template <int B>
__device__ __forceinline__ u64 p_offset(int lane) {
  return (1ull << 63) + (1ull << (63 - B)) + (B == 60 ? (u64)(lane & 1) << (64 - B) : 0ull);
}
template <int B>
__device__ __forceinline__ u64 factor(u64 q, u64 u, u64 p) {
  uint32_t below;
  const u64 h = mul_high(q, u, below);
  return B == 60 ? h + p : h + p + (below >> 31);
}
// f g for f in any units and g in units of 2^-(B - 1); f < 2^63 units, f g < 2^64 units, g <
// 2^62 units.  The result is truncated and its last bit set (odd = 1): off by less than a
// unit, and by nothing in the mean.  A lane's first product needs neither (odd = 0): f is a
// power of two.  (A correction after the last factor for the half units that the factors
// before it lose is wrong by the later factors: 8e-14 of an energy where the hidden units of a
// lane all pull one way.  Nearest rounding, an addition with carry, takes 2 to 4 % of a
// case's time, this 1 %.)
template <int B>
__device__ __forceinline__ u64 times_factor(u64 f, u64 g, uint32_t odd) {
  uint32_t below;
  const u64 h = mul_high(f, g, below);
  constexpr int s = 65 - B;
  const uint32_t lo = (uint32_t)h, hi = (uint32_t)(h >> 32);
  return (u64)__funnelshift_l(lo, hi, s) << 32 | (__funnelshift_l(below, lo, s) | odd);
}
// A lane's product: f 2^e, f within 2^(63 - 2 s) and 2^63 (s as in FlipTables' bound).
struct LaneProduct {
  u64 f;
  int e;
};
__device__ __forceinline__ LaneProduct lane_one(int s) { return {1ull << (63 - s), s - 63}; }
__device__ __forceinline__ UFloat lane_value(LaneProduct p) { return ufloat(p.f, p.e); }
// ready for further factors
__device__ __forceinline__ LaneProduct lane_renew(LaneProduct p, int s) {
  const UFloat v = lane_value(p);
  return {v.m >> s, v.e + s};
}
// Factors until lane_renew and S of rows with the summed bounds s8, s4, s2 (S >= 1 also for
// elements that change no site: f stays below 2^63); 0: FP64 form
__device__ __forceinline__ int fold_length(int s8, int s4, int s2, int &s) {
  s = max(1, s8 <= EF_S_MAX ? s8 : s4 <= EF_S_MAX ? s4 : s2);
  return s8 <= EF_S_MAX ? 8 : s4 <= EF_S_MAX ? 4 : s2 <= EF_S_MAX ? 2 : 0;
}

// ------------------------------------------------------------ Ising
// One CTA takes S samples (gridDim.y CTAs share their sites): their q in shared memory,
// then each warp takes pairs of sites: one read of the two sites' table rows serves all
// samples, one read of a sample's q both sites, and four products are reduced together
// (warp_prod4).  Lane group e accumulates sample e's (and e + 4's) sum.
// N = 256, M = 256, n = 2,048: 0.34 ms with the tables and theta (products in FP64
// 1.14 ms; one log_cosh per hidden unit and flip, eloc_ising_kernel<double>, 20.1 ms).
// The issue of the integer products bounds it: 50 % of the slots at 16 warps per SM,
// whatever a warp's samples and sites (four, eight; one, two).
template <int S>
constexpr int ising_threads() {
  return S == 8 ? 256 : 128;
}

template <int S>
__global__ void __launch_bounds__(ising_threads<S>(), S == 8 ? 2 : 4) eloc_ising_f64_kernel(
    const double *__restrict__ params, int N, int M, const int8_t *__restrict__ x, int64_t n,
    const int32_t *__restrict__ edges, int n_edges, double h, double J, FlipTables tab,
    double *__restrict__ eloc) {
  constexpr int THREADS = ising_threads<S>(), WARPS = THREADS / 32;
  constexpr int W4 = (S + 3) / 4;  // quartets of samples
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *rho = reinterpret_cast<double *>(smem_raw);  // [sample][M], FP64 form only
  u64 *qs = reinterpret_cast<u64 *>(rho + (size_t)S * M);  // [sample][M]
  int8_t *xs = reinterpret_cast<int8_t *>(qs + (size_t)S * M);  // [site][sample], 4 W4 samples
  __shared__ double red[WARPS][4 * W4];
  __shared__ double norm[4 * W4][32];
  __shared__ int diag[S];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, mine = lane >> 3;
  for (int64_t b0 = (int64_t)blockIdx.x * S; b0 < n; b0 += (int64_t)gridDim.x * S) {
    // the last CTA's missing samples repeat sample n - 1; their results are not stored
    for (int e = tid; e < 4 * W4 * N; e += THREADS) {
      const int s = e / N, i = e - s * N;
      const int64_t b = s < S && b0 + s < n ? b0 + s : n - 1;
      xs[i * 4 * W4 + s] = x[b * N + i];
    }
    if (tid < S) diag[tid] = 0;
    __syncthreads();
    for (int e = tid; e < S * n_edges; e += THREADS) {
      const int s = e / n_edges, q = e - s * n_edges;
      const int same =
          xs[edges[2 * q] * 4 * W4 + s] == xs[edges[2 * q + 1] * 4 * W4 + s] ? 1 : -1;
      atomicAdd(&diag[s], same);  // integers: the order does not matter
    }
    double acc[W4];
#pragma unroll
    for (int w = 0; w < W4; ++w) acc[w] = 0.0;
    if (h != 0.0) {
      bool odd = false;  // something needs the FP64 form
      for (int k = tid; k < N; k += THREADS) odd |= tab.bound[k].z > EF_S_MAX;
      bool finite = true;
      for (int j = tid; j < M; j += THREADS) {
        u64 q[S];
#pragma unroll
        for (int s = 0; s < S; ++s) q[s] = __ldg(tab.q + min(b0 + s, n - 1) * M + j);
#pragma unroll
        for (int s = 0; s < S; ++s) {
          finite &= q[s] <= 1ull << 63;
          qs[s * M + j] = q[s];
        }
      }
      finite = __syncthreads_and(finite);
      odd = __syncthreads_or(odd || !finite);
      if (odd) {
        for (int s = 0; s < S; ++s)
          for (int j = tid; j < M; j += THREADS)
            rho[s * M + j] = rho_of(tab.theta[min(b0 + s, n - 1) * M + j]);
        __syncthreads();
        for (int s = warp; s < S; s += WARPS) norm[s][lane] = lane_norm(rho + s * M, M);
        __syncthreads();
      }
      for (int k0 = 2 * (WARPS * (int)blockIdx.y + warp); k0 < N; k0 += 2 * WARPS * gridDim.y) {
        // site k0 + 1 = N stands for the row of ones
        int bits[2];  // bit s: sample s's spin of site k0 + t is down
        int fold = finite ? 8 : 0, S8 = 0, S4 = 0, S2 = 0, range = 0;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          bits[t] = 0;
          const uchar4 b = tab.bound[k0 + t];
          S8 = max(S8, (int)b.x);
          S4 = max(S4, (int)b.y);
          S2 = max(S2, (int)b.z);
          if (k0 + t < N)
#pragma unroll
            for (int s = 0; s < S; ++s)
              bits[t] |= (xs[(k0 + t) * 4 * W4 + s] < 0) << s;
        }
        if (fold) fold = fold_length(S8, S4, S2, range);
        LaneProduct g[2][4 * W4];
        if (fold) {
          const u64 offset = p_offset<60>(lane);
#pragma unroll
          for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int s = 0; s < 4 * W4; ++s) g[t][s] = lane_one(range);
          const u64 *up = tab.uup + (int64_t)k0 * M, *down = tab.udown + (int64_t)k0 * M;
#pragma unroll 1
          for (int js = 0; js < M; js += 32 * fold) {
            if (js > 0) {
#pragma unroll
              for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int s = 0; s < S; ++s) g[t][s] = lane_renew(g[t][s], range);
            }
            const int je = min(M, js + 32 * fold);
#pragma unroll 1
            for (int j = js + lane; j < je; j += 32) {
              const uint32_t odd = j >= 32;
              u64 u[2][2];
#pragma unroll
              for (int t = 0; t < 2; ++t) {
                u[t][0] = __ldg(down + (int64_t)t * M + j);
                u[t][1] = __ldg(up + (int64_t)t * M + j);
              }
#pragma unroll
              for (int s = 0; s < S; ++s) {
                const u64 q = qs[s * M + j], p = (offset - q) >> 4;
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                  const u64 ut = (bits[t] >> s) & 1 ? u[t][1] : u[t][0];
                  g[t][s].f = times_factor<60>(g[t][s].f, factor<60>(q, ut, p), odd);
                }
              }
            }
          }
        }
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const int k = k0 + t;
          if (k >= N) break;
          double ft[4 * W4];  // FP64 form
          if (!fold) {
#pragma unroll
            for (int s = 0; s < 4 * W4; ++s) ft[s] = s < S ? norm[s][lane] : 1.0;
            const double *eu = tab.up + (int64_t)k * M, *ed = tab.down + (int64_t)k * M;
#pragma unroll 1
            for (int j = lane; j < M; j += 32) {
              const double u = __ldg(eu + j), d = __ldg(ed + j);
#pragma unroll
              for (int s = 0; s < S; ++s)
                ft[s] *= fma(rho[s * M + j], (bits[t] >> s) & 1 ? u : d, 1.0);
            }
          }
#pragma unroll
          for (int w = 0; w < W4; ++w) {
            bool ok = true;
            double r;
            if (fold) {
              UFloat quad[4];
#pragma unroll
              for (int s = 0; s < 4; ++s) quad[s] = lane_value(g[t][4 * w + s]);
              ok = to_double(warp_prod4(quad), r);
            } else {
              const double quad[4] = {ft[4 * w], ft[4 * w + 1], ft[4 * w + 2], ft[4 * w + 3]};
#pragma unroll
              for (int s = 0; s < 4; ++s) ok &= in_range(quad[s]);
              r = warp_prod4(quad);
              ok &= in_range(r);
            }
            const double v = r * ((bits[t] >> (4 * w + mine)) & 1 ? tab.rup[k] : tab.rdown[k]);
            ok &= in_range(v);
            if (__all_sync(0xffffffffu, ok)) {
              acc[w] += v;
            } else {
#pragma unroll 1
              for (int s = 4 * w; s < 4 * w + 4 && s < S; ++s) {
                const int d = (bits[t] >> s) & 1 ? 2 : -2;
                const double lr = slow_log_ratio(params, N, M, xs + s, 4 * W4, &k, &d, 1);
                if (4 * w + mine == s) acc[w] += exp(lr);
              }
            }
          }
        }
      }
    }
#pragma unroll
    for (int w = 0; w < W4; ++w)
      if ((lane & 7) == 0) red[warp][4 * w + mine] = acc[w];
    __syncthreads();
    if (tid < S && b0 + tid < n) {
      double s = 0.0;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) s += red[w][tid];
      const double e = h != 0.0 ? -h * s : 0.0;
      if (gridDim.y == 1)
        eloc[b0 + tid] = e + J * (double)diag[tid];
      else  // two addends and zero: their order does not matter
        atomicAdd(eloc + b0 + tid, blockIdx.y == 0 ? e + J * (double)diag[tid] : e);
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------ LocalOperator
// One CTA per sample: q of the sample, the connected elements
// enumerated in shared memory (local_conn_enumerate), then each warp takes groups
// of four elements: NS table rows each (a site that the element leaves alone
// reads the row of ones), four products reduced together.  10 x 10 Heisenberg, M = 200,
// n = 4,096 (about 100 elements a sample): 0.38 ms with the tables and theta (products in
// FP64 1.02 ms; eloc_local_kernel<double> 14.4 ms).
template <int NS>
__global__ void __launch_bounds__(EF_THREADS) eloc_local_f64_kernel(
    const double *__restrict__ params, int N, int M, const int8_t *__restrict__ x, int64_t n,
    vmck_local_op op, FlipTables tab, double *__restrict__ eloc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  LocalConnShared sh = local_conn_shared_layout(smem_raw, op);
  double *rho = reinterpret_cast<double *>(sh.end);  // FP64 form only
  u64 *qs = reinterpret_cast<u64 *>(rho + M);
  __shared__ double red[32], norm[32];
  const Grp g = cta_grp();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, mine = lane >> 3;
  const int S = op.max_sites;
  const int64_t ones = (int64_t)N * M, down = tab.down - tab.up;
  bool odd = false;  // some row needs the FP64 form
  for (int k = tid; k < N; k += EF_THREADS) odd |= NS * (int)tab.bound[k].z > EF_S_MAX;
  for (int64_t b = blockIdx.x; b < n; b += gridDim.x) {
    for (int i = tid; i < N; i += EF_THREADS) sh.xs[i] = x[b * N + i];
    __syncthreads();
    bool finite = true;
    for (int j = tid; j < M; j += EF_THREADS) {
      const u64 q = __ldg(tab.q + b * M + j);
      finite &= q <= 1ull << 63;
      qs[j] = q;
    }
    finite = __syncthreads_and(finite);
    const bool fp64 = __syncthreads_or(NS > 2 || odd || !finite);
    const int kept = local_conn_enumerate(op, sh, g, true);
    if (fp64) {
      for (int j = tid; j < M; j += EF_THREADS) rho[j] = rho_of(tab.theta[b * M + j]);
      __syncthreads();
      if (warp == 0) norm[lane] = lane_norm(rho, M);
    }
    __syncthreads();
    double acc = 0.0;
    for (int k0 = 4 * warp; k0 < kept; k0 += 4 * EF_WARPS) {
      int64_t row[4][NS];  // of up (the row of down follows) and of uup
      int fix[NS];         // of this lane's element: of rup (rdown follows); -1: none
#pragma unroll
      for (int q = 0; q < NS; ++q) fix[q] = -1;
      int same = 0;  // bit e: element e leaves the configuration as it is (ratio 1)
      int s8 = 0, s4 = 0, s2 = 0;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        int b8 = 0, b4 = 0, b2 = 0;
#pragma unroll
        for (int q = 0; q < NS; ++q) row[e][q] = ones;
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
              row[e][q] = (int64_t)st * M + (d > 0 ? 0 : down);
              if (mine == e) fix[q] = d > 0 ? st : st + N;
              same &= ~(1 << e);
              const uchar4 b = tab.bound[st];
              b8 += b.x;
              b4 += b.y;
              b2 += b.z;
            }
          }
        }
        s8 = max(s8, b8);
        s4 = max(s4, b4);
        s2 = max(s2, b2);
      }
      int range;
      bool ok = true;
      double r;
      const int fold = NS <= 2 && finite ? fold_length(s8, s4, s2, range) : 0;
      if (NS <= 2 && fold) {
        constexpr int B = NS == 1 ? 60 : 56;  // units of an element's u
        const u64 offset = p_offset<B>(lane);
        LaneProduct g[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) g[e] = lane_one(range);
#pragma unroll 1
        for (int js = 0; js < M; js += 32 * fold) {
          if (js > 0) {
#pragma unroll
            for (int e = 0; e < 4; ++e) g[e] = lane_renew(g[e], range);
          }
          const int je = min(M, js + 32 * fold);
#pragma unroll 2
          for (int j = js + lane; j < je; j += 32) {
            const uint32_t odd = j >= 32;
            u64 u[4][NS];
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
              for (int q = 0; q < NS; ++q) u[e][q] = __ldg(tab.uup + row[e][q] + j);
            const u64 q = qs[j], p = (offset - q) >> (64 - B);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              u64 ue = u[e][0];
              if (NS == 2) {
                uint32_t below;
                ue = mul_high(ue, u[e][NS - 1], below);
                ue += below >> 31;
              }
              g[e].f = times_factor<B>(g[e].f, factor<B>(q, ue, p), odd);
            }
          }
        }
        UFloat quad[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) quad[e] = lane_value(g[e]);
        ok = to_double(warp_prod4(quad), r);
      } else {
        double f[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) f[e] = norm[lane];
#pragma unroll(NS <= 2 ? 2 : 1)
        for (int j = lane; j < M; j += 32) {
          const double rj = rho[j];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            double u = __ldg(tab.up + row[e][0] + j);
#pragma unroll
            for (int q = 1; q < NS; ++q) u *= __ldg(tab.up + row[e][q] + j);
            f[e] *= fma(rj, u, 1.0);
          }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) ok &= in_range(f[e]);
        r = warp_prod4(f);
        ok &= in_range(r);
      }
      double v = r;
#pragma unroll
      for (int q = 0; q < NS; ++q)
        if (fix[q] >= 0) v *= tab.rup[fix[q]];
      ok &= in_range(v);
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
          const double w = ns ? exp(slow_log_ratio(params, N, M, sh.xs, 1, site, d, ns)) : 1.0;
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

static int launch_flip_tables(cudaStream_t st, const double *params, int N, int M, double *ws) {
  flip_tables_kernel<<<N + 1, 256, 0, st>>>(params, N, M, ws);
  return check_launch("flip tables");
}

constexpr size_t EF_SMEM_MAX = 200 * 1024;
static size_t ising_smem(int S, int N, int M) {
  return (size_t)S * M * 16 + (size_t)N * (S == 8 ? 8 : 4);
}

template <int S>
static int launch_ising(cudaStream_t st, const double *params, int N, int M, const int8_t *x,
                        int64_t n, const int32_t *edges, int n_edges, double h, double J,
                        const FlipTables &tab, double *eloc, int split) {
  const size_t smem = ising_smem(S, N, M);
  if (smem > 40 * 1024)
    VMCK_CUDA(cudaFuncSetAttribute(eloc_ising_f64_kernel<S>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t grid = std::min<int64_t>((n + S - 1) / S, (int64_t)sm_count() * 32);
  if (split == 2) VMCK_CUDA(cudaMemsetAsync(eloc, 0, (size_t)n * 8, st));
  eloc_ising_f64_kernel<S><<<dim3((unsigned)grid, split), ising_threads<S>(), smem, st>>>(
      params, N, M, x, n, edges, n_edges, h, J, tab, eloc);
  return check_launch("rbm_eloc_ising_f64");
}

template <int NS>
static int launch_local(cudaStream_t st, const double *params, int N, int M, const int8_t *x,
                        int64_t n, const vmck_local_op &op, const FlipTables &tab, double *eloc,
                        size_t smem) {
  if (smem > 40 * 1024)
    VMCK_CUDA(cudaFuncSetAttribute(eloc_local_f64_kernel<NS>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t grid = std::min<int64_t>(n, (int64_t)sm_count() * 32);
  eloc_local_f64_kernel<NS><<<(unsigned)grid, EF_THREADS, smem, st>>>(params, N, M, x, n, op, tab,
                                                                      eloc);
  return check_launch("rbm_eloc_local_f64");
}

}  // namespace vmck

using namespace vmck;

extern "C" int64_t vmck_rbm_eloc_f64_workspace_size(int32_t N, int32_t M, int64_t n) {
  return flip_table_len(N, M, n);
}

extern "C" int vmck_rbm_eloc_ising_f64(vmck_stream s, const double *params, int32_t N, int32_t M,
                                       const int8_t *x, int64_t n, const int32_t *edges,
                                       int32_t n_edges, double h, double J, double *eloc,
                                       double *workspace, int64_t workspace_len) {
  VMCK_REQUIRE(params && x && eloc && workspace && N > 0 && M > 0 && n >= 0,
               "rbm_eloc_ising_f64 arguments");
  VMCK_REQUIRE(n_edges == 0 || edges, "edges");
  VMCK_REQUIRE(workspace_len >= flip_table_len(N, M, n), "rbm_eloc_ising_f64 workspace too small");
  if (n == 0) return VMCK_OK;
  cudaStream_t st = as_stream(s);
  // One log_cosh per hidden unit and flip where that is a single launch of a few us (at most
  // EF_DIRECT warp rounds of flips per SM: n = 16, N = M = 8: 17 us a call, 28 by the three
  // launches below; N = M = 16: 44 and 46; N = M = 24: 52 and 48), and where two samples'
  // vectors or the sites' sign indices do not fit.
  const int64_t rounds = (n + sm_count() - 1) / sm_count() * N * ((M + 31) / 32);
  if (rounds <= EF_DIRECT || ising_smem(2, N, M) > EF_SMEM_MAX || !signed_rows_fit(N))
    return vmck_rbm_eloc_ising(s, VMCK_F64, params, N, M, x, n, edges, n_edges, h, J, eloc,
                               nullptr);
  int rc;
  const int64_t chunk = ef_chunk(M, n);
  const FlipTables tab = flip_tables(workspace, N, M, chunk);
  if (h != 0.0 && (rc = launch_flip_tables(st, params, N, M, workspace))) return rc;
  for (int64_t c = 0; c < n; c += chunk, x += chunk * N, eloc += chunk) {
    const int64_t m = std::min(chunk, n - c);
    if (h != 0.0 && (rc = theta_q_f64(st, params, N, M, x, m, tab.theta, tab.q))) return rc;
    // Eight samples share a read of the tables, four while there are few.  Two CTAs share a
    // sample group's sites where each warp still has two pairs of them: the last round of
    // CTAs is shorter.  N = M = 256, n = 1,500 / 2,048 / 3,000 / 4,096 / 16,384: 350 / 352 /
    // 509 / 626 / 2,038 us with eight and no split, 305 / 340 / 437 / 565 / 1,998 so; N =
    // 32, M = 64: 40 us without the split, 45 with it.
    const int split = h != 0.0 && N >= 64 ? 2 : 1;
    if (m > 16 * (int64_t)sm_count() && ising_smem(8, N, M) <= EF_SMEM_MAX / 2)
      rc = launch_ising<8>(st, params, N, M, x, m, edges, n_edges, h, J, tab, eloc, split);
    else if (ising_smem(4, N, M) <= EF_SMEM_MAX)
      rc = launch_ising<4>(st, params, N, M, x, m, edges, n_edges, h, J, tab, eloc, split);
    else
      rc = launch_ising<2>(st, params, N, M, x, m, edges, n_edges, h, J, tab, eloc, 1);
    if (rc) return rc;
  }
  return VMCK_OK;
}

extern "C" int vmck_rbm_eloc_local_f64(vmck_stream s, const double *params, int32_t N, int32_t M,
                                       const int8_t *x, int64_t n, const vmck_local_op *op,
                                       double *eloc, double *workspace, int64_t workspace_len) {
  VMCK_REQUIRE(params && x && eloc && op && workspace && N > 0 && M > 0 && n >= 0,
               "rbm_eloc_local_f64 arguments");
  int rc = validate_local_op(*op);
  if (rc) return rc;
  VMCK_REQUIRE(op->n_sites == N, "operator and model sizes differ");
  VMCK_REQUIRE(workspace_len >= flip_table_len(N, M, n), "rbm_eloc_local_f64 workspace too small");
  if (n == 0) return VMCK_OK;
  cudaStream_t st = as_stream(s);
  const size_t smem = local_conn_shared_bytes(*op) + (size_t)M * 16 + 16;
  // (as vmck_rbm_eloc_local, whose kernel keeps two vectors too)
  VMCK_REQUIRE(smem <= 200 * 1024,
               "operator / M too large for the fused local-energy kernel");
  if (!signed_rows_fit(N))
    return vmck_rbm_eloc_local(s, VMCK_F64, params, N, M, x, n, op, eloc, nullptr);
  if ((rc = launch_flip_tables(st, params, N, M, workspace))) return rc;
  const int64_t chunk = ef_chunk(M, n);
  const FlipTables tab = flip_tables(workspace, N, M, chunk);
  for (int64_t c = 0; c < n; c += chunk, x += chunk * N, eloc += chunk) {
    const int64_t m = std::min(chunk, n - c);
    if ((rc = theta_q_f64(st, params, N, M, x, m, tab.theta, tab.q))) return rc;
    if (op->max_sites <= 1)
      rc = launch_local<1>(st, params, N, M, x, m, *op, tab, eloc, smem);
    else if (op->max_sites == 2)
      rc = launch_local<2>(st, params, N, M, x, m, *op, tab, eloc, smem);
    else
      rc = launch_local<4>(st, params, N, M, x, m, *op, tab, eloc, smem);
    if (rc) return rc;
  }
  return VMCK_OK;
}
