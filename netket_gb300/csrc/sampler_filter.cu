// Metropolis sweeps with a filtered decision: the Local and Exchange rules for an
// RBM whose weights, as FP32, fit in one SM's shared memory.
//
// A proposal is accepted iff ln u < 2 s + corr, s the change of logpsi.  The
// decision needs s only as far as it separates ln u from 2 s + corr, so s is
// first formed cheaply, with a bound eps on its distance from what the plain
// kernel (metropolis_kernel) computes:
//   s = sum_j (|t_j| - |theta_j|) + ln prod_j (1 + e^(-2|t_j|)) / (1 + e^(-2|theta_j|)),
// theta and t = theta + delta in FP32: two FMAs, one exponential on the MUFU
// unit, one addition and one product per hidden unit, one logarithm per lane.
// Only when |ln u - (2 s + corr)| <= eps (about 1 proposal in 200 at M = 400) is
// s formed again exactly as metropolis_kernel<T> forms it, from the same values
// in the same order (FP32), or in FP64 from the parameters.  Every decision, and
// so every sample, is the plain kernel's.  (FP64: up to the rounding of theta,
// 1e-16, which the plain kernel carries from proposal to proposal within a sweep
// and the exact path here forms from scratch.)
//
// One warp drives one chain; lane l holds hidden units l + 32 r in registers.
// FP32: theta is the plain kernel's, recomputed once per sweep.  FP64: theta is a
// double-float pair of the sum over the FP32-rounded weights (the rounding is
// part of eps), so an accepted move costs no FP64 operation: GB300 issues two of
// them per clock and SM, and the plain kernel spent about 50 per hidden unit and
// proposal (FP64 pipe 85 % busy, ncu).
//
// What else a proposal needs is kept in registers: the spins and the hoppable
// clusters as bit words (word l in lane l), the clusters' prefix counts (rebuilt
// after an accepted move), and the random words of 32 proposals, which the lanes
// compute together.  Swapping the unequal spins u and v turns every hoppable
// cluster that holds exactly one of them into a non-hoppable one and back, so
// with inc_i the bit words of the clusters at site i the new set is
// hop ^ inc_u ^ inc_v (clusters holding both cancel).
//
// Measured (GB300, MCState.sample, before -> now; before = one log_cosh per hidden
// unit and proposal): FP64 Local, N = 64, M = 128, 1,024 chains x 9 sweeps 14.1 ->
// 0.26 ms; FP64 Exchange, N = 36, M = 72, 1,024 chains 7.77 -> 0.23 ms; FP32
// Exchange, 10 x 10 J1-J2, M = 400, 4,096 chains 3.45 -> 1.10 ms (about 880 warp
// instructions per proposal before, 312 now).
#include <algorithm>

#include "filter_common.cuh"

namespace vmck {

namespace {

constexpr int FS_MAX_WARPS = 28;

template <typename T, int R>
constexpr int max_warps() {  // by registers: theta, t (and the low parts)
  return sizeof(T) == 4 ? FS_MAX_WARPS : (R <= 8 ? 24 : 20);
}

// Row layout of the shared weights: hidden unit l + 32 r at quad r / 4 of lane l
// (one 16-byte load serves four r), the R % 4 last r behind them.
template <int R>
__device__ __forceinline__ int row_pos(int j) {
  constexpr int Q = R / 4;
  const int l = j & 31, r = j >> 5;
  return r < 4 * Q ? (r >> 2) * 128 + 4 * l + (r & 3) : Q * 128 + (r - 4 * Q) * 32 + l;
}
template <int R>
__device__ __forceinline__ void load_row(const float *row, int lane, float (&w)[R]) {
  constexpr int Q = R / 4;
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const float4 v = *reinterpret_cast<const float4 *>(row + q * 128 + 4 * lane);
    w[4 * q] = v.x;
    w[4 * q + 1] = v.y;
    w[4 * q + 2] = v.z;
    w[4 * q + 3] = v.w;
  }
#pragma unroll
  for (int r = 4 * Q; r < R; ++r) w[r] = row[Q * 128 + (r - 4 * Q) * 32 + lane];
}

// Shared-memory layout (bytes from the start).
struct FilterSmem {
  size_t bias, vis, l1, logtab, cl, inc, total;
};
__host__ __device__ inline FilterSmem filter_smem(int rule, int N, int R, int C) {
  FilterSmem s;
  const size_t row = (size_t)32 * R * 4;
  s.bias = N * row;
  s.vis = s.bias + row;
  s.l1 = s.vis + 4 * (size_t)N;
  s.logtab = s.l1 + 4 * (size_t)N;
  s.cl = s.logtab + (rule == 1 ? 4 * (size_t)(C + 1) : 0);
  s.inc = s.cl + (rule == 1 ? 4 * (size_t)C : 0);
  s.total = s.inc + (rule == 1 ? 4 * (size_t)N * ((C + 31) / 32) : 0);
  return s;
}

}  // namespace

template <typename T, int RULE, int R>
__global__ void __launch_bounds__(32 * max_warps<T, R>(), 1)
    metropolis_filtered_kernel(SweepArgs A, int wpb) {
  constexpr bool F64 = sizeof(T) == 8;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int N = A.N, M = A.M, C = A.C;
  const int nwords = (C + 31) >> 5;
  const FilterSmem lay = filter_smem(RULE, N, R, C);
  float *Ws = reinterpret_cast<float *>(smem_raw);
  float *bs = reinterpret_cast<float *>(smem_raw + lay.bias);
  float *as = reinterpret_cast<float *>(smem_raw + lay.vis);
  float *l1 = reinterpret_cast<float *>(smem_raw + lay.l1);
  float *logtab = reinterpret_cast<float *>(smem_raw + lay.logtab);
  uint32_t *cl = reinterpret_cast<uint32_t *>(smem_raw + lay.cl);
  uint32_t *inc = reinterpret_cast<uint32_t *>(smem_raw + lay.inc);
  __shared__ float all_l1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const T *params = static_cast<const T *>(A.params);
  {  // stage the parameters (FP32), clusters and incidence words
    for (int e = tid; e < (N + 1) * 32 * R; e += blockDim.x) {
      const int i = e / (32 * R), j = e - i * (32 * R);
      // row N is the hidden bias; units beyond M are zero
      const float v = j < M ? (float)(i < N ? params[M + (int64_t)i * M + j] : params[j]) : 0.0f;
      Ws[i * (32 * R) + row_pos<R>(j)] = v;
    }
    for (int i = tid; i < N; i += blockDim.x) as[i] = (float)params[M + (int64_t)N * M + i];
    if (tid == 0) all_l1 = 0.0f;
    if (RULE == 1) stage_rule(A, nwords, logtab, cl, inc);
    __syncthreads();
    for (int i = warp; i <= N; i += (int)(blockDim.x >> 5)) {
      float w[R], s = 0.0f;
      load_row<R>(Ws + i * (32 * R), lane, w);
#pragma unroll
      for (int r = 0; r < R; ++r) s += fabsf(w[r]);
      s = warp_sum(s);
      if (i < N) s += fabsf(as[i]);
      if (lane == 0) {
        if (i < N) l1[i] = s;
        atomicAdd(&all_l1, s);  // a bound: the order of the sum does not matter
      }
    }
    __syncthreads();
  }
  const int b = blockIdx.x * wpb + warp;
  if (warp >= wpb || b >= A.B) return;  // the other warps only helped staging
  const RuleTables tables{logtab, cl, inc, C, nwords};
  ChainBits<RULE> ch;
  ch.load(A.sigma + (int64_t)b * N, N, tables);

  float th[R], lo[F64 ? R : 1];
  float sum_abs = 0.0f, log_prod = 0.0f;  // this lane's sum |theta|, lg2 prod (1 + e)
  auto totals = [&](const float (&v)[R], float &sa, float &lp) {
    float s = 0.0f, p = 1.0f;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float m = fabsf(v[r]);
      s += m;
      p = fmaf(p, ex2_fast(-2.885390043f * m), p);
    }
    sa = s;
    lp = __log2f(p);
  };
  // theta = b + x W: FP32 in the plain kernel's order, FP64 as double-float sums
  auto recompute = [&]() {
    load_row<R>(bs, lane, th);
    if (F64) {
#pragma unroll
      for (int r = 0; r < R; ++r) lo[r] = 0.0f;
    }
    for (int w = 0; 32 * w < N; ++w) {
      const uint32_t bits = __shfl_sync(0xffffffffu, ch.xb, w);
      const int i1 = min(32, N - 32 * w);
      for (int q = 0; q < i1; ++q) {
        const float x = (bits >> q) & 1u ? 1.0f : -1.0f;
        float wr[R];
        load_row<R>(Ws + (32 * w + q) * (32 * R), lane, wr);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if (F64) {
            const df32 s = df_two_sum(th[r], x * wr[r]);
            th[r] = s.hi;
            lo[r] += s.lo;
          } else {
            th[r] += x * wr[r];
          }
        }
      }
    }
    if (F64) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const df32 s = df_quick_two_sum(th[r], lo[r]);
        th[r] = s.hi;
        lo[r] = s.lo;
      }
    }
    totals(th, sum_abs, log_prod);
  };
  if (F64) recompute();

  const float eps0 = 2.0f * (32 * R * (A_UNIT + (F64 ? 0.0f : B_UNIT)) + FIXED +
                             (F64 ? 6.0f * ROUND * all_l1 : 0.0f)) + LN_U;
  const float eps_s = 2.0f * (2 * R + 16) * ROUND;
  const float eps_d = F64 ? 0.0f : 2.0f * 2.0f * (R + 6) * 1.5f * ROUND;
  const int total = A.n_discard + A.L;
  int64_t acc_count = 0;
  for (int step = 0; step < total; ++step) {
    if (!F64) recompute();
    RandomWords<F64> rnd;
    for (int p = 0; p < A.sweep; ++p) {
      if ((p & 31) == 0) rnd.draw(A, A.counter + (uint64_t)step * A.sweep + p, b);
      Proposal pr;
      if (!ch.propose(__shfl_sync(0xffffffffu, rnd.x, p & 31), N, tables, pr)) continue;
      const int su = pr.su, sv = pr.sv;
      const float corr = pr.corr;
      const int du = ch.up(su) ? -2 : 2;  // an Exchange partner changes by -du
      const float fu = (float)du;
      float t[R];
      {
        float w[R];
        load_row<R>(Ws + su * (32 * R), lane, w);
#pragma unroll
        for (int r = 0; r < R; ++r) t[r] = th[r] + fu * w[r];
        if (RULE == 1) {
          load_row<R>(Ws + sv * (32 * R), lane, w);
#pragma unroll
          for (int r = 0; r < R; ++r) t[r] -= fu * w[r];
        }
      }
      float new_abs, new_prod;
      totals(t, new_abs, new_prod);
      const float d = (new_abs - sum_abs) + 0.693147181f * (new_prod - log_prod);
      const bool far = !(fabsf(d) < SUM_MAX);
      const int sum = __reduce_add_sync(0xffffffffu, far ? 0 : __float2int_rn(d * 524288.0f));
      // sum |t| + |theta|, rounded up (a lane's part capped: it is far beyond that)
      const int size = __reduce_add_sync(
          0xffffffffu, __float2int_ru(fminf(new_abs + sum_abs, 1e7f)));
      float s = (float)sum * SUM_UNIT + fu * as[su];
      if (RULE == 1) s -= fu * as[sv];
      const float x = 2.0f * s + corr;
      float eps = eps0 + eps_s * (float)size + X_REL * (fabsf(x) + fabsf(corr));
      if (!F64) eps += eps_d * (RULE == 1 ? l1[su] + l1[sv] : l1[su]);
      const float margin = __shfl_sync(0xffffffffu, rnd.ln_u, p & 31) - x;
      bool accept = margin < 0.0f;
      if (!(fabsf(margin) > eps) || __any_sync(0xffffffffu, far)) {
        // too close to call: the plain kernel's own evaluation
        if constexpr (F64) {
          accept = exact_accept_f64<(R > 1)>(static_cast<const double *>(A.params), N, M, ch.xb, su,
                                    sv, du, ch.hop, pr.hop_new,
                                    __shfl_sync(0xffffffffu, rnd.y, p & 31),
                                    __shfl_sync(0xffffffffu, rnd.z, p & 31));
        } else {
          float e = 0.0f;
#pragma unroll
          for (int r = 0; r < R; ++r)
            if (lane + 32 * r < M) e += log_cosh_fast(t[r]) - log_cosh_fast(th[r]);
          e = warp_sum(e);
          e += fu * as[su];
          if (RULE == 1) e += -fu * as[sv];
          const float dlp = 2.0f * e;
          accept = u01f(__shfl_sync(0xffffffffu, rnd.y, p & 31)) < expf(dlp + corr);
        }
      }
      if (accept) {
        if constexpr (F64) {
          float w[R];
          load_row<R>(Ws + su * (32 * R), lane, w);
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const df32 v = df_two_sum(th[r], fu * w[r]);
            th[r] = v.hi;
            lo[r] += v.lo;
          }
          if (RULE == 1) {
            load_row<R>(Ws + sv * (32 * R), lane, w);
#pragma unroll
            for (int r = 0; r < R; ++r) {
              const df32 v = df_two_sum(th[r], -fu * w[r]);
              th[r] = v.hi;
              lo[r] += v.lo;
            }
          }
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const df32 v = df_quick_two_sum(th[r], lo[r]);
            th[r] = v.hi;
            lo[r] = v.lo;
          }
        } else {
#pragma unroll
          for (int r = 0; r < R; ++r) th[r] = t[r];
        }
        sum_abs = new_abs;
        log_prod = new_prod;
        ch.apply(pr);
        ++acc_count;
      }
    }
    if (step >= A.n_discard)
      ch.store(A.samples + ((int64_t)b * A.L + (step - A.n_discard)) * N, N);
  }
  T logpsi;
  if constexpr (F64) {
    logpsi = final_logpsi_f64(static_cast<const double *>(A.params), N, M, ch.xb);
  } else {
    recompute();
    float part = 0.0f;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (lane + 32 * r < M) part += log_cosh_fast(th[r]);
    for (int w = 0; 32 * w < N; ++w) {
      const uint32_t bits = __shfl_sync(0xffffffffu, ch.xb, w);
      const int i = 32 * w + lane;
      if (i < N) part += ((bits >> lane) & 1u ? 1.0f : -1.0f) * as[i];
    }
    logpsi = warp_sum(part);
  }
  ch.store(A.sigma + (int64_t)b * N, N);
  if (lane == 0) {
    A.log_prob[b] = 2.0 * (double)logpsi;
    A.n_accepted[b] += acc_count;
  }
}

// Registers per lane for the hidden layer: 32 R >= M.  Thirteen beside sixteen: what a
// proposal issues and the shared memory of a row follow R (10 x 10 J1-J2, 4,096 chains, kernel
// time with R = 13 / 16, us: M = 400 Exchange FP32 1,089 / 1,230, FP64 2,959 / 3,382, Local 655 /
// 772, 2,922 / 3,114; M = 260 Exchange FP64 2,729 / 3,259, Local FP32 659 / 777).
static int filter_regs(int M) {
  for (int r : {1, 2, 4, 8, 13, 16})
    if (M <= 32 * r) return r;
  return 0;
}

// Spins and clusters are one bit word per lane; the weights' rows and the tables
// have to fit the SM's shared memory.
bool filtered_fits(int rule, int N, int M, int C) {
  const int R = filter_regs(M);
  return R > 0 && N <= 1024 && (rule == 0 || C <= 1024) &&
         filter_smem(rule, N, R, rule == 1 ? C : 0).total <= FS_SMEM_MAX;
}

template <typename T, int RULE, int R>
static int launch_filtered_as(cudaStream_t st, const SweepArgs &a) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // as few waves as the registers allow, each with an even share of the chains
  const int most = max_warps<T, R>();
  const int waves = (a.B + sms * most - 1) / (sms * most);
  const int wpb = (a.B + sms * waves - 1) / (sms * waves);
  const size_t smem = filter_smem(RULE, a.N, R, a.C).total;
  VMCK_CUDA(cudaFuncSetAttribute(metropolis_filtered_kernel<T, RULE, R>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  // at least eight warps stage the weights
  metropolis_filtered_kernel<T, RULE, R>
      <<<(a.B + wpb - 1) / wpb, 32 * std::max(wpb, 8), smem, st>>>(a, wpb);
  return check_launch("metropolis_sample (filtered)");
}

template <typename T, int RULE>
static int launch_filtered_r(cudaStream_t st, const SweepArgs &a) {
  switch (filter_regs(a.M)) {
    case 1: return launch_filtered_as<T, RULE, 1>(st, a);
    case 2: return launch_filtered_as<T, RULE, 2>(st, a);
    case 4: return launch_filtered_as<T, RULE, 4>(st, a);
    case 8: return launch_filtered_as<T, RULE, 8>(st, a);
    case 13: return launch_filtered_as<T, RULE, 13>(st, a);
    default: return launch_filtered_as<T, RULE, 16>(st, a);
  }
}

int launch_filtered(cudaStream_t st, int dtype, int rule, const SweepArgs &args) {
  SweepArgs a = args;
  if (rule == 0) a.C = 0;
  if (dtype == VMCK_F64)
    return rule == 0 ? launch_filtered_r<double, 0>(st, a) : launch_filtered_r<double, 1>(st, a);
  return rule == 0 ? launch_filtered_r<float, 0>(st, a) : launch_filtered_r<float, 1>(st, a);
}

}  // namespace vmck
