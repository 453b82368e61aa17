// Filtered Metropolis sweeps (see sampler_filter.cu) for weights that do not fit in
// an SM's shared memory: W is read through L2, theta lives in the warp's shared
// memory and the proposal's t in registers, so that an accepted move reads nothing
// again.
//
// What bounds it is the traffic from L2: a proposal reads two rows of W (16 KB at
// M = 2048 in FP32).  The recomputation of theta once per sweep (FP32, so that
// theta stays the plain kernel's) is therefore shared: all warps of the block
// form theta of six chains at a time, each thread a few hidden units of all six,
// so W is read once for six chains instead of once per chain.  The block's chains
// move through the sweeps together.
//
// 16 x 16 Heisenberg, M = 2,048, 16,384 chains x 9 sweeps (FP32): 171 -> 69 ms; the
// proposals' rows alone are 600 GB, 8.9 TB/s over the launch.  Before: theta in
// shared memory with log_cosh of theta and t per hidden unit and proposal, every
// chain's own recomputation and a second read of the rows on acceptance.
//
// FP64: the FP32 roundings of the weights are formed from the doubles' bits as
// they are read (no FP64-pipe conversion), theta is a double-float pair, and
// nothing is recomputed.
#include <algorithm>

#include "filter_common.cuh"

namespace vmck {

namespace {

constexpr int FL_CHAINS = 6;  // chains whose theta a pass over W forms

template <typename T, int Q>
constexpr int l2_warps() {  // by registers: 4 Q values of t per lane
  return Q >= 16 ? 18 : (Q >= 8 ? 24 : 28);
}

// FP32 value of a double toward zero, by its bits: 0 below the normal range,
// infinity above it (no FP64 instruction; GB300 converts two doubles per clock
// and SM).
__device__ __forceinline__ float f32_of(double v) {
  const uint32_t hi = (uint32_t)__double2hiint(v), lo = (uint32_t)__double2loint(v);
  const uint32_t e = hi & 0x7ff00000u, sign = hi & 0x80000000u;
  uint32_t r = (__funnelshift_l(lo, hi, 3) ^ 0x40000000u) & 0x7fffffffu;
  if (e < 0x38100000u) r = 0u;
  if (e >= 0x47f00000u) r = 0x7f800000u;
  return __uint_as_float(r | sign);
}
__device__ __forceinline__ float f32_of(float v) { return v; }

__device__ __forceinline__ void load4(const float *p, float (&w)[4]) {
  const float4 v = __ldg(reinterpret_cast<const float4 *>(p));
  w[0] = v.x;
  w[1] = v.y;
  w[2] = v.z;
  w[3] = v.w;
}
__device__ __forceinline__ void load4(const double *p, float (&w)[4]) {
  const double2 a = __ldg(reinterpret_cast<const double2 *>(p));
  const double2 b = __ldg(reinterpret_cast<const double2 *>(p) + 1);
  w[0] = f32_of(a.x);
  w[1] = f32_of(a.y);
  w[2] = f32_of(b.x);
  w[3] = f32_of(b.y);
}

// Hidden unit of entry c of a lane's quad q: four neighbours (one wide load) when
// the rows are aligned for it, else lane-strided.
template <bool VEC>
__device__ __forceinline__ int unit(int q, int c, int lane) {
  return VEC ? 128 * q + 4 * lane + c : 128 * q + 32 * c + lane;
}
template <bool VEC, typename T>
__device__ __forceinline__ void load_quad(const T *row, int M, int q, int lane, float (&w)[4]) {
  if (VEC) {
    if (128 * q + 4 * lane < M) {
      load4(row + 128 * q + 4 * lane, w);
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c) w[c] = 0.0f;
    }
  } else {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int j = unit<false>(q, c, lane);
      w[c] = j < M ? f32_of(__ldg(row + j)) : 0.0f;
    }
  }
}

struct L2Smem {
  size_t vis, l1, xs, logtab, cl, inc, theta, per_warp, total;
};
__host__ __device__ inline L2Smem l2_smem(bool f64, int rule, int N, int Q, int C, int wpb) {
  L2Smem s;
  s.vis = 0;
  s.l1 = 4 * (size_t)N;
  s.xs = s.l1 + 4 * (size_t)N;
  // spins of the block's chains as +-1.0f, [site][chain]
  const size_t chains = (size_t)(wpb + FL_CHAINS - 1) / FL_CHAINS * FL_CHAINS;
  s.logtab = s.xs + (f64 ? 0 : 4 * (size_t)N * chains);
  s.cl = s.logtab + (rule == 1 ? 4 * (size_t)(C + 1) : 0);
  s.inc = s.cl + (rule == 1 ? 4 * (size_t)C : 0);
  s.theta = s.inc + (rule == 1 ? 4 * (size_t)N * ((C + 31) / 32) : 0);
  s.theta = (s.theta + 15) & ~size_t(15);
  s.per_warp = (size_t)128 * Q * 4 * (f64 ? 2 : 1);
  s.total = s.theta + wpb * s.per_warp;
  return s;
}

}  // namespace

template <typename T, int RULE, int Q, bool VEC>
__global__ void __launch_bounds__(32 * l2_warps<T, Q>(), 1)
    metropolis_filtered_l2_kernel(SweepArgs A, int wpb) {
  constexpr bool F64 = sizeof(T) == 8;
  constexpr int MP = 128 * Q;  // hidden units, padded with zeros
  constexpr int THREADS = 32 * l2_warps<T, Q>();
  constexpr int JPT = (MP + THREADS - 1) / THREADS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int N = A.N, M = A.M, C = A.C;
  const int nwords = (C + 31) >> 5;
  const L2Smem lay = l2_smem(F64, RULE, N, Q, C, wpb);
  float *as = reinterpret_cast<float *>(smem_raw + lay.vis);
  float *l1 = reinterpret_cast<float *>(smem_raw + lay.l1);
  float *xs = reinterpret_cast<float *>(smem_raw + lay.xs);
  float *logtab = reinterpret_cast<float *>(smem_raw + lay.logtab);
  uint32_t *cl = reinterpret_cast<uint32_t *>(smem_raw + lay.cl);
  uint32_t *inc = reinterpret_cast<uint32_t *>(smem_raw + lay.inc);
  __shared__ float all_l1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int chains = (wpb + FL_CHAINS - 1) / FL_CHAINS * FL_CHAINS;
  const T *params = static_cast<const T *>(A.params);
  const T *W = params + M;
  {
    for (int i = tid; i < N; i += blockDim.x) as[i] = (float)W[(int64_t)N * M + i];
    if (tid == 0) all_l1 = 0.0f;
    if (RULE == 1) stage_rule(A, nwords, logtab, cl, inc);
    __syncthreads();
    for (int i = warp; i <= N; i += THREADS / 32) {
      const T *row = i < N ? W + (int64_t)i * M : params;
      float s = 0.0f;
      for (int j = lane; j < M; j += 32) s += fabsf(f32_of(row[j]));
      s = warp_sum(s);
      if (i < N) s += fabsf(as[i]);
      if (lane == 0) {
        if (i < N) l1[i] = s;
        atomicAdd(&all_l1, s);  // a bound: the order of the sum does not matter
      }
    }
    __syncthreads();
  }
  const RuleTables tables{logtab, cl, inc, C, nwords};
  float *ths = reinterpret_cast<float *>(smem_raw + lay.theta + warp * lay.per_warp);
  float *los = ths + MP;  // FP64: the low parts
  const int R = (M + 31) >> 5;
  const float eps0 = 2.0f * (MP * (A_UNIT + (F64 ? 0.0f : B_UNIT)) + FIXED +
                             (F64 ? 12.0f * ROUND * all_l1 : 0.0f)) + LN_U;
  const float eps_s = 2.0f * (8 * Q + 16) * ROUND;
  const float eps_d = F64 ? 0.0f : 2.0f * 2.0f * (R + 6) * 1.5f * ROUND;
  const int total = A.n_discard + A.L;
  // every warp of the block takes part in the shared recomputation; warps without a
  // chain do nothing else
  for (int first = blockIdx.x * wpb; first < A.B; first += gridDim.x * wpb) {
    const int b = first + warp;
    const bool live = warp < wpb && b < A.B;
    ChainBits<RULE> ch;
    if (live) ch.load(A.sigma + (int64_t)b * N, N, tables);
    float sum_abs = 0.0f, log_prod = 0.0f;
    auto totals = [&]() {
      float s = 0.0f, p = 1.0f;
#pragma unroll 4
      for (int j = lane; j < MP; j += 32) {
        const float m = fabsf(ths[j]);
        s += m;
        p = fmaf(p, ex2_fast(-2.885390043f * m), p);
      }
      sum_abs = s;
      log_prod = __log2f(p);
    };
    // theta = b + x W of all the block's chains, in the plain kernel's order (FP32)
    auto recompute_all = [&]() {
      __syncthreads();
      if (warp < chains) {
        for (int w = 0; 32 * w < N; ++w) {
          const uint32_t bits = __shfl_sync(0xffffffffu, ch.xb, w);
          const int i = 32 * w + lane;
          if (i < N) xs[i * chains + warp] = (bits >> lane) & 1u ? 1.0f : -1.0f;
        }
      }
      __syncthreads();
      for (int c0 = 0; c0 < wpb; c0 += FL_CHAINS) {
        float acc[JPT][FL_CHAINS];
#pragma unroll
        for (int k = 0; k < JPT; ++k) {
          const int j = tid + k * THREADS;
          const float bj = j < M ? f32_of(params[j]) : 0.0f;
#pragma unroll
          for (int c = 0; c < FL_CHAINS; ++c) acc[k][c] = bj;
        }
#pragma unroll 4
        for (int i = 0; i < N; ++i) {
          float w[JPT];
#pragma unroll
          for (int k = 0; k < JPT; ++k) {
            const int j = tid + k * THREADS;
            w[k] = j < M ? f32_of(__ldg(W + (int64_t)i * M + j)) : 0.0f;
          }
#pragma unroll
          for (int c = 0; c < FL_CHAINS; ++c) {
            const float x = xs[i * chains + c0 + c];
#pragma unroll
            for (int k = 0; k < JPT; ++k) acc[k][c] += x * w[k];
          }
        }
#pragma unroll
        for (int c = 0; c < FL_CHAINS; ++c) {
          if (c0 + c < wpb) {
            float *to = reinterpret_cast<float *>(smem_raw + lay.theta + (c0 + c) * lay.per_warp);
#pragma unroll
            for (int k = 0; k < JPT; ++k)
              if (tid + k * THREADS < MP) to[tid + k * THREADS] = acc[k][c];
          }
        }
      }
      __syncthreads();
    };
    if (F64 && live) {  // theta as double-float sums over the FP32 weights
      for (int j = lane; j < MP; j += 32) {
        float hi = j < M ? f32_of(params[j]) : 0.0f, lo = 0.0f;
        for (int w = 0; 32 * w < N; ++w) {
          const uint32_t bits = __shfl_sync(0xffffffffu, ch.xb, w);
          const int i1 = min(32, N - 32 * w);
          for (int q = 0; q < i1; ++q) {
            const float v = j < M ? f32_of(W[(int64_t)(32 * w + q) * M + j]) : 0.0f;
            const df32 s = df_two_sum(hi, (bits >> q) & 1u ? v : -v);
            hi = s.hi;
            lo += s.lo;
          }
        }
        const df32 s = df_quick_two_sum(hi, lo);
        ths[j] = s.hi;
        los[j] = s.lo;
      }
      __syncwarp();
      totals();
    }
    int64_t acc_count = 0;
    for (int step = 0; step < total; ++step) {
      if (!F64) {
        recompute_all();
        if (live) totals();
      }
      if (!live) continue;
      RandomWords<F64> rnd;
      for (int p = 0; p < A.sweep; ++p) {
        if ((p & 31) == 0) rnd.draw(A, A.counter + (uint64_t)step * A.sweep + p, b);
        Proposal pr;
        if (!ch.propose(__shfl_sync(0xffffffffu, rnd.x, p & 31), N, tables, pr)) continue;
        const int su = pr.su, sv = pr.sv;
        const float corr = pr.corr;
        const int du = ch.up(su) ? -2 : 2;  // an Exchange partner changes by -du
        const float fu = (float)du;
        const T *Wu = W + (int64_t)su * M;
        const T *Wv = W + (int64_t)(RULE == 1 ? sv : su) * M;
        float t[4 * Q];
        float new_abs = 0.0f, prod = 1.0f;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          float wu[4], wv[4], th4[4];
          load_quad<VEC>(Wu, M, q, lane, wu);
          if (RULE == 1) load_quad<VEC>(Wv, M, q, lane, wv);
          if (VEC) {
            const float4 v = *reinterpret_cast<const float4 *>(ths + 128 * q + 4 * lane);
            th4[0] = v.x;
            th4[1] = v.y;
            th4[2] = v.z;
            th4[3] = v.w;
          } else {
#pragma unroll
            for (int c = 0; c < 4; ++c) th4[c] = ths[unit<VEC>(q, c, lane)];
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            float v = th4[c] + fu * wu[c];
            if (RULE == 1) v -= fu * wv[c];
            t[4 * q + c] = v;
            const float m = fabsf(v);
            new_abs += m;
            prod = fmaf(prod, ex2_fast(-2.885390043f * m), prod);  // at most 2^(4 Q)
          }
        }
        const float new_prod = __log2f(prod);
        const float d = (new_abs - sum_abs) + 0.693147181f * (new_prod - log_prod);
        const bool far = !(fabsf(d) < SUM_MAX);
        const int sum = __reduce_add_sync(0xffffffffu, far ? 0 : __float2int_rn(d * 524288.0f));
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
          if constexpr (F64) {
            accept = exact_accept_f64<true>(static_cast<const double *>(A.params), N, M, ch.xb, su, sv,
                                      du, ch.hop, pr.hop_new,
                                      __shfl_sync(0xffffffffu, rnd.y, p & 31),
                                      __shfl_sync(0xffffffffu, rnd.z, p & 31));
          } else {
            float e = 0.0f;
            for (int j = lane; j < M; j += 32) {
              const float th = ths[j];
              float v = th + fu * f32_of(__ldg(Wu + j));
              if (RULE == 1) v -= fu * f32_of(__ldg(Wv + j));
              e += log_cosh_fast(v) - log_cosh_fast(th);
            }
            e = warp_sum(e);
            e += fu * as[su];
            if (RULE == 1) e += -fu * as[sv];
            const float dlp = 2.0f * e;
            accept = u01f(__shfl_sync(0xffffffffu, rnd.y, p & 31)) < expf(dlp + corr);
          }
        }
        if (accept) {
          if constexpr (F64) {
#pragma unroll 2
            for (int q = 0; q < Q; ++q) {
              float wu[4], wv[4];
              load_quad<VEC>(Wu, M, q, lane, wu);
              if (RULE == 1) load_quad<VEC>(Wv, M, q, lane, wv);
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                const int j = unit<VEC>(q, c, lane);
                df32 v = df_two_sum(ths[j], fu * wu[c]);
                float low = los[j] + v.lo;
                if (RULE == 1) {
                  v = df_two_sum(v.hi, -fu * wv[c]);
                  low += v.lo;
                }
                v = df_quick_two_sum(v.hi, low);
                ths[j] = v.hi;
                los[j] = v.lo;
              }
            }
          } else {
#pragma unroll
            for (int q = 0; q < Q; ++q) {
              if (VEC) {
                *reinterpret_cast<float4 *>(ths + 128 * q + 4 * lane) =
                    make_float4(t[4 * q], t[4 * q + 1], t[4 * q + 2], t[4 * q + 3]);
              } else {
#pragma unroll
                for (int c = 0; c < 4; ++c) ths[unit<VEC>(q, c, lane)] = t[4 * q + c];
              }
            }
          }
          __syncwarp();
          sum_abs = new_abs;
          log_prod = new_prod;
          ch.apply(pr);
          ++acc_count;
        }
      }
      if (step >= A.n_discard)
        ch.store(A.samples + ((int64_t)b * A.L + (step - A.n_discard)) * N, N);
    }
    if (!F64) recompute_all();
    if (live) {
      T logpsi;
      if constexpr (F64) {
        logpsi = final_logpsi_f64(static_cast<const double *>(A.params), N, M, ch.xb);
      } else {
        float part = 0.0f;
        for (int j = lane; j < M; j += 32) part += log_cosh_fast(ths[j]);
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
  }
}

// Quads per lane: 128 Q >= M.
static int l2_quads(int M) {
  for (int q : {2, 4, 8, 16})
    if (M <= 128 * q) return q;
  return 0;
}

template <typename T, int Q>
static int l2_chains(int rule, int N, int C, int most) {
  int w = std::min(l2_warps<T, Q>(), most);
  while (w > 0 && l2_smem(sizeof(T) == 8, rule, N, Q, C, w).total > FS_SMEM_MAX) --w;
  return w;
}

// Spins and clusters are one bit word per lane, t is in registers; at least four
// chains' theta have to fit beside the tables.
bool filtered_l2_fits(int dtype, int rule, int N, int M, int C) {
  const int Q = l2_quads(M);
  return Q > 0 && N <= 1024 && (rule == 0 || C <= 1024) &&
         l2_smem(dtype == VMCK_F64, rule, N, Q, rule == 1 ? C : 0, 4).total <= FS_SMEM_MAX;
}

template <typename T, int RULE, int Q, bool VEC>
static int launch_l2_as(cudaStream_t st, const SweepArgs &a) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int most = l2_chains<T, Q>(RULE, a.N, a.C, l2_warps<T, Q>());
  // as few rounds as shared memory allows, each with an even share of the chains
  const int rounds = (a.B + sms * most - 1) / (sms * most);
  const int wpb = (a.B + sms * rounds - 1) / (sms * rounds);
  const size_t smem = l2_smem(sizeof(T) == 8, RULE, a.N, Q, a.C, wpb).total;
  VMCK_CUDA(cudaFuncSetAttribute(metropolis_filtered_l2_kernel<T, RULE, Q, VEC>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int grid = std::min((a.B + wpb - 1) / wpb, sms);
  metropolis_filtered_l2_kernel<T, RULE, Q, VEC>
      <<<grid, 32 * l2_warps<T, Q>(), smem, st>>>(a, wpb);
  return check_launch("metropolis_sample (filtered, weights through L2)");
}

template <typename T, int RULE, bool VEC>
static int launch_l2_q(cudaStream_t st, const SweepArgs &a) {
  switch (l2_quads(a.M)) {
    case 2: return launch_l2_as<T, RULE, 2, VEC>(st, a);
    case 4: return launch_l2_as<T, RULE, 4, VEC>(st, a);
    case 8: return launch_l2_as<T, RULE, 8, VEC>(st, a);
    default: return launch_l2_as<T, RULE, 16, VEC>(st, a);
  }
}

template <typename T>
static int launch_l2_t(cudaStream_t st, int rule, const SweepArgs &a) {
  // rows of W start at params + M + i M: 16-byte loads need M a multiple of four
  const bool vec = a.M % 4 == 0 && reinterpret_cast<uintptr_t>(a.params) % 16 == 0;
  if (rule == 0) return vec ? launch_l2_q<T, 0, true>(st, a) : launch_l2_q<T, 0, false>(st, a);
  return vec ? launch_l2_q<T, 1, true>(st, a) : launch_l2_q<T, 1, false>(st, a);
}

int launch_filtered_l2(cudaStream_t st, int dtype, int rule, const SweepArgs &args) {
  SweepArgs a = args;
  if (rule == 0) a.C = 0;
  return dtype == VMCK_F64 ? launch_l2_t<double>(st, rule, a) : launch_l2_t<float>(st, rule, a);
}

}  // namespace vmck
