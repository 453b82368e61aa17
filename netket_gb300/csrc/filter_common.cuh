// What the two filtered Metropolis kernels share (sampler_filter.cu: weights in
// shared memory; sampler_filter_l2.cu: weights through L2): the chain's discrete
// state as bit words, its random words, the exact FP64 decision and the constants of
// the filter's margin.
#pragma once

#include "sampler_filter.cuh"

namespace vmck {

namespace {

constexpr size_t FS_SMEM_MAX = 227 * 1024 - 256;

__device__ __forceinline__ float ex2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// theta_j for the spins in the words xb (word l in lane l), from scratch, the sites in
// order, four loads in flight.  j < 0: this lane has no hidden unit.
__device__ __forceinline__ double theta_f64(const double *__restrict__ params, int N, int M,
                                            uint32_t xb, int j) {
  const double *W = params + M + max(j, 0);
  double th = __ldg(params + max(j, 0));
  for (int w = 0; 32 * w < N; ++w) {
    const uint32_t bits = __shfl_sync(0xffffffffu, xb, w);
    const int i1 = min(32, N - 32 * w);
    for (int q0 = 0; q0 < i1; q0 += 4) {
      double v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        v[q] = __ldg(W + (int64_t)(32 * w + min(q0 + q, i1 - 1)) * M);
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (q0 + q < i1) {
          const uint32_t flip = (bits >> (q0 + q)) & 1u ? 0u : 0x80000000u;
          th += __hiloint2double(__double2hiint(v[q]) ^ (int)flip, __double2loint(v[q]));
        }
    }
  }
  return th;
}

// The plain kernel's decision in FP64, theta formed from scratch for the spins in the
// words xb (word l in lane l).  MANY hidden units per lane: s as a sum of |t| - |theta|
// and one logarithm of a quotient of products per lane, half the FP64 operations of a
// log_cosh per hidden unit.  The launch ends with the chain that meets the most of these:
// 1,024 chains, N = 64, M = 128: 314 -> 245 us (one load at a time and log_cosh before;
// 275 with log_cosh); N = 36, M = 72: 246 -> 228 us; one unit per lane (N = M = 16): 234
// with log_cosh, 253 without.
template <bool MANY>
__device__ __noinline__ bool exact_accept_f64(const double *__restrict__ params, int N, int M,
                                              uint32_t xb, int su, int sv, int du, int hop,
                                              int hop_new, uint32_t ry, uint32_t rz) {
  const int lane = threadIdx.x & 31;
  const double *W = params + M, *a = params + M + (int64_t)N * M;
  double s = 0.0, p_new = 1.0, p_old = 1.0;
  for (int j0 = 0; j0 < M; j0 += 32) {
    const int j = j0 + lane < M ? j0 + lane : -1;
    const double th = theta_f64(params, N, M, xb, j);
    if (j >= 0) {
      double t = th + (double)du * W[(int64_t)su * M + j];
      if (sv >= 0) t -= (double)du * W[(int64_t)sv * M + j];
      if (MANY) {
        s += fabs(t) - fabs(th);
        p_new = fma(p_new, exp(-2.0 * fabs(t)), p_new);  // at most 2^(M / 32)
        p_old = fma(p_old, exp(-2.0 * fabs(th)), p_old);
      } else {
        s += log_cosh(t) - log_cosh(th);
      }
    }
  }
  if (MANY) s += log(p_new / p_old);
  s = warp_sum(s);
  s += (double)du * a[su];
  double corr = 0.0;
  if (sv >= 0) {
    s -= (double)du * a[sv];
    corr = log((double)hop) - log((double)hop_new);
  }
  return u01d(ry, rz) < exp(2.0 * s + corr);
}

// log psi of the final state in FP64, in metropolis_kernel's order.
__device__ __noinline__ double final_logpsi_f64(const double *__restrict__ params, int N, int M,
                                                uint32_t xb) {
  const int lane = threadIdx.x & 31;
  const double *a = params + M + (int64_t)N * M;
  double part = 0.0;
  for (int j0 = 0; j0 < M; j0 += 32) {
    const int j = j0 + lane < M ? j0 + lane : -1;
    const double th = theta_f64(params, N, M, xb, j);
    if (j >= 0) part += log_cosh(th);
  }
  for (int w = 0; 32 * w < N; ++w) {
    const uint32_t bits = __shfl_sync(0xffffffffu, xb, w);
    const int i = 32 * w + lane;
    if (i < N) part += (bits >> lane) & 1u ? a[i] : -a[i];
  }
  return warp_sum(part);
}

// The Exchange rule's tables in shared memory.
struct RuleTables {
  const float *logtab;   // C + 1: log k
  const uint32_t *cl;    // C: u | v << 16
  const uint32_t *inc;   // [site][word]: clusters that hold the site once
  int C, nwords;
};

struct Proposal {
  int su, sv, hop_new;
  uint32_t flip;
  float corr;
};

// A chain's discrete state: bit i of word l (lane l) of xb is set where x_i = +1;
// hb holds the hoppable clusters the same way, with this lane's count, the counts
// before it and their sum.
template <int RULE>
struct ChainBits {
  uint32_t xb = 0u, hb = 0u;
  int hop = 0, before = 0, cnt = 0;

  __device__ bool up(int i) const {
    return (__shfl_sync(0xffffffffu, xb, i >> 5) >> (i & 31)) & 1u;
  }
  __device__ void prefix() {
    const int lane = threadIdx.x & 31;
    cnt = __popc(hb);
    int inclusive = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inclusive, o);
      if (lane >= o) inclusive += v;
    }
    before = inclusive - cnt;
  }
  __device__ void load(const int8_t *row, int N, const RuleTables &t) {
    const int lane = threadIdx.x & 31;
    xb = hb = 0u;
    for (int w = 0; 32 * w < N; ++w) {
      const int i = 32 * w + lane;
      const uint32_t m = __ballot_sync(0xffffffffu, i < N && row[i] > 0);
      if (lane == w) xb = m;
    }
    if (RULE == 1) {
      for (int w = 0; w < t.nwords; ++w) {
        const int q = 32 * w + lane;
        const uint32_t c = q < t.C ? t.cl[q] : 0u;
        const int u = (int)(c & 0xffffu), v = (int)(c >> 16);
        const uint32_t xu = __shfl_sync(0xffffffffu, xb, u >> 5) >> (u & 31);
        const uint32_t xv = __shfl_sync(0xffffffffu, xb, v >> 5) >> (v & 31);
        const uint32_t m = __ballot_sync(0xffffffffu, q < t.C && ((xu ^ xv) & 1u));
        if (lane == w) hb = m;
      }
      prefix();
      hop = __reduce_add_sync(0xffffffffu, cnt);
    }
  }
  __device__ void store(int8_t *row, int N) const {
    const int lane = threadIdx.x & 31;
    for (int w = 0; 32 * w < N; ++w) {
      const uint32_t bits = __shfl_sync(0xffffffffu, xb, w);
      if (32 * w + lane < N) row[32 * w + lane] = (bits >> lane) & 1u ? 1 : -1;
    }
  }
  // The proposal of a random word; false where there is no move (rejected).
  __device__ bool propose(uint32_t word, int N, const RuleTables &t, Proposal &p) const {
    const int lane = threadIdx.x & 31;
    p.sv = -1;
    p.hop_new = 0;
    p.flip = 0u;
    p.corr = 0.0f;
    if (RULE == 0) {
      p.su = (int)below(word, (uint32_t)N);
      return true;
    }
    if (hop == 0) return false;
    // the k-th hoppable cluster: its word, then its bit
    const int k = (int)below(word, (uint32_t)hop);
    const unsigned own = __ballot_sync(0xffffffffu, before <= k && k < before + cnt);
    if (own == 0u) return false;  // unreachable while the counts match the words
    const int src = __ffs(own) - 1;
    const uint32_t hw = __shfl_sync(0xffffffffu, hb, src);
    const int nth = k - __shfl_sync(0xffffffffu, before, src);
    const unsigned at = __ballot_sync(
        0xffffffffu, ((hw >> lane) & 1u) && __popc(hw & ((1u << lane) - 1u)) == nth);
    const int pick = 32 * src + __ffs(at) - 1;
    if (pick >= t.C || at == 0u) return false;  // likewise; never index out of range
    const uint32_t c = t.cl[pick];
    p.su = (int)(c & 0xffffu);
    p.sv = (int)(c >> 16);
    if (lane < t.nwords)
      p.flip = t.inc[p.su * t.nwords + lane] ^ t.inc[p.sv * t.nwords + lane];
    p.hop_new =
        hop + __reduce_add_sync(0xffffffffu, __popc(p.flip) - 2 * __popc(p.flip & hb));
    p.corr = t.logtab[hop] - t.logtab[p.hop_new];
    return true;
  }
  __device__ void apply(const Proposal &p) {
    const int lane = threadIdx.x & 31;
    if (lane == (p.su >> 5)) xb ^= 1u << (p.su & 31);
    if (RULE == 1) {
      if (lane == (p.sv >> 5)) xb ^= 1u << (p.sv & 31);
      hb ^= p.flip;
      prefix();
      hop = p.hop_new;
    }
  }
};

// The random words of 32 proposals, one proposal per lane, and ln u of each: NaN (no
// decision by the filter) where the logarithm says too little.
template <bool F64>
struct RandomWords {
  uint32_t x = 0, y = 0, z = 0;
  float ln_u = 0.0f;
  __device__ void draw(const SweepArgs &A, uint64_t first, int b) {
    const uint64_t idx = first + (threadIdx.x & 31);
    const u32x4 r = philox4x32_10(u32x4{(uint32_t)idx, (uint32_t)(idx >> 32), (uint32_t)b, 0u},
                                  A.k0, A.k1);
    x = r.x;
    y = r.y;
    z = r.z;
    if (F64)
      ln_u = y >= 65536u ? (__log2f((float)y) - 32.0f) * 0.693147181f : __int_as_float(-1);
    else
      ln_u = (y >> 8) ? __logf(u01f(y)) : __int_as_float(-1);
  }
};

// Clusters, their logarithms and the incidence words into shared memory, by the
// whole block; barriers inside.
__device__ inline void stage_rule(const SweepArgs &A, int nwords, float *logtab, uint32_t *cl,
                                  uint32_t *inc) {
  const int tid = threadIdx.x, C = A.C;
  for (int k = tid; k <= C; k += blockDim.x) logtab[k] = logf((float)k);
  for (int q = tid; q < C; q += blockDim.x)
    cl[q] = (uint32_t)A.clusters[2 * q] | (uint32_t)A.clusters[2 * q + 1] << 16;
  for (int e = tid; e < A.N * nwords; e += blockDim.x) inc[e] = 0u;
  __syncthreads();
  for (int q = tid; q < C; q += blockDim.x) {
    const int u = (int)(cl[q] & 0xffffu), v = (int)(cl[q] >> 16);
    if (u != v) {  // a cluster of one site twice is never hoppable
      atomicOr(&inc[u * nwords + (q >> 5)], 1u << (q & 31));
      atomicOr(&inc[v * nwords + (q >> 5)], 1u << (q & 31));
    }
  }
}

// eps, the filter's margin on ln u - (2 s + corr).  Per hidden unit: ex2.approx
// and lg2.approx are off by 2^-22 each, the product and the argument of the
// exponential by 2^-24, in t and in theta (A_UNIT); FP32 only: the plain kernel's
// log_cosh_fast by 5e-7 + 2^-23 |x| (B_UNIT, with its |x| part in the next term).
// Per unit of S = sum |t| + |theta|: the roundings of theta + delta and of the
// lane's R additions, 2^-24 each.  The lanes' sums go to the warp total as
// integers in units of 2^-19 (FIXED: half a unit per lane).  FP32 only: the plain
// kernel's summation rounds R + 6 times, each time by 2^-24 of at most
// sum_j |t - theta| <= 2 (|W_u|_1 + |W_v|_1).  FP64 only: the FP32 weights (and
// visible biases) are off by 2^-24 of themselves (2^-23 where they are truncated),
// theta and t by as much of sum |W| + |b| each and delta by 2 more of it.  ln u:
// lg2.approx (2^-22 of at most 32) and, in FP64, the 21 low bits of u, left out
// (2^-16).  Each constant is at least 1.5 times the bound it stands for.
constexpr float A_UNIT = 1.3e-6f, B_UNIT = 1.6e-6f, ROUND = 5.97e-8f, FIXED = 4.6e-5f,
                LN_U = 4e-5f, X_REL = 1e-6f;
constexpr float SUM_UNIT = 1.0f / 524288.0f, SUM_MAX = 126.0f;  // 32 * 126 * 2^19 < 2^31

}  // namespace

}  // namespace vmck
