// FP32 local energies of the RBM: operators of one- and two-site terms and Ising.
//
// Every value is the one of eloc_local_kernel<float> / eloc_ising_kernel<float>
// (rbm.cu) bit for bit up to the FP64 sum over connected elements: theta sums the
// sites in order, and the log-ratio of an element sums hidden units j = l + 32 r
// in r for each of 32 partial sums l, which are added pairwise (l ^ 16, 8, 4, 2,
// 1).  Those kernels spent 51 warp instructions per 32 hidden units of an element,
// 17 of them on the arithmetic; the rest went into one four-byte load per operand,
// a five-step butterfly per element and a group-wide scan per sample.
//
// Here eight lanes take one element, lane l holding the partial sums 4 l .. 4 l + 3:
// operands come in 16-byte loads and one butterfly serves the four elements of a
// warp.  Weights that fit are kept in shared memory (one CTA per SM, several
// groups of four warps, each with its own sample and barrier) where the elements are many
// enough (e3_any); the others are read through L1.  Each warp lists the connected elements of its share of the terms
// by ballots, with nothing shared between warps before the sample's sum.
//
// What bounds it: FP32 issue (27 instructions per 32 hidden units of an element).
// 10 x 10 J1-J2, M = 400, n = 16,384 (about 200 elements a sample): 2.10 -> 1.17 ms.
#include <algorithm>

#include "eloc_f32.cuh"
#include "localop.cuh"

namespace vmck {

namespace {

constexpr int E3_GROUP = 128;       // threads of a sample's group
constexpr int E3_MAX_GROUPS = 6;    // groups per CTA with the weights in shared memory
constexpr size_t E3_SMEM_MAX = 227 * 1024 - 2048;

// log_cosh_fast, bit for bit (test_gpu_eloc_f32.py compares the energies), with e^(-2|x|) = 2^(-2
// |x| log2 e) in one multiplication and one MUFU operation; what the operation flushes to
// zero (|x| > 43) is below 1e-37 and leaves the polynomial at its constant either way.
__device__ __forceinline__ float log_cosh_ftz(float x) {
  x = fabsf(x);
  float e;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x * -2.885390043f));
  float p = 0.003752624150365591f;
  p = __fmaf_rn(p, e, -0.02303827926516533f);
  p = __fmaf_rn(p, e, 0.06651248037815094f);
  p = __fmaf_rn(p, e, -0.12526661157608032f);
  p = __fmaf_rn(p, e, 0.1846884787082672f);
  p = __fmaf_rn(p, e, -0.24635660648345947f);
  p = __fmaf_rn(p, e, 0.3328184187412262f);
  p = __fmaf_rn(p, e, -0.4999622404575348f);
  p = __fmaf_rn(p, e, 0.999998927116394f);
  p = __fmaf_rn(p, e, 5.239402245393876e-09f);
  return x + p - 0.693147180559945309f;
}

// A connected element: its two sites and their spin changes (-2, 0, 2), packed.
// Sites take 14 bits, a change two (1: -2, 2: 0, 3: +2).
__device__ __forceinline__ uint32_t pack_element(int s0, int d0, int s1, int d1) {
  return (uint32_t)s0 | (uint32_t)(2 + d0 / 2) << 14 | (uint32_t)s1 << 16 |
         (uint32_t)(2 + d1 / 2) << 30;
}
__device__ __forceinline__ int element_site0(uint32_t e) { return (int)(e & 0x3fffu); }
__device__ __forceinline__ int element_site1(uint32_t e) { return (int)((e >> 16) & 0x3fffu); }
__device__ __forceinline__ float element_d0(uint32_t e) {
  return (float)(2 * ((int)((e >> 14) & 3u) - 2));
}
__device__ __forceinline__ float element_d1(uint32_t e) { return (float)(2 * ((int)(e >> 30) - 2)); }

// Bytes of shared memory: the weights (rows padded to MP) and visible biases, then
// per group theta, log_cosh theta, the spins as floats and four warps' element lists.
struct E3Smem {
  size_t vis, group, th, lc, xs, mel, elem, per_group;
};
__host__ __device__ inline E3Smem e3_smem(bool wsm, int N, int M, int cap) {
  E3Smem s;
  const size_t MP = ((size_t)M + 31) & ~size_t(31);
  s.vis = wsm ? (size_t)N * MP * 4 : 0;
  s.group = align16(s.vis + (wsm ? (size_t)N * 4 : 0));
  s.th = 0;
  s.lc = MP * 4;
  s.xs = 2 * MP * 4;
  s.mel = align16(s.xs + 4 * (size_t)N);
  s.elem = s.mel + 4 * (size_t)cap * 8;
  s.per_group = align16(s.elem + 4 * (size_t)cap * 4);
  return s;
}

}  // namespace

struct IsingArgs {
  const int32_t *edges;
  int n_edges;
  double h, J;
};

// cap: list entries per warp (local operators)
template <bool ISING, bool WSM, bool VEC>
__global__ void __launch_bounds__(WSM ? E3_GROUP *E3_MAX_GROUPS : E3_GROUP)
    eloc_f32_kernel(const float *__restrict__ params, int N, int M, const int8_t *__restrict__ x,
                    int64_t n, vmck_local_op op, IsingArgs ising, int cap,
                    double *__restrict__ eloc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[WSM ? E3_MAX_GROUPS : 1][2][4];
  const int MP = (M + 31) & ~31;
  const E3Smem lay = e3_smem(WSM, N, M, cap);
  const int group = WSM ? threadIdx.x / E3_GROUP : 0;
  const int groups = WSM ? blockDim.x / E3_GROUP : 1;
  const Grp g{(int)threadIdx.x - group * E3_GROUP, E3_GROUP, WSM ? 1 + group : 0};
  const int warp = g.tid >> 5, lane = g.tid & 31;
  const int sub = lane >> 3, l4 = 4 * (lane & 7);  // element of the four, first partial sum
  const float *W = params + M, *a = W + (int64_t)N * M;
  float *ws = reinterpret_cast<float *>(smem_raw);
  float *as = reinterpret_cast<float *>(smem_raw + lay.vis);
  if (WSM) {
    for (int e = threadIdx.x; e < N * MP; e += blockDim.x) {
      const int i = e / MP, j = e - i * MP;
      ws[e] = j < M ? W[(int64_t)i * M + j] : 0.0f;
    }
    for (int i = threadIdx.x; i < N; i += blockDim.x) as[i] = a[i];
    __syncthreads();
  }
  unsigned char *mine = smem_raw + lay.group + group * lay.per_group;
  float *th = reinterpret_cast<float *>(mine + lay.th);
  float *lc = reinterpret_cast<float *>(mine + lay.lc);
  float *xs = reinterpret_cast<float *>(mine + lay.xs);
  double *mel = reinterpret_cast<double *>(mine + lay.mel) + (size_t)warp * cap;
  uint32_t *elem = reinterpret_cast<uint32_t *>(mine + lay.elem) + (size_t)warp * cap;

  // log-ratio of the element e for the eight lanes of this sub-group
  auto log_ratio = [&](uint32_t e) -> float {
    const int s0 = element_site0(e), s1 = element_site1(e);
    const float d0 = element_d0(e), d1 = element_d1(e);
    const float *w0 = WSM ? ws + s0 * MP : W + (int64_t)s0 * M;
    const float *w1 = WSM ? ws + s1 * MP : W + (int64_t)s1 * M;
    float p[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 2
    for (int j = l4; j < MP; j += 32) {
      float u[4], v[4], t[4], c[4];
      if (WSM || (VEC && j < M)) {
        const float4 f = *reinterpret_cast<const float4 *>(w0 + j);
        u[0] = f.x, u[1] = f.y, u[2] = f.z, u[3] = f.w;
        if (!ISING) {
          const float4 f1 = *reinterpret_cast<const float4 *>(w1 + j);
          v[0] = f1.x, v[1] = f1.y, v[2] = f1.z, v[3] = f1.w;
        }
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          u[k] = !VEC && j + k < M ? __ldg(w0 + j + k) : 0.0f;
          if (!ISING) v[k] = !VEC && j + k < M ? __ldg(w1 + j + k) : 0.0f;
        }
      }
      const float4 f2 = *reinterpret_cast<const float4 *>(th + j);
      const float4 f3 = *reinterpret_cast<const float4 *>(lc + j);
      t[0] = f2.x, t[1] = f2.y, t[2] = f2.z, t[3] = f2.w;
      c[0] = f3.x, c[1] = f3.y, c[2] = f3.z, c[3] = f3.w;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        t[k] += d0 * u[k];
        if (!ISING) t[k] += d1 * v[k];
        p[k] += log_cosh_ftz(t[k]) - c[k];
      }
    }
    // the butterfly over 32 partial sums: l ^ 16, 8, 4 across lanes, 2, 1 within
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
#pragma unroll
      for (int k = 0; k < 4; ++k) p[k] += __shfl_xor_sync(0xffffffffu, p[k], o);
    float s = (p[0] + p[2]) + (p[1] + p[3]);
    s += d0 * (WSM ? as[s0] : __ldg(a + s0));
    // (a one-site element's second site is a placeholder)
    if (!ISING && d1 != 0.0f) s += d1 * (WSM ? as[s1] : __ldg(a + s1));
    return s;
  };

  for (int64_t b = (int64_t)blockIdx.x * groups + group; b < n; b += (int64_t)gridDim.x * groups) {
    const int8_t *xb = x + b * N;
    for (int i = g.tid; i < N; i += E3_GROUP) xs[i] = (float)xb[i];
    grp_sync(g);
    // theta and log_cosh(theta); the padding adds zeros to every log-ratio
    for (int j = g.tid; j < MP; j += E3_GROUP) {
      float acc = 0.0f;
      if (j < M) {
        acc = params[j];
        const float *w = WSM ? ws + j : W + j;
        const int ld = WSM ? MP : M;
#pragma unroll 4
        for (int i = 0; i < N; ++i) acc += xs[i] * w[(int64_t)i * ld];
      }
      th[j] = acc;
      lc[j] = log_cosh_ftz(acc);
    }
    double acc = 0.0, diag = 0.0;
    int count = 0;  // this warp's elements
    if (ISING) {
      int same = 0;
      for (int e = g.tid; e < ising.n_edges; e += E3_GROUP)
        same += xs[ising.edges[2 * e]] == xs[ising.edges[2 * e + 1]] ? 1 : -1;
      diag = (double)same;
      count = ising.h != 0.0 ? (N - warp + 3) >> 2 : 0;  // sites warp, warp + 4, ...
    } else {
      // connected elements of terms 32 (4 k + warp) + lane
      const int S = op.max_sites, R = op.max_rows;
      for (int t0 = 32 * warp; t0 < op.n_terms; t0 += E3_GROUP) {
        const int t = t0 + lane;
        const bool in = t < op.n_terms;
        int s0 = 0, s1 = 0, r = 0, nc = 0, sz = 0;
        float x0 = 0.0f, x1 = 0.0f;
        if (in) {
          sz = op.acting_size[t];
          if (sz > 0) {
            s0 = op.acting_on[t * S];
            x0 = xs[s0];
            r = x0 < 0.0f;
          }
          if (sz > 1) {
            s1 = op.acting_on[t * S + 1];
            x1 = xs[s1];
            r = (r << 1) | (x1 < 0.0f);
          }
          nc = op.n_conns[(int64_t)t * R + r];
          if (op.nonzero_diagonal) diag += op.diag_mels[(int64_t)t * R + r];
        }
        for (int c = 0; __any_sync(0xffffffffu, c < nc); ++c) {
          bool keep = false;
          double v = 0.0;
          uint32_t e = 0u;
          if (c < nc) {
            const int64_t at = ((int64_t)t * R + r) * op.max_conns + c;
            v = op.mels[at];
            if (fabs(v) > op.mel_cutoff) {
              const int8_t *xp = op.x_prime + at * S;
              const int d0 = sz > 0 ? (int)xp[0] - (int)x0 : 0;
              const int d1 = sz > 1 ? (int)xp[1] - (int)x1 : 0;
              if (d0 == 0 && d1 == 0) {
                acc += v;  // x' = x
              } else {
                keep = true;
                e = pack_element(s0, d0, s1, d1);
              }
            }
          }
          const unsigned m = __ballot_sync(0xffffffffu, keep);
          if (keep) {
            const int at = count + __popc(m & ((1u << lane) - 1u));
            mel[at] = v;
            elem[at] = e;
          }
          count += __popc(m);
        }
      }
    }
    grp_sync(g);  // theta and log_cosh(theta) of all warps; this warp's list
    for (int k0 = 0; k0 < count; k0 += 4) {
      const int k = k0 + sub;
      uint32_t e = 2u << 14 | 2u << 30;  // no element: no change, not added
      double v = 0.0;
      if (k < count) {
        if (ISING) {
          const int i = warp + 4 * k;
          e = pack_element(i, xs[i] < 0.0f ? 2 : -2, 0, 0);
          v = -ising.h;
        } else {
          e = elem[k];
          v = mel[k];
        }
      }
      const float s = log_ratio(e);
      if (k < count && (lane & 7) == 0) acc += v * exp_ratio(s);
    }
    acc = warp_sum(acc);
    diag = warp_sum(diag);
    if (lane == 0) {
      red[group][0][warp] = acc;
      red[group][1][warp] = diag;
    }
    grp_sync(g);
    if (g.tid == 0) {
      const double *ra = red[group][0], *rd = red[group][1];
      const double e = (ra[0] + ra[1]) + (ra[2] + ra[3]);
      const double d = (rd[0] + rd[1]) + (rd[2] + rd[3]);
      if (ISING) {
        eloc[b] = e + ising.J * d;
      } else {
        const double dd = op.nonzero_diagonal ? op.constant + d : 0.0;
        eloc[b] = e + (fabs(dd) > op.mel_cutoff ? dd : 0.0);
      }
    }
    // the next sample's spins and lists are written by threads past this barrier's
    // reads: thread 0 reads red, which the next sample writes after two barriers
  }
}

template <bool ISING, bool WSM, bool VEC>
static int launch_e3(cudaStream_t st, const float *params, int N, int M, const int8_t *x,
                     int64_t n, const vmck_local_op &op, const IsingArgs &ising, int cap,
                     int groups, double *eloc) {
  const int sms = sm_count();
  const E3Smem s = e3_smem(WSM, N, M, cap);
  const size_t smem = s.group + groups * s.per_group;
  if (smem > 40 * 1024)
    VMCK_CUDA(cudaFuncSetAttribute(eloc_f32_kernel<ISING, WSM, VEC>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t grid = WSM ? std::min<int64_t>((n + groups - 1) / groups, sms)
                           : std::min<int64_t>(n, (int64_t)sms * 32);
  eloc_f32_kernel<ISING, WSM, VEC><<<(unsigned)grid, E3_GROUP * groups, smem, st>>>(
      params, N, M, x, n, op, ising, cap, eloc);
  return check_launch(ISING ? "rbm_eloc_ising (FP32)" : "rbm_eloc_local (FP32)");
}

// Entries a warp's list can need: its terms (32 of every 128) times the stored
// columns of a row.
static int e3_cap(const vmck_local_op &op) {
  return (int)std::min<int64_t>((int64_t)((op.n_terms + E3_GROUP - 1) / E3_GROUP) * 32 *
                                    op.max_conns,
                                1 << 20);
}

template <bool ISING>
static int e3_any(cudaStream_t st, const float *params, int N, int M, const int8_t *x, int64_t n,
                  const vmck_local_op &op, const IsingArgs &ising, double *eloc) {
  const int cap = ISING ? 0 : e3_cap(op);
  const E3Smem s = e3_smem(true, N, M, cap);
  int groups = s.group < E3_SMEM_MAX ? (int)((E3_SMEM_MAX - s.group) / s.per_group) : 0;
  groups = std::min(groups, E3_MAX_GROUPS);
  // Weights in shared memory where at least four groups (16 warps) fit beside them and the
  // connected elements are many enough to pay for the copy and for the warps that do not
  // fit: about a million single-site ones, 0.75 million of samples with 128 and more (half
  // of the terms).  L2 / shared memory, us: Ising N = 100, M = 400: n = 3,000 136 / 147,
  // 16,384 672 / 571; J1-J2 8 x 8, M = 256: 3,000 114 / 120, 6,000 205 / 196; 10 x 10, M = 400:
  // 16,384 1,360 / 1,172; Heisenberg 10 x 10 (200 terms), M = 500: 16,384 1,044 / 1,100.
  const bool many = ISING ? n * N >= 1000000 : op.n_terms >= 256 && n * op.n_terms >= 1500000;
  if (groups >= 4 && many)
    return launch_e3<ISING, true, true>(st, params, N, M, x, n, op, ising, cap, groups, eloc);
  const bool vec = M % 4 == 0 && reinterpret_cast<uintptr_t>(params) % 16 == 0;
  return vec ? launch_e3<ISING, false, true>(st, params, N, M, x, n, op, ising, cap, 1, eloc)
             : launch_e3<ISING, false, false>(st, params, N, M, x, n, op, ising, cap, 1, eloc);
}

// Terms of at most two sites, sites in 14 bits, and the lists in shared memory; what
// the general kernel's vectors do not fit stays refused by it.
bool eloc_f32_takes(int N, int M, int64_t n, const vmck_local_op *op) {
  if (N >= (1 << 14)) return false;
  // a handful of samples with wide layers wait for W from L2 either way; the general kernel
  // has more of its rows in flight (12 x 12 J1-J2, M = 1,152: n = 600 336 us here, 333 there;
  // n = 5,000 1,553 here, 1,941 there)
  if (M >= 1024 && n <= 4 * (int64_t)sm_count()) return false;
  const size_t general =
      2 * 4 * (size_t)M + (op ? local_conn_shared_bytes(*op) + 16 : align16((size_t)N));
  if (general > 200 * 1024) return false;
  if (op && op->max_sites > 2) return false;
  const E3Smem s = e3_smem(false, N, M, op ? e3_cap(*op) : 0);
  return s.group + s.per_group <= 200 * 1024;
}

int eloc_f32_ising(cudaStream_t st, const float *params, int N, int M, const int8_t *x, int64_t n,
                   const int32_t *edges, int n_edges, double h, double J, double *eloc) {
  return e3_any<true>(st, params, N, M, x, n, vmck_local_op{}, IsingArgs{edges, n_edges, h, J},
                      eloc);
}

int eloc_f32_local(cudaStream_t st, const float *params, int N, int M, const int8_t *x, int64_t n,
                   const vmck_local_op &op, double *eloc) {
  return e3_any<false>(st, params, N, M, x, n, op, IsingArgs{}, eloc);
}

}  // namespace vmck
