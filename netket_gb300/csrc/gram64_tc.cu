// T = O_L O_L^T + diag_shift I for FP64 tanh(theta), the contraction t t^T on the
// tcgen05 tensor cores.
//
// A row of t (|t| <= 1), times the power of two that brings its largest entry to [1/2, 1), is
// rounded to a multiple of 2^-55 and written in balanced base-128 digits, t 2^s = sum_a
// q_a 2^(-6 - 7 a), a = 0 .. 7, |q_a| <= 64: eight matrices of small integers, exact in
// FP16.  t t^T is then 2^(-s - s') sum_d 2^(-12 - 7 d) D_d with
//   D_d = sum_{a + b = d} q_a q_b^T.
// An entry of D_d is an integer of at most (d + 1) K 4096 <= 2^24 for K <= 512, so
// the tensor core forms it exactly in its FP32 accumulator, whatever the order and
// rounding of its additions.  Diagonals d = 0 .. 7 are kept (36 products), and of
// d = 8 the squares: where two rows are equal (on the matrix diagonal, and for a
// configuration that was sampled twice) q_4 q_4 is positive, 2^-57.6 per hidden unit
// in the mean, while the other products of d = 8 change sign.  They join D_7 as
// q_4 (q_4 2^-7)^T, a ninth operand plane (with its fractions D_7 may be rounded to 24
// bits, a unit of 2^-61 at most per MMA).  What is left out is at most 6.1 2^-56 per hidden
// unit, about 2^-56 sqrt(hidden units) in a sum, of the product of the rows' largest
// entries.  Error of T, rms, over that of FP64 sums: 0.15 to 0.86 (weights of 0.001 to 0.3, N =
// 8 .. 100, M = 32 .. 400).  The eight integers of an entry are added in two 64-bit integers
// (more than 512 hidden units: chunk by chunk) and only the assembly (x . x', g, 1 / n) is FP64.
//
// The FP64 pipe (two operations per clock and SM) bounded the plain form:
// n = 4,096, M = 400: 5.74 -> 0.41 ms (digits 0.012 of it; 0.38 without the ninth plane).
//
// Kernel: persistent, warp-specialised (TMA warp, MMA warp, 16 epilogue warps),
// tiles of 128 rows x 64 columns of the lower triangle.  The eight diagonals fill
// tensor memory (8 x 64 columns); a stage holds all planes of 32 hidden units
// (64-byte swizzle; A 64 KB, B 36 KB; two stages) for the 74 MMAs that use it.  The
// epilogue empties tensor memory into registers first, so its FP64 arithmetic and
// stores overlap the next tile's MMAs.  Waits are bounded by the library's wait
// limit (VMCK_DEV_TIMEOUT).
#include <cuda_fp16.h>

#include <algorithm>

#include "gram_tc.cuh"
#include "tc_common.cuh"
#include "units_f64.cuh"

namespace vmck {

namespace {

constexpr int H_DIGITS = 8, H_PLANES = H_DIGITS + 1;  // + q_4 2^-7
constexpr int H_BM = 128, H_BN = 64, H_BK = 32, H_STAGES = 2;
constexpr int H_A_BYTES = H_BM * H_BK * 2, H_B_BYTES = H_BN * H_BK * 2;  // one digit
constexpr int H_STAGE_BYTES = H_DIGITS * H_A_BYTES + H_PLANES * H_B_BYTES;
constexpr int H_EPI_WARPS = 16, H_THREADS = 32 * (2 + H_EPI_WARPS);
constexpr int H_COLS = H_BN / 4;  // columns per epilogue warp (four per lane quarter)
constexpr int H_TMEM = H_DIGITS * H_BN;
constexpr int H_CHUNK = 512 / H_BK;  // stages whose sums stay below 2^24
constexpr int H_WORDS = 9;           // sign words of N <= 288
constexpr int H_SHIFT_MAX = 480;     // 2^(-61 - 2 s) is a normal number

// K-major operand with 64-byte swizzle: 8-row groups 512 bytes apart, layout
// SWIZZLE_64B = 4 (fields as in umma_desc_sw128).
__device__ __forceinline__ uint64_t umma_desc_sw64(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr >> 4) & 0x3FFF);
  d |= static_cast<uint64_t>(1) << 16;
  d |= static_cast<uint64_t>(512 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(4) << 61;
  return d;
}

struct Gram64Params {
  const uint32_t *bits;  // sign words of the samples
  const double *g, *c;   // O obar per sample, |obar|^2
  double *T64;
  float *T32;
  double inv_n, shift;
  int64_t n;
  int words, N, M;
  const int *skip;  // nonzero: t is out of range, the plain kernel forms T
  const int *shift_of;  // s of each row
  int32_t *status;
  unsigned long long wait_ns;
  int64_t tiles;
};

// Tile t -> (row tile, column tile): row tile I has column tiles 0 .. 2 I + 1.
__device__ __forceinline__ void gram64_tile(int64_t t, int &I, int &J) {
  int64_t i = (int64_t)((sqrt(4.0 * (double)t + 1.0) - 1.0) * 0.5);
  while (i * (i + 1) > t) --i;
  while ((i + 1) * (i + 2) <= t) ++i;
  I = (int)i;
  J = (int)(t - i * (i + 1));
}

// digits[a][row][k] of t 2^s and the ninth plane, zero for k in [M, ldk), and s of each row;
// *flag is set where |t| > 1 or NaN.  A warp per row, two neighbouring k per lane.
__global__ void __launch_bounds__(256) gram64_digits_kernel(const double *__restrict__ t,
                                                            int64_t n, int M, int ldk,
                                                            __half2 *__restrict__ digits,
                                                            int *__restrict__ shift_of,
                                                            int *flag) {
  const int64_t r = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= n) return;
  const double *row = t + r * M;
  uint32_t most = 0u;
  for (int k = lane; k < M; k += 32) most = max(most, size_word(__ldg(row + k)));
  most = __reduce_max_sync(0xffffffffu, most);
  if (most > 0x3ff00000u) {  // |t| > 1 or NaN
    if (lane == 0) atomicOr(flag, 1);
    return;
  }
  const int s = most == 0u ? 0 : min(max(1022 - (int)(most >> 20), 0), H_SHIFT_MAX);
  if (lane == 0) shift_of[r] = s;
  const double scale = __hiloint2double((1023 + 55 + s) << 20, 0);
  const int half_ld = ldk / 2;
  __half2 *out = digits + r * half_ld;
  for (int h = lane; h < half_ld; h += 32) {
    float d[2][H_DIGITS];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      long long v = 2 * h + q < M ? __double2ll_rn(__ldg(row + 2 * h + q) * scale) : 0ll;
#pragma unroll
      for (int a = H_DIGITS - 1; a > 0; --a) {
        const int low = (int)((v + 64) & 127) - 64;
        d[q][a] = (float)low;
        v = (v - low) >> 7;
      }
      d[q][0] = (float)(int)v;
    }
#pragma unroll
    for (int a = 0; a < H_DIGITS; ++a)
      out[a * n * half_ld + h] = __floats2half2_rn(d[0][a], d[1][a]);
    out[H_DIGITS * n * half_ld + h] = __floats2half2_rn(0x1p-7f * d[0][4], 0x1p-7f * d[1][4]);
  }
}

__global__ void __launch_bounds__(H_THREADS, 1)
    gram64_kernel(const __grid_constant__ CUtensorMap mA, const __grid_constant__ CUtensorMap mB,
                  Gram64Params g) {
  extern __shared__ __align__(1024) unsigned char h_smem_raw[];
  unsigned char *smem = reinterpret_cast<unsigned char *>(
      (reinterpret_cast<uintptr_t>(h_smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + H_STAGES * H_STAGE_BYTES);
  uint64_t *empty = full + H_STAGES;
  uint64_t *d_full = empty + H_STAGES;
  uint64_t *d_empty = d_full + 1;
  uint64_t *drain = d_empty + 1;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drain + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0)
    *abort_flag = (*g.skip != 0 ||
                   (g.status &&
                    (*reinterpret_cast<volatile int32_t *>(g.status) & VMCK_DEV_TIMEOUT)))
                      ? 1
                      : 0;
  __syncthreads();
  if (*abort_flag) return;
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(H_TMEM)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int s = 0; s < H_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(d_full, 1);
    mbar_init(d_empty, H_EPI_WARPS);
    mbar_init(drain, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int num_kb = (g.M + H_BK - 1) / H_BK;

  auto fail = [&]() {
    if (g.status) atomicOr(g.status, VMCK_DEV_TIMEOUT);
    *abort_flag = 1;
  };

  if (warp == 0) {
    // ---------------- TMA producer: digit a of rows [y, ..) is at tensor row a n + y
    if (lane == 0) {
      int64_t it = 0;
      for (int64_t tile = blockIdx.x; tile < g.tiles && !*abort_flag; tile += gridDim.x) {
        int I, J;
        gram64_tile(tile, I, J);
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = (int)(it % H_STAGES);
          if (it >= H_STAGES &&
              !mbar_wait(&empty[s], (uint32_t)(((it / H_STAGES) - 1) & 1), g.wait_ns)) {
            fail();
            break;
          }
          if (*abort_flag) break;
          unsigned char *st = smem + s * H_STAGE_BYTES;
          mbar_expect_tx(&full[s], H_STAGE_BYTES);
          for (int a = 0; a < H_DIGITS; ++a)
            tma_load_2d(st + a * H_A_BYTES, &mA, &full[s], kb * H_BK,
                        (int)(a * g.n) + I * H_BM);
          for (int a = 0; a < H_PLANES; ++a)
            tma_load_2d(st + H_DIGITS * H_A_BYTES + a * H_B_BYTES, &mB, &full[s], kb * H_BK,
                        (int)(a * g.n) + J * H_BN);
        }
      }
      // every copy issued must land before the CTA may exit
      const int64_t first = it > H_STAGES ? it - H_STAGES : 0;
      for (int64_t q = first; q < it; ++q)
        mbar_wait(&full[q % H_STAGES], (uint32_t)((q / H_STAGES) & 1));
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer
    if (lane == 0) {
      const uint32_t idesc = umma_idesc_f16(H_BM, H_BN);
      int64_t it = 0, drained = 0;  // chunks handed to the epilogue
      bool issued_any = false, ok = true;
      for (int64_t tile = blockIdx.x; tile < g.tiles && ok && !*abort_flag; tile += gridDim.x) {
        for (int kb = 0; kb < num_kb && ok; ++kb, ++it) {
          const int in_chunk = kb % H_CHUNK;
          if (in_chunk == 0 && drained > 0 &&
              !mbar_wait(d_empty, (uint32_t)((drained - 1) & 1), g.wait_ns)) {
            fail();
            ok = false;
            break;
          }
          const int s = (int)(it % H_STAGES);
          if (!mbar_wait(&full[s], (uint32_t)((it / H_STAGES) & 1), g.wait_ns)) {
            fail();
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a0 = smem_u32(smem + s * H_STAGE_BYTES);
          const uint32_t b0 = a0 + H_DIGITS * H_A_BYTES;
#pragma unroll 1
          for (int d = 0; d < H_DIGITS; ++d) {
            const uint32_t dst = tmem_base + d * H_BN;
#pragma unroll 1
            for (int a = 0; a <= d; ++a) {
              const uint32_t as = a0 + a * H_A_BYTES, bs = b0 + (d - a) * H_B_BYTES;
#pragma unroll
              for (int k = 0; k < H_BK / 16; ++k)
                umma_f16(dst, umma_desc_sw64(as + 32 * k), umma_desc_sw64(bs + 32 * k), idesc,
                         (in_chunk == 0 && a == 0 && k == 0) ? 0u : 1u);
            }
          }
#pragma unroll
          for (int k = 0; k < H_BK / 16; ++k)  // q_4 (q_4 2^-7)^T
            umma_f16(tmem_base + (H_DIGITS - 1) * H_BN, umma_desc_sw64(a0 + 4 * H_A_BYTES + 32 * k),
                     umma_desc_sw64(b0 + H_DIGITS * H_B_BYTES + 32 * k), idesc, 1u);
          umma_commit(&empty[s]);
          issued_any = true;
          if (in_chunk == H_CHUNK - 1 || kb == num_kb - 1) {
            umma_commit(d_full);
            ++drained;
          }
        }
      }
      if (issued_any) {
        umma_commit(drain);
        mbar_wait(drain, 0);
      }
    }
  } else {
    // ---------------- epilogue: warp e reads lane quarter (warp & 3), columns
    // [16 (e >> 2), +16); a thread holds 16 columns of one row
    const int e = warp - 2, quarter = warp & 3, part = e >> 2;
    const uint32_t tm = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) +
                        (uint32_t)(part * H_COLS);
    const double cc = *g.c;
    int64_t chunk = 0;
    bool alive = true;
    for (int64_t tile = blockIdx.x; tile < g.tiles && alive; tile += gridDim.x) {
      int I, J;
      gram64_tile(tile, I, J);
      // sum_d D_d 2^(-12 - 7 d) = hi 2^-33 + lo 2^-61 (times 2^(-s - s'))
      long long hi[H_COLS], lo[H_COLS];
#pragma unroll
      for (int j = 0; j < H_COLS; ++j) hi[j] = lo[j] = 0;
      for (int kb = 0; kb < num_kb; kb += H_CHUNK, ++chunk) {
        if (!mbar_wait(d_full, (uint32_t)(chunk & 1), g.wait_ns)) {
          fail();
          alive = false;
          break;
        }
        tc_fence_after();
#pragma unroll
        for (int d = 0; d < H_DIGITS; ++d) {
          float v[H_COLS];
          tmem_ld_16cols(tm + d * H_BN, v);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < H_COLS; ++j) {
            const long long w = (long long)__float2int_rn(v[j]) * (1 << (7 * (3 - (d & 3))));
            if (d < 4) hi[j] += w;
            else lo[j] += w;
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(d_empty);
      }
      if (!alive) break;
      const int64_t row = (int64_t)I * H_BM + quarter * 32 + lane;
      const int64_t col0 = (int64_t)J * H_BN + part * H_COLS;
      if (row < g.n && col0 <= row) {
        uint32_t rb[H_WORDS];
#pragma unroll
        for (int w = 0; w < H_WORDS; ++w)
          rb[w] = w < g.words ? __ldg(g.bits + row * g.words + w) : 0u;
        const double gr = cc - __ldg(g.g + row);
        const int sr = 1023 - __ldg(g.shift_of + row);
        double *out = g.T64 ? g.T64 + row * g.n + col0 : nullptr;
        float *out32 = g.T32 ? g.T32 + row * g.n + col0 : nullptr;
#pragma unroll
        for (int j = 0; j < H_COLS; ++j) {
          const int64_t col = col0 + j;
          if (col <= row) {
            int diff = 0;
#pragma unroll
            for (int w = 0; w < H_WORDS; ++w)
              if (w < g.words) diff += __popc(rb[w] ^ __ldg(g.bits + col * g.words + w));
            const int B = g.N - 2 * diff;
            const int es = (sr - __ldg(g.shift_of + col)) << 20;  // exponent of 2^(-s - s')
            const double A = fma((double)hi[j], __hiloint2double(es - (33 << 20), 0),
                                 (double)lo[j] * __hiloint2double(es - (61 << 20), 0));
            double v = (fma(A, (double)(1 + B), (double)B) + (gr - __ldg(g.g + col))) * g.inv_n;
            if (col == row) v += g.shift;
            if (out) out[j] = v;
            if (out32) out32[j] = (float)v;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(H_TMEM)
                 : "memory");
  }
}

int64_t digits_ld(int M) { return (M + H_BK - 1) / H_BK * H_BK; }

int digits_map(CUtensorMap *map, const __half *base, int64_t ldk, int64_t rows, int box_rows) {
  auto fn = encode_fn();
  if (!fn) {
    set_last_error("cuTensorMapEncodeTiled is unavailable");
    return VMCK_ERR_CUDA;
  }
  cuuint64_t dims[2] = {(cuuint64_t)ldk, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)(ldk * 2)};
  cuuint32_t box[2] = {(cuuint32_t)H_BK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  const CUresult r =
      fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half *>(base), dims, strides, box,
         estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_last_error("cuTensorMapEncodeTiled failed (%d)", (int)r);
    return VMCK_ERR_CUDA;
  }
  return VMCK_OK;
}

}  // namespace

// Bytes: the range flag, the digits (1,024-byte aligned) and the rows' shifts.
int64_t gram64_tc_workspace_doubles(int M, int64_t n) {
  return (H_PLANES * n * digits_ld(M) * 2 + 1024 + 64 + 4 * n) / 8 + 1;
}

// The plain kernel's time is its M steps of one 64 x 64 tile until the tiles fill the
// SMs (n about 1,100), this kernel's about 20 us more of set-up, then its stages.
// Whole call, tensor cores / plain, us: M = 16, n = 1,024: 73 / 55, n = 2,048: 106 /
// 133; M = 64, n = 64: 70 / 113, n = 2,048: 123 / 341; M = 400, n = 64: 187 / 551,
// n = 4,096: 609 / 5,979.
bool gram64_tc_takes(int M, int64_t n) {
  // rows of all digits are TMA coordinates (32-bit)
  return (M > 32 || n >= 1536) && H_PLANES * n + H_BM < (1ll << 31);
}

// *flag_out: device word, nonzero after the launch where t was out of range (the
// caller runs the plain kernel under it).
int gram64_tc_launch(cudaStream_t st, const double *t, const uint32_t *bits, int words, int N,
                     int M, int64_t n, const double *g, const double *c, double inv_n,
                     double shift, double *T64, float *T32, double *ws, int32_t *status,
                     const int **flag_out) {
  int *flag = reinterpret_cast<int *>(ws);
  __half *digits = reinterpret_cast<__half *>(
      (reinterpret_cast<uintptr_t>(ws) + 64 + 1023) & ~uintptr_t(1023));
  *flag_out = flag;
  const int ldk = (int)digits_ld(M);
  VMCK_CUDA(cudaMemsetAsync(flag, 0, sizeof(int), st));
  int *shift_of = reinterpret_cast<int *>(digits + H_PLANES * n * ldk);
  gram64_digits_kernel<<<(unsigned)((n + 7) / 8), 256, 0, st>>>(
      t, n, M, ldk, reinterpret_cast<__half2 *>(digits), shift_of, flag);
  int rc = check_launch("gram digits");
  if (rc) return rc;
  CUtensorMap mA, mB;
  if ((rc = digits_map(&mA, digits, ldk, H_DIGITS * n, H_BM))) return rc;
  if ((rc = digits_map(&mB, digits, ldk, H_PLANES * n, H_BN))) return rc;
  const int64_t row_tiles = (n + H_BM - 1) / H_BM;
  Gram64Params p{bits, g,  c, T64, T32,  inv_n,  shift,           n,
                 words, N, M, flag, shift_of, status, wait_limit_ns(),
                 row_tiles * (row_tiles + 1)};
  const size_t smem = 1024 + H_STAGES * H_STAGE_BYTES + 128;
  VMCK_CUDA(cudaFuncSetAttribute(gram64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  gram64_kernel<<<(unsigned)std::min<int64_t>(p.tiles, sms), H_THREADS, smem, st>>>(mA, mB, p);
  return check_launch("gram (FP64 on tensor cores)");
}

}  // namespace vmck
