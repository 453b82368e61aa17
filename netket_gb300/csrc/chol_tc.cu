// Blocked Cholesky factorisation of an FP32 matrix on the tcgen05 tensor cores
// (factor_mode 4 of vmck_cholesky_solve_refined): the factor of the FP32 copy
// of T that iterative refinement against the FP64 matrix turns into an
// FP64-accurate solve.  It replaces jax.scipy.linalg.cho_factor in
// netket/optimizer/solver/solvers.py:266-268.
//
// Storage: the matrix is column-major with its UPPER triangle valid (row-major
// lower triangle, the library's convention); the factor U (A = U^T U) replaces
// it in place.
//
// Algorithm: right-looking, 512-row block rows, each factored in 128-row inner
// panels:
//   leaf   chol_leaf_kernel: one CTA factors the 128 x 128 diagonal block in
//          shared memory and forms its inverse X = U_pp^-1;
//   panel  U[r0:r1, r1:n] = X^T A[r0:r1, r1:n]  (a GEMM with K = 128);
//   inner  A[r1:k1, r1:n] -= U[r0:r1, r1:k1]^T U[r0:r1, r1:n]  (K = 128), the
//          rest of the block row;
//   bulk   A[k1:n, k1:n] -= U[k0:k1, k1:n]^T U[k0:k1, k1:n]  (K = 512), once per
//          block row.
// Every GEMM runs in tc_gemm_kernel.  Its operands are FP32 values split into
// two FP16 terms, t * s = hi + lo with s a power of two that keeps the operand
// inside FP16's normal range (|t| s < 2^13), and it accumulates hi_a hi_b +
// hi_a lo_b + lo_a hi_b in FP32 in tensor memory: 22 significant bits per
// operand, so each product carries ~2^-21 relative error (lo_a lo_b, ~2^-22, is
// dropped) - FP32-GEMM class, at three half-precision MMAs where a BF16 split
// needs six.  Each GEMM's epilogue also writes the split form of the values the
// next GEMM consumes (the panel rows), so no separate conversion pass runs.
//
// Scales: for SPD A every trailing-matrix entry is bounded by max_i A_ii and
// every factor entry by sqrt(max_i A_ii); the leaf measures max |X| itself.
// A matrix that is not SPD reports VMCK_DEV_NOT_SPD from the leaf (the pivot is
// replaced by 1 so the run stays finite); the caller falls back.
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "chol_tc.cuh"
#include "tc_common.cuh"

namespace vmck {

// scales[0] = s(max diag A), scales[1] = s(sqrt(max diag A)); status gets
// NONFINITE for a non-finite diagonal.  One block.
__global__ void __launch_bounds__(256) chol_bounds_kernel(const float *__restrict__ A, int64_t n,
                                                          float *scales, int32_t *status) {
  __shared__ float red[8];
  float m = 0.0f;
  bool bad = false;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
    const float d = A[i + i * n];
    bad |= !isfinite(d);
    m = fmaxf(m, fabsf(d));
  }
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  bad = __syncthreads_or(bad);
  if (threadIdx.x == 0) {
    float t = 0.0f;
    for (int w = 0; w < 8; ++w) t = fmaxf(t, red[w]);
    scales[0] = split_scale(t);
    scales[1] = split_scale(sqrtf(t));
    if (bad && status) atomicOr(status, VMCK_DEV_NONFINITE);
  }
}

// B operand of the first panel GEMM: out[j * ldo + i] = split(A(r0 + i, c0 + j))
// for i < rows (column-major A), zero for i in [rows, ldo).
__global__ void chol_split_rows_kernel(const float *__restrict__ A, int64_t n, int64_t r0,
                                       int64_t c0, int rows, int64_t cols, int ldo,
                                       const float *scales, __half *oh, __half *ol) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= cols * ldo) return;
  const int64_t j = e / ldo;
  const int i = (int)(e - j * ldo);
  __half hi = __float2half_rn(0.0f), lo = hi;
  if (i < rows) split_f16(A[(r0 + i) + (c0 + j) * n], scales[0], hi, lo);
  oh[e] = hi;
  ol[e] = lo;
}

// ------------------------------------------------------------ the GEMM
// C[m + nn ldc] = alpha (A_op B_op^T)(m, nn) / (sa sb) + beta C[m + nn ldc]
// with A_op (M x K) and B_op (N x K) given as split FP16 pairs whose rows are
// K-contiguous (TMA tensors: x = K, y = row).  tri: only m <= nn is written and
// tiles wholly below the diagonal are skipped.  Optional split output of the
// result: oh/ol[(nn - o_col0) ldo + m] = split(value * so) for m < o_rows,
// nn >= o_col0.
//
// Launched with programmatic dependent launch: the prologue (tensor-memory
// allocation, barriers, descriptor prefetch) overlaps the previous kernel of the
// stream.  Persistent and warp-specialised: warp 0 streams 64-wide K slabs of the four
// operand tiles with TMA (128-byte swizzle) into a 2-stage ring; warp 1 issues
// the tcgen05.mma (kind::f16, M = 128, N = 256) from one thread; warps 2-17 hold
// the tile's FP32 sums in registers (64 per thread).
//
// Accumulation.  The tensor core adds each MMA's products into its FP32
// accumulator with a truncating alignment, an error of up to an ulp of the
// running sum per MMA that does not average out: over K = 512 (96 MMAs) it left
// the factor's backward error at ~4e-6 and refinement converging by only ~0.08
// per pass.  Here the large hi * hi products accumulate in tensor memory for one
// 64-wide slab only (4 MMAs, region D1), and the epilogue adds each slab's sum
// to its registers with round-to-nearest FP32 additions; the small cross terms
// hi * lo + lo * hi (2^-11 of the sum) accumulate over the whole tile in region
// D2 (with lolo also lo * lo: the result is then the exact product of the split
// operands up to FP32 summation, so a Gram matrix stays positive semidefinite;
// without it the missing 2^-22 part is a positive semidefinite matrix taken
// away).  The MMA thread issues a slab's cross terms first, so the epilogue drains
// D1 of the previous slab meanwhile.  With beta != 0 the register sums start
// from the old C values, loaded while the tile's first slab runs, so the
// write-out only stores.  Waits for work are bounded by the library's wait limit; a wait that
// runs out sets VMCK_DEV_TIMEOUT and the CTA winds down.
//
// BN = 256 columns per tile; one-row-tile launches (the factorisation's chain, which
// waits for them) take 128 or 64 where the columns then still fit one wave: the
// write-out of a tile (4 + 4 bytes per entry, one SM's stores) is most of such a
// launch, so it shrinks with the tile.  Panel row and next rows at n = 4,096, K =
// 128: 13 and 14 us -> 5 and 7 us (with the split copy stored two rows at a time).
constexpr int G_BM = 128, G_BK = 64, G_STAGES = 2;
constexpr int G_EPI_WARPS = 16;  // four per tensor-memory lane quarter, BN / 4 columns each
constexpr int G_THREADS = 32 * (2 + G_EPI_WARPS);
constexpr int G_A_BYTES = G_BM * G_BK * 2;  // 16 KB (one of hi / lo)
constexpr int G_UMMA_K = 16;
constexpr int G_CHUNK = 8;  // epilogue columns per tensor-memory load
template <int BN>
struct GemmTile {
  static constexpr int TMEM_COLS = 2 * BN;  // D1 (hi * hi, one slab), D2 (cross terms, one tile)
  static constexpr int COLS = BN / 4;       // columns per epilogue warp
  static constexpr int B_BYTES = BN * G_BK * 2;
  static constexpr int STAGE_BYTES = 2 * G_A_BYTES + 2 * B_BYTES;
  static constexpr int BOX = BN < G_BM ? BN : G_BM;  // rows of a B operand copy
};

struct GemmParams {
  int M, N, K;
  int a_row0, b_row0, k_off;  // TMA coordinates of A_op row 0, B_op row 0, first K
  float *C;
  int64_t ldc;
  float alpha, beta;
  const float *sa, *sb;
  int tri;
  int lolo;  // also lo * lo (a Gram matrix of the split operand stays one)
  // split K: tile t of kz * base_tiles covers K range [z kchunk, +kchunk) of
  // output tile t % base_tiles, z = t / base_tiles, into C + z zstride
  int kz, kchunk;
  int64_t zstride, base_tiles;
  __half *oh, *ol;
  int64_t ldo;
  int o_rows, o_col0;
  const float *so;
  int32_t *status;
  unsigned long long wait_ns;
  int mt, nt;
  int64_t tiles;
};

// Tile t -> (mi, ni).  Upper-triangular launches (BN = 2 BM, common origin):
// column tile ni holds row tiles 0 .. min(mt, 2 ni + 2) - 1.  With one row tile
// (any BN) tile t is column tile t.
__device__ __forceinline__ int64_t tri_cum(int64_t ni, int64_t mt) {
  const int64_t h = mt / 2;
  return ni <= h ? ni * (ni + 1) : h * (h + 1) + (ni - h) * mt;
}
__device__ __forceinline__ void gemm_tile(const GemmParams &g, int64_t t, int &mi, int &ni) {
  if (g.mt == 1) {
    mi = 0;
    ni = (int)t;
    return;
  }
  if (!g.tri) {
    mi = (int)(t % g.mt);
    ni = (int)(t / g.mt);
    return;
  }
  int lo = 0, hi = g.nt - 1;  // largest ni with tri_cum(ni) <= t
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (tri_cum(mid, g.mt) <= t) lo = mid;
    else hi = mid - 1;
  }
  ni = lo;
  mi = (int)(t - tri_cum(lo, g.mt));
}

// Tile t -> (mi, ni), its K slab range [kb0, kb0 + nkb) and output C.
__device__ __forceinline__ void gemm_work(const GemmParams &g, int64_t t, int &mi, int &ni,
                                          int &kb0, int &nkb, float *&C) {
  if (g.kz == 1) {  // no split: skip the 64-bit division
    gemm_tile(g, t, mi, ni);
    kb0 = 0;
    nkb = (g.K + G_BK - 1) / G_BK;
    C = g.C;
    return;
  }
  const int64_t z = t / g.base_tiles;
  gemm_tile(g, t - z * g.base_tiles, mi, ni);
  const int k0 = (int)z * g.kchunk;
  const int k1 = min(g.K, k0 + g.kchunk);
  kb0 = k0 / G_BK;
  nkb = (k1 - k0 + G_BK - 1) / G_BK;
  C = g.C + z * g.zstride;
}

template <int BN>
__global__ void __launch_bounds__(G_THREADS, 1)
    tc_gemm_kernel(const __grid_constant__ CUtensorMap mAh, const __grid_constant__ CUtensorMap mAl,
                   const __grid_constant__ CUtensorMap mBh, const __grid_constant__ CUtensorMap mBl,
                   GemmParams g) {
  constexpr int G_BN = BN, G_TMEM_COLS = GemmTile<BN>::TMEM_COLS, G_COLS = GemmTile<BN>::COLS;
  constexpr int G_B_BYTES = GemmTile<BN>::B_BYTES, G_STAGE_BYTES = GemmTile<BN>::STAGE_BYTES;
  constexpr int G_NCH = G_COLS / G_CHUNK;
  extern __shared__ __align__(1024) unsigned char g_smem_raw[];
  unsigned char *smem = reinterpret_cast<unsigned char *>(
      (reinterpret_cast<uintptr_t>(g_smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + G_STAGES * G_STAGE_BYTES);
  uint64_t *empty = full + G_STAGES;
  uint64_t *d1_full = empty + G_STAGES;
  uint64_t *d1_empty = d1_full + 1;
  uint64_t *d2_full = d1_empty + 1;
  uint64_t *d2_empty = d2_full + 1;
  uint64_t *drain = d2_empty + 1;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drain + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0)
    *abort_flag =
        (g.status && (*reinterpret_cast<volatile int32_t *>(g.status) & VMCK_DEV_TIMEOUT)) ? 1 : 0;
  __syncthreads();
  if (*abort_flag) return;
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(G_TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int s = 0; s < G_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(d1_full, 1);
    mbar_init(d1_empty, G_EPI_WARPS);
    mbar_init(d2_full, 1);
    mbar_init(d2_empty, G_EPI_WARPS);
    mbar_init(drain, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&mAh)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&mAl)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&mBh)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&mBl)) : "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // the prologue above overlaps the previous kernel of the stream; its output
  // (operands, C) is read only from here on
  pdl_wait();
  pdl_trigger();

  auto fail = [&]() {
    if (g.status) atomicOr(g.status, VMCK_DEV_TIMEOUT);
    *abort_flag = 1;
  };

  if (warp == 0) {
    // ---------------- TMA producer
    if (lane == 0) {
      int64_t it = 0;
      for (int64_t tile = blockIdx.x; tile < g.tiles && !*abort_flag; tile += gridDim.x) {
        int mi, ni, kb0, num_kb;
        float *Ct;
        gemm_work(g, tile, mi, ni, kb0, num_kb, Ct);
        const int ya = g.a_row0 + mi * G_BM, yb = g.b_row0 + ni * G_BN;
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = (int)(it % G_STAGES);
          if (it >= G_STAGES &&
              !mbar_wait(&empty[s], (uint32_t)(((it / G_STAGES) - 1) & 1), g.wait_ns)) {
            fail();
            break;
          }
          if (*abort_flag) break;
          unsigned char *st = smem + s * G_STAGE_BYTES;
          const int x = g.k_off + (kb0 + kb) * G_BK;
          mbar_expect_tx(&full[s], G_STAGE_BYTES);
          tma_load_2d(st, &mAh, &full[s], x, ya);
          tma_load_2d(st + G_A_BYTES, &mAl, &full[s], x, ya);
          constexpr int BOX = GemmTile<BN>::BOX;
#pragma unroll
          for (int r = 0; r < G_BN; r += BOX) {
            tma_load_2d(st + 2 * G_A_BYTES + r * G_BK * 2, &mBh, &full[s], x, yb + r);
            tma_load_2d(st + 2 * G_A_BYTES + G_B_BYTES + r * G_BK * 2, &mBl, &full[s], x, yb + r);
          }
        }
      }
      // every copy issued must land before the CTA may exit
      const int64_t first = it > G_STAGES ? it - G_STAGES : 0;
      for (int64_t q = first; q < it; ++q)
        mbar_wait(&full[q % G_STAGES], (uint32_t)((q / G_STAGES) & 1));
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer
    if (lane == 0) {
      const uint32_t idesc = umma_idesc_f16(G_BM, G_BN);
      const uint32_t d1 = tmem_base, d2 = tmem_base + G_BN;
      int64_t it = 0, slab = 0, tcount = 0;
      bool issued_any = false, ok = true;
      for (int64_t tile = blockIdx.x; tile < g.tiles && ok && !*abort_flag;
           tile += gridDim.x, ++tcount) {
        if (tcount > 0 && !mbar_wait(d2_empty, (uint32_t)((tcount - 1) & 1), g.wait_ns)) {
          fail();
          break;
        }
        tc_fence_after();
        int mi, ni, kb0, num_kb;
        float *Ct;
        gemm_work(g, tile, mi, ni, kb0, num_kb, Ct);
        for (int kb = 0; kb < num_kb; ++kb, ++it, ++slab) {
          const int s = (int)(it % G_STAGES);
          if (!mbar_wait(&full[s], (uint32_t)((it / G_STAGES) & 1), g.wait_ns)) {
            fail();
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t ah = smem_u32(smem + s * G_STAGE_BYTES);
          const uint32_t al = ah + G_A_BYTES, bh = ah + 2 * G_A_BYTES, bl = bh + G_B_BYTES;
          // cross terms of this slab into D2 (accumulates over the tile)
#pragma unroll
          for (int k = 0; k < G_BK / G_UMMA_K; ++k) {
            const uint32_t off = k * G_UMMA_K * 2;
            umma_f16(d2, umma_desc_sw128(ah + off), umma_desc_sw128(bl + off), idesc,
                     (kb == 0 && k == 0) ? 0u : 1u);
            umma_f16(d2, umma_desc_sw128(al + off), umma_desc_sw128(bh + off), idesc, 1u);
            if (g.lolo)
              umma_f16(d2, umma_desc_sw128(al + off), umma_desc_sw128(bl + off), idesc, 1u);
          }
          // hi * hi of this slab into D1 once the epilogue has read the last slab
          if (slab > 0 && !mbar_wait(d1_empty, (uint32_t)((slab - 1) & 1), g.wait_ns)) {
            fail();
            ok = false;
            issued_any = true;
            break;
          }
          tc_fence_after();
#pragma unroll
          for (int k = 0; k < G_BK / G_UMMA_K; ++k) {
            const uint32_t off = k * G_UMMA_K * 2;
            umma_f16(d1, umma_desc_sw128(ah + off), umma_desc_sw128(bh + off), idesc,
                     k == 0 ? 0u : 1u);
          }
          umma_commit(&empty[s]);
          umma_commit(d1_full);
          issued_any = true;
        }
        if (!ok) break;
        umma_commit(d2_full);
      }
      if (issued_any) {
        umma_commit(drain);
        mbar_wait(drain, 0);
      }
    }
  } else {
    // ---------------- epilogue: warp e reads TMEM lane quarter (warp & 3),
    // columns [64 * (e >> 2), +64) of the 256-column tile
    const int e = warp - 2, quarter = warp & 3, part = e >> 2;
    const float inv_s = 1.0f / ((g.sa ? *g.sa : 1.0f) * (g.sb ? *g.sb : 1.0f));
    const float alpha = g.alpha * inv_s;  // a power of two times +-1: exact scaling
    const float cscale = g.beta / alpha;  // old C in units of the sums
    const float so = g.so ? *g.so : 1.0f;
    const uint32_t lane_off = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t t1 = tmem_base + lane_off + (uint32_t)(part * G_COLS);
    const uint32_t t2 = t1 + G_BN;
    int64_t tcount = 0, slab = 0;
    bool alive = true;
    for (int64_t tile = blockIdx.x; tile < g.tiles && alive; tile += gridDim.x, ++tcount) {
      int mi, ni, kb0, num_kb;
      float *Ct;
      gemm_work(g, tile, mi, ni, kb0, num_kb, Ct);
      const int m = mi * G_BM + quarter * 32 + lane;
      const int nbase = ni * G_BN + part * G_COLS;
      const bool row_ok = m < g.M;
      float *Crow = Ct + m;
      // the sums start from the old C values (loaded while the first slab's MMAs
      // run), so the write-out only stores
      float acc[G_COLS];
      if (g.beta != 0.0f) {
        const float *cp = Crow + (int64_t)nbase * g.ldc;
#pragma unroll
        for (int i = 0; i < G_COLS; ++i) {
          const int nn = nbase + i;
          acc[i] = (row_ok && nn < g.N && (!g.tri || m <= nn)) ? *cp * cscale : 0.0f;
          cp += g.ldc;
        }
      } else {
#pragma unroll
        for (int i = 0; i < G_COLS; ++i) acc[i] = 0.0f;
      }
      for (int kb = 0; kb < num_kb; ++kb, ++slab) {
        if (!mbar_wait(d1_full, (uint32_t)(slab & 1), g.wait_ns)) {
          fail();
          alive = false;
          break;
        }
        tc_fence_after();
#pragma unroll
        for (int ch = 0; ch < G_NCH; ++ch) {
          float v[G_CHUNK];
          tmem_ld_8cols(t1 + ch * G_CHUNK, v);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < G_CHUNK; ++j) acc[ch * G_CHUNK + j] += v[j];
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(d1_empty);
      }
      if (!alive) break;
      if (!mbar_wait(d2_full, (uint32_t)(tcount & 1), g.wait_ns)) {
        fail();
        break;
      }
      tc_fence_after();
#pragma unroll
      for (int ch = 0; ch < G_NCH; ++ch) {
        float v[G_CHUNK];
        tmem_ld_8cols(t2 + ch * G_CHUNK, v);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < G_CHUNK; ++j) acc[ch * G_CHUNK + j] += v[j];
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(d2_empty);
      // write-out (stores only).  The split copy goes out two rows at a time: lane
      // pairs exchange one column each, so an even lane stores rows m, m + 1 of the
      // even column and an odd lane rows m - 1, m of the odd one
      float *cp = Crow + (int64_t)nbase * g.ldc;
      const bool odd = lane & 1;
#pragma unroll
      for (int i = 0; i < G_COLS; i += 2) {
        const int nn = nbase + i;
        const float v0 = alpha * acc[i], v1 = alpha * acc[i + 1];
        if (row_ok && nn < g.N && (!g.tri || m <= nn)) *cp = v0;
        if (row_ok && nn + 1 < g.N && (!g.tri || m <= nn + 1)) cp[g.ldc] = v1;
        cp += 2 * g.ldc;
        if (g.oh && nn + 1 >= g.o_col0) {  // warp-uniform
          __half h0, l0, h1, l1;
          split_f16(v0, so, h0, l0);
          split_f16(v1, so, h1, l1);
          const __half2 mine = odd ? __halves2half2(h1, l1) : __halves2half2(h0, l0);
          const __half2 give = odd ? __halves2half2(h0, l0) : __halves2half2(h1, l1);
          const __half2 got = __shfl_xor_sync(0xffffffffu, give, 1);
          const __half2 first = odd ? got : mine, second = odd ? mine : got;  // rows in order
          const int c = nn + (odd ? 1 : 0), m0 = m & ~1;
          const int rows = min(g.o_rows, g.tri ? min(g.M, c + 1) : g.M);
          if (c < g.N && c >= g.o_col0 && m0 < rows) {
            const int64_t o = (int64_t)(c - g.o_col0) * g.ldo + m0;
            if (m0 + 1 < rows) {
              *reinterpret_cast<__half2 *>(g.oh + o) = __lows2half2(first, second);
              *reinterpret_cast<__half2 *>(g.ol + o) = __highs2half2(first, second);
            } else {
              g.oh[o] = __low2half(first);
              g.ol[o] = __high2half(first);
            }
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
                 "r"(G_TMEM_COLS)
                 : "memory");
  }
}

// ------------------------------------------------------------ the leaf
// One CTA factors the mp x mp (mp <= 128) diagonal block at (r0, r0) of the
// column-major upper A in shared memory, A = U^T U, and forms X = U^-1.  Per 32-row
// panel p:
//   (a) warp 0 factors the 32 x 32 diagonal block, lane l holding column l in
//       registers, four pivots at a time: every lane factors the 4 x 4 pivot block
//       from a shared-memory broadcast (no shuffle in the pivot chain) and solves its
//       own four entries, and the rows below get one rank-4 update with a row's four
//       multipliers in one 16-byte broadcast.  The next four rows are updated first,
//       so their pivot chain overlaps the update of the others; the rows shift down
//       four registers per step, so the step loop has one compact body;
//   (b) the panel row U_pp^-T A_p,j by forward substitution, one thread per column;
//   (c) the rank-32 update of the trailing block in 4 x 4 register tiles: the next
//       diagonal block first, so that warp 0 goes on to its (a) while the other
//       warps update the rest;
//   (d) meanwhile warp 7 inverts U_pp (lane l solves U x = e_l from the bottom row
//       up).
// The off-diagonal blocks X_IJ = -X_II sum_K U_IK X_KJ follow as far as they can
// behind the last factor and inversion, then the last block column, four warps a
// block (one warp issues an FMA every 1.75 clocks; with eight warps the operands'
// shared-memory reads bound it).
// Every entry takes the same operations in the same order as a right-looking
// elimination one pivot at a time would give it.
// Writes U in place, X split into K-contiguous rows (xh/xl[m * 128 + k] = X(k, m),
// scale from max |X| into *scale_x) and Y = X^T zero-padded column-major
// 128 x 128 (the refinement's triangular solves).  Rows / columns past mp are
// the identity.  A non-positive or NaN pivot raises VMCK_DEV_NOT_SPD and is
// replaced by 1.
//
// One SM is busy and 128 of these are in a row at n = 16,384, so only its latency
// counts: 62,000 clocks, 33 us (50 us with one pivot at a time in one warp and each
// phase after the other; of these now: load 4, factors 23, panel rows and updates 9,
// X 16, outputs 9 thousand).
constexpr int LB = 128, LLD = LB + 4, LEAF_T = 256;
constexpr int LRD = 36;  // row stride of a diagonal block's shifted rows
constexpr size_t CHOL_LEAF_SMEM =
    (size_t)(2 * LB * LLD + 2 * 32 * LRD + 3 * 32 * LRD + LB + 4 * 32 + 4 * 64) * sizeof(float);

// All threads, or the seven warps that factor.
__device__ __forceinline__ void leaf_sync_all() { __syncthreads(); }
__device__ __forceinline__ void leaf_sync_main() {
  asm volatile("bar.sync 1, 224;" ::: "memory");
}

// The 4 x 4 pivot block (columns a0 .. a3, upper part) of the four rows c: the lane's
// own entries of U in v, the inverse roots in inv.
struct LeafPivots {
  float v[4], inv[4];
  int bad;  // bit m: pivot m was not positive and is replaced by 1
};
__device__ __forceinline__ LeafPivots leaf_pivots(const float4 &a0, const float4 &a1,
                                                  const float4 &a2, const float4 &a3,
                                                  const float (&c)[4]) {
  LeafPivots p;
  p.bad = 0;
  auto root = [&](float d, int m) {
    if (!(d > 0.0f)) {
      p.bad |= 1 << m;
      d = 1.0f;
    }
    return rsqrtf(d);
  };
  const float i0 = root(a0.x, 0);
  const float u01 = a1.x * i0, u02 = a2.x * i0, u03 = a3.x * i0;
  const float i1 = root(fmaf(-u01, u01, a1.y), 1);
  const float u12 = fmaf(-u01, u02, a2.y) * i1, u13 = fmaf(-u01, u03, a3.y) * i1;
  const float i2 = root(fmaf(-u12, u12, fmaf(-u02, u02, a2.z)), 2);
  const float u23 = fmaf(-u12, u13, fmaf(-u02, u03, a3.z)) * i2;
  const float i3 = root(fmaf(-u23, u23, fmaf(-u13, u13, fmaf(-u03, u03, a3.w))), 3);
  p.v[0] = c[0] * i0;
  p.v[1] = fmaf(-u01, p.v[0], c[1]) * i1;
  p.v[2] = fmaf(-u12, p.v[1], fmaf(-u02, p.v[0], c[2])) * i2;
  p.v[3] = fmaf(-u23, p.v[2], fmaf(-u13, p.v[1], fmaf(-u03, p.v[0], c[3]))) * i3;
  p.inv[0] = i0;
  p.inv[1] = i1;
  p.inv[2] = i2;
  p.inv[3] = i3;
  return p;
}

// (a): U_pp into S, its rows shifted left of their diagonal into shifted[k][q] =
// U(k, k + 1 + q) (zero past the block), 1 / U(k, k) into rd.  Returns whether a
// pivot was replaced.
__device__ __forceinline__ bool leaf_factor32(float *S, int P, float *shifted, float *rd,
                                              float *piv, float *mul) {
  const int lane = threadIdx.x & 31;
  // at step k0, c[i] holds row k0 + i of column P + lane
  float c[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) c[i] = S[(P + i) * LLD + P + lane];
#pragma unroll
  for (int i = 0; i < 32; ++i) shifted[i * LRD + lane] = 0.0f;
  int bad = 0;
  const float4 *pv = reinterpret_cast<const float4 *>(piv);
  const float4 *mv = reinterpret_cast<const float4 *>(mul);
  *reinterpret_cast<float4 *>(piv + 4 * lane) = make_float4(c[0], c[1], c[2], c[3]);
  __syncwarp();
  LeafPivots f;
  {
    const float c4[4] = {c[0], c[1], c[2], c[3]};
    f = leaf_pivots(pv[0], pv[1], pv[2], pv[3], c4);
  }
#pragma unroll 1
  for (int k0 = 0; k0 < 32; k0 += 4) {
    bad |= f.bad;  // (not the pivots formed past the last row)
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int k = k0 + m;
      if (lane < k) f.v[m] = 0.0f;  // left of the diagonal
      if (lane == k && ((f.bad >> m) & 1)) f.v[m] = 1.0f;
      S[(P + k) * LLD + P + lane] = f.v[m];
      if (lane > k) shifted[k * LRD + lane - k - 1] = f.v[m];
      if (lane == k) rd[P + k] = f.inv[m];
    }
    __syncwarp();  // the last step's readers of mul are done
    *reinterpret_cast<float4 *>(mul + 4 * lane) = make_float4(f.v[0], f.v[1], f.v[2], f.v[3]);
    __syncwarp();
    // rows k0 + 4 .. k0 + 7 first: their pivot chain overlaps the other rows
    float c4[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 m = mv[k0 + 4 + i];
      c4[i] = fmaf(-m.w, f.v[3], fmaf(-m.z, f.v[2], fmaf(-m.y, f.v[1],
                                                         fmaf(-m.x, f.v[0], c[4 + i]))));
    }
    *reinterpret_cast<float4 *>(piv + 4 * lane) = make_float4(c4[0], c4[1], c4[2], c4[3]);
    __syncwarp();
    const int k1 = (k0 + 4) & 31;
    const LeafPivots next = leaf_pivots(pv[k1], pv[k1 + 1], pv[k1 + 2], pv[k1 + 3], c4);
#pragma unroll
    for (int i = 8; i < 32; ++i) {
      const float4 m = mv[k0 + i];  // rows past the block: zeros, never used
      c[i - 4] = fmaf(-m.w, f.v[3], fmaf(-m.z, f.v[2], fmaf(-m.y, f.v[1],
                                                            fmaf(-m.x, f.v[0], c[i]))));
    }
    f = next;
  }
  return bad != 0;
}

// (d): X_pp = U_pp^-1 by back substitution, lane l solving U x = e_l; x[q] holds row
// i + 1 + q at row i (rows past the block are 0).  Four rows per body, so the rows
// shift four registers at a time.  Returns max |X| over the valid columns.
__device__ __forceinline__ float leaf_invert32(float *X, int P, const float *shifted,
                                               const float *rd, int mp) {
  const int lane = threadIdx.x & 31;
  float am = 0.0f;
  float x[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) x[i] = 0.0f;
#pragma unroll 1
  for (int s = 0; s < 32; s += 4) {
    float n[4];  // the body's rows, newest first
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int i = 31 - s - m;
      const float4 *row = reinterpret_cast<const float4 *>(shifted + i * LRD);
      float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int q4 = 0; q4 < 8; ++q4) {
        const float4 u4 = row[q4];
        const float u[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int q = 4 * q4 + t;  // row i + 1 + q: q < m from this body
          if (q < m) a[t] = fmaf(u[t], n[m - 1 - q], a[t]);
          else if (q - m < 32) a[t] = fmaf(u[t], x[q - m], a[t]);
        }
      }
      const float ri = rd[P + i];
      const float xi = (i == lane) ? ri : (i < lane ? -((a[0] + a[1]) + (a[2] + a[3])) * ri : 0.0f);
      X[(P + i) * LLD + P + lane] = xi;
      if (P + lane < mp) am = fmaxf(am, fabsf(xi));
      n[m] = xi;
    }
#pragma unroll
    for (int q = 31; q >= 4; --q) x[q] = x[q - 4];
#pragma unroll
    for (int q = 0; q < 4; ++q) x[q] = n[3 - q];
  }
  return am;
}

// Threads of two (b: 2) or four warps.
__device__ __forceinline__ void leaf_sync_pair() { asm volatile("bar.sync 2, 64;" ::: "memory"); }
__device__ __forceinline__ void leaf_sync_four() { asm volatile("bar.sync 3, 128;" ::: "memory"); }

// 2 x 4 outputs (rows r2 .., columns c4 ..) of A B, K a multiple of 4: A row-major
// (ld la), B row-major (ld lb).
__device__ __forceinline__ void leaf_product(const float *A, int la, const float *B, int lb,
                                             int K, int r2, int c4, float (&acc)[2][4]) {
  const float *ar = A + r2 * la, *bc = B + c4;
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[r][q] = 0.0f;
#pragma unroll 4
  for (int k = 0; k < K; k += 4) {
    const float4 a0 = *reinterpret_cast<const float4 *>(ar + k);
    const float4 a1 = *reinterpret_cast<const float4 *>(ar + la + k);
    const float x0[4] = {a0.x, a0.y, a0.z, a0.w}, x1[4] = {a1.x, a1.y, a1.z, a1.w};
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const float4 v = *reinterpret_cast<const float4 *>(bc + (k + m) * lb);
      acc[0][0] = fmaf(x0[m], v.x, acc[0][0]);
      acc[0][1] = fmaf(x0[m], v.y, acc[0][1]);
      acc[0][2] = fmaf(x0[m], v.z, acc[0][2]);
      acc[0][3] = fmaf(x0[m], v.w, acc[0][3]);
      acc[1][0] = fmaf(x1[m], v.x, acc[1][0]);
      acc[1][1] = fmaf(x1[m], v.y, acc[1][1]);
      acc[1][2] = fmaf(x1[m], v.z, acc[1][2]);
      acc[1][3] = fmaf(x1[m], v.w, acc[1][3]);
    }
  }
}

// S(i0 .., j0 ..) -= U(P .., i0 ..)^T U(P .., j0 ..), a 4 x 4 tile.  (Below the
// diagonal of a diagonal block: entries nothing reads.)
__device__ __forceinline__ void leaf_update_tile(float *S, int P, int i0, int j0) {
  float acc[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const float4 v = *reinterpret_cast<const float4 *>(S + (i0 + r) * LLD + j0);
    acc[r][0] = v.x, acc[r][1] = v.y, acc[r][2] = v.z, acc[r][3] = v.w;
  }
#pragma unroll 4
  for (int k = 0; k < 32; ++k) {
    const float *row = S + (P + k) * LLD;
    const float4 av = *reinterpret_cast<const float4 *>(row + i0);
    const float4 bv = *reinterpret_cast<const float4 *>(row + j0);
    const float a[4] = {av.x, av.y, av.z, av.w}, bq[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[r][q] = fmaf(-a[r], bq[q], acc[r][q]);
  }
#pragma unroll
  for (int r = 0; r < 4; ++r)
    *reinterpret_cast<float4 *>(S + (i0 + r) * LLD + j0) =
        make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
}

__global__ void __launch_bounds__(LEAF_T, 1) chol_leaf_kernel(float *__restrict__ A, int64_t n,
                                                           int64_t r0, int mp,
                                                           __half *__restrict__ xh,
                                                           __half *__restrict__ xl,
                                                           float *scale_x, float *__restrict__ yinv,
                                                           int32_t *status) {
  extern __shared__ __align__(16) float lsm[];
  float *S = lsm;                       // S[i * LLD + j]: A, then U(i, j), i <= j
  float *X = S + LB * LLD;              // X[i * LLD + j] = U^-1(i, j), blocks I <= J only
  float *shifted = X + LB * LLD;        // two panels' U_pp rows (factor / inversion overlap)
  float *Tb = shifted + 2 * 32 * LRD;   // 3 x [32][LRD] temporaries of the inverse
  float *rd = Tb + 3 * 32 * LRD;        // rd[i] = 1 / U(i, i)
  float *piv = rd + LB;                 // 32 x float4: the four pivot rows' columns
  float *mul = piv + 4 * 32;            // 64 x float4: four multipliers of each row
  __shared__ float red[LEAF_T / 32];
  __shared__ int not_spd;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) not_spd = 0;
  for (int e = tid; e < 4 * 64; e += LEAF_T) mul[e] = 0.0f;
  pdl_wait();  // the block was written by the previous kernel of the stream
  pdl_trigger();
  // lane = row i of block row warp & 3, columns 8 u + 4 (warp >> 2) + q
  const int li = 32 * (warp & 3) + lane, lj = 4 * (warp >> 2);
  {
    float v[16][4];  // all of a thread's loads in flight at once
    const float *col = A + (r0 + li) + (r0 + lj) * n;
#pragma unroll
    for (int u = 0; u < 16; ++u)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int j = lj + 8 * u + q;
        v[u][q] = li == j ? 1.0f : 0.0f;
        if (li <= j && j < mp) v[u][q] = col[(8 * u + q) * n];
      }
#pragma unroll
    for (int u = 0; u < 16; ++u)
      *reinterpret_cast<float4 *>(S + li * LLD + lj + 8 * u) =
          make_float4(v[u][0], v[u][1], v[u][2], v[u][3]);
  }
  leaf_sync_all();
  float am = 0.0f;  // max |X| over the valid block (this thread's writes)
  // off-diagonal block X_IJ by 128 threads (t)
  auto x_block = [&](int I, int J, int t) {
    const int r2 = 2 * (t >> 3), c4 = 4 * (t & 7);
    float acc[2][4];
    float *T = Tb + I * 32 * LRD;
    leaf_product(S + 32 * I * LLD + 32 * (I + 1), LLD, X + 32 * (I + 1) * LLD + 32 * J, LLD,
                 32 * (J - I), r2, c4, acc);
#pragma unroll
    for (int r = 0; r < 2; ++r)
      *reinterpret_cast<float4 *>(T + (r2 + r) * LRD + c4) =
          make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
    leaf_sync_four();
    leaf_product(X + 32 * I * LLD + 32 * I, LLD, T, LRD, 32, r2, c4, acc);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      *reinterpret_cast<float4 *>(X + (32 * I + r2 + r) * LLD + 32 * J + c4) =
          make_float4(-acc[r][0], -acc[r][1], -acc[r][2], -acc[r][3]);
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (32 * J + c4 + q < mp) am = fmaxf(am, fabsf(acc[r][q]));
    }
    leaf_sync_four();
  };
  auto factor = [&](int p) {
    if (leaf_factor32(S, 32 * p, shifted + (p & 1) * 32 * LRD, rd, piv, mul) && lane == 0)
      not_spd = 1;
  };
  if (warp == 0) factor(0);
#pragma unroll 1
  for (int p = 0; p < 4; ++p) {
    const int P = 32 * p;
    leaf_sync_all();  // (a) of this panel and (c) of the last one are done
    if (warp == 7) {
      am = fmaxf(am, leaf_invert32(X, P, shifted + (p & 1) * 32 * LRD, rd, mp));
      continue;
    }
    const int ncols = LB - P - 32;
    if (ncols == 0) break;
    // (b) one thread per column right of the block
    if (tid < ncols) {
      float *col = S + P * LLD + P + 32 + tid;
      float y[32];
#pragma unroll
      for (int r = 0; r < 32; ++r) y[r] = col[r * LLD];
#pragma unroll
      for (int k = 0; k < 32; ++k) {
        y[k] *= rd[P + k];
        const float *urow = S + (P + k) * LLD + P;  // U(k, r) = urow[r]
#pragma unroll
        for (int r4 = 4 * (k / 4); r4 < 32; r4 += 4) {
          const float4 u = *reinterpret_cast<const float4 *>(urow + r4);
          if (r4 > k) y[r4] = fmaf(-u.x, y[k], y[r4]);
          if (r4 + 1 > k) y[r4 + 1] = fmaf(-u.y, y[k], y[r4 + 1]);
          if (r4 + 2 > k) y[r4 + 2] = fmaf(-u.z, y[k], y[r4 + 2]);
          if (r4 + 3 > k) y[r4 + 3] = fmaf(-u.w, y[k], y[r4 + 3]);
        }
      }
#pragma unroll
      for (int r = 0; r < 32; ++r) col[r * LLD] = y[r];
    }
    leaf_sync_main();
    // (c) the next diagonal block by warps 0 and 1, then warp 0 factors it
    const int base = P + 32;
    if (warp < 2) {
      leaf_update_tile(S, P, base + 4 * (tid >> 3), base + 4 * (tid & 7));
      leaf_sync_pair();
    }
    if (warp == 0) {
      factor(p + 1);
    } else {
      // the other blocks (i <= j, not the first): 64 tiles each, warps 1 .. 6
      const int below = 3 - p, tiles = 64 * (below * (below + 1) / 2 - 1);
#pragma unroll 1
      for (int t = tid - 32; t < tiles; t += 192) {
        int blk = 1 + (t >> 6), bi = 0;
        while (blk >= below - bi) blk -= below - bi++;
        leaf_update_tile(S, P, base + 32 * bi + 4 * ((t >> 3) & 7),
                         base + 32 * (bi + blk) + 4 * (t & 7));
      }
      // behind the last factor: X_01 (X_00 and X_11 are there)
      if (p == 2 && warp >= 3) x_block(0, 1, tid - 96);
    }
  }
  // behind the last inversion: X_12 and X_02; then the last block column
  if (warp < 4) {
    x_block(1, 2, tid);
    x_block(0, 2, tid);
  }
  leaf_sync_all();  // X_33 too
  if (warp < 4) {
#pragma unroll 1
    for (int I = 2; I >= 0; --I) x_block(I, 3, tid);
  }
  leaf_sync_all();
  // max |X| over the valid block -> split scale
  for (int o = 16; o > 0; o >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
  if (lane == 0) red[warp] = am;
  __syncthreads();
  float amax = 0.0f;
#pragma unroll
  for (int w = 0; w < LEAF_T / 32; ++w) amax = fmaxf(amax, red[w]);
  const float sx = split_scale(amax);
  if (tid == 0) {
    *scale_x = sx;
    if (not_spd && status) atomicOr(status, VMCK_DEV_NOT_SPD);
  }
  // outputs.  X split: lane = two rows, four columns at a time; the blocks of the
  // operand that are zero for every leaf were cleared once by the caller
  for (int t = warp; t < 64; t += LEAF_T / 32) {
    const int i = 64 * (t & 1) + 2 * lane, j0 = 4 * (t >> 1);
    if (64 * (t & 1) > j0 + 3) continue;
    const float4 x0 = *reinterpret_cast<const float4 *>(X + i * LLD + j0);
    const float4 x1 = *reinterpret_cast<const float4 *>(X + (i + 1) * LLD + j0);
    const float a[4] = {x0.x, x0.y, x0.z, x0.w}, c[4] = {x1.x, x1.y, x1.z, x1.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int j = j0 + q;  // row j of the split operand = column j of X
      __half h0 = __float2half_rn(0.0f), l0 = h0, h1 = h0, l1 = h0;
      if (j < mp && i <= j) split_f16(a[q], sx, h0, l0);
      if (j < mp && i + 1 <= j) split_f16(c[q], sx, h1, l1);
      *reinterpret_cast<__half2 *>(xh + j * LB + i) = __halves2half2(h0, h1);
      *reinterpret_cast<__half2 *>(xl + j * LB + i) = __halves2half2(l0, l1);
    }
  }
  {
    float *col = A + (r0 + li) + (r0 + lj) * n;
#pragma unroll 4
    for (int u = 0; u < 16; ++u) {
      if (32 * (warp & 3) > lj + 8 * u + 3) continue;  // below the diagonal
      const float4 v = *reinterpret_cast<const float4 *>(S + li * LLD + lj + 8 * u);
      const float us[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int j = lj + 8 * u + q;
        if (li <= j && j < mp) col[(8 * u + q) * n] = us[q];
      }
    }
  }
  for (int c = warp; c < LB; c += LEAF_T / 32) {
    const int r = 4 * lane;  // Y(r, c) = X(c, r); above the diagonal cleared by the caller
    if (r + 3 < c) continue;
    const float4 v = *reinterpret_cast<const float4 *>(X + c * LLD + r);
    *reinterpret_cast<float4 *>(yinv + c * LB + r) =
        make_float4(r < mp && c <= r ? v.x : 0.0f, r + 1 < mp && c <= r + 1 ? v.y : 0.0f,
                    r + 2 < mp && c <= r + 2 ? v.z : 0.0f, r + 3 < mp && c <= r + 3 ? v.w : 0.0f);
  }
}

// ------------------------------------------------------------ host side
static int make_f16_map(CUtensorMap *map, const __half *base, int64_t kdim, int64_t rows,
                        int64_t ld, int box_rows) {
  auto fn = encode_fn();
  if (!fn) {
    set_last_error("cuTensorMapEncodeTiled is unavailable");
    return VMCK_ERR_CUDA;
  }
  cuuint64_t dims[2] = {(cuuint64_t)kdim, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)(ld * 2)};
  cuuint32_t box[2] = {(cuuint32_t)G_BK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half *>(base), dims,
                  strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_last_error("cuTensorMapEncodeTiled failed (%d)", (int)r);
    return VMCK_ERR_CUDA;
  }
  return VMCK_OK;
}


static int num_sms_dev() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

template <int BN>
static int launch_gemm(cudaStream_t st, const SplitOperand &a, const SplitOperand &b,
                       GemmParams g, int sms) {
  CUtensorMap mAh, mAl, mBh, mBl;
  int rc;
  constexpr int box = GemmTile<BN>::BOX;
  if ((rc = make_f16_map(&mAh, a.hi, a.kdim, a.rows, a.ld, G_BM))) return rc;
  if ((rc = make_f16_map(&mAl, a.lo, a.kdim, a.rows, a.ld, G_BM))) return rc;
  if ((rc = make_f16_map(&mBh, b.hi, b.kdim, b.rows, b.ld, box))) return rc;
  if ((rc = make_f16_map(&mBl, b.lo, b.kdim, b.rows, b.ld, box))) return rc;
  g.mt = (g.M + G_BM - 1) / G_BM;
  g.nt = (g.N + BN - 1) / BN;
  if (g.tri && g.mt > 1) {
    const int64_t h = g.mt / 2;
    g.base_tiles = g.nt <= h ? (int64_t)g.nt * (g.nt + 1) : h * (h + 1) + (int64_t)(g.nt - h) * g.mt;
  } else {
    g.base_tiles = (int64_t)g.mt * g.nt;
  }
  g.tiles = g.base_tiles * g.kz;
  const size_t smem = 1024 + G_STAGES * GemmTile<BN>::STAGE_BYTES + 8 * 16 + 64;
  VMCK_CUDA(cudaFuncSetAttribute(tc_gemm_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
  const unsigned grid = (unsigned)std::min<int64_t>(g.tiles, sms);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(G_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  VMCK_CUDA(cudaLaunchKernelEx(&cfg, tc_gemm_kernel<BN>, mAh, mAl, mBh, mBl, g));
  return check_launch("tc_gemm");
}

int tc_gemm(cudaStream_t st, const SplitOperand &a, int a_row0, const SplitOperand &b, int b_row0,
            int k_off, int M, int N, int K, float *C, int64_t ldc, float alpha, float beta,
            const float *sa, const float *sb, int tri, __half *oh, __half *ol, int64_t ldo,
            int o_rows, int o_col0, const float *so, int32_t *status, int max_ctas, int lolo,
            int kchunk, int64_t zstride) {
  if (M <= 0 || N <= 0 || K <= 0) return VMCK_OK;
  if (kchunk <= 0 || kchunk >= K) kchunk = K;
  if (kchunk < K && (kchunk % G_BK != 0 || tri || oh || beta != 0.0f)) {
    set_last_error("tc_gemm: split K needs kchunk %% %d == 0, no tri / split output / beta", G_BK);
    return VMCK_ERR_ARG;
  }
  GemmParams g{};
  g.M = M;
  g.N = N;
  g.K = K;
  g.a_row0 = a_row0;
  g.b_row0 = b_row0;
  g.k_off = k_off;
  g.C = C;
  g.ldc = ldc;
  g.alpha = alpha;
  g.beta = beta;
  g.sa = sa;
  g.sb = sb;
  g.tri = tri;
  g.lolo = lolo;
  g.oh = oh;
  g.ol = ol;
  g.ldo = ldo;
  g.o_rows = o_rows;
  g.o_col0 = o_col0;
  g.so = so;
  g.status = status;
  g.wait_ns = wait_limit_ns();
  g.kchunk = kchunk;
  g.kz = (K + kchunk - 1) / kchunk;
  g.zstride = zstride;
  const int sms = max_ctas > 0 ? max_ctas : num_sms_dev();
  if (M <= G_BM && g.kz == 1) {
    if (N <= 64 * sms) return launch_gemm<64>(st, a, b, g, sms);
    if (N <= 128 * sms) return launch_gemm<128>(st, a, b, g, sms);
  }
  return launch_gemm<256>(st, a, b, g, sms);
}

int chol_block_rows(int64_t n) {
  static const int forced = [] {
    const char *v = getenv("VMCK_CHOL_BLOCK");
    const int r = v ? atoi(v) : 0;
    return (r == 128 || r == 256 || r == 512 || r == 1024 || r == 2048 || r == 4096) ? r : 0;
  }();
  if (forced) return forced;
  // measured on GB300 (factor + refinement): n = 16,384: 18.5 / 18.2 / 19.7 ms
  // for 512 / 1024 / 2048 rows; 32,768: 86 / 68 / 71 ms; 65,536: 609 / 440 /
  // 385 / 412 ms (4096)
  return n >= 3 * CHOL_BIG_N / 2 ? 2048 : (n >= CHOL_BIG_N / 2 ? 1024 : CHOL_BLOCK);
}

int64_t chol_tc_workspace_bytes(int64_t n) {
  const int64_t nb = (n + LB - 1) / LB;
  int64_t b = 0;
  b += 4 * (int64_t)chol_block_rows(n) * n * 2;  // Ph hi / lo, two buffers (K = block rows)
  b += 2 * (int64_t)LB * n * 2;          // Bs hi / lo
  b += 2 * (int64_t)LB * LB * 2;         // Xs hi / lo
  b += 64;                               // scales
  b += nb * LB * LB * 4;                 // Yinv
  return b + 8 * 1024;                   // alignment
}

int chol_events_needed(int64_t n) {
  const int64_t blk = chol_block_rows(n);
  return (int)(3 * ((n + blk - 1) / blk) + 2 + 2 * ((n + LB - 1) / LB));
}

// Trailing-update CTAs of the side stream: every SM but a reserve that stays
// free for the chain's kernels: 48 below n = CHOL_BIG_N, 24 from there on
// (measured: the chain's share of the work shrinks with n; n = 65,536: 385 /
// 366 / 371 ms with 48 / 24 / 12), unless VMCK_CHOL_RESERVE (read once per
// process) sets it.
static int side_ctas(int sms, int64_t n) {
  static const int forced = [] {
    const char *v = getenv("VMCK_CHOL_RESERVE");
    return v ? std::max(0, atoi(v)) : -1;
  }();
  const int reserve = forced >= 0 ? forced : (n >= CHOL_BIG_N ? 24 : 48);
  return std::max(8, sms - reserve);
}

static char *align_up(char *p, size_t a) {
  return reinterpret_cast<char *>((reinterpret_cast<uintptr_t>(p) + a - 1) & ~uintptr_t(a - 1));
}

int chol_tc_factor(cudaStream_t st, float *A, int64_t n, void *ws, int32_t *status,
                   float **yinv_out, const CholStreams *ls) {
  if (n <= 0) return VMCK_OK;
  if (n >= (1ll << 30)) {
    set_last_error("chol_tc: n must be below 2^30");
    return VMCK_ERR_UNSUPPORTED;
  }
  const int64_t blk = chol_block_rows(n);
  char *p = align_up(static_cast<char *>(ws), 1024);
  __half *ph_hi[2], *ph_lo[2];
  for (int q = 0; q < 2; ++q) {
    ph_hi[q] = reinterpret_cast<__half *>(p);
    p = align_up(p + (size_t)blk * n * 2, 1024);
    ph_lo[q] = reinterpret_cast<__half *>(p);
    p = align_up(p + (size_t)blk * n * 2, 1024);
  }
  __half *bs_hi = reinterpret_cast<__half *>(p);
  p = align_up(p + (size_t)LB * n * 2, 1024);
  __half *bs_lo = reinterpret_cast<__half *>(p);
  p = align_up(p + (size_t)LB * n * 2, 1024);
  __half *xs_hi = reinterpret_cast<__half *>(p);
  p = align_up(p + (size_t)LB * LB * 2, 1024);
  __half *xs_lo = reinterpret_cast<__half *>(p);
  p = align_up(p + (size_t)LB * LB * 2, 1024);
  float *scales = reinterpret_cast<float *>(p);  // [0] A entries, [1] U entries, [2] X
  p = align_up(p + 64, 1024);
  float *yinv = reinterpret_cast<float *>(p);
  if (yinv_out) *yinv_out = yinv;

  const int nblocks = (int)((n + blk - 1) / blk);
  // look-ahead: the chain stream factors block row b and updates block row b + 1
  // (LA); the side stream updates rows b + 2 .. with block row b, first block row
  // b + 2 (event E[b]: LA(b + 1) waits for it), then the rest (event G[b]: block
  // row b + 2 reuses block row b's split-panel buffer).  F[b]: block row b's
  // panel is complete.
  const bool two = ls && ls->chain && ls->side && ls->n_events >= 3 * nblocks + 2;
  cudaStream_t chain = two ? ls->chain : st, side = two ? ls->side : st;
  cudaEvent_t *F = two ? ls->events : nullptr, *E = F ? F + nblocks : nullptr;
  cudaEvent_t *G = E ? E + nblocks : nullptr;
  // split block-row updates: PA[p] panel p's rows are written (chain), PB[p] the
  // update of the rows below panel p + 1 by panel p is done (chain2)
  const int npanels = (int)((n + LB - 1) / LB);
  const bool split = two && ls->chain2 && ls->n_events >= 3 * nblocks + 2 + 2 * npanels;
  cudaEvent_t *PA = split ? G + nblocks + 2 : nullptr, *PB = split ? PA + npanels : nullptr;
  int rc;
  if (two) {
    VMCK_CUDA(cudaEventRecord(ls->events[3 * nblocks], st));
    VMCK_CUDA(cudaStreamWaitEvent(chain, ls->events[3 * nblocks], 0));
    VMCK_CUDA(cudaStreamWaitEvent(side, ls->events[3 * nblocks], 0));
    if (split) VMCK_CUDA(cudaStreamWaitEvent(ls->chain2, ls->events[3 * nblocks], 0));
  }
  const int side_grid = two ? side_ctas(num_sms_dev(), n) : 0;
  // chain2's updates leave two of the SMs that the side stream does not use: a grid
  // over all of them keeps the next leaf waiting for its last wave (n = 16,384: factor
  // and two refinements 11.87 -> 11.30 ms; 11.75 with none left, 11.36 with four, 11.63
  // with sixteen; n = 24,000: 27.7 -> 26.35).  Before the first trailing update the
  // whole chip is the chain's, and a reserve there changes nothing.
  // From CHOL_BIG_N on, with 24 SMs reserved, 22 are too few for the updates once the side
  // stream is done: the whole grid (32,768 / 40,960 / 49,152: 54.5 / 95 / 150 ms; limited
  // 55.3 / 95 / 194).
  const int chain2_grid =
      n >= CHOL_BIG_N ? 0 : std::max(8, num_sms_dev() - side_grid - 2);
  VMCK_CUDA(cudaFuncSetAttribute(chol_leaf_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)CHOL_LEAF_SMEM));
  // the leaf writes X and Y on and above, or below, their diagonals
  VMCK_CUDA(cudaMemsetAsync(yinv, 0, (size_t)((n + LB - 1) / LB) * LB * LB * 4, chain));
  VMCK_CUDA(cudaMemsetAsync(xs_hi, 0, (size_t)LB * LB * 2, chain));
  VMCK_CUDA(cudaMemsetAsync(xs_lo, 0, (size_t)LB * LB * 2, chain));
  chol_bounds_kernel<<<1, 256, 0, chain>>>(A, n, scales, status);
  if ((rc = check_launch("chol_tc bounds"))) return rc;
  {
    const int rows = (int)std::min<int64_t>(LB, n);
    const int64_t cols = n - rows;
    if (cols > 0) {
      chol_split_rows_kernel<<<ceil_div(cols * LB, 256), 256, 0, chain>>>(
          A, n, 0, rows, rows, cols, LB, scales, bs_hi, bs_lo);
      if ((rc = check_launch("chol_tc split"))) return rc;
    }
  }
  for (int b = 0; b < nblocks; ++b) {
    const int64_t k0 = b * blk;
    const int64_t k1 = std::min<int64_t>(n, k0 + blk), w = k1 - k0;
    const int64_t k2 = std::min<int64_t>(n, k1 + blk), k3 = std::min<int64_t>(n, k2 + blk);
    __half *qh = ph_hi[two ? (b & 1) : 0], *ql = ph_lo[two ? (b & 1) : 0];
    // the block row's split panel: row (c - k0) holds U(k0 .. k1, c) (K = w)
    const SplitOperand ph{qh, ql, blk, w, n - k0};
    if (two && b >= 2)
      VMCK_CUDA(cudaStreamWaitEvent(chain, G[b - 2], 0));  // side is done with this buffer
    bool pb_pending = false;  // PB[pi - 1] recorded in this block row
    for (int64_t r0 = k0; r0 < k1; r0 += LB) {
      const int64_t r1 = std::min<int64_t>(k1, r0 + LB);
      const int mp = (int)(r1 - r0), pp = (int)((r0 - k0) / LB);
      const int pi = (int)(r0 / LB);
      {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(1);
        cfg.blockDim = dim3(LEAF_T);
        cfg.dynamicSmemBytes = CHOL_LEAF_SMEM;
        cfg.stream = chain;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        VMCK_CUDA(cudaLaunchKernelEx(&cfg, chol_leaf_kernel, A, n, r0, mp, xs_hi, xs_lo,
                                     scales + 2, yinv + (r0 / LB) * LB * LB, status));
        if ((rc = check_launch("chol_tc leaf"))) return rc;
      }
      if (r1 == n) break;
      const SplitOperand xop{xs_hi, xs_lo, LB, mp, mp};
      const SplitOperand bop{bs_hi, bs_lo, LB, mp, n - r1};
      // panel: U[r0:r1, r1:n] = X^T A[r0:r1, r1:n], split copy into Ph
      if ((rc = tc_gemm(chain, xop, 0, bop, 0, 0, mp, (int)(n - r1), mp, A + r0 + r1 * n, n,
                        1.0f, 0.0f, scales + 2, scales + 0, 0,
                        qh + (r1 - k0) * blk + pp * LB, ql + (r1 - k0) * blk + pp * LB, blk,
                        mp, 0, scales + 1,
                        status, 0)))
        return rc;
      if (r1 < k1) {
        // rest of the block row; rows [r1, r1 + next) feed the next panel (split)
        const int next = (int)std::min<int64_t>(LB, k1 - r1);
        const SplitOperand pk{qh, ql, blk, pp * LB + mp, n - k0};
        if (!split) {
          if ((rc = tc_gemm(chain, pk, (int)(r1 - k0), pk, (int)(r1 - k0), pp * LB,
                            (int)(k1 - r1), (int)(n - r1), mp, A + r1 + r1 * n, n, -1.0f, 1.0f,
                            scales + 1, scales + 1, 1, bs_hi, bs_lo, LB, next, next,
                            scales + 0, status, 0)))
            return rc;
        } else {
          // the next panel's rows on the chain (after the previous panel's update
          // of the same rows on chain2), the rows below them on chain2
          const int64_t r2 = r1 + next;
          if (r2 < k1) VMCK_CUDA(cudaEventRecord(PA[pi], chain));
          if (pb_pending) VMCK_CUDA(cudaStreamWaitEvent(chain, PB[pi - 1], 0));
          pb_pending = false;
          if ((rc = tc_gemm(chain, pk, (int)(r1 - k0), pk, (int)(r1 - k0), pp * LB, next,
                            (int)(n - r1), mp, A + r1 + r1 * n, n, -1.0f, 1.0f, scales + 1,
                            scales + 1, 1, bs_hi, bs_lo, LB, next, next, scales + 0, status, 0)))
            return rc;
          if (r2 < k1) {
            VMCK_CUDA(cudaStreamWaitEvent(ls->chain2, PA[pi], 0));
            if ((rc = tc_gemm(ls->chain2, pk, (int)(r2 - k0), pk, (int)(r2 - k0), pp * LB,
                              (int)(k1 - r2), (int)(n - r2), mp, A + r2 + r2 * n, n, -1.0f,
                              1.0f, scales + 1, scales + 1, 1, nullptr, nullptr, 0, 0, 0,
                              nullptr, status, b == 0 ? 0 : chain2_grid)))
              return rc;
            VMCK_CUDA(cudaEventRecord(PB[pi], ls->chain2));
            pb_pending = true;
          }
        }
      }
    }
    if (k1 == n) break;
    const int next = (int)std::min<int64_t>(LB, n - k1);
    if (!two) {
      // trailing matrix by the whole block row; rows [k1, k1 + next) feed the
      // next block row's first panel (split)
      if ((rc = tc_gemm(st, ph, (int)w, ph, (int)w, 0, (int)(n - k1), (int)(n - k1), (int)w,
                        A + k1 + k1 * n, n, -1.0f, 1.0f, scales + 1, scales + 1, 1, bs_hi, bs_lo,
                        LB, next, next, scales + 0, status, 0)))
        return rc;
      continue;
    }
    VMCK_CUDA(cudaEventRecord(F[b], chain));
    // LA(b): block row b + 1 by this block row, once the side stream has applied
    // the previous block row to it
    if (b >= 1) VMCK_CUDA(cudaStreamWaitEvent(chain, E[b - 1], 0));
    if ((rc = tc_gemm(chain, ph, (int)w, ph, (int)w, 0, (int)(k2 - k1), (int)(n - k1), (int)w,
                      A + k1 + k1 * n, n, -1.0f, 1.0f, scales + 1, scales + 1, 1, bs_hi, bs_lo,
                      LB, next, next, scales + 0, status, 0)))
      return rc;
    // side: block row b + 2, then the rest
    VMCK_CUDA(cudaStreamWaitEvent(side, F[b], 0));
    if (k2 < n) {
      const int off2 = (int)(k2 - k0);
      if ((rc = tc_gemm(side, ph, off2, ph, off2, 0, (int)(k3 - k2), (int)(n - k2), (int)w,
                        A + k2 + k2 * n, n, -1.0f, 1.0f, scales + 1, scales + 1, 1, nullptr,
                        nullptr, 0, 0, 0, nullptr, status, side_grid)))
        return rc;
    }
    VMCK_CUDA(cudaEventRecord(E[b], side));
    if (k3 < n) {
      const int off3 = (int)(k3 - k0);
      if ((rc = tc_gemm(side, ph, off3, ph, off3, 0, (int)(n - k3), (int)(n - k3), (int)w,
                        A + k3 + k3 * n, n, -1.0f, 1.0f, scales + 1, scales + 1, 1, nullptr,
                        nullptr, 0, 0, 0, nullptr, status, side_grid)))
        return rc;
    }
    VMCK_CUDA(cudaEventRecord(G[b], side));
  }
  if (two) {
    VMCK_CUDA(cudaEventRecord(ls->events[3 * nblocks], chain));
    VMCK_CUDA(cudaStreamWaitEvent(st, ls->events[3 * nblocks], 0));
    VMCK_CUDA(cudaEventRecord(ls->events[3 * nblocks + 1], side));
    VMCK_CUDA(cudaStreamWaitEvent(st, ls->events[3 * nblocks + 1], 0));
    if (split) {  // (already ordered through the chain; kept explicit)
      VMCK_CUDA(cudaEventRecord(ls->events[3 * nblocks], ls->chain2));
      VMCK_CUDA(cudaStreamWaitEvent(st, ls->events[3 * nblocks], 0));
    }
  }
  return VMCK_OK;
}

}  // namespace vmck
