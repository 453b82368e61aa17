// Tensor-core (tcgen05) forms of the structured Gram contraction; implemented in
// gram_tc.cu (FP32 tanh(theta)) and gram64_tc.cu (FP64).
#pragma once

#include "common.cuh"

namespace vmck {

int64_t gram_tc_workspace_doubles(int M, int64_t n);

// c: shifted, rounded tanh(theta); h, w, s0sq: double-float epilogue terms
// (see gram.cu); T64 nullable.
int gram_tc_launch(vmck_ctx *ctx, cudaStream_t st, const float *c, const uint32_t *bits,
                   int words, int N, int M, int64_t n, const float2 *h, const float2 *w,
                   const float2 *s0sq, double inv_n, double diag_shift, double *T64, float *T32,
                   double *ws, int split, int32_t *status);

// FP64 tanh(theta) (gram64_tc.cu): T64 and / or T32 from exact integer products of
// base-128 digits.  *flag_out is a device word that is nonzero after the launch where
// |t| > 1 or NaN; nothing is written then.
int64_t gram64_tc_workspace_doubles(int M, int64_t n);
bool gram64_tc_takes(int M, int64_t n);
int gram64_tc_launch(cudaStream_t st, const double *t, const uint32_t *bits, int words, int N,
                     int M, int64_t n, const double *g, const double *c, double inv_n,
                     double shift, double *T64, float *T32, double *ws, int32_t *status,
                     const int **flag_out);

}  // namespace vmck
