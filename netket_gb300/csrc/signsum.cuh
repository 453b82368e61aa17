// FP64 products with the spin matrix by tables of signed sums (signsum_f64.cu).
#pragma once

#include "units_f64.cuh"

namespace vmck {

// logpsi (and theta, tanh theta where not null) of n samples; false when N is too
// large for the tables (the caller's general kernel takes it).
bool signed_rows_fit(int N);
int logpsi_f64(cudaStream_t st, const double *params, int N, int M, const int8_t *x, int64_t n,
               double *logpsi, double *theta, double *tanh_out);
// theta and q_units(theta) of n samples
int theta_q_f64(cudaStream_t st, const double *params, int N, int M, const int8_t *x, int64_t n,
                double *theta, u64 *q);
// out_s = t_s . (v_bias + x_s V) + x_s . v_visible
int o_v_f64(cudaStream_t st, const double *t, const int8_t *x, int N, int M, int64_t n,
            const double *v, double *out);
// O^T v: partial sums over ot_v_f64_chunks(N, M, n) chunks of samples in ws
int ot_v_f64_chunks(int N, int M, int64_t n);
int ot_v_f64(cudaStream_t st, const double *t, const int8_t *x, int N, int M, int64_t n,
             const double *v, double *ws);

}  // namespace vmck
