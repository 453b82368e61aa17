// FP32 local energies for one- and two-site terms (eloc_f32.cu).
#pragma once

#include "common.cuh"

namespace vmck {

// Whether the kernel takes this problem (op null: Ising).
bool eloc_f32_takes(int N, int M, int64_t n, const vmck_local_op *op);
int eloc_f32_ising(cudaStream_t st, const float *params, int N, int M, const int8_t *x, int64_t n,
                   const int32_t *edges, int n_edges, double h, double J, double *eloc);
int eloc_f32_local(cudaStream_t st, const float *params, int N, int M, const int8_t *x, int64_t n,
                   const vmck_local_op &op, double *eloc);

}  // namespace vmck
