// Metropolis sweeps whose decisions are filtered (sampler_filter.cu): entry
// points for vmck_metropolis_sample.
#pragma once

#include "common.cuh"

namespace vmck {

struct SweepArgs {
  const void *params;
  int N, M;
  int8_t *sigma;
  double *log_prob;
  int64_t *n_accepted;
  int B, sweep, n_discard, L;
  int8_t *samples;
  uint32_t k0, k1;
  uint64_t counter;
  const int32_t *clusters;  // Exchange rule only
  int C;
};

// Whether the weights-in-shared-memory kernel takes this problem.
bool filtered_fits(int rule, int N, int M, int C);
int launch_filtered(cudaStream_t st, int dtype, int rule, const SweepArgs &a);
// The same with the weights read through L2.
bool filtered_l2_fits(int dtype, int rule, int N, int M, int C);
int launch_filtered_l2(cudaStream_t st, int dtype, int rule, const SweepArgs &a);

}  // namespace vmck
