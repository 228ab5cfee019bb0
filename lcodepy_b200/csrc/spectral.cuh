// Field solver by fast transforms, for grids whose number of intervals N - 1
// factors into small primes, as the configuration's do, up to 3125 nodes a side
// (two buffers of a line in a block's shared memory).
#pragma once

#include "common.cuh"

namespace lcb {

// Whether the fast transforms take a grid of N nodes a side.
bool spectral_grid(int N);
// Constant tables (twiddle factors, spectral factors), FP64 in both
// precisions, and the scratch of one solve.
size_t spectral_ops_bytes(int N);
int spectral_ops_build(int N, double h, double c, void *ops, cudaStream_t st);
size_t spectral_work_bytes(int N);
int spectral_solve(const lcb_compute_fields_args *a, const void *ops, cudaStream_t st);

}  // namespace lcb
