// Kernel-matrix build in 64 x 64 tiles (declarations; implementation in km_build_small.cu).
#pragma once

#include "km_build_params.cuh"

namespace km {

// True when a 64 x 64 kernel exists for the inner step and the tile counts are in its range.
bool small_supported(const BuildParams& p);

// True when the kernel stages an operand 16 bytes at a time (along the points or along k).
bool small_wide_loads(const float* base, long long s_t, long long s_k, long long s_l, int K, int L);

// `tma`: both operands satisfy tma_supported() and the inner step is a square or a product.
int launch_build_small(const BuildParams& p, bool tma, cudaStream_t stream);

// Reads back and clears the kernel's wait-ran-out flag; the device must already be synchronised.
// 0 / 1, or -1 on error.
int small_take_wait_flag();

}  // namespace km
