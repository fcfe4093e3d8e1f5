// Host interface of the tcgen05 kernels for many activation rows (dq_gemm_umma.cu).
#pragma once

#include "dq_gemv.cuh"

namespace dq {

// x [m, K] against up to four packed matrices that share it, in one launch.  *taken stays false
// (nothing launched) when the kernel does not take a geometry: fp32 activations or metadata, groups
// that are not 64 * 2^n values, rows or pointers that TMA cannot address (16-byte multiples).
int32_t launch_gemm_umma(const GemvArgs* args, const int* bits, int count, cudaStream_t stream, bool* taken);

// 1 if this call is one of those that dq_gemm_fail_next lets fail, else 0.
int take_fail_next();

}  // namespace dq
