// Argument block and output store shared by the GEMV kernels.
#pragma once

#include "dq_common.cuh"

namespace dq {

struct GemvArgs {
  const void* x;
  const uint32_t* packed;
  const void* scales;
  const void* offsets;  // may be null
  const void* bias;     // may be null; [rows] in out_dtype, indexed from out_col0
  void* out;
  int64_t out_stride;  // elements between consecutive activation rows of out
  int64_t out_col0;    // first output column this weight writes
  int x_dtype, meta_dtype, out_dtype;
  int m;     // real activation rows
  int rows;  // output features of this weight
  int words_per_row, num_groups, words_per_group, group_values, in_features;
  int chunks_per_row, chunks_per_group;  // fast path only
  int read_again;  // 1: another launch of this call reads the same weights (row chunks, passes over half the rows)
};

// A launch attribute that lets the packed words of `jobs` leave L2 before anything else: an access policy window
// over all of them where they lie close together (a layer loaded in one go; up to a third of the window may be what lies
// between them, but nothing that this launch reads or writes besides weights), else over the largest, or over the first
// part of it if it is longer than a window can be (128 MB here, as against an lm_head of 500).  False: the launch goes
// without, because its weights are read again in this call, or because the stream has a window of its own, which a launch's would replace.
//
// Weights are read once per launch and are nine tenths of all traffic.  What they push out otherwise are the
// activations and above all the INSTRUCTIONS of the kernels that take turns in a decode step, whose first fetches
// then come from memory, launch after launch: the captured step of a 14B model's layers (15 layers, four rows) 1144 ->
// 1050 us, of a 2B model with its head (one row, launches of 2 to 11 MB) 465 -> 461, without it 381 -> 357; a launch whose
// kernel ran just before takes the same time as without (2 x 17408 x 5120, 4-bit, four rows 25.7 -> 25.2 us, 5120 x 5120, 3-bit,
// one row 8.3), and so does a step whose weights all stay in L2 (two layers of the 2B model, 38 MB: 50.1 -> 49.9).
// (The same by cp.async with an L2 cache hint costs registers and up to 3 % at 2 bits.  The many-rows kernel, the
// streaming launch of several matrices and the expert layers have not been measured with a window and go without.)
inline bool weights_leave_first(cudaLaunchAttribute* attr, const DeviceInfo& dev, cudaStream_t stream, const GemvArgs* jobs, int n) {
  const auto bytes = [](const GemvArgs& a) { return static_cast<int64_t>(a.rows) * a.words_per_row * 4; };
  uintptr_t low = ~uintptr_t{0}, high = 0;
  int64_t sum = 0;
  int most = 0;
  for (int i = 0; i < n; ++i) {
    if (jobs[i].read_again != 0) return false;
    for (int j = 0; j < i; ++j) {
      if (jobs[j].packed == jobs[i].packed) return false;
    }
    const auto at = reinterpret_cast<uintptr_t>(jobs[i].packed);
    low = at < low ? at : low, high = at + bytes(jobs[i]) > high ? at + bytes(jobs[i]) : high;
    sum += bytes(jobs[i]);
    if (bytes(jobs[i]) > bytes(jobs[most])) most = i;
  }
  cudaLaunchAttributeValue own = {};
  if (cudaStreamGetAttribute(stream, cudaLaunchAttributeAccessPolicyWindow, &own) != cudaSuccess) {
    cudaGetLastError();
  } else if (own.accessPolicyWindow.num_bytes != 0) {
    return false;
  }
  const int64_t span = static_cast<int64_t>(high - low);
  bool together = span <= dev.max_window && span <= sum + sum / 2;
  for (int i = 0; i < n && together; ++i) {
    const GemvArgs& a = jobs[i];
    const auto apart = [&](const void* p, int64_t elems, int dtype) {
      const auto at = reinterpret_cast<uintptr_t>(p);
      return at >= high || at + static_cast<uintptr_t>(elems) * dtype_size(dtype) <= low;
    };
    together = apart(a.x, static_cast<int64_t>(a.m) * a.in_features, a.x_dtype) && apart(a.out, a.m * a.out_stride, a.out_dtype) &&
               (a.bias == nullptr || apart(a.bias, a.out_col0 + a.rows, a.out_dtype));
  }
  attr->id = cudaLaunchAttributeAccessPolicyWindow;
  cudaAccessPolicyWindow& w = attr->val.accessPolicyWindow;
  w.base_ptr = together ? reinterpret_cast<void*>(low) : const_cast<uint32_t*>(jobs[most].packed);
  w.num_bytes = static_cast<size_t>(together ? span : bytes(jobs[most]) < dev.max_window ? bytes(jobs[most]) : dev.max_window);
  w.hitRatio = 1.0f;
  w.hitProp = cudaAccessPropertyStreaming;
  w.missProp = cudaAccessPropertyStreaming;
  return true;
}

namespace peerpush {
struct Push;  // dq_peer_push.cuh
}

// Tensor-core path (dq_gemv_mma.cu).  Returns DQ_ERR_UNSUPPORTED without touching
// the error buffer when the geometry or dtype is not one it handles, so the
// caller can fall through to the SIMT kernels.
bool mma_path_supports(const GemvArgs& a, int bits);
// `push` (optional): the launch also replicates its output rows into every rank's window and
// ends with the bounded wait for the other ranks' rows; only the streaming and the tiled kernel
// do that, so with `push` every other geometry returns DQ_ERR_UNSUPPORTED, nothing launched.
int32_t launch_gemv_mma(const GemvArgs& a, int bits, cudaStream_t stream, const peerpush::Push* push = nullptr);
// Up to four matrices that share one activation, in ONE launch.  *taken is false (and nothing
// was launched) when the jobs do not qualify; the caller then launches them one by one.
int32_t launch_gemv_mma_fused(const GemvArgs* jobs, const int* bits, int n, cudaStream_t stream, bool* taken,
                              const peerpush::Push* push = nullptr);

// Two to four long matrices that share an activation in one launch of the streaming kernel's body
// (dq_gemv_stream_multi.cu).  *taken stays false, nothing launched, when they do not qualify.
int32_t launch_gemv_stream_fused(const GemvArgs* jobs, const int* bits, int n, cudaStream_t stream, bool* taken);
// One to eight activation rows against one matrix of too few rows for the streaming kernel: its
// body with the reduction axis sliced over a thread-block cluster (dq_gemv_stream_sliced.cu).
int32_t launch_gemv_stream_sliced(const GemvArgs& a, int bits, cudaStream_t stream, bool* taken);
// The same for one to four matrices that share an activation, in one launch.
int32_t launch_gemv_stream_sliced_fused(const GemvArgs* jobs, const int* bits, int n, int least_ctas, cudaStream_t stream, bool* taken);
// min_rows..64 activation rows against one matrix in one pass over the weights (dq_gemv_rows.cu).
// *taken stays false, nothing launched, when the matrix or the activation does not qualify.
int32_t launch_gemv_rows(const GemvArgs& a, int bits, cudaStream_t stream, bool* taken, int min_rows = 9);
// False when DQ_B200_GEMV_PATH=simt forces the SIMT kernels.
bool mma_enabled_for_rows();
// False when DQ_B200_NO_PDL drops the programmatic-dependent-launch attribute.
bool pdl_enabled_for_rows();

#ifdef __CUDACC__
__device__ __forceinline__ void store_out(const GemvArgs& a, int m, int row, float v) {
  const int64_t col = a.out_col0 + row;
  if (a.bias != nullptr) {
    v += load_f32(a.bias, col, a.out_dtype);
  }
  store_f32(a.out, static_cast<int64_t>(m) * a.out_stride + col, a.out_dtype, v);
}

#endif

}  // namespace dq
