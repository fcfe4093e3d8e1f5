// The streaming kernel's body on matrices of too few rows to be a stream for it: the reduction
// axis sliced over a thread-block cluster (gemv_mma_stream_sliced_kernel, dq_gemv_mma_stream.cuh).
//
// The streaming kernel gives a warp whole rows, so it needs eight row tiles per SM and warp to fill
// the machine; below that the tiled kernel slices the reduction axis over the eight warps of ONE
// CTA (8, 4 or 2 ways, even slices), which leaves a down-projection such as 5120 x 17408 with 160
// CTAs of eight warps on 148 SMs -- a third of the warps the streaming kernel keeps resident, and the
// decode needs them.  Here the slices are CTAs of a cluster: a group of eight row tiles x up to
// eight slices of whole blocks in any proportion, two CTAs per SM, every CTA staging only its own
// part of the activation; the slices' sums meet in the cluster's first CTA through distributed
// shared memory in slice order.
#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>

#include "dq_gemv.cuh"
#include "dq_gemv_mma_stream.cuh"

namespace dq {
namespace {

// Clusters of `slices` CTAs with `smem` bytes each that the device holds at once, per kernel build.
template <typename Kernel>
int active_clusters(int tag, Kernel kernel, int slices, size_t smem) {
  static std::mutex mu;
  static std::map<std::tuple<int, int, size_t>, int> cache;
  const auto key = std::make_tuple(tag, slices, smem);
  {
    std::lock_guard<std::mutex> lock(mu);
    const auto it = cache.find(key);
    if (it != cache.end()) return it->second;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(1, static_cast<unsigned>(slices));
  cfg.blockDim = dim3(stream::kThreads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = static_cast<unsigned>(slices);
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (allow_shared(kernel, smem) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    n = 0;
  }
  std::lock_guard<std::mutex> lock(mu);
  cache[key] = n;
  return n;
}

template <int BITS>
int32_t launch_sliced(const GemvArgs& a, const DeviceInfo& dev, cudaStream_t stream_h, bool* taken) {
  using C = stream::Cfg<BITS>;
  const int steps = a.words_per_row / (4 * BITS);
  if (reinterpret_cast<uintptr_t>(a.packed) % 16 != 0 || (static_cast<int64_t>(a.words_per_row) * 4) % 16 != 0) return DQ_OK;
  if (a.group_values != 128 || steps % C::P != 0 || a.num_groups != steps || a.in_features != steps * 128) return DQ_OK;
  const auto align = static_cast<uintptr_t>(C::META_BYTES);
  if (reinterpret_cast<uintptr_t>(a.scales) % align != 0 || reinterpret_cast<uintptr_t>(a.offsets) % align != 0 ||
      (static_cast<int64_t>(a.num_groups) * 2) % C::META_BYTES != 0) {
    return DQ_OK;
  }
  if ((reinterpret_cast<uintptr_t>(a.x) & 15) != 0) return DQ_OK;  // a slice of x starts on a step: stays 16-byte aligned
  const bool plan16 = BITS == 8;  // the fp16-operand plan (see launch_stream, dq_gemv_mma.cu)
  const int aregs = plan16 ? 16 : (BITS == 8 ? 32 : 16);
  const int nblocks = steps / C::P;
  const int tiles = static_cast<int>(ceil_div(a.rows, 16));
  const int row_groups = static_cast<int>(ceil_div(tiles, stream::kWarps));
  stream::Params p = {};
  p.steps = steps;
  p.tiles = tiles;
  p.magic = (plan16 || a.x_dtype != DQ_BF16) ? 0x64006400u : 0x43004300u;
  auto smem_for = [&](int slices) {
    const int slice_steps = static_cast<int>(ceil_div(nblocks, slices)) * C::P;
    const size_t stride = static_cast<size_t>(slice_steps) * aregs + 4;
    const size_t need = C::RING_BYTES + (static_cast<size_t>(a.m) * stride + aregs) * 16 + static_cast<size_t>(slice_steps) * 8 * 4 * 2;
    // At least 80 KB: two CTAs per SM, not three.  With one activation row three would fit, and the
    // CTAs of a cluster are then placed so unevenly over the SMs that the launch is slower and its
    // time erratic in the slice count (measured at 2 / 3 / 4 / 8 bits, one row: 5120 x 17408 17 / 24 /
    // 23 / 31 us with three per SM, 14 / 20 / 17 / 21 with two; 3584 x 18944 17 / 23 / 22 / 30 against
    // 13 / 18 / 15 / 18; one per SM is level with two except on 10240 x 5120, 23 against 13 at 8 bits).
    return std::max(need, static_cast<size_t>(tuning_int("DQ_B200_SLICED_MIN_SMEM_KB", 80)) << 10);
  };
  auto run = [&](auto kernel, int tag) -> int32_t {
    // The largest slice count (two blocks a slice at least) whose clusters are all resident at once,
    // then the smallest with the same longest slice.
    const int forced = tuning_int("DQ_B200_STREAM_SLICES", 0);
    int slices = 0;
    const int max_slices = std::min(8, nblocks / 2);
    if (forced > 1) {
      slices = std::min(forced, std::max(1, nblocks));
      if (slices < 2 || active_clusters(tag, kernel, slices, smem_for(slices)) < 1) return DQ_OK;
    } else {
      for (int s = max_slices; s >= 2 && slices == 0; --s) {
        const size_t smem = smem_for(s);
        if (smem <= static_cast<size_t>(dev.max_smem_optin) && active_clusters(tag, kernel, s, smem) >= row_groups) slices = s;
      }
      if (slices == 0) return DQ_OK;
      while (slices > 2 && ceil_div(nblocks, slices - 1) == ceil_div(nblocks, slices)) --slices;
    }
    const size_t smem = smem_for(slices);
    if (smem > static_cast<size_t>(dev.max_smem_optin)) return DQ_OK;
    DQ_CUDA(allow_shared(kernel, smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(row_groups), static_cast<unsigned>(slices));
    cfg.blockDim = dim3(stream::kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream_h;
    cudaLaunchAttribute attr[3];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = static_cast<unsigned>(slices);
    attr[0].val.clusterDim.z = 1;
    unsigned count = weights_leave_first(&attr[1], dev, stream_h, &a, 1) ? 2 : 1;
    if (pdl_enabled_for_rows()) {
      attr[count].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[count++].val.programmaticStreamSerializationAllowed = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = count;
    DQ_CUDA(cudaLaunchKernelEx(&cfg, kernel, a, p));
    DQ_CHECK_LAUNCH("gemv");
    note_kernel("gemv_mma_stream_sliced_kernel");
    *taken = true;
    return DQ_OK;
  };
  const bool xbf = a.x_dtype == DQ_BF16, mbf = a.meta_dtype == DQ_BF16;
  const int tag = BITS * 4 + (xbf ? 2 : 0) + (mbf ? 1 : 0);
  constexpr bool P16 = BITS == 8;
  if (xbf && mbf) return run(stream::gemv_mma_stream_sliced_kernel<BITS, true, true, P16>, tag);
  if (xbf) return run(stream::gemv_mma_stream_sliced_kernel<BITS, true, false, P16>, tag);
  if (mbf) return run(stream::gemv_mma_stream_sliced_kernel<BITS, false, true, P16>, tag);
  return run(stream::gemv_mma_stream_sliced_kernel<BITS, false, false, P16>, tag);
}

}  // namespace

// One matrix, one to eight activation rows.  *taken stays false (nothing launched) when the matrix
// or the activation does not qualify or no slice count fits the device in one wave.
int32_t launch_gemv_stream_sliced(const GemvArgs& a, int bits, cudaStream_t stream_h, bool* taken) {
  *taken = false;
  const DeviceInfo* dev = device_info();
  if (dev == nullptr) return DQ_ERR_CUDA;
  if (a.m < 1 || a.m > 8) return DQ_OK;
  if (a.x_dtype != DQ_BF16 && a.x_dtype != DQ_F16) return DQ_OK;
  if (a.meta_dtype != DQ_BF16 && a.meta_dtype != DQ_F16) return DQ_OK;
  if ((a.in_features & 7) != 0) return DQ_OK;
  switch (bits) {
    case 2:
      return launch_sliced<2>(a, *dev, stream_h, taken);
    case 3:
      return launch_sliced<3>(a, *dev, stream_h, taken);
    case 4:
      return launch_sliced<4>(a, *dev, stream_h, taken);
    default:
      return launch_sliced<8>(a, *dev, stream_h, taken);
  }
}

namespace {

constexpr int kMaxJobs = 4;

struct SlicedJob {
  GemvArgs a;
  stream::Params p;
  int bits, group_begin, groups;  // row groups [group_begin, group_begin + groups) of the grid's x axis
};
struct SlicedLaunch {
  SlicedJob job[kMaxJobs];
  int njobs;
};

// Several matrices that share an activation: a range of row groups each, the same number of slices.
template <bool XBF16, bool MBF16>
__global__ void __launch_bounds__(stream::kThreads, 2) gemv_mma_stream_sliced_multi_kernel(const __grid_constant__ SlicedLaunch L) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int j = 0;
#pragma unroll
  for (int i = 1; i < kMaxJobs; ++i) {
    if (i < L.njobs && static_cast<int>(blockIdx.x) >= L.job[i].group_begin) j = i;
  }
  const SlicedJob& J = L.job[j];
  const unsigned int group = blockIdx.x - J.group_begin;
  switch (J.bits) {
    case 2: stream::sliced_body<2, XBF16, MBF16, false>(J.a, J.p, group, J.groups, smem_raw); break;
    case 3: stream::sliced_body<3, XBF16, MBF16, false>(J.a, J.p, group, J.groups, smem_raw); break;
    case 4: stream::sliced_body<4, XBF16, MBF16, false>(J.a, J.p, group, J.groups, smem_raw); break;
    default: stream::sliced_body<8, XBF16, MBF16, true>(J.a, J.p, group, J.groups, smem_raw); break;
  }
}

template <int BITS>
bool job_ok(const GemvArgs& a) {
  using C = stream::Cfg<BITS>;
  const int steps = a.words_per_row / (4 * BITS);
  const auto align = static_cast<uintptr_t>(C::META_BYTES);
  return reinterpret_cast<uintptr_t>(a.packed) % 16 == 0 && (static_cast<int64_t>(a.words_per_row) * 4) % 16 == 0 && a.group_values == 128 &&
         steps % C::P == 0 && a.num_groups == steps && a.in_features == steps * 128 && reinterpret_cast<uintptr_t>(a.scales) % align == 0 &&
         reinterpret_cast<uintptr_t>(a.offsets) % align == 0 && (static_cast<int64_t>(a.num_groups) * 2) % C::META_BYTES == 0;
}

template <int BITS>
size_t job_smem(const GemvArgs& a, int slices) {
  using C = stream::Cfg<BITS>;
  const int aregs = 16;  // (8 bits: the fp16-operand plan)
  const int slice_steps = static_cast<int>(ceil_div(a.in_features / 128 / C::P, slices)) * C::P;
  return C::RING_BYTES + (static_cast<size_t>(a.m) * (static_cast<size_t>(slice_steps) * aregs + 4) + aregs) * 16 +
         static_cast<size_t>(slice_steps) * 8 * 4 * 2;
}

}  // namespace

int32_t launch_gemv_stream_sliced_fused(const GemvArgs* jobs, const int* bits, int n, int least_ctas, cudaStream_t stream_h, bool* taken) {
  *taken = false;
  const DeviceInfo* dev = device_info();
  if (dev == nullptr) return DQ_ERR_CUDA;
  const GemvArgs& a0 = jobs[0];
  if (n < 1 || n > kMaxJobs || a0.m < 1 || a0.m > 8 || (a0.x_dtype != DQ_BF16 && a0.x_dtype != DQ_F16) ||
      (a0.meta_dtype != DQ_BF16 && a0.meta_dtype != DQ_F16) || (reinterpret_cast<uintptr_t>(a0.x) & 15) != 0) {
    return DQ_OK;
  }
  SlicedLaunch L = {};
  L.njobs = n;
  int groups = 0, nblocks = 1 << 30;
  for (int i = 0; i < n; ++i) {
    const GemvArgs& a = jobs[i];
    if (a.x != a0.x || a.m != a0.m || a.x_dtype != a0.x_dtype || a.meta_dtype != a0.meta_dtype || a.in_features != a0.in_features ||
        a.out_dtype != a0.out_dtype || a.rows < 1) {
      return DQ_OK;
    }
    if (!(bits[i] == 2 ? job_ok<2>(a) : bits[i] == 3 ? job_ok<3>(a) : bits[i] == 4 ? job_ok<4>(a) : job_ok<8>(a))) return DQ_OK;
    SlicedJob& J = L.job[i];
    J.a = a;
    J.bits = bits[i];
    J.p.steps = a.in_features / 128;
    J.p.tiles = static_cast<int>(ceil_div(a.rows, 16));
    J.p.magic = (bits[i] == 8 || a.x_dtype != DQ_BF16) ? 0x64006400u : 0x43004300u;
    J.group_begin = groups;
    J.groups = static_cast<int>(ceil_div(J.p.tiles, stream::kWarps));
    groups += J.groups;
    nblocks = std::min(nblocks, J.p.steps / (bits[i] == 2 ? stream::Cfg<2>::P : bits[i] == 3 ? stream::Cfg<3>::P : bits[i] == 4 ? stream::Cfg<4>::P : stream::Cfg<8>::P));
  }
  auto smem_for = [&](int slices) {
    size_t need = 80 << 10;  // two CTAs per SM, not three (see launch_sliced)
    for (int i = 0; i < n; ++i) {
      need = std::max(need, bits[i] == 2 ? job_smem<2>(jobs[i], slices) : bits[i] == 3 ? job_smem<3>(jobs[i], slices)
                                                                    : bits[i] == 4 ? job_smem<4>(jobs[i], slices) : job_smem<8>(jobs[i], slices));
    }
    return need;
  };
  auto run = [&](auto kernel, int tag) -> int32_t {
    // as launch_sliced: the most slices whose clusters are all resident, then the fewest with the same longest slice
    int slices = 0;
    for (int s = std::min(8, nblocks / 2); s >= 2 && slices == 0; --s) {
      const size_t smem = smem_for(s);
      if (smem <= static_cast<size_t>(dev->max_smem_optin) && active_clusters(tag, kernel, s, smem) >= groups) slices = s;
    }
    while (slices > 2 && ceil_div(nblocks, slices - 1) == ceil_div(nblocks, slices)) --slices;
    if (slices == 0) {  // whole rows per warp, if every CTA is resident
      const size_t smem = smem_for(1);
      int per_sm = 0;
      if (smem > static_cast<size_t>(dev->max_smem_optin)) return DQ_OK;
      DQ_CUDA(allow_shared(kernel, smem));
      DQ_CUDA(resident_ctas(&per_sm, kernel, stream::kThreads, smem));
      if (static_cast<int64_t>(per_sm) * dev->sm_count < groups) return DQ_OK;
      slices = 1;
    }
    if (groups * slices < least_ctas) return DQ_OK;
    const size_t smem = smem_for(slices);
    DQ_CUDA(allow_shared(kernel, smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(groups), static_cast<unsigned>(slices));
    cfg.blockDim = dim3(stream::kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream_h;
    cudaLaunchAttribute attr[3];
    int na = 0;
    if (weights_leave_first(&attr[na], *dev, stream_h, jobs, n)) ++na;
    if (slices > 1) {
      attr[na].id = cudaLaunchAttributeClusterDimension;
      attr[na].val.clusterDim.x = 1;
      attr[na].val.clusterDim.y = static_cast<unsigned>(slices);
      attr[na].val.clusterDim.z = 1;
      ++na;
    }
    if (pdl_enabled_for_rows()) {
      attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[na].val.programmaticStreamSerializationAllowed = 1;
      ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    DQ_CUDA(cudaLaunchKernelEx(&cfg, kernel, L));
    DQ_CHECK_LAUNCH("gemv");
    note_kernel("gemv_mma_stream_sliced_multi_kernel");
    *taken = true;
    return DQ_OK;
  };
  const bool xbf = a0.x_dtype == DQ_BF16, mbf = a0.meta_dtype == DQ_BF16;
  if (xbf && mbf) return run(gemv_mma_stream_sliced_multi_kernel<true, true>, 103);
  if (xbf) return run(gemv_mma_stream_sliced_multi_kernel<true, false>, 102);
  if (mbf) return run(gemv_mma_stream_sliced_multi_kernel<false, true>, 101);
  return run(gemv_mma_stream_sliced_multi_kernel<false, false>, 100);
}

}  // namespace dq
