// Metadata entry points, error plumbing and the host-side geometry check that
// every operator runs first.
//
// dq_resolve_geometry keeps the rules and the wording of the reference's
// resolve_geometry (packages/dynquant-kernels/csrc/include/dynquant/geometry.h:63-132):
// nothing is derived by guesswork, everything is either passed in or implied
// by a shape, and every implication is checked.
#include <algorithm>
#include <atomic>
#include <mutex>

#include "dq_common.cuh"

namespace dq {

char* error_buffer() {
  static thread_local char buffer[kErrorBufferSize] = {0};
  return buffer;
}

namespace {
std::atomic<int64_t> g_launches{0};
}
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
namespace {
thread_local const char* t_last_kernel = "";
}
void note_kernel(const char* name) { t_last_kernel = name; }
const char* last_kernel() { return t_last_kernel; }
int64_t launches_so_far() { return g_launches.load(std::memory_order_relaxed); }

namespace {
constexpr int kMaxDevices = 64;
DeviceInfo cache[kMaxDevices];
std::atomic<bool> ready[kMaxDevices];
std::mutex mu;
}  // namespace

const DeviceInfo* device_info() {
  int device = 0;
  cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess || device < 0 || device >= kMaxDevices) {
    fail(DQ_ERR_CUDA, "cudaGetDevice failed: %s", cudaGetErrorString(err));
    return nullptr;
  }
  if (ready[device].load(std::memory_order_acquire)) return &cache[device];
  std::lock_guard<std::mutex> lock(mu);
  if (!ready[device].load(std::memory_order_relaxed)) {
    DeviceInfo info = {};
    info.device = device;
    err = cudaDeviceGetAttribute(&info.sm_count, cudaDevAttrMultiProcessorCount, device);
    if (err == cudaSuccess) {
      err = cudaDeviceGetAttribute(&info.max_smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin,
                                   device);
    }
    int window = 0;
    if (err == cudaSuccess) err = cudaDeviceGetAttribute(&window, cudaDevAttrMaxAccessPolicyWindowSize, device);
    info.max_window = window;
    if (err != cudaSuccess) {
      fail(DQ_ERR_CUDA, "cudaDeviceGetAttribute failed: %s", cudaGetErrorString(err));
      return nullptr;
    }
    // Once per device and process; a call that is the first one inside a stream capture may do this too.
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    void *host = nullptr, *mapped = nullptr;
    err = cudaThreadExchangeStreamCaptureMode(&mode);
    if (err == cudaSuccess) {
      err = cudaHostAlloc(&host, kReportWords * sizeof(unsigned int), cudaHostAllocPortable | cudaHostAllocMapped);
      if (err == cudaSuccess) err = cudaHostGetDevicePointer(&mapped, host, 0);
      cudaThreadExchangeStreamCaptureMode(&mode);
    }
    if (err != cudaSuccess || mapped != host) {  // (one address space: the kernels' address is the host's)
      fail(DQ_ERR_CUDA, "no host memory for the kernels' reports: %s", cudaGetErrorString(err));
      return nullptr;
    }
    info.report = static_cast<unsigned int*>(host);
    for (int i = 0; i < kReportWords; ++i) info.report[i] = 0u;
    cache[device] = info;
    ready[device].store(true, std::memory_order_release);
  }
  return &cache[device];
}

int32_t take_report(int device) {
  if (device < 0 || device >= kMaxDevices || !ready[device].load(std::memory_order_acquire)) return DQ_OK;  // (nothing has run there)
  unsigned int* report = cache[device].report;
  const auto taken = [&](Report what) {
    return __atomic_load_n(report + what, __ATOMIC_RELAXED) != 0u && __atomic_exchange_n(report + what, 0u, __ATOMIC_RELAXED) != 0u;
  };
  if (taken(kReportWait)) {
    return fail(DQ_ERR_DEVICE, "gemm: a wait inside a block ran out; an output of an earlier call on this device is incomplete");
  }
  if (taken(kReportId)) {
    return fail(DQ_ERR_DEVICE, "embedding lookup: an earlier call on this device was given an id outside its table (its row is NaN)");
  }
  return DQ_OK;
}

namespace {
// A direct-mapped table per thread: no lock, and a collision only costs asking again.
struct KernelFact {
  const void* kernel;
  int device, threads;
  size_t bytes;
  int value;
};
constexpr int kFacts = 512;

KernelFact& fact_slot(KernelFact* table, const void* kernel, int device, size_t mix) {
  const size_t h = (reinterpret_cast<uintptr_t>(kernel) >> 4) * 0x9E3779B97F4A7C15ull + mix * 0xC2B2AE3D27D4EB4Full + static_cast<size_t>(device);
  return table[(h >> 32) % kFacts];
}
}  // namespace

cudaError_t allow_shared_bytes(const void* kernel, size_t bytes) {
  static thread_local KernelFact table[kFacts];
  int device = 0;
  if (const cudaError_t err = cudaGetDevice(&device)) return err;
  KernelFact& f = fact_slot(table, kernel, device, 0);
  if (f.kernel == kernel && f.device == device && f.bytes >= bytes) return cudaSuccess;
  // Always all that the device allows, so that no thread ever lowers what another one relies on.
  const DeviceInfo* dev = device_info();
  cudaFuncAttributes attr = {};
  if (dev == nullptr) return cudaErrorInvalidDevice;
  if (const cudaError_t err = cudaFuncGetAttributes(&attr, kernel)) return err;
  const size_t most = static_cast<size_t>(dev->max_smem_optin) - attr.sharedSizeBytes;
  const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(std::max(most, bytes)));
  if (err == cudaSuccess) f = {kernel, device, 0, std::max(most, bytes), 0};
  return err;
}

cudaError_t resident_ctas_of(int* per_sm, const void* kernel, int threads, size_t bytes) {
  static thread_local KernelFact table[kFacts];
  int device = 0;
  if (const cudaError_t err = cudaGetDevice(&device)) return err;
  KernelFact& f = fact_slot(table, kernel, device, bytes * 2048 + static_cast<size_t>(threads));
  if (f.kernel != kernel || f.device != device || f.threads != threads || f.bytes != bytes) {
    int n = 0;
    if (const cudaError_t err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, bytes)) return err;
    f = {kernel, device, threads, bytes, n};
  }
  *per_sm = f.value;
  return cudaSuccess;
}

}  // namespace dq

extern "C" {

int64_t dq_launch_count(void) { return dq::launches_so_far(); }
const char* dq_last_kernel(void) { return dq::last_kernel(); }


int32_t dq_poll_status(int32_t device) { return dq::take_report(device); }

int32_t dq_gemm_status(void* stream) {
  int device = 0;
  DQ_CUDA(cudaGetDevice(&device));
  DQ_CUDA(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)));
  return dq::take_report(device);
}

int32_t dq_abi_version(void) { return DQ_ABI_VERSION; }
int32_t dq_built_with_cuda(void) { return 1; }
const char* dq_compiled_architectures(void) { return "sm_100a"; }
int32_t dq_gemv_max_rows(void) { return DQ_GEMV_MAX_ROWS; }
int32_t dq_moe_max_tokens(void) { return DQ_MOE_MAX_TOKENS; }
const char* dq_last_error(void) { return dq::error_buffer(); }

int32_t dq_resolve_geometry(const char* op, const dq_weight* w, dq_geometry* out) {
  if (op == nullptr) op = "dynquant";
  DQ_REQUIRE(w != nullptr && out != nullptr, "%s: null weight descriptor", op);
  const int vpb = dq::values_per_block(w->bits);
  DQ_REQUIRE(vpb > 0, "%s: unsupported bit width %d; expected one of {2, 3, 4, 8}", op, w->bits);
  DQ_REQUIRE(dq::dtype_ok(w->meta_dtype), "%s: unsupported scales dtype tag %d", op, w->meta_dtype);
  DQ_REQUIRE(w->rows >= 0 && w->words_per_row >= 0,
             "%s: packed must be 2-D [rows, words], got [%lld, %lld]", op,
             static_cast<long long>(w->rows), static_cast<long long>(w->words_per_row));
  DQ_REQUIRE(w->in_features > 0, "%s: in_features must be positive, got %lld", op,
             static_cast<long long>(w->in_features));
  DQ_REQUIRE(w->group_values > 0,
             "%s: group_values must be a resolved positive count, got %lld. The per-row sentinel "
             "(-1) is the caller's to resolve.",
             op, static_cast<long long>(w->group_values));
  DQ_REQUIRE(w->num_groups > 0, "%s: scales has zero groups", op);
  DQ_REQUIRE(w->words_per_row % w->num_groups == 0,
             "%s: %lld words per row is not divisible by %lld groups; the checkpoint is inconsistent",
             op, static_cast<long long>(w->words_per_row), static_cast<long long>(w->num_groups));
  const int64_t words_per_group = w->words_per_row / w->num_groups;
  const int64_t group_bits = w->group_values * w->bits;
  DQ_REQUIRE(words_per_group * 32 >= group_bits,
             "%s: a group of %lld values at %d-bit needs %lld words but only %lld are stored", op,
             static_cast<long long>(w->group_values), w->bits,
             static_cast<long long>((group_bits + 31) / 32), static_cast<long long>(words_per_group));
  if (w->num_groups > 1) {
    DQ_REQUIRE(group_bits % 32 == 0,
               "%s: group_values=%lld at %d-bit occupies %lld bits, not a whole number of words, so "
               "group 1 would begin mid-word. group_values must be a multiple of %d unless the whole "
               "row is one group.",
               op, static_cast<long long>(w->group_values), w->bits,
               static_cast<long long>(group_bits), DQ_GROUP_SIZE_ALIGNMENT);
    DQ_REQUIRE(words_per_group * 32 == group_bits,
               "%s: %lld words per group does not match %lld bits of payload", op,
               static_cast<long long>(words_per_group), static_cast<long long>(group_bits));
    DQ_REQUIRE(w->num_groups * w->group_values >= w->in_features,
               "%s: %lld groups of %lld cover %lld values, short of in_features=%lld", op,
               static_cast<long long>(w->num_groups), static_cast<long long>(w->group_values),
               static_cast<long long>(w->num_groups * w->group_values),
               static_cast<long long>(w->in_features));
  } else {
    DQ_REQUIRE(w->group_values == w->in_features,
               "%s: a single group must span the row exactly; got group_values=%lld for "
               "in_features=%lld",
               op, static_cast<long long>(w->group_values), static_cast<long long>(w->in_features));
  }
  DQ_REQUIRE(w->rows == 0 || (w->packed != nullptr && w->scales != nullptr),
             "%s: null packed or scales pointer", op);
  DQ_REQUIRE(w->rows < (int64_t{1} << 31) && w->words_per_row < (int64_t{1} << 31) &&
                 w->in_features < (int64_t{1} << 31),
             "%s: tensor dimensions exceed 32-bit indexing", op);
  DQ_REQUIRE(reinterpret_cast<uintptr_t>(w->packed) % 4 == 0 &&
                 reinterpret_cast<uintptr_t>(w->scales) % dq::dtype_size(w->meta_dtype) == 0 &&
                 reinterpret_cast<uintptr_t>(w->offsets) % dq::dtype_size(w->meta_dtype) == 0,
             "%s: misaligned packed / scales / offsets pointer", op);

  out->group_values = static_cast<int32_t>(w->group_values);
  out->num_groups = static_cast<int32_t>(w->num_groups);
  out->words_per_group = static_cast<int32_t>(words_per_group);
  out->words_per_row = static_cast<int32_t>(w->words_per_row);
  out->in_features = static_cast<int32_t>(w->in_features);
  out->blocks_per_group = static_cast<int32_t>((w->group_values + vpb - 1) / vpb);
  out->blocks_per_row = out->num_groups * out->blocks_per_group;
  return DQ_OK;
}

}  // extern "C"
