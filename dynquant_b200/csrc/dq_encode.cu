// Dense matrix -> packed words, scales and offsets: the min/max group encoder of
// QuantTensor.from_dense (dynquant_b200/format.py; reference quant/tensor.py:239-396 without the
// clip search), bit for bit what that function computes on the host.
//
// Per group: lo / hi over its values (a last, partial group is padded with zeros, which take
// part), scale and offset rounded to the storage type BEFORE any code is derived from them, then
// code = clamp(rint((w - offset) / scale), 0, 2^bits - 1).  Every operation is one IEEE fp32
// operation in the order of the host code: __fsub_rn, __fdiv_rn (never a reciprocal), rintf.
//
// Bound by HBM: 2 bytes read and bits/8 + 4/group written per value.  A thread takes 8 consecutive
// values (one 16-byte load of a 16-bit weight) and keeps them in registers, so the matrix is read
// once; the group/8 lanes of a group agree on lo and hi by shuffles; a thread's 8 codes are 8*bits
// contiguous bits of the row, which leave as one 2-, 4- or 8-byte store (3 bits: the quad that
// shares 32 values exchanges its 24-bit pieces and three of its lanes store a word each).
// 2048 x 6144 at 4 bits: 37 ms through the host's tensor operations and two copies over PCIe; here
// the launch is a few microseconds.
//
// The kernels that multiply by packed weights request them BEFORE their griddepcontrol.wait, as data
// that no kernel in flight writes.  Launched right behind this one they would have a programmatic edge
// to it, which an ordinary kernel releases when its blocks exit and not when its stores are visible.
// So a memset follows: an ordinary edge on both sides, behind which the words are complete.
#include <algorithm>

#include "dq_common.cuh"

namespace dq {
namespace {

constexpr int kEncodeThreads = 256;

__device__ unsigned int g_after_encode;  // what the memset behind the kernel writes; nobody reads it

struct EncodeArgs {
  const void* w;
  uint32_t* packed;
  void* scales;
  void* offsets;
  int w_dtype, meta_dtype;
  int rows, in_features, octets_per_row;  // octets: of the padded row
  int words_per_row, num_groups;
  int symmetric;
};

// torch's amin / amax hand a NaN on; fminf and fmaxf would drop it.
__device__ __forceinline__ float min_nan(float a, float b) {
  float d;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ float max_nan(float a, float b) {
  float d;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}

__device__ __forceinline__ float round_through(float v, int dtype) {
  if (dtype == DQ_F16) return __half2float(__float2half_rn(v));
  if (dtype == DQ_BF16) return __bfloat162float(__float2bfloat16_rn(v));
  return v;
}

// LANES = group / 8 threads of a warp hold one group.
template <int BITS, int LANES>
__global__ void __launch_bounds__(kEncodeThreads) encode_kernel(const EncodeArgs a) {
  constexpr float kMax = static_cast<float>((1 << BITS) - 1);
  constexpr int kHalf = 1 << (BITS - 1);
  const int64_t total = static_cast<int64_t>(a.rows) * a.octets_per_row;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * kEncodeThreads;
  // (whole warps stay in the loop: octets_per_row is a multiple of LANES, so a group's lanes agree)
  const int64_t rounded = (total + kWarp - 1) / kWarp * kWarp;
  for (int64_t at = static_cast<int64_t>(blockIdx.x) * kEncodeThreads + threadIdx.x; at < rounded; at += stride) {
    const bool live = at < total;
    const int row = live ? static_cast<int>(at / a.octets_per_row) : 0;
    const int octet = live ? static_cast<int>(at - static_cast<int64_t>(row) * a.octets_per_row) : 0;
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = 0.0f;
    if (live && octet * 8 < a.in_features) {  // in_features is a multiple of 8: whole octets exist or are padding
      const int64_t base = static_cast<int64_t>(row) * a.in_features + octet * 8;
      if (a.w_dtype == DQ_F32) {
        const float4* p = reinterpret_cast<const float4*>(static_cast<const float*>(a.w) + base);
        const float4 x = __ldg(p), y = __ldg(p + 1);
        v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w, v[4] = y.x, v[5] = y.y, v[6] = y.z, v[7] = y.w;
      } else {
        const uint4 raw = ldg_stream_128(static_cast<const unsigned short*>(a.w) + base);
        const uint32_t r[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (a.w_dtype == DQ_F16) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&r[i]));
            v[2 * i] = f.x, v[2 * i + 1] = f.y;
          } else {
            v[2 * i] = __uint_as_float(r[i] << 16), v[2 * i + 1] = __uint_as_float(r[i] & 0xFFFF0000u);
          }
        }
      }
    }
    float lo = v[0], hi = v[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) lo = min_nan(lo, v[i]), hi = max_nan(hi, v[i]);
#pragma unroll
    for (int d = LANES / 2; d > 0; d >>= 1) {
      lo = min_nan(lo, __shfl_xor_sync(0xffffffffu, lo, d));
      hi = max_nan(hi, __shfl_xor_sync(0xffffffffu, hi, d));
    }
    float scale, offset;
    if (a.symmetric) {
      constexpr float kDiv = static_cast<float>(kHalf - 1 > 1 ? kHalf - 1 : 1);
      scale = round_through(__fdiv_rn(max_nan(fabsf(hi), fabsf(lo)), kDiv), a.meta_dtype);
      offset = round_through(__fmul_rn(-static_cast<float>(kHalf), scale), a.meta_dtype);
    } else {
      scale = round_through(__fdiv_rn(__fsub_rn(hi, lo), kMax), a.meta_dtype);
      offset = round_through(lo, a.meta_dtype);
    }
    if (hi == lo) scale = 0.0f, offset = round_through(lo, a.meta_dtype);  // a constant group

    uint32_t bits_lo = 0u, bits_hi = 0u;  // the octet's 8 * BITS bits
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float c = 0.0f;
      if (scale != 0.0f) c = fminf(fmaxf(rintf(__fdiv_rn(__fsub_rn(v[i], offset), scale)), 0.0f), kMax);
      const uint32_t q = static_cast<uint32_t>(__float2int_rz(c));
      if constexpr (BITS == 8) {
        if (i < 4) bits_lo |= q << (8 * i); else bits_hi |= q << (8 * (i - 4));
      } else {
        bits_lo |= q << (BITS * i);
      }
    }
    uint32_t next = 0u;
    if constexpr (BITS == 3) next = __shfl_down_sync(0xffffffffu, bits_lo, 1);
    if (live) {
      uint32_t* row_words = a.packed + static_cast<int64_t>(row) * a.words_per_row;
      if constexpr (BITS == 8) {
        *reinterpret_cast<uint2*>(row_words + octet * 2) = make_uint2(bits_lo, bits_hi);
      } else if constexpr (BITS == 4) {
        row_words[octet] = bits_lo;
      } else if constexpr (BITS == 2) {
        reinterpret_cast<unsigned short*>(row_words)[octet] = static_cast<unsigned short>(bits_lo);
      } else {
        const int j = octet & 3;  // word j of the 96-bit block: the rest of piece j, the start of piece j + 1
        if (j < 3) row_words[(octet >> 2) * 3 + j] = (bits_lo >> (8 * j)) | (next << (24 - 8 * j));
      }
      if (octet % LANES == 0) {
        const int64_t meta = static_cast<int64_t>(row) * a.num_groups + octet / LANES;
        store_f32(a.scales, meta, a.meta_dtype, scale);
        store_f32(a.offsets, meta, a.meta_dtype, offset);
      }
    }
  }
}

template <int BITS>
void launch_encode(const EncodeArgs& a, int lanes, int grid, cudaStream_t s) {
  switch (lanes) {
    case 4: encode_kernel<BITS, 4><<<grid, kEncodeThreads, 0, s>>>(a); break;
    case 8: encode_kernel<BITS, 8><<<grid, kEncodeThreads, 0, s>>>(a); break;
    case 16: encode_kernel<BITS, 16><<<grid, kEncodeThreads, 0, s>>>(a); break;
    default: encode_kernel<BITS, 32><<<grid, kEncodeThreads, 0, s>>>(a); break;
  }
}

}  // namespace
}  // namespace dq

extern "C" int32_t dq_encode(const void* w, int32_t w_dtype, int64_t rows, int64_t in_features, int32_t bits,
                             int64_t group_values, int32_t symmetric, void* packed, void* scales, void* offsets,
                             int32_t meta_dtype, void* stream) {
  DQ_REQUIRE(dq::values_per_block(bits) > 0, "encode: unsupported bit width %d; expected one of {2, 3, 4, 8}", bits);
  DQ_REQUIRE(dq::dtype_ok(w_dtype) && dq::dtype_ok(meta_dtype), "encode: unsupported dtype tag");
  DQ_REQUIRE(rows >= 0 && in_features > 0 && rows < (1LL << 31) && in_features < (1LL << 31), "encode: bad sizes");
  if (rows == 0) return DQ_OK;
  DQ_REQUIRE(w != nullptr && packed != nullptr && scales != nullptr && offsets != nullptr, "encode: null pointer");
  if ((group_values != 32 && group_values != 64 && group_values != 128 && group_values != 256) || in_features % 8 != 0 ||
      reinterpret_cast<uintptr_t>(w) % 16 != 0 || reinterpret_cast<uintptr_t>(packed) % 8 != 0) {
    return dq::fail(DQ_ERR_UNSUPPORTED, "encode: groups of 32, 64, 128 or 256 values, whole octets per row, aligned buffers");
  }
  const dq::DeviceInfo* dev = dq::device_info();
  if (dev == nullptr) return DQ_ERR_CUDA;
  dq::EncodeArgs a = {};
  a.w = w;
  a.packed = static_cast<uint32_t*>(packed);
  a.scales = scales;
  a.offsets = offsets;
  a.w_dtype = w_dtype;
  a.meta_dtype = meta_dtype;
  a.rows = static_cast<int>(rows);
  a.in_features = static_cast<int>(in_features);
  a.num_groups = static_cast<int>(dq::ceil_div(in_features, group_values));
  a.octets_per_row = static_cast<int>(a.num_groups * (group_values / 8));
  a.words_per_row = static_cast<int>(a.num_groups * group_values * bits / 32);
  a.symmetric = symmetric;
  const int64_t total = static_cast<int64_t>(a.rows) * a.octets_per_row;
  const int grid = static_cast<int>(std::min<int64_t>(dq::ceil_div(total, dq::kEncodeThreads), static_cast<int64_t>(dev->sm_count) * 64));
  const int lanes = static_cast<int>(group_values / 8);
  auto s = static_cast<cudaStream_t>(stream);
  switch (bits) {
    case 2: dq::launch_encode<2>(a, lanes, grid, s); break;
    case 3: dq::launch_encode<3>(a, lanes, grid, s); break;
    case 4: dq::launch_encode<4>(a, lanes, grid, s); break;
    default: dq::launch_encode<8>(a, lanes, grid, s); break;
  }
  DQ_CHECK_LAUNCH("encode");
  void* word = nullptr;
  DQ_CUDA(cudaGetSymbolAddress(&word, dq::g_after_encode));
  DQ_CUDA(cudaMemsetAsync(word, 0, sizeof(unsigned int), s));
  return DQ_OK;
}
