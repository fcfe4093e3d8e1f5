// Packed words -> dense [rows, in_features] matrix, bit-exact against the
// reference's QuantTensor.dequantize.
//
// Replaces dequant_kernel / dequant_cuda
// (packages/dynquant-kernels/csrc/quant/dequant.cu:47-93, :130-165).  It is the
// prefill (M > 8) feed for a dense GEMM, the embedding-row decoder, and the
// anchor of the parity suite: a wrong bit anywhere in the decode shows here as
// a wrong number, with no accumulation to hide behind.
//
// Arithmetic: w = float(q) * scale, then + offset, both rounded to fp32
// (packages/dynquant-core/src/dynquant/quant/tensor.py:417-426 multiplies and
// then adds), then one rounding to the output dtype.  With fp16/bf16 scales the
// product is exact in fp32, so this equals the reference CUDA kernel's single
// fmaf as well; with fp32 scales it follows the torch definition.  An absent
// offsets tensor means "no add", not "+0".
//
// Two kernels.  dequant_octet_kernel is the one nearly every tensor takes (in_features and
// the group size multiples of 8): a thread produces 8 consecutive values -- one 16-byte
// store for a 16-bit output, so a warp writes 512 contiguous bytes per store instruction --
// from the 8 * BITS bits at bit 8 * BITS * octet of its row (the packed row is one
// contiguous LSB-first bit string: groups are whole numbers of 32-value blocks).  dequant_kernel
// is the general one: one thread per block of 16/32/8/4 values at 2/3/4/8-bit, any tail.
#include <algorithm>
#include <type_traits>

#include "dq_decode.cuh"

namespace dq {
namespace {

constexpr int kDequantThreads = 128;

struct DequantArgs {
  const uint32_t* packed;
  const void* scales;
  const void* offsets;
  void* out;
  const void* ids;       // null, or the packed row of every output row
  int ids_are_32;        // int32 ids (else int64)
  int table_rows;        // rows of the packed tensor (ids lie below it)
  unsigned int* report;  // an id that does not is reported
  int meta_dtype, out_dtype;
  int rows;              // output rows
  int words_per_row, num_groups, words_per_group, group_values, in_features;
  int blocks_per_group, blocks_per_row;
};

// Which packed row an output row of an embedding lookup comes from: the id at its place.
// An id outside the table gives -1 -- the kernels then write a row of NaN and report it, which the host
// raises: the gather that this replaces failed a device assertion, which costs the caller the context.
__device__ __forceinline__ int source_row(const DequantArgs& a, int row) {
  const int64_t id = a.ids_are_32 ? static_cast<int64_t>(__ldg(static_cast<const int*>(a.ids) + row))
                                  : static_cast<int64_t>(__ldg(static_cast<const long long*>(a.ids) + row));
  return id >= 0 && id < a.table_rows ? static_cast<int>(id) : -1;
}

// U runs of 8 consecutive values per thread, kDequantThreads octets apart, so that a CTA
// writes one contiguous stretch of the output and the grid writes the output front to back.
// `group_shift` >= 0: the group size is 2^shift.  `per_row_magic` = ceil(2^64 / octets_per_row):
// the high half of its product with an octet's number is the octet's row (exact below 2^32).
//
// Bound by the stores (2 bytes written per value, bits/8 read): 14336 x 4096 at 3 / 4 / 8 bits takes
// 38 / 37 / 37 us where filling the output with zeros takes 33.  (Octets over blockIdx.x and rows
// over blockIdx.y, one octet per thread: 52 / 44 / 44 -- and 14 us against 10 on 14080 x 768, whose
// rows left most threads of a CTA idle.)  256 threads and 4 octets: 43; 2 octets: 39 to 41.
template <int BITS, int U, bool IDS>
__global__ void __launch_bounds__(kDequantThreads) dequant_octet_kernel(const DequantArgs a, unsigned octets_per_row,
                                                                        unsigned long long per_row_magic, unsigned total,
                                                                        int group_shift) {
  const bool has_offsets = a.offsets != nullptr;
  constexpr uint32_t kMask = (1u << BITS) - 1u;
  const bool fused = a.meta_dtype != DQ_F32;  // q * scale is exact in fp32: one fma is multiply, then add
  const unsigned first = blockIdx.x * (kDequantThreads * U) + threadIdx.x;
  uint32_t lo[U], hi[U];
  float scale[U], offset[U];
  bool known[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const unsigned at = first + u * kDequantThreads;
    lo[u] = hi[u] = 0u, scale[u] = offset[u] = 0.0f, known[u] = true;
    if (at < total) {
      const int row = static_cast<int>(__umul64hi(at, per_row_magic));
      const int o = static_cast<int>(at - row * octets_per_row);
      const int from = IDS ? source_row(a, row) : row;
      if constexpr (IDS) known[u] = from >= 0;
      if (!IDS || from >= 0) {
        const int bit = o * 8 * BITS;
        const int word = bit >> 5;
        const uint32_t* src = a.packed + static_cast<int64_t>(from) * a.words_per_row;
        // the octet's 8 * BITS bits (64 at 8-bit: two whole words)
        if constexpr (BITS == 8) {
          const uint2 v = __ldg(reinterpret_cast<const uint2*>(src) + o);
          lo[u] = v.x, hi[u] = v.y;
        } else {
          lo[u] = __ldg(src + word);
          if constexpr (BITS == 3) hi[u] = (bit & 31) > 8 ? __ldg(src + word + 1) : 0u;  // 24 bits from bit (bit & 31)
        }
        const int g = group_shift >= 0 ? ((o * 8) >> group_shift) : (o * 8) / a.group_values;
        const int64_t meta = static_cast<int64_t>(from) * a.num_groups + g;
        scale[u] = load_f32(a.scales, meta, a.meta_dtype);
        if (has_offsets) offset[u] = load_f32(a.offsets, meta, a.meta_dtype);
        if constexpr (BITS == 2) lo[u] >>= bit & 31;
        if constexpr (BITS == 3) lo[u] = __funnelshift_r(lo[u], hi[u], bit & 31);
      }
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const unsigned at = first + u * kDequantThreads;
    if (at >= total) break;
    float vals[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      uint32_t q;
      if constexpr (BITS == 8) {
        q = ((i < 4 ? lo[u] : hi[u]) >> (8 * (i & 3))) & 0xFFu;
      } else {
        q = (lo[u] >> (BITS * i)) & kMask;
      }
      // float(q) without the conversion unit (a quarter-rate pipe): 2^23 + q is exactly
      // representable, so OR-ing q into the mantissa of 2^23 and subtracting 2^23 is exact
      const float qf = __uint_as_float(0x4B000000u | q) - 8388608.0f;
      if (fused && has_offsets) {
        vals[i] = __fmaf_rn(qf, scale[u], offset[u]);
      } else {
        vals[i] = __fmul_rn(qf, scale[u]);
        if (has_offsets) vals[i] = __fadd_rn(vals[i], offset[u]);
      }
      if (IDS && !known[u]) vals[i] = __int_as_float(0x7FC00000);
    }
    if (IDS && !known[u]) report_to_host(a.report, kReportId);
    // rows are whole octets, so octet `at` of the output starts at value 8 * at
    if (a.out_dtype == DQ_F32) {
      float4* dst = reinterpret_cast<float4*>(a.out) + static_cast<size_t>(at) * 2;
      dst[0] = make_float4(vals[0], vals[1], vals[2], vals[3]);
      dst[1] = make_float4(vals[4], vals[5], vals[6], vals[7]);
    } else {
      uint32_t p16[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        p16[j] = round_pair_to_16(vals[2 * j], vals[2 * j + 1], a.out_dtype);
      }
      reinterpret_cast<uint4*>(a.out)[at] = make_uint4(p16[0], p16[1], p16[2], p16[3]);
    }
  }
}

template <int BITS>
__global__ void __launch_bounds__(kDequantThreads) dequant_kernel(const DequantArgs a) {
  constexpr int VB = Block<BITS>::kValues;
  constexpr int WB = Block<BITS>::kWords;
  const int64_t total = static_cast<int64_t>(a.rows) * a.blocks_per_row;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  const bool has_offsets = a.offsets != nullptr;

  for (int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total;
       idx += stride) {
    const int row = static_cast<int>(idx / a.blocks_per_row);
    const int blk = static_cast<int>(idx - static_cast<int64_t>(row) * a.blocks_per_row);
    const int g = blk / a.blocks_per_group;
    const int bg = blk - g * a.blocks_per_group;
    const int word_base = g * a.words_per_group + (bg * VB * BITS) / 32;
    const int words_left = a.words_per_row - word_base;
    const int value_base = g * a.group_values + bg * VB;
    // Values of this block that exist: bounded by the group (per-row tail) and
    // by in_features (zero pad of the last group).
    const int live = min(min(VB, a.group_values - bg * VB), a.in_features - value_base);
    if (live <= 0) {
      continue;
    }
    const int64_t out_base = static_cast<int64_t>(row) * a.in_features + value_base;
    const int from = a.ids == nullptr ? row : source_row(a, row);
    if (from < 0) {
      report_to_host(a.report, kReportId);
      for (int j = 0; j < live; ++j) store_f32(a.out, out_base + j, a.out_dtype, __int_as_float(0x7FC00000));
      continue;
    }
    const uint32_t* src = a.packed + static_cast<int64_t>(from) * a.words_per_row + word_base;
    const int64_t meta = static_cast<int64_t>(from) * a.num_groups + g;
    const float scale = load_f32(a.scales, meta, a.meta_dtype);
    const float offset = has_offsets ? load_f32(a.offsets, meta, a.meta_dtype) : 0.0f;

    if (live == VB && words_left >= WB) {
      uint32_t w[WB];
#pragma unroll
      for (int i = 0; i < WB; ++i) {
        w[i] = __ldg(src + i);
      }
      float vals[VB];
      for_each_pair<BITS>(w, [&](int p, float2 q2) {
        float lo = __fmul_rn(q2.x, scale);
        float hi = __fmul_rn(q2.y, scale);
        if (has_offsets) {
          lo = __fadd_rn(lo, offset);
          hi = __fadd_rn(hi, offset);
        }
        vals[2 * p] = lo;
        vals[2 * p + 1] = hi;
      });
      if (a.out_dtype == DQ_F32) {
        float* dst = reinterpret_cast<float*>(a.out) + out_base;
        if ((reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
#pragma unroll
          for (int j = 0; j < VB / 4; ++j) {
            reinterpret_cast<float4*>(dst)[j] =
                make_float4(vals[4 * j], vals[4 * j + 1], vals[4 * j + 2], vals[4 * j + 3]);
          }
        } else {
#pragma unroll
          for (int j = 0; j < VB; ++j) {
            dst[j] = vals[j];
          }
        }
      } else {
        unsigned short* dst = reinterpret_cast<unsigned short*>(a.out) + out_base;
        uint32_t packed16[VB / 2];
#pragma unroll
        for (int j = 0; j < VB / 2; ++j) {
          packed16[j] = round_to_16(vals[2 * j], a.out_dtype) |
                        (round_to_16(vals[2 * j + 1], a.out_dtype) << 16);
        }
        const uintptr_t addr = reinterpret_cast<uintptr_t>(dst);
        if (VB % 8 == 0 && (addr & 15) == 0) {
#pragma unroll
          for (int j = 0; j < VB / 8; ++j) {
            reinterpret_cast<uint4*>(dst)[j] = make_uint4(packed16[4 * j], packed16[4 * j + 1],
                                                          packed16[4 * j + 2], packed16[4 * j + 3]);
          }
        } else if ((addr & 3) == 0) {
#pragma unroll
          for (int j = 0; j < VB / 2; ++j) {
            reinterpret_cast<uint32_t*>(dst)[j] = packed16[j];
          }
        } else {
#pragma unroll
          for (int j = 0; j < VB / 2; ++j) {
            dst[2 * j] = static_cast<unsigned short>(packed16[j] & 0xFFFFu);
            dst[2 * j + 1] = static_cast<unsigned short>(packed16[j] >> 16);
          }
        }
      }
    } else {
      for (int j = 0; j < live; ++j) {
        const float q = static_cast<float>(code_at<BITS>(src, j, words_left));
        float v = __fmul_rn(q, scale);
        if (has_offsets) {
          v = __fadd_rn(v, offset);
        }
        store_f32(a.out, out_base + j, a.out_dtype, v);
      }
    }
  }
}

}  // namespace
}  // namespace dq

namespace dq {
namespace {

int32_t launch_dequant(const dq_weight* w, const dq_geometry& g, const void* ids, int ids_are_32, int64_t rows, void* out,
                       int32_t out_dtype, cudaStream_t s) {
  DequantArgs a = {};
  a.packed = static_cast<const uint32_t*>(w->packed);
  a.scales = w->scales;
  a.offsets = w->offsets;
  a.out = out;
  a.ids = ids;
  a.ids_are_32 = ids_are_32;
  a.table_rows = static_cast<int>(w->rows);
  a.meta_dtype = w->meta_dtype;
  a.out_dtype = out_dtype;
  a.rows = static_cast<int>(rows);
  a.words_per_row = g.words_per_row;
  a.num_groups = g.num_groups;
  a.words_per_group = g.words_per_group;
  a.group_values = g.group_values;
  a.in_features = g.in_features;
  a.blocks_per_group = g.blocks_per_group;
  a.blocks_per_row = g.blocks_per_row;

  const DeviceInfo* dev = device_info();
  if (dev == nullptr) return DQ_ERR_CUDA;
  a.report = dev->report;
  // The octet kernel: whole octets per row and per group, 16-byte aligned output rows, and
  // (8-bit) 8-byte aligned packed rows.
  const size_t out_elem = static_cast<size_t>(dtype_size(out_dtype));
  const bool octets = a.in_features % 8 == 0 && a.group_values % 8 == 0 &&
                      reinterpret_cast<uintptr_t>(out) % 16 == 0 && (a.in_features * out_elem) % 16 == 0 &&
                      (w->bits != 8 || (reinterpret_cast<uintptr_t>(a.packed) % 8 == 0 && a.words_per_row % 2 == 0));
  const int64_t num_octets = static_cast<int64_t>(a.rows) * (a.in_features / 8);
  if (octets && a.in_features > 8 && num_octets < (int64_t{1} << 32)) {
    const unsigned per_row = static_cast<unsigned>(a.in_features / 8);
    const unsigned long long magic = ~0ull / per_row + 1;  // ceil(2^64 / per_row)
    int shift = -1;
    if ((a.group_values & (a.group_values - 1)) == 0) {
      shift = 0;
      while ((1 << shift) < a.group_values) ++shift;
    }
    const unsigned total = static_cast<unsigned>(num_octets);
    // Four octets per thread from a full wave of such threads on; below it more CTAs are worth more
    // than loads in flight (6912 x 1024, 0.9 M octets: 7.1 us with one, 8.3 with four).
    const bool four = num_octets >= static_cast<int64_t>(dev->sm_count) * 2048 * 4;
    const unsigned grid = static_cast<unsigned>(ceil_div(num_octets, kDequantThreads * (four ? 4 : 1)));
    const auto run = [&](auto ids) {
      constexpr bool IDS = decltype(ids)::value;
      const auto pick = [&](auto one, auto many) { (four ? many : one)<<<grid, kDequantThreads, 0, s>>>(a, per_row, magic, total, shift); };
      switch (w->bits) {
        case 2: pick(dequant_octet_kernel<2, 1, IDS>, dequant_octet_kernel<2, 4, IDS>); break;
        case 3: pick(dequant_octet_kernel<3, 1, IDS>, dequant_octet_kernel<3, 4, IDS>); break;
        case 4: pick(dequant_octet_kernel<4, 1, IDS>, dequant_octet_kernel<4, 4, IDS>); break;
        default: pick(dequant_octet_kernel<8, 1, IDS>, dequant_octet_kernel<8, 4, IDS>); break;
      }
    };
    if (a.ids != nullptr) {
      run(std::true_type{});
    } else {
      run(std::false_type{});
    }
    DQ_CHECK_LAUNCH("dequant");
    return DQ_OK;
  }
  const int64_t total = static_cast<int64_t>(a.rows) * a.blocks_per_row;
  const int64_t want = ceil_div(total, kDequantThreads);
  const int grid = static_cast<int>(std::min<int64_t>(want, static_cast<int64_t>(dev->sm_count) * 32));
  switch (w->bits) {
    case 2:
      dequant_kernel<2><<<grid, kDequantThreads, 0, s>>>(a);
      break;
    case 3:
      dequant_kernel<3><<<grid, kDequantThreads, 0, s>>>(a);
      break;
    case 4:
      dequant_kernel<4><<<grid, kDequantThreads, 0, s>>>(a);
      break;
    default:
      dequant_kernel<8><<<grid, kDequantThreads, 0, s>>>(a);
      break;
  }
  DQ_CHECK_LAUNCH("dequant");
  return DQ_OK;
}

}  // namespace
}  // namespace dq

extern "C" int32_t dq_dequant(const dq_weight* w, void* out, int32_t out_dtype, void* stream) {
  dq_geometry g;
  if (const int32_t rc = dq_resolve_geometry("dequant", w, &g)) return rc;
  DQ_REQUIRE(dq::dtype_ok(out_dtype), "dequant: unsupported output dtype tag %d", out_dtype);
  if (w->rows == 0) return DQ_OK;
  DQ_REQUIRE(out != nullptr, "dequant: null output pointer");
  return dq::launch_dequant(w, g, nullptr, 0, w->rows, out, out_dtype, static_cast<cudaStream_t>(stream));
}

extern "C" int32_t dq_dequant_rows(const dq_weight* w, const void* ids, int32_t ids_are_int32, int64_t count, void* out,
                                   int32_t out_dtype, void* stream) {
  dq_geometry g;
  if (const int32_t rc = dq_resolve_geometry("dequant_rows", w, &g)) return rc;
  DQ_REQUIRE(dq::dtype_ok(out_dtype), "dequant_rows: unsupported output dtype tag %d", out_dtype);
  DQ_REQUIRE(count >= 0 && count < (1LL << 31), "dequant_rows: bad row count %lld", static_cast<long long>(count));
  if (count == 0) return DQ_OK;
  DQ_REQUIRE(ids != nullptr && out != nullptr, "dequant_rows: null pointer");
  return dq::launch_dequant(w, g, ids, ids_are_int32 != 0, count, out, out_dtype, static_cast<cudaStream_t>(stream));
}
