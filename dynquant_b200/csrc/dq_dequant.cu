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
// Three kernels.  dequant_pairs_kernel takes what models have: 16-bit metadata and output, in_features and
// the group size multiples of 16.  dequant_octet_kernel takes the rest of the regular tensors (in_features and
// the group size multiples of 8, any types): a thread produces 8 consecutive values -- one 16-byte
// store for a 16-bit output, so a warp writes 512 contiguous bytes per store instruction --
// from the 8 * BITS bits at bit 8 * BITS * octet of its row (the packed row is one
// contiguous LSB-first bit string: groups are whole numbers of 32-value blocks).  dequant_kernel
// is the general one: one thread per block of 16/32/8/4 values at 2/3/4/8-bit, any tail.
#include <algorithm>
#include <type_traits>

#include "dq_decode.cuh"
#include "dq_umma_decode.cuh"

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
// Bound by its instructions: 14336 x 4096 at 3 / 4 / 8 bits takes 36 / 33 / 36 us in a graph, filling its
// output 18.6.  (Octets over blockIdx.x and rows
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

// 16 codes -> eight registers of two, each as an exact 16-bit number of the METADATA's type: codes `first` and
// `second` of register j.  ONE AND-OR puts two codes into the mantissas of a power of two, one packed subtraction
// takes that off again.
template <int BITS, bool MBF16>
struct Codes16 {
  static constexpr int kMantissa = MBF16 ? 7 : 10;
  static constexpr int first(int j) { return BITS == 8 ? 2 * j : BITS == 4 ? j / 4 * 8 + j % 4 : j; }
  static constexpr int second(int j) { return BITS == 8 ? 2 * j + 1 : BITS == 4 ? j / 4 * 8 + j % 4 + 4 : j + 8; }
  static __device__ __forceinline__ uint32_t minus(uint32_t a, uint32_t b) {
    if constexpr (MBF16) {
      const __nv_bfloat162 d = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
      return *reinterpret_cast<const uint32_t*>(&d);
    } else {
      const __half2 d = __hsub2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
      return *reinterpret_cast<const uint32_t*>(&d);
    }
  }
  // The codes at bit `place` of both halves; place + BITS <= kMantissa.
  static __device__ __forceinline__ uint32_t take(uint32_t u, int place) {
    const uint32_t mask = ((1u << BITS) - 1u) << place, magic = static_cast<uint32_t>((MBF16 ? 127 : 15) + kMantissa - place) << kMantissa;
    return minus((u & (mask | (mask << 16))) | (magic | (magic << 16)), magic | (magic << 16));
  }
  // `w`: the words that hold the codes, from bit `shift` on (3 bits: 0 or 16; else 0)
  static __device__ __forceinline__ void get(const uint32_t* w, int shift, uint32_t* q) {
    if constexpr (BITS == 8) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if constexpr (MBF16) {
          // Seven bits fit the mantissa: 128 + low bits; the top bit toggles -256 / -128.  Their sum is code - 128.
          const uint32_t p = __byte_perm(w[j / 2], 0u, (j & 1) ? 0x4342u : 0x4140u);
          q[j] = minus((p & 0x007F007Fu) | 0x43004300u, (p & 0x00800080u) ^ 0x43804380u);
          q[j] = minus(q[j], 0xC300C300u);
        } else {
          q[j] = minus(__byte_perm(w[j / 2], 0x64006400u, (j & 1) ? 0x7372u : 0x7170u), 0x64006400u);
        }
      }
    } else if constexpr (BITS == 3) {
      // Codes 0..7 and 8..15 are 24 bits each: their lower and upper 16 bits side by side.
      const unsigned long long v = ((static_cast<unsigned long long>(w[1]) << 32) | w[0]) >> shift;
      const uint32_t a = static_cast<uint32_t>(v), b = static_cast<uint32_t>(v >> 24);
      const uint32_t low = __byte_perm(a, b, 0x5410u), high = __byte_perm(a, b, 0x6521u);
      constexpr int kPlaces = kMantissa / 3;
#pragma unroll
      for (int j = 0; j < 5; ++j) q[j] = take(low >> (3 * (j - j % kPlaces)), 3 * (j % kPlaces));
#pragma unroll
      for (int j = 0; j < 3; ++j) q[5 + j] = take(high >> (7 + 3 * (j - j % kPlaces)), 3 * (j % kPlaces));
    } else {
      constexpr int kPlaces = kMantissa / BITS, kOfWord = 16 / BITS;  // registers of a word: 8 or 4
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int i = j % kOfWord;
        q[j] = take(w[j / kOfWord] >> (BITS * (i - i % kPlaces)), BITS * (i % kPlaces));
      }
    }
  }
};

// U runs of 16 consecutive values per thread, one 32-byte store each, kDequantThreads runs apart (as
// dequant_octet_kernel; `runs_per_row`, `per_row_magic`, `total` count runs).  A code is an exact number of the
// metadata's type, so that ONE mixed-precision fma, q * s + o with 16-bit factors and an fp32 addend, is the
// exact product and the one rounding of the sum that the format asks for.  No offsets: the addend is -0, which
// changes no sum, not even a zero's sign.
//
// Bound by memory: bits / 8 bytes read and 2 written per value.  14336 x 4096 at 2 / 3 / 4 / 8 bits: 22.7 / 24.4 /
// 24.9 / 28.9 us (5.9 to 6.2 TB/s; filling such an output takes 18.6) where dequant_octet_kernel takes 36.4 /
// 36.5 / 33.0 / 35.7: that one decodes value by value and reads scale and offset for every eight.  This one executes
// 7.1 instructions a value in all (3 bits), at 69 % of the issue slots.
template <int BITS, bool MBF16, int U, bool IDS>
__global__ void __launch_bounds__(kDequantThreads) dequant_pairs_kernel(const DequantArgs a, unsigned runs_per_row, unsigned long long per_row_magic,
                                                                        unsigned total, int group_shift) {
  constexpr int kWords = BITS == 3 ? 2 : BITS / 2;
  const unsigned first = blockIdx.x * (kDequantThreads * U) + threadIdx.x;
  uint32_t w[U][kWords];
  unsigned short scale[U], offset[U];
  int shift[U];
  bool known[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const unsigned at = min(first + u * kDequantThreads, total - 1);
    const int row = static_cast<int>(__umul64hi(at, per_row_magic)), run = static_cast<int>(at - row * runs_per_row);
    int from = row;
    known[u] = true;
    if constexpr (IDS) {
      from = source_row(a, row);
      known[u] = from >= 0;
      from = max(from, 0);
    }
    const uint32_t* src = a.packed + static_cast<int64_t>(from) * a.words_per_row + run * BITS / 2;
    shift[u] = 0;
    if constexpr (BITS == 2) {
      w[u][0] = __ldg(src);
    } else if constexpr (BITS == 3) {
      shift[u] = (run & 1) * 16;
      w[u][0] = __ldg(src), w[u][1] = __ldg(src + 1);
    } else if constexpr (BITS == 4) {
      const uint2 v = __ldg(reinterpret_cast<const uint2*>(src));
      w[u][0] = v.x, w[u][1] = v.y;
    } else {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(src));
      w[u][0] = v.x, w[u][1] = v.y, w[u][2] = v.z, w[u][3] = v.w;
    }
    const int64_t meta = static_cast<int64_t>(from) * a.num_groups + (group_shift >= 0 ? (run * 16) >> group_shift : (run * 16) / a.group_values);
    scale[u] = __ldg(static_cast<const unsigned short*>(a.scales) + meta);
    offset[u] = a.offsets != nullptr ? __ldg(static_cast<const unsigned short*>(a.offsets) + meta) : 0x8000;
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const unsigned at = first + u * kDequantThreads;
    if (at >= total) break;
    float o = MBF16 ? __uint_as_float(static_cast<uint32_t>(offset[u]) << 16) : __half2float(__ushort_as_half(offset[u]));
    if constexpr (IDS) {
      if (!known[u]) {
        o = __int_as_float(0x7FC00000);
        report_to_host(a.report, kReportId);
      }
    }
    using C = Codes16<BITS, MBF16>;
    uint32_t q[8], out[8];
    float f[16];
    C::get(w[u], shift[u], q);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      f[C::first(j)] = umma::fma_half<MBF16>(q[j], false, scale[u], o);
      f[C::second(j)] = umma::fma_half<MBF16>(q[j], true, scale[u], o);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) out[j] = round_pair_to_16(f[2 * j], f[2 * j + 1], a.out_dtype);
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(static_cast<unsigned char*>(a.out) + static_cast<size_t>(at) * 32), "r"(out[0]),
                 "r"(out[1]), "r"(out[2]), "r"(out[3]), "r"(out[4]), "r"(out[5]), "r"(out[6]), "r"(out[7])
                 : "memory");
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
  int shift = -1;
  if ((a.group_values & (a.group_values - 1)) == 0) {
    shift = 0;
    while ((1 << shift) < a.group_values) ++shift;
  }
  // The pairs kernel: whole runs of 16 values per row and per group, 32-byte aligned output rows, and packed rows that
  // a run's words can be read from at once.
  const int run_bytes = w->bits == 3 ? 4 : 2 * w->bits;
  const bool pairs = out_dtype != DQ_F32 && a.meta_dtype != DQ_F32 && a.in_features % 16 == 0 && a.in_features > 16 && a.group_values % 16 == 0 &&
                     reinterpret_cast<uintptr_t>(out) % 32 == 0 && reinterpret_cast<uintptr_t>(a.packed) % run_bytes == 0 && a.words_per_row * 4 % run_bytes == 0;
  const int64_t num_runs = static_cast<int64_t>(a.rows) * (a.in_features / 16);
  if (pairs && num_runs < (int64_t{1} << 31)) {
    const unsigned per_row = static_cast<unsigned>(a.in_features / 16);
    const unsigned long long magic = ~0ull / per_row + 1;  // ceil(2^64 / per_row)
    const unsigned total = static_cast<unsigned>(num_runs);
    // Two runs per thread from a full wave of such threads on (4096 x 4096, 3-bit: 8.2 us, 9.0 with one, 9.6 with four;
    // 2048 x 2048 is level, 512 x 1024 takes 1.83 us with one, 1.95 with two).
    const bool two = num_runs >= static_cast<int64_t>(dev->sm_count) * 2048 * 2;
    const unsigned grid = static_cast<unsigned>(ceil_div(num_runs, kDequantThreads * (two ? 2 : 1)));
    const auto run = [&](auto bits, auto bf16, auto ids) {
      constexpr int B = decltype(bits)::value;
      constexpr bool M = decltype(bf16)::value, IDS = decltype(ids)::value;
      (two ? dequant_pairs_kernel<B, M, 2, IDS> : dequant_pairs_kernel<B, M, 1, IDS>)<<<grid, kDequantThreads, 0, s>>>(a, per_row, magic, total, shift);
    };
    const auto with_bits = [&](auto bf16, auto ids) {
      switch (w->bits) {
        case 2: run(std::integral_constant<int, 2>{}, bf16, ids); break;
        case 3: run(std::integral_constant<int, 3>{}, bf16, ids); break;
        case 4: run(std::integral_constant<int, 4>{}, bf16, ids); break;
        default: run(std::integral_constant<int, 8>{}, bf16, ids); break;
      }
    };
    const auto with_meta = [&](auto ids) { a.meta_dtype == DQ_BF16 ? with_bits(std::true_type{}, ids) : with_bits(std::false_type{}, ids); };
    a.ids != nullptr ? with_meta(std::true_type{}) : with_meta(std::false_type{});
    DQ_CHECK_LAUNCH("dequant");
    return DQ_OK;
  }
  const int64_t num_octets = static_cast<int64_t>(a.rows) * (a.in_features / 8);
  if (octets && a.in_features > 8 && num_octets < (int64_t{1} << 32)) {
    const unsigned per_row = static_cast<unsigned>(a.in_features / 8);
    const unsigned long long magic = ~0ull / per_row + 1;  // ceil(2^64 / per_row)
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
