// The pipeline that the tcgen05 kernels share: who does what in a block, the barriers between the
// roles, the decoding warpgroups.
//
// Warp 0 brings activations (TMA), warp 2 packed weights (TMA), warp 1 issues the MMAs, warp 3 owns the
// tensor memory, the warps from 4 on decode in warpgroups of four.  A weight tile is 128 rows x 128
// values; a thread of a warpgroup owns one of its rows (the tensor memory lane that it may write).
#pragma once

#include "dq_umma_decode.cuh"

namespace dq {
namespace umma {

#ifdef __CUDACC__

constexpr int kDecodeWarp0 = 4;        // warps 0..3: TMA x, MMA, TMA weights, tensor memory
// Decoding warpgroups and the operand tiles of 128 x 128 weights in tensor memory, one per warpgroup:
// stage (chunk of 128 values of K) i belongs to warpgroup i % kGroups and always to its tile, so that
// nobody can ever be two passes ahead of a tile's barrier.  Four groups and tiles of 64 columns, or
// (every weight as two 16-bit pieces) three groups and tiles of 128.
template <bool SPLIT>
struct Roles {
  static constexpr int kGroups = SPLIT ? 3 : 4, kTileColumns = SPLIT ? 128 : 64, kColumns = kGroups * kTileColumns;
  static constexpr int kThreads = (kDecodeWarp0 + 4 * kGroups) * 32;
};
constexpr int kMaxGroups = 4;
constexpr int kMaxRing = 16;
// fp16 operands hold nothing below 2^-25 and nothing above 65504, and two of them (split weights) no more
// than that: a weight of 1e-4 would be held to 3e-4 of itself.  The mma.sync kernels scale fp32 sums by
// group instead and have no such limits.  So each weight row of a tile is brought to 2^14..2^15 by a power
// of two of its own, which its fp32 sums lose again (row_power): nothing of a row is then held to less than
// 2^-39 of the row's largest weight.  bf16 has the range of fp32 and needs none of it.  The look at a tile's
// metadata ahead of its decode costs 0.9 to 1.8 us a launch (4097 x 4096, 3-bit, 24 rows: 12.6 -> 14.3 us; 4096
// x 14336, 64 rows: 24.8 -> 25.8) and the expert layer of 1000 tokens a fifth (278 -> 342 us).  Rows shared by
// the lanes of a warp, with shuffles, took 2 us more: it is bound by its instructions, and a thread per row
// has the fewest.
template <bool BF16, bool SPLIT>
constexpr bool kScaledRows = SPLIT && !BF16;
constexpr int kPowerSlots = 4;

struct Bars {
  uint32_t x_full, x_empty, w_full, w_empty, a_full, a_empty, d_full, d_empty, drain, p_full, p_empty;
};

// Where a role stands in a ring: a slot and the parity of its pass (run-time divisions would cost the
// single-thread roles more than their work: 0.3 us per stage, measured).
struct Cursor {
  uint32_t slot = 0, pass = 0;
  __device__ __forceinline__ void advance(uint32_t slots, uint32_t by = 1) {
    slot += by;
    if (slot >= slots) slot -= slots, pass ^= 1;  // (by <= slots)
  }
};

// The metadata of a packed matrix, and the weight ring that its tiles pass through.
struct Meta {
  const void* scales;
  const void* offsets;                 // may be null
  int num_groups, group_shift;         // group = 64 << group_shift
};
struct WeightRing {
  const unsigned char* tiles;
  int slots, bytes;
};

template <bool MBF16>
__device__ __forceinline__ float widen16(uint32_t v) {
  return MBF16 ? __uint_as_float(v << 16) : __half2float(__ushort_as_half(static_cast<unsigned short>(v)));
}
// 2^k, for a k of row_power or its negative.
__device__ __forceinline__ float power_of_two(int k) { return __uint_as_float(static_cast<uint32_t>(127 + k) << 23); }
template <bool MBF16>
__device__ __forceinline__ unsigned short scaled16(unsigned short s, float power) {  // (exact but for what goes below 2^-24)
  const float v = widen16<MBF16>(s) * power;
  return MBF16 ? static_cast<unsigned short>(__float_as_uint(v) >> 16) : __half_as_ushort(__float2half_rn(v));
}
// A row's power k: its weights in groups [g0, g0 + count) of that row, all below max|s| * (2^bits - 1) +
// max|o|, times 2^k stay below 2^15.  A thread takes a row, in 16-byte pieces that start on a 16-byte
// boundary (what they hold of the row's other groups may count; what belongs to its neighbours is masked),
// up to four of each array in flight; where a piece would reach past the arrays of `rows` rows, value by value.
template <bool MBF16>
__device__ __forceinline__ int row_power(const Meta& meta, int bits, int64_t rows, int64_t row, int g0, int count) {
  struct Pieces {
    uintptr_t row0, row1, at;  // bytes: the row's, and the next piece's
    int last;                  // pieces - 1
    bool inside;               // all of them in the array
  };
  const auto pieces = [&](const void* p) -> Pieces {
    const uintptr_t row0 = reinterpret_cast<uintptr_t>(p) + static_cast<uintptr_t>(row * meta.num_groups) * 2, from = row0 + static_cast<uintptr_t>(g0) * 2;
    const uintptr_t at = from & ~uintptr_t{15}, base = reinterpret_cast<uintptr_t>(p);
    const int last = static_cast<int>((from + static_cast<uintptr_t>(count) * 2 - 1 - at) >> 4);
    return {row0, row0 + static_cast<uintptr_t>(meta.num_groups) * 2, at, last,
            at >= base && at + (static_cast<uintptr_t>(last) + 1) * 16 <= base + static_cast<uintptr_t>(rows * meta.num_groups) * 2};
  };
  const auto fold = [](uint32_t most, uint4 v, const Pieces& p, int i) -> uint32_t {  // |.| as its bits: ordered like the values
    uint32_t w[4] = {v.x, v.y, v.z, v.w};
    const uintptr_t at = p.at + static_cast<uintptr_t>(i) * 16;
    if (at < p.row0 || at + 16 > p.row1) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uintptr_t low = at + j * 4, high = low + 2;
        w[j] &= (low >= p.row0 && low < p.row1 ? 0x0000FFFFu : 0u) | (high >= p.row0 && high < p.row1 ? 0xFFFF0000u : 0u);
      }
    }
    const uint32_t m = __vmaxu2(__vmaxu2(w[0] & 0x7FFF7FFFu, w[1] & 0x7FFF7FFFu), __vmaxu2(w[2] & 0x7FFF7FFFu, w[3] & 0x7FFF7FFFu));
    return __vmaxu2(most, m);
  };
  const auto load = [](const Pieces& p, int i) -> uint4 { return __ldg(reinterpret_cast<const uint4*>(p.at) + i); };
  constexpr int kBatch = 4;
  const bool has_offsets = meta.offsets != nullptr;
  const Pieces s = pieces(meta.scales), o = has_offsets ? pieces(meta.offsets) : s;
  uint32_t s_most = 0, o_most = 0;
  const bool inside = s.inside && o.inside;
  for (int g = 0; g < count && !inside; ++g) {
    const int64_t at = row * meta.num_groups + g0 + g;
    s_most = max(s_most, __ldg(static_cast<const unsigned short*>(meta.scales) + at) & 0x7FFFu);
    if (has_offsets) o_most = max(o_most, __ldg(static_cast<const unsigned short*>(meta.offsets) + at) & 0x7FFFu);
  }
  for (int i0 = 0; inside && (i0 <= s.last || i0 <= o.last); i0 += kBatch) {
    uint4 sv[kBatch], ov[kBatch];
#pragma unroll
    for (int i = 0; i < kBatch; ++i) sv[i] = load(s, min(i0 + i, s.last)), ov[i] = load(o, min(i0 + i, o.last));
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      s_most = fold(s_most, sv[i], s, min(i0 + i, s.last));
      if (has_offsets) o_most = fold(o_most, ov[i], o, min(i0 + i, o.last));
    }
  }
  s_most = max(s_most & 0xFFFFu, s_most >> 16), o_most = max(o_most & 0xFFFFu, o_most >> 16);
  const float bound = fmaf(widen16<MBF16>(s_most), static_cast<float>((1 << bits) - 1), widen16<MBF16>(o_most));
  const int e = static_cast<int>(__float_as_uint(bound) >> 23);  // (255: past fp32 itself, by less than 2^9)
  return e == 255 ? -123 : min(141 - e, 100);
}

// Warpgroup `group`'s chunks of a tile of 128 weight rows, `row` the one of this thread and `tile_row` its
// place in the staged tile: chunk c0 + i is stage stage0 + i, numbered over the life of the block.  `power`
// (kScaledRows): what the row is multiplied by.  False once a wait has run out.
template <int BITS, bool BF16, bool MBF16, bool SPLIT>
__device__ bool decode_tile(const Meta& meta, int64_t row, int tile_row, float power, int c0, int group, uint32_t stage0, int stages, const WeightRing& ring,
                            const Bars& bars, uint32_t tmem, Cursor& w_at, uint32_t& a_pass, volatile int* failed) {
  constexpr int kGroups = Roles<SPLIT>::kGroups;
  const int lane = threadIdx.x & 31;
  const int warp4 = (threadIdx.x >> 5) & 3;
  const unsigned short* s_row = static_cast<const unsigned short*>(meta.scales) + row * meta.num_groups;
  const unsigned short* o_row =
      meta.offsets == nullptr ? nullptr : static_cast<const unsigned short*>(meta.offsets) + row * meta.num_groups;
  auto set = [&](Affine<BITS, MBF16>& affine, unsigned short s, unsigned short o) {
    const float offset = o_row != nullptr ? widen16<MBF16>(o) : 0.0f;
    if constexpr (kScaledRows<BF16, SPLIT>) {
      affine.set(scaled16<MBF16>(s, power), offset * power);
    } else {
      affine.set(s, offset);
    }
  };
  const bool two_groups = meta.group_shift == 0;  // 64-value groups: a chunk holds two
  auto group_of = [&](int i, int half) -> int { return min((2 * (c0 + i) + half) >> meta.group_shift, meta.num_groups - 1); };
  unsigned short s_next[2], o_next[2] = {0, 0};
  auto fetch = [&](int i) {
    const int g0 = group_of(i, 0);
    s_next[0] = __ldg(s_row + g0);
    if (o_row != nullptr) o_next[0] = __ldg(o_row + g0);
    if (two_groups) {
      const int g1 = group_of(i, 1);
      s_next[1] = __ldg(s_row + g1);
      if (o_row != nullptr) o_next[1] = __ldg(o_row + g1);
    }
  };
  const int first = (group + kGroups - static_cast<int>(stage0 % kGroups)) % kGroups;
  if (first >= stages) return true;
  fetch(first);
  for (int i = first; i < stages; i += kGroups) {
    Affine<BITS, MBF16> affine;
    set(affine, s_next[0], o_next[0]);
    const unsigned short s_half = s_next[1], o_half = o_next[1];
    fetch(min(i + kGroups, stages - 1));  // the next chunk's metadata travels while this one is decoded
    const uint32_t slot = w_at.slot;
    if (!mbar_wait(bars.w_full + slot * 8, w_at.pass, failed)) return false;
    const uint32_t dst = tmem + group * Roles<SPLIT>::kTileColumns + (static_cast<uint32_t>(warp4 * 32) << 16);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      uint32_t w[2 * BITS], v[16], low[16];
      read_row64<BITS>(ring.tiles + slot * ring.bytes, tile_row, half, w);
      if (half == 1 && two_groups) set(affine, s_half, o_half);
      decode32<BITS, BF16, MBF16, SPLIT>(w, affine, v, low);
      if (half == 0) {  // the MMAs of this group's previous chunk are done with the tile
        if (!mbar_wait(bars.a_empty + group * 8, a_pass ^ 1, failed)) return false;
        fence_after_sync();
      }
      tmem_st16(dst + half * 32, v);
      if constexpr (SPLIT) tmem_st16(dst + 64 + half * 32, low);
      decode32<BITS, BF16, MBF16, SPLIT>(w + BITS, affine, v, low);
      tmem_st16(dst + half * 32 + 16, v);
      if constexpr (SPLIT) tmem_st16(dst + 64 + half * 32 + 16, low);
    }
    tmem_wait_st();
    fence_before_sync();
    __syncwarp();
    if (lane == 0) {
      mbar_arrive(bars.a_full + group * 8);
      // Only now: an arrival may overtake shared-memory loads still in flight, and the slot is refilled
      // at once.  By here every word has gone through the decode.
      mbar_arrive(bars.w_empty + slot * 8);
    }
    w_at.advance(static_cast<uint32_t>(ring.slots), kGroups);
    a_pass ^= 1;
  }
  return true;
}

// Barriers from `at` on (shared memory).
constexpr uint32_t kBarrierBytes = (4 * kMaxRing + 2 * kMaxGroups + 5 + 2 * kPowerSlots) * 8;
__device__ __forceinline__ Bars bars_at(uint32_t at) {
  Bars b;
  b.x_full = at;
  b.x_empty = b.x_full + kMaxRing * 8;
  b.w_full = b.x_empty + kMaxRing * 8;
  b.w_empty = b.w_full + kMaxRing * 8;
  b.a_full = b.w_empty + kMaxRing * 8;
  b.a_empty = b.a_full + kMaxGroups * 8;
  b.d_full = b.a_empty + kMaxGroups * 8;
  b.d_empty = b.d_full + 2 * 8;
  b.drain = b.d_empty + 2 * 8;
  b.p_full = b.drain + 8;
  b.p_empty = b.p_full + kPowerSlots * 8;
  return b;
}
// power_writers, power_readers: warps that write and that read a slot of row powers; 0: there are none
__device__ __forceinline__ void init_bars(const Bars& b, int x_slots, int w_slots, int groups, int epilogue_warps, int power_writers = 0,
                                          int power_readers = 0) {
  for (int i = 0; i < x_slots; ++i) mbar_init(b.x_full + i * 8, 1), mbar_init(b.x_empty + i * 8, 1);
  for (int i = 0; i < w_slots; ++i) mbar_init(b.w_full + i * 8, 1), mbar_init(b.w_empty + i * 8, 4);
  for (int i = 0; i < groups; ++i) mbar_init(b.a_full + i * 8, 4), mbar_init(b.a_empty + i * 8, 1);
  for (int i = 0; i < 2; ++i) mbar_init(b.d_full + i * 8, 1), mbar_init(b.d_empty + i * 8, static_cast<uint32_t>(epilogue_warps));
  for (int i = 0; i < kPowerSlots && power_readers > 0; ++i) {
    mbar_init(b.p_full + i * 8, static_cast<uint32_t>(power_writers)), mbar_init(b.p_empty + i * 8, static_cast<uint32_t>(power_readers));
  }
  mbar_init(b.drain, 1);
  fence_mbar_init();
}

// The MMAs of 64 values of K, four steps of 16: a piece of the operand tile at `a`, a slab of activations
// at `b`.
template <bool SPLIT>
__device__ __forceinline__ void mma_slab(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, bool accumulate) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    mma_ts(d, a + k * 8, b + k * 2, idesc, accumulate || k > 0);
    if constexpr (SPLIT) mma_ts(d, a + 64 + k * 8, b + k * 2, idesc, true);
  }
}
// One chunk's: an operand tile, two slabs.
template <bool SPLIT>
__device__ __forceinline__ void mma_chunk(uint32_t d, uint32_t a, uint64_t b0, uint64_t b1, uint32_t idesc, bool accumulate) {
  mma_slab<SPLIT>(d, a, b0, idesc, accumulate);
  mma_slab<SPLIT>(d, a + 32, b1, idesc, true);
}

// What the roles of a block leave in flight when they stop; only a block that gives up looks at it.
struct InFlight {
  uint32_t issued[3];  // copies, by the warp that issues them (0 and 2)
  int mma_lane;        // of warp 1: the thread whose MMAs a commit waits for
};
// Called by all threads once every role has stopped -- a producer may have issued its last copy long before
// another role's wait runs out, so a role cannot do it for itself: waits (bounded) until the copies and the
// MMAs are through with the memory that is about to change hands.
__device__ __forceinline__ void drain(const InFlight& left, const Bars& bars, int x_slots, int w_slots) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 1 && lane == left.mma_lane) {
    mma_commit(bars.drain);
    for (int i = 0; i < kSpins && !mbar_try(bars.drain, 0); ++i) {
    }
  }
  if ((warp == 0 || warp == 2) && lane == 0) {
    const uint32_t issued = left.issued[warp], slots = static_cast<uint32_t>(warp == 2 ? w_slots : x_slots);
    for (uint32_t k = issued > slots ? issued - slots : 0; k < issued; ++k) {
      for (int i = 0; i < kSpins && !mbar_try((warp == 2 ? bars.w_full : bars.x_full) + (k % slots) * 8, (k / slots) & 1); ++i) {
      }
    }
  }
}

#endif  // __CUDACC__

// ---- host -------------------------------------------------------------------
inline bool encode_map(CUtensorMap* map, CUtensorMapDataType type, const void* base, int64_t inner, int64_t outer, int64_t row_bytes,
                int box_inner, int box_outer, CUtensorMapSwizzle swizzle) {
  static const auto encode = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess) {
      fn = nullptr;
    }
    return reinterpret_cast<decltype(&cuTensorMapEncodeTiled)>(fn);
  }();
  if (encode == nullptr) return false;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(inner), static_cast<cuuint64_t>(outer)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(row_bytes)};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(box_inner), static_cast<cuuint32_t>(box_outer)};
  const cuuint32_t step[2] = {1, 1};
  return encode(map, type, 2, const_cast<void*>(base), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

inline CUtensorMapSwizzle weight_swizzle(int bits) {
  return bits == 2 ? CU_TENSOR_MAP_SWIZZLE_32B : bits == 3 ? CU_TENSOR_MAP_SWIZZLE_NONE : bits == 4 ? CU_TENSOR_MAP_SWIZZLE_64B
                                                                                                     : CU_TENSOR_MAP_SWIZZLE_128B;
}

// 64 << shift values per group, or -1.
inline int group_shift_of(int group_values) {
  for (int s = 0; s < 16; ++s) {
    if (group_values == (64 << s)) return s;
  }
  return -1;
}

}  // namespace umma
}  // namespace dq
