// Packed codes -> 16-bit weights, one weight row per thread, natural order: the A operand of
// tcgen05.mma as tensor memory holds it (lane = weight row, a 32-bit column = two values of K).
//
// A code is moved into the upper mantissa bits of 1.0f: f = 1 + q * 2^(p - 23) with its lowest bit
// at bit p, by one shift shared by the codes of a window and one AND-OR per code.  Then
//   w = f * (s * 2^(23 - p)) + (o - s * 2^(23 - p))
// is ONE fp32 fma per value (two per packed instruction), with no conversion and no unbiasing:
// the constant's own rounding is 2^(-1-p) of a scale step (p >= 14 at 2, 3 and 4 bits; p = 8 at 8
// bits, where a step is 1/128 of the range).  One rounding to the operand type follows.  About 4
// issue cycles per value, against 2 for the accumulator-side scaling of the mma.sync kernels --
// but here a decoded value is multiplied with up to 256 activation rows at once.
#pragma once

#include "dq_umma.cuh"

namespace dq {
namespace umma {

#ifdef __CUDACC__

template <int BITS>
struct DecodeCfg;
template <>
struct DecodeCfg<2> {
  static constexpr int kPairs = 2, kSwizzle = 1;
};
template <>
struct DecodeCfg<3> {
  static constexpr int kPairs = 3, kSwizzle = 0;
};
template <>
struct DecodeCfg<4> {
  static constexpr int kPairs = 1, kSwizzle = 2;
};
template <>
struct DecodeCfg<8> {
  static constexpr int kPairs = 1, kSwizzle = 3;
};

// Multiplier and addend of the two values of a register, per position pair.
template <int BITS>
struct Affine {
  float2 mul[DecodeCfg<BITS>::kPairs], add[DecodeCfg<BITS>::kPairs];
  __device__ __forceinline__ void set(float s, float o) {
    auto put = [&](int i, float lo, float hi) {
      mul[i] = make_float2(s * lo, s * hi);
      add[i] = make_float2(fmaf(-s, lo, o), fmaf(-s, hi, o));
    };
    if constexpr (BITS == 2) put(0, 256.0f, 64.0f), put(1, 16.0f, 4.0f);
    if constexpr (BITS == 3) put(0, 512.0f, 64.0f), put(1, 8.0f, 512.0f), put(2, 64.0f, 8.0f);
    if constexpr (BITS == 4) put(0, 256.0f, 16.0f);
    if constexpr (BITS == 8) put(0, 32768.0f, 32768.0f);
  }
};

template <bool BF16>
__device__ __forceinline__ uint32_t pack16(float2 v) {
  if constexpr (BF16) {
    const __nv_bfloat162 b = __floats2bfloat162_rn(v.x, v.y);
    return *reinterpret_cast<const uint32_t*>(&b);
  } else {
    const __half2 h = __floats2half2_rn(v.x, v.y);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
}

// 32 values (BITS words) -> 16 registers of two.
template <int BITS, bool BF16>
__device__ __forceinline__ void decode32(const uint32_t* w, const Affine<BITS>& c, uint32_t* out) {
  constexpr uint32_t kOne = 0x3F800000u;
  auto field = [&](uint32_t u, int p) -> float { return __uint_as_float((u & (((1u << BITS) - 1u) << p)) | kOne); };
  auto emit = [&](int n, float lo, float hi, int pair) {
    out[n] = pack16<BF16>(__ffma2_rn(make_float2(lo, hi), c.mul[pair], c.add[pair]));
  };
  if constexpr (BITS == 2 || BITS == 4) {
    constexpr int kPerWord = 32 / BITS;
#pragma unroll
    for (int i = 0; i < BITS; ++i) {
      const uint32_t u[4] = {w[i] << 15, w[i] << 7, w[i] >> 1, w[i] >> 9};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int n = (i * kPerWord + j * (8 / BITS)) / 2;
        if constexpr (BITS == 4) {
          emit(n, field(u[j], 15), field(u[j], 19), 0);
        } else {
          emit(n, field(u[j], 15), field(u[j], 17), 0);
          emit(n + 1, field(u[j], 19), field(u[j], 21), 1);
        }
      }
    }
  } else if constexpr (BITS == 3) {
    const uint32_t u[11] = {w[0] << 14, w[0] << 5, w[0] >> 4, __funnelshift_r(w[0], w[1], 13), w[1] << 10, w[1] << 1,
                            w[1] >> 8, __funnelshift_r(w[1], w[2], 17), w[2] << 6, w[2] >> 3, w[2] >> 12};
#pragma unroll
    for (int n = 0; n < 16; ++n) {
      const int a = 2 * n, b = 2 * n + 1;
      emit(n, field(u[a / 3], 14 + 3 * (a % 3)), field(u[b / 3], 14 + 3 * (b % 3)), n % 3);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float lo = __uint_as_float(__byte_perm(w[i], kOne, 0x7604u | ((2 * j) << 4)));
        const float hi = __uint_as_float(__byte_perm(w[i], kOne, 0x7604u | ((2 * j + 1) << 4)));
        emit(2 * i + j, lo, hi, 0);
      }
    }
  }
}

// The 64 values (2 * BITS words) of half `half` of row `row` in a staged 128 x 128-value tile.
template <int BITS>
__device__ __forceinline__ void read_row64(const unsigned char* tile, int row, int half, uint32_t* w) {
  constexpr int ROW = 16 * BITS;
  if constexpr (BITS == 3) {  // 24 bytes, not swizzled: rows 48 bytes apart spread over the banks by themselves
    const unsigned char* p = tile + row * ROW;
    if (half == 0) {
      const uint4 a = *reinterpret_cast<const uint4*>(p);
      const uint2 b = *reinterpret_cast<const uint2*>(p + 16);
      w[0] = a.x, w[1] = a.y, w[2] = a.z, w[3] = a.w, w[4] = b.x, w[5] = b.y;
    } else {
      const uint2 a = *reinterpret_cast<const uint2*>(p + 24);
      const uint4 b = *reinterpret_cast<const uint4*>(p + 32);
      w[0] = a.x, w[1] = a.y, w[2] = b.x, w[3] = b.y, w[4] = b.z, w[5] = b.w;
    }
  } else {
    constexpr int kMask = (1 << DecodeCfg<BITS>::kSwizzle) - 1;  // 16-byte pieces are XORed with address bits 7..
#pragma unroll
    for (int i = 0; i < BITS / 2; ++i) {
      int at = row * ROW + half * (8 * BITS) + i * 16;
      at ^= ((at >> 7) & kMask) << 4;
      const uint4 v = *reinterpret_cast<const uint4*>(tile + at);
      w[4 * i] = v.x, w[4 * i + 1] = v.y, w[4 * i + 2] = v.z, w[4 * i + 3] = v.w;
    }
  }
}

#endif  // __CUDACC__

}  // namespace umma
}  // namespace dq
