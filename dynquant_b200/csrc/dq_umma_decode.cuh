// Packed codes -> 16-bit weights, one weight row per thread, natural order: the A operand of
// tcgen05.mma as tensor memory holds it (lane = weight row, a 32-bit column = two values of K).
//
// ONE AND-OR puts two codes (one per 16-bit half) into the mantissa of a power of two of the
// METADATA's type -- with the code's lowest bit at mantissa bit p and the exponent chosen so that
// this bit is worth 1, a half is exactly M_p + q -- and ONE mixed-precision fma per value,
//   w = (M_p + q) * s + (o - M_p * s),   16-bit factors, fp32 addend and result,
// unbiases, scales and shifts it; the scale enters in its own type, and the addend's rounding is up to
// M_p * 2^-25 of a scale step: 2^-15 of it at most (M_p <= 1024) -- but 2^-10 for 8-bit codes with bf16
// metadata, whose addend is o - 32768 * s.  One conversion per pair rounds to the operand type; split in two,
// a weight keeps 16 bits (bf16) or 21 and more (fp16).  None of it shows behind the rounding of a 16-bit
// output: 24 rows x 1024 x 4096 at every width, metadata type and operand type, error against 64 bits in the
// norm within 1e-4 of itself of the mma.sync kernels' (1.65e-3 bf16, 2.07e-4 fp16).  Taking M_p off the codes
// first (one packed subtraction per pair, exact) changed no figure of that table and cost 1 to 6 %.
// That is about 1.1 (2, 4, 8 bits) to 1.5 (3 bits) ALU instructions per value -- logic, shifts and
// conversions issue at half rate and bound the loop -- plus one fma at full rate; building fp32
// values code by code (an AND-OR and half a conversion each) took 2 and ran 128 x 64 values in 680
// cycles per SM.  8-bit codes do not fit a bf16 mantissa: with bf16 metadata they take that way.
#pragma once

#include "dq_umma.cuh"

namespace dq {
namespace umma {

#ifdef __CUDACC__

// Bytes of a row of a 128-value tile are 16 * BITS: the TMA swizzle mode (log2 of the 16-byte pieces).
template <int BITS>
constexpr int kSwizzleBits = BITS == 2 ? 1 : BITS == 4 ? 2 : BITS == 8 ? 3 : 0;

// Scale and addends of one group.
template <int BITS, bool MBF16>
struct Affine {
  // code positions in the mantissa (bits): at 2 bits 0 2 4 (6), at 3 bits 0 3 (6), at 4 bits 0 (4)
  static constexpr int kWide = BITS == 8 && MBF16;  // fp32 codes
  static constexpr int kPlaces = BITS == 2 ? (MBF16 ? 3 : 4) : BITS == 3 ? (MBF16 ? 2 : 3) : BITS == 4 ? (MBF16 ? 1 : 2) : 1;
  static constexpr int kMantissa = MBF16 ? 7 : 10;
  unsigned short scale;
  float wide_mul, add[kPlaces];
  __device__ __forceinline__ void set(unsigned short s16, float o) {
    scale = s16;
    const float s = MBF16 ? __uint_as_float(static_cast<uint32_t>(s16) << 16) : __half2float(__ushort_as_half(s16));
    if constexpr (kWide) {
      wide_mul = s * 32768.0f;
      add[0] = fmaf(-s, 32768.0f, o);
    } else {
#pragma unroll
      for (int i = 0; i < kPlaces; ++i) add[i] = fmaf(-s, static_cast<float>(1 << (kMantissa - i * BITS)), o);
    }
  }
  // The magic number of place i in both halves: M = 2^(kMantissa - i * BITS).
  static constexpr uint32_t magic(int i) {
    const uint32_t half = MBF16 ? static_cast<uint32_t>(127 + kMantissa - i * BITS) << 7 : static_cast<uint32_t>(15 + kMantissa - i * BITS) << 10;
    return half | (half << 16);
  }
  static constexpr uint32_t mask(int i) {
    const uint32_t half = ((1u << BITS) - 1u) << (i * BITS);
    return half | (half << 16);
  }
};

template <bool BF16>
__device__ __forceinline__ uint32_t pack16(float lo, float hi) {
  if constexpr (BF16) {
    const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&b);
  } else {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
}

// (16-bit half of `pair`) * scale + add, in fp32.
template <bool MBF16>
__device__ __forceinline__ float fma_half(uint32_t pair, bool high, unsigned short scale, float add) {
  float d;
  if constexpr (MBF16) {
    if (high) {
      asm("{\n .reg .b16 l, h;\n mov.b32 {l, h}, %1;\n fma.rn.f32.bf16 %0, h, %2, %3;\n}" : "=f"(d) : "r"(pair), "h"(scale), "f"(add));
    } else {
      asm("{\n .reg .b16 l, h;\n mov.b32 {l, h}, %1;\n fma.rn.f32.bf16 %0, l, %2, %3;\n}" : "=f"(d) : "r"(pair), "h"(scale), "f"(add));
    }
  } else {
    if (high) {
      asm("{\n .reg .b16 l, h;\n mov.b32 {l, h}, %1;\n fma.rn.f32.f16 %0, h, %2, %3;\n}" : "=f"(d) : "r"(pair), "h"(scale), "f"(add));
    } else {
      asm("{\n .reg .b16 l, h;\n mov.b32 {l, h}, %1;\n fma.rn.f32.f16 %0, l, %2, %3;\n}" : "=f"(d) : "r"(pair), "h"(scale), "f"(add));
    }
  }
  return d;
}

// 32 values (BITS words) -> 16 registers of two; `low` (if not null): what the rounding of each value
// to 16 bits left over, rounded the same way, so that out + low carries the value to 16 bits (bf16) or
// 21 (fp16) -- the remainder is one exact mixed-precision fma per value.
template <int BITS, bool BF16, bool MBF16, bool SPLIT>
__device__ __forceinline__ void decode32(const uint32_t* w, const Affine<BITS, MBF16>& c, uint32_t* out, uint32_t* low) {
  using A = Affine<BITS, MBF16>;
  float f[32];
  // codes `lo` (low half of u) and `hi` (high half), at mantissa place i
  auto take = [&](uint32_t u, int i, int lo, int hi) {
    const uint32_t q = (u & A::mask(i)) | A::magic(i);
    f[lo] = fma_half<MBF16>(q, false, c.scale, c.add[i]);
    f[hi] = fma_half<MBF16>(q, true, c.scale, c.add[i]);
  };
  if constexpr (A::kWide) {
    // 1 + q * 2^-15 in fp32: byte q under the upper half of 1.0f
#pragma unroll
    for (int v = 0; v < 32; ++v) {
      f[v] = fmaf(__uint_as_float(__byte_perm(w[v / 4], 0x3F800000u, 0x7604u | ((v & 3) << 4))), c.wide_mul, c.add[0]);
    }
  } else if constexpr (BITS == 8) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {  // two bytes of w under the upper bytes of two 1024.0
      const uint32_t q = __byte_perm(w[i / 2], A::magic(0), (i & 1) ? 0x7352u : 0x7150u);
      f[2 * i] = fma_half<MBF16>(q, false, c.scale, c.add[0]);
      f[2 * i + 1] = fma_half<MBF16>(q, true, c.scale, c.add[0]);
    }
  } else if constexpr (BITS == 4) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int v = 8 * i;
      if constexpr (A::kPlaces == 2) {
        take(w[i], 0, v, v + 4), take(w[i], 1, v + 1, v + 5);
        take(w[i] >> 8, 0, v + 2, v + 6), take(w[i] >> 8, 1, v + 3, v + 7);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) take(w[i] >> (4 * j), 0, v + j, v + j + 4);
      }
    }
  } else if constexpr (BITS == 2) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
#pragma unroll
      for (int j = 0; j < 8; ++j) take(w[i] >> (2 * (j - j % A::kPlaces)), j % A::kPlaces, 16 * i + j, 16 * i + j + 8);
    }
  } else {
    // bits 16 t .. 16 t + 15 of the 96 below bits 48 + 16 t ..: code i in the low halves, i + 16 in the high ones
    const uint32_t h[3] = {__byte_perm(w[0], w[1], 0x7610u), __byte_perm(w[0], w[2], 0x5432u), __byte_perm(w[1], w[2], 0x7610u)};
    constexpr int P = A::kPlaces;
#pragma unroll
    for (int j = 0; j < 5; ++j) take(h[0] >> (3 * (j - j % P)), j % P, j, j + 16);               // codes 0..4 at bits 0..14
#pragma unroll
    for (int j = 0; j < 4; ++j) take(h[1] >> (2 + 3 * (j - j % P)), j % P, j + 6, j + 22);       // 6..9 at bits 2..13
#pragma unroll
    for (int j = 0; j < 5; ++j) take(h[2] >> (1 + 3 * (j - j % P)), j % P, j + 11, j + 27);      // 11..15 at bits 1..15
    // the two codes that straddle halves
    const uint32_t five = ((h[0] >> 15) & 0x00010001u) | ((h[1] << 1) & 0x00060006u);
    const uint32_t ten = ((h[1] >> 14) & 0x00030003u) | ((h[2] << 2) & 0x00040004u);
    take(five, 0, 5, 21);
    take(ten, 0, 10, 26);
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    out[i] = pack16<BF16>(f[2 * i], f[2 * i + 1]);
    if constexpr (SPLIT) {
      constexpr unsigned short kMinusOne = BF16 ? 0xBF80 : 0xBC00;
      low[i] = pack16<BF16>(fma_half<BF16>(out[i], false, kMinusOne, f[2 * i]), fma_half<BF16>(out[i], true, kMinusOne, f[2 * i + 1]));
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
    constexpr int kMask = (1 << kSwizzleBits<BITS>) - 1;  // 16-byte pieces are XORed with address bits 7..
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
