// Packed matrix x many activation rows on the fifth-generation tensor cores:
//   out[m, n] = sum_k x[m, k] * (q[n, k] * s[n, g] + o[n, g]) (+ bias[n])
// for prefill and large batches, in ONE pass -- the reference (and this library before) writes the
// dense matrix out and reads it back for a library GEMM (runtime/ops.py:205-231).
//
// A CTA computes 128 weight rows x n_tile activation rows (16..256) with the weights as the A
// operand of tcgen05.mma:
//   * warp 2 streams packed 128 x 128-value tiles into shared memory by TMA (they are 4..16 KB, so
//     a ring of them keeps HBM busy), warp 0 the activation in 64-value slabs with the 128-byte
//     swizzle, both zero-filled past the edges of their tensors;
//   * four warpgroups (warps 4..19) decode, 64 values of K in turn: a thread owns one weight row, so
//     its scale and offset are two registers and its packed words one contiguous piece of shared
//     memory; the 16-bit weights go straight to TENSOR MEMORY (tcgen05.st) in the
//     natural order -- not to shared memory, whose bandwidth the activation needs;
//   * warp 1 issues the MMAs (A from tensor memory, B from shared memory), accumulating in tensor
//     memory; two accumulator tiles where they fit (n_tile <= 192), so that the decode of the next
//     tile runs under the epilogue of this one.
// What bounds it: with n_tile >= 144 the tensor pipe (128 x n_tile x 64 take 2 n_tile cycles), below
// that the decode (about 290 cycles per 128 x 64 values on the SM's four schedulers).
//
// Small matrices: the reduction axis is sliced over a thread-block cluster (grid.y), each CTA leaves
// its fp32 tile in its own shared memory and the CTAs of the cluster add a share of the columns
// each, in slice order, over distributed shared memory -- deterministic.
//
// Every wait is bounded (dq_umma.cuh): when one runs out the block stops issuing, drains its own
// copies, frees its tensor memory, leaves its output unwritten and raises the device's error word
// (dq_gemm_status).
#include <algorithm>
#include <cmath>

#include "dq_gemm_umma.cuh"
#include "dq_gemv.cuh"
#include "dq_umma_decode.cuh"

namespace dq {
namespace {

using namespace umma;

constexpr int kJobs = 4;
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

struct Job {
  CUtensorMap wmap;
  const void* scales;
  const void* offsets;                 // may be null
  const void* bias;                    // may be null; element 0 belongs to output column 0 of this job
  int64_t col0;
  int rows, row_tiles, bits, num_groups, group_shift;  // group = 64 << group_shift
};

struct Params {
  Job job[kJobs];
  CUtensorMap xmap;
  void* out;
  int64_t out_stride;
  int jobs, m, chunks;                 // chunks of 128 values of K
  int row_tiles, tiles;                // over all jobs; tiles = row_tiles x token tiles
  int n_tile, d_buffers, tmem_columns;
  int x_slots, w_slots, w_bytes;       // rings; bytes of a weight slot
  int slices;
  uint32_t ring_offset, barrier_offset;
};

__device__ unsigned int g_gemm_failed = 0;

struct Bars {
  uint32_t x_full, x_empty, w_full, w_empty, a_full, a_empty, d_full, d_empty, drain;
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

// Warpgroup `group`'s chunks of a row tile: chunk c0 + i is stage stage0 + i, numbered over the life of
// the block.  False once a wait has run out.
template <int BITS, bool BF16, bool MBF16, bool SPLIT>
__device__ bool decode_tile(const Job& job, const Params& p, int row0, int c0, int group, uint32_t stage0, int stages,
                            const unsigned char* w_ring, const Bars& bars, uint32_t tmem, Cursor& w_at, uint32_t& a_pass,
                            volatile int* failed) {
  constexpr int kGroups = Roles<SPLIT>::kGroups;
  const int lane = threadIdx.x & 31;
  const int warp4 = (threadIdx.x >> 5) & 3;
  const int r = warp4 * 32 + lane;
  const int row = min(row0 + r, job.rows - 1);
  const unsigned short* s_row = static_cast<const unsigned short*>(job.scales) + static_cast<int64_t>(row) * job.num_groups;
  const unsigned short* o_row =
      job.offsets == nullptr ? nullptr : static_cast<const unsigned short*>(job.offsets) + static_cast<int64_t>(row) * job.num_groups;
  auto widen = [&](unsigned short v) -> float {
    return MBF16 ? __uint_as_float(static_cast<uint32_t>(v) << 16) : __half2float(__ushort_as_half(v));
  };
  const bool two_groups = job.group_shift == 0;  // 64-value groups: a chunk holds two
  auto group_of = [&](int i, int half) -> int { return min((2 * (c0 + i) + half) >> job.group_shift, job.num_groups - 1); };
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
    affine.set(s_next[0], o_row != nullptr ? widen(o_next[0]) : 0.0f);
    const unsigned short s_half = s_next[1], o_half = o_next[1];
    fetch(min(i + kGroups, stages - 1));  // the next chunk's metadata travels while this one is decoded
    const uint32_t slot = w_at.slot;
    if (!mbar_wait(bars.w_full + slot * 8, w_at.pass, failed)) return false;
    const uint32_t dst = tmem + group * Roles<SPLIT>::kTileColumns + (static_cast<uint32_t>(warp4 * 32) << 16);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      uint32_t w[2 * BITS], v[16], low[16];
      read_row64<BITS>(w_ring + slot * p.w_bytes, r, half, w);
      if (half == 1 && two_groups) affine.set(s_half, o_row != nullptr ? widen(o_half) : 0.0f);
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
    w_at.advance(static_cast<uint32_t>(p.w_slots), kGroups);
    a_pass ^= 1;
  }
  return true;
}

// SPLIT: the weights enter as the sum of two 16-bit operands, so that nothing of their fp32 values is
// lost that the sums could show.  Up to DQ_GEMV_CHUNKED_MAX_ROWS activation rows, where the mma.sync
// kernels scale fp32 accumulators and never round a weight; above that the dense path this kernel
// replaces rounds every weight once, and so does this kernel.
template <bool BF16, bool MBF16, bool SPLIT>
__global__ void __launch_bounds__(Roles<SPLIT>::kThreads, 1) gemm_umma_kernel(const __grid_constant__ Params p) {
  constexpr int kGroups = Roles<SPLIT>::kGroups;
  extern __shared__ __align__(1024) unsigned char smem[];
  // control block at the front: failure flag, tensor memory address, barriers
  volatile int* failed = reinterpret_cast<volatile int*>(smem);
  const uint32_t base = smem_addr(smem);
  Bars bars;
  bars.x_full = base + p.barrier_offset;
  bars.x_empty = bars.x_full + kMaxRing * 8;
  bars.w_full = bars.x_empty + kMaxRing * 8;
  bars.w_empty = bars.w_full + kMaxRing * 8;
  bars.a_full = bars.w_empty + kMaxRing * 8;
  bars.a_empty = bars.a_full + kMaxGroups * 8;
  bars.d_full = bars.a_empty + kMaxGroups * 8;
  bars.d_empty = bars.d_full + 2 * 8;
  bars.drain = bars.d_empty + 2 * 8;
  const int x_bytes = p.n_tile * 256;  // two slabs of 64 values
  unsigned char* x_ring = smem + p.ring_offset;
  unsigned char* w_ring = x_ring + p.x_slots * x_bytes;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    *failed = 0;
    for (int i = 0; i < p.x_slots; ++i) mbar_init(bars.x_full + i * 8, 1), mbar_init(bars.x_empty + i * 8, 1);
    for (int i = 0; i < p.w_slots; ++i) mbar_init(bars.w_full + i * 8, 1), mbar_init(bars.w_empty + i * 8, 4);
    for (int i = 0; i < kGroups; ++i) mbar_init(bars.a_full + i * 8, 4), mbar_init(bars.a_empty + i * 8, 1);
    for (int i = 0; i < 2; ++i) mbar_init(bars.d_full + i * 8, 1), mbar_init(bars.d_empty + i * 8, 4 * kGroups);
    mbar_init(bars.drain, 1);
    fence_mbar_init();
    tma_prefetch_map(&p.xmap);
  }
  if (warp == 3) tmem_alloc(base + 4, static_cast<uint32_t>(p.tmem_columns));
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + 4);
  const uint32_t d_tmem = tmem + Roles<SPLIT>::kColumns;
  pdl_launch_dependents();

  // this CTA's share of the reduction axis (slices: as equal as possible, in chunks)
  const int slice = static_cast<int>(blockIdx.y);
  const int c0 = static_cast<int>(static_cast<int64_t>(p.chunks) * slice / p.slices);
  const int c1 = static_cast<int>(static_cast<int64_t>(p.chunks) * (slice + 1) / p.slices);

  auto job_of = [&](int row_tile, int& local) -> int {
    int j = 0;
    local = row_tile;
    while (j + 1 < p.jobs && local >= p.job[j].row_tiles) local -= p.job[j++].row_tiles;
    return j;
  };

  if (warp == 0 || warp == 2) {
    if (elect_one()) {
      const bool weights = warp == 2;
      if (!weights) pdl_wait_prior_grid();  // the activation is the previous kernel's; weights are nobody's
      const uint32_t full = weights ? bars.w_full : bars.x_full, empty = weights ? bars.w_empty : bars.x_empty;
      const uint32_t slots = static_cast<uint32_t>(weights ? p.w_slots : p.x_slots);
      Cursor at;
      uint32_t issued = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x) {
        int local;
        const Job& job = p.job[job_of(tile % p.row_tiles, local)];
        const int token0 = (tile / p.row_tiles) * p.n_tile;
        const int count = c1 - c0;
        const int bytes = weights ? 2048 * job.bits : x_bytes;
        for (int i = 0; i < count; ++i, ++issued, at.advance(slots)) {
          const uint32_t slot = at.slot;
          if (!(ok = mbar_wait(empty + slot * 8, at.pass ^ 1, failed))) break;
          mbar_expect(full + slot * 8, static_cast<uint32_t>(bytes));
          if (weights) {
            tma_load_2d(smem_addr(w_ring) + slot * p.w_bytes, &job.wmap, (c0 + i) * 4 * job.bits, local * 128, full + slot * 8);
          } else {
            const uint32_t dst = smem_addr(x_ring) + slot * x_bytes;
            tma_load_2d(dst, &p.xmap, (c0 + i) * 128, token0, full + slot * 8);
            tma_load_2d(dst + x_bytes / 2, &p.xmap, (c0 + i) * 128 + 64, token0, full + slot * 8);
          }
        }
      }
      if (!ok || *failed != 0) {  // wait for the copies in flight
        for (uint32_t k = issued > slots ? issued - slots : 0; k < issued; ++k) {
          for (int i = 0; i < kSpins && !mbar_try(full + (k % slots) * 8, (k / slots) & 1); ++i) {
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = mma_descriptor(BF16, p.n_tile);
      Cursor x_at, a_at, d_at;
      bool ok = true;
      for (int tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x, d_at.advance(static_cast<uint32_t>(p.d_buffers))) {
        const uint32_t buffer = d_at.slot;
        if (!mbar_wait(bars.d_empty + buffer * 8, d_at.pass ^ 1, failed)) break;
        fence_after_sync();
        const uint32_t d = d_tmem + buffer * p.n_tile;
        for (int i = 0; i < c1 - c0; ++i) {
          const uint32_t xs = x_at.slot;
          if (!(ok = mbar_wait(bars.x_full + xs * 8, x_at.pass, failed))) break;
          const uint64_t b0 = smem_descriptor(smem_addr(x_ring) + xs * x_bytes);
          const uint64_t b1 = smem_descriptor(smem_addr(x_ring) + xs * x_bytes + x_bytes / 2);
          if (!(ok = mbar_wait(bars.a_full + a_at.slot * 8, a_at.pass, failed))) break;
          fence_after_sync();
          const uint32_t a = tmem + a_at.slot * Roles<SPLIT>::kTileColumns;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            mma_ts(d, a + k * 8, (k < 4 ? b0 : b1) + (k & 3) * 2, idesc, i > 0 || k > 0);
            if constexpr (SPLIT) mma_ts(d, a + 64 + k * 8, (k < 4 ? b0 : b1) + (k & 3) * 2, idesc, true);
          }
          mma_commit(bars.a_empty + a_at.slot * 8);
          a_at.advance(kGroups);
          mma_commit(bars.x_empty + xs * 8);
          x_at.advance(static_cast<uint32_t>(p.x_slots));
        }
        if (ok) mma_commit(bars.d_full + buffer * 8);
      }
      if (*failed != 0) {  // MMAs in flight read and write tensor memory: it is freed after them
        mma_commit(bars.drain);
        for (int i = 0; i < kSpins && !mbar_try(bars.drain, 0); ++i) {
        }
      }
    }
    __syncwarp();
  } else if (warp >= kDecodeWarp0) {
    const int group = (warp - kDecodeWarp0) >> 2;
    const int warp4 = warp & 3;
    const int r = warp4 * 32 + lane;
    const int stages = c1 - c0;
    uint32_t stage = 0;
    uint32_t a_pass = 0;
    Cursor w_at, d_at;
    w_at.advance(static_cast<uint32_t>(p.w_slots), static_cast<uint32_t>(group));
    for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x, d_at.advance(static_cast<uint32_t>(p.d_buffers)), stage += stages) {
      int local;
      const Job& job = p.job[job_of(tile % p.row_tiles, local)];
      bool ok;
#define DQ_DECODE(B) ok = decode_tile<B, BF16, MBF16, SPLIT>(job, p, local * 128, c0, group, stage, stages, w_ring, bars, tmem, w_at, a_pass, failed)
      switch (job.bits) {
        case 2: DQ_DECODE(2); break;
        case 3: DQ_DECODE(3); break;
        case 4: DQ_DECODE(4); break;
        default: DQ_DECODE(8); break;
      }
#undef DQ_DECODE
      if (!ok) break;
      const uint32_t buffer = d_at.slot;
      if (!mbar_wait(bars.d_full + buffer * 8, d_at.pass, failed)) break;
      fence_after_sync();
      const uint32_t src = d_tmem + buffer * p.n_tile + (static_cast<uint32_t>(warp4 * 32) << 16);
      const int row = local * 128 + r;
      const int token0 = (tile / p.row_tiles) * p.n_tile;
      const float bias = job.bias != nullptr && row < job.rows ? load_f32(job.bias, row, BF16 ? DQ_BF16 : DQ_F16) : 0.0f;
      unsigned short* dst = static_cast<unsigned short*>(p.out) + job.col0 + row;
      float* red = reinterpret_cast<float*>(smem + p.ring_offset);
      for (int col = group * 16; col < p.n_tile; col += kGroups * 16) {  // the warpgroups share the columns
        uint32_t v[16];
        tmem_ld16(src + col, v);
        tmem_wait_ld();
        if (p.slices > 1) {
#pragma unroll
          for (int i = 0; i < 16; ++i) red[(col + i) * 128 + r] = __uint_as_float(v[i]);
        } else if (row < job.rows) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int token = token0 + col + i;
            if (token < p.m) {
              dst[static_cast<int64_t>(token) * p.out_stride] =
                  static_cast<unsigned short>(round_to_16(__uint_as_float(v[i]) + bias, BF16 ? DQ_BF16 : DQ_F16));
            }
          }
        }
      }
      fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bars.d_empty + buffer * 8);
    }
  }

  __syncthreads();
  if (p.slices > 1) {  // one tile per cluster: add the slices' columns, a share of them per CTA
    cluster_sync();
    const int tile = blockIdx.x;
    int local;
    const Job& job = p.job[job_of(tile % p.row_tiles, local)];
    const int per = (p.n_tile + p.slices - 1) / p.slices;
    const int first = slice * per, last = min(first + per, p.n_tile);
    const int row = local * 128 + (threadIdx.x & 127);
    const int token0 = (tile / p.row_tiles) * p.n_tile;
    if (*failed == 0 && row < job.rows) {
      const float bias = job.bias != nullptr ? load_f32(job.bias, row, BF16 ? DQ_BF16 : DQ_F16) : 0.0f;
      unsigned short* dst = static_cast<unsigned short*>(p.out) + job.col0 + row;
      const uint32_t red = base + p.ring_offset + (threadIdx.x & 127) * 4;
      for (int col = first + (threadIdx.x >> 7); col < last && token0 + col < p.m; col += Roles<SPLIT>::kThreads / 128) {
        float part[8];  // all requested, then added in slice order
#pragma unroll
        for (int s = 0; s < 8; ++s) part[s] = s < p.slices ? cluster_ld(red + col * 512, s) : 0.0f;
        float sum = part[0];
#pragma unroll
        for (int s = 1; s < 8; ++s) sum += part[s];
        dst[static_cast<int64_t>(token0 + col) * p.out_stride] =
            static_cast<unsigned short>(round_to_16(sum + bias, BF16 ? DQ_BF16 : DQ_F16));
      }
    }
    cluster_sync();  // nobody leaves while its sums are being read
  }
  if (threadIdx.x == 0 && *failed != 0) atomicOr(&g_gemm_failed, 1u);
  fence_after_sync();
  if (warp == 3) tmem_free(tmem, static_cast<uint32_t>(p.tmem_columns));
}

// ---------------------------------------------------------------------------
// Host
// ---------------------------------------------------------------------------

constexpr uint32_t kBarrierOffset = 64;
constexpr uint32_t kRingOffset = 1024;

bool encode_map(CUtensorMap* map, CUtensorMapDataType type, const void* base, int64_t inner, int64_t outer, int64_t row_bytes,
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

CUtensorMapSwizzle weight_swizzle(int bits) {
  return bits == 2 ? CU_TENSOR_MAP_SWIZZLE_32B : bits == 3 ? CU_TENSOR_MAP_SWIZZLE_NONE : bits == 4 ? CU_TENSOR_MAP_SWIZZLE_64B
                                                                                                     : CU_TENSOR_MAP_SWIZZLE_128B;
}

// 64 << shift values per group, or -1.
int group_shift_of(int group_values) {
  for (int s = 0; s < 16; ++s) {
    if (group_values == (64 << s)) return s;
  }
  return -1;
}

bool geometry_ok(const GemvArgs& a, int bits) {
  const bool x16 = a.x_dtype == DQ_BF16 || a.x_dtype == DQ_F16, meta16 = a.meta_dtype == DQ_BF16 || a.meta_dtype == DQ_F16;
  if (!x16 || !meta16 || a.out_dtype != a.x_dtype || a.in_features % 8 != 0 || group_shift_of(a.group_values) < 0) return false;
  if (a.words_per_group * 32 != a.group_values * bits || a.words_per_row % 4 != 0) return false;
  return reinterpret_cast<uintptr_t>(a.x) % 16 == 0 && reinterpret_cast<uintptr_t>(a.packed) % 16 == 0;
}

struct Shape {
  int n_tile, token_tiles, slices;
};

// Token tiles and slices of the reduction axis with the least estimated time: waves of CTAs times
// the cycles of one -- 128-value stages, each bound by the hand-over between the block's roles or by
// the tensor pipe (2 n_tile cycles per 64 values), plus a start and an end.  The slices of all tiles
// are resident at once or there are none: a second wave of clusters costs more than it gives (4096 x
// 14336, 16 rows: 22 us with 4 slices, 38 with 8), and clusters of eight pack badly into the GPCs
// (1152 x 7936, 128 rows: 14 us with 6 slices, 21 with 8).
Shape pick_shape(int m, int row_tiles, int chunks, int sm_count) {
  Shape best = {};
  double best_cost = 1e30;
  const int min_tiles = static_cast<int>(ceil_div(m, 256));
  for (int tt = min_tiles; tt <= min_tiles + 2; ++tt) {
    const int n = static_cast<int>(ceil_div(ceil_div(m, tt), 16) * 16);
    if (n * (tt - 1) >= m) continue;
    const double stage = std::max(700.0, 4.0 * n + 60.0);
    for (int s = 1; s <= 6 && s <= chunks; ++s) {
      const int64_t ctas = static_cast<int64_t>(row_tiles) * tt * s;
      const int resident = s <= 2 ? sm_count : s <= 4 ? sm_count - 16 : sm_count - 24;
      if (s > 1 && ctas > resident) break;
      const double waves = std::ceil(static_cast<double>(ctas) / sm_count);
      const double hidden = s == 1 && n <= 128 ? 0.0 : 10.0 * n;  // an epilogue that the next tile does not cover
      const double cost = waves * (static_cast<double>(ceil_div(chunks, s)) * stage + hidden) + (s > 1 ? 1500.0 : 0.0) + 10.0 * n + 7000.0;
      if (cost < best_cost) best_cost = cost, best = {n, tt, s};
    }
  }
  return best;
}

}  // namespace

int32_t launch_gemm_umma(const GemvArgs* args, const int* bits, int count, cudaStream_t stream, bool* taken) {
  *taken = false;
  const DeviceInfo* dev = device_info();
  if (dev == nullptr) return DQ_ERR_CUDA;
  if (count < 1 || count > kJobs) return DQ_OK;
  Params p = {};
  const GemvArgs& a = args[0];
  int w_bytes = 0;
  for (int i = 0; i < count; ++i) {
    const GemvArgs& b = args[i];
    if (!geometry_ok(b, bits[i]) || b.x != a.x || b.m != a.m || b.out != a.out || b.out_stride != a.out_stride ||
        b.in_features != a.in_features || b.meta_dtype != a.meta_dtype || b.rows < 1) {
      return DQ_OK;
    }
    Job& job = p.job[i];
    if (!encode_map(&job.wmap, CU_TENSOR_MAP_DATA_TYPE_INT32, b.packed, b.words_per_row, b.rows, static_cast<int64_t>(b.words_per_row) * 4,
                    4 * bits[i], 128, weight_swizzle(bits[i]))) {
      return DQ_OK;
    }
    job.scales = b.scales;
    job.offsets = b.offsets;
    job.col0 = b.out_col0;
    job.bias = b.bias == nullptr ? nullptr : static_cast<const unsigned short*>(b.bias) + b.out_col0;
    job.rows = b.rows;
    job.row_tiles = static_cast<int>(ceil_div(b.rows, 128));
    job.bits = bits[i];
    job.num_groups = b.num_groups;
    job.group_shift = group_shift_of(b.group_values);
    p.row_tiles += job.row_tiles;
    w_bytes = std::max(w_bytes, 2048 * bits[i]);
  }
  p.jobs = count;
  p.m = a.m;
  p.out = a.out;
  p.out_stride = a.out_stride;
  p.chunks = static_cast<int>(ceil_div(a.in_features, 128));
  Shape shape = pick_shape(a.m, p.row_tiles, p.chunks, dev->sm_count);
  if (const int n = tuning_int("DQ_B200_UMMA_N", 0)) shape.n_tile = n, shape.token_tiles = static_cast<int>(ceil_div(a.m, n));
  if (const int s = tuning_int("DQ_B200_UMMA_SLICES", 0)) shape.slices = s;
  p.n_tile = shape.n_tile;
  p.slices = shape.slices;
  p.tiles = p.row_tiles * shape.token_tiles;
  if (!encode_map(&p.xmap, a.x_dtype == DQ_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, a.x, a.in_features, a.m,
                  static_cast<int64_t>(a.in_features) * 2, 64, p.n_tile, CU_TENSOR_MAP_SWIZZLE_128B)) {
    return DQ_OK;
  }
  const int grid_x = p.slices > 1 ? p.tiles : std::min(p.tiles, dev->sm_count);
  const bool split = a.m <= DQ_GEMV_CHUNKED_MAX_ROWS;
  const int a_columns = split ? Roles<true>::kColumns : Roles<false>::kColumns;
  p.d_buffers = p.slices == 1 && p.tiles > grid_x && a_columns + 2 * p.n_tile <= 512 ? 2 : 1;
  p.tmem_columns = 32;
  while (p.tmem_columns < a_columns + p.d_buffers * p.n_tile) p.tmem_columns *= 2;
  // Rings: activation slots of 128 values (2..6), then weight slots -- a multiple of the warpgroups, so
  // that a slot always belongs to the same one (its barrier then cannot be two passes behind).
  const int x_bytes = p.n_tile * 256;
  p.w_bytes = w_bytes;
  const int budget = dev->max_smem_optin - static_cast<int>(kRingOffset);
  p.x_slots = std::clamp((budget - kMaxGroups * w_bytes) / x_bytes, 2, 6);
  const int groups = split ? Roles<true>::kGroups : Roles<false>::kGroups;
  p.w_slots = std::clamp((budget - p.x_slots * x_bytes) / w_bytes / groups * groups, groups, 12);
  p.barrier_offset = kBarrierOffset;
  p.ring_offset = kRingOffset;
  const size_t smem = kRingOffset + static_cast<size_t>(p.x_slots) * x_bytes + static_cast<size_t>(p.w_slots) * w_bytes;

  const bool mbf = a.meta_dtype == DQ_BF16;
  auto run = [&](auto kernel) -> int32_t {
    DQ_CUDA(allow_shared(kernel, smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(grid_x), static_cast<unsigned>(p.slices));
    cfg.blockDim = dim3(static_cast<unsigned>(split ? Roles<true>::kThreads : Roles<false>::kThreads));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (p.slices > 1) {
      attr[n].id = cudaLaunchAttributeClusterDimension;
      attr[n].val.clusterDim.x = 1;
      attr[n].val.clusterDim.y = static_cast<unsigned>(p.slices);
      attr[n].val.clusterDim.z = 1;
      ++n;
    }
    if (pdl_enabled_for_rows()) {
      attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[n].val.programmaticStreamSerializationAllowed = 1;
      ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    DQ_CUDA(cudaLaunchKernelEx(&cfg, kernel, p));
    DQ_CHECK_LAUNCH("gemm");
    note_kernel("gemm_umma_kernel");
    *taken = true;
    return DQ_OK;
  };
  if (split) {
    if (a.x_dtype == DQ_BF16) return mbf ? run(gemm_umma_kernel<true, true, true>) : run(gemm_umma_kernel<true, false, true>);
    return mbf ? run(gemm_umma_kernel<false, true, true>) : run(gemm_umma_kernel<false, false, true>);
  }
  if (a.x_dtype == DQ_BF16) return mbf ? run(gemm_umma_kernel<true, true, false>) : run(gemm_umma_kernel<true, false, false>);
  return mbf ? run(gemm_umma_kernel<false, true, false>) : run(gemm_umma_kernel<false, false, false>);
}

}  // namespace dq

extern "C" int32_t dq_gemm_status(void* stream) {
  auto s = static_cast<cudaStream_t>(stream);
  unsigned int word = 0;
  DQ_CUDA(cudaMemcpyFromSymbolAsync(&word, dq::g_gemm_failed, sizeof(word), 0, cudaMemcpyDeviceToHost, s));
  DQ_CUDA(cudaStreamSynchronize(s));
  if (word != 0u) return dq::fail(DQ_ERR_DEVICE, "gemm: a wait inside a block ran out; an output of this device is incomplete");
  return DQ_OK;
}
