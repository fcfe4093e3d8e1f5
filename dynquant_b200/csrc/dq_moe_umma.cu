// An expert layer over many tokens on the fifth-generation tensor cores (the layer of dq_moe.cu, whose
// kernels take at most DQ_MOE_MAX_TOKENS tokens per call and read every active expert once per eight
// of its tokens).
//
// Five launches on the caller's stream, no host round trip:
//   1. route    one block: the assignments sorted by expert, and a table of column tiles -- up to
//               n_cap (64 or 128) tokens of one expert each, as equal as possible.
//   2. permute  the token rows in that order, so that a tile's activations are consecutive rows.
//   3. gate_up  the pipeline of dq_umma_pipeline.cuh, persistent over (column tile, 64 gate rows + the
//               64 matching up rows); each warp decodes 16 gate and the matching 16 up rows, so that the
//               epilogue pairs them by a shuffle; it stores h = silu(g) * u rounded to the activation
//               type, in sorted order.
//   4. down     the same over (column tile, 128 rows of the down bank) with h as the activation; fp32
//               results go back to assignment order.
//   5. combine  y[t] = sum_k p[t,k] * d[t,k] in slot order.
// Weights enter as two 16-bit operands (see SPLIT, dq_gemm_umma.cu), 16 (bf16) or 21 bits of each.  The
// order inside an expert is left to atomics: a column's result does not depend on its place, so the
// layer is bit-identical run to run all the same.
//
// Bound by the decode (every expert's values once per 128 of its tokens, about 0.5 us per 128 x 128
// values and SM) until experts have hundreds of tokens each.
#include <algorithm>
#include <cmath>

#include "dq_gemm_umma.cuh"
#include "dq_umma_pipeline.cuh"

namespace dq {
namespace {

using namespace umma;

constexpr int kRouteThreads = 1024;
constexpr int kMaxExperts = 1024;
constexpr int kGroups = Roles<true>::kGroups;
// Four warps more than the dense kernel: a tile is only 6 to 16 chunks long, so warps of their own finish
// it while the decoding warps work on the next (down, 6 chunks of 0.5 us per tile: 143 us per layer of
// 1000 tokens with the decoding warps doing it).
constexpr int kEpilogueWarp0 = kDecodeWarp0 + 4 * kGroups;
constexpr int kThreads = (kEpilogueWarp0 + 4) * 32;
// Activations come in boxes of 32 rows, as many as a tile has tokens for: 128 rows for every tile of 62
// tokens were 4.5 TB/s out of L2 (1000 tokens: gate_up 168 us).
constexpr int kBoxRows = 32;
constexpr int kColumns = 128;          // accumulator columns: one tile of up to 128 tokens, or two of up to 64

struct RouteTable {
  int num_tiles, num_rows, pad[2];  // column tiles; assignments that belong to a local expert
};

// tiles[i] = (expert, first sorted position, tokens, unused)
__global__ void __launch_bounds__(kRouteThreads) moe_route_kernel(const int32_t* ids, int first_expert, int num_experts, int assignments,
                                                                  int n_cap, RouteTable* table, int4* tiles, int32_t* order) {
  __shared__ int count[kMaxExperts], start[kMaxExperts], tile0[kMaxExperts];
  __shared__ int warp_rows[32], warp_tiles[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  pdl_launch_dependents();
  count[tid] = 0;
  __syncthreads();
  pdl_wait_prior_grid();
  for (int i = tid; i < assignments; i += kRouteThreads) {
    const int e = __ldcg(ids + i) - first_expert;
    if (e >= 0 && e < num_experts) atomicAdd(&count[e], 1);
  }
  __syncthreads();
  // exclusive sums over the experts of their rows and of their tiles
  const int mine = tid < num_experts ? count[tid] : 0;
  const int my_tiles = (mine + n_cap - 1) / n_cap;
  int rows = mine, nt = my_tiles;
#pragma unroll
  for (int d = 1; d < 32; d *= 2) {
    const int r = __shfl_up_sync(0xffffffffu, rows, d), t = __shfl_up_sync(0xffffffffu, nt, d);
    if (lane >= d) rows += r, nt += t;
  }
  if (lane == 31) warp_rows[warp] = rows, warp_tiles[warp] = nt;
  __syncthreads();
  if (warp == 0) {
    int r = warp_rows[lane], t = warp_tiles[lane];
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
      const int r2 = __shfl_up_sync(0xffffffffu, r, d), t2 = __shfl_up_sync(0xffffffffu, t, d);
      if (lane >= d) r += r2, t += t2;
    }
    warp_rows[lane] = r, warp_tiles[lane] = t;
  }
  __syncthreads();
  start[tid] = rows - mine + (warp > 0 ? warp_rows[warp - 1] : 0);
  tile0[tid] = nt - my_tiles + (warp > 0 ? warp_tiles[warp - 1] : 0);
  if (tid == 0) *table = {warp_tiles[31], warp_rows[31], {0, 0}};
  if (mine > 0) {
    const int each = (mine + my_tiles - 1) / my_tiles;
    for (int i = 0; i < my_tiles; ++i) {
      tiles[tile0[tid] + i] = make_int4(tid, start[tid] + i * each, min(each, mine - i * each), 0);
    }
  }
  __syncthreads();
  for (int i = tid; i < assignments; i += kRouteThreads) {
    const int e = __ldcg(ids + i) - first_expert;
    if (e >= 0 && e < num_experts) order[atomicAdd(&start[e], 1)] = i;
  }
}

// Row `i` of xs = the token of assignment order[i]; 16-byte pieces, a row per warp and round.
__global__ void __launch_bounds__(256) moe_permute_kernel(const uint4* x, const RouteTable* table, const int32_t* order, int topk,
                                                          int pieces, uint4* xs) {
  pdl_launch_dependents();
  pdl_wait_prior_grid();
  const int rows = __ldcg(&table->num_rows), lane = threadIdx.x & 31;
  for (int i = blockIdx.x * 8 + (threadIdx.x >> 5); i < rows; i += gridDim.x * 8) {
    const uint4* src = x + static_cast<int64_t>(__ldcg(order + i) / topk) * pieces;
    uint4* dst = xs + static_cast<int64_t>(i) * pieces;
    for (int p = lane; p < pieces; p += 32) dst[p] = __ldcg(src + p);
  }
}

struct Params {
  CUtensorMap wmap, xmap;
  Meta meta;
  const RouteTable* table;
  const int4* tiles;
  const int32_t* order;
  void* out;                 // h [sorted position, rows] or d [assignment, rows]
  int64_t bank_rows;         // rows of the whole bank
  int rows;                  // output rows per expert (inter, or hidden)
  int row_blocks;            // of 64 (gate_up) or 128 (down) rows per expert
  int chunks, bits;
  int n_cap;
  int x_slots, w_slots, w_bytes;
  int give_up;               // dq_gemm_fail_next
  unsigned int* report;
};

constexpr uint32_t kBarrierOffset = 64, kOrderOffset = 1024, kPowersOffset = 3072;
constexpr uint32_t ring_offset(bool scaled_rows) { return scaled_rows ? 4096 : kPowersOffset; }
static_assert(kBarrierOffset + kBarrierBytes <= kOrderOffset, "");

// Where a tile's accumulator lies.  Tiles of up to 64 tokens take the two halves of the columns in turn
// (the MMAs of one run under the epilogue of the other), a larger one takes both; every role walks the
// same sequence.
struct Halves {
  uint32_t at = 0, passes = 0;  // passes: a parity bit per half
  bool both = false;
  __device__ __forceinline__ void take(int tokens) {
    both = tokens > 64;
    if (both) at = 0;
  }
  __device__ __forceinline__ bool wait(uint32_t bars, uint32_t flip, volatile int* failed) const {
    return mbar_wait(bars + at * 8, ((passes >> at) & 1) ^ flip, failed) && (!both || mbar_wait(bars + 8, (passes >> 1) ^ flip, failed));
  }
  __device__ __forceinline__ void done() {
    passes ^= both ? 3u : 1u << at;
    if (!both) at ^= 1;
  }
};

template <bool BF16, bool MBF16, bool GATE_UP>
__global__ void __launch_bounds__(kThreads, 1) moe_umma_kernel(const __grid_constant__ Params p) {
  extern __shared__ __align__(1024) unsigned char smem[];
  volatile int* failed = reinterpret_cast<volatile int*>(smem);
  InFlight* left = reinterpret_cast<InFlight*>(smem + 8);
  const uint32_t base = smem_addr(smem);
  const Bars bars = bars_at(base + kBarrierOffset);
  const int x_bytes = p.n_cap * 256;
  unsigned char* x_ring = smem + ring_offset(kScaledRows<BF16, true>);
  signed char* powers = reinterpret_cast<signed char*>(smem + kPowersOffset);  // of a tile's rows, by slot
  unsigned char* w_ring = x_ring + p.x_slots * x_bytes;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    *failed = p.give_up;
    init_bars(bars, p.x_slots, p.w_slots, kGroups, 4, 4, 4 * kGroups + 4);
    tma_prefetch_map(&p.xmap);
    tma_prefetch_map(&p.wmap);
  }
  if (warp == 3) tmem_alloc(base + 4, 512);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + 4);
  const uint32_t d_tmem = tmem + Roles<true>::kColumns;
  pdl_launch_dependents();
  pdl_wait_prior_grid();  // the routing and the activation

  const int tiles = __ldcg(&p.table->num_tiles) * p.row_blocks;
  // (column tile, row block) of a tile; the next one's entry is requested while this one is worked on
  auto entry = [&](int tile) -> int4 { return tile < tiles ? __ldcg(p.tiles + tile / p.row_blocks) : make_int4(0, 0, 0, 0); };

  // The bank's row at `place` of a tile's 128.
  const auto row_of = [&](int4 e, int block, int place) -> int64_t {
    const int64_t row = GATE_UP ? static_cast<int64_t>(e.x) * 2 * p.rows + block * 64 + (place < 64 ? place : p.rows + place - 64)
                                : static_cast<int64_t>(e.x) * p.rows + block * 128 + place;
    return row < p.bank_rows ? row : p.bank_rows - 1;
  };

  if (warp == 0 || warp == 2) {
    if (elect_one()) {
      const bool weights = warp == 2;
      const uint32_t full = weights ? bars.w_full : bars.x_full, empty = weights ? bars.w_empty : bars.x_empty;
      const uint32_t slots = static_cast<uint32_t>(weights ? p.w_slots : p.x_slots);
      Cursor at;
      uint32_t issued = 0;
      bool ok = true;
      int4 next = entry(blockIdx.x);
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        const int4 e = next;
        next = entry(tile + gridDim.x);
        const int block = tile % p.row_blocks;
        const int boxes = (e.z + kBoxRows - 1) / kBoxRows;  // of activation rows, per slab of 64 values
        const uint32_t bytes = static_cast<uint32_t>(weights ? 2048 * p.bits : boxes * kBoxRows * 256);
        const int w_row = GATE_UP ? e.x * 2 * p.rows + block * 64 : e.x * p.rows + block * 128;
        for (int i = 0; i < p.chunks; ++i, ++issued, at.advance(slots)) {
          const uint32_t slot = at.slot;
          if (!(ok = mbar_wait(empty + slot * 8, at.pass ^ 1, failed))) break;
          mbar_expect(full + slot * 8, bytes);
          if (weights) {
            const uint32_t dst = smem_addr(w_ring) + slot * p.w_bytes;
            tma_load_2d(dst, &p.wmap, i * 4 * p.bits, w_row, full + slot * 8);
            if (GATE_UP) tma_load_2d(dst + 1024 * p.bits, &p.wmap, i * 4 * p.bits, w_row + p.rows, full + slot * 8);
          } else {
            const uint32_t dst = smem_addr(x_ring) + slot * x_bytes;
            for (int b = 0; b < boxes; ++b) {
              tma_load_2d(dst + b * (kBoxRows * 128), &p.xmap, i * 128, e.y + b * kBoxRows, full + slot * 8);
              tma_load_2d(dst + x_bytes / 2 + b * (kBoxRows * 128), &p.xmap, i * 128 + 64, e.y + b * kBoxRows, full + slot * 8);
            }
          }
        }
      }
      left->issued[warp] = issued;
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      Cursor x_at, a_at;
      Halves halves;
      bool ok = true;
      int4 next = entry(blockIdx.x);
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x, halves.done()) {
        const int4 e = next;
        next = entry(tile + gridDim.x);
        const uint32_t idesc = mma_descriptor(BF16, (e.z + 15) / 16 * 16);
        halves.take(e.z);
        if (!halves.wait(bars.d_empty, 1, failed)) break;
        fence_after_sync();
        const uint32_t d = d_tmem + halves.at * 64;
        for (int i = 0; i < p.chunks; ++i) {
          const uint32_t xs = x_at.slot;
          if (!(ok = mbar_wait(bars.x_full + xs * 8, x_at.pass, failed))) break;
          if (!(ok = mbar_wait(bars.a_full + a_at.slot * 8, a_at.pass, failed))) break;
          fence_after_sync();
          const uint32_t xb = smem_addr(x_ring) + xs * x_bytes;
          mma_chunk<true>(d, tmem + a_at.slot * Roles<true>::kTileColumns, smem_descriptor(xb), smem_descriptor(xb + x_bytes / 2), idesc, i > 0);
          mma_commit(bars.a_empty + a_at.slot * 8);
          mma_commit(bars.x_empty + xs * 8);
          x_at.advance(static_cast<uint32_t>(p.x_slots));
          a_at.advance(kGroups);
        }
        if (ok) {
          mma_commit(bars.d_full + halves.at * 8);
          if (halves.both) mma_commit(bars.d_full + 8);
        }
      }
      left->mma_lane = lane;
    }
    __syncwarp();
  } else if (warp >= kDecodeWarp0) {
    // The rows of a warp's 32 lanes: for gate_up 16 gate rows and the matching 16 up rows.
    const int warp4 = warp & 3, pair = warp4 * 16 + (lane & 15);
    const int tile_row = GATE_UP ? (lane < 16 ? 0 : 64) + pair : warp4 * 32 + lane;
    int4 next = entry(blockIdx.x);
    Cursor p_at;  // (kScaledRows) where this warp reads the rows' powers
    const auto read_power = [&](int& k) -> bool {
      if (!mbar_wait(bars.p_full + p_at.slot * 8, p_at.pass, failed)) return false;
      k = powers[p_at.slot * 128 + tile_row];
      __syncwarp();
      if (lane == 0) mbar_arrive(bars.p_empty + p_at.slot * 8);
      p_at.advance(kPowerSlots);
      return true;
    };
    if (warp < kEpilogueWarp0) {
      const int group = (warp - kDecodeWarp0) >> 2;
      const WeightRing ring = {w_ring, p.w_slots, p.w_bytes};
      uint32_t stage = 0, a_pass = 0;
      Cursor w_at;
      w_at.advance(static_cast<uint32_t>(p.w_slots), static_cast<uint32_t>(group));
      bool ok = true;
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x, stage += p.chunks) {
        const int4 e = next;
        next = entry(tile + gridDim.x);
        const int block = tile % p.row_blocks;
        const int64_t bank_row = row_of(e, block, tile_row);
        int k = 0;  // what the row is multiplied by: 2^k
        if constexpr (kScaledRows<BF16, true>) {
          if (!read_power(k)) break;
        }
#define DQ_DECODE(B) \
  ok = decode_tile<B, BF16, MBF16, true>(p.meta, bank_row, tile_row, power_of_two(k), 0, group, stage, p.chunks, ring, bars, tmem, w_at, a_pass, failed)
        switch (p.bits) {
          case 2: DQ_DECODE(2); break;
          case 3: DQ_DECODE(3); break;
          case 4: DQ_DECODE(4); break;
          default: DQ_DECODE(8); break;
        }
#undef DQ_DECODE
      }
    } else {
      int* places = reinterpret_cast<int*>(smem + kOrderOffset) + warp4 * kColumns;  // this warp's copy of the tile's assignments
      Halves halves;
      // The rows' powers (kScaledRows) for the decoding warps too, two tiles ahead of them: a scan of their own
      // would hold the decode up, and one warp for all four takes longer than a tile of the down projection.
      Cursor found;
      int4 ahead = entry(blockIdx.x);
      const auto find_power = [&](int tile) -> bool {
        if (tile >= tiles) return true;
        if (!mbar_wait(bars.p_empty + found.slot * 8, found.pass ^ 1, failed)) return false;
        const int4 e = ahead;
        ahead = entry(tile + gridDim.x);
        powers[found.slot * 128 + tile_row] =
            static_cast<signed char>(row_power<MBF16>(p.meta, p.bits, p.bank_rows, row_of(e, tile % p.row_blocks, tile_row), 0, p.meta.num_groups));
        __syncwarp();
        if (lane == 0) mbar_arrive(bars.p_full + found.slot * 8);
        found.advance(kPowerSlots);
        return true;
      };
      bool ok = true;
      if constexpr (kScaledRows<BF16, true>) ok = find_power(blockIdx.x) && find_power(blockIdx.x + gridDim.x);
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x, halves.done()) {
        const int4 e = next;
        next = entry(tile + gridDim.x);
        const int block = tile % p.row_blocks;
        const int row = GATE_UP ? block * 64 + pair : block * 128 + tile_row;  // of the expert's output rows
        if (!GATE_UP) {
          __syncwarp();
          for (int c = lane; c < e.z; c += 32) places[c] = __ldcg(p.order + e.y + c);
          __syncwarp();
        }
        int k = 0;
        if constexpr (kScaledRows<BF16, true>) {
          if (!read_power(k)) break;
        }
        halves.take(e.z);
        if (!halves.wait(bars.d_full, 0, failed)) break;
        fence_after_sync();
        const uint32_t src = d_tmem + halves.at * 64 + (static_cast<uint32_t>(warp4 * 32) << 16);
        for (int col = 0; col < e.z; col += 16) {
          uint32_t v[16];
          tmem_ld16(src + col, v);
          tmem_wait_ld();
          if constexpr (kScaledRows<BF16, true>) {
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * power_of_two(-k));
          }
          if constexpr (GATE_UP) {
            // lane l < 16 has gate row l, lane l + 16 the matching up row: each finishes eight of the columns
            const int first = col + (lane < 16 ? 0 : 8);
            unsigned short* dst = static_cast<unsigned short*>(p.out) + static_cast<int64_t>(e.y + first) * p.rows + row;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float other = __uint_as_float(__shfl_xor_sync(0xffffffffu, lane < 16 ? v[i + 8] : v[i], 16));
              const float g = lane < 16 ? __uint_as_float(v[i]) : other, u = lane < 16 ? other : __uint_as_float(v[i + 8]);
              if (row < p.rows && first + i < e.z) {
                dst[static_cast<int64_t>(i) * p.rows] =
                    static_cast<unsigned short>(round_to_16((g / (1.0f + __expf(-g))) * u, BF16 ? DQ_BF16 : DQ_F16));
              }
            }
          } else if (row < p.rows) {
            float* dst = static_cast<float*>(p.out) + row;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              if (col + i < e.z) dst[static_cast<int64_t>(places[col + i]) * p.rows] = __uint_as_float(v[i]);
            }
          }
        }
        fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(bars.d_empty + halves.at * 8);
          if (halves.both) mbar_arrive(bars.d_empty + 8);
        }
        if constexpr (kScaledRows<BF16, true>) ok = find_power(tile + 2 * gridDim.x);
      }
    }
  }

  __syncthreads();
  if (*failed != 0) {  // (the same for all: every role has stopped)
    drain(*left, bars, p.x_slots, p.w_slots);
    __syncthreads();
  }
  if (threadIdx.x == 0 && *failed != 0) report_to_host(p.report, kReportWait);
  fence_after_sync();
  if (warp == 3) tmem_free(tmem, 512);
}

// A quad of columns per thread, the tokens over the grid's y axis (which ends at 65535) and round it.
constexpr int64_t kMaxGridY = 65535;
__global__ void __launch_bounds__(256) moe_combine_rows_kernel(const float4* d, const float* w, const int32_t* ids, int first_expert,
                                                               int tokens, int topk, int quads, int num_experts, void* y, int y_dtype) {
  pdl_launch_dependents();
  pdl_wait_prior_grid();
  const int q = blockIdx.x * 256 + threadIdx.x;
  if (q >= quads) return;
  for (int token = blockIdx.y; token < tokens; token += gridDim.y) {
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int k = 0; k < topk; ++k) {
      const int a = token * topk + k, e = __ldcg(ids + a) - first_expert;
      if (e < 0 || e >= num_experts) continue;
      const float p = __ldcg(w + a);
      const float4 v = __ldcg(d + static_cast<int64_t>(a) * quads + q);
      acc.x = fmaf(p, v.x, acc.x), acc.y = fmaf(p, v.y, acc.y), acc.z = fmaf(p, v.z, acc.z), acc.w = fmaf(p, v.w, acc.w);
    }
    const int64_t at = static_cast<int64_t>(token) * quads + q;
    if (y_dtype == DQ_F32) {
      static_cast<float4*>(y)[at] = acc;
    } else {
      static_cast<uint2*>(y)[at] = make_uint2(round_pair_to_16(acc.x, acc.y, y_dtype), round_pair_to_16(acc.z, acc.w, y_dtype));
    }
  }
}

// ---------------------------------------------------------------------------
// Host
// ---------------------------------------------------------------------------

struct Layout {
  size_t table, tiles, order, xs, h, d, total;
};

Layout layout_of(int64_t tokens, int64_t topk, int64_t hidden, int64_t inter, int64_t experts, int act_bytes) {
  auto up = [](size_t v) { return (v + 255) / 256 * 256; };
  const size_t a = static_cast<size_t>(tokens * topk);
  Layout l = {};
  size_t at = 0;
  l.table = at, at = up(at + sizeof(RouteTable));
  l.tiles = at, at = up(at + (a / 64 + static_cast<size_t>(experts) + 1) * sizeof(int4));
  l.order = at, at = up(at + a * 4);
  l.xs = at, at = up(at + a * hidden * act_bytes);
  l.h = at, at = up(at + a * inter * act_bytes);
  l.d = at, at = up(at + a * hidden * 4);
  l.total = at;
  return l;
}

template <typename Kernel, typename... Args>
int32_t launch(Kernel kernel, dim3 grid, int threads, size_t smem, cudaStream_t stream, const char* name, Args... args) {
  if (smem > 48 * 1024) DQ_CUDA(allow_shared(kernel, smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(static_cast<unsigned>(threads));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled_for_rows() ? 1 : 0;
  DQ_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
  DQ_CHECK_LAUNCH(name);
  return DQ_OK;
}

template <bool GATE_UP>
int32_t launch_bank(const dq_weight& w, const dq_geometry& g, const void* act, int act_dtype, int64_t act_rows, int rows, Params p,
                    const DeviceInfo& dev, cudaStream_t stream) {
  p.meta = {w.scales, w.offsets, g.num_groups, 1};
  p.bank_rows = w.rows;
  p.rows = rows;
  p.row_blocks = static_cast<int>(ceil_div(rows, GATE_UP ? 64 : 128));
  p.chunks = static_cast<int>(ceil_div(g.in_features, 128));
  p.bits = w.bits;
  p.w_bytes = 2048 * w.bits;
  if (!encode_map(&p.wmap, CU_TENSOR_MAP_DATA_TYPE_INT32, w.packed, g.words_per_row, w.rows, static_cast<int64_t>(g.words_per_row) * 4, 4 * w.bits,
                  GATE_UP ? 64 : 128, weight_swizzle(w.bits)) ||
      !encode_map(&p.xmap, act_dtype == DQ_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, act, g.in_features, act_rows,
                  static_cast<int64_t>(g.in_features) * 2, 64, kBoxRows, CU_TENSOR_MAP_SWIZZLE_128B)) {
    return fail(DQ_ERR_CUDA, "moe_gemm: a tensor map could not be encoded");
  }
  const bool bf = act_dtype == DQ_BF16, mbf = w.meta_dtype == DQ_BF16;
  const uint32_t front = ring_offset(!bf);
  const int x_bytes = p.n_cap * 256, budget = dev.max_smem_optin - static_cast<int>(front);
  p.x_slots = std::clamp((budget - kGroups * p.w_bytes) / x_bytes, 2, 4);
  p.w_slots = std::clamp((budget - p.x_slots * x_bytes) / p.w_bytes / kGroups * kGroups, kGroups, 12);
  const size_t smem = front + static_cast<size_t>(p.x_slots) * x_bytes + static_cast<size_t>(p.w_slots) * p.w_bytes;
  const auto kernel = bf ? (mbf ? moe_umma_kernel<true, true, GATE_UP> : moe_umma_kernel<true, false, GATE_UP>)
                         : (mbf ? moe_umma_kernel<false, true, GATE_UP> : moe_umma_kernel<false, false, GATE_UP>);
  return launch(kernel, dim3(static_cast<unsigned>(dev.sm_count)), kThreads, smem, stream, "moe_gemm", p);
}

}  // namespace

}  // namespace dq

extern "C" {

int32_t dq_moe_gemm_scratch_bytes(int64_t tokens, int64_t topk, int64_t hidden, int64_t inter, int64_t num_experts, int32_t act_dtype,
                                  int64_t* bytes) {
  DQ_REQUIRE(bytes != nullptr, "moe_gemm_scratch_bytes: null result pointer");
  DQ_REQUIRE(tokens >= 0 && topk > 0 && hidden > 0 && inter > 0 && num_experts > 0 && dq::dtype_ok(act_dtype) && tokens * topk < (1LL << 24),
             "moe_gemm: bad sizes (tokens=%lld topk=%lld hidden=%lld inter=%lld experts=%lld)", static_cast<long long>(tokens),
             static_cast<long long>(topk), static_cast<long long>(hidden), static_cast<long long>(inter), static_cast<long long>(num_experts));
  *bytes = static_cast<int64_t>(dq::layout_of(tokens, topk, hidden, inter, num_experts, dq::dtype_size(act_dtype)).total);
  return DQ_OK;
}

int32_t dq_moe_gemm(const void* x, int32_t x_dtype, int64_t tokens, const int32_t* topk_ids, const float* topk_w, int64_t topk,
                    int64_t first_expert, int64_t num_experts, const dq_weight* gate_up, const dq_weight* down, int64_t hidden, int64_t inter,
                    void* y, int32_t y_dtype, void* scratch, int64_t scratch_bytes, void* stream) {
  int64_t need = 0;
  if (const int32_t rc = dq_moe_gemm_scratch_bytes(tokens, topk, hidden, inter, num_experts, x_dtype, &need)) return rc;
  DQ_REQUIRE(first_expert >= 0 && first_expert < (1LL << 30), "moe_gemm: first_expert=%lld out of range", static_cast<long long>(first_expert));
  DQ_REQUIRE(gate_up != nullptr && down != nullptr, "moe_gemm: null bank descriptor");
  dq_geometry g_gu, g_dn;
  if (const int32_t rc = dq_resolve_geometry("moe_gemm(gate_up)", gate_up, &g_gu)) return rc;
  if (const int32_t rc = dq_resolve_geometry("moe_gemm(down)", down, &g_dn)) return rc;
  DQ_REQUIRE(gate_up->rows == num_experts * 2 * inter && gate_up->in_features == hidden && down->rows == num_experts * hidden &&
                 down->in_features == inter,
             "moe_gemm: the banks must be [experts * 2 * inter, hidden] and [experts * hidden, inter]");
  DQ_REQUIRE(dq::dtype_ok(y_dtype), "moe_gemm: unsupported output dtype tag %d", y_dtype);
  if (tokens == 0) return DQ_OK;
  DQ_REQUIRE(x != nullptr && topk_ids != nullptr && topk_w != nullptr && y != nullptr, "moe_gemm: null pointer");
  DQ_REQUIRE(scratch != nullptr && scratch_bytes >= need && reinterpret_cast<uintptr_t>(scratch) % 256 == 0,
             "moe_gemm: scratch must be 256-byte aligned and at least %lld bytes (dq_moe_gemm_scratch_bytes), got %lld",
             static_cast<long long>(need), static_cast<long long>(scratch_bytes));
  const auto half = [](int32_t t) { return t == DQ_BF16 || t == DQ_F16; };
  const auto rows16 = [](const dq_weight* w) { return reinterpret_cast<uintptr_t>(w->packed) % 16 == 0 && w->words_per_row % 4 == 0; };
  const auto aligned = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  if (!half(x_dtype) || !half(gate_up->meta_dtype) || !half(down->meta_dtype) || gate_up->group_values != 128 || down->group_values != 128 ||
      !rows16(gate_up) || !rows16(down) || !aligned(x) || !aligned(y) || hidden % 8 != 0 || inter % 8 != 0 || num_experts > dq::kMaxExperts ||
      !dq::mma_enabled_for_rows()) {
    return dq::fail(DQ_ERR_UNSUPPORTED,
                    "moe_gemm: this build handles fp16/bf16 activations and metadata, 128-value groups, 16-byte aligned rows and up to %d experts",
                    dq::kMaxExperts);
  }
  const dq::DeviceInfo* dev = dq::device_info();
  if (dev == nullptr) return DQ_ERR_CUDA;
  auto s = static_cast<cudaStream_t>(stream);
  const dq::Layout lay = dq::layout_of(tokens, topk, hidden, inter, num_experts, dq::dtype_size(x_dtype));
  auto* base = static_cast<unsigned char*>(scratch);
  const int assignments = static_cast<int>(tokens * topk), experts = static_cast<int>(num_experts), first = static_cast<int>(first_expert);
  auto* table = reinterpret_cast<dq::RouteTable*>(base + lay.table);
  auto* tiles = reinterpret_cast<int4*>(base + lay.tiles);
  auto* order = reinterpret_cast<int32_t*>(base + lay.order);
  // Columns of a tile (and rows of an activation slot): 64 where hardly an expert has more tokens than
  // that, else 128, so that an expert's weights are decoded once.
  const double mean = static_cast<double>(assignments) / experts;
  const int n_cap = mean + 3.0 * std::sqrt(mean) <= 64.0 ? 64 : dq::kColumns;
  if (const int32_t rc = dq::launch(dq::moe_route_kernel, dim3(1), dq::kRouteThreads, 0, s, "moe_gemm(route)", topk_ids, first, experts,
                                    assignments, n_cap, table, tiles, order)) {
    return rc;
  }
  const unsigned permute_ctas = static_cast<unsigned>(std::min<int64_t>(dq::ceil_div(assignments, 8), static_cast<int64_t>(dev->sm_count) * 8));
  if (const int32_t rc = dq::launch(dq::moe_permute_kernel, dim3(permute_ctas), 256, 0, s, "moe_gemm(permute)", static_cast<const uint4*>(x),
                                    static_cast<const dq::RouteTable*>(table), static_cast<const int32_t*>(order), static_cast<int>(topk),
                                    static_cast<int>(hidden / 8), reinterpret_cast<uint4*>(base + lay.xs))) {
    return rc;
  }
  dq::Params p = {};
  p.table = table;
  p.tiles = tiles;
  p.order = order;
  p.n_cap = n_cap;
  p.give_up = dq::take_fail_next();
  p.report = dev->report;
  p.out = base + lay.h;
  if (const int32_t rc = dq::launch_bank<true>(*gate_up, g_gu, base + lay.xs, x_dtype, assignments, static_cast<int>(inter), p, *dev, s)) return rc;
  p.out = base + lay.d;
  if (const int32_t rc = dq::launch_bank<false>(*down, g_dn, base + lay.h, x_dtype, assignments, static_cast<int>(hidden), p, *dev, s)) return rc;
  const int quads = static_cast<int>(hidden / 4);
  const dim3 combine(static_cast<unsigned>(dq::ceil_div(quads, 256)), static_cast<unsigned>(std::min(tokens, dq::kMaxGridY)));
  if (const int32_t rc = dq::launch(dq::moe_combine_rows_kernel, combine, 256, 0, s, "moe_gemm(combine)",
                                    reinterpret_cast<const float4*>(base + lay.d), topk_w, topk_ids, first, static_cast<int>(tokens),
                                    static_cast<int>(topk), quads, experts, y, y_dtype)) {
    return rc;
  }
  dq::note_kernel("moe_umma_kernel");
  return DQ_OK;
}

}  // extern "C"
