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
//   * four warpgroups (three where weights are split in two operands) decode, 128 values of K in turn:
//     a thread owns one weight row, so its scale and offset are two registers and its packed words one
//     contiguous piece of shared memory; the 16-bit weights go straight to TENSOR MEMORY (tcgen05.st)
//     in the natural order -- not to shared memory, whose bandwidth the activation needs;
//   * warp 1 issues the MMAs (A from tensor memory, B from shared memory), accumulating in tensor
//     memory; two accumulator tiles where they fit, so that the decode of the next tile runs under the
//     epilogue of this one.
// What bounds it: for wide tiles the tensor pipe (n_tile / 2 cycles per 16 values of K) at the clock that
// the power cap leaves, below that the decode's issue slots (14336 x 4096, 4-bit: issue 55 %, integer
// pipe 54 %, tensor 31 % at 65 rows, with 112 of 148 SMs at work; 0.5 us per 128 x 128 values and SM split
// in two operands).  14336 x 4096, 4-bit, at 16 / 128 / 512 / 4096 rows: 21 / 22 / 53 / 427 us (1.13
// PFLOP/s, 79 % of the sustained dense peak; 366 us in bursts too short for the power cap) where dequantize +
// dense took 215 us at the first two and 558 at the last.
//
// Small matrices: the reduction axis is sliced over a thread-block cluster (grid.y), each CTA leaves
// its fp32 tile in its own shared memory and the CTAs of the cluster add a share of the columns
// each, in slice order, over distributed shared memory -- deterministic.
//
// Every wait is bounded (dq_umma.cuh): when one runs out the block's roles stop one after the other, its
// copies and MMAs in flight are drained, its tensor memory is freed, its output is left incomplete and
// the host is told (DeviceInfo::report).
#include <algorithm>
#include <cmath>

#include "dq_gemm_umma.cuh"
#include "dq_gemv.cuh"
#include "dq_umma_pipeline.cuh"

namespace dq {
namespace {

using namespace umma;

constexpr int kJobs = 4;
constexpr int kMaxSlices = 6;
struct Job {
  CUtensorMap wmap;
  Meta meta;
  const void* bias;                    // may be null; element 0 belongs to output column 0 of this job
  int64_t col0;
  int rows, row_tiles, bits;
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
  int x_slabs;                         // slabs of 64 values in an activation slot: 2 (a chunk) or 1
  int slices;
  int give_up;                         // dq_gemm_fail_next
  unsigned int* report;
  uint32_t ring_offset, barrier_offset;
};

constexpr uint32_t kBarrierOffset = 64, kRingOffset = 1024;
static_assert(kBarrierOffset + kBarrierBytes <= kRingOffset, "");

// SPLIT: the weights enter as the sum of two 16-bit operands, so that nothing of their fp32 values is
// lost that a 16-bit output could show (figures: dq_umma_decode.cuh).  Up to DQ_GEMV_CHUNKED_MAX_ROWS activation rows, where the mma.sync
// kernels scale fp32 accumulators and never round a weight; above that the dense path this kernel
// replaces rounds every weight once, and so does this kernel.
template <bool BF16, bool MBF16, bool SPLIT>
__global__ void __launch_bounds__(Roles<SPLIT>::kThreads, 1) gemm_umma_kernel(const __grid_constant__ Params p) {
  constexpr int kGroups = Roles<SPLIT>::kGroups;
  extern __shared__ __align__(1024) unsigned char smem[];
  // control block at the front: failure flag, tensor memory address, barriers
  volatile int* failed = reinterpret_cast<volatile int*>(smem);
  InFlight* left = reinterpret_cast<InFlight*>(smem + 8);
  const uint32_t base = smem_addr(smem);
  const Bars bars = bars_at(base + p.barrier_offset);
  const int x_slabs = SPLIT ? 2 : p.x_slabs;
  const int slab_bytes = p.n_tile * 128, x_bytes = slab_bytes * x_slabs;
  unsigned char* x_ring = smem + p.ring_offset;
  unsigned char* w_ring = x_ring + p.x_slots * x_bytes;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

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

  // groups [g0, g0 + groups_of(job)) hold the values of this share
  const auto first_group = [&](const Job& job) -> int { return (2 * c0) >> job.meta.group_shift; };
  const auto groups_of = [&](const Job& job) -> int {
    return min((2 * c1 - 1) >> job.meta.group_shift, job.meta.num_groups - 1) - first_group(job) + 1;
  };

  if (threadIdx.x == 0) {
    *failed = p.give_up;
    init_bars(bars, p.x_slots, p.w_slots, kGroups, 4 * kGroups);
    tma_prefetch_map(&p.xmap);
  }
  if (warp == 3) tmem_alloc(base + 4, static_cast<uint32_t>(p.tmem_columns));
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + 4);
  const uint32_t d_tmem = tmem + Roles<SPLIT>::kColumns;
  pdl_launch_dependents();

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
        const int count = weights || x_slabs == 2 ? c1 - c0 : (c1 - c0) * 2;
        const int bytes = weights ? 2048 * job.bits : x_bytes;
        for (int i = 0; i < count; ++i, ++issued, at.advance(slots)) {
          const uint32_t slot = at.slot;
          if (!(ok = mbar_wait(empty + slot * 8, at.pass ^ 1, failed))) break;
          mbar_expect(full + slot * 8, static_cast<uint32_t>(bytes));
          if (weights) {
            tma_load_2d(smem_addr(w_ring) + slot * p.w_bytes, &job.wmap, (c0 + i) * 4 * job.bits, local * 128, full + slot * 8);
          } else {
            const uint32_t dst = smem_addr(x_ring) + slot * x_bytes;
            const int x0 = c0 * 128 + i * 64 * x_slabs;
            tma_load_2d(dst, &p.xmap, x0, token0, full + slot * 8);
            if (x_slabs == 2) tma_load_2d(dst + slab_bytes, &p.xmap, x0 + 64, token0, full + slot * 8);
          }
        }
      }
      left->issued[warp] = issued;
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
          uint32_t xs = x_at.slot;
          if (!(ok = mbar_wait(bars.x_full + xs * 8, x_at.pass, failed))) break;
          if (!(ok = mbar_wait(bars.a_full + a_at.slot * 8, a_at.pass, failed))) break;
          fence_after_sync();
          const uint32_t a = tmem + a_at.slot * Roles<SPLIT>::kTileColumns;
          uint32_t slab = smem_addr(x_ring) + xs * x_bytes;
          mma_slab<SPLIT>(d, a, smem_descriptor(slab), idesc, i > 0);
          if (x_slabs == 1) {
            mma_commit(bars.x_empty + xs * 8);
            x_at.advance(static_cast<uint32_t>(p.x_slots));
            xs = x_at.slot;
            if (!(ok = mbar_wait(bars.x_full + xs * 8, x_at.pass, failed))) break;
            slab = smem_addr(x_ring) + xs * x_bytes;
          } else {
            slab += slab_bytes;
          }
          mma_slab<SPLIT>(d, a + 32, smem_descriptor(slab), idesc, true);
          mma_commit(bars.a_empty + a_at.slot * 8);
          a_at.advance(kGroups);
          mma_commit(bars.x_empty + xs * 8);
          x_at.advance(static_cast<uint32_t>(p.x_slots));
        }
        if (ok) mma_commit(bars.d_full + buffer * 8);
      }
      left->mma_lane = lane;
    }
    __syncwarp();
  } else if (warp >= kDecodeWarp0) {
    const int group = (warp - kDecodeWarp0) >> 2;
    const int warp4 = warp & 3;
    const int r = warp4 * 32 + lane;
    const int stages = c1 - c0;
    const WeightRing ring = {w_ring, p.w_slots, p.w_bytes};
    uint32_t stage = 0;
    uint32_t a_pass = 0;
    Cursor w_at, d_at;
    w_at.advance(static_cast<uint32_t>(p.w_slots), static_cast<uint32_t>(group));
    for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x, d_at.advance(static_cast<uint32_t>(p.d_buffers)), stage += stages) {
      int local;
      const Job& job = p.job[job_of(tile % p.row_tiles, local)];
      float power = 1.0f, back = 1.0f;
      if constexpr (kScaledRows<BF16, SPLIT>) {
        const int k = row_power<MBF16>(job.meta, job.bits, job.rows, min(local * 128 + r, job.rows - 1), first_group(job), groups_of(job));
        power = power_of_two(k), back = power_of_two(-k);
      }
      bool ok;
#define DQ_DECODE(B) ok = decode_tile<B, BF16, MBF16, SPLIT>(job.meta, min(local * 128 + r, job.rows - 1), r, power, c0, group, stage, stages, ring, bars, tmem, w_at, a_pass, failed)
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
        if constexpr (kScaledRows<BF16, SPLIT>) {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * back);
        }
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
  if (*failed != 0) {  // (the same for all: every role has stopped)
    drain(*left, bars, p.x_slots, p.w_slots);
    __syncthreads();
  }
  if (p.slices > 1) {
    // One tile per cluster: add the slices' columns, a share of them per CTA.  A warp takes a column, a
    // lane four of its rows, all slices' loads of two columns requested before the first is used (one
    // row and column at a time, slice after slice, two slices took 3 us at 64 columns and 5.6 at 128).
    cluster_sync();
    const int tile = blockIdx.x;
    int local;
    const Job& job = p.job[job_of(tile % p.row_tiles, local)];
    const int per = (p.n_tile + p.slices - 1) / p.slices;
    const int token0 = (tile / p.row_tiles) * p.n_tile;
    const int first = slice * per, last = min(min(first + per, p.n_tile), p.m - token0);
    const int row = local * 128 + lane * 4;
    if (*failed == 0 && row < job.rows) {
      constexpr int kType = BF16 ? DQ_BF16 : DQ_F16, kWarps = Roles<SPLIT>::kThreads / 32;
      float bias[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      if (job.bias != nullptr) {
#pragma unroll
        for (int i = 0; i < 4; ++i) bias[i] = load_f32(job.bias, min(row + i, job.rows - 1), kType);
      }
      const uint32_t red = base + p.ring_offset + lane * 16;
      for (int col0 = first + warp; col0 < last; col0 += 2 * kWarps) {
        float4 part[2][kMaxSlices];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int col = min(col0 + c * kWarps, last - 1);
#pragma unroll
          for (int s = 0; s < kMaxSlices; ++s) {
            part[c][s] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (s < p.slices) part[c][s] = cluster_ld4(red + col * 512, s);
          }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int col = col0 + c * kWarps;
          if (col >= last) break;
          float4 sum = part[c][0];
#pragma unroll
          for (int s = 1; s < kMaxSlices; ++s) {  // in slice order
            sum.x += part[c][s].x, sum.y += part[c][s].y, sum.z += part[c][s].z, sum.w += part[c][s].w;
          }
          unsigned short* dst = static_cast<unsigned short*>(p.out) + static_cast<int64_t>(token0 + col) * p.out_stride + job.col0 + row;
          const uint2 packed = make_uint2(round_pair_to_16(sum.x + bias[0], sum.y + bias[1], kType),
                                          round_pair_to_16(sum.z + bias[2], sum.w + bias[3], kType));
          if (row + 3 < job.rows && (reinterpret_cast<uintptr_t>(dst) & 7) == 0) {
            *reinterpret_cast<uint2*>(dst) = packed;
          } else {
            const uint32_t half[4] = {packed.x & 0xFFFFu, packed.x >> 16, packed.y & 0xFFFFu, packed.y >> 16};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (row + i < job.rows) dst[i] = static_cast<unsigned short>(half[i]);
            }
          }
        }
      }
    }
    cluster_sync();  // nobody leaves while its sums are being read
  }
  if (threadIdx.x == 0 && *failed != 0) report_to_host(p.report, kReportWait);
  fence_after_sync();
  if (warp == 3) tmem_free(tmem, static_cast<uint32_t>(p.tmem_columns));
}

// ---------------------------------------------------------------------------
// Host
// ---------------------------------------------------------------------------

bool geometry_ok(const GemvArgs& a, int bits) {
  const bool x16 = a.x_dtype == DQ_BF16 || a.x_dtype == DQ_F16, meta16 = a.meta_dtype == DQ_BF16 || a.meta_dtype == DQ_F16;
  if (!x16 || !meta16 || a.out_dtype != a.x_dtype || a.in_features % 8 != 0 || group_shift_of(a.group_values) < 0) return false;
  if (a.words_per_group * 32 != a.group_values * bits || a.words_per_row % 4 != 0) return false;
  return reinterpret_cast<uintptr_t>(a.x) % 16 == 0 && reinterpret_cast<uintptr_t>(a.packed) % 16 == 0;
}

// Whether this kernel takes ALL the matrices at once.  Asked before anything is launched: the caller's other paths
// compute every one of them, and a second launch (first_launch_tiles) has to be one that is taken.
bool jobs_ok(const GemvArgs* args, const int* bits, int count) {
  if (count < 1 || count > kJobs) return false;
  const GemvArgs& a = args[0];
  for (int i = 0; i < count; ++i) {
    const GemvArgs& b = args[i];
    if (!geometry_ok(b, bits[i]) || b.x != a.x || b.m != a.m || b.out != a.out || b.out_stride != a.out_stride ||
        b.in_features != a.in_features || b.meta_dtype != a.meta_dtype || b.rows < 1) {
      return false;
    }
  }
  return true;
}

struct Shape {
  int n_tile, token_tiles, slices;
  double cost;                         // us, estimated
};

// Token tiles and slices of the reduction axis with the least estimated time (us, fitted to measurements
// at 16..1024 rows on matrices of 128 x 128 to 14336 x 4096): waves of CTAs times the chunks of one, each
// bound by the decode or by the tensor pipe, a start and an end, and what a cluster costs -- the sums
// that cross it and, the more of the chip it fills, its launch.  The slices of all tiles are resident at
// once or there are none: a second wave of clusters costs more than it gives (4096 x 14336, 16 rows: 22
// us with 4 slices, 38 with 8), and clusters of eight pack badly into the GPCs (1152 x 7936, 128 rows: 14
// us with 6 slices, 21 with 8).
Shape pick_shape(int m, int row_tiles, int chunks, bool split, int sm_count) {
  Shape best = {};
  best.cost = 1e30;
  const int min_tiles = static_cast<int>(ceil_div(m, 256));
  for (int tt = min_tiles; tt <= min_tiles + (m > 256 ? 2 : 0); ++tt) {  // (up to 256 rows a second tile only decodes twice)
    const int n = static_cast<int>(ceil_div(ceil_div(m, tt), 16) * 16);
    if (n * (tt - 1) >= m) continue;
    const double again = 1.0 + 0.08 * (tt - min_tiles);
    const double chunk = (split ? 0.49 + 0.001 * n : std::max(0.42, 0.22 + 0.0022 * n)) * again;
    for (int s = 1; s <= kMaxSlices && s <= chunks; ++s) {
      const int64_t ctas = static_cast<int64_t>(row_tiles) * tt * s;
      const int resident = s <= 2 ? sm_count : s <= 4 ? sm_count - 16 : sm_count - 24;
      if (s > 1 && ctas > resident) break;
      const double waves = std::ceil(static_cast<double>(ctas) / sm_count);
      const double hidden = s == 1 && n <= 128 ? 0.0 : 0.005 * n;  // an epilogue that the next tile does not cover
      const double cluster = s > 1 ? 1.0 + 0.004 * n * s + 1.1 * (s - 1) * static_cast<double>(ctas) / sm_count : 0.0;
      const double cost = waves * (static_cast<double>(ceil_div(chunks, s)) * chunk + hidden) + cluster + 2.2 + 0.01 * n;
      if (cost < best.cost) best = {n, tt, s, cost};
    }
  }
  return best;
}

// The row tiles that a launch of its own should have, the rest in a second one; all of them: one launch.
//
// Up to 256 activation rows a wave is bound by the decode, and a last wave of a few tiles costs as much as a full
// one.  So the first launch gets whole waves and the second, whose tiles are few, slices the reduction axis over
// clusters: 4-bit 20480 x 4096 (160 row tiles) at 16 / 64 / 128 rows 37.2 / 41.8 / 41.9 -> 29.9 / 34.7 / 34.0 us; of 60
// matrices of 149 to 300 row tiles 12 change and gain 2 to 31 %, none loses.  With more token tiles the waves run into
// one another and the second launch, which waits for the first to end, loses up to 7 % (1500 rows, 5120 x 5120:
// 61 -> 65 us).
int first_launch_tiles(int m, int row_tiles, int chunks, bool split, int sm_count) {
  const int tiles = row_tiles / sm_count * sm_count;
  if (m > 256 || tiles == 0 || tiles == row_tiles) return row_tiles;
  const auto cost = [&](int t) -> double { return pick_shape(m, t, chunks, split, sm_count).cost; };
  return cost(tiles) + cost(row_tiles - tiles) < 0.95 * cost(row_tiles) ? tiles : row_tiles;
}

int32_t launch_jobs(const GemvArgs* args, const int* bits, int count, const DeviceInfo* dev, cudaStream_t stream, bool* taken);

}  // namespace

int32_t launch_gemm_umma(const GemvArgs* args, const int* bits, int count, cudaStream_t stream, bool* taken) {
  *taken = false;
  const DeviceInfo* dev = device_info();
  if (dev == nullptr) return DQ_ERR_CUDA;
  if (!jobs_ok(args, bits, count)) return DQ_OK;
  int row_tiles = 0;
  for (int i = 0; i < count; ++i) row_tiles += static_cast<int>(ceil_div(args[i].rows, 128));
  const int first = tuning_int("DQ_B200_UMMA_LAST_WAVE", 1) == 0
                        ? row_tiles
                        : first_launch_tiles(args[0].m, row_tiles, static_cast<int>(ceil_div(args[0].in_features, 128)), args[0].m <= DQ_GEMV_CHUNKED_MAX_ROWS, dev->sm_count);
  if (first >= row_tiles) return launch_jobs(args, bits, count, dev, stream, taken);
  GemvArgs part[2][kJobs];
  int part_bits[2][kJobs], parts[2] = {0, 0}, tile0 = 0;
  for (int i = 0; i < count; ++i) {
    const int tiles = static_cast<int>(ceil_div(args[i].rows, 128)), cut = std::clamp(first - tile0, 0, tiles) * 128;  // rows of the first part
    tile0 += tiles;
    for (int k = 0; k < 2; ++k) {
      const int64_t row0 = k == 0 ? 0 : cut;
      const int rows = k == 0 ? std::min(cut, args[i].rows) : args[i].rows - cut;
      if (rows <= 0) continue;
      GemvArgs& b = part[k][parts[k]];
      b = args[i];
      b.rows = rows;
      b.packed += row0 * b.words_per_row;
      b.scales = static_cast<const unsigned short*>(b.scales) + row0 * b.num_groups;
      if (b.offsets != nullptr) b.offsets = static_cast<const unsigned short*>(b.offsets) + row0 * b.num_groups;
      b.out_col0 += row0;
      part_bits[k][parts[k]++] = bits[i];
    }
  }
  if (const int32_t rc = launch_jobs(part[0], part_bits[0], parts[0], dev, stream, taken)) return rc;
  if (!*taken) return DQ_OK;
  if (const int32_t rc = launch_jobs(part[1], part_bits[1], parts[1], dev, stream, taken)) return rc;
  return *taken ? DQ_OK : fail(DQ_ERR_CUDA, "gemm: the second launch of a matrix was refused");
}

namespace {

int32_t launch_jobs(const GemvArgs* args, const int* bits, int count, const DeviceInfo* dev, cudaStream_t stream, bool* taken) {
  *taken = false;
  Params p = {};
  const GemvArgs& a = args[0];
  int w_bytes = 0;
  for (int i = 0; i < count; ++i) {
    const GemvArgs& b = args[i];
    Job& job = p.job[i];
    if (!encode_map(&job.wmap, CU_TENSOR_MAP_DATA_TYPE_INT32, b.packed, b.words_per_row, b.rows, static_cast<int64_t>(b.words_per_row) * 4,
                    4 * bits[i], 128, weight_swizzle(bits[i]))) {
      return DQ_OK;
    }
    job.meta = {b.scales, b.offsets, b.num_groups, group_shift_of(b.group_values)};
    job.col0 = b.out_col0;
    job.bias = b.bias == nullptr ? nullptr : static_cast<const unsigned short*>(b.bias) + b.out_col0;
    job.rows = b.rows;
    job.row_tiles = static_cast<int>(ceil_div(b.rows, 128));
    job.bits = bits[i];
    p.row_tiles += job.row_tiles;
    w_bytes = std::max(w_bytes, 2048 * bits[i]);
  }
  p.jobs = count;
  p.m = a.m;
  p.out = a.out;
  p.out_stride = a.out_stride;
  p.chunks = static_cast<int>(ceil_div(a.in_features, 128));
  Shape shape = pick_shape(a.m, p.row_tiles, p.chunks, a.m <= DQ_GEMV_CHUNKED_MAX_ROWS, dev->sm_count);
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
  // Rings: activation slots of 128 values (up to 6), then weight slots -- a multiple of the warpgroups, so
  // that a slot always belongs to the same one (its barrier then cannot be two passes behind).  Where the
  // activation of three chunks does not fit (8 bits, from 224 columns on) the slots are of 64 values: two
  // of 128 leave a copy only one chunk's time (8-bit 17280 x 1152 at 512 / 4096 rows 26.8 / 186 us against
  // 25.7 / 175, 4096 x 4096 at 4096 rows 128 against 111).  Elsewhere the second wait per chunk only
  // costs (14336 x 4096, 4-bit, 65 rows: 19.4 us against 17.4).
  p.w_bytes = w_bytes;
  const int budget = dev->max_smem_optin - static_cast<int>(kRingOffset);
  const int x_room = (budget - kMaxGroups * w_bytes) / (p.n_tile * 128);  // slabs of 64 values
  p.x_slabs = x_room < 6 ? 1 : 2;
  p.x_slots = std::min(x_room / p.x_slabs, 6);
  const int x_bytes = p.n_tile * 128 * p.x_slabs;
  const int groups = split ? Roles<true>::kGroups : Roles<false>::kGroups;
  p.w_slots = std::clamp((budget - p.x_slots * x_bytes) / w_bytes / groups * groups, groups, 12);
  p.give_up = take_fail_next();
  p.report = dev->report;
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

}  // namespace
}  // namespace dq

namespace dq {
namespace {
thread_local int t_fail_next = 0;
}
int take_fail_next() { return t_fail_next > 0 ? (--t_fail_next, 1) : 0; }
}  // namespace dq

extern "C" int32_t dq_gemm_fail_next(int32_t calls) {
  dq::t_fail_next = std::max(calls, 0);
  return DQ_OK;
}
