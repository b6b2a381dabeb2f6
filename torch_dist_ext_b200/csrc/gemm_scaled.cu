// Block-scaled e4m3 GEMM for sm_100a, any token count:
//   D[x, y] = sum_kb x_scale[x, kb] * y_scale[y / 128, kb] * (sum_{k in block kb} X[x, k] * Y[y, k])
// X: activations (one fp32 scale per row and 128-wide K block), Y: weights (one per 128 x 128 block), both K-major.
//
// What bounds it. Every 128-wide K block has to leave the tensor core and be promoted, acc += partial * scale, because
// the scales are arbitrary fp32 numbers. The activations sit on the 128-row (TMEM lane) side and 256 weight rows on the
// narrow side, so a thread's 128 columns share ONE scale per K block (its row's times its weight block's): a promotion
// is one multiply-add per value. With the weights on the lanes, as the decode kernel of gemm_tcgen05.cu has
// it, every value needs a scale product and a shuffle of its own, and a tile is 64 columns wide; that kernel ran
// 2048 x 28672 x 8192 at 484 TFLOP/s.
//
// kCtas = 2 (more than 128 rows): a CTA pair computes 256 x 256 tiles with tcgen05.mma.cta_group::2, each CTA staging
// its own 128 rows of X and half of the Y tile; kCtas = 1 (decode): 128 x 256 tiles, the tile's 256 weight rows
// streamed once. The 256 columns are two halves with a pipeline of their own each: warp 0 copies (TMA), warp 1 + h issues
// the MMAs of half h, warps 4 + 4 h .. 7 + 4 h promote it: warp w owns TMEM lanes 32 * (w % 4), 128 fp32 sums per thread
// in registers. Each half has two partial buffers of 128 columns (together all of the tensor memory), so block i is
// promoted while block i + 1 multiplies; a promoting warp multiplies 32 columns in while the next 32 travel, hands the
// buffer back before the last 32 and looks for the next block's completion before it multiplies those. What bounds it now
// is that warp's chain, about 1000 cycles per K block against 512 of tensor work (measured with clock stamps; without
// the multiply-adds 850, without the tensor-memory reads 720). 16 promoting warps of 64 columns spilled and were slower.
// A warp whose 32 rows lie beyond X only hands the buffers on. Warp 3 stages the products of row and weight scales in
// shared memory, four K blocks at a time (fetched by the promoting threads themselves, each load touched 32 lines).
//
// The loops of the copying and issuing warps are walked by the whole warp and only the asynchronous instructions sit
// inside `if (elect_one())`: with one thread in the loop each of them cost 70-90 cycles (operands moved to uniform
// registers in front of every instruction): 2048 x 28672 x 8192 went from 895 to 547 us with that change alone, and with
// the rest above to 499 us in isolation (575 in a loop of changing operands, 1690 TFLOP/s), against 1900 to 1970 before.
//
// Work split. Pairs take whole tiles in full rounds; the tiles of a last, partly filled round are cut along K into `parts`
// pieces, one pair each. A piece leaves its sums in a scratch slice of its own and whoever arrives last at the tile (an
// atomic counter, no waiting) adds the slices in the order of the pieces. At decode sizes a tile's pieces are the CTAs of
// one cluster: they leave their sums in shared memory, and after a cluster barrier each adds up and stores its part of
// the columns, out of the others' shared memory: no scratch, no counters, and every CTA takes part (with slices in global
// memory 64 x 7168 x 8192 spent 9 of 20 us on the meeting). Either way the result does not depend on who is last.
//
// Every wait is bounded; a wait that runs out records a status word, raises the abort flag (of both CTAs) and falls
// through to the common exit. The reference (xytpai/torch_dist_ext) has no GEMM.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <array>
#include <map>
#include <mutex>
#include <string>
#include "tdx/comm.h"
#include "tdx/gemm.h"
#include "tdx/gemm_core.cuh"
#include "tdx/launch.h"
#include "tdx/ptx.cuh"
#include "tdx/tc.cuh"
#include "tdx/tma_host.h"

namespace tdx {
namespace {

using gemm_core::store_chunk;

constexpr int kPromoteWarps = 8;
constexpr int kFirstPromoteWarp = 4;              // warps 0-3: copies, MMAs of either column half, scales
constexpr int kThreads = (kFirstPromoteWarp + kPromoteWarps) * 32;
// 384 threads start with 168 registers each; a promoting thread holds 128 sums and up to 64 values on their way, so the
// role warps hand registers over: 128 x 56 + 256 x 216 = 62464 of the launch's 384 x 168 = 64512.
constexpr int kRoleRegs = 56, kPromoteRegs = 216;
constexpr int kRows = 128;                        // X rows per CTA (TMEM lanes)
constexpr int kCols = 256;                        // Y rows of a tile (MMA N)
constexpr int kHalf = 128;                        // columns of one MMA pipeline = one weight scale block
constexpr int kXBytes = kRows * 128;
constexpr uint32_t kTmemCols = 2 * kCols;
constexpr uint32_t kWaitLimit = 1u << 22;
constexpr size_t kSliceFloats = (size_t)kRows * kCols;   // partial sums of one CTA
constexpr int kSumPitch = gemm_core::kSumPitch<kCols>;                 // decode: row pitch of the sums in shared memory, in 16-byte quads
// Scale products: a ring of 16 K blocks, handed over in groups of four, [K block][half][row]; a block's pitch is padded by
// eight floats so that the writing lanes (eight rows x four blocks) hit distinct banks.
constexpr int kGroup = 4;
constexpr int kGroups = 4;
constexpr int kScalePitch = 2 * kRows + 8;
constexpr int kScaleBytes = kGroup * kGroups * kScalePitch * 4;

template <int kCtas>
struct Shape {
  static constexpr int kHalfRows = kHalf / kCtas;        // Y rows of a column half staged by one CTA
  static constexpr int kYBytes = 2 * kHalfRows * 128;
  static constexpr int kStageBytes = kXBytes + kYBytes;  // 48 KB alone, 32 KB in a pair
  static constexpr int kStages = kCtas == 2 ? 6 : 4;
  static constexpr int kBarrierOffset = kStages * kStageBytes;
  static constexpr int kScaleOffset = kBarrierOffset + 1024;
  static constexpr int kSmem = kScaleOffset + kScaleBytes + 1024 /* alignment slack */;
  static_assert(kSmem <= 227 * 1024, "shared memory of one CTA");
  static_assert(kRows * kSumPitch * 16 <= kBarrierOffset, "the sums of a decode tile take the ring's place");
};

struct ScaledArgs {
  int x_rows, y_rows, kblocks;
  int tiles_x, tiles_y;
  int full_rounds;         // tiles worker, worker + workers, ... for this many rounds (0 at decode sizes with parts > 1)
  int parts;               // pieces per remaining tile
  int per;                 // K blocks per piece
  float* ws;               // pairs: [worker][CTA of the pair] slices of [64 column quads][128 rows][4] fp32
  uint32_t* counters;      // pairs: [remaining tile][CTA of the pair], zero on entry and on exit
  const float* x_scale;    // [x_rows, kblocks]
  const float* y_scale;    // [ceil(y_rows / 128), kblocks]
  void* out;
  int64_t sx, sy;
  int out_dtype;
  int whole_sectors;       // 16-bit output whose rows and base are 32-byte aligned: stored a sector per lane
  uint32_t idesc;
  uint32_t* status;
};

// The n-th piece of work of `worker`: the K blocks [kb0, kb1) of a tile. Every role of both CTAs walks the same sequence.
struct Work {
  int tile, kb0, kb1;
};
__device__ __forceinline__ bool next_work(const ScaledArgs& a, int worker, int workers, int n, Work* w) {
  const int ntiles = a.tiles_x * a.tiles_y;
  if (n < a.full_rounds || a.parts == 1) {
    const int t = worker + n * workers;
    *w = Work{t, 0, a.kblocks};
    return t < ntiles;
  }
  const int t = a.full_rounds * workers + worker / a.parts, kb0 = worker % a.parts * a.per;
  *w = Work{t, kb0, min(a.kblocks, kb0 + a.per)};
  return n == a.full_rounds && t < ntiles;
}
// The K blocks of a worker, counted through all its work: how many there are, and where the i-th one lies.
__device__ __forceinline__ int block_count(const ScaledArgs& a, int worker, int workers) {
  const int ntiles = a.tiles_x * a.tiles_y;
  if (a.parts == 1) return worker < ntiles ? ((ntiles - 1 - worker) / workers + 1) * a.kblocks : 0;
  Work w;
  const bool piece = next_work(a, worker, workers, a.full_rounds, &w);
  return a.full_rounds * a.kblocks + (piece ? w.kb1 - w.kb0 : 0);
}
__device__ __forceinline__ void block_at(const ScaledArgs& a, int worker, int workers, int i, int* tile, int* kb) {
  const int n = i / a.kblocks;
  Work w;
  next_work(a, worker, workers, min(n, a.parts == 1 ? n : a.full_rounds), &w);
  *tile = w.tile;
  *kb = w.kb0 + i - n * a.kblocks;
}

// acc += v * s, kept where it is written: between the request of the next values and the wait for them.
__device__ __forceinline__ void multiply_add(float& acc, uint32_t v, float s) {
  asm volatile("fma.rn.f32 %0, %1, %2, %0;" : "+f"(acc) : "f"(__uint_as_float(v)), "f"(s));
}

// 16 columns of a row as 16-bit values: one 32-byte store, a whole sector of memory.
__device__ __forceinline__ void store_sector(void* dst, const uint32_t (&w)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]),
               "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}

template <int kCtas>
__global__ void __launch_bounds__(kThreads, 1)
gemm_scaled_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_y, const ScaledArgs a) {
  using S = Shape<kCtas>;
  constexpr int kStages = S::kStages;
  // identical carve-up in both CTAs of a pair: descriptors, barriers and the TMEM slot sit at the same offsets
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + S::kBarrierOffset);   // used in the leader
  uint64_t* empty = full + kStages;          // one per CTA: both halves' MMAs have read the stage
  uint64_t* part_full = empty + kStages;     // [half][2 buffers], one per CTA
  uint64_t* part_empty = part_full + 4;      // [half][2 buffers], used in the leader
  uint64_t* scale_full = part_empty + 4;     // [4]
  uint64_t* scale_empty = scale_full + kGroups;
  float* scale_ring = reinterpret_cast<float*>(smem + S::kScaleOffset);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(scale_empty + kGroups);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  uint32_t* last_flag = tmem_slot + 2;

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint32_t rank = kCtas == 2 ? tc::cluster_ctarank() : 0u;      // 0: leader
  const uint32_t other = rank ^ 1u;
  const int worker = kCtas == 2 ? blockIdx.x >> 1 : blockIdx.x;
  const int workers = kCtas == 2 ? gridDim.x >> 1 : gridDim.x;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 2);
    }
    for (int i = 0; i < 4; ++i) {
      tc::mbar_init(&part_full[i], 1);
      tc::mbar_init(&part_empty[i], kPromoteWarps / 2 * kCtas);
    }
    for (int i = 0; i < kGroups; ++i) {
      tc::mbar_init(&scale_full[i], 32);
      tc::mbar_init(&scale_empty[i], kPromoteWarps);
    }
    *abort_flag = 0;
    tc::fence_barrier_init();
    tc::tma_prefetch_desc(&map_x);
    tc::tma_prefetch_desc(&map_y);
  }
  __syncthreads();
  if constexpr (kCtas == 2) {
    tc::cluster_arrive();
    tc::cluster_wait();        // both CTAs' barriers exist before anyone arrives on them remotely
  }
  if (warp == 1) {
    if constexpr (kCtas == 2) {
      tc::tmem_alloc_pair(tmem_slot, kTmemCols);
      tc::tmem_relinquish_pair();
    } else {
      tc::tmem_alloc(tmem_slot, kTmemCols);
      tc::tmem_relinquish();
    }
  }
  tc::fence_before_thread_sync();
  __syncthreads();
  tc::fence_after_thread_sync();
  const uint32_t tmem_base = *tmem_slot;

  const int blocks = block_count(a, worker, workers);   // the same in both CTAs of a pair

  // a role that gives up tells the whole pair, so that the other roles stop early too
  auto fail = [&]() {
    *abort_flag = 1;
    if constexpr (kCtas == 2)
      tc::st_cluster_u32(tc::map_to_cta(tc::smem_u32(const_cast<uint32_t*>(abort_flag)), other), 1u);
    if (a.status) atomicExch(a.status, (uint32_t)kTimeoutGemmPipeline);
  };

  if (warp < kFirstPromoteWarp) {
    tc::registers_down<kRoleRegs>();
    if (warp == 0 && blocks > 0) {
      // ---- producer (both CTAs of a pair): own X rows and own part of the Y rows, bytes credited to the leader ----
      const uint32_t bar0 = kCtas == 2 ? tc::map_to_cta(tc::smem_u32(&full[0]), 0) : tc::smem_u32(&full[0]);
      auto load = [&](const CUtensorMap* map, uint32_t dst, uint32_t s, int kb, int row) {
        if constexpr (kCtas == 2) tc::tma_load_2d_pair(dst, map, bar0 + s * 8u, kb * 128, row);
        else tc::tma_load_2d(smem + (dst - tc::smem_u32(smem)), map, &full[s], kb * 128, row);
      };
      const uint32_t ring = tc::smem_u32(smem);
      auto load_y = [&](uint32_t s, int kb, int row) {   // this CTA's rows of either column half
        load(&map_y, ring + s * S::kStageBytes + kXBytes, s, kb, row);
        load(&map_y, ring + s * S::kStageBytes + kXBytes + S::kHalfRows * 128, s, kb, row + kHalf);
      };
      int tile, kb;
      auto load_x = [&](uint32_t s) {
        load(&map_x, ring + s * S::kStageBytes, s, kb, (tile % a.tiles_x) * (kRows * kCtas) + (int)rank * kRows);
      };
      auto load_weights = [&](uint32_t s) { load_y(s, kb, (tile / a.tiles_x) * kCols + (int)rank * S::kHalfRows); };
      // the weights are written by no kernel: their first ring is requested before the previous kernel of the stream
      // has finished, the activations after it
      const int ahead = min(kStages, blocks);
      if (tc::elect_one()) {
        for (int i = 0; i < ahead; ++i) {
          block_at(a, worker, workers, i, &tile, &kb);
          if (rank == 0) tc::mbar_arrive_expect_tx(&full[i], kCtas * S::kStageBytes);
          load_weights(i);
        }
      }
      __syncwarp();
      ptx::pdl_wait();
      if (tc::elect_one()) {
        for (int i = 0; i < ahead; ++i) {
          block_at(a, worker, workers, i, &tile, &kb);
          load_x(i);
        }
      }
      __syncwarp();
      ptx::pdl_launch_dependents();
      bool ok = true;
      for (int it = ahead; it < blocks; ++it) {
        const uint32_t s = it % kStages;
        block_at(a, worker, workers, it, &tile, &kb);
        ok = tc::mbar_wait_warp(&empty[s], ((it / kStages) - 1) & 1, kWaitLimit, abort_flag);
        if (!ok) break;
        if (tc::elect_one()) {
          if (rank == 0) tc::mbar_arrive_expect_tx(&full[s], kCtas * S::kStageBytes);
          load_x(s);
          load_weights(s);
        }
        __syncwarp();
      }
      if (!ok) fail();
    } else if (warp <= 2 && rank == 0) {
      // ---- MMA issue (leader; warp 1: columns 0-127, warp 2: columns 128-255) ----
      const uint32_t half = warp - 1;
      ptx::pdl_wait();         // a poll-counted wait must not begin while an earlier kernel may still run for seconds
      bool ok = true;
      for (int it = 0; it < blocks; ++it) {
        const uint32_t s = it % kStages, buf = it & 1;
        // the operands first: they are there long before the partial buffer is handed back
        ok = tc::mbar_wait_warp(&full[s], (it / kStages) & 1, kWaitLimit, abort_flag) &&
             (it < 2 || tc::mbar_wait_warp(&part_empty[half * 2 + buf], ((it >> 1) - 1) & 1, kWaitLimit, abort_flag));
        if (!ok) break;
        tc::fence_after_thread_sync();
        const uint32_t xa = tc::smem_u32(smem + s * S::kStageBytes);
        const uint64_t dx = tc::make_smem_desc_sw128(xa);
        const uint64_t dy = tc::make_smem_desc_sw128(xa + kXBytes + half * (S::kHalfRows * 128));
        const uint32_t dst = tmem_base + buf * kCols + half * kHalf;
        if (tc::elect_one()) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {   // 32 bytes of K per instruction, stepped inside the swizzle span
            if constexpr (kCtas == 2) tc::umma_pair<true>(dst, dx + (uint64_t)(k * 2), dy + (uint64_t)(k * 2), a.idesc, k > 0 ? 1u : 0u);
            else tc::umma<true>(dst, dx + (uint64_t)(k * 2), dy + (uint64_t)(k * 2), a.idesc, k > 0 ? 1u : 0u);
          }
          if constexpr (kCtas == 2) {
            tc::umma_commit_both(&part_full[half * 2 + buf], 3);
            tc::umma_commit_both(&empty[s], 3);
          } else {
            tc::umma_commit(&part_full[half * 2 + buf]);
            tc::umma_commit(&empty[s]);
          }
        }
        __syncwarp();
      }
      if (!ok) fail();
    } else if (warp == 3) {
      // ---- scale products of this CTA's rows and both weight blocks, four K blocks at a time: lane = (row, block) ----
      ptx::pdl_wait();
      const int r = lane >> 2, k = lane & 3;
      const int last_block = (a.y_rows - 1) / 128;
      bool ok = true;
      for (int i0 = 0; i0 < blocks; i0 += kGroup) {
        const uint32_t group = i0 / kGroup;
        int tile, kb;
        block_at(a, worker, workers, min(i0 + k, blocks - 1), &tile, &kb);
        const float* x_at = a.x_scale + kb;
        const int row = (tile % a.tiles_x) * (kRows * kCtas) + (int)rank * kRows + r;
        float xs[kRows / 8];
#pragma unroll
        for (int i = 0; i < kRows / 8; ++i) xs[i] = __ldg(x_at + (int64_t)min(row + i * 8, a.x_rows - 1) * a.kblocks);
        const int block = (tile / a.tiles_x) * 2;
        const float lo = __ldg(a.y_scale + (int64_t)block * a.kblocks + kb);
        const float hi = __ldg(a.y_scale + (int64_t)min(block + 1, last_block) * a.kblocks + kb);
        ok = group < kGroups || tc::mbar_wait_warp(&scale_empty[group % kGroups], ((group / kGroups) - 1) & 1, kWaitLimit, abort_flag);
        if (!ok) break;
        float* dst = scale_ring + ((i0 + k) % (kGroup * kGroups)) * kScalePitch + r;
#pragma unroll
        for (int i = 0; i < kRows / 8; ++i) {
          dst[i * 8] = xs[i] * lo;
          dst[kRows + i * 8] = xs[i] * hi;
        }
        tc::mbar_arrive(&scale_full[group % kGroups]);
      }
      if (!ok) fail();
    }
  } else {
    // ---- promotion (warps 4..11 of every CTA) ----
    tc::registers_up<kPromoteRegs>();
    ptx::pdl_wait();           // scales, scratch and output belong to the stream's order
    const int q = warp & 3, half = (warp - kFirstPromoteWarp) >> 2;
    const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(half * kHalf);
    const uint32_t leader_empty = kCtas == 2 ? tc::map_to_cta(tc::smem_u32(&part_empty[half * 2]), 0) : 0u;
    const int row_in_cta = q * 32 + lane;
    const float* my_scales = scale_ring + half * kRows + row_in_cta;
    // This warp has read its part of a partial buffer. Nothing but tensor-memory reads that have completed goes before
    // it, so the arrival at the leader of a pair needs no release of ordinary memory at cluster scope (which took longer
    // than a K block).
    auto release = [&](uint32_t buf) {
      __syncwarp();
      if (tc::elect_one()) {
        if (kCtas == 1 || rank == 0) tc::mbar_arrive(&part_empty[half * 2 + buf]);
        else tc::mbar_arrive_cluster_relaxed(leader_empty + buf * 8u);
      }
    };
    uint32_t it = 0;
    bool ready = false;        // the next block's partial product has been seen to be complete
    // A warp whose wait ran out leaves the loop and still attends the meeting of its worker's piece, behind the loop: the
    // barriers count all eight warps, and the other column half may have had its last block. (Walking on inside the loop
    // instead cost it 2 %: 2048 x 28672 x 8192 577 / 589 us.)
    bool lost = false;
    Work w;
    for (int n = 0; next_work(a, worker, workers, n, &w); ++n) {
      const int tile_row = (w.tile % a.tiles_x) * (kRows * kCtas) + (int)rank * kRows + q * 32;
      const int x = tile_row + lane;
      const int y0 = (w.tile / a.tiles_x) * kCols + half * kHalf;
      const bool live = tile_row < a.x_rows && y0 < a.y_rows;       // the same for the whole warp
      float acc[kHalf];
#pragma unroll
      for (int j = 0; j < kHalf; ++j) acc[j] = 0.f;
      bool ok = true;
      const uint32_t end = it + (uint32_t)(w.kb1 - w.kb0);
      for (; it != end; ++it) {
        // the warp leaves the loop as a whole (tcgen05.ld is a warp-wide instruction)
        if (it % kGroup == 0)
          ok = tc::mbar_wait_warp(&scale_full[(it / kGroup) % kGroups], (it / (kGroup * kGroups)) & 1, kWaitLimit, abort_flag);
        if (!ready) ok = ok && tc::mbar_wait_warp(&part_full[half * 2 + (it & 1)], (it >> 1) & 1, kWaitLimit, abort_flag);
        if (!ok) break;
        tc::fence_after_thread_sync();
        const float sc = my_scales[(it % (kGroup * kGroups)) * kScalePitch];
        if (live) {
          // 32 columns are multiplied in while the next 32 travel
          const uint32_t src = taddr + (it & 1) * kCols;
          uint32_t v[2][32];
          tc::tmem_ld_32_start(src, v[0]);
#pragma unroll
          for (int c = 0; c < kHalf / 32; ++c) {
            tc::tmem_ld_wait_32(v[c & 1]);
            if (c + 1 < kHalf / 32) {
              tc::tmem_ld_32_start(src + (c + 1) * 32, v[(c + 1) & 1]);
            } else {                       // every value is in registers: the buffer may be multiplied into again
              tc::fence_before_thread_sync();
              release(it & 1);
              ready = __all_sync(0xffffffffu, tc::mbar_test(&part_full[half * 2 + ((it + 1) & 1)], ((it + 1) >> 1) & 1));
            }
#pragma unroll
            for (int j = 0; j < 32; ++j) multiply_add(acc[c * 32 + j], v[c & 1][j], sc);
          }
        } else {
          release(it & 1);
          ready = false;
        }
        if (it % kGroup == kGroup - 1) {   // the group's products have been read
          __syncwarp();
          if (tc::elect_one()) tc::mbar_arrive(&scale_empty[(it / kGroup) % kGroups]);
        }
      }
      if (!ok) {
        lost = true;
        break;
      }
      if (kCtas == 1 && a.parts > 1) {
        // the meeting in the cluster, below: the sums go to shared memory once every MMA of this CTA has read its stages
        tc::named_barrier_sync(1, kPromoteWarps * 32);
        if (live) {
          float4* mine = reinterpret_cast<float4*>(smem) + row_in_cta * kSumPitch + half * (kHalf / 4);
#pragma unroll
          for (int j = 0; j < kHalf / 4; ++j) mine[j] = make_float4(acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]);
        }
        break;
      }
      if (kCtas == 2 && n == a.full_rounds && a.parts > 1) {
        // a piece of a tile: leave the sums in this worker's slice (a warp's lanes write 512 consecutive bytes)
        const size_t column = ((size_t)half * (kHalf / 4) * kRows + row_in_cta) * 4;
        if (live) {
          float* mine = a.ws + ((size_t)worker * kCtas + rank) * kSliceFloats + column;
#pragma unroll
          for (int j = 0; j < kHalf / 4; ++j)
            __stcg(reinterpret_cast<float4*>(mine + (size_t)j * kRows * 4), make_float4(acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]));
        }
        __threadfence();
        tc::named_barrier_sync(1, kPromoteWarps * 32);
        uint32_t* counter = a.counters + (size_t)(w.tile - a.full_rounds * workers) * kCtas + rank;
        if (threadIdx.x == kFirstPromoteWarp * 32) {
          // an aborted piece is not counted: nobody adds the tile up, and the status says so
          *last_flag = !*abort_flag && atomicAdd(counter, 1u) == (uint32_t)a.parts - 1u ? 1u : 0u;
        }
        tc::named_barrier_sync(1, kPromoteWarps * 32);
        if (!*last_flag) break;
        __threadfence();
        if (threadIdx.x == kFirstPromoteWarp * 32) *counter = 0;
        if (live) {
#pragma unroll
          for (int j = 0; j < kHalf; ++j) acc[j] = 0.f;
          const int first = worker - worker % a.parts;
          for (int piece = first; piece < first + a.parts; ++piece) {
            const float* src = a.ws + ((size_t)piece * kCtas + rank) * kSliceFloats + column;
#pragma unroll
            for (int j0 = 0; j0 < kHalf / 4; j0 += 16) {     // 16 loads in flight before the first is used
              float4 in[16];
#pragma unroll
              for (int j = 0; j < 16; ++j) in[j] = __ldcg(reinterpret_cast<const float4*>(src + (size_t)(j0 + j) * kRows * 4));
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                acc[4 * (j0 + j)] += in[j].x;
                acc[4 * (j0 + j) + 1] += in[j].y;
                acc[4 * (j0 + j) + 2] += in[j].z;
                acc[4 * (j0 + j) + 3] += in[j].w;
              }
            }
          }
        }
      }
      if (live) {
        if (a.whole_sectors && y0 + kHalf <= a.y_rows) {
          if (x < a.x_rows) {
            char* dst = static_cast<char*>(a.out) + ((int64_t)x * a.sx + y0) * 2;
#pragma unroll
            for (int c = 0; c < kHalf; c += 16) {
              uint32_t o[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) o[j] = gemm_core::pack2(a.out_dtype, acc[c + 2 * j], acc[c + 2 * j + 1]);
              store_sector(dst + c * 2, o);
            }
          }
        } else {
#pragma unroll
          for (int c = 0; c < kHalf; c += 16) {
            float v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = acc[c + j];
            if (y0 + c < a.y_rows) store_chunk(a, x, y0 + c, v);
          }
        }
      }
    }
    if (lost) {
      if (lane == 0) fail();
      __syncwarp();
      if (a.parts > 1 && a.full_rounds * workers + worker / a.parts < a.tiles_x * a.tiles_y) {
        tc::named_barrier_sync(1, kPromoteWarps * 32);
        if (kCtas == 2) {      // the second one says who adds the tile up
          if (threadIdx.x == kFirstPromoteWarp * 32) *last_flag = 0u;
          __syncwarp();
          tc::named_barrier_sync(1, kPromoteWarps * 32);
        }
      }
    }
  }

  // ---- common exit ----
  tc::fence_before_thread_sync();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(1000);   // copies already issued land before shared memory goes away
  }
  if (kCtas == 2 || a.parts > 1) {
    tc::cluster_arrive();
    tc::cluster_wait();        // pairs: no CTA leaves while its peer may still read its shared memory or write its barriers
  }
  if (kCtas == 1 && a.parts > 1) {
    if (warp >= kFirstPromoteWarp && !*abort_flag) {
      const int tile = worker / a.parts, x0 = (tile % a.tiles_x) * kRows;
      gemm_core::add_up_cluster<kCols, kPromoteWarps * 32>(a, tc::smem_u32(smem), threadIdx.x - kFirstPromoteWarp * 32, worker % a.parts, a.parts,
                                                           0, 1, min(kRows, a.x_rows - x0), x0, (tile / a.tiles_x) * kCols);
    }
    tc::cluster_arrive();
    tc::cluster_wait();        // no CTA leaves while another may still read its sums
  }
  if (warp == 1) {
    tc::fence_after_thread_sync();
    if constexpr (kCtas == 2) tc::tmem_dealloc_pair(tmem_base, kTmemCols);
    else tc::tmem_dealloc(tmem_base, kTmemCols);
  }
}

template <int kCtas>
std::string launch(const CUtensorMap& mx, const CUtensorMap& my, const ScaledArgs& a, int workers, cudaStream_t stream) {
  auto kern = gemm_scaled_kernel<kCtas>;
  const std::string err = reserve_dynamic_smem(kern, Shape<kCtas>::kSmem);
  if (!err.empty()) return err;
  cudaLaunchConfig_t cfg{};
  const int cluster = kCtas == 2 ? 2 : a.parts;
  cfg.gridDim = dim3(workers * kCtas);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = Shape<kCtas>::kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, mx, my, a);
  return e == cudaSuccess ? "" : std::string("GEMM launch failed: ") + cudaGetErrorString(e);
}

int sm_count() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

}  // namespace

// How the problem is divided (see the head of this file). Measured: a K block takes 0.55 us (both forms), a meeting
// of pairs about 6 us and 1 us per piece, one inside a cluster about 3.5 us.
ScaledGemmPlan gemm_scaled_plan(int x_rows, int y_rows, int kblocks, int sms, const int (&clusters)[3]) {
  ScaledGemmPlan p{};
  p.ctas = x_rows > kRows ? 2 : 1;
  const long long tiles_x = (x_rows + kRows * p.ctas - 1) / (kRows * p.ctas), tiles_y = (y_rows + kCols - 1) / kCols;
  const long long ntiles = tiles_x * tiles_y;
  const int most = sms / p.ctas;
  p.full_rounds = (int)(ntiles / most);
  const int rem = (int)(ntiles - (long long)p.full_rounds * most);
  p.workers = p.full_rounds > 0 ? most : rem;
  p.parts = 1;
  p.per = kblocks;
  if (rem == 0 || (p.ctas == 1 && p.full_rounds > 0)) return p;
  double best = kblocks * 0.55;
  for (int parts = 2; parts <= 8; ++parts) {
    if (p.ctas == 1 && (parts & (parts - 1) || rem > clusters[parts == 2 ? 0 : parts == 4 ? 1 : 2])) continue;
    const int per = (kblocks + parts - 1) / parts;
    if (rem * parts > most || per < 2 || (parts - 1) * per >= kblocks) continue;
    const double us = per * 0.55 + (p.ctas == 2 ? 6.0 + parts : 3.5);
    if (us >= best) continue;
    best = us;
    p.parts = parts;
    p.per = per;
  }
  if (p.parts > 1 && p.full_rounds == 0) p.workers = rem * p.parts;
  if (p.parts > 1 && p.ctas == 2) {
    p.slice_floats = (size_t)rem * p.parts * p.ctas * kSliceFloats;
    p.counters = (size_t)rem * p.ctas;
  }
  return p;
}

// Clusters of 2, 4 and 8 CTAs of the decode form that the current device holds at a time.
static const int (&resident_clusters())[3] {
  static std::mutex mu;
  static std::map<int, std::array<int, 3>> known;
  static thread_local int out[3];
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(mu);
  auto it = known.find(dev);
  if (it == known.end()) {
    std::array<int, 3> n{0, 0, 0};
    if (reserve_dynamic_smem(gemm_scaled_kernel<1>, Shape<1>::kSmem).empty()) {
      for (int i = 0; i < 3; ++i) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(sm_count() / (2 << i) * (2 << i));
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = Shape<1>::kSmem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2 << i;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&n[i], gemm_scaled_kernel<1>, &cfg) != cudaSuccess) n[i] = 0;
      }
    }
    it = known.emplace(dev, n).first;
  }
  for (int i = 0; i < 3; ++i) out[i] = it->second[i];
  return out;
}

std::string gemm_scaled(const GemmProblem& g, const ScaledGemmPlan& p, cudaStream_t stream) {
  if (g.elem_size != 1 || !g.x_scale || !g.y_scale) return "block-scaled GEMM: e4m3 operands with both scales";
  if (g.k <= 0 || g.k % 128) return "K must be a positive multiple of 128";
  if (g.x_rows <= 0 || g.y_rows <= 0) return "";
  ScaledArgs a{};
  a.x_rows = g.x_rows;
  a.y_rows = g.y_rows;
  a.kblocks = g.k / 128;
  a.tiles_x = (g.x_rows + kRows * p.ctas - 1) / (kRows * p.ctas);
  a.tiles_y = (g.y_rows + kCols - 1) / kCols;
  a.full_rounds = p.full_rounds;
  a.parts = p.parts;
  a.per = p.per;
  if (p.slice_floats > 0) {
    if (!g.ws || !g.counters || g.ws_bytes < p.slice_floats * sizeof(float) || g.counter_count < p.counters)
      return "block-scaled GEMM: the scratch is too small for this problem";
    if (reinterpret_cast<uintptr_t>(g.ws) % 16) return "block-scaled GEMM: the scratch must be 16-byte aligned";
  }
  a.ws = g.ws;
  a.counters = g.counters;
  a.x_scale = g.x_scale;
  a.y_scale = g.y_scale;
  a.out = g.out;
  a.sx = g.sx;
  a.sy = g.sy;
  a.out_dtype = g.out_dtype;
  a.whole_sectors = g.out_dtype != kF32 && g.sy == 1 && (g.sx * 2) % 32 == 0 && reinterpret_cast<uintptr_t>(g.out) % 32 == 0;
  a.idesc = tc::make_idesc(kRows * p.ctas, kHalf, 0, 0);
  a.status = g.status;
  CUtensorMap mx, my;
  std::string err = tma::kmajor_2d(&mx, g.x, g.x_rows, g.k, g.ldx, 1, g.elem_kind, kRows);
  if (!err.empty()) return err;
  err = tma::kmajor_2d(&my, g.y, g.y_rows, g.k, g.ldy, 1, g.elem_kind, kHalf / p.ctas);
  if (!err.empty()) return err;
  return p.ctas == 2 ? launch<2>(mx, my, a, p.workers, stream) : launch<1>(mx, my, a, p.workers, stream);
}

ScaledGemmPlan gemm_scaled_plan_here(int x_rows, int y_rows, int kblocks) {
  return gemm_scaled_plan(x_rows, y_rows, kblocks, sm_count(), resident_clusters());
}

}  // namespace tdx
