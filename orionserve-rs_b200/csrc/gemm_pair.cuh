// Products of many rows on the tensor cores: persistent CTA pairs, shared by the projections (gemm_tc.cu) and the mixtures (moe_gemm_tc.cu).
//
// Prompts and continuous batching are bound by the tensor cores, with the rate at which operands reach shared memory close behind. Two CTAs of a
// cluster work as one MMA unit (tcgen05 cta_group::2) on a tile of 256 weight rows x up to 256 tokens: each loads its own 128 weight rows and HALF of
// the token rows, so 64 k cost 32 KiB of loads per CTA for 4.2 MFLOP. The accumulator takes 256 of the 512 columns of tensor memory; there are two, and
// the pairs stay on their SMs and go from tile to tile: the epilogue of one tile (an activation, or 128 KiB of f32 stores) runs under the main loop of
// the next, and the rings never drain in between. What the issuing warp does between two MMAs counts (128 cycles each): its loop is uniform over
// the warp and one elected lane issues, stages hold 128 k, and ONE commit a stage frees both CTAs' halves. Measured on 8192 x 14336 x 4096: one lane
// in a divergent branch with four commits every 64 k 735 us, with one commit 617, like this 612; with 128 tokens a tile 1310, 994, 799.
//
// The epilogue has eight warps: with four, the activations of a mixture (k 2048, 13 us of main loop a tile) took longer than the main loop (up
// projection of 7006 rows, 331 us against 210; of 2048 rows with the exact GELU, 125 against 87).
//
// A CTA has 384 threads: warp 0 loads, warp 1 of the leader issues the MMAs, warps 4-11 are the epilogue. Every wait is bounded; a wait that runs out
// sets the error word, and the CTAs still free their tensor memory.
#pragma once

#include "kernels.h"
#include "tcgen05.cuh"

namespace orion {
namespace {

__device__ __forceinline__ void tmem_alloc_pair(uint32_t *dst_smem, uint32_t ncols) {  // one warp in EACH CTA of the pair
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// 2-D tiled TMA load of one CTA of a pair: the data lands in THIS CTA's shared memory, the bytes are
// counted on the barrier at cluster address `bar_cluster_addr` (the leader's). No multicast.
__device__ __forceinline__ void tma_load_2d_pair(void *dst_smem, const void *tensor_map, int c0, int c1, uint32_t bar_cluster_addr) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst_smem)),
      "l"(tensor_map), "r"(c0), "r"(c1), "r"(bar_cluster_addr)
      : "memory");
}
__device__ __forceinline__ void cluster_arrive_release() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait_acquire() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// Address of the same shared-memory location in cluster member `rank`.
__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}
// Arrives on this barrier in both CTAs of the pair once every MMA issued so far by this thread has completed.
__device__ __forceinline__ void umma_commit_both(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "h"((uint16_t)3)
               : "memory");
}

// Order in which CTAs take output tiles: eight token tiles against every weight tile before the next eight, token tiles first. With the weight tiles
// first, a wave of 148 CTAs would meet nearly all of them with one token tile, and a matrix larger than L2 would come from HBM again for every 256
// tokens; like this a wave works on about as many tokens as weight rows.
struct TileXy {
  uint32_t x, y;
};
constexpr uint32_t kRasterTokens = 8;
__device__ __forceinline__ TileXy raster(uint32_t id, uint32_t tiles_x, uint32_t tiles_y) {
  const uint32_t first = id / (kRasterTokens * tiles_x) * kRasterTokens, in = id - first * tiles_x, tall = min(kRasterTokens, tiles_y - first);
  return {in / tall, first + in % tall};
}

struct PairConfig {
  static constexpr uint32_t kThreads = 384, kRows = 128, kSlabK = 64;  // threads and weight rows per CTA, k of a TMA box (one swizzle atom)
  static constexpr uint32_t kMaxTokens = 256, kStages = 3, kStageK = 2 * kSlabK;
  static constexpr uint32_t kWSlab = kRows * kSlabK * 2, kXSlab = kMaxTokens / 2 * kSlabK * 2;  // 64 k of either operand
  static constexpr uint32_t kWBytes = 2 * kWSlab, kXBytes = 2 * kXSlab;                          // one stage of either ring
  static constexpr uint32_t kXRingOffset = kStages * kWBytes, kBarrierOffset = kXRingOffset + kStages * kXBytes;
  static constexpr uint32_t kTmemCols = 512, kEpilogueWarps = 8;
  static constexpr int kSmemBytes = kBarrierOffset + 1024 /*align*/ + 512 /*barriers*/;
  static_assert(kSmemBytes <= 232448, "ring exceeds the shared memory of an SM");
};
constexpr uint32_t kPairs = 74;  // of 148 SMs

// A tile: weight rows w_row .. + 255 of *w against token rows x_row .. + cols - 1 of *x (cols a multiple of 32 up to 256, as a pair's MMA takes them; boxes of `box` token rows, at
// least half of cols and a multiple of 8), stages kb .. end of k.
struct PairJob {
  const CUtensorMap *w, *x;
  uint32_t w_row, x_row, cols, box, kb, end;
};

// The body of a kernel of pairs (grid: two CTAs each, cluster of two). Work provides
//   total()          tiles of the launch
//   early(id)        whether tile `id` is known before the preceding kernel has ended
//   job(id)          the tile, a Job; one without stages (kb == end) is passed over
//   Job              what job() returns: a PairJob, and what store() needs
//   store(j, row, c, r)  columns c .. c + 15 of weight row w_row + row (of 32 in a warp, one a lane), f32
template <typename Work>
__device__ __forceinline__ void run_pairs(const Work &work, ReadyWait ready, uint32_t *error) {
  using Cfg = PairConfig;
  constexpr uint32_t kStages = Cfg::kStages;
  extern __shared__ uint8_t raw_smem[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(raw_smem) + 1023) & ~uintptr_t(1023));
  uint8_t *w_ring = smem, *x_ring = smem + Cfg::kXRingOffset;
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + Cfg::kBarrierOffset);
  uint64_t *empty = full + kStages, *acc_full = empty + kStages, *acc_empty = acc_full + 2;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 2);

  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = blockIdx.x & 1u, pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const bool leader = rank == 0;
  const uint32_t total = work.total();

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 2 * Cfg::kEpilogueWarps);  // both CTAs' epilogues (used in the leader)
    }
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, Cfg::kTmemCols);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_arrive_release();  // the peer's barriers exist before anything of this CTA signals them
  cluster_wait_acquire();
  tc_fence_after();
  // only now: a dependent CTA that waits for this grid must not hold tensor memory that a CTA of it still needs
  pdl_trigger();
  const uint32_t tmem_base = *tmem_slot;
  bool ok = true;
  auto wait = [](uint64_t *bar, uint32_t parity) { return (bool)__all_sync(0xffffffffu, mbar_wait(bar, parity)); };  // one answer for a warp

  if (warp == 0) {
    // Producer: this CTA's weight rows and its half of the token rows; the bytes of both CTAs are counted on the leader's barrier. Weights are
    // immutable: those of the first tile are asked for before the wait for the kernel that makes the activations, where the tile is known.
    const bool elected = elect_one();
    uint32_t it = 0, early = 0;
    auto load_w = [&](uint32_t s, uint32_t kb, const PairJob &j) {
      if (!elected) return;
      const uint32_t bar = mapa_u32(smem_u32(&full[s]), 0);
      if (leader) mbar_arrive_expect_tx(&full[s], 2 * (Cfg::kWBytes + 2 * j.box * Cfg::kSlabK * 2));
#pragma unroll
      for (uint32_t h = 0; h < 2; ++h)
        tma_load_2d_pair(w_ring + s * Cfg::kWBytes + h * Cfg::kWSlab, j.w, (int)(kb * Cfg::kStageK + h * Cfg::kSlabK), (int)(j.w_row + rank * Cfg::kRows), bar);
    };
    if (pair < total && work.early(pair)) {
      const typename Work::Job j = work.job(pair);
      for (uint32_t kb = j.kb; kb < j.end && early < kStages; ++kb, ++early) load_w(early, kb, j);
    }
    if (ready.counter) {
      if (!wait_ready(ready)) atomicOr(error, 2u);
      fence_proxy_async_all();
    } else {
      pdl_wait();
    }
    for (uint32_t t = pair; ok && t < total; t += pairs) {
      const typename Work::Job j = work.job(t);
      for (uint32_t kb = j.kb; kb < j.end; ++kb, ++it) {
        const uint32_t s = it % kStages;
        if (it >= early) {
          if (!wait(&empty[s], ((it / kStages) & 1) ^ 1)) { ok = false; break; }
          load_w(s, kb, j);
        }
        if (elected) {
          const uint32_t bar = mapa_u32(smem_u32(&full[s]), 0);
#pragma unroll
          for (uint32_t h = 0; h < 2; ++h)
            tma_load_2d_pair(x_ring + s * Cfg::kXBytes + h * Cfg::kXSlab, j.x, (int)(kb * Cfg::kStageK + h * Cfg::kSlabK), (int)(j.x_row + rank * (j.cols / 2)), bar);
        }
        __syncwarp();
      }
    }
    // the slots that are still being read: nobody signals a barrier of a CTA that is gone
    for (uint32_t i = it > kStages ? it - kStages : 0; ok && i < it; ++i) ok = wait(&empty[i % kStages], (i / kStages) & 1);
  } else if (warp == 1) {
    if (leader) {  // issues for both CTAs
      const uint64_t w_desc = desc_k_sw128(smem_u32(w_ring)), x_desc = desc_k_sw128(smem_u32(x_ring));
      const bool elected = elect_one();
      if (!Work::kStaticTiles) pdl_wait();  // the list of tiles
      uint32_t it = 0, turn = 0;
      for (uint32_t t = pair; ok && t < total; t += pairs) {
        const typename Work::Job j = work.job(t);
        if (j.kb >= j.end) continue;
        const uint32_t id = idesc(2 * Cfg::kRows, j.cols, false), buf = turn & 1, acc = tmem_base + buf * Cfg::kMaxTokens;
        if (!wait(&acc_empty[buf], ((turn >> 1) & 1) ^ 1)) { ok = false; break; }
        tc_fence_after();
        for (uint32_t kb = j.kb; kb < j.end; ++kb, ++it) {
          const uint32_t s = it % kStages;
          if (!wait(&full[s], (it / kStages) & 1)) { ok = false; break; }
          tc_fence_after();
          if (elected) {
            const uint64_t a = w_desc + s * (Cfg::kWBytes >> 4), b = x_desc + s * (Cfg::kXBytes >> 4);
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h)
#pragma unroll
              for (uint32_t k = 0; k < Cfg::kSlabK / 16; ++k)  // 16 k elements inside the swizzle atom = 32 bytes on the start address
                umma_bf16_pair(acc, a + ((h * Cfg::kWSlab + k * 32) >> 4), b + ((h * Cfg::kXSlab + k * 32) >> 4), id, (kb > j.kb || h > 0 || k > 0) ? 1u : 0u);
            umma_commit_both(&empty[s]);  // the stage of both CTAs is free once these MMAs have read it
          }
          __syncwarp();
        }
        if (ok && elected) umma_commit_both(&acc_full[buf]);
        ++turn;
      }
    }
  } else if (warp >= 4) {
    // Epilogue: warp w reads tensor-memory lanes 32 * (w % 4) .. + 31 (lane = weight row, column = token); the two warps of the same lanes take
    // turns, 16 columns each. With two or four loads of 16 in flight the loop was that much longer, and the eight warps waited for instructions: GELU of
    // 512 x 8192, k 512, four at a time 22.5 us, two 20.2, one 18.4; with all activations in one kernel, told apart for every value, 23.0.
    // The output may still be read by the kernel before the producer of x. (With a ready counter the producer has read it before it counted.)
    if (!ready.counter) pdl_wait();
    uint32_t turn = 0;
    for (uint32_t t = pair; ok && t < total; t += pairs) {
      const typename Work::Job j = work.job(t);
      if (j.kb >= j.end) continue;
      const uint32_t buf = turn & 1, acc = tmem_base + (((warp & 3) * 32u) << 16) + buf * Cfg::kMaxTokens;
      if (!wait(&acc_full[buf], (turn >> 1) & 1)) { ok = false; break; }
      ++turn;
      tc_fence_after();
      constexpr uint32_t kStep = 16 * (Cfg::kEpilogueWarps / 4);
      uint32_t mb = 16 * ((warp - 4) / 4);
      // once this warp's last columns are in registers, the MMAs of the tile after the next may write them
      auto release = [&] {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&acc_empty[buf]), 0));
      };
      if (mb >= j.cols) release();
#pragma unroll 1
      for (; mb < j.cols; mb += kStep) {
        uint32_t rr[16];
        tmem_ld16(acc + mb, rr);
        tmem_ld_wait();
        if (mb + kStep >= j.cols) release();
        work.store(j, rank * Cfg::kRows + (warp & 3) * 32 + lane, mb, rr);
      }
    }
  }
  if (!ok) atomicOr(error, 1u);
  tc_fence_before();
  __syncthreads();
  // Neither CTA leaves, nor frees the tensor memory the pair allocated together, while the other may still be read by an MMA or be reading
  // its accumulator.
  cluster_arrive_release();
  cluster_wait_acquire();
  if (warp == 1) tmem_dealloc_pair(tmem_base, Cfg::kTmemCols);
}

}  // namespace
}  // namespace orion
