// bf16 GEMM on the 5th-generation tensor cores:  partial[s][r][n] = sum_k x[r][k] * w[n][k]
// (tensor.rs:114-128 without the bias), f32 accumulation in tensor memory.
//
// The weight matrix is the M operand of the MMA ("swap A/B"): a CTA owns a tile
// of 128 weight rows x TOKN tokens, so the batch size only changes the N extent
// of the instruction and a decode step (1..256 tokens) streams every weight
// byte exactly once. W [n][k] and x [r][k] are both K-major as stored, so no
// transposition is needed.
//
// Per CTA (256 threads):
//   warp 0   one lane streams the W tile (TMA tensor loads, 128B-swizzled 64-wide k
//            slabs) into the deep weight ring; it never waits for the preceding kernel;
//   warp 2   one lane waits for the preceding kernel (programmatic dependent launch),
//            then keeps the short activation ring full (x tiles come from L2);
//   warp 1   allocates tensor memory, one lane issues tcgen05.mma (128 x TOKN x 16,
//            four per k slab) and commits to the "empty" barriers of both stages;
//   warps 4-7 epilogue: tcgen05.ld the accumulator (lane = weight row, column =
//            token) and store f32 partials, 128 contiguous bytes per warp store.
// Split-K: blockIdx.z owns a contiguous range of k slabs and writes its own slab
// of the partial buffer; the consumer kernel sums the slabs.
// Every CTA loads its own tiles, nothing is multicast. Clusters appear in two forms only: CTA pairs
// for batches of more than 256 rows (gemm_pair_kernel), and the split-K reduction over distributed shared
// memory (off by default). The activation producer can take its dependency from a counter in device
// memory instead of the preceding kernel's completion (ReadyWait, used after a tensor-parallel hand-over).
// Every wait is bounded; a wait that runs out sets a device error word and the
// CTA still releases its tensor memory before returning.
#include "gemm_pair.cuh"
#include "value_cache.h"

#include <algorithm>
#include <cstdlib>
#include <tuple>

namespace orion {
namespace {

constexpr int kTileN = 128;   // weight rows per CTA (M of the MMA)
constexpr int kSlabK = 64;    // k elements per stage: 128 bytes = one swizzle atom
constexpr int kUmmaK = 16;
constexpr int kThreads = 256;

__device__ uint32_t g_gemm_error = 0;
#ifdef ORION_TRACE
// Phase trace, compiled in with -DORION_TRACE only and switched on by ORION_GEMM_TRACE=1:
// %globaltimer stamps of CTA (0,0,0) of the last launches.
constexpr int kTraceLaunches = 160, kTraceStamps = 8;
__device__ unsigned long long g_gemm_trace[kTraceLaunches][kTraceStamps];
__device__ uint32_t g_gemm_trace_on = 0, g_gemm_trace_next = 0;
__device__ __forceinline__ void gtrace(uint32_t slot, int k) {
  if (slot != 0xFFFFFFFFu) g_gemm_trace[slot][k] = global_timer_ns();
}
#define ORION_GTRACE(slot, k) gtrace(slot, k)
#else
#define ORION_GTRACE(slot, k) ((void)0)
#endif

// Two rings per CTA. Weight tiles come from HBM (long latency, the stream that must never
// stall): WST stages of 16 KiB. Activation tiles come from L2 (every CTA re-reads them):
// XST stages of TOKN x 128 B are enough. Measured on decode shapes, weight bandwidth follows
// the weight bytes in flight per SM (160 KiB -> 6.0 TB/s, 128 KiB -> 5.3 TB/s), so shared
// memory goes to the W ring first.
// MT = weight tiles of 128 rows per CTA. Decode batches stream weights (MT = 1, as many CTAs as
// possible); 129 to 256 rows feel the shared-memory fill rate as well, so a CTA there takes two weight
// tiles against one activation tile (MT = 2: 64 KiB of operands per 8.4 MFLOP instead of 48 KiB per 4.2),
// with two accumulators in tensor memory.
template <int TOKN, int WST, int XST, int MT = 1>
struct TcConfig {
  static constexpr int kWBytes = MT * kTileN * kSlabK * 2;
  static constexpr int kXBytes = TOKN * kSlabK * 2;
  static constexpr int kWStages = WST;
  static constexpr int kXStages = XST;
  static constexpr int kXRingOffset = WST * kWBytes;
  static constexpr int kBarrierOffset = kXRingOffset + XST * kXBytes;
  static constexpr int kTmemCols = MT * TOKN < 32 ? 32 : MT * TOKN;
  static_assert(kTmemCols <= 512 && (kTmemCols & (kTmemCols - 1)) == 0, "tensor memory columns: a power of two up to 512");
  static constexpr int kSmemBytes = kBarrierOffset + 1024 /*align*/ + 512 /*barriers*/;
};

__device__ __forceinline__ float ld_dsmem_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
// ACT: the epilogue stores activations (kGemmGelu, kGemmRelu2, kGemmGeglu, kGemmStore); else f32 partials, or SwiGLU where `act` is given. A
// template parameter, since the larger epilogue costs the weight-streaming shapes 0.8 us per launch.
template <int TOKN, int WST, int XST, int MT, bool ACT>
__global__ void __launch_bounds__(kThreads)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
               float *__restrict__ partial, bf16 *__restrict__ act, uint32_t M, uint32_t N, uint32_t K,
               uint32_t splits, uint32_t cluster_reduce, uint32_t ldc, uint32_t epilogue, ReadyWait ready, const float *__restrict__ bias) {
  using Cfg = TcConfig<TOKN, WST, XST, MT>;
  extern __shared__ uint8_t raw_smem[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(raw_smem) + 1023) &
                                              ~uintptr_t(1023));
  uint8_t *w_ring = smem, *x_ring = smem + Cfg::kXRingOffset;
  uint64_t *full_w = reinterpret_cast<uint64_t *>(smem + Cfg::kBarrierOffset);
  uint64_t *empty_w = full_w + WST;
  uint64_t *full_x = empty_w + WST;
  uint64_t *empty_x = full_x + XST;
  uint64_t *acc_ready = empty_x + XST;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_ready + 1);

  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t n0 = blockIdx.x * (MT * kTileN), t0 = blockIdx.y * TOKN, split = blockIdx.z;
  const uint32_t nkb = (K + kSlabK - 1) / kSlabK;
  const uint32_t kb_begin = (uint32_t)((uint64_t)split * nkb / splits);
  const uint32_t kb_end = (uint32_t)((uint64_t)(split + 1) * nkb / splits);
  const uint32_t my_kb = kb_end - kb_begin;

  pdl_trigger();
#ifdef ORION_TRACE
  __shared__ uint32_t trace_slot_s;
#endif
  if (threadIdx.x == 0) {
#ifdef ORION_TRACE
    uint32_t slot = 0xFFFFFFFFu;
    if (g_gemm_trace_on && blockIdx.x + blockIdx.y + blockIdx.z == 0) {
      slot = atomicAdd(&g_gemm_trace_next, 1u) % kTraceLaunches;
      g_gemm_trace[slot][7] = ((unsigned long long)gridDim.x << 32) | (gridDim.z << 16) | my_kb;
    }
    trace_slot_s = slot;
    gtrace(slot, 0);
#endif
    for (int s = 0; s < WST; ++s) {
      mbar_init(&full_w[s], 1);
      mbar_init(&empty_w[s], 1);
    }
    for (int s = 0; s < XST; ++s) {
      mbar_init(&full_x[s], 1);
      mbar_init(&empty_x[s], 1);
    }
    mbar_init(acc_ready, 1);
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
#ifdef ORION_TRACE
  const uint32_t tslot = trace_slot_s;
#endif
  bool ok = true;

  if (warp == 0) {
    // Weight producer. Weights are immutable, so this stream starts while the kernel that
    // produces the activations is still running and never waits for it.
    if (lane == 0) {
      ORION_GTRACE(tslot, 1);
      for (uint32_t i = 0; i < my_kb; ++i) {
        const uint32_t s = i % WST, use = i / WST;
        if (!mbar_wait(&empty_w[s], (use & 1) ^ 1)) { ok = false; break; }
        mbar_arrive_expect_tx(&full_w[s], Cfg::kWBytes);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)  // rows past the matrix read as zeros and still count their bytes
          tma_load_2d(w_ring + s * Cfg::kWBytes + mt * (kTileN * kSlabK * 2), &map_w, (int)((kb_begin + i) * kSlabK),
                      (int)(n0 + mt * kTileN), &full_w[s]);
      }
    }
  } else if (warp == 2) {
    // Activation producer: waits for the preceding kernel, then keeps the short x ring full.
    if (lane == 0) {
      if (ready.counter) {  // the activations' producer counts its finished CTAs: no wait for its completion
        if (!wait_ready(ready)) atomicOr(&g_gemm_error, 2u);
        fence_proxy_async_all();
      } else {
        pdl_wait();
      }
      ORION_GTRACE(tslot, 3);
      for (uint32_t i = 0; i < my_kb; ++i) {
        const uint32_t s = i % XST, use = i / XST;
        if (!mbar_wait(&empty_x[s], (use & 1) ^ 1)) { ok = false; break; }
        mbar_arrive_expect_tx(&full_x[s], Cfg::kXBytes);
        tma_load_2d(x_ring + s * Cfg::kXBytes, &map_x, (int)((kb_begin + i) * kSlabK), (int)t0, &full_x[s]);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t id = idesc(kTileN, TOKN, false);
      for (uint32_t i = 0; i < my_kb; ++i) {
        const uint32_t sw = i % WST, sx = i % XST;
        if (!mbar_wait(&full_w[sw], (i / WST) & 1)) { ok = false; break; }
        if (i == 0) ORION_GTRACE(tslot, 2);
        if (!mbar_wait(&full_x[sx], (i / XST) & 1)) { ok = false; break; }
        tc_fence_after();
        const uint32_t wt = smem_u32(w_ring + sw * Cfg::kWBytes);
        const uint32_t xt = smem_u32(x_ring + sx * Cfg::kXBytes);
#pragma unroll
        for (int k = 0; k < kSlabK / kUmmaK; ++k) {
          // advancing 16 k elements inside the swizzle atom = +32 bytes on the start address
          const uint64_t b = desc_k_sw128(xt + k * kUmmaK * 2);
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {  // one accumulator of TOKN columns per weight tile
            const uint64_t a = desc_k_sw128(wt + mt * (kTileN * kSlabK * 2) + k * kUmmaK * 2);
            umma_bf16(tmem_base + (uint32_t)(mt * TOKN), a, b, id, (i > 0 || k > 0) ? 1u : 0u);
          }
        }
        umma_commit(&empty_w[sw]);  // both stages are free once these MMAs have read them
        umma_commit(&empty_x[sx]);
      }
      umma_commit(acc_ready);  // arrives when every MMA above has completed
      ORION_GTRACE(tslot, 4);
    }
  } else if (!ACT && warp >= 4) {
    // Epilogue warps: warp w may touch tensor-memory lanes 32*(w%4) .. +31.
    const uint32_t lq = warp & 3;
    // The partial buffer may still be read by the kernel before the producer of x: wait for the
    // predecessor here, while the main loop runs, rather than after the accumulator is ready. (With a
    // ready counter the producer has read the buffer before it counted, and the accumulator follows the count.)
    if (!ready.counter) pdl_wait();
    if (my_kb > 0) {
      if (!mbar_wait(acc_ready, 0)) ok = false;
    }
    tc_fence_after();
    if (threadIdx.x == 128) ORION_GTRACE(tslot, 5);
    float *dst = partial + (size_t)split * M * N;
    // Split-K inside a cluster: the tile goes to shared memory as stage[token][128 weight rows]
    // (the rings are idle: every load has landed and every MMA has read its operands).
    float *stage = reinterpret_cast<float *>(smem);
    // Tensor-memory loads are issued for up to four 16-column chunks before the one wait, so the
    // round trips of a batch overlap; stores follow chunk by chunk.
    constexpr int kBatch = TOKN >= 64 ? 4 : TOKN / 16;
#pragma unroll 1
    for (int mb = 0; mb < MT * TOKN; mb += 16 * kBatch) {
      uint32_t rr[kBatch][16];
      if (ok && my_kb > 0) {
#pragma unroll
        for (int b = 0; b < kBatch; ++b) tmem_ld16(tmem_base + ((lq * 32u) << 16) + (uint32_t)(mb + 16 * b), rr[b]);
        tmem_ld_wait();
      } else {
#pragma unroll
        for (int b = 0; b < kBatch; ++b)
#pragma unroll
          for (int j = 0; j < 16; ++j) rr[b][j] = 0u;
      }
#pragma unroll
      for (int b = 0; b < kBatch; ++b) {
      const int mc = mb + 16 * b;
      const int mt = mc / TOKN, c = mc % TOKN;  // weight tile, first token column of this chunk
      const uint32_t n = n0 + mt * kTileN + lq * 32 + lane;
      if (t0 + c >= M) continue;  // warp-uniform
      uint32_t (&r)[16] = rr[b];
      if (cluster_reduce) {
#pragma unroll
        for (int j = 0; j < 16; ++j) stage[(c + j) * kTileN + lq * 32 + lane] = __uint_as_float(r[j]);
      } else if (act != nullptr) {
        // Fused SwiGLU (tensor.rs:167-189): weight rows are interleaved, lane 2i holds gate_f and
        // lane 2i + 1 holds up_f of the same f for these 16 tokens. Each lane of a pair trades
        // half of its values with the other and finishes one token of every token pair.
        const uint32_t odd = lane & 1u;
        const uint32_t f = n >> 1, F = N >> 1;
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) {
          const uint32_t send = odd ? r[2 * jj] : r[2 * jj + 1];
          const uint32_t recv = __shfl_xor_sync(0xffffffffu, send, 1);
          const float g = __uint_as_float(odd ? recv : r[2 * jj]);
          const float u = __uint_as_float(odd ? r[2 * jj + 1] : recv);
          const uint32_t tok = t0 + c + 2 * jj + odd;
          if (tok < M && n < N) act[(size_t)tok * F + f] = __float2bfloat16_rn(__fmul_rn(g / (1.0f + __expf(-g)), u));
        }
      } else if (n < N) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const uint32_t tok = t0 + c + j;
          if (tok < M) dst[(size_t)tok * ldc + n] = __uint_as_float(r[j]);  // ldc: row stride of the output
        }
      }
      }
    }
  }
  if constexpr (ACT) {
    // Activations in bf16, row stride ldc. All eight warps: the conversion is as long as a short k loop, and the
    // producers and the issuing warp have nothing left to do. Warps 0-3 take the second half of the columns.
    __syncwarp();
    const uint32_t lq = warp & 3;
    pdl_wait();  // `act` may still be read by the kernel before the producer of x
    if (!mbar_wait(acc_ready, 0)) ok = false;
    tc_fence_after();
    constexpr int kCols = MT * TOKN, kHalf = kCols >= 32 ? kCols / 2 : kCols;
    const int begin = warp >= 4 ? 0 : kHalf, end = warp >= 4 ? kHalf : kCols;
#pragma unroll 1
    for (int mc = begin; mc < end; mc += 16) {
      uint32_t r[16];
      tmem_ld16(tmem_base + ((lq * 32u) << 16) + (uint32_t)mc, r);
      tmem_ld_wait();
      const int mt = mc / TOKN, c = mc % TOKN;
      const uint32_t n = n0 + mt * kTileN + lq * 32 + lane;
      if (epilogue == kGemmGeglu) {
        // lane 2i holds gate f, lane 2i + 1 up f; a pair trades halves and each finishes one token of every two
        const uint32_t odd = lane & 1u;
        bf16 *dst = act + (size_t)(t0 + c) * ldc + (n >> 1);
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) {
          const uint32_t recv = __shfl_xor_sync(0xffffffffu, odd ? r[2 * jj] : r[2 * jj + 1], 1);
          const float g = __uint_as_float(odd ? recv : r[2 * jj]), u = __uint_as_float(odd ? r[2 * jj + 1] : recv);
          const uint32_t j = 2 * jj + odd;
          if (t0 + c + j < M && n < N) dst[(size_t)j * ldc] = __float2bfloat16_rn(gelu_tanh<bf16>(g) * u);
        }
        continue;
      }
      if (t0 + c >= M || n >= N) continue;
      bf16 *dst = act + (size_t)(t0 + c) * ldc + n;
      const uint32_t valid = M - (t0 + c);
      const float b = bias ? bias[n] : 0.f;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float v = __uint_as_float(r[j]) + b;
        if ((uint32_t)j < valid) dst[(size_t)j * ldc] = __float2bfloat16_rn(epilogue == kGemmGelu ? gelu_tanh<bf16>(v) : (epilogue == kGemmRelu2 ? relu2(v) : v));
      }
    }
    __syncwarp();
  }
  if (cluster_reduce) {
    // The `splits` CTAs of one tile form a cluster (1, 1, splits). Every CTA sums a share of the
    // tile's tokens over all members' staged tiles (distributed shared memory, member order, so
    // the result is the same as summing slabs in order) and writes slab 0 only.
    __syncthreads();
    cluster_arrive_release();
    cluster_wait_acquire();
    if (warp >= 4) {
      const uint32_t row = (warp & 3) * 32 + lane, n = n0 + row;
      const uint32_t valid = (M - t0) < (uint32_t)TOKN ? (M - t0) : (uint32_t)TOKN;
      const uint32_t tb = split * valid / splits, te = (split + 1) * valid / splits;
      const uint32_t base = smem_u32(smem) + row * 4;
#pragma unroll 2
      for (uint32_t tok = tb; tok < te; ++tok) {
        float x[8];
#pragma unroll
        for (uint32_t s = 0; s < 8; ++s) x[s] = s < splits ? ld_dsmem_f32(mapa_u32(base + tok * (kTileN * 4), s)) : 0.f;
        float acc = 0.f;
#pragma unroll
        for (uint32_t s = 0; s < 8; ++s)
          if (s < splits) acc += x[s];
        if (n < N) partial[(size_t)(t0 + tok) * N + n] = acc;
      }
    }
    cluster_arrive_release();  // nobody leaves while a peer may still read its staged tile
    cluster_wait_acquire();
  }
  if (threadIdx.x == 128) ORION_GTRACE(tslot, 6);
  if (!ok) atomicOr(&g_gemm_error, 1u);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, Cfg::kTmemCols);
}

// ---- many rows: persistent CTA pairs (gemm_pair.cuh) ------------------------------

template <GemmEpilogue OUT>
struct ProjectionWork {
  static constexpr bool kStaticTiles = true;
  struct Job : PairJob {
    float *out;
  };
  const CUtensorMap *map_w, *map_x, *map_tail;
  float *partial;
  bf16 *act;
  const float *bias;
  uint32_t M, N, splits, tokn, whole, tail, ldc, tiles_x, tiles_y, stages;

  // `whole` tiles, and those after them in `tail` pieces each
  __device__ __forceinline__ uint32_t total() const { return whole + (tiles_x * tiles_y * splits - whole) * tail; }
  __device__ __forceinline__ bool early(uint32_t) const { return true; }
  __device__ __forceinline__ Job job(uint32_t id) const {  // the k split slowest
    const bool piece = id >= whole;
    const uint32_t at = piece ? (id - whole) % tail : 0, cols = piece ? tokn / tail : tokn;
    if (piece) id = whole + (id - whole) / tail;
    const uint32_t plane = tiles_x * tiles_y, split = id / plane;
    const TileXy t = raster(id % plane, tiles_x, tiles_y);
    return {{map_w, piece ? map_tail : map_x, t.x * (2 * kTileN), t.y * tokn + at * cols, cols, cols / 2, (uint32_t)((uint64_t)split * stages / splits),
             (uint32_t)((uint64_t)(split + 1) * stages / splits)},
            partial + (size_t)split * M * N};
  }
  __device__ __forceinline__ void store(const Job &j, uint32_t row, uint32_t c, uint32_t (&r)[16]) const {
    const uint32_t n = j.w_row + row, t0 = j.x_row + c;
    if (t0 >= M) return;  // warp-uniform
    if (OUT == kGemmPartials) {
      if (n < N) {
#pragma unroll
        for (uint32_t i = 0; i < 16; ++i)
          if (t0 + i < M) j.out[(size_t)(t0 + i) * ldc + n] = __uint_as_float(r[i]);
      }
    } else if (OUT == kGemmSwiglu || OUT == kGemmGeglu) {
      // Weight rows are interleaved: lane 2i holds gate f, lane 2i + 1 up f of these 16 tokens. The lanes of a pair trade halves and each
      // finishes one token of every two (SwiGLU: tensor.rs:167-189).
      const uint32_t odd = row & 1u;
      const size_t stride = OUT == kGemmSwiglu ? N >> 1 : ldc;
      bf16 *to = act + (t0 + odd) * stride + (n >> 1);
#pragma unroll
      for (uint32_t jj = 0; jj < 8; ++jj, to += 2 * stride) {
        const uint32_t recv = __shfl_xor_sync(0xffffffffu, odd ? r[2 * jj] : r[2 * jj + 1], 1);
        const float g = __uint_as_float(odd ? recv : r[2 * jj]), u = __uint_as_float(odd ? r[2 * jj + 1] : recv);
        const float v = OUT == kGemmSwiglu ? __fmul_rn(g / (1.0f + __expf(-g)), u) : gelu_tanh<bf16>(g) * u;
        if (t0 + 2 * jj + odd < M && n < N) *to = __float2bfloat16_rn(v);
      }
    } else if (n < N) {
      bf16 *to = act + (size_t)t0 * ldc + n;
      const float b = bias ? bias[n] : 0.f;
#pragma unroll
      for (uint32_t i = 0; i < 16; ++i, to += ldc) {
        const float v = __uint_as_float(r[i]) + b;
        if (t0 + i < M) *to = __float2bfloat16_rn(OUT == kGemmGelu ? gelu_tanh<bf16>(v) : (OUT == kGemmRelu2 ? relu2(v) : v));
      }
    }
  }
};

template <GemmEpilogue OUT>
__global__ void __launch_bounds__(PairConfig::kThreads)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_tail,
                 float *__restrict__ partial, bf16 *__restrict__ act, uint32_t M, uint32_t N, uint32_t K, uint32_t splits, uint32_t tokn, uint32_t whole,
                 uint32_t tail, uint32_t ldc, ReadyWait ready, const float *__restrict__ bias) {
  const ProjectionWork<OUT> work{&map_w, &map_x, &map_tail, partial, act, bias, M, N, splits, tokn, whole, tail, ldc, (N + 2 * kTileN - 1) / (2 * kTileN),
                                 (M + tokn - 1) / tokn, (K + PairConfig::kStageK - 1) / PairConfig::kStageK};
  run_pairs(work, ready, &g_gemm_error);
}

// ---- host side -----------------------------------------------------------------

// [rows][k] bf16 matrix with row stride ld; box = 64 k x box_rows, 128-byte swizzle.
int make_map(CUtensorMap *map, const void *base, uint64_t rows, uint64_t k, uint64_t ld,
             uint32_t box_rows) {
  EncodeFn fn = encode_fn();
  if (!fn) return set_error(ORION_ERR_BACKEND, "backend cuda failed at tensor map: driver entry point missing");
  const cuuint64_t dims[2] = {k, rows};
  const cuuint64_t strides[1] = {ld * 2};
  const cuuint32_t box[2] = {(cuuint32_t)kSlabK, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides,
                  box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return set_error(ORION_ERR_BACKEND, "backend cuda failed at tensor map: encode returned %d (rows %llu k %llu ld %llu)",
                     (int)r, (unsigned long long)rows, (unsigned long long)k, (unsigned long long)ld);
  return ORION_OK;
}

int cached_map(const void *base, uint64_t rows, uint64_t k, uint64_t ld, uint32_t box_rows, CUtensorMap *out) {
  static ValueCache<std::tuple<const void *, uint64_t, uint64_t, uint64_t, uint32_t>, CUtensorMap> cache(65536);
  return cache.get({base, rows, k, ld, box_rows}, out, [&](CUtensorMap *m) { return make_map(m, base, rows, k, ld, box_rows); });
}

template <bool ACT, int TOKN, int WST, int XST, int MT>
int launch_tc_form(const bf16 *x, uint32_t ldx, const bf16 *w, uint32_t ldw, float *partial, bf16 *act,
              uint32_t rows, uint32_t n, uint32_t k, uint32_t splits, bool cluster_reduce, uint32_t ldc, GemmEpilogue epi,
              cudaStream_t stream, ReadyWait ready, const float *bias) {
  if (ldc == 0) ldc = n;
  if (ldc != n && (splits != 1 || epi == kGemmSwiglu))
    return set_error(ORION_ERR_INTERNAL, "a strided GEMM output needs one k split and no SwiGLU");
  using Cfg = TcConfig<TOKN, WST, XST, MT>;
  static_assert(Cfg::kSmemBytes <= 232448, "ring exceeds the shared memory of an SM");
  if (MT > 1 && cluster_reduce) return set_error(ORION_ERR_INTERNAL, "cluster split-K is built for one weight tile per CTA");
  static bool attr_set[kMaxDeviceOrdinals] = {};
  ORION_CUDA_CHECK("gemm_tc attr", ensure_dynamic_smem(gemm_tc_kernel<TOKN, WST, XST, MT, ACT>, Cfg::kSmemBytes, attr_set));
  CUtensorMap mw, mx;
  ORION_TRY(cached_map(w, n, k, ldw, kTileN, &mw));
  ORION_TRY(cached_map(x, rows, k, ldx, TOKN, &mx));
  dim3 grid((n + MT * kTileN - 1) / (MT * kTileN), (rows + TOKN - 1) / TOKN, splits);
  if (cluster_reduce)
    ORION_CUDA_CHECK("gemm_tc", launch_pdl_cluster(gemm_tc_kernel<TOKN, WST, XST, MT, ACT>, grid, dim3(kThreads), dim3(1, 1, splits),
                                                   Cfg::kSmemBytes, stream, mw, mx, partial, act, rows, n, k, splits,
                                                   1u, ldc, (uint32_t)epi, ready, bias));
  else
    ORION_CUDA_CHECK("gemm_tc", launch_pdl(gemm_tc_kernel<TOKN, WST, XST, MT, ACT>, grid, dim3(kThreads), Cfg::kSmemBytes, stream,
                                           mw, mx, partial, act, rows, n, k, splits, 0u, ldc, (uint32_t)epi, ready, bias));
  count_launch();
  ORION_CUDA_CHECK("gemm_tc", cudaGetLastError());
  return ORION_OK;
}

template <int TOKN, int WST, int XST, int MT = 1>
int launch_tc(const bf16 *x, uint32_t ldx, const bf16 *w, uint32_t ldw, float *partial, bf16 *act, uint32_t rows, uint32_t n,
              uint32_t k, uint32_t splits, bool cluster_reduce, uint32_t ldc, GemmEpilogue epi, cudaStream_t stream, ReadyWait ready,
              const float *bias) {
  auto form = epi == kGemmGelu || epi == kGemmStore || epi == kGemmRelu2 || epi == kGemmGeglu ? launch_tc_form<true, TOKN, WST, XST, MT>
                                                    : launch_tc_form<false, TOKN, WST, XST, MT>;
  return form(x, ldx, w, ldw, partial, act, rows, n, k, splits, cluster_reduce, ldc, epi, stream, ready, bias);
}

// How a projection of many rows is cut for the persistent pairs: 74 pairs take the tiles (and k splits) round by round, so the time is the number of
// rounds times a tile's. Unit: 1.14 ns, what one token column costs a k slab of 64. A slab takes the tensor cores tokn + 16 units (measured 311 ns
// with 256 tokens, 162 with 128, few tiles at work), and with all pairs at work the loads of 256 + tokn rows, which reach shared memory at 14 TB/s in
// all (359-399 ns with 256 tokens, 285-308 with 192, 240-255 with 128). About 3 us for the last tile's epilogue; the consumer reads every k split's
// slab again. Against a sweep of 22 shapes of 300 to 7006 rows, every tile and 1 to 4 splits, the choice is 1.8 % off the best on average.
uint32_t pair_tiles(uint32_t rows, uint32_t n, uint32_t tokn) { return (n + 2 * kTileN - 1) / (2 * kTileN) * ((rows + tokn - 1) / tokn); }
// A last round that is nearly empty costs as much as a full one: its tiles are cut into `tail` pieces of tokn / tail tokens each, so that all pairs have
// work (512 rows of the 8B shape's gate/up: 224 tiles are three rounds and two tiles; those go as 16 pieces of 32 tokens, 101 -> 95 us).
struct PairPlan {
  uint32_t tokn = PairConfig::kMaxTokens, tail = 1;
  uint64_t cost = ~0ull;
};
PairPlan pair_plan(uint32_t rows, uint32_t n, uint32_t k, uint32_t splits) {
  const uint64_t stages = (k + PairConfig::kStageK - 1) / PairConfig::kStageK, slabs = 2 * ((stages + splits - 1) / splits);
  auto round = [&](uint64_t busy, uint32_t cols) { return slabs * std::max<uint64_t>(cols + 16, busy * (2 * kTileN + cols) / 128) + 2 * cols; };
  PairPlan best;
  for (uint32_t t = PairConfig::kMaxTokens; t >= 128; t -= 32) {  // a pair's MMA takes multiples of 32 columns
    const uint64_t tiles = (uint64_t)pair_tiles(rows, n, t) * splits, rest = tiles % kPairs, full = tiles / kPairs * round(kPairs, t);
    for (uint32_t s = 1; s <= t / 32; ++s) {
      if (t / 32 % s || (s > 1 && (rest == 0 || rest * s > kPairs))) continue;
      const uint64_t cost = full + (rest ? round(rest * s, t / s) : 0) + 9 * (t / s) + (uint64_t)(splits - 1) * ((rows + 15) / 16 * 16) * n / 1300;
      if (cost < best.cost) best = {t, s, cost};
    }
  }
  return best;
}
// A k split has to gain a tenth: it keeps an activation out of the epilogue. Two full rounds and more are never split. The same for all row counts
// of a run 16 j + 1 .. 16 (j + 1), since token tiles are multiples of 32.
uint32_t pair_splits(uint32_t rows, uint32_t n, uint32_t k) {
  const uint32_t tiles = pair_tiles(rows, n, PairConfig::kMaxTokens);
  uint32_t best = 1;
  if (tiles > 2 * kPairs) return best;
  // One weight tile is mostly latency, and slabs of so few columns cost little: up to four splits of 512 k and more while half of the pairs are
  // enough for them. k 2048, 16 rows of weights and the norm that reads the result: 1280 tokens 10.7 -> 9.8 us, 2048 tokens 13.5 -> 11.1.
  if (n <= (uint32_t)kTileN) return std::max(1u, std::min({4u, k / (8 * kSlabK), kPairs / 2 / tiles}));
  uint64_t cost = pair_plan(rows, n, k, 1).cost * 9 / 10;
  for (uint32_t s = 2; s <= 4 && k / s >= 8 * kSlabK; ++s) {
    const uint64_t c = pair_plan(rows, n, k, s).cost;
    if (c < cost) best = s, cost = c;
  }
  return best;
}

template <GemmEpilogue OUT>
int launch_pair_form(const bf16 *x, uint32_t ldx, const bf16 *w, uint32_t ldw, float *partial, bf16 *act, uint32_t rows, uint32_t n, uint32_t k,
                     uint32_t splits, uint32_t ldc, cudaStream_t stream, ReadyWait ready, const float *bias) {
  if (ldc == 0) ldc = n;
  if (ldc != n && (splits != 1 || OUT == kGemmSwiglu))
    return set_error(ORION_ERR_INTERNAL, "a strided GEMM output needs one k split and no SwiGLU");
  using Cfg = PairConfig;
  static bool attr_set[kMaxDeviceOrdinals] = {};
  ORION_CUDA_CHECK("gemm_pair attr", ensure_dynamic_smem(gemm_pair_kernel<OUT>, Cfg::kSmemBytes, attr_set));
  const PairPlan plan = pair_plan(rows, n, k, splits);
  const uint32_t tokn = plan.tokn, tiles = pair_tiles(rows, n, tokn) * splits, whole = plan.tail > 1 ? tiles / kPairs * kPairs : tiles;
  CUtensorMap mw, mx, mt;
  ORION_TRY(cached_map(w, n, k, ldw, kTileN, &mw));
  ORION_TRY(cached_map(x, rows, k, ldx, tokn / 2, &mx));
  mt = mx;
  if (plan.tail > 1) ORION_TRY(cached_map(x, rows, k, ldx, tokn / plan.tail / 2, &mt));
  const uint32_t jobs = whole + (tiles - whole) * plan.tail;
  ORION_CUDA_CHECK("gemm_pair", launch_pdl_cluster(gemm_pair_kernel<OUT>, dim3(2 * std::min(jobs, kPairs)), dim3(Cfg::kThreads), dim3(2, 1, 1), Cfg::kSmemBytes,
                                                   stream, mw, mx, mt, partial, act, rows, n, k, splits, tokn, whole, plan.tail, ldc, ready, bias));
  count_launch();
  ORION_CUDA_CHECK("gemm_pair", cudaGetLastError());
  return ORION_OK;
}

int launch_pair(const bf16 *x, uint32_t ldx, const bf16 *w, uint32_t ldw, float *partial, bf16 *act, uint32_t rows, uint32_t n, uint32_t k,
                uint32_t splits, uint32_t ldc, GemmEpilogue epi, cudaStream_t stream, ReadyWait ready, const float *bias) {
  auto form = epi == kGemmPartials ? launch_pair_form<kGemmPartials>
              : epi == kGemmSwiglu ? launch_pair_form<kGemmSwiglu>
              : epi == kGemmGelu   ? launch_pair_form<kGemmGelu>
              : epi == kGemmRelu2  ? launch_pair_form<kGemmRelu2>
              : epi == kGemmGeglu  ? launch_pair_form<kGemmGeglu>
                                   : launch_pair_form<kGemmStore>;
  return form(x, ldx, w, ldw, partial, act, rows, n, k, splits, ldc, stream, ready, bias);
}

// Who takes the persistent pairs: batches of more than 256 rows, with ORION_GEMM_PAIR=2 of more than 128 (the parity tests run this). The four
// projections of the 8B shape at 512 / 2048 / 8192 rows, f32 out: 188 / 611 / 2380 us with pairs, 239 / 775 / 2540 with one CTA per 256-token tile. At 129 to
// 256 rows the two are equal: the wider gate/up 3-6 % slower with pairs, the others 5-13 % faster.
// Matrices of one weight tile (routers) are the exception: the second CTA of a pair has nothing but padding, and with more than kRouterRows tokens single
// CTAs are faster. 16 rows of k 2048 and the norm that reads the result, 2048 / 3000 / 4096 / 8192 tokens: single CTAs 12.0 / 12.6 / 13.6 / 19.5 us, pairs
// with the best k splits 11.1 / 12.8 / 15.3 / 23.1; 64 rows of k 4096: 14.7 / 15.4 / 16.3 / 21.4 and 12.2 / 14.6 / 17.3 / 25.3.
const uint32_t g_pair_rows = std::getenv("ORION_GEMM_PAIR") && std::atoi(std::getenv("ORION_GEMM_PAIR")) >= 2 ? 128 : 256;
constexpr uint32_t kRouterRows = 3072;
bool takes_pairs(uint32_t rows, uint32_t n) { return rows > g_pair_rows && (n > (uint32_t)kTileN || rows <= kRouterRows); }

// Batches of 129..256 rows stream weights like decode but already feel the fill rate (48 KiB of operands per
// 4.2 MFLOP with one weight tile): ORION_GEMM_MID_MT=2 (default) gives a CTA two weight tiles there, 1 one.
int g_mid_mt = std::getenv("ORION_GEMM_MID_MT") ? std::atoi(std::getenv("ORION_GEMM_MID_MT")) : 2;
uint32_t weight_tiles_per_cta(uint32_t rows, uint32_t n) { return rows > 128 && rows <= 256 && g_mid_mt >= 2 && n >= 2 * (uint32_t)kTileN ? 2 : 1; }
int g_small_stages = 5;  // 5: deep weight ring + short activation ring for decode batches; 4: equal rings
// Batches of 65..128 rows: 0 (default) = 4 weight + 2 activation stages, 96 KiB, two CTAs per SM like the
// smaller tiles (the split-K planner counts on two); 1 = 6 + 6 stages, 192 KiB, one CTA per SM, k splits
// sized for one wave of 148; 2 = the same tile with k splits sized for 296 CTAs, also for 129..256 rows
// (two waves of uneven length). ORION_GEMM_MID_TILE overrides (tuning A/B).
int g_mid_tile = std::getenv("ORION_GEMM_MID_TILE") ? std::atoi(std::getenv("ORION_GEMM_MID_TILE")) : 0;

uint32_t token_tile(uint32_t rows) {
  if (rows <= 16) return 16;
  if (rows <= 32) return 32;
  if (rows <= 64) return 64;
  if (rows <= 128) return 128;
  return 256;
}

}  // namespace

bool gemm_tc_supported(uint32_t rows, uint32_t n, uint32_t k, uint32_t ldx, uint32_t ldw,
                       const void *x, const void *w) {
  return rows > 0 && n > 0 && k >= (uint32_t)kSlabK && k % 8 == 0 && ldx % 8 == 0 && ldw % 8 == 0 &&
         (reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0 &&
         encode_fn() != nullptr;
}

int launch_gemm_tc(const bf16 *x, uint32_t ldx, const bf16 *w, uint32_t ldw, float *partial,
                   uint32_t rows, uint32_t n, uint32_t k, uint32_t splits, cudaStream_t stream,
                   bf16 *act, bool cluster_reduce, uint32_t ldc, ReadyWait ready, GemmEpilogue epi, const float *bias) {
  const uint32_t nkb = (k + kSlabK - 1) / kSlabK;
  if (cluster_reduce && (splits < 2 || splits > 8 || act != nullptr))
    return set_error(ORION_ERR_INTERNAL, "cluster split-K needs 2..8 splits and f32 output");
  if ((epi == kGemmSwiglu || epi == kGemmGeglu) && (splits != 1 || n % 2 != 0))
    return set_error(ORION_ERR_INTERNAL, "a gated epilogue needs one k split and an even row count");
  if ((act != nullptr) != (epi != kGemmPartials) || (act != nullptr && splits != 1))
    return set_error(ORION_ERR_INTERNAL, "a GEMM epilogue that stores activations needs one k split and a place for them");
  if (splits < 1 || splits > nkb)
    return set_error(ORION_ERR_INTERNAL, "gemm split count %u outside 1..%u", splits, nkb);
  const bool deep = g_small_stages >= 5;
  const uint32_t tt = token_tile(rows);
  if (takes_pairs(rows, n) && !cluster_reduce) {
    if (splits > (k + PairConfig::kStageK - 1) / PairConfig::kStageK) return set_error(ORION_ERR_INTERNAL, "gemm split count %u leaves a split empty", splits);
    return launch_pair(x, ldx, w, ldw, partial, act, rows, n, k, splits, ldc, epi, stream, ready, bias);
  }
  switch (tt) {
    case 16:
      return deep ? launch_tc<16, 6, 3>(x, ldx, w, ldw, partial, act, rows, n, k, splits, cluster_reduce, ldc, epi, stream, ready, bias)
                  : launch_tc<16, 5, 3>(x, ldx, w, ldw, partial, act, rows, n, k, splits, cluster_reduce, ldc, epi, stream, ready, bias);
    case 32:
      return deep ? launch_tc<32, 6, 3>(x, ldx, w, ldw, partial, act, rows, n, k, splits, cluster_reduce, ldc, epi, stream, ready, bias)
                  : launch_tc<32, 5, 3>(x, ldx, w, ldw, partial, act, rows, n, k, splits, cluster_reduce, ldc, epi, stream, ready, bias);
    case 64:
      return deep ? launch_tc<64, 5, 3>(x, ldx, w, ldw, partial, act, rows, n, k, splits, cluster_reduce, ldc, epi, stream, ready, bias)
                  : launch_tc<64, 4, 4>(x, ldx, w, ldw, partial, act, rows, n, k, splits, cluster_reduce, ldc, epi, stream, ready, bias);
    case 128:
      return g_mid_tile == 0
                 ? launch_tc<128, 4, 2>(x, ldx, w, ldw, partial, act, rows, n, k, splits, cluster_reduce, ldc, epi, stream, ready, bias)
                 : launch_tc<128, 6, 6>(x, ldx, w, ldw, partial, act, rows, n, k, splits, cluster_reduce, ldc, epi, stream, ready, bias);
    default: {
      const uint32_t mt = cluster_reduce ? 1 : weight_tiles_per_cta(rows, n);
      return mt == 2 ? launch_tc<256, 3, 3, 2>(x, ldx, w, ldw, partial, act, rows, n, k, splits, cluster_reduce, ldc, epi, stream, ready, bias)
                     : launch_tc<256, 4, 4>(x, ldx, w, ldw, partial, act, rows, n, k, splits, cluster_reduce, ldc, epi, stream, ready, bias);
    }
  }
}

const void *gemm_tc_error_word() { return device_symbol(g_gemm_error); }

int gemm_tc_poll_error(uint32_t *code) {
#ifdef ORION_TRACE
  static const bool tracing = std::getenv("ORION_GEMM_TRACE") != nullptr &&
                              (std::getenv("LOCAL_RANK") == nullptr || std::atoi(std::getenv("LOCAL_RANK")) == 0);  // one rank prints
  if (tracing) {
    static unsigned long long t[kTraceLaunches][kTraceStamps];
    uint32_t next = 0, on = 1;
    cudaMemcpyFromSymbol(t, g_gemm_trace, sizeof t);
    cudaMemcpyFromSymbol(&next, g_gemm_trace_next, sizeof next);
    cudaMemcpyToSymbol(g_gemm_trace_on, &on, sizeof on);
    if (next >= (uint32_t)kTraceLaunches) {
      unsigned long long prev_end = 0;
      fprintf(stderr, "gemm trace of CTA 0 (us): entry(abs mod 1e5) grid.x splits slabs | gap-from-prev-end setup first-W pdl-wait last-mma acc-ready epilogue total\n");
      for (int i = 0; i < kTraceLaunches; ++i) {
        const unsigned long long *r = t[(next + i) % kTraceLaunches];
        fprintf(stderr, "  gemm %10.2f %4u %2u %3u | %7.2f %6.2f %6.2f %6.2f %6.2f %6.2f %6.2f %6.2f\n", (double)(r[0] % 100000000ull) / 1e3, (unsigned)(r[7] >> 32),
                (unsigned)((r[7] >> 16) & 0xFFFF), (unsigned)(r[7] & 0xFFFF), prev_end ? ((double)r[0] - (double)prev_end) / 1e3 : 0.0,
                (r[1] - r[0]) / 1e3, (r[2] - r[0]) / 1e3, (r[3] - r[0]) / 1e3, (r[4] - r[0]) / 1e3, (r[5] - r[0]) / 1e3,
                (r[6] - r[0]) / 1e3, (r[6] - r[0]) / 1e3);
        prev_end = r[6];
      }
    }
  }
#endif
  uint32_t v = 0;
  ORION_CUDA_CHECK("gemm error word", cudaMemcpyFromSymbol(&v, g_gemm_error, sizeof v));
  if (v) {
    uint32_t zero = 0;
    ORION_CUDA_CHECK("gemm error word", cudaMemcpyToSymbol(g_gemm_error, &zero, sizeof zero));
  }
  *code = v;
  return ORION_OK;
}

// ---- planning and dispatch -------------------------------------------------------

namespace {
uint32_t g_target_ctas = 296;  // two CTAs fit on each of the 148 SMs
// Split-K reduction inside a thread-block cluster (distributed shared memory) instead of one f32
// slab per split summed by the consumer. Off by default: measured on the headline step it removes
// 8/9 of the slab traffic but costs more than it saves (5.27 vs 5.01 ms per step): clusters of 8
// CTAs of 105 KiB must be co-scheduled, which delays the dependent-launch overlap, and each GEMM
// gains two cluster barriers. ORION_CLUSTER_SPLITK=1 turns it on (tests cover both).
bool g_cluster_splitk = std::getenv("ORION_CLUSTER_SPLITK") ? std::atoi(std::getenv("ORION_CLUSTER_SPLITK")) != 0 : false;
}

void gemm_set_target_ctas(uint32_t v) { g_target_ctas = v ? v : 296; }
void gemm_set_small_stages(int stages) { g_small_stages = stages >= 5 ? 5 : 4; }

GemmPlan gemm_plan(bool is_bf16, uint32_t rows, uint32_t n, uint32_t k, uint32_t ldx,
                   uint32_t ldw) {
  GemmPlan p{1, false, false, 1, 0};
  if (!is_bf16) return p;
  // alignment of the pointers is checked at launch; shapes decide the plan
  if (!(rows > 0 && n > 0 && k >= (uint32_t)kSlabK && k % 8 == 0 && ldx % 8 == 0 && ldw % 8 == 0 &&
        encode_fn() != nullptr))
    return p;
  p.tensor_core = true;
  if (takes_pairs(rows, n)) {
    p.splits = p.out_slabs = pair_splits(rows, n, k);
    return p;
  }
  const uint32_t nkb = (k + kSlabK - 1) / kSlabK;
  if (rows > 256) {  // one weight tile and many tokens: up to four k splits of at least eight slabs, in at most two waves
    const uint32_t tiles = (rows + 255) / 256;
    if (tiles < 148) p.splits = p.out_slabs = std::max(1u, std::min({296 / tiles, nkb / 8, 4u}));
    return p;
  }
  const uint32_t rows_per_cta = kTileN * (g_cluster_splitk ? 1 : weight_tiles_per_cta(rows, n));
  const uint32_t tiles = ((n + rows_per_cta - 1) / rows_per_cta) * ((rows + token_tile(rows) - 1) / token_tile(rows));
  // the 256-token tile (and the 6 + 6 stage 128-token one) fills an SM by itself: one wave is 148 CTAs
  const bool one_per_sm = g_mid_tile != 2 && (token_tile(rows) == 256 || (token_tile(rows) == 128 && g_mid_tile == 1));
  uint32_t s = (one_per_sm ? g_target_ctas / 2 : g_target_ctas) / (tiles ? tiles : 1);
  const uint32_t cap = nkb / 4 ? nkb / 4 : 1;  // at least four k slabs per split
  if (s > cap) s = cap;
  if (s > 16) s = 16;
  if (g_cluster_splitk && s > 8) s = 8;  // portable cluster size
  p.splits = s < 1 ? 1 : s;
  p.cluster_reduce = g_cluster_splitk && p.splits > 1;
  p.out_slabs = p.cluster_reduce ? 1 : p.splits;
  return p;
}

size_t gemm_partial_floats(bool is_bf16, uint32_t max_rows, uint32_t n, uint32_t k) {
  size_t best = (size_t)max_rows * n;
  if (!is_bf16) return best;
  for (uint32_t r = 1; r <= max_rows; r = takes_pairs(r, n) && r < max_rows ? std::min(max_rows, (r / 16 + 1) * 16) : r + 1) {  // as in pair_splits
    const GemmPlan p = gemm_plan(true, r, n, k, k, k);
    const size_t need = (size_t)p.splits * r * n;
    if (need > best) best = need;
  }
  return best;
}

int launch_gemm_swiglu(const bf16 *x, uint32_t ldx, const bf16 *w_interleaved, uint32_t ldw, bf16 *act, uint32_t rows,
                       uint32_t ffn, uint32_t k, cudaStream_t stream, ReadyWait ready) {
  if (!gemm_tc_supported(rows, 2 * ffn, k, ldx, ldw, x, w_interleaved))
    return set_error(ORION_ERR_INTERNAL, "tensor-core GEMM planned for an unaligned operand");
  return launch_gemm_tc(x, ldx, w_interleaved, ldw, nullptr, rows, 2 * ffn, k, 1, stream, act, false, 0, ready, kGemmSwiglu);
}

int launch_gemm_act(const bf16 *x, uint32_t ldx, const bf16 *w, uint32_t ldw, bf16 *act, uint32_t ld_act, uint32_t rows, uint32_t n,
                    uint32_t k, GemmEpilogue epi, cudaStream_t stream, const float *bias) {
  if (epi != kGemmGelu && epi != kGemmStore && epi != kGemmRelu2 && epi != kGemmGeglu) return set_error(ORION_ERR_INTERNAL, "not an epilogue of this entry point");
  if (!gemm_tc_supported(rows, n, k, ldx, ldw, x, w))
    return set_error(ORION_ERR_INTERNAL, "tensor-core GEMM planned for an unaligned operand");
  return launch_gemm_tc(x, ldx, w, ldw, nullptr, rows, n, k, 1, stream, act, false, ld_act, ReadyWait{}, epi, bias);
}

template <>
int launch_gemm<float>(const float *x, uint32_t ldx, const float *w, uint32_t ldw, float *partial,
                       uint32_t rows, uint32_t n, uint32_t k, GemmPlan, cudaStream_t stream, ReadyWait) {
  return launch_gemm_simt<float>(x, ldx, w, ldw, partial, rows, n, k, stream);
}

template <>
int launch_gemm<bf16>(const bf16 *x, uint32_t ldx, const bf16 *w, uint32_t ldw, float *partial,
                      uint32_t rows, uint32_t n, uint32_t k, GemmPlan plan, cudaStream_t stream,
                      ReadyWait ready) {
  if (plan.tensor_core) {
    if (!gemm_tc_supported(rows, n, k, ldx, ldw, x, w))
      return set_error(ORION_ERR_INTERNAL, "tensor-core GEMM planned for an unaligned operand");
    return launch_gemm_tc(x, ldx, w, ldw, partial, rows, n, k, plan.splits, stream, nullptr, plan.cluster_reduce,
                          plan.ldc, ready);
  }
  if (plan.ldc != 0 && plan.ldc != n) return set_error(ORION_ERR_INTERNAL, "a strided GEMM output needs the tensor-core path");
  return launch_gemm_simt<bf16>(x, ldx, w, ldw, partial, rows, n, k, stream);
}

}  // namespace orion
