// SIMT GEMM  out[r][n] = sum_k x[r][k] * w[n][k]  (tensor.rs:114-128 without bias).
//
// This is the arithmetic of the f32 correctness build and the fallback for bf16
// shapes the tensor-core kernel does not take (K not a multiple of 8, unaligned
// rows). Every output element is accumulated by ONE thread with k ascending;
// for f32 storage the multiply and the add are rounded separately (no FMA), so
// the result equals the reference's `acc += a * b` loop bit for bit.
#include "kernels.h"

namespace orion {
namespace {

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

template <typename T>
__device__ __forceinline__ float mac(float acc, float a, float b);
template <>
__device__ __forceinline__ float mac<float>(float acc, float a, float b) {
  return __fadd_rn(acc, __fmul_rn(a, b));
}
template <>
__device__ __forceinline__ float mac<bf16>(float acc, float a, float b) {
  return fmaf(a, b, acc);
}

template <typename T>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const T *__restrict__ x, uint32_t ldx, const T *__restrict__ w, uint32_t ldw,
                 float *__restrict__ out, uint32_t M, uint32_t N, uint32_t K) {
  __shared__ float xs[BK][BM + 1];
  __shared__ float ws[BK][BN + 1];
  pdl_trigger();
  pdl_wait();
  const uint32_t m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const uint32_t tx = threadIdx.x % 16, ty = threadIdx.x / 16;  // tx -> n, ty -> m
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;

  for (uint32_t k0 = 0; k0 < K; k0 += BK) {
    for (uint32_t idx = threadIdx.x; idx < BM * BK; idx += 256) {
      const uint32_t r = idx / BK, kk = idx % BK;
      const uint32_t gm = m0 + r, gk = k0 + kk;
      xs[kk][r] = (gm < M && gk < K) ? to_f32<T>(x[(size_t)gm * ldx + gk]) : 0.0f;
    }
    for (uint32_t idx = threadIdx.x; idx < BN * BK; idx += 256) {
      const uint32_t r = idx / BK, kk = idx % BK;
      const uint32_t gn = n0 + r, gk = k0 + kk;
      ws[kk][r] = (gn < N && gk < K) ? to_f32<T>(w[(size_t)gn * ldw + gk]) : 0.0f;
    }
    __syncthreads();
    const uint32_t kmax = min((uint32_t)BK, K - k0);  // never accumulate padded k (keeps -0.0 exact)
    for (uint32_t kk = 0; kk < kmax; ++kk) {
      float a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = xs[kk][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = ws[kk][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = mac<T>(acc[i][j], a[i], b[j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const uint32_t gm = m0 + ty * TM + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const uint32_t gn = n0 + tx * TN + j;
      if (gn < N) out[(size_t)gm * N + gn] = acc[i][j];
    }
  }
}

// The same arithmetic for the few rows of a decode step of the f32 build, where the kernel above is a chain of exposed latencies: a tile of 64 x 64
// leaves most of its threads on rows that are not there, and every 16 k wait for their loads. Here a thread has one output, a CTA eight rows x 16
// outputs (16 CTAs for 256 outputs, 86 for 1376), and the k slabs arrive by asynchronous copies kStages ahead. What remains is mostly the chain of
// k dependent additions, which the order of the sum asks for. 8 rows: 67 -> 5 us with k 688 and 256 outputs, 35 -> 3.4 with k 256 and 1024 outputs.
constexpr uint32_t kFewRows = 8, kFewCols = 16, kFewK = 128, kFewStages = 3, kFewPitch = kFewK + 4;  // + 4: rows of a quarter warp on different banks

__device__ __forceinline__ void copy16(float *dst, const float *src, bool real) {  // zeros where there is nothing to copy
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(real ? 16 : 0) : "memory");
}

__global__ void __launch_bounds__(kFewRows * kFewCols)
gemm_simt_few_kernel(const float *__restrict__ x, uint32_t ldx, const float *__restrict__ w, uint32_t ldw, float *__restrict__ out, uint32_t M,
                     uint32_t N, uint32_t K) {
  __shared__ __align__(16) float xs[kFewStages][kFewRows][kFewPitch], ws[kFewStages][kFewCols][kFewPitch];
  constexpr uint32_t kThreads = kFewRows * kFewCols, kVec = kFewK / 4;
  pdl_trigger();
  const uint32_t m0 = blockIdx.y * kFewRows, n0 = blockIdx.x * kFewCols, tn = threadIdx.x % kFewCols, tm = threadIdx.x / kFewCols;
  const uint32_t slabs = (K + kFewK - 1) / kFewK;
  auto load_w = [&](uint32_t i) {
#pragma unroll
    for (uint32_t v = threadIdx.x; v < kFewCols * kVec; v += kThreads) {
      const uint32_t r = v / kVec, c = v % kVec * 4, k = i * kFewK + c;
      const bool real = n0 + r < N && k < K;
      copy16(&ws[i % kFewStages][r][c], real ? w + (size_t)(n0 + r) * ldw + k : w, real);
    }
  };
  auto load_x = [&](uint32_t i) {
#pragma unroll
    for (uint32_t v = threadIdx.x; v < kFewRows * kVec; v += kThreads) {
      const uint32_t r = v / kVec, c = v % kVec * 4, k = i * kFewK + c;
      const bool real = m0 + r < M && k < K;
      copy16(&xs[i % kFewStages][r][c], real ? x + (size_t)(m0 + r) * ldx + k : x, real);
    }
  };
  // weights are immutable: the first slabs' are asked for before the wait for the kernel that makes x
  for (uint32_t i = 0; i < kFewStages - 1 && i < slabs; ++i) load_w(i);
  pdl_wait();
  for (uint32_t i = 0; i < kFewStages - 1; ++i) {
    if (i < slabs) load_x(i);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  float acc = 0.0f;
  for (uint32_t i = 0; i < slabs; ++i) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kFewStages - 2) : "memory");
    __syncthreads();  // slab i has arrived for everyone, and everyone has read the one that the next copies replace
    if (i + kFewStages - 1 < slabs) {
      load_w(i + kFewStages - 1);
      load_x(i + kFewStages - 1);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float *xr = xs[i % kFewStages][tm], *wr = ws[i % kFewStages][tn];
    const uint32_t n = min(kFewK, K - i * kFewK);  // never a padded k (keeps -0.0 exact)
#pragma unroll 8
    for (uint32_t k = 0; k < n; k += 4) {
      const float4 a = *reinterpret_cast<const float4 *>(xr + k), b = *reinterpret_cast<const float4 *>(wr + k);
      acc = mac<float>(acc, a.x, b.x);
      acc = mac<float>(acc, a.y, b.y);
      acc = mac<float>(acc, a.z, b.z);
      acc = mac<float>(acc, a.w, b.w);
    }
  }
  if (m0 + tm < M && n0 + tn < N) out[(size_t)(m0 + tm) * N + n0 + tn] = acc;
}

}  // namespace

template <typename T>
int launch_gemm_simt(const T *x, uint32_t ldx, const T *w, uint32_t ldw, float *out, uint32_t rows,
                     uint32_t n, uint32_t k, cudaStream_t stream) {
  if (rows == 0 || n == 0) return ORION_OK;
  if constexpr (sizeof(T) == 4) {
    // Decode batches. The 4 x 4 outputs of a thread above need a quarter of the shared-memory reads, so that kernel wins where it fills the chip: with more
    // than 32 rows against many outputs (the head of a large vocabulary). Few / tile, us, with k 256: 16384 outputs and 64 rows 55 / 61; 28000 outputs
    // 59 / 65 with 40 rows, 70 / 66 with 48, 92 / 69 with 64; 128256 outputs 209 / 233 with 32 rows, 259 / 235 with 40, 411 / 240 with 64; k 4096, 14336
    // outputs and 64 rows 716 / 1152.
    const bool few_rows = rows <= 32 || (rows <= 64 && (uint64_t)((rows + 7) / 8 * 8) * n < 1300000);
    if (few_rows && k % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) == 0) {
      const dim3 few((n + kFewCols - 1) / kFewCols, (rows + kFewRows - 1) / kFewRows);
      ORION_CUDA_CHECK("gemm_simt", launch_pdl(gemm_simt_few_kernel, few, dim3(kFewRows * kFewCols), 0, stream, x, ldx, w, ldw, out, rows, n, k));
      count_launch();
      ORION_CUDA_CHECK("gemm_simt", cudaGetLastError());
      return ORION_OK;
    }
  }
  dim3 grid((n + BN - 1) / BN, (rows + BM - 1) / BM);
  ORION_CUDA_CHECK("gemm_simt", launch_pdl(gemm_simt_kernel<T>, grid, dim3(256), 0, stream, x, ldx, w, ldw, out,
                                           rows, n, k));
  count_launch();
  ORION_CUDA_CHECK("gemm_simt", cudaGetLastError());
  return ORION_OK;
}
template int launch_gemm_simt<float>(const float *, uint32_t, const float *, uint32_t, float *,
                                     uint32_t, uint32_t, uint32_t, cudaStream_t);
template int launch_gemm_simt<bf16>(const bf16 *, uint32_t, const bf16 *, uint32_t, float *,
                                    uint32_t, uint32_t, uint32_t, cudaStream_t);

}  // namespace orion
