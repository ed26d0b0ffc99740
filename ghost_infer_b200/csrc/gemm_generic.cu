// Plain matrix product on CUDA cores with 32-bit accumulation: out[M,N] (op)= A[M,K] * W[N,K]^T, for any types, sizes and strides.
//
// The true 32-bit path's rows that start on 16-byte boundaries go to gemm_f32.cu; this kernel takes the rest (odd K, rows off such
// boundaries, mixed and 16-bit types) and is the reference beside every faster product.  It has that file's order of
// additions, which follows from K alone: the same bits whichever kernel ran, whatever else is in the batch.  Weights are
// row-major [out, in] without bias, as the reference keeps them (src/model.rs:1019, src/quant.rs:73-78).
//
// Bound by the FFMA pipe where there are many rows, else by the chain over K (load, barrier, multiply).  Operands lie in k order
// in shared memory, rows padded to 20 numbers (eight lanes' 16-byte reads fall into different banks), so that a packed
// multiply-add takes the even and the odd k of two operands at once; two blocks an SM, whose 124 registers let loads and products
// overlap.  32-bit rows off 16-byte boundaries: 300 x 8,192 x 2,047 527 us, 2,000 x 2,048 x 8,191 3.18 ms, one row x 2,048 x
// 2,047 120 us; single multiply-adds, even and odd k in accumulators of their own, 820 us, 4.74 ms and 189 us; one running
// sum over K 696 us, 3.10 ms and 192 us.
#include "api.h"
#include "common.cuh"

namespace {

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4, PITCH = BK + 4;

// (lo, hi) of acc += the products of the halves, each rounded once, as fmaf would
__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float join2(uint64_t v) { return __fadd_rn(__uint_as_float((uint32_t)v), __uint_as_float((uint32_t)(v >> 32))); }

template <typename TA, typename TW, typename TO, int MODE>
__global__ void __launch_bounds__(256, 2)
gemm_tile_kernel(void* __restrict__ out_, const TA* __restrict__ A, const TW* __restrict__ W, int M, int N, int K,
                 long lda, long ldw, long ldo, int seg) {
  __shared__ __align__(16) float As[BM * PITCH];
  __shared__ __align__(16) float Ws[BN * PITCH];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tx = tid % 16, ty = tid / 16;  // thread owns rows ty + 16 i, columns tx + 16 j
  uint64_t acc[TM][TN];                    // (even k, odd k)
  float sum[TM][TN];                       // finished stretches
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0, sum[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
    // 64 rows x 16 k per operand = 1024 elements, 4 per thread; consecutive threads walk k (contiguous)
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int r = (tid >> 4) + 16 * it, k = tid & 15;
      float av = 0.f, wv = 0.f;
      if (m0 + r < M && k0 + k < K) av = gi::ldf(A + (size_t)(m0 + r) * lda + k0 + k);
      if (n0 + r < N && k0 + k < K) wv = gi::ldf(W + (size_t)(n0 + r) * ldw + k0 + k);
      As[r * PITCH + k] = av;
      Ws[r * PITCH + k] = wv;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; k += 4) {
      ulonglong2 w[TN];
#pragma unroll
      for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(Ws + (tx + 16 * j) * PITCH + k);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(As + (ty + 16 * i) * PITCH + k);
#pragma unroll
        for (int j = 0; j < TN; ++j) fma2(acc[i][j], a.x, w[j].x);
#pragma unroll
        for (int j = 0; j < TN; ++j) fma2(acc[i][j], a.y, w[j].y);
      }
    }
    __syncthreads();
    if ((k0 + BK) % seg == 0 || k0 + BK >= K) {  // a stretch ends
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          sum[i][j] = __fadd_rn(sum[i][j], join2(acc[i][j]));
          acc[i][j] = 0;
        }
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty + 16 * i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx + 16 * j;
      if (n >= N) continue;
      if (MODE == GI_GEMM_ACCUM_F32) {
        float* o = (float*)out_ + (size_t)m * ldo + n;
        *o = *o + sum[i][j];
      } else {
        gi::stf((TO*)out_ + (size_t)m * ldo + n, sum[i][j]);
      }
    }
  }
}

template <typename TA, typename TW>
int launch(void* out, int out_dtype, int mode, const void* A, const void* W, int M, int N, int K, long lda, long ldw,
           long ldo, cudaStream_t s) {
  const int seg = gi::sum_segment(K);
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (mode == GI_GEMM_ACCUM_F32) {
    gemm_tile_kernel<TA, TW, float, GI_GEMM_ACCUM_F32><<<grid, 256, 0, s>>>(out, (const TA*)A, (const TW*)W, M, N, K, lda, ldw, ldo, seg);
  } else if (out_dtype == GI_F32) {
    gemm_tile_kernel<TA, TW, float, GI_GEMM_STORE><<<grid, 256, 0, s>>>(out, (const TA*)A, (const TW*)W, M, N, K, lda, ldw, ldo, seg);
  } else {
    gemm_tile_kernel<TA, TW, __nv_bfloat16, GI_GEMM_STORE><<<grid, 256, 0, s>>>(out, (const TA*)A, (const TW*)W, M, N, K, lda, ldw, ldo, seg);
  }
  return gi::check_launch("gemm_generic");
}

}  // namespace

extern "C" int gi_gemm_generic(void* out, int out_dtype, int mode, const void* A, int a_dtype, const void* W,
                               int w_dtype, int M, int N, int K, long lda, long ldw, long ldo, void* stream) {
  if (M <= 0 || N <= 0) return GI_OK;
  if (K <= 0) return gi::fail(GI_ERR_ARG, "gemm: K must be positive, got %d", K);
  if (mode != GI_GEMM_STORE && mode != GI_GEMM_ACCUM_F32) return gi::fail(GI_ERR_ARG, "gemm: unknown mode %d", mode);
  if (mode == GI_GEMM_ACCUM_F32 && out_dtype != GI_F32) return gi::fail(GI_ERR_ARG, "gemm: accumulation needs a float output");
  if ((N + BN - 1) / BN > 2147483647 || (M + BM - 1) / BM > 65535)
    return gi::fail(GI_ERR_UNSUPPORTED, "gemm: %d rows are more than one launch takes (%d)", M, 65535 * BM);
  if (a_dtype == GI_F32 && w_dtype == GI_F32 && out_dtype == GI_F32 && gi::gemm_f32_takes(A, W, N, K, lda, ldw))
    return gi::gemm_f32((float*)out, mode == GI_GEMM_ACCUM_F32, (const float*)A, (const float*)W, M, N, K, lda, ldw, ldo, (cudaStream_t)stream);
  GI_DISPATCH_DTYPE(a_dtype, TA, GI_DISPATCH_DTYPE(w_dtype, TW,
      return (launch<TA, TW>(out, out_dtype, mode, A, W, M, N, K, lda, ldw, ldo, (cudaStream_t)stream))));
  return GI_OK;
}
