// The products of the true 32-bit path where rows are 16-byte aligned: out[M,N] (op)= A[M,K] * W[N,K]^T, all float, FFMA
// only.  gi_gemm_generic sends such operands here and keeps its own kernel for the rest.  (Prompt steps' products of larger matrices go to
// gemm_f32_split.cu; steps of one token a sequence and smaller matrices come here.)
//
// One order of additions serves every kernel of the 32-bit path, so that a token's bits do not depend on which of them
// ran: K is cut into SUM_SEGMENTS stretches of gi::sum_segment(K) numbers (it follows from K alone); in a stretch the
// even and the odd k are summed each in k order by fused multiply-adds from zero (the two halves of a packed
// multiply-add, which needs fewer issue slots and register reads than two single ones), the two are added, and the
// stretches' sums are added in their order.  (One running sum over all of K, the order before, leaves no parallelism
// but the outputs, and its error grows with K instead of K / 64.)
//
// few_rows (a decode step): bound by the bytes of W.  A block walks 16-row tiles of W, the 32 stretches of a row side by
// side: lane = (one of 4 groups of rows, one of 8 stretches), so each thread sums whole stretches in order and 256
// threads share a tile that K alone would leave to 16 x M threads.  W arrives by cp.async in pieces of 16 numbers of
// every stretch, each stretch padded to 20 so that eight lanes' 16-byte reads fall into different banks.
// (Two blocks per SM with 8 rows each were slower: a stage's fixed costs are then paid twice as often.)  L2 is asked for the first tile before the dependency
// wait (a prefetch reads no values, so it is right whoever wrote W).
// B200, repeated launches, 16,384 x 2,048 (134 MB): M = 1 30.5 us, M = 4 33.0 us (4.1 TB/s), M = 16 65 us, which is bound by
// the shared memory reads of the tokens; 128,256 x 2,048, M = 4: 226 us (4.65 TB/s).  The tiled kernel that served these
// before took 844 us on average over a decode step's products of a 1B model (a 64-row tile for 4 rows, a fifth of the SMs).
//
// many_rows (a prompt): bound by the FFMA pipe (72 TFLOP/s at the maximum clock, 54-63 with three different operands).
// Tiles of 32 (to 48) x 128, 8 (to 12) x 4 outputs a thread, operands kept in k order in shared memory (rows padded to 36 numbers) and read
// 16 bytes at a time, a warp's lanes along the columns so that a row's number is one broadcast; three blocks per SM:
// small tiles because 600 rows x 2,048 columns are only 80 tiles of 128 x 128.  600 rows: 16,384 x 2,048 956 us (42 TFLOP/s;
// single multiply-adds in 64 x 64 tiles 1,079 us, the kernel before 2,480 us), 2,048 x 2,048 142 us in tiles
// of 36 rows, 184 us in tiles of 32 (three on the fullest SM where 2.05 would do; single multiply-adds in 64 x 64 tiles 245 us,
// the kernel before 300 us).
#include "api.h"
#include "common.cuh"

namespace {

using gi::SUM_SEGMENTS;

__device__ __forceinline__ void cp16(void* dst, const float* src, bool valid) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int n = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// (lo, hi) of acc += the products of the halves, each rounded once, as fmaf would
__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float join2(uint64_t v) { return __fadd_rn(__uint_as_float((uint32_t)v), __uint_as_float((uint32_t)(v >> 32))); }

constexpr int PIECE = 16, PITCH = PIECE + 4;                 // numbers of a stretch a stage, padded
constexpr int LINE = SUM_SEGMENTS * PITCH;                   // floats of one row in a stage
constexpr int FEW_THREADS = 256;

constexpr int ROWS = 16;                                     // rows of W a tile
template <int MT> constexpr int FEW_STAGES = MT <= 4 ? 4 : (MT <= 8 ? 3 : 2);
template <int MT>
constexpr size_t FEW_SMEM = sizeof(float) * ((size_t)FEW_STAGES<MT> * (ROWS + MT) * LINE + SUM_SEGMENTS * (ROWS * MT + 1));

// MT tokens a block (blockIdx.y picks them).  Up to 8 tokens the two halves of the warps take 8 rows each; with 16 they
// take 8 tokens each and all rows, so that a number read from shared memory serves more products.
template <int MT, bool ACCUM>
__global__ void __launch_bounds__(FEW_THREADS, 1)
few_rows_kernel(float* __restrict__ out, const float* A, const float* W, int M, int N, int K, long lda, long ldw, long ldo, int seg) {
  constexpr int STAGES = FEW_STAGES<MT>;
  constexpr bool SPLIT_TOKENS = MT > 8;
  constexpr int RT = SPLIT_TOKENS ? 4 : 2, TT = SPLIT_TOKENS ? MT / 2 : MT;
  extern __shared__ __align__(16) float smem[];
  float* red = smem + (size_t)STAGES * (ROWS + MT) * LINE;   // [SEGMENTS][ROWS * MT + 1]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int half = warp & 1, s = (warp >> 1) * 8 + (lane & 7), rg = lane >> 3;
  const int row0 = SPLIT_TOKENS ? rg : half * 8 + rg, tok0 = SPLIT_TOKENS ? half * TT : 0;
  const int m0 = blockIdx.y * MT;
  const int n_tiles = (N + ROWS - 1) / ROWS, per_tile = seg / PIECE;
  const int mine = (n_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const int total = mine * per_tile;                         // stages this block works through

  gi::pdl_launch_dependents();
  if (tid < ROWS && (int)blockIdx.x * ROWS + tid < N) {
    const uint32_t bytes = (uint32_t)min(K, 2048) * 4u;      // K % 4 == 0: a multiple of 16
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(W + ((size_t)blockIdx.x * ROWS + tid) * ldw), "r"(bytes) : "memory");
  }
  gi::pdl_wait();

  // thread's part of a stage: 16 bytes q of stretch sg of rows r0, r0 + 2, ...
  const int q = tid & 3, sg = (tid >> 2) & 31, r0 = tid >> 7;
  const int k0 = sg * seg + q * 4;
  const float* x_row = A + (size_t)(m0 + r0) * lda + k0;
  int in_tile = 0, at_stage = 0, left = total, n0 = (int)blockIdx.x * ROWS;       // where the next load stands
  auto load = [&]() {
    if (left > 0) {
      float* st = smem + (size_t)at_stage * (ROWS + MT) * LINE + sg * PITCH + q * 4;
      const bool in_k = k0 + in_tile * PIECE < K;
      const int rows = in_k ? N - n0 - r0 : 0, toks = in_k ? M - m0 - r0 : 0;
      const float* src = W + (size_t)(n0 + r0) * ldw + k0 + in_tile * PIECE;
#pragma unroll
      for (int i = 0; i < ROWS; i += 2, src += 2 * ldw) cp16(st + (r0 + i) * LINE, i < rows ? src : W, i < rows);
      src = x_row + in_tile * PIECE;
#pragma unroll
      for (int i = 0; i < MT; i += 2, src += 2 * lda)
        if (r0 + i < MT) cp16(st + (ROWS + r0 + i) * LINE, i < toks ? src : A, i < toks);
      --left;
      at_stage = at_stage + 1 == STAGES ? 0 : at_stage + 1;
      if (++in_tile == per_tile) in_tile = 0, n0 += (int)gridDim.x * ROWS;
    }
    cp_commit();
  };

  uint64_t acc[RT][TT];                                      // (even k, odd k)
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int t = 0; t < TT; ++t) acc[r][t] = 0;
#pragma unroll
  for (int g = 0; g < STAGES - 1; ++g) load();

  int stage = 0, done = 0, n_out = (int)blockIdx.x * ROWS;
  for (int g = 0; g < total; ++g) {
    cp_wait<STAGES - 2>();
    __syncthreads();
    load();                                                  // into the stage that was read before this barrier
    const float* st = smem + (size_t)stage * (ROWS + MT) * LINE + s * PITCH;
    stage = stage + 1 == STAGES ? 0 : stage + 1;
#pragma unroll
    for (int j = 0; j < PIECE; j += 4) {
      ulonglong2 w[RT];
#pragma unroll
      for (int r = 0; r < RT; ++r) w[r] = *reinterpret_cast<const ulonglong2*>(st + (row0 + 4 * r) * LINE + j);
#pragma unroll
      for (int t = 0; t < TT; ++t) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(st + (ROWS + tok0 + t) * LINE + j);
#pragma unroll
        for (int r = 0; r < RT; ++r) fma2(acc[r][t], x.x, w[r].x);
#pragma unroll
        for (int r = 0; r < RT; ++r) fma2(acc[r][t], x.y, w[r].y);
      }
    }
    if (++done < per_tile) continue;
    done = 0;
    // the tile is summed: stretches meet in shared memory and are added in their order
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
      for (int t = 0; t < TT; ++t) {
        red[s * (ROWS * MT + 1) + (tok0 + t) * ROWS + row0 + 4 * r] = join2(acc[r][t]);
        acc[r][t] = 0;
      }
    __syncthreads();
    if (tid < ROWS * MT) {
      const int n = n_out + tid % ROWS, m = m0 + tid / ROWS;
      float sum = 0.f;
#pragma unroll
      for (int i = 0; i < SUM_SEGMENTS; ++i) sum += red[i * (ROWS * MT + 1) + tid];
      if (n < N && m < M) {
        float* o = out + (size_t)m * ldo + n;
        *o = ACCUM ? *o + sum : sum;
      }
    }
    n_out += (int)gridDim.x * ROWS;
    // `red` is written again only after the next stage's barrier
  }
}

constexpr int BN = 128, BK = 32, TN = 4, KP = BK + 4, MANY_STAGES = 3, MANY_THREADS = 128;
template <int TM>
constexpr size_t MANY_SMEM = sizeof(float) * MANY_STAGES * (4 * TM + BN) * KP;

// TM: rows a thread takes, a tile has 4 TM
template <int TM, bool ACCUM>
__global__ void __launch_bounds__(MANY_THREADS, TM == 8 ? 3 : 2)
many_rows_kernel(float* __restrict__ out, const float* A, const float* W, int M, int N, int K, long lda, long ldw, long ldo, int seg) {
  constexpr int BM = 4 * TM;
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x, tx = tid % 32, ty = tid / 32;  // thread owns rows ty + 4 i, columns tx + 32 j
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int steps = (K + BK - 1) / BK, per_seg = seg / BK;
  gi::pdl_wait();

  const int q = tid % 8, r0 = tid / 8;                       // 16 bytes q of rows r0, r0 + 16, ...
  auto load = [&](int g) {
    if (g < steps) {
      float* st = smem + (size_t)(g % MANY_STAGES) * (BM + BN) * KP + q * 4;
      const int k = g * BK + q * 4;
#pragma unroll
      for (int i = 0; i < (BM + 15) / 16; ++i) {
        const int r = r0 + 16 * i;
        const bool ok = k < K && m0 + r < M;
        if (r < BM) cp16(st + r * KP, ok ? A + (size_t)(m0 + r) * lda + k : A, ok);
      }
#pragma unroll
      for (int i = 0; i < BN / 16; ++i) {
        const int r = r0 + 16 * i;
        const bool ok = k < K && n0 + r < N;
        cp16(st + (BM + r) * KP, ok ? W + (size_t)(n0 + r) * ldw + k : W, ok);
      }
    }
    cp_commit();
  };

  uint64_t acc[TM][TN];                                      // (even k, odd k)
  float sum[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0, sum[i][j] = 0.f;
#pragma unroll
  for (int g = 0; g < MANY_STAGES - 1; ++g) load(g);

  int left = per_seg;
  for (int g = 0; g < steps; ++g) {
    cp_wait<MANY_STAGES - 2>();
    __syncthreads();
    load(g + MANY_STAGES - 1);
    const float* sa = smem + (size_t)(g % MANY_STAGES) * (BM + BN) * KP + ty * KP;
    const float* sw = smem + (size_t)(g % MANY_STAGES) * (BM + BN) * KP + (BM + tx) * KP;
#pragma unroll
    for (int k = 0; k < BK; k += 4) {
      ulonglong2 w[TN];
#pragma unroll
      for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(sw + 32 * j * KP + k);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(sa + 4 * i * KP + k);
#pragma unroll
        for (int j = 0; j < TN; ++j) fma2(acc[i][j], a.x, w[j].x);
#pragma unroll
        for (int j = 0; j < TN; ++j) fma2(acc[i][j], a.y, w[j].y);
      }
    }
    if (--left == 0 || g + 1 == steps) {                     // a stretch ends
      left = per_seg;
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          sum[i][j] = __fadd_rn(sum[i][j], join2(acc[i][j]));
          acc[i][j] = 0;
        }
    }
  }
  // only now: blocks of the next kernel that move in early take places that this one's remaining blocks should spread over
  gi::pdl_launch_dependents();
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty + 4 * i;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx + 32 * j;
      if (m < M && n < N) {
        float* o = out + (size_t)m * ldo + n;
        *o = ACCUM ? *o + sum[i][j] : sum[i][j];
      }
    }
  }
}

template <typename Kern>
int allow_smem(Kern kern, size_t bytes, bool (&seen)[gi::MAX_DEVICES_SEEN]) {
  int dev;
  if (!gi::unconfigured_here(seen, &dev)) return GI_OK;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess)
    return gi::check_launch("gemm_f32: shared memory");
  if (dev >= 0) seen[dev] = true;
  return GI_OK;
}

template <int MT, bool ACCUM>
int launch_few(float* out, const float* A, const float* W, int M, int N, int K, long lda, long ldw, long ldo, int seg, cudaStream_t s) {
  static bool seen[gi::MAX_DEVICES_SEEN];
  const int rc = allow_smem(few_rows_kernel<MT, ACCUM>, FEW_SMEM<MT>, seen);
  if (rc != GI_OK) return rc;
  const int tiles = (N + ROWS - 1) / ROWS, blocks = gi::sm_count();
  const dim3 grid(tiles < blocks ? tiles : blocks, (M + MT - 1) / MT);
  return gi::check(gi::launch(few_rows_kernel<MT, ACCUM>, grid, dim3(FEW_THREADS), FEW_SMEM<MT>, s, out, A, W, M, N, K, lda, ldw, ldo, seg), "gemm_f32");
}

// Which of the two, by a model of what they measure (us), fitted to 1,134 sizes of 1 to 600 rows, 64 to 32,000 columns and K of 32
// to 8,192; the faster of the two is missed by 0.1% on average, by 12% at most.  An SM of few_rows takes 4.8 / 7.9 / 9.4 a 16-row
// tile of W and pass of up to 4 / 8 / 16 tokens and 2,048 of K, and works through all 32 stretches however short they are;
// one of many_rows 63.5 for a round of 32-row tiles and 2,048 of K (its tiles share the FFMA pipe), 17.5 once.  2,048 columns:
// 48 rows 32 against 75, 100 rows 57 against 77; 16,384 columns: 48 rows 186 against 128; 128,256 columns: 16 rows 468 against
// about 400; K of 64, 4,096 columns: 64 rows 31 against 5.
// A tile has 32 rows, or 36, 40 or 48 where that spares the fullest SM a tile: 601 rows x 2,048 columns are 304 tiles of 32
// rows, three on some SMs (184 us), and 272 of 36, two at most (142 us).
// The wider tiles leave room for two blocks an SM instead of three and cost 5% more for their rows (16,384 columns: 985 us
// against 956).
double few_cost(int M, int N, int seg) {
  const int mt = M <= 4 ? M : M <= 8 ? 8 : 16, sms = gi::sm_count();
  const long tiles = (N + ROWS - 1) / ROWS, blocks = tiles < sms ? tiles : sms, passes = (M + mt - 1) / mt;
  return 4.1 + (M <= 4 ? 4.8 : M <= 8 ? 7.9 : 9.4) * (SUM_SEGMENTS * seg / 2048.0) * (double)((tiles + blocks - 1) / blocks) * (double)((blocks * passes + sms - 1) / sms);
}
double many_cost(int M, int N, int K, int tm) {
  const long tiles = (long)((M + 4 * tm - 1) / (4 * tm)) * ((N + BN - 1) / BN), sms = gi::sm_count();
  return 5.0 + (17.5 + (tm == 8 ? 63.5 : 8.3 * tm) * (double)((tiles + sms - 1) / sms)) * (K / 2048.0);
}

template <int TM, bool ACCUM>
int launch_many(float* out, const float* A, const float* W, int M, int N, int K, long lda, long ldw, long ldo, int seg, cudaStream_t s) {
  static bool seen[gi::MAX_DEVICES_SEEN];
  const int rc = allow_smem(many_rows_kernel<TM, ACCUM>, MANY_SMEM<TM>, seen);
  if (rc != GI_OK) return rc;
  // row tiles fastest: blocks that run together share a tile of W, the larger operand
  const dim3 grid((M + 4 * TM - 1) / (4 * TM), (N + BN - 1) / BN);
  return gi::check(gi::launch(many_rows_kernel<TM, ACCUM>, grid, dim3(MANY_THREADS), MANY_SMEM<TM>, s, out, A, W, M, N, K, lda, ldw, ldo, seg), "gemm_f32");
}

template <bool ACCUM>
int launch_product(float* out, const float* A, const float* W, int M, int N, int K, long lda, long ldw, long ldo, cudaStream_t s) {
  const int seg = gi::sum_segment(K);
  int tm = 8;
  for (int t : {9, 10, 12})
    if (many_cost(M, N, K, t) < many_cost(M, N, K, tm)) tm = t;
  // (few_rows has 16 tokens to a block of the grid's y, which takes 65,535)
  if (few_cost(M, N, seg) > many_cost(M, N, K, tm) || M > 16 * 65535) {
    if (tm == 8) return launch_many<8, ACCUM>(out, A, W, M, N, K, lda, ldw, ldo, seg, s);
    if (tm == 9) return launch_many<9, ACCUM>(out, A, W, M, N, K, lda, ldw, ldo, seg, s);
    if (tm == 10) return launch_many<10, ACCUM>(out, A, W, M, N, K, lda, ldw, ldo, seg, s);
    return launch_many<12, ACCUM>(out, A, W, M, N, K, lda, ldw, ldo, seg, s);
  }
  if (M == 1) return launch_few<1, ACCUM>(out, A, W, M, N, K, lda, ldw, ldo, seg, s);
  if (M == 2) return launch_few<2, ACCUM>(out, A, W, M, N, K, lda, ldw, ldo, seg, s);
  if (M <= 4) return launch_few<4, ACCUM>(out, A, W, M, N, K, lda, ldw, ldo, seg, s);
  if (M <= 8) return launch_few<8, ACCUM>(out, A, W, M, N, K, lda, ldw, ldo, seg, s);
  return launch_few<16, ACCUM>(out, A, W, M, N, K, lda, ldw, ldo, seg, s);
}

}  // namespace

namespace gi {
// 16-byte reads need rows that start on 16-byte boundaries and hold a multiple of four numbers; the grid's y takes 65,535
// column tiles.
bool gemm_f32_takes(const void* A, const void* W, int N, int K, long lda, long ldw) {
  return K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0 && (N + BN - 1) / BN <= 65535;
}
int gemm_f32(float* out, bool accum, const float* A, const float* W, int M, int N, int K, long lda, long ldw, long ldo, cudaStream_t s) {
  return accum ? launch_product<true>(out, A, W, M, N, K, lda, ldw, ldo, s) : launch_product<false>(out, A, W, M, N, K, lda, ldw, ldo, s);
}
}  // namespace gi
