// The true 32-bit path's larger products on tcgen05 tensor cores: out[M,N] (op)= A[M,K] * W[N,K]^T, all float, for the matrices
// that gi_gemm_f32_split_scratch takes (1,024 rows and columns or more: with fewer columns its distance from 64 bits is not below
// the multiply-adds').  The matrix alone decides (N and K), never the rows: one order of additions serves every number of rows,
// so a prompt token's bits do not depend on its step.
//
// A number becomes two 16-bit floats: 64 neighbours of a row (a chunk) share a power of two that brings their largest to
// [2^14, 2^15); hi is the scaled number rounded to 11 bits, lo what is left rounded to 11 bits: 23 bits of each number or
// 2^-39 of its chunk's largest, whichever is more.  A chunk's sum is lo hi' + hi lo' + hi hi', twelve instructions of 16 numbers
// into a fresh accumulator (products are exact, the tensor cores cut off what does not fit into a sum they add to
// themselves, hence no longer chains); it leaves tensor memory, gets both powers of two back and is added with one rounding
// to its stretch's sum, and the at most eight stretches (they follow from K alone) are added in their order.
// A result that is no finite number is worked out again in plain multiply-adds (a split infinity is none any more).
//
// A tile is 128 rows of W (the "M" side of the instruction, split by four warps on the way from shared into tensor memory)
// times up to 128 tokens (the "N" side, in shared memory).  One thread feeds both rings with TMA, one issues the
// products, four warps split W, eight drain accumulators; two chunks of W and two accumulators in tensor memory, so that all
// four overlap.  Up to 32 tokens (FEW, tiles of 16) two more warps split the tokens themselves, eight warps split W in turns, and
// where there are few tiles the blocks of a cluster share the stretches of a tile, which meet in distributed shared memory;
// more tokens are split once by a kernel of their own, into scratch.
//
// Steps of one token a sequence keep gemm_f32.cu's kernels (ops.one_token_step): they are bound by the bytes of W, and there the
// chain of a chunk (32 KB: split 0.4 us, twelve products 0.5 us at 16 tokens as at 128, since each reads 128 rows of W out of
// tensor memory) is longer than the chunk's share of the memory's time: a 1B model's step of four 1.98 ms against 1.72.
// B200, one launch beside one of gemm_f32.cu: 601 rows 16,384 x 2,048 223 us (181 TFLOP/s) against 960; 2,048 x 8,192 150 against
// 550; 64 rows 46 against 134 and 112 against 150; 16 rows 51 against 72 and 48 against 48.  What bounds it with many rows is
// the draining warps (64 columns a thread and chunk), with few the one thread's products.
// Distance from 64 bits (2-norms): 1.2e-7 against 1.5e-7 (K 2,048), 1.4e-7 against 2.3e-7 (K 8,192), 1.2e-7 against 1.3e-7 (K 1,024).
#include <cuda.h>
#include <cuda_fp16.h>
#include <float.h>

#include "api.h"
#include "common.cuh"
#include "tc_utils.cuh"

namespace {

using namespace gi::tc;

constexpr int ROWS = 128;              // rows of W a tile = lanes of tensor memory
constexpr int CK = 64;                 // numbers of K a chunk
constexpr int STRETCHES = 8;
constexpr int FEW_TILE = 16, FEW_MAX = 32;   // tokens a tile of the FEW form, and tokens up to which it is taken
constexpr int SLAB = 8192;             // tokens split into scratch at a time
constexpr uint32_t W_STAGE = ROWS * CK * 4;

__device__ int g_split_status = 0;

// A wait of this kernel is over in microseconds (its inputs are complete when it starts); it gives up after a second or so.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int who) {
  for (uint32_t i = 0; i < (1u << 20); ++i)
    if (mbar_try_wait(bar, parity)) return true;
  atomicCAS(&g_split_status, 0, who);
  return false;
}

struct Args {
  float* out;
  const float *A, *W, *fx;             // fx: [chunk][ldf] what brings a token's chunk back to size (not FEW)
  long lda, ldw, ldo;
  int M, N, K, ldf, nt, tiles_m, tiles, chunks, per_stretch, seg, cluster, a_vec, accumulate;
};

template <bool FEW, bool CLUSTER>
struct Shape {
  static constexpr int NT = FEW ? FEW_TILE : 128;             // tokens a tile at most
  static constexpr int W_STAGES = CLUSTER ? 4 : FEW ? 6 : 3, X_STAGES = FEW ? 4 : 3, A_STAGES = FEW ? 4 : 2;
  // Slots of a chunk's powers of two and of its two barriers, from splitting to draining.  W is split at most A_STAGES chunks
  // ahead of the products, tokens X_STAGES, and the products are at most two ahead of the drained ones: six would do.
  static constexpr int SLOTS = 8;
  static constexpr uint32_t X_HALF = NT * 128, X_STAGE = 2 * X_HALF;     // hi rows, then lo rows, 128 bytes each, swizzled
  static constexpr uint32_t X_AT = W_STAGES * W_STAGE, FW_AT = X_AT + X_STAGES * X_STAGE, FX_AT = FW_AT + SLOTS * ROWS * 4,
                            RED_AT = FX_AT + SLOTS * NT * 4, BAR_AT = RED_AT + (CLUSTER ? STRETCHES / 2 * NT * ROWS * 4 : 0);
  static constexpr int N_BARS = 2 * W_STAGES + 2 * SLOTS;
  static constexpr size_t SMEM = BAR_AT + N_BARS * 8 + 16 + 1024;
  // warp 0 loads, 1 issues products, FEW: 2-3 split tokens, in turns; then the warps that split W, in SETS of four that take
  // turns, and those that drain, in PARTS of four that share a tile's columns, 16 at a time
  static constexpr int SETS = FEW ? 2 : 1, PARTS = FEW ? 1 : 2;
  static constexpr int SPLIT_WARP = FEW ? 4 : 2, DRAIN_WARP = SPLIT_WARP + 4 * SETS, THREADS = 32 * (DRAIN_WARP + 4 * PARTS);
  static constexpr int COLS = NT / PARTS;                    // columns a draining thread holds
  // columns of tensor memory: two accumulators, the chunks of W (hi 32, lo 32), and the stretches' sum where registers have no room
  static constexpr int A_AT = 2 * NT, SUM_AT = A_AT + 64 * A_STAGES, TMEM = 512;
  // A wait names a phase by its parity: whoever takes turns must see every phase of the stages that it waits for.  (With five
  // stages of W a set met a stage every second time round, and its wait was over while the phase before was still open.)
  static_assert(W_STAGES % SETS == 0, "a stage of W belongs to one set");
  static_assert(SUM_AT + (FEW ? 0 : NT) <= TMEM && SMEM <= 227 * 1024 && SPLIT_WARP % 2 == 0, "what a block has");
};

__device__ __forceinline__ uint64_t pack2(float a, float b) { return (uint64_t)__float_as_uint(a) | (uint64_t)__float_as_uint(b) << 32; }
__device__ __forceinline__ float lo_of(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi_of(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t a, uint64_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// The tensor cores cut off: a chunk's sum comes out small by 8.8e-8 of itself on average (measured, random numbers; 7e-8 with
// numbers of one sign), so the whole does, and gets that back here.
__device__ __forceinline__ float whole(float v) { return fmaf(v, 8.5e-8f, v); }

// the power of two that brings `top` to [2^14, 2^15) (a chunk of zeros or of the smallest numbers: 2^126), and its inverse
__device__ __forceinline__ float scale_of(float top, float* back) {
  const int s = min(141 - (int)(__float_as_uint(top) >> 23), 126);
  *back = __uint_as_float((uint32_t)(127 - s) << 23);
  return __uint_as_float((uint32_t)(127 + s) << 23);
}
// two neighbours as 16-bit pairs
__device__ __forceinline__ void split2(float a, float b, float scale, uint32_t* hi, uint32_t* lo) {
  const uint64_t y = mul2(pack2(a, b), pack2(scale, scale));
  const __half2 h = __floats2half2_rn(lo_of(y), hi_of(y));
  const float2 f = __half22float2(h);
  const __half2 l = __floats2half2_rn(lo_of(y) - f.x, hi_of(y) - f.y);
  *hi = *reinterpret_cast<const uint32_t*>(&h);
  *lo = *reinterpret_cast<const uint32_t*>(&l);
}

__device__ __forceinline__ void mma_a_tmem(uint32_t d, uint32_t a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d), "r"(a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}
// (the registers are named, so that nothing that reads them moves above the wait)
__device__ __forceinline__ void wait_ld16(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                 "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]) :: "memory");
}
__device__ __forceinline__ void wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float ld_remote(uint32_t addr, int rank) {
  uint32_t at;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// one result by plain multiply-adds, in the order of gemm_f32.cu
__device__ __noinline__ void plain_result(const Args& args, int m, int n) {
  const float *a = args.A + (size_t)m * args.lda, *w = args.W + (size_t)n * args.ldw;
  float sum = 0.f;
  for (int s = 0; s < args.K; s += args.seg) {
    float even = 0.f, odd = 0.f;
    const int end = min(args.K, s + args.seg);
    for (int k = s; k < end; k += 2) {
      even = fmaf(a[k], w[k], even);
      if (k + 1 < end) odd = fmaf(a[k + 1], w[k + 1], odd);
    }
    sum += even + odd;
  }
  float* o = args.out + (size_t)m * args.ldo + n;
  *o = args.accumulate ? *o + sum : sum;
}

// Splits `rows` rows of A into two 16-bit planes [rows][chunks * 64] (zeros past K) and fx.  Sixteen lanes take a chunk.
__global__ void __launch_bounds__(256)
split_rows_kernel(uint2* __restrict__ hi, uint2* __restrict__ lo, float* __restrict__ fx, const float* A, long lda, int rows, int K, int chunks,
                  int ldf, int a_vec) {
  gi::pdl_prologue();
  const long i = (long)blockIdx.x * 16 + (threadIdx.x >> 4);
  const int l = threadIdx.x & 15;
  const bool live = i < (long)rows * chunks;
  const int m = live ? (int)(i / chunks) : 0, c = live ? (int)(i % chunks) : 0, k = c * CK + l * 4;
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  if (live) {
    const float* src = A + (size_t)m * lda + k;
    if (a_vec && k + 4 <= K) {
      const float4 f = *reinterpret_cast<const float4*>(src);
      v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (k + e < K) v[e] = src[e];
    }
  }
  float top = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
  float back;
  const float scale = scale_of(top, &back);
  uint2 h, w;
  split2(v[0], v[1], scale, &h.x, &w.x);
  split2(v[2], v[3], scale, &h.y, &w.y);
  if (live) {
    hi[i * 16 + l] = h;
    lo[i * 16 + l] = w;
    if (l == 0) fx[(size_t)c * ldf + m] = back;
  }
}

// CLUSTER: `a.cluster` blocks share a tile's stretches (FEW only).  W_TMA: rows of W start on 16-byte boundaries; else its
// warps load their rows themselves.
template <bool FEW, bool CLUSTER, bool W_TMA>
__global__ void __launch_bounds__(Shape<FEW, CLUSTER>::THREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_lo,
                  const __grid_constant__ Args a) {
  using S = Shape<FEW, CLUSTER>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  float* fw = reinterpret_cast<float*>(smem + S::FW_AT);     // [SLOTS][ROWS]
  float* fx = reinterpret_cast<float*>(smem + S::FX_AT);     // [SLOTS][NT]
  const uint32_t bars = smem_u32(smem + S::BAR_AT);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + S::BAR_AT + S::N_BARS * 8);
  // Two barriers a chunk, so that the one thread that issues products waits once and signals once: `full` - its rows of W are
  // split (4 warps), its tokens are there (1) and its accumulator is drained (the chunk before the last one's; 4 warps a part);
  // `done` - its products are: its operands' places are free and its accumulator is ready.
  const uint32_t w_full = bars, w_empty = w_full + 8 * S::W_STAGES, full = w_empty + 8 * S::W_STAGES, done = full + 8 * S::SLOTS;
  auto wait_full = [&](int it, int who) { return mbar_wait(full + 8 * (it % S::SLOTS), (uint32_t)((it / S::SLOTS) & 1), who); };
  auto wait_done = [&](int it, int who) { return it < 0 || mbar_wait(done + 8 * (it % S::SLOTS), (uint32_t)((it / S::SLOTS) & 1), who); };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < S::W_STAGES; ++i) {
      mbar_init(w_full + 8 * i, 1);
      mbar_init(w_empty + 8 * i, 4);
    }
    for (int i = 0; i < S::SLOTS; ++i) {
      mbar_init(full + 8 * i, 5 + 4 * S::PARTS);
      mbar_init(done + 8 * i, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)S::TMEM) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  const int rank = CLUSTER ? (int)blockIdx.x % a.cluster : 0, mine = CLUSTER ? STRETCHES / a.cluster : STRETCHES;   // stretches of this block
  const int tile0 = CLUSTER ? (int)blockIdx.x / a.cluster : (int)blockIdx.x, tile_step = CLUSTER ? a.tiles : (int)gridDim.x;
  const int c_first = CLUSTER ? min(a.chunks, rank * mine * a.per_stretch) : 0, c_last = CLUSTER ? min(a.chunks, c_first + mine * a.per_stretch) : a.chunks;
  if (W_TMA && threadIdx.x == 0) {     // a prefetch reads no values: right whoever wrote W
    const int n0 = tile0 / a.tiles_m * ROWS;
    for (int c = c_first; c < min(c_last, c_first + S::W_STAGES); ++c) {
      tma_prefetch_l2_2d(&map_w, c * CK, n0);
      tma_prefetch_l2_2d(&map_w, c * CK + 32, n0);
    }
  }
  if constexpr (FEW) {                 // rows of tokens that do not exist stay zero
    for (int i = threadIdx.x; i < S::X_STAGES * (int)S::X_STAGE / 16; i += S::THREADS) reinterpret_cast<uint4*>(smem + S::X_AT)[i] = make_uint4(0, 0, 0, 0);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  gi::pdl_launch_dependents();
  gi::pdl_wait();

  if (warp == 0) {
    if (lane == 0 && (W_TMA || !FEW)) {
      bool ok = true;
      int it = 0, loaded = 0;
      for (int tile = tile0; tile < a.tiles && ok; tile += tile_step) {
        const int m0 = tile % a.tiles_m * a.nt, n0 = tile / a.tiles_m * ROWS;
        for (int c = c_first; c < c_last && ok; ++c, ++it) {
          if (W_TMA) {
            const int st = it % S::W_STAGES;
            ok = mbar_wait(w_empty + 8 * st, (uint32_t)((it / S::W_STAGES) & 1) ^ 1, 1);
            if (!ok) break;
            mbar_expect_tx(w_full + 8 * st, W_STAGE);
            const uint32_t dst = smem_u32(smem + st * W_STAGE);
            tma_load_2d(dst, &map_w, c * CK, n0, w_full + 8 * st);
            tma_load_2d(dst + W_STAGE / 2, &map_w, c * CK + 32, n0, w_full + 8 * st);
          }
          if (!FEW) {
            const int st = it % S::X_STAGES, slot = it % S::SLOTS;
            ok = wait_done(it - S::X_STAGES, 1);
            if (!ok) break;
            const uint32_t dst = smem_u32(smem + S::X_AT + st * S::X_STAGE), bar = full + 8 * slot;
            mbar_expect_tx(bar, (uint32_t)a.nt * 260u);
            tma_load_2d(dst, &map_hi, c * CK, m0, bar);
            tma_load_2d(dst + S::X_HALF, &map_lo, c * CK, m0, bar);
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         ::"r"(smem_u32(fx + slot * S::NT)), "l"(a.fx + (size_t)c * a.ldf + m0), "r"((uint32_t)a.nt * 4u), "r"(bar) : "memory");
          }
          ++loaded;
        }
      }
      // the block does not leave before its copies have landed, also where somebody gave up
      for (int i = max(0, loaded - S::W_STAGES); W_TMA && i < loaded; ++i) mbar_wait(w_full + 8 * (i % S::W_STAGES), (uint32_t)((i / S::W_STAGES) & 1), 1);
      for (int i = max(0, loaded - S::X_STAGES); !FEW && i < loaded; ++i) wait_full(i, 1);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = (1u << 4) | ((uint32_t)(a.nt >> 3) << 17) | ((uint32_t)(ROWS >> 4) << 24);   // float sums of 16-bit floats
      bool ok = true;
      int it = 0;
      for (int tile = tile0; tile < a.tiles && ok; tile += tile_step)
        for (int c = c_first; c < c_last && ok; ++c, ++it) {
          const int st = it & 1, as = it % S::A_STAGES, xs = it % S::X_STAGES;
          ok = wait_full(it, 2);
          if (!ok) break;
          tc_fence_after();
          const uint32_t d = tmem + st * S::NT, hi = tmem + S::A_AT + as * 64, lo = hi + 32;
          const uint64_t x_hi = smem_desc(smem_u32(smem + S::X_AT + xs * S::X_STAGE)), x_lo = x_hi + (S::X_HALF >> 4);
#pragma unroll
          for (int k = 0; k < CK / 16; ++k) mma_a_tmem(d, lo + 8 * k, x_hi + 2 * k, idesc, k > 0);
#pragma unroll
          for (int k = 0; k < CK / 16; ++k) mma_a_tmem(d, hi + 8 * k, x_lo + 2 * k, idesc, 1);
#pragma unroll
          for (int k = 0; k < CK / 16; ++k) mma_a_tmem(d, hi + 8 * k, x_hi + 2 * k, idesc, 1);
          tc_commit(done + 8 * (it % S::SLOTS));
        }
      wait_done(it - 1, 2);                                  // its products, as the loads above
    }
  } else if (warp >= S::SPLIT_WARP && warp < S::DRAIN_WARP) {
    // a row of W a thread
    const int set = (warp - S::SPLIT_WARP) / 4;
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    bool ok = true;
    int it = 0;
    for (int tile = tile0; tile < a.tiles && ok; tile += tile_step) {
      const int n = tile / a.tiles_m * ROWS + row;
      for (int c = c_first; c < c_last && ok; ++c, ++it) {
        if (it % S::SETS != set) continue;
        const int ws = it % S::W_STAGES, as = it % S::A_STAGES;
        const unsigned char* staged = smem + ws * W_STAGE + row * 128;
        auto piece = [&](int p) {                            // numbers 4 p .. + 3 of this row's chunk
          if constexpr (W_TMA) return *reinterpret_cast<const float4*>(staged + (p >> 3) * (W_STAGE / 2) + ((p & 7) ^ (row & 7)) * 16);
          const float* src = a.W + (size_t)n * a.ldw + c * CK + 4 * p;
          const int live = n < a.N ? a.K - c * CK - 4 * p : 0;
          return make_float4(live > 0 ? src[0] : 0.f, live > 1 ? src[1] : 0.f, live > 2 ? src[2] : 0.f, live > 3 ? src[3] : 0.f);
        };
        if (W_TMA) ok = mbar_wait(w_full + 8 * ws, (uint32_t)((it / S::W_STAGES) & 1), 3);
        if (!ok) break;
        float4 v[CK / 4];
        float top = 0.f, top1 = 0.f;
#pragma unroll
        for (int p = 0; p < CK / 4; ++p) v[p] = piece(p);
        if (W_TMA) {
          __syncwarp();
          if (lane == 0) mbar_arrive(w_empty + 8 * ws);
        }
#pragma unroll
        for (int p = 0; p < CK / 4; ++p) {
          top = fmaxf(top, fmaxf(fabsf(v[p].x), fabsf(v[p].y)));
          top1 = fmaxf(top1, fmaxf(fabsf(v[p].z), fabsf(v[p].w)));
        }
        float back;
        const float scale = scale_of(fmaxf(top, top1), &back);
        ok = wait_done(it - S::A_STAGES, 3);
        if (!ok) break;
        tc_fence_after();
        const uint32_t dst = tmem + lane_base + S::A_AT + as * 64;
#pragma unroll
        for (int q = 0; q < CK / 16; ++q) {
          uint32_t hi[8], lo[8];
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            const float4 f = v[4 * q + p];
            split2(f.x, f.y, scale, &hi[2 * p], &lo[2 * p]);
            split2(f.z, f.w, scale, &hi[2 * p + 1], &lo[2 * p + 1]);
          }
          tc_st8(dst + 8 * q, hi);
          tc_st8(dst + 32 + 8 * q, lo);
        }
        fw[it % S::SLOTS * ROWS + row] = back;
        wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(full + 8 * (it % S::SLOTS));
      }
    }
  } else if (warp >= S::DRAIN_WARP) {
    const int row = (warp & 3) * 32 + lane, part = (warp - S::DRAIN_WARP) / 4;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    constexpr int GROUP = 16, GROUPS = S::COLS / GROUP;      // columns leave tensor memory 16 at a time
    auto col_of = [&](int g) { return (g * S::PARTS + part) * GROUP; };
    bool ok = true;
    int it = 0;
    if (lane == 0) {                                         // nothing to drain before the first two chunks
      mbar_arrive(full);
      mbar_arrive(full + 8);
    }
    for (int tile = tile0; tile < a.tiles && ok; tile += tile_step) {
      const int m0 = tile % a.tiles_m * a.nt, n = tile / a.tiles_m * ROWS + row, nt = a.nt;
      uint64_t acc[S::COLS / 2], sum[FEW ? S::COLS / 2 : 1];
#pragma unroll
      for (int j = 0; j < S::COLS / 2; ++j) acc[j] = 0;
      int left = a.per_stretch, stretch = 0;
      for (int c = c_first; c < c_last && ok; ++c, ++it) {
        const int st = it & 1, slot = it % S::SLOTS;
        ok = wait_full(it, 4) && wait_done(it, 4);
        if (!ok) break;
        tc_fence_after();
        const float f = fw[slot * ROWS + row];
        const uint64_t f2 = pack2(f, f);
        const uint32_t d = tmem + lane_base + st * S::NT;
        auto take = [&](int g, const uint32_t (&r)[GROUP]) {
#pragma unroll
          for (int j = 0; j < GROUP; j += 4) {
            const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(fx + slot * S::NT + col_of(g) + j);
            fma2(acc[(g * GROUP + j) / 2], (uint64_t)r[j] | (uint64_t)r[j + 1] << 32, mul2(x.x, f2));
            fma2(acc[(g * GROUP + j) / 2 + 1], (uint64_t)r[j + 2] | (uint64_t)r[j + 3] << 32, mul2(x.y, f2));
          }
        };
        // (a third of a chunk's time; one group asked for while the one before is added was slower: 253 against 223 us at 601 x 16,384 x 2,048)
#pragma unroll
        for (int g = 0; g < GROUPS; g += 2) {                // (columns past the tile's tokens hold what nobody reads)
          if (col_of(g) < nt) {
            uint32_t r[GROUP], r1[GROUP];
            tc_ld16(d + col_of(g), r);
            if (g + 1 < GROUPS) {
              tc_ld16(d + col_of(g + 1), r1);
              wait_ld16(r1);
            }
            wait_ld16(r);
            take(g, r);
            if (g + 1 < GROUPS) take(g + 1, r1);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(full + 8 * ((it + 2) % S::SLOTS));
        if (--left > 0 && c + 1 < c_last) continue;
        left = a.per_stretch;                                // a stretch ends
        if constexpr (CLUSTER) {
          // where the cluster reads it
          float* red = reinterpret_cast<float*>(smem + S::RED_AT) + stretch * FEW_TILE * ROWS;
#pragma unroll
          for (int j = 0; j < S::COLS / 2; ++j) {
            red[(2 * j) * ROWS + row] = lo_of(acc[j]);
            red[(2 * j + 1) * ROWS + row] = hi_of(acc[j]);
            acc[j] = 0;
          }
        } else if constexpr (FEW) {
#pragma unroll
          for (int j = 0; j < S::COLS / 2; ++j) {
            sum[j] = stretch == 0 ? acc[j] : add2(sum[j], acc[j]);
            acc[j] = 0;
          }
        } else {
          const uint32_t t = tmem + lane_base + S::SUM_AT;
          const bool last = c + 1 == c_last;
#pragma unroll
          for (int g = 0; g < GROUPS; ++g) {
            const int col = col_of(g);
            if (col < nt) {
              uint32_t s[GROUP];
              if (stretch > 0) {
                tc_ld16(t + col, s);
                wait_ld16(s);
#pragma unroll
                for (int j = 0; j < GROUP; j += 2) {
                  uint64_t& v = acc[(g * GROUP + j) / 2];
                  v = add2((uint64_t)s[j] | (uint64_t)s[j + 1] << 32, v);
                }
              }
              if (!last) {
#pragma unroll
                for (int j = 0; j < GROUP; j += 2) {
                  uint64_t& v = acc[(g * GROUP + j) / 2];
                  s[j] = (uint32_t)v;
                  s[j + 1] = (uint32_t)(v >> 32);
                  v = 0;
                }
                tc_st16(t + col, s);
              }
            }
          }
          if (!last) wait_st();
        }
        ++stretch;
      }
      if (!ok) break;
      if (!CLUSTER && n < a.N) {
        const int live = min(nt, a.M - m0);
        const long ldo = a.ldo;
        const bool add = a.accumulate != 0;
        float* o = a.out + (size_t)m0 * ldo + n;
        uint32_t odd[(S::NT + 31) / 32] = {};                // results that are no finite numbers: after the others
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
          const int col = col_of(g);
#pragma unroll
          for (int j = 0; j < GROUP; ++j) {
            const uint64_t both = FEW ? sum[FEW ? (g * GROUP + j) / 2 : 0] : acc[(g * GROUP + j) / 2];
            const float v = whole((j & 1) ? hi_of(both) : lo_of(both));
            const bool fine = fabsf(v) <= FLT_MAX;
            float* at = o + (size_t)(col + j) * ldo;
            if (col + j < live) {
              if (fine) *at = add ? *at + v : v;
              else odd[g * S::PARTS * GROUP / 32] |= 1u << (g * S::PARTS * GROUP % 32 + j);
            }
          }
        }
#pragma unroll
        for (int i = 0; i < (S::NT + 31) / 32; ++i)
          for (uint32_t rest = odd[i]; rest; rest &= rest - 1) plain_result(a, m0 + 32 * i + part * GROUP + __ffs((int)rest) - 1, n);
      }
    }
  } else if constexpr (FEW) {
    // tokens: sixteen lanes a chunk of a token; the two warps take turns, and a chunk's numbers are asked for a turn early
    const int l = lane & 15, sub = lane >> 4, n_chunks = c_last - c_first;
    const int total = tile0 < a.tiles ? ((a.tiles - tile0 + tile_step - 1) / tile_step) * n_chunks : 0;
    float4 next[FEW_TILE / 2];
    auto ask = [&](int it) {
      const int k = (c_first + it % n_chunks) * CK + l * 4, m0 = (tile0 + it / n_chunks * tile_step) % a.tiles_m * FEW_TILE;
#pragma unroll
      for (int i = 0; i < FEW_TILE / 2; ++i) {
        const int m = m0 + 2 * i + sub;
        const float* src = a.A + (size_t)m * a.lda + k;
        next[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (m < a.M) {
          if (a.a_vec && k + 4 <= a.K) {
            next[i] = *reinterpret_cast<const float4*>(src);
          } else {
            if (k < a.K) next[i].x = src[0];
            if (k + 1 < a.K) next[i].y = src[1];
            if (k + 2 < a.K) next[i].z = src[2];
            if (k + 3 < a.K) next[i].w = src[3];
          }
        }
      }
    };
    bool ok = true;
    if (warp - 2 < total) ask(warp - 2);
    for (int it = warp - 2; it < total && ok; it += 2) {
      const int xs = it % S::X_STAGES, slot = it % S::SLOTS;
      float4 v[FEW_TILE / 2];
#pragma unroll
      for (int i = 0; i < FEW_TILE / 2; ++i) v[i] = next[i];
      if (it + 2 < total) ask(it + 2);
      ok = wait_done(it - S::X_STAGES, 5);
      if (!ok) break;
#pragma unroll
      for (int i = 0; i < FEW_TILE / 2; ++i) {
        if (2 * i >= a.M) break;                             // (a later tile's missing tokens: zeros)
        const int m = 2 * i + sub;
        float top = fmaxf(fmaxf(fabsf(v[i].x), fabsf(v[i].y)), fmaxf(fabsf(v[i].z), fabsf(v[i].w)));
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
        float back;
        const float scale = scale_of(top, &back);
        uint2 h, w;
        split2(v[i].x, v[i].y, scale, &h.x, &w.x);
        split2(v[i].z, v[i].w, scale, &h.y, &w.y);
        unsigned char* dst = smem + S::X_AT + xs * S::X_STAGE + m * 128 + ((l >> 1) ^ (m & 7)) * 16 + (l & 1) * 8;
        *reinterpret_cast<uint2*>(dst) = h;
        *reinterpret_cast<uint2*>(dst + S::X_HALF) = w;
        if (l == 0) fx[slot * S::NT + m] = back;
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(full + 8 * slot);
    }
  }
  if constexpr (CLUSTER) {
    __syncwarp();
    cluster_sync();
    const int used = (a.chunks + a.per_stretch - 1) / a.per_stretch;
    const uint32_t red = smem_u32(smem + S::RED_AT);
    const int m0 = tile0 % a.tiles_m * FEW_TILE, n0 = tile0 / a.tiles_m * ROWS;
    for (int i = rank * S::THREADS + (int)threadIdx.x; i < min(FEW_TILE, a.M - m0) * ROWS; i += a.cluster * S::THREADS) {
      const int m = m0 + i / ROWS, n = n0 + i % ROWS;
      float parts[STRETCHES];
#pragma unroll
      for (int r = 0; r < STRETCHES; ++r) parts[r] = r < used ? ld_remote(red + 4u * (uint32_t)(r % mine * FEW_TILE * ROWS + i), r / mine) : 0.f;
      float v = parts[0];
#pragma unroll
      for (int r = 1; r < STRETCHES; ++r)
        if (r < used) v += parts[r];
      v = whole(v);
      if (n < a.N) {
        float* o = a.out + (size_t)m * a.ldo + n;
        if (fabsf(v) <= FLT_MAX) *o = a.accumulate ? *o + v : v;
        else plain_result(a, m, n);
      }
    }
    cluster_sync();                                          // nobody leaves while its sums are read
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)S::TMEM) : "memory");
}

template <bool FEW, bool CLUSTER, bool W_TMA>
int allow_smem() {
  static bool seen[gi::MAX_DEVICES_SEEN];
  int dev;
  if (!gi::unconfigured_here(seen, &dev)) return GI_OK;
  if (cudaFuncSetAttribute(gemm_split_kernel<FEW, CLUSTER, W_TMA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Shape<FEW, CLUSTER>::SMEM) != cudaSuccess)
    return gi::check_launch("gemm_f32_split: shared memory");
  if (dev >= 0) seen[dev] = true;
  return GI_OK;
}

// Blocks that share a tile's stretches: as many as let every cluster of the launch run at once.
template <bool W_TMA>
int cluster_of(int tiles) {
  static int room[gi::MAX_DEVICES_SEEN][4] = {};             // clusters of 2, 4 and 8 blocks that a device holds, plus one
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= gi::MAX_DEVICES_SEEN || allow_smem<true, true, W_TMA>() != GI_OK) return 1;
  for (int k = 3; k > 0; --k) {
    if (room[dev][k] == 0) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(1 << k);
      cfg.blockDim = dim3(Shape<true, true>::THREADS);
      cfg.dynamicSmemBytes = Shape<true, true>::SMEM;
      cudaLaunchAttribute attr;
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim.x = 1 << k;
      attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
      cfg.attrs = &attr;
      cfg.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, gemm_split_kernel<true, true, W_TMA>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        n = 0;
      }
      room[dev][k] = n + 1;
    }
    if (tiles <= room[dev][k] - 1) return 1 << k;
  }
  return 1;
}

template <bool FEW, bool CLUSTER, bool W_TMA>
int launch_split(const CUtensorMap& mw, const CUtensorMap& mh, const CUtensorMap& ml, const Args& a, int blocks, cudaStream_t s) {
  const int rc = allow_smem<FEW, CLUSTER, W_TMA>();
  if (rc != GI_OK) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(Shape<FEW, CLUSTER>::THREADS);
  cfg.dynamicSmemBytes = Shape<FEW, CLUSTER>::SMEM;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (CLUSTER) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = a.cluster;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (gi::pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return gi::check(cudaLaunchKernelEx(&cfg, gemm_split_kernel<FEW, CLUSTER, W_TMA>, mw, mh, ml, a), "gemm_f32_split");
}

int pad16(int m) { return (m + 15) / 16 * 16; }
long plane_bytes(long rows, int chunks) { return rows * chunks * CK * 2; }

}  // namespace

// Bytes of scratch that a product of these sizes needs, -1 where the plain kernels take it.
extern "C" long gi_gemm_f32_split_scratch(int M, int N, int K) {
  if (M <= 0 || N < 1024 || K < 1024) return -1;
  if (M <= FEW_MAX) return 0;
  const int rows = M < SLAB ? M : SLAB, chunks = (K + CK - 1) / CK;
  return 2 * plane_bytes(rows, chunks) + (long)chunks * (pad16(rows) + 128) * 4;
}

extern "C" int gi_gemm_f32_split(float* out, int mode, const float* A, const float* W, int M, int N, int K, long lda, long ldw, long ldo,
                                 void* scratch, long scratch_bytes, void* stream) {
  if (M <= 0 || N <= 0) return GI_OK;
  if (mode != GI_GEMM_STORE && mode != GI_GEMM_ACCUM_F32) return gi::fail(GI_ERR_ARG, "gemm_f32_split: unknown mode %d", mode);
  const long want = gi_gemm_f32_split_scratch(M, N, K);
  if (want < 0) return gi::fail(GI_ERR_UNSUPPORTED, "gemm_f32_split: a matrix of %d x %d is for the plain kernels", N, K);
  if (scratch_bytes < want || (want > 0 && (scratch == nullptr || ((uintptr_t)scratch & 15))))
    return gi::fail(GI_ERR_ARG, "gemm_f32_split: %ld bytes of scratch, wanted %ld on a 16-byte boundary", scratch_bytes, want);
  cudaStream_t s = (cudaStream_t)stream;
  const int sms = gi::sm_count(), tiles_n = (N + ROWS - 1) / ROWS;
  Args a = {};
  a.W = W;
  a.lda = lda; a.ldw = ldw; a.ldo = ldo;
  a.N = N; a.K = K;
  a.chunks = (K + CK - 1) / CK;
  a.per_stretch = (a.chunks + STRETCHES - 1) / STRETCHES;
  a.seg = gi::sum_segment(K);
  a.a_vec = (lda % 4 == 0 && ((uintptr_t)A & 15) == 0) ? 1 : 0;
  a.accumulate = mode == GI_GEMM_ACCUM_F32 ? 1 : 0;
  const bool w_tma = ldw % 4 == 0 && ((uintptr_t)W & 15) == 0 && K % 4 == 0;
  CUtensorMap mw = {}, mh = {}, ml = {};
  if (w_tma) {
    const int rc = gi::tensor_map_2d_ex(&mw, W, N, K, ldw, GI_F32, 32, ROWS);
    if (rc != GI_OK) return rc;
  }
  if (M <= FEW_MAX) {
    a.out = out; a.A = A;
    a.M = M; a.nt = FEW_TILE; a.tiles_m = (M + FEW_TILE - 1) / FEW_TILE; a.tiles = a.tiles_m * tiles_n;
    a.cluster = w_tma ? cluster_of<true>(a.tiles) : cluster_of<false>(a.tiles);
    if (a.cluster > 1)
      return w_tma ? launch_split<true, true, true>(mw, mh, ml, a, a.tiles * a.cluster, s) : launch_split<true, true, false>(mw, mh, ml, a, a.tiles * a.cluster, s);
    const int blocks = a.tiles < sms ? a.tiles : sms;
    return w_tma ? launch_split<true, false, true>(mw, mh, ml, a, blocks, s) : launch_split<true, false, false>(mw, mh, ml, a, blocks, s);
  }
  for (int m0 = 0; m0 < M; m0 += SLAB) {
    const int rows = M - m0 < SLAB ? M - m0 : SLAB;
    unsigned char* hi = (unsigned char*)scratch;
    unsigned char* lo = hi + plane_bytes(rows, a.chunks);
    float* fx = reinterpret_cast<float*>(lo + plane_bytes(rows, a.chunks));
    a.out = out + (size_t)m0 * ldo;
    a.A = A + (size_t)m0 * lda;
    a.M = rows;
    a.ldf = pad16(rows) + 128;
    a.fx = fx;
    int rc = gi::check(gi::launch(split_rows_kernel, dim3((unsigned)(((long)rows * a.chunks + 15) / 16)), dim3(256), 0, s, (uint2*)hi, (uint2*)lo, fx, a.A, lda,
                                  rows, K, a.chunks, a.ldf, a.a_vec), "gemm_f32_split: tokens");
    if (rc != GI_OK) return rc;
    // tokens a tile: a chunk takes a block about 512 + 5 tokens clocks (shared memory's and tensor memory's reads), a launch as
    // many rounds of tiles as the fullest SM has
    long best = 0;
    for (int nt = 16; nt <= 128; nt += 16) {
      const long tiles = (long)((rows + nt - 1) / nt) * tiles_n, cost = (tiles + sms - 1) / sms * (512 + 5 * nt);
      if (best == 0 || cost <= best) best = cost, a.nt = nt, a.tiles_m = (rows + nt - 1) / nt;
    }
    a.tiles = a.tiles_m * tiles_n;
    rc = gi::tensor_map_2d_ex(&mh, hi, rows, (long)a.chunks * CK, (long)a.chunks * CK, GI_BF16, 64, a.nt);
    if (rc == GI_OK) rc = gi::tensor_map_2d_ex(&ml, lo, rows, (long)a.chunks * CK, (long)a.chunks * CK, GI_BF16, 64, a.nt);
    if (rc != GI_OK) return rc;
    const int blocks = a.tiles < sms ? a.tiles : sms;
    rc = w_tma ? launch_split<false, false, true>(mw, mh, ml, a, blocks, s) : launch_split<false, false, false>(mw, mh, ml, a, blocks, s);
    if (rc != GI_OK) return rc;
  }
  return GI_OK;
}

// 0, or the role whose wait ran out since the last call (1 loads, 2 products, 3 rows of W, 4 results, 5 tokens).
extern "C" int gi_gemm_f32_split_status(int* status) {
  int zero = 0;
  if (cudaMemcpyFromSymbol(status, g_split_status, sizeof(int)) != cudaSuccess || cudaMemcpyToSymbol(g_split_status, &zero, sizeof(int)) != cudaSuccess)
    return gi::check_launch("gemm_f32_split: status");
  return GI_OK;
}
