// The true 32-bit path's larger products on tcgen05 tensor cores: out[M,N] (op)= A[M,K] * W[N,K]^T, all float, for the matrices
// that gi_gemm_f32_split_scratch takes (1,024 rows and columns or more).  Between this kernel and the multiply-adds of gemm_f32.cu the
// matrix (N and K) and the kind of step decide, never the number of rows: a prompt token's bits do not depend on its step.
//
// A number becomes three bfloat16 (the splitting of Henry, Tang and Heinecke, "Leveraging the bfloat16 Artificial Intelligence
// Datatype For Higher-Precision Computations", 2019): hi is the number rounded to 8 bits, mid what is left rounded to 8 bits, lo what
// is left then, which has 8 bits at most.  They have a float's exponent, so the three sum up to the number itself whatever its
// neighbours are; it is multiplied by 2^24 first, so that this holds down to the smallest floats.  Numbers from 2^103 on and sums from
// 2^79 on become no finite numbers, and such results are worked out again in plain multiply-adds, as those that really are none.
// Of the nine products six are made; mid lo', lo mid' and lo lo' are 2^-24 of |a w| together at most, random in sign.
//
// The tensor cores cut off what does not fit into a sum that they add to themselves, so no long chain is left to them: hi hi'
// of 32 numbers of K (two instructions, products of 16 bits) goes into a fresh accumulator, which leaves tensor memory and is
// added with one rounding to its stretch's sum; a chunk of K is 64 numbers.  The five small products (2^-8 of the whole) have an
// accumulator of their own, which is read at the end of a stretch.  The at most eight stretches (they follow from K alone) are added in
// their order.  (With 64 numbers an accumulator, sums of one sign were further from 64 bits than the multiply-adds'.)
//
// A tile is 128 rows of W (the "M" side of the instruction, split by four warps on the way from shared into tensor memory)
// times up to 96 tokens (the "N" side, in shared memory; 96, since a chunk's two accumulators of hi hi', one of the small products and
// two chunks of W's parts are 480 of tensor memory's 512 columns).  A chunk's hi hi' is made first and drained while its small
// products are.  One thread feeds both rings with TMA, one issues the products, four warps
// split W, twelve drain accumulators.  Up to 32 tokens (FEW, tiles of 16) two more warps split the tokens themselves, eight warps
// split W in turns, and where there are few tiles the blocks of a cluster share the stretches of a tile, which meet in distributed
// shared memory; more tokens are split once by a kernel of their own, into scratch (6 bytes a number, 8,192 tokens at a time).
//
// An instruction takes 17 + 0.45 clocks a token when a warp issues it together and one lane is elected, and 96 or more when one thread
// does so in a branch of its own (its operands then have to be brought together first).
//
// Steps of one token a sequence keep gemm_f32.cu's kernels (ops.one_token_step): a layer of a 1B model takes 105 us here and 102
// there with one to four sequences, the common case (119 and 164 with 16; the number of sequences must not decide, or a
// token's bits would depend on it).  The smaller matrices do as well, since a launch here has 10 us of set-up and pipeline
// to fill, longer than what they take there (1,024 x 1,024: 12 us here for 16 rows, 12 there; 24 against 16 for 33).
// B200, cold L2, one launch beside one of gemm_f32.cu (us): 601 rows 16,384 x 2,048 234 (172 TFLOP/s) against 960; 2,048 x 8,192 136 against
// 548; 64 rows 46 against 133 and 115 against 151; 16 rows 43 against 72 and 38 against 47; 4 rows 39 against 45 and 32 against 27.
// What bounds it with many rows: tensor cores busy 57 % of the time, issue slots 55 % (splitting and draining warps), shared memory's
// 128 bytes a clock about 60 % (W, tokens and their parts: 170 KB a chunk), one waiting for another; eight splitting warps in the
// place of four were slower (601 rows 269 us), as was a first half split before its place is free (241).  With few rows: the bytes of W.
// Distance from 64 bits (2-norms, random numbers): 0.84e-7 against 1.32e-7 (K 1,024), 0.92e-7 against 1.51e-7 (K 2,048), 1.3e-7
// against 2.3e-7 (K 8,192); of one sign 0.64e-7 against 0.90e-7; rows of W with eight numbers 5.3e-8 against 5.9e-8, with one (where the
// multiply-adds round once) 2.6e-8 against 2.5e-8.
#include <cuda.h>
#include <cuda_bf16.h>
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

// No wait depends on what the numbers are but for the time that a tile full of results that are no finite numbers takes (a few
// milliseconds); all end after WAIT_LIMIT tries.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int who) { return gi::tc::mbar_wait(bar, parity, who, &g_split_status); }

struct Args {
  float* out;
  const float *A, *W;
  long lda, ldw, ldo;
  int M, N, K, nt, tiles_m, tiles, chunks, per_stretch, seg, cluster, a_vec, w_vec, accumulate;
};

template <bool FEW, bool CLUSTER>
struct Shape {
  static constexpr int NT = FEW ? FEW_TILE : 96;              // tokens a tile at most
  static constexpr int W_STAGES = CLUSTER ? 4 : FEW ? 6 : 3, X_STAGES = FEW ? 4 : 3, A_STAGES = FEW ? 4 : 2;
  // Slots of a chunk's barriers.  W is split at most A_STAGES chunks ahead of the products, tokens X_STAGES, and the products are
  // at most one ahead of the drained ones: six would do.
  static constexpr int SLOTS = 8;
  static constexpr uint32_t X_PART = NT * 128, X_STAGE = 3 * X_PART;     // hi rows, mid rows, lo rows, 128 bytes each, swizzled
  static constexpr uint32_t X_AT = W_STAGES * W_STAGE, RED_AT = X_AT + X_STAGES * X_STAGE,
                            BAR_AT = RED_AT + (CLUSTER ? STRETCHES / 2 * NT * ROWS * 4 : 0);
  static constexpr int N_BARS = 2 * W_STAGES + 3 * SLOTS + 1;
  static constexpr size_t SMEM = BAR_AT + N_BARS * 8 + 16 + 1024;
  // warp 0 loads, 1 issues products, FEW: 2-3 split tokens, in turns; then the warps that split W, in SETS of four that take
  // turns, and those that drain, in PARTS of four that share a tile's columns, 16 at a time
  static constexpr int SETS = FEW ? 2 : 1, PARTS = FEW ? 1 : 3;
  static constexpr int SPLIT_WARP = FEW ? 4 : 2, DRAIN_WARP = SPLIT_WARP + 4 * SETS, THREADS = 32 * (DRAIN_WARP + 4 * PARTS);
  static constexpr int COLS = NT / PARTS;                    // columns a draining thread holds
  // columns of tensor memory: a chunk's two accumulators of hi hi', one of the small products, the chunks of W (hi, mid, lo: 32 each)
  static constexpr int SMALL_AT = 2 * NT, A_AT = (3 * NT + 31) / 32 * 32, A_COLS = 96, TMEM = 512;
  // A wait names a phase by its parity: whoever takes turns must see every phase of the stages that it waits for.  (With five
  // stages of W a set met a stage every second time round, and its wait was over while the phase before was still open.)
  static_assert(W_STAGES % SETS == 0, "a stage of W belongs to one set");
  static_assert(A_AT + A_COLS * A_STAGES <= TMEM && SMEM <= 227 * 1024 && COLS % 16 == 0 && COLS <= 32, "what a block has");
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

constexpr float SCALE = 16777216.f, BACK = 1.f / (SCALE * SCALE);      // what both operands are multiplied by, and the result's way back

// two neighbours as pairs of bfloat16 whose sums they are, times SCALE (lo has 8 bits: the rest's upper half as it is)
__device__ __forceinline__ void split2(float a, float b, uint32_t* hi, uint32_t* mid, uint32_t* lo) {
  const uint64_t minus1 = pack2(-1.f, -1.f);
  uint64_t rest = mul2(pack2(a, b), pack2(SCALE, SCALE));
  auto part = [&](uint32_t* to) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo_of(rest), hi_of(rest));
    *to = *reinterpret_cast<const uint32_t*>(&h);
  };
  auto subtract = [&](uint32_t v) { fma2(rest, (uint64_t)(v << 16) | (uint64_t)(v & 0xffff0000u) << 32, minus1); };     // exact
  part(hi);
  subtract(*hi);
  part(mid);
  subtract(*mid);
  *lo = __byte_perm((uint32_t)rest, (uint32_t)(rest >> 32), 0x7632);
}

// One lane of a warp that is together, the same at every call.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
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
  const bool vec = args.a_vec && args.w_vec;
  float sum = 0.f;
  for (int s = 0; s < args.K; s += args.seg) {
    float even = 0.f, odd = 0.f;
    const int end = min(args.K, s + args.seg);
    int k = s;
    for (; vec && k + 4 <= end; k += 4) {
      const float4 x = *reinterpret_cast<const float4*>(a + k), y = *reinterpret_cast<const float4*>(w + k);
      even = fmaf(x.z, y.z, fmaf(x.x, y.x, even));
      odd = fmaf(x.w, y.w, fmaf(x.y, y.y, odd));
    }
    for (; k < end; k += 2) {
      even = fmaf(a[k], w[k], even);
      if (k + 1 < end) odd = fmaf(a[k + 1], w[k + 1], odd);
    }
    sum += even + odd;
  }
  float* o = args.out + (size_t)m * args.ldo + n;
  *o = args.accumulate ? *o + sum : sum;
}
// A warp's results of token m that are no finite numbers (`mine`: this lane's is none).  A token that holds a NaN has no other results,
// and reading it is all that takes: a sequence that has diverged does not hold up the others of its step.
__device__ __noinline__ void again(const Args& args, int m, int n, bool mine) {
  const float* a = args.A + (size_t)m * args.lda;
  bool nan = false;
  for (int k = threadIdx.x & 31; k < args.K; k += 32) nan |= a[k] != a[k];
  if (__any_sync(0xffffffffu, nan)) {
    if (mine) args.out[(size_t)m * args.ldo + n] = __int_as_float(0x7fffffff);
  } else if (mine) {
    plain_result(args, m, n);
  }
}

// Splits `rows` rows of A into three planes [rows][chunks * 64] of 16-bit parts (zeros past K), four numbers a thread.
__global__ void __launch_bounds__(256)
split_rows_kernel(uint2* __restrict__ planes, const float* A, long lda, int rows, int K, int chunks, int a_vec) {
  gi::pdl_prologue();
  const long quads = (long)chunks * (CK / 4), i = (long)blockIdx.x * 256 + threadIdx.x, plane = rows * quads;
  if (i >= plane) return;
  const int m = (int)(i / quads), k = (int)(i % quads) * 4;
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  const float* src = A + (size_t)m * lda + k;
  if (a_vec && k + 4 <= K) {
    const float4 f = *reinterpret_cast<const float4*>(src);
    v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (k + e < K) v[e] = src[e];
  }
  uint2 hi, mid, lo;
  split2(v[0], v[1], &hi.x, &mid.x, &lo.x);
  split2(v[2], v[3], &hi.y, &mid.y, &lo.y);
  planes[i] = hi;
  planes[plane + i] = mid;
  planes[2 * plane + i] = lo;
}

// CLUSTER: `a.cluster` blocks share a tile's stretches (FEW only).  W_TMA: rows of W start on 16-byte boundaries; else its
// warps load their rows themselves.
template <bool FEW, bool CLUSTER, bool W_TMA>
__global__ void __launch_bounds__(Shape<FEW, CLUSTER>::THREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ Args a) {
  using S = Shape<FEW, CLUSTER>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t bars = smem_u32(smem + S::BAR_AT);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + S::BAR_AT + S::N_BARS * 8);
  // Barriers of a chunk: `full` - its rows of W are split (4 warps), its tokens are there (1) and its accumulators are drained (of the
  // chunk before; 4 warps a part); `large` - its hi hi' are made; `done` - all its products are, its operands' places are free.
  // `small` - a stretch's small products are read.
  const uint32_t w_full = bars, w_empty = w_full + 8 * S::W_STAGES, full = w_empty + 8 * S::W_STAGES, done = full + 8 * S::SLOTS,
                 large = done + 8 * S::SLOTS, small = large + 8 * S::SLOTS;
  auto wait_full = [&](int it, int who) { return mbar_wait(full + 8 * (it % S::SLOTS), (uint32_t)((it / S::SLOTS) & 1), who); };
  auto wait_done = [&](int it, int who) { return it < 0 || mbar_wait(done + 8 * (it % S::SLOTS), (uint32_t)((it / S::SLOTS) & 1), who); };
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < S::W_STAGES; ++i) {
      mbar_init(w_full + 8 * i, 1);
      mbar_init(w_empty + 8 * i, 4);
    }
    for (int i = 0; i < S::SLOTS; ++i) {
      mbar_init(full + 8 * i, 5 + 4 * S::PARTS);
      mbar_init(done + 8 * i, 1);
      mbar_init(large + 8 * i, 1);
    }
    mbar_init(small, 4 * S::PARTS);
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
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  gi::pdl_launch_dependents();
  gi::pdl_wait();

  if (warp == 0) {
    if (lane == 0 && (W_TMA || !FEW)) {
      bool ok = true;
      int it = 0, w_loaded = 0, x_loaded = 0;
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
            ++w_loaded;
          }
          if (!FEW) {
            const int st = it % S::X_STAGES, slot = it % S::SLOTS;
            ok = wait_done(it - S::X_STAGES, 1);
            if (!ok) break;
            const uint32_t dst = smem_u32(smem + S::X_AT + st * S::X_STAGE), bar = full + 8 * slot;
            mbar_expect_tx(bar, (uint32_t)a.nt * 384u);
            for (int p = 0; p < 3; ++p) tma_load_2d(dst + p * S::X_PART, &map_x, c * CK, p * a.M + m0, bar);
            ++x_loaded;
          }
        }
      }
      // the block does not leave before its copies have landed, also where somebody gave up
      for (int i = max(0, w_loaded - S::W_STAGES); i < w_loaded; ++i) mbar_wait(w_full + 8 * (i % S::W_STAGES), (uint32_t)((i / S::W_STAGES) & 1), 1);
      for (int i = max(0, x_loaded - S::X_STAGES); i < x_loaded; ++i) wait_full(i, 1);
    }
  } else if (warp == 1) {
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(a.nt >> 3) << 17) | ((uint32_t)(ROWS >> 4) << 24);   // float sums of bfloat16
    const uint32_t x_at = __shfl_sync(0xffffffffu, smem_u32(smem + S::X_AT), 0);
    bool ok = true;
    int it = 0, stretches = 0;
    for (int tile = tile0; tile < a.tiles && ok; tile += tile_step) {
      int left = 0;
      for (int c = c_first; c < c_last && ok; ++c, ++it) {
        const int as = it % S::A_STAGES, xs = it % S::X_STAGES;
        const bool fresh = left == 0;                        // a stretch begins
        left = (fresh ? a.per_stretch : left) - 1;
        ok = __all_sync(0xffffffffu, wait_full(it, 2));
        if (!ok) break;
        tc_fence_after();
        const uint32_t s = tmem + S::SMALL_AT, hi = tmem + S::A_AT + as * S::A_COLS, mid = hi + 32, lo = hi + 64;
        const uint64_t x_hi = smem_desc(x_at + xs * S::X_STAGE), x_mid = x_hi + (S::X_PART >> 4), x_lo = x_hi + (2 * S::X_PART >> 4);
        auto product = [&](uint32_t w, uint64_t x, bool first) {
#pragma unroll
          for (int k = 0; k < CK / 16; ++k) mma_a_tmem(s, w + 8 * k, x + 2 * k, idesc, !(first && k == 0));
        };
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < CK / 16; ++k) mma_a_tmem(tmem + k / 2 * S::NT, hi + 8 * k, x_hi + 2 * k, idesc, k & 1);
          tc_commit(large + 8 * (it % S::SLOTS));
        }
        if (fresh && stretches++ > 0) {
          ok = __all_sync(0xffffffffu, mbar_wait(small, (uint32_t)(stretches & 1), 2));
          if (!ok) break;
          tc_fence_after();
        }
        if (elect_one()) {
          product(mid, x_hi, fresh);
          product(hi, x_mid, false);
          product(mid, x_mid, false);
          product(lo, x_hi, false);
          product(hi, x_lo, false);
          tc_commit(done + 8 * (it % S::SLOTS));
        }
        __syncwarp();
      }
    }
    wait_done(it - 1, 2);                                    // its products, as the loads above
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
        ok = wait_done(it - S::A_STAGES, 3);
        if (!ok) break;
        tc_fence_after();
        const uint32_t dst = tmem + lane_base + S::A_AT + as * S::A_COLS;
#pragma unroll
        for (int q = 0; q < CK / 16; ++q) {
          uint32_t hi[8], mid[8], lo[8];
          float4 v[4];
#pragma unroll
          for (int p = 0; p < 4; ++p) v[p] = piece(4 * q + p);
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            const float4 f = v[p];
            split2(f.x, f.y, &hi[2 * p], &mid[2 * p], &lo[2 * p]);
            split2(f.z, f.w, &hi[2 * p + 1], &mid[2 * p + 1], &lo[2 * p + 1]);
          }
          tc_st8(dst + 8 * q, hi);
          tc_st8(dst + 32 + 8 * q, mid);
          tc_st8(dst + 64 + 8 * q, lo);
        }
        if (W_TMA) {
          __syncwarp();
          if (lane == 0) mbar_arrive(w_empty + 8 * ws);
        }
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
    if (lane == 0) mbar_arrive(full);                        // nothing to drain before the first chunk
    for (int tile = tile0; tile < a.tiles && ok; tile += tile_step) {
      const int m0 = tile % a.tiles_m * a.nt, n = tile / a.tiles_m * ROWS + row, nt = a.nt;
      uint64_t acc[S::COLS / 2], sum[S::COLS / 2];
#pragma unroll
      for (int j = 0; j < S::COLS / 2; ++j) acc[j] = sum[j] = 0;
      // an accumulator's columns of this part, added (columns past the tile's tokens hold what nobody reads)
      auto take = [&](uint32_t d) {
#pragma unroll
        for (int g = 0; g < GROUPS; ++g)
          if (col_of(g) < nt) {
            uint32_t r[GROUP];
            tc_ld16(d + col_of(g), r);
            wait_ld16(r);
#pragma unroll
            for (int j = 0; j < GROUP; j += 2) {
              uint64_t& v = acc[(g * GROUP + j) / 2];
              v = add2(v, (uint64_t)r[j] | (uint64_t)r[j + 1] << 32);
            }
          }
      };
      int left = a.per_stretch, stretch = 0;
      for (int c = c_first; c < c_last && ok; ++c, ++it) {
        ok = mbar_wait(large + 8 * (it % S::SLOTS), (uint32_t)((it / S::SLOTS) & 1), 4);
        if (!ok) break;
        tc_fence_after();
        take(tmem + lane_base);
        take(tmem + lane_base + S::NT);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(full + 8 * ((it + 1) % S::SLOTS));
        const bool ends = --left == 0 || c + 1 == c_last;    // a stretch ends
        if (ends) {
          ok = wait_done(it, 4);
          if (!ok) break;
          tc_fence_after();
          take(tmem + lane_base + S::SMALL_AT);
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(small);
        }
        if (!ends) continue;
        left = a.per_stretch;
        if constexpr (CLUSTER) {
          // where the cluster reads it
          float* red = reinterpret_cast<float*>(smem + S::RED_AT) + stretch * FEW_TILE * ROWS;
#pragma unroll
          for (int j = 0; j < S::COLS / 2; ++j) {
            red[(2 * j) * ROWS + row] = lo_of(acc[j]);
            red[(2 * j + 1) * ROWS + row] = hi_of(acc[j]);
          }
        } else {
#pragma unroll
          for (int j = 0; j < S::COLS / 2; ++j) sum[j] = stretch == 0 ? acc[j] : add2(sum[j], acc[j]);
        }
#pragma unroll
        for (int j = 0; j < S::COLS / 2; ++j) acc[j] = 0;
        ++stretch;
      }
      if (!ok) break;
      if constexpr (!CLUSTER) {
        const int live = n < a.N ? min(nt, a.M - m0) : 0;
        const long ldo = a.ldo;
        const bool add = a.accumulate != 0;
        float* o = a.out + (size_t)m0 * ldo + n;
        uint32_t odd = 0;                                    // results that are no finite numbers: after the others
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
          const int col = col_of(g);
#pragma unroll
          for (int j = 0; j < GROUP; ++j) {
            const uint64_t both = sum[(g * GROUP + j) / 2];
            const float v = ((j & 1) ? hi_of(both) : lo_of(both)) * BACK;
            float* at = o + (size_t)(col + j) * ldo;
            if (col + j < live) {
              if (fabsf(v) <= FLT_MAX) *at = add ? *at + v : v;
              else odd |= 1u << (g * GROUP + j);
            }
          }
        }
        for (uint32_t rest = __reduce_or_sync(0xffffffffu, odd); rest; rest &= rest - 1) {
          const int i = __ffs((int)rest) - 1;
          again(a, m0 + col_of(i / GROUP) + i % GROUP, n, (odd >> i & 1) != 0);
        }
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
        uint2 hi, mid, lo;
        split2(v[i].x, v[i].y, &hi.x, &mid.x, &lo.x);
        split2(v[i].z, v[i].w, &hi.y, &mid.y, &lo.y);
        unsigned char* dst = smem + S::X_AT + xs * S::X_STAGE + m * 128 + ((l >> 1) ^ (m & 7)) * 16 + (l & 1) * 8;
        *reinterpret_cast<uint2*>(dst) = hi;
        *reinterpret_cast<uint2*>(dst + S::X_PART) = mid;
        *reinterpret_cast<uint2*>(dst + 2 * S::X_PART) = lo;
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
    for (int i = rank * S::THREADS + (int)threadIdx.x; i < min(FEW_TILE, a.M - m0) * ROWS; i += a.cluster * S::THREADS) {     // whole warps
      const int m = m0 + i / ROWS, n = n0 + i % ROWS;
      float parts[STRETCHES];
#pragma unroll
      for (int r = 0; r < STRETCHES; ++r) parts[r] = r < used ? ld_remote(red + 4u * (uint32_t)(r % mine * FEW_TILE * ROWS + i), r / mine) : 0.f;
      float v = parts[0];
#pragma unroll
      for (int r = 1; r < STRETCHES; ++r)
        if (r < used) v += parts[r];
      v *= BACK;
      const bool fine = fabsf(v) <= FLT_MAX;
      if (n < a.N && fine) {
        float* o = a.out + (size_t)m * a.ldo + n;
        *o = a.accumulate ? *o + v : v;
      }
      const bool odd = n < a.N && !fine;
      if (__any_sync(0xffffffffu, odd)) again(a, m, n, odd);
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
int launch_split(const CUtensorMap& mw, const CUtensorMap& mx, const Args& a, int blocks, cudaStream_t s) {
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
  return gi::check(cudaLaunchKernelEx(&cfg, gemm_split_kernel<FEW, CLUSTER, W_TMA>, mw, mx, a), "gemm_f32_split");
}

long planes_bytes(long rows, int chunks) { return 3 * rows * chunks * CK * 2; }

}  // namespace

// Bytes of scratch that a product of these sizes needs, -1 where the plain kernels take it.
extern "C" long gi_gemm_f32_split_scratch(int M, int N, int K) {
  if (M <= 0 || N < 1024 || K < 1024) return -1;
  if (M <= FEW_MAX) return 0;
  const int rows = M < SLAB ? M : SLAB, chunks = (K + CK - 1) / CK;
  return planes_bytes(rows, chunks);
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
  a.w_vec = (ldw % 4 == 0 && ((uintptr_t)W & 15) == 0) ? 1 : 0;
  a.accumulate = mode == GI_GEMM_ACCUM_F32 ? 1 : 0;
  const bool w_tma = a.w_vec && K % 4 == 0;
  CUtensorMap mw = {}, mx = {};
  if (w_tma) {
    const int rc = gi::tensor_map_2d_ex(&mw, W, N, K, ldw, GI_F32, 32, ROWS);
    if (rc != GI_OK) return rc;
  }
  if (M <= FEW_MAX) {
    a.out = out; a.A = A;
    a.M = M; a.nt = FEW_TILE; a.tiles_m = (M + FEW_TILE - 1) / FEW_TILE; a.tiles = a.tiles_m * tiles_n;
    a.cluster = w_tma ? cluster_of<true>(a.tiles) : cluster_of<false>(a.tiles);
    if (a.cluster > 1)
      return w_tma ? launch_split<true, true, true>(mw, mx, a, a.tiles * a.cluster, s) : launch_split<true, true, false>(mw, mx, a, a.tiles * a.cluster, s);
    const int blocks = a.tiles < sms ? a.tiles : sms;
    return w_tma ? launch_split<true, false, true>(mw, mx, a, blocks, s) : launch_split<true, false, false>(mw, mx, a, blocks, s);
  }
  for (int m0 = 0; m0 < M; m0 += SLAB) {
    const int rows = M - m0 < SLAB ? M - m0 : SLAB;
    a.out = out + (size_t)m0 * ldo;
    a.A = A + (size_t)m0 * lda;
    a.M = rows;
    const long quads = (long)rows * a.chunks * (CK / 4);
    int rc = gi::check(gi::launch(split_rows_kernel, dim3((unsigned)((quads + 255) / 256)), dim3(256), 0, s, (uint2*)scratch, a.A, lda, rows, K,
                                  a.chunks, a.a_vec), "gemm_f32_split: tokens");
    if (rc != GI_OK) return rc;
    // tokens a tile: a chunk takes a block about 1,100 + 11 tokens clocks (2,048 x 8,192: 1,640 in tiles of 48, 2,000 in tiles of 80), a
    // launch as many rounds of tiles as the fullest SM has
    long best = 0;
    for (int nt = 16; nt <= Shape<false, false>::NT; nt += 16) {
      const long tiles = (long)((rows + nt - 1) / nt) * tiles_n, cost = (tiles + sms - 1) / sms * (1100 + 11 * nt);
      if (best == 0 || cost <= best) best = cost, a.nt = nt, a.tiles_m = (rows + nt - 1) / nt;
    }
    a.tiles = a.tiles_m * tiles_n;
    // one map over the three planes (a tile's rows past the last token are the next plane's: nobody reads their results)
    rc = gi::tensor_map_2d_ex(&mx, scratch, 3L * rows, (long)a.chunks * CK, (long)a.chunks * CK, GI_BF16, 64, a.nt);
    if (rc != GI_OK) return rc;
    const int blocks = a.tiles < sms ? a.tiles : sms;
    rc = w_tma ? launch_split<false, false, true>(mw, mx, a, blocks, s) : launch_split<false, false, false>(mw, mx, a, blocks, s);
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
