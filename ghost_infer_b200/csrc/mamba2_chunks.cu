// The Mamba-2 recurrence of a prompt step in 16-bit rows, 64 tokens at a time as matrix products (the "state-space dual"
// form of Dao and Gu, 2024), beside the token-by-token walk of mamba2.cu, which serves short stretches and the 32-bit path.
//
// With a_t = -exp(A_log) dt_t and c_t the sum of a over a chunk's tokens up to t, S the state before the chunk:
//     y_i  = exp(c_i) C_i S  +  sum_{j <= i} (C_i . B_j) exp(c_i - c_j) dt_j x_j  +  D x_i
//     S   <- exp(c_last) S   +  sum_j B_j (exp(c_last - c_j) dt_j x_j)^T
// The walk was bound by its chain: 64 heads x 64 columns of one prompt are 7 warps an SM, each with 2,048 dependent steps.
// Here a block takes a head's 32 columns of S (128 blocks for 64 heads of 64) and walks the chunks; eight warps form the
// four products with mma.sync.  B, C and x are 16-bit numbers and enter exactly; what is 32-bit (S, the weighted x, the
// decayed scores) enters as three 16-bit parts, 24 bits together, in three products.  Sums are 32-bit.  The tensor cores cut
// off what does not fit into a sum that they add to themselves, so the products that make up most of y (C . B, scores x)
// leave them 16 numbers at a time and are added with one rounding to nearest, and a chunk's addition to S is summed apart
// and joined with one rounding.  c is summed in 64 bits: exp(c_i - c_j) of neighbours would lose the digits that c has grown
// by.  Distance of y from 64 bits, 64 heads of 64, N 128, 512 tokens (the walk's beside it): 0.95e-7 (0.95e-7) where a state
// lasts a few tokens, 1.2e-7 (39e-7) where it lasts hundreds, 0.88e-7 (0.71e-7) where it is gone at the next token; with sums
// left to the tensor cores 1.2e-7, 1.2e-7 and 1.1e-7, for 1% less time.
// Between different 16-token tiles decays are products of two factors, both at most 1, taken at the later tile's start:
// 64 + 96 exponentials a chunk for 1,536 pairs.  The pairs inside the four diagonal tiles take one each (544, in both halves
// of the columns), and a token's weight for S is worked out by the four threads that apply it.
// Rows and columns past N, P and the chunk's end are zeros.  A block that meets an infinity or a not-a-number walks its
// tokens one by one after all (`walk_all`), so that neither reaches an earlier token.
// B200, 2,048 tokens, 64 heads of 64, N 128: 176 us, the walk 660 us; 64 heads of 40, N 96: 165 and 536 us.  What bounds it
// now is the chain of a chunk (about 5 us: operands out of shared memory, four products one after the other, two barriers),
// not the tensor cores' rate.
#include <math.h>

#include <type_traits>

#include "api.h"
#include "common.cuh"
#include "mma_utils.cuh"

namespace {

constexpr int Q = 64, PT = 32, THREADS = 256;
constexpr int XP = PT * 2 + 16;                    // bytes of a row of 32 columns, padded: an odd number of 16-byte words

__device__ __forceinline__ float softplus_f(float v) { return v > 20.f ? v : log1pf(expf(v)); }

// v = parts[0] + parts[1] + parts[2] to 24 bits
__device__ __forceinline__ void split3(float v, __nv_bfloat16 (&part)[3]) {
  part[0] = __float2bfloat16_rn(v);
  const float r = v - __bfloat162float(part[0]);
  part[1] = __float2bfloat16_rn(r);
  part[2] = __float2bfloat16_rn(r - __bfloat162float(part[1]));
}
__device__ __forceinline__ void split3_pair(float lo, float hi, uint32_t (&out)[3]) {
  __nv_bfloat16 a[3], b[3];
  split3(lo, a);
  split3(hi, b);
#pragma unroll
  for (int i = 0; i < 3; ++i) out[i] = (uint32_t)__bfloat16_as_ushort(a[i]) | (uint32_t)__bfloat16_as_ushort(b[i]) << 16;
}

// acc + a b, the product over 16 numbers added with one rounding to nearest: the tensor cores cut off what does not fit into a
// sum that they add to themselves
__device__ __forceinline__ void add_mma(float (&acc)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  float t[4] = {};
  gi::mma_16816(t, a, b0, b1);
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i] += t[i];
}

template <int NT>
struct Layout {
  static constexpr int NP = 16 * NT;                         // rows of S with padding
  static constexpr int BP = NP * 2 + 16;                     // bytes of a row of B or C, padded
  static constexpr int C_AT = 0, B_AT = Q * BP, X_AT = 2 * Q * BP, BUF = X_AT + Q * XP;
  static constexpr int S_AT = 2 * BUF, S_PART = NP * XP;     // two buffers of S in three parts, [n][column]
  static constexpr int W_AT = S_AT + 2 * 3 * S_PART, W_PART = Q * XP;   // weighted x in three parts
  static constexpr int CUM_AT = W_AT + 3 * W_PART;           // double[2][Q]
  static constexpr int DT_AT = CUM_AT + 2 * 8 * Q;           // float[2][Q]
  static constexpr int EI_AT = DT_AT + 2 * 4 * Q, EJ_AT = EI_AT + 4 * Q, IN_AT = EJ_AT + 16 * Q, BYTES = IN_AT + 4 * Q;
};

// The whole stretch token by token, by a block that met an infinity or a not-a-number: a product over 16 tokens lets one
// token's meet the zero weights of earlier ones, and a split infinity is none any more, where the recurrence carries both
// forward only.  The state in memory is still that before the step, and `y` is written again.  `bc`, `x`, `dt_in`: the first
// token's row of B, of x from this block's first column on (`cols` of them exist), its step size before softplus; C is
// `c_after` numbers behind B.  Thread: column tid % 32, every eighth row from tid / 32 on.
template <int NT>
__device__ __noinline__ void walk_all(unsigned char* smem, float* y, int inner, const __nv_bfloat16* bc, const __nv_bfloat16* x, int channels,
                                      int c_after, const __nv_bfloat16* dt_in, long ld_proj, float* S_cols, int qlen, int cols, int N,
                                      float A, float D, float bias) {
  using L = Layout<NT>;
  constexpr int ROWS = L::NP / 8;
  const int tid = threadIdx.x, p = tid & 31, first = tid >> 5;
  float* sB = reinterpret_cast<float*>(smem);                // [32][NP]
  float* sC = sB + 32 * L::NP;
  float* sx = sC + 32 * L::NP;                               // [32][PT]
  float* sdt = sx + 32 * PT;
  float* sums = sdt + 32;                                    // [8][32]
  float S[ROWS];
#pragma unroll
  for (int k = 0; k < ROWS; ++k) S[k] = p < cols && first + 8 * k < N ? S_cols[(size_t)p * N + first + 8 * k] : 0.f;
  for (int c0 = 0; c0 < qlen; c0 += 32) {
    const int nc = min(32, qlen - c0);
    __syncthreads();
    for (int i = tid; i < nc * N; i += THREADS) {
      const __nv_bfloat16* at = bc + (size_t)(c0 + i / N) * channels + i % N;
      sB[i / N * L::NP + i % N] = gi::ldf(at);
      sC[i / N * L::NP + i % N] = gi::ldf(at + c_after);
    }
    for (int i = tid; i < nc * PT; i += THREADS) sx[i] = i % PT < cols ? gi::ldf(x + (size_t)(c0 + i / PT) * channels + i % PT) : 0.f;
    if (tid < nc) sdt[tid] = softplus_f(gi::ldf(dt_in + (size_t)(c0 + tid) * ld_proj) + bias);
    __syncthreads();
    for (int t = 0; t < nc; ++t) {
      const float dt = sdt[t], keep = expf(A * dt), xv = sx[t * PT + p];
      float sum = 0.f;
#pragma unroll
      for (int k = 0; k < ROWS; ++k) {
        const int n = first + 8 * k;
        if (n < N) {
          S[k] = fmaf(keep, S[k], xv * (sB[t * L::NP + n] * dt));
          sum = fmaf(S[k], sC[t * L::NP + n], sum);
        }
      }
      sums[tid] = sum;
      __syncthreads();
      if (first == 0 && p < cols) {
        sum = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) sum += sums[w * 32 + p];
        y[(size_t)(c0 + t) * inner + p] = fmaf(D, xv, sum);
      }
      __syncthreads();
    }
  }
#pragma unroll
  for (int k = 0; k < ROWS; ++k)
    if (p < cols && first + 8 * k < N) S_cols[(size_t)p * N + first + 8 * k] = S[k];
}

// grid (heads, sequences, column tiles of 32)
template <int NT>
__global__ void __launch_bounds__(THREADS, 1)
mamba2_chunks_kernel(float* __restrict__ y, const __nv_bfloat16* xbc, const __nv_bfloat16* proj, long ld_proj, const float* dt_bias,
                     const float* a_log, const float* d_skip, float* state, long state_ld, int state_rows, const int* cu_seqlens,
                     const int* seq_slots, int heads, int P, int N, int groups, int from) {
  using L = Layout<NT>;
  extern __shared__ __align__(16) unsigned char smem[];
  const uint32_t base = gi::smem_u32(smem);
  double* cum_s = reinterpret_cast<double*>(smem + L::CUM_AT);
  float* dt_s = reinterpret_cast<float*>(smem + L::DT_AT);
  float* ei = reinterpret_cast<float*>(smem + L::EI_AT);
  float* ej = reinterpret_cast<float*>(smem + L::EJ_AT);     // [row tile][token]
  float* e_in = reinterpret_cast<float*>(smem + L::IN_AT);
  gi::pdl_prologue();
  const int h = blockIdx.x, b = blockIdx.y, p0 = blockIdx.z * PT;
  const int tok0 = cu_seqlens[b], qlen = cu_seqlens[b + 1] - tok0;
  if (qlen < from) return;
  const int slot = seq_slots[b];
  float* S_row = state + (size_t)(slot >= 0 ? slot : state_rows - 1) * state_ld + (size_t)h * N * P;
  const int g = h / (heads / groups);
  const int inner = heads * P, channels = inner + 2 * groups * N;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int lr = lane >> 2, lc = (lane & 3) * 2;             // row and first column of a lane in an accumulator tile
  const float A = -expf(a_log[h]), D = d_skip[h], bias = dt_bias[h];
  const __nv_bfloat16* dt_in = proj + 2 * (size_t)inner + 2 * (size_t)groups * N + h;

  auto load = [&](int c0, int buf) {
    const int nc = min(Q, qlen - c0);
    const uint32_t dst = base + buf * L::BUF;
    const __nv_bfloat16* rows = xbc + (size_t)(tok0 + c0) * channels;
    for (int i = tid; i < Q * NT * 2; i += THREADS) {
      const int t = i / (NT * 2), w = i % (NT * 2);
      const bool ok = t < nc && w * 8 < N;
      const __nv_bfloat16* src = rows + (ok ? (size_t)t * channels + inner + (size_t)g * N + w * 8 : 0);
      gi::cp_async_16(dst + L::B_AT + t * L::BP + w * 16, src, ok ? 16 : 0);
      gi::cp_async_16(dst + L::C_AT + t * L::BP + w * 16, ok ? src + (size_t)groups * N : rows, ok ? 16 : 0);
    }
    {
      const int t = tid >> 2, w = tid & 3;
      const bool ok = t < nc && p0 + w * 8 < P;
      gi::cp_async_16(dst + L::X_AT + t * XP + w * 16, ok ? rows + (size_t)t * channels + (size_t)h * P + p0 + w * 8 : rows, ok ? 16 : 0);
    }
    gi::cp_async_commit();
  };
  // warp 0, whose row tile has the least to do, works out the next chunk's step sizes and their sums, two a lane; what it
  // reads for that was asked for a chunk earlier
  float raw[2] = {0.f, 0.f};
  auto load_dt = [&](int c0) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = c0 + 2 * lane + i;
      raw[i] = t < qlen ? gi::ldf(dt_in + (size_t)(tok0 + t) * ld_proj) : 0.f;
    }
  };
  auto sum_dt = [&](int c0, int buf) {
    float dt[2];
    double s[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      dt[i] = c0 + 2 * lane + i < qlen ? softplus_f(raw[i] + bias) : 0.f;
      s[i] = (double)(A * dt[i]);
    }
    double run = s[0] + s[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double up = __shfl_up_sync(0xffffffffu, run, o);
      if (lane >= o) run += up;
    }
    double* cum = cum_s + buf * Q + 2 * lane;
    cum[0] = run - s[1];
    cum[1] = run;
    *reinterpret_cast<float2*>(dt_s + buf * Q + 2 * lane) = make_float2(dt[0], dt[1]);
  };
  load(0, 0);
  if (warp == 0) {
    load_dt(0);
    sum_dt(0, 0);
    load_dt(Q);
  }

  // warps below NT hold 16 rows of S each: sacc[k] is columns 8 k .. + 7
  float sacc[4][4];
  const int srow = 16 * warp + lr;
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int n = srow + (i >> 1) * 8, p = p0 + 8 * k + lc + (i & 1);
      sacc[k][i] = (warp < NT && n < N && p < P) ? S_row[(size_t)p * N + n] : 0.f;
    }
  auto put_state = [&](int buf) {
    if (warp < NT) {
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          uint32_t part[3];
          split3_pair(sacc[k][2 * r], sacc[k][2 * r + 1], part);
#pragma unroll
          for (int s = 0; s < 3; ++s)
            *reinterpret_cast<uint32_t*>(smem + L::S_AT + (3 * buf + s) * L::S_PART + (srow + 8 * r) * XP + (8 * k + lc) * 2) = part[s];
        }
    }
  };
  // 0 while all that this thread found is finite, the state also when rounded to 16 bits; not-a-number after that
  float odd = 0.f;
  auto check_state = [&] {
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int i = 0; i < 4; ++i) odd = fmaf(sacc[k][i] * 1.0625f, 0.f, odd);
  };
  check_state();
  put_state(0);

  // this warp's rows and columns of y: of the two warps a scheduler holds one has a late row tile, one an early one
  const int rt = warp < 4 ? warp : 7 - warp, ch = warp >> 2;
  const uint32_t a_row = (uint32_t)((lane & 7) + ((lane >> 3) & 1) * 8), a_col = (uint32_t)(lane >> 4) * 16;   // ldmatrix rows, bytes
  const uint32_t b_row = (uint32_t)((lane & 7) + (lane >> 4) * 8), b_col = (uint32_t)((lane >> 3) & 1) * 16;

  // A chunk.  Only a sequence's last one may have fewer tokens; its late row tiles are then left out (65 tokens of 16 sequences,
  // 64 heads of 64, N 128: 185 us -> 164), in a copy of its own, since the tests alone cost full chunks 2%.
  auto chunk = [&](int c0, int buf, auto full) {
    constexpr bool FULL = decltype(full)::value;
    const int nc = FULL ? Q : qlen - c0;
    const double* cum = cum_s + buf * Q;
    const float* sdt = dt_s + buf * Q;
    const double last = cum[Q - 1];
    const unsigned char* bx = smem + buf * L::BUF + L::X_AT;
    {
      // tables: exp(c_i - c at its tile's start), exp(c at a tile's start - c_j) dt_j for earlier j, exp(c_i)
      const int r = tid >> 6, t = tid & 63;
      const double start = r > 0 ? cum[16 * r - 1] : 0.0;
      if (r == 0) {
        const int ti = t >> 4;
        ei[t] = expf((float)(cum[t] - (ti > 0 ? cum[16 * ti - 1] : 0.0)));
        e_in[t] = expf((float)cum[t]);
      } else if (t < 16 * r) {
        ej[r * Q + t] = expf((float)(start - cum[t])) * sdt[t];
      }
      // weighted x in three parts: eight columns of a token
      const int j = tid >> 2, w8 = (tid & 3) * 16;
      const float we = expf((float)(last - cum[j])) * sdt[j];
      const uint4 xv = *reinterpret_cast<const uint4*>(bx + j * XP + w8);
      const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
      uint32_t part[4][3];
#pragma unroll
      for (int k = 0; k < 4; ++k) split3_pair(__uint_as_float(xw[k] << 16) * we, __uint_as_float(xw[k] & 0xffff0000u) * we, part[k]);
#pragma unroll
      for (int s = 0; s < 3; ++s)
        *reinterpret_cast<uint4*>(smem + L::W_AT + s * L::W_PART + j * XP + w8) = make_uint4(part[0][s], part[1][s], part[2][s], part[3][s]);
    }
    __syncthreads();

    const uint32_t cb = base + buf * L::BUF;
    if (FULL || 16 * rt < nc) {
      float main[2][4] = {}, main1[2][4] = {}, small[2][4] = {};
      uint32_t cf[NT][4];
#pragma unroll
      for (int k = 0; k < NT; ++k) {
        gi::ldmatrix_x4(cf[k], cb + L::C_AT + (16 * rt + a_row) * L::BP + k * 32 + a_col);
#pragma unroll
        for (int s = 2; s >= 0; --s) {
          uint32_t f[4];
          gi::ldmatrix_x4_trans(f, base + L::S_AT + (3 * buf + s) * L::S_PART + (16 * k + a_row) * XP + ch * 32 + a_col);
          float (&acc)[2][4] = s > 0 ? small : (k & 1) ? main1 : main;
          gi::mma_16816(acc[0], cf[k], f[0], f[1]);
          gi::mma_16816(acc[1], cf[k], f[2], f[3]);
        }
      }
      const int i0 = 16 * rt + lr;
      float yin[2][4];                                         // what the state before the chunk gives
      {
        const float t0 = e_in[i0], t1 = e_in[i0 + 8];
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            yin[k][i] = ((main[k][i] + main1[k][i]) + small[k][i]) * (i < 2 ? t0 : t1);
            main[k][i] = small[k][i] = 0.f;
          }
      }
      const float e0 = ei[i0], e1 = ei[i0 + 8];
      for (int jt = 0; jt <= rt; ++jt) {
        float m[2][4] = {};
#pragma unroll
        for (int k = 0; k < NT; ++k) {
          uint32_t f[4];
          gi::ldmatrix_x4(f, cb + L::B_AT + (16 * jt + b_row) * L::BP + k * 32 + b_col);
          add_mma(m[0], cf[k], f[0], f[1]);
          add_mma(m[1], cf[k], f[2], f[3]);
        }
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int j = 16 * jt + 8 * k + lc + e;
            if (jt < rt) {
              const float w = ej[rt * Q + j];
              m[k][e] *= e0 * w;
              m[k][2 + e] *= e1 * w;
            } else {
              const double cj = cum[j];
              const float dt = sdt[j];
              m[k][e] = i0 >= j ? m[k][e] * (expf((float)(cum[i0] - cj)) * dt) : 0.f;
              m[k][2 + e] = i0 + 8 >= j ? m[k][2 + e] * (expf((float)(cum[i0 + 8] - cj)) * dt) : 0.f;
            }
          }
        uint32_t a01[3], a23[3], b01[3], b23[3], xf[4];
        split3_pair(m[0][0], m[0][1], a01);
        split3_pair(m[0][2], m[0][3], a23);
        split3_pair(m[1][0], m[1][1], b01);
        split3_pair(m[1][2], m[1][3], b23);
        gi::ldmatrix_x4_trans(xf, cb + L::X_AT + (16 * jt + a_row) * XP + ch * 32 + a_col);
#pragma unroll
        for (int s = 2; s >= 0; --s) {
          const uint32_t af[4] = {a01[s], a23[s], b01[s], b23[s]};
          if (s > 0) {
            gi::mma_16816(small[0], af, xf[0], xf[1]);
            gi::mma_16816(small[1], af, xf[2], xf[3]);
          } else {
            add_mma(main[0], af, xf[0], xf[1]);
            add_mma(main[1], af, xf[2], xf[3]);
          }
        }
      }
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          yin[k][i] += main[k][i] + small[k][i];
          odd = fmaf(yin[k][i], 0.f, odd);
        }
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int i = i0 + 8 * r, col = ch * 16 + 8 * k + lc;
          if (i < nc && p0 + col < P) {
            const uint32_t xv = *reinterpret_cast<const uint32_t*>(bx + i * XP + col * 2);
            const float2 o = make_float2(fmaf(D, __uint_as_float(xv << 16), yin[k][2 * r]),
                                         fmaf(D, __uint_as_float(xv & 0xffff0000u), yin[k][2 * r + 1]));
            *reinterpret_cast<float2*>(y + (size_t)(tok0 + c0 + i) * inner + (size_t)h * P + p0 + col) = o;
          }
        }
    }

    if (warp < NT) {
      float add[4][4] = {}, low[4][4] = {};
#pragma unroll
      for (int k = 0; k < Q / 16; ++k) {
        if (!FULL && 16 * k >= nc) break;
        uint32_t af[4];
        gi::ldmatrix_x4_trans(af, cb + L::B_AT + (16 * k + b_row) * L::BP + warp * 32 + b_col);
#pragma unroll
        for (int s = 2; s >= 0; --s)
#pragma unroll
          for (int n2 = 0; n2 < 2; ++n2) {
            uint32_t f[4];
            gi::ldmatrix_x4_trans(f, base + L::W_AT + s * L::W_PART + (16 * k + a_row) * XP + n2 * 32 + a_col);
            gi::mma_16816(s > 0 ? low[2 * n2] : add[2 * n2], af, f[0], f[1]);
            gi::mma_16816(s > 0 ? low[2 * n2 + 1] : add[2 * n2 + 1], af, f[2], f[3]);
          }
      }
      const float keep = expf((float)last);
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int i = 0; i < 4; ++i) sacc[k][i] = fmaf(keep, sacc[k][i], add[k][i] + low[k][i]);
      check_state();
      put_state(buf ^ 1);
    }
    if (warp == 0 && c0 + Q < qlen) {
      sum_dt(c0 + Q, buf ^ 1);
      load_dt(c0 + 2 * Q);
    }
  };
  bool walk = false;
  for (int c0 = 0, buf = 0; c0 < qlen; c0 += Q, buf ^= 1) {
    gi::cp_async_wait<0>();
    // the chunk, its sums and S are in shared memory; the other buffers are free
    walk = __syncthreads_or(odd != 0.f);
    if (walk) break;
    if (c0 + Q < qlen) load(c0 + Q, buf ^ 1);
    if (qlen - c0 >= Q) chunk(c0, buf, std::true_type());
    else chunk(c0, buf, std::false_type());
  }
  if (walk || __syncthreads_or(odd != 0.f)) {
    walk_all<NT>(smem, y + (size_t)tok0 * inner + (size_t)h * P + p0, inner, xbc + (size_t)tok0 * channels + inner + (size_t)g * N,
                 xbc + (size_t)tok0 * channels + (size_t)h * P + p0, channels, groups * N, dt_in + (size_t)tok0 * ld_proj, ld_proj,
                 S_row + (size_t)p0 * N, qlen, min(PT, P - p0), N, A, D, bias);
    return;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int n = srow + (i >> 1) * 8, p = p0 + 8 * k + lc + (i & 1);
      if (warp < NT && n < N && p < P) S_row[(size_t)p * N + n] = sacc[k][i];
    }
}

template <int NT>
int launch_chunks(dim3 grid, cudaStream_t s, float* y, const void* xbc, const void* proj, long ld_proj, const float* dt_bias, const float* a_log,
           const float* d_skip, float* state, long state_ld, int state_rows, const int* cu, const int* slots, int heads, int P, int N, int groups, int from) {
  static bool seen[gi::MAX_DEVICES_SEEN];
  int dev;
  if (gi::unconfigured_here(seen, &dev)) {
    if (cudaFuncSetAttribute(mamba2_chunks_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Layout<NT>::BYTES) != cudaSuccess)
      return gi::check_launch("mamba2 chunks: shared memory");
    if (dev >= 0) seen[dev] = true;
  }
  return gi::check(gi::launch(mamba2_chunks_kernel<NT>, grid, dim3(THREADS), Layout<NT>::BYTES, s, y, (const __nv_bfloat16*)xbc,
                              (const __nv_bfloat16*)proj, ld_proj, dt_bias, a_log, d_skip, state, state_ld, state_rows, cu, slots, heads, P, N,
                              groups, from), "mamba2 chunks");
}

}  // namespace

extern "C" int gi_mamba2_chunks(float* y, const void* xbc, const void* proj, long ld_proj, const float* dt_bias, const float* a_log,
                                const float* d_skip, float* state, long state_ld, int state_rows, const int* cu_seqlens,
                                const int* seq_slots, int n_seqs, int heads, int P, int N, int groups, int from, void* stream) {
  if (n_seqs <= 0) return GI_OK;
  if (heads <= 0 || P <= 0 || N <= 0 || groups <= 0 || heads % groups != 0 || from < 1)
    return gi::fail(GI_ERR_ARG, "mamba2 chunks: %d heads, %d groups, head size %d, state %d", heads, groups, P, N);
  if (P % 8 != 0 || N % 8 != 0 || N > 128 || ((uintptr_t)xbc & 15) || ((uintptr_t)y & 7))
    return gi::fail(GI_ERR_UNSUPPORTED, "mamba2 chunks: head size and state must be multiples of 8, the state at most 128, rows aligned");
  if (n_seqs > 65535 || (P + PT - 1) / PT > 65535) return gi::fail(GI_ERR_UNSUPPORTED, "mamba2 chunks: more than one launch takes");
  const dim3 grid(heads, n_seqs, (P + PT - 1) / PT);
  cudaStream_t s = (cudaStream_t)stream;
#define GI_CHUNKS(NT) launch_chunks<NT>(grid, s, y, xbc, proj, ld_proj, dt_bias, a_log, d_skip, state, state_ld, state_rows, cu_seqlens, seq_slots, heads, P, N, groups, from)
  if (N <= 32) return GI_CHUNKS(2);
  if (N <= 64) return GI_CHUNKS(4);
  if (N <= 96) return GI_CHUNKS(6);
  return GI_CHUNKS(8);
#undef GI_CHUNKS
}
