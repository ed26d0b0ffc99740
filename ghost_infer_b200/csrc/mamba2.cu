// The Mamba-2 (state-space duality) mixer's own steps, between its input and output projections.
//
// The input projection's rows are [z: inner | x: inner | B: G*N | C: G*N | dt: heads], inner = heads * P.
//  * conv:  the channels [x | B | C] pass a causal convolution over `taps` tokens per channel, plus bias, then silu.
//           Inputs before a step's first token come from the sequence's state (zeros for a fresh sequence).
//  * scan:  dt <- softplus(dt + dt_bias); per head (head h reads group h / (heads / G) of B and C)
//           S <- exp(-exp(A_log) dt) S + dt B x^T   (S is N x P),   y = S^T C + D x.
//           Everything here is 32-bit; the tokens of a sequence are walked in order, thirty-two at a time through shared
//           memory; a warp owns two or four columns p of S, its lanes the rows n, kept in registers across the step.
//           One token or a thousand, alone or in a batch, take the same arithmetic in the same order: no bit changes.
//           (In 16-bit rows a sequence's stretch of many tokens goes by chunks as matrix products instead: mamba2_chunks.cu.
//           Its own length decides, whatever else is in the step.)
//  * gate + norm: y * silu(z), divided by the root mean square of each of `parts` equal parts, times a weight.
// Per-sequence state: one float row per slot, [S: heads * P * N, a column's N rows side by side (a lane's rows are then
// neighbours in memory: a one-token step, which is all loading and storing of S, moves whole lines) | last taps - 1 conv
// inputs: (taps - 1) * channels];
// slot -1 (a padding row of a fixed-size launch) uses the last row of the matrix.
#include <math.h>

#include "api.h"
#include "common.cuh"

namespace {


__device__ __forceinline__ float silu_f(float v) { return v / (1.0f + expf(-v)); }
__device__ __forceinline__ float softplus_f(float v) { return v > 20.f ? v : log1pf(expf(v)); }

// grid (token tiles of 8, sequences, channel tiles of 256): a thread takes one channel of eight tokens
template <typename T, typename TW>
__global__ void __launch_bounds__(256)
conv_kernel(T* __restrict__ out, const T* __restrict__ proj, long ld_proj, const TW* __restrict__ w,
            const TW* __restrict__ bias, const float* __restrict__ state, long state_ld, int state_rows,
            const int* __restrict__ cu_seqlens, const int* __restrict__ seq_slots, int inner, int channels, int taps,
            int s_floats) {
  gi::pdl_prologue();
  const int b = blockIdx.y;
  const int tok0 = cu_seqlens[b], qlen = cu_seqlens[b + 1] - tok0;
  const int i0 = blockIdx.x * 8;
  if (i0 >= qlen) return;
  const int slot = seq_slots[b];
  const float* cs = state + (size_t)(slot >= 0 ? slot : state_rows - 1) * state_ld + s_floats;
  const int n_here = min(8, qlen - i0);
  const int c = blockIdx.z * 256 + threadIdx.x;
  if (c < channels) {
    const float bc = gi::ldf(bias + c);
    for (int ii = 0; ii < n_here; ++ii) {
      const int i = i0 + ii;
      float acc = bc;
      for (int j = 0; j < taps; ++j) {
        const int src = i - (taps - 1) + j;
        const float v = src >= 0 ? gi::ldf(proj + (size_t)(tok0 + src) * ld_proj + inner + c)
                                 : cs[(size_t)(src + taps - 1) * channels + c];
        acc = fmaf(gi::ldf(w + (size_t)c * taps + j), v, acc);
      }
      gi::stf(out + (size_t)(tok0 + i) * channels + c, silu_f(acc));
    }
  }
}

// The same for 16-bit rows and weights whose channels come in eights: a thread takes eight channels of eight tokens, one 16-byte
// load a row, all rows before anything is computed, where the kernel above loads every input TAPS times two bytes at a time
// and waits for each token's.  The same sums in the same order: the same bits.  Bound by memory and silu's exponential and
// division; 2,048 tokens of 6,144 channels: 38 us, before 79 us.
template <int TAPS>
__global__ void __launch_bounds__(128)
conv8_kernel(__nv_bfloat16* __restrict__ out, const __nv_bfloat16* proj, long ld_proj, const __nv_bfloat16* __restrict__ w,
             const __nv_bfloat16* __restrict__ bias, const float* state, long state_ld, int state_rows, const int* __restrict__ cu_seqlens,
             const int* __restrict__ seq_slots, int inner, int channels, int s_floats) {
  constexpr int TOK = 8;
  gi::pdl_prologue();
  const int b = blockIdx.y;
  const int tok0 = cu_seqlens[b], qlen = cu_seqlens[b + 1] - tok0;
  const int i0 = blockIdx.x * TOK, c = (blockIdx.z * 128 + threadIdx.x) * 8;
  if (i0 >= qlen || c >= channels) return;
  const __nv_bfloat16* in = proj + (size_t)tok0 * ld_proj + inner + c;
  uint4 raw[TOK + TAPS - 1];                                 // inputs i0 - (TAPS - 1) .. i0 + 7
#pragma unroll
  for (int r = 0; r < TOK + TAPS - 1; ++r) {
    const int src = i0 + r - (TAPS - 1);
    raw[r] = src >= 0 && src < qlen ? *reinterpret_cast<const uint4*>(in + (size_t)src * ld_proj) : make_uint4(0, 0, 0, 0);
  }
  float wt[8][TAPS];
#pragma unroll
  for (int k = 0; k < 8; ++k)
#pragma unroll
    for (int j = 0; j < TAPS; ++j) wt[k][j] = gi::ldf(w + (size_t)(c + k) * TAPS + j);
  const uint4 b8 = *reinterpret_cast<const uint4*>(bias + c);
  const int slot = seq_slots[b];
  const float* cs = state + (size_t)(slot >= 0 ? slot : state_rows - 1) * state_ld + s_floats + c;
  auto number = [](const uint4& v, int k) {
    const uint32_t word = k < 2 ? v.x : k < 4 ? v.y : k < 6 ? v.z : v.w;
    return __uint_as_float(k & 1 ? word & 0xffff0000u : word << 16);
  };
#pragma unroll
  for (int t = 0; t < TOK; ++t) {
    if (i0 + t >= qlen) break;
    uint32_t o[4];
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
      float y[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float acc = number(b8, k + e);
#pragma unroll
        for (int j = 0; j < TAPS; ++j) {
          const int src = i0 + t + j - (TAPS - 1);
          const float v = src >= 0 ? number(raw[t + j], k + e) : cs[(size_t)(src + TAPS - 1) * channels + k + e];
          acc = fmaf(wt[k + e][j], v, acc);
        }
        y[e] = silu_f(acc);
      }
      const __nv_bfloat162 two = __floats2bfloat162_rn(y[0], y[1]);
      o[k / 2] = *reinterpret_cast<const uint32_t*>(&two);
    }
    *reinterpret_cast<uint4*>(out + (size_t)(tok0 + i0 + t) * channels + c) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// grid (channel blocks, sequences): the state takes the last taps - 1 inputs of [old state | this step's inputs]
template <typename T>
__global__ void conv_update_kernel(const T* __restrict__ proj, long ld_proj, float* __restrict__ state, long state_ld,
                                   int state_rows, const int* __restrict__ cu_seqlens,
                                   const int* __restrict__ seq_slots, int inner, int channels, int taps, int s_floats) {
  gi::pdl_prologue();
  const int b = blockIdx.y;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= channels) return;
  const int tok0 = cu_seqlens[b], qlen = cu_seqlens[b + 1] - tok0;
  if (qlen <= 0) return;
  const int slot = seq_slots[b];
  float* cs = state + (size_t)(slot >= 0 ? slot : state_rows - 1) * state_ld + s_floats;
  const int keep = taps - 1;
  // place k of the new state is place qlen + k of [old state (keep) | inputs (qlen)]; walking k upwards reads old
  // places qlen + k > k only, which are not yet overwritten
  for (int k = 0; k < keep; ++k) {
    const int at = qlen + k;
    const float v = at < keep ? cs[(size_t)at * channels + c] : gi::ldf(proj + (size_t)(tok0 + at - keep) * ld_proj + inner + c);
    cs[(size_t)k * channels + c] = v;
  }
}

// grid (heads, sequences, column tiles of SC_W * SC_CPW); a warp owns SC_CPW (two or four) columns p of the head's state, its lanes the
// rows (lane l of NPT >= 4 rows owns rows (32 j + l) 4 .. + 3 for j = 0 .. NPT / 4 - 1, so that a warp reads B and C as
// whole 16-byte words side by side; of fewer rows, l NPT .. + NPT - 1), in registers for the whole step.  Tokens go
// through shared memory SC_CH at a time (rows past N padded with zeros, which leave their state at zero); B_t and C_t
// are read once per token for all of a warp's columns.  A token's sum over the rows stays per lane for SC_RB tokens,
// then the 32 (token, column) sums of a warp are added across its lanes in one halving exchange (31 shuffles instead of
// 160), after which lane SC_CPW t + c holds token t, column c.  The order of every sum follows from N alone.
constexpr int SC_W = 4, SC_CH = 32;

// One halving step of the exchange: of 2 * HALF values a lane keeps the half its bit `BIT` of the lane number names and
// adds the other lane's partial sums of the same values.
template <int HALF, int BIT>
__device__ __forceinline__ void halve(float (&v)[32], int lane) {
  const bool upper = (lane & BIT) != 0;
#pragma unroll
  for (int k = 0; k < HALF; ++k) {
    const float send = upper ? v[k] : v[k + HALF];
    const float keep = upper ? v[k + HALF] : v[k];
    v[k] = keep + __shfl_xor_sync(0xffffffffu, send, BIT);
  }
}

template <typename T, typename TW, int NPT, int SC_CPW>
__global__ void __launch_bounds__(SC_W * 32)
scan_kernel(float* __restrict__ y, const T* __restrict__ xbc, const T* __restrict__ proj, long ld_proj,
            const TW* __restrict__ dt_bias, const TW* __restrict__ a_log, const TW* __restrict__ d_skip,
            float* __restrict__ state, long state_ld, int state_rows, const int* __restrict__ cu_seqlens,
            const int* __restrict__ seq_slots, int heads, int P, int N, int groups, int below) {
  constexpr int NP = 32 * NPT;       // rows with padding
  constexpr int SC_COLS = SC_W * SC_CPW, SC_RB = 32 / SC_CPW, SC_CPW_LOG2 = SC_CPW == 2 ? 1 : 2;
  static_assert(SC_CPW == 2 || SC_CPW == 4, "a warp takes 2 or 4 columns");
  extern __shared__ __align__(16) float sm[];
  float* sB = sm;                    // [SC_CH][NP]
  float* sC = sB + SC_CH * NP;       // [SC_CH][NP]
  float* sx = sC + SC_CH * NP;       // [SC_CH][SC_COLS]
  float* sdt = sx + SC_CH * SC_COLS; // [SC_CH]
  float* sdA = sdt + SC_CH;          // [SC_CH]
  gi::pdl_prologue();
  const int h = blockIdx.x, b = blockIdx.y, p0 = blockIdx.z * SC_COLS;
  const int tok0 = cu_seqlens[b], qlen = cu_seqlens[b + 1] - tok0;
  if (qlen <= 0 || qlen >= below) return;
  const int slot = seq_slots[b];
  float* S_row = state + (size_t)(slot >= 0 ? slot : state_rows - 1) * state_ld + (size_t)h * N * P;
  const int g = h / (heads / groups);
  const int inner = heads * P, channels = inner + 2 * groups * N;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int pw = p0 + warp * SC_CPW;             // this warp's first column
  // row of this lane's i-th value
  auto row_of = [&](int i) { return NPT >= 4 ? ((i >> 2) * 32 + lane) * 4 + (i & 3) : lane * NPT + i; };
  float S[SC_CPW][NPT];
#pragma unroll
  for (int c = 0; c < SC_CPW; ++c)
#pragma unroll
    for (int i = 0; i < NPT; ++i) {
      const int n = row_of(i);
      S[c][i] = (pw + c < P && n < N) ? S_row[(size_t)(pw + c) * N + n] : 0.f;
    }
  const float A = -expf(gi::ldf(a_log + h)), D = gi::ldf(d_skip + h), bias = gi::ldf(dt_bias + h);

  for (int c0 = 0; c0 < qlen; c0 += SC_CH) {
    const int nc = min(SC_CH, qlen - c0);
    __syncthreads();
    for (int idx = tid; idx < nc * NP; idx += SC_W * 32) {
      const int t = idx / NP, n = idx % NP;
      float bv = 0.f, cv = 0.f;
      if (n < N) {
        const T* r = xbc + (size_t)(tok0 + c0 + t) * channels + inner + (size_t)g * N + n;
        bv = gi::ldf(r);
        cv = gi::ldf(r + (size_t)groups * N);
      }
      sB[idx] = bv;
      sC[idx] = cv;
    }
    for (int idx = tid; idx < nc * SC_COLS; idx += SC_W * 32) {
      const int t = idx / SC_COLS, j = idx % SC_COLS;
      sx[idx] = (p0 + j < P) ? gi::ldf(xbc + (size_t)(tok0 + c0 + t) * channels + (size_t)h * P + p0 + j) : 0.f;
    }
    for (int t = tid; t < nc; t += SC_W * 32) {
      const float dt = softplus_f(gi::ldf(proj + (size_t)(tok0 + c0 + t) * ld_proj + 2 * inner + 2 * groups * N + h) + bias);
      sdt[t] = dt;
      sdA[t] = expf(A * dt);
    }
    __syncthreads();
    for (int t0 = 0; t0 < nc; t0 += SC_RB) {
      float acc[32];                                  // [SC_RB tokens][SC_CPW columns]
#pragma unroll
      for (int tl = 0; tl < SC_RB; ++tl) {
        const int t = t0 + tl;
#pragma unroll
        for (int c = 0; c < SC_CPW; ++c) acc[tl * SC_CPW + c] = 0.f;
        if (t < nc) {                                 // the same for the whole block
          const float dA = sdA[t], dt = sdt[t];
          float bv[NPT], cv[NPT];
          if (NPT >= 4) {
#pragma unroll
            for (int j = 0; j < NPT / 4; ++j) {
              const float4 b4 = *reinterpret_cast<const float4*>(sB + t * NP + (j * 32 + lane) * 4);
              const float4 c4 = *reinterpret_cast<const float4*>(sC + t * NP + (j * 32 + lane) * 4);
              bv[4 * j] = b4.x; bv[4 * j + 1] = b4.y; bv[4 * j + 2] = b4.z; bv[4 * j + 3] = b4.w;
              cv[4 * j] = c4.x; cv[4 * j + 1] = c4.y; cv[4 * j + 2] = c4.z; cv[4 * j + 3] = c4.w;
            }
          } else {
#pragma unroll
            for (int i = 0; i < NPT; ++i) {
              bv[i] = sB[t * NP + lane * NPT + i];
              cv[i] = sC[t * NP + lane * NPT + i];
            }
          }
#pragma unroll
          for (int i = 0; i < NPT; ++i) bv[i] *= dt;
#pragma unroll
          for (int c = 0; c < SC_CPW; ++c) {
            const float x = sx[t * SC_COLS + warp * SC_CPW + c];
            float a = 0.f;
#pragma unroll
            for (int i = 0; i < NPT; ++i) {
              S[c][i] = fmaf(dA, S[c][i], x * bv[i]);
              a = fmaf(S[c][i], cv[i], a);
            }
            acc[tl * SC_CPW + c] = a;
          }
        }
      }
      halve<16, 16>(acc, lane);
      halve<8, 8>(acc, lane);
      halve<4, 4>(acc, lane);
      halve<2, 2>(acc, lane);
      halve<1, 1>(acc, lane);
      // lane SC_CPW tl + c now holds token t0 + tl, column c
      const int t = t0 + (lane >> SC_CPW_LOG2), c = lane & (SC_CPW - 1);
      if (t < nc && pw + c < P)
        y[(size_t)(tok0 + c0 + t) * inner + (size_t)h * P + pw + c] = acc[0] + D * sx[t * SC_COLS + warp * SC_CPW + c];
    }
  }
#pragma unroll
  for (int c = 0; c < SC_CPW; ++c)
#pragma unroll
    for (int i = 0; i < NPT; ++i) {
      const int n = row_of(i);
      if (pw + c < P && n < N) S_row[(size_t)(pw + c) * N + n] = S[c][i];
    }
}

// grid (tokens, parts)
template <typename TO, typename T, typename TW>
__global__ void __launch_bounds__(256)
gate_norm_kernel(TO* __restrict__ out, const float* __restrict__ y, const T* __restrict__ proj, long ld_proj,
                 const TW* __restrict__ w, int inner, int parts, float eps) {
  __shared__ float scratch[33];
  gi::pdl_prologue();
  const int t = blockIdx.x, part = blockIdx.y, gw = inner / parts, c0 = part * gw;
  float ss = 0.f;
  for (int i = threadIdx.x; i < gw; i += blockDim.x) {
    const float v = y[(size_t)t * inner + c0 + i] * silu_f(gi::ldf(proj + (size_t)t * ld_proj + c0 + i));
    ss = fmaf(v, v, ss);
  }
  ss = gi::block_sum(ss, scratch);
  const float inv = 1.0f / sqrtf(ss / (float)gw + eps);
  for (int i = threadIdx.x; i < gw; i += blockDim.x) {
    const float v = y[(size_t)t * inner + c0 + i] * silu_f(gi::ldf(proj + (size_t)t * ld_proj + c0 + i));
    gi::stf(out + (size_t)t * inner + c0 + i, v * inv * gi::ldf(w + c0 + i));
  }
}

// The same for 16-bit rows and parts of up to 1,024 numbers in fours: TPP threads share a part, 4 VEC numbers each, kept in
// registers, so that y and z are read once, 16 and 8 bytes at a time, and silu is worked out once.  The order of a part's sum
// follows from its width alone, the same for one token and for many.  A block has 256 threads, fewer where the parts are fewer;
// grid (tokens, ceil(parts / parts a block)).  Bound by silu's exponential and division where there are many tokens, else by
// the chain from load to store.  4,096 numbers in 8 parts: one token 2.2 us, 2,048 tokens 14.5 us; the kernel above 2.4 and
// 40 us, a warp per part with 16 numbers a lane 3.6 and 14.4 us, four numbers a thread 1.8 and 18 us.
template <typename TW, int TPP, int VEC>
__global__ void __launch_bounds__(256)
gate_norm_vec_kernel(__nv_bfloat16* __restrict__ out, const float* y, const __nv_bfloat16* proj, long ld_proj, const TW* __restrict__ w,
                     int inner, int parts, float eps) {
  __shared__ float sums[8];
  gi::pdl_prologue();
  const int t = blockIdx.x, part = blockIdx.y * (blockDim.x / TPP) + threadIdx.x / TPP, lane = threadIdx.x % TPP;
  const int gw = inner / parts, c0 = part * gw, width = part < parts ? gw : 0;
  float4 v[VEC], z[VEC];
#pragma unroll
  for (int k = 0; k < VEC; ++k) {
    const int i = 4 * (lane + TPP * k);
    v[k] = z[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < width) {
      v[k] = gi::ld4(y + (size_t)t * inner + c0 + i);
      z[k] = gi::ld4(proj + (size_t)t * ld_proj + c0 + i);
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < VEC; ++k) {
    if (4 * (lane + TPP * k) >= width) continue;
    v[k].x *= silu_f(z[k].x);
    v[k].y *= silu_f(z[k].y);
    v[k].z *= silu_f(z[k].z);
    v[k].w *= silu_f(z[k].w);
    ss = fmaf(v[k].w, v[k].w, fmaf(v[k].z, v[k].z, fmaf(v[k].y, v[k].y, fmaf(v[k].x, v[k].x, ss))));
  }
  ss = gi::warp_sum(ss);
  if (TPP > 32) {
    if ((threadIdx.x & 31) == 0) sums[threadIdx.x >> 5] = ss;
    __syncthreads();
    ss = 0.f;
#pragma unroll
    for (int k = 0; k < TPP / 32; ++k) ss += sums[threadIdx.x / TPP * (TPP / 32) + k];
  }
  const float inv = 1.0f / sqrtf(ss / (float)gw + eps);
#pragma unroll
  for (int k = 0; k < VEC; ++k) {
    const int i = 4 * (lane + TPP * k);
    if (i >= width) continue;
    const float4 g = gi::ld4(w + c0 + i);
    gi::st4(out + (size_t)t * inner + c0 + i, make_float4(v[k].x * inv * g.x, v[k].y * inv * g.y, v[k].z * inv * g.z, v[k].w * inv * g.w));
  }
}

template <typename T, typename TW, int NPT, int CPW>
int launch_scan(dim3 grid, size_t smem, cudaStream_t s, float* y, const T* xbc, const T* proj, long ld_proj, const TW* dt_bias,
                const TW* a_log, const TW* d_skip, float* state, long state_ld, int state_rows, const int* cu, const int* slots,
                int heads, int P, int N, int groups, int below) {
  auto kern = scan_kernel<T, TW, NPT, CPW>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return gi::fail(GI_ERR_CUDA, "mamba2 scan: %s", cudaGetErrorString(e));
  }
  return gi::check(gi::launch(kern, grid, dim3(SC_W * 32), smem, s, y, xbc, proj, ld_proj, dt_bias, a_log, d_skip, state, state_ld,
                              state_rows, cu, slots, heads, P, N, groups, below), "mamba2 scan");
}

}  // namespace

extern "C" int gi_mamba2_conv(void* xbc_out, const void* proj, int dtype, long ld_proj, const void* conv_w,
                              const void* conv_b, int w_dtype, const float* state, long state_ld, int state_rows,
                              const int* cu_seqlens, const int* seq_slots, int n_seqs, int max_q_len, int inner,
                              int channels, int taps, int s_floats, void* stream) {
  if (n_seqs <= 0 || max_q_len <= 0) return GI_OK;
  if (taps < 1 || channels <= 0 || inner < 0) return gi::fail(GI_ERR_ARG, "mamba2 conv: bad sizes");
  if (n_seqs > 65535) return gi::fail(GI_ERR_UNSUPPORTED, "mamba2 conv: more than 65535 sequences in one launch");
  if ((channels + 255) / 256 > 65535) return gi::fail(GI_ERR_UNSUPPORTED, "mamba2 conv: %d channels are more than one launch takes", channels);
  cudaError_t e = cudaSuccess;
  // Eight channels of eight tokens a thread leave too few threads where there are few tokens: the line lies at 64 tiles of
  // eight tokens of 6,144 channels.  Kernel below and this one in us, 6,144 channels: one token 2.1 and 3.9, 64 sequences
  // of one 4.8 and 8.8, 32 tokens 6.1 and 9.0, 256 13.4 and 13.1, 512 22 and 14; 3,328 channels: 512 tokens 13.4 and 13.8, 1,024
  // 24 and 15.  (State rows and `s_floats` in eights are not needed: the state is read number by number.)
  const long tiles = (long)((max_q_len + 7) / 8) * n_seqs;
  if (max_q_len >= 8 && tiles * channels >= 64L * 6144 && dtype == GI_BF16 && w_dtype == GI_BF16 && taps >= 2 && taps <= 4 && channels % 8 == 0 && inner % 8 == 0 && ld_proj % 8 == 0 &&
      (((uintptr_t)xbc_out | (uintptr_t)proj | (uintptr_t)conv_b) & 15) == 0) {
    const dim3 grid((max_q_len + 7) / 8, n_seqs, (channels / 8 + 127) / 128);
#define GI_CONV8(TAPS)                                                                                                              \
  e = gi::launch(conv8_kernel<TAPS>, grid, dim3(128), 0, (cudaStream_t)stream, (__nv_bfloat16*)xbc_out, (const __nv_bfloat16*)proj, \
                 ld_proj, (const __nv_bfloat16*)conv_w, (const __nv_bfloat16*)conv_b, state, state_ld, state_rows, cu_seqlens,      \
                 seq_slots, inner, channels, s_floats)
    if (taps == 2) GI_CONV8(2);
    else if (taps == 3) GI_CONV8(3);
    else GI_CONV8(4);
#undef GI_CONV8
    return gi::check(e, "mamba2 conv");
  }
  dim3 grid((max_q_len + 7) / 8, n_seqs, (channels + 255) / 256);
  GI_DISPATCH_DTYPE(dtype, T, GI_DISPATCH_DTYPE(w_dtype, TW,
      e = gi::launch(conv_kernel<T, TW>, grid, dim3(256), 0, (cudaStream_t)stream, (T*)xbc_out, (const T*)proj, ld_proj,
                     (const TW*)conv_w, (const TW*)conv_b, state, state_ld, state_rows, cu_seqlens, seq_slots, inner, channels,
                     taps, s_floats)));
  return gi::check(e, "mamba2 conv");
}

extern "C" int gi_mamba2_conv_update(const void* proj, int dtype, long ld_proj, float* state, long state_ld, int state_rows,
                                     const int* cu_seqlens, const int* seq_slots, int n_seqs, int inner, int channels,
                                     int taps, int s_floats, void* stream) {
  if (n_seqs <= 0 || taps <= 1) return GI_OK;
  if (n_seqs > 65535) return gi::fail(GI_ERR_UNSUPPORTED, "mamba2 conv: more than 65535 sequences in one launch");
  dim3 grid((channels + 127) / 128, n_seqs);
  cudaError_t e = cudaSuccess;
  GI_DISPATCH_DTYPE(dtype, T,
      e = gi::launch(conv_update_kernel<T>, grid, dim3(128), 0, (cudaStream_t)stream, (const T*)proj, ld_proj, state, state_ld,
                     state_rows, cu_seqlens, seq_slots, inner, channels, taps, s_floats));
  return gi::check(e, "mamba2 conv update");
}

extern "C" int gi_mamba2_scan(float* y, const void* xbc, const void* proj, int dtype, long ld_proj, const void* dt_bias,
                              const void* a_log, const void* d_skip, int w_dtype, float* state, long state_ld,
                              int state_rows, const int* cu_seqlens, const int* seq_slots, int n_seqs, int heads, int P,
                              int N, int groups, void* stream) {
  return gi_mamba2_scan_below(y, xbc, proj, dtype, ld_proj, dt_bias, a_log, d_skip, w_dtype, state, state_ld, state_rows, cu_seqlens,
                              seq_slots, n_seqs, heads, P, N, groups, 2147483647, stream);
}

extern "C" int gi_mamba2_scan_below(float* y, const void* xbc, const void* proj, int dtype, long ld_proj, const void* dt_bias,
                                    const void* a_log, const void* d_skip, int w_dtype, float* state, long state_ld,
                                    int state_rows, const int* cu_seqlens, const int* seq_slots, int n_seqs, int heads, int P,
                                    int N, int groups, int below, void* stream) {
  if (n_seqs <= 0) return GI_OK;
  if (heads <= 0 || P <= 0 || N <= 0 || groups <= 0 || heads % groups != 0)
    return gi::fail(GI_ERR_ARG, "mamba2 scan: %d heads, %d groups, head size %d, state %d", heads, groups, P, N);
  if (n_seqs > 65535 || heads > 65535) return gi::fail(GI_ERR_UNSUPPORTED, "mamba2 scan: more than 65535 sequences or heads");
  if (N > 1024) return gi::fail(GI_ERR_UNSUPPORTED, "mamba2 scan: a state of %d rows is more than a warp's lanes take", N);
  int npt = 1;
  while (32 * npt < N) npt *= 2;
  // four columns a warp where that still gives every SM several blocks (B_t and C_t are then read once for four columns);
  // two where there are few heads and sequences (one prompt), for twice the warps.  Either way a sum's additions are
  // the same ones in the same order, so the choice changes no bit.
  const int cpw = ((long)heads * n_seqs * ((P + SC_W * 4 - 1) / (SC_W * 4)) >= 400) ? 4 : 2;
  const int cols = SC_W * cpw;
  dim3 grid(heads, n_seqs, (P + cols - 1) / cols);
  if (grid.z > 65535) return gi::fail(GI_ERR_UNSUPPORTED, "mamba2 scan: head size %d is more than one launch takes", P);
  const size_t smem = (2 * (size_t)SC_CH * 32 * npt + (size_t)SC_CH * cols + 2 * SC_CH) * sizeof(float);
  cudaStream_t s = (cudaStream_t)stream;
  int rc = GI_OK;
#define GI_SCAN_LAUNCH(NPT, CPW)                                                                                       \
  GI_DISPATCH_DTYPE(dtype, T, GI_DISPATCH_DTYPE(w_dtype, TW,                                                           \
      rc = (launch_scan<T, TW, NPT, CPW>(grid, smem, s, y, (const T*)xbc, (const T*)proj, ld_proj, (const TW*)dt_bias, \
                                         (const TW*)a_log, (const TW*)d_skip, state, state_ld, state_rows, cu_seqlens, \
                                         seq_slots, heads, P, N, groups, below))))
#define GI_SCAN_CASE(NPT)                                                                                              \
  case NPT:                                                                                                            \
    if (cpw == 4) GI_SCAN_LAUNCH(NPT, 4);                                                                              \
    else GI_SCAN_LAUNCH(NPT, 2);                                                                                       \
    break;
  switch (npt) {
    GI_SCAN_CASE(1)
    GI_SCAN_CASE(2)
    GI_SCAN_CASE(4)
    GI_SCAN_CASE(8)
    GI_SCAN_CASE(16)
    GI_SCAN_CASE(32)
  }
#undef GI_SCAN_LAUNCH
#undef GI_SCAN_CASE
  return rc;
}

extern "C" int gi_mamba2_gate_norm(void* out, int out_dtype, const float* y, const void* proj, int dtype, long ld_proj,
                                   const void* w, int w_dtype, int n_tokens, int inner, int parts, float eps,
                                   void* stream) {
  if (n_tokens <= 0) return GI_OK;
  if (parts <= 0 || inner <= 0 || inner % parts != 0)
    return gi::fail(GI_ERR_ARG, "mamba2 norm: %d values do not divide into %d parts", inner, parts);
  if (parts > 65535) return gi::fail(GI_ERR_UNSUPPORTED, "mamba2 norm: more than 65535 parts");
  cudaError_t e = cudaSuccess;
  const int gw = inner / parts;
  if (dtype == GI_BF16 && out_dtype == GI_BF16 && gw % 4 == 0 && gw <= 1024 && ld_proj % 4 == 0 && ((uintptr_t)y & 15) == 0 &&
      (((uintptr_t)proj | (uintptr_t)out) & 7) == 0 && ((uintptr_t)w & (w_dtype == GI_F32 ? 15 : 7)) == 0) {
    const int tpp = gw <= 256 ? 32 : gw <= 512 ? 64 : 128, here = parts < 256 / tpp ? parts : 256 / tpp;
    const dim3 grid(n_tokens, (parts + here - 1) / here);
#define GI_NORM(TPP, VEC)                                                                                                        \
  GI_DISPATCH_DTYPE(w_dtype, TW,                                                                                                 \
      e = gi::launch(gate_norm_vec_kernel<TW, TPP, VEC>, grid, dim3(here * tpp), 0, (cudaStream_t)stream, (__nv_bfloat16*)out, y, \
                     (const __nv_bfloat16*)proj, ld_proj, (const TW*)w, inner, parts, eps))
    if (gw <= 128) GI_NORM(32, 1);
    else if (tpp == 32) GI_NORM(32, 2);
    else if (tpp == 64) GI_NORM(64, 2);
    else GI_NORM(128, 2);
#undef GI_NORM
    return gi::check(e, "mamba2 norm");
  }
  dim3 grid(n_tokens, parts);
  GI_DISPATCH_DTYPE(out_dtype, TO, GI_DISPATCH_DTYPE(dtype, T, GI_DISPATCH_DTYPE(w_dtype, TW,
      e = gi::launch(gate_norm_kernel<TO, T, TW>, grid, dim3(256), 0, (cudaStream_t)stream, (TO*)out, y, (const T*)proj, ld_proj,
                     (const TW*)w, inner, parts, eps))));
  return gi::check(e, "mamba2 norm");
}
