// Linear attention with a matrix of state per head, walked token by token: the recurrence of a gated delta rule and of
// decayed ("lightning") linear attention, one kernel with the differences as parameters.
//
// Per head, with S a K x V matrix of 32-bit numbers kept per sequence, and per token a decay g, a key k (K), a query q (K),
// a value v (V) and, for the delta rule, a write strength beta:
//     S <- g S;   u = delta ? beta (v - S^T k) : v;   S <- S + k u^T;   o = S^T q          (o sees the token's own write)
//  * decay: a constant per head, or exp(-exp(A_log[h]) * softplus(a[t, h] + dt_bias[h])) from a projected row;
//  * beta: sigmoid of a projected row;
//  * q and k may pass silu on the way in, and may be made unit vectors (x / sqrt(sum x^2 + eps)), q times a constant;
//  * query/key head of head h: h / (heads / qk_heads).
// Everything after the loads is 32-bit.  The tokens of a sequence are walked in order whatever the step holds, so a prompt
// cut anywhere, alone or in a batch, gives the same bits.
//
// Work split: grid (heads, sequences, tiles of 32, 16 or 8 columns of S; the widest tile that still gives every SM a
// block is chosen by the launcher).  A column of S (K numbers) belongs to 8 neighbouring lanes; lane l holds rows
// 4 (l + 8 m) .. + 3 for m = 0, 1, ..., so a column's rows are read from the state, and a token's key and query from shared
// memory, sixteen bytes at a time.  The delta rule's S^T k ends with three exchanges among a column's lanes, token by
// token, since the next write depends on it; the read-outs S^T q of eight tokens are exchanged together (seven exchanges
// instead of twenty-four).  The order of every sum follows from K alone: one token or a thousand, alone or in a batch,
// whatever the tile, give the same bits.
// Four more warps of the block prepare the next tokens while these work: together they load a chunk's rows (sixteen bytes a
// thread where the rows allow it, every load before anything is computed from it, so a chunk costs one trip to memory),
// apply silu on the way into shared memory, then the unit norms (one warp per token, in place), the decay and the write
// strength, and write the previous chunk's read-outs to memory in whole lines.  Two buffers in shared memory, one barrier
// of the block per chunk.
// ROT: queries and keys turn on the way in: once a chunk's rows are in shared memory the preparing threads turn the pairs of
// their first numbers by the step's table of angles (loaded with the rows), keys having been scaled when they were stored.
// KEYED: the decay is a number per token and key channel (ready made, float32 rows [heads * K]), S <- diag(g_t) S + k_t v_t^T,
// and goes through shared memory beside queries and keys; queries are multiplied by a constant on the way in.
// State per slot: [heads][V][K] floats (a column's rows side by side) at the start of the slot's row; slot -1 (a padding row
// of a fixed-size launch) uses the last row of the matrix.
#pragma once

#include <math.h>

#include "api.h"
#include "common.cuh"

namespace {

constexpr int LS_LANES = 8;        // lanes of a column
constexpr int LS_PREP = 128;       // threads that prepare tokens and write read-outs
constexpr int LS_TB = 8;           // read-outs exchanged together

__device__ __forceinline__ float ls_silu(float v) { return v / (1.0f + expf(-v)); }
__device__ __forceinline__ float ls_softplus(float v) { return v > 20.f ? v : log1pf(expf(v)); }

// One halving step among a column's 8 lanes: of 2 * HALF values a lane keeps the half its bit `BIT` of the lane number
// names and adds the other lane's partial sums of the same values.
template <int HALF, int BIT, int C>
__device__ __forceinline__ void ls_halve(float (&v)[LS_TB * C], int lane) {
  const bool upper = (lane & BIT) != 0;
#pragma unroll
  for (int k = 0; k < HALF * C; ++k) {
    const float send = upper ? v[k] : v[k + HALF * C];
    const float keep = upper ? v[k + HALF * C] : v[k];
    v[k] = keep + __shfl_xor_sync(0xffffffffu, send, BIT);
  }
}

// two products, two fused multiply-adds in one instruction; each half is rounded as the single one would be
__device__ __forceinline__ uint64_t ls_pair(float a, float b) { return (uint64_t)__float_as_uint(a) | (uint64_t)__float_as_uint(b) << 32; }
__device__ __forceinline__ float ls_lo(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float ls_hi(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ uint64_t ls_mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t ls_fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// Sixteen bytes of a row as 32-bit numbers.
__device__ __forceinline__ void ls_load16(const float* p, float (&out)[4]) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
}
__device__ __forceinline__ void ls_load16(const __nv_bfloat16* p, float (&out)[8]) {
  const uint4 v = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    out[2 * i] = __uint_as_float(w[i] << 16);
    out[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
// All of the block's threads, from wherever they are.
__device__ __forceinline__ void ls_block_barrier() { asm volatile("bar.sync 0;" ::: "memory"); }
// The preparing threads among themselves (barrier 1; the block's own barrier is 0).
__device__ __forceinline__ void ls_prep_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(LS_PREP) : "memory"); }

struct LsArgs {
  float* o;
  const void *q, *k, *v, *a_in, *b_in;
  long ldq, ldk, ldv, lda, ldb;
  const float *decay_c, *dt_bias;
  const float *g_direct, *u_direct;      // per token and head, ready made: the decay itself and what multiplies the written value
  float* state;
  long state_ld;
  int state_rows;
  const int *cu_seqlens, *seq_slots;
  int heads, qk_heads, K, V, in_act, unit_norm, vec_state, vec_in;
  float norm_eps, q_scale;
  const float2* table;                   // ROT: [tokens][half] (cos, sin)
  int half, adjacent;                    // pairs that turn: (i, i + half), or neighbours
  float k_scale;
  const float* g_key;                    // KEYED: [tokens][heads * K] decays
};

// tokens per chunk: two buffers of it stay under 48 KB of shared memory
template <int KR> struct LsChunk { static constexpr int value = KR >= 32 ? 8 : 16; };

// For steps in which some sequence brings several tokens; the others (about one token a sequence) take linear_state_step_kernel.
// Two blocks an SM for the narrower tiles: a grid of about as many blocks as SMs times two then runs as one round.
// C: columns a thread holds.  A token's key and query (and decays) leave shared memory once per thread, sixteen bytes a lane, and
// a walk with one column a thread spends about half its time on that (four wavefronts a load, eight loads a token and warp);
// without the delta rule a thread therefore holds several columns, two numbers an instruction.  B200, us a launch with several and with
// one column: 8 prompts of 150 to 410 tokens, 16 heads of 128 x 128 (tiles of 32, four columns): turned 191 and 306, keyed 175 and 310,
// constant decays 256 and 365, ready-made gates 154 and 224; 8 heads of 256 x 256 (two columns): 416 and 586, 365 and 586, 646 and 670, 277
// and 412.  One prompt of 2,048 tokens in tiles of 8 (two columns): 16 heads of 128 x 128 308 and 367, 263 and 314, 517 and 494, 222 and
// 250; where the grid is no more than a block an SM a warp's own length is all there is, and one column would be faster with
// gates and decays per key (12 heads of 96 x 64: 236 and 256, 213 and 191, 449 and 439, 197 and 158).
template <typename T, int KR, int COLS, int C, bool DELTA, bool ROT, bool KEYED>
__global__ void __launch_bounds__(COLS / C * LS_LANES + LS_PREP, (COLS <= 16 || (C > 1 && KR < 32)) ? 2 : 1)
linear_state_kernel(const LsArgs a) {
  constexpr int Kp = KR * LS_LANES;            // rows with padding
  constexpr int M = KR / 4;                    // groups of four rows per lane; also a preparing lane's share of a row
  constexpr int NC = COLS / C * LS_LANES;      // threads that hold S
  constexpr int CH = LsChunk<KR>::value;
  constexpr int BUF = 2 * CH * Kp + 2 * CH * COLS + 2 * CH + (KEYED ? CH * Kp : 0);     // the decays come last
  constexpr int KEYS_AT = 2 * CH * Kp + 2 * CH * COLS + 2 * CH;
  static_assert(KEYS_AT % 4 == 0, "the decays start on a 16-byte boundary");
  constexpr int VW = 16 / (int)sizeof(T);      // numbers of a row in sixteen bytes
  static_assert(COLS % C == 0 && (C == 1 || !DELTA), "whole threads; the delta rule's column is one thread's");
  static_assert(CH % LS_TB == 0 && CH <= LS_PREP && (CH * Kp) % LS_PREP == 0 && COLS % VW == 0 && CH * COLS / VW <= LS_PREP,
                "whole exchanges; a preparing thread per token, and per group of a chunk's values");
  extern __shared__ __align__(16) float sm[];
  gi::pdl_prologue();
  const int h = blockIdx.x, b = blockIdx.y, j0 = blockIdx.z * COLS;
  const int tok0 = a.cu_seqlens[b], qlen = a.cu_seqlens[b + 1] - tok0;
  if (qlen <= 0) return;
  const int K = a.K, V = a.V;
  const int slot = a.seq_slots[b];
  float* S_row = a.state + (size_t)(slot >= 0 ? slot : a.state_rows - 1) * a.state_ld + (size_t)h * V * K;
  const int hk = h / (a.heads / a.qk_heads);
  const int tid = threadIdx.x;
  const bool prep = tid >= NC;
  const int n_chunks = (qlen + CH - 1) / CH;
  const size_t o_ld = (size_t)a.heads * V;
  const T* qp = (const T*)a.q; const T* kp = (const T*)a.k; const T* vp = (const T*)a.v;
  const T* ap = (const T*)a.a_in; const T* bp = (const T*)a.b_in;
  const float dc = a.decay_c != nullptr ? a.decay_c[h] : 1.0f;
  const float rate = ap != nullptr ? expf(dc) : 0.f, bias = (ap != nullptr && a.dt_bias != nullptr) ? a.dt_bias[h] : 0.f;

  // A chunk's tokens are made ready by the 128 preparing threads together, in two parts.  `fetch`: every thread loads its share
  // of the chunk's rows into registers (sixteen bytes at a time where the rows allow it), a chunk before they are wanted, so
  // that the trip to memory passes while the chunk before is walked.  `put`: silu on the way into shared memory; then the
  // turns, and for unit vectors one warp per token sums the squares of its row in shared memory and scales it in place.
  const bool act = a.in_act != 0;
  constexpr int RG = (CH * Kp / 2 + LS_PREP - 1) / LS_PREP;          // pairs a thread turns, per operand
  constexpr int DG = KEYED ? (CH * Kp / 4 + LS_PREP - 1) / LS_PREP : 1;
  constexpr int QG = (CH * Kp / VW + LS_PREP - 1) / LS_PREP;         // groups of VW numbers a thread moves, per operand
  constexpr int QS = CH * Kp / LS_PREP, VS = (CH * COLS + LS_PREP - 1) / LS_PREP;
  constexpr int QN = QG * VW > QS ? QG * VW : QS, VN = VW > VS ? VW : VS;
  float av, bv, qr[QN], kr[QN], vr[VN];
  float2 cs[ROT ? RG : 1];
  float4 dr[DG];                                                     // per-key decays
  const int pt = tid - NC;
  const int vpr = COLS / VW, vt = pt / vpr, vc = (pt - vt * vpr) * VW;      // at most CH * COLS / VW <= 128 groups
  // A thread's places in a chunk (token << 16 | number) are the same in every chunk: their divisions are made once (they were half
  // of what the preparing warps did, and those are the longer part of a narrow tile's chunk).
  int q_at[QG], d_at[DG], r_at[ROT ? RG : 1];
  auto place = [](int g, int per) { return per > 0 ? g / per << 16 | g % per : 0x7fff0000; };
#pragma unroll
  for (int i = 0; i < QG; ++i) q_at[i] = place(pt + i * LS_PREP, K / VW);
#pragma unroll
  for (int i = 0; i < DG; ++i) d_at[i] = place(pt + i * LS_PREP, (K + 3) / 4);
#pragma unroll
  for (int i = 0; i < (ROT ? RG : 1); ++i) r_at[i] = place(pt + i * LS_PREP, a.half);
  auto fetch = [&](int c) {
    const int n = min(CH, qlen - c * CH);
    const size_t tokc = (size_t)tok0 + (size_t)c * CH;
    // decay and write strength: one thread per token
    av = bv = 0.f;
    if (pt < n) {
      if (ap != nullptr) av = gi::ldf(ap + (tokc + pt) * a.lda + h);
      if (bp != nullptr) bv = gi::ldf(bp + (tokc + pt) * a.ldb + h);
    }
    if (ROT) {
#pragma unroll
      for (int i = 0; i < RG; ++i) {
        cs[i] = (r_at[i] >> 16) < n ? a.table[tokc * a.half + pt + i * LS_PREP] : make_float2(1.f, 0.f);
      }
    }
    if (KEYED) {
      const size_t ldg = (size_t)a.heads * K;
#pragma unroll
      for (int i = 0; i < DG; ++i) {
        const int t = d_at[i] >> 16, r0 = (d_at[i] & 0xffff) * 4;
        dr[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < n) {
          const float* p = a.g_key + (tokc + t) * ldg + (size_t)h * K + r0;
          if (K % 4 == 0) {
            dr[i] = *reinterpret_cast<const float4*>(p);
          } else {
            dr[i].x = p[0];
            if (r0 + 1 < K) dr[i].y = p[1];
            if (r0 + 2 < K) dr[i].z = p[2];
            if (r0 + 3 < K) dr[i].w = p[3];
          }
        }
      }
    }
    if (a.vec_in) {
#pragma unroll
      for (int i = 0; i < QG; ++i) {
        const int t = q_at[i] >> 16, r0 = (q_at[i] & 0xffff) * VW;
        if (t < n) {
          ls_load16(qp + (tokc + t) * a.ldq + (size_t)hk * K + r0, *reinterpret_cast<float (*)[VW]>(qr + i * VW));
          ls_load16(kp + (tokc + t) * a.ldk + (size_t)hk * K + r0, *reinterpret_cast<float (*)[VW]>(kr + i * VW));
        }
      }
      if (vt < n && j0 + vc < V) ls_load16(vp + (tokc + vt) * a.ldv + (size_t)h * V + j0 + vc, *reinterpret_cast<float (*)[VW]>(vr));
    } else {
      const int total = n * K;
#pragma unroll
      for (int i = 0; i < QS; ++i) {
        const int e = pt + i * LS_PREP;
        if (e < total) {
          const int t = e / K, r = e - t * K;
          qr[i] = gi::ldf(qp + (tokc + t) * a.ldq + (size_t)hk * K + r);
          kr[i] = gi::ldf(kp + (tokc + t) * a.ldk + (size_t)hk * K + r);
        }
      }
#pragma unroll
      for (int i = 0; i < VS; ++i) {
        const int e = pt + i * LS_PREP, t = e / COLS, cc = e % COLS;
        vr[i] = (t < n && j0 + cc < V) ? gi::ldf(vp + (tokc + t) * a.ldv + (size_t)h * V + j0 + cc) : 0.f;
      }
    }
  };
  auto put = [&](int c, float* buf) {
    float* sq = buf; float* sk = sq + CH * Kp; float* sv = sk + CH * Kp; float* sg = sv + CH * COLS; float* sb = sg + CH;
    const int n = min(CH, qlen - c * CH);
    const size_t tokc = (size_t)tok0 + (size_t)c * CH;
    const float qs = KEYED ? a.q_scale : 1.0f;
    if (a.vec_in) {
#pragma unroll
      for (int i = 0; i < QG; ++i) {
        const int t = q_at[i] >> 16, r0 = (q_at[i] & 0xffff) * VW;
        if (t < n) {
#pragma unroll
          for (int e = 0; e < VW; e += 4) {
            float4 q4 = make_float4(qr[i * VW + e], qr[i * VW + e + 1], qr[i * VW + e + 2], qr[i * VW + e + 3]);
            float4 k4 = make_float4(kr[i * VW + e], kr[i * VW + e + 1], kr[i * VW + e + 2], kr[i * VW + e + 3]);
            if (act) {
              q4.x = ls_silu(q4.x); q4.y = ls_silu(q4.y); q4.z = ls_silu(q4.z); q4.w = ls_silu(q4.w);
              k4.x = ls_silu(k4.x); k4.y = ls_silu(k4.y); k4.z = ls_silu(k4.z); k4.w = ls_silu(k4.w);
            }
            if (ROT) { k4.x *= a.k_scale; k4.y *= a.k_scale; k4.z *= a.k_scale; k4.w *= a.k_scale; }
            if (KEYED) { q4.x *= qs; q4.y *= qs; q4.z *= qs; q4.w *= qs; }
            *reinterpret_cast<float4*>(sq + t * Kp + r0 + e) = q4;
            *reinterpret_cast<float4*>(sk + t * Kp + r0 + e) = k4;
          }
        }
      }
      if (vt < n && j0 + vc < V) {
#pragma unroll
        for (int e = 0; e < VW; ++e) sv[vt * COLS + vc + e] = act ? ls_silu(vr[e]) : vr[e];     // V is a multiple of VW here
      }
    } else {
      const int total = n * K;
#pragma unroll
      for (int i = 0; i < QS; ++i) {
        const int e = pt + i * LS_PREP;
        if (e < total) {
          const int t = e / K, r = e - t * K;
          sq[t * Kp + r] = (act ? ls_silu(qr[i]) : qr[i]) * qs;
          sk[t * Kp + r] = (act ? ls_silu(kr[i]) : kr[i]) * (ROT ? a.k_scale : 1.0f);
        }
      }
#pragma unroll
      for (int i = 0; i < VS; ++i) {
        const int e = pt + i * LS_PREP;
        if (e < n * COLS) sv[e] = act ? ls_silu(vr[i]) : vr[i];
      }
    }
    if (KEYED) {
      float* sd = buf + KEYS_AT;
#pragma unroll
      for (int i = 0; i < DG; ++i) {
        const int t = d_at[i] >> 16;
        if (t < n) {
          *reinterpret_cast<float4*>(sd + t * Kp + (d_at[i] & 0xffff) * 4) = dr[i];       // numbers past K: zeros, inside the padding
        }
      }
    }
    if (pt < n && !KEYED) {
      sg[pt] = ap != nullptr ? expf(-rate * ls_softplus(av + bias)) : dc;
      sb[pt] = bp != nullptr ? 1.0f / (1.0f + expf(-bv)) : 1.0f;
      if (a.g_direct != nullptr) sg[pt] = a.g_direct[(tokc + pt) * a.heads + h];
      if (a.u_direct != nullptr) sb[pt] = a.u_direct[(tokc + pt) * a.heads + h];
    }
    if (ROT && a.half > 0) {
      ls_prep_barrier();             // the chunk's rows are in shared memory
#pragma unroll
      for (int i = 0; i < RG; ++i) {
        const int t = r_at[i] >> 16, p = r_at[i] & 0xffff;
        if (t < n) {
          const int ia = t * Kp + (a.adjacent ? 2 * p : p), ib = a.adjacent ? ia + 1 : ia + a.half;
          float x, y;
          gi::rotate_pair(sq[ia], sq[ib], cs[i], &x, &y);
          sq[ia] = x; sq[ib] = y;
          gi::rotate_pair(sk[ia], sk[ib], cs[i], &x, &y);
          sk[ia] = x; sk[ib] = y;
        }
      }
    }
    if (a.unit_norm) {
      ls_prep_barrier();             // the chunk's rows are in shared memory
      const int pw = pt >> 5, pl = pt & 31;
      for (int t = pw; t < n; t += LS_PREP / 32) {
        float qv[M], kv[M];
        float s1 = 0.f, s2 = 0.f;
#pragma unroll
        for (int i = 0; i < M; ++i) {
          qv[i] = sq[t * Kp + pl + 32 * i];
          kv[i] = sk[t * Kp + pl + 32 * i];
          s1 = fmaf(qv[i], qv[i], s1);
          s2 = fmaf(kv[i], kv[i], s2);
        }
        s1 = gi::warp_sum(s1);
        s2 = gi::warp_sum(s2);
        const float fq = a.q_scale / sqrtf(s1 + a.norm_eps), fk = 1.0f / sqrtf(s2 + a.norm_eps);
#pragma unroll
        for (int i = 0; i < M; ++i) {
          sq[t * Kp + pl + 32 * i] = qv[i] * fq;
          sk[t * Kp + pl + 32 * i] = kv[i] * fk;
        }
      }
    }
  };
  // a chunk's read-outs from buffer `buf` to memory, by the threads [first, first + count)
  auto write_out = [&](int c, const float* buf, int first, int count) {
    const float* so = buf + 2 * CH * Kp + CH * COLS + 2 * CH;
    const int n = min(CH, qlen - c * CH);
    for (int idx = tid - first; idx < n * COLS; idx += count) {
      const int t = idx / COLS, cc = idx % COLS;
      if (j0 + cc < V) a.o[((size_t)tok0 + (size_t)c * CH + t) * o_ld + (size_t)h * V + j0 + cc] = so[idx];
    }
  };

  const int col = tid / LS_LANES * C, lane = tid % LS_LANES;    // of the threads that hold S: the first of their columns
  uint64_t S[C][KR / 2];                                        // two rows side by side
  if (prep) {
    if (K < Kp) {                  // rows past K stay zero in both buffers: nothing writes them again
      for (int e = tid - NC; e < 2 * CH * Kp; e += LS_PREP) {
        if (e % Kp >= K) { sm[e] = 0.f; sm[BUF + e] = 0.f; }
      }
      if (KEYED) {
        for (int e = tid - NC; e < CH * Kp; e += LS_PREP) {
          if (e % Kp >= K) { sm[KEYS_AT + e] = 0.f; sm[BUF + KEYS_AT + e] = 0.f; }
        }
      }
      ls_prep_barrier();
    }
    fetch(0);
    put(0, sm);
    if (n_chunks > 1) fetch(1);
    // (the two kinds of threads have loops of their own, which keeps either's registers out of the other's)
    for (int c = 0; c < n_chunks; ++c) {
      ls_block_barrier();
      if (c > 0) write_out(c - 1, sm + ((c - 1) & 1) * BUF, NC, LS_PREP);
      if (c + 1 < n_chunks) put(c + 1, sm + ((c + 1) & 1) * BUF);
      if (c + 2 < n_chunks) fetch(c + 2);
    }
  } else {
#pragma unroll
    for (int cc = 0; cc < C; ++cc)
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const int i = 4 * (lane + LS_LANES * m), j = j0 + col + cc;
        float s4[4] = {0.f, 0.f, 0.f, 0.f};
        if (a.vec_state && j < V && i < K) {
          const float4 v = *reinterpret_cast<const float4*>(S_row + (size_t)j * K + i);
          s4[0] = v.x; s4[1] = v.y; s4[2] = v.z; s4[3] = v.w;
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) s4[e] = (j < V && i + e < K) ? S_row[(size_t)j * K + i + e] : 0.f;
        }
        S[cc][2 * m] = ls_pair(s4[0], s4[1]);
        S[cc][2 * m + 1] = ls_pair(s4[2], s4[3]);
      }
  for (int c = 0; c < n_chunks; ++c) {
    ls_block_barrier();          // chunk c is ready in buffer c & 1; the other buffer's tokens and this one's read-outs are used up
    float* buf = sm + (c & 1) * BUF;
    const float* sq = buf; const float* sk = sq + CH * Kp; const float* sv = sk + CH * Kp;
    const float* sg = sv + CH * COLS; const float* sb = sg + CH;
    float* so = buf + 2 * CH * Kp + CH * COLS + 2 * CH;
    const int n = min(CH, qlen - c * CH);
    // one token: the state's columns walk on, `out` takes this lane's share of the read-outs
    auto token = [&](int t, float* out) {
      const float g = KEYED ? 1.0f : sg[t];
      const float* sd = buf + KEYS_AT;
      ulonglong2 kk[M], qq[M];
#pragma unroll
      for (int m = 0; m < M; ++m) {
        kk[m] = *reinterpret_cast<const ulonglong2*>(sk + t * Kp + 4 * (lane + LS_LANES * m));
        qq[m] = *reinterpret_cast<const ulonglong2*>(sq + t * Kp + 4 * (lane + LS_LANES * m));
      }
      float u[C];
#pragma unroll
      for (int cc = 0; cc < C; ++cc) u[cc] = sv[t * COLS + col + cc];
      if (DELTA) {
        uint64_t d01 = 0, d23 = 0;                        // four chains, then a tree: the order is fixed by K alone
#pragma unroll
        for (int m = 0; m < M; ++m) {
          d01 = ls_fma2(S[0][2 * m], kk[m].x, d01);
          d23 = ls_fma2(S[0][2 * m + 1], kk[m].y, d23);
        }
        float d = (ls_lo(d01) + ls_hi(d01)) + (ls_lo(d23) + ls_hi(d23));
        d += __shfl_xor_sync(0xffffffffu, d, 1);
        d += __shfl_xor_sync(0xffffffffu, d, 2);
        d += __shfl_xor_sync(0xffffffffu, d, 4);
        u[0] = sb[t] * (u[0] - g * d);
      } else if (a.u_direct != nullptr) {
#pragma unroll
        for (int cc = 0; cc < C; ++cc) u[cc] *= sb[t];
      }
      uint64_t a01[C], a23[C];
      const uint64_t g2 = ls_pair(g, g);
#pragma unroll
      for (int cc = 0; cc < C; ++cc) a01[cc] = a23[cc] = 0;
#pragma unroll
      for (int m = 0; m < M; ++m) {
        ulonglong2 d2;
        if (KEYED) d2 = *reinterpret_cast<const ulonglong2*>(sd + t * Kp + 4 * (lane + LS_LANES * m));
        else d2.x = d2.y = g2;
#pragma unroll
        for (int cc = 0; cc < C; ++cc) {
          const uint64_t u2 = ls_pair(u[cc], u[cc]);
          uint64_t &lo = S[cc][2 * m], &hi = S[cc][2 * m + 1];
          lo = ls_fma2(kk[m].x, u2, ls_mul2(d2.x, lo));
          hi = ls_fma2(kk[m].y, u2, ls_mul2(d2.y, hi));
          a01[cc] = ls_fma2(lo, qq[m].x, a01[cc]);
          a23[cc] = ls_fma2(hi, qq[m].y, a23[cc]);
        }
      }
#pragma unroll
      for (int cc = 0; cc < C; ++cc) out[cc] = (ls_lo(a01[cc]) + ls_hi(a01[cc])) + (ls_lo(a23[cc]) + ls_hi(a23[cc]));
    };
    for (int t0 = 0; t0 < n; t0 += LS_TB) {
      float acc[LS_TB * C];                              // [token][column]
      if (t0 + LS_TB <= n) {     // eight whole tokens: nothing to test between them, so the next one's loads start early
#pragma unroll
        for (int tl = 0; tl < LS_TB; ++tl) token(t0 + tl, acc + tl * C);
      } else {
#pragma unroll
        for (int tl = 0; tl < LS_TB; ++tl) {
#pragma unroll
          for (int cc = 0; cc < C; ++cc) acc[tl * C + cc] = 0.f;
          if (t0 + tl < n) token(t0 + tl, acc + tl * C);      // the same for the whole block
        }
      }
      ls_halve<4, 4, C>(acc, lane);
      ls_halve<2, 2, C>(acc, lane);
      ls_halve<1, 1, C>(acc, lane);
      // lane l of a column now holds token t0 + l
      if (t0 + lane < n) {
#pragma unroll
        for (int cc = 0; cc < C; ++cc) so[(t0 + lane) * COLS + col + cc] = acc[cc];
      }
    }
  }
  }
  __syncthreads();
  write_out(n_chunks - 1, sm + ((n_chunks - 1) & 1) * BUF, 0, NC + LS_PREP);
  if (!prep) {
#pragma unroll
    for (int cc = 0; cc < C; ++cc)
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const int i = 4 * (lane + LS_LANES * m), j = j0 + col + cc;
        const float s4[4] = {ls_lo(S[cc][2 * m]), ls_hi(S[cc][2 * m]), ls_lo(S[cc][2 * m + 1]), ls_hi(S[cc][2 * m + 1])};
        if (j >= V) continue;
        if (a.vec_state && i < K) {
          *reinterpret_cast<float4*>(S_row + (size_t)j * K + i) = make_float4(s4[0], s4[1], s4[2], s4[3]);
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (i + e < K) S_row[(size_t)j * K + i + e] = s4[e];
        }
      }
  }
}

// The same walk for a step of about one token a sequence: bound by the bytes of S and the trips to memory, of which the kernel
// above would make three one after the other (rows, the barrier behind their preparation, S beside it) with a third of its threads
// waiting.  Here the threads that hold S prepare the token themselves; S is asked for in L2 before the dependency wait (a prefetch
// reads no values) and loaded beside the rows.  64 registers and 256 threads: four blocks an SM, where the other has two (keys of more
// than 128 numbers: 128 registers, two).  Every sum has the other's order, so the bits are the same.  B200, in a step of 8
// sequences (16 heads of 128 x 128, 17 MB of state read and written): 5.3 us of the step's time, 16.7 in the kernel above.  One launch
// of 64 sequences, us, here and there: the same heads turned 31 and 66, constant decays 37 and 72, ready-made gates 35 and 50 (64 with
// several columns a thread), delta rule 35 and 82; 8 heads of 256 x 256 66 and 84, delta rule 74 and 111.
template <typename T, int KR, int COLS, bool DELTA, bool ROT, bool KEYED>
__global__ void __launch_bounds__(COLS * LS_LANES, (KR < 32 ? 1024 : 512) / (COLS * LS_LANES))
linear_state_step_kernel(const __grid_constant__ LsArgs a) {
  constexpr int Kp = KR * LS_LANES, M = KR / 4, NC = COLS * LS_LANES;
  __shared__ __align__(16) float sq[Kp], sk[Kp], sd[KEYED ? Kp : 1], sv[COLS];
  const int h = blockIdx.x, b = blockIdx.y, j0 = blockIdx.z * COLS, tid = threadIdx.x;
  const int K = a.K, V = a.V;
  const int col = tid / LS_LANES, lane = tid % LS_LANES, j = j0 + col;
  gi::pdl_launch_dependents();
  const int slot = gi::ld_step(a.seq_slots + b);
  float* S_col = a.state + (size_t)(slot >= 0 ? slot : a.state_rows - 1) * a.state_ld + ((size_t)h * V + j) * K;
  if (j < V) {
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const int i = 4 * (lane + LS_LANES * m);
      if (i < K) asm volatile("prefetch.global.L2 [%0];" ::"l"(S_col + i));
    }
  }
  gi::pdl_wait();
  const int tok0 = a.cu_seqlens[b], qlen = a.cu_seqlens[b + 1] - tok0;
  if (qlen <= 0) return;
  constexpr bool GATES = !ROT && !KEYED;               // projected or ready made, and unit vectors
  const float dc = KEYED || a.decay_c == nullptr ? 1.0f : a.decay_c[h];
  const float rate = GATES && a.a_in != nullptr ? expf(dc) : 0.f, bias = GATES && a.a_in != nullptr && a.dt_bias != nullptr ? a.dt_bias[h] : 0.f;
  const int hk = h / (a.heads / a.qk_heads);
  float S[KR];
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const int i = 4 * (lane + LS_LANES * m);
    float4 s4 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (j < V && i < K) {
      if (a.vec_state) {
        s4 = *reinterpret_cast<const float4*>(S_col + i);
      } else {
        s4.x = S_col[i];
        if (i + 1 < K) s4.y = S_col[i + 1];
        if (i + 2 < K) s4.z = S_col[i + 2];
        if (i + 3 < K) s4.w = S_col[i + 3];
      }
    }
    S[4 * m] = s4.x; S[4 * m + 1] = s4.y; S[4 * m + 2] = s4.z; S[4 * m + 3] = s4.w;
  }
  const bool act = a.in_act != 0;
  const float qs = KEYED ? a.q_scale : 1.0f, ks = ROT ? a.k_scale : 1.0f;
  for (int t = 0; t < qlen; ++t) {
    const size_t tok = (size_t)tok0 + t;
    const T *q = (const T*)a.q + tok * a.ldq + (size_t)hk * K, *k = (const T*)a.k + tok * a.ldk + (size_t)hk * K;
    if (t > 0) __syncthreads();                        // the token before is used up
    float g = dc, strength = 1.f;
    if (GATES) {
      if (a.a_in != nullptr) g = expf(-rate * ls_softplus(gi::ldf((const T*)a.a_in + tok * a.lda + h) + bias));
      if (DELTA) strength = 1.0f / (1.0f + expf(-gi::ldf((const T*)a.b_in + tok * a.ldb + h)));
      if (a.g_direct != nullptr) g = a.g_direct[tok * a.heads + h];
      if (!DELTA && a.u_direct != nullptr) strength = a.u_direct[tok * a.heads + h];
    }
    // a pair that turns is loaded, turned and stored by one thread; the numbers past the pairs one a thread
    auto query = [&](int i) { const float v = gi::ldf(q + i); return (act ? ls_silu(v) : v) * qs; };
    auto key = [&](int i) { const float v = gi::ldf(k + i); return (act ? ls_silu(v) : v) * ks; };
    const int half = ROT ? a.half : 0;
    for (int i = tid; i < Kp - half; i += NC) {
      if (i < half) {
        const int ia = a.adjacent ? 2 * i : i, ib = a.adjacent ? ia + 1 : ia + half;
        const float2 cs = a.table[tok * half + i];
        const float qa = query(ia), qb = query(ib), ka = key(ia), kb = key(ib);
        gi::rotate_pair(qa, qb, cs, &sq[ia], &sq[ib]);
        gi::rotate_pair(ka, kb, cs, &sk[ia], &sk[ib]);
      } else {
        const int at = i + half;
        sq[at] = at < K ? query(at) : 0.f;
        sk[at] = at < K ? key(at) : 0.f;
      }
    }
    if (KEYED)
      for (int i = tid; i < Kp; i += NC) sd[i] = i < K ? a.g_key[tok * (size_t)a.heads * K + (size_t)h * K + i] : 0.f;
    if (tid < COLS && j0 + tid < V) {
      const float v = gi::ldf((const T*)a.v + tok * a.ldv + (size_t)h * V + j0 + tid);
      sv[tid] = act ? ls_silu(v) : v;
    }
    __syncthreads();
    if (GATES && a.unit_norm) {
      if (tid < 32) {
        float qv[M], kv[M], s1 = 0.f, s2 = 0.f;
#pragma unroll
        for (int i = 0; i < M; ++i) {
          qv[i] = sq[tid + 32 * i];
          kv[i] = sk[tid + 32 * i];
          s1 = fmaf(qv[i], qv[i], s1);
          s2 = fmaf(kv[i], kv[i], s2);
        }
        s1 = gi::warp_sum(s1);
        s2 = gi::warp_sum(s2);
        const float fq = a.q_scale / sqrtf(s1 + a.norm_eps), fk = 1.0f / sqrtf(s2 + a.norm_eps);
#pragma unroll
        for (int i = 0; i < M; ++i) {
          sq[tid + 32 * i] = qv[i] * fq;
          sk[tid + 32 * i] = kv[i] * fk;
        }
      }
      __syncthreads();
    }
    float u = j < V ? sv[col] : 0.f;
    if (DELTA) {
      float d0 = 0.f, d1 = 0.f, d2 = 0.f, d3 = 0.f;
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const float4 k4 = *reinterpret_cast<const float4*>(sk + 4 * (lane + LS_LANES * m));
        d0 = fmaf(S[4 * m], k4.x, d0);
        d1 = fmaf(S[4 * m + 1], k4.y, d1);
        d2 = fmaf(S[4 * m + 2], k4.z, d2);
        d3 = fmaf(S[4 * m + 3], k4.w, d3);
      }
      float d = (d0 + d1) + (d2 + d3);
      d += __shfl_xor_sync(0xffffffffu, d, 1);
      d += __shfl_xor_sync(0xffffffffu, d, 2);
      d += __shfl_xor_sync(0xffffffffu, d, 4);
      u = strength * (u - g * d);
    } else if (GATES && a.u_direct != nullptr) {
      u *= strength;
    }
    float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const int i = 4 * (lane + LS_LANES * m);
      const float4 k4 = *reinterpret_cast<const float4*>(sk + i), q4 = *reinterpret_cast<const float4*>(sq + i);
      if (KEYED) {
        const float4 d4 = *reinterpret_cast<const float4*>(sd + i);
        S[4 * m] *= d4.x; S[4 * m + 1] *= d4.y; S[4 * m + 2] *= d4.z; S[4 * m + 3] *= d4.w;
      }
      S[4 * m] = fmaf(k4.x, u, g * S[4 * m]);
      S[4 * m + 1] = fmaf(k4.y, u, g * S[4 * m + 1]);
      S[4 * m + 2] = fmaf(k4.z, u, g * S[4 * m + 2]);
      S[4 * m + 3] = fmaf(k4.w, u, g * S[4 * m + 3]);
      a0 = fmaf(S[4 * m], q4.x, a0);
      a1 = fmaf(S[4 * m + 1], q4.y, a1);
      a2 = fmaf(S[4 * m + 2], q4.z, a2);
      a3 = fmaf(S[4 * m + 3], q4.w, a3);
    }
    float o = (a0 + a1) + (a2 + a3);
    o += __shfl_xor_sync(0xffffffffu, o, 4);
    o += __shfl_xor_sync(0xffffffffu, o, 2);
    o += __shfl_xor_sync(0xffffffffu, o, 1);
    if (lane == 0 && j < V) a.o[tok * (size_t)a.heads * V + (size_t)h * V + j] = o;
  }
  if (j < V) {
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const int i = 4 * (lane + LS_LANES * m);
      if (a.vec_state && i < K) {
        *reinterpret_cast<float4*>(S_col + i) = make_float4(S[4 * m], S[4 * m + 1], S[4 * m + 2], S[4 * m + 3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (i + e < K) S_col[i + e] = S[4 * m + e];
      }
    }
  }
}

int ls_sm_count() {
  static int n[gi::MAX_DEVICES_SEEN] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= gi::MAX_DEVICES_SEEN) return 148;
  if (n[dev] == 0 && cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) n[dev] = 148;
  return n[dev];
}

template <typename T, int KR, int COLS, bool ROT, bool KEYED>
cudaError_t ls_launch(const LsArgs& a, int n_seqs, bool delta, cudaStream_t stream) {
  constexpr int CH = LsChunk<KR>::value;
  // columns a thread: wide tiles come with many blocks, narrow ones with few, whose warps' own length counts more
  constexpr int C = KR < 32 && COLS >= 32 ? 4 : 2;
  const size_t smem = 2 * (size_t)((KEYED ? 3 : 2) * CH * KR * LS_LANES + 2 * CH * COLS + 2 * CH) * sizeof(float);
  const dim3 grid(a.heads, n_seqs, (a.V + COLS - 1) / COLS), block((delta ? COLS : COLS / C) * LS_LANES + LS_PREP);
  if constexpr (KEYED) {
    auto kern = linear_state_kernel<T, KR, COLS, C, false, false, true>;
    if (smem > 48 * 1024) {
      static bool configured[gi::MAX_DEVICES_SEEN] = {};
      int dev;
      if (gi::unconfigured_here(configured, &dev)) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        if (dev >= 0) configured[dev] = true;
      }
    }
    return gi::launch(kern, grid, block, smem, stream, a);
  } else if constexpr (ROT) {
    return gi::launch(linear_state_kernel<T, KR, COLS, C, false, true, false>, grid, block, smem, stream, a);
  } else {
    return delta ? gi::launch(linear_state_kernel<T, KR, COLS, 1, true, false, false>, grid, block, smem, stream, a)
                 : gi::launch(linear_state_kernel<T, KR, COLS, C, false, false, false>, grid, block, smem, stream, a);
  }
}

template <typename T, int KR, int COLS, bool ROT, bool KEYED>
cudaError_t ls_launch_step(const LsArgs& a, int n_seqs, bool delta, cudaStream_t stream) {
  const dim3 grid(a.heads, n_seqs, (a.V + COLS - 1) / COLS), block(COLS * LS_LANES);
  if constexpr (!ROT && !KEYED) {
    if (delta) return gi::launch(linear_state_step_kernel<T, KR, COLS, true, false, false>, grid, block, 0, stream, a);
  }
  return gi::launch(linear_state_step_kernel<T, KR, COLS, false, ROT, KEYED>, grid, block, 0, stream, a);
}

template <typename T, int KR, bool ROT, bool KEYED>
cudaError_t ls_pick_tile(const LsArgs& a, int n_seqs, bool delta, bool walk, cudaStream_t stream) {
  // the widest tile that still gives every SM a block: with fewer blocks than SMs the token-by-token walk, whose length a
  // block cannot shorten, runs on a part of the device only
  const long per = (long)a.heads * n_seqs, sms = ls_sm_count();
  if (per * ((a.V + 31) / 32) >= sms || a.V <= 8)
    return walk ? ls_launch<T, KR, 32, ROT, KEYED>(a, n_seqs, delta, stream) : ls_launch_step<T, KR, 32, ROT, KEYED>(a, n_seqs, delta, stream);
  if (per * ((a.V + 15) / 16) >= sms)
    return walk ? ls_launch<T, KR, 16, ROT, KEYED>(a, n_seqs, delta, stream) : ls_launch_step<T, KR, 16, ROT, KEYED>(a, n_seqs, delta, stream);
  return walk ? ls_launch<T, KR, 8, ROT, KEYED>(a, n_seqs, delta, stream) : ls_launch_step<T, KR, 8, ROT, KEYED>(a, n_seqs, delta, stream);
}

// What every entry point checks and fills in alike (the pointers and sizes are set).
template <bool ROT, bool KEYED = false>
int ls_run(LsArgs& a, int dtype, int n_seqs, int delta, int n_tokens, void* stream) {
  const int K = a.K, V = a.V;
  if (a.heads <= 0 || a.qk_heads <= 0 || a.heads % a.qk_heads || K <= 0 || V <= 0)
    return gi::fail(GI_ERR_ARG, "linear_state: bad sizes (heads %d, query/key heads %d, keys %d, values %d)", a.heads, a.qk_heads, K, V);
  if (K > 32 * LS_LANES) return gi::fail(GI_ERR_UNSUPPORTED, "linear_state: keys of %d numbers (at most %d)", K, 32 * LS_LANES);
  if (!a.o || !a.q || !a.k || !a.v || (!a.decay_c && !a.g_direct && !a.g_key) || !a.state || !a.cu_seqlens || !a.seq_slots)
    return gi::fail(GI_ERR_ARG, "linear_state: a missing pointer");
  if (a.state_ld < (long)a.heads * K * V)
    return gi::fail(GI_ERR_ARG, "linear_state: state rows of %ld floats, wanted %ld", a.state_ld, (long)a.heads * K * V);
  // sixteen bytes of a column at a time where every column of every slot starts on such a boundary
  a.vec_state = (K % 4 == 0 && a.state_ld % 4 == 0 && ((size_t)a.state & 15) == 0) ? 1 : 0;
  {
    // sixteen bytes of a row at a time where every piece a block reads starts on such a boundary
    const int vw = dtype == GI_BF16 ? 8 : 4;
    const size_t esz = dtype == GI_BF16 ? 2 : 4;
    a.vec_in = (K % vw == 0 && V % vw == 0 && a.ldq % vw == 0 && a.ldk % vw == 0 && a.ldv % vw == 0 &&
                (((uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.v) & 15) == 0 && esz * vw == 16) ? 1 : 0;
  }
  // more tokens than sequences: some sequence brings several, the step is a prompt step (n_tokens 0: not known)
  const bool walk = n_tokens <= 0 || n_tokens > n_seqs;
  cudaError_t e = cudaSuccess;
  GI_DISPATCH_DTYPE(dtype, T, {
    if (K <= 4 * LS_LANES) e = ls_pick_tile<T, 4, ROT, KEYED>(a, n_seqs, delta != 0, walk, (cudaStream_t)stream);
    else if (K <= 8 * LS_LANES) e = ls_pick_tile<T, 8, ROT, KEYED>(a, n_seqs, delta != 0, walk, (cudaStream_t)stream);
    else if (K <= 16 * LS_LANES) e = ls_pick_tile<T, 16, ROT, KEYED>(a, n_seqs, delta != 0, walk, (cudaStream_t)stream);
    else e = ls_pick_tile<T, 32, ROT, KEYED>(a, n_seqs, delta != 0, walk, (cudaStream_t)stream);
  });
  return gi::check(e, "linear_state");
}

}  // namespace
