// Row-local integer stages between the linears of exact mode: RMSNorm + quantisation, RoPE + per-head
// quantisation + KV limb store, attention output division, SiLU * up + quantisation.
// One CTA per row (or per token and KV head); row maxima and sums are exact integer reductions (the warp's
// reduce instructions, then shared memory), so the thread count cannot change a bit. Bound violations set the sticky flag word.
//
// Same integers as src/bitexact/exact/segs.py:49-128 and the fused kernels of
// src/bitexact/vllm_plugin/exact_fuse.py:136-334.
#pragma once

#include <cooperative_groups.h>

#include "bx_ptx.cuh"
#include "bx_rules.cuh"
#include "stage_math.cuh"

namespace bx {

// ---- exact division helpers ----
// floor(x / d) and remainder for 0 <= x < 2^63 from inv = floor((2^64 - 1) / d): one high multiply, one fix-up.
__device__ __forceinline__ u64 uqr_recip(u64 x, u64 d, u64 inv, u64& rem) {
  u64 q = __umul64hi(x, inv);
  u64 r = x - q * d;
  if (r >= d) { q += 1; r -= d; }
  rem = r;
  return q;
}

// div_round (exact/ops.py:37-57) with the row-constant divisor r given with its reciprocal.
template <int NIT>
__device__ __forceinline__ i64 div_round_recip(i64 a, i64 p, u64 r, u64 inv) {
  u64 rem;
  const u64 mag = (u64)iabs(a);
  const u64 q0 = uqr_recip(mag, r, inv, rem);
  i64 Q, R;
  if (a < 0) { Q = -(i64)q0 - (rem != 0 ? 1 : 0); R = rem != 0 ? (i64)(r - rem) : 0; }
  else { Q = (i64)q0; R = (i64)rem; }
  i64 left = imax(p, 0);
#pragma unroll
  for (int i = 0; i < NIT; ++i) {
    if (left > 0) {                                    // a step with nothing left to shift in would change nothing
      const int c = (int)imin(left, 28);
      const u64 q1 = uqr_recip((u64)R << c, r, inv, rem);
      Q = shl(Q, c) + (i64)q1;
      R = (i64)rem;
      left -= c;
    }
  }
  if (p >= 0) return Q + (2 * R >= (i64)r ? 1 : 0);
  const int k = (int)iclamp(-p, 1, 62);
  return (Q + (1ll << (k - 1))) >> k;
}

// The same for a single element (out of line: the stages come here once in 10^6 elements).
template <int NIT>
__device__ __noinline__ i64 long_division(i64 a, i64 p, u64 r) {
  return div_round_recip<NIT>(a, p, r, ~0ull / r);
}

// floor(num / den) for 0 <= num < 2^62 and 2^31 <= den <= 2^33 (quotient below 2^31): float64 estimate, exact integer
// fix-up. The conversion of num loses at most 2^8, i.e. 2^-23 of a quotient unit, and the division rounds by less
// than 2^-22, so the truncated estimate is the floor or one off; one correction each way settles it.
__device__ __forceinline__ i64 fdiv_pos_est(i64 num, i64 den) {
  i64 q = (i64)((double)num / (double)den);
  i64 r = num - q * den;
  if (r < 0) { q -= 1; r += den; }
  if (r >= den) { q += 1; }
  return q;
}

// ---- block reductions (exact, order free) ----
// High words first, then the low words of the lanes that hold the largest (two 32-bit warp reductions).
__device__ __forceinline__ i64 warp_max(i64 v) {
  const int hi = __reduce_max_sync(0xffffffffu, (int)(v >> 32));
  const uint32_t lo = __reduce_max_sync(0xffffffffu, (int)(v >> 32) == hi ? (uint32_t)v : 0u);
  return (i64)(((u64)(uint32_t)hi << 32) | lo);
}
__device__ __forceinline__ i64 warp_sum(i64 v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// All threads of the CTA get the result. `buf` holds 33 i64 in shared memory.
template <bool IS_MAX>
__device__ __forceinline__ i64 block_reduce(i64 v, i64* buf) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = IS_MAX ? warp_max(v) : warp_sum(v);
  __syncthreads();                       // buf may still be read from a previous reduction
  if (lane == 0) buf[warp] = v;
  __syncthreads();
  if (warp == 0) {
    i64 t = lane < nw ? buf[lane] : (IS_MAX ? (i64)0x8000000000000000ull : 0);
    t = IS_MAX ? warp_max(t) : warp_sum(t);
    if (lane == 0) buf[32] = t;
  }
  __syncthreads();
  return buf[32];
}

// Bits of a row maximum. The row exponents and the power-of-two bounds need only the bit length of max |v|, and the OR of the
// magnitudes has the same: two logic operations per value and two warp reductions of 32 bits, where a 64-bit maximum
// costs eight issue slots per value and a shuffle tree (measured; 64-bit compares are the dearest common operation).
// (-2^63, whose magnitude does not exist, counts as 0, as it does for a maximum.)
__device__ __forceinline__ i64 mag_or(i64 acc, i64 v) { return acc | (iabs(v) & 0x7fffffffffffffffll); }
__device__ __forceinline__ i64 warp_or(i64 v) {
  const uint32_t lo = __reduce_or_sync(0xffffffffu, (uint32_t)v), hi = __reduce_or_sync(0xffffffffu, (uint32_t)((u64)v >> 32));
  return (i64)(((u64)hi << 32) | lo);
}
// Sum of 0 <= v < 2^57 over the warp, 26 bits at a time.
__device__ __forceinline__ i64 warp_sum_pos(i64 v) {
  const u64 a = __reduce_add_sync(0xffffffffu, (uint32_t)v & 0x3ffffffu), b = __reduce_add_sync(0xffffffffu, (uint32_t)(v >> 26) & 0x3ffffffu);
  const u64 c = __reduce_add_sync(0xffffffffu, (uint32_t)(v >> 52));
  return (i64)(a + (b << 26) + (c << 52));
}
// Over the CTA, for all threads, with one barrier: every warp folds the warps' results itself. `buf` holds 32 i64 in shared
// memory that no other reduction of the kernel uses (between two calls with the same buffer stands another barrier).
__device__ __forceinline__ i64 block_or(i64 v, i64* buf) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_or(v);
  if (lane == 0) buf[warp] = v;
  __syncthreads();
  return warp_or(lane < nw ? buf[lane] : 0);
}
__device__ __forceinline__ i64 block_max(i64 v, i64* buf) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  if (lane == 0) buf[warp] = v;
  __syncthreads();
  return warp_max(lane < nw ? buf[lane] : (i64)0x8000000000000000ull);
}
__device__ __forceinline__ i64 block_sum_pos(i64 v, i64* buf) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum_pos(v);
  if (lane == 0) buf[warp] = v;
  __syncthreads();
  return warp_sum(lane < nw ? buf[lane] : 0);
}

// 2^-t at out_bits for t >= 0 at 26 fractional bits: table 2^-f at 2^60 (step 2^-14) + linear interpolation
// (exact/ops.py:108-116).
template <bool SMEM_TABLE = false>
__device__ __forceinline__ i64 exp2neg_lut(i64 t, const i64* __restrict__ lut, int out_bits) {
  const i64 n = t >> FT2;
  const i64 f = t & ((1ll << FT2) - 1);
  const int idx = (int)(f >> (FT2 - EXP2_BITS));
  const i64 rr = f & ((1ll << (FT2 - EXP2_BITS)) - 1);
  const i64 a = SMEM_TABLE ? lut[idx] : __ldg(lut + idx);
  const i64 b = SMEM_TABLE ? lut[idx + 1] : __ldg(lut + idx + 1);
  const i64 v = a + rshs<FT2 - EXP2_BITS>((b - a) * rr);
  return rshc(v, (i64)(EXP2_ONE - out_bits) + n);
}

// Activation row -> limb planes a8[l][row][col] (optional), one element.
__device__ __forceinline__ void store_limb_planes(int8_t* a8, int64_t plane, int64_t off, int q) {
  int r = q;
  a8[off] = (int8_t)split8(r);
  a8[plane + off] = (int8_t)split8(r);
  a8[2 * plane + off] = (int8_t)split8(r);
}

// ---- RMSNorm + quant (segs.add_y + norm_q; exact_fuse._norm_kernel) ----
// MODE 0: x = emb[ids[row]] (int32 table); 1: x = xin + yin; 2: x = xin.
constexpr int NORM_THREADS = 256;
constexpr int NORM_EPT = 16;     // D <= 4096
constexpr int NORM_MAX_D = NORM_THREADS * NORM_EPT;

// One row by the integer rule, for rows whose values (or gamma) leave the ranges of the double-precision form below.
template <int MODE, int NT>
__device__ __noinline__ void norm_row(const void* xin, const i64* yin, const i64* ids, const i64* gm, const i64* ge, const i64* xo,
                                      int32_t* q, i64* sh_out, int8_t* a8, int64_t row, int M, int D, int lg, i64 (*red)[32]) {
  constexpr int EPT = NORM_MAX_D / NT;
  i64 x[EPT];
  i64 ax = 0;
#pragma unroll
  for (int k = 0; k < EPT; ++k) {
    const int c = 4 * threadIdx.x + (k / 4) * 4 * NT + k % 4;        // the columns this thread has stored to xo
    x[k] = 0;
    if (c < D) {
      if (xo) x[k] = xo[row * D + c];
      else if (MODE == 0) x[k] = (i64) reinterpret_cast<const int32_t*>(xin)[ids[row] * D + c];
      else if (MODE == 1) x[k] = reinterpret_cast<const i64*>(xin)[row * D + c] + yin[row * D + c];
      else x[k] = reinterpret_cast<const i64*>(xin)[row * D + c];
      ax = mag_or(ax, x[k]);
    }
  }
  ax = block_or(ax, red[0]);                 // the bits of the maximum: what follows reads no more of it
  // rms (exact/ops.py:92-105)
  const i64 amax = imax(ax, 1);
  const i64 shx = imax((i64)bitlen(amax) - 25, -6);
  i64 S = 0;
#pragma unroll
  for (int k = 0; k < EPT; ++k) {
    const i64 xs = rshc(x[k], shx);
    S += xs * xs;
  }
  S = block_sum_pos(S, red[1]);              // at most EPT squares of 2^25 per thread
  const i64 T = S + rshc(EPS60 * D, 60 - 2 * (FR - shx));
  const i64 m = (62 + lg - (i64)bitlen(T)) >> 1;
  const i64 s = 2 * m - lg;
  const i64 V = s >= 0 ? (s >= 64 ? 0 : shl(T, (int)s)) : (T >> (int)imin(-s, 63));
  const i64 r = isqrt(V);
  const i64 er = shx - FR - m;
  const u64 inv = ~0ull / (u64)r;
  // ndiv + quant(., -FN)
  i64 pmax = 0;
#pragma unroll
  for (int k = 0; k < EPT; ++k) {
    const int c = 4 * threadIdx.x + (k / 4) * 4 * NT + k % 4;
    if (c < D) {
      x[k] = div_round_recip<3>(x[k] * gm[c], ge[c] - FR - er + FN, (u64)r, inv);
      pmax = mag_or(pmax, x[k]);
    }
  }
  pmax = block_or(pmax, red[2]);
  const i64 sh = quant_sh(pmax, -FN);
  if (threadIdx.x == 0) sh_out[row] = sh;
  const int64_t plane = (int64_t)M * D;
#pragma unroll
  for (int k = 0; k < EPT; ++k) {
    const int c = 4 * threadIdx.x + (k / 4) * 4 * NT + k % 4;
    if (c < D) {
      const int qv = (int)rshc(x[k], sh + FN);
      q[row * D + c] = qv;
      if (a8) store_limb_planes(a8, plane, row * D + c, qv);
    }
  }
  __syncthreads();                           // the buffers are free for the next row
}

// NT threads walk the rows blockIdx.x + k gridDim.x, four consecutive columns and Q such groups per thread; gamma stays in
// registers. Per element: 31 bytes moved and about 60 issue slots (before: 200, in 64-bit integers), so with a few thousand
// rows the memory bounds it; a decode batch is one chain of loads and three reductions. 3750 rows of 2048: 117 -> 54 us
// (4.4 TB/s), 256 rows 11.0 -> 6.3 us, one row 5.8 -> 3.4 us.
//
// floor(x gm 2^p / r + 1/2) in double precision: where |x| < 2^40 (more sets the flag) and x gm has at most 53 bits; 2^p / r is
// held as two doubles (the second from the exact remainder of the first), so the quotient is known to 2^-90 of itself, and
// for |y| < 2^50 its distance to a rounding boundary to 2^-40. An element nearer to one than 2^-20 (one in 10^6) takes the long
// division. p >= 0 and p < 0 are one formula: floor((floor(a / r) + 2^(k-1)) / 2^k) = floor(a / (r 2^k) + 1/2).
template <int MODE, int NT, int Q>
__global__ void __launch_bounds__(NT, 1024 / NT)
norm_kernel(const void* __restrict__ xin, const i64* __restrict__ yin, const i64* __restrict__ ids,
            const i64* __restrict__ gm, const i64* __restrict__ ge, i64* xo, int32_t* __restrict__ q,
            i64* __restrict__ sh_out, int8_t* __restrict__ a8, int32_t* flag, int M, int D, int lg, int do_norm, bool wide) {
  __shared__ i64 red[3][32];
  uint32_t* red32 = reinterpret_cast<uint32_t*>(red);
  // A decode step's weights have pushed gamma out of L2: asked for (32 bytes a thread) while the previous kernel ends.
  // Read behind the wait without this, a step of 19 sequences took 2051 us in place of 2024.
  if (do_norm)
    for (int c = 4 * threadIdx.x; c < D; c += 4 * NT) {
      prefetch_l2(gm + c);
      prefetch_l2(ge + c);
    }
  wait_previous();
  launch_next();
  double G[Q][4];                            // gm 2^ge
  uint32_t gtop = 0;
#pragma unroll
  for (int k = 0; k < Q; ++k) {
    const int c = 4 * (threadIdx.x + k * NT);
    i64 m4[4] = {0, 0, 0, 0}, e4[4] = {0, 0, 0, 0};
    if (do_norm && c < D) {
      load4(gm + c, wide, m4);
      load4(ge + c, wide, e4);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const double v = to_f64(m4[j]);
      const bool fits = in_f64(m4[j]) && e4[j] >= -40 && e4[j] <= 8;
      gtop = max(gtop, fits ? (uint32_t)__double2hiint(v) & 0x7fffffffu : 0x7fefffffu);
      G[k][j] = fits ? v * pow2_f64((int)e4[j]) : 0.0;
    }
  }
  const int gbits = do_norm ? f64_bits(group_max<NT>(gtop, red32 + 128, 0)) : 0;
  const int64_t plane = (int64_t)M * D;
  for (int64_t row = blockIdx.x; row < M; row += gridDim.x) {
    double x[Q][4];
    uint32_t top = 0;
#pragma unroll
    for (int k = 0; k < Q; ++k) {
      const int c = 4 * (threadIdx.x + k * NT);
      i64 v[4] = {0, 0, 0, 0};
      if (c < D) {
        if (MODE == 0) {
          const int32_t* e = reinterpret_cast<const int32_t*>(xin) + ids[row] * D + c;
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] = e[j];
        } else {
          load4(reinterpret_cast<const i64*>(xin) + row * D + c, wide, v);
        }
        if (MODE == 1) {
          i64 y[4];
          load4(yin + row * D + c, wide, y);
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] += y[j];
        }
        if (xo) store4(xo + row * D + c, wide, v);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        x[k][j] = to_f64(v[j]);
        top = max(top, in_f64(v[j]) ? (uint32_t)__double2hiint(x[k][j]) & 0x7fffffffu : 0x7fefffffu);
      }
    }
    top = group_max<NT>(top, red32, 0);
    const int bits = f64_bits(top);
    const bool general = bits > 40 || bits + gbits > 53;
    if (general) {
      i64 ax = 0;
#pragma unroll
      for (int k = 0; k < Q; ++k) {
        const int c = 4 * (threadIdx.x + k * NT);
        if (c < D) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            i64 v;
            if (xo) v = xo[row * D + c + j];
            else if (MODE == 0) v = (i64) reinterpret_cast<const int32_t*>(xin)[ids[row] * D + c + j];
            else if (MODE == 1) v = reinterpret_cast<const i64*>(xin)[row * D + c + j] + yin[row * D + c + j];
            else v = reinterpret_cast<const i64*>(xin)[row * D + c + j];
            ax = mag_or(ax, v);
          }
        }
      }
      ax = group_or<NT>(ax, red[1], 0);
      if (threadIdx.x == 0 && ax >= (1ll << 40)) *flag = 1;
      __syncthreads();
      if (do_norm) norm_row<MODE, NT>(xin, yin, ids, gm, ge, xo, q, sh_out, a8, row, M, D, lg, red);
      continue;
    }
    if (!do_norm) {
      __syncthreads();
      continue;
    }
    // rms (exact/ops.py:92-105)
    const int shx = max((bits ? bits : 1) - 25, -6);
    double S = 0.0;                          // at most 8 squares of 2^25 per thread: exact
    {
      const double half = shx > 0 ? pow2_f64(shx - 1) : 0.0, scale = pow2_f64(-shx);
#pragma unroll
      for (int k = 0; k < Q; ++k)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const double xs = __fma_rd(x[k][j] + half, scale, F2I) - F2I;
          S = fma(xs, xs, S);
        }
    }
    const i64 T = group_sum<NT>((i64)S, red[1], 0) + rshc(EPS60 * D, 60 - 2 * (FR - shx));
    const i64 m = (62 + lg - (i64)bitlen(T)) >> 1;
    const i64 s = 2 * m - lg;
    const i64 V = s >= 0 ? (s >= 64 ? 0 : shl(T, (int)s)) : (T >> (int)imin(-s, 63));
    const i64 r = isqrt(V);
    const i64 er = shx - FR - m;
    const double rd = (double)r, inv = 1.0 / rd, low = fma(-inv, rd, 1.0) * inv;
    const int p0 = (int)(FN - FR - er);      // the exponent of the quotient, without gamma's
    const double scale = pow2_f64(p0), c_hi = inv * scale, c_lo = low * scale;
    // ndiv + quant(., -FN)
    const bool far = p0 < -22 || p0 > 76;    // p = p0 + ge: outside -62 .. 84 the long division has rules of its own
    top = 0;
#pragma unroll
    for (int k = 0; k < Q; ++k)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const double a = x[k][j] * G[k][j];
        const double h = a * c_hi, l = fma(a, c_lo, fma(a, c_hi, -h));
        const double n = __dadd_rd(h, F2I) - F2I;
        const double d = ((h - n) + l) - 0.5;                          // distance to the boundary between n and n + 1
        const int dh = __double2hiint(d);
        const uint32_t size = (uint32_t)__double2hiint(h) & 0x7fffffffu;
        double y = n + __hiloint2double(~(dh >> 31) & 0x3ff00000, 0);
        // within 2^-20 of it, or |y| from 2^49 on: the long division
        if ((uint32_t)(dh & 0x7fffffff) < (1003u << 20) || size >= (1072u << 20) || far) {
          const int c = 4 * (threadIdx.x + k * NT) + j;
          if (c < D) {
            const i64 xi = f64_to_int(x[k][j] + F2I);
            const i64 v = long_division<3>(xi * gm[c], ge[c] - FR - er + FN, (u64)r);
            if (!in_f64(v)) top = 0x7fefffffu;
            y = to_f64(v);
          }
        }
        x[k][j] = y;
        top = max(top, (uint32_t)__double2hiint(y) & 0x7fffffffu);
      }
    top = group_max<NT>(top, red32 + 128, 0);
    if (top >= 0x7fe00000u) {                // a quotient of 2^51 or more
      norm_row<MODE, NT>(xin, yin, ids, gm, ge, xo, q, sh_out, a8, row, M, D, lg, red);
      continue;
    }
    const i64 sh = top ? (i64)f64_bits(top) - FN - QB : NEG_BIG;       // quant_sh
    if (threadIdx.x == 0) sh_out[row] = sh;
    const int c = top ? f64_bits(top) - QB : 0;
    const double half = c > 0 ? pow2_f64(c - 1) : 0.0, down = pow2_f64(-c);
#pragma unroll
    for (int k = 0; k < Q; ++k) {
      const int col = 4 * (threadIdx.x + k * NT);
      int v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = __double2loint(__fma_rd(x[k][j] + half, down, F2I));
      if (col < D) store_q4(q, a8, plane, row * D + col, wide, v);
    }
  }
}

// ---- RoPE + per-head q quant + K / V limb store (segs.rope_y + q_group + tri_paged.store; _qkv_kernel) ----
// One CTA per (token, KV head); G query heads, head_dim HD (HD / 2 threads, each owning one rotation pair).
struct QkvParams {
  const i64* y;        // [N, (H + 2 HKV) HD] at FR
  const i64* cos;      // [max_pos, HD / 2] at 30 bits
  const i64* sin;
  const i64* pos;      // [N]
  const i64* slot;     // [N] flat cache slot, < 0: not stored (may be null with cache null)
  int8_t* cache;       // limb planes [nb, HKV, bs, 8 HD] or null
  int64_t sc_nb, sc_h, sc_bs;
  int bs;
  int32_t* q;          // [N, H HD]
  i64* sh;             // [N, H]
  int32_t* flag;
  int H, HKV, HD;
};

__global__ void qkv_kernel(const QkvParams p) {
  __shared__ i64 red[2][32];
  int turn = 0;
  const int64_t row = blockIdx.x;
  const int h = blockIdx.y;
  const int HH = p.HD / 2;
  const int G = p.H / p.HKV;
  const int dd = threadIdx.x;              // 0 .. HH-1
  const int64_t NT = (int64_t)(p.H + 2 * p.HKV) * p.HD;
  wait_previous();
  launch_next();
  const i64 pos = p.pos[row];
  const i64* yr = p.y + row * NT;
  // Everything the thread reads is requested before the first use: the row's q / k / v values and the slot are in
  // flight together with the position and the rotation pair that depends on it (the kernel is a latency chain).
  constexpr int GPRE = 8;
  i64 xa[GPRE], xb[GPRE];
#pragma unroll
  for (int g = 0; g < GPRE; ++g) {
    xa[g] = 0;
    xb[g] = 0;
    if (g < G) {
      const int64_t qc = (int64_t)(h * G + g) * p.HD + dd;
      xa[g] = yr[qc];
      xb[g] = yr[qc + HH];
    }
  }
  const int64_t kc = (int64_t)p.H * p.HD + (int64_t)h * p.HD + dd;
  const int64_t vc = (int64_t)(p.H + p.HKV) * p.HD + (int64_t)h * p.HD + dd;
  const i64 k1 = yr[kc], k2 = yr[kc + HH];
  const i64 v1r = yr[vc], v2r = yr[vc + HH];
  const i64 slot = p.cache ? p.slot[row] : -1;
  const i64 cs = p.cos[pos * HH + dd];
  const i64 sn = p.sin[pos * HH + dd];
  i64 big = 0;
  i64 shmax = NEG_BIG;
  auto head = [&](int g, i64 x1, i64 x2) {
    const int64_t qc = (int64_t)(h * G + g) * p.HD + dd;
    big = mag_or(mag_or(big, x1), x2);
    const i64 p1 = x1 * cs - x2 * sn;
    const i64 p2 = x2 * cs + x1 * sn;
    const i64 amax = block_or(mag_or(mag_or(0, p1), p2), red[turn ^= 1]);
    const i64 sh = quant_sh(amax, -(FR + FT));
    shmax = imax(shmax, sh);
    int32_t* qo = p.q + row * ((int64_t)p.H * p.HD) + qc;
    qo[0] = (int32_t)rshc(p1, sh + (FR + FT));
    qo[HH] = (int32_t)rshc(p2, sh + (FR + FT));
    if (threadIdx.x == 0) p.sh[row * p.H + h * G + g] = sh;
  };
#pragma unroll
  for (int g = 0; g < GPRE; ++g)
    if (g < G) head(g, xa[g], xb[g]);                   // G is the same for every thread of the grid
  for (int g = GPRE; g < G; ++g) {
    const int64_t qc = (int64_t)(h * G + g) * p.HD + dd;
    head(g, yr[qc], yr[qc + HH]);
  }
  big = mag_or(mag_or(mag_or(mag_or(big, k1), k2), v1r), v2r);
  const i64 k1o = rshs<FR + FT - FK>(k1 * cs - k2 * sn);
  const i64 k2o = rshs<FR + FT - FK>(k2 * cs + k1 * sn);
  const i64 v1 = rshs<FR - FV>(v1r);
  const i64 v2 = rshs<FR - FV>(v2r);
  const i64 kvbig = imax(imax(iabs(k1o), iabs(k2o)), imax(iabs(v1), iabs(v2)));
  const int over = __syncthreads_or(big >= (1ll << 31) || kvbig > LIM3);
  if (threadIdx.x == 0 && (over || shmax > FK + 3 - FZ)) *p.flag = 1;
  if (p.cache) {
    if (slot >= 0) {
      int8_t* base = p.cache + (slot / p.bs) * p.sc_nb + (int64_t)h * p.sc_h + (slot % p.bs) * p.sc_bs;
      int kk1 = (int)k1o, kk2 = (int)k2o, vv1 = (int)v1, vv2 = (int)v2;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        base[i * p.HD + dd] = (int8_t)split8(kk1);
        base[i * p.HD + HH + dd] = (int8_t)split8(kk2);
        base[(3 + i) * p.HD + dd] = (int8_t)split8(vv1);
        base[(3 + i) * p.HD + HH + dd] = (int8_t)split8(vv2);
      }
    }
  }
}

// K / V int64 [N, HKV, HD] -> limb planes at flat slots (tri_paged.store, src/bitexact/vllm_plugin/tri_paged.py:311-335).
__global__ void kv_store_kernel(int8_t* cache, const i64* __restrict__ slot, const i64* __restrict__ k,
                                const i64* __restrict__ v, int64_t skz, int64_t skh, int64_t svz, int64_t svh,
                                int64_t sc_nb, int64_t sc_h, int64_t sc_bs, int bs, int HD) {
  const int64_t n = blockIdx.x;
  const int h = blockIdx.y;
  const i64 s = slot[n];
  if (s < 0) return;
  int8_t* base = cache + (s / bs) * sc_nb + (int64_t)h * sc_h + (s % bs) * sc_bs;
  for (int dd = threadIdx.x; dd < HD; dd += blockDim.x) {
    int kk = (int)k[n * skz + h * skh + dd], vv = (int)v[n * svz + h * svh + dd];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      base[i * HD + dd] = (int8_t)split8(kk);
      base[(3 + i) * HD + dd] = (int8_t)split8(vv);
    }
  }
}

// ---- attention output: o = div_round(num, 5, den), quant(o, -FR) (segs.attn_div + quant; _attn_out_kernel) ----
constexpr int AO_THREADS = 512;  // a row is a latency chain: more threads, fewer serial divisions each
constexpr int AO_EPT = 8;      // H * HD <= 4096
constexpr int AO_MAXH = 64;

// Head sizes that are no multiple of four.
__global__ void __launch_bounds__(AO_THREADS)
attn_out_any_kernel(const i64* __restrict__ num, const i64* __restrict__ den, int32_t* __restrict__ q,
                i64* __restrict__ sh_out, int8_t* __restrict__ a8, int M, int K2, int HD) {
  __shared__ i64 red[32];
  __shared__ u64 dens[AO_MAXH], invs[AO_MAXH];
  const int64_t row = blockIdx.x;
  const int nh = K2 / HD;
  i64 o[AO_EPT];
  wait_previous();
  launch_next();
#pragma unroll
  for (int k = 0; k < AO_EPT; ++k) {                  // the numerators are in flight while the reciprocals are made
    const int c = threadIdx.x + k * AO_THREADS;
    o[k] = c < K2 ? num[row * K2 + c] : 0;
  }
  if (threadIdx.x < nh) {
    const u64 dv = (u64)den[row * nh + threadIdx.x];
    dens[threadIdx.x] = dv;
    invs[threadIdx.x] = dv ? ~0ull / dv : 0;
  }
  __syncthreads();
  i64 omax = 0;
#pragma unroll
  for (int k = 0; k < AO_EPT; ++k) {
    const int c = threadIdx.x + k * AO_THREADS;
    if (c < K2) {
      const int hd = c / HD;
      o[k] = dens[hd] ? div_round_recip<1>(o[k], FR - FV, dens[hd], invs[hd]) : 0;
      omax = mag_or(omax, o[k]);
    }
  }
  omax = block_or(omax, red);
  const i64 sh = quant_sh(omax, -FR);
  if (threadIdx.x == 0) sh_out[row] = sh;
  const int64_t plane = (int64_t)M * K2;
#pragma unroll
  for (int k = 0; k < AO_EPT; ++k) {
    const int c = threadIdx.x + k * AO_THREADS;
    if (c < K2) {
      const int qv = (int)rshc(o[k], sh + FR);
      q[row * K2 + c] = qv;
      if (a8) store_limb_planes(a8, plane, row * K2 + c, qv);
    }
  }
}

// One row by the integer rule (quotients that leave the ranges of the form below).
template <int NT, int Q>
__device__ __noinline__ void attn_out_row(const i64* num, const i64* den, int32_t* q, i64* sh_out, int8_t* a8, int64_t row, int M, int K2,
                                          int HD, i64* red) {
  i64 o[4 * Q];
  i64 omax = 0;
#pragma unroll
  for (int k = 0; k < 4 * Q; ++k) {
    const int c = threadIdx.x + k * NT;
    o[k] = 0;
    if (c < K2) {
      const i64 d = den[row * (K2 / HD) + c / HD];
      if (d) o[k] = div_round_recip<1>(num[row * K2 + c], FR - FV, (u64)d, ~0ull / (u64)d);
      omax = mag_or(omax, o[k]);
    }
  }
  omax = group_or<NT>(omax, red, 0);
  const i64 sh = quant_sh(omax, -FR);
  if (threadIdx.x == 0) sh_out[row] = sh;
  const int64_t plane = (int64_t)M * K2;
#pragma unroll
  for (int k = 0; k < 4 * Q; ++k) {
    const int c = threadIdx.x + k * NT;
    if (c < K2) {
      const int qv = (int)rshc(o[k], sh + FR);
      q[row * K2 + c] = qv;
      if (a8) store_limb_planes(a8, plane, row * K2 + c, qv);
    }
  }
}

// One row per CTA; a thread has four consecutive entries of one head (HD is a multiple of four) and Q such groups.
// o = floor(32 num / den + 1/2): num is one rounding (its halves are exact), 32 / den another and the product a third, so
// for |o| < 2^29 the quotient is known to 2^-21; nearer to a boundary than 2^-20 the integer division decides.
// 3750 rows of 2048: 66 -> 26 us (4.5 TB/s), 256 rows 6.7 -> 4.1 us, one row 3.9 -> 2.1 us; with an entry from 32 on in every row,
// which takes the integer rule for the row, 72 -> 106 us.
template <int NT, int Q>
__global__ void __launch_bounds__(NT)
attn_out_kernel(const i64* __restrict__ num, const i64* __restrict__ den, int32_t* __restrict__ q,
                i64* __restrict__ sh_out, int8_t* __restrict__ a8, int M, int K2, int HD, bool wide) {
  __shared__ uint32_t red32[32];
  __shared__ i64 red[32];
  const int64_t row = blockIdx.x;
  const int nh = K2 / HD;
  i64 o[Q][4], d[Q];
  wait_previous();
  launch_next();
#pragma unroll
  for (int k = 0; k < Q; ++k) {
    const int c = 4 * (threadIdx.x + k * NT);
    d[k] = 0;
    if (c < K2) {
      load4(num + row * K2 + c, wide, o[k]);
      d[k] = den[row * nh + c / HD];
    }
  }
  uint32_t omax = 0;
  int v[Q][4];
#pragma unroll
  for (int k = 0; k < Q; ++k) {
    const double inv = 32.0 / (double)d[k];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[k][j] = 0;
      if (d[k] != 0) {
        const double y = fma(s32_to_f64((int)(o[k][j] >> 32)), 4294967296.0, u32_to_f64((uint32_t)o[k][j])) * inv;
        const double t = __dadd_rd(y, F2I), e = (y - (t - F2I)) - 0.5;
        const int eh = __double2hiint(e);
        v[k][j] = __double2loint(t) + 1 + (eh >> 31);
        uint32_t size = (uint32_t)__double2hiint(y) & 0x7fffffffu;
        if ((uint32_t)(eh & 0x7fffffff) < (1003u << 20) && size < (1052u << 20))
          v[k][j] = (int)long_division<1>(o[k][j], FR - FV, (u64)d[k]);
        omax = max(omax, size >= (1052u << 20) || d[k] < 0 ? 0xffffffffu : (uint32_t)abs(v[k][j]));
      }
    }
  }
  omax = group_max<NT>(omax, red32, 0);
  if (omax == 0xffffffffu) {
    attn_out_row<NT, Q>(num, den, q, sh_out, a8, row, M, K2, HD, red);
    return;
  }
  const i64 sh = quant_sh(omax, -FR);
  if (threadIdx.x == 0) sh_out[row] = sh;
  const int64_t plane = (int64_t)M * K2;
  const int c = omax ? (int)sh + FR : 0;
  const int half = c > 0 ? 1 << (c - 1) : 0, right = max(c, 0), left = max(-c, 0);
#pragma unroll
  for (int k = 0; k < Q; ++k) {
    const int col = 4 * (threadIdx.x + k * NT);
#pragma unroll
    for (int j = 0; j < 4; ++j) v[k][j] = ((v[k][j] + half) >> right) << left;
    if (col < K2) store_q4(q, a8, plane, row * K2 + col, wide, v[k]);
  }
}

// ---- SiLU(g) * u + quant(., -2 FR) (segs.silu_y + quant_silu; exact/ops.py:119-130; _silu_kernel) ----
constexpr int SILU_THREADS = 512;

template <bool SMEM_TABLE = false>
__device__ __forceinline__ i64 silu_p(i64 g, i64 u, const i64* __restrict__ lut, bool& bad) {
  const i64 a = imin(iabs(g), 64ll << FR);                       // <= 2^30: the product below is 32 x 32 -> 64 bits
  const i64 t = rshs<FR + 30 - FT2>((i64)((u64)(uint32_t)a * (u64)(uint32_t)L2E30));
  const i64 E = exp2neg_lut<SMEM_TABLE>(t, lut, 30);
  const i64 den = (1ll << 30) + E;
  const i64 nume = g >= 0 ? (1ll << 60) : shl(E, 30);
  const i64 sig = fdiv_pos_est(2 * nume + den, 2 * den);          // rdiv
  const i64 gc = iclamp(g, -(1ll << 32), 1ll << 32);
  const i64 s = rshs<30>(gc * sig);
  const u64 as = (u64)iabs(s), au = (u64)iabs(u);
  bad = iabs(g) > (1ll << 32);
  if ((as | au) >> 31) bad |= bitlen((i64)as) + bitlen((i64)au) > 62;      // both below 2^31: 62 bits cannot be passed
  return (i64)((u64)s * (u64)u);
}

// The same for |g|, |u| < 2^30 (below 64 in value), otherwise silu_p itself. About 80 issue slots (silu_p: 200):
// the sigmoid's quotient r = floor(2^60 / den + 1/2) from a rough reciprocal and one Newton step (off by at most one,
// which the low 32 bits of 2^60 - r den tell; it is never a tie, 2^61 / den being odd only for den = 2^61), and
// floor(E 2^30 / den + 1/2) = 2^30 - r, as E = den - 2^30.
template <bool SMEM_TABLE>
__device__ __noinline__ i64 silu_rare(i64 g, i64 u, const i64* __restrict__ lut, bool& bad) {
  return silu_p<SMEM_TABLE>(g, u, lut, bad);
}
template <bool SMEM_TABLE = false>
__device__ __forceinline__ i64 silu_fast(i64 gl, i64 ul, const i64* __restrict__ lut, bool& anybad) {
  const int g = (int)gl, u = (int)ul;
  const int out = ((int)(gl >> 32) ^ (g >> 31)) | ((int)(ul >> 32) ^ (u >> 31)) |
                  (int)(((uint32_t)(g + 0x40000000) | (uint32_t)(u + 0x40000000)) >> 31);
  const uint32_t a = (uint32_t)abs(g);
  const u64 tt = (u64)a * (uint32_t)L2E30 + (1ull << (FR + 30 - FT2 - 1));
  const uint32_t t = (uint32_t)(tt >> (FR + 30 - FT2));
  const uint32_t n = (t >> FT2) + ((uint32_t)(tt >> 32) >> (FR + 30 - FT2)) * 64u;      // t has up to 33 bits
  const int idx = (int)(t >> (FT2 - EXP2_BITS)) & ((1 << EXP2_BITS) - 1);
  const i64 e0 = SMEM_TABLE ? lut[idx] : __ldg(lut + idx), e1 = SMEM_TABLE ? lut[idx + 1] : __ldg(lut + idx + 1);
  const i64 v = e0 + rshs<FT2 - EXP2_BITS>((e1 - e0) * (i64)(t & ((1u << (FT2 - EXP2_BITS)) - 1)));
  if (out != 0 || (u64)v >> 61) {
    bool bad;
    const i64 P = silu_rare<SMEM_TABLE>(gl, ul, lut, bad);
    anybad |= bad;
    return P;
  }
  const uint32_t E = (shr_clamp((uint32_t)((u64)v >> 29), n) + 1) >> 1;
  const uint32_t den = (1u << 30) + E;
  const double dd = u32_to_f64(den), x0 = rcp_f64_rough(dd), x1 = fma(x0, fma(-dd, x0, 1.0), x0);
  uint32_t r = (uint32_t)__double2loint(fma(x1, 1152921504606846976.0, F2I));
  const int rem = (int)(0u - r * den), half = (int)(den >> 1);
  r += (rem > half ? 1 : 0) - (rem < -half ? 1 : 0);
  const int sig = g >= 0 ? (int)r : (1 << 30) - (int)r;
  const int s = (int)(((i64)g * sig + (1ll << 29)) >> 30);
  return (i64)s * u;
}

template <int EPT>
__global__ void __launch_bounds__(SILU_THREADS)
silu_kernel(const i64* __restrict__ y, const i64* __restrict__ lut, int32_t* __restrict__ q, i64* __restrict__ sh_out,
            int8_t* __restrict__ a8, int32_t* flag, int M, int FF) {
  __shared__ i64 red[33];
  const int64_t row = blockIdx.x;
  const i64* yr = y + row * (2 * (int64_t)FF);
  i64 P[EPT];
  i64 pmax = 0;
  bool anybad = false;
  wait_previous();
  launch_next();
#pragma unroll
  for (int k = 0; k < EPT; ++k) {
    const int c = threadIdx.x + k * SILU_THREADS;
    P[k] = 0;
    if (c < FF) {
      bool bad;
      P[k] = silu_p(yr[c], yr[FF + c], lut, bad);
      anybad |= bad;
      pmax = mag_or(pmax, P[k]);
    }
  }
  if (anybad) *flag = 1;
  pmax = block_or(pmax, red);
  const i64 sh = quant_sh(pmax, -2 * FR);
  if (threadIdx.x == 0) sh_out[row] = sh;
  const int64_t plane = (int64_t)M * FF;
#pragma unroll
  for (int k = 0; k < EPT; ++k) {
    const int c = threadIdx.x + k * SILU_THREADS;
    if (c < FF) {
      const int qv = (int)rshc(P[k], sh + 2 * FR);
      q[row * FF + c] = qv;
      if (a8) store_limb_planes(a8, plane, row * FF + c, qv);
    }
  }
}

// P 2^-c of four consecutive entries, rounded half up, 1 <= c <= 62 or (c <= 0) shifted left.
__device__ __forceinline__ void quant4(const i64 (&P)[4], int c, int (&v)[4]) {
  if (c > 0) {
    const i64 half = 1ll << (c - 1);
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = (int)((P[j] + half) >> c);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = (int)shl(P[j], -c);
  }
}

// Cluster form of silu_kernel for decode batches: the columns of a row are split over the CTAs of a thread-block
// cluster (one row of 8192: 7.3 -> 4.4 us; 256 threads, Q groups of four consecutive columns each), the row maximum is exchanged through distributed
// shared memory: a row alone is a latency chain, and its CTAs gather from the table at the same time. FF % 4 == 0.
constexpr int SILU_CL_THREADS = 256;

template <int Q>
__global__ void __launch_bounds__(SILU_CL_THREADS)
silu_cluster_kernel(const i64* __restrict__ y, const i64* __restrict__ lut, int32_t* __restrict__ q,
                    i64* __restrict__ sh_out, int8_t* __restrict__ a8, int32_t* flag, int M, int FF, bool wide) {
  namespace cg = cooperative_groups;
  __shared__ i64 red[32];
  __shared__ i64 cta_max;
  cg::cluster_group cluster = cg::this_cluster();
  const int part = (int)cluster.block_rank(), parts = (int)cluster.num_blocks();
  const int64_t row = blockIdx.x / parts;
  const int per = (FF / 4 + parts - 1) / parts;            // groups of four columns per CTA
  const i64* yr = y + row * (2 * (int64_t)FF);
  i64 P[Q][4];
  i64 pmax = 0;
  bool anybad = false;
  wait_previous();
  launch_next();
#pragma unroll
  for (int k = 0; k < Q; ++k) {
    const int own = threadIdx.x + k * SILU_CL_THREADS, c = 4 * (part * per + own);
    i64 u[4] = {0, 0, 0, 0};
#pragma unroll
    for (int j = 0; j < 4; ++j) P[k][j] = 0;
    if (own < per && c < FF) {
      load4(yr + c, wide, P[k]);
      load4(yr + FF + c, wide, u);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      P[k][j] = silu_fast(P[k][j], u[j], lut, anybad);
      pmax = mag_or(pmax, P[k][j]);
    }
  }
  if (anybad) *flag = 1;
  pmax = group_or<SILU_CL_THREADS>(pmax, red, 0);
  if (threadIdx.x == 0) cta_max = pmax;
  cluster.sync();
  i64 rmax = 0;
  for (int r = 0; r < parts; ++r) rmax |= *cluster.map_shared_rank(&cta_max, r);
  const i64 sh = quant_sh(rmax, -2 * FR);
  if (part == 0 && threadIdx.x == 0) sh_out[row] = sh;
  const int64_t plane = (int64_t)M * FF;
  const int c = (int)imax(sh + 2 * FR, -62);
#pragma unroll
  for (int k = 0; k < Q; ++k) {
    const int own = threadIdx.x + k * SILU_CL_THREADS, col = 4 * (part * per + own);
    int v[4];
    quant4(P[k], c, v);
    if (own < per && col < FF) store_q4(q, a8, plane, row * FF + col, wide, v);
  }
  cluster.sync();                                   // peers may still be reading cta_max
}

// Persistent form with the 2^-f table (131 KB) in shared memory: one 1024-thread CTA per SM walks the rows, in groups of
// GT threads with a row and a barrier each (a group's loads and barrier are hidden by the others), Q groups of four columns per
// thread. The table gathers are what the other forms wait for (they miss L1); from shared memory they cost a few cycles, and a
// CTA fetches the table once for all its rows. 23 bytes and 117 warp instructions per 32 elements. FF % 4 == 0, FF <= 4 GT Q.
// 3750 rows of 8192: 275 -> 164 us (4.3 TB/s), of 14336 1875 rows 405 -> 155 us; 256 rows of 8192 25.2 -> 17.5 us. ncu: issue 63 %, waits for
// loads (64 registers hold no second row and spill 124 bytes; asking for the next row's lines in L2 cost 20 %). Arguments beyond 64
// take the general form one by one: 1875 rows of 8192 98 us, 106 with one in 1000 of them, 150 with one in 100 (148 before).
constexpr int SILU_P_THREADS = 1024;
constexpr int SILU_TABLE = (1 << EXP2_BITS) + 1;

template <int GT, int Q>
__global__ void __launch_bounds__(SILU_P_THREADS, 1)
silu_persistent_kernel(const i64* __restrict__ y, const i64* __restrict__ lut, int32_t* __restrict__ q,
                       i64* __restrict__ sh_out, int8_t* __restrict__ a8, int32_t* flag, int M, int FF, bool wide) {
  constexpr int GROUPS = SILU_P_THREADS / GT;
  extern __shared__ __align__(16) uint8_t silu_smem[];
  i64* tab = reinterpret_cast<i64*>(silu_smem);
  __shared__ i64 red[GROUPS][2][32];
  const int group = threadIdx.x / GT, t = threadIdx.x % GT;
  int turn = 0;
  // the table into L2 while the previous kernel ends, a part per CTA (256 sequences: 6046 -> 6017 us a step, this and the
  // same for the streaming attention's table, which has since become an asynchronous copy)
  for (int i = 4 * (blockIdx.x * SILU_P_THREADS + threadIdx.x); i < SILU_TABLE; i += 4 * gridDim.x * SILU_P_THREADS) prefetch_l2(lut + i);
  wait_previous();
  launch_next();
  for (int i = threadIdx.x; i < SILU_TABLE; i += SILU_P_THREADS) tab[i] = __ldg(lut + i);
  __syncthreads();
  const int64_t plane = (int64_t)M * FF;
  bool anybad = false;
  for (int64_t row = (int64_t)group * gridDim.x + blockIdx.x; row < M; row += (int64_t)GROUPS * gridDim.x) {
    const i64* yr = y + row * (2 * (int64_t)FF);
    i64 P[Q][4];
    i64 pmax = 0;
#pragma unroll
    for (int k = 0; k < Q; ++k) {
      const int c = 4 * (t + k * GT);
      i64 u[4] = {0, 0, 0, 0};
#pragma unroll
      for (int j = 0; j < 4; ++j) P[k][j] = 0;
      if (c < FF) {
        load4(yr + c, wide, P[k]);
        load4(yr + FF + c, wide, u);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        P[k][j] = silu_fast<true>(P[k][j], u[j], tab, anybad);
        pmax = mag_or(pmax, P[k][j]);
      }
    }
    pmax = group_or<GT>(pmax, red[group][turn ^= 1], group);     // a warp is at most one row ahead of another of its group
    const i64 sh = quant_sh(pmax, -2 * FR);
    if (t == 0) sh_out[row] = sh;
    const int s = (int)imax(sh + 2 * FR, -62);
#pragma unroll
    for (int k = 0; k < Q; ++k) {
      const int c = 4 * (t + k * GT);
      int v[4];
      quant4(P[k], s, v);
      if (c < FF) store_q4(q, a8, plane, row * FF + c, wide, v);
    }
  }
  if (anybad) *flag = 1;
}

// ---- SiLU * up + quant in two kernels, for a gate / up projection sharded by output column over several GPUs ----
// silu_prod_kernel: y [N, 2 FFl] (the rank's gate columns, then its up columns) -> P int64 [N, FFl] and the row maximum
// of |P| over the rank's columns. The ranks then take the integer maximum of the row maxima (an exact all-reduce) and
// quant_rows_kernel quantises every shard with the same row exponent: the integers of silu_kernel on the full row.
template <int NT>
__global__ void __launch_bounds__(NT)
silu_prod_kernel(const i64* __restrict__ y, const i64* __restrict__ lut, i64* __restrict__ P, i64* __restrict__ rowmax,
                 int32_t* flag, int FFl) {
  __shared__ i64 red[33];
  const int64_t row = blockIdx.x;
  const i64* yr = y + row * (2 * (int64_t)FFl);
  i64 pmax = 0;
  bool anybad = false;
  for (int c = threadIdx.x; c < FFl; c += NT) {
    bool bad;
    const i64 v = silu_p(yr[c], yr[FFl + c], lut, bad);
    anybad |= bad;
    pmax = imax(pmax, iabs(v));
    P[row * FFl + c] = v;
  }
  if (anybad) *flag = 1;
  pmax = block_reduce<true>(pmax, red);
  if (threadIdx.x == 0) rowmax[row] = pmax;
}

// q = rshc(P, sh + fbits) with sh = quant_sh(rowmax, -fbits) (exact/ops.py:82-89); also the limb planes of q (optional)
// with row pitch `ldq` and plane size `plane` elements, so that a rank can write its columns into the full-width planes.
__global__ void __launch_bounds__(256)
quant_rows_kernel(const i64* __restrict__ P, const i64* __restrict__ rowmax, int fbits, int32_t* __restrict__ q,
                  int64_t ldq, i64* __restrict__ sh_out, int8_t* __restrict__ a8, int64_t plane, int K) {
  const int64_t row = blockIdx.x;
  const i64 sh = quant_sh(rowmax[row], -(i64)fbits);
  if (threadIdx.x == 0 && sh_out) sh_out[row] = sh;
  for (int c = threadIdx.x; c < K; c += 256) {
    const int qv = (int)rshc(P[row * K + c], sh + fbits);
    q[row * ldq + c] = qv;
    if (a8) store_limb_planes(a8, plane, row * ldq + c, qv);
  }
}

}  // namespace bx
