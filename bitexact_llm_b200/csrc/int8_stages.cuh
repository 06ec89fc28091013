// Row-local integer stages of int8 mode between its linears: RMSNorm + 2-limb row quantisation, RoPE + KV limb
// store, attention output division, SiLU-table * up + quantisation. They consume the int64 output y of the fused
// int8 linear (post already applied) and emit the next linear's input: activation limb planes int8 [2, M, K]
// (limb i of row m at row i * M + m, the layout of the reference's stack_limbs) and the row scale (mant, e).
//
// Same integers as src/bitexact/int8/ops.py:24-108 and int8/segs.py:48-118, and as the fused kernels of
// src/bitexact/vllm_plugin/tri_fuse.py:82-265 and vllm_plugin/tri_mlp.py:86-150.
#pragma once

#include "bx_rules.cuh"
#include "elementwise.cuh"
#include "int8_linear.cuh"

namespace bx {
namespace i8 {

constexpr int FR = 16, FG = 12, FA = 12, FT = 16, FQ = 14, FV = 14;
constexpr i64 EPS40 = 10995116;
constexpr i64 QMAX2 = 127 << 8;
constexpr i64 SILU_LO = -(32 << 12), SILU_HI = 32 << 12;

// floor(n / d) for d > 0 from inv = floor((2^64 - 1) / d), |n| < 2^63.
__device__ __forceinline__ i64 fdiv_recip(i64 n, u64 d, u64 inv) {
  u64 rem;
  const u64 q = uqr_recip((u64)iabs(n), d, inv, rem);
  return n < 0 ? -(i64)q - (rem != 0 ? 1 : 0) : (i64)q;
}

// quant_rows(z, 2) pieces from the row's max |z| (int8/ops.py:24-35): shift sh, scaled maximum as_.
__device__ __forceinline__ void quant_scale(i64 zmax, i64& sh, i64& as_) {
  const i64 amax = imax(zmax, 1);
  sh = (i64)bitlen(amax) - 30;
  as_ = rsh_t(amax, sh);
}
__device__ __forceinline__ int quant2(i64 z, i64 sh, i64 as_, u64 inv) {
  const i64 zs = rsh_t(z, sh);
  return (int)fdiv_recip(2 * (zs * QMAX2) + as_, (u64)(2 * as_), inv);     // rdiv(zs * qmax, as_)
}
__device__ __forceinline__ void store_limbs2(int8_t* a8, int64_t plane, int64_t off, int q) {
  const int lo = ((q + 128) & 255) - 128;
  a8[off] = (int8_t)lo;
  a8[plane + off] = (int8_t)((q - lo) >> 8);
}
// norm24 (int8/ops.py:70-73)
__device__ __forceinline__ void norm24(i64 mant, i64 e, i64& m_out, i64& e_out) {
  const i64 b = (i64)bitlen(mant) - 24;
  m_out = rsh_t(mant, b);
  e_out = e + b;
}

// The largest |v| of the CTA as a double (all threads), from each thread's.
template <int NT>
__device__ __forceinline__ i64 group_max_f64(double v, i64* buf, int group) {
  const int lane = threadIdx.x & 31, warp = (threadIdx.x % NT) >> 5;
  const i64 w = warp_max(__double_as_longlong(v));           // doubles from 0 up are ordered as their bits are
  if (lane == 0) buf[warp] = w;
  group_sync<NT>(group);
  return warp_max(lane < NT / 32 ? buf[lane] : 0);
}

// quant2 of four values z (whole numbers as doubles) with |z| <= amax, and their two limb planes.
// floor(zs 32512 / as + 1/2) with zs = z 2^-sh rounded half up: |quotient| <= 32512, known to 2^-36.
struct QuantRow {
  i64 sh, as_;
  double half, down, ratio;                                  // zs = floor((z + half) down)
};
__device__ __forceinline__ QuantRow quant_row(i64 amax) {
  QuantRow r;
  quant_scale(amax, r.sh, r.as_);
  r.half = r.sh > 0 ? pow2_f64((int)r.sh - 1) : 0.0;
  r.down = pow2_f64(-(int)r.sh);
  r.ratio = (double)QMAX2 / (double)r.as_;
  return r;
}
__device__ __noinline__ int quant2_exact(double z, i64 sh, i64 as_) {
  return quant2(f64_to_int(z + F2I), sh, as_, ~0ull / (u64)(2 * as_));
}
__device__ __forceinline__ void quant_store4(const double (&z)[4], const QuantRow& r, int8_t* a8, int64_t plane, int64_t off, bool on, bool wide) {
  uint32_t b[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const double zs = __fma_rd(z[j] + r.half, r.down, F2I) - F2I;
    const double t = __fma_rd(zs, r.ratio, F2I), d = fma(zs, r.ratio, F2I - t) - 0.5;
    const int dh = __double2hiint(d);
    int q = __double2loint(t) + 1 + (dh >> 31);
    if ((uint32_t)(dh & 0x7fffffff) < (1003u << 20)) q = quant2_exact(z[j], r.sh, r.as_);
    b[j] = limb_bytes((uint32_t)q);
  }
  if (!on) return;
  if (wide) {
    const uint32_t l01 = __byte_perm(b[0], b[1], 0x5140), l23 = __byte_perm(b[2], b[3], 0x5140);
    *reinterpret_cast<uint32_t*>(a8 + off) = __byte_perm(l01, l23, 0x5410);
    *reinterpret_cast<uint32_t*>(a8 + plane + off) = __byte_perm(l01, l23, 0x7632);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      a8[off + j] = (int8_t)b[j];
      a8[plane + off + j] = (int8_t)(b[j] >> 8);
    }
  }
}

// One row by the integer rules, for widths that are no multiple of four and values out of range of the form below.
template <int MODE, int NT>
__device__ __noinline__ void int8_norm_row(const void* xin, const i64* yin, const i64* ids, const i64* gamma, i64* xo, bool summed, int8_t* a8,
                                           i64* mant, i64* eo, int32_t* flag, int64_t row, int M, int D, int do_norm, i64 (*red)[32]) {
  constexpr int EPT = NORM_MAX_D / NT;
  i64 x[EPT];
  i64 ax = 0;
#pragma unroll
  for (int k = 0; k < EPT; ++k) {
    const int c = 4 * threadIdx.x + (k / 4) * 4 * NT + k % 4;
    x[k] = 0;
    if (c < D) {
      if (summed && xo) x[k] = xo[row * D + c];              // stored by this thread
      else if (MODE == 0) x[k] = (i64) reinterpret_cast<const int32_t*>(xin)[ids[row] * D + c];
      else if (MODE == 1) x[k] = reinterpret_cast<const i64*>(xin)[row * D + c] + yin[row * D + c];
      else x[k] = reinterpret_cast<const i64*>(xin)[row * D + c];
      if (xo && !summed) xo[row * D + c] = x[k];
      ax = mag_or(ax, x[k]);
    }
  }
  ax = block_or(ax, red[0]);                                          // its bit length and a power-of-two bound are what is read
  if (!do_norm) {
    if (threadIdx.x == 0 && ax >= (1ll << 42)) *flag = 1;
    __syncthreads();
    return;
  }
  const i64 shx = (i64)bitlen(imax(ax, 1)) - 24;                       // rms (int8/ops.py:76-84)
  i64 S = 0, zmax = 0;
#pragma unroll
  for (int k = 0; k < EPT; ++k) {
    const int c = 4 * threadIdx.x + (k / 4) * 4 * NT + k % 4;
    if (c < D) {
      const i64 xs = rsh_t(x[k], shx);
      S += xs * xs;
      x[k] = x[k] * gamma[c];
      zmax = imax(zmax, iabs(x[k]));
    }
  }
  S = block_sum_pos(S, red[1]);
  zmax = block_max(zmax, red[2]);
  const i64 r = isqrt(S / D + rsh_t(EPS40, 40 - 2 * (FR - shx)));
  i64 sh, as_;
  quant_scale(zmax, sh, as_);
  const u64 inv = ~0ull / (u64)(2 * as_);
  const int64_t plane = (int64_t)M * D;
#pragma unroll
  for (int k = 0; k < EPT; ++k) {
    const int c = 4 * threadIdx.x + (k / 4) * 4 * NT + k % 4;
    if (c < D) store_limbs2(a8, plane, row * D + c, quant2(x[k], sh, as_, inv));
  }
  if (threadIdx.x == 0) {
    const i64 mq = fdiv(2 * shl(as_, 30) + r, 2 * r);                  // rdiv(as_ << 30, r)
    norm24(mq, sh - FG - shx - 30, mant[row], eo[row]);
  }
  __syncthreads();                                                     // the buffers are free for the next row
}

// MODE 0: x = emb[ids]; 1: x = xin + yin; 2: x = xin. With do_norm: pre_norm(x, gamma) (int8/segs.py:48-53). As norm_kernel of
// exact mode: rows walked with gamma in registers, four consecutive columns per thread, products and quotients in double
// precision where |x gamma| < 2^51 (26 bytes an element). 1875 rows of 2048: 45 -> 26 us (3.8 TB/s), one row 7.3 -> 3.6 us.
template <int MODE, int NT, int Q>
__global__ void __launch_bounds__(NT, 1024 / NT)
int8_norm_kernel(const void* __restrict__ xin, const i64* __restrict__ yin, const i64* __restrict__ ids,
                 const i64* __restrict__ gamma, i64* xo, int8_t* __restrict__ a8, i64* __restrict__ mant,
                 i64* __restrict__ eo, int32_t* flag, int M, int D, int do_norm, bool wide) {
  __shared__ i64 red[3][32];
  uint32_t* red32 = reinterpret_cast<uint32_t*>(red);
  if (do_norm)
    for (int c = 4 * threadIdx.x; c < D; c += 4 * NT) prefetch_l2(gamma + c);
  wait_previous();
  launch_next();
  if (D % 4) {
    for (int64_t row = blockIdx.x; row < M; row += gridDim.x)
      int8_norm_row<MODE, NT>(xin, yin, ids, gamma, xo, false, a8, mant, eo, flag, row, M, D, do_norm, red);
    return;
  }
  double G[Q][4];
  uint32_t gtop = 0;
#pragma unroll
  for (int k = 0; k < Q; ++k) {
    const int c = 4 * (threadIdx.x + k * NT);
    i64 g4[4] = {0, 0, 0, 0};
    if (do_norm && c < D) load4(gamma + c, wide, g4);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      G[k][j] = to_f64(g4[j]);
      gtop = max(gtop, in_f64(g4[j]) ? (uint32_t)__double2hiint(G[k][j]) & 0x7fffffffu : 0x7fefffffu);
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
    if (bits + gbits > 51 || bits > 42) {
      __syncthreads();
      int8_norm_row<MODE, NT>(xin, yin, ids, gamma, xo, true, a8, mant, eo, flag, row, M, D, do_norm, red);
      continue;
    }
    if (!do_norm) {                                                    // below 2^42: no flag
      __syncthreads();
      continue;
    }
    const int shx = (bits ? bits : 1) - 24;                            // rms (int8/ops.py:76-84)
    double S = 0.0, zmax = 0.0;                                        // at most 8 squares of 2^24 per thread: exact
    {
      const double half = shx > 0 ? pow2_f64(shx - 1) : 0.0, down = pow2_f64(-shx);
#pragma unroll
      for (int k = 0; k < Q; ++k)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const double xs = __fma_rd(x[k][j] + half, down, F2I) - F2I;
          S = fma(xs, xs, S);
          x[k][j] *= G[k][j];
          zmax = fmax(zmax, fabs(x[k][j]));
        }
    }
    const i64 sum = group_sum<NT>((i64)S, red[1], 0);
    const QuantRow qr = quant_row(f64_to_int(__longlong_as_double(group_max_f64<NT>(zmax, red[2], 0)) + F2I));
#pragma unroll
    for (int k = 0; k < Q; ++k) {
      const int c = 4 * (threadIdx.x + k * NT);
      quant_store4(x[k], qr, a8, plane, row * D + c, c < D, wide);
    }
    if (threadIdx.x == 0) {
      const i64 r = isqrt(sum / D + rsh_t(EPS40, 40 - 2 * (FR - shx)));
      const i64 mq = fdiv(2 * shl(qr.as_, 30) + r, 2 * r);             // rdiv(as_ << 30, r)
      norm24(mq, qr.sh - FG - shx - 30, mant[row], eo[row]);
    }
  }
}

// RoPE (16-bit cos / sin) of q and k, v >> 2, bound flag, K / V limb planes stored in the paged cache
// (int8/segs.py:69-88; tri_fuse._qkv_kernel). One CTA per (token, KV head), HD / 2 threads.
struct Qkv8Params {
  const i64* y;
  const i64* cos;
  const i64* sin;
  const i64* pos;
  const i64* slot;
  int8_t* cache;
  int64_t sc_nb, sc_h, sc_bs;
  int bs;
  i64* q64;          // [N, HKV, G, HD] (may be null)
  int32_t* q32;      // same values as int32 (may be null)
  int32_t* flag;
  int H, HKV, HD;
};

__global__ void int8_qkv_kernel(const Qkv8Params p) {
  __shared__ i64 red[33];
  const int64_t row = blockIdx.x;
  const int h = blockIdx.y;
  const int HH = p.HD / 2, G = p.H / p.HKV, dd = threadIdx.x;
  const int64_t NT = (int64_t)(p.H + 2 * p.HKV) * p.HD;
  constexpr int SHR = FT + FR - FQ;
  wait_previous();
  launch_next();
  const i64 pos = p.pos[row];
  const i64 cs = p.cos[pos * HH + dd], sn = p.sin[pos * HH + dd];
  const i64* yr = p.y + row * NT;
  i64 big = 0;
  for (int g = 0; g < G; ++g) {
    const int64_t qc = (int64_t)(h * G + g) * p.HD + dd;
    const i64 x1 = yr[qc], x2 = yr[qc + HH];
    const i64 q1 = rshs<SHR>(x1 * cs - x2 * sn), q2 = rshs<SHR>(x2 * cs + x1 * sn);
    big = imax(big, imax(iabs(q1), iabs(q2)));
    const int64_t qo = row * ((int64_t)p.H * p.HD) + qc;            // [N, HKV, G, HD] == [N, H, HD]
    if (p.q64) { p.q64[qo] = q1; p.q64[qo + HH] = q2; }
    if (p.q32) { p.q32[qo] = (int32_t)q1; p.q32[qo + HH] = (int32_t)q2; }
  }
  const int64_t kc = (int64_t)p.H * p.HD + (int64_t)h * p.HD + dd;
  const int64_t vc = (int64_t)(p.H + p.HKV) * p.HD + (int64_t)h * p.HD + dd;
  const i64 k1 = yr[kc], k2 = yr[kc + HH];
  const i64 k1o = rshs<SHR>(k1 * cs - k2 * sn), k2o = rshs<SHR>(k2 * cs + k1 * sn);
  const i64 v1 = rshs<FR - FV>(yr[vc]), v2 = rshs<FR - FV>(yr[vc + HH]);
  big = imax(big, imax(imax(iabs(k1o), iabs(k2o)), imax(iabs(v1), iabs(v2))));
  big = block_reduce<true>(big, red);
  if (threadIdx.x == 0 && big > LIM3) *p.flag = 1;
  if (p.cache) {
    const i64 slot = p.slot[row];
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

// Head sizes that are no multiple of four.
// o = rdiv(num << 2, den) per head, then pre_plain(o) (int8/segs.py:101-109; tri_fuse._attn_out_kernel).
__global__ void __launch_bounds__(AO_THREADS)
int8_attn_out_any_kernel(const i64* __restrict__ num, const i64* __restrict__ den, int8_t* __restrict__ a8,
                     i64* __restrict__ mant, i64* __restrict__ eo, int M, int K2, int HD) {
  __shared__ i64 red[32];
  __shared__ u64 dens[AO_MAXH], invs[AO_MAXH];
  const int64_t row = blockIdx.x;
  const int nh = K2 / HD;
  wait_previous();
  launch_next();
  if (threadIdx.x < nh) {
    const u64 dv = 2 * (u64)den[row * nh + threadIdx.x];
    dens[threadIdx.x] = dv;
    invs[threadIdx.x] = dv ? ~0ull / dv : 0;
  }
  __syncthreads();
  i64 o[AO_EPT];
  i64 omax = 0;
#pragma unroll
  for (int k = 0; k < AO_EPT; ++k) {
    const int c = threadIdx.x + k * AO_THREADS;
    o[k] = 0;
    if (c < K2) {
      const int hd = c / HD;
      if (dens[hd]) o[k] = fdiv_recip(2 * shl(num[row * K2 + c], FR - FV) + (i64)(dens[hd] >> 1), dens[hd], invs[hd]);
      omax = imax(omax, iabs(o[k]));
    }
  }
  omax = block_max(omax, red);
  i64 sh, as_;
  quant_scale(omax, sh, as_);
  const u64 inv = ~0ull / (u64)(2 * as_);
  const int64_t plane = (int64_t)M * K2;
#pragma unroll
  for (int k = 0; k < AO_EPT; ++k) {
    const int c = threadIdx.x + k * AO_THREADS;
    if (c < K2) store_limbs2(a8, plane, row * K2 + c, quant2(o[k], sh, as_, inv));
  }
  if (threadIdx.x == 0) norm24(as_, sh - FR, mant[row], eo[row]);
}

// One row by the integer rules (quotients that leave the ranges of the form below).
template <int NT, int Q>
__device__ __noinline__ void int8_attn_out_row(const i64* num, const i64* den, int8_t* a8, i64* mant, i64* eo, int64_t row, int M, int K2, int HD,
                                               i64* red) {
  i64 o[4 * Q];
  i64 omax = 0;
#pragma unroll
  for (int k = 0; k < 4 * Q; ++k) {
    const int c = threadIdx.x + k * NT;
    o[k] = 0;
    if (c < K2) {
      const u64 d = 2 * (u64)den[row * (K2 / HD) + c / HD];
      if (d) o[k] = fdiv_recip(2 * shl(num[row * K2 + c], FR - FV) + (i64)(d >> 1), d, ~0ull / d);
      omax = imax(omax, iabs(o[k]));
    }
  }
  omax = block_max(omax, red);
  i64 sh, as_;
  quant_scale(omax, sh, as_);
  const u64 inv = ~0ull / (u64)(2 * as_);
  const int64_t plane = (int64_t)M * K2;
#pragma unroll
  for (int k = 0; k < 4 * Q; ++k) {
    const int c = threadIdx.x + k * NT;
    if (c < K2) store_limbs2(a8, plane, row * K2 + c, quant2(o[k], sh, as_, inv));
  }
  if (threadIdx.x == 0) norm24(as_, sh - FR, mant[row], eo[row]);
}
__device__ __noinline__ int attn_out_exact(i64 num, i64 den) {
  const u64 d = 2 * (u64)den;
  return (int)fdiv_recip(2 * shl(num, FR - FV) + (i64)(d >> 1), d, ~0ull / d);
}

// As attn_out_kernel of exact mode: floor(4 num / den + 1/2) in double precision, |o| < 2^29. 1875 rows of 2048: 36 -> 18 us, one
// row 4.7 -> 2.4 us.
template <int NT, int Q>
__global__ void __launch_bounds__(NT)
int8_attn_out_kernel(const i64* __restrict__ num, const i64* __restrict__ den, int8_t* __restrict__ a8,
                     i64* __restrict__ mant, i64* __restrict__ eo, int M, int K2, int HD, bool wide) {
  __shared__ uint32_t red32[32];
  __shared__ i64 red[32];
  const int64_t row = blockIdx.x;
  const int nh = K2 / HD;
  i64 n[Q][4], d[Q];
  wait_previous();
  launch_next();
#pragma unroll
  for (int k = 0; k < Q; ++k) {
    const int c = 4 * (threadIdx.x + k * NT);
    d[k] = 0;
    if (c < K2) {
      load4(num + row * K2 + c, wide, n[k]);
      d[k] = den[row * nh + c / HD];
    }
  }
  uint32_t omax = 0;
  double o[Q][4];
#pragma unroll
  for (int k = 0; k < Q; ++k) {
    const double inv = 4.0 / (double)d[k];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      o[k][j] = 0.0;
      if (d[k] != 0) {
        const double y = fma(s32_to_f64((int)(n[k][j] >> 32)), 4294967296.0, u32_to_f64((uint32_t)n[k][j])) * inv;
        const double t = __dadd_rd(y, F2I), e = (y - (t - F2I)) - 0.5;
        const int eh = __double2hiint(e);
        const uint32_t size = (uint32_t)__double2hiint(y) & 0x7fffffffu;
        int v = __double2loint(t) + 1 + (eh >> 31);
        if ((uint32_t)(eh & 0x7fffffff) < (1003u << 20) && size < (1052u << 20)) v = attn_out_exact(n[k][j], d[k]);
        omax = max(omax, size >= (1052u << 20) || d[k] < 0 || d[k] >= (1ll << 61) ? 0xffffffffu : (uint32_t)abs(v));
        o[k][j] = s32_to_f64(v);
      }
    }
  }
  omax = group_max<NT>(omax, red32, 0);
  if (omax == 0xffffffffu) {
    int8_attn_out_row<NT, Q>(num, den, a8, mant, eo, row, M, K2, HD, red);
    return;
  }
  const QuantRow qr = quant_row((i64)omax);
  const int64_t plane = (int64_t)M * K2;
#pragma unroll
  for (int k = 0; k < Q; ++k) {
    const int c = 4 * (threadIdx.x + k * NT);
    quant_store4(o[k], qr, a8, plane, row * K2 + c, c < K2, wide);
  }
  if (threadIdx.x == 0) norm24(qr.as_, qr.sh - FR, mant[row], eo[row]);
}

// SiLU at FR from the table at step 2^-12 with linear interpolation (int8/ops.py:100-108).
__device__ __forceinline__ i64 silu_tab(i64 g, const i64* __restrict__ lut) {
  const i64 gi = g >> (FR - FA);
  const i64 r = g - shl(gi, FR - FA);
  const i64 i = iclamp(gi, SILU_LO, SILU_HI - 1) - SILU_LO;
  const i64 a = __ldg(lut + i);
  const i64 v = a + rshs<FR - FA>((__ldg(lut + i + 1) - a) * r);
  return gi >= SILU_HI ? g : (gi < SILU_LO ? 0 : v);
}

// h = rsh(silu(g) * u, FR), pre_plain(h); the row maxima of |silu(g)| and |u| go to scr[0], scr[1] as atomic
// maxima (int8/segs.py:111-118; tri_mlp._h_kernel / _quant_kernel with ATOMIC).
template <int EPT>
__global__ void __launch_bounds__(SILU_THREADS)
int8_silu_kernel(const i64* __restrict__ y, const i64* __restrict__ lut, int8_t* __restrict__ a8,
                 i64* __restrict__ mant, i64* __restrict__ eo, i64* __restrict__ scr, int M, int FF) {
  __shared__ i64 red[3][32];
  const int64_t row = blockIdx.x;
  const i64* yr = y + row * (2 * (int64_t)FF);
  i64 hv[EPT];
  i64 hmax = 0, smax = 0, umax = 0;
  wait_previous();
  launch_next();
#pragma unroll
  for (int k = 0; k < EPT; ++k) {
    const int c = threadIdx.x + k * SILU_THREADS;
    hv[k] = 0;
    if (c < FF) {
      const i64 sg = silu_tab(yr[c], lut), u = yr[FF + c];
      hv[k] = rshs<FR>((i64)((u64)sg * (u64)u));
      hmax = imax(hmax, iabs(hv[k]));
      smax = imax(smax, iabs(sg));
      umax = imax(umax, iabs(u));
    }
  }
  hmax = block_max(hmax, red[0]);
  smax = block_max(smax, red[1]);
  umax = block_max(umax, red[2]);
  if (threadIdx.x == 0 && scr) {
    atomicMax(reinterpret_cast<long long*>(scr), (long long)smax);
    atomicMax(reinterpret_cast<long long*>(scr + 1), (long long)umax);
  }
  i64 sh, as_;
  quant_scale(hmax, sh, as_);
  const u64 inv = ~0ull / (u64)(2 * as_);
  const int64_t plane = (int64_t)M * FF;
#pragma unroll
  for (int k = 0; k < EPT; ++k) {
    const int c = threadIdx.x + k * SILU_THREADS;
    if (c < FF) store_limbs2(a8, plane, row * FF + c, quant2(hv[k], sh, as_, inv));
  }
  if (threadIdx.x == 0) norm24(as_, sh - FR, mant[row], eo[row]);
}

// The compact SiLU table (bitexact_llm_b200/int8/consts.py: silu_compact): max(x, 0) - silu(x) of the table's entries for
// |x| <= 8, 65537 x 16 bits (131 KB instead of 2 MB), which fits beside the rows of an SM. 1875 rows of 8192 (18 bytes an element):
// 152 -> 84 us (3.3 TB/s), of 14336 405 -> 128 us, 64 rows of 8192 20.8 -> 9.6 us, one row 12.7 -> 4.3 us. With 10 % of the arguments
// beyond 8, which go to the full table one by one, 1875 rows of 8192 158 -> 139 us. 64 registers a thread spill 192 bytes and load
// 420 (two rows at a time).
constexpr int SC_HALF = 8 << FA, SC_N = 2 * SC_HALF + 1, SC_BYTES = (SC_N * 2 + 15) / 16 * 16;

struct SiluAcc {
  uint32_t s, u;           // largest |silu(g)|, |u| of the fast form
  i64 rs, ru;              // and of the rest
};
struct SiluRare {
  i64 sg, h;
};
__device__ __noinline__ SiluRare silu8_rare(i64 g, i64 u, const i64* __restrict__ lut) {
  SiluRare r;
  r.sg = silu_tab(g, lut);
  r.h = rshs<FR>((i64)((u64)r.sg * (u64)u));
  return r;
}
// h of one element as a double; `big` where it does not fit one.
__device__ __forceinline__ double silu8(i64 gl, i64 ul, const uint16_t* tab, const i64* __restrict__ lut, SiluAcc& acc, bool& big) {
  const int g = (int)gl, u = (int)ul;
  const int gi = g >> (FR - FA), at = gi + SC_HALF;
  const bool fast = (int)(gl >> 32) == (g >> 31) && (int)(ul >> 32) == (u >> 31) && (uint32_t)at < (uint32_t)(SC_N - 1) &&
                    (uint32_t)(u + 0x40000000) >> 31 == 0;
  const int i = fast ? at : 0;
  const int a = max(gi, 0) * (1 << (FR - FA)) - (int)tab[i], b = max(gi + 1, 0) * (1 << (FR - FA)) - (int)tab[i + 1];
  const int r = g & ((1 << (FR - FA)) - 1);
  const int sg = a + (((b - a) * r + (1 << (FR - FA - 1))) >> (FR - FA));
  if (fast) {
    acc.s = max(acc.s, (uint32_t)abs(sg));
    acc.u = max(acc.u, (uint32_t)abs(u));
    // |sg u| < 2^50: floor((sg u + 2^15) 2^-16) in doubles
    return __fma_rd(fma(s32_to_f64(sg), s32_to_f64(u), 32768.0), 1.52587890625e-5, F2I) - F2I;
  }
  const SiluRare w = silu8_rare(gl, ul, lut);
  acc.rs = imax(acc.rs, iabs(w.sg));
  acc.ru = imax(acc.ru, iabs(ul));
  big |= !in_f64(w.h);
  return to_f64(w.h);
}

// One row by the integer rules (h beyond 2^51).
template <int NT>
__device__ __noinline__ void int8_silu_row(const i64* yr, const i64* lut, int8_t* a8, int64_t plane, int64_t off, i64* mant, i64* eo, int FF,
                                           i64* red, int group) {
  const int t = threadIdx.x % NT, lane = threadIdx.x & 31, warp = t >> 5;
  i64 hmax = 0;
  for (int c = t; c < FF; c += NT) hmax = imax(hmax, iabs(silu8_rare(yr[c], yr[FF + c], lut).h));
  hmax = warp_max(hmax);
  if (lane == 0) red[warp] = hmax;
  group_sync<NT>(group);
  hmax = warp_max(lane < NT / 32 ? red[lane] : 0);
  i64 sh, as_;
  quant_scale(hmax, sh, as_);
  const u64 inv = ~0ull / (u64)(2 * as_);
  for (int c = t; c < FF; c += NT) store_limbs2(a8, plane, off + c, quant2(silu8_rare(yr[c], yr[FF + c], lut).h, sh, as_, inv));
  if (t == 0) norm24(as_, sh - FR, *mant, *eo);
  group_sync<NT>(group);
}

// Many rows: one 1024-thread CTA per SM with the compact table in shared memory (one asynchronous copy) walks the rows, in
// groups of GT threads with a row and a barrier each, Q groups of four columns per thread. FF % 4 == 0, FF <= 4 GT Q.
template <int GT, int Q>
__global__ void __launch_bounds__(SILU_P_THREADS, 1)
int8_silu_persistent_kernel(const i64* __restrict__ y, const i64* __restrict__ lut, const uint16_t* __restrict__ compact, int8_t* __restrict__ a8,
                            i64* __restrict__ mant, i64* __restrict__ eo, i64* __restrict__ scr, int M, int FF, bool wide) {
  constexpr int GROUPS = SILU_P_THREADS / GT;
  extern __shared__ __align__(16) uint8_t silu_smem[];
  const uint16_t* tab = reinterpret_cast<const uint16_t*>(silu_smem);
  __shared__ i64 red[GROUPS][2][32];
  __shared__ uint64_t table_full;
  const int group = threadIdx.x / GT, t = threadIdx.x % GT;
  int turn = 0;
  if (threadIdx.x == 0) {
    mbar_init(&table_full, 1);
    fence_barrier_init();
  }
  __syncthreads();
  wait_previous();
  launch_next();
  if (threadIdx.x == 0) {
    mbar_arrive_expect_tx(&table_full, SC_BYTES);
    bulk_load(silu_smem, compact, &table_full, SC_BYTES);
  }
  const bool there = mbar_wait(&table_full, 0);
  if (!there && threadIdx.x == 0) atomicAdd(&g_wait_timeouts, 1);
  const int64_t plane = (int64_t)M * FF;
  SiluAcc acc{0u, 0u, 0, 0};
  for (int64_t row = (int64_t)group * gridDim.x + blockIdx.x; row < M; row += (int64_t)GROUPS * gridDim.x) {
    const i64* yr = y + row * (2 * (int64_t)FF);
    double h[Q][4];
    double hmax = 0.0;
    bool big = false;
#pragma unroll
    for (int k = 0; k < Q; ++k) {
      const int c = 4 * (t + k * GT);
#pragma unroll
      for (int j = 0; j < 4; ++j) h[k][j] = 0.0;
      if (c < FF) {
        i64 g[4], u[4];
        load4(yr + c, wide, g);
        load4(yr + FF + c, wide, u);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          h[k][j] = silu8(g[j], u[j], tab, lut, acc, big);
          hmax = fmax(hmax, fabs(h[k][j]));
        }
      }
    }
    if (big) hmax = 1e300;
    const double top = __longlong_as_double(group_max_f64<GT>(hmax, red[group][turn ^= 1], group));
    if (top > 1e299) {                                         // the barrier of the row function frees the other buffer
      group_sync<GT>(group);
      int8_silu_row<GT>(yr, lut, a8, plane, row * FF, mant + row, eo + row, FF, red[group][turn], group);
      continue;
    }
    const QuantRow qr = quant_row(f64_to_int(top + F2I));
#pragma unroll
    for (int k = 0; k < Q; ++k) {
      const int c = 4 * (t + k * GT);
      quant_store4(h[k], qr, a8, plane, row * FF + c, c < FF, wide);
    }
    if (t == 0) norm24(qr.as_, qr.sh - FR, mant[row], eo[row]);
  }
  if (scr) {
    const i64 s = warp_max(imax(acc.rs, (i64)acc.s)), u = warp_max(imax(acc.ru, (i64)acc.u));
    if ((threadIdx.x & 31) == 0) {
      atomicMax(reinterpret_cast<long long*>(scr), (long long)s);
      atomicMax(reinterpret_cast<long long*>(scr + 1), (long long)u);
    }
  }
  if (!there) mbar_wait(&table_full, 0);                       // a copy that is late lands before the CTA ends
}

// Decode batches: the columns of a row over the CTAs of a cluster (256 threads, Q groups of four columns each), the compact
// table read through L1.
template <int Q>
__global__ void __launch_bounds__(SILU_CL_THREADS)
int8_silu_cluster_kernel(const i64* __restrict__ y, const i64* __restrict__ lut, const uint16_t* __restrict__ compact, int8_t* __restrict__ a8,
                         i64* __restrict__ mant, i64* __restrict__ eo, i64* __restrict__ scr, int M, int FF, bool wide) {
  namespace cg = cooperative_groups;
  __shared__ i64 red[32];
  __shared__ i64 cta_max;
  cg::cluster_group cluster = cg::this_cluster();
  const int part = (int)cluster.block_rank(), parts = (int)cluster.num_blocks();
  const int64_t row = blockIdx.x / parts;
  const int per = (FF / 4 + parts - 1) / parts;            // groups of four columns per CTA
  const i64* yr = y + row * (2 * (int64_t)FF);
  double h[Q][4];
  double hmax = 0.0;
  bool big = false;
  SiluAcc acc{0u, 0u, 0, 0};
  wait_previous();
  launch_next();
#pragma unroll
  for (int k = 0; k < Q; ++k) {
    const int own = threadIdx.x + k * SILU_CL_THREADS, c = 4 * (part * per + own);
#pragma unroll
    for (int j = 0; j < 4; ++j) h[k][j] = 0.0;
    if (own < per && c < FF) {
      i64 g[4], u[4];
      load4(yr + c, wide, g);
      load4(yr + FF + c, wide, u);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        h[k][j] = silu8(g[j], u[j], compact, lut, acc, big);
        hmax = fmax(hmax, fabs(h[k][j]));
      }
    }
  }
  if (big) hmax = 1e300;
  const i64 mine = group_max_f64<SILU_CL_THREADS>(hmax, red, 0);
  if (threadIdx.x == 0) cta_max = mine;
  if (scr) {
    const i64 s = warp_max(imax(acc.rs, (i64)acc.s)), u = warp_max(imax(acc.ru, (i64)acc.u));
    if ((threadIdx.x & 31) == 0) {
      atomicMax(reinterpret_cast<long long*>(scr), (long long)s);
      atomicMax(reinterpret_cast<long long*>(scr + 1), (long long)u);
    }
  }
  cluster.sync();
  i64 all = 0;
  for (int r = 0; r < parts; ++r) all = imax(all, *cluster.map_shared_rank(&cta_max, r));
  const double top = __longlong_as_double(all);
  const int64_t plane = (int64_t)M * FF;
  if (top > 1e299) {
    if (part == 0) int8_silu_row<SILU_CL_THREADS>(yr, lut, a8, plane, row * FF, mant + row, eo + row, FF, red, 0);
  } else {
    const QuantRow qr = quant_row(f64_to_int(top + F2I));
#pragma unroll
    for (int k = 0; k < Q; ++k) {
      const int own = threadIdx.x + k * SILU_CL_THREADS, c = 4 * (part * per + own);
      quant_store4(h[k], qr, a8, plane, row * FF + c, own < per && c < FF, wide);
    }
    if (part == 0 && threadIdx.x == 0) norm24(qr.as_, qr.sh - FR, mant[row], eo[row]);
  }
  cluster.sync();                                   // peers may still be reading cta_max
}

// segs.post on a raw int_mm output (src/bitexact/int8/segs.py:62-67): c int32 [R, N] with limb i of row m at row
// i * M + m -> y int64 [M, N]; flag when checked and some |t| >= 2^38.
__global__ void int8_post_kernel(const int32_t* __restrict__ c, const i64* __restrict__ mul, i64 fmsh,
                                 const i64* __restrict__ mant, const i64* __restrict__ e, i64* __restrict__ y,
                                 int32_t* flag, int M, int N, int checked) {
  const int64_t total = (int64_t)M * N;
  bool bad = false;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t m = t / N, n = t % N;
    const i64 acc = (i64)c[t] + shl((i64)c[total + t], 8);
    const i64 tv = rsh_t((i64)((u64)acc * (u64)mul[n]), fmsh);
    bad |= iabs(tv) >= (1ll << 38);
    y[t] = rsh_t((i64)((u64)tv * (u64)mant[m]), 8 - e[m]);
  }
  if (checked && bad) *flag = 1;
}

// segs.post on the joined accumulator acc = c0 + (c1 << 8) as int64 [M, N] (the form the reference's `post` takes).
__global__ void int8_post_acc_kernel(const i64* __restrict__ acc, const i64* __restrict__ mul, i64 fmsh,
                                     const i64* __restrict__ mant, const i64* __restrict__ e, i64* __restrict__ y,
                                     int32_t* flag, int M, int N, int checked) {
  const int64_t total = (int64_t)M * N;
  bool bad = false;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t m = t / N, n = t % N;
    const i64 tv = rsh_t((i64)((u64)acc[t] * (u64)mul[n]), fmsh);
    bad |= iabs(tv) >= (1ll << 38);
    y[t] = rsh_t((i64)((u64)tv * (u64)mant[m]), 8 - e[m]);
  }
  if (checked && bad) *flag = 1;
}

// The same in two steps, for a gate / up projection sharded by output column over several GPUs: step 1 on the
// rank's columns writes h and the row maxima of |h| (and the |silu(g)|, |u| maxima for the bound flag); the caller
// takes the integer maximum of the row maxima over the ranks; step 2 quantises the rank's columns with the scale of
// the FULL row. Same integers as int8_silu_kernel on the full row.
template <int EPT>
__global__ void __launch_bounds__(SILU_THREADS)
int8_silu_prod_kernel(const i64* __restrict__ y, const i64* __restrict__ lut, i64* __restrict__ h,
                      i64* __restrict__ rowmax, i64* __restrict__ scr, int M, int FF) {
  __shared__ i64 red[33];
  const int64_t row = blockIdx.x;
  const i64* yr = y + row * (2 * (int64_t)FF);
  i64 hmax = 0, smax = 0, umax = 0;
#pragma unroll
  for (int k = 0; k < EPT; ++k) {
    const int c = threadIdx.x + k * SILU_THREADS;
    if (c < FF) {
      const i64 sg = silu_tab(yr[c], lut), u = yr[FF + c];
      const i64 hv = rshs<FR>((i64)((u64)sg * (u64)u));
      h[row * FF + c] = hv;
      hmax = imax(hmax, iabs(hv));
      smax = imax(smax, iabs(sg));
      umax = imax(umax, iabs(u));
    }
  }
  hmax = block_reduce<true>(hmax, red);
  smax = block_reduce<true>(smax, red);
  umax = block_reduce<true>(umax, red);
  if (threadIdx.x == 0) {
    rowmax[row] = hmax;
    if (scr) {
      atomicMax(reinterpret_cast<long long*>(scr), (long long)smax);
      atomicMax(reinterpret_cast<long long*>(scr + 1), (long long)umax);
    }
  }
}

// pre_plain of the rows of h [M, K] given the maxima of the full rows: limb planes a8 [2][M][K], mant, e.
__global__ void __launch_bounds__(256)
int8_quant_rows_kernel(const i64* __restrict__ h, const i64* __restrict__ rowmax, int8_t* __restrict__ a8,
                       i64* __restrict__ mant, i64* __restrict__ eo, int M, int K) {
  const int64_t row = blockIdx.x;
  i64 sh, as_;
  quant_scale(rowmax[row], sh, as_);
  const u64 inv = ~0ull / (u64)(2 * as_);
  const int64_t plane = (int64_t)M * K;
  for (int c = threadIdx.x; c < K; c += blockDim.x) store_limbs2(a8, plane, row * K + c, quant2(h[row * K + c], sh, as_, inv));
  if (threadIdx.x == 0 && mant) norm24(as_, sh - FR, mant[row], eo[row]);
}

// flag |= any layer's max|silu(g)| * max|u| >= 2^62 (int64 product, wrapping like the reference's), then reset
// (tri_fuse._flag_kernel, src/bitexact/vllm_plugin/tri_fuse.py:248-265).
__global__ void int8_flag_end_kernel(i64* scr, int32_t* flag, int L) {
  for (int i = threadIdx.x; i < L; i += blockDim.x) {
    const i64 s = scr[2 * i], u = scr[2 * i + 1];
    if ((i64)((u64)s * (u64)u) >= (1ll << 62)) *flag = 1;
    scr[2 * i] = 0;
    scr[2 * i + 1] = 0;
  }
}

}  // namespace i8
}  // namespace bx
