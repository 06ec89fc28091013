// Attention weights from products of doubles.
//
// Both weight tables are exponentials, so an entry is the product of two of 128 (exact rule: 2^-f in steps of 2^-7 and 2^-14) or of
// 512 and 256 (int8 rule: e^z in steps of 2^-4 and 2^-12) doubles in shared memory, 2 and 6 KB for 131 and 524, and a weight
// is known to 2^-27 (exact rule) or to the 2^-11 that its table was rounded by before (int8 rule). From 2^-22 below a rounding boundary
// to 2^-21 above it (exact rule), or within 2^-9 of it (int8 rule), the table itself decides. A table is known to be of this kind
// because every entry was held against the products: by the caller that prepared them (attn_table.py, the kernels that give a pair to
// a CTA or a cluster), or by the first kernel of the split decode attention, a slice per CTA. A table of another kind takes the general
// rule.
// Measured in the second kernel of the split attention, 32 sequences of 64 .. 8192 keys: 85 us with the 4097 entries of
// attn_weight_tables.cuh, which leave 1 % of the weights near the maximum undecided (most warps then gather from L2), 66 us so.
#pragma once

#include "attn_weight_tables.cuh"
#include "stage_math.cuh"

namespace bx {

constexpr int PW_EXACT = 128, PW_INT8 = 512, PW_DOUBLES = 768;
constexpr int PW_LAST = 131072;                                        // int8 rule: entry of z = 0

struct ProductTable {
  const double* t;      // shared memory: exact 2^-(i / 128), 2^-(i / 16384); int8 ptab[last] e^-(i / 16), e^-(i / 4096)
  double slope;         // exact: (2^-(1 / 16384) - 1) / 4096
};
__device__ __forceinline__ double exp2_entry(const i64* lut, int i) { return (double)__ldg(lut + i) * 8.673617379884035e-19; }      // 2^-60
__device__ __forceinline__ void load_products(const i64* lut, const int32_t* ptab, ProductTable& pt, double* t, int tid, int n) {
  pt.t = t;
  pt.slope = 0.0;
  if (ptab) {
    const double top = (double)__ldg(ptab + PW_LAST);
    for (int i = tid; i < PW_INT8 + 256; i += n) t[i] = i < PW_INT8 ? top * exp(-i / 16.0) : exp(-(i - PW_INT8) / 4096.0);
  } else {
    for (int i = tid; i < 2 * PW_EXACT; i += n) t[i] = exp2_entry(lut, i < PW_EXACT ? i * PW_EXACT : i - PW_EXACT);
    pt.slope = (exp2_entry(lut, 1) - 1.0) * (1.0 / 4096);
  }
}
// The same of the exact rule from a caller's copy that says whether it has found them to be its table's (bitexact_llm_b200/attn_table.py):
// the slope behind them, and in front of them a word that is 1 where they are; otherwise pt.t is null.
__device__ __forceinline__ void copy_products(const double* src, ProductTable& pt, double* t, int tid, int n) {
  for (int i = tid; i < 2 * PW_EXACT; i += n) t[i] = __ldg(src + i);
  pt.t = __ldg(reinterpret_cast<const int*>(src) - 1) == 1 ? t : nullptr;
  pt.slope = __ldg(src + 2 * PW_EXACT);
}
constexpr int PW_EXACT_BYTES = 8 * 2 * PW_EXACT;
// Entries [part of parts) of the caller's table against the products.
__device__ __forceinline__ bool check_products(const i64* lut, const int32_t* ptab, i64 l2e, const double* t, int part, int parts, int tid,
                                               int n) {
  bool ok = true;
  if (ptab) {
#pragma unroll 4
    for (int i = part * n + tid; i <= PW_LAST; i += parts * n) {
      const int v = __ldg(ptab + (PW_LAST - i));
      const double w = i < PW_LAST ? t[i >> 8] * t[PW_INT8 + (i & 255)] : 0.0;
      ok &= v >= 0 && v <= (1 << 22) && fabs((double)v - w) <= 0.50048828125;              // 1/2 + 2^-11
    }
  } else {
    for (int i = part * n + tid; i <= 1 << EXP2_BITS; i += parts * n) {
      const double w = i < 1 << EXP2_BITS ? t[i >> 7] * t[PW_EXACT + (i & 127)] : 0.5;
      ok &= fabs(exp2_entry(lut, i) - w) <= 8.881784197001252e-16;                       // 2^-50
    }
    ok &= t[0] == 1.0 && l2e >= (1ll << 28) && l2e < (1ll << 29);
  }
  return ok;
}
// The weight floor(v scale + 1/2), `unsure` about a boundary.
template <bool EXACT>
__device__ __forceinline__ uint32_t round_weight(double v, double scale, bool& unsure) {
  const double t = __fma_rd(v, scale, F2I);
  const int dh = __double2hiint(fma(v, scale, F2I - t));               // 0x3fe00000: one half
  unsure = EXACT ? (uint32_t)(dh - 0x3fdfffff) <= 1u : (uint32_t)(dh - 0x3fdfe000) < 0x3000u;
  return (uint32_t)__double2loint(t) + (dh >= 0x3fe00000 ? 1u : 0u);
}
// zz = (row maximum - score) + the rounding term of the shift, as exp2_weight and int8_weight take it.
__device__ __forceinline__ uint32_t product_weight(const ProductTable& pt, uint32_t l2e, i64 zz, int c, bool live, bool& unsure) {
  const uint32_t lo = (uint32_t)zz, hi = (uint32_t)((u64)zz >> 32);
  const u64 tt = (u64)__funnelshift_r(lo, hi, c) * l2e + (1ull << (FZ + 28 - FT2 - 1));
  const uint32_t t = __funnelshift_r((uint32_t)tt, (uint32_t)(tt >> 32), FZ + 28 - FT2);
  const double v = pt.t[(t >> 19) & 127] * pt.t[PW_EXACT + ((t >> 12) & 127)];
  const uint32_t w = round_weight<true>(fma(v, pt.slope * u32_to_f64(t & 4095), v), pow2_f64(FP - (int)(t >> FT2)), unsure);
  const bool on = live && (hi >> (c - 1)) == 0;                        // from 2^31 on: 0
  unsure &= on;
  return on ? w : 0u;
}
__device__ __forceinline__ uint32_t product_weight8(const ProductTable& pt, i64 zz, bool live, bool& unsure) {
  const uint32_t lo = (uint32_t)zz, hi = (uint32_t)((u64)zz >> 32);
  const uint32_t u = __funnelshift_r(lo, hi, WT_INT8_SHIFT);
  const bool on = live && (hi >> (WT_INT8_SHIFT - 1)) == 0 && u < (uint32_t)PW_LAST;     // the table's last entry is 0
  const uint32_t w = round_weight<false>(pt.t[(u >> 8) & (PW_INT8 - 1)], pt.t[PW_INT8 + (u & 255)], unsure);
  unsure &= on;
  return on ? w : 0u;
}

}  // namespace bx
