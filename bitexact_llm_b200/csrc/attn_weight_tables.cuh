// Attention weights from a shared-memory copy of the weight table.
//
// A weight needs two neighbouring 64-bit entries of the 2^-f table (exact rule, 131 KB) or one 32-bit entry of the
// e^z table (int8 rule, 524 KB). Neither fits L1 beside the staged keys, and 32 lanes gather from up to 32 lines: the
// kernels that read the tables through L1 spent most of their time waiting for those gathers. Here a CTA keeps a
// compact copy in shared memory, made from whatever table the caller gave:
//
//   exact rule   the top 31 bits of the entries (65 KB). The interpolated value is known to within two units of
//                2^29, hence the rounded 22-bit weight is known unless a rounding boundary lies between; only those
//                (one in 2^(8 + n) for a weight of 2^-n) are recomputed from the full table.
//   int8 rule    the entries within 8 of the maximum, as 16 low bits and, where a weight can exceed 65535, 8 high
//                bits (83 KB). Entries further down are read from the table itself.
//
// Both forms are checked while they are copied (range, and the steps between neighbours that the 32-bit interpolation
// assumes). A table that does not fit them, or a row whose shift does not, takes the general function for every weight:
// same integers for any table.
#pragma once

#include "bx_ptx.cuh"
#include "bx_rules.cuh"

namespace bx {

constexpr int WT_EXP2_N = (1 << EXP2_BITS) + 1;
constexpr int WT_EXP2_BYTES = (WT_EXP2_N * 4 + 127) / 128 * 128;       // 65664
constexpr int WT_NEAR = 32768, WT_HIGH = 17408;                        // 8 and 4.25 below the maximum in steps of 2^-12
constexpr int WT_INT8_BYTES = WT_NEAR * 2 + WT_HIGH;                   // 82944
constexpr int WT_PTAB_LAST = 131072;                                   // entry of z = 0

// Copies the table into `tab`; `tid` of `n` threads. Returns false where this thread saw an entry that does not fit.
__device__ __forceinline__ bool fill_exp2_table(uint8_t* tab, const i64* __restrict__ lut, int tid, int n) {
  uint32_t* t = reinterpret_cast<uint32_t*>(tab);
  bool ok = true;
  for (int i = tid; i < WT_EXP2_N; i += n) {
    const i64 v = __ldg(lut + i);
    ok &= v >= 0 && v <= (1ll << EXP2_ONE);
    t[i] = (uint32_t)((u64)v >> 29);
  }
  return ok;
}
// Second half of the check, after a barrier: neighbours differ by less than 2^19, so the product with a 12-bit
// remainder stays in 31 bits.
__device__ __forceinline__ bool check_exp2_table(const uint8_t* tab, int tid, int n) {
  const uint32_t* t = reinterpret_cast<const uint32_t*>(tab);
  bool ok = true;
  for (int i = tid; i < WT_EXP2_N - 1; i += n) {
    const int d = (int)(t[i + 1] - t[i]);
    ok &= d < (1 << 19) && d > -(1 << 19);
  }
  return ok;
}
__device__ __forceinline__ bool fill_int8_table(uint8_t* tab, const int32_t* __restrict__ ptab, int tid, int n) {
  uint16_t* lo = reinterpret_cast<uint16_t*>(tab);
  uint8_t* hi = tab + WT_NEAR * 2;
  bool ok = true;
  for (int u = tid; u < WT_NEAR; u += n) {
    const uint32_t v = (uint32_t)__ldg(ptab + (WT_PTAB_LAST - u));
    lo[u] = (uint16_t)v;
    if (u < WT_HIGH) {
      hi[u] = (uint8_t)(v >> 16);
      ok &= v < (1u << 24);
    } else {
      ok &= v < (1u << 16);
    }
  }
  return ok;
}

// The exact rule's weight of a key at zz = (row maximum - score) + 2^(c - 1), for a row shift of c = 1 .. 31 bits and
// 2^28 <= l2e < 2^29: zf = zz >> c; from zf = 2^31 on the weight is 0 (t >= 32 at 26 bits), below it t fits 32 bits.
// With a 31-bit table w = a + ((b - a) rr >> 12) the full value lies in [w, w + 2] 2^29, and rounding is monotone:
// where both ends round to the same weight that is the weight, else `unsure` is set.
__device__ __forceinline__ uint32_t exp2_weight(i64 zz, int c, uint32_t l2e, bool live, const uint8_t* tab, bool& unsure) {
  const uint32_t lo = (uint32_t)zz, hi = (uint32_t)((u64)zz >> 32);
  const uint32_t zf = __funnelshift_r(lo, hi, c);
  const u64 tt = (u64)zf * l2e + (1ull << (FZ + 28 - FT2 - 1));
  uint32_t t = __funnelshift_r((uint32_t)tt, (uint32_t)(tt >> 32), FZ + 28 - FT2);
  t = (live && (hi >> (c - 1)) == 0) ? t : 0xffffffffu;              // n = 63: weight 0
  const uint32_t* e = reinterpret_cast<const uint32_t*>(tab + ((t >> (FT2 - EXP2_BITS - 2)) & (((1 << EXP2_BITS) - 1) << 2)));
  const int rr = (int)(t & ((1u << (FT2 - EXP2_BITS)) - 1));
  const uint32_t a = e[0];
  const uint32_t w = a + (uint32_t)(((int)(e[1] - a) * rr) >> (FT2 - EXP2_BITS));
  const uint32_t s = (t >> FT2) + (EXP2_ONE - FP - 29 - 1);
  const uint32_t r0 = (shr_clamp(w, s) + 1) >> 1, r1 = (shr_clamp(w + 2, s) + 1) >> 1;
  unsure = r0 != r1;
  return r0;
}

// The int8 rule's weight of a key at zz = (row maximum - score) + 2^18 - 1: u = zz >> 19 table steps below the maximum
// (= -((score - maximum + 2^18) >> 19)).
constexpr int WT_INT8_SHIFT = 2 * 14 + 3 - 12;
__device__ __forceinline__ uint32_t int8_weight(i64 zz, bool live, const uint8_t* tab, const int32_t* __restrict__ ptab) {
  const uint32_t lo = (uint32_t)zz, hi = (uint32_t)((u64)zz >> 32);
  uint32_t u = __funnelshift_r(lo, hi, WT_INT8_SHIFT);
  u = (live && (hi >> (WT_INT8_SHIFT - 1)) == 0) ? u : 0xffffffffu;
  uint32_t v = 0;
  if (u < (uint32_t)WT_NEAR) {
    v = reinterpret_cast<const uint16_t*>(tab)[u];
    if (u < (uint32_t)WT_HIGH) v |= (uint32_t)tab[WT_NEAR * 2 + u] << 16;
  } else if (u <= (uint32_t)WT_PTAB_LAST) {
    v = (uint32_t)__ldg(ptab + (WT_PTAB_LAST - (int)u));
  }
  return v;
}

// The decode kernels' form: 4097 entries (16 KB; two CTAs share an SM, four with block tables of up to 64 keys) prepared by the caller from its table, with
// what that form cannot say (bitexact_llm_b200/attn_table.py works both out over all entries of the full table). The
// weight at t = factor (zz >> c) lies in [w, w + window] mtop 2^-n of the interpolated entry w, give or take `slack`, all
// in units of 2^-32; `unsure` where a rounding boundary lies in that range.
// Cost in cycles of a scheduler, measured: a gather from the 131 KB table 32 and an L2 round trip, the whole of this about
// 45, of which the two 32-bit gathers from shared memory take 14.
struct CompactTable {
  const uint32_t* tab;          // null: none
  const double* products;       // attn_weight_products.cuh, in place of tab (null: none)
  uint32_t window, slack, factor, mtop;
  int shift;
};
constexpr int CT_N = 4097;
constexpr int CT_BYTES = 16400;

// One thread asks for the table; it is complete when the phase of `bar` is (16-byte aligned ct.tab and dst). The copy runs
// behind the scores of the first pair. Copied by all threads in front of them instead, it held up batches of short
// contexts: 64 sequences of up to 64 keys 18 : 22.5 us.
__device__ __forceinline__ void fetch_compact(uint32_t* dst, const CompactTable& ct, uint64_t* bar) {
  mbar_arrive_expect_tx(bar, (CT_N - 1) * 4);
  bulk_load(dst, ct.tab, bar, (CT_N - 1) * 4);
  dst[CT_N - 1] = __ldg(ct.tab + CT_N - 1);
}
// hs: a distance with hi >> hs != 0 is out of range (weight 0).
__device__ __forceinline__ uint32_t compact_weight(const CompactTable& ct, const uint32_t* tab, i64 zz, int c, int hs, bool live,
                                                   bool& unsure) {
  const uint32_t lo = (uint32_t)zz, hi = (uint32_t)((u64)zz >> 32);
  const uint32_t zf = __funnelshift_r(lo, hi, c) << ct.shift;
  const uint32_t t = (uint32_t)(((u64)zf * ct.factor + (1ull << 31)) >> 32);
  const uint32_t n = (t >> FT2) + (hi >> hs) * 32u;
  const uint32_t* e = reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint8_t*>(tab) + ((t >> 12) & 0x3ffcu));
  const uint32_t a = e[0];
  const uint32_t w = a - __umulhi(a - e[1], t << 18);
  const uint32_t m = live ? shr_clamp(ct.mtop, n) : 0u;
  const u64 r = (u64)w * m + ((1ull << 31) - ct.slack);
  const uint32_t rl = (uint32_t)r;
  unsure = live && rl + (m * ct.window + 2u * ct.slack) < rl;
  return (uint32_t)(r >> 32);
}

}  // namespace bx
