// Integer rules of the row-local stages in double precision.
//
// The stages are bound by instruction issue, and 64-bit integer products and shifts are the dearest instructions they
// have (cycles of a scheduler per warp, measured: mul.hi.u64 17.6, mad.lo.s64 8.7, a 64-bit compare 8, div.u64 151),
// while an fma.f64 takes 2. Values below 2^51 are exact as doubles, a product of two doubles is exact as a rounded
// product and its fma remainder, and floor(v) is one addition of 1.5 2^52 that rounds down. So a quotient is known to
// far better than the distance to the rounding boundary in all but a few cases in 10^6; those, and values out of these
// ranges, take the integer rule itself. Nothing here changes a bit: the tests hold every form to the oracle.
#pragma once

#include "bx_ptx.cuh"
#include "bx_rules.cuh"

namespace bx {

constexpr double F2I = 6755399441055744.0;            // 1.5 2^52: v + F2I has the integer v in its low mantissa bits
constexpr int F2I_HI = 0x43380000;                    // its high word (the low word is 0)

// |x| < 2^51, exact.
__device__ __forceinline__ double to_f64(i64 x) {
  return __hiloint2double((int)(x >> 32) + F2I_HI, (int)x) - F2I;
}
__device__ __forceinline__ bool in_f64(i64 x) { return ((uint32_t)((int)(x >> 32) + 0x80000) >> 20) == 0; }
// The integer v of t = v + F2I.
__device__ __forceinline__ i64 f64_to_int(double t) {
  return ((i64)(__double2hiint(t) - F2I_HI) << 32) | (u64)(uint32_t)__double2loint(t);
}
__device__ __forceinline__ double u32_to_f64(uint32_t x) { return __hiloint2double(0x43300000, (int)x) - 4503599627370496.0; }
__device__ __forceinline__ double s32_to_f64(int x) { return __hiloint2double(0x43300000, x ^ (int)0x80000000) - 4503601774854144.0; }
// 2^e, -1022 <= e <= 1023.
__device__ __forceinline__ double pow2_f64(int e) { return __hiloint2double((1023 + e) << 20, 0); }
// Bit length of the largest |v| from the largest high word of |v| as a double (0 for 0).
__device__ __forceinline__ int f64_bits(uint32_t hi) { return hi ? (int)(hi >> 20) - 1022 : 0; }

__device__ __forceinline__ double rcp_f64_rough(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  return r;
}

// ---- four consecutive entries of a row ----
// wide: the addresses are multiples of what is moved (the host looks at every pointer and pitch).
__device__ __forceinline__ void load4(const i64* p, bool wide, i64 (&v)[4]) {
  if (wide) {
    asm volatile("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3]) : "l"(p));
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = p[j];
  }
}
__device__ __forceinline__ void store4(i64* p, bool wide, const i64 (&v)[4]) {
  if (wide) {
    st_global_v4(p, v[0], v[1], v[2], v[3]);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) p[j] = v[j];
  }
}
// q and its limb planes.
__device__ __forceinline__ void store_q4(int32_t* q, int8_t* a8, int64_t plane, int64_t off, bool wide, const int (&v)[4]) {
  if (!wide) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      q[off + j] = v[j];
      if (a8) {
        const uint32_t b = limb_bytes((uint32_t)v[j]);
#pragma unroll
        for (int i = 0; i < 3; ++i) a8[i * plane + off + j] = (int8_t)(b >> (8 * i));
      }
    }
    return;
  }
  *reinterpret_cast<int4*>(q + off) = make_int4(v[0], v[1], v[2], v[3]);
  if (a8) {
    const uint32_t b0 = limb_bytes((uint32_t)v[0]), b1 = limb_bytes((uint32_t)v[1]), b2 = limb_bytes((uint32_t)v[2]),
                   b3 = limb_bytes((uint32_t)v[3]);
    const uint32_t l01 = __byte_perm(b0, b1, 0x5140), l23 = __byte_perm(b2, b3, 0x5140);     // limbs 0 0 1 1 of a pair
    *reinterpret_cast<uint32_t*>(a8 + off) = __byte_perm(l01, l23, 0x5410);
    *reinterpret_cast<uint32_t*>(a8 + plane + off) = __byte_perm(l01, l23, 0x7632);
    *reinterpret_cast<uint32_t*>(a8 + 2 * plane + off) = __byte_perm(__byte_perm(b0, b1, 0x0062), __byte_perm(b2, b3, 0x0062), 0x5410);
  }
}

// ---- reductions over a group of NT threads (whole warps; barrier 1 + group) ----
// One barrier each; `buf` (32 words) is free again once another barrier of the group has been passed.
template <int NT>
__device__ __forceinline__ void group_sync(int group) {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(NT) : "memory");
}
template <int NT>
__device__ __forceinline__ uint32_t group_max(uint32_t v, uint32_t* buf, int group) {
  const int lane = threadIdx.x & 31, warp = (threadIdx.x % NT) >> 5;
  v = __reduce_max_sync(0xffffffffu, v);
  if (lane == 0) buf[warp] = v;
  group_sync<NT>(group);
  return __reduce_max_sync(0xffffffffu, lane < NT / 32 ? buf[lane] : 0u);
}
template <int NT>
__device__ __forceinline__ i64 group_or(i64 v, i64* buf, int group) {
  const int lane = threadIdx.x & 31, warp = (threadIdx.x % NT) >> 5;
  uint32_t lo = __reduce_or_sync(0xffffffffu, (uint32_t)v), hi = __reduce_or_sync(0xffffffffu, (uint32_t)((u64)v >> 32));
  if (lane == 0) buf[warp] = (i64)(((u64)hi << 32) | lo);
  group_sync<NT>(group);
  const i64 w = lane < NT / 32 ? buf[lane] : 0;
  lo = __reduce_or_sync(0xffffffffu, (uint32_t)w);
  hi = __reduce_or_sync(0xffffffffu, (uint32_t)((u64)w >> 32));
  return (i64)(((u64)hi << 32) | lo);
}
// Sum of 0 <= v < 2^57.
template <int NT>
__device__ __forceinline__ i64 group_sum(i64 v, i64* buf, int group) {
  const int lane = threadIdx.x & 31, warp = (threadIdx.x % NT) >> 5;
  auto warp_total = [](i64 x) -> i64 {                 // 26 bits at a time
    const u64 a = __reduce_add_sync(0xffffffffu, (uint32_t)x & 0x3ffffffu), b = __reduce_add_sync(0xffffffffu, (uint32_t)(x >> 26) & 0x3ffffffu);
    const u64 c = __reduce_add_sync(0xffffffffu, (uint32_t)(x >> 52));
    return (i64)(a + (b << 26) + (c << 52));
  };
  v = warp_total(v);
  if (lane == 0) buf[warp] = v;
  group_sync<NT>(group);
  return warp_total(lane < NT / 32 ? buf[lane] : 0);
}

}  // namespace bx
