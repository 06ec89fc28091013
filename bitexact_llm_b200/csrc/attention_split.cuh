// Decode attention split evenly over the chip, whatever the number and the lengths of the sequences: two kernels.
//
// The 64-key units of all (request, KV head) pairs lie in one line, request by request and head by head, and CTA b of G takes
// the units [T b / G, T (b + 1) / G): every SM streams the same number of keys, where a kernel that gives a pair to a CTA
// (or a cluster) waits for the longest pair. What lies between the two sweeps of a pair that several CTAs share is only
// its row maxima:
//
//   attention_scores_kernel   K limbs through a TMA ring, exact scores (int64) into scratch (32 bytes a key beside its 384; in L2
//                             up to about 3 million keys over all pairs, beyond that written to and read from HBM: 72 sequences
//                             of 8000 .. 8192 keys, 4.8 million, 384 us against 393 of the streaming kernel), the maxima of every
//                             piece (CTA x pair, index pair + CTA).
//   attention_values_kernel   maxima of the pair from its pieces, weights, p V on tcgen05 with the accumulators in TMEM over all
//                             keys of the piece; a piece that is a whole pair is stored, others are added to num and den, which the
//                             first kernel has cleared. Integer sums: any order gives the same bits.
//
// The arithmetic is that of the kernels in paged_attention.cuh.
#pragma once

#include "paged_attention.cuh"

namespace bx {

constexpr int SPL_KEYS = 64;                     // keys per unit and per stage
constexpr int SPL_WARPS = 8;                     // warps that compute
constexpr int SPL_K_STAGE = SPL_KEYS * ATT2_HALF, SPL_V_STAGE = SPL_KEYS * 256;
constexpr int SPL_K_STAGES = 8, SPL_V_STAGES = 5;
constexpr int SPL_WAVE = 8;                      // 32-key groups whose weights are made together, one per warp
constexpr int SPL_PTILE = 512;                   // weight limbs of a group: [16 rows = (limb, query)] x [32 keys]
constexpr int SPL_MAXREQ = 512;
constexpr int SPL_MAXPAGES = 1024;               // pages of a CTA's units
constexpr int SPL_TMEM = 64;                     // two pieces' accumulators of 32 columns

struct SplitParams {
  AttnParams a;
  i64* scores;          // [units][64 keys][4]
  i64* pmax;            // [pairs + CTAs][4]
  int* fits;            // [CTAs] the CTA's slice of the weight table is what the products say
  int nreq;
};

// A walk over the pieces of units [x, end): the part of pair (r, h) from unit u on, `count` units.
struct SplitWalk {
  const int* start;     // [nreq + 1] units of one head before request r
  int HKV, nreq, x, end;
  int r, h, u, n, count;
  __device__ __forceinline__ void begin(const int* s, int heads, int req, int from, int to) {
    start = s;
    HKV = heads;
    nreq = req;
    x = from;
    end = to;
    count = 0;
    if (x >= end) return;
    int lo = 0, hi = nreq;                       // the last request that starts at or before x
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (start[mid] * HKV <= x) lo = mid; else hi = mid;
    }
    r = lo;
    n = start[r + 1] - start[r];
    const int in = x - start[r] * HKV;
    h = in / n;
    u = in % n;
    count = min(n - u, end - x);
  }
  __device__ __forceinline__ bool more() const { return x < end; }
  __device__ __forceinline__ void next() {
    x += count;
    u = 0;
    if (x >= end) return;
    if (++h == HKV) {
      h = 0;
      do ++r; while (start[r + 1] == start[r]);
      n = start[r + 1] - start[r];
    }
    count = min(n, end - x);
  }
};

// Keys of request t as everywhere: up to its last query's position.
__device__ __forceinline__ i64 split_keys(const AttnParams& p, int t) {
  i64 kend = 0;
  for (int g = 0; g < p.M; ++g) kend = imax(kend, p.qpos[(int64_t)t * p.M + g] + 1);
  return imin(imax(kend, 0), (i64)p.nblk * p.bs);
}
// start[0 .. nreq] and keys[0 .. nreq), by all threads.
__device__ __forceinline__ void split_starts(const AttnParams& p, int nreq, int* start, int* keys) {
  for (int t = threadIdx.x; t < nreq; t += blockDim.x) {
    keys[t] = (int)split_keys(p, t);
    start[t + 1] = (keys[t] + SPL_KEYS - 1) / SPL_KEYS;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int run = 0;
    for (int t0 = 0; t0 < nreq; t0 += 32) {
      int v = t0 + lane < nreq ? start[t0 + lane + 1] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int w = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += w;
      }
      if (t0 + lane < nreq) start[t0 + lane + 1] = run + v;
      run += __shfl_sync(0xffffffffu, v, 31);
    }
    if (lane == 0) start[0] = 0;
  }
  __syncthreads();
}
// The first unit of CTA b, and the CTA that has unit x. No more CTAs take part than there are units, so that every CTA between
// the first and the last of a pair has a piece of it.
__device__ __forceinline__ int split_ctas(int units) { return min((int)gridDim.x, units); }
// Whether v holds in all threads of the warps that compute.
__device__ __forceinline__ bool split_and(bool v) {
  int all;
  asm volatile(
      "{\n\t.reg .pred a, b;\n\tsetp.ne.u32 a, %1, 0;\n\tbarrier.cta.red.and.pred b, 1, %2, a;\n\tselp.u32 %0, 1, 0, b;\n\t}"
      : "=r"(all)
      : "r"((int)v), "n"(32 * SPL_WARPS)
      : "memory");
  return all != 0;
}
__device__ __forceinline__ int split_bound(int units, int b) {
  const int ctas = split_ctas(units);
  return b >= ctas ? units : (int)((int64_t)units * b / ctas);
}
__device__ __forceinline__ int split_owner(int units, int x) { return (int)((((int64_t)x + 1) * split_ctas(units) - 1) / units); }

// The page numbers of the CTA's units, pages per unit each (-1 beyond the context), by all threads at once: one at a time, the
// producer warp would wait for each piece's.
__device__ __forceinline__ void split_pages(const AttnParams& p, int nreq, const int* start, const int* keys, int from, int to, int* list) {
  const int per = SPL_KEYS / p.bs;
  for (int i = threadIdx.x; i < (to - from) * per; i += blockDim.x) {
    SplitWalk v;
    v.begin(start, p.HKV, nreq, from + i / per, to);
    const int rel = v.u * per + i % per;
    int page = -1;
    if (rel * p.bs < keys[v.r]) {
      const i64 brow = p.rmap ? p.rmap[v.r] : v.r;
      page = p.bt64 ? (int)reinterpret_cast<const i64*>(p.bt)[brow * p.sbt + rel] : reinterpret_cast<const int32_t*>(p.bt)[brow * p.sbt + rel];
    }
    list[i] = page;
  }
  __syncthreads();
}

// The producer warp: the pages of every unit of the CTA's pieces into the ring, VALUES ? two boxes [V0|V1], [V1|V2] : one box of K
// limbs.
template <bool VALUES, int NS, class Small>
__device__ __forceinline__ void split_produce(const CUtensorMap& tmap, const AttnParams& p, SplitWalk w, uint8_t* ring, Small* sm, const int* list,
                                              int lane) {
  const int pages = SPL_KEYS / p.bs;
  volatile uint32_t* abort_flag = &sm->abort_flag;
  bool ok = true;
  int slot = 0, round = 0, issued = 0;
  for (; w.more() && ok; w.next()) {
    for (int u = 0; u < w.count && ok; ++u, list += pages) {
      const int page = lane < pages ? list[lane] : -1;
      const int live = __popc(__ballot_sync(0xffffffffu, page >= 0));
      if (round > 0) ok = mbar_wait(&sm->empty[slot], (round - 1) & 1);
      ok = __all_sync(0xffffffffu, ok && *abort_flag == 0);
      if (!ok) break;
      if (lane == 0) mbar_arrive_expect_tx(&sm->full[slot], (uint32_t)(live * p.bs * (VALUES ? 256 : ATT2_HALF)));
      __syncwarp();
      if (page >= 0) {
        if (!VALUES) {
          tma_load_4d(ring + slot * SPL_K_STAGE + lane * p.bs * ATT2_HALF, &tmap, &sm->full[slot], 0, 0, w.h, page);
        } else {
          uint8_t* st = ring + slot * SPL_V_STAGE + lane * p.bs * 128;
          tma_load_4d(st, &tmap, &sm->full[slot], 192, 0, w.h, page);
          tma_load_4d(st + SPL_KEYS * 128, &tmap, &sm->full[slot], 256, 0, w.h, page);
        }
      }
      if (issued < NS) ++issued;
      if (++slot == NS) { slot = 0; ++round; }
    }
  }
  if (!ok && lane == 0) { atomicAdd(&g_wait_timeouts, 1); sm->abort_flag = 1; }
  for (int i = 0; i < issued; ++i) {                                   // whatever happened elsewhere: copies in flight land before the exit
    if (--slot < 0) { slot = NS - 1; --round; }
    mbar_wait(&sm->full[slot], round & 1);
  }
}

struct SplitScoresSmall {
  uint64_t full[SPL_K_STAGES], empty[SPL_K_STAGES];
  i64 wmax[2][SPL_WARPS][4];
  uint32_t abort_flag;
  int start[SPL_MAXREQ + 1], keys[SPL_MAXREQ];
  double products[PW_DOUBLES];
};
__host__ __device__ constexpr int split_scores_smem(int pages) { return SPL_K_STAGES * SPL_K_STAGE + (int)sizeof(SplitScoresSmall) + 4 * pages + 128; }

__global__ void __launch_bounds__(32 * (SPL_WARPS + 1), 2)
attention_scores_kernel(const __grid_constant__ CUtensorMap tmap_k, const SplitParams sp) {
  extern __shared__ __align__(128) uint8_t att_smem[];
  const AttnParams& p = sp.a;
  uint8_t* ring = att_smem;
  SplitScoresSmall* sm = reinterpret_cast<SplitScoresSmall*>(ring + SPL_K_STAGES * SPL_K_STAGE);
  int* list = reinterpret_cast<int*>(sm + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < SPL_K_STAGES; ++s) {
      mbar_init(&sm->full[s], 1);
      mbar_init(&sm->empty[s], SPL_WARPS);
    }
    sm->abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmap_k);
  }
  wait_previous();
  launch_next();                                   // attention_values_kernel: its CTAs come as these end, and ask for V meanwhile
  split_starts(p, sp.nreq, sm->start, sm->keys);
  const int units = sm->start[sp.nreq] * p.HKV, from = split_bound(units, blockIdx.x), to = split_bound(units, blockIdx.x + 1);
  split_pages(p, sp.nreq, sm->start, sm->keys, from, to, list);
  SplitWalk w;
  w.begin(sm->start, p.HKV, sp.nreq, from, to);

  if (warp == SPL_WARPS) {
    split_produce<false, SPL_K_STAGES>(tmap_k, p, w, ring, sm, list, lane);
    return;
  }
  // num and den of every pair, for the pieces that are added up
  const int64_t rows = (int64_t)sp.nreq * p.HKV * p.M;
  for (int64_t i = blockIdx.x * (int64_t)(32 * SPL_WARPS) + threadIdx.x; i < rows * (ATT_HD / 2); i += (int64_t)gridDim.x * (32 * SPL_WARPS))
    reinterpret_cast<longlong2*>(p.num)[i] = make_longlong2(0, 0);
  for (int64_t i = blockIdx.x * (int64_t)(32 * SPL_WARPS) + threadIdx.x; i < rows; i += (int64_t)gridDim.x * (32 * SPL_WARPS)) p.den[i] = 0;

  {
    ProductTable pt;
    load_products(p.lut, p.ptab, pt, sm->products, threadIdx.x, 32 * SPL_WARPS);
    asm volatile("bar.sync 1, %0;" ::"n"(32 * SPL_WARPS) : "memory");
    const bool fits = check_products(p.lut, p.ptab, p.l2e, pt.t, blockIdx.x, gridDim.x, threadIdx.x, 32 * SPL_WARPS);
    const bool all = split_and(fits);
    if (threadIdx.x == 0) sp.fits[blockIdx.x] = all;
  }
  volatile uint32_t* abort_flag = &sm->abort_flag;
  bool ok = true;
  int slot = 0, phase = 0, turn = 0;
  const int g = (lane >> 2) & 3;                                       // this lane's query
  // the queries of a piece: 4 x 16 bytes of this lane's row, and its last visible key
  struct Query {
    int4 v[4];
    int qp;
  };
  auto load_query = [&](const SplitWalk& v, Query& q) {
    const int64_t pz = (int64_t)v.r * p.HKV + v.h;
    const bool on = v.more() && g < p.M;
    const int4* row = reinterpret_cast<const int4*>(p.q + (pz * p.M + g) * ATT_HD) + 4 * (lane & 3);
#pragma unroll
    for (int i = 0; i < 4; ++i) q.v[i] = on ? row[i] : make_int4(0, 0, 0, 0);
    q.qp = on ? (int)imin(p.qpos[(int64_t)v.r * p.M + g], (i64)0x7fffffff) : -1;
  };
  Query q;
  load_query(w, q);
  while (w.more()) {
    const int64_t pz = (int64_t)w.r * p.HKV + w.h;
    SplitWalk after = w;
    after.next();
    uint32_t afrag[2][4];
    {
      const int row_lo = lane >> 2, limb_lo = row_lo >> 2;             // limb 0 or 1; rows 8 .. 11 hold limb 2
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int4 qv = q.v[2 * t + half];
          const uint32_t b0 = limb_bytes((uint32_t)qv.x), b1 = limb_bytes((uint32_t)qv.y), b2 = limb_bytes((uint32_t)qv.z),
                         b3 = limb_bytes((uint32_t)qv.w);
          const uint32_t sel = limb_lo ? 0x0051u : 0x0040u;
          afrag[t][2 * half] = __byte_perm(__byte_perm(b0, b1, sel), __byte_perm(b2, b3, sel), 0x5410);
          afrag[t][2 * half + 1] = row_lo < 4 ? __byte_perm(__byte_perm(b0, b1, 0x0062), __byte_perm(b2, b3, 0x0062), 0x5410) : 0u;
        }
    }
    const int keys = sm->keys[w.r], qp = q.qp;
    load_query(after, q);                                              // the next piece's, behind this one's keys
    i64 mymax = ATT_NEG;
    for (int i = 0; i < w.count; ++i) {
      if (ok) ok = mbar_wait(&sm->full[slot], phase);
      ok = __all_sync(0xffffffffu, ok && *abort_flag == 0);
      const int key0 = (w.u + i) * SPL_KEYS + 8 * warp;
      if (ok && key0 < keys) {
        const uint8_t* kp = ring + slot * SPL_K_STAGE + (8 * warp + (lane >> 2)) * ATT2_HALF + 16 * (lane & 3);
        int acc[3][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}, {0, 0, 0, 0}};
        const bool kvalid = key0 + (lane >> 2) < keys;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          uint4 v = make_uint4(0, 0, 0, 0);
          if (kvalid) v = *reinterpret_cast<const uint4*>(kp + j * ATT_HD);
          mma_s8(acc[j], afrag[0], v.x, v.y);
          mma_s8(acc[j], afrag[1], v.z, v.w);
        }
        const i64 raw = fragment_score(acc, lane);
        const int in = 8 * warp + 2 * (lane & 3) + (lane >> 4), key = (w.u + i) * SPL_KEYS + in;
        sp.scores[((int64_t)(w.x + i) * SPL_KEYS + in) * 4 + g] = raw;
        if (key < keys && key <= qp) mymax = imax(mymax, raw);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm->empty[slot]);
      if (++slot == SPL_K_STAGES) { slot = 0; phase ^= 1; }
    }
    i64 m = imax(mymax, __shfl_xor_sync(0xffffffffu, mymax, 16));
    m = imax(m, __shfl_xor_sync(0xffffffffu, m, 1));
    m = imax(m, __shfl_xor_sync(0xffffffffu, m, 2));
    if (lane < 16 && (lane & 3) == 0) sm->wmax[turn][warp][lane >> 2] = m;
    asm volatile("bar.sync 1, %0;" ::"n"(32 * SPL_WARPS) : "memory");  // a warp is at most one piece ahead of another
    if (threadIdx.x < 4) {
      i64 best = ATT_NEG;
#pragma unroll
      for (int v = 0; v < SPL_WARPS; ++v) best = imax(best, sm->wmax[turn][v][threadIdx.x]);
      sp.pmax[(pz + blockIdx.x) * 4 + threadIdx.x] = best;
    }
    w = after;
    turn ^= 1;
  }
  if (!ok && lane == 0) { atomicAdd(&g_wait_timeouts, 1); sm->abort_flag = 1; }
}

struct SplitValuesSmall {
  uint64_t full[SPL_V_STAGES], empty[SPL_V_STAGES];
  uint64_t pfull[2], pfree[2];                   // a wave's weight tiles: written by the 8 warps, read by its MMAs
  uint64_t accfull[2], accfree[2];               // a piece's accumulators: committed by the MMAs, read by 4 warps
  double products[PW_DOUBLES];
  i64 cnum[2][4][ATT_HD];
  i64 pden[2][SPL_WARPS][4];
  uint32_t tmem_base;
  uint32_t abort_flag;
  int start[SPL_MAXREQ + 1], keys[SPL_MAXREQ];
};
__host__ __device__ constexpr int split_values_smem(int pages) {
  return 1024 + SPL_V_STAGES * SPL_V_STAGE + 2 * SPL_WAVE * SPL_PTILE + (int)sizeof(SplitValuesSmall) + 4 * pages;
}

__device__ __forceinline__ void add_i64(i64* p, i64 v) {
  asm volatile("red.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__global__ void __launch_bounds__(32 * (SPL_WARPS + 2), 2)
attention_values_kernel(const __grid_constant__ CUtensorMap tmap_v, const SplitParams sp) {
  extern __shared__ __align__(128) uint8_t att_smem[];
  const AttnParams& p = sp.a;
  uint8_t* ring = align_smem(att_smem);
  uint8_t* ptile = ring + SPL_V_STAGES * SPL_V_STAGE;                  // [2 waves][8 groups][512]
  SplitValuesSmall* sm = reinterpret_cast<SplitValuesSmall*>(ptile + 2 * SPL_WAVE * SPL_PTILE);
  int* list = reinterpret_cast<int*>(sm + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < SPL_V_STAGES; ++s) {
      mbar_init(&sm->full[s], 1);
      mbar_init(&sm->empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sm->pfull[i], SPL_WARPS);
      mbar_init(&sm->pfree[i], 1);
      mbar_init(&sm->accfull[i], 1);
      mbar_init(&sm->accfree[i], 4);
    }
    sm->abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmap_v);
  }
  if (warp == 0) {
    tmem_alloc(&sm->tmem_base, SPL_TMEM);
    tmem_relinquish();
  }
  // attention_scores_kernel is always the kernel in front, launched by the same call, and permits an early start behind its own
  // wait: what it reads (positions, block table, cache, tables) is complete. Its scores, maxima and cleared outputs are not before
  // the wait of the weight warps.
  ProductTable pt;
  load_products(p.lut, p.ptab, pt, sm->products, threadIdx.x, blockDim.x);
  split_starts(p, sp.nreq, sm->start, sm->keys);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm->tmem_base;
  const int units = sm->start[sp.nreq] * p.HKV, from = split_bound(units, blockIdx.x), to = split_bound(units, blockIdx.x + 1);
  split_pages(p, sp.nreq, sm->start, sm->keys, from, to, list);
  SplitWalk w;
  w.begin(sm->start, p.HKV, sp.nreq, from, to);
  volatile uint32_t* abort_flag = &sm->abort_flag;

  if (warp == SPL_WARPS) {
    split_produce<true, SPL_V_STAGES>(tmap_v, p, w, ring, sm, list, lane);
  } else if (warp == SPL_WARPS + 1) {
    // ---------------- MMA warp: one thread ----------------
    if (lane == 0) {
      constexpr uint32_t IDESC = umma_idesc_i8_amn(16);
      bool ok = true;
      int slot = 0, phase = 0;
      uint32_t piece = 0, wave = 0;
      for (; w.more() && ok; w.next(), ++piece) {
        const uint32_t acc = tmem + 32 * (piece & 1);
        if (piece >= 2) ok = mbar_wait(&sm->accfree[piece & 1], ((piece >> 1) - 1) & 1);
        tc_fence_after();
        const int waves = (2 * w.count + SPL_WAVE - 1) / SPL_WAVE;
        for (int v = 0; v < waves && ok; ++v, ++wave) {
          ok = mbar_wait(&sm->pfull[wave & 1], (wave >> 1) & 1);
          const uint32_t pt = smem_u32(ptile) + (wave & 1) * SPL_WAVE * SPL_PTILE;
          const int stages = min(SPL_WAVE / 2, w.count - v * (SPL_WAVE / 2));
          for (int s = 0; s < stages && ok; ++s) {
            ok = mbar_wait(&sm->full[slot], phase) && *abort_flag == 0;
            if (!ok) break;
            tc_fence_after();
            const uint32_t vb = smem_u32(ring) + slot * SPL_V_STAGE;
#pragma unroll
            for (int kg = 0; kg < 2; ++kg) {
              const uint64_t b = umma_desc_kmajor_plain(pt + (2 * s + kg) * SPL_PTILE, 256, 128);
              const uint32_t more = v > 0 || s > 0 || kg > 0 ? 1u : 0u;
              umma_i8(acc, umma_desc_sw128(vb + kg * 4096), b, IDESC, more);
              umma_i8(acc + 16, umma_desc_sw128(vb + SPL_KEYS * 128 + kg * 4096), b, IDESC, more);
            }
            umma_commit(&sm->empty[slot]);
            if (++slot == SPL_V_STAGES) { slot = 0; phase ^= 1; }
          }
          if (ok) umma_commit(&sm->pfree[wave & 1]);
        }
        if (ok) umma_commit(&sm->accfull[piece & 1]);
      }
      if (!ok) { atomicAdd(&g_wait_timeouts, 1); sm->abort_flag = 1; }
    }
    __syncwarp();
  } else {
    // ---------------- weight warps: from here on, what the first kernel writes ----------------
    wait_previous();
    bool ok = true;
    const int g = lane & 3;                                            // this lane's query
    uint32_t piece = 0, wave = 0;
    // this lane's four scores of group `grp` of the walk's piece (warp w takes group w of every wave)
    auto load_scores = [&](const SplitWalk& v, int grp, i64 (&sc)[4]) {
#pragma unroll
      for (int j = 0; j < 4; ++j) sc[j] = 0;
      if (!v.more() || grp >= 2 * v.count) return;
      const i64* s = sp.scores + ((int64_t)v.x * SPL_KEYS + grp * 32 + (lane >> 2)) * 4 + g;
#pragma unroll
      for (int j = 0; j < 4; ++j) sc[j] = s[32 * j];
    };
    // what a piece needs beside them, as loaded (nothing here waits for a load): the maximum of one CTA's part of the pair per
    // eight lanes, the query's position and row shift
    struct Piece {
      i64 mx, qpos, sh;
      int64_t pz;
      int b0, b1;                                                      // CTAs that have a part of the pair
    };
    auto load_piece = [&](const SplitWalk& v, Piece& q) {
      q.mx = ATT_NEG;
      q.qpos = -1;
      q.sh = 0;
      q.b0 = q.b1 = blockIdx.x;
      if (!v.more()) return;
      q.pz = (int64_t)v.r * p.HKV + v.h;
      if (g < p.M) {
        q.qpos = p.qpos[(int64_t)v.r * p.M + g];
        if (p.sh) q.sh = p.sh[q.pz * p.M + g];
      }
      if (v.u != 0 || v.count != v.n) {
        const int x0 = v.x - v.u;
        q.b0 = split_owner(units, x0);
        q.b1 = split_owner(units, x0 + v.n - 1);
      }
      if (q.b0 + (lane >> 2) <= q.b1) q.mx = sp.pmax[(q.pz + q.b0 + (lane >> 2)) * 4 + g];
    };
    // ---- accumulators of a piece: first tile lanes 0..63 = (V limb 0, dim), 64..127 = (V limb 1, dim); second tile lanes
    //      64..127 = (V limb 2, dim). Column 4 i + g = (weight limb i, query g). ----
    auto flush = [&](uint32_t piece, int64_t pz, bool whole) {
      const int turn = piece & 1;
      i64 part[4] = {0, 0, 0, 0};
      if (warp < 4) {
        if (ok) ok = mbar_wait(&sm->accfull[turn], (piece >> 1) & 1);
        ok = __all_sync(0xffffffffu, ok && *abort_flag == 0);
        if (ok) {
          tc_fence_after();
          uint32_t d01[16], d12[16];
          const uint32_t tb = tmem + 32 * turn + ((uint32_t)(warp * 32) << 16);
          tmem_ld16(tb, d01);
          tmem_ld16(tb + 16, d12);
          tmem_ld_wait();
          tc_fence_before();
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            i64 a = (i64)(int32_t)d01[q] + shl((i64)(int32_t)d01[4 + q], 8) + shl((i64)(int32_t)d01[8 + q], 16);
            if (warp >= 2) {
              const i64 b = (i64)(int32_t)d12[q] + shl((i64)(int32_t)d12[4 + q], 8) + shl((i64)(int32_t)d12[8 + q], 16);
              a = shl(a, 8) + shl(b, 16);
            }
            part[q] = a;
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm->accfree[turn]);
        if (warp < 2) {
#pragma unroll
          for (int q = 0; q < 4; ++q) sm->cnum[turn][q][warp * 32 + lane] = part[q];
        }
      }
      asm volatile("bar.sync 1, %0;" ::"n"(32 * SPL_WARPS) : "memory"); // cnum, pden written; a warp is at most one piece ahead
      if (ok && (warp == 2 || warp == 3)) {
        const int d = (warp - 2) * 32 + lane;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (q < p.M) {
            i64* o = p.num + (pz * p.M + q) * ATT_HD + d;
            const i64 x = sm->cnum[turn][q][d] + part[q];
            if (whole) *o = x; else add_i64(o, x);
          }
      }
      if (ok && threadIdx.x < p.M) {
        i64 x = 0;
#pragma unroll
        for (int v = 0; v < SPL_WARPS; ++v) x += sm->pden[turn][v][threadIdx.x];
        i64* o = p.den + pz * p.M + threadIdx.x;
        if (whole) *o = x; else add_i64(o, x);
      }
    };
    const uint32_t l2e = (uint32_t)p.l2e;
    i64 sc[4];
    Piece q, last{};
    load_scores(w, warp, sc);
    load_piece(w, q);
    bool product = true;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += 32 * SPL_WARPS) product &= sp.fits[i] != 0;
    product = split_and(product);
    while (w.more()) {
      SplitWalk after = w;
      after.next();
      const Piece cur = q;
      load_piece(after, q);
      i64 mx = cur.mx;
      for (int b = cur.b0 + 8 + (lane >> 2); b <= cur.b1; b += 8) mx = imax(mx, sp.pmax[(cur.pz + b) * 4 + g]);
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) mx = imax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const i64 rowshift = g < p.M && p.sh ? (i64)(FK + 3 - FZ) - cur.sh : 0;
      const bool fast = product && (p.ptab || (rowshift >= 1 && rowshift <= 31));
      const int c = p.ptab ? WT_INT8_SHIFT : fast ? (int)rowshift : 1;
      const i64 mxh = mx + (p.ptab ? (1ll << (WT_INT8_SHIFT - 1)) - 1 : 1ll << (c - 1));
      const int qp = (int)imin(cur.qpos, (i64)sm->keys[w.r] - 1);
      i64 den = 0;
      const int groups = 2 * w.count, waves = (groups + SPL_WAVE - 1) / SPL_WAVE;
      for (int v = 0; v < waves; ++v, ++wave) {
        const int grp = v * SPL_WAVE + warp;
        i64 nx[4];
        if (v + 1 < waves) load_scores(w, grp + SPL_WAVE, nx); else load_scores(after, warp, nx);
        uint32_t pv[4];
        int redo = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const bool live = grp < groups && w.u * SPL_KEYS + grp * 32 + 8 * j + (lane >> 2) <= qp;
          bool unsure;
          pv[j] = p.ptab ? product_weight8(pt, mxh - sc[j], live, unsure) : product_weight(pt, l2e, mxh - sc[j], c, live, unsure);
          redo |= (fast ? unsure : live) ? 1 << j : 0;
        }
        if (redo) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (redo >> j & 1) pv[j] = (uint32_t)attn_weight_any(p, sc[j], mx, rowshift);
        }
        if (ok && wave >= 2) ok = mbar_wait(&sm->pfree[wave & 1], ((wave >> 1) - 1) & 1);
        ok = __all_sync(0xffffffffu, ok && *abort_flag == 0);
        if (ok && grp < groups) {
          uint8_t* pt = ptile + ((wave & 1) * SPL_WAVE + warp) * SPL_PTILE;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int kl = 8 * j + (lane >> 2);
            den += (i64)(int32_t)pv[j];
            const uint32_t lb = limb_bytes(pv[j]);
            const int off = (kl >> 4) * 256 + (kl & 15) + g * 16;
            pt[off] = (uint8_t)lb;                                     // row g      (limb 0)
            pt[off + 64] = (uint8_t)(lb >> 8);                         // row 4 + g  (limb 1)
            pt[off + 128] = (uint8_t)(lb >> 16);                       // row 8 + g  (limb 2)
          }
          fence_proxy_async_smem();                                    // the tile is read by tcgen05 (async proxy)
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm->pfull[wave & 1]);
#pragma unroll
        for (int j = 0; j < 4; ++j) sc[j] = nx[j];
        if (v == 0 && piece > 0) flush(piece - 1, last.pz, last.b0 == last.b1);  // the piece before: its MMAs ran behind these weights
      }
      den += __shfl_xor_sync(0xffffffffu, den, 4);
      den += __shfl_xor_sync(0xffffffffu, den, 8);
      den += __shfl_xor_sync(0xffffffffu, den, 16);
      if (lane < 4) sm->pden[piece & 1][warp][lane] = den;
      last = cur;
      w = after;
      ++piece;
    }
    if (piece > 0) flush(piece - 1, last.pz, last.b0 == last.b1);
    if (!ok && lane == 0) { atomicAdd(&g_wait_timeouts, 1); sm->abort_flag = 1; }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, SPL_TMEM);
  }
}

}  // namespace bx
