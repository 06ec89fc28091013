// Prefill attention over the paged int8 limb-plane KV cache: tiles of consecutive query tokens of one request and one
// KV head, both integer sweeps inside the CTA, the limb products on tcgen05.
//
// A tile is BT = 32 / G consecutive tokens x the G query heads of the KV head: 32 query rows r = t G + g, so a K / V
// row staged for the tile serves 32 queries (the per-row decode kernel stages it once per token). Same integers as
// the per-row kernel and as the reference's prefill kernel (src/bitexact/vllm_plugin/tri_prefill.py:32-86, int8
// weight rule) and, with the exact weight rule, as bmm + softmax_w + bmm (src/bitexact/exact/model.py:114-119):
// every product is an exact limb dot, the maximum and the sums are exact integer reductions, and key s is visible
// to a query iff s <= its position, so the grouping of queries into tiles cannot change a bit.
//
// Per block of 128 keys (staged by TMA, one box of 128 bytes x page rows per page and cache-row third:
// [K0|K1], [K2|V0], [V1|V2], 128-byte swizzle, no byte fetched twice):
//   scores  S^T [128 keys = TMEM lanes] x [5 blocks x 32 queries]: A = K limb j tile (K-major), B = the three
//           stacked query limb tiles [96 x 64] written once per tile; 8 MMAs; block b = i + j as in the limb GEMM.
//   sweep 1 keeps a running maximum per (thread, query row); sweep 2 recomputes the scores (the MMAs are a few
//           hundred cycles; keeping 32 x S int64 scores on chip is not possible), turns them into weights with the
//           final row maximum, and writes the weights' three limbs as the B operand [96 x 128 keys] of
//   p.V     D1 [lanes = bytes of [K2|V0]] and D2 [lanes = bytes of [V1|V2]] x [96 = (weight limb, query)], A = the
//           staged cache rows read MN-major (no transposition), accumulated in TMEM over ALL keys of the tile and
//           read once at the end (|sum| <= keys * 2^14 < 2^31 for fewer than 43690 keys).
//
// What bounds it: the weight function, once per (query row, key) pair on the CUDA cores. So the weight table lies in
// shared memory (attn_weight_tables.cuh), and everything else is arranged so that the 16 weight warps never wait:
//   * one persistent CTA per SM walks the (tile, KV head) list backwards (the tiles of a prompt grow with its position:
//     the short ones come last and fill the last wave), so that the table is copied once per launch;
//   * a producer warp streams boxes of 16 KB through a ring across sweeps and tiles (8 boxes beside the 65 KB table of
//     the exact rule, 6 beside the 83 KB of the int8 rule; [K0|K1] is released by the score MMAs already);
//   * an MMA warp issues the scores of step i + 1 before p.V of step i: two score accumulators (2 x 160 TMEM columns)
//     and two weight tiles, so the tensor pipe works on the next block while the weights of this one are made;
//   * the next tile's queries are written as soon as the last score product of this one is complete.
// Weight warps: warp % 4 = TMEM lane quarter (32 keys), warp / 4 = group of 8 query rows.
// One B200, 4 prompts of 1700 .. 2048 tokens, 32 query heads, a launch of 3750 rows: 2.10 ms as one CTA per tile with the table
// gathered through L1, 0.80 ms so (int8 rule 1.13 -> 0.51 ms).
//
// Every wait is bounded; a timeout sets the device status word, after which the remaining steps run through without
// waiting or touching the results.
#pragma once

#include "attn_weight_tables.cuh"
#include "paged_attention.cuh"

namespace bx {

constexpr int PF_ROWS = 32;                     // query rows per tile
constexpr int PF_KEYS = 128;                    // keys per block
constexpr int PF_BOX = PF_KEYS * 128;           // one third of the cache rows of a block: 16 KB
constexpr int PF_WARPS = 16;                    // weight warps: 4 lane quarters x 4 groups of 8 rows
constexpr int PF_THREADS = 32 * (PF_WARPS + 2); // and a producer and an MMA warp
constexpr int PF_RG = 3 * PF_ROWS / 8;          // 8-row groups of the limb tiles
constexpr int PF_LBO = PF_RG * 128;             // bytes between the 16-byte K chunks of those tiles
constexpr int PF_QTILE = 4 * PF_LBO;            // query limbs [96 x 64 dims] as 8 x 16-byte core matrices
constexpr int PF_PTILE = 8 * PF_LBO;            // weight limbs [96 x 128 keys]
constexpr int PF_S_COLS = 5 * PF_ROWS;          // score accumulators of a step
constexpr int PF_D1 = 2 * PF_S_COLS, PF_D2 = PF_D1 + 3 * PF_ROWS;     // p.V accumulators; 512 columns in all
constexpr int PF_TMEM = 512;
constexpr int PF_MAXBOXES = 8;

__host__ __device__ constexpr int pf_boxes(bool exact) { return exact ? 8 : 6; }
__host__ __device__ constexpr int pf_table_bytes(bool exact) { return exact ? WT_EXP2_BYTES : WT_INT8_BYTES; }

struct PrefillParams {
  const int32_t* q;     // [N, HKV, G, 64]
  const i64* sh;        // [N, HKV, G] (exact mode; null with ptab)
  const i64* pos;       // [N] query position of each token
  const int32_t* tiles; // [T, 3] (block-table row, first token, tokens; more than 32 / G are taken 32 / G at a time)
  const void* bt;
  int bt64;
  int64_t sbt;
  int nblk, bs;
  AttnParams w;         // weight rule: lut / l2e (exact) or ptab (int8)
  i64* num;             // [N, HKV, G, 64]
  i64* den;             // [N, HKV, G]
  int HKV, G;
  int64_t work;         // tiles x KV heads
};

struct PrefillTile {    // what the producer warp hands on with a tile
  i64 out[PF_ROWS];     // row of q, num / 64 and den, -1: no query (its weights are 0, nothing is written)
  i64 rshift[PF_ROWS];
  int qp[PF_ROWS];
  int nb;               // blocks of 128 keys (at least 1)
  int live;             // 0: no key is visible to any query, nothing is written
};

struct PrefillSmall {
  uint64_t full[PF_MAXBOXES], empty[PF_MAXBOXES];
  uint64_t sready[2], sfree[2];       // score accumulators: committed by the MMAs, read by the 16 weight warps
  uint64_t pfull[2], pvdone[2];       // weight tiles: written by the 16 weight warps, read by the p.V MMAs
  uint64_t info_full[2], info_empty[2];
  uint64_t qfull;
  uint32_t tmem_base;
  uint32_t fail;
  uint32_t bad_table;
  i64 red[4][PF_ROWS];
  i64 mx[PF_ROWS], mxh[PF_ROWS];      // row maximum, and with the rounding term of the row shift
  int c[PF_ROWS];                     // row shift, 0: the row takes the general weight function
  PrefillTile tile[2];
};

__host__ __device__ constexpr int pf_smem(bool exact) {
  return pf_boxes(exact) * PF_BOX + PF_QTILE + 2 * PF_PTILE + pf_table_bytes(exact) + (int)sizeof(PrefillSmall) + 1024;
}
static_assert(pf_smem(true) <= 232448 && pf_smem(false) <= 232448, "shared memory of an SM");

template <bool EXACT>
__global__ void __launch_bounds__(PF_THREADS, 1)
prefill_attention_kernel(const __grid_constant__ CUtensorMap tmap, const PrefillParams p) {
  constexpr int NBOX = pf_boxes(EXACT);
  extern __shared__ uint8_t pf_raw[];
  uint8_t* ring = align_smem(pf_raw);
  uint8_t* qtile = ring + NBOX * PF_BOX;
  uint8_t* ptile = qtile + PF_QTILE;
  uint8_t* table = ptile + 2 * PF_PTILE;
  PrefillSmall* sm = reinterpret_cast<PrefillSmall*>(table + pf_table_bytes(EXACT));
  i64* comb = reinterpret_cast<i64*>(ptile);           // after a tile's last MMA: [32 rows][64 dims]
  i64* dens = comb + PF_ROWS * ATT_HD;                 // and the sums of the weights [4 quarters][32 rows]
  static_assert((PF_ROWS * ATT_HD + 4 * PF_ROWS) * 8 <= 2 * PF_PTILE, "exchange");

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile uint32_t* fail = &sm->fail;

  if (tid == 0) {
    for (int i = 0; i < NBOX; ++i) {
      mbar_init(&sm->full[i], 1);
      mbar_init(&sm->empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sm->sready[i], 1);
      mbar_init(&sm->sfree[i], PF_WARPS);
      mbar_init(&sm->pfull[i], PF_WARPS);
      mbar_init(&sm->pvdone[i], 1);
      mbar_init(&sm->info_full[i], 1);
      mbar_init(&sm->info_empty[i], PF_WARPS + 1);
    }
    mbar_init(&sm->qfull, PF_WARPS);
    sm->fail = *reinterpret_cast<volatile int*>(&g_wait_timeouts) != 0;
    sm->bad_table = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmap);
  }
  if (warp == 0) {
    tmem_alloc(&sm->tmem_base, PF_TMEM);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm->tmem_base;
  bool ok = sm->fail == 0;
  // a wait that ran out: note it once per role, run the rest of the loop without waiting
  auto give_up = [&]() {
    atomicAdd(&g_wait_timeouts, 1);
    *fail = 1;
  };
  auto item = [&](int64_t w) { return p.work - 1 - w; };
  // Pieces of 32 / G tokens of work item w. Every role reads it from the list itself, so that all go through the same number
  // of rounds (and barriers) whatever a wait came to.
  const int per = PF_ROWS / p.G;
  auto pieces = [&](int64_t w) -> int {
    if (w >= p.work) return 1;
    const int n = p.tiles[3 * (item(w) / p.HKV) + 2];
    return n > per ? (n + per - 1) / per : 1;
  };

  if (warp == PF_WARPS) {
    // ---------------- producer warp ----------------
    wait_previous();
    const int pages = PF_KEYS / p.bs;                  // pages per block, one per lane
    int slot = 0, round = 0, issued = 0;
    uint32_t k = 0;
    const bool start = ok;
    int piece = 0;
    for (int64_t w = blockIdx.x; w < p.work && ok; ++k) {
      const int64_t it = item(w);
      const int h = (int)(it % p.HKV);
      const int32_t* tl = p.tiles + 3 * (it / p.HKV);
      const int64_t brow = tl[0], tok0 = tl[1] + (int64_t)piece * per;
      const int rest = tl[2] - piece * per, ntok = min(rest, per);
      if (rest > per) ++piece; else { piece = 0; w += gridDim.x; }
      // ---- the tile's rows, one per lane ----
      if (k >= 2) ok = __all_sync(0xffffffffu, mbar_wait(&sm->info_empty[k & 1], ((k >> 1) - 1) & 1));
      if (!ok) break;
      PrefillTile& ti = sm->tile[k & 1];
      const int t = lane / p.G, g = lane % p.G;
      i64 qp = -1, rs = 0, out = -1;
      if (t < ntok) {
        qp = imin(p.pos[tok0 + t], (i64)p.nblk * p.bs - 1);
        out = ((tok0 + t) * p.HKV + h) * p.G + g;
        if (EXACT) rs = (i64)(FK + 3 - FZ) - p.sh[out];
      }
      ti.out[lane] = out;
      ti.rshift[lane] = rs;
      ti.qp[lane] = (int)qp;
      const int kend = __reduce_max_sync(0xffffffffu, (int)imax(qp, -1)) + 1;
      const int nb = kend > 0 ? (kend + PF_KEYS - 1) / PF_KEYS : 1;
      if (lane == 0) {
        ti.nb = nb;
        ti.live = kend > 0;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm->info_full[k & 1]);
      // ---- its boxes ----
      auto page = [&](int blk) -> int {                // pages past the table: the null block (its keys are masked)
        const int pidx = blk * pages + lane;
        if (lane >= pages || pidx >= p.nblk) return 0;
        return p.bt64 ? (int)reinterpret_cast<const int64_t*>(p.bt)[brow * p.sbt + pidx]
                      : reinterpret_cast<const int32_t*>(p.bt)[brow * p.sbt + pidx];
      };
      int blk = 0, sweep = 0, cur = page(0);
      for (int i = 0; i < 2 * nb && ok; ++i) {
        const int nblk = blk + 1 == nb ? 0 : blk + 1;
        const int nxt = page(nblk);                    // requested before this block's waits
        for (int third = 0; third < 2 + sweep && ok; ++third) {
          if (round > 0) ok = mbar_wait(&sm->empty[slot], (round - 1) & 1);
          ok = __all_sync(0xffffffffu, ok && *fail == 0);
          if (!ok) break;
          if (lane == 0) mbar_arrive_expect_tx(&sm->full[slot], PF_BOX);
          __syncwarp();
          if (lane < pages)
            tma_load_4d(ring + slot * PF_BOX + lane * p.bs * 128, &tmap, &sm->full[slot], 128 * third, 0, h, cur);
          if (issued < NBOX) ++issued;
          if (++slot == NBOX) { slot = 0; ++round; }
        }
        cur = nxt;
        blk = nblk;
        if (blk == 0) sweep = 1;
      }
    }
    if (start && !ok && lane == 0) give_up();
    for (int i = 0; i < issued; ++i) {                 // whatever happened elsewhere: copies in flight land before the exit
      if (--slot < 0) { slot = NBOX - 1; --round; }
      mbar_wait(&sm->full[slot], round & 1);
    }
  } else if (warp == PF_WARPS + 1) {
    // ---------------- MMA warp: one thread ----------------
    wait_previous();
    if (lane == 0) {
      constexpr uint32_t ID_ALL = umma_idesc_i8(3 * PF_ROWS), ID_ONE = umma_idesc_i8(PF_ROWS), ID_TWO = umma_idesc_i8(2 * PF_ROWS);
      constexpr uint32_t ID_PV = umma_idesc_i8_amn(3 * PF_ROWS);
      const uint32_t qaddr = smem_u32(qtile), raddr = smem_u32(ring);
      const bool start = ok;
      int slot = 0, phase = 0;
      uint32_t k = 0, s = 0, v = 0;                    // tiles, score steps, p.V steps so far
      int pv_k2v0 = -1, pv_v12 = 0;                    // boxes of the p.V step that is due, -1: none
      bool pv_first = false;
      auto next_box = [&]() -> int {                   // waits for the next box of the ring
        if (ok) ok = mbar_wait(&sm->full[slot], phase);
        const int b = slot;
        if (++slot == NBOX) { slot = 0; phase ^= 1; }
        return b;
      };
      auto pv_step = [&]() {
        const uint32_t buf = v & 1;
        if (ok) ok = mbar_wait(&sm->pfull[buf], (v >> 1) & 1);
        if (!ok) return;
        tc_fence_after();
        const uint32_t paddr = smem_u32(ptile) + buf * PF_PTILE;
#pragma unroll
        for (int kg = 0; kg < 4; ++kg) {
          const uint64_t pdesc = umma_desc_kmajor_plain(paddr + kg * 2 * PF_LBO, PF_LBO, 128);
          const uint32_t accum = (!pv_first || kg > 0) ? 1u : 0u;
          umma_i8(tmem + PF_D1, umma_desc_sw128(raddr + pv_k2v0 * PF_BOX + kg * 4096), pdesc, ID_PV, accum);
          umma_i8(tmem + PF_D2, umma_desc_sw128(raddr + pv_v12 * PF_BOX + kg * 4096), pdesc, ID_PV, accum);
        }
        umma_commit(&sm->empty[pv_k2v0]);
        umma_commit(&sm->empty[pv_v12]);
        umma_commit(&sm->pvdone[buf]);
        ++v;
        pv_k2v0 = -1;
      };
      int left = pieces(blockIdx.x);
      for (int64_t w = blockIdx.x; w < p.work && ok; ++k) {
        if (--left == 0) {
          w += gridDim.x;
          left = pieces(w);
        }
        ok = mbar_wait(&sm->info_full[k & 1], (k >> 1) & 1);
        const int nb = ok ? sm->tile[k & 1].nb : 0;
        mbar_arrive(&sm->info_empty[k & 1]);
        if (ok) ok = mbar_wait(&sm->qfull, k & 1);
        for (int i = 0; i < 2 * nb && ok; ++i, ++s) {
          const bool second = i >= nb;
          const uint32_t buf = s & 1;
          const int b0 = next_box(), b1 = next_box();
          if (ok && s >= 2) ok = mbar_wait(&sm->sfree[buf], ((s >> 1) - 1) & 1);
          if (!ok) break;
          tc_fence_after();
          const uint32_t acc = tmem + buf * PF_S_COLS;
#pragma unroll
          for (int ks = 0; ks < 2; ++ks) {
            const uint32_t qk = qaddr + ks * 2 * PF_LBO;
            const uint64_t q_all = umma_desc_kmajor_plain(qk, PF_LBO, 128);
            const uint64_t k0 = umma_desc_sw128(raddr + b0 * PF_BOX + ks * 32);
            const uint64_t k1 = umma_desc_sw128(raddr + b0 * PF_BOX + 64 + ks * 32);
            const uint64_t k2 = umma_desc_sw128(raddr + b1 * PF_BOX + ks * 32);
            if (ks == 0) {
              // every column block written once without accumulation
              const uint64_t q_last = umma_desc_kmajor_plain(qk + (2 * PF_ROWS / 8) * 128, PF_LBO, 128);
              umma_i8(acc, k0, q_all, ID_ALL, 0);
              umma_i8(acc + 3 * PF_ROWS, k1, q_last, ID_ONE, 0);
              umma_i8(acc + 1 * PF_ROWS, k1, q_all, ID_TWO, 1);
              umma_i8(acc + 4 * PF_ROWS, k2, q_last, ID_ONE, 0);
              umma_i8(acc + 2 * PF_ROWS, k2, q_all, ID_TWO, 1);
            } else {
              umma_i8(acc, k0, q_all, ID_ALL, 1);
              umma_i8(acc + 1 * PF_ROWS, k1, q_all, ID_ALL, 1);
              umma_i8(acc + 2 * PF_ROWS, k2, q_all, ID_ALL, 1);
            }
          }
          umma_commit(&sm->empty[b0]);
          if (!second) umma_commit(&sm->empty[b1]);
          umma_commit(&sm->sready[buf]);
          if (pv_k2v0 >= 0) pv_step();                 // the weights of the step before
          if (second) {
            pv_k2v0 = b1;
            pv_v12 = next_box();
            pv_first = i == nb;
          }
        }
      }
      if (ok && pv_k2v0 >= 0) pv_step();
      if (start && !ok) give_up();
    }
    __syncwarp();
  } else {
    // ---------------- weight warps ----------------
    const int quarter = warp & 3, group = warp >> 2;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    // One int4 of the tile's queries per thread: row (i, r) of the B operand, 16-byte K chunks PF_LBO apart.
    const int qr = tid >> 4, qd = (tid & 15) * 4;
    auto load_q = [&](const PrefillTile& ti) -> int4 {
      const i64 o = ti.out[qr];
      return o >= 0 ? *reinterpret_cast<const int4*>(p.q + o * ATT_HD + qd) : make_int4(0, 0, 0, 0);
    };
    auto write_q = [&](const int4& x) {
      const uint32_t b[4] = {limb_bytes((uint32_t)x.x), limb_bytes((uint32_t)x.y), limb_bytes((uint32_t)x.z), limb_bytes((uint32_t)x.w)};
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int row = i * PF_ROWS + qr;
        const uint32_t lo = __byte_perm(b[0], b[1], i | ((4 + i) << 4)), hi = __byte_perm(b[2], b[3], i | ((4 + i) << 4));
        *reinterpret_cast<uint32_t*>(qtile + (qd >> 4) * PF_LBO + (row >> 3) * 128 + (row & 7) * 16 + (qd & 15)) =
            __byte_perm(lo, hi, 0x5410);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm->qfull);
    };
    auto sync_weights = [&]() { asm volatile("bar.sync 1, %0;" ::"n"(32 * PF_WARPS) : "memory"); };
    const bool start = ok;
    // ---- the weight table, and the first tile's queries ----
    wait_previous();
    {
      bool fits = EXACT ? fill_exp2_table(table, p.w.lut, tid, 32 * PF_WARPS) : fill_int8_table(table, p.w.ptab, tid, 32 * PF_WARPS);
      if (EXACT) {
        sync_weights();
        fits &= check_exp2_table(table, tid, 32 * PF_WARPS) && p.w.l2e >= (1ll << 28) && p.w.l2e < (1ll << 29);
      }
      if (!fits) sm->bad_table = 1;
      if (ok && blockIdx.x < p.work) {
        ok = mbar_wait(&sm->info_full[0], 0);
        if (ok) write_q(load_q(sm->tile[0]));
      }
      sync_weights();
    }
    const bool fits = sm->bad_table == 0;
    const uint32_t l2e = (uint32_t)p.w.l2e;
    uint32_t k = 0, s = 0, v = 0;
    int left = pieces(blockIdx.x);
    for (int64_t w = blockIdx.x; w < p.work && start; ++k) {
      if (--left == 0) {
        w += gridDim.x;
        left = pieces(w);
      }
      const PrefillTile& ti = sm->tile[k & 1];
      if (ok) ok = mbar_wait(&sm->info_full[k & 1], (k >> 1) & 1);
      ok = __all_sync(0xffffffffu, ok && *fail == 0);
      const int nb = ok ? ti.nb : 0;
      const bool last_tile = w >= p.work;              // w is already that of the next piece
      int qmin = 0x7fffffff;                             // keys up to here are visible to the warp's 8 rows
#pragma unroll
      for (int j = 0; j < 8; ++j) qmin = min(qmin, ti.qp[8 * group + j]);
      // the scores of a step: this thread's key of the block x 8 query rows
      auto scores = [&](i64 (&raw)[8]) {
        const uint32_t buf = s & 1;
        if (ok) ok = mbar_wait(&sm->sready[buf], (s >> 1) & 1);
        ok = __all_sync(0xffffffffu, ok && *fail == 0);
        if (!ok) return;
        tc_fence_after();
        uint32_t acc[5][8];
#pragma unroll
        for (int b = 0; b < 5; ++b) tmem_ld8(tmem + lane_base + buf * PF_S_COLS + b * PF_ROWS + 8 * group, acc[b]);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm->sfree[buf]);
#pragma unroll
        for (int j = 0; j < 8; ++j) raw[j] = join5(acc[0][j], acc[1][j], acc[2][j], acc[3][j], acc[4][j]);
      };

      // ---- sweep 1: row maxima ----
      {
        i64 mx[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) mx[j] = ATT_NEG;
        for (int blk = 0; blk < nb && ok; ++blk, ++s) {
          i64 raw[8];
          scores(raw);
          if (!ok) break;
          if (blk * PF_KEYS + PF_KEYS - 1 <= qmin) {
#pragma unroll
            for (int j = 0; j < 8; ++j) mx[j] = imax(mx[j], raw[j]);
          } else {
            const int key = blk * PF_KEYS + quarter * 32 + lane;
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (key <= ti.qp[8 * group + j]) mx[j] = imax(mx[j], raw[j]);
          }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int hi = __reduce_max_sync(0xffffffffu, (int)(mx[j] >> 32));
          const uint32_t lo = __reduce_max_sync(0xffffffffu, (int)(mx[j] >> 32) == hi ? (uint32_t)mx[j] : 0u);
          if (lane == 0) sm->red[quarter][8 * group + j] = (i64)(((u64)(uint32_t)hi << 32) | lo);
        }
      }
      sync_weights();
      if (tid < PF_ROWS) {
        const i64 m = imax(imax(sm->red[0][tid], sm->red[1][tid]), imax(sm->red[2][tid], sm->red[3][tid]));
        const i64 rs = ti.rshift[tid];
        const int c = !EXACT ? WT_INT8_SHIFT : (rs >= 1 && rs <= 31) ? (int)rs : 0;
        sm->mx[tid] = m;
        sm->mxh[tid] = m + (EXACT ? (c > 0 ? 1ll << (c - 1) : 0) : (1ll << (WT_INT8_SHIFT - 1)) - 1);
        sm->c[tid] = fits ? c : 0;
      }
      sync_weights();

      // ---- sweep 2: weights with the final maxima; their limbs are the B operand of p.V ----
      i64 den[8];
      int general = 0;                                   // rows that take the general weight function
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        den[j] = 0;
        general |= sm->c[8 * group + j] == 0 ? 1 << j : 0;
      }
      for (int blk = 0; blk < nb && ok; ++blk, ++s) {
        i64 raw[8];
        const bool prefetch = blk == nb - 1 && !last_tile;
        int4 qn = make_int4(0, 0, 0, 0);
        if (prefetch) {
          const uint32_t kn = k + 1;
          ok = mbar_wait(&sm->info_full[kn & 1], (kn >> 1) & 1);
          if (ok) qn = load_q(sm->tile[kn & 1]);
        }
        scores(raw);
        if (!ok) break;
        if (prefetch) write_q(qn);                       // the tile's last score product is complete
        const uint32_t buf = v & 1;
        if (v >= 2) ok = mbar_wait(&sm->pvdone[buf], ((v >> 1) - 1) & 1);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const int key = blk * PF_KEYS + quarter * 32 + lane;
        const bool all = blk * PF_KEYS + PF_KEYS - 1 <= qmin;
        uint32_t pv[8];
        int redo = general;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int r = 8 * group + j;
          const bool vis = all || key <= ti.qp[r];
          if (EXACT) {
            bool unsure;
            pv[j] = exp2_weight(sm->mxh[r] - raw[j], sm->c[r] | (general >> j & 1), l2e, vis, table, unsure);
            redo |= unsure ? 1 << j : 0;
          } else {
            pv[j] = int8_weight(sm->mxh[r] - raw[j], vis, table, p.w.ptab);
          }
        }
        if (redo) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int r = 8 * group + j;
            if (redo >> j & 1)
              pv[j] = all || key <= ti.qp[r] ? (uint32_t)attn_weight_any(p.w, raw[j], sm->mx[r], ti.rshift[r]) : 0;
          }
        }
        uint8_t* pcol = ptile + buf * PF_PTILE + quarter * 2 * PF_LBO + (lane >> 4) * PF_LBO + group * 128 + (lane & 15);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          den[j] += (i64)(int32_t)pv[j];
          const uint32_t b = limb_bytes(pv[j]);
          pcol[j * 16] = (uint8_t)b;
          pcol[(PF_ROWS / 8) * 128 + j * 16] = (uint8_t)(b >> 8);
          pcol[2 * (PF_ROWS / 8) * 128 + j * 16] = (uint8_t)(b >> 16);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm->pfull[buf]);
        ++v;
      }

      // ---- p.V accumulators: lane = byte of the cache-row third, column 32 i + r = (weight limb i, query r) ----
      if (ok) ok = mbar_wait(&sm->pvdone[(v - 1) & 1], ((v - 1) >> 1) & 1);
      ok = __all_sync(0xffffffffu, ok && *fail == 0);
      i64 part[8];
      if (ok) {
        tc_fence_after();
        uint32_t d1[3][8], d2[3][8];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          tmem_ld8(tmem + lane_base + PF_D1 + i * PF_ROWS + 8 * group, d1[i]);
          tmem_ld8(tmem + lane_base + PF_D2 + i * PF_ROWS + 8 * group, d2[i]);
        }
        tmem_ld_wait();
        tc_fence_before();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          i64 a = 0;
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            // quarters 0, 1: D2 lanes = V limb 1; quarters 2, 3: D1 lanes = V limb 0, D2 lanes = V limb 2
            const i64 x = quarter < 2 ? shl((i64)(int32_t)d2[i][j], 8)
                                      : (i64)(int32_t)d1[i][j] + shl((i64)(int32_t)d2[i][j], 16);
            a += shl(x, 8 * i);
          }
          part[j] = a;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) part[j] = 0;
      }
      // This warp has seen the tile's last p.V product complete, so the weight tiles are free: they hold the exchange
      // between the quarters. They are written again only after both barriers of the next tile's sweep 1.
      const int d = (quarter & 1) * 32 + lane;
      if (quarter < 2) {
#pragma unroll
        for (int j = 0; j < 8; ++j) comb[(8 * group + j) * ATT_HD + d] = part[j];
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        i64 x = den[j];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0) dens[quarter * PF_ROWS + 8 * group + j] = x;
      }
      sync_weights();
      const bool write = ok && ti.live != 0;
      if (quarter >= 2 && write) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const i64 o = ti.out[8 * group + j];
          if (o >= 0) p.num[o * ATT_HD + d] = part[j] + comb[(8 * group + j) * ATT_HD + d];
        }
      }
      if (tid < PF_ROWS && write) {
        const i64 o = ti.out[tid];
        if (o >= 0) p.den[o] = dens[tid] + dens[PF_ROWS + tid] + dens[2 * PF_ROWS + tid] + dens[3 * PF_ROWS + tid];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm->info_empty[k & 1]);
    }
    if (start && !ok && lane == 0) give_up();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, PF_TMEM);
  }
}

}  // namespace bx
