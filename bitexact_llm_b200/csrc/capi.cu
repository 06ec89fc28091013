// C ABI of libbitexact_b200.so (declared in include/bitexact_b200.h). One translation unit: the kernel headers
// are included here so that the device-side status word is shared by every kernel.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

#include "../../include/bitexact_b200.h"
#include "host_util.cuh"
#include "exact_linear.cuh"
#include "exact_linear_splitk.cuh"
#include "exact_linear_rows.cuh"
#include "int8_linear.cuh"
#include "int8_linear_splitk.cuh"
#include "int8_stages.cuh"
#include "elementwise.cuh"
#include "attention_split.cuh"
#include "paged_attention.cuh"
#include "prefill_attention.cuh"
#include "sampler.cuh"
#include "logp.cuh"
#include "decompose.cuh"
#include "unfused.cuh"
#include "unfused_stages.cuh"
#include "peak_probe.cuh"
#include "bmm_limb.cuh"

namespace {

using namespace bx;

// int8 [planes, rows, K] row-major -> 3-D map (K, rows, planes), box (128 bytes, box_rows, planes), 128B swizzle.
bool make_map(CUtensorMap* m, const void* base, uint64_t K, uint64_t rows, uint64_t planes, uint32_t box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[3] = {K, rows, planes};
  cuuint64_t strides[2] = {K, rows * K};
  cuuint32_t box[3] = {128, box_rows, (cuuint32_t)planes};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// The same tensor with boxes of `box_rows` rows of ONE plane (the B-operand chunks of the CTA-pair kernels).
bool make_map_chunks(CUtensorMap* m, const void* base, uint64_t K, uint64_t rows, uint64_t planes, uint32_t box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[3] = {K, rows, planes};
  cuuint64_t strides[2] = {K, rows * K};
  cuuint32_t box[3] = {128, box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

template <int TA>
int launch_exact(const CUtensorMap& mw, const CUtensorMap& ma, const ExactEpiParams& ep, int K, cudaStream_t st) {
  using Cfg = GemmCfg<3, 3, TA>;
  static PerDevice configured;
  if (once_per_device(configured, [] {
        return cudaFuncSetAttribute(exact_linear_kernel<TA>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    Cfg::SMEM_BYTES);
      }) != BX_OK)
    return BX_ELAUNCH;
  const int m_tiles = (ep.M + TA - 1) / TA;
  const int n_tiles = (ep.N + WROWS - 1) / WROWS;
  return launch_chained(exact_linear_kernel<TA>, dim3(m_tiles * n_tiles), GEMM_THREADS, Cfg::SMEM_BYTES, st, 0, mw, ma, ep, K, m_tiles);
}

template <int TA>
int launch_exact_splitk(const CUtensorMap& mw, const CUtensorMap& ma, const ExactEpiParams& ep, int K, int split,
                        cudaStream_t st) {
  using Cfg = GemmCfg<3, 3, TA>;
  static PerDevice configured;
  if (once_per_device(configured, [] {
        return cudaFuncSetAttribute(exact_linear_splitk_kernel<TA>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    Cfg::SMEM_BYTES);
      }) != BX_OK)
    return BX_ELAUNCH;
  const int m_tiles = (ep.M + TA - 1) / TA;
  const int n_tiles = (ep.N + WROWS - 1) / WROWS;
  return launch_chained(exact_linear_splitk_kernel<TA>, dim3((unsigned)(m_tiles * n_tiles * split)), GEMM_THREADS, Cfg::SMEM_BYTES, st, split,
                        mw, ma, ep, K, m_tiles);
}

// Split-K with the activation rows as the 128-row operand (exact_linear_rows_splitk_kernel).
template <int TA>
int launch_exact_rows_splitk(const CUtensorMap& mact, const CUtensorMap& mwt, const ExactEpiParams& ep, int K, int split,
                             cudaStream_t st) {
  using Cfg = GemmCfg<3, 3, TA>;
  static PerDevice configured;
  if (once_per_device(configured, [] {
        return cudaFuncSetAttribute(exact_linear_rows_splitk_kernel<TA>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    Cfg::SMEM_BYTES);
      }) != BX_OK)
    return BX_ELAUNCH;
  const int w_tiles = (ep.N + TA - 1) / TA;
  const int row_blocks = (ep.M + WROWS - 1) / WROWS;
  return launch_chained(exact_linear_rows_splitk_kernel<TA>, dim3((unsigned)(w_tiles * row_blocks * split)), GEMM_THREADS, Cfg::SMEM_BYTES, st, split,
                        mact, mwt, ep, K, w_tiles);
}

template <int TA>
int launch_exact_persistent(const CUtensorMap& mw, const CUtensorMap& ma, const ExactEpiParams& ep, int K,
                            cudaStream_t st) {
  using Cfg = GemmCfg<3, 3, TA>;
  static PerDevice configured;
  if (once_per_device(configured, [] {
        return cudaFuncSetAttribute(exact_linear_persistent_kernel<TA>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    Cfg::SMEM_BYTES);
      }) != BX_OK)
    return BX_ELAUNCH;
  const int sms = device_sms();
  if (sms <= 0) return BX_ELAUNCH;
  const int m_tiles = (ep.M + TA - 1) / TA;
  const int n_tiles = (ep.N + WROWS - 1) / WROWS;
  const int total = m_tiles * n_tiles;
  const int grid = total < sms ? total : sms;
  return launch_chained(exact_linear_persistent_kernel<TA>, dim3(grid), GEMM_THREADS, Cfg::SMEM_BYTES, st, 0, mw, ma, ep, K, n_tiles, m_tiles);
}

// CTA pairs resident at a time for a pair kernel (clusters of 2 with its shared memory), cached per device.
template <class Kernel>
int max_active_pairs(Kernel kernel, int smem, PerDevice& cache) {
  const int dev = current_device();
  if (dev < 0) return 0;
  int n = cache.v[dev].load(std::memory_order_acquire);
  if (n > 0) return n;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * 148, 1, 1);
  cfg.blockDim = dim3(GEMM_THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n <= 0) {
    cudaGetLastError();
    return 0;
  }
  cache.v[dev].store(n, std::memory_order_release);
  return n;
}

template <int TA>
int launch_exact_pair(const CUtensorMap& mw, const CUtensorMap& mb, const ExactEpiParams& ep, int K, cudaStream_t st) {
  using Cfg = PairCfg<3, 3, TA>;
  static PerDevice configured, pairs_cache;
  if (once_per_device(configured, [] {
        return cudaFuncSetAttribute(exact_linear_pair_kernel<TA>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    Cfg::SMEM_BYTES);
      }) != BX_OK)
    return BX_ELAUNCH;
  const int pairs = max_active_pairs(exact_linear_pair_kernel<TA>, Cfg::SMEM_BYTES, pairs_cache);
  if (pairs <= 0) return BX_ELAUNCH;
  const int m_tiles = (ep.M + TA - 1) / TA;
  const int n_tiles2 = (ep.N + 2 * WROWS - 1) / (2 * WROWS);
  const int total = m_tiles * n_tiles2;
  const int grid = 2 * (total < pairs ? total : pairs);
  exact_linear_pair_kernel<TA><<<grid, GEMM_THREADS, Cfg::SMEM_BYTES, st>>>(mw, mb, ep, K, n_tiles2, m_tiles);
  return launched(1);
}

template <int TN, bool DBL>
int launch_exact_rows(const CUtensorMap& ma, const CUtensorMap& mw, const ExactEpiParams& ep, int K, cudaStream_t st) {
  using Cfg = RowsCfg<TN, DBL>;
  static PerDevice configured, pairs_cache;
  if (once_per_device(configured, [] {
        return cudaFuncSetAttribute(exact_linear_rows_kernel<TN, DBL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    Cfg::SMEM_BYTES);
      }) != BX_OK)
    return BX_ELAUNCH;
  const int pairs = max_active_pairs(exact_linear_rows_kernel<TN, DBL>, Cfg::SMEM_BYTES, pairs_cache);
  if (pairs <= 0) return BX_ELAUNCH;
  const int n_tiles = (ep.N + TN - 1) / TN;
  const int m_tiles2 = (ep.M + 2 * WROWS - 1) / (2 * WROWS);
  const long total = (long)n_tiles * m_tiles2;
  const int grid = 2 * (int)(total < pairs ? total : pairs);
  exact_linear_rows_kernel<TN, DBL><<<grid, GEMM_THREADS, Cfg::SMEM_BYTES, st>>>(ma, mw, ep, K, n_tiles, m_tiles2);
  return launched(1);
}

template <int TN, int NBUF>
int launch_exact_rows_one(const CUtensorMap& mact, const CUtensorMap& mwt, const ExactEpiParams& ep, int K,
                          cudaStream_t st) {
  using Cfg = GemmCfg<3, 3, TN>;
  static PerDevice configured;
  if (once_per_device(configured, [] {
        return cudaFuncSetAttribute(exact_linear_rows_one_kernel<TN, NBUF>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES);
      }) != BX_OK)
    return BX_ELAUNCH;
  const int sms = device_sms();
  if (sms <= 0) return BX_ELAUNCH;
  const int row_blocks = (ep.M + WROWS - 1) / WROWS;
  const int w_tiles = (ep.N + TN - 1) / TN;
  const long total = (long)row_blocks * w_tiles;
  const int grid = (int)(total < sms ? total : sms);
  // Chained (launch_chained) while a CTA has a few tiles: a decode step of 256 sequences (3.5 tiles per CTA) took 6011 us so, 6041
  // plainly. Plain on long lists: scoring 700 rows (LM head, 81 tiles per CTA) 1732 us plainly, 1760 chained; on other days
  // 1505 : 1522 and 1705 : 1712.
  if (total <= 8L * sms)
    return launch_chained(exact_linear_rows_one_kernel<TN, NBUF>, dim3(grid), GEMM_THREADS, Cfg::SMEM_BYTES, st, 0, mact, mwt, ep, K,
                          row_blocks, w_tiles);
  exact_linear_rows_one_kernel<TN, NBUF><<<grid, GEMM_THREADS, Cfg::SMEM_BYTES, st>>>(mact, mwt, ep, K, row_blocks, w_tiles);
  return launched(1);
}

template <int TA, bool POST>
int launch_int8(const CUtensorMap& mw, const CUtensorMap& ma, const Int8EpiParams& ep, int K, cudaStream_t st) {
  using Cfg = GemmCfg<1, 2, TA>;
  static PerDevice configured;
  if (once_per_device(configured, [] {
        return cudaFuncSetAttribute(int8_linear_kernel<TA, POST>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    Cfg::SMEM_BYTES);
      }) != BX_OK)
    return BX_ELAUNCH;
  const int m_tiles = (ep.M + TA - 1) / TA;
  const int n_tiles = (ep.N + WROWS - 1) / WROWS;
  // POST = false (raw products): its operands may be any tensors, so it does not start before the previous kernel has ended.
  if (POST)
    return launch_chained(int8_linear_kernel<TA, POST>, dim3(m_tiles * n_tiles), GEMM_THREADS, Cfg::SMEM_BYTES, st, 0, mw, ma, ep, K, m_tiles);
  int8_linear_kernel<TA, POST><<<m_tiles * n_tiles, GEMM_THREADS, Cfg::SMEM_BYTES, st>>>(mw, ma, ep, K, m_tiles);
  return launched(1);
}

template <int TA, bool POST>
int launch_int8_persistent(const CUtensorMap& mw, const CUtensorMap& ma, const Int8EpiParams& ep, int K,
                           cudaStream_t st) {
  using Cfg = GemmCfg<1, 2, TA>;
  static PerDevice configured;
  if (once_per_device(configured, [] {
        return cudaFuncSetAttribute(int8_linear_persistent_kernel<TA, POST>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES);
      }) != BX_OK)
    return BX_ELAUNCH;
  const int sms = device_sms();
  if (sms <= 0) return BX_ELAUNCH;
  const int m_tiles = (ep.M + TA - 1) / TA;
  const int n_tiles = (ep.N + WROWS - 1) / WROWS;
  const int total = m_tiles * n_tiles;
  const int grid = total < sms ? total : sms;
  // POST = false (raw products): its operands may be any tensors, so it does not start before the previous kernel has ended.
  if (POST)
    return launch_chained(int8_linear_persistent_kernel<TA, POST>, dim3(grid), GEMM_THREADS, Cfg::SMEM_BYTES, st, 0, mw, ma, ep, K, n_tiles, m_tiles);
  int8_linear_persistent_kernel<TA, POST><<<grid, GEMM_THREADS, Cfg::SMEM_BYTES, st>>>(mw, ma, ep, K, n_tiles, m_tiles);
  return launched(1);
}

template <int TA>
int launch_int8_splitk(const CUtensorMap& mw, const CUtensorMap& ma, const Int8EpiParams& ep, int K, int split,
                       cudaStream_t st) {
  using Cfg = GemmCfg<1, 2, TA>;
  static_assert((TA + SPLITK_MAX - 1) * WROWS * 8 <= Cfg::STAGES * Cfg::STAGE_BYTES, "partial columns fit in the ring");
  static PerDevice configured;
  if (once_per_device(configured, [] {
        return cudaFuncSetAttribute(int8_linear_splitk_kernel<TA>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    Cfg::SMEM_BYTES);
      }) != BX_OK)
    return BX_ELAUNCH;
  const int m_tiles = (ep.M + TA - 1) / TA;
  const int n_tiles = (ep.N + WROWS - 1) / WROWS;
  return launch_chained(int8_linear_splitk_kernel<TA>, dim3((unsigned)(m_tiles * n_tiles * split)), GEMM_THREADS, Cfg::SMEM_BYTES, st, split,
                        mw, ma, ep, K, m_tiles);
}

template <int TA>
int launch_bmm_limb(const CUtensorMap& mb, const CUtensorMap& ma, const BmmEpiParams& ep, int Z, int K16, cudaStream_t st) {
  using Cfg = GemmCfg<3, 3, TA>;
  static PerDevice configured;
  if (once_per_device(configured, [] {
        return cudaFuncSetAttribute(bmm_limb_kernel<TA>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES);
      }) != BX_OK)
    return BX_ELAUNCH;
  const int m_tiles = (ep.M + TA - 1) / TA, n_tiles = (ep.N + WROWS - 1) / WROWS;
  const long grid = (long)Z * m_tiles * n_tiles;
  if (grid > 0x7fffffffL) return BX_EARG;
  bmm_limb_kernel<TA><<<(unsigned)grid, GEMM_THREADS, Cfg::SMEM_BYTES, st>>>(mb, ma, ep, K16, n_tiles, m_tiles);
  return launched(1);
}

template <class TX>
void launch_bmm_pack(const void* x, int64_t sz, int64_t sr, int64_t sk, int8_t* planes, int Z, int R, int K, int K16,
                     cudaStream_t st) {
  const int64_t total = (int64_t)Z * R * (K16 / 16);
  int64_t blocks = (total + 255) / 256;
  if (blocks > 148 * 32) blocks = 148 * 32;
  bmm_pack_kernel<TX><<<(unsigned)blocks, 256, 0, st>>>((const TX*)x, sz, sr, sk, planes, Z, R, K, K16);
}

template <bool POST>
int run_int8(const int8_t* a, const int8_t* w, const Int8EpiParams& ep, int K, int tile_rows, cudaStream_t st) {
  const int M = ep.M, N = ep.N;
  if (!a || !w || M < 0 || N <= 0 || K <= 0 || K % 16 || K >= 65536 || !aligned16(a) || !aligned16(w)) return BX_EARG;
  if (M == 0) return BX_OK;
  int ta = tile_rows;
  bool persistent = false;
  if (ta < 0) {                       // negative: that tile size on the persistent kernel
    ta = -ta;
    persistent = true;
  } else if (ta == 0) {
    const long n_tiles = (N + WROWS - 1) / WROWS;
    ta = M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : (n_tiles * ((M + 127) / 128) >= 90 ? 128 : 64);
    // 64-row tiles that would cover less than half of the SMs: with a short K, 32-row tiles (wo at 256 rows:
    // 12.7 -> 10.6 us); with a long K the 64-row tiles stay and K is split over clusters below
    if (ta == 64 && M > 64 && K < 4096 && n_tiles * ((M + 63) / 64) * 2 <= 148) ta = 32;
    // more tiles than SMs: one CTA per SM with the epilogue of a tile behind the MMAs of the next
    persistent = n_tiles * ((M + ta - 1) / ta) > 148;
  }
  // Split-K over a cluster of CTAs (fused post only): 200 + rows (10000 S + 200 + rows: clusters of exactly S) asks
  // for it; automatic when the tile list covers less than half of the SMs and K is long enough for two K blocks per
  // slice, with as many slices (2, 4 or 8) as keep the CTA count within the SMs.
  int split = 0;
  if (POST) {
    int want = 0;
    if (ta >= 10000) { want = ta / 10000; ta %= 10000; if (want != 2 && want != 4 && want != 8) return BX_EARG; }
    if (ta >= 200 && ta < 300) {
      ta -= 200;
      if (ta != 16 && ta != 32 && ta != 64) return BX_EARG;
      split = want ? want : SPLITK_MAX;
    } else if (want) {
      return BX_EARG;
    } else if (tile_rows == 0 && !persistent && (ta == 16 || ta == 32 || ta == 64)) {
      const long tiles = ((N + WROWS - 1) / WROWS) * (long)((M + ta - 1) / ta);
      if (tiles * 2 <= 148) split = (int)(148 / tiles);
      if (split > 8) split = 8;
    }
    if (split > 0) {
      const int nkb = (K + BKB - 1) / BKB;
      if (split > nkb / 2) split = nkb / 2;
      while (split & (split - 1)) --split;
      if (tile_rows == 0 && split > 4) split = 4;
    }
  }
  CUtensorMap mw, ma;
  if (!make_map(&mw, w, (uint64_t)K, (uint64_t)N, 1, WROWS)) return BX_ELAUNCH;
  if (!make_map(&ma, a, (uint64_t)K, (uint64_t)M, 2, (uint32_t)ta)) return BX_ELAUNCH;
  if constexpr (POST) {
    if (split >= 2) {
      switch (ta) {
        case 16: return launch_int8_splitk<16>(mw, ma, ep, K, split, st);
        case 32: return launch_int8_splitk<32>(mw, ma, ep, K, split, st);
        default: return launch_int8_splitk<64>(mw, ma, ep, K, split, st);
      }
    }
  }
  if (persistent) {
    switch (ta) {
      case 16: return launch_int8_persistent<16, POST>(mw, ma, ep, K, st);
      case 32: return launch_int8_persistent<32, POST>(mw, ma, ep, K, st);
      case 64: return launch_int8_persistent<64, POST>(mw, ma, ep, K, st);
      case 128: return launch_int8_persistent<128, POST>(mw, ma, ep, K, st);
      default: return BX_EARG;
    }
  }
  switch (ta) {
    case 16: return launch_int8<16, POST>(mw, ma, ep, K, st);
    case 32: return launch_int8<32, POST>(mw, ma, ep, K, st);
    case 64: return launch_int8<64, POST>(mw, ma, ep, K, st);
    case 128: return launch_int8<128, POST>(mw, ma, ep, K, st);
    default: return BX_EARG;
  }
}

// What a tile list takes, in units of 10 ns: launch + waves of 148 tiles x (K blocks x block + tile). Fitted to 1026 pairs of a
// batch (128 .. 4096 rows) and a shape of weights (83 shapes, N 512 .. 128256, K 256 .. 14336; flushed L2), the lists with residual
// entries and those without on their own. Single times are off by up to 10 %; what counts is which form is ahead.
struct ListCost {
  int launch, block, tile;
  long of(long tiles, long nkb, long more = 0) const { return launch + (tiles + 147) / 148 * (block * nkb + tile + more); }
};
struct ListCosts {
  ListCost act64, act48, act32, act48p, act32p, w64, w48;     // activation rows per tile (p: persistent), weight rows per tile
};
constexpr ListCosts LIST_PLAIN = {{182, 71, 572}, {678, 62, 496}, {330, 60, 638}, {1008, 63, 131}, {877, 58, 90},
                                  {1274, 65, 335}, {1451, 60, 154}};
constexpr ListCosts LIST_RESIDUAL = {{0, 94, 888}, {467, 72, 742}, {360, 70, 786}, {1417, 68, 108}, {210, 63, 436},
                                     {1496, 68, 319}, {1445, 63, 138}};
// More for a tile of 64 / 48 weight rows where the rows of y start off 32-byte boundaries: they are written row by row.
constexpr int ODD_W64 = 580, ODD_W48 = 410;

// The tile form (a tile_rows value) of an exact linear.
int exact_linear_auto(int M, int N, int K, bool residual) {
  // Activation rows per CTA: the size that needs the fewest wave-rows (below); a tile list of more than two waves
  // goes to the persistent kernel (48 rows, overlapped epilogue).
  const long n_tiles = (N + WROWS - 1) / WROWS, nkb = (K + BKB - 1) / BKB;
  auto act_tiles = [&](int rows) { return n_tiles * ((M + rows - 1) / rows); };
  int ta = M <= 16 ? 16 : M <= 32 ? 32 : 48;
  if (M > 48) {
    // waves of 148 CTAs x (rows of a tile + a fixed cost of about 16 rows' worth of prologue and epilogue)
    long best = -1;
    const int cand[3] = {64, 48, 32};
    for (int i = 0; i < 3; ++i) {
      const long cost = ((act_tiles(cand[i]) + 147) / 148) * (cand[i] + 16);
      if (best < 0 || cost < best) { best = cost; ta = cand[i]; }
    }
  }
  bool persistent = ta <= 48 && act_tiles(ta) > 2 * 148;
  if (ta == 64 && K <= 4096 && act_tiles(48) > 2 * 148) { ta = 48; persistent = true; }
  const long blocks = (M + WROWS - 1) / WROWS, w64_tiles = blocks * ((N + 63) / 64);
  const bool full_blocks = 10 * blocks * WROWS <= 11 * (((M + 47) / 48) * 48L);     // 128-row blocks pad about as little as 48
  // Few tiles: K split over clusters, so that the tile list covers the SMs.
  if (!persistent && M >= WROWS && K >= 8192) {
    // a batch that fills blocks of 128 rows (the down projection at 256 rows): activation rows on the MMA M side, 64 weight
    // rows per tile, as many K slices as keep the CTA count within the SMs
    if (full_blocks && w64_tiles * 2 <= 148) return w64_tiles * 4 <= 148 ? 40764 : 20764;
    // 64-row tiles with K split over CTA pairs read less shared memory per product than one wave of 32-row tiles
    // (measured 47 -> 39 us)
    if (M > 128 && act_tiles(64) * 2 <= 148) return 20264;
  }
  if (!persistent && M <= 128 && ta != 48 && act_tiles(ta) * 2 <= 148) {
    int split = (int)(148 / act_tiles(ta));
    const int lim = ta == 16 ? splitk_limit<16>() : ta == 32 ? splitk_limit<32>() : splitk_limit<64>();
    if (split > lim) split = lim;
    if (split > nkb / 2) split = (int)(nkb / 2);
    while (split & (split - 1)) --split;
    // at most 4: clusters of 8 measured 1.3 - 1.5 x slower on these shapes (fewer of them are resident at a time)
    if (split > 4) split = 4;
    return split >= 2 ? 10000 * split + 200 + ta : ta;
  }
  if (M < WROWS) return persistent ? -ta : ta;
  // From 128 rows on: the activation rows on the MMA M side with 64 weight rows per tile (wider MMAs, residual lists
  // warp-uniform, epilogue not overlapped) or 48 (two accumulator buffers), or 48 activation rows on the persistent kernel,
  // where one of them is predicted to be faster than what the rules so far give. Over the fitted sizes that is 0.95 of the time
  // of those rules (8 of 1026 more than 2 % slower, with residual entries 7), and 0.96 / 0.98 of that of a choice by waves with
  // three fixed costs, which took up to 1.6 x as long (N 9601, K 272, 160 rows 22.5 -> 31.7 us; N 4096, K 14336, 560 rows
  // 223 -> 259 us).
  const int form = persistent ? (ta == 48 && full_blocks ? 664 : -ta) : ta;
  const ListCosts& c = residual ? LIST_RESIDUAL : LIST_PLAIN;
  const long t48 = act_tiles(48);
  const long cost[3] = {c.w64.of(w64_tiles, nkb, N % 4 ? ODD_W64 : 0), c.w48.of(blocks * ((N + 47) / 48), nkb, N % 4 ? ODD_W48 : 0),
                        c.act48p.of(t48, nkb)};
  const long given = form == 664 ? cost[0] : form == -48 ? cost[2] : form == -32 ? c.act32p.of(act_tiles(32), nkb)
                   : form == 64 ? c.act64.of(act_tiles(64), nkb) : form == 48 ? c.act48.of(t48, nkb)
                   : c.act32.of(act_tiles(32), nkb);
  const int forms[3] = {664, 648, -48};
  const int best = cost[0] <= cost[1] && cost[0] <= cost[2] ? 0 : cost[1] <= cost[2] ? 1 : 2;
  return 100 * cost[best] < 99 * given ? forms[best] : form;
}

}  // namespace

extern "C" {

int bx_version(void) { return 1; }

long long bx_launch_count(void) { return g_launches; }

int bx_device_status(void) { return status_read(); }

int bx_clear_device_status(void) { return status_clear(); }

int bx_set_device_status(int value) { return status_write(value); }

int bx_i8_tensor_peak(int iters, int repeats, double* tops, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (iters < 4 || iters > (1 << 22) || repeats < 1 || repeats > 64 || !tops) return BX_EARG;
  static PerDevice configured;
  if (once_per_device(configured, [] {
        return cudaFuncSetAttribute(i8_peak_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PEAK_SMEM);
      }) != BX_OK)
    return BX_ELAUNCH;
  const int sms = device_sms();
  if (sms <= 0) return BX_ELAUNCH;
  cudaStream_t st = (cudaStream_t)stream;
  cudaEvent_t e0, e1;
  if (cudaEventCreate(&e0) != cudaSuccess) return BX_ELAUNCH;
  if (cudaEventCreate(&e1) != cudaSuccess) { cudaEventDestroy(e0); return BX_ELAUNCH; }
  const double ops = (double)sms * iters * 4.0 * 2.0 * 128.0 * PEAK_N * 32.0;
  double best = 0.0, sum = 0.0;
  int rc = BX_OK;
  i8_peak_kernel<<<sms, 128, PEAK_SMEM, st>>>(iters / 4);          // warm-up
  for (int r = 0; r < repeats && rc == BX_OK; ++r) {
    cudaEventRecord(e0, st);
    i8_peak_kernel<<<sms, 128, PEAK_SMEM, st>>>(iters);
    cudaEventRecord(e1, st);
    float ms = 0.f;
    if (cudaEventSynchronize(e1) != cudaSuccess || cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess || ms <= 0.f) {
      rc = BX_ELAUNCH;
      break;
    }
    const double t = ops / (ms * 1e-3) / 1e12;
    best = t > best ? t : best;
    sum += t;
    g_launches += 1;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (rc != BX_OK || cudaGetLastError() != cudaSuccess) return BX_ELAUNCH;
  tops[0] = best;
  tops[1] = sum / repeats;
  return BX_OK;
}

size_t bx_exact_linear_scratch_bytes(int M, int K) { return (size_t)3 * (size_t)M * (size_t)K; }

int bx_split_limbs(const int32_t* q, int64_t ldq, int8_t* a8, int M, int K, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!q || !a8 || M < 0 || K <= 0 || K % 16 || ldq % 4 || ldq < K || !aligned16(q) || !aligned16(a8)) return BX_EARG;
  if (M == 0) return BX_OK;
  const int64_t total = (int64_t)M * (K / 16);
  int blocks = (int)((total + 255) / 256);
  if (blocks > 148 * 16) blocks = 148 * 16;
  split_limbs_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(q, ldq, a8, M, K);
  return launched(1);
}

static int exact_linear_core(const int32_t* q, int64_t ldq, const int64_t* sh, const int8_t* limbs, const int64_t* d,
                             const int64_t* g, const int32_t* cnt, const int32_t* ec, const int64_t* ev, int R,
                             const int8_t* planes, int64_t* y, int32_t* flag, int M, int N, int K, int checked,
                             int tile_rows, int early, void* stream) {
  int8_t* scratch = const_cast<int8_t*>(planes);
  cudaStream_t st = (cudaStream_t)stream;
  int ta = tile_rows == 0 ? exact_linear_auto(M, N, K, cnt != nullptr) : tile_rows;
  const bool persistent = ta < 0;     // negative: that tile size on the persistent kernel (16, 32, 48)
  if (persistent) {
    ta = -ta;
    if (ta != 16 && ta != 32 && ta != 48) return BX_EARG;
  }
  int want_split = 0;                 // 10000 S + 200 + rows: split-K over clusters of exactly S CTAs
  if (ta >= 10000) {
    want_split = ta / 10000;
    ta %= 10000;
    if (!((ta >= 200 && ta < 300) || ta == 764) || (want_split != 2 && want_split != 4 && want_split != 8)) return BX_EARG;
  }
  if (ta == 764) {
    int split = want_split ? want_split : 2;
    const int nkb = (K + BKB - 1) / BKB;
    if (split > nkb / 2) split = nkb / 2;
    while (split & (split - 1)) --split;
    if (split >= 2) {
      CUtensorMap mact, mwt;
      if (!make_map(&mact, scratch, (uint64_t)K, (uint64_t)M, 3, WROWS)) return BX_ELAUNCH;
      if (!make_map(&mwt, limbs, (uint64_t)K, (uint64_t)N, 3, 64)) return BX_ELAUNCH;
      ExactEpiParams ep{q, ldq, sh, d, g, cnt, ec, ev, R, y, flag, M, N, checked, early};
      return launch_exact_rows_splitk<64>(mact, mwt, ep, K, split, st);
    }
    ta = 664;                          // K too short to split: the same tile shape on the one-CTA kernel
  }
  if (ta == 416 || ta == 432 || ta == 448) {          // 400 + rows: that tile size on the CTA-pair kernel
    ta -= 400;
    CUtensorMap mw, mb;
    if (!make_map(&mw, limbs, (uint64_t)K, (uint64_t)N, 3, WROWS)) return BX_ELAUNCH;
    if (!make_map_chunks(&mb, scratch, (uint64_t)K, (uint64_t)M, 3, (uint32_t)(ta / 2))) return BX_ELAUNCH;
    ExactEpiParams ep{q, ldq, sh, d, g, cnt, ec, ev, R, y, flag, M, N, checked, early};
    switch (ta) {
      case 16: return launch_exact_pair<16>(mw, mb, ep, K, st);
      case 32: return launch_exact_pair<32>(mw, mb, ep, K, st);
      default: return launch_exact_pair<48>(mw, mb, ep, K, st);
    }
  }
  if (ta == 516 || ta == 532 || ta == 548 || ta == 564 || ta == 580) {
    // 500 + weight rows per tile: activation rows on the MMA M side, CTA pairs (16 .. 48: two accumulator buffers)
    ta -= 500;
    CUtensorMap ma, mw;
    if (!make_map(&ma, scratch, (uint64_t)K, (uint64_t)M, 3, WROWS)) return BX_ELAUNCH;
    if (!make_map_chunks(&mw, limbs, (uint64_t)K, (uint64_t)N, 3, (uint32_t)(ta / 2))) return BX_ELAUNCH;
    ExactEpiParams ep{q, ldq, sh, d, g, cnt, ec, ev, R, y, flag, M, N, checked, early};
    switch (ta) {
      case 16: return launch_exact_rows<16, true>(ma, mw, ep, K, st);
      case 32: return launch_exact_rows<32, true>(ma, mw, ep, K, st);
      case 48: return launch_exact_rows<48, true>(ma, mw, ep, K, st);
      case 64: return launch_exact_rows<64, false>(ma, mw, ep, K, st);
      default: return launch_exact_rows<80, false>(ma, mw, ep, K, st);
    }
  }
  if (ta == 616 || ta == 632 || ta == 648 || ta == 664 || ta == 680) {
    // 600 + weight rows per tile: activation rows on the MMA M side, one CTA (16 .. 48: two accumulator buffers)
    ta -= 600;
    CUtensorMap mact, mwt;
    if (!make_map(&mact, scratch, (uint64_t)K, (uint64_t)M, 3, WROWS)) return BX_ELAUNCH;
    if (!make_map(&mwt, limbs, (uint64_t)K, (uint64_t)N, 3, (uint32_t)ta)) return BX_ELAUNCH;
    ExactEpiParams ep{q, ldq, sh, d, g, cnt, ec, ev, R, y, flag, M, N, checked, early};
    switch (ta) {
      case 16: return launch_exact_rows_one<16, 2>(mact, mwt, ep, K, st);
      case 32: return launch_exact_rows_one<32, 2>(mact, mwt, ep, K, st);
      case 48: return launch_exact_rows_one<48, 2>(mact, mwt, ep, K, st);
      case 64: return launch_exact_rows_one<64, 1>(mact, mwt, ep, K, st);
      default: return launch_exact_rows_one<80, 1>(mact, mwt, ep, K, st);
    }
  }
  // Split-K over a cluster of CTAs: 200 + activation rows per tile.
  int split = 0;
  if (ta >= 200) {
    ta -= 200;
    split = want_split ? want_split : SPLITK_MAX;
    if (ta != 16 && ta != 32 && ta != 64) return BX_EARG;
  }
  if (split > 0) {
    const int nkb = (K + BKB - 1) / BKB;
    const int lim = ta == 16 ? splitk_limit<16>() : ta == 32 ? splitk_limit<32>() : splitk_limit<64>();
    if (split > lim) split = lim;
    if (split > nkb / 2) split = nkb / 2;                      // at least two K blocks per slice
    while (split & (split - 1)) --split;   // clusters of 2, 4 or 8: a cluster of 6 ran 1.6 x slower than one of 4
  }
  CUtensorMap mw, ma;
  if (!make_map(&mw, limbs, (uint64_t)K, (uint64_t)N, 3, WROWS)) return BX_ELAUNCH;
  if (!make_map(&ma, scratch, (uint64_t)K, (uint64_t)M, 3, (uint32_t)ta)) return BX_ELAUNCH;
  ExactEpiParams ep{q, ldq, sh, d, g, cnt, ec, ev, R, y, flag, M, N, checked, early};
  if (split >= 2) {
    switch (ta) {
      case 16: return launch_exact_splitk<16>(mw, ma, ep, K, split, st);
      case 32: return launch_exact_splitk<32>(mw, ma, ep, K, split, st);
      default: return launch_exact_splitk<64>(mw, ma, ep, K, split, st);
    }
  }
  if (persistent) {
    switch (ta) {
      case 16: return launch_exact_persistent<16>(mw, ma, ep, K, st);
      case 32: return launch_exact_persistent<32>(mw, ma, ep, K, st);
      default: return launch_exact_persistent<48>(mw, ma, ep, K, st);
    }
  }
  switch (ta) {
    case 16: return launch_exact<16>(mw, ma, ep, K, st);
    case 32: return launch_exact<32>(mw, ma, ep, K, st);
    case 48: return launch_exact<48>(mw, ma, ep, K, st);
    case 64: return launch_exact<64>(mw, ma, ep, K, st);
    case 80: return launch_exact<80>(mw, ma, ep, K, st);
    default: return BX_EARG;
  }
}

int bx_exact_norm(int mode, const void* xin, const int64_t* yin, const int64_t* ids, const int64_t* gm,
                  const int64_t* ge, int64_t* xo, int32_t* q, int64_t* sh, int8_t* a8, int32_t* flag, int M, int D,
                  int do_norm, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!xin || !flag || M < 0 || D < 32 || D > 4096 || (D & (D - 1))) return BX_EARG;
  if ((mode == 0 && !ids) || (mode == 1 && !yin) || mode < 0 || mode > 2) return BX_EARG;
  if (do_norm && (!gm || !ge || !q || !sh)) return BX_EARG;
  if (M == 0) return BX_OK;
  int lg = 0;
  while ((1 << lg) < D) ++lg;
  cudaStream_t st = (cudaStream_t)stream;
  const i64* y = (const i64*)yin; const i64* id = (const i64*)ids;
  const int sms = device_sms();
  if (sms <= 0) return BX_ELAUNCH;
  // rows of D int64, D a multiple of 32: every access is as wide as the base pointers are aligned
  const bool wide = aligned_to(xin, 32) && aligned_to(yin, 32) && aligned_to(gm, 32) && aligned_to(ge, 32) && aligned_to(xo, 32) &&
                    aligned_to(q, 16) && aligned_to(a8, 4);
#define BX_NORM_LAUNCH(MODE, NT, Q) \
  return launch_chained(norm_kernel<MODE, NT, Q>, dim3(even_grid(M, sms * (1024 / NT))), NT, 0, st, 0, xin, y, id, (const i64*)gm, \
                        (const i64*)ge, (i64*)xo, q, (i64*)sh, a8, flag, M, D, lg, do_norm, wide)
#define BX_NORM_MODES(NT, Q) \
  if (mode == 0) BX_NORM_LAUNCH(0, NT, Q); else if (mode == 1) BX_NORM_LAUNCH(1, NT, Q); else BX_NORM_LAUNCH(2, NT, Q)
  if (D <= 512) { BX_NORM_MODES(128, 1); }
  else if (D == 1024) { BX_NORM_MODES(256, 1); }
  else if (D == 2048) { BX_NORM_MODES(512, 1); }
  else { BX_NORM_MODES(512, 2); }
#undef BX_NORM_MODES
#undef BX_NORM_LAUNCH
}

int bx_exact_qkv(const int64_t* y, const int64_t* cos, const int64_t* sin, const int64_t* pos,
                 const int64_t* slot, int8_t* cache, int64_t sc_nb, int64_t sc_h, int64_t sc_bs, int bs, int32_t* q,
                 int64_t* sh, int32_t* flag, int N, int H, int HKV, int HD, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!y || !cos || !sin || !pos || !q || !sh || !flag || N < 0) return BX_EARG;
  if ((HD != 64 && HD != 128) || HKV <= 0 || H % HKV || (cache && (!slot || bs <= 0))) return BX_EARG;
  if (N == 0) return BX_OK;
  QkvParams p{(const i64*)y, (const i64*)cos, (const i64*)sin, (const i64*)pos, (const i64*)slot, cache, sc_nb, sc_h,
              sc_bs, bs, q, (i64*)sh, flag, H, HKV, HD};
  return launch_chained(qkv_kernel, dim3(N, HKV), HD / 2, 0, (cudaStream_t)stream, 0, p);
}

int bx_kv_store(int8_t* cache, int64_t sc_nb, int64_t sc_h, int64_t sc_bs, int bs, const int64_t* slot,
                const int64_t* k, int64_t skz, int64_t skh, const int64_t* v, int64_t svz, int64_t svh, int N,
                int HKV, int HD, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!cache || !slot || !k || !v || bs <= 0 || N < 0 || HKV <= 0 || HD <= 0) return BX_EARG;
  if (N == 0) return BX_OK;
  kv_store_kernel<<<dim3(N, HKV), 64, 0, (cudaStream_t)stream>>>(cache, (const i64*)slot, (const i64*)k, (const i64*)v,
                                                                 skz, skh, svz, svh, sc_nb, sc_h, sc_bs, bs, HD);
  return launched(1);
}

int bx_exact_attn_out(const int64_t* num, const int64_t* den, int32_t* q, int64_t* sh, int8_t* a8, int N, int K2,
                      int HD, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!num || !den || !q || !sh || N < 0 || K2 <= 0 || K2 > AO_THREADS * AO_EPT || HD <= 0 || K2 % HD ||
      K2 / HD > AO_MAXH)
    return BX_EARG;
  if (N == 0) return BX_OK;
  const i64 *nm = (const i64*)num, *dn = (const i64*)den;
  if (HD % 4)
    return launch_chained(attn_out_any_kernel, dim3(N), AO_THREADS, 0, (cudaStream_t)stream, 0, nm, dn, q, (i64*)sh, a8, N, K2, HD);
  const bool wide = aligned_to(num, 32) && aligned_to(q, 16) && aligned_to(a8, 4);
  return launch_chained(K2 <= 1024 ? attn_out_kernel<256, 1> : K2 <= 2048 ? attn_out_kernel<512, 1> : attn_out_kernel<512, 2>, dim3(N),
                        K2 <= 1024 ? 256 : 512, 0, (cudaStream_t)stream, 0, nm, dn, q, (i64*)sh, a8, N, K2, HD, wide);
}

// Rows at a time in a CTA of the persistent SiLU kernels: as many as its threads can hold, but no more than the rows there
// are for an SM.
static int silu_groups(int N, int FF, int sms) {
  const int room = FF <= 4096 ? 4 : FF <= 8192 ? 2 : 1, rows = N > 2 * sms ? 4 : N > sms ? 2 : 1;
  return room < rows ? room : rows;
}

int bx_exact_silu_quant(const int64_t* y, const int64_t* lut, int32_t* q, int64_t* sh, int8_t* a8, int32_t* flag,
                        int N, int FF, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!y || !lut || !q || !sh || !flag || N < 0 || FF <= 0 || FF > SILU_THREADS * 28) return BX_EARG;
  if (N == 0) return BX_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const bool wide = aligned_to(y, 32) && aligned_to(q, 16) && aligned_to(a8, 4);
  const int sms = device_sms();
  if (sms <= 0) return BX_ELAUNCH;
  // Many rows: one persistent CTA per SM, 2^-f table in shared memory (copied in about 4 us); up to 128 rows a row over a
  // cluster, with gathers from L2 (us, cluster : persistent, FF 8192: 64 rows 8.0 : 10.4, 100 rows 10.7 : 10.8, 200 rows 18.8 : 17.5;
  // FF 4096: 64 rows 5.4 : 9.4, 256 rows 13.8 : 11.8; FF 14336: 64 rows 13.8 : 15.4).
  if (FF % 4 == 0 && N > 128) {
    static PerDevice configured;
    const int smem = SILU_TABLE * 8;
    if (once_per_device(configured, [smem] {
          cudaError_t e = cudaSuccess;
          for (auto* k : {silu_persistent_kernel<256, 4>, silu_persistent_kernel<512, 2>, silu_persistent_kernel<512, 4>,
                          silu_persistent_kernel<1024, 2>, silu_persistent_kernel<1024, 4>})
            if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
          return e;
        }) != BX_OK)
      return BX_ELAUNCH;
    const int groups = silu_groups(N, FF, sms);
    auto* kernel = FF > 8192 ? silu_persistent_kernel<1024, 4> : FF > 4096 ? (groups == 2 ? silu_persistent_kernel<512, 4> : silu_persistent_kernel<1024, 2>)
                   : groups == 4 ? silu_persistent_kernel<256, 4> : groups == 2 ? silu_persistent_kernel<512, 2> : silu_persistent_kernel<1024, 2>;
    return launch_chained(kernel, dim3(even_grid((N + groups - 1) / groups, sms)), SILU_P_THREADS, smem, st, 0, (const i64*)y, (const i64*)lut, q,
                          (i64*)sh, a8, flag, N, FF, wide);
  }
  if (FF % 4 == 0 && FF >= 1024) {     // decode batches: a row over a cluster
    const int cl = N * 8 <= sms ? 8 : 4, per = (FF / 4 + cl - 1) / cl;
    return launch_chained(per <= SILU_CL_THREADS ? silu_cluster_kernel<1> : per <= 2 * SILU_CL_THREADS ? silu_cluster_kernel<2> : silu_cluster_kernel<4>,
                          dim3(cl * N), SILU_CL_THREADS, 0, st, cl, (const i64*)y, (const i64*)lut, q, (i64*)sh, a8, flag, N, FF, wide);
  }
  const int ept = (FF + SILU_THREADS - 1) / SILU_THREADS;
  return launch_chained(ept <= 4 ? silu_kernel<4> : ept <= 16 ? silu_kernel<16> : silu_kernel<28>, dim3(N), SILU_THREADS, 0, st, 0,
                        (const i64*)y, (const i64*)lut, q, (i64*)sh, a8, flag, N, FF);
}

constexpr int BX_ENOFIT = -100;
#ifndef BX_ATT_CHUNK
#define BX_ATT_CHUNK 512
#endif

// How the persistent streaming kernel (variants 5: 8 consumer warps, 6: 4) would run.
struct StreamPlan {
  int warps, per_sm, stages;      // per_sm 0: it does not fit
  bool chunked, table;            // scores of long contexts in scratch; with the compact weight table
  int64_t cap;                    // keys whose scores stay in shared memory
  size_t smem;
};

// chunked: scores of contexts beyond `cap` in the caller's scratch; else in shared memory for the widest context.
// table: bytes of the weight table's form in shared memory, 0: none.
static StreamPlan stream_plan(int NW, int64_t max_keys, bool chunked, int table) {
  const int KEYS = 8 * NW, STAGE = KEYS * 256;
  StreamPlan p{NW, 0, 0, chunked, false, chunked ? BX_ATT_CHUNK : (max_keys + KEYS - 1) / KEYS * KEYS, 0};  // chunks: a multiple of 32 NW keys
  if (p.cap / 32 > ATT6_MAXGROUPS) return p;
  int64_t fixed = 1024 + p.cap * 32 + (int64_t)sizeof(Attn6Small) + 1024 /* request order */;
  auto stages = [&](int64_t used) { return (int)((227 * 1024 / p.per_sm - 1024 - used) / STAGE); };
  for (p.per_sm = NW == 4 ? 4 : 2; p.per_sm >= 1; --p.per_sm) {  // most CTAs per SM that still leave a ring of 4 stages
    p.stages = stages(fixed);
    if (p.stages >= 4 || (p.per_sm == 1 && p.stages >= 3)) break;
  }
  if (p.per_sm < 1) return p;
  // The compact weight table where it costs neither a CTA nor the ring: 256 sequences of 512 .. 768 keys 155 -> 133 us; a
  // step that had to give up CTAs for it (and the cluster kernels, five small CTAs to an SM) lost up to 35 %. With
  // pages of 16 keys that is: tables of up to 64 keys, 592 .. 832, 1360 .. 1888, and all that are chunked; for the 2 KB of products
  // up to 512 keys, 592 .. 1280, 1360 .. 2336, and all that are chunked.
  p.table = table && stages(fixed + table) >= 4;
  if (p.table) {
    fixed += table;
    p.stages = stages(fixed);
  }
  if (p.stages > ATT6_MAXNS) p.stages = ATT6_MAXNS;
  p.smem = (size_t)fixed + (size_t)p.stages * STAGE;
  return p;
}

constexpr int64_t STREAM_PAIRS = 2 * 148;         // fewer (request, KV head) pairs than this leave SMs idle: cluster kernels

static bool stream_page_ok(int NW, int bs) { return bs <= 8 * NW && 8 * NW % bs == 0 && 32 % bs == 0; }

// The automatic choice, by CTAs that fit on an SM beside the score buffer: four 4-warp CTAs, else two 8-warp CTAs, else two or
// three 4-warp CTAs, else, with scratch, chunks; per_sm 0: the cluster kernels (they stream better than one CTA per SM).
static StreamPlan stream_auto(int64_t pairs, int64_t max_keys, int bs, bool scratch, int table) {
  const StreamPlan none{};
  if (pairs < STREAM_PAIRS) return none;
  const int tries[3][2] = {{4, 4}, {8, 2}, {4, 2}};
  for (int t = 0; t < 3; ++t) {
    const StreamPlan p = stream_plan(tries[t][0], max_keys, false, table);
    if (stream_page_ok(tries[t][0], bs) && p.per_sm >= tries[t][1]) return p;
  }
  if (!scratch) return none;
  // Chunks. Without the compact table four 4-warp CTAs per SM serve many pairs best (us, 4 : 8 warps; 64 sequences of 64 .. 8192
  // keys 311 : 307, 128 of 32 .. 256 / 64 .. 2048 / 64 .. 8192 39 : 45, 146 : 152, 512 : 499, 256 of the same 61 : 73, 246 : 260,
  // 917 : 945), few pairs two of 8 warps (48 sequences of 64 .. 8192 keys 300 : 244). With it 8 warps at any number of pairs (256
  // sequences of 64 .. 2048 / 64 .. 8192 keys 215 : 246, 731 : 917), which batches of contexts much shorter than their block
  // table pay for (256 of 8 .. 64 / 32 .. 256 / 200 .. 600 keys 50 : 41, 68 : 61, 108 : 109); the host does not know the contexts, and
  // a second launch that leaves at once where it is not wanted took 8 us.
  const int NW = !table && pairs >= 1024 ? 4 : 8;
  const StreamPlan p = stream_plan(NW, max_keys, true, table);
  return stream_page_ok(NW, bs) && p.per_sm >= 2 ? p : none;
}

// shift: bit 8 says that the products lie behind the entries; without it those serve an exact table too.
static CompactTable compact_table(const bx_compact_table* c) {
  const double* products = c->shift & 256 ? reinterpret_cast<const double*>(c->tab + CT_BYTES / 4) : nullptr;
  return CompactTable{c->tab, products, c->window, c->slack, c->factor, c->mtop, c->shift & 255};
}

static int run_attention_stream(const StreamPlan& plan, const int32_t* q, const int64_t* sh, const int64_t* qpos,
                                const int8_t* cache, int64_t nb, int64_t sc_nb, int64_t sc_h, int64_t sc_bs, int bs,
                                const void* bt, int bt_is_int64, int64_t sbt, int nblk, const int64_t* rmap,
                                const int64_t* lut, int64_t l2e, const int32_t* ptab, int64_t* num, int64_t* den, int R,
                                int HKV, int M, const CompactTable& given, void* spill, size_t spill_bytes, void* stream) {
  const int64_t npairs = (int64_t)R * HKV;
  const int64_t spill_keys = ((int64_t)nblk * bs + 63) / 64 * 64;
  const int64_t grid = npairs < (int64_t)plan.per_sm * 148 ? npairs : (int64_t)plan.per_sm * 148;
  if (spill && (size_t)grid * (size_t)spill_keys * 32 > spill_bytes) return BX_ENOFIT;      // one slice per CTA
  const CompactTable ct = plan.table ? given : CompactTable{};
  AttnParams p{q, (const i64*)sh, (const i64*)qpos, cache, sc_nb, sc_h, sc_bs, bs, bt, bt_is_int64, sbt, nblk,
               (const i64*)rmap, (const i64*)lut, (i64)l2e, (i64*)num, (i64*)den, M, HKV, (int)plan.cap, ptab, ct};
  static PerDevice configured;
  if (once_per_device(configured, [] {
        cudaError_t e = cudaFuncSetAttribute(exact_attention_stream_kernel<8>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        return e != cudaSuccess ? e
                                : cudaFuncSetAttribute(exact_attention_stream_kernel<4>,
                                                       cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
      }) != BX_OK)
    return BX_ELAUNCH;
  EncodeTiledFn fn = encode_fn();
  if (!fn) return BX_ELAUNCH;
  CUtensorMap tk, tv;
  cuuint64_t dims[4] = {512, (cuuint64_t)bs, (cuuint64_t)HKV, (cuuint64_t)nb};
  cuuint64_t strides[3] = {(cuuint64_t)sc_bs, (cuuint64_t)sc_h, (cuuint64_t)sc_nb};
  cuuint32_t boxk[4] = {ATT2_HALF, (cuuint32_t)bs, 1, 1};
  cuuint32_t boxv[4] = {128, (cuuint32_t)bs, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  // 64-byte L2 promotion on both maps: measured against none / 128 B / 256 B, it is the only setting that changes
  // anything (batch 256, contexts U[64, 8192]: 875 -> 817 us; neutral at short contexts; 256 B: 15 % slower).
  if (fn(&tk, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<int8_t*>(cache), dims, strides, boxk, estr,
         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_64B,
         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS ||
      fn(&tv, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<int8_t*>(cache), dims, strides, boxv, estr,
         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_64B,
         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return BX_ELAUNCH;
  return launch_chained(plan.warps == 8 ? exact_attention_stream_kernel<8> : exact_attention_stream_kernel<4>, dim3((unsigned)grid),
                        32 * plan.warps + 64, (int)plan.smem, (cudaStream_t)stream, 0, tk, tv, p, plan.stages, npairs, (i64*)spill,
                        spill_keys);
}

// Scratch of the even split (variant 7): scores of every 64-key unit that the block tables can hold, and the pieces' maxima.
static size_t split_bytes(int64_t pairs, int64_t max_keys, int sms) {
  return (size_t)pairs * ((max_keys + SPL_KEYS - 1) / SPL_KEYS) * SPL_KEYS * 32 + (size_t)(pairs + 2 * sms) * 32 + (size_t)2 * sms * 16;
}
static int64_t split_cta_pages(int64_t pairs, int64_t max_keys, int bs, int sms) {
  const int64_t units = pairs * ((max_keys + SPL_KEYS - 1) / SPL_KEYS);
  return ((units + 2 * sms - 1) / (2 * sms)) * (SPL_KEYS / bs);
}
static bool split_can(int64_t R, int64_t HKV, int64_t max_keys, int bs, int sms) {
  return R <= SPL_MAXREQ && bs >= 8 && SPL_KEYS % bs == 0 && split_cta_pages(R * HKV, max_keys, bs, sms) <= SPL_MAXPAGES;
}

// Where the automatic choice splits evenly, by what the host knows: pairs and the width of the block tables. The two kernels cost about
// 9 us more than one on the smallest batches and serve every mix of lengths alike (us, before : split, 8 KV heads: 32 sequences of
// 64 .. 8192 keys 223 : 110, 64 of 16 .. 4096 145 : 119, 100 of 100 .. 1500 111 : 84, 256 of 500 .. 1400 254 : 184, 256 of
// 512 .. 768 145 : 138, of 500 .. 620 129 : 119; 16 of 500 .. 1400 35 : 33; one of 4000 / 8000 keys 27 : 23, 39 : 27; 72 of 64 .. 8192
// 265 : 224; pages of 64 keys, which the streaming kernel does not take, 200 of 64 .. 8192 968 : 562). Narrower tables stay with the
// kernels that give a pair to a CTA or a cluster (64 of 16 .. 600 37 : 45, 256 of 16 .. 200 59 : 70), and so do few pairs of up to 3072
// keys (4 of 2000 25 : 27). Contexts much shorter than wide tables pay for it (64 of 16 .. 100 keys in 4096 23 : 28, 32 of the same 47 : 25).
// entries: the caller's exact table has a compact form but no products, which leaves every weight of the split to the full table; the
// streaming kernel has the entries (us, stream : split: 64 sequences of 16 .. 4096 keys 137 : 167, 100 of 100 .. 1500 109 : 122, 256 of
// 512 .. 768 138 : 175, of 500 .. 1400 254 : 247; 48 of 64 .. 8192 221 : 208).
static bool split_auto(int64_t pairs, int64_t max_keys, bool entries) {
  if (entries && pairs >= STREAM_PAIRS && max_keys <= 4096 + 64) return false;
  return max_keys > (pairs >= 1024 ? 512 : pairs >= 192 ? 896 : pairs >= 128 ? 1280 : pairs >= 64 ? 2048 : 3072);
}

static int run_attention_split(const int8_t* cache, int64_t nb, AttnParams p, int R, void* scratch, int sms, cudaStream_t st) {
  static PerDevice configured;
  if (once_per_device(configured, [] {
        cudaError_t e = cudaFuncSetAttribute(attention_scores_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, split_scores_smem(SPL_MAXPAGES));
        return e != cudaSuccess ? e
                                : cudaFuncSetAttribute(attention_values_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, split_values_smem(SPL_MAXPAGES));
      }) != BX_OK)
    return BX_ELAUNCH;
  EncodeTiledFn fn = encode_fn();
  if (!fn) return BX_ELAUNCH;
  CUtensorMap tk, tv;
  cuuint64_t dims[4] = {512, (cuuint64_t)p.bs, (cuuint64_t)p.HKV, (cuuint64_t)nb};
  cuuint64_t strides[3] = {(cuuint64_t)p.sc_bs, (cuuint64_t)p.sc_h, (cuuint64_t)p.sc_nb};
  cuuint32_t boxk[4] = {ATT2_HALF, (cuuint32_t)p.bs, 1, 1}, boxv[4] = {128, (cuuint32_t)p.bs, 1, 1}, estr[4] = {1, 1, 1, 1};
  if (fn(&tk, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<int8_t*>(cache), dims, strides, boxk, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
         CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_64B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS ||
      fn(&tv, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<int8_t*>(cache), dims, strides, boxv, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_64B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return BX_ELAUNCH;
  SplitParams sp;
  sp.a = p;
  sp.pmax = (i64*)scratch;                               // pieces first, so that both parts are aligned
  sp.fits = (int*)(sp.pmax + ((int64_t)R * p.HKV + 2 * sms) * 4);
  sp.scores = (i64*)(sp.fits + 4 * 2 * sms);
  sp.nreq = R;
  const int pages = (int)split_cta_pages((int64_t)R * p.HKV, (int64_t)p.nblk * p.bs, p.bs, sms);
  const int rc = launch_chained(attention_scores_kernel, dim3(2 * sms), 32 * (SPL_WARPS + 1), split_scores_smem(pages), st, 0, tk, sp);
  if (rc != BX_OK) return rc;
  return launch_chained(attention_values_kernel, dim3(2 * sms), 32 * (SPL_WARPS + 2), split_values_smem(pages), st, 0, tv, sp);
}

static int run_attention(const int32_t* q, const int64_t* sh, const int64_t* qpos, const int8_t* cache, int64_t nb,
                         int64_t sc_nb, int64_t sc_h, int64_t sc_bs, int bs, const void* bt, int bt_is_int64,
                         int64_t sbt, int nblk, const int64_t* rmap, const int64_t* lut, int64_t l2e,
                         const int32_t* ptab, int64_t* num, int64_t* den, int R, int HKV, int M, int HD,
                         int cluster_size, int variant, const CompactTable& given, void* spill, size_t spill_bytes,
                         void* stream) {
  CompactTable ct = aligned16(given.tab) ? given : CompactTable{};
  // The products of the exact rule (2 KB) everywhere; an int8 weight is one entry of its table, which the 16 KB form serves better than
  // 6 KB of products do (us, 64 sequences of 16 .. 600 keys 35 : 37, 4 of 16 .. 2000 20 : 22).
  if (ptab) ct.products = nullptr;
  if (ct.products) ct.tab = nullptr;
  const int table = ct.products ? PW_EXACT_BYTES : ct.tab ? CT_BYTES : 0;
  if (!q || !qpos || !cache || !bt || !num || !den) return BX_EARG;
  if (!ptab && (!sh || !lut)) return BX_EARG;
  if (R < 0 || HKV <= 0 || M < 1 || M > 4 || HD != ATT_HD || bs <= 0 || nblk <= 0 || nb <= 0) return BX_EARG;
  const int64_t max_keys = (int64_t)nblk * bs;
  if (max_keys >= 43690) return BX_EARG;
  if (R == 0) return BX_OK;
  const int64_t smem_limit = 227 * 1024;
  // TMA-staged kernel when the cache layout allows a tensor map over it, else the direct-load kernel.
  const bool tma_ok = (bs % 8 == 0) && (ATT2_STAGE_KEYS % bs == 0) && sc_bs % 16 == 0 && sc_h % 16 == 0 &&
                      sc_nb % 16 == 0 && sc_bs >= 384 && aligned16(cache);
  if (variant >= 2 && !tma_ok) return BX_EARG;
  if (variant < 0 || variant > 7 || (variant == 4 && bs > 32)) return BX_EARG;
  if (variant == 7 || (variant == 0 && cluster_size == 0 && tma_ok && split_auto((int64_t)R * HKV, max_keys, !ptab && ct.tab))) {
    const int sms = device_sms();
    if (sms <= 0) return BX_ELAUNCH;
    if (split_can(R, HKV, max_keys, bs, sms) && spill && aligned16(spill) && aligned16(num) && spill_bytes >= split_bytes((int64_t)R * HKV, max_keys, sms))
      return run_attention_split(cache, nb, AttnParams{q, (const i64*)sh, (const i64*)qpos, cache, sc_nb, sc_h, sc_bs, bs, bt, bt_is_int64, sbt,
                                 nblk, (const i64*)rmap, (const i64*)lut, (i64)l2e, (i64*)num, (i64*)den, M, HKV, 0, ptab, ct}, R, spill, sms,
                                 (cudaStream_t)stream);
    if (variant == 7) return BX_EARG;
  }
  if (variant == 5 || variant == 6 || (variant == 0 && tma_ok)) {
    const int NW = variant == 5 ? 8 : 4;
    if (variant != 0 && !stream_page_ok(NW, bs)) return BX_EARG;
    const StreamPlan plan = variant == 0 ? stream_auto((int64_t)R * HKV, max_keys, bs, spill != nullptr, table)
                                         : stream_plan(NW, max_keys, spill != nullptr, table);
    int rc = BX_ENOFIT;
    if (plan.per_sm > 0)
      rc = run_attention_stream(plan, q, sh, qpos, cache, nb, sc_nb, sc_h, sc_bs, bs, bt, bt_is_int64, sbt, nblk, rmap, lut, l2e,
                                ptab, num, den, R, HKV, M, ct, plan.chunked ? spill : nullptr,
                                spill_bytes, stream);
    if (variant != 0) return rc == BX_ENOFIT ? BX_EARG : rc;
    if (rc != BX_ENOFIT) return rc;
  }
  // 1 direct loads, 2 TMA-staged, 3 TMA + tcgen05 p.V with 8 consumer warps, 4 the same with 4 consumer warps
  const int kind = variant != 0 ? variant : (tma_ok ? ((bs <= 32 && (int64_t)R * HKV >= 64) ? 4 : 3) : 1);
  const int nw = kind == 4 ? 4 : 8;
  const bool use_tma = kind >= 2;
  const int64_t fixed = kind >= 3 ? 1024 + (int64_t)ATT3_NS * (8 * nw * 256) + (int64_t)sizeof(Attn3Small) + (ct.products ? table : 0)
                        : kind == 2 ? (int64_t)ATT2_NS * ATT2_STAGE_BYTES + (int64_t)sizeof(Attn2Small)
                                    : (int64_t)sizeof(AttnShared);
  const int64_t gran = kind >= 3 ? 8 * nw : use_tma ? ATT2_STAGE_KEYS : 8;
  const int64_t cap_limit = (smem_limit - fixed) / 32 / gran * gran;
  int cs = cluster_size;
  if (cs == 0) {
    cs = 1;
    const int64_t pairs = (int64_t)R * HKV;
    while (cs < ATT_MAXCS && pairs * cs < 2 * 148) cs *= 2;               // fill the SMs
    while (cs < ATT_MAXCS && (max_keys + cs - 1) / cs > (kind == 4 ? 512 : 704)) cs *= 2;   // small score buffer
  }
  if (cs != 1 && cs != 2 && cs != 4 && cs != 8) return BX_EARG;
  auto cap_of = [&](int c) { return ((max_keys + c - 1) / c + gran - 1) / gran * gran; };
  while (cs < ATT_MAXCS && cap_of(cs) > cap_limit) cs *= 2;
  const int chunk_cap = (int)cap_of(cs);
  if (chunk_cap > cap_limit) return BX_EARG;
  const size_t smem = (size_t)fixed + (size_t)chunk_cap * 32;
  AttnParams p{q, (const i64*)sh, (const i64*)qpos, cache, sc_nb, sc_h, sc_bs, bs, bt, bt_is_int64, sbt, nblk,
               (const i64*)rmap, (const i64*)lut, (i64)l2e, (i64*)num, (i64*)den, M, HKV, chunk_cap, ptab, kind >= 3 && ct.products ? ct : CompactTable{}};
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((int64_t)cs * R * HKV), 1, 1);
  cfg.blockDim = dim3(kind == 4 ? 160 : use_tma ? ATT2_THREADS : ATT_THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  static PerDevice configured[5];
  if (once_per_device(configured[kind], [kind, smem_limit] {
        return kind == 4 ? cudaFuncSetAttribute(exact_attention_tc_kernel<4>,
                                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_limit)
               : kind == 3 ? cudaFuncSetAttribute(exact_attention_tc_kernel<8>,
                                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_limit)
               : kind == 2 ? cudaFuncSetAttribute(exact_attention_tma_kernel,
                                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_limit)
                           : cudaFuncSetAttribute(exact_attention_kernel,
                                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_limit);
      }) != BX_OK)
    return BX_ELAUNCH;
  if (kind >= 3) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return BX_ELAUNCH;
    CUtensorMap tk, tv;
    cuuint64_t dims[4] = {512, (cuuint64_t)bs, (cuuint64_t)HKV, (cuuint64_t)nb};
    cuuint64_t strides[3] = {(cuuint64_t)sc_bs, (cuuint64_t)sc_h, (cuuint64_t)sc_nb};
    cuuint32_t boxk[4] = {ATT2_HALF, (cuuint32_t)bs, 1, 1};
    cuuint32_t boxv[4] = {128, (cuuint32_t)bs, 1, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    if (fn(&tk, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<int8_t*>(cache), dims, strides, boxk, estr,
           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS ||
        fn(&tv, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<int8_t*>(cache), dims, strides, boxv, estr,
           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return BX_ELAUNCH;
    return launch_chained(kind == 4 ? exact_attention_tc_kernel<4> : exact_attention_tc_kernel<8>, cfg.gridDim, (int)cfg.blockDim.x,
                          (int)smem, cfg.stream, cs, tk, tv, p);
  } else if (use_tma) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return BX_ELAUNCH;
    CUtensorMap tm;
    cuuint64_t dims[4] = {512, (cuuint64_t)bs, (cuuint64_t)HKV, (cuuint64_t)nb};
    cuuint64_t strides[3] = {(cuuint64_t)sc_bs, (cuuint64_t)sc_h, (cuuint64_t)sc_nb};
    cuuint32_t box[4] = {ATT2_HALF, (cuuint32_t)bs, 1, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    if (fn(&tm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<int8_t*>(cache), dims, strides, box, estr,
           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return BX_ELAUNCH;
    if (cudaLaunchKernelEx(&cfg, exact_attention_tma_kernel, tm, p) != cudaSuccess) return BX_ELAUNCH;
  } else {
    if (cudaLaunchKernelEx(&cfg, exact_attention_kernel, p) != cudaSuccess) return BX_ELAUNCH;
  }
  return launched(1);
}

int bx_exact_attention(const int32_t* q, const int64_t* sh, const int64_t* qpos, const int8_t* cache, int64_t nb,
                       int64_t sc_nb, int64_t sc_h, int64_t sc_bs, int bs, const void* bt, int bt_is_int64,
                       int64_t sbt, int nblk, const int64_t* rmap, const int64_t* lut, int64_t l2e, int64_t* num,
                       int64_t* den, int R, int HKV, int M, int HD, int cluster_size, int variant, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!sh || !lut) return BX_EARG;
  return run_attention(q, sh, qpos, cache, nb, sc_nb, sc_h, sc_bs, bs, bt, bt_is_int64, sbt, nblk, rmap, lut, l2e,
                       nullptr, num, den, R, HKV, M, HD, cluster_size, variant, CompactTable{}, nullptr, 0, stream);
}

int bx_attention_plan(int R, int HKV, int nblk, int bs, int scratch, int table) {
  if (R < 0 || HKV <= 0 || nblk <= 0 || bs <= 0) return BX_EARG;
  const int64_t pairs = (int64_t)R * HKV, keys = (int64_t)nblk * bs;
  const int sms = device_sms();
  if (scratch == 2 && R > 0 && split_auto(pairs, keys, table == 3) && split_can(R, HKV, keys, bs, sms > 0 ? sms : 148)) return 7;
  const StreamPlan p = stream_auto(pairs, keys, bs, scratch != 0, table == 2 ? PW_EXACT_BYTES : table ? CT_BYTES : 0);
  return p.per_sm == 0 ? 0 : 1000 * p.chunked + 100 * p.warps + 10 * p.per_sm + p.table;
}

int bx_attention_stream_pairs(void) { return (int)STREAM_PAIRS; }

size_t bx_attention_scratch_bytes(int nblk, int bs) {
  if (nblk <= 0 || bs <= 0) return 0;
  const size_t keys = ((size_t)nblk * bs + 63) / 64 * 64;
  return (size_t)4 * 148 * keys * 32;
}

size_t bx_attention_workspace(int R, int HKV, int nblk, int bs, int variant) {
  const int sms = device_sms();
  if (R <= 0 || HKV <= 0 || nblk <= 0 || bs <= 0 || sms <= 0) return 0;
  const int64_t pairs = (int64_t)R * HKV, keys = (int64_t)nblk * bs;
  if ((variant == 7 || (variant == 0 && split_auto(pairs, keys, false))) && split_can(R, HKV, keys, bs, sms)) {
    // room for the streaming kernel too: a cache that no tensor map can describe, or a forced cluster size, takes another kernel
    const size_t even = split_bytes(pairs, keys, sms), other = bx_attention_scratch_bytes(nblk, bs);
    return variant == 7 || pairs < STREAM_PAIRS || even > other ? even : other;
  }
  return keys <= 896 || pairs < STREAM_PAIRS ? 0 : bx_attention_scratch_bytes(nblk, bs);
}

int bx_exact_attention_ws(const int32_t* q, const int64_t* sh, const int64_t* qpos, const int8_t* cache, int64_t nb,
                          int64_t sc_nb, int64_t sc_h, int64_t sc_bs, int bs, const void* bt, int bt_is_int64,
                          int64_t sbt, int nblk, const int64_t* rmap, const int64_t* lut, int64_t l2e, int64_t* num,
                          int64_t* den, int R, int HKV, int M, int HD, int cluster_size, int variant, void* scratch,
                          size_t scratch_bytes, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!sh || !lut) return BX_EARG;
  return run_attention(q, sh, qpos, cache, nb, sc_nb, sc_h, sc_bs, bs, bt, bt_is_int64, sbt, nblk, rmap, lut, l2e,
                       nullptr, num, den, R, HKV, M, HD, cluster_size, variant, CompactTable{}, scratch, scratch_bytes, stream);
}

int bx_int8_attention_ws(const int32_t* q, const int64_t* qpos, const int8_t* cache, int64_t nb, int64_t sc_nb,
                         int64_t sc_h, int64_t sc_bs, int bs, const void* bt, int bt_is_int64, int64_t sbt, int nblk,
                         const int64_t* rmap, const int32_t* ptab, int64_t* num, int64_t* den, int R, int HKV, int M,
                         int HD, int cluster_size, int variant, void* scratch, size_t scratch_bytes, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!ptab) return BX_EARG;
  return run_attention(q, nullptr, qpos, cache, nb, sc_nb, sc_h, sc_bs, bs, bt, bt_is_int64, sbt, nblk, rmap, nullptr,
                       0, ptab, num, den, R, HKV, M, HD, cluster_size, variant, CompactTable{}, scratch, scratch_bytes, stream);
}

int bx_int8_attention(const int32_t* q, const int64_t* qpos, const int8_t* cache, int64_t nb, int64_t sc_nb,
                      int64_t sc_h, int64_t sc_bs, int bs, const void* bt, int bt_is_int64, int64_t sbt, int nblk,
                      const int64_t* rmap, const int32_t* ptab, int64_t* num, int64_t* den, int R, int HKV, int M,
                      int HD, int cluster_size, int variant, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!ptab) return BX_EARG;
  return run_attention(q, nullptr, qpos, cache, nb, sc_nb, sc_h, sc_bs, bs, bt, bt_is_int64, sbt, nblk, rmap, nullptr,
                       0, ptab, num, den, R, HKV, M, HD, cluster_size, variant, CompactTable{}, nullptr, 0, stream);
}

int bx_exact_attention_tab(const int32_t* q, const int64_t* sh, const int64_t* qpos, const int8_t* cache, int64_t nb,
                           int64_t sc_nb, int64_t sc_h, int64_t sc_bs, int bs, const void* bt, int bt_is_int64,
                           int64_t sbt, int nblk, const int64_t* rmap, const int64_t* lut, int64_t l2e, int64_t* num,
                           int64_t* den, int R, int HKV, int M, int HD, int cluster_size, int variant, void* scratch,
                           size_t scratch_bytes, const bx_compact_table* compact, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!sh || !lut || !compact) return BX_EARG;
  const CompactTable ct = compact_table(compact);
  return run_attention(q, sh, qpos, cache, nb, sc_nb, sc_h, sc_bs, bs, bt, bt_is_int64, sbt, nblk, rmap, lut, l2e,
                       nullptr, num, den, R, HKV, M, HD, cluster_size, variant, ct, scratch, scratch_bytes, stream);
}

int bx_int8_attention_tab(const int32_t* q, const int64_t* qpos, const int8_t* cache, int64_t nb, int64_t sc_nb,
                          int64_t sc_h, int64_t sc_bs, int bs, const void* bt, int bt_is_int64, int64_t sbt, int nblk,
                          const int64_t* rmap, const int32_t* ptab, int64_t* num, int64_t* den, int R, int HKV, int M,
                          int HD, int cluster_size, int variant, void* scratch, size_t scratch_bytes,
                          const bx_compact_table* compact, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!ptab || !compact) return BX_EARG;
  const CompactTable ct = compact_table(compact);
  return run_attention(q, nullptr, qpos, cache, nb, sc_nb, sc_h, sc_bs, bs, bt, bt_is_int64, sbt, nblk, rmap, nullptr,
                       0, ptab, num, den, R, HKV, M, HD, cluster_size, variant, ct, scratch, scratch_bytes, stream);
}

int bx_prefill_attention(const int32_t* q, const int64_t* sh, const int64_t* pos, const int32_t* tiles, int n_tiles,
                         const int8_t* cache, int64_t nb, int64_t sc_nb, int64_t sc_h, int64_t sc_bs, int bs,
                         const void* bt, int bt_is_int64, int64_t sbt, int nblk, const int64_t* lut, int64_t l2e,
                         const int32_t* ptab, int64_t* num, int64_t* den, int HKV, int G, int HD, int tile_rows,
                         void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!q || !pos || !tiles || !cache || !bt || !num || !den || n_tiles < 0) return BX_EARG;
  if (!ptab && (!sh || !lut)) return BX_EARG;
  if (tile_rows == 0) tile_rows = 32;
  if (tile_rows != 16 && tile_rows != 32) return BX_EARG;
  if (HD != ATT_HD || HKV <= 0 || HKV > 65535 || G < 1 || G > tile_rows || nblk <= 0 || nb <= 0) return BX_EARG;
  if (bs < 8 || bs > PF_KEYS || PF_KEYS % bs || (int64_t)nblk * bs >= 43690) return BX_EARG;
  if (sc_bs % 16 || sc_h % 16 || sc_nb % 16 || sc_bs < 384 || !aligned16(cache) || !aligned16(q)) return BX_EARG;
  if (n_tiles == 0) return BX_OK;
  EncodeTiledFn fn = encode_fn();
  if (!fn) return BX_ELAUNCH;
  CUtensorMap tm;
  cuuint64_t dims[4] = {512, (cuuint64_t)bs, (cuuint64_t)HKV, (cuuint64_t)nb};
  cuuint64_t strides[3] = {(cuuint64_t)sc_bs, (cuuint64_t)sc_h, (cuuint64_t)sc_nb};
  cuuint32_t box[4] = {128, (cuuint32_t)bs, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  if (fn(&tm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<int8_t*>(cache), dims, strides, box, estr,
         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return BX_ELAUNCH;
  const bool exact = !ptab;
  const int sms = device_sms();
  if (sms <= 0) return BX_ELAUNCH;
  static PerDevice configured;
  if (once_per_device(configured, [] {
        cudaError_t e = cudaFuncSetAttribute(prefill_attention_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             pf_smem(true));
        return e != cudaSuccess ? e
                                : cudaFuncSetAttribute(prefill_attention_kernel<false>,
                                                       cudaFuncAttributeMaxDynamicSharedMemorySize, pf_smem(false));
      }) != BX_OK)
    return BX_ELAUNCH;
  PrefillParams p{};
  p.q = q;
  p.sh = (const i64*)sh;
  p.pos = (const i64*)pos;
  p.tiles = tiles;
  p.bt = bt;
  p.bt64 = bt_is_int64;
  p.sbt = sbt;
  p.nblk = nblk;
  p.bs = bs;
  p.w.lut = (const i64*)lut;
  p.w.l2e = (i64)l2e;
  p.w.ptab = ptab;
  p.num = (i64*)num;
  p.den = (i64*)den;
  p.HKV = HKV;
  p.G = G;
  p.work = (int64_t)n_tiles * HKV;
  const unsigned grid = (unsigned)(p.work < sms ? p.work : sms);       // persistent: one CTA per SM
  return launch_chained(exact ? prefill_attention_kernel<true> : prefill_attention_kernel<false>, dim3(grid), PF_THREADS, pf_smem(exact),
                        (cudaStream_t)stream, 0, tm, p);
}

int bx_int8_norm(int mode, const void* xin, const int64_t* yin, const int64_t* ids, const int64_t* gamma,
                 int64_t* xo, int8_t* a8, int64_t* mant, int64_t* e, int32_t* flag, int M, int D, int do_norm,
                 void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!xin || !flag || M < 0 || D < 1 || D > NORM_THREADS * NORM_EPT || mode < 0 || mode > 2) return BX_EARG;
  if ((mode == 0 && !ids) || (mode == 1 && !yin) || (do_norm && (!gamma || !a8 || !mant || !e))) return BX_EARG;
  if (M == 0) return BX_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const int sms = device_sms();
  if (sms <= 0) return BX_ELAUNCH;
  const bool wide = D % 4 == 0 && aligned_to(xin, 32) && aligned_to(yin, 32) && aligned_to(gamma, 32) && aligned_to(xo, 32) && aligned_to(a8, 4);
#define BX_NORM_LAUNCH(MODE, NT, Q) \
  return launch_chained(i8::int8_norm_kernel<MODE, NT, Q>, dim3(even_grid(M, sms * (1024 / NT))), NT, 0, st, 0, xin, (const i64*)yin, \
                        (const i64*)ids, (const i64*)gamma, (i64*)xo, a8, (i64*)mant, (i64*)e, flag, M, D, do_norm, wide)
#define BX_NORM_MODES(NT, Q) \
  if (mode == 0) BX_NORM_LAUNCH(0, NT, Q); else if (mode == 1) BX_NORM_LAUNCH(1, NT, Q); else BX_NORM_LAUNCH(2, NT, Q)
  if (D <= 512) { BX_NORM_MODES(128, 1); }
  else if (D <= 1024) { BX_NORM_MODES(256, 1); }
  else if (D <= 2048) { BX_NORM_MODES(512, 1); }
  else { BX_NORM_MODES(512, 2); }
#undef BX_NORM_MODES
#undef BX_NORM_LAUNCH
}

int bx_int8_qkv(const int64_t* y, const int64_t* cos, const int64_t* sin, const int64_t* pos, const int64_t* slot,
                int8_t* cache, int64_t sc_nb, int64_t sc_h, int64_t sc_bs, int bs, int64_t* q64, int32_t* q32,
                int32_t* flag, int N, int H, int HKV, int HD, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!y || !cos || !sin || !pos || !flag || (!q64 && !q32) || N < 0) return BX_EARG;
  if ((HD != 64 && HD != 128) || HKV <= 0 || H % HKV || (cache && (!slot || bs <= 0))) return BX_EARG;
  if (N == 0) return BX_OK;
  i8::Qkv8Params p{(const i64*)y, (const i64*)cos, (const i64*)sin, (const i64*)pos, (const i64*)slot, cache, sc_nb,
                   sc_h, sc_bs, bs, (i64*)q64, q32, flag, H, HKV, HD};
  return launch_chained(i8::int8_qkv_kernel, dim3(N, HKV), HD / 2, 0, (cudaStream_t)stream, 0, p);
}

int bx_int8_attn_out(const int64_t* num, const int64_t* den, int8_t* a8, int64_t* mant, int64_t* e, int N, int K2,
                     int HD, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!num || !den || !a8 || !mant || !e || N < 0 || K2 <= 0 || K2 > AO_THREADS * AO_EPT || HD <= 0 || K2 % HD ||
      K2 / HD > AO_MAXH)
    return BX_EARG;
  if (N == 0) return BX_OK;
  const i64 *nm = (const i64*)num, *dn = (const i64*)den;
  if (HD % 4)
    return launch_chained(i8::int8_attn_out_any_kernel, dim3(N), AO_THREADS, 0, (cudaStream_t)stream, 0, nm, dn, a8, (i64*)mant, (i64*)e, N, K2, HD);
  const bool wide = aligned_to(num, 32) && aligned_to(a8, 4);
  return launch_chained(K2 <= 1024 ? i8::int8_attn_out_kernel<256, 1> : K2 <= 2048 ? i8::int8_attn_out_kernel<512, 1> : i8::int8_attn_out_kernel<512, 2>,
                        dim3(N), K2 <= 1024 ? 256 : 512, 0, (cudaStream_t)stream, 0, nm, dn, a8, (i64*)mant, (i64*)e, N, K2, HD, wide);
}

int bx_int8_silu_quant(const int64_t* y, const int64_t* lut, int8_t* a8, int64_t* mant, int64_t* e, int64_t* scr,
                       int N, int FF, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!y || !lut || !a8 || !mant || !e || N < 0 || FF <= 0 || FF > SILU_THREADS * 28) return BX_EARG;
  if (N == 0) return BX_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const int ept = (FF + SILU_THREADS - 1) / SILU_THREADS;
  return launch_chained(ept <= 4 ? i8::int8_silu_kernel<4> : ept <= 16 ? i8::int8_silu_kernel<16> : i8::int8_silu_kernel<28>, dim3(N),
                        SILU_THREADS, 0, st, 0, (const i64*)y, (const i64*)lut, a8, (i64*)mant, (i64*)e, (i64*)scr, N, FF);
}

int bx_int8_silu_quant_tab(const int64_t* y, const int64_t* lut, const uint16_t* compact, int8_t* a8, int64_t* mant, int64_t* e, int64_t* scr,
                           int N, int FF, void* stream) {
  if (!compact || !aligned16(compact) || FF % 4 || FF < 1024) return bx_int8_silu_quant(y, lut, a8, mant, e, scr, N, FF, stream);
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!y || !lut || !a8 || !mant || !e || N < 0 || FF > SILU_THREADS * 28) return BX_EARG;
  if (N == 0) return BX_OK;
  const bool wide = aligned_to(y, 32) && aligned_to(a8, 4);
  cudaStream_t st = (cudaStream_t)stream;
  const int sms = device_sms();
  if (sms <= 0) return BX_ELAUNCH;
  if (N > 128) {
    static PerDevice configured;
    const int smem = i8::SC_BYTES;
    if (once_per_device(configured, [smem] {
          cudaError_t r = cudaSuccess;
          for (auto* k : {i8::int8_silu_persistent_kernel<256, 4>, i8::int8_silu_persistent_kernel<512, 2>, i8::int8_silu_persistent_kernel<512, 4>,
                          i8::int8_silu_persistent_kernel<1024, 2>, i8::int8_silu_persistent_kernel<1024, 4>})
            if (r == cudaSuccess) r = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
          return r;
        }) != BX_OK)
      return BX_ELAUNCH;
    const int groups = silu_groups(N, FF, sms);
    auto* kernel = FF > 8192 ? i8::int8_silu_persistent_kernel<1024, 4>
                   : FF > 4096 ? (groups == 2 ? i8::int8_silu_persistent_kernel<512, 4> : i8::int8_silu_persistent_kernel<1024, 2>)
                   : groups == 4 ? i8::int8_silu_persistent_kernel<256, 4> : groups == 2 ? i8::int8_silu_persistent_kernel<512, 2>
                                                                                         : i8::int8_silu_persistent_kernel<1024, 2>;
    return launch_chained(kernel, dim3(even_grid((N + groups - 1) / groups, sms)), SILU_P_THREADS, smem, st, 0, (const i64*)y, (const i64*)lut,
                          compact, a8, (i64*)mant, (i64*)e, (i64*)scr, N, FF, wide);
  }
  const int cl = N * 8 <= sms ? 8 : 4, per = (FF / 4 + cl - 1) / cl;
  return launch_chained(per <= SILU_CL_THREADS ? i8::int8_silu_cluster_kernel<1> : per <= 2 * SILU_CL_THREADS ? i8::int8_silu_cluster_kernel<2>
                                                                                                  : i8::int8_silu_cluster_kernel<4>,
                        dim3(cl * N), SILU_CL_THREADS, 0, st, cl, (const i64*)y, (const i64*)lut, compact, a8, (i64*)mant, (i64*)e, (i64*)scr, N,
                        FF, wide);
}

int bx_int8_silu_prod(const int64_t* y, const int64_t* lut, int64_t* h, int64_t* rowmax, int64_t* scr, int N, int FFl,
                      void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!y || !lut || !h || !rowmax || N < 0 || FFl <= 0 || FFl > SILU_THREADS * 28) return BX_EARG;
  if (N == 0) return BX_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const int ept = (FFl + SILU_THREADS - 1) / SILU_THREADS;
  if (ept <= 4) i8::int8_silu_prod_kernel<4><<<N, SILU_THREADS, 0, st>>>((const i64*)y, (const i64*)lut, (i64*)h, (i64*)rowmax, (i64*)scr, N, FFl);
  else if (ept <= 16) i8::int8_silu_prod_kernel<16><<<N, SILU_THREADS, 0, st>>>((const i64*)y, (const i64*)lut, (i64*)h, (i64*)rowmax, (i64*)scr, N, FFl);
  else i8::int8_silu_prod_kernel<28><<<N, SILU_THREADS, 0, st>>>((const i64*)y, (const i64*)lut, (i64*)h, (i64*)rowmax, (i64*)scr, N, FFl);
  return launched(1);
}

int bx_int8_quant_rows(const int64_t* h, const int64_t* rowmax, int8_t* a8, int64_t* mant, int64_t* e, int N, int K,
                       void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!h || !rowmax || !a8 || N < 0 || K <= 0 || (mant && !e)) return BX_EARG;
  if (N == 0) return BX_OK;
  i8::int8_quant_rows_kernel<<<N, 256, 0, (cudaStream_t)stream>>>((const i64*)h, (const i64*)rowmax, a8, (i64*)mant, (i64*)e, N, K);
  return launched(1);
}

int bx_int8_post(const int32_t* c, const int64_t* mul, int64_t fmsh, const int64_t* mant, const int64_t* e, int64_t* y,
                 int32_t* flag, int M, int N, int checked, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!c || !mul || !mant || !e || !y || !flag || M < 0 || N <= 0) return BX_EARG;
  if (M == 0) return BX_OK;
  const int64_t total = (int64_t)M * N;
  int blocks = (int)((total + 255) / 256);
  if (blocks > 148 * 16) blocks = 148 * 16;
  i8::int8_post_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(c, (const i64*)mul, (i64)fmsh, (const i64*)mant, (const i64*)e, (i64*)y, flag, M, N, checked);
  return launched(1);
}

int bx_int8_flag_end(int64_t* scr, int32_t* flag, int L, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!scr || !flag || L <= 0) return BX_EARG;
  i8::int8_flag_end_kernel<<<1, 64, 0, (cudaStream_t)stream>>>((i64*)scr, flag, L);
  return launched(1);
}

int bx_pcg_raw(const int64_t* keys, int64_t* out, int n, int V, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!keys || !out || n < 0 || V <= 0) return BX_EARG;
  if (n == 0) return BX_OK;
  const int run = 16;
  const int blocks = (V + run * SAMPLE_THREADS - 1) / (run * SAMPLE_THREADS);
  pcg_raw_kernel<<<dim3(blocks, n), SAMPLE_THREADS, 0, (cudaStream_t)stream>>>((const i64*)keys, (i64*)out, V, run);
  return launched(1);
}

static int sample_chunks(int M, int V) {
  int nch = (8 * 148 + (M > 0 ? M : 1) - 1) / (M > 0 ? M : 1);       // eight 256-thread CTAs per SM
  const int maxch = (V + 2047) / 2048;
  if (nch > maxch) nch = maxch;
  return nch < 1 ? 1 : nch;
}

size_t bx_sample_scratch_bytes(int M, int V) { return (size_t)2 * 8 * (size_t)(M > 0 ? M : 0) * sample_chunks(M, V); }

static int run_sample(const int64_t* logits, int64_t ld, const int64_t* rows, const int64_t* lnt, void* scratch,
                      int64_t* tok, int64_t* omax, int M, int V, int64_t voff, int bits, void* stream) {
  if (!logits || !rows || !lnt || !scratch || !tok || M < 0 || V <= 0 || ld < V || voff < 0 || M > 65535) return BX_EARG;
  if (M == 0) return BX_OK;
  const int nch0 = sample_chunks(M, V);
  const int ch = ((V + nch0 - 1) / nch0 + 1) / 2 * 2;
  const int nch = (V + ch - 1) / ch;
  i64* pmax = (i64*)scratch;
  i64* pidx = pmax + (size_t)M * nch0;
  cudaStream_t st = (cudaStream_t)stream;
  const int rc = launch_chained(sample_part_kernel, dim3(nch, M), SAMPLE_THREADS, 0, st, 0, (const i64*)logits, ld, (const i64*)rows,
                                (const i64*)lnt, pmax, pidx, V, ch, nch, bits, (i64)voff);
  if (rc != BX_OK) return rc;
  return launch_chained(sample_combine_kernel, dim3((M + 3) / 4), 128, 0, st, 0, pmax, pidx, (i64*)tok, (i64*)omax, M, nch);
}

int bx_sample(const int64_t* logits, int64_t ld, const int64_t* rows, const int64_t* lnt, void* scratch,
              int64_t* tok, int M, int V, int bits, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  return run_sample(logits, ld, rows, lnt, scratch, tok, nullptr, M, V, 0, bits, stream);
}

int bx_sample_shard(const int64_t* logits, int64_t ld, const int64_t* rows, const int64_t* lnt, void* scratch,
                    int64_t* best, int64_t* idx, int M, int V_local, int64_t v_offset, int bits, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!best) return BX_EARG;
  return run_sample(logits, ld, rows, lnt, scratch, idx, best, M, V_local, v_offset, bits, stream);
}

// ---- weight preparation (load time) ----
int bx_decompose_rows(const uint16_t* w, int64_t ldw, int8_t* limbs, int64_t* g, int64_t* d, int32_t* cnt, int32_t* flag,
                      int N, int K, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!w || !limbs || !g || !d || !cnt || !flag || N < 0 || K <= 0 || ldw < K) return BX_EARG;
  if (N == 0) return BX_OK;
  decompose_rows_kernel<<<N, DEC_THREADS, 0, (cudaStream_t)stream>>>(w, ldw, limbs, (i64*)g, (i64*)d, cnt, flag, N, K);
  return launched(1);
}

int bx_decompose_residual(const uint16_t* w, int64_t ldw, const int64_t* g, const int64_t* d, const int64_t* start,
                          int64_t* rr, int64_t* rc, int64_t* rv, int N, int K, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!w || !g || !d || !start || !rr || !rc || !rv || N < 0 || K <= 0 || ldw < K) return BX_EARG;
  if (N == 0) return BX_OK;
  decompose_residual_kernel<<<N, DEC_THREADS, 0, (cudaStream_t)stream>>>(w, ldw, (const i64*)g, (const i64*)d,
                                                                         (const i64*)start, (i64*)rr, (i64*)rc, (i64*)rv, K);
  return launched(1);
}

// ---- integer log p ----------------------------------------------------------------------------------------------
static void logp_plan(int M, int V, int& ch, int& nch) {
  const int nch0 = sample_chunks(M, V);
  ch = (V + nch0 - 1) / nch0;
  nch = (V + ch - 1) / ch;
}

size_t bx_logp_scratch_bytes(int M, int V) {
  return (size_t)(2 * 8 + 4) * (size_t)(M > 0 ? M : 0) * sample_chunks(M, V > 0 ? V : 1);      // maxima, sums, and a word per CTA
}

static bool logp_args_ok(const void* lg, int64_t ld, const void* scratch, int M, int V) {
  return lg && scratch && M >= 0 && M <= 65535 && V > 0 && ld >= V;
}

int bx_logp_pair_table(const int64_t* tab, int tab_len, int64_t* tab2, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!tab || !tab2 || tab_len != LSE_LAST + 1 || ((uintptr_t)tab2 & 15)) return BX_EARG;
  logp_pair_table_kernel<<<(tab_len + 255) / 256, 256, 0, (cudaStream_t)stream>>>((const i64*)tab, (longlong2*)tab2, tab_len);
  return launched(1);
}

int bx_logp_rowmax(const int64_t* logits, int64_t ld, void* scratch, int64_t* rowmax, int M, int V, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!logp_args_ok(logits, ld, scratch, M, V) || !rowmax) return BX_EARG;
  if (M == 0) return BX_OK;
  int ch, nch;
  logp_plan(M, V, ch, nch);
  cudaStream_t st = (cudaStream_t)stream;
  i64* pmax = (i64*)scratch;
  logp_max_kernel<<<dim3(nch, M), LOGP_THREADS, 0, st>>>((const i64*)logits, ld, pmax, V, ch, nch, nullptr, nullptr);
  logp_rowfold_kernel<<<(M + 127) / 128, 128, 0, st>>>(pmax, nch, (i64*)rowmax, M, 0);
  return launched(2);
}

int bx_logp_rowsum(const int64_t* logits, int64_t ld, const int64_t* rowmax, const int64_t* tab2, int tab_len,
                   void* scratch, int64_t* S, int M, int V, int fr, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!logp_args_ok(logits, ld, scratch, M, V) || !rowmax || !tab2 || ((uintptr_t)tab2 & 15) || !S || tab_len != LSE_LAST + 1 || fr <= LSE_STEP ||
      fr > 24)
    return BX_EARG;
  if (M == 0) return BX_OK;
  int ch, nch;
  logp_plan(M, V, ch, nch);
  cudaStream_t st = (cudaStream_t)stream;
  i64* psum = (i64*)scratch;
  logp_sum_kernel<<<dim3(nch, M), LOGP_THREADS, 0, st>>>((const i64*)logits, ld, (const i64*)rowmax, nullptr, 0, nullptr,
                                                        (const longlong2*)tab2, nullptr, psum, V, ch, nch, fr);
  logp_rowfold_kernel<<<(M + 127) / 128, 128, 0, st>>>(psum, nch, (i64*)S, M, 1);
  return launched(2);
}

int bx_logp_finish(const int64_t* S, const int64_t* zt, const int64_t* lnt, int64_t* out, int M, int fr, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!S || !zt || !lnt || !out || M < 0 || fr <= LSE_STEP || fr > 24) return BX_EARG;
  if (M == 0) return BX_OK;
  logp_finish_kernel<<<(M + 127) / 128, 128, 0, (cudaStream_t)stream>>>((const i64*)S, 1, (const i64*)zt, nullptr, 0, nullptr,
                                                                        nullptr, (const i64*)lnt, (i64*)out, M, 0, fr);
  return launched(1);
}

int bx_int_logp(const int64_t* logits, int64_t ld, const int64_t* tok, const int64_t* lnt, const int64_t* tab2,
                int tab_len, void* scratch, int64_t* out, int M, int V, int fr, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!logp_args_ok(logits, ld, scratch, M, V) || !tok || !lnt || !tab2 || ((uintptr_t)tab2 & 15) || !out || tab_len != LSE_LAST + 1 ||
      fr <= LSE_STEP || fr > 24)
    return BX_EARG;
  if (M == 0) return BX_OK;
  int ch, nch;
  logp_plan(M, V, ch, nch);
  cudaStream_t st = (cudaStream_t)stream;
  const int nch0 = sample_chunks(M, V);
  i64* pmax = (i64*)scratch;                       // chunk maxima, then (entry 0 of each row) the row maximum
  i64* psum = pmax + (size_t)M * nch0;
  // below about eight table lengths of logits, checking the table costs what the gathers do (both 34 .. 39 us at 16 rows of 128256;
  // 64 rows 80 -> 66 us)
  int* fits = (i64)M * V >= (i64)8 * LSE_LAST ? (int*)(psum + (size_t)M * nch0) : nullptr;
  logp_max_kernel<<<dim3(nch, M), LOGP_THREADS, 0, st>>>((const i64*)logits, ld, pmax, V, ch, nch, (const longlong2*)tab2, fits);
  // the row maxima go to out[], which the last kernel overwrites after reading them
  logp_sum_kernel<<<dim3(nch, M), LOGP_THREADS, 0, st>>>((const i64*)logits, ld, nullptr, pmax, nch, (i64*)out,
                                                        (const longlong2*)tab2, fits, psum, V, ch, nch, fr);
  logp_finish_kernel<<<(M + 127) / 128, 128, 0, st>>>(psum, nch, nullptr, (const i64*)logits, ld, (const i64*)tok,
                                                      (const i64*)out, (const i64*)lnt, (i64*)out, M, V, fr);
  return launched(3);
}

int bx_exact_silu_prod(const int64_t* y, const int64_t* lut, int64_t* P, int64_t* rowmax, int32_t* flag, int N, int FFl,
                       void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!y || !lut || !P || !rowmax || !flag || N < 0 || FFl <= 0) return BX_EARG;
  if (N == 0) return BX_OK;
  silu_prod_kernel<512><<<N, 512, 0, (cudaStream_t)stream>>>((const i64*)y, (const i64*)lut, (i64*)P, (i64*)rowmax, flag,
                                                             FFl);
  return launched(1);
}

int bx_exact_quant_rows(const int64_t* P, const int64_t* rowmax, int fbits, int32_t* q, int64_t ldq, int64_t* sh,
                        int8_t* a8, int64_t plane, int N, int K, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!P || !rowmax || !q || N < 0 || K <= 0 || ldq < K || fbits < 0 || fbits > 62 || (a8 && plane < (int64_t)N * ldq))
    return BX_EARG;
  if (N == 0) return BX_OK;
  quant_rows_kernel<<<N, 256, 0, (cudaStream_t)stream>>>((const i64*)P, (const i64*)rowmax, fbits, q, ldq, (i64*)sh, a8,
                                                         plane, K);
  return launched(1);
}

// ---- stages of the reference's standalone engine, one kernel each (unfused_stages.cuh) ----
int bx_exact_rms(const int64_t* x, int64_t* r, int64_t* er, int64_t* amax, int M, int D, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!x || !r || !er || M < 0 || D < 1 || D > 4096 || (D & (D - 1))) return BX_EARG;
  if (M == 0) return BX_OK;
  int lg = 0;
  while ((1 << lg) < D) ++lg;
  rms_kernel<<<M, US_THREADS, 0, (cudaStream_t)stream>>>((const i64*)x, (i64*)r, (i64*)er, (i64*)amax, D, lg);
  return launched(1);
}

int bx_exact_ndiv(const int64_t* x, const int64_t* gm, const int64_t* ge, const int64_t* r, const int64_t* er,
                  int64_t* P, int M, int D, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!x || !gm || !ge || !r || !er || !P || M < 0 || D < 1) return BX_EARG;
  if (M == 0) return BX_OK;
  ndiv_kernel<<<M, US_THREADS, 0, (cudaStream_t)stream>>>((const i64*)x, (const i64*)gm, (const i64*)ge, (const i64*)r,
                                                        (const i64*)er, (i64*)P, D);
  return launched(1);
}

int bx_rowmax_abs(const int64_t* P, int64_t* rowmax, int M, int K, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!P || !rowmax || M < 0 || K < 1) return BX_EARG;
  if (M == 0) return BX_OK;
  rowmax_abs_kernel<<<M, US_THREADS, 0, (cudaStream_t)stream>>>((const i64*)P, (i64*)rowmax, K);
  return launched(1);
}

int bx_exact_rope(const int64_t* y, const int64_t* cos, const int64_t* sin, const int64_t* pos, int64_t* Pq, int64_t* k,
                  int64_t* v, int N, int H, int HKV, int HD, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!y || !cos || !sin || !pos || !Pq || !k || !v || N < 0 || H <= 0 || HKV <= 0 || HD <= 0 || HD % 2) return BX_EARG;
  if (N == 0) return BX_OK;
  rope_kernel<<<N, US_THREADS, 0, (cudaStream_t)stream>>>((const i64*)y, (const i64*)cos, (const i64*)sin,
                                                        (const i64*)pos, (i64*)Pq, (i64*)k, (i64*)v, H, HKV, HD);
  return launched(1);
}

int bx_softmax_w(const int64_t* raw, const uint8_t* ok, const int64_t* qpos, const int64_t* sh, const int64_t* lut,
                 int64_t l2e, const int32_t* ptab, int32_t* p, int64_t* den, int R, int S, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!raw || !p || !den || R < 0 || S < 1 || (!ok && !qpos)) return BX_EARG;
  if (!ptab && (!sh || !lut)) return BX_EARG;
  if (R == 0) return BX_OK;
  AttnParams w{};
  w.lut = (const i64*)lut;
  w.l2e = (i64)l2e;
  w.ptab = ptab;
  softmax_w_kernel<<<R, US_THREADS, 0, (cudaStream_t)stream>>>((const i64*)raw, ok, (const i64*)qpos,
                                                             ptab ? nullptr : (const i64*)sh, w, p, (i64*)den, S);
  return launched(1);
}

int bx_exact_attn_div(const int64_t* num, const int64_t* den, int64_t* o, int Z, int HD, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!num || !den || !o || Z < 0 || HD < 1) return BX_EARG;
  if (Z == 0) return BX_OK;
  attn_div_kernel<<<Z, US_THREADS, 0, (cudaStream_t)stream>>>((const i64*)num, (const i64*)den, (i64*)o, HD);
  return launched(1);
}

int bx_int8_post_acc(const int64_t* acc, const int64_t* mul, int64_t fmsh, const int64_t* mant, const int64_t* e,
                     int64_t* y, int32_t* flag, int M, int N, int checked, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!acc || !mul || !mant || !e || !y || !flag || M < 0 || N <= 0) return BX_EARG;
  if (M == 0) return BX_OK;
  const int64_t total = (int64_t)M * N;
  int blocks = (int)((total + 255) / 256);
  if (blocks > 148 * 16) blocks = 148 * 16;
  i8::int8_post_acc_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>((const i64*)acc, (const i64*)mul, (i64)fmsh,
                                                                   (const i64*)mant, (const i64*)e, (i64*)y, flag, M, N,
                                                                   checked);
  return launched(1);
}

int bx_pcg_seed_state(const int64_t* keys, int64_t* st, int n, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!keys || !st || n < 0) return BX_EARG;
  if (n == 0) return BX_OK;
  pcg_seed_state_kernel<<<(n + 127) / 128, 128, 0, (cudaStream_t)stream>>>((const i64*)keys, (i64*)st, n);
  return launched(1);
}

int bx_pcg_raw_from_state(const int64_t* st, int64_t* out, int n, int V, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!st || !out || n < 0 || V <= 0) return BX_EARG;
  if (n == 0) return BX_OK;
  const int run = 16;
  const int blocks = (V + run * SAMPLE_THREADS - 1) / (run * SAMPLE_THREADS);
  pcg_raw_state_kernel<<<dim3(blocks, n), SAMPLE_THREADS, 0, (cudaStream_t)stream>>>((const i64*)st, (i64*)out, V, run);
  return launched(1);
}

int bx_bmm(const void* a, int a_is_int64, const void* b, int b_is_int64, int64_t* c, int Z, int M, int N, int K,
           int64_t saz, int64_t sam, int64_t sak, int64_t sbz, int64_t sbk, int64_t sbn, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!a || !b || !c || Z < 0 || M < 0 || N < 0 || K < 0 || K >= 43690 || Z > 65535) return BX_EARG;
  if (Z == 0 || M == 0 || N == 0) return BX_OK;
  const dim3 grid((N + BMM_T - 1) / BMM_T, (M + BMM_T - 1) / BMM_T, Z);
  if (grid.y > 65535) return BX_EARG;
  cudaStream_t st = (cudaStream_t)stream;
  if (a_is_int64 && b_is_int64)
    bmm_kernel<i64, i64><<<grid, 256, 0, st>>>((const i64*)a, (const i64*)b, (i64*)c, M, N, K, saz, sam, sak, sbz, sbk, sbn);
  else if (a_is_int64)
    bmm_kernel<i64, int32_t><<<grid, 256, 0, st>>>((const i64*)a, (const int32_t*)b, (i64*)c, M, N, K, saz, sam, sak, sbz, sbk, sbn);
  else if (b_is_int64)
    bmm_kernel<int32_t, i64><<<grid, 256, 0, st>>>((const int32_t*)a, (const i64*)b, (i64*)c, M, N, K, saz, sam, sak, sbz, sbk, sbn);
  else
    bmm_kernel<int32_t, int32_t><<<grid, 256, 0, st>>>((const int32_t*)a, (const int32_t*)b, (i64*)c, M, N, K, saz, sam, sak, sbz, sbk, sbn);
  return launched(1);
}

// ---- bmm on the tensor pipe (bmm_limb.cuh) ----
size_t bx_bmm_limb_scratch_bytes(int Z, int M, int N, int K) {
  if (Z <= 0 || M < 0 || N < 0 || K < 0) return 0;
  const size_t K16 = ((size_t)K + 15) / 16 * 16;
  return 3 * (size_t)Z * ((size_t)M + (size_t)N) * K16 + 16;
}

int bx_bmm_limb(const void* a, int a_is_int64, const void* b, int b_is_int64, int64_t* c, int Z, int M, int N, int K,
                int64_t saz, int64_t sam, int64_t sak, int64_t sbz, int64_t sbk, int64_t sbn, int8_t* scratch,
                int tile_rows, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (Z < 0 || M < 0 || N < 0 || K < 0 || K >= 43690) return BX_EARG;
  if (Z == 0 || M == 0 || N == 0) return BX_OK;
  if (!c) return BX_EARG;
  cudaStream_t st = (cudaStream_t)stream;
  if (K == 0)                                        // an empty sum (the operands may be null pointers)
    return cudaMemsetAsync(c, 0, sizeof(int64_t) * (size_t)Z * M * N, st) == cudaSuccess ? BX_OK : BX_ELAUNCH;
  if (!a || !b || !scratch || !aligned16(scratch)) return BX_EARG;
  const int K16 = (K + 15) / 16 * 16;
  int8_t* pa = scratch;
  int8_t* pb = scratch + 3 * (size_t)Z * M * K16;
  if (a_is_int64) launch_bmm_pack<i64>(a, saz, sam, sak, pa, Z, M, K, K16, st);
  else launch_bmm_pack<int32_t>(a, saz, sam, sak, pa, Z, M, K, K16, st);
  if (b_is_int64) launch_bmm_pack<i64>(b, sbz, sbn, sbk, pb, Z, N, K, K16, st);      // rows of b^T: columns of b
  else launch_bmm_pack<int32_t>(b, sbz, sbn, sbk, pb, Z, N, K, K16, st);
  int ta = tile_rows;
  if (ta == 0) {
    ta = M <= 16 ? 16 : M <= 32 ? 32 : M <= 48 ? 48 : M <= 64 ? 64 : 80;
    if (M > 80) {
      long best = -1;
      const int cand[3] = {80, 64, 48};
      for (int i = 0; i < 3; ++i) {
        const long cost = (long)((M + cand[i] - 1) / cand[i]) * (cand[i] + 16);
        if (best < 0 || cost < best) { best = cost; ta = cand[i]; }
      }
    }
  }
  CUtensorMap mb, ma;
  if (!make_map(&mb, pb, (uint64_t)K16, (uint64_t)Z * N, 3, WROWS)) return BX_ELAUNCH;
  if (!make_map(&ma, pa, (uint64_t)K16, (uint64_t)Z * M, 3, (uint32_t)ta)) return BX_ELAUNCH;
  BmmEpiParams ep{c, M, N};
  switch (ta) {
    case 16: return launch_bmm_limb<16>(mb, ma, ep, Z, K16, st);
    case 32: return launch_bmm_limb<32>(mb, ma, ep, Z, K16, st);
    case 48: return launch_bmm_limb<48>(mb, ma, ep, Z, K16, st);
    case 64: return launch_bmm_limb<64>(mb, ma, ep, Z, K16, st);
    case 80: return launch_bmm_limb<80>(mb, ma, ep, Z, K16, st);
    default: return BX_EARG;
  }
}

int bx_exact_epilogue(const int64_t* T, const int64_t* B, const int32_t* q, int64_t ldq, const int32_t* cnt,
                      const int32_t* ec, const int64_t* ev, int R, const int64_t* d, const int64_t* g,
                      const int64_t* sh, int64_t* y, int32_t* flag, int M, int N, int checked, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!T || !d || !g || !sh || !y || !flag || M < 0 || N <= 0) return BX_EARG;
  if (cnt && (!q || !ec || !ev || R <= 0)) return BX_EARG;
  if (M == 0) return BX_OK;
  const int64_t total = (int64_t)M * N;
  int64_t blocks = (total + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  epilogue_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>((const i64*)T, (const i64*)B, q, ldq, cnt, ec,
                                                                      (const i64*)ev, R, (const i64*)d, (const i64*)g,
                                                                      (const i64*)sh, (i64*)y, flag, M, N, checked);
  return launched(1);
}

int bx_int8_mm(const int8_t* a, const int8_t* w, int32_t* c, int M, int N, int K, int tile_rows, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!c) return BX_EARG;
  Int8EpiParams ep{c, nullptr, 0, nullptr, nullptr, nullptr, nullptr, M, N, 0, 0};
  return run_int8<false>(a, w, ep, K, tile_rows, (cudaStream_t)stream);
}

static int int8_linear_post(const int8_t* a, const int8_t* w, const int64_t* mul, int64_t fmsh, const int64_t* mant,
                            const int64_t* e, int64_t* y, int32_t* flag, int M, int N, int K, int checked, int tile_rows,
                            int early, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!mul || !mant || !e || !y || !flag) return BX_EARG;
  Int8EpiParams ep{nullptr, mul, fmsh, mant, e, y, flag, M, N, checked, early};
  return run_int8<true>(a, w, ep, K, tile_rows, (cudaStream_t)stream);
}

int bx_int8_linear_post(const int8_t* a, const int8_t* w, const int64_t* mul, int64_t fmsh, const int64_t* mant,
                        const int64_t* e, int64_t* y, int32_t* flag, int M, int N, int K, int checked, int tile_rows,
                        void* stream) {
  return int8_linear_post(a, w, mul, fmsh, mant, e, y, flag, M, N, K, checked, tile_rows, 0, stream);
}

int bx_int8_linear_post_early(const int8_t* a, const int8_t* w, const int64_t* mul, int64_t fmsh, const int64_t* mant,
                              const int64_t* e, int64_t* y, int32_t* flag, int M, int N, int K, int checked,
                              int tile_rows, void* stream) {
  return int8_linear_post(a, w, mul, fmsh, mant, e, y, flag, M, N, K, checked, tile_rows, 1, stream);
}

int bx_exact_linear(const int32_t* q, int64_t ldq, const int64_t* sh, const int8_t* limbs, const int64_t* d,
                    const int64_t* g, const int32_t* cnt, const int32_t* ec, const int64_t* ev, int R,
                    int8_t* scratch, int64_t* y, int32_t* flag, int M, int N, int K, int checked, int tile_rows,
                    void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!q || !sh || !limbs || !d || !g || !scratch || !y || !flag) return BX_EARG;
  if (M < 0 || N <= 0 || K <= 0 || K % 16 || K >= 43690 || !aligned16(limbs) || !aligned16(scratch)) return BX_EARG;
  if (cnt && (!ec || !ev || R <= 0)) return BX_EARG;
  if (M == 0) return BX_OK;
  int rc = bx_split_limbs(q, ldq, scratch, M, K, stream);
  if (rc != BX_OK) return rc;
  return exact_linear_core(q, ldq, sh, limbs, d, g, cnt, ec, ev, R, scratch, y, flag, M, N, K, checked, tile_rows, 1, stream);
}

static int exact_linear_planes(const int8_t* planes, const int32_t* q, int64_t ldq, const int64_t* sh, const int8_t* limbs,
                           const int64_t* d, const int64_t* g, const int32_t* cnt, const int32_t* ec, const int64_t* ev,
                           int R, int64_t* y, int32_t* flag, int M, int N, int K, int checked, int tile_rows, int early,
                           void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (!planes || !sh || !limbs || !d || !g || !y || !flag) return BX_EARG;
  if (M < 0 || N <= 0 || K <= 0 || K % 16 || K >= 43690 || !aligned16(limbs) || !aligned16(planes)) return BX_EARG;
  if (cnt && (!ec || !ev || R <= 0 || !q)) return BX_EARG;
  if (M == 0) return BX_OK;
  return exact_linear_core(q, ldq, sh, limbs, d, g, cnt, ec, ev, R, planes, y, flag, M, N, K, checked, tile_rows, early, stream);
}

int bx_exact_linear_tile(int M, int N, int K, int residual) {
  if (M < 0 || N <= 0 || K <= 0 || K % 16 || K >= 43690) return BX_EARG;
  return exact_linear_auto(M, N, K, residual != 0);
}

int bx_exact_linear_planes(const int8_t* planes, const int32_t* q, int64_t ldq, const int64_t* sh, const int8_t* limbs,
                           const int64_t* d, const int64_t* g, const int32_t* cnt, const int32_t* ec, const int64_t* ev,
                           int R, int64_t* y, int32_t* flag, int M, int N, int K, int checked, int tile_rows,
                           void* stream) {
  return exact_linear_planes(planes, q, ldq, sh, limbs, d, g, cnt, ec, ev, R, y, flag, M, N, K, checked, tile_rows, 0, stream);
}

int bx_exact_linear_planes_early(const int8_t* planes, const int32_t* q, int64_t ldq, const int64_t* sh,
                                 const int8_t* limbs, const int64_t* d, const int64_t* g, const int32_t* cnt,
                                 const int32_t* ec, const int64_t* ev, int R, int64_t* y, int32_t* flag, int M, int N,
                                 int K, int checked, int tile_rows, void* stream) {
  return exact_linear_planes(planes, q, ldq, sh, limbs, d, g, cnt, ec, ev, R, y, flag, M, N, K, checked, tile_rows, 1, stream);
}

// ---- allocation-free variant of the exact linear ----
// Scratch for the activation limb planes lives in the library image instead of caller memory.
#define BX_STATIC_SCRATCH_BYTES (3u * 256u * 8192u)
static __device__ __align__(256) int8_t g_static_planes[BX_STATIC_SCRATCH_BYTES];

size_t bx_exact_linear_static_max_bytes(void) { return (size_t)BX_STATIC_SCRATCH_BYTES; }

int bx_exact_linear_static(const int32_t* q, int64_t ldq, const int64_t* sh, const int8_t* limbs, const int64_t* d,
                           const int64_t* g, const int32_t* cnt, const int32_t* ec, const int64_t* ev, int R,
                           int64_t* y, int32_t* flag, int M, int N, int K, int checked, int tile_rows, void* stream) {
  if (g_status_seen.load(std::memory_order_relaxed)) return BX_EDEVICE;
  if (M < 0 || K <= 0) return BX_EARG;
  if ((size_t)3 * (size_t)M * (size_t)K > (size_t)BX_STATIC_SCRATCH_BYTES) return BX_ELIMIT;
  // The host-side name of a __device__ array is not a device address; resolve it once per device, with that
  // device current, and hand the real address to the kernels.
  // The table is atomic: first calls that race on one device from several host threads store the same address.
  static std::atomic<int8_t*> dev_ptr[BX_MAX_DEVICES];
  const int dev = current_device();
  if (dev < 0) return BX_ELAUNCH;
  int8_t* planes = dev_ptr[dev].load(std::memory_order_acquire);
  if (!planes) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_static_planes) != cudaSuccess || !p) return BX_ELAUNCH;
    planes = static_cast<int8_t*>(p);
    dev_ptr[dev].store(planes, std::memory_order_release);
  }
  return bx_exact_linear(q, ldq, sh, limbs, d, g, cnt, ec, ev, R, planes, y, flag, M, N, K, checked, tile_rows,
                         stream);
}

}  // extern "C"

#include "forward.cuh"
