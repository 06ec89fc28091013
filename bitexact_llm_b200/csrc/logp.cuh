// Integer log p of given tokens from int64 logits rows [M, V] at fr fractional bits.
//
// log p(tok) = (l_tok - max) - ln(sum_v e^(l_v - max)), everything an int64: the terms e^z come from a table of e^x
// at 44 bits with step 2^-12 over [-40, 0] (linear interpolation on the fr - 12 low bits, rounded; arguments below
// -40 take the first entry), their sum S is < 2^62 and exact in any order, ln S comes from the sampler's ln table.
// The result is an integer at 2^-40. Same integers as int_logp (src/bitexact/vllm_plugin/rl.py:43-65) and as the
// chunked two-pass form of src/bitexact/vllm_plugin/tri_logp.py:27-91.
//
// Two passes over the rows: logp_max_kernel reduces every (row, column chunk) to
// its maximum, logp_sum_kernel first folds the row's chunk maxima (or takes a row maximum given by the caller: a
// column shard sums against the maximum of the full row), then sums its chunk's terms. logp_finish_kernel works on
// [M]: the sum over the chunks, ln S and the target term. The first pass is bound by HBM (8 M V bytes). Gathering the terms' entries
// from the 2.6 MB table bound the second one to 2.7 TB/s (700 rows of 128256: 267 us); made from products of doubles in shared memory it
// takes 187 us, bound by the random 8-byte reads of those (L1 / shared memory 82 % busy).
#pragma once

#include "sampler.cuh"
#include "stage_math.cuh"

namespace bx {

constexpr int LOGP_THREADS = 256;
constexpr int LSE_FE = 44, LSE_MIN = -40, LSE_STEP = 12;
constexpr int LSE_LAST = -LSE_MIN << LSE_STEP;             // index of e^0 = the last table entry
constexpr i64 LOGP_INVALID = (i64)(-0x7fffffffffffffffll - 1);

__device__ __forceinline__ i64 block_max_i64(i64 v, i64* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = imax(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  v = red[0];
#pragma unroll
  for (int w = 1; w < LOGP_THREADS / 32; ++w) v = imax(v, red[w]);
  return v;
}

// One term e^(x - mx) at LSE_FE bits (rl.py:51-59): table entry of the clamped argument's top bits, interpolated on
// the s = fr - 12 low bits with a rounding shift. tab2[i] = (entry i, entry min(i + 1, last)): the two entries of an
// interpolation come with one 16-byte gather (the table is 2.6 MB, so most gathers go to L2 and their count is what
// the pass is bound by).
__device__ __forceinline__ i64 lse_term(i64 x, i64 mx, const longlong2* __restrict__ tab2, int fr) {
  const int s = fr - LSE_STEP;
  const i64 zc = imax(x - mx, -((i64)(-LSE_MIN) << fr));
  const i64 zi = zc >> s;
  const i64 r = zc - shl(zi, s);
  const longlong2 ab = __ldg(tab2 + (int)(zi + LSE_LAST));
  return ab.x + (((ab.y - ab.x) * r + ((i64)1 << (s - 1))) >> s);
}

// The table's entries as products: 2^44 e^(-e / 4096) = t[e >> 8] t[LSE_A + (e & 255)], e steps below the last one; product and
// entry differ by at most 1/2 and 2^-49 of the product, so its rounding is the entry unless it lies that close to a boundary (one in 2^4
// at e^0, one in 2^(4 + 1.44 z) at e^-z). Whether a table is of this kind is seen by the first pass: each of its first LSE_PARTS CTAs
// holds a slice of it against e^x and leaves a word.
constexpr int LSE_A = LSE_LAST / 256 + 1, LSE_PARTS = 1024;
constexpr double LSE_ONE = 17592186044416.0, LSE_REL = 8.881784197001252e-16;      // 2^44, 2^-50
__device__ __forceinline__ void lse_products(double* t) {
  for (int i = threadIdx.x; i < LSE_A + 256; i += blockDim.x) t[i] = i < LSE_A ? LSE_ONE * exp(-i / 16.0) : exp(-(i - LSE_A) / 4096.0);
}
__device__ __forceinline__ bool lse_check(const longlong2* __restrict__ tab2, int part, int parts) {
  bool ok = true;
  for (int i = part * blockDim.x + threadIdx.x; i <= LSE_LAST; i += parts * blockDim.x) {
    const longlong2 ab = __ldg(tab2 + i);
    const double w = LSE_ONE * exp((i - LSE_LAST) / 4096.0);
    ok &= ab.x >= 0 && ab.x <= (1ll << LSE_FE) && fabs(to_f64(ab.x) - w) <= 0.5 + w * LSE_REL && ab.y == __ldg(tab2 + min(i + 1, LSE_LAST)).x;
  }
  return ok;
}
// lse_term as a whole double; `unsure` where an entry is.
__device__ __forceinline__ double lse_product(i64 x, i64 mx, const double* t, uint32_t lim, int s, bool& unsure) {
  const u64 far = (u64)(mx - x);
  const uint32_t d = (uint32_t)(far >> 32) ? lim : min((uint32_t)far, lim);
  const uint32_t e = (d + (1u << s) - 1) >> s, r = (e << s) - d;
  const double a = t[e >> 8] * t[LSE_A + (e & 255)], b = a * 1.000244170429747855;      // the entry above: e^(1 / 4096)
  const double na = a + F2I, nb = b + F2I;
  const int near = __double2hiint(fma(b, -2 * LSE_REL, 0.5));       // upper words: a difference of as much or more is unsure
  unsure = max(__double2hiint(a - (na - F2I)) & 0x7fffffff, __double2hiint(b - (nb - F2I)) & 0x7fffffff) >= near;
  const double rs = __hiloint2double(0x43300000 - (s << 20), (int)r) - __hiloint2double((1075 - s) << 20, 0);      // r 2^-s
  return __dadd_rd(fma(nb - na, rs, 0.5), na) - F2I;
}

// grid (nch, M): pmax[row * nch + chunk] = max of logits[row, chunk columns].
// fits (may be null): whether the CTA's slice of the table is what lse_product takes it for.
__global__ void __launch_bounds__(LOGP_THREADS) logp_max_kernel(const i64* __restrict__ lg, i64 ld, i64* __restrict__ pmax,
                                                                 int V, int ch, int nch, const longlong2* __restrict__ tab2,
                                                                 int* __restrict__ fits) {
  __shared__ i64 red[LOGP_THREADS / 32];
  const int row = blockIdx.y, c0 = blockIdx.x * ch, c1 = min(c0 + ch, V);
  const i64* x = lg + (i64)row * ld;
  i64 v = LOGP_INVALID;
  int c = c0 + threadIdx.x;
  for (; c + 3 * LOGP_THREADS < c1; c += 4 * LOGP_THREADS) {
    const i64 a0 = __ldg(x + c), a1 = __ldg(x + c + LOGP_THREADS), a2 = __ldg(x + c + 2 * LOGP_THREADS),
              a3 = __ldg(x + c + 3 * LOGP_THREADS);
    v = imax(imax(v, a0), imax(imax(a1, a2), a3));
  }
  for (; c < c1; c += LOGP_THREADS) v = imax(v, __ldg(x + c));
  v = block_max_i64(v, red);
  if (threadIdx.x == 0) pmax[(i64)row * nch + blockIdx.x] = v;
  const int id = blockIdx.y * gridDim.x + blockIdx.x;
  if (fits && id < LSE_PARTS) {
    const int ok = __syncthreads_and(lse_check(tab2, id, min((int)(gridDim.x * gridDim.y), LSE_PARTS)));
    if (threadIdx.x == 0) fits[id] = ok;
  }
}

// tab2[i] = (tab[i], tab[min(i + 1, n - 1)]).
__global__ void logp_pair_table_kernel(const i64* __restrict__ tab, longlong2* __restrict__ tab2, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) tab2[i] = make_longlong2(tab[i], tab[min(i + 1, n - 1)]);
}

// grid (nch, M): psum[row * nch + chunk] = sum of the chunk's terms against the row maximum: rowmax[row] when given,
// else the maximum of the row's nch_max chunk maxima in pmax (which it also leaves in rowmax_out[row], chunk 0).
__global__ void __launch_bounds__(LOGP_THREADS) logp_sum_kernel(const i64* __restrict__ lg, i64 ld,
                                                                 const i64* __restrict__ rowmax,
                                                                 const i64* __restrict__ pmax, int nch_max,
                                                                 i64* __restrict__ rowmax_out,
                                                                 const longlong2* __restrict__ tab, const int* __restrict__ fits,
                                                                 i64* __restrict__ psum, int V, int ch, int nch, int fr) {
  __shared__ i64 red[LOGP_THREADS / 32];
  __shared__ double products[LSE_A + 256];
  bool product = fits != nullptr;
  if (product) {
    lse_products(products);
    const int parts = min((int)(gridDim.x * gridDim.y), LSE_PARTS);
    for (int i = threadIdx.x; i < parts; i += LOGP_THREADS) product &= fits[i] != 0;
    product = __syncthreads_and(product);
  }
  const int row = blockIdx.y, c0 = blockIdx.x * ch, c1 = min(c0 + ch, V);
  i64 mx;
  if (rowmax) {
    mx = __ldg(rowmax + row);
  } else {
    i64 v = LOGP_INVALID;
    for (int j = threadIdx.x; j < nch_max; j += LOGP_THREADS) v = imax(v, pmax[(i64)row * nch_max + j]);
    mx = block_max_i64(v, red);
    if (blockIdx.x == 0 && threadIdx.x == 0) rowmax_out[row] = mx;
    __syncthreads();                                       // red is reused below
  }
  const i64* x = lg + (i64)row * ld;
  i64 acc = 0;
  int c = c0 + threadIdx.x;
  constexpr int U = 8;                                     // gathers in flight per thread: the pass is latency bound
  if (product) {
    const uint32_t lim = (uint32_t)(-LSE_MIN) << fr;
    const auto term = [&](i64 v) {
      bool unsure;
      const double w = lse_product(v, mx, products, lim, fr - LSE_STEP, unsure);
      return unsure ? to_f64(lse_term(v, mx, tab, fr)) : w;
    };
    for (; c + (U - 1) * LOGP_THREADS < c1; c += U * LOGP_THREADS) {
      i64 a[U];
#pragma unroll
      for (int k = 0; k < U; ++k) a[k] = __ldg(x + c + k * LOGP_THREADS);
      double sum = F2I;                                    // eight terms of at most 2^44
#pragma unroll
      for (int k = 0; k < U; ++k) sum += term(a[k]);
      acc += f64_to_int(sum);
    }
    for (; c < c1; c += LOGP_THREADS) acc += f64_to_int(term(__ldg(x + c)) + F2I);
  }
  for (; c + (U - 1) * LOGP_THREADS < c1; c += U * LOGP_THREADS) {
    i64 a[U];
#pragma unroll
    for (int k = 0; k < U; ++k) a[k] = __ldg(x + c + k * LOGP_THREADS);
#pragma unroll
    for (int k = 0; k < U; ++k) a[k] = lse_term(a[k], mx, tab, fr);
#pragma unroll
    for (int k = 0; k < U; ++k) acc += a[k];
  }
  for (; c < c1; c += LOGP_THREADS) acc += lse_term(__ldg(x + c), mx, tab, fr);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) red[warp] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    i64 t = 0;
#pragma unroll
    for (int w = 0; w < LOGP_THREADS / 32; ++w) t += red[w];
    psum[(i64)row * nch + blockIdx.x] = t;
  }
}

// One thread per row: out[row] = the maximum (sum = 0) or the sum (sum = 1) of the row's n partial values.
__global__ void logp_rowfold_kernel(const i64* __restrict__ part, int n, i64* __restrict__ out, int M, int sum) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= M) return;
  i64 v = part[(i64)row * n];
  for (int j = 1; j < n; ++j) {
    const i64 p = part[(i64)row * n + j];
    v = sum ? v + p : imax(v, p);
  }
  out[row] = v;
}

// One thread per row: S = the sum of nsum partial sums (or S itself, nsum = 1); the target term zt[row] when given,
// else logits[row, tok[row]] - rowmax[row]; out = (max(zt, -2^36) << (40 - fr)) - (ln S - 44 ln 2) (rl.py:61-65).
// A token outside [0, V) (a target term equal to the most negative int64), or a sum below 1, gives the most negative
// int64.
__global__ void logp_finish_kernel(const i64* __restrict__ psum, int nsum, const i64* __restrict__ zt,
                                   const i64* __restrict__ lg, i64 ld, const i64* __restrict__ tok,
                                   const i64* rowmax, const i64* __restrict__ lnt, i64* out, int M, int V, int fr) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= M) return;
  i64 S = 0;
  for (int j = 0; j < nsum; ++j) S += psum[(i64)row * nsum + j];
  i64 z;
  bool ok = S >= 1;
  if (zt) {
    z = zt[row];
    ok = ok && z != LOGP_INVALID;                          // no shard held the token
  } else {
    const i64 t = tok[row];
    ok = ok && t >= 0 && t < V;
    z = ok ? lg[(i64)row * ld + t] - rowmax[row] : 0;
  }
  if (!ok) {
    out[row] = LOGP_INVALID;
    return;
  }
  const i64 lse = ln_q(S, lnt) - (i64)LSE_FE * LN2Q;
  out[row] = shl(imax(z, -((i64)1 << 36)), FLN - fr) - lse;
}

}  // namespace bx
