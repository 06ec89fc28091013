// The kernels of all layers of a forward call, launched from one call: the same entry points in the same order as the
// engines' Python loops, with every intermediate in one workspace. A step of a few rows is about 150 kernels of 5 .. 20 us, and
// launching them one call at a time from Python took longer than running them (17 prompt tokens: 3.7 ms for 2.1 ms of
// kernels). Included at the end of capi.cu, whose entry points it calls.
#pragma once

namespace {

// Pieces of the workspace on 256-byte boundaries.
struct Carver {
  uint8_t* base;
  size_t used = 0;
  template <class T>
  T* take(size_t n) {
    T* p = base ? reinterpret_cast<T*>(base + used) : nullptr;
    used += (n * sizeof(T) + 255) / 256 * 256;
    return p;
  }
};

struct ExactBuffers {
  int64_t *x, *sh, *y, *shq, *num, *den;
  int32_t *q, *qq;
  int8_t* planes;
  void* scratch;
  size_t scratch_bytes, total;
};

inline int64_t largest(int64_t a, int64_t b, int64_t c) { return a > b ? (a > c ? a : c) : (b > c ? b : c); }

ExactBuffers exact_buffers(void* base, int64_t N, int64_t D, int64_t H, int64_t HKV, int64_t HD, int64_t FF, int nblk, int bs, bool tiles) {
  Carver w{(uint8_t*)base};
  const int64_t K = largest(D, H * HD, FF), O = largest(D, (H + 2 * HKV) * HD, 2 * FF);
  ExactBuffers b;
  b.x = w.take<int64_t>(N * D);
  b.y = w.take<int64_t>(N * O);
  b.q = w.take<int32_t>(N * K);
  b.planes = w.take<int8_t>(3 * N * K);
  b.sh = w.take<int64_t>(N);
  b.qq = w.take<int32_t>(N * H * HD);
  b.shq = w.take<int64_t>(N * H);
  b.num = tiles ? nullptr : w.take<int64_t>(N * H * HD);
  b.den = tiles ? nullptr : w.take<int64_t>(N * H);
  b.scratch_bytes = tiles ? 0 : bx_attention_workspace((int)N, (int)HKV, nblk, bs, 0);
  b.scratch = b.scratch_bytes ? w.take<uint8_t>(b.scratch_bytes) : nullptr;
  b.total = w.used;
  return b;
}

struct Int8Buffers {
  int64_t *x, *mant, *e, *y, *num, *den;
  int32_t* q;
  int8_t* a8;
  void* scratch;
  size_t scratch_bytes, total;
};

Int8Buffers int8_buffers(void* base, int64_t N, int64_t D, int64_t H, int64_t HKV, int64_t HD, int64_t FF, int nblk, int bs, bool tiles) {
  Carver w{(uint8_t*)base};
  const int64_t K = largest(D, H * HD, FF), O = largest(D, (H + 2 * HKV) * HD, 2 * FF);
  Int8Buffers b;
  b.x = w.take<int64_t>(N * D);
  b.y = w.take<int64_t>(N * O);
  b.a8 = w.take<int8_t>(2 * N * K);
  b.mant = w.take<int64_t>(N);
  b.e = w.take<int64_t>(N);
  b.q = w.take<int32_t>(N * H * HD);
  b.num = tiles ? nullptr : w.take<int64_t>(N * H * HD);
  b.den = tiles ? nullptr : w.take<int64_t>(N * H);
  b.scratch_bytes = tiles ? 0 : bx_attention_workspace((int)N, (int)HKV, nblk, bs, 0);
  b.scratch = b.scratch_bytes ? w.take<uint8_t>(b.scratch_bytes) : nullptr;
  b.total = w.used;
  return b;
}

bool step_ok(const bx_step* s, const void* layers) {
  return s && layers && s->emb && s->ids && s->pos && s->slot && s->bt && s->cos && s->sin && s->x && s->flag && s->work &&
         s->layers > 0 && s->N > 0 && s->N <= INT32_MAX && s->D > 0 && s->H > 0 && s->HKV > 0 && s->H % s->HKV == 0 && s->HD > 0 && s->FF > 0 &&
         s->bs > 0 && s->nblk > 0 && (s->tiles ? s->n_tiles >= 0 && s->num && s->den : s->qpos != nullptr);
}

}  // namespace

size_t bx_forward_bytes(int exact, int N, int D, int H, int HKV, int HD, int FF, int nblk, int bs, int tiles) {
  if (N <= 0 || D <= 0 || H <= 0 || HKV <= 0 || HD <= 0 || FF <= 0 || nblk <= 0 || bs <= 0) return 0;
  return exact ? exact_buffers(nullptr, N, D, H, HKV, HD, FF, nblk, bs, tiles != 0).total
               : int8_buffers(nullptr, N, D, H, HKV, HD, FF, nblk, bs, tiles != 0).total;
}

#define BX_TRY(call)                \
  do {                              \
    const int rc_ = (call);         \
    if (rc_ != BX_OK) return rc_;   \
  } while (0)

int bx_exact_forward(const bx_step* s, const bx_exact_layer* layers, void* stream) {
  if (!step_ok(s, layers) || !s->lut) return BX_EARG;
  const int N = (int)s->N, D = (int)s->D, H = (int)s->H, HKV = (int)s->HKV, HD = (int)s->HD, FF = (int)s->FF, G = H / HKV, bs = (int)s->bs,
            nblk = (int)s->nblk, K2 = H * HD;
  const bool tiles = s->tiles != nullptr;
  const ExactBuffers b = exact_buffers(s->work, N, D, H, HKV, HD, FF, nblk, bs, tiles);
  if (b.total > (size_t)s->work_bytes) return BX_EARG;
  int64_t *num = tiles ? s->num : b.num, *den = tiles ? s->den : b.den;
  // Every linear stands directly behind the stage that made its input: its weights may be read early.
  auto linear = [&](const bx_exact_lin& w, int checked) {
    return bx_exact_linear_planes_early(b.planes, b.q, w.K, b.sh, w.limbs, w.d, w.g, w.cnt, w.ec, w.ev, (int)w.R, b.y, s->flag, N, (int)w.N, (int)w.K,
                                        checked, (int)w.tile_rows, stream);
  };
  // The residual stream changes buffers with every sum, and ends in the caller's.
  int64_t *cur = s->x, *other = b.x;
  BX_TRY(bx_exact_norm(0, s->emb, nullptr, s->ids, layers[0].ga_m, layers[0].ga_e, cur, b.q, b.sh, b.planes, s->flag, N, D, 1, stream));
  for (int i = 0; i < (int)s->layers; ++i) {
    const bx_exact_layer& l = layers[i];
    if (l.wqkv.N != (H + 2 * HKV) * HD || l.wqkv.K != D || l.wo.N != D || l.wo.K != K2 || l.wgu.N != 2 * FF || l.wgu.K != D || l.wd.N != D || l.wd.K != FF)
      return BX_EARG;
    BX_TRY(linear(l.wqkv, 0));
    BX_TRY(bx_exact_qkv(b.y, s->cos, s->sin, s->pos, s->slot, l.cache, l.sc_nb, l.sc_h, l.sc_bs, bs, b.qq, b.shq, s->flag, N, H, HKV, HD, stream));
    if (tiles) {
      BX_TRY(bx_prefill_attention(b.qq, b.shq, s->pos, s->tiles, (int)s->n_tiles, l.cache, l.nb, l.sc_nb, l.sc_h, l.sc_bs, bs, s->bt, (int)s->bt64,
                                  s->sbt, nblk, s->lut, s->l2e, nullptr, num, den, HKV, G, HD, 32, stream));
    } else if (s->compact) {
      BX_TRY(bx_exact_attention_tab(b.qq, b.shq, s->qpos, l.cache, l.nb, l.sc_nb, l.sc_h, l.sc_bs, bs, s->bt, (int)s->bt64, s->sbt, nblk, s->rmap,
                                    s->lut, s->l2e, num, den, N, HKV, G, HD, 0, 0, b.scratch, b.scratch_bytes, s->compact, stream));
    } else {
      BX_TRY(bx_exact_attention_ws(b.qq, b.shq, s->qpos, l.cache, l.nb, l.sc_nb, l.sc_h, l.sc_bs, bs, s->bt, (int)s->bt64, s->sbt, nblk, s->rmap,
                                   s->lut, s->l2e, num, den, N, HKV, G, HD, 0, 0, b.scratch, b.scratch_bytes, stream));
    }
    BX_TRY(bx_exact_attn_out(num, den, b.q, b.sh, b.planes, N, K2, HD, stream));
    BX_TRY(linear(l.wo, 1));
    BX_TRY(bx_exact_norm(1, cur, b.y, nullptr, l.gm_m, l.gm_e, other, b.q, b.sh, b.planes, s->flag, N, D, 1, stream));
    BX_TRY(linear(l.wgu, 0));
    BX_TRY(bx_exact_silu_quant(b.y, s->lut, b.q, b.sh, b.planes, s->flag, N, FF, stream));
    BX_TRY(linear(l.wd, 1));
    const bool last = i + 1 == (int)s->layers;
    BX_TRY(bx_exact_norm(1, other, b.y, nullptr, last ? nullptr : layers[i + 1].ga_m, last ? nullptr : layers[i + 1].ga_e, cur, last ? nullptr : b.q,
                         last ? nullptr : b.sh, last ? nullptr : b.planes, s->flag, N, D, last ? 0 : 1, stream));
  }
  return BX_OK;
}

int bx_int8_forward(const bx_step* s, const bx_int8_layer* layers, void* stream) {
  if (!step_ok(s, layers) || !s->ptab || !s->silu || !s->scr) return BX_EARG;
  const int N = (int)s->N, D = (int)s->D, H = (int)s->H, HKV = (int)s->HKV, HD = (int)s->HD, FF = (int)s->FF, G = H / HKV, bs = (int)s->bs,
            nblk = (int)s->nblk, K2 = H * HD;
  const bool tiles = s->tiles != nullptr;
  const Int8Buffers b = int8_buffers(s->work, N, D, H, HKV, HD, FF, nblk, bs, tiles);
  if (b.total > (size_t)s->work_bytes) return BX_EARG;
  int64_t *num = tiles ? s->num : b.num, *den = tiles ? s->den : b.den;
  auto linear = [&](const bx_int8_lin& w) {
    return bx_int8_linear_post_early(b.a8, w.w, w.mul, w.fmsh, b.mant, b.e, b.y, s->flag, N, (int)w.N, (int)w.K, 1, 0, stream);
  };
  int64_t *cur = s->x, *other = b.x;
  BX_TRY(bx_int8_norm(0, s->emb, nullptr, s->ids, layers[0].ga, cur, b.a8, b.mant, b.e, s->flag, N, D, 1, stream));
  for (int i = 0; i < (int)s->layers; ++i) {
    const bx_int8_layer& l = layers[i];
    if (l.wqkv.N != (H + 2 * HKV) * HD || l.wqkv.K != D || l.wo.N != D || l.wo.K != K2 || l.wgu.N != 2 * FF || l.wgu.K != D || l.wd.N != D || l.wd.K != FF)
      return BX_EARG;
    BX_TRY(linear(l.wqkv));
    BX_TRY(bx_int8_qkv(b.y, s->cos, s->sin, s->pos, s->slot, l.cache, l.sc_nb, l.sc_h, l.sc_bs, bs, nullptr, b.q, s->flag, N, H, HKV, HD, stream));
    if (tiles) {
      BX_TRY(bx_prefill_attention(b.q, nullptr, s->pos, s->tiles, (int)s->n_tiles, l.cache, l.nb, l.sc_nb, l.sc_h, l.sc_bs, bs, s->bt, (int)s->bt64,
                                  s->sbt, nblk, nullptr, 0, s->ptab, num, den, HKV, G, HD, 32, stream));
    } else if (s->compact) {
      BX_TRY(bx_int8_attention_tab(b.q, s->qpos, l.cache, l.nb, l.sc_nb, l.sc_h, l.sc_bs, bs, s->bt, (int)s->bt64, s->sbt, nblk, s->rmap, s->ptab, num, den,
                                   N, HKV, G, HD, 0, 0, b.scratch, b.scratch_bytes, s->compact, stream));
    } else {
      BX_TRY(bx_int8_attention_ws(b.q, s->qpos, l.cache, l.nb, l.sc_nb, l.sc_h, l.sc_bs, bs, s->bt, (int)s->bt64, s->sbt, nblk, s->rmap, s->ptab, num, den,
                                  N, HKV, G, HD, 0, 0, b.scratch, b.scratch_bytes, stream));
    }
    BX_TRY(bx_int8_attn_out(num, den, b.a8, b.mant, b.e, N, K2, HD, stream));
    BX_TRY(linear(l.wo));
    BX_TRY(bx_int8_norm(1, cur, b.y, nullptr, l.gm, other, b.a8, b.mant, b.e, s->flag, N, D, 1, stream));
    BX_TRY(linear(l.wgu));
    BX_TRY(bx_int8_silu_quant_tab(b.y, s->silu, s->silu_compact, b.a8, b.mant, b.e, s->scr + 2 * i, N, FF, stream));
    BX_TRY(linear(l.wd));
    const bool last = i + 1 == (int)s->layers;
    BX_TRY(bx_int8_norm(1, other, b.y, nullptr, last ? nullptr : layers[i + 1].ga, cur, last ? nullptr : b.a8, last ? nullptr : b.mant,
                        last ? nullptr : b.e, s->flag, N, D, last ? 0 : 1, stream));
  }
  return bx_int8_flag_end(s->scr, s->flag, (int)s->layers, stream);
}

#undef BX_TRY
