"""The row-local stages in double precision hold every integer of the oracle: widths with and without remainders, one row, a
few and more than a launch holds at a time, pointers off the wide boundaries, values on and next to rounding boundaries
and values (or gammas) that leave the ranges of the fast forms."""

import numpy as np
import pytest
import torch

from bitexact_llm_b200 import _native as nv
from oracle import exact as ox
from oracle import int8 as o8

pytestmark = pytest.mark.gpu
RNG = np.random.RandomState


def T(a, off=0):
    """On the device, `off` elements behind a 512-byte boundary."""
    a = np.ascontiguousarray(a)
    t = torch.empty(a.size + off, dtype=torch.from_numpy(a).dtype, device="cuda")[off:]
    t.copy_(torch.from_numpy(a).reshape(-1))
    return t.view(a.shape)


def empty(shape, dtype, off):
    n = int(np.prod(shape))
    return torch.empty(n + off, dtype=dtype, device="cuda")[off:].view(shape)


def planes(q):
    out, r = [], q.astype(np.int64)
    for _ in range(3):
        lo = ((r + 128) & 255) - 128
        out.append(lo.astype(np.int8))
        r = (r - lo) >> 8
    return np.stack(out)


def same(q, a8, sh, wq, wsh):
    assert np.array_equal(sh.cpu().numpy().reshape(-1), wsh.reshape(-1))
    assert np.array_equal(q.cpu().numpy(), wq)
    assert np.array_equal(a8.cpu().numpy(), planes(wq))


def spread(rng, shape, bits):
    """Values of every size up to 2^bits."""
    return (rng.randint(-(1 << 62), 1 << 62, shape) >> rng.randint(62 - bits, 62, shape)).astype(np.int64)


@pytest.mark.parametrize("D,M,off", [(32, 3, 0), (256, 1, 0), (512, 1300, 0), (1024, 700, 0), (2048, 1, 0), (2048, 301, 1), (4096, 300, 0)])
def test_norm(D, M, off):
    rng = RNG(D + M)
    x = (rng.randn(M, D) * 2.0 ** rng.uniform(4, 30, (M, 1))).round().astype(np.int64)
    y = (rng.randn(M, D) * 2.0 ** 20).round().astype(np.int64)
    x[0] = 1 << 20                                               # all alike: the same quotient everywhere
    y[0] = 0
    if M > 2:
        x[1] = y[1] = 0
        x[2, ::2], x[2, 1::2], y[2] = 3, -5, 0
    if M > 6:
        x[3, 5] = 1 << 39                                        # the largest value without the flag
        x[4] = spread(rng, D, 38)
        x[5, 1] = -(1 << 30)
        x[6] = np.where(np.arange(D) % 3 == 0, 1 << 39, -(1 << 39)) - y[6]
    for gm, ge in ((rng.randint(128, 256, D), rng.randint(-9, -5, D)), (rng.randint(-(1 << 24), 1 << 24, D), rng.randint(-26, -20, D)),
                   (rng.randint(1, 4, D), np.where(np.arange(D) % 5, -1, 9))):
        gm, ge = gm.astype(np.int64), ge.astype(np.int64)
        flag = torch.zeros(1, dtype=torch.int32, device="cuda")
        q, a8 = empty((M, D), torch.int32, off), empty((3, M, D), torch.int8, off)
        sh, xo = empty((M,), torch.int64, 0), empty((M, D), torch.int64, off)
        tx, ty, tm, te = T(x, off), T(y, off), T(gm, off), T(ge, off)
        nv.check(nv.lib().bx_exact_norm(1, tx.data_ptr(), ty.data_ptr(), None, tm.data_ptr(), te.data_ptr(), xo.data_ptr(), q.data_ptr(),
                                        sh.data_ptr(), a8.data_ptr(), flag.data_ptr(), M, D, 1, nv.stream()), "bx_exact_norm")
        wq, wsh, werr = ox.norm_quant(x + y, gm, ge)
        assert np.array_equal(xo.cpu().numpy(), x + y) and bool(flag.item()) == bool(werr)
        same(q, a8, sh, wq, wsh)


@pytest.mark.parametrize("bad", [1 << 40, (1 << 52) + 1, -(1 << 60), (1 << 51) - 1])
def test_norm_of_values_out_of_range(bad):
    """Values that set the flag still give the oracle's integers, with and without the sum stored, and alone."""
    rng = RNG(1)
    M, D = 5, 2048
    x = rng.randint(-(1 << 28), 1 << 28, (M, D)).astype(np.int64)
    x[3, 700] = bad
    gm, ge = rng.randint(128, 256, D).astype(np.int64), np.full(D, -7, np.int64)
    wq, wsh, _ = ox.norm_quant(x, gm, ge)
    tx, tm, te, zero = T(x), T(gm), T(ge), torch.zeros(M, D, dtype=torch.long, device="cuda")
    for mode, store in ((1, True), (2, False), (1, False)):
        flag = torch.zeros(1, dtype=torch.int32, device="cuda")
        q, a8, sh = empty((M, D), torch.int32, 0), empty((3, M, D), torch.int8, 0), empty((M,), torch.int64, 0)
        xo = empty((M, D), torch.int64, 0) if store else None
        nv.check(nv.lib().bx_exact_norm(mode, tx.data_ptr(), zero.data_ptr() if mode == 1 else None, None, tm.data_ptr(), te.data_ptr(),
                                        nv.ptr(xo), q.data_ptr(), sh.data_ptr(), a8.data_ptr(), flag.data_ptr(), M, D, 1, nv.stream()), "norm")
        assert flag.item() == 1
        same(q, a8, sh, wq, wsh)


@pytest.mark.parametrize("FF,N,off", [(1000, 3, 0), (1026, 70, 0), (1028, 2, 0), (4096, 5, 0), (4096, 140, 0), (4096, 400, 0), (4096, 200, 1), (8192, 1, 0), (8192, 100, 0), (8192, 130, 0),
                                      (8192, 40, 1), (8192, 64, 0), (8192, 310, 0), (14336, 20, 0), (14336, 150, 0)])
def test_silu(FF, N, off):
    rng = RNG(FF + N)
    y = (rng.randn(N, 2 * FF) * 2.0 ** rng.uniform(18, 27, (N, 1))).round().astype(np.int64)
    y[0, :7] = [0, 1, -1, 1 << 30, -(1 << 30), (1 << 30) - 1, 1 - (1 << 30)]     # about the ends of the fast form
    y[0, FF:FF + 7] = [1 << 24, (1 << 30) - 1, -(1 << 30), 1 << 20, 5, 1 << 30, -1 - (1 << 30)]
    if N > 2:
        y[1, :FF] = np.arange(FF) * ((1 << 24) // 997) - (25 << 24)              # every size of the argument, where E passes 0
        y[2] = 0
    lut = ox.exp2_table()
    wq, wsh, werr = ox.silu_quant(y, lut)
    ty, tl = T(y, off), T(lut)
    q, a8, sh = empty((N, FF), torch.int32, off), empty((3, N, FF), torch.int8, off), empty((N,), torch.int64, 0)
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    nv.check(nv.lib().bx_exact_silu_quant(ty.data_ptr(), tl.data_ptr(), q.data_ptr(), sh.data_ptr(), a8.data_ptr(), flag.data_ptr(), N, FF,
                                          nv.stream()), "silu")
    assert bool(flag.item()) == bool(werr)
    same(q, a8, sh, wq, wsh)


@pytest.mark.parametrize("H,HD,N,off", [(16, 64, 1, 0), (32, 64, 3, 0), (32, 64, 500, 1), (32, 128, 9, 0), (64, 64, 2, 0), (4, 30, 3, 0)])
def test_attention_division(H, HD, N, off):
    rng = RNG(H + N)
    num = spread(rng, (N, H, HD), 57)
    den = rng.randint(1 << 29, 1 << 36, (N, H, 1)).astype(np.int64)
    num[0, 0] = 64 * (den[0, 0] // 64) * np.arange(HD) // 64                     # quotients on and about the boundaries
    den[0, 1], num[0, 1] = 1 << 30, (np.arange(HD) * 2 + 1) << 24
    den[0, 2] = 0
    if N > 2:
        den[1] = 1 << 28                                                         # the quotient of 2^57 2^5 / 2^28: the integer rule
        den[2] = (1 << 35) - rng.randint(0, 5, (H, 1))
    K2 = H * HD
    d = np.where(den == 0, 1, den)
    o = np.where(den == 0, 0, ox.div_round(num, ox.FR - ox.FV, d)).reshape(N, K2)
    wq, wsh = ox.quant(o, -ox.FR)
    tn, td = T(num, off), T(den)
    q, a8, sh = empty((N, K2), torch.int32, off), empty((3, N, K2), torch.int8, off), empty((N,), torch.int64, 0)
    nv.check(nv.lib().bx_exact_attn_out(tn.data_ptr(), td.data_ptr(), q.data_ptr(), sh.data_ptr(), a8.data_ptr(), N, K2, HD, nv.stream()), "out")
    same(q, a8, sh, wq, wsh)


def same8(a8, mant, e, M, want):
    wq, wm, we = want
    a = a8.cpu().numpy().reshape(2, M, -1).astype(np.int64)
    assert np.array_equal(mant.cpu().numpy(), wm) and np.array_equal(e.cpu().numpy(), we)
    assert np.array_equal(a[0] + (a[1] << 8), wq)


@pytest.mark.parametrize("D,M,off", [(7, 3, 0), (30, 2, 0), (256, 1, 0), (700, 5, 0), (1024, 700, 0), (2048, 301, 1), (3000, 4, 0), (4096, 300, 0)])
def test_int8_norm(D, M, off):
    rng = RNG(D + M)
    x = (rng.randn(M, D) * 2.0 ** rng.uniform(2, 34, (M, 1))).round().astype(np.int64)
    y = (rng.randn(M, D) * 2.0 ** 12).round().astype(np.int64)
    x[0], y[0] = 1 << 16, 0
    if M > 2:
        x[1] = y[1] = 0
        x[2], y[2] = spread(rng, D, 50), 0                        # beyond the flag, and beyond the fast form
    for gamma in ((4096 * (1 + 0.3 * rng.randn(D))).round().astype(np.int64), rng.randint(-(1 << 24), 1 << 24, D).astype(np.int64)):
        if D < 256 and abs(gamma).max() > 1 << 20:
            x[2 % M] >>= 20
        flag = torch.zeros(1, dtype=torch.int32, device="cuda")
        a8, mant, e, xo = empty((2, M, D), torch.int8, off), empty((M,), torch.int64, 0), empty((M,), torch.int64, 0), empty((M, D), torch.int64, off)
        tx, ty, tg = T(x, off), T(y, off), T(gamma, off)
        nv.check(nv.lib().bx_int8_norm(1, tx.data_ptr(), ty.data_ptr(), None, tg.data_ptr(), xo.data_ptr(), a8.data_ptr(), mant.data_ptr(),
                                       e.data_ptr(), flag.data_ptr(), M, D, 1, nv.stream()), "bx_int8_norm")
        assert np.array_equal(xo.cpu().numpy(), x + y)
        ok = [m for m in range(M) if abs(x[m] + y[m]).max() * float(abs(gamma).max()) < 2.0 ** 62]       # the oracle's own range
        wq, wm, we = o8.pre_norm((x + y)[ok], gamma)
        same8(a8.view(2, M, D)[:, ok], mant[ok], e[ok], len(ok), (wq, wm, we))


@pytest.mark.parametrize("bad,want", [((1 << 42) - 1, 0), (1 << 42, 1), (-(1 << 60), 1)])
def test_int8_sum_flag(bad, want):
    x = np.zeros((3, 64), np.int64)
    x[1, 17] = bad
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    tx, ty, xo = T(x), T(np.zeros_like(x)), empty(x.shape, torch.int64, 0)
    nv.check(nv.lib().bx_int8_norm(1, tx.data_ptr(), ty.data_ptr(), None, None, xo.data_ptr(), None, None, None, flag.data_ptr(), 3, 64, 0,
                                   nv.stream()), "bx_int8_norm")
    assert flag.item() == want and np.array_equal(xo.cpu().numpy(), x)


@pytest.mark.parametrize("FF,N,off", [(1000, 3, 0), (1028, 2, 0), (4096, 140, 0), (4096, 400, 0), (4096, 200, 1), (8192, 1, 0), (8192, 40, 1),
                                      (8192, 130, 0), (8192, 310, 0), (14336, 20, 0), (14336, 150, 0)])
def test_int8_silu(FF, N, off):
    from bitexact_llm_b200.int8.consts import silu_compact
    rng = RNG(FF + N)
    y = (rng.randn(N, 2 * FF) * 2.0 ** rng.uniform(8, 19, (N, 1))).round().astype(np.int64)
    edge = 8 << 16
    y[0, :9] = [0, edge, edge - 1, -edge, -edge - 1, -edge + 1, 32 << 16, (1 << 33) + 5, -(1 << 33)]     # the table's ends, and beyond
    y[0, FF:FF + 9] = [(1 << 30) - 1, 1 << 30, -(1 << 30), -(1 << 30) - 1, 1 << 31, 7, -(1 << 20), 1 << 20, 3]
    if N > 2:
        y[1, :FF] = np.arange(FF) * (edge // 997) - 3 * edge
        y[2] = 0
        y[N - 1, 5], y[N - 1, FF + 5] = 32 << 16, 1 << 41                        # h beyond 2^45, in one row
    if N > 5:
        y[4, 9], y[4, FF + 9] = 1 << 36, -(1 << 26)                              # and 2^46
    lut = o8.silu_table()
    wq, wm, we, _ = o8.silu_mul(y, lut)
    ty, tl = T(y, off), T(lut)
    tab = silu_compact(tl)
    a8, mant, e, scr = empty((2, N, FF), torch.int8, off), empty((N,), torch.int64, 0), empty((N,), torch.int64, 0), torch.zeros(2, dtype=torch.long, device="cuda")
    nv.check(nv.lib().bx_int8_silu_quant_tab(ty.data_ptr(), tl.data_ptr(), tab.data_ptr(), a8.data_ptr(), mant.data_ptr(), e.data_ptr(),
                                             scr.data_ptr(), N, FF, nv.stream()), "silu")
    same8(a8, mant, e, N, (wq, wm, we))
    assert scr.tolist() == [int(abs(o8.silu(y[:, :FF], lut)).max()), int(abs(y[:, FF:]).max())]


def test_int8_silu_of_products_beyond_doubles():
    """h of 2^51 and more: the row takes the integer rules, its neighbours do not."""
    from bitexact_llm_b200.int8.consts import silu_compact
    rng = RNG(0)
    lut = o8.silu_table()
    tl = T(lut)
    tab = silu_compact(tl)
    for N in (2, 300):
        y = rng.randint(-(1 << 18), 1 << 18, (N, 8192)).astype(np.int64)
        y[1, 70], y[1, 4096 + 70] = 1 << 36, 1 << 32                              # silu(g) = g there: h = 2^52
        wq, wm, we, _ = o8.silu_mul(y, lut)
        ty = T(y)
        a8, mant, e = empty((2, N, 4096), torch.int8, 0), empty((N,), torch.int64, 0), empty((N,), torch.int64, 0)
        nv.check(nv.lib().bx_int8_silu_quant_tab(ty.data_ptr(), tl.data_ptr(), tab.data_ptr(), a8.data_ptr(), mant.data_ptr(), e.data_ptr(), None,
                                                 N, 4096, nv.stream()), "silu")
        assert 2 ** 51 < (1 << 36) * (1 << 32) >> 16
        same8(a8, mant, e, N, (wq, wm, we))


@pytest.mark.parametrize("H,HD,N,off", [(16, 64, 1, 0), (32, 64, 3, 0), (32, 64, 500, 1), (32, 128, 9, 0), (64, 64, 2, 0), (4, 30, 3, 0)])
def test_int8_attention_division(H, HD, N, off):
    rng = RNG(H + N)
    num = spread(rng, (N, H, HD), 55)
    den = rng.randint(1 << 29, 1 << 36, (N, H, 1)).astype(np.int64)
    num[0, 0] = 64 * (den[0, 0] // 64) * np.arange(HD) // 64
    den[0, 1], num[0, 1] = 1 << 30, (np.arange(HD) * 2 + 1) << 27
    if N > 2:
        den[1] = 1 << 22                                                          # quotients from 2^29 on: the integer rules
        den[2] = (1 << 35) - rng.randint(0, 5, (H, 1))
    K2 = H * HD
    tn, td = T(num, off), T(den)
    a8, mant, e = empty((2, N, K2), torch.int8, off), empty((N,), torch.int64, 0), empty((N,), torch.int64, 0)
    nv.check(nv.lib().bx_int8_attn_out(tn.data_ptr(), td.data_ptr(), a8.data_ptr(), mant.data_ptr(), e.data_ptr(), N, K2, HD, nv.stream()), "out")
    same8(a8, mant, e, N, o8.attn_out(num, den))
