"""The row-local stages in double precision hold every integer of the oracle: widths with and without remainders, one row, a
few and more than a launch holds at a time, pointers off the wide boundaries, values on and next to rounding boundaries
and values (or gammas) that leave the ranges of the fast forms."""

import numpy as np
import pytest
import torch

from bitexact_llm_b200 import _native as nv
from oracle import exact as ox

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
