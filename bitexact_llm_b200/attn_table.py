"""Compact weight tables of the decode attention kernels, made once per engine from the engine's own table.

An attention weight is round(2^top 2^-t) with 2^-t from a 131 KB table with interpolation (exact mode) or an entry of a
524 KB table of e^z (int8 mode). The kernels gather from neither: a CTA keeps 4097 entries of 2^-f (16 KB) in shared
memory, from which a weight is known to within a small window, and goes to the full table only where a rounding boundary
lies in the window. The window is a property of the full table, worked out here over all of its entries; a table that
such a form cannot stand for gets none (None), and the kernels then read the full table for every weight.

In exact mode the doubles of which the entries of a 2^-f table are products (2 KB, `products`) serve better and take the place of the
entries where the table is one of products; any other table keeps the entries.

compact = (int32 tensor of the entries, in exact mode with room for the products behind them, window, slack, factor from a row
distance to t, its left shift, 2^(top + 1)): window in units of the interpolated entry, slack (for a table that was itself rounded) in
units of 2^-32 of a weight; an EntriesOnly where exact mode's table is none of products."""

import ctypes

import torch

T_BITS, W_BITS = 26, 31                # fractional bits of t, bits of an entry
STEP = 1 << 14                         # t steps per segment: 4096 segments
ENTRIES = 4097


class EntriesOnly(tuple):
    """A compact form of exact mode without products: the room behind the entries is empty, and the kernels are told so."""


class Native(ctypes.Structure):
    """bx_compact_table of include/bitexact_b200.h."""
    _fields_ = [("tab", ctypes.c_void_p)] + [(n, ctypes.c_uint32) for n in ("window", "slack", "factor", "mtop")] + [("shift", ctypes.c_int)]


def native(compact):
    tab, window, slack, factor, shift, mtop = compact
    products = tab.shape[0] > ENTRIES and not isinstance(compact, EntriesOnly)
    return Native(tab.data_ptr(), window, slack, factor, mtop, shift | (256 if products else 0))


def products(lut):
    """The doubles of which the entries of a 2^-f table (int64 [16385]) are products: 2^-(i / 128), 2^-(i / 16384) and the slope between
    entries; None where an entry is not, by the bound that csrc/attn_weight_products.cuh rounds weights by."""
    e = lut.detach().cpu().double() * 2.0 ** -60
    t = torch.cat([e[0:16384:128], e[:128], ((e[1] - 1.0) / 4096)[None]])
    w = (t[:128, None] * t[None, 128:256]).reshape(-1)
    ok = float(t[0]) == 1.0 and bool(((e[:-1] - w).abs() <= 2.0 ** -50).all()) and abs(float(e[-1]) - 0.5) <= 2.0 ** -50
    return t if ok else None


def _with_products(tab, t):
    """The entries, and behind them (from byte 16400 on) the products t, with a 1 in front of them; zeros for None."""
    word = torch.tensor([0, 0, 0 if t is None else 1], dtype=torch.int32)
    return torch.cat([tab, word, (torch.zeros(257, dtype=torch.float64) if t is None else t).view(torch.int32)])


def to(compact, device):
    return None if compact is None else type(compact)((compact[0].to(device), *compact[1:]))


def _walk(tab, t):
    """The kernel's w for t (int64 tensors): the interpolated entry below the true value by at most the window."""
    idx, rr = (t & ((1 << T_BITS) - 1)) >> 14, t & (STEP - 1)
    a, b = tab[idx], tab[idx + 1]
    return a - (((a - b) * rr) >> 14)


def _fits(tab):
    return bool((tab >= 1).all()) and bool((tab < 1 << 32).all()) and bool((tab[:-1] >= tab[1:]).all())


def exact(lut, l2e):
    """From the 2^-f table (int64 [16385] at 2^60, linear between the entries) and l2e = round(log2(e) 2^28)."""
    v = lut.detach().cpu().long()
    if v.shape != (16385,) or not (1 << 28) <= int(l2e) < (1 << 29) or int(v.min()) < 1 << 30 or int(v.max()) > 1 << 60:
        return None
    a = v[::4] >> (60 - W_BITS)
    i = torch.arange(16384)
    k, rr = i >> 2, (i & 3) << 12
    off = v[:-1] - ((a[k] << 29) - (a[k] - a[k + 1]) * (rr << 15))       # 2^29 times the distance to the straight line
    lo, hi = int(off.min() >> 29), int(-((-off.max()) >> 29))
    tab = a + (lo - 2)                 # one for the floor of the kernel's product, one for the rounding of the table's rule
    if not _fits(tab) or hi - lo > 60:
        return None
    t = products(v)
    form = _with_products(tab.to(torch.int32), t), hi - lo + 3, 0, int(l2e) * 8, 1, 1 << 23
    return form if t is not None else EntriesOnly(form)


def int8(ptab):
    """From the weight table (int32 [131073], entry 131072 - u is the weight u steps of 2^-12 below the maximum). Every
    entry is compared with what the kernel makes of the compact form."""
    from .exact.consts import exp2_table
    p = ptab.detach().cpu().long()
    if p.shape != (131073,) or int(p[0]) != 0 or not 1 <= int(p[-1]) <= 1 << 22 or int(p[-1]) & (int(p[-1]) - 1):
        return None
    mtop = 2 * int(p[-1])              # 2^(32 - 31) p[-1]: w mtop 2^-n is the weight at 32 fractional bits
    factor = 3098164009                # round(log2(e) 2^31)
    u = torch.arange(131072)
    t = _mulhi_round(u << 15, factor)
    n = t >> T_BITS
    m = torch.where(n < 32, mtop >> n.clamp(max=31), torch.zeros_like(n))
    want = p[131072 - u]
    a = exp2_table("cpu").long()[::4] >> (60 - W_BITS)
    slack = 1 << 21                    # the e^z table has 10 bits more than the weights: its own rounding
    for window in (12, 16, 24, 32):
        tab = a - window // 2 - 4
        if not _fits(tab):
            return None
        r = _walk(tab, t) * m + (1 << 31) - slack
        sure = (r & 0xFFFFFFFF) + window * m + 2 * slack < 1 << 32
        if bool(((r >> 32) == want)[sure].all()):
            return tab.to(torch.int32), window, slack, factor, 15, mtop
    return None


def _mulhi_round(x, k):
    """(x k + 2^31) >> 32 for 0 <= x, k < 2^32 in int64."""
    lo = x * (k & 0xFFFF) + (1 << 31)              # below 2^49
    return (x * (k >> 16) + (lo >> 16)) >> 16
