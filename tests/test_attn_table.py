"""The compact weight tables of the decode attention kernels (attn_table): the window they state holds for every interval of
the full table, tables they cannot stand for are declined, and the kernels give the integers of the full table with them."""

import numpy as np
import pytest
import torch

from bitexact_llm_b200 import attn_table
from bitexact_llm_b200.exact.consts import exp2_table
from bitexact_llm_b200.int8 import consts as consts8

L2E = 387270501


def test_exact_window_holds_over_the_table():
    lut = exp2_table("cpu").long()
    tab, window, slack, factor, shift, mtop = attn_table.exact(lut, L2E)
    assert slack == 0 and factor == 8 * L2E and shift == 1 and mtop == 1 << 23 and window <= 16
    i = torch.arange(16384)
    g = torch.Generator().manual_seed(0)
    for rr in (0, 1, 2047, 4095, *torch.randint(0, 4096, (40,), generator=g).tolist()):
        v = lut[i] + (((lut[i + 1] - lut[i]) * rr + (1 << 11)) >> 12)
        w = attn_table._walk(tab.long(), i * 4096 + rr)
        assert bool((w << 29 <= v).all()) and bool((v <= w + window << 29).all()), rr


def test_tables_without_a_compact_form():
    lut = exp2_table("cpu").long()
    rising = lut.clone()
    rising[5000] = 1 << 60
    assert attn_table.exact(rising, L2E) is None
    assert attn_table.exact(lut, 1 << 29) is None and attn_table.exact(lut * 2, L2E) is None
    ptab = consts8.weight_table(consts8.exp_table())
    assert attn_table.int8(ptab) is not None
    for at in (40000, 131000):
        other = ptab.clone()
        other[at] += 7
        assert attn_table.int8(other) is None


@pytest.mark.gpu
@pytest.mark.parametrize("variant", [0, 3, 4, 5, 6])
@pytest.mark.parametrize("mode", ["exact", "int8"])
@pytest.mark.parametrize("R,HKV,M,nblk", [(3, 2, 4, 9), (40, 8, 4, 5), (2, 1, 3, 70), (37, 8, 1, 64)])
def test_decode_attention_with_the_compact_table(mode, variant, R, HKV, M, nblk):
    from bitexact_llm_b200.vllm_plugin import tri_exact_attn, tri_paged
    bs, nb, g = 16, 1 + 80, torch.Generator().manual_seed(R + M)
    rng = lambda lo, hi, *n: torch.randint(lo, hi, n, generator=g)
    k, v = (rng(-(1 << 18), 1 << 18, nb, HKV, bs, 64) >> rng(0, 12, nb, 1, 1, 1) for _ in range(2))
    cache = tri_paged.to_limbs(torch.cat([k, v], -1).int()).cuda()
    bt = rng(1, nb, R, nblk).int().cuda()
    pos = rng(0, nblk * bs, R, 1)
    pos[0] = nblk * bs - 1
    pos[-1] = 0
    qpos = (pos - rng(0, 3, R, M)).clamp(min=0).cuda()
    q = (rng(-(1 << 21), 1 << 21, R, HKV, M, 64) >> rng(0, 9, R, HKV, M, 1)).int()
    if mode == "exact":
        shift = torch.tensor([0, 1, 5, 11, 14, 18, 24, 31, 32, 62])
        sh = (-6 - shift[rng(0, 10, R, HKV, M)]).cuda()
        lut = exp2_table("cuda").long()
        run = lambda c: tri_exact_attn.attend(q.cuda(), sh, qpos, cache, bt, None, lut, L2E, variant=variant, compact=c)
        compact = attn_table.exact(lut, L2E)
    else:
        q >>= 7
        ptab = consts8.weight_table(consts8.exp_table()).cuda()
        run = lambda c: tri_paged.attend(q.cuda(), qpos, cache, bt, ptab, variant=variant, compact=c)
        compact = attn_table.int8(ptab)
    num, den = run(attn_table.to(compact, "cuda"))
    want, wden = run(None)
    assert torch.equal(num, want) and torch.equal(den, wden)
    assert np.unique(den.cpu().numpy()).size > 1


def test_where_the_automatic_choice_uses_the_table():
    """Per block-table width in pages of 16 keys: warps, CTAs per SM, chunks and table of the streaming kernel."""
    from bitexact_llm_b200 import _native as nv
    plan = lambda R, keys, table: nv.lib().bx_attention_plan(R, 8, keys // 16, 16, int(keys > 896), table)
    assert [plan(37, keys, 1) for keys in (64, 80, 576, 592, 832, 848, 1344, 1360, 1888, 1904, 2400, 2416, 8192)] == \
        [441, 440, 440, 821, 821, 820, 820, 421, 421, 420, 420, 1821, 1821]
    assert [plan(37, keys, 0) for keys in (64, 592, 1360, 2416, 8192)] == [440, 820, 420, 1820, 1820]
    assert plan(127, 8192, 0) == 1820 and plan(128, 8192, 0) == 1440 and plan(256, 8192, 1) == 1821
    assert plan(36, 784, 1) == 0 and nv.lib().bx_attention_stream_pairs() == 296


def test_where_the_automatic_choice_splits():
    """With the scratch that bx_attention_workspace asks for: the split on both sides of its widths, what it cannot hold, and what
    an exact table without products takes in its place; the products' 2 KB leave room where 16 KB do not."""
    from bitexact_llm_b200 import _native as nv
    plan = lambda R, keys, table, HKV=8, bs=16: nv.lib().bx_attention_plan(R, HKV, keys // bs, bs, 2, table)
    assert [plan(37, keys, 1) for keys in (592, 832, 896, 912, 1360, 2400, 8192)] == [821, 821, 820, 7, 7, 7, 7]
    assert [plan(128, keys, 1) for keys in (512, 528)] == [440, 7] and [plan(24, keys, 1) for keys in (896, 912)] == [0, 7]
    assert [plan(16, keys, 1) for keys in (1280, 1296)] == [0, 7] and [plan(8, keys, 1) for keys in (2048, 2064)] == [0, 7]
    assert [plan(1, keys, 0) for keys in (3072, 3088)] == [0, 7]
    assert [plan(512, 1040, 1, 1), plan(513, 1040, 1, 1), plan(64, 43200, 1), plan(64, 2048, 1, 8, 128)] == [7, 820, 1821, 0]
    assert [plan(37, keys, 3) for keys in (592, 1360, 2416, 4160, 4176)] == [821, 421, 1821, 1821, 7] and plan(36, 1360, 3) == 7
    assert [plan(37, keys, 2) for keys in (64, 80, 512, 528, 592, 848, 896)] == [441, 441, 441, 440, 821, 821, 821]


def only_streaming(monkeypatch):
    """Variant 0 gets enough scratch for the streaming kernel's chunks, and less than the split asks for."""
    from bitexact_llm_b200.vllm_plugin import tri_exact_attn

    def scratch(device, R, HKV, nblk, bs, variant):
        n = R * HKV * ((nblk * bs + 63) // 64) * 64 * 32
        return torch.empty(n, dtype=torch.uint8, device=device), n
    monkeypatch.setattr(tri_exact_attn, "_scratch", scratch)


def launches(run):
    from bitexact_llm_b200 import _native as nv
    before = nv.lib().bx_launch_count()
    out = run()
    return out, nv.lib().bx_launch_count() - before


@pytest.mark.gpu
@pytest.mark.parametrize("R,nblk", [(37, 1), (75, 4), (37, 37), (40, 52), (37, 85), (41, 118), (37, 151), (38, 300)])
@pytest.mark.parametrize("mode", ["exact", "int8"])
def test_streaming_kernel_with_the_table_equals_the_oracle(mode, R, nblk, monkeypatch):
    """Every form of the streaming kernel that uses the table by itself (both ends of each band of widths), the forced ones, and what
    the automatic choice runs with all its scratch: the full table's integers for all pairs, the CPU oracle's for some; contexts of
    1 key up to the whole table."""
    from bitexact_llm_b200 import _native as nv
    from bitexact_llm_b200.vllm_plugin import tri_exact_attn, tri_paged
    from oracle import exact as ox
    from oracle import int8 as o8
    HKV, M, bs, nb = 8, 3, 16, 401
    assert nv.lib().bx_attention_plan(R, HKV, nblk, bs, int(nblk * bs > 896), 1) % 10 == 1
    g = torch.Generator().manual_seed(R * nblk)
    rng = lambda lo, hi, *n: torch.randint(lo, hi, n, generator=g)
    bits = 18 if mode == "exact" else 13
    k, v = (rng(-(1 << bits), 1 << bits, nb, HKV, bs, 64) >> rng(0, 4, nb, 1, 1, 1) for _ in range(2))
    cache = tri_paged.to_limbs(torch.cat([k, v], -1).int())
    bt = rng(1, nb, R, nblk).int()
    pos = rng(0, nblk * bs, R, 1)
    pos[:4, 0] = torch.tensor([nblk * bs - 1, 0, min(31, nblk * bs - 1), nblk * bs // 2])
    qpos = (pos - rng(0, 3, R, M)).clamp(min=0)
    q = (rng(-(1 << 20), 1 << 20, R, HKV, M, 64) >> rng(0, 6, R, HKV, M, 1)).int()
    pick = np.array([0, 1, 2, 3, R - 1])
    rows = [t.numpy() for t in (q[pick].long(), qpos[pick], cache, bt)]
    if mode == "exact":
        shift = torch.tensor([0, 1, 5, 11, 14, 16, 18, 24, 31, 32, 62])
        sh = -6 - shift[rng(0, 11, R, HKV, M)]
        lut = exp2_table("cuda").long()
        run = lambda c, var=0: tri_exact_attn.attend(q.cuda(), sh.cuda(), qpos.cuda(), cache.cuda(), bt.cuda(), None, lut, L2E,
                                                     variant=var, compact=c)
        compact = attn_table.exact(lut, L2E)
        want = ox.paged_attention(rows[0], sh[pick].numpy(), *rows[1:], pick, ox.exp2_table())
    else:
        q >>= 7
        ptab = consts8.weight_table(consts8.exp_table()).cuda()
        run = lambda c, var=0: tri_paged.attend(q.cuda(), qpos.cuda(), cache.cuda(), bt.cuda(), ptab, variant=var, compact=c)
        compact = attn_table.int8(ptab)
        want = o8.paged_attention(q[pick].long().numpy(), *rows[1:], pick, o8.exp_table())
    compact = attn_table.to(compact, "cuda")
    (num, den), count = launches(lambda: run(compact))
    table = 2 if mode == "exact" else 1
    assert count == (2 if nv.lib().bx_attention_plan(R, HKV, nblk, bs, 2, table) == 7 else 1)
    with monkeypatch.context() as m:
        only_streaming(m)
        assert nv.lib().bx_attention_plan(R, HKV, nblk, bs, 1, table) % 10 == 1
        streamed, count = launches(lambda: run(compact))
        assert count == 1
    for other in (streamed, run(None), run(compact, 5), run(compact, 6), run(None, 3)):
        assert torch.equal(num, other[0]) and torch.equal(den, other[1])
    assert np.array_equal(num.cpu().numpy()[pick], want[0])
    assert np.array_equal(den.cpu().numpy()[pick].reshape(want[1].shape), want[1])


@pytest.mark.gpu
def test_many_pairs_in_chunks_without_a_table(monkeypatch):
    """From 1024 pairs on 4-warp CTAs serve wide block tables for callers without a compact table, where the split has too little
    scratch."""
    from bitexact_llm_b200 import _native as nv
    from bitexact_llm_b200.vllm_plugin import tri_exact_attn, tri_paged
    R, HKV, M, bs, nblk, nb = 129, 8, 4, 16, 160, 200
    assert nv.lib().bx_attention_plan(R, HKV, nblk, bs, 1, 0) == 1440
    g = torch.Generator().manual_seed(5)
    rng = lambda lo, hi, *n: torch.randint(lo, hi, n, generator=g)
    cache = tri_paged.to_limbs((rng(-(1 << 18), 1 << 18, nb, HKV, bs, 128)).int()).cuda()
    bt, pos = rng(1, nb, R, nblk).int().cuda(), rng(0, nblk * bs, R, 1)
    pos[:20] = rng(0, 40, 20, 1)
    qpos = pos.expand(-1, M).contiguous().cuda()
    q, sh = rng(-(1 << 20), 1 << 20, R, HKV, M, 64).int().cuda(), (-6 - rng(12, 20, R, HKV, M)).cuda()
    run = lambda var: tri_exact_attn.attend(q, sh, qpos, cache, bt, None, exp2_table("cuda").long(), L2E, variant=var)
    num, den = run(0)
    for var in (3, 5, 6):
        other = run(var)
        assert torch.equal(num, other[0]) and torch.equal(den, other[1])
    only_streaming(monkeypatch)
    other, count = launches(lambda: run(0))
    assert count == 1 and torch.equal(num, other[0]) and torch.equal(den, other[1])


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["exact", "int8"])
@pytest.mark.parametrize("R,HKV,nblk", [(520, 1, 70), (513, 1, 160), (64, 8, 2700)])
def test_what_the_split_cannot_hold(mode, R, HKV, nblk):
    """More than 512 requests, or more than 1024 pages a CTA by table width: variant 0 streams, with and without a compact table."""
    from bitexact_llm_b200 import _native as nv
    from bitexact_llm_b200.vllm_plugin import tri_exact_attn, tri_paged
    M, bs, nb = 4, 16, 200
    g = torch.Generator().manual_seed(R + nblk)
    rng = lambda lo, hi, *n: torch.randint(lo, hi, n, generator=g)
    cache = tri_paged.to_limbs((rng(-(1 << 18), 1 << 18, nb, HKV, bs, 128) >> rng(0, 5, nb, 1, 1, 1)).int()).cuda()
    bt, pos = rng(1, nb, R, nblk).int().cuda(), rng(0, min(nblk * bs, 1500), R, 1)
    pos[3] = min(nblk * bs, 5000) - 1
    qpos = pos.expand(-1, M).contiguous().cuda()
    q, sh = rng(-(1 << 20), 1 << 20, R, HKV, M, 64).int().cuda(), (-6 - rng(12, 20, R, HKV, M)).cuda()
    if mode == "exact":
        lut = exp2_table("cuda").long()
        form = attn_table.to(attn_table.exact(lut, L2E), "cuda")
        run = lambda c, var: tri_exact_attn.attend(q, sh, qpos, cache, bt, None, lut, L2E, variant=var, compact=c)
    else:
        q >>= 7
        ptab = consts8.weight_table(consts8.exp_table()).cuda()
        form = attn_table.to(attn_table.int8(ptab), "cuda")
        run = lambda c, var: tri_paged.attend(q, qpos, cache, bt, ptab, variant=var, compact=c)
    want = run(None, 3 if nblk < 1000 else 5)
    for c, table in ((form, 2 if mode == "exact" else 1), (None, 0)):
        assert nv.lib().bx_attention_plan(R, HKV, nblk, bs, 2, table) > 100
        got, count = launches(lambda: run(c, 0))
        assert count == 1 and torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def test_products_are_the_tables_they_stand_for():
    """The doubles behind a compact table: every entry within the bound that weights are rounded by, and the mark of a table that
    is none of products."""
    lut = exp2_table("cpu").long()
    t = attn_table.products(lut)
    i = torch.arange(16384)
    for rr in (0, 1, 2048, 4095):
        v = lut[i].double() * 2.0 ** -60 + (lut[i + 1] - lut[i]).double() * rr * 2.0 ** -72
        w = t[i >> 7] * t[128 + (i & 127)]
        assert bool(((w + w * (t[256] * rr) - v).abs() <= 2.0 ** -49).all())      # a weight of 22 bits to 2^-27
    other = (lut >> 1) + (1 << 58)
    assert attn_table.products(other) is None
    a, b = attn_table.exact(lut, L2E)[0], attn_table.exact(other, L2E)[0]
    assert a.shape == b.shape and int(a[4099]) == 1 and int(b[4099]) == 0


def halved(lut):
    """A table with a compact form that is none of products."""
    return (lut >> 1) + (1 << 58)


def test_tables_of_another_kind_keep_their_entries():
    lut = exp2_table("cpu").long()
    assert attn_table.native(attn_table.exact(lut, L2E)).shift == 257
    form = attn_table.exact(halved(lut), L2E)
    assert attn_table.native(form).shift == 1 and attn_table.native(attn_table.to(form, "cpu")).shift == 1
    i, tab = torch.arange(16384), form[0][:attn_table.ENTRIES].long()
    for rr in (0, 1, 2047, 4095):                                # the window holds for what the kernels then read
        v = halved(lut)[i] + (((halved(lut)[i + 1] - halved(lut)[i]) * rr + (1 << 11)) >> 12)
        w = attn_table._walk(tab, i * 4096 + rr)
        assert bool((w << 29 <= v).all()) and bool((v <= w + form[1] << 29).all()), rr


@pytest.mark.gpu
@pytest.mark.parametrize("R,nblk", [(37, 4), (37, 37), (37, 85), (38, 150), (37, 261), (4, 261)])
def test_entries_of_an_exact_table_that_is_none_of_products(R, nblk):
    """The streaming kernel reads them, the others the full table; on both sides of where the split takes over."""
    from bitexact_llm_b200.vllm_plugin import tri_exact_attn, tri_paged
    HKV, M, bs, nb = 8, 4, 16, 301
    g = torch.Generator().manual_seed(R * nblk)
    rng = lambda lo, hi, *n: torch.randint(lo, hi, n, generator=g)
    cache = tri_paged.to_limbs((rng(-(1 << 18), 1 << 18, nb, HKV, bs, 128) >> rng(0, 4, nb, 1, 1, 1)).int()).cuda()
    bt, pos = rng(1, nb, R, nblk).int().cuda(), rng(0, nblk * bs, R, 1)
    pos[0] = nblk * bs - 1
    qpos = (pos - rng(0, 3, R, M)).clamp(min=0).cuda()
    q = (rng(-(1 << 20), 1 << 20, R, HKV, M, 64) >> rng(0, 6, R, HKV, M, 1)).int().cuda()
    sh = (-6 - rng(10, 20, R, HKV, M)).cuda()
    lut = halved(exp2_table("cuda").long())
    form = attn_table.to(attn_table.exact(lut, L2E), "cuda")
    run = lambda c, var: tri_exact_attn.attend(q, sh, qpos, cache, bt, None, lut, L2E, variant=var, compact=c)
    want = run(None, 3)
    for c, var in ((form, 0), (form, 5), (form, 6), (form, 3), (form, 7), (None, 0)):
        got = run(c, var)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]), var
    assert want[1].unique().numel() > 1
