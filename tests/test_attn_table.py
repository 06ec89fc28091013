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
