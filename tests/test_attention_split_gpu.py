"""The even split of decode attention over the chip (variant 7) against the oracle: pieces that are a whole pair and pairs cut
anywhere, every page size, contexts from none to thousands of keys, both weight rules, with and without a compact table."""

import numpy as np
import pytest
import torch

from bitexact_llm_b200 import _native as nv
from bitexact_llm_b200 import attn_table
from oracle import exact as ox
from oracle import int8 as o8

pytestmark = pytest.mark.gpu
HD = 64


def T(a, dtype=None):
    t = torch.from_numpy(np.ascontiguousarray(a))
    return (t if dtype is None else t.to(dtype)).cuda()


def cache_planes(rng, nb, HKV, bs, lim):
    c32 = rng.randint(-lim, lim + 1, (nb, HKV, bs, 2 * HD)).astype(np.int64)
    planes = np.zeros((nb, HKV, bs, 8 * HD), dtype=np.int8)
    for part, o in ((c32[..., :HD], 0), (c32[..., HD:], 3)):
        for i, lo in enumerate(ox.split_limbs(part, 3)[0]):
            planes[..., (o + i) * HD:(o + i + 1) * HD] = lo.astype(np.int8)
    planes[..., 6 * HD:] = rng.randint(-128, 128, planes[..., 6 * HD:].shape)       # unused tail: junk
    return planes


@pytest.mark.parametrize("bs", [8, 16, 32, 64])
@pytest.mark.parametrize("R,HKV,M,longest,width", [(1, 1, 1, 1, 64), (1, 8, 4, 70, 128), (3, 2, 4, 3000, 3072), (40, 8, 4, 200, 256),
                                                   (9, 4, 3, 1500, 4096), (130, 3, 2, 64, 64)])
def test_split_holds_the_oracle(bs, R, HKV, M, longest, width):
    from bitexact_llm_b200.vllm_plugin import tri_exact_attn, tri_paged
    rng = np.random.RandomState(R * 7 + bs)
    planes = cache_planes(rng, max(3, 1024 // bs), HKV, bs, 1 << (10 if R % 2 else 22))
    bt = rng.randint(1, planes.shape[0], (R + 2, width // bs)).astype(np.int32 if R % 2 else np.int64)
    rmap = rng.randint(0, R + 2, R).astype(np.int64)
    ctx = rng.randint(1, longest + 1, R)
    ctx[0] = longest
    for i, c in enumerate((64, 65, 128, 63)):                                        # ends of units
        if i + 1 < R and c <= longest:
            ctx[i + 1] = c
    qpos = np.repeat((ctx - 1)[:, None], M, 1).astype(np.int64)
    if R > 6:
        qpos[5] = -1                                                                 # no key at all
        qpos[6, 0] = 0                                                               # a query that sees one key of many
    q = rng.randint(-(1 << 22), (1 << 22) + 1, (R, HKV, M, HD)).astype(np.int64)
    sh = rng.randint(-40, -10, (R, HKV, M)).astype(np.int64)
    lut = ox.exp2_table()
    live = (qpos >= 0).any(1)                                                        # the oracle has no empty context
    wnum, wden = ox.paged_attention(q[live], sh[live], qpos[live], planes, bt, rmap[live], lut)
    tl = T(lut)
    forms = (None, attn_table.to(attn_table.exact(tl, ox.L2E28), "cuda"))
    for form in forms:
        num, den = tri_exact_attn.attend(T(q, torch.int32), T(sh), T(qpos), T(planes), T(bt), T(rmap), tl, ox.L2E28, variant=7, compact=form)
        num, den = num.cpu().numpy(), den.cpu().numpy()
        assert np.array_equal(num[live], wnum) and np.array_equal(den[live], wden)
        assert not num[~live].any() and not den[~live].any()
    expt = o8.exp_table()
    w8n, w8d = o8.paged_attention((q >> 9)[live], qpos[live], planes, bt, rmap[live], expt)
    ptab = T(o8.weight_table(expt), torch.int32)
    for form in (None, attn_table.to(attn_table.int8(ptab), "cuda")):
        num, den = tri_paged.attend(T(q >> 9), T(qpos), T(planes), T(bt), ptab, rmap=T(rmap), variant=7, compact=form)
        assert np.array_equal(num.cpu().numpy()[live], w8n) and np.array_equal(den.cpu().numpy()[live], w8d)
    assert nv.device_status() == 0


def test_split_refuses_what_it_cannot_hold():
    from bitexact_llm_b200.vllm_plugin import tri_exact_attn
    rng = np.random.RandomState(0)
    planes = T(cache_planes(rng, 4, 1, 16, 100))
    R = 513                                                                          # more requests than it has room for
    args = [torch.zeros(R, 1, 1, HD, dtype=torch.int32, device="cuda"), torch.full((R, 1, 1), -20, device="cuda"),
            torch.zeros(R, 1, dtype=torch.long, device="cuda"), planes, torch.zeros(R, 1, dtype=torch.int32, device="cuda"), None, T(ox.exp2_table()),
            ox.L2E28]
    with pytest.raises(RuntimeError):
        tri_exact_attn.attend(*args, variant=7)
    tri_exact_attn.attend(*[a[:512] if torch.is_tensor(a) and a.shape[0] == R else a for a in args], variant=7)
    torch.cuda.synchronize()
    assert nv.device_status() == 0


def test_inputs_rewritten_on_the_stream():
    """Positions, pages, keys and the weight table are overwritten by the kernels right in front of the call: the second kernel, which
    reads them before the first one has ended, sees the newest."""
    from bitexact_llm_b200.vllm_plugin import tri_exact_attn
    rng = np.random.RandomState(3)
    R, HKV, M, bs, nblk = 24, 8, 4, 16, 20
    caches = [T(cache_planes(rng, 40, HKV, bs, 1 << 16)) for _ in range(2)]
    bts = [T(rng.randint(1, 40, (R, nblk)).astype(np.int32)) for _ in range(2)]
    poss = [T(np.repeat(rng.randint(0, nblk * bs, (R, 1)), M, 1).astype(np.int64)) for _ in range(2)]
    luts = [T(ox.exp2_table()), T(ox.exp2_table() // 3)]                             # the second is no table of products
    q, sh = T(rng.randint(-(1 << 20), 1 << 20, (R, HKV, M, HD)), torch.int32), T(rng.randint(-26, -16, (R, HKV, M)))
    call = lambda c, b, p, l, v: tri_exact_attn.attend(q, sh, p, c, b, None, l, ox.L2E28, variant=v)
    want = {}
    for i in range(16):
        pick = [x[i >> k & 1] for k, x in enumerate((caches, bts, poss, luts))]
        want[i] = call(*pick, 3)
    live = [x[0].clone() for x in (caches, bts, poss, luts)]
    torch.cuda.synchronize()
    got = []
    for i in rng.randint(0, 16, 60):
        for k in rng.permutation(4):
            live[k].copy_((caches, bts, poss, luts)[k][i >> k & 1])
        got.append((i, call(*live, 7)))
    torch.cuda.synchronize()
    for i, (num, den) in got:
        assert torch.equal(num, want[i][0]) and torch.equal(den, want[i][1])
    assert nv.device_status() == 0
