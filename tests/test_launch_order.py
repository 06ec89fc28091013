"""Kernels that may start before the kernel in front of them has ended (programmatic dependent launch): what they read is
ordered behind everything that was put on the stream before them, weights, scales and tables included."""

import contextlib
import os
import re

import numpy as np
import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "bitexact_llm_b200", "csrc")
READS = re.compile(r"__ldg\(|fill_\w+\(|tma_load\w*\(|\bp\.(qpos|pos|bt|q|sh)\[")


def _integer_sources():
    return {f: open(os.path.join(SRC, f)).read() for f in sorted(os.listdir(SRC)) if f.endswith(".cuh") and not f.startswith("fl_")}


def test_no_kernel_reads_memory_before_its_wait():
    seen = 0
    for name, src in _integer_sources().items():
        for m in re.finditer(r"__global__ .*?^}", src, re.S | re.M):
            body = re.sub(r"//[^\n]*", "", m.group(0)[m.group(0).index("{"):])
            if "wait_previous();" in body:
                seen += 1
                assert not READS.search(body[:body.index("wait_previous();")]), (name, m.group(0)[:200])
            if "launch_next();" in body:                    # the next kernel starts only when all before this one has ended
                assert "wait_previous();" in body[:body.index("launch_next();")], (name, m.group(0)[:200])
    assert seen >= 12


def test_weight_tiles_are_requested_behind_the_wait_unless_asked_for_early():
    seen = 0
    for name, src in _integer_sources().items():
        for m in re.finditer(r"---- TMA producer.*?\n(.*?)wait_previous\(\);", src, re.S):
            seen += 1
            assert re.search(r"const int pre = !(ep\.)?early", m.group(1)) and "for (int i = 0; i < pre;" in m.group(1), name
            assert m.group(1).count("for (") == 1, name      # nothing but those first tiles is asked for in front of the wait
    assert seen == 3


def test_a_late_copy_lands_before_its_cta_ends():
    """Whoever copies into shared memory without a tensor map waits for the copy once more at its end where the first wait ran out."""
    src = _integer_sources()
    kernels = {m.group(1): m.group(0) for f in ("int8_stages.cuh", "paged_attention.cuh")
               for m in re.finditer(r"__global__ .*?(\w+)\(.*?^}", re.sub(r"__launch_bounds__\([^)]*\)*", "", src[f]), re.S | re.M)
               if "bulk_load(" in m.group(0) or "fetch_compact(" in m.group(0)}
    assert sorted(kernels) == ["exact_attention_stream_kernel", "int8_silu_persistent_kernel"]
    for name, body in kernels.items():
        again = re.search(r"if \(!(there|table)\) (mbar_wait\(&table_full, 0\)|wait_table\(\));", body[body.rindex("for (int64_t"):])
        assert again, name


def test_only_the_engines_ask_for_weights_early(monkeypatch):
    from bitexact_llm_b200 import _native as nv
    from bitexact_llm_b200.exact.model import Lin
    from bitexact_llm_b200.int8.gemm_skinny import linear_post
    from bitexact_llm_b200.vllm_plugin import exact_fuse
    from bitexact_llm_b200.vllm_plugin.exact_gemm import FusedLin
    called = []

    class Fake:
        def __getattr__(self, name):
            return lambda *a: called.append(name) or 0

    monkeypatch.setattr(nv, "lib", lambda: Fake())
    monkeypatch.setattr(nv, "stream", lambda: 0)
    empty = torch.zeros(0, dtype=torch.long)
    dec = {"limbs": torch.zeros(3, 8, 16, dtype=torch.int8), "g": torch.zeros(8, dtype=torch.long), "d": torch.zeros(8, dtype=torch.long),
           "rr": empty, "rc": empty, "rv": empty}
    lin, flag = FusedLin(Lin(dec, None, "cpu")), torch.zeros(1, dtype=torch.int32)
    q, sh = torch.zeros(2, 16, dtype=torch.int32), torch.zeros(2, dtype=torch.long)
    exact_fuse.attach_planes(q, torch.zeros(3, 2, 16, dtype=torch.int8))
    lin(q, sh, flag)
    lin(q, sh, flag, early=True)
    lin.timer = lambda *a: contextlib.nullcontext()          # a timer may put work of its own in between
    lin(q, sh, flag, early=True)
    a8, one = torch.zeros(4, 16, dtype=torch.int8), torch.ones(8, dtype=torch.long)
    linear_post(a8, torch.zeros(8, 16, dtype=torch.int8), one, 30, sh, sh, flag)
    linear_post(a8, torch.zeros(8, 16, dtype=torch.int8), one, 30, sh, sh, flag, early=True)
    assert called == ["bx_exact_linear_planes", "bx_exact_linear_planes_early", "bx_exact_linear_planes", "bx_int8_linear_post",
                      "bx_int8_linear_post_early"]


def _decomposed(rng, N, K):
    return {"limbs": rng.randint(-128, 128, (3, N, K)).astype(np.int8), "g": rng.randint(-34, -24, N).astype(np.int64),
            "d": rng.randint(0, 31, N).astype(np.int64), "rr": np.zeros(0, np.int64), "rc": np.zeros(0, np.int64),
            "rv": np.zeros(0, np.int64)}


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(1, 2048, 2048), (20, 3072, 512), (130, 4096, 256), (256, 16384, 256)])
def test_weights_rewritten_on_the_stream(M, N, K):
    """The weights of a linear are overwritten by the kernel in front of it, or by the one in front of the stage that feeds
    it: every call multiplies by the newest."""
    from bitexact_llm_b200.exact.model import Lin
    from bitexact_llm_b200.vllm_plugin import exact_fuse
    from bitexact_llm_b200.vllm_plugin.exact_gemm import FusedLin
    rng = np.random.RandomState(M + N)
    decs = [_decomposed(rng, N, K) for _ in range(2)]
    T = lambda d: {k: torch.from_numpy(v) for k, v in d.items()}
    lins = [FusedLin(Lin(T(d), None, "cuda")) for d in decs]
    live = FusedLin(Lin(T(decs[0]), None, "cuda"))

    class Model:
        D, dev = K, "cuda"
    gammas = [(torch.from_numpy(rng.randint(128, 256, K)).cuda(), torch.from_numpy(rng.randint(-8, -6, K)).cuda()) for _ in range(2)]
    gamma = tuple(t.clone() for t in gammas[0])
    h = torch.from_numpy(rng.randint(-(1 << 30), 1 << 30, (M, K))).cuda()
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    want = []
    for i in range(2):
        q, sh = exact_fuse.pre_norm(Model, h, gammas[i], flag)
        want.append([lin(q, sh, flag) for lin in lins])
    torch.cuda.synchronize()
    q, sh = exact_fuse.pre_norm(Model, h, gammas[0], flag)
    got = []
    for i in range(40):
        a, b = i & 1, (i >> 1) & 1
        for x, y in zip((live.limbs, live.g, live.d), (lins[a].limbs, lins[a].g, lins[a].d)):
            x.copy_(y)
        if i % 3 == 0:                                       # the stage stands between the new weights and the product
            for x, y in zip(gamma, gammas[b]):
                x.copy_(y)
            q, sh = exact_fuse.pre_norm(Model, h, gamma, flag)
            last, out = b, live(q, sh, flag, early=True)
        else:                                                # the new weights are the kernel in front
            live.d.copy_(lins[a].d)
            live.limbs.copy_(lins[a].limbs)
            out = live(q, sh, flag)
        got.append((torch.equal(out, want[last][a]), i))
    assert all(ok for ok, _ in got), got
    assert not torch.equal(want[0][0], want[0][1]) and not torch.equal(want[0][0], want[1][0])


@pytest.mark.gpu
def test_attention_tables_rewritten_on_the_stream():
    """The 2^-f table of an attention call, in full and in its compact form, and the SiLU stage's, made by the kernel in front."""
    from bitexact_llm_b200 import attn_table
    from bitexact_llm_b200.exact.consts import exp2_table
    from bitexact_llm_b200.vllm_plugin import exact_fuse, tri_exact_attn, tri_paged, tri_prefill
    g = torch.Generator().manual_seed(3)
    rng = lambda lo, hi, *n: torch.randint(lo, hi, n, generator=g)
    L2E, HKV, G, bs, nb, R = 387270501, 8, 4, 16, 9, 48
    luts = [exp2_table("cuda").long(), (exp2_table("cuda").long() >> 1) + (1 << 58)]
    compacts = [attn_table.to(attn_table.exact(lut, L2E), "cuda") for lut in luts]
    assert all(c is not None and c[1:] == (c[1], 0, 8 * L2E, 1, 1 << 23) for c in compacts)
    cache = tri_paged.to_limbs(rng(-(1 << 15), 1 << 15, nb, HKV, bs, 128).int()).cuda()
    bt = rng(1, nb, R, 4).int().cuda()
    q, sh = rng(-(1 << 15), 1 << 15, R, HKV, G, 64).int().cuda(), (-6 - rng(14, 22, R, HKV, G)).cuda()
    pos = rng(30, 64, R).cuda()
    qpos = pos.view(-1, 1).expand(-1, G).contiguous()
    tiles = torch.stack([torch.arange(R), torch.arange(R), torch.ones(R, dtype=torch.long)], 1).int().cuda()

    class Model:
        dev = "cuda"
    y = rng(-(1 << 26), 1 << 26, 64, 512).cuda()
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")

    calls = [lambda lut, c: tri_exact_attn.attend(q, sh, qpos, cache, bt, None, lut, L2E),
             lambda lut, c: tri_exact_attn.attend(q, sh, qpos, cache, bt, None, lut, L2E, compact=c),
             lambda lut, c: tri_prefill.attend_exact(q, sh, pos, cache, bt, tiles, lut, L2E),
             lambda lut, c: exact_fuse.silu_quant(Model, y, lut, flag)]
    want = [[call(luts[i], compacts[i]) for call in calls] for i in range(2)]
    torch.cuda.synchronize()
    lut, tab = luts[0].clone(), compacts[0][0].clone()
    window = max(c[1] for c in compacts)                     # a wider window only asks the full table more often
    for i in range(40):
        for call, (num, den) in zip(calls, want[i & 1]):
            lut.zero_()
            tab.fill_(1)
            lut.copy_(luts[i & 1])
            tab.copy_(compacts[i & 1][0])
            if i & 2:
                lut.copy_(luts[i & 1])                       # the full table or the compact one is the last thing written
            x, z = call(lut, (tab, window, *compacts[0][2:]))
            assert torch.equal(x, num) and torch.equal(z, den), i
    assert not torch.equal(want[0][0][1], want[1][0][1])
