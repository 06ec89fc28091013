"""All layers from one call of the library: the residual rows, caches and flag of the engines' own loop over single calls, for decoding
rows and prompt tiles, with and without what an engine may lack, and what that loop alone serves."""

import contextlib

import pytest
import torch

from bitexact_llm_b200 import _native as nv

pytestmark = pytest.mark.gpu


def engine(mode, width, layers, edit=lambda c: c, n_pos=700):
    from bitexact_llm_b200.exact import consts
    cfg = dict(consts.LLAMA_1B, hidden_size=width, intermediate_size=4 * width, num_hidden_layers=layers, num_attention_heads=width // 64,
               num_key_value_heads=width // 256, head_dim=64, vocab_size=512)
    sd = consts.random_state_dict(cfg, seed=width, device="cuda", gamma_jitter=0.1)
    if mode == "exact":
        from bitexact_llm_b200.vllm_plugin.exact_run import ExactEngine
        return ExactEngine(edit(consts.build(cfg, sd, n_pos=n_pos)), "cuda")
    from bitexact_llm_b200.int8 import consts as consts8
    from bitexact_llm_b200.int8.engine import IntEngine
    return IntEngine(edit(consts8.build(cfg, sd, n_pos=n_pos)), "cuda")


def step(eng, ses, seqs, lens, tiles, native, form=True):
    """One forward call on copies of the session's caches."""
    kvs = [c.clone() for c in ses.kvs]
    seq = torch.cat([torch.full((n,), s) for s, n in zip(seqs, lens)]).cuda()
    pos = torch.cat([torch.arange(n) for n in lens]).cuda()
    ids = (seq * 31 + pos * 7) % 512
    slot = ses._slots(seq, pos)
    if len(lens) > 1:
        slot[1] = -1                                             # padding: goes to the null page
    tt, row = [], 0
    for s, n in zip(seqs, lens):
        tt.append((s, row, n, n))
        row += n
    tt = eng.tile_table(tt, ses.bs).cuda() if tiles else None
    if tt is not None and len(lens) > 1:
        tt = tt[1:]                                              # the first tile's rows are in none
    keep = eng.compact
    eng.compact = keep if form else None
    with contextlib.ExitStack() as st:
        if not native:
            st.enter_context(pytest.MonkeyPatch.context()).setattr(type(eng), "_forward_native", lambda *a: None)
        eng.fl.zero_()
        before = nv.lib().bx_launch_count()
        x = eng.forward(kvs, ids, pos, slot, ses.bt, seq, tiles=tt)
        torch.cuda.synchronize()
        out = x, kvs, int(eng.fl), nv.lib().bx_launch_count() - before
    eng.compact = keep
    return out


@pytest.mark.parametrize("mode", ["exact", "int8"])
@pytest.mark.parametrize("width,layers", [(256, 1), (1024, 3)])
def test_the_same_rows_caches_and_flag(mode, width, layers):
    from bitexact_llm_b200.decode import Session
    eng = engine(mode, width, layers)
    ses = Session(eng, 40, 640, perm_seed=1)
    for seqs, lens, tiles, form in (([3], [1], False, True), ([0, 5], [40, 3], False, True), ([0, 5], [40, 3], False, False),
                                    (list(range(40)), [1] * 40, False, True), ([7, 2], [600, 9], True, True)):
        a, b = (step(eng, ses, seqs, lens, tiles, native, form) for native in (False, True))
        assert torch.equal(a[0], b[0]) and a[2] == b[2] and a[3] == b[3]
        assert all(torch.equal(u, v) for u, v in zip(a[1], b[1]))
    eng.check()


def test_what_the_loop_alone_serves():
    """A timer brackets single linears; a missing row map goes through the loop too."""
    from bitexact_llm_b200.decode import Session
    eng = engine("exact", 256, 2)
    ses = Session(eng, 2, 64)
    ids, pos, seq = torch.tensor([5, 9]).cuda(), torch.tensor([0, 0]).cuda(), torch.arange(2).cuda()
    args = (ses.kvs, ids, pos, ses._slots(seq, pos), ses.bt, seq)
    want = eng.forward(*args)
    seen = []
    for ly in eng.layers:
        ly["wo"].timer = lambda *a: (seen.append(a), contextlib.nullcontext())[1]
    assert torch.equal(eng.forward(*args), want) and len(seen) == 2
    for ly in eng.layers:
        ly["wo"].timer = None
    assert torch.equal(eng.forward(*args[:5], None), want)
    work = nv.lib().bx_forward_bytes(1, 2, 256, 4, 1, 64, 1024, 4, 16, 0)
    assert work > 0 and nv.lib().bx_forward_bytes(1, 0, 256, 4, 1, 64, 1024, 4, 16, 0) == 0
    assert nv.lib().bx_exact_forward(None, None, None) == nv.BX_EARG and nv.lib().bx_int8_forward(None, None, None) == nv.BX_EARG


@pytest.mark.parametrize("mode", ["exact", "int8"])
def test_the_feed_forward_width_is_that_of_the_weights(mode):
    """Constants whose config does not name it."""
    from bitexact_llm_b200.decode import Session

    def unnamed(c):
        del c["cfg"]["intermediate_size"]
        return c
    for n in (1, 600):
        got = []
        for edit in (unnamed, lambda c: c):
            eng = engine(mode, 256, 2, edit)
            assert mode == "exact" or eng.FF == 1024
            got.append(step(eng, Session(eng, 2, 640, perm_seed=1), [1], [n], n > 500, True))
        assert torch.equal(got[0][0], got[1][0]) and got[0][3] == got[1][3]


@pytest.mark.parametrize("layer", ["wqkv", "wo", "wgu", "wd"])
def test_linears_of_another_kind_are_called(layer):
    """A layer that is wrapped, or of a class of its own (exact mode); an engine's own _lin, of its class or its instance (int8 mode)."""
    from bitexact_llm_b200.decode import Session
    from bitexact_llm_b200.int8.engine import IntEngine
    from bitexact_llm_b200.vllm_plugin.exact_gemm import FusedLin
    seen = []

    class Counted(FusedLin):
        def __call__(self, *a, **k):
            seen.append(self)
            return super().__call__(*a, **k)

    class Own(IntEngine):
        def _lin(self, pre, lin):
            seen.append(lin)
            return super()._lin(pre, lin)

    def run(eng):
        return step(eng, Session(eng, 2, 64, perm_seed=1), [1], [3], False, True)
    eng = engine("exact", 256, 2)
    want, plain = run(eng), eng.layers[1][layer]
    eng.layers[1][layer] = lambda *a, **k: (seen.append(a), plain(*a, **k))[1]
    got = run(eng)
    assert len(seen) == 1 and torch.equal(got[0], want[0])
    eng.layers[1][layer] = plain
    plain.__class__ = Counted
    got = run(eng)
    assert len(seen) == 2 and torch.equal(got[0], want[0])
    plain.__class__ = FusedLin
    eng = engine("int8", 256, 2)
    want = run(eng)
    assert len(seen) == 2
    eng.__class__ = Own
    got = run(eng)
    assert len(seen) == 2 + 4 * eng.L and torch.equal(got[0], want[0])
    eng.__class__ = IntEngine
    eng._lin = lambda pre, lin: (seen.append(lin), IntEngine._lin(eng, pre, lin))[1]
    got = run(eng)
    assert len(seen) == 2 + 8 * eng.L and torch.equal(got[0], want[0])


def test_feed_of_device_tokens():
    """A server's sampled tokens stay on the device: no more waits than for tokens on the host, the same rows, lengths and caches,
    also beside entries on the host and portions cut by chunk_rows."""
    import warnings

    from bitexact_llm_b200.decode import Session
    eng, rng = engine("exact", 256, 2), torch.Generator().manual_seed(3)
    portions = [torch.randint(0, 512, (n,), generator=rng) for n in (1, 7, 1, 450, 1, 3)]

    def run(place, chunk_rows):
        ses = Session(eng, 6, 640, perm_seed=1)
        entries = [(s, t.cuda() if place == "device" or place == "mixed" and s % 2 else t) for s, t in enumerate(portions)]
        with warnings.catch_warnings(record=True) as waits:
            warnings.simplefilter("always")
            torch.cuda.set_sync_debug_mode("warn")
            try:
                rows = ses.feed(entries, chunk_rows)
            finally:
                torch.cuda.set_sync_debug_mode("default")
        return torch.cat(rows), ses.lens.clone(), torch.stack(ses.kvs), sum("synchroniz" in str(w.message) for w in waits)
    run("host", 4096)
    for chunk_rows in (4096, 100):
        want = run("host", chunk_rows)
        assert want[3] > 0
        for place in ("device", "mixed"):
            got = run(place, chunk_rows)
            assert all(torch.equal(a, b) for a, b in zip(want[:3], got[:3]))
            assert got[3] <= want[3]


@pytest.mark.parametrize("mode", ["exact", "int8"])
@pytest.mark.parametrize("B,keys", [(3, 3300), (48, 1000)])
def test_decoding_in_wide_tables(mode, B, keys):
    """The even split, whose scratch lies in the call's workspace, layer after layer over filled caches: few pairs and many."""
    from bitexact_llm_b200.decode import Session
    from bitexact_llm_b200.vllm_plugin import tri_paged
    eng = engine(mode, 1024, 3, n_pos=keys)
    ses = Session(eng, B, keys, perm_seed=1)
    assert nv.lib().bx_attention_plan(B, eng.HKV, ses.nblk, ses.bs, 2, 2 if mode == "exact" else 1) == 7
    g = torch.Generator(device="cuda").manual_seed(B)
    lens = torch.randint(0, keys, (B,), generator=g, device="cuda")
    lens[0] = keys - 1
    seq = torch.repeat_interleave(torch.arange(B, device="cuda"), lens)
    at = torch.arange(seq.shape[0], device="cuda") - torch.repeat_interleave(torch.cumsum(lens, 0) - lens, lens)
    bits = (17, 19) if mode == "exact" else (14, 14)
    for cache in ses.kvs:
        k, v = (torch.round(torch.randn(seq.shape[0], eng.HKV, 64, generator=g, device="cuda") * 2.0 ** b).long() for b in bits)
        tri_paged.store(cache, ses._slots(seq, at), k, v)
    ids, out = torch.arange(B, device="cuda") * 7 % 512, []
    for native in (False, True):
        kvs = [c.clone() for c in ses.kvs]
        with pytest.MonkeyPatch.context() as m:
            if not native:
                m.setattr(type(eng), "_forward_native", lambda *a: None)
            before = nv.lib().bx_launch_count()
            out.append((eng.forward(kvs, ids, lens, ses._slots(ses.rows, lens), ses.bt, ses.rows), nv.lib().bx_launch_count() - before, kvs))
    assert torch.equal(out[0][0], out[1][0]) and out[0][1] == out[1][1]
    assert all(torch.equal(a, b) for a, b in zip(out[0][2], out[1][2]))
    eng.check()


@pytest.mark.parametrize("mode,bound", [("exact", "wqkv"), ("exact", "wgu"), ("exact", "wd"), ("int8", "keys"), ("int8", "products")])
def test_a_bound_in_the_middle_layer_sets_the_flag(mode, bound):
    """Keys, values or products beyond their bounds in one layer of three; the product bound of int8 mode, which only the end of the
    call looks at, by itself. Without the edit there is no flag."""
    from bitexact_llm_b200.decode import Session
    from bitexact_llm_b200.vllm_plugin import tri_fuse
    eng = engine(mode, 256, 3)
    ses = Session(eng, 2, 64, perm_seed=1)
    run = lambda native: step(eng, ses, [0, 1], [3, 5], False, native)
    assert run(True)[2] == 0 and run(False)[2] == 0
    ly = eng.layers[1]
    if mode == "exact":
        ly[bound].g += 30
    elif bound == "keys":
        ly["ga"] <<= 12
    else:
        w, mul, fmsh = ly["wd"]
        ly["wd"], gamma = (w, mul, fmsh + 28), ly["gm"].clone()
        with pytest.MonkeyPatch.context() as m:                  # the maxima at 2^12 times the gamma, and the gamma for 2^62.5
            m.setattr(tri_fuse, "flag_end", lambda *a: None)
            ly["gm"] = gamma << 12
            assert run(False)[2] == 0
            s, u = eng.scr[1].tolist()
            ly["gm"] = gamma * int(2.0 ** 12 * (2.0 ** 62.5 / (s * u)) ** 0.5)
            eng.scr.zero_()
            assert run(False)[2] == 0                            # nothing else sets the flag
            s, u = eng.scr[1].tolist()
            assert 1 << 62 <= s * u < 1 << 63
            eng.scr.zero_()
    loop, native = run(False), run(True)
    assert loop[2] == native[2] == 1 and torch.equal(loop[0], native[0])
