"""All layers from one call of the library: the residual rows, caches and flag of the engines' own loop over single calls, for decoding
rows and prompt tiles, with and without what an engine may lack, and what that loop alone serves."""

import contextlib

import pytest
import torch

from bitexact_llm_b200 import _native as nv

pytestmark = pytest.mark.gpu


def engine(mode, width, layers, edit=lambda c: c):
    from bitexact_llm_b200.exact import consts
    cfg = dict(consts.LLAMA_1B, hidden_size=width, intermediate_size=4 * width, num_hidden_layers=layers, num_attention_heads=width // 64,
               num_key_value_heads=width // 256, head_dim=64, vocab_size=512)
    sd = consts.random_state_dict(cfg, seed=width, device="cuda", gamma_jitter=0.1)
    if mode == "exact":
        from bitexact_llm_b200.vllm_plugin.exact_run import ExactEngine
        return ExactEngine(edit(consts.build(cfg, sd, n_pos=700)), "cuda")
    from bitexact_llm_b200.int8 import consts as consts8
    from bitexact_llm_b200.int8.engine import IntEngine
    return IntEngine(edit(consts8.build(cfg, sd, n_pos=700)), "cuda")


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
