"""The work that users of this package have it do, as cases to be timed: decoding, prompts, mixed serving steps and scoring on
the integer engines (exact and int8 mode), decoding and prompts on the hybrid float models.

A case is a dict of plain values. `model`: exact | int8 (a Llama of `width` and `layers`) or fedatar | veredra (float models,
`dtype` bfloat16 or float32); `task`:

  decode  one step of a batch of `batch` sequences with `lo` .. `hi` keys before it: forward, head, sampler, replayed from a CUDA
          graph with the tokens copied in from pinned host memory
  prompt  `batch` new prompts of `lo` .. `hi` tokens through `Session.prefill` (integer engines, and the first tokens sampled) or
          `Session.feed` (float models, logits of every prompt's end)
  mixed   a step of a server with chunked prompts: `batch` running sequences decode a token each while `portion` tokens of a
          prompt are fed
  score   log p of the tokens of `rows` residual rows: head, then the integer log-softmax (integer engines)

Sizes within lo .. hi are spread evenly and deterministically, so that a case's work does not depend on the seed; weights,
tokens, caches and sampler seeds come from the seed. Widths and depths are those of the benchmarks (1024 and 2048 with 16 layers,
4096 with 4; the float models here with the 2 or 4 layers that hold each of their mechanisms), the vocabulary is 128256 throughout."""

import math

import torch

VOCAB = 128256
DEV = "cuda"
FR = {"exact": 24, "int8": 16}
KEY_BYTES = 384                     # three limbs of a key and of a value of 64 entries


def listed():
    return [
        # One user at a chat prompt's length: every kernel is latency.
        dict(name="exact-decode-1", model="exact", task="decode", width=2048, layers=16, batch=1, lo=512, hi=512),
        # A small server with sequences of any length.
        dict(name="exact-decode-19", model="exact", task="decode", width=2048, layers=16, batch=19, lo=16, hi=1100),
        # The throughput benchmark: 256 sequences, 512-token prompts, up to 256 tokens generated.
        dict(name="exact-decode-256", model="exact", task="decode", width=2048, layers=16, batch=256, lo=512, hi=768),
        # Long documents: contexts of 64 .. 8192 keys.
        dict(name="exact-decode-32-long", model="exact", task="decode", width=2048, layers=16, batch=32, lo=64, hi=8192),
        # A short question.
        dict(name="exact-prompt-17", model="exact", task="prompt", width=2048, layers=16, batch=1, lo=17, hi=17),
        # A batch of long prompts.
        dict(name="exact-prompt-4x2048", model="exact", task="prompt", width=2048, layers=16, batch=4, lo=1700, hi=2048),
        # Chunked prompts beside running sequences.
        dict(name="exact-mixed-48", model="exact", task="mixed", width=2048, layers=16, batch=48, lo=100, hi=1500, portion=700),
        # int8 mode: the mode for throughput, mixed prompt lengths up to 4096.
        dict(name="int8-decode-64", model="int8", task="decode", width=2048, layers=16, batch=64, lo=16, hi=4096),
        dict(name="int8-prompt-5", model="int8", task="prompt", width=2048, layers=16, batch=5, lo=16, hi=3000),
        # Reinforcement learning: log p of given tokens.
        dict(name="exact-score-700", model="exact", task="score", width=2048, layers=1, rows=700),
        # The float models: prompts of one, decoding of the other.
        dict(name="fedatar-prompt-3", model="fedatar", task="prompt", width=2048, layers=2, batch=3, lo=300, hi=1500,
             dtype="bfloat16"),
        dict(name="veredra-decode-64", model="veredra", task="decode", width=2048, layers=4, batch=64, lo=200, hi=200,
             dtype="bfloat16"),
    ]


def draw(rng):
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def span(lo, hi):
        a, b = log(lo, hi), log(lo, hi)
        return dict(lo=min(a, b), hi=max(a, b))
    kind = rng.choice(["decode"] * 4 + ["prompt"] * 3 + ["mixed"] + ["score"] + ["float"] * 3)
    if kind == "float":
        c = dict(model=rng.choice(["fedatar", "veredra"]), width=rng.choice([1024, 2048]),
                 dtype=rng.choice(["bfloat16", "bfloat16", "bfloat16", "float32"]))
        c["layers"] = 2 if c["model"] == "fedatar" else 4
        wide = c["dtype"] == "bfloat16"
        if rng.random() < 0.5:
            n = log(16, 400)
            return dict(c, task="decode", batch=log(1, 96 if wide else 16), lo=n, hi=n)
        return dict(c, task="prompt", batch=rng.randint(1, 4), **span(8, 1600 if wide else 300))
    c = dict(model=rng.choice(["exact", "exact", "int8"]))
    c["width"], c["layers"] = rng.choice([(2048, 16), (2048, 16), (1024, 16), (4096, 4)])
    if kind == "score":
        return dict(c, task="score", layers=1, rows=log(1, 1000))
    if kind == "prompt":
        return dict(c, task="prompt", batch=rng.randint(1, 4), **span(5, 2000))
    if kind == "mixed":
        return dict(c, task="mixed", batch=log(1, 100), portion=log(10, 1500), **span(16, 1500))
    batch = log(1, 256)
    return dict(c, task="decode", batch=batch, **span(16, min(8192, 180000 // batch)))


def sizes(case):
    """The contexts or prompt lengths of a case's sequences: lo .. hi in steps of the golden ratio, hi first."""
    lo, hi = case["lo"], case["hi"]
    return [hi - int((hi - lo) * ((0.6180339887498949 * i) % 1.0)) for i in range(case["batch"])]


# ---- models -------------------------------------------------------------------------------------------------------

def llama_config(case):
    from bitexact_llm_b200.exact import consts
    w = case["width"]
    return dict(consts.LLAMA_1B, hidden_size=w, intermediate_size=min(4 * w, 14336), num_hidden_layers=case["layers"],
                num_attention_heads=w // 64, num_key_value_heads=w // 256, head_dim=64)


def llama_engine(case, seed, n_pos):
    from bitexact_llm_b200.exact import consts
    cfg = llama_config(case)
    sd = consts.random_state_dict(cfg, seed=seed, device=DEV, gamma_jitter=0.1)
    if case["model"] == "exact":
        from bitexact_llm_b200.vllm_plugin.exact_run import ExactEngine
        return ExactEngine(consts.build(cfg, sd, n_pos=n_pos), DEV)
    from bitexact_llm_b200.int8 import consts as consts8
    from bitexact_llm_b200.int8.engine import IntEngine
    return IntEngine(consts8.build(cfg, sd, n_pos=n_pos), DEV)


def fedatar_config(width, layers):
    """minGRU and latent-attention layers in turn; a dense feed-forward first, then 8 experts (two per token) and a shared one."""
    out = []
    for i in range(layers):
        attention = {"heads": width // 64, "dim": 64, "rot_dim": 32, "vdim": 64, "q_rank": 3 * width // 8, "kv_rank": 256,
                     "rot": {"base": 1e6, "dims": 32}, "scale": 96 ** -0.5, "mask": {"size": 1024}}
        kind, m = ("latent_attention", attention) if i % 2 else ("mingru", {"width": width})
        ff = {"kind": "moe", "router": {"experts": 8, "top": 2}, "expert": {"ff": 2 * width}, "shared": {"ff": 2 * width}}
        out.append({"type": kind, "mixer": m, "mlp": ff if i else {"kind": "dense", "ff": 6 * width}})
    return {"architecture": "Fedatar", "vocab": VOCAB, "width": width, "norm": {"eps": 1e-6}, "layers": out}


def veredra_config(width, layers):
    """Gated linear attention, attention and Mamba-2 in turn, two streams, a gated feed-forward of 4 x width."""
    kinds = [("gla", {"heads": width // 256, "dim": 128, "vdim": 256, "tau": 16.0}),
             ("attention", {"heads": width // 128, "kv_heads": width // 512, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                            "rot": {"base": 1e6, "dims": 128}, "mask": {"size": 1024}}),
             ("mamba2", {"heads": width // 32, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8})]
    out = [{"type": kinds[i % 3][0], "mixer": kinds[i % 3][1], "mlp": {"kind": "dense", "ff": 4 * width}} for i in range(layers)]
    return {"architecture": "Veredra", "vocab": VOCAB, "width": width, "streams": 2, "norm": {"eps": 1e-6}, "logit_scale": 1.0,
            "logit_softcap": 30.0, "loop": None, "layers": out}


def matrix_shapes(cfg):
    """(name, rows, columns) of every weight matrix of a float model."""
    D, out = cfg["width"], [("embed", cfg["vocab"], cfg["width"]), ("head", cfg["vocab"], cfg["width"])]
    for i, ly in enumerate(cfg["layers"]):
        p, m, f = f"l{i}.mix.", ly["mixer"], ly["mlp"]
        kind = ly["type"]
        if kind == "mingru":
            out += [(p + n, m["width"], D) for n in "zxg"] + [(p + "o", D, m["width"])]
        elif kind == "latent_attention":
            H, R, qr = m["heads"], m["kv_rank"], m["q_rank"]
            out += [(p + "dq", qr, D), (p + "uq", H * (m["dim"] + m["rot_dim"]), qr), (p + "dkv", R + m["rot_dim"], D),
                    (p + "uk", H * m["dim"], R), (p + "uv", H * m["vdim"], R), (p + "g", H, D), (p + "o", D, H * m["vdim"])]
        elif kind == "attention":
            H, G = m["heads"], m["kv_heads"]
            out += [(p + "q", H * m["dim"], D), (p + "k", G * m["dim"], D), (p + "v", G * m["vdim"], D), (p + "o", D, H * m["vdim"])]
        elif kind == "gla":
            nk, nv = m["heads"] * m["dim"], m["heads"] * m["vdim"]
            out += [(p + "q", nk, D), (p + "k", nk, D), (p + "v", nv, D), (p + "g", nv, D), (p + "a1", 16, D), (p + "a2", nk, 16),
                    (p + "o", D, nv)]
        else:
            inner, bc = m["heads"] * m["vdim"], 2 * m["groups"] * m["state"]
            out += [(p + "in", 2 * inner + bc + m["heads"], D), (p + "conv", inner + bc, m["conv"]), (p + "o", D, inner)]
        p = f"l{i}.mlp."
        if cfg["architecture"] == "Veredra":
            out += [(p + "gate", f["ff"], D), (p + "up", f["ff"], D), (p + "down", D, f["ff"])]
        elif f["kind"] == "dense":
            out += [(p + "up", f["ff"], D), (p + "down", D, f["ff"])]
        else:
            for n, ff in [(f"e{e}", f["expert"]["ff"]) for e in range(f["router"]["experts"])] + [("shared", f["shared"]["ff"])]:
                out += [(p + n + ".up", ff, D), (p + n + ".down", D, ff)]
            out += [(p + "router", f["router"]["experts"], D)]
    return out


def float_weights(cfg, seed):
    """bf16 tensors under the designs' names."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    normal = lambda *n: torch.randn(*n, generator=g, device=DEV)
    t = {n: (normal(r, k) * k ** -0.5).to(torch.bfloat16) for n, r, k in matrix_shapes(cfg)}
    D = cfg["width"]

    def vec(name, n, mean=0.0):
        t[name] = (mean + 0.1 * normal(n)).to(torch.bfloat16)
    if cfg["architecture"] == "Fedatar":
        vec("final.norm", D, 1.0)
        vec("final.norm.b", D)
    else:
        vec("final.norm", D)
    for i, ly in enumerate(cfg["layers"]):
        p, m, f, kind = f"l{i}.", ly["mixer"], ly["mlp"], ly["type"]
        for q in (1, 2):
            if cfg["architecture"] == "Fedatar":
                vec(f"{p}norm{q}", D, 1.0)
                vec(f"{p}norm{q}.b", D)
            else:
                S = cfg["streams"]
                vec(f"{p}norm{q}", D)
                vec(f"{p}hc{q}.in", S, 1.0 / S)
                vec(f"{p}hc{q}.out", S, 0.7)
                t[f"{p}hc{q}.mix"] = torch.eye(S, device=DEV).to(torch.bfloat16)
        if f["kind"] == "moe":
            vec(p + "mlp.router.b", f["router"]["experts"])
        elif cfg["architecture"] == "Fedatar":
            vec(p + "mlp.act", 2)
        p += "mix."
        if kind == "mingru":
            vec(p + "z.b", m["width"], -1.0)
            vec(p + "x.b", m["width"])
        elif kind == "latent_attention":
            vec(p + "dq.norm", m["q_rank"], 1.0)
            vec(p + "dkv.norm", m["kv_rank"], 1.0)
            vec(p + "sink", m["heads"])
        elif kind == "attention":
            for n, rows in (("q", m["heads"] * m["dim"]), ("k", m["kv_heads"] * m["dim"]), ("v", m["kv_heads"] * m["vdim"])):
                vec(f"{p}{n}.b", rows)
                if n != "v":
                    vec(f"{p}{n}.norm", rows, 1.0)
            vec(p + "sink", m["heads"])
        elif kind == "gla":
            vec(p + "a2.b", m["heads"] * m["dim"], 2.0)
            vec(p + "norm", m["vdim"], 1.0)
        else:
            inner = m["heads"] * m["vdim"]
            for n, size, mean in (("conv.b", inner + 2 * m["groups"] * m["state"], 0.0), ("dt_bias", m["heads"], -3.0),
                                  ("A_log", m["heads"], 0.0), ("D", m["heads"], 1.0), ("norm", inner, 1.0)):
                vec(p + n, size, mean)
    return t


def float_config(case):
    return (fedatar_config if case["model"] == "fedatar" else veredra_config)(case["width"], case["layers"])


def float_engine(case, seed):
    from bitexact_llm_b200.hybrid import fedatar, veredra
    cfg = float_config(case)
    return (fedatar if case["model"] == "fedatar" else veredra).load(cfg, float_weights(cfg, seed), DEV, case["dtype"])


# ---- states -------------------------------------------------------------------------------------------------------

def tokens(case, seed, batch, n):
    return torch.randint(0, VOCAB, (batch, n), generator=torch.Generator().manual_seed(seed))


def fill_cache(case, ses, lens, seed):
    """Keys and values of the first lens[b] positions of every sequence, N(0, 1), different in every layer."""
    from bitexact_llm_b200.vllm_plugin import tri_paged
    g = torch.Generator(device=DEV).manual_seed(seed)
    n = torch.tensor(lens, device=DEV)
    seq = torch.repeat_interleave(torch.arange(len(lens), device=DEV), n)
    pos = torch.arange(seq.shape[0], device=DEV) - torch.repeat_interleave(torch.cumsum(n, 0) - n, n)
    slot = ses.bt[seq, pos // ses.bs].long() * ses.bs + pos % ses.bs
    kb, vb = (17, 19) if case["model"] == "exact" else (14, 14)       # fractional bits of cached keys and values
    for cache in ses.kvs:
        k, v = (torch.round(torch.randn(seq.shape[0], ses.eng.HKV, ses.eng.HD, generator=g, device=DEV) * 2.0 ** b).long()
                for b in (kb, vb))
        tri_paged.store(cache, slot, k, v)
    ses.lens.copy_(n)


def leaves(caches):
    return [t for c in caches for t in (c if isinstance(c, tuple) else (c,))]


def capture(body, keep=()):
    """body() as a CUDA graph, and what it returned; the tensors `keep` are put back as they were before the warm-up."""
    saved = [t.clone() for t in keep]
    for _ in range(2):
        body()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = body()
    for t, s in zip(keep, saved):
        t.copy_(s)
    return graph, out


def sampler_rows(batch, seed):
    """(seed, generated index, temperature 7 / 10) of every sequence."""
    rows = torch.zeros(batch, 4, dtype=torch.long)
    rows[:, 0], rows[:, 1], rows[:, 2], rows[:, 3] = seed + torch.arange(batch), 3, 7, 10
    return rows.to(DEV)


@torch.no_grad()
def prepare(case, seed):
    from bitexact_llm_b200.decode import Session
    from bitexact_llm_b200.vllm_plugin import sampler
    s = {"case": case}
    integer = case["model"] in FR
    if case["task"] == "score":
        s["eng"] = eng = llama_engine(case, seed, 64)
        g = torch.Generator(device=DEV).manual_seed(seed + 1)
        s["rows"] = torch.round(torch.randn(case["rows"], case["width"], generator=g, device=DEV) * 2.0 ** eng.FR).long()
        s["tokens"] = torch.randint(0, VOCAB, (case["rows"],), generator=g, device=DEV)
        return s
    lens = sizes(case)
    B, longest = len(lens), max(lens)
    s["lens"] = torch.tensor(lens)
    if case["task"] == "prompt":
        s["eng"] = eng = llama_engine(case, seed, longest + 1) if integer else float_engine(case, seed)
        s["ses"] = Session(eng, B, longest + 1, perm_seed=seed)
        s["prompts"] = tokens(case, seed, B, longest)
        s["sampler"] = sampler_rows(B, seed)
        return s
    if case["task"] == "mixed":
        n = case["portion"]
        s["eng"] = eng = llama_engine(case, seed, max(longest, n) + 1)
        s["ses"] = ses = Session(eng, B + 1, max(longest, n) + 1, perm_seed=seed)
        fill_cache(case, ses, lens + [0], seed)
        new = tokens(case, seed, 1, B + n)[0]
        s["entries"] = [(b, new[b:b + 1]) for b in range(B)] + [(B, new[B:])]
        s["start"] = ses.lens.clone()
        s["sampler"] = sampler_rows(B + 1, seed)
        return s
    s["eng"] = eng = llama_engine(case, seed, longest + 1) if integer else float_engine(case, seed)
    s["ses"] = ses = Session(eng, B, longest + 1, perm_seed=seed)
    if integer:
        fill_cache(case, ses, lens, seed)
    else:
        ses.prefill(tokens(case, seed, B, longest))
    s["sampler"] = rows = sampler_rows(B, seed)
    s["host"] = tokens(case, seed + 1, B, 1)[:, 0].pin_memory()
    s["in"] = tok = s["host"].to(DEV)
    s["pos"] = pos = ses.lens.clone()                   # the graph reads it: it lives as long as the state

    def step():
        x = ses.step(tok, pos)
        if not integer:
            return x, eng.logits_float(x)
        lg = eng.logits(x)
        return lg, sampler.sample_rows(lg, rows, eng.ln, eng.FR)
    s["graph"], s["out"] = capture(step, [ses.lens] + (leaves(ses.kvs) if not integer else []))
    return s


@torch.no_grad()
def run(s):
    from bitexact_llm_b200.vllm_plugin import rl, sampler
    case, eng = s["case"], s["eng"]
    if case["task"] == "decode":
        s["in"].copy_(s["host"], non_blocking=True)
        s["graph"].replay()
        return s["out"]
    if case["task"] == "score":
        lg = eng.logits(s["rows"])
        return lg, rl.int_logp_q(lg, s["tokens"], eng.ln, eng.FR)
    ses = s["ses"]
    if case["task"] == "mixed":
        ses.lens.copy_(s["start"])
        rows = ses.feed(s["entries"])
        lg = eng.logits(torch.cat([r[-1:] for r in rows]))
        return torch.cat(rows), lg, sampler.sample_rows(lg, s["sampler"], eng.ln, eng.FR)
    ses.lens.zero_()
    if case["model"] in FR:
        h = ses.prefill(s["prompts"], s["lens"])
        lg = eng.logits(h)
        return h, lg, sampler.sample_rows(lg, s["sampler"], eng.ln, eng.FR)
    rows = ses.feed([(b, p[:n]) for b, (p, n) in enumerate(zip(s["prompts"], s["lens"].tolist()))])
    return torch.cat(rows), eng.logits_float(torch.cat([r[-1:] for r in rows]))


# ---- work and accuracy --------------------------------------------------------------------------------------------

def work(case):
    """Weights once (those of a step's experts in expectation), every key and value that is seen, states in and out, outputs;
    operations of the products and of attention."""
    D, V, L = case["width"], VOCAB, case["layers"]
    task = case["task"]
    lens = [] if task == "score" else sizes(case)
    if task == "decode":
        rows, heads, keys, fresh = len(lens), len(lens), sum(n + 1 for n in lens), len(lens)
    elif task == "prompt":
        rows, heads, keys, fresh = sum(lens), len(lens), sum(lens), sum(lens)
    elif task == "mixed":
        n = case["portion"]
        rows, heads, keys, fresh = len(lens) + n, len(lens) + 1, sum(k + 1 for k in lens) + n, len(lens) + n
    else:
        rows, heads, keys, fresh = 0, case["rows"], 0, 0
    seen = sum(n + 1 for n in lens) if task != "prompt" else sum(n * (n + 1) // 2 for n in lens)    # (query row, key) pairs
    if task == "mixed":
        seen += case["portion"] * (case["portion"] + 1) // 2
    if case["model"] in FR:
        planes, products = (3, 9) if case["model"] == "exact" else (1, 2)       # bytes per weight, int8 products per pair
        cfg = llama_config(case)
        H, G, ff = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["intermediate_size"]
        per_layer = D * (2 * H * 64 + 2 * G * 64 + 3 * ff) if task != "score" else 0
        moved = planes * (L * per_layer + V * D) + L * G * KEY_BYTES * (keys + fresh) + 8 * V * heads + 4 * D * rows
        return {"bytes": moved, "flops": 2 * products * (rows * L * per_layer + heads * V * D) + 2 * 2 * 9 * 64 * H * L * seen}
    cfg = float_config(case)
    size = 2 if case["dtype"] == "bfloat16" else 4
    moved, ops = size * V * D + 4 * V * heads + (size + 4) * D * rows, 2 * heads * V * D
    for name, n, k in matrix_shapes(cfg):
        if name in ("embed", "head"):
            continue
        part = name.split(".")
        routed = part[1] == "mlp" and part[2][0] == "e" and part[2][1:].isdigit()
        used = 1 - (1 - 2 / 8) ** rows if routed else 1.0           # an expert's weights, when a row chose it
        moved += size * n * k * used
        ops += 2 * n * k * rows * (0.25 if routed else 1.0)
    for ly in cfg["layers"]:
        m = ly["mixer"]
        if ly["type"] in ("mingru", "gla", "mamba2"):
            state = m["width"] if ly["type"] == "mingru" else m["heads"] * m["vdim"] * (m["dim"] if ly["type"] == "gla" else m["state"])
            moved += 4 * state * len(lens) * (2 if task == "decode" else 1)
            ops += 4 * state * rows
        else:
            row = m["kv_rank"] + m["rot_dim"] if ly["type"] == "latent_attention" else m["kv_heads"] * (m["dim"] + m["vdim"])
            window = m["mask"]["size"]
            moved += size * row * (sum(min(n + 1, window) for n in lens) if task == "decode" else rows)
            entries = m["dim"] + m["vdim"] + m.get("rot_dim", 0)
            ops += 2 * m["heads"] * entries * sum(min(n + 1, window) if task == "decode" else n * (n + 1) // 2 - max(0, n - window) * (n - window + 1) // 2
                                                  for n in lens)
    return {"bytes": moved, "flops": ops}


def tolerance(case):
    """The integer engines are bit-exact by definition. The float models: see the comments."""
    if case["model"] in FR:
        return "exact"
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 2e-3}
    # Activations are rounded to bf16 between the kernels; a row whose second and third expert are nearly tied may take the other.
    return {"rel": 0.03, "max": 0.99}


# The float models in 64 bits, whole sequences at once ([sequence, token, entry]), padded behind their ends.

def sigmoid(v):
    return torch.sigmoid(v)


def silu(v):
    return v * torch.sigmoid(v)


def softplus(v):
    return v.clamp(min=0) + torch.log1p(torch.exp(-v.abs()))


def rms(v, w, eps):
    return v / torch.sqrt((v * v).mean(-1, keepdim=True) + eps) * w


def layer_norm(v, w, b, eps):
    c = v - v.mean(-1, keepdim=True)
    return c / torch.sqrt((c * c).mean(-1, keepdim=True) + eps) * w + b


def turn(v, base, dims, halves):
    """Rotates the first `dims` entries of v [.., T, heads, n] by position: pairs (i, i + dims / 2) or (2 i, 2 i + 1)."""
    T, half = v.shape[1], dims // 2
    ang = torch.arange(T, dtype=torch.float64, device=DEV)[:, None] * base ** (-2.0 * torch.arange(half, dtype=torch.float64, device=DEV) / dims)
    c, s = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
    a, b = (v[..., :half], v[..., half:dims]) if halves else (v[..., 0:dims:2], v[..., 1:dims:2])
    r = torch.stack([a * c - b * s, b * c + a * s], -2 if halves else -1).reshape(*v.shape[:-1], dims)
    return torch.cat([r, v[..., dims:]], -1)


def attend(q, k, v, scale, window, sink):
    """q, k [S, T, H, n], v [S, T, H, m]; exp(sink[h]) is added to every denominator."""
    T = q.shape[1]
    d = torch.arange(T, device=DEV)[:, None] - torch.arange(T, device=DEV)[None, :]
    hidden = (d < 0) | ((d >= window) if window else torch.zeros_like(d, dtype=torch.bool))
    out = torch.empty(*q.shape[:3], v.shape[3], dtype=torch.float64, device=DEV)
    for i in range(q.shape[0]):
        z = torch.einsum("ihd,jhd->hij", q[i], k[i]) * scale
        z.masked_fill_(hidden, -math.inf)
        top = torch.maximum(z.amax(-1, keepdim=True), sink[:, None, None])
        e = torch.exp(z - top)
        e /= e.sum(-1, keepdim=True) + torch.exp(sink[:, None, None] - top)
        out[i] = torch.einsum("hij,jhd->ihd", e, v[i])
    return out


def recur(q, k, v, decay):
    """S = decay S + k v^T, o = S^T q over the tokens; q, k, decay [S, T, H, n], v [S, T, H, m]."""
    S = torch.zeros(*k[:, 0].shape, v.shape[3], dtype=torch.float64, device=DEV)
    o = torch.empty_like(v)
    for t in range(k.shape[1]):
        S = decay[:, t, :, :, None] * S + k[:, t, :, :, None] * v[:, t, :, None, :]
        o[:, t] = torch.einsum("bhnm,bhn->bhm", S, q[:, t])
    return o


def mix64(kind, h, w, m, eps):
    S, T = h.shape[:2]
    H = m.get("heads")
    if kind == "mingru":
        z, u = sigmoid(h @ w["z"].T + w["z.b"]), h @ w["x"].T + w["x.b"]
        cand = torch.where(u >= 0, u + 0.5, sigmoid(u))
        s, out = torch.zeros_like(z[:, 0]), torch.empty_like(z)
        for t in range(T):
            s = (1 - z[:, t]) * s + z[:, t] * cand[:, t]
            out[:, t] = s
        return (out * silu(h @ w["g"].T)) @ w["o"].T
    if kind == "latent_attention":
        dn, dr, R, base = m["dim"], m["rot_dim"], m["kv_rank"], m["rot"]["base"]
        q = (rms(h @ w["dq"].T, w["dq.norm"], eps) @ w["uq"].T).reshape(S, T, H, dn + dr)
        q = torch.cat([q[..., :dn], turn(q[..., dn:], base, dr, False)], -1)
        kv = h @ w["dkv"].T
        c = rms(kv[..., :R], w["dkv.norm"], eps)
        kr = turn(kv[..., None, R:], base, dr, False).expand(-1, -1, H, -1)
        k = torch.cat([(c @ w["uk"].T).reshape(S, T, H, dn), kr], -1)
        o = attend(q, k, (c @ w["uv"].T).reshape(S, T, H, m["vdim"]), m["scale"], m["mask"]["size"], w["sink"])
        return (o * sigmoid(h @ w["g"].T)[..., None]).reshape(S, T, -1) @ w["o"].T
    if kind == "attention":
        G, dk, rot = m["kv_heads"], m["dim"], m["rot"]
        q = rms(h @ w["q"].T + w["q.b"], w["q.norm"], eps).reshape(S, T, H, dk)
        k = rms(h @ w["k"].T + w["k.b"], w["k.norm"], eps).reshape(S, T, G, dk)
        v = (h @ w["v"].T + w["v.b"]).reshape(S, T, G, m["vdim"])
        q, k = turn(q, rot["base"], rot["dims"], True), turn(k, rot["base"], rot["dims"], True)
        k, v = k.repeat_interleave(H // G, 2), v.repeat_interleave(H // G, 2)
        return attend(q, k, v, m["scale"], m["mask"]["size"], w["sink"]).reshape(S, T, -1) @ w["o"].T
    if kind == "gla":
        n, p = m["dim"], m["vdim"]
        q, k = ((h @ w[x].T).reshape(S, T, H, n) for x in "qk")
        decay = torch.exp(-softplus(-((h @ w["a1"].T) @ w["a2"].T + w["a2.b"])) / m["tau"]).reshape(S, T, H, n)
        o = recur(q * n ** -0.5, k, (h @ w["v"].T).reshape(S, T, H, p), decay)
        return (rms(o, w["norm"], eps).reshape(S, T, -1) * silu(h @ w["g"].T)) @ w["o"].T
    P, N, G = m["vdim"], m["state"], m["groups"]
    inner = H * P
    u = h @ w["in"].T
    z, x, dt = u[..., :inner], u[..., inner:2 * inner + 2 * G * N], softplus(u[..., 2 * inner + 2 * G * N:] + w["dt_bias"])
    pad = torch.cat([torch.zeros(S, m["conv"] - 1, x.shape[2], dtype=torch.float64, device=DEV), x], 1)
    x = silu(w["conv.b"] + sum(pad[:, j:j + T] * w["conv"][:, j] for j in range(m["conv"])))
    v = x[..., :inner].reshape(S, T, H, P)
    b, c = (x[..., inner + i * G * N:inner + (i + 1) * G * N].reshape(S, T, G, N).repeat_interleave(H // G, 2) for i in (0, 1))
    decay = torch.exp(-torch.exp(w["A_log"]) * dt)[..., None].expand(-1, -1, -1, N)
    y = recur(c, b * dt[..., None], v, decay) + w["D"][:, None] * v
    y = (y.reshape(S, T, inner) * silu(z)).reshape(S, T, m["norm_groups"], -1)
    return (rms(y, 1.0, eps).reshape(S, T, inner) * w["norm"]) @ w["o"].T


def ff64(f, gated, h, w):
    if gated:
        z = h @ w["gate"].T
        return (0.5 * z * (1 + torch.tanh(math.sqrt(2 / math.pi) * (z + 0.044715 * z ** 3))) * (h @ w["up"].T)) @ w["down"].T
    if f["kind"] == "dense":
        z, (a, b) = h @ w["up"].T, softplus(w["act"])
        neg = z.clamp(max=0)
        return (torch.where(z > 0, a * z * z, (0.5 + b) * (torch.expm1(neg) - neg)) + 0.5 * z) @ w["down"].T
    z = h @ w["router"].T + w["router.b"]
    top, idx = torch.sort(z, dim=-1, descending=True, stable=True)
    top, idx = torch.softmax(top[..., :f["router"]["top"]], -1), idx[..., :f["router"]["top"]]
    expert = lambda n, r: ((r @ w[n + ".up"].T).clamp(min=0) ** 2) @ w[n + ".down"].T
    out = expert("shared", h)
    for e in range(f["router"]["experts"]):
        at = (idx == e).any(-1)
        out[at] += (top * (idx == e)).sum(-1)[at][:, None] * expert(f"e{e}", h[at])
    return out


@torch.no_grad()
def exact(case, seed):
    """The float models' residual rows and logits in 64 bits. The integer engines' outputs are whole numbers."""
    if case["model"] in FR:
        return None
    lens = sizes(case)
    B, n = len(lens), max(lens)
    ids = tokens(case, seed, B, n)
    if case["task"] == "decode":
        ids = torch.cat([ids, tokens(case, seed + 1, B, 1)], 1)
    cfg = float_config(case)
    names = list(float_weights(cfg, seed).items())
    w = dict(names)
    under = lambda p: {k[len(p):]: v.double() for k, v in w.items() if k.startswith(p)}
    eps, streams = cfg["norm"]["eps"], cfg.get("streams")
    x = w["embed"][ids.to(DEV)].double()
    if streams:
        x = torch.stack([x] * streams)
    for i, ly in enumerate(cfg["layers"]):
        for q, part in ((1, "mix."), (2, "mlp.")):
            hc, norm = under(f"l{i}.hc{q}."), under(f"l{i}.norm{q}")
            if streams:
                h = rms(torch.einsum("s,sbtd->btd", hc["in"], x), 1 + norm[""], eps)
            else:
                h = layer_norm(x, norm[""], norm[".b"], eps)
            sub = under(f"l{i}.{part}")
            y = mix64(ly["type"], h, sub, ly["mixer"], eps) if q == 1 else ff64(ly["mlp"], bool(streams), h, sub)
            x = torch.einsum("st,sbnd->tbnd", hc["mix"], x) + hc["out"][:, None, None, None] * y if streams else x + y
    x = x.sum(0) if streams else x
    rows = x[:, -1] if case["task"] == "decode" else torch.cat([x[b, :k] for b, k in enumerate(lens)])
    last = rows if case["task"] == "decode" else torch.stack([x[b, k - 1] for b, k in enumerate(lens)])
    final = under("final.norm")
    if streams:
        z = rms(last, 1 + final[""], eps) @ w["head"].double().T * cfg["logit_scale"]
        return rows, cfg["logit_softcap"] * torch.tanh(z / cfg["logit_softcap"])
    # In bf16 a near tie sends a row to another expert than in 64 bits, so a handful of rows has no 64-bit value to be held to.
    if case["dtype"] == "bfloat16":
        return rows, None
    return rows, layer_norm(last, final[""], final[".b"], eps) @ w["head"].double().T
