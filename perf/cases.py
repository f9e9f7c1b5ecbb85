"""What this framework is measured on: steps of its engine as a program that serves or scores text makes them.

A case is a model, what its step brings (one token a sequence, whole prompts, the next turn of a conversation) and how
many sequences of which lengths take part.  Models have random weights and the sizes of this repository's presets and
benchmarks: the Qwen3-0.6B shape whole, the Qwen3-8B shape with its layers cut to twelve of 36 (a state has to fit the
card three times over; embedding and output head are whole), and Vabelorn and Lunadra at width 2,048 with four layers.
Everything runs through ``Engine``: ``alloc_slot``, ``step``, ``sample``, ``free_slot``; a decode step is taken back
with ``cache.truncate`` so that it can be made again.

Routed experts have no case: two correct 16-bit implementations choose different experts where two scores nearly tie,
and the logits of such a token differ by more than rounding.
"""
import math
import random

import torch

import pytorch_engine_b200 as pe

DEVICE = "cuda:0"
PREFILL_TOKENS = 16384      # prompt tokens a step of ``prepare`` brings at most
EXACT_FLOPS = 2.0e14        # above this a 64-bit run takes too long

QWEN3 = {
    "qwen3_0_6b": dict(hidden=1024, heads=16, kv_heads=8, dim=128, ff=3072, layers=28, vocab=151936, tied=True),
    "qwen3_8b": dict(hidden=4096, heads=32, kv_heads=8, dim=128, ff=12288, layers=12, vocab=151936, tied=False),
}
THETA, EPS = 1e6, 1e-6
# width 2,048, 16 heads of 128 over 4 key heads, feed-forward 6,144, vocabulary 32,768: the small size of bench.py --archs
WIDTH, HEADS, KV_HEADS, DIM, FF, VOCAB, LAYERS = 2048, 16, 4, 128, 6144, 32768, 4
YARN = {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}


# ---- the cases -----------------------------------------------------------------------------------------------------
def listed():
    return [
        # one user's chat on the small model: the smallest step there is, all launches and latency
        dict(name="decode 0.6B x 1", task="decode", model="qwen3_0_6b", dtype="bfloat16", seqs=1, shortest=300, longest=300),
        # a small server of the small model: more sequences than the few-row kernels take, lengths that do not line up
        dict(name="decode 0.6B x 24", task="decode", model="qwen3_0_6b", dtype="bfloat16", seqs=24, shortest=16, longest=2048),
        # the benchmark's step: eight long conversations on the 8B shape, bound by its weights
        dict(name="decode 8B x 8", task="decode", model="qwen3_8b", dtype="bfloat16", seqs=8, shortest=4000, longest=4090),
        # a full batch with conversations of every length, half of the traffic is cache
        dict(name="decode 8B x 64", task="decode", model="qwen3_8b", dtype="bfloat16", seqs=64, shortest=16, longest=4096),
        # the benchmark's prompt
        dict(name="prompt 8B 2048 tokens", task="prompt", model="qwen3_8b", dtype="bfloat16", seqs=1, shortest=2048, longest=2048, past=0),
        # a one-line question: time to the first token of a short chat turn
        dict(name="prompt 8B 45 tokens", task="prompt", model="qwen3_8b", dtype="bfloat16", seqs=1, shortest=45, longest=45, past=0),
        # the next turn of two conversations: some hundred new tokens behind a long cached past
        dict(name="next turns 8B", task="prompt", model="qwen3_8b", dtype="bfloat16", seqs=2, shortest=200, longest=350, past=3100),
        # a batch of prompts of very unequal lengths in one step (the 0.6B configuration of the benchmarks: 16 to 2,048 tokens)
        dict(name="prompts 0.6B ragged", task="prompt", model="qwen3_0_6b", dtype="bfloat16", seqs=16, shortest=16, longest=2048, past=0),
        # scoring texts in float32: logits at every position, the precision that parity runs use
        dict(name="score 0.6B float32", task="score", model="qwen3_0_6b", dtype="float32", seqs=3, shortest=5, longest=333, past=0),
        # a reply of a model with a linear recurrence beside attention: the prompt, then single tokens
        dict(name="reply Vabelorn", task="reply", model="vabelorn", dtype="bfloat16", seqs=1, shortest=1500, longest=1500, steps=8),
        # two replies of a model with a gated delta rule beside window attention, and matrix memories
        dict(name="reply Lunadra", task="reply", model="lunadra", dtype="bfloat16", seqs=2, shortest=400, longest=1100, steps=8),
        # drawing the next token of a full batch with the usual filters
        dict(name="sample 64 rows", task="sample", seqs=64, vocab=151936, temperature=0.8, top_k=50, top_p=0.95, min_p=0.0),
    ]


def draw(rng):
    def spread(lo, hi):
        return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    task = rng.choice(["decode", "decode", "decode", "prompt", "prompt", "prompt", "score", "reply", "sample"])
    if task == "sample":
        filters = rng.choice([(0.0, 0, 1.0, 0.0), (rng.uniform(0.3, 1.5), rng.randint(1, 200), rng.uniform(0.5, 1.0), 0.0),
                              (0.7, 40, 0.95, 0.05), (1.0, 0, 1.0, 0.0)])
        return dict(task=task, seqs=spread(1, 64), vocab=rng.choice([151936, rng.randint(1000, 151936)]), temperature=filters[0],
                    top_k=filters[1], top_p=filters[2], min_p=filters[3])
    if task == "reply":
        longest = spread(16, 1500)
        seqs = rng.randint(1, 2) if longest < 1000 else 1
        return dict(task=task, model=rng.choice(["vabelorn", "lunadra"]), dtype="bfloat16", seqs=seqs, shortest=rng.randint(1, longest),
                    longest=longest, steps=rng.randint(1, 8))
    if task == "score":
        longest = spread(16, 333)
        return dict(task=task, model="qwen3_0_6b", dtype="float32", seqs=rng.randint(1, 3), shortest=rng.randint(1, longest),
                    longest=longest, past=0)
    model = rng.choice(["qwen3_0_6b", "qwen3_8b"])
    if task == "decode":
        longest = spread(64, 3900)
        return dict(task=task, model=model, dtype="bfloat16", seqs=spread(1, 64), shortest=rng.randint(16, 64), longest=longest)
    seqs = spread(1, 16 if model == "qwen3_0_6b" else 8)
    past = rng.choice([0, 0, rng.randint(1, 3500)])
    longest = spread(16, min(2048, 2048 if model == "qwen3_0_6b" else 2048 // seqs))
    return dict(task=task, model=model, dtype="bfloat16", seqs=seqs, shortest=rng.randint(2, longest), longest=longest, past=past)


def lengths(case):
    """How many tokens each sequence has (a decode step: before it; a prompt: new ones): part of the case, not of the seed."""
    lo, hi, n = case["shortest"], case["longest"], case["seqs"]
    r = random.Random("%d %d %d" % (lo, hi, n))
    return [hi] + [r.randint(lo, hi) for _ in range(n - 1)]


def tokens_of(case, seed):
    """Per sequence: (cached before, new in the step under test, fed one by one behind it)."""
    r = random.Random(seed * 7919 + 17)
    vocab = QWEN3[case["model"]]["vocab"] if case["model"] in QWEN3 else VOCAB
    out = []
    for n in lengths(case):
        past = n if case["task"] == "decode" else case.get("past", 0)
        new = 1 if case["task"] == "decode" else n
        out.append(tuple([r.randrange(vocab) for _ in range(k)] for k in (past, new, case.get("steps", 0))))
    return out


# ---- models --------------------------------------------------------------------------------------------------------
def qwen3_shapes(m):
    h, q, kv = m["hidden"], m["heads"] * m["dim"], m["kv_heads"] * m["dim"]
    s = {"model.embed_tokens.weight": (m["vocab"], h)}
    for i in range(m["layers"]):
        p = "model.layers.%d." % i
        s.update({p + "input_layernorm.weight": (h,), p + "self_attn.q_proj.weight": (q, h), p + "self_attn.k_proj.weight": (kv, h),
                  p + "self_attn.v_proj.weight": (kv, h), p + "self_attn.o_proj.weight": (h, q), p + "self_attn.q_norm.weight": (m["dim"],),
                  p + "self_attn.k_norm.weight": (m["dim"],), p + "post_attention_layernorm.weight": (h,),
                  p + "mlp.gate_proj.weight": (m["ff"], h), p + "mlp.up_proj.weight": (m["ff"], h), p + "mlp.down_proj.weight": (h, m["ff"])})
    s["model.norm.weight"] = (h,)
    if not m["tied"]:
        s["lm_head.weight"] = (m["vocab"], h)
    return s


def vabelorn_config():
    att = {"type": "attention", "mixer": {"heads": HEADS, "kv_heads": KV_HEADS, "dim": DIM, "vdim": DIM, "scale": DIM ** -0.5,
                                          "rot": {"base": THETA, "dims": DIM // 2, "scaling": YARN}},
           "mlp": {"kind": "dense", "ff": FF}}
    wkv = {"type": "wkv", "mixer": {"heads": WIDTH // 64, "dim": 64, "decay_rank": 64}, "mlp": {"kind": "dense", "ff": FF}}
    return {"architecture": "Vabelorn", "vocab": VOCAB, "width": WIDTH, "logit_scale": 1.0, "norm": {"eps": EPS},
            "token_side": {"dim": 64}, "layers": [att if i % 2 == 0 else wkv for i in range(LAYERS)]}


def vabelorn_shapes(cfg):
    w, n, ds = WIDTH, LAYERS, cfg["token_side"]["dim"]
    s = {"embed": (VOCAB, w), "final.norm": (w,), "side.embed": (VOCAB, n * ds)}
    for i, layer in enumerate(cfg["layers"]):
        p, m = "l%d." % i, layer["mixer"]
        H, d = m["heads"], m["dim"]
        if layer["type"] == "attention":
            G = m["kv_heads"]
            s.update({p + "mix.q": (H * d, w), p + "mix.k": (G * d, w), p + "mix.v": (G * d, w), p + "mix.q.norm": (d,),
                      p + "mix.k.norm": (d,), p + "mix.o": (w, H * d)})
        else:
            s.update({p + "mix.mu." + x: (w,) for x in "rkvgw"})
            s.update({p + "mix." + x: (H * d, w) for x in "rkvg"})
            s.update({p + "mix.w1": (m["decay_rank"], w), p + "mix.w2": (H * d, m["decay_rank"]), p + "mix.w0": (H * d,),
                      p + "mix.u": (H, d), p + "mix.norm": (H * d,), p + "mix.o": (w, H * d)})
        s.update({p + "norm1": (w,), p + "norm2": (w,), p + "mlp.gate": (FF, w), p + "mlp.up": (FF, w), p + "mlp.down": (w, FF),
                  p + "side.gate": (ds, w), p + "side.proj": (w, ds), p + "side.norm": (w,)})
    return s


def lunadra_config():
    side = {"type": "parallel",
            "mixer": {"left": {"heads": HEADS, "kv_heads": KV_HEADS, "dim": DIM, "vdim": DIM, "scale": DIM ** -0.5, "mask": {"size": 1024},
                               "rot": {"base": THETA, "dims": DIM // 2}},
                      "right": {"heads": 8, "kv_heads": 4, "dim": 128, "vdim": 128, "conv": 4, "rank": 64},
                      "left_scale": 1.0, "right_scale": 1.0},
            "mlp": {"kind": "dense", "ff": FF}}
    mem = {"type": "mlstm", "mixer": {"heads": WIDTH // 256, "dim": 128, "vdim": 256, "gate_cap": 15.0}, "mlp": {"kind": "dense", "ff": FF}}
    return {"architecture": "Lunadra", "vocab": VOCAB, "width": WIDTH, "residual_mult": 1.0, "norm": {"eps": EPS},
            "embedding": {"bigram": {"buckets": 65521, "mul_prev": 31, "mul_cur": 7}},
            "layers": [side if i % 2 == 0 else mem for i in range(LAYERS)]}


def lunadra_shapes(cfg):
    w = WIDTH
    s = {"embed": (VOCAB, w), "bigram": (cfg["embedding"]["bigram"]["buckets"] + 1, w), "final.norm": (w,), "head": (VOCAB, w)}
    for i, layer in enumerate(cfg["layers"]):
        p, m = "l%d." % i, layer["mixer"]
        if layer["type"] == "parallel":
            a, b = m["left"], m["right"]
            q = p + "mix.left."
            s.update({q + "q": (a["heads"] * a["dim"], w), q + "k": (a["kv_heads"] * a["dim"], w), q + "v": (a["kv_heads"] * a["vdim"], w),
                      q + "o": (w, a["heads"] * a["vdim"])})
            q = p + "mix.right."
            for x, rows in (("q", b["kv_heads"] * b["dim"]), ("k", b["kv_heads"] * b["dim"]), ("v", b["heads"] * b["vdim"])):
                s.update({q + x: (rows, w), q + x + ".conv": (rows, b["conv"])})
            s.update({q + "b": (b["heads"], w), q + "A_log": (b["heads"],), q + "a1": (b["rank"], w), q + "a2": (b["heads"] * b["dim"], b["rank"]),
                      q + "dt_bias": (b["heads"] * b["dim"],), q + "g1": (b["rank"], w), q + "g2": (b["heads"] * b["vdim"], b["rank"]),
                      q + "norm": (b["vdim"],), q + "o": (w, b["heads"] * b["vdim"])})
        else:
            q, H, d, dv = p + "mix.", m["heads"], m["dim"], m["vdim"]
            s.update({q + "q": (H * d, w), q + "k": (H * d, w), q + "v": (H * dv, w), q + "g": (H * dv, w), q + "o": (w, H * dv),
                      q + "norm": (H * dv,), q + "i": (H, w), q + "i.b": (H,), q + "f": (H, w), q + "f.b": (H,)})
        s.update({p + "norm1": (w,), p + "mlp.gate": (FF, w), p + "mlp.up": (FF, w), p + "mlp.down": (w, FF)})
    return s


def shapes(model):
    if model in QWEN3:
        return qwen3_shapes(QWEN3[model])
    return vabelorn_shapes(vabelorn_config()) if model == "vabelorn" else lunadra_shapes(lunadra_config())


def weights_of(model, seed):
    """Weights by checkpoint name in bfloat16, made on the device: matrices N(0, 0.02), those that write into the residual
    stream smaller by the square root of their number (so that the stream keeps its embedding, as in trained models),
    norms and gates around the values that trained models have them at."""
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed * 1000003 + 5)
    out = {}
    untied = model in QWEN3 and not QWEN3[model]["tied"]
    into_stream = 0.02 / math.sqrt(2 * QWEN3[model]["layers"]) if model in QWEN3 else 0.02
    for name, shape in shapes(model).items():
        t = torch.empty(shape, dtype=torch.bfloat16, device=DEVICE)
        last = name.split(".")[-1]
        if "norm" in name:
            t.normal_(1.0, 0.1, generator=g)
        elif ".mu." in name:
            t.uniform_(0.0, 1.0, generator=g)
        elif last == "w0":                     # per-channel decay: some channels forget fast, some slowly
            t.uniform_(-6.0, 0.5, generator=g)
        elif last in ("u", "conv", "A_log"):
            t.normal_(0.0, 0.5, generator=g)
        elif last == "dt_bias":
            t.normal_(-3.0, 1.0, generator=g)
        elif name.endswith(".f.b"):            # forget gates of a memory are mostly open
            t.normal_(4.0, 1.0, generator=g)
        elif last in ("embed", "bigram"):
            t.normal_(0.0, 0.5, generator=g)
        elif untied and "embed_tokens" in name:    # a tied table is the output head too, and stays at 0.02
            t.normal_(0.0, 1.0, generator=g)
        elif "o_proj" in name or "down_proj" in name:
            t.normal_(0.0, into_stream, generator=g)
        else:
            t.normal_(0.0, 0.02, generator=g)
        out[name] = t
    return out


def engine_of(case, seed):
    model = case["model"]
    if model in QWEN3:
        m = QWEN3[model]
        cfg = pe.preset(model, num_hidden_layers=m["layers"])
    else:
        cfg = pe.VabelornConfig.from_dict(vabelorn_config()) if model == "vabelorn" else pe.LunadraConfig.from_dict(lunadra_config())
    ends = [len(a) + len(b) + len(c) + 1 for a, b, c in tokens_of(case, seed)]
    return pe.Engine(None, config=cfg, weights=weights_of(model, seed), dtype=case["dtype"], max_batch=max(case["seqs"], 1),
                     max_context_len=-(-max(ends) // 64) * 64, max_cache_tokens=sum(-(-n // 64) * 64 for n in ends))


# ---- a pass --------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    if case["task"] == "sample":
        # an engine of any size draws from rows of any vocabulary; rows as peaked as a trained model's
        g = torch.Generator(device=DEVICE)
        g.manual_seed(seed)
        logits = torch.randn(case["seqs"], case["vocab"], generator=g, device=DEVICE) * 2.5
        params = pe.SamplingParams(temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"], min_p=case["min_p"])
        engine = pe.Engine.from_random(pe.preset("tiny_b"), max_context_len=64, max_cache_tokens=64, max_batch=1)
        return dict(task="sample", engine=engine, logits=logits, params=params, seed=seed, requests=list(range(case["seqs"])),
                    steps=[3] * case["seqs"])
    state = dict(task=case["task"], engine=engine_of(case, seed), seqs=tokens_of(case, seed), steps=case.get("steps", 0))
    engine = state["engine"]
    if case["task"] == "reply":
        run(state)          # a serving engine has its decode graphs
        return state
    if case["task"] == "decode" or case.get("past", 0):
        state["slots"] = [engine.alloc_slot() for _ in state["seqs"]]
        step, used = [], 0
        for slot, (past, _, _) in zip(state["slots"], state["seqs"]):
            if used + len(past) > PREFILL_TOKENS:
                engine.step(step)
                step, used = [], 0
            step.append(pe.StepEntry(slot, past))
            used += len(past)
        engine.step(step)
    if case["task"] == "decode":
        run(state)          # likewise
    return state


def run(state):
    engine, task = state["engine"], state["task"]
    if task == "sample":
        return engine.sample(state["logits"], state["params"], state["seed"], state["requests"], state["steps"])
    seqs = state["seqs"]
    slots = state.get("slots") or [engine.alloc_slot() for _ in seqs]
    logits = engine.step([pe.StepEntry(s, new, range(len(new)) if task == "score" else (len(new) - 1,))
                          for s, (_, new, _) in zip(slots, seqs)])
    out = [logits]
    for i in range(state["steps"]):
        logits = engine.step([pe.StepEntry(s, (later[i],), (0,)) for s, (_, _, later) in zip(slots, seqs)])
    if state["steps"]:
        out.append(logits)
    for s, (past, _, _) in zip(slots, seqs):
        if "slots" in state:
            engine.cache.truncate(s, len(past))     # the step can be made again
        else:
            engine.free_slot(s)
    return out


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def work(case):
    if case["task"] == "sample":
        n = case["seqs"] * case["vocab"]
        return {"bytes": 4 * n + 4 * case["seqs"], "flops": 2 * n}
    size = 2 if case["dtype"] == "bfloat16" else 4
    lens, model = lengths(case), case["model"]
    past = lens if case["task"] == "decode" else [case.get("past", 0)] * len(lens)
    new = [1] * len(lens) if case["task"] == "decode" else lens
    steps = case.get("steps", 0)
    sh = shapes(model)
    tables = ("model.embed_tokens.weight", "embed", "bigram", "side.embed", "head", "lm_head.weight")
    layer_params = sum(math.prod(s) for n, s in sh.items() if n not in tables and len(s) == 2)
    head_params = math.prod(sh["model.embed_tokens.weight" if model in QWEN3 else "embed"])
    vocab, hidden = sh["model.embed_tokens.weight" if model in QWEN3 else "embed"]
    bytes_, flops = 0, 0
    for t in range(1 + steps):
        q = new if t == 0 else [1] * len(lens)
        p = past if t == 0 else [a + b + t - 1 for a, b in zip(past, new)]
        wanted = sum(q) if case["task"] == "score" else len(q)
        bytes_ += (layer_params + head_params) * size + sum(q) * hidden * size + wanted * vocab * 4
        flops += 2 * layer_params * sum(q) + 2 * head_params * wanted
        if model in QWEN3:
            m = QWEN3[model]
            layers, heads, kv, dim, window = m["layers"], m["heads"], m["kv_heads"], m["dim"], 1 << 30
        else:
            layers, heads, kv, dim = LAYERS // 2, HEADS, KV_HEADS, DIM
            window = 1024 if model == "lunadra" else 1 << 30
        for a, b in zip(p, q):
            pairs = sum(min(i + 1, window) for i in range(a, a + b)) if window < a + b else b * a + b * (b + 1) // 2
            flops += 4 * layers * heads * dim * pairs
            bytes_ += layers * 2 * kv * dim * size * (min(a, window) + b)
        # the recurrences: state elements of a token and layer, about three multiply-adds each, read and written once a step
        cells = {"vabelorn": (LAYERS // 2) * WIDTH * 64, "lunadra": (LAYERS // 2) * (8 * 128 * 128 + 8 * 128 * 256)}.get(model, 0)
        flops += 6 * cells * sum(q)
        bytes_ += 8 * cells * len(q)
    return {"bytes": int(bytes_), "flops": int(flops)}


def tolerance(case):
    """bfloat16: runs on other kernels (library products in place of the framework's own) differ by 0.5-0.8 % for Qwen3 and
    0.8-1.1 % for the recurrent models, and each is 0.5-1.4 % off the 64-bit logits.  float32: 2e-6 off them."""
    if case["task"] == "sample":
        return "exact"
    return {"rel": 1e-5} if case["dtype"] == "float32" else {"rel": 0.03}


# ---- the same in 64 bits, plainly --------------------------------------------------------------------------------------
def unit(x, eps=EPS):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def halves(x, angles):
    """Rotation of feature i together with feature i + n of the first 2n: ``x [T, heads, d]``, ``angles [T, n]``."""
    n = angles.shape[1]
    c, s = torch.cos(angles)[:, None], torch.sin(angles)[:, None]
    a, b = x[..., :n], x[..., n:2 * n]
    return torch.cat([a * c - b * s, b * c + a * s, x[..., 2 * n:]], dim=-1)


def pairs(x, angles, factor=1.0):
    """Rotation of features (2i, 2i + 1) of the first 2n."""
    n = angles.shape[1]
    c, s = torch.cos(angles)[:, None] * factor, torch.sin(angles)[:, None] * factor
    a, b = x[..., 0:2 * n:2], x[..., 1:2 * n:2]
    return torch.cat([torch.stack([a * c - b * s, b * c + a * s], dim=-1).flatten(-2), x[..., 2 * n:]], dim=-1)


def attend(q, k, v, scale, window=None, sink=False):
    """Causal grouped attention ``[T, H, d]`` over ``[T, G, d]``; ``sink`` adds one to the softmax's denominator."""
    T, H, _ = q.shape
    per = H // k.shape[1]
    i = torch.arange(T, device=q.device)
    out = torch.empty(T, H, v.shape[2], dtype=q.dtype, device=q.device)
    for r0 in range(0, T, 1024):
        r = i[r0:r0 + 1024, None]
        hidden = (i[None] > r) if window is None else (i[None] > r) | (r - i[None] >= window)
        for h in range(H):
            s = (q[r0:r0 + 1024, h] @ k[:, h // per].T * scale).masked_fill(hidden, -math.inf)
            if sink:
                top = s.amax(dim=-1, keepdim=True).clamp(min=0.0)
                e = torch.exp(s - top)
                prob = e / (torch.exp(-top) + e.sum(dim=-1, keepdim=True))
            else:
                prob = torch.softmax(s, dim=-1)
            out[r0:r0 + 1024, h] = prob @ v[:, h // per]
    return out.reshape(T, -1)


def frequencies(dims, base=THETA):
    return base ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device=DEVICE) / dims)


def yarn(dims):
    def turns(t):
        return dims * math.log(YARN["original"] / (2.0 * math.pi * t)) / (2.0 * math.log(THETA))

    lo, hi = max(math.floor(turns(YARN["fast"])), 0), min(math.ceil(turns(YARN["slow"])), dims - 1)
    ramp = ((torch.arange(dims // 2, dtype=torch.float64, device=DEVICE) - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    f = frequencies(dims)
    return f / YARN["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(YARN["factor"]) + 1.0


def silu(x):
    return x * torch.sigmoid(x)


def qwen3_exact(m, W, seqs, rows):
    xs = [W["model.embed_tokens.weight"][torch.tensor(t, device=DEVICE)].double() for t in seqs]
    cut = [len(t) for t in seqs]
    for i in range(m["layers"]):
        p = "model.layers.%d." % i
        w = {n[len(p):-7]: t.double() for n, t in W.items() if n.startswith(p)}
        x = torch.cat(xs)
        h = unit(x) * w["input_layernorm"]
        q, k, v = (torch.split((h @ w["self_attn.%s_proj" % c].T).view(x.shape[0], -1, m["dim"]), cut) for c in "qkv")
        del h
        outs = []
        for a, b, c in zip(q, k, v):
            ang = torch.arange(a.shape[0], dtype=torch.float64, device=DEVICE)[:, None] * frequencies(m["dim"])
            outs.append(attend(halves(unit(a) * w["self_attn.q_norm"], ang), halves(unit(b) * w["self_attn.k_norm"], ang), c, m["dim"] ** -0.5))
        x = x + torch.cat(outs) @ w["self_attn.o_proj"].T
        del q, k, v, outs
        h = unit(x) * w["post_attention_layernorm"]
        for r in range(0, x.shape[0], 8192):
            g = h[r:r + 8192]
            x[r:r + 8192] += (silu(g @ w["mlp.gate_proj"].T) * (g @ w["mlp.up_proj"].T)) @ w["mlp.down_proj"].T
        xs = list(torch.split(x, cut))
    x = torch.cat([x[torch.tensor(r, device=DEVICE)] for x, r in zip(xs, rows)])
    head = W["model.embed_tokens.weight" if m["tied"] else "lm_head.weight"]
    x = unit(x) * W["model.norm.weight"].double()
    return torch.cat([x @ head[r:r + 16384].double().T for r in range(0, head.shape[0], 16384)], dim=1)


def wkv_exact(h, w, p, m):
    T, H, d = h.shape[0], m["heads"], m["dim"]
    before = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
    mix = {s: h + (before - h) * w[p + "mu." + s] for s in "rkvgw"}
    r, k, v = ((mix[s] @ w[p + s].T).view(T, H, d) for s in "rkv")
    keep = torch.exp(-torch.exp(torch.tanh(mix["w"] @ w[p + "w1"].T) @ w[p + "w2"].T + w[p + "w0"])).view(T, H, d)
    S, o = torch.zeros(H, d, d, dtype=h.dtype, device=h.device), []
    for t in range(T):
        kv = k[t, :, :, None] * v[t, :, None]
        o.append((r[t, :, :, None] * (S + w[p + "u"][:, :, None] * kv)).sum(1))
        S = keep[t, :, :, None] * S + kv
    return (unit(torch.stack(o)).reshape(T, H * d) * w[p + "norm"] * silu(mix["g"] @ w[p + "g"].T)) @ w[p + "o"].T


def vabelorn_exact(W, tokens, rows):
    cfg = vabelorn_config()
    w = {n: t.double() for n, t in W.items()}
    tok = torch.tensor(tokens, device=DEVICE)
    T, ds = len(tokens), cfg["token_side"]["dim"]
    pos = torch.arange(T, dtype=torch.float64, device=DEVICE)[:, None]
    x = w["embed"][tok]
    for i, layer in enumerate(cfg["layers"]):
        p, m = "l%d." % i, layer["mixer"]
        if layer["type"] == "attention":
            q, k, v = ((x @ w[p + "mix." + c].T).view(T, -1, m["dim"]) for c in "qkv")
            f, factor = yarn(m["rot"]["dims"])
            turn = pos * frequencies(m["vdim"])
            o = attend(pairs(unit(q) * w[p + "mix.q.norm"], pos * f, factor), pairs(unit(k) * w[p + "mix.k.norm"], pos * f, factor),
                       pairs(unit(v), turn), m["scale"], sink=True)
            y = pairs(o.view(T, -1, m["vdim"]), -turn).reshape(T, -1) @ w[p + "mix.o"].T
        else:
            y = wkv_exact(x, w, p + "mix.", m)
        x = x + unit(y) * w[p + "norm1"]
        y = (silu(x @ w[p + "mlp.gate"].T) * (x @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T
        x = x + unit(y) * w[p + "norm2"]
        z = x @ w[p + "side.gate"].T
        z = 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))
        y = (z * w["side.embed"][tok][:, i * ds:(i + 1) * ds]) @ w[p + "side.proj"].T
        x = x + unit(y) * w[p + "side.norm"]
    return (unit(x[rows]) * w["final.norm"]) @ w["embed"].T


def delta_exact(h, w, p, m):
    T, H, G, d, dv = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]

    def short(c):
        y, taps = h @ w[p + c].T, w[p + c + ".conv"]
        y = torch.cat([torch.zeros(m["conv"] - 1, y.shape[1], dtype=y.dtype, device=y.device), y])
        return silu(sum(y[j:j + T] * taps[:, j] for j in range(m["conv"])))

    q, k, v = short("q").view(T, G, d), short("k").view(T, G, d), short("v").view(T, H, dv)
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    q, k = q.repeat_interleave(H // G, dim=1), k.repeat_interleave(H // G, dim=1)
    beta = torch.sigmoid(h @ w[p + "b"].T)
    step = torch.nn.functional.softplus((h @ w[p + "a1"].T) @ w[p + "a2"].T + w[p + "dt_bias"]).view(T, H, d)
    keep = torch.exp(-torch.exp(w[p + "A_log"])[None, :, None] * step)
    S, o = torch.zeros(H, d, dv, dtype=h.dtype, device=h.device), []
    for t in range(T):
        S = keep[t, :, :, None] * S
        u = beta[t, :, None] * (v[t] - (S * k[t, :, :, None]).sum(1))
        S = S + k[t, :, :, None] * u[:, None]
        o.append((S * q[t, :, :, None]).sum(1))
    gate = torch.sigmoid((h @ w[p + "g1"].T) @ w[p + "g2"].T).view(T, H, dv)
    return (unit(torch.stack(o)) * w[p + "norm"] * gate).reshape(T, H * dv) @ w[p + "o"].T


def mlstm_exact(h, w, p, m):
    T, H, d, dv, cap = h.shape[0], m["heads"], m["dim"], m["vdim"], m["gate_cap"]
    q = (h @ w[p + "q"].T).view(T, H, d) * d ** -0.5
    k, v = (h @ w[p + "k"].T).view(T, H, d), (h @ w[p + "v"].T).view(T, H, dv)
    gi = cap * torch.tanh((h @ w[p + "i"].T + w[p + "i.b"]) / cap)
    gf = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ w[p + "f"].T + w[p + "f.b"]) / cap))
    zeros = lambda *s: torch.zeros(*s, dtype=h.dtype, device=h.device)  # noqa: E731
    S, n, top, o = zeros(H, d, dv), zeros(H, d), zeros(H), []
    for t in range(T):
        new = torch.maximum(gf[t] + top, gi[t])
        keep, take = torch.exp(gf[t] + top - new)[:, None], torch.exp(gi[t] - new)[:, None]
        S = keep[:, :, None] * S + (take * k[t])[:, :, None] * v[t, :, None]
        n, top = keep * n + take * k[t], new
        den = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-top)) + 1e-6
        o.append((S * q[t, :, :, None]).sum(1) / den[:, None])
    return (unit(torch.stack(o)).reshape(T, H * dv) * w[p + "norm"] * torch.sigmoid(h @ w[p + "g"].T)) @ w[p + "o"].T


def lunadra_exact(W, tokens, rows):
    cfg = lunadra_config()
    w = {n: t.double() for n, t in W.items()}
    b, T = cfg["embedding"]["bigram"], len(tokens)
    hashed = [b["buckets"]] + [(x * b["mul_prev"] + y * b["mul_cur"]) % b["buckets"] for x, y in zip(tokens, tokens[1:])]
    x = w["embed"][torch.tensor(tokens, device=DEVICE)] + w["bigram"][torch.tensor(hashed, device=DEVICE)]
    pos = torch.arange(T, dtype=torch.float64, device=DEVICE)[:, None]
    for i, layer in enumerate(cfg["layers"]):
        p, m = "l%d." % i, layer["mixer"]
        h = unit(x) * w[p + "norm1"]
        if layer["type"] == "parallel":
            a = m["left"]
            q, k, v = ((h @ w[p + "mix.left." + c].T).view(T, -1, a["dim"]) for c in "qkv")
            ang = pos * frequencies(a["rot"]["dims"])
            y = attend(halves(q, ang), halves(k, ang), v, a["scale"], window=a["mask"]["size"]) @ w[p + "mix.left.o"].T
            y = y + delta_exact(h, w, p + "mix.right.", m["right"])
        else:
            y = mlstm_exact(h, w, p + "mix.", m)
        x = x + y + (torch.relu(h @ w[p + "mlp.gate"].T) * (h @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T
    return (unit(x[rows]) * w["final.norm"]) @ w["head"].T


def exact(case, seed):
    if case["task"] == "sample" or work(dict(case, task="prompt", past=0))["flops"] > EXACT_FLOPS:
        return None
    seqs, steps = tokens_of(case, seed), case.get("steps", 0)
    every = [a + b + c for a, b, c in seqs]
    if sum(len(t) for t in every) > 40000:
        return None
    rows = [list(range(len(a), len(a) + len(b))) if case["task"] == "score" else [len(a) + len(b) - 1] for a, b, _ in seqs]
    W = weights_of(case["model"], seed)
    if case["model"] in QWEN3:
        return [qwen3_exact(QWEN3[case["model"]], W, every, rows)]
    one = vabelorn_exact if case["model"] == "vabelorn" else lunadra_exact
    got = [one(W, t, r + [len(t) - 1] * (steps > 0)) for t, r in zip(every, rows)]
    return [torch.stack([g[0] for g in got])] + ([torch.stack([g[1] for g in got])] if steps else [])
