"""What this framework is timed on: the work that its users have it do, through the entry points they call.

Three ways in: the operations of a global layer that another program calls by themselves ("layer", "scan", "block"), and
the three models behind the engine ("atma", "rizurax", "zemivik"), whose steps are prompts, portions of prompts with
decoding sequences beside them, and decoding.  A decoding step is replayed from a CUDA graph, as the engine does it.

A case is a dict of plain values:
  path      layer | scan | block | atma | rizurax | zemivik
  dtype     bfloat16 | float16 | float32
  layer, scan, block: batch, tokens, heads, kv_heads, window (0 = every key)
  models:   width, layers, prompts (sequences that bring tokens), tokens (the longest's new tokens, the others are shorter),
            done (tokens of theirs that are in the cache already), decodes (decoding sequences), context (the longest
            one's tokens, the new one included)
Weights and inputs are random with the distributions of the benchmark's; token ids are uniform.
"""

import math

import numpy as np
import torch
import torch.nn.functional as F

DEV = "cuda"
HEAD = 128                    # head size of every configuration of this framework
PAGE = 256                    # tokens of a cache page
MODELS = ("atma", "rizurax", "zemivik")
VOCAB = {"atma": 50304, "rizurax": 32768, "zemivik": 32768}
POLAR = {"null_base": 2.0, "null_slope_raw": 0.5, "len_gain_raw": -1.0, "mag_beta_raw": -1.5}
GAMMA_BIAS = 3.9
WINDOW, KEEP = 1024, 4        # of three Zemivik layers in four


# ---- the cases -------------------------------------------------------------------------------------------------------
def op(name, path, batch, tokens, dtype="bfloat16", heads=8, kv_heads=2, window=0):
    return dict(name=name, path=path, dtype=dtype, batch=batch, tokens=tokens, heads=heads, kv_heads=kv_heads, window=window)


def step(name, path, layers, prompts=0, tokens=0, done=0, decodes=0, context=0, width=1024, dtype="bfloat16"):
    return dict(name=name, path=path, dtype=dtype, width=width, layers=layers, prompts=prompts, tokens=tokens, done=done, decodes=decodes,
                context=context)


def listed():
    return [
        # the benchmark's headline: attention and memory of one global layer over one long document
        op("layer_prompt_64k", "layer", 1, 65536),
        # the memory branch by itself over a batch of documents
        op("scan_8x16k", "scan", 8, 16384),
        # one global block in fp32: what a check of a checkpoint against another implementation runs
        op("block_fp32_2k", "block", 1, 2048, dtype="float32"),
        # the 378M model: the prompts of a chat server's step, of all lengths
        step("atma_prompts_7", "atma", 16, prompts=7, tokens=2900),
        # the same model decoding for a full batch with long contexts
        step("atma_decode_64x32k", "atma", 16, decodes=64, context=32768),
        # and for a few users with short ones: the smallest step
        step("atma_decode_3x1k", "atma", 16, decodes=3, context=1000),
        # a long document in one step
        step("rizurax_prompt_32k", "rizurax", 8, prompts=1, tokens=32768),
        # a server's mixed step: the next portion of two long prompts while others decode
        step("rizurax_mixed", "rizurax", 8, prompts=2, tokens=3001, done=9000, decodes=24, context=5000),
        # an agent's handful of conversations
        step("rizurax_decode_8x8k", "rizurax", 8, decodes=8, context=8192),
        # a batch of medium prompts, windowed attention
        step("zemivik_prompts_4x4k", "zemivik", 8, prompts=4, tokens=4096),
        # a full batch decoding, windowed attention
        step("zemivik_decode_64x8k", "zemivik", 8, decodes=64, context=8192),
        # --dtype float32: a prompt whose logits are compared with another implementation's
        step("rizurax_fp32_1500", "rizurax", 8, prompts=1, tokens=1500, dtype="float32"),
    ]


def draw(rng):
    """Another case of the ranges that the listed ones stand for."""
    def between(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("layer", "scan", "block", "prompts", "prompts", "portions", "decode", "decode", "fp32"))
    if kind in ("layer", "scan", "block"):
        heads, kv_heads = rng.choice(((8, 2), (8, 2), (16, 4), (4, 2), (8, 8)))
        dtype = "float32" if kind == "block" else rng.choice(("bfloat16", "bfloat16", "float16"))
        most = {"layer": 65536, "scan": 131072, "block": 4096}[kind] * 8 // max(8, heads)
        tokens = between(64, most if kind != "scan" else most // 2)
        batch = between(1, min(8, max(1, most // tokens)))
        return op("", kind, batch, tokens, dtype, heads, kv_heads, rng.choice((0, 0, WINDOW)) if kind != "scan" else 0)
    model = rng.choice(MODELS)
    width = rng.choice((512, 1024, 1024, 2048))
    layers = 16 if model == "atma" and width <= 1024 else 8
    if kind == "decode":
        decodes = between(1, 64)
        return step("", model, layers, decodes=decodes, context=between(100, 32768 if width <= 1024 else 8192), width=width)
    if kind == "fp32":                                                      # --dtype float32 is an option of these two
        return step("", rng.choice(MODELS[1:]), 8, prompts=rng.choice((1, 2)), tokens=between(32, 1500), width=min(width, 1024), dtype="float32")
    most = 32768 if width <= 1024 else 8192
    if kind == "portions":
        model = rng.choice(MODELS[1:])
        prompts = between(1, 4)
        return step("", model, 8, prompts=prompts, tokens=between(16, 8192 // prompts), done=between(100, 16384), decodes=between(1, 32),
                    context=between(100, 8192), width=width)
    prompts = between(1, 12)
    return step("", model, layers, prompts=prompts, tokens=between(16, min(most, 2 * most // prompts)), width=width)


def sequences(case):
    """[(tokens in the cache, new tokens)] of a step, decoding sequences first; their lengths differ."""
    n, m = case["decodes"], case["prompts"]
    out = [(max(case["context"] - 1 - case["context"] * i // (2 * n), 1), 1) for i in range(n)]
    return out + [(max(case["done"] - 37 * i, 0), max(case["tokens"] - case["tokens"] * 3 * i // (4 * m), 2)) for i in range(m)]


# ---- weights ---------------------------------------------------------------------------------------------------------
def config(case):
    """config.json of the step's model."""
    D, H, path = case["width"], case["width"] // HEAD, case["path"]
    G = max(2, H // 4)
    if path == "atma":
        return {"architecture": "Atma", "layers": case["layers"], "hidden": D, "head_dim": HEAD, "num_kv_heads": G, "gamma_bias": GAMMA_BIAS}
    if path == "rizurax":
        rot = {"dims": 32, "base": 500000.0, "scaling": {"factor": 4.0, "original": 8192, "fast": 32.0, "slow": 1.0}}
        mlp = {"kind": "dense", "ff": 4 * D}
        delta = {"type": "delta", "mlp": mlp, "mixer": {"heads": H, "kv_heads": H // 2, "dim": HEAD, "vdim": HEAD, "conv": 4}}
        att = {"type": "attention", "mlp": mlp, "mixer": {"heads": H, "kv_heads": G, "dim": HEAD // 2, "vdim": HEAD, "diff": 0.4, "scale": 0.125,
                                                          "rot": rot}}
        return {"architecture": "Rizurax", "vocab": VOCAB[path], "width": D, "norm": {"eps": 1e-6},
                "layers": [att if i % 4 == 2 else delta for i in range(case["layers"])],
                "embedding": {"bigram": {"buckets": 4093, "mul_prev": 101, "mul_cur": 7}}}
    most = max(32768, *(a + b for a, b in sequences(case)))

    def layer(size):
        return {"type": "attention", "mlp": {"kind": "dense", "ff": 6 * D},
                "mixer": {"heads": H, "kv_heads": G, "dim": HEAD, "vdim": HEAD, "scale": 0.1, "v_mix": True,
                          "mask": {"size": size, "keep_first": KEEP}}}

    return {"architecture": "Zemivik", "vocab": VOCAB[path], "width": D, "max_positions": most, "norm": {"eps": 1e-6}, "embedding": {"scale": 4.0},
            "layers": [layer(most if i % 4 == 3 else WINDOW) for i in range(case["layers"])]}


class Draws:
    """Random tensors of one seed, in the case's type."""

    def __init__(self, case, seed):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed))
        self.dtype = getattr(torch, case["dtype"])

    def normal(self, *shape, std=1.0, mean=0.0, dtype=None):
        return (torch.randn(shape, device=DEV, generator=self.g) * std + mean).to(dtype or self.dtype)

    def ints(self, most, *shape):
        return torch.randint(0, most, shape, device=DEV, generator=self.g)


def atma_block(put, i, D, G, layered):
    """The tensors of one Atma block; a global one if i % 4 == 2."""
    H, P = D // HEAD, f"blocks.{i}." if layered else ""

    def lin(name, rows, cols):
        put(P + name + ".weight", rows, cols), put(P + name + ".bias", rows, std=0.02)

    if i % 4 == 2:
        lin("attn.q", 2 * H * HEAD, D), lin("attn.k", G * HEAD, D), lin("attn.v", G * HEAD, D)
        for n, channels in (("q", H * HEAD), ("k", G * HEAD), ("v", G * HEAD)):
            put(P + f"attn.canon_{n}.weight", channels, 1, 4, std=0.3)
        lin("attn.proj", D, H * HEAD), lin("attn.mu_proj", D, H)
        put(P + "attn.v_null", H, HEAD, std=0.1, dtype=torch.float32)
        for n, value in POLAR.items():
            put(P + "attn." + n, H, std=0.1, mean=value, dtype=torch.float32)
        lin("attn.mem.w_gamma", H, D), lin("attn.mem.w_beta", H, D), lin("attn.mem.gate", H * HEAD, D), lin("attn.mem.proj", D, H * HEAD)
    else:
        lin("attn.in_proj", 3 * D, D), put(P + "attn.conv.weight", D, 1, 3, std=0.5), lin("attn.out_proj", D, D)
    lin("mlp.fc", 8 * D, D), lin("mlp.proj", D, 4 * D)
    put(P + "norm1.weight", D, std=0.1, mean=1.0), put(P + "norm2.weight", D, std=0.1, mean=1.0)


def weights(case, draws):
    w = {}

    def put(name, *shape, std=None, mean=0.0, dtype=None):
        w[name] = draws.normal(*shape, std=scale * shape[-1] ** -0.5 if std is None else std, mean=mean, dtype=dtype)

    scale = 3 ** -0.5 if case["path"] in ("atma", "block") else 1.0         # that of the default initialisation, +-1/sqrt(fan_in)
    if case["path"] == "block":
        atma_block(put, 2, case["heads"] * HEAD, case["kv_heads"], False)
        return w
    cfg, path = config(case), case["path"]
    D, V = case["width"], VOCAB[path]
    if path == "atma":
        put("embed.weight", V, D, std=1.0)
        for i in range(case["layers"]):
            atma_block(put, i, D, cfg["num_kv_heads"], True)
        put("norm.weight", D, std=0.1, mean=1.0), put("proj.weight", V, D), put("proj.bias", V, std=0.02)
        return w
    if path == "rizurax":
        put("embed", V, D, std=1.0), put("bigram", cfg["embedding"]["bigram"]["buckets"] + 1, D, std=0.5)
    else:
        put("embed", V, D, std=0.3), put("pos", cfg["max_positions"], D, std=0.5), put("embed.norm", D, std=0.1, mean=1.0)
    mean = 0.0 if path == "rizurax" else 1.0
    for i, e in enumerate(cfg["layers"]):
        p, m, ff = f"l{i}.", e["mixer"], e["mlp"]["ff"]
        H, G, d, vd = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        put(p + "norm1", D, std=0.1, mean=mean), put(p + "norm2", D, std=0.1, mean=mean), put(p + "mix.o", D, H * vd)
        if e["type"] == "delta":
            for n, rows in (("q", G * d), ("k", G * d), ("v", H * vd)):
                put(p + "mix." + n, rows, D), put(p + f"mix.{n}.conv", rows, m["conv"], std=0.5)
            put(p + "mix.a", H, D), put(p + "mix.b", H, D), put(p + "mix.g", H * vd, D)
            put(p + "mix.A_log", H, std=0.5, mean=-1.0), put(p + "mix.dt_bias", H, std=0.5, mean=-2.0), put(p + "mix.norm", vd, std=0.1, mean=1.0)
        elif path == "rizurax":
            put(p + "mix.q", H * 2 * d, D), put(p + "mix.k", G * 2 * d, D), put(p + "mix.v", G * vd, D)
            for n in ("lq1", "lk1", "lq2", "lk2"):
                put(p + "mix." + n, d, std=0.2)
        else:
            put(p + "mix.q", H * d, D), put(p + "mix.k", G * d, D), put(p + "mix.v", G * vd, D), put(p + "mix.g", H * vd, D)
            put(p + "mix.q.norm", H * d, std=0.1, mean=1.0), put(p + "mix.k.norm", G * d, std=0.1, mean=1.0), put(p + "mix.vmix", std=0.1, mean=0.3)
        if path == "rizurax":
            put(p + "mlp.gate", ff, D)
        else:
            put(p + "mlp.up.b", ff, std=0.1), put(p + "mlp.down.b", D, std=0.1)
        put(p + "mlp.up", ff, D), put(p + "mlp.down", D, ff)
    put("final.norm", D, std=0.1, mean=mean), put("head", V, D)
    return w


# ---- inputs ----------------------------------------------------------------------------------------------------------
def op_inputs(case, draws):
    B, T, H, G = (case[n] for n in ("batch", "tokens", "heads", "kv_heads"))
    x = {"q": draws.normal(B, T, H, HEAD), "k": draws.normal(B, T, G, HEAD), "v": draws.normal(B, T, G, HEAD)}
    x["g"] = -F.softplus(draws.normal(B, T, H, dtype=torch.float32))
    x["beta"] = torch.sigmoid(draws.normal(B, T, H, dtype=torch.float32))
    if case["path"] == "layer":
        x["g"] = F.logsigmoid(x["g"] + GAMMA_BIAS)         # the layer's slow decay; the scan alone is run with a fast one
    x["polar"] = {"v_null": draws.normal(H, HEAD, std=0.1, dtype=torch.float32)}
    for n, value in POLAR.items():
        x["polar"][n] = draws.normal(H, std=0.1, mean=value, dtype=torch.float32)
    return x


def page_count(case):
    return [-(-(a + b) // PAGE) for a, b in sequences(case)]


def page_lists(case, seed):
    """The cache pages of every sequence, in no order."""
    counts = page_count(case)
    order = np.random.RandomState(int(seed) % (1 << 31)).permutation(sum(counts)).tolist()
    at = np.cumsum([0] + counts)
    return [order[at[i]:at[i + 1]] for i in range(len(counts))]


def step_ids(case, draws):
    """Per sequence the ids of its new tokens, the one before them first."""
    ids = draws.ints(VOCAB[case["path"]], sum(n + 1 for _, n in sequences(case))).tolist()
    out, at = [], 0
    for _, n in sequences(case):
        out.append(ids[at:at + n + 1])
        at += n + 1
    return out


def buffers(case, state):
    """The caches and tables of a model's state by name, in one order."""
    if case["path"] == "atma":
        parts = (("k", state.k_cache), ("v", state.v_cache), ("conv", state.conv), ("mem", state.mem))
        return {f"{n}.{i}": d[i] for n, d in parts for i in sorted(d, key=str)}
    return {f"{i}.{n}": layer[n] for i, layer in enumerate(state) for n in sorted(layer)}


def fill(case, bufs, draws):
    """What sequences that are under way have left behind; nothing if all of them are new."""
    for name in sorted(bufs):
        t = bufs[name]
        if all(done == 0 for done, _ in sequences(case)):
            t.zero_()
        else:
            t.copy_(draws.normal(*t.shape, std=0.3 if "mem" in name or "state" in name else 1.0, dtype=t.dtype))


class Step:
    """A model and one step's batch, as a server holds them."""

    def __init__(self, case, seed):
        from atma_b200.engine import CacheManager, ModelRunner, Sequence
        from atma_b200.registry import model_class

        draws, cfg = Draws(case, seed), config(case)
        w, ids = weights(case, draws), step_ids(case, draws)
        pages, seqs, plan = page_lists(case, seed), sequences(case), []
        self.model = model_class(cfg).from_config(cfg, w, draws.dtype, DEV)
        widest = max(len(p) for p in pages)
        cache = CacheManager(sum(page_count(case)), PAGE, len(seqs), widest)
        self.state = self.model.new_state(len(seqs), cache.num_blocks, PAGE, widest * PAGE)
        for i, (done, new) in enumerate(seqs):
            tokens = [0] * (done - 1) + ids[i] if done else ids[i][1:]
            plan.append((Sequence(i, tokens, done=done, slot=i, pages=pages[i]), new))
        last = np.cumsum([n for _, n in seqs]) - 1
        decoding = not case["prompts"]
        self.batch = ModelRunner(self.model, cache, self.state).build(plan, last.tolist(), pad_decode_to=len(seqs) if decoding else None)
        self.bufs = buffers(case, self.state)
        self.graph = self._capture() if decoding else None
        fill(case, self.bufs, Draws(case, seed + 1_000_003))

    def _capture(self):
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(2):
                self.model.forward(self.batch, self.state)
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            self.logits = self.model.forward(self.batch, self.state)
        return graph

    def run(self):
        if self.graph is None:
            logits = self.model.forward(self.batch, self.state)
            return {"logits": logits, "state": self.bufs}
        self.graph.replay()
        # a decoding step writes one cache row of each sequence, which its own attention has read back
        return {"logits": self.logits, "state": {n: t for n, t in self.bufs.items() if not is_cache(n)}}


def is_cache(name):
    return name.split(".")[0] in ("k", "v") or name.split(".")[1] in ("k", "v")


def prepare(case, seed):
    if case["path"] in MODELS:
        return case, Step(case, seed)
    draws = Draws(case, seed)
    if case["path"] == "block":
        w = weights(case, draws)
        return case, {"w": w, "x": draws.normal(case["batch"], case["tokens"], case["heads"] * HEAD)}
    x = op_inputs(case, draws)
    x["n_keys"] = torch.arange(1, case["tokens"] + 1, device=DEV, dtype=torch.float32)
    return case, x


@torch.no_grad()
def run(state):
    case, x = state
    if isinstance(x, Step):
        return x.run()
    window = case["window"] or None
    if case["path"] == "layer":
        from atma_b200.mixing import global_layer_mixing
        return global_layer_mixing(x["q"], x["k"], x["v"], x["g"], x["beta"], x["n_keys"], x["polar"], window=window)
    if case["path"] == "scan":
        from atma_b200.gated_delta import chunk_gated_delta_rule
        return chunk_gated_delta_rule(q=x["q"], k=x["k"], v=x["v"], g=x["g"], beta=x["beta"], scale=1.0, output_final_state=True,
                                      use_qk_l2norm_in_kernel=True)
    from atma_b200.block import global_block_forward
    return global_block_forward(x["x"], x["w"], head_dim=HEAD, num_kv_heads=case["kv_heads"], window=window, return_state=True)


# ---- what a pass cannot do without -------------------------------------------------------------------------------------
def seen_keys(done, new, window, keep=0):
    """Keys that `new` tokens behind `done` others see, summed."""
    i = np.arange(done + 1, done + new + 1, dtype=np.float64)
    near = np.minimum(i, window) if window else i
    return float((near + np.minimum(i - near, keep)).sum())


def work(case):
    size = {"bfloat16": 2, "float16": 2, "float32": 4}[case["dtype"]]
    delta_flops = 6.0 * HEAD * HEAD                                     # of a token and head: S k, the update, S q
    if case["path"] not in MODELS:
        B, T, H, G = (case[n] for n in ("batch", "tokens", "heads", "kv_heads"))
        attention = 4.0 * HEAD * H * B * seen_keys(0, T, case["window"])
        scan = delta_flops * B * T * H
        moved = B * T * (H + 2 * G) * HEAD * size + B * T * H * 8 + B * T * H * HEAD * size + B * H * HEAD * HEAD * 4
        if case["path"] == "scan":
            return {"bytes": moved, "flops": scan}
        if case["path"] == "layer":
            return {"bytes": moved + B * T * H * (HEAD + 1) * size, "flops": scan + attention}
        D = H * HEAD
        matrices = D * (2 * D + 2 * G * HEAD) + D * (D + H) + 2 * H * D + 2 * D * D + 12 * D * D
        return {"bytes": matrices * size + 2 * B * T * D * size + B * H * HEAD * HEAD * 4, "flops": 2.0 * matrices * B * T + scan + attention}
    D, V, H = case["width"], VOCAB[case["path"]], case["width"] // HEAD
    G, seqs, n = max(2, H // 4), sequences(case), sum(new for _, new in sequences(case))
    matrices, attention, delta, cached, tables = 0, 0.0, 0.0, 0.0, 0.0
    for i in range(case["layers"]):
        window, delta_layer, short_conv = 0, False, False
        if case["path"] == "atma":
            short_conv = i % 4 != 2
            delta_layer = not short_conv
            matrices += 12 * D * D + (4 * D * D if short_conv else 5 * D * D + 2 * D * G * HEAD + 3 * D * H)
        elif case["path"] == "rizurax":
            delta_layer = i % 4 != 2
            matrices += 12 * D * D + (2 * D * (H // 2) * HEAD + 3 * D * D + 2 * D * H if delta_layer else 2 * D * D + 2 * D * G * HEAD)
        else:
            window = 0 if i % 4 == 3 else WINDOW
            matrices += 12 * D * D + 3 * D * D + 2 * D * G * HEAD
        if not short_conv and not (delta_layer and case["path"] == "rizurax"):
            maps = 1.5 if case["path"] == "rizurax" else 1.0                # two maps of half the size, both times the whole values
            attention += 4.0 * HEAD * H * maps * sum(seen_keys(a, b, window, KEEP if window else 0) for a, b in seqs)
            reach = [min(a, window + b + KEEP) if window else a for a, b in seqs]
            cached += 2 * G * HEAD * size * sum(r + b for r, (_, b) in zip(reach, seqs))
        if delta_layer:
            delta += delta_flops * H * n
            tables += H * HEAD * HEAD * 4 * sum(2 if a else 1 for a, _ in seqs)
    moved = (matrices + D * V) * size + 2 * n * D * size + cached + tables + len(seqs) * V * 4
    return {"bytes": moved, "flops": 2.0 * matrices * n + 2.0 * D * V * len(seqs) + attention + delta}


def tolerance(case):
    """Measured against `exact`, with a factor of about four."""
    if case["dtype"] == "float32":
        return {"rel": 1.5e-5, "max": 1e-3}
    if case["path"] in MODELS:
        return {"rel": 0.03, "max": 0.5}
    return {"rel": 0.015, "max": 0.3}


# ---- the same in 64 bits -----------------------------------------------------------------------------------------------
def rms(x, eps=torch.finfo(torch.float32).eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def short_conv(x, taps, before=None):
    """x (T, C), taps (C, K) with the last one on the current row, before (K-1, C): the rows in front."""
    K = taps.shape[1]
    rows = torch.cat([x.new_zeros(K - 1, x.shape[1]) if before is None else before, x])
    return sum(rows[j:j + x.shape[0]] * taps[:, j] for j in range(K)), rows[rows.shape[0] - (K - 1):]


def by_rows(T, keys, heads, f):
    """f(first row, past the last) in blocks whose scores take a gigabyte or so."""
    block = max(1, min(T, int(1.5e8 / max(1, keys * heads))))
    return [f(a, min(a + block, T)) for a in range(0, T, block)]


def scores(q, k, a, b, done, window, keep):
    """q (T, H, d), k (N, H, d): products of rows a..b with the keys up to theirs, and which of them are seen."""
    top = done + b
    i, j = torch.arange(done + a, done + b, device=DEV)[:, None], torch.arange(top, device=DEV)[None, :]
    see = j <= i
    if window:
        see &= (i - j < window) | (j < keep)
    return torch.einsum("thd,nhd->htn", q[a:b], k[:top]), see


def softmax_attention(q, k, v, scale, done, window=0, keep=0, sink=None):
    G = q.shape[1] // k.shape[1]
    k, v = k.repeat_interleave(G, 1), v.repeat_interleave(G, 1)

    def rows(a, b):
        s, see = scores(q, k, a, b, done, window, keep)
        s = (s * scale).masked_fill_(~see, float("-inf"))
        if sink is not None:
            s = torch.cat([s, torch.full_like(s[..., :1], sink)], -1)
        return torch.einsum("htn,nhd->thd", torch.softmax(s, -1)[..., :done + b], v[:done + b])

    return torch.cat(by_rows(q.shape[0], k.shape[0], q.shape[1], rows))


def polar_attention(q, k, v, p, done, window=0):
    """q (T, H, d); k, v (N, G, d).  Returns the directions (T, H, d) and the magnitudes (T, H)."""
    T, H, d = q.shape
    k, v = k.repeat_interleave(H // k.shape[1], 1), v.repeat_interleave(H // v.shape[1], 1)
    p = {n: t.double() for n, t in p.items()}
    gain, slope, beta = (F.softplus(p[n])[:, None] for n in ("len_gain_raw", "null_slope_raw", "mag_beta_raw"))

    def rows(a, b):
        s, see = scores(q, k, a, b, done, window, 0)
        n = torch.arange(done + a + 1, done + b + 1, device=DEV, dtype=torch.float64)
        n = n.clamp_max(window) if window else n
        heat = 1.0 + gain * torch.log(n)
        null = (p["null_base"][:, None] + slope * torch.sqrt(torch.log(n + 1.0))) * heat
        s = (s * (heat / math.sqrt(d))[..., None]).masked_fill_(~see, float("-inf"))
        w = torch.softmax(torch.cat([s, null[..., None]], -1), -1)
        w, w_null = w[..., :-1], w[..., -1]
        c = torch.einsum("htn,nhd->thd", w, v[:done + b]) + w_null.T[..., None] * p["v_null"]
        real = w.sum(-1)
        mag = torch.tanh(beta * torch.log1p(real * real / (w * w).sum(-1).clamp_min(1e-300) * real))
        return c / c.norm(dim=-1, keepdim=True).clamp_min(1e-6), mag.T

    c, mag = zip(*by_rows(T, k.shape[0], H, rows))
    return torch.cat(c), torch.cat(mag)


def delta_rule(q, k, v, g, beta, S=None, chunk=64):
    """q, k (T, H, K), v (T, H, V), g (log decay) and beta (T, H).  Returns the reads (T, H, V) and the last state (H, K, V)."""
    T, H, K = q.shape
    pad = -T % chunk
    q, k, v = (F.pad(x.transpose(0, 1), (0, 0, 0, pad)).unflatten(1, (-1, chunk)) for x in (q, k, v))      # (H, chunks, chunk, .)
    g, beta = (F.pad(x.T, (0, pad)).unflatten(1, (-1, chunk)) for x in (g, beta))
    total = g.cumsum(-1)
    decay = torch.exp((total[..., :, None] - total[..., None, :]).tril()).tril()
    A = beta[..., None] * decay * (k @ k.transpose(-1, -2))
    eye = torch.eye(chunk, device=DEV, dtype=torch.float64)
    solve = torch.linalg.solve_triangular(A.tril(-1) + eye, torch.diag_embed(beta), upper=False, unitriangular=True)
    inside, fade, left = decay * (q @ k.transpose(-1, -2)), torch.exp(total)[..., None], torch.exp(total[..., -1:] - total)[..., None]
    S = torch.zeros(H, K, v.shape[-1], device=DEV, dtype=torch.float64) if S is None else S
    out = torch.empty_like(v)
    for c in range(v.shape[1]):
        u = solve[:, c] @ (v[:, c] - fade[:, c] * (k[:, c] @ S))
        out[:, c] = fade[:, c] * (q[:, c] @ S) + inside[:, c] @ u
        S = fade[:, c, -1:] * S + (left[:, c] * k[:, c]).transpose(-1, -2) @ u
    return out.flatten(1, 2)[:, :T].transpose(0, 1), S


def unit(x, eps=0.0):
    return x * torch.rsqrt((x * x).sum(-1, keepdim=True) + eps)


class Doubles(dict):
    """Weights in 64 bits, each converted when it is asked for."""

    def __getitem__(self, name):
        return super().__getitem__(name).double()

    def lin(self, x, name):
        y = x @ self[name + ".weight"].T
        return y + self[name + ".bias"] if name + ".bias" in self else y


def atma_global(h, w, P, G, cached, conv, S, window=0):
    """The mixing of a global layer over one sequence's new rows h (T, D).  cached: (k, v) rows in front or None, conv: rows
    in front of the three convolutions, S: memory state or None.  Returns the mix, the new (k, v), conv rows and state."""
    T, H = h.shape[0], w[P + "null_base"].shape[0]
    q, gate = w.lin(h, P + "q").view(T, H, 2, HEAD).unbind(2)
    q, k, v = rms(q).flatten(1), rms(w.lin(h, P + "k").view(T, G, HEAD)).flatten(1), w.lin(h, P + "v")
    kept, ends = [], {}
    for n, x in (("q", q), ("k", k), ("v", v)):
        y, ends[n] = short_conv(x, w[P + f"canon_{n}.weight"][:, 0], None if conv is None else conv[n])
        kept.append((x + y).view(T, -1, HEAD))
    q, k, v = kept
    keys, values = (k, v) if cached is None else (torch.cat([cached[0], k]), torch.cat([cached[1], v]))
    params = {n: w[P + n] for n in (*POLAR, "v_null")}
    c, mag = polar_attention(q, keys, values, params, keys.shape[0] - T, window)
    mix = w.lin((c * torch.sigmoid(gate)).flatten(1), P + "proj") + w.lin(mag, P + "mu_proj")
    g, beta = F.logsigmoid(w.lin(h, P + "mem.w_gamma") + GAMMA_BIAS), torch.sigmoid(w.lin(h, P + "mem.w_beta"))
    r, S = delta_rule(unit(q), unit(k).repeat_interleave(H // G, 1), v.repeat_interleave(H // G, 1), g, beta, S)
    mix = mix + w.lin(rms(r).flatten(1) * torch.sigmoid(w.lin(h, P + "mem.gate")), P + "mem.proj")
    return mix, k, v, ends, S


def atma_mlp(x, w, P):
    a, gate = w.lin(rms(x, 1e-6) * w[P + "norm2.weight"], P + "mlp.fc").chunk(2, -1)
    return w.lin(gate * a.relu().square(), P + "mlp.proj")


def exact_ops(case, seed):
    draws, window = Draws(case, seed), case["window"]
    B, T, H, G = (case[n] for n in ("batch", "tokens", "heads", "kv_heads"))
    if case["path"] == "block":
        w = Doubles(weights(case, draws))
        xs, states = draws.normal(B, T, H * HEAD).double(), []
        out = torch.empty_like(xs)
        for b, x in enumerate(xs):
            mix, _, _, _, S = atma_global(rms(x, 1e-6) * w["norm1.weight"], w, "attn.", G, None, None, None, window)
            x = x + mix
            out[b] = x + atma_mlp(x, w, "")
            states.append(S)
        return out, torch.stack(states)
    x = op_inputs(case, draws)
    parts = []
    for b in range(B):
        q, k, v, g, beta = (x[n][b].double() for n in ("q", "k", "v", "g", "beta"))
        c = polar_attention(q, k, v, x["polar"], 0, window) if case["path"] == "layer" else ()
        o, S = delta_rule(unit(q), unit(k).repeat_interleave(H // G, 1), v.repeat_interleave(H // G, 1), g, beta)
        parts.append((*(t.transpose(0, 1) for t in c), o, S))
    return tuple(torch.stack(t) for t in zip(*parts))


class ExactStep:
    """One step of a model: the rows of all sequences through plain matrix products, each sequence's mixing by itself."""

    def __init__(self, case, seed):
        self.case, self.cfg, draws = case, config(case), Draws(case, seed)
        self.dtype = draws.dtype
        self.w, ids = Doubles(weights(case, draws)), step_ids(case, draws)
        self.pages, self.seqs = page_lists(case, seed), sequences(case)
        self.bufs = self._buffers(sum(page_count(case)), len(self.seqs))
        fill(case, self.bufs, Draws(case, seed + 1_000_003))
        self.ids = torch.tensor([t for i in ids for t in i[1:]], device=DEV)
        self.prev = torch.tensor([t if j or done else -1 for i, (done, _) in zip(ids, self.seqs) for j, t in enumerate(i[:-1])], device=DEV)
        ends = np.cumsum([0] + [n for _, n in self.seqs])
        self.rows = [slice(int(a), int(b)) for a, b in zip(ends, ends[1:])]
        self.last = torch.tensor(ends[1:] - 1, device=DEV)
        self.positions = torch.cat([torch.arange(a, a + n, device=DEV) for a, n in self.seqs])

    def _buffers(self, pages, n):
        """Empty caches and tables in the layouts that the framework documents."""
        D, H, path, dt = self.case["width"], self.case["width"] // HEAD, self.case["path"], self.dtype
        G, out = max(2, H // 4), {}
        zeros = lambda *s, dtype=dt: torch.zeros(s, device=DEV, dtype=dtype)  # noqa: E731
        for i in range(self.case["layers"]):
            if path == "atma" and i % 4 == 2:
                out.update({f"k.{i}": zeros(pages, PAGE, G, HEAD), f"v.{i}": zeros(pages, PAGE, G, HEAD),
                            f"mem.{i}": zeros(n, H, HEAD, HEAD, dtype=torch.float32)})
                out.update({f"conv.attn_{i}_{m}": zeros(n, c * HEAD, 3) for m, c in (("q", H), ("k", G), ("v", G))})
            elif path == "atma":
                out[f"conv.conv_{i}"] = zeros(n, D, 2)
            elif path == "rizurax" and i % 4 != 2:
                out.update({f"{i}.conv": zeros(n, 4, 2 * (H // 2) * HEAD + H * HEAD), f"{i}.state": zeros(n, H, HEAD, HEAD, dtype=torch.float32)})
            else:
                out.update({f"{i}.k": zeros(pages, PAGE, G, HEAD), f"{i}.v": zeros(pages, PAGE, G, HEAD)})
        return out

    def cached(self, name, s, new):
        """The rows of sequence s in cache `name`, the new ones behind those in front (and, in 64 bits, in the cache)."""
        done, n = self.seqs[s]
        pages = torch.tensor(self.pages[s], device=DEV)
        rows = self.bufs[name][pages].flatten(0, 1)[:done].double()
        at = torch.arange(done, done + n, device=DEV)
        if self.case["prompts"]:
            self.new.setdefault(name, self.bufs[name].double())[pages[at // PAGE], at % PAGE] = new
        return torch.cat([rows, new])

    def set(self, name, s, value):
        self.new.setdefault(name, self.bufs[name].double())[s] = value

    def run(self):
        self.new = {}
        logits = getattr(self, "_" + self.case["path"])()
        kept = {n: self.new.get(n, t) for n, t in self.bufs.items() if self.case["prompts"] or not is_cache(n)}
        return {"logits": logits, "state": kept}

    def _atma(self):
        w, G = self.w, self.cfg["num_kv_heads"]
        x = w.get("embed.weight")[self.ids].double()
        for i in range(self.case["layers"]):
            P = f"blocks.{i}."
            h = rms(x, 1e-6) * w[P + "norm1.weight"]
            proj = None if i % 4 == 2 else w.lin(h, P + "attn.in_proj")
            mix = torch.empty_like(x)
            for s, r in enumerate(self.rows):
                done = self.seqs[s][0]
                if proj is None:
                    before = {n: self.bufs[f"conv.attn_{i}_{n}"][s].double().T for n in "qkv"} if done else None
                    front = [self.cached(f"{n}.{i}", s, torch.zeros(self.seqs[s][1], G, HEAD, device=DEV, dtype=torch.float64))[:done]
                             for n in "kv"] if done else None
                    mix[r], k, v, conv, S = atma_global(h[r], w, P + "attn.", G, front, before, self.bufs[f"mem.{i}"][s].double() if done else None)
                    self.cached(f"k.{i}", s, k), self.cached(f"v.{i}", s, v), self.set(f"mem.{i}", s, S)
                    for n in "qkv":
                        self.set(f"conv.attn_{i}_{n}", s, conv[n].T)
                else:
                    b, c, value = proj[r].chunk(3, -1)
                    before = self.bufs[f"conv.conv_{i}"][s].double().T if done else None
                    y, last = short_conv(b * value, w[P + "attn.conv.weight"][:, 0], before)
                    mix[r] = c * y
                    self.set(f"conv.conv_{i}", s, last.T)
            x = x + (mix if proj is None else w.lin(mix, P + "attn.out_proj"))
            x = x + atma_mlp(x, w, P)
        z = w.lin(rms(x[self.last], 1e-6) * w["norm.weight"], "proj")
        return 15.0 * z * torch.rsqrt(z * z + 225.0)

    def _delta(self, h, i, m):
        w, p = self.w, f"l{i}.mix."
        H, G, K = m["heads"], m["kv_heads"], m["conv"]
        raw = torch.cat([h @ w[p + n].T for n in "qkv"], 1)
        taps = torch.cat([w[p + n + ".conv"] for n in "qkv"])
        beta, g = torch.sigmoid(h @ w[p + "b"].T), -torch.exp(w[p + "A_log"]) * F.softplus(h @ w[p + "a"].T + w[p + "dt_bias"])
        out = torch.empty(h.shape[0], H, HEAD, device=DEV, dtype=torch.float64)
        for s, r in enumerate(self.rows):
            done, n = self.seqs[s]
            table = self.bufs[f"{i}.conv"][s].double()                      # raw rows by position mod taps
            before = torch.stack([table[t % K] if t >= 0 else torch.zeros_like(table[0]) for t in range(done - K + 1, done)])
            y, _ = short_conv(raw[r], taps, before)
            q, k, v = F.silu(y).view(n, -1, HEAD).split((G, G, H), 1)
            q, k = (unit(t, 1e-6).repeat_interleave(H // G, 1) for t in (q, k))
            S = self.bufs[f"{i}.state"][s].double() if done else None
            out[r], S = delta_rule(q * HEAD ** -0.5, k, v, g[r], beta[r], S)
            for t in range(max(done, done + n - K), done + n):
                table[t % K] = raw[r][t - done]
            self.set(f"{i}.state", s, S), self.set(f"{i}.conv", s, table)
        return (rms(out, 1e-6) * w[p + "norm"]).flatten(1) * F.silu(h @ w[p + "g"].T)

    def _two_maps(self, h, i, m):
        w, p = self.w, f"l{i}.mix."
        H, G, d, rot = m["heads"], m["kv_heads"], m["dim"], m["rot"]
        lam = torch.exp((w[p + "lq1"] * w[p + "lk1"]).sum()) - torch.exp((w[p + "lq2"] * w[p + "lk2"]).sum()) + m["diff"]
        f, sc, n = rot["base"] ** (-2.0 * torch.arange(rot["dims"] // 2, device=DEV, dtype=torch.float64) / rot["dims"]), rot["scaling"], rot["dims"]
        at = [n * math.log(sc["original"] / (2 * math.pi * sc[e])) / (2 * math.log(rot["base"])) for e in ("fast", "slow")]
        lo, hi = max(math.floor(at[0]), 0), min(math.ceil(at[1]), n - 1)
        ramp = ((torch.arange(n // 2, device=DEV) - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        angle = self.positions[:, None] * (f / sc["factor"] * ramp + f * (1 - ramp))
        a = 0.1 * math.log(sc["factor"]) + 1
        cos, sin = (a * torch.cos(angle))[:, None], (a * torch.sin(angle))[:, None]

        def turn(x):
            even, odd = x[..., 0:n:2], x[..., 1:n:2]
            return torch.cat([torch.stack([even * cos - odd * sin, odd * cos + even * sin], -1).flatten(-2), x[..., n:]], -1)

        q, k, v = turn((h @ w[p + "q"].T).view(-1, H * 2, d)), turn((h @ w[p + "k"].T).view(-1, G * 2, d)), (h @ w[p + "v"].T).view(-1, G, HEAD)
        out = torch.empty(h.shape[0], H, HEAD, device=DEV, dtype=torch.float64)
        for s, r in enumerate(self.rows):
            done = self.seqs[s][0]
            keys = self.cached(f"{i}.k", s, k[r].reshape(-1, G, 2 * d)).view(-1, G, 2, d)
            values = self.cached(f"{i}.v", s, v[r])
            a1, a2 = (softmax_attention(q[r].view(-1, H, 2, d)[:, :, j], keys[:, :, j], values, m["scale"], done) for j in (0, 1))
            out[r] = rms(a1 - lam * a2, 1e-6) * (1 - m["diff"])
        return out.flatten(1)

    def _rizurax(self):
        w, big = self.w, self.cfg["embedding"]["bigram"]
        bucket = torch.where(self.prev < 0, big["buckets"], (self.prev * big["mul_prev"] + self.ids * big["mul_cur"]) % big["buckets"])
        x = w.get("embed")[self.ids].double() + w.get("bigram")[bucket].double()
        for i, e in enumerate(self.cfg["layers"]):
            p = f"l{i}."
            h1, h2 = (rms(x, 1e-6) * (1 + w[p + n]) for n in ("norm1", "norm2"))
            mixed = (self._delta if e["type"] == "delta" else self._two_maps)(h1, i, e["mixer"])
            x = x + mixed @ w[p + "mix.o"].T
            x = x + (F.gelu(h2 @ w[p + "mlp.gate"].T, approximate="tanh") * (h2 @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T
        return (rms(x[self.last], 1e-6) * (1 + w["final.norm"])) @ w["head"].T

    def _zemivik(self):
        w, first = self.w, None
        x = rms(w.get("embed")[self.ids].double() * self.cfg["embedding"]["scale"] + w.get("pos")[self.positions].double(), 1e-6) * w["embed.norm"]
        for i, e in enumerate(self.cfg["layers"]):
            p, m = f"l{i}.", e["mixer"]
            q, k = (rms(x @ w[p + "mix." + n].T, 1e-6) * w[p + f"mix.{n}.norm"] for n in "qk")
            q, k, v = q.view(-1, m["heads"], HEAD), k.view(-1, m["kv_heads"], HEAD), (x @ w[p + "mix.v"].T).view(-1, m["kv_heads"], HEAD)
            first, v = (v, v) if first is None else (first, (1 - w[p + "mix.vmix"]) * v + w[p + "mix.vmix"] * first)
            out = torch.empty_like(q)
            for s, r in enumerate(self.rows):
                keys, values = self.cached(f"{i}.k", s, k[r]), self.cached(f"{i}.v", s, v[r])
                out[r] = softmax_attention(q[r], keys, values, m["scale"], self.seqs[s][0], m["mask"]["size"], KEEP, 0.0)
            y = (out.flatten(1) * torch.sigmoid(x @ w[p + "mix.g"].T)) @ w[p + "mix.o"].T
            x = x + rms(y, 1e-6) * w[p + "norm1"]
            y = torch.relu(x @ w[p + "mlp.up"].T + w[p + "mlp.up.b"]).square() @ w[p + "mlp.down"].T + w[p + "mlp.down.b"]
            x = x + rms(y, 1e-6) * w[p + "norm2"]
        return (rms(x[self.last], 1e-6) * w["final.norm"]) @ w["head"].T


@torch.no_grad()
def exact(case, seed):
    return ExactStep(case, seed).run() if case["path"] in MODELS else exact_ops(case, seed)
