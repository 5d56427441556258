"""The work that users have this library do, as cases that can be timed and checked.

A case is one step of serving a decoder through ``Engine``: the prompt step of one or several requests (``kind`` "prompt":
the tokens go in, the logits of each request's last token come out, the requests' slots are given back), or one decode
step of sequences that are already in the cache (``kind`` "decode": one token of each goes in, its logits come out, the
sequences grow by one).  ``lengths`` are the tokens of each prompt, or of each cached sequence, as "8x500" or "45,300".

Sizes are those that the library is built and benchmarked for: the shapes of Llama 3.2 1B and 3B and of Llama 3.1 8B, the
1B shape in true 32 bits, and the Guduzen decoder (several residual streams, windowed, shared and latent attention, the
gated delta rule) of the 1B shape's width and depth, the nearest to a whole of the mechanisms that Llama 3 has not."""
import math
import random
import zlib

import torch

from gpullama3.java_b200.config.registry import architecture_of
from gpullama3.java_b200.engine.api import Engine
from gpullama3.java_b200.engine.step import SequenceInput

DEVICE = "cuda"
F64 = torch.float64
ROOM = 1024             # positions that a decoding sequence grows by before it is over and starts again
PASS_TOKENS = 16384     # tokens of context that go into the cache in one step


def _llama(layers, hidden, heads, head_dim, ff, tied, factor):
    return {"architectures": ["LlamaForCausalLM"], "num_hidden_layers": layers, "hidden_size": hidden,
            "num_attention_heads": heads, "num_key_value_heads": 8, "head_dim": head_dim, "intermediate_size": ff,
            "vocab_size": 128256, "rope_theta": 500000.0, "rms_norm_eps": 1e-5, "tie_word_embeddings": tied,
            "max_position_embeddings": 131072,
            "rope_scaling": {"rope_type": "llama3", "factor": factor, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
                             "original_max_position_embeddings": 8192}}


def _guduzen(layers=16, width=2048, heads=32, kv_heads=8, dim=64, ff=8192, window=1024, kv_rank=128, q_rank=768):
    att = {"heads": heads, "kv_heads": kv_heads, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "mask": {"size": window}}
    lat = {"heads": heads, "dim": dim, "vdim": dim, "kv_rank": kv_rank, "q_rank": q_rank, "scale": dim ** -0.5}
    delta = {"heads": heads, "kv_heads": heads, "dim": dim, "vdim": dim, "conv": 4, "a_rank": 64, "g_rank": 64}
    kinds = [("attention", lambda i: dict(att)), ("attention", lambda i: dict(att, kv_from=i - 1)),
             ("latent_attention", lambda i: dict(lat)), ("channel_delta", lambda i: dict(delta))]
    return {"architecture": "Guduzen", "vocab": 128256, "width": width, "streams": 3, "logit_softcap": 30.0,
            "norm": {"eps": 1e-6}, "layers": [{"type": kinds[i % 4][0], "mixer": kinds[i % 4][1](i),
                                               "mlp": {"kind": "dense", "ff": ff}} for i in range(layers)]}


MODELS = {
    "1b": _llama(16, 2048, 32, 64, 8192, True, 32.0),
    "3b": _llama(28, 3072, 24, 128, 8192, True, 32.0),
    "8b": _llama(32, 4096, 32, 128, 14336, False, 8.0),
    "guduzen": _guduzen(),
}
UNEQUAL = "218,1463,942,1029,117,1633,2026,687"


def listed():
    return [
        # a chat: one person's question, then one token after the other
        {"name": "1b short prompt", "model": "1b", "dtype": "bfloat16", "kind": "prompt", "lengths": "45"},
        {"name": "1b decode alone", "model": "1b", "dtype": "bfloat16", "kind": "decode", "lengths": "900"},
        # a document to be read, and the benchmark's headline: a small batch at a context of 4,096
        {"name": "1b prompt", "model": "1b", "dtype": "bfloat16", "kind": "prompt", "lengths": "2048"},
        {"name": "1b decode batch 8", "model": "1b", "dtype": "bfloat16", "kind": "decode", "lengths": "8x4096"},
        # requests as they come: eight of unequal length
        {"name": "3b unequal prompts", "model": "3b", "dtype": "bfloat16", "kind": "prompt", "lengths": UNEQUAL},
        {"name": "3b unequal decode", "model": "3b", "dtype": "bfloat16", "kind": "decode", "lengths": UNEQUAL},
        # serving at full load: 64 requests at a time
        {"name": "8b many prompts", "model": "8b", "dtype": "bfloat16", "kind": "prompt", "lengths": "64x512"},
        {"name": "8b decode batch 64", "model": "8b", "dtype": "bfloat16", "kind": "decode", "lengths": "64x512"},
        # runs in true 32 bits: to check a conversion, or where bfloat16 is not enough
        {"name": "1b float32 prompt", "model": "1b", "dtype": "float32", "kind": "prompt", "lengths": "2048"},
        {"name": "1b float32 decode", "model": "1b", "dtype": "float32", "kind": "decode", "lengths": "8x500"},
        # a decoder of another design through the same engine
        {"name": "guduzen prompt", "model": "guduzen", "dtype": "bfloat16", "kind": "prompt", "lengths": "2048"},
        {"name": "guduzen decode batch 8", "model": "guduzen", "dtype": "bfloat16", "kind": "decode", "lengths": "8x2000"},
    ]


def _log_uniform(rng, lo, hi):
    return lo if hi <= lo else min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    model, dtype, prompt_tokens, context_tokens = rng.choice([
        ("1b", "bfloat16", 16384, 65536), ("1b", "bfloat16", 16384, 65536), ("3b", "bfloat16", 8192, 16384),
        ("8b", "bfloat16", 4096, 16384), ("1b", "float32", 2048, 4096), ("guduzen", "bfloat16", 8192, 16384)])
    kind = rng.choice(["prompt", "decode"])
    if kind == "prompt":
        longest = _log_uniform(rng, 16, min(8192, prompt_tokens))
        batch = _log_uniform(rng, 1, min(16, prompt_tokens // longest))
    else:
        batch = _log_uniform(rng, 1, 64)
        longest = _log_uniform(rng, 32, min(8192, context_tokens // batch))
    lengths = [longest] + [rng.randint(max(1, longest // 16), longest) for _ in range(batch - 1)]
    rng.shuffle(lengths)
    return {"model": model, "dtype": dtype, "kind": kind, "lengths": ",".join(map(str, lengths))}


def _lengths(case):
    if "x" in case["lengths"]:
        count, length = case["lengths"].split("x")
        return [int(length)] * int(count)
    return [int(n) for n in case["lengths"].split(",")]


# ---- weights and tokens, made from the seed
#
# Matrices have the usual initial spread of 0.02.  The last product of a sublayer has a smaller one, so that what it adds is
# a part of what is in the residual stream already, as in a trained decoder; with the same spread everywhere the first
# layers would drown the embedding and every later rounding would weigh several times as much.

OUTPUT_STD = {"o": 1e-3, "down": 3e-4}


def _shapes(cfg):
    """Checkpoint name -> (shape, mean, standard deviation) of every tensor of a model."""
    if cfg.get("architecture") == "Guduzen":
        return _guduzen_shapes(cfg)
    h, ff, d = cfg["hidden_size"], cfg["intermediate_size"], cfg["head_dim"]
    q, kv = cfg["num_attention_heads"] * d, cfg["num_key_value_heads"] * d
    out = {"model.embed_tokens.weight": ((cfg["vocab_size"], h), 0.0, 0.02), "model.norm.weight": ((h,), 1.0, 0.1)}
    if not cfg["tie_word_embeddings"]:
        out["lm_head.weight"] = ((cfg["vocab_size"], h), 0.0, 0.02)
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        for n in ("input_layernorm", "post_attention_layernorm"):
            out[p + n + ".weight"] = ((h,), 1.0, 0.1)
        for n, shape in (("self_attn.q", (q, h)), ("self_attn.k", (kv, h)), ("self_attn.v", (kv, h)), ("self_attn.o", (h, q)),
                         ("mlp.gate", (ff, h)), ("mlp.up", (ff, h)), ("mlp.down", (h, ff))):
            out[p + n + "_proj.weight"] = (shape, 0.0, OUTPUT_STD.get(n.split(".")[1], 0.02))
    return out


def _guduzen_shapes(cfg):
    h, s = cfg["width"], cfg["streams"]
    out = {"embed": ((cfg["vocab"], h), 0.0, 0.02), "final.norm": ((h,), 0.0, 0.02)}
    for i, layer in enumerate(cfg["layers"]):
        p, m, ff = f"l{i}.", layer["mixer"], layer["mlp"]["ff"]
        H, G, d, dv = m["heads"], m.get("kv_heads", m["heads"]), m["dim"], m["vdim"]
        for j in (1, 2):
            out[p + f"norm{j}"] = ((h,), 0.0, 0.02)
            out.update({p + f"hc{j}.in": ((s,), 1.0 / s, 0.1), p + f"hc{j}.out": ((s,), 1.0, 0.1), p + f"hc{j}.mix": ((s, s), 1.0 / s, 0.05)})
        out.update({p + "mlp.gate": ((ff, h), 0.0, 0.02), p + "mlp.up": ((ff, h), 0.0, 0.02), p + "mlp.down": ((h, ff), 0.0, OUTPUT_STD["down"])})
        p += "mix."
        out[p + "o"] = ((h, H * dv), 0.0, OUTPUT_STD["o"])
        if layer["type"] == "attention":
            for n, rows in (("q", H * d),) if "kv_from" in m else (("q", H * d), ("k", G * d), ("v", G * dv)):
                out[p + n], out[p + n + ".b"] = ((rows, h), 0.0, 0.02), ((rows,), 0.0, 0.02)
        elif layer["type"] == "latent_attention":
            out.update({p + "dq": ((m["q_rank"], h), 0.0, 0.02), p + "dq.norm": ((m["q_rank"],), 1.0, 0.1),
                        p + "uq": ((H * d, m["q_rank"]), 0.0, 0.02), p + "dkv": ((m["kv_rank"], h), 0.0, 0.02),
                        p + "dkv.norm": ((m["kv_rank"],), 1.0, 0.1), p + "uk": ((H * d, m["kv_rank"]), 0.0, 0.02),
                        p + "uv": ((H * dv, m["kv_rank"]), 0.0, 0.02)})
        else:
            for n, rows in (("q", G * d), ("k", G * d), ("v", H * dv)):
                out[p + n], out[p + n + ".conv"] = ((rows, h), 0.0, 0.02), ((rows, m["conv"]), 0.0, m["conv"] ** -0.5)
            out.update({p + "b": ((H, h), 0.0, 0.02), p + "A_log": ((H,), -1.0, 0.5), p + "norm": ((dv,), 1.0, 0.1),
                        p + "a1": ((m["a_rank"], h), 0.0, 0.02), p + "a2": ((H * d, m["a_rank"]), 0.0, 0.02),
                        p + "dt_bias": ((H * d,), 0.0, 1.0), p + "g1": ((m["g_rank"], h), 0.0, 0.02),
                        p + "g2": ((H * dv, m["g_rank"]), 0.0, 0.02)})
    return out


class _Weights:
    """The checkpoint's tensors by name, each made on the GPU when it is asked for: a function of seed and name."""

    def __init__(self, case, seed):
        self.shapes, self.seed, self.dtype = _shapes(MODELS[case["model"]]), int(seed), getattr(torch, case["dtype"])

    def __getitem__(self, name):
        shape, mean, std = self.shapes[name]
        g = torch.Generator(DEVICE).manual_seed((self.seed * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFF)
        t = torch.randn(shape, generator=g, device=DEVICE, dtype=torch.float32).mul_(std).add_(mean)
        return t.to(self.dtype)

    def f64(self, name):
        return self[name].to(F64)


def _tokens(case, seed):
    """The tokens of every sequence, and those that a decoding sequence is fed after them."""
    rng = random.Random(int(seed) * 7919 + 13)
    cfg = MODELS[case["model"]]
    vocab = cfg.get("vocab_size") or cfg["vocab"]
    lengths = _lengths(case)
    return [rng.choices(range(vocab), k=n) for n in lengths], [rng.choices(range(vocab), k=ROOM) for _ in lengths]


# ---- the case itself


def prepare(case, seed):
    cfg = MODELS[case["model"]]
    arch = architecture_of(cfg)
    model = arch.model_factory(arch.config_class.from_dict(cfg), getattr(torch, case["dtype"]), DEVICE)
    model.load_tensors(_Weights(case, seed))
    sequences, fed = _tokens(case, seed)
    room = ROOM if case["kind"] == "decode" else 0
    engine = Engine(model, max_tokens=sum(-(-(len(s) + room) // 64) * 64 for s in sequences), max_batch=len(sequences))
    state = {"kind": case["kind"], "engine": engine, "sequences": sequences, "fed": fed, "slots": [], "at": ROOM}
    if case["kind"] == "decode":
        _start(state)
    return state


def _start(state):
    """The sequences go into the cache; those before them are over."""
    engine, sequences = state["engine"], state["sequences"]
    for slot in state["slots"]:
        engine.cache.release(slot)
    state["slots"], state["at"] = [engine.cache.acquire() for _ in sequences], 0
    batch, total = [], 0
    for slot, tokens in zip(state["slots"], sequences):
        if batch and total + len(tokens) > PASS_TOKENS:
            engine.step(batch)
            batch, total = [], 0
        batch.append(SequenceInput(slot, tokens, []))
        total += len(tokens)
    engine.step(batch)


def run(state):
    engine = state["engine"]
    if state["kind"] == "decode":
        if state["at"] == ROOM:
            _start(state)
        at = state["at"]
        state["at"] = at + 1
        return engine.step([SequenceInput(slot, [fed[at]], [0]) for slot, fed in zip(state["slots"], state["fed"])])
    slots = [engine.cache.acquire() for _ in state["sequences"]]
    try:
        return engine.step([SequenceInput(slot, tokens, [len(tokens) - 1]) for slot, tokens in zip(slots, state["sequences"])])
    finally:
        for slot in slots:
            engine.cache.release(slot)


def _attention_widths(cfg):
    """Of every layer: the floats of a position's keys and values that it keeps, the products of a query with a position
    (multiply-adds), and how many positions a query sees at most."""
    if cfg.get("architecture") != "Guduzen":
        d = cfg["head_dim"]
        return [(2 * cfg["num_key_value_heads"] * d, 2 * cfg["num_attention_heads"] * d, None)] * cfg["num_hidden_layers"]
    out = []
    for layer in cfg["layers"]:
        m = layer["mixer"]
        if layer["type"] == "attention":
            out.append((m["kv_heads"] * (m["dim"] + m["vdim"]), m["heads"] * (m["dim"] + m["vdim"]), m["mask"]["size"]))
        elif layer["type"] == "latent_attention":
            out.append((m["kv_rank"], m["heads"] * (m["dim"] + m["vdim"]), None))
        else:   # a state of fixed size: read, decayed, corrected and read out once for a token
            out.append((0, 0, 0))
    return out


def work(case):
    cfg = MODELS[case["model"]]
    lengths, size = _lengths(case), 4 if case["dtype"] == "float32" else 2
    vocab, hidden = (cfg["vocab"], cfg["width"]) if "width" in cfg else (cfg["vocab_size"], cfg["hidden_size"])
    shapes = _shapes(cfg)
    products = sum(math.prod(shape) for name, (shape, _, _) in shapes.items() if "embed" not in name and name != "lm_head.weight")
    decode, rows = case["kind"] == "decode", len(lengths)
    tokens = rows if decode else sum(lengths)
    flops = 2 * (products * tokens + rows * vocab * hidden)
    cells = 0
    for kept, multiply_adds, window in _attention_widths(cfg):
        reach = lambda n: n if window is None else min(n, window)  # noqa: E731
        if decode:
            seen = [reach(n + 1) for n in lengths]
            cells += kept * (sum(seen) + rows)
            flops += 2 * multiply_adds * sum(seen)
        else:
            cells += kept * tokens
            flops += 2 * multiply_adds * sum(n * (n + 1) // 2 if window is None or n <= window else
                                             window * (window + 1) // 2 + (n - window) * window for n in lengths)
    state_bytes = 0
    for layer in cfg.get("layers", ()):
        if layer["type"] == "channel_delta":
            m = layer["mixer"]
            state = m["heads"] * m["dim"] * m["vdim"]
            state_bytes += 4 * rows * state * (2 if decode else 1)
            flops += 7 * state * tokens
    # every weight once, of the embedding the rows of the tokens (and all of it as the output head), keys and values, logits
    return {"bytes": size * (products + vocab * hidden + tokens * hidden + cells) + state_bytes + 4 * rows * vocab, "flops": flops}


def tolerance(case):
    # four times what the same last token's logits differ by when it goes in as a decode step and as the end of a prompt
    # step, whose products and attention sum in another order: 1.3e-6 in 32 bits, 3.3e-3 (Llama 3) and 6.3e-3 (Guduzen,
    # with more roundings to bfloat16 in a layer); the largest difference was 5 to 6 times that of the norms
    if case["dtype"] == "float32":
        return {"rel": 8e-6, "max": 5e-5}
    return {"rel": 0.025, "max": 0.14} if case["model"] == "guduzen" else {"rel": 0.014, "max": 0.08}


# ---- the same results in 64 bits, from the weights and tokens alone


def exact(case, seed):
    cfg = MODELS[case["model"]]
    sequences, fed = _tokens(case, seed)
    if case["kind"] == "decode":
        sequences = [s + [f[0]] for s, f in zip(sequences, fed)]
    whole = work(dict(case, kind="prompt", lengths=",".join(str(len(s)) for s in sequences)))
    if whole["flops"] > 2e14:   # over some seconds in 64 bits
        return None
    weights = _Weights(case, seed)
    forward = _guduzen_forward if cfg.get("architecture") == "Guduzen" else _llama_forward
    return forward(cfg, weights, sequences)


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _pieces(x, sequences):
    return torch.split(x, [len(s) for s in sequences])


def _attend(q, k, v, scale, window=None):
    """Causal attention of one sequence: q [T, H, d], k and v [T, G, d]; H / G query heads share a key and value head."""
    T, H, d = q.shape
    G = k.shape[1]
    i = torch.arange(T, device=q.device)
    out = torch.empty((T, H, v.shape[2]), dtype=q.dtype, device=q.device)
    for start in range(0, T, 1024):   # (queries a part at a time, for the memory)
        rows = i[start:start + 1024]
        hidden = i[None, :] > rows[:, None]
        if window is not None:
            hidden = hidden | (rows[:, None] - i[None, :] >= window)
        for g in range(G):
            heads = slice(g * (H // G), (g + 1) * (H // G))
            s = torch.einsum("thd,jd->htj", q[rows[0]:rows[-1] + 1, heads], k[:, g]) * scale
            s = s.masked_fill_(hidden, float("-inf")).softmax(-1)
            out[rows[0]:rows[-1] + 1, heads] = torch.einsum("htj,jd->thd", s, v[:, g])
    return out


def _llama_frequencies(cfg):
    d, rule = cfg["head_dim"], cfg["rope_scaling"]
    f = cfg["rope_theta"] ** (-torch.arange(0, d, 2, dtype=F64) / d)
    wavelength = 2 * math.pi / f
    original = rule["original_max_position_embeddings"]
    blend = ((original / wavelength - rule["low_freq_factor"]) / (rule["high_freq_factor"] - rule["low_freq_factor"])).clamp(0, 1)
    return ((1 - blend) * f / rule["factor"] + blend * f).to(torch.float32).to(F64)


def _llama_forward(cfg, W, sequences):
    d, H, G = cfg["head_dim"], cfg["num_attention_heads"], cfg["num_key_value_heads"]
    eps = cfg["rms_norm_eps"]
    x = W.f64("model.embed_tokens.weight")[torch.tensor([t for s in sequences for t in s], device=DEVICE)]
    position = torch.cat([torch.arange(len(s)) for s in sequences]).to(F64)
    angle = (position[:, None] * _llama_frequencies(cfg)[None, :]).to(DEVICE)[:, None, :]
    cos, sin = angle.cos(), angle.sin()

    def rotate(y):
        a, b = y[..., :d // 2], y[..., d // 2:]
        return torch.cat([a * cos - b * sin, a * sin + b * cos], -1)

    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, eps) * W.f64(p + "input_layernorm.weight")
        q, k, v = (h @ W.f64(p + f"self_attn.{n}_proj.weight").T for n in "qkv")
        q, k, v = rotate(q.view(-1, H, d)), rotate(k.view(-1, G, d)), v.view(-1, G, d)
        o = torch.cat([_attend(*parts, d ** -0.5) for parts in zip(*(_pieces(t, sequences) for t in (q, k, v)))])
        x = x + o.reshape(-1, H * d) @ W.f64(p + "self_attn.o_proj.weight").T
        h = _rms(x, eps) * W.f64(p + "post_attention_layernorm.weight")
        gate = torch.nn.functional.silu(h @ W.f64(p + "mlp.gate_proj.weight").T).mul_(h @ W.f64(p + "mlp.up_proj.weight").T)
        x = x + gate @ W.f64(p + "mlp.down_proj.weight").T
    last = torch.cat([piece[-1:] for piece in _pieces(x, sequences)])
    last = _rms(last, eps) * W.f64("model.norm.weight")
    return last @ W.f64("model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight").T


def _guduzen_forward(cfg, W, sequences):
    eps = cfg["norm"]["eps"]
    x = W.f64("embed")[torch.tensor([t for s in sequences for t in s], device=DEVICE)]
    streams = x[:, None, :].expand(-1, cfg["streams"], -1).contiguous()
    kept = {}

    def attention(h, i, p, m):
        H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q = _rms((h @ W.f64(p + "q").T + W.f64(p + "q.b")).view(-1, H, d), eps)
        if "kv_from" not in m:
            kept[i] = (_rms((h @ W.f64(p + "k").T + W.f64(p + "k.b")).view(-1, G, d), eps),
                       (h @ W.f64(p + "v").T + W.f64(p + "v.b")).view(-1, G, dv))
        k, v = kept[m.get("kv_from", i)]
        return torch.cat([_attend(*parts, m["scale"], m["mask"]["size"]) for parts in zip(*(_pieces(t, sequences) for t in (q, k, v)))])

    def latent_attention(h, i, p, m):
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        c_q = _rms(h @ W.f64(p + "dq").T, eps) * W.f64(p + "dq.norm")
        c = _rms(h @ W.f64(p + "dkv").T, eps) * W.f64(p + "dkv.norm")
        q, k, v = ((a @ W.f64(p + n).T).view(-1, H, width) for a, n, width in ((c_q, "uq", d), (c, "uk", d), (c, "uv", dv)))
        return torch.cat([_attend(*parts, m["scale"]) for parts in zip(*(_pieces(t, sequences) for t in (q, k, v)))])

    def channel_delta(h, i, p, m):
        H, d, dv = m["heads"], m["dim"], m["vdim"]   # (as many key heads as heads)

        def convolved(n, width):
            w, outs = W.f64(p + n + ".conv"), []
            for y in _pieces(h @ W.f64(p + n).T, sequences):
                y = torch.nn.functional.pad(y, (0, 0, w.shape[1] - 1, 0))
                outs.append(sum(y[j:y.shape[0] - w.shape[1] + 1 + j] * w[:, j] for j in range(w.shape[1])))
            return torch.nn.functional.silu(torch.cat(outs)).view(-1, H, width)

        unit = lambda y: y * torch.rsqrt((y * y).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
        q, k, v = unit(convolved("q", d)) * d ** -0.5, unit(convolved("k", d)), convolved("v", dv)
        beta = torch.sigmoid(h @ W.f64(p + "b").T)
        step = torch.nn.functional.softplus(((h @ W.f64(p + "a1").T) @ W.f64(p + "a2").T + W.f64(p + "dt_bias")).view(-1, H, d))
        decay = torch.exp(-torch.exp(W.f64(p + "A_log"))[:, None] * step)
        out = []
        for q1, k1, v1, b1, g1 in zip(*(_pieces(t, sequences) for t in (q, k, v, beta, decay))):
            S = torch.zeros((H, d, dv), dtype=F64, device=DEVICE)
            for t in range(q1.shape[0]):
                S = S * g1[t, :, :, None]
                u = b1[t, :, None] * (v1[t] - torch.einsum("hdv,hd->hv", S, k1[t]))
                S = torch.baddbmm(S, k1[t, :, :, None], u[:, None, :])
                out.append(torch.einsum("hdv,hd->hv", S, q1[t]))
        gate = torch.sigmoid((h @ W.f64(p + "g1").T) @ W.f64(p + "g2").T).view(-1, H, dv)
        return _rms(torch.stack(out), eps) * W.f64(p + "norm") * gate

    mixers = {"attention": attention, "latent_attention": latent_attention, "channel_delta": channel_delta}
    for i, layer in enumerate(cfg["layers"]):
        for j in (1, 2):
            p = f"l{i}.hc{j}."
            h = _rms(torch.einsum("tsw,s->tw", streams, W.f64(p + "in")), eps) * (1 + W.f64(f"l{i}.norm{j}"))
            if j == 1:
                y = mixers[layer["type"]](h, i, f"l{i}.mix.", layer["mixer"]).flatten(1) @ W.f64(f"l{i}.mix.o").T
            else:
                gate = torch.nn.functional.gelu(h @ W.f64(f"l{i}.mlp.gate").T, approximate="tanh")
                y = (gate * (h @ W.f64(f"l{i}.mlp.up").T)) @ W.f64(f"l{i}.mlp.down").T
            streams = torch.einsum("tsw,sj->tjw", streams, W.f64(p + "mix")) + W.f64(p + "out")[None, :, None] * y[:, None, :]
    last = torch.cat([piece[-1:] for piece in _pieces(streams.sum(1), sequences)])
    logits = _rms(last, eps) * (1 + W.f64("final.norm")) @ W.f64("embed").T
    return cfg["logit_softcap"] * torch.tanh(logits / cfg["logit_softcap"])
