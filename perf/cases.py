"""Timed cases of the serving path: what a program that serves language models with this package has it do.

A pass is one scheduling step of such a program.  Its requests are open, their earlier tokens are in the paged cache, and it
hands the engine the next tokens of each request and gets logits back (`Engine.step`): a prompt, a further turn of a
conversation, or one token per sequence.  Portions are packed into batches of at most `MAX_BATCH_TOKENS` tokens, as
`Engine.generate` packs them.  Sampling runs on a batch of logits (`ops.topk_sample`).

Architectures are the presets of `zml_b200.models`, the smallest at full depth, of the others some of their equal layers
(`LAYERS`: what remains is several times the output head, and the oracle takes seconds).  Weights are N(0, 0.02), those that write to the residual stream smaller by
sqrt(2 layers) and embeddings N(0, 1), as models are set up for training: with equal weights everywhere a deep random network
amplifies roundings as no trained one does.  Norm weights lie near one, token ids are uniform; everything comes from the seed.
The lengths of a batch are spread evenly over [shortest, longest] in a shuffled order that the case alone decides.
"""
from __future__ import annotations

import math
import random
import zlib

import torch

from zml_b200 import ops
from zml_b200.models import llama, qwen3_5, qwen3_moe
from zml_b200.serving import Engine

PAGE = 64
MAX_BATCH_TOKENS = 8192
LAYERS = {"llama-3.2-1b": 16, "llama-3.1-8b": 16, "qwen3-30b-a3b": 8, "qwen3-30b-a3b-nvfp4": 8, "qwen3.5-9b": 16}
DEVICE = "cuda"
STD = 0.02
VOCAB_SAMPLED = 128256

FAMILIES = {
    "llama-3.2-1b": (llama.PRESETS, llama.LlamaConfig, llama.LlamaModel),
    "llama-3.1-8b": (llama.PRESETS, llama.LlamaConfig, llama.LlamaModel),
    "qwen3-30b-a3b": (qwen3_moe.PRESETS, qwen3_moe.Qwen3MoeConfig, qwen3_moe.Qwen3MoeModel),
    "qwen3-30b-a3b-nvfp4": (qwen3_moe.PRESETS, qwen3_moe.Qwen3MoeConfig, qwen3_moe.Qwen3MoeModel),
    "qwen3.5-9b": (qwen3_5.PRESETS, qwen3_5.Qwen35Config, qwen3_5.Qwen35Model),
}


def _step(name, model, batch, shortest, longest, past=0):
    return {"name": name, "do": "step", "model": model, "batch": batch, "shortest": shortest, "longest": longest, "past": past}


def _decode(name, model, batch, shortest, longest):
    """One token for each of `batch` sequences that hold [shortest, longest] tokens already."""
    return {"name": name, "do": "decode", "model": model, "batch": batch, "shortest": shortest, "longest": longest, "past": 0}


def listed():
    return [
        # the draw of one token per sequence with the settings of a chat service
        {"name": "sample-32-of-vocabulary", "do": "sample", "rows": 32, "topk": 40, "temperature": 0.8},
        # a chat with a small model on one GPU: first token, every further token, and a long document as the prompt
        _step("1b-prompt-512", "llama-3.2-1b", 1, 512, 512),
        _decode("1b-decode-1", "llama-3.2-1b", 1, 512, 512),
        _step("1b-document-16k", "llama-3.2-1b", 1, 16384, 16384),
        # a few sequences with long contexts
        _decode("1b-decode-6-long", "llama-3.2-1b", 6, 4000, 16000),
        # a service with 32 concurrent users: their prompts, their tokens, and a further turn of three conversations
        _step("8b-prompts-ragged", "llama-3.1-8b", 7, 128, 2048),
        _decode("8b-decode-32", "llama-3.1-8b", 32, 128, 2048),
        _step("8b-further-turn", "llama-3.1-8b", 3, 100, 400, past=3000),
        # a mixture of experts: prompts in bf16, 128 concurrent sequences in NVFP4
        _step("moe-prompts-8x1024", "qwen3-30b-a3b", 8, 1024, 1024),
        _decode("moe-nvfp4-decode-128", "qwen3-30b-a3b-nvfp4", 128, 1024, 1024),
        # a hybrid of gated delta nets and full attention
        _step("hybrid-prompts-ragged", "qwen3.5-9b", 7, 128, 2048),
        _decode("hybrid-decode-32", "qwen3.5-9b", 32, 128, 2048),
    ]


def _log_int(rng, lo, hi):
    return min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    """Any of the above with other sizes; a batch holds at most what the largest listed one of its kind holds."""
    kind = rng.choice(["sample", "step", "step", "step", "decode", "decode", "decode"])
    if kind == "sample":
        return {"do": "sample", "rows": _log_int(rng, 1, 128), "topk": _log_int(rng, 2, 128), "temperature": round(rng.uniform(0.3, 1.5), 2)}
    model = rng.choice(sorted(FAMILIES))
    if kind == "decode":
        most = {"llama-3.2-1b": 64, "llama-3.1-8b": 32, "qwen3.5-9b": 32}.get(model, 128)
        batch = _log_int(rng, 1, most)
        room = {"llama-3.2-1b": 60000, "llama-3.1-8b": 34816, "qwen3.5-9b": 34816}.get(model, 131072)    # tokens that the caches hold
        longest = _log_int(rng, 64, max(64, min(16384 if "llama" in model else 4096, room // batch)))
        return {"do": "decode", "model": model, "batch": batch, "shortest": _log_int(rng, max(1, longest // 16), longest), "longest": longest, "past": 0}
    total = _log_int(rng, 16, 16384 if model == "llama-3.2-1b" else 8192)
    batch = rng.choice([1, 1, 2, 3, 5, 8, 13, 32])
    longest = max(1, total // batch)
    past = rng.choice([0, 0, _log_int(rng, 16, 6000)]) if batch <= 5 else 0
    return {"do": "step", "model": model, "batch": batch, "shortest": _log_int(rng, max(1, longest // 16), longest), "longest": longest, "past": past}


# ------------------------------------------------------------------------------------------ sizes
def _config(case):
    presets, config, _ = FAMILIES[case["model"]]
    return config.from_hf(dict(presets[case["model"]], num_hidden_layers=LAYERS[case["model"]]))


def _lengths(case):
    n, lo, hi = case["batch"], case["shortest"], case["longest"]
    out = [hi] if n == 1 else [lo + (hi - lo) * i // (n - 1) for i in range(n)]
    random.Random(1000003 * n + 1009 * lo + hi).shuffle(out)
    return out


def _portions(case):
    """(tokens in the cache, tokens of the pass) of every sequence."""
    return [(n, 1) if case["do"] == "decode" else (case["past"], n) for n in _lengths(case)]


def work(case):
    if case["do"] == "sample":
        return {"bytes": case["rows"] * (VOCAB_SAMPLED * 4 + case["topk"] * 8 + 4), "flops": 0}
    c, parts = _config(case), _portions(case)
    d, hd, hq, hkv, layers = c.hidden_size, c.hd, c.num_attention_heads, c.num_key_value_heads, c.num_hidden_layers
    new, rows = sum(n for _, n in parts), len(parts)
    pairs = sum(n * p + n * (n + 1) // 2 for p, n in parts)          # (query, visible key) pairs of a causal layer
    keys = sum(p + n for p, n in parts)
    types = getattr(c, "layer_types", ["full_attention"] * layers)
    full, linear = types.count("full_attention"), types.count("linear_attention")
    gate = 1 if linear else 0                                        # the hybrid's attention has an output gate
    attn = full * d * hd * ((2 + gate) * hq + 2 * hkv)
    flops = 4 * full * hq * hd * pairs
    data = 2 * (full * 2 * hkv * hd * (keys + new)) + 2 * d * new    # cached keys and values, embedded rows
    if linear:
        kd, vd, hv = c.linear_num_key_heads * c.linear_key_head_dim, c.linear_num_value_heads * c.linear_value_head_dim, c.linear_num_value_heads
        attn += linear * d * (2 * kd + 3 * vd + 2 * hv)
        flops += linear * 6 * new * c.linear_key_head_dim * vd
        data += linear * rows * 2 * 4 * c.linear_key_head_dim * vd
    if getattr(c, "num_experts", 0):
        f, e, k = c.moe_intermediate_size, c.num_experts, c.num_experts_per_tok
        hit = e * (1 - (1 - k / e) ** new)
        mlp = layers * 3 * d * f
        data += mlp * hit * (9 / 16 if c.expert_dtype == "nvfp4" else 2) + 2 * layers * e * d
        mlp *= k
    else:
        mlp = layers * 3 * d * c.intermediate_size
        data += 2 * mlp
    data += 2 * (attn + c.vocab_size * d) + 4 * rows * c.vocab_size
    flops += 2 * new * (attn + mlp) + 2 * rows * c.vocab_size * d
    return {"bytes": data, "flops": flops}


# ------------------------------------------------------------------------------------------ inputs
_E2M1 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0)


def _nvfp4(w):
    """[E, N, K] -> (codes [E, N, K / 2], low nibble first, block scales [E, N, K / 16], matrix scales [E]), and what they stand for."""
    e, n, k = w.shape
    x = w.float().reshape(e, n, k // 16, 16)
    matrix = x.abs().amax((1, 2, 3)) / (6.0 * 448.0)
    scale = (x.abs().amax(-1) / 6.0 / matrix[:, None, None]).to(torch.float8_e4m3fn)
    step = (scale.float() * matrix[:, None, None])[..., None]
    grid = torch.tensor(_E2M1, device=w.device)
    code = torch.bucketize(x.abs() / step.clamp_min(1e-30), (grid[1:] + grid[:-1]) / 2)
    value = torch.where(x < 0, -grid[code], grid[code]) * step
    code = (code + torch.where(x < 0, 8, 0)).to(torch.uint8).reshape(e, n, k // 2, 2)
    return (code[..., 0] | (code[..., 1] << 4), scale, matrix), value.reshape(e, n, k)


class _Checkpoint:
    """Weights under their checkpoint names, made one by one from the seed as a loader asks for them (the two methods of
    `zml_b200.io.TensorStore` that the models' loaders call)."""

    def __init__(self, case, seed):
        self.c, self.seed = _config(case), seed
        self.hybrid = case["model"].startswith("qwen3.5")
        self.pre = "model.language_model." if self.hybrid else "model."
        self.fp4, self.made = getattr(self.c, "expert_dtype", "bf16") == "nvfp4", {}

    def has_key(self, name):
        if "mlp.experts." in name:
            return name.endswith(("weight_scale", "weight_scale_2")) if self.fp4 else name.endswith("gate_up_proj")
        if name == "lm_head.weight":
            return not self.c.tie_word_embeddings
        return self.c.qk_norm if name.endswith(("q_norm.weight", "k_norm.weight")) else not name.endswith("bias")

    def normal(self, name, *shape, std=STD, mean=0.0, dtype=torch.bfloat16):
        if "embed_tokens" in name:
            std = 1.0
        elif any(w in name for w in ("o_proj", "out_proj", "down_proj")):
            std = STD / math.sqrt(2 * self.c.num_hidden_layers)
        g = torch.Generator(device=DEVICE).manual_seed(self.seed * 4294967296 + zlib.crc32(name.encode()))
        return torch.empty(shape, dtype=dtype, device=DEVICE).normal_(mean, std, generator=g)

    def experts(self, layer, which):
        """(packed form, values) of one expert projection of a layer in NVFP4."""
        key = (layer, which)
        if key not in self.made:
            self.made = {k: v for k, v in self.made.items() if k[0] == layer}
            c = self.c
            shape = (c.hidden_size, c.moe_intermediate_size) if which == "down_proj" else (c.moe_intermediate_size, c.hidden_size)
            self.made[key] = _nvfp4(self.normal(f"{layer}.experts.{which}", c.num_experts, *shape))
        return self.made[key]

    def load_tensor(self, name, device=DEVICE, dtype=None, rows=None, cols=None):
        c = self.c
        d, hd, f = c.hidden_size, c.hd, c.intermediate_size
        last = name.rsplit(".", 1)[0].rsplit(".", 1)[-1] if name.endswith(".weight") else name.rsplit(".", 1)[-1]
        if "mlp.experts." in name and self.fp4:
            _, _, layer, _, _, expert, which, part = name.split(".")
            codes, scales, matrix = self.experts(layer, which)[0]
            return {"weight": codes, "weight_scale": scales, "weight_scale_2": matrix}[part][int(expert)]
        qg = 2 if self.hybrid else 1                                # the hybrid's q_proj rows are [query | gate] per head
        near = 0.0 if self.hybrid else 1.0                          # and its norms multiply by one plus their weight
        if name.endswith(("layernorm.weight", "model.norm.weight", "language_model.norm.weight")):
            return self.normal(name, d, std=0.1, mean=near)
        if last in ("q_norm", "k_norm"):
            return self.normal(name, hd, std=0.1, mean=near)
        if last == "norm":
            return self.normal(name, c.linear_value_head_dim, std=0.1, mean=1.0)
        if last == "A_log":
            return self.normal(name, c.linear_num_value_heads, std=0.7, mean=1.6, dtype=torch.float32)
        if last == "dt_bias":
            return self.normal(name, c.linear_num_value_heads, std=0.6, dtype=torch.float32)
        kd = vd = hv = 0
        if self.hybrid:
            kd, vd, hv = c.linear_num_key_heads * c.linear_key_head_dim, c.linear_num_value_heads * c.linear_value_head_dim, c.linear_num_value_heads
        if last == "conv1d":
            return self.normal(name, 2 * kd + vd, 1, c.linear_conv_kernel_dim, std=0.3)
        if "mlp.experts." in name:
            m = c.moe_intermediate_size
            return self.normal(name, c.num_experts, *((2 * m, d) if last == "gate_up_proj" else (d, m)))
        shape = {"embed_tokens": (c.vocab_size, d), "lm_head": (c.vocab_size, d), "q_proj": (qg * c.num_attention_heads * hd, d),
                 "k_proj": (c.num_key_value_heads * hd, d), "v_proj": (c.num_key_value_heads * hd, d), "o_proj": (d, c.num_attention_heads * hd),
                 "gate_proj": (f, d), "up_proj": (f, d), "down_proj": (d, f), "gate": (getattr(c, "num_experts", 0), d),
                 "in_proj_qkv": (2 * kd + vd, d), "in_proj_z": (vd, d), "in_proj_b": (hv, d), "in_proj_a": (hv, d), "out_proj": (d, vd)}[last]
        return self.normal(name, *shape)


def _tokens(case, seed):
    """All token ids of every sequence, those in the cache first."""
    g, v = torch.Generator().manual_seed(seed), _config(case).vocab_size
    return [torch.randint(0, v, (p + n,), generator=g).tolist() for p, n in _portions(case)]


def _batches(requests, portions):
    """Portions packed into batches of at most MAX_BATCH_TOKENS tokens; wanted: the logits behind a portion's last token."""
    batches, entries, want, used = [], [], [], 0
    for r, tokens in zip(requests, portions):
        at = 0
        while at < len(tokens):
            take = min(len(tokens) - at, MAX_BATCH_TOKENS - used)
            entries.append((r, tokens[at:at + take]))
            at += take
            want.append([take - 1] if at == len(tokens) else [])
            used += take
            if used == MAX_BATCH_TOKENS:
                batches.append((entries, want))
                entries, want, used = [], [], 0
    return batches + ([(entries, want)] if entries else [])


def prepare(case, seed):
    if case["do"] == "sample":
        g = torch.Generator(device=DEVICE).manual_seed(seed)
        logits = torch.empty((case["rows"], VOCAB_SAMPLED), device=DEVICE).normal_(0.0, 2.5, generator=g)
        return {"logits": logits, "topk": case["topk"], "temperature": case["temperature"], "seed": seed % 65536}
    _, _, cls = FAMILIES[case["model"]]
    model = cls(_config(case), device=DEVICE)
    model.load(_Checkpoint(case, seed))
    parts, tokens = _portions(case), _tokens(case, seed)
    longest = max(p + n for p, n in parts)
    pages = sum((p + n + PAGE - 1) // PAGE for p, n in parts)
    engine = Engine(model, num_pages=pages + 1, page_size=PAGE, max_batch=len(parts), max_seq_len=longest + 512, max_prefill_tokens=MAX_BATCH_TOKENS,
                    num_state_slots=len(parts))
    requests = [engine.open_request() for _ in parts]
    for entries, _ in _batches(requests, [t[:p] for (p, _), t in zip(parts, tokens)]):
        engine.step(entries)
    return {"engine": engine, "requests": requests, "past": [p for p, _ in parts],
            "batches": _batches(requests, [t[p:] for (p, _), t in zip(parts, tokens)])}


def run(state):
    if "logits" in state:
        tok, values, ids = ops.topk_sample(state["logits"], state["topk"], state["temperature"], seed=state["seed"], return_topk=True)
        return {"tokens": tok, "values": values, "ids": ids}
    for r, past in zip(state["requests"], state["past"]):           # back to where the pass begins: its rows of the cache are written again
        del r.prompt[past:]
        r.computed = past
    out = [state["engine"].step(entries, want) for entries, want in state["batches"]]
    return [lg for lg in out if lg is not None]


# ------------------------------------------------------------------------------------------ oracle
def tolerance(case):
    if case["do"] == "sample":
        return "exact"
    # bf16 activations through 8 to 16 layers: 0.9 - 1.5 % from 64 bits, and 0.2 - 1.7 % (0.09 of the result's root mean square at
    # one place) between runs whose norms, GEMMs and attention sum in another order
    return {"rel": 0.03, "max": 0.4}


def _rms(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _rope(x, pos, c, rot):
    """Rotation of the first `rot` dims of x [T, H, D], halves paired, with the frequencies of the configuration."""
    inv = c.rope_theta ** (-torch.arange(0, rot, 2, dtype=torch.float64, device=x.device) / rot)
    s = c.rope_scaling
    if s:                                                           # llama3: long waves stretched, a smooth passage between
        wave = 2 * math.pi / inv
        lo, hi, old = s["low_freq_factor"], s["high_freq_factor"], s["original_max_position_embeddings"]
        mix = ((old / wave - lo) / (hi - lo)).clamp(0, 1)
        inv = (1 - mix) * inv / s["factor"] + mix * inv
    a = pos[:, None].double() * inv[None]
    cos, sin = a.cos()[:, None], a.sin()[:, None]
    u, v = x[..., :rot // 2], x[..., rot // 2:rot]
    return torch.cat([u * cos - v * sin, v * cos + u * sin, x[..., rot:]], -1)


def _attend(q, k, v):
    """Causal attention of one sequence, q [T, Hq, D], k, v [T, Hkv, D], in blocks of queries."""
    t, hq, d = q.shape
    rep, out = hq // k.shape[1], torch.empty_like(q)
    block = max(64, min(t, (1 << 27) // (t * rep)))
    for h in range(k.shape[1]):
        for a in range(0, t, block):
            b = min(t, a + block)
            s = torch.einsum("qgd,kd->gqk", q[a:b, h * rep:(h + 1) * rep], k[:b, h]) / math.sqrt(d)
            s.masked_fill_(torch.arange(b, device=q.device)[None, None] > torch.arange(a, b, device=q.device)[None, :, None], -math.inf)
            out[a:b, h * rep:(h + 1) * rep] = torch.einsum("gqk,kd->qgd", torch.softmax(s, -1), v[:b, h])
    return out


def _delta_net(x, get, c, spans):
    """The gated delta net layer of the hybrid on normed inputs, token by token, all sequences side by side."""
    hk, hv, dk, dv = c.linear_num_key_heads, c.linear_num_value_heads, c.linear_key_head_dim, c.linear_value_head_dim
    mix, z = x @ get("in_proj_qkv.weight").t(), x @ get("in_proj_z.weight").t()
    beta = torch.sigmoid(x @ get("in_proj_b.weight").t())
    decay = torch.exp(-get("A_log").exp() * torch.nn.functional.softplus(x @ get("in_proj_a.weight").t() + get("dt_bias")))
    w = get("conv1d.weight")[:, 0]
    kk, n, longest = w.shape[1], len(spans), max(b - a for a, b in spans)
    pad = lambda m: torch.stack([torch.nn.functional.pad(m[a:b], (0, 0, 0, longest - (b - a))) for a, b in spans])   # noqa: E731
    mix = torch.nn.functional.conv1d(torch.nn.functional.pad(pad(mix).transpose(1, 2), (kk - 1, 0)), w[:, None], groups=w.shape[0]).transpose(1, 2)
    mix, beta, decay = torch.nn.functional.silu(mix), pad(beta), pad(decay)
    unit = lambda m: m * torch.rsqrt((m * m).sum(-1, keepdim=True) + 1e-6)                                           # noqa: E731
    q = unit(mix[..., :hk * dk].reshape(n, longest, hk, dk)).repeat_interleave(hv // hk, 2) * dk ** -0.5
    k = unit(mix[..., hk * dk:2 * hk * dk].reshape(n, longest, hk, dk)).repeat_interleave(hv // hk, 2)
    v = mix[..., 2 * hk * dk:].reshape(n, longest, hv, dv)
    state, y = torch.zeros((n, hv, dk, dv), dtype=x.dtype, device=x.device), torch.empty_like(v)
    for t in range(longest):
        state = state * decay[:, t, :, None, None]
        delta = (v[:, t] - (k[:, t, :, None] @ state)[:, :, 0]) * beta[:, t, :, None]
        state = state + k[:, t, :, :, None] * delta[:, :, None]
        y[:, t] = (q[:, t, :, None] @ state)[:, :, 0]
    y = torch.cat([y[i, :b - a] for i, (a, b) in enumerate(spans)])
    y = _rms(y, get("norm.weight"), c.rms_norm_eps) * torch.nn.functional.silu(z.reshape(-1, hv, dv))
    return y.reshape(-1, hv * dv) @ get("out_proj.weight").t()


def exact(case, seed):
    """The logits in 64 bits, all tokens of a sequence at once.  None where that takes too long, and for steps that round the
    experts' inputs to NVFP4 (up to 128 tokens per expert): there the result is a matter of that rounding."""
    if case["do"] == "sample":
        v, i = torch.topk(prepare(case, seed)["logits"], case["topk"])
        return {"tokens": None, "values": v.double(), "ids": i.to(torch.int32)}
    c, parts = _config(case), _portions(case)
    total = [p + n for p, n in parts]
    per_token = work(dict(case, do="step", batch=1, shortest=1, longest=1, past=0))["flops"] - 2 * c.vocab_size * c.hidden_size
    if per_token * sum(total) > 3e14:
        return None
    experts, top = getattr(c, "num_experts", 0), getattr(c, "num_experts_per_tok", 0)
    if getattr(c, "expert_dtype", "") == "nvfp4" and (len(parts) if case["do"] == "decode" else min(MAX_BATCH_TOKENS, sum(total))) * top // experts <= 128:
        return None
    store = _Checkpoint(case, seed)
    hybrid, hd = store.hybrid, c.hd
    one = 1.0 if hybrid else 0.0
    ids = torch.tensor([t for seq in _tokens(case, seed) for t in seq], device=DEVICE)
    spans = [(sum(total[:i]), sum(total[:i + 1])) for i in range(len(total))]
    pos = torch.cat([torch.arange(n, device=DEVICE) for n in total])
    x = store.load_tensor(store.pre + "embed_tokens.weight")[ids].double()
    for l in range(c.num_hidden_layers):
        get = lambda name: store.load_tensor(f"{store.pre}layers.{l}.{name}").double()                   # noqa: E731,B023
        n1 = _rms(x, one + get("input_layernorm.weight"), c.rms_norm_eps)
        if hybrid and c.layer_types[l] == "linear_attention":
            x = x + _delta_net(n1, lambda name: get("linear_attn." + name), c, spans)                    # noqa: B023
        else:
            q, gate = (n1 @ get("self_attn.q_proj.weight").t()).reshape(len(ids), c.num_attention_heads, -1), None
            if hybrid:
                q, gate = q[..., :hd], q[..., hd:]
            k = (n1 @ get("self_attn.k_proj.weight").t()).reshape(len(ids), c.num_key_value_heads, hd)
            v = (n1 @ get("self_attn.v_proj.weight").t()).reshape(len(ids), c.num_key_value_heads, hd)
            if c.qk_norm:
                q, k = _rms(q, one + get("self_attn.q_norm.weight"), c.rms_norm_eps), _rms(k, one + get("self_attn.k_norm.weight"), c.rms_norm_eps)
            rot = c.rotary_dim if hybrid else hd
            q, k = _rope(q, pos, c, rot), _rope(k, pos, c, rot)
            o = torch.cat([_attend(q[a:b], k[a:b], v[a:b]) for a, b in spans])
            o = o if gate is None else o * torch.sigmoid(gate)
            x = x + o.reshape(len(ids), -1) @ get("self_attn.o_proj.weight").t()
        n2 = _rms(x, one + get("post_attention_layernorm.weight"), c.rms_norm_eps)
        if not experts:
            x = x + (torch.nn.functional.silu(n2 @ get("mlp.gate_proj.weight").t()) * (n2 @ get("mlp.up_proj.weight").t())) @ get("mlp.down_proj.weight").t()
            continue
        w, chosen = torch.topk(n2 @ get("mlp.gate.weight").t(), top, dim=-1)
        w, f = torch.softmax(w, -1), c.moe_intermediate_size
        if c.expert_dtype == "nvfp4":
            gate_w, up_w, down_w = (store.experts(str(l), which)[1] for which in ("gate_proj", "up_proj", "down_proj"))
        else:
            gate_up, down_w = (store.load_tensor(f"{store.pre}layers.{l}.mlp.experts.{which}") for which in ("gate_up_proj", "down_proj"))
            gate_w, up_w = gate_up[:, :f], gate_up[:, f:]
        add = torch.zeros_like(x)
        for e in range(experts):
            tok, j = (chosen == e).nonzero(as_tuple=True)
            h = torch.nn.functional.silu(n2[tok] @ gate_w[e].double().t()) * (n2[tok] @ up_w[e].double().t())
            add.index_add_(0, tok, (h @ down_w[e].double().t()) * w[tok, j, None])
        x = x + add
    last = _rms(x[torch.tensor([b - 1 for _, b in spans], device=DEVICE)], one + store.load_tensor(store.pre + "norm.weight").double(), c.rms_norm_eps)
    logits = last @ store.load_tensor(store.pre + "embed_tokens.weight" if c.tie_word_embeddings else "lm_head.weight").double().t()
    out, at = [], 0                                                 # laid out as the batches bring them
    for _, want in _batches(range(len(parts)), [[0] * n for _, n in parts]):
        rows = sum(len(w) for w in want)
        out += [logits[at:at + rows]] if rows else []
        at += rows
    return out
