"""The work that a user of this framework has it do, through its public entry points, for timing one version against another.

What each kind of case stands for:

    graph     GPT-2 forward + tied head captured for one shape and replayed (``GraphedForward``): serving one request or one
              rank's share of a batch
    score     per-token cross-entropy of a batch (``FusedGPT.token_nll``), the logits never written: evaluation of a corpus
    logits    GPT-2 logits and greedy ids, launched call by call
    hidden    final hidden states (``FusedGPT.forward``), fp32 storage included
    generate  a whole request through a session: prompt, then token by token; the logits behind the last token come along
    prompt    the prompt pass of a session and the logits behind it, for the decoders with bounded memory
    attention the causal attention operator on its own

Weights are random with the spread of trained ones where that decides how the path behaves: the embedding rows are long
enough against what the layers add that the next token has a clear margin (GPT-2's head is tied: it repeats; the other two
have a permuted copy of the embeddings as head), so greedy ids do not hang on the last bit of a logit.
"""

import math

import torch

from gpt_triton_b200 import kernels as K
from gpt_triton_b200.fogilix import Fogilix
from gpt_triton_b200.generation import GenerationSession
from gpt_triton_b200.gpt import FusedGPT, GPTConfig, GraphedForward
from gpt_triton_b200.nufasun import Nufasun

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}
# GPT-2 small and medium; block_size is the position table
GPT2 = {"124m": (12, 12, 768), "355m": (24, 16, 1024)}
GPT2_VOCAB, GPT2_CONTEXT = 50257, 1024
# width -> layers, latent size, window of the two decoders with bounded memory
DECODERS = {1024: (8, 256, 512), 2048: (8, 512, 1024), 4096: (4, 512, 1024)}
VOCAB = 32768


def listed():
    return [
        # one short prompt: 87 small launches, latency only
        {"name": "gpt2-1x37", "kind": "graph", "model": "124m", "dtype": "fp16", "batch": 1, "n": 37},
        # one of eight ranks' share of the 512 x 300 benchmark batch
        {"name": "gpt2-64x300", "kind": "graph", "model": "124m", "dtype": "fp16", "batch": 64, "n": 300},
        # the benchmark batch itself, scored
        {"name": "gpt2-score-512x300", "kind": "score", "model": "124m", "dtype": "fp16", "batch": 512, "n": 300},
        # long sequences, the medium model
        {"name": "gpt2-355m-16x1024", "kind": "logits", "model": "355m", "dtype": "bf16", "batch": 16, "n": 1024},
        # fp32 storage (operands rounded to fp16 as in the reference): feature extraction
        {"name": "gpt2-fp32-16x300", "kind": "hidden", "model": "124m", "dtype": "fp32", "batch": 16, "n": 300},
        # a few interactive requests, greedy
        {"name": "gpt2-generate-8", "kind": "generate", "model": "124m", "dtype": "fp16", "batch": 8, "n": 300, "new": 64, "temperature": 0.0, "top_k": 0},
        # many sequences, sampled
        {"name": "gpt2-generate-256", "kind": "generate", "model": "124m", "dtype": "bf16", "batch": 256, "n": 300, "new": 32, "temperature": 0.8, "top_k": 50},
        # one long prompt
        {"name": "fogilix-prompt-1x4096", "kind": "prompt", "model": "fogilix", "dtype": "bf16", "width": 1024, "batch": 1, "n": 4096},
        # a serving batch
        {"name": "fogilix-generate-16", "kind": "generate", "model": "fogilix", "dtype": "bf16", "width": 2048, "batch": 16, "n": 512, "new": 64,
         "temperature": 0.0, "top_k": 0},
        # many long prompts
        {"name": "nufasun-prompt-16x2048", "kind": "prompt", "model": "nufasun", "dtype": "bf16", "width": 1024, "batch": 16, "n": 2048, "passes": 1},
        # one interactive request of ragged length
        {"name": "nufasun-generate-1", "kind": "generate", "model": "nufasun", "dtype": "bf16", "width": 2048, "batch": 1, "n": 333, "new": 64, "passes": 1,
         "temperature": 0.0, "top_k": 0},
        # the operator of the kernel sweep, a tensor per argument
        {"name": "attention-16x12x2048x64", "kind": "attention", "dtype": "fp16", "batch": 16, "heads": 12, "n": 2048, "dim": 64},
    ]


def draw(rng):
    def size(lo, hi):
        return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    kind = rng.choice(["graph", "score", "logits", "hidden", "generate", "generate", "prompt", "prompt", "attention"])
    if kind == "graph":
        n = size(8, 512)
        return {"kind": kind, "model": "124m", "dtype": rng.choice(["fp16", "bf16"]), "batch": size(1, min(64, max(1, 19200 // n))), "n": n}
    if kind == "score":
        n = size(64, GPT2_CONTEXT)
        return {"kind": kind, "model": "124m", "dtype": rng.choice(["fp16", "bf16"]), "batch": size(4, min(512, 131072 // n)), "n": n}
    if kind == "logits":
        n, model = size(16, GPT2_CONTEXT), rng.choice(["124m", "355m"])
        return {"kind": kind, "model": model, "dtype": rng.choice(["fp16", "bf16"]), "batch": size(1, max(1, 16384 // n)), "n": n}
    if kind == "hidden":
        n = size(16, GPT2_CONTEXT)
        return {"kind": kind, "model": "124m", "dtype": rng.choice(["fp32", "fp16"]), "batch": size(1, max(1, 8192 // n)), "n": n}
    if kind == "attention":
        n, dim = size(64, 2048), rng.choice([32, 64, 64, 128])
        return {"kind": kind, "dtype": rng.choice(["fp16", "bf16"]), "batch": size(1, max(1, 16384 // n)), "heads": rng.choice([4, 12, 16, 25]), "n": n, "dim": dim}
    model = rng.choice(["124m", "fogilix", "nufasun"]) if kind == "generate" else rng.choice(["fogilix", "nufasun"])
    case = {"kind": kind, "model": model, "dtype": "bf16"}
    if model == "124m":
        case["dtype"] = rng.choice(["fp16", "bf16"])
    else:
        case["width"] = rng.choice([1024, 1024, 2048]) if kind == "prompt" else rng.choice([1024, 2048, 4096])
    if model == "nufasun":
        case["passes"] = rng.choice([1, 1, 2])
    if kind == "prompt":
        n = size(65, 4096)
        return {**case, "batch": size(1, max(1, min(16, 16384 // n))), "n": n}
    n = size(17, 512)
    sampled = model == "124m" and rng.random() < 0.4
    return {**case, "batch": size(1, min(256 if model == "124m" else 128, 32768 // n)), "n": n, "new": rng.randint(12, 24),
            "temperature": 0.8 if sampled else 0.0, "top_k": 50 if sampled else 0}


# ----------------------------------------------------------------------------- weights and configurations
def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _generator(seed, stream):
    return torch.Generator(device=_device()).manual_seed(1000003 * (seed + 1) + stream)


class _Draws:
    """Normal tensors, rounded to the storage type."""

    def __init__(self, seed, stream, dtype):
        self.g, self.dtype = _generator(seed, stream), dtype

    def __call__(self, *shape, std=1.0, mean=0.0):
        return torch.randn(shape, generator=self.g, device=_device()).mul_(std).add_(mean).to(self.dtype)


def _gpt_weights(case, seed):
    layers, _, h = GPT2[case["model"]]
    r = _Draws(seed, 1, DTYPES[case["dtype"]])
    out = {"wte_weight": r(GPT2_VOCAB, h, std=0.14), "wpe_weight": r(GPT2_CONTEXT, h, std=0.02)}

    def norm(stem):
        return {stem + "layer_norm_weight": r(h, std=0.1, mean=1.0), stem + "layer_norm_bias": r(h, std=0.02)}

    def linear(stem, k, n, std):
        return {stem + "_weight": r(k, n, std=std), stem + "_bias": r(n, std=0.02)}

    deep = 0.02 / math.sqrt(2 * layers)
    for i in range(layers):
        a, m = f"blocks.{i}.0.", f"blocks.{i}.1."
        out |= norm(a) | linear(a + "c_attn", h, 3 * h, 0.02) | linear(a + "c_proj", h, h, deep)
        out |= norm(m) | linear(m + "ffn1", h, 4 * h, 0.02) | linear(m + "ffn2", 4 * h, h, deep)
    return out | norm("")


def _decoder_config(case):
    """Recurrent and window-attention layers in turn, feed-forwards everywhere."""
    width = case["width"]
    layers, rank, window = DECODERS[width]
    heads, out, owner = width // 128, [], None
    for i in range(layers):
        if case["model"] == "fogilix":
            mlp = {"kind": "dense", "ff": 4 * width}
            if i % 2 == 0:
                decay = [1.0 - 2.0 ** -(3 + 7 * h / max(heads - 1, 1)) for h in range(heads)]
                out.append({"type": "lightning", "mixer": {"heads": heads, "dim": 128, "vdim": 128, "decay": decay}, "mlp": mlp})
                continue
            mixer = {"heads": heads, "dim": 128, "vdim": 128, "kv_rank": rank, "mask": {"size": window}, "scale": 128 ** -0.5}
            if owner is None:
                owner = i
            else:
                mixer["kv_from"], owner = owner, None
            out.append({"type": "latent_attention", "mixer": mixer, "mlp": mlp})
            continue
        mlp = {"kind": "dense", "ff": round(8 * width / 3 / 64) * 64, "limit": 7.0}
        if i % 2 == 0:
            out.append({"type": "delta", "mixer": {"heads": heads, "kv_heads": heads // 2, "dim": 128, "vdim": 128, "conv": 4}, "mlp": mlp})
        else:
            mixer = {"heads": heads, "kv_heads": heads // 4, "dim": 64, "vdim": 128, "mask": {"size": window}, "diff": 0.6, "softcap": 30.0, "scale": 0.125,
                     "rot": {"base": 1e5, "dims": 64}}
            out.append({"type": "attention", "mixer": mixer, "mlp": mlp})
    if case["model"] == "fogilix":
        return {"architecture": "Fogilix", "vocab": VOCAB, "width": width, "layers": out, "norm": {"eps": 1e-5}, "logit_scale": 1.0}
    return {"architecture": "Nufasun", "vocab": VOCAB, "width": width, "layers": out, "norm": {"eps": 1e-6}, "embedding": {"scale": 1.0}, "logit_softcap": 30.0,
            "loop": {"start": 2, "stop": 4, "times": case["passes"]}}


def _decoder_weights(case, seed):
    cfg, w = _decoder_config(case), case["width"]
    r = _Draws(seed, 2, DTYPES[case["dtype"]])
    nufasun = case["model"] == "nufasun"

    def mat(n, k, s=1.0):
        return r(n, k, std=s / k ** 0.5)

    def gain(n, at=1.0, s=0.1):
        return r(n, std=s, mean=at)

    embed = r(VOCAB, w)
    successor = torch.randperm(VOCAB, generator=_generator(seed, 3), device=_device())
    head = torch.empty_like(embed)
    head[successor] = (embed.float() * w ** -0.5).to(embed.dtype)  # the token behind v scores high where v stands
    out = {"embed": embed, "head": head, "final.norm": gain(w, 1.0 if nufasun else 0.0)}
    if nufasun:
        out["loop.step"] = r(case["passes"], w, std=0.2)
    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], f"l{i}."
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        ff = layer["mlp"]["ff"]
        if not nufasun:
            out |= {p + "norm1": gain(w, 0.0), p + "norm2": gain(w, 0.0), p + "mlp.up": mat(ff, w), p + "mlp.down": mat(w, ff), p + "mix.q": mat(H * d, w)}
            out[p + "mix.o"] = mat(w, H * dv)
            if layer["type"] == "lightning":
                out |= {p + "mix.k": mat(H * d, w), p + "mix.v": mat(H * dv, w), p + "mix.g": mat(H * dv, w), p + "mix.norm": gain(H * dv)}
            else:
                out |= {p + "mix.uk": mat(H * d, m["kv_rank"]), p + "mix.uv": mat(H * dv, m["kv_rank"]), p + "mix.sink": r(H)}
                if "kv_from" not in m:
                    out |= {p + "mix.dkv": mat(m["kv_rank"], w), p + "mix.dkv.norm": gain(m["kv_rank"])}
            continue
        G = m["kv_heads"]
        out |= {p + "norm1": gain(w), p + "norm2": gain(w), p + "norm1b": gain(w, 0.4), p + "norm2b": gain(w, 0.4), p + "mix.o": mat(w, H * dv)}
        out |= {p + "mlp.gate": mat(ff, w), p + "mlp.up": mat(ff, w), p + "mlp.down": mat(w, ff), p + "mlp.gate.b": r(ff, std=0.1), p + "mlp.up.b": r(ff, std=0.1),
                p + "mlp.down.b": r(w, std=0.1)}
        if layer["type"] == "delta":
            out |= {p + "mix.q": mat(G * d, w), p + "mix.k": mat(G * d, w), p + "mix.v": mat(H * dv, w), p + "mix.g": mat(H * dv, w), p + "mix.a": mat(H, w),
                    p + "mix.b": mat(H, w), p + "mix.A_log": r(H, std=1.0, mean=-1.5), p + "mix.dt_bias": r(H, mean=-1.0), p + "mix.norm": gain(dv)}
            out |= {p + f"mix.{x}.conv": mat(n, m["conv"]) for x, n in (("q", G * d), ("k", G * d), ("v", H * dv))}
        else:
            out |= {p + "mix.q": mat(2 * H * d, w), p + "mix.k": mat(2 * G * d, w), p + "mix.v": mat(G * dv, w), p + "mix.g": mat(H, w), p + "mix.q.norm": gain(d),
                    p + "mix.k.norm": gain(d)}
            out |= {p + "mix." + x: r(d, std=0.1) for x in ("lq1", "lk1", "lq2", "lk2")}
    return out


def _weights(case, seed):
    return _gpt_weights(case, seed) if case["model"] in GPT2 else _decoder_weights(case, seed)


def _model(case, seed):
    with torch.device(_device()):
        if case["model"] in GPT2:
            layers, heads, h = GPT2[case["model"]]
            model = FusedGPT(GPTConfig(vocab_size=GPT2_VOCAB, block_size=GPT2_CONTEXT, n_layer=layers, n_head=heads, n_embd=h))
            model.load_state_dict(_weights(case, seed))
        else:
            model = {"fogilix": Fogilix, "nufasun": Nufasun}[case["model"]].from_checkpoint(_decoder_config(case), _weights(case, seed))
    return model.to(DTYPES[case["dtype"]]).eval()


def _ids(case, seed):
    vocab = GPT2_VOCAB if case["model"] in GPT2 else VOCAB
    return torch.randint(0, vocab, (case["batch"], case["n"]), generator=_generator(seed, 4), device=_device())


def _targets(ids):
    return ids.roll(-1, dims=1)  # the next token; the last one is scored against the first


def _qkv(case, seed):
    r = _Draws(seed, 5, DTYPES[case["dtype"]])
    return [r(case["batch"], case["heads"], case["n"], case["dim"]) for _ in range(3)]


# ----------------------------------------------------------------------------- the calls
def prepare(case, seed):
    kind = case["kind"]
    if kind == "attention":
        return {"kind": kind, "qkv": _qkv(case, seed)}
    model, ids = _model(case, seed), _ids(case, seed)
    state = {"kind": kind, "model": model, "ids": ids}
    if kind == "graph":
        state["forward"] = GraphedForward(model, ids, what="logits_and_next_ids")
    elif kind == "score":
        state["targets"] = _targets(ids)
    elif kind == "prompt":
        state["session"] = GenerationSession(model, case["batch"], capacity=case["n"] + 1)
    elif kind == "generate":
        state["new"] = case["new"]
        state["session"] = GenerationSession(model, case["batch"], capacity=case["n"] + case["new"], max_new_tokens=case["new"],
                                             temperature=case["temperature"], top_k=case["top_k"], seed=seed)
        state["session"].generate(ids[:, :8].contiguous(), min(8, case["new"]))  # a first request: the decode step is captured in it
    return state


@torch.no_grad()
def run(state):
    kind = state["kind"]
    if kind == "attention":
        return K.flash_attention_v1(*state["qkv"])
    model, ids = state["model"], state["ids"]
    if kind == "graph":
        logits, nxt = state["forward"](ids)
        return {"logits": logits, "ids": nxt}
    if kind == "score":
        return model.token_nll(ids, state["targets"])
    if kind == "logits":
        logits, nxt = model.logits_and_next_ids(ids)
        return {"logits": logits, "ids": nxt}
    if kind == "hidden":
        return model(ids)
    session = state["session"]
    if kind == "prompt":
        session.reset()
        return model.head_logits(session.extend(ids))
    tokens = session.generate(ids, state["new"])
    rows = session.extend(tokens[:, -1:].contiguous())
    return {"tokens": tokens, "logits": model.head_logits(rows)}


# ----------------------------------------------------------------------------- what a pass cannot do without
def _weight_count(case):
    """(weights of the layers' products, weights of the head)"""
    if case["model"] in GPT2:
        layers, _, h = GPT2[case["model"]]
        return 12 * h * h * layers, GPT2_VOCAB * h
    cfg, w, total = _decoder_config(case), case["width"], 0
    for i, layer in enumerate(cfg["layers"]):
        m = layer["mixer"]
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        ff = layer["mlp"]["ff"]
        if case["model"] == "fogilix":
            n = 2 * w * ff + w * H * dv
            n += w * 2 * H * (d + dv) if layer["type"] == "lightning" else w * H * d + m["kv_rank"] * (H * (d + dv) + (0 if "kv_from" in m else w))
        else:
            G = m["kv_heads"]
            n = 3 * w * ff + w * H * dv
            n += w * (2 * G * d + 2 * H * dv + 2 * H) if layer["type"] == "delta" else w * (2 * H * d + G * (2 * d + dv) + H)
            loop = cfg["loop"]
            n *= loop["times"] if loop["start"] <= i < loop["stop"] else 1
        total += n
    return total, VOCAB * w


def _pairs(first, count, window):
    """(query, key) pairs of `count` tokens behind `first` earlier ones."""
    return sum(min(first + i + 1, window) for i in range(count))


def _mixing(case, first, count):
    """(flops, bytes of what is remembered) of the layers' mixing for `count` tokens of one sequence behind `first`."""
    size = 4 if case["dtype"] == "fp32" else 2
    if case["model"] in GPT2:
        layers, _, h = GPT2[case["model"]]
        return 4.0 * layers * h * _pairs(first, count, 1 << 30), 2.0 * size * layers * h * (first + count)
    flops = memory = 0.0
    for layer in _decoder_config(case)["layers"]:
        m = layer["mixer"]
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        if "mask" in m:
            win = m["mask"]["size"]
            maps, per_key = (1, m["kv_rank"]) if case["model"] == "fogilix" else (2, m["kv_heads"] * (2 * d + dv))
            flops += 2.0 * maps * H * (d + dv) * _pairs(first, count, win)
            memory += size * per_key * min(first + count, win)
        else:
            flops += (4.0 if case["model"] == "fogilix" else 6.0) * H * d * dv * count
            memory += 8.0 * H * d * dv
    return flops, memory


def work(case):
    kind, B, n = case["kind"], case["batch"], case["n"]
    size = 4 if case["dtype"] == "fp32" else 2
    if kind == "attention":
        H, d = case["heads"], case["dim"]
        return {"bytes": 4.0 * size * B * H * n * d, "flops": 4.0 * B * H * d * _pairs(0, n, n)}
    body, head = _weight_count(case)
    T = B * n
    mix, memory = _mixing(case, 0, n)
    out = {"bytes": size * (body + 0.0), "flops": 2.0 * T * body + B * mix}
    vocab = GPT2_VOCAB if case["model"] in GPT2 else VOCAB
    out_size = 2 if case["model"] in GPT2 else 4
    if kind == "hidden":
        out["bytes"] += size * T * GPT2[case["model"]][2]
        return out
    scored = B if kind in ("prompt", "generate") else T
    out["bytes"] += size * head + 8.0 * T
    out["flops"] += 2.0 * scored * head
    if kind == "score":
        out["bytes"] += 12.0 * T
        return out
    out["bytes"] += out_size * float(scored) * vocab
    if kind in ("prompt", "generate"):
        out["bytes"] += B * memory
    if kind == "generate":
        for t in range(case["new"]):
            mix, memory = _mixing(case, n + t, 1)
            out["bytes"] += size * (body + head) + B * memory
            out["flops"] += B * (2.0 * (body + head) + mix)
    return out


def tolerance(case):
    """About four times the distance to 64-bit arithmetic that was measured, per storage type and depth of rounding."""
    if case["kind"] == "attention":
        return {"rel": 1e-3 if case["dtype"] == "fp16" else 8e-3, "max": 0.1}
    if case["kind"] == "score":
        return {"rel": 1e-3 if case["dtype"] == "fp16" else 1e-2, "max": 0.3}
    if case["dtype"] == "bf16":
        return {"rel": {"fogilix": 0.015, "nufasun": 0.025}.get(case["model"], 0.03), "max": 0.5, "differ": 0.01}
    return {"rel": 4e-3 if case["dtype"] == "fp16" else 2e-3, "max": 0.1, "differ": 0.01}


# ----------------------------------------------------------------------------- the same in 64 bits
def _layer_norm(x, w, b):
    x = x - x.mean(-1, keepdim=True)
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * w + b


def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _gelu(x):
    return 0.5 * x * (1 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x ** 3)))


def _causal(q, k, v, window=None, sink=None, scale=None, cap=None):
    """q, k (..., n, d), v (..., n, dv) of one sequence, head by head."""
    n = q.shape[-2]
    s = q @ k.transpose(-1, -2) * (q.shape[-1] ** -0.5 if scale is None else scale)
    if cap is not None:
        s = cap * torch.tanh(s / cap)
    age = torch.arange(n, device=q.device)[:, None] - torch.arange(n, device=q.device)[None, :]
    s.masked_fill_((age < 0) | (age >= (window or n)), -math.inf)
    if sink is None:
        return torch.softmax(s, -1) @ v
    top = torch.maximum(s.amax(-1, keepdim=True), sink.view(-1, 1, 1))
    e = torch.exp(s - top)
    return e @ v / (e.sum(-1, keepdim=True) + torch.exp(sink.view(-1, 1, 1) - top))


def _gpt_hidden(case, W, ids):
    layers, heads, h = GPT2[case["model"]]
    B, n = ids.shape
    x = W["wte_weight"][ids] + W["wpe_weight"][:n]
    for i in range(layers):
        a, m = f"blocks.{i}.0.", f"blocks.{i}.1."
        y = _layer_norm(x, W[a + "layer_norm_weight"], W[a + "layer_norm_bias"]) @ W[a + "c_attn_weight"] + W[a + "c_attn_bias"]
        q, k, v = (t.view(B, n, heads, h // heads).transpose(1, 2) for t in y.split(h, dim=-1))
        x = x + _causal(q, k, v).transpose(1, 2).reshape(B, n, h) @ W[a + "c_proj_weight"] + W[a + "c_proj_bias"]
        y = _gelu(_layer_norm(x, W[m + "layer_norm_weight"], W[m + "layer_norm_bias"]) @ W[m + "ffn1_weight"] + W[m + "ffn1_bias"])
        x = x + y @ W[m + "ffn2_weight"] + W[m + "ffn2_bias"]
    return _layer_norm(x, W["layer_norm_weight"], W["layer_norm_bias"])


def _heads(x, heads):
    return x.view(*x.shape[:2], heads, -1)


def _lightning(h, p, m, eps):
    q, k, v = (_heads(torch.nn.functional.silu(h @ p[x].T), m["heads"]) for x in "qkv")
    decay = torch.tensor(m["decay"], dtype=h.dtype, device=h.device)[:, None, None]
    s = torch.zeros((h.shape[0], m["heads"], m["dim"], m["vdim"]), dtype=h.dtype, device=h.device)
    o = torch.empty_like(v)
    for t in range(h.shape[1]):
        s.mul_(decay).addcmul_(k[:, t, :, :, None], v[:, t, :, None, :])
        o[:, t] = (q[:, t, :, None, :] @ s)[..., 0, :]
    return (_rms(o.flatten(2), p["norm"], eps) * torch.sigmoid(h @ p["g"].T)) @ p["o"].T


def _latent_attention(h, c, p, m):
    q, k, v = (_heads(x, m["heads"]).transpose(1, 2) for x in (h @ p["q"].T, c @ p["uk"].T, c @ p["uv"].T))
    y = torch.stack([_causal(q[b], k[b], v[b], m["mask"]["size"], p["sink"], m["scale"]) for b in range(h.shape[0])])
    return y.transpose(1, 2).flatten(2) @ p["o"].T


def _rotated(x, base, dims):
    """x (batch, n, heads, d): neighbouring columns turn by position * base^(-2i / dims)."""
    i = torch.arange(dims // 2, dtype=torch.float64, device=x.device)
    angle = torch.arange(x.shape[1], dtype=torch.float64, device=x.device)[:, None] * base ** (-2 * i / dims)
    c, s = torch.cos(angle)[:, None, :], torch.sin(angle)[:, None, :]
    u, v = x[..., 0:dims:2], x[..., 1:dims:2]
    out = x.clone()
    out[..., 0:dims:2], out[..., 1:dims:2] = u * c - v * s, v * c + u * s
    return out


def _differential(h, p, m, eps):
    H, G, d = m["heads"], m["kv_heads"], m["dim"]
    q = _rotated(_rms(_heads(h @ p["q"].T, 2 * H), p["q.norm"], eps), m["rot"]["base"], m["rot"]["dims"])
    k = _rotated(_rms(_heads(h @ p["k"].T, 2 * G), p["k.norm"], eps), m["rot"]["base"], m["rot"]["dims"])
    v = _heads(h @ p["v"].T, G)
    lam = torch.exp((p["lq1"] * p["lk1"]).sum()) - torch.exp((p["lq2"] * p["lk2"]).sum()) + m["diff"]
    out = []
    for b in range(h.shape[0]):
        vb = v[b].transpose(0, 1).repeat_interleave(H // G, 0)
        a = []
        for i in range(2):
            qb, kb = q[b, :, i::2].transpose(0, 1), k[b, :, i::2].transpose(0, 1).repeat_interleave(H // G, 0)
            a.append(_causal(qb, kb, vb, m["mask"]["size"], None, m["scale"], m["softcap"]))
        out.append(_rms(a[0] - lam * a[1], 1.0, eps).transpose(0, 1))
    y = torch.stack(out) * (1 - m["diff"]) * torch.sigmoid(h @ p["g"].T)[..., None]
    return y.flatten(2) @ p["o"].T


def _delta(h, p, m, eps):
    H, G, d, taps = m["heads"], m["kv_heads"], m["dim"], m["conv"]
    silu = torch.nn.functional.silu

    def conv(name):
        x = torch.nn.functional.pad(h @ p[name].T, (0, 0, taps - 1, 0))
        return silu(sum(x[:, t:t + h.shape[1]] * p[name + ".conv"][:, t] for t in range(taps)))

    def unit(x):
        return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)

    q, k = (unit(_heads(conv(x), G)).repeat_interleave(H // G, dim=2) for x in "qk")
    v = _heads(conv("v"), H)
    beta = torch.sigmoid(h @ p["b"].T)
    decay = torch.exp(-torch.exp(p["A_log"]) * torch.nn.functional.softplus(h @ p["a"].T + p["dt_bias"], threshold=100.0))
    s = torch.zeros((h.shape[0], H, d, m["vdim"]), dtype=h.dtype, device=h.device)
    o = torch.empty_like(v)
    for t in range(h.shape[1]):
        s.mul_(decay[:, t, :, None, None])
        u = beta[:, t, :, None] * (v[:, t] - (k[:, t, :, None, :] @ s)[..., 0, :])
        s.addcmul_(k[:, t, :, :, None], u[:, :, None, :])
        o[:, t] = (q[:, t, :, None, :] @ s)[..., 0, :]
    return (_rms(o * d ** -0.5, p["norm"], eps) * silu(_heads(h @ p["g"].T, H))).flatten(2) @ p["o"].T


def _decoder_rows(case, W, ids):
    """Rows behind the final norm (batch, n, width)."""
    cfg = _decoder_config(case)
    eps, nufasun = cfg["norm"]["eps"], case["model"] == "nufasun"
    x = start = W["embed"][ids]
    latents = {}
    order = [(i, None) for i in range(len(cfg["layers"]))]
    if nufasun:
        a, b = cfg["loop"]["start"], cfg["loop"]["stop"]
        order = order[:a] + [(i, t if i == a else None) for t in range(cfg["loop"]["times"]) for i in range(a, b)] + order[b:]
    for i, entered in order:
        layer = cfg["layers"][i]
        m, pre = layer["mixer"], f"l{i}."
        p = {k[len(pre) + 4:]: t for k, t in W.items() if k.startswith(pre + "mix.")}
        if not nufasun:
            h = _rms(x, 1 + W[pre + "norm1"], eps)
            if layer["type"] == "lightning":
                x = x + _lightning(h, p, m, eps)
            else:
                if "kv_from" not in m:
                    latents[i] = _rms(h @ p["dkv"].T, p["dkv.norm"], eps)
                x = x + _latent_attention(h, latents[m.get("kv_from", i)], p, m)
            x = x + _gelu(_rms(x, 1 + W[pre + "norm2"], eps) @ W[pre + "mlp.up"].T) @ W[pre + "mlp.down"].T
            continue
        if entered is not None:
            x = x + W["loop.step"][entered] + (start if entered > 0 else 0)
        h = _rms(x, W[pre + "norm1"], eps)
        x = x + _rms((_delta if layer["type"] == "delta" else _differential)(h, p, m, eps), W[pre + "norm1b"], eps)
        h, limit = _rms(x, W[pre + "norm2"], eps), layer["mlp"]["limit"]
        g = torch.clamp(h @ W[pre + "mlp.gate"].T + W[pre + "mlp.gate.b"], max=limit)
        u = torch.clamp(h @ W[pre + "mlp.up"].T + W[pre + "mlp.up.b"], -limit, limit)
        x = x + _rms((g * torch.sigmoid(1.702 * g) * (u + 1)) @ W[pre + "mlp.down"].T + W[pre + "mlp.down.b"], W[pre + "norm2b"], eps)
    return _rms(x, W["final.norm"] + (0 if nufasun else 1), eps)


def _exact_rows(case, W, ids):
    """Rows in front of the head, a few sequences at a time."""
    run_one = _gpt_hidden if case["model"] in GPT2 else _decoder_rows
    step = max(1, (16384 if case["model"] in GPT2 else 32768) // ids.shape[1])
    return torch.cat([run_one(case, W, part) for part in ids.split(step)])


def _exact_head(case, W, rows):
    if case["model"] in GPT2:
        return rows @ W["wte_weight"].T
    z = rows @ W["head"].T
    return 30.0 * torch.tanh(z / 30.0) if case["model"] == "nufasun" else z


@torch.no_grad()
def exact(case, seed):
    kind = case["kind"]
    if kind == "attention":
        q, k, v = _qkv(case, seed)
        return torch.stack([_causal(*(t[b].double() for t in (q, k, v))) for b in range(case["batch"])])
    W = {k: v.double() for k, v in _weights(case, seed).items()}
    ids = _ids(case, seed)
    B, n = ids.shape
    if kind == "hidden":
        return _exact_rows(case, W, ids)
    if kind == "prompt":
        return _exact_head(case, W, _exact_rows(case, W, ids)[:, -1])
    if kind == "score":
        out = []
        for rows, target in zip(_exact_rows(case, W, ids).flatten(0, 1).split(8192), _targets(ids).reshape(-1).split(8192)):
            z = _exact_head(case, W, rows)
            out.append(torch.logsumexp(z, -1) - z.gather(1, target[:, None])[:, 0])
        return torch.cat(out).view(B, n)
    if kind in ("graph", "logits"):
        logits = _exact_head(case, W, _exact_rows(case, W, ids))
        return {"logits": logits, "ids": logits.argmax(-1)}
    # Greedy continuation without one pass per token: guess it, run the whole sequences, take over what the guess got wrong
    # and everything behind it, until nothing changes.  (Sampled cases: every margin is far above what sampling bridges.)
    new = case["new"]
    seen = torch.cat([ids, ids[:, -1:].expand(B, new)], dim=1)
    if case["model"] not in GPT2:
        chain, token = [], ids[:, -1]
        successor = torch.randperm(VOCAB, generator=_generator(seed, 3), device=_device())
        for _ in range(new):
            token = successor[token]
            chain.append(token)
        seen = torch.cat([ids, torch.stack(chain, dim=1)], dim=1)
    for _ in range(4):
        logits = _exact_head(case, W, _exact_rows(case, W, seen)[:, n - 1:])
        picked = logits.argmax(-1)
        if torch.equal(picked[:, :new], seen[:, n:]):
            return {"tokens": picked[:, :new], "logits": logits[:, new]}
        seen = torch.cat([ids, picked[:, :new]], dim=1)
    return None
