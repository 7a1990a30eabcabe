"""Workloads that stand for what a program does with this framework, through the calls such a program makes.

A case is one pass of one kind of work on one model:

  step      one new token per row of a conversation that is under way: ids go up, the chosen ids come back (`call_host`, and
            `call` with a temperature where the token is sampled, as the chat loop does)
  prompt    a prompt of any length from position 0 (`forward`)
  request   a whole greedy request: the prompt in one call, then token after token (`generate`)

Models are the Llama sizes of `llama3.MODEL_PARAMS` with fp16, int8 or NF4 weights, and layer-list models in bf16 (Matulorn,
Rigazen) with the layer sizes of those Llamas.  Weights are random, made on the GPU from the seed.  The output matrix is the
embedding table, or that table moved on by one token, at a scale at which the stream still shows the token that went in: the
model is sure of its pick, as a trained one mostly is, so that ids do not hang on the last bit of a logit.

`exact` restates the models in 64 bits in plain torch.
"""
from __future__ import annotations

import gc
import math
import zlib

import numpy as np
import torch

from denograd_b200 import rand
from denograd_b200.llama3 import MODEL_PARAMS, Llama3
from denograd_b200.matulorn import Matulorn
from denograd_b200.nn import get_state_dict
from denograd_b200.rigazen import Rigazen

STD = 0.02            # of every matrix
GATES = ("i", "f")
EMBED_RMS = {"llama": 4.0, "matulorn": 4.0, "rigazen": 4.0, "tied": 1.0}  # of an embedding row as it enters the stream


# ------------------------------------------------------------------------------------------------ the cases
def listed() -> list[dict]:
    def llama(name, task, size, batch, tokens, quant="float16", temperature=0.0):
        return {"name": name, "family": "llama", "task": task, "size": size, "quant": quant, "batch": batch, "tokens": tokens, "temperature": temperature}

    def layers(name, family, task, size, batch, tokens, new=0):
        return {"name": name, "family": family, "task": task, "size": size, "batch": batch, "tokens": tokens, "new": new}

    return [
        # one user chatting with the smallest model: a sampled token at the driver's default temperature (smallest call)
        llama("1B chat token", "step", "1B", 1, 67, temperature=0.95),
        # the benchmark's headline: greedy decode of the 8B, one row behind a 512-token prompt
        llama("8B token", "step", "8B", 1, 547),
        # a server decoding 32 conversations at once
        llama("8B 32 tokens", "step", "8B", 32, 517),
        # int8 weights, eight conversations of 2000 tokens
        llama("8B int8 8 tokens", "step", "8B", 8, 2011, "int8"),
        # NF4 weights, the option for little memory: one row
        llama("8B nf4 token", "step", "8B", 1, 37, "nf4"),
        # a short question to the smallest model: time to first token
        llama("1B prompt 45", "prompt", "1B", 1, 45),
        # the benchmark's prompt
        llama("8B prompt 512", "prompt", "8B", 1, 512),
        # long documents, int8 weights: two rows, more than one pass of rows (largest call)
        llama("8B int8 prompt 2x1900", "prompt", "8B", 2, 1900, "int8"),
        # layer-list models: a request from one user, and a prompt of about the longest single pass, of each design
        layers("Matulorn request", "matulorn", "request", "1B", 1, 93, 24),
        layers("Matulorn prompt 1999", "matulorn", "prompt", "8B", 1, 1999),
        layers("Rigazen request x8", "rigazen", "request", "1B", 8, 60, 24),
        layers("Rigazen prompt 1999", "rigazen", "prompt", "8B", 1, 1999),
    ]


def draw(rng) -> dict:
    """One more case of the same ranges: steps of 1 to 32 rows behind 16 to 4096 tokens, prompts of 16 to 2048 tokens in up to
    four rows, requests of up to eight rows."""
    def spread(lo: int, hi: int) -> int:
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    family = rng.choice(["llama", "llama", "llama", "matulorn", "rigazen"])
    task = rng.choice(["step", "prompt"] if family == "llama" else ["request", "prompt"])
    size = rng.choice(["1B", "3B", "8B"])
    if family == "llama":
        case = {"family": family, "task": task, "size": size, "quant": rng.choice(["float16", "float16", "int8", "int8", "nf4"]) if task == "step" else rng.choice(["float16", "int8"])}
        if task == "prompt":
            batch = rng.choice([1, 1, 2, 3, 4])
            return dict(case, batch=batch, tokens=spread(16, min(2048, 3800 // batch)), temperature=0.0)
        if case["quant"] == "nf4":  # its prompts go in token by token
            return dict(case, batch=spread(1, 4), tokens=spread(16, 64), temperature=0.0)
        batch = spread(1, 32)
        return dict(case, batch=batch, tokens=spread(16, min(4096, 24000 // batch)), temperature=rng.choice([0.0, 0.0, 0.95]))
    case = {"family": family, "task": task, "size": size}
    if task == "prompt":
        batch = rng.choice([1, 1, 2])
        return dict(case, batch=batch, tokens=spread(16, 2048 // batch), new=0)
    batch = spread(1, 8)
    return dict(case, batch=batch, tokens=spread(16, 1024 // batch), new=rng.randint(8, 14 if size == "8B" else 24))


# ------------------------------------------------------------------------------------------------ models
def layer_list(family: str, size: str) -> dict:
    """A layer-list configuration with the layer sizes of that Llama: of every four Matulorn layers one latent attention, one
    minGRU and two gated delta; Rigazen layers take turns between mLSTM and window attention beside lightning attention."""
    p = MODEL_PARAMS[size]["args"]
    d, ff, L, H = p["dim"], p["hidden_dim"], p["n_layers"], p["dim"] // 128
    if family == "rigazen":
        window = {"heads": H, "kv_heads": H // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 4096, "keep_first": 64},
                  "rot": {"base": 500000.0, "dims": 128}}
        linear = {"heads": H, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** (-1 - 8.0 * (i + 1) / H) for i in range(H)]}
        mixers = [{"type": "mlstm", "mixer": {"heads": d // 512, "dim": 256, "vdim": 512, "gate_cap": 15.0}},
                  {"type": "parallel", "mixer": {"left": window, "right": linear, "left_scale": 0.8, "right_scale": 1.1}}]
        return {"architecture": "Rigazen", "width": d, "vocab": p["vocab_size"], "norm": {"eps": 1e-6}, "embedding": {"scale": d ** 0.5},
                "token_side": {"dim": 256}, "layers": [dict(mixers[i % 2], mlp={"kind": "dense", "ff": ff}) for i in range(L)]}
    rot = {"base": 500000.0, "dims": 64, "scaling": {"factor": 4.0, "original": 8192, "fast": 32.0, "slow": 1.0}}
    latent = {"heads": H, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "mask": {"size": 4096}, "rot": rot, "scale": 192 ** -0.5}
    delta = {"heads": H, "kv_heads": H // 2, "dim": 128, "vdim": 128, "conv": 4}
    mixers = [{"type": "latent_attention", "mixer": latent}, {"type": "delta", "mixer": delta}, {"type": "mingru", "mixer": {"width": d}},
              {"type": "delta", "mixer": delta}]
    return {"architecture": "Matulorn", "width": d, "vocab": p["vocab_size"], "norm": {"eps": 1e-6, "groups": 4},
            "layers": [dict(mixers[i % 4], mlp={"kind": "dense", "ff": ff, "limit": 7.0}) for i in range(L)]}


def shapes(case: dict) -> dict[str, tuple]:
    """The values of the model's tensors: name -> shape of the matrix or vector that it stands for."""
    p = MODEL_PARAMS[case["size"]]["args"]
    d, ff, V = p["dim"], p["hidden_dim"], p["vocab_size"]
    s: dict[str, tuple] = {}
    if case["family"] == "llama":
        kv = d // p["n_heads"] * p["n_kv_heads"]
        s["tok_embeddings.weight"], s["norm.weight"] = (V, d), (d,)
        if not MODEL_PARAMS[case["size"]]["tied"]:
            s["output.weight"] = (V, d)
        for i in range(p["n_layers"]):
            for n, shape in (("attention.wq", (d, d)), ("attention.wk", (kv, d)), ("attention.wv", (kv, d)), ("attention.wo", (d, d)),
                             ("feed_forward.w1", (ff, d)), ("feed_forward.w2", (d, ff)), ("feed_forward.w3", (ff, d)),
                             ("attention_norm", (d,)), ("ffn_norm", (d,))):
                s[f"layers.{i}.{n}.weight"] = shape
        return s
    c = layer_list(case["family"], case["size"])
    s["embed"], s["final.norm"] = (V, d), (d,)
    if case["family"] == "matulorn":
        s["head"] = (V, d)
    else:
        n = c["token_side"]["dim"]
        s["side.embed"] = (V, n * len(c["layers"]))
    for i, lc in enumerate(c["layers"]):
        L, M, m = f"l{i}.", f"l{i}.mix.", lc["mixer"]
        if case["family"] == "matulorn":
            s.update({L + n: (d,) for n in ("norm1", "norm1b", "norm2", "norm2b")})
            s.update({L + "mlp.gate": (ff, d), L + "mlp.gate.b": (ff,), L + "mlp.up": (ff, d), L + "mlp.up.b": (ff,), L + "mlp.down": (d, ff), L + "mlp.down.b": (d,)})
        else:
            s.update({L + "norm1": (d,), L + "norm2": (d,), L + "mlp.up": (ff, d), L + "mlp.down": (d, ff)})
            s.update({L + "side.gate": (n, d), L + "side.proj": (d, n), L + "side.norm": (d,)})
        if lc["type"] == "mingru":
            W = m["width"]
            s.update({M + "z": (W, d), M + "x": (W, d), M + "g": (W, d), M + "z.b": (W,), M + "x.b": (W,), M + "o": (d, W)})
        elif lc["type"] == "latent_attention":
            H = m["heads"]
            s.update({M + "q": (H * (m["dim"] + m["rot_dim"]), d), M + "dkv": (m["kv_rank"] + m["rot_dim"], d), M + "dkv.norm": (m["kv_rank"],),
                      M + "uk": (H * m["dim"], m["kv_rank"]), M + "uv": (H * m["vdim"], m["kv_rank"]), M + "sink": (H,), M + "o": (d, H * m["vdim"])})
        elif lc["type"] == "delta":
            H, G = m["heads"], m["kv_heads"]
            for n2, ch in (("q", G * m["dim"]), ("k", G * m["dim"]), ("v", H * m["vdim"])):
                s[M + n2], s[M + n2 + ".conv"] = (ch, d), (ch, m["conv"])
            s.update({M + "b": (H, d), M + "a": (H, d), M + "A_log": (H,), M + "dt_bias": (H,), M + "norm": (m["vdim"],), M + "g": (H * m["vdim"], d), M + "o": (d, H * m["vdim"])})
        else:
            r, Q = (m, M) if lc["type"] == "mlstm" else (m["right"], M + "right.")
            H, qk, v = r["heads"], r["heads"] * r["dim"], r["heads"] * r["vdim"]
            s.update({Q + "q": (qk, d), Q + "k": (qk, d), Q + "v": (v, d), Q + "g": (v, d), Q + "o": (d, v), Q + "norm": (v,)})
            if lc["type"] == "mlstm":
                s.update({M + "i": (H, d), M + "i.b": (H,), M + "f": (H, d), M + "f.b": (H,)})
            else:
                a, P = m["left"], M + "left."
                for n2, rows in (("q", a["heads"] * a["dim"]), ("k", a["kv_heads"] * a["dim"]), ("v", a["kv_heads"] * a["vdim"])):
                    s[P + n2], s[P + n2 + ".b"] = (rows, d), (rows,)
                    if n2 != "v":
                        s[P + n2 + ".norm"] = (rows,)
                s[P + "o"] = (d, a["heads"] * a["vdim"])
    return s


def generator(seed: int, name: str) -> torch.Generator:
    return torch.Generator("cuda").manual_seed(seed * 1_000_003 + zlib.crc32(name.encode()))


def normal(shape, std, seed, name, dtype):
    return torch.empty(shape, dtype=dtype, device="cuda").normal_(0.0, std, generator=generator(seed, name))


def uniform(shape, seed, name):
    return torch.rand(shape, device="cuda", generator=generator(seed, name))


def values(case: dict, seed: int, name: str) -> dict[str, torch.Tensor]:
    """What the checkpoint holds under this name: {"": values}, for quantised matrices {"weight", "scale"}."""
    shape = shapes(case)[name]
    leaf, quant = name.rsplit(".", 1)[-1], case.get("quant")
    tied = case["family"] == "llama" and MODEL_PARAMS[case["size"]]["tied"]
    if case["family"] == "llama":
        if len(shape) == 1:
            return {"": torch.ones(shape, dtype=torch.float16, device="cuda")}
        source, std = name, STD
        if name == "tok_embeddings.weight":
            std = EMBED_RMS["tied" if tied else "llama"]
        elif name == "output.weight":
            source = "tok_embeddings.weight"
        if quant == "int8":
            q = torch.randint(-127, 128, shape, dtype=torch.int8, device="cuda", generator=generator(seed, source))
            scale = (0.5 + uniform(shape[:1], seed, source + ".scale")) * (std / 73.3)
            if name == "output.weight":
                q, scale = q.roll(1, 0), scale.roll(1, 0)
            return {"weight": q, "scale": scale.half()}
        if quant == "nf4" and name.startswith("layers."):  # two codes per byte; blocks of 64 around a largest value of 2.4 deviations
            n = shape[0] * shape[1]
            codes = torch.randint(0, 256, (n // 2,), dtype=torch.uint8, device="cuda", generator=generator(seed, name))
            return {"weight": codes, "scale": ((0.8 + 0.4 * uniform((n // 64, 1), seed, name + ".scale")) * (2.4 * STD)).half()}
        w = normal(shape, std if source == name else STD, seed, source, torch.float16)
        return {"": w.roll(1, 0) if name == "output.weight" else w}
    if len(shape) == 2 and leaf != "conv":
        if name == "embed":
            rms = EMBED_RMS[case["family"]]
            return {"": normal(shape, rms if case["family"] == "matulorn" else rms / shape[1] ** 0.5, seed, name, torch.bfloat16)}
        if name == "head":
            return {"": normal(shape, STD, seed, "embed", torch.bfloat16).roll(1, 0)}
        if case["family"] == "rigazen" and name.endswith(".mix.k"):
            # a token's own key and query agree: the norm behind the recurrence would make anything of a first read-out near zero
            w = 0.6 * normal(shape, STD, seed, name[:-1] + "q", torch.bfloat16) + 0.8 * normal(shape, STD, seed, name, torch.bfloat16)
            return {"": w}
        # the exponential gates read a stream that no norm has scaled: a tenth, so that they stay near one as trained ones do
        return {"": normal(shape, STD / 10 if leaf in GATES else STD, seed, name, torch.bfloat16)}
    if "norm" in leaf:  # some are stored around zero
        around_zero = case["family"] == "rigazen" and (leaf in ("norm1", "norm2") or name == "final.norm")
        return {"": torch.full(shape, 0.0 if around_zero else 1.0, device="cuda")}
    u = uniform(shape, seed, name)
    if name.endswith(".f.b"):  # a state that is mostly kept
        return {"": 2.0 + u}
    return {"": torch.log(0.02 + u) if leaf == "A_log" else u - 0.25 if leaf == "conv" else 0.2 * (u - 0.5)}


class Memory:
    """Device memory of the framework as torch sees it; holds on to its owner."""

    TYPES = {"float16": "<f2", "float32": "<f4", "int8": "|i1", "uint8": "|u1", "int32": "<i4", "bfloat16": "<i2"}

    def __init__(self, owner, ptr: int, shape, dtype: str, ld: int | None = None):
        self.owner = owner
        size = int(self.TYPES[dtype][2])
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": self.TYPES[dtype], "data": (ptr, False), "version": 3,
                                         "strides": (ld * size, size) if ld and ld != shape[-1] else None}


def seen(owner, ptr, shape, dtype, ld=None) -> torch.Tensor:
    t = torch.as_tensor(Memory(owner, ptr, shape, dtype, ld), device="cuda")
    return t.view(torch.bfloat16) if dtype == "bfloat16" else t


def tokens_of(case: dict, seed: int, n: int) -> np.ndarray:
    V = MODEL_PARAMS[case["size"]]["args"]["vocab_size"]
    return np.random.RandomState(seed % (1 << 31)).randint(0, V, (case["batch"], n)).astype(np.int32)


def build(case: dict, seed: int):
    gc.collect()  # models of before give their memory back
    room = (case["tokens"] + case.get("new", 0) + 8 + 63) // 64 * 64
    if case["family"] == "llama":
        llm = Llama3(size=case["size"], quantize=case["quant"], max_context=room, max_batch=case["batch"], temperature=case["temperature"])
        there = get_state_dict(llm.model)
        for name in shapes(case):
            for part, v in values(case, seed, name).items():
                t = there[name if part in ("", "weight") else name.replace(".weight", ".scale")]
                seen(t, t.ptr, t.shape, t.dtype).copy_(v.reshape(t.shape))
    else:
        llm = {"matulorn": Matulorn, "rigazen": Rigazen}[case["family"]](layer_list(case["family"], case["size"]), max_context=room, max_batch=case["batch"], temperature=0.0)
        for name in shapes(case):
            q, v = llm.model.params[name], values(case, seed, name)[""]
            seen(q.tensor, q.ptr, q.shape, q.tensor.dtype, q.ld).copy_(v + q.offset if q.offset else v)
    torch.cuda.synchronize()
    return llm


# ------------------------------------------------------------------------------------------------ one pass
def prepare(case: dict, seed: int) -> dict:
    llm, toks = build(case, seed), tokens_of(case, seed, case["tokens"] + 1)
    V = MODEL_PARAMS[case["size"]]["args"]["vocab_size"]
    s = {"llm": llm, "case": case, "prompt": np.ascontiguousarray(toks[:, :-1]), "token": np.ascontiguousarray(toks[:, -1:]), "pos": case["tokens"], "seed": seed}
    logits = llm.model._workspace(case["batch"]).logits
    s["logits"] = seen(logits, logits.ptr, (case["batch"], V), logits.dtype)
    if case["task"] == "step":  # a conversation under way: its context is in the cache, its first tokens have been made
        llm.model.forward(s["prompt"], 0)
        for _ in range(2):
            llm.model.call_host(s["token"], s["pos"])
    return s


def run(s: dict) -> dict:
    llm, case = s["llm"], s["case"]
    if case["task"] == "step":
        if case["temperature"] > 0:
            rand.manual_seed(s["seed"])
            ids = llm.model.call(s["token"], s["pos"], llm.temperature, llm.top_k, llm.top_p, llm.alpha_f, llm.alpha_p).numpy()
        else:
            ids = llm.model.call_host(s["token"], s["pos"])
        return {"ids": ids, "logits": s["logits"]}
    if case["task"] == "prompt":
        ids = llm.model.forward(s["prompt"], 0)
        return {"ids": seen(ids, ids.ptr, ids.shape, ids.dtype), "logits": s["logits"]}
    llm.reset()
    return {"ids": llm.generate(s["prompt"], case["new"], batched=True), "logits": s["logits"]}


# ------------------------------------------------------------------------------------------------ work and tolerance
def work(case: dict) -> dict:
    """Every weight once per model call, what is cached of the tokens before it (or the recurrent state) once, logits written;
    multiplications of every token with every matrix, of causal attention and of state updates."""
    p = MODEL_PARAMS[case["size"]]["args"]
    V, B = p["vocab_size"], case["batch"]
    size = {"int8": 1.0, "nf4": 0.5 + 2.0 / 64}.get(case.get("quant"), 2.0)
    matrices = [(n, s) for n, s in shapes(case).items() if len(s) == 2 and not n.endswith(".conv") and "embed" not in n]
    inner = sum(s[0] * s[1] for n, s in matrices if n not in ("output.weight", "head"))
    head = V * p["dim"]
    weights = inner * size + head * (1.0 if case.get("quant") == "int8" else 2.0)
    T = case["tokens"]
    cached, state, attn, mix = 0.0, 0.0, 0.0, 0.0  # bytes per cached token, bytes of state, flops per pair of tokens, flops of a token's state
    if case["family"] == "llama":
        hd = p["dim"] // p["n_heads"]
        cached, attn = 4.0 * p["n_layers"] * p["n_kv_heads"] * hd, 4.0 * p["n_layers"] * p["dim"]
    else:
        for lc in layer_list(case["family"], case["size"])["layers"]:
            m = lc["mixer"]
            if lc["type"] == "latent_attention":
                cached, attn = cached + 2.0 * (m["kv_rank"] + m["rot_dim"]), attn + 2.0 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
            elif lc["type"] == "mingru":
                state += 8.0 * m["width"]
            else:
                r = m.get("right", m)
                state, mix = state + 8.0 * r["heads"] * r["dim"] * r["vdim"], mix + (8.0 if lc["type"] == "delta" else 4.0) * r["heads"] * r["dim"] * r["vdim"]
                if "left" in m:
                    a = m["left"]
                    cached, attn = cached + 2.0 * a["kv_heads"] * (a["dim"] + a["vdim"]), attn + 2.0 * a["heads"] * (a["dim"] + a["vdim"])
    width = 2.0 if case["family"] == "llama" else 4.0

    def call(n: int, before: int) -> tuple[float, float]:
        by = weights + B * (cached * (before + n) + state + V * width + 2.0 * n * p["dim"])
        return by, B * (2.0 * n * inner + 2.0 * head + attn * n * (before + (n + 1) / 2.0) + mix * n)

    calls = [call(1, T)] if case["task"] == "step" else [call(T, 0)] + [call(1, T + i) for i in range(max(case.get("new", 0) - 1, 0))]
    return {"bytes": sum(c[0] for c in calls), "flops": sum(c[1] for c in calls)}


def tolerance(case: dict) -> dict:
    """Logits; ids are whole numbers and stay the same."""
    return {"rel": 0.03 if case["family"] != "llama" else 0.015, "max": 0.3, "differ": 0.0}


# ------------------------------------------------------------------------------------------------ 64 bits
D = torch.float64
CODES = (-1.0, -0.6961928009986877, -0.5250730514526367, -0.39491748809814453, -0.28444138169288635, -0.18477343022823334, -0.09105003625154495, 0.0,
         0.07958029955625534, 0.16093020141124725, 0.24611230194568634, 0.33791524171829224, 0.44070982933044434, 0.5626170039176941, 0.7229568362236023, 1.0)


class Weights:
    def __init__(self, case: dict, seed: int, prefix: str = ""):
        self.case, self.seed, self.prefix = case, seed, prefix

    def sub(self, prefix: str) -> "Weights":
        return Weights(self.case, self.seed, self.prefix + prefix)

    def __getitem__(self, name: str) -> torch.Tensor:
        name = self.prefix + name
        v = values(self.case, self.seed, name)
        if "" in v:
            return v[""].to(D)
        if v["weight"].dtype == torch.int8:
            return v["weight"].to(D) * v["scale"].to(D)[:, None]
        codes = torch.stack([v["weight"] >> 4, v["weight"] & 15], -1).reshape(-1, 64).long()
        return (torch.tensor(CODES, dtype=D, device="cuda").half().to(D)[codes] * v["scale"].to(D)).reshape(shapes(self.case)[name])


def rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def causal(q, k, v, scale, sink=None):
    """Heads of one sequence [H, T, .]: softmax over the tokens so far, and a sink's weight where one is given."""
    T = q.shape[1]
    out = torch.empty(q.shape[0], T, v.shape[2], dtype=D, device="cuda")
    hidden = torch.ones(T, T, dtype=torch.bool, device="cuda").triu_(1)
    for h in range(q.shape[0]):
        g = h * k.shape[0] // q.shape[0]
        s = (q[h] @ k[g].T * scale).masked_fill_(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], 1)
        out[h] = torch.softmax(s, 1)[:, :T] @ v[g]
    return out


def heads(x, H):  # [T, H * n] -> [H, T, n]
    return x.reshape(x.shape[0], H, -1).transpose(0, 1)


def each_row(x, f):
    return torch.stack([f(r) for r in x])


def turn_pairs(x, theta):
    """Rotary on neighbouring entries of [H, T, n]."""
    T, n = x.shape[1:]
    a = torch.arange(T, dtype=D, device="cuda")[:, None] * theta ** (-torch.arange(0, n, 2, dtype=D, device="cuda") / n)
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * a.cos() - v * a.sin(), u * a.sin() + v * a.cos()], -1).reshape(x.shape)


def turn_halves(x, freqs, gain=1.0):
    """Rotary on entries n / 2 apart of [H, T, n]."""
    a = torch.arange(x.shape[1], dtype=D, device="cuda")[:, None] * freqs
    u, v = x.chunk(2, -1)
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1) * gain


def llama_stream(case, w, toks):
    p = MODEL_PARAMS[case["size"]]["args"]
    H, G, eps = p["n_heads"], p["n_kv_heads"], p["norm_eps"]
    x = w["tok_embeddings.weight"][toks]
    for i in range(p["n_layers"]):
        l = w.sub(f"layers.{i}.")
        h = rms(x, eps) * l["attention_norm.weight"]
        q, k, v = (h @ l[f"attention.{n}.weight"].T for n in ("wq", "wk", "wv"))
        a = torch.stack([causal(turn_pairs(heads(q[b], H), p["rope_theta"]), turn_pairs(heads(k[b], G), p["rope_theta"]), heads(v[b], G),
                                (p["dim"] // H) ** -0.5).transpose(0, 1).reshape(x.shape[1], -1) for b in range(len(x))])
        x = x + a @ l["attention.wo.weight"].T
        h = rms(x, eps) * l["ffn_norm.weight"]
        x = x + (torch.nn.functional.silu(h @ l["feed_forward.w1.weight"].T) * (h @ l["feed_forward.w3.weight"].T)) @ l["feed_forward.w2.weight"].T
    tied = MODEL_PARAMS[case["size"]]["tied"]
    return rms(x[:, -1], eps) * w["norm.weight"], w["tok_embeddings.weight" if tied else "output.weight"]


def mingru(h, w, m, eps):
    z, u, g = torch.sigmoid(h @ w["z"].T + w["z.b"]), h @ w["x"].T + w["x.b"], torch.nn.functional.silu(h @ w["g"].T)
    c = torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
    s, out = torch.zeros_like(z[:, 0]), torch.empty_like(z)
    for t in range(z.shape[1]):
        s = s + z[:, t] * (c[:, t] - s)
        out[:, t] = s
    return out * g @ w["o"].T


def latent_attention(h, w, m, eps):
    H, r, rot = m["heads"], m["kv_rank"], m["rot"]
    n, sc = rot["dims"], rot["scaling"]
    i = torch.arange(n // 2, dtype=D, device="cuda")
    f = rot["base"] ** (-2 * i / n)
    at = [n * math.log(sc["original"] / (2 * math.pi * t)) / (2 * math.log(rot["base"])) for t in (sc["fast"], sc["slow"])]
    lo, hi = max(math.floor(at[0]), 0), min(math.ceil(at[1]), n - 1)
    blend = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    f, gain = f / sc["factor"] * blend + f * (1 - blend), 0.1 * math.log(sc["factor"]) + 1
    q, c = h @ w["q"].T, h @ w["dkv"].T
    lat = rms(c[..., :r], eps) * w["dkv.norm"]
    kn, v, sink = lat @ w["uk"].T, lat @ w["uv"].T, w["sink"]

    def row(b):
        qh = heads(q[b], H)
        qh = torch.cat([qh[..., :m["dim"]], turn_halves(qh[..., m["dim"]:], f, gain)], -1)
        kr = turn_halves(c[b, :, r:][None], f, gain).expand(H, -1, -1)
        return causal(qh, torch.cat([heads(kn[b], H), kr], -1), heads(v[b], H), m["scale"], sink).transpose(0, 1).reshape(h.shape[1], -1)

    assert h.shape[1] <= m["mask"]["size"]
    return torch.stack([row(b) for b in range(len(h))]) @ w["o"].T


def delta(h, w, m, eps):
    H, G, n, v = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    B, T, _ = h.shape

    def conv(name):
        x, taps = h @ w[name].T, w[name + ".conv"]
        y = torch.zeros_like(x)
        for j in range(taps.shape[1]):
            back = taps.shape[1] - 1 - j
            y[:, back:] += taps[:, j] * x[:, :T - back]
        return torch.nn.functional.silu(y)

    q, k = (conv(c).reshape(B, T, G, n) for c in "qk")
    q, k = (x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
    q, k = q.repeat_interleave(H // G, 2) * n ** -0.5, k.repeat_interleave(H // G, 2)
    val, beta = conv("v").reshape(B, T, H, v), torch.sigmoid(h @ w["b"].T)
    decay = torch.exp(-torch.exp(w["A_log"]) * torch.nn.functional.softplus(h @ w["a"].T + w["dt_bias"]))
    S, out = torch.zeros(B, H, n, v, dtype=D, device="cuda"), torch.empty(B, T, H, v, dtype=D, device="cuda")
    for t in range(T):
        S = S * decay[:, t, :, None, None]
        u = beta[:, t, :, None] * (val[:, t] - (k[:, t, :, None] @ S)[:, :, 0])
        S = S + k[:, t, :, :, None] * u[:, :, None]
        out[:, t] = (q[:, t, :, None] @ S)[:, :, 0]
    g = torch.nn.functional.silu(h @ w["g"].T).reshape(out.shape)
    return (rms(out, eps) * w["norm"] * g).reshape(B, T, -1) @ w["o"].T


def matulorn_stream(case, w, toks):
    c = layer_list("matulorn", case["size"])
    eps, groups = c["norm"]["eps"], c["norm"]["groups"]

    def norm(x, g):
        return rms(x.reshape(x.shape[:-1] + (groups, -1)), eps).reshape(x.shape) * g

    x = w["embed"][toks]
    for i, lc in enumerate(c["layers"]):
        l, kind, lim = w.sub(f"l{i}."), {"mingru": mingru, "latent_attention": latent_attention, "delta": delta}[lc["type"]], lc["mlp"]["limit"]
        x = x + norm(kind(norm(x, l["norm1"]), l.sub("mix."), lc["mixer"], eps), l["norm1b"])
        h = norm(x, l["norm2"])
        g, u = (h @ l["mlp.gate"].T + l["mlp.gate.b"]).clamp(max=lim), (h @ l["mlp.up"].T + l["mlp.up.b"]).clamp(-lim, lim)
        x = x + norm((g * torch.sigmoid(1.702 * g) * (u + 1)) @ l["mlp.down"].T + l["mlp.down.b"], l["norm2b"])
    return norm(x[:, -1], w["final.norm"]), w["head"]


def mlstm(h, w, m, eps):
    H, n, v, cap = m["heads"], m["dim"], m["vdim"], m["gate_cap"]
    B, T, _ = h.shape
    q, k, val = ((h @ w[c].T).reshape(B, T, H, -1) for c in "qkv")
    q = q * n ** -0.5
    gi, gf = (cap * torch.tanh((h @ w[c].T + w[c + ".b"]) / cap) for c in "if")
    gf = torch.nn.functional.logsigmoid(gf)
    S, N, M = torch.zeros(B, H, n, v, dtype=D, device="cuda"), torch.zeros(B, H, n, dtype=D, device="cuda"), torch.zeros(B, H, dtype=D, device="cuda")
    out = torch.empty(B, T, H, v, dtype=D, device="cuda")
    for t in range(T):
        new = torch.maximum(gf[:, t] + M, gi[:, t])
        keep, put = torch.exp(gf[:, t] + M - new)[..., None], torch.exp(gi[:, t] - new)[..., None] * k[:, t]
        S = keep[..., None] * S + put[..., None] * val[:, t, :, None]
        N, M = keep * N + put, new
        over = torch.maximum((N * q[:, t]).sum(-1).abs(), torch.exp(-new)) + 1e-6
        out[:, t] = (q[:, t, :, None] @ S)[:, :, 0] / over[..., None]
    return (rms(out, eps).reshape(B, T, -1) * w["norm"] * torch.sigmoid(h @ w["g"].T)) @ w["o"].T


def window_attention(h, w, m, eps):
    H, G, dims = m["heads"], m["kv_heads"], m["rot"]["dims"]
    q, k, v = (h @ w[c].T + w[c + ".b"] for c in "qkv")
    q, k = rms(q, eps) * w["q.norm"], rms(k, eps) * w["k.norm"]
    f = m["rot"]["base"] ** (-torch.arange(0, dims, 2, dtype=D, device="cuda") / dims)
    assert h.shape[1] <= m["mask"]["size"] and dims == m["dim"]
    a = torch.stack([causal(turn_halves(heads(q[b], H), f), turn_halves(heads(k[b], G), f), heads(v[b], G), m["scale"]).transpose(0, 1).reshape(h.shape[1], -1)
                     for b in range(len(h))])
    return a @ w["o"].T


def lightning(h, w, m, eps):
    H, B, T = m["heads"], h.shape[0], h.shape[1]
    q, k, v = (torch.nn.functional.silu(h @ w[c].T).reshape(B, T, H, -1) for c in "qkv")
    decay = torch.tensor(m["decay"], dtype=torch.float32).to("cuda", D)[:, None, None]
    S, out = torch.zeros(B, H, m["dim"], m["vdim"], dtype=D, device="cuda"), torch.empty_like(v)
    for t in range(T):
        S = decay * S + k[:, t, :, :, None] * v[:, t, :, None]
        out[:, t] = (q[:, t, :, None] @ S)[:, :, 0]
    return (rms(out.reshape(B, T, -1), eps) * w["norm"] * torch.sigmoid(h @ w["g"].T)) @ w["o"].T


def rigazen_stream(case, w, toks):
    c = layer_list("rigazen", case["size"])
    eps, n = c["norm"]["eps"], c["token_side"]["dim"]
    x = w["embed"][toks] * c["embedding"]["scale"]
    side = values(w.case, w.seed, "side.embed")[""][toks].to(D)
    for i, lc in enumerate(c["layers"]):
        l, m, mix = w.sub(f"l{i}."), lc["mixer"], w.sub(f"l{i}.mix.")
        if lc["type"] == "mlstm":
            y = mlstm(x, mix, m, eps)
        else:
            y = m["left_scale"] * window_attention(x, mix.sub("left."), m["left"], eps) + m["right_scale"] * lightning(x, mix.sub("right."), m["right"], eps)
        x = x + rms(y, eps) * (1 + l["norm1"])
        x = x + rms(torch.relu(x @ l["mlp.up"].T) ** 2 @ l["mlp.down"].T, eps) * (1 + l["norm2"])
        gate = torch.nn.functional.gelu(x @ l["side.gate"].T, approximate="tanh")
        x = x + rms((gate * side[..., i * n:(i + 1) * n]) @ l["side.proj"].T, eps) * l["side.norm"]
    return rms(x[:, -1], eps) * (1 + w["final.norm"]), w["embed"]


def exact(case: dict, seed: int):
    toks = tokens_of(case, seed, case["tokens"] + 1)
    if case["task"] != "step":
        toks = toks[:, :-1]
    V = MODEL_PARAMS[case["size"]]["args"]["vocab_size"]
    for _ in range(case.get("new", 0) - 1):  # the token after each pick: the same one, or the next
        toks = np.concatenate([toks, (toks[:, -1:] + (case["family"] != "rigazen")) % V], 1)
    rows = torch.from_numpy(toks).long().cuda()
    if rows.numel() * MODEL_PARAMS[case["size"]]["args"]["n_layers"] > 700_000:
        return None
    stream = {"llama": llama_stream, "matulorn": matulorn_stream, "rigazen": rigazen_stream}[case["family"]]
    x, head = stream(case, Weights(case, seed), rows)
    return {"ids": None, "logits": x @ head.T}
