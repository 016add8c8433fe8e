"""The cases that this library's speed is judged by: whole requests, from token ids to token ids and logits.

A case is a model shape (the Llama shapes and decoder sizes of bench.py, the tiny test model), how many sequences
come together, how long their prompts are, how many tokens are generated for each, the dtype and the sampling.  One
pass is what a serving program does with such a batch: take slots, run all prompts in one step, generate the tokens
as `LLM.generate` does (captured decode steps, the device one step ahead of the host), ask for the logits behind the
last token, give the slots back.  Without generated tokens a pass is the prompt step and its logits alone.

Weights are seeded random numbers with what matters of trained ones: residual branches that add up to about the
embedding's size, a head that is sure of the next token (so that rounding does not send two correct runs down
different texts), experts chosen by the token and not by a coin's throw, decays of recurrences between fast and slow.
"""
from __future__ import annotations

import math
import zlib

import numpy as np
import torch
import torch.nn.functional as F

import cpp_minilamma_b200 as ml
from cpp_minilamma_b200 import api

# --------------------------------------------------------------------------------------------------- #
# model shapes                                                                                         #
# --------------------------------------------------------------------------------------------------- #
_LLAMA3 = {"rope_type": "llama3", "low_freq_factor": 1.0, "high_freq_factor": 4.0}
_LLAMA = {
    "llama31_8b": dict(vocab_size=128256, hidden_size=4096, intermediate_size=14336, num_hidden_layers=32,
                       num_attention_heads=32, num_key_value_heads=8, head_dim=128, max_position_embeddings=131072,
                       rope_theta=500000.0, rope_scaling=dict(_LLAMA3, factor=8.0, original_max_position_embeddings=8192),
                       rms_norm_eps=1e-5, tie_word_embeddings=False),
    "llama2_7b": dict(vocab_size=32000, hidden_size=4096, intermediate_size=11008, num_hidden_layers=32,
                      num_attention_heads=32, num_key_value_heads=32, head_dim=128, max_position_embeddings=4096,
                      rope_theta=10000.0, rope_scaling=None, rms_norm_eps=1e-5, tie_word_embeddings=False),
    "llama32_1b": dict(vocab_size=128256, hidden_size=2048, intermediate_size=8192, num_hidden_layers=16,
                       num_attention_heads=32, num_key_value_heads=8, head_dim=64, max_position_embeddings=131072,
                       rope_theta=500000.0, rope_scaling=dict(_LLAMA3, factor=32.0, original_max_position_embeddings=8192),
                       rms_norm_eps=1e-5, tie_word_embeddings=True),
    "tiny": dict(vocab_size=257, hidden_size=192, intermediate_size=512, num_hidden_layers=3, num_attention_heads=6,
                 num_key_value_heads=1, head_dim=32, max_position_embeddings=256, rope_theta=500000.0,
                 rope_scaling=dict(_LLAMA3, factor=8.0, original_max_position_embeddings=32), rms_norm_eps=1e-6,
                 tie_word_embeddings=True),
}
_WIDTHS = {2048: dict(ff=8192, heads=16, kv_heads=4, chunk=1024, ret_heads=8),
           4096: dict(ff=14336, heads=32, kv_heads=8, chunk=2048, ret_heads=16)}


def _kupirax(width):
    """Chunked attention, retention and the gated delta rule, twice over, a dense feed-forward beside each."""
    s = _WIDTHS[width]
    mlp = {"kind": "dense", "ff": s["ff"]}
    group = [
        {"type": "attention", "mlp": mlp,
         "mixer": {"heads": s["heads"], "kv_heads": s["kv_heads"], "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                   "mask": {"size": s["chunk"]},
                   "rot": {"base": 500000.0, "dims": 64,
                           "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}},
        {"type": "retention", "mlp": mlp,
         "mixer": {"heads": s["ret_heads"], "dim": 128, "vdim": 256, "rot": {"base": 10000.0, "dims": 128},
                   "decay": [1.0 - 2.0 ** (-5 - 4 * i / s["ret_heads"]) for i in range(s["ret_heads"])]}},
        {"type": "channel_delta", "mlp": mlp,
         "mixer": {"heads": s["heads"], "kv_heads": s["heads"], "dim": 128, "vdim": 128, "conv": 4, "decay_rank": 64,
                   "gate_rank": 64}}]
    return {"architecture": "Kupirax", "vocab": 32000, "width": width, "norm": {"eps": 1e-6}, "layers": group * 2}


def _badolix(width):
    """Window attention with capped scores (one layer on an earlier one's keys), latent attention and a state-space
    mixer; dense feed-forwards with biases and 4 of 16 experts out of 2 of 4 groups take turns."""
    s = _WIDTHS[width]
    dense = {"kind": "dense", "ff": s["ff"]}
    moe = {"kind": "moe", "router": {"experts": 16, "top": 4, "groups": {"count": 4, "keep": 2}}, "expert": {"ff": s["ff"] // 4}}
    window = {"heads": s["heads"], "kv_heads": s["kv_heads"], "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 30.0,
              "mask": {"size": 1024, "keep_first": 64}, "rot": {"base": 500000.0, "dims": 128, "scaling": {"factor": 8.0}}}
    latent = {"heads": s["heads"], "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 192, "scale": 192 ** -0.5,
              "rot": {"base": 500000.0, "dims": 64, "scaling": {"factor": 8.0, "original": 8192, "fast": 16.0, "slow": 1.0}}}
    ssm = {"heads": 2 * width // 64, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8}
    layers = [{"type": "attention", "mixer": window, "mlp": dense},
              {"type": "attention", "mixer": dict(window, kv_from=0), "mlp": moe},
              {"type": "latent_attention", "mixer": latent, "mlp": dense},
              {"type": "mamba2", "mixer": ssm, "mlp": moe},
              {"type": "attention", "mixer": window, "mlp": dense},
              {"type": "latent_attention", "mixer": latent, "mlp": moe}]
    return {"architecture": "Badolix", "vocab": 32000, "width": width, "norm": {"eps": 1e-5}, "embedding": {"scale": 2.0},
            "residual_mult": 0.7, "logit_scale": 0.5, "layers": layers}


def _config(case):
    """The config.json of the case's model."""
    stored = {"torch_dtype": case["dtype"]}
    if case["model"] == "kupirax":
        return dict(_kupirax(case["width"]), **stored)
    if case["model"] == "badolix":
        return dict(_badolix(case["width"]), **stored)
    raw = dict(_LLAMA[case["model"]], architectures=["LlamaForCausalLM"], **stored)
    if case["layers"]:
        raw["num_hidden_layers"] = case["layers"]
    return raw


# --------------------------------------------------------------------------------------------------- #
# cases                                                                                                #
# --------------------------------------------------------------------------------------------------- #
def _case(model, sequences, shortest, longest, new, layers=0, width=0, dtype="bfloat16", temperature=0.0, top_k=0):
    return {"model": model, "layers": layers, "width": width, "dtype": dtype, "sequences": sequences,
            "shortest": shortest, "longest": longest, "new": new, "temperature": temperature, "top_k": top_k}


def listed():
    return [
        # the smallest model and calls, in true float32: what a test suite or a toy model runs; launches and host work
        dict(_case("tiny", 4, 1, 40, 12, dtype="float32"), name="tiny float32 batch 4"),
        # one user and a small model: the time per token of a chat turn
        dict(_case("llama32_1b", 1, 97, 97, 64), name="1B chat turn"),
        # the headline workload: 8 sequences with unequal prompts on the 8B shape
        dict(_case("llama31_8b", 8, 128, 2047, 48), name="8B batch 8"),
        # a busy server of a small model: many unequal sequences, sampled
        dict(_case("llama32_1b", 64, 64, 1023, 48, temperature=0.8, top_k=40), name="1B batch 64 sampled"),
        # a prompt's way to its first token on the 8B shape
        dict(_case("llama31_8b", 1, 2048, 2048, 0), name="8B prompt 2048"),
        # many short prompts of odd lengths in one step: classification, scoring, a queue that filled up
        dict(_case("llama32_1b", 37, 3, 511, 0), name="1B ragged prompts"),
        # a long document, cut into portions by the engine
        dict(_case("llama32_1b", 1, 16383, 16383, 0), name="1B long prompt"),
        # the true float32 path at a real width: checking a model's numbers
        dict(_case("llama32_1b", 3, 17, 300, 16, dtype="float32"), name="1B float32"),
        # the decoder of chunked attention, retention and delta rule: a prompt of odd length, then a batch that decodes
        dict(_case("kupirax", 1, 2047, 2047, 0, width=2048), name="Kupirax prompt"),
        dict(_case("kupirax", 16, 64, 700, 48, width=2048), name="Kupirax batch 16"),
        # the decoder of window and latent attention, state space and routed experts: a few prompts, then a batch
        dict(_case("badolix", 3, 600, 2047, 0, width=2048), name="Badolix prompts"),
        dict(_case("badolix", 24, 32, 500, 48, width=2048), name="Badolix batch 24"),
    ]


def _spread(rng, low, high):
    """A whole number between low and high, even over their logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """One more case of the same ranges: any model, one sequence to many, prompts of a few tokens to thousands, with
    and without generated tokens; the 8B and 7B shapes with 8 of their 32 layers, both widths of the other decoders."""
    model = rng.choice(["tiny", "llama32_1b", "llama32_1b", "llama32_1b", "llama31_8b", "llama31_8b", "llama2_7b",
                        "kupirax", "kupirax", "badolix", "badolix"])
    dtype = "float32" if model == "tiny" or (model == "llama32_1b" and rng.random() < 0.2) else "bfloat16"
    new = 0 if rng.random() < 0.4 else _spread(rng, 8, 48)
    sequences = _spread(rng, 1, 64)
    budget = 20000  # prompt tokens of a case
    top = 2047
    if model == "tiny":
        sequences, budget, top = min(sequences, 16), 2000, 200
    elif dtype == "float32":
        sequences, budget, top = min(sequences, 8), 1200, 700
    elif new == 0 and model != "llama2_7b":
        top = 4095
    longest = _spread(rng, 16, max(17, min(top, budget // sequences)))
    shortest = _spread(rng, 1, longest)
    sampled = new > 0 and rng.random() < 0.3
    return _case(model, sequences, shortest, longest, new, layers=8 if model in ("llama31_8b", "llama2_7b") else 0,
                 width=rng.choice([2048, 4096]) if model in ("kupirax", "badolix") else 0, dtype=dtype,
                 temperature=0.8 if sampled else 0.0, top_k=_spread(rng, 2, 200) if sampled and rng.random() < 0.7 else 0)


def _vocab(case):
    raw = _config(case)
    return raw.get("vocab_size") or raw["vocab"]


def _prompts(case, seed):
    """Token id lists; lengths follow from the case alone (so that its work does), ids from the seed."""
    n, lo, hi = case["sequences"], case["shortest"], case["longest"]
    lens = [hi] if n == 1 else [lo + (hi - lo) * i // (n - 1) for i in range(n)]
    np.random.RandomState(7).shuffle(lens)
    ids = np.random.RandomState(seed % (1 << 32))
    return [[int(t) for t in ids.randint(0, _vocab(case), size=length)] for length in lens]


# --------------------------------------------------------------------------------------------------- #
# weights                                                                                              #
# --------------------------------------------------------------------------------------------------- #
class _Weights:
    """Seeded weights by tensor name: the same values for the library (`prepare`) and for `exact`."""

    def __init__(self, case, seed, device):
        self.raw, self.seed, self.device = _config(case), int(seed), device
        self.dtype = torch.bfloat16 if case["dtype"] == "bfloat16" else torch.float32
        self.runs = self.raw.get("num_hidden_layers") or len(self.raw["layers"])
        self.embed_name = "model.embed_tokens.weight" if "hidden_size" in self.raw else "embed"
        self.width = self.raw.get("hidden_size") or self.raw["width"]
        self.vocab = self.raw.get("vocab_size") or self.raw["vocab"]
        self.tied = self.raw.get("tie_word_embeddings", self.raw.get("architecture") == "Badolix")
        self.routed = self.raw.get("architecture") == "Badolix"
        self._embed = None

    def _gen(self, name):
        return torch.Generator(device=self.device).manual_seed(self.seed * 1000003 + zlib.crc32(name.encode()))

    def follow(self):
        """[vocab]: the token that the head is sure of behind each token (a tied head: the same one again)."""
        if self.tied:
            return torch.arange(self.vocab, device=self.device)
        return torch.randperm(self.vocab, generator=self._gen("follow"), device=self.device)

    def _experts(self):
        """([16, width] unit directions that the routers read, [vocab, 4] the experts that each token asks for: two of
        each of two groups)."""
        gen = self._gen("experts")
        u = F.normalize(torch.randn((16, self.width), generator=gen, device=self.device), dim=1)
        groups = torch.rand((self.vocab, 4), generator=gen, device=self.device).argsort(1)[:, :2]
        inside = torch.rand((self.vocab, 2, 4), generator=gen, device=self.device).argsort(2)[:, :, :2]
        return u, (groups[:, :, None] * 4 + inside).reshape(self.vocab, 4)

    def __call__(self, name, shape):
        if name == "lm_head.weight" or name == "head":
            out = torch.empty(shape, device=self.device)
            out[self.follow()] = 0.02 * self(self.embed_name, shape).float()
            return out.to(self.dtype)
        if name.endswith("router"):
            return (0.5 * self._experts()[0]).to(self.dtype)
        gen = self._gen(name)
        if name.endswith("A_log"):
            return (1.0 + 15.0 * torch.rand(shape, generator=gen, device=self.device)).log().to(self.dtype)
        if name.endswith("dt_bias"):
            dt = torch.exp(math.log(1e-3) + math.log(100.0) * torch.rand(shape, generator=gen, device=self.device))
            return dt.expm1().log().to(self.dtype)
        out = torch.randn(shape, generator=gen, device=self.device)
        if name == self.embed_name:
            if self.routed:
                u, wanted = self._experts()
                for j in range(wanted.shape[1]):
                    out += 10.0 * u[wanted[:, j]]
            return out.to(self.dtype)
        if "norm" in name or name.endswith("mix.D"):
            out.mul_(0.1).add_(1.0)
            if self.tied and name in ("model.norm.weight", "final.norm"):
                out.mul_(0.04)  # logits of an ordinary size behind a head that is the embedding
        elif name.endswith(".conv"):
            out.mul_(0.5)
        elif name.endswith((".o", ".down", "o_proj.weight", "down_proj.weight")):
            out.mul_(0.02 / math.sqrt(2.0 * self.runs))
        else:
            out.mul_(0.02)
        return out.to(self.dtype)


# --------------------------------------------------------------------------------------------------- #
# one pass                                                                                             #
# --------------------------------------------------------------------------------------------------- #
def prepare(case, seed):
    device = torch.device("cuda:0")
    prompts = _prompts(case, seed)
    weights = _Weights(case, seed, device)
    config = ml.config_from_dict(_config(case))
    positions = -(-(case["longest"] + case["new"] + 1) // 64) * 64
    model = ml.build_model(config, case["dtype"], device, positions)
    model.bind({spec.name: weights(spec.name, tuple(spec.shape)).to(torch.float32 if spec.kind == "vector" else weights.dtype)
                for spec in model.weight_specs()})
    tokens = sum(-(-(len(p) + case["new"] + 1) // 64) * 64 for p in prompts)
    llm = api.LLM(config, model, max_tokens=tokens, max_seqs=case["sequences"])
    params = ml.SamplingParams(case["temperature"], case["top_k"], seed=1 + seed % 1000)
    return {"llm": llm, "backend": ml.EngineBackend(llm.engine, params), "prompts": prompts, "new": case["new"]}


def run(state):
    llm, backend, prompts, new = state["llm"], state["backend"], state["prompts"], state["new"]
    n = len(prompts)
    requests = list(range(n))
    slots = llm.engine.acquire(n)
    try:
        entries = [ml.StepEntry(slot, prompt, [len(prompt) - 1]) for slot, prompt in zip(slots, prompts)]
        if new == 0:
            return {"logits": llm.step(entries)}
        tokens = []
        ticket = backend.submit(entries, requests, [0] * n)
        for i in range(1, new):
            ahead = backend.submit_ahead(slots, requests, [i] * n)
            tokens.append(backend.collect(ticket))
            ticket = ahead
        tokens.append(backend.collect(ticket))
        logits = llm.step([ml.StepEntry(slot, [token], [0]) for slot, token in zip(slots, tokens[-1])])
        return {"tokens": np.asarray(tokens, dtype=np.int64), "logits": logits}
    finally:
        for slot in slots:
            llm.engine.release(slot)


# --------------------------------------------------------------------------------------------------- #
# what a pass cannot do without                                                                        #
# --------------------------------------------------------------------------------------------------- #
def _layer_sizes(case):
    """Per layer: (weights every token reads, keys' and values' columns of all query heads, bytes cached per position,
    most positions a token sees, floats of recurrent state, weights of one expert, experts, experts per token)."""
    raw = _config(case)
    size = 2 if case["dtype"] == "bfloat16" else 4
    if "hidden_size" in raw:
        D, H, G, d = raw["hidden_size"], raw["num_attention_heads"], raw["num_key_value_heads"], raw["head_dim"]
        weights = D * d * (2 * H + 2 * G) + 3 * D * raw["intermediate_size"]
        return [(weights, 2 * H * d, 2 * G * d * size, 1 << 30, 0, 0, 0, 0)] * raw["num_hidden_layers"]
    D, rows = raw["width"], []
    for layer in raw["layers"]:
        m, kind = layer["mixer"], layer["type"]
        H, dv = m["heads"], m["vdim"]
        columns = cached = state = 0
        seen = 1 << 30
        if kind == "attention":
            d, G = m["dim"], m["kv_heads"]
            own = 0 if m.get("kv_from") is not None else G * (d + dv)
            weights, columns, cached = D * (H * d + own + H * dv), H * (d + dv), G * (d + dv) * size
            seen = m["mask"]["size"] + m["mask"].get("keep_first", 0)
        elif kind == "latent_attention":
            row = m["kv_rank"] + m["rot_dim"]
            weights = D * (H * (m["dim"] + m["rot_dim"]) + row + H * dv) + m["kv_rank"] * H * (m["dim"] + dv)
            columns, cached = H * (m["dim"] + m["rot_dim"] + dv), row * size
        elif kind == "retention":
            weights, state = D * H * (2 * m["dim"] + 3 * dv), H * m["dim"] * dv
        elif kind == "channel_delta":
            weights = D * (2 * m["kv_heads"] * m["dim"] + 2 * H * dv + H + m["decay_rank"] + m["gate_rank"]) \
                + m["decay_rank"] * H * m["dim"] + m["gate_rank"] * H * dv
            state = H * m["dim"] * dv
        else:
            inner, gn = H * dv, m["groups"] * m["state"]
            weights, state = D * (3 * inner + 2 * gn + H), H * m["state"] * dv
        mlp = layer["mlp"]
        if mlp["kind"] == "dense":
            rows.append((weights + 3 * D * mlp["ff"], columns, cached, seen, state, 0, 0, 0))
        else:
            rows.append((weights + D * 16, columns, cached, seen, state, 3 * D * mlp["expert"]["ff"], 16, mlp["router"]["top"]))
    return rows


def work(case):
    """Every step reads each weight it uses once and the cached positions and states of its sequences once, and writes
    what it adds to them; logits of the wanted rows are written.  Products count two operations a weight and token."""
    size = 2 if case["dtype"] == "bfloat16" else 4
    raw = _config(case)
    D, vocab = raw.get("hidden_size") or raw["width"], _vocab(case)
    lens = [len(p) for p in _prompts(case, 0)]
    n, new = len(lens), case["new"]
    layers = _layer_sizes(case)
    moved = flops = 0.0
    for step in range(new + 1):
        tokens = sum(lens) if step == 0 else n
        moved += D * vocab * size + n * vocab * 4 + tokens * D * size
        flops += 2.0 * n * D * vocab
        for weights, columns, cached, seen, state, expert, experts, top in layers:
            moved += (weights + expert * min(experts, tokens * top)) * size + tokens * cached
            flops += 2.0 * tokens * (weights + expert * top) + 6.0 * tokens * state
            moved += n * state * 4 * (1 if step == 0 else 2)
            for length in lens:
                if step == 0:
                    edge = min(length, seen)
                    flops += 2.0 * columns * (edge * (edge + 1) / 2 + (length - edge) * seen)
                else:
                    flops += 2.0 * columns * min(length + step, seen)
                    moved += cached * min(length + step, seen)
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    """Logits: 32-bit sums (against 64 bits 1e-7 on the tiny model, 4.4e-7 on the 1B shape), or values rounded to bfloat16
    between the parts of every layer (7.2e-3 behind 32 layers of width 4,096, 3.3e-3 behind 16 of 2,048 and 6 of the
    Kupirax decoder, 7.6e-4 where residual branches are scaled down); about four times those.  Tokens: ties."""
    if case["dtype"] == "float32":
        return {"rel": 2e-6, "max": 5e-5, "differ": 0.01}
    rel = {"badolix": 0.003, "kupirax": 0.013, "llama32_1b": 0.013}.get(case["model"], 0.028)
    return {"rel": rel, "max": 15 * rel, "differ": 0.01}


# --------------------------------------------------------------------------------------------------- #
# the same in 64 bits                                                                                  #
# --------------------------------------------------------------------------------------------------- #
def _rms(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _frequencies(dims, base, scaling):
    """(frequencies [dims / 2], factor on cosine and sine)."""
    f = base ** (-2.0 * np.arange(dims // 2) / dims)
    if not scaling:
        return f, 1.0
    factor = scaling["factor"]
    low, high = scaling.get("low", scaling.get("low_freq_factor")), scaling.get("high", scaling.get("high_freq_factor"))
    original = scaling.get("original", scaling.get("original_max_position_embeddings"))
    if low is not None:  # by wavelength
        s = np.clip((original * f / (2.0 * math.pi) - low) / (high - low), 0.0, 1.0)
        return (1.0 - s) * f / factor + s * f, 1.0
    if original is None:  # all alike
        return f / factor, 1.0
    pair = lambda turns: dims * math.log(original / (2.0 * math.pi * turns)) / (2.0 * math.log(base))  # noqa: E731
    lo, hi = max(math.floor(pair(scaling["fast"])), 0), min(math.ceil(pair(scaling["slow"])), dims - 1)
    ramp = np.clip((np.arange(dims // 2) - lo) / max(hi - lo, 0.001), 0.0, 1.0)
    return f / factor * ramp + f * (1.0 - ramp), 0.1 * math.log(factor) + 1.0


def _rotate(x, dims, base, scaling, neighbours=False):
    """x [..., T, heads, d]: the first `dims` dimensions turned in pairs (i, i + dims / 2), or (2i, 2i + 1)."""
    f, magnitude = _frequencies(dims, base, scaling)
    angle = torch.arange(x.shape[-3], dtype=x.dtype, device=x.device)[:, None, None] * torch.from_numpy(f).to(x.device)
    c, s = angle.cos() * magnitude, angle.sin() * magnitude
    out = x.clone()
    a, b = (slice(0, dims, 2), slice(1, dims, 2)) if neighbours else (slice(0, dims // 2), slice(dims // 2, dims))
    out[..., a] = x[..., a] * c - x[..., b] * s
    out[..., b] = x[..., b] * c + x[..., a] * s
    return out


def _attend(q, k, v, scale, seen, cap=0.0):
    """q [B, T, H, d], k [B, T, G, d], v [B, T, G, dv]; seen(i, j): whether query i sees key j."""
    B, T, H, _ = q.shape
    G = k.shape[2]
    out = q.new_empty(B, T, H, v.shape[-1])
    j = torch.arange(T, device=q.device)
    for b in range(B):
        for at in range(0, T, 512):
            rows = q[b, at:at + 512]
            n = rows.shape[0]
            rows = rows.view(n, G, H // G, -1).permute(1, 2, 0, 3).reshape(G, H // G * n, -1)
            s = (rows @ k[b, :at + n].permute(1, 2, 0)).mul_(scale)
            if cap:
                s = cap * torch.tanh(s / cap)
            hidden = ~seen((at + torch.arange(n, device=q.device))[:, None], j[None, :at + n])
            s = s.view(G, H // G, n, -1).masked_fill_(hidden, -math.inf).softmax(-1).view(G, H // G * n, -1)
            o = s @ v[b, :at + n].permute(1, 0, 2)
            out[b, at:at + n] = o.view(G, H // G, n, -1).permute(2, 0, 1, 3).reshape(n, H, -1)
    return out.flatten(2)


def _convolve(x, taps):
    """x [B, T, C], taps [C, n], the last one on the current token."""
    out = x * taps[:, -1]
    for back in range(1, taps.shape[1]):
        out[:, back:] += x[:, :-back] * taps[:, -1 - back]
    return out


class _Plain:
    """The decoders in float64, whole padded sequences [B, T], no cache."""

    def __init__(self, case, seed, device):
        self.draw = _Weights(case, seed, device)
        self.raw = self.draw.raw

    def w(self, name, *shape):
        return self.draw(name, shape).double()

    def product(self, x, name, out):
        return x @ self.w(name, out, x.shape[-1]).T

    def norm(self, x, name, eps):
        return _rms(x, eps) * self.w(name, x.shape[-1])

    def swiglu(self, h, pre, post, ff, biased=False):
        D = h.shape[-1]
        gate, up = (self.product(h, pre + p + post, ff) for p in ("gate", "up"))
        if biased:
            gate, up = gate + self.w(pre + "gate.b", ff), up + self.w(pre + "up.b", ff)
        out = self.product(F.silu(gate).mul_(up), pre + "down" + post, D)
        return out + self.w(pre + "down.b", D) if biased else out

    # ---- the three decoders: tokens [B, T] -> the rows in front of the head -------------------------- #
    def llama(self, tokens):
        c = self.raw
        D, H, G, d, eps = c["hidden_size"], c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"], c["rms_norm_eps"]
        x = self.w("model.embed_tokens.weight", c["vocab_size"], D)[tokens]
        causal = lambda i, j: j <= i  # noqa: E731
        for layer in range(c["num_hidden_layers"]):
            pre = f"model.layers.{layer}."
            h = self.norm(x, pre + "input_layernorm.weight", eps)
            q, k, v = (self.product(h, f"{pre}self_attn.{p}_proj.weight", n * d).unflatten(-1, (n, d))
                       for p, n in (("q", H), ("k", G), ("v", G)))
            q, k = (_rotate(z, d, c["rope_theta"], c["rope_scaling"]) for z in (q, k))
            x = x + self.product(_attend(q, k, v, d ** -0.5, causal), pre + "self_attn.o_proj.weight", D)
            h = self.norm(x, pre + "post_attention_layernorm.weight", eps)
            x = x + self.swiglu(h, pre + "mlp.", "_proj.weight", c["intermediate_size"])
        head = "model.embed_tokens.weight" if self.draw.tied else "lm_head.weight"
        return self.norm(x, "model.norm.weight", eps), head, 1.0

    def kupirax(self, tokens):
        c = self.raw
        D, eps = c["width"], c["norm"]["eps"]
        x = self.norm(self.w("embed", c["vocab"], D)[tokens], "embed.norm", eps)
        for i, layer in enumerate(c["layers"]):
            h = self.norm(x, f"l{i}.norm1", eps)
            mixed = getattr(self, "_" + layer["type"])(h, f"l{i}.mix.", layer["mixer"], eps)
            x = x + mixed + self.swiglu(h, f"l{i}.mlp.", "", layer["mlp"]["ff"])
        return self.norm(x, "final.norm", eps), "head", 1.0

    def _attention(self, h, pre, m, eps):
        H, G, d, rot, size = m["heads"], m["kv_heads"], m["dim"], m["rot"], m["mask"]["size"]
        q, k = (self.norm(self.product(h, pre + p, n * d), pre + p + ".norm", eps).unflatten(-1, (n, d))
                for p, n in (("q", H), ("k", G)))
        v = self.product(h, pre + "v", G * m["vdim"]).unflatten(-1, (G, -1))
        q, k = (_rotate(z, rot["dims"], rot["base"], rot["scaling"], neighbours=True) for z in (q, k))
        out = _attend(q, k, v, m["scale"], lambda i, j: (j <= i) & (j // size == i // size))
        return self.product(out, pre + "o", h.shape[-1])

    def _retention(self, h, pre, m, eps):
        H, d, dv, rot = m["heads"], m["dim"], m["vdim"], m["rot"]
        q, k = (_rotate(self.product(h, pre + p, H * d).unflatten(-1, (H, d)), rot["dims"], rot["base"], None) for p in "qk")
        k = k / math.sqrt(d)
        v = self.product(h, pre + "v", H * dv).unflatten(-1, (H, dv))
        decay = torch.tensor(m["decay"], dtype=h.dtype, device=h.device)[:, None, None]
        S = h.new_zeros(h.shape[0], H, d, dv)
        out = h.new_empty(h.shape[0], h.shape[1], H, dv)
        for t in range(h.shape[1]):
            S = S * decay + k[:, t, :, :, None] * v[:, t, :, None, :]
            out[:, t] = (q[:, t, :, None, :] @ S)[:, :, 0]
        return self.product(_rms(out, eps).flatten(2) * F.silu(self.product(h, pre + "g", H * dv)), pre + "o", h.shape[-1])

    def _channel_delta(self, h, pre, m, eps):
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        q, k, v = (F.silu(_convolve(self.product(h, pre + p, n), self.w(pre + p + ".conv", n, m["conv"]))).unflatten(-1, (H, -1))
                   for p, n in (("q", H * d), ("k", H * d), ("v", H * dv)))
        q, k = (z * torch.rsqrt(z.square().sum(-1, keepdim=True) + 1e-6) for z in (q, k))
        q = q / math.sqrt(d)
        beta = torch.sigmoid(self.product(h, pre + "b", H))
        rate = F.softplus(self.product(self.product(h, pre + "a1", m["decay_rank"]), pre + "a2", H * d)
                          + self.w(pre + "dt_bias", H * d)).unflatten(-1, (H, d))
        decay = torch.exp(-self.w(pre + "A_log", H).exp()[:, None] * rate)
        gate = torch.sigmoid(self.product(self.product(h, pre + "g1", m["gate_rank"]), pre + "g2", H * dv))
        S = h.new_zeros(h.shape[0], H, d, dv)
        out = h.new_empty(h.shape[0], h.shape[1], H, dv)
        for t in range(h.shape[1]):
            S = S * decay[:, t, :, :, None]
            u = beta[:, t, :, None] * (v[:, t] - (k[:, t, :, None, :] @ S)[:, :, 0])
            S = S + k[:, t, :, :, None] * u[:, :, None, :]
            out[:, t] = (q[:, t, :, None, :] @ S)[:, :, 0]
        out = _rms(out, eps) * self.w(pre + "norm", dv)
        return self.product(out.flatten(2) * gate, pre + "o", h.shape[-1])

    def badolix(self, tokens):
        c = self.raw
        D, eps, mult = c["width"], c["norm"]["eps"], c["residual_mult"]
        x = self.w("embed", c["vocab"], D)[tokens] * c["embedding"]["scale"]
        kept = {}
        for i, layer in enumerate(c["layers"]):
            m, pre = layer["mixer"], f"l{i}.mix."
            h = self.norm(x, f"l{i}.norm1", eps)
            if layer["type"] == "attention":
                mixed, kept[i] = self._window(h, pre, m, kept.get(m.get("kv_from")))
            elif layer["type"] == "latent_attention":
                mixed = self._latent(h, pre, m, eps)
            else:
                mixed = self._state_space(h, pre, m, eps)
            x = x + mult * mixed
            h, mlp = self.norm(x, f"l{i}.norm2", eps), layer["mlp"]
            if mlp["kind"] == "dense":
                x = x + mult * self.swiglu(h, f"l{i}.mlp.", "", mlp["ff"], biased=True)
            else:
                x = x + mult * self._routed(h.flatten(0, 1), f"l{i}.mlp.", mlp).view_as(h)
        return self.norm(x, "final.norm", eps), "embed", c["logit_scale"]

    def _window(self, h, pre, m, shared):
        H, G, d, rot = m["heads"], m["kv_heads"], m["dim"], m["rot"]
        turn = lambda z: _rotate(z, rot["dims"], rot["base"], rot["scaling"])  # noqa: E731
        q = turn(self.product(h, pre + "q", H * d).unflatten(-1, (H, d)))
        if shared is None:
            shared = (turn(self.product(h, pre + "k", G * d).unflatten(-1, (G, d))),
                      self.product(h, pre + "v", G * m["vdim"]).unflatten(-1, (G, -1)))
        size, keep = m["mask"]["size"], m["mask"]["keep_first"]
        out = _attend(q, *shared, m["scale"], lambda i, j: (j <= i) & ((i - j < size) | (j < keep)), m["softcap"])
        return self.product(out, pre + "o", h.shape[-1]), shared

    def _latent(self, h, pre, m, eps):
        H, d, r, dv, rank, rot = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"], m["rot"]
        turn = lambda z: _rotate(z, r, rot["base"], rot["scaling"])  # noqa: E731
        q = self.product(h, pre + "q", H * (d + r)).unflatten(-1, (H, d + r))
        down = self.product(h, pre + "dkv", rank + r)
        latent = self.norm(down[..., :rank], pre + "dkv.norm", eps)
        q = torch.cat([q[..., :d], turn(q[..., d:])], -1)
        k = torch.cat([self.product(latent, pre + "uk", H * d).unflatten(-1, (H, d)),
                       turn(down[..., None, rank:]).expand(-1, -1, H, -1)], -1)
        v = self.product(latent, pre + "uv", H * dv).unflatten(-1, (H, dv))
        return self.product(_attend(q, k, v, m["scale"], lambda i, j: j <= i), pre + "o", h.shape[-1])

    def _state_space(self, h, pre, m, eps):
        H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
        inner = H * P
        z, xbc, dt = self.product(h, pre + "in", 2 * inner + 2 * G * N + H).split([inner, inner + 2 * G * N, H], -1)
        channels = inner + 2 * G * N
        xbc = F.silu(_convolve(xbc, self.w(pre + "conv", channels, m["conv"])) + self.w(pre + "conv.b", channels))
        x, b, c = xbc.split([inner, G * N, G * N], -1)
        x = x.unflatten(-1, (H, P))
        b, c = (y.unflatten(-1, (G, N)).repeat_interleave(H // G, 2) for y in (b, c))
        dt = F.softplus(dt + self.w(pre + "dt_bias", H))
        decay = torch.exp(-self.w(pre + "A_log", H).exp() * dt)
        skip = self.w(pre + "D", H)[:, None]
        S = h.new_zeros(h.shape[0], H, N, P)
        out = torch.empty_like(x)
        for t in range(h.shape[1]):
            S = S * decay[:, t, :, None, None] + (dt[:, t, :, None] * b[:, t])[..., None] * x[:, t, :, None, :]
            out[:, t] = (c[:, t, :, None, :] @ S)[:, :, 0] + skip * x[:, t]
        out = out.flatten(2) * F.silu(z)
        parts = m["norm_groups"]
        out = _rms(out.unflatten(-1, (parts, -1)), eps).flatten(2) * self.w(pre + "norm", inner)
        return self.product(out, pre + "o", h.shape[-1])

    def _routed(self, h, pre, mlp):
        router = mlp["router"]
        groups = router["groups"]
        scores = torch.sigmoid(self.product(h, pre + "router", router["experts"]))
        by_group = scores.unflatten(-1, (groups["count"], -1))
        open_groups = by_group.topk(2, -1).values.sum(-1).topk(groups["keep"], -1).indices
        allowed = torch.zeros_like(by_group[..., 0]).scatter_(-1, open_groups, 1.0).bool()
        chosen = by_group.masked_fill(~allowed[..., None], -1.0).flatten(1).topk(router["top"], -1).indices
        weights = scores.gather(-1, chosen)
        weights = weights / (weights.sum(-1, keepdim=True) + 1e-20)
        out = torch.zeros_like(h)
        for e in range(router["experts"]):
            rows, place = (chosen == e).nonzero(as_tuple=True)
            if rows.numel():
                out[rows] += weights[rows, place, None] * self.swiglu(h[rows], f"{pre}e{e}.", "", mlp["expert"]["ff"])
        return out

    def logits(self, tokens, wanted):
        """float64 [len(wanted), vocab] for the (sequence, position) pairs of `wanted`."""
        x, head, scale = {"Kupirax": self.kupirax, "Badolix": self.badolix}.get(self.raw.get("architecture"), self.llama)(tokens)
        rows = torch.tensor(wanted, device=x.device).T
        return self.product(x[rows[0], rows[1]], head, self.draw.vocab) * scale


@torch.no_grad()
def exact(case, seed):
    device = torch.device("cuda:0" if torch.cuda.is_available() else "cpu")
    plain = _Plain(case, seed, device)
    prompts, new = _prompts(case, seed), case["new"]
    follow = plain.draw.follow().tolist() if new else []
    lines = []
    for prompt in prompts:  # the text that the head is sure of
        line = list(prompt)
        for _ in range(new):
            line.append(follow[line[-1]])
        lines.append(line)
    longest = max(len(line) for line in lines)
    tokens = torch.tensor([line + [0] * (longest - len(line)) for line in lines], device=device)
    wanted = [(i, len(line) - 1) for i, line in enumerate(lines)]
    if new == 0:
        return {"logits": plain.logits(tokens, wanted)}
    steps = [(i, len(prompt) + t - 1) for t in range(new) for i, prompt in enumerate(prompts)]
    logits = plain.logits(tokens, steps + wanted)
    said = logits[:len(steps)].argmax(-1).view(new, len(prompts)).cpu().numpy()
    return {"tokens": said, "logits": logits[len(steps):]}
