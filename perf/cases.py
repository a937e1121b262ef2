"""What the engine's speed is measured on: steps of language models through ``Engine.step`` (and
``Engine.sample``), as a serving loop calls them.

The sizes are those of the 4B preset and of the benchmark's table of layers (1b, 4b, 8b); weights and
token ids are made from a seed.  Three designs stand for the seven: the Qwen3 dense decoder in both
types, and the two whose layers between them hold every kind of mixer and feed-forward at work elsewhere
(state space recurrence, grouped-query attention with a sink, a cap and gates, routed experts, several
residual streams; latent attention, the gated delta rule, the token side).

One pass is one of four things (``"does"``):

* ``decode``: every live request gets one more token; its context is cut back first (a reply that is drawn
  again), so that a pass can be repeated.  Returns the logits, with ``sample`` also the tokens drawn.
* ``prompt``: new requests bring whole prompts in one step and are finished.  Returns the logits of each one's
  last ``want`` tokens.
* ``mixed``: live requests get one more token each beside the prompts of new requests, in one step.
* ``reply``: new requests from their prompts to the last of ``steps`` tokens, which are given (the scoring
  of known texts), then finished.  Returns the logits of every step.

Argmax feedback is left out on purpose: two correct engines may part at a tie, and nothing after it compares.
"""
from __future__ import annotations

import gc
import hashlib
import math

import torch

from kipp_b200.config import config_from_dict
from kipp_b200.config.registry import get_architecture
from kipp_b200.engine import Engine, StepEntry
from kipp_b200.sampling import SamplingParams

# (width, heads, kv heads, head size, feed-forward width), as the benchmark names them
SIZES = {"1b": (2048, 16, 4, 128, 6144), "4b": (2560, 32, 8, 128, 9728), "8b": (4096, 32, 8, 128, 12288)}
PORTION = 2048          # most tokens of a prompt fed in one step
PAGE = 16
F64 = torch.float64


# ---- the cases ---------------------------------------------------------------------------------------
def case(design, size, layers, does, requests, context, *, dtype="bfloat16", vocab=32000, ragged=False, **more):
    out = dict(design=design, size=size, layers=layers, vocab=vocab, dtype=dtype, does=does, requests=requests,
               context=context, ragged=ragged, prompts=0, prompt=0, want=1, steps=0, sample=False)
    out.update(more)
    return out


def listed():
    whole = dict(vocab=151936)
    return [
        # one user, a short exchange with a small model: launches and latency
        dict(case("qwen3", "1b", 4, "decode", 1, 77), name="decode 1x77 in 4 layers"),
        # one user of the 4B model after a page of text: weights read once for one token
        dict(case("qwen3", "4b", 36, "decode", 1, 2048, **whole), name="decode 1x2048"),
        # the benchmark's headline: eight requests near the end of their context
        dict(case("qwen3", "4b", 36, "decode", 8, 8100, **whole), name="decode 8x8100"),
        # a loaded server that draws its tokens
        dict(case("qwen3", "4b", 36, "decode", 64, 2048, sample=True, **whole), name="decode 64x2048 sampled"),
        # an odd number of requests, each at another place of its text
        dict(case("qwen3", "4b", 36, "decode", 13, 5003, ragged=True, **whole), name="decode 13 ragged"),
        # the benchmark's prompt
        dict(case("qwen3", "4b", 36, "prompt", 1, 2048, **whole), name="prompt 2048"),
        # continuous batching: three odd prompts arrive while twelve requests decode
        dict(case("qwen3", "4b", 36, "mixed", 12, 3001, ragged=True, prompts=3, prompt=421, **whole), name="mixed 12 + 3 prompts"),
        # the true 32-bit path, from short prompts to the end of the replies
        dict(case("qwen3", "1b", 4, "reply", 3, 203, dtype="float32", ragged=True, steps=8), name="reply in 32-bit"),
        # state space layers, routed experts, four residual streams: one long prompt, the last of it scored (an expert chosen
        # otherwise at a near tie changes one row by a third: few rows would compare nothing but that)
        dict(case("zunilorn", "1b", 4, "prompt", 1, 2048, want=64), name="zunilorn prompt 2048"),
        # the same design answers eight short questions
        dict(case("zunilorn", "4b", 4, "reply", 8, 101, ragged=True, steps=16), name="zunilorn reply 8"),
        # latent attention, gated delta rule, state space, token side: three odd prompts at once
        dict(case("nogavik", "4b", 4, "prompt", 3, 1277, ragged=True), name="nogavik prompts 3"),
        # the same design answers one question
        dict(case("nogavik", "1b", 4, "reply", 1, 300, steps=24), name="nogavik reply 1"),
    ]


def _log(rng, low, high):
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prompt", "mixed", "reply32", "design prompt", "design reply"])
    size = rng.choice(["1b", "4b", "4b", "8b"])
    layers = {"1b": 4, "4b": 36, "8b": 12}[size]
    vocab = 32000 if size == "1b" else 151936
    ragged = rng.random() < 0.6
    if kind in ("decode", "mixed"):
        n = _log(rng, 1, 64)
        context = _log(rng, 64, min(8100, 131072 // n))
        if kind == "decode":
            return case("qwen3", size, layers, "decode", n, context, vocab=vocab, ragged=ragged, sample=rng.random() < 0.25)
        k = rng.randint(1, 4)
        return case("qwen3", size, layers, "mixed", n, context, vocab=vocab, ragged=ragged, prompts=k, prompt=_log(rng, 17, 1500 // k))
    if kind == "prompt":
        k = rng.randint(1, 4)
        return case("qwen3", size, layers, "prompt", k, _log(rng, 33, 2048 // k), vocab=vocab, ragged=ragged)
    if kind == "reply32":
        return case("qwen3", "1b", 4, "reply", rng.randint(1, 6), _log(rng, 20, 240), dtype="float32", ragged=ragged, steps=rng.randint(2, 8))
    design, size = rng.choice(["zunilorn", "nogavik"]), rng.choice(["1b", "4b"])
    if kind == "design prompt":
        k = rng.randint(1, 4)
        return case(design, size, 4, "prompt", k, _log(rng, 65, 2048 // k), ragged=ragged, want=64 if design == "zunilorn" else 1)
    return case(design, size, 4, "reply", _log(rng, 1, 16), _log(rng, 20, 300), ragged=ragged, steps=rng.randint(4, 16))


def lengths(n, longest, ragged):
    """Tokens of each of n texts: all the longest, or spread between a tenth of it and all of it."""
    if not ragged:
        return [longest] * n
    return [longest] + [max(1, int(longest * (0.1 + 0.9 * ((i * 0.6180339887) % 1.0)))) for i in range(1, n)]


# ---- configurations ------------------------------------------------------------------------------------
def config_of(c):
    width, heads, kv, dim, ff = SIZES[c["size"]]
    if c["design"] == "qwen3":
        return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", vocab_size=c["vocab"], hidden_size=width,
                    intermediate_size=ff, num_hidden_layers=c["layers"], num_attention_heads=heads, num_key_value_heads=kv,
                    head_dim=dim, max_position_embeddings=8192, rope_theta=1e6, rms_norm_eps=1e-6, tie_word_embeddings=True,
                    hidden_act="silu", attention_bias=False, initializer_range=0.02, torch_dtype="bfloat16")
    ssm = {"heads": 2 * width // 64, "groups": 8, "vdim": 64, "state": 128, "conv": 4, "norm_groups": 8}
    if c["design"] == "zunilorn":
        moe = {"kind": "moe", "expert": {"ff": ff // 4, "limit": 7.0},
               "router": {"experts": 16, "identity": 2, "top": 4, "scale": 2.5}, "shared": {"ff": ff // 4, "limit": 7.0}}
        att = {"heads": heads, "kv_heads": kv, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "softcap": 50.0,
               "rot": {"base": 1e6, "dims": dim, "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
        order = [{"type": "mamba2", "mixer": ssm, "mlp": {"kind": "dense", "ff": ff, "limit": 7.0}},
                 {"type": "attention", "mixer": att, "mlp": moe}, {"type": "mamba2", "mixer": ssm, "mlp": moe},
                 {"type": "attention", "mixer": att, "mlp": moe}]
        return {"architecture": "Zunilorn", "vocab": c["vocab"], "width": width, "norm": {"eps": 1e-5}, "residual_mult": 0.5,
                "streams": 4, "logit_softcap": 30.0, "layers": [order[i % 4] for i in range(c["layers"])]}
    latent = {"heads": heads, "dim": dim, "rot_dim": dim // 2, "vdim": dim, "kv_rank": 4 * dim, "q_rank": width // 2,
              "rot": {"base": 1e6, "dims": dim // 2}, "scale": (dim + dim // 2) ** -0.5}
    par = {"left": {"heads": heads // 2, "kv_heads": kv // 2, "dim": dim, "vdim": 2 * dim, "scale": dim ** -0.5},
           "right": {"heads": heads // 2, "kv_heads": heads // 2, "dim": dim, "vdim": dim, "conv": 4, "decay_rank": dim,
                     "gate_rank": dim}}
    order = [("mamba2", ssm), ("latent_attention", latent), ("parallel", par), ("latent_attention", dict(latent, kv_from=1))]
    return {"architecture": "Nogavik", "vocab": c["vocab"], "width": width, "norm": {"eps": 1e-5}, "token_side": {"dim": 128},
            "layers": [{"type": t, "mixer": m, "mlp": {"kind": "dense", "ff": ff}}
                       for t, m in (order[i % 4] for i in range(c["layers"]))]}


# ---- preparation and the pass ----------------------------------------------------------------------------
def texts(c, seed):
    """(token ids of every live request's context and its next token, token ids of every new request's prompt and of the
    tokens given after it)"""
    g = torch.Generator().manual_seed(7919 * seed + 13)

    def some(n):
        return torch.randint(0, c["vocab"], (n,), generator=g).tolist()
    live = [some(n + 1) for n in lengths(c["requests"], c["context"], c["ragged"])] if c["does"] in ("decode", "mixed") else []
    if c["does"] == "mixed":
        new = [some(n) for n in lengths(c["prompts"], c["prompt"], c["ragged"])]
    elif c["does"] in ("prompt", "reply"):
        new = [some(n + c["steps"]) for n in lengths(c["requests"], c["context"], c["ragged"])]
    else:
        new = []
    return live, new


class State:
    pass


def prepare(c, seed):
    gc.collect()                                  # an engine that was given up has left its memory before the next one is made
    live, new = texts(c, seed)
    room = sum(len(t) + 2 * PAGE for t in live + new)
    s = State()
    s.case = c
    s.engine = Engine.from_config(config_from_dict(config_of(c)), seed, dtype=c["dtype"], page_size=PAGE,
                                  cache_tokens=room, max_requests=len(live) + len(new),
                                  max_batch_tokens=max(PORTION, len(live) + sum(len(t) for t in new)))
    s.live = [("live", i) for i in range(len(live))]
    s.kept = [len(t) - 1 for t in live]
    for rid, t in zip(s.live, live):
        for a in range(0, len(t) - 1, PORTION):
            s.engine.step([StepEntry(rid, t[a:min(a + PORTION, len(t) - 1)], [])])
    s.new = [("new", i) for i in range(len(new))]
    s.first = [StepEntry(rid, [t[-1]], [0]) for rid, t in zip(s.live, live)]
    for rid, t in zip(s.new, new):
        n = len(t) - c["steps"]
        s.first.append(StepEntry(rid, t[:n], list(range(max(0, n - c["want"]), n))))
    s.next = [[StepEntry(rid, [t[len(t) - c["steps"] + k]], [0]) for rid, t in zip(s.new, new)] for k in range(c["steps"])]
    s.params = [SamplingParams(temperature=0.0 if i % 4 == 0 else 0.8, top_p=0.95, top_k=0 if i % 2 else 50, seed=i + 1)
                for i in range(len(live))]
    return s


def run(s):
    e = s.engine
    for rid, n in zip(s.live, s.kept):
        e.truncate(rid, n)
    logits = e.step(s.first)
    out = {"logits": logits}
    if s.case["sample"]:
        out["tokens"] = torch.tensor(e.sample(s.params, [p.seed for p in s.params]))
    if s.next:
        out["logits"] = logits.new_empty(1 + len(s.next), *logits.shape)
        out["logits"][0].copy_(logits)
        for k, entries in enumerate(s.next):
            out["logits"][k + 1].copy_(e.step(entries))
    for rid in s.new:
        e.finish(rid)
    return out


# ---- what a pass cannot do without -----------------------------------------------------------------------
def work(c):
    config = config_from_dict(config_of(c))
    live, new = lengths(c["requests"], c["context"], c["ragged"]), []
    if c["does"] == "mixed":
        new = lengths(c["prompts"], c["prompt"], c["ragged"])
    elif c["does"] != "decode":
        live, new = [], live
    dense, expert, head = 0, 0, SIZES[c["size"]][0] * c["vocab"]
    for t in get_architecture(config.architecture).build(config).tensor_specs():
        if len(t.shape) == 2 and "embed" not in t.name and "conv" not in t.name and t.name not in ("head", "lm_head.weight"):
            n = t.shape[0] * t.shape[1]
            if ".mlp.e" in t.name:
                expert += n
            else:
                dense += n
    item = 4 if c["dtype"] == "float32" else 2
    width, heads, kv, dim, _ = SIZES[c["size"]]
    # (bytes of cache per token, bytes of state per request, attention's multiply-adds per pair of positions)
    if c["design"] == "qwen3":
        cache, state, pair = c["layers"] * 2 * kv * dim * item, 0, c["layers"] * 2 * heads * dim
    else:
        turn = [i % 4 for i in range(c["layers"])]
        ssm = 2 * width * 128 * 4
        if c["design"] == "zunilorn":
            cache = sum(2 * kv * dim * item for i in turn if i % 2)
            state, pair = sum(ssm for i in turn if i % 2 == 0), sum(2 * heads * dim for i in turn if i % 2)
        else:
            per = {0: 0, 1: (4 * dim + dim // 2) * item, 2: kv // 2 * 3 * dim * item, 3: 0}
            cache = sum(per[i] for i in turn)
            state = sum(ssm if i == 0 else heads // 2 * dim * dim * 4 if i == 2 else 0 for i in turn)
            pair = sum({0: 0, 1: heads * 5 * dim // 2, 2: heads // 2 * 3 * dim, 3: heads * 5 * dim // 2}[i] for i in turn)

    def step(fed, before):
        """(bytes, operations) of one step: ``fed`` tokens of each request onto ``before`` kept ones"""
        tokens = sum(fed)
        hit = 1.0 - (1.0 - 4.0 / 18.0) ** tokens
        b = (dense + expert * hit + head) * item + sum(f + p for f, p in zip(fed, before)) * cache
        b += len(fed) * (4 * c["vocab"] + 2 * state) + tokens * width * item
        f = 2.0 * tokens * (dense + expert / 16.0 * 4.0 * 16.0 / 18.0) + 2.0 * len(fed) * head
        f += sum(2.0 * pair * (q * p + q * (q + 1) / 2) for q, p in zip(fed, before))
        return b, f
    total = [step([1] * len(live) + new, live + [0] * len(new))]
    for k in range(c["steps"]):
        total.append(step([1] * len(new), [n + k for n in new]))
    return {"bytes": sum(t[0] for t in total), "flops": sum(t[1] for t in total)}


def tolerance(c):
    # about four times the distance measured from 64 bits (5e-6; 0.009 to 0.035 with experts chosen otherwise at near ties
    # among them; 0.005; 0.026 after 36 layers, 0.011 after 4)
    if c["dtype"] == "float32":
        return {"rel": 2e-5}
    t = {"rel": 0.15 if c["design"] == "zunilorn" else 0.02 if c["design"] == "nogavik" else 0.1 if c["layers"] > 4 else 0.05}
    if c["sample"]:
        t["differ"] = 0.2
    return t


# ---- the same in 64 bits -----------------------------------------------------------------------------------
class Weights:
    """The random weights of a seed, one tensor at a time: each has a generator of its own, named by the seed and the tensor."""

    def __init__(self, seed, device):
        self.seed, self.device = seed, device

    def __call__(self, name, *shape, kind="normal"):
        digest = hashlib.sha256(f"{self.seed}:{name}".encode()).digest()
        g = torch.Generator(device=self.device)
        g.manual_seed(int.from_bytes(digest[:8], "little") & ((1 << 63) - 1))
        t = torch.empty(shape, dtype=torch.float32, device=self.device)
        if kind == "normal":
            t.normal_(0.0, 0.02, generator=g)
        elif kind == "one":
            t.uniform_(-0.1, 0.1, generator=g).add_(1.0)
        else:
            t.normal_(0.0, 0.1, generator=g).add_(torch.eye(*shape, device=self.device))
        return t.to(torch.bfloat16).to(F64)


def rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def silu(x):
    return x * torch.sigmoid(x)


def turned(x, positions, freq, magnitude=1.0, neighbours=False):
    """x [T, H, D]: the first 2 len(freq) coordinates turn in pairs (i, i + half), or (2i, 2i + 1)."""
    half = freq.numel()
    ang = positions.to(F64)[:, None, None] * freq
    c, s = torch.cos(ang) * magnitude, torch.sin(ang) * magnitude
    out = x.clone()
    first, second = (slice(0, 2 * half, 2), slice(1, 2 * half, 2)) if neighbours else (slice(0, half), slice(half, 2 * half))
    u, v = x[..., first], x[..., second]
    out[..., first], out[..., second] = u * c - v * s, v * c + u * s
    return out


def frequencies(base, dims, device):
    return torch.tensor([base ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=F64, device=device)


def stretched(rot, device):
    """Frequencies of a rotation stretched by a factor: fast pairs keep theirs, slow ones are divided, a ramp between."""
    sc, dims, base = rot["scaling"], rot["dims"], rot["base"]
    at = [dims * math.log(sc["original"] / (2 * math.pi * t)) / (2 * math.log(base)) for t in (sc["fast"], sc["slow"])]
    low, high = max(math.floor(at[0]), 0), min(math.ceil(at[1]), dims - 1)
    ramp = ((torch.arange(dims // 2, dtype=F64, device=device) - low) / max(high - low, 0.001)).clamp(0, 1)
    f = frequencies(base, dims, device)
    return f / sc["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(sc["factor"]) + 1.0


def attend(q, k, v, scale, cap=None, sink=None):
    """q [T, H, D], k [T, G, D], v [T, G, V]: causal grouped-query attention; ``sink`` [H] joins the denominators."""
    T, H, _ = q.shape
    G = k.shape[1]
    out = torch.empty(T, H, v.shape[-1], dtype=F64, device=q.device)
    key = torch.arange(T, device=q.device)
    for h in range(H):
        for a in range(0, T, 2048):                       # rows of queries at a time
            b = min(T, a + 2048)
            s = q[a:b, h] @ k[:b, h * G // H].T * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            s = s.masked_fill(key[None, :b] > key[a:b, None], -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[h].expand(b - a, 1)], 1)
            out[a:b, h] = torch.softmax(s, -1)[:, :b] @ v[:b, h * G // H]
    return out


def convolved(x, weight, bias=None):
    taps = weight.shape[1]
    padded = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    out = sum(padded[j:j + x.shape[0]] * weight[:, j] for j in range(taps))
    return out if bias is None else out + bias


def state_space(m, w, p, h, eps):
    T, width = h.shape
    H, P, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
    inner, wide = H * P, H * P + 2 * G * N
    z, xbc, dt = (h @ w(p + "in", inner + wide + H, width).T).split([inner, wide, H], 1)
    xbc = silu(convolved(xbc, w(p + "conv", wide, m["conv"]), w(p + "conv.b", wide)))
    x, B, C = xbc.split([inner, G * N, G * N], 1)
    x = x.reshape(T, H, P)
    B, C = (t.reshape(T, G, 1, N).expand(T, G, H // G, N).reshape(T, H, N) for t in (B, C))
    dt = torch.nn.functional.softplus(dt + w(p + "dt_bias", H), threshold=1e9)
    decay = torch.exp(-torch.exp(w(p + "A_log", H)) * dt)
    S, y = h.new_zeros(H, N, P), torch.empty_like(x)
    for t in range(T):
        S = decay[t][:, None, None] * S + (dt[t][:, None] * B[t])[:, :, None] * x[t][:, None, :]
        y[t] = torch.einsum("hnp,hn->hp", S, C[t])
    y = (y + w(p + "D", H)[:, None] * x).reshape(T, inner) * silu(z)
    y = rms(y.view(T, m["norm_groups"], -1), eps).reshape(T, inner) * w(p + "norm", inner, kind="one")
    return y @ w(p + "o", width, inner).T


def gated(gate, up, limit):
    gate, up = gate.clamp(max=limit), up.clamp(-limit, limit)
    return gate * torch.sigmoid(1.702 * gate) * (up + 1)


class Qwen3:
    def __init__(self, c, w):
        self.c, self.w, self.n = config_of(c), w, c["layers"]
        self.embed = w("model.embed_tokens.weight", c["vocab"], self.c["hidden_size"])

    def start(self, ids):
        return [self.embed[t] for t in ids]

    def layer(self, i, xs, _ids):
        c, w, p = self.c, self.w, f"model.layers.{i}."
        W, D, H, G, eps = c["hidden_size"], c["head_dim"], c["num_attention_heads"], c["num_key_value_heads"], c["rms_norm_eps"]
        sizes = [x.shape[0] for x in xs]
        x = torch.cat(xs)
        n = rms(x, eps) * w(p + "input_layernorm.weight", W, kind="one")
        q, k, v = (n @ w(p + f"self_attn.{s}_proj.weight", r * D, W).T for s, r in (("q", H), ("k", G), ("v", G)))
        q = rms(q.view(-1, H, D), eps) * w(p + "self_attn.q_norm.weight", D, kind="one")
        k = rms(k.view(-1, G, D), eps) * w(p + "self_attn.k_norm.weight", D, kind="one")
        freq = frequencies(c["rope_theta"], D, x.device)
        out = []
        for q1, k1, v1 in zip(q.split(sizes), k.split(sizes), v.view(-1, G, D).split(sizes)):
            pos = torch.arange(q1.shape[0], device=x.device)
            out.append(attend(turned(q1, pos, freq), turned(k1, pos, freq), v1, D ** -0.5).reshape(-1, H * D))
        x = x + torch.cat(out) @ w(p + "self_attn.o_proj.weight", W, H * D).T
        n = rms(x, eps) * w(p + "post_attention_layernorm.weight", W, kind="one")
        F = c["intermediate_size"]
        a = silu(n @ w(p + "mlp.gate_proj.weight", F, W).T) * (n @ w(p + "mlp.up_proj.weight", F, W).T)
        return list((x + a @ w(p + "mlp.down_proj.weight", W, F).T).split(sizes))

    def finish(self, x):
        return rms(x, self.c["rms_norm_eps"]) * self.w("model.norm.weight", x.shape[-1], kind="one") @ self.embed.T


class Zunilorn:
    def __init__(self, c, w):
        self.c, self.w, self.n = config_of(c), w, c["layers"]
        self.embed = w("embed", c["vocab"], self.c["width"])

    def start(self, ids):
        return [self.embed[t][None].repeat(4, 1, 1) for t in ids]

    def attention(self, m, p, h):
        w, (T, W) = self.w, h.shape
        H, G, D = m["heads"], m["kv_heads"], m["dim"]
        freq, mag = stretched(m["rot"], h.device)
        pos = torch.arange(T, device=h.device)
        q, k, v = ((h @ w(p + s, r * D, W).T).view(T, r, D) for s, r in (("q", H), ("k", G), ("v", G)))
        o = attend(turned(q, pos, freq, mag), turned(k, pos, freq, mag), v, m["scale"], m["softcap"], w(p + "sink", H))
        return (o * torch.sigmoid(h @ w(p + "g", H, W).T)[:, :, None]).reshape(T, -1) @ w(p + "o", W, H * D).T

    def ff(self, f, p, h, size):
        w, W = self.w, h.shape[1]
        a = gated(h @ w(p + "gate", size, W).T, h @ w(p + "up", size, W).T, f["limit"])
        return a @ w(p + "down", W, size).T

    def feed_forward(self, f, p, h):
        w, W = self.w, h.shape[1]
        if f["kind"] == "dense":
            a = gated(h @ w(p + "gate", f["ff"], W).T + w(p + "gate.b", f["ff"]),
                      h @ w(p + "up", f["ff"], W).T + w(p + "up.b", f["ff"]), f["limit"])
            return a @ w(p + "down", W, f["ff"]).T + w(p + "down.b", W)
        r = f["router"]
        s = torch.softmax(h @ w(p + "router", r["experts"] + r["identity"], W).T, -1)
        chosen = torch.topk(s + w(p + "correction", s.shape[1]), r["top"], dim=-1).indices
        weight = s.gather(1, chosen)
        weight = torch.zeros_like(s).scatter(1, chosen, weight / (weight.sum(-1, keepdim=True) + 1e-20) * r["scale"])
        out = weight[:, r["experts"]:].sum(1, keepdim=True) * h
        for e in range(r["experts"]):
            rows = weight[:, e].nonzero()[:, 0]
            if rows.numel():
                out[rows] += weight[rows, e, None] * self.ff(f["expert"], f"{p}e{e}.", h[rows], f["expert"]["ff"])
        return out + torch.sigmoid(h @ w(p + "shared.sg", 1, W).T) * self.ff(f["shared"], p + "shared.", h, f["shared"]["ff"])

    def layer(self, i, streams, _ids):
        w, eps, l = self.w, self.c["norm"]["eps"], self.c["layers"][i]
        out = []
        for xs in streams:
            for q in (1, 2):
                c_in, c_out = (w(f"l{i}.hc{q}.{k}", 4, kind="one") for k in ("in", "out"))
                mix = w(f"l{i}.hc{q}.mix", 4, 4, kind="identity")
                u = torch.einsum("s,stw->tw", c_in, xs)
                h = rms(u, eps) * w(f"l{i}.norm{q}", u.shape[1], kind="one")
                if q == 2:
                    y = self.feed_forward(l["mlp"], f"l{i}.mlp.", h)
                elif l["type"] == "mamba2":
                    y = state_space(l["mixer"], w, f"l{i}.mix.", h, eps)
                else:
                    y = self.attention(l["mixer"], f"l{i}.mix.", h)
                xs = torch.einsum("sr,stw->rtw", mix, xs) + self.c["residual_mult"] * c_out[:, None, None] * y
            out.append(xs)
        return out

    def finish(self, x):
        x = rms(x.sum(0), self.c["norm"]["eps"]) * self.w("final.norm", x.shape[-1], kind="one") @ self.embed.T
        return self.c["logit_softcap"] * torch.tanh(x / self.c["logit_softcap"])


class Nogavik:
    def __init__(self, c, w):
        self.c, self.w, self.n = config_of(c), w, c["layers"]
        self.embed = w("embed", c["vocab"], self.c["width"])
        self.side = w("side.embed", c["vocab"], c["layers"] * self.c["token_side"]["dim"])
        self.lent = {}

    def start(self, ids):
        return [self.embed[t] for t in ids]

    def norm(self, x, name):
        return rms(x, self.c["norm"]["eps"]) * (1.0 + self.w(name, x.shape[-1]))

    def latent(self, i, which, m, p, h):
        w, (T, W), eps = self.w, h.shape, self.c["norm"]["eps"]
        H, D, R, K = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
        pos, freq = torch.arange(T, device=h.device), frequencies(m["rot"]["base"], m["rot"]["dims"], h.device)
        if m.get("kv_from") is None:
            both = h @ w(p + "dkv", K + R, W).T
            self.lent[i, which] = (rms(both[:, :K], eps) * w(p + "dkv.norm", K, kind="one"),
                                   turned(both[:, None, K:], pos, freq, neighbours=True))
        c, k_rot = self.lent[m.get("kv_from", i), which]
        c_q = rms(h @ w(p + "dq", m["q_rank"], W).T, eps) * w(p + "dq.norm", m["q_rank"], kind="one")
        q = (c_q @ w(p + "uq", H * (D + R), m["q_rank"]).T).view(T, H, D + R)
        q = torch.cat([q[..., :D], turned(q[..., D:], pos, freq, neighbours=True)], -1)
        k = torch.cat([(c @ w(p + "uk", H * D, K).T).view(T, H, D), k_rot.expand(T, H, R)], -1)
        v = (c @ w(p + "uv", H * m["vdim"], K).T).view(T, H, -1)
        o = attend(q, k, v, m["scale"]).reshape(T, -1)
        return (o * torch.sigmoid(h @ w(p + "g", o.shape[1], W).T)) @ w(p + "o", W, o.shape[1]).T

    def attention(self, m, p, h):
        w, (T, W), eps = self.w, h.shape, self.c["norm"]["eps"]
        H, G, D, V = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, k, v = (h @ w(p + s, r, W).T + w(p + s + ".b", r) for s, r in (("q", H * D), ("k", G * D), ("v", G * V)))
        q = rms(q.view(T, H, D), eps) * w(p + "q.norm", D, kind="one")
        k = rms(k.view(T, G, D), eps) * w(p + "k.norm", D, kind="one")
        return attend(q, k, v.view(T, G, V), m["scale"]).reshape(T, -1) @ w(p + "o", W, H * V).T

    def delta(self, m, p, h):
        w, (T, W) = self.w, h.shape
        H, D, V, G = m["heads"], m["dim"], m["vdim"], m["kv_heads"]
        q, k, v = (silu(convolved(h @ w(p + s, r, W).T, w(p + s + ".conv", r, m["conv"])))
                   for s, r in (("q", G * D), ("k", G * D), ("v", H * V)))
        head = torch.arange(H, device=h.device) // (H // G)
        q, k = (t.view(T, G, D) / torch.sqrt((t.view(T, G, D) ** 2).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        q, k, v = q[:, head] * D ** -0.5, k[:, head], v.view(T, H, V)
        beta = torch.sigmoid(h @ w(p + "b", H, W).T)
        rate = (h @ w(p + "a1", m["decay_rank"], W).T) @ w(p + "a2", H * D, m["decay_rank"]).T + w(p + "dt_bias", H * D)
        g = torch.exp(-torch.exp(w(p + "A_log", H))[:, None] * torch.nn.functional.softplus(rate, threshold=1e9).view(T, H, D))
        S, out = h.new_zeros(H, D, V), torch.empty_like(v)
        for t in range(T):
            S = g[t][:, :, None] * S
            u = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None, :]
            out[t] = torch.einsum("hdv,hd->hv", S, q[t])
        out = rms(out, self.c["norm"]["eps"]) * w(p + "norm", V, kind="one")
        gate = torch.sigmoid((h @ w(p + "g1", m["gate_rank"], W).T) @ w(p + "g2", H * V, m["gate_rank"]).T)
        return (out.reshape(T, -1) * gate) @ w(p + "o", W, H * V).T

    def layer(self, i, xs, ids):
        w, eps, l, p = self.w, self.c["norm"]["eps"], self.c["layers"][i], f"l{i}.mix."
        d, out = self.c["token_side"]["dim"], []
        for which, (x, t) in enumerate(zip(xs, ids)):
            W, m = x.shape[1], l["mixer"]
            h = self.norm(x, f"l{i}.norm1")
            if l["type"] == "mamba2":
                y = state_space(m, w, p, h, eps)
            elif l["type"] == "latent_attention":
                y = self.latent(i, which, m, p, h)
            else:
                y = 0.5 * (rms(self.attention(m["left"], p + "left.", h), eps) * w(p + "left.out", W, kind="one") +
                           rms(self.delta(m["right"], p + "right.", h), eps) * w(p + "right.out", W, kind="one"))
            F = l["mlp"]["ff"]
            up = torch.relu(self.norm(x, f"l{i}.norm2") @ w(f"l{i}.mlp.up", F, W).T) ** 2
            x = x + y + up @ w(f"l{i}.mlp.down", W, F).T
            z = x @ w(f"l{i}.side.gate", d, W).T
            z = 0.5 * z * (1 + torch.tanh(math.sqrt(2 / math.pi) * (z + 0.044715 * z ** 3)))
            side = (z * self.side[t][:, i * d:(i + 1) * d]) @ w(f"l{i}.side.proj", W, d).T
            out.append(x + rms(side, eps) * w(f"l{i}.side.norm", W, kind="one"))
        return out

    def finish(self, x):
        return self.norm(x, "final.norm") @ self.embed.T


def exact(c, seed):
    if c["design"] == "qwen3" and work_of_texts(c) > 4e14:
        return None                                     # over about 20 seconds in 64 bits
    device = torch.device("cuda")
    live, new = texts(c, seed)
    ids = [torch.tensor(t, device=device) for t in live + new]
    with torch.no_grad():
        model = {"qwen3": Qwen3, "zunilorn": Zunilorn, "nogavik": Nogavik}[c["design"]](c, Weights(seed, device))
        xs = model.start(ids)
        for i in range(model.n):
            xs = model.layer(i, xs, ids)
        # the last positions of every text: the token fed last, or the prompt's end and the tokens given after it
        rows = [model.finish(x[..., -c["want"] - c["steps"]:, :]) for x in xs]
    if c["steps"]:
        return {"logits": torch.stack(rows, 1)}
    out = {"logits": torch.cat(rows)}
    if c["sample"]:
        out["tokens"] = None
    return out


def work_of_texts(c):
    """Operations of the products and of the attention over whole texts."""
    width, heads, kv, dim, ff = SIZES[c["size"]]
    n = lengths(c["requests"], c["context"], c["ragged"]) + lengths(c["prompts"], c["prompt"], c["ragged"]) * (c["does"] == "mixed")
    per = 2 * (width * dim * (2 * heads + 2 * kv) + 3 * width * ff)
    return c["layers"] * sum(t * per + 4 * heads * dim * t * t for t in n)
