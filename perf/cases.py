"""What a user of this engine has it compute, as cases that can be timed and checked: single layers of the designs that it
serves, called the way the engine's own blocks call them, and two whole steps of a model that end in logits.

A layer is built from its spec by the registry of parts, gets random weights by `bind`, and is called as
`mixer.forward(x, step, cache)` or `feed_forward.forward(x, step)` on a batch that `BatchBuilder` describes; the whole steps go
through `make_driver` and its step function.  Sizes are those of `bench.py`'s design tables.  Single-token steps of a layer are
captured into a CUDA graph when they are prepared and replayed, as the engine runs its decode steps; prompts run eagerly.

    kind     state_space, delta, gla, memory    mixers that carry a matrix per head from token to token
             latent, attention                  mixers over a paged cache (rows of latent + rotated part; grouped queries under a
                                                window that keeps the first tokens, capped scores, a gate)
             experts                            routed experts beside a shared one
             model                              a whole step: embedding, layers, logits
    phase    prompt: `tokens` new tokens, cut unevenly into `entries` requests, behind `context` earlier tokens each
             decode: one new token for each of `tokens` requests that hold `context` tokens
"""

from __future__ import annotations

import math

import torch

from jax_vllm_b200 import make_driver, ops, random_model, registry
from jax_vllm_b200.cache import CacheManager
from jax_vllm_b200.config.model_spec import (GatedLinearAttentionSpec, DeltaRuleSpec, GeneralAttentionSpec, LatentAttentionSpec,
                                             MatrixMemorySpec, RopeSpec, RoutedExpertsSpec, StateSpaceSpec)
from jax_vllm_b200.engine import StepEntry
from jax_vllm_b200.engine.batch import BatchBuilder
from jax_vllm_b200.parts import BuildContext
from jax_vllm_b200.parts.registry import FEED_FORWARDS, MIXERS, build
from jax_vllm_b200.weights.random_init import random_tensors

PAGE = 16
EPS = 1e-5
DEVICE = "cuda"

# width; state-space (heads, values, state, groups); delta (heads, size, rank); memory and linear attention (heads, keys, values);
# latent (heads, plain, rotated, values, latent, query latent, window); attention (heads, key heads, size, window);
# experts (number, identity, top, size, shared); a whole model (layers, heads, key heads, size, feed-forward)
SIZES = {
    "small": dict(width=1024, ssm=(32, 64, 64, 2), delta=(16, 64, 32), mem=(4, 64, 128), lat=(8, 64, 32, 64, 256, 512, 512),
                  att=(16, 4, 64, 512), exp=(16, 2, 2, 1024, 512), model=(2, 16, 4, 64, 2816)),
    "w2k": dict(width=2048, ssm=(64, 64, 128, 1), delta=(32, 64, 64), mem=(8, 128, 256), lat=(16, 128, 64, 128, 512, 1536, 1024),
                att=(16, 4, 128, 1024), exp=(32, 4, 4, 1024, 1024), model=(4, 16, 4, 128, 5632)),
    "w4k": dict(width=4096, ssm=(128, 64, 128, 8), delta=(64, 64, 96), mem=(8, 256, 512), lat=(32, 128, 64, 128, 512, 1536, 1024),
                att=(32, 8, 128, 1024), exp=(32, 4, 4, 2048, 2048), model=(2, 32, 8, 128, 11008)),
}
KEEP, CAP, TAU, GATE_CAP, TAPS, ROTATION, VOCAB = 4, 30.0, 16.0, 15.0, 4, 5e5, 32000
RECURRENT = ("state_space", "delta", "gla", "memory")
PAGED = ("latent", "attention")


def _case(kind, size, phase, tokens, entries=1, context=0, dtype="bf16"):
    return {"kind": kind, "size": size, "phase": phase, "tokens": tokens, "entries": entries, "context": context, "dtype": dtype}


def listed():
    def c(name, *args, **more):
        return {"name": name, **_case(*args, **more)}
    return [
        # the smallest call there is: one user, one token, a small model's layer
        c("token_state_space", "state_space", "small", "decode", 1, context=40),
        # decode steps of a serving batch: a recurrent layer, both kinds of cache, experts
        c("decode_gla", "gla", "w2k", "decode", 48, context=500),
        c("decode_latent", "latent", "w2k", "decode", 8, context=2048),
        c("decode_attention", "attention", "w2k", "decode", 24, context=1500),
        c("decode_experts", "experts", "w2k", "decode", 8),
        # a whole decode step of a plain model, from token ids to logits
        c("decode_model", "model", "w2k", "decode", 8, context=2048),
        # a whole prompt in the 32-bit mode (reference outputs, checks of a conversion)
        c("prompt_model_f32", "model", "small", "prompt", 203, dtype="f32"),
        # prompts: one long one, several ragged ones, a portion behind earlier context, the largest
        c("prompt_delta", "delta", "w2k", "prompt", 2048),
        c("prompt_latent", "latent", "w2k", "prompt", 2048),
        c("prompt_attention", "attention", "small", "prompt", 2999, entries=3, context=77),
        c("prompt_experts", "experts", "w2k", "prompt", 777),
        c("prompt_state_space", "state_space", "w4k", "prompt", 4096, entries=3),
    ]


def _log_uniform(rng, low, high):
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high + 0.49))))))


def draw(rng):
    kind = rng.choice(RECURRENT + PAGED + ("experts", "model"))
    phase = rng.choice(("prompt", "decode"))
    size = rng.choice(tuple(SIZES))
    dtype = "bf16"
    if rng.random() < 0.2:                            # the 32-bit mode: small models, shorter prompts
        dtype, size = "f32", "small"
    if phase == "prompt":
        tokens = _log_uniform(rng, 16, 400 if dtype == "f32" else 2048 if size == "w4k" else 4096)
        entries = rng.choice((1, 1, 2, 3, 5))
        context = rng.choice((0, 0, _log_uniform(rng, 1, 1500)))
    else:
        tokens, entries = _log_uniform(rng, 1, 16 if dtype == "f32" else 64), 1
        context = _log_uniform(rng, 16, 1024 if dtype == "f32" else 4096)
    return _case(kind, size, phase, tokens, entries, context, dtype)


# --------------------------------------------------------------------------------------------------------- inputs
def _lengths(case):
    """New tokens of every entry."""
    n, parts = case["tokens"], case["entries"]
    if case["phase"] == "decode":
        return [1] * n
    shares = [1.0 + 0.7 * i for i in range(parts)]
    out = [max(1, int(n * s / sum(shares))) for s in shares]
    out[-1] += n - sum(out)
    return out


def _dtype(case):
    return torch.float32 if case["dtype"] == "f32" else torch.bfloat16


def _spec(case):
    z = SIZES[case["size"]]
    W = z["width"]
    kind = case["kind"]
    if kind == "state_space":
        h, e, n, g = z["ssm"]
        return StateSpaceSpec(W, h, e, n, g, g, TAPS, EPS)
    if kind == "delta":
        h, d, rank = z["delta"]
        return DeltaRuleSpec(W, h, d, EPS, decay_rank=rank)
    if kind == "gla":
        h, d, v = z["mem"]
        return GatedLinearAttentionSpec(W, h, d, v, TAU, d ** -0.5, EPS)
    if kind == "memory":
        h, d, v = z["mem"]
        return MatrixMemorySpec(W, h, d, v, GATE_CAP, EPS)
    if kind == "latent":
        h, p, r, v, c, q, window = z["lat"]
        return LatentAttentionSpec(W, h, p, r, v, c, (p + r) ** -0.5, RopeSpec(r, ROTATION, exact_table=True, layout="interleaved"),
                                   latent_norm_eps=EPS, query_latent_dim=q, window=window, sink="sink")
    if kind == "attention":
        h, g, d, window = z["att"]
        return GeneralAttentionSpec(W, h, g, d, d, d ** -0.5, RopeSpec(d, ROTATION, exact_table=True, layout="interleaved"),
                                    score_cap=CAP, gate="element", window=window, keep_first=KEEP)
    experts, identity, top, size, shared = z["exp"]
    return RoutedExpertsSpec(W, experts, top, size, renormalize=True, activation="swiglu", renorm_eps=1e-20, weight_scale=2.0,
                             correction="correction", identity=identity, shared_size=shared)


def _weights(part, case, gen):
    """Random tensors for a part: matrices that keep the size of what they multiply; vectors as models have them after
    training (decay rates and step sizes spread over their usual ranges, gates mostly open)."""
    def normal(shape):
        return torch.randn(shape, generator=gen, device=DEVICE)

    def between(shape, low, high):
        return low + (high - low) * torch.rand(shape, generator=gen, device=DEVICE)

    out = {}
    for name, t in part.tensor_specs().items():
        shape = tuple(16 if d == -1 else d for d in t.shape)
        last = name.rsplit(".", 1)[-1]
        if last == "A_log":
            w = between(shape, 1.0, 16.0).log()
        elif last == "dt_bias":
            w = torch.expm1(between(shape, math.log(1e-3), math.log(0.1)).exp()).log()
        elif name.endswith("f.b"):
            w = between(shape, 3.0, 6.0)
        elif last == "conv":
            w = between(shape, -0.5, 0.5)
        elif last == "correction":
            w = 0.01 * normal(shape)
        elif t.init == "ones_normal":
            w = 1.0 + 0.1 * normal(shape)
        elif t.kind == "vector":
            w = 0.5 * normal(shape)
        else:
            w = normal(shape) * shape[-1] ** -0.5
        out[name] = w.to(_dtype(case))
    return out


def _model_config(case):
    z = SIZES[case["size"]]
    layers, heads, kv, dim, ff = z["model"]
    return dict(architectures=["Qwen3ForCausalLM"], vocab_size=VOCAB, hidden_size=z["width"], intermediate_size=ff,
                num_hidden_layers=layers, num_attention_heads=heads, num_key_value_heads=kv, head_dim=dim, rms_norm_eps=1e-6,
                rope_theta=1e6, max_position_embeddings=8192, tie_word_embeddings=False)


def _requests(cache, lengths, context):
    """Live requests with pages for their context and their new tokens."""
    out = []
    for i, n in enumerate(lengths):
        rc = cache.admit(("request", i))
        cache.grow(rc, context + n)
        rc.num_tokens = context
        out.append(rc)
    return out


def _pages(lengths, context):
    return sum(-(-(context + n) // PAGE) for n in lengths) + 1


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed * 7919 + 11)
    dtype, lengths, context = _dtype(case), _lengths(case), case["context"]
    if case["kind"] == "model":
        model = random_model(registry.config_from_dict(_model_config(case)), seed=seed, dtype=case["dtype"] if case["dtype"] == "bf16"
                             else "fp32", device="cuda:0")
        most = context + max(lengths)
        decode = case["phase"] == "decode"
        driver = make_driver(model, max_num_seqs=len(lengths), max_model_len=most + PAGE, block_size=PAGE, prefix_cache=False,
                             max_tokens_per_step=case["tokens"], cuda_graphs=decode, num_blocks=_pages(lengths, context) + 2 * len(lengths))
        rcs = _requests(driver.cache, lengths, context)
        for group in driver.cache.groups:
            for t in (group.k, group.v):
                t.copy_(torch.randn(t.shape, generator=gen, device=DEVICE, dtype=torch.float32).to(t.dtype))
        ids = torch.randint(0, VOCAB, (sum(lengths),), generator=gen, device=DEVICE).tolist()
        entries, at = [], 0
        for rc, n in zip(rcs, lengths):               # a decode step wants every token's logits, a prompt those of its last
            entries.append(StepEntry(rc, ids[at:at + n], (n - 1,)))
            at += n
        if decode:
            for _ in range(2):                        # the first step of a batch size runs eagerly, the second is captured
                driver.runner.step(entries)
        return {"case": case, "driver": driver, "entries": entries}

    ctx = BuildContext(dtype=dtype, device=torch.device("cuda:0"))
    part = build(FEED_FORWARDS if case["kind"] == "experts" else MIXERS, "part", _spec(case), "l0", ctx)
    tensors = _weights(part, case, gen)
    part.bind(tensors)
    x = torch.randn((sum(lengths), SIZES[case["size"]]["width"]), generator=gen, device=DEVICE).to(dtype)
    state = {"case": case, "part": part, "x": x, "step": None, "cache": None}
    if case["kind"] != "experts":
        cache = CacheManager([part.cache_need()], PAGE, _pages(lengths, context), len(lengths), False)
        view = cache.allocate_storage(dtype, torch.device("cuda:0"))[0]
        rcs = _requests(cache, lengths, context)
        classes = getattr(part, "tile_classes", None)
        builder = BatchBuilder(len(cache.groups), PAGE, classes(PAGE) if classes else [], torch.device("cuda:0"))
        state.update(step=builder.build([StepEntry(rc, [0] * n, ()) for rc, n in zip(rcs, lengths)]), cache=view, manager=cache,
                     requests=rcs)
        if case["kind"] in PAGED:
            for t in (view.k,) if view.k is view.v else (view.k, view.v):
                t.copy_(torch.randn(t.shape, generator=gen, device=DEVICE).to(t.dtype))
        elif context:                                 # what earlier tokens left
            view.state.copy_(0.3 * torch.randn(view.state.shape, generator=gen, device=DEVICE))
    if case["phase"] == "decode":
        before = view.state.clone() if case["kind"] in RECURRENT else None
        _call(state)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            state["out"] = _call(state)
        state["graph"] = graph
        if before is not None:
            view.state.copy_(before)
    return state


# ------------------------------------------------------------------------------------------------------- one pass
def _call(state):
    case, part = state["case"], state["part"]
    if case["kind"] == "experts":
        y = part.forward(state["x"], None)
    else:
        y = part.forward(state["x"], state["step"], state["cache"])
    # a result given as parts or rows to add up is added up, as the reader behind the layer does
    return y if isinstance(y, torch.Tensor) else y.tensor()


@torch.no_grad()
def run(state):
    case = state["case"]
    if case["kind"] == "model":
        return {"logits": state["driver"].runner.step(state["entries"])}
    if "graph" in state:
        state["graph"].replay()
        y = state["out"]
    else:
        if case["kind"] in RECURRENT and not case["context"]:
            state["cache"].state.zero_()              # a new prompt starts from a zeroed slot
        y = _call(state)
    out = {"y": y}
    if case["kind"] in RECURRENT:
        out["state"] = state["cache"].state
    elif case["kind"] in PAGED:
        out["keys"] = state["cache"].k
    return out


# ------------------------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    z, n, lengths, context = SIZES[case["size"]], case["tokens"], _lengths(case), case["context"]
    W, item, kind = z["width"], 4 if case["dtype"] == "f32" else 2, case["kind"]

    def seen(window, keep=0):                         # pairs of a query and a key that it sees
        total = 0
        for q in lengths:
            for p in range(context, context + q):
                total += p + 1 if not window else min(p + 1, window + keep)
        return total

    def keys(window):                                 # cache rows read, and those written
        return sum(min(context, (window or context) + q) + q for q in lengths)

    if kind == "model":
        layers, h, g, d, ff = z["model"]
        weights = layers * (W * (h + 2 * g) * d + h * d * W + 3 * W * ff)
        head = VOCAB * W
        kv = keys(0) * layers * 2 * g * d * item
        return {"bytes": (weights + head) * item + kv + 2 * len(lengths) * VOCAB,
                "flops": 2 * n * weights + 2 * len(lengths) * head + layers * 4 * h * d * seen(0)}
    if kind == "experts":
        e, identity, top, size, shared = z["exp"]
        pairs = n * top * e / (e + identity)
        hit = e * (1 - (1 - top / (e + identity)) ** n)
        matrices = 3 * W * size
        return {"bytes": (hit * matrices + 3 * W * shared + W * (e + identity)) * item + n * W * item + n * W * 4,
                "flops": 2 * pairs * matrices + 2 * n * 3 * W * shared + 2 * n * W * (e + identity)}
    if kind == "state_space":
        h, e, s, g = z["ssm"]
        weights, per, size = W * (2 * h * e + 2 * g * s + h) + W * h * e, 6 * h * e * s, h * e * s + (TAPS - 1) * (h * e + 2 * g * s)
    elif kind == "delta":
        h, d, rank = z["delta"]
        weights, per, size = W * (5 * h * d + rank) + h * d * rank + W * h * d, 8 * h * d * d, h * d * d
    elif kind == "gla":
        h, d, v = z["mem"]
        weights, per, size = W * (2 * h * d + 2 * h * v + 16) + 16 * h * d + W * h * v, 6 * h * d * v, h * d * v
    elif kind == "memory":
        h, d, v = z["mem"]
        weights, per, size = W * (2 * h * d + 2 * h * v + 2 * h) + W * h * v, 6 * h * d * v, h * d * v + h * d + h
    elif kind == "latent":
        h, p, r, v, c, q, window = z["lat"]
        weights = W * (q + c + r) + q * h * (p + r) + h * (p + v) * c + W * h * v
        return {"bytes": weights * item + 2 * n * W * item + keys(window) * (c + r) * item,
                "flops": 2 * n * weights + 2 * h * (2 * c + r) * seen(window)}
    else:
        h, g, d, window = z["att"]
        weights = W * (2 * h + 2 * g) * d + W * h * d
        return {"bytes": weights * item + 2 * n * W * item + keys(window) * 2 * g * d * item,
                "flops": 2 * n * weights + 4 * h * d * seen(window, KEEP)}
    reads = 2 if context else 1
    return {"bytes": weights * item + 2 * n * W * item + reads * len(lengths) * size * 4, "flops": 2 * n * weights + per * n}


def tolerance(case):
    """About four times what these layers show against 64-bit arithmetic: 1e-6 to 3e-6 in 32-bit; in bfloat16, where operands and
    results of the products are rounded in between, 2e-3 to 5e-3, the delta rule 8e-3, a whole model 1e-2."""
    if case["dtype"] == "f32":
        return {"rel": 1.2e-5}
    return {"rel": {"model": 4e-2, "delta": 3e-2}.get(case["kind"], 2e-2)}


# ------------------------------------------------------------------------------------------- the same in 64 bits
def _unit(y, eps):
    return y / torch.sqrt((y * y).mean(-1, keepdim=True) + eps)


def _silu(z):
    return z * torch.sigmoid(z)


def _turn(x, positions, base, dims):
    """Interleaved pairs of the first `dims` elements of x [T, H, D] turned by position * base^(-2i/dims)."""
    freq = base ** (-torch.arange(0, dims, 2, dtype=torch.float64, device=x.device) / dims)
    a = positions[:, None].double() * freq.float().double()
    cos, sin = torch.cos(a)[:, None], torch.sin(a)[:, None]
    u, v = x[..., 0:dims:2], x[..., 1:dims:2]
    return torch.cat([torch.stack([u * cos - v * sin, v * cos + u * sin], -1).flatten(-2), x[..., dims:]], -1)


def _halves(x, positions, base):
    half = x.shape[-1] // 2
    freq = base ** (-torch.arange(half, dtype=torch.float64, device=x.device) / half)
    a = positions[:, None].double() * freq
    cos, sin = torch.cos(a)[:, None], torch.sin(a)[:, None]
    u, v = x[..., :half], x[..., half:]
    return torch.cat([u * cos - v * sin, v * cos + u * sin], -1)


def _attend(q, k, v, first, scale, window=0, keep=0, cap=0.0, sink=None):
    """q [n, H, D] at positions first.. against k [T, G, D], v [T, G, E], head by head."""
    n, H = q.shape[:2]
    T, G = k.shape[:2]
    i = first + torch.arange(n, device=q.device)[:, None]
    j = torch.arange(T, device=q.device)[None]
    see = j <= i
    if window:
        see = see & ((i - j < window) | (j < keep))
    out = q.new_zeros((n, H, v.shape[2]))
    for h in range(H):
        s = q[:, h] @ k[:, h * G // H].T * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill(~see, -math.inf)
        top = s.max(-1, keepdim=True).values
        if sink is not None:
            top = torch.maximum(top, sink[h])
        e = torch.exp(s - top)
        total = e.sum(-1, keepdim=True) + (torch.exp(sink[h] - top) if sink is not None else 0.0)
        out[:, h] = e @ v[:, h * G // H] / total
    return out


def _scan(r, k, v, w, S, u=None, b=None):
    """o_t = S^T r_t after S <- diag(w) S - b (u^T S) + k v^T, over the tokens of one entry; S [H, D, V] is updated."""
    o = v.new_empty(v.shape)
    for t in range(r.shape[0]):
        dot = torch.einsum("hd,hdv->hv", u[t], S) if u is not None else None
        S.mul_(w[t][:, :, None])
        if dot is not None:
            S.baddbmm_(b[t][:, :, None], dot[:, None, :], alpha=-1.0)
        S.baddbmm_(k[t][:, :, None], v[t][:, None, :])
        torch.bmm(r[t][:, None, :], S, out=o[t][:, None, :])
    return o


def _exact_recurrent(case, part, W, x, state):
    """The heads before the output product for one entry, and the state row as it is left."""
    n, kind = x.shape[0], case["kind"]
    new = state.clone()
    if kind == "state_space":
        H, E, N, G = SIZES[case["size"]]["ssm"]
        inner, mats, ch = H * E, H * N * E, H * E + 2 * G * N
        row = x @ W["in"].T
        old = state[mats:].view(TAPS - 1, ch)
        xbc = torch.cat([old, row[:, inner:inner + ch]])
        new[mats:] = xbc[-(TAPS - 1):].reshape(-1)
        xbc = _silu(sum(xbc[j:j + n] * W["conv"][:, j] for j in range(TAPS)) + W["conv.b"])
        xs = xbc[:, :inner].view(n, H, E)
        B, C = (xbc[:, inner + i * G * N:inner + (i + 1) * G * N].view(n, G, N).repeat_interleave(H // G, 1) for i in range(2))
        dt = torch.nn.functional.softplus(row[:, inner + ch:] + W["dt_bias"])
        decay = torch.exp(-torch.exp(W["A_log"]) * dt)
        S = state[:mats].view(H, N, E).clone()
        o = _scan(C, dt[:, :, None] * B, xs, decay[:, :, None].expand(n, H, N), S) + W["D"][:, None] * xs
        new[:mats] = S.reshape(-1)
        o = (o.reshape(n, inner) * _silu(row[:, :inner])).view(n, G, inner // G)
        return _unit(o, EPS).reshape(n, inner) * W["norm"], new
    if kind == "delta":
        H, D, _ = SIZES[case["size"]]["delta"]
        r, k, v = ((x @ W[t].T).view(n, H, D) for t in ("r", "k", "v"))
        w = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(x @ W["w1"].T) @ W["w2"].T + W["w0"])).view(n, H, D)
        a = torch.sigmoid(x @ W["a"].T + W["a.b"]).view(n, H, D)
        u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        S = state.view(H, D, D).clone()
        o = _scan(r, k, v, w, S, u, a * u)
        return _unit(o, EPS).reshape(n, -1) * W["norm"] * torch.sigmoid(x @ W["g"].T), S.reshape(-1)
    H, D, V = SIZES[case["size"]]["mem"]
    q, k = ((x @ W[t].T).view(n, H, D) for t in ("q", "k"))
    v, q = (x @ W["v"].T).view(n, H, V), q * D ** -0.5
    if kind == "gla":
        a = torch.exp(torch.nn.functional.logsigmoid((x @ W["a1"].T) @ W["a2"].T + W["a2.b"]) / TAU).view(n, H, D)
        S = state.view(H, D, V).clone()
        o = _scan(q, k, v, a, S)
        return (_unit(o, EPS) * W["norm"]).reshape(n, -1) * _silu(x @ W["g"].T), S.reshape(-1)
    gi = GATE_CAP * torch.tanh((x @ W["i"].T + W["i.b"]) / GATE_CAP)
    gf = torch.nn.functional.logsigmoid(GATE_CAP * torch.tanh((x @ W["f"].T + W["f.b"]) / GATE_CAP))
    m, marks = state[H * D * (V + 1):].clone(), []
    keep, take = torch.empty_like(gi), torch.empty_like(gi)
    for t in range(n):
        new_m = torch.maximum(gf[t] + m, gi[t])
        keep[t], take[t], m = torch.exp(gf[t] + m - new_m), torch.exp(gi[t] - new_m), new_m
        marks.append(m)
    S = torch.cat([state[:H * D * V].view(H, D, V), state[H * D * V:H * D * (V + 1)].view(H, D, 1)], -1)
    o = _scan(q, take[:, :, None] * k, torch.cat([v, torch.ones_like(v[..., :1])], -1), keep[:, :, None].expand(n, H, D), S)
    den = torch.maximum(o[..., V].abs(), torch.exp(-torch.stack(marks))) + 1e-6
    new = torch.cat([S[..., :V].reshape(-1), S[..., V].reshape(-1), m])
    o = _unit(o[..., :V] / den[..., None], EPS).reshape(n, -1) * W["norm"]
    return o * torch.sigmoid(x @ W["g"].T), new


def _cached(pool, rc, context):
    """The first `context` rows of a request in a page pool [pages, page, heads, size], in 64 bits."""
    pages = torch.as_tensor([p if p >= 0 else 0 for p in rc.tables[0]], device=pool.device)
    return pool[pages].reshape(-1, *pool.shape[2:])[:context].double()


def _exact_paged(case, part, W, x, rc, k_pool, v_pool):
    n, context, z = x.shape[0], case["context"], SIZES[case["size"]]
    pos = context + torch.arange(n, device=x.device)
    if case["kind"] == "attention":
        H, G, D, window = z["att"]
        q = _turn((x @ W["q"].T).view(n, H, D), pos, ROTATION, D)
        k = torch.cat([_cached(k_pool, rc, context), _turn((x @ W["k"].T).view(n, G, D), pos, ROTATION, D)])
        v = torch.cat([_cached(v_pool, rc, context), (x @ W["v"].T).view(n, G, D)])
        o = _attend(q, k, v, context, D ** -0.5, window, KEEP, CAP).reshape(n, -1)
        return o * torch.sigmoid(x @ W["g"].T) @ W["o"].T
    H, P, R, E, C, Q, window = z["lat"]
    q = ((_unit(x @ W["dq"].T, EPS) * W["dq.norm"]) @ W["uq"].T).view(n, H, P + R)
    down = x @ W["dkv"].T
    row = torch.cat([(_unit(down[:, :C], EPS) * W["dkv.norm"])[:, None], _turn(down[:, None, C:], pos, ROTATION, R)], -1)
    row = torch.cat([_cached(k_pool, rc, context), row])
    q = torch.cat([torch.einsum("nhp,hpc->nhc", q[..., :P], W["uk"].view(H, P, C)), _turn(q[..., P:], pos, ROTATION, R)], -1)
    o = _attend(q, row, row[..., :C], context, (P + R) ** -0.5, window, 0, 0.0, W["sink"])
    return torch.einsum("nhc,hec->nhe", o, W["uv"].view(H, E, C)).reshape(n, -1) @ W["o"].T


def _exact_experts(case, W, x):
    experts, identity, top, size, shared = SIZES[case["size"]]["exp"]
    glu = lambda u, p: (_silu(u @ W[f"{p}gate"].double().T) * (u @ W[f"{p}up"].double().T)) @ W[f"{p}down"].double().T
    s = torch.softmax(x @ W["router"].double().T, -1)
    ids = (s + W["correction"].double()).topk(top, -1).indices
    w = s.gather(1, ids)
    w = w / (w.sum(-1, keepdim=True) + 1e-20) * 2.0
    out = glu(x, "shared.")
    for e in range(experts + identity):
        rows = (ids == e).any(-1)
        if rows.any():
            y = glu(x[rows], f"e{e}.") if e < experts else x[rows]
            out[rows] += (w * (ids == e)).sum(-1)[rows][:, None] * y
    return out


def _exact_model(case, seed):
    state = prepare(case, seed)
    driver, entries = state["driver"], state["entries"]
    config = _model_config(case)
    H, G, D, context = (config["num_attention_heads"], config["num_key_value_heads"], config["head_dim"], case["context"])
    W = random_tensors(driver.model.tensor_specs(), seed, _dtype(case), "cuda:0")
    norm = lambda y, name: _unit(y, 1e-6) * W[name].double()
    times = lambda y, name: y @ W[name].double().T
    group, logits = driver.cache.groups[0], []
    for e in entries:
        h = W["model.embed_tokens.weight"][torch.as_tensor(e.tokens, device=DEVICE)].double()
        n = h.shape[0]
        pos = context + torch.arange(n, device=DEVICE)
        for i in range(config["num_hidden_layers"]):
            p = f"model.layers.{i}."
            x = norm(h, p + "input_layernorm.weight")
            q, k, v = (times(x, f"{p}self_attn.{t}_proj.weight").view(n, -1, D) for t in "qkv")
            q, k = (_halves(_unit(y, 1e-6) * W[f"{p}self_attn.{t}_norm.weight"].double(), pos, 1e6) for y, t in ((q, "q"), (k, "k")))
            k = torch.cat([_cached(group.k[i], e.cache, context), k])
            v = torch.cat([_cached(group.v[i], e.cache, context), v])
            h = h + times(_attend(q, k, v, context, D ** -0.5).reshape(n, -1), f"{p}self_attn.o_proj.weight")
            x = norm(h, p + "post_attention_layernorm.weight")
            h = h + times(_silu(times(x, p + "mlp.gate_proj.weight")) * times(x, p + "mlp.up_proj.weight"), p + "mlp.down_proj.weight")
        logits.append(times(norm(h[-1:], "model.norm.weight"), "lm_head.weight"))
    return {"logits": torch.cat(logits)}


@torch.no_grad()
def exact(case, seed):
    if case["kind"] == "model":
        return _exact_model(case, seed)
    state = prepare(case, seed)
    part, x = state["part"], state["x"].double()
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed * 7919 + 11)
    W = {name.removeprefix(part.prefix + "."): t if case["kind"] == "experts" else t.double()
         for name, t in _weights(part, case, gen).items()}
    if case["kind"] == "experts":
        return {"y": _exact_experts(case, W, x)}
    ys, rows, at = [], [], 0
    before = state["cache"].state.double() if case["kind"] in RECURRENT else None
    for e, n in enumerate(_lengths(case)):
        part_x = x[at:at + n]
        at += n
        if before is not None:
            heads, row = _exact_recurrent(case, part, W, part_x, before[state["requests"][e].slot])
            ys.append(heads @ W["o"].T)
            rows.append((state["requests"][e].slot, row))
        else:
            ys.append(_exact_paged(case, part, W, part_x, state["requests"][e], state["cache"].k, state["cache"].v))
    out = {"y": torch.cat(ys)}
    if before is None:
        out["keys"] = None
    else:
        out["state"] = before.clone()
        for slot, row in rows:
            out["state"][slot] = row
    return out
