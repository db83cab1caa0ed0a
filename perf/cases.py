"""The work that programs built on this package have it do, as cases that can be timed and compared.

Most cases are one part of a layer (a mixer or a feed-forward, from the part registries) run over the tokens of one step,
the way the engine runs it: the part is attached to a runtime and bound to weights once, the step's integer arrays and the
cache are laid out once, and a pass writes the residual stream (as the embedding does at a step's start), puts the
sequences' state where it stood before the step, and runs the part's ``forward`` with dependent launches on.  One case is a
whole model: prompts as one step, then decode steps with given tokens through ``Engine.decode_sample``, logits of each.

Sizes are those of the package's benchmark: Qwen3-8B and 0.6B layers, and the "lite" and "small" sizes of the other designs.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import zlm_b200  # noqa: F401  (fills the registries)
from zlm_b200 import Engine, StepEntry
from zlm_b200.cache import KVCache
from zlm_b200.config.spec import ScheduleEntry
from zlm_b200.engine.batch import MetaLayout, MetaStager, make_context, plan_step
from zlm_b200.kernels import PAGE_TOKENS, get_kernels
from zlm_b200.parts.base import Runtime
from zlm_b200.registry import FEED_FORWARDS, MIXERS, config_from_dict, lookup
from zlm_b200.sampling import SamplingParams

DEVICE = "cuda:0"
EPS = 1e-6
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}

# width of the model and sizes of the part, by part and size; see ``bench.py`` for the designs they belong to
GQA = {"8b": (4096, 32, 8), "0.6b": (1024, 16, 8), "lite": (2048, 16, 4)}                       # width, heads, kv heads
LATENT = {"lite": (2048, 16, 128, 64, 128, 512), "small": (1024, 8, 64, 32, 64, 256)}           # heads, dim, rot, vdim, rank
CONV = {"lite": (2048, 16, 4, 4096), "small": (1024, 8, 2, 512)}                                # heads, kv heads, window
RETENTION = {"lite": (2048, 16), "small": (1024, 8), "wide": (4096, 32)}                        # heads (128 x 128)
GLA = {"lite": (2048, 8), "small": (1024, 4), "wide": (4096, 16)}                               # heads (64 x 128)
RGLRU = {"lite": (2048, 8), "small": (1024, 4), "wide": (4096, 16)}                             # blocks of 256 channels
MLSTM = {"lite": (2048, 16), "small": (1024, 8), "wide": (4096, 32)}                            # heads (128 x 128)
EXPERTS = {"lite": (2048, 60, 4, 6, 768, 8, 4), "small": (1024, 30, 2, 4, 512, 4, 2)}           # experts, identity, top, ff, groups, keep
SIZES = {"gqa": GQA, "latent": LATENT, "conv": CONV, "retention": RETENTION, "gla": GLA, "rglru": RGLRU, "mlstm": MLSTM,
         "experts": EXPERTS}
MODEL = {"layers": 28, "width": 1024, "heads": 16, "kv": 8, "ff": 3072, "vocab": 151936}        # Qwen3-0.6B
TAPS = 4


def listed():
    def part(name, kind, size, tokens, seqs=1, start=0, dtype="bfloat16"):
        return {"name": name, "kind": kind, "size": size, "tokens": tokens, "seqs": seqs, "start": start, "dtype": dtype}
    return [
        # a chat server's smallest model: eight short prompts as one step, then captured decode steps (launch-bound)
        {"name": "model_b8_prompts_then_steps", "kind": "model", "size": "0.6b", "tokens": 8 * 40, "seqs": 8, "start": 0,
         "steps": 12, "dtype": "bfloat16"},
        # the headline model's attention layer over one ordinary prompt
        part("gqa_8b_prompt_2048", "gqa", "8b", 2048),
        # 64 prompts of unequal lengths as one step: the largest batch that the benchmark prefills
        part("gqa_0.6b_64_unequal_prompts", "gqa", "0.6b", 61037, seqs=64),
        # the true 32-bit path (trace replay, numerics work): a chunk of a prompt over a cached beginning
        part("gqa_lite_float32_chunk", "gqa", "lite", 509, start=515, dtype="float32"),
        # latent attention over a whole prompt (records to the cache, attention unfolded)
        part("latent_lite_prompt_2048", "latent", "lite", 2048),
        # attention behind short convolutions, three prompts of odd lengths
        part("conv_attention_lite_3_prompts", "conv", "lite", 2999, seqs=3),
        # linear attention with fixed decays: one ordinary prompt
        part("retention_lite_prompt_2048", "retention", "lite", 2048),
        # linear attention with a decay per channel and token: the next chunk of a long prompt
        part("gla_lite_chunk_2048", "gla", "lite", 2048, start=4096),
        # the recurrent gated unit over two unequal prompts
        part("rglru_lite_2_prompts", "rglru", "lite", 1999, seqs=2),
        # the matrix memory over four unequal prompts
        part("mlstm_lite_4_prompts", "mlstm", "lite", 3001, seqs=4),
        # routed experts in a prompt (sorted, grouped) ...
        part("experts_lite_prompt_2048", "experts", "lite", 2048),
        # ... and in a decode step of one sequence: the smallest call, a few microseconds of weights
        part("experts_small_one_token", "experts", "small", 1),
    ]


def draw(rng):
    kind = rng.choice(["gqa", "gqa", "latent", "conv", "retention", "gla", "rglru", "mlstm", "experts", "experts", "model"])
    if kind == "model":
        seqs = rng.randint(1, 12)
        return {"kind": kind, "size": "0.6b", "tokens": seqs * rng.randint(9, 60), "seqs": seqs, "start": 0,
                "steps": rng.randint(6, 14), "dtype": "bfloat16"}
    size = rng.choice(sorted(SIZES[kind]))
    tokens = min(int(round(2 ** rng.uniform(0, 13))),
                 (20_000_000 if kind in ("gqa", "latent", "conv") else 12_000_000) // SIZES[kind][size][0])
    dtype = "bfloat16"
    if kind != "latent" and rng.random() < 0.08:          # (the 32-bit path is for replays, chunks of some hundred tokens)
        dtype, tokens = "float32", max(1, int(round(2 ** rng.uniform(0, 9.5))))
    seqs = rng.randint(1, min(16, tokens))
    start = rng.randint(1, 4096) if kind in ("gqa", "retention", "gla", "rglru", "mlstm") and rng.random() < 0.4 else 0
    if kind == "gqa":
        start = min(start, 49152 // seqs)
    return {"kind": kind, "size": size, "tokens": tokens, "seqs": seqs, "start": start, "dtype": dtype}


# ---------------------------------------------------------------------------------------------- inputs and weights
def lengths(case):
    """New tokens of every sequence: unequal wherever there are more tokens than sequences."""
    T, R = case["tokens"], case["seqs"]
    if case["kind"] == "model" or T == R:
        return [T // R] * R
    w = np.random.RandomState(T * 131 + R).uniform(0.2, 1.8, R)
    n = np.maximum(1, np.floor(w / w.sum() * (T - R))).astype(int)
    while n.sum() != T:
        n[int(np.argmin(n)) if n.sum() < T else int(np.argmax(n))] += 1 if n.sum() < T else -1
    return [int(v) for v in n]


class Draws:
    """Random numbers by seed, always drawn in the same order."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEVICE).manual_seed(int(seed) * 2 + 1)

    def normal(self, shape, scale=1.0, shift=0.0, dtype=torch.float32):
        return (torch.randn(shape, generator=self.g, device=DEVICE) * scale + shift).to(dtype)

    def tokens(self, shape, n):
        return torch.randint(0, n, shape, generator=self.g, device=DEVICE).tolist()


def decays(heads):
    return [1.0 - 2.0 ** (-5 - 5 * h / max(1, heads - 1)) for h in range(heads)]


def part_spec(case):
    """(registry, name, width, parameters) of the case's part."""
    s = SIZES[case["kind"]][case["size"]]
    rot = {"kind": "rope_half_split", "theta": 1e4, "head_dim": 128, "n_rot": 128}
    if case["kind"] == "gqa":
        return MIXERS, "gqa_attention", s[0], dict(num_heads=s[1], num_kv_heads=s[2], head_dim=128, qk_norm=True,
                                                   qk_norm_eps=EPS, position=dict(rot, theta=1e6))
    if case["kind"] == "latent":
        return MIXERS, "latent_attention", s[0], dict(
            num_heads=s[1], head_dim=s[2], rot_dim=s[3], v_dim=s[4], kv_rank=s[5], scale=(s[2] + s[3]) ** -0.5, norm_eps=EPS,
            position={"kind": "rope_interleaved", "base": 1e4, "dims": s[3]})
    if case["kind"] == "conv":
        return MIXERS, "conv_attention", s[0], dict(num_heads=s[1], num_kv_heads=s[2], head_dim=128, v_dim=128, conv_taps=TAPS,
                                                    scale=128 ** -0.5, norm_eps=EPS, window=s[3])
    if case["kind"] == "retention":
        return MIXERS, "retention", s[0], dict(num_heads=s[1], head_dim=128, v_dim=128, decay=decays(s[1]), norm_eps=EPS,
                                               position=rot)
    if case["kind"] == "gla":
        return MIXERS, "gated_linear_attention", s[0], dict(num_heads=s[1], head_dim=64, v_dim=128, tau=8.0, norm_eps=EPS, rank=32)
    if case["kind"] == "rglru":
        return MIXERS, "rglru", s[0], dict(width=s[0], blocks=s[1], conv_taps=TAPS)
    if case["kind"] == "mlstm":
        return MIXERS, "mlstm", s[0], dict(num_heads=s[1], head_dim=128, v_dim=128, gate_cap=15.0, norm_eps=EPS)
    if case["kind"] == "experts":
        return FEED_FORWARDS, "routed_experts", s[0], dict(
            num_experts=s[1], identity=s[2], top_k=s[3], expert_ff=s[4], groups=s[5], keep=s[6], score="softmax",
            weight_on="output", activation="swiglu", correction=True, route_scale=2.5)
    raise ValueError(case["kind"])


def part_inputs(case, seed, part=None):
    """Everything random of a case, the same numbers whoever asks: weights by name in the dtype that the part is given, the
    part's input (a normed activation), the residual stream, what is cached of earlier tokens, the sequences' state."""
    if part is None:
        table, name, width, params = part_spec(case)
        part = lookup(table, "part", name)(hidden_size=width, **params)
    dt, width, d = DTYPES[case["dtype"]], SIZES[case["kind"]][case["size"]][0], Draws(seed)
    weights = {}
    for name, p in sorted(part.param_specs().items()):
        shape = p.concrete_shape()
        one = 1.0 if p.init == "one_plus_normal" else 0.0
        # matrices as trained ones are scaled; biases, which random models leave at zero, small and not zero; the taps of a
        # convolution of the order of one; what decides a recurrent unit's reach spread over its range
        scale = 0.5 if "conv.weight" in name else 1.0 if name == "lam" else 0.02
        keep32 = p.kind == "vector"
        weights[name] = d.normal(shape, scale, one, torch.float32 if keep32 else dt)
    x = d.normal((case["tokens"], width), dtype=dt)
    residual = d.normal((case["tokens"], width), 0.02)                # (as an embedding of the weights' scale leaves it)
    R, start = case["seqs"], case["start"]
    cached = state = None
    if start and case["kind"] == "gqa":
        kv = SIZES["gqa"][case["size"]][2]
        cached = (d.normal((R, start, kv, 128), dtype=dt), d.normal((R, start, kv, 128), dtype=dt))
    elif start:
        s = SIZES[case["kind"]][case["size"]]
        if case["kind"] == "rglru":
            state = (d.normal((R, TAPS, s[0])),)
        elif case["kind"] == "mlstm":
            state = (d.normal((R, s[1], 128, 128), 0.3), d.normal((R, s[1], 128)), d.normal((R, s[1])).abs())
        else:
            state = (d.normal((R, s[1], 64 if case["kind"] == "gla" else 128, 128)),)
    return {"weights": weights, "x": x, "residual": residual, "cached": cached, "state": state}


def model_inputs(case, seed):
    d, m = Draws(seed), MODEL
    H, Q, KV, F = m["width"], m["heads"] * 128, m["kv"] * 128, m["ff"]
    w = {"model.embed_tokens.weight": d.normal((m["vocab"], H), 0.02, dtype=torch.bfloat16), "model.norm.weight": d.normal((H,), 0.02, 1.0)}
    for i in range(m["layers"]):
        p = f"model.layers.{i}."
        for name, shape in (("self_attn.q_proj", (Q, H)), ("self_attn.k_proj", (KV, H)), ("self_attn.v_proj", (KV, H)),
                            ("self_attn.o_proj", (H, Q)), ("mlp.gate_proj", (F, H)), ("mlp.up_proj", (F, H)), ("mlp.down_proj", (H, F))):
            w[p + name + ".weight"] = d.normal(shape, 0.02, dtype=torch.bfloat16)
        for name, n in (("input_layernorm", H), ("post_attention_layernorm", H), ("self_attn.q_norm", 128), ("self_attn.k_norm", 128)):
            w[p + name + ".weight"] = d.normal((n,), 0.02, 1.0)
    prompts = [d.tokens((n,), m["vocab"]) for n in lengths(case)]
    steps = d.tokens((case["steps"], case["seqs"]), m["vocab"])
    return w, prompts, steps


# ---------------------------------------------------------------------------------------------- prepare and run
def prepare(case, seed):
    if case["kind"] == "model":
        w, prompts, steps = model_inputs(case, seed)
        m = MODEL
        config = config_from_dict({
            "architectures": ["Qwen3ForCausalLM"], "num_hidden_layers": m["layers"], "hidden_size": m["width"],
            "num_attention_heads": m["heads"], "num_key_value_heads": m["kv"], "head_dim": 128, "intermediate_size": m["ff"],
            "vocab_size": m["vocab"], "rope_theta": 1e6, "rms_norm_eps": EPS, "tie_word_embeddings": True,
            "max_position_embeddings": 40960, "hidden_act": "silu"})
        engine = Engine(config, w, torch.bfloat16, DEVICE, max_tokens=case["seqs"] * 512, max_batch=16, max_step_tokens=8192)
        return {"engine": engine, "prompts": prompts, "steps": steps}
    table, name, width, params = part_spec(case)
    dt = DTYPES[case["dtype"]]
    rt = Runtime(torch.device(DEVICE), dt, get_kernels())
    part = lookup(table, "part", name)(hidden_size=width, **params)
    part.attach(rt)
    given = part_inputs(case, seed, part)
    weights = given.pop("weights")
    part.bind(weights)
    news, start, R = lengths(case), case["start"], case["seqs"]
    is_mixer = table is MIXERS
    pages = sum(-(-(n + start) // PAGE_TOKENS) for n in news)
    cache = KVCache([ScheduleEntry(0)], [part.cache_request() if is_mixer else None], [part.state_request() if is_mixer else None],
                    pages * PAGE_TOKENS, R, max(news) + start, dt, rt.device)
    slots = [cache.alloc_slot() for _ in news]
    if start:
        before = [(s, start) for s in slots]
        cache.reserve(before)
        cache.commit(before)
    cache.reserve(list(zip(slots, news)))
    layout = MetaLayout(case["tokens"], R)
    stager = MetaStager(layout, rt.device)
    arrays, T, R, _ = plan_step([StepEntry(s, [0] * n) for s, n in zip(slots, news)], cache.lengths, 1, layout)
    stager.upload(arrays, T, R)
    ctx = make_context(stager, arrays, T, R, rt.ws)
    io = cache.ios[0]
    if given["cached"] is not None:
        where = torch.arange(start, device=DEVICE)
        for r, s in enumerate(slots):
            page = io.cache.block_table[s].long()[where // PAGE_TOKENS]
            for j in (0, 1):
                io.cache.pool[page, j, :, where % PAGE_TOKENS] = given["cached"][j][r]
    held = io.state if isinstance(io.state, tuple) else () if io.state is None else (io.state,)
    states = []
    for i, t in enumerate(held):
        first = t.clone()
        if given["state"] is not None:
            for r, s in enumerate(slots):
                first[s] = given["state"][i][r].view(first[s].shape)
        states.append((t, first))
    return {"part": part, "x": given["x"], "residual": given["residual"], "stream": torch.empty_like(given["residual"]),
            "ctx": ctx, "io": io, "states": states, "keep": (cache, stager)}


def run(state):
    if "engine" in state:
        engine, out = state["engine"], []
        slots = [engine.new_sequence() for _ in state["prompts"]]
        logits = engine.step([StepEntry(s, p, [len(p) - 1]) for s, p in zip(slots, state["prompts"])])
        out.append(logits.clone())
        for tokens in state["steps"]:
            engine.decode_sample(slots, tokens, GREEDY, range(len(slots)))
            out.append(engine.last_logits.clone())
        for s in slots:
            engine.release(s)
        return out
    part, ctx, io, stream = state["part"], state["ctx"], state["io"], state["stream"]
    k = part.rt.k
    ctx.extras.clear()                      # what the layers of one step share is made anew in every step
    k.forget_pending()
    stream.copy_(state["residual"])
    for held, first in state["states"]:
        held.copy_(first)
    k.set_pdl(True)
    try:
        if hasattr(part, "state_request"):
            part.forward(state["x"], stream, ctx, io)
        else:
            part.forward(state["x"], stream, ctx)
        k.flush_shares()
    finally:
        k.set_pdl(False)
    return {"stream": stream, "state": [held for held, _ in state["states"]]}


GREEDY = SamplingParams()


# ---------------------------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    T, R = case["tokens"], case["seqs"]
    if case["kind"] == "model":
        m, steps = MODEL, case["steps"]
        H, Q, KV, F, L, V = m["width"], m["heads"] * 128, m["kv"] * 128, m["ff"], m["layers"], m["vocab"]
        layer = H * (Q + 2 * KV) + Q * H + 3 * H * F
        n = T // R
        ctx = [n + j + 1 for j in range(steps)]
        attended = R * (n * (n + 1) // 2 + sum(ctx))
        nbytes = (1 + steps) * 2 * (L * layer + V * H) + 2 * L * 2 * KV * R * (n + sum(ctx)) + (1 + steps) * R * V * 4
        return {"bytes": nbytes, "flops": 2 * L * layer * (T + R * steps) + 2 * V * H * R * (1 + steps) + 4 * L * Q * attended}
    table, name, W, params = part_spec(case)
    part = lookup(table, "part", name)(hidden_size=W, **params)
    size = 2 if case["dtype"] == "bfloat16" else 4
    s = SIZES[case["kind"]][case["size"]]
    news, start = lengths(case), case["start"]
    weights = sum(math.prod(p.concrete_shape()) for p in part.param_specs().values())
    flops = 2 * T * sum(math.prod(p.concrete_shape()) for p in part.param_specs().values() if len(p.shape) == 2 and p.shape[1] > TAPS)
    nbytes = weights * size + T * W * (size + 8)                      # weights, the input, the stream read and written

    def pairs(window=0):
        full = sum(n * (n + 1) // 2 + n * start for n in news)
        return full - sum((n - window) * (n - window + 1) // 2 for n in news if window and n > window)
    if case["kind"] == "gqa":
        flops += 4 * s[1] * 128 * pairs()
        nbytes += 2 * s[2] * 128 * size * (T + R * start)
    elif case["kind"] == "latent":
        flops += 2 * s[1] * (s[2] + s[3] + s[4]) * pairs()
        nbytes += (s[5] + s[3]) * size * T
    elif case["kind"] == "conv":
        flops += 4 * s[1] * 128 * pairs(s[3]) + 2 * TAPS * T * (s[1] + 2 * s[2]) * 128
        nbytes += 2 * s[2] * 128 * size * T
    elif case["kind"] in ("retention", "mlstm", "gla"):
        per = s[1] * 128 * (64 if case["kind"] == "gla" else 128)
        flops += 4 * per * T                                          # k v^T into the state, the state read by q
        nbytes += 8 * per * R
    elif case["kind"] == "rglru":
        flops += 2 * T * (2 * 256 * W) + 2 * TAPS * T * W
        nbytes += 8 * TAPS * W * R
    elif case["kind"] == "experts":
        E, top, F = s[1], s[3], s[4]
        chosen = min(E, T * top)                                       # experts that this many choices reach at most
        flops = 2 * T * W * (E + s[2]) + 2 * T * top * 3 * W * F * E // (E + s[2])
        nbytes = (E + s[2]) * W * size + chosen * 3 * W * F * size + T * W * (size + 8)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # Measured against ``exact`` (which rounds nothing between the input and the result), one run of the listed cases and six
    # drawn ones: whole model 6.7e-3; attention and latent attention 3.1e-3 to 4.4e-3, retention, decayed linear attention and
    # the recurrent unit 3.1e-3 to 3.9e-3, matrix memory 5.1e-3, experts 0.9e-3 to 3.9e-3; 32-bit attention 4.4e-6.  About
    # four times that; experts a little more, since a choice between two experts of equal score is one row's whole difference.
    if case["dtype"] == "float32":
        return {"rel": 2e-5}
    return {"rel": {"model": 2.5e-2, "mlstm": 2e-2, "experts": 2e-2}.get(case["kind"], 1.5e-2)}


# ---------------------------------------------------------------------------------------------- the same in 64 bits
def _unit(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def _turn_half(x, pos, theta):
    half = x.shape[-1] // 2
    a = pos.double()[:, None, None] * torch.pow(torch.tensor(theta, dtype=torch.float64, device=x.device),
                                                -torch.arange(half, dtype=torch.float64, device=x.device) / half)
    u, v = x[..., :half], x[..., half:]
    return torch.cat([u * torch.cos(a) - v * torch.sin(a), v * torch.cos(a) + u * torch.sin(a)], -1)


def _turn_pairs(x, pos, theta):
    half = x.shape[-1] // 2
    a = pos.double()[:, None, None] * torch.pow(torch.tensor(theta, dtype=torch.float64, device=x.device),
                                                -torch.arange(half, dtype=torch.float64, device=x.device) / half)
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * torch.cos(a) - v * torch.sin(a), v * torch.cos(a) + u * torch.sin(a)], -1).flatten(-2)


def _attend(q, k, v, scale, start, window=0, sink=False):
    """q [n, H, D] at positions start ..; k [start + n, G, D], v [start + n, G, V]; heads in groups over G."""
    n, H = q.shape[:2]
    G, total = k.shape[1], k.shape[0]
    out = torch.empty((n, H, v.shape[2]), dtype=q.dtype, device=q.device)
    j = torch.arange(total, device=q.device)
    rows = max(1, (1 << 27) // total)
    for h in range(H):
        kh, vh = k[:, h * G // H], v[:, h * G // H]
        for a in range(0, n, rows):
            i = torch.arange(start + a, start + min(n, a + rows), device=q.device)[:, None]
            s = q[a:a + rows, h] @ kh.T * scale
            s = s.masked_fill((j > i) | ((j <= i - window) if window else (j < 0)), -math.inf)
            if sink:
                s = torch.cat([s, torch.zeros_like(s[:, :1])], 1)
            p = torch.softmax(s, 1)
            out[a:a + rows, h] = p[:, :total] @ vh
    return out


def _conv(x, w, before):
    """x [n, C], w [C, taps], before [taps - 1, C] -> [n, C]."""
    ext = torch.cat([before, x])
    return sum(ext[j:j + x.shape[0]] * w[:, j] for j in range(w.shape[1]))


def exact(case, seed):
    if case["kind"] == "model":
        return _exact_model(case, seed)
    given = part_inputs(case, seed)
    w = {n: t.double() for n, t in given["weights"].items()}
    x, residual = given["x"].double(), given["residual"].double()
    s, start = SIZES[case["kind"]][case["size"]], case["start"]
    if case["kind"] == "experts":
        return {"stream": residual + _experts(x, w, s), "state": []}
    outs, states = [], []
    at = 0
    for r, n in enumerate(lengths(case)):
        h, pos = x[at:at + n], torch.arange(start, start + n, device=x.device)
        first = [t[r].double() for t in given["state"]] if given["state"] is not None else None
        if case["kind"] == "gqa":
            q = _turn_half(_unit((h @ w["q_proj.weight"].T).view(n, -1, 128)) * w["q_norm.weight"], pos, 1e6)
            k = _turn_half(_unit((h @ w["k_proj.weight"].T).view(n, -1, 128)) * w["k_norm.weight"], pos, 1e6)
            v = (h @ w["v_proj.weight"].T).view(n, -1, 128)
            if start:
                k, v = (torch.cat([c[r].double(), t]) for c, t in zip(given["cached"], (k, v)))
            y, kept = _attend(q, k, v, 128 ** -0.5, start).flatten(1) @ w["o_proj.weight"].T, []
        elif case["kind"] == "latent":
            W, H, dn, dr, dv, rank = s
            q = (h @ w["q"].T).view(n, H, dn + dr)
            rec = h @ w["dkv"].T
            c = _unit(rec[:, :rank]) * w["dkv.norm"]
            kr = _turn_pairs(rec[:, None, rank:], pos, 1e4).expand(n, H, dr)
            k = torch.cat([(c @ w["uk"].T).view(n, H, dn), kr], -1)
            q = torch.cat([q[..., :dn], _turn_pairs(q[..., dn:], pos, 1e4)], -1)
            y = _attend(q, k, (c @ w["uv"].T).view(n, H, dv), (dn + dr) ** -0.5, 0).flatten(1) @ w["o"].T
            kept = []
        elif case["kind"] == "conv":
            raw = [h @ w[f"{c}_proj.weight"].T for c in "qkv"]
            q, k, v = (_conv(t, w[f"{c}_conv.weight"], torch.zeros(TAPS - 1, t.shape[1], dtype=t.dtype, device=t.device)).view(n, -1, 128)
                       for t, c in zip(raw, "qkv"))
            y = _attend(_unit(q), _unit(k), v, 128 ** -0.5, 0, s[3], sink=True).flatten(1)
            y = (y * torch.sigmoid(h @ w["g_proj.weight"].T)) @ w["o_proj.weight"].T
            full = torch.cat([torch.zeros(TAPS - 1, sum(t.shape[1] for t in raw), dtype=x.dtype, device=x.device), torch.cat(raw, 1)])
            kept = [full[-(TAPS - 1):]]
        elif case["kind"] == "rglru":
            y, kept = _rglru(h, w, s, first)
        else:
            y, kept = _matrix_state(case["kind"], h, w, s, first, pos)
        outs.append(y)
        states.append(kept)
        at += n
    slots = range(case["seqs"])                                       # (a fresh cache hands its slots out in order)
    return {"stream": residual + torch.cat(outs), "state": [torch.stack([states[r][i] for r in slots]) for i in range(len(states[0]))]}


def _matrix_state(kind, h, w, s, first, pos):
    n, H, D, V = h.shape[0], s[1], 64 if kind == "gla" else 128, 128
    q, k = ((h @ w[f"{c}_proj.weight"].T).view(n, H, D) for c in "qk")
    v = (h @ w["v_proj.weight"].T).view(n, H, V)
    zeros = torch.zeros((H, D, V), dtype=h.dtype, device=h.device)
    S = zeros if first is None else first[0]
    o = torch.empty((n, H, V), dtype=h.dtype, device=h.device)
    if kind == "retention":
        q, k = _turn_half(q, pos, 1e4), _turn_half(k, pos, 1e4) * D ** -0.5
        d = torch.tensor(decays(H), dtype=torch.float32, device=h.device).double()[:, None, None]
        for t in range(n):
            S = d * S + k[t, :, :, None] * v[t, :, None]
            o[t] = (S * q[t, :, :, None]).sum(1)
        z = h @ w["g_proj.weight"].T
        return (_unit(o).flatten(1) * z * torch.sigmoid(z)) @ w["o_proj.weight"].T, [S]
    if kind == "gla":
        z = h @ w["a_down.weight"].T @ w["a_up.weight"].T + w["a_up.bias"]
        a = torch.exp(torch.nn.functional.logsigmoid(z) / 8.0).view(n, H, D, 1)
        q = q * D ** -0.5
        for t in range(n):
            S = a[t] * S + k[t, :, :, None] * v[t, :, None]
            o[t] = (S * q[t, :, :, None]).sum(1)
        z = h @ w["g_proj.weight"].T
        return ((_unit(o) * w["norm.weight"]).flatten(1) * z * torch.sigmoid(z)) @ w["o_proj.weight"].T, [S]
    q = q * D ** -0.5
    i, f = (15.0 * torch.tanh((h @ w[f"{c}_gate.weight"].T + w[f"{c}_gate.bias"]) / 15.0) for c in "if")
    f = torch.nn.functional.logsigmoid(f)
    N, m = (zeros[:, :, 0], zeros[:, 0, 0]) if first is None else first[1:]
    for t in range(n):
        new = torch.maximum(f[t] + m, i[t])
        a, b = torch.exp(f[t] + m - new), torch.exp(i[t] - new)
        S = a[:, None, None] * S + b[:, None, None] * k[t, :, :, None] * v[t, :, None]
        N, m = a[:, None] * N + b[:, None] * k[t], new
        low = torch.maximum((N * q[t]).sum(1).abs(), torch.exp(-m)) + 1e-6
        o[t] = (S * q[t, :, :, None]).sum(1) / low[:, None]
    y = _unit(o).flatten(1) * w["norm.weight"] * torch.sigmoid(h @ w["g_proj.weight"].T)
    return y @ w["o_proj.weight"].T, [S, N, m]


def _rglru(h, w, s, first):
    n, W, B = h.shape[0], s[0], s[1]
    gelu = torch.nn.functional.gelu
    y = gelu(h @ w["y_proj.weight"].T + w["y_proj.bias"], approximate="tanh")
    raw = h @ w["x_proj.weight"].T + w["x_proj.bias"]
    before = torch.zeros((TAPS - 1, W), dtype=h.dtype, device=h.device) if first is None else first[0][1:]
    u = _conv(raw, w["conv.weight"], before) + w["conv.bias"]
    ub = u.view(n, B, W // B)
    r, i = (torch.sigmoid(torch.einsum("nbi,boi->nbo", ub, w[f"{c}_gate.weight"]) + w[f"{c}_gate.bias"]).flatten(1) for c in "ai")
    log_a = -8.0 * r * torch.nn.functional.softplus(w["lam"])
    a, b = torch.exp(log_a), torch.sqrt(-torch.expm1(2 * log_a)) * i * u
    S = torch.zeros((W,), dtype=h.dtype, device=h.device) if first is None else first[0][0]
    out = torch.empty_like(u)
    for t in range(n):
        S = a[t] * S + b[t]
        out[t] = S
    return (out * y) @ w["o_proj.weight"].T, [torch.cat([S[None], torch.cat([before, raw])[-(TAPS - 1):]])]


def _experts(x, w, s):
    W, E, identity, top, F, groups, keep = s
    score = torch.softmax(x @ w["router"].T, 1)
    choice = (score + w["correction"]).view(x.shape[0], groups, -1)
    best = torch.zeros(choice.shape[:2], dtype=torch.bool, device=x.device).scatter_(1, choice.amax(2).topk(keep, 1).indices, True)
    idx = choice.masked_fill(~best[:, :, None], -math.inf).flatten(1).topk(top, 1).indices
    weight = torch.zeros_like(score).scatter_(1, idx, score.gather(1, idx) * 2.5)
    y = weight[:, E:].sum(1, keepdim=True) * x
    for e in range(E):
        rows = weight[:, e].nonzero()[:, 0]
        if len(rows):
            z = x[rows] @ w[f"e{e}.gate"].T
            y[rows] += weight[rows, e, None] * ((z * torch.sigmoid(z) * (x[rows] @ w[f"e{e}.up"].T)) @ w[f"e{e}.down"].T)
    return y


def _exact_model(case, seed):
    w, prompts, steps = model_inputs(case, seed)
    R, n, m = case["seqs"], len(prompts[0]), MODEL
    ids = torch.tensor([p + [step[r] for step in steps] for r, p in enumerate(prompts)], device=DEVICE)
    T = ids.shape[1]
    pos = torch.arange(T, device=DEVICE)
    table = w["model.embed_tokens.weight"].double()
    x = table[ids]
    for i in range(m["layers"]):
        g = {name: w[f"model.layers.{i}.{name}.weight"].double() for name in (
            "input_layernorm", "post_attention_layernorm", "self_attn.q_norm", "self_attn.k_norm", "self_attn.q_proj",
            "self_attn.k_proj", "self_attn.v_proj", "self_attn.o_proj", "mlp.gate_proj", "mlp.up_proj", "mlp.down_proj")}
        h = _unit(x) * g["input_layernorm"]
        q = _turn_half((_unit((h @ g["self_attn.q_proj"].T).view(R * T, -1, 128)) * g["self_attn.q_norm"]), pos.repeat(R), 1e6)
        k = _turn_half((_unit((h @ g["self_attn.k_proj"].T).view(R * T, -1, 128)) * g["self_attn.k_norm"]), pos.repeat(R), 1e6)
        q, k, v = (t.view(R, T, -1, 128).transpose(1, 2) for t in (q, k, h @ g["self_attn.v_proj"].T))
        group = m["heads"] // m["kv"]
        k, v = (t.repeat_interleave(group, 1) for t in (k, v))
        score = (q @ k.transpose(2, 3) * 128 ** -0.5).masked_fill(pos[None, :] > pos[:, None], -math.inf)
        x = x + (torch.softmax(score, 3) @ v).transpose(1, 2).reshape(R, T, -1) @ g["self_attn.o_proj"].T
        h = _unit(x) * g["post_attention_layernorm"]
        z = h @ g["mlp.gate_proj"].T
        x = x + (z * torch.sigmoid(z) * (h @ g["mlp.up_proj"].T)) @ g["mlp.down_proj"].T
    x = _unit(x[:, n - 1:]) * w["model.norm.weight"].double()
    return [x[:, j] @ table.T for j in range(case["steps"] + 1)]
