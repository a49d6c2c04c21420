"""The work whose speed counts: the parts and the whole decoder as a program uses them.

Every case is one pass of one part of a decoder over one step's rows, or one call of a whole model:

  layer    token embedding, one decoder layer (attention over the paged cache, gated feed-forward) and the norm
           behind it, in bfloat16 and in true 32-bit
  latent   attention through a low-rank latent over a paged cache of latents
  experts  a mixture of experts, with its routing
  state    a recurrent mixer with a matrix state a head, over prompts that begin at a zeroed slot
  model    a whole decoder's step over prompts that arrive together, with the logits of their last tokens

Sizes are those of ``bench.py``: the 1B, 2B and 8B layer shapes, pages of 16.  Steps of at most 512 rows are
replayed from a recorded CUDA graph and larger ones are launched kernel by kernel, the way ``Engine`` runs them.
Every pass can be repeated: a new token's keys and values are written to the same place again, and a
recurrent state is zeroed as it is when a request is admitted.
"""

import math
from types import SimpleNamespace

import torch

from infernum_b200.cache import CacheManager
from infernum_b200.engine.step import ModelRunner, StepContext, StepEntry
from infernum_b200.models.model import Model
from infernum_b200.ops import core
from infernum_b200.parts.base import EMBEDDINGS, NORMS, LayerSpec, PartSpec, Runtime, build_layer, build_part
from infernum_b200.registry import resolve_config

PAGE = 16
RECORDED_ROWS = 512  # the engine replays steps of up to so many rows
EPS = 1e-5
THETA = 500000.0

# width -> the decoder layers of that width: heads, key/value heads, head size, feed-forward
LAYERS = {
    1024: dict(heads=16, kv_heads=4, head_dim=64, ff=2816),
    2048: dict(heads=32, kv_heads=8, head_dim=64, ff=8192),      # the 1B shape
    3072: dict(heads=24, kv_heads=8, head_dim=128, ff=8192),
    4096: dict(heads=32, kv_heads=8, head_dim=128, ff=14336),    # the 8B shape
}
# width -> latent attention of that width: heads of 128 + 64 rotated, values of 128, a latent of 512
LATENTS = {
    2048: dict(heads=16, q_rank=768),
    4096: dict(heads=32, q_rank=1536),
}


def listed():
    layer = dict(kind="layer", dtype="bfloat16")
    return [
        # one request of a small model being decoded: the least work a step can be, all of it latency
        dict(layer, name="layer decode 1 1B", width=2048, requests=1, tokens=1, past=700),
        # a server's ordinary step: many requests of uneven lengths, a token each
        dict(layer, name="layer decode 64 8B", width=4096, requests=64, tokens=64, past=1100),
        # a long prompt, as large as a step gets
        dict(layer, name="layer prompt 2048 8B", width=4096, requests=1, tokens=2048, past=0),
        # the true 32-bit engine: two prompts in one step, and a few requests being decoded
        dict(layer, name="layer prompts f32 1B", dtype="float32", width=2048, requests=2, tokens=700, past=0),
        dict(layer, name="layer decode 8 f32 1B", dtype="float32", width=2048, requests=8, tokens=8, past=500),
        # attention through a latent: a long prompt, and eight requests being decoded
        dict(kind="latent", name="latent prompt 2048 8B", width=4096, requests=1, tokens=2048, past=0),
        dict(kind="latent", name="latent decode 8 8B", width=4096, requests=8, tokens=8, past=1024),
        # sixteen experts of which a token uses four: a long prompt; a few decoded tokens, with an expert for all
        dict(kind="experts", name="experts prompt 2048 8B", width=4096, rule="softmax_top", ff=3584, experts=16,
             top=4, shared=0, tokens=2048),
        dict(kind="experts", name="experts decode 8 2B", width=2048, rule="softmax_all", ff=1024, experts=16,
             top=4, shared=4096, tokens=8),
        # recurrent mixers: a long prompt through a state space layer, two prompts through a delta rule
        dict(kind="state", name="ssd prompt 2048 2B", width=2048, rule="ssd", requests=1, tokens=2048),
        dict(kind="state", name="delta prompts 1500 2B", width=2048, rule="delta", requests=2, tokens=1500),
        # a whole decoder: three prompts that arrive together, odd lengths
        dict(kind="model", name="model prompts 1B", width=2048, layers=8, vocab=32000, requests=3, tokens=1019),
    ]


def _log(rng, low, high):
    """A whole number between the two, even over the logarithm."""
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


def draw(rng):
    kind = rng.choice(["layer", "layer", "layer", "latent", "latent", "experts", "experts", "state", "state", "model"])
    if kind == "layer":
        dtype = rng.choice(["bfloat16", "bfloat16", "float32"])
        width = rng.choice([1024, 2048] if dtype == "float32" else [1024, 2048, 3072, 4096])
        case = dict(kind=kind, dtype=dtype, width=width)
        if rng.random() < 0.5:
            n = _log(rng, 1, 16 if dtype == "float32" else 96)
            return dict(case, requests=n, tokens=n, past=_log(rng, 40, 600 if dtype == "float32" else 2000))
        tokens = _log(rng, 24, 700 if dtype == "float32" else 2048)
        return dict(case, requests=rng.randint(1, 3), tokens=tokens, past=rng.choice([0, 0, _log(rng, 30, 500)]))
    if kind == "latent":
        case = dict(kind=kind, width=rng.choice(sorted(LATENTS)))
        if rng.random() < 0.5:
            n = _log(rng, 1, 64)
            return dict(case, requests=n, tokens=n, past=_log(rng, 40, 2000))
        return dict(case, requests=rng.randint(1, 3), tokens=_log(rng, 24, 1800), past=rng.choice([0, 0, _log(rng, 30, 200)]))
    if kind == "experts":
        width = rng.choice([1024, 2048, 4096])
        rule = rng.choice(["softmax_top", "sigmoid", "softmax_all"])
        ff = {1024: 512, 2048: rng.choice([1024, 2048]), 4096: rng.choice([1792, 3584])}[width]
        return dict(kind=kind, width=width, rule=rule, ff=ff, experts=rng.choice([8, 16]) if ff > 1024 else 16,
                    top=rng.choice([2, 4]), shared=2 * ff if rule == "softmax_all" and rng.random() < 0.7 else 0,
                    tokens=_log(rng, 1, 2048))
    if kind == "state":
        return dict(kind=kind, width=rng.choice([1024, 2048]), rule=rng.choice(["ssd", "delta", "gla", "wkv"]),
                    requests=rng.randint(1, 4), tokens=_log(rng, 60, 2048))
    return dict(kind=kind, width=rng.choice([1024, 2048]), layers=rng.choice([2, 4, 8]), vocab=32000,
                requests=rng.randint(1, 4), tokens=_log(rng, 40, 1100))


# ---------------------------------------------------------------------------------------------
# the step's requests
# ---------------------------------------------------------------------------------------------
def _shares(total, parts):
    """``total`` cut in ``parts`` uneven shares."""
    weights = [3 + 5 * i for i in range(parts)]
    cuts = [total * sum(weights[: i + 1]) // sum(weights) for i in range(parts)]
    cuts[-1] = total
    out = [b - a for a, b in zip([0] + cuts, cuts)]
    return out if min(out) > 0 else [total // parts + (i < total % parts) for i in range(parts)]


def _requests(case):
    """(tokens cached before, tokens of this step) of every request."""
    n, tokens, past = case["requests"], case["tokens"], case.get("past", 0)
    if tokens == n:  # decoded tokens: lengths from a third of the mean to five thirds of it
        return [(max(1, past * (2 + 8 * i // max(n - 1, 1)) // 6 + i % 7) if n > 1 else past, 1) for i in range(n)]
    return [(past * (i + 1) // n, t) for i, t in enumerate(_shares(tokens, n))]


def _pairs(reqs):
    """(query, key) pairs that see one another."""
    return sum(t * p + t * (t + 1) // 2 for p, t in reqs)


class _Step:
    """A step over requests of a part: their cache, and the description that parts read."""

    def __init__(self, mixer, rt, reqs, dtype):
        need = SimpleNamespace(position=0, paged=mixer.cache_spec(), state=mixer.state_spec(), cache_of=None)
        total = [p + t for p, t in reqs]
        pages = sum(-(-n // PAGE) for n in total)
        self.cache = CacheManager([need], page_size=PAGE, num_pages=pages + 2, max_requests=len(reqs), dtype=dtype,
                                  device=rt.device)
        held = [self.cache.admit(i) for i in range(len(reqs))]
        for at in range(0, max(total), PAGE):  # the requests grow side by side: their pages lie between one another's
            for rc, n in zip(held, total):
                if at < n:
                    self.cache.extend(rc, min(PAGE, n - at))
        self.layer = self.cache.layer_caches[0]
        self.reqs = reqs
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=rt.device)  # noqa: E731
        rows = [t for _, t in reqs]
        cu = [sum(rows[:i]) for i in range(len(rows) + 1)]
        paged = len(self.cache.groups) > 0
        width = max(-(-n // PAGE) for n in total)
        self.tables = torch.full((len(reqs), width), -1, dtype=torch.int32)
        if paged:
            for e, rc in enumerate(held):
                t = torch.as_tensor(rc.tables[0], dtype=torch.int32)
                self.tables[e, : len(t)] = t
        self.fields = dict(
            n_rows=cu[-1], n_entries=len(reqs), token_ids=i32([0] * cu[-1]),
            positions=i32([p + j for p, t in reqs for j in range(t)]),
            row_entry=i32([e for e, t in enumerate(rows) for _ in range(t)]), cu_rows=i32(cu),
            q_start=i32([p for p, _ in reqs]), kv_len=i32(total), slot_ids=i32([rc.slot for rc in held]),
            logit_rows=None, block_tables=[self.tables.to(rt.device)] if paged else [], host_cu_rows=cu,
            host_kv_len=total, max_rows_per_entry=max(rows), max_kv_len=max(total), all_decode=max(rows) == 1)

    def context(self):
        return StepContext(**self.fields)


def _cached(pool, tables, entry, n):
    """The first ``n`` cached vectors of an entry: [heads, n, size]."""
    pages = tables[entry, : -(-n // PAGE)].long().to(pool.device)
    rows = pool[pages]  # [pages, heads, PAGE, size]
    return rows.permute(1, 0, 2, 3).reshape(pool.shape[1], -1, pool.shape[3])[:, :n]


# ---------------------------------------------------------------------------------------------
# weights and inputs, from the seed alone
# ---------------------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _draw_tensors(shapes, seed, dtype):
    """``shapes``: name -> (shape, mean, deviation)."""
    g = _generator(seed)
    return {name: (torch.randn(shape, generator=g, device="cuda") * dev + mean).to(dtype)
            for name, (shape, mean, dev) in shapes.items()}


def _layer_shapes(case, prefix):
    s, d = LAYERS[case["width"]], case["width"]
    h, g, hd, ff = s["heads"], s["kv_heads"], s["head_dim"], s["ff"]
    return {prefix + "input_layernorm.weight": ((d,), 1.0, 0.05),
            prefix + "self_attn.q_proj.weight": ((h * hd, d), 0.0, 0.02),
            prefix + "self_attn.k_proj.weight": ((g * hd, d), 0.0, 0.02),
            prefix + "self_attn.v_proj.weight": ((g * hd, d), 0.0, 0.02),
            prefix + "self_attn.o_proj.weight": ((d, h * hd), 0.0, 0.02),
            prefix + "post_attention_layernorm.weight": ((d,), 1.0, 0.05),
            prefix + "mlp.gate_proj.weight": ((ff, d), 0.0, 0.02),
            prefix + "mlp.up_proj.weight": ((ff, d), 0.0, 0.02),
            prefix + "mlp.down_proj.weight": ((d, ff), 0.0, 0.02)}


def _config(case):
    s = LAYERS[case["width"]]
    return {"model_type": "llama", "num_hidden_layers": case["layers"], "hidden_size": case["width"],
            "num_attention_heads": s["heads"], "num_key_value_heads": s["kv_heads"], "head_dim": s["head_dim"],
            "intermediate_size": s["ff"], "vocab_size": case["vocab"], "rope_theta": THETA, "rms_norm_eps": EPS,
            "tie_word_embeddings": False, "max_position_embeddings": 8192}


def _state_sizes(case):
    """Heads of 64 for a state space layer and wkv, of 128 for a delta rule, of 64 keys and 128 values for gated
    linear attention."""
    d = case["width"]
    return {"ssd": dict(heads=d // 64, vdim=64, state=128, groups=1, conv=4, norm_groups=1),
            "wkv": dict(heads=d // 64, dim=64, rank=64),
            "delta": dict(heads=d // 128, kv_heads=d // 256, dim=128, vdim=128, conv=4),
            "gla": dict(heads=d // 128, dim=64, vdim=128, rank=16, tau=16.0)}[case["rule"]]


def _shapes(case):
    """Every tensor of the case's part, by its checkpoint name."""
    kind, d = case["kind"], case["width"]
    if kind == "layer":
        out = _layer_shapes(case, "l.")
        out.update({"embed": ((4096, d), 0.0, 1.0), "norm": ((d,), 1.0, 0.05)})
        return out
    if kind == "model":
        out = {"model.embed_tokens.weight": ((case["vocab"], d), 0.0, 1.0), "model.norm.weight": ((d,), 1.0, 0.05),
               "lm_head.weight": ((case["vocab"], d), 0.0, 0.02)}
        for n in range(case["layers"]):
            out.update(_layer_shapes(case, "model.layers.%d." % n))
        return out
    if kind == "latent":
        h, qr = LATENTS[d]["heads"], LATENTS[d]["q_rank"]
        return {"dq": ((qr, d), 0.0, 0.02), "dq.norm": ((qr,), 1.0, 0.05), "uq": ((h * 192, qr), 0.0, 0.03),
                "dkv": ((576, d), 0.0, 0.02), "dkv.norm": ((512,), 1.0, 0.05), "uk": ((h * 128, 512), 0.0, 0.04),
                "uv": ((h * 128, 512), 0.0, 0.04), "o": ((d, h * 128), 0.0, 0.02)}
    if kind == "experts":
        f, n = case["ff"], case["experts"]
        out = {"router": ((n, d), 0.0, 0.02)}
        if case["rule"] != "softmax_all":
            out["router.b"] = ((n,), 0.0, 0.3)
        for e in range(n):
            out.update({"e%d.gate" % e: ((f, d), 0.0, 0.02), "e%d.up" % e: ((f, d), 0.0, 0.02),
                        "e%d.down" % e: ((d, f), 0.0, 0.02)})
        if case["shared"]:
            f = case["shared"]
            out.update({"shared.gate": ((f, d), 0.0, 0.02), "shared.up": ((f, d), 0.0, 0.02),
                        "shared.down": ((d, f), 0.0, 0.02)})
        return out
    s = _state_sizes(case)
    h = s["heads"]
    if case["rule"] == "ssd":
        inner = h * s["vdim"]
        channels = inner + 2 * s["groups"] * s["state"]
        return {"in": ((inner + channels + h, d), 0.0, 0.02), "conv": ((channels, s["conv"]), 0.0, 0.3),
                "conv.b": ((channels,), 0.0, 0.1), "dt_bias": ((h,), -1.0, 0.5), "A_log": ((h,), 0.0, 0.5),
                "D": ((h,), 1.0, 0.05), "norm": ((inner,), 1.0, 0.05), "o": ((d, inner), 0.0, 0.02)}
    if case["rule"] == "wkv":
        hk, r = h * s["dim"], s["rank"]
        out = {"mu." + m: ((d,), 0.5, 0.2) for m in "rkvgw"}
        out.update({m: ((hk, d), 0.0, 0.02) for m in "rkvg"})
        out.update({"w1": ((r, d), 0.0, 0.02), "w2": ((hk, r), 0.0, 0.05), "w0": ((hk,), -2.0, 0.8),
                    "u": ((h, s["dim"]), 0.0, 0.3), "norm": ((hk,), 1.0, 0.05), "o": ((d, hk), 0.0, 0.02)})
        return out
    if case["rule"] == "delta":
        qk, inner = s["kv_heads"] * s["dim"], h * s["vdim"]
        return {"q": ((qk, d), 0.0, 0.02), "k": ((qk, d), 0.0, 0.02), "v": ((inner, d), 0.0, 0.02),
                "g": ((inner, d), 0.0, 0.02), "b": ((h, d), 0.0, 0.02), "a": ((h, d), 0.0, 0.02),
                "q.conv": ((qk, s["conv"]), 0.0, 0.4), "k.conv": ((qk, s["conv"]), 0.0, 0.4),
                "v.conv": ((inner, s["conv"]), 0.0, 0.4), "A_log": ((h,), -1.0, 0.5), "dt_bias": ((h,), -2.0, 0.5),
                "norm": ((s["vdim"],), 1.0, 0.05), "o": ((d, inner), 0.0, 0.02)}
    qk, inner, r = h * s["dim"], h * s["vdim"], s["rank"]
    return {"q": ((qk, d), 0.0, 0.02), "k": ((qk, d), 0.0, 0.02), "v": ((inner, d), 0.0, 0.02),
            "g": ((inner, d), 0.0, 0.02), "a1": ((r, d), 0.0, 0.02), "a2": ((qk, r), 0.0, 0.2),
            "a2.b": ((qk,), 1.0, 0.5), "norm": ((s["vdim"],), 1.0, 0.05), "o": ((d, inner), 0.0, 0.02)}


def _dtype(case):
    return torch.float32 if case.get("dtype") == "float32" else torch.bfloat16


def _weights(case, seed):
    return _draw_tensors(_shapes(case), 4 * seed, _dtype(case))


def _rows(case, seed):
    """The step's input: token ids of a layer or a model, normed rows of a part."""
    n, g = case["tokens"], _generator(4 * seed + 1)
    if case["kind"] in ("layer", "model"):
        return torch.randint(0, 4096 if case["kind"] == "layer" else case["vocab"], (n,), generator=g, device="cuda",
                             dtype=torch.int32)
    return torch.randn((n, case["width"]), generator=g, device="cuda").to(_dtype(case))


def _fill(pool, seed):
    """What earlier steps left in the cache: normed latents, projected keys and values."""
    pool.copy_(torch.randn(pool.shape, generator=_generator(seed), device="cuda"))


# ---------------------------------------------------------------------------------------------
# the parts
# ---------------------------------------------------------------------------------------------
def _part(case, rt):
    kind, d = case["kind"], case["width"]
    if kind == "latent":
        return build_part("mixer", PartSpec("latent_attention", dict(
            hidden_size=d, num_heads=LATENTS[d]["heads"], dim=128, rot_dim=64, vdim=128, q_rank=LATENTS[d]["q_rank"],
            kv_rank=512, scale=192 ** -0.5, window=4096, eps=EPS, theta=10000.0)), rt)
    if kind == "experts":
        params = dict(hidden_size=d, expert_size=case["ff"], experts=case["experts"], top=case["top"],
                      scoring=case["rule"], router_bias=None if case["rule"] == "softmax_all" else "router.b")
        if case["rule"] == "sigmoid":
            params["groups"] = {"count": 4, "keep": 2}
        if case["shared"]:
            params["shared"] = {"size": case["shared"]}
        return build_part("ffn", PartSpec("moe", params), rt)
    s = _state_sizes(case)
    params = dict(hidden_size=d, num_heads=s["heads"], eps=EPS)
    if case["rule"] == "ssd":
        params.update(vdim=s["vdim"], state=s["state"], groups=s["groups"], conv=s["conv"], norm_groups=1)
    elif case["rule"] == "wkv":
        params.update(head_dim=s["dim"], decay_rank=s["rank"])
    elif case["rule"] == "delta":
        params.update(num_kv_heads=s["kv_heads"], head_dim=s["dim"], vdim=s["vdim"], conv=s["conv"])
    else:
        params.update(head_dim=s["dim"], vdim=s["vdim"], tau=s["tau"], decay_rank=s["rank"])
    return build_part("mixer", PartSpec(case["rule"], params), rt)


def _layer_parts(case, rt):
    s, d = LAYERS[case["width"]], case["width"]
    embed = EMBEDDINGS.get("token_embedding")(dict(vocab_size=4096, hidden_size=d, weight="embed"), rt)
    norm = lambda name: PartSpec("rmsnorm", dict(hidden_size=d, eps=EPS, weight=name))  # noqa: E731
    layer = build_layer(LayerSpec("prenorm", {
        "norm1": norm("l.input_layernorm.weight"),
        "mixer": PartSpec("attention", dict(
            hidden_size=d, num_heads=s["heads"], num_kv_heads=s["kv_heads"], head_dim=s["head_dim"], window=0,
            position={"kind": "rotary", "params": {"head_dim": s["head_dim"], "theta": THETA}}, prefix="l.self_attn.")),
        "norm2": norm("l.post_attention_layernorm.weight"),
        "ffn": PartSpec("swiglu", dict(hidden_size=d, intermediate_size=s["ff"], prefix="l.mlp.")),
    }, name="l."), rt)
    last = NORMS.get("rmsnorm")(dict(hidden_size=d, eps=EPS, weight="norm"), rt)
    return embed, layer, last


def prepare(case, seed):
    device = torch.device("cuda:0")
    weights = _weights(case, seed)
    if case["kind"] == "model":
        arch, cfg = resolve_config(_config(case))
        rt = Runtime(device, torch.bfloat16, options={})
        model = Model(arch.build_spec(cfg), rt)
        model.bind(weights)
        reqs = _requests(case)
        cache = CacheManager(model.cache_needs(), page_size=PAGE, max_requests=len(reqs), dtype=rt.dtype, device=device,
                             num_pages=sum(-(-t // PAGE) for _, t in reqs) + 2)
        ids = _rows(case, seed).tolist()
        prompts, at = [], 0
        for _, t in reqs:
            prompts.append(ids[at: at + t])
            at += t
        return dict(runner=ModelRunner(model, cache, max_rows=4096, max_entries=len(reqs)), cache=cache, prompts=prompts)

    dtype = _dtype(case)
    rt = Runtime(device, dtype, err=core.new_error_word(device), options={
        "sm_count": torch.cuda.get_device_properties(0).multi_processor_count})
    x = _rows(case, seed)
    if case["kind"] == "layer":
        embed, layer, last = _layer_parts(case, rt)
        for part in (embed, layer, last):
            part.bind(weights)
        step = _Step(layer.mixer, rt, _requests(case), dtype)
        _fill(step.layer.k_pool, 4 * seed + 2)
        _fill(step.layer.v_pool, 4 * seed + 3)
        step.fields["token_ids"] = x

        def forward():
            ctx = step.context()
            stream = embed.forward_step(ctx, None)
            layer.forward(stream, ctx, step.layer)
            normed = last.forward(stream)
            return {"normed": normed, "residual": stream.residual, "k": step.layer.k_pool, "v": step.layer.v_pool}
    elif case["kind"] == "experts":
        part = _part(case, rt)
        part.bind(weights)

        def forward():
            return {"out": part.forward(x)}
    else:
        part = _part(case, rt)
        part.bind(weights)
        step = _Step(part, rt, _requests(case), dtype)
        if case["kind"] == "latent":
            _fill(step.layer.k_pool, 4 * seed + 2)

        def forward():
            state = step.layer.state
            if state is not None:  # the requests have just been admitted
                state.zero_()
            out = part.forward(x, step.context(), step.layer)
            return {"out": out, "latents": step.layer.k_pool} if state is None else {"out": out, "state": state}

    def whole():
        with core.step_stream(device):
            core.step_fence(device)
            return forward()

    if case["tokens"] > RECORDED_ROWS:
        return dict(call=whole)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        whole()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="thread_local"):
        out = whole()
    return dict(graph=graph, out=out, call=whole)


def run(state):
    if "runner" in state:
        held = [state["cache"].admit(i) for i in range(len(state["prompts"]))]
        logits = state["runner"].step([StepEntry(rc, p, [len(p) - 1]) for rc, p in zip(held, state["prompts"])])
        for rc in held:
            state["cache"].release(rc)
        return {"logits": logits}
    if "graph" in state:
        state["graph"].replay()
        return state["out"]
    return state["call"]()


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
def _layer_work(case, reqs):
    s, d, n = LAYERS[case["width"]], case["width"], case["tokens"]
    qd, kd = s["heads"] * s["head_dim"], s["kv_heads"] * s["head_dim"]
    weights = d * (qd + 2 * kd) + qd * d + 3 * d * s["ff"]
    size = 4 if case.get("dtype") == "float32" else 2
    read = sum(p for p, _ in reqs)
    return (size * (weights + 2 * kd * (read + n)), 2.0 * n * weights + 4.0 * qd * _pairs(reqs))


def work(case):
    kind, d, n = case["kind"], case["width"], case["tokens"]
    if kind in ("layer", "model"):
        reqs = _requests(case)
        b, f = _layer_work(case, reqs)
        if kind == "model":
            return {"bytes": case["layers"] * b + 2 * d * case["vocab"] + 2 * n * d,
                    "flops": case["layers"] * f + 2.0 * len(reqs) * d * case["vocab"]}
        size = 4 if case["dtype"] == "float32" else 2
        return {"bytes": b + n * d * (4 + 2 * size), "flops": f}
    if kind == "latent":
        h, qr, reqs = LATENTS[d]["heads"], LATENTS[d]["q_rank"], _requests(case)
        down, keys = d * (qr + 576) + qr * h * 192 + h * 128 * d, sum(p + t for p, t in reqs)
        # the cheaper way of the two: keys and values made once for the cached vectors, or queries taken to the latents
        made = 2.0 * keys * 512 * h * 256 + 2.0 * h * (192 + 128) * _pairs(reqs)
        taken = 2.0 * n * h * 256 * 512 + 2.0 * h * (576 + 512) * _pairs(reqs)
        return {"bytes": 2 * (down + 2 * h * 128 * 512 + 576 * (keys + n) + 2 * n * d),
                "flops": 2.0 * n * down + min(made, taken)}
    if kind == "experts":
        e, top, ff = case["experts"], case["top"], case["ff"]
        used = e * (1 - (1 - top / e) ** n)  # experts that some token uses, at even odds
        cols = top * ff + case["shared"]
        return {"bytes": 2 * (3 * d * (used * ff + case["shared"]) + e * d + 2 * n * d), "flops": 2.0 * n * d * (3 * cols + e)}
    weights = sum(math.prod(shape) for shape, _, _ in _shapes(case).values())
    s = _state_sizes(case)
    per = {"ssd": (s.get("state", 0), s.get("vdim", 0), 5), "wkv": (s.get("dim", 0), s.get("dim", 0), 6),
           "delta": (s.get("dim", 0), s.get("vdim", 0), 7), "gla": (s.get("dim", 0), s.get("vdim", 0), 5)}[case["rule"]]
    state = s["heads"] * per[0] * per[1]
    return {"bytes": 2 * weights + 4 * n * d + 4 * state * case["requests"], "flops": 2.0 * n * weights + float(per[2]) * n * state}


def tolerance(case):
    # Measured against ``exact`` over the listed and drawn cases, times about four (bfloat16 rounds what passes from
    # one product to the next; 32-bit sums differ by their order).
    if case.get("dtype") == "float32":
        return {"rel": 1e-5}
    if case["kind"] == "model":
        return {"rel": 3e-2}
    return {"rel": 2e-2}


# ---------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------
def _rms(x, w=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)
    return y if w is None else y * w


def _silu(x):
    return x * torch.sigmoid(x)


def _rotate(x, pos, theta):
    """Pairs (i, i + half) of the last dimension; x [rows, heads, size]."""
    half = x.shape[-1] // 2
    freq = torch.tensor([theta ** (-2.0 * j / x.shape[-1]) for j in range(half)], dtype=torch.float64)
    ang = pos.double()[:, None, None] * freq.float().double().to(x.device)
    c, s = torch.cos(ang), torch.sin(ang)
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * c - b * s, a * s + b * c], -1)


def _attend(q, k, v, scale, past):
    """One head: q [t, .] at positions past.., k and v [past + t, .]."""
    s = (q @ k.T) * scale
    t, n = s.shape
    s.masked_fill_(torch.arange(n, device=s.device)[None, :] > past + torch.arange(t, device=s.device)[:, None], -math.inf)
    return torch.softmax(s, -1) @ v


def _exact_layer(case, w, prefix, x, reqs, cached):
    """x [rows, width] through one decoder layer; ``cached(e, n)``: an entry's first n keys and values."""
    s = LAYERS[case["width"]]
    h, g, hd = s["heads"], s["kv_heads"], s["head_dim"]
    m = lambda name: w[prefix + name].double()  # noqa: E731
    u = _rms(x, m("input_layernorm.weight"))
    pos = torch.cat([torch.arange(p, p + t) for p, t in reqs]).to(x.device)
    q = _rotate((u @ m("self_attn.q_proj.weight").T).view(-1, h, hd), pos, THETA)
    k = _rotate((u @ m("self_attn.k_proj.weight").T).view(-1, g, hd), pos, THETA)
    v = (u @ m("self_attn.v_proj.weight").T).view(-1, g, hd)
    o, at = torch.empty_like(q), 0
    for e, (p, t) in enumerate(reqs):
        rows = slice(at, at + t)
        at += t
        old = cached(e, p) if p else None
        for j in range(g):
            kk, vv = k[rows, j], v[rows, j]
            if old is not None:
                kk, vv = torch.cat([old[0][j].double(), kk]), torch.cat([old[1][j].double(), vv])
            for a in range(j * (h // g), (j + 1) * (h // g)):
                o[rows, a] = _attend(q[rows, a], kk, vv, hd ** -0.5, p)
    x = x + o.reshape(-1, h * hd) @ m("self_attn.o_proj.weight").T
    u = _rms(x, m("post_attention_layernorm.weight"))
    y = _silu(u @ m("mlp.gate_proj.weight").T) * (u @ m("mlp.up_proj.weight").T)
    return x + y @ m("mlp.down_proj.weight").T


class _PlainCache:
    """The cached vectors of every request as ``prepare`` lays them out: pages handed out request by request."""

    def __init__(self, reqs):
        total = [p + t for p, t in reqs]
        self.pages = sum(-(-n // PAGE) for n in total) + 3  # (two to spare, and one behind the pool for padding)
        mine, free = [[] for _ in reqs], 0
        for at in range(0, max(total), PAGE):
            for e, n in enumerate(total):
                if at < n:
                    mine[e].append(free)
                    free += 1
        self.tables = torch.full((len(reqs), max(len(t) for t in mine)), -1, dtype=torch.int32)
        for e, t in enumerate(mine):
            self.tables[e, : len(t)] = torch.tensor(t, dtype=torch.int32)

    def pool(self, heads, size, seed, dtype):
        out = torch.empty((self.pages, heads, PAGE, size), dtype=dtype, device="cuda")
        _fill(out, seed)
        return out


def _exact_experts(case, w, x):
    n, e, top = x.shape[0], case["experts"], case["top"]
    z = x @ w["router"].double().T
    if "router.b" in w:
        z = z + w["router.b"].double()
    if case["rule"] == "softmax_top":
        best = z.topk(top, -1)
        ids, wts = best.indices, torch.softmax(best.values, -1)
    elif case["rule"] == "sigmoid":
        s = torch.sigmoid(z)
        groups = s.view(n, 4, e // 4)
        open_ = groups.topk(2, -1).values.sum(-1).topk(2, -1).indices
        mask = torch.zeros((n, 4), dtype=torch.bool, device=x.device).scatter_(1, open_, True)
        ids = torch.where(mask[:, :, None], groups, -1.0).reshape(n, e).topk(top, -1).indices
        wts = s.gather(1, ids)
    else:
        best = torch.softmax(z, -1).topk(top, -1)
        ids, wts = best.indices, best.values / best.values.sum(-1, keepdim=True)
    out = torch.zeros_like(x)
    ffn = lambda p, rows: (_silu(rows @ w[p + "gate"].double().T) * (rows @ w[p + "up"].double().T)) @ w[p + "down"].double().T  # noqa: E731
    for i in range(e):
        row, slot = (ids == i).nonzero(as_tuple=True)
        if len(row):
            out[row] += wts[row, slot][:, None] * ffn("e%d." % i, x[row])
    return out + ffn("shared.", x) if case["shared"] else out


def _exact_latent(case, w, x, reqs, plain, pool):
    h, pos = LATENTS[case["width"]]["heads"], torch.cat([torch.arange(p, p + t) for p, t in reqs]).to(x.device)
    m = lambda name: w[name].double()  # noqa: E731
    q = (_rms(x @ m("dq").T, m("dq.norm")) @ m("uq").T).view(-1, h, 192)
    raw = x @ m("dkv").T
    c, r = _rms(raw[:, :512], m("dkv.norm")), _rotate(raw[:, None, 512:], pos, 10000.0)[:, 0]
    q = torch.cat([q[..., :128], _rotate(q[..., 128:], pos, 10000.0)], -1)
    uk, uv = m("uk").view(h, 128, 512), m("uv").view(h, 128, 512)
    o, at = torch.empty((x.shape[0], h, 128), dtype=torch.float64, device=x.device), 0
    for e, (p, t) in enumerate(reqs):
        rows = slice(at, at + t)
        at += t
        cc, rr = c[rows], r[rows]
        if p:
            old = _cached(pool, plain.tables, e, p)[0].double()
            cc, rr = torch.cat([old[:, :512], cc]), torch.cat([old[:, 512:], rr])
        for a in range(h):
            o[rows, a] = _attend(q[rows, a], torch.cat([cc @ uk[a].T, rr], -1), cc @ uv[a].T, 192 ** -0.5, p)
    return o.reshape(-1, h * 128) @ m("o").T


def _conv(x, weight, bias=None):
    taps = weight.shape[1]
    padded = torch.cat([torch.zeros((taps - 1, x.shape[1]), dtype=x.dtype, device=x.device), x])
    y = sum(padded[j: j + x.shape[0]] * weight[:, j] for j in range(taps))
    return _silu(y if bias is None else y + bias)


def _exact_state(case, w, x):
    """One request from a zeroed slot: (result, the slot's state as it is stored)."""
    s, rule, T = _state_sizes(case), case["rule"], x.shape[0]
    h = s["heads"]
    m = lambda name: w[name].double()  # noqa: E731
    if rule == "ssd":
        inner, gn = h * s["vdim"], s["groups"] * s["state"]
        proj = x @ m("in").T
        z, raw, dt = proj[:, :inner], proj[:, inner: 2 * inner + 2 * gn], proj[:, 2 * inner + 2 * gn:]
        xbc = _conv(raw, m("conv"), m("conv.b"))
        xs, b, c = xbc[:, :inner].view(T, h, -1), xbc[:, inner: inner + gn], xbc[:, inner + gn:]
        dt = torch.nn.functional.softplus(dt + m("dt_bias"))
        a = torch.exp(-torch.exp(m("A_log")) * dt)
        S = torch.zeros((h, s["state"], s["vdim"]), dtype=x.dtype, device=x.device)
        ys = []
        for t in range(T):
            S = a[t][:, None, None] * S + b[t][None, :, None] * (dt[t][:, None] * xs[t])[:, None, :]
            ys.append((c[t][None, :, None] * S).sum(1))
        y = torch.stack(ys) + m("D")[None, :, None] * xs
        y = _rms(y.reshape(T, inner) * _silu(z), m("norm"))
        tail = torch.cat([torch.zeros((3, raw.shape[1]), dtype=x.dtype, device=x.device), raw])[-3:]
        return y @ m("o").T, S, tail
    if rule == "wkv":
        k = s["dim"]
        prev = torch.cat([torch.zeros_like(x[:1]), x[:-1]])
        mix = {i: x + (prev - x) * m("mu." + i) for i in "rkvgw"}
        r, kk, v, g = (mix[i] @ m(i).T for i in "rkvg")
        wd = torch.exp(-torch.exp(torch.tanh(mix["w"] @ m("w1").T) @ m("w2").T + m("w0")))
        r, kk, v, wd = (i.view(T, h, k) for i in (r, kk, v, wd))
        S = torch.zeros((h, k, k), dtype=x.dtype, device=x.device)
        os = []
        for t in range(T):
            kv = kk[t][:, :, None] * v[t][:, None, :]
            os.append((r[t][:, :, None] * (S + m("u")[:, :, None] * kv)).sum(1))
            S = wd[t][:, :, None] * S + kv
        y = _rms(torch.stack(os)).reshape(T, h * k) * m("norm") * _silu(g)
        return y @ m("o").T, S, x[-1:]
    if rule == "delta":
        kv, dim, vd = s["kv_heads"], s["dim"], s["vdim"]
        raw = torch.cat([x @ m(i).T for i in "qkv"], -1)
        mixed = _conv(raw, torch.cat([m(i + ".conv") for i in "qkv"]))
        q, k, v = mixed.split([kv * dim, kv * dim, h * vd], -1)
        unit = lambda y: y / torch.sqrt((y * y).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
        per = h // kv
        q = (unit(q.view(T, kv, dim)) * dim ** -0.5).repeat_interleave(per, 1)
        k = unit(k.view(T, kv, dim)).repeat_interleave(per, 1)
        v = v.view(T, h, vd)
        beta = torch.sigmoid(x @ m("b").T)
        g = torch.exp(-torch.exp(m("A_log")) * torch.nn.functional.softplus(x @ m("a").T + m("dt_bias")))
        S = torch.zeros((h, dim, vd), dtype=x.dtype, device=x.device)
        os = []
        for t in range(T):
            S = g[t][:, None, None] * S
            u = beta[t][:, None] * (v[t] - (k[t][:, :, None] * S).sum(1))
            S = S + k[t][:, :, None] * u[:, None, :]
            os.append((q[t][:, :, None] * S).sum(1))
        y = (_rms(torch.stack(os)) * m("norm")).reshape(T, h * vd) * _silu(x @ m("g").T)
        tail = torch.cat([torch.zeros((3, raw.shape[1]), dtype=x.dtype, device=x.device), raw])[-3:]
        return y @ m("o").T, S, tail
    dim, vd = s["dim"], s["vdim"]
    q = (x @ m("q").T * dim ** -0.5).view(T, h, dim)
    k, v = (x @ m("k").T).view(T, h, dim), (x @ m("v").T).view(T, h, vd)
    a = torch.sigmoid(x @ m("a1").T @ m("a2").T + m("a2.b")).pow(1.0 / s["tau"]).view(T, h, dim)
    S = torch.zeros((h, dim, vd), dtype=x.dtype, device=x.device)
    os = []
    for t in range(T):
        S = a[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
        os.append((q[t][:, :, None] * S).sum(1))
    y = (_rms(torch.stack(os)) * m("norm")).reshape(T, h * vd) * _silu(x @ m("g").T)
    return y @ m("o").T, S, None


def exact(case, seed):
    w, rows, kind = _weights(case, seed), _rows(case, seed), case["kind"]
    if kind == "experts":
        return {"out": _exact_experts(case, w, rows.double())}
    reqs = _requests(case)
    if kind == "model":
        x = w["model.embed_tokens.weight"].double()[rows.long()]
        for n in range(case["layers"]):
            x = _exact_layer(case, w, "model.layers.%d." % n, x, reqs, None)
        last = torch.tensor([t for _, t in reqs]).cumsum(0) - 1
        x = _rms(x[last.to(x.device)], w["model.norm.weight"].double())
        return {"logits": x @ w["lm_head.weight"].double().T}
    if kind == "state":
        outs, at = [], 0
        for _, t in reqs:
            outs.append(_exact_state(case, w, rows[at: at + t].double())[0])
            at += t
        return {"out": torch.cat(outs), "state": None}
    plain = _PlainCache(reqs)
    if kind == "latent":
        pool = plain.pool(1, 576, 4 * seed + 2, _dtype(case))
        return {"out": _exact_latent(case, w, rows.double(), reqs, plain, pool), "latents": None}
    s = LAYERS[case["width"]]
    pools = [plain.pool(s["kv_heads"], s["head_dim"], 4 * seed + i, _dtype(case)) for i in (2, 3)]
    x = w["embed"].double()[rows.long()]
    x = _exact_layer(case, w, "l.", x, reqs, lambda e, n: [_cached(p, plain.tables, e, n) for p in pools])
    return {"normed": _rms(x, w["norm"].double()), "residual": x, "k": None, "v": None}
