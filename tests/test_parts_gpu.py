"""Each part alone against the plain function it stands for, and a model whose
schedule runs a layer twice and shares a cache."""
import math

import pytest
import torch

import plain_llama as pl

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
TOL = {torch.float32: 5e-6, torch.bfloat16: 2e-2}


def runtime(dtype, **options):
    from infernum_b200.ops import core
    from infernum_b200.parts.base import Runtime
    return Runtime(DEV, dtype, err=core.new_error_word(DEV), options=options)


def rel_err(got, ref):
    ref = ref.double().cpu()
    return float((got.double().cpu() - ref).abs().max() / max(ref.abs().max().item(), 1e-9))


def weights_for(part, dtype, seed=0):
    from infernum_b200.weights.random_init import random_tensors
    return random_tensors(part.weight_specs(), seed, DEV, dtype)


def step_ctx(cache, requests):
    """requests: list of (RequestCache, n_new tokens).  Builds the step inputs
    the way the engine does, with pages reserved."""
    from infernum_b200.engine.step import ModelRunner, StepEntry
    from types import SimpleNamespace
    fake = SimpleNamespace(rt=runtime(torch.float32), spec=SimpleNamespace(vocab_size=1 << 30))
    runner = ModelRunner(fake, cache)
    entries = [StepEntry(rc, [0] * n, []) for rc, n in requests]
    runner.reserve(entries)
    return runner._build(entries)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rmsnorm_part(dtype):
    from infernum_b200.parts import NORMS, ResidualStream
    rt = runtime(dtype)
    norm = NORMS.get("rmsnorm")({"hidden_size": 72, "eps": 2e-6, "weight": "w"}, rt)
    w = weights_for(norm, dtype)
    norm.bind(w)
    x = torch.randn(5, 72, device=DEV)
    d = torch.randn(5, 72, device=DEV).to(dtype)
    stream = ResidualStream(x.clone())
    stream.push(d)
    out = norm.forward(stream)
    assert stream.pending is None
    assert rel_err(stream.residual, x.double() + d.double()) < 1e-6
    assert rel_err(out, pl.rms_norm(x.double() + d.double(), w["w"].double(), 2e-6)) < TOL[dtype]
    assert rel_err(norm.apply(x), pl.rms_norm(x.double(), w["w"].double(), 2e-6)) < TOL[dtype]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rotary_part(dtype):
    from infernum_b200.parts import POSITION_ENCODINGS
    rt = runtime(dtype)
    scaling = {"rope_type": "llama3", "factor": 8.0, "low_freq_factor": 1.0,
               "high_freq_factor": 4.0, "original_max_position_embeddings": 64}
    rope = POSITION_ENCODINGS.get("rotary")({"head_dim": 48, "theta": 5e5, "scaling": scaling}, rt)
    q = torch.randn(6, 5, 48).to(dtype).to(DEV)
    k = torch.randn(6, 2, 48).to(dtype).to(DEV)
    pos = torch.tensor([0, 1, 63, 64, 200, 4000], dtype=torch.int32, device=DEV)
    q0, k0 = q.clone(), k.clone()
    rope.apply(q, k, pos)
    f = pl.rope_frequencies(48, 5e5, scaling)
    assert torch.equal(rope.inv_freq.cpu(), f)
    assert rel_err(q, pl.rope(q0.double().cpu(), pos.cpu(), f)) < TOL[dtype]
    assert rel_err(k, pl.rope(k0.double().cpu(), pos.cpu(), f)) < TOL[dtype]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_swiglu_part(dtype):
    from infernum_b200.parts import FEED_FORWARDS
    rt = runtime(dtype)
    ffn = FEED_FORWARDS.get("swiglu")({"hidden_size": 40, "intermediate_size": 104, "prefix": "m."}, rt)
    w = weights_for(ffn, dtype)
    for k in w:
        w[k] = (w[k].float() * 8).to(dtype)
    ffn.bind(w)
    x = torch.randn(9, 40).to(dtype).to(DEV)
    want = pl.swiglu(x.double().cpu(), *(w[f"m.{n}_proj.weight"].double().cpu() for n in ("gate", "up", "down")))
    assert rel_err(ffn.forward(x), want) < TOL[dtype]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("impl", ["auto", "plain"])
@pytest.mark.parametrize("nh, nkv, hd, window", [(4, 2, 16, 0), (3, 1, 32, 0), (6, 3, 48, 11)])
def test_attention_part_in_portions(dtype, impl, nh, nkv, hd, window):
    """The attention part fed a sequence in portions through a real cache
    equals plain attention over the whole sequence."""
    from infernum_b200.cache import CacheManager
    from infernum_b200.models.model import CacheNeed
    from infernum_b200.parts import MIXERS
    rt = runtime(dtype, attention=impl)
    H, T = 56, 45
    params = {"hidden_size": H, "num_heads": nh, "num_kv_heads": nkv, "head_dim": hd,
              "window": window, "prefix": "a.",
              "position": {"kind": "rotary", "params": {"head_dim": hd, "theta": 10000.0}}}
    attn = MIXERS.get("attention")(params, rt)
    w = weights_for(attn, dtype)
    for k in w:
        w[k] = (w[k].float() * 10).to(dtype)
    attn.bind(w)
    cache = CacheManager([CacheNeed(0, attn.cache_spec(), None, None)], page_size=4, num_pages=16,
                         max_requests=2, dtype=dtype, device=DEV)
    x = torch.randn(T, H).to(dtype).to(DEV)
    rc = cache.admit("r")
    outs, pos = [], 0
    for n in [7, 1, 2, 13, 1, 1, 20]:
        ctx = step_ctx(cache, [(rc, n)])
        outs.append(attn.forward(x[pos: pos + n], ctx, cache.layer_caches[0]))
        cache.commit(rc, n)
        pos += n
    got = torch.cat(outs)
    xd = x.double().cpu()
    W = {k: v.double().cpu() for k, v in w.items()}
    f = pl.rope_frequencies(hd, 10000.0, None)
    p = torch.arange(T)
    q = pl.rope((xd @ W["a.q_proj.weight"].T).view(T, nh, hd), p, f)
    k = pl.rope((xd @ W["a.k_proj.weight"].T).view(T, nkv, hd), p, f)
    v = (xd @ W["a.v_proj.weight"].T).view(T, nkv, hd)
    want = pl.attention(q, k, v, window=window).reshape(T, nh * hd) @ W["a.o_proj.weight"].T
    assert rt.err.item() == 0
    assert rel_err(got, want) < TOL[dtype]
    if window:
        assert sum(1 for page in rc.tables[0] if page == -1) > 0  # pages behind the window came back


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_embedding_and_head_parts(dtype):
    from infernum_b200.parts import EMBEDDINGS, HEADS
    rt = runtime(dtype)
    emb = EMBEDDINGS.get("token_embedding")({"vocab_size": 90, "hidden_size": 24, "weight": "e"}, rt)
    head = HEADS.get("linear_head")({"vocab_size": 90, "hidden_size": 24, "weight": "h", "tied_to": "e"}, rt)
    assert head.weight_specs() == {}
    w = weights_for(emb, dtype)
    emb.bind(w)
    head.bind(w)
    ids = torch.tensor([3, 89, 0], dtype=torch.int32, device=DEV)
    h = emb.forward(ids)
    assert h.dtype == torch.float32 and torch.equal(h.cpu(), w["e"].float().cpu()[[3, 89, 0]])
    x = torch.randn(4, 24).to(dtype).to(DEV)
    logits = head.forward(x)
    assert logits.dtype == torch.float32
    assert rel_err(logits, x.double().cpu() @ w["e"].double().cpu().T) < (5e-6 if dtype == torch.float32 else 3e-3)


def shared_schedule_spec(H=48, V=70):
    """Two layers; the schedule runs layer 0, layer 1, layer 0 again (its own
    cache), then a third attention that has no k/v of its own and reads the
    cache of the first run."""
    from infernum_b200.parts import LayerSpec, ModelSpec, PartSpec, ScheduleItem

    def layer(i, kv_shared=False):
        p = f"model.layers.{i}."
        norm = lambda n: PartSpec("rmsnorm", {"hidden_size": H, "eps": 1e-5, "weight": p + n})  # noqa: E731
        return LayerSpec("prenorm", name=p, parts={
            "norm1": norm("n1"),
            "mixer": PartSpec("attention", {"hidden_size": H, "num_heads": 4, "num_kv_heads": 2,
                                            "head_dim": 16, "prefix": p + "attn.", "kv_shared": kv_shared,
                                            "position": {"kind": "rotary", "params": {"head_dim": 16, "theta": 1e4}}}),
            "norm2": norm("n2"),
            "ffn": PartSpec("swiglu", {"hidden_size": H, "intermediate_size": 80, "prefix": p + "mlp."}),
        })

    return ModelSpec(
        hidden_size=H, vocab_size=V,
        embedding=PartSpec("token_embedding", {"vocab_size": V, "hidden_size": H, "weight": "emb"}),
        layers=(layer(0), layer(1), layer(2, kv_shared=True)),
        schedule=(ScheduleItem(0), ScheduleItem(1), ScheduleItem(0), ScheduleItem(2, cache_of=0)),
        final_norm=PartSpec("rmsnorm", {"hidden_size": H, "eps": 1e-5, "weight": "fn"}),
        lm_head=PartSpec("linear_head", {"vocab_size": V, "hidden_size": H, "weight": "head"}),
        max_position=256)


def plain_shared_schedule(W, tokens, H=48):
    T = len(tokens)
    W = {k: v.double().cpu() for k, v in W.items()}
    f = pl.rope_frequencies(16, 1e4, None)
    p = torch.arange(T)
    h = W["emb"][tokens]
    kept = {}
    for pos, (i, cache_of) in enumerate([(0, None), (1, None), (0, None), (2, 0)]):
        pre = f"model.layers.{i}."
        x = pl.rms_norm(h, W[pre + "n1"], 1e-5)
        q = pl.rope((x @ W[pre + "attn.q_proj.weight"].T).view(T, 4, 16), p, f)
        if cache_of is None:
            k = pl.rope((x @ W[pre + "attn.k_proj.weight"].T).view(T, 2, 16), p, f)
            v = (x @ W[pre + "attn.v_proj.weight"].T).view(T, 2, 16)
            kept[pos] = (k, v)
        else:
            k, v = kept[cache_of]
        h = h + pl.attention(q, k, v).reshape(T, 64) @ W[pre + "attn.o_proj.weight"].T
        m = pl.rms_norm(h, W[pre + "n2"], 1e-5)
        h = h + pl.swiglu(m, W[pre + "mlp.gate_proj.weight"], W[pre + "mlp.up_proj.weight"],
                          W[pre + "mlp.down_proj.weight"])
    return pl.rms_norm(h, W["fn"], 1e-5) @ W["head"].T


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_schedule_names_a_layer_twice_and_shares_a_cache(dtype):
    from infernum_b200.cache import CacheManager
    from infernum_b200.engine.step import ModelRunner, StepEntry
    from infernum_b200.models.model import Model
    from infernum_b200.weights.random_init import random_tensors
    rt = runtime(dtype)
    model = Model(shared_schedule_spec(), rt)
    specs = model.weight_specs()
    assert "model.layers.2.attn.k_proj.weight" not in specs
    W = random_tensors(specs, 5, DEV, dtype)
    for k in W:
        if "proj" in k:
            W[k] = (W[k].float() * 6).to(dtype)
    model.bind(W)
    needs = model.cache_needs()
    assert [n.cache_of for n in needs] == [None, None, None, 0]
    cache = CacheManager(needs, page_size=4, num_pages=32, max_requests=2, dtype=dtype, device=DEV)
    assert len(cache.groups) == 1 and cache.groups[0].positions == [0, 1, 2]
    assert cache.layer_caches[3].k_pool is cache.layer_caches[0].k_pool
    assert cache.layer_caches[2].k_pool is not cache.layer_caches[0].k_pool
    runner = ModelRunner(model, cache)
    tokens = [int(t) for t in torch.randint(0, 70, (33,))]
    rc = cache.admit("a")
    rows, pos = [], 0
    for n in [9, 1, 2, 20, 1]:
        rows.append(runner.step([StepEntry(rc, tokens[pos: pos + n], list(range(n)))]))
        pos += n
    runner.check_errors()
    got = torch.cat(rows)
    assert rel_err(got, plain_shared_schedule(W, tokens)) < (2e-5 if dtype == torch.float32 else 4e-2)


def test_products_report_into_the_runtimes_error_word(monkeypatch):
    """The tensor-core products report a wait that ran out in the device word
    they are handed.  Every product of a part must be handed the word of the
    part's Runtime (the one the engine reads after a step), not one of their
    own: the calls are watched at the C boundary, for both kernels, with and
    without the activation in the epilogue."""
    from infernum_b200.ops import gemm_tc
    from infernum_b200.parts import FEED_FORWARDS
    from infernum_b200.parts.linear import Linear
    rt = runtime(torch.bfloat16)
    seen = {"few": [], "pair": []}
    few, pair = gemm_tc.lib(), gemm_tc.pair_lib()
    real_few, real_pair = few.ib_gemm_tc, pair.ib_gemm_pair_scaled

    def spy_few(*args):
        seen["few"].append(args[12])
        return real_few(*args)

    def spy_pair(*args):
        seen["pair"].append(args[17])
        return real_pair(*args)

    monkeypatch.setattr(few, "ib_gemm_tc", spy_few)
    monkeypatch.setattr(pair, "ib_gemm_pair_scaled", spy_pair)
    lin = Linear(torch.randn(160, 96, device=DEV).to(torch.bfloat16), rt)
    lin(torch.randn(5, 96, device=DEV).to(torch.bfloat16))          # few tokens
    lin(torch.randn(768, 96, device=DEV).to(torch.bfloat16))        # a prompt: pairs of SMs
    ffn = FEED_FORWARDS.get("swiglu")({"hidden_size": 96, "intermediate_size": 256, "prefix": "m."}, rt)
    ffn.bind(weights_for(ffn, torch.bfloat16))
    ffn.forward(torch.randn(3, 96, device=DEV).to(torch.bfloat16))    # activation in the epilogue, few tokens
    ffn.forward(torch.randn(512, 96, device=DEV).to(torch.bfloat16))  # and on pairs of SMs
    torch.cuda.synchronize()
    word = rt.err.data_ptr()
    assert len(seen["few"]) >= 3 and len(seen["pair"]) >= 2
    assert set(seen["few"]) == {word} and set(seen["pair"]) == {word}
    assert int(rt.err.item()) == 0


def test_random_weights_are_the_same_on_the_device_and_in_a_written_folder(tmp_path):
    """A model drawn on the GPU from a configuration and a seed and the folder
    written for the same configuration and seed hold the same values bit for
    bit, so what was measured on one can be checked with the plain
    implementation on the other."""
    from helpers import TINY_B
    from infernum_b200.weights.random_init import model_specs_for, random_tensors, write_random_model
    folder = write_random_model(str(tmp_path / "m"), TINY_B, seed=21)
    stored = pl.read_weights(folder)
    _, _, specs = model_specs_for(TINY_B)
    drawn = random_tensors(specs, 21, DEV, torch.bfloat16)
    assert set(stored) == set(drawn)
    for name, t in drawn.items():
        assert torch.equal(t.cpu(), stored[name]), name
    other = random_tensors(specs, 22, DEV, torch.bfloat16)
    assert not torch.equal(other["model.embed_tokens.weight"], drawn["model.embed_tokens.weight"])


@pytest.mark.parametrize("scoring, experts, top, ff, shared, identity", [
    ("softmax_top", 16, 4, 192, 0, 0), ("softmax_top", 8, 2, 64, 0, 0), ("sigmoid", 16, 2, 128, 0, 0),
    ("softmax_all", 16, 4, 64, 128, 0), ("softmax_all", 40, 3, 128, 0, 2), ("softmax_all", 8, 4, 64, 64, 1),
    ("softmax_top", 40, 12, 64, 0, 0)])
@pytest.mark.parametrize("rows, hidden", [(65, 72), (100, 264), (300, 256), (1030, 128)])
def test_experts_of_the_chosen_tokens_only_against_every_expert_for_every_token(scoring, experts, top, ff, shared, identity,
                                                                                  rows, hidden):
    """The grouped products (above 64 rows) against 64 bits: with S the sum of the sizes of what an output adds up, an
    activated value rounds to bfloat16, eight bits, once (2^-8 of S in all), the result once (2^-8 of itself); the 32-bit sums of up
    to some hundred terms add less than a tenth to either."""
    from infernum_b200.ops import gemm_tc
    from infernum_b200.parts.base import PartSpec, build_part

    rt = runtime(torch.bfloat16, experts="grouped")  # (the sizes are too small for it to pay)
    params = dict(hidden_size=hidden, expert_size=ff, experts=experts, top=top, scoring=scoring, identity=identity,
                  router_bias="router.b" if scoring != "softmax_all" else None)
    if scoring == "sigmoid":
        params["groups"] = {"count": 4, "keep": 2}
    if shared:
        params["shared"] = {"size": shared, "gate": "g"}
    part = build_part("ffn", PartSpec("moe", params), rt)
    g = torch.Generator(device=DEV).manual_seed(rows + experts)
    w = {n: (torch.randn(s.shape, generator=g, device=DEV) * (0.3 if "router" in n else 0.1)).to(torch.bfloat16)
         for n, s in part.weight_specs().items()}
    part.bind(w)
    x = torch.randn(rows, hidden, generator=g, device=DEV).to(torch.bfloat16)
    x[rows // 2:] = x[: rows - rows // 2].clone()  # (crowds: half of the rows go where the others go)
    x[: rows // 4] = x[0]                          # (and one place gets a quarter of them)
    assert gemm_tc.grouped_suits(x, part.gate_up.weight, part.down.weight, ff, experts, top, "silu")
    got = part.forward(x)
    assert int(rt.error_word().item()) == 0
    ids, wts, gate = part.route(x)
    xd, ref, size = x.double(), torch.zeros(rows, hidden, dtype=torch.float64, device=DEV), 0
    every = [(f"e{e}.", (wts.double() * (ids == e)).sum(1)) for e in range(experts)]
    if shared:
        every.append(("shared.", torch.sigmoid(xd @ w["shared.g"].double().T)[:, 0]))
    for p, by in every:
        a = torch.nn.functional.silu(xd @ w[p + "gate"].double().T) * (xd @ w[p + "up"].double().T) * by[:, None]
        ref += a @ w[p + "down"].double().T
        size = size + a.abs() @ w[p + "down"].double().abs().T
    bound = 1.1 * 2 ** -8 * (size + ref.abs())
    if identity:  # (the input handed on is added to the rounded sum, and the whole rounds again)
        passed = (wts.double() * (ids >= experts)).sum(1)[:, None] * xd
        bound = bound + 1.1 * 2 ** -8 * (ref + passed).abs()
        ref = ref + passed
    assert bool(((got.double() - ref).abs() <= bound + 1e-6).all())
    again = part.forward(x)
    assert torch.equal(got, again)


@pytest.mark.parametrize("rows, experts, hidden", [(1, 1, 8), (3, 17, 264), (5, 2, 264), (6, 3, 1032), (9, 4, 64), (11, 12, 264), (8, 16, 2048), (70, 9, 1032), (2049, 16, 320)])
@pytest.mark.parametrize("dx, dw", [(torch.bfloat16,) * 2, (torch.float32,) * 2, (torch.bfloat16, torch.float32)])
def test_router_logits_of_rows_of_eights(rows, experts, hidden, dx, dw):
    """32-bit sums of ``hidden`` products in a fixed order: within sqrt(hidden) roundings of the sum of their sizes, and
    a row's logits do not depend on the batch."""
    from infernum_b200.ops import core

    x, w = torch.randn(rows, hidden, device=DEV).to(dx), torch.randn(experts, hidden, device=DEV).to(dw)
    out, one = torch.full((rows, experts), float("nan"), device=DEV), torch.empty(1, experts, device=DEV)
    core.router_logits(x, w, out)
    ref = x.double() @ w.double().T
    size = x.double().abs() @ w.double().abs().T
    assert bool(((out.double() - ref).abs() <= size * 2 ** -24 * max(4.0, hidden ** 0.5)).all())
    core.router_logits(x[rows - 1:], w, one)
    assert torch.equal(one[0], out[rows - 1])


@pytest.mark.parametrize("heads, window, sink, gate, q_rank", [(4, 0, False, False, 64), (3, 100, True, True, 0),
                                                               (8, 300, True, False, 64)])
@pytest.mark.parametrize("dim, vdim", [(128, 128), (128, 64), (64, 128), (64, 64)])
@pytest.mark.parametrize("past, new, page", [([0], [64], 16), ([0], [129], 4), ([0, 77, 300], [200, 65, 128], 16),
                                             ([513, 0], [300, 31], 32), ([128], [256], 128)])
def test_latent_attention_over_made_keys_against_the_plain_kernel(heads, window, sink, gate, q_rank, dim, vdim, past, new, page):
    """Prompts of many rows make every head's keys and values; the plain kernel attends over the latents in 32-bit.  Both
    round a handful of intermediate rows to bfloat16, other ones: bfloat16's tolerance of these tests.  Every page
    and slot without a token is NaN."""
    from types import SimpleNamespace

    from infernum_b200.cache import CacheManager
    from infernum_b200.ops import attention_expanded
    from infernum_b200.parts.base import PartSpec, build_part

    hidden, outs, made = 96, [], []
    for options in ({}, {"attention": "plain"}):
        rt = runtime(torch.bfloat16, **options)
        part = build_part("mixer", PartSpec("latent_attention", dict(
            hidden_size=hidden, num_heads=heads, dim=dim, rot_dim=64, vdim=vdim, q_rank=q_rank, kv_rank=64, scale=0.08,
            window=window, eps=1e-5, theta=10000.0, sink="sink" if sink else None, gate="g" if gate else None)), rt)
        gen = torch.Generator(device=DEV).manual_seed(heads + page)
        part.bind({n: (torch.randn(s.shape, generator=gen, device=DEV) * (1.0 if "norm" in n or n == "sink" else 0.15)).to(
            torch.bfloat16) for n, s in part.weight_specs().items()})
        need = SimpleNamespace(position=0, paged=part.cache_spec(), state=None, cache_of=None)
        cache = CacheManager([need], page_size=page, num_pages=sum(-(-(p + n) // page) for p, n in zip(past, new)) + 3,
                             max_requests=len(past), dtype=torch.bfloat16, device=DEV)
        held = []
        for e, p in enumerate(past):
            rc = cache.admit(e)
            cache.extend(rc, p)
            cache.commit(rc, p)
            held.append(rc)
        ctx = step_ctx(cache, list(zip(held, new)))
        pool = cache.layer_caches[0].k_pool
        pool.fill_(float("nan"))
        for rc, p in zip(held, past):
            for i, pg in enumerate(rc.tables[0]):
                n = min(page, p - i * page)
                if pg >= 0 and n > 0:
                    pool[pg, 0, :n] = torch.randn(n, 128, generator=gen, device=DEV).to(torch.bfloat16)
        x = torch.randn(sum(new), hidden, generator=gen, device=DEV).to(torch.bfloat16)
        made.append(attention_expanded.plan(ctx, sum(new), window, 1))
        outs.append(part.forward(x, ctx, cache.layer_caches[0]))
        assert int(rt.error_word().item()) == 0
    wide = sum(new) >= 64 * len(new)
    assert (made[0] > 0) == wide
    assert outs[0].isfinite().all() and rel_err(outs[0], outs[1]) < TOL[torch.bfloat16]


@pytest.mark.parametrize("short", [0, 1, 200])
def test_keys_that_find_no_row_in_the_buffer_are_reported(short):
    """The gathered latents end with the buffer: one that is too small sets the error word and is written to its end only."""
    from infernum_b200.ops import attention_expanded, core

    lib, i32 = attention_expanded.lib_for(128, 64, 128), lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    pool = torch.randn(40, 1, 16, 128, device=DEV).to(torch.bfloat16)
    tables, cu, start = i32([list(range(20)), list(range(20, 40))]), i32([0, 70, 170]), i32([230, 0])
    keys = (300 - 128) + 100  # (a window of 90: the first entry's first row sees keys from 141 on, its buffer begins at 128)
    out = torch.full((keys + 3, 128), 7.0, dtype=torch.bfloat16, device=DEV)
    err = core.new_error_word(DEV)
    core.check(lib.ib_gather_latents(pool.data_ptr(), out.data_ptr(), cu.data_ptr(), start.data_ptr(), tables.data_ptr(), 20, 2,
                                     16, 40, 90, 128, keys - short, err.data_ptr(), core.stream_ptr(out)), "gather_latents")
    want = torch.cat([torch.zeros(13, 128, device=DEV), pool.view(-1, 128)[141:300].float(), pool.view(-1, 128)[320:420].float()])
    assert torch.equal(out[: keys - short].float(), want[: keys - short]) and bool((out[keys - short:] == 7.0).all())
    assert int(err.item()) == (core.FLAG_KEYS_LOST if short else 0)
    assert "buffer made for them" in core.describe_flags(core.FLAG_KEYS_LOST)


@pytest.mark.parametrize("rule, heads, groups, rows, cols", [("ssd", 4, 2, 128, 64), ("ssd", 3, 1, 64, 128),
                                                             ("delta", 4, 2, 128, 128), ("delta", 3, 3, 64, 64),
                                                             ("delta", 2, 1, 128, 192)])
@pytest.mark.parametrize("lens", [[96], [128, 1, 63], [131, 64, 200], [0, 300], [65, 100, 193, 40]])
def test_scans_in_chunks_against_one_token_at_a_time(rule, heads, groups, rows, cols, lens):
    """The kernels for prompts against the token-by-token one, which a state whose rows are an odd number of floats apart
    asks for: the same 32-bit sums in another order, over states of some hundred decaying tokens.  A token's result does
    not see what comes after it, not even a NaN."""
    from types import SimpleNamespace

    from infernum_b200.ops import scan

    rt, N, E = runtime(torch.float32, scan="chunks"), sum(lens), len(lens)  # (also where they do not pay)
    g = torch.Generator(device=DEV).manual_seed(N + rows)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    cu = [sum(lens[:i]) for i in range(E + 1)]
    ctx = SimpleNamespace(n_entries=E, n_rows=N, max_rows_per_entry=max(lens), cu_rows=i32(cu), slot_ids=i32(list(range(E))),
                          row_entry=i32([e for e, n in enumerate(lens) for _ in range(n)]))
    size, inner = heads * rows * cols, heads * cols
    start = rnd(E, size)
    width = 2 * groups * rows + inner + 4 * heads  # (rows of fours)
    x, a_log, dt_bias, skip = rnd(N, width), rnd(heads) * 0.5, rnd(heads) - 1.0, rnd(heads)
    channels = width - 4 * heads
    taps = 3 if rule == "delta" and rows == 64 else 4  # (four: the pass before the scan by rows)
    conv, tail = (rnd(channels, taps) * 0.5, rnd(channels), size), size + (taps - 1) * channels  # (the last inputs behind)

    def walk(x, stride):
        state = torch.full((E + 1, stride), 7.0, device=DEV)
        state[:E, :size] = start
        out = torch.empty(N, inner, device=DEV)
        if rule == "ssd":
            scan.ssd_scan(x[:, : inner + 2 * groups * rows], x[:, width - heads:], dt_bias, a_log, skip, state, 0, ctx, out,
                          heads, groups, rows, cols, rt, conv=conv)
        else:
            scan.delta_scan(x, 0, width - 2 * heads, width - heads, conv[0], a_log, dt_bias, state, 0, size, ctx, out, heads,
                            groups, rows, cols, rt)
        return out, state

    assert scan.in_chunks(ctx, N, rows, cols, 0, tail + 8) and not scan.in_chunks(ctx, N, rows, cols, 0, tail + 9)
    assert not scan.in_chunks(ctx, N, rows, cols, 0, tail + 8, heads=1 << 17)  # (more scratch than it may have)
    out, state = walk(x, tail + 8)
    ref, ref_state = walk(x, tail + 9)
    assert rel_err(out, ref) < 1e-5 and rel_err(state[:E, :size], ref_state[:E, :size]) < 1e-5
    assert torch.equal(state[:, size: tail], ref_state[:, size: tail])
    assert bool((state[:, tail:] == 7.0).all()) and bool((state[E] == 7.0).all())
    last = next(e for e in range(E) if lens[e] >= 96)
    at = cu[last] + lens[last] - 2  # the token before the entry's last
    bad = x.clone()
    bad[at] = float("nan")
    got, _ = walk(bad, tail + 8)
    keep = torch.ones(N, dtype=torch.bool, device=DEV)
    keep[at: at + 2] = False
    assert torch.equal(got[keep], out[keep]) and bool(got[at].isnan().all())


@pytest.mark.parametrize("kind, params, step", [
    ("latent_attention", dict(num_heads=8, dim=128, rot_dim=64, vdim=128, q_rank=128, kv_rank=128, scale=0.07, window=0,
                              theta=10000.0, gate="g"), [(0, 700), (77, 300)]),      # keys made
    ("latent_attention", dict(num_heads=16, dim=128, rot_dim=64, vdim=128, q_rank=0, kv_rank=128, scale=0.07, window=0,
                              theta=10000.0, gate="g"), [(900, 1), (30, 1), (400, 1)]),   # slices of the latents
    ("ssd", dict(num_heads=8, vdim=64, state=128, groups=2, conv=4, norm_groups=1), [(0, 400), (0, 77)]),
    ("delta", dict(num_heads=8, num_kv_heads=4, head_dim=128, vdim=128, conv=4), [(0, 333), (0, 200)])])
def test_parts_whose_kernels_begin_early_give_the_same_bits(kind, params, step):
    """Pass after pass on other inputs, over the same buffers: a value read before the kernel in front wrote it, or from
    an older line of a cache, is another pass's.  Against the same passes with every kernel launched after the one before."""
    from types import SimpleNamespace

    from infernum_b200.cache import CacheManager
    from infernum_b200.csrc import build
    from infernum_b200.ops import core
    from infernum_b200.parts.base import PartSpec, build_part

    rt, width = runtime(torch.bfloat16), 512
    part = build_part("mixer", PartSpec(kind, dict(hidden_size=width, eps=1e-5, **params)), rt)
    gen = torch.Generator(device=DEV).manual_seed(3)
    part.bind({n: (torch.randn(s.shape, generator=gen, device=DEV) * (0.5 if len(s.shape) == 1 else 0.05)).to(torch.bfloat16)
               for n, s in part.weight_specs().items()})
    need = SimpleNamespace(position=0, paged=part.cache_spec(), state=part.state_spec(), cache_of=None)
    cache = CacheManager([need], page_size=16, num_pages=200, max_requests=len(step), dtype=torch.bfloat16, device=DEV)
    held = []
    for e, (past, _) in enumerate(step):
        held.append(cache.admit(e))
        if past:
            cache.extend(held[e], past)
            cache.commit(held[e], past)
    ctx, layer = step_ctx(cache, [(rc, n) for rc, (_, n) in zip(held, step)]), cache.layer_caches[0]
    inputs = torch.randn(12, sum(n for _, n in step), width, generator=gen, device=DEV).to(torch.bfloat16)
    old = torch.randn(layer.k_pool.shape, generator=gen, device=DEV).to(torch.bfloat16) if need.paged else None
    runs = []
    try:
        for early in (1, 0):
            for lib in build._loaded.values():
                if hasattr(lib, "ib_set_pdl"):
                    lib.ib_set_pdl(early)
            outs = []
            with core.step_stream(DEV):
                for x in [*inputs, *inputs]:
                    (layer.k_pool.copy_(old) if need.paged else layer.state.zero_())
                    core.step_fence(DEV)
                    outs.append(part.forward(x, ctx, layer).clone())
            torch.cuda.synchronize()
            runs.append(outs)
    finally:
        for lib in build._loaded.values():
            if hasattr(lib, "ib_set_pdl"):
                lib.ib_set_pdl(1)
    assert int(rt.error_word().item()) == 0
    for a, b in zip(*runs):
        assert a.isfinite().all() and torch.equal(a, b)
