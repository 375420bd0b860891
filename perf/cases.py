"""What is timed when this engine's speed is looked at: calls that a program makes through the engine's public parts, at
the sizes of bench.py's workloads.

Whole steps (``decode``: one step of a batch of requests from its CUDA graph; ``prompt``: a prompt in one step) run the
Llama-3.2-1B sizes with all layers.  Everything else is a part or a block on its own: built from its constructor, bound to
seeded weights, run over a cache manager's pages or state, as ``DecoderModel`` runs it.  Calls of up to 1,024 tokens are
replayed from a CUDA graph, as the engine replays its steps of that size; larger ones are launched kernel by kernel, as the
engine launches those.  A part's update goes through the RMS norm that folds it into the residual stream, as it does in
every model, so the outputs do not depend on the form in which the update travels.
"""

from __future__ import annotations

import math

import numpy as np
import torch

DEV = "cuda:0"
PAGE = 16
EPS = 1e-5
GRAPH_TOKENS = 1024  # the engine's default: steps of up to so many tokens are replayed from graphs
LLAMA_1B = dict(width=2048, heads=32, kv_heads=8, head_dim=64, inner=8192, layers=16, vocab=128256)
LLAMA_3B = dict(width=3072, heads=24, kv_heads=8, head_dim=128, inner=8192)
LLAMA_8B = dict(width=4096, heads=32, kv_heads=8, head_dim=128, inner=14336)
THETA = 500000.0
SCALING = dict(rope_type="llama3", factor=32.0, low_freq_factor=1.0, high_freq_factor=4.0,
               original_max_position_embeddings=8192)


# ------------------------------------------------------------------------------------------------------------ the cases
def listed():
    sizes = {k: v for k, v in LLAMA_1B.items() if k not in ("layers", "vocab")}
    return [
        # the headline workload: eight users' next tokens, every request with a 2,048-token prompt behind it
        dict(name="decode_8x2048", kind="decode", requests=8, context=2048),
        # time to the first token of one 2,048-token prompt
        dict(name="prompt_2048", kind="prompt", tokens=2048),
        # a server's mixed step, one layer of Llama-3.2-3B sizes: 32 users decode while a long prompt's portion comes in
        dict(name="block_mixed_3b", kind="block", dtype="bfloat16", decoding=32, context=4096, portion=2048, ahead=2048, **LLAMA_3B),
        # the exact path: a layer in float32, a short prompt
        dict(name="block_f32_prompt_500", kind="block", dtype="float32", decoding=0, context=0, portion=500, ahead=0, **sizes),
        # the exact path, four requests' next tokens: the smallest call of all
        dict(name="block_f32_decode_4", kind="block", dtype="float32", decoding=4, context=600, portion=0, ahead=0, **sizes),
        # a busy server's decode attention at long, unequal contexts
        dict(name="attention_decode_64", kind="attention", requests=64, context=8192, **LLAMA_8B),
        # the feed-forward of a medium batch, Llama-3.1-8B sizes
        dict(name="mlp_rows_48", kind="mlp", width=4096, inner=14336, rows=48),
        # decayed linear attention over one whole prompt
        dict(name="linear_decayed_2048", kind="linear", form="decayed", heads=16, width=2048, prompts=1, tokens=2048, decoding=0),
        # gated linear attention over several prompts of unequal length that arrived together
        dict(name="linear_gated_3x", kind="linear", form="gated", heads=16, width=2048, prompts=3, tokens=3001, decoding=0),
        # windowed attention with capped scores and a sink over two prompts
        dict(name="sink_prompts_4001", kind="sink", heads=32, kv_heads=8, dim=64, width=2048, window=1024, softcap=50.0,
             prompts=2, tokens=4001, decoding=0, context=0),
        # latent attention over one whole prompt
        dict(name="latent_2048", kind="latent", heads=16, width=2048, q_rank=768, window=1024, prompts=1, tokens=2048, decoding=0,
             context=0),
        # routed experts for a small batch of decoding requests
        dict(name="experts_rows_16", kind="experts", width=2048, inner=2048, experts=16, top=4, rows=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another case of the same kinds: batch sizes, prompt lengths and contexts over their whole range, odd ones among them."""
    kind = rng.choice(["decode", "prompt", "block", "block_f32", "attention", "mlp", "linear", "linear", "sink", "latent",
                       "experts"])
    sizes_1b = {k: v for k, v in LLAMA_1B.items() if k not in ("layers", "vocab")}
    if kind == "decode":
        n = _log(rng, 1, 32)
        return dict(kind=kind, requests=n, context=min(_log(rng, 64, 3000), 16384 // n))
    if kind == "prompt":
        return dict(kind=kind, tokens=_log(rng, 33, 2048))
    if kind == "block":
        return dict(kind=kind, dtype="bfloat16", decoding=rng.randint(0, 40), context=_log(rng, 256, 4096),
                    portion=_log(rng, 64, 2048), ahead=rng.choice([0, 0, rng.randint(1, 2048)]),
                    **rng.choice([sizes_1b, LLAMA_3B, LLAMA_8B]))
    if kind == "block_f32":
        if rng.random() < 0.5:
            return dict(kind="block", dtype="float32", decoding=_log(rng, 1, 24), context=_log(rng, 64, 1500), portion=0, ahead=0,
                        **sizes_1b)
        return dict(kind="block", dtype="float32", decoding=0, context=0, portion=_log(rng, 20, 700), ahead=0, **sizes_1b)
    if kind == "attention":
        z = rng.choice([sizes_1b, LLAMA_3B, LLAMA_8B])
        return dict(kind=kind, requests=_log(rng, 1, 64), context=_log(rng, 300, 8192), **z)
    if kind == "mlp":
        width, inner = rng.choice([(2048, 8192), (3072, 8192), (4096, 14336)])
        return dict(kind=kind, width=width, inner=inner, rows=_log(rng, 1, 600))
    if kind == "linear":
        heads = rng.choice([8, 16, 24, 32])
        case = dict(kind=kind, form=rng.choice(["decayed", "gated", "forget"]), heads=heads, width=128 * heads)
        if rng.random() < 0.25:
            return dict(case, prompts=0, tokens=0, decoding=_log(rng, 1, 64))
        prompts = rng.randint(1, 4)
        return dict(case, prompts=prompts, tokens=prompts * 8 + _log(rng, 100, 3000), decoding=rng.choice([0, 0, 5]))
    if kind == "sink":
        heads, kv, dim = rng.choice([(32, 8, 64), (16, 4, 64), (16, 4, 128), (32, 8, 128)])
        case = dict(kind=kind, heads=heads, kv_heads=kv, dim=dim, width=heads * dim, window=rng.choice([512, 1024, 0]),
                    softcap=rng.choice([0.0, 30.0, 50.0]))
        if rng.random() < 0.25:
            return dict(case, prompts=0, tokens=0, decoding=_log(rng, 1, 64), context=_log(rng, 300, 4096))
        prompts = rng.randint(1, 4)
        return dict(case, prompts=prompts, tokens=prompts * 8 + _log(rng, 200, 4000), decoding=rng.choice([0, 0, 7]), context=1500)
    if kind == "latent":
        heads = rng.choice([16, 32])
        case = dict(kind=kind, heads=heads, width=128 * heads, q_rank=48 * heads, window=rng.choice([512, 1024, 0]))
        if rng.random() < 0.25:
            return dict(case, prompts=0, tokens=0, decoding=_log(rng, 1, 64), context=_log(rng, 300, 4096))
        prompts = rng.randint(1, 3)
        return dict(case, prompts=prompts, tokens=prompts * 8 + _log(rng, 200, 2100), decoding=rng.choice([0, 0, 6]), context=1200)
    width, inner = rng.choice([(2048, 2048), (2048, 1024), (4096, 1024)])
    return dict(kind=kind, width=width, inner=inner, experts=16, top=rng.choice([2, 4]), rows=_log(rng, 1, 1024))


# ------------------------------------------------------------------------------------------------------------ the inputs
class _Seeded:
    """Tensors drawn one after the other from one seed, on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(DEV).manual_seed(int(seed))

    def normal(self, shape, std=1.0, dtype=torch.float32):
        return (torch.randn(shape, generator=self.g, device=DEV) * std).to(dtype)

    def uniform(self, shape, lo, hi):
        return torch.rand(shape, generator=self.g, device=DEV) * (hi - lo) + lo

    def matrix(self, rows, cols, dtype):
        return self.normal((rows, cols), cols ** -0.5, dtype)


def _dtype(case):
    return torch.float32 if case.get("dtype") == "float32" else torch.bfloat16


def _split(total, parts, least=8):
    """``total`` tokens in ``parts`` prompts of unequal length."""
    if parts <= 0:
        return []
    shares = [1.0 + 0.37 * ((i * 7) % 5) for i in range(parts)]
    lens = [max(least, int(total * s / sum(shares))) for s in shares]
    lens[0] += total - sum(lens)
    return lens


def _contexts(requests, most):
    """Unequal context lengths: from an eighth of ``most`` to all of it."""
    return [max(1, int(most * (0.125 + 0.875 * ((i * 29) % 64) / 63.0)) - (i * 13) % 7) for i in range(requests)]


def _requests(case):
    """[(new tokens, tokens before them)] of one step, the requests that decode first."""
    k = case["kind"]
    if k == "attention":
        return [(1, c) for c in _contexts(case["requests"], case["context"])]
    if k == "block":
        return [(1, c) for c in _contexts(case["decoding"], case["context"])] + ([(case["portion"], case["ahead"])] if case["portion"] else [])
    if k in ("sink", "latent"):
        return [(1, c) for c in _contexts(case["decoding"], case["context"])] + [(n, 0) for n in _split(case["tokens"], case["prompts"])]
    return [(1, 777) for _ in range(case["decoding"])] + [(n, 0) for n in _split(case["tokens"], case["prompts"])]


def _llama_weights(case, d):
    W, H, G, hd, I = case["width"], case["heads"], case["kv_heads"], case["head_dim"], case["inner"]
    t = _dtype(case)
    return dict(n1=d.uniform((W,), 0.5, 1.5), q=d.matrix(H * hd, W, t), k=d.matrix(G * hd, W, t), v=d.matrix(G * hd, W, t),
                o=d.matrix(W, H * hd, t), n2=d.uniform((W,), 0.5, 1.5), g=d.matrix(I, W, t), u=d.matrix(I, W, t),
                d=d.matrix(W, I, t), n3=d.uniform((W,), 0.5, 1.5))


def _linear_weights(case, d):
    W, H, C, b = case["width"], case["heads"], case["heads"] * 128, torch.bfloat16
    w = dict(q=d.matrix(C, W, b), k=d.matrix(C, W, b), v=d.matrix(C, W, b), g=d.matrix(C, W, b), o=d.matrix(W, C, b),
             n3=d.uniform((W,), 0.5, 1.5))
    if case["form"] == "decayed":
        w["norm"] = d.uniform((C,), 0.5, 1.5)
    elif case["form"] == "gated":
        w.update(a1=d.matrix(64, W, b), a2=d.matrix(C, 64, b), a2_bias=d.normal((C,), 0.5), norm=d.uniform((128,), 0.5, 1.5))
    else:
        w.update(f_bias=d.normal((C,), 0.5), lower=d.uniform((C,), 0.0, 0.9), norm=d.uniform((128,), 0.5, 1.5))
    return w


def _decays(heads):
    return [1.0 - 2.0 ** -(2 + 6 * h / (heads - 1)) for h in range(heads)]


def _sink_weights(case, d):
    W, H, G, e, b = case["width"], case["heads"], case["kv_heads"], case["dim"], torch.bfloat16
    return dict(q=d.matrix(H * e, W, b), k=d.matrix(G * e, W, b), v=d.matrix(G * e, W, b), o=d.matrix(W, H * e, b),
                sink=d.normal((H,)), qb=d.normal((H * e,), 0.1), kb=d.normal((G * e,), 0.1), vb=d.normal((G * e,), 0.1),
                n3=d.uniform((W,), 0.5, 1.5))


LAT = dict(dim=128, rot=64, vdim=128, rank=192)


def _latent_weights(case, d):
    W, H, r, b = case["width"], case["heads"], case["q_rank"], torch.bfloat16
    return dict(dq=d.matrix(r, W, b), dq_norm=d.uniform((r,), 0.5, 1.5), uq=d.matrix(H * 192, r, b), dkv=d.matrix(256, W, b),
                dkv_norm=d.uniform((192,), 0.5, 1.5), uk=d.matrix(H * 128, 192, b), uv=d.matrix(H * 128, 192, b),
                o=d.matrix(W, H * 128, b), n3=d.uniform((W,), 0.5, 1.5))


def _expert_weights(case, d):
    W, I, E, b = case["width"], case["inner"], case["experts"], torch.bfloat16
    w = dict(router=d.matrix(E, W, torch.float32), n3=d.uniform((W,), 0.5, 1.5))
    for e in range(E):
        w.update({f"g{e}": d.matrix(I, W, b), f"u{e}": d.matrix(I, W, b), f"d{e}": d.matrix(W, I, b)})
    return w


def _mlp_weights(case, d):
    W, I, b = case["width"], case["inner"], torch.bfloat16
    return dict(g=d.matrix(I, W, b), u=d.matrix(I, W, b), d=d.matrix(W, I, b), n3=d.uniform((W,), 0.5, 1.5))


def _model_weights(d):
    z, b = LLAMA_1B, torch.bfloat16
    W, H, G, hd, I = z["width"], z["heads"], z["kv_heads"], z["head_dim"], z["inner"]
    w = {"model.embed_tokens.weight": d.normal((z["vocab"], W), 0.02, b), "model.norm.weight": d.uniform((W,), 0.5, 1.5)}
    for i in range(z["layers"]):
        p = f"model.layers.{i}."
        w[p + "input_layernorm.weight"] = d.uniform((W,), 0.5, 1.5)
        w[p + "post_attention_layernorm.weight"] = d.uniform((W,), 0.5, 1.5)
        for name, rows, cols in (("self_attn.q_proj", H * hd, W), ("self_attn.k_proj", G * hd, W), ("self_attn.v_proj", G * hd, W),
                                 ("self_attn.o_proj", W, H * hd), ("mlp.gate_proj", I, W), ("mlp.up_proj", I, W),
                                 ("mlp.down_proj", W, I)):
            w[p + name + ".weight"] = d.normal((rows, cols), 0.02, b)
    return w


def _whole_inputs(case, seed):
    """The weights and each request's token ids (a decoding request's last id is the one that its step feeds)."""
    d = _Seeded(seed)
    w = _model_weights(d)
    n, length = (case["requests"], case["context"] + 1) if case["kind"] == "decode" else (1, case["tokens"])
    ids = torch.randint(0, LLAMA_1B["vocab"], (n, length), generator=d.g, device=DEV)
    return w, ids


def _past(case, d):
    """What stands in the cache before the step: for each request the rows of its earlier tokens, or its state."""
    k, reqs, t = case["kind"], _requests(case), _dtype(case)
    if k in ("block", "attention"):
        G, hd = case["kv_heads"], case["head_dim"]
        return [(d.normal((G, c, hd), 1.0, t), d.normal((G, c, hd), 1.0, t)) if c else None for _, c in reqs]
    if k == "sink":
        return [d.normal((case["kv_heads"], c, 2 * case["dim"]), 1.0, t) if c else None for _, c in reqs]
    if k == "latent":
        return [d.normal((1, c, 256), 1.0, t) if c else None for _, c in reqs]
    if k == "linear":  # the state S, [head][key channel][value]
        return [d.normal((case["heads"], 128, 128), 0.3) if c else None for _, c in reqs]
    return None


def _part_inputs(case, seed):
    d = _Seeded(seed)
    w = dict(block=_llama_weights, attention=_llama_weights, mlp=_mlp_weights, linear=_linear_weights, sink=_sink_weights,
             latent=_latent_weights, experts=_expert_weights)[case["kind"]](case, d)
    rows = case["rows"] if "rows" in case else sum(n for n, _ in _requests(case))
    x = d.normal((rows, case["width"]))
    h = d.normal((rows, case["width"]), 1.0, _dtype(case))
    past = _past(case, d) if "rows" not in case else None
    return w, x, h, past


# ------------------------------------------------------------------------------------------------------------- the calls
def prepare(case, seed):
    return _prepare_whole(case, seed) if case["kind"] in ("decode", "prompt") else _prepare_part(case, seed)


def _prepare_whole(case, seed):
    from tokasaurus_b200.engine.batch import StepEntry
    from tokasaurus_b200.engine.engine import Engine

    z = LLAMA_1B
    cfg = dict(architectures=["LlamaForCausalLM"], model_type="llama", num_hidden_layers=z["layers"], hidden_size=z["width"],
               num_attention_heads=z["heads"], num_key_value_heads=z["kv_heads"], intermediate_size=z["inner"],
               vocab_size=z["vocab"], rope_theta=THETA, rope_scaling=SCALING, rms_norm_eps=EPS, tie_word_embeddings=True,
               max_position_embeddings=131072)
    w, ids = _whole_inputs(case, seed)
    n, length = ids.shape
    eng = Engine(config_dict=cfg, random_weights=0, dtype="bfloat16", page_size=PAGE,
                 kv_cache_num_tokens=n * (-(-(length + 1) // PAGE) * PAGE), max_tokens_per_forward=8192, max_seqs_per_forward=64,
                 device=DEV)
    runner, cache = eng.runner, eng.runner.cache
    runner.model.bind(w, runner.rt)
    tokens = ids.tolist()
    names = [f"r{i}" for i in range(n)]
    for r in names:
        cache.admit(r)
        cache.ensure_capacity(r, length)
    if case["kind"] == "prompt":
        return dict(engine=eng, entries=[StepEntry(names[0], tokens[0], 0, [length - 1])])
    for r, t in zip(names, tokens):
        runner.step([StepEntry(r, t[:-1], 0, [length - 2])])
    extra = dict(temperature=np.zeros(n, dtype=np.float32), stream_key=np.zeros(n, dtype=np.int64),
                 sample_pos=np.full(n, length, dtype=np.int32),
                 row_slot=np.asarray([cache.slot(r) for r in names], dtype=np.int32))
    entries = [StepEntry(r, [t[-1]], length - 1, [0]) for r, t in zip(names, tokens)]
    eng.graphs.run(entries, extra)  # records the graph, as a server does before it takes requests
    return dict(engine=eng, entries=entries, extra=extra, n=n)


def _part(case):
    """The part under test and the norm that folds its update in."""
    from tokasaurus_b200 import parts as P

    k, W = case["kind"], case["width"]
    out_norm = P.RMSNorm(W, EPS, "n3")
    if k in ("block", "attention"):
        mixer = P.PagedAttention(W, case["heads"], case["kv_heads"], case["head_dim"], P.RotaryEncoding(case["head_dim"], THETA),
                                 "q", "k", "v", "o")
        if k == "attention":
            return mixer, out_norm
        return P.PreNormBlock(P.RMSNorm(W, EPS, "n1"), mixer, P.RMSNorm(W, EPS, "n2"),
                              P.GatedMLP(W, case["inner"], "g", "u", "d")), out_norm
    if k == "mlp":
        return P.GatedMLP(W, case["inner"], "g", "u", "d"), out_norm
    if k == "linear":
        H = case["heads"]
        if case["form"] == "decayed":
            return P.DecayedLinearAttention(W, H, 128, 128, _decays(H), EPS, "q", "k", "v", "g", "norm", "o"), out_norm
        if case["form"] == "gated":
            return P.GatedLinearAttention(W, H, 128, 128, 16.0, EPS, "q", "k", "v", "g", "a1", "a2", "a2_bias", "norm", "o"), out_norm
        return P.GatedLinearRecurrence(W, H, 128, 128, EPS, "q", "k", "f_bias", "lower", "v", "norm", "o"), out_norm
    if k == "sink":
        return P.SinkAttention(W, case["heads"], case["kv_heads"], case["dim"], case["dim"], case["dim"] ** -0.5,
                               case["softcap"] or None, case["window"] or None, EPS, "q", "k", "v", "o", "sink",
                               bias_names=("qb", "kb", "vb")), out_norm
    if k == "latent":
        return P.LatentAttention(W, case["heads"], LAT["dim"], LAT["rot"], LAT["vdim"], LAT["rank"], case["q_rank"], 192 ** -0.5,
                                 10000.0, LAT["rot"], EPS, case["window"] or None,
                                 names={n: n for n in ("dq", "dq_norm", "uq", "dkv", "dkv_norm", "uk", "uv", "o")}), out_norm
    return P.RoutedExperts(W, case["inner"], case["experts"], case["top"], "router", None,
                           lambda e: (f"g{e}", f"u{e}", f"d{e}")), out_norm


def _prepare_part(case, seed):
    from tokasaurus_b200.cache import CacheManager
    from tokasaurus_b200.engine.batch import Stager, StepContext, StepEntry, build_host_batch
    from tokasaurus_b200.engine.runtime import Runtime
    from tokasaurus_b200.parts import ResidualStream

    w, x, h, past = _part_inputs(case, seed)
    rt = Runtime.make(DEV, "float32" if _dtype(case) == torch.float32 else "bfloat16")
    part, norm = _part(case)
    part.bind(w, rt)
    norm.bind(w, rt)
    del w
    ctx = cache = state = None
    if past is not None:
        mixer = getattr(part, "mixer", part)
        reqs = _requests(case)
        pages = sum(-(-(n + c) // PAGE) for n, c in reqs)
        cm = CacheManager({0: mixer.cache_need()}, PAGE, max(pages, 1), max(len(reqs), 1), dtype=rt.dtype, device=rt.device)
        entries = []
        cache = cm.layer_cache(0)
        for i, (n, c) in enumerate(reqs):
            cm.admit(i)
            cm.ensure_capacity(i, n + c)
            entries.append(StepEntry(i, [0] * n, c, [n - 1]))
            if past[i] is None:
                continue
            if case["kind"] == "linear":
                cache.state[cm.slot(i)] = past[i].transpose(1, 2).reshape(cache.state.shape[1:])  # kept transposed
                continue
            table = torch.as_tensor(cm.requests[i].table_array(0)[: -(-c // PAGE)], device=DEV).long()
            for rows, pool in zip(past[i] if isinstance(past[i], tuple) else (past[i],), (cache.k, cache.v)):
                G, _, D = rows.shape
                padded = torch.zeros((G, table.numel() * PAGE, D), dtype=rows.dtype, device=DEV)
                padded[:, :c] = rows
                pool[table] = padded.view(G, table.numel(), PAGE, D).transpose(0, 1)
        host = build_host_batch(entries, cm)
        key = mixer.plan_key()
        plans = {key: mixer.plan(host)} if key is not None else {}
        ctx = StepContext(host, cm, rt.device, Stager(rt.device), None, plans)
        state = getattr(cache, "state", None)
    else:
        ctx = _Rows(x.shape[0])
    is_block = case["kind"] == "block"

    def call():
        stream = ResidualStream(x.clone())
        if is_block:
            stream = part.forward(ctx, stream, cache)
        elif past is None:
            stream.delta = part.forward(ctx, h)
        else:
            stream.delta = part.forward(ctx, h, cache)
        return dict(h=norm.forward(ctx, stream), x=stream.x, **({"state": state} if state is not None else {}))

    keep = dict(part=part, norm=norm, ctx=ctx, cache=cache, call=call, graph=None)
    if x.shape[0] <= GRAPH_TOKENS:
        before = state.clone() if state is not None else None
        call()
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            keep["out"] = call()
        keep["graph"] = g
        if state is not None:  # the call above moved the requests on
            state.copy_(before)
    return keep


class _Rows:
    """What a feed-forward wants to know of a step whose rows are all tokens."""

    def __init__(self, n):
        self.n_tokens = n
        self.token_seq = torch.arange(n, dtype=torch.int32, device=DEV)
        self.status = torch.zeros(1, dtype=torch.int32, device=DEV)


def run(state):
    if "engine" not in state:
        if state["graph"] is None:
            return state["call"]()
        state["graph"].replay()
        return state["out"]
    eng = state["engine"]
    if "extra" not in state:
        return dict(logits=eng.runner.step(state["entries"]), kv=eng.runner.cache.groups[0].storage)
    prep = eng.graphs.prepare(state["entries"], state["extra"])
    eng.graphs.launch(prep)
    return dict(logits=eng.graphs.graphs[prep["key"]]["logits"][:state["n"]])


# ------------------------------------------------------------------------------- what a pass cannot do without, tolerances
def _seen(case):
    """(query, key) pairs of a step, and key rows that are read from the cache."""
    pairs = rows = 0
    win = case.get("window") or 1 << 60
    for n, c in _requests(case):
        pairs += sum(min(c + i + 1, win) for i in range(n))
        rows += min(c, win + n)
    return pairs, rows


def work(case):
    k = case["kind"]
    if k in ("decode", "prompt"):
        z = LLAMA_1B
        W, H, G, hd, I = z["width"], z["heads"], z["kv_heads"], z["head_dim"], z["inner"]
        layer = W * (H + 2 * G) * hd + H * hd * W + 3 * W * I
        params = z["layers"] * layer + z["vocab"] * W
        row = 2 * G * hd * 2 * z["layers"]
        if k == "decode":
            n, c = case["requests"], case["context"]
            return dict(bytes=2 * params + n * (c + 1) * row + 4 * n * z["vocab"], flops=2 * n * params + 4 * n * c * H * hd * z["layers"])
        n = case["tokens"]
        return dict(bytes=2 * params + n * row, flops=2 * n * z["layers"] * layer + 2 * n * (n + 1) * H * hd * z["layers"] + 2 * z["vocab"] * W)
    W, s = case["width"], 4 if _dtype(case) == torch.float32 else 2
    rows = case["rows"] if "rows" in case else sum(n for n, _ in _requests(case))
    ends = rows * W * (4 + 4 + 2 * s)  # the stream in and out, the rows in and out
    if k in ("block", "attention"):
        H, G, hd, I = case["heads"], case["kv_heads"], case["head_dim"], case["inner"]
        params = W * (H + 2 * G) * hd + H * hd * W + (3 * W * I if k == "block" else 0)
        pairs, past = _seen(case)
        return dict(bytes=s * params + 2 * G * hd * s * (past + rows) + ends, flops=2 * rows * params + 4 * pairs * H * hd)
    if k == "mlp":
        params = 3 * W * case["inner"]
        return dict(bytes=s * params + ends, flops=2 * rows * params)
    if k == "linear":
        C = case["heads"] * 128
        params = W * C * (4 if case["form"] == "forget" else 5) + (64 * (W + C) if case["form"] == "gated" else 0)
        return dict(bytes=2 * params + ends + 2 * 4 * 128 * C * len(_requests(case)), flops=2 * rows * params + 6 * rows * C * 128)
    if k == "sink":
        H, G, e = case["heads"], case["kv_heads"], case["dim"]
        params = W * e * (2 * H + 2 * G)
        pairs, past = _seen(case)
        return dict(bytes=2 * params + ends + 2 * 2 * G * e * (past + rows), flops=2 * rows * params + 4 * pairs * H * e)
    if k == "latent":
        H, r = case["heads"], case["q_rank"]
        params = r * W + H * 192 * r + 256 * W + 2 * H * 128 * 192 + W * H * 128
        pairs, past = _seen(case)
        return dict(bytes=2 * params + ends + 2 * 256 * (past + rows), flops=2 * rows * params + 2 * pairs * H * (192 + 128))
    I, E, top = case["inner"], case["experts"], case["top"]
    touched = E * (1.0 - (1.0 - top / E) ** rows)  # experts that some row is expected to choose
    return dict(bytes=touched * 3 * W * I * 2 + 4 * E * W + ends, flops=2 * rows * top * 3 * W * I)


def tolerance(case):
    """About four times what the path showed against ``exact`` on a B200."""
    if case["kind"] in ("decode", "prompt"):
        return dict(rel=0.03, max=0.3)  # 16 layers, each of which rounds to 8 bits
    if _dtype(case) == torch.float32:
        return dict(rel=1e-5, max=2e-4)
    return dict(rel=1.5e-2, max=0.15)


# ------------------------------------------------------------------------------------------------ the same sums in 64 bits
def _rms(x, w=None):
    y = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS)
    return y if w is None else y * w


def _silu(x):
    return x * torch.sigmoid(x)


def _inv_freq(dim, scaled):
    f = 1.0 / THETA ** (torch.arange(0, dim, 2, dtype=torch.float64, device=DEV) / dim)
    if scaled:
        s = SCALING
        wave = 2 * math.pi / f
        smooth = (s["original_max_position_embeddings"] / wave - s["low_freq_factor"]) / (s["high_freq_factor"] - s["low_freq_factor"])
        mid = (1 - smooth) * f / s["factor"] + smooth * f
        low = wave > s["original_max_position_embeddings"] / s["low_freq_factor"]
        high = wave < s["original_max_position_embeddings"] / s["high_freq_factor"]
        f = torch.where(low, f / s["factor"], torch.where(high, f, mid))
    return f


def _rope(x, pos, freq):
    """x [T, heads, D], halves paired; the angle is the float32 product, which is how the encoding is defined."""
    ang = (pos.float()[:, None] * freq.float()[None, :]).double()[:, None, :]
    a, b = x.chunk(2, -1)
    return torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()], -1)


def _attend(q, k, v, scale, first, window=0, softcap=0.0, sink=None):
    """q [T, H, D] at positions first .., k and v [S, G, D]: causal attention, a block of queries at a time."""
    T, H, _ = q.shape
    S, G, E = v.shape
    out = torch.empty((T, H, E), dtype=torch.float64, device=DEV)
    j = torch.arange(S, device=DEV)[None, :]
    step = max(1, (1 << 27) // max(1, H * S))
    for a in range(0, T, step):
        qq = q[a:a + step]
        n = qq.shape[0]
        s = torch.einsum("tgrd,sgd->grts", qq.view(n, G, H // G, -1), k) * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        i = torch.arange(first + a, first + a + n, device=DEV)[:, None]
        s = s.masked_fill((j > i) | (j <= i - (window or 1 << 40)), float("-inf"))
        top = s.amax(-1, keepdim=True)
        if sink is not None:
            top = torch.maximum(top, sink.view(G, H // G, 1, 1))
        p = torch.exp(s - top)
        den = p.sum(-1, keepdim=True) + (torch.exp(sink.view(G, H // G, 1, 1) - top) if sink is not None else 0.0)
        out[a:a + n] = torch.einsum("grts,sgd->tgrd", p / den, v).reshape(n, H, E)
    return out.reshape(T, H * E)


def _spans(case):
    at = 0
    for i, (n, c) in enumerate(_requests(case)):
        yield i, at, n, c
        at += n


def _llama_mixer(h, w, case, past):
    H, G, hd = case["heads"], case["kv_heads"], case["head_dim"]
    freq = _inv_freq(hd, False)
    out = torch.empty((h.shape[0], H * hd), dtype=torch.float64, device=DEV)
    for i, at, n, c in _spans(case):
        hh = h[at:at + n]
        pos = torch.arange(c, c + n, device=DEV)
        q = _rope((hh @ w["q"].T).view(n, H, hd), pos, freq)
        k = _rope((hh @ w["k"].T).view(n, G, hd), pos, freq)
        v = (hh @ w["v"].T).view(n, G, hd)
        if c:
            k = torch.cat([past[i][0].double().transpose(0, 1), k])
            v = torch.cat([past[i][1].double().transpose(0, 1), v])
        out[at:at + n] = _attend(q, k, v, hd ** -0.5, c)
    return out @ w["o"].T


def _linear_mixer(h, w, case, past):
    H, T = case["heads"], h.shape[0]
    q, v = (h @ w["q"].T).view(T, H, 128), (h @ w["v"].T).view(T, H, 128)
    k = (h @ w["k"].T).view(T, H, 128)
    if case["form"] == "decayed":
        q, k, v = _silu(q), _silu(k), _silu(v)
        f = torch.tensor(_decays(H), dtype=torch.float32).double().to(DEV)[None, :, None].expand(T, H, 128)
    elif case["form"] == "gated":
        f = (torch.sigmoid((h @ w["a1"].T) @ w["a2"].T + w["a2_bias"]) ** (1 / 16.0)).view(T, H, 128)
        q = q * 128 ** -0.5
    else:
        f = (w["lower"] + (1 - w["lower"]) * torch.sigmoid(k.reshape(T, -1) + w["f_bias"])).view(T, H, 128)
        q, k = _silu(q), 1 - f
    o = torch.empty_like(v)
    states = []
    for i, at, n, c in _spans(case):
        S = past[i].double() if c else torch.zeros((H, 128, 128), dtype=torch.float64, device=DEV)
        for t in range(at, at + n):
            S = f[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
            o[t] = torch.einsum("hde,hd->he", S, q[t])
        states.append(S.transpose(1, 2))
    if case["form"] == "decayed":
        o = _rms(o.reshape(T, -1), w["norm"]) * torch.sigmoid(h @ w["g"].T)
    elif case["form"] == "gated":
        o = _rms(o, w["norm"]).reshape(T, -1) * _silu(h @ w["g"].T)
    else:
        o = _rms(o, w["norm"]).reshape(T, -1)
    return o @ w["o"].T, torch.stack(states)


def _sink_mixer(h, w, case, past):
    H, G, e = case["heads"], case["kv_heads"], case["dim"]
    T = h.shape[0]
    q = _rms((h @ w["q"].T + w["qb"]).view(T, H, e))
    k = _rms((h @ w["k"].T + w["kb"]).view(T, G, e))
    v = (h @ w["v"].T + w["vb"]).view(T, G, e)
    out = torch.empty((T, H * e), dtype=torch.float64, device=DEV)
    for i, at, n, c in _spans(case):
        kk, vv = k[at:at + n], v[at:at + n]
        if c:
            rows = past[i].double().transpose(0, 1)
            kk, vv = torch.cat([rows[..., :e], kk]), torch.cat([rows[..., e:], vv])
        out[at:at + n] = _attend(q[at:at + n], kk, vv, e ** -0.5, c, case["window"], case["softcap"], w["sink"])
    return out @ w["o"].T


def _turn(x, pos):
    """x [T, heads, rot]: neighbouring channels turned in pairs."""
    i = torch.arange(LAT["rot"] // 2, dtype=torch.float64, device=DEV)
    ang = pos.double()[:, None, None] * (10000.0 ** (-2 * i / LAT["rot"]))
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()], -1).reshape(x.shape)


def _latent_mixer(h, w, case, past):
    H, T, R = case["heads"], h.shape[0], LAT["rank"]
    q = (_rms(h @ w["dq"].T, w["dq_norm"]) @ w["uq"].T).view(T, H, 192)
    down = h @ w["dkv"].T
    lat = _rms(down[:, :R], w["dkv_norm"])
    out = torch.empty((T, H * 128), dtype=torch.float64, device=DEV)
    for i, at, n, c in _spans(case):
        pos = torch.arange(c, c + n, device=DEV)
        rows = torch.cat([lat[at:at + n], _turn(down[at:at + n, None, R:], pos)[:, 0]], -1)
        if c:
            rows = torch.cat([past[i][0].double(), rows])
        S = rows.shape[0]
        k = torch.cat([(rows[:, :R] @ w["uk"].T).view(S, H, 128), rows[:, None, R:].expand(S, H, LAT["rot"])], -1)
        v = (rows[:, :R] @ w["uv"].T).view(S, H, 128)
        qq = torch.cat([q[at:at + n, :, :128], _turn(q[at:at + n, :, 128:], pos)], -1)
        out[at:at + n] = _attend(qq, k, v, 192 ** -0.5, c, case["window"])
    return out @ w["o"].T


def _experts(h, w, case):
    E, top = case["experts"], case["top"]
    vals, idx = torch.topk(h @ w["router"].T, top, -1)
    wts = torch.softmax(vals, -1)
    out = torch.zeros_like(h)
    for e in range(E):
        share = (wts * (idx == e)).sum(-1)
        at = share.nonzero()[:, 0]
        if at.numel():
            hh = h[at]
            y = (_silu(hh @ w[f"g{e}"].double().T) * (hh @ w[f"u{e}"].double().T)) @ w[f"d{e}"].double().T
            out[at] += share[at, None] * y
    return out


def _glu(h, w):
    return (_silu(h @ w["g"].T) * (h @ w["u"].T)) @ w["d"].T


def _exact_whole(case, seed):
    z = LLAMA_1B
    w, ids = _whole_inputs(case, seed)
    n, length = ids.shape
    if n * length > 20000:
        return None
    H, G, hd = z["heads"], z["kv_heads"], z["head_dim"]
    freq, pos = _inv_freq(hd, True), torch.arange(length, device=DEV)
    x = w["model.embed_tokens.weight"][ids].double()
    for i in range(z["layers"]):
        p = {k[len(f"model.layers.{i}."):-len(".weight")]: t.double() for k, t in w.items() if k.startswith(f"model.layers.{i}.")}
        for r in range(n):
            h = _rms(x[r], p["input_layernorm"])
            q = _rope((h @ p["self_attn.q_proj"].T).view(length, H, hd), pos, freq)
            k = _rope((h @ p["self_attn.k_proj"].T).view(length, G, hd), pos, freq)
            v = (h @ p["self_attn.v_proj"].T).view(length, G, hd)
            y = x[r] + _attend(q, k, v, hd ** -0.5, 0) @ p["self_attn.o_proj"].T
            h = _rms(y, p["post_attention_layernorm"])
            x[r] = y + (_silu(h @ p["mlp.gate_proj"].T) * (h @ p["mlp.up_proj"].T)) @ p["mlp.down_proj"].T
    h = _rms(x[:, -1], w["model.norm.weight"].double())
    out = torch.cat([h @ part.double().T for part in w["model.embed_tokens.weight"].split(16384)], -1)
    return dict(logits=out, **({"kv": None} if case["kind"] == "prompt" else {}))


def exact(case, seed):
    k = case["kind"]
    if k in ("decode", "prompt"):
        return _exact_whole(case, seed)
    w, x, h, past = _part_inputs(case, seed)
    x, h = x.double(), h.double()
    if k != "experts":
        w = {n: t.double() for n, t in w.items()}
    state = None
    if k == "block":
        y = x + _llama_mixer(_rms(x, w["n1"]), w, case, past)
        y = y + _glu(_rms(y, w["n2"]), w)
    elif k == "attention":
        y = x + _llama_mixer(h, w, case, past)
    elif k == "mlp":
        y = x + _glu(h, w)
    elif k == "linear":
        d, state = _linear_mixer(h, w, case, past)
        y = x + d
    elif k == "sink":
        y = x + _sink_mixer(h, w, case, past)
    elif k == "latent":
        y = x + _latent_mixer(h, w, case, past)
    else:
        y = x + _experts(h, {n: (t.double() if n == "router" else t) for n, t in w.items()}, case)
    out = dict(h=_rms(y, w["n3"].double()), x=y)
    if state is not None:
        out["state"] = state if case["form"] == "forget" else state.reshape(state.shape[0], -1)
    return out
