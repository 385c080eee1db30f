"""Workloads that stand for what a program has this engine do, each one pass through the public entry points.

Whole steps go through `ModelRunner.step()` (decode steps replayed from recordings, a prompt portion beside decoded tokens, the
true FP32 path) and return logits.  Single layers go through the parts that every architecture of the registry is put together
from (`parts.base.MIXERS`, `FEED_FORWARDS`, `NORMS`), on the layer sizes that bench.py runs for those architectures, and return the
layer's result and the state it leaves.  `exact` restates each of them with plain tensor operations in double precision.
"""
import math

import numpy as np
import torch

from quench6k_b200.config import FlintConfig
from quench6k_b200.engine import ModelRunner, StepEntry
from quench6k_b200.engine.batch import StepContext
from quench6k_b200.models.decoder import DecoderModel
from quench6k_b200.models.flint import build_spec
from quench6k_b200.parts.base import FEED_FORWARDS, MIXERS, NORMS, LayerCache, Replaced, Runtime, make_part
from quench6k_b200.spec import PartSpec

DEV = "cuda:0"
F64 = torch.float64
PAGE = 16
EPS = 1e-6


def listed():
    return [
        # one user's decode step: latency, launches, matrix-vector products
        {"name": "decode_one", "kind": "decode", "size": "m", "batch": 1, "context": 4096, "portion": 0, "portion_start": 0},
        # a decode step of a batch deep in long contexts: the cache's bytes
        {"name": "decode_batch_long", "kind": "decode", "size": "m", "batch": 8, "context": 32768, "portion": 0, "portion_start": 0},
        # continuous batching: a portion of a long prompt beside requests that are decoding, no size a multiple of a tile
        {"name": "portion_beside_decode", "kind": "decode", "size": "m", "batch": 21, "context": 1789, "portion": 1501, "portion_start": 4111},
        # the true FP32 path on a prompt: what a check against another implementation runs
        {"name": "fp32_prompt", "kind": "fp32", "tokens": 509},
        # routed experts and the norm after them: a prompt (every expert's weights), a decode batch (the chosen experts' weights)
        {"name": "experts_prompt", "kind": "experts", "tokens": 2048, "experts": 256, "top": 8, "ff": 512},
        {"name": "experts_decode", "kind": "experts", "tokens": 32, "experts": 256, "top": 8, "ff": 512},
        # one layer's mixer on a prompt of 2,048 tokens, or on portions of two or three prompts at once
        {"name": "latent_prompt", "kind": "latent", "size": "m", "requests": 1, "tokens": 2048, "start": 0},
        {"name": "mixed_heads_prompt", "kind": "mixed_heads", "size": "m", "requests": 1, "tokens": 2048, "start": 0},
        {"name": "difference_prompts", "kind": "difference", "size": "m", "requests": 2, "tokens": 1409, "start": 0},
        {"name": "scan_prompt", "kind": "scan", "size": "m", "requests": 1, "tokens": 2048, "start": 0},
        {"name": "delta_prompt", "kind": "delta", "size": "m", "requests": 1, "tokens": 2048, "start": 0},
        {"name": "retention_portions", "kind": "retention", "size": "m", "requests": 3, "tokens": 1021, "start": 777},
    ]


def _between(rng, lo, hi):
    """A whole number from lo to hi, even over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "portion", "fp32", "experts", "latent", "mixed_heads", "difference", "scan", "delta", "retention"])
    if kind in ("decode", "portion"):
        batch = _between(rng, 1, 48)
        case = {"kind": "decode", "size": rng.choice("sm"), "batch": batch, "context": _between(rng, 64, 262144 // max(8, batch)),
                "portion": 0, "portion_start": 0}
        if kind == "portion":
            case.update(portion=_between(rng, 65, 2048), portion_start=rng.choice([0, _between(rng, 16, 8192)]))
        return case
    if kind == "fp32":
        return {"kind": "fp32", "tokens": _between(rng, 17, 512)}
    if kind == "experts":
        experts, top, ff = rng.choice([(256, 8, 512), (64, 4, 1024), (32, 4, 512)])
        return {"kind": "experts", "tokens": _between(rng, 1, 2048), "experts": experts, "top": top, "ff": ff}
    requests = rng.choice([1, 1, 2, 3])
    return {"kind": kind, "size": rng.choice("sm"), "requests": requests, "tokens": _between(rng, 130, 2048 // requests),
            "start": rng.choice([0, _between(rng, 16, 4096)])}


# ----------------------------------------------------------------------------------------------- inputs and weights
def _generator(*key):
    """A generator whose stream depends on every number of `key`."""
    seed = 0
    for k in key:
        seed = (seed * 1000003 + int(k) + 12345) % (2 ** 62)
    return torch.Generator(device=DEV).manual_seed(seed)


def _normal(gen, shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
    return (torch.randn(shape, generator=gen, device=DEV, dtype=torch.float32) * std + mean).to(dtype)


def _int32(values):
    return torch.tensor(values, dtype=torch.int32).to(DEV)


def _flint(case):
    """The configuration of a whole model: dense feed-forwards in bfloat16, routed experts, windows and q/k norms in FP32."""
    if case["kind"] == "fp32":
        return FlintConfig.from_dict({
            "architectures": ["FlintForCausalLM"], "hidden_size": 1024, "num_hidden_layers": 4, "num_attention_heads": 8,
            "num_key_value_heads": 2, "head_dim": 128, "vocab_size": 32768, "n_routed_experts": 32, "num_experts_per_tok": 4,
            "moe_intermediate_size": 512, "rms_norm_eps": EPS, "rope_theta": 10000.0, "qk_norm": True, "first_k_dense_replace": 1,
            "intermediate_size": 4096, "sliding_window": 128, "sliding_window_pattern": [False, True, False, True], "kv_page_size": PAGE})
    width, ff, heads, kv = {"s": (1024, 4096, 8, 2), "m": (2048, 8192, 16, 4)}[case["size"]]
    return FlintConfig.from_dict({
        "architectures": ["FlintForCausalLM"], "hidden_size": width, "num_hidden_layers": 8, "num_attention_heads": heads,
        "num_key_value_heads": kv, "head_dim": 128, "vocab_size": 32768, "n_routed_experts": 8, "num_experts_per_tok": 2,
        "moe_intermediate_size": 64, "rms_norm_eps": EPS, "rope_theta": 10000.0, "first_k_dense_replace": 8, "intermediate_size": ff,
        "kv_page_size": PAGE})


def _flint_weights(cfg, seed, dtype):
    """{tensor name: tensor}: matrices N(0, 0.02), norms of ones."""
    gen, w, D, hd = _generator(seed, 1), {}, cfg.hidden_size, cfg.head_dim
    matrix = lambda *shape: _normal(gen, shape, 0.02, dtype=dtype)
    ones = lambda n: torch.ones(n, device=DEV)
    w["model.embed_tokens.weight"] = matrix(cfg.vocab_size, D)
    for i in range(cfg.num_hidden_layers):
        p = f"model.layers.{i}."
        w[p + "input_layernorm.weight"], w[p + "post_attention_layernorm.weight"] = ones(D), ones(D)
        for name, rows in (("q", cfg.num_attention_heads), ("k", cfg.num_key_value_heads), ("v", cfg.num_key_value_heads)):
            w[p + f"self_attn.{name}_proj.weight"] = matrix(rows * hd, D)
        w[p + "self_attn.o_proj.weight"] = matrix(D, cfg.num_attention_heads * hd)
        if cfg.qk_norm:
            w[p + "self_attn.q_norm.weight"], w[p + "self_attn.k_norm.weight"] = ones(hd), ones(hd)
        if cfg.layer_is_dense(i):
            F = cfg.intermediate_size
            w[p + "mlp.gate_proj.weight"], w[p + "mlp.up_proj.weight"], w[p + "mlp.down_proj.weight"] = matrix(F, D), matrix(F, D), matrix(D, F)
        else:
            E, F = cfg.n_routed_experts, cfg.moe_intermediate_size
            w[p + "mlp.gate.weight"] = matrix(E, D)
            for name, shape in (("gate", (E, F, D)), ("up", (E, F, D)), ("down", (E, D, F))):
                w[p + f"mlp.experts.{name}_proj.weight"] = matrix(*shape)
    w["model.norm.weight"], w["lm_head.weight"] = ones(D), matrix(cfg.vocab_size, D)
    return w


def _requests(case, seed):
    """[(positions cached before, token ids of this step)] of a whole step."""
    rng = np.random.default_rng([seed, 7])
    ids = lambda n: rng.integers(0, 32768, n).tolist()
    if case["kind"] == "fp32":
        return [(0, ids(case["tokens"]))]
    reqs = [(case["context"] - 3 * i if case["context"] > 200 else case["context"], ids(1)) for i in range(case["batch"])]
    return reqs + ([(case["portion_start"], ids(case["portion"]))] if case["portion"] else [])


def _cached(cfg, seed, layer, request, n):
    """Keys and values of a request's first n positions, [n, kv heads, head size] each, as earlier steps have left them."""
    gen, shape = _generator(seed, 2, layer, request), (n, cfg.num_key_value_heads, cfg.head_dim)
    return _normal(gen, shape, 0.9), _normal(gen, shape, 0.9)


def _into_pages(cache, pages, values, which):
    """values [n, heads, width] into the first n places of `pages`."""
    n, heads, width = values.shape
    blocks = -(-n // PAGE)
    padded = torch.zeros((blocks * PAGE, heads, width), dtype=values.dtype, device=DEV)
    padded[:n] = values
    which[:, torch.tensor(pages[:blocks], device=DEV)] = padded.view(blocks, PAGE, heads, width).permute(2, 0, 1, 3)


# Per mixer: its registered kind and parameters (the layer sizes of bench.py's designs), and its tensors with the mean and spread
# they are drawn with: ("name", shape, spread, mean), spread None for a constant.
def _mixer(case):
    D, H, G, rank, inner, chunk = {"s": (1024, 8, 2, 256, 2048, 512), "m": (2048, 16, 4, 512, 4096, 1024)}[case["size"]]
    hd, kind = 128, case["kind"]
    rope = lambda n: PartSpec("rope", {"head_dim": n, "theta": 10000.0, "rotary_dim": n})
    if kind == "latent":
        return D, "latent_attention", dict(num_heads=H, head_dim=hd, rot_dim=64, v_dim=hd, kv_rank=rank, scale=192 ** -0.5, eps=EPS, pos=rope(64)), [
            ("q_proj.weight", (H * 192, D), 0.02, 0), ("kv_down_proj.weight", (rank + 64, D), 0.02, 0), ("kv_norm.weight", (rank,), 0.1, 1),
            ("k_up_proj.weight", (H * hd, rank), 0.04, 0), ("v_up_proj.weight", (H * hd, rank), 0.04, 0), ("o_proj.weight", (D, H * hd), 0.02, 0)]
    if kind in ("mixed_heads", "difference"):
        diff = kind == "difference"
        hd = 64 if diff else 128
        maps = 2 if diff else 1
        p = dict(num_heads=H, num_kv_heads=G, head_dim=hd, v_dim=128, eps=EPS, pos=PartSpec("none", {"head_dim": hd}), qk_norm=True, scale=hd ** -0.5)
        t = [("q_proj.weight", (H * maps * hd, D), 0.02, 0), ("k_proj.weight", (G * maps * hd, D), 0.02, 0), ("v_proj.weight", (G * 128, D), 0.02, 0),
             ("o_proj.weight", (D, H * 128), 0.02, 0), ("q_norm.weight", (hd,), 0.1, 1), ("k_norm.weight", (hd,), 0.1, 1)]
        if not diff:
            return D, "attention", dict(p, chunk=chunk, talk=True), t + [("talk.weight", (H, H), 0.25, 0)]
        t += [(n + ".bias", (c,), 0.1, 0) for n, c in (("q_proj", H * 2 * hd), ("k_proj", G * 2 * hd), ("v_proj", G * 128), ("o_proj", D))]
        t += [(n, (hd,), 0.1, 0) for n in ("lambda_q1", "lambda_k1", "lambda_q2", "lambda_k2")]
        return D, "attention", dict(p, chunk=chunk, bias=True, o_bias=True, softcap=30.0, maps=2, diff=0.4), t
    if kind == "scan":
        R = D // 16
        return D, "selective_scan", dict(inner=inner, state=16, conv=4, dt_rank=R), [
            ("in_proj.weight", (2 * inner, D), 0.02, 0), ("conv1d.weight", (inner, 4), 0.4, 0), ("conv1d.bias", (inner,), 0.1, 0),
            ("x_proj.weight", (R + 32, inner), 0.02, 0), ("dt_proj.weight", (inner, R), R ** -0.5, 0), ("dt_proj.bias", (inner,), 1.0, -4.0),
            ("A_log", (inner, 16), 0.8, 1.7), ("D", (inner,), 0.1, 1), ("out_proj.weight", (D, inner), 0.02, 0)]
    if kind == "delta":
        return D, "gated_delta", dict(num_heads=H, num_kv_heads=G, head_dim=hd, v_dim=hd, conv=4, eps=EPS), [
            ("q_proj.weight", (G * hd, D), 0.02, 0), ("k_proj.weight", (G * hd, D), 0.02, 0), ("v_proj.weight", (H * hd, D), 0.02, 0),
            ("q_conv.weight", (G * hd, 4), 0.5, 0), ("k_conv.weight", (G * hd, 4), 0.5, 0), ("v_conv.weight", (H * hd, 4), 0.5, 0),
            ("b_proj.weight", (H, D), 0.02, 0), ("a_proj.weight", (H, D), 0.02, 0), ("g_proj.weight", (H * hd, D), 0.02, 0),
            ("A_log", (H,), 1.0, -2.5), ("dt_bias", (H,), 0.5, 0), ("norm.weight", (hd,), 0.1, 1), ("o_proj.weight", (D, H * hd), 0.02, 0)]
    assert kind == "retention"
    decay = [1.0 - 2.0 ** (-5.0 - 5.0 * h / H) for h in range(H)]
    return D, "retention", dict(num_heads=H, head_dim=hd, v_dim=hd, decay=decay, eps=EPS, pos=rope(hd)), [
        (n + "_proj.weight", (H * hd, D), 0.02, 0) for n in "qkvg"] + [("o_proj.weight", (D, H * hd), 0.02, 0)]


_MATRICES = ("_proj.weight",)


def _mixer_weights(case, seed):
    gen = _generator(seed, 3)
    return {name: _normal(gen, shape, std, mean, torch.bfloat16 if name.endswith(_MATRICES) else torch.float32)
            for name, shape, std, mean in _mixer(case)[3]}


def _lengths(case):
    """Tokens of each request of a layer's step: no two the same."""
    n, R = case["tokens"], case["requests"]
    return [max(1, n - i * (n // (2 * R) + 1)) for i in range(R)]


def _layer_rows(seed, T, D):
    """Normed rows as a layer's first norm hands them over."""
    return _normal(_generator(seed, 4), (T, D))


def _earlier_rows(seed, request, n, width, heads=1):
    """What earlier portions of a request have left in its pages, [n, heads, width]."""
    return _normal(_generator(seed, 5, request, width, heads), (n, heads, width))


def _earlier_state(case, seed, name, shape):
    """A recurrent state [requests, *shape]: zeros for a prompt's first portion, else what earlier portions left."""
    if not case["start"]:
        return torch.zeros((case["requests"], *shape), device=DEV)
    return _normal(_generator(seed, 6, sum(name.encode())), (case["requests"], *shape), 0.3, dtype=torch.float32)


# ----------------------------------------------------------------------------------------------- prepare and run
def _runtime(dtype=torch.bfloat16):
    return Runtime(torch.device(DEV), dtype)


def prepare(case, seed):
    kind = case["kind"]
    return (_prepare_step if kind in ("decode", "fp32") else _prepare_experts if kind == "experts" else _prepare_mixer)(case, seed)


def run(state):
    return state["run"](state)


def _prepare_step(case, seed):
    cfg, reqs = _flint(case), _requests(case, seed)
    dtype = torch.float32 if case["kind"] == "fp32" else torch.bfloat16
    model, weights = DecoderModel(build_spec(cfg)), _flint_weights(cfg, seed, dtype)
    model.bind(lambda name: weights[name], _runtime(dtype))
    pages = sum(-(-(n + max(len(t), GROWTH)) // PAGE) + 1 for n, t in reqs)
    runner = ModelRunner(model, model.rt, PAGE, pages, len(reqs))
    state = {"runner": runner, "reqs": reqs, "steps": 0, "run": _run_prompt if case["kind"] == "fp32" else _run_decode}
    if case["kind"] != "fp32":
        _stand_at_context(state)
        for layer, cache in enumerate(runner.caches):
            for r, (n, _) in enumerate(reqs):
                table, (k, v) = runner.manager.table(r, cache.group), _cached(cfg, seed, layer, r, n)
                if n:
                    _into_pages(cache, table, k, cache.k)
                    _into_pages(cache, table, v, cache.v)
    return state


GROWTH = 256          # decode steps before a request ends and one of the same length takes its place


def _stand_at_context(state):
    """Every request at its context length, pages taken as chunked prefills would: a portion of each in turn."""
    runner, reqs = state["runner"], state["reqs"]
    for r in range(len(reqs)):
        runner.add_request(r)
    for at in range(0, max(n for n, _ in reqs), 2048):
        for r, (n, _) in enumerate(reqs):
            if n > at:
                runner.assume_cached(r, min(2048, n - at))


def _run_decode(state):
    runner, reqs = state["runner"], state["reqs"]
    portion = len(reqs[-1][1]) > 1
    if state["steps"] == GROWTH or (portion and state["steps"]):
        # a request has its tokens (or its prompt is through): it ends and the next one comes
        again = range(len(reqs)) if state["steps"] == GROWTH else [len(reqs) - 1]
        for r in again:
            runner.end_request(r)
        for r in again:
            runner.add_request(r)
            if reqs[r][0]:
                runner.assume_cached(r, reqs[r][0])
        state["steps"] = 0 if len(again) == len(reqs) else state["steps"]
    state["steps"] += 1
    return runner.step([StepEntry(r, tokens, [len(tokens) - 1]) for r, (_, tokens) in enumerate(reqs)])


def _run_prompt(state):
    runner, (_, tokens) = state["runner"], state["reqs"][0]
    runner.add_request(0)
    logits = runner.step([StepEntry(0, tokens, range(max(0, len(tokens) - 16), len(tokens)))])
    runner.end_request(0)
    return logits


def _experts_weights(case, seed):
    gen, E, F, D = _generator(seed, 8), case["experts"], case["ff"], 2048
    shapes = {"gate.weight": (E, D), "experts.gate_proj.weight": (E, F, D), "experts.up_proj.weight": (E, F, D), "experts.down_proj.weight": (E, D, F)}
    return {name: _normal(gen, shape, 0.02) for name, shape in shapes.items()}


def _prepare_experts(case, seed):
    T, D, rt = case["tokens"], 2048, _runtime()
    ffn = make_part(FEED_FORWARDS, "feed-forward", PartSpec("moe", dict(num_experts=case["experts"], top_k=case["top"], intermediate_size=case["ff"])),
                    hidden_size=D)
    weights = _experts_weights(case, seed)
    ffn.bind(lambda name: weights[name], rt)
    norm = make_part(NORMS, "norm", PartSpec("rmsnorm", {"eps": EPS}), size=D)
    norm.bind(lambda name: torch.ones(D), rt)
    stream = _normal(_generator(seed, 9), (T, D), 0.5, dtype=torch.float32)
    lens = [T] if T > 64 else [1] * T
    return {"ffn": ffn, "norm": norm, "x": _layer_rows(seed, T, D), "stream": stream, "h": torch.empty_like(stream),
            "ctx": _context(lens, [0] * len(lens), []), "run": _run_experts}


def _run_experts(state):
    """The routed experts' results, left to the norm that opens the next layer: the stream and its normed rows."""
    h = state["h"]
    h.copy_(state["stream"])
    rows = state["ffn"].forward(state["x"], state["ctx"], h, defer=True)
    return {"normed": state["norm"].forward(h, add=rows), "stream": h}


def _context(lens, starts, tables):
    T, R = sum(lens), len(lens)
    positions = [s + i for s, n in zip(starts, lens) for i in range(n)]
    offsets = [sum(lens[:i]) for i in range(R + 1)]
    return StepContext(T=T, R=R, token_ids=_int32([0] * T), positions=_int32(positions), req_of_token=_int32([r for r, n in enumerate(lens) for _ in range(n)]),
                       q_start=_int32(offsets), pos_start=_int32(starts), slot_ids=_int32(list(range(R))), block_tables=tables,
                       logit_rows=_int32([]), n_logit_rows=0, q_lens=list(lens), pos_starts=list(starts), slots=list(range(R)),
                       max_context=max(s + n for s, n in zip(starts, lens)), max_q_len=max(lens))


def _prepare_mixer(case, seed):
    D, kind, params, _ = _mixer(case)
    rt, lens = _runtime(), _lengths(case)
    mixer = make_part(MIXERS, "mixer", PartSpec(kind, params), hidden_size=D)
    weights = _mixer_weights(case, seed)
    mixer.bind(lambda name: weights[name], rt)
    starts, R, cache, tables, begin, states = [case["start"]] * len(lens), len(lens), None, [], None, None
    request = mixer.cache_request()
    if request is not None:
        blocks = [-(-(s + n) // PAGE) for s, n in zip(starts, lens)]
        order = np.random.default_rng([seed, 10]).permutation(sum(blocks)).tolist()        # pages as a pool hands them out after a while
        table = [order[sum(blocks[:r]):sum(blocks[:r + 1])] for r in range(R)]
        tables = [_int32([t + [0] * (max(blocks) - len(t)) for t in table])]
        k = torch.zeros((request.kv_heads, sum(blocks), PAGE, request.head_dim), dtype=rt.dtype, device=DEV)
        v = (k[..., :request.v_dim] if request.values_in_keys else
             torch.zeros((request.v_heads or request.kv_heads, sum(blocks), PAGE, request.v_dim or request.head_dim), dtype=rt.dtype, device=DEV))
        cache = LayerCache(0, k, v, PAGE)
        for r in range(R):
            if case["start"]:
                _into_pages(cache, table[r], _earlier_rows(seed, r, case["start"], k.shape[3], k.shape[0]), k)
                if not request.values_in_keys:
                    _into_pages(cache, table[r], _earlier_rows(seed, r + 100, case["start"], v.shape[3], v.shape[0]), v)
    shapes = mixer.state_shape()
    if shapes is not None:
        begin = {name: _earlier_state(case, seed, name, shape) for name, (shape, _) in shapes.items()}
        states = {name: torch.empty_like(t) for name, t in begin.items()}
    x = _layer_rows(seed, sum(lens), D)
    return {"mixer": mixer, "x": x, "ctx": _context(lens, starts, tables), "cache": cache, "begin": begin, "states": states,
            "out": torch.empty((sum(lens), D), device=DEV), "run": _run_mixer}


def _run_mixer(state):
    """The layer's result, FP32, and the recurrent state it leaves (the request's slot as it was before the portion is put there first)."""
    ctx = state["ctx"]
    ctx.made.clear()
    for name, t in (state["begin"] or {}).items():
        state["states"][name].copy_(t)
    y = state["mixer"].forward(state["x"], ctx, state["cache"], state["states"], state["out"])
    if y.dim() == 3:                        # split-K partial sums: added as the block that takes them would
        Replaced(y).apply(state["out"])
        y = state["out"]
    return {"out": y, **{"state." + n: t for n, t in (state["states"] or {}).items()}}


# ----------------------------------------------------------------------------------------------- work and tolerance
def _pairs_seen(starts, lens, window=None, chunk=None):
    """Query-key pairs of one head under the mask."""
    total = 0
    for s, n in zip(starts, lens):
        p = np.arange(s, s + n, dtype=np.int64) + 1
        p = np.minimum(p, window) if window else (p - 1) % chunk + 1 if chunk else p
        total += int(p.sum())
    return total


def work(case):
    kind = case["kind"]
    if kind in ("decode", "fp32"):
        cfg, reqs = _flint(case), _requests(case, 0)
        size = 4 if kind == "fp32" else 2
        T, D, hd, Hq, Hkv, V = sum(len(t) for _, t in reqs), cfg.hidden_size, cfg.head_dim, cfg.num_attention_heads, cfg.num_key_value_heads, cfg.vocab_size
        wanted = 16 if kind == "fp32" else len(reqs)
        weights, products, pairs = V * D, wanted * V * D, 0
        for i in range(cfg.num_hidden_layers):
            att = (2 * Hq + 2 * Hkv) * hd * D
            if cfg.layer_is_dense(i):
                ffn_w = ffn_p = 3 * cfg.intermediate_size * D
            else:
                one = 3 * cfg.moe_intermediate_size * D
                ffn_w = cfg.n_routed_experts * (one * (1 - (1 - cfg.num_experts_per_tok / cfg.n_routed_experts) ** T) + D)
                ffn_p = cfg.num_experts_per_tok * one + cfg.n_routed_experts * D
            weights, products = weights + att + ffn_w, products + T * (att + ffn_p)
            pairs += _pairs_seen([n for n, _ in reqs], [len(t) for _, t in reqs], cfg.sliding_window if cfg.layer_is_sliding(i) else None)
        kv = cfg.num_hidden_layers * sum(n + 2 * len(t) for n, t in reqs) * 2 * Hkv * hd
        return {"bytes": (weights + kv) * size + wanted * V * 4, "flops": 2.0 * products + 4.0 * Hq * hd * pairs}
    if kind == "experts":
        T, E, k, F, D = case["tokens"], case["experts"], case["top"], case["ff"], 2048
        touched = E * (1 - (1 - k / E) ** T)
        return {"bytes": 2.0 * (touched * 3 * F * D + E * D) + T * D * (2 + 4 + 4 + 2), "flops": 2.0 * T * (k * 3 * F * D + E * D)}
    D, _, p, tensors = _mixer(case)
    lens, T = _lengths(case), sum(_lengths(case))
    starts = [case["start"]] * len(lens)
    matrices = sum(math.prod(s) for n, s, _, _ in tensors if n.endswith(_MATRICES))
    nbytes, flops = 2.0 * matrices + T * D * (2 + 4), 2.0 * T * matrices
    if kind == "latent":
        H, pairs = p["num_heads"], _pairs_seen(starts, lens)
        expanded = 2 * p["head_dim"] + p["rot_dim"]             # keys and values expanded from the latent: the fewest operations a pair takes
        flops += 2.0 * H * expanded * pairs + sum(starts) * 2.0 * H * 2 * p["head_dim"] * p["kv_rank"]
        nbytes += 2.0 * (T + sum(starts)) * (p["kv_rank"] + p["rot_dim"])
    elif kind in ("mixed_heads", "difference"):
        H, G, maps, pairs = p["num_heads"], p["num_kv_heads"], p.get("maps", 1), _pairs_seen(starts, lens, chunk=p["chunk"])
        flops += 2.0 * pairs * H * (maps * p["head_dim"] + 128) + (2.0 * pairs * H * H if kind == "mixed_heads" else 0)
        nbytes += 2.0 * (T + sum(s % p["chunk"] for s in starts)) * G * (maps * p["head_dim"] + 128)
    else:
        cells, passes = {"scan": lambda: (p["inner"] * p["state"], 3), "delta": lambda: (p["num_heads"] * 128 * 128, 3),
                         "retention": lambda: (p["num_heads"] * 128 * 128, 2)}[kind]()
        flops += 2.0 * passes * cells * T
        nbytes += 8.0 * cells * len(lens)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """bfloat16 operands: a rounding of 2^-9 at each of a few places; the recurrent state of a layer is FP32 on inputs of FP32."""
    return TOLERANCES[case["kind"]]


# about four times what one implementation is off the double-precision result, two of them apart from one another
TOLERANCES = {"decode": {"rel": 2e-2, "max": 0.15}, "fp32": {"rel": 1e-5, "max": 2e-4}, "experts": {"rel": 7e-3, "max": 0.1},
              "latent": {"rel": 1.2e-2, "max": 0.15}, "mixed_heads": {"rel": 1.1e-2, "max": 0.15}, "difference": {"rel": 1.2e-2, "max": 0.15},
              "scan": {"rel": 1e-2, "max": 0.15}, "delta": {"rel": 7e-3, "max": 0.1}, "retention": {"rel": 7e-3, "max": 0.1}}


# ----------------------------------------------------------------------------------------------- the same in double precision
def _rms(x, w=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)
    return y if w is None else y * w


def _silu(x):
    return x * torch.sigmoid(x)


def _rotated(x, positions, theta):
    """x [T, heads, n]: entry d turns with entry d + n/2 by the float32 product of position and inverse frequency."""
    half = x.shape[-1] // 2
    inv = (theta ** (-(2.0 * torch.arange(half, dtype=F64, device=DEV)) / (2 * half))).float()
    angle = (positions.float()[:, None] * inv).to(F64)[:, None]
    a, b, c, s = x[..., :half], x[..., half:], torch.cos(angle), torch.sin(angle)
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _seen(q_pos, k_pos, window=None, chunk=None):
    d = q_pos[:, None] - k_pos[None, :]
    ok = d >= 0
    if window:
        ok &= d < window
    if chunk:
        ok &= q_pos[:, None] // chunk == k_pos[None, :] // chunk
    return ok


def exact(case, seed):
    kind = case["kind"]
    if kind in ("decode", "fp32"):
        return _exact_step(case, seed)
    return _exact_experts(case, seed) if kind == "experts" else _exact_mixer(case, seed)


def _exact_experts_rows(x, router, gate, up, down, top):
    """Softmax over the router's logits, the `top` largest renormalised, their SwiGLU experts' weighted sum."""
    p, chosen = torch.softmax(x @ router.to(F64).T, -1).topk(top, -1)
    p = p / p.sum(-1, keepdim=True)
    y = torch.zeros_like(x)
    for e in torch.unique(chosen).tolist():
        row, slot = torch.nonzero(chosen == e, as_tuple=True)
        xe = x[row]
        y.index_add_(0, row, ((_silu(xe @ gate[e].to(F64).T) * (xe @ up[e].to(F64).T)) @ down[e].to(F64).T) * p[row, slot][:, None])
    return y


def _exact_experts(case, seed):
    w, T = _experts_weights(case, seed), case["tokens"]
    y = _exact_experts_rows(_layer_rows(seed, T, 2048).to(F64), w["gate.weight"], w["experts.gate_proj.weight"], w["experts.up_proj.weight"],
                            w["experts.down_proj.weight"], case["top"])
    h = _normal(_generator(seed, 9), (T, 2048), 0.5, dtype=torch.float32).to(F64) + y
    return {"normed": _rms(h), "stream": h}


def _exact_step(case, seed):
    cfg, reqs = _flint(case), _requests(case, seed)
    dtype = torch.float32 if case["kind"] == "fp32" else torch.bfloat16
    weights = _flint_weights(cfg, seed, dtype)
    Hq, Hkv, hd = cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim
    tokens = torch.tensor([t for _, ts in reqs for t in ts], device=DEV)
    at = np.cumsum([0] + [len(t) for _, t in reqs])
    positions = torch.cat([torch.arange(n, n + len(t), device=DEV) for n, t in reqs])
    x = weights["model.embed_tokens.weight"][tokens].to(F64)
    for i in range(cfg.num_hidden_layers):
        w = lambda name, i=i: weights[f"model.layers.{i}." + name].to(F64)
        xn, T = _rms(x), x.shape[0]
        q, k, v = ((xn @ w(f"self_attn.{n}_proj.weight").T).view(T, -1, hd) for n in "qkv")
        if cfg.qk_norm:
            q, k = _rms(q), _rms(k)
        q, k = _rotated(q, positions, cfg.rope_theta), _rotated(k, positions, cfg.rope_theta)
        a = torch.empty((T, Hq, hd), dtype=F64, device=DEV)
        for r, (n, ts) in enumerate(reqs):
            rows = slice(int(at[r]), int(at[r + 1]))
            kr, vr = k[rows], v[rows]
            if n:
                kc, vc = _cached(cfg, seed, i, r, n)
                kr, vr = torch.cat([kc.to(F64), kr]), torch.cat([vc.to(F64), vr])
            ok = _seen(positions[rows], torch.arange(n + len(ts), device=DEV), cfg.sliding_window if cfg.layer_is_sliding(i) else None)
            for h in range(Hq):
                s = (q[rows, h] @ kr[:, h * Hkv // Hq].T) * hd ** -0.5
                a[rows, h] = torch.softmax(s.masked_fill(~ok, -math.inf), -1) @ vr[:, h * Hkv // Hq]
        x = x + a.view(T, Hq * hd) @ w("self_attn.o_proj.weight").T
        xn = _rms(x)
        if cfg.layer_is_dense(i):
            x = x + (_silu(xn @ w("mlp.gate_proj.weight").T) * (xn @ w("mlp.up_proj.weight").T)) @ w("mlp.down_proj.weight").T
        else:
            p = f"model.layers.{i}.mlp."
            x = x + _exact_experts_rows(xn, weights[p + "gate.weight"], weights[p + "experts.gate_proj.weight"], weights[p + "experts.up_proj.weight"],
                                        weights[p + "experts.down_proj.weight"], cfg.num_experts_per_tok)
    rows = [int(a) - 1 for a in at[1:]] if case["kind"] != "fp32" else range(max(0, len(tokens) - 16), len(tokens))
    return _rms(x[list(rows)]) @ weights["lm_head.weight"].to(F64).T


def _exact_mixer(case, seed):
    D, _, p, _ = _mixer(case)
    lens, w = _lengths(case), {n: t.to(F64) for n, t in _mixer_weights(case, seed).items()}
    x, outs, states, at = _layer_rows(seed, sum(lens), D).to(F64), [], [], 0
    for r, n in enumerate(lens):
        y, left = _EXACT[case["kind"]](case, seed, r, p, w, x[at:at + n])
        outs.append(y)
        states.append(left)
        at += n
    return {"out": torch.cat(outs), **{"state." + name: torch.stack([s[name] for s in states]) for name in states[0]}}


def _exact_latent(case, seed, r, p, w, x):
    H, hd, rd, rank, n, start = p["num_heads"], p["head_dim"], p["rot_dim"], p["kv_rank"], x.shape[0], case["start"]
    pos = torch.arange(start, start + n, device=DEV)
    q = (x @ w["q_proj.weight"].T).view(n, H, hd + rd)
    qr = _rotated(q[..., hd:], pos, 10000.0)
    ckv = x @ w["kv_down_proj.weight"].T
    rows = torch.cat([_rms(ckv[:, :rank], w["kv_norm.weight"]), _rotated(ckv[:, None, rank:], pos, 10000.0)[:, 0]], -1)
    rows = torch.cat([_earlier_rows(seed, r, start, rank + rd)[:, 0].to(F64), rows])
    ok, a = _seen(pos, torch.arange(start + n, device=DEV)), torch.empty((n, H, hd), dtype=F64, device=DEV)
    for h in range(H):
        up = slice(h * hd, (h + 1) * hd)
        s = (q[:, h, :hd] @ (rows[:, :rank] @ w["k_up_proj.weight"][up].T).T + qr[:, h] @ rows[:, rank:].T) * p["scale"]
        a[:, h] = torch.softmax(s.masked_fill(~ok, -math.inf), -1) @ (rows[:, :rank] @ w["v_up_proj.weight"][up].T)
    return a.view(n, H * hd) @ w["o_proj.weight"].T, {}


def _exact_chunked(case, seed, r, p, w, x):
    """Attention inside chunks: heads mixed by a matrix, or two maps per head whose results are subtracted."""
    H, G, hd, M, n, start = p["num_heads"], p["num_kv_heads"], p["head_dim"], p.get("maps", 1), x.shape[0], case["start"]
    bias = lambda name: w[name + "_proj.bias"] if M > 1 else 0.0
    pos = torch.arange(start, start + n, device=DEV)
    q = _rms((x @ w["q_proj.weight"].T + bias("q")).view(n, H, M, hd), w["q_norm.weight"])
    k = _rms((x @ w["k_proj.weight"].T + bias("k")).view(n, G * M, hd), w["k_norm.weight"])
    v = (x @ w["v_proj.weight"].T + bias("v")).view(n, G, 128)
    if start:
        k = torch.cat([_earlier_rows(seed, r, start, hd, G * M).to(F64), k])
        v = torch.cat([_earlier_rows(seed, r + 100, start, 128, G).to(F64), v])
    ok = _seen(pos, torch.arange(start + n, device=DEV), chunk=p["chunk"])
    k, a = k.view(-1, G, M, hd), torch.zeros((n, H, 128), dtype=F64, device=DEV)

    def weights(h, m):
        s = (q[:, h, m] @ k[:, h * G // H, m].T) * p["scale"]
        s = p["softcap"] * torch.tanh(s / p["softcap"]) if "softcap" in p else s
        return torch.softmax(s.masked_fill(~ok, -math.inf), -1)

    if M == 1:
        for g in range(H):                  # head g's weights enter every head's mixture
            pg = weights(g, 0)
            for j in range(G):              # the heads whose values are value head j
                heads = range(j * H // G, (j + 1) * H // G)
                a[:, heads.start:heads.stop] += (pg @ v[:, j])[:, None] * w["talk.weight"][heads.start:heads.stop, g][None, :, None]
        return a.reshape(n, H * 128) @ w["o_proj.weight"].T, {}
    lam = torch.exp((w["lambda_q1"] * w["lambda_k1"]).sum()) - torch.exp((w["lambda_q2"] * w["lambda_k2"]).sum()) + p["diff"]
    for h in range(H):
        a[:, h] = _rms((weights(h, 0) - lam * weights(h, 1)) @ v[:, h * G // H]) * (1.0 - p["diff"])
    return a.reshape(n, H * 128) @ w["o_proj.weight"].T + w["o_proj.bias"], {}


def _convolved(u, tail, taps):
    """Causal convolution per channel after the `tail` (the inputs before the portion): the results and the tail it leaves."""
    k, full = taps.shape[1], torch.cat([tail, u])
    return sum(taps[:, j] * full[j:j + u.shape[0]] for j in range(k)), full[-(k - 1):]


def _exact_scan(case, seed, r, p, w, x):
    C, N, R = p["inner"], p["state"], p["dt_rank"]
    xz = x @ w["in_proj.weight"].T
    u, tail = _convolved(xz[:, :C], _earlier_state(case, seed, "conv", (3, C))[r].to(F64), w["conv1d.weight"])
    u = _silu(u + w["conv1d.bias"])
    proj = u @ w["x_proj.weight"].T
    dt = torch.nn.functional.softplus(proj[:, :R] @ w["dt_proj.weight"].T + w["dt_proj.bias"])
    A, S, y = -torch.exp(w["A_log"]), _earlier_state(case, seed, "ssm", (C, N))[r].to(F64), torch.empty_like(u)
    for t in range(x.shape[0]):
        S = torch.exp(dt[t][:, None] * A) * S + (dt[t] * u[t])[:, None] * proj[t, R:R + N][None, :]
        y[t] = S @ proj[t, R + N:]
    y = (y + w["D"] * u) * _silu(xz[:, C:])
    return y @ w["out_proj.weight"].T, {"ssm": S, "conv": tail}


def _exact_delta(case, seed, r, p, w, x):
    H, G, d, n = p["num_heads"], p["num_kv_heads"], p["head_dim"], x.shape[0]
    raw = torch.cat([x @ w[f"{c}_proj.weight"].T for c in "qkv"], -1)
    u, tail = _convolved(raw, _earlier_state(case, seed, "conv", (3, raw.shape[1]))[r].to(F64), torch.cat([w[f"{c}_conv.weight"] for c in "qkv"]))
    q, k, v = _silu(u).split([G * d, G * d, H * d], -1)
    unit = lambda z: z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6)
    q, k = (unit(z.view(n, G, d)).repeat_interleave(H // G, 1) for z in (q, k))
    q, v, beta = q * d ** -0.5, v.view(n, H, d), torch.sigmoid(x @ w["b_proj.weight"].T)
    decay = torch.exp(-torch.exp(w["A_log"]) * torch.nn.functional.softplus(x @ w["a_proj.weight"].T + w["dt_bias"]))
    S, o = _earlier_state(case, seed, "S", (H, d, d))[r].to(F64), torch.empty_like(v)              # kept as [head, value, key]
    for t in range(n):
        S = decay[t][:, None, None] * S
        S = S + (beta[t][:, None] * (v[t] - torch.einsum("hvk,hk->hv", S, k[t])))[:, :, None] * k[t][:, None, :]
        o[t] = torch.einsum("hvk,hk->hv", S, q[t])
    y = _rms(o, w["norm.weight"]).view(n, H * d) * _silu(x @ w["g_proj.weight"].T)
    return y @ w["o_proj.weight"].T, {"S": S, "conv": tail}


def _exact_retention(case, seed, r, p, w, x):
    H, d, n = p["num_heads"], p["head_dim"], x.shape[0]
    pos = torch.arange(case["start"], case["start"] + n, device=DEV)
    q, k, v = ((x @ w[f"{c}_proj.weight"].T).view(n, H, d) for c in "qkv")
    q, k = _rotated(q, pos, 10000.0), _rotated(k, pos, 10000.0) * d ** -0.5
    decay = torch.tensor(p["decay"], dtype=torch.float32).to(DEV, F64)[:, None, None]
    S, o = _earlier_state(case, seed, "S", (H, d, d))[r].to(F64), torch.empty_like(v)              # kept as [head, key, value]
    for t in range(n):
        S = decay * S + k[t][:, :, None] * v[t][:, None, :]
        o[t] = torch.einsum("hkv,hk->hv", S, q[t])
    y = _rms(o).view(n, H * d) * _silu(x @ w["g_proj.weight"].T)
    return y @ w["o_proj.weight"].T, {"S": S}


_EXACT = {"latent": _exact_latent, "mixed_heads": _exact_chunked, "difference": _exact_chunked, "scan": _exact_scan, "delta": _exact_delta,
          "retention": _exact_retention}
