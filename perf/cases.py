"""The work this framework is used for, as cases that can be timed and compared.

A case is one call of a layer's part (an attention, a feed-forward, a recurrence) on the token rows of one step, or one
decode step of a whole small model.  Sizes are those of the layers in ``bench.py``: the Qwen3 family from 0.6B to 32B, and
the "2k" and "4k" layer sizes of the other designs.  ``listed`` gives the cases by name, ``draw`` more of the same ranges.

Fields of a case
    part      "attention" (grouped-query, q/k norm, rotation, paged cache, output projection), "mlp" (norm and gated
              feed-forward), "experts" (router, routed and shared experts), "mlstm" (matrix memory), "latent" (attention
              over a cache of one vector a token), "model" (a whole Qwen3 decode step)
    dtype     "bf16", or "f32" for the engine's true 32-bit mode
    size      a key of SIZES
    prompts, new, behind      requests that bring ``new`` tokens each, behind ``behind`` cached ones
    singles, least, most      requests that bring one token each, behind ``least`` to ``most`` cached ones
"""
import math

import numpy as np
import torch

import tffinfer_b200 as tff
from tffinfer_b200.cache import GroupSpec, make_cache_manager
from tffinfer_b200.config import Qwen3Config
from tffinfer_b200.engine.batch import packed_to_device
from tffinfer_b200.parts import LayerContext, PartSpec, build_part
from tffinfer_b200.weights import random_tensors_on_device

DEV = "cuda"
PAGE = 16
EPS = 1e-6
THETA = 1e6
# width, query heads, feed-forward of the Qwen3 family: 8 key/value heads of 128 everywhere
QWEN = {"0.6B": (1024, 16, 3072), "1.7B": (2048, 16, 6144), "4B": (2560, 32, 9728), "8B": (4096, 32, 12288),
        "14B": (5120, 40, 17408), "32B": (5120, 64, 25600)}
KV_HEADS, HEAD = 8, 128
# width, experts' feed-forward, experts, chosen, (groups, kept), shared feed-forward
EXPERTS = {"2k": (2048, 3072, 16, 2, (4, 2), 3072), "4k": (4096, 6144, 16, 2, (4, 2), 6144)}
# width, heads, key and value size
MLSTM = {"2k": (2048, 16, 128, 128), "4k": (4096, 32, 128, 128)}
# width, heads, unrotated and rotated key size, value size, query rank, latent rank
LATENT = {"2k": (2048, 16, 128, 64, 128, 768, 512), "4k": (4096, 32, 128, 64, 128, 1536, 512)}
# width, heads, key/value heads, feed-forward, layers, vocabulary of the whole models
MODEL = {"2k": (2048, 16, 4, 6144, 8, 32768), "4k": (4096, 32, 8, 12288, 8, 32768)}
SIZES = {"attention": QWEN, "mlp": QWEN, "experts": EXPERTS, "mlstm": MLSTM, "latent": LATENT, "model": MODEL}


def _case(part, dtype, size, name=None, prompts=0, new=0, behind=0, singles=0, least=0, most=0):
    c = dict(part=part, dtype=dtype, size=size, prompts=prompts, new=new, behind=behind, singles=singles, least=least, most=most)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # decoding for many users at once: a layer's attention streams 64 caches (bench.py, batch 64 behind 2,048 tokens)
        _case("attention", "bf16", "8B", "attention_decode_64", singles=64, least=2048, most=2304),
        # one long document read in: a layer's attention over a whole prompt of 8,192 tokens (bench.py sweep)
        _case("attention", "bf16", "8B", "attention_prompt_8192", prompts=1, new=8192),
        # a served mix: a portion of a prompt beside requests that decode (bench.py mixed14b), ragged everywhere
        _case("attention", "bf16", "14B", "attention_mixed_14b", prompts=1, new=484, behind=1501, singles=28, least=200, most=4200),
        # the headline decode step's largest product pair: 8 rows (bench.py, batch 8)
        _case("mlp", "bf16", "8B", "mlp_decode_8", singles=8),
        # a step's token budget of the mixed workload: portion and decoded tokens, 540 rows
        _case("mlp", "bf16", "14B", "mlp_step_540", prompts=1, new=540),
        # the 32-bit mode: feed-forward of four requests that decode (bench.py fp32_short)
        _case("mlp", "f32", "8B", "mlp_f32_decode_4", singles=4),
        # the 32-bit mode: four short prompts
        _case("attention", "f32", "8B", "attention_f32_prompts", prompts=4, new=134),
        # routed experts with a shared one: 64 requests that decode touch every expert
        _case("experts", "bf16", "2k", "experts_decode_64", singles=64),
        # the same on a prompt of 2,048 tokens
        _case("experts", "bf16", "2k", "experts_prompt_2048", prompts=1, new=2048),
        # a matrix memory over a prompt of 2,048 tokens
        _case("mlstm", "bf16", "2k", "mlstm_prompt_2048", prompts=1, new=2048),
        # latent attention, 32 requests that decode behind about 4,000 tokens
        _case("latent", "bf16", "2k", "latent_decode_32", singles=32, least=3000, most=5000),
        # one user's decode step of a small whole model, launches and latency
        _case("model", "bf16", "2k", "model_decode_1", singles=1, least=500, most=600),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _drawn(rng):
    part = rng.choice(["attention", "attention", "attention", "mlp", "mlp", "f32", "f32", "experts", "mlstm", "latent", "model"])
    if part == "f32":                                   # the 32-bit mode: short prompts and few requests
        size = rng.choice(["0.6B", "1.7B", "4B", "8B"])
        if rng.random() < 0.5:
            if rng.random() < 0.5:
                return _case("mlp", "f32", size, singles=_log(rng, 1, 16))
            return _case("mlp", "f32", size, prompts=1, new=_log(rng, 17, 512))
        if rng.random() < 0.5:
            least = _log(rng, 64, 1024)
            return _case("attention", "f32", size, singles=_log(rng, 1, 8), least=least, most=least + rng.randrange(256))
        return _case("attention", "f32", size, prompts=rng.randint(1, 4), new=_log(rng, 16, 256))
    if part == "attention":
        size = rng.choice(sorted(QWEN))
        kind = rng.choice(["decode", "prompt", "mixed"])
        if kind == "decode":
            least = _log(rng, 256, 8192)
            return _case(part, "bf16", size, singles=_log(rng, 8, 128), least=least, most=int(least * rng.uniform(1, 2)))
        if kind == "prompt":
            return _case(part, "bf16", size, prompts=rng.choice([1, 1, 2]), new=_log(rng, 256, 8192),
                         behind=rng.choice([0, 0, rng.randrange(4096)]))
        return _case(part, "bf16", size, prompts=1, new=_log(rng, 64, 512), behind=rng.randrange(4096),
                     singles=_log(rng, 4, 48), least=_log(rng, 100, 1000), most=_log(rng, 1000, 6000))
    if part == "mlp":
        size = rng.choice(sorted(QWEN))
        if rng.random() < 0.5:
            return _case(part, "bf16", size, singles=_log(rng, 1, 64))
        return _case(part, "bf16", size, prompts=1, new=_log(rng, 65, 2048))
    if part == "latent":
        size = rng.choice(["2k", "4k"])
        if rng.random() < 0.6:
            least = _log(rng, 256, 8192)
            return _case(part, "bf16", size, singles=_log(rng, 4, 64), least=least, most=int(least * rng.uniform(1, 2)))
        return _case(part, "bf16", size, prompts=rng.choice([1, 2]), new=_log(rng, 128, 4096))
    if part == "model":
        least = _log(rng, 64, 1800)
        return _case(part, "bf16", rng.choice(["2k", "4k"]), singles=_log(rng, 1, 8), least=least, most=least + rng.randrange(200))
    size = rng.choice(["2k", "4k"])                      # experts, mlstm
    if rng.random() < 0.5:
        return _case(part, "bf16", size, singles=_log(rng, 8, 128), least=100, most=_log(rng, 200, 4000))
    return _case(part, "bf16", size, prompts=rng.choice([1, 1, 3]), new=_log(rng, 100, 2048))


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / (2.5 if case["dtype"] == "f32" else 50.0))


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        c = _drawn(rng)
        if _cost(c) <= most:
            return c


# ------------------------------------------------------------------------------------------------- what a case consists of
def _spread(case):
    """Cached tokens of the requests that decode: spread evenly between least and most, in an order of no pattern."""
    n = case["singles"]
    if n == 0:
        return []
    span = case["most"] - case["least"]
    return [case["least"] + (span * ((i * 7 + 3) % n)) // max(1, n - 1) if n > 1 else case["least"] for i in range(n)]


def _requests(case):
    """[(cached tokens, new tokens)] of the step's requests: those that decode first."""
    return [(p, 1) for p in _spread(case)] + [(case["behind"], case["new"])] * case["prompts"]


def _rows(case):
    return sum(n for _, n in _requests(case))


def _act(case):
    return torch.float32 if case["dtype"] == "f32" else torch.bfloat16


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _spec(case):
    """(registry family, PartSpec) of the case's part."""
    part, size = case["part"], case["size"]
    if part == "attention":
        W, H, _ = QWEN[size]
        return "mixer", PartSpec("gqa_attention", dict(hidden_size=W, num_heads=H, num_kv_heads=KV_HEADS, head_dim=HEAD,
                                                       qk_norm=True, qk_norm_eps=EPS))
    if part == "mlp":
        W, _, F = QWEN[size]
        return "feed_forward", PartSpec("swiglu", dict(hidden_size=W, intermediate_size=F))
    if part == "experts":
        W, F, E, top, groups, shared = EXPERTS[size]
        return "feed_forward", PartSpec("routed_experts", dict(
            hidden_size=W, intermediate_size=F, num_experts=E, top=top, renormalize=True, router_score="softmax",
            correction=True, groups=groups, shared_intermediate=shared, shared_gate=True))
    if part == "mlstm":
        W, H, K, V = MLSTM[size]
        return "mixer", PartSpec("mlstm", dict(hidden_size=W, num_heads=H, head_dim=K, v_head_dim=V, gate_cap=15.0, eps=EPS))
    W, H, D, R, V, QR, KR = LATENT[size]
    return "mixer", PartSpec("latent_attention", dict(hidden_size=W, num_heads=H, head_dim=D, rot_dim=R, v_head_dim=V,
                                                      q_rank=QR, kv_rank=KR, eps=EPS))


def _weights(part, case, gen):
    """Tensors by name, as a file of the engine's dtype would hold them: matrices N(0, 0.02) unless the part says otherwise."""
    out = {}
    for name, spec in part.weight_specs().items():
        if spec.optional:
            continue
        std = spec.init_scale if spec.init_scale is not None else (0.1 if spec.init == "one_plus_normal" else 0.02)
        t = torch.randn(spec.shape, generator=gen, device=DEV) * std
        if spec.init == "one_plus_normal":
            t += 1.0
        out[name] = t if spec.role == "vector" else t.to(_act(case))
    return out


def _inputs(case, seed):
    """What both ``prepare`` and ``exact`` start from: the part's weights, its input rows, the residual and the cache."""
    gen = _generator(seed)
    family, spec = _spec(case)
    part = build_part(family, spec)
    weights = _weights(part, case, gen)
    T, W = _rows(case), part.hidden_size
    rows = torch.randn((T, W), generator=gen, device=DEV)
    d = dict(part=part, weights=weights, x=rows, h=rows.to(_act(case)))
    if case["part"] != "mlp":
        d["x"] = torch.randn((T, W), generator=gen, device=DEV) * 0.01
    else:
        d["norm_w"] = 1.0 + 0.1 * torch.randn((W,), generator=gen, device=DEV)
    return d, gen


def _cache_plan(case, part):
    """A cache manager that holds the step's requests with their cached tokens, pages handed out in turns."""
    need = part.cache_need() if hasattr(part, "cache_need") else None
    paged = need is not None and hasattr(need, "num_kv_heads")
    reqs = _requests(case)
    pages = sum(-(-(p + n) // PAGE) for p, n in reqs) if paged else 1
    groups = [GroupSpec(1, need.num_kv_heads, need.head_dim, need.window, need.planes)] if paged else []
    cache = make_cache_manager(groups, PAGE, [pages] if paged else [], len(reqs))
    left = [p for p, _ in reqs]
    for i in range(len(reqs)):
        cache.admit(i)
    while any(left):
        for i, n in enumerate(left):
            if n:
                cache.reserve(i, min(n, 256))
                cache.commit(i, min(n, 256))
                left[i] = n - min(n, 256)
    entries = [tff.StepEntry(i, [1] * n, (n - 1,)) for i, (_, n) in enumerate(reqs)]
    arrays = cache.gather_step(entries)
    status, detail = cache.reserve_step(arrays)
    if status != 1:
        raise RuntimeError(f"the step does not fit its cache: {status} {detail}")
    return cache, entries, arrays, (need, pages) if paged else None


def _cache_tensor(need, pages, case, gen):
    """Cached keys and values of unit size (queries and keys are normed), layers outermost as the engine stores them."""
    return torch.randn((1, pages, need.planes, need.num_kv_heads, PAGE, need.head_dim), generator=gen, device=DEV,
                       dtype=torch.float32 if case["dtype"] == "f32" else torch.bfloat16).permute(1, 0, 2, 3, 4, 5)


_kernels = None


def _ops():
    """The kernel library, loaded once as a program does."""
    global _kernels
    if _kernels is None:
        from tffinfer_b200.kernels.library import CudaKernels
        _kernels = CudaKernels()
    return _kernels


def prepare(case, seed):
    if case["part"] == "model":
        return _prepare_model(case, seed)
    ops, act = _ops(), _act(case)
    d, gen = _inputs(case, seed)
    part = d["part"]
    part.load(dict(d["weights"]), ops, act)
    cache, entries, arrays, paged = _cache_plan(case, part)
    batch = packed_to_device(*cache.pack_step(entries, arrays=arrays), DEV, pinned=True)
    ctx = LayerContext(batch=batch, ops=ops, page_size=PAGE, shared={})
    if paged is not None:
        ctx.kv_cache, ctx.block_table = _cache_tensor(*paged, case, gen), batch.block_tables[0]
    if case["part"] in ("attention", "latent"):
        ctx.position = _position(case)
        ctx.position.prepare(ops, DEV, max(p + n for p, n in _requests(case)) + 1)
    if case["part"] == "mlstm":
        ctx.state = torch.zeros((len(entries), *part.cache_need().shape), device=DEV)
        _fill_memory(ctx.state, case, gen)
    s = dict(part=part, ctx=ctx, x=d["x"], h=d["h"], case=case, norm=None)
    if case["part"] == "mlp":
        s["norm"] = build_part("norm", PartSpec("rms_norm", dict(dim=part.hidden_size, eps=EPS)))
        s["norm"].load({"weight": d["norm_w"]}, ops, act)
    return s


def _position(case):
    if case["part"] == "attention":
        return build_part("position", PartSpec("rotary", dict(head_dim=HEAD, theta=THETA)))
    return build_part("position", PartSpec("scaled_rotary", dict(rotary_dim=LATENT[case["size"]][3], theta=5e5,
                                                                 pairing="interleaved")))


def _fill_memory(state, case, gen):
    """Memories in mid-sequence for requests that decode: S, n and m (prompts start theirs from zeros)."""
    _, H, K, V = MLSTM[case["size"]]
    if case["singles"]:
        n = case["singles"]
        state[:n, :H * K * V] = torch.randn((n, H * K * V), generator=gen, device=DEV)
        state[:n, H * K * V:H * K * V + H * K] = torch.randn((n, H * K), generator=gen, device=DEV)
        state[:n, H * K * V + H * K:H * K * V + H * K + H] = 1.0


def run(s):
    if "runner" in s:
        runner = s["runner"]
        return runner.run_batch(runner.make_batch(s["entries"]))
    ctx, x, part = s["ctx"], s["x"], s["part"]
    ctx.shared = {}
    if s["norm"] is not None:                            # as a layer does: the norm folded into the product where that is faster
        act = _act(s["case"])
        h = s["norm"].deferred(x, ctx.ops, act)
        if h is None:
            h = s["norm"].forward(x, ctx.ops, act)
        return part.forward(h, ctx, residual=x)
    y = part.forward(s["h"], ctx, residual=x)
    return (y, ctx.state) if ctx.state is not None else y


# ------------------------------------------------------------------------------------------------------ a whole model
def _model_config(case):
    W, H, G, F, L, V = MODEL[case["size"]]
    return Qwen3Config(architecture="Qwen3ForCausalLM", hidden_size=W, num_layers=L, num_heads=H, num_kv_heads=G,
                       head_dim=HEAD, intermediate_size=F, vocab_size=V, rms_norm_eps=EPS, rope_theta=THETA,
                       max_position=4096, tie_word_embeddings=False, layer_types=("full_attention",) * L).validate()


def _model_tokens(case, seed):
    rng = np.random.default_rng(int(seed))
    return [rng.integers(0, MODEL[case["size"]][5], p + 1).tolist() for p in _spread(case)]


def _prepare_model(case, seed):
    """The engine's runner with its prompts read in; the first step of a size captures its launches, as a server's does."""
    tensors = random_tensors_on_device(_model_config(case), int(seed), DEV, "bfloat16", norm_noise=0.1)
    tokens = _model_tokens(case, seed)
    cap = sum(-(-(len(t) + 1) // PAGE) * PAGE for t in tokens)
    runner = tff.ModelRunner(config=_model_config(case), tensors=tensors, ops=_ops(), engine_config=tff.EngineConfig(
        dtype="bfloat16", page_size=PAGE, max_cache_tokens=cap, max_live_requests=max(8, len(tokens)), max_model_len=4096))
    for i, t in enumerate(tokens):
        runner.add_request(i)
        if len(t) > 1:
            runner.step([tff.StepEntry(i, t[:-1])])
    entries = [tff.StepEntry(i, [t[-1]], (0,)) for i, t in enumerate(tokens)]
    runner.run_batch(runner.make_batch(entries))
    return dict(runner=runner, entries=entries)


# -------------------------------------------------------------------------------------------------- work and tolerance
def work(case):
    part, T, reqs = case["part"], _rows(case), _requests(case)
    e = 4 if case["dtype"] == "f32" else 2
    pairs = sum(n * p + n * (n + 1) // 2 for p, n in reqs)         # (query, key) pairs
    cached, fresh = sum(p for p, _ in reqs), T
    if part == "attention":
        W, H, _ = QWEN[case["size"]]
        w = (2 * H + 2 * KV_HEADS) * HEAD * W
        kv = 2 * KV_HEADS * HEAD * e
        return {"bytes": w * e + (cached + fresh) * kv + T * W * (e + 8), "flops": 2.0 * T * w + 4.0 * pairs * H * HEAD}
    if part == "mlp":
        W, _, F = QWEN[case["size"]]
        return {"bytes": 3 * W * F * e + T * W * 8, "flops": 6.0 * T * W * F}
    if part == "experts":
        W, F, E, top, _, shared = EXPERTS[case["size"]]
        touched = E * (1.0 - (1.0 - top / E) ** T)
        return {"bytes": 3 * W * (touched * F + shared) * e + E * W * e + T * W * (e + 8),
                "flops": 6.0 * T * W * (top * F + shared) + 2.0 * T * W * E}
    if part == "mlstm":
        W, H, K, V = MLSTM[case["size"]]
        w = (2 * H * K + 2 * H * V + 2 * H) * W + H * V * W
        state = 4 * (H * K * V + H * K + H)
        return {"bytes": w * e + (2 * case["singles"] + case["prompts"]) * state + T * W * (e + 8),
                "flops": 2.0 * T * w + 4.0 * T * H * K * V}
    if part == "latent":
        W, H, D, R, V, QR, KR = LATENT[case["size"]]
        w = (QR + KR + R) * W + H * (D + R) * QR + H * (D + V) * KR + H * V * W
        return {"bytes": w * e + (cached + fresh) * (KR + R) * e + T * W * (e + 8),
                "flops": 2.0 * T * w + 2.0 * pairs * H * (D + R + V)}
    W, H, G, F, L, V = MODEL[case["size"]]
    w = L * ((2 * H + 2 * G) * HEAD * W + 3 * W * F) + V * W
    return {"bytes": w * e + L * (cached + fresh) * 2 * G * HEAD * e + T * V * 4,
            "flops": 2.0 * T * w + 4.0 * L * pairs * H * HEAD}


def tolerance(case):
    """About four times what the path is off 64-bit arithmetic, or what two runs of it differ by where that is more: 2.4e-6 in
    32 bits; in bfloat16 6e-3 for a memory over a prompt and for the logits of eight layers, 3e-3 for the other parts."""
    if case["dtype"] == "f32":
        return {"rel": 1e-5}
    return {"rel": {"model": 4e-2, "mlstm": 2e-2}.get(case["part"], 1.2e-2)}


# ------------------------------------------------------------------------------------------- the same in 64-bit arithmetic
def _rms(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * w


def _rotate(x, positions, theta, interleaved=False):
    """x [T, heads, d] turned by its position, pairs (i, i + d/2), or (2i, 2i + 1) when interleaved."""
    d = x.shape[-1]
    freq = theta ** (-2.0 * torch.arange(d // 2, device=x.device, dtype=torch.float64) / d)
    a = positions.double()[:, None] * freq
    c, s = a.cos()[:, None], a.sin()[:, None]
    if interleaved:
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * c - v * s, u * s + v * c], dim=-1).flatten(-2)
    u, v = x[..., :d // 2], x[..., d // 2:]
    return torch.cat([u * c - v * s, u * s + v * c], dim=-1)


def _softmax_attend(q, k, v, first, scale):
    """q [n, d] at positions first .. behind keys k [m, d], values v [m, e]."""
    out = torch.empty((q.shape[0], v.shape[1]), dtype=torch.float64, device=q.device)
    at = torch.arange(k.shape[0], device=q.device)
    for i in range(0, q.shape[0], 2048):
        s = (q[i:i + 2048] @ k.T) * scale
        mine = first + i + torch.arange(s.shape[0], device=q.device)
        s.masked_fill_(at[None] > mine[:, None], float("-inf"))
        out[i:i + 2048] = torch.softmax(s, dim=-1) @ v
    return out


def _gathered(cache, pages, first, kv_cache):
    """Cached rows 0 .. first of a request: [planes, kv heads, first, head] in float64."""
    n = -(-first // PAGE)
    got = kv_cache[torch.tensor(pages[:n], device=DEV, dtype=torch.long), 0].double()      # [n, planes, kv heads, page, head]
    return got.permute(1, 2, 0, 3, 4).flatten(2, 3)[:, :, :first]


def exact(case, seed):
    if case["part"] == "model":
        return _exact_model(case, seed)
    d, gen = _inputs(case, seed)
    w = {k: v.double() for k, v in d["weights"].items()}
    h, x = d["h"].double(), d["x"].double()
    if case["part"] == "mlp":
        h = _rms(x, d["norm_w"].double())
        g = h @ w["gate_proj.weight"].T
        return x + (g * torch.sigmoid(g) * (h @ w["up_proj.weight"].T)) @ w["down_proj.weight"].T
    if case["part"] == "experts":
        return x + _exact_experts(case, w, h)
    if case["part"] == "mlstm":
        return _exact_mlstm(case, w, h, x, gen)
    cache, entries, _, paged = _cache_plan(case, d["part"])
    kv_cache = _cache_tensor(*paged, case, gen)
    positions = torch.cat([torch.arange(p, p + n, device=DEV) for p, n in _requests(case)])
    mixed, row = [], 0
    if case["part"] == "attention":
        T, H = h.shape[0], QWEN[case["size"]][1]
        q = _rotate(_rms((h @ w["q_proj.weight"].T).view(T, H, HEAD), w["q_norm.weight"]), positions, THETA)
        k = _rotate(_rms((h @ w["k_proj.weight"].T).view(T, KV_HEADS, HEAD), w["k_norm.weight"]), positions, THETA)
        v = (h @ w["v_proj.weight"].T).view(T, KV_HEADS, HEAD)
        for r, (p, n) in enumerate(_requests(case)):
            old = _gathered(cache, cache.block_table(r, 0), p, kv_cache)
            heads = []
            for i in range(H):
                g = i // (H // KV_HEADS)
                heads.append(_softmax_attend(q[row:row + n, i], torch.cat([old[0, g], k[row:row + n, g]]),
                                             torch.cat([old[1, g], v[row:row + n, g]]), p, HEAD ** -0.5))
            mixed.append(torch.cat(heads, dim=1))
            row += n
        return x + torch.cat(mixed) @ w["o_proj.weight"].T
    _, H, D, R, V, QR, KR = LATENT[case["size"]]
    T = h.shape[0]
    q = (_rms(h @ w["dq"].T, w["dq.norm"]) @ w["uq"].T).view(T, H, D + R)
    q = torch.cat([q[..., :D], _rotate(q[..., D:], positions, 5e5, True)], dim=-1)
    down = h @ w["dkv"].T
    fresh = torch.cat([_rms(down[:, :KR], w["dkv.norm"]), _rotate(down[:, None, KR:], positions, 5e5, True)[:, 0]], dim=1)
    for r, (p, n) in enumerate(_requests(case)):
        c = torch.cat([_gathered(cache, cache.block_table(r, 0), p, kv_cache)[0, 0], fresh[row:row + n]])
        heads = []
        for i in range(H):
            k = torch.cat([c[:, :KR] @ w["uk"].view(H, D, KR)[i].T, c[:, KR:]], dim=1)
            heads.append(_softmax_attend(q[row:row + n, i], k, c[:, :KR] @ w["uv"].view(H, V, KR)[i].T, p, (D + R) ** -0.5))
        mixed.append(torch.cat(heads, dim=1))
        row += n
    return x + torch.cat(mixed) @ w["o"].T


def _exact_experts(case, w, h):
    W, F, E, top, (count, keep), shared = EXPERTS[case["size"]]
    s = torch.softmax(h @ w["router"].T, dim=-1)
    c = s + w["correction"]
    best = c.view(-1, count, E // count).amax(-1)
    kept = torch.zeros_like(best).scatter_(1, best.topk(keep, dim=1).indices, 1.0).bool()
    c = c.masked_fill(~kept.repeat_interleave(E // count, dim=1), float("-inf"))
    chosen = torch.zeros_like(s).scatter_(1, c.topk(top, dim=1).indices, 1.0) * s
    weight = chosen / chosen.sum(-1, keepdim=True)

    def f(rows, name):
        g = rows @ w[name + ".gate"].T
        return (g * torch.sigmoid(g) * (rows @ w[name + ".up"].T)) @ w[name + ".down"].T
    out = torch.sigmoid(h @ w["shared.sg"].T) * f(h, "shared")
    for e in range(E):
        rows = weight[:, e].nonzero()[:, 0]
        if rows.numel():
            out[rows] += weight[rows, e, None] * f(h[rows], f"e{e}")
    return out


def _exact_mlstm(case, w, h, x, gen):
    _, H, K, V = MLSTM[case["size"]]
    T, reqs = h.shape[0], _requests(case)
    size = build_part(*_spec(case)).cache_need().shape
    state = torch.zeros((len(reqs), *size), device=DEV)
    _fill_memory(state, case, gen)
    state = state.double()
    q, k = (h @ w["q"].T).view(T, H, K) * K ** -0.5, (h @ w["k"].T).view(T, H, K)
    v = (h @ w["v"].T).view(T, H, V)
    i = 15.0 * torch.tanh((h @ w["i"].T + w["i.b"]) / 15.0)
    f = torch.nn.functional.logsigmoid(15.0 * torch.tanh((h @ w["f"].T + w["f.b"]) / 15.0))
    o = torch.empty((T, H, V), dtype=torch.float64, device=DEV)
    # all requests of one length step by step together
    for group in ([r for r, (_, n) in enumerate(reqs) if n == 1 and r < case["singles"]],
                  [r for r in range(case["singles"], len(reqs))]):
        if not group:
            continue
        first = [sum(n for _, n in reqs[:r]) for r in group]
        # a request that decodes is in mid-sequence only when it has cached tokens; others start from zeros
        live = torch.tensor([1.0 if reqs[r][0] > 0 else 0.0 for r in group], device=DEV, dtype=torch.float64)[:, None]
        st = state[group] * live
        S, nn, m = (st[:, :H * K * V].reshape(-1, H, K, V), st[:, H * K * V:H * K * V + H * K].reshape(-1, H, K),
                    st[:, H * K * V + H * K:H * K * V + H * K + H].clone())
        for t in range(reqs[group[0]][1]):
            rows = [a + t for a in first]
            m2 = torch.maximum(f[rows] + m, i[rows])
            a, b = torch.exp(f[rows] + m - m2), torch.exp(i[rows] - m2)
            S = a[..., None, None] * S + (b[..., None] * k[rows])[..., None] * v[rows][:, :, None, :]
            nn = a[..., None] * nn + b[..., None] * k[rows]
            m = m2
            den = torch.maximum((nn * q[rows]).sum(-1).abs(), torch.exp(-m)) + 1e-6
            o[rows] = (S * q[rows][..., None]).sum(-2) / den[..., None]
        state[group, :H * K * V], state[group, H * K * V:H * K * V + H * K] = S.flatten(1), nn.flatten(1)
        state[group, H * K * V + H * K:H * K * V + H * K + H] = m
    o = (o * torch.rsqrt(o.square().mean(-1, keepdim=True) + EPS)).flatten(1) * w["norm"] * torch.sigmoid(h @ w["g"].T)
    return x + o @ w["o"].T, state


def _exact_model(case, seed):
    W, H, G, F, L, V = MODEL[case["size"]]
    tensors = random_tensors_on_device(_model_config(case), int(seed), DEV, "bfloat16", norm_noise=0.1)
    w = {k: v.double() for k, v in tensors.items()}
    logits = []
    for tokens in _model_tokens(case, seed):
        x = w["model.embed_tokens.weight"][torch.tensor(tokens, device=DEV)]
        T = x.shape[0]
        at = torch.arange(T, device=DEV)
        for i in range(L):
            p = f"model.layers.{i}."
            h = _rms(x, w[p + "input_layernorm.weight"])
            q = _rotate(_rms((h @ w[p + "self_attn.q_proj.weight"].T).view(T, H, HEAD), w[p + "self_attn.q_norm.weight"]), at, THETA)
            k = _rotate(_rms((h @ w[p + "self_attn.k_proj.weight"].T).view(T, G, HEAD), w[p + "self_attn.k_norm.weight"]), at, THETA)
            v = (h @ w[p + "self_attn.v_proj.weight"].T).view(T, G, HEAD)
            o = torch.cat([_softmax_attend(q[:, j], k[:, j // (H // G)], v[:, j // (H // G)], 0, HEAD ** -0.5)
                           for j in range(H)], dim=1)
            x = x + o @ w[p + "self_attn.o_proj.weight"].T
            h = _rms(x, w[p + "post_attention_layernorm.weight"])
            g = h @ w[p + "mlp.gate_proj.weight"].T
            x = x + (g * torch.sigmoid(g) * (h @ w[p + "mlp.up_proj.weight"].T)) @ w[p + "mlp.down_proj.weight"].T
        logits.append(_rms(x[-1:], w["model.norm.weight"]) @ w["lm_head.weight"].T)
    return torch.cat(logits)
