"""The work that a user of the engine has it do, as cases that can be timed and compared.

Kinds of cases:

``model``      a whole step of a Qwen3 decoder through ``ModelRunner.step``: decoded tokens (the captured graphs), prompt
               portions beside decoded tokens, in bfloat16 and on the float32 path
``attention``  paged attention of one layer (``ops.paged_attention``): prompts, portions behind cached keys, decoded tokens
``mlp``        a gated feed-forward (``FEED_FORWARDS`` kind ``swiglu``)
``moe``        a mixture of experts (``FEED_FORWARDS`` kind ``moe``), prompts and decoded tokens
``mixer``      a mixer with a matrix state per head (``MIXERS`` kinds ``retention`` and ``channel_delta``)

Sizes are those of ``bench.py`` (Qwen3-8B layers), of ``return_b200.benchmark`` (its 0.6B workload and its ``DESIGN_SIZES``)
and ragged ones of the same ranges.
"""
import math
import zlib

import numpy as np
import torch

from return_b200.cache.manager import CacheManager, GroupSpec
from return_b200.cache.storage import CacheStorage
from return_b200.config.model_config import Qwen3Config
from return_b200.engine.batch import BatchStaging, StepBatch, StepEntry, build_host_batch
from return_b200.engine.config import EngineConfig
from return_b200.engine.runner import ModelRunner
from return_b200.ext import ops
from return_b200.models import qwen3
from return_b200.models.decoder import DecoderModel
from return_b200.parts import FEED_FORWARDS, MIXERS
from return_b200.parts.base import BuildEnv, Tiling
from return_b200.parts.spec import ChannelDeltaSpec, ClampedGLUSpec, MoESpec, RetentionSpec, ScaledRopeSpec, SwiGLUSpec

DEVICE = "cuda:0"
PAGE = 16
EPS = 1e-6
THETA = 1e6


# ------------------------------------------------------------------------------------------------ the cases

def listed():
    """Requests of a case are written "cached+new" per request, separated by commas, "n*..." for n alike."""
    return [
        # the headline of bench.py at four of the 8B model's layers: a decode step of 8 requests behind 2,048 tokens
        {"name": "decode_8b_8x2048", "kind": "model", "dtype": "bfloat16", "hidden": 4096, "ff": 12288, "heads": 32, "kv_heads": 8,
         "layers": 4, "vocab": 151936, "requests": "8*2047+1"},
        # a serving step of the 0.6B workload: a portion of a long prompt and a short prompt beside decoded tokens
        {"name": "mixed_step_0.6b", "kind": "model", "dtype": "bfloat16", "hidden": 1024, "ff": 3072, "heads": 16, "kv_heads": 8,
         "layers": 6, "vocab": 32768, "requests": "1024+401,0+87,24*900+1"},
        # trace replay on the true float32 path: a ragged prompt beside a decoded token
        {"name": "trace_float32", "kind": "model", "dtype": "float32", "hidden": 1024, "ff": 3072, "heads": 16, "kv_heads": 8,
         "layers": 2, "vocab": 8192, "requests": "0+219,128+37,64+1"},
        # one layer's attention over a whole prompt, 8B heads
        {"name": "attention_prompt_2048", "kind": "attention", "heads": 32, "kv_heads": 8, "head_dim": 128, "window": 0,
         "requests": "0+2048"},
        # prompt portions of a serving step: the end of a long prompt, a fresh prompt, a resumed one
        {"name": "attention_portions", "kind": "attention", "heads": 16, "kv_heads": 8, "head_dim": 128, "window": 0,
         "requests": "7680+512,0+200,1500+61"},
        # one layer's attention of a full decode batch, 8B heads
        {"name": "attention_decode_64x2048", "kind": "attention", "heads": 32, "kv_heads": 8, "head_dim": 128, "window": 0,
         "requests": "64*2047+1"},
        # the 8B feed-forward over a prompt
        {"name": "mlp_prompt_2048", "kind": "mlp", "hidden": 4096, "ff": 12288, "tokens": 2048},
        # experts of the "2k" design size over a prompt, and for a decode step
        {"name": "moe_prompt_2048", "kind": "moe", "hidden": 2048, "ff": 1536, "experts": 32, "top": 4, "tokens": 2048},
        {"name": "moe_decode_8", "kind": "moe", "hidden": 2048, "ff": 1536, "experts": 32, "top": 4, "tokens": 8},
        # state mixers of the "2k" design size over a prompt, and the delta rule in a full decode batch
        {"name": "retention_prompt_2048", "kind": "mixer", "mixer": "retention", "hidden": 2048, "heads": 16, "kv_heads": 16,
         "dim": 128, "vdim": 128, "requests": "0+2048"},
        {"name": "delta_prompt_2048", "kind": "mixer", "mixer": "channel_delta", "hidden": 2048, "heads": 16, "kv_heads": 4,
         "dim": 128, "vdim": 128, "requests": "0+2048"},
        {"name": "delta_decode_64", "kind": "mixer", "mixer": "channel_delta", "hidden": 2048, "heads": 16, "kv_heads": 4,
         "dim": 128, "vdim": 128, "requests": "64*900+1"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _prompts(rng, longest):
    """One to three requests that bring several tokens, some of them behind cached ones."""
    parts = []
    for _ in range(rng.choice((1, 1, 2, 3))):
        parts.append("%d+%d" % (rng.choice((0, 0, _log(rng, 16, longest))), max(2, _log(rng, 32, longest) // (1 + len(parts)))))
    return ",".join(parts)


def draw(rng):
    kind = rng.choice(("model", "attention", "attention", "mlp", "moe", "mixer", "mixer"))
    if kind == "model":
        hidden, ff, heads, layers = rng.choice(((1024, 3072, 16, 6), (2048, 6144, 16, 3), (4096, 12288, 32, 2)))
        case = {"kind": kind, "dtype": rng.choice(("bfloat16", "bfloat16", "float32")), "hidden": hidden, "ff": ff, "heads": heads,
                "kv_heads": 8, "layers": layers, "vocab": rng.choice((8192, 32768))}
        if case["dtype"] == "float32":
            case.update(hidden=1024, ff=3072, heads=16, layers=rng.choice((1, 2)), vocab=8192,
                        requests="%d+%d,%d+1" % (_log(rng, 16, 200), _log(rng, 16, 250), _log(rng, 16, 200)))
        elif rng.random() < 0.5:
            case["requests"] = "%d*%d+1" % (_log(rng, 1, 64), _log(rng, 60, 1500))
        else:
            case["requests"] = "%d+%d,%d*%d+1" % (_log(rng, 16, 2000), _log(rng, 32, 600), _log(rng, 1, 40), _log(rng, 60, 1000))
        return case
    if kind == "attention":
        heads, kv_heads = rng.choice(((16, 8), (32, 8), (16, 4)))
        case = {"kind": kind, "heads": heads, "kv_heads": kv_heads, "head_dim": rng.choice((128, 128, 128, 64)),
                "window": rng.choice((0, 0, 0, 1024))}
        if rng.random() < 0.5:
            n = _log(rng, 1, 64)
            case["requests"] = "%d*%d+1" % (n, _log(rng, 100, 120000 // n if n > 8 else 12000))
        else:
            case["requests"] = _prompts(rng, 2000)
        return case
    if kind == "mlp":
        hidden, ff = rng.choice(((1024, 3072), (2048, 6144), (4096, 12288)))
        return {"kind": kind, "hidden": hidden, "ff": ff, "tokens": _log(rng, 1, 2040)}
    if kind == "moe":
        hidden, ff = rng.choice(((1024, 768), (2048, 1536)))
        return {"kind": kind, "hidden": hidden, "ff": ff, "experts": rng.choice((16, 32, 64)), "top": rng.choice((2, 4)),
                "tokens": _log(rng, 1, 2040)}
    heads = rng.choice((4, 8, 16))
    mixer = rng.choice(("retention", "channel_delta"))
    case = {"kind": kind, "mixer": mixer, "hidden": 128 * heads, "heads": heads,
            "kv_heads": heads if mixer == "retention" else rng.choice((heads, heads // 4)),
            "dim": rng.choice((128, 128, 64)), "vdim": rng.choice((128, 128, 64, 256))}
    case["requests"] = _prompts(rng, 2000) if rng.random() < 0.7 else "%d*%d+1" % (_log(rng, 1, 64), _log(rng, 60, 1000))
    return case


def _requests(case):
    """[(tokens cached before the step, tokens the step brings)]"""
    out = []
    for part in case["requests"].split(","):
        n, _, rest = part.rpartition("*")
        cached, new = rest.split("+")
        out += [(int(cached), int(new))] * (int(n) if n else 1)
    return out


# ------------------------------------------------------------------------------------------------ inputs

def _normal(seed, tag, shape, dtype=torch.bfloat16, mean=0.0, std=1.0):
    """A tensor that depends on the seed and its name alone."""
    g = torch.Generator(device=DEVICE).manual_seed((int(seed) * 1000003 + zlib.crc32(tag.encode())) % (1 << 62))
    return torch.empty(shape, dtype=torch.float32, device=DEVICE).normal_(mean, std, generator=g).to(dtype)


def _tokens(seed, tag, n, vocab):
    return np.random.RandomState((int(seed) * 7919 + zlib.crc32(tag.encode())) % (1 << 32)).randint(0, vocab, n).tolist()


def _model_weights(case, seed):
    """The parameters of the decoder by name, with the laws of the engine's random-weights mode."""
    h, ff, D = case["hidden"], case["ff"], 128
    dt = getattr(torch, case["dtype"])
    q, kv = case["heads"] * D, case["kv_heads"] * D
    shapes = {"embed": (case["vocab"], h), "lm_head": (case["vocab"], h), "final_norm.weight": (h,)}
    for i in range(case["layers"]):
        p = "layers.%d." % i
        shapes.update({p + "mixer.qkv": (q + 2 * kv, h), p + "mixer.o": (h, q), p + "mixer.q_norm.weight": (D,),
                       p + "mixer.k_norm.weight": (D,), p + "feed_forward.gate_up": (2 * ff, h), p + "feed_forward.down": (h, ff),
                       p + "mixer_norm.weight": (h,), p + "feed_forward_norm.weight": (h,)})
    return {n: _normal(seed, n, s, dt, 1.0, 0.1) if len(s) == 1 else _normal(seed, n, s, dt, 0.0, 0.02) for n, s in shapes.items()}


def _swiglu_weights(case, seed):
    return {"gate_up": _normal(seed, "gate_up", (2 * case["ff"], case["hidden"]), std=0.02),
            "down": _normal(seed, "down", (case["hidden"], case["ff"]), std=0.02)}


def _moe_weights(case, seed):
    h, f, e = case["hidden"], case["ff"], case["experts"]
    shapes = {"router": (e, h), "experts.gate_up": (e * 2 * f, h), "experts.down": (e * h, f), "shared.gate_up": (2 * f, h),
              "shared.down": (h, f)}
    return {n: _normal(seed, n, s, std=0.02) for n, s in shapes.items()}


def _mixer_weights(case, seed):
    W, H, G, D, V = (case[k] for k in ("hidden", "heads", "kv_heads", "dim", "vdim"))
    if case["mixer"] == "retention":
        return {"in": _normal(seed, "in", (2 * H * D + 2 * H * V, W), std=0.02), "o": _normal(seed, "o", (W, H * V), std=0.02)}
    C = 2 * G * D + H * V
    return {"in": _normal(seed, "in", (C + 128, W), std=0.02), "conv": _normal(seed, "conv", (C, 4), std=0.5),
            "beta": _normal(seed, "beta", (H, W), std=0.02), "decay_up": _normal(seed, "decay_up", (H * D, 64), std=0.2),
            "gate_up": _normal(seed, "gate_up", (H * V, 64), std=0.2), "A_log": _normal(seed, "A_log", (H,), std=0.5),
            "dt_bias": _normal(seed, "dt_bias", (H * D,), std=0.5), "norm": _normal(seed, "norm", (V,), mean=1.0, std=0.1),
            "o": _normal(seed, "o", (W, H * V), std=0.02)}


def _decays(case):
    return [1.0 - 2.0 ** -(5 + 4 * i / max(1, case["heads"] - 1)) for i in range(case["heads"])]


def _mixer_spec(case):
    W, H, D, V = (case[k] for k in ("hidden", "heads", "dim", "vdim"))
    if case["mixer"] == "retention":
        return RetentionSpec(hidden_size=W, num_heads=H, key_dim=D, value_dim=V, decay=tuple(_decays(case)), eps=1e-5,
                             position=ScaledRopeSpec(rotary_dim=D, theta=THETA, max_positions=8192))
    return ChannelDeltaSpec(hidden_size=W, num_heads=H, num_kv_heads=case["kv_heads"], key_dim=D, value_dim=V, conv_taps=4,
                            decay_rank=64, gate_rank=64, eps=1e-5)


def _fill(manager, requests, stride=256):
    """Takes the requests in and makes room for their cached tokens, a run at a time in turn, so that their pages lie among
    each other as they do in serving."""
    for i in range(len(requests)):
        manager.add(i)
    longest = max(c for c, _ in requests)
    for at in range(0, longest, stride):
        for i, (cached, _) in enumerate(requests):
            if at < cached:
                manager.append(i, min(stride, cached - at))


def _step_batch(manager, requests, tilings=None):
    entries = []
    for i, (_, new) in enumerate(requests):
        entries.append(StepEntry(rid=i, tokens=[0] * new, start=manager.append(i, new)))
    return StepBatch(build_host_batch(entries, manager, tilings=tilings), DEVICE, BatchStaging(DEVICE))


def _rows(case):
    return sum(n for _, n in _requests(case)) if "requests" in case else case["tokens"]


def _x(case, seed):
    """Rows as they come out of a norm."""
    return _normal(seed, "x", (_rows(case), case["hidden"]))


# ------------------------------------------------------------------------------------------------ prepare and run

def _prepare_model(case, seed):
    requests = _requests(case)
    room = sum((c + n + 63) // 64 * 64 for c, n in requests)
    limit = max(2048, max(c + n for c, n in requests))
    cfg = Qwen3Config.from_dict(dict(vocab_size=case["vocab"], hidden_size=case["hidden"], intermediate_size=case["ff"],
                                     num_hidden_layers=case["layers"], num_attention_heads=case["heads"],
                                     num_key_value_heads=case["kv_heads"], head_dim=128, rope_theta=THETA, rms_norm_eps=EPS,
                                     tie_word_embeddings=False, max_position_embeddings=40960))
    ecfg = EngineConfig(max_token=room + 64, max_reside=len(requests), page_size=PAGE, prefill_chunk=8192, dtype=case["dtype"],
                        max_model_len=limit)
    env = BuildEnv(ecfg.act_dtype, torch.device(DEVICE))
    model = DecoderModel(qwen3.decoder_spec(cfg, limit), env)
    model.bind(_model_weights(case, seed))
    runner = ModelRunner(model, ecfg, limit)
    entries = []
    for i, (cached, new) in enumerate(requests):
        ids = _tokens(seed, "request %d" % i, cached + new, case["vocab"])
        runner.add_request(i)
        if cached:
            runner.step([runner.reserve(i, ids[:cached])])
        # a decoded token's logits, and those of a portion's last token
        entries.append((i, ids[cached:], [new - 1]))
    entries = [runner.reserve(*e) for e in entries]
    runner.step(entries)              # a serving program has captured its decode graphs
    return {"runner": runner, "entries": entries}


def _prepare_attention(case, seed):
    requests = _requests(case)
    H, G, D, window = case["heads"], case["kv_heads"], case["head_dim"], case["window"] or None
    pages = sum((c + n + PAGE - 1) // PAGE + 1 for c, n in requests)
    manager = CacheManager([GroupSpec("keys", PAGE, pages, window)], len(requests))
    _fill(manager, requests)
    batch = _step_batch(manager, requests, {ops.TILES_TC5: Tiling(ops.TC5_TILE_ROWS, heaviest_first=True)})
    T = batch.num_tokens
    return {"batch": batch, "heads": H, "kv_heads": G, "head_dim": D, "window": window,
            "qkv": _normal(seed, "qkv", (T, (H + 2 * G) * D)), "k": _normal(seed, "k", (pages, G, PAGE, D)),
            "v": _normal(seed, "v", (pages, G, PAGE, D)), "out": torch.empty((T, H * D), dtype=torch.bfloat16, device=DEVICE)}


def _prepare_part(case, seed):
    env = BuildEnv(torch.bfloat16, torch.device(DEVICE))
    if case["kind"] == "mlp":
        part = FEED_FORWARDS.build(SwiGLUSpec(case["hidden"], case["ff"], interleave=8), env)
        weights, requests = _swiglu_weights(case, seed), [(0, case["tokens"])]
    elif case["kind"] == "moe":
        unit = ClampedGLUSpec(case["hidden"], case["ff"], 7.0)
        part = FEED_FORWARDS.build(MoESpec(case["hidden"], case["experts"], case["top"], unit, groups=8, keep_groups=4, shared=unit), env)
        weights, requests = _moe_weights(case, seed), [(0, case["tokens"])]
    else:
        part = MIXERS.build(_mixer_spec(case), env)
        weights, requests = _mixer_weights(case, seed), _requests(case)
    part.bind(weights)
    need = part.cache_need() if case["kind"] == "mixer" else None
    storage = CacheStorage([need], PAGE, sum((c + n + PAGE - 1) // PAGE + 1 for c, n in requests), len(requests), env)
    manager = storage.make_manager()
    storage.allocate()
    _fill(manager, requests)
    ctx = storage.layer_context(0, _step_batch(manager, requests), True)
    if need is not None:              # requests in the middle of their sequence carry a state; others start from zero
        for i, (cached, _) in enumerate(requests):
            if cached:
                ctx.state[i].copy_(_normal(seed, "state %d" % i, ctx.state[i].shape, torch.float32, std=0.3))
    return {"part": part, "ctx": ctx, "x": _x(case, seed), "storage": storage,
            "fresh": [i for i, (cached, _) in enumerate(requests) if not cached] if need is not None else []}


def prepare(case, seed):
    return {"model": _prepare_model, "attention": _prepare_attention}.get(case["kind"], _prepare_part)(case, seed)


@torch.no_grad()
def run(state):
    if "runner" in state:
        return state["runner"].step(state["entries"])
    if "qkv" in state:
        s = state
        ops.paged_attention(s["qkv"], s["k"], s["v"], s["batch"], s["batch"].block_tables[0], PAGE, s["out"], s["heads"],
                            s["kv_heads"], s["head_dim"], s["head_dim"] ** -0.5, s["window"])
        return s["out"]
    for slot in state["fresh"]:       # a request that starts takes its slot anew
        state["storage"].reset_slot(slot)
    y = state["part"].forward(state["x"], state["ctx"])
    held = state["ctx"].state
    return y if held is None else (y, held[:-1])


# ------------------------------------------------------------------------------------------------ what a pass cannot do without

def _seen(cached, new, window):
    """(keys that a request's tokens read between them, pairs of a token and a key that it sees)"""
    pairs = sum(min(cached + i + 1, window) if window else cached + i + 1 for i in range(new))
    keys = min(cached + new, window + new - 1) if window else cached + new
    return keys, pairs


def work(case):
    rows = _rows(case)
    if case["kind"] == "attention":
        H, G, D = case["heads"], case["kv_heads"], case["head_dim"]
        seen = [_seen(c, n, case["window"]) for c, n in _requests(case)]
        return {"bytes": 2 * (2 * G * D * sum(k for k, _ in seen) + 2 * rows * H * D), "flops": 4 * H * D * sum(p for _, p in seen)}
    h, f = case["hidden"], case.get("ff", 0)
    if case["kind"] == "mlp":
        return {"bytes": 2 * (3 * h * f + 2 * rows * h), "flops": 6 * rows * h * f}
    if case["kind"] == "moe":
        pairs, E = rows * case["top"], case["experts"]
        reached = E * (1 - (1 - case["top"] / E) ** rows)
        return {"bytes": 2 * (3 * h * f * (reached + 1) + E * h + 2 * rows * h), "flops": 6 * h * f * (pairs + rows) + 2 * rows * E * h}
    if case["kind"] == "mixer":
        H, D, V = case["heads"], case["dim"], case["vdim"]
        weights = sum(math.prod(s) for s in (((2 * H * D + 2 * H * V, h), (h, H * V)) if case["mixer"] == "retention" else
                                             ((2 * case["kv_heads"] * D + H * V + 128 + H, h), (H * (D + V), 64), (h, H * V))))
        states = sum((4 if c else 0) + 4 for c, _ in _requests(case)) * H * D * V
        return {"bytes": 2 * weights + states + 6 * rows * h,
                "flops": 2 * rows * weights + (4 if case["mixer"] == "retention" else 8) * rows * H * D * V}
    q, kv, D = case["heads"] * 128, case["kv_heads"] * 128, 128
    size = 4 if case["dtype"] == "float32" else 2
    layer = (q + 2 * kv) * h + q * h + 3 * h * f
    seen = [_seen(c, n, 0) for c, n in _requests(case)]
    n = len(seen)
    return {"bytes": size * (case["layers"] * (layer + 2 * kv * sum(k for k, _ in seen)) + case["vocab"] * h + rows * h) + 4 * n * case["vocab"],
            "flops": 2 * rows * case["layers"] * layer + 4 * q * case["layers"] * sum(p for _, p in seen) + 2 * n * case["vocab"] * h}


def tolerance(case):
    if case["kind"] == "model":
        return {"rel": 2e-5} if case["dtype"] == "float32" else {"rel": 2e-2}
    return {"rel": 1e-2}


# ------------------------------------------------------------------------------------------------ the same in 64 bits

def _silu(x):
    return x * torch.sigmoid(x)


def _rms(x, eps, weight=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if weight is None else y * weight


def _rotate(x, positions, theta=THETA):
    """x [T, heads, D], the two halves of a head are the pairs' parts."""
    half = x.shape[-1] // 2
    f = float(theta) ** (-torch.arange(half, dtype=torch.float64, device=x.device) / half)
    a = positions.double()[:, None, None] * f
    u, v = x[..., :half], x[..., half:]
    return torch.cat((u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()), -1)


def _softmax_attention(q, k, v, first, window=0):
    """q [n, H, D] at positions first, first + 1, ...; k, v [keys, G, D] from position 0."""
    n, H, D = q.shape
    rep = H // k.shape[1]
    i = torch.arange(first, first + n, device=q.device)[:, None]
    j = torch.arange(k.shape[0], device=q.device)[None, :]
    hidden = (j > i) | ((j <= i - window) if window else torch.zeros_like(j > i))
    out = torch.empty_like(q)
    for h in range(H):
        s = (q[:, h] @ k[:, h // rep].T) * D ** -0.5
        out[:, h] = torch.softmax(s.masked_fill(hidden, -math.inf), -1) @ v[:, h // rep]
    return out


def _exact_model(case, seed):
    requests = _requests(case)
    if sum(c + n for c, n in requests) * case["layers"] * case["hidden"] * case["ff"] > 1e13:
        return None
    w = _model_weights(case, seed)
    H, G, D = case["heads"], case["kv_heads"], 128
    last = []
    for r, (cached, new) in enumerate(requests):
        ids = torch.tensor(_tokens(seed, "request %d" % r, cached + new, case["vocab"]), device=DEVICE)
        x = w["embed"][ids].double()
        positions = torch.arange(len(ids), device=DEVICE)
        for i in range(case["layers"]):
            p = {n: t.double() for n, t in w.items() if n.startswith("layers.%d." % i)}
            p = {n.split(".", 2)[2]: t for n, t in p.items()}
            qkv = (_rms(x, EPS, p["mixer_norm.weight"]) @ p["mixer.qkv"].T).view(len(ids), H + 2 * G, D)
            q = _rotate(_rms(qkv[:, :H], EPS, p["mixer.q_norm.weight"]), positions)
            k = _rotate(_rms(qkv[:, H:H + G], EPS, p["mixer.k_norm.weight"]), positions)
            x = x + _softmax_attention(q, k, qkv[:, H + G:], 0).reshape(len(ids), H * D) @ p["mixer.o"].T
            x = x + _exact_swiglu(_rms(x, EPS, p["feed_forward_norm.weight"]), p["feed_forward.gate_up"], p["feed_forward.down"])
        last.append(_rms(x[-1], EPS, w["final_norm.weight"].double()))
    last = torch.stack(last)
    return torch.cat([last @ part.double().T for part in w["lm_head"].split(16384)], 1)


def _exact_swiglu(x, gate_up, down):
    """The rows of gate_up come in blocks: 8 gate rows, then their 8 up rows."""
    gu = (x @ gate_up.T).view(x.shape[0], -1, 2, 8)
    return (_silu(gu[:, :, 0]) * gu[:, :, 1]).reshape(x.shape[0], -1) @ down.T


def _exact_attention(case, seed):
    s = _prepare_attention(case, seed)
    H, G, D = case["heads"], case["kv_heads"], case["head_dim"]
    out, row = [], 0
    for r, (cached, new) in enumerate(_requests(case)):
        q = s["qkv"][row:row + new, :H * D].double().view(new, H, D)
        pages = s["batch"].block_tables[0][r, :(cached + new + PAGE - 1) // PAGE].long().clamp(min=0)
        k, v = (t[pages].transpose(1, 2).reshape(-1, G, D)[:cached + new].double() for t in (s["k"], s["v"]))
        out.append(_softmax_attention(q, k, v, cached, case["window"]).reshape(new, H * D))
        row += new
    return torch.cat(out)


def _clamped_unit(x, gate_up, down):
    f = down.shape[1]
    gu = x @ gate_up.T
    g, u = gu[:, :f].clamp(max=7.0), gu[:, f:].clamp(-7.0, 7.0)
    return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ down.T


def _exact_moe(case, seed):
    w, x = _moe_weights(case, seed), _x(case, seed).double()
    E, T = case["experts"], x.shape[0]
    score = torch.softmax(x @ w["router"].double().T, -1).view(T, 8, E // 8)
    best = score.amax(-1).topk(4, -1).indices
    score = torch.zeros_like(score).scatter(1, best[:, :, None].expand(-1, -1, E // 8), 1.0) * score
    value, chosen = score.view(T, E).topk(case["top"], -1)
    value = value / (value.sum(-1, keepdim=True) + 1e-20)
    y = _clamped_unit(x, w["shared.gate_up"].double(), w["shared.down"].double())
    up, down = w["experts.gate_up"].view(E, -1, case["hidden"]), w["experts.down"].view(E, case["hidden"], -1)
    for e in range(E):
        t, k = (chosen == e).nonzero(as_tuple=True)
        y[t] += value[t, k, None] * _clamped_unit(x[t], up[e].double(), down[e].double())
    return y


def _state_rows(S):
    """A state [heads, key rows, columns] in the order in which a request's slot holds it."""
    H, D, V = S.shape
    return S.view(H, D // 8, 8, V).transpose(2, 3).reshape(-1)


def _exact_mixer(case, seed):
    w = {n: t.double() for n, t in _mixer_weights(case, seed).items()}
    x = _x(case, seed).double()
    W, H, G, D, V = (case[k] for k in ("hidden", "heads", "kv_heads", "dim", "vdim"))
    delta = case["mixer"] == "channel_delta"
    C = 2 * G * D + H * V
    floats = H * D * V + (3 * C if delta else 0)
    ys, states, row = [], [], 0
    for r, (cached, new) in enumerate(_requests(case)):
        held = _normal(seed, "state %d" % r, (floats,), torch.float32, std=0.3).double() if cached else torch.zeros(
            floats, dtype=torch.float64, device=DEVICE)
        S = held[:H * D * V].view(H, D // 8, V, 8).transpose(2, 3).reshape(H, D, V).clone()
        h = x[row:row + new]
        p = h @ w["in"].T
        if delta:
            full = torch.cat((held[H * D * V:].view(C, 3).T, p[:, :C]))
            conv = _silu(sum(full[i:i + new] * w["conv"][:, i] for i in range(4)))
            q, k = (_unit(conv[:, i * G * D:(i + 1) * G * D].view(new, G, D)).repeat_interleave(H // G, 1) for i in (0, 1))
            q = q * D ** -0.5
            v = conv[:, 2 * G * D:].view(new, H, V)
            beta = torch.sigmoid(h @ w["beta"].T)
            step = torch.nn.functional.softplus(p[:, C:C + 64] @ w["decay_up"].T + w["dt_bias"]).view(new, H, D)
            decay = torch.exp(-torch.exp(w["A_log"])[None, :, None] * step)
        else:
            positions = torch.arange(cached, cached + new, device=DEVICE)
            q = _rotate(p[:, :H * D].view(new, H, D), positions)
            k = _rotate(p[:, H * D:2 * H * D].view(new, H, D), positions) * D ** -0.5
            v = p[:, 2 * H * D:2 * H * D + H * V].view(new, H, V)
            decay = torch.tensor(_decays(case), dtype=torch.float64, device=DEVICE)[None, :, None].expand(new, H, 1)
        o = torch.empty((new, H, V), dtype=torch.float64, device=DEVICE)
        for t in range(new):
            S *= decay[t][:, :, None]
            u = v[t]
            if delta:
                u = beta[t][:, None] * (u - torch.bmm(k[t][:, None], S)[:, 0])
            S.baddbmm_(k[t][:, :, None], u[:, None])
            o[t] = torch.bmm(q[t][:, None], S)[:, 0]
        if delta:
            o = _rms(o, 1e-5, w["norm"]) * torch.sigmoid(p[:, C + 64:] @ w["gate_up"].T).view(new, H, V)
        else:
            o = _rms(o, 1e-5) * _silu(p[:, 2 * H * D + H * V:]).view(new, H, V)
        ys.append(o.reshape(new, H * V) @ w["o"].T)
        rest = [full[-3:].T.reshape(-1)] if delta else []
        states.append(torch.cat([_state_rows(S)] + rest))
        row += new
    return torch.cat(ys), torch.stack(states)


def _unit(x):
    return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)


@torch.no_grad()
def exact(case, seed):
    if case["kind"] == "model":
        return _exact_model(case, seed)
    if case["kind"] == "attention":
        return _exact_attention(case, seed)
    if case["kind"] == "mlp":
        w = _swiglu_weights(case, seed)
        return _exact_swiglu(_x(case, seed).double(), w["gate_up"].double(), w["down"].double())
    return (_exact_moe if case["kind"] == "moe" else _exact_mixer)(case, seed)
