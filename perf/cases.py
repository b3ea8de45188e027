"""What a user of this engine has it do, as cases that can be timed and compared.

Whole steps of a Qwen2 decoder (a decoded token for every request of a batch, a prompt) in both data types, through
``ModelRunner``; the draw of the next tokens from a step's logits; and single layers of the other architectures over a
prompt, each through the part's own ``forward`` (weights, page pools and the step's context in hand, as in a model).

``exact`` is the same in plain torch in 64 bits, from the same weights and inputs.
"""
import hashlib
import math
from dataclasses import replace

import torch

from mimirmind_b200.config.spec import PartSpec
from mimirmind_b200.engine.engine import Engine
from mimirmind_b200.engine.loader import make_runtime
from mimirmind_b200.engine.model import Model
from mimirmind_b200.engine.runner import StepEntry
from mimirmind_b200.kernels import ops
from mimirmind_b200.parts.base import LayerCache, StepContext, WeightView
from mimirmind_b200.registry import FEED_FORWARDS, MIXERS, get_architecture
from mimirmind_b200.weights.store import expected_tensors

DEV = "cuda"
PAGE = 16
LAYERS = 2                      # of the whole-step cases: a layer's hand-over to the next is in them, and 16-bit roundings stay comparable

# layer sizes of two published decoders of the architecture
SHAPES = {
    "7b": dict(hidden_size=3584, num_attention_heads=28, num_key_value_heads=4, head_dim=128, intermediate_size=18944,
               vocab_size=152064, tie_word_embeddings=False),
    "0.5b": dict(hidden_size=896, num_attention_heads=14, num_key_value_heads=2, head_dim=64, intermediate_size=4864,
                 vocab_size=151936, tie_word_embeddings=True),
}
# layer sizes at which the other architectures are compared with one another
SIZES = {
    "w2048": dict(width=2048, heads=16, kv_heads=4, dim=128, vdim=64, window=1024, ff=8192),
    "w4096": dict(width=4096, heads=32, kv_heads=8, dim=128, vdim=128, window=4096, ff=16384),
}
STEPS = ("decode", "prompt")
MIXER_KINDS = ("sink", "delta", "retention", "forget", "differential")


def listed():
    return [
        # a decode step of a small batch on a 7B-shaped decoder: what serving spends its time on
        dict(name="decode-7b-b8", kind="decode", shape="7b", dtype="bfloat16", batch=8, context=2048),
        # the smallest call: one token of one request on a small model, where launches and latency count
        dict(name="decode-0.5b-b1", kind="decode", shape="0.5b", dtype="bfloat16", batch=1, context=130),
        # a long prompt in one step, the largest call
        dict(name="prompt-7b-4096", kind="prompt", shape="7b", dtype="bfloat16", tokens=4096),
        # the 32-bit runs, which exist for results that do not depend on how the work is cut: a prompt and a decode step
        dict(name="prompt-0.5b-f32", kind="prompt", shape="0.5b", dtype="float32", tokens=509),
        dict(name="decode-0.5b-f32", kind="decode", shape="0.5b", dtype="float32", batch=4, context=300),
        # sampled decoding: the draw that follows every decode step
        dict(name="sample-32", kind="sample", rows=32, vocab=152064, temperature=0.8, top_k=0, top_p=0.95),
        # windowed attention with a sink over several prompts of unequal length in one step
        dict(name="sink-3x", kind="sink", size="w2048", tokens=4001, requests=3),
        # the gated delta rule over a long prompt
        dict(name="delta-4096", kind="delta", size="w2048", tokens=4096, requests=1),
        # a matrix state with a constant decay, two prompts
        dict(name="retention-2x", kind="retention", size="w4096", tokens=3000, requests=2),
        # a matrix state with a forget gate per key channel
        dict(name="forget-2048", kind="forget", size="w2048", tokens=2048, requests=1),
        # routed experts over an ordinary prompt
        dict(name="experts-1500", kind="experts", size="w2048", tokens=1500),
        # differential attention over an ordinary prompt
        dict(name="differential-2048", kind="differential", size="w2048", tokens=2048, requests=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "prompt", "f32 decode", "f32 prompt", "sample", "sink", "delta", "retention", "forget", "experts",
                       "differential"])
    if kind == "decode":
        return dict(kind="decode", shape=rng.choice(["7b", "7b", "0.5b"]), dtype="bfloat16", batch=_log(rng, 1, 64), context=_log(rng, 100, 2500))
    if kind == "prompt":
        return dict(kind="prompt", shape=rng.choice(["7b", "0.5b"]), dtype="bfloat16", tokens=_log(rng, 65, 4096))
    if kind == "f32 decode":
        return dict(kind="decode", shape="0.5b", dtype="float32", batch=_log(rng, 1, 16), context=_log(rng, 30, 1000))
    if kind == "f32 prompt":
        return dict(kind="prompt", shape="0.5b", dtype="float32", tokens=_log(rng, 17, 1024))
    if kind == "sample":
        return dict(kind="sample", rows=_log(rng, 1, 64), vocab=rng.choice([32768, 65536, 151936, 152064]),
                    temperature=round(rng.uniform(0.3, 1.5), 2), top_k=rng.choice([0, 0, 20, 50, 200]), top_p=rng.choice([1.0, 0.8, 0.9, 0.95, 0.99]))
    size = rng.choice(sorted(SIZES))
    top = 4096 if size == "w2048" else 3000
    if kind == "experts":
        return dict(kind=kind, size=size, tokens=_log(rng, 8, top))
    return dict(kind=kind, size=size, tokens=_log(rng, 260, top), requests=rng.randint(1, 4))


# ---- weights and inputs --------------------------------------------------------------------------------------------------
def _generator(seed, name):
    g = torch.Generator(device=DEV)
    g.manual_seed(int.from_bytes(hashlib.sha256(f"{seed}:{name}".encode()).digest()[:7], "little"))
    return g


def _fill(spec, seed, dtype):
    """A tensor of the size and spread that its role has in a trained layer."""
    x = torch.randn(spec.shape, generator=_generator(seed, spec.name), device=DEV)
    if spec.role == "norm":
        x = 1.0 + 0.1 * x
    elif spec.role == "taps":
        x = 0.5 * x
    elif spec.role == "router":
        x = 0.2 * x
    elif spec.role == "lower_bound":
        x = torch.sigmoid(x)
    else:
        x = 0.02 * x
    return x.to(dtype)


def _dtype(case):
    return torch.float32 if case.get("dtype") == "float32" else torch.bfloat16


def _decoder(case):
    arch = get_architecture("Qwen2ForCausalLM")
    return arch.build_spec(arch.parse_config(dict(
        architectures=["Qwen2ForCausalLM"], model_type="qwen2", num_hidden_layers=LAYERS, rope_theta=1000000.0, rms_norm_eps=1e-6,
        max_position_embeddings=8192, use_sliding_window=False, torch_dtype=case["dtype"], **SHAPES[case["shape"]]), "cases"))


def _layer(case):
    """The layer of the case's architecture, as its configuration describes it."""
    z, kind = SIZES[case["size"]], case["kind"]
    d, H, G, dk, dv = z["width"], z["heads"], z["kv_heads"], z["dim"], z["vdim"]
    decay = [1.0 - 2.0 ** (-3 - 5 * h / max(1, H - 1)) for h in range(H)]
    ff = -(-(2 * z["ff"] // 12) // 64) * 64
    state = {"heads": H, "dim": dk, "vdim": dk}
    layer = {
        "sink": {"type": "attention", "mlp": None, "mixer": {"heads": H, "kv_heads": G, "dim": dk, "vdim": dv, "scale": dk ** -0.5,
                                                            "mask": {"size": z["window"]}, "rot": {"dims": dk, "base": 10000.0}, "v_mix": False}},
        "delta": {"type": "delta", "mlp": None, "mixer": dict(state, kv_heads=G, conv=4)},
        "retention": {"type": "retention", "mlp": None, "mixer": dict(state, decay=decay, rot={"dims": dk, "base": 10000.0})},
        "experts": {"type": "delta", "mixer": dict(state, kv_heads=G, conv=4),
                    "mlp": {"kind": "moe", "expert": {"ff": ff}, "router": {"experts": 16, "top": 4, "groups": {"count": 4, "keep": 2}}}},
        "forget": {"type": "parallel", "mlp": None,
                   "mixer": {"left": {"heads": H, "kv_heads": G, "dim": dk, "vdim": dv, "scale": dk ** -0.5, "conv": 4,
                                      "rot": {"dims": dk, "base": 10000.0}},
                             "right": {"heads": H, "dim": dk, "vdim": dv}, "left_scale": 1.0, "right_scale": 1.0}},
        "differential": {"type": "attention", "mlp": None,
                         "mixer": {"heads": H, "kv_heads": G, "dim": dk // 2, "vdim": dk, "scale": (dk // 2) ** -0.5, "softcap": 30.0, "diff": 0.5,
                                   "conv": 4, "mask": {"size": z["window"]}}},
    }[kind]
    name = {"sink": "Bigerax", "forget": "Zubarax", "differential": "Tupunex"}.get(kind, "Domelix")
    cfg = {"architecture": name, "vocab": 64, "width": d, "norm": {"eps": 1e-6}, "layers": [layer]}
    if name == "Bigerax":
        cfg.update(norm={"eps": 1e-6, "groups": 2}, embedding={"bigram": {"buckets": 61, "mul_prev": 33, "mul_cur": 7}})
    if name == "Zubarax":
        cfg.update(postln_alpha=2.0, embedding={"scale": 1.0})
    if name == "Tupunex":
        cfg.update(streams=4, embedding={"scale": 1.0})
    arch = get_architecture(name)
    spec = arch.build_spec(arch.parse_config(cfg, "cases")).layers[0]
    if kind == "experts":
        return FEED_FORWARDS, spec.feed_forward
    return MIXERS, spec.mixer["right"] if kind == "forget" else spec.mixer


def _layer_weights(registry, part, seed):
    return {s.name: _fill(s, seed, torch.bfloat16) for s in registry.get(part.kind).tensor_specs(part, "")}


def _decoder_weights(spec, seed, dtype):
    return {n: _fill(replace(s, name=n), seed, dtype) for n, s in expected_tensors(spec).items() if not s.optional}


def _tokens(seed, name, shape, vocab):
    return torch.randint(0, vocab, shape, generator=_generator(seed, name), device=DEV)


def _rows(case, seed):
    """What a layer gets: normalised activations of the step's tokens."""
    width = SIZES[case["size"]]["width"]
    return torch.randn((case["tokens"], width), generator=_generator(seed, "rows"), device=DEV).to(torch.bfloat16)


def _lengths(case):
    """The tokens shared out unequally over the requests."""
    r = case.get("requests", 1)
    total, weights = case["tokens"], [2 * i + 3 for i in range(r)]
    out = [total * w // sum(weights) for w in weights]
    out[-1] += total - sum(out)
    return out


def _logits(case, seed):
    """A row of logits with a few likely tokens above a wide tail, as a language model's."""
    g = _generator(seed, "logits")
    x = 2.0 * torch.randn((case["rows"], case["vocab"]), generator=g, device=DEV)
    best = torch.randint(0, case["vocab"], (case["rows"], 24), generator=g, device=DEV)
    lift = 10.0 * torch.rand((case["rows"], 24), generator=g, device=DEV)
    return x.scatter_add_(1, best, lift)


# ---- what a program has in hand, and one pass ----------------------------------------------------------------------------
def prepare(case, seed):
    if case["kind"] in STEPS:
        return _prepare_step(case, seed)
    if case["kind"] == "sample":
        r = case["rows"]
        full = lambda v, t: torch.full((r,), v, dtype=t, device=DEV)      # noqa: E731
        return dict(kind="sample", args=(_logits(case, seed), full(case["temperature"], torch.float32), full(case["top_k"], torch.int32),
                                         full(case["top_p"], torch.float32), torch.arange(1, r + 1, device=DEV) + 1000 * seed,
                                         torch.arange(r, device=DEV) + 7))
    rt = make_runtime("bfloat16")
    registry, part_spec = _layer(case)
    part = registry.get(part_spec.kind)(part_spec, WeightView(_layer_weights(registry, part_spec, seed)), rt)
    lens = _lengths(case)
    starts = [sum(lens[:i]) for i in range(len(lens))]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)        # noqa: E731
    positions = torch.cat([torch.arange(n, dtype=torch.int32, device=DEV) for n in lens])
    request = torch.cat([torch.full((n,), i, dtype=torch.int32, device=DEV) for i, n in enumerate(lens)])
    ctx = StepContext(n_tokens=sum(lens), n_requests=len(lens), token_ids=torch.zeros_like(positions), positions=positions, token_req=request,
                      q_start=starts, q_len=lens, kv_len=lens, req_meta=i32([[s, n, n, i] for i, (s, n) in enumerate(zip(starts, lens))]),
                      state_slots=i32(list(range(len(lens)))), block_tables={}, logit_rows=None, n_logit_rows=0, page_size=PAGE, runtime=rt,
                      max_kv_len=max(lens), max_q_len=max(lens))
    state = dict(kind=case["kind"], part=part, ctx=ctx, x=_rows(case, seed))
    if registry is MIXERS:
        cache = LayerCache(page_size=PAGE)
        if part.kv_cache_spec() is not None:
            width = -(-max(lens) // PAGE)
            pages = len(lens) * width
            cache.block_table = torch.randperm(pages, generator=_generator(seed, "pages"), device=DEV).to(torch.int32).view(len(lens), width)
            cache.arrays = {a.name: torch.zeros((pages,) + tuple(a.shape[:-1]) + (PAGE, a.shape[-1]), dtype=torch.bfloat16, device=DEV)
                            for a in part.kv_cache_spec().token_arrays()}
        if part.state_spec() is not None:
            cache.state = torch.zeros((len(lens),) + tuple(part.state_spec().shape), dtype=torch.float32, device=DEV)
        state["cache"] = cache
    return state


def _prepare_step(case, seed):
    spec = _decoder(case)
    model = Model(spec, _decoder_weights(spec, seed, _dtype(case)), make_runtime(case["dtype"]))
    decode = case["kind"] == "decode"
    batch, held = (case["batch"], case["context"]) if decode else (1, case["tokens"])
    engine = Engine(model, page_size=PAGE, cache_tokens=batch * (held + 2 * PAGE), max_context=held + 1, token_budget=batch * held, max_active=batch + 1)
    ids = _tokens(seed, "tokens", (batch, held + 1), spec.vocab_size).tolist()
    state = dict(kind=case["kind"], runner=engine.runner, engine=engine)
    if not decode:
        state["prompt"] = ids[0][:held]
        return state
    for i in range(batch):          # the contexts, a few requests to a step
        engine.runner.add_request(i)
    per = max(1, 8192 // held)
    for at in range(0, batch, per):
        engine.runner.step([StepEntry(i, ids[i][:held]) for i in range(at, min(batch, at + per))])
    for i in range(batch):
        engine.runner.manager.reserve(i, held + 1)
    state["entries"] = [StepEntry(i, ids[i][held:], [0]) for i in range(batch)]
    return state


def run(state):
    kind = state["kind"]
    if kind == "decode":            # one step over the batch, whose pages a scheduler has reserved: logits of every request
        return state["runner"].execute(state["entries"])
    if kind == "prompt":            # a request comes, its prompt is one step, its last token's logits are read
        runner, toks = state["runner"], state["prompt"]
        runner.add_request("prompt")
        logits = runner.step([StepEntry("prompt", toks, [len(toks) - 1])])
        runner.release("prompt")
        return logits
    if kind == "sample":
        return ops.sample_rows(*state["args"])
    if kind == "experts":
        return state["part"].forward(state["x"], state["ctx"])
    cache = state["cache"]
    y = state["part"].forward(state["x"], state["ctx"], cache)
    return y if cache.state is None else (y, cache.state)


# ---- what a pass cannot do without ---------------------------------------------------------------------------------------
def _seen(lens, window):
    """Query-key pairs of causal attention over whole prompts."""
    w = window or max(lens)
    return sum(min(n, w) * (min(n, w) + 1) // 2 + max(0, n - w) * w for n in lens)


def work(case):
    kind = case["kind"]
    if kind in STEPS:
        z, size = SHAPES[case["shape"]], 4 if case["dtype"] == "float32" else 2
        d, F, V = z["hidden_size"], z["intermediate_size"], z["vocab_size"]
        qs, kvs = z["num_attention_heads"] * z["head_dim"], z["num_key_value_heads"] * z["head_dim"]
        layer = d * (qs + 2 * kvs) + qs * d + 3 * d * F
        if kind == "decode":
            n, rows, pairs, held = case["batch"], case["batch"], case["batch"] * (case["context"] + 1), case["batch"] * case["context"]
        else:
            n, rows, pairs, held = case["tokens"], 1, _seen([case["tokens"]], 0), 0
        return {"bytes": size * (LAYERS * (layer + 2 * kvs * (held + n)) + V * d + n * d) + 4 * rows * V,
                "flops": 2 * (LAYERS * (n * layer + 2 * pairs * qs) + rows * V * d)}
    if kind == "sample":
        return {"bytes": 4 * case["rows"] * case["vocab"], "flops": 0}
    z, n = SIZES[case["size"]], case["tokens"]
    d, H, G, dk, dv = z["width"], z["heads"], z["kv_heads"], z["dim"], z["vdim"]
    rows = 2 * 2 * n * d
    if kind == "experts":
        ff = -(-(2 * z["ff"] // 12) // 64) * 64
        return {"bytes": 2 * 16 * 3 * ff * d + rows, "flops": 2 * n * (4 * 3 * ff * d + 16 * d)}
    lens = _lengths(case)
    if kind == "sink":
        weights, math_ = d * (H * dk + G * (dk + dv) + H * dv), _seen(lens, z["window"]) * H * (dk + dv)
        kept = 2 * n * G * (dk + dv)
    elif kind == "differential":
        weights, math_ = d * (H * dk + G * 2 * dk + H + H * dk), _seen(lens, z["window"]) * H * 2 * (dk // 2 + dk)
        kept = 2 * n * G * 2 * dk
    else:               # the recurrence as it is written: a multiply-add into and one out of every number of the state, with the delta rule two
        q, v, gate = {"delta": (G, dk, 2), "retention": (H, dk, 1), "forget": (H, dv, 0)}[kind]
        weights = d * (2 * q * dk + 2 * H * v + (H * v if gate else 0) + (2 * H if kind == "delta" else 0))
        math_ = n * H * dk * v * (3 if kind == "delta" else 2)
        kept = 4 * len(lens) * H * dk * v
    return {"bytes": 2 * weights + rows + kept, "flops": 2 * (n * weights + math_)}


def tolerance(case):
    kind = case["kind"]
    if kind == "sample":
        return "exact"                      # tokens
    if case.get("dtype") == "float32":
        return {"rel": 1e-5}                # sums of 32-bit products over up to 4,864 terms, two layers deep
    if kind in STEPS:
        return {"rel": 2.5e-2}              # 16-bit roundings through two layers
    if kind == "differential":
        return {"rel": 2e-2}                # a difference of two maps, brought to unit size
    return {"rel": 1e-2}                    # one layer in 16 bits


# ---- the same in 64 bits -------------------------------------------------------------------------------------------------
def _rms(x, eps=1e-6):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def _turned(x, angles, pairs):
    """x [n, heads, dim] with its pairs of numbers turned: ``pairs`` "half" (i, i + dim/2) or "next" (2i, 2i + 1)."""
    c, s = torch.cos(angles)[:, None], torch.sin(angles)[:, None]
    if pairs == "half":
        a, b = x.chunk(2, dim=-1)
        return torch.cat([a * c - b * s, b * c + a * s], dim=-1)
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * c - b * s, b * c + a * s], dim=-1).flatten(-2)


def _angles(n, dim, base):
    freq = base ** (-2.0 * torch.arange(dim // 2, dtype=torch.float64, device=DEV) / dim)
    return torch.arange(n, dtype=torch.float64, device=DEV)[:, None] * freq


def _attend(q, k, v, scale, window=0, sink=0.0, cap=0.0, last=None):
    """Causal attention of one sequence, a head at a time; ``last``: only the last so many queries."""
    n, H = q.shape[0], q.shape[1]
    m = last or n
    at = torch.arange(n - m, n, device=DEV)[:, None]
    key = torch.arange(n, device=DEV)[None]
    hidden = (key > at) | ((at - key >= window) if window else False)
    out = []
    for h in range(H):
        s = q[n - m:, h] @ k[:, h * k.shape[1] // H].T * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill_(hidden, -math.inf)
        top = s.amax(dim=-1, keepdim=True).clamp_min_(0.0 if sink else -math.inf)
        p = torch.exp(s - top)
        out.append(p @ v[:, h * v.shape[1] // H] / (p.sum(dim=-1, keepdim=True) + sink * torch.exp(-top)))
    return torch.stack(out, dim=1)


def _exact_step(case, seed):
    spec, z = _decoder(case), SHAPES[case["shape"]]
    w = _decoder_weights(spec, seed, _dtype(case))
    H, G, hd = z["num_attention_heads"], z["num_key_value_heads"], z["head_dim"]
    decode = case["kind"] == "decode"
    batch, n = (case["batch"], case["context"] + 1) if decode else (1, case["tokens"])
    if batch * n * sum(t.numel() for t in w.values()) > 1.2e14:
        return None                         # over the time that a check may take
    ids = _tokens(seed, "tokens", (batch, n if decode else n + 1), spec.vocab_size)[:, :n]
    table, rows = w["model.embed_tokens.weight"], []
    angles = _angles(n, hd, 1000000.0)
    xs = [table[ids[b]].double() for b in range(batch)]
    for i in range(LAYERS):
        at = f"model.layers.{i}."
        t = {k[len(at):]: v.double() for k, v in w.items() if k.startswith(at)}
        last = 1 if i == LAYERS - 1 else None        # of the last layer only the wanted token goes on
        for b in range(batch):
            h = _rms(xs[b]) * t["input_layernorm.weight"]
            q, k, v = (torch.addmm(t[f"self_attn.{c}_proj.bias"], h, t[f"self_attn.{c}_proj.weight"].T).view(n, -1, hd) for c in "qkv")
            o = _attend(_turned(q, angles, "half"), _turned(k, angles, "half"), v, hd ** -0.5, last=last)
            x = xs[b][-1:] if last else xs[b]
            x = x + o.flatten(1) @ t["self_attn.o_proj.weight"].T
            h = _rms(x) * t["post_attention_layernorm.weight"]
            gate = h @ t["mlp.gate_proj.weight"].T
            xs[b] = x + (torch.nn.functional.silu(gate) * (h @ t["mlp.up_proj.weight"].T)) @ t["mlp.down_proj.weight"].T
        del t
    head = table if z["tie_word_embeddings"] else w["lm_head.weight"]
    for x in xs:
        rows.append(_rms(x[-1:]) * w["model.norm.weight"].double())
    rows = torch.cat(rows)
    return torch.cat([rows @ part.double().T for part in head.split(16384)], dim=1)


def _conv(x, taps):
    """A causal convolution over the tokens per channel, the last tap on the token itself."""
    K = taps.shape[1]
    padded = torch.cat([x.new_zeros(K - 1, x.shape[1]), x])
    return sum(padded[j:j + x.shape[0]] * taps[:, j] for j in range(K))


def _exact_mixer(case, seed):
    _, spec = _layer(case)
    w = {n: t.double() for n, t in _layer_weights(MIXERS, spec, seed).items()}
    x, z, kind = _rows(case, seed).double(), SIZES[case["size"]], case["kind"]
    G, H, lens, outs, states = z["kv_heads"], z["heads"], _lengths(case), [], []
    silu = torch.nn.functional.silu
    for h in x.split(lens):
        n = h.shape[0]
        proj = lambda name, heads: (h @ w[spec[name]].T).view(n, heads, -1)        # noqa: E731
        if kind == "sink":
            dk, dv = spec["key_dim"], spec["value_dim"]
            biased = lambda name, heads: proj(name, heads) + w[spec[name] + ".b"].view(heads, -1)    # noqa: E731
            ang = _angles(n, dk, 10000.0)
            o = _attend(_turned(biased("q", H), ang, "next"), _turned(biased("k", G), ang, "next"), biased("v", G), spec["scale"], z["window"], sink=1.0)
            outs.append(o.flatten(1) @ w[spec["o"]].T + w[spec["o"] + ".b"])
            continue
        if kind == "differential":
            dk, raw = spec["key_dim"], {c: h @ w[spec[c]].T + w[spec[c] + spec["bias_suffix"]] for c in "qkv"}
            q, k, v = (_conv(raw[c], w[spec[c] + spec["conv_suffix"]]) for c in "qkv")
            q, k, v = q.view(n, H, 2, dk), k.view(n, G, 2, dk), v.view(n, G, -1)
            lam = torch.exp((w[spec["lq1"]] * w[spec["lk1"]]).sum()) - torch.exp((w[spec["lq2"]] * w[spec["lk2"]]).sum()) + spec["diff"]
            a, b = (_attend(q[:, :, m], k[:, :, m], v, spec["scale"], z["window"], cap=spec["softcap"]) for m in (0, 1))
            o = _rms(a - lam * b, spec["eps"]) * (1.0 - spec["diff"])
            if spec.get("g"):
                o = o * torch.sigmoid(h @ w[spec["g"]].T)[:, :, None]
            outs.append(o.flatten(1) @ w[spec["o"]].T)
            # the convolution's last inputs, the newest first, by channel: the first maps of all heads before the second ones
            tail = torch.cat([raw["q"].view(n, H, 2, dk).transpose(1, 2).flatten(1), raw["k"].view(n, G, 2, dk).transpose(1, 2).flatten(1), raw["v"]], dim=1)
            states.append(tail[-3:].flip(0).flatten())
            continue
        qh = spec["qk_heads"]
        q, k, v, tail = proj("q", qh), proj("k", qh), proj("v", H), []
        f = beta = None
        if kind == "delta":
            flat = [t.flatten(1) for t in (q, k, v)]
            tail = [torch.cat(flat, dim=1)[-3:].flip(0).flatten()]
            q, k, v = (silu(_conv(t, w[spec[c] + ".conv"])).view(n, heads, -1) for c, t, heads in zip("qkv", flat, (qh, qh, H)))
            q, k = (t / torch.sqrt((t * t).sum(dim=-1, keepdim=True) + spec["unit_eps"]) for t in (q, k))
            q = q * spec["q_scale"]
            f = torch.exp(-torch.exp(w[spec["A_log"]]) * torch.nn.functional.softplus(h @ w[spec["a"]].T + w[spec["dt_bias"]]))[..., None, None]
            beta = torch.sigmoid(h @ w[spec["delta"]].T)[..., None]
        elif kind == "retention":
            ang = _angles(n, spec["key_dim"], 10000.0)
            q, k = _turned(q, ang, "half"), _turned(k, ang, "half") * spec["k_scale"]
            f = torch.tensor(spec["decay"], dtype=torch.float32, device=DEV).double()[None, :, None, None].expand(n, -1, -1, -1)
        else:
            low = w[spec["lower"]].view(H, -1)
            gate = low + (1.0 - low) * torch.sigmoid(k + w[spec["f_bias"]].view(H, -1))
            q, k, f = silu(q), 1.0 - gate, gate[..., None]
        q, k = q.repeat_interleave(H // qh, dim=1), k.repeat_interleave(H // qh, dim=1)
        S, o = h.new_zeros(H, k.shape[2], v.shape[2]), torch.empty_like(v)
        for t in range(n):
            S = S * f[t]
            u = v[t] if beta is None else beta[t] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
            S = torch.baddbmm(S, k[t][:, :, None], u[:, None])
            o[t] = torch.bmm(q[t][:, None], S)[:, 0]
        o = _rms(o, spec["eps"])
        if spec.get("out_weight"):
            o = o * w[spec["out_weight"]]
        o = o.flatten(1)
        if spec.get("g"):
            o = o * silu(h @ w[spec["g"]].T)
        outs.append(o @ w[spec["o"]].T)
        states.append(torch.cat([S.transpose(1, 2).flatten()] + tail))
    y = torch.cat(outs)
    return (y, torch.stack(states)) if states else y


def _exact_experts(case, seed):
    registry, spec = _layer(case)
    w, x = _layer_weights(registry, spec, seed), _rows(case, seed).double()
    score = torch.softmax(x @ w[spec["router"]].double().T, dim=-1)
    n, E = score.shape
    runs = score.view(n, spec["groups"], -1).amax(dim=-1)
    kept = torch.zeros_like(runs).scatter_(1, runs.topk(spec["keep"], dim=1).indices, 1.0)
    best, chosen = (score * kept.repeat_interleave(E // spec["groups"], dim=1)).topk(spec["top"], dim=1)
    best = best / best.sum(dim=1, keepdim=True)
    y = torch.zeros_like(x)
    for e in range(E):
        rows, place = torch.nonzero(chosen == e, as_tuple=True)
        gate, up, down = (w[spec["expert"].format(e) + s].double() for s in (".gate", ".up", ".down"))
        h = x[rows]
        y.index_add_(0, rows, best[rows, place][:, None] * ((torch.nn.functional.silu(h @ gate.T) * (h @ up.T)) @ down.T))
    return y


def exact(case, seed):
    if case["kind"] in STEPS:
        return _exact_step(case, seed)
    if case["kind"] == "sample":
        return None
    return _exact_experts(case, seed) if case["kind"] == "experts" else _exact_mixer(case, seed)
