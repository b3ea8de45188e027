"""Kernels of single layers where their forms change hands: prompt attention with unequal key and value sizes against the mma.sync kernel,
the convolution's runs, norms by groups, the lists and sums of routed experts."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("dk,dv", [(128, 64), (64, 128), (64, 64), (128, 128)])
@pytest.mark.parametrize("what", ["plain", "cap", "hard cap", "logits", "shared values", "fp32", "window", "kept"])
def test_prompt_attention_on_tensor_memory(dk, dv, what, monkeypatch):
    from mimirmind_b200.kernels import attention
    from mimirmind_b200.kernels import ops
    from mimirmind_b200.parts.base import LayerCache, StepContext
    gen = torch.Generator(device=DEV).manual_seed(dk + dv + len(what))
    rnd = lambda *s: torch.randn(s, generator=gen, device=DEV).to(torch.bfloat16)     # noqa: E731
    H, G, page = 8, 4, 16
    Gv = 2 if what == "shared values" else G
    lens, begin = [300, 16, 129], [0, 100, 3]
    kv = [b + n for b, n in zip(begin, lens)]
    n, width = sum(lens), -(-max(kv) // page)
    starts = [0, 300, 316]
    cache = LayerCache(page_size=page, block_table=torch.randperm(3 * width, generator=gen, device=DEV).to(torch.int32).view(3, width),
                       arrays={"k": rnd(3 * width, G, page, dk), "v": rnd(3 * width, Gv, page, dv)})
    q = rnd(n, H * dk)
    options = {"cap": dict(softcap=30.0), "hard cap": dict(softcap=0.7), "logits": dict(sink_logit=torch.linspace(-3, 3, H, device=DEV)),
               "shared values": dict(value_heads=Gv), "window": dict(), "kept": dict(keep=5, chunk=64)}.get(what, {})
    outs = []
    for tensor_memory in (True, False):
        monkeypatch.setattr(attention, "USE_SINK_TCGEN05", tensor_memory)
        pos = torch.cat([torch.arange(b, b + m, dtype=torch.int32, device=DEV) for b, m in zip(begin, lens)])
        ctx = StepContext(n_tokens=n, n_requests=3, token_ids=None, positions=pos, token_req=i32(sum(([r] * m for r, m in enumerate(lens)), [])),
                          q_start=starts, q_len=lens, kv_len=kv, req_meta=None, state_slots=None, block_tables={}, logit_rows=None, n_logit_rows=0,
                          page_size=page, runtime=None, max_kv_len=max(kv), max_q_len=max(lens))
        out = torch.full((n, H * dv), float("nan"), dtype=torch.float32 if what == "fp32" else torch.bfloat16, device=DEV)
        attention.paged_sink_attention(q, cache, out, ctx, H, G, dk, dv, 70 if what == "window" else 0, dk ** -0.5, what != "plain", **options)
        outs.append(out.float())
    ops.check_tcgen05_errors(torch.device(DEV))
    a, b = outs
    # both round the weights to bf16 (2^-9 each, relative to another reference) and, but for fp32, the result
    assert ((a - b).norm() / b.norm()).item() <= 2.0 ** -7 and (a - b).abs().max() <= 2.0 ** -5 * b.abs().max()


@pytest.mark.parametrize("lens,tall", [([64], True), ([63], False), ([1, 1], True), ([20, 300], True), ([20] * 4 + [300], False), ([128, 15], True)])
def test_short_portions_stay_in_short_tiles(lens, tall):
    from types import SimpleNamespace

    from mimirmind_b200.kernels.attention import fills_tall_tiles
    assert fills_tall_tiles(SimpleNamespace(q_len=lens, plans={})) is tall


@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("n,d,ff,E,top", [(17, 64, 40, 6, 2), (100, 200, 136, 3, 3), (33, 2048, 256, 40, 8), (255, 72, 264, 5, 4)])
def test_grouped_products_of_small_steps_stay_in_32_bits(n, d, ff, E, top, gated, monkeypatch):
    from mimirmind_b200.config.spec import PartSpec
    from mimirmind_b200.kernels import ops
    from mimirmind_b200.parts import moe
    from mimirmind_b200.parts.base import Runtime, WeightView
    gen = torch.Generator(device=DEV).manual_seed(n + d)
    rnd = lambda *s: torch.randn(s, generator=gen, device=DEV)                       # noqa: E731
    w = {"router": rnd(E, d) * 4 * d ** -0.5}
    for e in range(E):
        w.update({f"e{e}.gate": rnd(ff, d) * d ** -0.5, f"e{e}.up": rnd(ff, d) * d ** -0.5, f"e{e}.down": rnd(d, ff) * ff ** -0.5})
    spec = PartSpec("routed_experts", {"hidden": d, "ff": ff, "experts": E, "top": top, "router": "router", "expert": "e{}", "gated": gated,
                                       "activation": "silu" if gated else "gelu_erf"})
    part = moe.RoutedExperts(spec, WeightView({k: v.to(torch.bfloat16) for k, v in w.items()}), Runtime(torch.bfloat16, torch.device(DEV)))
    x = rnd(n, d).to(torch.bfloat16)
    got = {}
    for least in (0, 1 << 40):
        monkeypatch.setattr(moe, "GROUPED_MIN_WEIGHTS", least)
        split, whole = part.forward_split(x, None), part.forward(x, None)
        assert split.rows.dtype == torch.float32 and (split.place is None) == (least > 0)
        y = split.rows if split.place is None else split.rows[split.place.long()]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            replayed = part.forward(x, None)
        graph.replay()
        assert torch.equal(replayed, whole)
        assert torch.equal(whole, ops.moe_combine(split.rows, split.weights, torch.bfloat16, place=split.place, top=top))
        got[least] = y
    ops.check_tcgen05_errors(torch.device(DEV))
    # the hidden rows are rounded to bf16 on both sides, mostly alike: 2^-9 each at most
    assert ((got[0] - got[1 << 40]).norm() / got[1 << 40].norm()).item() <= 2.0 ** -8


@pytest.mark.parametrize("taps", [1, 2, 4, 8])
@pytest.mark.parametrize("C", [128, 260])
def test_convolution_in_runs_of_tokens(taps, C):
    """Runs that start, end or lie inside a portion, with and without earlier inputs; the same bits as the walk's."""
    from mimirmind_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(taps + C)
    lens, begin, slots = [37, 1, 3, 64, 7], [0, 9, 0, 20, 50], [1, 0, 4, 2, 5]
    n, starts = sum(lens), [sum(lens[:i]) for i in range(5)]
    x = torch.randn((n, C + 8), generator=gen, device=DEV)
    w = torch.randn((C, taps), generator=gen, device=DEV)
    tail = torch.randn((6, max(1, (taps - 1) * C)), generator=gen, device=DEV)
    pos = torch.cat([torch.arange(b, b + m, dtype=torch.int32, device=DEV) for b, m in zip(begin, lens)])
    meta = i32([[s, m, b + m, sl] for s, m, b, sl in zip(starts, lens, begin, slots)])
    walked, tail2 = x.clone(), tail.clone()
    y = ops.causal_conv_tokens(x, C, w, tail, i32(sum(([r] * m for r, m in enumerate(lens)), [])), meta, i32(slots), pos, 5, silu=True)
    ops.causal_conv_walk(walked, C, w, tail2, meta, i32(slots), pos, 5, silu=True)
    assert torch.equal(y, walked[:, :C]) and torch.equal(tail, tail2)


@pytest.mark.parametrize("groups,gs", [(5, 16), (3, 64), (4, 100), (2, 128), (3, 200), (2, 512), (3, 516), (7, 10)])
@pytest.mark.parametrize("kind", ["fp32", "bf16", "no norm"])
def test_norm_by_groups(groups, gs, kind):
    from mimirmind_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(groups * gs)
    dt = torch.bfloat16 if kind == "bf16" else torch.float32
    rows = torch.randn((33, groups * gs + 4), generator=gen, device=DEV).to(dt)
    gate = torch.randn((33, groups * gs + 8), generator=gen, device=DEV)[:, 4:4 + groups * gs]
    w = torch.randn(gs, generator=gen, device=DEV)
    x = rows[:, :groups * gs]
    y = ops.gated_group_norm(x, groups, gs, dt, eps=1e-5, normalize=kind != "no norm", weight=w, gate=gate, activation="silu")
    xx = x.double().view(33, groups, gs)
    inv = 1.0 if kind == "no norm" else 1.0 / torch.sqrt((xx * xx).mean(-1, keepdim=True) + 1e-5)
    want = (xx * inv * w.double()).reshape(33, -1) * torch.nn.functional.silu(gate.double())
    # 32 bits: a sum of up to 516 squares and four factors; bf16: the result's rounding
    assert (y.double() - want).abs().max() <= (2.0 ** -8 if dt == torch.bfloat16 else 4e-6) * want.abs().max()


@pytest.mark.parametrize("E", [1, 7, 16, 33, 300])
@pytest.mark.parametrize("n,top", [(1, 1), (31, 2), (257, 1), (700, 4), (8193, 2)])
def test_rows_by_expert(E, n, top):
    from mimirmind_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(E + n)
    idx = (torch.rand((n, top), generator=gen, device=DEV) ** 2 * E).to(torch.int32).clamp_(max=E - 1)      # uneven, some experts empty
    rows = ops.moe_sort(idx, E, with_tiles=True)
    want = torch.sort(idx.flatten(), stable=True).indices.to(torch.int32)
    assert torch.equal(rows.order, want) and torch.equal(rows.row_token, (want // top).to(torch.int32))
    assert torch.equal(rows.place[want.long()], torch.arange(n * top, dtype=torch.int32, device=DEV))
    counts = torch.bincount(idx.flatten().long(), minlength=E).tolist()
    offsets, tiles = [0], []
    for e, c in enumerate(counts):
        tiles += [[offsets[-1] + lo, offsets[-1] + min(lo + 128, c), e] for lo in range(0, c, 128)]
        offsets.append(offsets[-1] + c)
    assert rows.offsets.tolist() == offsets
    assert rows.n_tiles.item() == len(tiles) and rows.tiles.view(-1, 3)[:len(tiles)].tolist() == tiles


@pytest.mark.parametrize("d", [8, 100, 2048, 2056, 5000])
@pytest.mark.parametrize("top", [1, 4, 6])
@pytest.mark.parametrize("weighed", [True, False])
def test_weighted_sum_of_experts(d, top, weighed):
    from mimirmind_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(d + top)
    n = 19
    y = torch.randn((n * top, d), generator=gen, device=DEV).to(torch.bfloat16)
    w = torch.rand((n, top), generator=gen, device=DEV) if weighed else None
    place = torch.randperm(n * top, generator=gen, device=DEV).to(torch.int32)
    got = ops.moe_combine(y, w, torch.bfloat16, place=place, top=top)
    rows = y[place.long()].double().view(n, top, d)
    want = (rows * (w.double()[:, :, None] if weighed else 1.0)).sum(1)
    assert (got.double() - want).abs().max() <= 2.0 ** -8 * want.abs().max()


@pytest.mark.parametrize("dk", [64, 128, 72])
@pytest.mark.parametrize("Gq", [1, 3, 40])
@pytest.mark.parametrize("rot,act,unit", [(True, False, False), (False, True, True), (True, True, True)])
def test_preparation_of_a_matrix_state(dk, Gq, rot, act, unit):
    from mimirmind_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(dk + Gq)
    n, H, n_v = 5, 6, 36
    q_off, k_off, v_off = 4, 4 + Gq * dk, 4 + 2 * Gq * dk
    a_off, b_off = v_off + n_v, v_off + n_v + H
    x = torch.randn((n, b_off + H + 4), generator=gen, device=DEV)
    before = x.double()
    angles = torch.randn((n, dk // 2), generator=gen, device=DEV) * 3
    table = torch.stack([angles.cos(), angles.sin()], dim=-1).contiguous()
    A, dt = torch.randn(H, generator=gen, device=DEV), torch.randn(H, generator=gen, device=DEV)
    gate, beta = ops.linear_state_prep(x, q_off, k_off, v_off, Gq, dk, n_v, silu=act, rot=table if rot else None, rot_dims=dk if rot else 0, unit=unit,
                                       unit_eps=1e-6, q_scale=0.3, k_scale=2.0, a_off=a_off, b_off=b_off, heads=H, A_log=A, dt_bias=dt)
    f = torch.nn.functional.silu if act else (lambda t: t)
    want = before.clone()
    for off, scale in ((q_off, 0.3), (k_off, 2.0)):
        y = f(before[:, off:off + Gq * dk]).view(n, Gq, dk)
        if rot:
            a, b = y.chunk(2, dim=-1)
            c, s = table[:, None, :, 0].double(), table[:, None, :, 1].double()
            y = torch.cat([a * c - b * s, b * c + a * s], dim=-1)
        if unit:
            y = y / torch.sqrt((y * y).sum(-1, keepdim=True) + 1e-6)
        want[:, off:off + Gq * dk] = (y * scale).reshape(n, -1)
    want[:, v_off:v_off + n_v] = f(before[:, v_off:v_off + n_v])
    # a dozen roundings of 2^-24 on numbers up to the largest
    assert (x - want).abs().max() <= 2e-6 * want.abs().max()
    assert torch.allclose(gate.double(), torch.exp(-A.double().exp() * torch.nn.functional.softplus(before[:, a_off:a_off + H] + dt.double())), rtol=3e-6, atol=1e-7)
    assert torch.allclose(beta.double(), torch.sigmoid(before[:, b_off:b_off + H]), rtol=1e-6, atol=1e-7)


@pytest.mark.parametrize("dk,dv", [(64, 128), (128, 64), (36, 20), (10, 6)])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_rows_cut_into_queries_keys_and_values(dk, dv, dt):
    from mimirmind_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(dk)
    n, Hq, Gk, Gv, page = 21, 12, 4, 2, 8
    x = torch.randn((n, Hq * dk + Gk * dk + Gv * dv + 4), generator=gen, device=DEV)
    q_off, k_off, v_off = 4, 4 + Hq * dk, 4 + (Hq + Gk) * dk
    slots = torch.randperm(64, generator=gen, device=DEV)[:n].to(torch.int32)
    slots[3] = -1
    q = torch.empty((n, Hq * dk), dtype=dt, device=DEV)
    k, v = torch.zeros((8, Gk, page, dk), dtype=dt, device=DEV), torch.zeros((8, Gv, page, dv), dtype=dt, device=DEV)
    ops.qkv_split_post(x, q_off, k_off, v_off, q, k, v, slots, page, Hq, Gk, dk, Gv, dv)
    assert torch.equal(q, x[:, q_off:k_off].to(dt))
    wk, wv = torch.zeros_like(k), torch.zeros_like(v)
    for t, s in enumerate(slots.tolist()):
        if s >= 0:
            wk[s // page, :, s % page] = x[t, k_off:v_off].to(dt).view(Gk, dk)
            wv[s // page, :, s % page] = x[t, v_off:v_off + Gv * dv].to(dt).view(Gv, dv)
    assert torch.equal(k, wk) and torch.equal(v, wv)


@pytest.mark.parametrize("dv", [64, 128, 256, 96])
@pytest.mark.parametrize("pair,gated,out", [(True, True, torch.bfloat16), (False, False, torch.float32), (True, False, torch.float32)])
def test_heads_finished(dv, pair, gated, out):
    from mimirmind_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(dv)
    n, H = 13, 5
    att = torch.randn((n, (2 if pair else 1) * H * dv), generator=gen, device=DEV)
    gate = torch.randn((n, H + 3), generator=gen, device=DEV)[:, 1:1 + H] if gated else None
    got = ops.head_finish(att, H, dv, pair=pair, lam=0.37, eps=1e-5, post=0.5, gate=gate, out_dtype=out)
    x = att.double().view(n, -1, dv)
    o = x[:, :H] - (0.37 * x[:, H:] if pair else 0.0)
    o = 0.5 * o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-5)
    if gated:
        o = o * torch.sigmoid(gate.double())[:, :, None]
    assert (got.double() - o.reshape(n, -1)).abs().max() <= (2.0 ** -8 if out == torch.bfloat16 else 3e-6) * o.abs().max()
