"""Prompt attention on tensor memory sees what its rows see and nothing else: what stands in the pages behind a request's last token and in front of
its window may be NaN, and neither that nor the other requests of the step change a bit of the result."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
H, G, PAGE = 8, 4, 16
LENS, BEGIN = [300, 16, 129], [0, 100, 3]
FORMS = {"plain": {}, "sink": {}, "cap": dict(softcap=30.0), "hard cap": dict(softcap=0.7), "logits": {}, "shared values": dict(value_heads=2), "fp32": {},
         "capped fp32": dict(softcap=20.0), "window": {}, "capped window": dict(softcap=20.0), "kept": dict(keep=5, chunk=64)}


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def attend(q, k, v, table, dk, dv, form, lens=LENS, begin=BEGIN, sink=None):
    from mimirmind_b200.kernels import attention, ops
    from mimirmind_b200.parts.base import LayerCache, StepContext
    n, kv = sum(lens), [b + m for b, m in zip(begin, lens)]
    starts = [sum(lens[:r]) for r in range(len(lens))]
    pos = torch.cat([torch.arange(b, b + m, dtype=torch.int32, device=DEV) for b, m in zip(begin, lens)])
    ctx = StepContext(n_tokens=n, n_requests=len(lens), token_ids=None, positions=pos, token_req=i32(sum(([r] * m for r, m in enumerate(lens)), [])),
                      q_start=starts, q_len=lens, kv_len=kv, req_meta=None, state_slots=None, block_tables={}, logit_rows=None, n_logit_rows=0,
                      page_size=PAGE, runtime=None, max_kv_len=max(kv), max_q_len=max(lens))
    assert attention.fills_tall_tiles(ctx)
    wide = "fp32" in form or "cap" in form
    out = torch.full((n, H * dv), float("nan"), dtype=torch.float32 if wide else torch.bfloat16, device=DEV)
    more = dict(FORMS[form])
    if form == "logits":
        more["sink_logit"] = torch.linspace(-3, 3, H, device=DEV)
    attention.paged_sink_attention(q, LayerCache(page_size=PAGE, block_table=table, arrays={"k": k, "v": v}), out, ctx, H, G, dk, dv,
                                   70 if "window" in form else 0, dk ** -0.5, form != "plain" if sink is None else sink, **more)
    ops.check_tcgen05_errors(torch.device(DEV))
    return out


def setting(dk, dv, form, seed=0):
    gen = torch.Generator(device=DEV).manual_seed(dk + 3 * dv + len(form) + seed)
    rnd = lambda *s: torch.randn(s, generator=gen, device=DEV).to(torch.bfloat16)     # noqa: E731
    width = -(-max(b + m for b, m in zip(BEGIN, LENS)) // PAGE) + 1
    table = torch.randperm(len(LENS) * width, generator=gen, device=DEV).to(torch.int32).view(len(LENS), width)
    return rnd(sum(LENS), H * dk), rnd(len(LENS) * width, G, PAGE, dk), rnd(len(LENS) * width, 2 if form == "shared values" else G, PAGE, dv), table


def unseen(form):
    """(request, token) of the slots in the requests' pages that none of their rows sees."""
    for r, (b, m) in enumerate(zip(BEGIN, LENS)):
        low = max(0, b + 1 - 70) if "window" in form else b // 64 * 64 if form == "kept" else 0
        for j in list(range(5 if form == "kept" else 0, low)) + list(range(b + m, -(-(b + m) // PAGE) * PAGE + PAGE)):
            yield r, j


@pytest.mark.parametrize("dk,dv", [(128, 64), (64, 128), (64, 64), (128, 128)])
@pytest.mark.parametrize("form", list(FORMS))
def test_what_no_row_sees_does_not_count(dk, dv, form):
    q, k, v, table = setting(dk, dv, form)
    clean = attend(q, k, v, table, dk, dv, form)
    assert torch.isfinite(clean).all()
    for junk in (float("nan"), float("inf"), 200.0):          # what an earlier owner of the pages may have left there
        kk, vv = k.clone(), v.clone()
        for r, j in unseen(form):
            kk[table[r, j // PAGE], :, j % PAGE] = junk
            vv[table[r, j // PAGE], :, j % PAGE] = junk
        assert torch.equal(attend(q, kk, vv, table, dk, dv, form), clean)


@pytest.mark.parametrize("dk,dv", [(128, 64), (64, 128), (64, 64)])
@pytest.mark.parametrize("form", ["cap", "hard cap", "capped window", "fp32"])
def test_other_requests_of_the_step_do_not_count(dk, dv, form):
    """Scores on both sides of 0.35 of the cap: the form that a score takes is its own."""
    q, k, v, table = setting(dk, dv, form)
    together = attend(q, k, v, table, dk, dv, form)
    loud = q.clone()
    loud[316:] *= 100                                          # the request behind, some of whose rows stand in the tile of the one before
    assert torch.equal(attend(loud, k, v, table, dk, dv, form)[:316], together[:316])
    for r, (b, m) in enumerate(zip(BEGIN, LENS)):
        s = sum(LENS[:r])
        if m >= 64:
            alone = attend(q[s:s + m].contiguous(), k, v, table[r:r + 1].contiguous(), dk, dv, form, lens=[m], begin=[b])
            assert torch.equal(alone, together[s:s + m])


@pytest.mark.parametrize("cap,spread", [(0.7, 1.0), (5.0, 3.0), (30.0, 1.0), (30.0, 12.0)])
def test_capped_scores_against_64_bits(cap, spread):
    """One request in one tile per head; the weights are rounded to bf16 once, the rest is 32-bit work on scores of at most ``cap``."""
    dk, dv, n = 64, 64, 128
    gen = torch.Generator(device=DEV).manual_seed(int(10 * cap))
    q = (spread * torch.randn((n, H * dk), generator=gen, device=DEV)).to(torch.bfloat16)
    k, v = (torch.randn((n // PAGE, G, PAGE, d), generator=gen, device=DEV).to(torch.bfloat16) for d in (dk, dv))
    FORMS["one"] = dict(softcap=cap)
    table = torch.arange(n // PAGE, dtype=torch.int32, device=DEV).view(1, -1)
    try:
        out = attend(q, k, v, table, dk, dv, "one", lens=[n], begin=[0], sink=False)
    finally:
        del FORMS["one"]
    kk, vv = (t.transpose(1, 2).reshape(n, G, -1).double().repeat_interleave(H // G, dim=1) for t in (k, v))
    s = cap * torch.tanh(torch.einsum("nhd,mhd->hnm", q.view(n, H, dk).double(), kk) * dk ** -0.5 / cap)
    p = torch.softmax(s.masked_fill(torch.ones(n, n, device=DEV).triu(1).bool(), float("-inf")), dim=-1)
    want, size = torch.einsum("hnm,mhd->nhd", p, vv).flatten(1), torch.einsum("hnm,mhd->nhd", p, vv.abs()).flatten(1)
    # every weight within 2^-9 (its rounding) and what its score is off in the exponent: a sum of 64 products, each addition within 2^-23 of the sum of
    # their sizes (the tensor core cuts off), and tanh within 2^-23 of the cap; the division by the sum at most as much; bf16 at the end
    sizes = torch.einsum("nhd,mhd->hnm", q.view(n, H, dk).double().abs(), kk.abs()).amax() * dk ** -0.5
    score = 64 * 2.0 ** -23 * sizes + 2.0 ** -23 * cap
    assert ((out.double() - want).abs() <= 2 * (2.0 ** -9 + 1.01 * score) * size + 2.0 ** -9 * want.abs() + 1e-30).all()


@pytest.mark.parametrize("dk,dv", [(128, 64), (128, 128)])
def test_a_learned_sink_needs_no_flag(dk, dv):
    q, k, v, table = setting(dk, dv, "logits")
    assert torch.equal(attend(q, k, v, table, dk, dv, "logits", sink=False), attend(q, k, v, table, dk, dv, "logits", sink=True))


@pytest.mark.parametrize("dk,dv", [(128, 64), (64, 128), (128, 128), (64, 64)])
@pytest.mark.parametrize("form,spread", [("fp32", 1.0), ("fp32", 4.0), ("capped fp32", 1.0), ("capped fp32", 4.0), ("shared values", 4.0)])
def test_no_further_from_64_bits_than_the_kernel_before(dk, dv, form, spread, monkeypatch):
    """Of the forms that came from the mma.sync kernel, whose reference follows every row's maximum: the largest weight is 1 before its division, exactly."""
    from mimirmind_b200.kernels import attention
    n = 700
    gen = torch.Generator(device=DEV).manual_seed(dk + dv)
    rnd = lambda *s: torch.randn(s, generator=gen, device=DEV).to(torch.bfloat16)     # noqa: E731
    Gv = 2 if form == "shared values" else G
    q, k, v = spread * rnd(n, H * dk), rnd(-(-n // PAGE), G, PAGE, dk), rnd(-(-n // PAGE), Gv, PAGE, dv)
    table = torch.arange(k.shape[0], dtype=torch.int32, device=DEV).view(1, -1)
    errs = []
    kk, vv = (t.transpose(1, 2).reshape(-1, t.shape[1], t.shape[3])[:n].double() for t in (k, v))
    s = torch.einsum("nhd,mhd->hnm", q.view(n, H, dk).double(), kk.repeat_interleave(H // G, dim=1)) * dk ** -0.5
    s = 20.0 * torch.tanh(s / 20.0) if "cap" in form else s
    s = s.masked_fill(torch.ones(n, n, device=DEV).triu(1).bool(), float("-inf"))
    top = s.amax(dim=-1, keepdim=True).clamp_min(0.0)          # the sink's score
    p = torch.exp(s - top) / (torch.exp(s - top).sum(dim=-1, keepdim=True) + torch.exp(-top))
    heads = torch.arange(H, device=DEV) // (H // G) % Gv
    want = torch.einsum("hnm,mhd->nhd", p, vv[:, heads]).flatten(1)
    for tensor_memory in (True, False):
        monkeypatch.setattr(attention, "USE_SINK_TCGEN05", tensor_memory)
        out = attend(q, k, v, table, dk, dv, form, lens=[n], begin=[0])
        errs.append(((out.double() - want).norm() / want.norm()).item())
    print(form, spread, dk, dv, "%.3e %.3e" % tuple(errs))
    assert errs[0] <= 1.002 * errs[1]


def test_shared_memory_is_reserved_once():
    """Not on every launch: the host's time is what bounds a layer over a short prompt."""
    from torch.profiler import ProfilerActivity, profile
    q, k, v, table = setting(128, 64, "window")
    attend(q, k, v, table, 128, 64, "window")
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as seen:
        attend(q, k, v, table, 128, 64, "window")
    names = [e.key for e in seen.key_averages()]
    assert any("Launch" in n for n in names) and not any("FuncSetAttribute" in n for n in names)
