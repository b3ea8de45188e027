"""The matrix-state recurrence as products over chunks against 64 bits and against the token-by-token walk: edges of chunks, requests of
unequal length, heads narrower than a tile, decays that underflow within a chunk, correlated keys, a state carried on."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def plain(q, k, v, decay, beta, S):
    """In 64 bits; q, k [n, H, dk], v [n, H, dv], decay [n, H], S [H, dk, dv]."""
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        S = S * decay[t][:, None, None]
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None]
        out[t] = torch.einsum("hkv,hk->hv", S, q[t])
    return out, S


@pytest.mark.parametrize("H,G,dk,dv", [(4, 2, 128, 128), (3, 3, 64, 128), (2, 1, 128, 64), (6, 2, 24, 36), (20, 5, 100, 128)])
@pytest.mark.parametrize("delta", [False, True])
@pytest.mark.parametrize("decay", ["near 1", "strong", "constant", "zero"])
def test_products(H, G, dk, dv, delta, decay):
    from mimirmind_b200.kernels import ops
    if decay == "constant" and delta:
        pytest.skip("the delta rule's decay is learned")
    gen = torch.Generator(device=DEV).manual_seed(H * dk + dv + delta)
    lens, begin, slots = [200, 1, 64, 129], [0, 5, 70, 0], [2, 0, 3, 4]
    n = sum(lens)
    rnd = lambda *s: torch.randn(s, generator=gen, device=DEV)                       # noqa: E731
    ld = 2 * G * dk + H * dv + 4
    row = rnd(n, ld)
    q, k, v = row[:, :G * dk], row[:, G * dk:2 * G * dk], row[:, 2 * G * dk + 4:]
    q *= dk ** -0.5
    if delta:           # unit keys, neighbouring ones alike
        kk = k.reshape(n, G, dk) + 2.0 * rnd(1, G, dk)
        k.copy_((kk / kk.norm(dim=-1, keepdim=True)).reshape(n, G * dk))
    else:
        k *= dk ** -0.5
    gate = {"near 1": 0.9 + 0.1 * torch.rand((n, H), generator=gen, device=DEV), "strong": 0.02 + 0.3 * torch.rand((n, H), generator=gen, device=DEV),
            "constant": None, "zero": (torch.rand((n, H), generator=gen, device=DEV) > 0.1).float()}[decay]
    head = torch.linspace(0.5, 0.9995, H, device=DEV) if gate is None else None
    beta = torch.rand((n, H), generator=gen, device=DEV) if delta else None
    state = rnd(5, H * dv * dk + 8)
    before = state.clone()
    starts = [sum(lens[:i]) for i in range(4)]
    meta, per = [], []
    for r, (s, m) in enumerate(zip(starts, lens)):
        per.append([len(meta), -(-m // 64)])
        meta += [[s + o, min(64, m - o), r, 0] for o in range(0, m, 64)]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)                   # noqa: E731
    pos = torch.cat([torch.arange(b, b + m, dtype=torch.int32, device=DEV) for b, m in zip(begin, lens)])
    assert ops.linear_state_products_supported(q, k, v, state, dk, dv)
    walked = before.clone()
    got = ops.linear_state_products(q, k, v, state, i32(meta), i32(per), i32(slots), pos, H, G, dk, dv, gate=gate, beta=beta, head_decay=head)
    walk = ops.linear_state_walk(q, k, v, walked, i32([[s, m, b + m, x] for s, m, b, x in zip(starts, lens, begin, slots)]), i32(slots), pos, 4, H, G,
                                 dk, dv, gate=gate, beta=beta, head_decay=head)
    assert torch.equal(state[1], before[1]) and torch.equal(state[:, H * dv * dk:], before[:, H * dv * dk:])      # nobody else's
    for r, (s, m) in enumerate(zip(starts, lens)):
        rep = lambda t, w: t[s:s + m].reshape(m, G, w).repeat_interleave(H // G, dim=1).double()                  # noqa: E731
        S = torch.zeros(H, dk, dv, dtype=torch.float64, device=DEV) if begin[r] == 0 else \
            before[slots[r], :H * dv * dk].view(H, dv, dk).transpose(1, 2).double()
        g = (gate[s:s + m] if gate is not None else head.expand(m, H)).double()
        want, S = plain(rep(q, dk), rep(k, dk), v[s:s + m].reshape(m, H, dv).double(), g, None if beta is None else beta[s:s + m].double(), S)
        kept = S.transpose(1, 2).reshape(-1)
        for mine, old, ref in ((got[s:s + m], walk[s:s + m], want.reshape(m, -1)), (state[slots[r], :H * dv * dk], walked[slots[r], :H * dv * dk], kept)):
            scale = ref.norm()
            err, was = ((mine - ref).norm() / scale).item(), ((old - ref).norm() / scale).item()
            print(f"err {err:.2e} walk {was:.2e}")
            # up to 64 + 128 + 128 products one after the other, their sums rounded like the walk's: a few 2^-22
            assert err <= max(5e-7, 1.5 * was), (r, err, was)


@pytest.mark.parametrize("H,dk,dv", [(148, 64, 20), (148, 100, 32), (74, 128, 100), (160, 48, 64)])
def test_blocks_of_32_columns(H, dk, dv):
    """So many heads that a block of the delta rule's chain takes 32 columns of a state: the bits of a few heads alone, whose blocks take sixteen."""
    from mimirmind_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(H + dv)
    lens, begin = [150, 64, 3], [0, 7, 0]
    n = sum(lens)
    rnd = lambda *s: torch.randn(s, generator=gen, device=DEV)                       # noqa: E731
    unit = lambda t: t / t.norm(dim=-1, keepdim=True)                                # noqa: E731
    q, k, v = rnd(n, H, dk) * dk ** -0.5, unit(rnd(n, H, dk) + rnd(1, H, dk)), rnd(n, H, dv)
    gate, beta = 0.8 + 0.2 * torch.rand((n, H), generator=gen, device=DEV), torch.rand((n, H), generator=gen, device=DEV)
    before = rnd(3, H, dv, dk)
    meta, per, s = [], [], 0
    for r, m in enumerate(lens):
        per.append([len(meta), -(-m // 64)])
        meta += [[s + o, min(64, m - o), r, 0] for o in range(0, m, 64)]
        s += m
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)                   # noqa: E731
    pos = torch.cat([torch.arange(b, b + m, dtype=torch.int32, device=DEV) for b, m in zip(begin, lens)])

    def run(heads):
        state = before[:, heads].reshape(3, -1).contiguous()
        flat = lambda t: t[:, heads].reshape(n, -1).contiguous()                     # noqa: E731
        h = len(heads)
        out = ops.linear_state_products(flat(q), flat(k), flat(v), state, i32(meta), i32(per), i32([0, 1, 2]), pos, h, h, dk, dv,
                                        gate=gate[:, heads].contiguous(), beta=beta[:, heads].contiguous())
        return out.view(n, h, dv), state.view(3, h, dv, dk)

    out, state = run(list(range(H)))
    few = [0, 1, H // 2, H - 1]
    some, kept = run(few)
    assert torch.isfinite(out).all() and torch.equal(out[:, few], some) and torch.equal(state[:, few], kept)


@pytest.mark.parametrize("H,dk,dv", [(4, 128, 64), (2, 128, 128), (3, 64, 64), (5, 36, 100)])
@pytest.mark.parametrize("gates", ["near 1", "wide", "near 0"])
def test_forget_gate_products(H, dk, dv, gates):
    from mimirmind_b200.kernels import ops
    gen = torch.Generator(device=DEV).manual_seed(H * dk + dv)
    lens, begin, slots = [150, 17, 64, 81], [0, 5, 70, 0], [2, 0, 3, 4]
    n = sum(lens)
    rnd = lambda *s: torch.randn(s, generator=gen, device=DEV)                       # noqa: E731
    row = rnd(n, 2 * H * dk + H * dv + 4)
    q, f, v = row[:, :H * dk], row[:, H * dk:2 * H * dk], row[:, 2 * H * dk + 4:]
    f.copy_({"near 1": 0.9 + 0.1 * torch.sigmoid(f), "wide": torch.sigmoid(4 * f), "near 0": 1e-6 + 0.05 * torch.sigmoid(f)}[gates])
    state = rnd(5, H * dv * dk + 8)
    before, walked = state.clone(), state.clone()
    starts = [sum(lens[:i]) for i in range(4)]
    meta, per = [], []
    for r, (s, m) in enumerate(zip(starts, lens)):
        per.append([len(meta), -(-m // 64)])
        meta += [[s + o, min(64, m - o), r, 0] for o in range(0, m, 64)]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)                   # noqa: E731
    pos = torch.cat([torch.arange(b, b + m, dtype=torch.int32, device=DEV) for b, m in zip(begin, lens)])
    got = ops.forget_gate_products(q, f, v, state, i32(meta), i32(per), i32(slots), pos, H, dk, dv)
    walk = ops.forget_gate_walk(q, f, v, walked, i32([[s, m, b + m, x] for s, m, b, x in zip(starts, lens, begin, slots)]), i32(slots), pos, 4, H, dk, dv)
    assert torch.equal(state[1], before[1]) and torch.equal(state[:, H * dv * dk:], before[:, H * dv * dk:])
    for r, (s, m) in enumerate(zip(starts, lens)):
        S = torch.zeros(H, dk, dv, dtype=torch.float64, device=DEV) if begin[r] == 0 else \
            before[slots[r], :H * dv * dk].view(H, dv, dk).transpose(1, 2).double()
        qq, ff, vv = (t[s:s + m].reshape(m, H, -1).double() for t in (q, f, v))
        want = torch.empty_like(vv)
        for t in range(m):
            S = S * ff[t][:, :, None] + (1.0 - ff[t])[:, :, None] * vv[t][:, None]
            want[t] = torch.einsum("hkv,hk->hv", S, qq[t])
        for mine, old, ref in ((got[s:s + m], walk[s:s + m], want.reshape(m, -1)),
                               (state[slots[r], :H * dv * dk], walked[slots[r], :H * dv * dk], S.transpose(1, 2).reshape(-1))):
            scale = ref.norm()
            err, was = ((mine - ref).norm() / scale).item(), ((old - ref).norm() / scale).item()
            print(f"err {err:.2e} walk {was:.2e}")
            assert err <= max(5e-7, 1.5 * was), (r, err, was)      # as above


@pytest.mark.parametrize("kind", ["plain", "delta", "forget"])
@pytest.mark.parametrize("lens", [[70, 1, 300, 127, 128], [256, 1], [1, 400, 3]])
def test_short_portions_beside_long_ones_are_walked(kind, lens):
    """Every request bit for bit what its own kernel makes of it, whatever stands beside it."""
    from types import SimpleNamespace

    from mimirmind_b200.kernels import ops
    from mimirmind_b200.parts.chunks import split_portions
    H, dk, dv, R, n = 3, 64, 128, len(lens), sum(lens)
    gen = torch.Generator(device=DEV).manual_seed(n)
    rnd = lambda *s: torch.randn(s, generator=gen, device=DEV)                       # noqa: E731
    q, k, v = rnd(n, H * dk) * dk ** -0.5, rnd(n, H * dk) * dk ** -0.5, rnd(n, H * dv)
    k = torch.sigmoid(k) if kind == "forget" else k
    gate, beta = 0.9 + 0.1 * torch.rand((n, H), generator=gen, device=DEV), torch.rand((n, H), generator=gen, device=DEV)
    more = {} if kind == "forget" else {"gate": gate, "beta": beta if kind == "delta" else None}
    heads = (H,) if kind == "forget" else (H, H)
    products, walk = (ops.forget_gate_products, ops.forget_gate_walk) if kind == "forget" else (ops.linear_state_products, ops.linear_state_walk)
    starts = [sum(lens[:i]) for i in range(R)]
    ctx = SimpleNamespace(q_start=starts, q_len=lens, kv_len=[m + 7 for m in lens], derived={}, token_ids=torch.zeros(1, device=DEV))
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)                   # noqa: E731
    pos = torch.cat([torch.arange(7, 7 + m, dtype=torch.int32, device=DEV) for m in lens])
    slots = i32(list(range(R))[::-1])
    before = rnd(R, H * dv * dk)
    chunk_meta, req_chunks, walked = split_portions(ctx, 64, 128)
    state = before.clone()
    out = products(q, k, v, state, chunk_meta, req_chunks, slots, pos, *heads, dk, dv, **more)
    out = walk(q, k, v, state, walked, slots, pos, R, *heads, dk, dv, out=out, **more)
    for r, (s, m) in enumerate(zip(starts, lens)):
        lone = before.clone()
        one = SimpleNamespace(q_start=[s], q_len=[m], kv_len=[m + 7], derived={}, token_ids=ctx.token_ids)
        if m >= 128:
            a, b, none = split_portions(one, 64, 128)
            assert none is None
            want = products(q, k, v, lone, a, b, slots[r:r + 1], pos, *heads, dk, dv, **more)
        else:
            want = walk(q, k, v, lone, i32([[s, m, m + 7, 0]]), slots[r:r + 1], pos, 1, *heads, dk, dv, **more)
        assert torch.equal(out[s:s + m], want[s:s + m]) and torch.equal(state[R - 1 - r], lone[R - 1 - r])


def test_which_steps_the_delta_rule_takes_to_the_products():
    """As measured: long portions of wide heads; not what a walk over many portions does as fast."""
    from mimirmind_b200.parts.linear_state import delta_by_products
    for lens, heads, dk, dv in (([512], 8, 64, 64), ([4096], 32, 128, 128), ([256] * 16, 32, 128, 128), ([2048] + [1] * 200, 32, 128, 128)):
        assert delta_by_products(lens, heads, dk, dv)
    for lens, heads, dk, dv in (([255], 8, 128, 128), ([256], 16, 128, 128), ([512] * 4, 32, 64, 64), ([512] + [1] * 200, 32, 128, 128), ([128] * 16, 32, 128, 128)):
        assert not delta_by_products(lens, heads, dk, dv)
