"""The matrix states as products over chunks, number by number: how far they are from 64 bits beside the token-by-token walk, very large numbers,
and what a number that is none does to the tokens around it."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
ROUNDING = 2.0 ** -24 / 3 ** 0.5 * 0.72          # root mean square of a rounding to 24 bits, relative, over the places of a binade


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


class Portion:
    """One request's portion of n tokens from its start; kind "plain", "delta" or "forget"."""

    def __init__(self, kind, n, H=4, G=4, dk=128, dv=128, seed=0, keys="independent", decay="strong"):
        gen = torch.Generator(device=DEV).manual_seed(seed + n + dk)
        rnd = lambda *s: torch.randn(s, generator=gen, device=DEV)                       # noqa: E731
        self.kind, self.n, self.H, self.G, self.dk, self.dv = kind, n, H, G, dk, dv
        self.q, self.k, self.v = rnd(n, G * dk), rnd(n, G * dk), rnd(n, H * dv)
        self.gate = self.beta = None
        if keys == "the same":        # nearly, with values that turn every 32 tokens: what a half of a chunk adds, the other takes back
            self.k = rnd(1, G * dk) + 1e-3 * self.k
            self.v = 0.1 * self.v + (1.0 - 2.0 * ((torch.arange(n, device=DEV) // 32) % 2))[:, None]
        if kind == "forget":
            self.q, low = torch.nn.functional.silu(self.q), torch.sigmoid(rnd(H * dk))
            self.k = low + (1 - low) * torch.sigmoid(self.k)
            return
        self.gate = {"strong": torch.sigmoid(rnd(n, H)), "near 1": torch.exp(-0.01 * torch.sigmoid(rnd(n, H))), "none": torch.ones(n, H, device=DEV)}[decay]
        if kind == "delta":
            unit = lambda t: (t.view(n, G, dk) / t.view(n, G, dk).norm(dim=-1, keepdim=True)).reshape(n, G * dk)    # noqa: E731
            self.q, self.k, self.beta = unit(self.q), unit(self.k), torch.sigmoid(rnd(n, H) + (3.0 if keys == "the same" else 0.0))

    def run(self, products):
        from mimirmind_b200.kernels import ops
        n, H, state = self.n, self.H, torch.zeros(1, self.H * self.dv * self.dk, device=DEV)
        if products:
            where = (i32([[o, min(64, n - o), 0, 0] for o in range(0, n, 64)]), i32([[0, -(-n // 64)]]), i32([0]), i32(list(range(n))))
        else:
            where = (i32([[0, n, n, 0]]), i32([0]), i32(list(range(n))), 1)
        if self.kind == "forget":
            out = (ops.forget_gate_products if products else ops.forget_gate_walk)(self.q, self.k, self.v, state, *where, H, self.dk, self.dv)
        else:
            out = (ops.linear_state_products if products else ops.linear_state_walk)(self.q, self.k, self.v, state, *where, H, self.G, self.dk, self.dv,
                                                                                     gate=self.gate, beta=self.beta)
        return out, state[0]

    def exact(self):
        n, H, dk, dv = self.n, self.H, self.dk, self.dv
        wide = lambda t: t.double().view(n, self.G, dk).repeat_interleave(H // self.G, dim=1)                        # noqa: E731
        q, k, v = wide(self.q), wide(self.k), self.v.double().view(n, H, dv)
        g = k if self.kind == "forget" else self.gate.double()[:, :, None]
        k = 1.0 - k if self.kind == "forget" else k
        S, out = torch.zeros(H, dk, dv, dtype=torch.float64, device=DEV), torch.empty_like(v)
        for t in range(n):
            S = S * g[t][:, :, None]
            u = v[t] if self.beta is None else self.beta[t].double()[:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
            S = torch.baddbmm(S, k[t][:, :, None], u[:, None])
            out[t] = torch.bmm(q[t][:, None], S)[:, 0]
        return out.reshape(n, -1), S.transpose(1, 2).reshape(-1)


def errors(got, want):
    return [((a.double() - b).norm() / b.norm()).item() for a, b in zip(got, want)]


@pytest.mark.parametrize("kind,decay", [("plain", "near 1"), ("plain", "none"), ("delta", "near 1"), ("delta", "none")])
@pytest.mark.parametrize("n,dk,dv", [(300, 128, 128), (1000, 128, 64), (700, 64, 128)])
def test_sums_over_many_tokens_are_closer_than_the_walk(kind, decay, n, dk, dv):
    p = Portion(kind, n, dk=dk, dv=dv, decay=decay)
    want = p.exact()
    for mine, walk in zip(errors(p.run(True), want), errors(p.run(False), want)):
        assert mine <= 0.6 * walk, (mine, walk)


@pytest.mark.parametrize("kind,roundings", [("plain", 16), ("delta", 30), ("forget", 16)])
@pytest.mark.parametrize("n,dk,dv", [(300, 128, 128), (1000, 128, 64), (700, 64, 128)])
def test_a_few_roundings_where_the_decays_are_strong(kind, roundings, n, dk, dv):
    """The walk rounds twice per token here and forgets most of it; the products round the decayed factors, the sums of 16 tokens or channels and
    their sums, with the delta rule those of W, U and the chunk's solution too: factors enter with all of their 24 bits."""
    p = Portion(kind, n, dk=dk, dv=dv)
    for e in errors(p.run(True), p.exact()):
        assert e <= roundings ** 0.5 * ROUNDING, e


@pytest.mark.parametrize("kind", ["plain", "delta", "forget"])
def test_very_large_numbers(kind):
    p = Portion(kind, 150)
    p.v *= 2e34
    got, want = p.run(True), p.exact()
    for mine, ref in zip(got, want):
        assert torch.isfinite(mine).all() and ((mine.double() - ref).norm() / ref.norm()).item() <= 2e-7


@pytest.mark.parametrize("kind", ["plain", "delta"])
@pytest.mark.parametrize("token", [0, 37, 64, 149])
def test_a_decay_that_is_no_number(kind, token):
    """It makes the state one that is no number, as in the walk: not an empty one."""
    p = Portion(kind, 150)
    p.gate[token, 1] = float("nan")
    (out, state), (walk, walked) = p.run(True), p.run(False)
    assert torch.equal(torch.isnan(out[token:]), torch.isnan(walk[token:])) and torch.equal(torch.isnan(state), torch.isnan(walked))
    assert torch.isnan(state.view(p.H, -1)[1]).all() and not torch.isnan(state.view(p.H, -1)[[0, 2, 3]]).any()


@pytest.mark.parametrize("n", [2048])
def test_what_a_chunk_writes_and_takes_back(n):
    p = Portion("delta", n, keys="the same", decay="none")
    want = p.exact()
    for mine, walk in zip(errors(p.run(True), want), errors(p.run(False), want)):
        assert mine <= 1.2 * walk, (mine, walk)


@pytest.mark.parametrize("kind,what", [(k, w) for k in ("plain", "delta", "forget") for w in ("q", "k", "v", "gate", "beta")
                                       if not (k == "forget" and w == "gate") and (k == "delta" or w != "beta")])
@pytest.mark.parametrize("number", [float("nan"), float("inf")])
@pytest.mark.parametrize("token", [0, 37, 64, 70, 127, 149])
@pytest.mark.parametrize("dk,dv", [(128, 128), (64, 64)])
def test_a_number_that_is_none_reaches_later_tokens_only(kind, what, number, token, dk, dv):
    if number == float("inf") and (what in ("gate", "beta") or (kind == "forget" and what == "k")):
        pytest.skip("decays and strengths are logistic values: a NaN is the only one that can stand there")
    p = Portion(kind, 150, dk=dk, dv=dv)
    clean = p.run(True)[0].clone()
    getattr(p, what)[token, 5 if what in ("q", "k", "v") else 1] = number
    (out, state), (walk, walked) = p.run(True), p.run(False)
    # before the token nothing has changed, but for the order of a chunk's sums
    assert torch.isfinite(out[:token]).all() and (out[:token] - clean[:token]).norm() <= 1e-6 * clean.norm()
    assert torch.equal(torch.isfinite(out), torch.isfinite(walk)) and torch.equal(torch.isfinite(state), torch.isfinite(walked))
