"""The draw of tokens where the search for an element changes its way: flat rows (more elements in a bin than its list holds, then equal
ones), rows that hold few finite logits, a NaN, very low and very high temperatures, every number of CTAs per row."""
import math

import numpy as np
import pytest
import torch

import plain_qwen2 as plain

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rows_of(kind, R, V, rng):
    if kind == "flat":
        return np.full((R, V), 1.25, dtype=np.float32)
    if kind == "nearly flat":
        return (1e-5 * rng.randn(R, V)).astype(np.float32)
    if kind == "few values":
        return rng.choice([-1.0, 0.0, 0.0, 0.5, 3.0], size=(R, V)).astype(np.float32)
    if kind == "mostly -inf":
        x = np.full((R, V), -np.inf, dtype=np.float32)
        for r in range(R):
            x[r, rng.choice(V, 9, replace=False)] = rng.randn(9) * 2
        return x
    return (3 * rng.randn(R, V)).astype(np.float32)


def check(row, T, k, p, u, token):
    """The token's share of the kept mass holds u, up to what 32-bit weights (relative error below 4e-6: exponents up to 28 in
    32 bits) can move a boundary."""
    order = np.lexsort((np.arange(row.size), -row.astype(np.float64)))
    x = row[order].astype(np.float64)
    kept = np.ones(row.size, dtype=bool) if not (0 < k < row.size) else x >= x[k - 1]
    with np.errstate(over="ignore", invalid="ignore"):
        w = np.where(kept, np.exp((x - x[0]) / T), 0.0)
    w[w < 2.0 ** -40] = 0.0
    cum, slack = np.cumsum(w), 4e-6
    lo = hi = cum[-1]
    if 0.0 < p < 1.0:           # the cut keeps equal logits together; a cut within the slack may fall on either side
        lo, hi = (cum[np.searchsorted(x[0] - x, x[0] - x[min(row.size - 1, np.searchsorted(cum, q * cum[-1]))], side="right") - 1]
                  for q in (max(0.0, p - slack), min(1.0, p + slack)))
    at = int(np.nonzero(order == token)[0][0])
    before = cum[at] - w[at]
    assert before <= u * hi + slack * cum[-1] and cum[at] >= u * lo - slack * cum[-1], (T, k, p, u, before / cum[-1], cum[at] / cum[-1])


@pytest.mark.parametrize("kind", ["flat", "nearly flat", "few values", "mostly -inf", "normal"])
@pytest.mark.parametrize("R,V", [(2, 300), (8, 9001), (16, 40000), (5, 152064), (70, 65536), (150, 33000)])
def test_draws(kind, R, V):
    from mimirmind_b200.kernels import ops
    rng = np.random.RandomState(V % 997 + R)
    logits = rows_of(kind, R, V, rng)
    temps = rng.choice([0.02, 0.3, 0.8, 1.5, 50.0], size=R).astype(np.float32)
    ks = rng.choice([0, 0, 2, 40, 5000], size=R).astype(np.int32)
    ps = rng.choice([1.0, 0.95, 0.5, 0.05], size=R).astype(np.float32)
    seeds, counters = rng.randint(1, 2 ** 31, size=R), rng.randint(0, 1000, size=R)
    t = lambda a, dt: torch.tensor(a, dtype=dt, device=DEV)                  # noqa: E731
    args = [t(temps, torch.float32), t(ks, torch.int32), t(ps, torch.float32), t(seeds, torch.int64), t(counters, torch.int64)]
    got = ops.sample_rows(t(logits, torch.float32), *args).cpu().tolist()
    for r in list(range(R))[:24]:
        u = plain.uniform_from(int(seeds[r]), int(counters[r]))
        check(logits[r], float(temps[r]), int(ks[r]), float(ps[r]), u, got[r])
    # a row alone is shared by another number of CTAs and draws the same token
    for r in (0, R - 1):
        one = ops.sample_rows(t(logits[r:r + 1], torch.float32), *[a[r:r + 1].contiguous() for a in args]).item()
        assert one == got[r]


def test_a_row_with_a_nan_or_an_infinite_logit_leaves_the_others_alone():
    from mimirmind_b200.kernels import ops
    rng = np.random.RandomState(4)
    x = torch.tensor(rng.randn(4, 20000), dtype=torch.float32, device=DEV)
    full = lambda v, dt: torch.full((4,), v, dtype=dt, device=DEV)           # noqa: E731
    args = [full(0.9, torch.float32), full(30, torch.int32), full(0.9, torch.float32), full(5, torch.int64), torch.arange(4, device=DEV)]
    want = ops.sample_rows(x, *args).cpu().tolist()
    x[1, 77] = math.nan
    x[2, 5] = math.inf
    got = ops.sample_rows(x, *args).cpu().tolist()
    assert got[0] == want[0] and got[3] == want[3] and all(0 <= v < 20000 for v in got)


@pytest.mark.parametrize("T", [1e-3, 1e-5, 1e-6])
@pytest.mark.parametrize("R,V", [(150, 33000), (5, 152064)])
def test_equal_logits_at_a_very_low_temperature(R, V, T):
    """logit / T - max / T is then off zero by its rounding: every weight is above one, and their sums have to hold them.  (At 1e-6 the
    rounding is at most 1, V e 2^40 < 2^59; at 1e-7 it may be 8, and 33000 e^8 2^40 is beyond the 64 bits of the total.)"""
    from mimirmind_b200.kernels import ops
    rng = np.random.RandomState(11)
    logits = np.repeat(rng.uniform(1.0, 20.0, size=(R, 1)).astype(np.float32), V, axis=1)
    seeds, counters = rng.randint(1, 2 ** 31, size=R), rng.randint(0, 1000, size=R)
    t = lambda a, dt: torch.tensor(a, dtype=dt, device=DEV)                  # noqa: E731
    got = ops.sample_rows(t(logits, torch.float32), torch.full((R,), T, device=DEV), torch.zeros(R, dtype=torch.int32, device=DEV),
                          torch.ones(R, device=DEV), t(seeds, torch.int64), t(counters, torch.int64)).cpu().tolist()
    for r in range(R):          # equal weights: the share of token i is [i, i+1) / V; u has 24 or more bits, the product rounds once
        u = plain.uniform_from(int(seeds[r]), int(counters[r]))
        assert abs(got[r] - u * V) <= 1.0 + 1e-6 * V, (r, T, got[r], u * V)


@pytest.mark.parametrize("R,V,scale,T,k,p,shift", [
    (6, 152064, 2.0, 0.8, 0, 0.95, 0),       # the bins of the cut and the draw hold less than a list, or a little more
    (4, 152064, 2.0, 1.5, 0, 0.9, 0),        # ... several lists: the bins are cut finer
    (3, 152064, 2.0, 8.0, 0, 0.9, 0),        # ... and more of them than a warp keeps
    (4, 152064, 2.0, 1.5, 5000, 0.95, 0),    # top-k's own bin leaves the others' places in doubt
    (40, 152061, 2.0, 1.0, 0, 0.95, 0),      # rows that start off 16 bytes
    (40, 65536, 2.0, 1.0, 300, 0.99, 1),     # ... and a first row that does
    (5, 8 * 38016, 2.0, 0.7, 0, 0.9, 0),     # the widest row whose slices are kept in shared memory
    (3, 8 * 38016 + 4, 2.0, 0.7, 0, 0.9, 0),
    (2, 8 * 65024 + 4, 2.0, 0.7, 0, 0.9, 0),   # beyond what the sums of the bins hold
])
def test_draws_where_the_search_changes_its_way(R, V, scale, T, k, p, shift):
    from mimirmind_b200.kernels import ops
    rng = np.random.RandomState(V % 991 + k)
    logits = (scale * rng.randn(R, V)).astype(np.float32)
    for r in range(R):
        logits[r, rng.choice(V, 24, replace=False)] += 10 * rng.rand(24).astype(np.float32)
    full = lambda v, dt: torch.full((R,), v, dtype=dt, device=DEV)           # noqa: E731
    seeds = rng.randint(1, 2 ** 31, size=R)
    buf = torch.empty(R * V + shift, device=DEV)
    x = buf[shift:].view(R, V)
    x.copy_(torch.tensor(logits))
    got = ops.sample_rows(x, full(T, torch.float32), full(k, torch.int32), full(p, torch.float32), torch.tensor(seeds, device=DEV), full(3, torch.int64)).cpu().tolist()
    for r in list(range(R))[:6]:
        check(logits[r], T, k, p, plain.uniform_from(int(seeds[r]), 3), got[r])


@pytest.mark.parametrize("T", [1e36, 1e38, 3e38])
@pytest.mark.parametrize("k,p", [(0, 0.9), (40000, 1.0)])
def test_temperatures_whose_reciprocal_is_below_the_normal_numbers(T, k, p):
    """The first bins and the finer ones have to agree on every logit where 1 / (32 T) has fewer than 24 bits."""
    from mimirmind_b200.kernels import ops
    R, V = 6, 152064
    rng = np.random.RandomState(int(np.log10(T)) + k)
    logits = (rng.uniform(-1.0, 1.0, size=(R, V)) * min(3.3e38, 4.0 * T)).astype(np.float32)
    seeds = rng.randint(1, 2 ** 31, size=R)
    full = lambda v, dt: torch.full((R,), v, dtype=dt, device=DEV)           # noqa: E731
    got = ops.sample_rows(torch.tensor(logits, device=DEV), full(T, torch.float32), full(k, torch.int32), full(p, torch.float32),
                          torch.tensor(seeds, device=DEV), full(3, torch.int64)).cpu().tolist()
    for r in range(R):
        check(logits[r], float(np.float32(T)), k, p, plain.uniform_from(int(seeds[r]), 3), got[r])


def test_wide_rows_are_not_slow():
    """A row of more numbers than the bins' 32-bit sums have room for goes through them in segments; without them it took eight to nine times
    as long as a row that is a little shorter."""
    from mimirmind_b200.kernels import ops
    times = []
    for V in (8 * 60800, 8 * 60800 + 320):
        x = 2 * torch.randn((2, V), device=DEV)
        full = lambda v, dt: torch.full((2,), v, dtype=dt, device=DEV)       # noqa: E731
        args = [full(0.8, torch.float32), full(0, torch.int32), full(0.95, torch.float32), full(5, torch.int64), torch.arange(2, device=DEV)]
        taken = []
        for _ in range(8):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            ops.sample_rows(x, *args)
            end.record()
            end.synchronize()
            taken.append(start.elapsed_time(end))
        times.append(sorted(taken)[2])
    assert times[1] <= 4 * times[0], times


@pytest.mark.parametrize("R,V,scale,T,k,p", [(2, 8 * 60800 + 4, 2.0, 0.7, 0, 0.9), (2, 1000003, 2.0, 0.8, 50, 0.95), (3, 1000000, 0.5, 1.5, 0, 0.9),
                                             (2, 2 * 8 * 60800 + 4, 3.0, 0.3, 0, 1.0), (1, 700000, 0.0, 1.0, 0, 1.0)])
def test_draws_from_rows_in_segments(R, V, scale, T, k, p):
    from mimirmind_b200.kernels import ops
    rng = np.random.RandomState(V % 991 + k)
    logits = (1.0 + scale * rng.randn(R, V)).astype(np.float32)
    full = lambda v, dt: torch.full((R,), v, dtype=dt, device=DEV)           # noqa: E731
    seeds = rng.randint(1, 2 ** 31, size=R)
    got = ops.sample_rows(torch.tensor(logits, device=DEV), full(T, torch.float32), full(k, torch.int32), full(p, torch.float32),
                          torch.tensor(seeds, device=DEV), full(3, torch.int64)).cpu().tolist()
    for r in range(R):
        check(logits[r], T, k, p, plain.uniform_from(int(seeds[r]), 3), got[r])
