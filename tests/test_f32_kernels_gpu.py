"""The 32-bit path's product and attention where their kernels change hands: edges of tiles, a few rows against many, short runs
against long ones.  Every form does the same operations in the same order, so a row's bits do not depend on what stands beside it."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def ops():
    from mimirmind_b200.kernels import ops as o
    return o


@pytest.mark.parametrize("N,K", [(8, 4), (131, 260), (896, 4864), (4736, 72), (37888, 68), (200, 67)])
@pytest.mark.parametrize("M", [1, 2, 4, 5, 8, 9, 16, 17, 33, 130])
def test_product(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M * N + K)
    a, w, b = (torch.randn(s, generator=g, device=DEV) for s in ((M, K), (N, K), (N,)))
    out = torch.empty((M, N), device=DEV)
    ops().gemm_simt(a, w, b, out)
    ref, size = a.double() @ w.double().T + b.double(), a.double().abs() @ w.double().abs().T + b.double().abs()
    # K products added one after the other and a bias: each addition rounds by at most 2^-24 of what has been added up
    assert ((out - ref).abs() <= (K + 1) * 2.0 ** -24 * size).all()
    for m in {0, M // 2, M - 1}:                # alone: the kernel for a few rows
        one = torch.empty((1, N), device=DEV)
        ops().gemm_simt(a[m:m + 1].contiguous(), w, b, one)
        assert torch.equal(one[0], out[m])


# rows and tokens around the tiles of 16 and 128 rows and of 8, 16, 32, 64 and 128 tokens; k in one, two, four and eight parts, whole steps of 64 and not
@pytest.mark.parametrize("N,K", [(128, 128), (131, 260), (200, 644), (257, 1540), (1000, 2052)])
@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17, 33, 64, 65, 129, 300])
def test_product_of_split_numbers(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M * N + K)
    a, w, b = (torch.randn(s, generator=g, device=DEV) for s in ((M, K), (N, K), (N,)))
    a *= torch.exp2(torch.randint(-12, 13, (M, K), generator=g, device=DEV))
    loose = torch.empty(M * K + 1, device=DEV)[1:].view(M, K).copy_(a)          # rows off the 16-byte boundaries
    out, two = torch.empty((M, N), device=DEV), torch.empty((M, N), device=DEV)
    ops().gemm_simt(a, w, b, out)
    ref, size = a.double() @ w.double().T + b.double(), a.double().abs() @ w.double().abs().T + b.double().abs()
    # K / 16 rounded additions, two dozen roundings of whole sums beside them (the parts, what is cut off sixteen terms of one sum), and five sums of K / 16 steps of
    # 2^-7 of the size
    assert ((out - ref).abs() <= (K / 16 + 24 + 5 * K / 16 / 128) * 2.0 ** -24 * size).all()
    ops().gemm_simt(loose, w, b, two)
    assert torch.equal(two, out)
    for m in {0, M // 2, M - 1}:                # alone: the kernel for a few rows
        one = torch.empty((1, N), device=DEV)
        ops().gemm_simt(a[m:m + 1].contiguous(), w, b, one)
        assert torch.equal(one[0], out[m])


@pytest.mark.parametrize("M,N,K", [(1000, 512, 516), (4900, 100, 260), (5000, 16, 2048), (37, 4864, 200), (9, 4864, 252), (3, 40000, 64)])
def test_product_of_weights_that_are_not_split(M, N, K):
    """Tiles of 64 rows with steps of 32 and of 64, of 32 rows, and the kernels that stream the weights, each against a row alone."""
    g = torch.Generator(device=DEV).manual_seed(M + N)
    a, w, b = (torch.randn(s, generator=g, device=DEV) for s in ((M, K), (N, K), (N,)))
    out = ops().gemm_simt(a, w, b, torch.empty((M, N), device=DEV))
    ref, size = a.double() @ w.double().T + b.double(), a.double().abs() @ w.double().abs().T + b.double().abs()
    assert ((out - ref).abs() <= (K + 1) * 2.0 ** -24 * size).all()             # as in test_product
    for m in {0, M // 2, M - 1}:
        assert torch.equal(ops().gemm_simt(a[m:m + 1].contiguous(), w, b, torch.empty((1, N), device=DEV))[0], out[m])


def split_forms(a, w, b):
    """The product in every form of the kernels for split numbers, by name."""
    out = {}
    for tile in (16, 32, 64, 128):
        for side_by_side in (False, True):
            if tile > 16 or (a.shape[0] <= 16 and not side_by_side):
                y = torch.empty((a.shape[0], w.shape[0]), device=DEV)
                out[tile, side_by_side] = ops().gemm_split(a, w, b, y, tile, side_by_side)
    return out


# k in one, two, four and eight parts, whole steps of 64 and not: walked by one block, whose sums of the parts before wait in tensor memory, or by one each
@pytest.mark.parametrize("N,K", [(128, 128), (131, 260), (200, 644), (257, 1540), (1000, 2052)])
@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 33, 65, 130, 300])
def test_forms_of_the_split_product(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M * N + K)
    a, w, b = (torch.randn(s, generator=g, device=DEV) for s in ((M, K), (N, K), (N,)))
    forms = split_forms(a, w, b)
    out = forms[32, False]
    for name, y in forms.items():
        assert torch.equal(y, out), name
    ref = a.double() @ w.double().T + b.double()
    # K / 16 rounded additions to a part's sum and a few to the whole, each off by an ulp / sqrt(12), at most 2^-23 / sqrt(12) of a sum that grows like the root of
    # their number.  A partial product that half of the steps leave out is 1.7e-6 of it
    assert (out - ref).norm() <= ((K / 16 + 8) / 6) ** 0.5 * 2.0 ** -24 * ref.norm()
    loose = torch.empty((M, K + 3), device=DEV)[:, :K].copy_(a)                 # rows off the 16-byte boundaries
    wide = torch.full((M, N + 5), 7.0, device=DEV)
    for tile in (16, 32, 64, 128):
        if tile > 16 or M <= 16:
            ops().gemm_split(loose, w, b, wide[:, :N], tile, tile == 64)
            assert torch.equal(wide[:, :N], out) and (wide[:, N:] == 7.0).all()


@pytest.mark.parametrize("numbers", ["powers", "cancelling", "small", "subnormal", "one large"])
@pytest.mark.parametrize("N,K", [(160, 644), (130, 1664)])
def test_bits_of_a_row_do_not_depend_on_the_others(numbers, N, K):
    """mma.sync for a few tokens and tcgen05.mma for more add sixteen products up to the same bits.  No document says so: it is what
    they do, for operands far apart as well."""
    g = torch.Generator(device=DEV).manual_seed(K)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)                         # noqa: E731
    powers = lambda top, *s: torch.exp2(torch.randint(-top, top + 1, s, generator=g, device=DEV).float())     # noqa: E731
    a, w = rnd(130, K), rnd(N, K)
    if numbers == "powers":
        a, w = a * powers(30, 130, K), w * powers(30, N, K)
    elif numbers == "cancelling":               # pairs that take each other away but for the last bits
        a[:, 1::2], w[:, 1::2] = -a[:, ::2] * (1 + 2.0 ** -20 * rnd(130, K // 2)), w[:, ::2]
    elif numbers == "small":
        a, w = a * 2.0 ** -118, w * powers(20, N, K)
    elif numbers == "subnormal":
        a, w = a * 2.0 ** -126 * powers(10, 130, K).clamp(max=1.0), w * 2.0 ** 40
    else:
        a[:, ::97] *= 2.0 ** 40
    for M in (1, 7, 16, 17, 130):
        forms = split_forms(a[:M].contiguous(), w, None)
        if M == 1:
            first = forms[16, False]
        for name, y in forms.items():
            assert torch.isfinite(y).all() and torch.equal(y, forms[32, False]), (M, name)
            assert torch.equal(y[:1], first), (M, name)
    ref, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    assert ((y - ref).abs() <= (K / 16 + 24 + 5 * K / 16 / 128) * 2.0 ** -24 * size + 2.0 ** -150).all()      # as in test_product_of_split_numbers


@pytest.mark.parametrize("M", [5, 12, 40, 150])
def test_split_product_of_numbers_that_cannot_be_split(M):
    """As below, in every form: what 32-bit FMAs over k in order give, and nothing beside them changes."""
    N, K = 140, 520
    g = torch.Generator(device=DEV).manual_seed(M)
    a, w = (torch.randn(s, generator=g, device=DEV) for s in ((M, K), (N, K)))
    clean = split_forms(a, w, None)[32, False]
    a[1, 3], a[2, 500], a[3, 17], w[130, 7], w[139, 519], w[5] = float("inf"), float("nan"), 3.4e38, float("-inf"), 3.4e38, 0.0
    a[4] = 3e38                                 # sums that overflow
    keep = torch.ones((M, N), dtype=torch.bool, device=DEV)
    keep[1:5] = False
    keep[:, [5, 130, 139]] = False
    narrow = torch.empty((M, N), device=DEV)    # by FMAs
    for n0 in (0, 70):
        narrow[:, n0:n0 + 70] = ops().gemm_simt(a, w[n0:n0 + 70].contiguous(), None, torch.empty((M, 70), device=DEV))
    for name, out in split_forms(a, w, None).items():
        assert torch.equal(out[keep], clean[keep]), name
        assert torch.equal(torch.isnan(out), torch.isnan(narrow)) and torch.equal(torch.isinf(out), torch.isinf(narrow)), name
        assert torch.equal(out[torch.isinf(out)], narrow[torch.isinf(narrow)]), name


@pytest.mark.parametrize("M", [5, 12, 40, 150])
def test_product_of_numbers_that_cannot_be_split(M):
    """An infinity, a NaN, a number beyond bf16's largest and sums that overflow: what 32-bit FMAs over k in order give, and nothing beside them changes."""
    N, K = 260, 520
    g = torch.Generator(device=DEV).manual_seed(M)
    a, w = (torch.randn(s, generator=g, device=DEV) for s in ((M, K), (N, K)))
    clean = torch.empty((M, N), device=DEV)
    ops().gemm_simt(a, w, None, clean)
    a[1, 3], a[2, 500], a[3, 17], w[130, 7], w[259, 519], w[5] = float("inf"), float("nan"), 3.4e38, float("-inf"), 3.4e38, 0.0
    a[4] = 3e38                                 # sums that overflow
    out = torch.empty((M, N), device=DEV)
    ops().gemm_simt(a, w, None, out)
    rows, cols = [1, 2, 3, 4], [130, 259, 5]
    keep = torch.ones((M, N), dtype=torch.bool, device=DEV)
    keep[rows] = False
    keep[:, cols] = False
    assert torch.equal(out[keep], clean[keep])
    narrow = torch.empty((M, 96), device=DEV)   # the product by FMAs: fewer than 128 rows of weights
    for n0 in (0, 96, 164):
        ops().gemm_simt(a, w[n0:n0 + 96].contiguous(), None, narrow)
        got = out[:, n0:n0 + 96]
        assert torch.equal(torch.isnan(got), torch.isnan(narrow)) and torch.equal(torch.isinf(got), torch.isinf(narrow))
        assert torch.equal(got[torch.isinf(got)], narrow[torch.isinf(narrow)])


@pytest.mark.parametrize("M", [4, 12, 40, 150])
@pytest.mark.parametrize("a_exp,w_exp", [(-112, 0), (-120, 0), (-125, 20), (-140, 100), (0, -120), (-70, -70), (90, 0), (100, 20), (60, 60)])
def test_product_of_small_and_large_numbers(M, a_exp, w_exp):
    """Operands near either end of the exponents: as exact as in the middle, up to the subnormal result's own rounding."""
    N, K = 200, 640
    g = torch.Generator(device=DEV).manual_seed(M)
    a, w = torch.randn((M, K), generator=g, device=DEV), torch.randn((N, K), generator=g, device=DEV)
    a, w = (torch.ldexp(x.double(), torch.tensor(e, device=DEV)).float() for x, e in ((a, a_exp), (w, w_exp)))
    out = torch.empty((M, N), device=DEV)
    ops().gemm_simt(a, w, None, out)
    ref, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    # as in test_product_of_split_numbers
    assert ((out - ref).abs() <= (K / 16 + 24 + 5 * K / 16 / 128) * 2.0 ** -24 * size + 2.0 ** -150).all()
    # n = K / 16 rounded additions to a sum that grows like the root of their number, each off by an ulp / sqrt(12), at most 2^-23 / sqrt(12) of it
    # (2-norms): together 2^-24 sqrt(n / 6) of the result.  By FMAs over k, n = K, it would be four times as much
    assert (out - ref).norm() <= (K / 16 / 6) ** 0.5 * 2.0 ** -24 * ref.norm() + 2.0 ** -150 * (M * N) ** 0.5


@pytest.mark.parametrize("N,K,split", [(131, 260, False), (512, 576, False), (1024, 256, False), (2048, 512, False), (128, 580, True), (2344, 512, True), (200, 640, True)])
def test_which_weights_are_split(N, K, split):
    """Small ones are not, for any number of tokens: their products by FMAs are the bits of narrow pieces of the weights, which always go that way."""
    g = torch.Generator(device=DEV).manual_seed(N + K)
    w = torch.randn((N, K), generator=g, device=DEV)
    for M in (1, 8, 16, 40, 200):
        a = torch.randn((M, K), generator=g, device=DEV)
        out, part = torch.empty((M, N), device=DEV), torch.empty((M, 96), device=DEV)
        ops().gemm_simt(a, w, None, out)
        ops().gemm_simt(a, w[:96].contiguous(), None, part)
        assert torch.equal(out[:, :96], part) != split


@pytest.mark.parametrize("M", [4, 300])
def test_product_of_rows_that_are_no_numbers_is_not_slow(M):
    """What a state that has gone wrong brings into every product after it: a NaN in every row.  Number by number it took some two hundred times as long
    as other rows; twice as long is what it takes."""
    N, K = 4096, 896
    g = torch.Generator(device=DEV).manual_seed(M)
    w, out, times = torch.randn((N, K), generator=g, device=DEV), torch.empty((M, N), device=DEV), []
    for bad in (False, True):
        a = torch.randn((M, K), generator=g, device=DEV)
        if bad:
            a[:, 5] = float("nan")
        taken = []
        for _ in range(8):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            ops().gemm_simt(a, w, None, out)
            end.record()
            end.synchronize()
            taken.append(start.elapsed_time(end))
        times.append(sorted(taken)[2])
        assert bool(torch.isnan(out).all()) == bad
    assert times[1] <= 10 * times[0], times


@pytest.mark.parametrize("tile", [32, 64, 128])
@pytest.mark.parametrize("side_by_side", [False, True])
@pytest.mark.parametrize("M,N,K", [(40, 130, 128), (150, 260, 1540)])
def test_product_whose_waits_run_out(tile, side_by_side, M, N, K):
    """As if a wait had run out at the start: the kernel returns, the error flag is set and the result is a sum in 64 bits.
    The next product is as if nothing had been."""
    g = torch.Generator(device=DEV).manual_seed(M + tile)
    a, w, b = (torch.randn(s, generator=g, device=DEV) for s in ((M, K), (N, K), (N,)))
    whole, gone, again = (torch.empty((M, N), device=DEV) for _ in range(3))
    flag = ops().tcgen05_error_flag(a.device)
    ops().gemm_split(a, w, b, whole, tile, side_by_side)
    assert int(flag.item()) == 0
    try:
        ops().gemm_split(a, w, b, gone, tile, side_by_side, give_up=True)
        assert int(flag.item()) == 1
    finally:
        flag.zero_()
    ops().gemm_split(a, w, b, again, tile, side_by_side)
    assert int(flag.item()) == 0 and torch.equal(again, whole)
    ref, size = a.double() @ w.double().T + b.double(), a.double().abs() @ w.double().abs().T + b.double().abs()
    assert ((gone - ref).abs() <= 2.0 ** -23 * size).all()           # rounded to 32 bits, and the bias added in 32 bits


@pytest.mark.parametrize("M,N,K", [(3, 70, 96), (40, 130, 100), (300, 257, 36)])
@pytest.mark.parametrize("ta,tw,tc", [(torch.bfloat16, torch.float32, torch.bfloat16), (torch.float32, torch.bfloat16, torch.float32)])
def test_product_of_mixed_types(M, N, K, ta, tw, tc):
    g = torch.Generator(device=DEV).manual_seed(M)
    a, w = torch.randn((M, K), generator=g, device=DEV).to(ta), torch.randn((N, K), generator=g, device=DEV).to(tw)
    out = torch.empty((M, N), dtype=tc, device=DEV)
    ops().gemm_simt(a, w, None, out)
    wide = torch.empty((M, N), device=DEV)
    ops().gemm_simt(a.float(), w.float(), None, wide)
    assert torch.equal(out, wide.to(tc))        # the same products of the same numbers


@pytest.mark.parametrize("hd,H,G", [(64, 6, 2), (128, 4, 4)])
@pytest.mark.parametrize("window", [0, 40])
@pytest.mark.parametrize("runs", [[(0, 1)], [(0, 100), (70, 3), (300, 1), (31, 33), (0, 4)], [(5, 1), (260, 1), (127, 1), (128, 1), (1000, 2)]])
def test_attention(hd, H, G, window, runs):
    """runs: (first position, tokens) of the requests of a step, their earlier keys in the cache."""
    page = 16
    g = torch.Generator(device=DEV).manual_seed(hd + window + len(runs))
    width = -(-max(p + n for p, n in runs) // page)
    pages = len(runs) * width
    k, v = (torch.randn((pages, G, page, hd), generator=g, device=DEV) for _ in range(2))
    table = torch.randperm(pages, generator=g, device=DEV).to(torch.int32).view(len(runs), width)
    n = sum(c for _, c in runs)
    q = torch.randn((n, H * hd), generator=g, device=DEV) * 2
    pos = torch.cat([torch.arange(p, p + c, dtype=torch.int32, device=DEV) for p, c in runs])
    req = torch.cat([torch.full((c,), r, dtype=torch.int32, device=DEV) for r, (_, c) in enumerate(runs)])
    for r, (p, c) in enumerate(runs):           # what lies behind a request's last token is nobody's: it must not be touched
        for j in range(p + c, width * page):
            k[table[r, j // page], :, j % page] = float("nan")
            v[table[r, j // page], :, j % page] = float("nan")
    out = ops().attention_generic(q, k, v, torch.empty_like(q), pos, req, table, page, H, G, hd, window, 0.1)
    at = 0
    for r, (p, c) in enumerate(runs):
        kk, vv = (t[table[r].long()].transpose(1, 2).reshape(width * page, G, hd).double() for t in (k, v))
        for i in {0, c // 2, c - 1}:
            hi = p + i + 1
            lo = max(0, hi - window) if window else 0
            for h in range(H):
                s = kk[lo:hi, h * G // H] @ q[at + i].view(H, hd)[h].double() * 0.1
                want = torch.softmax(s, 0) @ vv[lo:hi, h * G // H]
                # scores of up to 128 products of size ~2, weights and a sum over the keys in 32 bits
                assert (out[at + i].view(H, hd)[h] - want).abs().max() <= 2e-5 * max(1.0, vv[lo:hi].abs().max())
            one = ops().attention_generic(q[at + i:at + i + 1].contiguous(), k, v, torch.empty((1, H * hd), device=DEV), pos[at + i:at + i + 1].contiguous(),
                                          req[at + i:at + i + 1].contiguous(), table, page, H, G, hd, window, 0.1)
            assert torch.equal(one[0], out[at + i])          # as a single token, bit for bit
        at += c


def test_attention_skips_infinite_values_that_a_row_does_not_see():
    page, hd = 16, 64
    g = torch.Generator(device=DEV).manual_seed(1)
    k, v, q = (torch.randn(s, generator=g, device=DEV) for s in ((3, 1, page, hd), (3, 1, page, hd), (40, hd)))
    v[2, 0, 5] = float("inf")                   # the value of token 37
    table = torch.arange(3, dtype=torch.int32, device=DEV).view(1, 3)
    pos, req = torch.arange(40, dtype=torch.int32, device=DEV), torch.zeros(40, dtype=torch.int32, device=DEV)
    out = ops().attention_generic(q, k, v, torch.empty_like(q), pos, req, table, page, 1, 1, hd, 0, 0.125)
    assert torch.isfinite(out[:37]).all() and torch.isinf(out[37:]).all()
