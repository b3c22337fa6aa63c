"""GPU parity at the edges of tiles, alignments and splits: contractions with ragged extents and with few tiles, f32 products and
attention on the tensor cores, attention of a few queries, convolutions gathered from the image, folds and maps with remainders.
References are float64 on the CPU."""
import ctypes as C
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

BF16, F32 = torch.bfloat16, torch.float32
# a bf16 result is off by half a unit in its last place, 2^-9 of its value, and by what f32 sums of up to 4096 terms lose
BF16_ROUND = 2.0 ** -8
# an f32 product cut into bf16 pieces leaves out less than 2^-22 of each |a b|, its sums and the accumulators' updates lose no more
F32_CELL = 2.0 ** -20
# three TF32 products leave out less than 2^-20 of each |a b|; a chunk of 256 k is 96 updates of an accumulator that cut off at
# most 2^-22 of it each
TF32_CELL = 2.0 ** -15


@pytest.fixture(scope="module")
def T():
    from mimir_b200 import tensor
    return tensor


def rnd(shape, seed, dtype=F32, offset=0):
    """Normal values; `offset` elements into its storage, so that the base address is not a multiple of 16 bytes."""
    g = torch.Generator().manual_seed(seed)
    n = math.prod(shape)
    t = torch.empty(n + offset, dtype=dtype, device="cuda")
    t[offset:] = torch.randn(n, generator=g).to(dtype).cuda()
    return t[offset:].view(shape)


def d64(t):
    return t.detach().cpu().double()


def close_cells(got, want, scale, tol):
    """|got - want| <= tol * scale cell by cell (scale: the sum of the terms' magnitudes); infinities and NaN in the same places."""
    g, w = d64(got), want
    assert torch.equal(g.isnan(), w.isnan()) and torch.equal(g.isinf(), w.isinf()) and torch.equal(g[w.isinf()], w[w.isinf()])
    ok = w.isfinite()
    assert ((g - w).abs()[ok] <= (tol * scale)[ok]).all(), ((g - w).abs() / scale)[ok].max().item()


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("outer,length,inner", [(1, 15, 3), (2, 16, 8), (3, 17, 33), (2, 333, 20), (1, 2049, 40), (4, 64, 1028)])
def test_folds_and_maps_along_a_middle_axis(T, outer, length, inner, dtype):
    x, y = rnd((outer, length, inner), 1, dtype), rnd((outer, inner), 2, dtype)
    xd, yd = d64(x), d64(y)
    tol = 2.0 ** -20 if dtype == F32 else BF16_ROUND
    close_cells(T.reduce("sum", 1, x), xd.sum(1), xd.abs().sum(1), tol)
    close_cells(T.reduce_fused("sum", 1, x, "square"), xd.square().sum(1), xd.square().sum(1), tol)
    close_cells(T.reduce_fused("sum", 1, x, "mul", y), (xd * yd[:, None]).sum(1), (xd * yd[:, None]).abs().sum(1), tol)
    assert torch.equal(d64(T.reduce("max", 1, x)), xd.amax(1)) and torch.equal(d64(T.reduce("min", 1, x)), xd.amin(1))
    want = (xd * yd[:, None]).clamp(min=0)
    close_cells(T.binary_ax("mul", 1, x, y, then="relu"), want, want.abs() + 1e-30, tol)


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("outer,length,inner,offset", [
    (1, 256, 32, 0), (3, 255, 32, 0), (2, 257, 36, 0), (3, 128, 64, 0), (2, 64, 128, 0), (5, 63, 128, 0), (1, 2048, 4, 0), (2, 2049, 8, 0),
    (1, 100003, 12, 0), (2, 4100, 260, 0), (1, 20000, 96, 0), (40, 300, 100, 0), (300, 64, 1028, 0),
    (2, 300, 64, 1), (1, 64, 33, 0), (2, 63, 95, 0), (3, 191, 31, 0), (1, 513, 2, 0), (1, 100003, 7, 0), (2, 4099, 65, 0), (80, 70, 1023, 0)])
def test_folds_in_tiles_of_columns(T, outer, length, inner, offset, dtype):
    """One and four columns to a thread, lanes of 1 to 32, slices or none, tails of the axis and of the rows, with each placement of a second
    operand; extremes are the same values. No term of a sum passes more than length / 8 additions of a thread and 60 of the joins and
    slices (100 where a column is one thread's), each off by 2^-24 of the sum of the magnitudes at most, and one rounding of its own."""
    x, y = rnd((outer, length, inner), 1, dtype, offset=offset), rnd((outer, length, inner), 2, dtype, offset=offset)
    xd, yd, tol = d64(x), d64(y), (length / 8 + 101) * 2.0 ** -24 + (0 if dtype == F32 else BF16_ROUND)
    close_cells(T.reduce("sum", 1, x), xd.sum(1), xd.abs().sum(1), tol)
    close_cells(T.reduce_fused("sum", 1, x, "square"), xd.square().sum(1), xd.square().sum(1), tol)
    close_cells(T.reduce_fused("sum", 1, x, "mul", y), (xd * yd).sum(1), (xd * yd).abs().sum(1), tol)
    close_cells(T.reduce_fused("sum", 1, x, "mul", y[:, 0]), (xd * yd[:, :1]).sum(1), (xd * yd[:, :1]).abs().sum(1), tol)
    close_cells(T.reduce_fused("sum", 1, x, "add", y[0]), (xd + yd[0]).sum(1), (xd + yd[0]).abs().sum(1), tol)
    x[0, length // 2, 0], x[0, length - 1, 1], x[-1, 0, inner - 1] = math.inf, -math.inf, math.nan
    for monoid in ("max", "min"):
        want = x.float().nan_to_num(-math.inf if monoid == "max" else math.inf, math.inf, -math.inf)
        want = want.amax(1) if monoid == "max" else want.amin(1)
        assert torch.equal(T.reduce(monoid, 1, x).float(), want)
    got = T.reduce("sum", 1, x).float()
    assert got[0, 0] == math.inf and (inner == 2 or got[0, 1] == -math.inf) and torch.isnan(got[-1, inner - 1])


def attention_reference(q, k, v, scale, causal):
    s = d64(q) @ d64(k).transpose(1, 2) * scale
    if causal:
        hidden = torch.ones(s.shape[1:], dtype=torch.bool).triu_(s.shape[2] - s.shape[1] + 1)
        s = s.masked_fill(hidden, -math.inf)
        p = torch.softmax(s, -1).masked_fill(hidden, 0.0)
        p = p.masked_fill(hidden.all(1)[None, :, None], 0.0)
    else:
        p = torch.softmax(s, -1)
    return p @ d64(v), torch.logsumexp(s, -1)


@pytest.mark.parametrize("bh,sq,sk,d,causal", [
    (2, 128, 64, 64, False), (3, 129, 65, 32, False), (2, 300, 191, 33, False), (2, 257, 257, 96, True), (1, 130, 200, 97, True),
    (2, 200, 100, 128, True), (1, 1, 1000, 80, False), (2, 127, 63, 1, True), (40, 150, 150, 64, False)])
def test_f32_attention_of_any_length(T, bh, sq, sk, d, causal):
    q, k, v = rnd((bh, sq, d), 1), rnd((bh, sk, d), 2), rnd((bh, sk, d), 3)
    got, lse = T.attention(q, k, v, scale=d ** -0.5, causal=causal, return_lse=True)
    T.device_status()
    want, want_lse = attention_reference(q, k, v, d ** -0.5, causal)
    # scores off by F32_CELL of their terms, which the exponential turns into a relative error of the weights
    assert ((d64(got) - want).abs() <= 64 * F32_CELL).all()
    seen = want_lse.isfinite()
    assert torch.equal(d64(lse).isfinite(), seen) and ((d64(lse) - want_lse).abs()[seen] <= 64 * F32_CELL).all()
    assert torch.equal(got, T.attention(q, k, v, scale=d ** -0.5, causal=causal))


@pytest.mark.parametrize("sq,sk,d,causal", [(50, 60, 33, False), (200, 130, 128, True), (130, 300, 64, False)])
@pytest.mark.parametrize("qs,ks,vs", [(1.0, 1.0, 1e-36), (1.0, 1.0, 1e-38), (1.0, 1.0, 1e-41), (1e-37, 1e37, 1.0), (30.0, 30.0, 1.0)])
def test_f32_attention_of_tiny_values(T, sq, sk, d, causal, qs, ks, vs):
    # values below 2^-109, and weights (the last case), do not fit three bf16 pieces
    q, k, v = rnd((2, sq, d), 1) * qs, rnd((2, sk, d), 2) * ks, rnd((2, sk, d), 3)
    v[:, :, d // 2:] *= vs
    if qs > 1:  # the key with nearly all the weight holds nothing: the rest of the row is what the smallest weights bring
        k[:, 7, 0], q[..., 0] = 5000.0, 1.0
        k[:, 7, 1:] = k[:, 7, 1:] * 0.01
        q[..., 0] *= 1.0 / (5000.0 * 0.1) * 80.0
        q[..., 1:] *= 0.01
        v[:, 7] = 0.0
    got = T.attention(q, k, v, scale=0.1, causal=causal)
    T.device_status()
    want, _ = attention_reference(q, k, v, 0.1, causal)
    weights = attention_reference(q, k, v.abs(), 0.1, causal)[0]
    # scores of up to 100, off by F32_CELL of their terms and by the rounding of the exponential's argument
    assert ((d64(got) - want).abs() <= 200 * F32_CELL * weights + 1e-43).all()


@pytest.mark.parametrize("bh,sq,sk,d,causal", [
    (2, 129, 384, 64, False), (90, 300, 449, 64, True), (90, 257, 400, 30, False), (3, 200, 513, 97, True), (2, 500, 385, 128, True), (2, 1000, 450, 33, True)])
@pytest.mark.parametrize("vs", [1.0, 1e-38, 1e-41, math.inf])
def test_f32_attention_with_keys_cut_beforehand(T, bh, sq, sk, d, causal, vs):
    # one and two query tiles to an SM, tiles without a partner and of different lengths, values that do not fit the pieces, infinities
    q, k, v = rnd((bh, sq, d), 1), rnd((bh, sk, d), 2), rnd((bh, sk, d), 3)
    if vs == math.inf:
        q[0, 5, 3], k[1, 7, 2] = math.inf, -math.inf
        if not causal:   # (a hidden key's value is not read; the reference would multiply it by zero)
            v[0, 9, 1], v[1, 300, 1] = math.nan, math.inf
    else:
        v[:, :, d // 2:] *= vs
    got, lse = T.attention(q, k, v, scale=d ** -0.5, causal=causal, return_lse=True)
    T.device_status()
    want, want_lse = attention_reference(q, k, v, d ** -0.5, causal)
    g, w = d64(got), want
    assert torch.equal(g.isnan(), w.isnan()) and torch.equal(g.isinf(), w.isinf())
    weights = attention_reference(q, k, v.abs().nan_to_num(1, 1, 1), d ** -0.5, causal)[0].nan_to_num(1)
    ok = w.isfinite()
    assert ((g - w).abs() <= 64 * F32_CELL * weights + 1e-43)[ok].all()
    seen = want_lse.isfinite()
    assert ((d64(lse) - want_lse).abs()[seen] <= 64 * F32_CELL).all()


@pytest.mark.parametrize("d", [16, 64, 128])
@pytest.mark.parametrize("bh,sq,sk", [(1, 3, 1), (1, 3, 24), (700, 2, 20), (700, 40, 20), (700, 2, 64)])
def test_f32_attention_of_few_keys(T, bh, sq, sk, d):
    # a warp per row up to some number of rows and keys, which lies between these
    q, k, v = rnd((bh, sq, d), 1), rnd((bh, sk, d), 2), rnd((bh, sk, d), 3)
    got, lse = T.attention(q, k, v, scale=d ** -0.5, return_lse=True)
    T.device_status()
    want, want_lse = attention_reference(q, k, v, d ** -0.5, False)
    assert ((d64(got) - want).abs() <= 64 * F32_CELL).all() and ((d64(lse) - want_lse).abs() <= 64 * F32_CELL).all()


def test_f32_attention_with_infinities_takes_the_general_path(T):
    q, k, v = rnd((2, 300, 64), 1), rnd((2, 200, 64), 2), rnd((2, 200, 64), 3)
    q[0, 5, 3], k[1, 7, 2], v[0, 9, 1], v[1, 8, 1] = math.inf, -math.inf, math.nan, math.inf
    got = T.attention(q, k, v, scale=0.125)
    want, _ = attention_reference(q, k, v, 0.125, False)
    g = d64(got)
    assert torch.equal(g.isnan(), want.isnan()) and torch.equal(g.isinf(), want.isinf())
    assert ((g - want).abs()[want.isfinite()] <= 64 * F32_CELL).all()


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("bh,sq,sk,causal", [
    (3, 1, 1, False), (2, 1, 15, False), (5, 16, 17, True), (2, 16, 9, True), (1, 9, 4097, True), (160, 2, 300, False), (300, 1, 70, True),
    (1, 1, 5000, False), (7, 5, 1024, False)])
def test_attention_of_a_few_queries(T, bh, sq, sk, d, causal):
    q, k, v = rnd((bh, sq, d), 1, BF16), rnd((bh, sk, d), 2, BF16), rnd((bh, sk, d), 3, BF16)
    got, lse = T.attention(q, k, v, scale=d ** -0.5, causal=causal, return_lse=True)
    T.device_status()
    want, want_lse = attention_reference(q, k, v, d ** -0.5, causal)
    # weights and result are rounded to bf16: 2^-9 of every term
    weights = attention_reference(q, k, v.abs(), d ** -0.5, causal)[0]
    assert ((d64(got) - want).abs() <= BF16_ROUND * (want.abs() + weights) + 1e-6).all()
    seen = want_lse.isfinite()
    assert torch.equal(d64(lse).isfinite(), seen) and ((d64(lse) - want_lse).abs()[seen] <= 1e-4).all()


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("bh,sq,sk,causal", [
    (1, 8, 16, False), (1, 9, 16, True), (148, 1, 768, False), (128, 8, 1000, False), (128, 9, 1000, True), (2, 8, 3000, True), (3, 7, 47, False), (1, 16, 1, False)])
def test_attention_of_a_few_queries_in_tiles_of_eight_rows(T, bh, sq, sk, d, causal):
    # one and two tiles of rows, rings that wrap or are never full, heads that fill the SMs; the bound of test_attention_of_a_few_queries
    q, k, v = rnd((bh, sq, d), 4, BF16), rnd((bh, sk, d), 5, BF16), rnd((bh, sk, d), 6, BF16)
    got, lse = T.attention(q, k, v, scale=d ** -0.5, causal=causal, return_lse=True)
    T.device_status()
    want, want_lse = attention_reference(q, k, v, d ** -0.5, causal)
    weights = attention_reference(q, k, v.abs(), d ** -0.5, causal)[0]
    assert ((d64(got) - want).abs() <= BF16_ROUND * (want.abs() + weights) + 1e-6).all()
    seen = want_lse.isfinite()
    assert torch.equal(d64(lse).isfinite(), seen) and ((d64(lse) - want_lse).abs()[seen] <= 1e-4).all()


@pytest.mark.parametrize("bh,sq,sk", [(118, 16, 400), (120, 10, 400), (120, 11, 825), (120, 11, 826), (128, 16, 1), (128, 16, 1200), (148, 12, 1999), (148, 14, 4097), (149, 16, 130)])
def test_attention_of_a_few_queries_where_heads_fill_the_chip(T, bh, sq, sk):
    # on both sides of the line between the streaming kernel and the 128-row kernel; the bound of test_attention_of_a_few_queries
    q, k, v = rnd((bh, sq, 128), 7, BF16), rnd((bh, sk, 128), 8, BF16), rnd((bh, sk, 128), 9, BF16)
    got, lse = T.attention(q, k, v, scale=128 ** -0.5, return_lse=True)
    T.device_status()
    want, want_lse = attention_reference(q, k, v, 128 ** -0.5, False)
    weights = attention_reference(q, k, v.abs(), 128 ** -0.5, False)[0]
    assert ((d64(got) - want).abs() <= BF16_ROUND * (want.abs() + weights) + 1e-6).all()
    assert ((d64(lse) - want_lse).abs() <= 1e-4).all()


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("bh,sq,sk,causal,scale", [(3, 1, 40, True, 0.1), (2, 16, 1000, True, 0.1), (9, 2, 5000, True, 0.1), (200, 3, 300, True, 0.1), (4, 5, 700, False, -0.1)])
def test_attention_of_a_few_queries_keeps_f32_weights(T, bh, sq, sk, d, causal, scale):
    # fewer queries than keys under a mask, or a negative scale: f32 weights, so that only the result is rounded to bf16
    q, k, v = rnd((bh, sq, d), 1, BF16), rnd((bh, sk, d), 2, BF16), rnd((bh, sk, d), 3, BF16)
    got = T.attention(q, k, v, scale=scale, causal=causal)
    T.device_status()
    want, _ = attention_reference(q, k, v, scale, causal)
    weights = attention_reference(q, k, v.abs(), scale, causal)[0]
    # half a unit in the last of eight bits: 2^-8 of the result; scores off by F32_CELL of their terms
    assert ((d64(got) - want).abs() <= BF16_ROUND * want.abs() + 64 * F32_CELL * weights).all()


def test_attention_of_a_few_queries_does_not_read_hidden_keys(T):
    q, k, v = rnd((2, 4, 64), 1, BF16), rnd((2, 40, 64), 2, BF16), rnd((2, 40, 64), 3, BF16)
    v[0, 39, 5], v[1, 38, 7] = math.inf, math.nan   # seen by the last query, and by the last two
    got = d64(T.attention(q, k, v, scale=0.125, causal=True))
    assert got[0, :3].isfinite().all() and got[0, 3, 5].isinf() and got[1, :2].isfinite().all() and got[1, 2:, 7].isnan().all()
    want, _ = attention_reference(q, k, v.nan_to_num(0, 0, 0), 0.125, True)
    assert ((got - want).abs()[0, :3] <= 0.03).all() and ((got - want).abs()[1, :2] <= 0.03).all()


@pytest.mark.parametrize("dtype,d", [(BF16, 64), (BF16, 128), (BF16, 80), (F32, 64), (F32, 130)])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("sq,sk,hidden", [
    (1, 17, [16]), (1, 49, [48]), (2, 49, range(32)), (3, 4096, range(3896, 4094)), (4, 4096, range(0, 300)), (16, 200, range(16)),
    (2, 700, range(64, 700, 2)), (3, 129, range(0, 128)), (2, 40, range(40))])
def test_attention_with_scores_of_minus_infinity(T, dtype, d, causal, sq, sk, hidden):
    # keys hidden by a coordinate of minus infinity against a query coordinate of one, as padding is, anywhere among the keys
    q, k, v = rnd((3, sq, d), 1, dtype), rnd((3, sk, d), 2, dtype), rnd((3, sk, d), 3, dtype)
    q[..., 0], k[..., 0] = 1.0, 0.0
    k[:, list(hidden), 0] = -math.inf
    got, lse = T.attention(q, k, v, scale=d ** -0.5, causal=causal, return_lse=True)
    T.device_status()
    want, want_lse = attention_reference(q, k, v, d ** -0.5, causal)
    tol = 64 * F32_CELL if dtype == F32 else BF16_ROUND * (want.abs() + attention_reference(q, k, v.abs(), d ** -0.5, causal)[0]) + 1e-6
    g = d64(got)
    assert torch.equal(g.isnan(), want.isnan())   # no value where no key that a row sees has a finite score
    assert (((g - want).abs() <= tol) | want.isnan()).all()
    assert torch.equal(d64(lse).isfinite(), want_lse.isfinite()) and ((d64(lse) - want_lse).abs()[want_lse.isfinite()] <= 1e-4).all()


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (31, 65, 33), (128, 64, 512), (129, 127, 31), (600, 700, 260), (40, 30, 5000), (1500, 1301, 300)])
@pytest.mark.parametrize("b_nk,offset,out", [(True, 0, F32), (False, 0, F32), (True, 1, F32), (False, 1, BF16)])
def test_f32_products_of_any_extent(T, m, n, k, b_nk, offset, out):
    a, b = rnd((m, k), 1, F32, offset), rnd((n, k) if b_nk else (k, n), 2, F32, offset)
    b = b.t() if b_nk else b
    bias = rnd((n,), 3)
    got = T.product_2d(a, b, post="bias", bias=bias, out_dtype=out)
    T.device_status()
    scale = d64(a).abs() @ d64(b).abs() + d64(bias).abs()
    close_cells(got, d64(a) @ d64(b) + d64(bias), scale, F32_CELL if out == F32 else BF16_ROUND)


@pytest.mark.parametrize("batch,m,n,k,b_nk,offset,out", [
    (1, 1500, 1300, 300, True, 0, F32), (1, 1500, 1300, 301, False, 1, F32), (1, 1281, 1544, 257, True, 1, BF16),
    (1, 1281, 1544, 260, False, 0, BF16), (3, 1153, 1156, 515, True, 0, F32), (2, 4100, 4100, 33, False, 0, F32)])
def test_f32_products_with_many_tiles(T, batch, m, n, k, b_nk, offset, out):
    lead = (batch,) if batch > 1 else ()
    a, b = rnd(lead + (m, k), 1, F32, offset), rnd(lead + ((n, k) if b_nk else (k, n)), 2, F32, offset)
    b = b.transpose(-1, -2) if b_nk else b
    a[..., 5, 3], b[..., 7, 9] = math.inf, math.nan
    run = lambda: T.bmm(a, b) if batch > 1 else T.product_2d(a, b, out_dtype=out)
    run()
    got = run()
    T.device_status()
    want, scale = d64(a) @ d64(b), (d64(a).abs() @ d64(b).abs()).nan_to_num(0, 0, 0)
    close_cells(got, want, scale, TF32_CELL if out == F32 else BF16_ROUND)
    # a captured call holds no buffer of the library: it takes the kernel that needs none, whose error is smaller
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = run()
    graph.replay()
    T.device_status()
    close_cells(got, want, scale, F32_CELL if out == F32 else BF16_ROUND)


@pytest.mark.parametrize("out,gap", [(F32, 1), (F32, 4), (BF16, 4), (BF16, 8)])
def test_batched_f32_results_at_any_stride(T, out, gap):
    # entries of a result `gap` elements apart: 16-byte stores only where every entry starts on 16 bytes
    from mimir_b200 import _lib as L
    import ctypes as C
    batch, m, n, k = 3, 1153, 1160, 515
    a, b = rnd((batch, m, k), 1), rnd((batch, n, k), 2)
    room = torch.full((batch * (m * n + gap),), 7.0, dtype=out, device="cuda")
    d = L.GemmDesc()
    d.batch, d.m, d.n, d.k = batch, m, n, k
    d.a, d.b, d.c = a.data_ptr(), b.data_ptr(), room.data_ptr()
    d.stride_a, d.stride_b, d.stride_c = m * k, n * k, m * n + gap
    d.in_dtype, d.out_dtype, d.b_layout, d.post = L.F32, L.F32 if out == F32 else L.BF16, L.B_NK, L.POST_ID
    L.check(L.lib().mimk_gemm(C.byref(d), T._stream()), "gemm")
    T.device_status()
    room = room.view(batch, m * n + gap)
    assert (room[:, m * n:] == 7.0).all()
    bt = b.transpose(1, 2)
    close_cells(room[:, :m * n].reshape(batch, m, n), d64(a) @ d64(bt), d64(a).abs() @ d64(bt).abs(), TF32_CELL if out == F32 else BF16_ROUND)


@pytest.mark.parametrize("nk", [False, True])
@pytest.mark.parametrize("m,n,k,offset", [(1, 1, 1, 0), (17, 31, 77, 1), (1024, 10, 128, 0), (100, 130, 70, 3), (33, 100, 3, 1), (128, 257, 250, 2), (1200, 62, 129, 0)])
def test_small_f32_products_of_any_alignment(T, m, n, k, offset, nk):
    # tiles of 16 and of 32 rows, copies of 4 and of 16 bytes: one ascending fold per cell, so a corner of a product on the 64 x 64 kernel
    # (several hundred of its tiles) has the same bits
    M, N = 1280, 961
    a, b = rnd((M, k), 1, F32, offset), rnd((N, k) if nk else (k, N), 2, F32, offset)
    big = T.product_2d(a, b.t() if nk else b)
    bs = b[:n].contiguous() if nk else b[:, :n].contiguous()
    got = T.product_2d(a[:m].contiguous(), bs.t() if nk else bs)
    T.device_status()
    assert torch.equal(got, big[:m, :n])
    bd = d64(bs).t() if nk else d64(bs)
    # k roundings of an f32 sum at most
    close_cells(got, d64(a[:m]) @ bd, d64(a[:m]).abs() @ bd.abs(), k * 2.0 ** -24)


@pytest.mark.parametrize("nk", [False, True])
@pytest.mark.parametrize("m,n,k", [(416, 1121, 17), (448, 1057, 17), (448, 1057, 48), (880, 1053, 47), (960, 931, 50), (733, 635, 16), (107, 205, 188), (33, 65, 256)])
def test_small_f32_products_on_either_kernel_have_one_result(T, m, n, k, nk):
    # both sides of the lines between tiles of 32 x 32 and of 64 x 64, with copies of 4 and of 16 bytes: a corner has the same bits
    a, b = rnd((m, k), 1), rnd((n, k) if nk else (k, n), 2)
    got = T.product_2d(a, b.t() if nk else b)
    corner = b[:21].contiguous() if nk else b[:, :21].contiguous()
    part = T.product_2d(a[:33].contiguous(), corner.t() if nk else corner)
    T.device_status()
    assert torch.equal(part, got[:33, :21])
    bd = d64(b).t() if nk else d64(b)
    close_cells(got, d64(a) @ bd, d64(a).abs() @ bd.abs(), k * 2.0 ** -24)


@pytest.mark.parametrize("m,n,k,tiles", [
    (1710, 104, 233, 30), (23, 720, 472, 10), (172, 740, 340, 6), (260, 1268, 115, 3), (100, 320, 512, 20), (129, 256, 577, 15), (96, 80, 520, 30)])
def test_f32_products_dealt_out_by_pairs_and_singly_have_one_result(T, m, n, k, tiles):
    # whatever share of a tile's accumulators each CTA of a cluster has, a product has the bits of the same rows of one with more tiles (with
    # fewer than three TF32 products per term are made for)
    a, b = rnd((m, k), 1), rnd((n, k), 2)
    got, large = T.product_2d(a, b.t()), T.product_2d(torch.cat([a, rnd((128 * tiles, k), 3)]), b.t())
    T.device_status()
    assert torch.equal(got, large[:m])
    close_cells(got, d64(a) @ d64(b).t(), d64(a).abs() @ d64(b).t().abs(), F32_CELL)


def test_f32_products_keep_infinities_and_extremes(T):
    a, b = rnd((200, 600), 1), rnd((600, 300), 2)
    a[3, 5], a[7, 0], b[9, 11] = math.inf, math.nan, -math.inf
    a[100] *= 1e-30
    b[:, 30] *= 1e25
    close_cells(T.product_2d(a, b), d64(a) @ d64(b), d64(a).abs() @ d64(b).abs(), F32_CELL)


@pytest.mark.parametrize("batch,m,n,k,b_nk,out", [
    (1, 100, 130, 300, True, F32), (1, 129, 70, 5000, False, F32), (1, 300, 200, 1000, True, BF16), (1, 40, 1301, 2000, False, F32), (20, 65, 100, 700, True, F32)])
@pytest.mark.parametrize("low,high", [(1e-36, 1.0), (1e-38, 1e30), (1.0, 1e-37), (3e-42, 1e10)])
def test_f32_products_of_tiny_values(T, batch, m, n, k, b_nk, out, low, high):
    # values below 2^-109 do not fit three bf16 pieces; a third of the rows of A and of the columns of B are left as they are
    lead = (batch,) if batch > 1 else ()
    a, b = rnd(lead + (m, k), 1), rnd(lead + ((n, k) if b_nk else (k, n)), 2)
    b = b.transpose(-1, -2) if b_nk else b
    a[..., m // 3:, :] *= low
    b[..., n // 3:] *= high
    b[..., n // 2] = 0.0
    got = T.bmm(a, b, out_dtype=out) if batch > 1 else T.product_2d(a, b, out_dtype=out)
    T.device_status()
    # (near the end of its range an f32 sum is rounded to multiples of 2^-149, a bf16 result to multiples of 2^-133)
    cell, end = (F32_CELL, k * 2.0 ** -149) if out == F32 else (BF16_ROUND, 2.0 ** -133)
    close_cells(got, d64(a) @ d64(b), d64(a).abs() @ d64(b).abs() + end / cell, cell)


@pytest.mark.parametrize("n,cin,h,w,cout,kh,kw,stride,dil,pad,dtype", [
    (2, 5, 17, 23, 16, 3, 3, (1, 1), (1, 1), (1, 1), F32), (1, 33, 30, 31, 65, 3, 2, (2, 1), (1, 2), (0, 1), F32),
    (3, 16, 40, 40, 130, 1, 1, (1, 1), (1, 1), (0, 0), F32), (2, 3, 50, 41, 40, 7, 5, (2, 2), (1, 1), (3, 2), BF16),
    (9, 64, 20, 20, 96, 3, 3, (1, 1), (2, 2), (2, 2), BF16), (24, 8, 60, 60, 100, 5, 5, (1, 1), (1, 1), (4, 0), F32)])
def test_convolutions_gathered_from_the_image(T, monkeypatch, n, cin, h, w, cout, kh, kw, stride, dil, pad, dtype):
    monkeypatch.setattr(T, "CONV_CONTRACTION_MIN_WORK", 1)
    x, f = rnd((n, cin, h, w), 1, dtype), rnd((cout, cin, kh, kw), 2, dtype)
    got = T.conv(x, f, stride=stride, dilation=dil, padding=pad)
    T.device_status()
    conv = torch.nn.functional.conv2d
    want, scale = (conv(u, v, stride=stride, dilation=dil, padding=pad) for u, v in ((d64(x), d64(f)), (d64(x).abs(), d64(f).abs())))
    close_cells(got, want, scale + 1e-6, F32_CELL if dtype == F32 else BF16_ROUND)
    if dtype == F32:   # an infinity reaches the cells whose window holds it, and no other
        x[0, 0, h // 2, w // 2] = math.inf
        assert torch.equal(d64(T.conv(x, f, stride=stride, dilation=dil, padding=pad)).isfinite(),
                           conv(d64(x), d64(f), stride=stride, dilation=dil, padding=pad).isfinite())


@pytest.mark.parametrize("n,cin,h,w,cout,kh,kw,stride", [(2, 8, 64, 64, 128, 3, 3, (1, 1)), (1, 16, 65, 31, 256, 1, 5, (2, 1)), (2, 8, 30, 30, 40, 1, 1, (1, 1))])
@pytest.mark.parametrize("dtype", [BF16, F32])
def test_convolutions_with_and_without_a_patch_matrix(T, monkeypatch, n, cin, h, w, cout, kh, kw, stride, dtype):
    monkeypatch.setattr(T, "CONV_CONTRACTION_MIN_WORK", 1)
    x, f = rnd((n, cin, h, w), 1, dtype), rnd((cout, cin, kh, kw), 2, dtype)
    want, scale = (torch.nn.functional.conv2d(u, v, stride=stride) for u, v in ((d64(x), d64(f)), (d64(x).abs(), d64(f).abs())))
    for patches in (True, False):
        monkeypatch.setattr(T, "_patches_pay", lambda *sizes: patches)
        got = T.conv(x, f, stride=stride)
        T.device_status()
        close_cells(got, want, scale + 1e-6, BF16_ROUND if dtype == BF16 else TF32_CELL)


@pytest.mark.parametrize("n,cin,h,w,cout,kh,kw,stride,dil,pad,dtype", [
    (2, 3, 256, 259, 40, 32, 32, (32, 32), (1, 1), (0, 0), F32), (2, 3, 96, 128, 40, 32, 32, (32, 32), (1, 1), (0, 0), BF16),
    (3, 3, 1, 700, 33, 1, 64, (1, 2), (1, 1), (0, 5), F32), (3, 2, 1, 700, 64, 1, 64, (1, 1), (1, 1), (0, 0), BF16),
    (1, 20, 80, 9, 130, 33, 1, (1, 1), (2, 1), (3, 0), F32)])
def test_windows_too_wide_to_gather_go_through_patches(T, monkeypatch, n, cin, h, w, cout, kh, kw, stride, dil, pad, dtype):
    monkeypatch.setattr(T, "CONV_CONTRACTION_MIN_WORK", 1)
    calls, through = [], T._conv_as_contraction
    monkeypatch.setattr(T, "_conv_as_contraction", lambda *a: calls.append(1) or through(*a))
    x, f = rnd((n, cin, h, w), 1, dtype), rnd((cout, cin, kh, kw), 2, dtype)
    got = T.conv(x, f, stride=stride, dilation=dil, padding=pad)
    T.device_status()
    conv = torch.nn.functional.conv2d
    want, scale = (conv(u, v, stride=stride, dilation=dil, padding=pad) for u, v in ((d64(x), d64(f)), (d64(x).abs(), d64(f).abs())))
    close_cells(got, want, scale + 1e-6, F32_CELL if dtype == F32 else BF16_ROUND)
    assert calls and got.is_contiguous()
    other = BF16 if dtype == F32 else F32
    with pytest.raises(TypeError):
        T.conv(x, f.to(other), stride=stride, dilation=dil, padding=pad)


@pytest.mark.parametrize("n,cin,h,w,cout,kh,kw,stride,dil,pad", [
    (1, 1, 5, 7, 1, 1, 1, (1, 1), (1, 1), (0, 0)), (2, 5, 17, 23, 16, 3, 3, (1, 1), (1, 1), (1, 1)),
    (3, 33, 30, 31, 65, 3, 2, (2, 1), (1, 2), (0, 1)), (2, 64, 15, 66, 130, 3, 3, (2, 2), (1, 1), (1, 1)),
    (5, 72, 20, 70, 128, 1, 1, (2, 2), (1, 1), (0, 0)), (2, 130, 13, 9, 257, 5, 5, (3, 2), (2, 3), (4, 6)),
    (1, 64, 65, 130, 129, 1, 4, (1, 3), (1, 1), (0, 2)), (40, 16, 28, 28, 96, 3, 3, (1, 1), (1, 1), (1, 1))])
@pytest.mark.parametrize("by_tap", [0, 1])
@pytest.mark.parametrize("dtype", [F32, BF16])
def test_convolutions_over_an_image_laid_out_once(T, n, cin, h, w, cout, kh, kw, stride, dil, pad, by_tap, dtype):
    # the kernel itself, whatever the estimate says: ragged channels and filters, strided and dilated windows, tiles across images
    L = T.L
    run = L.lib()["_ZN4mimk11conv_piecesERK14mimk_conv_descP11CUstream_st"]
    run.restype, run.argtypes = C.c_int, [C.POINTER(L.ConvDesc), C.c_void_p]
    x, f = rnd((n, cin, h, w), 1, dtype), rnd((cout, cin, kh, kw), 2, dtype)
    stored = f.flatten(2).transpose(1, 2).contiguous() if by_tap else f
    oh, ow = ((e + 2 * p - d * (k - 1) - 1) // s + 1 for e, p, d, k, s in zip((h, w), pad, dil, (kh, kw), stride))
    d = L.ConvDesc()
    d.n, d.cin, d.h, d.w, d.cout, d.kh, d.kw = n, cin, h, w, cout, kh, kw
    d.stride_h, d.stride_w, d.dil_h, d.dil_w, d.pad_h, d.pad_w = *stride, *dil, *pad
    d.dtype, d.by_tap, d.x, d.filters = T._dt(x), by_tap, x.data_ptr(), stored.data_ptr()

    def conv():
        out = torch.full((n, cout, oh, ow), 7.0, dtype=dtype, device="cuda")
        d.out = out.data_ptr()
        L.check(run(C.byref(d), T._stream()), "conv")
        T.device_status()
        return out
    ref = lambda u, v: torch.nn.functional.conv2d(u, v, stride=stride, dilation=dil, padding=pad)
    close_cells(conv(), ref(d64(x), d64(f)), ref(d64(x).abs(), d64(f).abs()) + 1e-6, F32_CELL if dtype == F32 else BF16_ROUND)
    x[0, 0, h // 2, w // 2] = math.inf   # it reaches the cells whose window holds it, and no other
    assert torch.equal(d64(conv()).isfinite(), ref(d64(x), d64(f)).isfinite())


@pytest.mark.parametrize("cin,k,laid_out", [
    (15, 3, False), (17, 3, True), (24, 5, False), (24, 11, False), (32, 5, True), (32, 7, False), (56, 3, True), (64, 7, True), (72, 3, False), (128, 5, True)])
def test_f32_images_are_laid_out_where_the_error_is_no_larger(T, cin, k, laid_out):
    n, side, cout = 16, 56, 128
    d = T.L.ConvDesc()
    d.n, d.cin, d.h, d.w, d.cout, d.kh, d.kw, d.dtype = n, cin, side, side, cout, k, k, T.L.F32
    d.stride_h = d.stride_w = d.dil_h = d.dil_w = 1
    d.pad_h = d.pad_w = k // 2
    assert T.L.lib().mimk_conv_laid_out(C.byref(d), T._stream()) == laid_out


@pytest.mark.parametrize("n,cin,h,w,cout,k,pad", [(1, 16, 28, 28, 32, 3, 1), (2, 64, 20, 21, 24, 3, 0), (1, 128, 17, 16, 64, 1, 0)])
@pytest.mark.parametrize("dtype,other", [(F32, BF16), (BF16, F32)])
def test_convolutions_of_two_element_types(T, n, cin, h, w, cout, k, pad, dtype, other):
    # above the least work of the tensor cores, which take operands of one type: one fold per cell, as below it
    x, f = rnd((n, cin, h, w), 1, dtype), rnd((cout, cin, k, k), 2, other)
    got = T.conv(x, f, padding=(pad, pad))
    T.device_status()
    want, scale = (torch.nn.functional.conv2d(u, v, padding=pad) for u, v in ((d64(x), d64(f)), (d64(x).abs(), d64(f).abs())))
    close_cells(got, want, scale, cin * k * k * 2.0 ** -24 if dtype == F32 else BF16_ROUND)


@pytest.mark.parametrize("n,cin,h,w,cout,k", [(1, 8192, 4, 4, 64, 3), (2, 120, 9, 12, 32, 5), (4, 256, 28, 29, 256, 3)])
def test_bf16_convolutions_round_like_an_f32_fold(T, n, cin, h, w, cout, k):
    # off by half a unit of the result's last place and what an f32 sum may lose; operands of one sign, so that what an accumulator cuts off adds up
    x, f = rnd((n, cin, h, w), 1, BF16).abs_(), rnd((cout, cin, k, k), 2, BF16).abs_()
    got = T.conv(x, f, padding=(k // 2, k // 2))
    T.device_status()
    want = torch.nn.functional.conv2d(d64(x), d64(f), padding=k // 2)
    half_unit = 2.0 ** (want.log2().floor() - 8)
    assert ((d64(got) - want).abs() <= half_unit + F32_CELL * want).all()


@pytest.mark.parametrize("n,cin,h,w,cout,k,stride,pad", [
    (3, 16, 14, 14, 32, 3, 1, 1), (4, 65, 25, 19, 64, 5, 2, 2), (40, 24, 6, 5, 40, 3, 1, 1), (3, 128, 9, 30, 130, 1, 1, 0)])
@pytest.mark.parametrize("low,high", [(1.0, 1.0), (1e-36, 1.0), (1e-38, 1e30), (1.0, 1e-37), (3e-42, 1e10)])
@pytest.mark.parametrize("laid_out", [False, True])
def test_f32_convolutions_of_tiny_values(T, n, cin, h, w, cout, k, stride, pad, low, high, laid_out):
    # as test_f32_products_of_tiny_values, from the least work on that takes the tensor cores, gathered and over an image laid out once
    x, f = rnd((n, cin, h, w), 1), rnd((cout, cin, k, k), 2)
    x[n // 3:] *= low
    f[cout // 3:] *= high
    f[cout // 2] = 0.0
    oh, ow = (h + 2 * pad - k) // stride + 1, (w + 2 * pad - k) // stride + 1
    assert T._conv_on_tensor_cores(F32, n, cin, cout, k, k, oh, ow)
    if laid_out:
        run = T.L.lib()["_ZN4mimk11conv_piecesERK14mimk_conv_descP11CUstream_st"]
        run.restype, run.argtypes = C.c_int, [C.POINTER(T.L.ConvDesc), C.c_void_p]
        got, d = torch.empty((n, cout, oh, ow), device="cuda"), T.L.ConvDesc()
        d.n, d.cin, d.h, d.w, d.cout, d.kh, d.kw, d.dtype = n, cin, h, w, cout, k, k, T.L.F32
        d.stride_h = d.stride_w = stride
        d.pad_h = d.pad_w = pad
        d.dil_h = d.dil_w = 1
        d.x, d.filters, d.out = x.data_ptr(), f.data_ptr(), got.data_ptr()
        T.L.check(run(C.byref(d), T._stream()), "conv")
    else:
        got = T.conv(x, f, stride=(stride, stride), padding=(pad, pad))
    T.device_status()
    want, scale = (torch.nn.functional.conv2d(u, v, stride=stride, padding=pad) for u, v in ((d64(x), d64(f)), (d64(x).abs(), d64(f).abs())))
    close_cells(got, want, scale + cin * k * k * 2.0 ** -149 / F32_CELL, F32_CELL)


@pytest.mark.parametrize("n,cin,side,cout,k,tiny", [(16, 64, 30, 130, 3, 1e-40), (16, 64, 30, 128, 3, 3e-42), (16, 128, 28, 100, 5, 1e-40)])
def test_f32_convolutions_of_a_few_tiny_values(T, n, cin, side, cout, k, tiny):
    # a few positions whose cells are folded again for all filters, beside zeros and ordinary cells
    x, f = rnd((n, cin, side, side), 1), rnd((cout, cin, k, k), 2)
    x[0], x[1, :, 2:] = 0.0, 0.0
    x[0, 0, 0, 0], x[0, 3, 9, 9], x[1, 5, side - 1, side - 1] = tiny, -tiny, tiny
    d = T.L.ConvDesc()
    d.n, d.cin, d.h, d.w, d.cout, d.kh, d.kw, d.dtype = n, cin, side, side, cout, k, k, T.L.F32
    d.stride_h = d.stride_w = d.dil_h = d.dil_w = 1
    d.pad_h = d.pad_w = k // 2
    assert T.L.lib().mimk_conv_laid_out(C.byref(d), T._stream()) == 1
    got = T.conv(x, f, padding=(k // 2, k // 2))
    T.device_status()
    want, scale = (torch.nn.functional.conv2d(u, v, padding=k // 2) for u, v in ((d64(x), d64(f)), (d64(x).abs(), d64(f).abs())))
    close_cells(got, want, scale + cin * k * k * 2.0 ** -149 / F32_CELL, F32_CELL)


@pytest.mark.parametrize("m,n,k,b_nk,post,out,offset", [
    (2000, 1003, 520, True, "bias_relu", BF16, 0), (300, 257, 1031, True, None, BF16, 0), (129, 255, 1033, False, "bias", F32, 0),
    (640, 5003, 264, False, None, BF16, 0), (640, 5001, 257, True, "bias_tanh", F32, 1), (65, 2056, 512, True, None, BF16, 1),
    (3, 9001, 513, False, None, BF16, 3), (1, 8193, 1024, True, "relu", BF16, 0),
    (16, 4096, 4096, True, None, BF16, 0), (1, 520, 4104, False, None, F32, 0), (17, 130, 4096, True, "bias", BF16, 0),
    (129, 72, 4160, False, "add", BF16, 0), (31, 1000, 512, False, None, BF16, 0), (250, 1016, 1032, True, "bias", F32, 0), (128, 64, 64, True, None, F32, 0), (700, 1000, 72, True, "bias_relu", BF16, 0)])
def test_bf16_products_of_any_extent(T, m, n, k, b_nk, post, out, offset):
    a = rnd((m, k), 1, BF16, offset)
    b = rnd((n, k) if b_nk else (k, n), 2, BF16, offset)
    b = b.t() if b_nk else b
    bias = rnd((n,), 3) if post and post.startswith("bias") else None
    full = rnd((m, n), 4, out) if post == "add" else None
    got = T.product_2d(a, b, post=post, bias=bias, full=full, out_dtype=out)
    T.device_status()
    want = d64(a) @ d64(b)
    scale = d64(a).abs() @ d64(b).abs() * 2.0 ** -14   # the f32 sums, next to the rounding of the result
    want = want + (d64(bias) if bias is not None else 0) + (d64(full) if full is not None else 0)
    rounding = want.abs() * (BF16_ROUND if out == BF16 else 2.0 ** -20)
    if post and post.endswith("relu"):
        want = want.clamp(min=0)
    if post and post.endswith("tanh"):
        want = want.tanh()
    assert got.dtype == out and ((d64(got) - want).abs() <= rounding + scale + 1e-6).all()


@pytest.mark.parametrize("m,n,k", [(4864, 576, 64), (8192, 832, 72), (4865, 640, 64), (300, 320, 264)])
@pytest.mark.parametrize("offset", [1, 2, 7])
def test_bf16_results_that_start_anywhere(T, m, n, k, offset):
    # widths of whole 64s, where an odd start leaves the last element of a row to a piece without columns; nothing around the result is touched
    a, b = rnd((m, k), 1, BF16), rnd((n, k), 2, BF16)
    want = T.product_2d(a, b.t())
    room = torch.full((m * n + 64,), 7.0, dtype=BF16, device="cuda")
    d = T.L.GemmDesc()
    d.batch, d.m, d.n, d.k, d.stride_c = 1, m, n, k, m * n
    d.a, d.b, d.c = a.data_ptr(), b.data_ptr(), room.data_ptr() + 2 * offset
    d.in_dtype, d.out_dtype, d.b_layout, d.post = T.L.BF16, T.L.BF16, T.L.B_NK, T.L.POST_ID
    T.L.check(T.L.lib().mimk_gemm(C.byref(d), T._stream()), "gemm")
    T.device_status()
    assert (room[:offset] == 7.0).all() and (room[offset + m * n:] == 7.0).all()
    assert ((d64(room[offset:offset + m * n].view(m, n)) - d64(want)).abs() <= BF16_ROUND * d64(want).abs() + 1e-6).all()


@pytest.mark.parametrize("batch,m,n,k,b_nk,offset", [
    (1, 2000, 1003, 2048, True, 0), (1, 129, 255, 4001, False, 0), (1, 640, 1001, 2056, False, 1), (1, 65, 2056, 4096, True, 1), (3, 130, 203, 1030, True, 0)])
def test_f32_results_of_bf16_products_of_any_extent(T, batch, m, n, k, b_nk, offset):
    # as an f32 fold gives them (2^-20 of the terms, like an f32 product), whichever kernel the extents lead to
    lead = (batch,) if batch > 1 else ()
    a, b = rnd(lead + (m, k), 1, BF16, offset), rnd(lead + ((n, k) if b_nk else (k, n)), 2, BF16, offset)
    a.abs_(), b.abs_()   # one sign: what an accumulator cuts off adds up
    b = b.transpose(-1, -2) if b_nk else b
    got = T.bmm(a, b, out_dtype=F32) if batch > 1 else T.product_2d(a, b, out_dtype=F32)
    T.device_status()
    want = d64(a) @ d64(b)
    close_cells(got, want, want, F32_CELL)


@pytest.mark.parametrize("B,m,n,k,b_nk", [(3, 129, 255, 67, True), (5, 40, 200, 286, False), (2, 130, 64, 1000, True), (70, 16, 24, 72, False)])
def test_bf16_batches_of_any_extent(T, B, m, n, k, b_nk):
    a, b = rnd((B, m, k), 1, BF16), rnd((B, n, k) if b_nk else (B, k, n), 2, BF16)
    b = b.transpose(1, 2) if b_nk else b
    got = T.bmm(a, b)
    T.device_status()
    want = d64(a) @ d64(b)
    assert ((d64(got) - want).abs() <= want.abs() * BF16_ROUND + d64(a).abs() @ d64(b).abs() * 2.0 ** -14 + 1e-6).all()


@pytest.mark.parametrize("m,k,f,n,b_nk", [(1, 2048, 1024, 512, True), (17, 1544, 2056, 264, False), (128, 1536, 2048, 512, False), (200, 1600, 640, 520, True)])
def test_gated_mlp_of_few_rows(T, m, k, f, n, b_nk):
    x = rnd((m, k), 1, BF16)
    w = [(rnd((o, i) if b_nk else (i, o), s, BF16) * 0.05) for s, (i, o) in enumerate([(k, f), (k, f), (f, n)], 2)]
    w = [t.t() if b_nk else t for t in w]
    got = T.mlp_gated(x, *w)
    T.device_status()
    h = torch.nn.functional.silu(d64(x) @ d64(w[0])) * (d64(x) @ d64(w[1]))
    want, terms = h @ d64(w[2]), h.abs() @ d64(w[2]).abs()
    # the hidden layer is rounded to bf16: 2^-9 of every term, like the result itself
    assert ((d64(got) - want).abs() <= BF16_ROUND * (want.abs() + terms) + 1e-6).all()


@pytest.mark.parametrize("m,panels,kp,n", [(300, 8, 256, 264), (16, 4, 512, 2048), (129, 2, 1024, 72), (5, 16, 64, 1000)])
@pytest.mark.parametrize("b_nk", [True, False])
def test_products_of_few_tiles_keep_their_bits_as_panels_and_gathered(T, m, panels, kp, n, b_nk):
    from mimir_b200 import _lib as L
    import ctypes as C
    k = panels * kp
    a, b, b2 = rnd((m, k), 1, BF16), rnd((n, k) if b_nk else (k, n), 2, BF16), rnd((n, k) if b_nk else (k, n), 3, BF16)
    want = T.product_2d(a, b.t() if b_nk else b)
    got = T.product_2d_panels(a.view(m, panels, kp).transpose(0, 1).contiguous(), b.t() if b_nk else b)
    T.device_status()
    assert torch.equal(got, want)
    # the gated block's hidden layer, and both gathered into three copies of a wider matrix
    hidden = torch.empty((m, n), dtype=BF16, device="cuda")
    w2 = rnd((8, n) if b_nk else (n, 8), 4, BF16)
    T.mlp_gated(a, *((w.t() if b_nk else w) for w in (b, b2, w2)), h=hidden)
    for second, whole in ((None, want), (b2, hidden)):
        copies = [torch.full((m, n + 24), 3.0, dtype=BF16, device="cuda") for _ in range(3)]
        d = L.GemmDesc()
        d.batch, d.m, d.n, d.k = 1, m, n, k
        d.a, d.b = a.data_ptr(), b.data_ptr()
        d.in_dtype, d.out_dtype, d.b_layout, d.post = L.BF16, L.BF16, L.B_NK if b_nk else L.B_KN, L.POST_ID
        g = L.GatherDst()
        g.n_dst, g.ldc, g.col_off = 3, n + 24, 8
        for i, t in enumerate(copies):
            g.dst[i] = t.data_ptr()
        L.check(L.lib().mimk_gemm_gather(C.byref(d), second.data_ptr() if second is not None else None, C.byref(g), T._stream()), "gather")
        T.device_status()
        for t in copies:
            assert torch.equal(t[:, 8:8 + n], whole) and (t[:, :8] == 3.0).all() and (t[:, 8 + n:] == 3.0).all()


def test_two_streams_at_once_give_what_one_gives(T):
    # kernels with clusters, with copies in the library's buffer (one per stream) and without, two callers beside one another
    def work(i):
        bf, f = (lambda *shape: rnd(shape, i, BF16)), (lambda *shape: rnd(shape, i + 50))
        a, b, w = bf(300, 1031), bf(257, 1031), bf(2048, 16)
        x, y, q, k = f(1280, 516), f(516, 1284), f(3, 130, 64), f(3, 200, 64)
        few, keys, image, filters = bf(4, 3, 128), bf(4, 900, 128), f(12, 16, 40, 40), f(64, 16, 3, 3)
        return lambda: [T.product_2d(a, b.t()), T.product_2d(w.t(), bf2), T.product_2d(x, y), T.attention(q, k, k, scale=0.1),
                        T.attention(few, keys, keys, scale=0.1, causal=True), T.conv(image, filters, padding=(1, 1)),
                        T.product_2d(x[:200], y[:, :300].contiguous())]
    bf2 = rnd((2048, 1000), 7, BF16)
    calls = [work(1), work(2)]
    want = [c() for c in calls]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in calls]
    for _ in range(4):
        got = []
        for c, s in zip(calls, streams):
            with torch.cuda.stream(s):
                got.append(c())
        torch.cuda.synchronize()
        for g, w in zip(got, want):
            assert all(torch.equal(u, v) for u, v in zip(g, w))
    T.device_status()


def test_two_threads_on_one_stream_give_what_one_gives(T):
    # calls of two launches that meet in the stream's cached buffer, of different sizes, so that it also grows under them
    import threading
    x = [rnd((n, 64, 56, 56), n) for n in (14, 9)]
    f, q = rnd((128, 64, 3, 3), 7), [rnd((n, 700, 64), 40 + n) for n in (6, 11)]
    b = [rnd((1000, 301), i, BF16) for i in (1, 2)]
    calls = [lambda i=i: [T.conv(x[i], f, padding=(1, 1)), *T.attention(q[i], q[i], q[i], scale=0.1, return_lse=True), T.attention(q[i], q[i], q[i], scale=0.1),
                          T.product_2d(b[i], b[i].t())] for i in range(2)]
    want = [c() for c in calls]
    torch.cuda.synchronize()
    got, errors = [[], []], []

    def work(i):
        try:
            got[i] = [calls[i]() for _ in range(60)]
        except Exception as e:   # noqa: BLE001 -- shown by the main thread
            errors.append(e)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    T.device_status()
    assert not errors
    for g, w in zip(got, want):
        assert len(g) == 60 and all(torch.equal(u, v) for one in g for u, v in zip(one, w))


def test_a_handle_that_names_a_stream_per_thread(T):
    # cudaStreamPerThread is another stream in each thread: calls of two launches do not meet in one buffer there
    import threading
    per_thread, convs = 2, []
    for n in (14, 9):
        x, f = rnd((n, 64, 56, 56), n), rnd((128, 64, 3, 3), 7 + n)
        outs = [torch.empty((n, 128, 56, 56), device="cuda") for _ in range(21)]
        d = T.L.ConvDesc()
        d.n, d.cin, d.h, d.w, d.cout, d.kh, d.kw, d.dtype = n, 64, 56, 56, 128, 3, 3, T.L.F32
        d.stride_h = d.stride_w = d.dil_h = d.dil_w = d.pad_h = d.pad_w = 1
        d.x, d.filters = x.data_ptr(), f.data_ptr()
        assert T.L.lib().mimk_conv_laid_out(C.byref(d), T._stream()) == 1
        convs.append((d, outs, x, f))
    statuses = [[], []]

    def run(i, outs, stream):
        d = convs[i][0]
        for out in outs:
            d.out = out.data_ptr()
            statuses[i].append(T.L.lib().mimk_conv(C.byref(d), stream))
    for i in range(2):
        run(i, convs[i][1][:1], T._stream())
    torch.cuda.synchronize()
    threads = [threading.Thread(target=run, args=(i, convs[i][1][1:], per_thread)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    T.device_status()
    for (_, outs, _, _), status in zip(convs, statuses):
        assert status == [0] * 21 and all(torch.equal(out, outs[0]) for out in outs[1:])


@pytest.mark.parametrize("what", ["reduce", "mlp", "attention", "scatter"])
def test_calls_that_have_their_buffer_may_be_captured(T, what):
    x, h, q = rnd((1, 60000, 8), 1), [rnd(s, 2, BF16) for s in ((256, 512), (512, 512), (512, 512), (512, 256))], rnd((4, 512, 160), 3)
    big, index, updates = rnd((5000, 8), 4), (rnd((5000, 8), 5).abs() * 40).long().clamp_(max=4999), rnd((5000, 8), 6)
    call = {"reduce": lambda: T.reduce("sum", 1, x), "mlp": lambda: T.mlp_gated(*h), "attention": lambda: T.attention(q, q, q, scale=0.1),
            "scatter": lambda: T.scatter(0, big, index, updates)}[what]
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        want = call()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            got = call()
    graph.replay()
    torch.cuda.synchronize()
    T.device_status()
    assert torch.equal(got, want)
