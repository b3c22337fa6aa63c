"""GPU parity at the edges of tiles, alignments and splits: contractions with ragged extents and with few tiles, f32 products and
attention on the tensor cores, attention of a few queries, convolutions gathered from the image, folds and maps with remainders.
References are float64 on the CPU."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

BF16, F32 = torch.bfloat16, torch.float32
# a bf16 result is off by half a unit in its last place, 2^-9 of its value, and by what f32 sums of up to 4096 terms lose
BF16_ROUND = 2.0 ** -8
# an f32 product cut into bf16 pieces leaves out less than 2^-22 of each |a b|, its sums and the accumulators' updates lose no more
F32_CELL = 2.0 ** -20


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
