"""Slice products in every tile width of every slice count, on operands whose
slices are exact: what a wrong level, column or piece of a product changes is
larger than the tolerance at any slice count."""
import numpy as np
import pytest

from libtensor_b200.core import (MODE_OZAKI_BF16, MODE_OZAKI_FP8, MODE_OZAKI_INT8, Context, block_tensor,
                                 btod_contract2, contraction2)
from libtensor_b200.spec import BTSpec

pytestmark = pytest.mark.gpu

KS = [1100, 33]                 # more than one accumulation chunk of BF16 and FP8


def widest(slices):
    """Level accumulators of `slices` levels in 512 columns, at most 128 each."""
    return min(512 // slices // 16 * 16, 128)


def tile_width(rows, slices):
    """The width the products take for `rows` columns: fewest clocks per k block,
    a tile costing its products or the copy of its operand images."""
    def clocks(nt):
        return max(0.25 * slices * (slices + 1) * nt, slices * (4096 + 32 * nt) / 42.0)
    widths = range(16, widest(slices) + 1, 16)
    return min(reversed(widths), key=lambda nt: -(-rows // nt) * clocks(nt))


def _digits(rng, rows, k, top, beta, slices):
    """Rows of one digit each (|d| <= top, the first slice's largest) in one of
    `slices` slices; the first element sets the row's scale."""
    x = rng.integers(-top, top + 1, (rows, k)).astype(float)
    x *= 2.0 ** (beta * rng.integers(0, slices, (rows, k)))
    x[:, 0] = top * 2.0 ** (beta * (slices - 1))
    return x


def _matrix(ctx, x):
    t = block_tensor(ctx, BTSpec(dims=list(x.shape), splits=[[], [KS[0]]]))
    for bidx, blk in t.blocks(np.zeros(t.nelems)):
        k0 = sum(KS[:bidx[1]])
        t.set_block(bidx, x[:, k0:k0 + blk.shape[1]])
    return t


@pytest.mark.parametrize("mode,top,beta", [(MODE_OZAKI_INT8, 63, 7), (MODE_OZAKI_BF16, 63, 7), (MODE_OZAKI_FP8, 15, 5)],
                         ids=["int8", "bf16", "fp8"])
@pytest.mark.parametrize("slices", range(1, 9))
def test_every_width_exactly(mode, top, beta, slices):
    """640 rows along the MMA rows, `width` along its columns, either operand
    first.  One side fills p slices, the other S + 1 - p, so no product lies
    beyond the levels that are formed and the result is exact up to FP64
    rounding of the sums (numpy's too): (K + 4) 2^-53 of the magnitudes."""
    ctx = Context(0)
    rng = np.random.default_rng(slices)
    for width in range(16, widest(slices) + 1, 16):
        assert tile_width(width, slices) == width
        for p in sorted({1, (slices + 1) // 2, slices}):
            a = _digits(rng, 640, sum(KS), top, beta, p)
            b = _digits(rng, width, sum(KS), top, beta, slices + 1 - p)
            a[5] = 0.0
            for x, y in ((a, b), (b, a)):
                X, Y = _matrix(ctx, x), _matrix(ctx, y)
                op = btod_contract2(contraction2(1, 1, 1).contract(1, 1), X, Y)
                C = op.make_result()
                op.perform(C, mode=mode, nslices=slices)
                ctx.synchronize()
                got = C.get_block((0, 0), (len(x), len(y)))
                tol = (sum(KS) + 4) * 2.0 ** -53 * (np.abs(x) @ np.abs(y).T)
                assert np.all(np.abs(got - x @ y.T) <= tol), (width, p, len(x))
                for t in (op, C, X, Y):
                    t.close()
    ctx.close()


def test_width_of_the_four_slice_ladder():
    """400 rows in 4 slices take 112 columns: pieces of 224, 224 | 168, 168 |
    224 and 112 columns, 56 columns per half of the epilogue."""
    assert tile_width(400, 4) == 112
