"""Slice modes at the edges of their tiles: one MMA row tile is 128 rows, the
other side is cut into tiles of 16..128 columns by the slice count, and either
C side can take either place."""
import numpy as np
import pytest

from libtensor_b200.core import (MODE_OZAKI_BF16, MODE_OZAKI_FP8, MODE_OZAKI_INT8, Context, block_tensor,
                                 btod_contract2, contraction2)
from libtensor_b200.spec import BTSpec

pytestmark = pytest.mark.gpu

# C(i,j) = sum_k A(i,k) B(j,k): rows, columns, contracted blocks
SHAPES = [(1, 1, [1]), (16, 130, [32, 7]), (129, 65, [33]), (113, 128, [100, 31]), (400, 257, [1030]), (257, 400, [640, 390])]


def _matrix(ctx, rows, ks, x):
    t = block_tensor(ctx, BTSpec(dims=[rows, sum(ks)], splits=[[], [int(s) for s in np.cumsum(ks)[:-1]]]))
    for bidx, blk in t.blocks(np.zeros(t.nelems)):
        k0 = sum(ks[:bidx[1]])
        t.set_block(bidx, x[:, k0:k0 + blk.shape[1]])
    return t


@pytest.mark.parametrize("mode,beta", [(MODE_OZAKI_INT8, 7), (MODE_OZAKI_BF16, 7), (MODE_OZAKI_FP8, 5)],
                         ids=["int8", "bf16", "fp8"])
@pytest.mark.parametrize("slices", range(1, 9))
def test_slice_products_at_tile_edges(mode, beta, slices):
    """Slices of beta bits (the first of beta - 1 and a sign): an operand's
    dropped tail is at most 2^-(beta S) of its row's power-of-two bound, at
    most S products of 2^-(beta l) per dropped level l >= S, so an element is
    within K 2^(e_row + e_col) (S + 3) 2^-(beta S), 2^e at most twice the
    largest magnitude, and FP64 rounding."""
    ctx = Context(0)
    rng = np.random.default_rng(slices)
    for m, n, ks in SHAPES:
        a, b = rng.standard_normal((m, sum(ks))), rng.standard_normal((n, sum(ks)))
        a[m // 2] = 0.0                                  # a row without elements
        A, B = _matrix(ctx, m, ks, a), _matrix(ctx, n, ks, b)
        op = btod_contract2(contraction2(1, 1, 1).contract(1, 1), A, B, kc=-0.5)
        C = op.make_result()
        op.perform(C, mode=mode, nslices=slices)
        op.perform(C, 2.0, mode=mode, nslices=slices)
        ctx.synchronize()
        got = C.get_block((0, 0), (m, n))
        scale = sum(ks) * np.abs(a).max() * np.abs(b).max()
        bound = 1.5 * scale * (4.0 * (slices + 3) * 2.0 ** (-beta * slices) + 1e-14)
        assert np.abs(got + 1.5 * (a @ b.T)).max() <= bound, (m, n, ks)
        for x in (op, C, A, B):
            x.close()
    ctx.close()
