"""Symmetrizers fused into the contraction, every arithmetic mode, against dense
numpy: small blocks through the grouped products' and the modular
recombination's scatter, larger ones with either C side along the tile rows."""
import numpy as np
import pytest

from libtensor_b200.core import (MODE_OZAKI_BF16, MODE_OZAKI_CRT, MODE_OZAKI_FP8, MODE_OZAKI_INT8, MODE_PLAIN_FP64,
                                 Context, block_tensor, btod_contract2, contraction2)
from libtensor_b200.spec import BTSpec

pytestmark = pytest.mark.gpu

# error of one term relative to K times the operands' largest elements: slices
# of beta bits drop 2^-(beta S) per operand and dropped level (S + 3 of them) of
# a bound twice the largest element on either side; modular rounds operands to 43
# bits or more of a bound four times theirs
MODES = [(MODE_PLAIN_FP64, 0, 2.0 ** -52), (MODE_OZAKI_CRT, 13, 16 * 2 * 2.0 ** -44), (MODE_OZAKI_CRT, 8, 16 * 2 * 2.0 ** -25),
         (MODE_OZAKI_INT8, 7, 4 * 10 * 2.0 ** -49), (MODE_OZAKI_BF16, 7, 4 * 10 * 2.0 ** -49),
         (MODE_OZAKI_FP8, 8, 4 * 11 * 2.0 ** -40)]
IDS = ["plain", "modular13", "modular8", "int8", "bf16", "fp8"]

# blocks of i and j, of a and b, of k; grouped or not
SHAPES = [([5, 3], [20, 7], [40, 9], True), ([5, 3], [20, 7], [40, 9], False), ([20, 7], [5, 3], [1100, 9], False),
          ([3], [16, 5, 1], [33], False), ([12, 1], [4], [64], True)]


def _tensor(ctx, x, cuts):
    t = block_tensor(ctx, BTSpec(dims=list(x.shape), splits=[[int(s) for s in np.cumsum(c)[:-1]] for c in cuts]))
    for bidx, blk in t.blocks(np.zeros(t.nelems)):
        t.set_block(bidx, x[_at(bidx, blk.shape, cuts)])
    return t


def _at(bidx, shape, cuts):
    return tuple(slice(sum(c[:b]), sum(c[:b]) + n) for b, n, c in zip(bidx, shape, cuts))


@pytest.mark.parametrize("mode,slices,eps", MODES, ids=IDS)
@pytest.mark.parametrize("ij,ab,k,group", SHAPES, ids=["grouped", "wide", "tall", "one row block", "one column block"])
def test_symmetrized_contraction(ij, ab, k, group, mode, slices, eps):
    """r(i,j,a,b) = c (T(i,j,a,b) + s T(P(i,j,a,b))), T = sum_k A(i,j,k) B(a,b,k)."""
    ctx = Context(0)
    rng = np.random.default_rng(len(ij) + 10 * len(ab))
    ni, na, nk = sum(ij), sum(ab), sum(k)
    x, y = rng.standard_normal((ni, ni, nk)), rng.standard_normal((na, na, nk))
    A, B = _tensor(ctx, x, [ij, ij, k]), _tensor(ctx, y, [ab, ab, k])
    op = btod_contract2(contraction2(2, 2, 1).contract(2, 2), A, B)
    op.set_grouping(group)
    t = np.einsum("ijk,abk->ijab", x, y)
    bound = 2 * 0.5 * nk * np.abs(x).max() * np.abs(y).max() * (eps + nk * 2.0 ** -52)
    for symm, kw, perm in ((False, dict(idx=(0, 1)), (1, 0, 2, 3)), (True, dict(idx=(2, 3)), (0, 1, 3, 2)),
                           (True, dict(perm=(1, 0, 3, 2)), (1, 0, 3, 2))):
        r = op.make_symmetrized(symm, **kw)
        r.upload(np.full(r.nelems, 7.0))                 # the call overwrites it
        op.perform_symmetrized(r, symm, c=0.5, mode=mode, nslices=slices, **kw)
        ctx.synchronize()
        want = 0.5 * (t + (1 if symm else -1) * t.transpose(perm))
        for bidx, blk in r.blocks(r.download()):
            assert np.abs(blk - want[_at(bidx, blk.shape, [ij, ij, ab, ab])]).max() <= bound, (kw, bidx)
        r.close()
    for z in (op, A, B):
        z.close()
    ctx.close()
