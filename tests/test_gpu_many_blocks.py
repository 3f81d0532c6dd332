"""Plain FP64 products of stacks with hundreds to thousands of small C blocks."""
import numpy as np
import pytest

from libtensor_b200.core import Context, block_tensor, btod_contract2, contraction2
from libtensor_b200.spec import BTSpec

pytestmark = pytest.mark.gpu


def _cut(total, sizes):
    """Inner block boundaries of extents that repeat `sizes` up to `total`."""
    at, k = [sizes[0]], 1
    while at[-1] < total:
        at.append(at[-1] + sizes[k % len(sizes)])
        k += 1
    return at[:-1]


def _product(ctx, m, n, k, rows, cols, split=0):
    """(operation, result, operands, dense operands): rows and columns cut into
    the given extents, grouping off, so that the blocks form one stack."""
    out = []
    for d, sizes, seed in ((m, rows, 1), (n, cols, 2)):
        t = block_tensor(ctx, BTSpec(dims=[d, k], splits=[_cut(d, sizes), []]))
        x = np.random.default_rng(seed).standard_normal((d, k))
        arena = np.zeros(t.nelems)
        at = [0] + _cut(d, sizes)
        for bidx, blk in t.blocks(arena):
            blk[...] = x[at[bidx[0]]:at[bidx[0]] + blk.shape[0]]
        t.upload(arena)
        out.append((t, x))
    (A, a), (B, b) = out
    op = btod_contract2(contraction2(1, 1, 1).contract(1, 1), A, B)
    op.set_grouping(False)
    op.set_split_k(split)
    return op, op.make_result(), (A, B), (a, b)


@pytest.mark.parametrize("split", [1, 2])
@pytest.mark.parametrize("m,n,rows,cols", [(700, 90, [1], [90]), (90, 700, [90], [1]), (331, 257, [1, 2, 5], [3, 1, 40]),
                                           (515, 130, [127, 1], [2, 64, 1])],
                         ids=["rows of one", "columns of one", "grid", "tile edges"])
def test_stacks_of_many_blocks(m, n, rows, cols, split):
    """Each element within (K + 4) 2^-53 of its sum of magnitudes."""
    ctx = Context(0)
    op, C, ops, (a, b) = _product(ctx, m, n, 70, rows, cols, split)
    op.perform(C)
    op.perform(C, 2.0)
    ctx.synchronize()
    got = np.zeros((m, n))
    r0, c0 = [0] + _cut(m, rows), [0] + _cut(n, cols)
    for bidx, blk in C.blocks(C.download()):
        got[r0[bidx[0]]:r0[bidx[0]] + blk.shape[0], c0[bidx[1]]:c0[bidx[1]] + blk.shape[1]] = blk
    want, mag = 3.0 * a @ b.T, 3.0 * np.abs(a) @ np.abs(b).T
    assert np.all(np.abs(got - want) <= 74 * 2.0 ** -53 * mag)
    for x in (op, C, *ops):
        x.close()
    ctx.close()


def test_a_stack_of_many_blocks_is_not_slower_than_its_blocks_one_by_one():
    """48000 rows as one block (51 us) and as 48000 blocks of a row: one product
    per block takes 30 times as long (2.1 ms), a stack 11 times; counting up to
    each tile's first block made it 223 times.  The bound has a third to spare
    over the products one by one."""
    ctx = Context(0)
    best = []
    for rows in ([48000], [1]):
        op, C, ops, _ = _product(ctx, 48000, 64, 64, rows, [64], 1)
        for _ in range(3):
            op.perform(C)
        ctx.set_timing(True)
        for _ in range(20):
            op.perform(C)
        best.append(ctx.kernel_times()["contract_fp64"][0])
        ctx.set_timing(False)
        for x in (op, C, *ops):
            x.close()
    assert best[1] <= 40 * best[0], best
    ctx.close()
