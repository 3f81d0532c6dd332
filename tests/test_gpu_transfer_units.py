"""Transfers large enough for the staged tiles and for several units per job, and
the time of a transpose in many small blocks."""
from itertools import permutations

import numpy as np
import pytest

from libtensor_b200.core import Context, block_tensor, btod_add, btod_copy, btod_dotprod
from libtensor_b200.spec import BTSpec, permuted_spec

pytestmark = pytest.mark.gpu


def _spec(sizes, order):
    return BTSpec(dims=[sum(sizes)] * order, splits=[[int(x) for x in np.cumsum(sizes)[:-1]]] * order)


def _dense(t, arena, sizes):
    x = np.zeros([sum(sizes)] * t.order)
    at = np.concatenate([[0], np.cumsum(sizes)])
    for bidx, blk in t.blocks(arena):
        x[tuple(slice(at[b], at[b] + n) for b, n in zip(bidx, blk.shape))] = blk
    return x


# above 2^19 elements: planes of 1024 elements or more in tiles, smaller ones in
# place, and both; rows cut into chunks; one block and many
@pytest.mark.parametrize("order,sizes", [(2, [900]), (2, [33, 500, 200]), (3, [40, 60]), (3, [31, 70, 5]), (4, [33]),
                                         (4, [20, 13])], ids=str)
def test_large_permuted_copies_and_sums(order, sizes):
    """Copies must be exact; a sum of T terms in T multiply-adds is within
    (T + 1) 2^-53 of the sum of magnitudes; the dot product of N terms within
    N 2^-53 of it."""
    ctx = Context(0)
    spec = _spec(sizes, order)
    a = block_tensor(ctx, spec)
    arena = np.random.default_rng(order).standard_normal(a.nelems)
    a.upload(arena)
    x = _dense(a, arena, sizes)
    perms = list(permutations(range(order)))
    for p in perms:
        b = block_tensor(ctx, permuted_spec(spec, p))
        btod_copy(a, p, -1.0).perform(b)
        btod_copy(a, p, 1.0).perform(b, 3.0)                     # -x + 3 x
        assert np.array_equal(_dense(b, b.download(), sizes), 2.0 * x.transpose(p)), p
        e = btod_dotprod(a, p, b, None).calculate()
        assert abs(e - 2.0 * np.sum(x * x)) <= 2.0 * x.size * 2.0 ** -53 * np.sum(x * x)
        b.close()
    for terms in (2, 4, 6):
        use = (perms[::-1] + perms * 3)[:terms]
        cs = [(-0.5) ** k for k in range(terms)]
        op = btod_add(a, use[0], cs[0])
        for p, c in zip(use[1:], cs[1:]):
            op.add_op(a, p, c)
        b = block_tensor(ctx, spec)
        op.perform(b)
        want = sum(c * x.transpose(p) for p, c in zip(use, cs))
        mag = sum(abs(c) * np.abs(x.transpose(p)) for p, c in zip(use, cs))
        assert np.all(np.abs(_dense(b, b.download(), sizes) - want) <= (terms + 1) * 2.0 ** -53 * mag)
        b.close()
    a.close()
    ctx.close()


def test_transpose_in_blocks_just_below_the_tiled_size():
    """Blocks of 28 read in place against blocks of 32 in staged tiles, 1.5e7
    elements: the same bytes and 1.3 times the blocks.  163 and 166 us; with one
    warp of a CTA to a block 381."""
    ctx = Context(0)
    took = []
    for s in (32, 28):
        spec = _spec([s] * (3840 // s), 2)
        a, b = block_tensor(ctx, spec), block_tensor(ctx, spec)
        a.fill_seeded(1, 1.0)
        op = btod_copy(a, (1, 0), 1.0)
        for _ in range(3):
            op.perform(b)
        ctx.set_timing(True)
        for _ in range(10):
            op.perform(b)
        took.append(ctx.kernel_times()["transfer"][0])
        ctx.set_timing(False)
        a.close(); b.close()
    assert took[1] <= 1.6 * took[0], took
    ctx.close()
