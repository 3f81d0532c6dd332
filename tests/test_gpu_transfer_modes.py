"""Copies and adds where the ways of moving a block meet: rows, staged tiles and
small planes read directly, with extents from 1 to just above a plane of 1024
elements, and transfers from a few elements to many units."""
from itertools import permutations

import numpy as np
import pytest

from libtensor_b200.core import Context, block_tensor, btod_add, btod_copy, btod_dotprod
from libtensor_b200.spec import BTSpec, permuted_spec

pytestmark = pytest.mark.gpu

# block extents per dimension (all dims of one tensor are cut alike, so that
# every permutation maps it onto itself)
SIZES = [[1, 2], [5], [4, 33], [31, 1], [32, 33], [8, 65]]


def _dense(t, arena, dims):
    x = np.zeros(dims)
    starts = [np.concatenate([[0], np.cumsum([t.block_dims([b if e == d else 0 for e in range(t.order)])[d]
                                              for b in range(t.bidims[d])])]) for d in range(t.order)]
    for bidx, blk in t.blocks(arena):
        x[tuple(slice(starts[d][b], starts[d][b] + blk.shape[d]) for d, b in enumerate(bidx))] = blk
    return x


@pytest.mark.parametrize("sizes", SIZES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_permuted_copies_and_adds(sizes, order):
    """Copies must be exact; a sum of T terms in T multiply-adds is within
    (T + 1) 2^-53 of the sum of magnitudes."""
    n = sum(sizes)
    if n ** order > 3_000_000:
        pytest.skip("covered by the lower orders")
    ctx = Context(0)
    spec = BTSpec(dims=[n] * order, splits=[[int(x) for x in np.cumsum(sizes)[:-1]]] * order)
    a = block_tensor(ctx, spec)
    rng = np.random.default_rng(order)
    arena = rng.standard_normal(a.nelems)
    a.upload(arena)
    x = _dense(a, arena, spec.dims)
    perms = list(permutations(range(order)))
    for p in perms:
        b = block_tensor(ctx, permuted_spec(spec, p))
        btod_copy(a, p, -1.0).perform(b)
        btod_copy(a, p, 1.0).perform(b, 3.0)                     # -x + 3 x
        got = _dense(b, b.download(), spec.dims)
        assert np.array_equal(got, 2.0 * x.transpose(p)), p
        e = btod_dotprod(a, p, b, None).calculate()
        assert abs(e - 2.0 * np.sum(x * x)) <= 1e-12 * np.sum(x * x)
        b.close()
    for terms in (2, 3, 4, min(8, len(perms))):
        use = (perms[::-1] + perms)[:terms]
        cs = [(-0.5) ** k for k in range(len(use))]
        op = btod_add(a, use[0], cs[0])
        for p, c in zip(use[1:], cs[1:]):
            op.add_op(a, p, c)
        b = block_tensor(ctx, spec)
        op.perform(b)
        want = sum(c * x.transpose(p) for p, c in zip(use, cs))
        mag = sum(abs(c) * np.abs(x.transpose(p)) for p, c in zip(use, cs))
        assert np.all(np.abs(_dense(b, b.download(), spec.dims) - want) <= (len(use) + 1) * 2.0 ** -53 * mag)
        b.close()
    a.close()
    ctx.close()
