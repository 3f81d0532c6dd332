"""Plain FP64 products of stacked C blocks: tiles that several blocks share, in
every tile shape, with and without k chunks, and grids with missing blocks."""
import numpy as np
import pytest

from libtensor_b200 import spec as S
from libtensor_b200.core import Context, block_tensor, btod_contract2, contraction2
from oracle import restate as X

pytestmark = pytest.mark.gpu

CFG = S.LadderConfig("stacked", [3, 2, 4], [7, 4, 1])


@pytest.fixture(scope="module")
def case():
    ctx = Context(0)
    A, B = block_tensor(ctx, CFG.t_spec()), block_tensor(ctx, CFG.v_spec())
    A.upload(A.fill_seeded_host(11, 1.0))
    B.upload(B.fill_seeded_host(23, 1.0))
    a, b = X.seeded_dense(CFG.t_spec(), 11, 1.0), X.seeded_dense(CFG.v_spec(), 23, 1.0)
    yield ctx, A, B, a, b
    A.close(); B.close(); ctx.close()


def _plan(A, B):
    return btod_contract2(contraction2(2, 2, 2).contract(2, 2).contract(3, 3), A, B, kc=0.5)


def _starts(spec):
    return [[0] + list(s) for s in spec.splits]


def _check(C, arena, a, b, times):
    """Each element within (K + 4) 2^-53 of its sum of magnitudes."""
    K = a.shape[2] * a.shape[3]
    want = 0.5 * times * np.einsum("ijcd,abcd->ijab", a, b)
    mag = 0.5 * times * np.einsum("ijcd,abcd->ijab", np.abs(a), np.abs(b))
    st = _starts(CFG.t_spec())
    for bidx, blk in C.blocks(arena):
        at = tuple(slice(st[d][x], st[d][x] + blk.shape[d]) for d, x in enumerate(bidx))
        assert np.all(np.abs(blk - want[at]) <= (K + 4) * 2.0 ** -53 * mag[at]), bidx


@pytest.mark.parametrize("split", [0, 1, 3])
@pytest.mark.parametrize("tile", range(-1, 22))
def test_stacks_in_every_tile_shape(case, tile, split):
    ctx, A, B, a, b = case
    op = _plan(A, B)
    op.set_tile(tile)
    op.set_split_k(split)
    C = op.make_result()
    op.perform(C)
    op.perform(C, 2.0)
    _check(C, C.download(), a, b, 3.0)
    C.close(); op.close()


def test_stack_with_missing_blocks(case):
    """A zero amplitude block shortens the pair lists of its C blocks and leaves
    the grid of the others; the antisymmetrised result goes to its destinations
    from the same tiles."""
    ctx, A, B, a, b = case
    t = A.permuted((0, 1, 2, 3))
    t.upload(A.download())
    t.zero_block((0, 1, 0, 1))
    z, st = a.copy(), _starts(CFG.t_spec())
    sizes = [np.diff(s + [d]) for s, d in zip(st, CFG.t_spec().dims)]
    for p, _ in X.perm_group(4, CFG.t_spec().perms):
        blk = [(0, 1, 0, 1)[q] for q in p]
        z[tuple(slice(st[d][x], st[d][x] + sizes[d][x]) for d, x in enumerate(blk))] = 0.0
    op = _plan(t, B)
    C = op.make_result()
    op.perform(C)
    _check(C, C.download(), z, b, 1.0)
    R = op.make_symmetrized(False, perm=(1, 0, 3, 2))
    op.perform_symmetrized(R, False, perm=(1, 0, 3, 2))
    # C is symmetric under the pair exchange, so its antisymmetriser vanishes
    assert not np.any(R.download())
    R2 = op.make_symmetrized(True, perm=(1, 0, 3, 2))
    op.perform_symmetrized(R2, True, perm=(1, 0, 3, 2), c=0.5)
    _check(R2, R2.download(), z, b, 1.0)
    for x in (R, R2, C, op, t):
        x.close()
