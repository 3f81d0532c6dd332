"""Modular mode: rows of C fed by long (sampled) and short panels together."""
import numpy as np
import pytest

from libtensor_b200 import spec as S
from libtensor_b200.core import MODE_OZAKI_CRT, Context, block_tensor, btod_contract2, contraction2

pytestmark = pytest.mark.gpu


def _worst(got, want, t):
    """Largest block error relative to its block's largest element."""
    worst = 0.0
    for (_, g), (_, w) in zip(t.blocks(got), t.blocks(want)):
        m = float(np.max(np.abs(w))) if w.size else 0.0
        if m > 0:
            worst = max(worst, float(np.max(np.abs(g - w))) / m)
    return worst


@pytest.mark.parametrize("vir", [[34, 28], [34, 28, 5]], ids=["rows", "rows and core tiles"])
def test_redone_rows_take_their_short_panels_along(vir):
    """Rows of C fed by sampled panels (34 x 34 = 1156 contracted words) and by
    panels too short to be sampled (34 x 28; 28 x 5 and 5 x 5 in core tiles):
    when a row's sampled bound is too small, both kinds must be redone with the
    row's exact exponent, as the recombination scales the row once.  Every
    long V row gets an element 2^13 times its block's magnitude between the
    sampled runs; residues of one row scaled two ways would give errors of
    order one, consistent ones keep P - 13 - 1 > 28 bits of the other
    elements, hence 2^-28 < 1e-8."""
    ctx = Context(0)
    cfg = S.LadderConfig("mixed", [3], vir)
    A, B = block_tensor(ctx, cfg.t_spec()), block_tensor(ctx, cfg.v_spec())
    A.fill_seeded(11, cfg.t_scale)
    arena = B.fill_seeded_host(23, cfg.v_scale)
    for bidx, blk in B.blocks(arena):
        rows = blk.reshape(blk.shape[0] * blk.shape[1], -1)
        if rows.shape[1] >= 1024:
            rows[:, 40] = 8192.0 * float(np.max(np.abs(rows)))
    B.upload(arena)
    op = btod_contract2(contraction2(2, 2, 2).contract(2, 2).contract(3, 3), A, B, kc=cfg.kc)
    P, C = op.make_result(), op.make_result()
    op.perform(P)
    op.perform(C, mode=MODE_OZAKI_CRT, nslices=13)
    ctx.synchronize()
    assert _worst(C.download(), P.download(), C) <= 1e-8
    for x in (op, P, C, A, B):
        x.close()
    ctx.close()


def test_redo_follows_the_operands_of_each_call():
    """One plan, called with operands whose sampled bounds are too small, then
    with bounds that hold, then too small again: whether rows are redone is
    found anew in each call, so every result has the bits of a fresh plan's
    (the integers are exact, nothing depends on timing)."""
    ctx = Context(0)
    cfg = S.LadderConfig("redo", [3], [34])
    A, B = block_tensor(ctx, cfg.t_spec()), block_tensor(ctx, cfg.v_spec())
    A.fill_seeded(11, cfg.t_scale)
    plain = B.fill_seeded_host(23, cfg.v_scale)
    planted = plain.copy()
    B.upload(plain)
    for bidx, blk in B.blocks(planted):
        rows = blk.reshape(blk.shape[0] * blk.shape[1], -1)
        rows[:, 40] = 8192.0 * float(np.max(np.abs(rows)))

    def plan():
        op = btod_contract2(contraction2(2, 2, 2).contract(2, 2).contract(3, 3), A, B, kc=cfg.kc)
        return op, op.make_result()

    kept, C = plan()
    for arena in (planted, plain, planted, plain):
        B.upload(arena)
        fresh, D = plan()
        for op, r in ((kept, C), (fresh, D)):
            op.perform(r, mode=MODE_OZAKI_CRT, nslices=13)
        ctx.synchronize()
        assert np.array_equal(C.download(), D.download())
        for x in (fresh, D):
            x.close()
    for x in (kept, C, A, B):
        x.close()
    ctx.close()


def test_no_products_leave_or_zero_the_result():
    """An operand without non-zero blocks: the schedule is empty, so adding
    leaves the result as it is and assigning zeroes it."""
    ctx = Context(0)
    cfg = S.LadderConfig("empty", [3], [5, 4])
    A, B = block_tensor(ctx, cfg.t_spec()), block_tensor(ctx, cfg.v_spec())
    A.set_zero()
    B.fill_seeded(23, cfg.v_scale)
    op = btod_contract2(contraction2(2, 2, 2).contract(2, 2).contract(3, 3), A, B, kc=cfg.kc)
    C = op.make_result()
    C.upload(np.full(C.nelems, 3.0))
    op.perform(C, 1.0, mode=MODE_OZAKI_CRT, nslices=13)
    ctx.synchronize()
    assert all(np.all(blk == 3.0) for _, blk in C.blocks(C.download()))
    op.perform(C, mode=MODE_OZAKI_CRT, nslices=13)
    ctx.synchronize()
    assert not any(np.any(blk) for _, blk in C.blocks(C.download())) and C.nonzero() == []
    for x in (op, C, A, B):
        x.close()
    ctx.close()


@pytest.mark.parametrize("moduli", range(8, 17))
@pytest.mark.parametrize("m,n", [(300, 40), (37, 259), (1, 130)], ids=["rows long", "columns long", "one row"])
def test_recombination_is_exact_on_integers(moduli, m, n):
    """Integers below 2^11 are exact in the P >= 24 bits of every modulus count
    and 100 of their products stay below 2^53, so the recombined result must
    equal the integer result, either side along the tile rows; the last terms
    cancel in one column, whose exact zeros must come out as zeros."""
    ctx = Context(0)
    rng = np.random.default_rng(moduli)
    a = rng.integers(-2047, 2048, (m, 100)).astype(float)
    b = rng.integers(-2047, 2048, (n, 100)).astype(float)
    b[n // 2] = 0.0
    b[n // 2, :2], a[:, 1] = (1.0, -1.0), a[:, 0]
    A = block_tensor(ctx, S.BTSpec(dims=[m, 100], splits=[[], [60]]))
    B = block_tensor(ctx, S.BTSpec(dims=[n, 100], splits=[[], [60]]))
    for t, x in ((A, a), (B, b)):
        t.set_block((0, 0), x[:, :60])
        t.set_block((0, 1), x[:, 60:])
    op = btod_contract2(contraction2(1, 1, 1).contract(1, 1), A, B)
    C = op.make_result()
    op.perform(C, mode=MODE_OZAKI_CRT, nslices=moduli)
    ctx.synchronize()
    assert np.array_equal(C.get_block((0, 0), (m, n)), a @ b.T)
    for x in (op, C, A, B):
        x.close()
    ctx.close()
