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
