"""Split passes of the slice and modular modes where the contracted elements are
not contiguous: offsets tabulated (up to 4096 of them) and computed."""
import numpy as np
import pytest

from libtensor_b200.core import (MODE_OZAKI_BF16, MODE_OZAKI_CRT, MODE_OZAKI_FP8, MODE_OZAKI_INT8, Context,
                                 block_tensor, btod_contract2, contraction2)
from libtensor_b200.spec import BTSpec

pytestmark = pytest.mark.gpu


def _tensor(ctx, x):
    t = block_tensor(ctx, BTSpec(dims=list(x.shape), splits=[[]] * x.ndim))
    t.set_block([0] * x.ndim, x)
    return t


# operand error relative to its row's bound of 2^-(beta S) per slice and dropped
# level (as S + 3 of them), and of 2^-44 per operand for 13 moduli and K near 4096
MODES = [(MODE_OZAKI_INT8, 7, 10 * 2.0 ** -49), (MODE_OZAKI_BF16, 4, 7 * 2.0 ** -28),
         (MODE_OZAKI_FP8, 8, 11 * 2.0 ** -40), (MODE_OZAKI_CRT, 13, 2 * 2.0 ** -44)]


@pytest.mark.parametrize("nk,nl", [(64, 64), (65, 64), (64, 65), (9, 7)], ids=str)
@pytest.mark.parametrize("mode,slices,eps", MODES, ids=["int8", "bf16", "fp8", "modular"])
def test_scattered_contracted_elements(mode, slices, eps, nk, nl):
    """C(i,j) = sum_kl A(k,i,l) B(k,l,j): A's offsets have two sub-dimensions,
    B's one with a stride.  A row's bound is at most 4 times its largest element
    (2 exact, and the sampled bound's binade)."""
    ctx = Context(0)
    rng = np.random.default_rng(nk)
    a, b = rng.standard_normal((nk, 21, nl)), rng.standard_normal((nk, nl, 37))
    A, B = _tensor(ctx, a), _tensor(ctx, b)
    op = btod_contract2(contraction2(1, 1, 2).contract(0, 0).contract(2, 1), A, B)
    C = op.make_result()
    op.perform(C, mode=mode, nslices=slices)
    ctx.synchronize()
    want = np.einsum("kil,klj->ij", a, b)
    bound = nk * nl * 16.0 * np.abs(a).max() * np.abs(b).max() * (eps + 2.0 ** -52)
    assert np.abs(C.get_block((0, 0), (21, 37)) - want).max() <= bound
    for x in (op, C, A, B):
        x.close()
    ctx.close()
