"""Modular mode with the largest integers its scaling lets through: products of
one sign, of elements just below a power of two, as many as fit."""
import math

import numpy as np
import pytest

from libtensor_b200.core import MODE_OZAKI_CRT, Context, block_tensor, btod_contract2, contraction2
from libtensor_b200.spec import BTSpec

pytestmark = pytest.mark.gpu

MODULI = [256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193]


def _longest(L):
    """(P, K): P bits per operand and the K whose K 4^P comes closest to M / 2 from
    below, for the largest P of at most 50 that leaves a thousand products."""
    M = math.prod(MODULI[:L])
    P = min(50, int((math.log2(M) - 1 - 10) // 2))
    return P, M * (10 ** 9 - 1) // (2 * 10 ** 9) // 4 ** P - 1


@pytest.mark.parametrize("L", range(8, 16))
def test_sums_near_half_the_modulus(L):
    """A quotient off by one would give the sum less M: the opposite sign.  The
    operands round to 2^P (2^-53 off) and the result within three roundings.
    (16 moduli: 50-bit operands and sums exact in INT32 end at 2^-7 of M / 2.)"""
    P, K = _longest(L)
    assert 0.99 * math.prod(MODULI[:L]) / 2 <= K * 4.0 ** P
    ctx = Context(0)
    x = np.nextafter(1.0, 0.0)
    a = np.full((3, K), x)
    a[1] = -x
    a[2, ::2] = 0.0
    A = block_tensor(ctx, BTSpec(dims=[3, K], splits=[[], []]))
    B = block_tensor(ctx, BTSpec(dims=[2, K], splits=[[], []]))
    A.set_block((0, 0), a)
    B.set_block((0, 0), np.full((2, K), x))
    op = btod_contract2(contraction2(1, 1, 1).contract(1, 1), A, B)
    op.set_crt_bound(False)                      # exact exponents: no spare binade
    C = op.make_result()
    op.perform(C, mode=MODE_OZAKI_CRT, nslices=L)
    ctx.synchronize()
    got = C.get_block((0, 0), (3, 2))
    want = np.array([K, -K, K // 2])[:, None] * np.ones((1, 2))
    assert np.all(np.abs(got - want) <= 8 * 2.0 ** -53 * K), got
    for t in (op, C, A, B):
        t.close()
    ctx.close()
