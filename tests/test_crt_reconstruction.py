"""The modular mode's reconstruction (limb sums, quotient, joining) restated in
exact and FP64 arithmetic at the ends of the integers' range.  No GPU."""
from fractions import Fraction as F
import math
import random

import pytest

MODULI = [256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193]
BITS = 41                                   # bits per limb of the weights and of M
MAGIC = 1.5 * 2.0 ** 52


def fma(a, b, c):
    return float(F(a) * F(b) + F(c))        # one rounding


def quotient_limbs(M):
    """Two, or three where the highest limb of M has 8 bits or fewer."""
    n = -(-M.bit_length() // BITS)
    return 3 if n > 2 and M >> (BITS * (n - 1) + 8) == 0 else 2


def reconstruct(residues, moduli):
    M = math.prod(moduli)
    W = [M // m * pow(M // m, -1, m) for m in moduli]
    n = -(-M.bit_length() // BITS)
    limb = lambda x, i: (x >> (BITS * i)) & ((1 << BITS) - 1)
    S = [sum(r * limb(w, i) for r, w in zip(residues, W)) for i in range(n)]
    assert max(S) < 2 ** 53                 # so FP64 multiply-adds form them exactly
    share = [float(F(2 ** (BITS * i), M)) for i in range(n)]
    low = float(S[-2]) * share[-2]
    if quotient_limbs(M) == 3:
        low = fma(float(S[-3]), share[-3], low)
    q = fma(float(S[-1]), share[-1], low) + MAGIC - MAGIC
    x = 0.0
    for i in reversed(range(n)):
        d = fma(-q, float(limb(M, i)), float(S[i]))
        assert F(d) == S[i] - int(q) * limb(M, i)           # exact again
        x = d if i == n - 1 else fma(x, 2.0 ** BITS, d)
    return x, n


def largest(L):
    """Largest |X| of L moduli: the scaling keeps it 2^-1e-9 inside M / 2, and at
    most 2^17 products of two 50-bit integers are summed exactly in INT32."""
    M = math.prod(MODULI[:L])
    return min(int(F(M, 2) * F(2.0 ** -1e-9)), 2 ** 117)


@pytest.mark.parametrize("L", range(8, 17))
def test_integers_come_back_at_both_ends_of_the_range(L):
    """Exact below 2^53, else within one rounding per limb joined."""
    rng = random.Random(L)
    top = largest(L)
    xs = [top - i for i in range(20)] + [rng.randrange(top // 2, top) for _ in range(50)]
    xs += [rng.getrandbits(rng.randrange(1, top.bit_length())) for _ in range(100)] + [0, 1]
    for x in xs:
        for y in (x, -x):
            got, n = reconstruct([y % m for m in MODULI[:L]], MODULI[:L])
            assert abs(F(got) - y) <= (0 if x < 2 ** 53 else (n - 1) * x * F(1, 2 ** 53)), (L, y)


@pytest.mark.parametrize("L", range(8, 17))
def test_quotient_margin(L):
    """What the quotient leaves out (the lower limbs, and the rounding of its
    products, which are below 2^12) against the distance of the largest |X| / M
    from a half: a factor of 200 at least."""
    M = math.prod(MODULI[:L])
    n = -(-M.bit_length() // BITS)
    left_out = sum(F(sum(m - 1 for m in MODULI[:L]) * 2 ** BITS * 2 ** (BITS * i), M) for i in range(n - quotient_limbs(M)))
    assert 200 * (left_out + 3 * F(2 ** 12, 2 ** 53)) <= F(1, 2) - F(largest(L), M)
