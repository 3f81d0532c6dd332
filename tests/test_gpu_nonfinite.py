"""A NaN or an infinity in an operand, split-precision modes: the slice modes
give NaN in every element of C that reads it, as FP64 arithmetic does, and no
mode lets it change an element that does not read it."""
import numpy as np
import pytest

from libtensor_b200.core import (MODE_OZAKI_BF16, MODE_OZAKI_CRT, MODE_OZAKI_FP8, MODE_OZAKI_INT8, Context,
                                 block_tensor, btod_contract2, contraction2)
from libtensor_b200.spec import BTSpec

pytestmark = pytest.mark.gpu

BAD = [np.nan, np.inf, -np.inf]


def _matrix(ctx, x, rows, ks, zero=()):
    t = block_tensor(ctx, BTSpec(dims=list(x.shape), splits=[[int(s) for s in np.cumsum(c)[:-1]] for c in (rows, ks)]))
    at = [np.concatenate([[0], np.cumsum(c)]) for c in (rows, ks)]
    for i in range(len(rows)):
        for k in range(len(ks)):
            if (i, k) not in zero:
                t.set_block((i, k), x[at[0][i]:at[0][i + 1], at[1][k]:at[1][k + 1]])
    return t


def _results(ctx, a, b, m, n, ks, bad, side, where, mode, slices):
    """C with the value `bad` at `where` of one operand and with zero there.
    B's block (last, last) is a zero block, so that the last column block of C
    does not read A's last k block."""
    out = []
    for v in (bad, 0.0):
        x, y = a.copy(), b.copy()
        (x if side == 0 else y)[where] = v
        A = _matrix(ctx, x, m, ks)
        B = _matrix(ctx, y, n, ks, [(len(n) - 1, len(ks) - 1)])
        op = btod_contract2(contraction2(1, 1, 1).contract(1, 1), A, B, kc=0.75)
        C = op.make_result()
        op.perform(C, mode=mode, nslices=slices)
        ctx.synchronize()
        c = np.zeros((sum(m), sum(n)))
        r0, c0 = np.concatenate([[0], np.cumsum(m)]), np.concatenate([[0], np.cumsum(n)])
        for (i, j), blk in C.blocks(C.download()):
            c[r0[i]:r0[i + 1], c0[j]:c0[j + 1]] = blk
        out.append(c)
        for t in (op, C, A, B):
            t.close()
    return out


def _operands(m, n, ks, seed):
    rng = np.random.default_rng(seed)
    # (magnitudes above 1, so that a row scaled by an exponent of zero would
    # leave the integers' range)
    a, b = 1e3 * rng.standard_normal((sum(m), sum(ks))), 1e3 * rng.standard_normal((sum(n), sum(ks)))
    a[:, ks[0]:] *= 16.0                    # a row's largest elements are in its last block
    return a, b


# either C side along the tile rows; the second pair's columns take two lanes each
SHAPES = [([130, 5], [20, 3]), ([20, 3], [130, 5]), ([9, 40], [150, 17])]


@pytest.mark.parametrize("mode,slices", [(MODE_OZAKI_INT8, 7), (MODE_OZAKI_BF16, 7), (MODE_OZAKI_BF16, 2),
                                         (MODE_OZAKI_FP8, 8), (MODE_OZAKI_FP8, 3)],
                         ids=["int8x7", "bf16x7", "bf16x2", "fp8x8", "fp8x3"])
@pytest.mark.parametrize("m,n", SHAPES, ids=str)
def test_slice_modes_give_nan_where_it_is_read(mode, slices, m, n):
    ctx = Context(0)
    ks = [40, 33]
    a, b = _operands(m, n, ks, 3)
    for bad in BAD:
        for side in (0, 1):
            # in the last row of the first row block and the last k block
            r = (m if side == 0 else n)[0] - 1
            got, clean = _results(ctx, a, b, m, n, ks, bad, side, (r, sum(ks) - 2), mode, slices)
            reads = np.zeros(got.shape, bool)
            if side == 0:
                reads[r, :n[0]] = True                       # not the columns of the zero block
            else:
                reads[:, r] = True
            assert np.all(np.isnan(got[reads])), (bad, side)
            assert np.array_equal(got[~reads], clean[~reads]), (bad, side)
    ctx.close()


@pytest.mark.parametrize("ks,k,big", [([40, 33], 50, 1024.0), ([40, 600], 50, 1024.0), ([40, 1100], 41, 1024.0),
                                      ([40, 1100], 40 + 700, 1.0)],
                         ids=["exact, core tiles", "exact, rows", "sampled, seen", "sampled, not seen"])
def test_modular_mode_keeps_the_scale_of_the_finite_elements(ks, k, big):
    """Rows of up to 1023 elements have exact maxima, longer ones a bound from
    elements 0-31, 512-543 and so on, checked by the residue pass.  The result
    with a zero in the place of the bad element has the same row maxima (the
    element beside the bad one, where it is read with it), so what does not read
    it has the same bits."""
    ctx = Context(0)
    m, n = [130, 5], [20, 3]
    a, b = _operands(m, n, ks, 5)
    r = m[0] - 1
    a[r, k ^ 1] = big * np.abs(a[r]).max()
    for bad in BAD:
        got, clean = _results(ctx, a, b, m, n, ks, bad, 0, (r, k), MODE_OZAKI_CRT, 13)
        reads = np.zeros(got.shape, bool)
        reads[r, :n[0]] = True
        assert np.array_equal(got[~reads], clean[~reads]), bad
        # products with exact zeros: what is left of the row is finite and right
        b0 = b.copy()
        b0[:, k] = 0.0
        got, clean = _results(ctx, a, b0, m, n, ks, bad, 0, (r, k), MODE_OZAKI_CRT, 13)
        assert np.array_equal(got, clean), bad
    ctx.close()
