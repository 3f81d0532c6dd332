"""Workspace of the k-split partial tiles: shared by the plans of a context and
given back with them."""
import gc

import numpy as np
import pytest

from libtensor_b200.core import Context, block_tensor, btod_contract2, contraction2
from libtensor_b200.spec import BTSpec

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MB = 1 << 20


def _plan(ctx, A, B):
    op = btod_contract2(contraction2(1, 1, 1).contract(1, 1), A, B)
    op.set_split_k(4)
    return op, op.make_result()


def _used(ctx):
    ctx.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def test_workspace_goes_with_its_plans():
    """Four chunks of every tile of a 4096 x 4096 result are 512 MB; a second
    plan shares them, the first may go, and with the last plan they go too (but
    for 32 MB the context keeps, and 16 MB for what the driver rounds to)."""
    gc.collect()                                 # nothing of other tests is freed meanwhile
    ctx = Context(0)
    rng = np.random.default_rng(1)
    x = rng.standard_normal((4096, 256))
    spec = BTSpec(dims=[4096, 256], splits=[[], []])
    A, B = block_tensor(ctx, spec), block_tensor(ctx, spec)
    A.upload(x.ravel())
    B.upload(x[::-1].ravel())
    op, C = _plan(ctx, A, B)                     # modules and context memory come with a first call
    op.set_split_k(1)
    op.perform(C)
    op.close()
    before = _used(ctx)
    op1, C1 = _plan(ctx, A, B)
    op1.perform(C)
    one = _used(ctx)
    assert one - before >= 512 * MB
    op2, C2 = _plan(ctx, A, B)
    op2.perform(C)
    assert _used(ctx) - one <= 48 * MB + 2 * C.nelems * 8
    want = C.download()
    op1.close()
    C.upload(np.zeros(C.nelems))
    op2.perform(C)                               # the workspace outlives the plan that brought it
    assert np.array_equal(C.download(), want)
    op2.close()
    for t in (C1, C2):
        t.close()
    assert _used(ctx) - before <= 48 * MB
    for t in (C, A, B):
        t.close()
    ctx.close()
