"""Solves of a few iterations enqueue the chunks of eight iterations they need and no more: a solve whose cap or tolerance
ends it in the first chunk, and one whose cap is the end of the second.  A chunk is three kernels per iteration, the window
update and the poll; the initial kernel makes one more."""
import numpy as np
import pytest

import kuqcd_b200 as K
from oracle import oracle as O

CHUNK = 3 * 8 + 2


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(4, 4, 4, 4), (16, 12, 12, 12)])
@pytest.mark.parametrize("solver", [K.KQ_SOLVER_CGM, K.KQ_SOLVER_CGM_WINDOWED])
def test_short_solves_run_no_chunk_in_vain(cuda, dims, solver):
    fat, lng = O.make_links(dims, 0.3, 5)
    ctx = K.Context(dims)
    ctx.load_links(K.KUQCD_FAT_LINK, fat)
    ctx.load_links(K.KUQCD_LONG_LINK, lng)
    b = O.make_source(dims, 0, 3)
    for cap, chunks in ((1, 1), (7, 1), (8, 1), (9, 2), (16, 2)):
        _, info = ctx.solve(b, [0.01, 0.1], solver=solver, tol=0.0, max_iter=cap)
        assert info.iter == cap and info.kernel_launches == 1 + chunks * CHUNK, cap
    # sigma far above the operator's norm: every shift below tolerance within eight iterations
    xs, info = ctx.solve(b, [100.0, 300.0], solver=solver, tol=1e-20 * float(b @ b), max_iter=1000)
    assert 1 < info.iter <= 8 and info.kernel_launches == 1 + CHUNK
    for x, s in zip(xs, (100.0, 300.0)):
        assert O.true_residual(dims, fat, lng, 0, s, b, x) <= 1.5e-10
    ctx.close()
