"""GPU tests of what runs in a smaller workspace (kq_set_workspace_limit): the FP64 multishift CG in the reference's
kernel order and the true residuals with few temporaries, against the oracle (oracle/hisq_oracle.c).  Tolerances as for
the same calls without a limit: solutions to 1e-9 at convergence and 1e-11 at an iteration cap, residuals to 1e-12."""
import numpy as np
import pytest

import kuqcd_b200 as K
from oracle import oracle as O
from tests.conftest import dev_buffer


def context(dims, seed):
    fat, lng = O.make_links(dims, 0.3, seed)
    ctx = K.Context(dims)
    ctx.load_links(K.KUQCD_FAT_LINK, fat)
    ctx.load_links(K.KUQCD_LONG_LINK, lng)
    return ctx, fat, lng


def launches_in_reference_order(it):
    """One initial kernel, then chunks of eight iterations of four kernels."""
    return 1 + 32 * -(-it // 8)


@pytest.mark.gpu
@pytest.mark.parametrize("dims,parity", [((8, 8, 8, 8), 0), ((8, 8, 8, 8), 1), ((6, 4, 4, 6), 0), ((4, 4, 4, 1), 1),
                                         ((14, 12, 10, 18), 0)])
def test_reference_order_cgm_converges_as_the_oracle(cuda, dims, parity):
    ctx, fat, lng = context(dims, 1234)
    b = O.make_source(dims, parity, 99)
    sig = list(0.05 ** 2 + np.logspace(-4, 0, 12))
    tol = (1e-10) ** 2 * float(b @ b)
    want, it = O.cgm(dims, fat, lng, parity, [sig[0]] + [s - sig[0] for s in sig[1:]], b, tol, 10000)
    ctx.set_workspace_limit(1)
    xs, info = ctx.solve(b, sig, parity=parity, solver=K.KQ_SOLVER_CGM, tol=tol)
    assert info.kernel_launches == launches_in_reference_order(info.iter)
    xw, iw = ctx.solve(b, sig, parity=parity, solver=K.KQ_SOLVER_CGM_WINDOWED, tol=tol)
    ctx.set_workspace_limit(0)
    xa, ia = ctx.solve(b, sig, parity=parity, solver=K.KQ_SOLVER_CGM, tol=tol)
    assert ia.kernel_launches != launches_in_reference_order(ia.iter)  # the windowed solver, without a limit
    for x, i in ((xs, info), (xw, iw), (xa, ia)):
        assert abs(i.iter - it) <= 1 and i.status == 0
        for k in range(12):
            assert np.abs(x[k] - want[k]).max() <= 1e-9 * np.abs(want[k]).max(), k
            assert O.true_residual(dims, fat, lng, parity, sig[k], b, x[k]) <= 1.5e-10, k
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("max_iter", [1, 7, 8, 9, 17])
def test_reference_order_cgm_stops_at_the_cap(cuda, max_iter):
    dims = (6, 6, 4, 4)
    ctx, fat, lng = context(dims, 5)
    b = O.make_source(dims, 0, 3)
    rel = [0.0125, 0.05, 0.3]
    want, it = O.cgm(dims, fat, lng, 0, rel, b, 0.0, max_iter)
    ctx.set_workspace_limit(1)
    xs, info = ctx.solve(b, rel, solver=K.KQ_SOLVER_CGM, tol=0.0, max_iter=max_iter, shift_mode=0)
    assert info.iter == it == max_iter and info.status == 2
    assert info.kernel_launches == launches_in_reference_order(max_iter)
    for x, w in zip(xs, want):
        assert np.linalg.norm(x - w) <= 1e-11 * np.linalg.norm(w)
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(8, 6, 5, 4), (18, 17, 19, 18)])
@pytest.mark.parametrize("ns", [17, 20, 33])
@pytest.mark.parametrize("full", [False, True])
def test_true_residuals_in_several_launches(cuda, dims, ns, full):
    """More shifts than temporaries: sixteen without a limit, then four and one.  On the smaller lattice one shift per
    thread, on the larger one groups of up to four, so 17 shifts are groups of four and three, and 20 and 33 take
    several launches of one group size."""
    ctx, fat, lng = context(dims, 11)
    halves, vh = (2 if full else 1), int(np.prod(dims)) // 2
    vb = ctx.spinor_bytes(K.KUQCD_DOUBLE)
    rng = np.random.default_rng(ns)
    b = rng.standard_normal((halves, vh * 6))
    xs = rng.standard_normal((ns, halves, vh * 6))
    sig = list(0.01 + np.logspace(-3, 0, ns))
    d_b, d_x = dev_buffer(vb * halves), dev_buffer(vb * halves * ns)
    for h in range(halves):
        ctx.upload(K.KUQCD_DOUBLE, b[h], d_b[h * vb:(h + 1) * vb])
        for k in range(ns):
            ctx.upload(K.KUQCD_DOUBLE, xs[k, h], d_x[(k * halves + h) * vb:(k * halves + h + 1) * vb])
    want = [np.sqrt(sum((O.true_residual(dims, fat, lng, h, s, b[h], xs[k, h]) * np.linalg.norm(b[h])) ** 2
                        for h in range(halves))) / np.linalg.norm(b) for k, s in enumerate(sig)]
    partials = 8 * -(-vh // 128) * (ns + 1)
    for fields in (16, 4, 1):
        ctx.set_workspace_limit(fields * vb + partials + 2048)
        got = ctx.true_residuals(K.KQ_PARITY_FULL if full else 0, sig, d_b, d_x)
        assert max(abs(g / w - 1) for g, w in zip(got, want)) <= 1e-12, fields
    ctx.close()
