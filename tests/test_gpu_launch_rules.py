"""GPU tests of the launch rules: sizes on either side of every limit between the kernels that share the dslash, the
grouping of the true-residual kernels, and the multishift loop's iteration caps, against the oracle
(oracle/hisq_oracle.c).  Tolerances: FP64 1e-13 relative to the largest component, as in the dslash tests (sixteen
terms, each a 3x3 mat-vec, in another order of summation); FP32 1e-6 and HALF 3e-4 in relative 2-norm."""
import numpy as np
import pytest
import torch

import kuqcd_b200 as K
from oracle import oracle as O
from oracle import ptc_oracle as P
from tests.conftest import dev_buffer

# Sites per parity (twice that on full fields).  Threads per site change at 11,750 / 23,500 / 47,000 (FP64), 21,875 /
# 43,750 / 87,500 (FP32) and 18,750 / 37,500 / 75,000 (HALF); the HALF kernel of two sites per thread starts above
# 150,000; FP64 takes four CTAs per SM between one and two waves of three (113,664 and 151,552 sites).
DIMS = [(12, 11, 9, 19), (14, 13, 11, 21), (16, 15, 17, 22), (18, 17, 19, 18), (20, 19, 21, 30), (24, 23, 25, 24)]
TOL = {K.KUQCD_SINGLE: 1e-6, K.KUQCD_HALF: 3e-4}


def context(dims, seed=7):
    fat, lng = O.make_links(dims, 0.3, seed)
    ctx = K.Context(dims)
    ctx.load_links(K.KUQCD_FAT_LINK, fat)
    ctx.load_links(K.KUQCD_LONG_LINK, lng)
    return ctx, fat, lng


def near(out, ref, prec):
    if prec == K.KUQCD_DOUBLE:
        return np.abs(out - ref).max() <= 1e-13 * np.abs(ref).max()
    return np.linalg.norm(out - ref) <= TOL[prec] * np.linalg.norm(ref)


@pytest.mark.gpu
@pytest.mark.parametrize("dims", DIMS)
def test_operators_on_both_sides_of_the_launch_limits(cuda, dims):
    ctx, fat, lng = context(dims)
    vh = int(np.prod(dims)) // 2
    src = np.random.default_rng(3).standard_normal(2 * vh * 6)
    one, sigma = src[:vh * 6].copy(), 0.37
    want_d = O.dslash(dims, fat, lng, one, 1)
    # O.mdagm is D D (tests/test_gpu_dslash.py)
    want_m = sigma * one - O.dslash(dims, fat, lng, want_d, 0)
    want_f = O.dslash_full(dims, fat, lng, src)
    want_mf = sigma * src - O.dslash_full(dims, fat, lng, want_f)
    for prec in (K.KUQCD_DOUBLE, K.KUQCD_SINGLE, K.KUQCD_HALF):
        nb = ctx.spinor_bytes(prec)
        a, b, t = dev_buffer(nb), dev_buffer(nb), dev_buffer(nb)
        ctx.upload(prec, one, a)
        ctx.dslash(prec, a, b, 1)
        assert near(ctx.download(prec, b), want_d, prec), ("dslash", prec)
        ctx.mdagm(prec, sigma, a, b, t, 0)
        assert near(ctx.download(prec, b), want_m, prec), ("mdagm", prec)
        fa, fb, ft = dev_buffer(2 * nb), dev_buffer(2 * nb), dev_buffer(2 * nb)
        ctx.upload_full(prec, src, fa)
        ctx.dslash_full(prec, fa, fb)
        assert near(ctx.download_full(prec, fb), want_f, prec), ("full", prec)
        ctx.mdagm_full(prec, sigma, fa, fb, ft)
        assert near(ctx.download_full(prec, fb), want_mf, prec), ("mdagm_full", prec)
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("dims,ns", [((8, 6, 5, 4), 1), ((8, 6, 5, 4), 3), ((8, 6, 5, 4), 12), ((18, 17, 19, 18), 2),
                                     ((18, 17, 19, 18), 3), ((18, 17, 19, 18), 4), ((18, 17, 19, 18), 5),
                                     ((18, 17, 19, 18), 9)])
@pytest.mark.parametrize("full", [False, True])
def test_true_residuals_in_groups_of_every_size(cuda, dims, ns, full):
    """Groups of one shift per thread while all fit one wave (ns sites <= 113,664), else of up to four, of sizes that
    differ by at most one; 9 shifts also take more than one launch per group size."""
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
    got = ctx.true_residuals(K.KQ_PARITY_FULL if full else 0, sig, d_b, d_x)
    for k, s in enumerate(sig):
        rr = sum((O.true_residual(dims, fat, lng, h, s, b[h], xs[k, h]) * np.linalg.norm(b[h])) ** 2
                 for h in range(halves))
        assert abs(got[k] - np.sqrt(rr) / np.linalg.norm(b)) <= 1e-12 * got[k], k
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(6, 6, 4, 4), (14, 12, 10, 18)])
@pytest.mark.parametrize("max_iter", [1, 7, 8, 9, 16, 17, 33])
def test_multishift_stops_at_the_cap(cuda, dims, max_iter):
    """Caps at and around the ends of chunks (8 iterations) and windows (16), with chunks launched ahead: the iteration
    count is the cap and the solutions are the reference recurrences' after that many iterations."""
    ctx, fat, lng = context(dims, 5)
    b = O.make_source(dims, 0, 3)
    sig = list(0.05 ** 2 + np.logspace(-2, 0, 5))
    rel = [sig[0]] + [s - sig[0] for s in sig[1:]]
    want, it = O.cgm(dims, fat, lng, 0, rel, b, 0.0, max_iter)
    assert it == max_iter
    for solver in (K.KQ_SOLVER_CGM, K.KQ_SOLVER_CGM_WINDOWED):
        xs, info = ctx.solve(b, sig, solver=solver, tol=0.0, max_iter=max_iter)
        assert info.iter == max_iter and info.status == 2
        for x, w in zip(xs, want):
            assert np.linalg.norm(x - w) <= 1e-11 * np.linalg.norm(w)
    ctx.close()


@pytest.mark.gpu
def test_net_gradient_on_a_ragged_lattice(cuda):
    """The weight gradient where the last tile of 128 sites is partly past the end (Vh = 1350), held to the bound of the
    layers' output against the BF16-rounding oracle (5e-4, tests/test_gpu_net.py)."""
    dims, ch = (10, 6, 5, 9), (1, 8, 8)
    ctx, fat, lng = context(dims, 4)
    net = K.Net(ctx, ch)
    w = (0.3 * np.random.default_rng(1).standard_normal(net.nw)).astype(np.float32)
    net.weights = w
    r, e = O.make_source(dims, 0, 5), O.make_source(dims, 0, 6)
    dr, de = dev_buffer(ctx.spinor_bytes(K.KUQCD_DOUBLE)), dev_buffer(ctx.spinor_bytes(K.KUQCD_DOUBLE))
    ctx.upload(K.KUQCD_DOUBLE, r, dr)
    ctx.upload(K.KUQCD_DOUBLE, e, de)
    torch.cuda.synchronize()
    net.zero_grad()
    loss = net.train_pair(dr, de, 0, float(e @ e))
    g = net.grad().astype(np.float64)
    want, grads = P.loss_and_grad(P.Lattice(dims, fat), P.weights_from_flat(w.astype(np.float64), ch), r, e, 0, bf=True)
    flat = P.flat_from_weights(grads)
    assert abs(loss - want) <= 5e-4 * want
    assert np.linalg.norm(g - flat) <= 5e-4 * np.linalg.norm(flat)
    ctx.close()
