// Scalar steps of the windowed multishift CG (device side), shared by the single-system solver (kq_msrelax.cu)
// and the batched multi-system solver (kq_batch.cu).  They restate the recurrences of inverter_cgm.cpp:45-77 and
// accumulate the window coefficients of the deferred shift updates.
#pragma once
#include "kq_dslash_core.cuh"
#include "kq_msrelax.h"

namespace kq {

// ---------------------------------------------------------------------------------------------------- scalar steps
// What the next kernel of the iteration waits for is taken at the end of each reduction by one thread: B_0 after the
// first dslash (ms_beta), a_0 after the second (ms_alpha).  Everything else -- the shifted recurrences, the window
// coefficients of the deferred updates, the dropping of converged shifts -- is one shift step per iteration, run by
// a whole block beside the update of p0 (ms_shift_step).  With the shift work inside the two reductions, one warp
// looping over (shift, position) items in global memory, the tail of either dslash kernel cost about 9 us: at 16^4
// with 12 shifts the FP64 kernels took 23 us for 14 us of dslash.

// beta step (inverter_cgm.cpp:48-50): B_0 = -|r|^2 / <p, A p>, <p, A p> = sigma_0 |p|^2 + |D p|^2.  One thread;
// `slot`: the flag of the running iteration.
__device__ __forceinline__ void ms_beta(MsState *st, int slot, double rNorm2, double pAp)
{
    const double B0 = -rNorm2 / pAp;
    if (!(pAp != 0.0) || !isfinite(B0)) {
        st->status = KQ_STATUS_BREAKDOWN;
        st->active[slot] = 0;
        st->halt = 1;
        return;
    }
    st->b0 = B0;
}

// alpha step (inverter_cgm.cpp:58-60): a_0 = |r_new|^2 / |r|^2, and the next iteration's operator precision (the
// batched solver's).  One thread.
__device__ __forceinline__ void ms_alpha(MsState *st, double rNorm2, double lambda2)
{
    const double a0 = lambda2 / rNorm2;
    st->a0 = a0;
    st->lambda2 = lambda2;
    st->rNorm2 = lambda2;
    // |p_new|^2 = |r_new|^2 + a0^2 |p|^2, since the step makes r_new orthogonal to p
    st->pp = lambda2 + a0 * a0 * st->pp;
    st->iter += 1;
    if (!isfinite(lambda2)) {
        st->status = KQ_STATUS_BREAKDOWN;
        st->halt = 1;
    }
    const double rel2 = lambda2 / st->bnorm2;
    st->next_mode = (st->rho16_2 > 0.0 && rel2 < st->rho16_2) ? 2 : (st->rho32_2 > 0.0 && rel2 < st->rho32_2) ? 1 : 0;
}

// Shift step of one iteration (inverter_cgm.cpp:51-57, 61-77), run by every thread of one block of at least 64
// threads after ms_alpha: thread k < 64 takes shift k's recurrences (the shifted B_k, zeta_k, a_k, and whether the
// shift is still above tolerance), then the (shift, position) items of the window coefficients are spread over the
// block.  x_k -= B_k p_k and p_k = Z_k r_new + a_k p_k in the window representation are
//     e_k -= B_k c_k, f_kl -= B_k d_kl, then c_k *= a_k, d_kl *= a_k, d_k,new = Z_k.
// Every value is loaded once, all loads of a phase are independent, and each value has one writer.  Returns (to every
// thread) whether the solve goes on.
__device__ __forceinline__ bool ms_shift_step(MsState *st)
{
    __shared__ double sB[kMaxShift], sa[kMaxShift], sZ[kMaxShift];
    __shared__ unsigned keep_mask[kMaxShift / 32];
    const int tid = threadIdx.x, nt = blockDim.x;
    const int mt0 = st->maxTerm, ns = st->ns, jw = st->wpos;  // ring positions 0..jw-1 are in use
    const double B0 = st->b0, a0 = st->a0, a0m1 = st->a[0], Bm1 = st->Bm1, lambda2 = st->lambda2, tol = st->tol;
    if (tid < kMaxShift) {
        const int k = tid;
        double Bk = B0, ak = a0, z = 1.0;
        bool keep = false;
        if (k < mt0) {
            z = st->Z[k];
            if (k > 0) {
                const double zm1 = st->Zm1[k], sh = st->shift[k];
                const double rr1 = Bm1 * zm1 / (B0 * a0m1 * (zm1 - z) + zm1 * Bm1 * (1.0 - sh * B0));
                const double zn = z * rr1;
                Bk = B0 * rr1;
                ak = a0 * zn * Bk / (z * B0);
                st->Zm1[k] = z;
                st->Z[k] = zn;
                z = zn;
            }
            st->B[k] = Bk;
            keep = !(z * z * lambda2 < tol);  // converged shifts drop from the top
            sB[k] = Bk;
            sa[k] = ak;
            sZ[k] = z;
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if ((tid & 31) == 0) keep_mask[tid >> 5] = m;
    }
    __syncthreads();
    if (tid < mt0) st->a[tid] = sa[tid];
    // the new maxTerm: one above the highest shift still above tolerance (the reference's do-while)
    int mt = 0;
#pragma unroll
    for (int w = 0; w < kMaxShift / 32; ++w)
        if (keep_mask[w]) mt = 32 * (w + 1) - __clz((int)keep_mask[w]);
    if (jw == 0) {
        // first iteration of a window: from the identity representation p = p_old, x = x_old
        for (int t = tid; t < ns * kWin; t += nt) {
            const int k = t / kWin, l = t - k * kWin;
            const bool on = k < mt0;
            st->d[k][l] = on && l == 0 ? sZ[k] : 0.0;
            st->f[k][l] = 0.0;
            if (l == 0) {
                st->c[k] = on ? sa[k] : 1.0;
                st->e[k] = on ? -sB[k] : 0.0;
            }
        }
    } else {
        // item l = jw: c_k, e_k and the weight of the new residual; items l < jw: d_kl, f_kl
        const int per = jw + 1;
#pragma unroll 4
        for (int t = tid; t < mt0 * per; t += nt) {
            const int k = t / per, l = t - k * per;
            double *dp = l == jw ? &st->c[k] : &st->d[k][l], *fp = l == jw ? &st->e[k] : &st->f[k][l];
            const double dv = *dp, fv = *fp;
            *fp = fv - sB[k] * dv;
            *dp = dv * sa[k];
            if (l == jw) st->d[k][jw] = sZ[k];
        }
    }
    const bool go = mt > 0 && st->iter < st->max_iter && !st->halt && isfinite(lambda2);
    __syncthreads();  // every thread has read what thread 0 overwrites
    if (tid == 0) {
        st->maxTerm = mt;
        st->Bm1 = B0;
        st->wpos = jw + 1;
        if (jw == 0) st->wmax = mt0;
    }
    return go;
}

// Windowed shift update of one site, one colour component at a time (keeps W ring values in registers, not 6 W):
//   p_k <- c_k p_k + sum_l d_kl r_l ,  x_k <- x_k + e_k p_k + sum_l f_kl r_l   for k < kmax.
// Window position l (0-based) holds r^(i0+l+1) in ring slot (l+1) % W; positions >= n are unused (zero weight).
// FP64 spinor fields are three double2 planes of pv sites (kq_prec.cuh).  KU shifts at a time: their p and x are
// loaded before any of them is stored (the stores could alias later loads for the compiler), so KU x 2 loads per
// thread are in flight instead of 2.
__device__ __forceinline__ void window_update_one(const double2 p, const double2 x, const double2 *rl, double c,
                                                  double e, const double *d, const double *f, double2 &pn,
                                                  double2 &xn)
{
    pn = make_double2(c * p.x, c * p.y);
    xn = make_double2(x.x + e * p.x, x.y + e * p.y);
#pragma unroll
    for (int l = 0; l < kWin; ++l) {
        pn.x += d[l] * rl[l].x;
        pn.y += d[l] * rl[l].y;
        xn.x += f[l] * rl[l].x;
        xn.y += f[l] * rl[l].y;
    }
}

template <int KU = 1>
__device__ __forceinline__ void window_update_site(const char *ring, size_t vb, int pv, int i, int n, int kmax,
                                                   const double *sc, const double *se, const double (*sd)[kWin],
                                                   const double (*sf)[kWin], char *pw0, char *x0)
{
#pragma unroll 1
    for (int c = 0; c < 3; ++c) {
        const size_t off = (size_t)c * pv + i;
        double2 rl[kWin];
#pragma unroll
        for (int l = 0; l < kWin; ++l)
            rl[l] = l < n ? __ldg(reinterpret_cast<const double2 *>(ring + (size_t)((l + 1) % kWin) * vb) + off)
                          : make_double2(0.0, 0.0);
        int k = 0;
#pragma unroll 1
        for (; k + KU <= kmax; k += KU) {
            double2 p[KU], x[KU];
#pragma unroll
            for (int u = 0; u < KU; ++u) {
                p[u] = reinterpret_cast<const double2 *>(pw0 + (k + u) * vb)[off];
                x[u] = reinterpret_cast<const double2 *>(x0 + (k + u) * vb)[off];
            }
#pragma unroll
            for (int u = 0; u < KU; ++u) {
                double2 pn, xn;
                window_update_one(p[u], x[u], rl, sc[k + u], se[k + u], sd[k + u], sf[k + u], pn, xn);
                reinterpret_cast<double2 *>(pw0 + (k + u) * vb)[off] = pn;
                reinterpret_cast<double2 *>(x0 + (k + u) * vb)[off] = xn;
            }
        }
#pragma unroll 1
        for (; k < kmax; ++k) {
            double2 *pp = reinterpret_cast<double2 *>(pw0 + k * vb) + off;
            double2 *xp = reinterpret_cast<double2 *>(x0 + k * vb) + off;
            double2 pn, xn;
            window_update_one(*pp, *xp, rl, sc[k], se[k], sd[k], sf[k], pn, xn);
            *pp = pn;
            *xp = xn;
        }
    }
}

}  // namespace kq
