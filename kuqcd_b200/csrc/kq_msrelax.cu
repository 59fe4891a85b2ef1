// Multishift CG with windowed shift updates and a relaxed-precision operator.
//
// Recurrences and stopping rule are those of CGM::Invert (inverter_cgm.cpp:17-87).  Two changes of schedule:
//
// 1. Windowed shift updates.  The classic iteration reads and writes every shift's x_k and p_k every iteration
//    (Ymax + Axpby, inverter_cgm.cpp:61-69: 4 vectors per shift).  Here the base direction p_0 is updated every
//    iteration (the operator needs it), the residuals r^(i) go to a ring of W slots, and every W iterations one
//    kernel applies  p_k <- c_k p_k + sum_l d_kl r^(l),  x_k <- x_k + e_k p_k + sum_l f_kl r^(l)  for all shifts,
//    with coefficients accumulated by the scalar code from the same B_k, Z_k, a_k.  Per iteration the shift traffic
//    drops from 4N vectors to (4N + W)/W.
//
// 2. Relaxed operator precision (inexact Krylov).  The operator may be computed less accurately as the residual
//    shrinks: a matvec error eps*|A||p| made when |r| = rho |b| perturbs the final residual by about eps_eff * rho.
//    For multishift CG every shifted residual gap is a sum of the same matvec errors weighted by zeta_k <= 1, so it
//    is bounded by the base gap.  The host therefore switches the operator from FP64 to FP32 links (FP32 temporary)
//    at |r| < rho32 |b| and to HALF links (16-bit temporary) at |r| < rho16 |b|; all vectors and scalars stay FP64.
//    With rho = 0 the solver is the plain FP64 multishift CG with windowed updates.
//
// 3. Three kernels per iteration.  The operator is A = sigma0 - D_pq D_qp with D_pq = -D_qp^dag (the backward hops
//    apply the adjoints of the same stored links), so <p, A p> = sigma0 |p|^2 + |D_qp p|^2: the beta step can run
//    at the end of the first dslash, and the second dslash applies r <- r + B0 s directly, never storing s
//    (inverter_cgm.cpp:45-50 forms s, then <p, s>, then r).  In FP64 the two forms of <p, A p> agree to rounding;
//    with a 16-bit temporary the step length uses |D p|^2 before the temporary is rounded (relative 3e-5), while
//    the residual update uses the operator actually applied, so the recurrence stays exact.
//
// Kernels per iteration: K1 tmp = D p0, |tmp|^2 (beta step);  K2 r <- r + B0 (sigma0 p0 - D tmp) into the ring,
// |r|^2 (alpha step + |p0|^2 = |r|^2 + a0^2 |p0|^2, r being orthogonal to the old p0);  K3 p0 <- r + a0 p0, with the
// shift step (shifted recurrences, window coefficients, shift dropping) in one block of its own beside it.
// One CUDA graph per operator precision, kChunk iterations each followed by K4, the windowed shift update, which
// applies the window once it is full (W = 2 kChunk iterations) or the solve has stopped, and otherwise returns at
// once.  The window sets the shift-update traffic, the chunk the granularity of the precision switches.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <vector>

#include "kq_context.h"
#include "kq_dslash_core.cuh"
#include "kq_ms_device.cuh"
#include "kq_msrelax.h"

namespace kq {

constexpr int kBSm = 256;

// ---------------------------------------------------------------------------------------------------- kernels
__global__ void __launch_bounds__(kBSm) ms_init_kernel(int vh, int pv, const void *__restrict__ b, char *x0,
                                                       char *pw0, size_t vb, void *p0, char *ring, int ns,
                                                       MsState *st, double *partials)
{
    __shared__ double sm[32];
    const int i = blockIdx.x * kBSm + threadIdx.x;
    double nn = 0.0;
    if (i < vh) {
        double v[6], z[6] = {0, 0, 0, 0, 0, 0};
        ld_spinor<0>(b, pv, i, v);
        st_spinor<0>(p0, pv, i, v);
        st_spinor<0>(ring, pv, i, v);  // r^(0) in slot 0; the other slots are written before they are read
        for (int k = 0; k < ns; ++k) {
            st_spinor<0>(pw0 + k * vb, pv, i, v);
            st_spinor<0>(x0 + k * vb, pv, i, z);
        }
#pragma unroll
        for (int e = 0; e < 6; ++e) nn += v[e] * v[e];
    }
    double tot;
    if (grid_sum_last(nn, partials, &st->ticket[0], sm, &tot)) {
        st->rNorm2 = tot;
        st->bnorm2 = tot;
        st->pp = tot;  // p0 = b
        st->Bm1 = 1.0;
        for (int k = 0; k < st->ns; ++k) {
            st->a[k] = 0.0;
            st->B[k] = 1.0;
            st->Z[k] = 1.0;
            st->Zm1[k] = 1.0;
        }
        st->maxTerm = st->ns;
        st->wmax = st->ns;
        st->iter = 0;
        st->wpos = 0;
        st->halt = 0;
        // b = 0: x = 0 is the solution; a non-finite source is a breakdown
        const bool finite = isfinite(tot);
        st->status = finite ? 0 : KQ_STATUS_BREAKDOWN;
        st->active[0] = (finite && tot > 0.0) ? 1 : 0;
        st->active[1] = 0;
    }
}

// threads per CTA and sites per CTA of the dslash steps with S threads per site
__host__ __device__ constexpr int ms_threads(int S) { return S == 1 ? kBSm : S * split_sites(S); }
__host__ __device__ constexpr int ms_sites(int S) { return S == 1 ? kBSm : split_sites(S); }

// acc = (D src)(i) for this thread's output site i of parity p; false in threads without one.  *on: whether iterations
// still run (`active`).  With S > 1 the kernel may have been started beside the end of the one before it.
template <int LP, int SP, typename T, int S>
__device__ __forceinline__ bool ms_site(const Geom &g, int pv, const LinkSet &fat, const LinkSet &lng, const void *src,
                                        int p, const int *active, int &i, T acc[6], bool *on)
{
    i = blockIdx.x * ms_sites(S) + threadIdx.x % ms_sites(S);
    if constexpr (S == 1) {
        *on = *active != 0;
        if (!*on || i >= g.vh) return false;
        dslash_site_t<LP, SP, T>(g, pv, fat, lng, src, p, i, acc);
        return true;
    } else {
        const auto ready = [&] {
            pdl_wait();
            return *active != 0;
        };
        __shared__ T part[(S - 1) * 6 * ms_sites(S)];
        return dslash_site_split<LP, SP, T, S>(g, pv, fat, lng, src, p, i, i < g.vh, part, acc, ready, on);
    }
}

// K1: tmp = D p0 (p0 FP64; links LP; tmp stored in SO); |tmp|^2, then the beta step with
// <p0, A p0> = sigma0 |p0|^2 + |tmp|^2 (|p0|^2 from the alpha step's recurrence).  slot: parity of the iteration
// within its chunk.  S > 1: S threads per site (dslash_site_split).
template <int LP, int SO, int S, int MB>
__global__ void __launch_bounds__(ms_threads(S), MB) ms_dslash1_kernel(Geom g, int pv, LinkSet fat, LinkSet lng,
                                                          const void *p0, void *tmp, int q, int slot, MsState *st,
                                                          double *partials)
{
    pdl_trigger();
    __shared__ double sm[32];
    typedef typename Acc2<LP, LP>::T T;
    T acc[6];
    double tt = 0.0;
    int i;
    bool on;
    const bool mine = ms_site<LP, 0, T, S>(g, pv, fat, lng, p0, q, &st->active[slot], i, acc, &on);
    if (!on) return;
    if (mine) {
        st_spinor_as<SO>(tmp, pv, i, acc);
#pragma unroll
        for (int k = 0; k < 6; ++k) tt += (double)acc[k] * (double)acc[k];
    }
    if (!grid_arrive(tt, partials, &st->ticket[1], sm)) return;
    const double sp = st->shift[0] * st->pp, rr = st->rNorm2;  // in flight with the partials
    const double tot = partials_sum(partials, (int)gridDim.x, sm);
    if (threadIdx.x == 0) {
        st->ticket[1] = 0u;
        ms_beta(st, slot, rr, sp + tot);
    }
}

// K2: s = sigma0 p0 - D tmp (tmp stored in SI, links LP; s stays in registers); r^(i+1) = r^(i) + B0 s into the
// ring; |r|^2, then the alpha step
template <int LP, int SI, int S, int MB>
__global__ void __launch_bounds__(ms_threads(S), MB) ms_dslash2_kernel(Geom g, int pv, LinkSet fat, LinkSet lng,
                                                          const void *tmp, const void *p0, char *ring, size_t vb,
                                                          int p, int slot, MsState *st, double *partials)
{
    pdl_trigger();
    __shared__ double sm[32];
    typedef typename Acc2<LP, LP>::T T;
    T acc[6];
    double nn = 0.0;
    int i;
    bool on;
    const bool mine = ms_site<LP, SI, T, S>(g, pv, fat, lng, tmp, p, &st->active[slot], i, acc, &on);
    if (!on) return;
    if (mine) {
        const int it = st->iter;  // iterations completed before this one
        const char *rin = ring + (size_t)(it % kWin) * vb;
        char *rout = ring + (size_t)((it + 1) % kWin) * vb;
        double pv6[6], rv[6];
        ld_spinor_coherent<0>(p0, pv, i, pv6);
        ld_spinor_coherent<0>(rin, pv, i, rv);
        const double sig = st->shift[0], b0 = st->b0;
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            rv[k] += b0 * (sig * pv6[k] - (double)acc[k]);
            nn += rv[k] * rv[k];
        }
        st_spinor<0>(rout, pv, i, rv);
    }
    if (!grid_arrive(nn, partials, &st->ticket[2], sm)) return;
    const double rr = st->rNorm2;
    const double tot = partials_sum(partials, (int)gridDim.x, sm);
    if (threadIdx.x == 0) {
        st->ticket[2] = 0u;
        ms_alpha(st, rr, tot);
    }
}

// K3: p0 = r^(i) + a0 p0; block 0 takes the shift step meanwhile
__global__ void __launch_bounds__(kBSm) ms_p0_kernel(int vh, int pv, const char *ring, size_t vb, void *p0,
                                                     int slot, MsState *st)
{
    pdl_trigger();
    pdl_wait();
    const bool on = st->active[slot] != 0;
    if (blockIdx.x == 0) {
        const bool go = on && ms_shift_step(st);
        if (threadIdx.x == 0) st->active[1 - slot] = go ? 1 : 0;
        return;
    }
    if (!on) return;
    const int i = (blockIdx.x - 1) * kBSm + threadIdx.x;
    if (i >= vh) return;
    const char *r = ring + (size_t)(st->iter % kWin) * vb;
    double rv[6], pv6[6];
    ld_spinor_coherent<0>(r, pv, i, rv);
    ld_spinor_coherent<0>(p0, pv, i, pv6);
    const double a0 = st->a0;
#pragma unroll
    for (int k = 0; k < 6; ++k) pv6[k] = rv[k] + a0 * pv6[k];
    st_spinor<0>(p0, pv, i, pv6);
}

// K4: windowed shift update p_k <- c_k p_k + sum_l d_kl r_l ; x_k <- x_k + e_k p_k + sum_l f_kl r_l
template <int KU>
__global__ void __launch_bounds__(kBSm, 2) ms_window_kernel(int vh, int pv, const char *ring, size_t vb, char *pw0,
                                                         char *x0, MsState *st)
{
    __shared__ double sc[kMaxShift], se[kMaxShift], sd[kMaxShift][kWin], sf[kMaxShift][kWin];
    __shared__ int nw, km, act;
    if (threadIdx.x == 0) {
        nw = st->wpos;
        km = st->wmax;
        act = st->active[0];
    }
    __syncthreads();
    const int n = nw, kmax = km;
    // every block reads the same wpos / active (the reset below comes after all blocks have arrived)
    if (n == 0 || (n < kWin && act)) return;  // window not full and the solve still iterating
    for (int t = threadIdx.x; t < kmax; t += kBSm) {
        sc[t] = st->c[t];
        se[t] = st->e[t];
        for (int l = 0; l < kWin; ++l) {
            sd[t][l] = st->d[t][l];
            sf[t][l] = st->f[t][l];
        }
    }
    __syncthreads();
    const int i = blockIdx.x * kBSm + threadIdx.x;
    if (i < vh) window_update_site<KU>(ring, vb, pv, i, n, kmax, sc, se, sd, sf, pw0, x0);
    // last block resets the window
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(&st->ticket[0], 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (last && threadIdx.x == 0) {
        st->wpos = 0;
        st->ticket[0] = 0;
    }
}

// Writes the polled words of the state to the host page, chunk n to slot n & 1 (slots kPollSlot bytes apart).  A kernel
// at the end of the chunk's graph: a copy behind it costs the GPU about 6 us more per chunk.
constexpr int kPollSlot = 256;
static_assert(sizeof(MsPoll) <= kPollSlot, "poll slot");
__global__ void ms_poll_kernel(char *host, MsState *st)
{
    static_assert(sizeof(MsPoll) % sizeof(int) == 0, "copied by words");
    const int slot = st->polls & 1;
    __syncwarp();
    volatile int *dst = reinterpret_cast<volatile int *>(host + slot * kPollSlot);
    const int *src = reinterpret_cast<const int *>(st);
    for (int t = threadIdx.x; t < (int)(sizeof(MsPoll) / sizeof(int)); t += 32) dst[t] = src[t];
    if (threadIdx.x == 0) st->polls += 1;
}

// shifts updated per step of the window kernel's loop (KUQCD_WINDOW_UNROLL = 1 | 2 | 4)
static int window_unroll()
{
    static const int k = [] {
        const char *e = getenv("KUQCD_WINDOW_UNROLL");
        const int v = e ? atoi(e) : 4;
        return v == 1 || v == 2 ? v : 4;
    }();
    return k;
}

// ---------------------------------------------------------------------------------------------------- driver
// Threads per site of the dslash steps, by the limits of the stand-alone kernels.  (With the launches overlapped, 16^4
// and twelve shifts: FP64 with two threads per site 12.5 ms, with four 14.3 ms; the mixed solve with the HALF steps at
// one thread per site 10.76 ms, at four 10.59 ms.)
static int ms_split(int lp, int vh)
{
    return split_of(vh, lp == P64 ? kSplitLimit64 : lp == P32 ? kSplitLimit32 : kSplitLimit16);
}

// MB: resident CTAs per SM the kernels are compiled for (0: no bound, best for S > 1: at one the compiler takes 112
// registers for FP64, S = 2 and the 16^4 solve goes from 12.8 to 13.9 ms)
template <int LP, int S, int MB>
static void enqueue_ms_dslash(const Geom &g, const GaugeDev &gd, const MsBuffers &w, int parity, int it, cudaStream_t s)
{
    const int pv = pad_sites(g.vh), nb = (g.vh + ms_sites(S) - 1) / ms_sites(S), nt = ms_threads(S);
    if constexpr (S > 1) {
        launch_pdl(ms_dslash1_kernel<LP, LP, S, MB>, nb, nt, s, g, pv, gd.fat[LP], gd.lng[LP], w.p0, w.tmp, 1 - parity,
                   it & 1, w.st, w.partials);
        launch_pdl(ms_dslash2_kernel<LP, LP, S, MB>, nb, nt, s, g, pv, gd.fat[LP], gd.lng[LP], w.tmp, w.p0, (char *)w.ring,
                   w.vb, parity, it & 1, w.st, w.partials);
    } else {
        ms_dslash1_kernel<LP, LP, S, MB><<<nb, nt, 0, s>>>(g, pv, gd.fat[LP], gd.lng[LP], w.p0, w.tmp, 1 - parity, it & 1,
                                                           w.st, w.partials);
        ms_dslash2_kernel<LP, LP, S, MB><<<nb, nt, 0, s>>>(g, pv, gd.fat[LP], gd.lng[LP], w.tmp, w.p0, (char *)w.ring, w.vb,
                                                           parity, it & 1, w.st, w.partials);
    }
}

template <int LP>
static void enqueue_ms_chunk(const Geom &g, const GaugeDev &gd, const MsBuffers &w, int parity, char *host_poll,
                             cudaStream_t s)
{
    const int pv = pad_sites(g.vh), nb = (g.vh + kBSm - 1) / kBSm;
    const int S = ms_split(LP, g.vh);
    for (int it = 0; it < kChunk; ++it) {
        switch (S) {
            case 8: enqueue_ms_dslash<LP, 8, 0>(g, gd, w, parity, it, s); break;
            case 4: enqueue_ms_dslash<LP, 4, 0>(g, gd, w, parity, it, s); break;
            case 2: enqueue_ms_dslash<LP, 2, 0>(g, gd, w, parity, it, s); break;
            default:
                if (LP == 0 && fp64_four_ctas(g.vh)) enqueue_ms_dslash<LP, 1, LP == 0 ? 4 : SiteCtas<LP>::v>(g, gd, w, parity, it, s);
                else enqueue_ms_dslash<LP, 1, SiteCtas<LP>::v>(g, gd, w, parity, it, s);
                break;
        }
        if (S > 1) launch_pdl(ms_p0_kernel, nb + 1, kBSm, s, g.vh, pv, (const char *)w.ring, w.vb, w.p0, it & 1, w.st);
        else ms_p0_kernel<<<nb + 1, kBSm, 0, s>>>(g.vh, pv, (const char *)w.ring, w.vb, w.p0, it & 1, w.st);
    }
    switch (window_unroll()) {
        case 1: ms_window_kernel<1><<<nb, kBSm, 0, s>>>(g.vh, pv, (const char *)w.ring, w.vb, (char *)w.pw, (char *)w.x, w.st); break;
        case 2: ms_window_kernel<2><<<nb, kBSm, 0, s>>>(g.vh, pv, (const char *)w.ring, w.vb, (char *)w.pw, (char *)w.x, w.st); break;
        default: ms_window_kernel<4><<<nb, kBSm, 0, s>>>(g.vh, pv, (const char *)w.ring, w.vb, (char *)w.pw, (char *)w.x, w.st); break;
    }
    ms_poll_kernel<<<1, 32, 0, s>>>(host_poll, w.st);
}

static void enqueue_ms_chunk(int m, const Geom &g, const GaugeDev &gd, const MsBuffers &w, int parity, char *host_poll,
                             cudaStream_t s)
{
    if (m == 0) enqueue_ms_chunk<0>(g, gd, w, parity, host_poll, s);
    else if (m == 1) enqueue_ms_chunk<1>(g, gd, w, parity, host_poll, s);
    else enqueue_ms_chunk<2>(g, gd, w, parity, host_poll, s);
}

size_t ms_workspace_bytes(const Geom &g, int ns)
{
    MsBuffers w;
    Carve c(nullptr);
    ms_layout(c, g, ns, nullptr, nullptr, w);
    return c.off;
}

void ms_layout(Carve &c, const Geom &g, int ns, const void *d_b, void *d_x, MsBuffers &w)
{
    const size_t vb = spinor_bytes(g, P64);
    const int nb = (g.vh + 31) / 32;  // the most blocks a reduction kernel has (32 sites per CTA)
    w.vb = vb;
    w.b = d_b;
    w.x = d_x;
    w.p0 = c.take(vb);
    w.tmp = c.take(vb);  // big enough for any temporary precision
    w.ring = c.take(vb * kWin);
    w.pw = c.take(vb * ns);
    w.partials = static_cast<double *>(c.take(sizeof(double) * nb));
    w.st = static_cast<MsState *>(c.take(sizeof(MsState)));
}

cudaError_t ms_solve(::kq_context *ctx, const MsBuffers &w, int parity, int ns, const double *shifts_ref, double tol,
                     int max_iter, double rho32, double rho16, MsResult *res)
{
    const Geom &g = ctx->g;
    cudaStream_t s = ctx->stream;
    if (ns < 1 || ns > kMaxShift) {
        set_last_error("multishift: num_shift out of range (1..64)");
        return cudaErrorInvalidValue;
    }
    const bool use32 = rho32 > 0.0, use16 = rho16 > 0.0;
    if (!ctx->gd.have[P64] || (use32 && !ctx->gd.have[P32]) || (use16 && !ctx->gd.have[P16])) {
        set_last_error("multishift: links not resident in a precision the schedule needs");
        return cudaErrorInvalidValue;
    }
    MsState h;
    memset(&h, 0, sizeof(h));
    h.ns = ns;
    h.max_iter = max_iter;
    h.tol = tol;
    for (int k = 0; k < ns; ++k) h.shift[k] = shifts_ref[k];
    KQ_CUDA_TRY(cudaMemcpyAsync(w.st, &h, sizeof(MsState), cudaMemcpyHostToDevice, s));
    const int pv = pad_sites(g.vh), nb = (g.vh + kBSm - 1) / kBSm;
    ms_init_kernel<<<nb, kBSm, 0, s>>>(g.vh, pv, w.b, (char *)w.x, (char *)w.pw, w.vb, w.p0, (char *)w.ring, ns, w.st,
                                       w.partials);
    KQ_CUDA_TRY(cudaGetLastError());
    long long launches = 1;

    // One graph per operator precision, each kChunk iterations + the window update.  Building one takes the host about
    // 130 us (and its first launch more): the first three chunks are enqueued kernel by kernel and the graphs built
    // once two of them are in flight, so that a solve of one chunk builds none.
    cudaGraphExec_t *exec = res->exec;
    char *host_poll = reinterpret_cast<char *>(ctx->poll);
    auto build = [&](int m) -> cudaError_t {
        cudaGraph_t graph = nullptr;
        KQ_CUDA_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        enqueue_ms_chunk(m, g, ctx->gd, w, parity, host_poll, s);
        cudaError_t ee = cudaStreamEndCapture(s, &graph);
        if (ee == cudaSuccess) ee = cudaGraphInstantiate(&exec[m], graph, 0);
        if (graph) cudaGraphDestroy(graph);
        if (ee == cudaSuccess) ee = cudaGraphUpload(exec[m], s);
        if (ee != cudaSuccess) set_last_error(std::string("multishift: graph build failed: ") + cudaGetErrorString(ee));
        return ee;
    };
    // Up to two chunks are in flight: the one whose state the host waits for and, launched ahead of it, the next, so
    // that the GPU does not idle through a poll and a graph launch after every kChunk iterations (35 us of a chunk's
    // 170 us at 8^4).  The next chunk is launched ahead only where the last two states predict that the one in flight
    // neither ends the solve nor reaches a switch of precision; a wrong guess costs a chunk of no-ops, or keeps the
    // higher precision for kChunk more iterations.  Nothing is launched ahead of the first state, which is all that a
    // short solve has (two iterations at 4^4: 130 us; with a second chunk ahead and a graph built beside the first
    // 430 us).  The guess depends on the iterates alone, so a solve repeats exactly.
    cudaEvent_t done[2] = {nullptr, nullptr};
    cudaError_t err = cudaSuccess;
    for (auto &ev : done)
        if (err == cudaSuccess) err = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    int chunks[3] = {0, 0, 0};
    int launched = 0, polled = 0;
    auto mode_of = [&](double rel2) { return use16 && rel2 < rho16 * rho16 ? 2 : use32 && rel2 < rho32 * rho32 ? 1 : 0; };
    auto launch = [&](int m) {
        if (err == cudaSuccess && launched >= 3 && !exec[m]) err = build(m);
        if (err == cudaSuccess) {
            if (exec[m]) err = cudaGraphLaunch(exec[m], s);
            else {
                enqueue_ms_chunk(m, g, ctx->gd, w, parity, host_poll, s);
                err = cudaGetLastError();
            }
        }
        if (err == cudaSuccess) err = cudaEventRecord(done[launched & 1], s);
        chunks[m] += 1;
        launched += 1;
        launches += 3 * kChunk + 2;
    };
    // Shifts k >= final_from have been reported final.  A shift dropped from the iteration (k >= maxTerm) receives
    // its last update in the next window flush; once the window is flushed (wpos = 0), x_k no longer changes.
    int final_from = ns;
    auto report = [&](int mt) {
        if (ctx->solution_ready)
            for (int k = final_from - 1; k >= mt; --k) ctx->solution_ready(ctx, k, ctx->solution_ready_user);
        final_from = std::min(final_from, mt);
    };
    const int most = max_iter / kChunk + 3;  // chunks: every solve has stopped by then while its state is consistent
    double rel2 = 1.0, fall = 1.0;  // |r|^2 / |b|^2 of the last state read, and its factor over the chunk before it
    double stop2 = 0.0;              // the tolerance in the same units, once |b|^2 is known
    launch(mode_of(rel2));
    while (err == cudaSuccess) {
        const int m = mode_of(rel2);
        const double guess = rel2 * std::min(fall, 1.0);  // state after the chunk in flight
        // (a chunk runs kChunk iterations unless it ends the solve, so the cap says when the last one has been launched)
        const auto more = [&] { return launched < most && (long long)launched * kChunk < max_iter; };
        if (polled > 0 && more() && guess > stop2 && mode_of(0.1 * guess) == m) launch(m);
        // a graph that will be wanted, one per chunk in flight
        if (polled > 0 && more())
            for (int b : {m, use32 ? 1 : 0, use16 ? 2 : 0})
                if (err == cudaSuccess && !exec[b] && b >= m) {
                    err = build(b);
                    break;
                }
        if (err != cudaSuccess) break;
        err = cudaEventSynchronize(done[polled & 1]);
        if (err != cudaSuccess) break;
        const MsPoll st = *reinterpret_cast<const MsPoll *>(host_poll + (polled & 1) * kPollSlot);
        polled += 1;
        if (!st.active[0]) {
            if (st.wpos == 0) report(0);  // stopped, last window flushed: every x_k is final
            break;
        }
        const double now = st.rNorm2 / st.bnorm2;
        fall = now / rel2;
        rel2 = now;
        stop2 = tol / st.bnorm2;
        if (polled >= most) break;
        if (launched == polled) launch(mode_of(rel2));
        if (st.wpos == 0) report(st.maxTerm);  // the work it enqueues runs behind the chunks in flight
    }
    if (err == cudaSuccess) err = cudaMemcpyAsync(&h, w.st, sizeof(MsState), cudaMemcpyDeviceToHost, s);
    const cudaError_t es = cudaStreamSynchronize(s);
    for (auto &ev : done)
        if (ev) cudaEventDestroy(ev);
    if (err == cudaSuccess) err = es;
    if (err != cudaSuccess) {
        res->release();
        KQ_CUDA_TRY(err);
    }
    res->iter = h.iter;
    res->status = h.status ? h.status : (h.iter >= max_iter && h.maxTerm > 0 ? KQ_STATUS_MAXITER : 0);
    res->launches = launches;
    for (int m = 0; m < 3; ++m) res->chunks[m] = chunks[m];
    return cudaSuccess;
}

}  // namespace kq
