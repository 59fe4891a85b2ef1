// FP64 true residuals |b - (sigma - D_pq D_qp) x| / |b| on the device (the check the reference never makes,
// inverter_cgm.cpp:71-77 only tracks the recursive residual).
#include <vector>

#include "kq_dslash_core.cuh"
#include "kq_solver.h"

namespace kq {

__global__ void __launch_bounds__(256) resid_partials_kernel(int vh, int pv, const void *__restrict__ b,
                                                             const void *__restrict__ s, double *partials)
{
    __shared__ double sm[32];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double rr = 0.0, bb = 0.0;
    if (i < vh) {
        double bv[6], sv[6];
        ld_spinor<0>(b, pv, i, bv);
        ld_spinor<0>(s, pv, i, sv);
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const double d = bv[k] - sv[k];
            rr += d * d;
            bb += bv[k] * bv[k];
        }
    }
    rr = block_sum(rr, sm);
    __syncthreads();
    bb = block_sum(bb, sm);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = rr;
        partials[2 * blockIdx.x + 1] = bb;
    }
}

// Residuals of several shifts together: the links of a site are loaded once for R solutions, in both halves of the
// operator, and nothing but D x_k is stored.  One operator application per shift read every link 2 n times (12 shifts
// at 24^3 x 48: 24 launches of 102 us).  FP64 accumulators of R = 4 fit 128-thread CTAs at three per SM: 12 D x_k at
// 24^3 x 48 took 768 us one at a time, 488 with R = 2, 465 with R = 3, 442 with R = 4 (455 with 6, whose registers
// leave two CTAs).  The shifts are dealt to groups of equal size, or of two sizes that differ by one, each size a launch
// of its own without idle slots.  Groups are the fastest index of the grid: a tile's groups find its links in the L2.
constexpr int kBSr = 128;
template <int R> struct ResidCtas { static constexpr int v = R >= 3 ? 3 : R == 2 ? 4 : 6; };

struct ResidSigma {
    double v[kMaxShift];
};

// t_k = D x_k on parity q for ng groups of R shifts
template <int R>
__global__ void __launch_bounds__(kBSr, ResidCtas<R>::v) resid_dslash_kernel(Geom g, int pv, LinkSet fat, LinkSet lng,
                                                                             const char *__restrict__ x, size_t xstride,
                                                                             char *__restrict__ t, size_t vb, int ng,
                                                                             int q)
{
    const int k0 = (int)(blockIdx.x % ng) * R, i = (int)(blockIdx.x / ng) * kBSr + (int)threadIdx.x;
    if (i >= g.vh) return;
    double acc[R][6];
    dslash_site_mrhs_t<0, 0, double, R, true>(g, pv, fat, lng, x + k0 * xstride, xstride, 0, q, i, acc);
#pragma unroll
    for (int r = 0; r < R; ++r) st_spinor<0>(t + (k0 + r) * vb, pv, i, acc[r]);
}

// partial sums of |b - (sigma_k x_k - D t_k)|^2 (slot k) and, from the first group, of |b|^2 (slot bslot), one per tile
template <int R>
__global__ void __launch_bounds__(kBSr, ResidCtas<R>::v) resid_norm_kernel(Geom g, int pv, LinkSet fat, LinkSet lng,
                                                                           const char *__restrict__ t, size_t vb,
                                                                           const char *__restrict__ x, size_t xstride,
                                                                           const void *__restrict__ b, ResidSigma sigma,
                                                                           int ng, int p, double *partials, int ntiles,
                                                                           int slot0, int bslot)
{
    __shared__ double sm[32];
    const int k0 = (int)(blockIdx.x % ng) * R, tile = blockIdx.x / ng, i = tile * kBSr + (int)threadIdx.x;
    double rr[R], bb = 0.0;
#pragma unroll
    for (int r = 0; r < R; ++r) rr[r] = 0.0;
    if (i < g.vh) {
        double acc[R][6], bv[6];
        dslash_site_mrhs_t<0, 0, double, R, true>(g, pv, fat, lng, t + k0 * vb, vb, 0, p, i, acc);
        ld_spinor<0>(b, pv, i, bv);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            double xv[6];
            ld_spinor<0>(x + (k0 + r) * xstride, pv, i, xv);
            const double sg = sigma.v[slot0 + k0 + r];
#pragma unroll
            for (int e = 0; e < 6; ++e) {
                const double d = bv[e] - (sg * xv[e] - acc[r][e]);
                rr[r] += d * d;
            }
        }
#pragma unroll
        for (int e = 0; e < 6; ++e) bb += bv[e] * bv[e];
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const double v = block_sum(rr[r], sm);
        if (threadIdx.x == 0) partials[(size_t)(slot0 + k0 + r) * ntiles + tile] = v;
    }
    if (bslot >= 0 && k0 == 0) {
        const double v = block_sum(bb, sm);
        if (threadIdx.x == 0) partials[(size_t)bslot * ntiles + tile] = v;
    }
}

// out[slot] = sum of the slot's partials, in a fixed order (one block per slot)
__global__ void __launch_bounds__(256) resid_sum_kernel(const double *__restrict__ partials, int ntiles,
                                                        double *__restrict__ out)
{
    __shared__ double sm[32];
    const double v = partials_sum(partials + (size_t)blockIdx.x * ntiles, ntiles, sm);
    if (threadIdx.x == 0) out[blockIdx.x] = v;
}

template <int R>
static void launch_resid(const Geom &g, const GaugeDev &gd, int parity, int ng, const ResidSigma &sigma, const void *b,
                         const char *x, size_t xstride, char *tmp, double *partials, int ntiles, int slot0, int bslot,
                         cudaStream_t s)
{
    const int pv = pad_sites(g.vh);
    const size_t vb = spinor_bytes(g, P64);
    resid_dslash_kernel<R><<<ntiles * ng, kBSr, 0, s>>>(g, pv, gd.fat[P64], gd.lng[P64], x, xstride, tmp, vb, ng,
                                                        1 - parity);
    resid_norm_kernel<R><<<ntiles * ng, kBSr, 0, s>>>(g, pv, gd.fat[P64], gd.lng[P64], tmp, vb, x, xstride, b, sigma,
                                                      ng, parity, partials, ntiles, slot0, bslot);
}

// Workspace of true_residuals: `fields` temporaries, the partial sums and the totals.
int resid_tiles(const Geom &g) { return (g.vh + kBSr - 1) / kBSr; }
size_t resid_partials_bytes(const Geom &g, int ns) { return sizeof(double) * (size_t)resid_tiles(g) * (ns + 1); }

// |b - (sigma_k - D D) x_k|^2 for every k and |b|^2 of one parity: sums[0 .. ns - 1], sums[ns] on the host (pinned).
// x fields xstride bytes apart; tmp holds `fields` >= 1 of them, so at most that many shifts go in a launch.
cudaError_t residual_norms(const Geom &g, const GaugeDev &gd, int parity, int ns, const double *sigma, const void *d_b,
                           const void *d_x, size_t xstride, void *tmp, int fields, double *partials, double *d_sums,
                           double *sums, cudaStream_t s)
{
    const int ntiles = resid_tiles(g);
    char *t = static_cast<char *>(tmp);
    ResidSigma sg;
    for (int k = 0; k < ns; ++k) sg.v[k] = sigma[k];
    // one solution per thread while all of them fit one wave (8^4, 12 shifts: 10.6 us per half, four per thread 14.6 us;
    // 16^4: 80.8 and 46.4 us); the links then come from the L2
    const int fit = fields < 4 ? fields : 4;
    const int most = (long long)g.vh * ns <= 148 * 3 * 256 ? 1 : fit;
    const int groups = (ns + most - 1) / most, base = ns / groups, larger = ns % groups;  // `larger` groups of base + 1
    int k0 = 0;
    for (int part = 0; part < 2; ++part) {
        const int R = part == 0 ? base + 1 : base;
        for (int left = part == 0 ? larger : groups - larger; left > 0;) {
            const int ng = left < fields / R ? left : fields / R;
            const char *x = static_cast<const char *>(d_x) + k0 * xstride;
            const int bslot = k0 == 0 ? ns : -1;
            switch (R) {
                case 1: launch_resid<1>(g, gd, parity, ng, sg, d_b, x, xstride, t, partials, ntiles, k0, bslot, s); break;
                case 2: launch_resid<2>(g, gd, parity, ng, sg, d_b, x, xstride, t, partials, ntiles, k0, bslot, s); break;
                case 3: launch_resid<3>(g, gd, parity, ng, sg, d_b, x, xstride, t, partials, ntiles, k0, bslot, s); break;
                default: launch_resid<4>(g, gd, parity, ng, sg, d_b, x, xstride, t, partials, ntiles, k0, bslot, s); break;
            }
            k0 += ng * R;
            left -= ng;
        }
    }
    resid_sum_kernel<<<ns + 1, 256, 0, s>>>(partials, ntiles, d_sums);
    KQ_CUDA_TRY(cudaGetLastError());
    KQ_CUDA_TRY(cudaMemcpyAsync(sums, d_sums, sizeof(double) * (ns + 1), cudaMemcpyDeviceToHost, s));
    return cudaStreamSynchronize(s);
}

// |v|^2 of one FP64 parity field (partials: 2 * nb doubles)
cudaError_t norm2_p64(const Geom &g, const void *v, double *partials, double *out, cudaStream_t s)
{
    const int nb = (g.vh + 255) / 256;
    resid_partials_kernel<<<nb, 256, 0, s>>>(g.vh, pad_sites(g.vh), v, v, partials);  // |v - v|^2, |v|^2
    KQ_CUDA_TRY(cudaGetLastError());
    std::vector<double> h(2 * (size_t)nb);
    KQ_CUDA_TRY(cudaMemcpyAsync(h.data(), partials, sizeof(double) * 2 * nb, cudaMemcpyDeviceToHost, s));
    KQ_CUDA_TRY(cudaStreamSynchronize(s));
    double bb = 0;
    for (int b = 0; b < nb; ++b) bb += h[2 * b + 1];
    *out = bb;
    return cudaSuccess;
}

}  // namespace kq
