// The HISQ even-odd hopping term for one output site, shared by every kernel that applies it.
//
//   (D v)(x) = sum_mu [ F_mu(x) v(x+mu) + L_mu(x) v(x+3mu) - F_mu(x-mu)^dag v(x-mu) - L_mu(x-3mu)^dag v(x-3mu) ]
//
// with the reference's factors 1/2 and c3 = -1/48 already folded into the device links (dirac_hisq.cpp:464-502,
// dirac_hisq.cpp:40).  Output sites have parity p; neighbours are read from the parity-(1-p) field at their
// checkerboard index, with periodic wrap in every direction (Position::Normalize, space_time.cpp:187-197); the
// backward links live at the neighbour site on the other parity (dirac_hisq.cpp:492,499).
#pragma once
#include "kq_internal.h"
#include "kq_prec.cuh"

namespace kq {

// Periodic coordinate for hops of at most 3 (any extent >= 1, so nt = 1 wraps onto itself as in the reference).
__device__ __forceinline__ int wrap3(int v, int n)
{
    if (n > 3) return v < 0 ? v + n : (v >= n ? v - n : v);
    v %= n;
    return v < 0 ? v + n : v;
}

template <typename T>
__device__ __forceinline__ void mv_add(const T u[18], const T v[6], T acc[6])
{
    // acc += U v, U row-major
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        T re = acc[2 * r], im = acc[2 * r + 1];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const T ur = u[2 * (c + 3 * r)], ui = u[2 * (c + 3 * r) + 1];
            re += ur * v[2 * c] - ui * v[2 * c + 1];
            im += ur * v[2 * c + 1] + ui * v[2 * c];
        }
        acc[2 * r] = re;
        acc[2 * r + 1] = im;
    }
}

template <typename T>
__device__ __forceinline__ void mdv_sub(const T u[18], const T v[6], T acc[6])
{
    // acc -= U^dag v : (U^dag v)_r = sum_c conj(U_cr) v_c
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        T re = acc[2 * r], im = acc[2 * r + 1];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const T ur = u[2 * (r + 3 * c)], ui = u[2 * (r + 3 * c) + 1];
            re -= ur * v[2 * c] + ui * v[2 * c + 1];
            im -= ur * v[2 * c + 1] - ui * v[2 * c];
        }
        acc[2 * r] = re;
        acc[2 * r + 1] = im;
    }
}

// Checkerboard coordinates of output site i on parity p.
struct SiteCoord {
    int x, y, z, t, xcb;
};

__device__ __forceinline__ SiteCoord site_coord(const Geom &g, int i, int p)
{
    SiteCoord c;
    int r = i / g.hx;
    c.xcb = i - r * g.hx;
    const int r2 = r / g.n[1];
    c.y = r - r2 * g.n[1];
    c.t = r2 / g.n[2];
    c.z = r2 - c.t * g.n[2];
    c.x = 2 * c.xcb + ((c.y + c.z + c.t + p) & 1);
    return c;
}

// Neighbour checkerboard index for a hop of `hop` in direction dir.
__device__ __forceinline__ int nbr_index(const Geom &g, const SiteCoord &c, int i, int dir, int hop)
{
    switch (dir) {
        case 0: return i - c.xcb + (wrap3(c.x + hop, g.n[0]) >> 1);
        case 1: return i + (wrap3(c.y + hop, g.n[1]) - c.y) * g.sy;
        case 2: return i + (wrap3(c.z + hop, g.n[2]) - c.z) * g.sz;
        default: return i + (wrap3(c.t + hop, g.n[3]) - c.t) * g.st;
    }
}

// One link as type T.  HALF links (LP = 2) come back as raw int16 values: a site's fat-link terms are accumulated
// in units of the fat field's scale, the long-link terms have their spinor multiplied by scale_long / scale_fat
// (6 products instead of 18 on the link), and the sum is scaled once at the end (fold_scale_*).
template <int LP, typename T, bool KEEP = false>
__device__ __forceinline__ void ld_link_fold(const void *base, int pv, int dir, int i, const LinkSet &L, T u[18])
{
    if constexpr (LP == 2) {
        float q[18];
        ld_link_q16<KEEP>(base, pv, dir, i, q);
#pragma unroll
        for (int k = 0; k < 18; ++k) u[k] = (T)q[k];
    } else {
        typename Acc<LP>::T w[18];
        ld_link_any<LP, KEEP>(base, pv, dir, i, L.scale, L.recon, w);
#pragma unroll
        for (int k = 0; k < 18; ++k) u[k] = (T)w[k];
    }
}

template <int LP, typename T>
__device__ __forceinline__ T fold_scale_long(const LinkSet &fat, const LinkSet &lng)
{
    return LP == 2 ? (T)(lng.scale / fat.scale) : T(1);
}

template <int LP, typename T>
__device__ __forceinline__ void fold_scale_site(const LinkSet &fat, T acc[6])
{
    if constexpr (LP == 2) {
        const T s = (T)(fat.scale * (1.0f / 32767.0f));
#pragma unroll
        for (int k = 0; k < 6; ++k) acc[k] *= s;
    }
}

template <int LP, typename T>
__device__ __forceinline__ void fold_long_spinor(T rl, T v[6])
{
    if constexpr (LP == 2) {
#pragma unroll
        for (int k = 0; k < 6; ++k) v[k] *= rl;
    }
}

// Accumulation type of a (link precision, spinor precision) pair: double only when both are FP64.
template <int LP, int SP> struct Acc2 { using T = float; };
template <> struct Acc2<0, 0> { using T = double; };

// acc = (D src)(i) for output parity p.  src is the parity-(1-p) field.  Links in precision LP, spinors in SP.  KEEP: the
// forward links will be read again, by the backward hops of the other parity's sites in the same launch.
template <int LP, int SP, bool KEEP = false>
__device__ __forceinline__ void dslash_site2(const Geom &g, int pv, const LinkSet &fat, const LinkSet &lng,
                                             const void *src, int p, int i, typename Acc2<LP, SP>::T acc[6])
{
    using T = typename Acc2<LP, SP>::T;
    static_assert(sizeof(typename Acc<LP>::T) == sizeof(T) && sizeof(typename Acc<SP>::T) == sizeof(T),
                  "FP64 links go with FP64 spinors");
    const SiteCoord c = site_coord(g, i, p);
    // select parity planes without indexing the parameter arrays dynamically (keeps them out of local memory)
    const void *fat_p = p ? fat.par[1] : fat.par[0], *fat_q = p ? fat.par[0] : fat.par[1];
    const void *lng_p = p ? lng.par[1] : lng.par[0], *lng_q = p ? lng.par[0] : lng.par[1];
    const T rl = fold_scale_long<LP, T>(fat, lng);
#pragma unroll
    for (int k = 0; k < 6; ++k) acc[k] = T(0);
#pragma unroll
    for (int dir = 0; dir < 4; ++dir) {
        const int nf1 = nbr_index(g, c, i, dir, 1);
        const int nf3 = nbr_index(g, c, i, dir, 3);
        const int nb1 = nbr_index(g, c, i, dir, -1);
        const int nb3 = nbr_index(g, c, i, dir, -3);
        T u[18], v[6];
        ld_link_fold<LP, T, KEEP>(fat_p, pv, dir, i, fat, u);
        ld_spinor<SP>(src, pv, nf1, v);
        mv_add(u, v, acc);
        ld_link_fold<LP, T, KEEP>(lng_p, pv, dir, i, lng, u);
        ld_spinor<SP>(src, pv, nf3, v);
        fold_long_spinor<LP>(rl, v);
        mv_add(u, v, acc);
        ld_link_fold<LP>(fat_q, pv, dir, nb1, fat, u);
        ld_spinor<SP>(src, pv, nb1, v);
        mdv_sub(u, v, acc);
        ld_link_fold<LP>(lng_q, pv, dir, nb3, lng, u);
        ld_spinor<SP>(src, pv, nb3, v);
        fold_long_spinor<LP>(rl, v);
        mdv_sub(u, v, acc);
    }
    fold_scale_site<LP>(fat, acc);
}

template <int P>
__device__ __forceinline__ void dslash_site(const Geom &g, int pv, const LinkSet &fat, const LinkSet &lng,
                                            const void *src, int p, int i, typename Acc<P>::T acc[6])
{
    dslash_site2<P, P>(g, pv, fat, lng, src, p, i, acc);
}

// General form: links in LP, input spinors stored in SP, arithmetic in T (double only for FP64 links).
// Used where a sloppy operator reads an FP64 vector (the inexact-matvec phases of the multishift solver).
template <int LP, int SP, typename T>
__device__ __forceinline__ void dslash_site_t(const Geom &g, int pv, const LinkSet &fat, const LinkSet &lng,
                                              const void *src, int p, int i, T acc[6])
{
    const SiteCoord c = site_coord(g, i, p);
    const void *fat_p = p ? fat.par[1] : fat.par[0], *fat_q = p ? fat.par[0] : fat.par[1];
    const void *lng_p = p ? lng.par[1] : lng.par[0], *lng_q = p ? lng.par[0] : lng.par[1];
    const T rl = fold_scale_long<LP, T>(fat, lng);
#pragma unroll
    for (int k = 0; k < 6; ++k) acc[k] = T(0);
#pragma unroll
    for (int dir = 0; dir < 4; ++dir) {
        const int nf1 = nbr_index(g, c, i, dir, 1);
        const int nf3 = nbr_index(g, c, i, dir, 3);
        const int nb1 = nbr_index(g, c, i, dir, -1);
        const int nb3 = nbr_index(g, c, i, dir, -3);
        T u[18], v[6];
        ld_link_fold<LP>(fat_p, pv, dir, i, fat, u);
        ld_spinor_as<SP>(src, pv, nf1, v);
        mv_add(u, v, acc);
        ld_link_fold<LP>(lng_p, pv, dir, i, lng, u);
        ld_spinor_as<SP>(src, pv, nf3, v);
        fold_long_spinor<LP>(rl, v);
        mv_add(u, v, acc);
        ld_link_fold<LP>(fat_q, pv, dir, nb1, fat, u);
        ld_spinor_as<SP>(src, pv, nb1, v);
        mdv_sub(u, v, acc);
        ld_link_fold<LP>(lng_q, pv, dir, nb3, lng, u);
        ld_spinor_as<SP>(src, pv, nb3, v);
        fold_long_spinor<LP>(rl, v);
        mdv_sub(u, v, acc);
    }
    fold_scale_site<LP>(fat, acc);
}

// Split form, for lattices whose sites alone do not fill the GPU: S threads share an output site, each taking 16 / S
// terms of the sum (S = 2: two directions, 4: one direction, 8: one direction's forward or backward pair); thread
// sub * NS + s of a CTA of S * NS threads works on site s of the CTA's NS, so a warp still reads 32 consecutive
// sites of every plane.  The partial sums meet in shared memory and are added in the order of sub.  One thread per
// site is a chain of sixteen link loads in too few warps to hide them: at 8^4 (8 CTAs) the FP64 dslash took 9.5 us for
// 4 MB of links, with S = 8 3.3 us; at 16^4 14.0 us, with S = 2 9.3 us.
// Sites per CTA for a given S.
__host__ __device__ constexpr int split_sites(int S) { return S == 2 ? 64 : 32; }

// Threads per site for `sites` output sites: the most (up to 8) that keep sites * S within `limit` threads, about one
// wave of the kernel (FP64 113,664 threads, FP32 189,440).  Beyond it the extra CTAs only add partial sums.  Measured
// with S = 1 / 2 / 4 / 8 (us): FP64 12,096 sites 9.7 / 6.4 / 4.8 / 4.5, 24,192 10.8 / 7.7 / 8.7 / 7.9, 41,472 17.2 / 11.5
// / 12.9 / 14.9, 52,488 20.0 / 22.3; FP32 24,192 8.4 / 5.8 / 4.7 / 5.0, 41,472 9.1 / 6.6 / 6.3 / 6.8, 80,000 15.0 / 11.0,
// 120,000 20.6 / 22.8; HALF 19,208 6.3 / 5.4 / 4.7 / 5.1, 41,472 9.0 / 7.3 / 7.0 / 7.6, 65,536 9.2 / 9.4.  One limit per
// precision gives up 0.3 us at two of these sizes (FP64 12,096 and HALF 41,472 would run 0.3 us faster with twice the
// threads that the rule takes).
constexpr int kSplitLimit64 = 94000, kSplitLimit32 = 175000, kSplitLimit16 = 150000;
inline int split_of(int sites, int limit)
{
    return sites <= limit / 8 ? 8 : sites <= limit / 4 ? 4 : sites <= limit / 2 ? 2 : 1;
}

// Resident 256-thread CTAs per SM that the one-thread-per-site kernels are compiled for.  FP32: five (48 registers, as
// without a bound; three or four at more registers are slower: 32^4 88 and 83 against 77 us).  HALF: four; without a
// bound the compiler takes 44 registers, with too few loads in flight (solver kernels at 32^4: 72.6 and 84.7 us
// unbounded, 64.3 and 70.0 us bounded).  FP64: three (80 registers; two to three per cent over no bound on lattices from
// 16^4 to 48^4), but four where that saves the last of up to three waves: 120,000 sites are 1.06 waves of three CTAs
// per SM and 0.79 of four, 47.4 and 38.5 us; 240,000 on a full lattice 77.9 and 69.0 us.
template <int LP> struct SiteCtas { static constexpr int v = LP == 0 ? 3 : LP == 1 ? 5 : 4; };
inline bool fp64_four_ctas(int sites)
{
    constexpr int wave3 = 148 * 3 * 256, wave4 = 148 * 4 * 256;
    const int w3 = (sites + wave3 - 1) / wave3, w4 = (sites + wave4 - 1) / wave4;
    return w3 <= 3 && w4 < w3;
}

// the two terms (fat hop 1, long hop 3) of direction dir and sign `sgn`; fat_b / lng_b: the parity whose links they use
template <int LP, int SP, typename T>
__device__ __forceinline__ void dslash_hop_pair(const Geom &g, int pv, const LinkSet &fat, const LinkSet &lng,
                                                const void *fat_b, const void *lng_b, const void *src,
                                                const SiteCoord &c, int i, int dir, int sgn, T rl, T acc[6])
{
    const int n1 = nbr_index(g, c, i, dir, sgn), n3 = nbr_index(g, c, i, dir, 3 * sgn);
    T u[18], v[6];
    ld_link_fold<LP>(fat_b, pv, dir, sgn > 0 ? i : n1, fat, u);
    ld_spinor_coherent<SP>(src, pv, n1, v);
    if (sgn > 0) mv_add(u, v, acc);
    else mdv_sub(u, v, acc);
    ld_link_fold<LP>(lng_b, pv, dir, sgn > 0 ? i : n3, lng, u);
    ld_spinor_coherent<SP>(src, pv, n3, v);
    fold_long_spinor<LP>(rl, v);
    if (sgn > 0) mv_add(u, v, acc);
    else mdv_sub(u, v, acc);
}

// Programmatic dependent launch: a kernel launched with cudaLaunchAttributeProgrammaticStreamSerialization may start
// once every CTA of the kernel before it has called pdl_trigger (or ended); pdl_wait returns when that kernel is complete
// and its writes are visible.  Both do nothing in kernels launched without the attribute.  What the kernel before wrote
// is read with plain loads after the wait (ld_spinor_coherent), never through the read-only path, which assumes data
// that no one writes while the kernel runs, nor through a __restrict__ pointer, which the compiler may send there.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// acc = (D src)(i) in the threads of sub 0, which return true if `valid` (the site exists); every thread of the CTA
// calls this.  part: (S - 1) * 6 * NS values of shared memory.  ready() is called by every thread once its first two
// links are on their way and before any field is read; where it returns false (for the whole CTA) nothing is computed and
// *on is false.  A kernel that waits there for the one before it (pdl_wait) has its launch, its index arithmetic and
// these link loads overlap that kernel's end.
template <int LP, int SP, typename T, int S, typename Ready>
__device__ __forceinline__ bool dslash_site_split(const Geom &g, int pv, const LinkSet &fat, const LinkSet &lng,
                                                  const void *src, int p, int i, bool valid, T *part, T acc[6],
                                                  Ready ready, bool *on)
{
    static_assert(S == 2 || S == 4 || S == 8, "threads per site");
    constexpr int NS = split_sites(S);
    constexpr int ND = S == 2 ? 2 : 1;  // directions per thread
    const int sub = threadIdx.x / NS, s = threadIdx.x % NS;
#pragma unroll
    for (int k = 0; k < 6; ++k) acc[k] = T(0);
    const SiteCoord c = site_coord(g, valid ? i : 0, p);
    const void *fat_p = p ? fat.par[1] : fat.par[0], *fat_q = p ? fat.par[0] : fat.par[1];
    const void *lng_p = p ? lng.par[1] : lng.par[0], *lng_q = p ? lng.par[0] : lng.par[1];
    const T rl = fold_scale_long<LP, T>(fat, lng);
    const int dir0 = S == 8 ? sub >> 1 : ND * sub;
    const bool fwd0 = S < 8 || !(sub & 1);
    const int n1 = valid ? nbr_index(g, c, i, dir0, fwd0 ? 1 : -1) : 0;
    const int n3 = valid ? nbr_index(g, c, i, dir0, fwd0 ? 3 : -3) : 0;
    T u1[18], u3[18];
    if (valid) {
        ld_link_fold<LP>(fwd0 ? fat_p : fat_q, pv, dir0, fwd0 ? i : n1, fat, u1);
        ld_link_fold<LP>(fwd0 ? lng_p : lng_q, pv, dir0, fwd0 ? i : n3, lng, u3);
    }
    *on = ready();
    if (!*on) return false;
    if (valid) {
        T v[6], w[6];
        ld_spinor_coherent<SP>(src, pv, n1, v);
        ld_spinor_coherent<SP>(src, pv, n3, w);
        fold_long_spinor<LP>(rl, w);
        if (fwd0) {
            mv_add(u1, v, acc);
            mv_add(u3, w, acc);
        } else {
            mdv_sub(u1, v, acc);
            mdv_sub(u3, w, acc);
        }
        if (S < 8) dslash_hop_pair<LP, SP, T>(g, pv, fat, lng, fat_q, lng_q, src, c, i, dir0, -1, rl, acc);
#pragma unroll
        for (int d = 1; d < ND; ++d) {
            dslash_hop_pair<LP, SP, T>(g, pv, fat, lng, fat_p, lng_p, src, c, i, dir0 + d, 1, rl, acc);
            dslash_hop_pair<LP, SP, T>(g, pv, fat, lng, fat_q, lng_q, src, c, i, dir0 + d, -1, rl, acc);
        }
    }
    if (sub) {
#pragma unroll
        for (int k = 0; k < 6; ++k) part[((sub - 1) * 6 + k) * NS + s] = acc[k];
    }
    __syncthreads();
    if (sub) return false;
#pragma unroll
    for (int r = 0; r < S - 1; ++r)
#pragma unroll
        for (int k = 0; k < 6; ++k) acc[k] += part[(r * 6 + k) * NS + s];
    fold_scale_site<LP>(fat, acc);
    return valid;
}

// Multi-RHS form: the links of site i are loaded once and applied to R right-hand sides whose fields are
// src0 + sys[r] * stride (sys[r] < 0: slot unused).  acc[r] receives (D src_r)(i).  ALL: every slot is used, and no test
// keeps the compiler from loading several systems' spinors ahead of their mat-vecs (FP64, R = 4, 24^3 x 48: twelve D x
// in 647 us with the tests, 442 without).
template <int LP, int SP, int R, bool ALL = false>
__device__ __forceinline__ void dslash_site_mrhs(const Geom &g, int pv, const LinkSet &fat, const LinkSet &lng,
                                                 const char *src0, size_t stride, const int sys[R], int p, int i,
                                                 typename Acc2<LP, SP>::T acc[R][6])
{
    using T = typename Acc2<LP, SP>::T;
    const SiteCoord c = site_coord(g, i, p);
    const void *fat_p = p ? fat.par[1] : fat.par[0], *fat_q = p ? fat.par[0] : fat.par[1];
    const void *lng_p = p ? lng.par[1] : lng.par[0], *lng_q = p ? lng.par[0] : lng.par[1];
    const T rl = fold_scale_long<LP, T>(fat, lng);
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int k = 0; k < 6; ++k) acc[r][k] = T(0);
#pragma unroll
    for (int dir = 0; dir < 4; ++dir) {
        const int nf1 = nbr_index(g, c, i, dir, 1);
        const int nf3 = nbr_index(g, c, i, dir, 3);
        const int nb1 = nbr_index(g, c, i, dir, -1);
        const int nb3 = nbr_index(g, c, i, dir, -3);
        T u[18], v[6];
        ld_link_fold<LP>(fat_p, pv, dir, i, fat, u);
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (ALL || sys[r] >= 0) {
                ld_spinor<SP>(src0 + sys[r] * stride, pv, nf1, v);
                mv_add(u, v, acc[r]);
            }
        ld_link_fold<LP>(lng_p, pv, dir, i, lng, u);
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (ALL || sys[r] >= 0) {
                ld_spinor<SP>(src0 + sys[r] * stride, pv, nf3, v);
                fold_long_spinor<LP>(rl, v);
                mv_add(u, v, acc[r]);
            }
        ld_link_fold<LP>(fat_q, pv, dir, nb1, fat, u);
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (ALL || sys[r] >= 0) {
                ld_spinor<SP>(src0 + sys[r] * stride, pv, nb1, v);
                mdv_sub(u, v, acc[r]);
            }
        ld_link_fold<LP>(lng_q, pv, dir, nb3, lng, u);
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (ALL || sys[r] >= 0) {
                ld_spinor<SP>(src0 + sys[r] * stride, pv, nb3, v);
                fold_long_spinor<LP>(rl, v);
                mdv_sub(u, v, acc[r]);
            }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) fold_scale_site<LP>(fat, acc[r]);
}

// Multi-RHS form with the input fields in any storage precision SP and arithmetic in T (the batched solver's
// grouped systems: R systems on one gauge field, fields at src0 + r * stride).  The links of site i are loaded
// once per call and applied to every right-hand side r with use & (1 << r), or to all of them (ALL).
template <int LP, int SP, typename T, int R, bool ALL = false>
__device__ __forceinline__ void dslash_site_mrhs_t(const Geom &g, int pv, const LinkSet &fat, const LinkSet &lng,
                                                   const char *src0, size_t stride, unsigned use, int p, int i,
                                                   T acc[R][6])
{
    const SiteCoord c = site_coord(g, i, p);
    const void *fat_p = p ? fat.par[1] : fat.par[0], *fat_q = p ? fat.par[0] : fat.par[1];
    const void *lng_p = p ? lng.par[1] : lng.par[0], *lng_q = p ? lng.par[0] : lng.par[1];
    const T rl = fold_scale_long<LP, T>(fat, lng);
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int k = 0; k < 6; ++k) acc[r][k] = T(0);
#pragma unroll
    for (int dir = 0; dir < 4; ++dir) {
        const int nf1 = nbr_index(g, c, i, dir, 1);
        const int nf3 = nbr_index(g, c, i, dir, 3);
        const int nb1 = nbr_index(g, c, i, dir, -1);
        const int nb3 = nbr_index(g, c, i, dir, -3);
        T u[18], v[6];
        ld_link_fold<LP>(fat_p, pv, dir, i, fat, u);
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (ALL || (use & (1u << r))) {
                ld_spinor_as<SP>(src0 + r * stride, pv, nf1, v);
                mv_add(u, v, acc[r]);
            }
        ld_link_fold<LP>(lng_p, pv, dir, i, lng, u);
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (ALL || (use & (1u << r))) {
                ld_spinor_as<SP>(src0 + r * stride, pv, nf3, v);
                fold_long_spinor<LP>(rl, v);
                mv_add(u, v, acc[r]);
            }
        ld_link_fold<LP>(fat_q, pv, dir, nb1, fat, u);
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (ALL || (use & (1u << r))) {
                ld_spinor_as<SP>(src0 + r * stride, pv, nb1, v);
                mdv_sub(u, v, acc[r]);
            }
        ld_link_fold<LP>(lng_q, pv, dir, nb3, lng, u);
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (ALL || (use & (1u << r))) {
                ld_spinor_as<SP>(src0 + r * stride, pv, nb3, v);
                fold_long_spinor<LP>(rl, v);
                mdv_sub(u, v, acc[r]);
            }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) fold_scale_site<LP>(fat, acc[r]);
}

// ------------------------------------------------------------------------------------------------ reductions
// Deterministic block sum of a double (fixed shuffle tree, then warp 0 over the per-warp sums).
__device__ __forceinline__ double block_sum(double v, double *smem32)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) smem32[w] = v;
    __syncthreads();
    const int nw = (blockDim.x + 31) >> 5;
    v = (threadIdx.x < nw) ? smem32[threadIdx.x] : 0.0;
    if (w == 0) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    }
    return v;  // valid in thread 0
}

// Publish this block's partial sum; returns true in every thread of the last block to arrive.  Every block calls
// this unconditionally.
__device__ __forceinline__ bool grid_arrive(double v, double *partials, unsigned *ticket, double *smem32)
{
    __shared__ bool am_last;
    v = block_sum(v, smem32);
    if (threadIdx.x == 0) {
        partials[blockIdx.x] = v;
        __threadfence();
        am_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!am_last) return false;
    __threadfence();
    return true;
}

// Fixed-order sum of n partials by the last block (the total in thread 0).  Each thread adds every blockDim.x-th
// partial; eight loads are in flight before the first is added (one at a time, the 2048 partials of a 32^4 lattice
// cost eight round trips to L2 in the tail of the kernel).
__device__ __forceinline__ double partials_sum(const double *partials, int n, double *smem32)
{
    constexpr int U = 8;
    double s = 0.0;
    for (int b0 = threadIdx.x; b0 < n; b0 += U * blockDim.x) {
        double w[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int b = b0 + u * (int)blockDim.x;
            w[u] = b < n ? *((volatile const double *)partials + b) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) s += w[u];
    }
    return block_sum(s, smem32);
}

// grid_arrive + partials_sum: true in the 32 threads of warp 0 of the last block to arrive, each holding in *total
// the fixed-order sum of all partials; the ticket is reset.
__device__ __forceinline__ bool grid_sum_last_warp(double v, double *partials, unsigned *ticket, double *smem32,
                                                   double *total)
{
    if (!grid_arrive(v, partials, ticket, smem32)) return false;
    const double s = partials_sum(partials, (int)gridDim.x, smem32);
    if (threadIdx.x >= 32) return false;
    *total = __shfl_sync(0xffffffffu, s, 0);
    if (threadIdx.x == 0) *ticket = 0u;
    return true;
}

// As grid_sum_last_warp, but true in exactly one thread (thread 0 of the last block).
__device__ __forceinline__ bool grid_sum_last(double v, double *partials, unsigned *ticket, double *smem32,
                                              double *total)
{
    return grid_sum_last_warp(v, partials, ticket, smem32, total) && threadIdx.x == 0;
}

}  // namespace kq
