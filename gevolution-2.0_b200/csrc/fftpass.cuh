// fftpass.cuh -- pencil passes of the 3-D real-to-complex transforms with the
// reference's pointwise physics fused into their load and solve stages.
//
// Fourier layout: kx + PP*(ky + N*kz) for kx < P = N/2 + 1 (half spectrum
// along x); the row pitch PP = N/2 + 2 is even so that every row starts on a
// 16-byte boundary.
//   fx_fwd : R2C along x for T rows (y0..y0+T-1, z); fused prepareFTsource
//   fy     : complex FFT along y for T kx-columns at one z (in place)
//   fz     : FFT along z, pointwise Fourier-space solver, inverse FFT along z,
//            for T kx-columns at one y and all components of the solve
//   fx_inv : C2R along x for T rows
#pragma once

#include "common.cuh"
#include "fftreg.cuh"
#include "kernels.h"
#include "tma.cuh"

namespace gev {

// ---------------------------------------------------------------------------
// fused source preparation (PHINONLINEAR): T00 in FP64, Tij in the field precision
// ---------------------------------------------------------------------------
// FX_COPY, FX_PREP_T00, FX_PREP_TIJ: common.cuh

template <class R> struct FxArgs {
    const R *in;          // field (component plane) to transform
    const R *phi;
    const R *chi;
    double bg, c, c2, c3; // prepareFTsource_T00 params (bgmodel, coeff, coeff2, coeff3) / Tij coeff in c
    typename CT<R>::C *out;
    double *partial;      // per-block partial sums of the source (FX_PREP_T00)
    bool clear;           // FX_COPY: leave zeros in place of the values read
};

template <class R>
__device__ __forceinline__ R ldr(const R *f, int N, int x, int y, int z)
{
    return __ldg(f + sidx(N, wrapi(x, N), wrapi(y, N), wrapi(z, N)));
}

// grids whose x and y transforms run as plane kernels, launched early
// (pdl_entry); the pass kernels of the others have more blocks than that
template <int N> __host__ __device__ constexpr bool plane_pass() { return N <= 128; }

// two adjacent values (x even: 8- or 16-byte aligned) in one load
template <bool EARLY, class R> __device__ __forceinline__ typename CT<R>::C ld_pair(const R *p)
{
    return ld<EARLY>(reinterpret_cast<const typename CT<R>::C *>(p));
}

// prepareFTsource_T00 (gevolution.hpp:160-171) at one point, in FP64: source
// s, phi and chi there, phi at the six neighbours
template <class R>
__device__ __forceinline__ double t00_point(const FxArgs<R> &a, R s_, R p_, R chi, R pxm, R pxp, R pym, R pyp, R pzm, R pzp)
{
    const double ph = (double)p_;
    double r = a.c2 * ((double)s_ - a.bg);
    r *= 1.0 - 2.0 * ph * (1.0 - ph);
    double g;
    g = (double)pxm - (double)pxp; r += 0.125 * g * g;
    g = (double)pym - (double)pyp; r += 0.125 * g * g;
    g = (double)pzm - (double)pzp; r += 0.125 * g * g;
    r += (a.c3 * (1.0 - 3.0 * ph) - a.c) * ph - a.c3 * (double)chi;
    return r;
}

template <class R>
__device__ __forceinline__ double prep_t00(const FxArgs<R> &a, int N, int x, int y, int z, double &src)
{
    const int64_t i = sidx(N, x, y, z);
    src = (double)a.in[i];
    return t00_point(a, a.in[i], a.phi[i], a.chi[i], ldr(a.phi, N, x - 1, y, z), ldr(a.phi, N, x + 1, y, z),
                     ldr(a.phi, N, x, y - 1, z), ldr(a.phi, N, x, y + 1, z), ldr(a.phi, N, x, y, z - 1),
                     ldr(a.phi, N, x, y, z + 1));
}

// prepareFTsource_Tij for one symmetric component c (00,01,02,11,12,22),
// gevolution.hpp:64-107, in the field precision R.  Diagonal:
// (phi(x+e_i) - phi(x-e_i))^2 / 2 + coeff T_ii.  Off-diagonal, the reference's
//   pi pj - p0 pij + (p0^2 - pi^2 - pj^2 + pij^2) / 2
// is evaluated in the algebraically identical form 2uv + w (u + v + w/2), with
// u = pi - p0, v = pj - p0, w = pij - pi - pj + p0: the squares of the
// potential cancel exactly in that form, so it keeps full relative accuracy in
// FP32 where the reference's form loses (phi / grad phi)^2 to cancellation.
template <class R>
__device__ __forceinline__ R prep_tij(const R *T, const R *phi, R coeff, int c, int N, int x, int y, int z)
{
    const int64_t i = sidx(N, x, y, z);
    const R t = __ldg(T + i);
    const int ai = (c == 0 || c == 1 || c == 2) ? 0 : (c == 5 ? 2 : 1);
    const int aj = (c == 0) ? 0 : (c == 1 ? 1 : ((c == 2 || c == 4 || c == 5) ? 2 : 1));
    const int ei[3] = {ai == 0, ai == 1, ai == 2}, ej[3] = {aj == 0, aj == 1, aj == 2};
    if (ai == aj) {
        const R g = ldr(phi, N, x + ei[0], y + ei[1], z + ei[2]) - ldr(phi, N, x - ei[0], y - ei[1], z - ei[2]);
        return (R)0.5 * g * g + coeff * t;
    }
    const R p0 = __ldg(phi + i);
    const R pi_ = ldr(phi, N, x + ei[0], y + ei[1], z + ei[2]);
    const R pj = ldr(phi, N, x + ej[0], y + ej[1], z + ej[2]);
    const R pij = ldr(phi, N, x + ei[0] + ej[0], y + ei[1] + ej[1], z + ei[2] + ej[2]);
    const R u = pi_ - p0, v = pj - p0, w = (pij - pi_) - (pj - p0);
    return (R)2 * u * v + w * (u + v + (R)0.5 * w) + coeff * t;
}

// ---------------------------------------------------------------------------
// x pass, forward: real rows -> half spectrum.  grid (N/T, N, ncomp), R2 * T
// threads.  A row of N reals is transformed as N/2 complex pairs (two-step
// register FFT) and unfolded into kx = 0 .. N/2.
// ---------------------------------------------------------------------------
// the transform of `LINES` rows whose step 1 is stored: step 2 in place (R2
// threads per line), then each warp unfolds whole rows.  With Z the transform
// of the row's pairs, ze = (Z[k] + conj Z[M-k]) / 2 and
// zo = (Z[k] - conj Z[M-k]) / 2i: kx = k gets ze + w zo, kx = M - k its mirror
// conj(ze - w zo), from the same two values.  dst(l) is the output row of
// line l.
template <int M, int LINES, int NT, bool EX, class C, class DST>
__device__ __forceinline__ void fx_finish(C *smem, const C *__restrict__ tw_full, DST &&dst)
{
    using R = decltype(smem->x);
    constexpr int R1 = RegPlan<M>::R1, R2 = RegPlan<M>::R2, ES = exch_size<M, 1>();
    constexpr int GRP = NT / R2, NW = (NT + 31) / 32;
    const int u = threadIdx.x % R2;
#pragma unroll 1
    for (int l = threadIdx.x / R2; l < LINES; l += GRP) {
        C *buf = smem + l * ES;
        for (int q = u; q < R1; q += R2) {
            C v[R2];
            step2_load<M, -1, EX, 1>(v, buf, q);
#pragma unroll
            for (int p = 0; p < R2; p++) buf[q * (R2 + 1) + p] = v[p];
        }
    }
    __syncthreads();
#pragma unroll 1
    for (int l = threadIdx.x / 32; l < LINES; l += NW) {
        const C *buf = smem + l * ES;
        C *out = dst(l);
#pragma unroll 4
        for (int k = threadIdx.x % 32; k <= M / 2; k += 32) {
            const int m = k == 0 ? 0 : M - k;
            const C zk = buf[(k % R1) * (R2 + 1) + k / R1];
            C zm = buf[(m % R1) * (R2 + 1) + m / R1];
            zm.y = -zm.y;
            const C ze = cscale(cadd(zk, zm), R(0.5)), d = csub(zk, zm);
            const C wo = cmul(__ldg(tw_full + k), mk(R(0.5) * d.y, R(-0.5) * d.x));
            out[k] = cadd(ze, wo);
            if (k < M / 2) out[M - k] = cconj(csub(ze, wo));
        }
    }
}

// the pair of sources at x = 2n, 2n + 1 of row (y, z)
template <class R, int N, int MODE, int COMP>
__device__ __forceinline__ typename CT<R>::C fx_pair(const FxArgs<R> &a, const R *in, int n, int y, int z, double &lsum)
{
    constexpr bool E = plane_pass<N>();
    const int x0 = 2 * n;
    if constexpr (MODE == FX_COPY) {
        // a caller's own array (gev_poisson_noalloc) may be aligned to single values only
        const R *p = in + sidx(N, x0, y, z);
        if (reinterpret_cast<uintptr_t>(in) % (2 * sizeof(R)) == 0) return *reinterpret_cast<const typename CT<R>::C *>(p);
        return mk(p[0], p[1]);
    } else if constexpr (MODE == FX_PREP_T00) {
        const int xm = x0 == 0 ? N - 1 : x0 - 1, x2 = x0 + 2 == N ? 0 : x0 + 2;
        const int ym = y == 0 ? N - 1 : y - 1, yp = y == N - 1 ? 0 : y + 1;
        const int zm = z == 0 ? N - 1 : z - 1, zp = z == N - 1 ? 0 : z + 1;
        const auto s = ld_pair<E>(in + sidx(N, x0, y, z)), ch = ld_pair<E>(a.chi + sidx(N, x0, y, z));
        const R *row = a.phi + sidx(N, 0, y, z);
        const auto p0 = ld_pair<E>(row + x0);
        const R pm = ld<E>(row + xm), p2 = ld<E>(row + x2);
        const auto ya = ld_pair<E>(a.phi + sidx(N, x0, ym, z)), yb = ld_pair<E>(a.phi + sidx(N, x0, yp, z));
        const auto za = ld_pair<E>(a.phi + sidx(N, x0, y, zm)), zb = ld_pair<E>(a.phi + sidx(N, x0, y, zp));
        lsum += (double)s.x + (double)s.y;
        return mk((R)t00_point(a, s.x, p0.x, ch.x, pm, p0.y, ya.x, yb.x, za.x, zb.x),
                  (R)t00_point(a, s.y, p0.y, ch.y, p0.x, p2, ya.y, yb.y, za.y, zb.y));
    } else if constexpr (MODE == FX_PREP_TIJ) {
        // one component of prepareFTsource_Tij (COMP in the order 00,01,02,11,12,22),
        // the expressions of tij6_point
        const R rc = (R)a.c;
        const auto t = ld_pair<E>(in + sidx(N, x0, y, z));
        const int ym = y == 0 ? N - 1 : y - 1, yp = y == N - 1 ? 0 : y + 1;
        const int zm = z == 0 ? N - 1 : z - 1, zp = z == N - 1 ? 0 : z + 1;
        const int xm = x0 == 0 ? N - 1 : x0 - 1, x2 = x0 + 2 == N ? 0 : x0 + 2;
        auto pair = [&](int yy, int zz) { return ld_pair<E>(a.phi + sidx(N, x0, yy, zz)); };
        auto one = [&](int x, int yy, int zz) { return ld<E>(a.phi + sidx(N, x, yy, zz)); };
        auto diag = [&](R p, R m, R tv) { const R g = p - m; return (R)0.5 * g * g + rc * tv; };
        auto off = [&](R p0, R pi, R pj, R pij, R tv) {
            const R u = pi - p0, v = pj - p0, w = (pij - pi) - (pj - p0);
            return (R)2 * u * v + w * (u + v + (R)0.5 * w) + rc * tv;
        };
        if constexpr (COMP == 0) {
            const auto c = pair(y, z);
            return mk(diag(c.y, one(xm, y, z), t.x), diag(one(x2, y, z), c.x, t.y));
        } else if constexpr (COMP == 3 || COMP == 5) {
            const auto p = COMP == 3 ? pair(yp, z) : pair(y, zp), m = COMP == 3 ? pair(ym, z) : pair(y, zm);
            return mk(diag(p.x, m.x, t.x), diag(p.y, m.y, t.y));
        } else if constexpr (COMP == 4) {
            const auto c = pair(y, z), py = pair(yp, z), pz = pair(y, zp), pyz = pair(yp, zp);
            return mk(off(c.x, py.x, pz.x, pyz.x, t.x), off(c.y, py.y, pz.y, pyz.y, t.y));
        } else {
            // 01 and 02: x and the other axis
            const auto c = pair(y, z), o = COMP == 1 ? pair(yp, z) : pair(y, zp);
            const R c2 = one(x2, y, z), o2 = COMP == 1 ? one(x2, yp, z) : one(x2, y, zp);
            return mk(off(c.x, c.y, o.x, o.y, t.x), off(c.y, c2, o.y, o2, t.y));
        }
    } else {
        // FX_PREP_T0I: T0i component c completed from its potential-free sum S_c at
        // vertex x: T0i_c(x) = (1 + phi(x) + phi(x + e_c)) S_c(x) -- the per-vertex
        // factor of particle_T0i_project (gevolution.hpp:2031-2201), applied once
        // per vertex with the current phi
        static_assert(MODE == FX_PREP_T0I, "mode");
        const auto s = ld_pair<E>(in + sidx(N, x0, y, z));
        const R *row = a.phi + sidx(N, 0, y, z);
        const auto p0 = ld_pair<E>(row + x0);
        typename CT<R>::C pe;
        if constexpr (COMP == 0) pe = mk(p0.y, ld<E>(row + (x0 + 2 == N ? 0 : x0 + 2)));
        else if constexpr (COMP == 1) pe = ld_pair<E>(a.phi + sidx(N, x0, y == N - 1 ? 0 : y + 1, z));
        else pe = ld_pair<E>(a.phi + sidx(N, x0, y, z == N - 1 ? 0 : z + 1));
        return mk(((R)1 + p0.x + pe.x) * s.x, ((R)1 + p0.y + pe.y) * s.y);
    }
}

// sum of v over the block's NT threads (any NT), written by thread 0
template <int NT> __device__ __forceinline__ void block_sum(double v, double *out)
{
    __shared__ double red[(NT + 31) / 32];
    for (int o = 16; o > 0; o >>= 1) {
        const double up = __shfl_down_sync(__activemask(), v, o);
        if ((int)(threadIdx.x & 31) + o < 32 && (int)threadIdx.x + o < NT) v += up;
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < (NT + 31) / 32; w++) s += red[w];
        *out = s;
    }
}

// zeros in place of the pairs that thread u of row (y, z) has read (every pair
// has one reader), after all of its loads
template <class R, int N>
__device__ __forceinline__ void fx_clear(const R *in, int u, int y, int z)
{
    constexpr int R1 = RegPlan<N / 2>::R1, R2 = RegPlan<N / 2>::R2;
#pragma unroll
    for (int r = 0; r < R1; r++) {
        R *w = const_cast<R *>(in) + sidx(N, 2 * (u + R2 * r), y, z);
        w[0] = R(0);
        w[1] = R(0);
    }
}

template <class R, int N, int T, int MODE, bool EX, int MINB>
__global__ void __launch_bounds__(RegPlan<N / 2>::R2 *T, MINB) k_fx_fwd(FxArgs<R> a, int64_t in_stride, int64_t out_stride,
                                                                       const typename CT<R>::C *__restrict__ tw_half,
                                                                       const typename CT<R>::C *__restrict__ tw_full)
{
    pdl_entry<false>();
    using C = typename CT<R>::C;
    constexpr int M = N / 2, PP = N / 2 + 2, R1 = RegPlan<M>::R1, R2 = RegPlan<M>::R2, NT = R2 * T, ES = exch_size<M, 1>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *smem = reinterpret_cast<C *>(smem_raw);
    const int u = threadIdx.x % R2, l = threadIdx.x / R2;
    const int y0 = blockIdx.x * T, z = blockIdx.y, comp = blockIdx.z;
    const R *in = a.in + (int64_t)comp * in_stride;
    C *out = a.out + (int64_t)comp * out_stride;
    double lsum = 0.0;
    {
        C v[R1];
        auto load = [&](auto cc) {
#pragma unroll
            for (int r = 0; r < R1; r++) v[r] = fx_pair<R, N, MODE, decltype(cc)::v>(a, in, u + R2 * r, y0 + l, z, lsum);
        };
        // the component is uniform over the block: branch around the loads, not between them
        if (MODE != FX_PREP_T0I || comp == 0) load(IntC<0>{});
        else if (comp == 1) load(IntC<1>{});
        else load(IntC<2>{});
        if (MODE == FX_COPY && a.clear) fx_clear<R, N>(in, u, y0 + l, z);
        step1_store<M, -1, EX, 1>(v, smem + l * ES, u, tw_half);
    }
    __syncthreads();
    fx_finish<M, T, NT, EX>(smem, tw_full, [&](int i) { return out + (int64_t)PP * (y0 + i + (int64_t)N * z); });

    if constexpr (MODE == FX_PREP_T00) block_sum<NT>(lsum, a.partial + blockIdx.x + gridDim.x * blockIdx.y);
}

// prepareFTsource_Tij for all six components at one point from the ten
// potential values they share (p0 = phi(x), pxp = phi(x + e_x), ..., pxy =
// phi(x + e_x + e_y)); the arithmetic of each component is that of prep_tij
// (same expressions, same order), so the results are identical.
template <class R>
__device__ __forceinline__ void tij6_point(R p0, R pxp, R pxm, R pyp, R pym, R pzp, R pzm, R pxy, R pxz, R pyz,
                                           const R t[6], R coeff, R o[6])
{
    R g;
    g = pxp - pxm; o[0] = (R)0.5 * g * g + coeff * t[0];
    g = pyp - pym; o[3] = (R)0.5 * g * g + coeff * t[3];
    g = pzp - pzm; o[5] = (R)0.5 * g * g + coeff * t[5];
    R u, v, w;
    u = pxp - p0; v = pyp - p0; w = (pxy - pxp) - (pyp - p0);
    o[1] = (R)2 * u * v + w * (u + v + (R)0.5 * w) + coeff * t[1];
    u = pxp - p0; v = pzp - p0; w = (pxz - pxp) - (pzp - p0);
    o[2] = (R)2 * u * v + w * (u + v + (R)0.5 * w) + coeff * t[2];
    u = pyp - p0; v = pzp - p0; w = (pyz - pyp) - (pzp - p0);
    o[4] = (R)2 * u * v + w * (u + v + (R)0.5 * w) + coeff * t[4];
}

// x pass, forward, for the six Tij components at once: each potential value
// is loaded once for all six sources.  grid (N/T, N); G thread groups per
// line: every group forms the sources of its share of the pairs, and
// transforms its share of the components.
template <class R, int N, int T, int G, int MINB>
__global__ void __launch_bounds__(RegPlan<N / 2>::R2 *T *G, MINB) k_fx_fwd_tij6(const R *__restrict__ Tij, int64_t n3,
                                                                              const R *__restrict__ phi, double coeff,
                                                                              typename CT<R>::C *out, int64_t out_stride,
                                                                              const typename CT<R>::C *__restrict__ tw_half,
                                                                              const typename CT<R>::C *__restrict__ tw_full)
{
    pdl_entry<false>();
    constexpr bool EX = true;   // fftreg.cuh: not a vector field
    using C = typename CT<R>::C;
    constexpr int M = N / 2, PP = N / 2 + 2, R1 = RegPlan<M>::R1, R2 = RegPlan<M>::R2, NT = R2 * T * G, ES = exch_size<M, 1>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *smem = reinterpret_cast<C *>(smem_raw);   // line c * T + l
    const int y0 = blockIdx.x * T, z = blockIdx.y;
    const R rc = (R)coeff;
    {
        const int zm = z == 0 ? N - 1 : z - 1, zp = z == N - 1 ? 0 : z + 1;
#pragma unroll 2
        for (int idx = threadIdx.x; idx < M * T; idx += NT) {
            // the points x0 = 2n and x0 + 1 of row (y, z): the potential rows
            // they touch are read as aligned pairs plus the four values beyond
            const int n = idx % M, l = idx / M, y = y0 + l;
            const int x0 = 2 * n, xm = x0 == 0 ? N - 1 : x0 - 1, x2 = x0 + 2 == N ? 0 : x0 + 2;
            const int ym = y == 0 ? N - 1 : y - 1, yp = y == N - 1 ? 0 : y + 1;
            // 32-bit offsets (N <= 768): one base register per plane
            auto row = [&](int yy, int zz) { return ((uint32_t)zz * N + (uint32_t)yy) * N; };
            const uint32_t r00 = row(y, z), rp0 = row(yp, z), r0p = row(y, zp);
            const C c00 = ld_pair<false>(phi + (r00 + x0)), cm0 = ld_pair<false>(phi + (row(ym, z) + x0)), cp0 = ld_pair<false>(phi + (rp0 + x0));
            const C c0p = ld_pair<false>(phi + (r0p + x0)), c0m = ld_pair<false>(phi + (row(y, zm) + x0)), cpp = ld_pair<false>(phi + (row(yp, zp) + x0));
            const R f00m = ld<false>(phi + (r00 + xm)), f002 = ld<false>(phi + (r00 + x2)), fp02 = ld<false>(phi + (rp0 + x2)),
                    f0p2 = ld<false>(phi + (r0p + x2));
            R t0[6], t1[6];
#pragma unroll
            for (int c = 0; c < 6; c++) {
                const C tv = ld_pair<false>(Tij + c * n3 + (r00 + x0));
                t0[c] = tv.x;
                t1[c] = tv.y;
            }
            R a0[6], a1[6];
            tij6_point(c00.x, c00.y, f00m, cp0.x, cm0.x, c0p.x, c0m.x, cp0.y, c0p.y, cpp.x, t0, rc, a0);
            tij6_point(c00.y, f002, c00.x, cp0.y, cm0.y, c0p.y, c0m.y, fp02, f0p2, cpp.y, t1, rc, a1);
            // pair n = j + R2 r waits at slot (r, j), where step 1 of thread j reads it
            C *b = smem + l * ES + (n / R2) * (R2 + 1) + n % R2;
#pragma unroll
            for (int c = 0; c < 6; c++) b[c * T * ES] = mk(a0[c], a1[c]);
        }
    }
    __syncthreads();
    const int u = threadIdx.x % R2;
#pragma unroll 1
    for (int l = threadIdx.x / R2; l < 6 * T; l += T * G) {
        C *b = smem + l * ES;
        C v[R1];
#pragma unroll
        for (int r = 0; r < R1; r++) v[r] = b[r * (R2 + 1) + u];
        step1_store<M, -1, EX, 1>(v, b, u, tw_half);
    }
    __syncthreads();
    fx_finish<M, 6 * T, NT, EX>(smem, tw_full, [&](int i) {
        return out + (i / T) * out_stride + (int64_t)PP * (y0 + i % T + (int64_t)N * z);
    });
}

// ---------------------------------------------------------------------------
// x pass, inverse: half spectrum -> real rows (imaginary parts of the kx = 0
// and kx = N/2 entries do not contribute).  grid (N/T, N, ncomp)
// ---------------------------------------------------------------------------
template <class R, int N, int T, bool EX, int MINB>
__global__ void __launch_bounds__(RegPlan<N / 2>::R2 *T, MINB) k_fx_inv(const typename CT<R>::C *in, int64_t in_stride, R *out,
                                                                       int64_t out_stride,
                                                                       const typename CT<R>::C *__restrict__ tw_half,
                                                                       const typename CT<R>::C *__restrict__ tw_full)
{
    pdl_entry<false>();
    using C = typename CT<R>::C;
    constexpr int M = N / 2, PP = N / 2 + 2, R1 = RegPlan<M>::R1, R2 = RegPlan<M>::R2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int u = threadIdx.x % R2, l = threadIdx.x / R2;   // neighbouring threads share a line
    const int y = blockIdx.x * T + l, z = blockIdx.y;
    C *buf = reinterpret_cast<C *>(smem_raw) + l * exch_size<M, 1>();
    const C *row = in + (int64_t)blockIdx.z * in_stride + (int64_t)PP * (y + (int64_t)N * z);
    {
        C v[R1];
#pragma unroll
        for (int r = 0; r < R1; r++) {
            const int k = u + R2 * r;
            C A = ld<false>(row + k), B = ld<false>(row + M - k);
            if (k == 0) { A.y = R(0); B.y = R(0); }
            B.y = -B.y;
            C w = __ldg(tw_full + k);
            w.y = -w.y;                                // exp(+2 pi i k / N)
            const C dd = cmul(csub(A, B), w), s = cadd(A, B);
            v[r] = mk(s.x - dd.y, s.y + dd.x);         // (A+B) + i (A-B) w
        }
        step1_store<M, 1, EX, 1>(v, buf, u, tw_half);
    }
    __syncthreads();
    R *dst = out + (int64_t)blockIdx.z * out_stride + sidx(N, 0, y, z);
    // a caller's own array (gev_poisson_noalloc) may be aligned to single values only
    const bool pairs = reinterpret_cast<uintptr_t>(out) % sizeof(C) == 0;
    for (int q = u; q < R1; q += R2) {
        C v[R2];
        step2_load<M, 1, EX, 1>(v, buf, q);
#pragma unroll
        for (int p = 0; p < R2; p++) {
            R *d = dst + 2 * (q + R1 * p);
            if (pairs) {
                *reinterpret_cast<C *>(d) = v[p];
            } else {
                d[0] = v[p].x;
                d[1] = v[p].y;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Small grids (N <= 128): the x and y transforms of a whole z plane in one
// kernel, the plane in shared memory between them.  At these sizes a pass is
// bound by its launch and by latency, not by its traffic: two launches of a
// solve and one pass over the spectrum go in each direction.  At 128^3 this is
// at its end: phi, chi and B_i solves take 37, 84 and 66 us in FP32 and 59, 152
// and 210 us in FP64; with the forward transforms as two passes 39, 83 and 69
// us, and 53, 142 and 205 us.
// ---------------------------------------------------------------------------
template <int N> struct PlaneShape {
    static constexpr int M = N / 2, P = M + 1;
    static constexpr int XU = RegPlan<M>::R2, YU = RegPlan<N>::R2;   // threads per row, per column
    static constexpr int NT = (P * YU + 31) / 32 * 32;               // one thread per (column, u)
    static constexpr int XES = exch_size<M, 1>(), XITEMS = N * XU, XPER = (XITEMS + NT - 1) / NT;
    static constexpr int VALUES = exch_size<N, P>() > N * XES ? exch_size<N, P>() : N * XES;
    // slot of (column k, y) while the columns are the lines (k fastest)
    __device__ __forceinline__ static int ycol(int k, int y) { return ((y / YU) * (YU + 1) + y % YU) * P + k; }
    // slot of (k, y) after the columns' transform (row y % R1 of the exchange)
    __device__ __forceinline__ static int yrow(int k, int y)
    {
        constexpr int R1 = RegPlan<N>::R1;
        return ((y % R1) * (YU + 1) + y / R1) * P + k;
    }
};

// resident CTAs: two FP32 planes of 128^2 fit an SM if the registers do too
template <class R, int N> constexpr int plane_minb() { return sizeof(R) == 4 && N == 128 ? 2 : 1; }

// forward: rows (with their source preparation), then columns; grid (N, ncomp)
template <class R, int N, int MODE, bool EX>
__global__ void __launch_bounds__(PlaneShape<N>::NT, plane_minb<R, N>()) k_plane_fwd(FxArgs<R> a, int64_t in_stride, int64_t out_stride,
                                                                 const typename CT<R>::C *__restrict__ tw_half,
                                                                 const typename CT<R>::C *__restrict__ tw_full)
{
    pdl_entry<true>();
    using C = typename CT<R>::C;
    using S = PlaneShape<N>;
    constexpr int M = S::M, P = S::P, PP = N / 2 + 2, NT = S::NT;
    constexpr int XR1 = RegPlan<M>::R1, XR2 = RegPlan<M>::R2, YR1 = RegPlan<N>::R1, YR2 = RegPlan<N>::R2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *smem = reinterpret_cast<C *>(smem_raw);
    const int z = blockIdx.x, comp = blockIdx.y;
    const R *in = a.in + (int64_t)comp * in_stride;
    double lsum = 0.0;
    auto load = [&](auto cc) {
#pragma unroll 1
        for (int w = threadIdx.x; w < S::XITEMS; w += NT) {
            const int u = w % XR2, y = w / XR2;
            C v[XR1];
#pragma unroll
            for (int r = 0; r < XR1; r++) v[r] = fx_pair<R, N, MODE, decltype(cc)::v>(a, in, u + XR2 * r, y, z, lsum);
            if (MODE == FX_COPY && a.clear) fx_clear<R, N>(in, u, y, z);
            step1_store<M, -1, EX, 1>(v, smem + y * S::XES, u, tw_half);
        }
    };
    if constexpr (MODE == FX_PREP_T0I || MODE == FX_PREP_TIJ) {
        if (comp == 0) load(IntC<0>{});
        else if (comp == 1) load(IntC<1>{});
        else if (MODE == FX_PREP_T0I || comp == 2) load(IntC<2>{});
        if constexpr (MODE == FX_PREP_TIJ) {
            if (comp == 3) load(IntC<3>{});
            else if (comp == 4) load(IntC<4>{});
            else if (comp == 5) load(IntC<5>{});
        }
    } else {
        load(IntC<0>{});
    }
    __syncthreads();
#pragma unroll 1
    for (int w = threadIdx.x; w < S::XITEMS; w += NT) {
        C *buf = smem + (w / XR2) * S::XES;
        for (int q = w % XR2; q < XR1; q += XR2) {
            C v[XR2];
            step2_load<M, -1, EX, 1>(v, buf, q);
#pragma unroll
            for (int p = 0; p < XR2; p++) buf[q * (XR2 + 1) + p] = v[p];
        }
    }
    __syncthreads();
    // unfold the rows through registers into the columns' layout
    constexpr int PAIRS = N * (M / 2 + 1), PPT = (PAIRS + NT - 1) / NT;
    C lo[PPT], hi[PPT];
#pragma unroll
    for (int i = 0; i < PPT; i++) {
        const int w = threadIdx.x + i * NT, k = w % (M / 2 + 1), y = w / (M / 2 + 1);
        if (w >= PAIRS) continue;
        const C *buf = smem + y * S::XES;
        const int m = k == 0 ? 0 : M - k;
        const C zk = buf[(k % XR1) * (XR2 + 1) + k / XR1];
        C zm = buf[(m % XR1) * (XR2 + 1) + m / XR1];
        zm.y = -zm.y;
        const C ze = cscale(cadd(zk, zm), R(0.5)), d = csub(zk, zm);
        const C wo = cmul(__ldg(tw_full + k), mk(R(0.5) * d.y, R(-0.5) * d.x));
        lo[i] = cadd(ze, wo);
        hi[i] = cconj(csub(ze, wo));
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < PPT; i++) {
        const int w = threadIdx.x + i * NT, k = w % (M / 2 + 1), y = w / (M / 2 + 1);
        if (w >= PAIRS) continue;
        smem[S::ycol(k, y)] = lo[i];
        if (k < M / 2) smem[S::ycol(M - k, y)] = hi[i];
    }
    __syncthreads();
    const int k = threadIdx.x % P, u = threadIdx.x / P;
    if (u < YR2) {
        C *buf = smem + k;
        C v[YR1];
#pragma unroll
        for (int r = 0; r < YR1; r++) v[r] = buf[(r * (YR2 + 1) + u) * P];
        step1_store<N, -1, EX, P>(v, buf, u, tw_full);
    }
    __syncthreads();
    if (u < YR2) {
        C *out = a.out + (int64_t)comp * out_stride + (int64_t)PP * N * z + k;
        for (int q = u; q < YR1; q += YR2) {
            C v[YR2];
            step2_load<N, -1, EX, P>(v, smem + k, q);
#pragma unroll
            for (int p = 0; p < YR2; p++) out[PP * (q + YR1 * p)] = v[p];
        }
    }
    if constexpr (MODE == FX_PREP_T00) block_sum<NT>(lsum, a.partial + z);
}

// inverse: columns, then rows; grid (N, ncomp)
template <class R, int N, bool EX>
__global__ void __launch_bounds__(PlaneShape<N>::NT, plane_minb<R, N>()) k_plane_inv(const typename CT<R>::C *in, int64_t in_stride, R *out,
                                                                 int64_t out_stride,
                                                                 const typename CT<R>::C *__restrict__ tw_half,
                                                                 const typename CT<R>::C *__restrict__ tw_full)
{
    pdl_entry<true>();
    using C = typename CT<R>::C;
    using S = PlaneShape<N>;
    constexpr int M = S::M, P = S::P, PP = N / 2 + 2, NT = S::NT;
    constexpr int XR1 = RegPlan<M>::R1, XR2 = RegPlan<M>::R2, YR1 = RegPlan<N>::R1, YR2 = RegPlan<N>::R2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *smem = reinterpret_cast<C *>(smem_raw);
    const int z = blockIdx.x;
    const int k0 = threadIdx.x % P, u0 = threadIdx.x / P;
    if (u0 < YR2) {
        const C *col = in + (int64_t)blockIdx.y * in_stride + (int64_t)PP * N * z + k0;
        C v[YR1];
#pragma unroll
        for (int r = 0; r < YR1; r++) v[r] = ld(col + PP * (u0 + YR2 * r));
        step1_store<N, 1, EX, P>(v, smem + k0, u0, tw_full);
    }
    __syncthreads();
    if (u0 < YR2) {
        for (int q = u0; q < YR1; q += YR2) {
            C v[YR2];
            step2_load<N, 1, EX, P>(v, smem + k0, q);
#pragma unroll
            for (int p = 0; p < YR2; p++) smem[(q * (YR2 + 1) + p) * P + k0] = v[p];
        }
    }
    __syncthreads();
    // the rows' first step in registers, then into the rows' layout
    C v[S::XPER][XR1];
#pragma unroll
    for (int i = 0; i < S::XPER; i++) {
        const int w = threadIdx.x + i * NT, u = w % XR2, y = w / XR2;
        if (w >= S::XITEMS) continue;
#pragma unroll
        for (int r = 0; r < XR1; r++) {
            const int k = u + XR2 * r;
            C A = smem[S::yrow(k, y)], B = smem[S::yrow(M - k, y)];
            if (k == 0) { A.y = R(0); B.y = R(0); }
            B.y = -B.y;
            C t = __ldg(tw_full + k);
            t.y = -t.y;                                // exp(+2 pi i k / N)
            const C dd = cmul(csub(A, B), t), sm = cadd(A, B);
            v[i][r] = mk(sm.x - dd.y, sm.y + dd.x);    // (A+B) + i (A-B) w
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < S::XPER; i++) {
        const int w = threadIdx.x + i * NT;
        if (w < S::XITEMS) step1_store<M, 1, EX, 1>(v[i], smem + (w / XR2) * S::XES, w % XR2, tw_half);
    }
    __syncthreads();
    // a caller's own array (gev_poisson_noalloc) may be aligned to single values only
    const bool pairs = reinterpret_cast<uintptr_t>(out) % sizeof(C) == 0;
#pragma unroll 1
    for (int w = threadIdx.x; w < S::XITEMS; w += NT) {
        const int y = w / XR2;
        R *dst = out + (int64_t)blockIdx.y * out_stride + sidx(N, 0, y, z);
        for (int q = w % XR2; q < XR1; q += XR2) {
            C x[XR2];
            step2_load<M, 1, EX, 1>(x, smem + y * S::XES, q);
#pragma unroll
            for (int p = 0; p < XR2; p++) {
                R *d = dst + 2 * (q + XR1 * p);
                if (pairs) {
                    *reinterpret_cast<C *>(d) = x[p];
                } else {
                    d[0] = x[p].x;
                    d[1] = x[p].y;
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// z pass with the Fourier-space solvers (gevolution.hpp:251-852).  All solver
// arithmetic is FP64; k tables hold gridk2[i] = (2N sin(pi i/N))^2 and
// kshift[i] = 2N sin(pi i/N) exp(-i pi i/N) (gevolution.hpp:269-275).
// ---------------------------------------------------------------------------
// OP_POISSON, OP_SCALAR, OP_VECTOR, OP_BIN and the EXTRA_* flags: common.cuh
// optional extras of OP_SCALAR

template <class R> struct FzArgs {
    typename CT<R>::C *data;   // component planes (stride nk)
    int64_t stride;
    const double *k2;          // gridk2[N]
    const double2 *ks;         // kshift[N]
    double p0, p1, p2, p3;     // op parameters
    int extra;
    typename CT<R>::C *hij;    // tensor state (6 planes) / B state (3 planes)
    typename CT<R>::C *hijp;
    typename CT<R>::C *bstate;
    double *phi_hom;           // k = 0 mode after the Poisson solve
    const double *partial;     // OP_POISSON: partial sums (npartial of them, null: none) summed into *sum
    int64_t npartial;
    double *sum;
    double *bins;              // OP_BIN: copies x 4 x numbins accumulators (k, k^2, P, P^2)
    unsigned long long *occ;   // OP_BIN: copies x numbins mode counts
    int *err;                  // device error word (may be null)
    const double *tab;         // OP_ZELD: ln k [h/Mpc] (ntab values) then ln P(k) (ntab values)
    int ntab;
    const double2 *modes;      // OP_ICS: [kz][ky][kx] numerators of the displacement potential
};

__device__ __forceinline__ double2 zmul(double2 a, double2 b) { return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ double2 zadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 zsub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 zsc(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
__device__ __forceinline__ double2 zcj(double2 a) { return make_double2(a.x, -a.y); }
template <class C> __device__ __forceinline__ double2 z2d(C a) { return make_double2((double)a.x, (double)a.y); }

// transverse-traceless numerators of projectFTtensor (gevolution.hpp:744-769)
__device__ __forceinline__ void tt_num(const double *g, const double2 *k, double k2, const double2 *S, double2 *o)
{
    double2 Sxx = S[0], Sxy = S[1], Sxz = S[2], Syy = S[3], Syz = S[4], Szz = S[5];
    o[0] = zadd(zadd(zsc(zadd(zsc(Sxx, g[0] - k2), zsc(zmul(k[0], zadd(zmul(k[1], Sxy), zmul(k[2], Sxz))), 2.0)), g[0] - k2),
                     zsc(Syy, (g[0] + k2) * (g[1] + k2) - 2.0 * k2 * k2)),
                zadd(zsc(Szz, (g[0] + k2) * (g[2] + k2) - 2.0 * k2 * k2), zsc(zmul(zmul(k[1], k[2]), Syz), 2.0 * (g[0] + k2))));
    o[1] = zadd(zadd(zsc(Sxy, 2.0 * (g[0] - k2) * (g[1] - k2)), zsc(zmul(zmul(zcj(k[0]), zcj(k[1])), Szz), g[2] + k2)),
                zadd(zsc(zmul(zcj(k[1]), zadd(zmul(zcj(k[0]), Sxx), zsc(zmul(k[2], Sxz), 2.0))), g[0] - k2),
                     zsc(zmul(zcj(k[0]), zadd(zmul(zcj(k[1]), Syy), zsc(zmul(k[2], Syz), 2.0))), g[1] - k2)));
    o[2] = zadd(zadd(zsc(Sxz, 2.0 * (g[0] - k2) * (g[2] - k2)), zsc(zmul(zmul(zcj(k[0]), zcj(k[2])), Syy), g[1] + k2)),
                zadd(zsc(zmul(zcj(k[2]), zadd(zmul(zcj(k[0]), Sxx), zsc(zmul(k[1], Sxy), 2.0))), g[0] - k2),
                     zsc(zmul(zcj(k[0]), zadd(zmul(zcj(k[2]), Szz), zsc(zmul(k[1], Syz), 2.0))), g[2] - k2)));
    o[3] = zadd(zadd(zsc(zadd(zsc(Syy, g[1] - k2), zsc(zmul(k[1], zadd(zmul(k[0], Sxy), zmul(k[2], Syz))), 2.0)), g[1] - k2),
                     zsc(Sxx, (g[1] + k2) * (g[0] + k2) - 2.0 * k2 * k2)),
                zadd(zsc(Szz, (g[1] + k2) * (g[2] + k2) - 2.0 * k2 * k2), zsc(zmul(zmul(k[0], k[2]), Sxz), 2.0 * (g[1] + k2))));
    o[4] = zadd(zadd(zsc(Syz, 2.0 * (g[1] - k2) * (g[2] - k2)), zsc(zmul(zmul(zcj(k[1]), zcj(k[2])), Sxx), g[0] + k2)),
                zadd(zsc(zmul(zcj(k[2]), zadd(zmul(zcj(k[1]), Syy), zsc(zmul(k[0], Sxy), 2.0))), g[1] - k2),
                     zsc(zmul(zcj(k[1]), zadd(zmul(zcj(k[2]), Szz), zsc(zmul(k[0], Sxz), 2.0))), g[2] - k2)));
    o[5] = zadd(zadd(zsc(zadd(zsc(Szz, g[2] - k2), zsc(zmul(k[2], zadd(zmul(k[0], Sxz), zmul(k[1], Syz))), 2.0)), g[2] - k2),
                     zsc(Sxx, (g[2] + k2) * (g[0] + k2) - 2.0 * k2 * k2)),
                zadd(zsc(Syy, (g[2] + k2) * (g[1] + k2) - 2.0 * k2 * k2), zsc(zmul(zmul(k[0], k[1]), Sxy), 2.0 * (g[2] + k2))));
}

template <int OP, int EXTRA> struct OpShape {
    static constexpr int CIN = (OP == OP_POISSON || OP == OP_BIN || OP == OP_ZELD || OP == OP_ICS) ? 1 : (OP == OP_SCALAR ? 6 : 3);
    static constexpr int COUT = (OP == OP_BIN) ? 0 : ((OP == OP_POISSON || OP == OP_ICS) ? 1 : (OP == OP_SCALAR ? ((EXTRA & EXTRA_VECTOR_EVOLVE) ? 4 : 1) : 3));
    static constexpr int CMAX = CIN > COUT ? CIN : COUT;   // columns the pass holds at once
    // projectFTscalar alone needs only three kz-independent combinations of the
    // six S_ij (see k_fz): the z pass transforms three columns instead of six
    static constexpr bool CONTRACT = (OP == OP_SCALAR && EXTRA == 0);
    static constexpr int CBUF = CONTRACT ? 3 : CMAX;   // exchange buffers of k_fz
    static constexpr int CTMA = CONTRACT ? 4 : CMAX;   // buffers of k_fz_tma
};

// Element-wise solver for one (kx, ky, kz): reads CIN values from v, writes
// COUT values back into v[0..COUT-1].
template <class R, int OP, int EXTRA>
__device__ __forceinline__ void fz_apply(const FzArgs<R> &a, int N, int kx, int ky, int kz, int64_t kidx, double2 *v)
{
    using C = typename CT<R>::C;
    const double g[3] = {__ldg(a.k2 + kx), __ldg(a.k2 + ky), __ldg(a.k2 + kz)};
    const double2 k[3] = {__ldg(a.ks + kx), __ldg(a.ks + ky), __ldg(a.ks + kz)};
    const double k2 = g[0] + g[1] + g[2];
    if constexpr (OP == OP_ZELD) {
        // Zel'dovich displacement of a white-noise spectrum (the generator's
        // counterpart of generateDisplacementField, ic_basic.hpp:1165-1610):
        // psi_c = i 2 pi n_c / |2 pi n|^2 * sqrt(P(k) N^3 / L^3) * w / N^3 in box
        // units, n the signed integer wavevector (numpy fftfreq convention),
        // k = 2 pi |n| / L.  p0 = L [Mpc/h], p1 != 0 cuts |n| > N/2 (k-sphere).
        const int n0 = kx, n1 = (ky < N / 2) ? ky : ky - N, n2 = (kz < N / 2) ? kz : kz - N;
        const double kk = (double)n0 * n0 + (double)n1 * n1 + (double)n2 * n2;
        const double2 w = v[0];
        v[0] = v[1] = v[2] = make_double2(0.0, 0.0);
        if (kk == 0.0 || (a.p1 != 0.0 && 4.0 * kk > (double)N * N)) return;
        const double lk = log(2.0 * 3.14159265358979323846 * sqrt(kk) / a.p0);
        int lo = 0, hi = a.ntab - 1;
        double lp;
        if (lk <= a.tab[0]) lp = a.tab[a.ntab];
        else if (lk >= a.tab[hi]) lp = a.tab[a.ntab + hi];
        else {
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (a.tab[mid] <= lk) lo = mid; else hi = mid;
            }
            const double t = (lk - a.tab[lo]) / (a.tab[hi] - a.tab[lo]);
            lp = a.tab[a.ntab + lo] + t * (a.tab[a.ntab + hi] - a.tab[a.ntab + lo]);
        }
        const double n3 = (double)N * N * N;
        const double amp = sqrt(exp(lp) * n3 / (a.p0 * a.p0 * a.p0)) / n3 / (2.0 * 3.14159265358979323846 * kk);
        const double nc[3] = {(double)n0, (double)n1, (double)n2};
#pragma unroll
        for (int c = 0; c < 3; c++) v[c] = make_double2(-nc[c] * amp * w.y, nc[c] * amp * w.x);   // i nc amp w
    } else if constexpr (OP == OP_ICS) {
        // generateDisplacementField's last factor (ic_basic.hpp:1270-1281):
        // potFT(k) = numerator(k) / potFT(k), the field holding the Fourier
        // transform of the CIC kernel; modes the generator sets to zero stay
        // zero (their numerator is exactly zero).  Complex division as
        // (n ker*) / |ker|^2.
        const double2 num = ld(a.modes + (int64_t)kx + (int64_t)(N / 2 + 1) * ((int64_t)ky + (int64_t)N * kz));
        if (num.x == 0.0 && num.y == 0.0) {
            v[0] = make_double2(0.0, 0.0);
        } else {
            const double2 ker = v[0];
            const double den = ker.x * ker.x + ker.y * ker.y;
            v[0] = make_double2((num.x * ker.x + num.y * ker.y) / den, (num.y * ker.x - num.x * ker.y) / den);
        }
    } else if constexpr (OP == OP_POISSON) {
        // solveModifiedPoissonFT: gevolution.hpp:806-852; p0 = coeff / (-N^3), p1 = modif;
        // p2 != 0 removes the k = 0 mode first (ic_basic.hpp:2419-2421)
        double den = k2 + a.p1;
        v[0] = (den != 0.0) ? zsc(v[0], a.p0 / den) : make_double2(0.0, 0.0);
        if (kx == 0 && ky == 0 && kz == 0) {
            if (a.p1 == 0.0 || a.p2 != 0.0) v[0] = make_double2(0.0, 0.0);
            if (a.phi_hom) *a.phi_hom = v[0].x;
        }
    } else if constexpr (OP == OP_VECTOR) {
        // projectFTvector: gevolution.hpp:449-515; p0 = coeff, p1 = modif
        if (k2 > 0.0) {
            double2 tmp = zsc(zadd(zadd(zmul(k[0], v[0]), zmul(k[1], v[1])), zmul(k[2], v[2])), 1.0 / k2);
            double f = 4.0 * a.p0 / (k2 + a.p1);
            for (int c = 0; c < 3; c++) v[c] = zsc(zsub(v[c], zmul(zcj(k[c]), tmp)), f);
        } else {
            v[0] = v[1] = v[2] = make_double2(0.0, 0.0);
        }
    } else {
        // projectFTscalar: gevolution.hpp:251-340 (add = 0)
        double2 S[6] = {v[0], v[1], v[2], v[3], v[4], v[5]};
        double2 chi = make_double2(0.0, 0.0);
        if (k2 > 0.0) {
            chi = zadd(zadd(zsc(S[0], g[1] + g[2] - 2.0 * g[0]), zsc(S[3], g[0] + g[2] - 2.0 * g[1])), zsc(S[5], g[0] + g[1] - 2.0 * g[2]));
            chi = zsub(chi, zsc(zmul(zmul(k[0], k[1]), S[1]), 6.0));
            chi = zsub(chi, zsc(zmul(zmul(k[0], k[2]), S[2]), 6.0));
            chi = zsub(chi, zsc(zmul(zmul(k[1], k[2]), S[4]), 6.0));
            chi = zsc(chi, 1.0 / (2.0 * k2 * k2 * N));
        }
        if constexpr ((EXTRA & EXTRA_TENSOR_PROJECT) != 0) {
            // projectFTtensor: gevolution.hpp:693-787
            double2 o[6];
            if (k2 > 0.0) {
                tt_num(g, k, k2, S, o);
                double k6 = k2 * k2 * k2 * N;
                for (int c = 0; c < 6; c++) a.hij[c * a.stride + kidx] = mk(R(o[c].x / k6), R(o[c].y / k6));
            } else {
                for (int c = 0; c < 6; c++) a.hij[c * a.stride + kidx] = mk(R(0), R(0));
            }
        }
        if constexpr ((EXTRA & EXTRA_TENSOR_EVOLVE) != 0) {
            // evolveFTtensor: gevolution.hpp:537-674; p0 = hubble, p1 = dtau, p2 = dtau_old
            const double dm = 0.5 * (a.p2 + a.p1), opd = 1.0 + a.p0 * dm, omd = 1.0 - a.p0 * dm;
            const double k4 = k2 * k2 * N;
            double2 h[6], hp[6], o[6];
            for (int c = 0; c < 6; c++) { h[c] = z2d(a.hij[c * a.stride + kidx]); hp[c] = z2d(a.hijp[c * a.stride + kidx]); }
            if (k2 * dm * dm < 1.0) {
                for (int c = 0; c < 6; c++) h[c] = zadd(h[c], zsc(hp[c], a.p2));
                if (k2 > 0.0) {
                    tt_num(g, k, k2, S, o);
                    for (int c = 0; c < 6; c++) hp[c] = zsc(zadd(zsc(hp[c], omd), zsc(zsub(zsc(o[c], 1.0 / k4), zsc(h[c], k2)), dm)), 1.0 / opd);
                } else {
                    double2 tr = zadd(zadd(S[0], S[3]), S[5]);
                    double2 Sm[6] = {zsub(S[0], zsc(tr, 1.0 / 3.0)), S[1], S[2], zsub(S[3], zsc(tr, 1.0 / 3.0)), S[4], zsub(S[5], zsc(tr, 1.0 / 3.0))};
                    for (int c = 0; c < 6; c++) hp[c] = zsc(zadd(zsc(hp[c], omd), zsc(Sm[c], 2.0 * dm / N)), 1.0 / opd);
                }
            } else {
                tt_num(g, k, k2, S, o);
                for (int c = 0; c < 6; c++) {
                    hp[c] = make_double2(0.0, 0.0);
                    h[c] = zsc(zadd(zsc(o[c], a.p2 / k4), zsc(h[c], 2.0 * a.p0)), 1.0 / (k2 * a.p2 + 2.0 * a.p0));
                }
            }
            for (int c = 0; c < 6; c++) {
                a.hij[c * a.stride + kidx] = mk(R(h[c].x), R(h[c].y));
                a.hijp[c * a.stride + kidx] = mk(R(hp[c].x), R(hp[c].y));
            }
        }
        if constexpr ((EXTRA & EXTRA_VECTOR_EVOLVE) != 0) {
            // evolveFTvector: gevolution.hpp:359-429; p3 = a^2 dtau
            double2 B[3];
            for (int c = 0; c < 3; c++) B[c] = z2d(a.bstate[c * a.stride + kidx]);
            double k4 = k2 * k2;
            if (k4 > 0.0) {
                double2 fac = make_double2(0.0, -2.0 * a.p3 / k4);
                B[0] = zadd(B[0], zmul(fac, zadd(zmul(zcj(k[0]), zsub(zsub(zsub(zsc(S[0], g[1] + g[2]), zsc(S[3], g[1])), zsc(S[5], g[2])), zsc(zmul(zmul(k[1], k[2]), S[4]), 2.0))),
                                                 zsc(zadd(zmul(k[1], S[1]), zmul(k[2], S[2])), g[1] + g[2] - g[0]))));
                B[1] = zadd(B[1], zmul(fac, zadd(zmul(zcj(k[1]), zsub(zsub(zsub(zsc(S[3], g[0] + g[2]), zsc(S[0], g[0])), zsc(S[5], g[2])), zsc(zmul(zmul(k[0], k[2]), S[2]), 2.0))),
                                                 zsc(zadd(zmul(k[0], S[1]), zmul(k[2], S[4])), g[0] + g[2] - g[1]))));
                B[2] = zadd(B[2], zmul(fac, zadd(zmul(zcj(k[2]), zsub(zsub(zsub(zsc(S[5], g[0] + g[1]), zsc(S[0], g[0])), zsc(S[3], g[1])), zsc(zmul(zmul(k[0], k[1]), S[1]), 2.0))),
                                                 zsc(zadd(zmul(k[0], S[2]), zmul(k[1], S[4])), g[0] + g[1] - g[2]))));
            } else {
                B[0] = B[1] = B[2] = make_double2(0.0, 0.0);
            }
            for (int c = 0; c < 3; c++) {
                a.bstate[c * a.stride + kidx] = mk(R(B[c].x), R(B[c].y));
                v[1 + c] = B[c];
            }
        }
        v[0] = chi;
    }
}

// OP_POISSON: the forward x pass's partial sums, by one block at the end of
// its own work
template <class R, int NT> __device__ __forceinline__ void sum_partials(const FzArgs<R> &a)
{
    if (a.partial && blockIdx.x == 0 && blockIdx.y == 0) {
        double v = 0.0;
        for (int64_t i = threadIdx.x; i < a.npartial; i += NT) v += a.partial[i];
        block_sum<NT>(v, a.sum);
    }
}

// OP_BIN: extractCrossSpectrum's binning (tools.hpp:105-215; KTYPE_LINEAR, CIC
// deconvolution; p0 = numbins, p1 = kmax) of the modes (kx, ky, kz) and
// (kx, ky, N - kz), which share their |k|: one warp, lanes at consecutive kz,
// v0 and v1 the two values (v1 ignored unless `two`).  Along the lanes the
// bin does not decrease, so lanes of one bin are neighbours: each run of them
// is summed by shuffles and only its first lane adds to the bins.  Five
// global additions per mode on a few hundred addresses take 1450 us at 256^3
// (FP64); this takes a few of them per warp, spread over bin_copies copies.
template <class R>
__device__ __forceinline__ void bin_modes(const FzArgs<R> &a, int N, int kx, int ky, int kz, bool on, bool two,
                                          typename CT<R>::C v0, typename CT<R>::C v1, int copy)
{
    const int lane = threadIdx.x & 31, nb = (int)a.p0;
    double s4[4] = {0.0, 0.0, 0.0, 0.0};
    unsigned int cnt = 0;
    int bin = nb;
    if (on && !(kx == 0 && ky == 0 && kz == 0)) {
        // k^2 and the bin index with separately rounded operations (no fused
        // multiply-add), as the reference evaluates them on the host: modes on a
        // bin edge (|n|^2 = 3 m^2 for the default kmax) land in the same bin
        auto lin = [&](int i) {
            const double t = __dmul_rn(2.0 * 3.14159265358979323846, (double)(i <= N / 2 ? i : N - i));
            return __dmul_rn(t, t);
        };
        const double kk2 = __dadd_rn(__dadd_rn(lin(kx), lin(ky)), lin(kz)), sk = sqrt(kk2);
        const double q = floor(__ddiv_rn(__dmul_rn((double)nb, sk), a.p1));
        if (q < (double)nb) {
            bin = (int)q;
            const int weight = (kx == 0 || (kx == N / 2 && (N % 2) == 0)) ? 1 : 2;
            double s = __ldg(a.tab + kx) * __ldg(a.tab + (ky <= N / 2 ? ky : N - ky)) * __ldg(a.tab + kz);
            s *= s;
            const double p0 = (double)v0.x * v0.x + (double)v0.y * v0.y, p1 = two ? (double)v1.x * v1.x + (double)v1.y * v1.y : 0.0;
            const double wt = two ? 2.0 * weight : (double)weight, f = kk2 * sk / s;
            cnt = two ? 2 * weight : weight;
            s4[0] = wt * sk;
            s4[1] = wt * kk2;
            s4[2] = weight * ((p0 + p1) * f);
            s4[3] = weight * ((p0 * p0 + p1 * p1) * f * f);
        }
    }
    const int prev = __shfl_up_sync(0xffffffffu, bin, 1);
    for (int o = 1; o < 32; o <<= 1) {
        const bool same = __shfl_down_sync(0xffffffffu, bin, o) == bin && lane + o < 32;
        if (!__any_sync(0xffffffffu, same)) break;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const double d = __shfl_down_sync(0xffffffffu, s4[i], o);
            if (same) s4[i] += d;
        }
        const unsigned int d = __shfl_down_sync(0xffffffffu, cnt, o);
        if (same) cnt += d;
    }
    if (bin < nb && (lane == 0 || prev != bin)) {
        double *b = a.bins + (size_t)copy * 4 * nb + bin;
#pragma unroll
        for (int i = 0; i < 4; i++) atomicAdd(b + i * nb, s4[i]);
        atomicAdd(a.occ + (size_t)copy * nb + bin, (unsigned long long)cnt);
    }
}

// z pass: grid (ceil(P/T), N), G * R2 * T threads; T kx-columns at one ky over
// all kz, every component of the solve: forward transform, pointwise solver,
// inverse transform in one kernel (two-step register FFT, fftreg.cuh), G
// thread groups sharing the components.
//
//   1. step 1 of every component, from global memory: one component (and the
//      contracted scalar sources) through registers, several by asynchronous
//      copies into the exchange buffers;
//   2. per row q (the modes kz = q + R1 p): step 2, the solver and the
//      inverse's step over p.  With one component the row stays in its
//      thread's registers; several components wait in their rows, where all
//      threads solve the modes;
//   3. the inverse's last step, straight to global memory.
//
// projectFTscalar (gevolution.hpp:251-340) without tensor or vector extras:
//   chi 2 k^4 N = S00 (g1+g2-2g0) + S11 (g0+g2-2g1) + S22 (g0+g1-2g2)
//                 - 6 (k0 k1 S01 + k0 k2 S02 + k1 k2 S12)
//               = A + g2 B - 6 k2 C, with
//   A = S00 (g1-2g0) + S11 (g0-2g1) + S22 (g0+g1) - 6 k0 k1 S01,
//   B = S00 + S11 - 2 S22,   C = k0 S02 + k1 S12.
// A, B, C have coefficients that depend on kx, ky only, so they are formed
// (in FP64) while the pencils load and the z transform -- linear, along kz --
// acts on three columns instead of six.
template <class R, int N, int T, int G, int OP, int EXTRA, int MINB>
__global__ void __launch_bounds__(RegPlan<N>::R2 *T *G, MINB) k_fz(FzArgs<R> a, const typename CT<R>::C *__restrict__ tw)
{
    constexpr bool EARLY = (uint64_t)((N / 2 + 1 + T - 1) / T) * N <= PDL_BLOCKS;   // the launch's grid
    pdl_entry<EARLY>();
    constexpr bool EX = OP != OP_VECTOR;   // fftreg.cuh
    using C = typename CT<R>::C;
    constexpr int P = N / 2 + 1, PP = N / 2 + 2;
    constexpr int R1 = RegPlan<N>::R1, R2 = RegPlan<N>::R2;
    constexpr int CIN = OpShape<OP, EXTRA>::CIN, COUT = OpShape<OP, EXTRA>::COUT;
    constexpr bool CONTRACT = OpShape<OP, EXTRA>::CONTRACT;
    constexpr int CT1 = CONTRACT ? 3 : CIN;   // columns transformed forward
    constexpr int ES = exch_size<N, T>();
    static_assert(CT1 > 1 || G == 1, "one component is one group's work");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *smem = reinterpret_cast<C *>(smem_raw);
    const int t = threadIdx.x % T, u = (threadIdx.x / T) % R2, g = threadIdx.x / (T * R2);
    const int kx = blockIdx.x * T + t, ky = blockIdx.y;
    const bool live = kx < P;
    C *buf = smem + t;   // this line's exchange buffers
    const int64_t col = (int64_t)(live ? kx : 0) + (int64_t)PP * ky;
    constexpr int64_t PLANE = (int64_t)PP * N;
    // slot of mode n of line t2
    auto slot = [](int n, int t2) { return ((n % R1) * (R2 + 1) + n / R1) * T + t2; };

    // 1. forward step 1
    if constexpr (CT1 > 1) {
        // row z = j + R2 r goes where step 1 of thread j reads it
        if constexpr (CONTRACT) {
            const double g0 = __ldg(a.k2 + (live ? kx : 0)), g1 = __ldg(a.k2 + ky);
            const double2 k0 = __ldg(a.ks + (live ? kx : 0)), k1 = __ldg(a.ks + ky), k01 = zmul(k0, k1);
#pragma unroll 2
            for (int r = g; r < R1; r += G) {
                const C *s = a.data + col + PLANE * (u + R2 * r);
                C x[6];
#pragma unroll
                for (int c = 0; c < 6; c++) x[c] = live ? __ldcs(s + c * a.stride) : mk(R(0), R(0));
                const double2 S0 = z2d(x[0]), S1 = z2d(x[1]), S2 = z2d(x[2]), S3 = z2d(x[3]), S4 = z2d(x[4]), S5 = z2d(x[5]);
                const double2 A = zsub(zadd(zadd(zsc(S0, g1 - 2.0 * g0), zsc(S3, g0 - 2.0 * g1)), zsc(S5, g0 + g1)),
                                       zsc(zmul(k01, S1), 6.0));
                const double2 B = zsub(zadd(S0, S3), zsc(S5, 2.0));
                const double2 Cc = zadd(zmul(k0, S2), zmul(k1, S4));
                C *o = buf + (r * (R2 + 1) + u) * T;
                o[0] = mk(R(A.x), R(A.y));
                o[ES] = mk(R(B.x), R(B.y));
                o[2 * ES] = mk(R(Cc.x), R(Cc.y));
            }
            if constexpr (G > 1) __syncthreads();
        } else {
            // every component in flight at once, no registers held
#pragma unroll 1
            for (int c = g; c < CIN; c += G) {
                const C *s = a.data + c * a.stride + col;
#pragma unroll
                for (int r = 0; r < R1; r++) copy_async(buf + c * ES + (r * (R2 + 1) + u) * T, s + PLANE * (u + R2 * r), live);
            }
            copy_async_commit();
            copy_async_wait<0>();
        }
#pragma unroll 1
        for (int c = g; c < CT1; c += G) {
            C v[R1];
#pragma unroll
            for (int r = 0; r < R1; r++) v[r] = buf[c * ES + (r * (R2 + 1) + u) * T];
            step1_store<N, -1, EX, T>(v, buf + c * ES, u, tw);
        }
    } else {
        C v[R1];
#pragma unroll
        for (int r = 0; r < R1; r++) v[r] = live ? __ldcs(a.data + col + PLANE * (u + R2 * r)) : mk(R(0), R(0));
        step1_store<N, -1, EX, T>(v, buf, u, tw);
    }
    __syncthreads();

    // 2. step 2, solver, inverse step 2
    if constexpr (OP == OP_BIN) {
        for (int q = u; q < R1; q += R2) {
            C v[R2];
            step2_load<N, -1, EX, T>(v, buf, q);
#pragma unroll
            for (int p = 0; p < R2; p++) buf[(q * (R2 + 1) + p) * T] = v[p];
        }
        __syncthreads();
        constexpr int NW = R2 * T / 32 > 0 ? R2 * T / 32 : 1;
        static_assert(R2 * T % 32 == 0, "whole warps bin the modes");
        for (int l = threadIdx.x / 32; l < T; l += NW) {
            const int kxl = blockIdx.x * T + l;
            for (int z0 = 0; z0 <= N / 2; z0 += 32) {
                const int z = z0 + (threadIdx.x & 31);
                const bool on = kxl < P && z <= N / 2, two = z > 0 && z < N / 2;
                const C v0 = on ? smem[slot(z, l)] : mk(R(0), R(0)), v1 = on && two ? smem[slot(N - z, l)] : mk(R(0), R(0));
                bin_modes(a, N, kxl, ky, z, on, two, v0, v1, (int)((blockIdx.x + gridDim.x * blockIdx.y) % bin_copies((int)a.p0)));
            }
        }
    } else if constexpr (CT1 == 1) {
        for (int q = u; q < R1; q += R2) {
            C v[R2];
            step2_load<N, -1, EX, T>(v, buf, q);
            if (live) {
#pragma unroll
                for (int p = 0; p < R2; p++) {
                    double2 w[COUT > 1 ? COUT : 1];
                    w[0] = z2d(v[p]);
                    const int n = q + R1 * p;
                    fz_apply<R, OP, EXTRA>(a, N, kx, ky, n, (int64_t)kx + PP * ((int64_t)ky + (int64_t)N * n), w);
                    if constexpr (COUT > 0) v[p] = mk(R(w[0].x), R(w[0].y));
#pragma unroll
                    for (int c = 1; c < COUT; c++)   // OP_ZELD: one column in, three out
                        buf[c * ES + (q * (R2 + 1) + p) * T] = mk(R(w[c].x), R(w[c].y));
                }
            }
            if constexpr (COUT > 0) step2_store<N, 1, EX, T>(v, buf, q, tw);
#pragma unroll 1
            for (int c = 1; c < COUT; c++) {
#pragma unroll
                for (int p = 0; p < R2; p++) v[p] = buf[c * ES + (q * (R2 + 1) + p) * T];
                step2_store<N, 1, EX, T>(v, buf + c * ES, q, tw);
            }
        }
    } else {
#pragma unroll 1
        for (int w = u + R2 * g; w < CT1 * R1; w += R2 * G) {
            C *row = buf + (w / R1) * ES;
            C v[R2];
            step2_load<N, -1, EX, T>(v, row, w % R1);
#pragma unroll
            for (int p = 0; p < R2; p++) row[((w % R1) * (R2 + 1) + p) * T] = v[p];
        }
        __syncthreads();
        if (live) {
            // threads of one line keep its kx: their kx and ky tables load once
#pragma unroll 1
            for (int n = u + R2 * g; n < N; n += R2 * G) {
                const int o = slot(n, 0);
                if constexpr (CONTRACT) {
                    const double g0 = __ldg(a.k2 + kx), g1 = __ldg(a.k2 + ky), g2 = __ldg(a.k2 + n);
                    const double2 k2c = __ldg(a.ks + n);
                    const double k2 = g0 + g1 + g2;
                    double2 chi = make_double2(0.0, 0.0);
                    if (k2 > 0.0) {
                        const double2 A = z2d(buf[o]), B = z2d(buf[ES + o]), Cc = z2d(buf[2 * ES + o]);
                        chi = zsub(zadd(A, zsc(B, g2)), zsc(zmul(k2c, Cc), 6.0));
                        chi = zsc(chi, 1.0 / (2.0 * k2 * k2 * N));
                    }
                    buf[o] = mk(R(chi.x), R(chi.y));
                } else {
                    double2 v[6];
#pragma unroll
                    for (int c = 0; c < CIN; c++) v[c] = z2d(buf[c * ES + o]);
                    fz_apply<R, OP, EXTRA>(a, N, kx, ky, n, (int64_t)kx + PP * ((int64_t)ky + (int64_t)N * n), v);
#pragma unroll
                    for (int c = 0; c < COUT; c++) buf[c * ES + o] = mk(R(v[c].x), R(v[c].y));
                }
            }
        }
        __syncthreads();
#pragma unroll 1
        for (int w = u + R2 * g; w < COUT * R1; w += R2 * G) {
            C *row = buf + (w / R1) * ES;
            C v[R2];
#pragma unroll
            for (int p = 0; p < R2; p++) v[p] = row[((w % R1) * (R2 + 1) + p) * T];
            step2_store<N, 1, EX, T>(v, row, w % R1, tw);
        }
    }
    if constexpr (COUT > 0) {
        __syncthreads();
        // 3. the inverse's last step
#pragma unroll 1
        for (int c = g; c < COUT; c += G) {
            C v[R1];
            step1_load<N, 1, EX, T>(v, buf + c * ES, u);
            if (live) {
#pragma unroll
                for (int r = 0; r < R1; r++) a.data[c * a.stride + col + PLANE * (u + R2 * r)] = v[r];
            }
        }
    }
    if constexpr (OP == OP_POISSON) sum_partials<R, R2 * T>(a);
}

// z pass with tensor-memory-access staging: one elected thread loads the
// CTA's T kx-columns of every input component over all kz as bulk tensor
// copies (boxes of at most 256 kz) into dense per-component shared buffers,
// the CTA transforms, solves and inverse-transforms them, and the results
// leave by bulk tensor stores.  Columns kx >= P of the last CTA are zero-filled
// on load and clipped on store.  Same arithmetic as k_fz, with block-wide
// Stockham passes (fft.cuh).  Taken (z_staged) where it is the faster of the
// two, which is where the two-step form holds too many registers for the
// warps that would hide its latency; us here / by k_fz:
//   FP32 contracted scalar   256: 187 / 222      512: 1425 / 2100
//   FP32 vector              256: 202 / 180      384: 726 / 686     512: 1196 / 1731
//   FP32 Poisson             256: 72 / 60        384: 246 / 272     512: 455 / 556
//   FP32 displacement        128: 40 / 41        256: 239 / 336     512: 1594 / 3666
//   FP64 contracted scalar   256: 471 / 334      384: 1941 / 1452   512: 3811 / 6495   768: 20.8 / 15.6 ms
//   FP64 vector              384: 2329 / 1192    768: 25.1 / 13.7 ms
//   FP64 Poisson             256: 126 / 104      384: 397 / 482     512: 801 / 1120    768: 3.0 / 5.0 ms
//   FP64 displacement        128: 84 / 68        256: 452 / 537     384: 1747 / 3639   512: 3612 / 6962
// The scalar solve with h_ij or parabolic B_i and the binning are k_fz's.
template <int N> struct ZBox {
    static constexpr int ZB = N <= 256 ? N : (N % 256 == 0 ? 256 : 128);
    static constexpr int NZB = N / ZB;
};

// resident CTAs of 256 threads the staged z pass is compiled for.  FP64: three
// where a thread's share of the lines is larger than one butterfly (the
// Poisson pass at 512: 801 us with three, 1664 with four, which spill), four
// otherwise (the scalar pass at 512: 4434 us with three, 3811 with four).
template <class R, int N, int OP, int EXTRA> constexpr int fz_staged_minb()
{
    return sizeof(R) == 8 && (OpShape<OP, EXTRA>::CMAX == 1 || N > 512) ? 3 : 4;
}

// PAD: the transforms use padded rows (fft.cuh), each component buffer then
// holds N + N / 8 rows of T values
template <class R, int N, int T, int NT, int OP, int EXTRA, bool PAD, int MINB>
__global__ void __launch_bounds__(NT, MINB)
    k_fz_tma(FzArgs<R> a, const typename CT<R>::C *__restrict__ tw, const __grid_constant__ CUtensorMap tmap)
{
    pdl_entry<false>();
    using C = typename CT<R>::C;
    constexpr int P = N / 2 + 1, PP = N / 2 + 2;
    constexpr int CIN = OpShape<OP, EXTRA>::CIN, COUT = OpShape<OP, EXTRA>::COUT;
    constexpr bool CONTRACT = OpShape<OP, EXTRA>::CONTRACT;
    constexpr int ZB = ZBox<N>::ZB, NZB = ZBox<N>::NZB;
    constexpr int CS = N * T;   // one component: [kz][t], dense
    constexpr int CSTR = PAD ? (N + N / 8) * T : CS;   // component buffer stride
    // bulk tensor copies want 128-byte aligned shared addresses: the launch
    // adds 128 bytes of slack and the buffers start at the next boundary
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *buf = reinterpret_cast<C *>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~(uintptr_t)127);
    __shared__ __align__(8) uint64_t bar;
    const int kx0 = blockIdx.x * T, ky = blockIdx.y;

    // the contracted scalar solve loads S00, S01, S11, S22 into buffers 0..3,
    // folds them into A and B (buffers 0, 1), then loads S02, S12 into
    // buffers 2, 3 and folds them into C (buffer 2): four buffers instead of six
    constexpr int NL1 = CONTRACT ? 4 : CIN;
    auto first_comp = [](int s) { return CONTRACT ? (s == 2 ? 3 : (s == 3 ? 5 : s)) : s; };
    auto load = [&](int slot, int comp) {
#pragma unroll 1
        for (int zc = 0; zc < NZB; zc++) tma_load_4d(buf + slot * CSTR + zc * ZB * T, &tmap, 2 * kx0, ky, zc * ZB, comp, &bar);
    };
    if (threadIdx.x == 0) mbar_init(&bar, 1);
    __syncthreads();
    if (threadIdx.x == 0) {
        mbar_expect_tx(&bar, (uint32_t)(NL1 * CS * sizeof(C)));
#pragma unroll 1
        for (int s = 0; s < NL1; s++) load(s, first_comp(s));
    }
    bool ok = mbar_wait(&bar, 0);
    if (__syncthreads_or(!ok)) {
        if (threadIdx.x == 0 && a.err) atomicOr(a.err, ERR_TMA_TIMEOUT);
        return;
    }

    if constexpr (CONTRACT) {
        // A, B, C of k_fz's projectFTscalar factorisation
        for (int idx = threadIdx.x; idx < CS; idx += NT) {
            const int t = idx % T, kx = kx0 + t;
            double2 A = make_double2(0.0, 0.0), B = A;
            if (kx < P) {
                const double2 S0 = z2d(buf[idx]), S1 = z2d(buf[CSTR + idx]);
                const double2 S3 = z2d(buf[2 * CSTR + idx]), S5 = z2d(buf[3 * CSTR + idx]);
                const double g0 = __ldg(a.k2 + kx), g1 = __ldg(a.k2 + ky);
                const double2 k0 = __ldg(a.ks + kx), k1 = __ldg(a.ks + ky);
                A = zsub(zadd(zadd(zsc(S0, g1 - 2.0 * g0), zsc(S3, g0 - 2.0 * g1)), zsc(S5, g0 + g1)),
                         zsc(zmul(zmul(k0, k1), S1), 6.0));
                B = zsub(zadd(S0, S3), zsc(S5, 2.0));
            }
            buf[idx] = mk(R(A.x), R(A.y));
            buf[CSTR + idx] = mk(R(B.x), R(B.y));
        }
        __syncthreads();   // buffers 2 and 3 are free
        if (threadIdx.x == 0) {
            fence_async_smem();
            mbar_expect_tx(&bar, (uint32_t)(2 * CS * sizeof(C)));
            load(2, 2);
            load(3, 4);
        }
        ok = mbar_wait(&bar, 1);
        if (__syncthreads_or(!ok)) {
            if (threadIdx.x == 0 && a.err) atomicOr(a.err, ERR_TMA_TIMEOUT);
            return;
        }
        for (int idx = threadIdx.x; idx < CS; idx += NT) {
            const int t = idx % T, kx = kx0 + t;
            double2 Cc = make_double2(0.0, 0.0);
            if (kx < P) {
                const double2 S2 = z2d(buf[2 * CSTR + idx]), S4 = z2d(buf[3 * CSTR + idx]);
                const double2 k0 = __ldg(a.ks + kx), k1 = __ldg(a.ks + ky);
                Cc = zadd(zmul(k0, S2), zmul(k1, S4));
            }
            buf[2 * CSTR + idx] = mk(R(Cc.x), R(Cc.y));
        }
        __syncthreads();
    }
#pragma unroll 1
    for (int c = 0; c < (CONTRACT ? 3 : CIN); c++) fft_lines<N, -1, T, NT, PAD>(buf + c * CSTR, T, tw);

    for (int idx = threadIdx.x; idx < CS; idx += NT) {
        const int t = idx % T, n = idx / T, kx = kx0 + t;
        if (kx >= P) continue;
        if constexpr (CONTRACT) {
            const double g0 = __ldg(a.k2 + kx), g1 = __ldg(a.k2 + ky), g2 = __ldg(a.k2 + n);
            const double2 k2c = __ldg(a.ks + n);
            const double k2 = g0 + g1 + g2;
            double2 chi = make_double2(0.0, 0.0);
            if (k2 > 0.0) {
                const double2 A = z2d(buf[idx]), B = z2d(buf[CSTR + idx]), Cc = z2d(buf[2 * CSTR + idx]);
                chi = zsub(zadd(A, zsc(B, g2)), zsc(zmul(k2c, Cc), 6.0));
                chi = zsc(chi, 1.0 / (2.0 * k2 * k2 * N));
            }
            buf[idx] = mk(R(chi.x), R(chi.y));
        } else {
            double2 v[6];
#pragma unroll
            for (int c = 0; c < CIN; c++) v[c] = z2d(buf[c * CSTR + idx]);
            const int64_t kidx = kx + (int64_t)PP * (ky + (int64_t)N * n);
            fz_apply<R, OP, EXTRA>(a, N, kx, ky, n, kidx, v);
#pragma unroll
            for (int c = 0; c < COUT; c++) buf[c * CSTR + idx] = mk(R(v[c].x), R(v[c].y));
        }
    }
    if constexpr (COUT > 0) {
        __syncthreads();
#pragma unroll 1
        for (int c = 0; c < COUT; c++) fft_lines<N, 1, T, NT, PAD>(buf + c * CSTR, T, tw);
        fence_async_smem();
        __syncthreads();
        if (threadIdx.x == 0) {
#pragma unroll 1
            for (int c = 0; c < COUT; c++)
#pragma unroll 1
                for (int zc = 0; zc < NZB; zc++) tma_store_4d(&tmap, 2 * kx0, ky, zc * ZB, c, buf + c * CSTR + zc * ZB * T);
            tma_store_drain();
        }
    }
    if constexpr (OP == OP_POISSON) sum_partials<R, NT>(a);
}

// y pass (in place): T kx-columns over all ky at one kz; grid (ceil(P/T), N, ncomp)
template <class R, int N, int T, int S, bool EX, int MINB>
__global__ void __launch_bounds__(RegPlan<N>::R2 *T, MINB) k_fy(typename CT<R>::C *data, int64_t stride,
                                                               const typename CT<R>::C *__restrict__ tw)
{
    pdl_entry<false>();
    using C = typename CT<R>::C;
    constexpr int P = N / 2 + 1, PP = N / 2 + 2, R1 = RegPlan<N>::R1, R2 = RegPlan<N>::R2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int t = threadIdx.x % T, u = threadIdx.x / T;
    const int kx = blockIdx.x * T + t;
    const bool live = kx < P;
    C *buf = reinterpret_cast<C *>(smem_raw) + t;
    C *d = data + (int64_t)blockIdx.z * stride + (live ? kx : 0) + (int64_t)PP * N * blockIdx.y;
    {
        C v[R1];
#pragma unroll
        for (int r = 0; r < R1; r++) v[r] = live ? d[PP * (u + R2 * r)] : mk(R(0), R(0));
        step1_store<N, S, EX, T>(v, buf, u, tw);
    }
    __syncthreads();
    for (int q = u; q < R1; q += R2) {
        C v[R2];
        step2_load<N, S, EX, T>(v, buf, q);
        if (live) {
#pragma unroll
            for (int p = 0; p < R2; p++) d[PP * (q + R1 * p)] = v[p];
        }
    }
}

// y pass with bulk-tensor-copy staging, the same grid and Stockham passes in
// shared memory: for the FP64 lines of 512, whose two-step form holds 32
// values per thread and two blocks of 128 threads per SM (six components
// forward 1517 us by k_fy, 1304 here; one back 734 and 661; with half or twice
// the columns k_fy takes 1480 and 1662).  Elsewhere k_fy is the faster one
// (FP64 256: 139 against 224 us, 384: 505 and 637, 768: 6.1 and 6.6 ms; FP32
// 512: 691 and 710 us).
constexpr int FY_STAGED_NT = 512;

template <class R, int N, int T, int S>
__global__ void __launch_bounds__(FY_STAGED_NT, 2) k_fy_tma(const typename CT<R>::C *__restrict__ tw, int *err,
                                                            const __grid_constant__ CUtensorMap tmap)
{
    pdl_entry<false>();
    using C = typename CT<R>::C;
    constexpr int YB = ZBox<N>::ZB, NYB = ZBox<N>::NZB;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *buf = reinterpret_cast<C *>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~(uintptr_t)127);
    __shared__ __align__(8) uint64_t bar;
    const int kx0 = blockIdx.x * T, z = blockIdx.y, comp = blockIdx.z;
    if (threadIdx.x == 0) mbar_init(&bar, 1);
    __syncthreads();
    if (threadIdx.x == 0) {
        mbar_expect_tx(&bar, (uint32_t)(N * T * sizeof(C)));
#pragma unroll 1
        for (int yc = 0; yc < NYB; yc++) tma_load_4d(buf + yc * YB * T, &tmap, 2 * kx0, yc * YB, z, comp, &bar);
    }
    const bool ok = mbar_wait(&bar, 0);
    if (__syncthreads_or(!ok)) {   // the data never arrived: leave the array untouched and say so
        if (threadIdx.x == 0 && err) atomicOr(err, ERR_TMA_TIMEOUT);
        return;
    }
    fft_lines<N, S, T, FY_STAGED_NT>(buf, T, tw);
    fence_async_smem();
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll 1
        for (int yc = 0; yc < NYB; yc++) tma_store_4d(&tmap, 2 * kx0, yc * YB, z, comp, buf + yc * YB * T);
        tma_store_drain();
    }
}

}  // namespace gev
