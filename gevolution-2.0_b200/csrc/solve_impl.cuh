// solve_impl.cuh -- launchers of the pencil passes for every supported grid
// size; included once per precision (solve_f32.cu, solve_f64.cu).
#pragma once

#include <algorithm>
#include <stdexcept>
#include <string>

#include "fftpass.cuh"
#include "kernels.h"

namespace gev {

// Lines (x passes) or kx-columns (y, z passes) per CTA, and the registers per
// thread (FP32; twice that in FP64) that set the resident CTAs, from sweeps at
// 128^3 to 512^3 (FP32) and 256^3 (FP64).
constexpr int PASS_TX = 8, PASS_TY = 16, PASS_TZ1 = 8, PASS_TIJ = 4, PASS_TIJ_G = 4, PASS_GZ = 3;
constexpr int REGS_X = 72, REGS_Y = 96;
template <class R> constexpr int REGS_TIJ = sizeof(R) == 4 ? 72 : 96;
template <class R> constexpr int REGS_Z1 = sizeof(R) == 4 ? 72 : 96;
// The tensor solve holds six components in FP64 and moves 24 values of tensor
// state per mode: eight columns make its rows 64-byte segments.  Chi solves
// with parabolic B_i and h_ij, eight against four columns (FP64: four against
// two): 256^3 1523 and 1696 us, FP64 2655 and 2780; 384^3 5.20 and 6.68 ms;
// 512^3 12.5 and 15.7 ms.  At 768 the six lines of eight columns (307,200
// bytes) are beyond a block's shared memory: four columns, 58.6 ms.
template <int N> constexpr int PASS_TZ6 = N <= 512 ? 8 : 4;
constexpr int REGS_Z6 = 168;
// three components: eight columns while a thread's values leave the registers
// for it (256^3: 180 against 191 us with four), four columns beyond
template <int N> constexpr int PASS_TZ3 = N <= 256 ? 8 : 4;
template <int N> constexpr int REGS_Z3 = N <= 256 ? 80 : 64;

// resident CTAs of nt threads with a budget of `regs` 32-bit registers per thread
// (FP64 values take twice the registers)
template <class R> constexpr int resident(int nt, int regs)
{
    const int r = regs * (sizeof(R) == 8 ? 2 : 1), lim = r > 248 ? 248 : r;
    const int b = 65536 / (lim * nt);
    return b < 1 ? 1 : (b > 32 ? 32 : b);
}

// dynamic shared memory that every block here may ask for: the 227 KB of a
// block less 1 KB for the kernels' static arrays
constexpr size_t BLOCK_SMEM = 226 * 1024;

template <size_t BYTES, class K> inline void set_smem(K kernel)
{
    static_assert(BYTES <= BLOCK_SMEM, "more shared memory than a block may have");
    if (BYTES <= 48 * 1024) return;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BYTES);
    if (e != cudaSuccess) {
        cudaGetLastError();
        throw std::runtime_error(std::string("shared memory limit: ") + cudaGetErrorString(e));
    }
}

#define GEV_SWITCH_N(N, CALL)                          \
    switch (N) {                                       \
    case 16: { constexpr int NN = 16; CALL; } break;   \
    case 32: { constexpr int NN = 32; CALL; } break;   \
    case 64: { constexpr int NN = 64; CALL; } break;   \
    case 128: { constexpr int NN = 128; CALL; } break; \
    case 256: { constexpr int NN = 256; CALL; } break; \
    case 384: { constexpr int NN = 384; CALL; } break; \
    case 512: { constexpr int NN = 512; CALL; } break; \
    case 768: { constexpr int NN = 768; CALL; } break; \
    default: throw std::runtime_error("unsupported grid size"); \
    }

template <class R> constexpr int cols(int t) { return sizeof(R) == 8 ? t / 2 : t; }
template <class R, int L> constexpr int regs_for(int regs) { return RegPlan<L>::R1 >= 24 ? regs + 32 : regs; }
// forward x passes.  The T00 source in FP32 waits for its seven loads per pair
// and wants warps more than registers (768^3: 3.58 ms with 104, 3.06 with 80)
template <class R, int N, int MODE> constexpr int regs_fx()
{
    return MODE == FX_PREP_T00 && sizeof(R) == 4 && RegPlan<N / 2>::R1 >= 24 ? 80 : regs_for<R, N / 2>(REGS_X);
}

template <class R, int N, int MODE, bool EX>
void fx_fwd_n(const FxArgs<R> &a, int ncomp, int64_t in_stride, int64_t out_stride, const FftTables<R> &tb, cudaStream_t st)
{
    using C = typename CT<R>::C;
    constexpr int T = PASS_TX, NT = RegPlan<N / 2>::R2 * T;
    static_assert((uint64_t)N * (N / T) > PDL_BLOCKS, "compiled for launches that are not early");
    constexpr size_t smem = (size_t)T * exch_size<N / 2, 1>() * sizeof(C);
    auto k = k_fx_fwd<R, N, T, MODE, EX, resident<R>(NT, regs_fx<R, N, MODE>())>;
    set_smem<smem>(k);
    pdl_launch(k, dim3(N / T, N, ncomp), NT, smem, st, a, in_stride, out_stride, tb.tw_half, tb.tw_full);
}

template <class R, int N>
void fx_tij6_n(const FxArgs<R> &a, int64_t in_stride, int64_t out_stride, const FftTables<R> &tb, cudaStream_t st)
{
    using C = typename CT<R>::C;
    static_assert((uint64_t)N * (N / PASS_TIJ) > PDL_BLOCKS, "compiled for launches that are not early");
    constexpr int T = cols<R>(PASS_TIJ), G = PASS_TIJ_G, NT = RegPlan<N / 2>::R2 * T * G;
    constexpr size_t smem = (size_t)6 * T * exch_size<N / 2, 1>() * sizeof(C);
    auto k = k_fx_fwd_tij6<R, N, T, G, resident<R>(NT, regs_for<R, N / 2>(REGS_TIJ<R>))>;
    set_smem<smem>(k);
    pdl_launch(k, dim3(N / T, N), NT, smem, st, a.in, in_stride, a.phi, a.c, a.out, out_stride, tb.tw_half, tb.tw_full);
}

template <class R, int N, int MODE, bool EX>
void plane_fwd_n(const FxArgs<R> &a, int ncomp, int64_t in_stride, int64_t out_stride, const FftTables<R> &tb, cudaStream_t st)
{
    using C = typename CT<R>::C;
    constexpr size_t smem = (size_t)PlaneShape<N>::VALUES * sizeof(C);
    auto k = k_plane_fwd<R, N, MODE, EX>;
    set_smem<smem>(k);
    pdl_launch(k, dim3(N, ncomp), PlaneShape<N>::NT, smem, st, a, in_stride, out_stride, tb.tw_half, tb.tw_full);
}

// y pass staged by bulk copies (k_fy_tma) or the two-step one (k_fy)
template <class R, int N> constexpr bool y_staged() { return sizeof(R) == 8 && N == 512; }

template <class R, int N, int S, bool EX>
void fy_n(typename CT<R>::C *data, int64_t stride, int ncomp, const FftTables<R> &tb, cudaStream_t st)
{
    using C = typename CT<R>::C;
    constexpr int T = cols<R>(PASS_TY);
    static_assert((uint64_t)N * (N / 2 / T) > PDL_BLOCKS, "compiled for launches that are not early");
    const dim3 grid((N / 2 + 1 + T - 1) / T, N, ncomp);
    if constexpr (y_staged<R, N>()) {
        constexpr size_t smem = (size_t)N * T * sizeof(C) + 128;
        const CUtensorMap map = fourier_tensor_map<R>(data, N, stride, ncomp, T, ZBox<N>::ZB, 1);
        auto k = k_fy_tma<R, N, T, S>;
        set_smem<smem>(k);
        pdl_launch(k, grid, FY_STAGED_NT, smem, st, tb.tw_full, tb.err, map);
    } else {
        constexpr int NT = RegPlan<N>::R2 * T;
        constexpr size_t smem = (size_t)exch_size<N, T>() * sizeof(C);
        auto k = k_fy<R, N, T, S, EX, resident<R>(NT, regs_for<R, N>(REGS_Y))>;
        set_smem<smem>(k);
        pdl_launch(k, grid, NT, smem, st, data, stride, tb.tw_full);
    }
}

template <class R, int N, int MODE, bool EX>
int fxy_fwd_ex(const FxArgs<R> &a, int ncomp, int64_t in_stride, int64_t out_stride, const FftTables<R> &tb, cudaStream_t st)
{
    if constexpr (plane_pass<N>()) {
        plane_fwd_n<R, N, MODE, EX>(a, ncomp, in_stride, out_stride, tb, st);
        return 1;
    } else {
        if constexpr (MODE == FX_PREP_TIJ) fx_tij6_n<R, N>(a, in_stride, out_stride, tb, st);
        else fx_fwd_n<R, N, MODE, EX>(a, ncomp, in_stride, out_stride, tb, st);
        fy_n<R, N, -1, EX>(a.out, out_stride, ncomp, tb, st);
        return 2;
    }
}

// three components are a vector field: no exact roots (fftreg.cuh)
template <class R, int N, int MODE>
int fxy_fwd_n(const FxArgs<R> &a, int ncomp, int64_t in_stride, int64_t out_stride, const FftTables<R> &tb, cudaStream_t st)
{
    if constexpr (MODE == FX_PREP_T0I) return fxy_fwd_ex<R, N, MODE, false>(a, ncomp, in_stride, out_stride, tb, st);
    else if constexpr (MODE != FX_COPY || sizeof(R) == 8) return fxy_fwd_ex<R, N, MODE, true>(a, ncomp, in_stride, out_stride, tb, st);
    else if (ncomp == 3) return fxy_fwd_ex<R, N, MODE, false>(a, ncomp, in_stride, out_stride, tb, st);
    else return fxy_fwd_ex<R, N, MODE, true>(a, ncomp, in_stride, out_stride, tb, st);
}

template <class R>
int fxy_forward(int N, int mode, const R *in, int64_t in_stride, int ncomp, const R *phi, const R *chi, double bg, double c,
                double c2, double c3, typename CT<R>::C *out, int64_t out_stride, double *partial, const FftTables<R> &tb,
                cudaStream_t st, bool clear)
{
    FxArgs<R> a;
    a.in = in; a.phi = phi; a.chi = chi;
    a.bg = bg; a.c = c; a.c2 = c2; a.c3 = c3;
    a.out = out; a.partial = partial; a.clear = clear;
    if (mode == FX_PREP_TIJ && ncomp != 6) throw std::runtime_error("the Tij sources are prepared together");
    int n = 0;
    if (mode == FX_COPY) { GEV_SWITCH_N(N, (n = fxy_fwd_n<R, NN, FX_COPY>(a, ncomp, in_stride, out_stride, tb, st))) }
    else if (mode == FX_PREP_T00) { GEV_SWITCH_N(N, (n = fxy_fwd_n<R, NN, FX_PREP_T00>(a, ncomp, in_stride, out_stride, tb, st))) }
    else if (mode == FX_PREP_T0I) { GEV_SWITCH_N(N, (n = fxy_fwd_n<R, NN, FX_PREP_T0I>(a, ncomp, in_stride, out_stride, tb, st))) }
    else { GEV_SWITCH_N(N, (n = fxy_fwd_n<R, NN, FX_PREP_TIJ>(a, ncomp, in_stride, out_stride, tb, st))) }
    return n;
}

template <class R, int N, bool EX>
void fxi_n(const typename CT<R>::C *in, int64_t in_stride, R *out, int64_t out_stride, int ncomp, const FftTables<R> &tb,
           cudaStream_t st)
{
    using C = typename CT<R>::C;
    constexpr int T = PASS_TX, NT = RegPlan<N / 2>::R2 * T;
    static_assert((uint64_t)N * (N / T) > PDL_BLOCKS, "compiled for launches that are not early");
    constexpr size_t smem = (size_t)T * exch_size<N / 2, 1>() * sizeof(C);
    auto k = k_fx_inv<R, N, T, EX, resident<R>(NT, regs_for<R, N / 2>(REGS_X))>;
    set_smem<smem>(k);
    pdl_launch(k, dim3(N / T, N, ncomp), NT, smem, st, in, in_stride, out, out_stride, tb.tw_half, tb.tw_full);
}

template <class R, int N, bool EX>
int fyx_inv_ex(typename CT<R>::C *in, int64_t in_stride, R *out, int64_t out_stride, int ncomp, const FftTables<R> &tb,
              cudaStream_t st)
{
    using C = typename CT<R>::C;
    if constexpr (plane_pass<N>()) {
        constexpr size_t smem = (size_t)PlaneShape<N>::VALUES * sizeof(C);
        auto k = k_plane_inv<R, N, EX>;
        set_smem<smem>(k);
        pdl_launch(k, dim3(N, ncomp), PlaneShape<N>::NT, smem, st, in, in_stride, out, out_stride, tb.tw_half, tb.tw_full);
        return 1;
    } else {
        fy_n<R, N, 1, EX>(in, in_stride, ncomp, tb, st);
        fxi_n<R, N, EX>(in, in_stride, out, out_stride, ncomp, tb, st);
        return 2;
    }
}

template <class R, int N>
int fyx_inv_n(typename CT<R>::C *in, int64_t in_stride, R *out, int64_t out_stride, int ncomp, const FftTables<R> &tb,
              cudaStream_t st)
{
    if constexpr (sizeof(R) == 4) {
        if (ncomp == 3) return fyx_inv_ex<R, N, false>(in, in_stride, out, out_stride, ncomp, tb, st);
    }
    return fyx_inv_ex<R, N, true>(in, in_stride, out, out_stride, ncomp, tb, st);
}

template <class R>
int fyx_inverse(int N, typename CT<R>::C *in, int64_t in_stride, R *out, int64_t out_stride, int ncomp, const FftTables<R> &tb,
                cudaStream_t st)
{
    int n = 0;
    GEV_SWITCH_N(N, (n = fyx_inv_n<R, NN>(in, in_stride, out, out_stride, ncomp, tb, st)))
    return n;
}

// CTAs of `bytes` dynamic shared memory that fit one SM (228 KB, 1 KB reserved per CTA)
constexpr int smem_ctas(size_t bytes) { return (int)(233472 / (bytes + 1024)); }

// z pass staged by bulk copies (k_fz_tma) or the two-step one (k_fz); the
// measured lines between them are in k_fz_tma's comment
template <class R, int N, int OP, int EXTRA> constexpr bool z_staged()
{
    using S = OpShape<OP, EXTRA>;
    if (OP == OP_BIN || (OP == OP_SCALAR && !S::CONTRACT)) return false;
    if (OP == OP_ZELD) return N >= 256;
    if (S::CMAX == 1) return N >= 384;
    if (sizeof(R) == 8) return N == 512 && S::CONTRACT;
    return N >= 512 || (N >= 256 && S::CONTRACT);
}

template <class R, int N, int OP, int EXTRA>
void fz_n(const FzArgs<R> &a, const FftTables<R> &tb, cudaStream_t st)
{
    using C = typename CT<R>::C;
    using S = OpShape<OP, EXTRA>;
    if constexpr (z_staged<R, N, OP, EXTRA>()) {
        static_assert((uint64_t)N * (N / 2 / 8) > PDL_BLOCKS, "compiled for launches that are not early");
        constexpr int T = S::CMAX == 1 ? cols<R>(8) : 4, NT = 256, MINB = fz_staged_minb<R, N, OP, EXTRA>();
        constexpr size_t dense = (size_t)S::CTMA * N * T * sizeof(C) + 128;
        constexpr size_t padded = (size_t)S::CTMA * (N + N / 8) * T * sizeof(C) + 128;
        // padded rows where they spread the banks, keep every component buffer on
        // a 128-byte boundary, and cost no resident CTA
        constexpr bool PAD = pad_helps<T, C>() && ((N + N / 8) * T * sizeof(C)) % 128 == 0 &&
                             smem_ctas(padded) >= std::min(MINB, smem_ctas(dense));
        constexpr size_t smem = PAD ? padded : dense;
        const CUtensorMap map = fourier_tensor_map<R>(a.data, N, a.stride, S::CMAX, T, 1, ZBox<N>::ZB);
        auto k = k_fz_tma<R, N, T, NT, OP, EXTRA, PAD, MINB>;
        set_smem<smem>(k);
        pdl_launch(k, dim3((N / 2 + 1 + T - 1) / T, N), NT, smem, st, a, tb.tw_full, map);
    } else {
        constexpr int CT1 = S::CONTRACT ? 3 : S::CIN, G = CT1 > 1 ? PASS_GZ : 1, R2 = RegPlan<N>::R2;
        constexpr int T0 = cols<R>(CT1 == 1 ? PASS_TZ1 : (CT1 == 3 ? PASS_TZ3<N> : PASS_TZ6<N>));
        constexpr int T = OP == OP_BIN && R2 * T0 < 32 ? 32 / R2 : T0, NT = R2 * T * G;   // OP_BIN works in whole warps
        constexpr size_t smem = (size_t)S::CBUF * exch_size<N, T>() * sizeof(C);
        constexpr int REGS = CT1 == 6 ? REGS_Z6 : (CT1 == 3 ? REGS_Z3<N> : REGS_Z1<R>);
        auto k = k_fz<R, N, T, G, OP, EXTRA, resident<R>(NT, regs_for<R, N>(REGS))>;
        set_smem<smem>(k);
        pdl_launch(k, dim3((N / 2 + 1 + T - 1) / T, N), NT, smem, st, a, tb.tw_full);
    }
}

template <class R, int N>
void fz_dispatch(const FzParams &fp, const FzArgs<R> &a, const FftTables<R> &tb, cudaStream_t st)
{
    if (fp.op == OP_POISSON) fz_n<R, N, OP_POISSON, 0>(a, tb, st);
    else if (fp.op == OP_ZELD) fz_n<R, N, OP_ZELD, 0>(a, tb, st);
    else if (fp.op == OP_ICS) fz_n<R, N, OP_ICS, 0>(a, tb, st);
    else if (fp.op == OP_BIN) fz_n<R, N, OP_BIN, 0>(a, tb, st);
    else if (fp.op == OP_VECTOR) fz_n<R, N, OP_VECTOR, 0>(a, tb, st);
    else {
        switch (fp.extra) {
        case 0: fz_n<R, N, OP_SCALAR, 0>(a, tb, st); break;
        case EXTRA_TENSOR_PROJECT: fz_n<R, N, OP_SCALAR, EXTRA_TENSOR_PROJECT>(a, tb, st); break;
        case EXTRA_TENSOR_EVOLVE: fz_n<R, N, OP_SCALAR, EXTRA_TENSOR_EVOLVE>(a, tb, st); break;
        case EXTRA_VECTOR_EVOLVE: fz_n<R, N, OP_SCALAR, EXTRA_VECTOR_EVOLVE>(a, tb, st); break;
        case EXTRA_TENSOR_PROJECT | EXTRA_VECTOR_EVOLVE: fz_n<R, N, OP_SCALAR, EXTRA_TENSOR_PROJECT | EXTRA_VECTOR_EVOLVE>(a, tb, st); break;
        case EXTRA_TENSOR_EVOLVE | EXTRA_VECTOR_EVOLVE: fz_n<R, N, OP_SCALAR, EXTRA_TENSOR_EVOLVE | EXTRA_VECTOR_EVOLVE>(a, tb, st); break;
        default: throw std::runtime_error("unsupported solver combination");
        }
    }
}

template <class R>
void fz_pass(int N, const FzParams &fp, typename CT<R>::C *data, int64_t stride, typename CT<R>::C *hij,
             typename CT<R>::C *hijp, typename CT<R>::C *bstate, const FftTables<R> &tb, cudaStream_t st)
{
    FzArgs<R> a;
    a.data = data; a.stride = stride;
    a.k2 = tb.k2; a.ks = tb.ks;
    a.p0 = fp.p0; a.p1 = fp.p1; a.p2 = fp.p2; a.p3 = fp.p3;
    a.extra = fp.extra;
    a.hij = hij; a.hijp = hijp; a.bstate = bstate;
    a.phi_hom = fp.phi_hom;
    a.err = fp.err;
    a.partial = fp.partial;
    a.npartial = fp.npartial;
    a.sum = fp.sum;
    a.bins = fp.bins;
    a.occ = fp.occ;
    a.tab = fp.tab;
    a.ntab = fp.ntab;
    a.modes = fp.modes;
    GEV_SWITCH_N(N, (fz_dispatch<R, NN>(fp, a, tb, st)))
}

// prepareFTsource as standalone passes, in place (the reference's call shape,
// main.cu:725, :822): T00 form into the source field with per-block sums of
// the source (row blocks of N points, one partial per (y, z) row); Tij form
// on the six Sij planes
template <class R>
__global__ void k_prep_t00(FxArgs<R> a, int N, R *out, double *partial)
{
    __shared__ double red[256 / 32];
    const int y = blockIdx.x, z = blockIdx.y;
    double lsum = 0.0;
    for (int x = threadIdx.x; x < N; x += blockDim.x) {
        double src;
        const double r = prep_t00(a, N, x, y, z, src);
        lsum += src;
        out[sidx(N, x, y, z)] = (R)r;   // the same point was read above: in place is safe
    }
    for (int o = 16; o > 0; o >>= 1) lsum += __shfl_down_sync(0xffffffffu, lsum, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = lsum;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < (int)(blockDim.x / 32); w++) s += red[w];
        partial[y + (int64_t)N * z] = s;
    }
}

template <class R>
__global__ void k_prep_tij(R *Sij, int64_t n3, const R *__restrict__ phi, R coeff, int N)
{
    const int y = blockIdx.x, z = blockIdx.y;
    for (int x = threadIdx.x; x < N; x += blockDim.x) {
        R o[6];
#pragma unroll
        for (int c = 0; c < 6; c++) o[c] = prep_tij(Sij + c * n3, phi, coeff, c, N, x, y, z);
#pragma unroll
        for (int c = 0; c < 6; c++) Sij[c * n3 + sidx(N, x, y, z)] = o[c];
    }
}

template <class R>
void prep_t00_pass(int N, R *source, const R *phi, const R *chi, double bg, double c, double c2, double c3, double *partial,
                   cudaStream_t st)
{
    FxArgs<R> a{};
    a.in = source; a.phi = phi; a.chi = chi;
    a.bg = bg; a.c = c; a.c2 = c2; a.c3 = c3;
    k_prep_t00<R><<<dim3(N, N), 256, 0, st>>>(a, N, source, partial);
}

template <class R>
void prep_tij_pass(int N, R *Sij, const R *phi, double coeff, cudaStream_t st)
{
    k_prep_tij<R><<<dim3(N, N), 128, 0, st>>>(Sij, (int64_t)N * N * N, phi, (R)coeff, N);
}

#define GEV_SOLVE_INST(R)                                                                                            \
    template int fxy_forward<R>(int, int, const R *, int64_t, int, const R *, const R *, double, double, double, double, \
                                CT<R>::C *, int64_t, double *, const FftTables<R> &, cudaStream_t, bool);            \
    template int fyx_inverse<R>(int, CT<R>::C *, int64_t, R *, int64_t, int, const FftTables<R> &, cudaStream_t);     \
    template void fz_pass<R>(int, const FzParams &, CT<R>::C *, int64_t, CT<R>::C *, CT<R>::C *, CT<R>::C *,          \
                             const FftTables<R> &, cudaStream_t);                                                    \
    template void prep_t00_pass<R>(int, R *, const R *, const R *, double, double, double, double, double *,          \
                                   cudaStream_t);                                                                    \
    template void prep_tij_pass<R>(int, R *, const R *, double, cudaStream_t);

}  // namespace gev
