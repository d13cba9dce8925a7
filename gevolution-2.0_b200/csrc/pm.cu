// pm.cu -- differentiable Newtonian particle-mesh run and its hand-written
// adjoint (C ABI gev_pm_*, include/gev.h).
//
// Forward step n (main.cu's gr_flag == 0 branch, CDM only):
//   rho   = scalarProjectionCIC_project          (gevolution.hpp:1902)
//   psi   = solveModifiedPoissonFT(rho, pc_n)     (gevolution.hpp:806, main.cu:765)
//   q    -= kq_n * grad psi (x)                   (update_q_Newton, gevolution.hpp:1051-1118,
//                                                  GRADIENT_ORDER 2; kq_n = dtau_kick * a * N)
//   x    += kx_n * q                              (update_pos_Newton, gevolution.hpp:1270-1273;
//                                                  kx_n = dtau / a_half)
// and after the last step the CIC density contrast delta = CIC(x) N^3/Np - 1.
//
// Particles are kept in ID order with unwrapped FP64 positions (box units), so
// the state is a smooth function of the initial conditions and no
// permutation has to be undone in the reverse pass; deposits use atomics
// (the grids of a differentiable run fit in L2).
//
// Reverse step n, given the cotangents (lx, lq) of (x_{n+1}, q_{n+1}):
//   lq'  = lq + kx lx                                   (drift)
//   lx  += -kq (d grad psi / dx)^T lq'                   (kick, at fixed psi)
//   Lam  = CIC deposit of lq' (3 components)             (transpose of the force gather)
//   lpsi = -kq sum_i (Lam_i(v - e_i) - Lam_i(v + e_i))/2 (transpose of the gradient stencil)
//   lrho = Poisson(lpsi, pc_n)                           (the solve is self-adjoint)
//   lx  += mass N^3 (d CIC / dx)^T lrho                  (transpose of the deposit)
//   lq   = lq'
// States x_n and potentials psi_n are recomputed segment by segment from
// checkpoints (x, q) stored every `checkpoint_every` steps.
#include <cmath>
#include <cstring>
#include <memory>
#include <stdexcept>
#include <string>
#include <vector>

#include "gev.h"
#include "kernels.h"

namespace gev {
namespace {

struct PmError : std::runtime_error {
    int code;
    PmError(int c, const std::string &m) : std::runtime_error(m), code(c) {}
};

void pck(cudaError_t e, const char *what)
{
    if (e == cudaSuccess) return;
    cudaGetLastError();   // reported here: not to be found by the next call's launch check
    throw PmError(e == cudaErrorMemoryAllocation ? GEV_ERR_NOMEM : GEV_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

template <class T> struct PBuf {
    T *p = nullptr;
    size_t n = 0;
    void alloc(size_t count, const char *what)
    {
        if (count == n && p) return;
        release();
        if (count == 0) return;
        pck(cudaMalloc((void **)&p, count * sizeof(T)), what);
        n = count;
    }
    void release()
    {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
    ~PBuf() { release(); }
};

constexpr int PM_NT = 256;

// cell corner and in-cell offset of an unwrapped box-unit coordinate.  The
// cell is reduced into the box in FP64 (floor of the quotient, at most one
// off, then one correction): a 64-bit integer remainder per coordinate costs
// more than the whole interpolation.  A non-finite coordinate gives cell 0.
__device__ __forceinline__ void pm_cell(double x, int N, double invN, int &c, double &d)
{
    const double p = x * (double)N;
    const double f = floor(p);
    d = p - f;
    int ci = (int)(f - (double)N * floor(f * invN));
    if (ci < 0) ci += N;
    if (ci >= N) ci -= N;
    c = (unsigned)ci < (unsigned)N ? ci : 0;
}

__device__ __forceinline__ int pm_wrap1(int i, int N) { return i >= N ? i - N : (i < 0 ? i + N : i); }

// The run's own particle arrays are three planes of np values (the caller's
// are triples): a warp's load of one coordinate is 256 contiguous bytes where
// triples spread it over 768, and the particle passes are bound by the L1
// wavefronts of their loads.
struct Vec3 {
    double v[3];
};
__device__ __forceinline__ Vec3 pm_get(const double *p, int64_t np, int64_t i)
{
    return Vec3{{p[i], p[np + i], p[2 * np + i]}};
}
__device__ __forceinline__ void pm_put(double *p, int64_t np, int64_t i, const double (&v)[3])
{
    p[i] = v[0];
    p[np + i] = v[1];
    p[2 * np + i] = v[2];
}

// triples -> planes and back
__global__ void k_pm_planes(const double *__restrict__ in, double *__restrict__ out, int64_t np)
{
    pdl_entry();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np; i += (int64_t)gridDim.x * blockDim.x) {
        const double v[3] = {in[3 * i], in[3 * i + 1], in[3 * i + 2]};
        pm_put(out, np, i, v);
    }
}
__global__ void k_pm_triples(const double *in, double *out, int64_t np)
{
    pdl_entry();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np; i += (int64_t)gridDim.x * blockDim.x) {
        const Vec3 v = pm_get(in, np, i);
#pragma unroll
        for (int k = 0; k < 3; k++) out[3 * i + k] = v.v[k];
    }
}

// A particle's cell and the grid offsets (x; N y; N^2 z, all below 2^31) of
// the four planes c - 1 .. c + 2 per axis.
struct PmSite {
    double d[3];
    int x[4], y[4], z[4];
    __device__ __forceinline__ PmSite(const double (&pos)[3], int N, double invN)
    {
        int c[3];
#pragma unroll
        for (int k = 0; k < 3; k++) pm_cell(pos[k], N, invN, c[k], d[k]);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            x[k] = pm_wrap1(c[0] + k - 1, N);
            y[k] = pm_wrap1(c[1] + k - 1, N) * N;
            z[k] = pm_wrap1(c[2] + k - 1, N) * N * N;
        }
    }
    __device__ __forceinline__ int at(int bx, int by, int bz) const { return x[bx + 1] + y[by + 1] + z[bz + 1]; }
    __device__ __forceinline__ double w(int axis, int b) const { return b ? d[axis] : 1.0 - d[axis]; }
};

template <bool EARLY, class R> __device__ __forceinline__ double pm_ld(const R *f, int i) { return (double)ld<EARLY>(f + i); }

// CIC deposit of cst at the particle's 8 corners
template <class R> __device__ __forceinline__ void pm_scatter(const PmSite &s, double cst, R *out)
{
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int bx = (k >> 2) & 1, by = (k >> 1) & 1, bz = k & 1;
        const double w = s.w(0, bx) * s.w(1, by) * s.w(2, bz);
        atomicAdd(out + s.at(bx, by, bz), (R)(w * cst));
    }
}

// one site's three values, interleaved with a pad: a corner's three additions
// are one 16-byte vector addition in FP32
__device__ __forceinline__ void pm_add3(float *out, double a, double b, double c)
{
    atomicAdd(reinterpret_cast<float4 *>(out), make_float4((float)a, (float)b, (float)c, 0.0f));
}
__device__ __forceinline__ void pm_add3(double *out, double a, double b, double c)
{
    atomicAdd(out, a);
    atomicAdd(out + 1, b);
    atomicAdd(out + 2, c);
}

// G[i][k] = (psi(c_k + e_i) - psi(c_k - e_i)) / 2 at the 8 corners c_k of the
// cell: 32 distinct values (the 8 corners and the 24 one step outside them)
template <bool EARLY, class R>
__device__ __forceinline__ void pm_grad_corners(const R *psi, const PmSite &s, double G[3][8])
{
    double in[8];
#pragma unroll
    for (int k = 0; k < 8; k++) in[k] = pm_ld<EARLY>(psi, s.at((k >> 2) & 1, (k >> 1) & 1, k & 1));
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int bx = (k >> 2) & 1, by = (k >> 1) & 1, bz = k & 1;
        // the neighbour inside the cell is a corner, the other one lies outside
        const double ox = pm_ld<EARLY>(psi, s.at(bx ? 2 : -1, by, bz)), oy = pm_ld<EARLY>(psi, s.at(bx, by ? 2 : -1, bz)),
                     oz = pm_ld<EARLY>(psi, s.at(bx, by, bz ? 2 : -1));
        G[0][k] = 0.5 * (bx ? ox - in[k & 3] : in[k | 4] - ox);
        G[1][k] = 0.5 * (by ? oy - in[k & 5] : in[k | 2] - oy);
        G[2][k] = 0.5 * (bz ? oz - in[k & 6] : in[k | 1] - oz);
    }
}

// mass deposit alone (the start of a run or of a recomputed segment)
template <class R>
__global__ void k_pm_deposit(const double *x, int64_t np, int N, double cst, R *out)
{
    pdl_entry();
    const double invN = 1.0 / N;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np; i += (int64_t)gridDim.x * blockDim.x)
        pm_scatter(PmSite(pm_get(x, np, i).v, N, invN), cst, out);
}

// forward kick (update_q_Newton) and drift (update_pos_Newton) from (xi, qi)
// to (xo, qo) (the same arrays or others), and the deposit of cst at the new
// position that the next step (or the final density) needs: the moved
// positions are not read back
template <class R, bool EARLY>
__global__ void __launch_bounds__(PM_NT, 3) k_pm_kick_drift(const double *xi, const double *qi, double *xo, double *qo, int64_t np, int N,
                                const R *psi, double kq, double kx, double cst, R *rho)
{
    pdl_entry<EARLY>();
    const double invN = 1.0 / N;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np; i += (int64_t)gridDim.x * blockDim.x) {
        double x[3], q[3];
#pragma unroll
        for (int a = 0; a < 3; a++) {
            x[a] = xi[a * np + i];
            q[a] = qi[a * np + i];
        }
        {
            const PmSite s(x, N, invN);
            double G[3][8];
            pm_grad_corners<EARLY>(psi, s, G);
            double g[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const double w = s.w(0, (k >> 2) & 1) * s.w(1, (k >> 1) & 1) * s.w(2, k & 1);
#pragma unroll
                for (int a = 0; a < 3; a++) g[a] += w * G[a][k];
            }
#pragma unroll
            for (int a = 0; a < 3; a++) {
                q[a] -= kq * g[a];
                x[a] += kx * q[a];
            }
        }
        pm_put(qo, np, i, q);
        pm_put(xo, np, i, x);
        if (rho) pm_scatter(PmSite(x, N, invN), cst, rho);
    }
}

// dw_k/dd_m v_k summed over the corners: gradient of the CIC interpolation
__device__ __forceinline__ void pm_weight_grad(const PmSite &s, const double v[8], double gm[3])
{
    gm[0] = gm[1] = gm[2] = 0.0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int bx = (k >> 2) & 1, by = (k >> 1) & 1, bz = k & 1;
        const double fx = s.w(0, bx), fy = s.w(1, by), fz = s.w(2, bz);
        gm[0] += (bx ? fy : -fy) * fz * v[k];
        gm[1] += (by ? fx : -fx) * fz * v[k];
        gm[2] += (bz ? fx : -fx) * fy * v[k];
    }
}

// One reverse pass over the particles, the end of step n + 1 and the start of
// step n together (both update the cotangents lx):
//   1. transpose of the CIC deposit of weight mf at xb (step n + 1's mass
//      deposit, or the final density): lx_m += mf N sum_k dw_k/dd_m f(c_k);
//   2. when xa is given, reverse of the drift and of the kick at fixed psi at
//      xa = x_n: lq becomes lq' (the cotangent of the kicked momentum), and
//      lq' is deposited into lam (three interleaved components) for the field
//      part of the step.
// (lxi, lqi) null: the cotangents start at zero.
template <class R, bool EARLY>
__global__ void __launch_bounds__(PM_NT, 2) k_pm_reverse(const double *xb, const R *f, double mf, const double *xa,
                             const R *psi, double kq, double kx, const double *lxi, const double *lqi,
                             double *lxo, double *lqo, R *lam, int64_t np, int N)
{
    pdl_entry<EARLY>();
    const double invN = 1.0 / N;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < np; i += (int64_t)gridDim.x * blockDim.x) {
        double lx[3], lq[3];
#pragma unroll
        for (int a = 0; a < 3; a++) {
            lx[a] = lxi ? lxi[a * np + i] : 0.0;
            lq[a] = lqi ? lqi[a * np + i] : 0.0;
        }
        {
            const PmSite s(pm_get(xb, np, i).v, N, invN);
            double v[8], gm[3];
#pragma unroll
            for (int k = 0; k < 8; k++) v[k] = pm_ld<EARLY>(f, s.at((k >> 2) & 1, (k >> 1) & 1, k & 1));
            pm_weight_grad(s, v, gm);
#pragma unroll
            for (int a = 0; a < 3; a++) lx[a] += mf * (double)N * gm[a];
        }
        if (xa) {
            const PmSite s(pm_get(xa, np, i).v, N, invN);
#pragma unroll
            for (int a = 0; a < 3; a++) lq[a] += kx * lx[a];
            double G[3][8], v[8], gm[3];
            pm_grad_corners<EARLY>(psi, s, G);
            // lx_m -= kq N sum_k dw_k/dd_m (sum_a lq'_a G[a][k])
#pragma unroll
            for (int k = 0; k < 8; k++) v[k] = lq[0] * G[0][k] + lq[1] * G[1][k] + lq[2] * G[2][k];
            pm_weight_grad(s, v, gm);
#pragma unroll
            for (int a = 0; a < 3; a++) lx[a] -= kq * (double)N * gm[a];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int bx = (k >> 2) & 1, by = (k >> 1) & 1, bz = k & 1;
                const double w = s.w(0, bx) * s.w(1, by) * s.w(2, bz);
                pm_add3(lam + 4 * (int64_t)s.at(bx, by, bz), w * lq[0], w * lq[1], w * lq[2]);
            }
        }
        pm_put(lxo, np, i, lx);
        pm_put(lqo, np, i, lq);
    }
}

// lpsi(v) = -kq sum_i (Lam_i(v - e_i) - Lam_i(v + e_i)) / 2; grid (N/32 or 1, N/4, N/2), block (min(N,32), 4, 2)
template <class R, bool EARLY>
__global__ void k_pm_adj_div(const R *lam, int N, double kq, R *lpsi)
{
    pdl_entry<EARLY>();
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y,
              z = blockIdx.z * blockDim.z + threadIdx.z;
    if (x >= N || y >= N || z >= N) return;
    auto at = [&](int xx, int yy, int zz, int c) {
        return (double)ld<EARLY>(lam + 4 * (int64_t)(pm_wrap1(xx, N) + N * (pm_wrap1(yy, N) + N * pm_wrap1(zz, N))) + c);
    };
    double s = at(x - 1, y, z, 0) - at(x + 1, y, z, 0);
    s += at(x, y - 1, z, 1) - at(x, y + 1, z, 1);
    s += at(x, y, z - 1, 2) - at(x, y, z + 1, 2);
    lpsi[x + N * (y + N * z)] = (R)(-kq * 0.5 * s);
}

template <class R>
__global__ void k_pm_contrast(const R *rho, int64_t n3, double *out)
{
    pdl_entry();
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < n3; g += (int64_t)gridDim.x * blockDim.x)
        out[g] = (double)rho[g] - 1.0;
}

template <class R>
__global__ void k_pm_to_field(const double *__restrict__ in, int64_t n3, R *out)
{
    pdl_entry();
    for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < n3; g += (int64_t)gridDim.x * blockDim.x)
        out[g] = (R)in[g];
}

struct PmBase {
    virtual ~PmBase() = default;
    virtual void forward(int nsteps, const double *coef, const double *x0, const double *q0, double *delta,
                         double *xo, double *qo) = 0;
    virtual void adjoint(const double *ddelta, double *gx0, double *gq0) = 0;
    virtual cudaStream_t stream() = 0;
};

template <class R> struct Pm final : PmBase {
    using C = typename CT<R>::C;
    int N;
    int64_t np, n3, nk;
    double mass;
    int every;
    int device;
    cudaStream_t st = nullptr;
    PBuf<R> fields;          // one allocation for rho, fld and lam
    R *rho = nullptr;        // deposited density of the step
    R *fld = nullptr;        // potential of a forward step; cotangent of a density (reverse)
    R *lam = nullptr;        // deposited momentum cotangents, [N^3][4]
    PBuf<C> W, twf, twh;
    PBuf<double> k2;
    PBuf<double2> ks;
    PBuf<double> state;      // one allocation for the particles and their cotangents
    double *x = nullptr, *q = nullptr, *lx = nullptr, *lq = nullptr;
    PBuf<int> derr;                                        // device error word of the Fourier passes
    std::vector<std::unique_ptr<PBuf<double>>> ckx, ckq;   // checkpoints (x, q) before steps 0, k, 2k, ...
    std::vector<std::unique_ptr<PBuf<double>>> segx;       // x_n within the segment being reversed
    std::vector<std::unique_ptr<PBuf<R>>> segpsi;          // psi_n within the segment
    std::vector<double> coefs;                             // 3 per step: kq, kx, pc
    int nsteps = 0;
    bool have_forward = false;

    Pm(const gev_pm_config &cfg) : N(cfg.N), np(cfg.np), mass(cfg.mass), every(cfg.checkpoint_every), device(cfg.device)
    {
        pck(cudaSetDevice(cfg.device), "cudaSetDevice");
        pck(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking), "stream");
        n3 = (int64_t)N * N * N;
        nk = (int64_t)(N / 2 + 2) * N * N;   // Fourier rows of pitch N/2+2
        fields.alloc(6 * n3, "fields");
        rho = fields.p;
        fld = rho + n3;
        lam = fld + n3;   // 16-byte aligned: n3 is a multiple of 4096
        W.alloc(nk, "spectrum");
        state.alloc(12 * np, "particles");
        x = state.p;
        q = x + 3 * np;
        lx = q + 3 * np;
        lq = lx + 3 * np;
        derr.alloc(1, "error word");
        pck(cudaMemset(derr.p, 0, sizeof(int)), "memset");
        std::vector<C> tf(N), th(N / 2);
        for (int k = 0; k < N; k++) {
            const double ang = -2.0 * M_PI * (double)k / N;
            tf[k].x = (R)std::cos(ang);
            tf[k].y = (R)std::sin(ang);
        }
        for (int k = 0; k < N / 2; k++) {
            const double ang = -2.0 * M_PI * (double)k / (N / 2);
            th[k].x = (R)std::cos(ang);
            th[k].y = (R)std::sin(ang);
        }
        std::vector<double> hk2(N);
        std::vector<double2> hks(N);
        for (int i = 0; i < N; i++) {   // gevolution.hpp:269-275
            const double gk = 2.0 * (double)N * std::sin(M_PI * (double)i / (double)N);
            hks[i] = make_double2(gk * std::cos(M_PI * (double)i / (double)N), -gk * std::sin(M_PI * (double)i / (double)N));
            hk2[i] = gk * gk;
        }
        twf.alloc(N, "tables"); twh.alloc(N / 2, "tables"); k2.alloc(N, "tables"); ks.alloc(N, "tables");
        pck(cudaMemcpy(twf.p, tf.data(), N * sizeof(C), cudaMemcpyHostToDevice), "tables");
        pck(cudaMemcpy(twh.p, th.data(), (N / 2) * sizeof(C), cudaMemcpyHostToDevice), "tables");
        pck(cudaMemcpy(k2.p, hk2.data(), N * sizeof(double), cudaMemcpyHostToDevice), "tables");
        pck(cudaMemcpy(ks.p, hks.data(), N * sizeof(double2), cudaMemcpyHostToDevice), "tables");
    }
    ~Pm() override
    {
        if (st) {
            cudaStreamSynchronize(st);
            cudaStreamDestroy(st);
        }
    }
    cudaStream_t stream() override { return st; }

    // after a synchronisation: a bulk tensor copy of a y or z pass that timed out
    // leaves its pencils untransformed and sets the error word
    void check_device(const char *what)
    {
        int e = 0;
        pck(cudaMemcpy(&e, derr.p, sizeof(int), cudaMemcpyDeviceToHost), "error word");
        if (e) {
            pck(cudaMemset(derr.p, 0, sizeof(int)), "memset");
            throw PmError(GEV_ERR_DEVICE, std::string(what) + ": device error word (bulk tensor copy timed out)");
        }
    }

    unsigned pgrid() const { return (unsigned)std::min<int64_t>((np + PM_NT - 1) / PM_NT, 148 * 16); }
    unsigned fgrid() const { return (unsigned)std::min<int64_t>((n3 + PM_NT - 1) / PM_NT, 148 * 16); }
    FftTables<R> tables() const { return FftTables<R>{twf.p, twh.p, k2.p, ks.p, derr.p}; }

    // out <- Poisson(in) with coefficient pc (modif 0): the pass sequence of gev_solve_phi
    // (clear: `in`, another array, is left zero)
    void poisson(const R *in, R *out, double pc, bool clear = false)
    {
        const FftTables<R> tb = tables();
        fxy_forward<R>(N, FX_COPY, in, n3, 1, nullptr, nullptr, 0.0, 0.0, 0.0, 0.0, W.p, nk, nullptr, tb, st, clear);
        FzParams fp{};
        fp.op = OP_POISSON;
        fp.err = derr.p;
        fp.p0 = pc / -((double)N * (double)N * (double)N);
        fp.p1 = 0.0;
        fz_pass<R>(N, fp, W.p, nk, nullptr, nullptr, nullptr, tb, st);
        fyx_inverse<R>(N, W.p, nk, out, n3, 1, tb, st);
    }

    void clear(R *f, int64_t n) { pck(cudaMemsetAsync(f, 0, n * sizeof(R), st), "memset"); }

    // density of the state xs into rho (the start of a chain of steps)
    void deposit(const double *xs, double cst)
    {
        clear(rho, n3);
        pdl_launch(k_pm_deposit<R>, pgrid(), PM_NT, 0, st, xs, np, N, cst, rho);
    }

    // potential of the density in rho, which is left cleared for the next deposit
    void potential(double pc, R *out)
    {
        poisson(rho, out, pc, true);
    }

    // whether the kernels may address a caller's array themselves: doubles on
    // their boundary, in this device's memory (or managed)
    bool direct(const double *a) const
    {
        cudaPointerAttributes at;
        if (reinterpret_cast<uintptr_t>(a) % sizeof(double) != 0) return false;
        if (cudaPointerGetAttributes(&at, a) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        return at.type == cudaMemoryTypeManaged || (at.type == cudaMemoryTypeDevice && at.device == device);
    }
    // a caller's triples to planes and back; through a copy into `spare` (3 np
    // values) where the array is not direct, so that whatever a copy accepts
    // (another device's memory, any alignment) is accepted and all else is an
    // error of the copy, not a fault of the kernel
    void from_caller(const double *in, double *planes, double *spare)
    {
        if (!direct(in)) {
            pck(cudaMemcpyAsync(spare, in, 3 * np * sizeof(double), cudaMemcpyDeviceToDevice, st), "copy in");
            in = spare;
        }
        pdl_launch(k_pm_planes, pgrid(), PM_NT, 0, st, in, planes, np);
    }
    void to_caller(const double *planes, double *out, double *spare)
    {
        double *to = direct(out) ? out : spare;
        pdl_launch(k_pm_triples, pgrid(), PM_NT, 0, st, planes, to, np);
        if (to != out) pck(cudaMemcpyAsync(out, to, 3 * np * sizeof(double), cudaMemcpyDeviceToDevice, st), "copy out");
    }

    void forward(int ns, const double *coef, const double *x0, const double *q0, double *delta, double *xo,
                 double *qo) override
    {
        have_forward = false;   // until the checkpoints of this run are all there
        nsteps = ns;
        coefs.assign(coef, coef + 3 * (size_t)ns);
        const int nck = (ns + every - 1) / every;
        while ((int)ckx.size() < nck) {
            ckx.emplace_back(new PBuf<double>());
            ckq.emplace_back(new PBuf<double>());
        }
        for (int s = 0; s < nck; s++) {
            ckx[s]->alloc(3 * np, "checkpoint");
            ckq[s]->alloc(3 * np, "checkpoint");
        }
        from_caller(x0, ckx[0]->p, x);
        from_caller(q0, ckq[0]->p, q);
        const double mcell = mass * (double)n3, contrast = (double)n3 / (double)np;
        deposit(ckx[0]->p, mcell);
        for (int n = 0; n < ns; n++) {
            potential(coefs[3 * n + 2], fld);
            // a step reads its state where the last one wrote it; the states
            // before steps 0, every, 2 every, ... are the checkpoints
            const bool from = n % every == 0, to = (n + 1) % every == 0 && n + 1 < ns;
            const int cf = n / every, ct = (n + 1) / every;
            pdl_launch(k_pm_kick_drift<R, true>, k_pm_kick_drift<R, false>, pgrid(), PM_NT, 0, st, from ? ckx[cf]->p : x,
                       from ? ckq[cf]->p : q, to ? ckx[ct]->p : x, to ? ckq[ct]->p : q, np, N, fld, coefs[3 * n],
                       coefs[3 * n + 1], n + 1 < ns ? mcell : contrast, rho);
        }
        // final CIC density contrast: mass N^3/Np per particle, minus one
        pdl_launch(k_pm_contrast<R>, fgrid(), PM_NT, 0, st, rho, n3, delta);
        if (xo) to_caller(x, xo, lx);
        if (qo) to_caller(q, qo, lq);
        pck(cudaGetLastError(), "forward launch");
        pck(cudaStreamSynchronize(st), "forward");
        check_device("forward");
        have_forward = true;
    }

    void adjoint(const double *ddelta, double *gx0, double *gq0) override
    {
        if (!have_forward) throw PmError(GEV_ERR_STATE, "gev_pm_adjoint needs a preceding gev_pm_forward");
        const double mcell = mass * (double)n3;
        const int nseg = (nsteps + every - 1) / every;
        while ((int)segx.size() < every) {
            segx.emplace_back(new PBuf<double>());
            segpsi.emplace_back(new PBuf<R>());
        }
        const int nb = N < 32 ? N : 32;
        const dim3 db(nb, 4, 2), dg(N / nb, N / 4, N / 2);
        // fld: the cotangent of the density deposited at xb (the final density first)
        pdl_launch(k_pm_to_field<R>, fgrid(), PM_NT, 0, st, ddelta, n3, fld);
        const double *xb = x;
        double mb = (double)n3 / (double)np;
        bool first = true;
        for (int s = nseg - 1; s >= 0; s--) {
            const int n0 = s * every, n1 = std::min(nsteps, n0 + every);
            // recompute x_n and psi_n of the segment from its checkpoint; q (the
            // forward's final momenta were already copied out) is the working q
            auto xn = [&](int n) { return n == n0 ? ckx[s]->p : segx[n - n0]->p; };
            deposit(ckx[s]->p, mcell);
            for (int n = n0; n < n1; n++) {
                PBuf<R> &sp = *segpsi[n - n0];
                sp.alloc(n3, "segment");
                potential(coefs[3 * n + 2], sp.p);
                if (n + 1 < n1) {
                    segx[n + 1 - n0]->alloc(3 * np, "segment");
                    pdl_launch(k_pm_kick_drift<R, true>, k_pm_kick_drift<R, false>, pgrid(), PM_NT, 0, st, xn(n),
                               n == n0 ? ckq[s]->p : q, xn(n + 1), q, np, N, sp.p, coefs[3 * n], coefs[3 * n + 1], mcell, rho);
                }
            }
            for (int n = n1 - 1; n >= n0; n--) {
                const double kq = coefs[3 * n], kx = coefs[3 * n + 1], pc = coefs[3 * n + 2];
                clear(lam, 4 * n3);
                pdl_launch(k_pm_reverse<R, true>, k_pm_reverse<R, false>, pgrid(), PM_NT, 0, st, xb, fld, mb, xn(n),
                           segpsi[n - n0]->p, kq, kx, first ? nullptr : lx, first ? nullptr : lq, lx, lq, lam, np, N);
                first = false;
                pdl_launch(k_pm_adj_div<R, true>, k_pm_adj_div<R, false>, dg, db, 0, st, lam, N, kq, fld);
                poisson(fld, fld, pc);
                mb = mcell;
                xb = xn(n);   // of the segment's first step the checkpoint, which outlives the segment
            }
        }
        pdl_launch(k_pm_reverse<R, true>, k_pm_reverse<R, false>, pgrid(), PM_NT, 0, st, xb, fld, mb, nullptr,
                   nullptr, 0.0, 0.0, lx, lq, lx, lq, nullptr, np, N);
        to_caller(lx, gx0, q);   // q is free by now
        to_caller(lq, gq0, q);
        pck(cudaGetLastError(), "adjoint launch");
        pck(cudaStreamSynchronize(st), "adjoint");
        check_device("adjoint");
    }
};

}  // namespace
}  // namespace gev

struct gev_pm {
    std::unique_ptr<gev::PmBase> impl;
    std::string err;
};

namespace {
thread_local std::string g_pm_create_error;

template <class F> int pm_guarded(gev_pm *h, F &&f)
{
    if (!h || !h->impl) return GEV_ERR_ARG;
    try {
        f(*h->impl);
        return GEV_OK;
    } catch (const gev::PmError &e) {
        h->err = e.what();
        return e.code;
    } catch (const std::exception &e) {
        h->err = e.what();
        return GEV_ERR_CUDA;
    }
}
}  // namespace

extern "C" {

int gev_pm_create(const gev_pm_config *cfg, gev_pm **out)
{
    if (!cfg || !out) return GEV_ERR_ARG;
    *out = nullptr;
    const int N = cfg->N;
    const bool okN = N == 16 || N == 32 || N == 64 || N == 128 || N == 256 || N == 384 || N == 512 || N == 768;
    if (!okN || (cfg->precision != GEV_FP64 && cfg->precision != GEV_MIXED) || cfg->np <= 0 ||
        cfg->checkpoint_every <= 0) {
        g_pm_create_error = "invalid configuration (N one of 16..768, np > 0, checkpoint_every > 0)";
        return GEV_ERR_ARG;
    }
    auto *h = new gev_pm;
    try {
        if (cfg->precision == GEV_FP64) h->impl.reset(new gev::Pm<double>(*cfg));
        else h->impl.reset(new gev::Pm<float>(*cfg));
    } catch (const gev::PmError &e) {
        g_pm_create_error = e.what();
        delete h;
        return e.code;
    } catch (const std::exception &e) {
        g_pm_create_error = e.what();
        delete h;
        return GEV_ERR_CUDA;
    }
    *out = h;
    return GEV_OK;
}

int gev_pm_destroy(gev_pm *h)
{
    delete h;
    return GEV_OK;
}

const char *gev_pm_last_error(const gev_pm *h) { return h ? h->err.c_str() : g_pm_create_error.c_str(); }

int gev_pm_forward(gev_pm *h, int32_t nsteps, const double *coef, const double *x0, const double *q0, double *delta,
                   double *x_out, double *q_out)
{
    if (!coef || !x0 || !q0 || !delta || nsteps <= 0) return GEV_ERR_ARG;
    return pm_guarded(h, [&](gev::PmBase &p) { p.forward(nsteps, coef, x0, q0, delta, x_out, q_out); });
}

int gev_pm_adjoint(gev_pm *h, const double *ddelta, double *gx0, double *gq0)
{
    if (!ddelta || !gx0 || !gq0) return GEV_ERR_ARG;
    return pm_guarded(h, [&](gev::PmBase &p) { p.adjoint(ddelta, gx0, gq0); });
}

void *gev_pm_stream(gev_pm *h) { return (h && h->impl) ? (void *)h->impl->stream() : nullptr; }

}  // extern "C"
