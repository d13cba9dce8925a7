// noalloc.cu -- gev_poisson_noalloc: the Poisson solve of the phi update on
// caller-owned device arrays, with all scratch in static device memory.
//
// Why it exists: gev_solve_phi works on fields that a context allocated.  Some
// callers cannot allocate device memory at the point where they want the
// solve: a host code that owns every device buffer through its own memory
// pool (a caching allocator that must see every allocation), or a caller in
// the middle of recording work into a stream where a cudaMalloc would either
// synchronise the device or be refused.  This entry point takes the source and
// the output as plain device pointers and keeps its one large temporary -- the
// complex half spectrum of the transform -- in a file-scope __device__ array
// of fixed size, so a call launches kernels and nothing else.
//
// Limits and rules (the same text is in include/gev.h):
//   * N in {16, 32, 64, 128}: the static scratch holds the half spectrum of a
//     128^3 grid in FP64 (N/2+2)*N*N*16 bytes = 17,301,504 bytes.  Larger N is
//     rejected with GEV_ERR_SIZE.
//   * Nothing in the scratch has to start at zero: every call writes the whole
//     spectrum before any of it is read.  The FFT and k tables are constants
//     of the library's device code.
//   * There is one scratch per device, shared by every caller of this entry
//     point in the process: two calls on the same device whose work overlaps
//     in time (different streams, no ordering between them) race on it.
//     Order such calls on one stream or synchronise between them.
//   * The host needs the device address of the scratch: the first call on a
//     device (and the first call after that device's context was destroyed and
//     re-created, e.g. by cudaDeviceReset) looks it up with
//     cudaGetSymbolAddress, which can also load the library's device code;
//     make that first call before any stream capture begins.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>

#include "gev.h"
#include "kernels.h"

namespace gev {
namespace {

constexpr int NA_MAX_N = 128;
constexpr size_t NA_SCRATCH_BYTES = (size_t)(NA_MAX_N / 2 + 2) * NA_MAX_N * NA_MAX_N * sizeof(double2);

static __device__ __align__(256) unsigned char na_scratch[NA_SCRATCH_BYTES];

// cos(2 pi k / 256), 0 <= k <= 64, rounded to FP64
constexpr double NA_QUADRANT[65] = {
    1.0, 0.9996988186962042, 0.9987954562051724, 0.9972904566786902, 0.9951847266721969, 0.99247953459871,
    0.989176509964781, 0.9852776423889412, 0.9807852804032304, 0.9757021300385286, 0.970031253194544,
    0.9637760657954398, 0.9569403357322088, 0.9495281805930367, 0.9415440651830208, 0.932992798834739,
    0.9238795325112867, 0.9142097557035307, 0.9039892931234433, 0.8932243011955153, 0.881921264348355,
    0.8700869911087115, 0.8577286100002721, 0.8448535652497071, 0.8314696123025452, 0.8175848131515837,
    0.8032075314806449, 0.7883464276266063, 0.773010453362737, 0.7572088465064846, 0.7409511253549591,
    0.724247082951467, 0.7071067811865476, 0.6895405447370668, 0.6715589548470183, 0.6531728429537768,
    0.6343932841636455, 0.6152315905806268, 0.5956993044924334, 0.5758081914178453, 0.5555702330196022,
    0.5349976198870972, 0.5141027441932217, 0.49289819222978404, 0.47139673682599764, 0.44961132965460654,
    0.4275550934302821, 0.40524131400498986, 0.3826834323650898, 0.3598950365349881, 0.33688985339222005,
    0.3136817403988915, 0.29028467725446233, 0.26671275747489837, 0.24298017990326387, 0.2191012401568698,
    0.19509032201612825, 0.17096188876030122, 0.14673047445536175, 0.1224106751992162, 0.0980171403295606,
    0.07356456359966743, 0.049067674327418015, 0.024541228522912288, 0.0};
constexpr double na_cos(int k)   // cos(2 pi k / 256), k >= 0
{
    k %= 256;
    if (k > 128) k = 256 - k;
    return k <= 64 ? NA_QUADRANT[k] : -NA_QUADRANT[128 - k];
}
constexpr double na_sin(int k) { return na_cos(k + 192); }

// FFT twiddles exp(-2 pi i k / N) and exp(-2 pi i k / (N/2)), and the k tables
// of gevolution.hpp:269-275, for one grid size; constants, so that a solve
// does not begin with a launch that writes them
template <class R, int N> struct NaTables {
    typename CT<R>::C full[N], half[N / 2];
    double k2[N];
    double2 ks[N];
    constexpr NaTables() : full(), half(), k2(), ks()
    {
        for (int k = 0; k < N; k++) {
            full[k].x = (R)na_cos(k * (256 / N));
            full[k].y = (R)-na_sin(k * (256 / N));
            if (k < N / 2) {
                half[k].x = (R)na_cos(k * (512 / N));
                half[k].y = (R)-na_sin(k * (512 / N));
            }
            const double c = na_cos(k * (128 / N)), s = na_sin(k * (128 / N)), gk = 2.0 * N * s;   // angle pi k / N
            k2[k] = gk * gk;
            ks[k].x = gk * c;
            ks[k].y = -gk * s;
        }
    }
};
template <class R> struct NaTableSet {
    NaTables<R, 16> n16;
    NaTables<R, 32> n32;
    NaTables<R, 64> n64;
    NaTables<R, 128> n128;
    constexpr NaTableSet() : n16(), n32(), n64(), n128() {}
};
struct NaAllTables {
    NaTableSet<float> f;
    NaTableSet<double> d;
    constexpr NaAllTables() : f(), d() {}
};
static __device__ const NaAllTables na_tables;

constexpr int NA_MAX_DEVICES = 64;
std::mutex na_mutex;
// per device: the scratch and table addresses and the unique id of the context it was
// resolved in (a device address is only valid inside its own context)
struct NaSlot {
    unsigned long long ctx_id = 0;
    void *ptr = nullptr;
    const void *tables = nullptr;
};
NaSlot na_slot[NA_MAX_DEVICES];

// the unique id of the calling thread's current context (0 if there is none)
int na_current_context_id(unsigned long long *id)
{
    static PFN_cuCtxGetCurrent_v4000 get_current = nullptr;
    static PFN_cuCtxGetId_v12000 get_id = nullptr;
    if (!get_current || !get_id) {
        void *p1 = nullptr, *p2 = nullptr;
        cudaDriverEntryPointQueryResult q1, q2;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p1, cudaEnableDefault, &q1) != cudaSuccess ||
            q1 != cudaDriverEntryPointSuccess || !p1 ||
            cudaGetDriverEntryPoint("cuCtxGetId", &p2, cudaEnableDefault, &q2) != cudaSuccess ||
            q2 != cudaDriverEntryPointSuccess || !p2)
            return GEV_ERR_CUDA;
        get_current = reinterpret_cast<PFN_cuCtxGetCurrent_v4000>(p1);
        get_id = reinterpret_cast<PFN_cuCtxGetId_v12000>(p2);
    }
    CUcontext cur = nullptr;
    if (get_current(&cur) != CUDA_SUCCESS) return GEV_ERR_CUDA;
    *id = 0;
    if (cur && get_id(cur, id) != CUDA_SUCCESS) return GEV_ERR_CUDA;
    return GEV_OK;
}

// device addresses of the scratch and the tables in the current context of device `dev`,
// resolved once per context
int na_addresses(int dev, unsigned char **base, const NaAllTables **tables)
{
    std::lock_guard<std::mutex> lock(na_mutex);
    unsigned long long id = 0;
    if (na_current_context_id(&id) != GEV_OK) return GEV_ERR_CUDA;
    NaSlot &s = na_slot[dev];
    if (id == 0 || !s.ptr || s.ctx_id != id) {
        void *p = nullptr, *t = nullptr;
        // makes the device's primary context current if no context is yet
        if (cudaGetSymbolAddress(&p, na_scratch) != cudaSuccess || !p) return GEV_ERR_CUDA;
        if (cudaGetSymbolAddress(&t, na_tables) != cudaSuccess || !t) return GEV_ERR_CUDA;
        if (na_current_context_id(&id) != GEV_OK || id == 0) return GEV_ERR_CUDA;
        s.ptr = p;
        s.tables = t;
        s.ctx_id = id;
    }
    *base = static_cast<unsigned char *>(s.ptr);
    *tables = static_cast<const NaAllTables *>(s.tables);
    return GEV_OK;
}

// pointers to one grid size's tables (addresses only: no device memory is read here)
template <class R, int N> FftTables<R> na_fft_tables(const NaTables<R, N> &t) { return FftTables<R>{t.full, t.half, t.k2, t.ks}; }
template <class R> FftTables<R> na_fft_tables(const NaTableSet<R> &t, int N)
{
    return N == 16 ? na_fft_tables(t.n16) : (N == 32 ? na_fft_tables(t.n32) : (N == 64 ? na_fft_tables(t.n64) : na_fft_tables(t.n128)));
}

template <class R>
int na_solve(int N, const R *src, R *dst, double coeff, double modif, unsigned char *base, const FftTables<R> &tb,
             cudaStream_t st)
{
    using C = typename CT<R>::C;
    C *spec = reinterpret_cast<C *>(base);
    const int64_t n3 = (int64_t)N * N * N, nk = (int64_t)(N / 2 + 2) * N * N;   // Fourier rows of pitch N/2+2

    // same pass sequence as the context's phi update without prepareFTsource
    fxy_forward<R>(N, FX_COPY, src, n3, 1, nullptr, nullptr, 0.0, 0.0, 0.0, 0.0, spec, nk, nullptr, tb, st);
    FzParams fp{};
    fp.op = OP_POISSON;
    fp.p0 = coeff / -((double)N * (double)N * (double)N);
    fp.p1 = modif;
    fp.phi_hom = nullptr;
    fz_pass<R>(N, fp, spec, nk, nullptr, nullptr, nullptr, tb, st);
    fyx_inverse<R>(N, spec, nk, dst, n3, 1, tb, st);
    return cudaGetLastError() == cudaSuccess ? GEV_OK : GEV_ERR_CUDA;
}

}  // namespace
}  // namespace gev

extern "C" int gev_poisson_noalloc(int32_t N, int32_t precision, const void *source, void *phi, double poisson_coeff,
                                   double modif, void *stream)
{
    using namespace gev;
    if (!source || !phi || (precision != GEV_FP64 && precision != GEV_MIXED)) return GEV_ERR_ARG;
    if (N != 16 && N != 32 && N != 64 && N != 128) {
        if (N == 256 || N == 384 || N == 512 || N == 768) return GEV_ERR_SIZE;
        return GEV_ERR_ARG;
    }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return GEV_ERR_CUDA;
    if (dev < 0 || dev >= NA_MAX_DEVICES) return GEV_ERR_ARG;
    unsigned char *base = nullptr;
    const NaAllTables *tables = nullptr;
    if (na_addresses(dev, &base, &tables) != GEV_OK) return GEV_ERR_CUDA;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    try {
        if (precision == GEV_FP64)
            return na_solve<double>(N, static_cast<const double *>(source), static_cast<double *>(phi), poisson_coeff,
                                    modif, base, na_fft_tables(tables->d, N), st);
        return na_solve<float>(N, static_cast<const float *>(source), static_cast<float *>(phi), poisson_coeff, modif,
                               base, na_fft_tables(tables->f, N), st);
    } catch (...) {
        return GEV_ERR_CUDA;
    }
}
