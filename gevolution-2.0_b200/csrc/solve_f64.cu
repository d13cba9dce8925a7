// solve_f64.cu -- FP64 instantiation of the pencil passes.
#include "solve_impl.cuh"

namespace gev {
GEV_SOLVE_INST(double)

// one thread per bin and sum: adds the copies in order
__global__ void k_bin_reduce(double *bins, unsigned long long *occ, int nb, int copies)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 4 * nb) {
        double s = bins[i];
        for (int c = 1; c < copies; c++) s += bins[(size_t)c * 4 * nb + i];
        bins[i] = s;
    } else if (i < 5 * nb) {
        unsigned long long n = occ[i - 4 * nb];
        for (int c = 1; c < copies; c++) n += occ[(size_t)c * nb + (i - 4 * nb)];
        occ[i - 4 * nb] = n;
    }
}

void launch_bin_reduce(double *bins, unsigned long long *occ, int nb, int copies, cudaStream_t st)
{
    k_bin_reduce<<<cdiv(5 * (int64_t)nb, 128), 128, 0, st>>>(bins, occ, nb, copies);
}
}  // namespace gev
