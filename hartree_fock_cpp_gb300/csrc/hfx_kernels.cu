// hfx_kernels.cu -- elementwise kernels around the Fock builds (sm_103a):
// symmetrisation of the accumulators, float density copies, density block
// maxima, index shifts of session task lists.
#include <cuda_runtime.h>

#include <algorithm>

#include "hfx_engine.hpp"
#include "hfx_smem.hpp"

namespace hfx {

// sum of an accumulator element over its copies
__device__ __forceinline__ double copies(const double* A, long long e, int ncopy, long long cstride)
{
    double v = A[e];
    for (int c = 1; c < ncopy; ++c) v += A[c * cstride + e];
    return v;
}

// G = (Jacc + Jacc^T)/4 - 1/2 (Kacc + Kacc^T)/8   (RHF, linalg.hpp:100-129),
// per molecule block of the packed buffers (blockIdx.y = molecule); blocks of
// molecules switched off for this build (active[f] == 0) are left untouched
__global__ void k_finish_rhf(const double* Jacc, const double* Kacc, double* G, const int* fk, const long long* fmoff,
                             const unsigned char* active, int ncopy, long long cstride)
{
    if (active && !active[blockIdx.y]) return;
    const int K = fk[blockIdx.y];
    const long long o = fmoff[blockIdx.y];
    const int n = K * K;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
        int i = e / K, j = e - i * K;
        double J = 0.25 * (copies(Jacc, o + e, ncopy, cstride) + copies(Jacc, o + j * K + i, ncopy, cstride));
        double X = 0.125 * (copies(Kacc, o + e, ncopy, cstride) + copies(Kacc, o + j * K + i, ncopy, cstride));
        G[o + e] = J - 0.5 * X;
    }
}

// J = (Jacc + Jacc^T)/4, K = (Kacc + Kacc^T)/8  (UHF, linalg.hpp:215-296)
__global__ void k_finish_uhf(const double* Jacc, const double* Ka, const double* Kb, double* J, double* Kao,
                             double* Kbo, const int* fk, const long long* fmoff, const unsigned char* active, int ncopy,
                             long long cstride)
{
    if (active && !active[blockIdx.y]) return;
    const int K = fk[blockIdx.y];
    const long long o = fmoff[blockIdx.y];
    const int n = K * K;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
        int i = e / K, j = e - i * K;
        J[o + e] = 0.25 * (copies(Jacc, o + e, ncopy, cstride) + copies(Jacc, o + j * K + i, ncopy, cstride));
        Kao[o + e] = 0.125 * (copies(Ka, o + e, ncopy, cstride) + copies(Ka, o + j * K + i, ncopy, cstride));
        Kbo[o + e] = 0.125 * (copies(Kb, o + e, ncopy, cstride) + copies(Kb, o + j * K + i, ncopy, cstride));
    }
}

// float copy of a packed density (the FP32 kernels' digestion products)
__global__ void k_to_float(const double* A, float* B, long long n)
{
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
        B[e] = (float)A[e];
}

__global__ void k_add(const double* A, const double* B, double* C, long long n)
{
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
        C[e] = A[e] + B[e];
}

// Dsh[p] = max over the (A, B) block of max(|D1|, |D2|), for every shell pair
// p (D2 may be null); the density-weighted screening of incremental builds.
__global__ void k_density_blocks(const DPair* pairs, int npairs, const double* D1, const double* D2, double* Dsh)
{
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npairs) return;
    const DPair pr = pairs[p];
    const int n0 = dncart(pr.l0), n1 = dncart(pr.l1);
    double m = 0.0;
    for (int a = 0; a < n0; ++a)
        for (int b = 0; b < n1; ++b) {
            long long e = pr.moff + (long long)(pr.bf0 + a) * pr.kdim + pr.bf1 + b;
            m = fmax(m, fabs(D1[e]));
            if (D2) m = fmax(m, fabs(D2[e]));
        }
    Dsh[p] = m;
}

KernelSpec density_blocks_spec(int npairs)
{
    KernelSpec s;
    s.func = (const void*)k_density_blocks;
    s.grid = dim3((unsigned)((npairs + 127) / 128));
    s.block = dim3(128);
    return s;
}

// Grid-stride elementwise kernels: 256 threads, at most 1024 CTAs per grid row.
static KernelSpec elementwise_spec(const void* func, long long n, int rows)
{
    KernelSpec s;
    s.func = func;
    long long grid = (n + 255) / 256;
    s.grid = dim3((unsigned)std::max(1LL, std::min(grid, 1024LL)), (unsigned)std::max(1, rows));
    s.block = dim3(256);
    return s;
}

KernelSpec finish_rhf_spec(int Kmax, int nfrag)
{
    return elementwise_spec((const void*)k_finish_rhf, (long long)Kmax * Kmax, nfrag);
}
KernelSpec finish_uhf_spec(int Kmax, int nfrag)
{
    return elementwise_spec((const void*)k_finish_uhf, (long long)Kmax * Kmax, nfrag);
}
// Shift the pair indices of a task list copied into a combined list (the
// multi-job Fock session, hfx_session.cpp).
__global__ void k_rebase_tasks(Task* t, long long n, int delta)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        t[i].bra += delta;
        t[i].ket += delta;
    }
}

KernelSpec rebase_tasks_spec(long long n) { return elementwise_spec((const void*)k_rebase_tasks, n, 1); }
KernelSpec add_spec(long long n) { return elementwise_spec((const void*)k_add, n, 1); }
KernelSpec to_float_spec(long long n) { return elementwise_spec((const void*)k_to_float, n, 1); }

cudaError_t allow_max_smem(const void* kernel)
{
    static OncePerDevice raised;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    return raised.run(dev, kernel, [&] {
        int optin = 0;
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        cudaFuncAttributes fa{};
        const cudaError_t g = cudaFuncGetAttributes(&fa, kernel);
        if (g != cudaSuccess) return g;
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes);
    });
}

}  // namespace hfx
