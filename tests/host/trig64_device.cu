// trig64_harness.cu's functions as the GPU runs them, with nvcc's contractions as in the engine: the special
// function unit's seeds, the table in global memory.  One thread an item; a CUDA error code or 0.
#include <cuda_runtime.h>
#include "model.cuh"

namespace {
__global__ void sincos_k(int n, const double* x, double* out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) ast::sincos_tab(x[i], out + 2 * i, out + 2 * i + 1);
}
__global__ void magnitude_k(int n, const double* v, double* out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    v += 8 * i;
    out[i] = ast::ls_algebraic(v[0], v[1], 1.0 / (v[0] * v[0]), 1.0 / (v[1] * v[1]), v[2], v[3], v[4], v[5], v[6], v[7]);
}
__global__ void quotients_k(int n, const double* us, double* out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[2 * i] = ast::quot(us[i], us[n + i]);
    out[2 * i + 1] = ast::inv_sqrt(fabs(us[n + i]));
}
__global__ void recip_k(int n, const double* s, double* out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = ast::recip(s[i]);
}
__global__ void seeds_k(int n, const double* x, double* out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[2 * i] = ast::rcp_seed(x[i]);
    out[2 * i + 1] = ast::rsqrt_seed(fabs(x[i]));
}

template <class K>
int run(K kernel, int n, const double* in, size_t n_in, double* out, size_t n_out)
{
    double *a = nullptr, *b = nullptr;
    cudaError_t e = cudaMalloc(&a, 8 * n_in);
    if (e == cudaSuccess) e = cudaMalloc(&b, 8 * n_out);
    if (e == cudaSuccess) e = cudaMemcpy(a, in, 8 * n_in, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        kernel<<<(n + 127) / 128, 128>>>(n, a, b);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, b, 8 * n_out, cudaMemcpyDeviceToHost);
    cudaFree(a);
    cudaFree(b);
    return (int)e;
}
}  // namespace

extern "C" int h_sincos_tab(int n, const double* x, double* out) { return run(sincos_k, n, x, n, out, 2 * (size_t)n); }

extern "C" int h_ls_algebraic(int n, const double* v, double* out) { return run(magnitude_k, n, v, 8 * (size_t)n, out, n); }

// us: the numerators, then the divisors.
extern "C" int h_quotients_us(int n, const double* us, double* out) { return run(quotients_k, n, us, 2 * (size_t)n, out, 2 * (size_t)n); }

extern "C" int h_recip(int n, const double* s, double* out) { return run(recip_k, n, s, n, out, n); }

// out: the seeds of 1 / x[i] and 1 / sqrt(|x[i]|).
extern "C" int h_seeds(int n, const double* x, double* out) { return run(seeds_k, n, x, n, out, 2 * (size_t)n); }
