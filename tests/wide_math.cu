/* The wide rows' arithmetic against what the multi-pass path computes, on the device: built and called by
 * test_gpu_wide_math.py. */
#include "../geistlib_b200/csrc/sampler_wide_math.cuh"

/* Arguments -|x| by their bits, first and up: how many come out otherwise than exp_exact's, and the bits of one. */
__global__ void exp_kernel(unsigned first, unsigned n, unsigned long long *differ, unsigned *which) {
    const double   t32  = exp2((double) (threadIdx.x & 31u) * 0x1p-5);
    const unsigned step = gridDim.x * blockDim.x;
    for (unsigned i0 = blockIdx.x * blockDim.x; i0 < n; i0 += step) { /* whole warps: the table is shared among the lanes */
        const unsigned bits = first + min(i0 + threadIdx.x, n - 1u);
        const float    a    = -__uint_as_float(bits);
        if (__float_as_uint(gb::wide_exp(a, t32)) != __float_as_uint(gb::exp_exact(a)) && i0 + threadIdx.x < n) {
            atomicAdd(differ, 1ull);
            *which = bits;
        }
    }
}
__global__ void quot_kernel(const float *e, const double *S, float *p, int *unsure, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        bool                   divide = false;
        const gb::WideQuotient quot(S[i]);
        (void) quot.quick(e[i], divide);
        p[i] = quot(e[i]);
        if (divide) {
            atomicAdd(unsure, 1);
        }
    }
}

extern "C" int exp_differs(unsigned first, unsigned n, unsigned long long *differ, unsigned *which) {
    struct Out {
        unsigned long long differ;
        unsigned           which;
    } h{}, *d = nullptr;
    cudaError_t e = cudaMalloc(&d, sizeof h);
    if (e == cudaSuccess) e = cudaMemset(d, 0, sizeof h);
    if (e == cudaSuccess) {
        exp_kernel<<<148 * 8, 256>>>(first, n, &d->differ, &d->which);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(&h, d, sizeof h, cudaMemcpyDeviceToHost);
    cudaFree(d);
    *differ = h.differ;
    *which  = h.which;
    return (int) e;
}
/* Probabilities by their bits, from 0 to 1: how many get another mass than the multi-pass path's histograms give them. */
__global__ void mass_kernel(unsigned last, unsigned long long *differ) {
    for (unsigned k = blockIdx.x * blockDim.x + threadIdx.x; k <= last; k += gridDim.x * blockDim.x) {
        const float p = __uint_as_float(k);
        if ((unsigned long long) gb::wide_mass(p) != __double2ull_rz((double) p * 0x1p62)) {
            atomicAdd(differ, 1ull);
        }
    }
}

extern "C" int mass_differs(unsigned last, unsigned long long *differ) {
    unsigned long long *d = nullptr;
    cudaError_t         e = cudaMalloc(&d, sizeof *d);
    if (e == cudaSuccess) e = cudaMemset(d, 0, sizeof *d);
    if (e == cudaSuccess) {
        mass_kernel<<<148 * 8, 256>>>(last, d);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(differ, d, sizeof *d, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int) e;
}
extern "C" int quotients(const float *e_dev, const double *S_dev, float *p_dev, int *unsure_dev, int n) {
    quot_kernel<<<(n + 255) / 256, 256>>>(e_dev, S_dev, p_dev, unsure_dev, n);
    const cudaError_t e = cudaGetLastError();
    return (int) (e != cudaSuccess ? e : cudaDeviceSynchronize());
}
