/*
 * fast_math_check.cu -- the device's float functions against the kernels that
 * define them, for every float argument: expf, logf, log10f, exp10f, and powf
 * at the exponents given on the command line.  Prints the number of arguments
 * whose results differ in any bit (two NaNs are alike).
 */
#include <cstdio>
#include <cstdlib>
#include <cuda_runtime.h>
#include "../../galfast_b200/csrc/gf_math.h"

__device__ __forceinline__ bool alike(float a, float b)
{
    return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b);
}

__global__ void check(unsigned long long *bad, int kind, float y)
{
    unsigned long long n = 0;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < (1ull << 32);
         i += (unsigned long long)gridDim.x * blockDim.x) {
        const float x = __uint_as_float((unsigned)i);
        bool ok = true;
        if (kind == 0) ok = alike(gfm::expf_(x), gfm::expf_kernel(x));
        if (kind == 1) ok = alike(gfm::logf_(x), gfm::logf_kernel(x));
        if (kind == 2) ok = alike(gfm::log10f_(x), gfm::log10f_kernel(x));
        if (kind == 3) ok = alike(gfm::exp10f_(x), gfm::exp10f_kernel(x));
        if (kind == 4) ok = alike(gfm::powf_(x, y), gfm::powf_kernel(x, y));
        if (kind == 5) ok = alike(gfm::powf_(y, x), gfm::powf_kernel(y, x));
        n += ok ? 0 : 1;
    }
    if (n) atomicAdd(bad, n);
}

int main(int argc, char **argv)
{
    unsigned long long *bad, total = 0;
    if (cudaMalloc(&bad, 8) != cudaSuccess) return 2;
    const char *name[] = {"expf", "logf", "log10f", "exp10f", "powf(x, y)", "powf(y, x)"};
    for (int kind = 0; kind < 6; kind++)
        for (int k = 0; k < (kind < 4 ? 1 : argc - 1); k++) {
            const float y = kind < 4 ? 0.f : (float)atof(argv[1 + k]);
            unsigned long long n = 0;
            cudaMemset(bad, 0, 8);
            check<<<148 * 8, 256>>>(bad, kind, y);
            if (cudaMemcpy(&n, bad, 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
            printf("%s y=%g differ=%llu\n", name[kind], y, n);
            total += n;
        }
    printf("differ=%llu\n", total);
    return total == 0 ? 0 : 1;
}
