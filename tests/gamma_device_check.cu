// gamma_f32 (grad_f32.cuh) against std.math.pow(x, 2.2) as the library
// restates it, on the device, for every float in [0, 1.001]: the largest
// difference must stay below kGammaErr.
#include <cstdio>

#include "z2d_internal.h"
using namespace z2dg;

__global__ void check(uint32_t last, uint32_t *worst) {
    uint32_t w = 0;
    for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b <= last; b += gridDim.x * blockDim.x) {
        const float x = __uint_as_float(b);
        w = max(w, __float_as_uint(fabsf(gamma_f32(x) - zpow(x, kGamma))));  // (a NaN is the largest)
    }
    atomicMax(worst, w);
}

int main() {
    uint32_t *d, h = 0;
    float top = 1.001f;
    uint32_t last;
    memcpy(&last, &top, 4);
    if (cudaMalloc(&d, 4) || cudaMemset(d, 0, 4)) return 2;
    check<<<1216, 256>>>(last, d);
    if (cudaMemcpy(&h, d, 4, cudaMemcpyDeviceToHost)) return 2;
    float worst;
    memcpy(&worst, &h, 4);
    printf("floats %u worst %.4g limit %.4g\n", last + 1, worst, kGammaErr);
    return worst < kGammaErr ? 0 : 1;
}
