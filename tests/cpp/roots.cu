// Largest distance, in units in the last place, of the flux arithmetic's
// FP64 reciprocal and roots from CUDA's IEEE ones over n arguments spread
// over the logarithm of [1e-200, 1e200], and what they give at 0 and below.
#include <cstdio>

#include "roots.cuh"

__device__ double ulps(double a, double b) {
    return fabs((double)(__double_as_longlong(a) - __double_as_longlong(b)));
}

__global__ void worst(int n, unsigned long long* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    // a low-discrepancy exponent and mantissa
    const double a = fmod(i * 0.6180339887498949, 1.0), b = fmod(i * 0.7548776662466927, 1.0);
    const double x = exp10(400.0 * a - 200.0) * (1.0 + b);
    double r, ir;
    rkdg::roots_f64(x, r, ir);
    atomicMax(out + 0, (unsigned long long)ulps(rkdg::rcp_f64(x), 1.0 / x));
    atomicMax(out + 1, (unsigned long long)ulps(rkdg::rcp_f64(-x), -1.0 / x));
    atomicMax(out + 2, (unsigned long long)ulps(r, sqrt(x)));
    atomicMax(out + 3, (unsigned long long)(fabs(ir * sqrt(x) - 1.0) * 4503599627370496.0));
    if (i == 0) {
        rkdg::roots_f64(0.0, r, ir);
        out[4] = r >= 0.0 && r <= 1e-140;
        rkdg::roots_f64(-1.0, r, ir);
        out[5] = r != r;
    }
}

int main() {
    const int n = 1 << 22;
    unsigned long long *d, h[6];
    if (cudaMalloc(&d, sizeof(h)) != cudaSuccess) return 1;
    cudaMemset(d, 0, sizeof(h));
    worst<<<n / 256, 256>>>(n, d);
    if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    for (unsigned long long v : h) std::printf("%llu ", v);
    std::printf("\n");
    return 0;
}
