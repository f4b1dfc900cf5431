// How many of n arguments, spread over the exponents of FP32's normal range,
// the limiter's FP32 reciprocal and roots do not round as IEEE does.
#include <cmath>
#include <cstdio>
#include <vector>

#include "device.cuh"

__global__ void eval(int n, float* x, float* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    x[i] = exp2f(-120.0f + 240.0f * i / n) * (1.0f + (float)(i % 997) / 997.0f);
    float root, inv;
    rkdg::lim_lengths(x[i], root, inv);
    out[3 * i] = rkdg::lim_rcp(x[i]), out[3 * i + 1] = root, out[3 * i + 2] = inv;
}

int main() {
    const int n = 1 << 20;
    float *dx, *dout;
    if (cudaMalloc(&dx, sizeof(float) * n) != cudaSuccess || cudaMalloc(&dout, sizeof(float) * 3 * n) != cudaSuccess) return 1;
    eval<<<n / 256, 256>>>(n, dx, dout);
    std::vector<float> x(n), out(3 * n);
    if (cudaMemcpy(x.data(), dx, sizeof(float) * n, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    if (cudaMemcpy(out.data(), dout, sizeof(float) * 3 * n, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    int bad[3] = {0, 0, 0};
    for (int i = 0; i < n; ++i) {
        const float root = std::sqrt(x[i]);
        bad[0] += out[3 * i] != 1.0f / x[i], bad[1] += out[3 * i + 1] != root, bad[2] += out[3 * i + 2] != 1.0f / root;
    }
    std::printf("%d %d %d\n", bad[0], bad[1], bad[2]);
    return 0;
}
