// The FP64 HLLC and LLF fluxes between two equal states, whose flux is the
// physical one, over scales of density and at zero pressure.  Prints the
// largest error of each, relative to the largest term of its sums.
#include <cstdio>
#include <vector>

#include "device.cuh"

namespace rkdg {
__global__ void fluxes(const double* u, int n, double gamma, double* f) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double nx = 0.6, ny = 0.8;
    hllc_flux(u + 4 * i, u + 4 * i, nx, ny, gamma, f + 8 * i);
    llf_flux(u + 4 * i, u + 4 * i, nx, ny, 0.0, gamma - 1.0, f + 8 * i + 4);
}

int run() {
    std::vector<double> u;
    const double dirs[5][2] = {{2, 1}, {-2, -1}, {0.25, 0.5}, {-0.25, -0.5}, {0, 0}};
    for (double scale : {1e-200, 1e-170, 1.0, 1e150, 1e200})
        for (double p : {0.0, 1.0})
            for (const auto& d : dirs)  // E = p / (gamma - 1) + rho |v|^2 / 2, exact at p = 0
                for (double v : {scale, scale * d[0], scale * d[1], scale * (p * 2.5 + 0.5 * (d[0] * d[0] + d[1] * d[1]))})
                    u.push_back(v);
    const int n = (int)u.size() / 4;
    std::vector<double> f(8 * n);
    double *du, *df;
    RKDG_CUDA_TRY(cudaMalloc(&du, sizeof(double) * u.size()));
    RKDG_CUDA_TRY(cudaMalloc(&df, sizeof(double) * f.size()));
    RKDG_CUDA_TRY(cudaMemcpy(du, u.data(), sizeof(double) * u.size(), cudaMemcpyHostToDevice));
    fluxes<<<(n + 63) / 64, 64>>>(du, n, 1.4, df);
    RKDG_CUDA_TRY(cudaMemcpy(f.data(), df, sizeof(double) * f.size(), cudaMemcpyDeviceToHost));
    double worst[2] = {0, 0};
    for (int i = 0; i < n; ++i) {
        const long double r = u[4 * i], vx = u[4 * i + 1] / r, vy = u[4 * i + 2] / r, E = u[4 * i + 3];
        const long double p = 0.4L * (E - 0.5L * r * (vx * vx + vy * vy)), q = 0.6L * vx + 0.8L * vy;
        const long double c = sqrtl(1.4L * fabsl(p) / r), size = (r + E + fabsl(p)) * (fabsl(vx) + fabsl(vy) + c) + fabsl(p);
        const long double want[4] = {r * q, r * vx * q + p * 0.6L, r * vy * q + p * 0.8L, (E + p) * q};
        for (int k = 0; k < 8; ++k) {
            const double e = size > 0 ? (double)(fabsl(f[8 * i + k] - want[k % 4]) / size) : fabs(f[8 * i + k]);
            if (!(e <= worst[k / 4])) worst[k / 4] = e == e ? e : 1e300;
        }
    }
    std::printf("%.3g %.3g\n", worst[0], worst[1]);
    return 0;
}
}  // namespace rkdg

int main() {
    try {
        return rkdg::run();
    } catch (const rkdg::Error& e) {
        std::fprintf(stderr, "%s\n", e.msg.c_str());
        return 1;
    }
}
