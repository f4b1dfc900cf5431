// The resident solve kernel (128 threads per tile, P1 with the limiter) on one
// tile of one element, its own neighbour across an edge, whose tables also name
// a neighbour's mean that nobody publishes in the first stage of a step and
// that lies ready in the second: the wait for it runs out after its two
// seconds.  Prints the error word, the done flag, the steps and the
// milliseconds of that launch and of a second one behind it, then whether a
// launch of more tiles than the device holds is refused, and the error it leaves.
#include <chrono>
#include <cstdio>
#include <cstring>
#include <vector>

#include "device.cuh"

namespace rkdg {
#include "resident.cuh"

template <typename T>
T* up(const std::vector<T>& h) {
    T* d = nullptr;
    RKDG_CUDA_TRY(cudaMalloc(&d, sizeof(T) * h.size()));
    RKDG_CUDA_TRY(cudaMemcpy(d, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice));
    return d;
}

void run() {
    upload_module_tables(3, 2);
    constexpr int ld = 128, slots = 16, lost = 7;
    const int rim = EDGE_BOUNDARY | (RKDG_BC_OUTFLOW << 2);
    std::vector<double2> U(6 * ld, make_double2(0, 0)), jinv(2 * ld, make_double2(0, 1)), lim(3 * ld, make_double2(0.5, 0.5));
    U[0] = make_double2(1.0, 0.0), U[ld] = make_double2(0.0, 2.5);
    jinv[0] = make_double2(1, 0);
    U[2 * ld] = make_double2(0.1, 0.0);  // a slope that the limiter (M = 0) must act on
    const int tags = (RKDG_BC_OUTFLOW << 8) | (RKDG_BC_OUTFLOW << 10);
    // edge 0: halo entry 0, the element's own edge 0; of edge 1 the flux sees
    // the rim, the limiter a neighbour in another tile
    const std::vector<int4> code(ld, make_int4(EDGE_HALO, rim | (lost << 4), rim, 0)), conn(ld, make_int4(1, 1, -1, tags));
    const std::vector<int4> desc = {{0, 1, 0, 1}, {0, 1, 0, 3}};
    const std::vector<int2> halo(slots, make_int2(0, 0));
    const std::vector<uint16_t> task = {0, 1, 2, 0};
    std::vector<int> slot(3 * ld, -1);
    slot[0] = 0;
    std::vector<ulonglong2> trace(2 * 4 * 2 * slots, ulonglong2{0, 0}), mean(2 * 2 * 2 * slots, ulonglong2{0, 0});
    const double value[4] = {1.0, 0.0, 0.0, 2.5};
    for (int half = 0; half < 4; ++half) {  // stage 2's mean of the lost slot (even stages use the first buffer)
        unsigned long long b;
        memcpy(&b, &value[half], 8);
        mean[half * slots + lost] = ulonglong2{2ull << 32 | (b & 0xffffffffull), 2ull << 32 | b >> 32};
    }
    StepCtl c{};
    c.dt_fixed = 1e-3, c.cfl = 0.1;
    ResidentArgs a{};
    StepCtl* ctl = up(std::vector<StepCtl>{c});
    unsigned char* sums = up(std::vector<unsigned char>(kResidentSums, 0));
    a.U = up(U), a.jinv = reinterpret_cast<double*>(up(jinv)), a.conn = up(conn), a.lim = up(lim), a.ctl = ctl;
    a.gamma = 1.4, a.tvb_m = 0.0, a.far = up(std::vector<double>(value, value + 4));
    a.ld = ld, a.rk = 2, a.nsteps = 1;
    a.slot = up(slot), a.slots = slots, a.trace = up(trace), a.mean = up(mean);
    a.wave = reinterpret_cast<unsigned long long*>(sums);
    a.mon = a.wave + kResidentSteps;
    a.count = reinterpret_cast<unsigned*>(a.mon + 2);
    TileArgs t{};
    t.code = up(code), t.desc = up(desc), t.halo = up(halo), t.task = up(task), t.max_halo = 8, t.ntiles = 1;
    using Form = ResidentForm<double, 3, 3, 2, RKDG_FLUX_HLLC, 1, 0>;
    Form::fit<128>(t.max_halo);  // sets the kernels' attributes
    for (int launch = 0; launch < 2; ++launch) {
        void* args[] = {&a, &t};
        const auto t0 = std::chrono::steady_clock::now();
        RKDG_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)Form::kernel<128>(), dim3(1), dim3(128), args,
                                                  Form::SM::bytes(t.max_halo), 0));
        RKDG_CUDA_TRY(cudaDeviceSynchronize());
        const double ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
        RKDG_CUDA_TRY(cudaMemcpy(&c, ctl, sizeof(c), cudaMemcpyDeviceToHost));
        std::printf("%d %d %d %.0f\n", c.error, c.done, c.step, ms);
        a.epoch += 2;
    }
    t.ntiles = 1 << 20;
    const bool refused = !Form::launch(a, t, false, 0);
    std::printf("%d %d\n", refused, (int)cudaPeekAtLastError());
}
}  // namespace rkdg

int main() {
    try {
        rkdg::run();
    } catch (const rkdg::Error& e) {
        std::fprintf(stderr, "%s\n", e.msg.c_str());
        return 1;
    }
    return 0;
}
