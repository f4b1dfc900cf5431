// The resident solve kernel's FP32 and FP32C forms (resident.cuh).
#include "device.cuh"

namespace rkdg {

#include "resident.cuh"

int resident_bound_fp32(int order, int flux, bool limiter, bool comp, int max_halo) {
    return with_resident<float>(order, 6, flux, limiter, comp, [&](auto form) { return form.bound(max_halo); });
}

int resident_tiles_fp32(int order, int nq, int flux, bool limiter, bool comp, int max_halo) {
    return with_resident<float>(order, nq, flux, limiter, comp, [&](auto form) { return form.tiles(max_halo); });
}

bool launch_resident_fp32(const StageArgs& a, const TileArgs& t, const void* lim, ResidentWork& w, int order, int nq,
                          int flux, int rk, int steps, bool monitor, cudaStream_t stream) {
    return launch_resident_of<float>(a, t, lim, w, order, nq, flux, rk, steps, monitor, stream);
}

void upload_resident_tables_fp32(int nq, int ng) { upload_module_tables(nq, ng); }

}  // namespace rkdg
