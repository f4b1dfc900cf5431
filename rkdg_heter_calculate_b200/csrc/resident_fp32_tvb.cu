// The resident solve kernel's FP32 forms with the limiter (resident.cuh).
#include "device.cuh"

namespace rkdg {

#include "resident.cuh"

extern const ResidentUnit resident_fp32_tvb = resident_unit_of<float, 1>();

}  // namespace rkdg
