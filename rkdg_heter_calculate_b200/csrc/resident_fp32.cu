// The resident solve kernel's FP32 forms without the limiter (resident.cuh).
#include "device.cuh"

namespace rkdg {

#include "resident.cuh"

extern const ResidentUnit resident_fp32 = resident_unit_of<float, 0>();

}  // namespace rkdg
