// The resident solve kernel's FP64 forms with the limiter (resident.cuh).
#include "device.cuh"

namespace rkdg {

#include "resident.cuh"

extern const ResidentUnit resident_fp64_tvb = resident_unit_of<double, 1>();

}  // namespace rkdg
