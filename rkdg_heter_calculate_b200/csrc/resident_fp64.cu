// The resident solve kernel's FP64 forms without the limiter (resident.cuh).
#include "device.cuh"

namespace rkdg {

#include "resident.cuh"

extern const ResidentUnit resident_fp64 = resident_unit_of<double, 0>();

}  // namespace rkdg
