// FP32 step kernels, 3D.
#include "fused32_kernels.h"

namespace dugks {

Kernels32 kernels32_3d(bool h, int npl, bool row, bool open) { return kernels32_d<3>(h, npl, row, open); }

}  // namespace dugks
