// FP32 step kernels, 2D.
#include "fused32_kernels.h"

namespace dugks {

Kernels32 kernels32_2d(bool h, int npl, bool row, bool open) { return kernels32_d<2>(h, npl, row, open); }

}  // namespace dugks
