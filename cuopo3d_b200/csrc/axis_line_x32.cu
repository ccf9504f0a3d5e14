// Line-specialised x-pass kernels, FP32.
#include "axis_line_kernels.cuh"

namespace opo {
OPO_AXIS_LINE_INSTANCE(float2, true)
}
