// Line-specialised y-pass kernels, FP64.
#include "axis_line_kernels.cuh"

namespace opo {
OPO_AXIS_LINE_INSTANCE(double2, false)
}
