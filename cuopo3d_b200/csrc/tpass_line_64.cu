// Line-specialised t-pass kernels, FP64.
#include "tpass_line_kernels.cuh"

namespace opo {
OPO_TPASS_LINE_INSTANCE(double2)
}
