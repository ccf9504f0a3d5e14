// Line-specialised t-pass kernels, FP32.
#include "tpass_line_kernels.cuh"

namespace opo {
OPO_TPASS_LINE_INSTANCE(float2)
}
