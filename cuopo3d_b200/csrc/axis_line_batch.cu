// Batched line-specialised x- and y-passes: one kernel per precision and axis, a CTA per tile
// (one field each) of every instance whose axis length has a compiled body; the instance's
// length selects the body (axis_line.cuh).
#include "axis_line.cuh"
#include "batch_device.cuh"

namespace opo {

// CTA size of the batched kernels: 128 x 6 (FP32, 80 registers) or 64 x 8 (FP64, 128
// registers) per SM, the single-instance kernels' sizes at 128-point lines.
template <typename C> constexpr int kBatchThreads = sizeof(C) == 16 ? 64 : 128;

template <typename C, bool X>
__global__ void __launch_bounds__(kBatchThreads<C>, sizeof(C) == 16 ? 8 : 6)
    axis_line_batch_kernel(const AxisArgs<C> *descs, const unsigned *prefix, const BatchHeader *hdr)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *sm = reinterpret_cast<C *>(smem_raw);
    const unsigned gt = blockIdx.x;
    if (gt >= hdr->total_tiles) return;
    prefix += hdr->pfirst;
    const int i = find_inst(prefix, hdr->ninst, gt);
    const AxisArgs<C> &d = descs[hdr->first + i];
    unsigned tile = gt - __ldg(prefix + i), f = 0;
    const unsigned nt = (unsigned)d.g.ntiles;
    while (tile >= nt) {
        tile -= nt;
        f++;
    }
    if (!(d.tmask >> f & 1u)) return;
    unsigned lim;
    const unsigned base = axis_line_base(d.g, tile, d.line_extent, lim);
    switch (d.line_n) {
#define OPO_CASE(N)                                                                                 \
    case N:                                                                                         \
        axis_line_tile<C, AxisLine<C, X, N>, kBatchThreads<C>, 0u>(d.f[f] + base, lim, d.g.gs_j, d.tab[f], d.tw, sm); \
        break;
        OPO_AXIS_LINES(OPO_CASE)
#undef OPO_CASE
    default: break;
    }
}

template <typename C, bool X> const void *axis_line_batch_func(int *threads)
{
    *threads = kBatchThreads<C>;
    return reinterpret_cast<const void *>(axis_line_batch_kernel<C, X>);
}

template const void *axis_line_batch_func<float2, true>(int *);
template const void *axis_line_batch_func<float2, false>(int *);
template const void *axis_line_batch_func<double2, true>(int *);
template const void *axis_line_batch_func<double2, false>(int *);

}  // namespace opo
