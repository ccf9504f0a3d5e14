// Kernels and launcher of the line-specialised axis passes (axis_line.cuh) for one
// precision and axis: included by the axis_line_*.cu files, which compile in parallel.
#pragma once

#include <type_traits>

#include "axis_line.cuh"

namespace opo {

// CTA u of a launch: tile u mod ntiles of the (u / ntiles)-th field of the mask.
template <typename C, typename G, unsigned GS>
__global__ void __launch_bounds__(G::THREADS, G::MINB) axis_line_kernel(AxisArgs<C> a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned fi = 0, tile = blockIdx.x;
    while (tile >= (unsigned)a.g.ntiles) {
        tile -= (unsigned)a.g.ntiles;
        fi++;
    }
    unsigned m = a.tmask;
    while (fi--) m &= m - 1;  // the fi-th field of the mask is the lowest left
    C *fp = (m & 1u) ? a.f[0] : (m & 2u) ? a.f[1] : a.f[2];
    const C *tab = (m & 1u) ? a.tab[0] : (m & 2u) ? a.tab[1] : a.tab[2];
    unsigned lim;
    fp += axis_line_base(a.g, tile, a.line_extent, lim);
    axis_line_tile<C, G, G::THREADS, GS>(fp, lim, a.g.gs_j, tab, a.tw, reinterpret_cast<C *>(smem_raw));
}

template <typename C, bool X> const void *axis_line_func(int n, bool square, int *threads)
{
    switch (n) {
#define OPO_CASE(N)                                                                                 \
    case N: {                                                                                       \
        using G = AxisLine<C, X, N>;                                                                \
        *threads = G::THREADS;                                                                      \
        if (!X && square) return reinterpret_cast<const void *>(axis_line_kernel<C, G, X ? 0u : (unsigned)N>); \
        return reinterpret_cast<const void *>(axis_line_kernel<C, G, 0u>);                          \
    }
        OPO_AXIS_LINES(OPO_CASE)
#undef OPO_CASE
    default: return nullptr;
    }
}

template <typename C, bool X>
cudaError_t launch_axis_line_t(const AxisArgs<C> &a, bool square, size_t smem, cudaStream_t st)
{
    int threads = 0;
    const void *fn = axis_line_func<C, X>(a.plan.n, square, &threads);
    if (!fn) return cudaErrorInvalidValue;
    void *args[] = {const_cast<AxisArgs<C> *>(&a)};
    return cudaLaunchKernel(fn, dim3((unsigned)a.g.ntiles * (unsigned)__builtin_popcount(a.tmask)), dim3(threads), args,
                            smem, st);
}

// Shared memory above the default 48 KB needs the attribute; set once per function.
template <typename C, bool X> cudaError_t configure_axis_line_t(int n)
{
    for (int square = 0; square < (X ? 1 : 2); square++) {
        int threads = 0;
        const void *fn = axis_line_func<C, X>(n, square != 0, &threads);
        if (!fn) return cudaErrorInvalidValue;
        cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

#define OPO_AXIS_LINE_INSTANCE(C, X)                                                                \
    template cudaError_t launch_axis_line_t<C, X>(const AxisArgs<C> &, bool, size_t, cudaStream_t);  \
    template cudaError_t configure_axis_line_t<C, X>(int);

}  // namespace opo
