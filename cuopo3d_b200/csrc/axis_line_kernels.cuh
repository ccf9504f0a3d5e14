// Kernels and launcher of the line-specialised axis passes (axis_line.cuh) for one
// precision and axis: included by the axis_line_*.cu files, which compile in parallel.
#pragma once

#include <type_traits>

#include "axis_line.cuh"

namespace opo {

// Tensor maps of the fields (y: boxes of L columns, N rows).
struct AxisLineTma {
    CUtensorMap map[3];
};

// CTA u of a launch: tile u mod ntiles of the (u / ntiles)-th field of the mask.
template <typename C, typename G, unsigned GS, bool TMA>
__device__ __forceinline__ void axis_line_cta(const AxisArgs<C> &a, const CUtensorMap *maps, int *err, long long wait)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    C *sm = reinterpret_cast<C *>(smem_raw);
    unsigned fi = 0, tile = blockIdx.x;
    while (tile >= (unsigned)a.g.ntiles) {
        tile -= (unsigned)a.g.ntiles;
        fi++;
    }
    unsigned m = a.tmask;
    while (fi--) m &= m - 1;  // the fi-th field of the mask is the lowest left
    const int f = (m & 1u) ? 0 : (m & 2u) ? 1 : 2;
    C *fp = f == 0 ? a.f[0] : f == 1 ? a.f[1] : a.f[2];
    const C *tab = f == 0 ? a.tab[0] : f == 1 ? a.tab[1] : a.tab[2];
    unsigned lim;
    fp += axis_line_base(a.g, tile, a.line_extent, lim);
    if constexpr (TMA) {
        const unsigned hi = fdiv(a.g.tdiv, tile), lo = tile - hi * a.g.tdiv.d;
        unsigned long long *bar = reinterpret_cast<unsigned long long *>(smem_raw + G::BYTES);
        if (!axis_line_load<C, G>(fp, lim, maps + f, (int)(lo * G::L * (sizeof(C) / 8)), (int)hi, sm, bar, wait)) {
            // The host reports the error and takes the fields for lost.  The copy must not land
            // in a later CTA's memory: this wait keeps the full bound.  (The threads that gave up go on
            // with the others, which meet them at the tile's barriers.)
            if (err) atomicExch(err, kAxisLineTimeout);
            mbar_wait(bar, 0);
        }
    }
    axis_line_tile<C, G, G::THREADS, GS, TMA>(fp, lim, a.g.gs_j, tab, a.tw, sm);
}

template <typename C, typename G, unsigned GS>
__global__ void __launch_bounds__(G::THREADS, G::MINB) axis_line_kernel(AxisArgs<C> a)
{
    axis_line_cta<C, G, GS, false>(a, nullptr, nullptr, 0);
}
template <typename C, typename G, unsigned GS>
__global__ void __launch_bounds__(G::THREADS, G::MINB)
    axis_line_tma_kernel(AxisArgs<C> a, const __grid_constant__ AxisLineTma t, int *err, long long wait)
{
    axis_line_cta<C, G, GS, G::TMA>(a, t.map, err, wait);
}

// Kernel of an axis of n points: square: the grid is, tma: TMA-fed (axis_line_tma).
template <typename C, bool X> const void *axis_line_func(int n, bool square, bool tma, int *threads)
{
    switch (n) {
#define OPO_CASE(N)                                                                                 \
    case N: {                                                                                       \
        using G = AxisLine<C, X, N>;                                                                \
        *threads = G::THREADS;                                                                      \
        constexpr unsigned SQ = X ? 0u : (unsigned)N;                                               \
        if constexpr (G::TMA) {                                                                     \
            if (tma && square) return reinterpret_cast<const void *>(axis_line_tma_kernel<C, G, SQ>); \
            if (tma) return reinterpret_cast<const void *>(axis_line_tma_kernel<C, G, 0u>);         \
            /* y rows off 16 bytes; an x line is always fed by TMA */                               \
            if constexpr (X) return nullptr;                                                        \
            else return reinterpret_cast<const void *>(axis_line_kernel<C, G, 0u>);                 \
        } else {                                                                                    \
            if (square) return reinterpret_cast<const void *>(axis_line_kernel<C, G, SQ>);          \
            return reinterpret_cast<const void *>(axis_line_kernel<C, G, 0u>);                      \
        }                                                                                           \
    }
        OPO_AXIS_LINES(OPO_CASE)
#undef OPO_CASE
    default: return nullptr;
    }
}

template <typename C, bool X>
cudaError_t launch_axis_line_t(const AxisArgs<C> &a, bool square, const CUtensorMap *maps, int *err, long long wait,
                               size_t smem, cudaStream_t st)
{
    int threads = 0;
    const void *fn = axis_line_func<C, X>(a.plan.n, square, maps != nullptr, &threads);
    if (!fn) return cudaErrorInvalidValue;
    const dim3 grid((unsigned)a.g.ntiles * (unsigned)__builtin_popcount(a.tmask));
    if (!maps) {
        void *args[] = {const_cast<AxisArgs<C> *>(&a)};
        return cudaLaunchKernel(fn, grid, dim3(threads), args, smem, st);
    }
    if (wait <= 0) wait = kWaitCycles;
    void *args[] = {const_cast<AxisArgs<C> *>(&a), const_cast<CUtensorMap *>(maps), &err, &wait};
    return cudaLaunchKernel(fn, grid, dim3(threads), args, smem, st);
}

// Shared memory above the default 48 KB needs the attribute.
template <typename C, bool X> cudaError_t configure_axis_line_t(int n)
{
    for (int k = 0; k < 4; k++) {
        int threads = 0;
        const void *fn = axis_line_func<C, X>(n, k & 1, k & 2, &threads);
        cudaError_t e = fn ? cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) : cudaSuccess;
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

#define OPO_AXIS_LINE_INSTANCE(C, X)                                                                \
    template cudaError_t launch_axis_line_t<C, X>(const AxisArgs<C> &, bool, const CUtensorMap *, int *, long long, \
                                                  size_t, cudaStream_t);                            \
    template cudaError_t configure_axis_line_t<C, X>(int);

}  // namespace opo
