// Kernels and launchers of the line-specialised t-pass (tile body in tpass_line.cuh) for one
// precision: included by tpass_line_32.cu and tpass_line_64.cu, which compile in parallel.
//  * tpass_line_kernel: one CTA per tile;
//  * tpass_line_batch_kernel: one CTA per tile of every instance of a batch whose time axis has
//    the body (each body a kernel of its own: one kernel holding every body and the
//    generic one needed 168 registers and spilled; a persistent form, whose CTAs walked the
//    tiles, took 377 instead of 335 us for 19.4 M voxels of 256 samples in FP32);
//  * tpass_line_fallback_kernel: the generic tile body at the line setting's CTA size and
//    radix, for grids without a line body.
#pragma once

#include "batch_device.cuh"
#include "tpass_line.cuh"

namespace opo {

template <typename C, int NT>
__global__ void __launch_bounds__(LineGeom<C, NT>::THREADS, LineGeom<C, NT>::MINB) tpass_line_kernel(TPassArgs<C> a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    tpass_line_tile<C, LineGeom<C, NT>>(a, blockIdx.x, smem_raw);
}

template <typename C, int NT>
__global__ void __launch_bounds__(LineGeom<C, NT>::THREADS, LineGeom<C, NT>::MINB)
    tpass_line_batch_kernel(const TPassArgs<C> *descs, const unsigned *prefix, const BatchHeader *hdr, int tp)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TPassArgs<C> *d = reinterpret_cast<TPassArgs<C> *>(smem_raw);
    unsigned char *buf = smem_raw + desc_bytes<TPassArgs<C>>();
    const unsigned gt = blockIdx.x;
    if (gt >= hdr->total_tiles) return;
    descs += hdr->first;
    prefix += hdr->pfirst;
    const int i = find_inst(prefix, hdr->ninst, gt);
    stage_desc(descs + i, d);
    __syncthreads();
    if (d->ph_steps) {
        if (threadIdx.x < 6) d->ph[threadIdx.x / 3][threadIdx.x % 3] = d->ph_steps[tp * 6 + threadIdx.x];
        __syncthreads();
    }
    tpass_line_tile<C, LineGeom<C, NT>>(*d, gt - __ldg(prefix + i), buf);
}

template <typename C, int R1, int THREADS>
__global__ void __launch_bounds__(THREADS, 4) tpass_line_fallback_kernel(TPassArgs<C> a)
{
    constexpr int RMAX = LineFallback<C, THREADS>::RMAX;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C *sm = reinterpret_cast<C *>(smem_raw);
    const C *src[3] = {a.psrc, a.f[1], a.f[2]};
    const unsigned lmask = tpass_load_mask(a);
    for (unsigned tile = blockIdx.x; tile < (unsigned)a.g.ntiles; tile += gridDim.x) {
        stage_tile<C, THREADS, false>(a.g, (unsigned)a.plan.n, tile, src, lmask, sm);
        tpass_tile<C, R1, THREADS, RMAX, true>(a, tile, sm);
    }
}

// Single-instance or batched kernel of line body nt, or null.
template <typename C> const void *tpass_line_func(int nt, bool batch)
{
    switch (nt) {
#define OPO_CASE(NT)                                                                                \
    case NT:                                                                                        \
        return batch ? reinterpret_cast<const void *>(tpass_line_batch_kernel<C, NT>)                \
                     : reinterpret_cast<const void *>(tpass_line_kernel<C, NT>);
        OPO_TPASS_LINE_SETTINGS(OPO_CASE)
        OPO_TPASS_LINES(OPO_CASE)
#undef OPO_CASE
    default: return nullptr;
    }
}
template <typename C> const void *tpass_line_batch_func(int nt) { return tpass_line_func<C>(nt, true); }

// Fallback radices: FP32 4, 8 and 16, FP64 4.
template <typename C> const void *tpass_fallback_func(int r)
{
    if (r == 4) return reinterpret_cast<const void *>(tpass_line_fallback_kernel<C, 4, 128>);
    if constexpr (sizeof(C) == 8) {
        if (r == 8) return reinterpret_cast<const void *>(tpass_line_fallback_kernel<C, 8, 128>);
        if (r == 16) return reinterpret_cast<const void *>(tpass_line_fallback_kernel<C, 16, 128>);
    }
    return nullptr;
}

// A tile and its twiddles (the units are 16 bytes in both precisions; the twiddles are C).
template <typename C> size_t tpass_line_smem(int nt)
{
    switch (nt) {
#define OPO_CASE(NT) case NT: return LineGeom<C, NT>::tile_bytes();
        OPO_TPASS_LINE_SETTINGS(OPO_CASE)
        OPO_TPASS_LINES(OPO_CASE)
#undef OPO_CASE
    default: return 0;
    }
}

template <typename C> cudaError_t configure_line_kernels(int nt, size_t smem)
{
    if (nt) return cudaFuncSetAttribute(tpass_line_func<C>(nt, false), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    for (int r : {4, 8, 16})
        if (const void *fn = tpass_fallback_func<C>(r)) {
            cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return e;
        }
    return cudaSuccess;
}

template <typename C> cudaError_t launch_tpass_line(const TPassArgs<C> &a, int nt, int grid, size_t smem, cudaStream_t st)
{
    const void *fn = tpass_line_func<C>(nt, false);
    if (!fn) return cudaErrorInvalidValue;
    void *args[] = {const_cast<TPassArgs<C> *>(&a)};
    return cudaLaunchKernel(fn, dim3(grid), dim3(tpass_line_shape(sizeof(C) == 16, nt).threads), args, smem, st);
}

template <typename C>
cudaError_t launch_tpass_line_fallback(const TPassArgs<C> &a, PassVariant v, int r_fallback, int grid, size_t smem,
                                       cudaStream_t st)
{
    const void *fn = v.threads == 128 ? tpass_fallback_func<C>(r_fallback) : nullptr;
    if (!fn) return cudaErrorInvalidValue;
    void *args[] = {const_cast<TPassArgs<C> *>(&a)};
    return cudaLaunchKernel(fn, dim3(grid), dim3(v.threads), args, smem, st);
}

#define OPO_TPASS_LINE_INSTANCE(C)                                                                  \
    template const void *tpass_line_batch_func<C>(int);                                             \
    template size_t tpass_line_smem<C>(int);                                                        \
    template cudaError_t configure_line_kernels<C>(int, size_t);                                    \
    template cudaError_t launch_tpass_line<C>(const TPassArgs<C> &, int, int, size_t, cudaStream_t); \
    template cudaError_t launch_tpass_line_fallback<C>(const TPassArgs<C> &, PassVariant, int, int, size_t, cudaStream_t);

}  // namespace opo
