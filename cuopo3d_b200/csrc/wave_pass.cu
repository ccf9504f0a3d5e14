// Plane-wave (1 x 1) solver: all z-steps of a crystal pass or cavity round trip in one launch.
//
// Without diffraction a time line never meets another one, and with one line a t-pass is
// one CTA: 4096 FP64 samples cost 13 us a step, the FP64 pipe of a single SM, and a
// launch per step.  Here a thread-block cluster of K CTAs (1, 4, 8 or 16) holds the line of
// all three fields in its shared memory from the first half step to the last
// (reference Solver1D.cuh / Solver3D.cuh:946-997: RK4, dispersion, RK4, ..., EOM, GDD and
// mirrors).  The transform's plan starts with radices of product K:
//   * CTA r holds the samples t = m M + r M / K + b (M = n / K, m < K, b < M / K): the coupled-
//     wave half steps are pointwise, and the first K-fold stages act on m alone -- local;
//   * their outputs for m are block m of M spectrum positions: each CTA stores them straight
//     into CTA m's block buffer (distributed shared memory); one cluster barrier;
//   * CTA r transforms its block (the plan's remaining stages, phase table, inverse) and
//     stores the result back to the owners of the samples; a second cluster barrier.
// Two cluster barriers a step order everything: a CTA's block buffer is last read before
// the second barrier and written again after it, its sample buffer is last read before the
// first barrier and written by its peers after it.
// B200, a round trip of 100 steps with EOM and GDD on 4096 FP64 samples: 3.83 -> 0.83 ms, three
// solvers in turn 1.31 -> 0.28 ms each; 256 FP32 samples 0.69 -> 0.43 ms.
//
// The barriers are the hardware's cluster barriers; no CTA leaves before the last one.

#include "pass_body.cuh"
#include "wave_pass.h"

namespace opo {

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ unsigned cluster_rank()
{
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// Generic address of p (this CTA's shared memory) in CTA `rank` of the cluster.
template <typename T> __device__ __forceinline__ T *peer(T *p, unsigned rank)
{
    unsigned long long r;
    asm("mapa.u64 %0, %1, %2;" : "=l"(r) : "l"(p), "r"(rank));
    return reinterpret_cast<T *>(r);
}

// Butterflies of sample-buffer stage (radix R, nb blocks) of the fields in mask: element
// m of butterfly (blk, a, b) at row blk R sub + a + m sub, sub = K / (nb R).  FWD with
// dst != null: output k of the last such stage goes to position `pos` + b of CTA (row)'s
// block buffer.
template <typename C, int R, bool FWD>
__device__ __forceinline__ void sample_stage(const WaveArgs<C> &w, C *X, C *blockbuf, int s, int nb, unsigned rank, unsigned mask,
                                             bool last)
{
    const unsigned bw = w.bw, K = w.K, sub = K / (nb * R), per = nb * sub * bw, nf = __popc(mask), q = sub * w.M;
    const C *tw = w.tw + w.plan.twoff[s];
    for (unsigned u = threadIdx.x; u < nf * per; u += kThreads) {
        const unsigned fi = (u >= per) + (u >= 2 * per), v = u - fi * per;
        const int f = field_id(mask, (int)fi);
        const unsigned c = v / bw, b = v - c * bw, blk = c / sub, a = c - blk * sub;
        const unsigned j = a * w.M + rank * bw + b, row0 = blk * R * sub + a;
        C *x0 = X + f * w.xregion + b;
        C x[R];
#pragma unroll
        for (int m = 0; m < R; m++) x[m] = x0[(row0 + m * sub) * bw];
        if constexpr (!FWD) {
#pragma unroll
            for (int m = 1; m < R; m++) x[m] = cmul(x[m], __ldg(tw + (m - 1) * q + j));
        }
        dft<R, FWD ? +1 : -1>(x);
        if constexpr (FWD) {
#pragma unroll
            for (int k = 1; k < R; k++) x[k] = cmulc(x[k], __ldg(tw + (k - 1) * q + j));
        }
        if (FWD && last) {
            C *y = blockbuf + f * w.g.region + prow(w.g, rank * bw + b);
#pragma unroll
            for (int k = 0; k < R; k++) *peer(y, row0 + k * sub) = x[k];
        } else {
#pragma unroll
            for (int k = 0; k < R; k++) x0[(row0 + k * sub) * bw] = x[k];
        }
    }
}

// Transform, table `tab` of this CTA's block, inverse transform of the fields in mask.
template <typename C, bool CL>
__device__ __forceinline__ void line_transform(const WaveArgs<C> &w, C *X, C *Y, unsigned rank, const C *const *tab, unsigned mask)
{
    const AxisPlan &p = w.plan;
    const int s0 = w.nsample;  // sample-buffer stages
    if constexpr (CL) {
        if (w.K == 8) {
            sample_stage<C, 8, true>(w, X, Y, 0, 1, rank, mask, true);
        } else {
            sample_stage<C, 4, true>(w, X, Y, 0, 1, rank, mask, w.K == 4);
            if (w.K == 16) {
                __syncthreads();
                sample_stage<C, 4, true>(w, X, Y, 1, 4, rank, mask, true);
            }
        }
        cluster_sync();
    }
    const C *tb[3] = {tab[0] + rank * w.M, tab[1] + rank * w.M, tab[2] + rank * w.M};
    for (int s = s0; s < p.ns - 1; s++) {
        smem_stage_dispatch<C, +1, false, kThreads, 8, true>(p.radix[s], Y, w.g, (int)w.M, p.len[s], p.q[s],
                                                             w.tw + p.twoff[s], mask);
        __syncthreads();
    }
    fused_dispatch<C, +1, kThreads, 8, true>(p.radix[p.ns - 1], Y, w.g, (int)w.M, tb, mask);
    __syncthreads();
    for (int s = p.ns - 2; s >= s0; s--) {
        smem_stage_dispatch<C, -1, true, kThreads, 8, true>(p.radix[s], Y, w.g, (int)w.M, p.len[s], p.q[s],
                                                            w.tw + p.twoff[s], mask);
        __syncthreads();
    }
    if constexpr (CL) {
        const unsigned bw = w.bw;
        for (unsigned fb = mask; fb; fb &= fb - 1) {
            const int f = __ffs(fb) - 1;
            for (unsigned j = threadIdx.x; j < w.M; j += kThreads) {
                const unsigned c = j / bw;
                *peer(X + f * w.xregion + rank * bw + (j - c * bw), c) = Y[f * w.g.region + prow(w.g, j)];
            }
        }
        cluster_sync();
        if (w.K == 8) {
            sample_stage<C, 8, false>(w, X, Y, 0, 1, rank, mask, false);
        } else {
            if (w.K == 16) {
                sample_stage<C, 4, false>(w, X, Y, 1, 4, rank, mask, false);
                __syncthreads();
            }
            sample_stage<C, 4, false>(w, X, Y, 0, 1, rank, mask, false);
        }
        __syncthreads();
    }
}

template <typename C, bool CL> __global__ void __launch_bounds__(kThreads, 1) wave_kernel(const __grid_constant__ WaveArgs<C> w)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(16) unsigned char phased_raw[sizeof(TPassArgs<C>)];
    TPassArgs<C> &phased = *reinterpret_cast<TPassArgs<C> *>(phased_raw);  // w.rk with this t-pass's phases
    C *Y = reinterpret_cast<C *>(smem_raw);
    C *X = CL ? Y + 3 * w.g.region : Y;
    const unsigned rank = CL ? cluster_rank() : 0u;
    const TPassArgs<C> &a = w.rk;
    const unsigned ns = CL ? w.K * w.bw : w.M;  // samples of this CTA
    // sample i: its time index, and its place in a field's region of the sample buffer
    auto time_of = [&](unsigned i) { return CL ? i / w.bw * w.M + rank * w.bw + i % w.bw : i; };
    auto at = [&](int f, unsigned i) -> C & { return CL ? X[f * w.xregion + i] : Y[f * w.g.region + prow(w.g, i)]; };
    for (unsigned i = threadIdx.x; i < ns; i += kThreads) {
        const unsigned t = time_of(i);
        at(0, i) = a.psrc[t];
        at(1, i) = a.f[1][t];
        at(2, i) = a.f[2][t];
    }
    if (a.use_phase)
        for (unsigned k = threadIdx.x; k < sizeof(a) / 4; k += kThreads)
            reinterpret_cast<unsigned *>(&phased)[k] = reinterpret_cast<const unsigned *>(&a)[k];
    if constexpr (CL) cluster_sync();  // every CTA of the cluster runs before the first remote store
    __syncthreads();
    for (int tp = 0; tp <= w.n_steps; tp++) {
        const bool close = tp == w.n_steps;
        const int halves = tp == 0 || close ? 1 : 2;
        if (a.use_phase) {
            if (threadIdx.x < 6) phased.ph[threadIdx.x / 3][threadIdx.x % 3] = w.ph_steps[tp * 6 + threadIdx.x];
            __syncthreads();
        }
        for (unsigned i = threadIdx.x; i < ns; i += kThreads) {
            C p = at(0, i), s = at(1, i), d = at(2, i);
            for (int h = 0; h < halves; h++) {
                if (a.use_phase) rk4_half_step<true>(phased, h, p, s, d);
                else rk4_half_step<false>(a, h, p, s, d);
            }
            if (close && w.closing && w.eom) {
                const C e = __ldg(w.eom + time_of(i));
                s = cmul(s, e);
                d = cmul(d, e);
            }
            at(0, i) = p;
            at(1, i) = s;
            at(2, i) = d;
        }
        __syncthreads();
        const unsigned mask = close ? (w.closing ? w.close_mask : 0u) : w.mask;
        if (mask) line_transform<C, CL>(w, X, Y, rank, w.tab[close ? 1 : 0], mask);
    }
    for (unsigned i = threadIdx.x; i < ns; i += kThreads) {
        const unsigned t = time_of(i);
#pragma unroll
        for (int f = 0; f < 3; f++) a.f[f][t] = at(f, i);
    }
}

}  // namespace

template <typename C> cudaError_t configure_wave_kernels()
{
    cudaError_t e = cudaFuncSetAttribute(wave_kernel<C, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(wave_kernel<C, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(wave_kernel<C, true>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}

namespace {
template <typename C> cudaLaunchConfig_t wave_config(int K, size_t smem, cudaStream_t st, cudaLaunchAttribute *attr)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(K);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = K;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = K > 1 ? 1 : 0;
    return cfg;
}
}  // namespace

template <typename C> bool wave_fits(int K, size_t smem)
{
    if (smem > 220 * 1024) return false;
    if (K == 1) return true;
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = wave_config<C>(K, smem, nullptr, &attr);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, wave_kernel<C, true>, &cfg) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    return n >= 1;
}

template <typename C> cudaError_t launch_wave(const WaveArgs<C> &w, size_t smem, cudaStream_t st)
{
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = wave_config<C>((int)w.K, smem, st, &attr);
    return w.K > 1 ? cudaLaunchKernelEx(&cfg, wave_kernel<C, true>, w) : cudaLaunchKernelEx(&cfg, wave_kernel<C, false>, w);
}

#define OPO_WAVE(C)                                                     \
    template cudaError_t configure_wave_kernels<C>();                   \
    template bool wave_fits<C>(int, size_t);                            \
    template cudaError_t launch_wave<C>(const WaveArgs<C> &, size_t, cudaStream_t);
OPO_WAVE(float2)
OPO_WAVE(double2)

}  // namespace opo
