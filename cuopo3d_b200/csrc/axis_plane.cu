// The x and then the y diffraction factor of a square grid in one launch, a plane of one field
// per CTA (reference Solver3D.cuh:282-301, 700-788): the stages of the two line bodies
// (axis_line.cuh) one after the other on a plane that stays in shared memory, so that results
// equal the separate passes' bit for bit.
//
// Small grids are bound by the launches' latency and by the plane's way through L2 between the
// passes; here a z-step has two launches instead of three and one crossing of the field instead
// of two.  What is left is the chain of six stages with a barrier after each, which the CTAs of
// an SM overlap (64 points: 4 of 36 KB in FP32, 3 of 72 KB in FP64).  axis_plane_pays (axis_line.cuh) has the figures.
#include "axis_line.cuh"

namespace opo {

template <typename C, int N_> struct AxisPlane {
    static constexpr int N = N_;
    static constexpr bool F64 = sizeof(C) == 16;
    using GX = AxisLine<C, true, N>;
    using GY = AxisLine<C, false, N>;
    static_assert(GX::RC == 1 && GY::RC == 1, "two-stage plans");
    static constexpr int LS = GX::LS;  // the x body's rows: padded, few bank conflicts in x, none along a row
    static constexpr int BYTES = N * LS * (int)sizeof(C);
    static constexpr int ITEMS = N * N / (GX::RA < GX::RB ? GX::RA : GX::RB);  // of its longest x stage
    static constexpr int REGS = F64 ? (GX::RA > 8 || GX::RB > 8 ? 128 : 96) : 80;
    // an equal number of items for every thread of at most 256 (FP64 at 96 registers 192, three
    // CTAs per SM instead of two: 64 x 64 x 128 27.3 -> 25.9 us a step).  512 threads were slower
    // (32 / 62 -> 35 / 77 us a step of 64 x 64 x 256, FP32 / FP64), 128 within 5 % either way
    static constexpr int CAP = REGS == 96 ? 192 : 256;
    static constexpr int PER = (ITEMS + CAP - 1) / CAP;
    static constexpr int THREADS = ((ITEMS + PER - 1) / PER + 31) / 32 * 32;
    static constexpr int MINB = 65536 / REGS / THREADS;
    __device__ __forceinline__ static constexpr int at(int row, int col) { return row * LS + col + col / GX::RL; }
};

// One axis of the plane in sm: x reads its first stage from global memory, y stores its last.
template <typename C, typename P, typename G>
__device__ __forceinline__ void axis_plane_axis(C *gp, const C *__restrict__ tab, const C *__restrict__ tw, C *sm)
{
    constexpr int N = G::N, RA = G::RA, Q = G::Q, RL = G::RL, NG = G::NG;
    auto at = [](int line, int j) { return G::X ? P::at(line, j) : P::at(j, line); };
    auto item = [](int w, int nb, int &line, int &b) {
        line = G::X ? w / nb : w % N;
        b = G::X ? w % nb : w / N;
    };
#pragma unroll 1
    for (int w = threadIdx.x; w < Q * N; w += P::THREADS) {
        int l, b;
        item(w, Q, l, b);
        C x[RA];
#pragma unroll
        for (int m = 0; m < RA; m++) x[m] = G::X ? gp[l * N + b + m * Q] : sm[at(l, b + m * Q)];
        dft<RA, -1>(x);
#pragma unroll
        for (int k = 1; k < RA; k++) x[k] = cmul(x[k], __ldg(tw + (k - 1) * Q + b));
#pragma unroll
        for (int k = 0; k < RA; k++) sm[at(l, b + k * Q)] = x[k];
    }
    __syncthreads();
#pragma unroll 1
    for (int w = threadIdx.x; w < NG * N; w += P::THREADS) {
        int l, g;
        item(w, NG, l, g);
        C x[RL];
#pragma unroll
        for (int m = 0; m < RL; m++) x[m] = sm[at(l, g * RL + m)];
        dft<RL, -1>(x);
#pragma unroll
        for (int k = 0; k < RL; k++) x[k] = cmul(x[k], __ldg(G::X ? tab + k * NG + g : tab + g * RL + k));
        dft<RL, +1>(x);
#pragma unroll
        for (int k = 0; k < RL; k++) sm[at(l, g * RL + k)] = x[k];
    }
    __syncthreads();
#pragma unroll 1
    for (int w = threadIdx.x; w < Q * N; w += P::THREADS) {
        int l, b;
        item(w, Q, l, b);
        C x[RA];
#pragma unroll
        for (int m = 0; m < RA; m++) x[m] = sm[at(l, b + m * Q)];
#pragma unroll
        for (int k = 1; k < RA; k++) x[k] = cmulc(x[k], __ldg(tw + (k - 1) * Q + b));
        dft<RA, +1>(x);
#pragma unroll
        for (int k = 0; k < RA; k++) {
            if (G::X)
                sm[at(l, b + k * Q)] = x[k];
            else
                gp[(b + k * Q) * N + l] = x[k];
        }
    }
    if (G::X) __syncthreads();
}

// CTA u of a launch: plane u mod nt of the (u / nt)-th field of the mask.
template <typename C, typename P>
__global__ void __launch_bounds__(P::THREADS, P::MINB) axis_plane_kernel(AxisPlaneArgs<C> a)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    C *sm = reinterpret_cast<C *>(smem_raw);
    unsigned fi = 0, t = blockIdx.x;
    while (t >= a.nt) {
        t -= a.nt;
        fi++;
    }
    unsigned m = a.tmask;
    while (fi--) m &= m - 1;
    const int f = (m & 1u) ? 0 : (m & 2u) ? 1 : 2;
    C *gp = (f == 0 ? a.f[0] : f == 1 ? a.f[1] : a.f[2]) + (size_t)t * (P::N * P::N);
    axis_plane_axis<C, P, typename P::GX>(gp, f == 0 ? a.tabx[0] : f == 1 ? a.tabx[1] : a.tabx[2], a.twx, sm);
    axis_plane_axis<C, P, typename P::GY>(gp, f == 0 ? a.taby[0] : f == 1 ? a.taby[1] : a.taby[2], a.twy, sm);
}

template <typename C> static const void *axis_plane_func(int n, int *threads, size_t *smem)
{
    switch (n) {
#define OPO_CASE(N)                                                                                 \
    case N:                                                                                         \
        if constexpr (axis_plane(sizeof(C) == 16, N)) {                                             \
            *threads = AxisPlane<C, N>::THREADS;                                                    \
            *smem = AxisPlane<C, N>::BYTES;                                                         \
            return reinterpret_cast<const void *>(axis_plane_kernel<C, AxisPlane<C, N>>);           \
        }                                                                                           \
        return nullptr;
        OPO_AXIS_LINES(OPO_CASE)
#undef OPO_CASE
    default: return nullptr;
    }
}

template <typename C> cudaError_t launch_axis_plane(const AxisPlaneArgs<C> &a, int n, cudaStream_t st)
{
    int threads = 0;
    size_t smem = 0;
    const void *fn = axis_plane_func<C>(n, &threads, &smem);
    if (!fn) return cudaErrorInvalidValue;
    void *args[] = {const_cast<AxisPlaneArgs<C> *>(&a)};
    return cudaLaunchKernel(fn, dim3(a.nt * (unsigned)__builtin_popcount(a.tmask)), dim3(threads), args, smem, st);
}

template <typename C> cudaError_t configure_axis_plane(int n)
{
    int threads = 0;
    size_t smem = 0;
    const void *fn = axis_plane_func<C>(n, &threads, &smem);
    if (!fn || smem <= 48 * 1024) return cudaSuccess;
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
}

template cudaError_t launch_axis_plane<float2>(const AxisPlaneArgs<float2> &, int, cudaStream_t);
template cudaError_t launch_axis_plane<double2>(const AxisPlaneArgs<double2> &, int, cudaStream_t);
template cudaError_t configure_axis_plane<float2>(int);
template cudaError_t configure_axis_plane<double2>(int);

}  // namespace opo
