// Line-specialised x- and y-passes: the diffraction factor of one axis (reference
// Solver3D.cuh:282-301, 700-788) for an axis length whose radix plan is a compile-time
// constant, one field per tile.
//
// The generic axis tile (pass_body.cuh) holds all three fields of its lines: at 128 x 128 x
// 256 four CTAs of 128 threads fit an SM, and their first-stage loads, three fields one
// after the other, left the pass waiting on global memory (45 / 50 us for x / y in FP32,
// 99 / 102 us in FP64 against 31 / 62 us of HBM at the measured rate).  The diffraction
// factors do not couple the fields, so a tile here is L lines of one field: a third of the
// shared memory and one load phase per tile, 8 (FP32 x, 64 registers), 7 (FP32 y, 72) or 8
// (FP64, 64-thread CTAs at 128 registers) of them per SM whose phases overlap, every index and
// stride but the y-pass's row stride a constant (and that one too on square grids).  128 x 128 x
// 256, B200: FP32 x / y 39 / 40 us, FP64 70 / 79 us (5.7 / 5.1 TB/s); 256 x 256 x 512 FP32
// 350 / 387 -> 245 / 285 us.
//
// Stages of a tile, all threads on one stage at a time: the RA-point stage from global
// memory; with three radices the RB-point stage; the last radix's stage fused with the
// phase table and its inverse; back up; the inverse RA-point stage to global memory.  Items
// of x tiles run along the line (consecutive threads on consecutive elements), items of y
// tiles across the lines (consecutive threads on consecutive x).
//
// Shared memory: y tiles keep the global order (row of L elements per position, 128 bytes:
// no bank conflicts).  x tiles keep lines apart (stride LS) with one padding element after
// every RL = last-radix elements, so that the last stage's threads, RL + 1 elements apart,
// fall on different banks; LS is the stride with the fewest bank conflicts over the stages'
// access patterns, counted at compile time (axis_line_stride).
//
// Phase tables: position order g RL + k for y (a warp's threads share g: broadcast loads);
// x wants neighbouring g together, entry (g, k) at k (N / RL) + g -- in position order the
// table loads alone took 16 cache lines each and the FP32 x-pass 47 us instead of 37.
#pragma once

#include <type_traits>

#include "fft_radix.cuh"
#include "opo_internal.h"
#include "tma_copy.cuh"

namespace opo {

// Compiled axis lengths.
#define OPO_AXIS_LINES(X)                                                                          \
    X(16) X(24) X(32) X(36) X(48) X(64) X(72) X(96) X(108) X(128) X(144) X(192) X(216) X(256) X(384) X(512)

// Radix of stage 0, 1 or 2 of the body for n points (n = product; 1: no such stage; 0: no
// body).  Each is the fastest of the two- and three-stage orders tried per length on n x n
// grids; only 32 differs between the axes (x 4 x 8: a line's loads start 64 or 128
// contiguous bytes wide, FP32 43 against 54 us; y 8 x 4: 35 against 41 us).
__host__ __device__ constexpr int axis_line_radix(bool x, int n, int stage)
{
    const int v = n == 16    ? 40401
                  : n == 24  ? 40601
                  : n == 32  ? (x ? 40801 : 80401)
                  : n == 36  ? 90401
                  : n == 48  ? 60801
                  : n == 64  ? 80801
                  : n == 72  ? 90801
                  : n == 96  ? 120801
                  : n == 108 ? 91201
                  : n == 128 ? 160801
                  : n == 144 ? 121201
                  : n == 192 ? 161201
                  : n == 216 ? 90604
                  : n == 256 ? 161601
                  : n == 384 ? 80608
                  : n == 512 ? 80808
                             : 0;
    return stage == 0 ? v / 10000 : stage == 1 ? v / 100 % 100 : v % 100;
}

// Lines per tile.  y rows of L elements are 128 bytes (whole cache lines); long axes take
// half, so that several tiles still fit an SM.
__host__ __device__ constexpr int axis_line_lines(bool fp64, bool x, int n)
{
    return fp64 ? (x && n >= 216 ? 4 : 8) : (n >= 384 || n == 216 || (x && n == 256) ? 8 : 16);
}

// Square n x n grids with a body that runs x and y in one launch (axis_plane.cu).
__host__ __device__ constexpr bool axis_plane(bool fp64, int n) { return n <= (fp64 ? 72 : 64); }
// Whether it is the faster one on this many planes (fields times nt).  Up to 48 points always:
// us a z-step, one solver / three in turn, two launches -> one: 32 x 32 x 64 FP64 11.7 / 5.8 ->
// 10.3 / 5.2, 16 x 16 x 32 FP32 10.3 / 3.9 -> 9.0 / 3.3, 48 x 48 x 256 FP64 43.7 / 36.5 -> 42.1 /
// 31.7.  From 64 points on two planes per SM are needed (64 x 64 x 64 FP64 22.5 -> 23.9 alone;
// 64 x 64 x 128 40.0 / 28.8 -> 38.9 / 25.9), and in FP32, whose CTAs a plane's six stages keep
// longer than the x and y tiles, all planes resident at once, four per SM (64 x 64 x 128 25.0 /
// 16.3 -> 24.4 / 15.4; x 256 41.9 / 32.3 -> 43.5 / 31.2).  On 64 points and the nine time axes from
// 64 to 256 samples, alone: inside the rule FP32 gains 2-6 % (108 samples loses 6), FP64 -2 to +6;
// outside it 4-7 % are lost (96 samples, 288 planes, gains 3 and 9).  FP32 72 and 96 points: alone
// 5 and 9 % slower at 256 samples, no body.
inline bool axis_plane_pays(bool fp64, int n, unsigned planes)
{
    return axis_plane(fp64, n) && (n <= 48 || (planes >= 2 * 148 && (fp64 || planes <= 4 * 148)));
}

// Wavefronts of one shared-memory access of an x stage with nb butterflies per line, butterfly
// b of line l at element l ls + pos(b), consecutive threads on consecutive butterflies, for
// elements of which `banks` fill a wavefront (16 FP32, 8 FP64), over 16 wavefronts' threads.
template <typename P> __host__ __device__ constexpr int axis_line_waves(int ls, int nb, int banks, P pos)
{
    int total = 0;
    for (int w0 = 0; w0 < 16 * banks; w0 += banks) {
        int worst = 0;
        for (int i = 0; i < banks; i++) {
            int same = 0;
            const int bi = (w0 + i) / nb * ls + pos((w0 + i) % nb);
            for (int j = 0; j < banks; j++)
                same += ((w0 + j) / nb * ls + pos((w0 + j) % nb)) % banks == bi % banks;
            worst = same > worst ? same : worst;
        }
        total += worst;
    }
    return total;
}
// Line stride of an x tile: the least of PADN .. PADN + 15 with the fewest wavefronts.
__host__ __device__ constexpr int axis_line_stride(int n, int ra, int rb, int rc, int banks)
{
    const int q = n / ra, rl = rc > 1 ? rc : rb, padn = n + n / rl;
    int best = padn, cost = 1 << 30;
    for (int ls = padn; ls < padn + 16; ls++) {
        int c = axis_line_waves(ls, q, banks, [=](int b) { return b + b / rl; }) +
                axis_line_waves(ls, n / rl, banks, [=](int g) { return g * (rl + 1); });
        if (rc > 1) c += axis_line_waves(ls, n / rb, banks, [=](int b) {
            const int p = b / rc * q + b % rc;
            return p + p / rl;
        });
        if (c < cost) {
            cost = c;
            best = ls;
        }
    }
    return best;
}

template <typename C, bool X_, int N_> struct AxisLine {
    static constexpr bool X = X_;
    static constexpr int N = N_, RA = axis_line_radix(X, N, 0), RB = axis_line_radix(X, N, 1),
                         RC = axis_line_radix(X, N, 2);
    static constexpr bool F64 = sizeof(C) == 16;
    static constexpr int L = axis_line_lines(F64, X, N);
    static constexpr int Q = N / RA;              // butterflies of the first stage per line
    static constexpr int RL = RC > 1 ? RC : RB;   // radix of the last forward stage
    static constexpr int NG = N / RL;             // its butterflies per line
    static constexpr int LS = X ? axis_line_stride(N, RA, RB, RC, F64 ? 8 : 16) : 0;
    // TMA-fed tiles (axis_line_load): the raw stride of an x line, for which the first stage's
    // reads of consecutive elements fill whole wavefronts across lines
    static constexpr int NB = F64 ? 8 : 16;
    static constexpr int LSR = N + (Q % NB + NB - N % NB) % NB;
    static constexpr int BYTES = ((X ? L * (LS > LSR ? LS : LSR) : N * L) * (int)sizeof(C) + 127) / 128 * 128;
    // one first-stage item per thread up to 256 threads, then two
    static constexpr int ITEMS = Q * L;
    static constexpr int THREADS = ((ITEMS <= 256 ? ITEMS : (ITEMS + 1) / 2) + 31) / 32 * 32;
    // TMA-fed: one item per thread, and from 128 points on -- loads through registers hold their
    // bytes in flight in L1, which beside the t-pass's shared memory (three solvers in turn, the
    // SMs' split at its largest) is 28 KB: 128 x 128 x 256 FP32 15.0 -> 14.0 ms a round trip, FP64
    // 30.3 -> 27.7; alone, and below 128 points, the two are within 1-5 %, registers ahead.  (At 384
    // and 512 points only FP64 x has one item per thread.)
    static constexpr bool TMA = ITEMS <= THREADS && N >= 128;
    // Registers: FP32 80 (at 64 the radix-16 y-pass of ragged grids spills: 47 us against 39),
    // FP64 128 with a radix above 8, else 96.
    static constexpr int REGS = F64 ? (RA > 8 || RB > 8 ? 128 : 96) : X && RA == 16 && RB == 8 ? 64 : 80;
    static constexpr int MINB = 65536 / REGS / THREADS;
    __device__ __forceinline__ static constexpr int at(int l, int j) { return X ? l * LS + j + j / RL : j * L + l; }
    // item w of a stage with nb butterflies per line -> (line, butterfly)
    __device__ __forceinline__ static void item(int w, int nb, int &l, int &b)
    {
        if (X) {
            b = w % nb;
            l = w / nb;
        } else {
            b = w / L;
            l = w % L;
        }
    }
};

// Shared memory of one tile.
template <typename C, bool X> inline size_t axis_line_smem(int n)
{
    switch (n) {
#define OPO_CASE(N) case N: return AxisLine<C, X, N>::BYTES;
        OPO_AXIS_LINES(OPO_CASE)
#undef OPO_CASE
    default: return 0;
    }
}

// Whether the body for n points can be TMA-fed.
template <typename C, bool X> inline bool axis_line_tma(int n)
{
    switch (n) {
#define OPO_CASE(N) case N: return AxisLine<C, X, N>::TMA;
        OPO_AXIS_LINES(OPO_CASE)
#undef OPO_CASE
    default: return false;
    }
}

// One tile: lines [0, lim) of the L starting at fp (lim < L: the last tile of a row or
// field), row stride gs (elements; y: between positions, GS != 0 fixes it at compile time).
// Offsets within a tile are 32-bit byte counts.  A caller that reuses sm synchronises first.
template <typename C, typename G, int THREADS, unsigned GS, bool LOADED = false>
__device__ __forceinline__ void axis_line_tile(C *fp, unsigned lim, unsigned gs, const C *__restrict__ tab,
                                               const C *__restrict__ tw, C *sm)
{
    constexpr int RA = G::RA, RB = G::RB, RC = G::RC, Q = G::Q, RL = G::RL, NG = G::NG, L = G::L;
    // lines past lim load the last line's values and store nothing
    constexpr bool FULL = !G::X && GS % L == 0 && GS > 0;  // square grid of whole tiles
    const unsigned gsj = (G::X ? 1u : (GS ? GS : gs)) * (unsigned)sizeof(C), gsl = (G::X ? G::N : 1u) * (unsigned)sizeof(C);
    char *const gp = reinterpret_cast<char *>(fp);
    if constexpr (LOADED) {
        // first stage from the raw tile (x: lines LSR apart; y: in place)
        static_assert(G::ITEMS <= THREADS, "one item per thread");
        int l, b;
        G::item(min((int)threadIdx.x, G::ITEMS - 1), Q, l, b);
        C x[RA];
#pragma unroll
        for (int m = 0; m < RA; m++) x[m] = sm[G::X ? l * G::LSR + b + m * Q : (b + m * Q) * L + l];
        __syncthreads();  // x: the padded tile overlaps the raw one
        if (threadIdx.x < G::ITEMS) {
            dft<RA, -1>(x);
#pragma unroll
            for (int k = 1; k < RA; k++) x[k] = cmul(x[k], __ldg(tw + (k - 1) * Q + b));
#pragma unroll
            for (int k = 0; k < RA; k++) sm[G::at(l, b + k * Q)] = x[k];
        }
    } else
#pragma unroll 1
    for (int w = threadIdx.x; w < G::ITEMS; w += THREADS) {
        int l, b;
        G::item(w, Q, l, b);
        const unsigned o = (FULL ? (unsigned)l : min((unsigned)l, lim - 1)) * gsl + b * gsj;
        C x[RA];
#pragma unroll
        for (int m = 0; m < RA; m++) x[m] = *reinterpret_cast<const C *>(gp + (o + m * Q * gsj));
        dft<RA, -1>(x);
#pragma unroll
        for (int k = 1; k < RA; k++) x[k] = cmul(x[k], __ldg(tw + (k - 1) * Q + b));
#pragma unroll
        for (int k = 0; k < RA; k++) sm[G::at(l, b + k * Q)] = x[k];
    }
    __syncthreads();
    // middle stage of a three-radix plan, forward or inverse
    auto middle = [&](auto fwd) {
        constexpr bool F = decltype(fwd)::value;
        constexpr int NB = G::N / RB;
        const C *tw1 = tw + (RA - 1) * Q;
#pragma unroll 1
        for (int w = threadIdx.x; w < NB * L; w += THREADS) {
            int l, b;
            G::item(w, NB, l, b);
            const int j = b % RC, p0 = b / RC * Q + j;
            C x[RB];
#pragma unroll
            for (int m = 0; m < RB; m++) x[m] = sm[G::at(l, p0 + m * RC)];
            if constexpr (!F) {
#pragma unroll
                for (int m = 1; m < RB; m++) x[m] = cmulc(x[m], __ldg(tw1 + (m - 1) * RC + j));
            }
            dft<RB, F ? -1 : +1>(x);
            if constexpr (F) {
#pragma unroll
                for (int k = 1; k < RB; k++) x[k] = cmul(x[k], __ldg(tw1 + (k - 1) * RC + j));
            }
#pragma unroll
            for (int k = 0; k < RB; k++) sm[G::at(l, p0 + k * RC)] = x[k];
        }
        __syncthreads();
    };
    if constexpr (RC > 1) middle(std::true_type{});
#pragma unroll 1
    for (int w = threadIdx.x; w < NG * L; w += THREADS) {
        int l, g;
        G::item(w, NG, l, g);
        C x[RL];
#pragma unroll
        for (int m = 0; m < RL; m++) x[m] = sm[G::at(l, g * RL + m)];
        dft<RL, -1>(x);
        if constexpr (!G::X && !G::F64 && RL % 2 == 0) {
            const float4 *t2 = reinterpret_cast<const float4 *>(tab + g * RL);
#pragma unroll
            for (int k = 0; k < RL; k += 2) {
                const float4 t = __ldg(t2 + k / 2);
                x[k] = cmul(x[k], C{t.x, t.y});
                x[k + 1] = cmul(x[k + 1], C{t.z, t.w});
            }
        } else {
#pragma unroll
            for (int k = 0; k < RL; k++) x[k] = cmul(x[k], __ldg(G::X ? tab + k * NG + g : tab + g * RL + k));
        }
        dft<RL, +1>(x);
#pragma unroll
        for (int k = 0; k < RL; k++) sm[G::at(l, g * RL + k)] = x[k];
    }
    __syncthreads();
    if constexpr (RC > 1) middle(std::false_type{});
#pragma unroll 1
    for (int w = threadIdx.x; w < G::ITEMS; w += THREADS) {
        int l, b;
        G::item(w, Q, l, b);
        if (!FULL && (unsigned)l >= lim) continue;
        const unsigned o = l * gsl + b * gsj;
        C x[RA];
#pragma unroll
        for (int m = 0; m < RA; m++) x[m] = sm[G::at(l, b + m * Q)];
#pragma unroll
        for (int k = 1; k < RA; k++) x[k] = cmulc(x[k], __ldg(tw + (k - 1) * Q + b));
        dft<RA, +1>(x);
#pragma unroll
        for (int k = 0; k < RA; k++) *reinterpret_cast<C *>(gp + (o + k * Q * gsj)) = x[k];
    }
}

// Brings the raw tile into sm with the TMA: x one bulk copy per line, y one tensor box (L
// columns of N rows of the plane; columns past the grid read as zero).  Every thread returns
// when the tile has landed; false when the bounded wait (wait clock cycles) expired.
template <typename C, typename G>
__device__ __forceinline__ bool axis_line_load(const C *fp, unsigned lim, const CUtensorMap *map, int c0, int plane, C *sm,
                                               unsigned long long *bar, long long wait)
{
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const unsigned lines = min(lim, (unsigned)G::L);
    if (threadIdx.x < 32) {
        if (threadIdx.x == 0) mbar_arrive_expect_tx(bar, (G::X ? lines : (unsigned)G::L) * G::N * (unsigned)sizeof(C));
        __syncwarp();
        if constexpr (G::X) {
            if (threadIdx.x < lines)
                tma_bulk(sm + threadIdx.x * G::LSR, fp + threadIdx.x * G::N, G::N * (unsigned)sizeof(C), bar);
        } else {
            if (threadIdx.x == 0) tma_tensor_3d(sm, map, c0, 0, plane, bar);
        }
    }
    __syncthreads();  // the barrier is initialised
    return mbar_wait(bar, 0, wait);
}

// First element and line count of tile `tile` of a line-specialised pass.
__device__ __forceinline__ unsigned axis_line_base(const TileGeom &g, unsigned tile, unsigned extent, unsigned &lim)
{
    const unsigned hi = fdiv(g.tdiv, tile), lo = tile - hi * g.tdiv.d;
    lim = extent - lo * (unsigned)g.nlines;
    return lo * g.tmulA + hi * g.tmulB;
}

}  // namespace opo
