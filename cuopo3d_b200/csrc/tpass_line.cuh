// Line-specialised t-pass: the tile body of tpass_tile / tpass_tile_split for a time
// axis whose length and radix plan are compile-time constants, in FP32 and FP64.
//
// It computes what the generic t-pass computes (reference Solver3D.cuh:872-943 RK4 half
// steps, then Solver3D.cuh:572-639 dispersion: transform, phase, inverse transform) on
// tiles of 16-byte units: PP units per time sample, one time sample per shared-memory
// row.  A unit is one FP64 pixel, or in FP32 a split pair: the same time sample of
// pixels l and l + 1, real parts in one packed f32x2 register pair and imaginary parts
// in another, in registers and in shared memory (re_l, re_l+1, im_l, im_l+1).  Every FP32
// butterfly, twiddle and phase product then serves two lines with one packed instruction
// per component (a complex product: 4 packed instructions for two values; multiplying by
// +-i only renames registers), each twiddle and phase factor is loaded once for both
// lines, and all index arithmetic is compile-time.  The pixels of a tile are consecutive in
// the (x, y) plane, whatever nx; the plane holds whole tiles.  The transforms are two-stage plans [RA, RB] up to 256
// samples and three-stage plans [RA, RB, RC] beyond (decimation in frequency forward, in
// time inverse, phase tables in the plan's digit-reversed order), so the twiddles and
// phase tables are the host's tables of that plan.
//
// Shapes (tpass_line_shape): PP and the CTA size give each stage about one item per thread of
// half or a third of a CTA (two or three (stage, field) jobs run at a time) and 12-24 warps
// per SM beside tiles of 20-110 KB.  The pass is bound by its arithmetic pipes and shared
// memory together (128 x 128 x 256: FP32 FMA pipe 61 %, FP64 pipe 65 % busy): 512 samples took
// 167-170 us in FP32 with 16, 24 or 32 warps per SM, 256 samples were slower with three jobs
// (76 against 70 us, register spills) or radix 8 throughout (80 us); three jobs won by 9 % on
// 64 x 64 x 128 in FP32 (18.4 -> 16.8 us) and by 1-4 % at 384 and 512.
//
// Shared memory per field: NT rows of PP units.  With PP < 8 the last stage's threads, RL
// rows apart, would share banks: two-stage bodies put a padding row after every RL rows,
// three-stage ones (whose tiles leave no room) put time sample t in row t ^ (t / RL mod 8 / PP),
// a permutation inside each group of RL rows (at 256 samples the permutation's index
// arithmetic cost 4 %: FP32 73.7 against 70.7 us).  The first stage's twiddles are staged with
// the tile, after the three field regions (shared-memory latency instead of L1 for the
// twiddle loads of a first- and last-stage item; the other tables stay in global memory).
#pragma once

#include "pass_body.cuh"

namespace opo {

struct X2C {
    f32x2 r, i;
};

// Packed FP32 arithmetic with explicit rounding (no contraction left to the compiler):
// the single-instance and batched kernels that share this body compute bit-identical
// results.
__device__ __forceinline__ f32x2 xr_add(f32x2 a, f32x2 b)
{
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 xr_sub(f32x2 a, f32x2 b)
{
    f32x2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 xr_mul(f32x2 a, f32x2 b)
{
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 xr_fma(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

__device__ __forceinline__ X2C xadd(X2C a, X2C b) { return X2C{xr_add(a.r, b.r), xr_add(a.i, b.i)}; }
__device__ __forceinline__ X2C xsub(X2C a, X2C b) { return X2C{xr_sub(a.r, b.r), xr_sub(a.i, b.i)}; }
// a (c + i s) and a (c - i s); ns = -s
__device__ __forceinline__ X2C xmul(X2C a, f32x2 c, f32x2 s, f32x2 ns)
{
    return X2C{xr_fma(a.i, ns, xr_mul(a.r, c)), xr_fma(a.r, s, xr_mul(a.i, c))};
}
__device__ __forceinline__ X2C xmulc(X2C a, f32x2 c, f32x2 s, f32x2 ns)
{
    return X2C{xr_fma(a.i, s, xr_mul(a.r, c)), xr_fma(a.r, ns, xr_mul(a.i, c))};
}
// a (c + S i s) for constants c, s
template <int S> __device__ __forceinline__ X2C xrot(X2C a, float c, float s)
{
    const f32x2 C = x2_dup(c), P = x2_dup(s), N = x2_dup(-s);
    return S > 0 ? xmul(a, C, P, N) : xmulc(a, C, P, N);
}
// a times a table entry t = c + i s: a t (CONJ: a conj(t))
template <bool CONJ> __device__ __forceinline__ X2C xmul_tab(X2C a, float2 t)
{
    const f32x2 c = x2_dup(t.x), s = x2_dup(t.y);
    const f32x2 ns = xr_sub(0ull, s);
    return CONJ ? xmulc(a, c, s, ns) : xmul(a, c, s, ns);
}

// DFT4 of sign S; ROT2: the third input enters multiplied by S i (folded into the sums).
template <int S, bool ROT2 = false> __device__ __forceinline__ void xdft4(X2C &x0, X2C &x1, X2C &x2, X2C &x3)
{
    X2C t0, t1;
    if (!ROT2) {
        t0 = xadd(x0, x2);
        t1 = xsub(x0, x2);
    } else if (S > 0) {  // x2 i = (-x2.i, x2.r)
        t0 = X2C{xr_sub(x0.r, x2.i), xr_add(x0.i, x2.r)};
        t1 = X2C{xr_add(x0.r, x2.i), xr_sub(x0.i, x2.r)};
    } else {  // x2 (-i) = (x2.i, -x2.r)
        t0 = X2C{xr_add(x0.r, x2.i), xr_sub(x0.i, x2.r)};
        t1 = X2C{xr_sub(x0.r, x2.i), xr_add(x0.i, x2.r)};
    }
    const X2C t2 = xadd(x1, x3), d = xsub(x1, x3);
    x0 = xadd(t0, t2);
    x2 = xsub(t0, t2);
    // t3 = d (S i): x1 = t1 + t3, x3 = t1 - t3
    if (S > 0) {
        x1 = X2C{xr_sub(t1.r, d.i), xr_add(t1.i, d.r)};
        x3 = X2C{xr_add(t1.r, d.i), xr_sub(t1.i, d.r)};
    } else {
        x1 = X2C{xr_add(t1.r, d.i), xr_sub(t1.i, d.r)};
        x3 = X2C{xr_sub(t1.r, d.i), xr_add(t1.i, d.r)};
    }
}

template <int R, int S> struct XDft;

template <int S> struct XDft<2, S> {
    __device__ __forceinline__ static void run(X2C *x)
    {
        const X2C t = x[0];
        x[0] = xadd(t, x[1]);
        x[1] = xsub(t, x[1]);
    }
};

template <int S> struct XDft<3, S> {
    __device__ __forceinline__ static void run(X2C *x)
    {
        const f32x2 h = x2_dup(-0.5f), s3 = x2_dup(S * Roots<float>::s3), n3 = x2_dup(-S * Roots<float>::s3);
        const X2C t = xadd(x[1], x[2]), d = xsub(x[1], x[2]);
        const X2C m{xr_fma(t.r, h, x[0].r), xr_fma(t.i, h, x[0].i)};
        x[0] = xadd(x[0], t);
        x[1] = X2C{xr_fma(d.i, n3, m.r), xr_fma(d.r, s3, m.i)};  // m + S i s3 d
        x[2] = X2C{xr_fma(d.i, s3, m.r), xr_fma(d.r, n3, m.i)};
    }
};

template <int S> struct XDft<4, S> {
    __device__ __forceinline__ static void run(X2C *x) { xdft4<S>(x[0], x[1], x[2], x[3]); }
};

// 6 = 2 x 3 and 12 = 4 x 3 by the prime-factor map (dft_3xm)
template <int M, int S> __device__ __forceinline__ void xdft_3xm(X2C *x)
{
    constexpr int N = 3 * M, E = M == 4 ? 9 : 3;
    X2C y[N];
#pragma unroll
    for (int n2 = 0; n2 < M; n2++) {
        X2C t[3] = {x[3 * n2 % N], x[(M + 3 * n2) % N], x[(2 * M + 3 * n2) % N]};
        XDft<3, S>::run(t);
        y[n2] = t[0];
        y[M + n2] = t[1];
        y[2 * M + n2] = t[2];
    }
#pragma unroll
    for (int k1 = 0; k1 < 3; k1++) {
        XDft<M, S>::run(y + M * k1);
#pragma unroll
        for (int k2 = 0; k2 < M; k2++) x[(4 * k1 + E * k2) % N] = y[M * k1 + k2];
    }
}
template <int S> struct XDft<6, S> {
    __device__ __forceinline__ static void run(X2C *x) { xdft_3xm<2, S>(x); }
};
template <int S> struct XDft<12, S> {
    __device__ __forceinline__ static void run(X2C *x) { xdft_3xm<4, S>(x); }
};

// 9 = 3 x 3 as Dft<9>
template <int S> struct XDft<9, S> {
    __device__ __forceinline__ static void run(X2C *x)
    {
        using K = Roots<float>;
        X2C u[3][3];
#pragma unroll
        for (int m = 0; m < 3; m++) {
            X2C t[3] = {x[m], x[m + 3], x[m + 6]};
            XDft<3, S>::run(t);
            u[0][m] = t[0];
            u[1][m] = t[1];
            u[2][m] = t[2];
        }
        u[1][1] = xrot<S>(u[1][1], K::c9, K::s9);
        u[1][2] = xrot<S>(u[1][2], K::c9_2, K::s9_2);
        u[2][1] = xrot<S>(u[2][1], K::c9_2, K::s9_2);
        u[2][2] = xrot<S>(u[2][2], K::c9_4, K::s9_4);
#pragma unroll
        for (int r = 0; r < 3; r++) {
            XDft<3, S>::run(u[r]);
#pragma unroll
            for (int k = 0; k < 3; k++) x[3 * k + r] = u[r][k];
        }
    }
};

// 8 = 2 x 4: a_m = x_m + x_{m+4}, b_m = (x_m - x_{m+4}) W8^m, y_{2k} = DFT4(a), y_{2k+1} = DFT4(b)
template <int S> struct XDft<8, S> {
    __device__ __forceinline__ static void run(X2C *x)
    {
        const float r2 = Roots<float>::r2;
        X2C a0 = xadd(x[0], x[4]), a1 = xadd(x[1], x[5]), a2 = xadd(x[2], x[6]), a3 = xadd(x[3], x[7]);
        X2C b0 = xsub(x[0], x[4]);
        X2C b1 = xrot<S>(xsub(x[1], x[5]), r2, r2);
        X2C b2 = xsub(x[2], x[6]);  // enters DFT4(b) times S i
        X2C b3 = xrot<S>(xsub(x[3], x[7]), -r2, r2);
        xdft4<S>(a0, a1, a2, a3);
        xdft4<S, true>(b0, b1, b2, b3);
        x[0] = a0; x[2] = a1; x[4] = a2; x[6] = a3;
        x[1] = b0; x[3] = b1; x[5] = b2; x[7] = b3;
    }
};

// 16 = 4 x 4: u_{m,r} = DFT4_j(x_{m+4j})_r, u_{m,r} *= W16^{m r}, y_{4k+r} = DFT4_m(u_{m,r})_k
template <int S> struct XDft<16, S> {
    __device__ __forceinline__ static void run(X2C *x)
    {
        const float r2 = Roots<float>::r2, c8 = Roots<float>::c8, s8 = Roots<float>::s8;
#pragma unroll
        for (int m = 0; m < 4; m++) xdft4<S>(x[m], x[m + 4], x[m + 8], x[m + 12]);
        x[1 + 4 * 1] = xrot<S>(x[1 + 4 * 1], c8, s8);    // W^1
        x[1 + 4 * 2] = xrot<S>(x[1 + 4 * 2], r2, r2);    // W^2
        x[1 + 4 * 3] = xrot<S>(x[1 + 4 * 3], s8, c8);    // W^3
        x[2 + 4 * 1] = xrot<S>(x[2 + 4 * 1], r2, r2);    // W^2
        // x[2 + 4 * 2] times W^4 = S i: folded into its DFT4 below
        x[2 + 4 * 3] = xrot<S>(x[2 + 4 * 3], -r2, r2);   // W^6
        x[3 + 4 * 1] = xrot<S>(x[3 + 4 * 1], s8, c8);    // W^3
        x[3 + 4 * 2] = xrot<S>(x[3 + 4 * 2], -r2, r2);   // W^6
        x[3 + 4 * 3] = xrot<S>(x[3 + 4 * 3], -c8, -s8);  // W^9
        xdft4<S>(x[0], x[1], x[2], x[3]);
        xdft4<S>(x[4], x[5], x[6], x[7]);
        xdft4<S, true>(x[8], x[9], x[10], x[11]);
        xdft4<S>(x[12], x[13], x[14], x[15]);
        // x[4 r + k] = y_{4 k + r}: transpose the 4 x 4 block (register renaming)
        X2C t;
        t = x[1]; x[1] = x[4]; x[4] = t;
        t = x[2]; x[2] = x[8]; x[8] = t;
        t = x[3]; x[3] = x[12]; x[12] = t;
        t = x[6]; x[6] = x[9]; x[9] = t;
        t = x[7]; x[7] = x[13]; x[13] = t;
        t = x[11]; x[11] = x[14]; x[14] = t;
    }
};

template <int R, int S> __device__ __forceinline__ void xdft(X2C *x) { XDft<R, S>::run(x); }

__device__ __forceinline__ X2C split_of(float4 q)
{
    return X2C{f2pack(float2{q.x, q.z}), f2pack(float2{q.y, q.w})};
}
__device__ __forceinline__ float4 interleaved_of(X2C v)
{
    const float2 re = f2unpack(v.r), im = f2unpack(v.i);
    return make_float4(re.x, im.x, re.y, im.y);
}

// The 16-byte unit of each precision: its register form, loads and stores of the raw
// layout (the global one, C values interleaved: staged tiles and the fields), the
// butterflies, table products and the coupled-wave half steps.
template <typename C> struct LineUnit;

template <> struct LineUnit<float2> {
    using U = X2C;
    static constexpr int PX = 2;  // pixels per unit
    __device__ __forceinline__ static U lds(const void *p)
    {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(p);
        return X2C{v.x, v.y};
    }
    __device__ __forceinline__ static void sts(void *p, U v) { *reinterpret_cast<ulonglong2 *>(p) = make_ulonglong2(v.r, v.i); }
    __device__ __forceinline__ static U load_raw(const void *p) { return split_of(*reinterpret_cast<const float4 *>(p)); }
    __device__ __forceinline__ static void store_raw(void *p, U v) { *reinterpret_cast<float4 *>(p) = interleaved_of(v); }
    template <int R, int S> __device__ __forceinline__ static void dft(U *x) { xdft<R, S>(x); }
    // x t (CONJ: x conj(t)) for a table entry t
    template <bool CONJ> __device__ __forceinline__ static U tmul(U x, float2 t) { return xmul_tab<CONJ>(x, t); }
    __device__ __forceinline__ static U zero() { return X2C{0ull, 0ull}; }
    // n half steps of every voxel of the units p, s, i
    __device__ __forceinline__ static void rk4(const TPassArgs<float2> &a, U &p, U &s, U &i)
    {
        f32x2 v[3][2] = {{p.r, p.i}, {s.r, s.i}, {i.r, i.i}};
        for (int h = 0; h < a.n_rk4; h++) rk4_half_x2(a, h, v[0], v[1], v[2]);
        p = X2C{v[0][0], v[0][1]};
        s = X2C{v[1][0], v[1][1]};
        i = X2C{v[2][0], v[2][1]};
    }
};

template <> struct LineUnit<double2> {
    using U = double2;
    static constexpr int PX = 1;
    __device__ __forceinline__ static U lds(const void *p) { return *reinterpret_cast<const double2 *>(p); }
    __device__ __forceinline__ static void sts(void *p, U v) { *reinterpret_cast<double2 *>(p) = v; }
    __device__ __forceinline__ static U load_raw(const void *p) { return *reinterpret_cast<const double2 *>(p); }
    __device__ __forceinline__ static void store_raw(void *p, U v) { *reinterpret_cast<double2 *>(p) = v; }
    template <int R, int S> __device__ __forceinline__ static void dft(U *x) { opo::dft<R, S>(x); }
    template <bool CONJ> __device__ __forceinline__ static U tmul(U x, double2 t) { return CONJ ? cmulc(x, t) : cmul(x, t); }
    __device__ __forceinline__ static U zero() { return double2{0.0, 0.0}; }
    __device__ __forceinline__ static void rk4(const TPassArgs<double2> &a, U &p, U &s, U &i)
    {
        if (a.use_phase) {
            for (int h = 0; h < a.n_rk4; h++) rk4_half_step<true>(a, h, p, s, i);
        } else {
            for (int h = 0; h < a.n_rk4; h++) rk4_half_step<false>(a, h, p, s, i);
        }
    }
};

template <typename C, int NT_> struct LineGeom {
    static constexpr int NT = NT_;
    static constexpr LineShape S = tpass_line_shape(sizeof(C) == 16, NT);
    static constexpr int RA = S.ra, RB = S.rb, RC = S.rc, PP = S.pp, THREADS = S.threads, MINB = S.ctas, JOBS = S.jobs;
    static constexpr int PX = LineUnit<C>::PX;
    static constexpr int P = PP * PX;            // pixels per tile
    static constexpr int Q = NT / RA;            // butterflies per line of the first stage
    static constexpr int RL = RC > 1 ? RC : RB;  // radix of the last forward stage
    static constexpr int NG = NT / RL;           // its butterflies per line
    static constexpr bool PAD = PP == 4 && RC == 1;
    static constexpr int MASK = !PAD && PP < 8 ? 8 / PP - 1 : 0;
    static constexpr int REGION = (NT + (PAD ? NG : 0)) * PP * 16;  // bytes per field region
    static constexpr int A = PP * Q;             // first-stage items per field
    static constexpr int B = PP * (NT / RB);     // middle-stage items (three radices)
    static constexpr int LAST = PP * NG;         // last-stage items
    static constexpr int NTW = (RA - 1) * Q;     // first-stage twiddles, staged after the tile
    static constexpr int TILE_BYTES = 3 * REGION;
    static constexpr size_t tile_bytes() { return (size_t)TILE_BYTES + (size_t)NTW * sizeof(C); }
    static_assert(RL % (MASK + 1) == 0, "rows permute inside a group");
    // shared-memory row of sample g RL + k, and byte offset of (row, unit) in a field region
    __device__ __forceinline__ static constexpr int row(int g, int k) { return PAD ? g * (RL + 1) + k : g * RL + (k ^ (g & MASK)); }
    __device__ __forceinline__ static constexpr int off(int row, int u) { return (row * PP + u) * 16; }
};

// Issue the cp.async copies of a tile (the fields in lmask) into buffer buf.
template <typename C, typename G>
__device__ __forceinline__ void line_stage_in(const TPassArgs<C> &a, unsigned base, unsigned lmask, unsigned char *buf)
{
    const unsigned gs = a.g.gs_j;
    const C *src[3] = {a.psrc, a.f[1], a.f[2]};
#pragma unroll
    for (int f = 0; f < 3; f++) {
        if (!(lmask & (1u << f))) continue;
        const C *gsrc = src[f] + base;
        for (unsigned e = threadIdx.x; e < G::NT * G::PP; e += G::THREADS) {
            const int t = (int)(e / G::PP), u = (int)(e % G::PP);
            cp_async<16>(buf + f * G::REGION + G::off(G::row(t / G::RL, t % G::RL), u),
                         gsrc + (size_t)t * gs + u * G::PX);
        }
    }
}

// Sweep over the staged tile: half steps and EOM per unit, two units per thread at a time
// (items e and e + THREADS: two independent chains to interleave); transformed fields go
// back to shared memory as units, the others (loaded, not transformed) to global memory.
template <typename C, typename G>
__device__ __forceinline__ void line_sweep(const TPassArgs<C> &a, unsigned base, unsigned lmask, unsigned tmask, unsigned char *buf)
{
    using L = LineUnit<C>;
    using U = typename L::U;
    constexpr unsigned THREADS = G::THREADS;
    const unsigned gs = a.g.gs_j;
    auto at = [&](int f, unsigned e) {
        const int t = (int)(e / G::PP), u = (int)(e % G::PP);
        return buf + f * G::REGION + G::off(G::row(t / G::RL, t % G::RL), u);
    };
    auto load = [&](unsigned e, U (&v)[3]) {
#pragma unroll
        for (int f = 0; f < 3; f++) v[f] = (lmask & (1u << f)) ? L::load_raw(at(f, e)) : L::zero();
    };
    auto finish = [&](unsigned e, U (&v)[3]) {
        const int t = (int)(e / G::PP), u = (int)(e % G::PP);
        if (a.eom) {
            const C ev = __ldg(a.eom + t);
            v[1] = L::template tmul<false>(v[1], ev);
            v[2] = L::template tmul<false>(v[2], ev);
        }
#pragma unroll
        for (int f = 0; f < 3; f++) {
            if (tmask & (1u << f))
                L::sts(at(f, e), v[f]);
            else if (lmask & (1u << f))
                L::store_raw(a.f[f] + base + (unsigned)t * gs + u * G::PX, v[f]);
        }
    };
    constexpr unsigned NI = G::NT * G::PP;
    constexpr unsigned PER = 65536 / (G::THREADS * G::MINB) > 100 ? 2 : 1;
    for (unsigned e = threadIdx.x; e < NI; e += PER * THREADS) {
        const bool two = PER == 2 && e + THREADS < NI;
        U v0[3], v1[3];
        load(e, v0);
        if (two) load(e + THREADS, v1);
        L::rk4(a, v0[0], v0[1], v0[2]);
        if (two) L::rk4(a, v1[0], v1[1], v1[2]);
        finish(e, v0);
        if (two) finish(e + THREADS, v1);
    }
}

// Row of first-stage value m of butterfly j (sample j + Q m).  Q is a multiple of RL: the
// group is j / RL + (Q / RL) m; with two stages j < Q = RL and the group is m.
template <typename G> __device__ __forceinline__ int line_row_a(int j, int m)
{
    if constexpr (G::RC == 1) return G::row(m, j);
    return G::row(j / G::RL + G::Q / G::RL * m, j % G::RL);
}

// Item w of a field in the forward first stage (stride Q): butterfly, then the twiddles
// W_NT^{j k}.
template <typename C, typename G>
__device__ __forceinline__ void line_stage_a(const unsigned char *tws_, unsigned char *buf, unsigned w)
{
    using L = LineUnit<C>;
    constexpr int Q = G::Q, RA = G::RA;
    const int u = (int)(w % G::PP), j = (int)(w / G::PP);
    typename L::U x[RA];
#pragma unroll
    for (int m = 0; m < RA; m++) x[m] = L::lds(buf + G::off(line_row_a<G>(j, m), u));
    L::template dft<RA, +1>(x);
    const C *tws = reinterpret_cast<const C *>(tws_);
#pragma unroll
    for (int k = 1; k < RA; k++) x[k] = L::template tmul<true>(x[k], tws[(k - 1) * Q + j]);
#pragma unroll
    for (int k = 0; k < RA; k++) L::sts(buf + G::off(line_row_a<G>(j, k), u), x[k]);
}

// Item w of a field in the middle stage of a three-radix plan (stride RC inside blocks of
// Q samples), forward or inverse.
template <typename C, typename G, bool FWD>
__device__ __forceinline__ void line_stage_m(const C *tw1, unsigned char *buf, unsigned w)
{
    using L = LineUnit<C>;
    constexpr int RB = G::RB, RC = G::RC;
    const int u = (int)(w % G::PP), b = (int)(w / G::PP), blk = b / RC, j = b % RC;
    typename L::U x[RB];
#pragma unroll
    for (int m = 0; m < RB; m++) x[m] = L::lds(buf + G::off(G::row(blk * RB + m, j), u));
    if constexpr (!FWD) {
#pragma unroll
        for (int m = 1; m < RB; m++) x[m] = L::template tmul<false>(x[m], __ldg(tw1 + (m - 1) * RC + j));
    }
    L::template dft<RB, FWD ? +1 : -1>(x);
    if constexpr (FWD) {
#pragma unroll
        for (int k = 1; k < RB; k++) x[k] = L::template tmul<true>(x[k], __ldg(tw1 + (k - 1) * RC + j));
    }
#pragma unroll
    for (int k = 0; k < RB; k++) L::sts(buf + G::off(G::row(blk * RB + k, j), u), x[k]);
}

// Item w of a field in the last forward stage: butterfly, phase table, inverse butterfly.
template <typename C, typename G>
__device__ __forceinline__ void line_stage_b(const C *tab, unsigned char *buf, unsigned w)
{
    using L = LineUnit<C>;
    constexpr int RL = G::RL;
    const int u = (int)(w % G::PP), g = (int)(w / G::PP);
    const C *tb = tab + RL * g;
    typename L::U x[RL];
#pragma unroll
    for (int m = 0; m < RL; m++) x[m] = L::lds(buf + G::off(G::row(g, m), u));
    L::template dft<RL, +1>(x);
    if constexpr (sizeof(C) == 8) {
        // two FP32 table entries per 16-byte load (tb is 16-byte aligned: RL g even)
#pragma unroll
        for (int k = 0; k < RL; k += 2) {
            const float4 t2 = __ldg(reinterpret_cast<const float4 *>(tb + k));
            x[k] = L::template tmul<false>(x[k], C{t2.x, t2.y});
            x[k + 1] = L::template tmul<false>(x[k + 1], C{t2.z, t2.w});
        }
    } else {
#pragma unroll
        for (int k = 0; k < RL; k++) x[k] = L::template tmul<false>(x[k], __ldg(tb + k));
    }
    L::template dft<RL, -1>(x);
#pragma unroll
    for (int k = 0; k < RL; k++) L::sts(buf + G::off(G::row(g, k), u), x[k]);
}

// Item w of a field in the inverse first stage (twiddles before the butterfly), written to
// global memory.
template <typename C, typename G>
__device__ __forceinline__ void line_stage_c(const unsigned char *tws_, const unsigned char *buf, C *dst, unsigned w, unsigned gs)
{
    using L = LineUnit<C>;
    constexpr int Q = G::Q, RA = G::RA;
    const int u = (int)(w % G::PP), j = (int)(w / G::PP);
    typename L::U x[RA];
#pragma unroll
    for (int m = 0; m < RA; m++) x[m] = L::lds(buf + G::off(line_row_a<G>(j, m), u));
    const C *tws = reinterpret_cast<const C *>(tws_);
#pragma unroll
    for (int m = 1; m < RA; m++) x[m] = L::template tmul<false>(x[m], tws[(m - 1) * Q + j]);
    L::template dft<RA, -1>(x);
    C *d = dst + (unsigned)j * gs + u * G::PX;
#pragma unroll
    for (int k = 0; k < RA; k++) L::store_raw(d + (size_t)(Q * k) * gs, x[k]);
}

// The transform stages of every field in tmask as jobs (stage, field) in stage-major
// order, two or three jobs per phase (PER; an equal share of the CTA each; one job when one
// field is transformed) and a CTA barrier between phases.  A job's stage of a field always
// ran in an earlier phase (nf >= PER jobs apart).
template <typename C, typename G, int BAR, int PER>
__device__ __forceinline__ void line_jobs(const TPassArgs<C> &a, unsigned base, unsigned tmask, unsigned nf, unsigned char *buf)
{
    constexpr unsigned GROUP = G::THREADS / PER, STAGES = G::RC > 1 ? 5 : 3;
    static_assert(GROUP % 32 == 0, "a warp runs one job");
    const unsigned gs = a.g.gs_j, njobs = STAGES * nf;
    const unsigned slot = threadIdx.x / GROUP, w0 = threadIdx.x % GROUP;
    const unsigned char *tws = buf + G::TILE_BYTES;
    for (unsigned j0 = 0; j0 < njobs; j0 += PER) {
        const unsigned j = j0 + slot;
        if (j < njobs) {
            // stage j / nf and field j % nf for nf = 1, 2, 3 (j < 15: j / 3 = (11 j) >> 5)
            const unsigned stage = nf == 1 ? j : (nf == 2 ? j >> 1 : (11 * j) >> 5);
            const int f = field_id(tmask, (int)(j - stage * nf));
            unsigned char *fb = buf + f * G::REGION;
            if (stage == 0) {
                for (unsigned w = w0; w < G::A; w += GROUP) line_stage_a<C, G>(tws, fb, w);
            } else if (stage == STAGES - 1) {
                for (unsigned w = w0; w < G::A; w += GROUP) line_stage_c<C, G>(tws, fb, a.f[f] + base, w, gs);
            } else if (G::RC == 1 || stage == 2) {
                for (unsigned w = w0; w < G::LAST; w += GROUP) line_stage_b<C, G>(a.tab[f], fb, w);
            } else if constexpr (G::RC > 1) {
                const C *tw1 = a.tw + G::NTW;
                if (stage == 1)
                    for (unsigned w = w0; w < G::B; w += GROUP) line_stage_m<C, G, true>(tw1, fb, w);
                else
                    for (unsigned w = w0; w < G::B; w += GROUP) line_stage_m<C, G, false>(tw1, fb, w);
            }
        }
        tile_sync<BAR>();
    }
}

// One tile: the fields in the load mask staged with cp.async, the sweep, then per
// transformed field the transform stages, the last one written to global memory.  Ends
// with the CTA synchronised.
template <typename C, typename G, int BAR = 0>
__device__ __forceinline__ void tpass_line_tile(const TPassArgs<C> &a, unsigned tile, unsigned char *buf)
{
    const unsigned base = tile * (unsigned)G::P;
    const unsigned tmask = a.tmask, lmask = tpass_load_mask(a);
    line_stage_in<C, G>(a, base, lmask, buf);
    {  // the first stage's twiddles
        C *tws = reinterpret_cast<C *>(buf + G::TILE_BYTES);
        for (int e = threadIdx.x; e < G::NTW; e += G::THREADS) cp_async<sizeof(C)>(tws + e, a.tw + e);
    }
    cp_async_wait_all();
    tile_sync<BAR>();
    line_sweep<C, G>(a, base, lmask, tmask, buf);
    tile_sync<BAR>();
    if (!tmask) return;
    const unsigned nf = __popc(tmask);
    if (G::JOBS == 3 && nf == 3)
        line_jobs<C, G, BAR, G::JOBS>(a, base, tmask, nf, buf);
    else if (nf >= 2)
        line_jobs<C, G, BAR, 2>(a, base, tmask, nf, buf);
    else
        line_jobs<C, G, BAR, 1>(a, base, tmask, nf, buf);
}

}  // namespace opo
