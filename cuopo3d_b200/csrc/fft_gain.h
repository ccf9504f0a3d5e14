// Gain compensation of the transform pairs (host code, shared by the solver's table builder
// and the host-side checks in tests/native/gain_check.cu and gain64_check.cu).
//
// The FP32 kernels' roots of unity -- the butterflies' constants (fft_radix.cuh) and the
// stage twiddles, computed in FP64 and rounded -- have |W|^2 - 1 of a few 1e-8, mostly
// negative, so forward transform -> phase table -> inverse transform is not exactly
// norm-preserving: it drains ~2e-8 of the energy per pass, coherently, every split step
// (about 5e-6 of the energy per 100-step round trip and pass kind).  Every input-output
// pair of a Cooley-Tukey network is joined by one chain of butterflies, so the squared
// row norms r_p of the forward operator and the squared column norms c_p of the inverse
// follow from running the network on squared magnitudes: r = |F|^2 1, c = (|F_inv|^2)^T 1.
// A pair with exact constants has r_p = c_p = n; a phase table scaled by n / sqrt(r_p c_p)
// at spectrum position p gives the pair the energy gain of the table itself for white
// inputs, which removes the coherent drain.  What remains is the arithmetic's own
// rounding.
//
// FP64 likewise, a factor 2^29 smaller: the double nearest cos(pi/4) is 1 + 6.8e-17 of it, so
// a pair of radices 8 x 8 multiplies amplitudes by 1 + 6.5e-17 on average where 4 x 4 x 4 leaves
// 1 + 3e-18, in phase at every step: 1.5e-14 of the power over 120 steps.  The factors are held
// and applied to the table entries in extended precision; the entries' own rounding to FP64
// is as large but differs in sign from entry to entry.
#pragma once

#include "fft_radix.cuh"
#include "opo_internal.h"

#include <cmath>
#include <complex>
#include <vector>

namespace opo {

// |B_km|^2 of the radix-R butterfly as the FP32 kernels compute it: dft<R> run on float2
// unit vectors, whose outputs are exactly the FP32 constants (sums of them, for radix 3).
template <int R> inline void butterfly_sq(std::vector<double> &b2)
{
    b2.assign((size_t)R * R, 0.0);
    for (int m = 0; m < R; m++) {
        float2 x[R];
        for (int k = 0; k < R; k++) x[k] = make_float2(k == m ? 1.f : 0.f, 0.f);
        dft<R, +1>(x);
        for (int k = 0; k < R; k++) b2[(size_t)k * R + m] = (double)x[k].x * x[k].x + (double)x[k].y * x[k].y;
    }
}

// Per position of the digit-reversed spectrum: n / sqrt(r_p c_p) for plan pl, whose
// FP64 stage twiddles tw (AxisPlan layout) the kernels get rounded to FP32.
inline std::vector<double> fp32_pair_compensation(const AxisPlan &pl, const std::vector<std::complex<double>> &tw)
{
    const int n = pl.n;
    std::vector<double> r(n, 1.0), c(n, 1.0), nx(n);
    std::vector<double> b2[17];
    butterfly_sq<2>(b2[2]);
    butterfly_sq<3>(b2[3]);
    butterfly_sq<4>(b2[4]);
    butterfly_sq<6>(b2[6]);
    butterfly_sq<8>(b2[8]);
    butterfly_sq<9>(b2[9]);
    butterfly_sq<12>(b2[12]);
    butterfly_sq<16>(b2[16]);
    auto w2 = [&](int s, int k, int j) {
        if (k == 0) return 1.0;
        const std::complex<double> w = tw[(size_t)pl.twoff[s] + (size_t)(k - 1) * (pl.len[s] / pl.radix[s]) + j];
        const double a = (double)(float)w.real(), b = (double)(float)w.imag();
        return a * a + b * b;
    };
    // forward (decimation in frequency): butterfly, then the twiddle of output k
    for (int s = 0; s < pl.ns; s++) {
        const int R = pl.radix[s], L = pl.len[s], q = L / R;
        const std::vector<double> &B = b2[R];
        for (int g0 = 0; g0 < n; g0 += L)
            for (int j = 0; j < q; j++)
                for (int k = 0; k < R; k++) {
                    double v = 0;
                    for (int m = 0; m < R; m++) v += B[(size_t)k * R + m] * r[g0 + m * q + j];
                    nx[g0 + k * q + j] = v * w2(s, k, j);
                }
        r.swap(nx);
    }
    // inverse (decimation in time, stages last to first: twiddle of input m, then the
    // butterfly); its column norms come from the transposed network, stages first to last
    for (int s = 0; s < pl.ns; s++) {
        const int R = pl.radix[s], L = pl.len[s], q = L / R;
        const std::vector<double> &B = b2[R];
        for (int g0 = 0; g0 < n; g0 += L)
            for (int j = 0; j < q; j++)
                for (int m = 0; m < R; m++) {
                    double v = 0;
                    for (int k = 0; k < R; k++) v += B[(size_t)k * R + m] * c[g0 + k * q + j];
                    nx[g0 + m * q + j] = v * w2(s, m, j);
                }
        c.swap(nx);
    }
    std::vector<double> comp(n);
    for (int p = 0; p < n; p++) comp[p] = n / std::sqrt(r[p] * c[p]);
    return comp;
}

// Mean over the inputs m of output k, and over the outputs of input m, of |B_km|^2 - 1 for the
// radix-R butterfly as the FP64 kernels compute it.
struct ButterflyDeviation {
    std::vector<double> row, col;
};
template <int R> inline ButterflyDeviation butterfly_deviation()
{
    ButterflyDeviation d{std::vector<double>(R, 0.0), std::vector<double>(R, 0.0)};
    auto dev = [](double a, double b) { return (double)((long double)a * a + (long double)b * b - 1); };
    using K = Roots<double>;
    for (int m = 0; m < R; m++) {
        double2 x[R];
        for (int k = 0; k < R; k++) x[k] = make_double2(k == m ? 1.0 : 0.0, 0.0);
        dft<R, +1>(x);
        for (int k = 0; k < R; k++) {
            double v;
            if (R != 9) {
                v = dev(x[k].x, x[k].y);  // constants, unrounded
            } else {
                // two 3-point butterflies and a root W9^(m1 r) between them: the constants' product
                const int m1 = m % 3, r = k % 3, w = m1 * r;
                const double d3 = dev(0.5, K::s3);
                v = (r && m / 3 ? d3 : 0.0) + (m1 && k / 3 ? d3 : 0.0) +
                    (w == 1 ? dev(K::c9, K::s9) : w == 2 ? dev(K::c9_2, K::s9_2) : w == 4 ? dev(K::c9_4, K::s9_4) : 0.0);
            }
            d.row[k] += v / R;
            d.col[m] += v / R;
        }
    }
    return d;
}

// The FP64 factors minus 1, from the roots of unity as the FP64 kernels hold them: r_p and
// c_p are n (1 + O(1e-16)), so the network runs on the deviations to first order.
inline std::vector<double> fp64_pair_deviation(const AxisPlan &pl, const std::vector<std::complex<double>> &tw)
{
    static const std::vector<ButterflyDeviation> devs = [] {
        std::vector<ButterflyDeviation> d(17);
        d[2] = butterfly_deviation<2>();
        d[3] = butterfly_deviation<3>();
        d[4] = butterfly_deviation<4>();
        d[6] = butterfly_deviation<6>();
        d[8] = butterfly_deviation<8>();
        d[9] = butterfly_deviation<9>();
        d[12] = butterfly_deviation<12>();
        d[16] = butterfly_deviation<16>();
        return d;
    }();
    const int n = pl.n;
    std::vector<double> r(n, 0.0), c(n, 0.0);
    for (int s = 0; s < pl.ns; s++) {
        const int R = pl.radix[s], L = pl.len[s], q = L / R;
        const ButterflyDeviation &B = devs[R];
        for (int g0 = 0; g0 < n; g0 += L)
            for (int j = 0; j < q; j++) {
                double rm = 0, cm = 0;
                for (int m = 0; m < R; m++) {
                    rm += r[g0 + m * q + j];
                    cm += c[g0 + m * q + j];
                }
                for (int k = 0; k < R; k++) {
                    double w = 0;
                    if (k) {
                        const std::complex<double> &t = tw[(size_t)pl.twoff[s] + (size_t)(k - 1) * q + j];
                        w = (double)((long double)t.real() * t.real() + (long double)t.imag() * t.imag() - 1);
                    }
                    r[g0 + k * q + j] = rm / R + B.row[k] + w;
                    c[g0 + k * q + j] = cm / R + B.col[k] + w;
                }
            }
    }
    for (int p = 0; p < n; p++) r[p] = -0.5 * (r[p] + c[p]);
    return r;
}

// Factors of the phase table's entries for the kernels of one precision.
inline std::vector<long double> pair_compensation(bool fp64, const AxisPlan &pl, const std::vector<std::complex<double>> &tw)
{
    std::vector<long double> f(pl.n);
    const std::vector<double> v = fp64 ? fp64_pair_deviation(pl, tw) : fp32_pair_compensation(pl, tw);
    for (int p = 0; p < pl.n; p++) f[p] = fp64 ? 1.0L + v[p] : (long double)v[p];
    return f;
}

inline void scale_table(std::vector<std::complex<long double>> &tab, const std::vector<long double> &comp)
{
    for (size_t k = 0; k < tab.size(); k++) tab[k] *= comp[k];
}

}  // namespace opo
