// Host-side check of the FP64 transform-pair gain compensation (cuopo3d_b200/csrc/fft_gain.h),
// compiled and run by tests/test_fp64_gain.py; no GPU needed.
//
// For each plan of the line and plane-wave kernels the forward and inverse transforms are built as
// dense operators in extended precision with the FP64 kernels' constants: the squared row
// and column norms must give fp64_pair_deviation, to the extended arithmetic's rounding.  Then the power gain of the pair for white inputs with tables
// rounded to FP64 as the solver rounds them, averaged over random phase tables.  An entry's
// components are each off by at most 2^-53 of themselves, uniformly: its squared modulus by
// 2 x 2^-53 / sqrt(3) = 1.28e-16 r.m.s. at most, the mean over T tables of n entries by that /
// sqrt(T n); the bound is five times it.
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdio>
#include <random>
#include <vector>

#include "../../cuopo3d_b200/csrc/fft_gain.h"

using cd = std::complex<double>;
using cl = std::complex<long double>;

static const double kPi = 3.14159265358979323846;

static opo::AxisPlan make_plan(const std::vector<int> &rad, std::vector<cd> &tw)
{
    opo::AxisPlan p{};
    int n = 1;
    for (int r : rad) n *= r;
    p.n = n;
    p.ns = (int)rad.size();
    int L = n;
    for (int s = 0; s < p.ns; s++) {
        const int R = rad[s], q = L / R;
        p.radix[s] = R;
        p.len[s] = L;
        p.twoff[s] = (int)tw.size();
        for (int k = 1; k < R; k++)
            for (int j = 0; j < q; j++) tw.push_back(std::polar(1.0, -2 * kPi * (double)j * k / L));
        L = q;
    }
    return p;
}

// The 2- to 16-point butterflies of fft_radix.cuh in extended arithmetic with FP64 constants.
static void dft3(cl *x, int S)
{
    const long double s3 = opo::Roots<double>::s3;
    const cl t = x[1] + x[2], d = x[1] - x[2], m = x[0] - 0.5L * t, e(-S * s3 * d.imag(), S * s3 * d.real());
    x[0] += t;
    x[1] = m + e;
    x[2] = m - e;
}
static void dft4(cl *x, int S)
{
    const cl a = x[0] + x[2], b = x[0] - x[2], c = x[1] + x[3], d = x[1] - x[3], e(-S * d.imag(), S * d.real());
    x[0] = a + c;
    x[1] = b + e;
    x[2] = a - c;
    x[3] = b - e;
}
static void butterfly(int R, int S, cl *x)
{
    using K = opo::Roots<double>;
    auto w = [&](double c, double s) { return cl(c, S * (long double)s); };
    if (R == 2) {
        const cl t = x[0];
        x[0] = t + x[1];
        x[1] = t - x[1];
    } else if (R == 3) {
        dft3(x, S);
    } else if (R == 4) {
        dft4(x, S);
    } else if (R == 6 || R == 12) {
        const int M = R / 3;
        cl y[12];
        for (int n2 = 0; n2 < M; n2++) {
            cl t[3];
            for (int n1 = 0; n1 < 3; n1++) t[n1] = x[(3 * n2 + M * n1) % R];
            dft3(t, S);
            for (int k1 = 0; k1 < 3; k1++) y[k1 * M + n2] = t[k1];
        }
        for (int k1 = 0; k1 < 3; k1++) {
            butterfly(M, S, y + k1 * M);
            for (int k = 0; k < R; k++)
                if (k % 3 == k1) x[k] = y[k1 * M + k % M];
        }
    } else if (R == 8) {
        cl a[4], b[4];
        for (int m = 0; m < 4; m++) {
            a[m] = x[m] + x[m + 4];
            b[m] = x[m] - x[m + 4];
        }
        b[1] *= w(K::r2, K::r2);
        b[2] = cl(-S * b[2].imag(), S * b[2].real());
        b[3] *= w(-K::r2, K::r2);
        dft4(a, S);
        dft4(b, S);
        for (int k = 0; k < 4; k++) {
            x[2 * k] = a[k];
            x[2 * k + 1] = b[k];
        }
    } else {  // 9 = 3 x 3, 16 = 4 x 4
        const int Q = R == 9 ? 3 : 4;
        cl u[4][4];
        for (int m = 0; m < Q; m++) {
            cl t[4];
            for (int j = 0; j < Q; j++) t[j] = x[m + Q * j];
            butterfly(Q, S, t);
            for (int r = 0; r < Q; r++) {
                const int e = m * r;
                cl f(1, 0);
                if (R == 9) f = e == 1 ? w(K::c9, K::s9) : e == 2 ? w(K::c9_2, K::s9_2) : e == 4 ? w(K::c9_4, K::s9_4) : f;
                else
                    f = e == 1 ? w(K::c8, K::s8) : e == 2 ? w(K::r2, K::r2) : e == 3 ? w(K::s8, K::c8) : e == 4 ? w(0, 1)
                        : e == 6 ? w(-K::r2, K::r2) : e == 9 ? w(-K::c8, -K::s8) : f;
                u[r][m] = t[r] * f;
            }
        }
        for (int r = 0; r < Q; r++) {
            butterfly(Q, S, u[r]);
            for (int k = 0; k < Q; k++) x[Q * k + r] = u[r][k];
        }
    }
}

static cl twiddle(const opo::AxisPlan &p, const std::vector<cd> &tw, int s, int k, int j)
{
    if (k == 0) return cl(1, 0);
    const cd w = tw[(size_t)p.twoff[s] + (size_t)(k - 1) * (p.len[s] / p.radix[s]) + j];
    return cl(w.real(), w.imag());
}

static void transform(const opo::AxisPlan &p, const std::vector<cd> &tw, std::vector<cl> &x, bool fwd)
{
    for (int i = 0; i < p.ns; i++) {
        const int s = fwd ? i : p.ns - 1 - i, R = p.radix[s], L = p.len[s], q = L / R;
        for (int g0 = 0; g0 < p.n; g0 += L)
            for (int j = 0; j < q; j++) {
                cl v[16];
                for (int m = 0; m < R; m++)
                    v[m] = x[g0 + m * q + j] * (fwd ? cl(1, 0) : std::conj(twiddle(p, tw, s, m, j)));
                butterfly(R, fwd ? -1 : +1, v);
                for (int k = 0; k < R; k++) x[g0 + k * q + j] = v[k] * (fwd ? twiddle(p, tw, s, k, j) : cl(1, 0));
            }
    }
}

int main()
{
    const std::vector<std::vector<int>> plans = {{4, 4}, {6, 4}, {8, 4}, {9, 4}, {6, 6}, {6, 8}, {8, 8}, {9, 8}, {12, 8},
                                                 {9, 12}, {16, 8}, {12, 12}, {16, 12}, {9, 6, 4}, {16, 16}, {6, 6, 8},
                                                 {4, 4, 4}, {8, 3, 4, 2}, {4, 4, 8, 2}, {8, 8, 8}};
    int bad = 0;
    std::mt19937_64 rng(11);
    std::uniform_real_distribution<double> ph(-kPi, kPi);
    for (const auto &rad : plans) {
        std::vector<cd> tw;
        const opo::AxisPlan p = make_plan(rad, tw);
        const int n = p.n;
        const std::vector<double> dev = opo::fp64_pair_deviation(p, tw);
        const std::vector<long double> comp = opo::pair_compensation(true, p, tw);
        std::vector<long double> r(n, 0), c(n, 0);
        for (int i = 0; i < n; i++) {
            std::vector<cl> e(n, cl(0, 0)), u(n, cl(0, 0));
            e[i] = u[i] = 1;
            transform(p, tw, e, true);
            for (int q = 0; q < n; q++) r[q] += std::norm(e[q]);
            transform(p, tw, u, false);
            for (int q = 0; q < n; q++) c[i] += std::norm(u[q]);
        }
        long double worst = 0, plain = 0;
        for (int q = 0; q < n; q++) {
            worst = std::max(worst, std::abs(dev[q] - (n / std::sqrt(r[q] * c[q]) - 1)));
            plain += (r[q] * c[q] / ((long double)n * n) - 1) / n;
        }
        const int T = 200000 / n;
        long double gain = 0;
        for (int t = 0; t < T; t++)
            for (int q = 0; q < n; q++) {
                const double x = ph(rng);
                const cl v = cl(std::cos((long double)x), std::sin((long double)x)) * (comp[q] / n);
                const long double a = (double)v.real(), b = (double)v.imag();
                gain += ((a * a + b * b) * r[q] * c[q] - 1) / n;
            }
        gain /= T;
        const long double bound = 5 * 1.28e-16L / std::sqrt((long double)T * n);
        // the norms: up to 512 terms of a few roundings of 5.4e-20 each, most of which cancel
        const bool ok = worst < 2e-18L && std::abs(gain) < bound;
        std::printf("n=%4d ns=%d: network vs dense %.1Le, power gain plain %+.2Le compensated %+.2Le (bound %.1Le) %s\n", n,
                    p.ns, worst, plain, gain, bound, ok ? "ok" : "FAIL");
        bad += !ok;
    }
    return bad ? 1 : 0;
}
