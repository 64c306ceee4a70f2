// The tests by which the tensor kernels reject combinations (host side, plain C++):
// upper bounds on the mutual information that a threshold is compared through,
// and the error bounds of the single-precision key estimates.
//
// With q the control fraction, D(p||q) the binary relative entropy in bits and
// s, b the size and the controls of a cell, N MI = sum over the cells of
// s D(b/s || q); the sizes add up to N and the controls to n_ctrls.
#pragma once

#include <algorithm>
#include <cmath>

namespace fiu {

// D(p||q) <= c (p - q)^2 on [0, 1] for
//     c = max(1 / (2 ln2 q (1-q)), -lg(1-q) / q^2, -lg(q) / (1-q)^2):
// f(p) = D(p||q) - c (p-q)^2 has f(q) = f'(q) = 0 and
// f'' = 1 / (ln2 p (1-p)) - 2c, which is <= 0 on an interval around q (first
// term of the maximum) and > 0 beyond it, so f falls from 0 up to where the
// interval ends and lies below its chord to the end point (second and third
// terms) after that.  So
//     N MI <= c (sum b^2 / s - n_ctrls^2 / N)      [bits].
//
// A combination whose N MI reaches thr_bits has
// sum b^2 / s >= bound_k * thr_bits + bound_c.  Slack: each of `cells` terms, at
// most b <= n_ctrls, carries at most 12 roundings or approximations of 2^-22 and
// the sum `cells` more of 2^-24 of the total n_ctrls; the 2^-20 shift of s lowers a
// term by at most 2^-20 of it.  Doubled.
inline void f4_quadratic(int n_cases, int n_ctrls, int cells, double& bound_k, double& bound_c) {
    const double N = (double)n_cases + n_ctrls, q = n_ctrls / N;
    const double lg_q = std::log2(q), lg_1q = std::log2(1 - q);
    const double c = std::max({1 / (2 * std::log(2.0) * q * (1 - q)), -lg_1q / (q * q), -lg_q / ((1 - q) * (1 - q))});
    const double u = std::ldexp(1.0, -24);
    bound_k = (1 - 1e-9) / c;
    bound_c = q * n_ctrls * (1 - 1e-9) - (2 * n_ctrls * (12 * 4 * u + 16 * u + cells * u) + 1e-3);
}

// A closer bound, for tables of many cells.  g(p) = D(p||q) / (p-q)^2 is the average
// over u, weighted with 1 - u, of D''(q + u (p-q)) = (1/t + 1/(1-t)) / ln2 at
// t = q + u (p-q).  For fixed u the two parts are 1/(a + u p) and 1/(b + u (1-p)) with
// a = q (1-u) and b = (1-q) (1-u): convex in p, so g lies below its chord
// L(p) = g(0) + (g(1) - g(0)) p.  The chord of 1/(a + u p) exceeds it by p (1-p) times
// u^2 / (a (a+u) (a + u p)), its divided difference at 0, p and 1, and the other
// likewise, so
//     R(p) = (L - g) / (p (1-p))
// is an average of such fractions, positive and convex in p.  With k its least value
// D <= (p-q)^2 Q(p), Q = L - k p (1-p), exact at p = 0, p = 1 and where R is least
// (near q).  Summed over the cells with p = b/s the powers below the second give
// constants:
//     N MI <= a0 N + a1 n_ctrls + sum b p (a2 + a3 p + a4 p^2).
struct F4Quartic {
    float a2, a3, a4;
};
// Least value of R, lowered by 0.1 % (the search ends within 1e-9 of the place, and R is computed to 1e-5).
inline double f4_least_ratio(double q) {
    const double r = 1 - q, l2 = std::log(2.0), L0 = -std::log1p(-q) / l2 / (q * q), L1 = -std::log(q) / l2 / (r * r);
    auto R = [&](double x) {  // p = 1 / (1 + e^-x): even steps towards both ends
        const double p = 1 / (1 + std::exp(-x)), p1 = 1 / (1 + std::exp(x)), d = p - q;
        const double g = std::fabs(d) < 1e-5 * std::min(q, r)
                             ? 1 / (2 * l2 * q * r)
                             : (p * std::log1p(d / q) + p1 * std::log1p(-d / r)) / l2 / (d * d);
        return (L0 + (L1 - L0) * p - g) / (p * p1);
    };
    double lo = -25, hi = 25;  // convex in p, so it falls and then rises in x too
    for (int it = 0; it < 60; ++it) {
        const double m = (hi - lo) / 3, a = lo + m, b = hi - m;
        if (R(a) <= R(b)) hi = b;
        else lo = a;
    }
    return std::max(0.0, R((lo + hi) / 2) * 0.999 - 1e-4);
}
// The coefficients and the test (as f4_quadratic).  Slack, in units of 2^-24 n_ctrls S with
// S = |a2| + |a3| + |a4| (a term is at most b S, and the b add up to n_ctrls): 12 roundings and
// approximations of a term, 64 for the 2^-20 shift of s in up to four powers of b/s, 3 of the
// coefficients, `cells` of the sum; taken as 2 (15 + cells).
inline F4Quartic f4_quartic(int n_cases, int n_ctrls, int cells, double& bound_k, double& bound_c) {
    const double N = (double)n_cases + n_ctrls, q = n_ctrls / N, r = 1 - q;
    const double L0 = -std::log2(r) / (q * q), L1 = -std::log2(q) / (r * r), k = f4_least_ratio(q);
    const double A = L0, B = L1 - L0 - k, C = k;
    const double a4 = C, a3 = B - 2 * q * C, a2 = A - 2 * q * B + q * q * C, a1 = q * q * B - 2 * q * A, a0 = q * q * A;
    const double S = std::fabs(a2) + std::fabs(a3) + std::fabs(a4), u = std::ldexp(1.0, -24);
    const double slack = 2 * n_ctrls * S * (15 + cells) * u + 1e-3;
    bound_k = 1 - 1e-9;
    bound_c = -a0 * N - a1 * n_ctrls - slack;
    return F4Quartic{(float)a2, (float)a3, (float)a4};
}

// Bound (in bits) on |order 3's estimate (t3x_survivor, tensor3m.cu) - exact key / (ln2 * 2^32)| over the 81
// terms of one combination: with N the number of samples every partial sum is
// at most 2 N lg2 N (81 roundings of at most 2^-24 of it), lg2.approx is
// within 2^-18 of log2 on every input the kernel can see (measured worst case
// 1.93e-6, checked exhaustively against FP64 by fiu_probe_lg2_error), the
// x + 2^-20 shift moves each term by at most 2^-20 / ln 2 (counts below 16)
// or one rounding of the count, and the integer table rounds each term by
// 1/2.  Doubled.
inline double t3_margin(int n_samples) {
    const double N = n_samples, lgN = std::log2(std::max(2.0, N)), B = 2 * N * lgN;
    const double u = std::ldexp(1.0, -24), e20 = std::ldexp(1.0, -20), e_lg2 = std::ldexp(1.0, -18);
    const double err = 81 * u * B + 2 * N * (18 * u + e_lg2) + 81 * e20 / std::log(2.0) +
                       2 * N * std::ldexp(1.0, -23) / std::log(2.0) + 81 * 0.5 / (std::log(2.0) * 4294967296.0);
    return 2 * err + 1e-3;
}

// Bound (in bits) on |t4x_estimate - exact key / (ln2 * 2^32)|, N samples: each sample lies in one of the 81
// cells, so sum s over the cells is N and sum s lg2 s <= N lg2 N.  A cell's products and sums round at most 5
// times by 2^-24 of at most s lg2 s; lg2.approx is within 2^-18 of log2 on every input the kernel can see (checked
// exhaustively by fiu_probe_lg2_error), which moves a cell by at most 2 s 2^-18; the x + 2^-20 shift moves each
// of the 243 products by at most 2^-20 / ln 2 and its rounding each logarithm by at most 2^-24 / ln 2; the
// running sum, below N, rounds 81 times; the integer table rounds each of the 243 exact terms by 1/2 of 2^-32
// nats.  Doubled.  (0.3 bits at 8 000 samples, 4.6 at 130 000.)
inline double t4x_margin(int n_samples) {
    const double N = n_samples, lgN = std::log2(std::max(2.0, N)), l2 = std::log(2.0);
    const double u = std::ldexp(1.0, -24), e20 = std::ldexp(1.0, -20), e_lg2 = std::ldexp(1.0, -18);
    const double err = 5 * u * N * lgN + 2 * N * e_lg2 + 243 * e20 / l2 + 2 * N * u / l2 + 82 * u * N +
                       243 * 0.5 / (l2 * 4294967296.0);
    return 2 * err + 1e-3;
}

}  // namespace fiu
