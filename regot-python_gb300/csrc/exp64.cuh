// FP64 exponential of the plan entries, exp(arg / reg).
//
// Table-driven evaluation after P. T. P. Tang, "Table-driven implementation of
// the exponential function in IEEE floating-point arithmetic" (ACM TOMS 15,
// 1989): z = arg (1 / reg), n = round(z 4096 / ln 2), r = z - n ln2 / 4096 in
// two exact-product steps (Cody and Waite), exp(z) = 2^(n / 4096) e^r, with
// 2^(i / 4096) = T_i (1 + t_i) from a table of 4096 pairs (64 KB, gathered
// through L1), T_i correctly rounded, and e^r by its Taylor polynomial of degree
// three (|r| < 2^-13.5: the next term is below 2^-58). The t_i keep the table's
// own rounding out of the result: within 0.52 units in the last place of the
// exponential of z, 0.29 root mean square (1.01 and 0.41 without them).
//
// Twelve FP64 instructions an entry with the argument, where the passes with
// exp() took about twenty-two: FP64 issue bounds every FP64 pass (a GB300 SM
// starts two FP64 operations a clock). The range tests look at exponent
// bits.
#pragma once

#include <cuda_runtime.h>

namespace regot {

struct Exp64 {
    const double2* table;  // (T_i, t_i), i < 4096 (device)
    const double2* phi;    // (phi(x), e^x - 1) at x = (i - 3072) ln2 / 4096, i < 6144
    double inv_reg;
};

// The tables of the current device (made with its first context and kept) and 1 / reg.
Exp64 exp64_for(double reg);

// exp(arg / reg); arg = -infinity gives 0.
__device__ __forceinline__ double exp_scaled(double arg, const Exp64& e) {
    constexpr double kMagic = 6755399441055744.0;  // 1.5 * 2^52: rounds to an integer
    const double z = arg * e.inv_reg;
    const unsigned hz = (unsigned)__double2hiint(z);
    if ((hz & 0x7fffffffu) < 0x40862000u) {  // |z| < 708: a normal result
        const double t = fma(z, 5909.278887481194, kMagic);
        const int n = __double2loint(t);
        const double k = t - kMagic;
        double r = fma(k, -0.00016922538566177536, z);
        r = fma(k, -2.1711753512906926e-13, r);
        const double2 T = __ldg(e.table + (n & 4095));
        // (1 + t) e^r - 1
        const double q = fma(r * r, fma(r, 0.16666666666666666, 0.5), r + T.y);
        const double v = fma(T.x, q, T.x);
        return __hiloint2double(__double2hiint(v) + ((n >> 12) << 20), __double2loint(v));
    }
    // below -746 the exponential is 0 (-infinity included, NaN not)
    if (hz >= 0xc0875000u && (hz < 0xfff00000u || (hz == 0xfff00000u && __double2loint(z) == 0)))
        return 0.0;
    return exp(z);
}

// phi(x) = e^x - 1 - x without cancellation, for x <= 700. With x = n c + r,
// c = ln2 / 4096, |r| <= c / 2, A = phi(n c) and B = e^(n c) - 1 tabulated
// (|n| <= 3072),
//     phi(x) = A + B r + (1 + B) phi(r),
// phi(r) by its series to r^7. Below 2^-9, where A + B r would cancel, n = 0 and
// r = x instead (A = B = 0, the series still a few 1e-17 relative); from
// |x| = 1/2 on, where phi > 0.1, as it stands with e^x as above. Some nineteen
// FP64 instructions without a divergent branch, where the series to x^17 beside
// expm1(x) - x in one warp took about thirty-four. Largest error 1.97 units in
// the last place below 1/2 and 2.5 beyond (2.01 and 3.0 for series and expm1).
__device__ __forceinline__ double phi_tabled(double x, const Exp64& e) {
    constexpr double kMagic = 6755399441055744.0;
    const unsigned ax = (unsigned)__double2hiint(x) & 0x7fffffffu;
    const double t = fma(x, 5909.278887481194, kMagic);
    int n = __double2loint(t);
    const double k = t - kMagic;
    double r = fma(k, -0.00016922538566177536, x);
    r = fma(k, -2.1711753512906926e-13, r);
    if (ax < 0x3f600000u) {  // |x| < 2^-9
        n = 0;
        r = x;
    }
    double s = fma(r, 1.9841269841269841e-04, 1.3888888888888889e-03);
    s = fma(r, s, 0.0083333333333333332);
    s = fma(r, s, 0.041666666666666664);
    s = fma(r, s, 0.16666666666666666);
    s = fma(r, s, 0.5);
    const double q = (r * r) * s;  // phi(r)
    if (ax < 0x3fe00000u) {  // |n| <= 2955
        const double2 ab = __ldg(e.phi + (n + 3072));
        return fma(ab.y, r, ab.x) + fma(ab.y, q, q);
    }
    if (ax < 0x40862000u) {
        const double2 T = __ldg(e.table + (n & 4095));
        const double E = __hiloint2double(__double2hiint(T.x) + ((n >> 12) << 20), __double2loint(T.x));
        return fma(E, (r + T.y) + q, (E - 1.0) - x);
    }
    return expm1(x) - x;
}

}  // namespace regot
