// fastmath.cuh -- branch-free FP64 exponential, tanh on [0, 1] and square
// root for the per-pair arithmetic of the symmetry-function kernels.
//
// The library routines handle every argument range and special value, and
// their range tests are branches: inside a warp whose lanes hold different
// pairs the lanes can take different sides, and a branch also keeps the
// compiler from interleaving two independent sequences.  The arguments here
// are bounded by the cutoff geometry (exp of a non-positive number, tanh of
// u = 1 - r/rc in [0, 1], sqrt of a squared distance), so each function is
// one straight-line sequence:
//
//  * exp_clamped(x), x clamped to [-708, 709]: Cody-Waite argument
//    reduction x = k ln2 + r, |r| <= ln2/2 (W. J. Cody and W. Waite, "Software Manual for the
//    Elementary Functions", 1980), with the reduction done by fused
//    multiply-adds against ln2 split into its double rounding and the
//    remainder; e^r - 1 by its Taylor series to degree 13 evaluated with
//    Estrin's scheme (depth 4 instead of a 13-deep Horner chain), 1 added
//    last; 2^k applied through the exponent field (e^-708 ~ 3e-308, the
//    smallest result without a subnormal scale).  Error within 1 ulp of
//    libm (tests/test_fastmath.py emulates these operations on the host
//    with exact fused multiply-adds, and checks the device functions, run
//    through hdnnp_debug_math, against libm's exp, tanh and sqrt).
//  * exp_neg(x): exp_clamped's operations for x in [-700, 0], without the
//    clamp.  exp_small(x) for x in [-1.5, 0]: the same reduction (W. J. Cody,
//    W. Waite, "Software Manual for the Elementary Functions", 1980) with ln 2
//    in one double (at most two of them are taken off) and a polynomial
//    interpolated at Chebyshev nodes on [-ln 2 / 2, ln 2 / 2].
//  * tanh01(u) for u in [0, 1]: a polynomial interpolated at Chebyshev nodes;
//    no reduction, no reciprocal.  (Both interpolants in 60 decimal digits,
//    then rounded; two Horner chains each.)
//  * sqrt_rsqrt(x) and rsqrt_pos(x): the hardware reciprocal square-root
//    approximation refined by one third-order Newton step; the root as
//    x * rsqrt with one residual correction.  x = 0 gives 0 (the reciprocal
//    is taken of max(x, 1e-300)).
// The constants are ln 2 and 1/ln 2 rounded to double, the remainder
// ln 2 - double(ln 2), 1.5 * 2^52 (the round-to-integer shifter), 1/n! and
// the interpolants'.
#pragma once

namespace hdnnp {

__device__ __forceinline__ double rsqrt_approx(double x) {
    double y;
    asm("rsqrt.approx.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}

// e^x for x in [-708, 709] (arguments outside are clamped to the range)
__device__ __forceinline__ double exp_clamped(double x) {
    constexpr double kLog2e = 1.4426950408889634;
    constexpr double kLn2Hi = 0.6931471805599453;
    constexpr double kLn2Lo = 2.3190468138462996e-17;
    constexpr double kShift = 6755399441055744.0;  // 1.5 * 2^52
    x = fmin(fmax(x, -708.0), 709.0);
    const double t = fma(x, kLog2e, kShift);
    const int k = __double2loint(t);
    const double kd = t - kShift;
    double r = fma(kd, -kLn2Hi, x);
    r = fma(kd, -kLn2Lo, r);
    // e^r - 1 = sum_{n=1..13} r^n / n!, Estrin's scheme
    const double r2 = r * r, r4 = r2 * r2, r8 = r4 * r4;
    const double q0 = r;                                                  // r
    const double q1 = fma(0.16666666666666666, r, 0.5);                   // 1/2! + r/3!
    const double q2 = fma(0.008333333333333333, r, 0.041666666666666664);  // 1/4! + r/5!
    const double q3 = fma(0.0001984126984126984, r, 0.001388888888888889);
    const double q4 = fma(2.7557319223985893e-06, r, 2.48015873015873e-05);
    const double q5 = fma(2.505210838544172e-08, r, 2.755731922398589e-07);
    const double q6 = fma(1.6059043836821613e-10, r, 2.08767569878681e-09);
    const double s0 = fma(q1, r2, q0);
    const double s1 = fma(q3, r2, q2);
    const double s2 = fma(q5, r2, q4);
    const double t0 = fma(s1, r4, s0);
    const double t1 = fma(q6, r4, s2);
    const double p = 1.0 + fma(t1, r8, t0);
    return p * __hiloint2double((k + 1023) << 20, 0);
}

// Coefficients, read as constant-bank operands of the multiply-adds: as
// literals each would cost two moves into registers per use.
__constant__ double kExpSmall[13] = {1.4426950408889634, 6755399441055744.0, 0.6931471805599453, 0.5000000000000001,
                                     0.16666666666666669, 0.041666666666623824, 0.008333333333330039,
                                     0.0013888888917367081, 0.00019841269863171557, 2.4801521057868204e-05,
                                     2.7557268276905696e-06, 2.7620201591031547e-07, 2.5100472505694996e-08};
__constant__ double kTanh01[16] = {1.0, -0.3333333333333273, 0.13333333333282113, -0.05396825395091773,
                                   0.021869488226930838, -0.008863232181130274, 0.003592104115230281,
                                   -0.00145571559077928, 0.0005896028950856166, -0.00023801236323479905,
                                   9.472256075732066e-05, -3.603918536997382e-05, 1.2306805295349983e-05,
                                   -3.402993826979274e-06, 6.496857637862531e-07, -6.20675330545365e-08};

// e^x for x in [-1.5, 0]: x = k ln 2 + r, k = 0, -1, -2, and 2^k (1 + r +
// r^2 q(r)), q the degree-9 interpolant of (e^r - 1 - r) / r^2 (error 1e-16 of
// q, 2e-17 of the sum).  Relative error below 2^-52 (0.71 of it measured).  As
// many FP64 operations as one polynomial 1 + x + x^2 q(x) over the whole
// interval, whose terms cancel near -1.5 (6.1 of 2^-52 there).
__device__ __forceinline__ double exp_small(double x) {
    const double t = fma(x, kExpSmall[0], kExpSmall[1]);
    const double r = fma(t - kExpSmall[1], -kExpSmall[2], x), r2 = r * r;
    double a = kExpSmall[11], b = kExpSmall[12];
#pragma unroll
    for (int n = 9; n >= 3; n -= 2) a = fma(a, r2, kExpSmall[n]);
#pragma unroll
    for (int n = 10; n >= 4; n -= 2) b = fma(b, r2, kExpSmall[n]);
    const double p = 1.0 + fma(fma(b, r, a), r2, r);
    return __hiloint2double(__double2hiint(p) + (int)((unsigned)__double2loint(t) << 20), __double2loint(p));
}

// tanh(u) for u in [0, 1]: u p(u^2), p the degree-15 Chebyshev interpolant of
// tanh(sqrt v) / sqrt v on [0, 1] (error 6e-17)
__device__ __forceinline__ double tanh01(double u) {
    const double v = u * u, w = v * v;
    double a = kTanh01[14], b = kTanh01[15];
#pragma unroll
    for (int k = 12; k >= 0; k -= 2) a = fma(a, w, kTanh01[k]);
#pragma unroll
    for (int k = 13; k >= 1; k -= 2) b = fma(b, w, kTanh01[k]);
    return u * fma(b, v, a);
}

// e^x for x in [-700, 0], the operations of exp_clamped without the range
// clamp and with its coefficients in the constant bank
__constant__ double kExpNeg[16] = {1.4426950408889634, 6755399441055744.0, 0.6931471805599453, 2.3190468138462996e-17,
                                   0.5, 0.16666666666666666, 0.041666666666666664, 0.008333333333333333,
                                   0.001388888888888889, 0.0001984126984126984, 2.48015873015873e-05,
                                   2.7557319223985893e-06, 2.755731922398589e-07, 2.505210838544172e-08,
                                   2.08767569878681e-09, 1.6059043836821613e-10};
__device__ __forceinline__ double exp_neg(double x) {
    const double t = fma(x, kExpNeg[0], kExpNeg[1]);
    const int k = __double2loint(t);
    const double kd = t - kExpNeg[1];
    double r = fma(kd, -kExpNeg[2], x);
    r = fma(kd, -kExpNeg[3], r);
    const double r2 = r * r, r4 = r2 * r2, r8 = r4 * r4;
    const double q1 = fma(kExpNeg[5], r, kExpNeg[4]), q2 = fma(kExpNeg[7], r, kExpNeg[6]);
    const double q3 = fma(kExpNeg[9], r, kExpNeg[8]), q4 = fma(kExpNeg[11], r, kExpNeg[10]);
    const double q5 = fma(kExpNeg[13], r, kExpNeg[12]), q6 = fma(kExpNeg[15], r, kExpNeg[14]);
    const double s0 = fma(q1, r2, r), s1 = fma(q3, r2, q2), s2 = fma(q5, r2, q4);
    const double t0 = fma(s1, r4, s0), t1 = fma(q6, r4, s2);
    const double p = 1.0 + fma(t1, r8, t0);
    return p * __hiloint2double((k + 1023) << 20, 0);
}

// x^y, y not an integer, of an angular function's base x = 1 + lambda cos: a
// base that rounding takes below zero (collinear atoms, lambda = 1 or -1) is
// zero, not NaN.  The limits lie above the rounding of the cosine.
__device__ __forceinline__ double base_pow(double x, double y) { return pow(x < 0.0 && x > -1e-10 ? 0.0 : x, y); }
__device__ __forceinline__ float base_pow(float x, float y) { return powf(x < 0.0f && x > -1e-4f ? 0.0f : x, y); }

// 1 / sqrt(x) for x > 0 (x = 0 gives 1e150)
__device__ __forceinline__ double rsqrt_pos(double x) {
    // max(x, 1e-300) on the high word (x >= 0; the low word only matters above)
    const double xc = __hiloint2double(max(__double2hiint(x), 0x01a56e1f), __double2loint(x));
    const double y = rsqrt_approx(xc);
    const double e = fma(-xc * y, y, 1.0);                     // 1 - x y^2
    return fma(y * e, fma(0.375, e, 0.5), y);                  // y (1 + e/2 + 3e^2/8)
}

// sqrt(x) and 1/sqrt(x) for x >= 0 (x = 0: r = 0, ir = 1e150)
__device__ __forceinline__ void sqrt_rsqrt(double x, double& r, double& ir) {
    ir = rsqrt_pos(x);
    const double s = x * ir;
    r = fma(0.5 * ir, fma(-s, s, x), s);
}

}  // namespace hdnnp
