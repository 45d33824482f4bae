// exercise.cuh — the arithmetic of the exercise decision (american.cu): moneyness, the continuation
// polynomial, its test in single precision, and the solver's quotients. Plain functions of their
// arguments, the same on the host, where the tests compare them with exact arithmetic.
#pragma once

#include <cmath>

#include "exact.cuh"

namespace lsm {

// double-precision operations rounded to nearest, none contracted into another (the host compiles
// with contraction off)
#ifdef __CUDA_ARCH__
FX_HD double mul(double a, double b) { return __dmul_rn(a, b); }
FX_HD double add(double a, double b) { return __dadd_rn(a, b); }
FX_HD double div(double a, double b) { return __ddiv_rn(a, b); }
FX_HD double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
#else
FX_HD double mul(double a, double b) { return a * b; }
FX_HD double add(double a, double b) { return a + b; }
FX_HD double div(double a, double b) { return a / b; }
FX_HD double fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
#endif

// S / norm rounded to nearest, from y = 1 / norm rounded to nearest (see moneyness_short for a norm
// of few digits). q0 = RN(S y) may be more than one ulp off near a power of two; one correction
// step q1 = RN(q0 + RN(S - norm q0) y) brings it within one ulp, and then the remainder S - norm q1 is exact and the second step
// q1 + r y rounded once is the correctly rounded quotient (P. Markstein, IBM J. Res. Dev.
// 34(1), 1990: y within half an ulp of 1 / norm, q1 within one ulp of S / norm).
// Five FP64 operations in place of a full division.
template <class K>
FX_HD double moneyness(double s, const K& A)
{
    const double y = A.inv_norm, b = A.norm;
    const double q0 = mul(s, y);
    const double q1 = fma_rn(fma_rn(-q0, b, s), y, q0);
    return fma_rn(fma_rn(-q1, b, s), y, q1);
}

// The same for a norm of at most 45 significant bits, from y and ylo = RN(1 / norm - y): the sum
// before its one rounding is within 2^-105 of S / norm, and a quotient of a 24-bit by a 45-bit number
// is never nearer than 2^-99 to a midpoint of two doubles (it would have to be a fraction with the
// 54-bit midpoint's numerator), so it rounds as the quotient does. Two FP64 operations.
FX_HD bool few_digits(double norm)
{
    return (fx_bits(norm) & 0xff) == 0 && norm >= 0x1p-200 && norm <= 0x1p200;
}
FX_HD double reciprocal_rest(double norm, double inv_norm) { return div(fma_rn(-norm, inv_norm, 1.0), norm); }
FX_HD double moneyness_short(double s, double y, double ylo)
{
    return fma_rn(s, y, mul(s, ylo));
}

// b0 + b1 m + b2 m m, evaluated left to right
FX_HD double continuation(double b0, double b1, double b2, double m)
{
    return add(add(b0, mul(b1, m)), mul(mul(b2, m), m));
}

// One date's exercise test in single precision (screen_exercise), with h = (S - K) / norm:
// continuation a0 + a1 h + a2 h^2, and its error bound 2^-19 |iv| + e0 + e1 |h| + e2 h^2.
struct alignas(16) LsmScreen {
    float a0, a1, a2, e0, e1, e2;
    int fit; // 1 where the date has a regression
    int pad;
};

// the screen of beta; m0 = (float) strike / norm. The expansion about the strike keeps the terms at
// the size of the values that are compared: about 0 they are tens of times larger and cancel (near
// the exercise boundary the polynomial hugs the payoff), and 4 % of the in-the-money paths of a daily
// Heston put stayed open. The e's carry 2^-19 of each term (32 units of single precision; a term has
// at most 10) and 2^-48 of the terms about 0, where the reference's own rounding and that of the
// shift lie.
FX_HD LsmScreen lsm_screen(const double* beta, int fit, double strike, double norm, double m0)
{
    LsmScreen s;
    const double a1 = fma(2.0 * beta[2], m0, beta[1]), a0 = fma(fma(beta[2], m0, beta[1]), m0, beta[0]);
    s.a0 = (float)a0;
    s.a1 = (float)a1;
    s.a2 = (float)beta[2];
    s.fit = fit;
    s.pad = 0;
    constexpr float U = 0x1p-19f, D = 0x1p-48f;
    const float k = fabsf((float)strike), q = fabsf((float)norm), m = fabsf((float)m0);
    const float b0 = fabsf((float)beta[0]), b1 = fabsf((float)beta[1]), b2 = fabsf(s.a2);
    s.e0 = U * (fabsf(s.a0) + fabsf((float)((double)(float)strike - strike))) + D * (2.0f * k + b0 + (b1 + b2 * m) * m) +
           1e-30f;
    s.e1 = U * fabsf(s.a1) + D * (q + b1 + 2.0f * b2 * m);
    s.e2 = U * b2;
    // far from single precision's range: the test stays open
    if (!(fmaxf(fmaxf(fmaxf(fabsf(s.a0), fabsf(s.a1)), fmaxf(b0, b1)), fmaxf(fmaxf(k, q), fmaxf(b2, m))) < 1e30f))
        s.e0 = INFINITY;
    return s;
}

// The exercise test iv >= b0 + b1 m + b2 m^2 (iv = phi (S - K), m = S / norm) of an
// in-the-money spot sf, in single precision: 1 exercise, 0 hold, -1 too close to call.
// With u = 2^-24, x = S - K_f (one rounding, relative) and h = x / norm, the inputs rounded to float
// and the rounded operations leave iv with 2 u (|iv| + |K_f - K|), a0 with 2 u, a1 h with 6 u and
// a2 h^2 with 9 u of their sizes, and the difference with one u of iv and c: below 10 u of each term,
// against 32 u in the bound (lsm_screen), which also holds the reference's own rounding. So |d| above
// the bound fixes the sign of the double-precision difference and hence the reference's test; inputs
// too large for single precision give an infinite or NaN d or bound and come back undecided, as does
// the thin band around the exercise boundary: the caller then runs the double-precision test.
template <class K>
FX_HD int screen_exercise(float sf, const LsmScreen& P, const K& A)
{
    const float x = sf - A.strike_f, v = x + A.strike_lo;
    const float iv = A.call ? v : -v;
    const float h = x * A.inv_norm_f, ah = fabsf(h);
    const float d = iv - fmaf(fmaf(P.a2, h, P.a1), h, P.a0);
    const float e = fmaf(fabsf(iv), 0x1p-19f, fmaf(fmaf(P.e2, ah, P.e1), ah, P.e0));
    return d > e ? 1 : (d < -e ? 0 : -1);
}

// A divisor and its reciprocal in two pieces: r = 1 / l rounded, rl = 1 / l - r rounded.
struct Pivot {
    double l, r, rl;
};
FX_HD Pivot pivot(double l)
{
    const double r = div(1.0, l);
    return Pivot{l, r, mul(fma_rn(-l, r, 1.0), r)};
}

// a / P.l from the two-piece reciprocal: within half an ulp and 2^-50 of one, so the correctly
// rounded quotient unless a tie is nearer than that. `sure` stays set where the exact remainder
// a - q l is below half an ulp of q (of the ulp below a power of two) times l by a clear margin,
// which an integer comparison of its bits decides; elsewhere, and near the ends of the range, the
// caller takes the division. Two dependent FP64 operations, the test beside the next ones: the
// solver's chain of six divisions is on every date's critical path (a division takes about nine).
FX_HD double divide_by(double a, const Pivot& P, bool& sure)
{
    const double q = fma_rn(a, P.r, mul(a, P.rl));
    const unsigned long long rem = fx_bits(fma_rn(-q, P.l, a)) & 0x7fffffffffffffffull;
    const unsigned long long qb = fx_bits(q), lb = fx_bits(P.l);
    const int ea = (int)(fx_bits(a) >> 52 & 0x7ff), eq = (int)(qb >> 52 & 0x7ff), el = (int)(lb >> 52 & 0x7ff);
    // half an ulp of q times |l|, less 2^-19 of it; half that at a power of two
    const long long half = (long long)(lb & 0x7fffffffffffffffull) - (1ll << 34) +
                           ((long long)(eq - 1023 - 53 - ((qb << 12) == 0)) << 52);
    sure &= (unsigned)(ea - 623) <= 800u && (unsigned)(el - 623) <= 800u && (long long)rem < half;
    return q;
}

} // namespace lsm
