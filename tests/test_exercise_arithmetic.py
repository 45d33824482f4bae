"""The arithmetic of the exercise decision (csrc/exercise.cuh), compiled for the host and compared
with the reference's double-precision expressions and with exact rationals:

* the single-precision screen, expanded about the strike, never decides against the reference's test
  iv >= (b0 + b1 m) + (b2 m) m and leaves a thin band open;
* the two-operation quotient S / norm for a norm of at most 45 bits is the correctly rounded one;
* the solver's quotient is the correctly rounded one wherever it says that it is sure.

Each is tried where it could go wrong: continuations that hug the payoff, quotients built next to a
tie, divisors and quotients at powers of two, the ends of the range.
"""
import ctypes as C
import os
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r'''
#include "exercise.cuh"
using namespace lsm;
struct Contract {
    int call;
    double strike, norm, inv_norm;
    float strike_f, strike_lo, inv_norm_f;
};
extern "C" {
// the screen of each spot under its own policy, as the kernels set it up
void screens(long n, const float* s, double strike, double norm, int call, const double* beta, int* out)
{
    Contract A{call, strike, norm, 1.0 / norm, (float)strike, 0.f, 0.f};
    A.strike_lo = (float)((double)A.strike_f - strike);
    A.inv_norm_f = (float)A.inv_norm;
    for (long i = 0; i < n; i++) {
        const LsmScreen P = lsm_screen(beta + 3 * i, 1, strike, norm, (double)A.strike_f / norm);
        out[i] = screen_exercise(s[i], P, A);
    }
}
void reference(long n, const float* s, double strike, double norm, int call, const double* beta, int* out)
{
    for (long i = 0; i < n; i++) {
        const double d = s[i], iv = call ? d - strike : strike - d, m = d / norm;
        out[i] = iv >= continuation(beta[3 * i], beta[3 * i + 1], beta[3 * i + 2], m);
    }
}
int short_quotients(long n, const float* s, double norm, double* out, double* markstein)
{
    const double y = 1.0 / norm, lo = reciprocal_rest(norm, y);
    Contract A{0, 0.0, norm, y, 0.f, 0.f, 0.f};
    for (long i = 0; i < n; i++) {
        out[i] = moneyness_short((double)s[i], y, lo);
        markstein[i] = moneyness((double)s[i], A);
    }
    return few_digits(norm);
}
void quotients(long n, const double* a, const double* l, double* out, int* sure)
{
    for (long i = 0; i < n; i++) {
        bool ok = true;
        out[i] = divide_by(a[i], pivot(l[i]), ok);
        sure[i] = ok;
    }
}
}
'''


@pytest.fixture(scope="module")
def arith(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("exercise")
    (d / "exercise.cpp").write_text(SOURCE)
    subprocess.run([gxx, "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "thoth_gb300", "csrc"), str(d / "exercise.cpp"), "-o", str(d / "exercise.so")],
                   check=True)
    return C.CDLL(str(d / "exercise.so"))


def ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def decisions(arith, s, K, norm, call, beta):
    s = np.ascontiguousarray(s, dtype=np.float32)
    beta = np.ascontiguousarray(beta, dtype=np.float64)
    scr, ref = np.zeros(len(s), dtype=np.int32), np.zeros(len(s), dtype=np.int32)
    for f, out in ((arith.screens, scr), (arith.reference, ref)):
        f(C.c_long(len(s)), ptr(s), C.c_double(K), C.c_double(norm), int(call), ptr(beta), ptr(out))
    return scr, ref


@pytest.mark.parametrize("call", [False, True])
@pytest.mark.parametrize("K,norm", [(100.0, 100.0), (103.7, 103.7), (1e-3 / 3, 1e-3 / 3), (4.2e7 / 3, 4.2e7 / 3),
                                    (100.0, 0.37), (0.37, 100.0), (0.0, 100.0)])
def test_screen_never_contradicts_the_reference(arith, call, K, norm):
    rng = np.random.default_rng(11 + call)
    n = 200000
    scale = K if K > 0 else norm
    s = (scale * np.exp(0.25 * rng.standard_normal(n))).astype(np.float32)
    sd = s.astype(np.float64)
    itm = (sd > K) if call else (sd < K)
    s, sd = s[itm], sd[itm]
    n = len(s)
    if n == 0:
        return  # a put struck at zero is never in the money
    iv = (sd - K) if call else (K - sd)
    m = sd / norm
    # slopes of the payoff's size and far above it; b0 then puts the continuation a signed distance
    # from the payoff, from 1e-16 of the scale to ten times it
    b2 = scale * rng.standard_normal(n) * 10.0 ** rng.uniform(-3, 3, n)
    b1 = scale * rng.standard_normal(n) * 10.0 ** rng.uniform(-3, 3, n)
    hug = rng.random(n) < 0.5  # the payoff's own slope at the spot: the polynomial hugs the payoff
    b1 = np.where(hug, (norm if call else -norm) - 2.0 * b2 * m, b1)
    gap = scale * np.sign(rng.standard_normal(n)) * 10.0 ** rng.uniform(-16, 1, n)
    b0 = iv - (b1 * m + (b2 * m) * m) - gap
    scr, ref = decisions(arith, s, K, norm, call, np.stack([b0, b1, b2], axis=1))
    closed = scr >= 0
    assert np.array_equal(scr[closed], ref[closed])
    # the band: 2^-19 of each term about the strike, 2^-48 of each about zero, with room for the
    # rounding of the bound itself
    Kf = np.float64(np.float32(K))
    m0 = Kf / norm
    h = (sd - Kf) / norm
    a1, a0 = 2.0 * b2 * m0 + b1, (b2 * m0 + b1) * m0 + b0
    about_strike = np.abs(iv) + np.abs(Kf - K) + np.abs(a0) + np.abs(a1 * h) + np.abs(b2) * h * h
    about_zero = (2 * K + np.abs(b0) + (np.abs(b1) + np.abs(b2) * m0) * m0 +
                  (norm + np.abs(b1) + 2 * np.abs(b2) * m0) * np.abs(h))
    assert closed[np.abs(gap) > 1.5 * (2.0 ** -19 * about_strike + 2.0 ** -48 * about_zero)].all()


@pytest.mark.parametrize("call", [False, True])
@pytest.mark.parametrize("K,norm", [(100.0, 100.0), (103.7, 103.7), (100.0, 0.37)])
def test_screen_beside_the_strike(arith, call, K, norm):
    """Spots a few floats from the strike, under policies whose terms about zero are up to 1e12 times
    the scale and cancel there: the reference's own rounding is then what decides."""
    rng = np.random.default_rng(17 + call)
    n = 200000
    Kf = np.float32(K)
    step = rng.integers(1, 200, n).astype(np.int32)
    s = (Kf.view(np.int32) + (step if call else -step)).astype(np.int32).view(np.float32)
    sd = s.astype(np.float64)
    iv = (sd - K) if call else (K - sd)
    m, m0 = sd / norm, np.float64(Kf) / norm
    b2 = K * 10.0 ** rng.uniform(0, 12, n) * rng.choice([-1.0, 1.0], n) / max(m0, 1.0) ** 2
    b1 = (norm if call else -norm) - 2.0 * b2 * m0
    gap = K * rng.choice([-1.0, 1.0], n) * 10.0 ** rng.uniform(-16, -2, n)
    b0 = iv - (b1 * m + (b2 * m) * m) - gap
    scr, ref = decisions(arith, s, K, norm, call, np.stack([b0, b1, b2], axis=1))
    closed = scr >= 0
    assert closed.any() and not closed.all()
    assert np.array_equal(scr[closed], ref[closed])


def test_screen_leaves_what_single_precision_cannot_hold(arith):
    """Terms beyond 1e30, infinities and values that are no number stay open: the caller's
    double-precision test decides."""
    s = np.full(8, 90.0, dtype=np.float32)
    big = [1e31, -1e31, 1e300, np.inf, -np.inf, np.nan, 1e38, 1e30]
    for col in range(3):
        beta = np.ones((8, 3))
        beta[:, col] = big
        scr, _ = decisions(arith, s, 100.0, 100.0, False, beta)
        assert (scr == -1).all(), (col, scr)
    for K, norm in ((1e31, 1e31), (100.0, 1e-38), (100.0, 1e35)):
        scr, _ = decisions(arith, s, K, norm, False, np.ones((8, 3)))
        assert (scr == -1).all()
    scr, _ = decisions(arith, np.array([np.inf, np.nan], dtype=np.float32), 100.0, 100.0, True, np.ones((2, 3)))
    assert (scr == -1).all()


@pytest.mark.parametrize("norm", [100.0, 3.0, 1.0, 2.0 ** 40, 1e-3 * 2 ** 10 // 1, 123456.75, (2.0 ** 45 - 1) * 2.0 ** -40,
                                  (2.0 ** 44 + 1) * 2.0 ** -30, (2.0 ** 45 - 1) * 2.0 ** 100, (2.0 ** 44 + 3) * 2.0 ** -230])
def test_short_quotient_is_correctly_rounded(arith, norm):
    """Random spots, every spot's neighbours at powers of two, and the spots of 24 bits whose quotients
    lie nearest a tie among a million."""
    if norm == 0.0:
        norm = 1.0
    mant, exp = np.frexp(norm)
    n45 = int(mant * 2 ** 53)
    assert n45 % 2 ** 8 == 0
    rng = np.random.default_rng(5)
    ints = rng.integers(1 << 23, 1 << 24, 1 << 20)
    # (2 S 2^k mod n) nearest 0 or n with k such that the quotient has 54 bits: a tie has remainder 0
    odd = n45 // (n45 & -n45)
    k = 54 + odd.bit_length() - 24
    pw = pow(2, k, 2 * odd)
    dist = [(min(r, 2 * odd - r), int(s)) for s in ints[:200000] for r in [int(s) * pw % (2 * odd)]]
    hard = np.array([s for _, s in sorted(dist)[:2000]])
    edges = np.concatenate([2 ** 23 + np.arange(64), 2 ** 24 - 1 - np.arange(64)])
    for e in (-149 + 23, -60, -23, 0, 3, 100):
        s = np.ldexp(np.concatenate([ints, hard, edges]).astype(np.float64), e).astype(np.float32)
        s = s[(s > 0) & np.isfinite(s)]
        q, mk = np.zeros(len(s)), np.zeros(len(s))
        short = arith.short_quotients(C.c_long(len(s)), ptr(s), C.c_double(norm), ptr(q), ptr(mk))
        assert short == (2.0 ** -200 <= norm <= 2.0 ** 200)
        want = s.astype(np.float64) / norm
        if short:
            np.testing.assert_array_equal(q, want)
            np.testing.assert_array_equal(mk, want)


def test_sure_quotients_are_correctly_rounded(arith):
    rng = np.random.default_rng(3)
    n = 400000
    l = np.ldexp(rng.integers(1 << 52, 1 << 53, n).astype(np.float64), rng.integers(-120, 20, n))
    a = np.ldexp(rng.integers(1 << 52, 1 << 53, n).astype(np.float64), rng.integers(-120, 20, n)) * rng.choice([-1.0, 1.0], n)
    plain = n
    # next to a tie: a = RN(l (q + 1/2 ulp)) and its neighbours; and next to powers of two
    m = 20000
    tie_a, tie_l = [], []
    for li, qi, e in zip(rng.integers(1 << 52, 1 << 53, m), rng.integers(1 << 52, 1 << 53, m), range(m)):
        li, qi = int(li), int(qi)
        if e % 4 == 0:
            qi = 1 << 52
        if e % 8 == 3:
            qi = (1 << 53) - 1
        if e % 16 == 5:
            li = 1 << 52
        if e % 16 == 9:
            li = (1 << 53) - 1
        x = float(Fraction(2 * qi + (1 if e % 2 else -1), 2) * li)  # correctly rounded
        for y in (np.nextafter(x, 0.0), x, np.nextafter(x, np.inf)):
            tie_a.append(y)
            tie_l.append(float(li))
    # as near a tie as a quotient can be: a 2^54 = x l - d for an odd x of 54 bits and a small odd d
    for li in rng.integers(1 << 51, 1 << 52, 6000):
        li = 2 * int(li) + 1
        inv = pow(li, -1, 1 << 54)
        for d in (1, -1, 3, -7, 4095, -65535):
            x = d * inv % (1 << 54)
            y = (x * li - d) >> 54
            if x >> 53 and y >> 52 and (y << 54) == x * li - d and y < (1 << 53):
                tie_a.append(float(y))
                tie_l.append(float(li))
    ties = len(tie_a)
    ends = [2.0 ** -400, 2.0 ** 400, 2.0 ** -399, 2.0 ** 399, 1e-300, 1e300, 2.0 ** -1060, 0.0, 1.0, 3.0, np.inf]
    ea, el = np.meshgrid(ends, [x for x in ends if 0.0 < x < np.inf])
    a = np.concatenate([a, tie_a, ea.ravel(), -ea.ravel()])
    l = np.concatenate([l, tie_l, el.ravel(), el.ravel()])
    q, sure = np.zeros(len(a)), np.zeros(len(a), dtype=np.int32)
    arith.quotients(C.c_long(len(a)), ptr(a), ptr(l), ptr(q), ptr(sure))
    with np.errstate(over="ignore", under="ignore", invalid="ignore"):
        want = a / l
    s = sure != 0
    np.testing.assert_array_equal(q[s], want[s])
    assert s[:plain].mean() > 0.999          # the division is the exception
    assert ties - 3 * m > 5000 and not s[a == 0.0].any()
