// calib.cu — LSV leverage calibration by the binned particle method, the algorithm of
// Single::CalibrateLeverage and its helpers (pricer/src/marketdata/single.cpp:240-473) with
// the reference Rng (helpers/rng.hpp) and inverse normal (helpers/distributions.cpp:37-81).
//
// One cooperative launch walks the dates. Per date, two rounds build the conditional variance of
// the current ensemble: (A) the extremes of ln S and the sum of v, (B) per-bin counts and sums of
// v between those extremes. In a round every CTA adds its contribution into the date's totals
// (exact integer sums), arrives at a counter and waits for the others there; every CTA then forms
// the bin means and the layer itself, from the same totals. Everything of the step into the date
// that needs no layer runs between an arrival and its wait: the Gaussians, the generator's jump
// and the layer coordinate behind round A, the variance step behind round B.
//
// GB300 issues FP64 at 1/64 of the FP32 rate: an FP64 instruction holds its scheduler's pipe for
// 64 clocks, and 16384 particles are one warp a scheduler on 128 SMs, so the FP64 instructions of
// a date are what it costs. The step is therefore kept short: constants of a date come from the
// host; the tail of the inverse normal (its logarithm and square root, 4.85 % of draws) runs on
// draws collected over the CTA; the layer is looked up from ln S - ln S0, which the ensemble
// carries, instead of from the logarithm of a spot kept through an exponential; the part of the
// log-spot step that no leverage enters waits ready for it; a CTA builds the layer only where the
// ensemble is (a CTA without particles writes the whole of it out). Per date 29 us as a
// restatement of the reference's expressions, both branches of the inverse normal evaluated and a
// last CTA building the layer: 13.3 ms for 16384 particles x 365 dates; like this 18 us, 6.5 ms.
//
// The Gaussians are the reference's stream: xoshiro256++ seeded by splitmix64, one 64-bit
// draw per Gaussian through Acklam's inverse normal, two per particle per date in particle
// order. Each particle keeps its own generator state: it starts 2p draws into the stream and
// jumps 2P - 2 draws after each date. The generator is linear over GF(2), so a jump by d
// draws is the polynomial x^d mod chi (chi the characteristic polynomial of the transition)
// evaluated at the transition: 256 transitions and XORs (F. Haramoto et al., "Efficient jump
// ahead for F2-linear random number generators", INFORMS J. Computing 20(3), 2008).
//
// Compiled without FMA contraction (the book kernel's tail Gaussians round as the reference's do);
// the ensemble's own arithmetic uses fused multiply-adds where written. It differs from the
// reference's in rounding only, about one part in 10^16 an operation; the sums of v are exact
// (exact.cuh), independent of the grid.
#include "calib.cuh"
#include "phi.cuh"

#include <cmath>

#include <mutex>
#include <vector>

namespace {

constexpr int CALIB_WARPS = CALIB_THREADS / 32;
static_assert(CALIB_WARPS == 4, "four warps share the results of round A");
constexpr unsigned long long WAIT_LIMIT_NS = 2000000000ull; // 2 s

__host__ __device__ __forceinline__ uint64_t rotl64(uint64_t x, int k) { return (x << k) | (x >> (64 - k)); }

// xoshiro256++: output, then the state transition (helpers/rng.hpp:50-62)
__host__ __device__ __forceinline__ uint64_t xo_next(uint64_t* s)
{
    const uint64_t result = rotl64(s[0] + s[3], 23) + s[0];
    const uint64_t t = s[1] << 17;
    s[2] ^= s[0];
    s[3] ^= s[1];
    s[1] ^= s[2];
    s[0] ^= s[3];
    s[2] ^= t;
    s[3] = rotl64(s[3], 45);
    return result;
}

__host__ __device__ __forceinline__ void xo_step(uint64_t* s)
{
    const uint64_t t = s[1] << 17;
    s[2] ^= s[0];
    s[3] ^= s[1];
    s[1] ^= s[2];
    s[0] ^= s[3];
    s[2] ^= t;
    s[3] = rotl64(s[3], 45);
}

// s <- q(A) s for q = sum_i poly_i x^i: the state sum_i poly_i A^i s
__host__ __device__ void xo_jump(const uint64_t* poly, uint64_t* s)
{
    uint64_t r0 = 0, r1 = 0, r2 = 0, r3 = 0;
    for (int w = 0; w < 4; w++) {
        uint64_t bits = poly[w];
        for (int b = 0; b < 64; b++) {
            if (bits & 1u) {
                r0 ^= s[0];
                r1 ^= s[1];
                r2 ^= s[2];
                r3 ^= s[3];
            }
            bits >>= 1;
            xo_step(s);
        }
    }
    s[0] = r0;
    s[1] = r1;
    s[2] = r2;
    s[3] = r3;
}

// the fixed date-to-date jump by its nibble table in shared memory: the XOR of the table
// rows the state's 64 nibbles select (the matrix-vector product over GF(2))
__device__ __forceinline__ void xo_jump_tab(const uint64_t* tab, uint64_t* s)
{
    uint64_t r0 = 0, r1 = 0, r2 = 0, r3 = 0;
#pragma unroll
    for (int w = 0; w < 4; w++) {
        uint64_t x = s[w];
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const ulonglong2* t = reinterpret_cast<const ulonglong2*>(tab + ((w * 16 + k) * 16 + (int)(x & 15u)) * 4);
            const ulonglong2 a = t[0], b = t[1];
            r0 ^= a.x;
            r1 ^= a.y;
            r2 ^= b.x;
            r3 ^= b.y;
            x >>= 4;
        }
    }
    s[0] = r0;
    s[1] = r1;
    s[2] = r2;
    s[3] = r3;
}

constexpr double ACKLAM_P_LOW = 0.02425;

// Acklam's inverse normal (the reference's NormalCdfInv), its two branches apart, each the
// expression the reference evaluates there
__device__ __forceinline__ double acklam_central(double P) // P in [p_low, 1 - p_low]
{
    const double a0 = -3.969683028665376e+01, a1 = 2.209460984245205e+02, a2 = -2.759285104469687e+02,
                 a3 = 1.383577518672690e+02, a4 = -3.066479806614716e+01, a5 = 2.506628277459239e+00;
    const double b0 = -5.447609879822406e+01, b1 = 1.615858368580409e+02, b2 = -1.556989798598866e+02,
                 b3 = 6.680131188771972e+01, b4 = -1.328068155288572e+01;
    const double q = P - 0.5;
    const double r = q * q;
    const double cn = (((((a0 * r + a1) * r + a2) * r + a3) * r + a4) * r + a5) * q;
    const double cd = ((((b0 * r + b1) * r + b2) * r + b3) * r + b4) * r + 1.0;
    return cn / cd;
}

__device__ __forceinline__ double acklam_tail(double P) // P < p_low or P > 1 - p_low
{
    const double c0 = -7.784894002430293e-03, c1 = -3.223964580411365e-01, c2 = -2.400758277161838e+00,
                 c3 = -2.549732539343734e+00, c4 = 4.374664141464968e+00, c5 = 2.938163982698783e+00;
    const double d0 = 7.784695709041462e-03, d1 = 3.224671290700398e-01, d2 = 2.445134137142996e+00,
                 d3 = 3.754408661907416e+00;
    const bool lower = P < ACKLAM_P_LOW;
    const double qt = sqrt(-2.0 * log(lower ? P : 1.0 - P));
    const double tn = ((((c0 * qt + c1) * qt + c2) * qt + c3) * qt + c4) * qt + c5;
    const double td = (((d0 * qt + d1) * qt + d2) * qt + d3) * qt + 1.0;
    return (lower ? tn : -tn) / td;
}

// a uniform in (0, 1) of 53 bits, as Rng::Gaussian forms it
__device__ __forceinline__ double uniform53(uint64_t* s)
{
    const double u0 = (double)(xo_next(s) >> 11) * (1.0 / 9007199254740992.0);
    return u0 > 0.0 ? u0 : (1.0 / 9007199254740992.0);
}

__device__ __forceinline__ bool in_tail(double u) { return u < ACKLAM_P_LOW || !(u <= 1.0 - ACKLAM_P_LOW); }

// the inverse normal's branches with fused multiply-adds
__device__ __forceinline__ double gauss_tail(double P)
{
    const bool lower = P < ACKLAM_P_LOW;
    const double q = sqrt(-2.0 * log(lower ? P : 1.0 - P));
    double n = -7.784894002430293e-03, d = 7.784695709041462e-03;
    n = fma(n, q, -3.223964580411365e-01);
    d = fma(d, q, 3.224671290700398e-01);
    n = fma(n, q, -2.400758277161838e+00);
    d = fma(d, q, 2.445134137142996e+00);
    n = fma(n, q, -2.549732539343734e+00);
    d = fma(d, q, 3.754408661907416e+00);
    n = fma(n, q, 4.374664141464968e+00);
    d = fma(d, q, 1.0);
    n = fma(n, q, 2.938163982698783e+00);
    return (lower ? n : -n) / d;
}

__device__ __forceinline__ double gauss_central(double P)
{
    const double q = P - 0.5, r = q * q;
    double n = -3.969683028665376e+01, d = -5.447609879822406e+01;
    n = fma(n, r, 2.209460984245205e+02);
    d = fma(d, r, 1.615858368580409e+02);
    n = fma(n, r, -2.759285104469687e+02);
    d = fma(d, r, -1.556989798598866e+02);
    n = fma(n, r, 1.383577518672690e+02);
    d = fma(d, r, 6.680131188771972e+01);
    n = fma(n, r, -3.066479806614716e+01);
    d = fma(d, r, -1.328068155288572e+01);
    n = fma(n, r, 2.506628277459239e+00);
    d = fma(d, r, 1.0);
    return n * q / d;
}

// QeVarianceStep (single.cpp:344-368): psi = s2 / m^2 <= 1.5 is tested as s2 <= 1.5 m^2, and the
// quadratic branch takes c = 2 / psi from m and s2 and sqrt(c) sqrt(c - 1) as one square root (c
// capped where its square would overflow: the step's random part is below FP64 there)
__device__ double qe_step(double V, double Z, const CalibStep& C, const double* phi)
{
    const double m = fma(V, C.e, C.th1e), s2 = fma(V, C.qa, C.qb), m2 = m * m;
    if (s2 <= 1.5 * m2) {
        double c = 2.0 * m2 / s2;
        if (c > 1e150 && c < INFINITY) c = 1e150;
        const double b2 = c - 1.0 + sqrt(c * (c - 1.0));
        const double bz = sqrt(b2) + Z;
        return m / (1.0 + b2) * bz * bz;
    }
    // 1 - p = 2 m^2 / (s2 + m^2), 1 - u = Phi(-Z), 1 / beta = (s2 + m^2) / (2 m)
    const double num = s2 + m2;
    const double r = 2.0 * m2 / (num * thoth::phi_table(phi, -Z)); // (1 - p) / (1 - u)
    return r <= 1.0 ? 0.0 : log(r) * (num / (2.0 * m));
}

// LeveragedLogSpotStep (single.cpp:370-388) as carry + L b - L^2 d: its parts b and d
__device__ __forceinline__ void spot_parts(double Vp, double Vc, double Z, const CalibStep& C, double& b, double& d)
{
    if (C.flat == 0.0) {
        const double s = Vp + Vc;
        const double var = C.k3 * s;
        b = fma(sqrt(var < 0 ? 0.0 : var), Z, fma(C.r, Vc - Vp, fma(C.a1, s, C.k0)));
        d = C.a2 * s;
    } else {
        b = sqrt(Vp * C.dt) * Z;
        d = 0.5 * Vp * C.dt;
    }
}

// LeverageSurface::LayerAt (leverage_surface.cpp:19-40) at grid coordinate f on a layer in shared
// memory: the clamps select instead of branching (the interpolation index is clamped to the layer,
// and its value is only selected where the reference interpolates)
__device__ __forceinline__ double layer_at(const double* lev, int points, double f)
{
    const int last = points - 1;
    const bool inside = f > 0.0 && f < (double)last;
    const int i = inside ? (int)f : 0;
    const double w = f - (double)i;
    const double mid = fma(w, lev[i + 1] - lev[i], lev[i]);
    return !(f > 0.0) ? lev[0] : (f >= (double)last ? lev[last] : mid);
}

__device__ __forceinline__ void warp_sum(Fx128& a)
{
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const unsigned long long lo = __shfl_xor_sync(0xffffffffu, (unsigned long long)a.lo, o);
        const unsigned long long hi = __shfl_xor_sync(0xffffffffu, (unsigned long long)a.hi, o);
        fx_add(a, (uint64_t)lo, (uint64_t)hi);
    }
}

__device__ __forceinline__ unsigned long long now_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// wait until *flag >= want; false (status 2) after 2 s, or at once when another CTA failed
__device__ bool wait_for(const unsigned* flag, unsigned want, int* status)
{
    const unsigned long long t0 = now_ns();
    while (ld_acquire(flag) < want) {
        if (*(volatile int*)status != 0) return false;
        if (now_ns() - t0 > WAIT_LIMIT_NS) {
            atomicExch(status, 2);
            return false;
        }
        __nanosleep(32);
    }
    return true;
}

// a double's bit pattern as a signed integer with the same order (not a number: not_a_number first)
__device__ __forceinline__ long long order_key(double x)
{
    const long long b = __double_as_longlong(x);
    return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}

__device__ __forceinline__ bool not_a_number(double x)
{
    return ((unsigned long long)__double_as_longlong(x) << 1) > 0xffe0000000000000ull;
}

__device__ __forceinline__ double from_key(long long k)
{
    return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffll));
}

// An exact 128-bit sum added into global memory as limbs of 42, 42 and 44 bits, each into a word
// of its own by a reduction that returns nothing (as in american.cu): a CTA's sum is below 2^108,
// so fewer than 2^20 CTAs cannot overflow a word.
__device__ __forceinline__ void fx_red3(unsigned long long* dst, const Fx128& a)
{
    const uint64_t m = (1ull << 42) - 1;
    atomicAdd(dst, (unsigned long long)(a.lo & m));
    atomicAdd(dst + 1, (unsigned long long)((a.lo >> 42) | ((a.hi & ((1ull << 20) - 1)) << 22)));
    atomicAdd(dst + 2, (unsigned long long)(a.hi >> 20));
}

__device__ __forceinline__ Fx128 fx_load3(const unsigned long long* p)
{
    const uint64_t l0 = __ldcg(p), l1 = __ldcg(p + 1), l2 = __ldcg(p + 2);
    Fx128 r = {l0, 0};
    fx_add(r, l1 << 42, l1 >> 22);
    fx_add(r, 0, l2 << 20);
    return r;
}

// the two 64-bit words x adds to an Fx128 (x >= 0, truncated to 2^-64); bad when out of range
__device__ __forceinline__ void fx_words(double x, uint64_t& lo, uint64_t& hi, bool& bad)
{
    Fx128 t = {0, 0};
    fx_add_checked(t, x, bad);
    lo = t.lo;
    hi = t.hi;
}

// A bin's sum of v in shared memory, one particle a thread: v's fixed-point value (below 2^36 by
// its check, in units of 2^-64) as five 20-bit limbs, each added into its own 32-bit word, which
// 2^12 addends cannot overflow. (A 64-bit shared atomic is a compare-and-swap loop, and the
// particles crowd into a few bins.)
constexpr int BIN_LIMBS = 5;
static_assert(CALIB_THREADS <= 4096, "a limb's word holds 2^12 addends");

__device__ __forceinline__ uint64_t limb_bits(uint64_t lo, uint64_t hi, int i)
{
    const int b = 20 * i;
    const uint64_t w = b >= 64 ? hi >> (b - 64) : (b == 0 ? lo : (lo >> b) | (hi << (64 - b)));
    return w & 0xfffffu;
}

// one particle's state and what its next step has so far
struct Particle {
    double x, var, lns;
    double z1, z2, vc, sb, sd;
    uint64_t s[4];
};

// ONE: at most one particle a thread, held in registers
template <bool ONE>
__global__ void __launch_bounds__(CALIB_THREADS, 4) lsv_calib_kernel(const CalibArgs A, int G)
{
    extern __shared__ __align__(16) unsigned char s_dyn[]; // the jump table, then the layer [points]
    uint64_t* s_jtab = reinterpret_cast<uint64_t*>(s_dyn);
    double* s_layer = reinterpret_cast<double*>(s_dyn + sizeof(uint64_t) * CALIB_JTAB_WORDS);
    __shared__ long long s_min[CALIB_WARPS], s_max[CALIB_WARPS];
    __shared__ Fx128 s_sum[CALIB_WARPS];
    static_assert(CALIB_MAX_BINS >= CALIB_THREADS, "the tail queue fits the bins' arrays");
    __shared__ unsigned s_cnt[CALIB_MAX_BINS];
    __shared__ unsigned long long s_bin[2 * CALIB_MAX_BINS]; // 64-bit sums, or three of the limbs
    __shared__ double s_two[2 * CALIB_MAX_BINS];             // the others; then sums and means
    unsigned long long *s_blo = s_bin, *s_bhi = s_bin + CALIB_MAX_BINS;
    unsigned *s_l0 = reinterpret_cast<unsigned*>(s_bin), *s_l4 = reinterpret_cast<unsigned*>(s_two); // limbs 0..3, 4
    double *s_bsum = s_two, *s_mean = s_two + CALIB_MAX_BINS;
    // behind round A, when the bins are not in use: the tail draws, whose they are, their Gaussians
    double *s_qu = reinterpret_cast<double*>(s_bin), *s_z = s_two;
    unsigned short* s_qi = reinterpret_cast<unsigned short*>(s_cnt);
    __shared__ int s_qn[2];    // how many
    __shared__ double s_bc[4]; // min ln S, bin width and its reciprocal, ensemble mean of v
    __shared__ int s_flat;             // every particle at one spot
    __shared__ unsigned short s_span[2]; // the layer's points around the ensemble: first, one past the last
    const int T = G * CALIB_THREADS; // the CTAs past G have no particles and take no part in the rounds
    const int t = threadIdx.x, gt = blockIdx.x * CALIB_THREADS + t;
    const int lane = t & 31, warp = t >> 5;
    const int P = (int)blockIdx.x < G ? A.P : 0, bins = A.bins;
    const bool writes = (int)blockIdx.x == A.writer;
    const int R = ONE ? 1 : (A.P + T - 1) / T; // particles a thread, the same for every thread
    bool bad = false;
    int tog = 0;
    Particle q{};

    for (int i = t; i < (int)CALIB_JTAB_WORDS; i += CALIB_THREADS) s_jtab[i] = A.jtab[i];
    if (t < 2) s_qn[t] = 0;
    __syncthreads();
    // the ensemble at today; particle p's generator at draw 2p of the stream
    for (int p = gt; p < P; p += T) {
        q.x = 0.0;
        q.var = A.v0;
        q.lns = A.ln_s0;
        for (int w = 0; w < 4; w++) q.s[w] = A.seed_state[w];
        const uint64_t off = 2ull * (uint64_t)p;
        for (int i = 0; i < CALIB_JUMP_BITS; i++)
            if ((off >> i) & 1u) xo_jump(A.jpow + 4 * i, q.s);
        if (!ONE) {
            A.x[p] = q.x;
            A.var[p] = q.var;
            A.lns[p] = q.lns;
            for (int w = 0; w < 4; w++) A.rng[(size_t)w * P + p] = q.s[w];
        }
    }

    unsigned round = 0;
    auto arrive = [&] { // after a __syncthreads that follows every contribution's fence
        ++round;
        if (t == 0 && P > 0) atomicAdd(A.bar, 1u);
    };
    for (int k = 0; k < A.n; k++) {
        // ---- round A: extremes of ln S (as integer keys), sum of v ----
        if (P > 0) {
            long long mn = 0x7fffffffffffffffll, mx = -0x7fffffffffffffffll;
            Fx128 sv = {0, 0};
            for (int p = gt; p < P; p += T) {
                if (!ONE) {
                    q.lns = A.lns[p];
                    q.var = A.var[p];
                }
                if (!not_a_number(q.lns)) { // a particle lost to a layer without a value moves no bin
                    const long long key = order_key(q.lns);
                    mn = min(mn, key);
                    mx = max(mx, key);
                }
                fx_add_checked(sv, q.var, bad);
            }
#pragma unroll
            for (int o = 16; o; o >>= 1) {
                mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
                mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            }
            warp_sum(sv);
            if (lane == 0) {
                s_min[warp] = mn;
                s_max[warp] = mx;
                s_sum[warp] = sv;
            }
            if (bad) atomicExch(A.status, 3);
            __syncthreads();
            if (t == 0) {
                long long cm = s_min[0], cx = s_max[0];
                Fx128 cs = s_sum[0];
                for (int w = 1; w < CALIB_WARPS; w++) {
                    cm = min(cm, s_min[w]);
                    cx = max(cx, s_max[w]);
                    fx_add(cs, s_sum[w]);
                }
                if (cm <= cx) { // a CTA whose particles are all lost adds nothing
                    atomicMin(A.kmin + k, cm);
                    atomicMax(A.kmax + k, cx);
                    fx_red3(A.vsum + 3 * (size_t)k, cs);
                }
                __threadfence();
            }
        }
        arrive();
        // ---- behind round A: the Gaussians of the step into date k in draw order (the variance's
        // first) and the generator's jump ----
        if (k > 0 && P > 0)
            for (int it = 0; it < R; ++it, tog ^= 1) {
                const int p = gt + it * T;
                const bool act = p < P;
                bool tail1 = false, tail2 = false;
                if (act) {
                    if (!ONE)
                        for (int w = 0; w < 4; w++) q.s[w] = A.rng[(size_t)w * P + p];
                    const double u1 = uniform53(q.s), u2 = uniform53(q.s);
                    tail1 = in_tail(u1);
                    tail2 = in_tail(u2);
                    if (tail1) {
                        const int o = atomicAdd(&s_qn[tog], 1);
                        s_qu[o] = u1;
                        s_qi[o] = (unsigned short)(2 * t);
                    }
                    if (tail2) {
                        const int o = atomicAdd(&s_qn[tog], 1);
                        s_qu[o] = u2;
                        s_qi[o] = (unsigned short)(2 * t + 1);
                    }
                    q.z1 = gauss_central(u1);
                    q.z2 = gauss_central(u2);
                }
                __syncthreads();
                // the CTA's tail draws, a dozen of 256: one warp's work while the others go on
                for (int o = t; o < s_qn[tog]; o += CALIB_THREADS) s_z[s_qi[o]] = gauss_tail(s_qu[o]);
                if (t == 0) s_qn[tog ^ 1] = 0;
                if (act) xo_jump_tab(s_jtab, q.s);
                __syncthreads();
                if (tail1) q.z1 = s_z[2 * t];
                if (tail2) q.z2 = s_z[2 * t + 1];
                if (!ONE && act) {
                    for (int w = 0; w < 4; w++) A.rng[(size_t)w * P + p] = q.s[w];
                    A.z1[p] = q.z1;
                    A.z2[p] = q.z2;
                }
            }
        __syncthreads(); // the Gaussians are read: the arrays below are theirs
        for (int b = t; b < CALIB_MAX_BINS; b += CALIB_THREADS) {
            s_cnt[b] = 0;
            s_blo[b] = 0; // or limbs 0..3
            s_bhi[b] = 0;
            s_l4[b] = 0;
        }
        // one thread a warp forms its share of the round's results: the bins' origin and width; their
        // reciprocal; the layer's points around the ensemble (below the lowest, above the highest);
        // the ensemble's mean
        bool ok = true;
        if (lane == 0) {
            ok = wait_for(A.bar, round * (unsigned)G, A.status);
            if (ok && warp == 1) {
                s_bc[3] = fx_to_double(fx_load3(A.vsum + 3 * (size_t)k)) * A.rP;
            } else if (ok) {
                const double gmn = from_key((long long)__ldcg((const unsigned long long*)(A.kmin + k)));
                const double gmx = from_key((long long)__ldcg((const unsigned long long*)(A.kmax + k)));
                if (warp == 0) {
                    s_bc[0] = gmn;
                    s_bc[1] = (gmx - gmn) * A.rbins;
                    s_flat = gmx - gmn < 1e-10;
                } else if (warp == 2) {
                    s_bc[2] = 1.0 / ((gmx - gmn) * A.rbins);
                } else {
                    const double off = (double)A.offset[k], top = (double)A.points;
                    s_span[0] = (unsigned short)fmin(fmax(floor(fma(gmn, A.rln_step[k], -off)) - 1.0, 0.0), top - 1.0);
                    s_span[1] = (unsigned short)fmin(fmax(floor(fma(gmx, A.rln_step[k], -off)) + 3.0, 1.0), top);
                }
            }
        }
        // The four waits end apart, and where another CTA has failed some of them fail and others still
        // find the count complete: the CTA goes on only if all four did, and so wrote their results
        if (!__syncthreads_and(ok)) return;
        const bool flat = s_flat != 0;
        const double bmn = s_bc[0], width = s_bc[1], rwidth = s_bc[2], fallback = s_bc[3];
        // the layer's points this CTA needs: those around the ensemble, or all to write out
        const int i0 = writes ? 0 : s_span[0];
        const int i1 = writes ? A.points : s_span[1];

        if (!flat) {
            // ---- round B: per-bin counts and sums of v ----
            if (P > 0) {
                for (int p = gt; p < P; p += T) {
                    if (!ONE) {
                        q.lns = A.lns[p];
                        q.var = A.var[p];
                    }
                    int b = (int)((q.lns - bmn) * rwidth);
                    b = b < 0 ? 0 : (b > bins - 1 ? bins - 1 : b);
                    uint64_t lo, hi;
                    fx_words(q.var, lo, hi, bad);
                    atomicAdd(&s_cnt[b], 1u);
                    if (ONE) {
#pragma unroll
                        for (int i = 0; i < BIN_LIMBS; i++)
                            atomicAdd(i < 4 ? s_l0 + i * CALIB_MAX_BINS + b : s_l4 + b, (unsigned)limb_bits(lo, hi, i));
                    } else {
                        const unsigned long long old = atomicAdd(&s_blo[b], (unsigned long long)lo);
                        atomicAdd(&s_bhi[b], (unsigned long long)(hi + ((uint64_t)old + lo < lo ? 1u : 0u)));
                    }
                }
                __syncthreads();
                for (int b = t; b < bins; b += CALIB_THREADS)
                    if (s_cnt[b]) {
                        atomicAdd(A.bcnt + (size_t)k * bins + b, s_cnt[b]);
                        Fx128 v = {0, 0};
                        if (ONE) {
                            for (int i = 0; i < BIN_LIMBS; i++) {
                                const uint64_t w = i < 4 ? s_l0[i * CALIB_MAX_BINS + b] : s_l4[b];
                                const int sh = 20 * i;
                                if (sh >= 64) fx_add(v, 0, w << (sh - 64));
                                else fx_add(v, w << sh, sh ? w >> (64 - sh) : 0);
                            }
                        } else {
                            v = Fx128{s_blo[b], s_bhi[b]};
                        }
                        fx_red3(A.bsum + 3 * ((size_t)k * bins + b), v);
                        __threadfence();
                    }
                if (bad) atomicExch(A.status, 3);
            }
            __syncthreads();
            arrive();
        }
        // ---- behind round B: the variance step and the log-spot step's parts ----
        const CalibStep C = A.steps[k];
        if (k > 0)
            for (int p = gt; p < P; p += T) {
                if (!ONE) {
                    q.var = A.var[p];
                    q.z1 = A.z1[p];
                    q.z2 = A.z2[p];
                }
                q.vc = qe_step(q.var, q.z1, C, A.phi);
                spot_parts(q.var, q.vc, q.z2, C, q.sb, q.sd);
                if (!ONE) {
                    A.vc[p] = q.vc;
                    A.sb[p] = q.sb;
                    A.sd[p] = q.sd;
                }
            }
        if (!flat) {
            // the layer's points on the bins' grid
            const double x0 = fma(0.5, width, bmn), ls = A.ln_step[k];
            const int64_t off = A.offset[k];
            for (int i = i0 + t; i < i1; i += CALIB_THREADS) s_layer[i] = ((double)(off + i) * ls - x0) * rwidth;
            ok = t != 0 || wait_for(A.bar, round * (unsigned)G, A.status);
            if (!__syncthreads_and(ok)) return;
            for (int b = t; b < bins; b += CALIB_THREADS) {
                s_bsum[b] = fx_to_double(fx_load3(A.bsum + 3 * ((size_t)k * bins + b)));
                s_cnt[b] = __ldcg(A.bcnt + (size_t)k * bins + b);
            }
            __syncthreads();
            // populated bins, then each thin bin from its nearest populated one, left first
            // (one thread a bin: the fill reads only populated bins)
            const unsigned mc = (unsigned)A.min_count;
            for (int b = t; b < bins; b += CALIB_THREADS) {
                int from = s_cnt[b] >= mc ? b : -1;
                for (int d = 1; d < bins && from < 0; d++) {
                    if (b - d >= 0 && s_cnt[b - d] >= mc) from = b - d;
                    else if (b + d < bins && s_cnt[b + d] >= mc) from = b + d;
                }
                s_mean[b] = from >= 0 ? s_bsum[from] / s_cnt[from] : fallback;
            }
            __syncthreads();
        }
        // ---- layer k from the conditional variance of the bins (the same in every CTA) ----
        for (int i = i0 + t; i < i1; i += CALIB_THREADS) {
            double ev = fallback;
            if (!flat) {
                // linear between bin centres, the outer bins' means beyond them
                const double f = fmin(fmax(s_layer[i], 0.0), (double)(bins - 1));
                const int j = min((int)f, max(bins - 2, 0));
                const double m0 = s_mean[j];
                ev = fma(f - (double)j, s_mean[min(j + 1, bins - 1)] - m0, m0);
            }
            if (ev < A.min_cv) ev = A.min_cv;
            double L = A.local_vol[(size_t)k * A.points + i] * rsqrt(ev);
            L = L < A.lmin ? A.lmin : (L > A.lmax ? A.lmax : L);
            s_layer[i] = L;
            if (writes) A.lev[(size_t)k * A.points + i] = L;
        }
        __syncthreads();
        if (k == 0) continue;

        // ---- the step into date k with layer k ----
        const double rls = A.rln_step[k], f0 = A.f0[k];
        for (int p = gt; p < P; p += T) {
            if (!ONE) {
                q.x = A.x[p];
                q.lns = A.lns[p];
                q.vc = A.vc[p];
                q.sb = A.sb[p];
                q.sd = A.sd[p];
            }
            const double L = layer_at(s_layer, A.points, fma(q.x, rls, f0));
            const double step = fma(-L * L, q.sd, fma(L, q.sb, C.carry));
            q.var = q.vc;
            q.x += step;
            q.lns += step;
            if (!ONE) {
                A.var[p] = q.var;
                A.x[p] = q.x;
                A.lns[p] = q.lns;
            }
        }
    }
}

// ---- host: GF(2) polynomials of degree < 256 as 4 words, bit i = coefficient of x^i ----
struct Poly {
    uint64_t w[4];
};

std::mutex g_chi_mu;
bool g_chi_ready = false;
Poly g_chi;                           // chi - x^256
Poly g_pow2[CALIB_JUMP_BITS + 24];    // x^(2^i) mod chi

bool bit(const Poly& p, int i) { return (p.w[i >> 6] >> (i & 63)) & 1u; }

// a b mod chi (Horner over the bits of b, high to low)
Poly mulmod(const Poly& a, const Poly& b)
{
    Poly r = {{0, 0, 0, 0}};
    for (int i = 255; i >= 0; i--) {
        const bool top = (r.w[3] >> 63) & 1u; // r x overflows into x^256 = chi - x^256
        r.w[3] = (r.w[3] << 1) | (r.w[2] >> 63);
        r.w[2] = (r.w[2] << 1) | (r.w[1] >> 63);
        r.w[1] = (r.w[1] << 1) | (r.w[0] >> 63);
        r.w[0] <<= 1;
        if (top)
            for (int j = 0; j < 4; j++) r.w[j] ^= g_chi.w[j];
        if (bit(b, i))
            for (int j = 0; j < 4; j++) r.w[j] ^= a.w[j];
    }
    return r;
}

// chi from the minimal polynomial of one state bit's sequence (Berlekamp-Massey over GF(2));
// the transition's characteristic polynomial is primitive of degree 256, so any nonzero
// sequence has it as its minimal polynomial
bool find_chi()
{
    const int N = 512;
    std::vector<uint8_t> s(N);
    uint64_t st[4];
    xo_seed_state(1, st);
    for (int i = 0; i < N; i++) {
        s[i] = (uint8_t)(st[0] & 1u);
        xo_advance(st);
    }
    std::vector<uint8_t> C(N + 1, 0), B(N + 1, 0), Tm;
    C[0] = B[0] = 1;
    int L = 0, m = 1;
    for (int n = 0; n < N; n++) {
        uint8_t d = s[n];
        for (int i = 1; i <= L; i++) d ^= (uint8_t)(C[i] & s[n - i]);
        if (!d) {
            m++;
        } else if (2 * L <= n) {
            Tm = C;
            for (int i = 0; i + m <= N; i++) C[i + m] ^= B[i];
            L = n + 1 - L;
            B = Tm;
            m = 1;
        } else {
            for (int i = 0; i + m <= N; i++) C[i + m] ^= B[i];
            m++;
        }
    }
    if (L != 256) return false;
    // chi(x) = x^256 C(1/x): the coefficient of x^(256 - i) is C[i]
    Poly c = {{0, 0, 0, 0}};
    for (int i = 1; i <= 256; i++)
        if (C[i]) {
            const int e = 256 - i;
            c.w[e >> 6] |= 1ull << (e & 63);
        }
    g_chi = c;
    Poly x = {{2, 0, 0, 0}};
    g_pow2[0] = x;
    for (int i = 1; i < CALIB_JUMP_BITS + 24; i++) g_pow2[i] = mulmod(g_pow2[i - 1], g_pow2[i - 1]);
    return true;
}

// ---- the reference Rng's stream for the book kernel's tail dimensions -------------------
__constant__ uint64_t c_xo_pow2[64 * 4]; // x^(2^i) mod chi for i < 64

struct TailSeed {
    uint64_t s[4];
};

constexpr int TAIL_THREADS = 128;
constexpr int TAIL_WARPS = TAIL_THREADS / 32;
constexpr int TAIL_PATHS_PER_THREAD = 16;
// thread k draws the tail Gaussians of paths [16 k, 16 k + 16): one jump to its first path's
// place in the stream (p dt draws in: the binary powers of x), then its paths' draws in stream
// order, as the reference's NextPath draws them. A draw in the central region is inverted at
// once; one in a tail (4.85 % of them) waits in its warp's queue in shared memory, and 32
// queued draws are inverted at once on the warp's 32 lanes, so the logarithm runs on full
// warps instead of on most warps' iterations.
__global__ void __launch_bounds__(TAIL_THREADS) tail_normals_kernel(const TailSeed s0, int dt, int64_t paths,
                                                                    float* __restrict__ out)
{
    __shared__ double q_u[TAIL_WARPS][64];
    __shared__ uint32_t q_i[TAIL_WARPS][64];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t p0 = ((int64_t)blockIdx.x * TAIL_THREADS + threadIdx.x) * TAIL_PATHS_PER_THREAD;
    const bool live = p0 < paths;
    if (__all_sync(0xffffffffu, !live)) return; // warp-uniform
    const int np = live ? (int)(paths - p0 < TAIL_PATHS_PER_THREAD ? paths - p0 : TAIL_PATHS_PER_THREAD) : 0;
    uint64_t s[4] = {s0.s[0], s0.s[1], s0.s[2], s0.s[3]};
    if (live) {
        const uint64_t pos = (uint64_t)p0 * (uint64_t)dt;
        for (int i = 0; i < 64; i++)
            if ((pos >> i) & 1u) xo_jump(c_xo_pow2 + 4 * i, s);
    }
    int qn = 0; // the warp's queue length (the same on every lane)
    for (int pl = 0; pl < TAIL_PATHS_PER_THREAD; pl++) {
        const bool act = pl < np;
        for (int d = 0; d < dt; d++) {
            double u = 0.0;
            uint32_t idx = 0;
            bool tail = false;
            if (act) {
                const double u0 = (double)(xo_next(s) >> 11) * (1.0 / 9007199254740992.0);
                u = u0 > 0.0 ? u0 : (1.0 / 9007199254740992.0);
                idx = (uint32_t)((size_t)d * (size_t)paths + (size_t)(p0 + pl)); // < 2^31: the table's size limit
                tail = u < ACKLAM_P_LOW || !(u <= 1.0 - ACKLAM_P_LOW);
                if (!tail) out[idx] = (float)acklam_central(u);
            }
            const unsigned m = __ballot_sync(0xffffffffu, tail);
            if (tail) {
                const int slot = qn + __popc(m & ((1u << lane) - 1u)); // < 63
                q_u[w][slot] = u;
                q_i[w][slot] = idx;
            }
            qn += __popc(m);
            if (qn >= 32) { // 32 to 63 entries: invert the first 32, keep the rest
                __syncwarp();
                out[q_i[w][lane]] = (float)acklam_tail(q_u[w][lane]);
                const int rest = qn - 32;
                double mu = 0.0;
                uint32_t mi = 0;
                if (lane < rest) {
                    mu = q_u[w][32 + lane];
                    mi = q_i[w][32 + lane];
                }
                __syncwarp();
                if (lane < rest) {
                    q_u[w][lane] = mu;
                    q_i[w][lane] = mi;
                }
                __syncwarp();
                qn = rest;
            }
        }
    }
    __syncwarp();
    if (lane < qn) out[q_i[w][lane]] = (float)acklam_tail(q_u[w][lane]);
}

} // namespace

void xo_seed_state(uint64_t seed, uint64_t s[4])
{
    uint64_t z = seed;
    for (int i = 0; i < 4; i++) {
        z += 0x9e3779b97f4a7c15ULL;
        uint64_t x = z;
        x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
        x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
        s[i] = x ^ (x >> 31);
    }
}

void xo_advance(uint64_t s[4]) { xo_step(s); }

bool xo_jump_poly(uint64_t d, uint64_t out[4])
{
    {
        std::lock_guard<std::mutex> lk(g_chi_mu);
        if (!g_chi_ready) {
            if (!find_chi()) return false;
            g_chi_ready = true;
        }
    }
    Poly r = {{1, 0, 0, 0}};
    for (int i = 0; i < 64; i++)
        if ((d >> i) & 1u) {
            if (i >= CALIB_JUMP_BITS + 24) return false;
            r = mulmod(r, g_pow2[i]);
        }
    for (int j = 0; j < 4; j++) out[j] = r.w[j];
    return true;
}

void xo_apply_jump(const uint64_t poly[4], uint64_t s[4]) { xo_jump(poly, s); }

void xo_jump_table(const uint64_t poly[4], uint64_t* tab)
{
    // column i of the jump matrix: the jump of the state with only bit i set
    std::vector<uint64_t> col(256 * 4);
    for (int i = 0; i < 256; i++) {
        uint64_t e[4] = {0, 0, 0, 0};
        e[i >> 6] = 1ull << (i & 63);
        xo_jump(poly, e);
        for (int w = 0; w < 4; w++) col[i * 4 + w] = e[w];
    }
    for (int n = 0; n < 64; n++)
        for (int v = 0; v < 16; v++) {
            uint64_t r[4] = {0, 0, 0, 0};
            for (int b = 0; b < 4; b++)
                if ((v >> b) & 1)
                    for (int w = 0; w < 4; w++) r[w] ^= col[(4 * n + b) * 4 + w];
            for (int w = 0; w < 4; w++) tab[(n * 16 + v) * 4 + w] = r[w];
        }
}

int calib_max_grid(int sms, size_t smem)
{
    int per = 0, per1 = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, lsv_calib_kernel<false>, CALIB_THREADS, smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per1, lsv_calib_kernel<true>, CALIB_THREADS, smem) != cudaSuccess)
        return 0;
    return (per < per1 ? per : per1) * sms;
}

cudaError_t launch_calib(const CalibArgs& A, int grid, int cap, size_t smem, cudaStream_t st)
{
    // one more CTA, without particles, writes the layers out where the device has room for it
    CalibArgs a = A;
    int G = grid;
    if (grid < cap) ++grid;
    a.writer = grid - 1;
    void* args[] = {&a, &G};
    auto k = (int64_t)G * CALIB_THREADS >= A.P ? lsv_calib_kernel<true> : lsv_calib_kernel<false>;
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k), dim3(grid), dim3(CALIB_THREADS), args, smem, st);
}

cudaError_t tail_normals_prepare()
{
    static std::mutex mu;
    static bool ready[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu);
    if (dev >= 0 && dev < 64 && ready[dev]) return cudaSuccess;
    std::vector<uint64_t> pw(64 * 4);
    for (int i = 0; i < 64; i++)
        if (!xo_jump_poly(1ull << i, pw.data() + 4 * i)) return cudaErrorUnknown;
    e = cudaMemcpyToSymbol(c_xo_pow2, pw.data(), sizeof(uint64_t) * pw.size());
    if (e == cudaSuccess && dev >= 0 && dev < 64) ready[dev] = true;
    return e;
}

cudaError_t launch_tail_normals(uint64_t seed, int dt, int64_t paths, float* out, cudaStream_t st)
{
    if (dt <= 0 || paths <= 0) return cudaSuccess;
    TailSeed s0;
    xo_seed_state(seed, s0.s);
    const int64_t threads = (paths + TAIL_PATHS_PER_THREAD - 1) / TAIL_PATHS_PER_THREAD;
    const unsigned blocks = (unsigned)((threads + TAIL_THREADS - 1) / TAIL_THREADS);
    tail_normals_kernel<<<blocks, TAIL_THREADS, 0, st>>>(s0, dt, paths, out);
    return cudaGetLastError();
}
