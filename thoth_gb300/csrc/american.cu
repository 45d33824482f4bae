// american.cu — Longstaff-Schwartz exercise of a vanilla on its asset's stored paths, the
// algorithm of pricer_mcl_american.cpp:263-447 (FitAmericanPolicy / ApplyAmericanPolicy)
// with the normal-equation solve of helpers/maths.cpp:354-381 and 419-470.
//
// Fit: one cooperative, persistent launch fits every contract of an asset on the same stored
// paths, walking the exercise dates backwards. A date's regression needs the sums of the powers of
// the in-the-money paths' moneyness, which no decision changes, and the sums with their cashflows,
// which date t + 1's decisions change. So while date t's policy is being found, the CTAs already
// list date t - 1's in-the-money paths and form its moneyness sums, and the normal equations'
// matrix is factored beside the cashflow sums: the round of all CTAs that each date needs (publish,
// wait, solve) lies behind the next date's work. Every CTA solves from the contracts' per-date
// totals (exact 128-bit integer atomics) itself, one contract a lane, so no CTA releases the
// others. The decision at date t + 1 is taken where its cashflow is used, on the way to date t, and
// a path keeps the date of its earliest exercise: the frozen policy's exercise on the same paths
// (the same test at the same dates), so the premium comes out of the fit without a second walk.
//
// What bounds the fit is FP64: an SM finishes one warp's instruction in 16 clocks, and a date needs
// one product a path and eight operations an in-the-money path (2^20 paths, half of them in the
// money: 16.6 thousand clocks of the 25 thousand a date takes; with a publish-and-release per date,
// FP64 decisions, FP64 conversions and branches between the products it took 71 thousand).
// 2^20 Heston paths x 365 dates: 13.4 ms before, 4.7 ms.
//
// Apply: the frozen policy on another path set (the bumped scenarios of the Greeks), one
// forward walk per path that stops at the first exercise.
//
// Sums are exact (exact.cuh), so the regressions, the decisions and the premium do not
// depend on the grid; the arithmetic of each addend, of the solve and of the decision is
// the reference's, operation for operation, in round-to-nearest double with no fused
// multiply-adds (those inside the moneyness quotient give its correctly rounded value).
// GB300 runs FP64 at a small fraction of its FP32 rate, so the per-path work keeps FP64
// to what the result depends on: the in-the-money test is an integer compare on the
// spot's bits, the quotient S / norm is two operations where norm has few digits and five
// elsewhere, spots widen by integer operations, and the exercise test runs in FP32 wherever a
// proven margin shows that it decides as the FP64 test (screen_exercise), which then runs only in a
// thin band around the boundary (0.3 paths in a thousand).
#include "american.cuh"

#include <type_traits>

using namespace lsm;

namespace {

constexpr unsigned long long BARRIER_LIMIT_NS = 2000000000ull; // 2 s

// intrinsic(S) > 0, decided on the single-precision bits of S (integer compare; the
// threshold is exact, see itm_bits)
template <class K>
__device__ __forceinline__ bool in_the_money(float s, const K& A)
{
    const int b = __float_as_int(s);
    return A.call ? b >= A.itm_bits : b <= A.itm_bits;
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

__device__ __forceinline__ void prefetch_l2(const void* p)
{
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// wait until *flag >= want; false (status 2) after 2 s, or soon when another CTA has failed: the
// caller stops working and waits no more
__device__ bool wait_for(const unsigned* flag, unsigned want, int* status)
{
    const unsigned long long t0 = now_ns();
    for (unsigned polls = 1; ld_acquire(flag) < want; ++polls) {
        if (polls % 64) continue;
        if (*(volatile int*)status != 0) return false;
        if (now_ns() - t0 > BARRIER_LIMIT_NS) {
            atomicExch(status, 2);
            return false;
        }
    }
    return true;
}

// An exact 128-bit sum split into three limbs of 42, 42 and 44 bits, each added into its own
// 64-bit word by a reduction that returns nothing (no round trip for a carry). The limbs of a
// per-CTA sum are below 2^44, so fewer than 2^20 CTAs cannot overflow a word; the solving CTA
// reassembles the exact value.
constexpr uint64_t LIMB42 = (1ull << 42) - 1;

__device__ __forceinline__ void fx_red3(unsigned long long* dst, const Fx128& a)
{
    atomicAdd(dst, (unsigned long long)(a.lo & LIMB42));
    atomicAdd(dst + 1, (unsigned long long)((a.lo >> 42) | ((a.hi & ((1ull << 20) - 1)) << 22)));
    atomicAdd(dst + 2, (unsigned long long)(a.hi >> 20));
}

__device__ __forceinline__ Fx128 fx_from3(const unsigned long long* src)
{
    const uint64_t l0 = __ldcg(src), l1 = __ldcg(src + 1), l2 = __ldcg(src + 2);
    Fx128 r = {l0, 0};
    fx_add(r, l1 << 42, l1 >> 22);
    fx_add(r, 0, l2 << 20);
    return r;
}

// a float spot as a double, without the conversion's pass through the FP64 unit (out of line where
// it is needed: the compiler would convert every spot and select)
__device__ __noinline__ double widen_rare(float s) { return (double)s; }
__device__ __forceinline__ double widen(float s)
{
    const unsigned b = (unsigned)__float_as_int(s), a = b & 0x7fffffffu;
    if (a - 0x00800000u < 0x7f000000u)
        return __hiloint2double((int)((a >> 3) + 0x38000000u | (b & 0x80000000u)), (int)(b << 29));
    return widen_rare(s); // zero, subnormal, infinite or NaN
}

// phi (S - K) in double precision, the reference's intrinsic value of an in-the-money spot: one FP64
// operation (K - S rounds to -(S - K))
template <class K>
__device__ __forceinline__ double itm_value(float sf, const K& A)
{
    const double v = __dsub_rn(widen(sf), A.strike);
    return __hiloint2double(__double2hiint(v) ^ (A.call ? 0 : (int)0x80000000), __double2loint(v));
}

// max(phi (S - K), 0): payoff_vanilla with a floor at 0 (helpers/finance.cpp:9-32); a spot that is
// not a number is paid, so that the sums' checks see it
template <class K>
__device__ __forceinline__ double payoff(float sf, const K& A)
{
    return in_the_money(sf, A) || sf != sf ? itm_value(sf, A) : 0.0;
}

// CTA-wide exact sum of one accumulator per thread into out (thread 0 writes)
template <int WARPS>
__device__ void block_sum(Fx128 a, Fx128 (&s_w)[WARPS][LSM_NACC], int slot, Fx128* out)
{
    warp_sum(a);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) s_w[warp][slot] = a;
    __syncthreads();
    if (threadIdx.x == 0) {
        Fx128 s = {0, 0};
        for (int w = 0; w < WARPS; w++) fx_add(s, s_w[w][slot]);
        *out = s;
    }
    __syncthreads();
}

// The fit's CTA: 16 warps walk the paths; two more publish the CTA's sums, wait for the others' and
// find the policies, one (the factorer) from the moneyness sums, one (the solver) from the cashflow
// sums. Both are on the SM's scheduler 0 (warps 0 and 4).
constexpr int FIT_WARPS = 18, FIT_FACTORER = 0, FIT_SOLVER = 4;
constexpr int FIT_THREADS = 32 * FIT_WARPS;
constexpr int FIT_WALKERS = FIT_THREADS - 64;
constexpr int FIT_MIN_PATHS = 128; // paths a CTA walks before the grid grows: a chunk a scheduler
constexpr int FIT_SOLVER_CHUNKS = 24; // see lsm_fit_kernel
constexpr int FIT_AHEAD = 256; // elements of a block requested ahead, paths in global memory (512: 2 % slower)
constexpr int SUM_LIMBS = 5; // a warp's 128-bit sum in 26-bit limbs, added in shared memory

constexpr int FIT_X = 5, FIT_Y = 3; // a date's moneyness sums (with the count), its cashflow sums
static_assert(FIT_X + FIT_Y == LSM_PART, "the totals hold both");
// A contract's sums in shared memory: the moneyness sums of even and of odd dates, the cashflow
// sums. The walkers form date t - 1's moneyness sums before they wait for date t's policy, and the
// solver may still hold date t's then; date t - 2's and the next cashflow sums come behind that wait.
constexpr int FIT_SUMS = 2 * FIT_X + FIT_Y;

// named barriers: date t's moneyness sums are in shared memory (by the parity of t, as the
// sums); its cashflow sums; its policy; its factors, from factorer to solver (by parity)
enum { BAR_X = 1, BAR_Y = 3, BAR_POLICY = 4, BAR_FACTOR = 5 };
constexpr int FIT_HANDOVER = FIT_WALKERS + 32; // the walkers and one of the two
template <int N>
__device__ __forceinline__ void bar_sync(int id)
{
    __syncwarp();
    asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(N) : "memory");
}
template <int N>
__device__ __forceinline__ void bar_arrive(int id)
{
    __syncwarp();
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(N) : "memory");
}

// the Cholesky factor of one date's normal equations
struct FitFactor {
    Pivot p1, p2, p3;
    double l21, l31, l32;
    int ok;
};

// one contract's policy at a date: coefficients and screen
struct FitPolicy {
    double b[3], df; // df: the discount from this date to the one before
    LsmScreen s;
};

// shared memory of one contract beside its paths
constexpr size_t FIT_CONTRACT_BYTES = sizeof(LsmContract) + 2 * sizeof(FitFactor) + sizeof(FitPolicy) +
                                      sizeof(unsigned) * FIT_SUMS * SUM_LIMBS + sizeof(int) * FIT_WARPS;

static_assert(sizeof(LsmContract) % 16 == 0 && 2 * sizeof(FitFactor) % 16 == 0 && sizeof(FitPolicy) % 16 == 0,
              "the policies lie on 16-byte boundaries behind the contracts and factors");

__host__ __device__ inline size_t fit_control_bytes(int C) { return (FIT_CONTRACT_BYTES * (size_t)C + 15) & ~size_t(15); }

// and of its paths: spots of two dates, then per contract cashflow, list moneyness and list index
__host__ __device__ inline size_t fit_path_bytes(int C, int64_t ppc)
{
    return (size_t)ppc * (2 * sizeof(float) + (size_t)C * (2 * sizeof(double) + sizeof(uint16_t)));
}

// the warp's sums of four accumulators: halves of them change hands, so a lane adds 5 values where
// four butterflies add 20; lanes 0, 8, 16, 24 are left with sums 0..3, which they add into dst
__device__ __forceinline__ void warp_sum4(Fx128 (&q)[4], int lane, unsigned* dst, int n)
{
    auto swap = [](const Fx128& give, int o) {
        Fx128 r;
        r.lo = __shfl_xor_sync(0xffffffffu, (unsigned long long)give.lo, o);
        r.hi = __shfl_xor_sync(0xffffffffu, (unsigned long long)give.hi, o);
        return r;
    };
    const bool up = lane & 16, odd = lane & 8;
    Fx128 k0 = up ? q[2] : q[0], k1 = up ? q[3] : q[1];
    const Fx128 g0 = up ? q[0] : q[2], g1 = up ? q[1] : q[3];
    fx_add(k0, swap(g0, 16));
    fx_add(k1, swap(g1, 16));
    Fx128 k = odd ? k1 : k0;
    const Fx128 g = odd ? k0 : k1;
    fx_add(k, swap(g, 8));
#pragma unroll
    for (int o = 4; o; o >>= 1) fx_add(k, swap(k, o));
    const int i = lane >> 3;
    if ((lane & 7) == 0 && i < n) {
        constexpr unsigned L26 = (1u << 26) - 1;
        unsigned* d = dst + i * SUM_LIMBS;
        atomicAdd(d, (unsigned)k.lo & L26);
        atomicAdd(d + 1, (unsigned)(k.lo >> 26) & L26);
        atomicAdd(d + 2, (unsigned)((k.lo >> 52) | (k.hi << 12)) & L26);
        atomicAdd(d + 3, (unsigned)(k.hi >> 14) & L26);
        atomicAdd(d + 4, (unsigned)(k.hi >> 40));
    }
}

// the limbs' value (each below 2^30: 16 warps), and the limbs cleared for the next date
__device__ __forceinline__ Fx128 take_limbs(unsigned* d)
{
    Fx128 r = {d[0], 0};
    fx_add(r, (uint64_t)d[1] << 26, 0);
    fx_add(r, (uint64_t)d[2] << 52, (uint64_t)d[2] >> 12);
    fx_add(r, 0, (uint64_t)d[3] << 14);
    fx_add(r, 0, (uint64_t)d[4] << 40);
#pragma unroll
    for (int i = 0; i < SUM_LIMBS; i++) d[i] = 0;
    return r;
}

// the factor of (X^T X) for X = {1, m, m^2}: Cholesky A = L L^T (maths.cpp:354-381), the
// operations of a column loop in its order
__device__ void factor3(double n, double s1, double s2, double s3, double s4, FitFactor& F)
{
    F.ok = 0;
    if (n <= 0.0) return;
    F.p1 = pivot(__dsqrt_rn(n));
    F.l21 = __ddiv_rn(s1, F.p1.l);
    F.l31 = __ddiv_rn(s2, F.p1.l);
    const double p22 = __dsub_rn(s2, __dmul_rn(F.l21, F.l21));
    if (p22 <= 0.0) return;
    F.p2 = pivot(__dsqrt_rn(p22));
    F.l32 = __ddiv_rn(__dsub_rn(s3, __dmul_rn(F.l31, F.l21)), F.p2.l);
    const double p33 = __dsub_rn(__dsub_rn(s4, __dmul_rn(F.l31, F.l31)), __dmul_rn(F.l32, F.l32));
    if (p33 <= 0.0) return;
    F.p3 = pivot(__dsqrt_rn(p33));
    F.ok = 1;
}

// beta of L L^T beta = g: forward, then back substitution (maths.cpp:419-470)
template <class Divide>
__device__ __forceinline__ void substitute3(const FitFactor& F, double g0, double g1, double g2, double* beta, Divide div)
{
    const double z0 = div(g0, F.p1);
    const double z1 = div(__dsub_rn(g1, __dmul_rn(F.l21, z0)), F.p2);
    const double z2 = div(__dsub_rn(__dsub_rn(g2, __dmul_rn(F.l31, z0)), __dmul_rn(F.l32, z1)), F.p3);
    beta[2] = div(z2, F.p3);
    beta[1] = div(__dsub_rn(z1, __dmul_rn(F.l32, beta[2])), F.p2);
    beta[0] = div(__dsub_rn(__dsub_rn(z0, __dmul_rn(F.l21, beta[1])), __dmul_rn(F.l31, beta[2])), F.p1);
}

__device__ __noinline__ void substitute3_divisions(const FitFactor* F, double g0, double g1, double g2, double* beta)
{
    substitute3(*F, g0, g1, g2, beta, [](double a, const Pivot& P) { return __ddiv_rn(a, P.l); });
}

// what the walk's loops need of a contract, in registers (their stores to shared memory would make
// every use of the contract there a load again)
struct FitScreen {
    int call, itm_bits, float_strike;
    float strike_f, strike_lo, inv_norm_f;
};
__device__ __forceinline__ FitScreen screen_of(const LsmContract& K)
{
    return FitScreen{K.call, K.itm_bits, K.float_strike, K.strike_f, K.strike_lo, K.inv_norm_f};
}

// S - K in single precision, and 1 where it is exact and a normal number: where the strike is a
// float that holds for S within a factor of two of K (and often beyond: the rounding error, the
// two-sum's, is zero). It is then the double-precision difference.
__device__ __forceinline__ int difference(float sf, const FitScreen& E, float& d)
{
    d = sf - E.strike_f;
    const float bv = d - sf;
    const float err = (sf - (d - bv)) - (E.strike_f + bv);
    return (int)(err == 0.0f) & E.float_strike & (int)(((unsigned)__float_as_int(d) & 0x7fffffffu) - 0x00800000u < 0x7f000000u);
}

// the test that the screen leaves open, out of the walk's line
__device__ __noinline__ bool exercises_exactly(float sf, const FitPolicy* Q, const LsmContract* K)
{
    return itm_value(sf, *K) >= continuation(Q->b[0], Q->b[1], Q->b[2], moneyness((double)sf, *K));
}

// IN_SMEM: the CTA's paths (spots of two dates, every contract's cashflows and in-the-money list)
// live in shared memory, wherever they fit: 26 bytes a path of one contract, 18 more a contract. Else
// in global memory, with the spots read from their rows; then 16 warps an SM have too few loads in
// flight for the latency of DRAM, so each loop's next block is requested into L2 (ahead). 14 dates,
// one contract, the fit alone: 2^24 paths 7.07 ms without, 5.6 with; 2^22 paths 1.44 and 1.14. (Eight
// chunks' loads together instead of four: 1 % faster there, and 15 % slower where a warp has two or
// three chunks, 64 contracts of 2^17 paths.)
template <bool IN_SMEM>
__global__ void __launch_bounds__(FIT_THREADS, 1) lsm_fit_kernel(const LsmFitArgs A)
{
    extern __shared__ __align__(16) unsigned char fit_smem[];
    __shared__ Fx128 s_w[FIT_WARPS][LSM_NACC];
    // What each of the two waiting warps tells the others when it gives up. s_stop, the solver's
    // word for the whole CTA: set before the policy's barrier, read by the walkers behind it. s_lost,
    // the factorer's: set before the factors' barrier, read by the solver behind it. Both stay set.
    __shared__ int s_stop, s_lost;
    using Index = typename std::conditional<IN_SMEM, uint16_t, int32_t>::type;
    const int G = gridDim.x;
    const int C = A.C;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    LsmContract* const s_ct = reinterpret_cast<LsmContract*>(fit_smem);
    FitFactor* const s_fac = reinterpret_cast<FitFactor*>(s_ct + C); // [2][C], by the parity of the date
    FitPolicy* const s_pol = reinterpret_cast<FitPolicy*>(s_fac + 2 * C);
    unsigned* const s_limb = reinterpret_cast<unsigned*>(s_pol + C); // [C][FIT_SUMS][SUM_LIMBS]
    int* const s_nout = reinterpret_cast<int*>(s_limb + C * FIT_SUMS * SUM_LIMBS); // [C][FIT_WARPS]
    unsigned char* const paths = fit_smem + fit_control_bytes(C);
    float* const s_spot = reinterpret_cast<float*>(paths);                              // [2][ppc]
    double* const s_cf = reinterpret_cast<double*>(paths + 2 * sizeof(float) * A.ppc);  // [C][2][ppc]
    uint16_t* const s_idx = reinterpret_cast<uint16_t*>(s_cf + 2 * (size_t)C * A.ppc);  // [C][ppc]

    // this CTA's paths: [p0, p0 + len); a warp's: [la, lb) of them, whole chunks of 32 (the last
    // may end early). The factorer and the solver on scheduler 0 issue FP64 work worth
    // FIT_SOLVER_CHUNKS chunks of a contract a date, so that scheduler's three walkers take that much
    // less than the five, four and four of the others (2^20 paths x 365 dates, fit alone: 0 chunks
    // 5.83 ms, 12 5.70, 24 5.54, 40 5.79).
    const int64_t p0 = (int64_t)blockIdx.x * A.ppc;
    const int len = (int)max((int64_t)0, min(A.ppc, A.n - p0));
    int la, lb;
    {
        const int chunks = (len + 31) / 32;
        const int first = max(0, (chunks - 3 * ((FIT_SOLVER_CHUNKS + C - 1) / C)) / 4); // scheduler 0's
        const int s = warp & 3, k = s ? warp >> 2 : (warp >> 2) - 2, of = s == 0 ? 3 : (s == 1 ? 5 : 4);
        const int from = s ? first + (chunks - first) * (s - 1) / 3 : 0;
        const int to = s ? first + (chunks - first) * s / 3 : first;
        la = 32 * (from + (to - from) * k / of);
        lb = min(len, 32 * (from + (to - from) * (k + 1) / of));
    }
    bool bad = false;

    for (int c = threadIdx.x; c < C; c += FIT_THREADS) s_ct[c] = A.ct[c];
    for (int i = threadIdx.x; i < C * FIT_SUMS * SUM_LIMBS; i += FIT_THREADS) s_limb[i] = 0;
    if (threadIdx.x == 0) s_stop = s_lost = 0;
    __syncthreads();

    auto spots = [&](int t) -> const float* { // date t's spots of this CTA
        if constexpr (IN_SMEM) return s_spot + (size_t)(t & 1) * A.ppc;
        return A.S + (int64_t)t * A.ld + p0;
    };
    auto cashflows = [&](const LsmContract& K, int c) -> double* {
        if constexpr (IN_SMEM) return s_cf + (size_t)(2 * c) * A.ppc;
        return K.cf + p0;
    };
    auto list_m = [&](const LsmContract& K, int c) -> double* {
        if constexpr (IN_SMEM) return s_cf + (size_t)(2 * c + 1) * A.ppc + la;
        return K.c_m + p0 + la;
    };
    auto list_idx = [&](const LsmContract& K, int c) -> Index* {
        if constexpr (IN_SMEM) return s_idx + (size_t)c * A.ppc + la;
        else return K.c_idx + p0 + la;
    };

    // the CTA's sums at `slot` of each contract into the totals of date t at `first`
    auto publish = [&](int t, int slot, int first, int count, unsigned* bar) {
        for (int x = lane; x < C * count; x += 32) {
            const int c = x / count, i = x - c * count;
            if (t > s_ct[c].M - 2) continue;
            fx_red3(s_ct[c].tot + ((size_t)t * LSM_PART + first + i) * 3,
                    take_limbs(s_limb + (c * FIT_SUMS + slot + i) * SUM_LIMBS));
        }
        __threadfence();
        __syncwarp();
        if (lane == 0) atomicAdd(bar, 1u);
    };
    auto await = [&](const unsigned* bar, unsigned want) {
        int ok = 1;
        if (lane == 0) ok = wait_for(bar, want, A.status);
        ok = __shfl_sync(0xffffffffu, ok, 0);
        __syncwarp(); // lane 0's acquire orders the warp's reads of the totals
        return ok != 0;
    };
    // one reading for the warp of a word that another warp may be writing
    auto told = [&](const int& word) { return __shfl_sync(0xffffffffu, *(const volatile int*)&word, 0) != 0; };
    auto total = [&](int c, int t, int i) { return fx_from3(s_ct[c].tot + ((size_t)t * LSM_PART + i) * 3); };

    // A wait that fails takes no warp out of the loops: a named barrier counts its threads, so one
    // that a warp no longer comes to would hold the others for good. Whoever gives up goes on through
    // every barrier of the dates left without working, and all leave together behind the loops.
    bool ok = true;
    if (warp == FIT_FACTORER) {
        // the moneyness sums of a date are complete while the CTAs still form its cashflow sums:
        // the normal equations' matrix is factored beside them
        unsigned phase = 0;
        for (int t = A.Tmax - 2; t >= 1; --t) {
            phase += (unsigned)G;
            bar_sync<FIT_HANDOVER>(BAR_X + (t & 1));
            ok = ok && !told(s_stop);
            if (ok) {
                publish(t, (t & 1) * FIT_X, 0, FIT_X, A.bar_x);
                ok = await(A.bar_x, phase);
                if (!ok) s_lost = 1;
            }
            for (int c = lane; ok && c < C; c += 32) {
                if (t > s_ct[c].M - 2) continue;
                const Fx128 a1 = total(c, t, 0), a2 = total(c, t, 1), a3 = total(c, t, 2), a4 = total(c, t, 3);
                const double n = (double)total(c, t, 4).lo;
                FitFactor& F = s_fac[(t & 1) * C + c];
                F.ok = 0;
                if (n >= (double)s_ct[c].min_itm)
                    factor3(n, fx_to_double(a1), fx_to_double(a2), fx_to_double(a3), fx_to_double(a4), F);
            }
            bar_arrive<64>(BAR_FACTOR + (t & 1));
        }
    } else if (warp == FIT_SOLVER) {
        unsigned phase = 0;
        for (int t = A.Tmax - 2; t >= 1; --t) {
            phase += (unsigned)G;
            bar_sync<FIT_HANDOVER>(BAR_Y);
            if (ok) {
                publish(t, 2 * FIT_X, FIT_X, FIT_Y, A.bar_y);
                ok = await(A.bar_y, phase);
            }
            bar_sync<64>(BAR_FACTOR + (t & 1));
            // (the factorer may be a date ahead: its word then stops the CTA a date early)
            ok = ok && !told(s_lost);
            if (!ok) s_stop = 1;
            for (int c = lane; ok && c < C; c += 32) {
                const LsmContract& K = s_ct[c];
                if (t > K.M - 2) continue;
                const Fx128 g0 = total(c, t, FIT_X), g1 = total(c, t, FIT_X + 1), g2 = total(c, t, FIT_X + 2);
                double b[3] = {0.0, 0.0, 0.0};
                const FitFactor& F = s_fac[(t & 1) * C + c];
                const int f = F.ok;
                const double df = K.df[t - 1];
                if (f) {
                    const double h0 = fx_to_double(g0), h1 = fx_to_double(g1), h2 = fx_to_double(g2);
                    bool sure = true;
                    substitute3(F, h0, h1, h2, b, [&](double a, const Pivot& P) { return divide_by(a, P, sure); });
                    if (!sure) substitute3_divisions(&F, h0, h1, h2, b);
                }
                FitPolicy& Q = s_pol[c];
                Q.s = lsm_screen(b, f, K.strike, K.norm, K.m0);
                Q.df = df;
                for (int i = 0; i < 3; i++) Q.b[i] = b[i];
                if (blockIdx.x == 0) {
                    K.fit[t] = f;
                    for (int i = 0; i < 3; i++) K.beta[3 * t + i] = b[i];
                }
            }
            bar_arrive<FIT_HANDOVER>(BAR_POLICY);
        }
    } else {
        // ---- the walkers -----------------------------------------------------------
        // Paths in global memory: FIT_AHEAD elements from `at` on (below end) into L2, a line a lane,
        // one block ahead of a loop that starts its blocks here
        auto ahead = [&](const auto* base, int at, int end) {
            constexpr int LINE = 128 / (int)sizeof(*base);
            static_assert(FIT_AHEAD <= 32 * LINE, "a warp requests a block at once");
            const int l = at + LINE * lane;
            if (!IN_SMEM && LINE * lane < FIT_AHEAD && l < end) prefetch_l2(base + l);
        };
        auto block_starts = [&](int l) { return !IN_SMEM && l % FIT_AHEAD == 0; };
        auto request_spots = [&](int t) { // each thread copies the spots it will screen itself
            if constexpr (IN_SMEM) {
                float* const dst = s_spot + (size_t)(t & 1) * A.ppc;
                const float* const row = A.S + (int64_t)t * A.ld + p0;
                for (int l = la + lane; l < lb; l += 32)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                                     (unsigned)__cvta_generic_to_shared(dst + l)),
                                 "l"(row + l)
                                 : "memory");
            }
            ahead(spots(t), la, lb);
            if (IN_SMEM && t > 1) // the date after next: into L2
                for (int l = la + 32 * lane; l < lb; l += 1024) prefetch_l2(A.S + (int64_t)(t - 1) * A.ld + p0 + l);
        };
        // the moneyness sums of date t for every contract whose exercise grid reaches it: list
        // the in-the-money paths, then full warps of them do the FP64 work
        auto moneyness_sums = [&](int t) {
            if constexpr (IN_SMEM) {
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncwarp();
            }
            const float* const S = spots(t);
            for (int c = 0; c < C; ++c) {
                const LsmContract& K = s_ct[c];
                if (t > K.M - 2) continue;
                Index* const idx = list_idx(K, c);
                double* const lm = list_m(K, c);
                const FitScreen E = screen_of(K);
                int nout = 0;
#pragma unroll 4
                for (int l0 = la; l0 < lb; l0 += 32) {
                    const int l = l0 + lane;
                    if (block_starts(l0 - la)) ahead(S, l0 + FIT_AHEAD, lb);
                    const bool itm = l < lb && in_the_money(S[l < lb ? l : la], E);
                    const unsigned mk = __ballot_sync(0xffffffffu, itm);
                    if (itm) idx[nout + __popc(mk & below)] = (Index)l;
                    nout += __popc(mk);
                }
                __syncwarp();
                Fx128 q[4] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};
                auto sums = [&](auto money) {
                    for (int j = lane; j < nout; j += 32) {
                        const double m = money(widen(S[idx[j]])), m2 = __dmul_rn(m, m);
                        const double m3 = __dmul_rn(m2, m), m4 = __dmul_rn(m2, m2);
                        lm[j] = m;
                        fx_add_checked(q[0], m, bad);
                        fx_add_checked(q[1], m2, bad);
                        fx_add_checked(q[2], m3, bad);
                        fx_add_checked(q[3], m4, bad);
                    }
                };
                if (K.short_norm)
                    sums([y = K.inv_norm, lo = K.inv_norm_lo](double s) { return moneyness_short(s, y, lo); });
                else
                    sums([&K](double s) { return moneyness(s, K); });
                __syncwarp();
                unsigned* const limb = s_limb + (c * FIT_SUMS + (t & 1) * FIT_X) * SUM_LIMBS;
                warp_sum4(q, lane, limb, 4);
                if (lane == 0) {
                    s_nout[c * FIT_WARPS + warp] = nout;
                    atomicAdd(limb + 4 * SUM_LIMBS, (unsigned)nout);
                }
            }
        };
        // every path through date t + 1's decision and to date t
        auto roll = [&](int t) {
            const float* const Sn = spots(t + 1);
            for (int c = 0; c < C; ++c) {
                const LsmContract& K = s_ct[c];
                if (t > K.M - 2) continue;
                const bool last = t == K.M - 2; // the date before maturity: no decision to take
                const FitPolicy& Q = s_pol[c];
                const double d = last ? K.df[t] : Q.df;
                const bool decide = !last && Q.s.fit;
                double* const cf = cashflows(K, c);
                const LsmScreen P = Q.s;
                const FitScreen E = screen_of(K);
                const int sign = E.call ? 0 : (int)0x80000000; // K - S rounds to -(S - K)
                int32_t* const tau = K.tau + p0;
                // without a branch from the screen to the product, so that the chunks' chains of
                // single-precision operations overlap and an FP64 instruction serves a whole warp
                constexpr int U = 4;
                for (int l0 = la + lane; l0 - lane < lb; l0 += 32 * U) {
                    if (block_starts(l0 - lane - la)) {
                        ahead(cf, l0 - lane + FIT_AHEAD, lb);
                        if (decide) ahead(Sn, l0 - lane + FIT_AHEAD, lb);
                    }
                    double v[U];
                    float sf[U];
                    int ex[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int l = min(l0 + 32 * u, lb - 1);
                        v[u] = cf[l];
                        sf[u] = Sn[decide ? l : 0];
                    }
                    if (decide) {
                        int open = 0, rest = 0;
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            ex[u] = screen_exercise(sf[u], P, E) & -(int)((l0 + 32 * u < lb) & in_the_money(sf[u], E));
                            open |= ex[u];
                        }
                        if (__any_sync(0xffffffffu, open)) { // no path of the chunks exercises: nothing to find
                            if (__any_sync(0xffffffffu, open < 0)) {
#pragma unroll
                                for (int u = 0; u < U; ++u)
                                    if (ex[u] < 0) ex[u] = exercises_exactly(sf[u], &Q, &K);
                                __syncwarp();
                            }
#pragma unroll
                            for (int u = 0; u < U; ++u) {
                                float x;
                                const int exact = difference(sf[u], E, x);
                                const unsigned xb = (unsigned)__float_as_int(x);
                                const int hi = (int)(((xb & 0x7fffffffu) >> 3) + 0x38000000u | (xb & 0x80000000u)) ^ sign;
                                const bool now = ex[u] & exact;
                                v[u] = __hiloint2double(now ? hi : __double2hiint(v[u]), now ? (int)(xb << 29) : __double2loint(v[u]));
                                rest |= ex[u] & (exact ^ 1);
                            }
                            if (__any_sync(0xffffffffu, rest)) {
#pragma unroll
                                for (int u = 0; u < U; ++u) {
                                    float x;
                                    if (ex[u] && !difference(sf[u], E, x)) v[u] = itm_value(sf[u], K);
                                }
                                __syncwarp();
                            }
#pragma unroll
                            for (int u = 0; u < U; ++u)
                                if (ex[u]) tau[l0 + 32 * u] = t + 1;
                        }
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        v[u] = __dmul_rn(v[u], d);
                        if (l0 + 32 * u < lb) cf[l0 + 32 * u] = v[u];
                    }
                }
            }
            __syncwarp();
        };
        // the cashflow sums of date t over the lists
        auto cashflow_sums = [&](int t) {
            for (int c = 0; c < C; ++c) {
                const LsmContract& K = s_ct[c];
                if (t > K.M - 2) continue;
                const double* const cf = cashflows(K, c);
                const Index* const idx = list_idx(K, c);
                const double* const lm = list_m(K, c);
                const int nout = s_nout[c * FIT_WARPS + warp];
                Fx128 q[4] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};
                for (int j = lane; j < nout; j += 32) {
                    if (block_starts(j - lane)) {
                        const int next = j - lane + FIT_AHEAD;
                        ahead(lm, next, nout);
                        ahead(idx, next, nout);
                        if (next < nout) // the cashflows of the next block's paths
                            for (int l = idx[next] + 16 * lane; l <= idx[min(next + FIT_AHEAD, nout) - 1]; l += 512)
                                prefetch_l2(cf + l);
                    }
                    const double y = cf[idx[j]], m = lm[j], m2 = __dmul_rn(m, m);
                    const double my = __dmul_rn(m, y), m2y = __dmul_rn(m2, y);
                    fx_add_checked(q[0], y, bad);
                    fx_add_checked(q[1], my, bad);
                    fx_add_checked(q[2], m2y, bad);
                }
                __syncwarp();
                warp_sum4(q, lane, s_limb + (c * FIT_SUMS + 2 * FIT_X) * SUM_LIMBS, FIT_Y);
            }
            if (bad) atomicExch(A.status, 3);
        };

        // maturity: each contract's cashflow is its payoff
        for (int c = 0; c < C; ++c) {
            const LsmContract& K = s_ct[c];
            const float* row = A.S + (int64_t)(K.M - 1) * A.ld + p0;
            double* const cf = cashflows(K, c);
            for (int l = la + lane; l < lb; l += 32) {
                cf[l] = payoff(row[l], K);
                K.tau[p0 + l] = 0;
            }
        }
        const int t0 = A.Tmax - 2;
        if (t0 >= 1) {
            request_spots(t0);
            moneyness_sums(t0);
            bar_arrive<FIT_HANDOVER>(BAR_X + (t0 & 1));
        }
        for (int t = t0; t >= 1; --t) {
            if (t < t0) {
                ahead(cashflows(s_ct[0], 0), la, lb);
                ahead(spots(t + 1), la, lb);
                bar_sync<FIT_HANDOVER>(BAR_POLICY);
                ok = ok && !s_stop;
            }
            if (ok) {
                roll(t);
                // date t + 1's spots have been used: date t - 1's take their place
                if (t > 1) request_spots(t - 1);
                cashflow_sums(t);
            }
            bar_arrive<FIT_HANDOVER>(BAR_Y);
            if (t > 1) { // the next date's moneyness sums, while this date's policy is found
                if (ok) moneyness_sums(t - 1);
                bar_arrive<FIT_HANDOVER>(BAR_X + ((t - 1) & 1));
            }
        }
        if (t0 >= 1) bar_sync<FIT_HANDOVER>(BAR_POLICY);
    }
    __syncthreads(); // every warp is out of the loops
    if (s_stop) return;

    // the value of each path's earliest exercise (date 1's decision here), else of its maturity
    for (int c = 0; c < C; ++c) {
        const LsmContract& K = s_ct[c];
        Fx128 v = {0, 0}, v2 = {0, 0}, eu = {0, 0};
        if (warp != FIT_FACTORER && warp != FIT_SOLVER) {
            const bool decide = K.M > 2 && s_pol[c].s.fit;
            const float* const S1 = spots(1);
            const float* const last = A.S + (int64_t)(K.M - 1) * A.ld + p0;
            const double dT = K.disc[K.M - 1];
            constexpr int U = 4; // paths a lane whose loads are in flight together
            for (int l0 = la + lane; l0 < lb; l0 += 32 * U) {
                int t[U];
                float s1[U], sT[U], sx[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int l = min(l0 + 32 * u, lb - 1);
                    t[u] = K.tau[p0 + l];
                    s1[u] = decide ? S1[l] : 0.f;
                    sT[u] = last[l];
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (decide && in_the_money(s1[u], K)) {
                        const FitPolicy& Q = s_pol[c];
                        int ex = screen_exercise(s1[u], Q.s, K);
                        if (ex < 0) ex = exercises_exactly(s1[u], &Q, &K);
                        if (ex) t[u] = 1;
                    }
                    sx[u] = t[u] ? A.S[(int64_t)t[u] * A.ld + p0 + min(l0 + 32 * u, lb - 1)] : 0.f;
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (l0 + 32 * u < lb) {
                        const double e = __dmul_rn(payoff(sT[u], K), dT);
                        const double x = t[u] ? __dmul_rn(itm_value(sx[u], K), K.disc[t[u]]) : e;
                        fx_add_checked(v, x, bad);
                        fx_add_checked(v2, __dmul_rn(x, x), bad);
                        fx_add_checked(eu, e, bad);
                    }
            }
        }
        Fx128* const acc = K.acc + (size_t)blockIdx.x * LSM_NACC;
        block_sum(v, s_w, 0, acc);
        block_sum(v2, s_w, 1, acc + 1);
        block_sum(eu, s_w, 2, acc + 2);
    }
    if (bad) atomicExch(A.status, 3);
}

constexpr int APPLY_AHEAD = 8; // dates whose spots one thread loads together

// The frozen policy on a path set. A path's walk ends at its first exercise, but nothing on the way
// branches: the dates that are loaded together are screened together, and the first that may
// exercise is picked. The FP64 work comes once a path, after the walk, where the warp is whole again
// (five products and differences; with the conversions and tests on the way, and three block sums,
// 300,000 paths of 13 dates took 34 us, now 18).
__global__ void __launch_bounds__(LSM_THREADS, 2) lsm_apply_kernel(const LsmArgs A)
{
    __shared__ unsigned s_limb[LSM_NACC * SUM_LIMBS];
    if (threadIdx.x < LSM_NACC * SUM_LIMBS) s_limb[threadIdx.x] = 0;
    __syncthreads();
    const int64_t T = (int64_t)gridDim.x * LSM_THREADS;
    const int64_t g0 = (int64_t)blockIdx.x * LSM_THREADS + threadIdx.x;
    const int lane = threadIdx.x & 31;
    bool bad = false;
    Fx128 q[4] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}}; // values, their squares, maturity payoffs
    const float* last = A.S + (int64_t)(A.M - 1) * A.ld;
    const double dT = A.disc[A.M - 1];
    const int tend = A.M - 1; // exercise dates 1 .. M-2; the maturity pays the European payoff
    const int sign = A.call ? 0 : (int)0x80000000; // as in itm_value
    auto value = [&](float sf, double d) {
        const double v = __dsub_rn(widen(sf), A.strike);
        return __dmul_rn(__hiloint2double(__double2hiint(v) ^ sign, __double2loint(v)), d);
    };
    for (int64_t p = g0; p < A.n; p += T) {
        const float sT = __ldg(last + p);
        int tau = 0;
        float sx = 0.f;
        // row t + u of the date-major paths: coalesced in p
        for (int t = 1; t < tend && !tau; t += APPLY_AHEAD) {
            float sv[APPLY_AHEAD];
            int ex[APPLY_AHEAD], open = 0;
#pragma unroll
            for (int u = 0; u < APPLY_AHEAD; ++u)
                sv[u] = __ldg(A.S + (int64_t)min(t + u, tend) * A.ld + p);
#pragma unroll
            for (int u = 0; u < APPLY_AHEAD; ++u) {
                const float4* w = reinterpret_cast<const float4*>(A.screen + min(t + u, tend));
                const float4 a = __ldg(w), b = __ldg(w + 1);
                const LsmScreen P = {a.x, a.y, a.z, a.w, b.x, b.y, __float_as_int(b.z), 0};
                ex[u] = screen_exercise(sv[u], P, A) & -(int)((t + u < tend) & (P.fit != 0) & in_the_money(sv[u], A));
                open |= ex[u];
            }
            if (open < 0) { // rare: the dates that the screen leaves open
#pragma unroll
                for (int u = 0; u < APPLY_AHEAD; ++u)
                    if (ex[u] < 0) {
                        const double* be = A.beta + 3 * (t + u);
                        ex[u] = itm_value(sv[u], A) >= continuation(be[0], be[1], be[2], moneyness((double)sv[u], A));
                    }
            }
#pragma unroll
            for (int u = APPLY_AHEAD - 1; u >= 0; --u) {
                tau = ex[u] ? t + u : tau;
                sx = ex[u] ? sv[u] : sx;
            }
        }
        // (a NaN spot is paid, so that the sum's check sees it)
        const double e = in_the_money(sT, A) || sT != sT ? value(sT, dT) : 0.0;
        const double x = tau ? value(sx, A.disc[tau]) : e;
        fx_add_checked(q[0], x, bad);
        fx_add_checked(q[1], __dmul_rn(x, x), bad);
        fx_add_checked(q[2], e, bad);
    }
    __syncwarp();
    if (bad) atomicExch(A.status, 3);
    warp_sum4(q, lane, s_limb, LSM_NACC);
    __syncthreads();
    if (threadIdx.x < LSM_NACC)
        A.acc[(size_t)blockIdx.x * LSM_NACC + threadIdx.x] = take_limbs(s_limb + threadIdx.x * SUM_LIMBS);
}

} // namespace

// dynamic shared memory of a fit whose CTAs walk ppc paths each (in_smem: the paths' too)
static size_t fit_smem(int C, int64_t ppc, bool in_smem)
{
    return fit_control_bytes(C) + (in_smem ? fit_path_bytes(C, ppc) : 0);
}

cudaError_t lsm_fit_shape(int64_t n, int C, int sms, LsmFitShape* out)
{
    int dev = 0, most = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncAttributes at;
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&at, lsm_fit_kernel<true>);
    if (e != cudaSuccess) return e;
    // one CTA an SM, all resident
    const int64_t want = (n + FIT_MIN_PATHS - 1) / FIT_MIN_PATHS;
    out->grid = (int)(want < 1 ? 1 : (want < sms ? want : sms));
    out->ppc = ((n + out->grid - 1) / out->grid + 31) / 32 * 32;
    out->in_smem = fit_smem(C, out->ppc, true) + at.sharedSizeBytes <= (size_t)most;
    const size_t smem = fit_smem(C, out->ppc, out->in_smem);
    const void* fn = out->in_smem ? reinterpret_cast<const void*>(lsm_fit_kernel<true>)
                                  : reinterpret_cast<const void*>(lsm_fit_kernel<false>);
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(most - (int)at.sharedSizeBytes));
    int per = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, FIT_THREADS, smem);
    if (e == cudaSuccess && per < 1) e = cudaErrorLaunchOutOfResources;
    return e;
}

cudaError_t launch_lsm_fit(const LsmFitArgs& A, const LsmFitShape& shape, cudaStream_t st)
{
    LsmFitArgs a = A;
    void* args[] = {&a};
    const void* fn = shape.in_smem ? reinterpret_cast<const void*>(lsm_fit_kernel<true>)
                                   : reinterpret_cast<const void*>(lsm_fit_kernel<false>);
    return cudaLaunchCooperativeKernel(fn, dim3(shape.grid), dim3(FIT_THREADS), args,
                                       fit_smem(A.C, A.ppc, shape.in_smem), st);
}

cudaError_t launch_lsm_apply(const LsmArgs& A, int grid, cudaStream_t st)
{
    lsm_apply_kernel<<<grid, LSM_THREADS, 0, st>>>(A);
    return cudaGetLastError();
}
