// surrogate.cu — BF16 tensor-core (tcgen05) kernels of the learned Heston
// surrogate: a validation GEMM, the fused MLP inference kernel, the training
// tile (forward, head, backward for inputs and weights) and Adam.
#include "engine.cuh"
#include "phi.cuh"
#include "surrogate.cuh"
#include "tc.cuh"

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

namespace thoth {

// ---------------------------------------------------------------------------
// Validation GEMM: one CTA of 128 threads computes D (128 x N, FP32, row-major)
// = A (128 x K) * B (N x K)^T with A, B bf16 row-major in global memory.
// N in {16..256} multiple of 16, K multiple of 16 up to 256.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128) tc_gemm_test_kernel(const __nv_bfloat16* __restrict__ A,
                                                           const __nv_bfloat16* __restrict__ B, int N, int K,
                                                           float* __restrict__ D, int* status)
{
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ uint64_t mbar;
    __shared__ uint32_t taddr_s;
    unsigned char* sA = sm;
    unsigned char* sB = sm + 128 * K * 2;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    uint32_t ncols = 32;
    while (ncols < (uint32_t)N) ncols <<= 1;
    if (warp == 0) tc::tmem_alloc(&taddr_s, ncols);
    if (t == 0) tc::mbar_init(&mbar, 1);
    // stage A and B into the K-major core-matrix layout (16-byte chunks)
    const int kc = K / 8;
    for (int c = t; c < 128 * kc; c += 128) {
        const int r = c / kc, kb = c % kc;
        *reinterpret_cast<uint4*>(sA + tc::cm_offset(r, kb * 8, 128)) =
            *reinterpret_cast<const uint4*>(A + (size_t)r * K + kb * 8);
    }
    for (int c = t; c < N * kc; c += 128) {
        const int r = c / kc, kb = c % kc;
        *reinterpret_cast<uint4*>(sB + tc::cm_offset(r, kb * 8, N)) =
            *reinterpret_cast<const uint4*>(B + (size_t)r * K + kb * 8);
    }
    tc::fence_smem_async();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tm = taddr_s;
    if (t == 0) {
        const uint32_t idesc = tc::make_idesc_bf16(128, N);
        const uint32_t a0 = tc::smem_u32(sA), b0 = tc::smem_u32(sB);
        for (int kk = 0; kk < K / 16; ++kk) {
            const uint64_t ad = tc::make_desc(a0 + (uint32_t)(2 * kk) * (128 * 16), 128 * 16, 128);
            const uint64_t bd = tc::make_desc(b0 + (uint32_t)(2 * kk) * (uint32_t)(N * 16), (uint32_t)N * 16, 128);
            tc::mma_bf16(tm, ad, bd, idesc, kk > 0 ? 1u : 0u);
        }
        tc::mma_commit(&mbar);
    }
    const bool ok = tc::mbar_wait(&mbar, 0);
    if (!ok && lane == 0) atomicExch(status, 1);
    tc::fence_after_sync();
    if (ok) {
        const int row = warp * 32 + lane;
        for (int c0 = 0; c0 < N; c0 += 16) {
            float v[16];
            tc::tmem_ld16(tm + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, v);
#pragma unroll
            for (int j = 0; j < 16; ++j) D[(size_t)row * N + c0 + j] = v[j];
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tm, ncols);
}

cudaError_t launch_tc_gemm_test(const void* A, const void* B, int N, int K, float* D, int* status, cudaStream_t st)
{
    // padded far beyond the operands so that every descriptor-generated address stays
    // inside this CTA's shared memory even if an offset field were misread
    const size_t need = (size_t)(128 + N) * K * 2;
    const size_t smem = need > 200 * 1024 ? need : 200 * 1024;
    cudaError_t e = cudaFuncSetAttribute(tc_gemm_test_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    tc_gemm_test_kernel<<<1, 128, smem, st>>>(reinterpret_cast<const __nv_bfloat16*>(A),
                                              reinterpret_cast<const __nv_bfloat16*>(B), N, K, D, status);
    return cudaGetLastError();
}

namespace mlp {

// ---------------------------------------------------------------------------
// One training tile: 128 rows of the batch through the whole network and back, one CTA.
//
// Weights, activations and gradients of the tile never leave the SM: seven 32 KB operand
// buffers in shared memory (W2, W3, W4, the activations a1..a3, and one that holds W1 and the
// inputs during layer 1 and dz4 afterwards), and the four pre-activations' derivatives in the
// 512 TMEM columns, where each layer's accumulator was. A buffer is reused as soon as the
// products that read it are done: dz3 goes over W4, dz2 over W3, dz1 over dz4, the inputs (kept
// in registers) over a3. dW = dz^T a and da = dz W read the same tiles as transposed operands
// (tc::make_desc_mn), so nothing is transposed or stored twice. The da chain is the critical
// path; each dW runs behind it into columns that are free by then, and is read out while the
// next product runs.
//
// 512 threads do the epilogues: warp w owns rows 32 (w % 4) .. + 31 (its TMEM lanes) and columns
// 32 (w / 4) .. + 31. The special-function unit bounds the forward half (two operations an
// activation, 128 x 128 of them a layer at 16 a clock: 1.1 us); SiLU' is taken there as well,
// from the same reciprocal, and kept, so the backward half has none. Four more warps add the bias
// gradients, a column a thread in row order, beside the products that follow (in the epilogue
// warps they held up every layer: 41 000 clocks a tile, about 33 000 beside them). Per-tile partial
// gradients go to memory, dW as [in][out] so that a warp's lanes (out) store 128 consecutive
// bytes; adam_kernel adds them in tile order. The two kernels are launched as programmatic
// dependents: gathering the batch's rows and the launch itself overlap the other's end.
//
// As eight layer kernels with row-per-thread global accesses a step of 8192 rows took 0.50 ms
// (64 CTAs, 12 to 29 warps stalled on global memory per issue); as this kernel and Adam, 35 us with
// its host work.
// ---------------------------------------------------------------------------
constexpr int TILE_MAIN = 512; // the epilogue threads
constexpr int TILE_THREADS = TILE_MAIN + H;
constexpr uint32_t TILE_BUF = H * H * 2; // one 128 x 128 bf16 operand
constexpr size_t TILE_SMEM = 7 * (size_t)TILE_BUF;

// issue D = A B^T over K (one thread); a tile of 128 rows is read as it lies (K along its
// columns) or transposed (mn: K along its rows). The descriptors of a K slice differ from the
// first's in the start address alone (16-byte units): formed per slice, in a loop, the issuing
// thread held the products up (inference of 2^20 cells 198 us, 185 like this)
template <int K>
__device__ __forceinline__ void issue(uint32_t d, const unsigned char* A, bool a_mn, const unsigned char* B, bool b_mn,
                                      int N)
{
    const uint32_t idesc = tc::make_idesc_bf16(128, N, a_mn, b_mn);
    const uint32_t a0 = tc::smem_u32(A), b0 = tc::smem_u32(B);
    const uint64_t ad = a_mn ? tc::make_desc_mn(a0, 128) : tc::make_desc(a0, 2048, 128);
    const uint64_t bd = b_mn ? tc::make_desc_mn(b0, 128) : tc::make_desc(b0, 2048, 128);
#pragma unroll
    for (uint32_t kk = 0; kk < K / 16; ++kk)
        tc::mma_bf16(d, ad + kk * (a_mn ? 16u : 256u), bd + kk * (b_mn ? 16u : 256u), idesc, kk > 0 ? 1u : 0u);
}

// SiLU and its derivative from one reciprocal: z sigmoid(z) equals __fdividef(z, 1 + e^-z) bit for
// bit (checked for every float z)
__device__ __forceinline__ void silu_both(float z, float& a, float& d)
{
    const float s = __fdividef(1.0f, 1.0f + __expf(-z));
    a = z * s;
    d = s * (1.0f + z * (1.0f - s));
}

// named barriers of the tile kernel: the epilogue threads' own; one for each dz tile, ready for its
// bias gradient (each used once); dz4's bias gradient done, its buffer free
enum : int { BAR_MAIN = 1, BAR_DZ = 2, BAR_D4_FREE = 6 };
__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n)
{
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// 16 values of a row into columns c0 .. c0 + 15 of an operand tile, as bf16
__device__ __forceinline__ void put16(unsigned char* tile, int row, int c0, const float (&v)[16])
{
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        __align__(16) __nv_bfloat16 o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = __float2bfloat16(v[8 * h + j]);
        *reinterpret_cast<uint4*>(tile + tc::cm_offset(row, c0 + 8 * h, ROWS)) = *reinterpret_cast<const uint4*>(o);
    }
}

__global__ void __launch_bounds__(TILE_THREADS, 1) train_tile_kernel(const TileArgs A)
{
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ uint64_t mb_w, mb_a, mb_b; // weights arrived; the da chain; the dW products
    __shared__ uint32_t tm_s;
    __shared__ float red[4][H];
    __shared__ float red2[4][2];
    float* const s_y = red[0];            // a row's partial head sum, then dL/dy
    unsigned char *W2 = sm, *W3 = sm + TILE_BUF, *W4 = sm + 2 * TILE_BUF, *A1 = sm + 3 * TILE_BUF,
                  *A2 = sm + 4 * TILE_BUF, *A3 = sm + 5 * TILE_BUF, *D4 = sm + 6 * TILE_BUF;
    unsigned char *W1 = D4, *X = D4 + H * KIN * 2; // until dz4 is formed
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, cg = warp >> 2;
    const int row = (warp & 3) * 32 + lane, c0 = cg * 32;
    float* gp = A.part + (size_t)blockIdx.x * N_PARAMS;
    if (t == 0) {
        tc::mbar_init(&mb_w, 1);
        tc::mbar_init(&mb_a, 1);
        tc::mbar_init(&mb_b, 1);
        tc::fence_mbar_init();
        tc::fence_smem_async();
    }
    if (warp == 0) tc::tmem_alloc(&tm_s, 512);
    // this thread's row of the set (perm and the set do not change while a step may overlap)
    const int64_t r0 = A.first + (int64_t)blockIdx.x * ROWS;
    uint4 x0 = make_uint4(0, 0, 0, 0), x1 = x0;
    float yt = 0.f, wt = 0.f;
    if (cg == 0 || cg == 3) {
        const int64_t src = A.perm ? (int64_t)__ldg(A.perm + r0 + row) : r0 + row;
        if (cg == 0) {
            const uint4* xs = reinterpret_cast<const uint4*>(A.x + src * KIN);
            x0 = __ldg(xs);
            x1 = __ldg(xs + 1);
            *reinterpret_cast<uint4*>(X + tc::cm_offset(row, 0, ROWS)) = x0;
            *reinterpret_cast<uint4*>(X + tc::cm_offset(row, 8, ROWS)) = x1;
        } else {
            yt = __ldg(A.y + src);
            wt = __ldg(A.w + src);
        }
    }
    // The weights are there, and the partials free. Nothing the previous kernel writes is read
    // before this, and the parameters never through the read-only path, which may run ahead of it.
    tc::wait_previous();
    if (t == 0) {
        tc::mbar_expect(&mb_w, N_BF * 2);
        tc::bulk_load(W1, A.wbf + OFF_BF_W1, H * KIN * 2, &mb_w);
        tc::bulk_load(W2, A.wbf + OFF_BF_W2, 3 * TILE_BUF, &mb_w); // W2, W3, W4 follow on
    }
    tc::fence_smem_async();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tm = tm_s;
    bool ok = true;

    if (t >= TILE_MAIN) {
        // db = the sum of dz over the tile's rows, in row order, a column a thread
        const int o = t - TILE_MAIN;
#pragma unroll 1
        for (int l = 4; l >= 1; --l) {
            bar_sync(BAR_DZ + 4 - l, TILE_THREADS);
            const unsigned char* dz = l == 3 ? W4 : l == 2 ? W3 : D4;
            float s = 0.f;
#pragma unroll 16
            for (int r = 0; r < ROWS; ++r)
                s += __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(dz + tc::cm_offset(r, o, ROWS)));
            gp[b_off(l) + o] = s;
            if (l == 4) bar_arrive(BAR_D4_FREE, TILE_THREADS);
        }
    } else {
        uint32_t ph_a = 0, ph_b = 0;
        auto operands_ready = [&] { // operand and TMEM accesses of every thread -> the next products
            tc::fence_smem_async();
            tc::fence_before_sync();
            bar_sync(BAR_MAIN, TILE_MAIN);
            tc::fence_after_sync();
        };
        auto wait_a = [&] {
            ok = tc::mbar_wait(&mb_a, ph_a) && ok;
            ph_a ^= 1u;
            tc::fence_after_sync();
        };
        auto wait_b = [&] {
            ok = tc::mbar_wait(&mb_b, ph_b) && ok;
            ph_b ^= 1u;
            tc::fence_after_sync();
        };
        const uint32_t at = tm + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0; // this thread's lane, column
        ok = tc::mbar_wait(&mb_w, 0) && ok;

        // ---- forward: layer l's accumulator in columns 128 (l - 1) ..; SiLU into the next operand,
        // SiLU' over the accumulator ----------------------------------------------------------
        unsigned char* const in[4] = {X, A1, A2, A3};
        unsigned char* const wl[4] = {W1, W2, W3, W4};
        const float4* w5 = reinterpret_cast<const float4*>(A.params + OFF_W5 + c0); // 16-byte aligned: OFF_W5 is a multiple of 4
        static_assert(OFF_W5 % 4 == 0, "head weights are read four at a time");
        float s4[32]; // layer 4: SiLU of this thread's columns
#pragma unroll
        for (int l = 1; l <= 4; ++l) {
            if (t == 0) {
                const uint32_t d = tm + (uint32_t)(128 * (l - 1));
                if (l == 1) issue<KIN>(d, X, false, W1, false, H);
                else issue<H>(d, in[l - 1], false, wl[l - 1], false, H);
                tc::mma_commit(&mb_a);
            }
            const float* b = A.params + b_off(l) + c0;
            float bv[16]; // requested before the wait, which covers their latency
#pragma unroll
            for (int j = 0; j < 16; ++j) bv[j] = b[j];
            wait_a();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float v[16], d[16];
                const uint32_t col = at + (uint32_t)(128 * (l - 1) + 16 * h);
                tc::tmem_ld16(col, v);
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const float z = v[j] + bv[j];
                    silu_both(z, v[j], d[j]);
                    if (l == 4) s4[16 * h + j] = v[j];
                }
                if (h == 0)
#pragma unroll
                    for (int j = 0; j < 16; ++j) bv[j] = b[16 + j];
                if (l < 4) put16(in[l < 4 ? l : 0], row, c0 + 16 * h, v);
                tc::tmem_st16(col, d);
            }
            tc::tmem_wait_st();
            if (l < 4) operands_ready();
        }
        // ---- head: y = b5 + sum_j w5[j] a4[j], one column group after the other so that the sum
        // runs in column order; weighted MSE, dL/dy ---------------------------------------------
#pragma unroll 1
        for (int g = 0; g < 4; ++g) {
            if (cg == g) {
                float yh = g == 0 ? A.params[OFF_B5] : s_y[row];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float4 w = w5[j];
                    yh = fmaf(w.x, s4[4 * j], yh);
                    yh = fmaf(w.y, s4[4 * j + 1], yh);
                    yh = fmaf(w.z, s4[4 * j + 2], yh);
                    yh = fmaf(w.w, s4[4 * j + 3], yh);
                }
                if (g < 3) {
                    s_y[row] = yh;
                } else {
                    const float e = yh - yt;
                    const float dy = 2.f * e * wt / (float)A.rows;
                    s_y[row] = dy;
                    float sdy = dy, sl = e * e * wt;
                    for (int o = 16; o > 0; o >>= 1) {
                        sdy += __shfl_xor_sync(0xffffffffu, sdy, o);
                        sl += __shfl_xor_sync(0xffffffffu, sl, o);
                    }
                    if (lane == 0) {
                        red2[warp & 3][0] = sdy;
                        red2[warp & 3][1] = sl;
                    }
                }
            }
            bar_sync(BAR_MAIN, TILE_MAIN);
        }
        const float dy = s_y[row];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float d[16];
            tc::tmem_ld16(at + (uint32_t)(384 + 16 * h), d);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float4 w = w5[4 * h + j];
                d[4 * j] = dy * w.x * d[4 * j];
                d[4 * j + 1] = dy * w.y * d[4 * j + 1];
                d[4 * j + 2] = dy * w.z * d[4 * j + 2];
                d[4 * j + 3] = dy * w.w * d[4 * j + 3];
            }
            put16(D4, row, c0 + 16 * h, d);
        }
        bar_arrive(BAR_DZ, TILE_THREADS);
        operands_ready();
        if (t == 0) { // da3 = dz4 W4
            issue<H>(tm + 384, D4, false, W4, true, H);
            tc::mma_commit(&mb_a);
        }
        // the head's weight gradients: every column's sum over the warp's 32 rows by the butterfly
        // tree of a shuffle reduction; at each level a lane keeps one half of its columns, so that
        // lane k ends with column k
#pragma unroll
        for (int j = 0; j < 32; ++j) s4[j] *= dy;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int k = 0; k < 32; ++k)
                if (k < o) {
                    const float keep = up ? s4[k + o] : s4[k], send = up ? s4[k] : s4[k + o];
                    s4[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
        }
        red[warp & 3][c0 + lane] = s4[0];

        // ---- backward --------------------------------------------------------------------------
        // dz_{l} = da_l SiLU'(z_l) into an operand tile: da_l in columns 384.., SiLU' in 128 (l - 1)..
        auto input_grad = [&](int l, unsigned char* dst) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float v[16], d[16];
                tc::tmem_ld16(at + (uint32_t)(384 + 16 * h), v);
                tc::tmem_ld16(at + (uint32_t)(128 * (l - 1) + 16 * h), d);
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] *= d[j];
                put16(dst, row, c0 + 16 * h, v);
            }
            bar_arrive(BAR_DZ + 4 - l, TILE_THREADS);
        };
        // dW (rows out, columns in) from TMEM column dcol to the partials, [in][out]
        auto weight_grad = [&](int l, uint32_t dcol) {
            float* g = gp + w_off(l) + row;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float v[16];
                tc::tmem_ld16(at + dcol + (uint32_t)(16 * h), v);
#pragma unroll
                for (int j = 0; j < 16; ++j) g[(c0 + 16 * h + j) * H] = v[j];
            }
        };
        wait_a();
        input_grad(3, W4);
        operands_ready();
        if (t == 0) {
            issue<H>(tm + 384, W4, false, W3, true, H); // da2 = dz3 W3
            tc::mma_commit(&mb_a);
            issue<H>(tm + 256, D4, true, A3, true, H);  // dW4 = dz4^T a3
            tc::mma_commit(&mb_b);
            gp[OFF_B5] = red2[0][0] + red2[1][0] + red2[2][0] + red2[3][0];
            A.loss_part[blockIdx.x] = red2[0][1] + red2[1][1] + red2[2][1] + red2[3][1];
        }
        if (cg == 1) gp[OFF_W5 + row] = red[0][row] + red[1][row] + red[2][row] + red[3][row];
        wait_a();
        input_grad(2, W3);
        wait_b();
        if (cg == 0) { // a3 is done with: the inputs again, for dW1
            *reinterpret_cast<uint4*>(A3 + tc::cm_offset(row, 0, ROWS)) = x0;
            *reinterpret_cast<uint4*>(A3 + tc::cm_offset(row, 8, ROWS)) = x1;
        }
        operands_ready();
        if (t == 0) {
            issue<H>(tm + 384, W3, false, W2, true, H); // da1 = dz2 W2
            tc::mma_commit(&mb_a);
            issue<H>(tm + 128, W4, true, A2, true, H);  // dW3 = dz3^T a2
            tc::mma_commit(&mb_b);
        }
        weight_grad(4, 256);
        bar_sync(BAR_D4_FREE, TILE_THREADS);
        wait_a();
        tc::launch_dependents();
        input_grad(1, D4);
        wait_b();
        operands_ready();
        if (t == 0) {
            issue<H>(tm + 384, D4, true, A3, true, KIN); // dW1 = dz1^T x
            issue<H>(tm + 256, W3, true, A1, true, H);   // dW2 = dz2^T a1
            tc::mma_commit(&mb_a);
        }
        weight_grad(3, 128);
        wait_a();
        weight_grad(2, 256);
        if (cg == 0) {
            float v[16];
            tc::tmem_ld16(at + 384, v);
#pragma unroll
            for (int j = 0; j < KIN; ++j) gp[w_off(1) + j * H + row] = v[j];
        }
    }
    if (!ok && lane == 0) atomicExch(A.status, 1);
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tm, 512);
}

// bf16 operand copy of parameter j (a weight of layer 1..4): its place in wbf, -1 for the others
__host__ __device__ inline int bf_index(int j)
{
    if (j < OFF_B1) return OFF_BF_W1 + (int)tc::cm_offset(j / KIN, j % KIN, H) / 2;
    if (j < OFF_W2 || j >= OFF_W5) return -1;
    const int l = (j - OFF_W2) / LAYER, o = (j - OFF_W2) % LAYER;
    return o < H * H ? OFF_BF_W2 + l * H * H + (int)tc::cm_offset(o / H, o % H, H) / 2 : -1;
}

// The partial gradients lie [in][out] where the parameters lie [out][in]. Blocks of 32 (out) x 8
// (in) weights: a warp sums one input's 32 outputs (128 consecutive bytes a tile), the sums cross
// in shared memory, and each thread then has the parameter of its place in the parameters' order
// (8 consecutive inputs of an output: 32 bytes). The last blocks take the biases and the head,
// which lie alike. g: the block's sums; returns this thread's parameter, or -1.
constexpr int GRAD_THREADS = 256;
constexpr int GRAD_W1_BLOCKS = H / 32;            // inputs 0..6, with their low parts 7..13
constexpr int GRAD_W_BLOCKS = (H / 32) * (H / 8); // per hidden layer
constexpr int GRAD_VEC = 4 * H + H + 1;           // biases of layers 1..4, head weights, head bias
constexpr int GRAD_BLOCKS = GRAD_W1_BLOCKS + 3 * GRAD_W_BLOCKS + (GRAD_VEC + GRAD_THREADS - 1) / GRAD_THREADS;

// where a block's sums come from: the partials' index j of thread t's sum (-1: none), and whether
// the low part's partials (7 inputs on) are added after it
__device__ __forceinline__ int grad_source(int blk, int t, bool& lo)
{
    lo = false;
    const int o = t & 31, i = t >> 5;
    if (blk < GRAD_W1_BLOCKS) {
        lo = true;
        return i < 7 ? OFF_W1 + i * H + blk * 32 + o : -1;
    }
    blk -= GRAD_W1_BLOCKS;
    if (blk < 3 * GRAD_W_BLOCKS) {
        const int l = blk / GRAD_W_BLOCKS, k = blk % GRAD_W_BLOCKS;
        return OFF_W2 + l * LAYER + ((k >> 2) * 8 + i) * H + (k & 3) * 32 + o;
    }
    const int v = (blk - 3 * GRAD_W_BLOCKS) * GRAD_THREADS + t;
    if (v >= GRAD_VEC) return -1;
    return v < 4 * H ? b_off(1 + v / H) + v % H : OFF_W5 + v - 4 * H;
}

// the parameter that thread t of the block holds after the crossing (-1: none)
__device__ __forceinline__ int grad_param(int blk, int t)
{
    const int o = t >> 3, i = t & 7;
    if (blk < GRAD_W1_BLOCKS) return i < 7 ? OFF_W1 + (blk * 32 + o) * KIN + i : -1;
    blk -= GRAD_W1_BLOCKS;
    if (blk < 3 * GRAD_W_BLOCKS) {
        const int l = blk / GRAD_W_BLOCKS, k = blk % GRAD_W_BLOCKS;
        return OFF_W2 + l * LAYER + ((k & 3) * 32 + o) * H + (k >> 2) * 8 + i;
    }
    bool lo;
    return grad_source(blk + GRAD_W1_BLOCKS, t, lo);
}

// SUM (float or double): the tiles' partials added in tile order
template <class SUM>
__device__ __forceinline__ SUM grad_sum(const float* part, int tiles, int j, SUM g)
{
    const float* p = part + j;
    int tl = 0;
    constexpr int F = 32; // loads in flight, added in order
    for (; tl + F <= tiles; tl += F) {
        float v[F];
#pragma unroll
        for (int k = 0; k < F; ++k) v[k] = __ldcg(p + (size_t)(tl + k) * N_PARAMS);
#pragma unroll
        for (int k = 0; k < F; ++k) g += (SUM)v[k];
    }
    for (; tl < tiles; ++tl) g += (SUM)__ldcg(p + (size_t)tl * N_PARAMS);
    return g;
}

// a block's sums crossed from the partials' order into the parameters'
template <class SUM>
__device__ __forceinline__ SUM grad_cross(SUM (&s)[8][33], int blk, int t, SUM g)
{
    if (blk >= GRAD_W1_BLOCKS + 3 * GRAD_W_BLOCKS) return g; // the vectors lie alike
    s[t >> 5][t & 31] = g;
    __syncthreads();
    return s[t & 7][t >> 3];
}

// grad[j] = sum over tiles of part[tile][j] (fixed order), then Adam on the FP32
// master and refresh of the bf16 operand copies
__global__ void __launch_bounds__(GRAD_THREADS) adam_kernel(float* params, float* m, float* v, const float* part,
                                                            int tiles, __nv_bfloat16* wbf, float lr, float b1, float b2,
                                                            float eps, float bc1, float bc2)
{
    __shared__ float s[8][33];
    const int t = threadIdx.x, blk = blockIdx.x;
    bool lo;
    const int js = grad_source(blk, t, lo);
    float g = 0.f;
    tc::wait_previous();
    if (js >= 0) {
        g = grad_sum(part, tiles, js, g);
        // W1 columns f and f + 7 carry the hi and lo bf16 parts of feature f with one
        // tied weight: column f's thread applies the summed gradient to both; columns
        // 14 and 15 are padding and stay zero
        if (lo) g = grad_sum(part, tiles, js + 7 * H, g);
    }
    tc::launch_dependents();
    g = grad_cross(s, blk, t, g);
    const int j = grad_param(blk, t);
    if (j < 0) return;
    const float mj = fmaf(b1, m[j], (1.f - b1) * g);
    const float vj = fmaf(b2, v[j], (1.f - b2) * g * g);
    m[j] = mj;
    v[j] = vj;
    const float p = params[j] - lr * (mj / bc1) / (sqrtf(vj / bc2) + eps);
    params[j] = p;
    const int bj = bf_index(j);
    if (bj >= 0) wbf[bj] = __float2bfloat16(p);
    if (j < OFF_B1) {
        params[j + 7] = p;
        wbf[bf_index(j + 7)] = __float2bfloat16(p);
    }
}

// the gradient alone, in the parameters' order (W1's tied columns apart): the tiles' partials
// summed in FP64 in tile order, rounded once
__global__ void __launch_bounds__(GRAD_THREADS) gradient_kernel(const float* part, int tiles, float* grad)
{
    __shared__ double s[8][33];
    const int t = threadIdx.x, blk = blockIdx.x;
    bool lo;
    const int js = grad_source(blk, t, lo);
    const double g = grad_cross(s, blk, t, js >= 0 ? grad_sum(part, tiles, js, 0.0) : 0.0);
    const int j = grad_param(blk, t);
    if (j >= 0) grad[j] = (float)g;
    if (blk < GRAD_W1_BLOCKS) { // the low parts' columns, and the padding's
        for (int k = t; k < 9 * 32; k += GRAD_THREADS) {
            const int i = 7 + k / 32, o = blk * 32 + k % 32;
            grad[OFF_W1 + o * KIN + i] = (float)grad_sum(part, tiles, OFF_W1 + i * H + o, 0.0);
        }
    }
}

// tail averaging of the weights: avg = params (k == 0), else avg += (params - avg) / (k + 1)
__global__ void weight_avg_kernel(const float* __restrict__ params, float* __restrict__ avg, int k)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= N_PARAMS) return;
    avg[j] = k == 0 ? params[j] : fmaf(params[j] - avg[j], 1.0f / (float)(k + 1), avg[j]);
}

// the model takes the averaged weights, and its bf16 operand copies follow (as in adam_kernel)
__global__ void weight_avg_finish_kernel(float* __restrict__ params, const float* __restrict__ avg,
                                         __nv_bfloat16* __restrict__ wbf)
{
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= N_PARAMS) return;
    if (j < OFF_B1 && j % KIN >= 7) return; // the tied hi/lo columns are written by their partner
    const float p = avg[j];
    params[j] = p;
    const int bj = bf_index(j);
    if (bj >= 0) wbf[bj] = __float2bfloat16(p);
    if (j < OFF_B1) {
        params[j + 7] = p;
        wbf[bf_index(j + 7)] = __float2bfloat16(p);
    }
}

__global__ void sum_kernel(const float* x, int n, float* out)
{
    __shared__ float s[256];
    float a = 0.f;
    for (int i = threadIdx.x; i < n; i += 256) a += x[i];
    s[threadIdx.x] = a;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = s[0];
}

// SiLU of two columns at once for inference: silu(z) = z sigmoid(z), sigmoid(z) = (1 + tanh(z/2)) / 2,
// with one special-function-unit tanh per value (the exponential and reciprocal form takes two)
// and the arithmetic on packed pairs. tanh.approx is within about 2^-11 of tanh, well inside the
// bf16 rounding (2^-9 relative) the next layer's operand gets anyway.
__device__ __forceinline__ float2 silu2_infer(float2 z)
{
    const float2 h = __fmul2_rn(z, make_float2(0.5f, 0.5f));
    float t0, t1;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t0) : "f"(h.x));
    asm("tanh.approx.f32 %0, %1;" : "=f"(t1) : "f"(h.y));
    return __ffma2_rn(h, make_float2(t0, t1), h); // z/2 (1 + tanh(z/2))
}

// ---------------------------------------------------------------------------
// Fused inference: one persistent CTA per SM, three tiles of 128 cells in flight, each with its
// own 256 threads, TMEM accumulator (128 columns), mbarrier and named barrier; the weights are
// resident in shared memory and shared by all. Two warps share a tile's 32 rows, one half of the
// columns each: an epilogue (bias, SiLU, the next operand) is bound by the latency of its column
// blocks rather than by the special-function unit (16 tanh a clock: 1024 clocks for a tile's
// layer), so it has two warps a scheduler and tile, and each block's accumulator is requested
// while the one before it is worked on. With one warp and no request ahead an epilogue took 3800
// clocks beside two others, and 2^20 cells 0.22 ms; like this 0.185. (What holds it above the
// special-function bound of 0.11 ms is the queue that those operations share with shared memory,
// which the products' operand reads fill.)
//
// Cells come as rows of normalised features, or as a lattice: its features are one word (the bf16
// pair hi, lo) a log-moneyness, maturity and parameter, from tables that a small kernel fills, so
// a tile's rows are put together from seven words and no feature is stored. Building them per
// cell, in FP64 with seven divisions, took 0.23 ms for 2^20 cells.
//
// An ensemble's members run one after the other in the same launch, their outputs added in member
// order. The price scale of a lattice cell is FP64 work (two normal distribution functions), and
// FP64 issues at 1/64 of the FP32 rate; four more warps do it beside the networks, whose pipes it
// does not use, and the outputs are scaled at the end. As a kernel of its own, with the library's
// normcdf, it took 0.48 ms.
// ---------------------------------------------------------------------------
constexpr int INFER_TILES = 3;                 // tiles in flight
constexpr int INFER_GROUP = 256;               // threads a tile
constexpr int INFER_MAIN = INFER_TILES * INFER_GROUP;
constexpr int INFER_LATTICE_THREADS = INFER_MAIN + ROWS; // and the scale's
constexpr uint32_t INFER_TMEM_COLS = 512;      // a power of two >= 128 x INFER_TILES
__device__ __forceinline__ uint32_t feature_word(float v)
{
    const __nv_bfloat16 h = __float2bfloat16(v), l = __float2bfloat16(v - __bfloat162float(h));
    return (uint32_t)__bfloat16_as_ushort(h) | ((uint32_t)__bfloat16_as_ushort(l) << 16);
}

template <bool LATTICE>
__global__ void __launch_bounds__(LATTICE ? INFER_LATTICE_THREADS : INFER_MAIN, 1) infer_kernel(const InferArgs A)
{
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ uint64_t mbar[INFER_TILES], mb_w;
    __shared__ uint32_t tm_s;
    __shared__ __align__(16) float sb[4 * H + H + 4]; // biases of layers 1..4, head weights, head bias
    unsigned char* sW1 = sm;               // 128 x 16
    unsigned char* sW = sW1 + H * KIN * 2; // 3 x (128 x 128)
    unsigned char* tiles_sm = sW + 3 * H * H * 2;
    double* s_phi = reinterpret_cast<double*>(tiles_sm + INFER_TILES * (ROWS * KIN * 2 + ROWS * H * 2));
    const int t = threadIdx.x, warp = t >> 5, g = t / INFER_GROUP; // g: the tile slot, or 3 for the scale's warps
    const int half = (t >> 7) & 1, r = t & 127;
    if (warp == 0) tc::tmem_alloc(&tm_s, INFER_TMEM_COLS);
    if (t == 0) {
        for (int w = 0; w < INFER_TILES; ++w) tc::mbar_init(&mbar[w], 1);
        tc::mbar_init(&mb_w, 1);
        tc::fence_mbar_init();
        tc::fence_smem_async();
    }
    if (LATTICE)
        for (int i = t; i < PHI_NODES * PHI_COEF; i += INFER_LATTICE_THREADS) s_phi[i] = A.L.phi[i];
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const int tiles = (A.n + ROWS - 1) / ROWS;
    const int stride = INFER_TILES * gridDim.x;
    const uint32_t per = LATTICE ? A.L.n_lm * A.L.n_T : 1;

    if (LATTICE && g == INFER_TILES) {
        // the price scale of every cell of this CTA's tiles
        for (int tile0 = INFER_TILES * blockIdx.x; tile0 < tiles && !A.scale_done; tile0 += stride)
            for (int tile = tile0; tile < min(tile0 + INFER_TILES, tiles); ++tile) {
                const uint32_t c = (uint32_t)tile * ROWS + (uint32_t)r;
                if (c >= (uint32_t)A.n) break;
                const uint32_t set = c / per, q = c % per, j = q / A.L.n_lm, k = q % A.L.n_lm;
                const double2 v = A.L.set_T[(size_t)set * A.L.n_T + j], m = A.L.lm[k];
                const double d1 = fma(-m.x, v.x, v.y);
                const double bs = fma(-m.y, phi_table(s_phi, fma(-2.0, v.y, d1)), phi_table(s_phi, d1));
                A.scale[c] = sqrt(fma(bs, bs, A.L.floor2));
            }
    } else {
        unsigned char* sX = tiles_sm + g * (ROWS * KIN * 2 + ROWS * H * 2); // this tile's 128 x 16
        unsigned char* sAct = sX + ROWS * KIN * 2;                          // and 128 x 128
        const uint32_t acc = tm_s + (uint32_t)(g * 128);
        const uint32_t at = acc + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(half * 64); // this thread's columns
        uint32_t phase = 0;
        bool ok = true;
#pragma unroll 1
        for (int m = 0; m < A.members; ++m) {
            // the member's weights, once every tile of the one before is done
            if (m > 0) asm volatile("bar.sync 8, %0;" ::"n"(INFER_MAIN) : "memory");
            if (t == 0) {
                tc::fence_smem_async();
                tc::mbar_expect(&mb_w, N_BF * 2);
                for (int i = 0; i < N_BF * 2; i += 4096) // W1 and W2..W4 follow on in both memories
                    tc::bulk_load(sm + i, reinterpret_cast<const unsigned char*>(A.wbf[m]) + i, 4096, &mb_w);
            }
            const float* params = A.params[m];
            for (int i = t; i < 4 * H; i += INFER_MAIN) sb[i] = params[b_off(1 + i / H) + i % H];
            for (int i = t; i <= H; i += INFER_MAIN) sb[4 * H + i] = params[OFF_W5 + i]; // and the head bias
            if (t == 0) ok = tc::mbar_wait(&mb_w, (uint32_t)(m & 1)) && ok;
            asm volatile("bar.sync 8, %0;" ::"n"(INFER_MAIN) : "memory");
#pragma unroll 1
            for (int tile = INFER_TILES * blockIdx.x + g; tile < tiles; tile += stride) {
                const int64_t c = (int64_t)tile * ROWS + r;
                // row r of the input tile: hi parts in columns 0..6, lo parts in 7..13; each half of
                // the group stores one 16-byte chunk
                uint32_t f[7] = {0u, 0u, 0u, 0u, 0u, 0u, 0u};
                if (c < A.n) {
                    if (LATTICE) {
                        const uint32_t set = (uint32_t)c / per, q = (uint32_t)c % per;
                        f[0] = __ldg(A.L.f_lm + q % A.L.n_lm);
                        f[1] = __ldg(A.L.f_T + q / A.L.n_lm);
#pragma unroll
                        for (int i = 0; i < 5; ++i) f[2 + i] = __ldg(A.L.f_set + (size_t)set * 5 + i);
                    } else {
#pragma unroll
                        for (int i = 0; i < 7; ++i) f[i] = feature_word(__ldg(A.x + c * 7 + i));
                    }
                }
                uint4 v;
                if (half == 0) // hi 0..6, lo 0
                    v = make_uint4(__byte_perm(f[0], f[1], 0x5410), __byte_perm(f[2], f[3], 0x5410),
                                   __byte_perm(f[4], f[5], 0x5410), __byte_perm(f[6], f[0], 0x7610));
                else // lo 1..6, padding
                    v = make_uint4(__byte_perm(f[1], f[2], 0x7632), __byte_perm(f[3], f[4], 0x7632),
                                   __byte_perm(f[5], f[6], 0x7632), 0u);
                *reinterpret_cast<uint4*>(sX + tc::cm_offset(r, 8 * half, ROWS)) = v;
                float o = sb[5 * H];
#pragma unroll 1
                for (int l = 1; l <= 4; ++l) {
                    // operand writes of every thread of the group -> visible to the tensor core
                    tc::fence_smem_async();
                    tc::fence_before_sync();
                    bar_sync(1 + g, INFER_GROUP);
                    tc::fence_after_sync();
                    if ((t & (INFER_GROUP - 1)) == 0) {
                        if (l == 1) issue<KIN>(acc, sX, false, sW1, false, H);
                        else issue<H>(acc, sAct, false, sW + (l - 2) * H * H * 2, false, H);
                        tc::mma_commit(&mbar[g]);
                    }
                    ok = tc::mbar_wait(&mbar[g], phase) && ok;
                    phase ^= 1u;
                    tc::fence_after_sync();
                    const float* bias = sb + (l - 1) * H + half * 64;
                    uint32_t u[2][16];
                    tc::tmem_ld16_start(at, u[0]);
#pragma unroll
                    for (int q = 0; q < 4; ++q) { // blocks of 16 columns, the next one's load in flight
                        tc::tmem_ld16_wait(u[q & 1]);
                        if (q < 3) tc::tmem_ld16_start(at + (uint32_t)(16 * (q + 1)), u[(q + 1) & 1]);
                        float a[16];
#pragma unroll
                        for (int j = 0; j < 16; j += 4) {
                            const float4 b4 = *reinterpret_cast<const float4*>(bias + 16 * q + j);
                            const float2 z0 = __fadd2_rn(make_float2(__uint_as_float(u[q & 1][j]), __uint_as_float(u[q & 1][j + 1])),
                                                         make_float2(b4.x, b4.y));
                            const float2 z1 = __fadd2_rn(make_float2(__uint_as_float(u[q & 1][j + 2]), __uint_as_float(u[q & 1][j + 3])),
                                                         make_float2(b4.z, b4.w));
                            const float2 s0 = silu2_infer(z0), s1 = silu2_infer(z1);
                            a[j] = s0.x;
                            a[j + 1] = s0.y;
                            a[j + 2] = s1.x;
                            a[j + 3] = s1.y;
                        }
                        if (l < 4) {
                            // the products that read sAct are done: the next operand goes over it
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                __align__(16) __nv_bfloat162 hv[4];
#pragma unroll
                                for (int j = 0; j < 4; ++j)
                                    hv[j] = __floats2bfloat162_rn(a[h * 8 + 2 * j], a[h * 8 + 2 * j + 1]);
                                *reinterpret_cast<uint4*>(sAct + tc::cm_offset(r, half * 64 + 16 * q + h * 8, ROWS)) =
                                    *reinterpret_cast<const uint4*>(hv);
                            }
                        } else if (half == 0) {
#pragma unroll
                            for (int j = 0; j < 16; ++j) o = fmaf(sb[4 * H + 16 * q + j], a[j], o);
                        } else {
                            tc::tmem_st16(at + (uint32_t)(16 * q), a); // for the head's sum, in column order
                        }
                    }
                }
                // the head: columns 0..63 are in o; the same thread goes on with the other half's
                if (half) tc::tmem_wait_st();
                tc::fence_before_sync();
                bar_sync(1 + g, INFER_GROUP);
                tc::fence_after_sync();
                if (half == 0) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        float a[16];
                        tc::tmem_ld16(at + (uint32_t)(64 + 16 * q), a);
#pragma unroll
                        for (int j = 0; j < 16; ++j) o = fmaf(sb[4 * H + 64 + 16 * q + j], a[j], o);
                    }
                    if (c < A.n) {
                        float s = m == 0 ? o : A.y[c] + o;
                        if (m == A.members - 1) s *= 1.0f / (float)A.members;
                        A.y[c] = s;
                    }
                }
            }
        }
        if (!ok && (t & 31) == 0) atomicExch(A.status, 1);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tm_s, INFER_TMEM_COLS);
    if (LATTICE) // the CTA's own tiles, outputs times scale
        for (int tile0 = INFER_TILES * blockIdx.x; tile0 < tiles; tile0 += stride)
            for (int c = tile0 * ROWS + t; c < min((tile0 + INFER_TILES) * ROWS, A.n); c += INFER_LATTICE_THREADS)
                A.price[c] = (float)((double)A.y[c] * A.scale[c]);
}

// the price scale of every cell by the library's distribution function (TABLE_FLOOR)
__global__ void __launch_bounds__(256) lattice_scale_kernel(const InferArgs A)
{
    const uint32_t per = A.L.n_lm * A.L.n_T;
    for (uint32_t c = blockIdx.x * 256 + threadIdx.x; c < (uint32_t)A.n; c += gridDim.x * 256) {
        const uint32_t set = c / per, q = c % per, j = q / A.L.n_lm, k = q % A.L.n_lm;
        const double2 v = A.L.set_T[(size_t)set * A.L.n_T + j], m = A.L.lm[k];
        const double d1 = fma(-m.x, v.x, v.y);
        const double bs = normcdf(d1) - m.y * normcdf(fma(-2.0, v.y, d1));
        A.scale[c] = sqrt(fma(bs, bs, A.L.floor2));
    }
}

} // namespace mlp

// ---- launchers -----------------------------------------------------------------
// the tile kernel's shared-memory limit, once per device (not inside a training loop)
cudaError_t mlp_train_prepare()
{
    return cudaFuncSetAttribute(mlp::train_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)mlp::TILE_SMEM);
}

// a launch whose start may overlap the end of the stream's previous kernel (tc::wait_previous)
template <class... P, class... Q>
static cudaError_t launch_overlapped(void (*k)(P...), int grid, int threads, size_t smem, cudaStream_t st, Q... args)
{
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3((unsigned)grid);
    c.blockDim = dim3((unsigned)threads);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, k, P(args)...);
}

// the partial gradients and losses of a batch's tiles
cudaError_t mlp_train_tiles(const mlp::TileArgs& A, cudaStream_t st)
{
    return launch_overlapped(mlp::train_tile_kernel, A.rows / mlp::ROWS, mlp::TILE_THREADS, mlp::TILE_SMEM, st, A);
}

cudaError_t mlp_adam(float* params, float* m, float* v, const float* part, int tiles, __nv_bfloat16* wbf, float lr,
                     float b1, float b2, float eps, float bc1, float bc2, cudaStream_t st)
{
    return launch_overlapped(mlp::adam_kernel, mlp::GRAD_BLOCKS, mlp::GRAD_THREADS, 0, st, params, m, v, part, tiles, wbf,
                             lr, b1, b2, eps, bc1, bc2);
}

cudaError_t mlp_gradient(const float* part, int tiles, float* grad, cudaStream_t st)
{
    mlp::gradient_kernel<<<mlp::GRAD_BLOCKS, mlp::GRAD_THREADS, 0, st>>>(part, tiles, grad);
    return cudaGetLastError();
}

cudaError_t mlp_loss(const float* loss_part, int tiles, float* loss, cudaStream_t st)
{
    mlp::sum_kernel<<<1, 256, 0, st>>>(loss_part, tiles, loss);
    return cudaGetLastError();
}

cudaError_t mlp_weight_avg(const float* params, float* avg, int k, cudaStream_t st)
{
    mlp::weight_avg_kernel<<<(mlp::N_PARAMS + 255) / 256, 256, 0, st>>>(params, avg, k);
    return cudaGetLastError();
}

cudaError_t mlp_weight_avg_finish(float* params, const float* avg, __nv_bfloat16* wbf, cudaStream_t st)
{
    mlp::weight_avg_finish_kernel<<<(mlp::N_PARAMS + 255) / 256, 256, 0, st>>>(params, avg, wbf);
    return cudaGetLastError();
}

// a training set as the tile kernel reads it: each feature a bf16 pair hi + lo (columns f and
// f + 7, tied weights), keeping about 16 significant bits of the input, and the loss weights
// 1 / scale^2 (scale null: 1)
__global__ void pack_set_kernel(const float* __restrict__ x, const float* __restrict__ scale, int64_t n,
                                __nv_bfloat16* __restrict__ X, float* __restrict__ W)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    __align__(16) __nv_bfloat16 h[mlp::KIN];
#pragma unroll
    for (int f = 0; f < 7; ++f) {
        const float v = x[i * 7 + f];
        h[f] = __float2bfloat16(v);
        h[7 + f] = __float2bfloat16(v - __bfloat162float(h[f]));
    }
    h[14] = h[15] = __float2bfloat16(0.f);
    uint4* dst = reinterpret_cast<uint4*>(X + i * mlp::KIN);
    dst[0] = reinterpret_cast<const uint4*>(h)[0];
    dst[1] = reinterpret_cast<const uint4*>(h)[1];
    if (W) {
        const double sc = scale ? (double)scale[i] : 1.0;
        W[i] = (float)(1.0 / (sc * sc));
    }
}

cudaError_t mlp_pack_set(const float* x, const float* scale, int64_t n, __nv_bfloat16* X, float* W, cudaStream_t st)
{
    pack_set_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(x, scale, n, X, W);
    return cudaGetLastError();
}

// the lattice's tables (LatticeArgs), one thread an entry
__device__ __forceinline__ double clip(const LatticeArgs& A, int q, double f)
{
    return fmin(fmax(f, A.lo[q]), A.hi[q]);
}

// 2 (f - lo) / (hi - lo) - 1 in FP64, then to FP32, as the host normalisation
__device__ __forceinline__ uint32_t lattice_word(const LatticeArgs& A, int q, double f)
{
    return mlp::feature_word((float)(2.0 * (clip(A, q, f) - A.lo[q]) / (A.hi[q] - A.lo[q]) - 1.0));
}

__global__ void __launch_bounds__(256) lattice_tables_kernel(const LatticeArgs A)
{
    const int n_st = A.n_sets * A.n_T; // at most the cells
    const int64_t total = (int64_t)n_st + (int64_t)A.n_sets * 5 + A.n_lm + A.n_T;
    for (int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x; e < total; e += (int64_t)gridDim.x * 256) {
        if (e < n_st) {
            // the expected average Heston variance over [0, T]: sd of the Black-Scholes price
            const double* p = A.params + (e / A.n_T) * 5;
            const double T = clip(A, 1, A.Ts[e % A.n_T]), kappa = clip(A, 2, p[0]), theta = clip(A, 3, p[1]),
                         v0 = clip(A, 6, p[4]);
            const double kt = kappa * T;
            const double var = theta + (v0 - theta) * (1.0 - exp(-kt)) / kt;
            const double sd = sqrt(fmax(var, 1e-8) * T);
            A.set_T[e] = make_double2(1.0 / sd, 0.5 * sd);
            continue;
        }
        int64_t i = e - n_st;
        if (i < (int64_t)A.n_sets * 5) {
            A.f_set[i] = lattice_word(A, 2 + (int)(i % 5), A.params[i]);
        } else if ((i -= (int64_t)A.n_sets * 5) < A.n_lm) {
            const double f = clip(A, 0, A.lms[i]);
            A.f_lm[i] = lattice_word(A, 0, A.lms[i]);
            A.lm[i] = make_double2(f, exp(f));
        } else {
            i -= A.n_lm;
            A.f_T[i] = lattice_word(A, 1, A.Ts[i]);
        }
    }
}

cudaError_t lattice_tables(const LatticeArgs& A, int sms, cudaStream_t st)
{
    const int64_t total = (int64_t)A.n_sets * (A.n_T + 5) + A.n_lm + A.n_T;
    lattice_tables_kernel<<<(unsigned)std::min<int64_t>((total + 255) / 256, 8 * sms), 256, 0, st>>>(A);
    return cudaGetLastError();
}

cudaError_t lattice_scale(const mlp::InferArgs& A, int sms, cudaStream_t st)
{
    mlp::lattice_scale_kernel<<<(unsigned)std::min((A.n + 255) / 256, 8 * sms), 256, 0, st>>>(A);
    return cudaGetLastError();
}

// Phi's Taylor coefficients about the nodes k / 8 (phi.cuh)
void phi_coefficients(double* out)
{
    for (int k = -PHI_MID; k <= PHI_MID; ++k, out += PHI_COEF) {
        const double x = k / 8.0, phi = std::exp(-0.5 * x * x) / std::sqrt(2.0 * 3.14159265358979323846);
        double he0 = 1.0, he1 = x, f = 1.0; // He_0, He_1; n!
        out[0] = 0.5 * std::erfc(-x / std::sqrt(2.0));
        for (int n = 1; n < PHI_COEF; ++n) {
            f *= n;
            out[n] = (n % 2 ? phi : -phi) * he0 / f;
            const double he2 = x * he1 - n * he0;
            he0 = he1;
            he1 = he2;
        }
    }
}

cudaError_t mlp_infer(const mlp::InferArgs& A, bool lattice, int sms, cudaStream_t st)
{
    using namespace mlp;
    const size_t smem = (size_t)N_BF * 2 + INFER_TILES * (size_t)(ROWS * KIN + ROWS * H) * 2 +
                        (lattice ? sizeof(double) * PHI_NODES * PHI_COEF : 0);
    auto k = lattice ? infer_kernel<true> : infer_kernel<false>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int tiles = (A.n + ROWS - 1) / ROWS, grid = std::min((tiles + INFER_TILES - 1) / INFER_TILES, sms);
    k<<<grid, lattice ? INFER_LATTICE_THREADS : INFER_MAIN, smem, st>>>(A);
    return cudaGetLastError();
}

} // namespace thoth
