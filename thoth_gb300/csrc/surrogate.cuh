// surrogate.cuh — the surrogate's network and the arguments and launchers of its kernels
// (surrogate.cu), shared with the C ABI (surrogate_host.cu).
#pragma once

#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace thoth {

// ===========================================================================
// The surrogate MLP: 7 inputs (padded to 16) -> 4 x 128 SiLU -> 1.
// Parameters (FP32 master, offsets in floats):
//   W1 [128][16], b1[128], W2..W4 [128][128] + b[128], w5[128], b5[1]
// BF16 copies of W1..W4 are the tensor-core operands, kept in global memory in the operand
// layout (tc::cm_offset), so a CTA's copy of them is a plain block copy.
// ===========================================================================
namespace mlp {

constexpr int H = 128;      // hidden width
constexpr int NF = 7;       // input features
constexpr int KIN = 16;     // a feature pair each (hi, lo), padded to one MMA K slice
constexpr int ROWS = 128;   // rows per tile = MMA M
constexpr int OFF_W1 = 0;
constexpr int OFF_B1 = OFF_W1 + H * KIN;
constexpr int OFF_W2 = OFF_B1 + H;
constexpr int LAYER = H * H + H; // W + b of a hidden layer 2..4
constexpr int OFF_W5 = OFF_W2 + 3 * LAYER;
constexpr int OFF_B5 = OFF_W5 + H;
constexpr int N_PARAMS = OFF_B5 + 1;
constexpr int OFF_BF_W1 = 0;                 // bf16 weights, offsets in elements
constexpr int OFF_BF_W2 = H * KIN;
constexpr int N_BF = H * KIN + 3 * H * H;

__host__ __device__ constexpr int w_off(int l) { return l == 1 ? OFF_W1 : OFF_W2 + (l - 2) * LAYER; }
__host__ __device__ constexpr int b_off(int l) { return w_off(l) + H * (l == 1 ? KIN : H); }

// one batch's tiles (train_tile_kernel)
struct TileArgs {
    const __nv_bfloat16* x; // [n][16] normalised inputs of the training set
    const float* y;         // [n] targets
    const float* w;         // [n] loss weights 1 / scale^2
    const int* perm;        // row r of the batch is perm[first + r] (null: first + r)
    int64_t first;
    int rows;               // batch rows (multiple of 128)
    const float* params;    // FP32 master
    const __nv_bfloat16* wbf; // bf16 W1..W4 in the operand layout
    float* part;            // per-tile partial gradients, [tiles][N_PARAMS]
    float* loss_part;       // [tiles]
    int* status;
};

constexpr int MAX_MEMBERS = 64; // networks of an ensemble

// a lattice's tables, and one serving call (infer_kernel)
struct LatticeTables {
    const uint32_t* f_lm;  // [n_lm] feature words (bf16 hi, lo << 16), clipped and normalised
    const uint32_t* f_T;   // [n_T]
    const uint32_t* f_set; // [n_sets][5]
    const double2* set_T;  // [n_sets][n_T] 1 / sd, sd / 2 of the price scale
    const double2* lm;     // [n_lm] clipped log-moneyness, its exponential
    const double* phi;     // [PHI_NODES][PHI_COEF]
    double floor2;         // squared scale floor
    uint32_t n_lm, n_T;
};

struct InferArgs {
    const float* x;   // [n][7] normalised rows (not a lattice)
    LatticeTables L;  // a lattice
    int n;            // cells
    int members;
    float* y;         // [n] outputs, the members' mean
    double* scale;    // [n] a lattice's price scale
    int scale_done;   // 1: the scale is there already (lattice_scale)
    float* price;     // [n] a lattice's prices
    int* status;
    const float* params[MAX_MEMBERS];
    const __nv_bfloat16* wbf[MAX_MEMBERS];
};

} // namespace mlp

// ---------------------------------------------------------------------------
// Lattice serving: the cells of n_sets parameter sets x n_T maturities x n_lm
// log-moneyness, cell c = (set * n_T + j) * n_lm + k with raw features
// (lm[k], T[j], kappa, theta, xi, rho, v0 of the set), clipped to the training
// box and normalised, and the network's output scaled back to a price in units
// of spot. Everything a cell needs is one word or number per axis value or per
// (set, maturity); lattice_tables fills those.
// ---------------------------------------------------------------------------
struct LatticeArgs {
    const double* params; // [n_sets][5] kappa, theta, xi, rho, v0
    const double* lms;    // [n_lm]
    const double* Ts;     // [n_T]
    double lo[7], hi[7];  // training box
    int n_sets, n_lm, n_T;
    uint32_t *f_lm, *f_T, *f_set;
    double2 *set_T, *lm;
};

cudaError_t mlp_train_prepare();
cudaError_t mlp_train_tiles(const mlp::TileArgs& A, cudaStream_t st);
cudaError_t mlp_adam(float* params, float* m, float* v, const float* part, int tiles, __nv_bfloat16* wbf, float lr,
                     float b1, float b2, float eps, float bc1, float bc2, cudaStream_t st);
cudaError_t mlp_gradient(const float* part, int tiles, float* grad, cudaStream_t st);
cudaError_t mlp_loss(const float* loss_part, int tiles, float* loss, cudaStream_t st);
cudaError_t mlp_pack_set(const float* x, const float* scale, int64_t n, __nv_bfloat16* X, float* W, cudaStream_t st);
cudaError_t mlp_weight_avg(const float* params, float* avg, int k, cudaStream_t st);
cudaError_t mlp_weight_avg_finish(float* params, const float* avg, __nv_bfloat16* wbf, cudaStream_t st);
cudaError_t lattice_tables(const LatticeArgs& A, int sms, cudaStream_t st);
// Below this floor the scale of a cell far out of the money is smaller than what the table of Phi holds
// of it (its tail ends at 3e-18, and is good to 2e-10 there), and lattice_scale takes the library's
// function for every cell. From 1e-9 on the prices are the same bits either way; at 1e-15 the table's
// differed by 2e-6, at 1e-30 they had nothing in common with the scale.
constexpr double TABLE_FLOOR = 1e-10;
cudaError_t lattice_scale(const mlp::InferArgs& A, int sms, cudaStream_t st);
cudaError_t mlp_infer(const mlp::InferArgs& A, bool lattice, int sms, cudaStream_t st);

} // namespace thoth
