// surrogate_host.cu — C ABI of the learned Heston surrogate: a 7 -> 4 x 128
// SiLU -> 1 MLP trained and served by the tcgen05 kernels of surrogate.cu.
// No reference counterpart: the reference has no learned pricer.
#include "thoth_gpu.h"
#include "phi.cuh"
#include "surrogate.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <new>
#include <stdexcept>
#include <random>
#include <string>
#include <vector>

using namespace thoth;

namespace {
thread_local std::string s_err;
std::mutex s_mu;
int sfail(int code, const std::string& m)
{
    s_err = m;
    return code;
}
#define STRY(expr)                                                                                              \
    do {                                                                                                        \
        cudaError_t e_ = (expr);                                                                                \
        if (e_ != cudaSuccess)                                                                                  \
            return sfail(e_ == cudaErrorMemoryAllocation ? THOTH_GPU_E_NOMEM : THOTH_GPU_E_CUDA,                \
                         std::string(#expr) + ": " + cudaGetErrorString(e_));                                    \
    } while (0)

using mlp::H, mlp::KIN, mlp::NF, mlp::LAYER, mlp::OFF_W1, mlp::OFF_W2, mlp::OFF_W5;

__nv_bfloat16 to_bf(float f)
{
    return __float2bfloat16(f);
}
} // namespace

struct ThothSurrogate {
    int np = 0, nbf = 0;
    float* params = nullptr; // FP32 master
    float* m = nullptr;
    float* v = nullptr;
    __nv_bfloat16* wbf = nullptr;
    int* status = nullptr;
    cudaStream_t st = nullptr;
    int dev = 0; // the device current when the handle was created; every call sets it
    int sms = 0;
    int64_t step = 0;
    // training buffers (grown on demand): the tiles' partial gradients and losses
    int cap_rows = 0;
    unsigned char* tb = nullptr;
    mlp::TileArgs A{};
    float* grad = nullptr;
    float* loss = nullptr;
    // inference buffer (grown on demand)
    size_t cap_inf = 0;
    unsigned char* ib = nullptr;
    // the running average of the weights over a training call's last epochs
    float* avg = nullptr;
    // device copy of a training set and its per-epoch permutation (grown on demand)
    int64_t cap_ds = 0;
    unsigned char* ds = nullptr;
    int* perm_host = nullptr; // pinned
    cudaEvent_t perm_copied = nullptr;
};

namespace {

void host_params_to_bf(const std::vector<float>& p, std::vector<__nv_bfloat16>& w)
{
    w.resize(mlp::N_BF);
    __nv_bfloat16* to = w.data();
    auto layer = [&](const float* from, int cols) { // the operand layout
        for (int kb = 0; kb < cols; kb += 8)
            for (int r = 0; r < H; r++)
                for (int k = 0; k < 8; k++) *to++ = to_bf(from[(size_t)r * cols + kb + k]);
    };
    layer(p.data() + OFF_W1, KIN);
    for (int l = 0; l < 3; l++) layer(p.data() + OFF_W2 + l * LAYER, H);
}

int upload_params(ThothSurrogate* s, const std::vector<float>& p)
{
    std::vector<__nv_bfloat16> w;
    host_params_to_bf(p, w);
    STRY(cudaMemcpyAsync(s->params, p.data(), sizeof(float) * s->np, cudaMemcpyHostToDevice, s->st));
    STRY(cudaMemcpyAsync(s->wbf, w.data(), sizeof(__nv_bfloat16) * w.size(), cudaMemcpyHostToDevice, s->st));
    STRY(cudaStreamSynchronize(s->st));
    return THOTH_GPU_OK;
}

int ensure_train(ThothSurrogate* s, int rows)
{
    if (rows <= s->cap_rows) return THOTH_GPU_OK;
    if (s->tb) cudaFree(s->tb);
    s->tb = nullptr;
    s->cap_rows = 0; // stays empty if the allocation fails
    const int tiles = rows / 128;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += (bytes + 255) & ~size_t(255);
        return o;
    };
    const size_t op = take((size_t)tiles * s->np * 4), ol = take((size_t)tiles * 4), og = take((size_t)s->np * 4),
                 oloss = take(4);
    STRY(cudaMalloc(&s->tb, off));
    s->cap_rows = rows;
    mlp::TileArgs& A = s->A;
    A.part = reinterpret_cast<float*>(s->tb + op);
    A.loss_part = reinterpret_cast<float*>(s->tb + ol);
    s->grad = reinterpret_cast<float*>(s->tb + og);
    s->loss = reinterpret_cast<float*>(s->tb + oloss);
    A.params = s->params;
    A.wbf = s->wbf;
    A.status = s->status;
    return THOTH_GPU_OK;
}

int check_status(ThothSurrogate* s)
{
    int st = 0;
    STRY(cudaMemcpyAsync(&st, s->status, sizeof(int), cudaMemcpyDeviceToHost, s->st));
    STRY(cudaStreamSynchronize(s->st));
    if (st) return sfail(THOTH_GPU_E_CUDA, "tensor-core MMA did not complete (bounded wait expired)");
    return THOTH_GPU_OK;
}

int ensure_infer(ThothSurrogate* s, size_t bytes)
{
    if (bytes <= s->cap_inf) return THOTH_GPU_OK;
    if (s->ib) cudaFree(s->ib);
    s->ib = nullptr;
    s->cap_inf = 0; // stays empty if the allocation fails
    STRY(cudaMalloc(&s->ib, bytes));
    s->cap_inf = bytes;
    return THOTH_GPU_OK;
}

// a timed region of the handle's stream: its two events, destroyed on every way out
struct Timed {
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    ~Timed()
    {
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
    }
    cudaError_t create()
    {
        const cudaError_t e = cudaEventCreate(&e0);
        return e == cudaSuccess ? cudaEventCreate(&e1) : e;
    }
};

// the results and the status word back in one wait, and the region's device time
int finish_infer(ThothSurrogate* s, Timed& T, const float* from, float* to, int64_t n, double* device_ms)
{
    int st = 0;
    STRY(cudaMemcpyAsync(to, from, sizeof(float) * (size_t)n, cudaMemcpyDeviceToHost, s->st));
    STRY(cudaMemcpyAsync(&st, s->status, sizeof(int), cudaMemcpyDeviceToHost, s->st));
    STRY(cudaStreamSynchronize(s->st));
    float ms = 0;
    cudaEventElapsedTime(&ms, T.e0, T.e1);
    if (device_ms) *device_ms = ms;
    if (st) return sfail(THOTH_GPU_E_CUDA, "tensor-core MMA did not complete (bounded wait expired)");
    return THOTH_GPU_OK;
}

// the handle's device copy of a training set of n rows: inputs packed to bf16 pairs, targets, loss
// weights, and a permutation; raw is where the caller's inputs and scales land before the packing
struct SetBuffers {
    __nv_bfloat16* x;
    float *y, *w;
    int* perm;
    float *raw_x, *raw_scale;
};

int upload_set(ThothSurrogate* s, const float* x, const float* y, const float* scale, int64_t n, SetBuffers& D)
{
    if (n > s->cap_ds) {
        if (s->ds) cudaFree(s->ds);
        if (s->perm_host) cudaFreeHost(s->perm_host);
        s->ds = nullptr;
        s->perm_host = nullptr;
        s->cap_ds = 0;
        STRY(cudaMalloc(&s->ds, (size_t)n * (KIN * 2 + 4 + 4 + 4 + NF * 4 + 4) + 2048));
        STRY(cudaHostAlloc(&s->perm_host, sizeof(int) * (size_t)n, cudaHostAllocDefault));
        if (!s->perm_copied) STRY(cudaEventCreateWithFlags(&s->perm_copied, cudaEventDisableTiming));
        s->cap_ds = n;
    }
    unsigned char* at = s->ds;
    auto take = [&](size_t bytes) {
        unsigned char* p = at;
        at += (bytes + 255) & ~size_t(255);
        return p;
    };
    D.x = reinterpret_cast<__nv_bfloat16*>(take((size_t)n * KIN * 2));
    D.y = reinterpret_cast<float*>(take((size_t)n * 4));
    D.w = reinterpret_cast<float*>(take((size_t)n * 4));
    D.perm = reinterpret_cast<int*>(take((size_t)n * 4));
    D.raw_x = reinterpret_cast<float*>(take((size_t)n * NF * 4));
    D.raw_scale = scale ? reinterpret_cast<float*>(take((size_t)n * 4)) : nullptr;
    STRY(cudaMemcpyAsync(D.raw_x, x, (size_t)n * NF * 4, cudaMemcpyHostToDevice, s->st));
    STRY(cudaMemcpyAsync(D.y, y, (size_t)n * 4, cudaMemcpyHostToDevice, s->st));
    if (scale) STRY(cudaMemcpyAsync(D.raw_scale, scale, (size_t)n * 4, cudaMemcpyHostToDevice, s->st));
    STRY(mlp_pack_set(D.raw_x, D.raw_scale, n, D.x, D.w, s->st));
    return THOTH_GPU_OK;
}

// one network's training call in three phases, so that several networks can train side by side
struct TrainRun {
    ThothSurrogate* s = nullptr;
    int64_t n = 0, steps_per_epoch = 0, total = 0, done = 0;
    int epochs = 0, avg_epochs = 0, batch = 0;
    // a cosine decay from lr to lr_lo over decay_steps steps, then lr_lo
    double lr = 0, lr_lo = 0;
    int64_t decay_steps = 1;
    SetBuffers D{};
    std::vector<int> idx; // the host permutation
    std::mt19937_64 rng;
};

// the training set up once on the member's device memory (bf16 hi/lo inputs, targets, loss
// weights) and the schedule of this call
int train_setup(TrainRun& R, ThothSurrogate* s, const float* x, const float* y, const float* scale, int64_t n,
                int epochs, int batch, double lr, uint64_t seed, int avg_epochs, double lr_avg)
{
    R.s = s;
    R.n = n;
    R.epochs = epochs;
    R.avg_epochs = avg_epochs;
    R.batch = (int)std::min<int64_t>(batch, n / 128 * 128);
    int rc = ensure_train(s, R.batch);
    if (rc) return rc;
    if (avg_epochs > 0 && !s->avg) STRY(cudaMalloc(&s->avg, sizeof(float) * s->np));
    rc = upload_set(s, x, y, scale, n, R.D);
    if (rc) return rc;
    R.idx.resize(n);
    for (int64_t i = 0; i < n; i++) R.idx[i] = (int)i;
    R.rng.seed(seed);
    R.steps_per_epoch = n / R.batch;
    R.total = R.steps_per_epoch * epochs;
    // without averaging the decay runs over every step down to zero; with it, over the steps
    // before the averaged epochs, down to lr_avg, which then holds
    R.lr = lr;
    R.lr_lo = avg_epochs > 0 ? lr_avg : 0.0;
    R.decay_steps = std::max<int64_t>(1, avg_epochs > 0 ? R.steps_per_epoch * (int64_t)(epochs - avg_epochs) : R.total);
    mlp::TileArgs& A = s->A;
    A.x = R.D.x;
    A.y = R.D.y;
    A.w = R.D.w;
    A.perm = R.D.perm;
    A.rows = R.batch;
    STRY(cudaMemsetAsync(s->status, 0, sizeof(int), s->st));
    STRY(mlp_train_prepare());
    STRY(cudaEventRecord(s->perm_copied, s->st));
    return THOTH_GPU_OK;
}

// epoch e: the next permutation is drawn on the host while the device runs the previous
// epoch; at the averaged epochs the weights at the epoch's end join the running average
int train_epoch(TrainRun& R, int e)
{
    ThothSurrogate* s = R.s;
    const double pi = 3.14159265358979323846;
    std::shuffle(R.idx.begin(), R.idx.end(), R.rng);
    STRY(cudaEventSynchronize(s->perm_copied)); // the previous permutation has left the pinned buffer
    std::memcpy(s->perm_host, R.idx.data(), sizeof(int) * (size_t)R.n);
    STRY(cudaMemcpyAsync(R.D.perm, s->perm_host, sizeof(int) * (size_t)R.n, cudaMemcpyHostToDevice, s->st));
    STRY(cudaEventRecord(s->perm_copied, s->st));
    const int tiles = R.batch / 128;
    for (int64_t b = 0; b < R.steps_per_epoch; b++, R.done++) {
        const double c = (double)std::min(R.done, R.decay_steps), step = (double)(s->step + R.done + 1);
        const float lr = (float)(R.lr_lo + (R.lr - R.lr_lo) * 0.5 * (1.0 + std::cos(pi * c / (double)R.decay_steps)) + 1e-6);
        s->A.first = b * R.batch;
        STRY(mlp_train_tiles(s->A, s->st));
        STRY(mlp_adam(s->params, s->m, s->v, s->A.part, tiles, s->wbf, lr, 0.9f, 0.999f, 1e-8f,
                      (float)(1.0 - std::pow(0.9, step)), (float)(1.0 - std::pow(0.999, step)), s->st));
    }
    if (R.avg_epochs > 0 && e >= R.epochs - R.avg_epochs)
        STRY(mlp_weight_avg(s->params, s->avg, e - (R.epochs - R.avg_epochs), s->st));
    return THOTH_GPU_OK;
}

int train_finish(TrainRun& R, double* final_loss)
{
    ThothSurrogate* s = R.s;
    if (R.avg_epochs > 0) STRY(mlp_weight_avg_finish(s->params, s->avg, s->wbf, s->st));
    s->step += R.total;
    float l = 0;
    STRY(mlp_loss(s->A.loss_part, R.batch / 128, s->loss, s->st)); // the last step's
    STRY(cudaMemcpyAsync(&l, s->loss, sizeof(float), cudaMemcpyDeviceToHost, s->st));
    STRY(cudaStreamSynchronize(s->st));
    const int rc = check_status(s);
    if (rc) return rc;
    if (final_loss) *final_loss = l / s->A.rows;
    return THOTH_GPU_OK;
}

} // namespace

extern "C" {

int thoth_gpu_surrogate_create(ThothSurrogate** out, uint64_t seed)
{
    try {
        if (!out) return sfail(THOTH_GPU_E_INVALID, "null handle pointer");
        std::lock_guard<std::mutex> lk(s_mu);
        int n = 0;
        if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) return sfail(THOTH_GPU_E_NODEVICE, "no CUDA device");
        int dev = 0;
        STRY(cudaGetDevice(&dev));
        cudaDeviceProp p;
        STRY(cudaGetDeviceProperties(&p, dev));
        if (!(p.major == 10 && p.minor == 3)) return sfail(THOTH_GPU_E_NODEVICE, "not an sm_103 device");
        ThothSurrogate* s = new ThothSurrogate();
        s->dev = dev;
        s->np = mlp::N_PARAMS;
        s->nbf = mlp::N_BF;
        s->sms = p.multiProcessorCount;
        cudaError_t e = cudaStreamCreateWithFlags(&s->st, cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaMalloc(&s->params, sizeof(float) * s->np * 3);
        if (e == cudaSuccess) e = cudaMalloc(&s->wbf, sizeof(__nv_bfloat16) * s->nbf);
        if (e == cudaSuccess) e = cudaMalloc(&s->status, sizeof(int));
        if (e != cudaSuccess) {
            delete s;
            return sfail(THOTH_GPU_E_NOMEM, std::string("surrogate allocation: ") + cudaGetErrorString(e));
        }
        s->m = s->params + s->np;
        s->v = s->params + 2 * s->np;
        // Xavier-uniform weights, zero biases; W1 only on the 7 real input columns
        std::mt19937_64 rng(seed);
        std::vector<float> h(s->np, 0.f);
        auto fill = [&](int off, int rows, int cols, int fan_in, int used_cols) {
            const double a = std::sqrt(6.0 / (fan_in + rows));
            std::uniform_real_distribution<double> U(-a, a);
            for (int r = 0; r < rows; r++)
                for (int c = 0; c < cols; c++) h[off + r * cols + c] = c < used_cols ? (float)U(rng) : 0.f;
        };
        fill(OFF_W1, H, KIN, NF, NF);
        for (int r = 0; r < H; r++) // tie the lo-part columns to the hi-part columns
            for (int f = 0; f < NF; f++) h[OFF_W1 + r * KIN + NF + f] = h[OFF_W1 + r * KIN + f];
        for (int l = 0; l < 3; l++) fill(OFF_W2 + l * LAYER, H, H, H, H);
        fill(OFF_W5, 1, H, H, H);
        int rc = upload_params(s, h);
        if (rc == THOTH_GPU_OK) {
            e = cudaMemsetAsync(s->m, 0, sizeof(float) * 2 * s->np, s->st);
            if (e == cudaSuccess) e = cudaMemsetAsync(s->status, 0, sizeof(int), s->st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s->st);
            if (e != cudaSuccess) rc = sfail(THOTH_GPU_E_CUDA, cudaGetErrorString(e));
        }
        if (rc) {
            delete s;
            return rc;
        }
        *out = s;
        return THOTH_GPU_OK;
    } catch (const std::bad_alloc&) {
        return sfail(THOTH_GPU_E_NOMEM, "out of host memory");
    } catch (const std::exception& e) {
        return sfail(THOTH_GPU_E_INVALID, std::string("host error: ") + e.what());
    }
}

int thoth_gpu_surrogate_destroy(ThothSurrogate* s)
{
    try {
        if (!s) return THOTH_GPU_OK;
        std::lock_guard<std::mutex> lk(s_mu);
        cudaSetDevice(s->dev); // frees below whatever this returns
        cudaFree(s->params);
        cudaFree(s->wbf);
        cudaFree(s->status);
        if (s->tb) cudaFree(s->tb);
        if (s->ib) cudaFree(s->ib);
        if (s->avg) cudaFree(s->avg);
        if (s->ds) cudaFree(s->ds);
        if (s->perm_host) cudaFreeHost(s->perm_host);
        if (s->perm_copied) cudaEventDestroy(s->perm_copied);
        if (s->st) cudaStreamDestroy(s->st);
        delete s;
        return THOTH_GPU_OK;
    } catch (const std::bad_alloc&) {
        return sfail(THOTH_GPU_E_NOMEM, "out of host memory");
    } catch (const std::exception& e) {
        return sfail(THOTH_GPU_E_INVALID, std::string("host error: ") + e.what());
    }
}

int thoth_gpu_surrogate_n_params(void) { return mlp::N_PARAMS; }

int thoth_gpu_surrogate_get_params(ThothSurrogate* s, float* params)
{
    try {
        if (!s || !params) return sfail(THOTH_GPU_E_INVALID, "null argument");
        std::lock_guard<std::mutex> lk(s_mu);
        STRY(cudaSetDevice(s->dev));
        STRY(cudaMemcpyAsync(params, s->params, sizeof(float) * s->np, cudaMemcpyDeviceToHost, s->st));
        STRY(cudaStreamSynchronize(s->st));
        return THOTH_GPU_OK;
    } catch (const std::bad_alloc&) {
        return sfail(THOTH_GPU_E_NOMEM, "out of host memory");
    } catch (const std::exception& e) {
        return sfail(THOTH_GPU_E_INVALID, std::string("host error: ") + e.what());
    }
}

int thoth_gpu_surrogate_set_params(ThothSurrogate* s, const float* params)
{
    try {
        if (!s || !params) return sfail(THOTH_GPU_E_INVALID, "null argument");
        std::lock_guard<std::mutex> lk(s_mu);
        STRY(cudaSetDevice(s->dev));
        std::vector<float> h(params, params + s->np);
        return upload_params(s, h);
    } catch (const std::bad_alloc&) {
        return sfail(THOTH_GPU_E_NOMEM, "out of host memory");
    } catch (const std::exception& e) {
        return sfail(THOTH_GPU_E_INVALID, std::string("host error: ") + e.what());
    }
}

int thoth_gpu_surrogate_gradient(ThothSurrogate* s, const float* x, const float* y, const float* scale, int32_t rows,
                                 float* grad, double* loss)
{
    try {
        if (!s || !x || !y || !grad || rows < 128 || rows % 128) return sfail(THOTH_GPU_E_INVALID, "rows must be a multiple of 128");
        std::lock_guard<std::mutex> lk(s_mu);
        STRY(cudaSetDevice(s->dev));
        int rc = ensure_train(s, rows);
        if (rc) return rc;
        SetBuffers D{};
        rc = upload_set(s, x, y, scale, rows, D);
        if (rc) return rc;
        mlp::TileArgs A = s->A;
        A.x = D.x;
        A.y = D.y;
        A.w = D.w;
        A.perm = nullptr;
        A.first = 0;
        A.rows = rows;
        const int tiles = rows / 128;
        STRY(cudaMemsetAsync(s->status, 0, sizeof(int), s->st));
        STRY(mlp_train_prepare());
        STRY(mlp_train_tiles(A, s->st));
        STRY(mlp_gradient(A.part, tiles, s->grad, s->st));
        STRY(mlp_loss(A.loss_part, tiles, s->loss, s->st));
        float l = 0;
        STRY(cudaMemcpyAsync(&l, s->loss, sizeof(float), cudaMemcpyDeviceToHost, s->st));
        STRY(cudaMemcpyAsync(grad, s->grad, sizeof(float) * s->np, cudaMemcpyDeviceToHost, s->st));
        rc = check_status(s);
        if (rc) return rc;
        if (loss) *loss = l / rows;
        return THOTH_GPU_OK;
    } catch (const std::bad_alloc&) {
        return sfail(THOTH_GPU_E_NOMEM, "out of host memory");
    } catch (const std::exception& e) {
        return sfail(THOTH_GPU_E_INVALID, std::string("host error: ") + e.what());
    }
}

int thoth_gpu_surrogate_train(ThothSurrogate* s, const float* x, const float* y, const float* scale, int64_t n,
                              int32_t epochs, int32_t batch, double lr, uint64_t seed, double* final_loss)
{
    return thoth_gpu_surrogate_train_avg(s, x, y, scale, n, epochs, batch, lr, seed, 0, 0.0, final_loss);
}

int thoth_gpu_surrogate_train_avg(ThothSurrogate* s, const float* x, const float* y, const float* scale, int64_t n,
                                  int32_t epochs, int32_t batch, double lr, uint64_t seed, int32_t avg_epochs,
                                  double lr_avg, double* final_loss)
{
    return thoth_gpu_surrogate_train_members(&s, 1, x, y, scale, n, epochs, batch, lr, seed, avg_epochs, lr_avg,
                                             final_loss);
}

int thoth_gpu_surrogate_train_members(ThothSurrogate* const* members, int32_t k, const float* x, const float* y,
                                      const float* scale, int64_t n, int32_t epochs, int32_t batch, double lr,
                                      uint64_t seed, int32_t avg_epochs, double lr_avg, double* final_loss)
{
    try {
        if (!members || k < 1 || k > mlp::MAX_MEMBERS || !x || !y || n < 128 || epochs < 1 || batch < 128 || batch % 128 ||
            !(lr > 0))
            return sfail(THOTH_GPU_E_INVALID, "bad training arguments (batch must be a multiple of 128)");
        if (avg_epochs < 0 || avg_epochs >= epochs || (avg_epochs > 0 && !(lr_avg > 0 && lr_avg <= lr)))
            return sfail(THOTH_GPU_E_INVALID, "bad weight averaging (0 <= avg_epochs < epochs, 0 < lr_avg <= lr)");
        if (n > ((int64_t)1 << 31) - 1) return sfail(THOTH_GPU_E_TOO_LARGE, "training set beyond 2^31 rows");
        for (int j = 0; j < k; j++) {
            if (!members[j]) return sfail(THOTH_GPU_E_INVALID, "null member");
            for (int i = 0; i < j; i++)
                if (members[i] == members[j]) return sfail(THOTH_GPU_E_INVALID, "a member appears twice");
            if (members[j]->dev != members[0]->dev) return sfail(THOTH_GPU_E_INVALID, "members on different devices");
        }
        std::lock_guard<std::mutex> lk(s_mu);
        STRY(cudaSetDevice(members[0]->dev));
        std::vector<TrainRun> runs(k);
        for (int j = 0; j < k; j++) {
            const int rc = train_setup(runs[j], members[j], x, y, scale, n, epochs, batch, lr, seed + (uint64_t)j,
                                       avg_epochs, lr_avg);
            if (rc) return rc;
        }
        // the members' epochs interleaved: each member launches its steps on its own stream, so their
        // kernels run side by side on the device
        for (int e = 0; e < epochs; e++)
            for (int j = 0; j < k; j++) {
                const int rc = train_epoch(runs[j], e);
                if (rc) return rc;
            }
        for (int j = 0; j < k; j++) {
            const int rc = train_finish(runs[j], final_loss ? final_loss + j : nullptr);
            if (rc) return rc;
        }
        return THOTH_GPU_OK;
    } catch (const std::bad_alloc&) {
        return sfail(THOTH_GPU_E_NOMEM, "out of host memory");
    } catch (const std::exception& e) {
        return sfail(THOTH_GPU_E_INVALID, std::string("host error: ") + e.what());
    }
}

int thoth_gpu_surrogate_predict(ThothSurrogate* s, const float* x, int64_t n, float* y, double* device_ms)
{
    try {
        if (!s || !x || !y || n < 1 || n > ((int64_t)1 << 30)) return sfail(THOTH_GPU_E_INVALID, "bad predict arguments");
        std::lock_guard<std::mutex> lk(s_mu);
        STRY(cudaSetDevice(s->dev));
        auto up = [](size_t b) { return (b + 255) & ~size_t(255); };
        const size_t o_y = up(sizeof(float) * NF * (size_t)n);
        int rc = ensure_infer(s, o_y + sizeof(float) * (size_t)n);
        if (rc) return rc;
        mlp::InferArgs A{};
        A.x = reinterpret_cast<const float*>(s->ib);
        A.n = (int)n;
        A.members = 1;
        A.y = reinterpret_cast<float*>(s->ib + o_y);
        A.status = s->status;
        A.params[0] = s->params;
        A.wbf[0] = s->wbf;
        Timed T;
        STRY(T.create());
        STRY(cudaMemcpyAsync(s->ib, x, sizeof(float) * NF * (size_t)n, cudaMemcpyHostToDevice, s->st));
        STRY(cudaMemsetAsync(s->status, 0, sizeof(int), s->st));
        STRY(cudaEventRecord(T.e0, s->st));
        STRY(mlp_infer(A, false, s->sms, s->st));
        STRY(cudaEventRecord(T.e1, s->st));
        return finish_infer(s, T, A.y, y, n, device_ms);
    } catch (const std::bad_alloc&) {
        return sfail(THOTH_GPU_E_NOMEM, "out of host memory");
    } catch (const std::exception& e) {
        return sfail(THOTH_GPU_E_INVALID, std::string("host error: ") + e.what());
    }
}

int thoth_gpu_surrogate_price_lattice(ThothSurrogate* s, const double* params, int32_t n_sets, const double* lms,
                                      int32_t n_lm, const double* Ts, int32_t n_T, const double* box_lo,
                                      const double* box_hi, double floor, float* prices, double* device_ms)
{
    return thoth_gpu_surrogate_price_lattice_mean(&s, 1, params, n_sets, lms, n_lm, Ts, n_T, box_lo, box_hi, floor,
                                                  prices, device_ms);
}

int thoth_gpu_surrogate_price_lattice_mean(ThothSurrogate* const* members, int32_t k, const double* params,
                                           int32_t n_sets, const double* lms, int32_t n_lm, const double* Ts,
                                           int32_t n_T, const double* box_lo, const double* box_hi, double floor,
                                           float* prices, double* device_ms)
{
    try {
        if (!members || k < 1 || k > mlp::MAX_MEMBERS || !params || !lms || !Ts || !box_lo || !box_hi || !prices || n_sets < 1 ||
            n_lm < 1 || n_T < 1 || !(floor > 0))
            return sfail(THOTH_GPU_E_INVALID, "bad lattice arguments");
        for (int j = 0; j < k; j++) {
            if (!members[j]) return sfail(THOTH_GPU_E_INVALID, "null member");
            if (members[j]->dev != members[0]->dev) return sfail(THOTH_GPU_E_INVALID, "members on different devices");
        }
        ThothSurrogate* s = members[0]; // its buffers and stream serve the call
        const int64_t n = (int64_t)n_sets * n_lm * n_T;
        if (n > ((int64_t)1 << 30)) return sfail(THOTH_GPU_E_TOO_LARGE, "more than 2^30 lattice cells");
        for (int q = 0; q < 7; q++)
            if (!(box_hi[q] > box_lo[q])) return sfail(THOTH_GPU_E_INVALID, "empty training box");
        std::lock_guard<std::mutex> lk(s_mu);
        STRY(cudaSetDevice(s->dev));
        // [inputs: sets, axes, Phi's table][feature words][per set and maturity][per log-moneyness]
        // [outputs][scales][prices]
        auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
        const size_t n_par = (size_t)n_sets * 5, n_in = n_par + n_lm + n_T + PHI_NODES * PHI_COEF;
        size_t off = 0;
        auto take = [&](size_t bytes) {
            const size_t o = off;
            off += up(bytes);
            return o;
        };
        const size_t o_in = take(sizeof(double) * n_in), o_w = take(sizeof(uint32_t) * (n_par + n_lm + n_T)),
                     o_st = take(sizeof(double2) * (size_t)n_sets * n_T), o_lm = take(sizeof(double2) * n_lm),
                     o_y = take(sizeof(float) * (size_t)n), o_sc = take(sizeof(double) * (size_t)n),
                     o_p = take(sizeof(float) * (size_t)n);
        int rc = ensure_infer(s, off);
        if (rc) return rc;
        std::vector<double> in(n_in);
        std::copy(params, params + n_par, in.begin());
        std::copy(lms, lms + n_lm, in.begin() + n_par);
        std::copy(Ts, Ts + n_T, in.begin() + n_par + n_lm);
        phi_coefficients(in.data() + n_par + n_lm + n_T);
        const double* d_in = reinterpret_cast<const double*>(s->ib + o_in);
        LatticeArgs B{};
        B.params = d_in;
        B.lms = d_in + n_par;
        B.Ts = d_in + n_par + n_lm;
        for (int q = 0; q < 7; q++) {
            B.lo[q] = box_lo[q];
            B.hi[q] = box_hi[q];
        }
        B.n_sets = n_sets;
        B.n_lm = n_lm;
        B.n_T = n_T;
        B.f_set = reinterpret_cast<uint32_t*>(s->ib + o_w);
        B.f_lm = B.f_set + n_par;
        B.f_T = B.f_lm + n_lm;
        B.set_T = reinterpret_cast<double2*>(s->ib + o_st);
        B.lm = reinterpret_cast<double2*>(s->ib + o_lm);
        mlp::InferArgs A{};
        A.L = mlp::LatticeTables{B.f_lm, B.f_T, B.f_set, B.set_T, B.lm, d_in + n_par + n_lm + n_T, floor * floor,
                                 (uint32_t)n_lm, (uint32_t)n_T};
        A.n = (int)n;
        A.members = k;
        A.y = reinterpret_cast<float*>(s->ib + o_y);
        A.scale = reinterpret_cast<double*>(s->ib + o_sc);
        A.price = reinterpret_cast<float*>(s->ib + o_p);
        A.status = s->status;
        for (int j = 0; j < k; j++) {
            A.params[j] = members[j]->params;
            A.wbf[j] = members[j]->wbf;
        }
        Timed T;
        STRY(T.create());
        STRY(cudaMemcpyAsync(s->ib + o_in, in.data(), sizeof(double) * n_in, cudaMemcpyHostToDevice, s->st));
        STRY(cudaMemsetAsync(s->status, 0, sizeof(int), s->st));
        STRY(cudaEventRecord(T.e0, s->st));
        STRY(lattice_tables(B, s->sms, s->st));
        A.scale_done = floor < TABLE_FLOOR;
        if (A.scale_done) STRY(lattice_scale(A, s->sms, s->st));
        STRY(mlp_infer(A, true, s->sms, s->st));
        STRY(cudaEventRecord(T.e1, s->st));
        return finish_infer(s, T, A.price, prices, n, device_ms);
    } catch (const std::bad_alloc&) {
        return sfail(THOTH_GPU_E_NOMEM, "out of host memory");
    } catch (const std::exception& e) {
        return sfail(THOTH_GPU_E_INVALID, std::string("host error: ") + e.what());
    }
}

const char* thoth_gpu_surrogate_last_error(void) { return s_err.c_str(); }

} // extern "C"
