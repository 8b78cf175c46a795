// mlp.cu -- host side of the surrogate ln g(E) network: a 4 x 256 SiLU MLP on
// the tcgen05 tensor cores (mlp_fused.cu), BF16 operands with FP32
// accumulation, trained with Adam on FP32 master weights.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "pticm.h"
#include "mlp_layout.h"
#include "pticm_engine.h"
#include "runtime_internal.h"

namespace pticm {
cudaError_t tc_gemm(const __nv_bfloat16* A, const __nv_bfloat16* B, int M, int N, int K, const float* bias, int act,
                    float* Cf, __nv_bfloat16* Cb, long long ldc, DevStatus* status, int* abort_flag,
                    cudaStream_t st);
}  // namespace pticm

using namespace pticm;

namespace {

int mlp_fail(int code, const std::string& m) {
    set_last_error(m);
    return code;
}

#define MLP_CK(x)                                                                                         \
    do {                                                                                                  \
        cudaError_t e_ = (x);                                                                             \
        if (e_ != cudaSuccess) return mlp_fail(PTICM_ERR_CUDA, std::string(#x) + ": " + cudaGetErrorString(e_)); \
    } while (0)

}  // namespace

extern "C" int pticm_tc_gemm_check(int M, int N, int K, const uint16_t* A, const uint16_t* B, const float* bias,
                                   int act, float* C, uint16_t* C_bf16) {
    if (M <= 0 || N <= 0 || K <= 0 || (K % 64) || !A || !B || !C)
        return mlp_fail(PTICM_ERR_INVALID, "need positive M, N and K a multiple of 64");
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0)
        return mlp_fail(PTICM_ERR_NODEVICE, "no CUDA device is available");
    __nv_bfloat16 *dA = nullptr, *dB = nullptr;
    float *dC = nullptr, *db = nullptr;
    __nv_bfloat16* dCb = nullptr;
    DevStatus* ds = nullptr;
    int* dab = nullptr;
    int rc = PTICM_OK;
    auto cleanup = [&]() {
        cudaFree(dA); cudaFree(dB); cudaFree(dC); cudaFree(dCb); cudaFree(db); cudaFree(ds); cudaFree(dab);
    };
    if (cudaMalloc(&dA, (size_t)M * K * 2) || cudaMalloc(&dB, (size_t)N * K * 2) ||
        cudaMalloc(&dC, (size_t)M * N * 4) || cudaMalloc(&ds, sizeof(DevStatus)) || cudaMalloc(&dab, 4) ||
        (bias && cudaMalloc(&db, (size_t)N * 4)) || (C_bf16 && cudaMalloc(&dCb, (size_t)M * N * 2))) {
        cleanup();
        return mlp_fail(PTICM_ERR_NOMEM, "device allocation failed");
    }
    cudaError_t e = cudaMemcpy(dA, A, (size_t)M * K * 2, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(dB, B, (size_t)N * K * 2, cudaMemcpyHostToDevice);
    if (e == cudaSuccess && bias) e = cudaMemcpy(db, bias, (size_t)N * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(ds, 0, sizeof(DevStatus));
    if (e == cudaSuccess) e = cudaMemset(dab, 0, 4);
    if (e == cudaSuccess) e = tc_gemm(dA, dB, M, N, K, db, act, dC, dCb, N, ds, dab, nullptr);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    DevStatus hs{};
    if (e == cudaSuccess) e = cudaMemcpy(&hs, ds, sizeof hs, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(C, dC, (size_t)M * N * 4, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && C_bf16) e = cudaMemcpy(C_bf16, dCb, (size_t)M * N * 2, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) rc = mlp_fail(PTICM_ERR_CUDA, std::string("tc_gemm: ") + cudaGetErrorString(e));
    else if (hs.error) rc = mlp_fail(PTICM_ERR_DEVICE, "tc_gemm: tensor-core wait expired");
    cleanup();
    return rc;
}

extern "C" int pticm_tc_gemm_bench(int M, int N, int K, int iters, double* ms_per_gemm, double* tflops) {
    if (M <= 0 || N <= 0 || K <= 0 || (K % 64) || iters <= 0 || !ms_per_gemm)
        return mlp_fail(PTICM_ERR_INVALID, "need positive M, N, iters and K a multiple of 64");
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0)
        return mlp_fail(PTICM_ERR_NODEVICE, "no CUDA device is available");
    __nv_bfloat16 *dA = nullptr, *dB = nullptr, *dC = nullptr;
    DevStatus* ds = nullptr;
    int* dab = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    auto cleanup = [&]() {
        cudaFree(dA); cudaFree(dB); cudaFree(dC); cudaFree(ds); cudaFree(dab);
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
    };
    if (cudaMalloc(&dA, (size_t)M * K * 2) || cudaMalloc(&dB, (size_t)N * K * 2) || cudaMalloc(&dC, (size_t)M * N * 2) ||
        cudaMalloc(&ds, sizeof(DevStatus)) || cudaMalloc(&dab, 4)) {
        cleanup();
        return mlp_fail(PTICM_ERR_NOMEM, "device allocation failed");
    }
    cudaError_t e = cudaMemset(dA, 0x3c, (size_t)M * K * 2);   // bf16 ~1.0 everywhere: finite sums
    if (e == cudaSuccess) e = cudaMemset(dB, 0x3c, (size_t)N * K * 2);
    if (e == cudaSuccess) e = cudaMemset(ds, 0, sizeof(DevStatus));
    if (e == cudaSuccess) e = cudaMemset(dab, 0, 4);
    if (e == cudaSuccess) e = cudaEventCreate(&e0);
    if (e == cudaSuccess) e = cudaEventCreate(&e1);
    if (e == cudaSuccess) e = tc_gemm(dA, dB, M, N, K, nullptr, 0, nullptr, dC, N, ds, dab, nullptr);   // warm-up
    if (e == cudaSuccess) e = cudaEventRecord(e0, nullptr);
    for (int i = 0; i < iters && e == cudaSuccess; i++)
        e = tc_gemm(dA, dB, M, N, K, nullptr, 0, nullptr, dC, N, ds, dab, nullptr);
    if (e == cudaSuccess) e = cudaEventRecord(e1, nullptr);
    if (e == cudaSuccess) e = cudaEventSynchronize(e1);
    float ms = 0.f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
    DevStatus hs{};
    if (e == cudaSuccess) e = cudaMemcpy(&hs, ds, sizeof hs, cudaMemcpyDeviceToHost);
    int rc = PTICM_OK;
    if (e != cudaSuccess) rc = mlp_fail(PTICM_ERR_CUDA, std::string("tc_gemm: ") + cudaGetErrorString(e));
    else if (hs.error) rc = mlp_fail(PTICM_ERR_DEVICE, "tc_gemm: tensor-core wait expired");
    else {
        *ms_per_gemm = (double)ms / iters;
        if (tflops) *tflops = 2.0 * M * N * (double)K / (*ms_per_gemm * 1e-3) / 1e12;
    }
    cleanup();
    return rc;
}

// ===================================================================== MLP
namespace {

// Rows of a prediction on the device at a time (128 MB with their results).
constexpr uint64_t kPredictRows = (uint64_t)4 << 20;

const size_t kWoff[MLP_LAYERS] = {kW1, kW2, kW3, kW4};
const int kKin[MLP_LAYERS] = {MLP_K0, MLP_H, MLP_H, MLP_H};

}  // namespace

struct pticm_mlp {
    int B = 0;                        // batch capacity (multiple of 128)
    MlpArgs a{};                      // parameters, images and training buffers
    float *dX = nullptr, *dY = nullptr;   // dataset on the device
    size_t cap_x = 0, cap_y = 0;      // and their capacities in rows
    float* y = nullptr;               // predictions, cap_p rows
    size_t cap_p = 0;
    long long* ctr = nullptr;         // device: [0] iteration of the current training call, [1] Adam steps taken
    std::vector<void*> allocs;
    ~pticm_mlp() {
        for (void* p : allocs) cudaFree(p);
        cudaFree(dX);
        cudaFree(dY);
        cudaFree(y);
    }
    template <typename T>
    cudaError_t alloc(T** p, size_t count) {
        void* q = nullptr;
        cudaError_t e = cudaMalloc(&q, count * sizeof(T));
        if (e != cudaSuccess) return e;
        allocs.push_back(q);
        *p = static_cast<T*>(q);
        return cudaMemset(q, 0, count * sizeof(T));
    }
};

namespace {

int mlp_check_status(pticm_mlp* m) {
    DevStatus hs{};
    MLP_CK(cudaMemcpy(&hs, m->a.status, sizeof hs, cudaMemcpyDeviceToHost));
    if (hs.error) return mlp_fail(PTICM_ERR_DEVICE, "surrogate network: tensor-core wait expired");
    return PTICM_OK;
}

// A buffer of at least `rows` elements of `per` floats each; kept between
// calls while the calls need at least a quarter of it.
int mlp_reserve(float** p, size_t* cap, size_t rows, size_t per) {
    if (*p && rows <= *cap && rows * 4 >= *cap) return PTICM_OK;
    cudaFree(*p);
    *p = nullptr;
    *cap = 0;
    MLP_CK(cudaMalloc(p, rows * per * sizeof(float)));
    *cap = rows;
    return PTICM_OK;
}

int mlp_upload_rows(pticm_mlp* m, const float* x, uint64_t n) {
    if (int rc = mlp_reserve(&m->dX, &m->cap_x, n, MLP_IN)) return rc;
    MLP_CK(cudaMemcpy(m->dX, x, n * MLP_IN * 4, cudaMemcpyHostToDevice));
    return PTICM_OK;
}

}  // namespace

extern "C" {

int pticm_mlp_create(uint64_t seed, uint32_t batch, pticm_mlp** out) {
    if (!out || batch == 0) return mlp_fail(PTICM_ERR_INVALID, "invalid arguments");
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0)
        return mlp_fail(PTICM_ERR_NODEVICE, "no CUDA device is available");
    auto m = new pticm_mlp();
    m->B = (int)((batch + 127) / 128 * 128);
    const size_t B = (size_t)m->B;
    MlpArgs& A = m->a;
    A.B = m->B;
    bool bad = false;
    bad |= m->alloc(&A.P, kParams) != cudaSuccess;
    bad |= m->alloc(&A.G, kParams) != cudaSuccess;
    bad |= m->alloc(&A.Mm, kParams) != cudaSuccess;
    bad |= m->alloc(&A.Vm, kParams) != cudaSuccess;
    for (int l = 0; l < MLP_LAYERS; l++) {
        bad |= m->alloc(&A.Wi[l], (size_t)MLP_H * kKin[l] * 2) != cudaSuccess;
        if (l > 0) bad |= m->alloc(&A.WTi[l], (size_t)MLP_H * kKin[l] * 2) != cudaSuccess;
        bad |= m->alloc(&A.Z[l], B * MLP_H / 4) != cudaSuccess;
        bad |= m->alloc(&A.dZf[l], B * MLP_H / 4) != cudaSuccess;
        bad |= m->alloc(&A.dZT[l], B * MLP_H * 2) != cudaSuccess;
        bad |= m->alloc(&A.HT[l], B * kKin[l] * 2) != cudaSuccess;   // (input columns past the features stay zero)
    }
    bad |= m->alloc(&A.H4, B * MLP_H / 8) != cudaSuccess;
    bad |= m->alloc(&A.dy, B) != cudaSuccess;
    bad |= m->alloc(&A.loss_tile, B / MLP_TILE) != cudaSuccess;
    bad |= m->alloc(&A.losses, 1) != cudaSuccess;
    bad |= m->alloc(&A.status, 1) != cudaSuccess;
    bad |= m->alloc(&A.abort_flag, 1) != cudaSuccess;
    bad |= m->alloc(&m->ctr, 2) != cudaSuccess;
    if (bad) {
        delete m;
        return mlp_fail(PTICM_ERR_NOMEM, "device allocation failed");
    }
    // He-style initialisation from a host generator; unused input columns 0
    std::vector<float> p(kParams, 0.0f);
    uint64_t s = seed * 0x9E3779B97F4A7C15ull + 0x1234567ull;
    auto gauss = [&]() {
        // Box-Muller on two splitmix64 draws
        auto next = [&]() {
            uint64_t z = (s += 0x9E3779B97F4A7C15ull);
            z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
            z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
            z ^= z >> 31;
            return ((z >> 11) + 0.5) * (1.0 / 9007199254740992.0);
        };
        const double u1 = next(), u2 = next();
        return (float)(std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2));
    };
    for (int l = 0; l < MLP_LAYERS; l++) {
        const int fan_in = l == 0 ? MLP_IN : MLP_H;
        const float sc = std::sqrt(2.0f / fan_in);
        for (int r = 0; r < MLP_H; r++)
            for (int c = 0; c < kKin[l]; c++)
                p[kWoff[l] + (size_t)r * kKin[l] + c] = (l == 0 && c >= MLP_IN) ? 0.0f : sc * gauss();
    }
    for (int j = 0; j < MLP_H; j++) p[kW5 + j] = std::sqrt(1.0f / MLP_H) * gauss();
    if (cudaMemcpy(A.P, p.data(), kParams * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
        mlp_images(A.P, A.Wi, A.WTi, nullptr) != cudaSuccess) {
        delete m;
        return mlp_fail(PTICM_ERR_CUDA, "parameter upload failed");
    }
    *out = m;
    return PTICM_OK;
}

void pticm_mlp_destroy(pticm_mlp* m) { delete m; }

uint64_t pticm_mlp_param_count(void) { return kParams; }

int pticm_mlp_get_params(pticm_mlp* m, float* out) {
    if (!m || !out) return mlp_fail(PTICM_ERR_INVALID, "null argument");
    MLP_CK(cudaMemcpy(out, m->a.P, kParams * 4, cudaMemcpyDeviceToHost));
    return PTICM_OK;
}

int pticm_mlp_set_params(pticm_mlp* m, const float* in) {
    if (!m || !in) return mlp_fail(PTICM_ERR_INVALID, "null argument");
    MLP_CK(cudaMemcpy(m->a.P, in, kParams * 4, cudaMemcpyHostToDevice));
    MLP_CK(mlp_images(m->a.P, m->a.Wi, m->a.WTi, nullptr));
    return PTICM_OK;
}

int pticm_mlp_set_data(pticm_mlp* m, const float* x, const float* y, uint64_t n) {
    if (!m || !x || !y || n == 0) return mlp_fail(PTICM_ERR_INVALID, "invalid arguments");
    if (int rc = mlp_upload_rows(m, x, n)) return rc;
    if (int rc = mlp_reserve(&m->dY, &m->cap_y, n, 1)) return rc;
    MLP_CK(cudaMemcpy(m->dY, y, n * 4, cudaMemcpyHostToDevice));
    return PTICM_OK;
}

int pticm_mlp_gradients(pticm_mlp* m, const float* x, const float* y, uint32_t n, float* grads, float* loss) {
    if (!m || !x || !y || n == 0 || (int)n > m->B) return mlp_fail(PTICM_ERR_INVALID, "invalid arguments");
    if (int rc = pticm_mlp_set_data(m, x, y, n)) return rc;
    MLP_CK(cudaMemset(m->a.status, 0, sizeof(DevStatus)));
    MLP_CK(cudaMemset(m->a.abort_flag, 0, sizeof(int)));
    MlpArgs A = m->a;
    A.X = m->dX;
    A.Y = m->dY;
    A.n_valid = (long long)n;
    MLP_CK(mlp_train_step(A, nullptr));
    MLP_CK(cudaDeviceSynchronize());
    if (int rc = mlp_check_status(m)) return rc;
    if (grads) MLP_CK(cudaMemcpy(grads, A.G, kParams * 4, cudaMemcpyDeviceToHost));
    if (loss) MLP_CK(cudaMemcpy(loss, A.losses, 4, cudaMemcpyDeviceToHost));
    return PTICM_OK;
}

int pticm_mlp_train(pticm_mlp* m, const float* x, const float* y, uint64_t n, uint32_t steps, float lr,
                    uint64_t seed, float* loss_per_step) {
    if (!m || !x || !y || n == 0 || n > 0xFFFFFFFFull) return mlp_fail(PTICM_ERR_INVALID, "invalid arguments");
    if (int rc = pticm_mlp_set_data(m, x, y, n)) return rc;
    if (steps == 0) return PTICM_OK;
    const int B = m->B;
    const int nb = (int)std::min<uint64_t>(n, (uint64_t)B);
    // Batches: an epoch-wise Fisher-Yates shuffle on the host (xorshift64),
    // written a chunk of kChunk steps at a time into one half of a pinned
    // two-chunk ring; the device ring (the same layout) is read by the
    // captured step at row (iteration mod 2 kChunk).  The host fills chunk
    // c + 2 while chunk c + 1 runs.
    constexpr uint32_t kChunk = 256;
    const size_t half = (size_t)kChunk * nb;
    std::vector<uint32_t> order(n);
    for (uint64_t i = 0; i < n; i++) order[i] = (uint32_t)i;
    uint64_t s = seed ^ 0xA0761D6478BD642Full;
    auto nxt = [&]() {
        s ^= s << 13; s ^= s >> 7; s ^= s << 17;
        return s;
    };
    uint64_t cursor = n;
    auto fill = [&](uint32_t* dst, uint32_t count) {
        for (size_t k = 0; k < (size_t)count * nb; k++) {
            if (cursor == n) {   // reshuffle each epoch
                for (uint64_t i = n - 1; i > 0; i--) std::swap(order[i], order[nxt() % (i + 1)]);
                cursor = 0;
            }
            dst[k] = order[cursor++];
        }
    };

    struct Res {
        cudaStream_t st = nullptr;
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
        uint32_t* ring = nullptr;    // device, 2 kChunk batches
        uint32_t* hring = nullptr;   // pinned host
        float* losses = nullptr;     // device, one per step
        cudaEvent_t copied[2] = {nullptr, nullptr};
        cudaEvent_t ready = nullptr;
        ~Res() {
            if (st) cudaStreamSynchronize(st);
            if (exec) cudaGraphExecDestroy(exec);
            if (graph) cudaGraphDestroy(graph);
            for (cudaEvent_t e : copied)
                if (e) cudaEventDestroy(e);
            if (ready) cudaEventDestroy(ready);
            if (st) cudaStreamDestroy(st);
            cudaFree(ring);
            cudaFree(losses);
            cudaFreeHost(hring);
        }
    } r;
    MLP_CK(cudaStreamCreateWithFlags(&r.st, cudaStreamNonBlocking));
    MLP_CK(cudaMalloc(&r.ring, 2 * half * 4));
    MLP_CK(cudaMalloc(&r.losses, (size_t)steps * 4));
    MLP_CK(cudaMallocHost(&r.hring, 2 * half * 4));
    for (cudaEvent_t& e : r.copied) MLP_CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    MLP_CK(cudaEventCreateWithFlags(&r.ready, cudaEventDisableTiming));
    // the dataset's copies and the weights' images were issued on the default
    // stream, which r.st does not wait for by itself
    MLP_CK(cudaEventRecord(r.ready, nullptr));
    MLP_CK(cudaStreamWaitEvent(r.st, r.ready, 0));
    MLP_CK(cudaMemsetAsync(m->a.status, 0, sizeof(DevStatus), r.st));
    MLP_CK(cudaMemsetAsync(m->a.abort_flag, 0, sizeof(int), r.st));
    MLP_CK(cudaMemsetAsync(m->ctr, 0, sizeof(long long), r.st));   // this call's iteration counter

    // one training step, captured once: the chain kernel (gather, forward,
    // loss, backward) and the gradient kernel (gradients, Adam, images,
    // counters)
    MlpArgs A = m->a;
    A.X = m->dX;
    A.Y = m->dY;
    A.idx = r.ring;
    A.ctr = m->ctr;
    A.ring = 2 * (int)kChunk;
    A.n_valid = nb;
    A.losses = r.losses;
    A.lr = lr;
    MLP_CK(cudaStreamBeginCapture(r.st, cudaStreamCaptureModeRelaxed));
    const cudaError_t es = mlp_train_step(A, r.st);
    const cudaError_t ec = cudaStreamEndCapture(r.st, &r.graph);
    MLP_CK(es);
    MLP_CK(ec);
    MLP_CK(cudaGraphInstantiate(&r.exec, r.graph, 0));

    for (uint32_t c0 = 0, chunk = 0; c0 < steps; c0 += kChunk, chunk++) {
        const uint32_t cnt = std::min(kChunk, steps - c0);
        const int h = (int)(chunk & 1);
        // the pinned half is free once its previous upload (two chunks ago) ran
        MLP_CK(cudaEventSynchronize(r.copied[h]));
        fill(r.hring + h * half, cnt);
        MLP_CK(cudaMemcpyAsync(r.ring + h * half, r.hring + h * half, (size_t)cnt * nb * 4, cudaMemcpyHostToDevice,
                               r.st));
        MLP_CK(cudaEventRecord(r.copied[h], r.st));
        for (uint32_t i = 0; i < cnt; i++) MLP_CK(cudaGraphLaunch(r.exec, r.st));
    }
    if (loss_per_step)
        MLP_CK(cudaMemcpyAsync(loss_per_step, r.losses, (size_t)steps * 4, cudaMemcpyDeviceToHost, r.st));
    MLP_CK(cudaStreamSynchronize(r.st));
    return mlp_check_status(m);
}

int pticm_mlp_predict(pticm_mlp* m, const float* x, uint64_t n, float* y) {
    if (!m || !x || !y) return mlp_fail(PTICM_ERR_INVALID, "null argument");
    if (n == 0) return PTICM_OK;
    for (uint64_t r0 = 0; r0 < n; r0 += kPredictRows) {
        const uint64_t rows = std::min(n - r0, kPredictRows);
        if (int rc = mlp_upload_rows(m, x + r0 * MLP_IN, rows)) return rc;
        if (int rc = mlp_reserve(&m->y, &m->cap_p, rows, 1)) return rc;
        if (r0 == 0) {   // (behind the copy, which would wait for them)
            MLP_CK(cudaMemsetAsync(m->a.status, 0, sizeof(DevStatus), nullptr));
            MLP_CK(cudaMemsetAsync(m->a.abort_flag, 0, sizeof(int), nullptr));
        }
        MlpArgs A = m->a;
        A.X = m->dX;
        A.y = m->y;
        A.n_valid = (long long)rows;
        MLP_CK(mlp_predict_rows(A, nullptr));
        MLP_CK(cudaMemcpy(y + r0, m->y, rows * 4, cudaMemcpyDeviceToHost));
    }
    return mlp_check_status(m);
}

int pticm_mlp_division_probe(const float* a, const float* b, float* q, int count) {
    if (!a || !b || !q || count <= 0) return mlp_fail(PTICM_ERR_INVALID, "invalid arguments");
    int devices = 0;
    if (cudaGetDeviceCount(&devices) != cudaSuccess || devices == 0)
        return mlp_fail(PTICM_ERR_NODEVICE, "no CUDA device is available");
    DArr<float> da, db, dq;
    MLP_CK(da.reserve((size_t)count));
    MLP_CK(db.reserve((size_t)count));
    MLP_CK(dq.reserve((size_t)count));
    MLP_CK(cudaMemcpy(da.p, a, (size_t)count * 4, cudaMemcpyHostToDevice));
    MLP_CK(cudaMemcpy(db.p, b, (size_t)count * 4, cudaMemcpyHostToDevice));
    MLP_CK(mlp_div(da.p, db.p, dq.p, count, nullptr));
    MLP_CK(cudaMemcpy(q, dq.p, (size_t)count * 4, cudaMemcpyDeviceToHost));
    return PTICM_OK;
}

}  // extern "C"
