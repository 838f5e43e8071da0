// surrogate.cu -- the calibration surrogate: a 4-256-256-256-3 GELU
// multilayer perceptron with BF16 weights and activations and FP32
// accumulation, trained with Adam, every GEMM on tcgen05 tensor cores
// (surrogate_gemm.cuh). C ABI in include/dem_surrogate.h.
//
// The reference has no such component: its calibration loop
// (Drivers/Calibration/py/smc.py:168-350) proposes parameters by sequential
// Monte Carlo over plain DEM runs; this network learns the map from contact
// parameters to bulk responses from batched DEM runs and proposes candidates
// for them, with DEM kept as the judge of its error.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/dem_surrogate.h"
#include "surrogate_gemm.cuh"
#include "surrogate_fused.cuh"

using namespace surrogate;

namespace {

constexpr int NI = DEM_MLP_INPUTS, NH = DEM_MLP_HIDDEN, NO = DEM_MLP_OUTPUTS;

// offsets of the flat FP32 parameter vector (include/dem_surrogate.h)
constexpr long long OFF_W1 = 0, OFF_B1 = OFF_W1 + (long long)NH * NI;
constexpr long long OFF_W2 = OFF_B1 + NH, OFF_B2 = OFF_W2 + (long long)NH * NH;
constexpr long long OFF_W3 = OFF_B2 + NH, OFF_B3 = OFF_W3 + (long long)NH * NH;
constexpr long long OFF_W4 = OFF_B3 + NH, OFF_B4 = OFF_W4 + (long long)NO * NH;
constexpr long long NPARAM = OFF_B4 + NO;
static_assert(NPARAM == DEM_MLP_NPARAMS, "parameter layout");

struct Mlp {
    int device = 0;
    int capacity = 0;
    cudaStream_t stream = nullptr;
    std::string err;
    char* block = nullptr;                                          // holds every array below
    unsigned* d_error = nullptr;
    float *p = nullptr, *g = nullptr, *m = nullptr, *v = nullptr; // params, grads, Adam moments (FP32)
    __nv_bfloat16* wb = nullptr;                                    // BF16 copy of the whole vector
    long long step = 0;
    float norm[2 * NI + 2 * NO];                                    // in_mean, in_std, out_mean, out_std
    float* d_norm = nullptr;
    // activations for `capacity` rows
    float *x = nullptr, *t = nullptr;        // raw inputs, raw targets (FP32)
    __nv_bfloat16* xb = nullptr;             // normalised inputs
    float *z1 = nullptr, *z2 = nullptr, *z3 = nullptr, *y = nullptr;
    __nv_bfloat16 *h1 = nullptr, *h2 = nullptr, *h3 = nullptr;
    __nv_bfloat16 *dyb = nullptr, *dz1 = nullptr, *dz2 = nullptr, *dz3 = nullptr;
    float *loss = nullptr, *loss_part = nullptr;
    float* partial = nullptr;                                       // weight-gradient slices, MAX_SLICES parameter vectors
};

int fail(Mlp* h, int code, const std::string& msg)
{
    if (h) h->err = msg;
    return code;
}

#define CK(call)                                                                                      \
    do {                                                                                              \
        cudaError_t e_ = (call);                                                                      \
        if (e_ != cudaSuccess) return fail(h, DEM_MLP_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

unsigned grid1(long long n, int b) { return (unsigned)std::max<long long>(1, (n + b - 1) / b); }

} // namespace

// ---------------------------------------------------------------------------
// element-wise and reduction kernels
// ---------------------------------------------------------------------------
namespace {

// x (raw, [n][4]) -> (x - mean) / std in BF16
__global__ void k_norm_inputs(const float* x, const float* norm, int n, __nv_bfloat16* xb)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n * NI) return;
    const int c = i % NI;
    xb[i] = __float2bfloat16_rn((x[i] - norm[c]) / norm[NI + c]);
}

// y (normalised, [n][3]) -> raw units
__global__ void k_denorm_outputs(const float* y, const float* norm, int n, float* out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n * NO) return;
    const int c = i % NO;
    out[i] = y[i] * norm[2 * NI + NO + c] + norm[2 * NI + c];
}

// dy = 2 (y - t') / (3 n) in BF16 with t' the normalised target, and each
// block's part of the sum of (y - t')^2, its elements in a fixed order
// (k_reduce_params adds the parts).
constexpr int LOSS_BLOCK = 256;
__global__ void __launch_bounds__(LOSS_BLOCK) k_loss(const float* y, const float* t, const float* norm, int n,
                                                     __nv_bfloat16* dyb, float* part)
{
    __shared__ float sh[LOSS_BLOCK];
    float acc = 0.f;
    const float scale = 2.0f / (3.0f * (float)n);
    for (int i = blockIdx.x * LOSS_BLOCK + threadIdx.x; i < n * NO; i += gridDim.x * LOSS_BLOCK) {
        const int c = i % NO;
        const float tn = (t[i] - norm[2 * NI + c]) / norm[2 * NI + NO + c];
        const float d = y[i] - tn;
        acc += d * d;
        dyb[i] = __float2bfloat16_rn(scale * d);
    }
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int s = LOSS_BLOCK / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

__global__ void k_to_bf16(const float* p, long long n, __nv_bfloat16* out)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = __float2bfloat16_rn(p[i]);
}

// The gradient of parameter i from the slices' partial sums in slice order, the
// loss from the blocks' parts, and (step) Adam (Kingma and Ba 2015) with bias
// correction, which refreshes the BF16 copy. Where a wait of this pass ran out
// (*error), a slice's sums are not of this batch: nothing changes.
__global__ void __launch_bounds__(256) k_reduce_params(const float* partial, int slices, long long stride, const float* loss_part,
                                                       int loss_blocks, float loss_scale, float* loss, float* g, bool step,
                                                       float* p, float* m, float* v, float lr, float bc1, float bc2,
                                                       __nv_bfloat16* wb, const unsigned* error)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (*error) return;
    if (i == 0) {
        float s = 0.f;
        for (int b = 0; b < loss_blocks; ++b) s += loss_part[b];
        *loss = s / loss_scale;
    }
    if (i >= NPARAM) return;
    float gi = 0.f;
#pragma unroll 8
    for (int s = 0; s < slices; ++s) gi += partial[(long long)s * stride + i];
    g[i] = gi;
    if (!step) return;
    const float mi = 0.9f * m[i] + 0.1f * gi;
    const float vi = 0.999f * v[i] + 0.001f * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float pi = p[i] - lr * (mi / bc1) / (sqrtf(vi / bc2) + 1e-8f);
    p[i] = pi;
    wb[i] = __float2bfloat16_rn(pi);
}

template <int BN>
int launch_layer(Mlp* h, GemmArgs a)
{
    static bool configured[64] = {false};
    if (!configured[h->device & 63]) {
        CK(cudaFuncSetAttribute(k_layer<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, LayerSmem<BN>::bytes(LAYER_MAX_K)));
        configured[h->device & 63] = true;
    }
    a.error = h->d_error;
    const dim3 grid(grid1(a.M, GEMM_BM), grid1(a.N, BN));
    k_layer<BN><<<grid, GEMM_THREADS, LayerSmem<BN>::bytes(a.K), h->stream>>>(a);
    CK(cudaGetLastError());
    return DEM_MLP_OK;
}

// C = A . B^T with the operand strides of GemmArgs, K <= 256; N <= 16 uses 16-wide tiles
int gemm(Mlp* h, const __nv_bfloat16* A, long long a_sm, long long a_sk, const __nv_bfloat16* B, long long b_sn,
         long long b_sk, int M, int N, int K, int epi, const float* bias, const float* aux, float* out_f32,
         __nv_bfloat16* out_bf16, int ldc)
{
    GemmArgs a{A, B, a_sm, a_sk, b_sn, b_sk, M, N, K, epi, bias, aux, out_f32, out_bf16, ldc, nullptr};
    if (N <= 16) return launch_layer<16>(h, a);
    return launch_layer<LAYER_BN>(h, a);
}

// Slices of the batch in the weight gradients: 64 samples each up to
// MAX_SLICES of them (a batch of 1,024), longer ones beyond.
constexpr int MAX_SLICES = 16;
int slice_length(int n)
{
    const int chunks = (n + GEMM_BK - 1) / GEMM_BK;
    return GEMM_BK * ((chunks + MAX_SLICES - 1) / MAX_SLICES);
}
constexpr int MAX_LOSS_BLOCKS = 64;
constexpr long long PARAM_STRIDE = (NPARAM + 3) / 4 * 4; // of a slice: 16-byte rows

} // namespace

// ---------------------------------------------------------------------------
// forward and backward passes (n rows already in h->x, h->t)
// ---------------------------------------------------------------------------
namespace {

// Inference: the whole pass in one kernel (surrogate_fused.cuh), one CTA per
// SM over 128-sample tiles; the activations stay on the SM.
int forward_fused(Mlp* h, int n)
{
    static bool configured[64] = {false};
    static int sms[64] = {0};
    if (!configured[h->device & 63]) {
        CK(cudaFuncSetAttribute(k_mlp_forward_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, FUSED_SMEM));
        CK(cudaDeviceGetAttribute(&sms[h->device & 63], cudaDevAttrMultiProcessorCount, h->device));
        configured[h->device & 63] = true;
    }
    const int tiles = (n + FUSED_TILE - 1) / FUSED_TILE;
    FusedArgs a{h->x, h->d_norm, h->wb, h->p, OFF_W1, OFF_B1, OFF_W2, OFF_B2, OFF_W3, OFF_B3, OFF_W4, OFF_B4,
                n, h->y, h->d_error};
    k_mlp_forward_fused<<<std::min(tiles, sms[h->device & 63]), FUSED_THREADS, FUSED_SMEM, h->stream>>>(a);
    CK(cudaGetLastError());
    return DEM_MLP_OK;
}

// the training pass: one product per layer, the pre-activations kept
int forward(Mlp* h, int n)
{
    int rc;
    const __nv_bfloat16* W = h->wb;
    const float* P = h->p;
    k_norm_inputs<<<grid1((long long)n * NI, 256), 256, 0, h->stream>>>(h->x, h->d_norm, n, h->xb);
    // z1 = x W1^T + b1, h1 = gelu(z1), ... (A rows = samples, B rows = output features)
    if ((rc = gemm(h, h->xb, NI, 1, W + OFF_W1, NI, 1, n, NH, NI, EPI_BIAS_GELU, P + OFF_B1, nullptr, h->z1, h->h1, NH)))
        return rc;
    if ((rc = gemm(h, h->h1, NH, 1, W + OFF_W2, NH, 1, n, NH, NH, EPI_BIAS_GELU, P + OFF_B2, nullptr, h->z2, h->h2, NH)))
        return rc;
    if ((rc = gemm(h, h->h2, NH, 1, W + OFF_W3, NH, 1, n, NH, NH, EPI_BIAS_GELU, P + OFF_B3, nullptr, h->z3, h->h3, NH)))
        return rc;
    return gemm(h, h->h3, NH, 1, W + OFF_W4, NH, 1, n, NO, NH, EPI_BIAS_F32, P + OFF_B4, nullptr, h->y, nullptr, NO);
}

// Gradient of the mean squared error into h->g, loss into h->loss; lr > 0: and
// the Adam step (bias corrections bc1, bc2).
int backward(Mlp* h, int n, float lr = 0.f, float bc1 = 1.f, float bc2 = 1.f)
{
    int rc;
    const __nv_bfloat16* W = h->wb;
    const int loss_blocks = std::min(MAX_LOSS_BLOCKS, (int)grid1((long long)n * NO, LOSS_BLOCK));
    k_loss<<<loss_blocks, LOSS_BLOCK, 0, h->stream>>>(h->y, h->t, h->d_norm, n, h->dyb, h->loss_part);
    // dz3 = (dy W4) gelu'(z3), dz2 = (dz3 W3) gelu'(z2), dz1 = (dz2 W2) gelu'(z1)
    // (the input gradient is not needed)
    if ((rc = gemm(h, h->dyb, NO, 1, W + OFF_W4, 1, NH, n, NH, NO, EPI_DGELU_BF16, nullptr, h->z3, nullptr, h->dz3, NH)))
        return rc;
    if ((rc = gemm(h, h->dz3, NH, 1, W + OFF_W3, 1, NH, n, NH, NH, EPI_DGELU_BF16, nullptr, h->z2, nullptr, h->dz2, NH)))
        return rc;
    if ((rc = gemm(h, h->dz2, NH, 1, W + OFF_W2, 1, NH, n, NH, NH, EPI_DGELU_BF16, nullptr, h->z1, nullptr, h->dz1, NH)))
        return rc;
    // every layer's dW = dz^T x and db = colsum(dz)
    static bool configured[64] = {false};
    const int smem = 2 * (LayerSmem<64>::A_BYTES + LayerSmem<64>::B_BYTES) + 1024;
    if (!configured[h->device & 63]) {
        CK(cudaFuncSetAttribute(k_weight_grads, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        configured[h->device & 63] = true;
    }
    WeightGradArgs a{};
    int tiles = 0;
    auto add = [&](int k, const __nv_bfloat16* dz, const __nv_bfloat16* x, int outs, int ins, long long ow, long long ob) {
        a.layer[k] = WeightGrad{dz, x, outs, ins, ow, ob, tiles, (outs + GEMM_BM - 1) / GEMM_BM};
        tiles += a.layer[k].m_tiles * ((ins + 63) / 64);
    };
    add(0, h->dz3, h->h2, NH, NH, OFF_W3, OFF_B3);
    add(1, h->dz2, h->h1, NH, NH, OFF_W2, OFF_B2);
    add(2, h->dz1, h->xb, NH, NI, OFF_W1, OFF_B1);
    add(3, h->dyb, h->h3, NO, NH, OFF_W4, OFF_B4);
    a.batch = n;
    a.slice = slice_length(n);
    a.partial = h->partial;
    a.n_params = PARAM_STRIDE;
    a.error = h->d_error;
    const int slices = (n + a.slice - 1) / a.slice;
    k_weight_grads<<<dim3(tiles, slices), GEMM_THREADS, smem, h->stream>>>(a);
    k_reduce_params<<<grid1(NPARAM, 256), 256, 0, h->stream>>>(h->partial, slices, PARAM_STRIDE, h->loss_part, loss_blocks,
                                                               3.0f * (float)n, h->loss, h->g, lr > 0.f, h->p, h->m, h->v,
                                                               lr, bc1, bc2, h->wb, h->d_error);
    CK(cudaGetLastError());
    return DEM_MLP_OK;
}

int check_device_status(Mlp* h)
{
    unsigned e = 0;
    CK(cudaMemcpyAsync(&e, h->d_error, sizeof(e), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    if (e) {
        CK(cudaMemsetAsync(h->d_error, 0, sizeof(unsigned), h->stream));
        return fail(h, DEM_MLP_ERR_TIMEOUT, "a tensor-core wait ran out");
    }
    return DEM_MLP_OK;
}

int load_batch(Mlp* h, const float* x, const float* t, int n)
{
    if (n <= 0 || n > h->capacity || !x) return fail(h, DEM_MLP_ERR_BAD_INPUT, "batch size out of range");
    CK(cudaSetDevice(h->device));
    CK(cudaMemcpyAsync(h->x, x, (size_t)n * NI * sizeof(float), cudaMemcpyHostToDevice, h->stream));
    if (t) CK(cudaMemcpyAsync(h->t, t, (size_t)n * NO * sizeof(float), cudaMemcpyHostToDevice, h->stream));
    return DEM_MLP_OK;
}

} // namespace

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
struct dem_mlp : Mlp {};

extern "C" {

int dem_mlp_create(int device, int capacity, uint64_t seed, dem_mlp** out)
{
    if (!out || capacity <= 0 || capacity > (1 << 24)) return DEM_MLP_ERR_BAD_INPUT;
    *out = nullptr;
    dem_mlp* h = new dem_mlp();
    h->device = device;
    h->capacity = capacity;
    auto cleanup = [&](int rc) {
        if (rc) dem_mlp_destroy(h);
        return rc;
    };
    if (cudaSetDevice(device) != cudaSuccess) return cleanup(DEM_MLP_ERR_CUDA);
    if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess) return cleanup(DEM_MLP_ERR_CUDA);
    const size_t c = (size_t)capacity;
    // one device block for every array (24 allocations took most of the set-up)
    size_t total = 0;
    char* block = nullptr;
    auto part = [&](auto** p, size_t count) {
        if (block) *p = reinterpret_cast<std::remove_reference_t<decltype(*p)>>(block + total);
        total += (std::max<size_t>(count, 1) * sizeof(**p) + 255) & ~(size_t)255;
    };
    for (int pass = 0; pass < 2; ++pass) {
        if (pass == 1) {
            if (cudaMalloc(reinterpret_cast<void**>(&block), total) != cudaSuccess)
                return cleanup(fail(h, DEM_MLP_ERR_CUDA, "cudaMalloc failed"));
            h->block = block;
            total = 0;
        }
        part(&h->d_error, 1);
        part(&h->p, NPARAM); part(&h->g, NPARAM); part(&h->m, NPARAM); part(&h->v, NPARAM);
        part(&h->wb, NPARAM);
        part(&h->d_norm, 2 * NI + 2 * NO);
        part(&h->x, c * NI); part(&h->t, c * NO); part(&h->xb, c * NI);
        part(&h->z1, c * NH); part(&h->z2, c * NH); part(&h->z3, c * NH); part(&h->y, c * NO);
        part(&h->h1, c * NH); part(&h->h2, c * NH); part(&h->h3, c * NH);
        part(&h->dyb, c * NO); part(&h->dz1, c * NH); part(&h->dz2, c * NH); part(&h->dz3, c * NH);
        part(&h->loss, 1);
        part(&h->loss_part, MAX_LOSS_BLOCKS);
        part(&h->partial, (size_t)std::min<long long>(MAX_SLICES, grid1(capacity, GEMM_BK)) * PARAM_STRIDE);
    }
    // He-uniform weights, zero biases
    std::vector<float> p(NPARAM, 0.0f);
    std::mt19937_64 rng(seed);
    auto fill = [&](long long off, int rows, int cols) {
        const float a = std::sqrt(6.0f / (float)cols);
        std::uniform_real_distribution<float> u(-a, a);
        for (long long i = 0; i < (long long)rows * cols; ++i) p[off + i] = u(rng);
    };
    fill(OFF_W1, NH, NI);
    fill(OFF_W2, NH, NH);
    fill(OFF_W3, NH, NH);
    fill(OFF_W4, NO, NH);
    for (int k = 0; k < NI; ++k) { h->norm[k] = 0.f; h->norm[NI + k] = 1.f; }
    for (int k = 0; k < NO; ++k) { h->norm[2 * NI + k] = 0.f; h->norm[2 * NI + NO + k] = 1.f; }
    int rc = dem_mlp_set_params(h, p.data());
    if (rc) return cleanup(rc);
    if (cudaMemcpyAsync(h->d_norm, h->norm, sizeof(h->norm), cudaMemcpyHostToDevice, h->stream) != cudaSuccess ||
        cudaMemsetAsync(h->d_error, 0, sizeof(unsigned), h->stream) != cudaSuccess ||
        cudaStreamSynchronize(h->stream) != cudaSuccess)
        return cleanup(DEM_MLP_ERR_CUDA);
    *out = h;
    return DEM_MLP_OK;
}

int dem_mlp_set_normalisation(dem_mlp* h, const float* in_mean, const float* in_std, const float* out_mean,
                              const float* out_std)
{
    if (!h || !in_mean || !in_std || !out_mean || !out_std) return DEM_MLP_ERR_BAD_INPUT;
    for (int k = 0; k < NI; ++k) {
        if (!(in_std[k] > 0.f)) return fail(h, DEM_MLP_ERR_BAD_INPUT, "input std must be positive");
        h->norm[k] = in_mean[k];
        h->norm[NI + k] = in_std[k];
    }
    for (int k = 0; k < NO; ++k) {
        if (!(out_std[k] > 0.f)) return fail(h, DEM_MLP_ERR_BAD_INPUT, "output std must be positive");
        h->norm[2 * NI + k] = out_mean[k];
        h->norm[2 * NI + NO + k] = out_std[k];
    }
    CK(cudaSetDevice(h->device));
    CK(cudaMemcpyAsync(h->d_norm, h->norm, sizeof(h->norm), cudaMemcpyHostToDevice, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return DEM_MLP_OK;
}

int dem_mlp_get_params(dem_mlp* h, float* params)
{
    if (!h || !params) return DEM_MLP_ERR_BAD_INPUT;
    CK(cudaSetDevice(h->device));
    CK(cudaMemcpyAsync(params, h->p, NPARAM * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return DEM_MLP_OK;
}

int dem_mlp_set_params(dem_mlp* h, const float* params)
{
    if (!h || !params) return DEM_MLP_ERR_BAD_INPUT;
    CK(cudaSetDevice(h->device));
    CK(cudaMemcpyAsync(h->p, params, NPARAM * sizeof(float), cudaMemcpyHostToDevice, h->stream));
    CK(cudaMemsetAsync(h->m, 0, NPARAM * sizeof(float), h->stream));
    CK(cudaMemsetAsync(h->v, 0, NPARAM * sizeof(float), h->stream));
    k_to_bf16<<<grid1(NPARAM, 256), 256, 0, h->stream>>>(h->p, NPARAM, h->wb);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(h->stream));
    h->step = 0;
    return DEM_MLP_OK;
}

int dem_mlp_forward(dem_mlp* h, const float* x, int n, float* y)
{
    if (!h || !y) return DEM_MLP_ERR_BAD_INPUT;
    int rc;
    if ((rc = load_batch(h, x, nullptr, n)) || (rc = forward_fused(h, n))) return rc;
    k_denorm_outputs<<<grid1((long long)n * NO, 256), 256, 0, h->stream>>>(h->y, h->d_norm, n, h->t);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(y, h->t, (size_t)n * NO * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    return check_device_status(h);
}

int dem_mlp_gradients(dem_mlp* h, const float* x, const float* t, int n, float* loss, float* grads)
{
    if (!h || !t || !loss || !grads) return DEM_MLP_ERR_BAD_INPUT;
    int rc;
    if ((rc = load_batch(h, x, t, n)) || (rc = forward(h, n)) || (rc = backward(h, n))) return rc;
    CK(cudaMemcpyAsync(loss, h->loss, sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaMemcpyAsync(grads, h->g, NPARAM * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    return check_device_status(h);
}

int dem_mlp_train_step(dem_mlp* h, const float* x, const float* t, int n, float lr, float* loss)
{
    if (!h || !t || !(lr > 0.f)) return DEM_MLP_ERR_BAD_INPUT;
    int rc;
    const float bc1 = 1.0f - std::pow(0.9f, (float)(h->step + 1));
    const float bc2 = 1.0f - std::pow(0.999f, (float)(h->step + 1));
    if ((rc = load_batch(h, x, t, n)) || (rc = forward(h, n)) || (rc = backward(h, n, lr, bc1, bc2))) return rc;
    if (loss) CK(cudaMemcpyAsync(loss, h->loss, sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    if ((rc = check_device_status(h))) return rc;
    h->step += 1;
    return DEM_MLP_OK;
}

int dem_mlp_time_forward(dem_mlp* h, int n, int reps, float* ms)
{
    if (!h || !ms || n <= 0 || n > h->capacity || reps <= 0) return DEM_MLP_ERR_BAD_INPUT;
    CK(cudaSetDevice(h->device));
    cudaEvent_t e0, e1;
    CK(cudaEventCreate(&e0));
    CK(cudaEventCreate(&e1));
    int rc = forward_fused(h, n); // warm-up
    CK(cudaEventRecord(e0, h->stream));
    for (int r = 0; r < reps && !rc; ++r) rc = forward_fused(h, n);
    CK(cudaEventRecord(e1, h->stream));
    CK(cudaEventSynchronize(e1));
    float t = 0.f;
    CK(cudaEventElapsedTime(&t, e0, e1));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) return rc;
    *ms = t / reps;
    return check_device_status(h);
}

int dem_mlp_selftest_expire(dem_mlp* h)
{
    if (!h) return DEM_MLP_ERR_BAD_INPUT;
    CK(cudaSetDevice(h->device));
    CK(cudaMemsetAsync(h->d_error, 1, sizeof(unsigned), h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return DEM_MLP_OK;
}

const char* dem_mlp_last_error(dem_mlp* h) { return h ? h->err.c_str() : "null handle"; }

void dem_mlp_destroy(dem_mlp* h)
{
    if (!h) return;
    cudaSetDevice(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    if (h->block) cudaFree(h->block);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
}

} // extern "C"
