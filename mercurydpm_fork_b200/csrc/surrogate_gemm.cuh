// surrogate_gemm.cuh -- BF16 x BF16 -> FP32 GEMM on the 5th-generation tensor
// cores (tcgen05.mma, accumulator in tensor memory) for the calibration
// surrogate's multilayer perceptron.
//
//   C[m, n] = sum_k A(m, k) B(n, k)      A(m, k) = A[m * a_sm + k * a_sk]
//                                        B(n, k) = B[n * b_sn + k * b_sk]
//
// k_layer (forward and input-gradient products, K <= 256): one CTA of 256
// threads computes a 128 x BN tile. All of K is staged at once, 64 at a time
// into shared memory of its own in the K-major canonical layout without swizzle
// (8 x 16-byte core matrices; LBO = 128 B between the two K halves of an
// instruction, SBO = 1024 B between 8-row groups); one thread issues the K=16
// tcgen05.mma of a chunk as it lands; the accumulator lives in tensor memory
// (128 lanes x BN columns of FP32) and the eight warps read it back with
// tcgen05.ld (each lane quarter by two warps) for the fused epilogue.
// k_weight_grads (all weight and bias gradients of a pass, one launch): the
// batch is the contraction, split over blockIdx.y into slices whose FP32
// partial sums k_reduce_params adds in slice order.
// Row-contiguous operands are staged with cp.async, column-contiguous ones
// (the transposed products of the backward pass) through 8 x 8 transposes in
// registers, others element by element.
//
// Every wait is bounded: a wait that runs out sets an error word and the
// kernel finishes without using the missing result; tensor memory is
// always released.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>

namespace surrogate {

constexpr int GEMM_BM = 128;
constexpr int GEMM_BK = 64;
constexpr int GEMM_THREADS = 256; // 8 warps: warps w and w + 4 share TMEM lanes 32 (w % 4) ..
constexpr int LAYER_MAX_K = 256;
constexpr int LAYER_BN = 32;      // output columns of a tile: a batch of 1,024 gives 64 CTAs a layer
constexpr unsigned long long WAIT_LIMIT = 1ull << 26; // try_wait polls before giving up

enum Epilogue : int {
    EPI_BIAS_GELU = 1,    // z = acc + bias[n]; out_f32 = z; out_bf16 = gelu(z)
    EPI_BIAS_F32 = 2,     // out_f32 = acc + bias[n]
    EPI_DGELU_BF16 = 3,   // out_bf16 = acc * gelu'(z[m, n]) with z = aux_f32
};

struct GemmArgs {
    const __nv_bfloat16* A;
    const __nv_bfloat16* B;
    long long a_sm, a_sk, b_sn, b_sk;
    int M, N, K;
    int epilogue;
    const float* bias;       // EPI_BIAS_*
    const float* aux_f32;    // EPI_DGELU_BF16: pre-activations z, ld = ldc
    float* out_f32;
    __nv_bfloat16* out_bf16;
    int ldc;
    unsigned int* error;     // set to 1 when a wait runs out
};

__device__ __forceinline__ float gelu_f(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }

// d/dz of z Phi(z): Phi(z) + z phi(z)
__device__ __forceinline__ float gelu_grad_f(float z)
{
    const float cdf = 0.5f * (1.0f + erff(z * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * z * z);
    return cdf + z * pdf;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// UMMA shared-memory matrix descriptor: start, leading and stride byte
// offsets (16-byte units), version 1, no swizzle.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// kind::f16 instruction descriptor: FP32 accumulator, BF16 A and B, both
// K-major, N = bn, M = 128.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int bn)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(smem_u32(bar)), "r"(parity)
                 : "memory");
    return ok != 0;
}

// bounded wait; false when the limit ran out
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity)
{
    for (unsigned long long i = 0; i < WAIT_LIMIT; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "setp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
                 "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void umma_commit(uint64_t* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32])
{
    uint32_t r[32];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                   "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
                   "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
                   "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16])
{
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// Stage rows [row0, row0 + rows) x k [k0, k0 + 64) of a strided BF16 matrix
// into the K-major no-swizzle layout: core matrix (row / 8, k / 8) at
// (row / 8) * 1024 + (k / 8) * 128 bytes, row % 8 selecting its 16-byte row.
// Out-of-range elements are zero.
__device__ __forceinline__ void stage_tile(unsigned char* dst, const __nv_bfloat16* src, long long s_row,
                                           long long s_k, int row0, int rows, int nrows, int k0, int K)
{
    const int items = rows * (GEMM_BK / 8); // (row, 8-element k group)
    for (int it = threadIdx.x; it < items; it += GEMM_THREADS) {
        const int r = it >> 3, g = it & 7;
        const int row = row0 + r;
        const int kb = k0 + g * 8;
        unsigned short e[8];
        if (row < nrows && kb + 8 <= K && s_k == 1 && ((((long long)row * s_row + kb) & 7) == 0)) {
            const uint4 v = *reinterpret_cast<const uint4*>(src + (long long)row * s_row + kb);
            *reinterpret_cast<uint4*>(dst + (r >> 3) * 1024 + g * 128 + (r & 7) * 16) = v;
            continue;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int k = kb + q;
            e[q] = (row < nrows && k < K) ? __bfloat16_as_ushort(src[(long long)row * s_row + (long long)k * s_k]) : 0;
        }
        uint4 v;
        v.x = e[0] | ((uint32_t)e[1] << 16);
        v.y = e[2] | ((uint32_t)e[3] << 16);
        v.z = e[4] | ((uint32_t)e[5] << 16);
        v.w = e[6] | ((uint32_t)e[7] << 16);
        *reinterpret_cast<uint4*>(dst + (r >> 3) * 1024 + g * 128 + (r & 7) * 16) = v;
    }
}

// The same staging for a row-contiguous matrix with 16-byte aligned rows:
// one cp.async of 16 bytes per (row, 8-element k group), zero-filled past
// the matrix edge, in flight together (cp.async.commit_group by the caller).
__device__ __forceinline__ void stage_tile_async(unsigned char* dst, const __nv_bfloat16* src, long long s_row,
                                                 int row0, int rows, int nrows, int k0, int K)
{
    const int items = rows * (GEMM_BK / 8);
    for (int it = threadIdx.x; it < items; it += GEMM_THREADS) {
        const int r = it >> 3, g = it & 7;
        const int row = row0 + r;
        const int kb = k0 + g * 8;
        int bytes = 0;
        const __nv_bfloat16* p = src;
        if (row < nrows && kb < K) {
            bytes = (K - kb >= 8) ? 16 : (K - kb) * 2;
            p = src + (long long)row * s_row + kb;
        }
        const uint32_t d = smem_u32(dst + (r >> 3) * 1024 + g * 128 + (r & 7) * 16);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(p), "r"(bytes) : "memory");
    }
}

// The same staging for a column-contiguous matrix (element (row, k) at
// src[k * s_k + row]; nrows, row0 and s_k multiples of 8, src 16-byte aligned):
// 8 x 8 blocks, eight 16-byte loads along the rows, transposed in registers.
// A warp takes 8 K groups x 4 row groups, so a load instruction covers whole
// 64-byte runs. `chunks` consecutive K chunks, `chunk_bytes` apart, at a time.
__device__ __forceinline__ void stage_tile_t(unsigned char* dst0, const __nv_bfloat16* src, long long s_k, int row0,
                                             int rows, int nrows, int kfirst, int K, int chunks, int chunk_bytes)
{
    for (int t = threadIdx.x; t < rows * chunks; t += GEMM_THREADS) { // rows / 8 row groups x 8 K groups a chunk
        const int c = t / rows, it = t - c * rows;
        const int k0 = kfirst + c * GEMM_BK;
        unsigned char* dst = dst0 + c * chunk_bytes;
        const int g = it & 7, f = it >> 3;
        const int row = row0 + 8 * f;
        uint32_t w[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int k = k0 + 8 * g + i;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (row < nrows && k < K) v = *reinterpret_cast<const uint4*>(src + (long long)k * s_k + row);
            w[i][0] = v.x; w[i][1] = v.y; w[i][2] = v.z; w[i][3] = v.w;
        }
        unsigned char* out = dst + f * 1024 + g * 128;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const uint32_t sel = (r & 1) ? 0x7632u : 0x5410u;
            uint4 v;
            v.x = __byte_perm(w[0][r >> 1], w[1][r >> 1], sel);
            v.y = __byte_perm(w[2][r >> 1], w[3][r >> 1], sel);
            v.z = __byte_perm(w[4][r >> 1], w[5][r >> 1], sel);
            v.w = __byte_perm(w[6][r >> 1], w[7][r >> 1], sel);
            *reinterpret_cast<uint4*>(out + r * 16) = v;
        }
    }
}

// How an operand is staged: by its strides and alignment alone.
enum Staging : int { STAGE_ANY, STAGE_ROWS, STAGE_COLUMNS };
__device__ __forceinline__ Staging staging_of(const __nv_bfloat16* p, long long s_row, long long s_k, int nrows)
{
    const bool aligned = (reinterpret_cast<uintptr_t>(p) & 15) == 0;
    if (aligned && s_k == 1 && (s_row & 7) == 0) return STAGE_ROWS;
    if (aligned && s_row == 1 && (s_k & 7) == 0 && (nrows & 7) == 0) return STAGE_COLUMNS;
    return STAGE_ANY;
}
__device__ __forceinline__ void stage_operand(Staging how, unsigned char* dst, const __nv_bfloat16* p, long long s_row,
                                              long long s_k, int row0, int rows, int nrows, int k0, int K)
{
    if (how == STAGE_ROWS) stage_tile_async(dst, p, s_row, row0, rows, nrows, k0, K);
    else if (how == STAGE_COLUMNS) stage_tile_t(dst, p, s_k, row0, rows, nrows, k0, K, 1, 0);
    else stage_tile(dst, p, s_row, s_k, row0, rows, nrows, k0, K);
}

// tensor memory and barriers of a CTA; every CTA releases what it took
__device__ __forceinline__ uint32_t tile_begin(uint64_t* bars, int n_bars, uint32_t* slot, int* failed, uint32_t cols)
{
    if (threadIdx.x == 0) {
        for (int i = 0; i < n_bars; ++i) mbar_init(&bars[i], 1);
        *failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return *slot;
}
__device__ __forceinline__ void tile_end(uint32_t tmem, uint32_t cols)
{
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (threadIdx.x < 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols));
}

// the MMAs of one staged chunk of `steps` x 16 of K (thread 0)
template <int BN>
__device__ __forceinline__ void chunk_mma(uint32_t tmem, const unsigned char* sA, const unsigned char* sB, int steps,
                                          bool accumulate)
{
    constexpr uint32_t idesc = umma_idesc_bf16(BN);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    for (int j = 0; j < steps; ++j)
        umma_bf16(tmem, umma_desc(smem_u32(sA) + j * 256, 128, 1024), umma_desc(smem_u32(sB) + j * 256, 128, 1024), idesc,
                  (accumulate || j > 0) ? 1u : 0u);
}

__device__ __forceinline__ unsigned char* align1024(unsigned char* p)
{
    return reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(p) + 1023) & ~static_cast<uintptr_t>(1023));
}

__host__ __device__ constexpr uint32_t tmem_cols(int bn) { return bn <= 32 ? 32u : (bn <= 64 ? 64u : 128u); }

template <int BN>
struct LayerSmem {
    static constexpr int A_BYTES = GEMM_BM * GEMM_BK * 2; // 16 KB per chunk
    static constexpr int B_BYTES = BN * GEMM_BK * 2;
    static int bytes(int K) { return ((K + GEMM_BK - 1) / GEMM_BK) * (A_BYTES + B_BYTES) + 1024; } // + alignment slack
};

// Bound by latency, not throughput (a batch of 1,024 is 0.13 GFLOP a layer):
// 32-column tiles give 64 CTAs instead of 8, and K is in flight as a whole
// instead of two chunks. A layer of 1,024 x 256 x 256: 39.7 -> 9.3 us (16.5 with
// 64-column tiles and transposed chunks staged one after the other).
template <int BN>
__global__ void __launch_bounds__(GEMM_THREADS, 1) k_layer(GemmArgs g)
{
    static_assert(BN == 16 || BN == 32, "UMMA N for M = 128; two warps per lane quarter read 16 columns each");
    using L = LayerSmem<BN>;
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;
    const int nk = (g.K + GEMM_BK - 1) / GEMM_BK;
    unsigned char* sA = align1024(smem_raw);
    unsigned char* sB = sA + nk * L::A_BYTES;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * GEMM_BM, n0 = blockIdx.y * BN;
    const uint32_t tmem = tile_begin(&bar, 1, &tmem_slot, &failed, tmem_cols(BN));

    const Staging how_a = staging_of(g.A, g.a_sm, g.a_sk, g.M), how_b = staging_of(g.B, g.b_sn, g.b_sk, g.N);
    // transposed operands: every chunk's loads in flight together
    if (how_a == STAGE_COLUMNS) stage_tile_t(sA, g.A, g.a_sk, m0, GEMM_BM, g.M, 0, g.K, nk, L::A_BYTES);
    if (how_b == STAGE_COLUMNS) stage_tile_t(sB, g.B, g.b_sk, n0, BN, g.N, 0, g.K, nk, L::B_BYTES);
    for (int c = 0; c < nk; ++c) { // row-contiguous chunks land in order while the later ones are in flight
        if (how_a != STAGE_COLUMNS)
            stage_operand(how_a, sA + c * L::A_BYTES, g.A, g.a_sm, g.a_sk, m0, GEMM_BM, g.M, c * GEMM_BK, g.K);
        if (how_b != STAGE_COLUMNS)
            stage_operand(how_b, sB + c * L::B_BYTES, g.B, g.b_sn, g.b_sk, n0, BN, g.N, c * GEMM_BK, g.K);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int c = 0; c < nk; ++c) {
        if (nk - 1 - c >= 3) asm volatile("cp.async.wait_group 3;" ::: "memory");
        else if (nk - 1 - c == 2) asm volatile("cp.async.wait_group 2;" ::: "memory");
        else if (nk - 1 - c == 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // generic/cp.async writes -> async-proxy reads
        __syncthreads();
        if (threadIdx.x == 0) {
            const int left = min(GEMM_BK, g.K - c * GEMM_BK);
            chunk_mma<BN>(tmem, sA + c * L::A_BYTES, sB + c * L::B_BYTES, (left + 15) / 16, c > 0);
            if (c == nk - 1) umma_commit(&bar);
        }
    }
    if (!mbar_wait(&bar, 0)) failed = 1;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncthreads();
    if (failed) {
        if (threadIdx.x == 0) atomicExch(g.error, 1u);
    } else {
        // ---- epilogue: thread = accumulator row (tensor-memory lane); the two
        // warps of a lane quarter take 16 columns each ----
        const int quarter = warp & 3, cc = warp >> 2;
        const int row = m0 + quarter * 32 + lane;
        if (16 * cc < BN) {
            float v[16];
            tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(cc * 16), v);
            const long long base = (long long)row * g.ldc;
            const int nb0 = n0 + cc * 16;
            if (row >= g.M) {
            } else if (nb0 + 16 <= g.N && (g.ldc & 7) == 0) {
                // a whole 16-column run of this row: 16-byte stores (the row's
                // 32 or 64 bytes are contiguous)
                const float4* x4 = reinterpret_cast<const float4*>(g.epilogue == EPI_DGELU_BF16 ? g.aux_f32 + base + nb0
                                                                                                 : g.bias + nb0);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 x = x4[i];
                    if (g.epilogue == EPI_DGELU_BF16) {
                        v[4 * i] *= gelu_grad_f(x.x);
                        v[4 * i + 1] *= gelu_grad_f(x.y);
                        v[4 * i + 2] *= gelu_grad_f(x.z);
                        v[4 * i + 3] *= gelu_grad_f(x.w);
                    } else {
                        v[4 * i] += x.x;
                        v[4 * i + 1] += x.y;
                        v[4 * i + 2] += x.z;
                        v[4 * i + 3] += x.w;
                    }
                }
                if (g.epilogue != EPI_DGELU_BF16) {
                    float4* o4 = reinterpret_cast<float4*>(g.out_f32 + base + nb0);
#pragma unroll
                    for (int i = 0; i < 4; ++i) o4[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                }
                if (g.epilogue != EPI_BIAS_F32) {
                    const bool act = g.epilogue != EPI_DGELU_BF16;
                    uint4* o4 = reinterpret_cast<uint4*>(g.out_bf16 + base + nb0);
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        uint32_t w[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const float x0 = act ? gelu_f(v[8 * i + 2 * j]) : v[8 * i + 2 * j];
                            const float x1 = act ? gelu_f(v[8 * i + 2 * j + 1]) : v[8 * i + 2 * j + 1];
                            w[j] = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(x0)) |
                                   ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(x1)) << 16);
                        }
                        o4[i] = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
            } else {
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const int n = nb0 + i;
                    if (n >= g.N) break;
                    const float a = v[i];
                    switch (g.epilogue) {
                    case EPI_BIAS_F32: g.out_f32[base + n] = a + g.bias[n]; break;
                    case EPI_BIAS_GELU: {
                        const float z = a + g.bias[n];
                        g.out_f32[base + n] = z;
                        g.out_bf16[base + n] = __float2bfloat16_rn(gelu_f(z));
                        break;
                    }
                    default: // EPI_DGELU_BF16
                        g.out_bf16[base + n] = __float2bfloat16_rn(a * gelu_grad_f(g.aux_f32[base + n]));
                    }
                }
            }
        }
    }
    tile_end(tmem, tmem_cols(BN));
}

// ---------------------------------------------------------------------------
// weight and bias gradients
// ---------------------------------------------------------------------------
// dW[o][i] = sum_b dz[b][o] x[b][i] and db[o] = sum_b dz[b][o] of one layer
struct WeightGrad {
    const __nv_bfloat16* dz; // [batch][outs]
    const __nv_bfloat16* x;  // [batch][ins]
    int outs, ins;
    long long off_w, off_b;  // in the flat parameter vector
    int first_tile;          // of the launch's tiles, 128 outputs x 64 inputs each
    int m_tiles;
};

struct WeightGradArgs {
    WeightGrad layer[4];     // by first_tile
    int batch, slice;        // samples, samples of a slice (a multiple of 64)
    float* partial;          // [slice][n_params]
    long long n_params;
    unsigned int* error;
};

// Few output tiles (22 over the four layers) and a long contraction: the batch
// is split over blockIdx.y so that a batch of 1,024 is 352 CTAs instead of the
// two of an unsplit 256 x 256 product (148 us, and 60 us for a column sum of
// one thread per output). All weight and bias gradients of that batch: 15.8 us.
__global__ void __launch_bounds__(GEMM_THREADS, 1) k_weight_grads(WeightGradArgs a)
{
    constexpr int BN = 64;
    using L = LayerSmem<BN>;
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;
    int li = 0;
#pragma unroll
    for (int k = 1; k < 4; ++k)
        if ((int)blockIdx.x >= a.layer[k].first_tile) li = k;
    const WeightGrad w = a.layer[li];
    const int tile = blockIdx.x - w.first_tile;
    const int m0 = (tile % w.m_tiles) * GEMM_BM, n0 = (tile / w.m_tiles) * BN;
    const int kb = blockIdx.y * a.slice, ke = min(a.batch, kb + a.slice);
    unsigned char* sA = align1024(smem_raw);
    unsigned char* sB = sA + 2 * L::A_BYTES;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t tmem = tile_begin(bar, 2, &tmem_slot, &failed, tmem_cols(BN));
    const Staging how_a = staging_of(w.dz, 1, w.outs, w.outs), how_b = staging_of(w.x, 1, w.ins, w.ins);
    const int nk = (ke - kb + GEMM_BK - 1) / GEMM_BK;
    float bias = 0.0f; // thread r < 128: output m0 + r
    for (int c = 0; c < nk; ++c) {
        const int b = c & 1, k0 = kb + c * GEMM_BK;
        unsigned char* cA = sA + b * L::A_BYTES;
        unsigned char* cB = sB + b * L::B_BYTES;
        // the MMAs of chunk c - 2 read this buffer: wait for them before overwriting it
        if (c >= 2 && !mbar_wait(&bar[b], ((c - 2) >> 1) & 1)) failed = 1;
        stage_operand(how_a, cA, w.dz, 1, w.outs, m0, GEMM_BM, w.outs, k0, ke);
        stage_operand(how_b, cB, w.x, 1, w.ins, n0, BN, w.ins, k0, ke);
        asm volatile("cp.async.wait_all;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (threadIdx.x == 0) {
            chunk_mma<BN>(tmem, cA, cB, (min(GEMM_BK, ke - k0) + 15) / 16, c > 0);
            umma_commit(&bar[b]);
        }
        if (n0 == 0 && threadIdx.x < GEMM_BM) { // the staged outputs of this chunk, in batch order
            const unsigned char* row = cA + (threadIdx.x >> 3) * 1024 + (threadIdx.x & 7) * 16;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const uint4 v = *reinterpret_cast<const uint4*>(row + q * 128);
                const uint32_t e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    bias += __uint_as_float(e[j] << 16);
                    bias += __uint_as_float(e[j] & 0xffff0000u);
                }
            }
        }
    }
    const int last = nk - 1;
    if (!mbar_wait(&bar[last & 1], (last >> 1) & 1)) failed = 1;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncthreads();
    float* out = a.partial + (long long)blockIdx.y * a.n_params;
    if (failed) {
        if (threadIdx.x == 0) atomicExch(a.error, 1u);
    } else {
        const int quarter = warp & 3, cc = warp >> 2;
        const int o = m0 + quarter * 32 + lane;
        float v[32];
        tmem_ld32(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(cc * 32), v);
        const int i0 = n0 + cc * 32;
        if (o < w.outs) {
            float* row = out + w.off_w + (long long)o * w.ins + i0;
            if (i0 + 32 <= w.ins && (w.ins & 3) == 0 && (w.off_w & 3) == 0 && (a.n_params & 3) == 0) {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    reinterpret_cast<float4*>(row)[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            } else {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (i0 + i < w.ins) row[i] = v[i];
            }
        }
        if (n0 == 0 && threadIdx.x < GEMM_BM && m0 + (int)threadIdx.x < w.outs) out[w.off_b + m0 + threadIdx.x] = bias;
    }
    tile_end(tmem, tmem_cols(BN));
}

} // namespace surrogate
