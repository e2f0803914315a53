// Learned plan scorer: a 3-layer MLP (in → H → H → 1, ReLU) that predicts a
// plan's log runtime from its features.  It stands in for the cost the
// reference's optimizer minimises (computeOrderCost / optCostOrder,
// plan/optimizer.cpp:319-577, fed by cardEstimateUnlabeled,
// plan/estimator.cpp:562-661); the cost model stays as the fallback and as
// the baseline the scorer is compared with.
//
// Training runs on the GPU in FP32 with this file's kernels (tiled SGEMM,
// bias/ReLU epilogues, column-sum bias gradients, Adam).  Batched inference
// runs in BF16 on the tensor cores (mma.sync m16n8k16, FP32 accumulate): the
// scorer is a few microseconds per pattern, far from any roofline that would
// justify the tcgen05 machinery.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.hpp"
#include "device_util.hpp"

using namespace sge;

struct sge_mlp {
    int device = 0;
    uint32_t in = 0, hid = 0;
    cudaStream_t stream = nullptr;
    // parameters (FP32): W1 [hid×in], b1 [hid], W2 [hid×hid], b2 [hid], W3 [hid], b3 [1]
    float *d_p = nullptr, *d_g = nullptr, *d_m = nullptr, *d_v = nullptr;
    size_t np = 0;
    uint64_t adam_t = 0;
    // BF16 copies of the weight matrices for inference
    __nv_bfloat16 *d_w1h = nullptr, *d_w2h = nullptr;
    bool bf16_stale = true;
    // workspace
    float *d_ws = nullptr;
    size_t ws_floats = 0;
};

namespace {

#define CUDA_TRY(expr)                                                                               \
    do {                                                                                             \
        cudaError_t _e = (expr);                                                                     \
        if (_e != cudaSuccess)                                                                       \
            return fail(_e == cudaErrorMemoryAllocation ? SGE_OOM : SGE_CUDA_ERROR, "%s: %s", #expr, \
                        cudaGetErrorString(_e));                                                     \
    } while (0)

constexpr int TILE = 16;

// C[M×N] = op(A)·op(B) (+ bias[N]) (ReLU) ; A is M×K (TA: stored K×M), B is K×N
// (TB: stored N×K), all row-major.  beta accumulates into C.
template <bool TA, bool TB>
__global__ void sgemm(const float *__restrict__ A, const float *__restrict__ B, float *__restrict__ C, int M, int N,
                      int K, const float *__restrict__ bias, int relu, float beta) {
    __shared__ float As[TILE][TILE + 1];
    __shared__ float Bs[TILE][TILE + 1];
    const int r = blockIdx.y * TILE + threadIdx.y, col = blockIdx.x * TILE + threadIdx.x;
    float acc = 0.f;
    for (int k0 = 0; k0 < K; k0 += TILE) {
        const int ka = k0 + threadIdx.x, kb = k0 + threadIdx.y;
        As[threadIdx.y][threadIdx.x] = (r < M && ka < K) ? (TA ? A[(size_t)ka * M + r] : A[(size_t)r * K + ka]) : 0.f;
        Bs[threadIdx.y][threadIdx.x] = (kb < K && col < N) ? (TB ? B[(size_t)col * K + kb] : B[(size_t)kb * N + col]) : 0.f;
        __syncthreads();
#pragma unroll
        for (int t = 0; t < TILE; ++t) acc += As[threadIdx.y][t] * Bs[t][threadIdx.x];
        __syncthreads();
    }
    if (r < M && col < N) {
        float v = acc;
        if (bias) v += bias[col];
        if (relu) v = v > 0.f ? v : 0.f;
        C[(size_t)r * N + col] = beta != 0.f ? beta * C[(size_t)r * N + col] + v : v;
    }
}

// dZ = dA ⊙ (Z > 0)
__global__ void relu_grad(float *dA, const float *Z, size_t n) {
    size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i < n && Z[i] <= 0.f) dA[i] = 0.f;
}

// out[j] = Σ_i X[i][j]  (bias gradient), X is rows×cols
__global__ void colsum(const float *X, float *out, int rows, int cols) {
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= cols) return;
    float s = 0.f;
    for (int i = 0; i < rows; ++i) s += X[(size_t)i * cols + j];
    out[j] = s;
}

// dy = (y - t) / B ; loss partials
__global__ void mse_grad(const float *y, const float *t, float *dy, float *loss, int B) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= B) return;
    float d = y[i] - t[i];
    dy[i] = d / (float)B;
    atomicAdd(loss, 0.5f * d * d / (float)B);
}

__global__ void adam(float *p, const float *g, float *m, float *v, size_t n, float lr, float b1, float b2,
                     float eps, float c1, float c2) {
    size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    float gi = g[i];
    m[i] = b1 * m[i] + (1.f - b1) * gi;
    v[i] = b2 * v[i] + (1.f - b2) * gi * gi;
    p[i] -= lr * (m[i] / c1) / (sqrtf(v[i] / c2) + eps);
}

__global__ void to_bf16(const float *x, __nv_bfloat16 *y, size_t n) {
    size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i < n) y[i] = __float2bfloat16_rn(x[i]);
}

// ---- BF16 tensor-core layer: Z[B×N] = X[B×K]·Wᵀ (W is N×K) + bias, ReLU ----
// One warp computes a 16×8 tile with mma.sync.m16n8k16 (row.col, f32 accumulate).
// Fragment layout (PTX ISA, m16n8k16 .bf16): g = lane/4, t = lane%4;
//   A regs: (g, 2t..2t+1), (g+8, 2t..), (g, 2t+8..), (g+8, 2t+8..)
//   B regs: (k 2t..2t+1, n g), (k 2t+8..2t+9, n g)
//   C/D:    (g, 2t), (g, 2t+1), (g+8, 2t), (g+8, 2t+1)
__device__ __forceinline__ uint32_t pack2(const __nv_bfloat16 *p, int stride_ok0, int stride_ok1) {
    __nv_bfloat162 v;
    v.x = stride_ok0 ? p[0] : __float2bfloat16_rn(0.f);
    v.y = stride_ok1 ? p[1] : __float2bfloat16_rn(0.f);
    return *reinterpret_cast<uint32_t *>(&v);
}

__global__ void bf16_linear(const __nv_bfloat16 *__restrict__ X, const __nv_bfloat16 *__restrict__ W,
                            const float *__restrict__ bias, float *__restrict__ Z, __nv_bfloat16 *__restrict__ Zh,
                            int B, int N, int K, int relu) {
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int tiles_n = (N + 7) / 8;
    const int tm = warp / tiles_n, tn = warp % tiles_n;
    if (tm * 16 >= B) return;
    const int g = lane >> 2, t = lane & 3;
    const int r0 = tm * 16 + g, r1 = r0 + 8, n = tn * 8 + g;
    float c0 = 0.f, c1 = 0.f, c2 = 0.f, c3 = 0.f;
    for (int k0 = 0; k0 < K; k0 += 16) {
        const int ka = k0 + 2 * t, kb = ka + 8;
        uint32_t a0 = pack2(X + (size_t)r0 * K + ka, r0 < B && ka < K, r0 < B && ka + 1 < K);
        uint32_t a1 = pack2(X + (size_t)r1 * K + ka, r1 < B && ka < K, r1 < B && ka + 1 < K);
        uint32_t a2 = pack2(X + (size_t)r0 * K + kb, r0 < B && kb < K, r0 < B && kb + 1 < K);
        uint32_t a3 = pack2(X + (size_t)r1 * K + kb, r1 < B && kb < K, r1 < B && kb + 1 < K);
        uint32_t b0 = pack2(W + (size_t)n * K + ka, n < N && ka < K, n < N && ka + 1 < K);
        uint32_t b1 = pack2(W + (size_t)n * K + kb, n < N && kb < K, n < N && kb + 1 < K);
        asm volatile(
            "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
            "{%0,%1,%2,%3};\n"
            : "+f"(c0), "+f"(c1), "+f"(c2), "+f"(c3)
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    }
    const int col0 = tn * 8 + 2 * t;
    float out[4] = {c0, c1, c2, c3};
    const int rows[4] = {r0, r0, r1, r1};
    const int cols[4] = {col0, col0 + 1, col0, col0 + 1};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (rows[q] < B && cols[q] < N) {
            float v = out[q] + (bias ? bias[cols[q]] : 0.f);
            if (relu) v = v > 0.f ? v : 0.f;
            if (Z) Z[(size_t)rows[q] * N + cols[q]] = v;
            if (Zh) Zh[(size_t)rows[q] * N + cols[q]] = __float2bfloat16_rn(v);
        }
    }
}

// y[i] = Σ_j A2[i][j]·w3[j] + b3 (FP32; the last layer has one output)
__global__ void dot_out(const float *A, const float *w, const float *b, float *y, int B, int H) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= B) return;
    float s = b[0];
    for (int j = 0; j < H; ++j) s += A[(size_t)i * H + j] * w[j];
    y[i] = s;
}

// ---- fused kernels for layers of at most FUSE_MAX units (the plan scorer's
// 64 -> 128 -> 128 -> 1) ----
// A call on this network is launch latency: the layer kernels above take 5
// launches per BF16 forward and 20 per training batch.  A block here keeps all
// weights in shared memory and takes its rows through every layer; sums run in
// the layer kernels' order (ascending, one FMA chain per element), so FP32
// results do not change.
constexpr int FUSE_MAX = 128;

// BF16 forward, 32 rows per block: warp (r, h) computes 16 rows x half of the
// columns of each layer with mma.sync, activations pass through shared memory.
// 4,992 x 64 features: 5 launches -> 1, the whole call 98 -> 51 us.
constexpr int BF_ROWS = 32;
struct BfSmem {
    __nv_bfloat16 w1[FUSE_MAX][FUSE_MAX + 8], w2[FUSE_MAX][FUSE_MAX + 8];   // (pitch: 4 words past a bank row)
    __nv_bfloat16 x[BF_ROWS][FUSE_MAX + 8], a1[BF_ROWS][FUSE_MAX + 8];
    float y[2][BF_ROWS];
};
// acc[t] (16 x 8 tiles, columns from col0) = rows of A [.. x K] times W^T
__device__ __forceinline__ void bf_layer(const __nv_bfloat16 (*A)[FUSE_MAX + 8], const __nv_bfloat16 (*W)[FUSE_MAX + 8],
                                         int row0, int col0, int K, float (*acc)[4]) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int n = 0; n < FUSE_MAX / 16; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
    for (int k0 = 0; k0 < K; k0 += 16) {
        auto two = [&](const __nv_bfloat16 *p) { return *reinterpret_cast<const uint32_t *>(p); };
        const uint32_t a0 = two(&A[row0 + g][k0 + 2 * t]), a1 = two(&A[row0 + g + 8][k0 + 2 * t]),
                       a2 = two(&A[row0 + g][k0 + 2 * t + 8]), a3 = two(&A[row0 + g + 8][k0 + 2 * t + 8]);
#pragma unroll
        for (int n = 0; n < FUSE_MAX / 16; ++n) {
            const uint32_t b0 = two(&W[col0 + n * 8 + g][k0 + 2 * t]), b1 = two(&W[col0 + n * 8 + g][k0 + 2 * t + 8]);
            asm volatile(
                "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                "{%0,%1,%2,%3};\n"
                : "+f"(acc[n][0]), "+f"(acc[n][1]), "+f"(acc[n][2]), "+f"(acc[n][3])
                : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
        }
    }
}
__global__ void __launch_bounds__(128) bf16_forward_fused(const float *__restrict__ X, const __nv_bfloat16 *__restrict__ W1,
                                                          const float *__restrict__ b1,
                                                          const __nv_bfloat16 *__restrict__ W2,
                                                          const float *__restrict__ b2, const float *__restrict__ w3,
                                                          const float *__restrict__ b3, float *__restrict__ y, int B,
                                                          int in, int hid) {
    extern __shared__ __align__(16) unsigned char raw[];
    BfSmem &S = *reinterpret_cast<BfSmem *>(raw);
    const int r0 = blockIdx.x * BF_ROWS, tid = threadIdx.x;
    const __nv_bfloat16 zero = __float2bfloat16_rn(0.f);
    if (in % 8 == 0 && hid % 8 == 0) {   // rows of 16-byte pieces
        const int q1 = in / 8, q2 = hid / 8;
        for (int i = tid; i < FUSE_MAX * q1; i += 128) {
            const int r = i / q1, c = i % q1;
            *reinterpret_cast<uint4 *>(&S.w1[r][c * 8]) =
                r < hid ? reinterpret_cast<const uint4 *>(W1)[(size_t)r * q1 + c] : make_uint4(0, 0, 0, 0);
        }
        for (int i = tid; i < FUSE_MAX * q2; i += 128) {
            const int r = i / q2, c = i % q2;
            *reinterpret_cast<uint4 *>(&S.w2[r][c * 8]) =
                r < hid ? reinterpret_cast<const uint4 *>(W2)[(size_t)r * q2 + c] : make_uint4(0, 0, 0, 0);
        }
    }
    const int ka = (in + 15) & ~15, kb = (hid + 15) & ~15;   // K padded with zeros
    if (in % 8 || hid % 8 || ka != in || kb != hid)
        for (int i = tid; i < FUSE_MAX * FUSE_MAX; i += 128) {
            const int r = i / FUSE_MAX, c = i % FUSE_MAX;
            S.w1[r][c] = r < hid && c < in ? W1[(size_t)r * in + c] : zero;
            S.w2[r][c] = r < hid && c < hid ? W2[(size_t)r * hid + c] : zero;
        }
    for (int i = tid; i < BF_ROWS * ka; i += 128) {
        const int r = i / ka, c = i % ka;
        S.x[r][c] = r0 + r < B && c < in ? __float2bfloat16_rn(X[(size_t)(r0 + r) * in + c]) : zero;
    }
    __syncthreads();
    const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int row0 = (warp & 1) * 16, half = warp >> 1, col0 = half * (FUSE_MAX / 2);
    float acc[FUSE_MAX / 16][4];
    bf_layer(S.x, S.w1, row0, col0, ka, acc);
#pragma unroll
    for (int n = 0; n < FUSE_MAX / 16; ++n)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int c = col0 + n * 8 + 2 * t + (q & 1), r = row0 + g + (q >> 1) * 8;
            const float v = acc[n][q] + (c < hid ? b1[c] : 0.f);
            S.a1[r][c] = __float2bfloat16_rn(v > 0.f ? v : 0.f);
        }
    __syncthreads();
    bf_layer(S.a1, S.w2, row0, col0, kb, acc);
    float s0 = 0.f, s1 = 0.f;   // this lane's columns of rows g and g + 8
#pragma unroll
    for (int n = 0; n < FUSE_MAX / 16; ++n)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int c = col0 + n * 8 + 2 * t + (q & 1);
            const float bias = c < hid ? b2[c] : 0.f, w = c < hid ? w3[c] : 0.f;
            const float v = acc[n][q] + bias;
            const float a = v > 0.f ? v : 0.f;
            if (q < 2) s0 += a * w;
            else s1 += a * w;
        }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
        s0 += __shfl_xor_sync(0xFFFFFFFFu, s0, o);
        s1 += __shfl_xor_sync(0xFFFFFFFFu, s1, o);
    }
    if (t == 0) {
        S.y[half][row0 + g] = s0;
        S.y[half][row0 + g + 8] = s1;
    }
    __syncthreads();
    if (tid < BF_ROWS && r0 + tid < B) y[r0 + tid] = b3[0] + S.y[0][tid] + S.y[1][tid];
}

// One batch's rows through the network and back, FT_ROWS per block: A1, A2 and
// the gradients at Z1, Z2 for the parameter kernel, and the loss.  Row i of the
// batch is row idx[i] of x and t (i itself when idx is null).  x may be X: a
// batch that is in order already gathers onto itself, so neither is __restrict__.
constexpr int FT_ROWS = 4, FT_THREADS = 256;
struct FtSmem {
    float w1[FUSE_MAX][FUSE_MAX + 1], w2[FUSE_MAX][FUSE_MAX + 1];
    float x[FT_ROWS][FUSE_MAX], a1[FT_ROWS][FUSE_MAX], a2[FT_ROWS][FUSE_MAX], z[FT_ROWS][FUSE_MAX];
    float w3[FUSE_MAX], dy[FT_ROWS], loss[FT_ROWS];
};
// A row-major matrix of `cols` <= FUSE_MAX columns into padded rows, a warp per
// row and four columns per lane.
__device__ __forceinline__ void fill_rows(float (*out)[FUSE_MAX + 1], const float *__restrict__ w, int rows, int cols) {
    constexpr int STEP = FT_THREADS / 32, AHEAD = 8;   // rows in flight per warp
    const int c0 = 4 * (threadIdx.x & 31);
    const bool vec = cols % 4 == 0;
    for (int r0 = threadIdx.x >> 5; r0 < rows; r0 += STEP * AHEAD) {
        float4 v[AHEAD];
#pragma unroll
        for (int q = 0; q < AHEAD; ++q) {
            const int r = r0 + q * STEP;
            const float *p = w + (size_t)r * cols + c0;
            v[q] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r >= rows || c0 >= cols) continue;
            if (vec) v[q] = *reinterpret_cast<const float4 *>(p);
            else {
                v[q].x = p[0];
                if (c0 + 1 < cols) v[q].y = p[1];
                if (c0 + 2 < cols) v[q].z = p[2];
                if (c0 + 3 < cols) v[q].w = p[3];
            }
        }
#pragma unroll
        for (int q = 0; q < AHEAD; ++q) {
            const int r = r0 + q * STEP;
            if (r >= rows) break;
            if (c0 < cols) out[r][c0] = v[q].x;
            if (c0 + 1 < cols) out[r][c0 + 1] = v[q].y;
            if (c0 + 2 < cols) out[r][c0 + 2] = v[q].z;
            if (c0 + 3 < cols) out[r][c0 + 3] = v[q].w;
        }
    }
}
__global__ void __launch_bounds__(FT_THREADS) train_rows_fused(const float *__restrict__ P, const float *x,
                                                               const float *__restrict__ t,
                                                               const uint32_t *__restrict__ idx, int B, int in, int hid,
                                                               float *X, float *__restrict__ A1,
                                                               float *__restrict__ A2, float *__restrict__ dZ1,
                                                               float *__restrict__ dZ2, float *__restrict__ dY,
                                                               float *__restrict__ loss) {
    extern __shared__ __align__(16) unsigned char raw[];
    FtSmem &S = *reinterpret_cast<FtSmem *>(raw);
    const int r0 = blockIdx.x * FT_ROWS, tid = threadIdx.x;
    const float *W1 = P, *b1 = W1 + (size_t)hid * in, *W2 = b1 + hid, *b2 = W2 + (size_t)hid * hid, *w3 = b2 + hid,
                *b3 = w3 + hid;
    fill_rows(S.w1, W1, hid, in);
    fill_rows(S.w2, W2, hid, hid);
    if (tid < hid) S.w3[tid] = w3[tid];
    for (int i = tid; i < FT_ROWS * in; i += FT_THREADS) {
        const int r = r0 + i / in, c = i % in;
        const float v = r < B ? x[(size_t)(idx ? idx[r] : r) * in + c] : 0.f;
        S.x[i / in][c] = v;
        if (r < B) X[(size_t)r * in + c] = v;
    }
    __syncthreads();
    // thread (j, q): column j of rows q and q + 2
    const int j = tid % FUSE_MAX, q = tid / FUSE_MAX;
    constexpr int R = FT_ROWS * FUSE_MAX / FT_THREADS;
    float z1[R], z2[R];
    if (j < hid) {
        float acc[R] = {};
#pragma unroll 8
        for (int k = 0; k < in; ++k)
#pragma unroll
            for (int r = 0; r < R; ++r) acc[r] = fmaf(S.x[q + 2 * r][k], S.w1[j][k], acc[r]);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            z1[r] = acc[r] + b1[j];
            S.a1[q + 2 * r][j] = z1[r] <= 0.f ? 0.f : z1[r];
        }
    }
    __syncthreads();
    if (j < hid) {
        float acc[R] = {};
#pragma unroll 8
        for (int k = 0; k < hid; ++k)
#pragma unroll
            for (int r = 0; r < R; ++r) acc[r] = fmaf(S.a1[q + 2 * r][k], S.w2[j][k], acc[r]);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            z2[r] = acc[r] + b2[j];
            S.a2[q + 2 * r][j] = z2[r] <= 0.f ? 0.f : z2[r];
        }
    }
    __syncthreads();
    if (tid < FT_ROWS) {
        float s = b3[0];
#pragma unroll 8
        for (int k = 0; k < hid; ++k) s += S.a2[tid][k] * S.w3[k];
        float l = 0.f, g = 0.f;
        if (r0 + tid < B) {
            const float d = s - t[idx ? idx[r0 + tid] : r0 + tid];
            g = d / (float)B;
            l = 0.5f * d * d / (float)B;
            dY[r0 + tid] = g;
        }
        S.dy[tid] = g;
        S.loss[tid] = l;
    }
    __syncthreads();
    if (tid == 0) {
        float l = 0.f;
        for (int r = 0; r < FT_ROWS; ++r) l += S.loss[r];
        atomicAdd(loss, l);
    }
    if (j < hid) {
#pragma unroll
        for (int r = 0; r < R; ++r) S.z[q + 2 * r][j] = z2[r] <= 0.f ? 0.f : S.dy[q + 2 * r] * S.w3[j];
    }
    __syncthreads();
    if (j < hid) {
        float acc[R] = {};
#pragma unroll 8
        for (int k = 0; k < hid; ++k)
#pragma unroll
            for (int r = 0; r < R; ++r) acc[r] = fmaf(S.z[q + 2 * r][k], S.w2[k][j], acc[r]);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int row = r0 + q + 2 * r;
            if (row >= B) continue;
            const size_t o = (size_t)row * hid + j;
            A1[o] = S.a1[q + 2 * r][j];
            A2[o] = S.a2[q + 2 * r][j];
            dZ2[o] = S.z[q + 2 * r][j];
            dZ1[o] = z1[r] <= 0.f ? 0.f : acc[r];
        }
    }
}

// Gradients over the batch (rows in order), then the gradient itself (G) or one
// Adam step.  A block takes PG_OUT rows of W2 or W1 (dZ columns) against every
// column: 128 batch rows at a time in shared memory, four elements a thread;
// the last blocks take the biases and W3, one element a thread.  (One thread
// per element reading global memory took 24 us a batch, this 11.)
struct AdamState {
    float p, m, v;
};
__device__ __forceinline__ AdamState adam_load(const float *p, const float *m, const float *v, int e) {
    return AdamState{p[e], m[e], v[e]};
}
__device__ __forceinline__ void adam_step(AdamState &s, float gi, float lr, float b1, float b2, float eps, float c1,
                                          float c2) {
    s.m = b1 * s.m + (1.f - b1) * gi;
    s.v = b2 * s.v + (1.f - b2) * gi * gi;
    s.p -= lr * (s.m / c1) / (sqrtf(s.v / c2) + eps);
}
constexpr int PG_OUT = 8, PG_K = 128;
struct PgSmem {
    float a[PG_K][PG_OUT], b[PG_K][FUSE_MAX];
};
__global__ void __launch_bounds__(256) param_grads_fused(const float *__restrict__ X, const float *__restrict__ A1,
                                                         const float *__restrict__ A2, const float *__restrict__ dZ1,
                                                         const float *__restrict__ dZ2, const float *__restrict__ dY,
                                                         int B, int in, int hid, float *__restrict__ G, float *p,
                                                         float *m, float *v, float lr, float c1, float c2) {
    extern __shared__ __align__(16) unsigned char raw[];
    PgSmem &S = *reinterpret_cast<PgSmem *>(raw);
    const int n1 = hid * in, n2 = hid * hid, tid = threadIdx.x;
    auto put = [&](int e, float s, AdamState &st) {
        if (G) { G[e] = s; return; }
        adam_step(st, s, lr, 0.9f, 0.999f, 1e-8f, c1, c2);
        p[e] = st.p;
        m[e] = st.m;
        v[e] = st.v;
    };
    const int groups = (hid + PG_OUT - 1) / PG_OUT;
    if ((int)blockIdx.x < 2 * groups) {
        const bool second = (int)blockIdx.x < groups;
        const int r0 = ((int)blockIdx.x % groups) * PG_OUT, cols = second ? hid : in;
        const float *dZ = second ? dZ2 : dZ1, *in_act = second ? A1 : X;
        const int c = tid % FUSE_MAX, q = tid / FUSE_MAX;   // column c of rows q, q + 2, q + 4, q + 6
        float acc[PG_OUT / 2] = {};
        // this thread's parameters and moments, asked for before the sums
        AdamState st[PG_OUT / 2] = {};
        auto index = [&](int r) { return (second ? n1 + hid : 0) + (r0 + q + 2 * r) * cols + c; };
        if (!G && c < cols)
#pragma unroll
            for (int r = 0; r < PG_OUT / 2; ++r)
                if (r0 + q + 2 * r < hid) st[r] = adam_load(p, m, v, index(r));
        for (int k0 = 0; k0 < B; k0 += PG_K) {
            const int kn = min(PG_K, B - k0);
            __syncthreads();
            float va[PG_K * PG_OUT / 256];
#pragma unroll
            for (int i = 0; i < PG_K * PG_OUT / 256; ++i) {
                const int k = (i * 256 + tid) / PG_OUT, r = (i * 256 + tid) % PG_OUT;
                va[i] = k < kn && r0 + r < hid ? dZ[(size_t)(k0 + k) * hid + r0 + r] : 0.f;
            }
#pragma unroll
            for (int h = 0; h < PG_K / 2; h += 16) {   // 16 loads in flight
                float vb[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const int k = 2 * (h + i) + q;
                    vb[i] = k < kn && c < cols ? in_act[(size_t)(k0 + k) * cols + c] : 0.f;
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) S.b[2 * (h + i) + q][c] = vb[i];
            }
#pragma unroll
            for (int i = 0; i < PG_K * PG_OUT / 256; ++i) S.a[(i * 256 + tid) / PG_OUT][(i * 256 + tid) % PG_OUT] = va[i];
            __syncthreads();
            if (c < cols) {
#pragma unroll 8
                for (int k = 0; k < kn; ++k) {
                    const float y = S.b[k][c];
#pragma unroll
                    for (int r = 0; r < PG_OUT / 2; ++r) acc[r] = fmaf(S.a[k][q + 2 * r], y, acc[r]);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < PG_OUT / 2; ++r) {
            const int row = r0 + q + 2 * r;
            if (row < hid && c < cols) put(index(r), acc[r], st[r]);
        }
        return;
    }
    // biases, W3 and its bias: Σ_i a[i * as] * b[i] (b null: Σ a)
    const int e = ((int)blockIdx.x - 2 * groups) * 256 + tid;
    if (e >= 3 * hid + 1) return;
    const float *a, *b = nullptr;
    int as = hid, o = e, at;
    if (o < hid) { a = dZ1 + o; at = n1 + o; }
    else if ((o -= hid) < hid) { a = dZ2 + o; at = n1 + hid + n2 + o; }
    else if ((o -= hid) < hid) { a = A2 + o; b = dY; at = n1 + 2 * hid + n2 + o; }
    else { a = dY; as = 1; at = n1 + 3 * hid + n2; }
    float s = 0.f;
    if (b) {
#pragma unroll 16
        for (int i = 0; i < B; ++i) s = fmaf(a[(size_t)i * as], b[i], s);
    } else {
#pragma unroll 16
        for (int i = 0; i < B; ++i) s += a[(size_t)i * as];
    }
    AdamState st{};
    if (!G) st = adam_load(p, m, v, at);
    put(at, s, st);
}

inline bool fused(const sge_mlp *m) { return m->in <= FUSE_MAX && m->hid <= FUSE_MAX; }

inline dim3 gemm_grid(int M, int N) { return dim3((N + TILE - 1) / TILE, (M + TILE - 1) / TILE); }

struct Layout {
    size_t w1, b1, w2, b2, w3, b3, n;
};
Layout layout(uint32_t in, uint32_t hid) {
    Layout L;
    L.w1 = 0;
    L.b1 = L.w1 + (size_t)hid * in;
    L.w2 = L.b1 + hid;
    L.b2 = L.w2 + (size_t)hid * hid;
    L.w3 = L.b2 + hid;
    L.b3 = L.w3 + hid;
    L.n = L.b3 + 1;
    return L;
}

sge_status ensure_ws(sge_mlp *m, uint32_t B) {
    // X, Z1, A1, Z2, A2, y, t, dy, dA, loss
    size_t need = (size_t)B * m->in + 4ull * B * m->hid + 3ull * B + (size_t)B * m->hid + 64;
    if (m->ws_floats >= need) return SGE_OK;
    cudaFree(m->d_ws);
    m->d_ws = nullptr;
    CUDA_TRY(cudaMalloc(&m->d_ws, need * sizeof(float)));
    m->ws_floats = need;
    return SGE_OK;
}

// Forward in FP32; leaves Z1, A1, Z2, A2, y in the workspace.
void forward_fp32(sge_mlp *m, const Layout &L, float *X, float *Z1, float *A1, float *Z2, float *A2, float *y,
                  uint32_t B) {
    const dim3 blk(TILE, TILE);
    float *P = m->d_p;
    sgemm<false, true><<<gemm_grid(B, m->hid), blk, 0, m->stream>>>(X, P + L.w1, Z1, B, m->hid, m->in, P + L.b1, 0, 0.f);
    cudaMemcpyAsync(A1, Z1, sizeof(float) * B * m->hid, cudaMemcpyDeviceToDevice, m->stream);
    size_t nh = (size_t)B * m->hid;
    relu_grad<<<(unsigned)((nh + 255) / 256), 256, 0, m->stream>>>(A1, Z1, nh);  // A1 = relu(Z1)
    sgemm<false, true><<<gemm_grid(B, m->hid), blk, 0, m->stream>>>(A1, P + L.w2, Z2, B, m->hid, m->hid, P + L.b2, 0, 0.f);
    cudaMemcpyAsync(A2, Z2, sizeof(float) * nh, cudaMemcpyDeviceToDevice, m->stream);
    relu_grad<<<(unsigned)((nh + 255) / 256), 256, 0, m->stream>>>(A2, Z2, nh);
    dot_out<<<(B + 255) / 256, 256, 0, m->stream>>>(A2, P + L.w3, P + L.b3, y, B, m->hid);
}

}  // namespace

extern "C" {

sge_status sge_mlp_create(uint32_t in_dim, uint32_t hidden, uint64_t seed, int device, sge_mlp **out) {
    if (!out || in_dim == 0 || hidden == 0 || in_dim > 4096 || hidden > 4096)
        return fail(SGE_BAD_INPUT, "sge_mlp_create: bad dimensions");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) { cudaGetLastError(); return fail(SGE_NO_DEVICE, "no CUDA device visible"); }
    DeviceGuard restore_device;
    CUDA_TRY(cudaSetDevice(device));
    sge_mlp *m = new sge_mlp();
    m->device = device;
    m->in = in_dim;
    m->hid = hidden;
    Layout L = layout(in_dim, hidden);
    m->np = L.n;
    std::vector<float> h(L.n, 0.f);
    Rng rng(seed);
    auto uni = [&](float a) { return (float)(((double)(rng.next() >> 11) / 9007199254740992.0) * 2.0 - 1.0) * a; };
    const float s1 = std::sqrt(6.f / (in_dim + hidden)), s2 = std::sqrt(6.f / (2.f * hidden)), s3 = std::sqrt(6.f / (hidden + 1.f));
    for (size_t i = 0; i < (size_t)hidden * in_dim; ++i) h[L.w1 + i] = uni(s1);
    for (size_t i = 0; i < (size_t)hidden * hidden; ++i) h[L.w2 + i] = uni(s2);
    for (size_t i = 0; i < hidden; ++i) h[L.w3 + i] = uni(s3);
    cudaError_t e;
    if ((e = cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking)) != cudaSuccess ||
        (e = cudaMalloc(&m->d_p, 4 * L.n * sizeof(float))) != cudaSuccess ||
        (e = cudaMalloc(&m->d_w1h, sizeof(__nv_bfloat16) * hidden * in_dim)) != cudaSuccess ||
        (e = cudaMalloc(&m->d_w2h, sizeof(__nv_bfloat16) * hidden * hidden)) != cudaSuccess) {
        sge_mlp_destroy(m);
        return fail(SGE_OOM, "sge_mlp_create: %s", cudaGetErrorString(e));
    }
    m->d_g = m->d_p + L.n;
    m->d_m = m->d_g + L.n;
    m->d_v = m->d_m + L.n;
    cudaMemcpy(m->d_p, h.data(), L.n * sizeof(float), cudaMemcpyHostToDevice);
    cudaMemset(m->d_m, 0, 2 * L.n * sizeof(float));
    *out = m;
    return SGE_OK;
}

sge_status sge_mlp_destroy(sge_mlp *m) {
    if (!m) return SGE_OK;
    DeviceGuard restore_device;
    cudaSetDevice(m->device);
    if (m->stream) cudaStreamSynchronize(m->stream);
    cudaFree(m->d_p);
    cudaFree(m->d_w1h);
    cudaFree(m->d_w2h);
    cudaFree(m->d_ws);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
    return SGE_OK;
}

sge_status sge_mlp_num_params(const sge_mlp *m, size_t *n) {
    if (!m || !n) return fail(SGE_BAD_INPUT, "null argument");
    *n = m->np;
    return SGE_OK;
}

sge_status sge_mlp_get_params(const sge_mlp *m, float *out) {
    if (!m || !out) return fail(SGE_BAD_INPUT, "null argument");
    DeviceGuard restore_device;
    CUDA_TRY(cudaSetDevice(m->device));
    CUDA_TRY(cudaMemcpy(out, m->d_p, m->np * sizeof(float), cudaMemcpyDeviceToHost));
    return SGE_OK;
}

sge_status sge_mlp_set_params(sge_mlp *m, const float *in) {
    if (!m || !in) return fail(SGE_BAD_INPUT, "null argument");
    DeviceGuard restore_device;
    CUDA_TRY(cudaSetDevice(m->device));
    CUDA_TRY(cudaMemcpy(m->d_p, in, m->np * sizeof(float), cudaMemcpyHostToDevice));
    m->bf16_stale = true;
    m->adam_t = 0;
    CUDA_TRY(cudaMemset(m->d_m, 0, 2 * m->np * sizeof(float)));
    return SGE_OK;
}

sge_status sge_mlp_forward(sge_mlp *m, const float *x, uint32_t B, float *y) {
    if (!m || (!x && B) || (!y && B)) return fail(SGE_BAD_INPUT, "null argument");
    if (B == 0) return SGE_OK;
    DeviceGuard restore_device;
    CUDA_TRY(cudaSetDevice(m->device));
    sge_status st = ensure_ws(m, B);
    if (st != SGE_OK) return st;
    Layout L = layout(m->in, m->hid);
    float *X = m->d_ws, *Z1 = X + (size_t)B * m->in, *A1 = Z1 + (size_t)B * m->hid, *Z2 = A1 + (size_t)B * m->hid,
          *A2 = Z2 + (size_t)B * m->hid, *Y = A2 + (size_t)B * m->hid;
    CUDA_TRY(cudaMemcpyAsync(X, x, sizeof(float) * B * m->in, cudaMemcpyHostToDevice, m->stream));
    forward_fp32(m, L, X, Z1, A1, Z2, A2, Y, B);
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaMemcpyAsync(y, Y, sizeof(float) * B, cudaMemcpyDeviceToHost, m->stream));
    CUDA_TRY(cudaStreamSynchronize(m->stream));
    return SGE_OK;
}

sge_status sge_mlp_forward_bf16(sge_mlp *m, const float *x, uint32_t B, float *y) {
    if (!m || (!x && B) || (!y && B)) return fail(SGE_BAD_INPUT, "null argument");
    if (B == 0) return SGE_OK;
    DeviceGuard restore_device;
    CUDA_TRY(cudaSetDevice(m->device));
    sge_status st = ensure_ws(m, B);
    if (st != SGE_OK) return st;
    Layout L = layout(m->in, m->hid);
    if (m->bf16_stale) {
        size_t n1 = (size_t)m->hid * m->in, n2 = (size_t)m->hid * m->hid;
        to_bf16<<<(unsigned)((n1 + 255) / 256), 256, 0, m->stream>>>(m->d_p + L.w1, m->d_w1h, n1);
        to_bf16<<<(unsigned)((n2 + 255) / 256), 256, 0, m->stream>>>(m->d_p + L.w2, m->d_w2h, n2);
        m->bf16_stale = false;
    }
    if (fused(m)) {
        float *X = m->d_ws, *Y = X + (size_t)B * m->in;
        CUDA_TRY(cudaFuncSetAttribute(bf16_forward_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BfSmem)));
        CUDA_TRY(cudaMemcpyAsync(X, x, sizeof(float) * B * m->in, cudaMemcpyHostToDevice, m->stream));
        bf16_forward_fused<<<(B + BF_ROWS - 1) / BF_ROWS, 128, sizeof(BfSmem), m->stream>>>(
            X, m->d_w1h, m->d_p + L.b1, m->d_w2h, m->d_p + L.b2, m->d_p + L.w3, m->d_p + L.b3, Y, (int)B, (int)m->in,
            (int)m->hid);
        CUDA_TRY(cudaGetLastError());
        CUDA_TRY(cudaMemcpyAsync(y, Y, sizeof(float) * B, cudaMemcpyDeviceToHost, m->stream));
        CUDA_TRY(cudaStreamSynchronize(m->stream));
        return SGE_OK;
    }
    // workspace reuse: X (fp32) | Xh | A1h | A2 (fp32) | y
    float *X = m->d_ws;
    __nv_bfloat16 *Xh = reinterpret_cast<__nv_bfloat16 *>(X + (size_t)B * m->in);
    __nv_bfloat16 *A1h = Xh + (size_t)B * m->in + 8;
    float *A2 = reinterpret_cast<float *>(A1h + (size_t)B * m->hid + 8);
    A2 = reinterpret_cast<float *>((reinterpret_cast<uintptr_t>(A2) + 15) & ~(uintptr_t)15);
    float *Y = A2 + (size_t)B * m->hid;
    CUDA_TRY(cudaMemcpyAsync(X, x, sizeof(float) * B * m->in, cudaMemcpyHostToDevice, m->stream));
    size_t nx = (size_t)B * m->in;
    to_bf16<<<(unsigned)((nx + 255) / 256), 256, 0, m->stream>>>(X, Xh, nx);
    const int tiles = ((B + 15) / 16) * ((m->hid + 7) / 8);
    const int threads = 128, blocks = (tiles * 32 + threads - 1) / threads;
    bf16_linear<<<blocks, threads, 0, m->stream>>>(Xh, m->d_w1h, m->d_p + L.b1, nullptr, A1h, B, m->hid, m->in, 1);
    bf16_linear<<<blocks, threads, 0, m->stream>>>(A1h, m->d_w2h, m->d_p + L.b2, A2, nullptr, B, m->hid, m->hid, 1);
    dot_out<<<(B + 255) / 256, 256, 0, m->stream>>>(A2, m->d_p + L.w3, m->d_p + L.b3, Y, B, m->hid);
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaMemcpyAsync(y, Y, sizeof(float) * B, cudaMemcpyDeviceToHost, m->stream));
    CUDA_TRY(cudaStreamSynchronize(m->stream));
    return SGE_OK;
}

// Workspace of a fused batch: its rows and labels, activations and gradients
// at the layers, one loss (ensure_ws(B) holds it).
struct TrainBufs {
    float *x, *X, *A1, *A2, *dZ1, *dZ2, *t, *dY, *loss;
};
static TrainBufs train_bufs(sge_mlp *m, uint32_t B) {
    const size_t bi = (size_t)B * m->in, bh = (size_t)B * m->hid;
    TrainBufs b;
    b.X = b.x = m->d_ws;   // (a batch that is already in order gathers onto itself)
    b.A1 = b.X + bi;
    b.A2 = b.A1 + bh;
    b.dZ1 = b.A2 + bh;
    b.dZ2 = b.dZ1 + bh;
    b.t = b.dZ2 + bh;
    b.dY = b.t + B;
    b.loss = b.dY + B;
    return b;
}
// One batch: rows forward and back, then the gradient into G, or an Adam step
// (G null).
static sge_status fused_batch(sge_mlp *m, const TrainBufs &b, const float *x, const float *t, const uint32_t *idx,
                              uint32_t B, float *loss, float *G, float lr, float c1, float c2) {
    CUDA_TRY(cudaFuncSetAttribute(train_rows_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FtSmem)));
    train_rows_fused<<<(B + FT_ROWS - 1) / FT_ROWS, FT_THREADS, sizeof(FtSmem), m->stream>>>(
        m->d_p, x, t, idx, (int)B, (int)m->in, (int)m->hid, b.X, b.A1, b.A2, b.dZ1, b.dZ2, b.dY, loss);
    CUDA_TRY(cudaFuncSetAttribute(param_grads_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PgSmem)));
    param_grads_fused<<<2 * ((m->hid + PG_OUT - 1) / PG_OUT) + (3 * m->hid + 256) / 256, 256, sizeof(PgSmem), m->stream>>>(
        b.X, b.A1, b.A2, b.dZ1, b.dZ2, b.dY, (int)B, (int)m->in, (int)m->hid, G, m->d_p, m->d_m, m->d_v, lr, c1, c2);
    CUDA_TRY(cudaGetLastError());
    return SGE_OK;
}

// Training with fused batches: the set and every epoch's order go up once, the
// batches follow each other on the stream (two launches each) and the last
// epoch's losses come back at the end.  1,152 rows, 4 epochs of 128: 36
// batches with two copies, 20 launches and a synchronisation each 4.9 ms,
// now 0.9 ms (bound by the two launches' load latency, some 11 us each).
static sge_status train_fused(sge_mlp *m, const float *x, const float *t, uint32_t n, uint32_t epochs, uint32_t batch,
                              float lr, uint64_t seed, float *final_loss) {
    batch = std::min(batch, n);
    sge_status st = ensure_ws(m, batch);
    if (st != SGE_OK) return st;
    const TrainBufs b = train_bufs(m, batch);
    const uint32_t nb = (n + batch - 1) / batch;
    // x | t | one epoch's losses | a group of epochs' orders (4 MB, or one epoch)
    const uint32_t group = std::max<uint32_t>(1, std::min<uint32_t>(epochs, (1u << 20) / n));
    const size_t floats = (size_t)n * m->in + n + nb;
    float *d = nullptr;
    CUDA_TRY(cudaMalloc(&d, 4 * (floats + (size_t)group * n)));
    float *dx = d, *dt = dx + (size_t)n * m->in, *dloss = dt + n;
    uint32_t *didx = reinterpret_cast<uint32_t *>(dloss + nb);
    std::vector<uint32_t> idx(n), orders((size_t)group * n);
    for (uint32_t i = 0; i < n; ++i) idx[i] = i;
    Rng rng(seed);
    cudaError_t e = cudaMemcpyAsync(dx, x, sizeof(float) * (size_t)n * m->in, cudaMemcpyHostToDevice, m->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dt, t, sizeof(float) * n, cudaMemcpyHostToDevice, m->stream);
    for (uint32_t ep = 0; ep < epochs && st == SGE_OK && e == cudaSuccess; ++ep) {
        if (ep % group == 0) {
            if (ep) e = cudaStreamSynchronize(m->stream);   // (the last group's orders are in use until then)
            const uint32_t some = std::min(group, epochs - ep);
            for (uint32_t q = 0; q < some; ++q) {
                for (uint32_t i = n - 1; i > 0; --i) std::swap(idx[i], idx[(uint32_t)rng.below(i + 1)]);
                memcpy(&orders[(size_t)q * n], idx.data(), 4 * (size_t)n);
            }
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(didx, orders.data(), 4 * (size_t)some * n, cudaMemcpyHostToDevice, m->stream);
        }
        if (e == cudaSuccess) e = cudaMemsetAsync(dloss, 0, sizeof(float) * nb, m->stream);
        for (uint32_t q = 0; q < nb && st == SGE_OK && e == cudaSuccess; ++q) {
            const uint32_t s = q * batch, B = std::min(batch, n - s);
            ++m->adam_t;
            const float b1 = 0.9f, b2 = 0.999f;
            const float c1 = 1.f - std::pow(b1, (float)m->adam_t), c2 = 1.f - std::pow(b2, (float)m->adam_t);
            st = fused_batch(m, b, dx, dt, didx + (size_t)(ep % group) * n + s, B, dloss + q, nullptr, lr, c1, c2);
        }
    }
    std::vector<float> losses(nb, 0.f);
    if (st == SGE_OK && e == cudaSuccess && epochs)
        e = cudaMemcpyAsync(losses.data(), dloss, sizeof(float) * nb, cudaMemcpyDeviceToHost, m->stream);
    const cudaError_t e2 = cudaStreamSynchronize(m->stream);
    cudaFree(d);
    m->bf16_stale = true;
    if (st != SGE_OK) return st;
    if (e != cudaSuccess || e2 != cudaSuccess)
        return fail(SGE_CUDA_ERROR, "sge_mlp_train: %s", cudaGetErrorString(e != cudaSuccess ? e : e2));
    double sum = 0;
    for (float l : losses) sum += l;
    if (final_loss) *final_loss = epochs ? (float)(sum / nb) : 0.f;
    return SGE_OK;
}

// Loss 0.5·mean((f(x)-t)²) and its gradient (flat, parameter layout) for one batch.
static sge_status loss_grad_dev(sge_mlp *m, const float *x, const float *t, uint32_t B, float *loss_out,
                                bool copy_grads, float *grads_out) {
    sge_status st = ensure_ws(m, B);
    if (st != SGE_OK) return st;
    Layout L = layout(m->in, m->hid);
    const uint32_t H = m->hid;
    if (fused(m)) {
        TrainBufs b = train_bufs(m, B);
        CUDA_TRY(cudaMemcpyAsync(b.x, x, sizeof(float) * B * m->in, cudaMemcpyHostToDevice, m->stream));
        CUDA_TRY(cudaMemcpyAsync(b.t, t, sizeof(float) * B, cudaMemcpyHostToDevice, m->stream));
        CUDA_TRY(cudaMemsetAsync(b.loss, 0, sizeof(float), m->stream));
        if ((st = fused_batch(m, b, b.x, b.t, nullptr, B, b.loss, m->d_g, 0.f, 1.f, 1.f)) != SGE_OK) return st;
        if (loss_out) CUDA_TRY(cudaMemcpyAsync(loss_out, b.loss, sizeof(float), cudaMemcpyDeviceToHost, m->stream));
        if (copy_grads && grads_out)
            CUDA_TRY(cudaMemcpyAsync(grads_out, m->d_g, sizeof(float) * m->np, cudaMemcpyDeviceToHost, m->stream));
        CUDA_TRY(cudaStreamSynchronize(m->stream));
        return SGE_OK;
    }
    float *X = m->d_ws, *Z1 = X + (size_t)B * m->in, *A1 = Z1 + (size_t)B * H, *Z2 = A1 + (size_t)B * H,
          *A2 = Z2 + (size_t)B * H, *Y = A2 + (size_t)B * H, *T = Y + B, *dY = T + B, *dA = dY + B,
          *loss = dA + (size_t)B * H;
    CUDA_TRY(cudaMemcpyAsync(X, x, sizeof(float) * B * m->in, cudaMemcpyHostToDevice, m->stream));
    CUDA_TRY(cudaMemcpyAsync(T, t, sizeof(float) * B, cudaMemcpyHostToDevice, m->stream));
    CUDA_TRY(cudaMemsetAsync(loss, 0, sizeof(float), m->stream));
    forward_fp32(m, L, X, Z1, A1, Z2, A2, Y, B);
    mse_grad<<<(B + 255) / 256, 256, 0, m->stream>>>(Y, T, dY, loss, (int)B);
    float *G = m->d_g;
    const dim3 blk(TILE, TILE);
    // layer 3: dW3[j] = Σ_i A2[i][j] dY[i] ; db3 = Σ dY ; dA2 = dY w3ᵀ
    sgemm<true, false><<<gemm_grid(H, 1), blk, 0, m->stream>>>(A2, dY, G + L.w3, H, 1, B, nullptr, 0, 0.f);
    colsum<<<1, 32, 0, m->stream>>>(dY, G + L.b3, B, 1);
    sgemm<false, false><<<gemm_grid(B, H), blk, 0, m->stream>>>(dY, m->d_p + L.w3, dA, B, H, 1, nullptr, 0, 0.f);
    size_t nh = (size_t)B * H;
    relu_grad<<<(unsigned)((nh + 255) / 256), 256, 0, m->stream>>>(dA, Z2, nh);  // dZ2
    // layer 2: dW2 = dZ2ᵀ A1 ; db2 = colsum dZ2 ; dA1 = dZ2 W2
    sgemm<true, false><<<gemm_grid(H, H), blk, 0, m->stream>>>(dA, A1, G + L.w2, H, H, B, nullptr, 0, 0.f);
    colsum<<<(H + 127) / 128, 128, 0, m->stream>>>(dA, G + L.b2, B, H);
    float *dA1 = Z2;  // Z2 no longer needed once dZ2 exists: reuse its storage
    sgemm<false, false><<<gemm_grid(B, H), blk, 0, m->stream>>>(dA, m->d_p + L.w2, dA1, B, H, H, nullptr, 0, 0.f);
    relu_grad<<<(unsigned)((nh + 255) / 256), 256, 0, m->stream>>>(dA1, Z1, nh);  // dZ1
    // layer 1: dW1 = dZ1ᵀ X ; db1 = colsum dZ1
    sgemm<true, false><<<gemm_grid(H, m->in), blk, 0, m->stream>>>(dA1, X, G + L.w1, H, m->in, B, nullptr, 0, 0.f);
    colsum<<<(H + 127) / 128, 128, 0, m->stream>>>(dA1, G + L.b1, B, H);
    CUDA_TRY(cudaGetLastError());
    if (loss_out) CUDA_TRY(cudaMemcpyAsync(loss_out, loss, sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    if (copy_grads && grads_out)
        CUDA_TRY(cudaMemcpyAsync(grads_out, G, sizeof(float) * m->np, cudaMemcpyDeviceToHost, m->stream));
    CUDA_TRY(cudaStreamSynchronize(m->stream));
    return SGE_OK;
}

sge_status sge_mlp_loss_grad(sge_mlp *m, const float *x, const float *t, uint32_t B, float *loss, float *grads) {
    if (!m || !x || !t || B == 0) return fail(SGE_BAD_INPUT, "sge_mlp_loss_grad: bad argument");
    DeviceGuard restore_device;
    CUDA_TRY(cudaSetDevice(m->device));
    return loss_grad_dev(m, x, t, B, loss, true, grads);
}

sge_status sge_mlp_train(sge_mlp *m, const float *x, const float *t, uint32_t n, uint32_t epochs, uint32_t batch,
                         float lr, uint64_t seed, float *final_loss) {
    if (!m || !x || !t || n == 0 || batch == 0) return fail(SGE_BAD_INPUT, "sge_mlp_train: bad argument");
    DeviceGuard restore_device;
    CUDA_TRY(cudaSetDevice(m->device));
    if (fused(m)) return train_fused(m, x, t, n, epochs, batch, lr, seed, final_loss);
    std::vector<uint32_t> idx(n);
    for (uint32_t i = 0; i < n; ++i) idx[i] = i;
    std::vector<float> bx((size_t)batch * m->in), bt(batch);
    Rng rng(seed);
    float last = 0.f;
    for (uint32_t ep = 0; ep < epochs; ++ep) {
        for (uint32_t i = n - 1; i > 0; --i) std::swap(idx[i], idx[(uint32_t)rng.below(i + 1)]);
        double ep_loss = 0;
        uint32_t nb = 0;
        for (uint32_t s = 0; s < n; s += batch) {
            const uint32_t B = std::min(batch, n - s);
            for (uint32_t r = 0; r < B; ++r) {
                memcpy(&bx[(size_t)r * m->in], x + (size_t)idx[s + r] * m->in, sizeof(float) * m->in);
                bt[r] = t[idx[s + r]];
            }
            float loss = 0.f;
            sge_status st = loss_grad_dev(m, bx.data(), bt.data(), B, &loss, false, nullptr);
            if (st != SGE_OK) return st;
            ++m->adam_t;
            const float b1 = 0.9f, b2 = 0.999f;
            const float c1 = 1.f - std::pow(b1, (float)m->adam_t), c2 = 1.f - std::pow(b2, (float)m->adam_t);
            adam<<<(unsigned)((m->np + 255) / 256), 256, 0, m->stream>>>(m->d_p, m->d_g, m->d_m, m->d_v, m->np, lr,
                                                                          b1, b2, 1e-8f, c1, c2);
            ep_loss += loss;
            ++nb;
        }
        last = (float)(ep_loss / std::max(nb, 1u));
    }
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaStreamSynchronize(m->stream));
    m->bf16_stale = true;
    if (final_loss) *final_loss = last;
    return SGE_OK;
}

}  // extern "C"
