// mlp.cu - FP32 surrogate network of include/orkan_mlp.h: tiled GEMMs with fused bias/GELU
// epilogues, deterministic reductions, Adam, minibatch gather, a captured training step and
// input-space ascent for proposals.  Everything runs in the caller's stream.
#include "../../../include/orkan_mlp.h"

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <vector>

namespace {

std::atomic<unsigned long long> g_launches{0};

constexpr int kBM = 64, kBN = 64, kBK = 16, kGemmThreads = 256;   // default tile; 32 x 32 for small grids
constexpr float kInvSqrt2 = 0.70710678118654752440f;
constexpr float kInvSqrt2Pi = 0.39894228040143267794f;

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * kInvSqrt2)); }
__device__ __forceinline__ float gelu_grad(float z) {
    return 0.5f * (1.0f + erff(z * kInvSqrt2)) + z * kInvSqrt2Pi * expf(-0.5f * z * z);
}
// Both from one erff.
__device__ __forceinline__ void gelu_both(float z, float& act, float& slope) {
    const float e = 1.0f + erff(z * kInvSqrt2);
    act = 0.5f * z * e;
    slope = 0.5f * e + z * kInvSqrt2Pi * expf(-0.5f * z * z);
}

enum Epi : int { kEpiStore = 0, kEpiBiasGelu = 1, kEpiGeluBack = 2 };

// C[m][n] = sum_k opA[m][k] opB[k][n];  opA[m][k] = TA ? A[k][m] : A[m][k],
// opB[k][n] = TB ? B[n][k] : B[k][n] (row-major with leading dimensions lda, ldb).
// Epilogues: store; z = acc + bias[n] into C and gelu(z) into out2; acc * gelu'(aux[m][n]).
// Each output is one thread's fixed-order sum over k, so results are deterministic.
template <bool TA, bool TB, int EPI, int kBM = 64, int kBN = 64>
__global__ void __launch_bounds__(kGemmThreads) k_gemm(int M, int N, int K, const float* __restrict__ A, int lda,
                                                       const float* __restrict__ B, int ldb, float* __restrict__ C,
                                                       int ldc, const float* __restrict__ bias,
                                                       const float* __restrict__ aux, float* __restrict__ out2) {
    constexpr int TM = kBM / 16, TN = kBN / 16;          // outputs per thread: TM x TN
    __shared__ float As[kBK][kBM + 4];
    __shared__ float Bs[kBK][kBN + 4];
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const int m0 = blockIdx.y * kBM, n0 = blockIdx.x * kBN;
    // split over k (gridDim.z slices of whole kBK tiles): slice z sums its own k range and
    // stores to its own M x ldc plane of C
    const int ktiles = (K + kBK - 1) / kBK, per = (ktiles + gridDim.z - 1) / gridDim.z;
    const int kbeg = blockIdx.z * per * kBK, kend = min(K, (int)(blockIdx.z + 1) * per * kBK);
    C += (size_t)blockIdx.z * M * ldc;
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
    for (int k0 = kbeg; k0 < kend; k0 += kBK) {
        for (int e = threadIdx.x; e < kBM * kBK; e += kGemmThreads) {
            const int mm = TA ? e % kBM : e / kBK, kk = TA ? e / kBM : e % kBK;
            const int gm = m0 + mm, gk = k0 + kk;
            float v = 0.f;
            if (gm < M && gk < kend) v = TA ? A[(size_t)gk * lda + gm] : A[(size_t)gm * lda + gk];
            As[kk][mm] = v;
        }
        for (int e = threadIdx.x; e < kBN * kBK; e += kGemmThreads) {
            const int nn = TB ? e / kBK : e % kBN, kk = TB ? e % kBK : e / kBN;
            const int gn = n0 + nn, gk = k0 + kk;
            float v = 0.f;
            if (gn < N && gk < kend) v = TB ? B[(size_t)gn * ldb + gk] : B[(size_t)gk * ldb + gn];
            Bs[kk][nn] = v;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kBK; ++kk) {
            float a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[kk][ty + 16 * i];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = Bs[kk][tx + 16 * j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int m = m0 + ty + 16 * i, n = n0 + tx + 16 * j;
            if (m >= M || n >= N) continue;
            const size_t o = (size_t)m * ldc + n;
            if (EPI == kEpiStore) {
                C[o] = acc[i][j];
            } else if (EPI == kEpiBiasGelu) {
                const float z = acc[i][j] + bias[n];
                C[o] = z;
                out2[o] = gelu(z);
            } else {
                C[o] = acc[i][j] * gelu_grad(aux[o]);
            }
        }
}

// out[i] = sum over the slices z < nz of part[z * count + i], in slice order.
__global__ void k_sum_slices(const float* __restrict__ part, int nz, size_t count, float* __restrict__ out) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    float s = 0.f;
    for (int z = 0; z < nz; ++z) s += part[(size_t)z * count + i];
    out[i] = s;
}

// y[b] = sum_h A[b][h] w[h] + w0, one warp per row, fixed shuffle tree.
__global__ void k_rowdot(const float* __restrict__ A, int rows, int h, const float* __restrict__ w,
                         const float* __restrict__ w0, float* __restrict__ y) {
    const int row = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32, lane = threadIdx.x % 32;
    if (row >= rows) return;
    float s = 0.f;
    for (int k = lane; k < h; k += 32) s = fmaf(A[(size_t)row * h + k], w[k], s);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) y[row] = s + w0[0];
}

// dy[b] = 2 (y[b] - t[b]) / batch (or 1 when t is NULL: the gradient of f itself);
// loss_slot[0] = mean squared error (one block, fixed order).
__global__ void k_loss(const float* __restrict__ y, const float* __restrict__ t, int batch, float* __restrict__ dy,
                       float* __restrict__ loss_slot) {
    __shared__ float red[1024];
    float s = 0.f;
    for (int b = threadIdx.x; b < batch; b += blockDim.x) {
        if (t) {
            const float d = y[b] - t[b];
            dy[b] = 2.0f * d / (float)batch;
            s = fmaf(d, d, s);
        } else {
            dy[b] = 1.0f;
        }
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0 && loss_slot) loss_slot[0] = red[0] / (float)batch;
}

// out[n] = sum_m X[m][n] v[m] (v == NULL: 1), in a fixed order: a block of 32 columns x 32 row
// lanes, lane l takes rows l, l + 32, ..., and the lanes' sums are added in lane order.  (One
// thread per column walked the 1024 rows of a batch in 23-44 us.)
constexpr int kColRows = 32;
__global__ void __launch_bounds__(32 * kColRows) k_colsum(const float* __restrict__ X, int rows, int cols,
                                                          const float* __restrict__ v, float* __restrict__ out) {
    __shared__ float sh[kColRows][33];
    const int n = blockIdx.x * 32 + threadIdx.x;
    float s = 0.f;
    if (n < cols)
        for (int m = threadIdx.y; m < rows; m += kColRows)
            s = v ? fmaf(X[(size_t)m * cols + n], v[m], s) : s + X[(size_t)m * cols + n];
    sh[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y == 0 && n < cols) {
        for (int l = 1; l < kColRows; ++l) s += sh[l][threadIdx.x];
        out[n] = s;
    }
}

// dZ2[b][h] = dy[b] w3[h] gelu'(Z2[b][h])
__global__ void k_outer_gelu(const float* __restrict__ dy, const float* __restrict__ w, const float* __restrict__ Z,
                             int rows, int cols, float* __restrict__ out) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)rows * cols) return;
    const int b = (int)(i / cols), h = (int)(i % cols);
    out[i] = dy[b] * w[h] * gelu_grad(Z[i]);
}

__global__ void k_step_begin(unsigned* step) {
    ++step[0];
    ++step[1];
}

// Adam with bias correction at step t = step[0] (1-based, all steps of the network).
__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m1,
                       float* __restrict__ m2, size_t count, float lr, const unsigned* __restrict__ step) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const float t = (float)step[0];
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float mi = b1 * m1[i] + (1.0f - b1) * g[i];
    const float vi = b2 * m2[i] + (1.0f - b2) * g[i] * g[i];
    m1[i] = mi;
    m2[i] = vi;
    const float mh = mi / (1.0f - powf(b1, t)), vh = vi / (1.0f - powf(b2, t));
    p[i] -= lr * mh / (sqrtf(vh) + eps);
}

// Adam ascent on inputs, clamped to [lo, hi].
__global__ void k_adam_inputs(float* __restrict__ x, const float* __restrict__ g, float* __restrict__ m1,
                              float* __restrict__ m2, size_t count, float lr, int t, float lo, float hi) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float mi = b1 * m1[i] + (1.0f - b1) * g[i];
    const float vi = b2 * m2[i] + (1.0f - b2) * g[i] * g[i];
    m1[i] = mi;
    m2[i] = vi;
    const float mh = mi / (1.0f - powf(b1, (float)t)), vh = vi / (1.0f - powf(b2, (float)t));
    x[i] = fminf(hi, fmaxf(lo, x[i] + lr * mh / (sqrtf(vh) + eps)));
}

__host__ __device__ inline uint64_t mix64(uint64_t z) {
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
__host__ __device__ inline uint64_t gcd64(uint64_t a, uint64_t b) {
    while (b) { const uint64_t t = a % b; a = b; b = t; }
    return a;
}

// Minibatch of the current step (schedule counter step[1], 1-based): epoch e = (s - 1) / spe,
// position j = (s - 1) % spe; sample i of the epoch is (a_e i + c_e) mod count.
__global__ void k_gather(const float* __restrict__ X, const float* __restrict__ T, unsigned count, int n_in, int batch,
                         unsigned spe, uint64_t seed, const unsigned* __restrict__ step, float* __restrict__ xb,
                         float* __restrict__ tb) {
    const unsigned s = step[1] - 1, e = s / spe, j = s % spe;
    uint64_t a = mix64(seed ^ (0x5851f42d4c957f2dull * (e + 1))) % count;
    if (a == 0) a = 1;
    while (gcd64(a, count) != 1) a = (a + 1) % count == 0 ? 1 : a + 1;
    const uint64_t c = mix64(seed + 0x632be59bd9b4e019ull * (e + 1)) % count;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < batch; r += gridDim.x * blockDim.x) {
        const uint64_t i = (uint64_t)j * batch + r;
        const uint64_t src = (a * i + c) % count;
        for (int k = 0; k < n_in; ++k) xb[(size_t)r * n_in + k] = X[src * n_in + k];
        tb[r] = T[src];
    }
}

// Mean of the per-step losses of the last epoch.
__global__ void k_epoch_loss(const float* __restrict__ losses, unsigned spe, float* __restrict__ out) {
    float s = 0.f;
    for (unsigned k = 0; k < spe; ++k) s += losses[k];
    out[0] = s / (float)spe;
}

__global__ void k_copy_loss(const float* __restrict__ src, const unsigned* __restrict__ step, unsigned spe,
                            float* __restrict__ losses) {
    losses[(step[1] - 1) % spe] = src[0];
}

// ---- networks of 256 hidden units and at most 64 inputs -----------------------------------
// The whole layer width fits one block, so a block carries a tile of rows through the network in
// shared memory and registers: forward only (k_rows<RG, false>), or forward and backward up to
// dL/dz1, dL/dz2 and dL/dx (k_rows<RG, true>); k_wgrad forms the weight gradients (reductions over
// the rows) in k slices and k_reduce adds slices and per-tile column sums in order.
//
// A thread computes 8 rows x RG columns (columns lane + 32 c of its warp's range); 8 / RG warps cover
// the 256 columns of 8 rows, so a tile has BM = 8 RG rows.  Rows are the fastest index of the
// staged activations: their 8 values per k are two broadcast 16-byte loads and come as pairs for
// fma.rn.f32x2 (two FMAs per instruction, each rounded as fmaf).  Tall tiles raise the work per
// staged weight, short ones the number of blocks: see rows_tile.
//
// Bound: FP32 FMAs (60 us for 32768 rows at 74 TFLOP/s) for tall tiles; latency for one batch, where an
// SM has one 8-row tile.  Measured against one tiled GEMM, row dot and column sum after the other:
// forward of 32768 rows 131 us (32 calls of 1024 rows: 1115 us), gradients of 1024 rows 67 us with the
// host's part (264 us), of which k_rows 21 us, k_wgrad 7.7 us and k_reduce 2.9 us, a training step of
// 1024 rows 44 us (210 us).
constexpr int kFH = 256, kFMaxIn = 64, kFThreads = 256, kFK = 16, kFP = 260, kFPT = 258;

struct RowsArgs {
    const float *x, *t;                 // t NULL with backward: gradient of f itself (dy = 1)
    int rows, n_in;
    const float *W1, *b1, *W2, *b2, *w3, *b3;
    float* y;                           // f(x), may be NULL with backward
    float *A1, *dZ1, *dZ2, *gx;         // backward outputs; gx may be NULL
    float *colp;                        // [db1, db2, dw3][part][256]: sums over 8 rows each
    float *rowp;                        // [loss, db3][tile]
    int parts, tiles;
};

__device__ __forceinline__ unsigned long long pack2(float v) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float half_of(unsigned long long v, int i) {
    return __uint_as_float((unsigned)(i ? v >> 32 : v & 0xffffffffull));
}
__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

// acc[rows 8][columns RG] += A[k][rows] W[k][columns] over kFK staged k: A at (k BM), W at (k pitch).
template <int RG>
__device__ __forceinline__ void rows_mma(unsigned long long (&acc)[4][RG], const float* A, const float* W, int pitch) {
    constexpr int BM = 8 * RG;
#pragma unroll
    for (int k = 0; k < kFK; ++k) {
        const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(A + k * BM);
        const ulonglong2 a1 = *reinterpret_cast<const ulonglong2*>(A + k * BM + 4);
#pragma unroll
        for (int c = 0; c < RG; ++c) {
            const unsigned long long w = pack2(W[k * pitch + 32 * c]);
            fma2(acc[0][c], a0.x, w);
            fma2(acc[1][c], a0.y, w);
            fma2(acc[2][c], a1.x, w);
            fma2(acc[3][c], a1.y, w);
        }
    }
}

// An 8-row tile has one column per thread in that form, and five shared-memory wavefronts for eight FMAs a
// lane.  There the k of a chunk are split over four groups of two warps instead, a thread takes 4 columns
// (8 wavefronts for 32 FMAs), and the four partial sums meet in shared memory in the order of k
// (k_rows<1, true> of 1024 rows 28.3 -> 20.8 us, with the biases and W1 fetched ahead; forward 14.6 -> 12.6 us).
// acc[row pair][column c]: columns of the forward pass 128 half + 4 lane + c (a 16-byte load per k), of the
// backward pass 128 half + lane + 32 c, whose W2 rows are staged as they lie, kFS floats apart (a 16-byte
// load is four k of one column, and 8 lanes fall on all banks).
constexpr int kFS = 20, kFSlot = 34;
__device__ __forceinline__ void split_fma(unsigned long long (&acc)[4][4], const float* A, int c, float w) {
    const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(A), a1 = *reinterpret_cast<const ulonglong2*>(A + 4);
    const unsigned long long ww = pack2(w);
    fma2(acc[0][c], a0.x, ww);
    fma2(acc[1][c], a0.y, ww);
    fma2(acc[2][c], a1.x, ww);
    fma2(acc[3][c], a1.y, ww);
}
__device__ __forceinline__ void split_forward(unsigned long long (&acc)[4][4], const float* A, const float* W) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float4 w = *reinterpret_cast<const float4*>(W + k * kFP);
        split_fma(acc, A + k * 8, 0, w.x);
        split_fma(acc, A + k * 8, 1, w.y);
        split_fma(acc, A + k * 8, 2, w.z);
        split_fma(acc, A + k * 8, 3, w.w);
    }
}
__device__ __forceinline__ void split_backward(unsigned long long (&acc)[4][4], const float* A, const float* W) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const float4 w = *reinterpret_cast<const float4*>(W + 32 * c * kFS);
        split_fma(acc, A, c, w.x);
        split_fma(acc, A + 8, c, w.y);
        split_fma(acc, A + 16, c, w.z);
        split_fma(acc, A + 24, c, w.w);
    }
}
// The sums over the four groups, for column tid: slot (half, c) starts at 34 (4 half + c) and holds one
// 16-byte element per lane, so that the reads of either column order are free of conflicts.
template <bool FWD>
__device__ __forceinline__ void split_sum(const unsigned long long (&acc)[4][4], float* P, unsigned long long (&out)[4][1]) {
    const int tid = threadIdx.x, lane = tid % 32, warp = tid / 32;
    ulonglong2* B = reinterpret_cast<ulonglong2*>(P);
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int q = 0; q < 2; ++q)
            B[(warp / 2 * 2 + q) * 8 * kFSlot + (warp % 2 * 4 + c) * kFSlot + lane] =
                make_ulonglong2(acc[2 * q][c], acc[2 * q + 1][c]);
    __syncthreads();
    const int slot = FWD ? (tid / 128 * 4 + tid % 4) * kFSlot + tid % 128 / 4 : tid / 32 * kFSlot + tid % 32;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        ulonglong2 s = B[q * 8 * kFSlot + slot];
#pragma unroll
        for (int g = 1; g < 4; ++g) {
            const ulonglong2 v = B[(2 * g + q) * 8 * kFSlot + slot];
            s.x = add2(s.x, v.x);
            s.y = add2(s.y, v.y);
        }
        out[2 * q][0] = s.x;
        out[2 * q + 1][0] = s.y;
    }
}

// W2 chunks in shared memory: three for the 8-row tiles (two of them on their way), else two.
template <int RG>
constexpr int kFChunk = RG == 1 ? kFH * kFS : kFK * kFP;
template <int RG>
constexpr int kFChunks = RG == 1 ? 3 : 2;
template <int RG>
size_t rows_smem(int n_in) {
    return sizeof(float) * (size_t)(kFP * 8 * RG + kFChunks<RG> * kFChunk<RG> + n_in * 8 * RG + 64 + 16 * RG);
}

template <int RG, bool BWD>
__global__ void __launch_bounds__(kFThreads, BWD && RG > 1 ? 1 : 2) k_rows(const RowsArgs a) {
    constexpr int BM = 8 * RG, CG = 8 / RG, NC = kFChunks<RG>, kW = kFChunk<RG>, kChunks = kFH / kFK;
    extern __shared__ __align__(16) float fsm[];
    float* As = fsm;                                   // [256][BM]; later dz1 as [BM][260]
    float* Ws = As + kFP * BM;                         // NC chunks of kFK rows
    float* Xs = Ws + NC * kW;                    // [n_in][BM]
    float* red = Xs + a.n_in * BM;                     // [8 warps][8 rows]
    float* dys = red + 64;                             // [BM]
    float* errs = dys + BM;                            // [BM]
    const int tid = threadIdx.x, lane = tid % 32, warp = tid / 32;
    const int rg = warp / CG, col0 = (warp % CG) * 32 * RG + lane;
    const int row0 = blockIdx.x * BM, my0 = row0 + rg * 8;
    auto load_w2 = [&](int kc, int buf) {              // W2 rows 16 kc .. + 15
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = tid + kFThreads * i, r = e / 64, c = (e % 64) * 4;
            cp_async16(Ws + buf * kW + r * kFP + c, a.W2 + (size_t)(kc * kFK + r) * kFH + c);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    auto load_w2t = [&](int kc, int buf) {             // columns 16 kc .. + 15 of W2, row by row
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = tid + kFThreads * i;
            cp_async16(Ws + buf * kW + e / 4 * kFS + e % 4 * 4, a.W2 + (size_t)(e / 4) * kFH + kc * kFK + e % 4 * 4);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
#pragma unroll
    for (int c = 0; c + 1 < NC; ++c) load_w2(c, c);
    for (int e = tid; e < a.n_in * BM; e += kFThreads) {
        const int r = e / a.n_in, k = e % a.n_in;
        Xs[k * BM + r] = row0 + r < a.rows ? a.x[(size_t)(row0 + r) * a.n_in + k] : 0.f;
    }
    __syncthreads();
    unsigned long long acc[4][RG];
    float d1[BWD ? 8 : 1][RG];                         // gelu'(z1)
    auto clear = [&] {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c < RG; ++c) acc[i][c] = 0ull;
    };
    clear();
#pragma unroll 4
    for (int k = 0; k < a.n_in; ++k) {
        const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(Xs + k * BM + rg * 8);
        const ulonglong2 a1 = *reinterpret_cast<const ulonglong2*>(Xs + k * BM + rg * 8 + 4);
#pragma unroll
        for (int c = 0; c < RG; ++c) {
            const unsigned long long w = pack2(__ldg(a.W1 + (size_t)k * kFH + col0 + 32 * c));
            fma2(acc[0][c], a0.x, w);
            fma2(acc[1][c], a0.y, w);
            fma2(acc[2][c], a1.x, w);
            fma2(acc[3][c], a1.y, w);
        }
    }
#pragma unroll
    for (int c = 0; c < RG; ++c) {
        const int col = col0 + 32 * c;
        const float bias = __ldg(a.b1 + col);
        float v[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const float z = half_of(acc[r / 2][c], r % 2) + bias;
            if (BWD) gelu_both(z, v[r], d1[r][c]);
            else v[r] = gelu(z);
            if (BWD && a.A1 && my0 + r < a.rows) a.A1[(size_t)(my0 + r) * kFH + col] = v[r];
        }
        *reinterpret_cast<float4*>(As + col * BM + rg * 8) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4*>(As + col * BM + rg * 8 + 4) = make_float4(v[4], v[5], v[6], v[7]);
    }
    clear();
    // one column per thread: its bias and output weight arrive under the product
    const float bias2 = RG == 1 ? __ldg(a.b2 + col0) : 0.f, out3 = RG == 1 ? __ldg(a.w3 + col0) : 0.f;
    const int kg = warp / 2 * 4;                       // 8-row tiles: this warp's k of a chunk, and its columns
    // every chunk by mma(its index, its buffer), the next NC - 1 on their way
    auto chunks = [&](auto& load, auto mma) {
        for (int kc = 0; kc < kChunks; ++kc) {
            asm volatile("cp.async.wait_group %0;\n" ::"n"(NC - 2) : "memory");
            __syncthreads();                           // the chunk is in, the one before it is read
            if (kc + NC - 1 < kChunks) load(kc + NC - 1, (kc + NC - 1) % NC);
            else if (NC > 2) asm volatile("cp.async.commit_group;\n" ::: "memory");
            mma(kc, Ws + kc % NC * kW);
        }
    };
    if constexpr (RG == 1) {
        unsigned long long part[4][4] = {};
        chunks(load_w2, [&](int kc, const float* W) {
            split_forward(part, As + (kc * kFK + kg) * 8, W + kg * kFP + warp % 2 * 128 + lane * 4);
        });
        __syncthreads();
        split_sum<true>(part, Ws, acc);
    } else {
        chunks(load_w2, [&](int kc, const float* W) { rows_mma<RG>(acc, As + kc * kFK * BM + rg * 8, W + col0, kFP); });
    }
    // z2 = acc + b2; y = gelu(z2) . w3 + b3, over the lanes by a fixed tree, then over the warps
    float p[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) p[r] = 0.f;
#pragma unroll
    for (int c = 0; c < RG; ++c) {
        const float bias = RG == 1 ? bias2 : __ldg(a.b2 + col0 + 32 * c), w3 = RG == 1 ? out3 : __ldg(a.w3 + col0 + 32 * c);
#pragma unroll
        for (int r = 0; r < 8; ++r) p[r] = fmaf(gelu(half_of(acc[r / 2][c], r % 2) + bias), w3, p[r]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < 8; ++r) p[r] += __shfl_xor_sync(0xffffffffu, p[r], o);
    if (lane == 0)
        for (int r = 0; r < 8; ++r) red[warp * 8 + r] = p[r];
    __syncthreads();                                   // (also: As is read)
    if (tid < BM) {
        float s = 0.f;
        for (int w = 0; w < CG; ++w) s += red[(tid / 8 * CG + w) * 8 + tid % 8];
        s += __ldg(a.b3);
        const bool live = row0 + tid < a.rows;
        if (a.y && live) a.y[row0 + tid] = s;
        if (BWD) {
            const float d = a.t && live ? s - a.t[row0 + tid] : 0.f;
            dys[tid] = !live ? 0.f : a.t ? 2.0f * d / (float)a.rows : 1.0f;
            errs[tid] = d;
        }
    }
    if constexpr (BWD) {
        if constexpr (RG == 1) {
#pragma unroll
            for (int c = 0; c + 1 < NC; ++c) load_w2t(c, c);
        }
        __syncthreads();
        if (tid == 0 && a.rowp) {
            float loss = 0.f, db3 = 0.f;
            for (int r = 0; r < BM; ++r) {
                loss = fmaf(errs[r], errs[r], loss);
                db3 += dys[r];
            }
            a.rowp[blockIdx.x] = loss;
            a.rowp[a.tiles + blockIdx.x] = db3;
        }
        const size_t part = (size_t)blockIdx.x * RG + rg;
#pragma unroll
        for (int c = 0; c < RG; ++c) {
            const int col = col0 + 32 * c;
            const float bias = RG == 1 ? bias2 : __ldg(a.b2 + col), w3 = RG == 1 ? out3 : __ldg(a.w3 + col);
            float v[8], dw3 = 0.f, db2 = 0.f;
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const float z = half_of(acc[r / 2][c], r % 2) + bias, dy = dys[rg * 8 + r];
                float act, slope;
                gelu_both(z, act, slope);
                dw3 = fmaf(act, dy, dw3);
                v[r] = dy * w3 * slope;
                db2 += v[r];
                if (a.dZ2 && my0 + r < a.rows) a.dZ2[(size_t)(my0 + r) * kFH + col] = v[r];
            }
            if (a.colp) {
                a.colp[((size_t)a.parts + part) * kFH + col] = db2;
                a.colp[(2 * (size_t)a.parts + part) * kFH + col] = dw3;
            }
            *reinterpret_cast<float4*>(As + col * BM + rg * 8) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4*>(As + col * BM + rg * 8 + 4) = make_float4(v[4], v[5], v[6], v[7]);
        }
        // dz1 = (dz2 W2^T) gelu'(z1)
        if constexpr (RG == 1) {
            unsigned long long part[4][4] = {};
            chunks(load_w2t, [&](int kc, const float* W) {
                split_backward(part, As + (kc * kFK + kg) * 8, W + (warp % 2 * 128 + lane) * kFS + kg);
            });
            __syncthreads();
            split_sum<false>(part, Ws, acc);
        } else {
            // chunk kc holds W2[:][16 kc .. + 15] transposed (pitch 258: the stores of a warp, 8 rows x 4 k,
            // fall on 32 banks)
            float4 w[4];
            auto get_t = [&](int kc) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int e = tid + kFThreads * i;
                    w[i] = __ldg(reinterpret_cast<const float4*>(a.W2 + (size_t)(e / 4) * kFH + kc * kFK + (e % 4) * 4));
                }
            };
            auto put_t = [&](int buf) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int e = tid + kFThreads * i;
                    float* d = Ws + buf * kW + (e % 4) * 4 * kFPT + e / 4;
                    d[0] = w[i].x;
                    d[kFPT] = w[i].y;
                    d[2 * kFPT] = w[i].z;
                    d[3 * kFPT] = w[i].w;
                }
            };
            get_t(0);
            put_t(0);
            clear();
            __syncthreads();
            for (int kc = 0; kc < kFH / kFK; ++kc) {
                if (kc + 1 < kFH / kFK) get_t(kc + 1);
                rows_mma<RG>(acc, As + kc * kFK * BM + rg * 8, Ws + (kc & 1) * kW + col0, kFPT);
                if (kc + 1 < kFH / kFK) put_t((kc + 1) & 1);
                __syncthreads();
            }
        }
#pragma unroll
        for (int c = 0; c < RG; ++c) {
            const int col = col0 + 32 * c;
            float db1 = 0.f;
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const float v = half_of(acc[r / 2][c], r % 2) * d1[r][c];
                db1 += v;
                if (a.dZ1 && my0 + r < a.rows) a.dZ1[(size_t)(my0 + r) * kFH + col] = v;
                if (a.gx) As[(rg * 8 + r) * kFP + col] = v;
            }
            if (a.colp) a.colp[part * kFH + col] = db1;
        }
        if (!a.gx) return;
        __syncthreads();
        for (int r = warp; r < BM; r += kFThreads / 32) {              // dL/dx[r], one warp each
            float dz[kFH / 32];
#pragma unroll
            for (int i = 0; i < kFH / 32; ++i) dz[i] = As[r * kFP + lane + 32 * i];
#pragma unroll 4
            for (int k = 0; k < a.n_in; ++k) {
                float s = 0.f;
#pragma unroll
                for (int i = 0; i < kFH / 32; ++i) s = fmaf(dz[i], __ldg(a.W1 + k * kFH + lane + 32 * i), s);
#pragma unroll
                for (int q = 16; q > 0; q >>= 1) s += __shfl_xor_sync(0xffffffffu, s, q);
                if (lane == 0 && row0 + r < a.rows) a.gx[(size_t)(row0 + r) * a.n_in + k] = s;
            }
        }
    }
}

// Weight gradients over a slice of the rows: part[z][W1 then W2] = sum over rows of slice z of
// X^T dZ1 and A1^T dZ2, in 64 x 64 tiles, 4 x 4 outputs per thread.  blockIdx.x < 4: tiles of W1 (n_in <=
// 64 inputs x 256), then the 16 tiles of W2; blockIdx.y: slice.
__global__ void __launch_bounds__(256) k_wgrad(const float* __restrict__ X, const float* __restrict__ A1,
                                               const float* __restrict__ dZ1, const float* __restrict__ dZ2, int rows,
                                               int n_in, int per, float* __restrict__ part) {
    __shared__ __align__(16) float As[2][kFK][64], Bs[2][kFK][64];
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    const bool first = blockIdx.x < 4;
    const int tile = first ? blockIdx.x : blockIdx.x - 4;
    const int i0 = first ? 0 : tile / 4 * 64, j0 = tile % 4 * 64;
    const int M = first ? n_in : kFH;
    const float* A = first ? X : A1;
    const float* B = first ? dZ1 : dZ2;
    const int rbeg = blockIdx.y * per, rend = min(rows, rbeg + per);
    float* out = part + (size_t)blockIdx.y * (n_in + kFH) * kFH + (first ? 0 : n_in * kFH);
    float4 av, bv;
    auto get = [&](int r0) {                           // one row and 4 columns of each operand per thread
        const int r = r0 + ty, c = tx * 4;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        bv = r < rend ? __ldg(reinterpret_cast<const float4*>(B + (size_t)r * kFH + j0 + c)) : zero;
        if (!first) {
            av = r < rend ? __ldg(reinterpret_cast<const float4*>(A + (size_t)r * kFH + i0 + c)) : zero;
        } else {
            const float* q = A + (size_t)r * n_in + c;
            av = zero;
            if (r < rend) {
                if (c < M) av.x = q[0];
                if (c + 1 < M) av.y = q[1];
                if (c + 2 < M) av.z = q[2];
                if (c + 3 < M) av.w = q[3];
            }
        }
    };
    auto put = [&](int buf) {
        *reinterpret_cast<float4*>(&As[buf][ty][tx * 4]) = av;
        *reinterpret_cast<float4*>(&Bs[buf][ty][tx * 4]) = bv;
    };
    float acc[4][4] = {};
    get(rbeg);
    put(0);
    __syncthreads();
    int buf = 0;
    for (int r0 = rbeg; r0 < rend; r0 += kFK, buf ^= 1) {
        const bool more = r0 + kFK < rend;
        if (more) get(r0 + kFK);
#pragma unroll
        for (int k = 0; k < kFK; ++k) {
            const float4 x = *reinterpret_cast<const float4*>(&As[buf][k][ty * 4]);
            const float4 w = *reinterpret_cast<const float4*>(&Bs[buf][k][tx * 4]);
            const float xa[4] = {x.x, x.y, x.z, x.w}, wa[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xa[i], wa[j], acc[i][j]);
        }
        if (more) put(buf ^ 1);
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = i0 + ty * 4 + i;
        if (m < M)
            *reinterpret_cast<float4*>(out + (size_t)m * kFH + j0 + tx * 4) =
                make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    }
}

// Gradient vector from the slices and the per-tile sums, each in order: blocks [0, nw) the
// weights W1 and W2, then 24 blocks of 32 columns of (b1, b2, w3), then b3 and the loss.
__global__ void __launch_bounds__(256) k_reduce(const float* __restrict__ part, int nz, const float* __restrict__ colp,
                                                int parts, const float* __restrict__ rowp, int tiles, int rows, int n_in,
                                                int nw, float* __restrict__ g, float* __restrict__ loss) {
    __shared__ float sh[256];
    const int tid = threadIdx.x, b = blockIdx.x;
    const int w1 = n_in * kFH, weights = w1 + kFH * kFH;
    if (b < nw) {
        const int i = b * 256 + tid;
        if (i >= weights) return;
        float s = 0.f;
        for (int z = 0; z < nz; ++z) s += part[(size_t)z * weights + i];
        g[i < w1 ? i : i + kFH] = s;                   // b1 lies between W1 and W2
        return;
    }
    if (b < nw + 24) {
        const int e = (b - nw) * 32 + tid % 32, kind = e / kFH, col = e % kFH, seg = tid / 32;
        float s = 0.f;
        for (int q = seg; q < parts; q += 8) s += colp[((size_t)kind * parts + q) * kFH + col];
        sh[tid] = s;
        __syncthreads();
        if (seg == 0) {
            for (int l = 1; l < 8; ++l) s += sh[l * 32 + tid];
            g[(kind == 0 ? w1 : kind == 1 ? weights + kFH : weights + 2 * kFH) + col] = s;
        }
        return;
    }
    float sl = 0.f, sb = 0.f;
    for (int q = tid; q < tiles; q += 256) {
        sl += rowp[q];
        sb += rowp[tiles + q];
    }
    for (int pass = 0; pass < 2; ++pass) {
        sh[tid] = pass ? sb : sl;
        __syncthreads();
        for (int o = 128; o > 0; o >>= 1) {
            if (tid < o) sh[tid] += sh[tid + o];
            __syncthreads();
        }
        if (tid == 0) {
            if (pass) g[weights + 3 * kFH] = sh[0];
            else if (loss) loss[0] = sh[0] / (float)rows;
        }
        __syncthreads();
    }
}

unsigned blocks(size_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

struct orkan_mlp {
    int n_in = 0, h = 0, maxb = 0;
    size_t np = 0;
    // parameter-vector offsets
    size_t oW1, ob1, oW2, ob2, oW3, ob3;
    float *P = nullptr, *G = nullptr, *M1 = nullptr, *M2 = nullptr;
    float *Z1 = nullptr, *A1 = nullptr, *Z2 = nullptr, *A2 = nullptr, *y = nullptr, *dy = nullptr;
    float *dZ2 = nullptr, *dZ1 = nullptr, *xb = nullptr, *tb = nullptr, *loss = nullptr, *losses = nullptr;
    float* split = nullptr;             // k-slice partial products of the weight gradients
    size_t split_cap = 0;
    bool fused = false;                 // 256 hidden units, few inputs: k_rows, k_wgrad, k_reduce
    float *colp = nullptr, *rowp = nullptr;   // their per-tile sums
    unsigned* step = nullptr;
    size_t losses_cap = 0;
};

namespace {

template <bool TA, bool TB, int EPI>
void gemm(cudaStream_t st, int M, int N, int K, const float* A, int lda, const float* B, int ldb, float* C, int ldc,
          const float* bias = nullptr, const float* aux = nullptr, float* out2 = nullptr) {
    const dim3 grid((N + kBN - 1) / kBN, (M + kBM - 1) / kBM);
    if (grid.x * grid.y >= 148) {
        k_gemm<TA, TB, EPI><<<grid, kGemmThreads, 0, st>>>(M, N, K, A, lda, B, ldb, C, ldc, bias, aux, out2);
    } else {                                   // 32 x 32 tiles: four times the blocks
        const dim3 g2((N + 31) / 32, (M + 31) / 32);
        k_gemm<TA, TB, EPI, 32, 32><<<g2, kGemmThreads, 0, st>>>(M, N, K, A, lda, B, ldb, C, ldc, bias, aux, out2);
    }
    ++g_launches;
}

// C[M][N] (ldc = N) = sum over a long k (the batch) of A^T B, split into k slices so that
// the grid covers the SMs; the slices are summed in order (deterministic).
void gemm_tn_split(orkan_mlp* m, cudaStream_t st, int M, int N, int K, const float* A, int lda, const float* B,
                   int ldb, float* C) {
    const int tiles = ((N + kBN - 1) / kBN) * ((M + kBM - 1) / kBM);
    int nz = (296 + tiles - 1) / tiles;
    nz = std::max(1, std::min(nz, (K + kBK - 1) / kBK));
    if (nz == 1 || (size_t)nz * M * N > m->split_cap) {
        gemm<true, false, kEpiStore>(st, M, N, K, A, lda, B, ldb, C, N);
        return;
    }
    const dim3 grid((N + kBN - 1) / kBN, (M + kBM - 1) / kBM, nz);
    k_gemm<true, false, kEpiStore><<<grid, kGemmThreads, 0, st>>>(M, N, K, A, lda, B, ldb, m->split, N, nullptr,
                                                                  nullptr, nullptr);
    const size_t cnt = (size_t)M * N;
    k_sum_slices<<<blocks(cnt, 256), 256, 0, st>>>(m->split, nz, cnt, C);
    g_launches += 2;
}

// Forward of `batch` rows of x into m->Z1, A1, Z2, A2, y.
void forward(orkan_mlp* m, const float* x, int batch, float* y, cudaStream_t st) {
    const int I = m->n_in, H = m->h;
    gemm<false, false, kEpiBiasGelu>(st, batch, H, I, x, I, m->P + m->oW1, H, m->Z1, H, m->P + m->ob1, nullptr, m->A1);
    gemm<false, false, kEpiBiasGelu>(st, batch, H, H, m->A1, H, m->P + m->oW2, H, m->Z2, H, m->P + m->ob2, nullptr,
                                     m->A2);
    k_rowdot<<<blocks(batch, 8), 256, 0, st>>>(m->A2, batch, H, m->P + m->oW3, m->P + m->ob3, y);
    ++g_launches;
}

// Backward from dy (m->dy) into the gradient vector g and, optionally, dL/dx.
void backward(orkan_mlp* m, const float* x, int batch, float* g, float* gx, cudaStream_t st) {
    const int I = m->n_in, H = m->h;
    const dim3 cols((H + 31) / 32), lanes(32, kColRows);
    k_colsum<<<cols, lanes, 0, st>>>(m->A2, batch, H, m->dy, g + m->oW3);
    k_colsum<<<1, lanes, 0, st>>>(m->dy, batch, 1, nullptr, g + m->ob3);
    k_outer_gelu<<<blocks((size_t)batch * H, 256), 256, 0, st>>>(m->dy, m->P + m->oW3, m->Z2, batch, H, m->dZ2);
    g_launches += 3;
    gemm_tn_split(m, st, H, H, batch, m->A1, H, m->dZ2, H, g + m->oW2);
    k_colsum<<<cols, lanes, 0, st>>>(m->dZ2, batch, H, nullptr, g + m->ob2);
    ++g_launches;
    gemm<false, true, kEpiGeluBack>(st, batch, H, H, m->dZ2, H, m->P + m->oW2, H, m->dZ1, H, nullptr, m->Z1);
    gemm_tn_split(m, st, I, H, batch, x, I, m->dZ1, H, g + m->oW1);
    k_colsum<<<cols, lanes, 0, st>>>(m->dZ1, batch, H, nullptr, g + m->ob1);
    ++g_launches;
    if (gx) gemm<false, true, kEpiStore>(st, batch, I, H, m->dZ1, H, m->P + m->oW1, H, gx, I);
}

RowsArgs rows_args(const orkan_mlp* m, const float* x, int rows) {
    RowsArgs a{};
    a.x = x;
    a.rows = rows;
    a.n_in = m->n_in;
    a.W1 = m->P + m->oW1;
    a.b1 = m->P + m->ob1;
    a.W2 = m->P + m->oW2;
    a.b2 = m->P + m->ob2;
    a.w3 = m->P + m->oW3;
    a.b3 = m->P + m->ob3;
    return a;
}

template <int RG, bool BWD>
int rows_launch_t(RowsArgs a, cudaStream_t st) {
    a.tiles = (a.rows + 8 * RG - 1) / (8 * RG);
    a.parts = a.tiles * RG;
    k_rows<RG, BWD><<<a.tiles, kFThreads, rows_smem<RG>(a.n_in), st>>>(a);
    ++g_launches;
    return (int)cudaGetLastError();
}

// Shared-memory limits of the row kernels on the current device (at creation: launches may be captured).
int rows_prepare() {
    auto allow = [](const void* f, size_t bytes) {
        return (int)cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    };
    int rc = allow((const void*)k_rows<1, true>, rows_smem<1>(kFMaxIn));
    if (!rc) rc = allow((const void*)k_rows<1, false>, rows_smem<1>(kFMaxIn));
    if (!rc) rc = allow((const void*)k_rows<4, true>, rows_smem<4>(kFMaxIn));
    if (!rc) rc = allow((const void*)k_rows<4, false>, rows_smem<4>(kFMaxIn));
    if (!rc) rc = allow((const void*)k_rows<8, false>, rows_smem<8>(kFMaxIn));
    return rc;
}

// Rows per tile: 8 while that leaves at most two tiles per SM (measured 18.7 us for 2368 rows forward
// and 23.1 us with 32-row tiles at 2400), then 32 (with backward z1 stays in registers as well), and
// forward 64 once they fill two tiles per SM: 131 us for 32768 rows and 3.3 ns a row beyond, 4.1 ns
// in 32-row tiles.
int rows_tile(int rows, bool bwd) {
    if (rows <= 2 * 8 * 148) return 8;
    return bwd || rows < 2 * 64 * 148 ? 32 : 64;
}
int rows_forward(const orkan_mlp* m, const float* x, int rows, float* y, cudaStream_t st) {
    RowsArgs a = rows_args(m, x, rows);
    a.y = y;
    switch (rows_tile(rows, false)) {
        case 8: return rows_launch_t<1, false>(a, st);
        case 32: return rows_launch_t<4, false>(a, st);
        default: return rows_launch_t<8, false>(a, st);
    }
}

// Forward, loss and backward of the fused form: t NULL takes the gradient of f itself; g NULL leaves
// the parameter gradients out; loss and gx may be NULL.
int rows_backward(orkan_mlp* m, const float* x, const float* t, int rows, float* loss, float* g, float* gx,
                  cudaStream_t st) {
    RowsArgs a = rows_args(m, x, rows);
    a.t = t;
    a.gx = gx;
    if (g) {
        a.A1 = m->A1;
        a.dZ1 = m->dZ1;
        a.dZ2 = m->dZ2;
        a.colp = m->colp;
        a.rowp = m->rowp;
    }
    const int tile = rows_tile(rows, true), tiles = (rows + tile - 1) / tile, parts = tiles * (tile / 8);
    int rc = tile == 8 ? rows_launch_t<1, true>(a, st) : rows_launch_t<4, true>(a, st);
    if (rc || !g) return rc;
    // slices of whole chunks, about two blocks per SM over the 20 tiles, at least 64 rows each
    const int want = std::max(1, std::min(15, (rows + 63) / 64));
    const int per = ((rows + want - 1) / want + kFK - 1) / kFK * kFK, nz = (rows + per - 1) / per;
    k_wgrad<<<dim3(20, nz), 256, 0, st>>>(x, m->A1, m->dZ1, m->dZ2, rows, m->n_in, per, m->split);
    const int nw = ((m->n_in + kFH) * kFH + 255) / 256;
    k_reduce<<<nw + 25, 256, 0, st>>>(m->split, nz, m->colp, parts, m->rowp, tiles, rows, m->n_in, nw, g, loss);
    g_launches += 2;
    return (int)cudaGetLastError();
}

// Do the arrays of na floats at a and nb floats at b share memory?  The row kernel writes results of some rows while
// others are still to be read, so results that lie on its inputs go through the network's own buffers.
bool overlap(const float* a, size_t na, const float* b, size_t nb) {
    return a && b && a < b + nb && b < a + na;
}
int copy_out(float* dst, const float* src, size_t count, cudaStream_t st) {
    return (int)cudaMemcpyAsync(dst, src, count * sizeof(float), cudaMemcpyDeviceToDevice, st);
}

// One training step on the minibatch of the device step counter (captured into a graph).
void train_step(orkan_mlp* m, const float* X, const float* T, unsigned count, int batch, unsigned spe, uint64_t seed,
                float lr, cudaStream_t st) {
    k_step_begin<<<1, 1, 0, st>>>(m->step);
    k_gather<<<blocks(batch, 128), 128, 0, st>>>(X, T, count, m->n_in, batch, spe, seed, m->step, m->xb, m->tb);
    g_launches += 2;
    if (m->fused) {
        rows_backward(m, m->xb, m->tb, batch, m->loss, m->G, nullptr, st);
    } else {
        forward(m, m->xb, batch, m->y, st);
        k_loss<<<1, 1024, 0, st>>>(m->y, m->tb, batch, m->dy, m->loss);
        ++g_launches;
        backward(m, m->xb, batch, m->G, nullptr, st);
    }
    k_copy_loss<<<1, 1, 0, st>>>(m->loss, m->step, spe, m->losses);
    ++g_launches;
    k_adam<<<blocks(m->np, 256), 256, 0, st>>>(m->P, m->G, m->M1, m->M2, m->np, lr, m->step);
    ++g_launches;
}

}  // namespace

extern "C" {

int orkan_mlp_create(orkan_mlp_t** out, unsigned n_in, unsigned hidden, unsigned max_batch, unsigned long long seed) {
    if (!out) return (int)cudaErrorInvalidValue;
    *out = nullptr;
    if (n_in == 0 || hidden == 0 || max_batch == 0 || n_in > 4096 || hidden > 8192 || max_batch > (1u << 22))
        return (int)cudaErrorInvalidValue;
    orkan_mlp* m = new orkan_mlp();
    m->n_in = (int)n_in;
    m->h = (int)hidden;
    m->maxb = (int)max_batch;
    const size_t I = n_in, H = hidden, B = max_batch;
    m->oW1 = 0;
    m->ob1 = m->oW1 + I * H;
    m->oW2 = m->ob1 + H;
    m->ob2 = m->oW2 + H * H;
    m->oW3 = m->ob2 + H;
    m->ob3 = m->oW3 + H;
    m->np = m->ob3 + 1;
    int rc = 0;
    auto al = [&](float** p, size_t n) {
        if (!rc) rc = (int)cudaMalloc(reinterpret_cast<void**>(p), (n ? n : 1) * sizeof(float));
    };
    al(&m->P, m->np);
    al(&m->G, m->np);
    al(&m->M1, m->np);
    al(&m->M2, m->np);
    m->fused = hidden == (unsigned)kFH && n_in <= (unsigned)kFMaxIn;
    al(&m->A1, B * H);
    if (m->fused) {                             // column sums of every 8 rows, row sums of every tile
        al(&m->colp, 3 * ((B + 7) / 8 + 4) * H);
        al(&m->rowp, 2 * ((B + 7) / 8));
    } else {
        al(&m->Z1, B * H);
        al(&m->Z2, B * H);
        al(&m->A2, B * H);
    }
    al(&m->dZ2, B * H);
    al(&m->dZ1, B * H);
    al(&m->y, B);
    al(&m->dy, B);
    al(&m->xb, B * I);
    al(&m->tb, B);
    al(&m->loss, 1);
    m->split_cap = (size_t)32 * std::max(I, H) * H;
    al(&m->split, m->split_cap);
    if (!rc) rc = (int)cudaMalloc(reinterpret_cast<void**>(&m->step), 2 * sizeof(unsigned));
    if (rc) {
        orkan_mlp_destroy(m);
        return rc;
    }
    // deterministic initialisation: splitmix64 stream, uniform in +-sqrt(6 / fan_in) for W
    std::vector<float> p(m->np, 0.0f);
    uint64_t st = seed;
    auto uni = [&](float bound) {
        st += 0x9e3779b97f4a7c15ull;
        const uint64_t z = mix64(st);
        return (float)(((double)(z >> 11) * (1.0 / 9007199254740992.0)) * 2.0 - 1.0) * bound;
    };
    const float b1 = sqrtf(6.0f / (float)I), b2 = sqrtf(6.0f / (float)H);
    for (size_t i = 0; i < I * H; ++i) p[m->oW1 + i] = uni(b1);
    for (size_t i = 0; i < H * H; ++i) p[m->oW2 + i] = uni(b2);
    for (size_t i = 0; i < H; ++i) p[m->oW3 + i] = uni(b2);
    rc = orkan_mlp_set_params(m, p.data());
    if (!rc && m->fused) rc = rows_prepare();
    if (rc) {
        orkan_mlp_destroy(m);
        return rc;
    }
    *out = m;
    return 0;
}

void orkan_mlp_destroy(orkan_mlp_t* m) {
    if (!m) return;
    float* bufs[] = {m->P, m->G, m->M1, m->M2, m->Z1, m->A1, m->Z2, m->A2, m->dZ2, m->dZ1,
                     m->y, m->dy, m->xb, m->tb, m->loss, m->losses, m->split, m->colp, m->rowp};
    for (float* b : bufs) cudaFree(b);
    cudaFree(m->step);
    delete m;
}

size_t orkan_mlp_param_count(const orkan_mlp_t* m) { return m ? m->np : 0; }

int orkan_mlp_get_params(const orkan_mlp_t* m, float* host) {
    if (!m || !host) return (int)cudaErrorInvalidValue;
    return (int)cudaMemcpy(host, m->P, m->np * sizeof(float), cudaMemcpyDeviceToHost);
}

int orkan_mlp_set_params(orkan_mlp_t* m, const float* host) {
    if (!m || !host) return (int)cudaErrorInvalidValue;
    int rc = (int)cudaMemcpy(m->P, host, m->np * sizeof(float), cudaMemcpyHostToDevice);
    if (!rc) rc = (int)cudaMemset(m->M1, 0, m->np * sizeof(float));
    if (!rc) rc = (int)cudaMemset(m->M2, 0, m->np * sizeof(float));
    if (!rc) rc = (int)cudaMemset(m->step, 0, 2 * sizeof(unsigned));
    return rc;
}

int orkan_mlp_forward(orkan_mlp_t* m, const float* x_dev, unsigned batch, float* y_dev, void* stream) {
    if (!m || !x_dev || !y_dev || batch == 0 || (int)batch > m->maxb) return (int)cudaErrorInvalidValue;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (m->fused) {
        const bool own = overlap(y_dev, batch, x_dev, (size_t)batch * m->n_in);
        const int rc = rows_forward(m, x_dev, (int)batch, own ? m->y : y_dev, st);
        return rc || !own ? rc : copy_out(y_dev, m->y, batch, st);
    }
    forward(m, x_dev, (int)batch, y_dev, st);
    return (int)cudaGetLastError();
}

int orkan_mlp_predict(orkan_mlp_t* m, const float* x_dev, unsigned count, float* y_dev, void* stream) {
    if (!m || !x_dev || !y_dev || count == 0) return (int)cudaErrorInvalidValue;
    // the fused form needs no activations in memory: any count at once, in int-sized pieces
    const bool whole = m->fused && !overlap(y_dev, count, x_dev, (size_t)count * m->n_in);
    const unsigned most = whole ? 1u << 24 : (unsigned)m->maxb;
    int rc = 0;
    for (unsigned c0 = 0; c0 < count && !rc; c0 += std::min(most, count - c0))
        rc = whole ? rows_forward(m, x_dev + (size_t)c0 * m->n_in, (int)std::min(most, count - c0), y_dev + c0,
                                     reinterpret_cast<cudaStream_t>(stream))
                      : orkan_mlp_forward(m, x_dev + (size_t)c0 * m->n_in, std::min(most, count - c0), y_dev + c0, stream);
    return rc;
}

int orkan_mlp_gradients(orkan_mlp_t* m, const float* x_dev, const float* t_dev, unsigned batch, float* loss_dev,
                        float* grad_dev, float* gx_dev, void* stream) {
    if (!m || !x_dev || !t_dev || !grad_dev || batch == 0 || (int)batch > m->maxb) return (int)cudaErrorInvalidValue;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (m->fused) {
        const size_t nx = (size_t)batch * m->n_in;
        const bool own = overlap(gx_dev, nx, x_dev, nx) || overlap(gx_dev, nx, t_dev, batch);
        const int rc = rows_backward(m, x_dev, t_dev, (int)batch, loss_dev, grad_dev, own ? m->xb : gx_dev, st);
        return rc || !own ? rc : copy_out(gx_dev, m->xb, nx, st);
    }
    forward(m, x_dev, (int)batch, m->y, st);
    k_loss<<<1, 1024, 0, st>>>(m->y, t_dev, (int)batch, m->dy, loss_dev);
    ++g_launches;
    backward(m, x_dev, (int)batch, grad_dev, gx_dev, st);
    return (int)cudaGetLastError();
}

int orkan_mlp_train(orkan_mlp_t* m, const float* x_dev, const float* t_dev, unsigned count, unsigned epochs,
                    unsigned batch, float lr, unsigned long long seed, float* loss_dev, void* stream) {
    if (!m || !x_dev || !t_dev || batch == 0 || (int)batch > m->maxb || count < batch)
        return (int)cudaErrorInvalidValue;
    if (epochs == 0) return 0;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const unsigned spe = count / batch;
    int rc = 0;
    if (spe > m->losses_cap) {
        cudaFree(m->losses);
        m->losses = nullptr;
        m->losses_cap = 0;
        if ((rc = (int)cudaMalloc(reinterpret_cast<void**>(&m->losses), spe * sizeof(float)))) return rc;
        m->losses_cap = spe;
    }
    // step[0] counts every Adam step of this network (bias correction); step[1] restarts at
    // 0 for this call and drives the epoch schedule
    if ((rc = (int)cudaMemsetAsync(m->step + 1, 0, sizeof(unsigned), st))) return rc;
    cudaStream_t cap = nullptr;
    if ((rc = (int)cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking))) return rc;
    cudaGraph_t g = nullptr;
    cudaGraphExec_t ge = nullptr;
    const unsigned long long l0 = g_launches.load();
    rc = (int)cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
    if (!rc) {
        train_step(m, x_dev, t_dev, count, (int)batch, spe, seed, lr, cap);
        const int erc = (int)cudaGetLastError();
        rc = (int)cudaStreamEndCapture(cap, &g);
        if (!rc) rc = erc;
    }
    const unsigned long long per_step = g_launches.load() - l0;
    g_launches -= per_step;                       // counted per replay below
    if (!rc) rc = (int)cudaGraphInstantiate(&ge, g, 0);
    if (g) cudaGraphDestroy(g);
    cudaEvent_t ev = nullptr;                     // the replays follow the caller's stream
    if (!rc) rc = (int)cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    if (!rc) rc = (int)cudaEventRecord(ev, st);
    if (!rc) rc = (int)cudaStreamWaitEvent(cap, ev, 0);
    const unsigned long long total = (unsigned long long)epochs * spe;
    for (unsigned long long s = 0; s < total && !rc; ++s) {
        rc = (int)cudaGraphLaunch(ge, cap);
        g_launches += per_step;
    }
    if (!rc && loss_dev) {
        k_epoch_loss<<<1, 1, 0, cap>>>(m->losses, spe, loss_dev);
        ++g_launches;
        rc = (int)cudaGetLastError();
    }
    if (!rc) rc = (int)cudaEventRecord(ev, cap);
    if (!rc) rc = (int)cudaStreamWaitEvent(st, ev, 0);
    if (!rc) rc = (int)cudaStreamSynchronize(cap);
    if (ge) cudaGraphExecDestroy(ge);
    if (ev) cudaEventDestroy(ev);
    cudaStreamDestroy(cap);
    return rc;
}

int orkan_mlp_ascend(orkan_mlp_t* m, float* x_dev, unsigned count, unsigned steps, float lr, float lo, float hi,
                     float* y_dev, void* stream) {
    if (!m || !x_dev || count == 0) return (int)cudaErrorInvalidValue;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const size_t nx = (size_t)count * m->n_in;
    float *gx = nullptr, *m1 = nullptr, *m2 = nullptr;
    int rc = 0;
    if ((rc = (int)cudaMalloc(reinterpret_cast<void**>(&gx), nx * sizeof(float))) ||
        (rc = (int)cudaMalloc(reinterpret_cast<void**>(&m1), nx * sizeof(float))) ||
        (rc = (int)cudaMalloc(reinterpret_cast<void**>(&m2), nx * sizeof(float)))) {
        cudaFree(gx);
        cudaFree(m1);
        return rc;
    }
    cudaMemsetAsync(m1, 0, nx * sizeof(float), st);
    cudaMemsetAsync(m2, 0, nx * sizeof(float), st);
    for (unsigned t = 1; t <= steps && !rc; ++t) {
        for (unsigned c0 = 0; c0 < count; c0 += (unsigned)m->maxb) {
            const int b = (int)((count - c0) < (unsigned)m->maxb ? count - c0 : (unsigned)m->maxb);
            const float* xc = x_dev + (size_t)c0 * m->n_in;
            if (m->fused) {                     // inputs' gradient alone
                if (!rc) rc = rows_backward(m, xc, nullptr, b, nullptr, nullptr, gx + (size_t)c0 * m->n_in, st);
                continue;
            }
            forward(m, xc, b, m->y, st);
            k_loss<<<1, 1024, 0, st>>>(m->y, nullptr, b, m->dy, nullptr);
            ++g_launches;
            backward(m, xc, b, m->G, gx + (size_t)c0 * m->n_in, st);
        }
        k_adam_inputs<<<blocks(nx, 256), 256, 0, st>>>(x_dev, gx, m1, m2, nx, lr, (int)t, lo, hi);
        ++g_launches;
        if (!rc) rc = (int)cudaGetLastError();
    }
    if (!rc && y_dev) rc = orkan_mlp_predict(m, x_dev, count, y_dev, stream);
    if (!rc) rc = (int)cudaStreamSynchronize(st);
    cudaFree(gx);
    cudaFree(m1);
    cudaFree(m2);
    return rc;
}

unsigned long long orkan_mlp_launch_count(void) { return g_launches.load(); }

}  // extern "C"
