// qaoa.cu - the batched QAOA entry points of include/orkan_batch.h: the batch context,
// resident cost vectors (one per distinct graph), waves of state vectors, the fused pass
// kernels, one CUDA graph per batch and the autotuner of the launch configuration.
#include "qaoa.cuh"

#include "../../../include/orkan_batch.h"

#include <stdint.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <string>
#include <vector>

using namespace orkan;

namespace {

// One graph's place in the resident arrays: its edges and weights, and its costs.
struct QaoaEdges {
    const unsigned char* uv;
    const double* w;
    unsigned ne;
};

// Costs of one kind of pass in its order (qaoa_cost_slot):
// cost[i] = sum_e w_e [bit u_e of x != bit v_e of x], x = qaoa_cost_state(i), edges in the
// given order.
template <class CostT>
__global__ void k_qaoa_cost(CostT* cost, QaoaGeo g, idx_t count, QaoaEdges E) {
    for (idx_t i = (idx_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (idx_t)gridDim.x * blockDim.x) {
        const unsigned x = (unsigned)qaoa_cost_state(g, sizeof(CostT) == 1, i);
        double c = 0.0;
        for (unsigned e = 0; e < E.ne; ++e)
            if (((x >> E.uv[2 * e]) ^ (x >> E.uv[2 * e + 1])) & 1u) c += E.w[e];
        cost[i] = (CostT)c;
    }
}

// The whole cost vector from the resident costs of the low (or full) passes.
template <class CostT>
__global__ void k_qaoa_cost_vector(const CostT* cost, QaoaGeo g, idx_t count, double* out) {
    const idx_t all = (idx_t(1) << g.n) - 1;
    for (idx_t i = (idx_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (idx_t)gridDim.x * blockDim.x) {
        const idx_t x = qaoa_cost_state(g, sizeof(CostT) == 1, i);
        out[x] = (double)cost[i];
        if (g.kind != kQaoaFull) out[all ^ x] = (double)cost[i];
    }
}

// table[(pos p + k) tstride + c] = fs (cos, sin)(c * gamma[pos p + k]) for c <= cmax of pos
__global__ void k_qaoa_tables(const unsigned* cmax, const double* gamma, const QaoaRx* rx, unsigned count, unsigned p,
                              unsigned tstride, double2* table) {
    const unsigned pos = blockIdx.x;
    if (pos >= count || cmax[pos] >= kQaoaMaxTable) return;
    const unsigned m = cmax[pos] + 1;
    for (unsigned t = threadIdx.x; t < p * m; t += blockDim.x) {
        const unsigned k = t / m, c = t % m;
        const idx_t row = (idx_t)pos * p + k;
        const double fs = rx[row].fs;
        double sn, cs;
        sincos((double)c * gamma[row], &sn, &cs);
        table[row * tstride + c] = c2(cs * fs, sn * fs);
    }
}

// ---- device accessors ------------------------------------------------------------------
__device__ __forceinline__ unsigned sm_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

struct QaoaDevPsi {
    double2* p;
    __device__ __forceinline__ void st(idx_t i, double2 v) const { p[i] = v; }
    __device__ __forceinline__ void cp16(double2* dst, idx_t i) const {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sm_u32(dst)), "l"(p + i) : "memory");
    }
    __device__ __forceinline__ void bulk_load(double2* dst, idx_t i, unsigned n, void* bar) const {
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                     ::"r"(sm_u32(dst)), "l"(p + i), "r"(n * 16u), "r"(sm_u32(bar)) : "memory");
    }
};
template <class CostT>
struct QaoaDevCost;
template <>
struct QaoaDevCost<double> {
    const double* p;
    __device__ __forceinline__ double ld(unsigned i) const { return __ldg(p + i); }
};
template <>
struct QaoaDevCost<uint8_t> {
    const uint8_t* p;
    __device__ __forceinline__ uint8_t ld(unsigned i) const { return __ldg(p + i); }
    // the 2^K costs at i, a multiple of 2^K
    template <int K>
    __device__ __forceinline__ void words(uint32_t* w, unsigned i) const {
        if constexpr (K == 4) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(p + i));
            w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
        } else if constexpr (K == 3) {
            const uint2 v = __ldg(reinterpret_cast<const uint2*>(p + i));
            w[0] = v.x; w[1] = v.y;
        } else if constexpr (K == 2) {
            w[0] = __ldg(reinterpret_cast<const unsigned*>(p + i));
        } else {
            w[0] = __ldg(reinterpret_cast<const unsigned short*>(p + i));
        }
    }
};

__device__ __forceinline__ void mb_init(void* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(sm_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mb_arrive(void* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(sm_u32(bar)) : "memory");
}
__device__ __forceinline__ void mb_expect(void* bar, unsigned bytes) {
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;\n" ::"r"(sm_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mb_try(void* bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                 " selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok) : "r"(sm_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait: false when the limit is reached.
__device__ __forceinline__ bool mb_wait(void* bar, unsigned parity, unsigned long long limit) {
    for (unsigned long long i = 0; i < limit; ++i)
        if (mb_try(bar, parity)) return true;
    return false;
}

// Shape of a pass block by chunk size: `groups` groups of 2^C / 16 threads work on one item
// each, and the other buffers hold staged items.  Four more warps stage the items.
//
// Registers: a block of 640 threads is launched with 96 each (61440); the staging warps give
// back all but 32 (4096 in all) and the computing ones then take 112 (57344), which holds the
// 16 amplitudes of a set (64) with little spilled.  The split waits forever for registers that the launch
// did not bring, so it is used where the compiler gave the kernel exactly those 96 (prepare_kernels);
// SPLIT = false is the same pass at whatever it gave, for every other build.
constexpr unsigned kStageThreads = 128;
constexpr unsigned kComputeThreads = 512;
constexpr unsigned kLaunchRegs = 96, kStageRegs = 32, kComputeRegs = 112;
static_assert(kStageThreads * kStageRegs + kComputeThreads * kComputeRegs <=
              (kStageThreads + kComputeThreads) * kLaunchRegs, "register split within the launch's registers");
template <unsigned C>
struct PassShape {
    static constexpr unsigned kThreads = (1u << C) / 16;
    static constexpr unsigned kGroups = kComputeThreads / kThreads;
    static constexpr unsigned kBuffers = C >= 13 ? 1 : kGroups + kGroups / 2;
    static constexpr unsigned kBlock = kComputeThreads + kStageThreads;
};

// One pass over the items of a launch.  Block b takes items b, b + grid, ... in turn; group g
// computes every kGroups-th of them, and the staging warps keep the free buffers filled: low
// items by one bulk copy of 2^C amplitudes, high items by 16-byte copies of runs.  A group
// hands its buffer back as soon as its last stage has its amplitudes in registers; no such
// stage reads the phase table that goes back with them (qaoa_pass_setup).
//
// Bound: HBM (32 bytes per stored amplitude in a middle pass) and shared memory (2 m - 1
// stages of 32 bytes) are close at C = 12; the registers of the 16 computing warps leave one
// block per SM, so the copies run ahead of the arithmetic instead of in another block.
// Measured (16 instances, p = 4, ms per run) against two 256-thread blocks per SM that filled,
// computed and stored one item after the other on the whole state: 24 qubits 5.61 against
// 17.17, 22 qubits 1.41 against 4.13, 20 qubits 0.41 against 0.95, 16 qubits 0.086 against
// 0.098; 8 weighted instances of 24 qubits at p = 6 5.89 against 19.8.  Half of the state's
// amplitudes account for a factor of two, the staging and the shorter stages for the rest.
template <class CostT, unsigned C, bool SPLIT>
__global__ void __launch_bounds__(PassShape<C>::kBlock, 1)
    k_qaoa_pass(const __grid_constant__ QaoaPass P, const QaoaTables T) {
    using Sh = PassShape<C>;
    constexpr unsigned NB = Sh::kBuffers, GT = Sh::kThreads, NG = Sh::kGroups;
    constexpr bool kBytes = sizeof(CostT) == 1;
    extern __shared__ __align__(128) unsigned char smem_q[];
    const QaoaSmem L = qaoa_smem(C, NB, kBytes ? T.tstride : 0u, 512);
    unsigned long long* full = reinterpret_cast<unsigned long long*>(smem_q + L.bar);
    unsigned long long* empty = full + NB;
    unsigned char* flags = reinterpret_cast<unsigned char*>(empty + NB);
    if (threadIdx.x == 0) {
        for (unsigned b = 0; b < NB; ++b) {
            mb_init(full + b, kStageThreads + 1);      // the staging threads' copies, and the first one
            mb_init(empty + b, GT / 32);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    const unsigned warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const unsigned items = (unsigned)P.items;          // checked to fit by the host
    if (warp >= kComputeThreads / 32) {                // staging
        if constexpr (SPLIT) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(kStageRegs));
        const unsigned st = threadIdx.x - kComputeThreads;
        unsigned k = 0;
        bool ok = true;
        for (unsigned w = blockIdx.x; w < items; w += gridDim.x, ++k) {
            const unsigned b = k % NB;
            const QaoaInst I = P.inst[w >> P.li];
            if (k >= NB && !mb_wait(empty + b, (k / NB - 1) & 1u, P.wait_limit)) { ok = false; break; }
            if (st == 0) {
                *reinterpret_cast<QaoaItem*>(smem_q + L.item + kQaoaItemBytes * b) = qaoa_item(P, T, I, w, sizeof(CostT));
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                if (P.layer_a >= 0 && P.kind == kQaoaLow) mb_expect(full + b, 16u << C);
            }
            if (kBytes && P.layer_phase >= 0) {
                const double2* row = T.phase + ((idx_t)I.pos * P.p + P.layer_phase) * T.tstride;
                double2* tab = reinterpret_cast<double2*>(smem_q + L.tab + L.tab_stride * b);
                for (unsigned e = st; e < T.tstride; e += kStageThreads)
                    QaoaDevPsi{const_cast<double2*>(row)}.cp16(tab + e, e);
            }
            if (!kBytes && st == 0) {                  // the item's FP64 costs on their way to L2
                const double* src = static_cast<const double*>(I.cost) + ((size_t)(w & ((1u << P.li) - 1)) << C);
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(src), "r"(8u << C) : "memory");
            }
            if (P.layer_a >= 0)
                qaoa_fill(P.geo, QaoaDevPsi{I.psi}, w & ((1u << P.li) - 1), reinterpret_cast<double2*>(smem_q + L.buf_stride * b),
                          full + b, st, kStageThreads);
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(sm_u32(full + b)) : "memory");
            if (st == 0) mb_arrive(full + b);
        }
        if (!ok) *P.status = 1.0;
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        // the bulk copies land before the block's shared memory is given up, also where a wait
        // of the computing warps ran out and no one else sees to it
        if (st == 0)
            for (unsigned b = 0; b < NB && b < k; ++b)
                mb_wait(full + b, ((k - 1 - b) / NB) & 1u, kQaoaPolls);
        return;
    }
    if constexpr (SPLIT) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(kComputeRegs));
    const unsigned gid = warp / (GT / 32), tid = threadIdx.x % GT;
    double* red = reinterpret_cast<double*>(smem_q + L.red) + gid * (GT / 32);
    auto group_sync = [&] { asm volatile("bar.sync %0, %1;\n" ::"r"(1 + gid), "n"(GT) : "memory"); };
    unsigned k = gid;
    for (unsigned w = blockIdx.x + gid * gridDim.x; w < items; w += NG * gridDim.x, k += NG) {
        const unsigned b = k % NB, parity = (k / NB) & 1u;
        unsigned char* flag = flags + 2 * gid + ((k / NG) & 1u);
        if (tid == 0) *flag = mb_wait(full + b, parity, P.wait_limit) ? 1 : 0;
        group_sync();
        if (!*flag || !mb_wait(full + b, parity, P.wait_limit)) {
            if (tid == 0) *P.status = 1.0;
            break;
        }
        const QaoaItem& J = *reinterpret_cast<const QaoaItem*>(smem_q + L.item + kQaoaItemBytes * b);
        double2* vb = reinterpret_cast<double2*>(smem_q + L.buf_stride * b);
        const double2* tab = reinterpret_cast<const double2*>(smem_q + L.tab + L.tab_stride * b);
        auto release = [&] {
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) mb_arrive(empty + b);
        };
        double acc = 0.0;
        for (unsigned r = 0; r < P.nreg; ++r) {
            acc = qaoa_stage<CostT>(P, r, J, QaoaDevPsi{J.psi}, QaoaDevCost<CostT>{static_cast<const CostT*>(J.cost)},
                                    vb, tab, C, tid, GT, release);
            if (r + 1 < P.nreg) {
                if (P.stage[r].warp_sync) __syncwarp();
                else group_sync();
            }
        }
        if (P.layer_phase < 0) {                       // the item's share of the mean, in fixed order
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
            if (lane == 0) red[tid / 32] = acc;
            group_sync();
            if (tid == 0) {
                double s = 0.0;
                for (unsigned i = 0; i < GT / 32; ++i) s += red[i];
                P.partial[w] = s;
            }
            group_sync();                              // red is read before the next item writes it
        }
    }
}

// Full items: one block per instance holds all 2^n amplitudes and runs the whole circuit.
template <class CostT>
__global__ void __launch_bounds__(512, 1) k_qaoa_full(const __grid_constant__ QaoaPass P, const QaoaTables T) {
    extern __shared__ __align__(128) unsigned char smem_q[];
    __shared__ double red[16];
    double2* vb = reinterpret_cast<double2*>(smem_q);
    const QaoaInst I = P.inst[blockIdx.x];
    const unsigned nst = qaoa_full_stages(P.geo.m, P.p);
    double acc = 0.0;
    for (unsigned r = 0; r < nst; ++r) {
        acc = qaoa_full_stage<CostT>(P, T, I.pos, I.n, r, QaoaDevCost<CostT>{static_cast<const CostT*>(I.cost)}, vb,
                                     threadIdx.x, blockDim.x);
        if (r + 1 < nst) __syncthreads();
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (unsigned i = 0; i < blockDim.x / 32; ++i) s += red[i];
        P.partial[blockIdx.x] = s;
    }
}

// out[pos] = sum of the instance's partials (a fixed share per thread, then a fixed tree) times
// the factor of its last layer.  One thread per instance took 212 us for the 4096 partials of a
// 24-qubit instance; one block takes a few.
constexpr unsigned kFoldThreads = 128;
__global__ void __launch_bounds__(kFoldThreads) k_qaoa_fold(const QaoaInst* inst, unsigned ninst,
                                                            const double* partial, idx_t items, const QaoaRx* rx,
                                                            unsigned p, double* out) {
    __shared__ double sh[kFoldThreads];
    const unsigned i = blockIdx.x;
    const idx_t a = inst[i].item0, b = (i + 1 < ninst) ? inst[i + 1].item0 : items;
    double s = 0.0;
    for (idx_t w = a + threadIdx.x; w < b; w += kFoldThreads) s += partial[w];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (unsigned o = kFoldThreads / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[inst[i].pos] = sh[0] * rx[(idx_t)inst[i].pos * p + p - 1].fm;
}

int sm_count() {
    int dev = 0, v = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v > 0 ? v : 148;
}

constexpr unsigned kQaoaMinC = 11;      // smallest chunk of the pass kernel

// Dynamic shared memory of a pass or full launch.
size_t pass_smem(unsigned kind, unsigned C, bool bytes, unsigned tstride) {
    if (kind == kQaoaFull) return size_t(16) << C;
    const unsigned nb = C >= 13 ? 1u : C == 12 ? 3u : 6u;
    return qaoa_smem(C, nb, bytes ? tstride : 0u, 512).total;
}

template <class K>
int allow_smem(K kern) {
    return (int)cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024);
}
// *split is cleared unless the kernel was compiled to the registers of the split.
template <class CostT, unsigned C>
int prepare_pass(bool* split) {
    cudaFuncAttributes fa;
    const int rc = (int)cudaFuncGetAttributes(&fa, k_qaoa_pass<CostT, C, true>);
    if (!rc && fa.numRegs != (int)kLaunchRegs) *split = false;
    return rc ? rc : allow_smem(k_qaoa_pass<CostT, C, true>);
}
int prepare_plain() {
    int rc;
    if ((rc = allow_smem(k_qaoa_pass<uint8_t, 11, false>)) || (rc = allow_smem(k_qaoa_pass<uint8_t, 12, false>)) ||
        (rc = allow_smem(k_qaoa_pass<uint8_t, 13, false>)) || (rc = allow_smem(k_qaoa_pass<double, 11, false>)) ||
        (rc = allow_smem(k_qaoa_pass<double, 12, false>)) || (rc = allow_smem(k_qaoa_pass<double, 13, false>)))
        return rc;
    return 0;
}
// Sets the kernels' shared-memory limits on the current device (before any graph capture) and picks the form.
int prepare_kernels(bool* split) {
    *split = true;
    int rc;
    if ((rc = prepare_pass<uint8_t, 11>(split)) || (rc = prepare_pass<uint8_t, 12>(split)) ||
        (rc = prepare_pass<uint8_t, 13>(split)) || (rc = prepare_pass<double, 11>(split)) ||
        (rc = prepare_pass<double, 12>(split)) || (rc = prepare_pass<double, 13>(split)) ||
        (rc = allow_smem(k_qaoa_full<uint8_t>)) || (rc = allow_smem(k_qaoa_full<double>)))
        return rc;
    return *split ? 0 : prepare_plain();
}

template <class CostT, unsigned C>
void launch_chunks(bool split, unsigned grid, size_t smem, const QaoaPass& P, const QaoaTables& T, cudaStream_t st) {
    if (split) k_qaoa_pass<CostT, C, true><<<grid, PassShape<C>::kBlock, smem, st>>>(P, T);
    else k_qaoa_pass<CostT, C, false><<<grid, PassShape<C>::kBlock, smem, st>>>(P, T);
}
template <class CostT>
int launch_pass_t(bool split, unsigned nt, unsigned grid, size_t smem, const QaoaPass& P, const QaoaTables& T,
                  cudaStream_t st) {
    if (P.kind == kQaoaFull) k_qaoa_full<CostT><<<grid, nt, smem, st>>>(P, T);
    else if (P.C == 11) launch_chunks<CostT, 11>(split, grid, smem, P, T, st);
    else if (P.C == 12) launch_chunks<CostT, 12>(split, grid, smem, P, T, st);
    else launch_chunks<CostT, 13>(split, grid, smem, P, T, st);
    return (int)cudaGetLastError();
}

// Launch configuration of the instances of one qubit count: log2 chunk, threads, ring depth.
struct QaoaCfg {
    unsigned C, nt, ring;
};

struct Graph {                     // one distinct cost function
    unsigned n;
    std::vector<unsigned char> edges;
    std::vector<double> w;
    unsigned cmax;                 // byte costs: integer maximum; else 0xffffffff
    // 2^n costs: those of the low and of the high passes (2^(n-1) each), or of the full pass
    unsigned char* d_cost = nullptr;
    size_t cost_bytes = 0;         // of one cost
    unsigned cost_C = 0;           // chunk size they are ordered for (0: not filled yet)
    QaoaEdges dev{};               // edges and weights on the device
    void* high() const { return d_cost + (cost_bytes << (n - 1)); }
};

struct Launch {
    int what;                      // 0 pass, 1 fold
    unsigned inst_off, ninst;      // slice of the plan's instance records
    idx_t items;
    unsigned pass, C, kind, nt;
    unsigned n;                    // qubit count of every instance of the launch
    unsigned grid;                 // blocks (pass launches)
    size_t smem;                   // dynamic shared memory of a block (pass launches)
    bool bytes;                    // byte costs
    size_t partial_off;
};

struct Plan {
    std::vector<Launch> launches;
    std::vector<QaoaInst> inst;    // psi holds an arena offset until the arena is known
    size_t arena = 0, partial = 0;
    unsigned waves = 0;
};

}  // namespace

struct orkan_qaoa {
    int device = 0;
    unsigned count = 0, p = 0;
    std::vector<unsigned> n;            // by instance
    std::vector<unsigned> gid;          // graph of each instance
    std::vector<Graph> graphs;
    std::vector<unsigned> cmax;         // by instance (byte costs) or 0xffffffff
    unsigned tstride = 1;
    bool any_bytes = false;
    unsigned long long budget = 0;
    QaoaCfg cfg[27];                    // launch configuration by qubit count
    // device buffers
    unsigned* d_cmax = nullptr;
    double* d_gamma = nullptr;          // [instance][p]
    QaoaRx* d_rx = nullptr;
    double2* d_table = nullptr;         // [instance][p][tstride]
    double* d_out = nullptr;            // means, then the status of the bounded waits
    unsigned char* d_costs = nullptr;   // every graph's costs
    unsigned char* d_uv = nullptr;      // every graph's edges and weights
    double* d_w = nullptr;
    double* d_partial = nullptr;
    unsigned char* d_arena = nullptr;
    size_t arena_bytes = 0, partial_cap = 0;
    QaoaInst* d_inst = nullptr;
    size_t inst_cap = 0;
    bool split = true;                      // the passes re-divide their registers
    unsigned long long polls = kQaoaPolls;  // limit of the passes' waits (orkan_qaoa_test_expire)
    // pinned host staging
    double* h_gamma = nullptr;
    QaoaRx* h_rx = nullptr;
    double* h_out = nullptr;
    Plan plan;
    cudaStream_t cap = nullptr;
    cudaGraphExec_t exec = nullptr;
};

namespace {

template <class T>
int dalloc(T** p, size_t count) {
    return (int)cudaMalloc(reinterpret_cast<void**>(p), (count ? count : 1) * sizeof(T));
}

unsigned default_C(unsigned n) { return n <= 12 ? n : std::max(12u, (n + 1) / 2); }
bool is_full(const orkan_qaoa* b, unsigned n) { return n <= b->cfg[n].C; }

// The launch shape that goes with a chunk size: threads per item (16 amplitudes each; a full
// item of fewer amplitudes than that takes one warp at least) and buffers per item in work.
QaoaCfg cfg_for(unsigned n, unsigned C) {
    QaoaCfg c;
    c.C = C;
    c.nt = C >= 13 ? 512u : C == 12 ? 256u : 128u;
    c.ring = (C >= 13 || n <= C) ? 1u : 2u;
    return c;
}

// Default: 2^12-slot chunks, two items in work per block and a third one staged; instances up
// to 12 qubits in one full pass, 25 and 26 qubits in 2^13-slot chunks (n <= 2 C).  A high pass
// of up to 20 qubits then mixes 8 bits in two groups (three stages instead of five).
QaoaCfg default_cfg(unsigned n) { return cfg_for(n, default_C(n)); }
size_t state_bytes(const orkan_qaoa* b, unsigned n) { return is_full(b, n) ? 0 : (size_t(1) << (n - 1)) * 16; }

// Launch plan for the instances `sel` (qubit counts descending), in waves under the budget.
Plan make_plan(const orkan_qaoa* b, const std::vector<unsigned>& sel) {
    Plan pl;
    size_t first = 0;
    while (first < sel.size()) {
        size_t bytes = 0, last = first;
        while (last < sel.size() && (last == first || bytes + state_bytes(b, b->n[sel[last]]) <= b->budget))
            bytes += state_bytes(b, b->n[sel[last++]]);
        pl.arena = std::max(pl.arena, bytes);
        ++pl.waves;
        std::vector<size_t> off(last - first);              // state offsets of the wave
        size_t o = 0;
        for (size_t k = first; k < last; ++k) {
            off[k - first] = o;
            o += state_bytes(b, b->n[sel[k]]);
        }
        size_t partial = 0;
        size_t g0 = first;                                  // one group per (qubit count, cost type)
        while (g0 < last) {
            const unsigned nq = b->n[sel[g0]];
            for (int bytes_cost = 1; bytes_cost >= 0; --bytes_cost) {
                std::vector<size_t> grp;
                for (size_t k = g0; k < last && b->n[sel[k]] == nq; ++k)
                    if ((b->cmax[sel[k]] < kQaoaMaxTable) == (bool)bytes_cost) grp.push_back(k);
                if (grp.empty()) continue;
                const bool full = is_full(b, nq);
                const unsigned C = full ? nq : b->cfg[nq].C;
                const unsigned npass = full ? 1 : b->p + 1;
                Launch meas{};
                for (unsigned j = 0; j < npass; ++j) {
                    Launch L{};
                    L.what = 0;
                    L.inst_off = (unsigned)pl.inst.size();
                    L.ninst = (unsigned)grp.size();
                    L.pass = full ? 0 : j;
                    L.C = C;
                    L.kind = full ? kQaoaFull : ((j % 2 == 0) ? kQaoaLow : kQaoaHigh);
                    L.nt = b->cfg[nq].nt;
                    L.n = nq;
                    L.bytes = bytes_cost;
                    idx_t acc = 0;
                    for (size_t k : grp) {
                        QaoaInst r;
                        r.psi = reinterpret_cast<double2*>(off[k - first]);
                        const Graph& gr = b->graphs[b->gid[sel[k]]];
                        r.cost = L.kind == kQaoaHigh ? gr.high() : gr.d_cost;
                        r.item0 = acc;
                        r.n = nq;
                        r.pos = sel[k];
                        acc += qaoa_items(nq, C, L.kind);
                        pl.inst.push_back(r);
                    }
                    L.items = acc;
                    if (j + 1 == npass) {
                        L.partial_off = partial;
                        partial += (size_t)acc;
                        meas = L;
                    }
                    pl.launches.push_back(L);
                }
                meas.what = 1;
                pl.launches.push_back(meas);
            }
            while (g0 < last && b->n[sel[g0]] == nq) ++g0;
        }
        pl.partial = std::max(pl.partial, partial);
        first = last;
    }
    return pl;
}

// Fill a graph's costs in the orders of its passes for chunks of 2^C.
int fill_costs(orkan_qaoa* b, Graph& g, unsigned C) {
    const bool full = g.n <= C, bytes = g.cost_bytes == 1;
    const unsigned Cc = full ? g.n : C;
    for (unsigned kind : {(unsigned)kQaoaFull, (unsigned)kQaoaLow, (unsigned)kQaoaHigh}) {
        if (full != (kind == kQaoaFull)) continue;
        const idx_t count = idx_t(1) << (full ? g.n : g.n - 1);
        const unsigned grid = (unsigned)std::min<idx_t>((count + 255) / 256, (idx_t)sm_count() * 16);
        void* dst = kind == kQaoaHigh ? g.high() : g.d_cost;
        const QaoaGeo geo = qaoa_geo(g.n, Cc, kind);
        if (bytes) k_qaoa_cost<<<grid, 256, 0, b->cap>>>((uint8_t*)dst, geo, count, g.dev);
        else k_qaoa_cost<<<grid, 256, 0, b->cap>>>((double*)dst, geo, count, g.dev);
        if (const int rc = (int)cudaGetLastError()) return rc;
    }
    g.cost_C = C;
    return 0;
}

// The captured graph reads the buffers and the cost order of the plan that it was made for.
void drop_exec(orkan_qaoa* b) {
    if (b->exec) cudaGraphExecDestroy(b->exec);
    b->exec = nullptr;
}

// Device side of a plan: the costs in the order of its passes, arena, partial sums, launch
// shapes and the instance records.
int upload_plan(orkan_qaoa* b, Plan& pl) {
    int rc;
    drop_exec(b);
    bool filled = false;
    for (const auto& L : pl.launches) {
        if (L.what != 0) continue;
        for (unsigned k = L.inst_off; k < L.inst_off + L.ninst; ++k) {
            Graph& g = b->graphs[b->gid[pl.inst[k].pos]];
            const unsigned C = b->cfg[g.n].C;
            if (g.cost_C == C) continue;
            if ((rc = fill_costs(b, g, C))) return rc;
            filled = true;
        }
    }
    if (filled && (rc = (int)cudaStreamSynchronize(b->cap))) return rc;
    if (pl.arena > b->arena_bytes) {
        cudaFree(b->d_arena);
        b->d_arena = nullptr;
        b->arena_bytes = 0;
        if ((rc = dalloc(&b->d_arena, pl.arena))) return rc;
        b->arena_bytes = pl.arena;
    }
    if (pl.partial > b->partial_cap) {
        cudaFree(b->d_partial);
        b->d_partial = nullptr;
        b->partial_cap = 0;
        if ((rc = dalloc(&b->d_partial, pl.partial))) return rc;
        b->partial_cap = pl.partial;
    }
    for (auto& L : pl.launches) {
        if (L.what != 0) continue;
        if (L.items > 0xffffffffull / 4) return (int)cudaErrorInvalidConfiguration;     // 32-bit item counters
        L.smem = pass_smem(L.kind, L.C, L.bytes, b->tstride);
        L.grid = L.kind == kQaoaFull ? L.ninst : (unsigned)std::min<idx_t>(L.items, (idx_t)sm_count());
    }
    for (auto& r : pl.inst) r.psi = reinterpret_cast<double2*>(b->d_arena + reinterpret_cast<size_t>(r.psi));
    if (pl.inst.size() > b->inst_cap) {
        cudaFree(b->d_inst);
        b->d_inst = nullptr;
        b->inst_cap = 0;
        if ((rc = dalloc(&b->d_inst, pl.inst.size()))) return rc;
        b->inst_cap = pl.inst.size();
    }
    return (int)cudaMemcpy(b->d_inst, pl.inst.data(), pl.inst.size() * sizeof(QaoaInst), cudaMemcpyHostToDevice);
}

// The device work of a plan (no copies).
int enqueue_kernels(const orkan_qaoa* b, const Plan& pl, cudaStream_t st) {
    const QaoaTables T{b->d_table, b->d_rx, b->tstride};
    for (const auto& L : pl.launches) {
        const QaoaInst* inst = b->d_inst + L.inst_off;
        int rc = 0;
        if (L.what == 0) {
            QaoaPass P;
            P.inst = inst;
            P.ninst = L.ninst;
            P.items = L.items;
            P.gamma = b->d_gamma;
            P.partial = b->d_partial + L.partial_off;
            P.p = b->p;
            P.pass = L.pass;
            P.C = L.C;
            P.kind = L.kind;
            P.status = b->d_out + b->count;
            qaoa_pass_setup(P, L.n, L.bytes);
            P.wait_limit = b->polls;
            rc = L.bytes ? launch_pass_t<uint8_t>(b->split, L.nt, L.grid, L.smem, P, T, st)
                         : launch_pass_t<double>(b->split, L.nt, L.grid, L.smem, P, T, st);
        } else {
            k_qaoa_fold<<<L.ninst, kFoldThreads, 0, st>>>(inst, L.ninst, b->d_partial + L.partial_off, L.items, b->d_rx,
                                                          b->p, b->d_out);
            rc = (int)cudaGetLastError();
        }
        if (rc) return rc;
    }
    return 0;
}

int enqueue_tables(const orkan_qaoa* b, cudaStream_t st) {
    if (!b->any_bytes) return 0;
    k_qaoa_tables<<<b->count, 128, 0, st>>>(b->d_cmax, b->d_gamma, b->d_rx, b->count, b->p, b->tstride, b->d_table);
    return (int)cudaGetLastError();
}

// One evaluation: angles in, tables, the plan's kernels, means out.
int enqueue_run(const orkan_qaoa* b, const Plan& pl, cudaStream_t st) {
    const size_t np = (size_t)b->count * b->p;
    int rc;
    if ((rc = (int)cudaMemcpyAsync(b->d_gamma, b->h_gamma, np * 8, cudaMemcpyHostToDevice, st))) return rc;
    if ((rc = (int)cudaMemcpyAsync(b->d_rx, b->h_rx, np * sizeof(QaoaRx), cudaMemcpyHostToDevice, st))) return rc;
    if ((rc = enqueue_tables(b, st))) return rc;
    if ((rc = enqueue_kernels(b, pl, st))) return rc;
    return (int)cudaMemcpyAsync(b->h_out, b->d_out, ((size_t)b->count + 1) * 8, cudaMemcpyDeviceToHost, st);
}

int rebuild(orkan_qaoa* b) {
    std::vector<unsigned> sel(b->count);
    for (unsigned i = 0; i < b->count; ++i) sel[i] = i;
    std::stable_sort(sel.begin(), sel.end(), [&](unsigned a, unsigned c) { return b->n[a] > b->n[c]; });
    Plan pl = make_plan(b, sel);
    int rc = upload_plan(b, pl);
    if (rc) return rc;
    b->plan = pl;
    cudaGraph_t g = nullptr;
    if ((rc = (int)cudaStreamBeginCapture(b->cap, cudaStreamCaptureModeThreadLocal))) return rc;
    const int erc = enqueue_run(b, b->plan, b->cap);
    rc = (int)cudaStreamEndCapture(b->cap, &g);
    if (erc || rc) {
        if (g) cudaGraphDestroy(g);
        return erc ? erc : rc;
    }
    rc = (int)cudaGraphInstantiate(&b->exec, g, 0);
    if (rc) b->exec = nullptr;
    cudaGraphDestroy(g);
    return rc;
}

// The passes only ever set the status of their waits; whoever has read it set clears it.
int clear_status(const orkan_qaoa* b, cudaStream_t st) {
    const int rc = (int)cudaMemsetAsync(b->d_out + b->count, 0, 8, st);
    return rc ? rc : (int)cudaStreamSynchronize(st);
}

// Angles into the pinned staging buffers; rx coefficients with the host's libm, as the
// per-call rx takes them (cos(theta / 2), sin(theta / 2) with theta = 2 beta).
void stage_angles(orkan_qaoa* b, const double* gammas, const double* betas) {
    double c[64], s[64];
    for (unsigned i = 0; i < b->count; ++i) {
        const size_t row = (size_t)i * b->p;
        for (unsigned k = 0; k < b->p; ++k) {
            const double theta = 2.0 * betas[row + k];
            b->h_gamma[row + k] = gammas[row + k];
            c[k] = cos(theta / 2.0);
            s[k] = sin(theta / 2.0);
        }
        qaoa_rx_coeffs(c, s, b->p, b->n[i], b->cfg[b->n[i]].C, b->h_rx + row);
    }
}

std::string cache_key(const orkan_qaoa* b, unsigned nq, bool bytes) {
    cudaDeviceProp prop;
    cudaGetDeviceProperties(&prop, b->device);
    return std::string(prop.name) + "|n" + std::to_string(nq) + "|p" + std::to_string(b->p) + (bytes ? "|u8" : "|f64") + "|v3";
}

}  // namespace

extern "C" {

int orkan_qaoa_create(orkan_qaoa_t** out, unsigned count, const unsigned* n_qubits, const unsigned* edge_offsets,
                      const unsigned* edges, const double* weights, unsigned p, unsigned long long mem_budget,
                      unsigned flags) {
    if (!out) return (int)cudaErrorInvalidValue;
    *out = nullptr;
    if (!count || !n_qubits || !edge_offsets || p == 0 || p > 64) return (int)cudaErrorInvalidValue;
    for (unsigned i = 0; i < count; ++i) {
        if (n_qubits[i] < 1 || n_qubits[i] > 26 || edge_offsets[i + 1] < edge_offsets[i])
            return (int)cudaErrorInvalidValue;
        for (unsigned e = edge_offsets[i]; e < edge_offsets[i + 1]; ++e)
            if (!edges || edges[2 * e] >= n_qubits[i] || edges[2 * e + 1] >= n_qubits[i] ||
                edges[2 * e] == edges[2 * e + 1])
                return (int)cudaErrorInvalidValue;
    }
    orkan_qaoa* b = new orkan_qaoa();
    cudaGetDevice(&b->device);
    b->count = count;
    b->p = p;
    b->n.assign(n_qubits, n_qubits + count);
    for (unsigned q = 0; q <= 26; ++q) {
        b->cfg[q] = default_cfg(q);
    }
    // distinct graphs (same qubit count, edges in the same order, same weights)
    std::map<std::vector<unsigned char>, unsigned> seen;
    b->gid.resize(count);
    b->cmax.resize(count);
    unsigned cm_all = 0;
    int rc = 0;
    for (unsigned i = 0; i < count; ++i) {
        Graph g;
        g.n = n_qubits[i];
        double wsum = 0.0;
        bool integral = true;
        for (unsigned e = edge_offsets[i]; e < edge_offsets[i + 1]; ++e) {
            g.edges.push_back((unsigned char)edges[2 * e]);
            g.edges.push_back((unsigned char)edges[2 * e + 1]);
            const double w = weights ? weights[e] : 1.0;
            g.w.push_back(w);
            if (!(w >= 0.0 && w == std::floor(w))) integral = false;
            wsum += w;
        }
        g.cmax = (integral && wsum < kQaoaMaxTable && !(flags & ORKAN_QAOA_F64_COSTS)) ? (unsigned)wsum : 0xffffffffu;
        std::vector<unsigned char> key(1, (unsigned char)g.n);
        key.insert(key.end(), g.edges.begin(), g.edges.end());
        const unsigned char* wb = reinterpret_cast<const unsigned char*>(g.w.data());
        key.insert(key.end(), wb, wb + g.w.size() * 8);
        auto it = seen.find(key);
        unsigned id;
        if (it == seen.end()) {
            id = (unsigned)b->graphs.size();
            seen.emplace(key, id);
            b->graphs.push_back(g);
        } else {
            id = it->second;
        }
        b->gid[i] = id;
        b->cmax[i] = b->graphs[id].cmax;
        if (b->cmax[i] != 0xffffffffu) {
            cm_all = std::max(cm_all, b->cmax[i]);
            b->any_bytes = true;
        }
    }
    b->tstride = cm_all + 1;
    // resident costs, edges and weights of every graph (costs in whole 256-byte units)
    size_t cost_total = 0, ne = 0;
    for (auto& g : b->graphs) {
        g.cost_bytes = g.cmax != 0xffffffffu ? 1 : 8;
        cost_total += ((g.cost_bytes << g.n) + 255) & ~size_t(255);
        ne += g.w.size();
    }
    if ((rc = dalloc(&b->d_costs, cost_total)) || (rc = dalloc(&b->d_uv, 2 * ne)) || (rc = dalloc(&b->d_w, ne))) {
        orkan_qaoa_destroy(b);
        return rc;
    }
    {
        std::vector<unsigned char> uv;
        std::vector<double> w;
        size_t at = 0;
        for (auto& g : b->graphs) {
            g.d_cost = b->d_costs + at;
            at += ((g.cost_bytes << g.n) + 255) & ~size_t(255);
            g.dev = QaoaEdges{b->d_uv + uv.size(), b->d_w + w.size(), (unsigned)g.w.size()};
            uv.insert(uv.end(), g.edges.begin(), g.edges.end());
            w.insert(w.end(), g.w.begin(), g.w.end());
        }
        if (ne && ((rc = (int)cudaMemcpy(b->d_uv, uv.data(), uv.size(), cudaMemcpyHostToDevice)) ||
                   (rc = (int)cudaMemcpy(b->d_w, w.data(), w.size() * 8, cudaMemcpyHostToDevice)))) {
            orkan_qaoa_destroy(b);
            return rc;
        }
    }
    size_t freeb = 0, totalb = 0;
    cudaMemGetInfo(&freeb, &totalb);
    b->budget = mem_budget ? mem_budget : (unsigned long long)(0.6 * (double)freeb);
    const size_t np = (size_t)count * p;
    if ((rc = dalloc(&b->d_cmax, count)) || (rc = dalloc(&b->d_gamma, np)) || (rc = dalloc(&b->d_rx, np)) ||
        (rc = dalloc(&b->d_table, b->any_bytes ? np * b->tstride : 1)) || (rc = dalloc(&b->d_out, (size_t)count + 1)) ||
        (rc = (int)cudaMallocHost(&b->h_gamma, np * 8)) || (rc = (int)cudaMallocHost(&b->h_rx, np * sizeof(QaoaRx))) ||
        (rc = (int)cudaMallocHost(&b->h_out, ((size_t)count + 1) * 8)) ||
        (rc = (int)cudaMemset(b->d_out, 0, ((size_t)count + 1) * 8)) || (rc = prepare_kernels(&b->split)) ||
        (rc = (int)cudaStreamCreateWithFlags(&b->cap, cudaStreamNonBlocking))) {
        orkan_qaoa_destroy(b);
        return rc;
    }
    cudaMemcpy(b->d_cmax, b->cmax.data(), count * sizeof(unsigned), cudaMemcpyHostToDevice);
    memset(b->h_gamma, 0, np * 8);
    memset(b->h_rx, 0, np * sizeof(QaoaRx));
    if ((rc = rebuild(b))) {
        orkan_qaoa_destroy(b);
        return rc;
    }
    *out = b;
    return 0;
}

int orkan_qaoa_run(orkan_qaoa_t* b, const double* gammas, const double* betas, double* means, void* stream) {
    if (!b || !gammas || !betas || !means) return (int)cudaErrorInvalidValue;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    int rc = (int)cudaStreamSynchronize(st);                // the staging buffers may still be read
    if (rc) return rc;
    if (!b->exec && (rc = rebuild(b))) return rc;           // the last tuning ended in an error
    stage_angles(b, gammas, betas);
    if ((rc = (int)cudaGraphLaunch(b->exec, st))) return rc;
    if ((rc = (int)cudaStreamSynchronize(st))) return rc;
    if (b->h_out[b->count] != 0.0) {                        // a wait for staged data ran out
        rc = clear_status(b, st);
        return rc ? rc : (int)cudaErrorLaunchTimeout;
    }
    memcpy(means, b->h_out, (size_t)b->count * 8);
    return 0;
}

int orkan_qaoa_test_expire(orkan_qaoa_t* b, int on) {
    if (!b) return (int)cudaErrorInvalidValue;
    b->polls = on ? 0 : kQaoaPolls;
    return rebuild(b);
}

int orkan_qaoa_test_plain_registers(orkan_qaoa_t* b) {
    if (!b) return (int)cudaErrorInvalidValue;
    b->split = false;
    const int rc = prepare_plain();
    return rc ? rc : rebuild(b);
}

int orkan_qaoa_config(const orkan_qaoa_t* b, unsigned n, unsigned* log_chunk, unsigned* threads, unsigned* ring) {
    if (!b || n > 26) return (int)cudaErrorInvalidValue;
    if (log_chunk) *log_chunk = b->cfg[n].C;
    if (threads) *threads = b->cfg[n].nt;
    if (ring) *ring = b->cfg[n].ring;
    return 0;
}

int orkan_qaoa_stats(const orkan_qaoa_t* b, unsigned* waves, unsigned* launches) {
    if (!b) return (int)cudaErrorInvalidValue;
    if (waves) *waves = b->plan.waves;
    if (launches) *launches = (unsigned)b->plan.launches.size() + (b->any_bytes ? 1u : 0u);
    return 0;
}

int orkan_qaoa_cost_vector(orkan_qaoa_t* b, unsigned i, double* host_out) {
    if (!b || !host_out || i >= b->count) return (int)cudaErrorInvalidValue;
    const Graph& g = b->graphs[b->gid[i]];
    const idx_t dim = idx_t(1) << g.n;
    const bool full = g.n <= g.cost_C;
    const QaoaGeo geo = qaoa_geo(g.n, full ? g.n : g.cost_C, full ? kQaoaFull : kQaoaLow);
    double* out = nullptr;
    int rc = dalloc(&out, dim);
    if (rc) return rc;
    const idx_t count = full ? dim : dim / 2;
    const unsigned grid = (unsigned)std::min<idx_t>((count + 255) / 256, (idx_t)sm_count() * 16);
    if (g.cost_bytes == 1) k_qaoa_cost_vector<<<grid, 256, 0, b->cap>>>((const uint8_t*)g.d_cost, geo, count, out);
    else k_qaoa_cost_vector<<<grid, 256, 0, b->cap>>>((const double*)g.d_cost, geo, count, out);
    rc = (int)cudaGetLastError();
    if (!rc) rc = (int)cudaStreamSynchronize(b->cap);
    if (!rc) rc = (int)cudaMemcpy(host_out, out, dim * 8, cudaMemcpyDeviceToHost);
    cudaFree(out);
    return rc;
}

int orkan_qaoa_tune(orkan_qaoa_t* b, const double* gammas, const double* betas, const char* cache_path) {
    if (!b || !gammas || !betas) return (int)cudaErrorInvalidValue;
    std::vector<std::pair<unsigned, bool>> groups;          // distinct (qubit count, cost type)
    for (unsigned i = 0; i < b->count; ++i) {
        const auto key = std::make_pair(b->n[i], b->cmax[i] < kQaoaMaxTable);
        if (std::find(groups.begin(), groups.end(), key) == groups.end()) groups.push_back(key);
    }
    std::string cached;
    if (cache_path) {
        if (FILE* f = fopen(cache_path, "r")) {
            char line[512];
            while (fgets(line, sizeof line, f)) cached += line;
            fclose(f);
        }
    }
    stage_angles(b, gammas, betas);
    const size_t np = (size_t)b->count * b->p;
    int rc;
    if ((rc = (int)cudaMemcpyAsync(b->d_gamma, b->h_gamma, np * 8, cudaMemcpyHostToDevice, b->cap)) ||
        (rc = (int)cudaMemcpyAsync(b->d_rx, b->h_rx, np * sizeof(QaoaRx), cudaMemcpyHostToDevice, b->cap)) ||
        (rc = enqueue_tables(b, b->cap)) || (rc = (int)cudaStreamSynchronize(b->cap)))
        return rc;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    std::string append;
    for (const auto& grp : groups) {
        const unsigned nq = grp.first;
        const std::string key = cache_key(b, nq, grp.second);
        const size_t at = cached.find("\"" + key + "\"");
        QaoaCfg c{};
        if (at != std::string::npos &&
            sscanf(cached.c_str() + at + key.size() + 2, ": {\"C\": %u, \"threads\": %u, \"ring\": %u", &c.C, &c.nt,
                   &c.ring) == 3 &&
            c.C <= kQaoaMaxC && (c.C >= nq || (2 * c.C >= nq && c.C >= kQaoaMinC))) {
            b->cfg[nq] = cfg_for(nq, c.C);
            continue;
        }
        // up to 64 instances of the group, within one wave's budget
        std::vector<unsigned> sel;
        size_t bytes = 0;
        for (unsigned i = 0; i < b->count && sel.size() < 64; ++i)
            if (b->n[i] == nq && (b->cmax[i] < kQaoaMaxTable) == grp.second) {
                if (!sel.empty() && bytes + (size_t(1) << (nq - 1)) * 16 > b->budget) break;
                bytes += (size_t(1) << (nq - 1)) * 16;
                sel.push_back(i);
            }
        // candidates: chunks from the smallest that keeps the high pass possible (2C >= n)
        // up to 2^13 (a chunk of at least n qubits is the full pass, where only n matters)
        std::vector<QaoaCfg> cands;
        const unsigned c_lo = std::min(kQaoaMaxC, std::max(nq <= kQaoaMinC ? nq : kQaoaMinC, (nq + 1) / 2));
        for (unsigned Cc = c_lo; Cc <= kQaoaMaxC; ++Cc) {
            cands.push_back(cfg_for(nq, Cc));
            if (Cc >= nq) break;                            // a full pass: larger chunks change nothing
        }
        // three rounds over the candidates, interleaved, each timing three runs of the
        // sample; a candidate's figure is its median round, so that a drift of the clocks
        // or a single disturbed round does not decide.  The rx coefficients depend on the
        // chunk and are staged for each candidate.
        constexpr int kRounds = 3;
        std::vector<std::array<float, kRounds>> times(cands.size());
        std::vector<bool> usable(cands.size(), true);
        for (int round = 0; round < kRounds; ++round) {
            for (size_t ci = 0; ci < cands.size(); ++ci) {
                if (!usable[ci]) continue;
                b->cfg[nq] = cands[ci];
                stage_angles(b, gammas, betas);
                Plan pl = make_plan(b, sel);
                bool ok = upload_plan(b, pl) == 0 &&
                          cudaMemcpyAsync(b->d_rx, b->h_rx, np * sizeof(QaoaRx), cudaMemcpyHostToDevice, b->cap) == cudaSuccess;
                if (ok && round == 0) ok = enqueue_kernels(b, pl, b->cap) == 0;       // warm-up
                if (ok) ok = cudaEventRecord(e0, b->cap) == cudaSuccess;
                for (int r = 0; r < 3 && ok; ++r) ok = enqueue_kernels(b, pl, b->cap) == 0;
                if (ok) ok = cudaEventRecord(e1, b->cap) == cudaSuccess && cudaEventSynchronize(e1) == cudaSuccess;
                float ms = 0.f;
                if (ok) ok = cudaEventElapsedTime(&ms, e0, e1) == cudaSuccess;
                double expired = 0.0;                       // a candidate whose waits ran out was not timed
                if (ok) ok = cudaMemcpy(&expired, b->d_out + b->count, 8, cudaMemcpyDeviceToHost) == cudaSuccess;
                if (!ok || expired != 0.0) {
                    cudaGetLastError();
                    clear_status(b, b->cap);
                    usable[ci] = false;
                    continue;
                }
                times[ci][round] = ms;
            }
        }
        // the default stays unless a candidate's median beats the default's by the margin
        // (a sample of <= 64 instances times differently from box to box; small wins are noise)
        constexpr float kMargin = 0.93f;
        const QaoaCfg dflt = default_cfg(nq);
        float best = 1e30f, dflt_ms = 1e30f;
        QaoaCfg bestc = dflt;
        for (size_t ci = 0; ci < cands.size(); ++ci) {
            if (!usable[ci]) continue;
            auto t = times[ci];
            std::sort(t.begin(), t.end());
            const QaoaCfg& c = cands[ci];
            if (c.C == dflt.C && c.nt == dflt.nt && c.ring == dflt.ring) dflt_ms = t[kRounds / 2];
            if (t[kRounds / 2] < best) {
                best = t[kRounds / 2];
                bestc = c;
            }
        }
        if (dflt_ms < 1e29f && best > kMargin * dflt_ms) {
            bestc = dflt;
            best = dflt_ms;
        }
        b->cfg[nq] = bestc;
        if (best > 1e29f) continue;                         // nothing was timed: nothing to record
        char line[512];
        snprintf(line, sizeof line,
                 "{\"%s\": {\"C\": %u, \"threads\": %u, \"ring\": %u, \"ms_per_instance\": %.5f}}\n", key.c_str(),
                 bestc.C, bestc.nt, bestc.ring, best / 3 / (sel.empty() ? 1 : sel.size()));
        append += line;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (cache_path && !append.empty()) {
        if (FILE* f = fopen(cache_path, "a")) {
            fputs(append.c_str(), f);
            fclose(f);
        }
    }
    return rebuild(b);
}

void orkan_qaoa_destroy(orkan_qaoa_t* b) {
    if (!b) return;
    drop_exec(b);
    if (b->cap) cudaStreamDestroy(b->cap);
    cudaFree(b->d_costs);
    cudaFree(b->d_uv);
    cudaFree(b->d_w);
    cudaFree(b->d_cmax);
    cudaFree(b->d_gamma);
    cudaFree(b->d_rx);
    cudaFree(b->d_table);
    cudaFree(b->d_out);
    cudaFree(b->d_partial);
    cudaFree(b->d_arena);
    cudaFree(b->d_inst);
    cudaFreeHost(b->h_gamma);
    cudaFreeHost(b->h_rx);
    cudaFreeHost(b->h_out);
    delete b;
}

}  // extern "C"
