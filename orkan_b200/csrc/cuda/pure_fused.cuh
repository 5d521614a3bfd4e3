// pure_fused.cuh - several consecutive statevector gates in one pass over HBM.
//
// The reference applies every gate as its own pass over the 2^n amplitudes
// (src/gate/gate_pure.c:33-48, TRAVERSE_PURE_1Q, and the quarter/eighth loops of
// gate_pure.c:282-434).  Here a run of gates is applied chunk by chunk: a chunk is the set of
// 2^C amplitudes whose indices differ only in C chosen "local" qubits, it is loaded into
// shared memory once, every gate of the run is applied to it there, and it is stored once.
// Inside the chunk the run is cut into stages: a stage holds consecutive gates whose mixed
// qubits fit a group of K local qubits; every thread takes the 2^K amplitudes of a set that
// differ only in the group's qubits into registers, applies all of the stage's gates there,
// and puts them back, so the shared memory is read and written once per stage, not per gate.
// K = 4 where the state has many chunks: a gate's decoding is then shared by 16 amplitudes and
// a run has fewer stages.  K = 3 where one block holds the whole state (up to 12 qubits): the
// block then has twice the threads and each thread half the arithmetic, which is what a run
// waits for there.
//
// * A gate can join a run when the qubits it mixes are local: the target of X, Y, H, Hy, Rx,
//   Ry, CX, CY and CCX, both qubits of SWAP.  Controls and diagonal gates (Z, S, Sdg, T, Tdg,
//   P, Rz, CZ) may sit on any qubit: a non-local bit is constant over a chunk, so a non-local
//   control becomes a condition on the chunk and a non-local diagonal gate a factor applied
//   to the whole chunk (or to nothing).
// * The local set always holds the lowest qubits that are free, at least qubits 0-2, so a
//   chunk is made of contiguous runs of >= 8 amplitudes (128-byte lines): loads and stores
//   stay coalesced wherever the mixed qubits lie.
// * Every gate uses the same per-pair arithmetic as its one-gate kernel (pair_op of
//   pure.cuh), so a fused run gives bit-identical results to the gates applied one by one.
//
// The index logic is written as per-thread, per-phase __host__ __device__ functions so the
// CPU emulator of the test suite runs it with bounds-checked memory before any GPU run.
#pragma once

#include "common.cuh"
#include "pure.cuh"

#include "../../../include/orkan_cu.h"

namespace orkan {

constexpr unsigned kFuseMaxGates = 48;   // gates of one fused launch
constexpr unsigned kFuseMaxLog = 12;     // chunk of at most 2^12 amplitudes (64 KB)
constexpr unsigned kFuseThreads = 512;   // threads of a block at most
constexpr unsigned kFuseGroup = 4;       // local qubits of a register stage at most (16 amplitudes)

// What a gate does to a thread's registers v[j], j = the set's element.  A gate acts where the
// chunk has all bits of gmask, the set all bits of lm and the element all bits of jm.
enum FOp : unsigned char {
    kFMix = 0,          // + 4 op + rt: pair_op<op> on elements j, j | 1 << rt (X, Y, H, Hy, Rx, Ry)
    kFPhase = 24,       // + 5 k + (0: every element, 1 + b: those with bit b): the |1>-factor of diagonal op k
    kFCz = 54,          // sign of the elements with all bits of jm
    kFRz = 55,          // + b: Rz, the element's bit b picks the factor
    kFRzOut = 59,       // Rz, the set's bit lm or the chunk's bit gq - 1 picks the factor
    kFSwap = 60         // + 0..5: exchange of element bits (0,1) (0,2) (0,3) (1,2) (1,3) (2,3)
};

struct FGate {
    unsigned char h;           // FOp
    unsigned char jm;
    unsigned char gq;          // kFRzOut
    unsigned char pad_;
    unsigned lm;               // chunk-index bits outside the stage's group
    unsigned long long gmask;  // global bits
    double c, s;
};

struct FStage {
    unsigned char first;                   // first gate
    unsigned char g[kFuseGroup];           // local bits of the group, ascending
    unsigned char f[kFuseMaxLog];          // the other local bits: bit i of a set's number goes to bit f[i]
};

struct FusedPlan {
    unsigned n, C;             // qubits, log2 chunk
    unsigned ngates;
    unsigned nnl;              // non-local bits
    unsigned long long nlmask; // global bits that are not local (the chunk id's bits)
    unsigned char lq[kFuseMaxLog];   // global position of local bit i (ascending)
    unsigned char nlq[32];     // global position of chunk id bit i (the first 32)
    unsigned K;                // qubits of a stage's group
    unsigned nstages;
    bool din, dout;            // the first stage reads HBM, the last one writes HBM: fused_direct
    FStage st[kFuseMaxGates + 1];    // st[nstages].first = ngates
    FGate g[kFuseMaxGates];
    ORKAN_HD unsigned chunk() const { return 1u << C; }
    ORKAN_HD idx_t nchunks() const { return idx_t(1) << (n - C); }
    ORKAN_HD unsigned sets() const { return 1u << (C - K); }
};
static_assert(sizeof(FusedPlan) <= 4000, "a kernel parameter");

// Global qubits a gate mixes (must be local) as a bit mask; ~0 for an unknown op.
inline unsigned long long fused_need(const orkan_fgate_t& q) {
    switch (q.op) {
        case ORKAN_OP_X: case ORKAN_OP_Y: case ORKAN_OP_H: case ORKAN_OP_HY: case ORKAN_OP_RX: case ORKAN_OP_RY:
            return 1ull << q.q[0];
        case ORKAN_OP_Z: case ORKAN_OP_S: case ORKAN_OP_SDG: case ORKAN_OP_T: case ORKAN_OP_TDG: case ORKAN_OP_P:
        case ORKAN_OP_RZ: case ORKAN_FOP_CZ:
            return 0;
        case ORKAN_FOP_CX: case ORKAN_FOP_CY: return 1ull << q.q[1];
        case ORKAN_FOP_SWAP: return (1ull << q.q[0]) | (1ull << q.q[1]);
        case ORKAN_FOP_CCX: return 1ull << q.q[2];
        default: return ~0ull;
    }
}

inline unsigned fused_arity(int op) {
    return op < ORKAN_FOP_CX ? 1u : (op == ORKAN_FOP_CCX ? 3u : 2u);
}

// A stage moves its amplitudes between HBM and registers itself, without the shared memory, where its
// group leaves the lowest three qubits to the lanes: 8 lanes then have the 128 bytes of a line.  Not
// where one block holds the state: it has no other block to wait behind, and all its copies to shared memory in
// flight at once (200 gates at 12 qubits 162 us; 165 us with direct stages).
inline bool fused_direct(const FusedPlan& P, const FStage& st) {
    for (unsigned i = 0; i < P.K; ++i)
        if (st.g[i] < 3) return false;
    return P.C >= P.K + 3 && P.C < P.n;
}

// Build the plan of a run on an n-qubit statevector with chunks of 2^C amplitudes.  False
// when the run does not fit (too many mixed qubits, bad qubits or op codes, too many gates).
inline bool fused_plan(unsigned n, unsigned C, unsigned ngates, const orkan_fgate_t* gates, FusedPlan* P) {
    if (n < 1 || n > 62 || C < 1 || C > kFuseMaxLog || C > n || ngates < 1 || ngates > kFuseMaxGates) return false;
    const unsigned long long all = (n >= 64) ? ~0ull : ((1ull << n) - 1ull);
    unsigned long long need = 7ull & all;
    for (unsigned i = 0; i < ngates; ++i) {
        const orkan_fgate_t& q = gates[i];
        const unsigned k = fused_arity(q.op);
        if (q.op < 0 || (q.op > ORKAN_OP_P && q.op < ORKAN_FOP_CX) || q.op > ORKAN_FOP_CCX) return false;
        for (unsigned j = 0; j < k; ++j) {
            if (q.q[j] >= n) return false;
            for (unsigned l = 0; l < j; ++l) if (q.q[l] == q.q[j]) return false;
        }
        need |= fused_need(q);
    }
    if (popc64(need) > C) return false;
    for (unsigned b = 0; b < n && popc64(need) < C; ++b) need |= 1ull << b;   // lowest free bits
    P->n = n;
    P->C = C;
    P->ngates = ngates;
    P->nlmask = all & ~need;
    unsigned pos[64];
    unsigned i = 0;
    for (unsigned b = 0; b < n; ++b)
        if ((need >> b) & 1ull) { P->lq[i] = (unsigned char)b; pos[b] = i++; }
    P->nnl = n - C;
    for (unsigned b = 0, k = 0; b < n && k < 32; ++b)
        if ((P->nlmask >> b) & 1ull) P->nlq[k++] = (unsigned char)b;
    const unsigned most = C == n ? 3u : kFuseGroup;
    P->K = C < most ? C : most;
    // stages: consecutive gates whose mixed local bits fit a group of K bits; a group with fewer is
    // filled with the highest other local bits for the sake of fused_direct, or the lowest
    P->nstages = 0;
    unsigned cur = 0;
    auto close = [&](unsigned first, unsigned last) {
        for (unsigned b = 0; b < C && popc64(cur) < P->K; ++b) cur |= 1u << (C < n ? C - 1 - b : b);
        FStage& st = P->st[P->nstages++];
        st.first = (unsigned char)first;
        unsigned k = 0, e[kFuseMaxLog] = {};             // element bit of a local bit of the group
        for (unsigned b = 0; b < C; ++b)
            if ((cur >> b) & 1u) { e[b] = k; st.g[k++] = (unsigned char)b; }
        for (; k < kFuseGroup; ++k) st.g[k] = 0;
        // lanes: the three lowest bits of a set's number go to free bits of different residues mod 3
        // where there are such, which fused_phys spreads over the shared-memory banks
        unsigned left = (P->chunk() - 1) & ~cur, nf = 0;
        for (unsigned r = 0; r < 3; ++r)
            for (unsigned b = 0; b < C; ++b)
                if (((left >> b) & 1u) && b % 3 == r) {
                    st.f[nf++] = (unsigned char)b;
                    left &= ~(1u << b);
                    break;
                }
        for (unsigned b = 0; b < C; ++b)
            if ((left >> b) & 1u) st.f[nf++] = (unsigned char)b;
        for (; nf < kFuseMaxLog; ++nf) st.f[nf] = 0;
        for (unsigned gi = first; gi < last; ++gi) {
            const orkan_fgate_t& q = gates[gi];
            FGate f{};
            f.c = q.c;
            f.s = q.s;
            auto local = [&](unsigned b) { return ((need >> b) & 1ull) != 0; };
            auto grouped = [&](unsigned b) { return local(b) && ((cur >> pos[b]) & 1u); };
            auto bit = [&](unsigned b) { return e[pos[b]]; };
            auto control = [&](unsigned b) {
                if (grouped(b)) f.jm |= (unsigned char)(1u << bit(b));
                else if (local(b)) f.lm |= 1u << pos[b];
                else f.gmask |= 1ull << b;
            };
            switch (q.op) {
                case ORKAN_OP_X: case ORKAN_OP_Y: case ORKAN_OP_H: case ORKAN_OP_HY: case ORKAN_OP_RX: case ORKAN_OP_RY: {
                    const unsigned k6 = q.op == ORKAN_OP_X ? 0 : q.op == ORKAN_OP_Y ? 1 : q.op == ORKAN_OP_H ? 2
                                        : q.op == ORKAN_OP_HY ? 3 : q.op == ORKAN_OP_RX ? 4 : 5;
                    f.h = (unsigned char)(kFMix + 4 * k6 + bit(q.q[0]));
                    break;
                }
                case ORKAN_FOP_CX: case ORKAN_FOP_CY:
                    f.h = (unsigned char)(kFMix + 4 * (q.op == ORKAN_FOP_CX ? 0 : 1) + bit(q.q[1]));
                    control(q.q[0]);
                    break;
                case ORKAN_FOP_CCX:
                    f.h = (unsigned char)(kFMix + bit(q.q[2]));
                    control(q.q[0]);
                    control(q.q[1]);
                    break;
                case ORKAN_OP_Z: case ORKAN_OP_S: case ORKAN_OP_SDG: case ORKAN_OP_T: case ORKAN_OP_TDG: case ORKAN_OP_P: {
                    const unsigned k6 = q.op == ORKAN_OP_Z ? 0 : q.op == ORKAN_OP_S ? 1 : q.op == ORKAN_OP_SDG ? 2
                                        : q.op == ORKAN_OP_T ? 3 : q.op == ORKAN_OP_TDG ? 4 : 5;
                    if (grouped(q.q[0])) f.h = (unsigned char)(kFPhase + 5 * k6 + 1 + bit(q.q[0]));
                    else { f.h = (unsigned char)(kFPhase + 5 * k6); control(q.q[0]); }
                    break;
                }
                case ORKAN_FOP_CZ:
                    control(q.q[0]);
                    control(q.q[1]);
                    f.h = kFCz;
                    break;
                case ORKAN_OP_RZ:
                    if (grouped(q.q[0])) f.h = (unsigned char)(kFRz + bit(q.q[0]));
                    else {
                        f.h = kFRzOut;
                        if (local(q.q[0])) f.lm = 1u << pos[q.q[0]];
                        else f.gq = (unsigned char)(q.q[0] + 1);
                    }
                    break;
                default: {                               // SWAP
                    unsigned x = bit(q.q[0]), y = bit(q.q[1]);
                    if (x > y) { const unsigned t = x; x = y; y = t; }
                    f.h = (unsigned char)(kFSwap + (x == 0 ? y - 1 : x == 1 ? y + 1 : 5u));
                    break;
                }
            }
            P->g[gi] = f;
        }
        cur = 0;
    };
    unsigned first = 0;
    for (unsigned gi = 0; gi < ngates; ++gi) {
        unsigned mixed = 0;
        for (unsigned long long r = fused_need(gates[gi]); r; r &= r - 1) mixed |= 1u << pos[ctz64(r)];
        if (popc64(cur | mixed) > P->K) {
            close(first, gi);
            first = gi;
        }
        cur |= mixed;
    }
    close(first, ngates);
    P->st[P->nstages].first = (unsigned char)ngates;
    P->din = fused_direct(*P, P->st[0]);
    P->dout = fused_direct(*P, P->st[P->nstages - 1]);
    return true;
}

// Shared-memory slot of chunk index s: the low 3 bits XORed with the three 3-bit fields above
// them, so the 8 lanes of a quarter warp that differ in bits of distinct residues mod 3 (and
// any 8 consecutive indices) hit distinct 16-byte bank groups.
ORKAN_HD unsigned fused_phys(unsigned s) { return s ^ (((s >> 3) ^ (s >> 6) ^ (s >> 9)) & 7u); }

// Global index of the chunk's amplitude 0: the chunk id's bits deposited on the non-local bits.
ORKAN_HD idx_t fused_base(const FusedPlan& P, idx_t chunk) {
#ifdef __CUDA_ARCH__
    if (P.nnl <= 32) {                               // one bit per lane
        const unsigned lane = threadIdx.x & 31u;
        const idx_t one = lane < P.nnl && ((chunk >> lane) & 1u) ? idx_t(1) << P.nlq[lane] : 0;
        const unsigned lo = __reduce_or_sync(0xffffffffu, (unsigned)one);
        const unsigned hi = P.n <= 32 ? 0u : __reduce_or_sync(0xffffffffu, (unsigned)(one >> 32));
        return ((idx_t)hi << 32) | lo;
    }
#endif
    idx_t base = 0;
    unsigned long long rest = P.nlmask;
    while (rest && chunk) {
        const unsigned b = ctz64(rest);
        base |= (chunk & 1u) << b;
        chunk >>= 1;
        rest &= rest - 1ull;
    }
    return base;
}

// Global offset of chunk index j: its bits at the local bits' global positions.
ORKAN_HD idx_t fused_off(const FusedPlan& P, unsigned j) {
    idx_t o = 0;
#pragma unroll
    for (unsigned i = 0; i < kFuseMaxLog; ++i)
        if (i < P.C) o |= idx_t((j >> i) & 1u) << P.lq[i];
    return o;
}

// Chunk index of set r's element 0 in a stage.
template <int K>
ORKAN_HD unsigned fused_set(const FusedPlan& P, const FStage& st, unsigned r) {
    unsigned sb = 0;
#pragma unroll
    for (unsigned i = 0; i < kFuseMaxLog - K; ++i)
        if (i < P.C - K) sb |= ((r >> i) & 1u) << st.f[i];
    return sb;
}

// A thread's share of a chunk for load and store.  Through the shared memory: the 2^K amplitudes
// j = tid | u << (C - K), whose offsets and slots are those of tid with the bits of u added, so that an
// amplitude costs a few logic instructions.  Directly: the set of the stage.
struct FusedWalk {
    idx_t in, out;             // global offset of the share's amplitude 0
};
template <int K>
ORKAN_HD FusedWalk fused_walk(const FusedPlan& P, unsigned tid) {
    return {fused_off(P, P.din ? fused_set<K>(P, P.st[0], tid) : tid),
            fused_off(P, P.dout ? fused_set<K>(P, P.st[P.nstages - 1], tid) : tid)};
}
// f(u, global offset) of the 2^K elements whose bit b lies at local bit l(b).
template <int K, class L, class F>
ORKAN_HD void fused_spread(const FusedPlan& P, idx_t off, const L& l, const F& f) {
    idx_t go[K];
#pragma unroll
    for (int b = 0; b < K; ++b) go[b] = idx_t(1) << P.lq[l(b)];
#pragma unroll
    for (int u = 0; u < (1 << K); ++u) {
        idx_t o = off;
#pragma unroll
        for (int b = 0; b < K; ++b)
            if ((u >> b) & 1) o |= go[b];
        f(u, o);
    }
}
// f(global offset, slot) of the share that goes through the shared memory.
template <int K, class F>
ORKAN_HD void fused_each(const FusedPlan& P, idx_t off, unsigned tid, const F& f) {
    if (tid >= P.sets()) return;
    const unsigned slot = fused_phys(tid);
    unsigned so[K];
#pragma unroll
    for (int b = 0; b < K; ++b) so[b] = fused_phys(1u << (P.C - K + b));
    fused_spread<K>(P, off, [&](int b) { return P.C - K + b; }, [&](int u, idx_t o) {
        unsigned s = slot;
#pragma unroll
        for (int b = 0; b < K; ++b)
            if ((u >> b) & 1) s ^= so[b];
        f(o, s);
    });
}
// Mem::cp16(dst, x) copies amplitude x (asynchronously on the GPU).
template <int K, class Mem>
ORKAN_HD void fused_load(const Mem& mem, const FusedPlan& P, const FusedWalk& w, unsigned tid, idx_t base, double2* buf) {
    fused_each<K>(P, w.in, tid, [&](idx_t o, unsigned s) { mem.cp16(buf + s, base | o); });
}
template <int K, class Mem>
ORKAN_HD void fused_store(const Mem& mem, const FusedPlan& P, const FusedWalk& w, unsigned tid, idx_t base,
                          const double2* buf) {
    fused_each<K>(P, w.out, tid, [&](idx_t o, unsigned s) { mem.st(base | o, buf[s]); });
}

// ---- register stages -------------------------------------------------------------------
// v[j] holds the amplitude at chunk index sb | (bit b of j at group bit g[b]).

//
// Where a gate has a condition, the new value is computed and selected instead of branched to, and
// exchanges are selects on the condition even where there is none (`on` is then true, which the
// compiler cannot know).  A divergent branch, or an exchange that the compiler may carry out by
// renaming registers, makes it copy all 64 registers of the 16 amplitudes at the switch's ends:
// 284 instructions per H and 342 per X then, 92 and 150 now (64 and 0 of them arithmetic).
ORKAN_HD double2 reg_select(bool p, double2 a, double2 b) { return c2(p ? a.x : b.x, p ? a.y : b.y); }

// X and Y on element bit RT where the set (on) and the element have the controls.
template <int OP, int RT, int NV>
ORKAN_HD void reg_flip(double2 (&v)[NV], const FGate& g, bool on) {
    if constexpr ((1 << RT) < NV) {
#pragma unroll
        for (int j = 0; j < NV; ++j)
            if (!(j & (1 << RT))) {
                const bool p = on && (j & g.jm) == g.jm;
                const double2 a = v[j], b = v[j | (1 << RT)];
                double2 na = a, nb = b;
                pair_op<OP>(na, nb, 0.0, 0.0);
                v[j] = reg_select(p, na, a);
                v[j | (1 << RT)] = reg_select(p, nb, b);
            }
    }
}

// H, Hy, Rx, Ry on element bit RT (they have no controls).
template <int OP, int RT, int NV>
ORKAN_HD void reg_mix(double2 (&v)[NV], const FGate& g) {
    if constexpr ((1 << RT) < NV) {
#pragma unroll
        for (int j = 0; j < NV; ++j)
            if (!(j & (1 << RT))) pair_op<OP>(v[j], v[j | (1 << RT)], g.c, g.s);
    }
}

// A diagonal 1-qubit op's |1>-factor on the elements with bit B (no condition then), or, B < 0, on all
// elements of the sets that have the bit (on).
template <int OP, int B, int NV>
ORKAN_HD void reg_phase(double2 (&v)[NV], const FGate& g, bool on) {
    if constexpr (B < 0 || (1 << (B < 0 ? 0 : B)) < NV) {
        constexpr bool plain = B >= 0 && OP != kOpS && OP != kOpSdg;     // S exchanges re and im
#pragma unroll
        for (int j = 0; j < NV; ++j)
            if (B < 0 || ((j >> (B < 0 ? 0 : B)) & 1)) {
                double2 a = c2(0.0, 0.0), x = v[j];
                pair_op<OP>(a, x, g.c, g.s);
                v[j] = plain ? x : reg_select(on, x, v[j]);
            }
    }
}

template <int NV>
ORKAN_HD void reg_cz(double2 (&v)[NV], const FGate& g, bool on) {
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        double2 a = c2(0.0, 0.0), x = v[j];
        pair_op<kOpZ>(a, x, 0.0, 0.0);
        v[j] = reg_select(on && (j & g.jm) == g.jm, x, v[j]);
    }
}

// Rz: the |1> factor is the |0> factor with s negated, (c x + s y, c y - s x) -> (c x - s y, c y + s x),
// the same roundings as pair_op<kOpRz>.  B < 0: every element takes the factor that `one` picks.
template <int B, int NV>
ORKAN_HD void reg_rz(double2 (&v)[NV], const FGate& g, bool one) {
    if constexpr (B < 0 || (1 << (B < 0 ? 0 : B)) < NV) {
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const double s = (B < 0 ? one : (bool)((j >> (B < 0 ? 0 : B)) & 1)) ? -g.s : g.s;
            v[j] = c2(lin2(g.c, v[j].x, s, v[j].y), lin2(g.c, v[j].y, -s, v[j].x));
        }
    }
}

template <int X, int Y, int NV>
ORKAN_HD void reg_swap(double2 (&v)[NV], bool on) {
    if constexpr ((1 << Y) < NV) {
#pragma unroll
        for (int j = 0; j < NV; ++j)
            if (!(j & (1 << X)) && !(j & (1 << Y))) {
                const double2 a = v[j | (1 << X)], b = v[j | (1 << Y)];
                v[j | (1 << X)] = reg_select(on, b, a);
                v[j | (1 << Y)] = reg_select(on, a, b);
            }
    }
}

// One gate of a stage on a thread's registers: one jump per gate, everything a case needs known
// at compile time but the angles and conditions.
template <int NV>
ORKAN_HD void fused_apply(const FGate& g, double2 (&v)[NV], unsigned sb, idx_t base) {
    if ((base & g.gmask) != g.gmask) return;                 // the same for the whole block
    const bool on = g.h == kFRzOut || (sb & g.lm) == g.lm;
    switch (g.h) {
#define ORKAN_RT(F, K6, OP, A) \
    case kFMix + 4 * K6: F<OP, 0> A; break; \
    case kFMix + 4 * K6 + 1: F<OP, 1> A; break; \
    case kFMix + 4 * K6 + 2: F<OP, 2> A; break; \
    case kFMix + 4 * K6 + 3: F<OP, 3> A; break;
        ORKAN_RT(reg_flip, 0, kOpX, (v, g, on)) ORKAN_RT(reg_flip, 1, kOpY, (v, g, on))
        ORKAN_RT(reg_mix, 2, kOpH, (v, g)) ORKAN_RT(reg_mix, 3, kOpHy, (v, g))
        ORKAN_RT(reg_mix, 4, kOpRx, (v, g)) ORKAN_RT(reg_mix, 5, kOpRy, (v, g))
#undef ORKAN_RT
#define ORKAN_PH1(K6, OP, B) case kFPhase + 5 * K6 + 1 + (B): reg_phase<OP, B>(v, g, on); break;
#define ORKAN_PH(K6, OP) ORKAN_PH1(K6, OP, -1) ORKAN_PH1(K6, OP, 0) ORKAN_PH1(K6, OP, 1) ORKAN_PH1(K6, OP, 2) \
    ORKAN_PH1(K6, OP, 3)
        ORKAN_PH(0, kOpZ) ORKAN_PH(1, kOpS) ORKAN_PH(2, kOpSdg) ORKAN_PH(3, kOpT) ORKAN_PH(4, kOpTdg) ORKAN_PH(5, kOpP)
#undef ORKAN_PH
#undef ORKAN_PH1
        case kFCz: reg_cz(v, g, on); break;
        case kFRz: reg_rz<0>(v, g, false); break;
        case kFRz + 1: reg_rz<1>(v, g, false); break;
        case kFRz + 2: reg_rz<2>(v, g, false); break;
        case kFRz + 3: reg_rz<3>(v, g, false); break;
        case kFRzOut: reg_rz<-1>(v, g, (sb & g.lm) != 0 || (g.gq && ((base >> (g.gq - 1)) & 1u))); break;
        case kFSwap: reg_swap<0, 1>(v, on); break;
        case kFSwap + 1: reg_swap<0, 2>(v, on); break;
        case kFSwap + 2: reg_swap<0, 3>(v, on); break;
        case kFSwap + 3: reg_swap<1, 2>(v, on); break;
        case kFSwap + 4: reg_swap<1, 3>(v, on); break;
        case kFSwap + 5: reg_swap<2, 3>(v, on); break;
        default: break;
    }
}

// Stage s of the run on a chunk (all threads of the block; a barrier follows).
// Thread tid takes set tid: the set's 2^K amplitudes go to registers, every gate of the stage
// whose chunk condition holds is applied, and they go back; the first stage reads HBM and the last
// one writes it where they are direct.  The swizzle is
// linear over disjoint bits, so element j lies at phys(sb) ^ phys(its group bits).
template <int K, class Mem>
ORKAN_HD void fused_stage_k(const Mem& mem, const FusedPlan& P, const FusedWalk& w, unsigned s, idx_t base, double2* buf,
                            unsigned r) {
    constexpr int NV = 1 << K;
    const FStage& st = P.st[s];
    const unsigned g0 = st.first, g1 = P.st[s + 1].first;
    unsigned ph[K];
#pragma unroll
    for (int b = 0; b < K; ++b) ph[b] = fused_phys(1u << st.g[b]) * 16u;
    if (r >= P.sets()) return;
    const unsigned sb = fused_set<K>(P, st, r), psb = fused_phys(sb) * 16u;
    unsigned char* raw = reinterpret_cast<unsigned char*>(buf);
    auto at = [&](int j) -> double2& {
        unsigned a = psb;
#pragma unroll
        for (int b = 0; b < K; ++b)
            if ((j >> b) & 1) a ^= ph[b];
        return *reinterpret_cast<double2*>(raw + a);
    };
    auto bit = [&](int b) { return (unsigned)st.g[b]; };
    double2 v[NV];
    if (s == 0 && P.din) {
        fused_spread<K>(P, base | w.in, bit, [&](int j, idx_t o) { v[j] = mem.ld(o); });
    } else {
#pragma unroll
        for (int j = 0; j < NV; ++j) v[j] = at(j);
    }
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
    for (unsigned gi = g0; gi < g1; ++gi) fused_apply(P.g[gi], v, sb, base);
    if (s + 1 == P.nstages && P.dout) {
        fused_spread<K>(P, base | w.out, bit, [&](int j, idx_t o) { mem.st(o, v[j]); });
    } else {
#pragma unroll
        for (int j = 0; j < NV; ++j) at(j) = v[j];
    }
}

// Shared memory of one block: the chunk.
ORKAN_HD size_t fused_smem_bytes(const FusedPlan& P) { return (size_t)P.chunk() * sizeof(double2); }

// Threads of a block: one set each, whole warps (at most kFuseThreads: 2^12 amplitudes, K >= 3).
inline unsigned fused_threads(const FusedPlan& P) { return P.sets() < 32 ? 32u : P.sets(); }

#ifdef __CUDACC__
struct FusedDevMem {
    double2* p;
    __device__ __forceinline__ double2 ld(idx_t i) const { return p[i]; }
    __device__ __forceinline__ void st(idx_t i, double2 v) const { p[i] = v; }
    __device__ __forceinline__ void cp16(double2* dst, idx_t i) const {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                     "l"(p + i) : "memory");
    }
};

// Persistent blocks walk the chunks; every gate whose chunk condition holds is applied in
// shared memory between one load and one store of the chunk.
//
// Bound: instructions and their latency at 4 warps per scheduler (128 registers: 16 amplitudes); 45 % of the
// issue slots are used, 18 % of FP64, a third of HBM.  At 28 qubits HBM takes 1.32 ms of a run, 8 gates of one
// stage hide under it (1.39 ms), 16 H take 1.89 ms, further ones 80 us each.  200 random gates: 30 qubits
// 208.7 ms with 8-amplitude sets whose gates copied registers, 124.7 ms with 16-amplitude sets, 122 ms
// with direct stages (both measured side by side: 125.9 and 122.3); 12 qubits, one block, 117 us on the GPU (277).  Fetching the next chunk to L2 ahead
// and letting half of the blocks start later gave nothing; chunks of 2^12 save a fifth of the runs but leave two
// blocks per SM (118.4 against 116.9 ms for 192 gates).
template <int K>
__global__ void __launch_bounds__(K == 4 ? 256 : kFuseThreads, K == 4 ? 2 : 1)
    k_pure_fused(FusedDevMem mem, const __grid_constant__ FusedPlan P) {
    extern __shared__ __align__(128) double2 fbuf[];
    const unsigned tid = threadIdx.x;
    const FusedWalk w = fused_walk<K>(P, tid);
    const idx_t nch = P.nchunks();
    const bool alone = P.nstages == 1 && P.din && P.dout;    // the chunk never meets the shared memory
    for (idx_t ch = blockIdx.x; ch < nch; ch += gridDim.x) {
        const idx_t base = fused_base(P, ch);
        if (!P.din) {
            fused_load<K>(mem, P, w, tid, base, fbuf);
            asm volatile("cp.async.wait_all;\n" ::: "memory");
            __syncthreads();
        }
        for (unsigned st = 0; st < P.nstages; ++st) {
            fused_stage_k<K>(mem, P, w, st, base, fbuf, tid);
            if (!alone) __syncthreads();
        }
        if (!P.dout) {
            fused_store<K>(mem, P, w, tid, base, fbuf);
            __syncthreads();
        }
    }
}
#endif

}  // namespace orkan
