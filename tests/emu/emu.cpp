// emu.cpp - CPU emulation of the CUDA kernels' index logic -- TEST INFRASTRUCTURE ONLY.
//
// The kernels in orkan_b200/csrc/cuda are written as __host__ __device__ per-thread
// (and per-phase) functions over a memory accessor.  This file instantiates the same
// functions with a checking accessor and runs every thread of every block on the CPU,
// with block barriers honoured by running each phase for all threads before the next.
// The accessor rejects out-of-range indices and counts reads and writes per element, so
// the tests can prove, before any GPU run, that every access of a launch stays inside
// the storage and that each stored element is read and written exactly as often as the
// layout's ownership rules require.  It is never used by the product library.
#include "../../orkan_b200/csrc/cuda/common.cuh"
#include "../../orkan_b200/csrc/cuda/dm_direct.cuh"
#include "../../orkan_b200/csrc/cuda/dm_engine.cuh"
#include "../../orkan_b200/csrc/cuda/dm_phase.cuh"
#include "../../orkan_b200/csrc/cuda/pure.cuh"
#include "../../orkan_b200/csrc/cuda/pure_fused.cuh"
#include "../../orkan_b200/csrc/cuda/qaoa.cuh"

#include <stdint.h>
#include <stdlib.h>
#include <string.h>
#include <vector>

using namespace orkan;

namespace {

struct EmuMem {
    double2* p;
    idx_t len;
    uint32_t* reads;
    uint32_t* writes;
    uint64_t* oob;
    double2 ld(idx_t i) const {
        if (i >= len) { ++*oob; return c2(0.0, 0.0); }
        ++reads[i];
        return p[i];
    }
    void st(idx_t i, double2 v) const {
        if (i >= len) { ++*oob; return; }
        ++writes[i];
        p[i] = v;
    }
    // asynchronous copy of the GPU path: lands immediately here; counted as one read per
    // element even when an element is copied to two shared-memory slots
    void cp(double2* dst, idx_t i) const {
        if (i >= len) { ++*oob; return; }
        if (i != last_cp) ++reads[i];
        last_cp = i;
        *dst = p[i];
    }
    mutable idx_t last_cp = ~idx_t(0);
    void cp16(double2* dst, idx_t i) const {
        if (i >= len) { ++*oob; return; }
        ++reads[i];
        *dst = p[i];
    }
    // asynchronous copy of a phase-table entry (not state storage): lands immediately here
    void cpg(double2* dst, const double2* src) const { *dst = *src; }
    // bulk copies of the GPU path (TMA): n consecutive elements, land immediately here
    void bulk_load(double2* sdst, idx_t i, unsigned n, void*) const {
        for (unsigned k = 0; k < n; ++k) sdst[k] = ld(i + k);
    }
    void bulk_store(idx_t i, const double2* ssrc, unsigned n) const {
        for (unsigned k = 0; k < n; ++k) st(i + k, ssrc[k]);
    }
};

struct EmuMemR {
    const double* p;
    idx_t len;
    uint64_t* oob;
    double ld(idx_t i) const {
        if (i >= len) { ++*oob; return 0.0; }
        return p[i];
    }
};

struct EmuMemC2 {
    const double2* p;
    idx_t len;
    uint64_t* oob;
    double2 ld(idx_t i) const {
        if (i >= len) { ++*oob; return c2(0.0, 0.0); }
        return p[i];
    }
};

// Cost accessor of the QAOA stages: the FP64 or byte cost i of an item whose costs start at
// base, or the 2^K byte costs at i (a multiple of 2^K) as words.
template <class CostT>
struct EmuCost {
    const CostT* p;
    idx_t base, len;
    uint64_t* oob;
    CostT ld(idx_t i) const {
        if (base + i >= len) { ++*oob; return CostT(0); }
        return p[base + i];
    }
    template <int K>
    void words(uint32_t* w, idx_t i) const {
        const idx_t nb = idx_t(1) << K;
        if ((base + i) % nb || base + i + nb > len) { ++*oob; return; }
        w[0] = 0;
        memcpy(w, reinterpret_cast<const uint8_t*>(p) + base + i, nb);
    }
};

constexpr unsigned kSms = 148;

unsigned grid_for(idx_t per_block, idx_t total, unsigned cap) {
    idx_t g = (total + per_block - 1) / per_block;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return (unsigned)g;
}

double2 ldc(const double* p, unsigned i) { return c2(p[2 * i], p[2 * i + 1]); }

// The operation phase of an item for all threads; a chain runs stage by stage.
template <class Op>
bool run_stages(const Op&, const DmGeom&, double2*, unsigned) { return false; }
bool run_stages(const OpChain& op, const DmGeom& g, double2* vb, unsigned nthr) {
    for (unsigned i = 0; i < op.nst; ++i)
        for (unsigned t = 0; t < nthr; ++t) op.stage(i, g, vb, t, nthr);
    return true;
}

template <class Map, class Op>
void run_engine(const EmuMem& mem, const Map& map, const DmGeom& g, const Op& op) {
    const unsigned grid = grid_for(1, g.items, kSms * 32u);
    std::vector<double2> vb((size_t)g.V() * g.P());
    std::vector<DmPos> pd(kDmMaxPos + 1);
    Op o = op;
    dm_orient(o, !Map::kMirrors);           // the packed layout stages rho^T
    for (unsigned b = 0; b < grid; ++b) {
        for (idx_t w = b; w < g.items; w += grid) {
            for (int phase = 0; phase < kDmPhases; ++phase) {
                const unsigned nthr = (phase == 1 || phase == 5) ? kDmIssueThreads : kDmBlock;
                if (phase == 3 && run_stages(o, g, vb.data(), nthr)) continue;
                for (unsigned t = 0; t < nthr; ++t)
                    dm_engine_item_phase(phase, mem, map, g, o, w, pd.data(), vb.data(), t, nthr);
            }
        }
    }
}

template <class Op>
int engine_dispatch(int layout, unsigned log_tile, double* rho, idx_t len, unsigned n, const DmGeom& g,
                    const Op& op, uint32_t* reads, uint32_t* writes, uint64_t* oob) {
    EmuMem mem{reinterpret_cast<double2*>(rho), len, reads, writes, oob};
    if (layout == 1) run_engine(mem, PackedMap{idx_t(1) << n}, g, op);
    else run_engine(mem, TiledMap{idx_t(1) << n, log_tile}, g, op);
    return 0;
}

unsigned ls_max_for(int layout, unsigned log_tile) { return layout == 2 ? log_tile : 6u; }

// block-side cap of the engine (the GPU default 64, or ORKAN_DM_MAX_V)
unsigned emu_max_v() {
    unsigned x = 64;
    if (const char* e = getenv("ORKAN_DM_MAX_V")) {
        const unsigned y = (unsigned)atoi(e);
        if (y == 8 || y == 16 || y == 32 || y == 64) x = y;
    }
    return x;
}

template <class Factor>
void run_phase(int layout, unsigned log_tile, const EmuMem& mem, unsigned n, const Factor& fac) {
    if constexpr (std::is_same<Factor, GateFactor1>::value) {
        if (layout == 1 && n > 10) {                    // as the GPU launcher picks it
            for (idx_t b = 0; b < phase_column_blocks(n); ++b)
                for (unsigned t = 0; t < kColThreads; ++t) dm_phase_columns(mem, PackedMap{idx_t(1) << n}, fac, b, t);
            return;
        }
    }
    const PhaseGeom g = phase_geometry(n, layout == 2 ? log_tile : 5u);
    const unsigned grid = grid_for(1, g.items, kSms * 32u);
    for (unsigned b = 0; b < grid; ++b)
        for (idx_t w = b; w < g.items; w += grid) {
            double2 srow[32], scol[32];
            for (unsigned t = 0; t < kPhaseThreads; ++t) dm_phase_stage(g, fac, w, srow, scol, t, kPhaseThreads);
            for (unsigned t = 0; t < kPhaseThreads; ++t) {
                if (layout == 1) dm_phase_item(mem, PackedMap{idx_t(1) << n}, g, fac, w, t, kPhaseThreads, srow, scol);
                else dm_phase_item(mem, TiledMap{idx_t(1) << n, log_tile}, g, fac, w, t, kPhaseThreads, srow, scol);
            }
        }
}


// One instance through the fused QAOA passes 0..upto (the GPU launch plan with a single
// instance): full pass when n <= C, else p + 1 low/high passes of 2^C-slot items over the
// stored half of the state.  psi, reads and writes are given for all 2^n basis states: each
// gets what its stored image holds.
template <class CostT>
int run_qaoa(unsigned n, const CostT* cost, unsigned p, const double* gamma, const double* beta, unsigned C,
             unsigned nthr, unsigned upto, double* psi, double* mean, uint32_t* reads, uint32_t* writes,
             uint64_t* oob) {
    const bool full = n <= C;
    if (p == 0 || nthr % 32 || (!full && 2 * C < n) || C > kQaoaMaxC) return -1;
    const idx_t dim = idx_t(1) << n, half = full ? 0 : dim / 2;
    std::vector<double> co(p), si(p);
    for (unsigned k = 0; k < p; ++k) {
        co[k] = cos(2.0 * beta[k] / 2.0);
        si[k] = sin(2.0 * beta[k] / 2.0);
    }
    std::vector<QaoaRx> rx(p);
    qaoa_rx_coeffs(co.data(), si.data(), p, n, C, rx.data());
    std::vector<double2> table(1, c2(1.0, 0.0));
    unsigned tstride = 1;
    if (sizeof(CostT) == 1) {
        unsigned cmax = 0;
        for (idx_t x = 0; x < dim; ++x) cmax = cost[x] > cmax ? (unsigned)cost[x] : cmax;
        tstride = cmax + 1;
        table.assign((size_t)p * tstride, c2(0.0, 0.0));
        for (unsigned k = 0; k < p; ++k)
            for (unsigned c = 0; c <= cmax; ++c) {
                double sn, cs;
                sincos((double)c * gamma[k], &sn, &cs);
                table[(size_t)k * tstride + c] = c2(cs * rx[k].fs, sn * rx[k].fs);
            }
    }
    std::vector<double2> st((size_t)half);
    std::vector<uint32_t> rd((size_t)half), wr((size_t)half);
    const EmuMem mem{st.data(), half, rd.data(), wr.data(), oob};
    QaoaInst I;
    I.psi = st.data();
    I.item0 = 0;
    I.n = n;
    I.pos = 0;
    const unsigned npass = full ? 1 : p + 1;
    for (unsigned j = 0; j < npass && j <= upto; ++j) {
        QaoaPass P;
        P.inst = &I;
        P.ninst = 1;
        P.kind = full ? kQaoaFull : ((j % 2 == 0) ? kQaoaLow : kQaoaHigh);
        P.C = full ? n : C;
        P.items = qaoa_items(n, P.C, P.kind);
        P.gamma = gamma;
        P.p = p;
        P.pass = full ? 0 : j;
        qaoa_pass_setup(P, n);
        const QaoaTables T{table.data(), rx.data(), tstride};
        // the costs in the order of the pass, as the batch context makes them
        const idx_t ncost = full ? dim : half;
        std::vector<CostT> ordered((size_t)ncost);
        for (idx_t i = 0; i < ncost; ++i) ordered[(size_t)i] = cost[qaoa_cost_state(P.geo, sizeof(CostT) == 1, i)];
        I.cost = ordered.data();
        const unsigned lc = qaoa_lc(n, P.C, P.kind);
        std::vector<double2> vb((size_t)1 << lc);
        double sum = 0.0;
        for (idx_t w = 0; w < P.items; ++w) {
            std::vector<double> acc(nthr, 0.0);
            const EmuCost<CostT> cm{ordered.data(), full ? 0 : w << P.C, ncost, oob};
            if (full) {
                for (unsigned r = 0; r < qaoa_full_stages(P.geo.m, p); ++r)
                    for (unsigned t = 0; t < nthr; ++t)
                        acc[t] = qaoa_full_stage<CostT>(P, T, 0, n, r, cm, vb.data(), t, nthr);
            } else {
                const QaoaItem J = qaoa_item(P, T, I, w, sizeof(CostT));
                if (P.layer_a >= 0)
                    for (unsigned t = 0; t < nthr; ++t) qaoa_fill(P.geo, mem, J.item, vb.data(), nullptr, t, nthr);
                for (unsigned r = 0; r < P.nreg; ++r)
                    for (unsigned t = 0; t < nthr; ++t)
                        acc[t] = qaoa_stage<CostT>(P, r, J, mem, cm, vb.data(), table.data() + (P.layer_phase < 0 ? 0 : P.layer_phase) * tstride,
                                                   lc, t, nthr, QaoaNoRelease{});
            }
            for (unsigned t = 0; t < nthr; ++t) sum += acc[t];
        }
        if (full || j == p) *mean = sum * rx[p - 1].fm;
    }
    if (!full)
        for (idx_t x = 0; x < dim; ++x) {
            const idx_t i = qaoa_index_of(n, C, x);
            reinterpret_cast<double2*>(psi)[x] = st[(size_t)i];
            reads[x] = rd[(size_t)i];
            writes[x] = wr[(size_t)i];
        }
    return 0;
}

// Slots that thread t of nthr touches in group gi of a chunked item, marked with its half-warp.
template <int K, int B0>
void mark_s(const QaoaGeo& g, std::vector<unsigned>& own) {
    for (unsigned r = 0; r < (1u << (g.C - K)); ++r)
        for (unsigned e = 0; e < (1u << K); ++e) own[qaoa_s_base<K, B0>(g.MM, r) + (e << B0)] = r >> 4;
}

}  // namespace

extern "C" {

// All entry points: data arrays are interleaved complex; reads/writes are per-element
// counters (zeroed by the caller); *oob receives the number of out-of-range accesses.
// Return 0, or -1 when the launch parameters are rejected (as the CUDA layer would).

int emu_dm_unitary(int layout, unsigned log_tile, double* rho, uint64_t len, unsigned n, unsigned k,
                   const unsigned* qubits, const double* u, uint32_t* reads, uint32_t* writes, uint64_t* oob) {
    DmGeom g;
    if (!dm_geometry(n, k, qubits, ls_max_for(layout, log_tile), &g, emu_max_v())) return -1;
    if (k == 1) {
        OpMix1 op;
        for (unsigned i = 0; i < 4; ++i) op.u[i] = ldc(u, i);
        return engine_dispatch(layout, log_tile, rho, len, n, g, op, reads, writes, oob);
    }
    OpMix2 op;
    for (unsigned i = 0; i < 16; ++i) op.u[i] = ldc(u, i);
    return engine_dispatch(layout, log_tile, rho, len, n, g, op, reads, writes, oob);
}

int emu_dm_monomial(int layout, unsigned log_tile, double* rho, uint64_t len, unsigned n, unsigned k,
                    const unsigned* qubits, const unsigned* src, const double* phase, uint32_t* reads,
                    uint32_t* writes, uint64_t* oob) {
    OpMonomial op;
    for (unsigned y = 0; y < 8; ++y) { op.src[y] = y; op.phase[y] = c2(1.0, 0.0); }
    for (unsigned y = 0; y < (1u << k); ++y) { op.src[y] = src[y]; op.phase[y] = ldc(phase, y); }
    DmGeom g;
    if (!dm_monomial_setup(n, k, qubits, op, ls_max_for(layout, log_tile), emu_max_v(), &g)) return -1;
    return engine_dispatch(layout, log_tile, rho, len, n, g, op, reads, writes, oob);
}

int emu_dm_superop1(int layout, unsigned log_tile, double* rho, uint64_t len, unsigned n, unsigned target,
                    const double* sop, uint32_t* reads, uint32_t* writes, uint64_t* oob) {
    OpSuper1 op;
    for (unsigned i = 0; i < 16; ++i) op.s[i] = ldc(sop, i);
    DmGeom g;
    const unsigned q[1] = {target};
    if (!dm_geometry(n, 1, q, ls_max_for(layout, log_tile), &g, emu_max_v())) return -1;
    return engine_dispatch(layout, log_tile, rho, len, n, g, op, reads, writes, oob);
}

int emu_dm_superop2(int layout, unsigned log_tile, double* rho, uint64_t len, unsigned n, unsigned q0, unsigned q1,
                    const double* sop, uint32_t* reads, uint32_t* writes, uint64_t* oob) {
    OpSuper2 op;
    for (unsigned i = 0; i < 256; ++i) op.s[i] = ldc(sop, i);
    DmGeom g;
    const unsigned q[2] = {q0, q1};
    if (!dm_geometry(n, 2, q, ls_max_for(layout, log_tile), &g, emu_max_v())) return -1;
    return engine_dispatch(layout, log_tile, rho, len, n, g, op, reads, writes, oob);
}

// Geometry of channel_2q on (q0, q1): -1 when there is none, else bit 0 set when the items
// take the tensor-core form and bit 1 when the staged block holds the 256 superoperator
// entries that the engine stages there before the first item (the device code stages only
// when both hold); out = {V, P, dynamic shared-memory bytes of an engine block}.
int emu_super2_geometry(int layout, unsigned log_tile, unsigned n, unsigned q0, unsigned q1, uint64_t* out) {
    DmGeom g;
    const unsigned q[2] = {q0, q1};
    if (!dm_geometry(n, 2, q, ls_max_for(layout, log_tile), &g, emu_max_v())) return -1;
    out[0] = g.V();
    out[1] = g.P();
    out[2] = dm_block_smem_bytes(g);
    return (super2_mma_form(g, kDmBlock) ? 1 : 0) | (super2_stage_fits(g) ? 2 : 0);
}

int emu_dm_phase(int layout, unsigned log_tile, double* rho, uint64_t len, unsigned n, unsigned k,
                 const unsigned* qubits, const double* phase, uint32_t* reads, uint32_t* writes, uint64_t* oob) {
    EmuMem mem{reinterpret_cast<double2*>(rho), len, reads, writes, oob};
    if (k == 1 && phase[0] == 1.0 && phase[1] == 0.0) {
        GateFactor1 f1;
        f1.q = qubits[0];
        f1.ph1 = ldc(phase, 1);
        run_phase(layout, log_tile, mem, n, f1);
        return 0;
    }
    {                                                   // controlled phase, as the GPU launcher picks it
        bool ctrl = true;
        for (unsigned y = 0; y + 1 < (1u << k); ++y) ctrl = ctrl && phase[2 * y] == 1.0 && phase[2 * y + 1] == 0.0;
        if (ctrl) {
            GateFactorCtrl fc;
            fc.mask = 0;
            for (unsigned j = 0; j < k; ++j) fc.mask |= 1ull << qubits[j];
            fc.ph = ldc(phase, (1u << k) - 1);
            run_phase(layout, log_tile, mem, n, fc);
            return 0;
        }
    }
    GateFactor fac;
    fac.k = k;
    for (unsigned j = 0; j < 3; ++j) fac.q[j] = j < k ? qubits[j] : 0;
    for (unsigned y = 0; y < 8; ++y) fac.phase[y] = y < (1u << k) ? ldc(phase, y) : c2(1.0, 0.0);
    run_phase(layout, log_tile, mem, n, fac);
    return 0;
}

// The direct kernels (dm_direct.cuh).  op: 0 unitary (u = 4 complex), 1 superoperator (16), 2 controlled flip with
// the qubits' last as target (p0, p1), 3 SWAP, 4 phase of a controlled diagonal gate (ph); tile != 0 takes
// k_direct_tile (n >= 6), else one thread per group.
}  // extern "C"

namespace {
template <class Map, class Op>
void run_direct(const EmuMem& mem, const Map& map, unsigned n, unsigned q, const Op& op, int tile) {
    if (!tile) {
        for (idx_t t = 0; t < (idx_t(1) << (2 * (n - 1))); ++t) direct_small(mem, map, n, q, op, t);
        return;
    }
    const idx_t nt = idx_t(1) << (n - 6);
    std::vector<double2> sh(kDirectTile * kDirectPitch);
    for (idx_t b = 0; b < nt * (nt + 1) / 2; ++b) {
        const DirectWhere w = direct_where<Map>(b, n, q);
        if (w.diag) {
            for (unsigned e = 0; e < kDirectTile * kDirectTile; ++e) {
                idx_t u, v;
                direct_tile_uv<Map>(w, e % kDirectTile, e / kDirectTile, &u, &v);
                direct_group(mem, map, q, op, u, v);
            }
            continue;
        }
        for (int phase = w.transposed ? 0 : 1; phase < (w.transposed ? 3 : 2); ++phase)
            for (unsigned t = 0; t < kDirectThreads; ++t)
                direct_tile_phase(phase, mem, map, q, op, w, sh.data(), t, kDirectThreads);
    }
}
template <class Map>
int run_direct_op(const EmuMem& mem, const Map& map, unsigned n, int op, unsigned k, const unsigned* q, const double* par,
                  int tile) {
    if (op == 0) {
        DirectMix1 o;
        for (unsigned i = 0; i < 4; ++i) o.u[i] = ldc(par, i);
        run_direct(mem, map, n, q[0], o, tile);
    } else if (op == 1) {
        DirectSuper1 o;
        for (unsigned i = 0; i < 16; ++i) o.s[i] = ldc(par, i);
        run_direct(mem, map, n, q[0], o, tile);
    } else if (op == 2) {
        unsigned long long ctrl = 0;
        for (unsigned j = 0; j + 1 < k; ++j) ctrl |= 1ull << q[j];
        const double2 p0 = ldc(par, 0), p1 = ldc(par, 1);
        if (p0.x == 1.0 && p1.x == 1.0) run_direct(mem, map, n, q[k - 1], DirectFlip<true>{ctrl, p0, p1}, tile);
        else run_direct(mem, map, n, q[k - 1], DirectFlip<false>{ctrl, p0, p1}, tile);
    } else if (op == 3) {
        for (idx_t t = 0; t < (idx_t(1) << (2 * n)); ++t) direct_swap(mem, map, n, q[0], q[1], t);
    } else {
        GateFactorCtrl f;
        f.mask = 0;
        for (unsigned j = 0; j < k; ++j) f.mask |= 1ull << q[j];
        f.ph = ldc(par, 0);
        for (idx_t t = 0; t < (idx_t(1) << (2 * n)); ++t) direct_phase(mem, map, n, f, t);
    }
    return 0;
}
}  // namespace

extern "C" {

int emu_dm_direct(int layout, unsigned log_tile, double* rho, uint64_t len, unsigned n, int op, unsigned k,
                  const unsigned* qubits, const double* par, int tile, uint32_t* reads, uint32_t* writes,
                  uint64_t* oob) {
    const EmuMem mem{reinterpret_cast<double2*>(rho), len, reads, writes, oob};
    if (layout == 1) return run_direct_op(mem, PackedMap{idx_t(1) << n}, n, op, k, qubits, par, tile);
    return run_direct_op(mem, TiledMap{idx_t(1) << n, log_tile}, n, op, k, qubits, par, tile);
}

// One chain of 1-qubit channels on ascending distinct qubits (k <= 6); -2: they do not fit one
// staged block.
int emu_dm_chain(int layout, unsigned log_tile, double* rho, uint64_t len, unsigned n, unsigned k,
                 const unsigned* qubits, const double* sops, uint32_t* reads, uint32_t* writes, uint64_t* oob) {
    DmGeom g;
    unsigned vbit[kChainMax];
    if (!dm_chain_geometry(n, k, qubits, ls_max_for(layout, log_tile), &g, vbit)) return -2;
    OpChain op;
    for (unsigned j = 0; j < kChainMax; ++j)
        for (unsigned e = 0; e < 16; ++e) op.s[j][e] = j < k ? ldc(sops + 32 * j, e) : c2(0.0, 0.0);
    dm_chain_stages(op, k, vbit);
    return engine_dispatch(layout, log_tile, rho, len, n, g, op, reads, writes, oob);
}

// exp_diag on a density matrix: phase table from diag, then the phase pass (as the GPU path).
int emu_dm_exp_diag(int layout, unsigned log_tile, double* rho, uint64_t len, unsigned n, const double* diag,
                    double t, uint32_t* reads, uint32_t* writes, uint64_t* oob) {
    if (t == 0.0) return 0;
    const idx_t d = idx_t(1) << n;
    std::vector<double2> tab(d);
    for (idx_t x = 0; x < d; ++x) {
        double sn, cs;
        sincos(diag[x] * t, &sn, &cs);
        tab[x] = c2(cs, sn);
    }
    TableFactor<EmuMemC2> fac{EmuMemC2{tab.data(), d, oob}};
    EmuMem mem{reinterpret_cast<double2*>(rho), len, reads, writes, oob};
    run_phase(layout, log_tile, mem, n, fac);
    return 0;
}

int emu_pure_gate1(double* psi, unsigned n, unsigned target, int op, double c, double s, uint32_t* reads,
                   uint32_t* writes, uint64_t* oob) {
    if (n < 1 || target >= n) return -1;
    const idx_t npairs = idx_t(1) << (n - 1);
    const unsigned grid = grid_for(kPureThreads * kVec, npairs, kSms * 8u);
    const idx_t nthr = (idx_t)grid * kPureThreads;
    EmuMem mem{reinterpret_cast<double2*>(psi), idx_t(1) << n, reads, writes, oob};
    for (idx_t tid = 0; tid < nthr; ++tid) {
        switch (op) {
#define ORKAN_EMU_CASE(OPC) case OPC: pure1q_thread<OPC>(mem, npairs, target, c, s, tid, nthr); break;
            ORKAN_EMU_CASE(kOpX) ORKAN_EMU_CASE(kOpY) ORKAN_EMU_CASE(kOpZ) ORKAN_EMU_CASE(kOpH)
            ORKAN_EMU_CASE(kOpS) ORKAN_EMU_CASE(kOpSdg) ORKAN_EMU_CASE(kOpT) ORKAN_EMU_CASE(kOpTdg)
            ORKAN_EMU_CASE(kOpHy) ORKAN_EMU_CASE(kOpRx) ORKAN_EMU_CASE(kOpRy) ORKAN_EMU_CASE(kOpRz)
            ORKAN_EMU_CASE(kOpP)
#undef ORKAN_EMU_CASE
            default: return -1;
        }
    }
    return 0;
}

int emu_pure_gate2(double* psi, unsigned n, unsigned qa, unsigned qb, int op, uint32_t* reads, uint32_t* writes,
                   uint64_t* oob) {
    if (n < 2 || qa >= n || qb >= n || qa == qb) return -1;
    const idx_t nq = idx_t(1) << (n - 2);
    const unsigned grid = grid_for(kPureThreads * kVec, nq, kSms * 8u);
    const idx_t nthr = (idx_t)grid * kPureThreads;
    EmuMem mem{reinterpret_cast<double2*>(psi), idx_t(1) << n, reads, writes, oob};
    for (idx_t tid = 0; tid < nthr; ++tid) {
        switch (op) {
            case kOpCX: pure2q_thread<kOpCX>(mem, nq, qa, qb, tid, nthr); break;
            case kOpCY: pure2q_thread<kOpCY>(mem, nq, qa, qb, tid, nthr); break;
            case kOpCZ: pure2q_thread<kOpCZ>(mem, nq, qa, qb, tid, nthr); break;
            case kOpSwap: pure2q_thread<kOpSwap>(mem, nq, qa, qb, tid, nthr); break;
            default: return -1;
        }
    }
    return 0;
}

int emu_pure_ccx(double* psi, unsigned n, unsigned c1, unsigned c2q, unsigned t, uint32_t* reads, uint32_t* writes,
                 uint64_t* oob) {
    if (n < 3) return -1;
    const idx_t no = idx_t(1) << (n - 3);
    const unsigned grid = grid_for(kPureThreads * kVec, no, kSms * 8u);
    const idx_t nthr = (idx_t)grid * kPureThreads;
    EmuMem mem{reinterpret_cast<double2*>(psi), idx_t(1) << n, reads, writes, oob};
    for (idx_t tid = 0; tid < nthr; ++tid) pure_ccx_thread(mem, no, c1, c2q, t, tid, nthr);
    return 0;
}

int emu_pure_exp_diag(double* psi, unsigned n, const double* diag, double t, uint32_t* reads, uint32_t* writes,
                      uint64_t* oob) {
    const idx_t d = idx_t(1) << n;
    const unsigned grid = grid_for(kPureThreads * kVec, d, kSms * 8u);
    const idx_t nthr = (idx_t)grid * kPureThreads;
    EmuMem mem{reinterpret_cast<double2*>(psi), d, reads, writes, oob};
    EmuMemR dg{diag, d, oob};
    for (idx_t tid = 0; tid < nthr; ++tid) pure_exp_diag_thread(mem, dg, d, t, tid, nthr);
    return 0;
}

int emu_fill(double* data, uint64_t len, double re, double im, unsigned corner_log_tile, uint64_t corner_dim,
             uint32_t* reads, uint32_t* writes, uint64_t* oob) {
    const unsigned grid = grid_for(kPureThreads * 4, len, kSms * 8u);
    const idx_t nthr = (idx_t)grid * kPureThreads;
    EmuMem mem{reinterpret_cast<double2*>(data), len, reads, writes, oob};
    for (idx_t tid = 0; tid < nthr; ++tid) fill_thread(mem, len, c2(re, im), corner_log_tile, corner_dim, tid, nthr);
    return 0;
}

// A fused run of statevector gates (k_pure_fused): every block of the grid, phase by phase (per
// chunk: load, each register stage, store), with a block-local chunk buffer.
}  // extern "C"

namespace {
template <int K>
void run_fused(const EmuMem& mem, const FusedPlan& P, unsigned grid_cap) {
    const unsigned nthr = fused_threads(P);
    const idx_t nch = P.nchunks();
    const unsigned grid = grid_for(1, nch, grid_cap ? grid_cap : kSms * 4u);
    std::vector<double2> buf(P.chunk());
    for (unsigned b = 0; b < grid; ++b)
        for (idx_t ch = b; ch < nch; ch += grid) {
            const idx_t base = fused_base(P, ch);
            for (unsigned t = 0; t < nthr && !P.din; ++t) fused_load<K>(mem, P, fused_walk<K>(P, t), t, base, buf.data());
            for (unsigned st = 0; st < P.nstages; ++st)
                for (unsigned t = 0; t < nthr; ++t) fused_stage_k<K>(mem, P, fused_walk<K>(P, t), st, base, buf.data(), t);
            for (unsigned t = 0; t < nthr && !P.dout; ++t) fused_store<K>(mem, P, fused_walk<K>(P, t), t, base, buf.data());
        }
}
}  // namespace

extern "C" {

int emu_pure_fused(double* psi, unsigned n, unsigned log_chunk, unsigned ngates, const orkan_fgate_t* gates,
                   unsigned grid_cap, uint32_t* reads, uint32_t* writes, uint64_t* oob) {
    FusedPlan P;
    if (!fused_plan(n, log_chunk, ngates, gates, &P)) return -1;
    const EmuMem mem{reinterpret_cast<double2*>(psi), idx_t(1) << n, reads, writes, oob};
    switch (P.K) {
        case 4: run_fused<4>(mem, P, grid_cap); break;
        case 3: run_fused<3>(mem, P, grid_cap); break;
        case 2: run_fused<2>(mem, P, grid_cap); break;
        default: run_fused<1>(mem, P, grid_cap); break;
    }
    return 0;
}

unsigned long long emu_fused_need(const orkan_fgate_t* g) { return fused_need(*g); }

// Register stages the plan cuts a run into (-1: the run does not fit).
int emu_fused_stages(unsigned n, unsigned log_chunk, unsigned ngates, const orkan_fgate_t* gates) {
    FusedPlan P;
    if (!fused_plan(n, log_chunk, ngates, gates, &P)) return -1;
    return (int)P.nstages;
}

// Shared-memory layout of the QAOA pass kernel: 1 when every region is aligned for the chunk
// sizes and buffer counts of the launches and any table length.
int emu_qaoa_smem_aligned(void) {
    for (unsigned C = 1; C <= kQaoaMaxC; ++C)
        for (unsigned buffers = 1; buffers <= 6; ++buffers)
            for (unsigned tstride = 0; tstride <= kQaoaMaxTable; ++tstride)
                if (!qaoa_smem_aligned(C, buffers, tstride, 512)) return 0;
    return 1;
}

// Groups 0 and 1 of a pass's items, when both hold 16 amplitudes: 1 when every half-warp
// touches the same slots in both, every slot once (0 otherwise, -1: not such a pass).
int emu_qaoa_half_warp_closed(unsigned n, unsigned C, unsigned kind) {
    const QaoaGeo g = qaoa_geo(n, C, kind);
    if (g.m < 2 || qaoa_group_bits(g, 0) != 4 || qaoa_group_bits(g, 1) != 4) return -1;
    std::vector<unsigned> a((size_t)1 << C, ~0u), b((size_t)1 << C, ~0u);
    for (unsigned r = 0; r < (1u << (C - 4)); ++r)
        for (unsigned e = 0; e < 16; ++e) {
            unsigned& o = a[qaoa_m_slot(qaoa_m_set<4>(g.MM, r), 4, e)];
            if (o != ~0u) return 0;
            o = r >> 4;
        }
    mark_s<4, 4>(g, b);
    return a == b ? 1 : 0;
}

// Fused QAOA passes of one instance; byte_cost selects byte costs (cost_b) over doubles.
int emu_qaoa(unsigned n, const double* cost_d, const uint8_t* cost_b, int byte_cost, unsigned p, const double* gamma,
             const double* beta, unsigned C, unsigned nthr, unsigned upto, double* psi, double* mean,
             uint32_t* reads, uint32_t* writes, uint64_t* oob) {
    if (byte_cost) return run_qaoa<uint8_t>(n, cost_b, p, gamma, beta, C, nthr, upto, psi, mean, reads, writes, oob);
    return run_qaoa<double>(n, cost_d, p, gamma, beta, C, nthr, upto, psi, mean, reads, writes, oob);
}

}  // extern "C"
