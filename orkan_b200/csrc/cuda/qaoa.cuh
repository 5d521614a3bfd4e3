// qaoa.cuh - batched QAOA-style circuits of uneven sizes, fused into p + 1 passes over half
// of each statevector.
//
// Each instance (n qubits, diagonal cost vector cost, angles gamma_k, beta_k) is the
// composition of the reference's own calls (no reference counterpart as a whole):
//     state_plus(n)                                     src/state/state_pure.c:30-43
//     for k < p:  exp_diag(cost, gamma_k)               src/circ/circ_pure.c:21-33
//                 rx(q, 2 beta_k) for every qubit q     src/gate/gate_pure.c:230-234
//     mean(cost)                                        src/meas/meas_pure.c:20-30
// The mixer of layer k factors into L_k (rx on qubits < C) and H_k (rx on qubits >= C),
// which commute, so the circuit D1 L1 H1 D2 L2 H2 ... Dp Lp Hp M regroups as
//     pass 0 (low):           init, D1, L1
//     pass j (1 <= j < p):    Mix_j, D_{j+1}, Mix_{j+1}   with Mix = H (j odd) or L (j even)
//     pass p:                 Mix_p, M
// and each pass touches every stored amplitude once.  Instances with n <= C run the whole
// circuit in one pass ("full") and never touch a state vector in memory.
//
// Half states.  The cost of a cut does not change when every bit is flipped, and neither do
// |+> and the mixer, so psi(~x) = psi(x) throughout the circuit: only the 2^N amplitudes
// with the top bit clear are kept (N = n - 1), and rx on the top qubit pairs y with ~y
// (its partner's stored image).  That halves the bytes, the arithmetic and the cost vectors.
//
// Order in memory.  y = row 2^C + c.  Column c sits at position
//     pos(c) = ((c ^ (t ? m : 0)) << 1) | t,   t = c >> (C - 1),  m = 2^(C-1) - 1
// of its row (in those low C - 1 bits), so columns c and ~c are neighbours: the high pass,
// which needs both for the top qubit, reads runs of at least 32 bytes.  On positions, the flip
// of qubit q < C - 1 is the flip of bit q + 1, the flip of qubit C - 1 is the complement of
// all C bits, and the flip of the top qubit is the complement of bit 0 and of every row bit.
// A low item is one row (2^C consecutive amplitudes, slot s = position).  A high item is
// 2^lw column pairs of all 2^R rows (R = N - C, lw = 2C - n), slot s = t | row << 1 | w << (R + 1).
// So both have the same mixers on slots: the single bits 1 .. nb - 1 and the complement M of
// bits 0 .. nb - 1 (nb = C for low items, R + 1 for high ones).
//
// Groups.  The mixers of an item run in register stages: group 0 is M with the single bits
// 1-3, group g > 0 the single bits 4g .. 4g + 3.  A thread holds the 16 amplitudes of a set
// (all combinations of a group's flips) and applies the group's butterflies there.  Rx on
// different qubits commute, so segment A runs the groups downwards to 0, the phase of the next
// layer is applied in group 0, and segment B runs them upwards: 2m - 1 stages with one
// phase point, always in the same register arrangement, so the costs are stored in the order
// in which the threads want them (qaoa_cost_slot) and go straight to registers.  The last
// stage stores from registers, with lanes on neighbouring amplitudes.  Groups 0 and 1 mix
// subcubes of 256 slots that one half-warp owns in both, so no block barrier lies between them.
//
// Arithmetic (checked against the per-call path at 1e-12): the rx pair update
// (a, b) -> (c a - i s b, c b - i s a) with c = cos(beta), s = sin(beta) (rx(2 beta) of
// gate_pure.c) is applied as k-form (a - i t b, b - i t a), t = s / c, when |c| >= |s|, or as
// (u a - i b, u b - i a), u = c / s, otherwise -- four FMAs per pair -- and the product of
// the dropped factors of a pass's segments scales the phase of that pass (or its mean); the
// phase is (c re + s im, c im - s re) with (s, c) = sincos(cost[x] * gamma) (taken from a
// per-layer table, made by the same sincos, when the costs are stored as bytes); the mean is
// sum cost[x] |psi_x|^2 in a fixed order per item.
#pragma once

#include "common.cuh"

#include <math.h>

#include <type_traits>

namespace orkan {

constexpr unsigned kQaoaMaxTable = 256;   // integer costs up to 255 are stored as bytes
constexpr unsigned kQaoaGroup = 4;        // mixers per register stage
constexpr unsigned kQaoaMaxC = 13;        // 2^13 amplitudes (128 KB) staged per work item

enum QaoaKind : unsigned { kQaoaFull = 0, kQaoaLow = 1, kQaoaHigh = 2 };

struct QaoaInst {
    double2* psi;          // 2^(n-1) amplitudes (unused by full passes)
    const void* cost;      // costs in the order of this kind of pass (qaoa_cost_slot)
    idx_t item0;           // first work item of this instance in the pass
    unsigned n;
    unsigned pos;          // row of the instance in the angle arrays and tables
};

// The mixer of one layer of one instance in the four-FMA form, and the factors that the
// dropped ones leave: fs scales the phase of this layer (the dropped factors of every segment
// of the pass that applies it), fm the mean (taken from the last layer; chunked instances sum
// half of the state, so it doubles the sum).
struct QaoaRx {
    double k;
    double fs;
    double fm;
    int sform;             // 0: (a - i k b) with k = s / c, scale = c; 1: (k a - i b), k = c / s, scale = s
    int pad_;
};

// Host side: the mixer coefficients of the p layers of an instance of n qubits in chunks of
// 2^C, layer k from c = cos(theta_k / 2), s = sin(theta_k / 2) of rx(theta_k).  Phase l of a
// chunked instance lies in pass l, between the segments of layers l - 1 and l.
inline void qaoa_rx_coeffs(const double* c, const double* s, unsigned p, unsigned n, unsigned C, QaoaRx* out) {
    const bool full = n <= C;
    auto power = [](double x, unsigned e) {
        double f = 1.0;
        for (unsigned i = 0; i < e; ++i) f *= x;
        return f;
    };
    double prev = 1.0;
    for (unsigned l = 0; l < p; ++l) {
        QaoaRx r;
        double scale;
        if (fabs(c[l]) >= fabs(s[l])) { r.k = s[l] / c[l]; scale = c[l]; r.sform = 0; }
        else { r.k = c[l] / s[l]; scale = s[l]; r.sform = 1; }
        if (full) {
            r.fs = power(scale, n);
            r.fm = 1.0;
        } else {
            const unsigned nq = (l % 2 == 0) ? C : n - C, nqm = ((l + 1) % 2 == 0) ? C : n - C;
            r.fs = power(scale, nq) * (l ? power(prev, nq) : 1.0);
            const double f = power(scale, nqm);
            r.fm = 2.0 * f * f;
        }
        r.pad_ = 0;
        prev = scale;
        out[l] = r;
    }
}

struct QaoaTables {
    const double2* phase;  // [pos][layer][tstride]: fs (cos, sin)(c * gamma) for byte costs c
    const QaoaRx* rx;      // [pos][layer]
    unsigned tstride;
};

// log2 of the slots of one item, of the stored amplitudes, and the items of an instance
// (chunked: low and high alike).
ORKAN_HD unsigned qaoa_lc(unsigned n, unsigned C, unsigned kind) { return kind == kQaoaFull ? n : C; }
ORKAN_HD unsigned qaoa_log_items(unsigned n, unsigned C, unsigned kind) { return kind == kQaoaFull ? 0u : n - 1 - C; }
ORKAN_HD idx_t qaoa_items(unsigned n, unsigned C, unsigned kind) { return idx_t(1) << qaoa_log_items(n, C, kind); }

// Position of column c in its row, and back.
ORKAN_HD unsigned qaoa_pos(unsigned C, unsigned c) {
    const unsigned t = c >> (C - 1), m = (1u << (C - 1)) - 1;
    return (((c & m) ^ (t ? m : 0u)) << 1) | t;
}
ORKAN_HD unsigned qaoa_col(unsigned C, unsigned pos) {
    const unsigned t = pos & 1u, m = (1u << (C - 1)) - 1;
    return ((pos >> 1) ^ (t ? m : 0u)) | (t << (C - 1));
}

// Shape of the items of a pass.
struct QaoaGeo {
    unsigned n, C, kind;
    unsigned R, lw;            // row bits; log2 of a high item's column pairs
    unsigned nb;               // mixed slot bits: singles 1 .. nb - 1 and M (full: singles 0 .. nb - 1)
    unsigned MM;               // mask of M over the slot bits (full: 0)
    unsigned m;                // groups
};
ORKAN_HD QaoaGeo qaoa_geo(unsigned n, unsigned C, unsigned kind) {
    QaoaGeo g;
    g.n = n;
    g.C = C;
    g.kind = kind;
    g.R = g.lw = 0;
    if (kind == kQaoaFull) {
        g.nb = n;
        g.MM = 0;
    } else {
        g.R = n - 1 - C;
        g.lw = 2 * C - n;
        g.nb = kind == kQaoaLow ? C : g.R + 1;
        g.MM = (1u << g.nb) - 1;
    }
    g.m = (g.nb + kQaoaGroup - 1) / kQaoaGroup;
    return g;
}
// log2 of the register set of group gi
ORKAN_HD unsigned qaoa_group_bits(const QaoaGeo& g, unsigned gi) {
    const unsigned left = g.nb - gi * kQaoaGroup;
    return left < kQaoaGroup ? left : kQaoaGroup;
}

// Storage index of slot s of an item.
ORKAN_HD idx_t qaoa_index(const QaoaGeo& g, idx_t item, unsigned s) {
    if (g.kind == kQaoaLow) return (item << g.C) | s;
    const unsigned row = (s >> 1) & ((1u << g.R) - 1), w = s >> (1 + g.R);
    return ((idx_t)row << g.C) | (item << (g.lw + 1)) | (w << 1) | (s & 1u);
}
// Basis state (top bit clear) of storage index i.
ORKAN_HD idx_t qaoa_state_of(unsigned C, idx_t i) {
    return (i >> C << C) | qaoa_col(C, (unsigned)(i & ((idx_t(1) << C) - 1)));
}
// Storage index of basis state x (any top bit).
ORKAN_HD idx_t qaoa_index_of(unsigned n, unsigned C, idx_t x) {
    const idx_t full = (idx_t(1) << n) - 1;
    if ((x >> (n - 1)) & 1u) x = ~x & full;
    return (x >> C << C) | qaoa_pos(C, (unsigned)(x & ((idx_t(1) << C) - 1)));
}

// ---- register sets ---------------------------------------------------------------------
// Set r of group 0 (M and the single bits 1 .. K - 1, K = qaoa_group_bits): slots
// r 2^K + 2j for element (j, m = 0) and their complements under MM for m = 1.  Register
// e = j | m << (K - 1) of a thread holds the element whose index is e with the bits of a
// lane-dependent key flipped, so that the 8 lanes of a shared-memory phase fall on 8
// different 16-byte banks; the butterflies are symmetric, so the flip needs no other care.
struct QaoaMSet {
    unsigned p0, p1;           // slot of register (j, m) is p_m ^ (j << 1)
};
template <int K>
ORKAN_HD QaoaMSet qaoa_m_set(unsigned MM, unsigned r) {
    constexpr unsigned nbk = K < 3 ? K : 3, sh = 3 - nbk;
    const unsigned k = (r >> sh) & ((1u << nbk) - 1);
    const unsigned km = k >> (nbk - 1), kj = k & ((1u << (nbk - 1)) - 1);
    QaoaMSet s;
    s.p0 = ((r << K) | (kj << 1)) ^ (km ? MM : 0u);
    s.p1 = s.p0 ^ MM;
    return s;
}
ORKAN_HD unsigned qaoa_m_slot(const QaoaMSet& s, int K, unsigned e) {
    const unsigned h = 1u << (K - 1);
    return ((e & h) ? s.p1 : s.p0) ^ ((e & (h - 1)) << 1);
}

// Set r of the K single bits at B0: base slot, element e at base | e << B0.  For B0 = 4 the
// sets of a chunked item are numbered so that set r lies in the subcube that sets r & ~15 ..
// r | 15 of group 0 cover (the complement M moves the odd slots to the complemented bits).
template <int K, int B0>
ORKAN_HD unsigned qaoa_s_base(unsigned MM, unsigned r) {
    unsigned b = (r & ((1u << B0) - 1)) | ((r >> B0) << (B0 + K));
    if (B0 == 4 && (b & 1u)) b ^= MM & ~((1u << (B0 + K)) - 1);
    return b;
}
// The same sets of a high item in the order for its stores (and, with K = 0, all slots in
// the order for its loads): lanes take t and the two lowest free row bits first (8
// neighbouring slots, distinct banks), then up to two column-pair bits, so that a warp covers
// whole 32- to 128-byte runs, then the other row bits, then the other column pairs.
ORKAN_HD unsigned qaoa_high_base(unsigned R, unsigned lw, unsigned r, unsigned B0, unsigned K) {
    const unsigned nr = R - K;
    const unsigned t = r & 1u;
    r >>= 1;
    const unsigned a = nr < 2 ? nr : 2, c = lw < 2 ? lw : 2;
    const unsigned rl = r & ((1u << a) - 1);
    r >>= a;
    const unsigned wl = r & ((1u << c) - 1);
    r >>= c;
    const unsigned rh = r & ((1u << (nr - a)) - 1);
    const unsigned wh = r >> (nr - a);
    unsigned x = t | ((rl | (rh << a)) << 1);
    if (K) x = (x & ((1u << B0) - 1)) | ((x >> B0) << (B0 + K));
    return x | ((wl | (wh << c)) << (1 + R));
}

// Cost order: within an item, byte costs set by set (a thread's 2^K costs are one aligned
// word), FP64 costs register by register (lanes read neighbouring values).  Slot whose cost
// is entry q of an item.
template <int K>
ORKAN_HD unsigned qaoa_cost_slot_k(const QaoaGeo& g, bool bytes, unsigned q) {
    const unsigned ls = g.C - K;                       // log2 of the sets
    const unsigned r = bytes ? q >> K : q & ((1u << ls) - 1), e = bytes ? q & ((1u << K) - 1) : q >> ls;
    return qaoa_m_slot(qaoa_m_set<K>(g.MM, r), K, e);
}
ORKAN_HD unsigned qaoa_cost_slot(const QaoaGeo& g, bool bytes, unsigned q) {
    switch (qaoa_group_bits(g, 0)) {
        case 1: return qaoa_cost_slot_k<1>(g, bytes, q);
        case 2: return qaoa_cost_slot_k<2>(g, bytes, q);
        case 3: return qaoa_cost_slot_k<3>(g, bytes, q);
        default: return qaoa_cost_slot_k<4>(g, bytes, q);
    }
}
// Basis state whose cost is entry i of the cost array of a kind of pass.
ORKAN_HD idx_t qaoa_cost_state(const QaoaGeo& g, bool bytes, idx_t i) {
    if (g.kind == kQaoaFull) return i;
    const idx_t item = i >> g.C;
    return qaoa_state_of(g.C, qaoa_index(g, item, qaoa_cost_slot(g, bytes, (unsigned)(i & ((idx_t(1) << g.C) - 1)))));
}

// ---- stages ----------------------------------------------------------------------------
enum : unsigned { kQaoaFromSmem = 0, kQaoaFromInit = 2 };
enum : unsigned { kQaoaToSmem = 0, kQaoaToGlobal = 1, kQaoaToMeasure = 2 };

struct QaoaStage {
    uint8_t g;                 // group
    int8_t sa, sb;             // segments applied before / after the phase (-1: none)
    uint8_t src, dst;
    int8_t phase;              // layer of the phase, -1: none
    uint8_t warp_sync;         // what the stage wrote is read by the same half-warp next
    uint8_t pad_;
};

// A pass launch: its instances (all of one qubit count) and the pass's stages, computed once
// on the host.
constexpr unsigned kQaoaStageTable = 8;    // 2 m - 1 with m <= 4
static_assert((kQaoaMaxC + kQaoaGroup - 1) / kQaoaGroup <= (kQaoaStageTable + 1) / 2, "the stages of every pass fit");
constexpr unsigned long long kQaoaPolls = 1ull << 24;   // limit of a bounded wait

struct QaoaPass {
    const QaoaInst* inst;
    unsigned ninst;
    idx_t items;           // total work items of the pass
    const double* gamma;   // [pos][p]
    double* partial;       // measuring pass: one partial sum per work item
    double* status;        // set non-zero when a wait for staged data ran out
    unsigned p;
    unsigned pass;         // j in [0, p] (0 for full passes)
    unsigned C;            // log2 of the chunk (slots per item)
    unsigned kind;         // QaoaKind
    unsigned li;           // log2 of the work items per instance: item w is item w mod 2^li
                           // of instance w >> li of the list (every instance has n qubits)
    unsigned long long wait_limit;   // polls of a bounded wait
    QaoaGeo geo;
    unsigned nreg;             // register stages (chunked passes)
    int layer_a, layer_b;      // layers of segments A and B (-1: none)
    int layer_phase;           // layer of the phase, -1: none
    QaoaStage stage[kQaoaStageTable];
};

// Fill in the geometry and the stages of a pass of n-qubit instances, whose phases are read from the staged
// tables (byte costs) or not.
//
// A stage that stores an item hands its buffers back before its arithmetic when a thread has one set, and the
// next item's table may then arrive while slower threads still read this one's.  So where group 0 alone makes up
// a middle pass (high items of 4 mixed bits, n = C + 4), byte costs take two stages: mixers A and the phase,
// then mixers B and the stores.  (512 instances of 16 qubits, p = 4: 727 us.  A release after the stores instead
// changes the registers of every byte-cost pass: 715 us there, but 16 instances of 24 qubits 5.71 against 5.59 ms.)
inline void qaoa_pass_setup(QaoaPass& P, unsigned n, bool tables = true) {
    P.geo = qaoa_geo(n, P.C, P.kind);
    P.li = qaoa_log_items(n, P.C, P.kind);
    P.nreg = 0;
    P.layer_a = P.layer_b = P.layer_phase = -1;
    P.wait_limit = kQaoaPolls;
    for (auto& s : P.stage) s = QaoaStage{};
    if (P.kind == kQaoaFull) return;
    const int j = (int)P.pass, p = (int)P.p, most = (kQaoaStageTable + 1) / 2;
    const int m = (int)P.geo.m < most ? (int)P.geo.m : most;       // (kQaoaMaxC bits are 4 groups)
    const bool first = j == 0, last = j == p;
    P.layer_a = first ? -1 : j - 1;
    P.layer_b = last ? -1 : j;
    P.layer_phase = last ? -1 : j;
    auto add = [&](int g, int sa, int sb) {
        QaoaStage& s = P.stage[P.nreg++];
        s.g = (uint8_t)g;
        s.sa = (int8_t)sa;
        s.sb = (int8_t)sb;
        s.src = kQaoaFromSmem;
        s.dst = kQaoaToSmem;
        s.phase = (int8_t)(g == 0 ? P.layer_phase : -1);
    };
    if (!first)
        for (int g = m - 1; g > 0; --g) add(g, 0, -1);
    if (tables && !first && !last && m == 1 && qaoa_group_bits(P.geo, 0) == kQaoaGroup) {
        add(0, 0, -1);
        add(0, -1, 1);
        P.stage[1].phase = -1;
    } else {
        add(0, first ? -1 : 0, last ? -1 : 1);
    }
    if (!last)
        for (int g = 1; g < m; ++g) add(g, -1, 1);
    if (first) P.stage[0].src = kQaoaFromInit;
    P.stage[P.nreg - 1].dst = last ? kQaoaToMeasure : kQaoaToGlobal;
    // groups 0 and 1 of 16 amplitudes each stay within a half-warp, unless group 1 stores a
    // high item (its sets are then numbered for the stores); the same group twice stays within a thread
    for (unsigned r = 0; r + 1 < P.nreg; ++r) {
        const QaoaStage &a = P.stage[r], &b = P.stage[r + 1];
        const bool pair = a.g + b.g == 1 && qaoa_group_bits(P.geo, 0) == 4 && qaoa_group_bits(P.geo, 1) == 4;
        P.stage[r].warp_sync = a.g == b.g || (pair && !(P.kind == kQaoaHigh && b.dst == kQaoaToGlobal));
    }
}

ORKAN_HD double2 qaoa_apply_phase(double2 ph, double2 v) {
    return c2(ph.x * v.x + ph.y * v.y, ph.x * v.y - ph.y * v.x);
}

// fs (cos, sin)(c gamma): from the table (which holds the factor) for byte costs.
template <class CostT>
ORKAN_HD double2 qaoa_phase(CostT c, double gamma, double fs, const double2* table) {
    if constexpr (std::is_same<CostT, double>::value) {
        (void)table;
        double sn, cs;
        sincos(c * gamma, &sn, &cs);
        return c2(cs * fs, sn * fs);
    } else {
        (void)gamma;
        (void)fs;
        return table[c];
    }
}

// The butterflies of K mixers on 2^K registers.
template <int K>
ORKAN_HD void qaoa_mix(double2 (&v)[1 << K], double k, int sform) {
    constexpr unsigned NV = 1u << K;
    if (sform == 0) {
#pragma unroll
        for (unsigned b = 0; b < (unsigned)K; ++b)
#pragma unroll
            for (unsigned j = 0; j < NV; ++j)
                if (!(j & (1u << b))) {
                    double2& a = v[j];
                    double2& c = v[j | (1u << b)];
                    const double2 na = c2(fma(k, c.y, a.x), fma(-k, c.x, a.y));
                    c = c2(fma(k, a.y, c.x), fma(-k, a.x, c.y));
                    a = na;
                }
    } else {
#pragma unroll
        for (unsigned b = 0; b < (unsigned)K; ++b)
#pragma unroll
            for (unsigned j = 0; j < NV; ++j)
                if (!(j & (1u << b))) {
                    double2& a = v[j];
                    double2& c = v[j | (1u << b)];
                    const double2 na = c2(fma(k, a.x, c.y), fma(k, a.y, -c.x));
                    c = c2(fma(k, c.x, a.y), fma(k, c.y, -a.x));
                    a = na;
                }
    }
}

// What a work item needs besides its amplitudes: the mixers of its two segments, the phase,
// where its amplitudes and costs are.  Written by the thread that stages the item.
struct QaoaItem {
    double2* psi;
    const void* cost;      // first cost of the item
    double ka, kb;
    double gamma, fs;
    int sa, sb;            // forms
    idx_t item;            // index within the instance
};
ORKAN_HD QaoaItem qaoa_item(const QaoaPass& P, const QaoaTables& T, const QaoaInst& I, idx_t w, unsigned cost_size) {
    QaoaItem J;
    const idx_t row = (idx_t)I.pos * P.p;
    J.psi = I.psi;
    J.item = w & ((idx_t(1) << P.li) - 1);
    J.cost = static_cast<const unsigned char*>(I.cost) + (J.item << P.C) * cost_size;
    J.ka = J.kb = J.gamma = J.fs = 0.0;
    J.sa = J.sb = 0;
    if (P.layer_a >= 0) {
        const QaoaRx& r = T.rx[row + P.layer_a];
        J.ka = r.k;
        J.sa = r.sform;
    }
    if (P.layer_b >= 0) {
        const QaoaRx& r = T.rx[row + P.layer_b];
        J.kb = r.k;
        J.sb = r.sform;
        J.fs = r.fs;
        J.gamma = P.gamma[row + P.layer_b];
    }
    return J;
}

// Amplitudes of an item into its buffer by threads tid of nthr: a low item is one run, a high
// item one element per slot (consecutive threads on runs of 2^(lw+1) neighbours).
// Mem::bulk_load(dst, x, count, bar) copies a run, Mem::cp16(dst, x) one amplitude.
template <class Mem>
ORKAN_HD void qaoa_fill(const QaoaGeo& g, const Mem& psi, idx_t item, double2* vb, void* bar, unsigned tid,
                        unsigned nthr) {
    if (g.kind == kQaoaLow) {
        if (tid == 0) psi.bulk_load(vb, item << g.C, 1u << g.C, bar);
        return;
    }
    for (unsigned e = tid; e < (1u << g.C); e += nthr) {
        const unsigned s = qaoa_high_base(g.R, g.lw, e, 0, 0);
        psi.cp16(vb + s, qaoa_index(g, item, s));
    }
}

struct QaoaNoRelease {
    ORKAN_HD void operator()() const {}
};

// The costs of one set of group 0, register by register through at(e), e ascending.  Byte costs come as
// words through CostMem::words.  FP64 costs, CostMem::ld(i), are read two registers ahead: the first two
// before the stage's mixers, the next two before the current two are used, so that no sincos waits for its
// own argument (8 instances of 24 qubits at p = 6: 5.89 ms with the staging warps' prefetch to L2, 6.60 ms
// with loads where they are used; four ahead spill).
template <int K, class CostT>
struct QaoaCosts;
template <int K>
struct QaoaCosts<K, uint8_t> {
    static constexpr unsigned kWords = (1u << K) < 4 ? 1 : (1u << K) / 4;
    uint32_t w[kWords];
    template <class CostMem>
    ORKAN_HD void begin(const CostMem& cost, unsigned r, unsigned) {
        cost.template words<K>(w, r << K);
    }
    template <class CostMem>
    ORKAN_HD unsigned char at(const CostMem&, unsigned e, unsigned, unsigned) {
        return (unsigned char)(w[e >> 2] >> (8 * (e & 3u)));
    }
};
template <int K>
struct QaoaCosts<K, double> {
    static constexpr unsigned NV = 1u << K, kAhead = NV < 2 ? NV : 2;
    double c[2][kAhead];
    template <class CostMem>
    ORKAN_HD void begin(const CostMem& cost, unsigned r, unsigned sets) {
#pragma unroll
        for (unsigned e = 0; e < kAhead; ++e) c[0][e] = cost.ld(e * sets + r);
    }
    template <class CostMem>
    ORKAN_HD double at(const CostMem& cost, unsigned e, unsigned r, unsigned sets) {
        if (e % kAhead == 0 && e + kAhead < NV)
#pragma unroll
            for (unsigned d = 0; d < kAhead; ++d) c[(e / kAhead + 1) & 1u][d] = cost.ld((e + kAhead + d) * sets + r);
        return c[(e / kAhead) & 1u][e % kAhead];
    }
};

// Group 0 of a chunked item: mixers of segment A, the phase, mixers of segment B, each if the
// stage has it.  Returns the thread's share of the mean when measuring.
template <int K, class CostT, class Mem, class CostMem, class Rel>
ORKAN_HD double qaoa_m_stage(const QaoaGeo& g, const QaoaStage& sg, const QaoaItem& J, const Mem& psi,
                             const CostMem& cost, double2* vb, const double2* tab, unsigned lc, unsigned tid,
                             unsigned nthr, const Rel& release) {
    constexpr unsigned NV = 1u << K;
    const unsigned sets = 1u << (lc - K);
    const bool costs = sg.phase >= 0 || sg.dst == kQaoaToMeasure;
    const double gamma = J.gamma, fs = J.fs;
    // The release lets the next item overwrite J, the amplitudes and the phase table.  J and the costs' place are
    // read before it; the table is not, so no stage reads the table and releases (qaoa_pass_setup).
    const double ka = J.ka, kb = J.kb;
    const int sa = J.sa, sb = J.sb;
    const idx_t item = J.item;
    double acc = 0.0;
    for (unsigned r = tid; r < sets; r += nthr) {
        const QaoaMSet ms = qaoa_m_set<K>(g.MM, r);
        QaoaCosts<K, CostT> c;
        if (costs) c.begin(cost, r, sets);
        double2 v[NV];
        if (sg.src == kQaoaFromInit) {
            const double amp0 = 1.0 / sqrt((double)(idx_t(1) << g.n));
#pragma unroll
            for (unsigned e = 0; e < NV; ++e) v[e] = c2(amp0, 0.0);
        } else {
#pragma unroll
            for (unsigned e = 0; e < NV; ++e) v[e] = vb[qaoa_m_slot(ms, K, e)];
        }
        if (sg.dst != kQaoaToSmem && sets == nthr) release();
        if (sg.sa >= 0) qaoa_mix<K>(v, ka, sa);
        if (sg.phase >= 0) {
#pragma unroll
            for (unsigned e = 0; e < NV; ++e)
                v[e] = qaoa_apply_phase(qaoa_phase<CostT>(c.at(cost, e, r, sets), gamma, fs, tab), v[e]);
        }
        if (sg.sb >= 0) qaoa_mix<K>(v, kb, sb);
        if (sg.dst == kQaoaToMeasure) {
#pragma unroll
            for (unsigned e = 0; e < NV; ++e) acc += (double)c.at(cost, e, r, sets) * (v[e].x * v[e].x + v[e].y * v[e].y);
        } else if (sg.dst == kQaoaToGlobal) {
#pragma unroll
            for (unsigned e = 0; e < NV; ++e) psi.st(qaoa_index(g, item, qaoa_m_slot(ms, K, e)), v[e]);
        } else {
#pragma unroll
            for (unsigned e = 0; e < NV; ++e) vb[qaoa_m_slot(ms, K, e)] = v[e];
        }
    }
    if (sg.dst != kQaoaToSmem && sets != nthr) release();
    return acc;
}

// Group of the K single bits at B0 (4, 8 or 12) of a chunked item.
template <int K, int B0, class Mem, class Rel>
ORKAN_HD void qaoa_s_stage(const QaoaGeo& g, const QaoaStage& sg, const QaoaItem& J, const Mem& psi, double2* vb,
                           unsigned lc, unsigned tid, unsigned nthr, const Rel& release) {
    constexpr unsigned NV = 1u << K;
    const unsigned sets = 1u << (lc - K);
    const double k = sg.sa >= 0 ? J.ka : J.kb;
    const int form = sg.sa >= 0 ? J.sa : J.sb;
    const idx_t item = J.item;                 // read before the release
    const bool high_out = g.kind == kQaoaHigh && sg.dst == kQaoaToGlobal;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (unsigned r = tid; r < sets; r += nthr) {
        const unsigned base = high_out ? qaoa_high_base(g.R, g.lw, r, B0, K) : qaoa_s_base<K, B0>(g.MM, r);
        double2 v[NV];
#pragma unroll
        for (unsigned e = 0; e < NV; ++e) v[e] = vb[base + (e << B0)];
        if (sg.dst == kQaoaToGlobal && sets == nthr) release();
        qaoa_mix<K>(v, k, form);
        if (sg.dst == kQaoaToGlobal) {
            const idx_t x = qaoa_index(g, item, base);
            const idx_t xs = g.kind == kQaoaHigh ? idx_t(1) << (B0 - 1 + g.C) : idx_t(1) << B0;
#pragma unroll
            for (unsigned e = 0; e < NV; ++e) psi.st(x + e * xs, v[e]);
        } else {
#pragma unroll
            for (unsigned e = 0; e < NV; ++e) vb[base + (e << B0)] = v[e];
        }
    }
    if (sg.dst == kQaoaToGlobal && sets != nthr) release();
}

// Stage r of a chunked item (barriers between stages are the caller's).
template <class CostT, class Mem, class CostMem, class Rel>
ORKAN_HD double qaoa_stage(const QaoaPass& P, unsigned r, const QaoaItem& J, const Mem& psi, const CostMem& cost,
                           double2* vb, const double2* tab, unsigned lc, unsigned tid, unsigned nthr,
                           const Rel& release) {
    const QaoaStage sg = P.stage[r];
    const QaoaGeo& g = P.geo;
    const unsigned K = qaoa_group_bits(g, sg.g);
#define ORKAN_QAOA_M(KK) \
    case KK: return qaoa_m_stage<KK, CostT>(g, sg, J, psi, cost, vb, tab, lc, tid, nthr, release);
#define ORKAN_QAOA_S(KK, BB) \
    case KK: qaoa_s_stage<KK, BB>(g, sg, J, psi, vb, lc, tid, nthr, release); break;
    if (sg.g == 0) {
        switch (K) { ORKAN_QAOA_M(1) ORKAN_QAOA_M(2) ORKAN_QAOA_M(3) default: ORKAN_QAOA_M(4) }
    } else if (sg.g == 1) {
        switch (K) { ORKAN_QAOA_S(1, 4) ORKAN_QAOA_S(2, 4) ORKAN_QAOA_S(3, 4) default: ORKAN_QAOA_S(4, 4) }
    } else if (sg.g == 2) {
        switch (K) { ORKAN_QAOA_S(1, 8) ORKAN_QAOA_S(2, 8) ORKAN_QAOA_S(3, 8) default: ORKAN_QAOA_S(4, 8) }
    } else {
        qaoa_s_stage<1, 12>(g, sg, J, psi, vb, lc, tid, nthr, release);     // 2^13 slots: bit 12
    }
#undef ORKAN_QAOA_M
#undef ORKAN_QAOA_S
    return 0.0;
}

// ---- full items: every one of the 2^n amplitudes in one block ------------------------------
// Layer t runs its m groups rotated, (i + m - t mod m) mod m, so that it starts with the
// group layer t - 1 ended with: that stage applies the end of layer t - 1, the phase of layer t and the
// start of layer t.
struct QaoaFullStage {
    unsigned g, t0, t1;        // group; layers applied in this stage
    bool init, measure, ends;  // first stage; last stage; layer t0's last group
};
ORKAN_HD unsigned qaoa_full_stages(unsigned m, unsigned p) { return m == 1 ? 1u : p * (m - 1) + 1; }
ORKAN_HD QaoaFullStage qaoa_full_stage_desc(unsigned m, unsigned p, unsigned r) {
    QaoaFullStage s;
    s.init = r == 0;
    s.measure = r + 1 == qaoa_full_stages(m, p);
    if (m == 1) {
        s.g = 0;
        s.t0 = 0;
        s.t1 = p - 1;
        s.ends = true;
        return s;
    }
    unsigned t, i;
    if (r < m) { t = 0; i = r; }
    else { t = 1 + (r - m) / (m - 1); i = 1 + (r - m) % (m - 1); }
    s.g = (i + m - (t % m)) % m;
    s.t0 = t;
    s.ends = i == m - 1;
    s.t1 = s.ends && t + 1 < p ? t + 1 : t;
    return s;
}

// Register r's element of a full item's set: the lanes' key flips the low element bits of the
// group at bit 0, whose sets are 2^K slots apart (qaoa_m_set).
template <int K, int B0, class CostT, class CostMem>
ORKAN_HD double qaoa_full_group(const QaoaPass& P, const QaoaTables& T, unsigned pos, unsigned n,
                                const QaoaFullStage& sg, const CostMem& cost, double2* vb, unsigned tid,
                                unsigned nthr) {
    constexpr unsigned NV = 1u << K, nbk = K < 3 ? K : 3;
    const unsigned sets = 1u << (n - K);
    const idx_t row = (idx_t)pos * P.p;
    double acc = 0.0;
    for (unsigned r = tid; r < sets; r += nthr) {
        const unsigned base = (r & ((1u << B0) - 1)) | ((r >> B0) << (B0 + K));
        const unsigned key = B0 == 0 ? (r >> (3 - nbk)) & ((1u << nbk) - 1) : 0u;
        auto slot = [&](unsigned e) { return base | ((e ^ key) << B0); };
        auto phase = [&](double2 (&v)[NV], unsigned l) {
            const double gam = P.gamma[row + l], fs = T.rx[row + l].fs;
            const double2* tab = T.phase + (row + l) * T.tstride;
#pragma unroll
            for (unsigned e = 0; e < NV; ++e)
                v[e] = qaoa_apply_phase(qaoa_phase<CostT>(cost.ld(slot(e)), gam, fs, tab), v[e]);
        };
        double2 v[NV];
        if (sg.init) {
            const double amp0 = 1.0 / sqrt((double)(idx_t(1) << n));
#pragma unroll
            for (unsigned e = 0; e < NV; ++e) v[e] = c2(amp0, 0.0);
            phase(v, 0);
        } else {
#pragma unroll
            for (unsigned e = 0; e < NV; ++e) v[e] = vb[slot(e)];
        }
        for (unsigned t = sg.t0; t <= sg.t1; ++t) {
            if (t > sg.t0) phase(v, t);
            const QaoaRx& rx = T.rx[row + t];
            qaoa_mix<K>(v, rx.k, rx.sform);
        }
        if (sg.measure) {
#pragma unroll
            for (unsigned e = 0; e < NV; ++e) acc += (double)cost.ld(slot(e)) * (v[e].x * v[e].x + v[e].y * v[e].y);
        } else {
#pragma unroll
            for (unsigned e = 0; e < NV; ++e) vb[slot(e)] = v[e];
        }
    }
    return acc;
}

template <class CostT, class CostMem>
ORKAN_HD double qaoa_full_stage(const QaoaPass& P, const QaoaTables& T, unsigned pos, unsigned n, unsigned r,
                                const CostMem& cost, double2* vb, unsigned tid, unsigned nthr) {
    const QaoaFullStage sg = qaoa_full_stage_desc(P.geo.m, P.p, r);
    const unsigned K = qaoa_group_bits(P.geo, sg.g);
#define ORKAN_QAOA_F(KK, BB) \
    case (KK) * 16 + (BB): return qaoa_full_group<KK, BB, CostT>(P, T, pos, n, sg, cost, vb, tid, nthr);
    switch (K * 16 + 4 * sg.g) {
        ORKAN_QAOA_F(1, 0) ORKAN_QAOA_F(2, 0) ORKAN_QAOA_F(3, 0) ORKAN_QAOA_F(4, 0)
        ORKAN_QAOA_F(1, 4) ORKAN_QAOA_F(2, 4) ORKAN_QAOA_F(3, 4) ORKAN_QAOA_F(4, 4)
        ORKAN_QAOA_F(1, 8) ORKAN_QAOA_F(2, 8) ORKAN_QAOA_F(3, 8) ORKAN_QAOA_F(4, 8)
        ORKAN_QAOA_F(1, 12)
        default: break;
    }
#undef ORKAN_QAOA_F
    return 0.0;
}

// ---- shared memory of a pass block -------------------------------------------------------
// [buffers: 2^C amplitudes each][phase tables, one per buffer (byte costs)][items, one per
// buffer][8 partial sums per group warp ...][barriers].  Buffers come first, so every region
// keeps the 128-byte alignment of the base.
constexpr unsigned kQaoaItemBytes = 128;
static_assert(sizeof(QaoaItem) <= kQaoaItemBytes, "item record");

struct QaoaSmem {
    size_t buf, tab, item, red, bar, total;    // offsets
    size_t buf_stride, tab_stride;
};
ORKAN_HD QaoaSmem qaoa_smem(unsigned C, unsigned buffers, unsigned tstride, unsigned threads) {
    QaoaSmem s;
    s.buf_stride = size_t(16) << C;
    s.tab_stride = (size_t(16) * tstride + 127) & ~size_t(127);
    s.buf = 0;
    s.tab = (s.buf_stride * buffers + 127) & ~size_t(127);
    s.item = s.tab + s.tab_stride * buffers;
    s.red = s.item + size_t(kQaoaItemBytes) * buffers;
    s.bar = s.red + ((size_t(8) * (threads / 32 + 1) + 127) & ~size_t(127));
    s.total = s.bar + 8 * (2 * buffers) + 64;
    return s;
}
// Every region aligned for its accesses (16-byte amplitudes, table entries and copies,
// 8-byte sums and barriers).
ORKAN_HD bool qaoa_smem_aligned(unsigned C, unsigned buffers, unsigned tstride, unsigned threads) {
    const QaoaSmem s = qaoa_smem(C, buffers, tstride, threads);
    return s.tab % 16 == 0 && s.buf_stride % 16 == 0 && s.tab_stride % 16 == 0 && s.item % 16 == 0 && s.red % 8 == 0 &&
           s.bar % 8 == 0;
}

}  // namespace orkan
