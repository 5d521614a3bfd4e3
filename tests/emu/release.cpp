// release.cpp - what a batched pass reads after it hands its buffers back -- TEST INFRASTRUCTURE ONLY.
//
// A stage that stores an item releases the item's buffer, phase table and record as soon as it needs them no
// more, and the staging warps may then overwrite all three with the next item's.  Threads of a block arrive in
// any order, so a thread must read none of them after its own release.  Here every release overwrites the
// three, and what the thread stores or sums afterwards is compared with a run whose releases do nothing.
// It is never used by the product library.
#include "../../orkan_b200/csrc/cuda/qaoa.cuh"

#include <math.h>
#include <string.h>
#include <vector>

using namespace orkan;

namespace {

struct Psi {
    double2* p;
    void st(idx_t i, double2 v) const { p[i] = v; }
    void cp16(double2* dst, idx_t i) const { *dst = p[i]; }
    void bulk_load(double2* dst, idx_t i, unsigned n, void*) const { memcpy(dst, p + i, n * sizeof(double2)); }
};
template <class CostT>
struct Costs {
    const CostT* p;
    CostT ld(unsigned i) const { return p[i]; }
    template <int K>
    void words(uint32_t* w, unsigned i) const { memcpy(w, p + i, size_t(1) << K); }
};

// What a release gives up, and the number of releases of the running thread.
struct Shared {
    std::vector<double2> vb, tab;
    QaoaItem J;
    unsigned released = 0;
};
struct Poison {
    Shared* s;
    bool armed;
    void operator()() const {
        ++s->released;
        if (!armed) return;
        const double2 bad = c2(NAN, NAN);
        for (auto& v : s->vb) v = bad;
        for (auto& v : s->tab) v = bad;
        s->J.psi = nullptr;
        s->J.cost = nullptr;
        s->J.ka = s->J.kb = s->J.gamma = s->J.fs = NAN;
        s->J.sa = s->J.sb = 1 - s->J.sa;
        s->J.item = ~idx_t(0);
    }
};

bool same(double2 a, double2 b) { return a.x == b.x && a.y == b.y; }

// One item of pass j: threads whose result depends on what they gave up (*late), threads that do not
// release exactly once (*count).
template <class CostT>
int run(unsigned n, unsigned C, unsigned p, unsigned j, unsigned nthr, unsigned* late, unsigned* count) {
    const unsigned tstride = 8;
    std::vector<double> co(p), si(p), gamma(p);
    for (unsigned k = 0; k < p; ++k) {
        co[k] = cos(0.3 + 0.7 * k);
        si[k] = sin(0.3 + 0.7 * k);
        gamma[k] = 0.4 + 0.2 * k;
    }
    std::vector<QaoaRx> rx(p);
    qaoa_rx_coeffs(co.data(), si.data(), p, n, C, rx.data());
    const idx_t half = idx_t(1) << (n - 1);
    std::vector<double2> psi((size_t)half), want, got;
    std::vector<CostT> cost((size_t)half);
    for (idx_t i = 0; i < half; ++i) {
        psi[(size_t)i] = c2(1.0 + (double)(i % 97), 2.0 - (double)(i % 89));
        cost[(size_t)i] = (CostT)(i % tstride);
    }
    QaoaInst I{};
    I.psi = psi.data();
    I.cost = cost.data();
    I.n = n;
    QaoaPass P{};
    P.inst = &I;
    P.ninst = 1;
    P.kind = j % 2 == 0 ? kQaoaLow : kQaoaHigh;
    P.C = C;
    P.items = qaoa_items(n, C, P.kind);
    P.gamma = gamma.data();
    P.p = p;
    P.pass = j;
    qaoa_pass_setup(P, n, sizeof(CostT) == 1);
    std::vector<double2> phase((size_t)p * tstride);
    for (unsigned i = 0; i < p * tstride; ++i) phase[i] = c2(cos(0.1 * i), sin(0.1 * i));
    const QaoaTables T{phase.data(), rx.data(), tstride};
    const idx_t w = P.items - 1;
    Shared s;
    s.vb.resize(size_t(1) << C);
    s.tab.assign(tstride, c2(0.0, 0.0));
    if (P.layer_phase >= 0) s.tab.assign(phase.begin() + P.layer_phase * tstride, phase.begin() + (P.layer_phase + 1) * tstride);
    s.J = qaoa_item(P, T, I, w, sizeof(CostT));
    if (P.layer_a >= 0)
        for (unsigned t = 0; t < nthr; ++t) qaoa_fill(P.geo, Psi{psi.data()}, w, s.vb.data(), nullptr, t, nthr);
    *late = *count = 0;
    for (unsigned r = 0; r < P.nreg; ++r)
        for (unsigned t = 0; t < nthr; ++t) {
            const bool last = r + 1 == P.nreg;
            auto go = [&](std::vector<double2>& out, bool poison) {
                s.released = 0;
                return qaoa_stage<CostT>(P, r, s.J, Psi{out.data()}, Costs<CostT>{static_cast<const CostT*>(s.J.cost)},
                                         s.vb.data(), s.tab.data(), C, t, nthr, Poison{&s, poison});
            };
            if (!last) {
                go(psi, false);
                *count += s.released != 0;
                continue;
            }
            want = psi;
            got = psi;
            const double a = go(want, false);
            *count += s.released != 1;
            const Shared keep = s;
            const double b = go(got, true);
            s = keep;
            bool ok = a == b;
            for (idx_t i = 0; i < half && ok; ++i) ok = same(want[(size_t)i], got[(size_t)i]);
            *late += !ok;
        }
    return 0;
}

}  // namespace

extern "C" int emu_qaoa_release(unsigned n, unsigned C, int bytes, unsigned p, unsigned j, unsigned nthr,
                                unsigned* late, unsigned* count) {
    if (n <= C || n > 2 * C || j > p || C > kQaoaMaxC) return -1;
    return bytes ? run<uint8_t>(n, C, p, j, nthr, late, count) : run<double>(n, C, p, j, nthr, late, count);
}
