// dm_direct.cuh - 1-qubit gates and superoperators and controlled flips on density matrices, one element
// group per thread straight from and to memory.
//
// The engine (dm_engine.cuh) stages blocks of the matrix in shared memory, which operations on several qubits
// at once need.  An operation on one qubit needs 2 x 2 groups only, so a thread loads the elements of a
// group, updates and stores them, and no copy descriptor, barrier or staged line lies in between:
//   * small matrices (k_direct_group, up to kDirectSmall qubits) lie in L2 and are bound by the length of one
//     block's chain of steps; one round trip to L2 takes its place (a gate at 8 qubits: 10.4 us of chain
//     down to the 3.5-4 us that its launch takes);
//   * larger ones (k_direct_tile) are bound by HBM; consecutive lanes take consecutive elements and blocks follow
//     the storage order.  H at 14 qubits, us, engine -> direct: packed 856 -> 645 on qubits 0-4, 963 -> 662 on 7, 876
//     -> 832 on the top one; tiled 703 -> 635, 703 -> 652, and 762 against 796 on the top one, which stays with
//     the engine there (direct_wins).  Its 512-byte lines came as one bulk copy each, about 80 copies per us and
//     SM whatever their length; packed lines start at any 16-byte offset on top of that.
//
// Groups of a 1-qubit operation on bit q: rows r0 = u with a zero at q, r1 = r0 | bit, columns c0 (from v)
// and c1 likewise, u >= v.  Then (r0, c0), (r1, c0) and (r1, c1) lie in the stored lower triangle; (r0, c1) does
// where r0 >= c1, and is the conjugate of the stored (c1, r0) otherwise -- for u = v that is (r1, c0) itself.
// Every stored element belongs to one group.  Reference behaviour: src/gate/packed/gate_packed_1q.c:65-104,
// src/gate/tiled/gate_tiled_h.c:28-223, src/channel/channel_packed.c:8-46.
#pragma once

#include "common.cuh"
#include "dm_engine.cuh"
#include "dm_phase.cuh"

namespace orkan {

constexpr unsigned kDirectThreads = 256;
constexpr unsigned kDirectSmall = 10;        // qubits up to which one thread per group is the faster form

// Store element (r, c), r >= c, and, in a diagonal tile of the tiled layout, its mirror image.
template <class Map, class Mem>
ORKAN_HD void direct_store(const Mem& mem, const Map& map, idx_t r, idx_t c, double2 x) {
    mem.st(map.at(r, c), x);
    if (Map::kMirrors && r != c && map.same_storage_block(r, c)) mem.st(map.at(c, r), cconj(x));
}

// Thread t's pair (row index, column index) of a 2^b x 2^b square: the lanes of a warp take the index
// that is contiguous in memory.
template <class Map>
ORKAN_HD void direct_pair(idx_t t, unsigned b, idx_t* row, idx_t* col) {
    const idx_t fast = t & ((idx_t(1) << b) - 1), slow = t >> b;
    *row = Map::kRowContig ? fast : slow;
    *col = Map::kRowContig ? slow : fast;
}

// Operations on a group x = (x00, x01, x10, x11).  above: (r0, c1) lies above the diagonal, and its conjugate
// (c1, r0) is what is stored.
struct DirectMix1 {
    double2 u[4];
    ORKAN_HD bool active(idx_t, idx_t) const { return true; }
    ORKAN_HD void apply(const double2 (&x)[4], double2 (&z)[4], idx_t, idx_t, bool) const {
        double2 y[4];                                  // y = u x, z = y u^dagger
        for (unsigned j = 0; j < 2; ++j) {
            y[j] = cadd(cmul(u[0], x[j]), cmul(u[1], x[2 + j]));
            y[2 + j] = cadd(cmul(u[2], x[j]), cmul(u[3], x[2 + j]));
        }
        for (unsigned i = 0; i < 2; ++i) {
            z[2 * i] = cadd(cmulc(y[2 * i], u[0]), cmulc(y[2 * i + 1], u[1]));
            z[2 * i + 1] = cadd(cmulc(y[2 * i], u[2]), cmulc(y[2 * i + 1], u[3]));
        }
    }
};
struct DirectSuper1 {
    double2 s[16];
    ORKAN_HD bool active(idx_t, idx_t) const { return true; }
    // A superoperator that does not map Hermitian matrices to Hermitian ones has two values for (r0, c1): row 01 of its
    // own, and the conjugate of what row 10 gives (c1, r0).  The stored element's counts.
    ORKAN_HD void apply(const double2 (&x)[4], double2 (&z)[4], idx_t, idx_t, bool above) const {
#pragma unroll
        for (unsigned m = 0; m < 4; ++m) {
            double2 acc = c2(0.0, 0.0);
            if (m == 1 && above) {
#pragma unroll
                for (unsigned j = 0; j < 4; ++j) super_fma(acc, cconj(s[8 + (j == 1 ? 2 : j == 2 ? 1 : j)]), x[j]);
            } else {
#pragma unroll
                for (unsigned j = 0; j < 4; ++j) super_fma(acc, s[4 * m + j], x[j]);
            }
            z[m] = acc;
        }
    }
};
// Controlled flip (X, CX, CCX, and any other phases of the kernel layer): rows that have all control bits exchange with phases p0 (new target
// bit 0) and p1, columns likewise with the conjugate phases; groups without either stay.  UNIT: both
// phases are 1 and values only move.
template <bool UNIT>
struct DirectFlip {
    unsigned long long ctrl;
    double2 p0, p1;
    ORKAN_HD bool active(idx_t r0, idx_t c0) const { return (r0 & ctrl) == ctrl || (c0 & ctrl) == ctrl; }
    ORKAN_HD void apply(const double2 (&x)[4], double2 (&z)[4], idx_t r0, idx_t c0, bool) const {
        const bool cr = (r0 & ctrl) == ctrl, cc = (c0 & ctrl) == ctrl;
        double2 y[4];
#pragma unroll
        for (unsigned j = 0; j < 2; ++j) {
            y[j] = cr ? x[2 + j] : x[j];
            y[2 + j] = cr ? x[j] : x[2 + j];
            if (!UNIT && cr) {
                y[j] = cmul(p0, y[j]);
                y[2 + j] = cmul(p1, y[2 + j]);
            }
        }
#pragma unroll
        for (unsigned i = 0; i < 2; ++i) {
            z[2 * i] = cc ? y[2 * i + 1] : y[2 * i];
            z[2 * i + 1] = cc ? y[2 * i] : y[2 * i + 1];
            if (!UNIT && cc) {
                z[2 * i] = cmulc(z[2 * i], p0);
                z[2 * i + 1] = cmulc(z[2 * i + 1], p1);
            }
        }
    }
};

// Y and CY: as DirectFlip with p0 = -i, p1 = i.  The values move and turn by quarters: no product that would make NaN of
// an infinity's zero part.
struct DirectFlipY {
    unsigned long long ctrl;
    static ORKAN_HD double2 turn(double2 a) { return c2(-a.y, a.x); }           // times i
    static ORKAN_HD double2 back(double2 a) { return c2(a.y, -a.x); }           // times -i
    ORKAN_HD bool active(idx_t r0, idx_t c0) const { return (r0 & ctrl) == ctrl || (c0 & ctrl) == ctrl; }
    ORKAN_HD void apply(const double2 (&x)[4], double2 (&z)[4], idx_t r0, idx_t c0, bool) const {
        const bool cr = (r0 & ctrl) == ctrl, cc = (c0 & ctrl) == ctrl;
        double2 y[4];
#pragma unroll
        for (unsigned j = 0; j < 2; ++j) {
            y[j] = cr ? back(x[2 + j]) : x[j];
            y[2 + j] = cr ? turn(x[j]) : x[2 + j];
        }
#pragma unroll
        for (unsigned i = 0; i < 2; ++i) {
            z[2 * i] = cc ? turn(y[2 * i + 1]) : y[2 * i];
            z[2 * i + 1] = cc ? back(y[2 * i]) : y[2 * i + 1];
        }
    }
};

// Group (u, v) of an operation on bit q.
template <class Map, class Mem, class Op>
ORKAN_HD void direct_group(const Mem& mem, const Map& map, unsigned q, const Op& op, idx_t u, idx_t v) {
    if (u < v) return;
    const idx_t bit = idx_t(1) << q;
    const idx_t r0 = insert0(u, q), c0 = insert0(v, q), r1 = r0 | bit, c1 = c0 | bit;
    if (!op.active(r0, c0)) return;
    const bool below = r0 >= c1;                       // (r0, c1) is stored as itself
    double2 x[4], z[4];
    x[0] = mem.ld(map.at(r0, c0));
    x[2] = mem.ld(map.at(r1, c0));
    x[3] = mem.ld(map.at(r1, c1));
    x[1] = u == v ? cconj(x[2]) : below ? mem.ld(map.at(r0, c1)) : cconj(mem.ld(map.at(c1, r0)));
    op.apply(x, z, r0, c0, !below);
    direct_store(mem, map, r0, c0, z[0]);
    direct_store(mem, map, r1, c0, z[2]);
    direct_store(mem, map, r1, c1, z[3]);
    if (u != v) {
        if (below) direct_store(mem, map, r0, c1, z[1]);
        else direct_store(mem, map, c1, r0, cconj(z[1]));
    }
}

// Small matrices: the group of thread t.
template <class Map, class Mem, class Op>
ORKAN_HD void direct_small(const Mem& mem, const Map& map, unsigned n, unsigned q, const Op& op, idx_t t) {
    if (t >> (2 * (n - 1))) return;
    idx_t u, v;
    direct_pair<Map>(t, n - 1, &u, &v);
    direct_group(mem, map, q, op, u, v);
}

// Larger matrices: a block takes a 32 x 32 tile (U, V) of groups, U >= V.  The partner of (r0, c1) is uniform over a
// tile off the diagonal when q >= 5 (the bits of u and v from q up decide), and itself stored when q < 5.
// Where it is transposed, neighbouring lanes would fetch neighbouring columns, so the tile of (c1, r0) goes through
// shared memory: lanes run along the index that is contiguous for (c1, r0) on the way in and out (phases 0 and
// 2) and along the other one for the update (phase 1).  Tiles on the diagonal take direct_group.
constexpr unsigned kDirectTile = 32, kDirectPitch = 33;

struct DirectWhere {
    idx_t U, V;
    bool diag, transposed;
};
// Tiles in storage order: row by row for the tiled layout, column by column for the packed one.
template <class Map>
ORKAN_HD DirectWhere direct_where(idx_t block, unsigned n, unsigned q) {
    DirectWhere w;
    tri_unrank_f(block, &w.U, &w.V);
    if (Map::kRowContig) {
        const idx_t last = (idx_t(1) << (n - 6)) - 1, a = w.U, b = w.V;
        w.U = last - b;
        w.V = last - a;
    }
    w.diag = w.U == w.V;
    w.transposed = !w.diag && q >= 5 && (w.U >> (q - 5)) == (w.V >> (q - 5));
    return w;
}
// Group (u, v) of a tile for fast index f (contiguous in memory) and slow index o.
template <class Map>
ORKAN_HD void direct_tile_uv(const DirectWhere& w, unsigned f, unsigned o, idx_t* u, idx_t* v) {
    *u = w.U * kDirectTile + (Map::kRowContig ? f : o);
    *v = w.V * kDirectTile + (Map::kRowContig ? o : f);
}
// Can an element off the diagonal tiles have a mirror image?  (Storage tiles of 32 and less hold no two rows of
// a tile of groups there.)
template <class Map>
ORKAN_HD bool direct_mirrors(const Map& map) { return Map::kMirrors && map.log_tdim() > 5; }

// Phase 1: the update of a tile's groups.  TR: the tile of (c1, r0) is staged in sh.
template <bool TR, class Map, class Mem, class Op>
ORKAN_HD void direct_tile_update(const Mem& mem, const Map& map, unsigned q, const Op& op, const DirectWhere& w,
                                 double2* sh, unsigned tid, unsigned nthr) {
    const idx_t bit = idx_t(1) << q;
    const bool mirrors = direct_mirrors(map);
    // one group at a time: two (their loads issued together) need 78-128 registers instead of 56-80, and
    // the blocks lost cost more than they gain (H at 14 q: 740 against 640 us tiled, 650 against 645 packed)
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
    for (unsigned e = tid; e < kDirectTile * kDirectTile; e += nthr) {
        const unsigned f = e % kDirectTile, o = e / kDirectTile;
        idx_t u, v;
        direct_tile_uv<Map>(w, f, o, &u, &v);
        const idx_t r0 = insert0(u, q), c0 = insert0(v, q), r1 = r0 | bit, c1 = c0 | bit;
        if (!op.active(r0, c0)) continue;
        const idx_t a00 = map.at(r0, c0), a10 = map.at(r1, c0), a11 = map.at(r1, c1);
        const idx_t a01 = TR ? 0 : map.at(r0, c1);
        double2& s01 = sh[f * kDirectPitch + o];
        double2 x[4], z[4];
        x[0] = mem.ld(a00);
        x[2] = mem.ld(a10);
        x[3] = mem.ld(a11);
        x[1] = TR ? s01 : mem.ld(a01);
        op.apply(x, z, r0, c0, TR);
        if (mirrors) {
            direct_store(mem, map, r0, c0, z[0]);
            direct_store(mem, map, r1, c0, z[2]);
            direct_store(mem, map, r1, c1, z[3]);
        } else {
            mem.st(a00, z[0]);
            mem.st(a10, z[2]);
            mem.st(a11, z[3]);
        }
        if (TR) s01 = z[1];
        else if (mirrors) direct_store(mem, map, r0, c1, z[1]);
        else mem.st(a01, z[1]);
    }
}
template <class Map, class Mem, class Op>
ORKAN_HD void direct_tile_phase(int phase, const Mem& mem, const Map& map, unsigned q, const Op& op,
                                const DirectWhere& w, double2* sh, unsigned tid, unsigned nthr) {
    if (phase == 1) {
        if (w.transposed) direct_tile_update<true>(mem, map, q, op, w, sh, tid, nthr);
        else direct_tile_update<false>(mem, map, q, op, w, sh, tid, nthr);
        return;
    }
    const idx_t bit = idx_t(1) << q;
    for (unsigned e = tid; e < kDirectTile * kDirectTile; e += nthr) {
        const unsigned o = e % kDirectTile, f = e / kDirectTile;
        idx_t u, v;
        direct_tile_uv<Map>(w, f, o, &u, &v);
        const idx_t r0 = insert0(u, q), c0 = insert0(v, q), c1 = c0 | bit;
        if (!op.active(r0, c0)) continue;
        double2& s = sh[f * kDirectPitch + o];
        if (phase == 0) s = cconj(mem.ld(map.at(c1, r0)));
        else if (direct_mirrors(map)) direct_store(mem, map, c1, r0, cconj(s));
        else mem.st(map.at(c1, r0), cconj(s));
    }
}

// SWAP of bits a and b: element (r, c) takes the value at (pi r, pi c).  The thread of the element that comes
// first in (row, column) order exchanges the pair; an element that is its own conjugate partner is conjugated.
template <class Map, class Mem>
ORKAN_HD void direct_swap(const Mem& mem, const Map& map, unsigned n, unsigned a, unsigned b, idx_t t) {
    if (t >> (2 * n)) return;
    idx_t r, c;
    direct_pair<Map>(t, n, &r, &c);
    if (r < c) return;
    const idx_t m = (idx_t(1) << a) | (idx_t(1) << b);
    auto pi = [&](idx_t x) { return (x & m) && (x & m) != m ? x ^ m : x; };
    const idx_t pr = pi(r), pc = pi(c);
    if (pr == r && pc == c) return;
    const bool flip = pr < pc;
    const idx_t r2 = flip ? pc : pr, c2i = flip ? pr : pc;
    if (r2 == r && c2i == c) {
        direct_store(mem, map, r, c, cconj(mem.ld(map.at(r, c))));
        return;
    }
    if (r2 < r || (r2 == r && c2i < c)) return;
    const double2 x = mem.ld(map.at(r, c)), y = mem.ld(map.at(r2, c2i));
    direct_store(mem, map, r, c, flip ? cconj(y) : y);
    direct_store(mem, map, r2, c2i, flip ? cconj(x) : x);
}

// Phase update of element (r, c), r > c (the diagonal has factor 1).
template <class Map, class Mem, class Factor>
ORKAN_HD void direct_phase(const Mem& mem, const Map& map, unsigned n, const Factor& fac, idx_t t) {
    if (t >> (2 * n)) return;
    idx_t r, c;
    direct_pair<Map>(t, n, &r, &c);
    double2 f;
    if (r <= c || !fac.factor(r, c, &f)) return;
    direct_store(mem, map, r, c, phase_apply(f, mem.ld(map.at(r, c))));
}

#ifdef __CUDACC__
template <class Map, class Op>
__global__ void __launch_bounds__(kDirectThreads) k_direct_tile(DevMem mem, Map map, unsigned n, unsigned q, Op op) {
    __shared__ double2 sh[kDirectTile * kDirectPitch];
    const unsigned tid = threadIdx.x;
    const DirectWhere w = direct_where<Map>(blockIdx.x, n, q);
    if (w.diag) {
        for (unsigned e = tid; e < kDirectTile * kDirectTile; e += kDirectThreads) {
            idx_t u, v;
            direct_tile_uv<Map>(w, e % kDirectTile, e / kDirectTile, &u, &v);
            direct_group(mem, map, q, op, u, v);
        }
        return;
    }
    if (w.transposed) {
        direct_tile_phase(0, mem, map, q, op, w, sh, tid, kDirectThreads);
        __syncthreads();
    }
    direct_tile_phase(1, mem, map, q, op, w, sh, tid, kDirectThreads);
    if (w.transposed) {
        __syncthreads();
        direct_tile_phase(2, mem, map, q, op, w, sh, tid, kDirectThreads);
    }
}
template <class Map, class Op>
__global__ void __launch_bounds__(kDirectThreads) k_direct_group(DevMem mem, Map map, unsigned n, unsigned q, Op op) {
    direct_small(mem, map, n, q, op, (idx_t)blockIdx.x * kDirectThreads + threadIdx.x);
}
template <class Map>
__global__ void __launch_bounds__(kDirectThreads) k_direct_swap(DevMem mem, Map map, unsigned n, unsigned a, unsigned b) {
    direct_swap(mem, map, n, a, b, (idx_t)blockIdx.x * kDirectThreads + threadIdx.x);
}
template <class Map, class Factor>
__global__ void __launch_bounds__(kDirectThreads) k_direct_phase(DevMem mem, Map map, unsigned n, Factor fac) {
    direct_phase(mem, map, n, fac, (idx_t)blockIdx.x * kDirectThreads + threadIdx.x);
}
#endif

}  // namespace orkan
