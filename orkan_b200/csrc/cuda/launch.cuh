// launch.cuh - launch helpers shared by the translation units of the kernel layer:
// the SM count of the current device, grid sizing, the counted launch check, and the
// density-matrix phase-pass launcher used by gates and exp_diag.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "dm_direct.cuh"
#include "dm_phase.cuh"

namespace orkan {

// Multiprocessors of the current device (cached per device; 148 on B200).
int sm_count();

// Counts one kernel launch (orkan_cu_launch_count) and returns the launch status.
int finish_launch();

// Grid cap of the streaming kernels: one block per share of work, no persistent loop.  The
// blocks are scheduled by the hardware as SMs free up, which measured 15 % faster at 30
// qubits than grid-stride loops over 8 blocks per SM (the register use of those kernels
// leaves room for four 256-thread blocks per SM, so such a grid ran in two rounds).
constexpr unsigned kFullGrid = 0x7fffffffu;

// Blocks for total_units of work at work_per_block_units per block, at least 1, at most cap.
inline unsigned grid_for(idx_t work_per_block_units, idx_t total_units, unsigned cap) {
    idx_t g = (total_units + work_per_block_units - 1) / work_per_block_units;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return (unsigned)g;
}

// Items (S x S sub-tiles) per block of the phase pass: 2, or 1 / 4 / 8 through the tuning
// knob ORKAN_PHASE_ITEMS, read once.
unsigned phase_items_per_block();

// Threads one per index of a 2^bits range.
inline unsigned direct_grid(unsigned bits) { return grid_for(kDirectThreads, idx_t(1) << bits, kFullGrid); }

// Elementwise phase pass over a packed (layout 1) or tiled (layout 2) density matrix: one thread per element
// up to kDirectSmall qubits (8 q: 4.0 against 6.2 us; from 11 q on the pass that skips whole inactive items
// is faster, 8.3 against 12.4 us).  Above that, 1-qubit gates on packed storage go column by column.
template <class Factor>
int launch_phase(int layout, unsigned log_tile, void* rho, unsigned n, const Factor& fac, cudaStream_t st) {
    if (n <= kDirectSmall) {
        DevMem mem{static_cast<double2*>(rho)};
        const unsigned grid = direct_grid(2 * n);
        if (layout == 1) k_direct_phase<<<grid, kDirectThreads, 0, st>>>(mem, PackedMap{idx_t(1) << n}, n, fac);
        else k_direct_phase<<<grid, kDirectThreads, 0, st>>>(mem, TiledMap{idx_t(1) << n, log_tile}, n, fac);
        return finish_launch();
    }
    if constexpr (std::is_same<Factor, GateFactor1>::value) {
        if (layout == 1 && n <= 21) {                   // (more blocks than a grid has beyond)
            k_dm_phase_columns<<<(unsigned)phase_column_blocks(n), kColThreads, 0, st>>>(
                DevMem{static_cast<double2*>(rho)}, PackedMap{idx_t(1) << n}, fac);
            return finish_launch();
        }
    }
    const PhaseGeom g = phase_geometry(n, layout == 2 ? log_tile : 5u);
    const unsigned grid = grid_for(phase_items_per_block(), g.items, kFullGrid);
    DevMem mem{static_cast<double2*>(rho)};
    if (layout == 1) {
        k_dm_phase<PackedMap, Factor><<<grid, kPhaseThreads, 0, st>>>(mem, PackedMap{idx_t(1) << n}, g, fac);
    } else {
        k_dm_phase<TiledMap, Factor><<<grid, kPhaseThreads, 0, st>>>(mem, TiledMap{idx_t(1) << n, log_tile}, g, fac);
    }
    return finish_launch();
}

}  // namespace orkan
