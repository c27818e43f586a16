// The persistent work-queue solve kernel (sm_100a), shared by the per-G
// instantiation files gf_persist_g*.cu (one translation unit per group size,
// so that the variants compile in parallel).
//
// CTAs sized to the SMs; groups of G threads pull cells from an atomic work
// queue until it is empty. G <= 32: several groups per CTA (at most 128
// threads); G = 64, 128, 256: one group (one cell at a time) per CTA. The
// per-cell workspace lives in shared memory (SHARED) or in an HBM slot per
// resident group. Mixed mechanisms are selected by the per-cell id.
#pragma once

#include <cuda_runtime.h>

#include "gf_device.cuh"
#include "gf_internal.h"

namespace gf {

constexpr int kMaxMechs = 4;


struct MechSet {
    DevMech m[kMaxMechs];
    int n;
};

// The cell's mechanism, or null for an id outside the solver's mechanisms: the
// cell is then not integrated, its status says so, and it counts as failed.
__device__ __forceinline__ const DevMech* pick(const MechSet& P, const LaunchArgs& a, long long cell) {
    const int id = a.mech_id ? a.mech_id[cell] : 0;
    return (id >= 0 && id < P.n) ? &P.m[id] : nullptr;
}

// Such a cell leaves the solve unchanged: its output row is a copy of its
// input row (the whole row stride), its RR row is zero, its counters are zero
// and its deltaTChem is left as it was; it is left out of the min over cells.
template <int G>
__device__ __forceinline__ void reject_cell(const Grp<G>& g, const LaunchArgs& a, long long cell) {
    if (a.Ynew) {
        const double* yi = a.Y0 + (size_t)cell * a.ld_y;
        double* yo = a.Ynew + (size_t)cell * a.ld_y;
        for (int i = g.lane; i < a.ld_y; i += G) yo[i] = yi[i];
    }
    if (a.RR)
        for (int i = g.lane; i < a.ld_rr; i += G) a.RR[(size_t)cell * a.ld_rr + i] = 0.0;
    if (g.lane == 0) {
        if (a.status) a.status[cell] = GF_CELL_BAD_MECHANISM;
        if (a.counters) {
            a.counters[2 * cell] = 0;
            a.counters[2 * cell + 1] = 0;
        }
        atomicAdd(a.queue + 4, 1ull);
    }
}

// Registers per thread the kernel is compiled for: SLIM = 1, at most 128
// (512 resident threads per SM); SLIM = 2 (a warp per cell, more cells than are
// resident otherwise), at most 168: twelve warps per SM instead of eight;
// otherwise up to 255, except for 64 threads per cell, capped at 200 so that five 64-thread CTAs fit an SM's registers
// (their workspaces fit its shared memory: 45 KB each at 53 species).
template <int G>
struct PersistShape {
    static constexpr int max_regs(int slim) { return slim == 2 ? 168 : (slim ? 128 : (G == 64 ? 200 : 255)); }
};

// NB: columns per LU panel of the blocked form (groups of less than 32 threads,
// m > 128); MS: the matrix sizes that it is compiled for (process_cell); with a
// range of sizes the workspace is padded to its largest (persistent_ranged_fn).
// kAllRanges: every range of sizes to 128, each with its own code and layout.
constexpr int kAllRanges = -1;
template <int G, bool SHARED, int SLIM, int NB = 8, int MS = 0>
__global__ void __maxnreg__(PersistShape<G>::max_regs(SLIM))
    persistent_kernel(const MechSet P, const LaunchArgs a, int ws_per_cell, long long n_slots) {
    extern __shared__ double smem[];
    Grp<G> g;
    const int gpb = G > 32 ? 1 : blockDim.x / G;
    const int gib = G > 32 ? 0 : threadIdx.x / G;
    const long long slot = (long long)blockIdx.x * gpb + gib;
    for (;;) {
        long long cell = 0;
        if (g.lane == 0) cell = (long long)atomicAdd(a.queue, 1ull);
        cell = g.bcast_ll(cell, 0);
        if (cell >= a.n_cells) break;
        const DevMech* Mp = pick(P, a, cell);
        if (!Mp) {
            reject_cell(g, a, cell);
            continue;
        }
        const DevMech& M = *Mp;
        if (SHARED) {
            const WsC w{smem + (size_t)gib * ws_per_cell};
            if constexpr (MS == kAllRanges) {
                if (!(process_cell<G, WsC, false, NB, -32, 32>(g, M, w, a, (int)cell) ||
                      process_cell<G, WsC, false, NB, -64, 64>(g, M, w, a, (int)cell) ||
                      process_cell<G, WsC, false, NB, -128, 128>(g, M, w, a, (int)cell)))
                    reject_cell(g, a, cell);
            } else {
                if (!process_cell<G, WsC, false, NB, MS, size_pad(MS)>(g, M, w, a, (int)cell))
                    reject_cell(g, a, cell);
            }
        } else if (G == 1) {
            process_cell<G, WsS, false, NB, MS>(g, M, WsS{a.ws + slot, n_slots}, a, (int)cell);
        } else {
            process_cell<G, WsC, false, NB, MS>(g, M, WsC{a.ws + slot * ws_per_cell}, a, (int)cell);
        }
    }
}

template <int G, int NB = 8, int MS = 0>
const void* persistent_variant(bool shared, int slim) {
    if (shared)
        return slim ? reinterpret_cast<const void*>(&persistent_kernel<G, true, 1, NB, MS>)
                    : reinterpret_cast<const void*>(&persistent_kernel<G, true, 0, NB, MS>);
    return slim ? reinterpret_cast<const void*>(&persistent_kernel<G, false, 1, NB, MS>)
                : reinterpret_cast<const void*>(&persistent_kernel<G, false, 0, NB, MS>);
}

// The tuned variants of the 32-, 64-, 96- and 128-thread forms (gf_persist_g<G>_tuned.cu):
// LU panels of 4 or 16 columns (workspace in shared memory; they matter for m > 128
// only, lu_factor), and the matrix size fixed at compile time for the 10-, 53- and
// 100-species mechanisms (m = 11, 54, 101; workspace in shared memory or HBM; 4-column
// panels are accepted for m = 54, and are the same kernel). Each with the register budget the form is usually run with
// (SLIM for 96 and 128 threads); nullptr for a variant that is not compiled.
constexpr int kTunedSlim(int G) { return (G == 128 || G == 96) ? 1 : 0; }
template <int G, int S, int NB, int MS>
const void* tuned_kernel(bool shared) {
    return shared ? reinterpret_cast<const void*>(&persistent_kernel<G, true, S, NB, MS>)
                  : reinterpret_cast<const void*>(&persistent_kernel<G, false, S, NB, MS>);
}
template <int G>
const void* persistent_tuned_variant(bool shared, int slim, int nb, int ms) {
    if (slim != kTunedSlim(G)) return nullptr;
    constexpr int S = kTunedSlim(G);
    if (ms == 0) {
        if (!shared) return nullptr;
        if (nb == 4) return tuned_kernel<G, S, 4, 0>(true);
        if (nb == 16) return tuned_kernel<G, S, 16, 0>(true);
        return nullptr;
    }
    if (ms == 54 && (nb == 8 || nb == 4)) return tuned_kernel<G, S, 8, 54>(shared);
    if (nb != 8) return nullptr;
    if (ms == 11) return tuned_kernel<G, S, 8, 11>(shared);
    if (ms == 101) return tuned_kernel<G, S, 8, 101>(shared);
    return nullptr;
}

// defined in gf_persist_g<G>.cu
const void* persistent_fn_g1(bool shared, int slim);
const void* persistent_fn_g2(bool shared, int slim);
const void* persistent_fn_g4(bool shared, int slim);
const void* persistent_fn_g8(bool shared, int slim);
const void* persistent_fn_g16(bool shared, int slim);
const void* persistent_fn_g32(bool shared, int slim);
// a warp per cell with at most 168 registers, workspace in shared memory; ms: 11 or 0
const void* persistent_dense_fn_g32(int ms);
const void* persistent_fn_g64(bool shared, int slim);
const void* persistent_fn_g96(bool shared, int slim);
const void* persistent_fn_g128(bool shared, int slim);
const void* persistent_fn_g256(bool shared, int slim);
// The 256-thread form, workspace in shared memory, for matrix sizes to 128: the
// form of launches that mix mechanisms and of those with one cell per SM. Each
// range of sizes (fix_size) has its own code, with its own rows per lane and
// tiles, and a vector of the workspace has room for the range's largest size, so
// that the vectors lie at places known at compile time. Against one code for any
// size, 701 cells of 70, 75, 90 and 120 species: 26.5, 20.3, 62.4 and 61.3 ->
// 22.3, 16.9, 52.1 and 50.3 ms, 148 cells of 70: 7.7 -> 6.5 ms. With several CTAs
// per SM the ranges' instructions would compete for the caches.
const void* persistent_ranged_fn_g256();
// The same for the other forms that the default rule takes (default_launch), a kernel
// per range (32, 64 or 128, the largest size) for launches whose mechanisms share
// one; nullptr for a pair that is not compiled. gf_persist_g<G>_ranged.cu
// 8,192 cells against one code for any size: a warp per cell, 20 and 31 species
// 16.7 -> 12.2 and 27.5 -> 18.3 ms (65,536 of 10 species 38.1 -> 22.3; compiled for
// m = 11 19.1); 64 threads, 44, 52 and 60 species 59.4, 36.6 and 135 -> 50.1, 30.1 and
// 106; 128 threads, 66, 75 and 90 species 148, 119 and 275 -> 128, 99 and 230.
const void* persistent_ranged_fn_g32(int range, bool dense);
const void* persistent_ranged_fn_g64(int range);
const void* persistent_ranged_fn_g128(int range);
// defined in gf_persist_g<G>_tuned.cu
const void* persistent_tuned_fn_g32(bool shared, int slim, int nb, int ms);
const void* persistent_tuned_fn_g64(bool shared, int slim, int nb, int ms);
const void* persistent_tuned_fn_g96(bool shared, int slim, int nb, int ms);
const void* persistent_tuned_fn_g128(bool shared, int slim, int nb, int ms);

#ifdef GF_PHASE_TIMERS
// phase-timer accumulators of the gf_persist_g<G>.cu units (profiling builds)
int phase_cycles_g1(unsigned long long* out, int reset);
int phase_cycles_g2(unsigned long long* out, int reset);
int phase_cycles_g4(unsigned long long* out, int reset);
int phase_cycles_g8(unsigned long long* out, int reset);
int phase_cycles_g16(unsigned long long* out, int reset);
int phase_cycles_g32(unsigned long long* out, int reset);
int phase_cycles_g64(unsigned long long* out, int reset);
int phase_cycles_g96(unsigned long long* out, int reset);
int phase_cycles_g128(unsigned long long* out, int reset);
int phase_cycles_g256(unsigned long long* out, int reset);
int phase_cycles_adj(unsigned long long* out, int reset);
// the tuned variants' units (gf_persist_g<G>_tuned.cu)
int phase_cycles_g32t(unsigned long long* out, int reset);
int phase_cycles_g64t(unsigned long long* out, int reset);
int phase_cycles_g96t(unsigned long long* out, int reset);
int phase_cycles_g128t(unsigned long long* out, int reset);
// the ranged kernels' units (gf_persist_g<G>_ranged.cu)
int phase_cycles_g32r(unsigned long long* out, int reset);
int phase_cycles_g64r(unsigned long long* out, int reset);
int phase_cycles_g128r(unsigned long long* out, int reset);
#endif

}  // namespace gf
