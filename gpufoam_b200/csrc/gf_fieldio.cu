// The plugin's host glue on the device: the gather of OpenFOAM's per-species
// fields into the solve's cell-major states (getY0,
// gpuChemistryModels/gpuChemistryModel/gpuChemistryModel.C:33-53) and the
// scatter of the cell-major rates back into per-species fields
// (computeRRAndChemDeltaT, gpuChemistryModel.C:351-356). Both are transposes
// through a shared-memory tile of kTileCells cells, so that the field-side
// accesses (a warp: 32 consecutive cells of one field) and the cell-side
// accesses (a warp: one cell's row) are both coalesced. HBM-bound data movement,
// no arithmetic: what counts is the bytes in flight, so every warp issues all
// loads of its share of a tile before it stores them. 500,000 cells of 53 species, heat release
// included (1.08 GB): 222 us; tiles of 16 cells with a division per element and
// an output cleared first took 334.
#include <algorithm>

#include "gf_internal.h"

namespace gf {

namespace {

constexpr int kTileCells = 32;
constexpr int kTileThreads = 256;
constexpr int kTileWarps = kTileThreads / 32;
constexpr int kInFlight = 8;  // loads of a thread in flight

struct FieldPtrs {
    const double* p[GF_MAX_SPECIES];
};
struct FieldOutPtrs {
    double* p[GF_MAX_SPECIES];
};

// y[c * ld + e] = field_e[c], e < nS the species, nS T, nS + 1 p
__global__ void __launch_bounds__(kTileThreads)
    gather_states_kernel(const FieldPtrs Y, const double* T, const double* p, int n, int nS, double* y, int ld) {
    extern __shared__ double tile[];  // [kTileCells][ne | 1]
    const int ne = nS + 2, lt = ne | 1;
    const int wid = threadIdx.x >> 5, l = threadIdx.x & 31;
    for (long long c0 = (long long)blockIdx.x * kTileCells; c0 < n; c0 += (long long)gridDim.x * kTileCells) {
        const int nc = n - c0 < kTileCells ? (int)(n - c0) : kTileCells;
        for (int e0 = wid; e0 < ne; e0 += kTileWarps * kInFlight) {
            double v[kInFlight];
#pragma unroll
            for (int k = 0; k < kInFlight; ++k) {
                const int e = e0 + k * kTileWarps;
                if (e < ne && l < nc) v[k] = __ldcs((e < nS ? Y.p[e] : (e == nS ? T : p)) + c0 + l);
            }
#pragma unroll
            for (int k = 0; k < kInFlight; ++k) {
                const int e = e0 + k * kTileWarps;
                if (e < ne && l < nc) tile[l * lt + e] = v[k];
            }
        }
        __syncthreads();
        for (int j = wid; j < nc; j += kTileWarps)
            for (int e = l; e < ne; e += 32) y[(c0 + j) * ld + e] = tile[j * lt + e];
        __syncthreads();
    }
}

// field_i[c] = RR[c * ld + i], i < nS
__global__ void __launch_bounds__(kTileThreads)
    scatter_rates_kernel(const double* RR, int ld, int n, int nS, const FieldOutPtrs out) {
    extern __shared__ double tile[];  // [kTileCells][nS | 1]
    const int lt = nS | 1;
    const int wid = threadIdx.x >> 5, l = threadIdx.x & 31;
    constexpr int R = kTileCells / kTileWarps;  // rows of a warp
    for (long long c0 = (long long)blockIdx.x * kTileCells; c0 < n; c0 += (long long)gridDim.x * kTileCells) {
        const int nc = n - c0 < kTileCells ? (int)(n - c0) : kTileCells;
        for (int i0 = l; i0 < nS; i0 += 64) {
            double v[R][2];
#pragma unroll
            for (int k = 0; k < R; ++k)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int j = wid + k * kTileWarps, i = i0 + 32 * h;
                    if (j < nc && i < nS) v[k][h] = __ldcs(RR + (c0 + j) * ld + i);
                }
#pragma unroll
            for (int k = 0; k < R; ++k)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int j = wid + k * kTileWarps, i = i0 + 32 * h;
                    if (j < nc && i < nS) tile[j * lt + i] = v[k][h];
                }
        }
        __syncthreads();
        if (l < nc)
            for (int i = wid; i < nS; i += kTileWarps) out.p[i][c0 + l] = tile[l * lt + i];
        __syncthreads();
    }
}

long long tile_grid(int n) {
    const long long tiles = (n + kTileCells - 1) / kTileCells;
    return std::min<long long>(tiles, 32LL * device_sm_count());
}

}  // namespace

int launch_gather_states(int n, int nS, const double* const* Y, const double* T, const double* p, double* y, int ld,
                         void* stream) {
    if (n <= 0) return 0;
    FieldPtrs P{};
    for (int i = 0; i < nS; ++i) P.p[i] = Y[i];
    const size_t smem = (size_t)kTileCells * ((nS + 2) | 1) * sizeof(double);
    const cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(&gather_states_kernel), smem);
    if (e != cudaSuccess) return (int)e;
    gather_states_kernel<<<(unsigned)tile_grid(n), kTileThreads, smem, reinterpret_cast<cudaStream_t>(stream)>>>(
        P, T, p, n, nS, y, ld);
    return (int)cudaGetLastError();
}

int launch_scatter_rates(int n, int nS, const double* RR, int ld, double* const* out, void* stream) {
    if (n <= 0) return 0;
    FieldOutPtrs P{};
    for (int i = 0; i < nS; ++i) P.p[i] = out[i];
    const size_t smem = (size_t)kTileCells * (nS | 1) * sizeof(double);
    const cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(&scatter_rates_kernel), smem);
    if (e != cudaSuccess) return (int)e;
    scatter_rates_kernel<<<(unsigned)tile_grid(n), kTileThreads, smem, reinterpret_cast<cudaStream_t>(stream)>>>(
        RR, ld, n, nS, P);
    return (int)cudaGetLastError();
}

}  // namespace gf
