// The plugin's per-cell side paths on the GPU. The reference computes them on
// the CPU, one cell at a time through OpenFOAM's reactions
// (gpuChemistryModels/gpuChemistryModel/gpuChemistryModel.C):
//   calculate()            :145-186  RR_i = W_i dN_i/dt / V
//   reactionRR(r)          :188-229  omega of reaction r
//   specieReactionRR(r)    :231-298  W_i dN_i/dt / V of reaction r alone
//   tc()                   :366-427  chemical time scale
//   Qdot()                 :429-450  -sum_i hf_i RR_i
// all at the concentrations c_i = rho Y_i / W_i of the thermo's density field
// (:163-166), the rates as gpuReaction::omega computes them
// (gpuReaction.H:472-488: kf Cf - kr Cr at the clipped temperature).
//
// calculate() and tc(): a lane per cell (cell_lanes_kernel). One reaction, few
// cells: one warp per cell with the cell's concentrations, third-body sums and
// per-reaction staging in shared memory: the same device functions as the
// solve (third_body_all, fast_kf, fast_lnKc, fast_C, the dN/dt gather
// stream). Qdot is one thread per cell with the reference's sequential sum.
#include <algorithm>
#include <cfloat>

#include "gf_device.cuh"

namespace gf {

namespace {

constexpr int kFieldCellsMax = 4;  // cells (warps) per CTA of the warp-per-cell form
// Cells from which the lane-per-cell form is taken: from there its 256 CTAs of 32 cells
// keep the SMs busy. 8,191 cells with a warp each / 8,192 with a lane each: 10 species
// 33 / 32 us, 53 159 / 156, 75 273 / 218, 100 656 / 417, 126 883 / 787; 20 and 31 species
// 38 / 45 and 55 / 77, and level with the warps near 12,000.
constexpr int kLaneCells = 8192;

struct FieldLayout {
    WsLayout L;  // only c, Mtb, stage and part are used
    int out;     // dN/dt of every species (one reaction)
    int size;
};

// Mechanisms with thousands of reactions fill a block's shared memory with their
// staging slots, so nothing lies beside them but c, out and the third-body sums:
//  * the 1 for the absent species of a reaction side is out[0], which takes its
//    dN/dt only after the rates;
//  * the 0 for the gather's missing records (behind the last slot) is c[0] and the
//    parts of dN/dt lie on the rest of c, out and the sums: all free by then. There are at
//    most max(nS, 32) parts for a warp, or 2 m for few species.
__host__ __device__ inline FieldLayout field_layout(const DevMech& M) {
    FieldLayout F{};
    int o = 0;
    F.L.stage = o;
    o += M.n_slots;
    F.L.c = o;
    F.L.part = o + 1;
    o += M.nS;
    F.out = o;
    o += M.nS;
    F.L.Mtb = o;
    o += M.n_tb > 0 ? M.n_tb : 1;
    const int parts = M.nS >= 32 ? M.nS : (2 * M.m < 32 ? 2 * M.m : 32);
    F.size = o > F.L.part + parts ? o : F.L.part + parts;
    return F;
}

// Per reaction (compute order, lanes): omega = kf Cf - kr Cr into staging
// slot 0 for the dN/dt gather; with want_tc the lane's shares of tc()'s two
// sums over reactions, sumW and sum of squares (wf = sum_rhs stoich * kf Cf,
// wr = sum_lhs stoich * kr Cr, each counted once in both).
template <class W>
__device__ __forceinline__ void stage_fields(const Grp<32>& g, const DevMech& M, const W& w, const WsLayout& L,
                                             const TCache& tc, bool want_tc, double* sumW, double* sumW2) {
    double sW = 0.0, sW2 = 0.0;
    for (int q = g.lane; q < M.nR; q += 32) {
        const RxnF R = load_fast(M, q);
        const LnK a = load_lnK(M, q, tc.T);
        double Ak;
        const double kf = fast_kf(M, q, R, tc, fast_M(M, w, L.Mtb, R, q), &Ak);
        const double kr = R.irr() ? 0.0 : kf * exp(-fast_lnKc(R, a, tc));
        const double omegaf = kf * fast_C(M, w, L.c, R, q, 0);
        const double omegar = kr * fast_C(M, w, L.c, R, q, 1);
        w[L.stage + R.slot] = omegaf - omegar;
        if (want_tc) {
            double wf = 0.0, wr = 0.0;
            const double* st = M.sst + ldg(M.sp_off + q);
            for (int e = 0; e < R.nr(); ++e) wf += ldg(st + R.nl() + e) * omegaf;
            for (int e = 0; e < R.nl(); ++e) wr += ldg(st + e) * omegar;
            sW += wf + wr;
            sW2 += wf * wf + wr * wr;
        }
    }
    *sumW = sW;
    *sumW2 = sW2;
}

__global__ void __launch_bounds__(32 * kFieldCellsMax) cell_fields_kernel(const DevMech M, const FieldArgs a) {
    extern __shared__ double smem[];
    Grp<32> g;
    const FieldLayout F = field_layout(M);
    const int per_cta = blockDim.x >> 5;
    const int warp = threadIdx.x >> 5;
    WsC w{smem + (size_t)warp * F.size};
    const int nS = M.nS;
    for (long long cell = (long long)blockIdx.x * per_cta + warp; cell < a.n_cells;
         cell += (long long)gridDim.x * per_cta) {
        const double* y = a.y + cell * a.ld_y;
        const double rho = a.rho[cell];
        double csum = 0.0;
        for (int i = g.lane; i < nS; i += 32) {
            const double ci = rho * y[i] / ldg(M.W + i);
            w[F.L.c + i] = ci;
            csum += ci;
        }
        if (g.lane == 0) w[F.out] = 1.0;  // c[nS]
        g.sync();
        if (M.n_tb > 0) {
            third_body_all(g, M, w, F.L.c, F.L.Mtb);
            g.sync();
        }
        const double T = y[nS];
        const TCache tcache = make_tcache(fmin(fmax(T, M.Tlow), M.Thigh));
        if (a.reaction >= 0) {
            // reactionRR / specieReactionRR: one reaction, lane 0
            double* rr = a.RR ? a.RR + cell * a.ld_rr : nullptr;
            if (rr)
                for (int i = 1 + g.lane; i < nS; i += 32) w[F.out + i] = 0.0;
            g.sync();
            if (g.lane == 0) {
                const int q = a.reaction_q;
                const RxnF R = load_fast(M, q);
                double Ak;
                const double kf = fast_kf(M, q, R, tcache, fast_M(M, w, F.L.Mtb, R, q), &Ak);
                const double kr = R.irr() ? 0.0 : kf * exp(-fast_lnKc(R, load_lnK(M, q, tcache.T), tcache));
                const double om = kf * fast_C(M, w, F.L.c, R, q, 0) - kr * fast_C(M, w, F.L.c, R, q, 1);
                if (a.omega) a.omega[cell] = om;
                if (rr) {
                    w[F.out] = 0.0;
                    // gpuReaction::dNdtByV (gpuReaction.H:490-508): lhs, then rhs
                    const int b0 = ldg(M.sp_off + q);
                    for (int e = 0; e < R.nl(); ++e) {
                        const int b = b0 + e;
                        w[F.out + ldg(M.sidx + b)] -= ldg(M.sst + b) * om;
                    }
                    for (int e = 0; e < R.nr(); ++e) {
                        const int b = b0 + R.nl() + e;
                        w[F.out + ldg(M.sidx + b)] += ldg(M.sst + b) * om;
                    }
                }
            }
            g.sync();
            if (rr)
                for (int i = g.lane; i < nS; i += 32) rr[i] = w[F.out + i] * ldg(M.W + i);
            g.sync();
            continue;
        }
        double sW, sW2;
        stage_fields(g, M, w, F.L, tcache, a.tc != nullptr, &sW, &sW2);
        g.sync();
        if (a.RR) {
            if (g.lane == 0) w[F.L.stage + M.n_slots] = 0.0;  // c[0]
            g.sync();
            stream_gather(g, M.dst[stream_index(32)], w, F.L.stage, w, F.L.part);
            g.sync();
            const int* part = M.dst_part[stream_index(32)];
            double* rr = a.RR + cell * a.ld_rr;
            for (int i = g.lane; i < nS; i += 32) rr[i] = part_sum(w, F.L.part, part, i) * ldg(M.W + i);
        }
        if (a.tc) {
            const double sumW = g.sum(sW), sumW2 = g.sum(sW2), ctot = g.sum(csum);
            if (g.lane == 0) a.tc[cell] = sumW2 == 0.0 ? DBL_MAX / 10.0 : sumW / sumW2 * ctot;
        }
        g.sync();
    }
}

// calculate() and tc() with a lane per cell: a CTA takes 32 cells, its warps
// share out the reactions, and every lane evaluates a reaction for its own cell,
// so the reaction's data is one broadcast load for 32 cells, no warp mixes rate
// types, and there is no gather. Concentrations and each warp's own dN/dt live in
// shared memory, species by species over the lanes (stride 33: the transposes in
// and out are free of bank conflicts too). Per species the order of the
// reference's sum inside a warp's reactions, then the warps in order. Bound by
// instructions: some 500 per reaction and 32 cells, at twelve warps per SM, where
// a warp per cell took 415 per 32 reactions of one cell and the gather besides.
// 60,000 cells of 53 species: 1028 -> 813 us.
constexpr int kLaneStride = 33;

// A value per species of one lane's cell.
struct WsLane {
    double* p;
    __device__ __forceinline__ double& operator[](int i) const { return p[i * kLaneStride]; }
};

__global__ void __launch_bounds__(128, 4) cell_lanes_kernel(const DevMech M, const FieldArgs a) {
    extern __shared__ double smem[];
    const int nS = M.nS, NW = blockDim.x >> 5;
    const int wid = threadIdx.x >> 5, l = threadIdx.x & 31;
    double* cs = smem;                                              // [nS + 1][33]
    double* dN = smem + (size_t)(nS + 1) * kLaneStride;             // [NW][nS][33]
    double* red = dN + (size_t)NW * nS * kLaneStride;               // [NW][2][32]
    const WsLane c{cs + l}, d{dN + (size_t)wid * nS * kLaneStride + l};
    for (long long c0 = (long long)blockIdx.x * 32; c0 < a.n_cells; c0 += (long long)gridDim.x * 32) {
        const int nc = a.n_cells - c0 < 32 ? (int)(a.n_cells - c0) : 32;
        for (int j = wid; j < 32; j += NW) {
            // lanes past the last cell work on a copy of it
            const long long cell = c0 + min(j, nc - 1);
            const double rho = a.rho[cell];
            const double* y = a.y + cell * a.ld_y;
            for (int i = l; i < nS; i += 32) cs[i * kLaneStride + j] = rho * y[i] / ldg(M.W + i);
        }
        if (wid == 0) c[nS] = 1.0;
        for (int i = 0; i < nS; ++i) d[i] = 0.0;
        const double T = a.y[(c0 + min(l, nc - 1)) * a.ld_y + nS];
        const TCache tc = make_tcache(fmin(fmax(T, M.Tlow), M.Thigh));
        __syncthreads();
        double sW = 0.0, sW2 = 0.0;
        for (int q = wid; q < M.nR; q += NW) {
            const RxnF R = load_fast(M, q);
            const LnK lk = load_lnK(M, q, tc.T);
            double Mc = 0.0;
            int t = (int)((unsigned)R.meta >> kRxnTbShift);
            if (t != 0) {
                if (t == kRxnTbFar) t = ldg(M.tb_row + q) + 1;
                const double* eff = M.eff + (size_t)(t - 1) * nS;
#pragma unroll 8
                for (int i = 0; i < nS; ++i) Mc = fma(ldg(eff + i), c[i], Mc);
            }
            double Ak;
            const double kf = fast_kf(M, q, R, tc, Mc, &Ak);
            const double kr = R.irr() ? 0.0 : kf * exp(-fast_lnKc(R, lk, tc));
            const double of = kf * fast_C(M, c, 0, R, q, 0), orv = kr * fast_C(M, c, 0, R, q, 1);
            const double om = of - orv;
            // dN/dt (gpuReaction.H:490-508): lhs, then rhs
            const int nl = R.nl(), nr = R.nr(), b = ldg(M.sp_off + q);
            double wf = 0.0, wr = 0.0;
            for (int e = 0; e < nl; ++e) {
                const int sp = ldg(M.sidx + b + e);
                const double st = ldg(M.sst + b + e);
                d[sp] = fma(-st, om, d[sp]);
                wr = fma(st, orv, wr);
            }
            for (int e = nl; e < nl + nr; ++e) {
                const int sp = ldg(M.sidx + b + e);
                const double st = ldg(M.sst + b + e);
                d[sp] = fma(st, om, d[sp]);
                wf = fma(st, of, wf);
            }
            // tc()'s two sums over reactions
            sW += wf + wr;
            sW2 += wf * wf + wr * wr;
        }
        red[wid * 64 + l] = sW;
        red[wid * 64 + 32 + l] = sW2;
        __syncthreads();
        if (a.RR)
            for (int j = wid; j < nc; j += NW)
                for (int i = l; i < nS; i += 32) {
                    double v = 0.0;
                    for (int k = 0; k < NW; ++k) v += dN[((size_t)k * nS + i) * kLaneStride + j];
                    a.RR[(c0 + j) * a.ld_rr + i] = v * ldg(M.W + i);
                }
        if (a.tc && wid == 0 && l < nc) {
            double w1 = 0.0, w2 = 0.0, ctot = 0.0;
            for (int k = 0; k < NW; ++k) {
                w1 += red[k * 64 + l];
                w2 += red[k * 64 + 32 + l];
            }
            for (int i = 0; i < nS; ++i) ctot += c[i];
            a.tc[c0 + l] = w2 == 0.0 ? DBL_MAX / 10.0 : w1 / w2 * ctot;
        }
        __syncthreads();
    }
}

// Qdot = 0 - hf_0 RR_0 - hf_1 RR_1 - ... in species order, each product
// rounded before the subtraction (no contraction), as the reference's loop: a
// thread per cell, after the warp has brought the rows of its 32 cells to
// shared memory with coalesced loads, kQdotRows rows in flight. Bound by HBM.
constexpr int kQdotRows = 8;
__global__ void __launch_bounds__(128) qdot_kernel(const DevMech M, int n, const double* RR, int ld_rr, double* qdot) {
    extern __shared__ double smem[];
    const int nS = M.nS, lt = nS | 1, l = threadIdx.x & 31;
    const int warps = blockDim.x >> 5;
    double* tile = smem + (size_t)(threadIdx.x >> 5) * 32 * lt;
    for (long long c0 = ((long long)blockIdx.x * warps + (threadIdx.x >> 5)) * 32; c0 < n;
         c0 += (long long)gridDim.x * warps * 32) {
        const int nc = n - c0 < 32 ? (int)(n - c0) : 32;
        for (int j0 = 0; j0 < nc; j0 += kQdotRows)
            for (int i0 = l; i0 < nS; i0 += 64) {
                double v[kQdotRows][2];
#pragma unroll
                for (int k = 0; k < kQdotRows; ++k)
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        if (j0 + k < nc && i0 + 32 * h < nS) v[k][h] = __ldcs(RR + (c0 + j0 + k) * ld_rr + i0 + 32 * h);
#pragma unroll
                for (int k = 0; k < kQdotRows; ++k)
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        if (j0 + k < nc && i0 + 32 * h < nS) tile[(j0 + k) * lt + i0 + 32 * h] = v[k][h];
            }
        __syncwarp();
        if (l < nc) {
            double q = 0.0;
            for (int i = 0; i < nS; ++i) q = __dsub_rn(q, __dmul_rn(ldg(M.hf + i), tile[l * lt + i]));
            qdot[c0 + l] = q;
        }
        __syncwarp();
    }
}

}  // namespace

int launch_cell_fields(const DevMech& M, const FieldArgs& a, void* stream) {
    if (a.n_cells <= 0) return 0;
    // all reactions: a lane per cell, with as many warps as leave room for two
    // CTAs per SM, while the cells fill the machine and there are at least two of
    // them; a warp per cell for one reaction, for few cells and for the species
    // (145 and more) that leave one. 16,384 cells, lane / warp per cell: 140 species
    // 1.93 / 2.06 ms; 150 species, with one warp, 4.14 / 2.18 ms.
    if (a.reaction < 0 && a.n_cells >= kLaneCells) {
        int warps = 4;
        auto bytes = [&](int w) {
            return ((size_t)(M.nS + 1) * kLaneStride + (size_t)w * (M.nS * kLaneStride + 64)) * sizeof(double);
        };
        while (warps > 1 && bytes(warps) > 113 * 1024) --warps;
        if (warps > 1) {
            const size_t smem = bytes(warps);
            const void* fn = reinterpret_cast<const void*>(&cell_lanes_kernel);
            cudaError_t e = allow_dynamic_smem(fn, smem);
            if (e != cudaSuccess) return (int)e;
            int per_sm = 0;
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cell_lanes_kernel, 32 * warps, smem);
            if (e != cudaSuccess) return (int)e;
            const long long grid =
                std::min<long long>((a.n_cells + 31) / 32, (long long)std::max(per_sm, 1) * device_sm_count());
            cell_lanes_kernel<<<(unsigned)grid, 32 * warps, smem, reinterpret_cast<cudaStream_t>(stream)>>>(M, a);
            return (int)cudaGetLastError();
        }
    }
    const FieldLayout F = field_layout(M);
    const size_t per_cell = (size_t)F.size * sizeof(double);
    int dev = 0, max_smem = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    int cells = kFieldCellsMax;
    while (cells > 1 && per_cell * cells > (size_t)max_smem) --cells;
    if (per_cell * cells > (size_t)max_smem) return (int)cudaErrorInvalidValue;
    const size_t smem = per_cell * cells;
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(&cell_fields_kernel), smem);
    if (e != cudaSuccess) return (int)e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cell_fields_kernel, 32 * cells, smem);
    if (e != cudaSuccess) return (int)e;
    const long long want = (a.n_cells + cells - 1) / cells;
    const long long grid = std::min<long long>(want, (long long)std::max(per_sm, 1) * device_sm_count());
    cell_fields_kernel<<<(unsigned)grid, 32 * cells, smem, reinterpret_cast<cudaStream_t>(stream)>>>(M, a);
    return (int)cudaGetLastError();
}

int launch_qdot(const DevMech& M, int n, const double* RR, int ld_rr, double* qdot, void* stream) {
    if (n <= 0) return 0;
    // a tile per warp: four warps, or as many as fit
    const size_t per_warp = (size_t)32 * (M.nS | 1) * sizeof(double);
    int warps = 4;
    while (warps > 1 && per_warp * warps > 100 * 1024) --warps;
    const size_t smem = per_warp * warps;
    const cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(&qdot_kernel), smem);
    if (e != cudaSuccess) return (int)e;
    const long long grid = std::min<long long>((n + 32LL * warps - 1) / (32LL * warps), 8LL * device_sm_count());
    qdot_kernel<<<(unsigned)grid, 32 * warps, smem, reinterpret_cast<cudaStream_t>(stream)>>>(M, n, RR, ld_rr, qdot);
    return (int)cudaGetLastError();
}

}  // namespace gf
