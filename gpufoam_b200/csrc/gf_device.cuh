// Device code of the per-cell chemistry path (sm_100a, FP64 on CUDA cores, the
// factorisation's trailing updates on the FP64 matrix units).
//
// One templated code path serves every launch form: a "group" of G threads
// (G = 1, 2, 4, 8, 16, 32, aligned inside a warp, or 64, 96, 128, 256, a whole CTA)
// integrates one cell. G = 1 is the reference's one-thread-per-cell model; from
// G = 32 on the cell's Jacobian/LU is usually held in shared memory. Loops over species, reactions,
// rows and columns are strided over the group's lanes; everything that decides
// control flow (error norm, step size, status) is group-uniform.
//
// The arithmetic follows gpuFoam's device code (paths below are relative to
// gpu_chemistry/src/ of the reference): gpuThermo/gpuThermo.H,
// gpuReaction/*.H, gpuOde/gpuODESystem.H, ludecompose.H, gpuRosenbrock*.H,
// gpuAdaptiveSolver.H, gpuODESolverBase.H and
// gpuKernelEvaluator/singleCellSolver.H. Where the order of a floating-point
// reduction is changed for parallelism it is noted; those change results at
// the ulp level only.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "gf_internal.h"

namespace gf {

// gpu_utils/common/gpu_constants.H:13-82
constexpr double kRR = 6.02214e+26 * 1.38065e-23;
constexpr double kPstd = 1e5;
constexpr double kLnPstdR = 2.4871731053390858;  // ln(kPstd / kRR)
constexpr double kVSmall = 2.2250738585072014e-308;  // numeric_limits<double>::min()
constexpr double kSmall = 2.220446049250313e-16;     // numeric_limits<double>::epsilon()
constexpr double kVGreat = 1.7976931348623157e+308 / 10.0;
constexpr int kMaxRejects = 100000;  // rejected attempts within one substep

// ------------------------------------------------------- phase timers
// Built only with -DGF_PHASE_TIMERS (a profiling variant of the library):
// lane 0 of each group accumulates clock64() cycles per phase of the solve.
#ifdef GF_PHASE_TIMERS
// one accumulator per translation unit (each has its own device module)
static __device__ unsigned long long g_phase_cycles[20];
// adds this translation unit's accumulators to out[20], optionally clearing them
static inline int phase_cycles_local(unsigned long long* out, int reset) {
    unsigned long long v[20];
    cudaMemcpyFromSymbol(v, g_phase_cycles, sizeof(v));
    for (int i = 0; i < 20; ++i) out[i] += v[i];
    if (reset) {
        unsigned long long z[20] = {};
        cudaMemcpyToSymbol(g_phase_cycles, z, sizeof(z));
    }
    return (int)cudaGetLastError();
}
#define GF_PH_BEGIN(g) \
    (g).sync();        \
    const long long _gf_ph0 = clock64();
#define GF_PH_END(g, k) \
    (g).sync();         \
    if ((g).lane == 0) atomicAdd(&g_phase_cycles[k], (unsigned long long)(clock64() - _gf_ph0));
#else
#define GF_PH_BEGIN(g)
#define GF_PH_END(g, k)
#endif
enum { PH_MIX = 0, PH_OMEGA, PH_GATHER_RHS, PH_JPARAMS, PH_JROWS, PH_TROW, PH_SHIFT, PH_LU, PH_SOLVE,
       PH_ADJ_RXN, PH_ATTEMPT, PH_ADJ_RECOMPUTE, PH_ADJ_TSOLVE, PH_ADJ_VJP, PH_ADJ_JTERM, PH_LU_PANEL, PH_LU_U12,
       PH_LU_TRAIL, PH_LU_PERM };

// ---------------------------------------------------------------- groups

// Cross-warp reduction buffers of a multi-warp group (one group per CTA): two,
// used in turn, so that a reduction needs one barrier (a warp writes a buffer
// again only after the barrier of the reduction in between, which every warp
// reaches after reading it).
constexpr int kRedMax = 3;  // values reduced together
template <int NW>
__device__ __forceinline__ double* grp_red_buf() {
    __shared__ double buf[2 * NW * kRedMax];
    return buf;
}

// G <= 32: G aligned lanes of one warp, several groups per warp/CTA.
// G = 64, 96, 128, 256: the whole CTA (one cell per CTA); barriers are
// __syncthreads and reductions go through a small shared buffer, in a fixed
// warp order (deterministic).
template <int G>
struct Grp {
    static constexpr int W = G > 32 ? G / 32 : 1;  // warps in the group
    int lane;
    unsigned mask;
    mutable int ph = 0;  // which reduction buffer is next (the same in every thread)
    __device__ __forceinline__ int warp() const { return G > 32 ? lane >> 5 : 0; }  // warp in the group
    __device__ __forceinline__ Grp() {
        const int wl = threadIdx.x & 31;
        if constexpr (G >= 32) {
            lane = G > 32 ? (int)threadIdx.x : wl;
            mask = 0xffffffffu;
        } else {
            lane = wl & (G - 1);
            mask = ((1u << G) - 1u) << (wl & ~(G - 1));
        }
    }
    __device__ __forceinline__ void sync() const {
        if (G > 32)
            __syncthreads();
        else if (G > 1)
            __syncwarp(mask);
    }
    __device__ __forceinline__ long long bcast_ll(long long v, int src) const {
        if (G == 1) return v;
        if constexpr (G > 32) {
            long long* b = reinterpret_cast<long long*>(grp_red_buf<W>()) + (ph ? W * kRedMax : 0);
            ph ^= 1;
            if (lane == src) b[0] = v;
            __syncthreads();
            return b[0];
        }
        return __shfl_sync(mask, v, src, G);
    }
    // N sums (or maxima) over the group at once, the same in every thread:
    // a shuffle tree inside a warp, then the warps in order (deterministic)
    template <int N, bool MAX>
    __device__ __forceinline__ void reduce(double (&v)[N]) const {
        static_assert(N <= kRedMax, "reduction buffer");
        constexpr int L = G > 32 ? 32 : G;
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) {
#pragma unroll
            for (int n = 0; n < N; ++n) {
                const double x = __shfl_xor_sync(mask, v[n], o, L);
                v[n] = MAX ? fmax(v[n], x) : v[n] + x;
            }
        }
        if constexpr (G > 32) {
            double* b = grp_red_buf<W>() + (ph ? W * kRedMax : 0);
            ph ^= 1;
            if ((threadIdx.x & 31) == 0) {
#pragma unroll
                for (int n = 0; n < N; ++n) b[(lane >> 5) * kRedMax + n] = v[n];
            }
            __syncthreads();
#pragma unroll
            for (int n = 0; n < N; ++n) {
                v[n] = b[n];
#pragma unroll
                for (int k = 1; k < W; ++k) {
                    const double x = b[k * kRedMax + n];
                    v[n] = MAX ? fmax(v[n], x) : v[n] + x;
                }
            }
        }
    }
    __device__ __forceinline__ double sum(double v) const {
        double x[1] = {v};
        reduce<1, false>(x);
        return x[0];
    }
    template <int N>
    __device__ __forceinline__ void sums(double (&v)[N]) const {
        reduce<N, false>(v);
    }
    // max with fmax semantics: a NaN operand is ignored (normaliseError.H:22)
    __device__ __forceinline__ double fmax_(double v) const {
        double x[1] = {v};
        reduce<1, true>(x);
        return x[0];
    }
    __device__ __forceinline__ int any(int p) const {
        if (G == 1) return p;
        if (G > 32) return __syncthreads_or(p) != 0;
        return (__ballot_sync(mask, p) & mask) != 0;
    }
};

// ------------------------------------------------------------- workspace

// Contiguous per-cell workspace (shared memory, or a per-cell block in HBM).
struct WsC {
    double* p;
    __device__ __forceinline__ double& operator[](int i) const { return p[i]; }
    __device__ __forceinline__ int& ip(int i) const { return *reinterpret_cast<int*>(p + i); }
    // the element `bytes` behind element i of a contiguous one
    __device__ __forceinline__ double at(int i, int bytes) const {
        return *reinterpret_cast<const double*>(reinterpret_cast<const char*>(p + i) + bytes);
    }
};
// Interleaved workspace: element i of a cell at p[i * s] (p already offset by
// the cell's slot), so that consecutive threads touch consecutive addresses.
struct WsS {
    double* p;
    long long s;
    __device__ __forceinline__ double& operator[](int i) const { return p[(long long)i * s]; }
    __device__ __forceinline__ int& ip(int i) const { return *reinterpret_cast<int*>(p + (long long)i * s); }
    __device__ __forceinline__ double at(int i, int bytes) const { return p[(long long)(i + (bytes >> 3)) * s]; }
};

template <class T>
__device__ __forceinline__ T ldg(const T* p) {
    return __ldg(p);
}


// ------------------------------------------------------------ thermo

// JANAF coefficient set of species i at T (gpuThermo.H:29-32)
__device__ __forceinline__ int coef_branch(double T, double Tcommon) { return T < Tcommon ? 0 : 1; }

struct Poly7 {
    double a0, a1, a2, a3, a4, a5, a6;
};

__device__ __forceinline__ Poly7 species_coeffs(const DevMech& M, int i, double T) {
    const int b = coef_branch(T, ldg(M.Tcommon + i));
    const double* c = M.coef + (size_t)b * 7 * M.nS + i;
    Poly7 a;
    a.a0 = ldg(c);
    a.a1 = ldg(c + M.nS);
    a.a2 = ldg(c + 2 * M.nS);
    a.a3 = ldg(c + 3 * M.nS);
    a.a4 = ldg(c + 4 * M.nS);
    a.a5 = ldg(c + 5 * M.nS);
    a.a6 = ldg(c + 6 * M.nS);
    return a;
}

// A reaction's packed data (RxnHead) and the species entries of both sides,
// requested with independent 16-byte loads before any of them is used.
struct Rxn {
    int type, irr, slot, tb_row, nl, nr, sp_off, nm_small;
    double lnA0, beta0, Ta0, sA0, Tcommon, Y, nm;
    int idx[2][kSideInline], iexp[2][kSideInline];
    double sexp[2][kSideInline];
};

__device__ __forceinline__ void load_rxn(const DevMech& M, int q, Rxn& R) {
    const int4* h = reinterpret_cast<const int4*>(M.rxh + q);
    const int4 h0 = __ldg(h), h1 = __ldg(h + 1);
    const double2* hd = reinterpret_cast<const double2*>(M.rxh + q) + 2;
    const double2 d0 = __ldg(hd), d1 = __ldg(hd + 1);
    const int4* sp = reinterpret_cast<const int4*>(M.rxs + (size_t)q * 2 * kSideInline);
    int4 v[2 * kSideInline];
#pragma unroll
    for (int e = 0; e < 2 * kSideInline; ++e) v[e] = __ldg(sp + e);
    R.type = h0.x;
    R.irr = h0.y;
    R.slot = h0.z;
    R.tb_row = h0.w;
    R.nl = h1.x;
    R.nr = h1.y;
    R.sp_off = h1.z;
    R.nm_small = h1.w;
    R.lnA0 = d0.x;
    R.beta0 = d0.y;
    R.Ta0 = d1.x;
    R.sA0 = d1.y;
    const double2 d2 = __ldg(hd + 2);
    R.Tcommon = d2.x;
    R.Y = d2.y;
    R.nm = __ldg(reinterpret_cast<const double*>(hd + 3));
#pragma unroll
    for (int e = 0; e < 2 * kSideInline; ++e) {
        R.idx[e / kSideInline][e % kSideInline] = v[e].x;
        R.iexp[e / kSideInline][e % kSideInline] = v[e].y;
        R.sexp[e / kSideInline][e % kSideInline] = __hiloint2double(v[e].w, v[e].z);
    }
}

__device__ __forceinline__ Poly7 reaction_coeffs_at(const DevMech& M, int r, double T, double Tcommon) {
    const int b = coef_branch(T, Tcommon);
    const double* c = M.rcoef + (size_t)b * 7 * M.nR + r;
    Poly7 a;
    a.a0 = ldg(c);
    a.a1 = ldg(c + M.nR);
    a.a2 = ldg(c + 2 * M.nR);
    a.a3 = ldg(c + 3 * M.nR);
    a.a4 = ldg(c + 4 * M.nR);
    a.a5 = ldg(c + 5 * M.nR);
    a.a6 = ldg(c + 6 * M.nR);
    return a;
}

// gpuThermo.H:177-184 (the perfect-gas Cp term is 0)
__device__ __forceinline__ double th_Cp(const Poly7& a, double T) {
    return ((((a.a4 * T + a.a3) * T + a.a2) * T + a.a1) * T + a.a0);
}
// gpuThermo.H:333-338
__device__ __forceinline__ double th_dCpdT(const Poly7& a, double T) {
    return (((4.0 * a.a4 * T + 3.0 * a.a3) * T + 2.0 * a.a2) * T + a.a1);
}
// gpuThermo.H:287-299
__device__ __forceinline__ double th_Gstd(const Poly7& a, double T, double logT) {
    return ((a.a0 * (1.0 - logT) - (((a.a4 / 20.0 * T + a.a3 / 12.0) * T + a.a2 / 6.0) * T + a.a1 / 2.0) * T - a.a6) *
                T +
            a.a5);
}
// gpuThermo.H:261-271 at p = pStd (the -R ln(p/pStd) term is zero there)
__device__ __forceinline__ double th_S_pstd(const Poly7& a, double T, double logT) {
    return ((((a.a4 / 4.0 * T + a.a3 / 3.0) * T + a.a2 / 2.0) * T + a.a1) * T + a.a0 * logT + a.a6);
}

// ------------------------------------------------------------ reactions
//
// Rate constants are evaluated in log space: k = sign(A) exp(ln|A| + beta ln T
// - Ta / T) (gpuArrheniusReactionRate.H:16-26 computes A * pow(T, beta) *
// exp(-Ta / T)), Kc = exp(lnK + nm ln(pStd / (RR T))) (gpuThermo.H:80-113,
// 139-169 compute exp and pow), the Troe function with exp/log instead of
// pow(10, .)/log10. The results differ from the reference at the level of a
// few ulp of the exponent argument (a relative 1e-14 for |arg| ~ 50), far
// inside the 1e-12 rate tolerance, and save the double-precision pow calls
// and divisions that dominate the reaction loops.

// temperature-dependent per-call quantities
struct TCache {
    double T, invT, logT, lx;  // lx = ln(pStd / (RR T))
};

__device__ __forceinline__ TCache make_tcache(double T) {
    TCache t;
    t.T = T;
    t.invT = 1.0 / T;
    t.logT = log(T);
    t.lx = kLnPstdR - t.logT;
    return t;
}

// gpuSpecieExponent.H:21-36
__device__ __forceinline__ double integer_pow(double x, int e) {
    if (e == 0) return 1;
    if (e == 1) return x;
    if (e == 2) return x * x;
    double xx = e > 0 ? x : 1 / x;
    double y = 1;
    for (int i = e; i != 0; i /= 2) {
        if (i % 2) y *= xx;
        xx *= xx;
    }
    return y;
}
// x^e for a non-integer exponent (rare: most mechanisms have integer
// exponents only), out of line: the many call sites share one copy of the
// math library's pow, which keeps the solve's instruction footprint smaller.
static __device__ __noinline__ double real_pow(double x, double e) { return pow(x, e); }
// gpuSpecieExponent.H:103-110
__device__ __forceinline__ double specie_pow(double x, int iexp, double sexp) {
    return iexp != kNoIntExp ? integer_pow(x, iexp) : real_pow(x, sexp);
}
// speciePow(c, e - 1) (gpuReaction.H:418-420 with gpuSpecieExponent::operator-)
__device__ __forceinline__ double specie_pow_m1(double x, int iexp, double sexp) {
    return iexp != kNoIntExp ? integer_pow(x, iexp - 1) : real_pow(x, sexp + (-1.0));
}

// ln|kInf| of a fall-off rate and dln(kInf)/dT = (beta + Ta/T)/T
__device__ __forceinline__ double arr_ln1(const DevMech& M, int q, const TCache& tc) {
    return fma(ldg(M.beta1 + q), tc.logT, ldg(M.lnA1 + q)) - ldg(M.Ta1 + q) * tc.invT;
}
__device__ __forceinline__ double arr_dlnkdT1(const DevMech& M, int q, const TCache& tc) {
    return (ldg(M.beta1 + q) + ldg(M.Ta1 + q) * tc.invT) * tc.invT;
}

// The solve's view of a reaction: its compact record (RxnFast).
struct RxnF {
    int meta, slot;
    unsigned lhs, rhs;
    double lnA0, beta0, Ta0, nm;
    __device__ __forceinline__ int type() const { return meta & kRxnType; }
    __device__ __forceinline__ bool irr() const { return meta & kRxnIrr; }
    __device__ __forceinline__ int nl() const { return (meta >> kRxnNlShift) & 15; }
    __device__ __forceinline__ int nr() const { return (meta >> kRxnNrShift) & 15; }
    __device__ __forceinline__ unsigned side(int sd) const { return sd ? rhs : lhs; }
    __device__ __forceinline__ bool sq(int sd, int e) const {
        return (meta >> (kRxnSqShift + kFastSide * sd + e)) & 1;
    }
    // sign(A): A = 0 gives k = 0 exactly
    __device__ __forceinline__ double sign() const {
        const int b = (meta >> kRxnSignShift) & 3;
        return b == 0 ? 1.0 : (b == 1 ? -1.0 : 0.0);
    }
};

__device__ __forceinline__ RxnF load_fast(const DevMech& M, int q) {
    const int4* h = reinterpret_cast<const int4*>(M.rxf + q);
    const int4 h0 = __ldg(h);
    const double2* hd = reinterpret_cast<const double2*>(h) + 1;
    const double2 d0 = __ldg(hd), d1 = __ldg(hd + 1);
    return RxnF{h0.x, h0.y, (unsigned)h0.z, (unsigned)h0.w, d0.x, d0.y, d1.x, d1.y};
}

// The reaction's third-body concentration (third_body_all), 0 for plain Arrhenius rates.
template <class W>
__device__ __forceinline__ double fast_M(const DevMech& M, const W& w, int m_off, const RxnF& R, int q) {
    int t = (int)((unsigned)R.meta >> kRxnTbShift);
    if (t == 0) return 0.0;
    if (t == kRxnTbFar) t = ldg(M.tb_row + q) + 1;
    return w[m_off + t - 1];
}

// The seven coefficients of ln K at this temperature's branch (DevMech::lnk).
struct LnK {
    double b0, b1, b2, b3, b4, b5, b6;
};
__device__ __forceinline__ LnK load_lnK(const DevMech& M, int q, double T) {
    // one Tcommon for every reaction (the usual case): no load to wait for
    const double Tc = M.Tc_all == M.Tc_all ? M.Tc_all : ldg(M.rTcommon + q);
    const double* c = M.lnk + (size_t)coef_branch(T, Tc) * 7 * M.nR + q;
    LnK a;
    a.b0 = ldg(c);
    a.b1 = ldg(c + M.nR);
    a.b2 = ldg(c + 2 * M.nR);
    a.b3 = ldg(c + 3 * M.nR);
    a.b4 = ldg(c + 4 * M.nR);
    a.b5 = ldg(c + 5 * M.nR);
    a.b6 = ldg(c + 6 * M.nR);
    return a;
}
// ln Kc with K capped as K() caps it (gpuThermo.H:80-113, 139-169): -Y G / (R T)
// with Y, R and the polynomial's divisors folded into the coefficients
__device__ __forceinline__ double fast_lnKc(const RxnF& R, const LnK& a, const TCache& tc) {
    const double T = tc.T;
    const double poly = fma(fma(fma(a.b4, T, a.b3), T, a.b2), T, a.b1);
    double lnK = fma(a.b0, 1.0 - tc.logT, -a.b6);
    lnK = fma(-poly, T, lnK);
    lnK = fma(a.b5, tc.invT, lnK);
    lnK = lnK < 600 ? lnK : 0.5 * log(kVGreat);
    return fma(R.nm, tc.lx, lnK);
}
// d ln Kc / dT (gpuThermo.H:160-166: (S + G/T) Y / (R T) - nm/T). S + G/T is H/T,
// whose polynomial has no logarithm and no cancellation between the two:
// -(b0 + 2 b1/2 T + ...) with G's divisors 2, 6, 12, 20 turned into H's 2, 3, 4, 5
__device__ __forceinline__ double fast_dlnKcdT(const RxnF& R, const LnK& a, const TCache& tc) {
    const double T = tc.T;
    double h = fma(4.0 * a.b4, T, 3.0 * a.b3);
    h = fma(h, T, 2.0 * a.b2);
    h = fma(h, T, a.b1);
    h = fma(h, T, a.b0);
    h = fma(a.b5, tc.invT, h);
    return -(h + R.nm) * tc.invT;
}

// Third-body concentrations M_t = sum_i eff_ti c_i of every third-body and
// fall-off reaction (gpuThirdBodyEfficiencies.H:28-35), written to Mtb[t]:
// threads over reactions, the even and the odd species each in order, the
// efficiencies species by species so that a warp's loads are consecutive. A
// warp per reaction with a shuffle tree took 4.8k warp instructions for 75
// reactions of 53 species; this takes 0.6k.
template <int G, class W>
__device__ __forceinline__ void third_body_all(const Grp<G>& g, const DevMech& M, const W& w, int c_off, int m_off) {
    const int n = M.n_tb;
    for (int t = g.lane; t < n; t += G) {
        const double* e = M.effT + t;
        double s0 = 0.0, s1 = 0.0;
        int i = 0;
        constexpr int U = 16;  // loads in flight
        for (; i + U <= M.nS; i += U) {
            double v[U];
#pragma unroll
            for (int k = 0; k < U; ++k) v[k] = ldg(e + (size_t)(i + k) * n);
#pragma unroll
            for (int k = 0; k < U; k += 2) {
                s0 = fma(v[k], w[c_off + i + k], s0);
                s1 = fma(v[k + 1], w[c_off + i + k + 1], s1);
            }
        }
#pragma unroll 4
        for (; i < M.nS; ++i) {
            const double t = s0;
            s0 = s1;
            s1 = fma(ldg(e + (size_t)i * n), w[c_off + i], t);
        }
        w[m_off + t] = s0 + s1;
    }
}

// Troe F (gpuTroeFallOffFunction.H:27-47); troe[] holds alpha, 1/T***, 1/T*, T**
__device__ __forceinline__ double troe_F(const DevMech& M, int q, const TCache& tc, double Pr) {
    const double* tp = M.troe + 4 * q;
    const double alpha = ldg(tp), iTsss = ldg(tp + 1), iTs = ldg(tp + 2), Tss = ldg(tp + 3);
    constexpr double kInvLn10 = 0.43429448190325182765;
    constexpr double kLn10 = 2.30258509299404568402;
    const double logPr = log(fmax(Pr, kSmall)) * kInvLn10;
    const double Fcent = (1.0 - alpha) * exp(-tc.T * iTsss) + alpha * exp(-tc.T * iTs) + exp(-Tss * tc.invT);
    const double logFcent = log(fmax(Fcent, kSmall)) * kInvLn10;
    const double c = -0.4 - 0.67 * logFcent;
    const double n = 0.75 - 1.27 * logFcent;
    const double x1 = n - 0.14 * (logPr + c);
    const double x2 = (logPr + c) / x1;
    const double x3 = 1.0 + x2 * x2;
    const double x4 = logFcent / x3;
    return exp(x4 * kLn10);
}

// Forward rate constant kf (operator(), gpuReactionRate.H:164-173) and, for
// third-body rates, its pure Arrhenius part Ak: plain and third-body Arrhenius
// (gpuArrheniusReactionRate.H, gpuThirdBodyArrheniusReactionRate.H), Lindemann
// and Troe fall-off (gpuFallOffReactionRate.H); the first exponential is one
// code site for all of them. Mc: the reaction's third-body concentration.
__device__ __forceinline__ double fast_kf(const DevMech& M, int q, const RxnF& R, const TCache& tc, double Mc,
                                          double* Ak_out) {
    const int type = R.type();
    const double l0 = fma(R.beta0, tc.logT, R.lnA0) - R.Ta0 * tc.invT;
    const bool falloff = type >= GF_RATE_LINDEMANN_FALLOFF;
    double l = l0, s = R.sign();
    if (falloff) {
        l = arr_ln1(M, q, tc);
        s = ldg(M.sA1 + q);
    }
    double k = s * exp(l);  // k, or the fall-off kInf
    *Ak_out = k;
    if (type == GF_RATE_THIRD_BODY_ARRHENIUS) k *= Mc;
    if (falloff) {
        // Pr = k0 / kInf * M, k = kInf Pr / (1 + Pr) F
        const double Pr = (R.sign() * s) * exp(l0 - l) * Mc;
        const double F = type == GF_RATE_TROE_FALLOFF ? troe_F(M, q, tc, Pr) : 1.0;
        k *= (Pr / (1.0 + Pr)) * F;
    }
    return k;
}

// Concentration products of reactions outside the compact record's terms (a
// side of more than kFastSide species, an exponent other than 1 and 2), out of
// line: rare, and their code would sit in the middle of every reaction loop.
// C = prod c^e in the reference's order (calcCf / calcCr, gpuReaction.H:372-386).
template <class W>
__device__ __noinline__ double general_C(const int* idx, const int* iexp, const double* sexp, int n, W w, int c_off) {
    double C = 1.0;
    for (int e = 0; e < n; ++e) C *= specie_pow(w[c_off + ldg(idx + e)], ldg(iexp + e), ldg(sexp + e));
    return C;
}
// C, and kmul dC/dc_j to out + j (calcdCfdcj / calcdCrdcj, gpuReaction.H:388-470).
template <class W>
__device__ __noinline__ double general_products(const int* idx, const int* iexp, const double* sexp, int n, W w,
                                                int c_off, double kmul, int out) {
    double C = 1.0;
    for (int e = 0; e < n; ++e) C *= specie_pow(w[c_off + ldg(idx + e)], ldg(iexp + e), ldg(sexp + e));
    for (int j = 0; j < n; ++j) {
        double d = 1;
        for (int i = 0; i < n; ++i) {
            const double x = w[c_off + ldg(idx + i)];
            const int ie = ldg(iexp + i);
            const double se = ldg(sexp + i);
            d *= (i == j) ? se * specie_pow_m1(x, ie, se) : specie_pow(x, ie, se);
        }
        w[out + j] = d * kmul;
    }
    return C;
}

// C = prod c^e of one side (0: lhs, 1: rhs): without a branch for the usual
// reaction (absent species read the 1 kept behind the concentrations).
template <class W>
__device__ __forceinline__ double fast_C(const DevMech& M, const W& w, int c_off, const RxnF& R, int q, int sd) {
    if (R.meta & kRxnGeneral) {
        const int b = ldg(M.sp_off + q) + (sd ? R.nl() : 0);
        return general_C(M.sidx + b, M.siexp + b, M.sexp + b, sd ? R.nr() : R.nl(), w, c_off);
    }
    double C = 1.0;
#pragma unroll
    for (int e = 0; e < kFastSide; ++e) {
        const double x = w[c_off + ((R.side(sd) >> (10 * e)) & 1023)];
        C *= R.sq(sd, e) ? x * x : x;
    }
    return C;
}
// C, and kmul dC/dc_j of the side's species to out + j.
template <class W>
__device__ __forceinline__ double fast_products(const DevMech& M, const W& w, int c_off, const RxnF& R, int q, int sd,
                                                double kmul, int out) {
    const int n = sd ? R.nr() : R.nl();
    if (R.meta & kRxnGeneral) {
        const int b = ldg(M.sp_off + q) + (sd ? R.nl() : 0);
        return general_products(M.sidx + b, M.siexp + b, M.sexp + b, n, w, c_off, kmul, out);
    }
    double pw[kFastSide], dm[kFastSide];
#pragma unroll
    for (int e = 0; e < kFastSide; ++e) {
        const double x = w[c_off + ((R.side(sd) >> (10 * e)) & 1023)];
        const bool sq = R.sq(sd, e);
        pw[e] = sq ? x * x : x;
        dm[e] = sq ? 2.0 * x : 1.0;
    }
    static_assert(kFastSide == 3, "the products below");
    w[out] = dm[0] * pw[1] * pw[2] * kmul;
    if (n > 1) w[out + 1] = pw[0] * dm[1] * pw[2] * kmul;
    if (n > 2) w[out + 2] = pw[0] * pw[1] * dm[2] * kmul;
    return pw[0] * pw[1] * pw[2];
}

// ------------------------------------------------------------- layout

// Per-cell workspace layout. The solve kernels (sweep = false) keep Cp, which only
// the Jacobian reads, in k2 and the parts of dN/dt in k3 and k4 (stage vectors, not
// yet written while f or the Jacobian is formed; v and rhoM/W are kept by the sweep
// alone, which has room for both), and have one pivot region: the solves
// follow either the pivots or their permutation (solve_layout places the other
// in k1, free until the first stage). The adjoint's sweep (sweep = true) needs
// both after the stages and gets separate regions. pad: the doubles given to a
// vector (m or more), or 0: as many as it needs.
__host__ __device__ inline WsLayout make_layout(int nS, int nR, int n_slots, int n_tb, bool sweep = false,
                                                int pad = 0) {
    WsLayout L;
    const int m = nS + 1, v = pad ? pad : m;
    L.ld = m | 1;
    L.ks = v;
    int o = 0;
    L.J = 0;
    if (!pad) o += m * L.ld;
    L.y0 = o; o += v;
    L.yt = o; o += v;
    L.dydx0 = o; o += v;
    L.dydx = o; o += v;
    L.dfdx = o; o += v;
    L.k1 = o; o += v;
    L.k2 = o; o += v;
    L.k3 = o; o += v;
    L.k4 = o; o += v;
    L.vv = o; o += v;
    L.piv = o; o += v;
    if (sweep) {
        L.perm = o; o += v;
    } else {
        L.perm = L.piv;
    }
    L.c = o; o += v;  // nS, and a 1 for the absent species of a reaction side
    L.Ha = o; o += pad ? v : nS;
    if (sweep) {
        L.Cp = o; o += pad ? v : nS;
        L.rhoMbyW = o; o += pad ? v : nS;
        L.vj = o; o += pad ? v : nS;
    } else {
        L.Cp = L.k2;
        L.vj = L.k3;
        L.rhoMbyW = L.k4;
    }
    if (pad) {  // behind the vectors, whose places are then known
        L.J = o; o += m * L.ld;
    }
    L.stage = o; o += n_slots + 1;  // and a 0 for the gathers' missing records
    L.part = L.k3;                  // k3, k4: no stage has written them when f is assembled
    L.Mtb = o; o += (n_tb > 0 ? n_tb : 1);
    L.size = o;
    return L;
}

// ------------------------------------------------------------ ODE system

// The mixture's scalars: density and its inverse, Cp, dCp/dT, the thermal
// expansion.
struct Mix {
    double rhoM, irho, CpM, dCpMdT, alphav;
};

// Mixture properties + concentrations (gpuMixture.H:33-121). The sums over
// species run lane-strided and are combined by a fixed shuffle tree
// (deterministic; the reference sums sequentially), all of them in one
// reduction. No division per species: 1/rho_i = (R/W_i) T/p, the polynomials'
// divisors and 1/W_i are in the tables, and the expansion coefficient
// sum(Y_i / (rho_i T)) rhoM of a perfect gas is 1/T. jac: also Cp; STORE: also
// the per-species v and rhoM/W that the adjoint reads.
template <bool STORE = false, int G, class W>
__device__ __forceinline__ Mix mixture(const Grp<G>& g, const DevMech& M, const W& w, const WsLayout& L, int y_off,
                                       double p, bool jac) {
    const int nS = M.nS;
    const double T = w[y_off + nS];
    const double ToP = T / p;
    double sm[3] = {};
    for (int i = g.lane; i < nS; i += G) {
        const double yi = fmax(w[y_off + i], 0.0);
        const double vi = ldg(M.Rsp + i) * ToP;
        const double* a = M.spc + (size_t)coef_branch(T, ldg(M.Tcommon + i)) * 10 * nS + i;
        const double a0 = ldg(a), a1 = ldg(a + nS), a2 = ldg(a + 2 * nS), a3 = ldg(a + 3 * nS), a4 = ldg(a + 4 * nS);
        const double h1 = ldg(a + 5 * nS), h2 = ldg(a + 6 * nS), h3 = ldg(a + 7 * nS), h4 = ldg(a + 8 * nS),
                     a5 = ldg(a + 9 * nS);
        const double Cpi = (((a4 * T + a3) * T + a2) * T + a1) * T + a0;
        sm[0] += yi * vi;
        sm[1] += yi * Cpi;
        w[L.Ha + i] = ((((h4 * T + h3) * T + h2) * T + h1) * T + a0) * T + a5;
        w[L.c + i] = yi * ldg(M.invW + i);
        if (jac) {
            sm[2] += yi * (((4.0 * a4 * T + 3.0 * a3) * T + 2.0 * a2) * T + a1);
            w[L.Cp + i] = Cpi;
        }
        if (STORE) w[L.vj + i] = vi;
    }
    g.sums(sm);
    Mix x;
    x.irho = sm[0];
    x.rhoM = 1.0 / sm[0];
    x.CpM = sm[1];
    x.dCpMdT = sm[2];
    x.alphav = jac ? 1.0 / T : 0.0;
    for (int i = g.lane; i < nS; i += G) {
        w[L.c + i] *= x.rhoM;
        if (STORE) w[L.rhoMbyW + i] = x.rhoM * ldg(M.invW + i);
    }
    if (g.lane == 0) w[L.c + nS] = 1.0;
    g.sync();
    return x;
}

// Net rate omega of every reaction at the clipped temperature (gpuReaction.H:472-488)
// With write_cache, kf, 1/Kc and the third-body Ak of every reaction are kept
// for the Jacobian at the same state (same T and concentrations, hence the
// same values: the reference evaluates them twice), in the reaction's own
// staging slots 1..3 (every reaction has at least four: omega, dwdT and one
// term per side); only the Jacobian's parameters overwrite them, after reading.
template <int G, class W>
__device__ __forceinline__ void stage_omega(const Grp<G>& g, const DevMech& M, const W& w, const WsLayout& L,
                                            const TCache& tc, bool write_cache) {
    for (int q = g.lane; q < M.nR; q += G) {
        const RxnF R = load_fast(M, q);
        const LnK a = load_lnK(M, q, tc.T);
        double Ak;
        const double kf = fast_kf(M, q, R, tc, fast_M(M, w, L.Mtb, R, q), &Ak);
        const double invKc = R.irr() ? 1.0 : exp(-fast_lnKc(R, a, tc));
        const double Cf = fast_C(M, w, L.c, R, q, 0);
        const double Cr = fast_C(M, w, L.c, R, q, 1);
        const int so = L.stage + R.slot;
        w[so] = kf * Cf - (R.irr() ? 0.0 : kf * invKc * Cr);
        if (write_cache) {
            w[so + 1] = kf;
            w[so + 2] = invKc;
            w[so + 3] = Ak;
        }
    }
    g.sync();
}

__host__ __device__ constexpr int log2_group(int G) { return G <= 1 ? 0 : 1 + log2_group(G / 2); }
// The index of a group size's gather streams in DevMech (group_size_of).
__host__ __device__ constexpr int stream_index(int G) { return G == 96 ? 9 : log2_group(G); }

// Runs this thread's share of a gather stream (gf_internal.h, Stream):
// wd[dst + pos] = sum of coef * ws[src + slot] over each entry's records, in
// order. The group's loads (48 coalesced bytes and the position) are
// independent of the sums, so they pipeline (U groups at a time); one thread
// owns each output entry (no barriers inside). Bound by instructions,
// of which 16-byte records that each carried a position took more.
template <int U = 2, int G, class WS, class WD>
__device__ __forceinline__ void stream_gather(const Grp<G>& g, const Stream& st, const WS& ws, int src, const WD& wd,
                                              int dst) {
    const int4* o = reinterpret_cast<const int4*>(st.off) + g.lane;
    const double2* c = reinterpret_cast<const double2*>(st.coef) + g.lane;
    const int* p = st.pos + g.lane;
    double acc = 0.0;
#pragma unroll U
    for (int k = 0; k < st.len; ++k) {
        const int4 v = __ldg(o + (size_t)k * G);
        const double2 a = __ldg(c + (size_t)k * 2 * G), b = __ldg(c + (size_t)k * 2 * G + G);
        const int pos = __ldg(p + (size_t)k * G);
        acc = fma(a.x, ws.at(src, v.x), acc);
        acc = fma(a.y, ws.at(src, v.y), acc);
        acc = fma(b.x, ws.at(src, v.z), acc);
        acc = fma(b.y, ws.at(src, v.w), acc);
        if (pos >= 0) {
            wd[dst + pos] = acc;
            acc = 0.0;
        }
    }
}

// The sum of a species' parts in the dN/dt gather.
template <class W>
__device__ __forceinline__ double part_sum(const W& w, int at, const int* part, int s) {
    const int e = ldg(part + s + 1);
    double acc = 0.0;
    for (int i = ldg(part + s); i < e; ++i) acc += w[at + i];
    return acc;
}

// dN_s/dt gathered in the reference's order, scaled to dY/dt (gpuODESystem.H:40-48,
// 184-189), then dT/dt (:53-63). Writes out[0..m).
template <int G, class W>
__device__ __forceinline__ void gather_rhs(const Grp<G>& g, const DevMech& M, const W& w, const WsLayout& L,
                                           int out_off, const Mix& x) {
    const int nS = M.nS;
    stream_gather(g, M.dst[stream_index(G)], w, L.stage, w, L.part);
    g.sync();
    const int* part = M.dst_part[stream_index(G)];
    double s_h = 0;
    for (int s = g.lane; s < nS; s += G) {
        const double acc = part_sum(w, L.part, part, s) * (ldg(M.W + s) * x.irho);
        w[out_off + s] = acc;
        s_h += acc * w[L.Ha + s];
    }
    const double sh = g.sum(s_h);
    if (g.lane == 0) w[out_off + nS] = (-sh) / x.CpM;
    g.sync();
}

// gpuODESystem::derivatives (gpuODESystem.H:164-196): out = f(y), entries 0..nS
// With write_cache it also leaves what the Jacobian at the same state needs: the
// rate constants, the species' Cp, and the mixture (returned).
template <int G, class W>
__device__ __forceinline__ Mix derivatives(const Grp<G>& g, const DevMech& M, const W& w, const WsLayout& L,
                                           int y_off, double p, int out_off, bool write_cache = false) {
    Mix x;
    g.sync();
    {
        GF_PH_BEGIN(g)
        x = mixture(g, M, w, L, y_off, p, write_cache);
        GF_PH_END(g, PH_MIX)
    }
    const double T = w[y_off + M.nS];
    const double Tc = fmin(fmax(T, M.Tlow), M.Thigh);
    {
        GF_PH_BEGIN(g)
        if (M.n_tb > 0) {
            third_body_all(g, M, w, L.c, L.Mtb);
            g.sync();
        }
        // The Jacobian takes its rate constants at the unclipped T: where the
        // clip changes T, a first pass leaves them in the cache.
        const bool two = write_cache && Tc != T;
#pragma unroll 1
        for (int pass = two ? 0 : 1; pass < 2; ++pass)
            stage_omega(g, M, w, L, make_tcache(pass == 0 ? T : Tc), write_cache && !(two && pass == 1));
        GF_PH_END(g, PH_OMEGA)
    }
    {
        GF_PH_BEGIN(g)
        gather_rhs(g, M, w, L, out_off, x);
        GF_PH_END(g, PH_GATHER_RHS)
    }
    return x;
}

// Per-reaction Jacobian parameters (computeReactionParameters, gpuReaction.H:650-702)
// from the rate constants kept by stage_omega.
template <int G, class W>
__device__ __forceinline__ void stage_jacobian_params(const Grp<G>& g, const DevMech& M, const W& w,
                                                      const WsLayout& L, const TCache& tc) {
    for (int q = g.lane; q < M.nR; q += G) {
        const RxnF R = load_fast(M, q);
        const LnK a = load_lnK(M, q, tc.T);
        const int so = L.stage + R.slot;
        const double kf = w[so + 1], invKc = w[so + 2], Ak = w[so + 3];
        // dk/dT = k dln(k)/dT with the kInf factor for fall-off rates
        // (gpuFallOffReactionRate.H:140-141)
        const double ddT = kf * (R.type() >= GF_RATE_LINDEMANN_FALLOFF ? arr_dlnkdT1(M, q, tc)
                                                                       : fma(R.Ta0, tc.invT, R.beta0) * tc.invT);
        const double Cf = fast_products(M, w, L.c, R, q, 0, kf, so + 2);
        double dwdT = Cf * ddT;
        double omega = Cf * kf;
        double Cr = 0.0;
        if (!R.irr()) {
            const double kr = kf * invKc;
            Cr = fast_products(M, w, L.c, R, q, 1, kr, so + 2 + R.nl());
            dwdT -= Cr * (ddT * invKc - kr * fast_dlnKcdT(R, a, tc));
            omega -= Cr * kr;
        }
        w[so] = omega;
        w[so + 1] = dwdT;
        if (R.type() == GF_RATE_THIRD_BODY_ARRHENIUS) w[so + 2 + R.nl() + R.nr()] = Ak * (Cf - Cr * invKc);
    }
    g.sync();
}

// gpuODESystem::jacobian (gpuODESystem.H:198-281): dfdx (entries 0..nS) and J
// (m x m, Y and T rows/columns; the p row/column are zero).
//   raw entries (gather stream, one thread per entry): dN/dc, T-column and
//     third-body terms in the reference's order per entry;
//   phase 3 (lanes over rows): ddY_dcdY (gpuODESystem.H:65-103);
//   then the T row (ddT_dtdY, ddT_dtdT, :108-146).
// The rate constants, Cp and the mixture x are those that derivatives() with
// write_cache left at the same state, and dfdx is the f that it wrote to f_off
// (the reference evaluates all of them again), except where the reaction
// temperature limits clipped its rates: the Jacobian's are not clipped.
template <int G, class W>
__device__ __forceinline__ void jacobian(const Grp<G>& g, const DevMech& M, const W& w, const WsLayout& L,
                                         int y_off, double p, int f_off, const Mix& x) {
    const int nS = M.nS;
    const int ld = L.ld;
    const double T = w[y_off + nS];
    const double alphav = x.alphav, rToP = x.rhoM * (T / p);
    {
        GF_PH_BEGIN(g)
        stage_jacobian_params(g, M, w, L, make_tcache(T));
        GF_PH_END(g, PH_JPARAMS)
    }
    {
        GF_PH_BEGIN(g)
        if (T < M.Tlow || T > M.Thigh) {
            gather_rhs(g, M, w, L, L.dfdx, x);
        } else {
            for (int i = g.lane; i < M.m; i += G) w[L.dfdx + i] = w[f_off + i];
            g.sync();
        }
        GF_PH_END(g, PH_GATHER_RHS)
    }
    {
    GF_PH_BEGIN(g)
    // raw dN/dc, T-column and third-body terms of every entry (species rows x
    // species and T columns), one thread per entry, in the reference's order
    stream_gather<4>(g, M.jst[stream_index(G)], w, L.stage, w, L.J);
    g.sync();
    // phase 3: a thread per row and, where the group has more threads than
    // rows, per part of its columns (a part may be empty: it still leaves its sum)
    const int rows = (nS + 31) & ~31, parts = min(2, max(1, G / rows));
    const int part = G > 32 ? g.lane / rows : 0;
    const int c0 = part * nS / parts, c1 = (part + 1) * nS / parts;
    for (int s = G > 32 ? g.lane - part * rows : g.lane; s < nS && part < parts; s += parts > 1 ? rows : G) {
        const double Ws = ldg(M.W + s);
        const double dfs = w[L.dfdx + s];
        const int row = L.J + s * ld;
        double ddN = 0.0;
#pragma unroll 4
        for (int c = c0; c < c1; ++c) {
            const double raw = w[row + c];
            ddN -= raw * w[L.c + c];
            // (W_s / rhoM) raw (rhoM / W_c) + rhoM v_c df_s
            w[row + c] = Ws * ldg(M.invW + c) * raw + rToP * ldg(M.Rsp + c) * dfs;
        }
        if (parts > 1)
            w[L.part + part * nS + s] = ddN;
        else
            w[row + nS] = Ws * x.irho * (w[row + nS] + ddN * alphav) + alphav * dfs;
    }
    if (parts > 1) {
        g.sync();
        for (int s = g.lane; s < nS; s += G) {
            double ddN = 0.0;
            for (int k = 0; k < parts; ++k) ddN += w[L.part + k * nS + s];
            const int row = L.J + s * ld;
            w[row + nS] = ldg(M.W + s) * x.irho * (w[row + nS] + ddN * alphav) + alphav * w[L.dfdx + s];
        }
    }
    g.sync();
    GF_PH_END(g, PH_JROWS)
    }
    GF_PH_BEGIN(g)
    // T row: ddT_dtdY (gpuODESystem.H:108-126)
    const double dTdt = w[L.dfdx + nS];
    for (int i = g.lane; i < nS; i += G) {
        double acc = 0.0;
        for (int j = 0; j < nS; ++j) acc -= w[L.J + j * ld + i] * w[L.Ha + j];
        acc -= w[L.Cp + i] * dTdt;
        w[L.J + nS * ld + i] = acc / x.CpM;
    }
    // ddT_dtdT (gpuODESystem.H:129-146)
    double s_tt = 0.0;
    for (int i = g.lane; i < nS; i += G) s_tt += w[L.dfdx + i] * w[L.Cp + i] + w[L.J + i * ld + nS] * w[L.Ha + i];
    const double stt = g.sum(s_tt);
    if (g.lane == 0) w[L.J + nS * ld + nS] = ((-stt) - dTdt * x.dCpMdT) / x.CpM;
    g.sync();
    GF_PH_END(g, PH_TROW)
}

// ------------------------------------------------------------------ LU

// a = -J + I/(gamma dx) (gpuAdaptiveSolver.H:51-73) and the implicit row
// scaling vv = 1/max|a_ij| of LUDecompose (ludecompose.H:9-21).
template <int G, class W>
__device__ __forceinline__ void shift_and_scale(const Grp<G>& g, const W& w, int A, int ld, int vv, int m,
                                                double diag) {
    for (int i = g.lane; i < m; i += G) {
        double mx = 0.0;
        for (int j = 0; j < m; ++j) {
            double v = -w[A + i * ld + j];
            if (j == i) v += diag;
            w[A + i * ld + j] = v;
            const double t = fabs(v);
            if (t > mx) mx = t;
        }
        w[vv + i] = 1.0 / mx;
    }
    g.sync();
}

template <int G, class W>
__device__ __forceinline__ void row_scale(const Grp<G>& g, const W& w, int A, int ld, int vv, int m) {
    for (int i = g.lane; i < m; i += G) {
        double mx = 0.0;
        for (int j = 0; j < m; ++j) {
            const double t = fabs(w[A + i * ld + j]);
            if (t > mx) mx = t;
        }
        w[vv + i] = 1.0 / mx;
    }
    g.sync();
}

// One elimination update a - l * u. The solve kernels contract it to one FMA
// (EXACT = false); EXACT = true rounds the product and the difference
// separately, as the reference's CPU build (no contraction) computes the Crout
// sums of ludecompose.H:36-55, so that parity kernels can compare factors bit
// for bit.
template <bool EXACT>
__device__ __forceinline__ double msub(double a, double l, double u) {
    if constexpr (EXACT)
        return __dsub_rn(a, __dmul_rn(l, u));
    else
        return fma(-l, u, a);
}

// LUDecompose (ludecompose.H:9-92) in right-looking form: at step k the pivot
// column holds exactly the Crout sums of the reference, the pivot is the last
// row with the largest vv*|a| (">=", :62), full rows are swapped, a zero pivot
// becomes gpuSmall and the column below is scaled by 1/pivot. Every entry
// receives its updates in the same k order as the reference's Crout loops.
template <int G, bool EXACT = false, class W>
__device__ __forceinline__ void lu_decompose(const Grp<G>& g, const W& w, int A, int ld, int piv, int vv, int m) {
    for (int k = 0; k < m; ++k) {
        // pivot search
        double best = -1.0;
        int bi = -1;
        for (int i = k + g.lane; i < m; i += G) {
            const double t = w[vv + i] * fabs(w[A + i * ld + k]);
            if (t >= best) {
                best = t;
                bi = i;
            }
        }
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) {
            const double ob = __shfl_xor_sync(g.mask, best, o, G);
            const int oi = __shfl_xor_sync(g.mask, bi, o, G);
            if (ob > best || (ob == best && oi > bi)) {
                best = ob;
                bi = oi;
            }
        }
        const int iMax = bi < 0 ? 0 : bi;
        if (iMax != k) {
            for (int j = g.lane; j < m; j += G) {
                const double t = w[A + k * ld + j];
                w[A + k * ld + j] = w[A + iMax * ld + j];
                w[A + iMax * ld + j] = t;
            }
        }
        g.sync();
        if (g.lane == 0) {
            w.ip(piv + k) = iMax;
            if (iMax != k) w[vv + iMax] = w[vv + k];
            if (w[A + k * ld + k] == 0.0) w[A + k * ld + k] = kSmall;
        }
        g.sync();
        if (k != m - 1) {
            const double rDiag = 1.0 / w[A + k * ld + k];
            for (int i = k + 1 + g.lane; i < m; i += G) w[A + i * ld + k] *= rDiag;
            g.sync();
            for (int j = k + 1 + g.lane; j < m; j += G) {
                const double ukj = w[A + k * ld + j];
                for (int i = k + 1; i < m; ++i) w[A + i * ld + j] = msub<EXACT>(w[A + i * ld + j], w[A + i * ld + k], ukj);
            }
            g.sync();
        }
    }
}

// Blocked form of lu_decompose (panels of NB columns). For every entry the
// sequence of updates is the same as in the unblocked loop (all steps k in
// ascending order; row exchanges move rows that have received the same
// updates), so the factors are identical; the trailing matrix receives NB
// updates per load/store instead of one.
// Panel steps k0 .. k1-1 of the blocked LU (a group of at most one warp):
// pivot search, row exchange, zero-pivot fix, column scaling and the update of
// the panel's remaining columns.
template <int G, bool EXACT = false, class W>
__device__ __forceinline__ void lu_panel(const Grp<G>& g, const W& w, int A, int ld, int piv, int vv, int m, int k0,
                                         int k1) {
    for (int k = k0; k < k1; ++k) {
        double best = -1.0;
        int bi = -1;
        for (int i = k + g.lane; i < m; i += G) {
            const double t = w[vv + i] * fabs(w[A + i * ld + k]);
            if (t >= best) {
                best = t;
                bi = i;
            }
        }
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) {
            const double ob = __shfl_xor_sync(g.mask, best, o, G);
            const int oi = __shfl_xor_sync(g.mask, bi, o, G);
            if (ob > best || (ob == best && oi > bi)) {
                best = ob;
                bi = oi;
            }
        }
        const int iMax = bi < 0 ? 0 : bi;
        if (iMax != k) {
            for (int j = g.lane; j < m; j += G) {
                const double t = w[A + k * ld + j];
                w[A + k * ld + j] = w[A + iMax * ld + j];
                w[A + iMax * ld + j] = t;
            }
        }
        g.sync();
        if (g.lane == 0) {
            w.ip(piv + k) = iMax;
            if (iMax != k) w[vv + iMax] = w[vv + k];
            if (w[A + k * ld + k] == 0.0) w[A + k * ld + k] = kSmall;
        }
        g.sync();
        if (k != m - 1) {
            const double rDiag = 1.0 / w[A + k * ld + k];
            for (int i = k + 1 + g.lane; i < m; i += G) {
                const double lik = w[A + i * ld + k] * rDiag;
                w[A + i * ld + k] = lik;
                for (int j = k + 1; j < k1; ++j) w[A + i * ld + j] = msub<EXACT>(w[A + i * ld + j], lik, w[A + k * ld + j]);
            }
            g.sync();
        }
    }
}

// c += a b for one 8 x 8 tile of doubles held by a warp (a: 8 x 4, b: 4 x 8;
// lane l holds a[l/4][l%4], b[l%4][l/4], c[l/4][2 (l%4) + 0, 1]). The unit
// accumulates its four products as a chain of FMAs in ascending k (measured on
// the B200: 262,144 results of random tiles bit for bit; the instruction's
// definition does not promise the order), so a tile update is the same as the
// scalar loop's. test_lu_edges (tests/test_gpu_edges.py) holds every form's factors
// to the scalar form's bit for bit, and would show a chip that adds otherwise.
__device__ __forceinline__ void mma_f64(double& c0, double& c1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1},{%2},{%3},{%0,%1};"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}

constexpr int kPanel = 8;  // columns per panel of lu_decompose_mma: two tile depths

// The pivot of a panel step by the reference's rule where the high words do not
// decide it: the last position with the largest vv |a| among the candidates
// (lab >= k; a NaN is never taken), row k where there is none. Returns the lane
// and register row that hold it. Out of line: reached on ties only.
template <int RP>
struct PivotRows {
    double t[RP];  // vv |a|
    int lab[RP];
};
template <int RP>
__device__ __noinline__ int pivot_exact(PivotRows<RP> c, int k) {
    double best = -1.0;
    int bi = -1, ri = 0;
#pragma unroll
    for (int r = 0; r < RP; ++r) {
        if (c.lab[r] >= k && (c.t[r] > best || (c.t[r] == best && c.lab[r] > bi))) {
            best = c.t[r];
            bi = c.lab[r];
            ri = r;
        }
    }
    const bool has = bi >= 0;
    const unsigned hi = has ? (unsigned)__double2hiint(best) : 0u;
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const bool c1 = has && hi == mh;
    const unsigned lo = c1 ? (unsigned)__double2loint(best) : 0u;
    const unsigned ml = __reduce_max_sync(0xffffffffu, lo);
    int mr = (int)__reduce_max_sync(0xffffffffu, (c1 && lo == ml) ? (unsigned)(bi + 1) : 0u) - 1;
    if (mr < 0) {
        mr = k;
#pragma unroll
        for (int r = 0; r < RP; ++r)
            if (c.lab[r] == k) {
                bi = k;
                ri = r;
            }
    }
    const int li = __ffs(__ballot_sync(0xffffffffu, bi == mr)) - 1;
    return li | (__shfl_sync(0xffffffffu, ri, li) << 5);
}

// Panel steps k0 .. k0+kb-1 with the panel held in registers (one full warp):
// lane l holds the rows at positions k0 + l + 32 r, each with its row scaling
// and a label, the position that it has in the reference's matrix after the
// exchanges so far (-1: no row). An exchange of rows k and iMax swaps two
// labels, and at the end perm[] takes the labels: perm[position] = the row of
// the workspace that holds it. Rows do not move. The pivot search (ludecompose.H
// :57-63) compares the high words of vv |a|: one integer warp reduction; where
// they tie, are zero or a NaN is the largest, pivot_exact decides. Meanwhile
// every lane has formed the reciprocal of its own candidate, so the division is
// off the chain of dependent operations. A zero pivot becomes gpuSmall (:81).
// Difference: when every candidate of a column is NaN, the reference exchanges
// row k with row 0 (its iMax starts at 0); here none is. The reciprocal pivots
// go to rd, the pivots to piv (unless piv < 0).
template <int RP, bool EXACT, class W>
__device__ __forceinline__ void lu_panel_reg(const W& w, int A, int ld, int piv, int sc, int rd, int perm, int m,
                                             int k0, int kb) {
    const int l = threadIdx.x & 31;
    double a[RP][kPanel], sv[RP];
    int lab[RP], row[RP];
#pragma unroll
    for (int r = 0; r < RP; ++r) {
        const int p = k0 + l + 32 * r;
        lab[r] = p < m ? p : -1;
        row[r] = p < m ? w.ip(perm + p) : 0;
        sv[r] = w[sc + row[r]];
#pragma unroll
        for (int t = 0; t < kPanel; ++t) a[r][t] = t < kb ? w[A + row[r] * ld + k0 + t] : 0.0;
    }
#pragma unroll
    for (int kk = 0; kk < kPanel; ++kk) {
        if (kk >= kb) break;
        const int k = k0 + kk;
        // the lane's candidate by high words (-1: no candidate)
        PivotRows<RP> c;
        int key = -1, ri = 0, tie = 0;
        double x = a[0][kk];
#pragma unroll
        for (int r = 0; r < RP; ++r) {
            c.t[r] = sv[r] * fabs(a[r][kk]);
            c.lab[r] = lab[r];
            const int h = lab[r] >= k ? __double2hiint(c.t[r]) : -1;
            if (r == 0) {
                key = h;
            } else {
                tie = h == key ? 1 : (h > key ? 0 : tie);
                if (h > key) {
                    key = h;
                    ri = r;
                    x = a[r][kk];
                }
            }
        }
        double rinv = 1.0 / x;
        const int mh = __reduce_max_sync(0xffffffffu, key);
        const unsigned own = __ballot_sync(0xffffffffu, key == mh);
        const unsigned tied = __ballot_sync(0xffffffffu, key == mh && tie);
        int li = __ffs(own) - 1;
        if (tied != 0 || (own & (own - 1)) != 0 || mh <= 0 || mh > 0x7ff00000) {
            const int v = pivot_exact<RP>(c, k);
            li = v & 31;
            if (l == li) {
                ri = v >> 5;
#pragma unroll
                for (int r = 0; r < RP; ++r)
                    if (r == ri) x = a[r][kk];
                if (x == 0.0) x = kSmall;
                rinv = 1.0 / x;
            }
        }
        // the pivot row's label, reciprocal and remaining entries, to every lane
        int mine = lab[0];
#pragma unroll
        for (int r = 1; r < RP; ++r)
            if (r == ri) mine = lab[r];
        const int iMax = __shfl_sync(0xffffffffu, mine, li);
        rinv = __shfl_sync(0xffffffffu, rinv, li);
        double u[kPanel];
#pragma unroll
        for (int t = kk + 1; t < kPanel; ++t) {
            double y = a[0][t];
#pragma unroll
            for (int r = 1; r < RP; ++r)
                if (r == ri) y = a[r][t];
            u[t] = __shfl_sync(0xffffffffu, y, li);
        }
#pragma unroll
        for (int r = 0; r < RP; ++r) {
            if (lab[r] == k) lab[r] = iMax;
            if (l == li && r == ri) {
                lab[r] = k;
                a[r][kk] = x;
            }
        }
        if (l == 0) {
            if (piv >= 0) w.ip(piv + k) = iMax;
            w[rd + k] = rinv;
        }
#pragma unroll
        for (int r = 0; r < RP; ++r) {
            if (lab[r] > k) {
                const double lik = a[r][kk] * rinv;
                a[r][kk] = lik;
#pragma unroll
                for (int t = kk + 1; t < kPanel; ++t) a[r][t] = msub<EXACT>(a[r][t], lik, u[t]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < RP; ++r) {
        if (lab[r] >= 0) {
#pragma unroll
            for (int t = 0; t < kPanel; ++t)
                if (t < kb) w[A + row[r] * ld + k0 + t] = a[r][t];
            w.ip(perm + lab[r]) = row[r];
        }
    }
}

// Blocked LU for a full warp or a multi-warp group (m <= 32 RP): warp 0 factors
// panels of 8 columns in registers (lu_panel_reg); the U12 rows take their
// updates with lanes over columns; the trailing matrix is updated in 8 x 8
// tiles by the FP64 matrix instruction, the tiles shared out to the warps in
// runs along a tile row (the run keeps its part of L in registers). Rows are
// not exchanged meanwhile: position i of the reference's matrix is row perm[i];
// one pass at the end puts them in order. Every entry receives its updates in k order, as in
// lu_decompose, so factors and pivots are the same bit for bit (EXACT: scalar
// updates with two roundings). sc: the row scalings; rd: out, 1 / U[i][i].
//
// Why: the factorisation was 30k of the 108k warp instructions of an attempt
// (m = 54, 128 threads): rank-4 updates spend most of theirs on addresses and
// loads, and the exchanges were another pass.
// A form with the whole matrix in registers and one barrier per column was
// slower (rank-1 updates: 62k instructions).
template <int G, int RP, bool EXACT, class W>
__device__ __forceinline__ void lu_decompose_mma(const Grp<G>& g, const W& w, int A, int ld, int piv, int sc, int rd,
                                                 int perm, int m) {
    constexpr int NW = G / 32;
    const int wid = g.warp();
    const int l = threadIdx.x & 31;
    for (int i = g.lane; i < m; i += G) w.ip(perm + i) = i;
    g.sync();
#pragma unroll 1
    for (int k0 = 0;; k0 += kPanel) {
        const int k1 = min(k0 + kPanel, m);
        {
            GF_PH_BEGIN(g)
            // the last panels have one row per lane: fewer instructions a step
            if (wid == 0) {
                if (RP == 1 || m - k0 <= 32)
                    lu_panel_reg<1, EXACT>(w, A, ld, piv, sc, rd, perm, m, k0, k1 - k0);
                else
                    lu_panel_reg<RP, EXACT>(w, A, ld, piv, sc, rd, perm, m, k0, k1 - k0);
            }
            g.sync();
            GF_PH_END(g, PH_LU_PANEL)
        }
        if (k1 >= m) break;
        {
            GF_PH_BEGIN(g)
            // U12: rows k0 .. k1-1 (a full panel), columns k1 .. m-1
            if (k1 + (g.lane & ~31) < m) {
                int ro[kPanel];
#pragma unroll
                for (int t = 0; t < kPanel; ++t) ro[t] = A + w.ip(perm + k0 + t) * ld;
                for (int j = k1 + g.lane; j < m; j += G) {
                    double u[kPanel];
#pragma unroll
                    for (int t = 0; t < kPanel; ++t) u[t] = w[ro[t] + j];
#pragma unroll
                    for (int t = 1; t < kPanel; ++t) {
#pragma unroll
                        for (int t2 = 0; t2 < t; ++t2) u[t] = msub<EXACT>(u[t], w[ro[t] + k0 + t2], u[t2]);
                        w[ro[t] + j] = u[t];
                    }
                }
            }
            g.sync();
            GF_PH_END(g, PH_LU_U12)
        }
        GF_PH_BEGIN(g)
        if constexpr (EXACT) {
            for (int j = k1 + l; j < m; j += 32)
                for (int i = k1 + wid; i < m; i += NW) {
                    const int ri = A + w.ip(perm + i) * ld;
                    double a = w[ri + j];
                    for (int t = k0; t < k1; ++t) a = msub<true>(a, w[ri + t], w[A + w.ip(perm + t) * ld + j]);
                    w[ri + j] = a;
                }
        } else {
            const int nt = (m - k1 + 7) >> 3;
            const int T = nt * nt;
            int t = wid * T / NW;
            const int t_end = (wid + 1) * T / NW;
            int tr = t / nt, tc = t - tr * nt;
            const int r8 = l >> 2, c4 = l & 3;
            const int p0 = A + w.ip(perm + k0 + c4) * ld, p1 = A + w.ip(perm + k0 + 4 + c4) * ld;
            while (t < t_end) {
                const int i = k1 + 8 * tr + r8;
                const bool rin = i < m;
                const int ri = A + (rin ? w.ip(perm + i) : 0) * ld;
                const double a0 = rin ? -w[ri + k0 + c4] : 0.0, a1 = rin ? -w[ri + k0 + 4 + c4] : 0.0;
                const int run = min(nt - tc, t_end - t);
                int col = k1 + 8 * tc;
                // two tiles of the run at a time: their loads and updates overlap
                for (int n = 0; n < run; n += 2, col += 16) {
                    double b0[2], b1[2], c0[2], c1[2];
                    bool in0[2], in1[2];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int cb = col + 8 * h + r8, j = col + 8 * h + 2 * c4;
                        const bool on = n + h < run;
                        b0[h] = on && cb < m ? w[p0 + cb] : 0.0;
                        b1[h] = on && cb < m ? w[p1 + cb] : 0.0;
                        in0[h] = on && rin && j < m;
                        in1[h] = on && rin && j + 1 < m;
                        c0[h] = in0[h] ? w[ri + j] : 0.0;
                        c1[h] = in1[h] ? w[ri + j + 1] : 0.0;
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h) mma_f64(c0[h], c1[h], a0, b0[h]);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int j = col + 8 * h + 2 * c4;
                        mma_f64(c0[h], c1[h], a1, b1[h]);
                        if (in0[h]) w[ri + j] = c0[h];
                        if (in1[h]) w[ri + j + 1] = c1[h];
                    }
                }
                t += run;
                ++tr;
                tc = 0;
            }
        }
        g.sync();
        GF_PH_END(g, PH_LU_TRAIL)
    }
    // rows to their positions, a few columns of a warp at a time
    {
        GF_PH_BEGIN(g)
        constexpr int CB = 4;
        int from[RP];
#pragma unroll
        for (int r = 0; r < RP; ++r) from[r] = l + 32 * r < m ? A + w.ip(perm + l + 32 * r) * ld : A;
        for (int j0 = wid * CB; j0 < m; j0 += NW * CB) {
            double v[RP][CB];
#pragma unroll
            for (int r = 0; r < RP; ++r)
#pragma unroll
                for (int c = 0; c < CB; ++c) v[r][c] = j0 + c < m ? w[from[r] + j0 + c] : 0.0;
            __syncwarp();
#pragma unroll
            for (int r = 0; r < RP; ++r)
#pragma unroll
                for (int c = 0; c < CB; ++c)
                    if (l + 32 * r < m && j0 + c < m) w[A + (l + 32 * r) * ld + j0 + c] = v[r][c];
            __syncwarp();
        }
        g.sync();
        GF_PH_END(g, PH_LU_PERM)
    }
}

template <int G, int NB, bool EXACT = false, class W>
__device__ __forceinline__ void lu_decompose_blocked(const Grp<G>& g, const W& w, int A, int ld, int piv, int vv,
                                                     int m) {
    if constexpr (G > 32) {
        // multi-warp group: warp 0 factors each panel; the U12 rows and the
        // trailing matrix are updated by all warps (lanes over columns, warps
        // over rows), each entry still receiving its updates in k order
        constexpr int NWp = G / 32;
        const int wid = g.warp(), l = threadIdx.x & 31;
        for (int k0 = 0; k0 < m; k0 += NB) {
            const int kb = min(NB, m - k0);
            const int k1 = k0 + kb;
            if (wid == 0) {
                Grp<32> g32;
                lu_panel<32, EXACT>(g32, w, A, ld, piv, vv, m, k0, k1);
            }
            __syncthreads();
            if (k1 >= m) break;
            for (int j = k1 + g.lane; j < m; j += G) {
                for (int t = 1; t < kb; ++t) {
                    double v = w[A + (k0 + t) * ld + j];
                    for (int t2 = 0; t2 < t; ++t2)
                        v = msub<EXACT>(v, w[A + (k0 + t) * ld + k0 + t2], w[A + (k0 + t2) * ld + j]);
                    w[A + (k0 + t) * ld + j] = v;
                }
            }
            __syncthreads();
            for (int j = k1 + l; j < m; j += 32) {
                double u[NB];
#pragma unroll
                for (int t = 0; t < NB; ++t) u[t] = t < kb ? w[A + (k0 + t) * ld + j] : 0.0;
                for (int i = k1 + wid; i < m; i += NWp) {
                    double a = w[A + i * ld + j];
#pragma unroll
                    for (int t = 0; t < NB; ++t)
                        if (t < kb) a = msub<EXACT>(a, w[A + i * ld + k0 + t], u[t]);
                    w[A + i * ld + j] = a;
                }
            }
            __syncthreads();
        }
    } else {
    for (int k0 = 0; k0 < m; k0 += NB) {
        const int kb = min(NB, m - k0);
        const int k1 = k0 + kb;
        // 1. panel: columns [k0, k1), rows [k0, m)
        lu_panel<G, EXACT>(g, w, A, ld, piv, vv, m, k0, k1);
        if (k1 >= m) break;
        // 2. U12: rows [k0, k1), columns [k1, m)
        for (int j = k1 + g.lane; j < m; j += G) {
            double u[NB];
#pragma unroll
            for (int t = 0; t < NB; ++t) {
                if (t < kb) {
                    double v = w[A + (k0 + t) * ld + j];
                    for (int t2 = 0; t2 < t; ++t2) v = msub<EXACT>(v, w[A + (k0 + t) * ld + k0 + t2], u[t2]);
                    u[t] = v;
                    w[A + (k0 + t) * ld + j] = v;
                }
            }
            // 3. trailing update of this column: rows [k1, m)
            for (int i = k1; i < m; ++i) {
                double a = w[A + i * ld + j];
#pragma unroll
                for (int t = 0; t < NB; ++t)
                    if (t < kb) a = msub<EXACT>(a, w[A + i * ld + k0 + t], u[t]);
                w[A + i * ld + j] = a;
            }
        }
        g.sync();
    }
    }
}

// LUBacksubstitute (ludecompose.H:94-130): the row exchanges first (equivalent
// to the reference's on-the-fly exchange, which only moves untouched values),
// then column-oriented forward and backward substitution. Forward: same
// subtraction order as the reference; backward: descending column order
// (the reference sums ascending), an ulp-level difference.
template <int G, class W>
__device__ __forceinline__ void lu_solve(const Grp<G>& g, const W& w, int A, int ld, int piv, int m, int b) {
    GF_PH_BEGIN(g)
    g.sync();
    if (g.lane == 0) {
        for (int i = 0; i < m; ++i) {
            const int ip = w.ip(piv + i);
            if (ip != i) {
                const double t = w[b + ip];
                w[b + ip] = w[b + i];
                w[b + i] = t;
            }
        }
    }
    g.sync();
    for (int j = 0; j < m - 1; ++j) {
        const double bj = w[b + j];
        for (int i = j + 1 + g.lane; i < m; i += G) w[b + i] -= w[A + i * ld + j] * bj;
        g.sync();
    }
    for (int j = m - 1; j >= 0; --j) {
        const double xj = w[b + j] / w[A + j * ld + j];
        g.sync();
        if (g.lane == 0) w[b + j] = xj;
        for (int i = g.lane; i < j; i += G) w[b + i] -= w[A + i * ld + j] * xj;
        g.sync();
    }
    GF_PH_END(g, PH_SOLVE)
}

// The row permutation LUBacksubstitute applies to a right-hand side (its
// sequence of exchanges b[i] <-> b[piv[i]]) as one gather: rhs'[i] = b[perm[i]].
// A group of 32 or more threads computes each position's source in parallel
// (the exchanges undone in reverse order: the row at position p came from
// piv-exchange k applied to the source so far, k = m-1 .. 0); smaller groups
// run the exchanges in order on one thread. Both give the same permutation.
template <int G, class W>
__device__ __forceinline__ void lu_perm(const Grp<G>& g, const W& w, int piv, int perm, int m) {
    g.sync();
    if constexpr (G >= 32) {
        for (int p = g.lane; p < m; p += G) {
            int s = p;
            for (int k = m - 1; k >= 0; --k) {
                const int q = w.ip(piv + k);
                s = s == k ? q : (s == q ? k : s);
            }
            w.ip(perm + p) = s;
        }
    } else if (g.lane == 0) {
        for (int i = 0; i < m; ++i) w.ip(perm + i) = i;
        for (int i = 0; i < m; ++i) {
            const int ip = w.ip(piv + i);
            if (ip != i) {
                const int t = w.ip(perm + i);
                w.ip(perm + i) = w.ip(perm + ip);
                w.ip(perm + ip) = t;
            }
        }
    }
    g.sync();
}

// LUBacksubstitute with the right-hand side in registers: lane l holds rows
// l, l + G, ...; the pivot value of each step is broadcast by a shuffle, so
// the substitution chain runs without shared-memory round trips or barriers.
// Same subtraction order as lu_solve; the backward step multiplies by the
// reciprocal of the diagonal, rdiag[j] = 1 / U[j][j] (computed once per LU),
// instead of dividing (ulp-level).
constexpr int kRegRows = 160;

// Whether the solves of a group of G threads (lu_solve_any) take the row
// permutation as a gather list (perm) or follow the pivots step by step (piv).
template <int G>
__host__ __device__ constexpr bool solve_uses_perm(int m) {
    return (G >= 32 && m <= 128) || (G >= 16 && G <= 32 && m <= kRegRows);
}

// The solve kernels' layout for a group of G threads: the pivot array the
// solves do not read (written by the factorisation or by lu_perm, consumed
// before the first stage) goes to k1.
template <int G>
__host__ __device__ inline WsLayout solve_layout(int nS, int nR, int n_slots, int n_tb, int pad = 0) {
    WsLayout L = make_layout(nS, nR, n_slots, n_tb, false, pad);
    if (solve_uses_perm<G>(nS + 1))
        L.piv = L.k1;
    else
        L.perm = L.k1;
    return L;
}
template <int G, class W>
__device__ __forceinline__ void lu_solve_reg(const Grp<G>& g, const W& w, int A, int ld, int perm, int rdiag, int m,
                                             int b) {
    constexpr int R = kRegRows / G;
    GF_PH_BEGIN(g)
    double x[R];
    g.sync();
#pragma unroll
    for (int t = 0; t < R; ++t) {
        const int i = t * G + g.lane;
        x[t] = i < m ? w[b + w.ip(perm + i)] : 0.0;
    }
    g.sync();
#pragma unroll
    for (int t = 0; t < R; ++t) {
        if (t * G < m - 1) {
            const int lmax = min(G, m - 1 - t * G);
            for (int l = 0; l < lmax; ++l) {
                const int j = t * G + l;
                const double bj = __shfl_sync(g.mask, x[t], l, G);
#pragma unroll
                for (int u = t; u < R; ++u) {
                    const int i = u * G + g.lane;
                    if (i > j && i < m) x[u] -= w[A + i * ld + j] * bj;
                }
            }
        }
    }
#pragma unroll
    for (int t = R - 1; t >= 0; --t) {
        if (t * G < m) {
            const int lmax = min(G, m - t * G);
            for (int l = lmax - 1; l >= 0; --l) {
                const int j = t * G + l;
                const double xj = __shfl_sync(g.mask, x[t], l, G) * w[rdiag + j];
                if (g.lane == l) x[t] = xj;
#pragma unroll
                for (int u = 0; u <= t; ++u) {
                    const int i = u * G + g.lane;
                    if (i < j) x[u] -= w[A + i * ld + j] * xj;
                }
            }
        }
    }
#pragma unroll
    for (int t = 0; t < R; ++t) {
        const int i = t * G + g.lane;
        if (i < m) w[b + i] = x[t];
    }
    g.sync();
    GF_PH_END(g, PH_SOLVE)
}

#ifndef GF_SOLVE_UNROLL
#define GF_SOLVE_UNROLL 1
#endif
constexpr int kSolveUnroll = GF_SOLVE_UNROLL;  // blocks of columns unrolled together
// Register form for one full warp with R rows per lane (m <= 32 R): lane l
// holds rows l + 32 u. Columns go in blocks of four: the block's four values
// are fetched with shuffles that do not wait for one another, every lane
// eliminates inside the block by itself (the six factors are at one address for
// all lanes), and then applies the four columns to its rows; columns that fill
// no block go one by one. Same operations and order per row as column by column
// (lu_solve_reg). Bound by the chain of dependent operations of one warp, then
// by its instructions: rows past m read row 0 and are never stored, so that the
// loops carry no predicate for them.
template <int R, class W>
__device__ __forceinline__ void lu_solve_warp(const W& w, int A, int ld, int perm, int rdiag, int m, int b) {
    const int lane = threadIdx.x & 31;
    double x[R];
    int ro[R];
    __syncwarp();
#pragma unroll
    for (int u = 0; u < R; ++u) {
        const int i = u * 32 + lane;
        ro[u] = i < m ? A + i * ld : A;
        x[u] = i < m ? w[b + w.ip(perm + i)] : 0.0;
    }
    // forward substitution with the unit lower factor: columns 0 .. m-2
#pragma unroll
    for (int t = 0; t < R; ++t) {
        const int n = min(32, m - 1 - 32 * t);  // columns of this tile
        int l0 = 0;
#pragma unroll kSolveUnroll
        for (; l0 + 4 <= n; l0 += 4) {
            const int j0 = 32 * t + l0, rb = A + j0 * ld + j0, d = lane - l0;
            double y[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) y[i] = __shfl_sync(0xffffffffu, x[t], l0 + i);
            const double l10 = w[rb + ld], l20 = w[rb + 2 * ld], l21 = w[rb + 2 * ld + 1], l30 = w[rb + 3 * ld],
                         l31 = w[rb + 3 * ld + 1], l32 = w[rb + 3 * ld + 2];
            y[1] -= l10 * y[0];
            y[2] -= l20 * y[0];
            y[3] -= l30 * y[0];
            y[2] -= l21 * y[1];
            y[3] -= l31 * y[1];
            y[3] -= l32 * y[2];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const double f = w[ro[t] + j0 + k];
                if (d > k) x[t] -= f * y[k];
#pragma unroll
                for (int u = t + 1; u < R; ++u) x[u] -= w[ro[u] + j0 + k] * y[k];
            }
        }
#pragma unroll 1
        for (; l0 < n; ++l0) {
            const int j = 32 * t + l0;
            const double bj = __shfl_sync(0xffffffffu, x[t], l0);
            if (lane > l0) x[t] -= w[ro[t] + j] * bj;
#pragma unroll
            for (int u = t + 1; u < R; ++u) x[u] -= w[ro[u] + j] * bj;
        }
    }
    // backward substitution, descending columns, x_j = (...) * (1 / U[j][j])
#pragma unroll
    for (int t = R - 1; t >= 0; --t) {
        int n = min(32, m - 32 * t);
#pragma unroll 1
        for (; n > 0 && (n & 3); --n) {
            const int l0 = n - 1, j = 32 * t + l0;
            const double xj = __shfl_sync(0xffffffffu, x[t], l0) * w[rdiag + j];
            const double f = w[ro[t] + j];
            if (lane < l0) x[t] -= f * xj;
            if (lane == l0) x[t] = xj;
#pragma unroll
            for (int u = 0; u < t; ++u) x[u] -= w[ro[u] + j] * xj;
        }
#pragma unroll kSolveUnroll
        for (int l0 = n - 4; l0 >= 0; l0 -= 4) {
            const int j0 = 32 * t + l0, rb = A + j0 * ld + j0, d = lane - l0;
            double y[4];
#pragma unroll
            for (int i = 3; i >= 0; --i) y[i] = __shfl_sync(0xffffffffu, x[t], l0 + i);
            const double u01 = w[rb + 1], u02 = w[rb + 2], u03 = w[rb + 3], u12 = w[rb + ld + 2], u13 = w[rb + ld + 3],
                         u23 = w[rb + 2 * ld + 3];
            y[3] *= w[rdiag + j0 + 3];
            y[2] -= u23 * y[3];
            y[1] -= u13 * y[3];
            y[0] -= u03 * y[3];
            y[2] *= w[rdiag + j0 + 2];
            y[1] -= u12 * y[2];
            y[0] -= u02 * y[2];
            y[1] *= w[rdiag + j0 + 1];
            y[0] -= u01 * y[1];
            y[0] *= w[rdiag + j0];
#pragma unroll
            for (int k = 3; k >= 0; --k) {
                const double f = w[ro[t] + j0 + k];
                if (d < k) x[t] -= f * y[k];
                if (d == k) x[t] = y[k];
#pragma unroll
                for (int u = 0; u < t; ++u) x[u] -= w[ro[u] + j0 + k] * y[k];
            }
        }
    }
#pragma unroll
    for (int u = 0; u < R; ++u)
        if (u * 32 + lane < m) w[b + 32 * u + lane] = x[u];
    __syncwarp();
}

// rdiag: 1 / diagonal of U, used by the register form (G >= 16).
template <int G, class W>
__device__ __forceinline__ void lu_solve_any(const Grp<G>& g, const W& w, int A, int ld, int piv, int perm, int rdiag,
                                             int m, int b) {
    if constexpr (G >= 32) {
        // the substitution chain is sequential: one warp (the cell's warp, or
        // warp 0 of a multi-warp group) runs it in registers
        if (m <= 64) {
            g.sync();
            GF_PH_BEGIN(g)
            if (G == 32 || g.lane < 32) {
                if (m <= 32)
                    lu_solve_warp<1>(w, A, ld, perm, rdiag, m, b);
                else
                    lu_solve_warp<2>(w, A, ld, perm, rdiag, m, b);
            }
            g.sync();
            GF_PH_END(g, PH_SOLVE)
            return;
        }
        // 64 < m <= 128 (the 100-species mechanism): four rows per lane
        if (m <= 128) {
            g.sync();
            if (G == 32 || g.lane < 32) lu_solve_warp<4>(w, A, ld, perm, rdiag, m, b);
            g.sync();
            return;
        }
    }
    if constexpr (G >= 16 && G <= 32) {
        if (m <= kRegRows) {
            lu_solve_reg(g, w, A, ld, perm, rdiag, m, b);
            return;
        }
    }
    lu_solve(g, w, A, ld, piv, m, b);
}

// The factorisation as the solve kernels run it, after the row scaling sc: by
// register panels and matrix tiles for 32 or more threads (m <= 128), the blocked form otherwise, with panels of NB columns and
// rows exchanged; then, for groups of 16 or more threads, the reciprocal pivots
// 1 / U[i][i] in rd (sc and rd may be the same array for fewer than 32 threads)
// and the row permutation of the solves (lu_solve_any).
template <int G, bool EXACT = false, int NB = 8, class W>
__device__ __forceinline__ void lu_factor(const Grp<G>& g, const W& w, int A, int ld, int piv, int sc, int rd,
                                          int perm, int m) {
    if constexpr (G >= 32) {
        if (m <= 128) {
            GF_PH_BEGIN(g)
            if (m <= 32)
                lu_decompose_mma<G, 1, EXACT>(g, w, A, ld, piv, sc, rd, perm, m);
            else if (m <= 64)
                lu_decompose_mma<G, 2, EXACT>(g, w, A, ld, piv, sc, rd, perm, m);
            else
                lu_decompose_mma<G, 4, EXACT>(g, w, A, ld, piv, sc, rd, perm, m);
            GF_PH_END(g, PH_LU)
            return;
        }
    }
    {
        GF_PH_BEGIN(g)
        lu_decompose_blocked<G, NB, EXACT>(g, w, A, ld, piv, sc, m);
        GF_PH_END(g, PH_LU)
    }
    if (G >= 16) {
        GF_PH_BEGIN(g)
        for (int i = g.lane; i < m; i += G) w[rd + i] = 1.0 / w[A + i * ld + i];
        lu_perm(g, w, piv, perm, m);
        GF_PH_END(g, PH_LU_PERM)
    }
}

// ------------------------------------------------------------- Rosenbrock

struct RosCoeffs {
    int s;  // stages with a linear solve
    double gamma, a21, a31, a32, c21, c31, c32, c41, c42, c43, b1, b2, b3, b4, e1, e2, e3, e4, d1, d2, d3, d4;
};

// gpuRosenbrock12.H:14-31, gpuRosenbrock23.H:13-37, gpuRosenbrock34.H:13-46
__device__ __forceinline__ RosCoeffs ros_coeffs(int solver) {
    RosCoeffs c = {};
    if (solver == GF_ROSENBROCK12) {
        const double gamma = 1.0 + 1.0 / 1.414213562373095;
        c.s = 2;
        c.gamma = gamma;
        c.a21 = 1.0 / gamma;
        c.c21 = -2.0 / gamma;
        c.b1 = (3.0 / 2.0) / gamma;
        c.b2 = (1.0 / 2.0) / gamma;
        c.e1 = c.b1 - 1.0 / gamma;
        c.e2 = c.b2;
        c.d1 = gamma;
        c.d2 = -gamma;
    } else if (solver == GF_ROSENBROCK23) {
        c.s = 3;
        c.a21 = 1;
        c.a31 = 1;
        c.a32 = 0;
        c.c21 = -1.0156171083877702091975600115545;
        c.c31 = 4.0759956452537699824805835358067;
        c.c32 = 9.2076794298330791242156818474003;
        c.b1 = 1;
        c.b2 = 6.1697947043828245592553615689730;
        c.b3 = -0.4277225654321857332623837380651;
        c.e1 = 0.5;
        c.e2 = -2.9079558716805469821718236208017;
        c.e3 = 0.2235406989781156962736090927619;
        c.gamma = 0.43586652150845899941601945119356;
        c.d1 = 0.43586652150845899941601945119356;
        c.d2 = 0.24291996454816804366592249683314;
        c.d3 = 2.1851380027664058511513169485832;
    } else {
        c.s = 4;
        c.a21 = 2.0;
        c.a31 = 48.0 / 25.0;
        c.a32 = 6.0 / 25.0;
        c.c21 = -8.0;
        c.c31 = 372.0 / 25.0;
        c.c32 = 12.0 / 5.0;
        c.c41 = -112.0 / 125.0;
        c.c42 = -54.0 / 125.0;
        c.c43 = -2.0 / 5.0;
        c.b1 = 19.0 / 9.0;
        c.b2 = 1.0 / 2.0;
        c.b3 = 25.0 / 108.0;
        c.b4 = 125.0 / 108.0;
        c.e1 = 34.0 / 108.0;
        c.e2 = 7.0 / 36.0;
        c.e3 = 0.0;
        c.e4 = 125.0 / 108.0;
        c.gamma = 1.0 / 2.0;
        c.d1 = 1.0 / 2.0;
        c.d2 = -3.0 / 2.0;
        c.d3 = 605.0 / 250.0;
        c.d4 = 29.0 / 250.0;
    }
    return c;
}

// Stage coefficients by (uniform) stage index: a_ij of the derivative points
// (stages 1 and 2), c_ij of the right-hand sides and d_i.
__device__ __forceinline__ double ros_a(const RosCoeffs& C, int i, int j) {
    return i == 1 ? C.a21 : (j == 0 ? C.a31 : C.a32);
}
__device__ __forceinline__ double ros_c(const RosCoeffs& C, int i, int j) {
    if (i == 1) return C.c21;
    if (i == 2) return j == 0 ? C.c31 : C.c32;
    return j == 0 ? C.c41 : (j == 1 ? C.c42 : C.c43);
}
__device__ __forceinline__ double ros_d(const RosCoeffs& C, int i) {
    return i == 0 ? C.d1 : (i == 1 ? C.d2 : (i == 2 ? C.d3 : C.d4));
}

// I/(gamma dx) - J of the Jacobian in L.J, and its LU (gpuAdaptiveSolver.H:51-73).
template <int G, class W, int NB = 8>
__device__ __forceinline__ void shift_and_factor(const Grp<G>& g, const DevMech& M, const W& w, const WsLayout& L,
                                                 const RosCoeffs& C, double dx) {
    const int m = M.m;
    const int ld = L.ld;
    const int sc = G >= 32 ? L.k2 : L.vv;  // the row scalings; the stages are not written yet
    {
        GF_PH_BEGIN(g)
        shift_and_scale(g, w, L.J, ld, sc, m, 1.0 / (C.gamma * dx));
        GF_PH_END(g, PH_SHIFT)
    }
    // (the solves of 32 or more threads follow perm)
    lu_factor<G, false, NB>(g, w, L.J, ld, G >= 32 && m <= 128 ? -1 : L.piv, sc, L.vv, L.perm, m);
}

// One attempt solve(y0, dydx0, dx, y) of gpuRosenbrock12/23/34 (their
// solve(y0, dydx0, dx, y, buffer)); returns the normalised error
// (normaliseError.H:6-29; the p entry contributes 0). y0 is at y0_off, the
// candidate is written to yt_off.
// SAVE (the adjoint sweep): the caller has factored the step (L.J holds the
// LU); the stage points are kept at save_y2 / save_y3 and f at them at
// save_f2 / save_f3.
// F0 (the solve kernel): the attempt also evaluates the step's f(y0) into
// dydx0, through the stage loop's derivative call: one call site, a smaller
// instruction footprint. A retried step evaluates it again (the same value),
// which brings back the rate constants that the Jacobian reads: cheaper than a
// second copy of the rate code for the few retries (4 % of the attempts).
// Without F0 (SAVE) the caller provides dydx0 and the factors.
template <int G, class W, bool SAVE = false, bool F0 = false, int NB = 8>
__device__ __forceinline__ double ros_attempt(const Grp<G>& g, const DevMech& M, const W& w, const WsLayout& L, const RosCoeffs& C,
                              const OdeParams& o, int y0_off, int yt_off, double p, double dx, int save_y2 = -1,
                              int save_y3 = -1, int save_f2 = -1, int save_f3 = -1) {
    const int m = M.m;
    const int ld = L.ld;
    // stages: k_i solves (I/(gamma dx) - J) k_i = f_i + dx d_i dfdx + sum_j c_ij k_j / dx,
    // f_0 = f(y0), f_i = f(y0 + sum_j a_ij k_j) where the method takes a new
    // derivative (stage 1; stage 2 of Rosenbrock34), else the previous one.
    // One loop, so the solve and the derivative each have a single call site;
    // with F0, pass st = -1 evaluates f(y0) and factors the step.
#pragma unroll 1
    for (int st = F0 ? -1 : 0; st < C.s; ++st) {
        const bool new_f = st < 0 || st == 1 || (st == 2 && C.s == 4);
        int at = y0_off, out = L.dydx0;
        if (st > 0 && new_f) {
            // the stage point (kept at save_y2 / save_y3 when asked: the adjoint sweep)
            const int pt = !SAVE ? yt_off : (st == 1 ? save_y2 : (st == 2 ? save_y3 : yt_off));
            for (int i = g.lane; i < m; i += G) {
                double v = w[y0_off + i];
                for (int j = 0; j < st; ++j) v += ros_a(C, st, j) * w[L.k1 + j * L.ks + i];
                w[pt + i] = v;
            }
            at = pt;
            out = L.dydx;
        }
        Mix x;
        if (new_f) x = derivatives(g, M, w, L, at, p, out, st < 0);
        if constexpr (SAVE) {
            if (st > 0 && new_f) {
                const int fs = st == 1 ? save_f2 : save_f3;
                for (int i = g.lane; i < m; i += G) w[fs + i] = w[L.dydx + i];
            }
        }
        if constexpr (F0) {
            if (st < 0) {
                jacobian(g, M, w, L, y0_off, p, L.dydx0, x);
                shift_and_factor<G, W, NB>(g, M, w, L, C, dx);
                continue;
            }
        }
        const int ki = L.k1 + st * L.ks;
        const int src = st == 0 ? L.dydx0 : L.dydx;
        const double dd = dx * ros_d(C, st);
        for (int i = g.lane; i < m; i += G) {
            double v = w[src + i] + dd * w[L.dfdx + i];
            if (st > 0) {
                double cs = ros_c(C, st, 0) * w[L.k1 + i];
                for (int j = 1; j < st; ++j) cs += ros_c(C, st, j) * w[L.k1 + j * L.ks + i];
                v += cs / dx;
            }
            w[ki + i] = v;
        }
        lu_solve_any(g, w, L.J, ld, L.piv, L.perm, L.vv, m, ki);
    }
    double emax = 0.0;
    for (int i = g.lane; i < m; i += G) {
        const double y0i = w[y0_off + i];
        double yi, ei;
        if (C.s == 2) {
            yi = y0i + C.b1 * w[L.k1 + i] + C.b2 * w[L.k2 + i];
            ei = C.e1 * w[L.k1 + i] + C.e2 * w[L.k2 + i];
        } else if (C.s == 3) {
            yi = y0i + C.b1 * w[L.k1 + i] + C.b2 * w[L.k2 + i] + C.b3 * w[L.k3 + i];
            ei = C.e1 * w[L.k1 + i] + C.e2 * w[L.k2 + i] + C.e3 * w[L.k3 + i];
        } else {
            yi = y0i + C.b1 * w[L.k1 + i] + C.b2 * w[L.k2 + i] + C.b3 * w[L.k3 + i] + C.b4 * w[L.k4 + i];
            ei = C.e1 * w[L.k1 + i] + C.e2 * w[L.k2 + i] + C.e4 * w[L.k4 + i];
        }
        w[yt_off + i] = yi;
        const double tol = o.absTol + o.relTol * fmax(fabs(y0i), fabs(yi));
        emax = fmax(emax, fabs(ei) / tol);
    }
    const double err = g.fmax_(emax);
    g.sync();
    return err;
}

// ------------------------------------------------------------ cell driver

struct CellResult {
    int status;
    int accepted;
    int attempts;
    double dxTry;
};

// odeSolve (gpuODESolverBase.H:67-111) + adaptiveSolve (gpuAdaptiveSolver.H:83-134).
// The state lives at *y_off (swapped with *yt_off on acceptance). Returns a
// gf_cell_status. maxSteps exhausted: dxTry is left unchanged (the reference
// returns without writing it).
// REC (the adjoint's forward pass): each accepted step's start state and
// size are recorded at rec (rec_cap steps at most, rec_ld doubles each).
template <int G, class W, bool REC = false, int NB = 8>
__device__ __forceinline__ int ode_solve(const Grp<G>& g, const DevMech& M, const W& w, const WsLayout& L, const OdeParams& o,
                         const RosCoeffs& C, double xStart, double xEnd, int* y_off, int* yt_off, double p,
                         double* dxTry, int* accepted, int* attempts, double* rec = nullptr, int rec_cap = 0,
                         int rec_ld = 0) {
    double step_dxTry = *dxTry;
    bool last = false;
    double x = xStart;
    const double inc_threshold = pow(o.maxScale / o.safeScale, -1.0 / o.alphaInc);
    for (int nStep = 0; nStep < o.maxSteps; nStep++) {
        const double dxTry0 = step_dxTry;
        if ((x + step_dxTry - xEnd) * (x + step_dxTry - xStart) > 0) {
            last = true;
            step_dxTry = xEnd - x;
        }
        double dx = step_dxTry;
        double err = 0.0;
        int rejects = 0;
        do {
            GF_PH_BEGIN(g)
            // adaptiveSolve's derivatives call (gpuAdaptiveSolver.H:96), which
            // also leaves what the attempt's Jacobian needs, is inside the attempt
            err = ros_attempt<G, W, false, true, NB>(g, M, w, L, C, o, *y_off, *yt_off, p, dx);
            GF_PH_END(g, PH_ATTEMPT)
            ++*attempts;
            if (err > 1) {
                const double scale = fmax(o.safeScale * pow(err, -o.alphaDec), o.minScale);
                dx *= scale;
                // the reference traps here (gpuAdaptiveSolver.H:111-114); the cap
                // also ends the loop for step controls that never shrink dx
                if (dx < kVSmall || ++rejects > kMaxRejects) return GF_CELL_STEP_UNDERFLOW;
            }
        } while (err > 1.0);
        x += dx;
        if constexpr (REC) {
            // the accepted step's start state and size, for the adjoint sweep
            if (*accepted >= rec_cap) return GF_CELL_MAX_STEPS;
            double* r = rec + (size_t)(*accepted) * rec_ld;
            for (int i = g.lane; i < M.m; i += G) r[i] = w[*y_off + i];
            if (g.lane == 0) r[M.m] = dx;
        }
        const int t = *y_off;
        *y_off = *yt_off;
        *yt_off = t;
        if (err > inc_threshold) {
            step_dxTry = fmin(fmax(o.safeScale * pow(err, -o.alphaInc), o.minScale), o.maxScale) * dx;
        } else {
            step_dxTry = o.safeScale * o.maxScale * dx;
        }
        ++*accepted;
        if ((x - xEnd) * (xEnd - xStart) >= 0) {
            if (nStep > 0 && last) step_dxTry = dxTry0;
            *dxTry = step_dxTry;
            return GF_CELL_OK;
        }
    }
    return GF_CELL_MAX_STEPS;
}

// order-preserving key of a double for atomicMin
__device__ __forceinline__ unsigned long long dbl_key(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

// singleCellSolver::operator() (singleCellSolver.H:27-51) with the
// computeYNew / computeRR epilogue (gpuKernelEvaluator.cu:84-96) fused:
// RR, the min of deltaTChemNew before clamping, and the clamp.
template <int G, class W, bool REC = false, int NB = 8, int PAD = 0>
__device__ __forceinline__ void process_cell_body(const Grp<G>& g, const DevMech& M, const W& w, const LaunchArgs& a,
                                                  int cell) {
    const WsLayout L = solve_layout<G>(M.nS, M.nR, M.n_slots, M.n_tb, PAD);
    const int nS = M.nS, m = M.m;
    const double* yin = a.Y0 + (size_t)cell * a.ld_y;
    int y_off = L.y0, yt_off = L.yt;
    for (int i = g.lane; i < m; i += G) w[y_off + i] = yin[i];
    const double p = yin[nS + 1];
    const double T0 = yin[nS];
    const double dT = a.deltaT_cell ? a.deltaT_cell[cell] : a.deltaT;
    double dxTry = a.deltaTChem[cell];
    if (g.lane == 0) w[L.stage + M.n_slots] = 0.0;
    int status = GF_CELL_OK, accepted = 0, attempts = 0;
    g.sync();
    if (T0 > a.Treact) {
        const RosCoeffs C = ros_coeffs(a.ode.solver);
        double timeLeft = dT;
        while (timeLeft > kSmall) {
            const double dt = timeLeft;
            double* rec = REC ? a.traj + (size_t)cell * a.traj_cap * a.traj_ld : nullptr;
            const int st = ode_solve<G, W, REC, NB>(g, M, w, L, a.ode, C, 0.0, dt, &y_off, &yt_off, p, &dxTry, &accepted,
                                                &attempts, rec, a.traj_cap, a.traj_ld);
            if (st != GF_CELL_OK && status == GF_CELL_OK) status = st;
            if (st == GF_CELL_STEP_UNDERFLOW) break;
            int bad = 0;
            for (int i = g.lane; i < m; i += G) {
                const double v = w[y_off + i];
                if (!isfinite(v)) bad = 1;
                if (i < nS) w[y_off + i] = fmax(0.0, v);
            }
            if (g.any(bad) && status == GF_CELL_OK) status = GF_CELL_NONFINITE;
            g.sync();
            timeLeft -= dt;
        }
    } else {
        dxTry = dT;
        status = GF_CELL_SKIPPED;
    }
    // outputs
    if (a.Ynew) {
        double* yo = a.Ynew + (size_t)cell * a.ld_y;
        for (int i = g.lane; i < m; i += G) yo[i] = w[y_off + i];
        if (g.lane == 0) yo[nS + 1] = p;
    }
    if (a.RR) {
        const double rho = a.rho[cell];
        double* rr = a.RR + (size_t)cell * a.ld_rr;
        for (int i = g.lane; i < nS; i += G) rr[i] = rho * (w[y_off + i] - yin[i]) / dT;
    }
    if (g.lane == 0) {
        a.deltaTChem[cell] = fmin(dxTry, a.deltaTChemMax);
        if (a.status) a.status[cell] = status;
        if (a.counters) {
            a.counters[2 * cell] = accepted;
            a.counters[2 * cell + 1] = attempts;
        }
    }
    // per-cell aggregates: min over cells before clamping, counters (queue[1..4])
    if (g.lane == 0) {
        atomicMin(a.queue + 1, dbl_key(dxTry));
        atomicAdd(a.queue + 2, (unsigned long long)accepted);
        atomicAdd(a.queue + 3, (unsigned long long)attempts);
        if (status != GF_CELL_OK && status != GF_CELL_SKIPPED) atomicAdd(a.queue + 4, 1ull);
    }
    g.sync();
}

// The matrix sizes that a kernel is compiled for. MS > 0: the size MS, the only one
// that its caller launches it for; MS < 0: the range of sizes up to -MS (and above
// half of it, from 64 on); 0: any size.
//
// fix_size: whether M has a size of the kernel's, with M.m and M.nS as far as the
// compiler can know them: all of a size, or its range, which decides the rows per
// lane, the tiles and many loops and drops the code of the other sizes. The caller
// leaves the mechanism alone where this says no.
template <int MS>
__device__ __forceinline__ bool fix_size(DevMech& M) {
    if (MS > 0) {
        M.m = MS;
        M.nS = MS - 1;
    } else if (MS < 0) {
        constexpr int above = MS < -32 ? -MS / 2 : 1;
        int m = M.m;
        if (m <= above || m > -MS) return false;
        // what the test has just shown, on a copy that the compiler knows nothing
        // else about: it loses the range of the test itself on the way to the loops
        asm("" : "+r"(m));
        __builtin_assume(m <= -MS);
        __builtin_assume(m > above);
        M.m = m;
        M.nS = m - 1;
    }
    return true;
}
// the largest size of m's range, 0 beyond the ranges
__host__ __device__ constexpr int size_range(int m) { return m <= 32 ? 32 : (m <= 64 ? 64 : (m <= 128 ? 128 : 0)); }
__host__ __device__ constexpr int size_pad(int MS) { return MS < 0 ? -MS : 0; }

// process_cell_body with the LU panel width NB and the kernel's matrix sizes MS.
// False: not a mechanism of the kernel's sizes, nothing done.
template <int G, class W, bool REC = false, int NB = 8, int MS = 0, int PAD = 0>
__device__ __forceinline__ bool process_cell(const Grp<G>& g, const DevMech& M, const W& w, const LaunchArgs& a,
                                             int cell) {
    if constexpr (MS == 0) {
        process_cell_body<G, W, REC, NB, PAD>(g, M, w, a, cell);
    } else {
        DevMech Ms = M;
        if (!fix_size<MS>(Ms)) return false;
        process_cell_body<G, W, REC, NB, PAD>(g, Ms, w, a, cell);
    }
    return true;
}

}  // namespace gf
