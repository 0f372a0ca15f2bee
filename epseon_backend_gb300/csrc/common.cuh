// common.cuh -- device-side data layout and arithmetic shared by the solver
// kernels of libepseon_cuda (sm_103a).
//
// The discrete problem is the one the FP64 oracle restates (Numerov on a
// uniform grid with E-independent Dirichlet cut-offs, twisted Sturm counts):
//   a = mu h^2 / 6,  T_i = aE - W_i with W_i = a V_i,  f_i = 1 + T_i,
//   g_i = 2 - 10 T_i,  projective step (A, B) <- (g A - f B, f A).
// Every FP64 expression on the count/bisection path is written with explicit
// __dadd_rn/__dmul_rn/__fma_rn so that nvcc cannot contract it differently
// from the oracle's explicit fma() calls.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "epscu.h"

// status bits kept per potential / level (public values from epscu.h)
#define EPSCU_STATUS_MAXITER EPSCU_LEVEL_MAXITER
#define EPSCU_STATUS_NONFINITE EPSCU_LEVEL_NONFINITE
#define EPSCU_STATUS_UNDER EPSCU_LEVEL_UNDER_RESOLVED
#define EPSCU_STATUS_CANCELLED EPSCU_LEVEL_CANCELLED
#define EPSCU_STATUS_NOTFOUND EPSCU_LEVEL_NOT_FOUND
#define EPSCU_STATUS_BAD EPSCU_LEVEL_BAD_INPUT

namespace epscu {

// the fast method's level lists (LevelWork::bucket / kBuckets), each ordered by
// window-length classes (quarter octaves)
enum { kListWarp = 0, kListLong, kListFragile, kListFragileLong, kListCluster, kLists };
constexpr int kBuckets = 64;
constexpr int kRenorm = 32;  // renormalise the projective state every kRenorm steps

// Per-potential constants, written by the prepare kernel.
struct PotMeta {
    double r_min, r_max, mu, e_cap;  // inputs
    double h, a, e_lo, delta;        // derived (same formulas as the oracle)
    int64_t off;                     // first element in V64 / W64
    int64_t offf;                    // first element in Wf2 (tile aligned)
    int64_t psi_off;                 // first element of this potential's psi rows
    int32_t N, i0, i1, k_scan;
    int32_t n_bisect, n_trial;
    int32_t n_total, n_out;
    int32_t level_base, status;
    int32_t prep_done;               // tiles of the prepare kernel that have finished (0 between solves)
    int32_t pad1;
};

// One level slot of the refinement stages.
struct LevelWork {
    double lo, hi;      // bracket (count(lo) <= v < count(hi))
    double lo0, hi0;    // the scan bracket
    double E;           // current energy
    double dE;          // last correction (error estimate)
    double norm_k_out;  // write-pass constants: psi scale on the outward side
    double norm_k_in;   //   and on the inward side
    double ck;          // psi at the match index
    int32_t ex_out, ex_in;  // binary exponents of the two side constants
    int32_t p, v;
    int32_t nodes, status;
    int32_t k;          // match index used by the write pass
    int32_t iters;
    int32_t j0, j1;     // grid window of the level's passes ([i0, i1] unless narrowed
                        // by the decay window of the fast method)
    int32_t bucket, rank;  // fast method: place in the order of falling window length
    int32_t n_in_bracket;  // levels the scan counted inside the scan bracket
    int32_t pad1;
};

// Global counters and flags of one solve (device memory).
struct Header {
    int32_t total_levels;
    int32_t queue_scan;
    int32_t queue_refine;
    int32_t queue_polish;
    int32_t error;          // first device-side error code (0 = none)
    int32_t fallbacks;      // levels that needed the bisection fallback
    int32_t n_units;        // warp work units (<= 32 levels of one potential)
    int32_t n_twist;        // levels handed to the twist-index search
    int32_t queue[16];      // work-queue heads of the per-level kernels
    int32_t n_long;         // levels whose window takes the CTA-per-level passes
    int32_t n_warp;         // levels whose window takes the warp-per-level passes
    int32_t n_cluster;      // levels whose window takes the passes of a cluster of CTAs
    int32_t stopped;        // a kernel has seen the host's cancel flag set
    int32_t n_under;        // potentials on under_list
    int32_t n_fragile;       // fragile levels on lanes, those with long windows,
    int32_t n_fragile_long;
    int32_t n_fragile_fall;  //   those the lane Newton handed over,
    int32_t n_fragile_twist; //   those for the twist-index search
    int32_t bis_items_n;    // bisection round: (potential, chunk) items listed
    int32_t bis_items_q;    //   and the work-queue head over them
    int32_t n_redo;         // norm passes redone at E + dE
    unsigned long long scan_updates;    // point-updates the windowed FP32 scan performed
    unsigned long long refine_updates;  // point-updates of the FP32 refinement passes
    unsigned long long df_updates;      // point-updates of the double-float passes
    long long psi_total;                // psi doubles of the batch (level setup)
    unsigned long long refine_max_updates;  // largest per-level FP32 point-updates
    unsigned long long df_max_updates;      // largest per-level double-float point-updates
    int32_t refine_max_iters;               // most FP32 passes of one level
    int32_t pad_hdr;
    int32_t hist[kLists * kBuckets];        // levels by list and window length
    unsigned long long long32_updates;      // CTA levels: FP32 pass point-updates
    unsigned long long longdf_updates;      //   and double-float pass point-updates
    unsigned long long psi_zero_points;     // psi points zeroed (outside the windows)
    unsigned long long psi_window_points;   // window points written
};

// queue ids of the per-level kernels
enum { kQBisect64 = 0, kQNorm64, kQWrite64, kQWarpLevels, kQLongLevels, kQRepair, kQWarpRewrite, kQLongRewrite,
       kQFragileLanes, kQFragileLong, kQFragileRepair, kQFragileRewrite,
       kQCountStride, kQCountListed, kQClusterLevels, kQClusterRewrite };

// internal level flags (not reported: gather keeps the public bits only)
// the level's final passes ran one CTA per level
#define EPSCU_STATUS_LONG 0x20000
// ... and those a cluster of CTAs
#define EPSCU_STATUS_CLUSTER 0x80000
// (fragile.cu) the lane Newton handed the level over: its refinement, norm pass
// and rewrite run on a CTA (the lane passes skip it)
#define EPSCU_STATUS_FALLBACK 0x10000
// (potential) a point inside the cut-offs lies above them: 1 + T can be small or
// negative there, and a fast pass renormalises after every point
#define EPSCU_STATUS_STEEP 0x40000
// (potential) ... so far above that f = 1 + T is negative there at some energy of
// the range.  A lane pass counts the sign changes of u times the product of the
// f before it, which are the levels below E only while u changes sign at every
// such point (all but ~0.1% of the energies, those next to the levels of the
// well on one side: up to 2 off), so the scans count these potentials point by
// point and their close levels take the group passes
#define EPSCU_STATUS_BELOW 0x100000
#define EPSCU_STATUS_PUBLIC 0xffff
// spacing of the samples of the twist-index search
constexpr int kTwistSample = 64;

// ---------------------------------------------------------------- FP64 helpers

// One divide-free projective Numerov step (identical to the oracle's
// numerov_step): state (A, B) ~ s (u_i, u_{i-1}) -> s f_i (u_{i+1}, u_i).
__device__ __forceinline__ void step64(double aE, double w, double& A, double& B) {
    const double T = __dsub_rn(aE, w);
    const double f = __dadd_rn(1.0, T);
    const double g = __fma_rn(-10.0, T, 2.0);
    const double An = __fma_rn(g, A, -__dmul_rn(f, B));
    B = __dmul_rn(f, A);
    A = An;
}

// x < 0 on the integer pipes: a FP64 comparison costs what a FP64 multiply-add
// does (64 cycles of its SM quarter's pipe a warp on GB300).  Above -0, up to
// -inf: a NaN, which an overflowing march leaves with its sign bit set, is not.
__device__ __forceinline__ bool negative(double x) {
    return (unsigned long long)__double_as_longlong(x) - 0x8000000000000001ull < 0x7ff0000000000000ull;
}

// frexp-style exponent of |m| (m = f 2^e, f in [0.5, 1)) for finite normal m.
__device__ __forceinline__ int exp_of(double m) {
    const int hi = __double2hiint(m);
    return ((hi >> 20) & 0x7ff) - 1022;
}

// Exact power of two 2^e for |e| < 1000.
__device__ __forceinline__ double pow2(int e) { return __hiloint2double((1023 + e) << 20, 0); }

// Rescale (x, y) by the power of two that brings max(|x|,|y|) into [0.5, 1);
// returns the exponent removed (0 when the pair is zero or not finite).
__device__ __forceinline__ int renorm_pair(double& x, double& y) {
    const double m = fmax(fabs(x), fabs(y));
    if (!(m > 0.0) || !isfinite(m)) return 0;
    const int e = exp_of(m);
    if (e > 1000 || e < -1000) return 0;
    const double s = pow2(-e);
    x *= s;
    y *= s;
    return e;
}

// E_j = E_lo + (j+1) delta (two roundings, as in the oracle).
__device__ __forceinline__ double trial_energy(const PotMeta& m, int j) {
    return __dadd_rn(m.e_lo, __dmul_rn((double)(j + 1), m.delta));
}

// bisection scan: the throughput scan on every kBisectCoarse-th trial
// energy, then counts inside the coarse cells whose end counts differ
constexpr int kBisectCoarse = 16;
// parts a cell with two or more levels is cut into per round (a power of two
// dividing kBisectCoarse; equal to it: one round, a count at every trial
// energy of the cell)
constexpr int kBisectSplit = 16;
// parts a coarse cell that holds exactly one level is cut into (a power of
// two dividing kBisectCoarse; 1: no count inside, the level's bracket is the
// whole cell, which isolates it already)
constexpr int kBisectSingle = 4;
// batches of at least this many potentials scan with a lane per energy (scan.cu;
// smaller ones have too few energies to cover a lane's march of its window),
// smaller ones with a group per energy (groupscan.cu).  The solve of uneven grids
// of 2048 to 65536 points, 8192 energies, ms, lanes / groups: 256 potentials 4.5 /
// 3.2, 384 4.8 / 3.8, 512 5.2 / 4.5, 700 7.5 / 7.0, 1024 7.7 / 7.9, 2048 16.3 /
// 17.8; of 2048 to 8192 points, 1024 energies: 256 2.8 / 3.0, 512 5.15 / 5.09,
// 1024 11.2 / 11.2, 2048 13.5 / 14.1
constexpr int kBisectMinPotentials = 512;

// e-folds of decay at the ends of the fast method's windows: e^-36 = 2.3e-16,
// psi at the cut is below FP64 resolution relative to its value at the
// turning point (dense eigen-decompositions of the discrete problem keep
// every level to 1e-12 and every eigenvector to 1e-10 in L2 down to 26)
constexpr float kWindowDecay = 36.0f;
// trial energies per entry of the scan's window table
constexpr int kScanWinBlock = 128;

// One side of a twisted Sturm count: the projective state from point `from` up
// (dir 1) or down (dir -1) to the twist index k, and its sign changes
// (identical arithmetic to the oracle's eo_count).
__device__ __forceinline__ int count_side64(const double* __restrict__ W, double aE, int from, int k, int dir, double& A,
                                            double& B) {
    A = 1.0;
    B = 0.0;
    int nodes = 0, s = 0;
    bool neg = false;
    // step64's operations, those of the next point (which do not depend on the
    // state) between this point's: the chain waits for ~2 FP64 latencies a
    // step instead of 4
    double T = __dsub_rn(aE, __ldg(W + from));
    double f = __dadd_rn(1.0, T), g = __fma_rn(-10.0, T, 2.0);
    for (int i = from; i != k; i += dir) {
        const double Tn = __dsub_rn(aE, __ldg(W + i + dir));  // (up to k: inside the grid)
        const double fB = __dmul_rn(f, B);
        const double Bn = __dmul_rn(f, A);
        const double An = __fma_rn(g, A, -fB);
        f = __dadd_rn(1.0, Tn);
        g = __fma_rn(-10.0, Tn, 2.0);
        A = An;
        B = Bn;
        const bool n = negative(A);
        nodes += n != neg;
        neg = n;
        if (++s == kRenorm) {
            s = 0;
            renorm_pair(A, B);
        }
    }
    return nodes;
}

// The count from the two sides' states at k.
__device__ __forceinline__ int count_join64(double aE, double wk, double A, double B, double C, double D) {
    const double Tk = __dsub_rn(aE, wk);
    const double fk = __dadd_rn(1.0, Tk);
    const double gk = __fma_rn(-10.0, Tk, 2.0);
    const double AC = __dmul_rn(A, C);
    const double num = __fma_rn(gk, AC, -__dmul_rn(fk, __fma_rn(B, C, __dmul_rn(D, A))));
    return (num < 0.0) != (AC < 0.0);
}

// Twisted Sturm count at E with twist index k.
__device__ __forceinline__ int count64(const PotMeta& m, const double* __restrict__ W, double E, int k) {
    const double aE = __dmul_rn(m.a, E);
    double A, B, C, D;
    int nodes = count_side64(W, aE, m.i0, k, +1, A, B);
    nodes += count_side64(W, aE, m.i1, k, -1, C, D);
    return nodes + count_join64(aE, __ldg(W + k), A, B, C, D);
}

// 1/f for 2^-100 <= |f| <= 2^100, of either sign: FP32 reciprocal refined by two
// FP64 Newton steps (relative error at the FP64 rounding level).  The two
// conversions run on the integer pipes (exact, and the same rounding): the
// magnitude there and back, the sign put into the double (the bits above the
// float's exponent fall off the first shift).
__device__ __forceinline__ double recip64_normal(double f) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(f);
    const uint32_t dropped = (uint32_t)u & 0x1fffffffu;
    uint32_t b = (uint32_t)((u >> 29) - (896ull << 23));  // truncated to a float's bits
    b += dropped > 0x10000000u || (dropped == 0x10000000u && (b & 1u));
    const uint32_t x = __float_as_uint(__frcp_rn(__uint_as_float(b)));
    double r = __hiloint2double((int)(((x >> 3) + (896u << 20)) | ((uint32_t)(u >> 32) & 0x80000000u)), (int)(x << 29));
    r = __fma_rn(r, __fma_rn(-f, r, 1.0), r);
    r = __fma_rn(r, __fma_rn(-f, r, 1.0), r);
    return r;
}

// ... for any f: the conversions themselves outside that range
__device__ __forceinline__ double recip64(double f) {
    if ((((uint32_t)__double2hiint(f) >> 20) & 0x7ffu) - 923u <= 200u) return recip64_normal(f);
    double r = (double)__frcp_rn((float)f);
    r = __fma_rn(r, __fma_rn(-f, r, 1.0), r);
    r = __fma_rn(r, __fma_rn(-f, r, 1.0), r);
    return r;
}

}  // namespace epscu
