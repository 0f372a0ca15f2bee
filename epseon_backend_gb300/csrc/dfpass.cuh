// dfpass.cuh -- pieces shared by the fast method's per-level passes
// (levelpass.cu, fragile.cu).
#pragma once

#include <math.h>

#include "common.cuh"
#include "dfloat.cuh"
#include "launch.h"

namespace epscu {

// Windows longer than a threshold take a CTA per level, the others a warp.  A
// warp per level costs the fewest instructions (no barriers, one scan), but a
// level's march is then 32 threads' and a batch of few levels leaves the GPU
// idle, so the threshold falls with the number of levels.  Solve times by
// threshold (Morse grids; the rule's choice in brackets):
//     levels x points     1024   4096  16384  65536
//        56 x 4096       [330]   398    401    411 us
//      3680 x 16384      1403  [1073]  1331   1330 us
//     14128 x 32768      6855   6281  [5233] 22050 us
//        37 x 65536     [1041]  1042   1721   3010 us
// DevBatch::long_window > 0 overrides it.
constexpr int kLongWindow = 65536;
constexpr int kLongWindowLevels = 45000;
constexpr int kMinLongWindow = 1024;

__host__ __device__ __forceinline__ int default_long_window(int total_levels) {
    int w = kMinLongWindow;
    while (w < kLongWindow && (long long)w * kLongWindowLevels < (long long)kLongWindow * total_levels) w <<= 1;
    return w;
}

// Windows longer than a second threshold take a cluster of four CTAs per level:
// 1024 threads on one march instead of 256, where the longest of a few levels'
// marches is what a solve waits for (280 levels on 2^20 points: 5.8 -> 2.0 ms
// of level passes; 37 levels on 65536 points, the solve 674 -> 487 us; 333
// levels on 65536 points with the threshold at 16384 instead of 32768: 888
// instead of 693 us, so it too rises with the number of levels).  Batches of
// more than kClusterPotentials potentials take CTAs, which are as fast or faster
// there unless each has very few levels.  The solve, us, clusters / CTAs, on
// Morse grids of 65536 points:
//     17 potentials,  958 levels   936 /  897      194 levels  1132 / 1024
//     24             1056          977 /  937      211         1214 / 1259
//     32             1591         1285 / 1210      318          951 / 1215
//     48             2516         1708 / 1639      515         1410 / 1392
constexpr int kMinClusterWindow = 16384;
constexpr int kClusterLevels = 256;
constexpr int kClusterPotentials = 16;

__host__ __device__ __forceinline__ int default_cluster_window(int total_levels) {
    long long w = kMinClusterWindow;
    while (w < (1ll << 30) && w * kClusterLevels < (long long)kMinClusterWindow * total_levels) w <<= 1;
    return (int)w;
}

// The threshold of the fragile levels' CTA passes (fragile.cu), which cost ~3x
// the point-updates of a lane's but cut its latency ~80x: 8192 points above 3e4
// levels, proportionally less below, never under 1024.  The solve, us, by
// threshold (uneven grids; the rule's choice in brackets):
//     levels               1024    2048    4096    8192    16384
//       705 (16 grids)    [569]             560              559
//      2829 (48)          [999]            1325             1304
//     11630 (256)         2666   [2732]    3153             6815
//     25362 (512)         6170            [7135]           10150
//     93060 (2048)       13016            12919  [14250]   15240
constexpr int kFragileLongWindow = 8192;
constexpr int kFragileLongLevels = 60000;
constexpr int kFragileMinLongWindow = 1024;

__host__ __device__ __forceinline__ int default_fragile_window(int total_levels) {
    int w = kFragileMinLongWindow;
    while (w < kFragileLongWindow && (long long)w * kFragileLongLevels < (long long)kFragileLongWindow * total_levels)
        w <<= 1;
    return w;
}

// Levels that share the scan's bracket with a neighbour, or whose brackets show
// them this close to one (Hartree), are fragile (fragile.cu).
constexpr double kFragileGap = 2e-5;

// the level's final passes ran on a CTA
__device__ __forceinline__ bool is_long(const LevelWork& w) { return (w.status & EPSCU_STATUS_LONG) != 0; }

// match points stay inside the level's window, off its two end points
__device__ __forceinline__ int clamp_k(const LevelWork& w, int k) { return max(w.j0 + 1, min(k, w.j1 - 1)); }

__device__ __forceinline__ dfl energy_df(const PotMeta& m, double E) {
    return df_from_double(__dmul_rn(m.a, E));
}

struct PassDF {
    double dE, gamma, sum;
    double pk_out, pk_in;
    int ex_out, ex_in;
    int nodes, count;
    int peak_i, peak_log2;
};

// Write the normalisation constants of pass r (match point k) into w.
__device__ __forceinline__ void finalize_df(const PotMeta& m, LevelWork& w, const PassDF& r, int k) {
    double ck = 1.0 / sqrt(m.h * r.sum);
    if (r.pk_out < 0.0) ck = -ck;  // psi > 0 next to the inner wall
    w.k = k;
    w.ck = ck;
    w.norm_k_out = ck / r.pk_out;
    w.norm_k_in = ck / r.pk_in;
    w.ex_out = r.ex_out;
    w.ex_in = r.ex_in;
    w.dE = r.dE;
    w.nodes = r.nodes;
    w.status &= ~EPSCU_STATUS_NOTFOUND;
    if (!isfinite(r.dE) || !isfinite(ck)) w.status |= EPSCU_STATUS_NONFINITE;
    if (r.nodes != w.v && !(m.status & EPSCU_STATUS_UNDER)) w.status |= EPSCU_STATUS_NOTFOUND;
}

// a converged level whose final pass disagrees (node count, or a Cooley
// correction far above the energy's accuracy) was matched at a poor point
__device__ __forceinline__ bool suspicious(const PotMeta& m, const LevelWork& w, int nodes, double dE) {
    return (nodes != w.v && !(m.status & EPSCU_STATUS_UNDER)) || !(fabs(dE) <= 1e-11 * fmax(1.0, fabs(w.E)));
}

// psi is only as accurate as the energy it is computed at (error ~ |E - E_v|
// over the gap to the next level, 1e-5 Eh near dissociation): a norm pass
// whose Cooley correction is above this is redone once at E + dE
__device__ __forceinline__ bool redo_norm(const LevelWork& w, const PassDF& r) {
    return r.nodes == w.v && isfinite(r.dE) && fabs(r.dE) > 1e-13 * fmax(1.0, fabs(w.E)) && fabs(r.dE) < 1e-8;
}

// The norm passes store psi-hat = (h + l) 2^X in the 8 bytes of each window
// point of the level's row as a tagged float pair: X = 64 r + x
// with x in [-32, 31], the pair (h 2^x, l 2^x) in floats, and r in the five
// low bits of the second float (which only cost l bits 2^-43 below h).  X can
// reach hundreds (a window edge deep in a steep wall lies far below the peak);
// |X| is clamped to the tag's range of about +-1000, beyond any value that
// survives the normalisation.
struct PsiTag {
    float sc;  // 2^x
    int r;     // the tag
};

__device__ __forceinline__ PsiTag psi_tag(int X) {
    X = max(-1000, min(X, 990));
    const int r = (X + 32) >> 6;  // floor((X + 32) / 64): x = X - 64 r in [-32, 31]
    return {fpow2(X - 64 * r), r};
}

__device__ __forceinline__ float2 psi_pair(dfl psi, PsiTag t) {
    const float l = __fmul_rn(psi.l, t.sc);
    const uint32_t lt = (__float_as_uint(l) & ~31u) | ((uint32_t)t.r & 31u);
    return make_float2(__fmul_rn(psi.h, t.sc), __uint_as_float(lt));
}

__device__ __forceinline__ void store_psi_pair(double* __restrict__ row, int i, dfl psi, PsiTag t) {
    reinterpret_cast<float2*>(row)[i] = psi_pair(psi, t);
}

// the stored pair back: (h, l) and the tag r (psi-hat = (h + l) 2^(64 r))
__device__ __forceinline__ dfl load_psi_pair(float2 v, int& r) {
    const uint32_t lt = __float_as_uint(v.y);
    r = ((int)(lt << 27)) >> 27;  // sign-extended five bits
    return {v.x, __uint_as_float(lt & ~31u)};
}

// the level's psi row, or nullptr (no psi requested, or the psi buffer
// overflowed: the level setup raised the capacity error)
__device__ __forceinline__ double* psi_row(const DevBatch& b, const PotMeta& m, const LevelWork& w) {
    if (!b.psi || b.hdr->error) return nullptr;
    return b.psi + m.psi_off + (int64_t)(w.v - b.min_level) * m.N;
}

__device__ __forceinline__ bool no_result(const LevelWork& w) {
    return (w.status & (EPSCU_STATUS_NOTFOUND | EPSCU_STATUS_CANCELLED | EPSCU_STATUS_NONFINITE)) != 0;
}

}  // namespace epscu
