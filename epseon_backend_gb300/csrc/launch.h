// launch.h -- host-side launchers of the libepseon_cuda kernels (one per
// translation unit), called by the orchestration in epscu.cu.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "common.cuh"

namespace epscu {

// the prepare kernel's tiles (a divisor of the tile the padded offsets align to)
constexpr int kPrepTile = 2048;
struct PrepTile {
    unsigned long long kall, kin, kmax;  // images of the minimum, the minimum over the interior, the maximum of V
    int32_t iin;                         // first interior point of the minimum
    int32_t bad;                         // inf or NaN among the points
};

struct DevBatch {
    int32_t n;                 // potentials
    PotMeta* meta;             // [n]
    const double* V64;         // concatenated potentials
    double* W64;               // a V (FP64)
    // minima over 32-point blocks, at offf / 32 + block: of V (order-preserving
    // images), of V from the block's start to i1, from i0 to its end, and of W
    // rounded down (the last two for the fast method, else nullptr)
    unsigned long long* Bkey;
    double* Bsuf;
    double* Bpre;
    float* Bmin;
    PrepTile* prep;            // [prep_tiles] summaries of the prepare kernel's tiles
    int32_t prep_tiles;        // padded points / kPrepTile
    float2* Wf2;               // a V as (hi, lo) floats, tile-aligned per potential
    int32_t* counts;           // [n * n_trial]
    float* gam;                // [n * n_trial] the scan's matching function f_k gamma_k at the counted trial
                               // energies (fast method: the refinement's first energy), or nullptr
    LevelWork* levels;         // [max_levels]
    int32_t* fallback_list;    // [max_levels] slots handed to the repair kernel
    int2* units;               // [max_units] (first slot, count) per warp work unit
    int32_t max_units;
    int32_t* twist_list;       // [max_twist] slots for the twist-index search
    double* twist_scratch;     // [max_twist * twist_stride] sampled outward ratios
    int32_t max_twist, twist_stride;
    int32_t max_levels;        // capacity of levels (n * level_capacity)
    int32_t level_capacity;    // slots per potential
    Header* hdr;
    int32_t* order;            // [n] potentials by decreasing cost
    int2* scan_win;            // [n * ceil(n_trial / kScanWinBlock)] scan windows, or nullptr (full grid)
    int32_t* cluster_list;     // [max_levels] slots with the longest windows (a cluster of CTAs each), or nullptr:
                               // none can be that long
    int32_t* long_list;        // [max_levels] slots with long windows (CTA-per-level passes), or nullptr
    int32_t* fragile_list;     // [max_levels] fragile levels (fragile.cu): a lane each, or nullptr
    int32_t* fragile_long;     // [max_levels]   long windows, a CTA each
    int32_t* fragile_fall;     // [max_levels]   handed over by the lane Newton
    int32_t* fragile_twist;    // [max_twist]    for the twist-index search
    int32_t* warp_list;        // [max_levels] the other slots (warp-per-level passes), or nullptr
    int32_t* bis_list;         // [n * n_trial] trial indices of the bisection scan's count round, or
                               // nullptr (every trial energy scanned)
    int32_t* bis_n;            // [n] entries of bis_list per potential
    int32_t* under_list;       // [n] group scan: the under-resolved potentials, scanned in full by lanes; nullptr:
                               // every potential scans alike
    int2* bis_items;           // [max_bis_items] (potential, first entry) chunks of a bisection round
    int32_t max_bis_items;
    double* psi;               // compact wavefunctions or nullptr
    int64_t psi_capacity;
    volatile int32_t* cancel;  // host-mapped cancel flag (device pointer) or nullptr
    int32_t n_trial;
    int32_t min_level, max_level;
    int32_t max_N;             // longest grid of the batch
    int32_t long_window;       // window length above which a level takes the CTA passes
    int32_t wait_polls;        // polls of a bounded wait on a staged scan tile (0: kWaitPolls)
    int32_t max_iter;          // cap on FP32 refinement passes (0: 48; fallback passes: twice it)
    double tol;
};

// Largest i in [i0, i1] with V_i <= E; k_scan when there is none: the last
// block whose suffix minimum is at or below E, then its points.
__device__ __forceinline__ int match_index(const PotMeta& m, const DevBatch& b, double E) {
    const double* S = b.Bsuf + m.offf / 32;
    int lo = m.i0 >> 5, hi = m.i1 >> 5;  // invariant: S[lo] <= E
    if (!(S[lo] <= E)) return m.k_scan;
    while (lo < hi) {
        const int mid = lo + (hi - lo + 1) / 2;
        if (S[mid] <= E) lo = mid;
        else hi = mid - 1;
    }
    const double* V = b.V64 + m.off;
    int i = min((lo << 5) + 31, m.i1);
    for (const int first = max(lo << 5, m.i0); i > first && !(V[i] <= E);) --i;
    return i;
}

constexpr int kWaitPolls = 1 << 22;       // default bound of the TMA scan's mbarrier waits
constexpr int kRefineMaxIter = 48;        // default cap on a level's FP32 refinement passes
__device__ __forceinline__ int refine_cap(const DevBatch& b) { return b.max_iter > 0 ? b.max_iter : kRefineMaxIter; }
// double-float fallback passes (bisection from the widened scan bracket)
__device__ __forceinline__ int fallback_cap(const DevBatch& b) { return 2 * refine_cap(b); }

// Whether the host asked to stop.  A read of the host-mapped flag goes over the
// host link, ~2 us each and slower the more warps read at once (a scan that
// read it per energy spent half its time there, 2432 warps without work took
// 19 us to find that out), so only the threads that poll read it and tell the
// others through the header.
__device__ __forceinline__ bool stop_asked(const DevBatch& b, bool poll) {
    volatile int32_t* stopped = &b.hdr->stopped;
    if (*stopped) return true;
    if (!poll || !b.cancel || !*b.cancel) return false;
    *stopped = 1;
    return true;
}

// prepare.cu
void launch_prepare(const DevBatch& b, cudaStream_t s);
void launch_level_setup(const DevBatch& b, cudaStream_t s);
void launch_window(const DevBatch& b, int sm_count, cudaStream_t s);
void launch_scan_window(const DevBatch& b, int sm_count, cudaStream_t s);

// tabulate.cu (knot_scratch: 4 n_knots doubles per potential; 6 for the adjoint)
constexpr int kTabTile = 2048;  // points per CTA; tiles[p]: the first tile of potential p
void launch_tabulate(int32_t n, const int32_t* kind, const double* params, const int64_t* offsets, const int32_t* N,
                     const double* r_min, const double* r_max, const int32_t* tiles, int32_t n_tiles, int32_t n_knots,
                     bool splines, double* knot_scratch, double* V, cudaStream_t s);

void launch_tabulate_adjoint(int32_t n, const int32_t* kind, const double* params, const int64_t* offsets,
                             const int32_t* N, const double* r_min, const double* r_max, int32_t n_knots,
                             double* knot_scratch, const double* gV, double* gP, cudaStream_t s);

// scan.cu
void launch_scan64(const DevBatch& b, cudaStream_t s);
struct ScanShape {
    int threads;      // threads per CTA (energies per CTA = threads)
    int tile;         // floats2 per TMA stage
    int stages;
    int ctas_per_sm;  // persistent grid = sm_count * ctas_per_sm
};
void launch_scan32(const DevBatch& b, const ScanShape& shape, int sm_count, cudaStream_t s, int stride = 1);
void launch_scan_under(const DevBatch& b, const ScanShape& shape, int sm_count, cudaStream_t s);
void launch_group_scan(const DevBatch& b, int sm_count, cudaStream_t s);
void launch_bisect_scan(const DevBatch& b, const ScanShape& shape, int sm_count, cudaStream_t s);
int64_t bisect_max_items(int n, int n_trial);  // capacity of DevBatch::bis_items
int scan32_max_tile();
void scan32_set_attributes();

// groupscan.cu
void groupscan_set_attributes();
void launch_count_stride(const DevBatch& b, int stride, int sm_count, cudaStream_t s);
void launch_count_listed(const DevBatch& b, int chunk, int sm_count, cudaStream_t s);

// levels.cu
void launch_bisect64(const DevBatch& b, int sm_count, cudaStream_t s);
void launch_norm64(const DevBatch& b, int sm_count, cudaStream_t s);
void launch_write64(const DevBatch& b, int sm_count, cudaStream_t s);
void launch_gather(const DevBatch& b, int32_t* n_total, int32_t* n_out, double* energy, int32_t* nodes,
                   int32_t* status, double* err_est, int apply_dE, cudaStream_t s);

void launch_twist64(const DevBatch& b, int sm_count, cudaStream_t s);

// levelpass.cu
void levels_set_attributes();
void launch_order_levels(const DevBatch& b, int sm_count, cudaStream_t s);
void launch_levels(const DevBatch& b, int sm_count, cudaStream_t s);
void launch_repair(const DevBatch& b, int sm_count, cudaStream_t s);
void launch_rewrite(const DevBatch& b, int sm_count, cudaStream_t s);

// fragile.cu
void launch_fragile(const DevBatch& b, int sm_count, cudaStream_t s);
void launch_fragile_repair(const DevBatch& b, int sm_count, cudaStream_t s);
void launch_fragile_rewrite(const DevBatch& b, int sm_count, cudaStream_t s);

// adjoint.cu
// points per CTA of the adjoint (one thread each)
constexpr int kAdjointPoints = 256;
void launch_adjoint(const DevBatch& b, const double* dL_dE, double* dL_dV, const int64_t* offsets_dev,
                    const int32_t* tiles_dev, int32_t n_tiles, cudaStream_t s);

void launch_adjoint_explicit(int32_t n, int32_t cap, int32_t max_N, const int64_t* offsets, const int32_t* N,
                             const double* h, const int32_t* n_out, const int64_t* psi_off, const double* psi,
                             const double* gE, double* gV, cudaStream_t s);

// epscu.cu: the calling thread's message for epscu_last_error()
void set_last_error(const std::string& msg);

// peaks.cu
void measure_fma_peaks(int sm_count, double* fp32_tflops, double* fp64_tflops);

}  // namespace epscu
