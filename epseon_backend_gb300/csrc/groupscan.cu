// groupscan.cu -- Sturm counts at trial energies, a group of threads per energy
// (the FP32 phase-1 pass of grouppass.cuh without its sums): a warp, or a CTA
// for grids longer than kScanCtaPoints.
//
// A lane per energy (scan.cu) marches the whole window as one chain, ~25 cycles
// a point: with few potentials the scan lasts as long as its longest window
// whatever the number of energies.  A group's chain is 32 or 256 times shorter,
// so batches under kBisectMinPotentials potentials count every kBisectCoarse-th
// trial energy and then inside the cells that hold a level (the bisection
// scan's plan) with these kernels, both rounds together against the lane scan
// of every energy:
//     1 x 2^20 points, 65536 energies      0.57 ms   12.8 ms
//     256 x 2048..65536 points, 8192       0.68 ms    2.1 ms
//     64 x 16384 points, 8192              0.21 ms    0.59 ms
//     48 x 4096..32768 points, 4096        0.14 ms    0.55 ms
//     24 x 6000 points                     0.09 ms    0.16 ms
//     1 x 10007 points, 1024 (all of them) 0.030 ms   0.133 ms  (static_scan.cu)
// Larger batches keep the lane kernels, which their many energies fill (a warp
// pass costs about twice a lane march's instructions per point), and so do
// under-resolved potentials (fragile.cu), in full and beside these kernels: the
// first energies of their levels' passes come from it.
//
// What bounds it: with a warp per energy 37% of the issue slots were used while
// every energy read the host's cancel flag; now it is the issue rate (0.76 per
// cycle on the long grid; ~30 instructions a point-update, of which 14 are the
// recurrence's).
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "dfpass.cuh"
#include "grouppass.cuh"
#include "launch.h"

namespace epscu {

namespace {

// A CTA's pass costs a barrier per step of its scan: 1024 energies on 10007
// points took 104 us with a CTA each and 30 us with a warp each, the two rounds
// of one 4096-point grid 46 us and 19 us; on 2^20 points a warp's march
// is 32768 steps long and the CTA's the shorter.
constexpr int kScanCtaPoints = 65536;
constexpr int kScanWarps = 8;

template <int NW>
struct ScanCta {
    static constexpr int kThreads = NW == 1 ? 128 : 32 * NW;
    static constexpr int kPerSm = NW == 1 ? 6 : 3;
};

// The count at trial energy j of potential p on the window [j0, j1] with the
// scan's twist index; with b.gam the matching function too (its scale is the
// potential's).
template <int NW>
__device__ __forceinline__ void count_at(const Grp<NW>& G, const DevBatch& b, int p, int j, int j0, int j1,
                                         Shared32<NW>& sh) {
    const PotMeta& m = b.meta[p];
    const float2* Wf = b.Wf2 + m.offf;
    const int k = max(j0 + 1, min(m.k_scan, j1 - 1));
    const dfl aE = df_from_double(__dmul_rn(m.a, trial_energy(m, j)));
    const Pass32 r = pass32<NW, false>(G, Wf, aE, j0, j1, k, (m.status & EPSCU_STATUS_STEEP) != 0, sh);
    if (G.leader()) {
        b.counts[(int64_t)p * b.n_trial + j] = r.count;
        if (b.gam) {
            const float2 w = __ldg(Wf + k);
            b.gam[(int64_t)p * b.n_trial + j] = r.g * (1.0f + ((aE.h - w.x) + (aE.l - w.y)));
        }
    }
}

// the scan window of trial energy j's block, with the twist index inside
__device__ __forceinline__ int2 scan_window(const DevBatch& b, int p, int j) {
    const PotMeta& m = b.meta[p];
    int2 w = make_int2(m.i0, m.i1);
    if (b.scan_win) {
        const int nb = (b.n_trial + kScanWinBlock - 1) / kScanWinBlock;
        w = b.scan_win[(int64_t)p * nb + j / kScanWinBlock];
        w.x = min(w.x, m.k_scan);
        w.y = max(w.y, m.k_scan);
    }
    return w;
}

// Runs count(i) for the items 0 .. total - 1 of a queue: the groups' own
// indices first, then the queue's, each asked for before the pass of the item
// in hand (the atomic's round trip runs beside the pass).
template <int NW, typename Count>
__device__ __forceinline__ void for_items(const Grp<NW>& G, const DevBatch& b, int* queue, int total, int& word,
                                          Count&& count) {
    const int groups = gridDim.x * (ScanCta<NW>::kThreads / Grp<NW>::kThreads);
    int item = NW == 1 ? blockIdx.x * (ScanCta<NW>::kThreads / 32) + (threadIdx.x >> 5) : blockIdx.x;
    while (item < total) {
        int q = 0, stop = 0;
        if (G.leader()) {
            q = atomicAdd(queue, 1);
            stop = stop_asked(b, (item & 15) == 0);
        }
        count(item);
        item = grp_bcast<NW>(G, stop ? total : groups + q, word);
    }
}

// Every stride-th trial energy (and the last): longest grids first, highest
// energies (longest windows) first.
template <int NW>
__global__ void __launch_bounds__(ScanCta<NW>::kThreads, ScanCta<NW>::kPerSm) count_stride_kernel(DevBatch b,
                                                                                                  int stride) {
    __shared__ Shared32<NW> sh;
    __shared__ int word;
    const Grp<NW> G;
    const int last = b.n_trial - 1, K = (b.n_trial + stride - 1) / stride;
    unsigned long long updates = 0;
    for_items<NW>(G, b, &b.hdr->queue[kQCountStride], b.n * K, word, [&](int item) {
        const int p = b.order[item / K];
        const int j = min((K - item % K) * stride - 1, last);
        const int status = b.meta[p].status;
        if (status & EPSCU_STATUS_BAD) {
            if (G.leader()) b.counts[(int64_t)p * b.n_trial + j] = 0;
            return;
        }
        if (b.under_list && (status & EPSCU_STATUS_UNDER)) return;  // (the lane scan's)
        const int2 w = scan_window(b, p, j);
        count_at<NW>(G, b, p, j, w.x, w.y, sh);
        updates += (unsigned long long)(w.y - w.x);
    });
    if (G.leader() && updates) atomicAdd(&b.hdr->scan_updates, updates);
}

// The trial energies the plan listed: its items are chunks of `chunk` entries
// of a potential's list.
template <int NW>
__global__ void __launch_bounds__(ScanCta<NW>::kThreads, ScanCta<NW>::kPerSm) count_listed_kernel(DevBatch b,
                                                                                                  int chunk) {
    __shared__ Shared32<NW> sh;
    __shared__ int word;
    const Grp<NW> G;
    const int total = min(b.hdr->bis_items_n, b.max_bis_items) * chunk;
    unsigned long long updates = 0;
    for_items<NW>(G, b, &b.hdr->queue[kQCountListed], total, word, [&](int item) {
        const int2 it = b.bis_items[item / chunk];
        const int q = it.y + item % chunk;
        if (q >= b.bis_n[it.x]) return;
        const int j = b.bis_list[(int64_t)it.x * b.n_trial + q];
        const int2 w = scan_window(b, it.x, j);
        count_at<NW>(G, b, it.x, j, w.x, w.y, sh);
        updates += (unsigned long long)(w.y - w.x);
    });
    if (G.leader() && updates) atomicAdd(&b.hdr->scan_updates, updates);
}

template <int NW>
constexpr size_t stage_bytes() {
    return (size_t)(ScanCta<NW>::kThreads / 32) * kStageFloat2 * sizeof(float2);
}

template <int NW>
int grid_of(int64_t energies, int sm_count) {
    const int64_t ctas = (energies * NW * 32 + ScanCta<NW>::kThreads - 1) / ScanCta<NW>::kThreads;
    return (int)(ctas < (int64_t)sm_count * ScanCta<NW>::kPerSm ? (ctas > 0 ? ctas : 1)
                                                                : (int64_t)sm_count * ScanCta<NW>::kPerSm);
}

}  // namespace

void groupscan_set_attributes() {
    cudaFuncSetAttribute(count_stride_kernel<kScanWarps>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)stage_bytes<kScanWarps>());
    cudaFuncSetAttribute(count_listed_kernel<kScanWarps>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)stage_bytes<kScanWarps>());
}

// a CTA per energy?
static bool cta_groups(const DevBatch& b) { return b.max_N > kScanCtaPoints; }

void launch_count_stride(const DevBatch& b, int stride, int sm_count, cudaStream_t s) {
    const int64_t energies = (int64_t)b.n * ((b.n_trial + stride - 1) / stride);
    if (cta_groups(b))
        count_stride_kernel<kScanWarps>
            <<<grid_of<kScanWarps>(energies, sm_count), ScanCta<kScanWarps>::kThreads, stage_bytes<kScanWarps>(), s>>>(
                b, stride);
    else
        count_stride_kernel<1>
            <<<grid_of<1>(energies, sm_count), ScanCta<1>::kThreads, stage_bytes<1>(), s>>>(b, stride);
}

void launch_count_listed(const DevBatch& b, int chunk, int sm_count, cudaStream_t s) {
    const int64_t energies = (int64_t)b.n * b.n_trial;  // (at most)
    if (cta_groups(b))
        count_listed_kernel<kScanWarps>
            <<<grid_of<kScanWarps>(energies, sm_count), ScanCta<kScanWarps>::kThreads, stage_bytes<kScanWarps>(), s>>>(
                b, chunk);
    else
        count_listed_kernel<1>
            <<<grid_of<1>(energies, sm_count), ScanCta<1>::kThreads, stage_bytes<1>(), s>>>(b, chunk);
}

}  // namespace epscu
