// levels.cu -- the plain method's per-level refinement, normalisation and
// write-back, and the results' gather of both methods.
//
// Every kernel here is persistent (grid = SMs x resident CTAs) and walks the
// level slots written by the bracket kernel; the number of slots is read from
// device memory, so the whole solve can be captured in one CUDA graph.
//
//  bisect64 : plain method, FP64 bisection on the twisted Sturm count with the
//             match index k(E) (outer classical turning point), n_bisect halvings
//             of the scan bracket -- identical arithmetic to the oracle.
//  norm64   : FP64 Cooley pass that also fixes the normalisation constants
//             (sum psi^2 h = 1, psi > 0 next to the inner wall) and the node
//             count reported for the level.
//  write64  : recomputes the FP64 recurrence and writes psi.
//  gather   : level slots -> the caller's [potential x capacity] layout; the
//             fast method reports E + dE of the last FP64 pass, the plain
//             method the bisection midpoint itself.
//
// Scale handling: the divide-free state after step i is s_{i+1} (u_{i+1}, u_i)
// with s_{i+1} = f_{i0} ... f_i, so psi_i = u_i / f_i = A_i / s_{i+1}.  Sums
// of psi^2 use S_{i+1} = f_i^2 S_i + A_i^2 (no division); the write pass
// carries q_i = 1 / s_i with a refined reciprocal of f_i.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "common.cuh"
#include "launch.h"

namespace epscu {

namespace {

__device__ __forceinline__ bool cancelled(const DevBatch& b) { return b.cancel && *b.cancel; }

// match points stay off the two boundary points (both sides non-empty)
__device__ __forceinline__ int clamp_inner(const PotMeta& m, int k) { return max(m.i0 + 1, min(k, m.i1 - 1)); }

// ------------------------------------------------------------------ FP64 pass

struct Side64 {
    double A, B, S, q;  // state, psi^2 sum, 1/s
    int eA, eQ;         // exponents removed from A/B and from q
    int nodes;
    int peak_L, peak_i;  // largest log2 |psi-hat| seen at a renormalisation point, and where
};

// STEEP: f may be anything (a barrier above the cut-offs); otherwise f >= 1/2, and
// its reciprocal needs no look at its range (4% of a small batch, 5.84 -> 6.07 ms)
template <bool WRITE, bool STEEP>
__device__ __forceinline__ void side64_of(const double* __restrict__ W, double aE, int from, int to, int dir, Side64& st,
                                          double* __restrict__ out, double L, int Xk) {
    auto recip = [](double f) { return STEEP ? recip64(f) : recip64_normal(f); };
    st.A = 1.0;
    st.B = 0.0;
    st.S = 0.0;
    st.q = 1.0;
    st.eA = 0;
    st.eQ = 0;
    st.nodes = 0;
    st.peak_L = -1 << 30;
    st.peak_i = from;
    int s = 0;
    double F = 0.0;
    if (WRITE) F = L * ldexp(1.0, min(1000, max(-1100, -Xk)));
    // (the next point's f, g and 1/f are formed beside this point's step, which
    // does not wait for them)
    double T = __dsub_rn(aE, __ldg(W + from));
    double f = __dadd_rn(1.0, T), rf = recip(f), g = __fma_rn(-10.0, T, 2.0);
    for (int i = from; i != to; i += dir) {
        const double Tn = __dsub_rn(aE, __ldg(W + i + dir));  // (up to `to`: inside the grid)
        const double qn = st.q * rf;
        if (WRITE) out[i] = st.A * qn * F;
        st.q = qn;
        if (!WRITE) st.S = __fma_rn(f * f, st.S, st.A * st.A);
        const double An = __fma_rn(g, st.A, -__dmul_rn(f, st.B));
        st.B = __dmul_rn(f, st.A);
        f = __dadd_rn(1.0, Tn);
        rf = recip(f);
        g = __fma_rn(-10.0, Tn, 2.0);
        st.nodes += negative(An) != negative(st.A);
        st.A = An;
        if (++s == kRenorm) {
            s = 0;
            const int e = renorm_pair(st.A, st.B);
            st.eA += e;
            if (!WRITE && e) st.S *= pow2(-2 * e);
            const int eq = exp_of(st.q);
            st.q *= pow2(-eq);
            st.eQ += eq;
            if (!WRITE) {
                const double mag = fabs(st.A * st.q);
                if (mag > 0.0) {
                    const int L = exp_of(mag) + st.eA + st.eQ;
                    if (L > st.peak_L) {
                        st.peak_L = L;
                        st.peak_i = i;
                    }
                }
            }
            if (WRITE) F = L * ldexp(1.0, min(1000, max(-1100, st.eA + st.eQ - Xk)));
        }
    }
}

template <bool WRITE>
__device__ __forceinline__ void side64(const PotMeta& m, const double* __restrict__ W, double aE, int from, int to,
                                       int dir, Side64& st, double* __restrict__ out, double L, int Xk) {
    if (m.status & EPSCU_STATUS_STEEP) side64_of<WRITE, true>(W, aE, from, to, dir, st, out, L, Xk);
    else side64_of<WRITE, false>(W, aE, from, to, dir, st, out, L, Xk);
}

struct Pass64 {
    double dE, gamma, sum;
    double pk_out, pk_in;  // psi-hat at k from each side
    int ex_out, ex_in;
    int nodes;
    int peak_i;       // where |psi| peaks (sampled every kRenorm points)
    int peak_log2;    // log2 of that peak over |psi| at k
};

// The two lanes of a pair (2 l, 2 l + 1) work on one level, the even one
// marching the outward side of every pass, the odd one the inward side, and
// hand each other the result; everything else both do alike.
__device__ __forceinline__ bool inward_lane() { return (threadIdx.x & 1) != 0; }
template <typename T>
__device__ __forceinline__ T pair_other(T v) {
    return __shfl_xor_sync(3u << (threadIdx.x & 30), v, 1);
}

__device__ Pass64 cooley64(const PotMeta& m, const double* __restrict__ W, double E, int k) {
    const double aE = __dmul_rn(m.a, E);
    const bool inw = inward_lane();
    Side64 mine, other;
    side64<false>(m, W, aE, inw ? m.i1 : m.i0, k, inw ? -1 : +1, mine, nullptr, 0.0, 0);
    other.A = pair_other(mine.A);
    other.B = pair_other(mine.B);
    other.S = pair_other(mine.S);
    other.q = pair_other(mine.q);
    other.eA = pair_other(mine.eA);
    other.eQ = pair_other(mine.eQ);
    other.nodes = pair_other(mine.nodes);
    other.peak_L = pair_other(mine.peak_L);
    other.peak_i = pair_other(mine.peak_i);
    const Side64 o = inw ? other : mine, in = inw ? mine : other;
    const double Tk = __dsub_rn(aE, __ldg(W + k));
    const double fk = __dadd_rn(1.0, Tk);
    const double gk = __fma_rn(-10.0, Tk, 2.0);
    Pass64 r;
    const double fk2 = fk * fk;
    r.sum = fk2 * (o.S / (o.A * o.A) + in.S / (in.A * in.A)) + 1.0;
    r.gamma = gk / fk - o.B / o.A - in.B / in.A;
    r.dE = r.gamma * fk2 / (12.0 * m.a * r.sum);
    r.nodes = o.nodes + in.nodes;
    const double rk = recip64(fk);
    r.pk_out = o.A * o.q * rk;
    r.pk_in = in.A * in.q * rk;
    r.ex_out = o.eA + o.eQ;
    r.ex_in = in.eA + in.eQ;
    const int Lo = (r.pk_out != 0.0 ? exp_of(fabs(r.pk_out)) : -1000) + r.ex_out;
    const int Li = (r.pk_in != 0.0 ? exp_of(fabs(r.pk_in)) : -1000) + r.ex_in;
    const int po = o.peak_L - Lo, pi = in.peak_L - Li;
    r.peak_log2 = max(po, pi);
    r.peak_i = po >= pi ? o.peak_i : in.peak_i;
    return r;
}

// ----------------------------------------------------------------- kernels

// A warp's next levels: up to `per` (a divisor of 32) consecutive slots of one
// unit (<= 32 levels of a potential, longest grids first).  turn: how often the
// warp has asked.  The first time it takes the item of its own number: CTAs are
// dealt to the SMs in turn, so with few items each has an SM quarter (and its
// FP64 pipe) to itself; after that from the queue.
__device__ __forceinline__ bool next_slots(const DevBatch& b, int qid, int per, int& turn, int2& slots) {
    const int split = 32 / per;
    for (;;) {
        int u = (int)blockIdx.x;
        if (turn > 0) {
            if ((threadIdx.x & 31) == 0) u = (int)gridDim.x + atomicAdd(&b.hdr->queue[qid], 1);
            u = __shfl_sync(0xffffffffu, u, 0);
        }
        ++turn;
        if (u / split >= min(b.hdr->n_units, b.max_units)) return false;
        const int2 unit = b.units[u / split];
        const int at = (u % split) * per;
        if (at >= unit.y) continue;
        slots = make_int2(unit.x + at, min(per, unit.y - at));
        return true;
    }
}

// Bisection of a level by 2^d lanes a side, d halvings per march: lanes 2 c and
// 2 c + 1 (c = 1 .. 2^d - 1) march the outward and the inward side of the count
// at node c of the tree of midpoints the next d halvings can visit (each
// midpoint formed from its ancestors by the bisection's own operations, so
// every energy and the final bracket are the sequential bisection's to the
// bit).  A FP64 instruction holds its SM quarter's FP64 pipe for 64 cycles
// however many lanes are active, and a march is a chain: with few levels the
// lanes are free.  d = 0: one lane per level, both sides in turn, which does
// the least work and is the form for many levels (the FP64 pipes' work is what
// counts then).  The form is the one with the shortest of (marches) x (warps
// per SM quarter); the longer side of a march is ~2/3 of its window.
// (145 levels on 3001 points, 27 halvings: 26.7 ms one lane per level.)
__device__ __forceinline__ int bisect_depth(int levels, int sms) {
    int best = 0;
    long long best_cost = 1ll << 60;
    for (int d = 0; d <= 4; ++d) {
        const long long marches = d == 0 ? 28 * 3 : (28 + d - 1) / d * 2;  // (of a typical bisection, in thirds)
        const long long warps = d == 0 ? (levels + 31) / 32 : ((long long)levels * (2 << d) + 31) / 32;
        const long long cost = marches * max(1ll, (warps + 4 * sms - 1) / (4 * sms));
        if (cost < best_cost) {
            best_cost = cost;
            best = d;
        }
    }
    return best;
}

__global__ void __launch_bounds__(32) bisect64_kernel(DevBatch b, int sms) {
    const int d = bisect_depth(b.hdr->total_levels, sms);
    const int lane = threadIdx.x;
    const int G = d == 0 ? 1 : 2 << d;              // lanes per level
    const int c = d == 0 ? 1 : max(1, (lane % G) / 2);  // this lane's node (0: none, it follows node 1)
    const bool inw = d > 0 && inward_lane();
    const int halvings = max(1, d);
    int turn = 0;
    for (int2 slots; next_slots(b, kQBisect64, 32 / G, turn, slots);) {
        // (lanes without a level do the unit's last one, and write nothing)
        const bool mine = lane / G < slots.y;
        const int slot = slots.x + min(lane / G, slots.y - 1);
        LevelWork w = b.levels[slot];
        const PotMeta m = b.meta[w.p];
        const double* W = b.W64 + m.off;
        const bool found = !(w.status & EPSCU_STATUS_NOTFOUND);
        // (one lane reads the host's flag, so the warp stays together)
        const bool stop = __shfl_sync(0xffffffffu, (int)(lane == 0 && cancelled(b)), 0) != 0;
        if (found && stop && mine && lane % G == 0) b.levels[slot].status = w.status | EPSCU_STATUS_CANCELLED;
        if (stop) continue;
        double lo = w.lo, hi = w.hi;
        // (levels of one unit share the potential, and with it n_bisect)
        for (int it = 0; it < m.n_bisect; it += halvings) {
            double l = lo, h = hi;
            double mid = __dmul_rn(0.5, __dadd_rn(l, h));
            for (int bit = 30 - __clz(c); bit >= 0; --bit) {
                if ((c >> bit) & 1) l = mid;
                else h = mid;
                mid = __dmul_rn(0.5, __dadd_rn(l, h));
            }
            const double aE = __dmul_rn(m.a, mid);
            const int k = match_index(m, b, mid);
            int count = 0;
            if (d == 0) {
                if (found) count = count64(m, W, mid, k);
            } else {
                double A = 1.0, B = 0.0;
                if (found) count = count_side64(W, aE, inw ? m.i1 : m.i0, k, inw ? -1 : 1, A, B);
                const double C = __shfl_xor_sync(0xffffffffu, A, 1), D = __shfl_xor_sync(0xffffffffu, B, 1);
                count += __shfl_xor_sync(0xffffffffu, count, 1);
                // (the even lane's: its own state is the outward one)
                count += count_join64(aE, __ldg(W + k), A, B, C, D);
            }
            const unsigned votes = __ballot_sync(0xffffffffu, found && count > w.v);
            int at = 1;
            for (int s = 0; s < halvings && it + s < m.n_bisect; ++s) {
                const double x = __dmul_rn(0.5, __dadd_rn(lo, hi));
                const bool up = (votes >> (d == 0 ? lane : lane - lane % G + 2 * at)) & 1u;
                if (up) hi = x;
                else lo = x;
                at = 2 * at + (up ? 0 : 1);
            }
        }
        if (found && mine && lane % G == 0) {
            w.lo = lo;
            w.hi = hi;
            w.E = __dmul_rn(0.5, __dadd_rn(lo, hi));
            w.iters = m.n_bisect;
            b.levels[slot] = w;
        }
    }
}

// Levels per warp of the pair kernels (two lanes each): as few as leave every
// SM quarter a warp (a warp costs its FP64 pipe the same whatever its lanes).
__device__ __forceinline__ int pairs_per_warp(int levels, int sms) {
    int per = 1;
    while (per < 16 && levels > 4 * sms * per) per <<= 1;
    return per;
}

// Write the normalisation constants of pass r (match point k) into w.
__device__ __forceinline__ void finalize64(const PotMeta& m, LevelWork& w, const Pass64& r, int k) {
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

// Matched at the outer turning point, moved to the peak of |psi| of the
// solution stitched there (as the oracle's match point).
__global__ void __launch_bounds__(32) norm64_kernel(DevBatch b, int sms) {
    const int per = pairs_per_warp(b.hdr->total_levels, sms);
    int turn = 0;
    for (int2 slots; next_slots(b, kQNorm64, per, turn, slots);) {
        const int lane = threadIdx.x & 31;
        if (lane / 2 >= slots.y) continue;
        const int slot = slots.x + lane / 2;
        LevelWork w = b.levels[slot];
        if (w.status & (EPSCU_STATUS_NOTFOUND | EPSCU_STATUS_CANCELLED)) continue;
        const PotMeta m = b.meta[w.p];
        int k = clamp_inner(m, match_index(m, b, w.E));
        Pass64 r = cooley64(m, b.W64 + m.off, w.E, k);
        if (r.peak_log2 >= 1) {
            k = clamp_inner(m, r.peak_i);
            r = cooley64(m, b.W64 + m.off, w.E, k);
        }
        finalize64(m, w, r, k);
        if (inward_lane()) continue;
        // a poor match point shows as a wrong node count or as a Cooley
        // correction far above the accuracy of the bisected energy
        const bool bad = (r.nodes != w.v && !(m.status & EPSCU_STATUS_UNDER)) ||
                         !(fabs(r.dE) <= 1e-11 * fmax(1.0, fabs(w.E)));
        if (bad && b.twist_list) {
            const int q = atomicAdd(&b.hdr->n_twist, 1);
            if (q < b.max_twist) b.twist_list[q] = slot;
        }
        b.levels[slot] = w;
    }
}

// Twist-index search of the plain method (FP64): sampled outward ratios
// u_{k-1}/u_k, inward ratios v_{k+1}/v_k, match point argmin |gamma_k|.
__global__ void __launch_bounds__(64) twist64_kernel(DevBatch b) {
    const int n = min(b.hdr->n_twist, b.max_twist);
    // (a pair of lanes per level: both sweep alike, then share the last pass)
    for (int q = (blockIdx.x * blockDim.x + threadIdx.x) / 2; q < n; q += gridDim.x * blockDim.x / 2) {
        const int slot = b.twist_list[q];
        LevelWork w = b.levels[slot];
        const PotMeta m = b.meta[w.p];
        const double* W = b.W64 + m.off;
        double* rho = b.twist_scratch + (int64_t)q * b.twist_stride;
        const double aE = __dmul_rn(m.a, w.E);
        double A = 1.0, B = 0.0;
        int s = 0;
        for (int i = m.i0; i < m.i1; ++i) {
            const int j = (i - m.i0) / kTwistSample;
            if ((i - m.i0) % kTwistSample == 0 && j < b.twist_stride && !inward_lane()) rho[j] = B / A;
            step64(aE, __ldg(W + i), A, B);
            if (++s == kRenorm) {
                s = 0;
                renorm_pair(A, B);
            }
        }
        __syncwarp(3u << (threadIdx.x & 30));  // rho is complete
        double C = 1.0, D = 0.0, best = INFINITY;
        int kbest = w.k;
        s = 0;
        for (int i = m.i1; i > m.i0; --i) {
            if ((i - m.i0) % kTwistSample == 0 && i <= m.i1 - 1) {
                const int j = (i - m.i0) / kTwistSample;
                if (j < b.twist_stride) {
                    const double T = __dsub_rn(aE, __ldg(W + i));
                    const double gam = (2.0 - 10.0 * T) / (1.0 + T) - rho[j] - D / C;
                    if (fabs(gam) < best) {
                        best = fabs(gam);
                        kbest = i;
                    }
                }
            }
            step64(aE, __ldg(W + i), C, D);
            if (++s == kRenorm) {
                s = 0;
                renorm_pair(C, D);
            }
        }
        const int k = clamp_inner(m, kbest);
        const Pass64 r = cooley64(m, W, w.E, k);
        finalize64(m, w, r, k);
        if (!inward_lane()) b.levels[slot] = w;
    }
}

__global__ void __launch_bounds__(32) write64_kernel(DevBatch b, int sms) {
    if (!b.psi || b.hdr->error) return;
    const int per = pairs_per_warp(b.hdr->total_levels, sms);
    const int lane = threadIdx.x & 31;
    int turn = 0;
    for (int2 slots; next_slots(b, kQWrite64, per, turn, slots);) {
        // zeros outside the cut-offs (everywhere without a result) by the warp
        for (int u = 0; u < slots.y; ++u) {
            const LevelWork w = b.levels[slots.x + u];
            const PotMeta& m = b.meta[w.p];
            double* out = b.psi + m.psi_off + (int64_t)(w.v - b.min_level) * m.N;
            const bool none = (w.status & (EPSCU_STATUS_NOTFOUND | EPSCU_STATUS_CANCELLED | EPSCU_STATUS_NONFINITE)) != 0;
            for (int i = lane; i < (none ? m.N : m.i0); i += 32) out[i] = 0.0;
            if (!none)
                for (int i = m.i1 + 1 + lane; i < m.N; i += 32) out[i] = 0.0;
        }
        if (lane / 2 >= slots.y) continue;
        const LevelWork w = b.levels[slots.x + lane / 2];
        if (w.status & (EPSCU_STATUS_NOTFOUND | EPSCU_STATUS_CANCELLED | EPSCU_STATUS_NONFINITE)) continue;
        const PotMeta m = b.meta[w.p];
        double* out = b.psi + m.psi_off + (int64_t)(w.v - b.min_level) * m.N;
        const double* W = b.W64 + m.off;
        const double aE = __dmul_rn(m.a, w.E);
        Side64 st;
        const bool inw = inward_lane();
        side64<true>(m, W, aE, inw ? m.i1 : m.i0, w.k, inw ? -1 : +1, st, out, inw ? w.norm_k_in : w.norm_k_out,
                     inw ? w.ex_in : w.ex_out);
        if (!inw) out[w.k] = w.ck;
    }
}

__global__ void gather_kernel(DevBatch b, int32_t* n_total, int32_t* n_out, double* energy, int32_t* nodes,
                              int32_t* status, double* err_est, int apply_dE) {
    const int p = blockIdx.x;
    const PotMeta m = b.meta[p];
    if (threadIdx.x == 0) {
        n_total[p] = m.n_total;
        n_out[p] = m.n_out;
    }
    for (int s = threadIdx.x; s < b.level_capacity; s += blockDim.x) {
        const int64_t o = (int64_t)p * b.level_capacity + s;
        if (s < m.n_out) {
            const LevelWork w = b.levels[m.level_base + s];
            energy[o] = (apply_dE && fabs(w.dE) <= 1e-9) ? w.E + w.dE : w.E;
            nodes[o] = w.nodes;
            status[o] = (w.status & EPSCU_STATUS_PUBLIC) | (m.status & EPSCU_STATUS_UNDER);
            if (err_est) err_est[o] = fabs(w.dE);
        } else {
            energy[o] = NAN;
            nodes[o] = -1;
            status[o] = EPSCU_STATUS_NOTFOUND | (m.status & (EPSCU_STATUS_BAD | EPSCU_STATUS_NONFINITE));
            if (err_est) err_est[o] = NAN;
        }
    }
}

}  // namespace

// CTAs of one warp, dealt to the SMs in turn: the first 4 sm_count work items
// have a quarter of an SM, and its FP64 pipe, each
constexpr int kWarpsPerSm = 16;

void launch_bisect64(const DevBatch& b, int sm_count, cudaStream_t s) {
    bisect64_kernel<<<sm_count * kWarpsPerSm, 32, 0, s>>>(b, sm_count);
}
void launch_norm64(const DevBatch& b, int sm_count, cudaStream_t s) {
    norm64_kernel<<<sm_count * kWarpsPerSm, 32, 0, s>>>(b, sm_count);
}
void launch_twist64(const DevBatch& b, int sm_count, cudaStream_t s) {
    twist64_kernel<<<sm_count, 64, 0, s>>>(b);
}
void launch_write64(const DevBatch& b, int sm_count, cudaStream_t s) {
    write64_kernel<<<sm_count * kWarpsPerSm, 32, 0, s>>>(b, sm_count);
}
void launch_gather(const DevBatch& b, int32_t* n_total, int32_t* n_out, double* energy, int32_t* nodes,
                   int32_t* status, double* err_est, int apply_dE, cudaStream_t s) {
    gather_kernel<<<b.n, 128, 0, s>>>(b, n_total, n_out, energy, nodes, status, err_est, apply_dE);
}

}  // namespace epscu
