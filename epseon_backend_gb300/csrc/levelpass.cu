// levelpass.cu -- the fast method's levels, from the scan's bracket to the
// written wavefunction, one group of threads per level (grouppass.cuh).
//
//  order_levels : the level slots by falling window length (counting sort of
//                 the window kernel's buckets), so that the queues below hand
//                 out the longest work first;
//  levels       : a group takes a level from a device queue and carries it
//                 through
//                   1. FP32 passes: safeguarded Cooley-Newton with the count
//                      bracket, to a Newton step of at most kTol32;
//                   2. double-float phase-1 passes (state and node count only,
//                      the FP32 pass's sum as the Newton denominator) until
//                      the correction is below the energy's resolution;
//                   3. phase 3 from the start states of the last of them: the
//                      normalisation, the correction with its own sum, and
//                      with psi requested the level's row, written unscaled
//                      as tagged float pairs, then turned into the normalised
//                      doubles and the row's rest zeroed while the window is
//                      still in the caches.
//                 The group is a warp where there are levels enough to fill
//                 the GPU, a CTA for windows above a threshold that falls with
//                 the number of levels, a cluster of four CTAs for the longest
//                 windows of a few potentials;
//  repair       : levels stage 2 could not settle (full double-float passes
//                 from the scan bracket widened by one trial spacing) and
//                 levels whose final pass disagrees (twist-index search), one
//                 CTA per level;
//  rewrite      : psi again from the final energies and match points (the
//                 adjoint of a solve that kept none), the same passes as the
//                 solve's, so the same bits.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "common.cuh"
#include "dfloat.cuh"
#include "dfpass.cuh"
#include "grouppass.cuh"
#include "launch.h"
#include "psirow.cuh"

namespace epscu {

namespace {

constexpr int kCtaWarps = 8;
constexpr int kClusterWarps = 32;  // four CTAs
constexpr int kCtaCtasPerSm = 2;

// FP32 Newton steps at most this large hand over to the double-float passes
// (Hartree); the energy after such a step is far inside their first step's
// range
constexpr double kTol32 = 3e-8;
// a double-float correction at most this large (Hartree, relative above 1) is
// left to the reported energy: psi keeps the energy it was computed at, and is
// off by what is left over the gap to the next level.  psi's error in L2 against
// FP64 at a bracket of 1e-15 (41137 levels of 1500 uneven grids; rms, median,
// 99th percentile), and the solve of 2048 uneven grids with psi and gradient:
//     1e-14     6.1e-12  3.2e-13  2.8e-11    17.4 ms
//      2e-15    1.7e-12  2.2e-13  6.3e-12    17.8 ms
//      1e-15    1.3e-12  1.9e-13  3.8e-12    17.9 ms
// (the passes of a lane per level before these: 2.7e-12, 2.2e-13, 6.8e-12)
constexpr double kSettled = 1e-15;
// halvings before the repair kernel looks for a better match point (256 bumped
// Morse wells: the kernel 1.0 ms without, 0.51 ms after 4, 0.39 ms after 2)
constexpr int kHalveFirst = 2;

// match points on a strip boundary (whole strips on the outward side) where
// the window allows it
__device__ __forceinline__ int align_k(const int j0, const int j1, int k) {
    const int a = k & ~(kStrip - 1);
    if (a > j0 && a < j1) k = a;
    return max(j0 + 1, min(k, j1 - 1));
}

__device__ __forceinline__ bool df_less(dfl a, dfl b) { return a.h < b.h || (a.h == b.h && a.l < b.l); }
__device__ __forceinline__ dfl df_neg(dfl a) { return {-a.h, -a.l}; }

// ------------------------------------------------------------------ phase 3

// The norm pass: this thread's chunk from its start state X.  sum, node
// count, peak and the psi values at k from each side; with a row the
// unnormalised psi-hat of every window point as tagged pairs.
template <int NW>
__device__ __noinline__ PassDF norm_pass(const Grp<NW> G, const Chunk& c, const float2* __restrict__ Wf, double a,
                                            double Wk, double E, int k, const StD& X, bool neg,
                                            double* __restrict__ row, SharedDF<NW>& sh) {
    constexpr unsigned full = 0xffffffffu;
    const int t = G.t(), lane = G.lane();
    const dfl aE = df_from_double(__dmul_rn(a, E));
    StD s = X;
    PsiTag tag = psi_tag(s.e);
    SqSum ss;
    ss.init();
    int nodes = 0, flip = 0, below = 0;
    int pk_L = -(1 << 30), pk_i = k;
    for_points(
        c, Wf, [&](float2 w, auto steep) { return df_point<true, steep.value>(aE, w); },
        [&](const PointDF& pt, float2* slot, int i) {
            const dfl psi = df_mul(s.u, pt.r);
            const float p = __fmul_rn(psi.h, psi.h);
            const float e = __fmaf_rn(psi.h, psi.h, -p);
            ss.add({p, __fmaf_rn(2.0f * psi.h, psi.l, e)});
            if (row) slot[i & (kStrip - 1)] = psi_pair(psi, tag);
            const float before = s.u.h;
            df_march(pt.q, s.u, s.d);
            flip = (int)((__float_as_uint(s.u.h) ^ __float_as_uint(before)) >> 31);
            nodes += flip;
        },
        [&](const PointDF& pt, float2*, int i, auto steep) {
            if (steep.value) below += pt.r.h < 0.0f;
            const float mm = fmaxf(fabsf(s.u.h), fabsf(s.d.h));
            if (mm > 0.0f && mm < INFINITY) {
                const int e = exp_clamped(mm, 120);
                const float sc = fpow2(-e);
                s.u = df_scale(s.u, sc);
                s.d = df_scale(s.d, sc);
                s.e += e;
                ss.rescale(-2 * e);
                tag = psi_tag(s.e);
            }
            if (s.u.h != 0.0f) {
                const int L = fexp(s.u.h) + s.e;
                if (L > pk_L) {
                    pk_L = L;
                    pk_i = i;
                }
            }
        },
        [&](int j, float2* buf) {
            if (!row) return;
            // the round's pairs to the row: 16 threads a strip
            __syncwarp();
            const int p0 = j < c.ns ? (c.s + c.dir * j) << 4 : -1;
            const int lo = c.lo, hi = c.hi;
#pragma unroll 2
            for (int x = 0; x < 16; ++x) {
                const int from = 2 * x + (lane >> 4);
                const int px = __shfl_sync(full, p0, from);
                const int lx = __shfl_sync(full, lo, from), hx = __shfl_sync(full, hi, from);
                const int i = px + (lane & 15);
                if (px >= 0 && i >= lx && i <= hx)
                    reinterpret_cast<float2*>(row)[i] = buf[from * kStageRow + (lane & 15)];
            }
        });
    const bool out = t < c.Lo;
    // A zero of psi on a chunk's end point (the centre of a symmetric well): the
    // march gives u there one sign, the next thread's start state may have the
    // other, and the change would be counted by both threads or by neither.
    // The start state's sign holds.
    if (c.ns > 0 && t != c.Lo - 1 && t != c.Lo + c.Li - 1 && neg != ((__float_as_uint(s.u.h) >> 31) != 0))
        nodes += flip ? -1 : 1;
    nodes = __reduce_add_sync(full, nodes - below);
    const DfE mine = c.ns > 0 ? sqsum_dfe(ss, 2 * s.e) : DfE{{0.0f, 0.0f}, 0};
    DfE so = warp_sum_dfe(out ? mine : DfE{{0.0f, 0.0f}, 0});
    DfE si = warp_sum_dfe(out ? DfE{{0.0f, 0.0f}, 0} : mine);
    int po_L = out ? pk_L : -(1 << 30), po_i = pk_i, pi_L = out ? -(1 << 30) : pk_L, pi_i = pk_i;
    warp_peak(po_L, po_i);
    warp_peak(pi_L, pi_i);
    StD Eo, Ei;
    double So = 0.0, Si = 0.0;
    if constexpr (NW == 1) {
        const int lo = c.Lo - 1, li = c.Lo + c.Li - 1;
        Eo = {shfl_df(s.u, lo), shfl_df(s.d, lo), __shfl_sync(full, s.e, lo)};
        Ei = {shfl_df(s.u, li), shfl_df(s.d, li), __shfl_sync(full, s.e, li)};
        so.e -= 2 * Eo.e;
        si.e -= 2 * Ei.e;
        So = dfe_to_double(so);
        Si = dfe_to_double(si);
    } else {
        if (t == c.Lo - 1) G.put(sh.eo3, s);
        if (t == c.Lo + c.Li - 1) G.put(sh.ei3, s);
        if (lane == 0) {
            const int w = G.warp();
            G.put(sh.nodes3[w], nodes);
            G.put(sh.so[w], so);
            G.put(sh.si[w], si);
            G.put(sh.po_L[w], po_L);
            G.put(sh.po_i[w], po_i);
            G.put(sh.pi_L[w], pi_L);
            G.put(sh.pi_i[w], pi_i);
        }
        G.sync();
        Eo = sh.eo3;
        Ei = sh.ei3;
        nodes = 0;
        po_L = pi_L = -(1 << 30);
#pragma unroll 1
        for (int w = 0; w < NW; ++w) {
            nodes += sh.nodes3[w];
            if (sh.po_L[w] > po_L) {
                po_L = sh.po_L[w];
                po_i = sh.po_i[w];
            }
            if (sh.pi_L[w] > pi_L) {
                pi_L = sh.pi_L[w];
                pi_i = sh.pi_i[w];
            }
        }
        if (G.warp() == 0) {
#pragma unroll 1
            for (int w = 0; w < NW; ++w) {
                DfE x = sh.so[w], y = sh.si[w];
                x.e -= 2 * Eo.e;
                y.e -= 2 * Ei.e;
                So += dfe_to_double(x);
                Si += dfe_to_double(y);
            }
        }
    }
    PassDF r;
    if (NW == 1 || G.warp() == 0) {
        double fk;
        r.gamma = gamma64(__dsub_rn(__dmul_rn(a, E), Wk), Eo, Ei, fk);
        r.nodes = nodes - (fk < 0.0 ? 1 : 0);
        r.count = r.nodes + (r.gamma < 0.0 ? 1 : 0);
        const double rfk = 1.0 / fk;
        r.pk_out = df_to_double(Eo.u) * rfk;
        r.pk_in = df_to_double(Ei.u) * rfk;
        r.ex_out = Eo.e;
        r.ex_in = Ei.e;
        r.sum = So / (r.pk_out * r.pk_out) + Si / (r.pk_in * r.pk_in) + 1.0;
        const int Lo = (r.pk_out != 0.0 ? exp_of(fabs(r.pk_out)) : -1000) + r.ex_out;
        const int Li = (r.pk_in != 0.0 ? exp_of(fabs(r.pk_in)) : -1000) + r.ex_in;
        const int po = po_L - Lo, pi = pi_L - Li;
        r.peak_log2 = max(po, pi);
        r.peak_i = po >= pi ? po_i : pi_i;
        r.dE = r.gamma * fk * fk / (12.0 * a * r.sum);
    }
    if constexpr (NW > 1) {
        if (t == 0) G.put(sh.res, r);
        G.sync();
        r = sh.res;
        G.sync();  // every thread has the result before the next pass's
    }
    return r;
}

// ------------------------------------------------------------------ a level

struct Tally {  // the leader's counters, added to the header at the kernel's end
    unsigned long long f32 = 0, df = 0, f32_max = 0, df_max = 0, zeros = 0, window = 0;
    int iters_max = 0, redos = 0;
};

__device__ __forceinline__ void flush(const DevBatch& b, const Tally& t, bool cta) {
    Header* h = b.hdr;
    if (t.f32) atomicAdd(&h->refine_updates, t.f32);
    if (t.df) atomicAdd(&h->df_updates, t.df);
    if (t.f32_max) atomicMax(&h->refine_max_updates, t.f32_max);
    if (t.df_max) atomicMax(&h->df_max_updates, t.df_max);
    if (t.zeros) atomicAdd(&h->psi_zero_points, t.zeros);
    if (t.window) atomicAdd(&h->psi_window_points, t.window);
    if (t.iters_max) atomicMax(&h->refine_max_iters, t.iters_max);
    if (t.redos) atomicAdd(&h->n_redo, t.redos);
    if (cta && t.f32) atomicAdd(&h->long32_updates, t.f32);
    if (cta && t.df) atomicAdd(&h->longdf_updates, t.df);
}

// What a level's passes read
struct Level {
    const float2* Wf;
    const double* W;
    double a, h;
    int j0, j1, v, N;
    bool under, steep;
};

__device__ __forceinline__ Level level_of(const DevBatch& b, const LevelWork& w) {
    const PotMeta& m = b.meta[w.p];
    return {b.Wf2 + m.offf,
            b.W64 + m.off,
            m.a,
            m.h,
            w.j0,
            w.j1,
            w.v,
            m.N,
            (m.status & EPSCU_STATUS_UNDER) != 0,
            (m.status & EPSCU_STATUS_STEEP) != 0};
}

// stages 2's state: the chunk and the start state of the last phase 1
template <int NW>
struct States {
    Chunk c;
    StD X, Eo, Ei;
    int nodes;
    bool neg;

    __device__ __forceinline__ void run(const Grp<NW>& G, const Level& L, double E, int k, SharedDF<NW>& sh) {
        c = make_chunk(G.t(), Grp<NW>::kThreads, L.j0, L.j1, k, L.steep);
        const double aE = __dmul_rn(L.a, E);
        states_df<NW>(G, c, L.Wf, df_from_double(aE), sh, X, Eo, Ei, nodes, neg);
        if (L.steep) nodes -= __dsub_rn(aE, __ldg(L.W + k)) < -1.0;  // (f < 0 at k)
    }

    // run() and the Cooley correction at its match point, with the sum of an
    // FP32 pass; count gets the number of levels below E.  (The FP64 part runs
    // in one warp: eight at it would queue for the FP64 pipe.)
    __device__ __forceinline__ double newton(const Grp<NW>& G, const Level& L, double E, int k, float sum,
                                             SharedDF<NW>& sh, int& count) {
        run(G, L, E, k, sh);
        double dE = 0.0;
        if (NW == 1 || G.warp() == 0) {
            double fk;
            const double gam = gamma64(__dsub_rn(__dmul_rn(L.a, E), __ldg(L.W + k)), Eo, Ei, fk);
            dE = gam * fk * fk / (12.0 * L.a * (double)sum);
            count = nodes + (gam < 0.0 ? 1 : 0);
        }
        if constexpr (NW > 1) {
            if (G.leader()) {
                G.put(sh.res.dE, dE);
                G.put(sh.res.count, count);
            }
            G.sync();
            dE = sh.res.dE;
            count = sh.res.count;
            G.sync();
        }
        return dE;
    }
};

// The norm pass at E and its match-point candidates: the FP32 one, the peak
// of |psi| seen by the pass, the outer turning point and its peak; the first
// whose stitched solution has v nodes wins.  (The peak itself, not the strip
// boundary before it: that can lie behind a wall, where psi is 2^-17 of the peak
// and the stitched solution off by the energy's rounding times that squared.)
// One more pass at E + dE when the correction is above the energy's resolution
// (psi is only as accurate as its energy).  `have`: st holds phase 1 at (E, k).
// Writes the constants and the energy into w.
template <int NW>
__device__ __forceinline__ void norm_level(const Grp<NW>& G, const DevBatch& b, const Level& L, LevelWork& w, double E,
                                           int k, States<NW>& st, bool have, double* row, SharedDF<NW>& sh, int& n_pass,
                                           int& redos) {
    auto pass = [&](int kk) {
        if (!have) {
            st.run(G, L, E, kk, sh);
            ++n_pass;
        }
        have = false;
        ++n_pass;
        return norm_pass<NW>(G, st.c, L.Wf, L.a, __ldg(L.W + kk), E, kk, st.X, st.neg, row, sh);
    };
    PassDF r, best;
    int kk = k, k_row = k;
    // (one pass in the loop: the candidates in their order)
    for (int step = 0;; ++step) {
        r = pass(kk);
        k_row = kk;
        if (step == 0) {
            best = r;
            k = kk;
            if (r.peak_log2 >= 2) {
                kk = clamp_k(w, r.peak_i);
                if (kk != k) continue;  // step 1: the peak's point
            }
            step = 1;
        } else if (step == 1) {
            best = r;
            k = kk;
        } else if (step == 2) {
            if (r.nodes != L.v && r.peak_log2 >= 1) {
                kk = clamp_k(w, r.peak_i);
                continue;  // step 3: its peak
            }
            step = 3;
        }
        if (step == 1 && best.nodes != L.v) {
            const PotMeta m = b.meta[w.p];
            kk = grp_bcast<NW>(G, G.leader() ? clamp_k(w, match_index(m, b, E)) : 0, sh.word);
            continue;  // step 2: the outer turning point
        }
        if (step == 3 && r.nodes == L.v) {
            best = r;
            k = kk;
        }
        if (step == 4) {
            best = r;
            break;
        }
        if (best.nodes == L.v && isfinite(best.dE) && fabs(best.dE) > 1e-13 * fmax(1.0, fabs(E)) &&
            fabs(best.dE) < 1e-8) {
            ++redos;
            E += best.dE;
        } else if (!(row && k_row != k)) {
            break;
        }
        kk = k;
        step = 3;  // step 4: the last pass
    }
    w.E = E;
    if (NW == 1 || G.warp() == 0) finalize_df(b.meta[w.p], w, best, k);
    if constexpr (NW > 1) {
        if (G.leader()) G.put(sh.w, w);
        G.sync();
        w = sh.w;
        G.sync();
    }
}

// twist-index search at w.E (the level's passes matched at a poor point): the
// outward solution's d/u every kTwistSample points, then |gamma_i| at the same
// points on the inward one; the match point becomes argmin |gamma_i| (Dhillon
// and Parlett's twisted-factorisation rule), then Newton and the norm pass
// there.
template <int NW>
__device__ __forceinline__ int twist_point(const Grp<NW>& G, const Level& L, double E, double* __restrict__ rho,
                                           int stride, int k_else, SharedDF<NW>& sh) {
    const dfl aE = df_from_double(__dmul_rn(L.a, E));
    const double aEd = __dmul_rn(L.a, E);
    double best = INFINITY;
    int at = 0x7fffffff;
#pragma unroll 1
    for (int dir = 1; dir >= -1; dir -= 2) {
        // one side over the whole window
        Chunk c;
        c.dir = dir;
        c.steep = L.steep;
        c.s_min = L.j0 >> 4;
        c.s_max = L.j1 >> 4;
        c.lo = dir > 0 ? L.j0 : L.j0 + 1;
        c.hi = dir > 0 ? L.j1 - 1 : L.j1;
        const int n = (c.hi >> 4) - (c.lo >> 4) + 1;
        c.m = (n + Grp<NW>::kThreads - 1) / Grp<NW>::kThreads;
        c.Lo = (n + c.m - 1) / c.m;
        c.Li = 0;
        c.ns = max(0, min(c.m, n - G.t() * c.m));
        c.s = dir > 0 ? (c.lo >> 4) + G.t() * c.m : (c.hi >> 4) - G.t() * c.m;
        c.seg = c.ns > 0 ? 0 : G.t();
        StD X, Eo, Ei;
        int nodes;
        bool neg;
        states_df<NW>(G, c, L.Wf, aE, sh, X, Eo, Ei, nodes, neg);
        dfl u = X.u, d = X.d;
        for_points(
            c, L.Wf, [&](float2 w, auto steep) { return df_point<false, steep.value>(aE, w); },
            [&](const PointDF& pt, float2*, int i) {
                const int rel = i - L.j0;
                if (rel % kTwistSample == 0 && rel / kTwistSample < stride) {
                    const double ratio = df_to_double(d) / df_to_double(u);
                    if (dir > 0) {
                        rho[rel / kTwistSample] = ratio;
                    } else if (i <= L.j1 - 1) {
                        const double Ti = aEd - __ldg(L.W + i);
                        const double out = rho[rel / kTwistSample];
                        // (with the rounding of the two ratios: at a node of psi they are huge
                        // and may cancel to anything)
                        const double gam =
                            fabs(-12.0 * Ti / (1.0 + Ti) + out + ratio) + 0x1p-44 * (fabs(out) + fabs(ratio));
                        if (gam < best || (gam == best && i < at)) {
                            best = gam;
                            at = i;
                        }
                    }
                }
                df_march(pt.q, u, d);
            },
            [&](const PointDF&, float2*, int, auto) {
                const int e = exp_clamped(fmaxf(fabsf(u.h), fabsf(d.h)), 120);
                const float sc = fpow2(-e);
                u = df_scale(u, sc);
                d = df_scale(d, sc);
            },
            [](int, float2*) {});
        __syncthreads();  // rho is complete
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double g2 = __shfl_xor_sync(0xffffffffu, best, o);
        const int k2 = __shfl_xor_sync(0xffffffffu, at, o);
        if (g2 < best || (g2 == best && k2 < at)) {
            best = g2;
            at = k2;
        }
    }
    if (G.lane() == 0) {
        sh.gb[G.warp()] = best;
        sh.gk[G.warp()] = at;
    }
    __syncthreads();
    best = INFINITY;
    at = 0x7fffffff;
    for (int w = 0; w < NW; ++w)
        if (sh.gb[w] < best || (sh.gb[w] == best && sh.gk[w] < at)) {
            best = sh.gb[w];
            at = sh.gk[w];
        }
    __syncthreads();
    return max(L.j0 + 1, min(at == 0x7fffffff ? k_else : at, L.j1 - 1));
}

// ---------------------------------------------------------------- kernels

// The counting sort's last step: slots to their place by bucket (longest
// windows first) and rank.
__global__ void __launch_bounds__(kLists * kBuckets) order_levels_kernel(DevBatch b) {
    static_assert(kBuckets == 64, "two warps scan a list's buckets");
    __shared__ int s_first[kLists * kBuckets];
    __shared__ int s_half[kLists];
    int32_t* const lists[kLists] = {b.warp_list, b.long_list, b.fragile_list, b.fragile_long, b.cluster_list};
    {
        // exclusive sums over falling bucket number, each list by two warps
        const int list = threadIdx.x / kBuckets, q = threadIdx.x % kBuckets;
        const int bucket = list * kBuckets + (kBuckets - 1 - q);
        const int n = b.hdr->hist[bucket];
        int x = n;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if ((int)(threadIdx.x & 31) >= o) x += y;
        }
        if (q == 31) s_half[list] = x;
        __syncthreads();
        if (q >= 32) x += s_half[list];
        s_first[bucket] = x - n;
        if (blockIdx.x == 0 && q == kBuckets - 1) {
            int32_t* const count[kLists] = {&b.hdr->n_warp, &b.hdr->n_long, &b.hdr->n_fragile, &b.hdr->n_fragile_long,
                                            &b.hdr->n_cluster};
            *count[list] = x;
        }
        __syncthreads();
    }
    const int total = b.hdr->total_levels;
    for (int slot = blockIdx.x * blockDim.x + threadIdx.x; slot < total; slot += gridDim.x * blockDim.x) {
        const LevelWork& w = b.levels[slot];
        lists[w.bucket / kBuckets][s_first[w.bucket] + w.rank] = slot;
    }
}

// The lists of the groups of NW warps
template <int NW>
__device__ __forceinline__ const int32_t* level_list(const DevBatch& b) {
    return NW == 1 ? b.warp_list : NW == kCtaWarps ? b.long_list : b.cluster_list;
}
template <int NW>
__device__ __forceinline__ int level_count(const DevBatch& b) {
    return min(NW == 1 ? b.hdr->n_warp : NW == kCtaWarps ? b.hdr->n_long : b.hdr->n_cluster, b.max_levels);
}

// The levels of one list, until its queue is empty.
template <int NW>
__device__ __forceinline__ void level_queue(const DevBatch& b, SharedDF<NW>& sh, Shared32<NW>& sh32) {
    const Grp<NW> G;
    const int32_t* list = level_list<NW>(b);
    const int n = level_count<NW>(b);
    int32_t* queue = &b.hdr->queue[NW == 1 ? kQWarpLevels : NW == kCtaWarps ? kQLongLevels : kQClusterLevels];
    Tally tally;
    for (;;) {
        const int2 next = grp_take<NW>(G, b, queue, n, sh.word);
        if (next.x >= n) break;
        const int slot = list[next.x];
        LevelWork w = b.levels[slot];
        const Level L = level_of(b, w);
        double* row = b.psi && !b.hdr->error
                          ? b.psi + b.meta[w.p].psi_off + (int64_t)(w.v - b.min_level) * L.N
                          : nullptr;
        if (next.y && !(w.status & EPSCU_STATUS_NOTFOUND)) w.status |= EPSCU_STATUS_CANCELLED;
        if (no_result(w)) {
            if (G.leader()) b.levels[slot].status = w.status;
            if (row) finish_row<Grp<NW>::kThreads>(G.t(), w, row, L.N);
            continue;
        }
        int k = w.k;
        // ---- stage 1, energies as a E in double-float
        dfl eps = df_from_double(L.a * w.E), lo = df_from_double(L.a * w.lo), hi = df_from_double(L.a * w.hi);
        const float tol = (float)(L.a * kTol32);
        float sum = 1.0f;
        bool ok = false, moved = false;
        int n32 = 0, ndf = 0;
        for (const int cap = refine_cap(b); n32 < cap;) {
            const Pass32 r = pass32<NW, true>(G, L.Wf, eps, L.j0, L.j1, k, L.steep, sh32);
            ++n32;
            sum = r.sum;
            if (r.count > L.v) hi = eps;
            else lo = eps;
            if (r.peak_log2 >= 2 && !moved) {
                const int kp = align_k(L.j0, L.j1, r.peak_i);
                if (kp != k) {
                    k = kp;
                    moved = true;
                    continue;  // the same energy at the new match point
                }
            }
            moved = false;
            const dfl en = df_add(eps, {r.de, 0.0f});
            const bool near = r.nodes == L.v && r.sum < 1e30f;
            if (near && isfinite(r.de) && df_less(lo, en) && df_less(en, hi)) {
                eps = en;
                if (fabsf(r.de) <= tol) {
                    ok = true;
                    break;
                }
            } else {
                eps = df_scale(df_add(lo, hi), 0.5f);
            }
            const dfl width = df_add(hi, df_neg(lo));
            if (width.h <= 2.0f * tol) {
                eps = df_scale(df_add(lo, hi), 0.5f);
                ok = true;
                break;
            }
        }
        // ---- stage 2
        States<NW> st;
        double E = 0.0;
        bool settled = false;
        if (ok) {
            E = df_to_double(eps) / L.a;
            double lo2 = df_to_double(lo) / L.a - 1e-8, hi2 = df_to_double(hi) / L.a + 1e-8;
#pragma unroll 1
            for (int it = 0; it < 6; ++it) {
                int count;
                const double dE = st.newton(G, L, E, k, sum, sh, count);
                ++ndf;
                if (count > L.v) hi2 = fmin(hi2, E);
                else lo2 = fmax(lo2, E);
                const double En = E + dE;
                if (!isfinite(En) || !(En >= lo2 && En <= hi2) || st.nodes != L.v) break;
                // (a correction at the energy's resolution: phase 3 goes on from
                // this pass's states, and its own correction is added to E)
                const double res = fmax(1.0, fabs(E));
                if (fabs(dE) <= kSettled * res || (it >= 4 && fabs(dE) <= 1e-12 * res)) {
                    settled = true;
                    break;
                }
                E = En;
            }
        }
        const unsigned long long pts = (unsigned long long)(L.j1 - L.j0);
        if (!settled) {
            // to the repair kernel, which goes on from the FP32 energy
            if (G.leader()) {
                if (ok) {
                    LevelWork& o = b.levels[slot];
                    o.E = df_to_double(eps) / L.a;
                    o.lo = df_to_double(lo) / L.a - 2e-8;
                    o.hi = df_to_double(hi) / L.a + 2e-8;
                    o.k = k;
                    o.iters = n32;
                }
                const int at = atomicAdd(&b.hdr->fallbacks, 1);
                if (at < b.max_levels) b.fallback_list[at] = slot;
            }
        } else {
            norm_level<NW>(G, b, L, w, E, k, st, true, row, sh, ndf, tally.redos);
            w.iters = n32 + ndf;
            if (row) finish_row<Grp<NW>::kThreads>(G.t(), w, row, L.N);
            if (G.leader()) {
                b.levels[slot] = w;
                if (b.twist_list && ((w.nodes != w.v && !L.under) || !(fabs(w.dE) <= 1e-11 * fmax(1.0, fabs(w.E))))) {
                    const int at = atomicAdd(&b.hdr->n_twist, 1);
                    if (at < b.max_twist) b.twist_list[at] = slot;
                }
            }
            if (row) {
                tally.zeros += (unsigned long long)(no_result(w) ? L.N : L.N - (L.j1 - L.j0 + 1));
                tally.window += (unsigned long long)(no_result(w) ? 0 : L.j1 - L.j0 + 1);
            }
        }
        tally.f32 += n32 * pts;
        tally.df += ndf * pts;
        tally.f32_max = max(tally.f32_max, n32 * pts);
        tally.df_max = max(tally.df_max, ndf * pts);
        tally.iters_max = max(tally.iters_max, n32);
    }
    if (G.leader()) flush(b, tally, NW > 1);
}

// The levels of all lists, the longest windows first: a CTA per level while
// there are long ones, then its warps a level each (one kernel: the warp list's
// longest marches run beside the last of the CTA list's instead of after them;
// 56 levels of one 4096-point grid 160 -> 85 us, 64 x 57 levels 670 -> 525 us).
__global__ void __launch_bounds__(32 * kCtaWarps, kCtaCtasPerSm) levels_kernel(DevBatch b) {
    __shared__ SharedDF<kCtaWarps> sh;
    __shared__ Shared32<kCtaWarps> sh32;
    __shared__ SharedDF<1> sh1;  // (a one-warp group uses neither)
    __shared__ Shared32<1> sh321;
    level_queue<kCtaWarps>(b, sh, sh32);
    level_queue<1>(b, sh1, sh321);
}

__global__ void __cluster_dims__(kClusterWarps / kCtaWarps, 1, 1)
    __launch_bounds__(32 * kCtaWarps, kCtaCtasPerSm) cluster_levels_kernel(DevBatch b) {
    __shared__ SharedDF<kClusterWarps> sh;
    __shared__ Shared32<kClusterWarps> sh32;
    Grp<kClusterWarps>().sync();  // (the other CTAs' shared memory exists)
    __shared__ SharedDF<kCtaWarps> sh8;
    __shared__ Shared32<kCtaWarps> sh328;
    __shared__ SharedDF<1> sh1;
    __shared__ Shared32<1> sh321;
    level_queue<kClusterWarps>(b, sh, sh32);
    level_queue<kCtaWarps>(b, sh8, sh328);
    level_queue<1>(b, sh1, sh321);
}

// Levels the queues above left over: first those stage 2 could not settle (the
// FP32 bracket may be off by its count errors: safeguarded Cooley-Newton with
// double-float passes from the FP32 stage's bracket, or the scan's widened by
// one trial spacing where its ends do not hold; Newton steps only while the pass
// sees the level's own node count and they stay inside the bracket, bisection
// otherwise), then those whose final pass disagrees.  Their psi is a CTA's from
// here on: they join the long list, which the rewrite's CTAs walk.
__global__ void __launch_bounds__(32 * kCtaWarps, kCtaCtasPerSm) repair_kernel(DevBatch b) {
    constexpr int NW = kCtaWarps;
    __shared__ SharedDF<NW> sh;
    __shared__ Shared32<NW> sh32;
    const Grp<NW> G;
    Tally tally;
    const int n_fall = min(b.hdr->fallbacks, b.max_levels);
    const int n_twist = min(b.hdr->n_twist, b.max_twist);
    for (;;) {
        const int2 next = grp_take<NW>(G, b, &b.hdr->queue[kQRepair], n_fall + n_twist, sh.word);
        const int q = next.x;
        if (q >= n_fall + n_twist) break;
        const bool fall = q < n_fall;
        const int slot = fall ? b.fallback_list[q] : b.twist_list[q - n_fall];
        LevelWork w = b.levels[slot];
        const Level L = level_of(b, w);
        const PotMeta m = b.meta[w.p];
        double* row = b.psi && !b.hdr->error ? b.psi + m.psi_off + (int64_t)(w.v - b.min_level) * L.N : nullptr;
        States<NW> st;
        int ndf = 0;
        double E = w.E;
        if (fall) {
            if (next.y) {
                w.status |= EPSCU_STATUS_CANCELLED;
                if (G.leader()) b.levels[slot].status = w.status;
                if (row) finish_row<Grp<NW>::kThreads>(G.t(), w, row, L.N);
                continue;
            }
            // the FP32 stage's bracket where its counts are right (a count
            // below and one above in double-float), the scan's otherwise
            int k = w.k;
            double lo = w.lo, hi = w.hi;
            auto count_at = [&](double e) {
                int count;
                st.newton(G, L, e, k, 1.0f, sh, count);
                ++ndf;
                return count;
            };
            if (!(w.iters > 0 && count_at(lo) <= L.v && count_at(hi) > L.v)) {
                lo = fmax(m.e_lo, w.lo0 - m.delta);
                hi = fmin(m.e_cap, w.hi0 + m.delta);
            }
            if (!(E > lo && E < hi)) E = 0.5 * (lo + hi);
            bool moved = false, done = false, twisted = false;
            int halved = 0;
            for (int it = 0, cap = fallback_cap(b); it < cap; ++it) {
                // sum psi^2 and the peak in FP32, the state and count in
                // double-float
                const Pass32 f = pass32<NW, true>(G, L.Wf, df_from_double(__dmul_rn(L.a, E)), L.j0, L.j1, k, L.steep, sh32);
                if (f.peak_log2 >= 2 && !moved && !twisted) {
                    const int kp = align_k(L.j0, L.j1, f.peak_i);
                    moved = true;
                    if (kp != k) {
                        k = kp;
                        continue;  // the same energy at the new match point
                    }
                }
                moved = false;
                int count;
                const double dE = st.newton(G, L, E, k, f.sum, sh, count);
                ++ndf;
                if (count > L.v) hi = E;
                else lo = E;
                const double tol = 1e-12 * fmax(1.0, fabs(E));
                const double En = E + dE;
                if (st.nodes == L.v && f.sum < 1e30f && isfinite(En) && En > lo && En < hi) {
                    E = En;
                    if (fabs(dE) <= tol) {
                        done = true;
                        break;
                    }
                } else {
                    E = 0.5 * (lo + hi);
                    // (matched in the wrong well the pass never has the level's
                    // nodes, and halving the bracket to the energy's resolution
                    // takes ~25 passes more: look for a better point instead)
                    twisted = b.twist_list && (++halved == kHalveFirst || halved == 2 * kHalveFirst);
                    if (twisted) {
                        k = twist_point<NW>(G, L, E, b.twist_scratch + (int64_t)blockIdx.x * b.twist_stride,
                                            b.twist_stride, k, sh);
                        ndf += 2;
                    }
                }
                if (hi - lo <= tol) {
                    E = 0.5 * (lo + hi);
                    done = true;
                    break;
                }
            }
            if (!done) w.status |= EPSCU_STATUS_MAXITER;
            norm_level<NW>(G, b, L, w, E, k, st, false, row, sh, ndf, tally.redos);
        }
        const bool off = (w.nodes != w.v && !L.under) || !(fabs(w.dE) <= 1e-11 * fmax(1.0, fabs(w.E)));
        if (!fall || (off && b.twist_list)) {
            // every CTA has scratch of its own
            E = w.E;
            const int k = twist_point<NW>(G, L, E, b.twist_scratch + (int64_t)blockIdx.x * b.twist_stride,
                                          b.twist_stride, w.k, sh);
            PassDF r;
#pragma unroll 1
            for (int it = 0;; ++it) {
                st.run(G, L, E, k, sh);
                r = norm_pass<NW>(G, st.c, L.Wf, L.a, __ldg(L.W + k), E, k, st.X, st.neg, row, sh);
                ndf += 2;
                if (it >= 8 || r.nodes != w.v || !isfinite(r.dE) || !(fabs(r.dE) < 1e-7)) break;
                if (fabs(r.dE) <= 1e-13 * fmax(1.0, fabs(E))) break;
                E += r.dE;
            }
            w.E = E;
            finalize_df(m, w, r, k);
        }
        if (row) finish_row<Grp<NW>::kThreads>(G.t(), w, row, L.N);
        if (G.leader()) {
            w.iters += ndf;
            if ((w.status & (EPSCU_STATUS_LONG | EPSCU_STATUS_CLUSTER)) != EPSCU_STATUS_LONG) {
                const int at = atomicAdd(&b.hdr->n_long, 1);
                if (at < b.max_levels) b.long_list[at] = slot;
                w.status = (w.status & ~EPSCU_STATUS_CLUSTER) | EPSCU_STATUS_LONG;
            }
            b.levels[slot] = w;
        }
        tally.df += ndf * (unsigned long long)(L.j1 - L.j0);
    }
    if (G.leader()) flush(b, tally, false);
}

// psi of the listed levels from their final energies and match points.
template <int NW>
__device__ __forceinline__ void rewrite_queue(const DevBatch& b, SharedDF<NW>& sh) {
    const Grp<NW> G;
    if (!b.psi || b.hdr->error) return;
    const int32_t* list = level_list<NW>(b);
    const int n = level_count<NW>(b);
    int32_t* queue = &b.hdr->queue[NW == 1 ? kQWarpRewrite : NW == kCtaWarps ? kQLongRewrite : kQClusterRewrite];
    for (;;) {
        const int2 next = grp_take<NW>(G, b, queue, n, sh.word);
        if (next.x >= n) break;
        LevelWork w = b.levels[list[next.x]];
        // (a repaired level: on the long list too)
        if (NW == 1 && (w.status & EPSCU_STATUS_LONG)) continue;
        if (NW == kClusterWarps && !(w.status & EPSCU_STATUS_CLUSTER)) continue;
        const Level L = level_of(b, w);
        double* row = b.psi + b.meta[w.p].psi_off + (int64_t)(w.v - b.min_level) * L.N;
        if (!no_result(w)) {
            States<NW> st;
            st.run(G, L, w.E, w.k, sh);
            const PassDF r = norm_pass<NW>(G, st.c, L.Wf, L.a, __ldg(L.W + w.k), w.E, w.k, st.X, st.neg, row, sh);
            finalize_df(b.meta[w.p], w, r, w.k);
        }
        finish_row<Grp<NW>::kThreads>(G.t(), w, row, L.N);
    }
}

__global__ void __launch_bounds__(32 * kCtaWarps, kCtaCtasPerSm) rewrite_kernel(DevBatch b) {
    __shared__ SharedDF<kCtaWarps> sh;
    __shared__ SharedDF<1> sh1;
    rewrite_queue<kCtaWarps>(b, sh);
    rewrite_queue<1>(b, sh1);
}

__global__ void __cluster_dims__(kClusterWarps / kCtaWarps, 1, 1)
    __launch_bounds__(32 * kCtaWarps, kCtaCtasPerSm) cluster_rewrite_kernel(DevBatch b) {
    __shared__ SharedDF<kClusterWarps> sh;
    Grp<kClusterWarps>().sync();
    __shared__ SharedDF<kCtaWarps> sh8;
    __shared__ SharedDF<1> sh1;
    rewrite_queue<kClusterWarps>(b, sh);
    rewrite_queue<kCtaWarps>(b, sh8);
    rewrite_queue<1>(b, sh1);
}

}  // namespace

namespace {

// the staging buffers of a CTA's warps, as dynamic shared memory
constexpr size_t stage_bytes(int threads) { return (size_t)(threads / 32) * kStageFloat2 * sizeof(float2); }
constexpr size_t kCtaStage = stage_bytes(32 * kCtaWarps);

}  // namespace

void levels_set_attributes() {
    const auto stage = [](const void* f) {
        cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCtaStage);
    };
    stage((const void*)levels_kernel);
    stage((const void*)cluster_levels_kernel);
    stage((const void*)rewrite_kernel);
    stage((const void*)cluster_rewrite_kernel);
    stage((const void*)repair_kernel);
}

void launch_order_levels(const DevBatch& b, int sm_count, cudaStream_t s) {
    order_levels_kernel<<<sm_count, kLists * kBuckets, 0, s>>>(b);
}
void launch_levels(const DevBatch& b, int sm_count, cudaStream_t s) {
    if (b.cluster_list)
        cluster_levels_kernel<<<sm_count / 4 * 4 * kCtaCtasPerSm, 32 * kCtaWarps, kCtaStage, s>>>(b);
    else
        levels_kernel<<<sm_count * kCtaCtasPerSm, 32 * kCtaWarps, kCtaStage, s>>>(b);
}
void launch_repair(const DevBatch& b, int sm_count, cudaStream_t s) {
    repair_kernel<<<sm_count * kCtaCtasPerSm, 32 * kCtaWarps, kCtaStage, s>>>(b);
}
void launch_rewrite(const DevBatch& b, int sm_count, cudaStream_t s) {
    if (b.cluster_list)
        cluster_rewrite_kernel<<<sm_count / 4 * 4 * kCtaCtasPerSm, 32 * kCtaWarps, kCtaStage, s>>>(b);
    else
        rewrite_kernel<<<sm_count * kCtaCtasPerSm, 32 * kCtaWarps, kCtaStage, s>>>(b);
}

}  // namespace epscu
