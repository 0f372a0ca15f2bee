// fragile.cu -- levels whose results the last bits of their passes decide.
//
//  * On grids that do not resolve the wavelength (k_max h > 1:
//    EPSCU_LEVEL_UNDER_RESOLVED) counts and energies of the discrete problem
//    are exact, but a level's matching function can have a pole within a
//    rounding error of its root: the node count of its shooting solution, and
//    now and then which of two close roots an iteration ends in, hang on the
//    rounding.
//  * Levels close to a neighbour (kFragileGap): psi mixes with the neighbour's
//    by the energy's resolution over the gap, 1e-13 / 1e-5 = 1e-8.
// These levels (12% and ~0.2% of the 2048-potential mixed batch) keep passes of
// their own, whose order of operations their results depend on: two lanes
// per level marching its window from both ends (lane32.cuh, lanedf.cuh), a CTA
// per level for windows above a threshold (the passes below), the twist-index
// search for levels whose final pass disagrees.  All other levels take
// levelpass.cu's.
//
// The CTA passes split each side of a pass (outward from j0 to the match point
// k, inward from j1 to k) into one contiguous chunk per thread:
//   1. every thread marches the two unit states (A, D) = (1, 0) and (0, 1)
//      through its chunk (the step D' = D + T (D - 12 A), A' = A + (T A + D')
//      is linear): the chunk's 2x2 transfer matrix, and the product of 1/f
//      over the chunk for the passes that need psi;
//   2. a prefix scan of the matrices, Hillis-Steele over the lanes with
//      shuffles, then over the warps through shared memory, gives every
//      chunk's exact starting state and scale (products renormalised by powers
//      of two, exponents in ints);
//   3. every thread re-runs its chunk from that state: node counts, the sum
//      of psi^2, the peak of |psi| or the psi write, reduced over the CTA.
// FP64 runs once per pass, in the CTA's thread 0 (the leader), which hands the
// pass's result on through shared memory.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "common.cuh"
#include "dfloat.cuh"
#include "dfpass.cuh"
#include "lane32.cuh"
#include "lanedf.cuh"
#include "launch.h"
#include "psirow.cuh"

namespace epscu {

namespace {

// CTA shape of the group passes: threads per CTA and the persistent grid's
// CTAs per SM
constexpr int kLongThreads = 256;
constexpr int kLongWarps = kLongThreads / 32;
constexpr int kLongCtasPerSm = 2;
// first of this file's rows of the twist scratch (levelpass.cu's CTAs, which may
// run at the same time, use the first ones)
constexpr int kFragileScratch = 2048;

// [[a, b], [c, d]] 2^e acting on the column (A, D)
struct Mat2 {
    dfl a, b, c, d;
    int e;
};

// v 2^e
struct Scal {
    dfl v;
    int e;
};

__device__ __forceinline__ Mat2 mat_identity() {
    return {{1.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}, {1.0f, 0.0f}, 0};
}

__device__ __forceinline__ void mat_norm(Mat2& m) {
    const float mm = fmaxf(fmaxf(fabsf(m.a.h), fabsf(m.b.h)), fmaxf(fabsf(m.c.h), fabsf(m.d.h)));
    if (mm > 0.0f && mm < INFINITY) {
        const int e = max(-120, min(120, fexp(mm)));
        const float sc = fpow2(-e);
        m.a = df_scale(m.a, sc);
        m.b = df_scale(m.b, sc);
        m.c = df_scale(m.c, sc);
        m.d = df_scale(m.d, sc);
        m.e += e;
    }
}

// x y (x applied after y)
__device__ __forceinline__ Mat2 mat_mul(const Mat2& x, const Mat2& y) {
    Mat2 r;
    r.a = df_add(df_mul(x.a, y.a), df_mul(x.b, y.c));
    r.b = df_add(df_mul(x.a, y.b), df_mul(x.b, y.d));
    r.c = df_add(df_mul(x.c, y.a), df_mul(x.d, y.c));
    r.d = df_add(df_mul(x.c, y.b), df_mul(x.d, y.d));
    r.e = x.e + y.e;
    mat_norm(r);
    return r;
}

__device__ __forceinline__ void scal_norm(Scal& s) {
    const float mm = fabsf(s.v.h);
    if (mm > 0.0f && mm < INFINITY) {
        const int e = max(-120, min(120, fexp(mm)));
        s.v = df_scale(s.v, fpow2(-e));
        s.e += e;
    }
}

__device__ __forceinline__ Scal scal_mul(const Scal& x, const Scal& y) {
    Scal r{df_mul(x.v, y.v), x.e + y.e};
    scal_norm(r);
    return r;
}

__device__ __forceinline__ dfl shfl_up_df(dfl v, int o) {
    return {__shfl_up_sync(0xffffffffu, v.h, o), __shfl_up_sync(0xffffffffu, v.l, o)};
}

__device__ __forceinline__ Mat2 shfl_up_mat(const Mat2& m, int o) {
    return {shfl_up_df(m.a, o), shfl_up_df(m.b, o), shfl_up_df(m.c, o), shfl_up_df(m.d, o),
            __shfl_up_sync(0xffffffffu, m.e, o)};
}

__device__ __forceinline__ Scal shfl_up_scal(const Scal& s, int o) {
    return {shfl_up_df(s.v, o), __shfl_up_sync(0xffffffffu, s.e, o)};
}

// T = aE - W as a double-float (the same operations as the lane passes)
__device__ __forceinline__ dfl t_of(dfl aE, float2 w) {
    const dfl T = two_sum(aE.h, -w.x);
    return fast_two_sum(T.h, __fadd_rn(T.l, __fsub_rn(aE.l, w.y)));
}

__device__ __forceinline__ void df_step(dfl T, dfl& A, dfl& D) {
    const dfl X = df_add(D, df_mulf(A, -12.0f));
    D = df_add(D, df_mul(T, X));
    A = df_add(A, df_add(df_mul(T, A), D));
}

// ---------------------------------------------------------------- groups
// A level's passes run on a CTA; its thread 0 is the leader.
struct Grp {
    static constexpr int kThreads = kLongThreads;
    __device__ __forceinline__ int t() const { return (int)threadIdx.x; }
    __device__ __forceinline__ int lane() const { return (int)(threadIdx.x & 31); }
    __device__ __forceinline__ int warp() const { return (int)(threadIdx.x >> 5); }
    __device__ __forceinline__ bool leader() const { return threadIdx.x == 0; }
};

// the leader's value to the whole CTA (slot: a shared word)
__device__ __forceinline__ int grp_bcast(const Grp& G, int v, int& slot) {
    if (G.leader()) slot = v;
    __syncthreads();
    const int r = slot;
    __syncthreads();  // every thread has read the slot
    return r;
}

// the next entry of a device queue for the group
__device__ __forceinline__ int grp_next(const Grp& G, int* queue, int& slot) {
    int q = 0;
    if (G.leader()) q = atomicAdd(queue, 1);
    return grp_bcast(G, q, slot);
}

// A non-negative sum (h + l) 2^e in double-float, and its warp-wide total:
// each lane's value aligned to the largest exponent of the warp (exact
// power-of-two scalings), then added with shuffles.  Lane 0's result is the
// one used (the butterfly's order is fixed, so it is reproducible).
struct DfE {
    dfl v;
    int e;
};

__device__ __forceinline__ DfE warp_sum_dfe(DfE x) {
    const bool has = x.v.h > 0.0f;
    int em = has ? x.e : -(1 << 30);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) em = max(em, __shfl_xor_sync(0xffffffffu, em, o));
    dfl v = {0.0f, 0.0f};
    if (has) {
        const int d = x.e - em;
        if (d > -120) v = df_scale(x.v, fpow2(d));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v = df_add(v, {__shfl_xor_sync(0xffffffffu, v.h, o), __shfl_xor_sync(0xffffffffu, v.l, o)});
    return {v, em};
}

// The same for FP32 sums v 2^e.
struct FE {
    float v;
    int e;
};

__device__ __forceinline__ FE warp_sum_fe(FE x) {
    const bool has = x.v > 0.0f;
    int em = has ? x.e : -(1 << 30);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) em = max(em, __shfl_xor_sync(0xffffffffu, em, o));
    float v = 0.0f;
    if (has) {
        const int d = x.e - em;
        if (d > -120) v = x.v * fpow2(d);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return {v, em};
}

// a thread's SqSum (in units of 2^e0) as a DfE; the FP64 spill is rare
__device__ __forceinline__ DfE sqsum_dfe(const SqSum& ss, int e0) {
    if (ss.x == 0.0) return {ss.d, e0};
    const double v = ss.value();
    if (!(v > 0.0) || !isfinite(v)) return {{0.0f, 0.0f}, e0};
    const int ex = exp_of(v);
    return {df_from_double(v * pow2(-ex)), e0 + ex};
}

// (h + l) 2^e in FP64 (the leader's combine)
__device__ __forceinline__ double dfe_to_double(DfE x) {
    if (!(x.v.h > 0.0f)) return 0.0;
    return (f2d(x.v.h) + f2d(x.v.l)) * pow2(max(-1000, min(1000, x.e)));
}

// ------------------------------------------------------- double-float sides
struct SharedDF {
    Mat2 wtot[kLongWarps], wpre[kLongWarps];
    Scal qtot[kLongWarps], qpre[kLongWarps];
    int nodes[kLongWarps];
    DfE s[kLongWarps];  // warp partial sums of psi-hat^2, absolute exponents
    int pk_L[kLongWarps], pk_s[kLongWarps];
    double gb[kLongWarps];  // MODE 5: warp minima of |gamma| and their points
    int gk[kLongWarps];
    // the side's final state (written by the thread holding the last chunk)
    dfl A, D, q;
    int eA, eQ;
    // the leader's broadcasts: the pass energy and the pass result
    dfl aE;
    PassDF res;
    int word;  // grp_bcast / grp_next slot
};

// One side of a pass over steps 0..nsteps-1 (point from + dir * step), the
// group-parallel twin of side_df<MODE>: the same outputs in the same scales
// (state and psi-hat at the end with their exponents, S relative to the
// final scale, peak in absolute log2), valid in the leader.  Called by every
// thread of the group.
template <int MODE>
struct LongSide {
    dfl A, D, q;
    int eA, eQ;
    int nodes;
    double S;
    int peak_L, peak_i;
};

// The twist-index search (MODE 4: outward sweep storing the sampled ratios,
// MODE 5: inward sweep forming |gamma_k| at the same samples) reuses the
// state-only chunked march; this is its scratch and result (the result is
// handed to every thread of the group).
struct TwistIO {
    double* rho;        // sampled outward ratios (one every kTwistSample points from j0)
    const double* W;    // a V (FP64) of the potential
    double aEd;         // a E in FP64
    int j0, j1, stride;
    double best;        // MODE 5 result: min |gamma_k| over the samples
    int k;              //   and its point
};

template <int MODE>
__device__ LongSide<MODE> long_side(const Grp& G, const float2* __restrict__ Wf, dfl aE, int from, int to,
                                    int dir, double* __restrict__ out, double L, int Xk, SharedDF& sh,
                                    TwistIO* tw = nullptr) {
    // MODE 0: state, 1: + sums/peak, 2: + psi write, 3: MODE 1 + unnormalised
    // psi-hat written in the absolute scale, 4/5: twist sweeps (state)
    constexpr bool kPsi = MODE == 1 || MODE == 2 || MODE == 3;
    constexpr bool kSums = MODE == 1 || MODE == 3;
    constexpr int kT = Grp::kThreads;
    const int tid = G.t(), lane = G.lane(), warp = G.warp();
    const int nsteps = (to - from) * dir;
    LongSide<MODE> res;
    if (nsteps <= 0) {  // uniform over the group: no barrier is skipped by part of it
        res.A = {1.0f, 0.0f};
        res.D = {1.0f, 0.0f};
        res.q = {1.0f, 0.0f};
        res.eA = res.eQ = 0;
        res.nodes = 0;
        res.S = 0.0;
        res.peak_L = -(1 << 30);
        res.peak_i = from;
        if (MODE == 5) {
            tw->best = INFINITY;
            tw->k = 0x7fffffff;
        }
        return res;
    }
    const int len = (nsteps + kT - 1) / kT;
    const int s0 = min(tid * len, nsteps), s1 = min(s0 + len, nsteps);

    // ---- phase 1: this chunk's transfer matrix (and product of 1/f)
    Mat2 M;
    Scal P{{1.0f, 0.0f}, 0};
    {
        dfl A1 = {1.0f, 0.0f}, D1 = {0.0f, 0.0f}, A2 = {0.0f, 0.0f}, D2 = {1.0f, 0.0f};
        int e = 0;
        for (int st = s0; st < s1; ++st) {
            const dfl T = t_of(aE, __ldg(Wf + from + dir * st));
            if (kPsi) P.v = df_mul(P.v, df_recip(df_add({1.0f, 0.0f}, T)));
            df_step(T, A1, D1);
            df_step(T, A2, D2);
            if (((st - s0) & 7) == 7) {
                const float mm = fmaxf(fmaxf(fabsf(A1.h), fabsf(D1.h)), fmaxf(fabsf(A2.h), fabsf(D2.h)));
                if (mm > 0.0f && mm < INFINITY) {
                    const int ee = max(-120, min(120, fexp(mm)));
                    const float sc = fpow2(-ee);
                    A1 = df_scale(A1, sc);
                    D1 = df_scale(D1, sc);
                    A2 = df_scale(A2, sc);
                    D2 = df_scale(D2, sc);
                    e += ee;
                }
                if (kPsi) scal_norm(P);
            }
        }
        M = {A1, A2, D1, D2, e};
        mat_norm(M);
        if (kPsi) scal_norm(P);
    }

    // ---- phase 2: exclusive prefix of the transfer matrices (later chunks on the left)
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const Mat2 y = shfl_up_mat(M, o);
        const Scal py = shfl_up_scal(P, o);
        if (lane >= o) {
            M = mat_mul(M, y);
            if (kPsi) P = scal_mul(P, py);
        }
    }
    Mat2 Mx = shfl_up_mat(M, 1);
    Scal Px = shfl_up_scal(P, 1);
    if (lane == 31) {
        sh.wtot[warp] = M;
        sh.qtot[warp] = P;
    }
    __syncthreads();
    if (tid == 0) {
        Mat2 acc = mat_identity();
        Scal qa{{1.0f, 0.0f}, 0};
        for (int w = 0; w < kLongWarps; ++w) {
            sh.wpre[w] = acc;
            sh.qpre[w] = qa;
            acc = mat_mul(sh.wtot[w], acc);
            if (kPsi) qa = scal_mul(sh.qtot[w], qa);
        }
    }
    __syncthreads();
    if (lane == 0) {
        Mx = sh.wpre[warp];
        Px = sh.qpre[warp];
    } else {
        Mx = mat_mul(Mx, sh.wpre[warp]);
        if (kPsi) Px = scal_mul(Px, sh.qpre[warp]);
    }

    // ---- phase 3: this chunk from its starting state (A, D) = Mx (1, 1)
    dfl A = df_add(Mx.a, Mx.b), D = df_add(Mx.c, Mx.d);
    int eA = Mx.e;
    {
        const float mm = fmaxf(fabsf(A.h), fabsf(D.h));
        if (mm > 0.0f && mm < INFINITY) {
            const int e = max(-120, min(120, fexp(mm)));
            const float sc = fpow2(-e);
            A = df_scale(A, sc);
            D = df_scale(D, sc);
            eA += e;
        }
    }
    dfl q = Px.v;
    int eQ = Px.e;
    PsiTag tag = psi_tag(MODE == 3 ? eA + eQ : 0);  // the stored pairs' scale and tag
    int nodes = 0;
    SqSum ss;
    ss.init();
    int peak_L = -(1 << 30), peak_s = 0x7fffffff;
    dfl F = {0.0f, 0.0f};
    if (MODE == 2) F = df_from_double(L * pow2(min(1000, max(-1000, eA + eQ - Xk))));
    double g_best = INFINITY;  // MODE 5
    int g_k = 0x7fffffff;
    for (int st = s0; st < s1; ++st) {
        const int i = from + dir * st;
        const dfl T = t_of(aE, __ldg(Wf + i));
        if (MODE == 4 || MODE == 5) {
            // twist search samples, before the step at i: outward, D/A of the
            // outward state; inward, gamma_i = -12 T_i / f_i + (D/A)_out +
            // (D/A)_in (the lane twist search's formula)
            const int rel = i - tw->j0;
            if (rel % kTwistSample == 0 && rel / kTwistSample < tw->stride) {
                const double ratio = df_to_double(D) / df_to_double(A);
                if (MODE == 4) {
                    tw->rho[rel / kTwistSample] = ratio;
                } else if (i <= tw->j1 - 1) {
                    const double Ti = tw->aEd - __ldg(tw->W + i);
                    const double gam = fabs(-12.0 * Ti / (1.0 + Ti) + tw->rho[rel / kTwistSample] + ratio);
                    if (gam < g_best || (gam == g_best && i < g_k)) {
                        g_best = gam;
                        g_k = i;
                    }
                }
            }
        }
        if (kPsi) {
            const dfl f = df_add({1.0f, 0.0f}, T);
            const dfl qn = df_mul(q, df_recip(f));
            const dfl psi = df_mul(A, qn);
            if (kSums) {
                const float p = __fmul_rn(psi.h, psi.h);
                const float e = __fmaf_rn(psi.h, psi.h, -p);
                ss.add({p, __fmaf_rn(2.0f * psi.h, psi.l, e)});
                if (MODE == 3 && out) store_psi_pair(out, i, psi, tag);  // absolute scale (as side_df)
            } else {
                const dfl v = df_mul(psi, F);
                out[i] = f2d(v.h) + f2d(v.l);
            }
            q = qn;
        }
        const dfl X = df_add(D, df_mulf(A, -12.0f));
        D = df_add(D, df_mul(T, X));
        const dfl An = df_add(A, df_add(df_mul(T, A), D));
        nodes += (__float_as_uint(An.h) ^ __float_as_uint(A.h)) >> 31;
        A = An;
        if (((st - s0) & 7) == 7 || st == s1 - 1) {
            const float mm = fmaxf(fabsf(A.h), fabsf(D.h));
            int e = 0, eq = 0;
            if (mm > 0.0f && mm < INFINITY) {
                e = max(-120, min(120, fexp(mm)));
                const float sc = fpow2(-e);
                A = df_scale(A, sc);
                D = df_scale(D, sc);
                eA += e;
            }
            if (kPsi) {
                eq = max(-120, min(120, fexp(q.h)));
                q = df_scale(q, fpow2(-eq));
                eQ += eq;
                if (kSums) {
                    ss.rescale(-2 * (e + eq));
                    if (MODE == 3) tag = psi_tag(eA + eQ);
                    const float mag = fabsf(__fmul_rn(A.h, q.h));
                    if (mag > 0.0f) {
                        const int Lm = fexp(mag) + eA + eQ;
                        if (Lm > peak_L) {
                            peak_L = Lm;
                            peak_s = st;
                        }
                    }
                } else if (e + eq != 0) {
                    F = df_from_double(L * pow2(min(1000, max(-1000, eA + eQ - Xk))));
                }
            }
        }
    }

    // ---- reductions: over each warp with shuffles, over the warps by the leader
    const int t_last = (nsteps - 1) / len;
    if (tid == t_last) {
        sh.A = A;
        sh.D = D;
        sh.q = q;
        sh.eA = eA;
        sh.eQ = eQ;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nodes += __shfl_xor_sync(0xffffffffu, nodes, o);
    DfE sw{{0.0f, 0.0f}, 0};
    if (kSums) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const int L2 = __shfl_xor_sync(0xffffffffu, peak_L, o);
            const int s2 = __shfl_xor_sync(0xffffffffu, peak_s, o);
            if (L2 > peak_L || (L2 == peak_L && s2 < peak_s)) {
                peak_L = L2;
                peak_s = s2;
            }
        }
        // this chunk's sum in the absolute scale 2^(2 (eA + eQ))
        sw = warp_sum_dfe(s1 > s0 ? sqsum_dfe(ss, 2 * (eA + eQ)) : DfE{{0.0f, 0.0f}, 0});
    }
    if (MODE == 5) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double g2 = __shfl_xor_sync(0xffffffffu, g_best, o);
            const int k2 = __shfl_xor_sync(0xffffffffu, g_k, o);
            if (g2 < g_best || (g2 == g_best && k2 < g_k)) {
                g_best = g2;
                g_k = k2;
            }
        }
    }
    if (lane == 0) {
        sh.nodes[warp] = nodes;
        sh.pk_L[warp] = peak_L;
        sh.pk_s[warp] = peak_s;
        if (kSums) sh.s[warp] = sw;
        if (MODE == 5) {
            sh.gb[warp] = g_best;
            sh.gk[warp] = g_k;
        }
    }
    __syncthreads();
    if (G.leader()) {
        res.A = sh.A;
        res.D = sh.D;
        res.q = sh.q;
        res.eA = sh.eA;
        res.eQ = sh.eQ;
        int nsum = 0;
        double Ssum = 0.0;
        int pL = -(1 << 30), ps = 0x7fffffff;
        for (int w = 0; w < kLongWarps; ++w) {
            nsum += sh.nodes[w];
            if (kSums) {
                // the warp's sum in the side's final scale
                DfE x = sh.s[w];
                x.e -= 2 * (res.eA + res.eQ);
                Ssum += dfe_to_double(x);
                if (sh.pk_L[w] > pL || (sh.pk_L[w] == pL && sh.pk_s[w] < ps)) {
                    pL = sh.pk_L[w];
                    ps = sh.pk_s[w];
                }
            }
        }
        res.nodes = nsum;
        res.S = Ssum;
        res.peak_L = pL;
        res.peak_i = ps == 0x7fffffff ? from : from + dir * ps;
    }
    if (MODE == 5) {
        // every thread of the group takes the search's result
        double gb = INFINITY;
        int gk = 0x7fffffff;
        for (int w = 0; w < kLongWarps; ++w)
            if (sh.gb[w] < gb || (sh.gb[w] == gb && sh.gk[w] < gk)) {
                gb = sh.gb[w];
                gk = sh.gk[w];
            }
        tw->best = gb;
        tw->k = gk;
    }
    // (no barrier here: the next writes of these fields come after the next
    // call's phase-2 barriers, which the leader reaches only after its reads)
    return res;
}

// One pass at E with match point k (the group twin of pass_df<MODE>): the
// leader turns the two sides into the Cooley correction, the count, the sum
// and the peak, and hands the result to the group.  MODE 3 also stores the
// unnormalised psi-hat of the window in row (if not null).
template <int MODE>
__device__ __forceinline__ PassDF long_pass(const Grp& G, const PotMeta& m, const LevelWork& w,
                                            const float2* __restrict__ Wf, const double* __restrict__ W64, double E,
                                            int k, double sum_fallback, SharedDF& sh,
                                            double* __restrict__ row = nullptr) {
    if (G.leader()) sh.aE = energy_df(m, E);
    __syncthreads();
    const dfl aE = sh.aE;
    const LongSide<MODE> o = long_side<MODE>(G, Wf, aE, w.j0, k, +1, row, 0.0, 0, sh);
    const LongSide<MODE> in = long_side<MODE>(G, Wf, aE, w.j1, k, -1, row, 0.0, 0, sh);
    if (G.leader()) {
        const double Tk = __dsub_rn(__dmul_rn(m.a, E), __ldg(W64 + k));
        const double fk = 1.0 + Tk;
        const double Ao = df_to_double(o.A), Do = df_to_double(o.D);
        const double Ai = df_to_double(in.A), Di = df_to_double(in.D);
        PassDF r;
        r.gamma = -12.0 * Tk / fk + Do / Ao + Di / Ai;
        r.nodes = o.nodes + in.nodes;
        r.count = r.nodes + (r.gamma < 0.0 ? 1 : 0);
        r.peak_i = k;
        r.peak_log2 = 0;
        r.pk_out = r.pk_in = 0.0;
        r.ex_out = r.ex_in = 0;
        if (MODE == 1 || MODE == 3) {
            const double rfk = 1.0 / fk;
            r.pk_out = Ao * df_to_double(o.q) * rfk;
            r.pk_in = Ai * df_to_double(in.q) * rfk;
            r.ex_out = o.eA + o.eQ;
            r.ex_in = in.eA + in.eQ;
            r.sum = o.S / (r.pk_out * r.pk_out) + in.S / (r.pk_in * r.pk_in) + 1.0;
            const int Lo = (r.pk_out != 0.0 ? exp_of(fabs(r.pk_out)) : -1000) + r.ex_out;
            const int Li = (r.pk_in != 0.0 ? exp_of(fabs(r.pk_in)) : -1000) + r.ex_in;
            const int po = o.peak_L - Lo, pi = in.peak_L - Li;
            r.peak_log2 = max(po, pi);
            r.peak_i = po >= pi ? o.peak_i : in.peak_i;
        } else {
            r.sum = sum_fallback;
        }
        r.dE = r.gamma * fk * fk / (12.0 * m.a * r.sum);
        sh.res = r;
    }
    __syncthreads();
    return sh.res;
}

// ------------------------------------------------------------------ FP32 passes
// The CTA-parallel twin of the lane kernel's FP32 Cooley pass (refine32): the
// same FP32 recurrence and sums, chunked and scanned as above.  It takes a
// long level from its scan bracket to ~1e-9 at ~1/7 of a double-float pass's
// cost; the double-float passes then only finish the last digits.

// [[a, b], [c, d]] 2^e in FP32
struct Mat2f {
    float a, b, c, d;
    int e;
};

struct Scalf {
    float v;
    int e;
};

__device__ __forceinline__ void matf_norm(Mat2f& m) {
    const float mm = fmaxf(fmaxf(fabsf(m.a), fabsf(m.b)), fmaxf(fabsf(m.c), fabsf(m.d)));
    if (mm > 0.0f && mm < INFINITY) {
        const int e = max(-120, min(120, fexp(mm)));
        const float sc = fpow2(-e);
        m.a *= sc;
        m.b *= sc;
        m.c *= sc;
        m.d *= sc;
        m.e += e;
    }
}

// x y (x applied after y)
__device__ __forceinline__ Mat2f matf_mul(const Mat2f& x, const Mat2f& y) {
    Mat2f r;
    r.a = fmaf(x.a, y.a, x.b * y.c);
    r.b = fmaf(x.a, y.b, x.b * y.d);
    r.c = fmaf(x.c, y.a, x.d * y.c);
    r.d = fmaf(x.c, y.b, x.d * y.d);
    r.e = x.e + y.e;
    matf_norm(r);
    return r;
}

__device__ __forceinline__ void scalf_norm(Scalf& s) {
    const float mm = fabsf(s.v);
    if (mm > 0.0f && mm < INFINITY) {
        const int e = max(-120, min(120, fexp(mm)));
        s.v *= fpow2(-e);
        s.e += e;
    }
}

__device__ __forceinline__ Scalf scalf_mul(const Scalf& x, const Scalf& y) {
    Scalf r{x.v * y.v, x.e + y.e};
    scalf_norm(r);
    return r;
}

__device__ __forceinline__ Mat2f shfl_up_matf(const Mat2f& m, int o) {
    return {__shfl_up_sync(0xffffffffu, m.a, o), __shfl_up_sync(0xffffffffu, m.b, o),
            __shfl_up_sync(0xffffffffu, m.c, o), __shfl_up_sync(0xffffffffu, m.d, o),
            __shfl_up_sync(0xffffffffu, m.e, o)};
}

__device__ __forceinline__ Scalf shfl_up_scalf(const Scalf& s, int o) {
    return {__shfl_up_sync(0xffffffffu, s.v, o), __shfl_up_sync(0xffffffffu, s.e, o)};
}

struct Shared32 {
    Mat2f wtot[kLongWarps], wpre[kLongWarps];
    Scalf ftot[kLongWarps], fpre[kLongWarps];
    Scalf fall;  // product of f^2 over the side
    int nodes[kLongWarps];
    FE s[kLongWarps];  // warp partial sums, absolute exponents
    int pk_L[kLongWarps], pk_s[kLongWarps];
    float A, D;  // the side's final state (thread holding the last chunk)
    int eA;
    // the leader's broadcasts: a E as a float pair and the pass result
    float aEh, aEl;
    PassDF res;
};

struct LongSide32 {
    float A, D;
    int eA;      // the final state is (A, D) 2^eA
    int nodes;
    double S;    // sum_j A_j^2 prod_{l>j} f_l^2 over the side, in units of 2^(2 eA)
    int peak_L;  // log2 of the largest |A_j| seen at the renormalisations
    int peak_i;
};

// One side in FP32 over steps 0..nsteps-1 (point from + dir * step): the
// state, the node count, the sum S and the peak of |A| exactly as the lane
// pass accumulates them (S' = f^2 S + A^2 before each step), chunked: phase 1
// gives each chunk's transfer matrix and product F of f^2, phase 2 scans
// them, phase 3 re-runs the chunk from its exact start state; a chunk's S is
// carried to the side's end by the product of F over the later chunks.  The
// result is valid in the leader.
__device__ LongSide32 long_side32(const Grp& G, const float2* __restrict__ Wf, float aEh, float aEl, int from,
                                  int to, int dir, Shared32& sh) {
    constexpr int kT = Grp::kThreads;
    const int tid = G.t(), lane = G.lane(), warp = G.warp();
    const int nsteps = (to - from) * dir;
    LongSide32 res;
    if (nsteps <= 0) {  // uniform over the group
        res.A = 1.0f;
        res.D = 1.0f;
        res.eA = 0;
        res.nodes = 0;
        res.S = 0.0;
        res.peak_L = -(1 << 30);
        res.peak_i = from;
        return res;
    }
    const int len = (nsteps + kT - 1) / kT;
    const int s0 = min(tid * len, nsteps), s1 = min(s0 + len, nsteps);

    // ---- phase 1: transfer matrix and product of f^2 of this chunk
    Mat2f M;
    Scalf F{1.0f, 0};
    {
        float A1 = 1.0f, D1 = 0.0f, A2 = 0.0f, D2 = 1.0f;
        int e = 0;
        for (int st = s0; st < s1; ++st) {
            const float2 w = __ldg(Wf + from + dir * st);
            const float T = (aEh - w.x) + (aEl - w.y);
            const float f = 1.0f + T;
            F.v *= f * f;
            float X = fmaf(-12.0f, A1, D1);
            D1 = fmaf(T, X, D1);
            A1 = A1 + fmaf(T, A1, D1);
            X = fmaf(-12.0f, A2, D2);
            D2 = fmaf(T, X, D2);
            A2 = A2 + fmaf(T, A2, D2);
            if (((st - s0) & 7) == 7) {
                const float mm = fmaxf(fmaxf(fabsf(A1), fabsf(D1)), fmaxf(fabsf(A2), fabsf(D2)));
                if (mm > 0.0f && mm < INFINITY) {
                    const int ee = max(-120, min(120, fexp(mm)));
                    const float sc = fpow2(-ee);
                    A1 *= sc;
                    D1 *= sc;
                    A2 *= sc;
                    D2 *= sc;
                    e += ee;
                }
                scalf_norm(F);
            }
        }
        M = {A1, A2, D1, D2, e};
        matf_norm(M);
        scalf_norm(F);
    }

    // ---- phase 2: exclusive prefix of the matrices, inclusive prefix of F
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const Mat2f y = shfl_up_matf(M, o);
        const Scalf fy = shfl_up_scalf(F, o);
        if (lane >= o) {
            M = matf_mul(M, y);
            F = scalf_mul(F, fy);
        }
    }
    Mat2f Mx = shfl_up_matf(M, 1);
    Scalf Fin = F;  // f^2 over the chunks up to this thread's
    Scalf Fall;     // f^2 over the side
    if (lane == 31) {
        sh.wtot[warp] = M;
        sh.ftot[warp] = F;
    }
    __syncthreads();
    if (tid == 0) {
        Mat2f acc = {1.0f, 0.0f, 0.0f, 1.0f, 0};
        Scalf fa{1.0f, 0};
        for (int w = 0; w < kLongWarps; ++w) {
            sh.wpre[w] = acc;
            sh.fpre[w] = fa;
            acc = matf_mul(sh.wtot[w], acc);
            fa = scalf_mul(sh.ftot[w], fa);
        }
        sh.fall = fa;
    }
    __syncthreads();
    if (lane == 0) Mx = sh.wpre[warp];
    else Mx = matf_mul(Mx, sh.wpre[warp]);
    Fin = scalf_mul(F, sh.fpre[warp]);
    Fall = sh.fall;

    // ---- phase 3: this chunk from its start state (A, D) = Mx (1, 1)
    float A = Mx.a + Mx.b, D = Mx.c + Mx.d;
    int eA = Mx.e;
    {
        const float mm = fmaxf(fabsf(A), fabsf(D));
        if (mm > 0.0f && mm < INFINITY) {
            const int e = max(-120, min(120, fexp(mm)));
            const float sc = fpow2(-e);
            A *= sc;
            D *= sc;
            eA += e;
        }
    }
    float S = 0.0f;  // in units of 2^(2 eA)
    int nodes = 0;
    int peak_L = -(1 << 30), peak_s = 0x7fffffff;
    for (int st = s0; st < s1; ++st) {
        const float2 w = __ldg(Wf + from + dir * st);
        const float T = (aEh - w.x) + (aEl - w.y);
        const float f = 1.0f + T;
        S = fmaf(f * f, S, A * A);
        const float X = fmaf(-12.0f, A, D);
        D = fmaf(T, X, D);
        const float An = A + fmaf(T, A, D);
        nodes += (__float_as_uint(An) ^ __float_as_uint(A)) >> 31;
        A = An;
        if (((st - s0) & 7) == 7 || st == s1 - 1) {
            const float mm = fmaxf(fabsf(A), fabsf(D));
            if (mm > 0.0f && mm < INFINITY) {
                const int e = max(-60, min(60, fexp(mm)));
                const float sc = fpow2(-e);
                A *= sc;
                D *= sc;
                S *= sc * sc;
                eA += e;
            }
            if (A != 0.0f) {
                const int L = eA + fexp(fabsf(A));
                if (L > peak_L) {
                    peak_L = L;
                    peak_s = st;
                }
            }
        }
    }

    // ---- reductions
    const int t_last = (nsteps - 1) / len;
    if (tid == t_last) {
        sh.A = A;
        sh.D = D;
        sh.eA = eA;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        nodes += __shfl_xor_sync(0xffffffffu, nodes, o);
        const int L2 = __shfl_xor_sync(0xffffffffu, peak_L, o);
        const int s2 = __shfl_xor_sync(0xffffffffu, peak_s, o);
        if (L2 > peak_L || (L2 == peak_L && s2 < peak_s)) {
            peak_L = L2;
            peak_s = s2;
        }
    }
    // this chunk's S carried to the side's end (times f^2 over the later
    // chunks = F_all / F_in), in the absolute scale: S (Fall.v / Fin.v)
    // 2^(2 eA + Fall.e - Fin.e)
    FE x{0.0f, 0};
    if (s1 > s0 && S != 0.0f && Fin.v != 0.0f) x = {S * __fdividef(Fall.v, Fin.v), 2 * eA + Fall.e - Fin.e};
    const FE sw = warp_sum_fe(x);
    if (lane == 0) {
        sh.nodes[warp] = nodes;
        sh.pk_L[warp] = peak_L;
        sh.pk_s[warp] = peak_s;
        sh.s[warp] = sw;
    }
    __syncthreads();
    if (G.leader()) {
        res.A = sh.A;
        res.D = sh.D;
        res.eA = sh.eA;
        int nsum = 0;
        double Ssum = 0.0;
        int pL = -(1 << 30), ps = 0x7fffffff;
        for (int w = 0; w < kLongWarps; ++w) {
            nsum += sh.nodes[w];
            const FE s = sh.s[w];
            if (s.v > 0.0f) Ssum += (double)s.v * pow2(max(-1000, min(1000, s.e - 2 * res.eA)));
            if (sh.pk_L[w] > pL || (sh.pk_L[w] == pL && sh.pk_s[w] < ps)) {
                pL = sh.pk_L[w];
                ps = sh.pk_s[w];
            }
        }
        res.nodes = nsum;
        res.S = Ssum;
        res.peak_L = pL;
        res.peak_i = ps == 0x7fffffff ? from : from + dir * ps;
    }
    return res;
}

// One FP32 pass at E with match point k (the group twin of the lane pass):
// Cooley correction, count, sum and the peak of |psi| relative to psi_k,
// formed by the leader and handed to the group.
__device__ __forceinline__ PassDF long_pass32(const Grp& G, const PotMeta& m, const LevelWork& w,
                                              const float2* __restrict__ Wf, const double* __restrict__ W64,
                                              double E, int k, Shared32& sh) {
    if (G.leader()) {
        const double aE = __dmul_rn(m.a, E);
        const float aEh = __double2float_rn(aE);
        sh.aEh = aEh;
        sh.aEl = __double2float_rn(aE - (double)aEh);
    }
    __syncthreads();
    const float aEh = sh.aEh, aEl = sh.aEl;
    const LongSide32 o = long_side32(G, Wf, aEh, aEl, w.j0, k, +1, sh);
    const LongSide32 in = long_side32(G, Wf, aEh, aEl, w.j1, k, -1, sh);
    if (G.leader()) {
        const double aE = __dmul_rn(m.a, E);
        const double Tk = aE - __ldg(W64 + k);
        const double fk = 1.0 + Tk;
        const double uA = o.A, vC = in.A;
        PassDF r;
        // gamma_k = -12 T_k / f_k + D_o / u_k + D_i / v_k   (no cancellation)
        r.gamma = -12.0 * Tk / fk + (double)o.D / uA + (double)in.D / vC;
        const double fk2 = fk * fk;
        r.sum = fk2 * (o.S / (uA * uA) + in.S / (vC * vC)) + 1.0;
        r.dE = r.gamma * fk2 / (12.0 * m.a * r.sum);
        r.nodes = o.nodes + in.nodes;
        r.count = r.nodes + (r.gamma < 0.0 ? 1 : 0);
        const int Lo = o.eA + (o.A != 0.0f ? fexp(fabsf(o.A)) : -1000);
        const int Li = in.eA + (in.A != 0.0f ? fexp(fabsf(in.A)) : -1000);
        const int po = o.peak_L - Lo, pi = in.peak_L - Li;
        r.peak_log2 = max(po, pi);
        r.peak_i = po >= pi ? o.peak_i : in.peak_i;
        r.pk_out = r.pk_in = 0.0;
        r.ex_out = r.ex_in = 0;
        sh.res = r;
    }
    __syncthreads();
    return sh.res;
}

// whether the host asked to stop, looked up by the leader and handed to the
// group (threads that look separately could see it change between their reads
// and part at the next barrier)
__device__ __forceinline__ bool grp_cancelled(const Grp& G, const DevBatch& b, int q, int& slot) {
    return grp_bcast(G, G.leader() && stop_asked(b, (q & 15) == 0) ? 1 : 0, slot) != 0;
}

// The refinement of a level, in up to three stages:
//   1. FP32 passes (long_pass32): safeguarded Cooley-Newton with the count
//      bracket, the match point moved to the peak of |psi|, until a Newton
//      step of at most kTol32Long is taken (the energy after it is then far
//      inside stage 2's first-pass acceptance);
//   2. double-float state-only passes with the FP32 sum as the Newton
//      denominator (as newton_df): usually one step, accepted from within
//      1e-8 (the chunked FP32 sum is accurate to ~1e-6);
//   3. if stage 2 does not settle (the FP32 counts are off near a trial
//      energy, or the pass sees another node count): safeguarded
//      Cooley-Newton in double-float with full sums from the scan bracket
//      widened by one trial spacing.  Every pass updates the count bracket;
//      Newton steps are taken only while the pass sees the level's own node
//      count (so a neighbouring level cannot attract the iteration) and stay
//      inside the bracket, bisection otherwise.  After the match point moves
//      to the peak of |psi| the pass is redone at the same E.
// mode 0: the long list (stages 1-3); 1: the levels newton_df handed over
// (stage 3 only); 2: the middle list, whose FP32 refinement the lane kernel
// refine32 did (stage 2 from its energy, bracket, match point and sum, with
// newton_df's acceptance rule, then stage 3 if it does not settle).  Every
// thread of a group runs the same control flow on the leader's pass results
// (the group's passes are collective).
// (Measured on the 2048-potential batch, refine_long / step: 2e-9 7.8 /
// 30.0 ms, 1e-8 7.4 / 29.8, 3e-8 7.4 / 29.6, 1e-7 7.0 / 29.6 with more
// double-float passes after it.)
constexpr double kTol32Long = 3e-8;

__device__ __noinline__ void refine_cta(const Grp& G, const DevBatch& b, LevelWork& w, bool fallback, SharedDF& sh,
                                        Shared32& sh32) {
    const PotMeta m = b.meta[w.p];
    const float2* Wf = b.Wf2 + m.offf;
    const double* W = b.W64 + m.off;
    double lo = w.lo, hi = w.hi, E = w.E, sum = 1.0;
    int k = grp_bcast(G, G.leader() ? clamp_k(w, match_index(m, b, E)) : 0, sh.word);
    bool done = false;
    int n_pass = 0, n_pass32 = 0;
    if (!fallback) {
        // ---- stage 1: FP32
        bool moved_last = false, ok32 = false;
        for (int it = 0, cap = refine_cap(b); it < cap; ++it) {
            const PassDF r = long_pass32(G, m, w, Wf, W, E, k, sh32);
            ++n_pass32;
            sum = r.sum;
            if (r.count > w.v) hi = E;
            else lo = E;
            if (r.peak_log2 >= 2 && !moved_last) {
                k = clamp_k(w, r.peak_i);
                moved_last = true;
                continue;  // the same energy at the new match point
            }
            moved_last = false;
            const double En = E + r.dE;
            const bool near = r.nodes == w.v || (m.status & EPSCU_STATUS_UNDER);
            if (near && isfinite(En) && En > lo && En < hi) {
                E = En;
                if (fabs(r.dE) <= kTol32Long) {
                    ok32 = true;
                    break;
                }
            } else {
                E = 0.5 * (lo + hi);
            }
            if (hi - lo <= 2.0 * kTol32Long) {
                E = 0.5 * (lo + hi);
                ok32 = true;
                break;
            }
        }
        // ---- stage 2: double-float state-only Newton (FP32 sum)
        if (ok32) {
            double lo2 = lo - 1e-8, hi2 = hi + 1e-8;
            for (int it = 0; it < 4 && !done; ++it) {
                const PassDF r = long_pass<0>(G, m, w, Wf, W, E, k, sum, sh);
                ++n_pass;
                if (r.count > w.v) hi2 = fmin(hi2, E);
                else lo2 = fmax(lo2, E);
                const double En = E + r.dE;
                if (!isfinite(En) || !(En >= lo2 && En <= hi2) || r.nodes != w.v) break;
                // the FP32 sum of the group pass is accurate to ~1e-6 (chunk
                // sums of a few hundred terms), so one step from within 1e-8
                // leaves ~1e-14: the first pass settles
                done = fabs(r.dE) <= (it == 0 ? 1e-8 * fmax(1.0, fabs(E)) : 1e-12 * fmax(1.0, fabs(E)));
                E = En;
            }
            if (done) {
                lo = lo2;
                hi = hi2;
            }
        }
    }
    if (!done) {
        // ---- stage 3: the FP32 bracket may be off by its count errors:
        // restart from the scan bracket widened by one trial spacing
        lo = fmax(m.e_lo, w.lo0 - m.delta);
        hi = fmin(m.e_cap, w.hi0 + m.delta);
        if (!(E > lo && E < hi)) E = 0.5 * (lo + hi);
        bool moved_last = false;
        for (int it = 0, cap = fallback_cap(b); it < cap; ++it) {
            const PassDF r = long_pass<1>(G, m, w, Wf, W, E, k, 1.0, sh);
            ++n_pass;
            sum = r.sum;
            if (r.count > w.v) hi = E;
            else lo = E;
            if (r.peak_log2 >= 2 && !moved_last) {
                k = clamp_k(w, r.peak_i);
                moved_last = true;
                continue;  // the same energy at the new match point
            }
            moved_last = false;
            const double tol = 1e-12 * fmax(1.0, fabs(E));
            const double En = E + r.dE;
            const bool near = r.nodes == w.v || (m.status & EPSCU_STATUS_UNDER);
            if (near && isfinite(En) && En > lo && En < hi) {
                E = En;
                if (fabs(r.dE) <= tol) {
                    done = true;
                    break;
                }
            } else {
                E = 0.5 * (lo + hi);
            }
            if (hi - lo <= tol) {
                E = 0.5 * (lo + hi);
                done = true;
                break;
            }
        }
    }
    if (!done) w.status |= EPSCU_STATUS_MAXITER;
    w.lo = lo;
    w.hi = hi;
    w.E = E;
    w.k = k;
    w.norm_k_in = sum;
    w.iters = n_pass32 + n_pass;
    if (G.leader()) {
        const unsigned long long pts = (unsigned long long)(w.j1 - w.j0);
        atomicAdd(&b.hdr->refine_updates, (unsigned long long)n_pass32 * pts);
        atomicAdd(&b.hdr->df_updates, (unsigned long long)n_pass * pts);
    }
}

// The norm pass of a level and its match-point candidates (as norm_df_level).
// With psi requested every pass also stores its unnormalised psi-hat (MODE 3)
// and the last pass is the one kept.  Returns whether the twist search is due.
__device__ __noinline__ bool norm_cta(const Grp& G, const DevBatch& b, LevelWork& w, double* row, SharedDF& sh) {
    const PotMeta m = b.meta[w.p];
    const float2* Wf = b.Wf2 + m.offf;
    const double* W = b.W64 + m.off;
    auto pass = [&](int kk) { return long_pass<3>(G, m, w, Wf, W, w.E, kk, 1.0, sh, row); };
    int k = w.k;
    PassDF r = pass(k);
    if (r.peak_log2 >= 2) {
        k = clamp_k(w, r.peak_i);
        r = pass(k);
    }
    int k_row = k;  // the pass whose psi-hat the row holds
    if (r.nodes != w.v) {
        const int kt = grp_bcast(G, G.leader() ? clamp_k(w, match_index(m, b, w.E)) : 0, sh.word);
        PassDF r2 = pass(kt);
        int k2 = kt;
        if (r2.nodes != w.v && r2.peak_log2 >= 1) {
            k2 = clamp_k(w, r2.peak_i);
            r2 = pass(k2);
        }
        k_row = k2;
        if (r2.nodes == w.v) {
            r = r2;
            k = k2;
        }
    }
    if (redo_norm(w, r)) {
        if (G.leader()) atomicAdd(&b.hdr->n_redo, 1);
        w.E += r.dE;
        r = pass(k);
    } else if (row && k_row != k) {
        r = pass(k);
    }
    finalize_df(m, w, r, k);
    return suspicious(m, w, r.nodes, r.dE);
}

// Twist-index search for a flagged level (any window length): a chunked
// outward sweep stores D/A every kTwistSample points, a chunked inward sweep
// forms |gamma_k| at the same points, the match point becomes argmin
// |gamma_k| (Dhillon and Parlett's twisted-factorisation rule), then Newton
// and the norm pass run there.
__device__ __noinline__ void twist_cta(const Grp& G, const DevBatch& b, LevelWork& w, double* row, SharedDF& sh) {
    const PotMeta m = b.meta[w.p];
    const float2* Wf = b.Wf2 + m.offf;
    const double* W = b.W64 + m.off;
    const dfl aE = energy_df(m, w.E);
    TwistIO tw;
    tw.rho = b.twist_scratch + (int64_t)(kFragileScratch + blockIdx.x) * b.twist_stride;
    tw.W = W;
    tw.aEd = __dmul_rn(m.a, w.E);
    tw.j0 = w.j0;
    tw.j1 = w.j1;
    tw.stride = b.twist_stride;
    tw.best = INFINITY;
    tw.k = w.k;
    long_side<4>(G, Wf, aE, w.j0, w.j1, +1, nullptr, 0.0, 0, sh, &tw);
    long_side<5>(G, Wf, aE, w.j1, w.j0, -1, nullptr, 0.0, 0, sh, &tw);
    const int k = clamp_k(w, tw.k == 0x7fffffff ? w.k : tw.k);
    auto pass = [&](double e) { return long_pass<3>(G, m, w, Wf, W, e, k, 1.0, sh, row); };
    double E1 = w.E;
    PassDF r = pass(E1);
    for (int it = 0; it < 8; ++it) {
        if (r.nodes != w.v || !isfinite(r.dE) || !(fabs(r.dE) < 1e-7)) break;
        if (fabs(r.dE) <= 1e-13 * fmax(1.0, fabs(E1))) break;
        E1 += r.dE;
        r = pass(E1);
    }
    w.E = E1;
    finalize_df(m, w, r, k);
}

// ---------------------------------------------------------------- kernels

// levels to a warp, two lanes each (the windows and pass counts differ, and the
// levels are few: more to a warp would only lengthen it)
constexpr int kLaneLevels = 8;

__device__ __forceinline__ bool next_levels(const DevBatch& b, int qid, int per, int2& unit) {
    int u = 0;
    if ((threadIdx.x & 31) == 0) u = atomicAdd(&b.hdr->queue[qid], 1);
    u = __shfl_sync(0xffffffffu, u, 0);
    const int n = min(b.hdr->n_fragile, b.max_levels);
    if (u >= (n + per - 1) / per) return false;
    unit = make_int2(u * per, min(per, n - u * per));
    return true;
}

// The fragile levels: the CTAs first take the long windows, a CTA each, then
// their warps the others, of similar window length and longest first: FP32
// refinement, double-float Newton and norm pass back to back, then the rows by
// the warp.
__global__ void __launch_bounds__(kLongThreads, kLongCtasPerSm) fragile_kernel(DevBatch b) {
    __shared__ SharedDF sh;
    __shared__ Shared32 sh32;
    const Grp G;
    const int n_long = min(b.hdr->n_fragile_long, b.max_levels);
    for (;;) {
        const int q = grp_next(G, &b.hdr->queue[kQFragileLong], sh.word);
        if (q >= n_long) break;
        const int slot = b.fragile_long[q];
        LevelWork w = b.levels[slot];
        double* row = psi_row(b, b.meta[w.p], w);
        bool off = false;
        if (grp_cancelled(G, b, q, sh.word)) {
            w.status |= EPSCU_STATUS_CANCELLED;
        } else {
            refine_cta(G, b, w, false, sh, sh32);
            off = norm_cta(G, b, w, row, sh);
        }
        if (row) finish_row<kLongThreads>(G.t(), w, row, b.meta[w.p].N);
        if (G.leader()) {
            b.levels[slot] = w;
            if (off && b.fragile_twist) {
                const int t = atomicAdd(&b.hdr->n_fragile_twist, 1);
                if (t < b.max_twist) b.fragile_twist[t] = slot;
            }
        }
    }
    const int lane = threadIdx.x & 31;
    for (int2 unit; next_levels(b, kQFragileLanes, kLaneLevels, unit);) {
        if (lane / 2 < unit.y) {
            const int slot = b.fragile_list[unit.x + lane / 2];
            refine32_level(b, slot);
            newton_df_level(b, slot);
            norm_df_level(b, slot);
        }
        __syncwarp();
        if (!b.psi || b.hdr->error) continue;
        for (int u = 0; u < unit.y; ++u) {
            const LevelWork w = b.levels[b.fragile_list[unit.x + u]];
            if (w.status & EPSCU_STATUS_FALLBACK) continue;
            const PotMeta& m = b.meta[w.p];
            finish_row<32>(lane, w, psi_row(b, m, w), m.N);
        }
    }
}

// Levels the lane Newton handed over (refinement from the scan bracket
// widened by one trial spacing, norm pass), then those whose final pass
// disagrees.  Theirs are the CTA passes' constants from here on.
__global__ void __launch_bounds__(kLongThreads, kLongCtasPerSm) fragile_repair_kernel(DevBatch b) {
    __shared__ SharedDF sh;
    __shared__ Shared32 sh32;
    const Grp G;
    const int n_fall = min(b.hdr->n_fragile_fall, b.max_levels);
    const int n_twist = min(b.hdr->n_fragile_twist, b.max_twist);
    for (;;) {
        const int q = grp_next(G, &b.hdr->queue[kQFragileRepair], sh.word);
        if (q >= n_fall + n_twist) break;
        const int slot = q < n_fall ? b.fragile_fall[q] : b.fragile_twist[q - n_fall];
        LevelWork w = b.levels[slot];
        double* row = psi_row(b, b.meta[w.p], w);
        bool off = true;
        if (q < n_fall) {
            if (grp_cancelled(G, b, q, sh.word)) {
                w.status |= EPSCU_STATUS_CANCELLED;
                off = false;
            } else {
                refine_cta(G, b, w, true, sh, sh32);
                off = norm_cta(G, b, w, row, sh) && b.fragile_twist;
            }
        }
        if (off) twist_cta(G, b, w, row, sh);
        if (row) finish_row<kLongThreads>(G.t(), w, row, b.meta[w.p].N);
        if (G.leader()) {
            if (!is_long(w) && !(w.status & EPSCU_STATUS_FALLBACK)) {
                const int t = atomicAdd(&b.hdr->n_fragile_long, 1);
                if (t < b.max_levels) b.fragile_long[t] = slot;
                w.status |= EPSCU_STATUS_LONG;
            }
            b.levels[slot] = w;
        }
    }
}

// psi again from the final constants (the adjoint of a solve that kept none):
// the rows' zeros (the whole row of a level without a result), then the
// windows, a lane per level and a CTA for the long and the handed-over levels.
__global__ void __launch_bounds__(256) fragile_zero_kernel(DevBatch b) {
    if (!b.psi || b.hdr->error) return;
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, n_warps = (gridDim.x * blockDim.x) >> 5;
    const int total = b.hdr->total_levels;
    for (int slot = warp; slot < total; slot += n_warps) {
        const LevelWork w = b.levels[slot];
        const int list = w.bucket / kBuckets;
        if (list != kListFragile && list != kListFragileLong) continue;
        const int N = b.meta[w.p].N;
        double* row = psi_row(b, b.meta[w.p], w);
        const bool none = no_result(w);
        zero_points<32>(lane, row, none ? N : w.j0);
        if (!none) zero_points<32>(lane, row + w.j1 + 1, N - 1 - w.j1);
    }
}

__global__ void __launch_bounds__(128) fragile_write_lanes_kernel(DevBatch b) {
    if (!b.psi || b.hdr->error) return;
    const int lane = threadIdx.x & 31;
    for (int2 unit; next_levels(b, kQFragileRewrite, 32, unit);) {
        if (lane >= unit.y) continue;
        const LevelWork w = b.levels[b.fragile_list[unit.x + lane]];
        if (no_result(w) || is_long(w) || (w.status & EPSCU_STATUS_FALLBACK)) continue;
        const PotMeta m = b.meta[w.p];
        double* out = psi_row(b, m, w);
        const float2* Wf = b.Wf2 + m.offf;
        const dfl aE = energy_df(m, w.E);
        SideDF<2> st;
        side_df<2>(Wf, aE, w.j0, w.k, +1, st, out, w.norm_k_out, w.ex_out);
        side_df<2>(Wf, aE, w.j1, w.k, -1, st, out, w.norm_k_in, w.ex_in);
        out[w.k] = w.ck;
    }
}

__global__ void __launch_bounds__(kLongThreads, kLongCtasPerSm) fragile_write_long_kernel(DevBatch b) {
    __shared__ SharedDF sh;
    const Grp G;
    if (!b.psi || b.hdr->error) return;
    const int n_long = min(b.hdr->n_fragile_long, b.max_levels), n_fall = min(b.hdr->n_fragile_fall, b.max_levels);
    for (int q = blockIdx.x; q < n_long + n_fall; q += gridDim.x) {
        const LevelWork w = b.levels[q < n_long ? b.fragile_long[q] : b.fragile_fall[q - n_long]];
        if (no_result(w)) continue;
        const PotMeta m = b.meta[w.p];
        double* out = psi_row(b, m, w);
        const float2* Wf = b.Wf2 + m.offf;
        const dfl aE = energy_df(m, w.E);
        long_side<2>(G, Wf, aE, w.j0, w.k, +1, out, w.norm_k_out, w.ex_out, sh);
        long_side<2>(G, Wf, aE, w.j1, w.k, -1, out, w.norm_k_in, w.ex_in, sh);
        if (G.leader()) out[w.k] = w.ck;
        __syncthreads();  // the shared scratch is reused by the next level
    }
}

}  // namespace

void launch_fragile(const DevBatch& b, int sm_count, cudaStream_t s) {
    fragile_kernel<<<sm_count * kLongCtasPerSm, kLongThreads, 0, s>>>(b);
}
void launch_fragile_repair(const DevBatch& b, int sm_count, cudaStream_t s) {
    fragile_repair_kernel<<<sm_count * kLongCtasPerSm, kLongThreads, 0, s>>>(b);
}
void launch_fragile_rewrite(const DevBatch& b, int sm_count, cudaStream_t s) {
    fragile_zero_kernel<<<sm_count * 8, 256, 0, s>>>(b);
    fragile_write_lanes_kernel<<<sm_count * 8, 128, 0, s>>>(b);
    fragile_write_long_kernel<<<sm_count * kLongCtasPerSm, kLongThreads, 0, s>>>(b);
}

}  // namespace epscu
