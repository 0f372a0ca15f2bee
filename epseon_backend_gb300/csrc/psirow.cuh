// psirow.cuh -- a level's psi row from the tagged pairs its norm pass stored.
#pragma once

#include <math.h>
#include <stdint.h>

#include "common.cuh"
#include "dfloat.cuh"
#include "dfpass.cuh"

namespace epscu {

namespace {

// the barrier of a group of NT threads: a warp, the CTA, a cluster of CTAs of 256
template <int NT>
__device__ __forceinline__ void group_sync() {
    if constexpr (NT == 32) __syncwarp();
    else if constexpr (NT <= 256) __syncthreads();
    else
        asm volatile(
            "barrier.cluster.arrive.release;\n\t"
            "barrier.cluster.wait.acquire;" ::
                : "memory");
}

// n zeros at p by NT threads (t: this one), 16 bytes a store
template <int NT>
__device__ __forceinline__ void zero_points(int t, double* p, int n) {
    if (n <= 0) return;
    const int head = (int)((reinterpret_cast<uintptr_t>(p) >> 3) & 1);
    if (head && t == 0) p[0] = 0.0;
    double2* q = reinterpret_cast<double2*>(p + head);
    const int pairs = (n - head) >> 1;
    for (int i = t; i < pairs; i += NT) q[i] = make_double2(0.0, 0.0);
    if (((n - head) & 1) && t == 0) p[n - 1] = 0.0;
}

// The level's row: the window's tagged pairs times the side constants (as
// norm_k 2^-ex = M 2^e with a double-float M in [0.5, 1): a double-float
// product and an integer assembly of the double, no FP64 instruction a
// point), psi_k, and zeros outside the window (everywhere without a result).
template <int NT>
__device__ __noinline__ void finish_row(int t, const LevelWork& w, double* __restrict__ row, int N) {
    const bool none = no_result(w);
    zero_points<NT>(t, row, none ? N : w.j0);
    if (none) return;
    zero_points<NT>(t, row + w.j1 + 1, N - 1 - w.j1);
    int e_out, e_in;
    const dfl M_out = df_from_double(frexp(w.norm_k_out, &e_out));
    const dfl M_in = df_from_double(frexp(w.norm_k_in, &e_in));
    e_out -= w.ex_out;
    e_in -= w.ex_in;
    // the pairs were stored by other threads of the group
    group_sync<NT>();
    const float2* pair = reinterpret_cast<const float2*>(row);
    constexpr int kS = NT;
    for (int i0 = w.j0; i0 <= w.j1; i0 += 4 * kS) {
        float2 raw[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const int i = i0 + x * kS + t;
            if (i <= w.j1 && i != w.k) raw[x] = pair[i];
        }
#pragma unroll 1
        for (int x = 0; x < 4; ++x) {
            const int i = i0 + x * kS + t;
            const float2 z4 = raw[0];
            raw[0] = raw[1];
            raw[1] = raw[2];
            raw[2] = raw[3];
            if (i > w.j1) continue;
            double v = w.ck;
            if (i != w.k) {
                int r;
                const dfl z = load_psi_pair(z4, r);
                const bool outward = i < w.k;
                const dfl p = df_mul(z, outward ? M_out : M_in);
                v = df_pair_to_double_scaled(p.h, p.l, 64 * r + (outward ? e_out : e_in));
            }
            row[i] = v;
        }
    }
}

}  // namespace

}  // namespace epscu
