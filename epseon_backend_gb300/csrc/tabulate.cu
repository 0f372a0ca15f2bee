// tabulate.cu -- device tabulation of parametric potentials and its adjoint
// (Morse, shifted Lennard-Jones 12-6, Morse + Gaussian bumps through a natural
// cubic spline on uniform knots).
//
// Everything is FP64, and on GB300 a FP64 instruction costs a warp 60 times an
// FP32 one's issue: the kernels are bound by the FP64 pipes (one instruction
// per point is 0.06 ms on the 2048-potential mixed batch, the write 0.05 ms).
// The values are the plain formulas' on tiles of points (a solve on an
// under-resolved grid amplifies their last bits, so no cheaper form of the
// exponential or the divisions is used), with the spline's Thomas sweeps by
// chunks: the LU recurrences contract by 2 - sqrt(3) = 0.268 a knot, so a lane
// starts them before its chunk instead of waiting for the whole sweep (a serial
// sweep by one thread, with a division a knot, was 1.2 ms of a launch whatever
// its size).  The adjoint, whose sums have no such readers, cuts the work per
// point:
//   * the Morse exponential is geometric along a uniform grid: the product of a
//     factor per 64-point block and a table of 64 factors (1 multiply instead of
//     an exp a point);
//   * 1/r by a FP32 reciprocal and two Newton steps;
//   * the spline's cubic weights in factored form, w^3 - w = -u w (1 + w);
//   * the tridiagonal system (1, 4, 1) by chunks, kWarm = 40 knots before each
//     (0.268^40 = 1e-23).
// Measured on the mixed batch (2048 potentials, 36.8 M points): values and
// adjoint together 7.8 -> 3.7 ms, the adjoint 4.30 -> 1.44 of them.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "common.cuh"
#include "launch.h"

namespace epscu {

namespace {

constexpr int kTabThreads = 256;
constexpr int kWarm = 40;
constexpr int kSweepWarm = 160;
constexpr int kBlock = 64;  // points per factor of the geometric exponential

// 1/r: an FP32 reciprocal and Newton steps where they hold, the division elsewhere
__device__ __forceinline__ double recip_r(double r) {
    return fabs(r) > 1e-30 && fabs(r) < 1e30 ? recip64_normal(r) : 1.0 / r;
}

// Knot value: Morse and up to three Gaussian bumps.
__device__ __forceinline__ double knot_value(const double* __restrict__ P, double r) {
    const double x = 1.0 - exp(-P[1] * (r - P[2]));
    double v = P[0] * x * x;
    for (int q = 0; q < 3; ++q) {
        const double amp = P[3 + 3 * q], w = P[4 + 3 * q], c = P[5 + 3 * q];
        if (amp != 0.0) v += amp * exp(-((r - c) * (r - c)) / (2.0 * w * w));
    }
    return v;
}

// 1 / (LU pivot) of row i of tridiag(1, 4, 1): U_i / U_{i+1}, U = 1, 4, 15, ...
// (integers below 2^53 for i < 27; the limit 2 - sqrt(3) beyond).
constexpr int kPivots = 26;
__device__ __forceinline__ double pivot_inverse(int i) {
    long long a = 1, b = 4;
    for (int q = 0; q < min(i, kPivots); ++q) {
        const long long c = 4 * b - a;
        a = b;
        b = c;
    }
    return (double)a / (double)b;
}

// x = tridiag(1, 4, 1)^-1 b on n rows, by the CTA: every thread its chunk of
// rows, the two sweeps started kWarm rows outside it (or at the matrix's end).
// d: scratch of n doubles.  b, d and x may not alias.  cp: kPivots + 1 inverse
// pivots in shared memory.
__device__ __forceinline__ void solve_141(const double* __restrict__ b, double* __restrict__ d, double* __restrict__ x,
                                          int n, const double* cp) {
    const int per = (n + kTabThreads - 1) / kTabThreads;
    const int lo = min((int)threadIdx.x * per, n), hi = min(lo + per, n);
    if (lo < hi) {
        double v = 0.0;
        for (int i = max(0, lo - kWarm); i < hi; ++i) {
            v = (b[i] - v) * cp[min(i, kPivots)];
            if (i >= lo) d[i] = v;
        }
    }
    __syncthreads();
    if (lo < hi) {
        double v = 0.0;
        for (int i = min(n, hi + kWarm) - 1; i >= lo; --i) {
            v = d[i] - cp[min(i, kPivots)] * v;
            if (i < hi) x[i] = v;
        }
    }
    __syncthreads();
}

// Knot values y and h^2/6 times the spline's second derivatives, one CTA per
// potential: M_{k-1} + 4 M_k + M_{k+1} = 6 (y_{k+1} - 2 y_k + y_{k-1}) / hk^2.
__global__ void __launch_bounds__(kTabThreads) knots_kernel(const int32_t* kind, const double* params,
                                                            const double* r_min, const double* r_max, int32_t K,
                                                            double* scratch) {
    __shared__ double cp[kPivots + 1];
    const int p = blockIdx.x;
    if (kind[p] != EPSCU_KIND_SPLINE) return;
    const double* P = params + (int64_t)p * 12;
    double* y = scratch + (int64_t)p * 4 * K;
    double* M = y + K;
    double* rhs = M + K;
    double* d = rhs + K;
    const double r0 = r_min[p], hk = (r_max[p] - r0) / (double)(K - 1);
    for (int j = threadIdx.x; j < K; j += kTabThreads) y[j] = knot_value(P, r0 + j * hk);
    __syncthreads();
    // the Thomas sweeps by one warp, a chunk a lane: started kSweepWarm knots
    // outside its chunk a sweep has the serial one's value to 1e-23 after 40 of
    // them and, since two neighbouring numbers fall together with probability
    // 0.73 a knot, its bits after the rest (but for a point in 10^4; the values a
    // solve of an under-resolved grid gets should not depend on the chunks)
    const int n = K - 2;
    const double s6 = 6.0 / (hk * hk);
    if (threadIdx.x == 0) {
        M[0] = M[K - 1] = 0.0;
        cp[0] = 1.0 / 4.0;
        for (int i = 1; i <= kPivots; ++i) cp[i] = 1.0 / (4.0 - cp[i - 1]);  // (its limit from 20 on)
    }
    for (int i = threadIdx.x; i < n; i += kTabThreads) rhs[i] = s6 * (y[i + 2] - 2.0 * y[i + 1] + y[i]);
    __syncthreads();
    if (threadIdx.x >= 32) return;
    const int per = (n + 31) / 32;
    const int lo = min((int)threadIdx.x * per, n), hi = min(lo + per, n);
    if (lo < hi) {
        double v = 0.0;
        for (int i = max(0, lo - kSweepWarm); i < hi; ++i) {
            v = i == 0 ? rhs[0] / 4.0 : (rhs[i] - v) / (4.0 - cp[min(i - 1, kPivots)]);
            if (i >= lo) d[i] = v;
        }
    }
    __syncwarp();
    if (lo < hi) {
        double v = 0.0;
        for (int i = min(n, hi + kSweepWarm) - 1; i >= lo; --i) {
            v = i == n - 1 ? d[i] : d[i] - cp[min(i, kPivots)] * v;
            if (i < hi) M[i + 1] = v;
        }
    }
}

// Values on the grid: one CTA per (potential, kTabTile points).
__global__ void __launch_bounds__(kTabThreads) tabulate_kernel(int32_t n, const int32_t* kind, const double* params,
                                                               const int64_t* offsets, const int32_t* Ns,
                                                               const double* r_min, const double* r_max,
                                                               const int32_t* tiles, int32_t K, const double* scratch,
                                                               double* V) {
    __shared__ int s_p;
    if (threadIdx.x == 0) {
        int lo = 0, hi = n - 1;  // the last p with tiles[p] <= blockIdx.x
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (tiles[mid] <= (int)blockIdx.x) lo = mid;
            else hi = mid - 1;
        }
        s_p = lo;
    }
    __syncthreads();
    const int p = s_p, N = Ns[p];
    const long long first = (long long)((int)blockIdx.x - tiles[p]) * kTabTile;
    const int count = (int)min((long long)kTabTile, N - first);
    const double r0 = r_min[p], r1 = r_max[p];
    const double h = (r1 - r0) / (double)(N - 1);
    const double* P = params + (int64_t)p * 12;
    double* out = V + offsets[p] + first;
    const int k = kind[p];
    if (k == EPSCU_KIND_SPLINE) {
        const double* y = scratch + (int64_t)p * 4 * K;
        const double* M = y + K;
        const double hk = (r1 - r0) / (double)(K - 1);
        const double h2 = hk * hk / 6.0;
        for (int x = threadIdx.x; x < count; x += kTabThreads) {
            const int i = (int)first + x;
            const double r = r0 + i * h;
            const double t = (r - r0) / hk;
            int j = (int)floor(t);
            j = max(0, min(j, K - 2));
            const double u = t - j, w = 1.0 - u;
            out[x] = w * y[j] + u * y[j + 1] + h2 * ((w * w * w - w) * M[j] + (u * u * u - u) * M[j + 1]);
        }
    } else if (k == EPSCU_KIND_LJ) {
        const double eps = P[0], sigma = P[1];
        for (int x = threadIdx.x; x < count; x += kTabThreads) {
            const int i = (int)first + x;
            const double r = r0 + i * h;
            const double s = sigma / r;
            const double s2 = s * s;
            const double s6 = s2 * s2 * s2;
            out[x] = 4.0 * eps * (s6 * s6 - s6) + eps;
        }
    } else {
        for (int x = threadIdx.x; x < count; x += kTabThreads) {
            const int i = (int)first + x;
            const double d = 1.0 - exp(-P[1] * (r0 + i * h - P[2]));
            out[x] = P[0] * d * d;
        }
    }
}

// The adjoint of the tabulation: dL/dparams from dL/dV, one CTA per potential.
//   Morse, LJ: sum_i g_i dV_i/dtheta over the grid.
//   Morse + bumps through the spline: V = w y_j + u y_{j+1}
//     - u w ((1 + w) m_j + (1 + u) m_{j+1}) with m = A^-1 D2 y (A = tridiag(1, 4, 1)
//     on the interior knots, m_0 = m_{K-1} = 0), so dL/dy = P^T g +
//     D2^T A^-1 Q^T g, with P^T g and Q^T g the grid's pull-back onto the knots
//     (the linear and the cubic weights); then sum_k dL/dy_k dy_k/dtheta over
//     the knots (Morse and Gaussian terms).
// The pull-back is deterministic: each thread owns a contiguous range of knot
// intervals and the grid points that fall in them, writing the interval's left
// and right sums; every sum runs in a fixed order (no atomics), so repeated
// calls give identical bits.

// deterministic sum of one value per thread over the CTA; the result in thread 0
__device__ __forceinline__ double cta_sum(double v, double* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < kTabThreads / 32; ++w) r += red[w];
    __syncthreads();
    return r;
}

constexpr int kAdjSegment = 65536;  // points per fill of the block factors

__global__ void __launch_bounds__(kTabThreads) tabulate_adjoint_kernel(
    const int32_t* kind, const double* params, const int64_t* offsets, const int32_t* Ns, const double* r_min,
    const double* r_max, int32_t n_knots, double* scratch, const double* gV, double* gP) {
    __shared__ double red[kTabThreads / 32];
    __shared__ double cp[kPivots + 1];
    __shared__ double s_q[kBlock], s_b[kAdjSegment / kBlock];
    const int p = blockIdx.x;
    const int N = Ns[p];
    const double r0 = r_min[p], r1 = r_max[p];
    const double h = (r1 - r0) / (double)(N - 1);
    const double* P = params + (int64_t)p * 12;
    const double* g = gV + offsets[p];
    double acc[12];
    for (int q = 0; q < 12; ++q) acc[q] = 0.0;
    const int k = kind[p];
    if (k == EPSCU_KIND_SPLINE) {
        const int K = n_knots;
        const double hk = (r1 - r0) / (double)(K - 1);
        double* Ly = scratch + (int64_t)p * 6 * K;  // per interval: left and right sums of the linear weights
        double* Ry = Ly + K;
        double* LM = Ry + K;                          // and of the cubic weights; then Q^T g
        double* RM = LM + K;
        double* z = RM + K;                           // A^-1 (Q^T g) on the interior knots
        double* d = z + K;
        if (threadIdx.x <= kPivots) cp[threadIdx.x] = pivot_inverse(threadIdx.x);
        // ---- pull-back onto the knot intervals [jb, je) owned by this thread
        const int nint = K - 1;
        const int per = (nint + kTabThreads - 1) / kTabThreads;
        const int jb = min((int)threadIdx.x * per, nint), je = min(jb + per, nint);
        const double inv = 1.0 / (double)(N - 1);
        if (jb < je) {
            // first grid point of interval jb: the least i with i (K - 1) >= jb (N - 1)
            long long i = ((long long)jb * (N - 1) + (K - 2)) / (K - 1);
            long long rem = i * (K - 1) - (long long)jb * (N - 1);
            for (int j = jb; j < je; ++j, rem -= N - 1) {
                double ly = 0.0, ry = 0.0, lm = 0.0, rm = 0.0;
                // (the last interval holds the grid's last point too)
                for (; i < N && (rem < N - 1 || j == K - 2); ++i, rem += K - 1) {
                    const double u = (double)(int)rem * inv, w = 1.0 - u;
                    const double gi = g[i];
                    ly = fma(gi, w, ly);
                    ry = fma(gi, u, ry);
                    const double c = gi * (u * w);
                    lm = fma(c, 1.0 + w, lm);
                    rm = fma(c, 1.0 + u, rm);
                }
                Ly[j] = ly;
                Ry[j] = ry;
                LM[j] = -lm;
                RM[j] = -rm;
            }
        }
        __syncthreads();
        // ---- z = A^-1 (Q^T g)_interior (A symmetric)
        for (int i = threadIdx.x; i < K - 2; i += kTabThreads) z[i] = LM[i + 1] + RM[i];
        __syncthreads();
        solve_141(z, d, LM, K - 2, cp);  // (LM[i]: knot i + 1)
        // ---- dL/dy_k = (P^T g)_k + (D2^T z)_k, then the knots' parameter derivatives
        for (int kk = threadIdx.x; kk < K; kk += kTabThreads) {
            // (intervals are 0..K-2: the last knot has no interval of its own)
            double gy = (kk < K - 1 ? Ly[kk] : 0.0) + (kk > 0 ? Ry[kk - 1] : 0.0);
            auto zk = [&](int q) { return q >= 1 && q <= K - 2 ? LM[q - 1] : 0.0; };
            gy += zk(kk - 1) - 2.0 * zk(kk) + zk(kk + 1);
            const double r = r0 + kk * hk;
            const double De = P[0], a = P[1], re = P[2];
            const double e = exp(-a * (r - re));
            const double x = 1.0 - e;
            acc[0] += gy * x * x;
            acc[1] += gy * 2.0 * De * x * e * (r - re);
            acc[2] += gy * -2.0 * De * x * e * a;
            for (int q = 0; q < 3; ++q) {
                const double amp = P[3 + 3 * q], wd = P[4 + 3 * q], c = P[5 + 3 * q];
                if (amp == 0.0) continue;
                const double dr = r - c, iw = 1.0 / wd;
                const double t = dr * iw;
                const double G = exp(-0.5 * t * t);
                const double gG = gy * G;
                acc[3 + 3 * q] += gG;
                acc[4 + 3 * q] += gG * amp * t * t * iw;
                acc[5 + 3 * q] += gG * amp * t * iw;
            }
        }
    } else if (k == EPSCU_KIND_LJ) {
        // dV/deps = 4 (s12 - s6) + 1, dV/dsigma = 4 eps (12 s12 - 6 s6) / sigma
        const double sigma = P[1];
        double a12 = 0.0, a6 = 0.0, a0 = 0.0;
        for (int i = threadIdx.x; i < N; i += kTabThreads) {
            const double r = fma((double)i, h, r0);
            const double s = sigma * recip_r(r);
            const double s2 = s * s;
            const double s6 = s2 * s2 * s2;
            const double t = g[i] * s6;
            a0 += g[i];
            a6 += t;
            a12 = fma(t, s6, a12);
        }
        acc[0] = fma(4.0, a12 - a6, a0);
        acc[1] = 4.0 * P[0] * (12.0 * a12 - 6.0 * a6) / sigma;
    } else {
        // x = 1 - e: dV/dDe = x^2, dV/da = 2 De x e (r - re), dV/dre = -2 De x e a
        const double a = P[1], re = P[2];
        if (threadIdx.x < kBlock) s_q[threadIdx.x] = exp(-a * (threadIdx.x * h));
        double b0 = 0.0, b1 = 0.0, b2 = 0.0;
        for (int s0 = 0; s0 < N; s0 += kAdjSegment) {
            const int cnt = min(kAdjSegment, N - s0);
            __syncthreads();  // the previous segment's factors are used up
            for (int b = threadIdx.x; b * kBlock < cnt; b += kTabThreads)
                s_b[b] = exp(-a * (fma((double)(s0 + b * kBlock), h, r0) - re));
            __syncthreads();
            for (int x = threadIdx.x; x < cnt; x += kTabThreads) {
                const double e = s_b[x / kBlock] * s_q[x % kBlock];
                const double d = 1.0 - e;
                const double gd = g[s0 + x] * d;
                b0 = fma(gd, d, b0);
                const double t = gd * e;
                b2 += t;
                b1 = fma(t, fma((double)(s0 + x), h, r0 - re), b1);
            }
        }
        acc[0] = b0;
        acc[1] = 2.0 * P[0] * b1;
        acc[2] = -2.0 * P[0] * a * b2;
    }
    const int used = k == EPSCU_KIND_SPLINE ? 12 : (k == EPSCU_KIND_LJ ? 2 : 3);
    for (int q = 0; q < 12; ++q) {
        const double v = q < used ? cta_sum(acc[q], red) : 0.0;
        if (threadIdx.x == 0) gP[(int64_t)p * 12 + q] = v;
    }
}

}  // namespace

void launch_tabulate(int32_t n, const int32_t* kind, const double* params, const int64_t* offsets, const int32_t* N,
                     const double* r_min, const double* r_max, const int32_t* tiles, int32_t n_tiles, int32_t n_knots,
                     bool splines, double* knot_scratch, double* V, cudaStream_t s) {
    if (splines) knots_kernel<<<n, kTabThreads, 0, s>>>(kind, params, r_min, r_max, n_knots, knot_scratch);
    tabulate_kernel<<<n_tiles, kTabThreads, 0, s>>>(n, kind, params, offsets, N, r_min, r_max, tiles, n_knots,
                                                    knot_scratch, V);
}

void launch_tabulate_adjoint(int32_t n, const int32_t* kind, const double* params, const int64_t* offsets,
                             const int32_t* N, const double* r_min, const double* r_max, int32_t n_knots,
                             double* knot_scratch, const double* gV, double* gP, cudaStream_t s) {
    tabulate_adjoint_kernel<<<n, kTabThreads, 0, s>>>(kind, params, offsets, N, r_min, r_max, n_knots, knot_scratch, gV,
                                                      gP);
}

}  // namespace epscu
