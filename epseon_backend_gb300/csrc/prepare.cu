// prepare.cu -- per-potential set-up of the discrete problem and level-slot
// bookkeeping.
//
// The set-up gives the oracle's eo_prepare() results exactly: minimum of V,
// E-independent Dirichlet cut-offs (a (V_i - E_lo) <= 1/2 in FP64), scan
// twist index (first argmin of V), trial spacing and the bisection step count.
#include <cuda_runtime.h>
#include <math.h>

#include "common.cuh"
#include "dfpass.cuh"
#include "launch.h"

namespace epscu {

namespace {

constexpr int kPrepThreads = 256;

// An unsigned integer image of a double that orders like the double (for
// non-NaN values): minima taken on it are exact and need no FP64 instruction.
constexpr unsigned long long kKeyMax = ~0ull;  // above every image (+inf's image is below it)
__device__ __forceinline__ unsigned long long dkey(double x) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(x);
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}
__device__ __forceinline__ double dkey_inv(unsigned long long k) {
    const unsigned long long u = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
    return __longlong_as_double((long long)u);
}
// the same with the two zeros on one key (they compare equal as doubles)
__device__ __forceinline__ unsigned long long dkey0(double x) {
    unsigned long long u = (unsigned long long)__double_as_longlong(x);
    if ((u << 1) == 0ull) u = 0ull;
    return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}
// the warp's smallest image / largest image, from 32-bit reductions of the halves
__device__ __forceinline__ unsigned long long warp_min_key(unsigned long long k) {
    const uint32_t h = __reduce_min_sync(0xffffffffu, (uint32_t)(k >> 32));
    const uint32_t l = __reduce_min_sync(0xffffffffu, (uint32_t)(k >> 32) == h ? (uint32_t)k : 0xffffffffu);
    return ((unsigned long long)h << 32) | l;
}
__device__ __forceinline__ unsigned long long warp_max_key(unsigned long long k) { return ~warp_min_key(~k); }

// (__double2float_rn(w), __double2float_rn(w - hi)) with integer operations
// for 2^-60 <= |w| < 2^101 (the conversions otherwise): hi rounds the 52-bit
// significand to 23 bits to nearest, ties to even; w - hi is the signed
// remainder of the 29 dropped bits times 2^(e-52), exact in a double, so one
// integer-to-float rounding of the remainder and two exact power-of-two
// scalings give the same float as converting w - hi.  No FP64 instruction.
__device__ __forceinline__ float2 split_double_rn(double w) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(w);
    const int e = (int)((u >> 52) & 0x7ffull) - 1023;
    if (e < -60 || e > 100) {
        const float hi = __double2float_rn(w);
        return make_float2(hi, __double2float_rn(__dsub_rn(w, (double)hi)));
    }
    const uint32_t sgn = (uint32_t)(u >> 32) & 0x80000000u;
    const unsigned long long mant = u & 0xfffffffffffffull;
    const uint32_t r = (uint32_t)(mant & 0x1fffffffull);
    uint32_t hb = ((uint32_t)(e + 127) << 23) | (uint32_t)(mant >> 29);
    const uint32_t up = (r > 0x10000000u || (r == 0x10000000u && (hb & 1u))) ? 1u : 0u;
    hb += up;  // a carry out of the significand raises the exponent
    const int rr = (int)r - (up ? 0x20000000 : 0);
    float lo = 0.0f;
    if (rr != 0) {
        lo = __fmul_rn(__fmul_rn(__int2float_rn(rr), 2.220446049250313e-16f), __int_as_float((127 + e) << 23));
        if (sgn) lo = -lo;
    }
    return make_float2(__uint_as_float(sgn | hb), lo);
}

// ------------------------------------------------------------------ set-up
// One CTA per tile of kPrepTile points, in one pass over V: W = a V (FP64 and
// the float pair, zeros in the padding), the minima of the 32-point blocks and
// the tile's summary.  The last CTA of a potential to finish derives what
// needs the whole grid from the summaries and from the points of the two tiles
// that hold the cut-offs; a second kernel, a warp per tile, turns the block
// minima into suffix and prefix minima.
//
// 24 bytes a point are moved (read V, write W twice).  With a CTA per potential,
// which read V six times and wrote point-wise suffix and prefix minima (16 bytes
// a point), a potential was one SM's work; both kernels together, before and now:
//     1 x 2^20 points              6.4 ms   27 us
//     256 x 2048..65536 points     490 us   71 us
//     2048 x 2048..65536 points    870 us  390 us  (3 TB/s)
//     1 x 4096 points               32 us   17 us
constexpr int kPrepUnroll = kPrepTile / kPrepThreads;

// the potential of tile x (its first tile, kPrepTile padded points each, is at
// or before x: the last such)
__device__ __forceinline__ int tile_potential(const DevBatch& b, int x) {
    const int64_t at = (int64_t)x * kPrepTile;
    int lo = 0, hi = b.n - 1;
    while (lo < hi) {
        const int mid = lo + (hi - lo + 1) / 2;
        if (b.meta[mid].offf <= at) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// The largest image whose double passes the cut-off test a (V - V_min) <= 1/2
// (it holds at V_min, is monotone in the image and fails for the NaNs, the
// images above +inf): a search outward from V_min + 1/(2a), then bisection.
__device__ unsigned long long cutoff_key(double a, double vmin, unsigned long long kmin) {
    auto inside = [&](unsigned long long k) { return __dmul_rn(a, __dsub_rn(dkey_inv(k), vmin)) <= 0.5; };
    unsigned long long lo = kmin, hi = kKeyMax;
    const unsigned long long g = dkey0(__dadd_rn(vmin, __ddiv_rn(0.5, a)));
    if (g > lo && g < hi) {
        unsigned long long step = 1ull;
        if (inside(g)) {
            lo = g;
            while (hi - lo > step) {
                if (!inside(lo + step)) {
                    hi = lo + step;
                    break;
                }
                lo += step;
                step <<= 1;
            }
        } else {
            hi = g;
            while (hi - lo > step) {
                if (inside(hi - step)) {
                    lo = hi - step;
                    break;
                }
                hi -= step;
                step <<= 1;
            }
        }
    }
    while (hi - lo > 1ull) {
        const unsigned long long mid = lo + (hi - lo) / 2;
        if (inside(mid)) lo = mid;
        else hi = mid;
    }
    return lo;
}

// halvings of the trial spacing down to tol (at most 200): the loop
// w = delta; while w > tol: w /= 2, whose steps are exact
__device__ __forceinline__ int halvings_to(double delta, double tol) {
    if (!(delta > tol)) return 0;
    const unsigned long long ud = (unsigned long long)__double_as_longlong(delta);
    const unsigned long long ut = (unsigned long long)__double_as_longlong(tol);
    const int ed = (int)((ud >> 52) & 0x7ff), et = (int)((ut >> 52) & 0x7ff);
    if (ed == 0x7ff || ed == 0 || et == 0) {  // (infinite, or a denormal halved inexactly)
        int K = 0;
        for (double w = delta; w > tol && K < 200; w = __dmul_rn(w, 0.5)) ++K;
        return K;
    }
    const unsigned long long mant = 0xfffffffffffffull;
    return min(200, ed - et + ((ud & mant) > (ut & mant) ? 1 : 0));
}

// What the whole grid decides, from the tile summaries (nt of them, at t0).
__device__ void finish_potential(const DevBatch& b, int p, int nt, const PrepTile* rec) {
    __shared__ unsigned long long s_k[3][kPrepThreads / 32];
    __shared__ int s_i[4][kPrepThreads / 32];
    __shared__ unsigned long long s_kt, s_kb;
    __shared__ double s_delta, s_kmax;
    __shared__ int s_K;
    constexpr int nw = kPrepThreads / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    PotMeta m = b.meta[p];
    const double* V = b.V64 + m.off;
    const int N = m.N;

    // minimum of V, and its first point in the interior (the scan's twist index)
    unsigned long long kall = kKeyMax, kin = kKeyMax;
    int iin = N, bad = 0;
    for (int t = tid; t < nt; t += kPrepThreads) {
        const PrepTile r = rec[t];
        kall = min(kall, r.kall);
        if (r.kin < kin) {
            kin = r.kin;
            iin = r.iin;
        }
        bad |= r.bad;
    }
    const unsigned long long wall = warp_min_key(kall), win = warp_min_key(kin);
    const int wi = __reduce_min_sync(0xffffffffu, kin == win ? iin : N);
    const int wb = __reduce_or_sync(0xffffffffu, bad);
    if (lane == 0) {
        s_k[0][warp] = wall;
        s_k[1][warp] = win;
        s_i[0][warp] = wi;
        s_i[1][warp] = wb;
    }
    __syncthreads();
    bad = 0;
    for (int w = 0; w < nw; ++w) bad |= s_i[1][w];
    kall = kin = kKeyMax;
    iin = N;
    for (int w = 0; w < nw; ++w) {
        kall = min(kall, s_k[0][w]);
        if (s_k[1][w] < kin || (s_k[1][w] == kin && s_i[0][w] < iin)) {
            kin = s_k[1][w];
            iin = s_i[0][w];
        }
    }
    const double vmin = dkey_inv(kall);
    if (tid == 0) s_kt = cutoff_key(m.a, vmin, kall);
    if (tid == 32) {  // (beside it, as is the next)
        s_delta = __ddiv_rn(__dsub_rn(m.e_cap, vmin), (double)m.n_trial);
        s_kmax = sqrt(2.0 * m.mu * (m.e_cap - vmin));
        s_K = halvings_to(s_delta, b.tol > 0.0 ? b.tol : 1e-12);
    }
    if (tid == 64) s_kb = dkey0(__dadd_rn(vmin, __ddiv_rn(1.0 - 1e-6, m.a)));
    __syncthreads();
    const unsigned long long kt = s_kt;

    // the tiles that hold the first and the last point inside the cut-off
    int ft = nt, lt = -1;
    for (int t = tid; t < nt; t += kPrepThreads)
        if (rec[t].kall <= kt) {
            ft = min(ft, t);
            lt = max(lt, t);
        }
    ft = __reduce_min_sync(0xffffffffu, ft);
    lt = __reduce_max_sync(0xffffffffu, lt);
    if (lane == 0) {
        s_i[2][warp] = ft;
        s_i[3][warp] = lt;
    }
    __syncthreads();
    for (int w = 0; w < nw; ++w) {
        ft = min(ft, s_i[2][w]);
        lt = max(lt, s_i[3][w]);
    }
    __syncthreads();
    int first = N, last = -1;
    if (lt >= 0)
        for (int x = tid; x < kPrepTile; x += kPrepThreads) {
            const int i = ft * kPrepTile + x, j = lt * kPrepTile + x;
            if (i < N && dkey0(V[i]) <= kt) first = min(first, i);
            if (j < N && dkey0(V[j]) <= kt) last = max(last, j);
        }
    first = __reduce_min_sync(0xffffffffu, first);
    last = __reduce_max_sync(0xffffffffu, last);
    if (lane == 0) {
        s_i[0][warp] = first;
        s_i[1][warp] = last;
    }
    __syncthreads();
    for (int w = 0; w < nw; ++w) {
        first = min(first, s_i[0][w]);
        last = max(last, s_i[1][w]);
    }
    const int i0 = first < 1 ? 1 : first;
    const int i1 = last > N - 2 ? N - 2 : last;

    // a barrier inside the cut-offs that rises above them (1), or to where f is
    // negative (2; from 1e-6 below, for the rounding of T), and the minima of the
    // two end tiles over [i0, i1]
    const unsigned long long kb = s_kb;
    auto above = [&](unsigned long long k) { return (k > kt ? 1 : 0) | (k > kb ? 2 : 0); };
    int steep = 0;
    unsigned long long ka = kKeyMax, kz = kKeyMax;
    for (int t = ft + 1 + tid; t < lt; t += kPrepThreads) steep |= above(rec[t].kmax);
    if (lt >= 0)
        for (int x = tid; x < kPrepTile; x += kPrepThreads) {
            const int i = ft * kPrepTile + x, j = lt * kPrepTile + x;
            if (i >= i0 && i <= i1) {
                const unsigned long long k = dkey0(V[i]);
                ka = min(ka, k);
                steep |= above(k);
            }
            if (j >= i0 && j <= i1) {
                const unsigned long long k = dkey0(V[j]);
                kz = min(kz, k);
                steep |= above(k);
            }
        }
    ka = warp_min_key(ka);
    kz = warp_min_key(kz);
    steep = __reduce_or_sync(0xffffffffu, steep);
    if (lane == 0) {
        s_k[0][warp] = ka;
        s_k[1][warp] = kz;
        s_i[2][warp] = steep;
    }
    __syncthreads();
    if (tid != 0) return;
    for (int w = 0; w < nw; ++w) {
        ka = min(ka, s_k[0][w]);
        kz = min(kz, s_k[1][w]);
        steep |= s_i[2][w];
    }
    PrepTile* out = const_cast<PrepTile*>(rec);
    if (lt >= 0) {
        out[ft].kall = ka;
        out[lt].kall = kz;  // (one tile: the same minimum)
    }
    int status = 0;
    if (bad) status |= EPSCU_STATUS_BAD | EPSCU_STATUS_NONFINITE;
    if (i1 - i0 < 2) status |= EPSCU_STATUS_BAD;
    if (!(m.e_cap > vmin)) status |= EPSCU_STATUS_BAD;
    m.e_lo = vmin;
    m.i0 = i0;
    m.i1 = i1;
    m.k_scan = i0 <= i1 && iin < N ? iin : i0;
    m.delta = s_delta;
    m.n_bisect = s_K;
    if (s_kmax * m.h > 1.0) status |= EPSCU_STATUS_UNDER;
    if (steep) status |= EPSCU_STATUS_STEEP;
    if (steep & 2) status |= EPSCU_STATUS_BELOW;
    m.status = status;
    if (b.under_list && (status & EPSCU_STATUS_UNDER) && !(status & EPSCU_STATUS_BAD))
        b.under_list[atomicAdd(&b.hdr->n_under, 1)] = p;
    m.n_total = 0;
    m.n_out = 0;
    m.prep_done = 0;
    b.meta[p] = m;
}

__global__ void __launch_bounds__(kPrepThreads) prepare_kernel(DevBatch b) {
    __shared__ unsigned long long s_k[3][kPrepThreads / 32];
    __shared__ int s_i[2][kPrepThreads / 32];
    __shared__ int s_last;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int p = tile_potential(b, blockIdx.x);
    const int64_t offf = b.meta[p].offf, off = b.meta[p].off;
    const int N = b.meta[p].N;
    const double a = b.meta[p].a;
    const int t = (int)((int64_t)blockIdx.x - offf / kPrepTile);
    const int base = t * kPrepTile;
    const double* V = b.V64 + off;
    double* W = b.W64 + off;
    float2* Wf = b.Wf2 ? b.Wf2 + offf : nullptr;

    double v[kPrepUnroll];
#pragma unroll
    for (int u = 0; u < kPrepUnroll; ++u) {
        const int i = base + u * kPrepThreads + tid;
        v[u] = i < N ? V[i] : 0.0;
    }
    // the comparisons run on order-preserving integer images of the doubles
    // (dkey0), exact and on the integer pipes; the only FP64 instruction per
    // point is W = a V
    unsigned long long kall = kKeyMax, kin = kKeyMax, kmax = 0ull;
    int iin = N, bad = 0;
#pragma unroll
    for (int u = 0; u < kPrepUnroll; ++u) {
        const int i = base + u * kPrepThreads + tid;
        const bool on = i < N;
        const double w = __dmul_rn(a, v[u]);
        if (on) W[i] = w;
        if (Wf) Wf[i] = on ? split_double_rn(w) : make_float2(0.0f, 0.0f);
        unsigned long long k = kKeyMax;
        if (on) {
            k = dkey0(v[u]);
            if ((((unsigned long long)__double_as_longlong(v[u]) >> 52) & 0x7ffull) == 0x7ffull) bad = 1;  // inf, NaN
            kmax = max(kmax, k);
        }
        const unsigned long long blk = warp_min_key(k);
        if (lane == 0 && on) b.Bkey[(offf + i) >> 5] = blk;
        kall = min(kall, blk);
        // the first interior point of the smallest image (i grows with u)
        const unsigned long long ki = i >= 1 && i <= N - 2 ? k : kKeyMax;
        if (ki < kin) {
            kin = ki;
            iin = i;
        }
    }
    if (base >= N) return;  // (padding only; uniform over the CTA)
    const unsigned long long win = warp_min_key(kin), wmax = warp_max_key(kmax);
    const int wi = __reduce_min_sync(0xffffffffu, kin == win ? iin : N);
    bad = __reduce_or_sync(0xffffffffu, bad);
    if (lane == 0) {
        s_k[0][warp] = kall;
        s_k[1][warp] = win;
        s_k[2][warp] = wmax;
        s_i[0][warp] = wi;
        s_i[1][warp] = bad;
    }
    __syncthreads();
    const int nt = (N + kPrepTile - 1) / kPrepTile;
    PrepTile* rec = b.prep + offf / kPrepTile;
    if (tid == 0) {
        PrepTile r{kKeyMax, kKeyMax, 0ull, N, 0};
        for (int w = 0; w < kPrepThreads / 32; ++w) {
            r.kall = min(r.kall, s_k[0][w]);
            r.kmax = max(r.kmax, s_k[2][w]);
            r.bad |= s_i[1][w];
            if (s_k[1][w] < r.kin || (s_k[1][w] == r.kin && s_i[0][w] < r.iin)) {
                r.kin = s_k[1][w];
                r.iin = s_i[0][w];
            }
        }
        rec[t] = r;
        __threadfence();
        s_last = nt == 1 || atomicAdd(&b.meta[p].prep_done, 1) == nt - 1;
        __threadfence();
    }
    __syncthreads();
    if (s_last) finish_potential(b, p, nt, rec);
}

// Suffix and prefix minima of V over the 32-point blocks of [i0, i1] (the
// minimum from a block's start to i1, and from i0 to its end), and for the
// fast method the block minima of a V rounded down to float (the decay-window
// bounds).  One warp per tile of 64 blocks; what lies beyond the tile comes
// from the tile summaries.
__global__ void __launch_bounds__(128) block_minima_kernel(DevBatch b, int n_tiles) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int x = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (x >= n_tiles) return;
    const int p = tile_potential(b, x);
    const PotMeta& m = b.meta[p];
    const int t = (int)((int64_t)x - m.offf / kPrepTile);
    if (t * kPrepTile >= m.N || (m.status & EPSCU_STATUS_BAD)) return;
    const int i0 = m.i0, i1 = m.i1;
    const int ft = i0 / kPrepTile, lt = i1 / kPrepTile;
    if (t < ft || t > lt) return;
    const PrepTile* rec = b.prep + m.offf / kPrepTile;
    unsigned long long right = kKeyMax, left = kKeyMax;
    for (int q = t + 1 + lane; q <= lt; q += 32) right = min(right, rec[q].kall);
    for (int q = ft + lane; q < t; q += 32) left = min(left, rec[q].kall);
    right = warp_min_key(right);
    left = warp_min_key(left);
    const int64_t B0 = m.offf / 32;
    const double* V = b.V64 + m.off;
    const double a = m.a;
    constexpr int kPer = kPrepTile / 32 / 32;  // blocks per lane
    unsigned long long k[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        const int B = t * (kPrepTile / 32) + u * 32 + lane;
        k[u] = B >= (i0 >> 5) && B <= (i1 >> 5) ? b.Bkey[B0 + B] : kKeyMax;
        // the blocks that the cut-offs cut: over their points inside
        for (int end = 0; end < 2; ++end) {
            const int Bc = (end ? i1 : i0) >> 5;
            if (Bc < t * (kPrepTile / 32) + u * 32 || Bc >= t * (kPrepTile / 32) + u * 32 + 32) continue;  // (uniform)
            const int i = (Bc << 5) + lane;
            const unsigned long long kc = warp_min_key(i >= i0 && i <= i1 ? dkey0(V[i]) : kKeyMax);
            if (B == Bc) k[u] = kc;
        }
    }
    unsigned long long suf[kPer], pre[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        suf[u] = pre[u] = k[u];
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_down_sync(full, suf[u], o), z = __shfl_up_sync(full, pre[u], o);
            if (lane + o < 32) suf[u] = min(suf[u], y);
            if (lane >= o) pre[u] = min(pre[u], z);
        }
    }
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        pre[u] = min(pre[u], left);
        left = __shfl_sync(full, pre[u], 31);
    }
#pragma unroll
    for (int u = kPer - 1; u >= 0; --u) {
        suf[u] = min(suf[u], right);
        right = __shfl_sync(full, suf[u], 0);
    }
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
        const int B = t * (kPrepTile / 32) + u * 32 + lane;
        if (B < (i0 >> 5) || B > (i1 >> 5)) continue;
        b.Bsuf[B0 + B] = dkey_inv(suf[u]);
        if (b.Bpre) {
            b.Bpre[B0 + B] = dkey_inv(pre[u]);
            b.Bmin[B0 + B] = __double2float_rd(__dmul_rn(a, dkey_inv(k[u])));
        }
    }
}

// Level counts per potential, exclusive prefix sums (level slots and psi
// offsets) and the total level count.  One CTA.
// A solve cancelled before this point, or whose scan gave up on a bounded wait
// (the error word is set), may have skipped scan work: its counts are
// incomplete and it gets no levels.  The cancel flag only goes from 0 to 1
// while a solve runs, so a scan that saw it is always followed by a set-up
// that does.
__global__ void __launch_bounds__(1024) level_setup_kernel(DevBatch b) {
    __shared__ int32_t s_lv[1024];
    __shared__ long long s_ps[1024];
    __shared__ int32_t carry_lv;
    __shared__ long long carry_ps;
    __shared__ int s_cancelled, s_failed;
    if (threadIdx.x == 0) {
        carry_lv = 0;
        carry_ps = 0;
        s_cancelled = b.cancel && *b.cancel;
        s_failed = b.hdr->error != 0;
    }
    __syncthreads();
    const bool cancelled = s_cancelled != 0, failed = s_failed != 0;
    for (int base = 0; base < b.n; base += blockDim.x) {
        const int p = base + threadIdx.x;
        int32_t n_out = 0;
        long long ps = 0;
        if (p < b.n) {
            PotMeta& m = b.meta[p];
            int32_t n_total = 0;
            if (cancelled) m.status |= EPSCU_STATUS_CANCELLED;
            else if (!failed && !(m.status & EPSCU_STATUS_BAD)) n_total = b.counts[(int64_t)p * b.n_trial + b.n_trial - 1];
            int32_t last = b.max_level < 0 ? n_total - 1 : min(b.max_level, n_total - 1);
            n_out = last - b.min_level + 1;
            n_out = max(0, min(n_out, b.level_capacity));
            m.n_total = n_total;
            m.n_out = n_out;
            ps = (long long)n_out * m.N;
        }
        s_lv[threadIdx.x] = n_out;
        s_ps[threadIdx.x] = ps;
        __syncthreads();
        // inclusive Hillis-Steele scan
        for (int o = 1; o < (int)blockDim.x; o <<= 1) {
            int32_t x = threadIdx.x >= o ? s_lv[threadIdx.x - o] : 0;
            long long y = threadIdx.x >= o ? s_ps[threadIdx.x - o] : 0;
            __syncthreads();
            s_lv[threadIdx.x] += x;
            s_ps[threadIdx.x] += y;
            __syncthreads();
        }
        if (p < b.n) {
            b.meta[p].level_base = carry_lv + s_lv[threadIdx.x] - n_out;
            b.meta[p].psi_off = carry_ps + s_ps[threadIdx.x] - ps;
        }
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) {
            carry_lv += s_lv[threadIdx.x];
            carry_ps += s_ps[threadIdx.x];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        b.hdr->total_levels = carry_lv;
        b.hdr->psi_total = carry_ps;
        b.hdr->queue_refine = 0;
        b.hdr->queue_polish = 0;
        if (b.psi && carry_ps > b.psi_capacity) atomicCAS(&b.hdr->error, 0, 5);
    }
}

// Warp work units for the per-level kernels: each potential's level slots in
// chunks of 32, potentials in decreasing grid length (the `order` array), so
// the warp queue hands out the longest work first.  (The plain method's.)
// One CTA.
__global__ void __launch_bounds__(1024) unit_setup_kernel(DevBatch b) {
    __shared__ int32_t s_u[1024];
    __shared__ int32_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < b.n; base += blockDim.x) {
        const int q = base + threadIdx.x;
        int32_t nu = 0;
        int p = 0;
        if (q < b.n) {
            p = b.order[q];
            nu = (b.meta[p].n_out + 31) / 32;
        }
        s_u[threadIdx.x] = nu;
        __syncthreads();
        for (int o = 1; o < (int)blockDim.x; o <<= 1) {
            const int32_t x = threadIdx.x >= o ? s_u[threadIdx.x - o] : 0;
            __syncthreads();
            s_u[threadIdx.x] += x;
            __syncthreads();
        }
        if (q < b.n) {
            const int32_t first = carry + s_u[threadIdx.x] - nu;
            const PotMeta& m = b.meta[p];
            for (int u = 0; u < nu; ++u) {
                const int32_t at = first + u;
                if (at < b.max_units) b.units[at] = make_int2(m.level_base + 32 * u, min(32, m.n_out - 32 * u));
            }
        }
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry += s_u[threadIdx.x];
        __syncthreads();
    }
    if (threadIdx.x == 0) b.hdr->n_units = min(carry, b.max_units);
}

// Bracket of every level slot from the scan counts: first trial j with
// count_j > v; bracket [E_{j-1}, E_j] (E_{-1} = E_lo).
__global__ void bracket_kernel(DevBatch b) {
    const int p = blockIdx.x;
    const PotMeta m = b.meta[p];
    const int32_t* c = b.counts + (int64_t)p * b.n_trial;
    for (int s = threadIdx.x; s < m.n_out; s += blockDim.x) {
        const int v = b.min_level + s;
        int lo = 0, hi = m.n_trial;
        int top = -1;  // trial index of the bracket's upper end (lo when -1)
        if (!b.bis_list || (b.under_list && (m.status & EPSCU_STATUS_UNDER))) {
            while (lo < hi) {
                const int mid = lo + (hi - lo) / 2;
                if (c[mid] > v) hi = mid;
                else lo = mid + 1;
            }
        } else {
            // bisection scan: counts exist at the coarse boundaries and at the
            // midpoints of every cell that held a level; descend the same
            // cells to the first trial index with a count above v
            const int last = m.n_trial - 1;
            const int ctop = c[last];
            if (v >= ctop) {
                lo = m.n_trial;
            } else {
                const int K = (m.n_trial + kBisectCoarse - 1) / kBisectCoarse;
                int kl = 1, kh = K;  // first coarse boundary with a count above v
                while (kl < kh) {
                    const int km = (kl + kh) / 2;
                    if (c[min(km * kBisectCoarse - 1, last)] > v) kh = km;
                    else kl = km + 1;
                }
                // then down the cell's halves while their midpoints have a
                // count (a cell cut into fewer parts ends the descent early:
                // the bracket is the last cell (a, a + W])
                int a = (kl - 1) * kBisectCoarse - 1;
                int W = kBisectCoarse;
                for (; W > 1; W >>= 1) {
                    const int mid = a + W / 2;
                    const int cm = mid >= last ? ctop : c[mid];
                    if (cm < 0) break;  // no count taken there
                    if (cm <= v) a = mid;
                }
                lo = min(a + 1, last);
                top = min(a + W, last);
            }
        }
        LevelWork w;
        w.p = p;
        w.v = v;
        w.status = m.status & EPSCU_STATUS_UNDER;
        w.nodes = -1;
        w.iters = 0;
        w.k = m.k_scan;
        w.dE = 0.0;
        w.norm_k_out = w.norm_k_in = 0.0;
        w.ex_out = w.ex_in = 0;
        w.n_in_bracket = 0;
        if (lo >= m.n_trial) {
            w.status |= EPSCU_STATUS_NOTFOUND;
            w.lo = w.hi = w.E = m.e_cap;
        } else {
            if (top < lo) top = lo;
            w.lo = lo == 0 ? m.e_lo : trial_energy(m, lo - 1);
            w.hi = trial_energy(m, top);
            w.E = __dmul_rn(0.5, __dadd_rn(w.lo, w.hi));
            w.n_in_bracket = c[top] - (lo == 0 ? 0 : c[lo - 1]);
            if (b.gam && lo > 0 && w.n_in_bracket == 1) {
                // the first energy of the refinement: the zero of the scan's
                // matching function interpolated between the bracket's ends,
                // when it falls from positive to negative there (one level, no
                // pole between); the midpoint otherwise
                const float* g = b.gam + (int64_t)p * b.n_trial;
                const float gl = g[lo - 1], gr = g[top];
                if (gl > 0.0f && gr < 0.0f && gl < INFINITY && gr > -INFINITY) {
                    const double t = fmin(0.95, fmax(0.05, (double)gl / ((double)gl - (double)gr)));
                    w.E = w.lo + t * (w.hi - w.lo);
                }
            }
        }
        w.lo0 = w.lo;
        w.hi0 = w.hi;
        w.j0 = m.i0;
        w.j1 = m.i1;
        w.bucket = w.rank = w.pad1 = 0;
        b.levels[m.level_base + s] = w;
    }
}

// Decay window at energy Eu (fast method; one call per warp, all lanes).
// Beyond the classical turning points of Eu (V > Eu there) the discrete
// solution decays at least by the constant-coefficient rate of the Numerov
// recurrence, acosh(1 + 6 t_i) per step with t_i = W_i - a Eu (for small t it
// is kappa h, the WKB exponent; for larger t it is below the true rate).  The
// window ends where that exponent, summed from the turning point, reaches
// `decay`: Dirichlet ends there change the solution by about e^-decay relative
// to its size at the turning point and an eigenvalue by a relative e^-2 decay,
// and every energy below Eu has a narrower window.  The classical choice of
// the start of the inward integration in Numerov-Cooley codes.
// Turning points come from binary searches on the suffix and prefix minima of
// V; the sums run over whole 32-point blocks beyond the turning point's block,
// a block of n points counting n acosh(1 + 6 (min W - a Eu)) (block minima
// rounded down, a Eu rounded up): a lower bound of the decay, so the window
// can only come out wider.  Returns [j0, j1] within [i0, i1].
__device__ int2 decay_window(const PotMeta& m, const DevBatch& b, double Eu, float decay) {
    const int lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    const float aEu = __double2float_ru(m.a * Eu);
    const float* Bm = b.Bmin + m.offf / 32;
    const int B_first = m.i0 >> 5, B_last = m.i1 >> 5;
    // the blocks of the outermost points at or below Eu: the last one whose
    // suffix minimum is, the first one whose prefix minimum is
    int t_out = m.k_scan >> 5, t_in = B_last;
    {
        const double* S = b.Bsuf + m.offf / 32;
        if (S[B_first] <= Eu) {
            int lo = B_first, hi = B_last;
            while (lo < hi) {
                const int mid = lo + (hi - lo + 1) / 2;
                if (S[mid] <= Eu) lo = mid;
                else hi = mid - 1;
            }
            t_out = lo;
        }
        const double* P = b.Bpre + m.offf / 32;
        int lo = B_first, hi = B_last;
        while (lo < hi) {
            const int mid = lo + (hi - lo) / 2;
            if (P[mid] <= Eu) hi = mid;
            else lo = mid + 1;
        }
        t_in = lo;
    }
    auto block_decay = [&](int B) {
        const int n = min((B << 5) + 31, m.i1) - max(B << 5, m.i0) + 1;
        return (float)n * acoshf(1.0f + 6.0f * fmaxf(Bm[B] - aEu, 0.0f));
    };
    // The block, going dir from B0, at which the e-folds summed from there on
    // reach decay (none: -1).  Four runs of 32 blocks at a time: their loads and
    // scans overlap, the sums are taken run by run (a run at a time waits ~700
    // cycles for each load: 0.33 ms a window kernel on a 2^20-point grid).
    auto reach = [&](int B0, int dir) {
        constexpr int kRuns = 4;
        const int n_blk = dir > 0 ? B_last - B0 + 1 : B0 - B_first + 1;
        float X = 0.0f;
        for (int q0 = 0; q0 < n_blk; q0 += 32 * kRuns) {
            float s[kRuns];
#pragma unroll
            for (int u = 0; u < kRuns; ++u) {
                const int q = q0 + 32 * u + lane;
                s[u] = q < n_blk ? block_decay(B0 + dir * q) : 0.0f;
            }
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
                for (int u = 0; u < kRuns; ++u) {
                    const float y = __shfl_up_sync(full, s[u], o);
                    if (lane >= o) s[u] += y;
                }
            }
#pragma unroll
            for (int u = 0; u < kRuns; ++u) {
                const unsigned hit = __ballot_sync(full, q0 + 32 * u + lane < n_blk && X + s[u] >= decay);
                if (hit) return B0 + dir * (q0 + 32 * u + __ffs(hit) - 1);
                X += __shfl_sync(full, s[u], 31);
            }
        }
        return -1;
    };
    const int b_out = reach(t_out + 1, 1), b_in = reach(t_in - 1, -1);
    const int j1 = b_out >= 0 ? min((b_out << 5) + 31, m.i1) : m.i1;
    const int j0 = b_in >= 0 ? max(b_in << 5, m.i0) : m.i0;
    if (j1 - j0 < 4) return make_int2(m.i0, m.i1);
    return make_int2(j0, j1);
}

// The order bucket of a window length: quarter octaves from 16 points up.
__device__ __forceinline__ int length_bucket(int len) {
    const int l = 31 - __clz(max(len, 16));
    return min(kBuckets - 1, 4 * (l - 4) + ((len >> (l - 2)) & 3));
}

// Decay window of every level slot (fast method), at E_up = hi0 + 2 delta:
// an energy above every energy the level's passes use (bracket, Newton steps,
// the repair's widened bracket), so one window serves all of them; its match
// point (the outer turning point at the first energy, on a strip boundary);
// and its place in the order of the level queues: windows longer than the
// long-window threshold (DevBatch::long_window, else default_long_window of
// the level count) on the long list (CTA per level), the rest on the warp
// list, fragile levels on two lists of their own, by length bucket and rank
// in it.  One warp per level.
__global__ void __launch_bounds__(128) window_kernel(DevBatch b) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int n_warps = (gridDim.x * blockDim.x) >> 5;
    const int total = b.hdr->total_levels;
    const int long_min = b.long_window > 0 ? b.long_window : default_long_window(total);
    const int cluster_min =
        b.cluster_list && b.long_window < kMinClusterWindow ? default_cluster_window(total) : 0x7fffffff;
    const int fragile_min = b.long_window > 0 ? b.long_window : default_fragile_window(total);
    for (int slot = warp; slot < total; slot += n_warps) {
        const LevelWork w = b.levels[slot];
        const PotMeta m = b.meta[w.p];
        int2 jw = make_int2(m.i0, m.i1);
        int k = w.k, len = 0, list = kListWarp;  // (a level without a bracket: last on the warp list)
        if (!(w.status & EPSCU_STATUS_NOTFOUND)) {
            jw = decay_window(m, b, w.hi0 + 2.0 * m.delta, kWindowDecay);
            k = match_index(m, b, w.E) & ~15;
            len = jw.y - jw.x;
            const int s = slot - m.level_base;
            const bool close = w.n_in_bracket > 1 || (s > 0 && w.hi0 - b.levels[slot - 1].lo0 < kFragileGap) ||
                               (s + 1 < m.n_out && b.levels[slot + 1].hi0 - w.lo0 < kFragileGap);
            // (where f can be negative the lane passes' counts are not the levels')
            const bool fragile = (m.status & EPSCU_STATUS_UNDER) || (close && !(m.status & EPSCU_STATUS_BELOW));
            list = fragile ? (len > fragile_min ? kListFragileLong : kListFragile)
                           : (len > cluster_min ? kListCluster : len > long_min ? kListLong : kListWarp);
        }
        if ((threadIdx.x & 31) == 0) {
            const int bucket = list * kBuckets + length_bucket(len);
            LevelWork* out = b.levels + slot;
            out->j0 = jw.x;
            out->j1 = jw.y;
            out->k = max(jw.x + 1, min(k, jw.y - 1));
            out->bucket = bucket;
            out->rank = atomicAdd(&b.hdr->hist[bucket], 1);
            if (list == kListLong || list == kListFragileLong) out->status = w.status | EPSCU_STATUS_LONG;
            if (list == kListCluster) out->status = w.status | EPSCU_STATUS_LONG | EPSCU_STATUS_CLUSTER;
        }
    }
}

// Decay windows of the scan: entry (p, q) is the window of the highest trial
// energy of block q (kScanWinBlock consecutive trial energies) of potential p,
// which contains the windows of every energy of the block.  One warp per entry.
__global__ void __launch_bounds__(128) scan_window_kernel(DevBatch b, int n_blk) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int n_warps = (gridDim.x * blockDim.x) >> 5;
    const int total = b.n * n_blk;
    for (int e = warp; e < total; e += n_warps) {
        const int p = e / n_blk, q = e % n_blk;
        const PotMeta m = b.meta[p];
        int2 jw = make_int2(m.i0, m.i1);
        if (!(m.status & EPSCU_STATUS_BAD)) {
            const int j = min((q + 1) * kScanWinBlock, b.n_trial) - 1;
            jw = decay_window(m, b, trial_energy(m, j), kWindowDecay);
        }
        if ((threadIdx.x & 31) == 0) b.scan_win[e] = jw;
    }
}

}  // namespace

void launch_prepare(const DevBatch& b, cudaStream_t s) {
    prepare_kernel<<<b.prep_tiles, kPrepThreads, 0, s>>>(b);
    block_minima_kernel<<<(b.prep_tiles + 3) / 4, 128, 0, s>>>(b, b.prep_tiles);
}

void launch_level_setup(const DevBatch& b, cudaStream_t s) {
    level_setup_kernel<<<1, 1024, 0, s>>>(b);
    if (!b.warp_list) unit_setup_kernel<<<1, 1024, 0, s>>>(b);
    bracket_kernel<<<b.n, 128, 0, s>>>(b);
}

void launch_window(const DevBatch& b, int sm_count, cudaStream_t s) {
    window_kernel<<<sm_count * 8, 128, 0, s>>>(b);
}

void launch_scan_window(const DevBatch& b, int sm_count, cudaStream_t s) {
    if (!b.scan_win) return;
    scan_window_kernel<<<sm_count * 8, 128, 0, s>>>(b, (b.n_trial + kScanWinBlock - 1) / kScanWinBlock);
}

}  // namespace epscu
