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

template <typename T, typename Op>
__device__ T block_reduce(T v, Op op, T* sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    const int nw = blockDim.x >> 5;
    v = threadIdx.x < nw ? sh[threadIdx.x] : sh[0];
    if (warp == 0)
        for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (threadIdx.x == 0) sh[0] = v;
    __syncthreads();
    v = sh[0];
    __syncthreads();
    return v;
}

struct MinI {
    __device__ int operator()(int a, int b) const { return min(a, b); }
};
struct MaxI {
    __device__ int operator()(int a, int b) const { return max(a, b); }
};
struct OrI {
    __device__ int operator()(int a, int b) const { return a | b; }
};

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
struct MinU {
    __device__ unsigned long long operator()(unsigned long long a, unsigned long long b) const { return min(a, b); }
};

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

__global__ void __launch_bounds__(kPrepThreads) prepare_kernel(DevBatch b) {
    __shared__ int shi[32];
    __shared__ unsigned long long shk[32];
    __shared__ unsigned long long s_kt;
    const int p = b.order[blockIdx.x];  // longest grids first (the tail is the last CTAs)
    PotMeta m = b.meta[p];
    const double* V = b.V64 + m.off;
    const int N = m.N;
    const int tid = threadIdx.x, nt = blockDim.x;

    // The per-point comparisons run on order-preserving integer images of the
    // doubles (dkey0), exact and on the integer pipes: min V and its finiteness,
    // the cut-off test a (V_i - V_min) <= 1/2 (monotone in V_i, so it holds
    // exactly up to a threshold image found once per potential by bisection
    // on the images with the FP64 test itself) and the first argmin; the only
    // FP64 instruction per point is W = a V.
    unsigned long long kmin = kKeyMax;
    int bad = 0;
    for (int i = tid; i < N; i += nt) {
        const double v = V[i];
        if ((((unsigned long long)__double_as_longlong(v) >> 52) & 0x7ffull) == 0x7ffull) bad = 1;  // inf, NaN
        else kmin = min(kmin, dkey0(v));
    }
    kmin = block_reduce(kmin, MinU(), shk);
    bad = block_reduce(bad, OrI(), shi);
    const double vmin = dkey_inv(kmin);

    const double h = __ddiv_rn(__dsub_rn(m.r_max, m.r_min), (double)(N - 1));
    const double a = __ddiv_rn(__dmul_rn(__dmul_rn(m.mu, h), h), 6.0);
    if (tid == 0) {
        // the largest image whose double passes the cut-off test (the test
        // holds at V_min; the images above +inf are NaNs, which fail it)
        unsigned long long lo = kmin, hi = kKeyMax;
        while (hi - lo > 1ull) {
            const unsigned long long mid = lo + (hi - lo) / 2;
            if (__dmul_rn(a, __dsub_rn(dkey_inv(mid), vmin)) <= 0.5) lo = mid;
            else hi = mid;
        }
        s_kt = lo;
    }
    __syncthreads();
    const unsigned long long kt = s_kt;
    int first = N, last = -1;
    for (int i = tid; i < N; i += nt) {
        if (dkey0(V[i]) <= kt) {
            first = min(first, i);
            last = max(last, i);
        }
    }
    first = block_reduce(first, MinI(), shi);
    last = block_reduce(last, MaxI(), shi);
    const int i0 = first < 1 ? 1 : first;
    const int i1 = last > N - 2 ? N - 2 : last;
    // a barrier inside the cut-offs that rises above them
    int steep = 0;
    for (int i = i0 + tid; i <= i1; i += nt) steep |= dkey0(V[i]) > kt;
    steep = block_reduce(steep, OrI(), shi);

    // argmin on [i0, i1], first occurrence
    unsigned long long bk = kKeyMax;
    int bi = N;
    for (int i = i0 + tid; i <= i1; i += nt) {
        const unsigned long long k = dkey0(V[i]);
        if (k < bk) {
            bk = k;
            bi = i;
        }
    }
    const unsigned long long gk = block_reduce(bk, MinU(), shk);
    int cand = (bk == gk) ? bi : N;
    const int k_scan = block_reduce(cand, MinI(), shi);

    // W = a V in FP64 and as an unevaluated (hi, lo) float pair; zero padding
    double* W = b.W64 + m.off;
    float2* Wf = b.Wf2 ? b.Wf2 + m.offf : nullptr;
    for (int i = tid; i < N; i += nt) {
        const double w = __dmul_rn(a, V[i]);
        W[i] = w;
        if (Wf) Wf[i] = split_double_rn(w);
    }

    // Suffix minima of V on [i0, i1] (M), and for the fast method prefix
    // minima (P) and the minima of a V over 32-point blocks clipped to
    // [i0, i1], rounded down to float (the decay-window bounds).  Coalesced
    // warp scans over the absolute 32-point blocks B0..B1: each warp owns a
    // contiguous run of blocks and scans it with shuffles, seeded with the
    // minimum of the runs to its right (suffix) or left (prefix).  Minima are
    // taken on an order-preserving integer image of the doubles (exact, and
    // no FP64 instruction at GB300's 1/64 rate).
    {
        const int lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
        const int B0 = i0 >> 5, B1 = i1 >> 5, nblk = i1 >= i0 ? B1 - B0 + 1 : 0;
        const int per = (nblk + nw - 1) / nw;
        const int wb0 = B0 + min(warp * per, nblk), wb1 = B0 + min((warp + 1) * per, nblk);  // [wb0, wb1)
        __shared__ unsigned long long s_run[32];
        auto load_key = [&](int B) {
            const int idx = (B << 5) + lane;
            return (idx >= i0 && idx <= i1) ? dkey(V[idx]) : kKeyMax;
        };
        // this warp's run minimum
        unsigned long long rm = kKeyMax;
        for (int B = wb0; B < wb1; ++B) rm = min(rm, load_key(B));
        for (int o = 16; o > 0; o >>= 1) rm = min(rm, __shfl_xor_sync(0xffffffffu, rm, o));
        if (lane == 0) s_run[warp] = rm;
        __syncthreads();
        double* M = b.Msuf + m.off;
        unsigned long long carry = kKeyMax;  // the minimum right of this warp's run
        for (int w = warp + 1; w < nw; ++w) carry = min(carry, s_run[w]);
        float* Bm = b.Mpre ? b.Bmin + m.offf / 32 : nullptr;
        for (int B = wb1 - 1; B >= wb0; --B) {
            unsigned long long k = load_key(B);
            // inclusive suffix minimum over the lanes (lane l: lanes l..31)
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long y = __shfl_down_sync(0xffffffffu, k, o);
                if (lane + o < 32) k = min(k, y);
            }
            const unsigned long long blk = __shfl_sync(0xffffffffu, k, 0);  // the block's minimum
            const int idx = (B << 5) + lane;
            if (idx >= i0 && idx <= i1) M[idx] = dkey_inv(min(k, carry));
            if (Bm && lane == 0) Bm[B] = __double2float_rd(__dmul_rn(a, dkey_inv(blk)));
            carry = min(carry, blk);
        }
        if (b.Mpre) {
            double* P = b.Mpre + m.off;
            carry = kKeyMax;  // the minimum left of this warp's run
            for (int w = 0; w < warp; ++w) carry = min(carry, s_run[w]);
            for (int B = wb0; B < wb1; ++B) {
                unsigned long long k = load_key(B);
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned long long y = __shfl_up_sync(0xffffffffu, k, o);
                    if (lane >= o) k = min(k, y);
                }
                const int idx = (B << 5) + lane;
                if (idx >= i0 && idx <= i1) P[idx] = dkey_inv(min(k, carry));
                carry = min(carry, __shfl_sync(0xffffffffu, k, 31));
            }
        }
    }

    if (tid == 0) {
        int status = 0;
        if (bad) status |= EPSCU_STATUS_BAD | EPSCU_STATUS_NONFINITE;
        if (i1 - i0 < 2) status |= EPSCU_STATUS_BAD;
        if (!(m.e_cap > vmin)) status |= EPSCU_STATUS_BAD;
        m.h = h;
        m.a = a;
        m.e_lo = vmin;
        m.i0 = i0;
        m.i1 = i1;
        m.k_scan = k_scan < N ? k_scan : i0;
        m.delta = __ddiv_rn(__dsub_rn(m.e_cap, vmin), (double)m.n_trial);
        const double tol = b.tol > 0.0 ? b.tol : 1e-12;
        int K = 0;
        for (double w = m.delta; w > tol && K < 200; w = __dmul_rn(w, 0.5)) ++K;
        m.n_bisect = K;
        const double kmax = sqrt(2.0 * m.mu * (m.e_cap - vmin));
        if (kmax * h > 1.0) status |= EPSCU_STATUS_UNDER;
        if (steep) status |= EPSCU_STATUS_STEEP;
        m.status = status;
        if (b.under_list && (status & EPSCU_STATUS_UNDER) && !(status & EPSCU_STATUS_BAD))
            b.under_list[atomicAdd(&b.hdr->n_under, 1)] = p;
        m.n_total = 0;
        m.n_out = 0;
        b.meta[p] = m;
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
    const int t_out = match_index(m, b.Msuf, Eu);
    int t_in;
    {
        // first i with min(V_i0 .. V_i) <= Eu (the prefix minima do not increase)
        const double* P = b.Mpre + m.off;
        int lo = m.i0, hi = m.i1;
        while (lo < hi) {
            const int mid = lo + (hi - lo) / 2;
            if (P[mid] <= Eu) hi = mid;
            else lo = mid + 1;
        }
        t_in = lo;
    }
    const int B_first = m.i0 >> 5, B_last = m.i1 >> 5;
    auto block_decay = [&](int B) {
        const int n = min((B << 5) + 31, m.i1) - max(B << 5, m.i0) + 1;
        return (float)n * acoshf(1.0f + 6.0f * fmaxf(Bm[B] - aEu, 0.0f));
    };
    int j1 = m.i1;
    float X = 0.0f;
    for (int B0 = (t_out >> 5) + 1; B0 <= B_last; B0 += 32) {
        const int B = B0 + lane;
        float s = B <= B_last ? block_decay(B) : 0.0f;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float y = __shfl_up_sync(full, s, o);
            if (lane >= o) s += y;
        }
        const unsigned hit = __ballot_sync(full, B <= B_last && X + s >= decay);
        if (hit) {
            j1 = min(((B0 + __ffs(hit) - 1) << 5) + 31, m.i1);
            break;
        }
        X += __shfl_sync(full, s, 31);
    }
    int j0 = m.i0;
    X = 0.0f;
    for (int B0 = (t_in >> 5) - 1; B0 >= B_first; B0 -= 32) {
        const int B = B0 - lane;
        float s = B >= B_first ? block_decay(B) : 0.0f;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float y = __shfl_up_sync(full, s, o);
            if (lane >= o) s += y;
        }
        const unsigned hit = __ballot_sync(full, B >= B_first && X + s >= decay);
        if (hit) {
            j0 = max((B0 - (__ffs(hit) - 1)) << 5, m.i0);
            break;
        }
        X += __shfl_sync(full, s, 31);
    }
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
    const int fragile_min = b.long_window > 0 ? b.long_window : default_fragile_window(total);
    for (int slot = warp; slot < total; slot += n_warps) {
        const LevelWork w = b.levels[slot];
        const PotMeta m = b.meta[w.p];
        int2 jw = make_int2(m.i0, m.i1);
        int k = w.k, len = 0, list = kListWarp;  // (a level without a bracket: last on the warp list)
        if (!(w.status & EPSCU_STATUS_NOTFOUND)) {
            jw = decay_window(m, b, w.hi0 + 2.0 * m.delta, kWindowDecay);
            k = match_index(m, b.Msuf, w.E) & ~15;
            len = jw.y - jw.x;
            const int s = slot - m.level_base;
            const bool fragile = (m.status & EPSCU_STATUS_UNDER) ||
                                 w.n_in_bracket > 1 || (s > 0 && w.hi0 - b.levels[slot - 1].lo0 < kFragileGap) ||
                                 (s + 1 < m.n_out && b.levels[slot + 1].hi0 - w.lo0 < kFragileGap);
            list = fragile ? (len > fragile_min ? kListFragileLong : kListFragile)
                           : (len > long_min ? kListLong : kListWarp);
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
    prepare_kernel<<<b.n, kPrepThreads, 0, s>>>(b);
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
