// sfwi_ot.cu — per-trace 1D quadratic-Wasserstein misfit and adjoint source.
//
// The reference declares OT, OT_power and OT_alltrace (sfwi-stage1/FD2DGPU.cuh:
// 21-25, argument order obs_x, obs_z, cal_x, cal_z, res_x, res_z, length,
// tracenum, misfit) and defines none of them.  This is the 1D W2 misfit
// between positive-normalised traces, written from its definition:
//   weights   p(u) = exp((u - max u)/sigma)          (OT, OT_alltrace)
//             p(u) = u^2 + 1e-3 sigma^2              (OT_power)
//             sigma = max|obs| of the trace, floored at 1e-3 max|obs| of the
//             gather (OT, OT_power), or max|obs| of the gather (OT_alltrace)
//   densities f = p(cal)/sum p(cal), g = p(obs)/sum p(obs)
//   CDFs      F_k = sum_{j<=k} f_j,  G_k likewise
//   transport T_k = G^-1(F_k) = dt (m + (F_k - G_{m-1})/g_m), G_{m-1} <= F_k < G_m
//   misfit    W = sum_k ((k+1) dt - T_k)^2 f_k
//   adjoint   A_j = ((j+1)dt - T_j)^2 - 2 sum_{k>=j} ((k+1)dt - T_k) f_k dt / g_m(k)
//             res_i = (1/2) (A_i - sum_j f_j A_j) / sum p(cal) * p'(cal_i)
// res is (1/2) dW/dcal, the scaling of the L2 residual (misfit sum r^2,
// adjoint source r).
//
// Two kernels.  k_ot_fp64 forms the adjoint sources of gradient runs, all sums,
// products and divisions in FP64 (the FP64 pipe, 1/64 of the FP32 rate, is 86 % busy:
// 2.87 ms for both components of 3760 traces of 3000 samples; 1 to 2 % of a gradient run).
// k_ot serves the calls that want a gather's misfit and residuals by themselves
// and takes 0.50 ms (OT_power 0.67): there the CDFs are 64-bit integers and the rest is in float
// pairs.  Its residuals differ from k_ot_fp64's in the last bit of one in 2000, which is
// nothing by itself; but an FP32 propagation of that source ends 7e-6 away from
// the other's after 3000 steps (as far as each is from FP64), so gradient
// runs stay with the FP64 form and their bits.
// The integers: CDFs are sums of positive weights, in units of 2^-s of the
// largest one, s such that a trace's sum stays below 2^62 (OT_power's weights are
// integers from the start, from the exact square of u's 24 bits).  Integer sums are
// exact in any order, so F_k - G_{m-1} and the search have no rounding but the weights'
// own (2^-50 at 3000 samples) and that of the ratio of the sums, 2^-63, upwards:
// densities of equal shape have equal CDFs.  What follows the search (r, its
// square, the adjoint weights and their sums) is in float pairs of 48 bits
// (D2, sfwi_d2.cuh).  The two cancellations are kept out of them: k+1 - T_k
// is done in integers, and A_j - sum f A relative to A at the largest weight,
// which matters where one sample holds nearly all of it.
// In both kernels the exponential weights are FP32 (expf of the argument rounded to
// FP32): their argument is at most 0, so a weight is 1 at the trace's maximum and
// its relative rounding of about 1e-7 stays far below the 1e-4 parity bar.  Against the
// formulas in quad precision, over 3000 random gathers: residuals (median) 2.9e-7 and
// misfits 9e-9 for OT, 1.8e-7 and 2e-8 for OT_alltrace in either kernel, from those
// weights; OT_power residuals 2.6e-8 in either, misfits 1.5e-15 (k_ot_fp64 4e-16).
// One CTA handles one (trace, component); prefix and suffix sums are block
// scans built on warp shuffles.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cudaTypedefs.h>
#include <mutex>

#include "sfwi_d2.cuh"
#include "sfwi_launch.h"

namespace sfwi {

using u64 = unsigned long long;

constexpr int OT_THREADS = 256;  // of k_ot_fp64

__device__ __forceinline__ double warp_incl_scan(double v) {
    const int l = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, v, o);
        if (l >= o) v += u;
    }
    return v;
}

// exclusive block scan of one value per thread (thread order)
__device__ double block_excl_scan(double v, double *wsum) {
    const double inc = warp_incl_scan(v);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 31) wsum[w] = inc;
    __syncthreads();
    if (w == 0) {
        const int nw = blockDim.x >> 5;
        double t = l < nw ? wsum[l] : 0.0;
        const double ti = warp_incl_scan(t);
        if (l < nw) wsum[l] = ti - t;
    }
    __syncthreads();
    const double r = wsum[w] + inc - v;
    __syncthreads();
    return r;
}

__device__ double block_reduce(double v, double *wsum) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) wsum[w] = v;
    __syncthreads();
    double t = 0.0;
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) t += wsum[i];
    __syncthreads();
    return t;
}

// exclusive suffix sums over the threads of the block: thread t gets the sum
// of v over threads t+1 .. blockDim.x-1 (cs: blockDim.x doubles of shared
// memory; wsum as block_excl_scan)
__device__ double block_excl_suffix(double v, double *cs, double *wsum) {
    const int t = threadIdx.x, T = blockDim.x;
    cs[t] = v;
    __syncthreads();
    const double e = block_excl_scan(cs[T - 1 - t], wsum);  // sum over threads after T-1-t
    cs[T - 1 - t] = e;
    __syncthreads();
    const double r = cs[t];
    __syncthreads();
    return r;
}

__device__ __forceinline__ D2 reciprocal(D2 d) {
    // two terms of the series from an approximate reciprocal of the high part
    const float x = __fdividef(1.f, d.h);
    float e = __fmaf_rn(-d.h, x, 1.f);
    e = __fmaf_rn(-d.l, x, e);
    return quick2(x, __fmul_rn(x, __fmaf_rn(e, e, e)));
}
__device__ __forceinline__ D2 to_d2(double v) {
    const float h = (float)v;
    return D2{h, (float)(v - (double)h)};
}
__device__ __forceinline__ double to_f64(D2 a) { return (double)a.h + (double)a.l; }
// an integer below 2^63, to 48 bits
__device__ __forceinline__ D2 to_d2(u64 x) {
    const float a = (float)(unsigned)(x >> 40), b = (float)((unsigned)(x >> 16) & 0xffffffu),
                c = (float)((unsigned)x & 0xffffu);
    const D2 s = quick2(a * 1099511627776.f, b * 65536.f);
    return quick2(s.h, __fadd_rn(s.l, c));
}
__device__ __forceinline__ D2 to_d2(long long x) {
    const D2 m = to_d2((u64)(x < 0 ? -x : x));
    return x < 0 ? -m : m;
}
// x 2^s of a float 0 <= x <= 1 (24 <= s <= 62), rounded
__device__ __forceinline__ u64 fixed_point(float x, int s) {
    const unsigned b = __float_as_uint(x), e = b >> 23;
    const u64 m = (u64)((b & 0x7fffffu) | 0x800000u) << (s - 22);
    return e == 0 ? 0 : ((m >> min(127u - e, 63u)) + 1) >> 1;
}

// ---------------------------------------------------------------------------
// block sums (blockDim.x a multiple of 32); `sm`: 66 64-bit words, not read
// by other threads when a call begins
// ---------------------------------------------------------------------------
__device__ __forceinline__ D2 shfl_down(D2 v, int o) {
    return D2{__shfl_down_sync(0xffffffffu, v.h, o), __shfl_down_sync(0xffffffffu, v.l, o)};
}
// exclusive sums over the threads before this one, of two values at once; the
// totals go to sm[64], sm[65] (the second level of these sums is one warp's work: done by
// every thread it was a quarter of the kernel's instructions)
__device__ void block_scan2(u64 &a, u64 &b, u64 *sm) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    auto warp_scan = [&](u64 &x, u64 &y) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const u64 u = __shfl_up_sync(0xffffffffu, x, o), v = __shfl_up_sync(0xffffffffu, y, o);
            if (l >= o) x += u, y += v;
        }
    };
    u64 x = a, y = b;
    warp_scan(x, y);
    if (l == 31) sm[w] = x, sm[32 + w] = y;
    __syncthreads();
    if (w == 0) {
        const u64 p = l < nw ? sm[l] : 0, q = l < nw ? sm[32 + l] : 0;
        u64 u = p, v = q;
        warp_scan(u, v);
        sm[l] = u - p, sm[32 + l] = v - q;
        if (l == 31) sm[64] = u, sm[65] = v;
    }
    __syncthreads();
    a = sm[w] + x - a;
    b = sm[32 + w] + y - b;
}
// the sum over the threads after this one
__device__ D2 block_suffix(D2 v, u64 *sm) {
    D2 *ws = reinterpret_cast<D2 *>(sm);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    auto warp_suffix = [&](D2 x) {  // this lane's and those after it
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const D2 u = shfl_down(x, o);
            if (l + o < 32) x = x + u;
        }
        return x;
    };
    auto drop_own = [&](D2 x) {
        x = shfl_down(x, 1);
        return l == 31 ? D2{0.f, 0.f} : x;
    };
    const D2 x = warp_suffix(v), after = drop_own(x);
    if (l == 0) ws[w] = x;
    __syncthreads();
    if (w == 0) {
        const D2 t = drop_own(warp_suffix(l < nw ? ws[l] : D2{0.f, 0.f}));
        ws[l] = t;
    }
    __syncthreads();
    return after + ws[w];
}
// the sums of two values; valid in thread 0
__device__ void block_sum2(D2 &v, D2 &u, u64 *sm) {
    D2 *ws = reinterpret_cast<D2 *>(sm);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    auto warp_sum = [&](D2 x) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x = x + shfl_down(x, o);
        return x;
    };
    v = warp_sum(v), u = warp_sum(u);
    if (l == 0) ws[w] = v, ws[32 + w] = u;
    __syncthreads();
    if (w == 0) {
        v = warp_sum(l < nw ? ws[l] : D2{0.f, 0.f});
        u = warp_sum(l < nw ? ws[32 + l] : D2{0.f, 0.f});
    }
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}
__device__ double block_max(double v, double *wsum) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) wsum[w] = v;
    __syncthreads();
    double t = -DBL_MAX;
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) t = fmax(t, wsum[i]);
    __syncthreads();
    return t;
}

// smallest m >= lo with G[m] > y, capped at n-1 (G non-decreasing and every
// index below lo known to hold G <= y): a galloping search from lo, so
// consecutive quantiles of one thread cost a few probes instead of a full
// binary search; the answer is that of a binary search over [0, n-1)
__device__ __forceinline__ int first_above(const u64 *G, int n, u64 y, int lo) {
    if (lo >= n - 1) return n - 1;
    if (G[lo] > y) return lo;
    int prev = lo, step = 1, hi;
    for (;;) {
        const int nx = prev + step;
        if (nx >= n - 1) {
            hi = n - 1;
            break;
        }
        if (G[nx] > y) {
            hi = nx;
            break;
        }
        prev = nx;
        step <<= 1;
    }
    int l = prev + 1;
    while (l < hi) {
        const int mid = (l + hi) >> 1;
        if (G[mid] > y)
            hi = mid;
        else
            l = mid + 1;
    }
    return l;
}

// ---------------------------------------------------------------------------
// the FP64 form, for gradient runs
// ---------------------------------------------------------------------------
// The GB300's FP64 rate is a small fraction of its FP32 rate, so the kernel
// spends FP64 operations sparingly: each thread owns one contiguous chunk of
// samples, the positivity transform (one exp per sample and trace) is
// evaluated once and kept, the CDF of the synthetic trace is formed on the
// fly from the chunk's running sum, the quantile search continues from the
// previous sample's quantile, and divisions by per-trace constants are
// multiplications by their reciprocals.
constexpr int OT_MAX_CHUNK = 32;  // samples per thread of the shared-memory form: nt <= 32 * OT_THREADS

// LONG = false: the per-trace arrays in shared memory (traces up to
// ot_max_nt() samples); LONG = true: in the caller's global scratch, five
// arrays of nt doubles per (trace, component), for longer traces (the
// transport residuals r then go to the fifth array instead of registers).
template <bool LONG>
__global__ void __launch_bounds__(OT_THREADS) k_ot_fp64(OtArgs a) {
    extern __shared__ double ot_sm[];
    __shared__ double wsum[32];
    __shared__ double cs[OT_THREADS];
    const int n = a.nt;
    // G: CDF of the observed trace; g: its density; P: p(cal); Q: the terms
    // r f dt / g, then the adjoint weights A; R (long form): r
    double *G = LONG ? a.scratch + (size_t)blockIdx.x * 5 * n : ot_sm;
    double *g = G + n, *P = g + n, *Q = P + n;
    double *R = LONG ? Q + n : nullptr;
    const int tr = blockIdx.x >> 1, comp = blockIdx.x & 1;
    const size_t o = (size_t)tr * n;
    const float *cal = (comp ? a.cal_x : a.cal_z) + o;
    const float *cal2 = a.cal2_z ? (comp ? a.cal2_x : a.cal2_z) + o : nullptr;
    const float *obs = (comp ? a.obs_x : a.obs_z) + o;
    float *res = (comp ? a.res_x : a.res_z) + o;
    double sigma = a.sigma[2 * tr + comp];
    if (!(sigma > 0.0)) sigma = 1.0;
    const double inv_sigma = 1.0 / sigma;
    const bool pw = a.kind == 2;
    auto pred = [&](int k) -> double { return cal2 ? (double)(cal[k] + cal2[k]) : (double)cal[k]; };
    const int chunk = (n + blockDim.x - 1) / blockDim.x;
    const int k0 = min(n, (int)threadIdx.x * chunk), k1 = min(n, k0 + chunk);

    float mc = -FLT_MAX, mo = -FLT_MAX;
    for (int k = k0; k < k1; k++) {
        mc = fmaxf(mc, cal2 ? cal[k] + cal2[k] : cal[k]);
        mo = fmaxf(mo, obs[k]);
    }
    const double cmax = block_max(mc, wsum), omax = block_max(mo, wsum);
    const double eps = 1e-3 * sigma * sigma;
    auto pf = [&](double u) { return pw ? u * u + eps : (double)expf((float)((u - cmax) * inv_sigma)); };
    auto pg = [&](double u) { return pw ? u * u + eps : (double)expf((float)((u - omax) * inv_sigma)); };

    double sf = 0.0, sg = 0.0;
    for (int k = k0; k < k1; k++) {
        const double x = pf(pred(k)), y = pg((double)obs[k]);
        P[k] = x;
        g[k] = y;
        sf += x;
        sg += y;
    }
    const double Sf = block_reduce(sf, wsum), Sg = block_reduce(sg, wsum);
    const double inv_Sf = 1.0 / Sf, inv_Sg = 1.0 / Sg;
    // densities, the chunk sums of both, and the CDF G of the observed trace
    double cf = 0.0, cg = 0.0;
    for (int k = k0; k < k1; k++) {
        g[k] *= inv_Sg;
        cg += g[k];
        cf += P[k] * inv_Sf;
    }
    const double offF = block_excl_scan(cf, wsum), offG = block_excl_scan(cg, wsum);
    {
        double run = offG;
        for (int k = k0; k < k1; k++) {
            run += g[k];
            G[k] = run;
        }
    }
    __syncthreads();

    // transport T_k = G^-1(F_k) and the misfit terms
    double w = 0.0, sq = 0.0, Fk = offF;
    double r_loc[LONG ? 1 : OT_MAX_CHUNK];
    int m = 0;
    for (int i = 0; i < k1 - k0; i++) {
        const int k = k0 + i;
        const double fk = P[k] * inv_Sf;
        Fk += fk;
        m = first_above(reinterpret_cast<const u64 *>(G), n, (u64)__double_as_longlong(Fk), m);  // (order of the bits)
        const double gm = g[m];
        const double inv_gm = 1.0 / gm;
        const double Gm1 = m > 0 ? G[m - 1] : 0.0;
        const double T = a.dt * (m + (Fk - Gm1) * inv_gm);
        const double r = (k + 1) * a.dt - T;
        w += r * r * fk;
        if (LONG)
            R[k] = r;
        else
            r_loc[i] = r;
        const double q = r * fk * a.dt * inv_gm;
        Q[k] = q;
        sq += q;
    }
    // suffix sums of q, the adjoint weights A_k = r_k^2 - 2 sum_{j>=k} q_j and
    // their f-weighted sum
    const double offQ = block_excl_suffix(sq, cs, wsum);
    double fa = 0.0, run = offQ;
    for (int i = k1 - k0 - 1; i >= 0; i--) {
        const int k = k0 + i;
        run += Q[k];
        const double rk = LONG ? R[k] : r_loc[i];
        const double A = rk * rk - 2.0 * run;
        Q[k] = A;
        fa += P[k] * inv_Sf * A;
    }
    const double FA = block_reduce(fa, wsum);
    const double W = block_reduce(w, wsum);
    for (int k = k0; k < k1; k++) {
        const double dp = pw ? 2.0 * pred(k) : P[k] * inv_sigma;
        res[k] = (float)(0.5 * (Q[k] - FA) * inv_Sf * dp);
    }
    if (threadIdx.x == 0) a.trace_misfit[2 * tr + comp] = W;
}

// ---------------------------------------------------------------------------
// integers and float pairs, for a gather's misfit by itself
// ---------------------------------------------------------------------------
// LONG = false: the per-trace arrays in shared memory (traces up to
// ot_max_nt() samples); LONG = true: in the caller's global scratch, five
// arrays of nt doubles per (trace, component), for longer traces.
// POWER: OT_power's weights, in units of sigma^2: v^2 + 1e-3 with v = u / sigma.
// Each thread owns one contiguous run of an odd number of samples (`run`), so that the
// threads' accesses to 64-bit arrays in shared memory fall into different
// banks; the quantile search continues from the previous sample's.
// Bound by instructions (500 us for 3760 traces of 3000 samples, 66 % of the issue slots, DRAM 6 %; OT_power
// 668 us, 57 %); 56 registers let three CTAs of 352 threads share an SM (64: two; 685 us for 590 in an
// earlier form).
template <bool LONG, bool POWER>
__global__ void __maxnreg__(56) k_ot(OtArgs a, int run) {
    extern __shared__ u64 ot_words[];
    // block sums; a call's words may be read until the next barrier, so calls alternate
    __shared__ u64 ws[2][66];
    // per-trace constants, formed by thread 0 in FP64
    __shared__ struct {
        float mc, mo;
        double inv_sigma, inv_S, scale;  // inv_S: of p's units
        D2 is, c, norm, sc, ref, FA;
        u64 ratio, kc, ko, least_c, least_o;
        int wide, ec, eo, bc, bo, shift, sc2, so2, kref;
    } tc;
    const int n = a.nt;
    // G: CDF of the observed trace; B: the adjoint weights but for a constant
    // per thread (first: obs); U: p(cal), POWER: cal
    u64 *G = LONG ? reinterpret_cast<u64 *>(a.scratch) + (size_t)blockIdx.x * 5 * n : ot_words;
    D2 *B = reinterpret_cast<D2 *>(G + n);
    float *U = reinterpret_cast<float *>(B + n), *O = reinterpret_cast<float *>(B);
    const int tr = blockIdx.x >> 1, comp = blockIdx.x & 1;
    const size_t o = (size_t)tr * n;
    const float *cal = (comp ? a.cal_x : a.cal_z) + o;
    const float *cal2 = a.cal2_z ? (comp ? a.cal2_x : a.cal2_z) + o : nullptr;
    const float *obs = (comp ? a.obs_x : a.obs_z) + o;
    float *res = (comp ? a.res_x : a.res_z) + o;
    // both traces (obs in B's place until its weights are taken), their
    // largest values and magnitudes
    float mc = -FLT_MAX, mo = -FLT_MAX, ac = 0.f, ao = 0.f;
#pragma unroll 4
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const float u = cal2 ? cal[k] + cal2[k] : cal[k], v = obs[k];
        U[k] = u;
        O[k] = v;
        mc = fmaxf(mc, u), ac = fmaxf(ac, fabsf(u));
        mo = fmaxf(mo, v), ao = fmaxf(ao, fabsf(v));
    }
    // units of the weights: 2^-bits of 2^ec, 2^eo, the powers of two above them
    const int all_ones = 62 - (32 - __clz((n - 1) | 1));
    int bc = all_ones, bo = all_ones;
    {
        float *w = reinterpret_cast<float *>(ws[0]);
        mc = warp_max(mc), mo = warp_max(mo), ac = warp_max(ac), ao = warp_max(ao);
        const int l = threadIdx.x & 31, nw = blockDim.x >> 5;
        if (l == 0) {
            float *q = w + 4 * (threadIdx.x >> 5);
            q[0] = mc, q[1] = mo, q[2] = ac, q[3] = ao;
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            mc = warp_max(l < nw ? w[4 * l] : -FLT_MAX), mo = warp_max(l < nw ? w[4 * l + 1] : -FLT_MAX);
            ac = warp_max(l < nw ? w[4 * l + 2] : 0.f), ao = warp_max(l < nw ? w[4 * l + 3] : 0.f);
        }
    }
    if (threadIdx.x == 0) {
        double sigma = a.sigma[2 * tr + comp];
        if (!(sigma > 0.0)) sigma = 1.0;
        const double inv = 1.0 / sigma;
        tc.mc = POWER ? ac : mc, tc.mo = mo;
        tc.kref = INT_MAX, tc.ref = D2{0.f, 0.f};
        tc.inv_sigma = inv;
        tc.is = to_d2(inv);
        // Scales at which a float pair could overflow or lose bits: the
        // weights' arguments and the last product are then formed in FP64.
        tc.wide = !(sigma > 1e-15 && sigma < 1e15 && fmaxf(ac, ao) < 1e9 * sigma);
        tc.ec = tc.eo = 0;
        if (POWER) {
            // (no finite magnitude: every weight is NaN, and the result)
            frexp(ac * inv * (ac * inv) + 1e-3, &tc.ec);
            frexp(ao * inv * (ao * inv) + 1e-3, &tc.eo);
        }
    }
    __syncthreads();
    mc = tc.mc, mo = tc.mo;
    const int ec = tc.ec, eo = tc.eo;
    const bool wide = tc.wide;
    const double inv_sigma = tc.inv_sigma;
    const D2 is = tc.is;
    if (POWER && !wide) {
        // A few large samples and many near 1e-3: the sum of the weights is
        // far below their number, which leaves bits for the small ones.
        const float qc = __int_as_float((127 - ec) << 23), qo = __int_as_float((127 - eo) << 23);
        float x = 0.f, y = 0.f;
        for (int k = threadIdx.x; k < n; k += blockDim.x) {
            const float u = U[k] * is.h, v = O[k] * is.h;
            x += (u * u + 1e-3f) * qc, y += (v * v + 1e-3f) * qo;
        }
        D2 sx{x, 0.f}, sy{y, 0.f};
        block_sum2(sx, sy, ws[1]);
        if (threadIdx.x == 0) {
            // (a margin for the rounding of these sums)
            auto room = [&](float t) {
                return t > 0.f ? min(max(all_ones, 62 - (ilogbf(1.01f * t) + 1)), 61) : all_ones;
            };
            tc.bc = room(sx.h), tc.bo = room(sy.h);
        }
        __syncthreads();
        bc = tc.bc, bo = tc.bo;
    }
    if (POWER) {
        if (threadIdx.x == 0) {
            // (u / sigma)^2 in the weights' units: u^2 times a factor of 53 bits
            auto factor = [&](int bits, u64 &k, int &s, u64 &least) {
                const u64 q = (u64)__double_as_longlong(ldexp(inv_sigma * inv_sigma, bits));
                k = ((q & 0xfffffffffffffULL) | 0x10000000000000ULL) << 11;
                s = 263 + 1075 - (int)(q >> 52);
                least = __double2ull_rn(ldexp(1e-3, bits));
            };
            factor(bc - ec, tc.kc, tc.sc2, tc.least_c);
            factor(bo - eo, tc.ko, tc.so2, tc.least_o);
        }
        __syncthreads();
    }
    // A weight: kinds 1 and 3 in FP32; POWER in units (its 62 bits, from the
    // exact square of u's 24)
    auto weight = [&](float u, float top) -> float {
        if (wide) return expf((float)(((double)u - (double)top) * inv_sigma));
        const D2 d = sum2(u, -top) * is;
        return expf(d.h + d.l);
    };
    auto power_units = [&](float u, u64 factor, int s, u64 least) -> u64 {
        const unsigned b = __float_as_uint(u), e = b >> 23 & 0xffu;
        const u64 m = (b & 0x7fffffu) | (e ? 0x800000u : 0u);
        const int r = min(max(s - 2 * (int)max(e, 1u) - 1, 0), 63);  // (the last place rounds)
        return (((__umul64hi(m * m << 16, factor) >> r) + 1) >> 1) + least;
    };
    const int k0 = min(n, (int)threadIdx.x * run), k1 = min(n, k0 + run);

    // weights, the sums of both runs, and the CDF G of the observed trace
    u64 F = 0, offG = 0;
    bool bad = POWER && inv_sigma == 0.0;  // (an infinite sigma, and with it every weight)
    for (int k = k0; k < k1; k++) {
        const float u = U[k], v = O[k];
        if (POWER) {
            if (fabsf(u) == mc) atomicMin(&tc.kref, k);
            bad |= !(fabsf(u) <= FLT_MAX && fabsf(v) <= FLT_MAX);
            F += power_units(u, tc.kc, tc.sc2, tc.least_c);
            offG += power_units(v, tc.ko, tc.so2, tc.least_o);
        } else {
            const float x = weight(u, mc), y = weight(v, mo);
            bad |= !(x <= 2.f && y <= 2.f);
            if (x == 1.f) atomicMin(&tc.kref, k);
            U[k] = x;
            F += fixed_point(x, bc);
            offG += fixed_point(y, bo);
        }
        G[k] = offG;
    }
    bad = __syncthreads_or(bad);
    block_scan2(F, offG, ws[1]);
    for (int k = k0; k < k1; k++) G[k] += offG;
    if (threadIdx.x == 0) {
        const double sf = (double)ws[1][64], sg = (double)ws[1][65], q = sg / sf;
        // ratio of the units, SG / SF = (ratio / 2^63) 2^shift, rounded up: F SG / SF
        // rounds down to the integer wherever it is one (equal shapes have r = 0)
        const u64 rb = (u64)__double_as_longlong(q);
        tc.ratio = ((rb & 0xfffffffffffffULL) | 0x10000000000000ULL) << 11;
        tc.shift = (int)(rb >> 52) - 1023;
        if (abs(tc.shift) < 62) {
            // (FP64's 53 bits, and the rest from the remainder)
            const u64 s = ws[1][64];
            __int128 d = ((unsigned __int128)ws[1][65] << (63 - tc.shift)) - (unsigned __int128)tc.ratio * s;
            const int c = __float2int_rn(__ll2float_rn((long long)(d >> 32)) * __fdividef(4294967296.f, (float)s));
            u64 r = tc.ratio + c;
            d -= (__int128)c * s;
            for (int i = 0; i < 4 && d > 0; i++, d -= s) r++;
            for (int i = 0; i < 4 && d <= -(__int128)s; i++, d += s) r--;
            tc.ratio = r;
        }
        // f / g = (p / SF) (SG / g), p and g in their units; sums of weights are
        // SF 2^-bc (p of kinds 1, 3: without the 2^-bc)
        const double inv_S = ldexp(1.0 / sf, bc);
        tc.c = to_d2(-2.0 * (POWER ? q : ldexp(q, bc)));
        tc.inv_S = POWER ? 1.0 / sf : inv_S;
        tc.norm = to_d2(-tc.inv_S);
        // res = (1/2) (A - FA) / S p'(u): p' = p / sigma, or (POWER, p in units
        // of 2^ec sigma^2) 2 (u / sigma) / sigma
        tc.scale = a.dt * a.dt * inv_S * (POWER ? ldexp(1.0, -ec) : 0.5);
        tc.sc = to_d2(tc.scale);
    }
    __syncthreads();
    if (bad) {
        // a weight without a finite value leaves none in the trace
        for (int k = threadIdx.x; k < n; k += blockDim.x) res[k] = __int_as_float(0x7fffffff);
        if (threadIdx.x == 0) a.trace_misfit[2 * tr + comp] = __longlong_as_double(0x7fffffffffffffffLL);
        return;
    }
    // transport, in samples: r_k = k + 1 - T_k = i - (F_k - G_{m-1}) / g_m, i = k + 1 - m
    // Adjoint weights in samples squared: A_k = r_k^2 + c sum_{j>=k} q_j, q_j = r_j p_j / g_m(j).
    // The sum is the block's after this thread's samples, plus the thread's own less what
    // comes before k, so a thread keeps B_k = r_k^2 - c sum_{j<k} q_j and adds a
    // constant when the block's sums are known.
    // Where one sample holds nearly all the weight, its A - FA is a small
    // difference: FA is formed relative to A of the sample of the largest
    // weight, kref, whose term is then none.
    const int kref = tc.kref;
    const u64 ratio = tc.ratio;
    const int up = 1 + min(max(tc.shift, 0), 62), down = min(max(-tc.shift, 0), 63);
    const D2 c = tc.c;
    D2 w{0.f, 0.f}, sq{0.f, 0.f}, fb{0.f, 0.f}, sp{0.f, 0.f};
    int m = 0;
    for (int k = k0; k < k1; k++) {
        D2 pk;
        if (POWER) {
            const u64 x = power_units(U[k], tc.kc, tc.sc2, tc.least_c);
            pk = to_d2(x);
            F += x;
        } else {
            pk = D2{U[k], 0.f};
            F += fixed_point(U[k], bc);
        }
        const u64 y = __umul64hi(F << up, ratio) >> down;
        m = first_above(G, n, y, m);
        const u64 below = m > 0 ? G[m - 1] : 0, g = G[m] - below;
        // (r of -1 to 1 from integers alone: near equal traces lose nothing)
        const int i = k + 1 - m;
        const u64 num = i == 1 ? g - (y - below) : y - below;
        const D2 ig = reciprocal(to_d2(g)), q1 = to_d2((long long)(i == 1 ? num : 0 - num)) * ig;
        const D2 r = i == 0 || i == 1 ? q1 : D2{(float)i, 0.f} + q1, rr = r * r;
        const D2 b = rr + -(c * sq);
        B[k] = b;
        w = w + pk * rr;
        if (k != kref) {
            fb = fb + pk * b;
            sp = sp + pk;
        }
        sq = sq + pk * r * ig;
    }
    const D2 rest = c * (block_suffix(sq, ws[0]) + sq);
    if (kref >= k0 && kref < k1) tc.ref = B[kref] + rest;
    __syncthreads();
    const D2 shift_a = rest + -tc.ref;  // A - A of kref = B + shift_a
    if (kref >= k0 && kref < k1) B[kref] = -shift_a;  // (its difference: none, exactly)
    fb = fb + shift_a * sp;
    block_sum2(fb, w, ws[1]);
    if (threadIdx.x == 0) {
        tc.FA = fb * tc.norm;
        a.trace_misfit[2 * tr + comp] = to_f64(w) * tc.inv_S * a.dt * a.dt;
    }
    __syncthreads();
    const D2 FA = tc.FA, sc = tc.sc;
    for (int k = k0; k < k1; k++) {
        const D2 d = (B[k] + shift_a) + FA, x{U[k], 0.f};
        if (wide) {
            res[k] = (float)(to_f64(d) * tc.scale * (POWER ? inv_sigma * U[k] : U[k]) * inv_sigma);
        } else {
            const D2 v = d * sc * (POWER ? is * x : x) * is;
            res[k] = v.h + v.l;
        }
    }
}

// longest trace held in shared memory: four FP64 arrays of nt samples next to the
// static block-scan buffers within 227 KB, and at most OT_MAX_CHUNK samples a
// thread (k_ot, which needs 20 bytes a sample, keeps the same limit)
int ot_max_nt() {
    const int by_smem = (int)((227 * 1024 - (OT_THREADS + 32) * sizeof(double) - 1024) / (4 * sizeof(double)));
    return by_smem < OT_MAX_CHUNK * OT_THREADS ? by_smem : OT_MAX_CHUNK * OT_THREADS;
}

size_t ot_scratch_doubles(int nt, int ntr) { return nt > ot_max_nt() ? (size_t)5 * nt * 2 * ntr : 0; }

template <bool LONG, bool POWER>
static cudaError_t launch_ot_form(const OtArgs &a, cudaStream_t st) {
    // Runs of an odd number of samples, at most 512 threads.  3760 traces of 3000 samples
    // (both components): runs of 7, 9, 11, 13, 15 samples 660, 585, 590, 606, 650 us, each thread's share
    // of the block sums (about four samples' work) against the threads that hide
    // latency; 8000 of 300 samples: 5, 7, 9, 11 samples 192, 217, 241, 191 us, by the
    // warps' idle threads.  Few traces want many threads each (37 of 120 samples: 3
    // samples 57 us, 9 samples 65 us).
    const int least = (a.nt + 511) / 512 | 1;
    auto threads_of = [&](int r) { return ((a.nt + r - 1) / r + 31) & ~31; };
    int run = std::max(3, least);
    if (a.ntr >= 256)
        for (int r = run = std::max(5, least); r <= 11; r += 2)
            if (threads_of(r) * (r + 4) < threads_of(run) * (run + 4)) run = r;
    const int threads = threads_of(run);
    const size_t sm = LONG ? 0 : (size_t)a.nt * 20;
    if (!LONG) {
        cudaError_t e = cudaFuncSetAttribute(k_ot<LONG, POWER>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e != cudaSuccess) return e;
    }
    k_ot<LONG, POWER><<<2 * a.ntr, threads, sm, st>>>(a, run);
    return cudaGetLastError();
}
cudaError_t launch_ot(const OtArgs &a, cudaStream_t st) {
    if (a.nt > ot_max_nt()) {
        if (!a.scratch) return cudaErrorInvalidValue;
        k_ot_fp64<true><<<2 * a.ntr, OT_THREADS, 0, st>>>(a);
        return cudaGetLastError();
    }
    const size_t sm = (size_t)4 * a.nt * sizeof(double);
    cudaError_t e = cudaFuncSetAttribute(k_ot_fp64<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    k_ot_fp64<false><<<2 * a.ntr, OT_THREADS, sm, st>>>(a);
    return cudaGetLastError();
}
cudaError_t launch_ot_gather(const OtArgs &a, cudaStream_t st) {
    const bool power = a.kind == 2;
    if (a.nt > ot_max_nt()) {
        if (!a.scratch) return cudaErrorInvalidValue;
        return power ? launch_ot_form<true, true>(a, st) : launch_ot_form<true, false>(a, st);
    }
    return power ? launch_ot_form<false, true>(a, st) : launch_ot_form<false, false>(a, st);
}

// ---------------------------------------------------------------------------
// Allocation-free OT entry point (sfwi_ot_noalloc in include/sfwi_gb300.h).
//
// Its working memory -- the per-trace scale of the positivity transform, the
// per-trace misfits and their sum -- lives in the fixed array below instead
// of buffers from cudaMalloc.  It serves callers that cannot allocate device
// memory: a host program whose own allocator has reserved every device byte
// up front, and inner loops where a cudaMalloc/cudaFree may synchronise the
// device and stall other work in flight.
// Every device that loads this library holds the array (256 KB) until the
// process exits.  All calls on a device share it: a call holds the device's lock
// from its first launch until its work has ended, so calls from several
// threads, on whatever streams, take turns.
// ---------------------------------------------------------------------------
constexpr int OT_NOALLOC_MAX_TRACES = 8192;
// [0, 2*max): scale per (trace, component); [2*max, 4*max): misfit per
// (trace, component); [4*max]: the summed misfit
static __device__ __align__(256) double g_ot_noalloc_scratch[4 * OT_NOALLOC_MAX_TRACES + 32];

// scale of trace `blockIdx.x>>1`, component `blockIdx.x&1`: max |obs| (a
// maximum of floats is exact: FP64 comparisons took 137 us for 3760 traces of 3000
// samples, now 44 us)
__global__ void k_ot_trace_scale(const float *obs_z, const float *obs_x, int nt, double *sigma) {
    __shared__ float wm[32];
    const int tr = blockIdx.x >> 1, comp = blockIdx.x & 1;
    const float *o = (comp ? obs_x : obs_z) + (size_t)tr * nt;
    float m = 0.f;
#pragma unroll 4
    for (int k = threadIdx.x; k < nt; k += blockDim.x) m = fmaxf(m, fabsf(o[k]));
    m = warp_max(m);
    if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < (int)(blockDim.x >> 5); i++) m = fmaxf(m, wm[i]);
        sigma[blockIdx.x] = m;
    }
}

// gather-wide scale: every trace of a component takes the largest (kind 3),
// or its own floored at OT_SIGMA_FLOOR times the largest (kinds 1, 2)
__global__ void k_ot_gather_scale(double *sigma, int ntr, int all) {
    __shared__ double wsum[32];
    const int comp = blockIdx.x;
    double m = 0.0;
    for (int t = threadIdx.x; t < ntr; t += blockDim.x) m = fmax(m, sigma[2 * t + comp]);
    const double g = block_max(m, wsum);
    __syncthreads();
    for (int t = threadIdx.x; t < ntr; t += blockDim.x)
        sigma[2 * t + comp] = all ? g : fmax(sigma[2 * t + comp], OT_SIGMA_FLOOR * g);
}

// per-shot floor of the trace scales (kinds 1, 2) or the shot's largest
// scale for every trace (kind 3); block = (shot, component)
__global__ void k_ot_shot_scale(double *sigma, const ShotGeo *geo, int all) {
    __shared__ double wsum[32];
    const int s = blockIdx.x >> 1, comp = blockIdx.x & 1;
    const int t0 = geo[s].tr0, n = geo[s].ntr;
    double m = 0.0;
    for (int t = threadIdx.x; t < n; t += blockDim.x) m = fmax(m, sigma[2 * (t0 + t) + comp]);
    const double g = block_max(m, wsum);
    __syncthreads();
    for (int t = threadIdx.x; t < n; t += blockDim.x) {
        double &v = sigma[2 * (t0 + t) + comp];
        v = all ? g : fmax(v, OT_SIGMA_FLOOR * g);
    }
}

void launch_ot_scales(const float *obs_z, const float *obs_x, int nt, int ntr, const ShotGeo *geo, int nshots,
                      int all, double *sigma, cudaStream_t st) {
    if (ntr < 1) return;
    k_ot_trace_scale<<<2 * ntr, 256, 0, st>>>(obs_z, obs_x, nt, sigma);
    k_ot_shot_scale<<<2 * nshots, 256, 0, st>>>(sigma, geo, all);
}

// misfit = sum over traces of the two components: 1024 partial sums in trace order,
// then a fixed tree (one thread's chain of 7520 additions took 450 us, this 10 us)
__global__ void __launch_bounds__(1024) k_ot_sum(const double *trace_misfit, int ntr, double *out) {
    __shared__ double p[1024];
    double w = 0.0;
    for (int i = threadIdx.x; i < 2 * ntr; i += 1024) w += trace_misfit[i];
    p[threadIdx.x] = w;
    __syncthreads();
    for (int h = 512; h > 0; h >>= 1) {
        if (threadIdx.x < h) p[threadIdx.x] += p[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = p[0];
}

}  // namespace sfwi

namespace {
// Device address of g_ot_noalloc_scratch, looked up once per CUDA context with
// the device current: host code cannot take the address of a __device__
// array (its name there is a host-side stand-in), and a new context on the
// same device (after cudaDeviceReset) loads the module, and the array, anew.
// The context is identified by cuCtxGetId, which never repeats in a process;
// where the driver does not offer it, the address is kept per device.
struct ScratchAddr {
    unsigned long long ctx;
    double *addr;
};
std::mutex g_noalloc_mu;            // of the addresses
std::mutex g_noalloc_call[128];     // of each device's array
ScratchAddr g_noalloc_addr[128] = {};

unsigned long long current_context_id() {
    static PFN_cuCtxGetCurrent_v4000 get_cur = nullptr;
    static PFN_cuCtxGetId_v12000 get_id = nullptr;
    static bool looked = false;
    if (!looked) {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 4000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_cur = reinterpret_cast<PFN_cuCtxGetCurrent_v4000>(f);
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = reinterpret_cast<PFN_cuCtxGetId_v12000>(f);
        looked = true;
    }
    CUcontext c = nullptr;
    unsigned long long id = 0;
    if (get_cur && get_id && get_cur(&c) == CUDA_SUCCESS && c && get_id(c, &id) == CUDA_SUCCESS) return id + 1;
    return 0;  // unknown: one address per device
}
}  // namespace

extern "C" int sfwi_ot_noalloc(int kind, const float *obs_x, const float *obs_z, const float *cal_x,
                               const float *cal_z, float *res_x, float *res_z, int length, int tracenum, float dt,
                               double *misfit, void *stream) {
    using namespace sfwi;
    if (kind < 1 || kind > 3) return record_error(-1, "sfwi_ot_noalloc: kind must be 1, 2 or 3");
    if (!misfit || length < 1 || tracenum < 0) return record_error(-1, "sfwi_ot_noalloc: bad argument");
    // an empty gather (a shot without receivers) adds nothing, as sfwi_ot
    if (tracenum == 0) return 0;
    if (!obs_x || !obs_z || !cal_x || !cal_z || !res_x || !res_z)
        return record_error(-1, "sfwi_ot_noalloc: bad argument");
    if (tracenum > OT_NOALLOC_MAX_TRACES)
        return record_error(-1, "sfwi_ot_noalloc: %d traces exceed the fixed scratch of %d traces", tracenum,
                            OT_NOALLOC_MAX_TRACES);
    if (length > ot_max_nt())
        return record_error(-1, "sfwi_ot_noalloc: length %d exceeds %d samples", length, ot_max_nt());
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return record_error(-2, "sfwi_ot_noalloc: %s", cudaGetErrorString(e));
    if (dev < 0 || dev >= 128) return record_error(-1, "sfwi_ot_noalloc: device %d out of range", dev);
    double *scratch = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        unsigned long long ctx = current_context_id();
        if (ctx == 0) {
            // no context current yet: make the device's primary context
            // current (it allocates nothing) so that its id can be read
            if ((e = cudaSetDevice(dev)) != cudaSuccess)
                return record_error(-2, "sfwi_ot_noalloc: %s", cudaGetErrorString(e));
            ctx = current_context_id();
        }
        ScratchAddr &a = g_noalloc_addr[dev];
        if (!a.addr || a.ctx != ctx) {
            void *p = nullptr;
            e = cudaGetSymbolAddress(&p, g_ot_noalloc_scratch);
            if (e != cudaSuccess) return record_error(-2, "sfwi_ot_noalloc: scratch address: %s", cudaGetErrorString(e));
            a.addr = static_cast<double *>(p);
            a.ctx = ctx;
        }
        scratch = a.addr;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    double *sigma = scratch, *tmis = scratch + 2 * OT_NOALLOC_MAX_TRACES, *sum = scratch + 4 * OT_NOALLOC_MAX_TRACES;
    std::lock_guard<std::mutex> turn(g_noalloc_call[dev]);
    k_ot_trace_scale<<<2 * tracenum, 256, 0, st>>>(obs_z, obs_x, length, sigma);
    k_ot_gather_scale<<<2, 256, 0, st>>>(sigma, tracenum, kind == 3);
    OtArgs o{};
    o.kind = kind;
    o.nt = length;
    o.ntr = tracenum;
    o.stage = 1;
    o.dt = dt;
    o.obs_z = obs_z;
    o.obs_x = obs_x;
    o.cal_z = cal_z;
    o.cal_x = cal_x;
    o.res_z = res_z;
    o.res_x = res_x;
    o.sigma = sigma;
    o.trace_misfit = tmis;
    double w = 0.0;
    if ((e = launch_ot_gather(o, st)) == cudaSuccess) {
        k_ot_sum<<<1, 1024, 0, st>>>(tmis, tracenum, sum);
        e = cudaMemcpyAsync(&w, sum, sizeof(double), cudaMemcpyDeviceToHost, st);
    }
    const cudaError_t end = cudaStreamSynchronize(st);  // (also after an error: the array is the next call's)
    if (e == cudaSuccess) e = end;
    if (e != cudaSuccess) return record_error(-2, "sfwi_ot_noalloc: %s", cudaGetErrorString(e));
    *misfit += w;
    return 0;
}
