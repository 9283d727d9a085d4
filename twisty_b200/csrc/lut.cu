// lut.cu -- weight lookup tables, built on the device in FP64.
//
// The reference builds its table with an OpenMP loop over bins, each bin a composite
// Simpson quadrature of IntegrandRT whose terms are sorted then summed
// (Twisty/PathWeightUtils.cpp:281-433). Here one thread sweeps a bin over node weights that all bins
// share (the integrand factors into a bin-independent weight times sin(kds p); the derivatives
// with respect to mu_s and eps into three more weights times its sine and cosine). The
// compensated sums replace the sort (they are at least as accurate), so the float table
// matches the reference's to within one float ulp rather than bit for bit (the faithful table
// mode is built on host threads).
//
// The node set keeps the reference's rule exactly: weights h/3 * {1, 4, 2, ..., 4, 2, 1}
// with the odd loop ending at node n-3 and the even loop at n-4 (nodes n-2 and n-1 are
// dropped), and the config mu/eps swap of IntegrandRT's call (PathWeightUtils.cpp:401).
#include "kernels.h"
#include "device_common.cuh"

#include <cfloat>
#include <cooperative_groups.h>
#include <math_constants.h>

namespace twisty {
namespace {

// bins whose secant (fixed-point form) errs by more than this per segment are steep; a table
// with more than bins / kSteepFractionDev of them takes the exact blend
constexpr double kSecantBoundDev = 1e-7;
constexpr uint32_t kSteepFractionDev = 16;

struct Neumaier {
    double s = 0.0, c = 0.0;
    __device__ __forceinline__ void add(double x)
    {
        const double t = s + x;
        c += (fabs(s) >= fabs(x)) ? (s - t) + x : (x - t) + s;
        s = t;
    }
    __device__ __forceinline__ double value() const { return s + c; }
};

// The FP64 form factors: node j contributes w_j sin(kds p_j) / kds with
// w_j = c_j (h/3) p_j exp(bds phase(p_j) - reg^2 p_j^2 / 2) the same for every bin. A CTA
// of kFastThreads threads covers that many consecutive bins of one table: it stages w_j for a
// chunk of nodes in shared memory and each thread sweeps its bin over the chunk, stepping
// (sin, cos)(kds j h) by the rotation through kds h and restarting from sincos every kRun
// nodes, so the phase drift stays at the level of the direct argument's own rounding
// (kds j h carries a relative error of one ulp either way). Runs are summed plainly and
// folded into a Neumaier total; node n (p = maxBound exactly) is added with a direct sin;
// bin 0 (kds = 0) takes the limit sin(kds p)/kds -> p.
constexpr int kFastThreads = 128;
constexpr uint32_t kFastChunk = 1024;
constexpr uint32_t kRun = 64;

__device__ __forceinline__ void build_fast(const LutBuildSpec &s, uint32_t bin0, double *out64, double *sw)
{
    const uint32_t n = s.num_steps_int;
    const double m = (double)s.eps, reg = (double)s.mu;
    const double ds = (double)s.ds;
    const double bds = (double)s.scatter * ds;
    const double maxb = 10.0 / m;
    const double h = maxb / (double)n;
    const double weight = h / 3.0;
    const double np_d = sqrt((CUDART_PI * m) * 0.5) / (1.0 - exp(-2.0 / m));
    const uint32_t bin = bin0 + threadIdx.x;
    const double kds = (double)bin * s.step64 * ds;
    const bool zero_k = !(kds > 0.0);
    double st, ct;
    sincos(kds * h, &st, &ct);
    // Past p_cut the weight is exactly zero in FP64 (bds phase(p) <= bds np_d, so the exponent
    // is below -750 and exp underflows to 0): those nodes add nothing and are not visited.
    // With the regulariser of the usual configurations most of [0, 10/eps] lies there.
    uint32_t n_eff = n;
    if (reg > 0.0) {
        const double p_cut = sqrt(2.0 * (bds * np_d + 750.0)) / reg;
        const double j_cut = ceil(p_cut / h) + 2.0;
        if (j_cut < (double)n) n_eff = (uint32_t)j_cut;
    }
    Neumaier acc;
    for (uint32_t c0 = 0; c0 < n_eff; c0 += kFastChunk) {
        const uint32_t cn = min(kFastChunk, n_eff - c0);
        __syncthreads();   // the previous chunk is consumed
        for (uint32_t i = threadIdx.x; i < cn; i += blockDim.x) {
            const uint32_t j = c0 + i;
            const double c = (j == 0) ? 1.0 : (j >= n - 2) ? 0.0 : ((j & 1u) ? 4.0 : 2.0);
            const double p = (double)j * h;
            const double ph = np_d * exp(-m * p * p * 0.5);
            sw[i] = (p * exp(bds * ph - reg * reg * p * p * 0.5)) * weight * c;
        }
        __syncthreads();
        if (zero_k) {
            double run = 0.0;
            for (uint32_t i = 0; i < cn; ++i) run = fma(sw[i], (double)(c0 + i) * h, run);
            acc.add(run);
        } else {
            for (uint32_t r0 = 0; r0 < cn; r0 += kRun) {
                double sn, cs;
                sincos(kds * ((double)(c0 + r0) * h), &sn, &cs);
                const uint32_t rn = min(kRun, cn - r0);
                double run = 0.0;
#pragma unroll 8
                for (uint32_t i = 0; i < rn; ++i) {
                    run = fma(sw[r0 + i], sn, run);
                    const double t = fma(sn, ct, cs * st);
                    cs = fma(cs, ct, -(sn * st));
                    sn = t;
                }
                acc.add(run);
            }
        }
    }
    const double ph = np_d * exp(-m * maxb * maxb * 0.5);
    const double wn = (maxb * exp(bds * ph - reg * reg * maxb * maxb * 0.5)) * weight;
    acc.add(zero_k ? wn * maxb : wn * sin(kds * maxb));
    if (bin < s.bins) {
        const double total = zero_k ? acc.value() : acc.value() / kds;
        out64[bin] = (total / (2.0 * CUDART_PI * CUDART_PI)) * (double)s.bias;
    }
}

__global__ void __launch_bounds__(kFastThreads) lut_build_fast_kernel(LutBuildSpec s, double *out64)
{
    __shared__ double sw[kFastChunk];
    build_fast(s, blockIdx.x * kFastThreads, out64, sw);
}

// Tables of many experiments (FP64 form, no derivatives): blockIdx.y selects the
// experiment, its table at out64 + y*bins.
__global__ void __launch_bounds__(kFastThreads) lut_build_batch_kernel(const LutBuildSpec *__restrict__ specs,
                                                                        uint32_t bins, double *out64)
{
    __shared__ double sw[kFastChunk];
    const LutBuildSpec s = specs[blockIdx.y];
    build_fast(s, blockIdx.x * kFastThreads, out64 + (size_t)blockIdx.y * bins, sw);
}

// Derivative tables of the adjoint, dL/dmu_s and dL/deps, from the same quadrature differentiated under
// the integral (the nodes move with maxBound = 10/eps). With e = exp(bds phase(p) - reg^2 p^2 / 2),
// s = sin(kds p)/kds and g = bds phase'(p) - reg^2 p, node j adds c_j times
//   w1 s,  w1 = p e                                   to the integral I,
//   w1 phase s                                        to dI/dbds,
//   w2 s + w3 cos(kds p),  w2 = p e (bds dphase/deps - (1 + p g)/eps),  w3 = -p^2 e/eps   to dI/deps + I/eps.
// A thread sweeps one bin, as build_fast does (the first form integrated each bin by a CTA with two
// exponentials and a sincos per node: 0.13-0.24 ms per 4096-bin table, one launch each).
// Out: per bin, one float4 of both tables. ratio 0: (dmu_i, dmu_{i+1} - dmu_i, deps_i, deps_{i+1} - deps_i), the form
// of the linear table. ratio 1: (dmu/L, deps/L) at the bin's left end and their change across the
// bin, the derivatives of ln L of the blend as chords over the bin. A chord is off the quotient of the
// blends by up to |step a| / 4 of the quotient's own change across the bin (to a factor near 1), a = L_{i+1}/L_i - 1; with
// no steep bin |step a| < 1.4e-3, so by 3.4e-4 of that change. In 64 bits (N = 20 to 600, 1024 and 4096 bins, sigma 0.08 to 0.2):
// a quarter of |step a| <= 2.4e-4 of the change, 1e-14 to 3e-8 of the table's largest entry, at or below a float's rounding.
constexpr int kDerivBins = kFastThreads - 1;   // the last thread of a CTA only serves as a neighbour
constexpr uint32_t kDerivChunk = 512;

__global__ void __launch_bounds__(kFastThreads)
deriv_tables_kernel(const LutBuildSpec *__restrict__ specs, const DerivJob *__restrict__ jobs, uint32_t bins)
{
    __shared__ double w1[kDerivChunk], w1p[kDerivChunk], w2[kDerivChunk], w3[kDerivChunk];
    __shared__ double s_mu[kFastThreads], s_eps[kFastThreads];
    const DerivJob job = jobs[blockIdx.y];
    const LutBuildSpec s = specs[job.spec];
    const uint32_t n = s.num_steps_int;
    const double m = (double)s.eps, reg = (double)s.mu, ds = (double)s.ds, bds = (double)s.scatter * ds;
    const double maxb = 10.0 / m, h = maxb / (double)n;
    const double em = exp(-2.0 / m);
    const double np_d = sqrt((CUDART_PI * m) * 0.5) / (1.0 - em);
    const double dlnnp = 0.5 / m - (2.0 / (m * m)) * em / (1.0 - em);
    auto node = [&](double p, double c, double &a1, double &a1p, double &a2, double &a3) {
        const double ph = np_d * exp(-m * p * p * 0.5);
        const double e = c * exp(bds * ph - reg * reg * p * p * 0.5);
        const double g = -bds * m * p * ph - reg * reg * p;
        a1 = p * e;
        a1p = a1 * ph;
        a2 = a1 * (bds * ph * (dlnnp - 0.5 * p * p) - (1.0 + p * g) / m);
        a3 = -p * p * e / m;
    };
    const uint32_t bin = blockIdx.x * kDerivBins + threadIdx.x;
    const double kds = (double)bin * s.step64 * ds;
    const bool zero_k = !(kds > 0.0);
    double st, ct;
    sincos(kds * h, &st, &ct);
    uint32_t n_eff = n;   // past p_cut every weight is zero (build_fast)
    if (reg > 0.0) {
        const double j_cut = ceil(sqrt(2.0 * (bds * np_d + 750.0)) / reg / h) + 2.0;
        if (j_cut < (double)n) n_eff = (uint32_t)j_cut;
    }
    Neumaier t1, tmu, teps;
    for (uint32_t c0 = 0; c0 < n_eff; c0 += kDerivChunk) {
        const uint32_t cn = min(kDerivChunk, n_eff - c0);
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < cn; i += blockDim.x) {
            const uint32_t j = c0 + i;
            const double c = (j == 0) ? 1.0 : (j >= n - 2) ? 0.0 : ((j & 1u) ? 4.0 : 2.0);
            node((double)j * h, c, w1[i], w1p[i], w2[i], w3[i]);
        }
        __syncthreads();
        for (uint32_t r0 = 0; r0 < cn; r0 += kRun) {
            double sn, cs;
            sincos(kds * ((double)(c0 + r0) * h), &sn, &cs);
            const uint32_t rn = min(kRun, cn - r0);
            double r1 = 0.0, rmu = 0.0, r2 = 0.0, r3 = 0.0;
#pragma unroll 4
            for (uint32_t i = r0; i < r0 + rn; ++i) {
                const double q = zero_k ? (double)(c0 + i) * h : sn;   // sin(kds p)/kds -> p
                r1 = fma(w1[i], q, r1);
                rmu = fma(w1p[i], q, rmu);
                r2 = fma(w2[i], q, r2);
                r3 = fma(w3[i], cs, r3);
                const double t = fma(sn, ct, cs * st);
                cs = fma(cs, ct, -(sn * st));
                sn = t;
            }
            const double k = zero_k ? 1.0 : kds;
            t1.add(r1 / k);
            tmu.add(rmu / k);
            teps.add(r2 / k);
            teps.add(r3);
        }
    }
    {
        double a1, a1p, a2, a3, sn, cs;
        node(maxb, 1.0, a1, a1p, a2, a3);
        sincos(kds * maxb, &sn, &cs);
        const double q = zero_k ? maxb : sn / kds;
        t1.add(a1 * q);
        tmu.add(a1p * q);
        teps.add(a2 * q);
        teps.add(a3 * cs);
    }
    const double scale = h / 3.0 / (2.0 * CUDART_PI * CUDART_PI) * (double)s.bias;
    s_mu[threadIdx.x] = tmu.value() * scale * ds;   // bds = mu_s ds
    s_eps[threadIdx.x] = -(t1.value() * scale) / m + teps.value() * scale;
    __syncthreads();
    if (bin >= bins || threadIdx.x == kFastThreads - 1) return;
    const int right = bin + 1 < bins ? threadIdx.x + 1 : threadIdx.x;
    const double mu0 = s_mu[threadIdx.x], mu1 = s_mu[right], e0 = s_eps[threadIdx.x], e1 = s_eps[right];
    float4 o;
    if (job.ratio) {
        const double L0 = (double)job.lut[bin], L1 = (double)job.lut[bin + 1 < bins ? bin + 1 : bin], x = (double)s.step;
        const double end = L0 + x * (L1 - L0);
        const double am = mu0 / L0, ae = e0 / L0;
        o = make_float4((float)am, (float)ae, (float)((mu0 + x * (mu1 - mu0)) / end - am), (float)((e0 + x * (e1 - e0)) / end - ae));
    } else {
        o = make_float4((float)mu0, (float)mu1 - (float)mu0, (float)e0, (float)e1 - (float)e0);
    }
    job.out[bin] = o;
}

// Replace non-positive entries by the smallest non-negative one and emit the float copy
// (WeightLookupTableIntegral::Initialize, PathWeightUtils.cpp:305-347). One CTA per table:
// blockIdx.x selects table x of a batch (lut + x*bins, out32 + x*bins, minmax + 3x).
__global__ void __launch_bounds__(1024) lut_finalize_kernel(uint32_t bins, double *lut, float *out32,
                                                            double *minmax)
{
    lut += (size_t)blockIdx.x * bins;
    if (out32) out32 += (size_t)blockIdx.x * bins;
    if (minmax) minmax += 3 * (size_t)blockIdx.x;
    __shared__ double smin[32], smax[32];
    __shared__ int sarg[32];
    // The reference keeps entries in float, so min/max selection runs on the float values.
    double mn = (double)(float)lut[0], mx = mn;
    int arg = 0;
    for (uint32_t i = 1 + threadIdx.x; i < bins; i += blockDim.x) {
        const double v = (double)(float)lut[i];
        if (v < mn && v >= 0.0) { mn = v; arg = (int)i; }
        if (v > mx && v >= 0.0) mx = v;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const double omn = __shfl_xor_sync(0xffffffffu, mn, o);
        const int oarg = __shfl_xor_sync(0xffffffffu, arg, o);
        if (omn < mn || (omn == mn && oarg < arg)) { mn = omn; arg = oarg; }
        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) { smin[w] = mn; smax[w] = mx; sarg[w] = arg; }
    __syncthreads();
    if (w == 0) {
        const int nw = blockDim.x >> 5;
        mn = l < nw ? smin[l] : DBL_MAX;
        mx = l < nw ? smax[l] : -DBL_MAX;
        arg = l < nw ? sarg[l] : 0;
        for (int o = 16; o > 0; o >>= 1) {
            const double omn = __shfl_xor_sync(0xffffffffu, mn, o);
            const int oarg = __shfl_xor_sync(0xffffffffu, arg, o);
            if (omn < mn || (omn == mn && oarg < arg)) { mn = omn; arg = oarg; }
            mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        }
        if (l == 0) { smin[0] = mn; smax[0] = mx; sarg[0] = arg; }
    }
    __syncthreads();
    mn = smin[0];
    const double mn64 = lut[sarg[0]];
    for (uint32_t i = threadIdx.x; i < bins; i += blockDim.x) {
        double v = lut[i];
        if ((float)v <= 0.0f) v = mn64;
        lut[i] = v;
        if (out32) out32[i] = (float)v;
    }
    if (threadIdx.x == 0 && minmax) {
        minmax[0] = mn;
        minmax[1] = smax[0];
        minmax[2] = (double)sarg[0];
    }
}

// Compensated-form tables of one experiment per CTA: lin = (L_i, L_{i+1} - L_i); fix = (round((log10 L_i - c0)
// 2^s) as uint32, log10(1 + step (L_{i+1}/L_i - 1))) with c0 = min log10 L - 64 2^-s and the
// largest s <= 30 keeping (N+1) (range 2^s + 65) below 2^31, else the wide form with
// 32 (range 2^s + 65) below 2^32. Bins whose secant error exceeds 1e-7 per segment are
// steep: slope NaN (paths crossing them are re-weighed through lin), counted in lf[x].steep.
// ok[x] = 1 when the fixed form is usable: every entry positive, at most bins/16 steep bins,
// s >= 22.
__global__ void __launch_bounds__(1024) comp_tables_kernel(uint32_t bins, const float *__restrict__ lut32,
                                                           const float *__restrict__ steps,
                                                           const uint32_t *__restrict__ nsegs, float2 *fix,
                                                           float2 *lin, LogFixed *lf, int *ok)
{
    __shared__ double s_lo[32], s_hi[32], s_err[32];
    __shared__ int s_bad[32], s_steep[32];
    const uint32_t x = blockIdx.x;
    const float *L = lut32 + (size_t)x * bins;
    fix += (size_t)x * table_pitch(bins);
    lin += (size_t)x * table_pitch(bins);
    const double st = (double)steps[x];
    double lo = DBL_MAX, hi = -DBL_MAX, err = 0.0;
    int bad = 0, steep = 0;
    for (uint32_t i = threadIdx.x; i < bins; i += blockDim.x) {
        const float a = L[i], b = L[i + 1 < bins ? i + 1 : i];
        lin[i] = make_float2(a, b - a);
        if (!(a > 0.0f) || !isfinite(a)) {
            bad = 1;
            continue;
        }
        const double lg = log10((double)a);
        lo = fmin(lo, lg);
        hi = fmax(hi, lg);
        if (i + 1 < bins) {
            const double r = (double)b / (double)a - 1.0;
            const double e = (st * r) * (st * r) / (8.0 * 2.302585092994046);
            if (e > kSecantBoundDev) ++steep;
            else err = fmax(err, e);
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        err = fmax(err, __shfl_xor_sync(0xffffffffu, err, o));
        bad |= __shfl_xor_sync(0xffffffffu, bad, o);
        steep += __shfl_xor_sync(0xffffffffu, steep, o);
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    if (l == 0) { s_lo[w] = lo; s_hi[w] = hi; s_err[w] = err; s_bad[w] = bad; s_steep[w] = steep; }
    __syncthreads();
    if (w == 0) {
        lo = l < nw ? s_lo[l] : DBL_MAX;
        hi = l < nw ? s_hi[l] : -DBL_MAX;
        err = l < nw ? s_err[l] : 0.0;
        bad = l < nw ? s_bad[l] : 0;
        steep = l < nw ? s_steep[l] : 0;
        for (int o = 16; o > 0; o >>= 1) {
            lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
            err = fmax(err, __shfl_xor_sync(0xffffffffu, err, o));
            bad |= __shfl_xor_sync(0xffffffffu, bad, o);
            steep += __shfl_xor_sync(0xffffffffu, steep, o);
        }
        if (l == 0) { s_lo[0] = lo; s_hi[0] = hi; s_err[0] = err; s_bad[0] = bad; s_steep[0] = steep; }
    }
    __syncthreads();
    lo = s_lo[0];
    hi = s_hi[0];
    err = s_err[0];
    bad = s_bad[0];
    steep = s_steep[0];
    double cap = floor(2147483647.0 / (double)(nsegs[x] + 1));
    int s = 30;
    while (s > 0 && (hi - lo) * ldexp(1.0, s) + 65.0 > cap) --s;
    int wide = 0;
    if (s < 22) {
        wide = 1;
        cap = floor(4294967295.0 / 32.0);
        s = 30;
        while (s > 0 && (hi - lo) * ldexp(1.0, s) + 65.0 > cap) --s;
    }
    const bool usable = !bad && (uint32_t)steep <= bins / kSteepFractionDev && s >= 22;
    const double inv_scale = ldexp(1.0, -s);
    if (threadIdx.x == 0) {
        lf[x] = usable ? LogFixed{lo - 64.0 * inv_scale, inv_scale, wide, steep} : LogFixed{0.0, 0.0, 0, steep};
        ok[x] = usable ? 1 : 0;
    }
    if (!usable) return;
    for (uint32_t i = threadIdx.x; i < bins; i += blockDim.x) {
        const double e = 64.0 + rint((log10((double)L[i]) - lo) * ldexp(1.0, s));
        const uint32_t u = (uint32_t)fmin(e, cap - 1.0);
        float delta = 0.0f;
        if (i + 1 < bins) {
            const double r = (double)L[i + 1] / (double)L[i] - 1.0;
            delta = ((st * r) * (st * r) / (8.0 * 2.302585092994046) > kSecantBoundDev) ? __int_as_float(0x7fffffff)
                                                                                       : (float)log10(1.0 + st * r);
        }
        fix[i] = make_float2(__uint_as_float(u), delta);
    }
}

// One table's finalisation and compensated forms in one launch of a cluster: the rules of
// lut_finalize_kernel (when `finalize`; else lut32 is the table) and of comp_tables_kernel, with
// the bins spread over kTabCtas SMs -- three FP64 logs a bin are 20 us on one SM at 8192 bins -- and the
// minima, maxima and counts combined through the cluster's shared memory. A single run used to
// read its table back, take the logs on the host and upload both forms: 0.15 ms at 4096 bins,
// 0.5 ms at 20000.
constexpr int kTabCtas = 8;

struct TabStats {
    double mn, mx, lo, hi, err;
    int arg, bad, steep, nonfinite;
    __device__ __forceinline__ void take(const TabStats &o)
    {
        if (o.mn < mn || (o.mn == mn && o.arg < arg)) { mn = o.mn; arg = o.arg; }
        mx = fmax(mx, o.mx);
        lo = fmin(lo, o.lo);
        hi = fmax(hi, o.hi);
        err = fmax(err, o.err);
        bad |= o.bad;
        steep += o.steep;
        nonfinite |= o.nonfinite;
    }
    __device__ __forceinline__ TabStats shuffled(int off) const
    {
        constexpr uint32_t F = 0xffffffffu;
        return TabStats{__shfl_xor_sync(F, mn, off), __shfl_xor_sync(F, mx, off), __shfl_xor_sync(F, lo, off), __shfl_xor_sync(F, hi, off),
                        __shfl_xor_sync(F, err, off), __shfl_xor_sync(F, arg, off), __shfl_xor_sync(F, bad, off),
                        __shfl_xor_sync(F, steep, off), __shfl_xor_sync(F, nonfinite, off)};
    }
};

// Combines the threads' statistics over the cluster (in every thread). s_cta: this CTA's part, `s_warp` scratch.
__device__ TabStats cluster_stats(TabStats t, const TabStats &none, TabStats *s_warp, TabStats *s_cta)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    for (int o = 16; o > 0; o >>= 1) t.take(t.shuffled(o));
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) s_warp[w] = t;
    __syncthreads();
    if (w == 0) {
        t = l < (int)(blockDim.x >> 5) ? s_warp[l] : none;
        for (int o = 16; o > 0; o >>= 1) t.take(t.shuffled(o));
        if (l == 0) *s_cta = t;
    }
    cl.sync();
    t = *cl.map_shared_rank(s_cta, 0);
    for (int r = 1; r < kTabCtas; ++r) t.take(*cl.map_shared_rank(s_cta, r));
    return t;
}

__global__ void __cluster_dims__(kTabCtas, 1, 1) __launch_bounds__(1024)
single_tables_kernel(uint32_t bins, float step, uint32_t n_segments, int finalize, double *lut64, float *lut32, float2 *lin, float2 *fix,
                     TableInfo *info)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    __shared__ TabStats s_warp[32], s_first, s_second;
    const uint32_t t0 = cl.block_rank() * blockDim.x + threadIdx.x, tn = kTabCtas * blockDim.x;
    const double first = finalize ? (double)(float)lut64[0] : 0.0;
    const TabStats none{first, first, DBL_MAX, -DBL_MAX, 0.0, 0, 0, 0, 0};
    TabStats a = none;
    if (finalize) {
        // min/max selection on the float values, as the reference keeps them; the first entry counts whatever its sign
        for (uint32_t i = t0; i < bins; i += tn) {
            const double v = (double)(float)lut64[i];
            if (i > 0 && v < a.mn && v >= 0.0) { a.mn = v; a.arg = (int)i; }
            if (i > 0 && v > a.mx && v >= 0.0) a.mx = v;
        }
        a = cluster_stats(a, none, s_warp, &s_first);
        const double mn64 = lut64[a.arg];
        cl.sync();   // every CTA has the replacement before any writes
        for (uint32_t i = t0; i < bins; i += tn) {
            double v = lut64[i];
            if ((float)v <= 0.0f) v = mn64;
            lut64[i] = v;
            lut32[i] = (float)v;
        }
        cl.sync();   // a bin's right neighbour may be another CTA's
    }
    const double st = (double)step;
    auto steepness = [&](float x, float y, double &r) {
        r = (double)y / (double)x - 1.0;
        return (st * r) * (st * r) / (8.0 * 2.302585092994046);
    };
    TabStats b = none;
    for (uint32_t i = t0; i < bins; i += tn) {
        const float x = lut32[i], y = lut32[i + 1 < bins ? i + 1 : i];
        lin[i] = make_float2(x, y - x);
        if (!isfinite(x)) b.nonfinite = 1;
        if (!(x > 0.0f) || !isfinite(x)) {
            b.bad = 1;
            continue;
        }
        const double lg = log10((double)x);
        b.lo = fmin(b.lo, lg);
        b.hi = fmax(b.hi, lg);
        if (i + 1 < bins) {
            double r;
            const double e = steepness(x, y, r);
            if (e > kSecantBoundDev) ++b.steep;
            else b.err = fmax(b.err, e);
        }
    }
    b = cluster_stats(b, none, s_warp, &s_second);
    double cap = floor(2147483647.0 / (double)(n_segments + 1));
    int s = 30;
    while (s > 0 && (b.hi - b.lo) * ldexp(1.0, s) + 65.0 > cap) --s;
    int wide = 0;
    if (s < 22) {
        wide = 1;
        cap = floor(4294967295.0 / 32.0);
        s = 30;
        while (s > 0 && (b.hi - b.lo) * ldexp(1.0, s) + 65.0 > cap) --s;
    }
    const bool usable = !b.bad && (uint32_t)b.steep <= bins / kSteepFractionDev && s >= 22;
    const double inv_scale = ldexp(1.0, -s);
    if (t0 == 0)
        *info = TableInfo{a.mn, a.mx, usable ? b.lo - 64.0 * inv_scale : 0.0, usable ? inv_scale : 0.0, b.bad ? INFINITY : b.err,
                          usable ? wide : 0, b.steep, usable ? 1 : 0, b.nonfinite};
    if (usable)
        for (uint32_t i = t0; i < bins; i += tn) {
            const float x = lut32[i];
            const double e = 64.0 + rint((log10((double)x) - b.lo) * ldexp(1.0, s));
            float delta = 0.0f;
            if (i + 1 < bins) {
                double r;
                delta = steepness(x, lut32[i + 1], r) > kSecantBoundDev ? __int_as_float(0x7fffffff) : (float)log10(1.0 + st * r);
            }
            fix[i] = make_float2(__uint_as_float((uint32_t)fmin(e, cap - 1.0)), delta);
        }
    cl.sync();   // the CTAs' shared memory stays until everyone has read it
}

}  // namespace

cudaError_t launch_single_tables(uint32_t bins, float step, uint32_t n_segments, int finalize, double *lut64, float *lut32, float2 *lin,
                                 float2 *fix, TableInfo *info, cudaStream_t st)
{
    single_tables_kernel<<<kTabCtas, 1024, 0, st>>>(bins, step, n_segments, finalize, lut64, lut32, lin, fix, info);
    return cudaGetLastError();
}

cudaError_t launch_lut_build_batch(const LutBuildSpec *d_specs, uint32_t n, uint32_t bins, double *out64,
                                   cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    if (bins < 2 || n > 65535u) return cudaErrorInvalidValue;
    lut_build_batch_kernel<<<dim3((bins + kFastThreads - 1) / kFastThreads, n), kFastThreads, 0, st>>>(d_specs, bins,
                                                                                                      out64);
    return cudaGetLastError();
}

cudaError_t launch_lut_finalize_batch(uint32_t n, uint32_t bins, double *lut64, float *out32, double *minmax,
                                      cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    lut_finalize_kernel<<<n, 1024, 0, st>>>(bins, lut64, out32, minmax);
    return cudaGetLastError();
}

cudaError_t launch_comp_tables_batch(uint32_t n, uint32_t bins, const float *lut32, const float *steps,
                                     const uint32_t *nsegs, float2 *fix, float2 *lin, LogFixed *lf, int *ok,
                                     cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    comp_tables_kernel<<<n, 1024, 0, st>>>(bins, lut32, steps, nsegs, fix, lin, lf, ok);
    return cudaGetLastError();
}

cudaError_t launch_lut_build(const LutBuildSpec &s, double *out64, cudaStream_t st)
{
    if (s.bins < 2 || s.num_steps_int < 4 || (s.num_steps_int & 1u)) return cudaErrorInvalidValue;
    lut_build_fast_kernel<<<(s.bins + kFastThreads - 1) / kFastThreads, kFastThreads, 0, st>>>(s, out64);
    return cudaGetLastError();
}

cudaError_t launch_deriv_tables(const LutBuildSpec *d_specs, const DerivJob *d_jobs, uint32_t n, uint32_t bins, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    if (n > 65535u) return cudaErrorInvalidValue;
    deriv_tables_kernel<<<dim3((bins + kDerivBins - 1) / kDerivBins, n), kFastThreads, 0, st>>>(d_specs, d_jobs, bins);
    return cudaGetLastError();
}

}  // namespace twisty
