// chain_plain.cu -- the plain FP32 drop-in form, the FP64 yardstick form, the FP64 global
// reduction over chains, and the reference-semantics weigher of given paths.
//
// Plain form: the arithmetic of the reference's GPU kernel
// (Twisty/FullExperimentRunnerOptimalPerturbOptimized_GPU.cu:689-918) -- positions rotated,
// every tangent and curvature recomputed each step, the float table blended, FP64 log weights and
// CombinedWeightValues_C accumulators -- with Philox in place of cuRAND and the reference CPU
// runner's proposal ranges (Twisty/FullExperimentRunnerOptimalPerturb.cpp:483-519). All FP32
// arithmetic is spelled with round-to-nearest intrinsics in the reference's operation order, so
// every position, tangent, curvature, bin and blend here is bit-identical to the same chain run
// by the CPU oracle; only the FP64 sums over segments and paths associate differently.
#include "kernels.h"

#include <algorithm>
#include "device_common.cuh"

#include <cfloat>
#include <cooperative_groups.h>

namespace twisty {
namespace {

using dev::CombinedWeight;

constexpr int kPlainThreads = 128;

// log10 weight of the path at x (planes of stride n_segments + 1), segment by segment in the
// reference's order and stopping where it stops: for the paths with a segment weight that is not a
// positive normal number (NaN curvatures, zero or negative table entries), which are rare.
__device__ __noinline__ bool plain_path_in_order(const float *x, const ChainSpec &c, const float *__restrict__ lut,
                                                 const dev::LutMeta &m, double &running, uint32_t &clamped)
{
    const uint32_t N = c.n_segments;
    const float *y = x + (N + 1), *z = y + (N + 1);
    float px = 0.f, py = 0.f, pz = 0.f;
    running = 0.0;
    for (uint32_t i = 0; i < N; ++i) {
        float vx = __fsub_rn(x[i + 1], x[i]), vy = __fsub_rn(y[i + 1], y[i]), vz = __fsub_rn(z[i + 1], z[i]);
        if (c.has_eval_shift && i == N - 2) {
            vx = __fadd_rn(vx, c.eval_shift[0]);
            vy = __fadd_rn(vy, c.eval_shift[1]);
            vz = __fadd_rn(vz, c.eval_shift[2]);
        }
        const float r = dev::rinvnorm(vx, vy, vz);
        const float tx = __fmul_rn(vx, r), ty = __fmul_rn(vy, r), tz = __fmul_rn(vz, r);
        if (i > 0) {
            const float kappa = __fsqrt_rn(dev::rdot3(__fmul_rn(__fsub_rn(tx, px), c.inv_ds), __fmul_rn(__fsub_rn(ty, py), c.inv_ds),
                                                      __fmul_rn(__fsub_rn(tz, pz), c.inv_ds)));
            double blend;
            if (dev::rbin_blend(kappa, lut, m, blend, clamped) < 0) return false;
            const double lg = log10(blend * c.absorption_factor);
            if (isnan(lg)) return false;
            running += lg;
        }
        px = tx; py = ty; pz = tz;
    }
    return !isnan(running);
}

// G lanes run one chain, its positions in shared memory as three planes (in `state` in global
// memory for chains too long for that, SMEM false, G = 32). Lane j takes the points and segments
// j, j + G, ... of a rotation and of the recompute, so neighbouring lanes read neighbouring points;
// the previous segment's tangent comes from the lane before by shuffle.
//  * The path weight is the product of the segment weights: each lane multiplies its
//    segments' mantissas and adds their exponents, the group combines them, and one FP64 log10 per path
//    replaces one per segment (a product of n FP64 factors errs by n 2^-53 relative, less than a sum of n logs).
//  * Lane j finishes the paths of steps j mod G: the log10 and the accumulator's power of ten
//    run once per G paths in each lane, not once per path in all of them.
// The first form of this kernel, one thread per chain with its state in global memory, was bound by
// its strided state traffic and the log10 per segment: the whole experiment of N = 64, 2^20 paths on
// 16384 chains took 7.20 ms, and takes 0.91 ms with this one.
template <int G, bool SMEM>
__global__ void __launch_bounds__(kPlainThreads, 1024 / kPlainThreads)
plain_chain_kernel(ChainSpec c, const float *__restrict__ init_pos, float *__restrict__ state, uint32_t stride,
                   const float *__restrict__ lut, LutMetaF mf, ChainOut *__restrict__ out, float *__restrict__ exp_pos,
                   double *__restrict__ exp_w)
{
    extern __shared__ float plain_smem[];
    const uint32_t j = threadIdx.x % G, slot = threadIdx.x / G;
    const uint32_t chain = blockIdx.x * (kPlainThreads / G) + slot;
    const bool real = chain < c.n_chains;
    if (!SMEM && !real) return;   // a whole warp
    const uint32_t N = c.n_segments;
    float *x = SMEM ? plain_smem + (size_t)slot * stride : state + (size_t)chain * stride;
    float *y = x + (N + 1), *z = y + (N + 1);
    for (uint32_t i = j; i <= N; i += G) {
        x[i] = init_pos[3 * i];
        y[i] = init_pos[3 * i + 1];
        z[i] = init_pos[3 * i + 2];
    }
    const dev::LutMeta m{mf.min_k, mf.max_k, mf.step, mf.bins};
    const uint32_t gmask = G == 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u) << ((threadIdx.x & 31u) / G * G);
    __syncwarp();

    // this lane's paths: the steps j mod G
    CombinedWeight cw;
    dev::cw_reset(cw);
    uint32_t valid = 0, failed = 0, clamped = 0;
    bool poisoned = false;
    enum : uint32_t { kNone, kProduct, kSum, kFailed, kZeroFirst, kZero };
    uint32_t kept = kNone;
    double kept_w = 0.0;      // kProduct: the mantissas' product, else log10 of the weight
    int kept_e = 0;
    bool met = false;         // the chain has met a valid path

    const uint32_t steps = !real ? 0 : (chain == c.n_chains - 1) ? c.last_steps : c.steps;
    const uint32_t total = c.burn_in + c.steps;
    for (uint32_t base = 0; base < total; base += G) {
        const dev::Proposal pr = dev::draw_step(c.seed, c.experiment, c.chain0 + chain, base + j, N, c.k_eff, c.max_angle);
        float psn, pcs;
        dev::sincos_half(pr.angle, psn, pcs);
        const uint32_t nstep = min((uint32_t)G, total - base);
        for (uint32_t jj = 0; jj < nstep; ++jj) {
            const uint32_t left = __shfl_sync(0xffffffffu, pr.left, jj, G);
            const uint32_t right = left + __shfl_sync(0xffffffffu, pr.k, jj, G);
            const float sn = __shfl_sync(0xffffffffu, psn, jj, G), cs = __shfl_sync(0xffffffffu, pcs, jj, G);
            const float lx = x[left], ly = y[left], lz = z[left];
            const float dx = __fsub_rn(x[right], lx), dy = __fsub_rn(y[right], ly), dz = __fsub_rn(z[right], lz);
            const float inv = dev::rinvnorm(dx, dy, dz);
            const float ax = __fmul_rn(dx, inv), ay = __fmul_rn(dy, inv), az = __fmul_rn(dz, inv);
            const float q[4] = {cs, __fmul_rn(ax, sn), __fmul_rn(ay, sn), __fmul_rn(az, sn)};
            for (uint32_t i = left + 1 + j; i < right; i += G) {
                float vx = __fsub_rn(x[i], lx), vy = __fsub_rn(y[i], ly), vz = __fsub_rn(z[i], lz);
                dev::rrotate(q, vx, vy, vz);
                x[i] = __fadd_rn(vx, lx);
                y[i] = __fadd_rn(vy, ly);
                z[i] = __fadd_rn(vz, lz);
            }
            __syncwarp();
            if (base + jj < c.burn_in) continue;
            const uint32_t wstep = base + jj - c.burn_in;
            const bool active = wstep < steps;

            double prod = 1.0;
            int esum = 0;
            bool odd = false;
            uint32_t cl = 0;
            float ptx = 0.f, pty = 0.f, ptz = 0.f;   // the tangent of this lane's previous round
            for (uint32_t r = 0; r * G < N; ++r) {
                const uint32_t i = r * G + j;
                const uint32_t at = min(i, N - 1);
                // UpdateTangentsFromPos (CurvePerturbUtils.cpp:147-154)
                float vx = __fsub_rn(x[at + 1], x[at]), vy = __fsub_rn(y[at + 1], y[at]), vz = __fsub_rn(z[at + 1], z[at]);
                if (c.has_eval_shift && at == N - 2) {
                    vx = __fadd_rn(vx, c.eval_shift[0]);
                    vy = __fadd_rn(vy, c.eval_shift[1]);
                    vz = __fadd_rn(vz, c.eval_shift[2]);
                }
                const float rn = dev::rinvnorm(vx, vy, vz);
                const float tx = __fmul_rn(vx, rn), ty = __fmul_rn(vy, rn), tz = __fmul_rn(vz, rn);
                // tangent i-1: of the lane before, of the last lane's previous round for lane 0
                const bool last = j == G - 1;
                const float bx = __shfl_sync(0xffffffffu, last ? ptx : tx, j + G - 1, G);
                const float by = __shfl_sync(0xffffffffu, last ? pty : ty, j + G - 1, G);
                const float bz = __shfl_sync(0xffffffffu, last ? ptz : tz, j + G - 1, G);
                if (i > 0 && i < N) {
                    // UpdateCurvaturesFromTangents_RadiativeTransfer (CurvePerturbUtils.cpp:157-166, bound N-1)
                    const float kappa = __fsqrt_rn(dev::rdot3(__fmul_rn(__fsub_rn(tx, bx), c.inv_ds), __fmul_rn(__fsub_rn(ty, by), c.inv_ds),
                                                              __fmul_rn(__fsub_rn(tz, bz), c.inv_ds)));
                    // WeightCurveViaCurvatureLog10_CudaSafe (PathWeighters.cpp:27-104)
                    double blend = 0.0;
                    const bool nan = dev::rbin_blend(kappa, lut, m, blend, cl) < 0;
                    const double v = blend * c.absorption_factor;
                    const int hi = __double2hiint(v);   // sign, exponent, high mantissa bits
                    odd |= nan || hi < 0x00100000 || hi >= 0x7ff00000;
                    esum += (hi >> 20) - 1023;
                    prod *= __hiloint2double((hi & 0x000fffff) | 0x3ff00000, __double2loint(v));
                }
                ptx = tx; pty = ty; ptz = tz;
                if ((r & 511u) == 511u) {   // 512 mantissas stay below 2^512
                    esum += (__double2hiint(prod) >> 20) - 1023;
                    prod = __hiloint2double((__double2hiint(prod) & 0x000fffff) | 0x3ff00000, __double2loint(prod));
                }
            }
            esum += (__double2hiint(prod) >> 20) - 1023;
            prod = __hiloint2double((__double2hiint(prod) & 0x000fffff) | 0x3ff00000, __double2loint(prod));
#pragma unroll
            for (int o = 1; o < G; o <<= 1) {
                prod *= __shfl_xor_sync(0xffffffffu, prod, o);
                esum += __shfl_xor_sync(0xffffffffu, esum, o);
            }
            uint32_t how = kProduct;
            if (__ballot_sync(0xffffffffu, odd) & gmask) {
                double running;
                cl = 0;
                const bool ok = plain_path_in_order(x, c, lut, m, running, cl);
                if (j > 0) cl = 0;   // every lane of the group weighed the same path
                how = !ok ? kFailed : running > -INFINITY ? kSum : met ? kZero : kZeroFirst;
                prod = running;
            }
            if (active) {
                clamped += cl;
                met |= how != kFailed;
                if (wstep % G == j) {
                    kept = how;
                    kept_w = prod;
                    kept_e = esum;
                }
            }
            if (wstep % G == G - 1 || wstep + 1 == c.steps) {
                if (kept != kNone) {
                    const double running = kept == kProduct ? log10(kept_w) + (double)kept_e * 0.30102999566398119521
                                           : kept == kFailed ? NAN : kept_w;
                    // a zero weight adds nothing, unless it is the accumulator's first: the
                    // reference's CombinedWeightValues_C then scales by 10^inf and stays NaN
                    if (kept == kProduct || kept == kSum) dev::cw_add(cw, running);
                    if (kept == kFailed) ++failed;
                    else ++valid;
                    poisoned |= kept == kZeroFirst;
                    if (exp_w) exp_w[(size_t)chain * c.steps + (wstep - wstep % G + j)] = running;
                    kept = kNone;
                }
            }
            if (exp_pos && active) {
                // export replay: every weighted path of this chain, in step order (a weights-only
                // replay passes no position buffer)
                float *dst = exp_pos + ((size_t)chain * c.steps + wstep) * 3 * (size_t)(N + 1);
                for (uint32_t e = j; e < 3 * (N + 1); e += G) dst[e] = x[(e % 3) * (N + 1) + e / 3];
            }
            __syncwarp();
        }
    }
    double part = dev::cw_log10(cw), mx = part;
#pragma unroll
    for (int o = 1; o < G; o <<= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    double sum = part > -INFINITY ? exp10(part - mx) : 0.0;
    if (poisoned || isnan(part)) sum = NAN;
#pragma unroll
    for (int o = 1; o < G; o <<= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        valid += __shfl_xor_sync(0xffffffffu, valid, o);
        failed += __shfl_xor_sync(0xffffffffu, failed, o);
        clamped += __shfl_xor_sync(0xffffffffu, clamped, o);
    }
    if (j == 0 && real) {
        ChainOut o;
        o.log10_sum = mx > -INFINITY || isnan(sum) ? mx + log10(sum) : -INFINITY;
        o.valid = valid;
        o.failed = failed;
        o.clamped = clamped;
        o.pad = 0;
        out[chain] = o;
    }
}

// Floats of shared memory per chain: three planes of N + 1, padded so that the chains of a warp
// start G banks apart (G lanes read G consecutive points).
uint32_t plain_smem_stride(uint32_t n, int G)
{
    const uint32_t f = 3 * (n + 1);
    if (G == 32) return f;
    return f + ((uint32_t)G + 32u - f % 32u) % 32u;
}

template <int G, bool SMEM>
cudaError_t launch_plain_t(const ChainSpec &c, const float *init_pos, float *state, const float *lut, LutMetaF m, ChainOut *out,
                           cudaStream_t st, float *exp_pos, double *exp_w)
{
    constexpr uint32_t per_block = kPlainThreads / G;
    const uint32_t blocks = (c.n_chains + per_block - 1) / per_block;
    const uint32_t stride = SMEM ? plain_smem_stride(c.n_segments, G) : (uint32_t)plain_state_floats_per_chain(c.n_segments);
    const size_t smem = SMEM ? sizeof(float) * (size_t)stride * per_block : 0;
    auto kern = plain_chain_kernel<G, SMEM>;
    if (SMEM) {
        const cudaError_t e = grant_smem(kern, smem);
        if (e != cudaSuccess) return e;
    }
    kern<<<blocks, kPlainThreads, smem, st>>>(c, init_pos, state, stride, lut, m, out, exp_pos, exp_w);
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------------
// FP64 form: positions, rotation, tangents, curvatures, table and weights in double. The
// proposal sequence is the same Philox draw; the rotation is the matrix of the unit
// quaternion (cos a/2, axis sin a/2) applied as q^-1 p q, as the reference's quaternion
// sandwich (CurvePerturbUtils.cpp:113-127). Tangents are recomputed on the fly, so only
// the positions live in global memory.
// ------------------------------------------------------------------------------------
__device__ __forceinline__ double lse_term(double &mx, double &sum, double &comp, double v, uint32_t n)
{
    if (n == 0) { mx = v; sum = 1.0; comp = 0.0; return 0.0; }
    if (v > mx) {
        const double f = exp10(mx - v);
        sum = sum * f;
        comp = comp * f;
        mx = v;
        v = 1.0;
    } else {
        v = exp10(v - mx);
    }
    const double y = v - comp, t = sum + y;
    comp = (t - sum) - y;
    sum = t;
    return 0.0;
}

__global__ void __launch_bounds__(kPlainThreads) fp64_chain_kernel(ChainSpec c, const float *__restrict__ init_pos,
                                                                    double *__restrict__ state,
                                                                    const double *__restrict__ lut, double min_k,
                                                                    double max_k, double step, int32_t bins,
                                                                    ChainOut *__restrict__ out)
{
    const uint32_t chain = blockIdx.x * blockDim.x + threadIdx.x;
    if (chain >= c.n_chains) return;
    const uint32_t N = c.n_segments;
    double *pos = state + (size_t)chain * 3 * (N + 1);
    for (uint32_t i = 0; i < 3 * (N + 1); ++i) pos[i] = (double)init_pos[i];
    const double arclength = (double)c.arclength;
    const double inv_ds = (double)N / arclength;
    const double absorption_factor = c.absorption_factor;
    double mx = 0.0, sum = 0.0, comp = 0.0;
    uint32_t valid = 0, failed = 0, clamped = 0;
    const uint32_t steps = (chain == c.n_chains - 1) ? c.last_steps : c.steps;
    const uint32_t total = c.burn_in + steps;
    for (uint32_t s = 0; s < total; ++s) {
        const dev::Proposal pr = dev::draw_step(c.seed, c.experiment, c.chain0 + chain, s, N, c.k_eff, c.max_angle);
        const uint32_t left = pr.left, right = pr.left + pr.k;
        const double lx = pos[3 * left], ly = pos[3 * left + 1], lz = pos[3 * left + 2];
        const double dx = pos[3 * right] - lx, dy = pos[3 * right + 1] - ly, dz = pos[3 * right + 2] - lz;
        const double inv = 1.0 / sqrt(dx * dx + dy * dy + dz * dz);
        const double ax = dx * inv, ay = dy * inv, az = dz * inv;
        double sn, cs;
        sincos(0.5 * (double)pr.angle, &sn, &cs);
        const double qw = cs, qx = ax * sn, qy = ay * sn, qz = az * sn;
        const double r00 = 1 - 2 * (qy * qy + qz * qz), r01 = 2 * (qx * qy - qw * qz), r02 = 2 * (qx * qz + qw * qy);
        const double r10 = 2 * (qx * qy + qw * qz), r11 = 1 - 2 * (qx * qx + qz * qz), r12 = 2 * (qy * qz - qw * qx);
        const double r20 = 2 * (qx * qz - qw * qy), r21 = 2 * (qy * qz + qw * qx), r22 = 1 - 2 * (qx * qx + qy * qy);
        for (uint32_t i = left + 1; i < right; ++i) {
            const double vx = pos[3 * i] - lx, vy = pos[3 * i + 1] - ly, vz = pos[3 * i + 2] - lz;
            pos[3 * i] = r00 * vx + r01 * vy + r02 * vz + lx;
            pos[3 * i + 1] = r10 * vx + r11 * vy + r12 * vz + ly;
            pos[3 * i + 2] = r20 * vx + r21 * vy + r22 * vz + lz;
        }
        if (s < c.burn_in) continue;
        double running = 0.0;
        bool ok = true;
        double px = 0, py = 0, pz = 0;  // previous tangent
        for (uint32_t i = 0; i < N; ++i) {
            double x = pos[3 * i + 3] - pos[3 * i], y = pos[3 * i + 4] - pos[3 * i + 1], z = pos[3 * i + 5] - pos[3 * i + 2];
            if (c.has_eval_shift && i == N - 2) {
                x += (double)c.eval_shift[0];
                y += (double)c.eval_shift[1];
                z += (double)c.eval_shift[2];
            }
            const double r = 1.0 / sqrt(x * x + y * y + z * z);
            const double tx = x * r, ty = y * r, tz = z * r;
            if (i > 0) {
                const double cx = (tx - px) * inv_ds, cy = (ty - py) * inv_ds, cz = (tz - pz) * inv_ds;
                double kappa = sqrt(cx * cx + cy * cy + cz * cz);
                if (isnan(kappa)) { ok = false; break; }
                if (kappa < min_k) kappa = min_k;
                if (kappa > max_k) {
                    if (kappa - max_k >= 1e-3) ++clamped;
                    kappa = max_k;
                }
                const double dist = kappa - min_k;
                int32_t l = (int32_t)floor(dist / step);
                if (l > bins - 1) l = bins - 1;
                const int32_t rr = (l == bins - 1) ? l : l + 1;
                const double interp = dist - (double)l * step;
                const double v = (lut[l] * (1.0 - interp) + lut[rr] * interp) * absorption_factor;
                const double lg = log10(v);
                if (isnan(lg)) { ok = false; break; }
                running += lg;
            }
            px = tx; py = ty; pz = tz;
        }
        if (ok) { lse_term(mx, sum, comp, running, valid); ++valid; }
        else ++failed;
    }
    ChainOut o;
    o.log10_sum = valid ? mx + log10(sum + comp) : -INFINITY;
    o.valid = valid;
    o.failed = failed;
    o.clamped = clamped;
    o.pad = 0;
    out[chain] = o;
}

// ------------------------------------------------------------------------------------
// FP64 global reduction over chains: log10 of the summed weight, and the standard error
// of that sum from the spread of the chain sums (chains are independent; their within-
// chain correlation is absorbed by treating each chain sum as one observation).
// ------------------------------------------------------------------------------------
__device__ ReduceOut reduce_result(double mx, double s1, double s2, uint32_t n, unsigned long long valid, unsigned long long failed,
                                   unsigned long long clamped)
{
    ReduceOut r;
    r.max_chain_log10 = mx;
    r.log10_sum = (mx > -INFINITY && s1 > 0.0) ? mx + log10(s1) : -INFINITY;
    double se = NAN;
    if (n > 1 && s1 > 0.0) {
        const double mean = s1 / n;
        const double var = fmax(0.0, (s2 - n * mean * mean) / (n - 1));
        se = sqrt(n * var) / s1;
    }
    r.rel_se = se;
    r.valid = valid;
    r.failed = failed;
    r.clamped = clamped;
    return r;
}

// With ranges set, CTA x reduces the chains ranges[x] = (first, count) into out[x] (one
// experiment of a batch per CTA).
__global__ void __launch_bounds__(1024) reduce_kernel(const ChainOut *__restrict__ chains, uint32_t n,
                                                       ReduceOut *__restrict__ out, const uint2 *__restrict__ ranges)
{
    if (ranges) {
        const uint2 rg = ranges[blockIdx.x];
        chains += rg.x;
        n = rg.y;
        out += blockIdx.x;
    }
    __shared__ double sd[32], sd2[32], sd3[32];
    __shared__ unsigned long long su[3][32];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
    double mx = -INFINITY;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) mx = fmax(mx, chains[i].log10_sum);
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (l == 0) sd[w] = mx;
    __syncthreads();
    if (w == 0) {
        double v = l < nw ? sd[l] : -INFINITY;
        for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (l == 0) sd[0] = v;
    }
    __syncthreads();
    mx = sd[0];
    __syncthreads();
    double s1 = 0.0, c1 = 0.0, s2 = 0.0;
    unsigned long long nv = 0, nf = 0, nc = 0;
    if (mx > -INFINITY) {
        for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
            const ChainOut ch = chains[i];
            const double x = (ch.log10_sum > -INFINITY) ? exp10(ch.log10_sum - mx) : 0.0;
            const double y = x - c1, t = s1 + y;
            c1 = (t - s1) - y;
            s1 = t;
            s2 += x * x;
        }
    }
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        nv += chains[i].valid;
        nf += chains[i].failed;
        nc += chains[i].clamped;
    }
    s1 -= c1;
    for (int o = 16; o > 0; o >>= 1) {
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
        nv += __shfl_xor_sync(0xffffffffu, nv, o);
        nf += __shfl_xor_sync(0xffffffffu, nf, o);
        nc += __shfl_xor_sync(0xffffffffu, nc, o);
    }
    if (l == 0) { sd2[w] = s1; sd3[w] = s2; su[0][w] = nv; su[1][w] = nf; su[2][w] = nc; }
    __syncthreads();
    if (w == 0) {
        s1 = l < nw ? sd2[l] : 0.0;
        s2 = l < nw ? sd3[l] : 0.0;
        nv = l < nw ? su[0][l] : 0;
        nf = l < nw ? su[1][l] : 0;
        nc = l < nw ? su[2][l] : 0;
        for (int o = 16; o > 0; o >>= 1) {
            s1 += __shfl_xor_sync(0xffffffffu, s1, o);
            s2 += __shfl_xor_sync(0xffffffffu, s2, o);
            nv += __shfl_xor_sync(0xffffffffu, nv, o);
            nf += __shfl_xor_sync(0xffffffffu, nf, o);
            nc += __shfl_xor_sync(0xffffffffu, nc, o);
        }
        if (l == 0) {
            *out = reduce_result(mx, s1, s2, n, nv, nf, nc);
        }
    }
}

// The same reduction of one pass's chains by a cluster of 8 CTAs, for the passes of many chains: one CTA
// makes two passes over them and an FP64 power of ten each on one SM. 16384 chains 17.8 -> 7.4 us, 40000 37.7 -> 10.0;
// both take 6.7 at 4096, where the line lies (3072: 5.9 by one CTA, 6.7 by the cluster, whose CTAs start and meet later).
constexpr int kReduceCtas = 8;
constexpr uint32_t kReduceClusterFrom = 4096;

struct ReducePart {
    double mx, s1, s2;
    unsigned long long nv, nf, nc;
};

__global__ void __cluster_dims__(kReduceCtas, 1, 1) __launch_bounds__(1024)
reduce_cluster_kernel(const ChainOut *__restrict__ chains, uint32_t n, ReduceOut *__restrict__ out)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    __shared__ ReducePart s_warp[32], s_cta;
    __shared__ double s_max;
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const uint32_t t0 = cl.block_rank() * blockDim.x + threadIdx.x, tn = kReduceCtas * blockDim.x;
    double mx = -INFINITY;
    for (uint32_t i = t0; i < n; i += tn) mx = fmax(mx, chains[i].log10_sum);
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (l == 0) s_warp[w].mx = mx;
    __syncthreads();
    if (w == 0) {
        mx = s_warp[l].mx;
        for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (l == 0) s_max = mx;
    }
    cl.sync();
    for (int r = 0; r < kReduceCtas; ++r) mx = fmax(mx, *cl.map_shared_rank(&s_max, r));
    ReducePart p{mx, 0.0, 0.0, 0, 0, 0};
    double c1 = 0.0;
    for (uint32_t i = t0; i < n; i += tn) {
        const ChainOut ch = chains[i];
        if (mx > -INFINITY) {
            const double x = (ch.log10_sum > -INFINITY) ? exp10(ch.log10_sum - mx) : 0.0;
            const double y = x - c1, t = p.s1 + y;
            c1 = (t - p.s1) - y;
            p.s1 = t;
            p.s2 += x * x;
        }
        p.nv += ch.valid;
        p.nf += ch.failed;
        p.nc += ch.clamped;
    }
    p.s1 -= c1;
    auto fold = [&] {
        for (int o = 16; o > 0; o >>= 1) {
            p.s1 += __shfl_xor_sync(0xffffffffu, p.s1, o);
            p.s2 += __shfl_xor_sync(0xffffffffu, p.s2, o);
            p.nv += __shfl_xor_sync(0xffffffffu, p.nv, o);
            p.nf += __shfl_xor_sync(0xffffffffu, p.nf, o);
            p.nc += __shfl_xor_sync(0xffffffffu, p.nc, o);
        }
    };
    fold();
    if (l == 0) s_warp[w] = p;
    __syncthreads();
    if (w == 0) {
        p = s_warp[l];
        fold();
        if (l == 0) s_cta = p;
    }
    cl.sync();
    if (t0 == 0) {
        for (int r = 1; r < kReduceCtas; ++r) {
            const ReducePart &q = *cl.map_shared_rank(&s_cta, r);
            p.s1 += q.s1;
            p.s2 += q.s2;
            p.nv += q.nv;
            p.nf += q.nf;
            p.nc += q.nc;
        }
        *out = reduce_result(mx, p.s1, p.s2, n, p.nv, p.nf, p.nc);
    }
    cl.sync();   // the CTAs' shared memory stays until it has been read
}

// ------------------------------------------------------------------------------------
// Weigh given paths with the reference's FP32 semantics: one path per thread.
// ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128) weigh_plain_kernel(const float *__restrict__ pos, uint64_t n_paths,
                                                           uint32_t N, float inv_ds, const float *__restrict__ lut,
                                                           LutMetaF mf, double absorption_factor,
                                                           double *__restrict__ log10w, uint8_t *__restrict__ valid,
                                                           int32_t *__restrict__ bins)
{
    const uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n_paths) return;
    const float *pp = pos + p * 3 * (uint64_t)(N + 1);
    const dev::LutMeta m{mf.min_k, mf.max_k, mf.step, mf.bins};
    double running = 0.0;
    bool ok = true;
    uint32_t clamped = 0;
    float px = 0.f, py = 0.f, pz = 0.f;
    for (uint32_t i = 0; i < N; ++i) {
        const float x = __fsub_rn(pp[3 * i + 3], pp[3 * i]), y = __fsub_rn(pp[3 * i + 4], pp[3 * i + 1]),
                    z = __fsub_rn(pp[3 * i + 5], pp[3 * i + 2]);
        const float r = dev::rinvnorm(x, y, z);
        const float tx = __fmul_rn(x, r), ty = __fmul_rn(y, r), tz = __fmul_rn(z, r);
        if (i > 0) {
            const float cx = __fmul_rn(__fsub_rn(tx, px), inv_ds), cy = __fmul_rn(__fsub_rn(ty, py), inv_ds),
                        cz = __fmul_rn(__fsub_rn(tz, pz), inv_ds);
            const float kappa = __fsqrt_rn(dev::rdot3(cx, cy, cz));
            double blend = 0.0;
            const int32_t b = ok ? dev::rbin_blend(kappa, lut, m, blend, clamped) : -1;
            if (bins) bins[p * (N - 1) + (i - 1)] = b;
            if (ok) {
                if (b < 0) ok = false;
                else {
                    const double lg = log10(blend * absorption_factor);
                    if (isnan(lg)) ok = false;
                    else running += lg;
                }
            }
        }
        px = tx; py = ty; pz = tz;
    }
    log10w[p] = ok ? running : 0.0;
    if (valid) valid[p] = ok ? 1 : 0;
}

}  // namespace

// Lanes per chain: the fewest of 8, 16 and 32 that give an SM at least 768 threads, from the chains
// of the pass and from those that fit in its shared memory (fewer lanes spend less on the work that
// every lane of a chain repeats; below 768 threads the latency of a step shows).
cudaError_t launch_plain_chains(const ChainSpec &c, const float *init_pos, float *state, const float *lut,
                                LutMetaF m, ChainOut *out, cudaStream_t st, float *exp_pos, double *exp_w)
{
    if (c.n_chains == 0) return cudaSuccess;
    if (plain_state_floats_per_chain(c.n_segments) > 0)
        return launch_plain_t<32, false>(c, init_pos, state, lut, m, out, st, exp_pos, exp_w);
    constexpr uint64_t kSms = 148, kSmem = 227 * 1024;
    auto threads_per_sm = [&](int G) {
        const uint64_t fit = kSmem / (sizeof(float) * plain_smem_stride(c.n_segments, G));
        return std::min<uint64_t>(fit, (c.n_chains + kSms - 1) / kSms) * (uint64_t)G;
    };
    if (threads_per_sm(8) >= 768) return launch_plain_t<8, true>(c, init_pos, state, lut, m, out, st, exp_pos, exp_w);
    if (threads_per_sm(16) >= 768) return launch_plain_t<16, true>(c, init_pos, state, lut, m, out, st, exp_pos, exp_w);
    return launch_plain_t<32, true>(c, init_pos, state, lut, m, out, st, exp_pos, exp_w);
}

cudaError_t launch_fp64_chains(const ChainSpec &c, const float *init_pos, double *state, const double *lut,
                               double min_k, double max_k, double step, int32_t bins, ChainOut *out, cudaStream_t st)
{
    const uint32_t blocks = (c.n_chains + kPlainThreads - 1) / kPlainThreads;
    fp64_chain_kernel<<<blocks, kPlainThreads, 0, st>>>(c, init_pos, state, lut, min_k, max_k, step, bins, out);
    return cudaGetLastError();
}

cudaError_t launch_reduce(const ChainOut *chains, uint32_t n, ReduceOut *out, cudaStream_t st)
{
    if (n >= kReduceClusterFrom) reduce_cluster_kernel<<<kReduceCtas, 1024, 0, st>>>(chains, n, out);
    else reduce_kernel<<<1, 1024, 0, st>>>(chains, n, out, nullptr);
    return cudaGetLastError();
}

cudaError_t launch_reduce_segments(const ChainOut *chains, const uint2 *ranges, uint32_t n_segments, ReduceOut *out,
                                   cudaStream_t st)
{
    if (n_segments == 0) return cudaSuccess;
    reduce_kernel<<<n_segments, 1024, 0, st>>>(chains, 0, out, ranges);
    return cudaGetLastError();
}

cudaError_t launch_weigh_plain(const float *pos, uint64_t n_paths, uint32_t n_segments, float inv_ds,
                               const float *lut, LutMetaF m, double absorption_factor, double *log10w,
                               uint8_t *valid, int32_t *bins, cudaStream_t st)
{
    if (n_paths == 0) return cudaSuccess;
    const uint64_t blocks = (n_paths + 127) / 128;
    weigh_plain_kernel<<<(unsigned)blocks, 128, 0, st>>>(pos, n_paths, n_segments, inv_ds, lut, m,
                                                         absorption_factor, log10w, valid, bins);
    return cudaGetLastError();
}

// ------------------------------------------------------------------------ path histogram
namespace {
// Linear path weights 10^(w + log10_norm) counted into nbins equal buckets over [lo, hi]: below
// lo into the first, above hi into the last (the reference's rule,
// FullExperimentRunnerOptimalPerturb.cpp:562-575, whose index for a weight of exactly hi is one
// past its last bucket: here the last); NaN (unwritten or invalid) weights are not counted.
__global__ void __launch_bounds__(256) weight_histogram_kernel(const double *__restrict__ w, uint64_t n,
                                                               double log10_norm, double lo, double hi,
                                                               uint32_t nbins, unsigned long long *__restrict__ counts)
{
    extern __shared__ unsigned int h[];
    for (uint32_t i = threadIdx.x; i < nbins; i += blockDim.x) h[i] = 0u;
    __syncthreads();
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (uint64_t)gridDim.x * blockDim.x) {
        const double x = w[p];
        if (isnan(x)) continue;
        const double v = exp10(x + log10_norm);
        uint32_t b;
        if (v < lo) b = 0;
        else if (v > hi) b = nbins - 1;
        else b = min((uint32_t)((v - lo) / (hi - lo) * (double)nbins), nbins - 1);
        atomicAdd(&h[b], 1u);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < nbins; i += blockDim.x)
        if (h[i]) atomicAdd(&counts[i], (unsigned long long)h[i]);
}
}  // namespace

cudaError_t launch_weight_histogram(const double *w, uint64_t n, double log10_norm, double lo, double hi, uint32_t nbins,
                                    unsigned long long *counts, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    const uint64_t blocks = std::min<uint64_t>((n + 255) / 256, 148 * 8);
    weight_histogram_kernel<<<(unsigned)blocks, 256, sizeof(unsigned int) * nbins, st>>>(w, n, log10_norm, lo, hi, nbins,
                                                                                         counts);
    return cudaGetLastError();
}

}  // namespace twisty
