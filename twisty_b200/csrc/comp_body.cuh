// comp_body.cuh -- the compensated B200 form of the Markov-chain hot path: the chain body
// shared by the single-run kernels (chain_comp.cu) and the batched kernels (batch.cu).
//
// Algorithm: the reference's GeometryRandom loop (Twisty/FullExperimentRunnerOptimalPerturb.cpp:
// 469-595): per step, rotate the points strictly between a random pivot `left` and
// `right = left + k` about the axis x_right - x_left by a random angle, recompute every
// tangent and curvature, gather each curvature's weight from the table, sum the log10
// weights, and accumulate the path weight into the experiment's running sum.
//
// B200 layout and arithmetic:
//  * G lanes cooperate on one chain (G = 1, 4, 8, 16 or 32); lane j owns the SPL contiguous
//    segments j*SPL .. j*SPL+SPL-1. The chain lives in shared memory as its unit tangents
//    t_i and segment lengths l_i. Rotating the points between left and right about the
//    chord x_right - x_left turns every tangent t_left .. t_{right-1} by the same rotation
//    (the chord is the axis and stays fixed) and leaves the lengths alone; each rotated
//    tangent is renormalised by one Newton step, so |t_i| = 1 to an ulp and the full
//    recompute needs no normalisation: kappa_i = |t_{i+1} - t_i| N/S.
//  * What bounds the step at 8 and 16 lanes per chain is the shared-memory pipe (16 x 16 at
//    N = 256: 90 % of its wavefronts, 83 % of the issue slots): 12 bytes per tangent
//    of the full recompute and 8 per table gather, then the shuffles. So a proposal takes three
//    shuffles (k and left in one word, sine and 1 - cosine ready), a chord's three sums travel
//    together (group_sum3), and four paths' totals are summed together (batch_step): N = 256
//    10.18 -> 9.55 ms per 2^25 paths. With 32 lanes the issue slots bind: those shapes keep pairs of
//    segments and compute on them with the packed FP32 instructions (Layout, for_curvatures):
//    N = 512 3.84 -> 3.40 ms per 2^23 paths.
//  * Rotation: the chord is summed across the group (for full-warp groups as 32-bit fixed
//    point with the warp reduction instruction, scaled by the chain's longest segment so
//    that 64 segments cannot overflow; otherwise by float shuffles), normalised, and each
//    tangent in the sub-chain is turned by Rodrigues' formula (groups of 1 and 4 lanes: by
//    v + (R - I) v, the matrix built once per step) with the angle's sin and 1 - cos taken
//    from the proposal's half-angle sine and cosine. Forward passes of short chains turn the
//    complement of a sub-chain longer than half the path instead (chain_body).
//  * The table is staged once per CTA in shared memory as float2. In the fixed-point form
//    entry i holds round((log10 L_i - c0) 2^s) as uint32 bits and the change of log10 of
//    the blend across the bin (secant): a segment costs one 8-byte LDS, one integer add
//    (exact) and one FMA (the interpolation correction). Each lane rounds its correction
//    sum to the same fixed point, the group adds the lanes' totals with integer shuffles
//    (exact, four paths together), and the chain's running log-sum-exp keeps its reference exponent as an
//    integer path total, so a path's weight relative to the running maximum is exp2 of an
//    exact integer difference. The host scales the table so that N+1 entries stay below
//    2^31; when that leaves fewer than 22 fraction bits, or the secant would lose more
//    than ~1e-7 per segment, the host selects the exact form instead: (L_i, L_{i+1} - L_i),
//    a log2 per segment, a Kahan-compensated FP32 sum combined across lanes by TwoSum and
//    a log-sum-exp over (hi, lo) float pairs.
//  * Incremental variant (ChainSpec.incr_resync = R > 0, fixed-point tables only): a rotation
//    turns the tangents of its sub-chain together, so of the path's curvatures only the two
//    at its ends change (interior ones are invariant up to rounding). Each weighted step
//    evaluates those two terms before and after the rotation and adds the difference to the
//    path's integer total; every R-th weighted step recomputes the total in full. This is an
//    algorithmic change of the recompute-everything definition and is reported separately.
//  * FP64 appears only per chain (assembling its log10 sum), in the per-CTA log-sum-exp of
//    the chains and in the global reduction (and per path in the exact form).
//  * Proposals: lane j of a group draws the Philox proposal of step base+j (one draw per
//    lane per G steps) and shuffles broadcast it.
#pragma once
#include "kernels.h"
#include "device_common.cuh"

#include <algorithm>
#include <cfloat>

namespace twisty {

// Shared by the translation units that instantiate the chain kernels (plain structs).
struct CompConsts {
    float kscale;        // (N/S) / step : |t_{i+1}-t_i| -> fractional bin index; the chain kernels keep
                         // their tangents scaled to length kscale, so |t'_{i+1}-t'_i| is the index
    float roff;          // -min_k / step
    float rmax;          // (max_k - min_k) / step
    float rsnap;         // 1e-3 / step: overshoot that counts as clamped
    float step;
    int32_t bins;
    float fscale;        // 2^s of the fixed-point table
    float l2s;           // 2^-s log2(10): fixed-point units -> log2
    int32_t wide;        // 64-bit path totals (the table's LogFixed.wide)
    double lw_offset;    // (N-1) c0 of the fixed-point table
    double inv_scale;    // 2^-s of the fixed-point table
};

struct ModeArgs {
    double log10_abs;    // log10 of the per-segment absorption factor
    // linear table (L_i, L_{i+1} - L_i) of the fixed-point table's curve: paths that cross a
    // steep bin (NaN slope) are re-weighed through it
    const float2 *lin;
    // export
    float *exp_pos;      // [chains][steps][N+1][3]; the chain kernel leaves unit tangents there (segment s at point s + 1)
    double *exp_w;       // [chains][steps] log10 weights (absorption included, normaliser not)
    // adjoint: the derivative tables, one 16-byte load per segment (deriv_tables_kernel: the ratio
    // form with the fixed-point table, the linear form with the exact blend)
    const float4 *dtab;
    double ref_log10;    // log10 of the forward sum of path weights (normaliser and absorption excluded)
    double *grad;        // [chains][6]: d/dmu_s, d/deps, d/dx, d/dy, d/dz (log10 units), sum of weights
};

namespace {

constexpr uint32_t FULL = 0xffffffffu;
constexpr int kMaxSubChain = 64;  // largest k the rotation rounds cover
constexpr float kLog2_10 = 3.32192809488736234787f;
constexpr float kLog10_2 = 0.30102999566398119521f;
constexpr float kInvLn10 = 0.43429448190325182765f;


__device__ __forceinline__ float sqrt_approx(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float ex2_approx(float x)
{
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Two floats in one 64-bit register: the packed FP32 instructions of sm_100 round each half as
// the scalar instruction does and take one issue slot for two operations (measured: 1.95
// packed FMAs per clock and SM against 3.8 scalar ones -- the same arithmetic rate from half
// the issue slots, which the loads, conversions and integer work beside it then use).
struct F2 {
    uint64_t v;
    __device__ __forceinline__ float lo() const { return __uint_as_float((uint32_t)v); }
    __device__ __forceinline__ float hi() const { return __uint_as_float((uint32_t)(v >> 32)); }
};

__device__ __forceinline__ F2 pack2(float lo, float hi)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b)
{
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 add2_rd(F2 a, F2 b)   // rounded toward -infinity
{
    F2 r;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b)
{
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c)
{
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ F2 sub2(F2 a, F2 b) { return fma2(b, pack2(-1.0f, -1.0f), a); }   // a - b, exactly rounded

// The lanes of a chain, from the chain's base lane qb. Lane j of it is lane qb + j; with 4 lanes per chain
// lane qb + 8j, so that the chains sit side by side in a row of shared memory (Layout).
template <int G>
struct Lanes {
    static constexpr int CPW = 32 / G;
    static constexpr int STRIDE = G == 4 ? CPW : 1;   // from one lane of a chain to the next
    static constexpr uint32_t MASK = G == 4 ? 0x01010101u : G == 32 ? FULL : (1u << (G & 31)) - 1u;   // ballot bits from qb on
    __device__ __forceinline__ static uint32_t base_of(uint32_t lane) { return G == 4 ? lane % CPW : lane / G * G; }
    __device__ __forceinline__ static uint32_t chain_of(uint32_t lane) { return G == 4 ? lane % CPW : lane / G; }
    __device__ __forceinline__ static uint32_t lane_of(uint32_t lane) { return G == 4 ? lane / CPW : lane % G; }
    // the value of the chain's lane j
    template <class T>
    __device__ __forceinline__ static T from(T v, uint32_t j, uint32_t qb)
    {
        return G == 4 ? __shfl_sync(FULL, v, j * CPW + qb) : __shfl_sync(FULL, v, j, G);
    }
};

template <int G, class T>
__device__ __forceinline__ T group_sum(T v)
{
#pragma unroll
    for (int o = 1; o < G; o <<= 1) v += __shfl_xor_sync(FULL, v, o * Lanes<G>::STRIDE);
    return v;
}

// The sums of three values over the chain's lanes, in every lane. From 8 lanes on the three
// travel together: the first exchange takes x and y (each lane keeps one and sends the other),
// the second adds z to them, the rest move one value each, and three broadcasts end it: 8
// shuffles for 16 lanes instead of 12 (the shuffles share the shared-memory pipe that bounds
// the step). The additions pair the same lanes in the same order as three butterflies do.
template <int G>
__device__ __forceinline__ void group_sum3(float &x, float &y, float &z, uint32_t j, uint32_t qb)
{
    constexpr int S = Lanes<G>::STRIDE;
    if constexpr (G < 8) {
        x = group_sum<G>(x);
        y = group_sum<G>(y);
        z = group_sum<G>(z);
    } else {
        const bool b0 = j & 1u, b1 = j & 2u;
        float p = b0 ? y : x;
        p += __shfl_xor_sync(FULL, b0 ? x : y, S);
        z += __shfl_xor_sync(FULL, z, S);
        float r = b1 ? z : p;
        r += __shfl_xor_sync(FULL, b1 ? p : z, 2 * S);
#pragma unroll
        for (int o = 4; o < G; o <<= 1) r += __shfl_xor_sync(FULL, r, o * S);
        x = Lanes<G>::from(r, 0, qb);
        y = Lanes<G>::from(r, 1, qb);
        z = Lanes<G>::from(r, 2, qb);
    }
}

// TwoSum-combine the lanes' Kahan pairs (hi, lo) of one group.
template <int G>
__device__ __forceinline__ void group_sum_pair(float &hi, float &lo)
{
#pragma unroll
    for (int o = 1; o < G; o <<= 1) {
        const float oh = __shfl_xor_sync(FULL, hi, o * Lanes<G>::STRIDE);
        const float ol = __shfl_xor_sync(FULL, lo, o * Lanes<G>::STRIDE);
        const float s = hi + oh;
        const float bp = s - hi;
        const float e = (hi - (s - bp)) + (oh - bp);
        hi = s;
        lo = lo + ol + e;
    }
}

__device__ __forceinline__ void kahan_add(float &s, float &c, float x)
{
    const float y = x - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
}

// Fractional bin index of |t_{i+1}-t_i|^2 and its bin. CLAMP handles tables whose curvature
// range a path can leave; tables spanning [0, 2.02 N/S] (the reference's) cannot be left by
// unit tangents (|t_{i+1}-t_i| <= 2). r >= 0 or NaN after the clamp. Returns the fraction
// r - L within bin L. floor(r) comes without conversion instructions (which share the MUFU
// pipe with the square root): r + 2^23 rounded toward -infinity carries floor(r) in its low
// mantissa bits for 0 <= r < 2^23. NaN and infinity, which only a degenerate zero-length
// chord can produce, land past the last bin, are bounded to it and get a NaN fraction.
template <bool B>
struct BoolTag {
    static constexpr bool value = B;
};

template <bool CLAMP>
__device__ __forceinline__ float bin_of(float qq, const CompConsts &k, bool valid, uint32_t &clamped, int32_t &L)
{
    // qq is |t'_{i+1} - t'_i|^2 of tangents scaled to length kscale: its root is the
    // fractional bin of a table starting at curvature 0 (tables that need no clamping do)
    float r = CLAMP ? sqrt_approx(qq) + k.roff : sqrt_approx(qq);
    if (CLAMP) {
        if (r < 0.0f) r = 0.0f;
        if (r > k.rmax) {
            clamped += (valid && r - k.rmax >= k.rsnap) ? 1u : 0u;
            r = k.rmax;
        }
    }
    const float fl = __fadd_rd(r, 8388608.0f);
    L = (int32_t)min(__float_as_uint(fl) - 0x4B000000u, (uint32_t)k.bins - 1u);
    return r - (fl - 8388608.0f);
}

// The bins of two squared lengths at once, for tables that need no clamping: bin_of<false> with
// its additions packed. Returns both fractions.
__device__ __forceinline__ F2 bins_of(F2 qq, const CompConsts &k, int32_t &L0, int32_t &L1)
{
    const F2 r = pack2(sqrt_approx(qq.lo()), sqrt_approx(qq.hi()));
    const F2 fl = add2_rd(r, pack2(8388608.0f, 8388608.0f));
    L0 = (int32_t)min((uint32_t)fl.v - 0x4B000000u, (uint32_t)k.bins - 1u);
    L1 = (int32_t)min((uint32_t)(fl.v >> 32) - 0x4B000000u, (uint32_t)k.bins - 1u);
    return sub2(r, add2(fl, pack2(-8388608.0f, -8388608.0f)));
}

// How a warp's tangents lie in shared memory (Layout, below). Measured against XYZ with the walk in
// order (precision geometry, the batched log-sum-exp in both): PAIRS at 32 lanes N = 512 +6 %,
// 701 +5 %, but 16 x 16 -5 % (more bank conflicts in the rotation, which that shape's
// shared-memory pipe at 90 % of its wavefronts pays for) and 8 x 16 -8 % (spills); PLANES
// at 4 lanes N = 64 +17 %, 66 +13 %, at one lane N = 16 +2 %, but under the 64 registers of the 4-lane
// shapes below 12 segments per lane -4 to -7 % (N = 18, 30, 34). ORDERED: a recompute that
// walks its segments in order (the exact blend of single runs) would keep the later halves of PAIRS in registers, and
// spills: N = 544 351 -> 324 us over 2^19 paths in XYZ, 768 371 -> 306, 1024 439 -> 330, receiver-shifted 669 -> 426.
// The incremental form, which reads single tangents more often than it recomputes, takes XYZ too (2^29 path-segments,
// a recompute every 64 steps: N = 512 -11 %, 530 -13 %, 768 -10 %, 1024 -10 %).
enum { kPairs = 0, kXyz = 1, kPlanes = 2 };
__host__ __device__ constexpr int comp_layout(int G, int SPL, bool ordered = false)
{
    return G == 32 ? (ordered ? kXyz : kPairs) : G == 1 || (G == 4 && SPL >= 12) ? kPlanes : kXyz;
}
// Whether the recompute works on pairs of segments with packed arithmetic.
__host__ __device__ constexpr bool comp_packed(int G, int SPL) { return comp_layout(G, SPL) != kXyz; }

// Three pairs: the tangents of a lane's segments h and h + H, H = (SPL + 1) / 2.
struct Tan2 {
    F2 x, y, z;
};

// Walk the curvatures this lane owns (curvature i lies between segments i and i + 1; the last one
// with the next lane's first tangent). load.one(m, x, y, z) gives the tangent of segment j*SPL + m,
// zero past the last segment; next(t0, n) the next lane's first tangent given this lane's (t0).
// Every slot is evaluated, with valid = false past curvature N-2, so no table load hides behind a
// branch (padding tangents are zero: their |t_{i+1}-t_i|^2 is 0 or 1, a bin in the table). FULLN:
// N == G*SPL, only the group's last boundary is invalid.
// In the layouts with packed arithmetic, seg2(i, i', qq, valid, valid') takes two curvatures at a
// time, H = (SPL + 1) / 2 apart, and seg1(i, qq, valid) the one left over when SPL is odd: pairs
// H apart keep every difference of neighbours a difference of two register pairs,
// P_{h+1} - P_h, with load.pair(h) = the tangents of segments j*SPL + h and j*SPL + h + H (the upper
// half of the last pair of an odd SPL is not read). The others walk their segments in order.
template <int G, int SPL, bool FULLN, bool PACKED = comp_packed(G, SPL), class Load, class NextFn, class Seg2Fn, class Seg1Fn>
__device__ __forceinline__ void for_curvatures(uint32_t j, uint32_t N, const Load &load, NextFn next, Seg2Fn seg2, Seg1Fn seg1)
{
    constexpr int H = (SPL + 1) / 2;
    constexpr bool ODD = SPL & 1;
    const uint32_t base = j * SPL;
    float nx, ny, nz;
    if constexpr (!PACKED) {
        float t0x = 0.f, t0y = 0.f, t0z = 0.f, px = 0.f, py = 0.f, pz = 0.f;
#pragma unroll
        for (int m = 0; m < SPL; ++m) {
            float tx, ty, tz;
            load.one(m, tx, ty, tz);
            if (m == 0) {
                t0x = tx; t0y = ty; t0z = tz;
            } else {
                const float dx = tx - px, dy = ty - py, dz = tz - pz;
                seg1(base + m - 1, fmaf(dx, dx, fmaf(dy, dy, dz * dz)), FULLN || base + m <= N - 1);
            }
            px = tx; py = ty; pz = tz;
        }
        next(t0x, t0y, t0z, nx, ny, nz);
        const float dx = nx - px, dy = ny - py, dz = nz - pz;
        seg1(base + SPL - 1, fmaf(dx, dx, fmaf(dy, dy, dz * dz)), base + SPL <= N - 1);
    } else {
        auto sq2 = [](const Tan2 &b, const Tan2 &a) {
            const F2 dx = sub2(b.x, a.x), dy = sub2(b.y, a.y), dz = sub2(b.z, a.z);
            return fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
        };
        Tan2 first = load.pair(0);
        next(first.x.lo(), first.y.lo(), first.z.lo(), nx, ny, nz);
        if (ODD && H == 1) first = Tan2{pack2(first.x.lo(), nx), pack2(first.y.lo(), ny), pack2(first.z.lo(), nz)};
        Tan2 prev = first;
#pragma unroll
        for (int h = 1; h < H; ++h) {
            Tan2 cur = load.pair(h);
            if (ODD && h == H - 1) cur = Tan2{pack2(cur.x.lo(), nx), pack2(cur.y.lo(), ny), pack2(cur.z.lo(), nz)};
            // the upper curvature, j*SPL + h + H - 1, is the group's last boundary only for odd SPL
            seg2(base + h - 1, base + h + H - 1, sq2(cur, prev), FULLN || base + h <= N - 1,
                 (FULLN && !(ODD && h == H - 1)) || base + h + H <= N - 1);
            prev = cur;
        }
        if constexpr (ODD) {
            const float dx = first.x.hi() - prev.x.lo(), dy = first.y.hi() - prev.y.lo(), dz = first.z.hi() - prev.z.lo();
            seg1(base + H - 1, fmaf(dx, dx, fmaf(dy, dy, dz * dz)), (FULLN && SPL > 1) || base + H <= N - 1);
        } else {
            const Tan2 cur{pack2(first.x.hi(), nx), pack2(first.y.hi(), ny), pack2(first.z.hi(), nz)};
            seg2(base + H - 1, base + SPL - 1, sq2(cur, prev), FULLN || base + H <= N - 1, base + SPL <= N - 1);
        }
    }
}

// next() for tangents held in registers: the next lane's t0 by shuffle.
template <int G>
struct ShflNext {
    __device__ __forceinline__ void operator()(float t0x, float t0y, float t0z, float &nx, float &ny, float &nz) const
    {
        if constexpr (G == 1) {   // a one-lane chain has no next lane: its last slot is padding
            nx = t0x; ny = t0y; nz = t0z;
        } else {
            nx = __shfl_down_sync(FULL, t0x, Lanes<G>::STRIDE);
            ny = __shfl_down_sync(FULL, t0y, Lanes<G>::STRIDE);
            nz = __shfl_down_sync(FULL, t0z, Lanes<G>::STRIDE);
        }
    }
};

// Table entry L. GLOBAL: the table is in global memory, read through L1 by an unconditional
// non-coherent load, so that the compiler cannot turn the padded slots' loads into predicated
// ones (measured: with plain loads the padded curvature loop ran 15 % slower through L1).
template <bool GLOBAL>
__device__ __forceinline__ float2 tab_load(const float2 *__restrict__ tab, int32_t L)
{
    if constexpr (GLOBAL) {
        float2 e;
        asm("ld.global.nc.v2.f32 {%0, %1}, [%2];" : "=f"(e.x), "=f"(e.y) : "l"(tab + L));
        return e;
    } else {
        return tab[L];
    }
}

// Generic full recompute of one path's log10 weight (absorption excluded), for the exact
// table or, with 64-bit lane sums, for the fixed-point table at any lane width. bin_sink(i,
// bin) receives every curvature's bin (-1 for NaN).
template <int G, int SPL, bool EXACT, bool CLAMP, bool GLOBAL = false, bool PACKED = comp_packed(G, SPL), class Load, class NextFn,
          class BinFn>
__device__ __forceinline__ double path_log10(uint32_t j, uint32_t N, const float2 *__restrict__ tab,
                                             const CompConsts &k, const Load &load, NextFn next, BinFn bin_sink,
                                             uint32_t &clamped)
{
    unsigned long long isum = 0;
    float csum = 0.f, ks = 0.f, kc = 0.f;
    auto seg = [&](uint32_t i, float qq, bool valid) {
        int32_t L;
        const float frac = bin_of<CLAMP>(qq, k, valid, clamped, L);
        if (valid) bin_sink(i, isnan(frac) ? -1 : L);
        const float2 e = tab_load<GLOBAL>(tab, L);
        if (EXACT) {
            const float term = __log2f(fmaf(frac * k.step, e.y, e.x)) * kLog10_2;
            kahan_add(ks, kc, valid ? term : 0.0f);
        } else {
            isum += valid ? __float_as_uint(e.x) : 0u;
            const float c2 = fmaf(frac, e.y, csum);
            csum = valid ? c2 : csum;
        }
    };
    auto seg2 = [&](uint32_t i0, uint32_t i1, F2 qq, bool v0, bool v1) {
        seg(i0, qq.lo(), v0);
        seg(i1, qq.hi(), v1);
    };
    // a chain that fills its group's slots: slot validity known at compile time
    if (N == (uint32_t)(G * SPL))
        for_curvatures<G, SPL, true, PACKED>(j, N, load, next, seg2, seg);
    else
        for_curvatures<G, SPL, false, PACKED>(j, N, load, next, seg2, seg);
    if (EXACT) {
        float hi = ks, lo = -kc;
        group_sum_pair<G>(hi, lo);
        return (double)hi + (double)lo;
    }
    const unsigned long long is = group_sum<G>(isum);
    const float cs = group_sum<G>(csum);
    return k.lw_offset + (double)is * k.inv_scale + (double)cs;
}

// Fixed-point full recompute for chains: this lane's share of the path total, table entries plus
// the rounded interpolation correction, in units of 2^-s. Each lane's sum is exact in 32 bits
// (its true value lies in [0, 2^32) by the table's scale); the group total is added in 32 bits
// for a narrow table, in 64 bits for a wide one (both exact). nan is set when one of the lane's
// curvatures is NaN or in a steep bin.
template <int G, int SPL, bool CLAMP, bool GLOBAL, class Load, class NextFn>
__device__ __forceinline__ uint32_t path_fixed(uint32_t j, uint32_t N, const float2 *__restrict__ tab,
                                               const CompConsts &k, const Load &load, NextFn next, bool &nan,
                                               uint32_t &clamped)
{
    uint32_t isum = 0;
    float c0 = 0.f, c1 = 0.f;
    // a padding slot leaves the sum alone even where the slope is NaN (a steep bin)
    auto entry = [&](int32_t L, float frac, bool valid, float &c) {
        const float2 e = tab_load<GLOBAL>(tab, L);
        isum += valid ? __float_as_uint(e.x) : 0u;
        const float c2 = fmaf(frac, e.y, c);
        c = valid ? c2 : c;
    };
    auto seg1 = [&](uint32_t, float qq, bool valid) {
        int32_t L;
        const float frac = bin_of<CLAMP>(qq, k, valid, clamped, L);
        entry(L, frac, valid, c0);
    };
    auto seg2 = [&](uint32_t i0, uint32_t i1, F2 qq, bool v0, bool v1) {
        if constexpr (CLAMP) {
            int32_t L0, L1;
            const float f0 = bin_of<true>(qq.lo(), k, v0, clamped, L0), f1 = bin_of<true>(qq.hi(), k, v1, clamped, L1);
            entry(L0, f0, v0, c0);
            entry(L1, f1, v1, c1);
        } else {
            int32_t L0, L1;
            const F2 f = bins_of(qq, k, L0, L1);
            entry(L0, f.lo(), v0, c0);
            entry(L1, f.hi(), v1, c1);
        }
    };
    if (N == (uint32_t)(G * SPL))
        for_curvatures<G, SPL, true>(j, N, load, next, seg2, seg1);
    else
        for_curvatures<G, SPL, false>(j, N, load, next, seg2, seg1);
    const float csum = comp_packed(G, SPL) ? c0 + c1 : c0;
    nan = isnan(csum);
    return isum + (uint32_t)__float2int_rn(csum * k.fscale);
}

// Row pitches of the XYZ layout (float2 and float elements), and with them the bytes of shared
// memory per warp that hold its chains' tangents whatever the layout: the chain count of a pass
// with num_chains 0 follows from how many warps fit, so the size is the same for all three.
__host__ __device__ constexpr int comp_pitch_xy(int G, int SPL)
{
    return G == 1 ? 32 : 32 + ((16 / SPL) > 1 ? (16 / SPL) : 1);
}
__host__ __device__ constexpr int comp_pitch_z(int G, int SPL)
{
    return G == 1 ? 32 : 32 + ((G / SPL) > 1 ? (G / SPL) : 1);
}
__host__ __device__ constexpr int warp_state_bytes(int G, int SPL)
{
    return (SPL * (comp_pitch_xy(G, SPL) * 8 + comp_pitch_z(G, SPL) * 4) + 15) / 16 * 16;
}

// Where segment m of lane o of a chain lies (qb: the chain's base lane): a for x (XYZ: for (x, y), in
// float2), b for z in XYZ.
struct Slot {
    uint32_t a, b;
};

// The layout of a warp's tangents in shared memory:
//  * PAIRS: three planes (x, y, z); row h of each holds, per lane, the pair of segments
//    h and h + H, H = (SPL + 1) / 2, as one float2: the recompute reads a pair of tangents by three
//    8-byte loads (consecutive columns of one row, no bank conflicts) straight into the register
//    pairs that its packed arithmetic works on. Of an odd SPL's last row only the lower half
//    exists, as one float per lane. Rows are padded to PP pairs, as many as the bytes allow.
//  * XYZ: (x, y) as float2 and z in planes of one row per segment, at immediate offsets from a
//    lane's base: 12 bytes per tangent too, in an 8-byte and a 4-byte load. The row pitches
//    (32 + 16/SPL float2, 32 + G/SPL floats) put the consecutive segments of a rotation in distinct
//    banks (at most 2-way conflicts).
//  * PLANES: x, y and z in rows of 32 floats, the column rotated by the row: 4 consecutive
//    segments of a 4-lane chain lie in the chain's own 4 banks where SPL = 1 mod 4 (and mostly so for
//    other SPL), and every access of a one-lane chain in its own bank.
template <int G, int SPL, bool ORDERED = false>
struct Layout {
    static constexpr int KIND = comp_layout(G, SPL, ORDERED);
    static constexpr int H = (SPL + 1) / 2;
    static constexpr bool ODD = SPL & 1;
    static constexpr int CPW = 32 / G;
    static constexpr int PXY = comp_pitch_xy(G, SPL), PZ = comp_pitch_z(G, SPL);
    static constexpr int WARP_BYTES = warp_state_bytes(G, SPL);
    static constexpr int PP = (WARP_BYTES / 12 - (ODD ? 32 : 0)) / (SPL / 2) / 2;
    static constexpr int PLANE = KIND == kPairs ? (SPL / 2) * 2 * PP + (ODD ? 32 : 0) : SPL * 32;   // floats
    static_assert(KIND == kXyz || (PP >= 32 && 3 * PLANE * 4 <= WARP_BYTES && PLANE % 2 == 0), "the planes fit");
    __device__ __forceinline__ static Slot slot(uint32_t o, uint32_t m, uint32_t qb)
    {
        if constexpr (KIND == kPlanes) {
            const uint32_t w = m * 32u + ((CPW * (o + m) + qb) & 31u);
            return Slot{w, w};
        } else if constexpr (KIND == kXyz) {
            const uint32_t col = G == 4 ? o * CPW + qb : qb + o;
            return Slot{m * PXY + col, m * PZ + col};
        } else {
            const uint32_t col = qb + o;
            const uint32_t up = m >= (uint32_t)H ? 1u : 0u;
            uint32_t w = (m - up * H) * (2u * PP) + 2u * col + up;
            if (ODD && m == (uint32_t)(H - 1)) w = (H - 1) * 2u * PP + col;
            return Slot{w, w};
        }
    }
    __device__ __forceinline__ static void get(const float *t, Slot s, float &x, float &y, float &z)
    {
        if constexpr (KIND == kXyz) {
            const float2 v = reinterpret_cast<const float2 *>(t)[s.a];
            x = v.x;
            y = v.y;
            z = (t + SPL * PXY * 2)[s.b];
        } else {
            x = t[s.a];
            y = t[s.a + PLANE];
            z = t[s.a + 2 * PLANE];
        }
    }
    __device__ __forceinline__ static void put(float *t, Slot s, float x, float y, float z)
    {
        if constexpr (KIND == kXyz) {
            reinterpret_cast<float2 *>(t)[s.a] = make_float2(x, y);
            (t + SPL * PXY * 2)[s.b] = z;
        } else {
            t[s.a] = x;
            t[s.a + PLANE] = y;
            t[s.a + 2 * PLANE] = z;
        }
    }
};

// Threads per CTA the chain kernel of a shape is compiled for (its register budget: 65536 /
// threads). With 12 or more segments per lane every shape fits 768 threads (24 warps) in 80
// registers without spills (forward variants), and the extra warps pay: N = 256 +6 %, 512
// +13 %, 1024 +24 % over the 16 (8) warps of a 512-thread budget.
__host__ __device__ constexpr int comp_max_threads(int G, int SPL)
{
    return (SPL >= 12) ? 768 : 1024;
}

// The segment lengths, one array per CTA: rotations never change a length, and every chain of
// a CTA starts from the same initial curve, so all its chains share them (G * SPL floats,
// padding segments 1).
__host__ __device__ constexpr size_t cta_len_bytes(int G, int SPL) { return ((size_t)G * SPL * 4 + 15) / 16 * 16; }

// One warp's tangents and the CTA's segment lengths.
struct Planes {
    float *t;    // Layout
    float *l;    // CTA-wide, by segment index
};

// The tangents of lane j of the chain in slot q, for for_curvatures. SHIFT: the weights see the
// receiver moved by the spec's eval_shift: v_{N-2} = l t + shift, renormalised.
template <int G, int SPL, bool SHIFT = false, bool ORDERED = false>
struct SmemLoad {
    using Lay = Layout<G, SPL, ORDERED>;
    const Planes &st;
    uint32_t qb, j;
    uint32_t N;
    const ChainSpec *c;   // SHIFT (through a copy of its members the shifted passes ran up to 20 % slower)
    float kscale, inv_ks;
    __device__ __forceinline__ void one(int m, float &x, float &y, float &z) const
    {
        Lay::get(st.t, Lay::slot(j, m, qb), x, y, z);
        if (SHIFT && j * SPL + m == N - 2) {
            const float l = st.l[j * SPL + m] * inv_ks;
            x = fmaf(l, x, c->eval_shift[0]);
            y = fmaf(l, y, c->eval_shift[1]);
            z = fmaf(l, z, c->eval_shift[2]);
            const float r = rsqrtf(fmaf(x, x, fmaf(y, y, z * z))) * kscale;
            x *= r; y *= r; z *= r;
        }
    }
    __device__ __forceinline__ Tan2 pair(int h) const
    {
        constexpr int H = Lay::H;
        const bool both = !(Lay::ODD && h == H - 1);
        if constexpr (Lay::KIND == kPairs && !SHIFT) {
            if (both) {
                const float2 *p = reinterpret_cast<const float2 *>(st.t) + (qb + j) + h * Lay::PP;
                const float2 x = p[0], y = p[Lay::PLANE / 2], z = p[Lay::PLANE];
                return Tan2{pack2(x.x, x.y), pack2(y.x, y.y), pack2(z.x, z.y)};
            }
        }
        float x0, y0, z0, x1 = 0.f, y1 = 0.f, z1 = 0.f;
        one(h, x0, y0, z0);
        if (both) one(h + H, x1, y1, z1);
        return Tan2{pack2(x0, x1), pack2(y0, y1), pack2(z0, z1)};
    }
};

enum { kModeForward = 0, kModeExport = 1, kModeAdjoint = 2 };


// Receiver-position gradient of one path's log10 weight, computed by one lane from the last
// three segments: moving the receiver moves points N-1 and N together, so only the segment
// vector v_{N-2} changes, hence t_{N-2} and the curvatures kappa_{N-3}, kappa_{N-2}. The
// reference's interpolation weight is in curvature units (PathWeighters.cpp:79-82), so its
// segment weight is almost constant within a bin and jumps by nearly L_{b+1} - L_b at each
// edge: its pathwise derivative misses almost all of the change an expectation over paths
// sees. The slope taken is that of the expected weight: averaged over a bin the staircase is
// the table's linear interpolant taken half a bin to the left, whose slope at fractional bin r
// is (L_{J+1} - L_J) / step with J = floor(r - 1/2); divided by the weight itself.
__device__ __forceinline__ void receiver_grad(const float t3[3], const float t2[3], const float t1[3], float len2,
                                              const float2 *lin, const CompConsts &k, float inv_ds, float g[3])
{
    const float r2 = 1.0f / len2;  // d t2 / d v2 = (I - t2 t2^T) / |v2|
    g[0] = g[1] = g[2] = 0.f;
    for (int which = 0; which < 2; ++which) {
        float d[3];
        float sign;
        if (which == 0) { for (int q = 0; q < 3; ++q) d[q] = t2[q] - t3[q]; sign = 1.f; }   // kappa_{N-3}
        else { for (int q = 0; q < 3; ++q) d[q] = t1[q] - t2[q]; sign = -1.f; }             // kappa_{N-2}
        const float dn = sqrtf(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
        if (!(dn > 0.f)) continue;
        float r = fmaf(dn, k.kscale, k.roff);
        if (r < 0.f) r = 0.f;
        if (r > k.rmax) continue;  // clamped: flat
        // the linear table (L_i, L_{i+1} - L_i): the blend at r and the slope of bin J
        const int32_t L = min((int32_t)r, k.bins - 1);
        const float2 e = lin[L];
        const float dd = (r - (float)L) * k.step;
        const float blend = fmaf(dd, e.y, e.x);
        const int32_t J = min(max((int32_t)floorf(r - 0.5f), 0), k.bins - 2);
        const float sl = lin[J].y;
        const float dlog = sl / (k.step * blend) * kInvLn10;  // d log10 w / d kappa
        const float dk = dlog * inv_ds * sign / dn;                  // d kappa / d t = inv_ds d/|d|
        const float dt = d[0] * t2[0] + d[1] * t2[1] + d[2] * t2[2];
        for (int q = 0; q < 3; ++q) g[q] += dk * (d[q] - dt * t2[q]) * r2;
    }
}

// A segment's length as the chain body computes it: |v| = |v|^2 rsqrt(|v|^2).
__device__ __forceinline__ float segment_length(const float *__restrict__ v)
{
    const float ss = fmaf(v[0], v[0], fmaf(v[1], v[1], v[2] * v[2]));
    return ss * rsqrtf(ss);
}

// The CTA's segment lengths from the initial segment vectors (padding segments 1); the CTA
// synchronises before use.
__device__ __forceinline__ void fill_lengths(float *s_len, const float *__restrict__ init_seg, uint32_t n, uint32_t slots)
{
    for (uint32_t s = threadIdx.x; s < slots; s += blockDim.x) {
        const float len = s < n ? segment_length(init_seg + 3 * s) : 1.f;
        s_len[s] = len;
    }
}

// Stage a table of `bins` float2 entries into shared memory (float4 vector loads: the table starts on 16 bytes, which
// table_pitch and the callers of single tables see to; a look at the address here cost 8 x 24 6 %).
__device__ __forceinline__ void stage_table(float4 *smem4, const float2 *__restrict__ tab_g, int bins)
{
    for (int i = threadIdx.x; i < bins / 2; i += blockDim.x) smem4[i] = reinterpret_cast<const float4 *>(tab_g)[i];
    if ((bins & 1) && threadIdx.x == 0) reinterpret_cast<float2 *>(smem4)[bins - 1] = tab_g[bins - 1];
}

// Exact-blend weight of the group's current path through the linear table, for paths of a
// fixed-point table that cross a steep bin: in segment order, as every exact blend sums. Not
// inlined: it runs rarely, and inlined its registers would count against the hot loop's.
template <int G, int SPL, bool CLAMP, bool ORDERED>
__device__ __noinline__ double steep_fallback(Planes st, uint32_t qb, uint32_t j, uint32_t N,
                                              const float2 *__restrict__ lin, CompConsts kc)
{
    const SmemLoad<G, SPL, false, ORDERED> load{st, qb, j, 0, nullptr, 0.f, 0.f};   // the chain's own layout
    uint32_t unused = 0;
    return path_log10<G, SPL, true, CLAMP, true, false>(j, N, lin, kc, load, ShflNext<G>{}, [](uint32_t, int32_t) {}, unused);
}

// One Markov chain run by the G lanes of one group on its own records st (tangent, length;
// warp-local slots): initial state from init_seg (segment vectors), burn_in + steps
// proposals, a full recompute of every weighted path, and the chain's running log-sum-exp.
// Writes out[chain] (when out is set and the chain is real) and returns the chain's log10 sum.
// STEEP: the fixed-point table has steep bins (NaN slopes); paths crossing one are re-weighed
// through ma.lin. Without it a NaN slope cannot occur and a NaN total means a NaN curvature.
template <int G, int SPL, bool EXACT, bool CLAMP, bool SHIFT, int MODE, bool INCR = false, bool STEEP = false,
          bool TAB_GLOBAL = false, bool ORDERED = (EXACT && MODE != kModeAdjoint) || INCR, bool GROUPED = true>
__device__ __forceinline__ double chain_body(const ChainSpec &c, const CompConsts &kc,
                                             const float *__restrict__ init_seg, const float2 *s_tab, Planes st,
                                             uint32_t qb, uint32_t j, uint32_t chain, bool real_chain,
                                             ChainOut *__restrict__ out, const ModeArgs &ma)
{
    constexpr bool FIX = !EXACT;
    constexpr bool ADJ = MODE == kModeAdjoint;
    const uint32_t N = c.n_segments;
    using Lay = Layout<G, SPL, ORDERED>;
    // segment record (tangent, length) of segment index s = owner*SPL + m
    // the tangents are stored at length kscale; records handed to export and the adjoint are unit
    const float inv_ks = 1.0f / kc.kscale;
    auto load_rec = [&](uint32_t owner, uint32_t m) {
        float x, y, z;
        Lay::get(st.t, Lay::slot(owner, m, qb), x, y, z);
        return make_float4(x * inv_ks, y * inv_ks, z * inv_ks, st.l[owner * SPL + m]);
    };

    float max_len = 0.f;
#pragma unroll
    for (int m = 0; m < SPL; ++m) {
        const uint32_t s = j * SPL + m;
        float x = 0.f, y = 0.f, z = 0.f, len = 1.f;
        if (s < N) {
            x = init_seg[3 * s];
            y = init_seg[3 * s + 1];
            z = init_seg[3 * s + 2];
            const float ss = fmaf(x, x, fmaf(y, y, z * z));
            const float r = rsqrtf(ss);
            len = ss * r;
            x *= r; y *= r; z *= r;
            const float h = fmaf(-0.5f, fmaf(x, x, fmaf(y, y, z * z)), 1.5f);   // one Newton step to |t| = 1
            x *= h * kc.kscale; y *= h * kc.kscale; z *= h * kc.kscale;       // stored at length kscale
            max_len = fmaxf(max_len, len);
        }
        Lay::put(st.t, Lay::slot(j, m, qb), x, y, z);
    }
#pragma unroll
    for (int o = 1; o < G; o <<= 1) max_len = fmaxf(max_len, __shfl_xor_sync(FULL, max_len, o * Lanes<G>::STRIDE));
    // fixed-point chord scale: a segment is at most 2^24 units, 64 of them at most 2^30
    const float chord_scale = 16777216.0f / (max_len * kc.kscale);   // the tangents have length kscale
    const float renorm = -0.5f * inv_ks * inv_ks;   // Newton step to |t'| = kscale: 1.5 + renorm |t'|^2
    __syncwarp();

    const uint32_t steps_c = real_chain ? ((chain == c.n_chains - 1) ? c.last_steps : c.steps) : 0;
    const uint32_t total = c.burn_in + c.steps;
    const uint32_t gchain = c.chain0 + (real_chain ? chain : 0);
    // rotation rounds: sub-chains have at most k_eff segments (a step takes the warp's longest)
    const uint32_t max_rounds = (c.k_eff + G - 1) / G;
    // Shorter side (forward passes of shapes that hold at most 36 segments, and 4 x 12, where a
    // sub-chain can be longer than half the path): turning the complement of the sub-chain, [right, N)
    // and [0, left), by -theta about the same chord gives the moved path up to one rotation of
    // the whole path, and the weights see only curvatures, which that rotation leaves alone.
    // The chain then lives in a frame that turns with it. The sub-chain's chord is d minus the
    // complement's, d = the sum of l_s t_s over the whole path in that frame: carried through
    // every complement move (d <- R(-theta) d) and re-summed from the state every 16 steps, so
    // that its rounding cannot build up over a long chain. (The 4 x 16 shape, N = 37..64, is
    // left out: it gained 2 % at N = 48 and its code lost 5 % at N = 64, where no sub-chain is
    // longer than half the path; 4 x 12 took N = 37..48 from it, +5-10 % with the shorter side
    // over without.) The incremental form turns the same side, so that it follows
    // the full recompute's trajectory. Shapes of 4 or fewer segments per lane on more than one
    // lane are left out too: at their 64-register budget the second code path spilled (4 x 4,
    // N = 13..16, measured 5-25 % slower).
    constexpr bool CMPL = MODE == kModeForward && !SHIFT && G < 32 && (G * SPL <= 36 || (G == 4 && SPL == 12)) &&
                          (G == 1 || SPL > 4);
    const bool cmpl_on = CMPL && N < 2 * c.k_eff;
    float dX = 0.f, dY = 0.f, dZ = 0.f;
    float lse_m = 0.f, lse_s = 0.f, lse_c = 0.f;  // exact form: running max (float) and Kahan sum
    unsigned long long lse_t = 0;                   // fixed form: running max as a path total
    uint32_t valid = 0, failed = 0, clamped = 0;
    float acc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    // incremental form: the current path's integer total and whether a NaN curvature was met
    // since the last full recompute
    unsigned long long inc_tot = 0;
    bool inc_bad = false;
    uint32_t inc_since_full = 0;   // incremental steps since the last full recompute
    // tangent of segment s (any lane's) and the fixed-point term of the curvature between two
    // tangents, with its interpolation correction rounded on its own
    auto tan_at = [&](uint32_t s, float &x, float &y, float &z) {
        Lay::get(st.t, Lay::slot(s / SPL, s % SPL, qb), x, y, z);
    };
    auto term = [&](float ax, float ay, float az, float bx, float by, float bz, bool &nan) -> uint32_t {
        const float dx = bx - ax, dy = by - ay, dz = bz - az;
        int32_t L;
        uint32_t unused = 0;
        const float frac = bin_of<CLAMP>(fmaf(dx, dx, fmaf(dy, dy, dz * dz)), kc, false, unused, L);
        const float2 e = s_tab[L];
        const float cor = frac * e.y;
        nan |= isnan(cor);   // a NaN curvature or a steep bin's NaN slope
        return __float_as_uint(e.x) + (uint32_t)__float2int_rn(cor * kc.fscale);
    };

    const SmemLoad<G, SPL, SHIFT, ORDERED> load_smem{st, qb, j, N, &c, kc.kscale, inv_ks};
    const ShflNext<G> next_smem{};
    // adjoint with the fixed-point table: the reference as a path total, and the tangents and weight of the
    // step whose receiver gradient this lane works out
    const long long adj_ref = ADJ && FIX ? llrint((ma.ref_log10 - kc.lw_offset) * (double)kc.fscale) : 0;
    [[maybe_unused]] float adj_w = 0.f, adj_t[9] = {};
    // The chain's running log-sum-exp (fixed-point form). It starts from the total 0 with an empty
    // sum: the first path's total is its new maximum.
    auto lse_add = [&](unsigned long long tot) {
        // exact integer difference: narrow totals stay below 2^31, wide ones are 64-bit
        const float dt = kc.wide ? (float)(long long)(tot - lse_t) : (float)(int32_t)((uint32_t)tot - (uint32_t)lse_t);
        const float x = dt * kc.l2s;
        float term = 1.f;
        if (x > 0.f) {
            const float f = ex2_approx(-x);
            lse_s *= f;
            lse_c *= f;
            lse_t = tot;
        } else {
            term = ex2_approx(x);
        }
        kahan_add(lse_s, lse_c, term);
    };
    // Forward passes of groups of 4 lanes and more (GROUPED: in the batched kernels only some shapes, batch_grouped) sum the
    // lanes' shares of four path totals together:
    // exchanges after every second and fourth weighted step leave one step's shares in each lane (step
    // j mod 4), the other levels add as a butterfly does, and each lane runs the log-sum-exp of
    // its own steps: 5 shuffles for four paths of 16 lanes instead of 16, and one log-sum-exp
    // update for four paths instead of one for each in every lane.
    constexpr bool BATCH = FIX && MODE == kModeForward && !INCR && G >= 4 && GROUPED;
    constexpr int LS = Lanes<G>::STRIDE;
    uint32_t even = 0, flags = 0;       // the even step's share; steps 0..3 met (bits 0..3) and weighed (bits 4..7)
    unsigned long long pair01 = 0;
    // the lower lane (by bit `up` of j) keeps x0 and sends x1, the upper one the other way round
    auto exchange = [&](unsigned long long x0, unsigned long long x1, bool up, int off) -> unsigned long long {
        if (kc.wide) return (up ? x1 : x0) + __shfl_xor_sync(FULL, up ? x0 : x1, off);
        return (uint32_t)(up ? x1 : x0) + __shfl_xor_sync(FULL, (uint32_t)(up ? x0 : x1), off);
    };
    auto exchange32 = [&](uint32_t x0, uint32_t x1, bool up, int off) -> unsigned long long {
        const uint32_t got = __shfl_xor_sync(FULL, up ? x0 : x1, off);
        return kc.wide ? (unsigned long long)(up ? x1 : x0) + got : (unsigned long long)((up ? x1 : x0) + got);
    };
    auto batch_step = [&](uint32_t slot, bool end, uint32_t part) {
        if (slot & 1u) {
            const unsigned long long two = exchange32(even, part, j & 1u, LS);
            if (slot == 1u) pair01 = two;
            if (slot == 3u || end) {
                unsigned long long tot = exchange(pair01, slot == 3u ? two : 0ull, j & 2u, 2 * LS);
                if (kc.wide) {
#pragma unroll
                    for (int o = 4; o < G; o <<= 1) tot += __shfl_xor_sync(FULL, tot, o * LS);
                } else {
                    uint32_t t32 = (uint32_t)tot;
#pragma unroll
                    for (int o = 4; o < G; o <<= 1) t32 += __shfl_xor_sync(FULL, t32, o * LS);
                    tot = t32;
                }
                if ((flags >> (4u + (j & 3u))) & 1u) lse_add(tot);
                valid += __popc(flags >> 4);
                failed += __popc(flags & 15u) - __popc(flags >> 4);
                flags = 0;
            }
        } else {
            even = part;
        }
    };
    auto no_bins = [](uint32_t, int32_t) {};
    // export: this lane's unit tangents, each in the place of its segment's end point
    // (export_positions_kernel makes the points of them, every path at once: in this loop, one chain's steps
    // wait for one another)
    auto export_tangents = [&](uint32_t wstep) {
        float *dst = ma.exp_pos + ((size_t)chain * c.steps + wstep) * 3 * (size_t)(N + 1);
#pragma unroll
        for (int m = 0; m < SPL; ++m) {
            const uint32_t s = j * SPL + m;
            if (s < N) {
                const float4 v = load_rec(j, m);
                dst[3 * (s + 1)] = v.x;
                dst[3 * (s + 1) + 1] = v.y;
                dst[3 * (s + 1) + 2] = v.z;
            }
        }
    };

    for (uint32_t base = 0; base < total; base += G) {
        const dev::Proposal pr = dev::draw_step(c.seed, c.experiment, gchain, base + j, N, c.k_eff, c.max_angle);
        // sin = 2 s c and 1 - cos = 2 s^2 of the turn (half angle s, c); k and left in one word, so
        // that three shuffles broadcast a proposal
        float psn, pcs;
        dev::sincos_half(pr.angle, psn, pcs);
        const float psth = 2.f * psn * pcs, pomc = 2.f * psn * psn;
        const uint32_t pkl = pr.k | (pr.left << 8);   // k <= 64, left < 1024
        const uint32_t nstep = min((uint32_t)G, total - base);
        for (uint32_t jj = 0; jj < nstep; ++jj) {
            const uint32_t kl = Lanes<G>::from(pkl, jj, qb);
            const uint32_t k = kl & 255u, left = kl >> 8;
            const float sth0 = Lanes<G>::from(psth, jj, qb);
            const float omc = Lanes<G>::from(pomc, jj, qb);
            const uint32_t right = left + k;
            // the segments this chain turns: the sub-chain, or its complement where that is
            // shorter, on the steps where that takes two or more rounds off the warp's rotation
            // (a step that turns complements pays for the wrap and for carrying d: saving one
            // round of three, as at N = 13 and 14 on 4 x 4, measured slower)
            bool cm = false, use_c = false;
            uint32_t kmax;   // the longest turned side among the warp's chains
            if constexpr (CMPL) {
                if (cmpl_on && ((base + jj) & 15u) == 0u) {
                    dX = 0.f; dY = 0.f; dZ = 0.f;
#pragma unroll
                    for (int m = 0; m < SPL; ++m) {   // padding slots hold zero tangents
                        float x, y, z;
                        Lay::get(st.t, Lay::slot(j, m, qb), x, y, z);
                        const float l = st.l[j * SPL + m];
                        dX = fmaf(l, x, dX);
                        dY = fmaf(l, y, dY);
                        dZ = fmaf(l, z, dZ);
                    }
                    group_sum3<G>(dX, dY, dZ, j, qb);
                }
                // whole-warp reductions: every chain of a warp belongs to one experiment (a CTA
                // runs one experiment's work item at a time), so cmpl_on is the same in every lane
                kmax = __reduce_max_sync(FULL, k);
                if (cmpl_on) {
                    const uint32_t kc = __reduce_max_sync(FULL, min(k, N - k));
                    use_c = (kc + G - 1) / G + 2 <= (kmax + G - 1) / G;   // the same for the whole warp
                    if (use_c) {
                        cm = N - k < k;
                        kmax = kc;
                    }
                }
            } else {
                kmax = k;
#pragma unroll
                for (int o = 1; o < Lanes<G>::CPW; o <<= 1)   // over the warp's chains
                    kmax = max(kmax, __shfl_xor_sync(FULL, kmax, G == 4 ? o : o * G));
            }
            const uint32_t rounds = min((kmax + G - 1) / G, max_rounds);
            // incremental form: the two end curvatures before the rotation (kappa_{left-1} and
            // kappa_{right-1}; left >= 1 and right <= N-1, so all four tangents exist)
            bool incr_now = false;
            uint32_t t_old = 0;
            float e0x = 0.f, e0y = 0.f, e0z = 0.f, e3x = 0.f, e3y = 0.f, e3z = 0.f;
            if constexpr (INCR) {
                incr_now = base + jj > c.burn_in && inc_since_full + 1 < c.incr_resync;
                if (incr_now) {
                    float a1x, a1y, a1z, b0x, b0y, b0z;
                    tan_at(left - 1, e0x, e0y, e0z);
                    tan_at(left, a1x, a1y, a1z);
                    tan_at(right - 1, b0x, b0y, b0z);
                    tan_at(right, e3x, e3y, e3z);
                    t_old = term(e0x, e0y, e0z, a1x, a1y, a1z, inc_bad) + term(b0x, b0y, b0z, e3x, e3y, e3z, inc_bad);
                }
            }
            // chord x_right - x_left = sum of l_s t_s over the k segments left .. right-1
            // (k <= N - 2 < G * SPL, so a sub-chain never needs more than SPL rounds; a
            // complement turned instead is shorter than its sub-chain)
            constexpr int R = (kMaxSubChain + G - 1) / G < SPL ? (kMaxSubChain + G - 1) / G : SPL;
            // more than 4 rounds (8-lane groups) under the 64-register budget of 1024-thread
            // CTAs (SPL < 16): the rotation pass reloads its tangents instead of keeping every
            // round's in registers (measured: no spills, N <= 64 up to 27 % faster)
            constexpr bool RELOAD = R > 4 && (SPL < 16 || G < 8);
            constexpr int RK = RELOAD ? 1 : R;
            // PLANES shapes turn the segments of two rounds at once with the packed instructions (16
            // for two segments instead of 32; the same roundings). Their 4-lane shapes keep the
            // chord pass's slots, two to a register, instead of finding each again. Together
            // N = 66 +11 % over PLANES without them, N = 24 on one lane +8 %, and 13 % off a burn-in step.
            // Under the 64 registers of the 4-lane shapes below 12 segments per lane the pairs spill
            // (N = 16..36 -10 to -25 %), and the Rodrigues form packed lost 6-18 % at 8 lanes.
            constexpr bool PACK_ROT = Lay::KIND == kPlanes;
            constexpr bool KEEP_SLOTS = PACK_ROT && G == 4;
            static_assert(!PACK_ROT || RELOAD, "the packed rotation reads its tangents again");
            // The move: the chord of the turned segments, the axis, the rotation. WRAP: the warp
            // turns complements this step (the chains with cm), which wrap past segment N-1 to 0,
            // turn by -theta and carry d; a step that turns none runs the plain code.
            auto turn = [&](auto wrap_tag) {
                constexpr bool WRAP = decltype(wrap_tag)::value;
                const bool cmw = WRAP && cm;
                const uint32_t first = cmw ? right : left;
                const uint32_t cnt = cmw ? N - k : k;
                auto seg_of = [&](uint32_t idx) {
                    uint32_t s = first + idx;
                    if (WRAP && s >= N) s -= N;
                    return s;
                };
                float vx[RK], vy[RK], vz[RK];
                Slot va[RK];
                [[maybe_unused]] uint32_t slots2[(R + 1) / 2];   // KEEP_SLOTS: below 2^16 each
                float cx = 0.f, cy = 0.f, cz = 0.f;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    if (r > 0 && (uint32_t)r >= rounds) break;
                    const uint32_t idx = j + r * G;
                    const uint32_t s = seg_of(idx);
                    const int ri = RELOAD ? 0 : r;
                    va[ri] = Lay::slot(s / SPL, s % SPL, qb);
                    if constexpr (KEEP_SLOTS) slots2[r / 2] = (r & 1) ? slots2[r / 2] + (va[0].a << 16) : va[0].a;
                    if (WRAP ? idx < cnt : s < right) {
                        Lay::get(st.t, va[ri], vx[ri], vy[ri], vz[ri]);
                        const float l = st.l[s];
                        cx = fmaf(l, vx[ri], cx);
                        cy = fmaf(l, vy[ri], cy);
                        cz = fmaf(l, vz[ri], cz);
                    }
                }
                if constexpr (G == 32) {
                    int ix = __float2int_rn(cx * chord_scale);
                    int iy = __float2int_rn(cy * chord_scale);
                    int iz = __float2int_rn(cz * chord_scale);
                    ix = __reduce_add_sync(FULL, ix);
                    iy = __reduce_add_sync(FULL, iy);
                    iz = __reduce_add_sync(FULL, iz);
                    cx = (float)ix;
                    cy = (float)iy;
                    cz = (float)iz;
                } else {
                    group_sum3<G>(cx, cy, cz, j, qb);
                }
                if (cmw) { cx = dX - cx; cy = dY - cy; cz = dZ - cz; }   // the sub-chain's chord
                // Rodrigues by +theta about the unit chord a -- the rotation the reference's
                // quaternion sandwich q^-1 p q applies with its product convention:
                // v cos + (a x v) sin + a (a.v)(1 - cos)
                const float inv = rsqrtf(fmaf(cx, cx, fmaf(cy, cy, cz * cz)));
                const float ax = cx * inv, ay = cy * inv, az = cz * inv;
                const float sth = cmw ? -sth0 : sth0;
                // Groups of 1 or 4 lanes (up to 32 or 8 rounds): the rotation as v + M v with
                // M = R - I = sin(theta) [a]x + (1 - cos(theta)) (a a^T - I), built once per step,
                // 9 FMAs per segment against 19 for the Rodrigues form (the correction is added
                // to v, so it rounds like the Rodrigues terms do). Measured +4.6-5.5 % at
                // N = 8..24 and +1-2 % at N = 32..96; with 8-lane groups (4 rounds) 1.9 % slower
                // at N = 128, so those keep the Rodrigues form.
                [[maybe_unused]] constexpr bool RMAT = G <= 4;
                if constexpr (PACK_ROT) {
                    const F2 ax2 = pack2(ax, ax), ay2 = pack2(ay, ay), az2 = pack2(az, az);
                    const F2 omc2 = pack2(omc, omc), nomc2 = pack2(-omc, -omc), sth2 = pack2(sth, sth), nsth2 = pack2(-sth, -sth);
                    const F2 oax = mul2(omc2, ax2), oay = mul2(omc2, ay2), oaz = mul2(omc2, az2);
                    const F2 m00 = fma2(oax, ax2, nomc2), m11 = fma2(oay, ay2, nomc2), m22 = fma2(oaz, az2, nomc2);
                    const F2 m01 = fma2(oax, ay2, mul2(nsth2, az2)), m10 = fma2(oax, ay2, mul2(sth2, az2));
                    const F2 m02 = fma2(oax, az2, mul2(sth2, ay2)), m20 = fma2(oax, az2, mul2(nsth2, ay2));
                    const F2 m12 = fma2(oay, az2, mul2(nsth2, ax2)), m21 = fma2(oay, az2, mul2(sth2, ax2));
                    const F2 renorm2 = pack2(renorm, renorm), c15 = pack2(1.5f, 1.5f);
                    __syncwarp();
#pragma unroll
                    for (int r = 0; r < R; r += 2) {
                        if (r > 0 && (uint32_t)r >= rounds) break;
                        const uint32_t i0 = j + r * G, i1 = i0 + G;
                        const uint32_t s0 = seg_of(i0), s1 = seg_of(i1);
                        const bool p0 = WRAP ? i0 < cnt : s0 < right;
                        const bool p1 = r + 1 < R && (WRAP ? i1 < cnt : s1 < right);
                        const Slot a0 = KEEP_SLOTS ? Slot{slots2[r / 2] & 0xFFFFu, 0} : Lay::slot(s0 / SPL, s0 % SPL, qb);
                        const Slot a1 = KEEP_SLOTS ? Slot{slots2[r / 2] >> 16, 0} : Lay::slot(s1 / SPL, s1 % SPL, qb);
                        float x0 = 0.f, y0 = 0.f, z0 = 0.f, x1 = 0.f, y1 = 0.f, z1 = 0.f;
                        if (p0) Lay::get(st.t, a0, x0, y0, z0);
                        if (p1) Lay::get(st.t, a1, x1, y1, z1);
                        const F2 x = pack2(x0, x1), y = pack2(y0, y1), z = pack2(z0, z1);
                        const F2 nx = fma2(m00, x, fma2(m01, y, fma2(m02, z, x)));
                        const F2 ny = fma2(m10, x, fma2(m11, y, fma2(m12, z, y)));
                        const F2 nz = fma2(m20, x, fma2(m21, y, fma2(m22, z, z)));
                        const F2 h = fma2(renorm2, fma2(nx, nx, fma2(ny, ny, mul2(nz, nz))), c15);
                        const F2 rx = mul2(nx, h), ry = mul2(ny, h), rz = mul2(nz, h);
                        if (p0) Lay::put(st.t, a0, rx.lo(), ry.lo(), rz.lo());
                        if (p1) Lay::put(st.t, a1, rx.hi(), ry.hi(), rz.hi());
                    }
                } else {
                    [[maybe_unused]] float m00 = 0.f, m01 = 0.f, m02 = 0.f, m10 = 0.f, m11 = 0.f, m12 = 0.f, m20 = 0.f, m21 = 0.f, m22 = 0.f;
                    if constexpr (RMAT) {
                        const float oax = omc * ax, oay = omc * ay, oaz = omc * az;
                        const float sax = sth * ax, say = sth * ay, saz = sth * az;
                        m00 = fmaf(oax, ax, -omc);
                        m11 = fmaf(oay, ay, -omc);
                        m22 = fmaf(oaz, az, -omc);
                        m01 = fmaf(oax, ay, -saz);
                        m10 = fmaf(oax, ay, saz);
                        m02 = fmaf(oax, az, say);
                        m20 = fmaf(oax, az, -say);
                        m12 = fmaf(oay, az, -sax);
                        m21 = fmaf(oay, az, sax);
                    }
                    __syncwarp();
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        if (r > 0 && (uint32_t)r >= rounds) break;
                        const uint32_t idx = j + r * G;
                        const uint32_t s = seg_of(idx);
                        const int ri = RELOAD ? 0 : r;
                        if (RELOAD) va[0] = Lay::slot(s / SPL, s % SPL, qb);
                        if (WRAP ? idx < cnt : s < right) {
                            if (RELOAD) Lay::get(st.t, va[0], vx[0], vy[0], vz[0]);
                            const float x = vx[ri], y = vy[ri], z = vz[ri];
                            float nx, ny, nz;
                            if constexpr (RMAT) {
                                nx = fmaf(m00, x, fmaf(m01, y, fmaf(m02, z, x)));
                                ny = fmaf(m10, x, fmaf(m11, y, fmaf(m12, z, y)));
                                nz = fmaf(m20, x, fmaf(m21, y, fmaf(m22, z, z)));
                            } else {
                                const float crx = ay * z - az * y, cry = az * x - ax * z, crz = ax * y - ay * x;
                                const float ad = (ax * x + ay * y + az * z) * omc;
                                nx = fmaf(ax, ad, fmaf(sth, crx, fmaf(-omc, x, x)));
                                ny = fmaf(ay, ad, fmaf(sth, cry, fmaf(-omc, y, y)));
                                nz = fmaf(az, ad, fmaf(sth, crz, fmaf(-omc, z, z)));
                            }
                            const float h = fmaf(renorm, fmaf(nx, nx, fmaf(ny, ny, nz * nz)), 1.5f);
                            Lay::put(st.t, va[ri], nx * h, ny * h, nz * h);
                        }
                    }
                }
                if constexpr (WRAP) {
                    // the whole path's chord turns with the complement (selected, not branched)
                    const float crx = ay * dZ - az * dY, cry = az * dX - ax * dZ, crz = ax * dY - ay * dX;
                    const float ad = (ax * dX + ay * dY + az * dZ) * omc;
                    const float nX = fmaf(ax, ad, fmaf(sth, crx, fmaf(-omc, dX, dX)));
                    const float nY = fmaf(ay, ad, fmaf(sth, cry, fmaf(-omc, dY, dY)));
                    const float nZ = fmaf(az, ad, fmaf(sth, crz, fmaf(-omc, dZ, dZ)));
                    dX = cm ? nX : dX;
                    dY = cm ? nY : dY;
                    dZ = cm ? nZ : dZ;
                }
            };
            if constexpr (CMPL) {
                if (use_c) turn(BoolTag<true>{});
                else turn(BoolTag<false>{});
            } else {
                turn(BoolTag<false>{});
            }
            __syncwarp();
            const uint32_t step = base + jj;
            if (step < c.burn_in) continue;
            const uint32_t wstep = step - c.burn_in;
            const bool active = wstep < steps_c;

            if constexpr (ADJ && FIX) {
                // The path's total as the forward pass takes it, and beside each table entry the derivatives of its
                // log in one 16-byte load: two packed operations a segment, where the exact blend takes a log2, a
                // compensated sum, a reciprocal and two blends. Image replay (48 pixels, N = 512, 2^17 paths
                // each): 1030 -> 504 warp-instructions per path, 6.76 -> 4.54 ms; the shared-memory and L1 pipe
                // then binds (92 % of its wavefronts).
                uint32_t isum = 0;
                float c0 = 0.f, c1 = 0.f;
                F2 g = pack2(0.f, 0.f);
                auto entry = [&](int32_t L, float frac, bool valid, float &cc) {
                    const float2 en = s_tab[L];
                    const float4 dv = __ldg(ma.dtab + L);
                    isum += valid ? __float_as_uint(en.x) : 0u;
                    const float c2 = fmaf(frac, en.y, cc);
                    cc = valid ? c2 : cc;
                    const F2 gn = add2(g, fma2(pack2(frac, frac), pack2(dv.z, dv.w), pack2(dv.x, dv.y)));
                    g.v = valid ? gn.v : g.v;
                };
                auto seg1 = [&](uint32_t, float qq, bool valid) {
                    int32_t L;
                    const float frac = bin_of<false>(qq, kc, valid, clamped, L);
                    entry(L, frac, valid, c0);
                };
                auto seg2 = [&](uint32_t, uint32_t, F2 qq, bool v0, bool v1) {
                    int32_t L0, L1;
                    const F2 f = bins_of(qq, kc, L0, L1);
                    entry(L0, f.lo(), v0, c0);
                    entry(L1, f.hi(), v1, c1);
                };
                if (N == (uint32_t)(G * SPL))
                    for_curvatures<G, SPL, true>(j, N, load_smem, next_smem, seg2, seg1);
                else
                    for_curvatures<G, SPL, false>(j, N, load_smem, next_smem, seg2, seg1);
                const float csum = c0 + c1;
                const bool bad = ((__ballot_sync(FULL, isnan(csum)) >> qb) & Lanes<G>::MASK) != 0u;
                isum += (uint32_t)__float2int_rn(csum * kc.fscale);
                const unsigned long long tot =
                      kc.wide ? group_sum<G>((unsigned long long)isum) : (unsigned long long)group_sum<G>(isum);
                const bool use = active && !bad;
                const float wt = use ? ex2_approx((float)((long long)tot - adj_ref) * kc.l2s) : 0.f;
                if (use) {
                    acc[0] = fmaf(wt, g.lo(), acc[0]);
                    acc[1] = fmaf(wt, g.hi(), acc[1]);
                    if (j == 0) acc[5] += wt;
                }
                // the receiver's part: lane j keeps the last three tangents of the steps j mod G, and
                // every G steps all lanes work out theirs together
                if (wstep % G == j) {
                    adj_w = wt;
                    Lay::get(st.t, Lay::slot((N - 3) / SPL, (N - 3) % SPL, qb), adj_t[0], adj_t[1], adj_t[2]);
                    Lay::get(st.t, Lay::slot((N - 2) / SPL, (N - 2) % SPL, qb), adj_t[3], adj_t[4], adj_t[5]);
                    Lay::get(st.t, Lay::slot((N - 1) / SPL, (N - 1) % SPL, qb), adj_t[6], adj_t[7], adj_t[8]);
                }
                if (wstep % G == G - 1 || wstep + 1u == c.steps) {
                    if (adj_w > 0.f) {
                        float t3[3], t2[3], t1[3], g3[3];
                        for (int i = 0; i < 3; ++i) {
                            t3[i] = adj_t[i] * inv_ks;
                            t2[i] = adj_t[3 + i] * inv_ks;
                            t1[i] = adj_t[6 + i] * inv_ks;
                        }
                        receiver_grad(t3, t2, t1, st.l[N - 2], ma.lin, kc, c.inv_ds, g3);
                        for (int i = 0; i < 3; ++i) acc[2 + i] += adj_w * g3[i];
                    }
                    adj_w = 0.f;
                }
                continue;
            }
            if (FIX) {
                bool bad = false;
                unsigned long long tot = 0;
                bool need_full = true;
                if constexpr (INCR) {
                    if (incr_now) {
                        // the two end curvatures after the rotation; the interior ones keep their terms
                        // (a turned complement moved the outer tangents of the two joints instead)
                        float a1x, a1y, a1z, b0x, b0y, b0z;
                        if (cm) {
                            tan_at(left - 1, e0x, e0y, e0z);
                            tan_at(right, e3x, e3y, e3z);
                        }
                        tan_at(left, a1x, a1y, a1z);
                        tan_at(right - 1, b0x, b0y, b0z);
                        const uint32_t t_new =
                              term(e0x, e0y, e0z, a1x, a1y, a1z, inc_bad) + term(b0x, b0y, b0z, e3x, e3y, e3z, inc_bad);
                        inc_tot += (unsigned long long)(long long)(int32_t)(t_new - t_old);
                        need_full = inc_bad;
                    }
                }
                // one decision per warp: the full recompute shuffles across the whole warp, and
                // every chain of the warp then stays on the same resync schedule
                if (INCR && !__any_sync(FULL, need_full)) {
                    tot = inc_tot;
                    ++inc_since_full;
                } else {
                    bool nan;
                    uint32_t part = path_fixed<G, SPL, CLAMP, TAB_GLOBAL>(j, N, s_tab, kc, load_smem, next_smem, nan, clamped);
                    bad = ((__ballot_sync(FULL, nan) >> qb) & Lanes<G>::MASK) != 0u;
                    // a NaN slope marks a steep bin, where the secant would err by more than
                    // 1e-7: weigh such paths (rare) with the exact blend through the linear
                    // table; only a NaN curvature leaves a path invalid
                    if constexpr (STEEP) {
                        if (__any_sync(FULL, bad)) {
                            const double wx = steep_fallback<G, SPL, CLAMP, ORDERED>(st, qb, j, N, ma.lin, kc);
                            if (bad && !isnan(wx)) {
                                bad = false;
                                // the total in shares of at most 32 bits, one per lane
                                const unsigned long long t =
                                      (unsigned long long)llrint(fmax(0.0, (wx - kc.lw_offset) * (double)kc.fscale));
                                part = (uint32_t)(t / G) + (j < (uint32_t)(t % G) ? 1u : 0u);
                            }
                        }
                    }
                    if constexpr (BATCH) {
                        const uint32_t slot = wstep & 3u;
                        flags |= active ? (bad ? 1u : 17u) << slot : 0u;
                        const bool end = wstep + 1u == c.steps;
                        batch_step(slot, end, part);
                        if (end && !(slot & 1u)) batch_step(slot + 1u, true, 0u);
                        continue;
                    }
                    tot = kc.wide ? group_sum<G>((unsigned long long)part) : (unsigned long long)group_sum<G>(part);
                    inc_tot = tot;
                    inc_bad = bad;
                    inc_since_full = 0;
                }
                if (MODE == kModeExport) {
                    const double w = bad ? NAN : kc.lw_offset + (double)tot * kc.inv_scale;
                    if (active) {
                        const size_t pidx = (size_t)chain * c.steps + wstep;
                        if (j == 0) ma.exp_w[pidx] = isnan(w) ? NAN : w + (N - 1) * ma.log10_abs;
                    }
                }
                if (MODE == kModeExport && ma.exp_pos && active) export_tangents(wstep);
                if (!active) continue;
                if (bad) {
                    ++failed;
                    continue;
                }
                lse_add(tot);
                ++valid;
                continue;
            }

            double w;
            if (ADJ) {
                // log10 weight and d/d(mu_s), d/d(eps) of this lane's segments (exact blend): the
                // blend from the staged linear table, the derivative blends from one 16-byte load
                float s = 0.f, cc = 0.f, gmu = 0.f, geps = 0.f;
                auto adj_seg = [&](uint32_t, float qq, bool valid) {
                    float r = sqrt_approx(qq) + kc.roff;   // scaled tangents: the root is the bin index
                    if (r < 0.f) r = 0.f;
                    if (r > kc.rmax) r = kc.rmax;
                    // floor(r) by a round-down add, as bin_of takes it (no float/int conversions
                    // on the MUFU pipe, which the blend's log2 and reciprocal already load;
                    // measured 1.8 % off the differentiation configuration's adjoint call)
                    const float fl = __fadd_rd(r, 8388608.0f);
                    const int32_t L = (int32_t)min(__float_as_uint(fl) - 0x4B000000u, (uint32_t)kc.bins - 1u);
                    const float d = (r - (fl - 8388608.0f)) * kc.step;
                    const float2 e = s_tab[L];
                    const float4 dv = __ldg(ma.dtab + L);
                    const float v = fmaf(d, e.y, e.x);
                    kahan_add(s, cc, valid ? __log2f(v) * kLog10_2 : 0.0f);
                    const float iv = __fdividef(1.0f, v);
                    gmu += valid ? fmaf(d, dv.y, dv.x) * iv : 0.0f;
                    geps += valid ? fmaf(d, dv.w, dv.z) * iv : 0.0f;
                };
                // a chain that fills its group's slots walks them with validity known at compile
                // time (every curvature but the group's last boundary), as the forward recompute does
                auto adj_seg2 = [&](uint32_t i0, uint32_t i1, F2 qq, bool v0, bool v1) {
                    adj_seg(i0, qq.lo(), v0);
                    adj_seg(i1, qq.hi(), v1);
                };
                if (N == (uint32_t)(G * SPL))
                    for_curvatures<G, SPL, true>(j, N, load_smem, next_smem, adj_seg2, adj_seg);
                else
                    for_curvatures<G, SPL, false>(j, N, load_smem, next_smem, adj_seg2, adj_seg);
                float hi = s, lo = -cc;
                group_sum_pair<G>(hi, lo);
                w = (double)hi + (double)lo;
                float g3[3] = {0.f, 0.f, 0.f};
                if (j == 0) {
                    const float4 v3 = load_rec((N - 3) / SPL, (N - 3) % SPL);
                    const float4 v2 = load_rec((N - 2) / SPL, (N - 2) % SPL);
                    const float4 v1 = load_rec((N - 1) / SPL, (N - 1) % SPL);
                    const float t3[3] = {v3.x, v3.y, v3.z}, t2[3] = {v2.x, v2.y, v2.z}, t1[3] = {v1.x, v1.y, v1.z};
                    receiver_grad(t3, t2, t1, v2.w, s_tab, kc, c.inv_ds, g3);
                }
                if (active && !isnan(w)) {
                    const float wt = exp2f((float)(w - ma.ref_log10) * kLog2_10);
                    acc[0] += wt * gmu * kInvLn10;
                    acc[1] += wt * geps * kInvLn10;
                    acc[2] += wt * g3[0];
                    acc[3] += wt * g3[1];
                    acc[4] += wt * g3[2];
                    if (j == 0) acc[5] += wt;
                }
            } else {
                // segments in order: the rounding of the blend's float terms follows the order
                w = path_log10<G, SPL, true, CLAMP, TAB_GLOBAL, false>(j, N, s_tab, kc, load_smem, next_smem, no_bins, clamped);
            }
            if (MODE == kModeExport && active) {
                if (ma.exp_pos) export_tangents(wstep);   // a weights-only replay passes no buffer
                if (j == 0) ma.exp_w[(size_t)chain * c.steps + wstep] = isnan(w) ? NAN : w + (N - 1) * ma.log10_abs;
            }
            if (!active) continue;
            if (isnan(w)) {
                ++failed;
                continue;
            }
            const float hi = (float)w;
            const float lo = (float)(w - (double)hi);
            if (valid == 0) {
                lse_m = hi;
                lse_s = exp2f(lo * kLog2_10);
                lse_c = 0.f;
                valid = 1;
            } else {
                const float x = (hi - lse_m) + lo;
                float term;
                if (x > 0.f) {
                    const float f = exp2f((lse_m - hi) * kLog2_10);
                    lse_s *= f;
                    lse_c *= f;
                    lse_m = hi;
                    term = exp2f(lo * kLog2_10);
                } else {
                    term = exp2f(x * kLog2_10);
                }
                kahan_add(lse_s, lse_c, term);
                ++valid;
            }
        }
    }
    clamped = group_sum<G>(clamped);
    if (ADJ) {
        if (FIX) {   // the fixed-point form leaves the natural log's factor to the end
            acc[0] *= kInvLn10;
            acc[1] *= kInvLn10;
        }
#pragma unroll
        for (int i = 0; i < 6; ++i) acc[i] = group_sum<G>(acc[i]);
        if (j == 0 && real_chain)
            for (int i = 0; i < 6; ++i) ma.grad[(size_t)chain * 6 + i] = (double)acc[i];
    }
    double chain_log10 = -INFINITY;
    if (valid) {
        const double head = FIX ? kc.lw_offset + (double)lse_t * kc.inv_scale : (double)lse_m;
        chain_log10 = head + log10((double)lse_s - (double)lse_c);   // -inf in a lane that met no path
    }
    if constexpr (BATCH) {
        // the chain's four interleaved sums, lanes j mod 4
        double m = chain_log10;
        m = fmax(m, __shfl_xor_sync(FULL, m, LS));
        m = fmax(m, __shfl_xor_sync(FULL, m, 2 * LS));
        double x = chain_log10 > -INFINITY ? exp10(chain_log10 - m) : 0.0;
        x += __shfl_xor_sync(FULL, x, LS);
        x += __shfl_xor_sync(FULL, x, 2 * LS);
        chain_log10 = m > -INFINITY ? m + log10(x) : -INFINITY;
    }
    if (valid) chain_log10 += (double)(N - 1) * ma.log10_abs;
    if (j == 0 && real_chain && out) {
        ChainOut o;
        o.log10_sum = chain_log10;
        o.valid = valid;
        o.failed = failed;
        o.clamped = clamped;
        o.pad = 0;
        out[chain] = o;
    }
    return real_chain ? chain_log10 : -INFINITY;
}

CompConsts make_consts(float inv_ds, const LutMetaF &m, uint32_t n_segments, const LogFixed &lf)
{
    CompConsts k;
    k.kscale = inv_ds / m.step;
    k.roff = -m.min_k / m.step;
    k.rmax = (m.max_k - m.min_k) / m.step;
    k.rsnap = 1e-3f / m.step;
    k.step = m.step;
    k.bins = m.bins;
    k.lw_offset = (double)(n_segments - 1) * lf.c0;
    k.inv_scale = lf.inv_scale;
    k.fscale = lf.inv_scale > 0.0 ? (float)(1.0 / lf.inv_scale) : 0.0f;
    k.l2s = (float)(lf.inv_scale * 3.321928094887362);
    k.wide = lf.wide;
    return k;
}

// A table whose range covers every curvature unit tangents can produce, |t_{i+1}-t_i| <= 2
// (with margin for rounding), needs no clamping.
bool table_needs_clamp(const CompConsts &k) { return !(k.roff == 0.0f && k.rmax >= 2.0001f * k.kscale); }

}  // namespace
}  // namespace twisty
