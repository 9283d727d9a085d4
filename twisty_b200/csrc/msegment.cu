// msegment.cu -- independent-sample M-segment Monte Carlo on the device.
//
// The reference's other estimator, MSegmentPathGenerationMC (Experiments/ExperimentBase.cpp:
// 1246-1386): every path is a fresh random curve from the recursive bootstrapper
// (ResolveEvenNumberOfSegments, Twisty/PathGeneration.cpp:47-414) between the fixed points
// 0, 1, N-1, N, weighed like the Markov-chain paths; the estimate is the mean weight.
//
// One thread builds and weighs one path at a time. The arithmetic follows the reference's mix of float
// vectors and double scalars; the random draws come from Philox-4x32-10, counter (draw index,
// path id lo, path id hi, experiment ^ 'MSEG'), key = seed, one 32-bit output per float draw and
// two per double draw -- the reference's std::mt19937_64 stream is not reproduced (its
// threads' interleaving makes it unreproducible anyway). A placement the reference would
// abort on (spheres that do not intersect, a NaN extent) marks the path invalid.
//  * The recursion (centre point, then the left half, then the right half) walks the leaves of a
//    perfect binary tree: before leaf t come the centres of the spans that begin at it, the largest
//    first, so the walk needs no stack and every thread of a warp places the same span.
//  * The reference draws an angle phi = acos(1 - 2u) and uses its sine and cosine only, and the
//    largest u from cos(asin(a / r)): in double those are 1 - 2u, 2 sqrt(u (1 - u)) and
//    d / (2r), so a centre costs one sincospi, one cube root, one square root and one
//    division in FP64 where the angles took two arc functions, three of sine and cosine, a power and four divisions.
//  * Points go to a scratch column per thread, element by element side by side, so that a warp's
//    stores and loads are whole lines, and the thread that placed a path weighs it. (Before, each
//    path's points were 12-byte pieces of its own row in a 1 GB batch, read again by a weigher of its
//    own: N = 66, 2^21 paths 5.7 ms on the device against 4.2, N = 258, 2^19 paths 6.9 against 4.4.)
#include "kernels.h"
#include "device_common.cuh"
#include "comp_body.cuh"

namespace twisty {
namespace {

constexpr float kPiF = 3.141592653589793f;

struct F3 {
    float x, y, z;
};
__device__ __forceinline__ F3 operator+(F3 a, F3 b) { return F3{a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ F3 operator-(F3 a, F3 b) { return F3{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ F3 operator*(F3 a, float s) { return F3{a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ float fdot(F3 a, F3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ F3 fcross(F3 a, F3 b)
{
    return F3{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ float fmag(F3 a) { return sqrtf(fdot(a, a)); }
__device__ __forceinline__ F3 funit(F3 a) { return a * (1.0f / sqrtf(fdot(a, a))); }

// Uniform draws from a per-path Philox stream. Only the draw index changes between the draws of a path:
// the half of the first round and the quarter of the second that do not depend on it are kept.
struct Draws {
    uint32_t k0, k1, tag;
    uint32_t x0, x1, y2, y3;   // round 1: words 0 and 1; round 2: the products of word 0
    uint32_t n = 0;
    __device__ Draws(uint64_t seed, uint32_t path_lo, uint32_t path_hi, uint32_t t)
        : k0((uint32_t)seed), k1((uint32_t)(seed >> 32)), tag(t)
    {
        const uint64_t a = (uint64_t)0xCD9E8D57u * path_hi;
        x0 = (uint32_t)(a >> 32) ^ path_lo ^ k0;
        x1 = (uint32_t)a;
        const uint64_t b = (uint64_t)0xD2511F53u * x0;
        y2 = (uint32_t)(b >> 32);
        y3 = (uint32_t)b;
    }
    // the next word: word 0 of the block with counter (n, path lo, path hi, tag)
    __device__ __forceinline__ uint32_t word()
    {
        const uint32_t i = n++;
        uint32_t a = k0, b = k1;
        const uint64_t m = (uint64_t)0xD2511F53u * i;
        const uint32_t z2 = (uint32_t)(m >> 32) ^ tag ^ b, z3 = (uint32_t)m;
        a += 0x9E3779B9u;
        b += 0xBB67AE85u;
        const uint64_t w = (uint64_t)0xCD9E8D57u * z2;
        uint32_t c0 = (uint32_t)(w >> 32) ^ x1 ^ a, c1 = (uint32_t)w, c2 = y2 ^ z3 ^ b, c3 = y3;
#pragma unroll
        for (int r = 2; r < 10; ++r) {
            a += 0x9E3779B9u;
            b += 0xBB67AE85u;
            const uint64_t p = (uint64_t)0xD2511F53u * c0, q = (uint64_t)0xCD9E8D57u * c2;
            c0 = (uint32_t)(q >> 32) ^ c1 ^ a;
            c1 = (uint32_t)q;
            c2 = (uint32_t)(p >> 32) ^ c3 ^ b;
            c3 = (uint32_t)p;
        }
        return c0;
    }
    __device__ float uf(float a, float b) { return a + (float)(word() >> 8) * (1.0f / 16777216.0f) * (b - a); }
    __device__ double ud(double a, double b)
    {
        const uint64_t hi = word(), lo = word();
        const double u = (double)(((hi << 32) | lo) >> 11) * (1.0 / 9007199254740992.0);
        return a + u * (b - a);
    }
    __device__ int coin() { return (int)(word() & 1u); }
};

// The path's points: element e = 3 i + k of this thread's column.
struct PathPts {
    float *p;
    size_t pitch;   // threads of the launch
    __device__ F3 get(uint32_t i) const
    {
        const float *q = p + 3 * (size_t)i * pitch;
        return F3{q[0], q[pitch], q[2 * pitch]};
    }
    __device__ void set(uint32_t i, F3 v) const
    {
        float *q = p + 3 * (size_t)i * pitch;
        q[0] = v.x;
        q[pitch] = v.y;
        q[2 * pitch] = v.z;
    }
};

// RotateQuatByQuat / RotateVectorByQuaternion (Twisty/CurvePerturbUtils.cpp:91-127).
__device__ void quat_product(const float A[4], const float B[4], float r[4])
{
    const float t0 = A[0] * B[0] - A[1] * B[1] - A[2] * B[2] - A[3] * B[3];
    const float t1 = A[0] * B[1] + A[1] * B[0] - A[2] * B[3] + A[3] * B[2];
    const float t2 = A[0] * B[2] + A[1] * B[3] + A[2] * B[0] - A[3] * B[1];
    const float t3 = A[0] * B[3] - A[1] * B[2] + A[2] * B[1] + A[3] * B[0];
    r[0] = t0;
    r[1] = t1;
    r[2] = t2;
    r[3] = t3;
}

__device__ F3 rotate_by_quaternion(const float q[4], F3 v)
{
    float p[4] = {0.0f, v.x, v.y, v.z};
    const float qi[4] = {q[0], -q[1], -q[2], -q[3]};
    quat_product(p, q, p);
    quat_product(qi, p, p);
    return F3{p[1], p[2], p[3]};
}

__device__ void frame(F3 a, F3 b, F3 &xa, F3 &ya, F3 &za)
{
    za = funit(b - a);
    F3 r{1.0f, 0.0f, 0.0f};
    if (fabsf(fdot(za, r)) > 0.999f) r = F3{0.0f, 1.0f, 0.0f};
    xa = funit(fcross(za, r));
    ya = funit(fcross(za, xa));
}

// ResolveTwoSegments: the point between l and l+2. Returns false when the reference would throw.
__device__ bool resolve_two(const PathPts &P, uint32_t l, uint32_t r, double ds, Draws &g)
{
    const F3 a = P.get(l), b = P.get(r);
    const float d = fmag(b - a);
    if (fabs((2.0f * ds) - (double)d) < 0.001f) {
        P.set(l + 1, (a + b) * 0.5f);
        return true;
    }
    if ((2.0f * ds) < (double)d) return false;
    const float theta = g.uf(0.0f, 2.0f * kPiF);
    if (d < 0.001f) {
        const float phi = (float)acos(1.0 - 2.0 * (double)g.uf(0.0f, 1.0f));
        P.set(l + 1, a + F3{sinf(phi) * cosf(theta), sinf(phi) * sinf(theta), cosf(phi)} * (float)ds);
        return true;
    }
    const F3 mid = (a + b) * 0.5f;
    const F3 axis = funit(b - a);
    F3 helper{1.0f, 0.0f, 0.0f};
    if ((double)fabsf(fdot(axis, helper)) >= 0.99) helper = F3{0.0f, 1.0f, 0.0f};
    const F3 normal = funit(fcross(axis, helper));
    const float half = d * 0.5f;
    float off = 0.0f;
    if (ds > (double)half) off = (float)sqrt((ds * ds) - (double)(half * half));
    const F3 pt = mid + normal * off;
    const float s = sinf(theta / 2.0f);
    const float q[4] = {cosf(theta / 2.0f), axis.x * s, axis.y * s, axis.z * s};
    P.set(l + 1, rotate_by_quaternion(q, pt - a) + a);
    return true;
}

// ResolveThreeSegments: the two points between l and l+3.
__device__ __noinline__ bool resolve_three(const PathPts &P, uint32_t l, uint32_t r, double ds, Draws &g)
{
    const F3 a = P.get(l), b = P.get(r);
    const float d = fmag(b - a);
    if (fabs((3.0f * ds) - (double)d) < 0.001f) {
        P.set(l + 1, a + (b - a) * (1.0f / 3.0f));
        return resolve_two(P, l + 1, r, ds, g);
    }
    if ((3.0f * ds) < (double)d) return false;
    const float theta = g.uf(0.0f, 2.0f * kPiF);
    if (d < 0.001f) {
        const float phi = (float)acos(1.0 - 2.0 * (double)g.uf(0.0f, 1.0f));
        P.set(l + 1, a + F3{sinf(phi) * cosf(theta), sinf(phi) * sinf(theta), cosf(phi)} * (float)ds);
        return resolve_two(P, l + 1, r, ds, g);
    }
    F3 xa, ya, za;
    frame(a, b, xa, ya, za);
    const double d2 = (double)(d * d);
    const double r1 = ds, r1s = r1 * r1;
    const double r2 = 2.0f * ds, r2s = r2 * r2;
    double extent;
    if (((double)d + r1) < r2) {
        extent = kPiF;
    } else {
        const double h = 0.5 + (r1s - r2s) / (2.0 * d2);
        double aa = 0.0;
        if (fabs(r1s - (h * h * d2)) >= 0.001) aa = sqrt(r1s - (h * h * d2));
        extent = (h * d < 0.0) ? (double)kPiF - asin(aa / r1) : asin(aa / r1);
        if (extent != extent) return false;
    }
    const float umax = (float)(0.5f - cos(extent) * 0.5f);
    const double phi = acos(1.0 - 2.0 * g.ud(0.0, (double)umax));
    const F3 dir = xa * (float)sin(phi) * cosf(theta) + ya * (float)sin(phi) * sinf(theta) + za * (float)cos(phi);
    P.set(l + 1, a + funit(dir) * (float)ds);
    return resolve_two(P, l + 1, r, ds, g);
}

// The centre point of m segments between l and r (ResolveEvenNumberOfSegments' placement);
// the halves are handled by the caller. inv_h = 2 / m.
__device__ bool place_centre(const PathPts &P, int m, double inv_h, uint32_t l, uint32_t r, double ds, double inv_ds, Draws &g)
{
    const int h = m / 2;
    const uint32_t c = l + (uint32_t)h;
    const F3 a = P.get(l), b = P.get(r);
    const double d = fmag(b - a);
    if (fabs((m * ds) - d) < 0.001f) {
        P.set(c, (b + a) * 0.5f);
        return true;
    }
    const double rad = ds * h;
    if ((rad + rad) < d) return false;
    F3 xa, ya, za;
    if (d < 0.001f) {
        const double phi = acos(1.0 - 2.0 * g.ud(0.0, 1.0));
        const double theta = g.ud(0.0, (double)(2.0f * kPiF));
        const double sr = rad * cbrt((double)g.uf(0.0f, 1.0f));
        frame(a, b, xa, ya, za);
        F3 off = xa * (float)sin(phi) * (float)cos(theta) + ya * (float)sin(phi) * (float)sin(theta) + za * (float)cos(phi);
        P.set(c, a + off * (float)sr);
        return true;
    }
    const F3 mid = (b + a) * 0.5f;
    const double to_mid = fmag(mid - a);
    // cos(asin(sqrt(rad^2 - d^2 / 4) / rad)) = d / (2 rad)
    const float umax = (float)(0.5 - 0.25 * d * (inv_ds * inv_h));
    const double u = g.ud(0.0, (double)umax);
    const double cphi = 1.0 - 2.0 * u, sphi = 2.0 * sqrt(u * (1.0 - u));
    const double theta = g.ud(0.0, (double)(2.0f * kPiF));
    const bool flip = g.coin() != 0;
    const double maxr = h * ds;
    const double minp = to_mid / (cphi * maxr);
    const double sr = maxr * cbrt(minp + (1.0f - minp) * (double)g.uf(0.0f, 1.0f));
    frame(a, b, xa, ya, za);
    double st, ct;
    sincospi(theta * 0.31830988618379067154, &st, &ct);
    const float sp = (float)sphi;
    F3 off = xa * sp * (float)ct + ya * sp * (float)st;
    if (!flip) {
        off = off + za * (float)cphi;
        P.set(c, a + off * (float)sr);
    } else {
        off = off + za * (float)cphi * -1.0f;
        P.set(c, b + off * (float)sr);
    }
    return true;
}

struct MSegSpec {
    uint32_t n_segments;
    float ds;
    float p0[3], p1[3], pm1[3], pm[3];
    uint64_t seed;
    uint32_t experiment;
    uint64_t path0;
    uint64_t n_paths;
};

// Places the points of one path; false when the reference would abort. N - 2 = LEAF << depth (the host validated N - 2 as
// resolvable). LEAF, 4 or 6, is the kernel's, a leaf's two halves share their code, and resolve_three is called, not
// inlined: with both kinds of leaves inlined twice in one kernel, compensated paths waited for their instructions
// (2^26 path-segments, N = 66 2.04 -> 1.76 ms, 98 3.40 -> 2.49, 386 5.35 -> 3.30, 770 8.33 -> 5.05; plain 2.22 -> 2.15,
// 3.13 -> 3.02, 4.11 -> 3.97, 6.57 -> 6.27; the same bits).
template <uint32_t LEAF>
__device__ bool build_path(const MSegSpec &s, const PathPts &P, uint64_t path)
{
    const uint32_t N = s.n_segments;
    Draws g(s.seed, (uint32_t)path, (uint32_t)(path >> 32), s.experiment ^ 0x4D534547u);
    const double ds = s.ds, inv_ds = 1.0 / ds;
    constexpr uint32_t leaf = LEAF;
    const uint32_t depth = 31u - (uint32_t)__clz((int)((N - 2) / leaf));
    const double inv_leaf = 2.0 / (double)leaf;
    for (uint32_t t = 0; t < (1u << depth); ++t) {
        const uint32_t l = 1 + t * leaf;
        const int top = t ? __ffs((int)t) - 1 : (int)depth;
        for (int k = top; k >= 0; --k) {
            const uint32_t m = leaf << k;
            // 2 / m = 2 / leaf scaled by 2^-k
            const double inv_h = __hiloint2double(__double2hiint(inv_leaf) - (k << 20), __double2loint(inv_leaf));
            if (!place_centre(P, (int)m, inv_h, l, l + m, ds, inv_ds, g)) return false;
        }
#pragma unroll 1
        for (uint32_t half = l; half < l + leaf; half += leaf / 2)
            if (LEAF == 4 ? !resolve_two(P, half, half + 2, ds, g) : !resolve_three(P, half, half + 3, ds, g)) return false;
    }
    return true;
}

// Walks the curvatures of a path: seg(kappa-like value of the two tangents) until it returns false.
template <class TanFn, class SegFn>
__device__ __forceinline__ bool walk_path(const PathPts &P, uint32_t N, TanFn tan, SegFn seg)
{
    F3 at = P.get(0), before{0.f, 0.f, 0.f};
    for (uint32_t i = 0; i < N; ++i) {
        const F3 next = P.get(i + 1);
        const F3 t = tan(next, at);
        if (i > 0 && !seg(t, before)) return false;
        before = t;
        at = next;
    }
    return true;
}

// log10 weight of a path with the compensated weigher's arithmetic (path_log10: the same
// tangents, bins, entries and fractions; the interpolation corrections add up in FP64).
template <bool EXACT>
__device__ bool weigh_comp(const PathPts &P, uint32_t N, const CompConsts &kc, const float2 *__restrict__ tab, double &w)
{
    unsigned long long isum = 0;
    double csum = 0.0;
    float ks = 0.f, kk = 0.f;
    uint32_t clamped = 0;
    auto tan = [&](F3 b, F3 a) {
        const float x = b.x - a.x, y = b.y - a.y, z = b.z - a.z;
        const float r = rsqrtf(fmaf(x, x, fmaf(y, y, z * z))) * kc.kscale;
        return F3{x * r, y * r, z * r};
    };
    walk_path(P, N, tan, [&](F3 t, F3 b) {
        const float dx = t.x - b.x, dy = t.y - b.y, dz = t.z - b.z;
        int32_t L;
        const float frac = bin_of<true>(fmaf(dx, dx, fmaf(dy, dy, dz * dz)), kc, true, clamped, L);
        const float2 e = tab_load<true>(tab, L);
        if (EXACT) {
            kahan_add(ks, kk, __log2f(fmaf(frac * kc.step, e.y, e.x)) * kLog10_2);
        } else {
            isum += __float_as_uint(e.x);
            csum += (double)frac * (double)e.y;
        }
        return true;
    });
    w = EXACT ? (double)ks - (double)kk : kc.lw_offset + (double)isum * kc.inv_scale + csum;
    return !isnan(w);
}

// The same with the plain weigher's arithmetic (weigh_plain_kernel, chain_plain.cu: the
// reference's FP32 operations), the segment weights multiplied as mantissas and exponents.
__device__ bool weigh_plain(const PathPts &P, uint32_t N, float inv_ds, const float *__restrict__ lut, const dev::LutMeta &m,
                            double absorption_factor, double &w)
{
    double prod = 1.0, logs = 0.0;
    int esum = 0;
    uint32_t clamped = 0;
    auto tan = [&](F3 b, F3 a) {
        const float x = __fsub_rn(b.x, a.x), y = __fsub_rn(b.y, a.y), z = __fsub_rn(b.z, a.z);
        const float r = dev::rinvnorm(x, y, z);
        return F3{__fmul_rn(x, r), __fmul_rn(y, r), __fmul_rn(z, r)};
    };
    auto normalise = [&] {
        esum += (__double2hiint(prod) >> 20) - 1023;
        prod = __hiloint2double((__double2hiint(prod) & 0x000fffff) | 0x3ff00000, __double2loint(prod));
    };
    const bool ok = walk_path(P, N, tan, [&](F3 t, F3 b) {
        const float kappa = __fsqrt_rn(dev::rdot3(__fmul_rn(__fsub_rn(t.x, b.x), inv_ds), __fmul_rn(__fsub_rn(t.y, b.y), inv_ds),
                                                  __fmul_rn(__fsub_rn(t.z, b.z), inv_ds)));
        double blend = 0.0;
        if (dev::rbin_blend(kappa, lut, m, blend, clamped) < 0) return false;
        const double v = __dmul_rn(blend, absorption_factor);
        const int hi = __double2hiint(v);
        if (hi < 0x00100000 || hi >= 0x7ff00000) {   // not a positive normal number: rare
            const double lg = log10(v);
            logs += lg;
            return !isnan(lg);
        }
        esum += (hi >> 20) - 1023;
        prod *= __hiloint2double((hi & 0x000fffff) | 0x3ff00000, __double2loint(v));
        if (prod >= 1e300) normalise();
        return true;
    });
    if (!ok) return false;
    w = log10(prod) + (double)esum * 0.30102999566398119521 + logs;
    return !isnan(w);
}

constexpr int kMsegThreads = 128;

// FORM 0: the plain weigher; 1: the compensated fixed-point table (a path through a steep bin, or with
// a NaN curvature, again through the linear one); 2: the linear table. Writes one sample per path.
template <int FORM, uint32_t LEAF>
__global__ void __launch_bounds__(kMsegThreads, 6)
msegment_kernel(MSegSpec s, MSegWeigh wg, CompConsts kc, float *__restrict__ scratch, ChainOut *__restrict__ out)
{
    const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x, threads = (size_t)gridDim.x * blockDim.x;
    const PathPts P{scratch + tid, threads};
    const uint32_t N = s.n_segments;
    P.set(0, F3{s.p0[0], s.p0[1], s.p0[2]});
    P.set(1, F3{s.p1[0], s.p1[1], s.p1[2]});
    P.set(N - 1, F3{s.pm1[0], s.pm1[1], s.pm1[2]});
    P.set(N, F3{s.pm[0], s.pm[1], s.pm[2]});
    const dev::LutMeta m{wg.meta.min_k, wg.meta.max_k, wg.meta.step, wg.meta.bins};
    for (uint64_t i = tid; i < s.n_paths; i += threads) {
        double w = 0.0;
        bool ok = build_path<LEAF>(s, P, s.path0 + i);
        if (ok) {
            if constexpr (FORM == 0) {
                ok = weigh_plain(P, N, wg.inv_ds, wg.lut, m, wg.absorption_factor, w);
            } else {
                ok = weigh_comp<FORM == 2>(P, N, kc, FORM == 2 ? wg.lin : wg.fix, w);
                if (FORM == 1 && !ok) ok = weigh_comp<true>(P, N, kc, wg.lin, w);
                w += (double)(N - 1) * wg.log10_absorption;
            }
        }
        ChainOut o;
        o.log10_sum = ok ? w : -INFINITY;
        o.valid = ok ? 1u : 0u;
        o.failed = ok ? 0u : 1u;
        o.clamped = 0;
        o.pad = 0;
        out[i] = o;
    }
}

template <int FORM>
void launch_form(const MSegSpec &s, const MSegWeigh &wg, const CompConsts &kc, unsigned blocks, float *scratch, ChainOut *out,
                 cudaStream_t st)
{
    uint32_t leaf = s.n_segments - 2;
    while (leaf > 6) leaf >>= 1;
    if (leaf == 4) msegment_kernel<FORM, 4><<<blocks, kMsegThreads, 0, st>>>(s, wg, kc, scratch, out);
    else msegment_kernel<FORM, 6><<<blocks, kMsegThreads, 0, st>>>(s, wg, kc, scratch, out);
}

}  // namespace

// Threads of a launch: 768 per SM (N = 66, 2^21 paths, before a kernel had one kind of leaf: 4.03 ms at 768, 4.07 at
// 1024, 4.35 at 512; the step is bound by issue, 40 k instructions per path, and instruction fetch), fewer while their columns
// exceed 384 MB (the context keeps them), and no more than there are paths.
uint32_t msegment_threads(uint32_t n_segments, uint64_t n_paths)
{
    constexpr uint64_t kSms = 148;
    const uint64_t column = 3 * sizeof(float) * (uint64_t)(n_segments + 1);
    const uint64_t t = std::min({kSms * 768, std::max<uint64_t>((384ull << 20) / column, 1), std::max<uint64_t>(n_paths, 1)});
    return (uint32_t)((t + kMsegThreads - 1) / kMsegThreads * kMsegThreads);
}

cudaError_t launch_msegment(uint32_t n_segments, float ds, const float p0[3], const float p1[3], const float pm1[3],
                            const float pm[3], uint64_t seed, uint32_t experiment, uint64_t path0, uint64_t n_paths,
                            uint32_t threads, const MSegWeigh &wg, float *scratch, ChainOut *out, cudaStream_t st)
{
    if (n_paths == 0) return cudaSuccess;
    MSegSpec s{};
    s.n_segments = n_segments;
    s.ds = ds;
    for (int k = 0; k < 3; ++k) {
        s.p0[k] = p0[k];
        s.p1[k] = p1[k];
        s.pm1[k] = pm1[k];
        s.pm[k] = pm[k];
    }
    s.seed = seed;
    s.experiment = experiment;
    s.path0 = path0;
    s.n_paths = n_paths;
    const CompConsts kc = make_consts(wg.inv_ds, wg.meta, n_segments, wg.lf);
    const unsigned blocks = threads / kMsegThreads;
    if (wg.plain) launch_form<0>(s, wg, kc, blocks, scratch, out, st);
    else if (wg.exact || wg.lf.inv_scale == 0.0) launch_form<2>(s, wg, kc, blocks, scratch, out, st);
    else launch_form<1>(s, wg, kc, blocks, scratch, out, st);
    return cudaGetLastError();
}

}  // namespace twisty
