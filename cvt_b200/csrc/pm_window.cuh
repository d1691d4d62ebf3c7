// Window loops of the PatchMatch-Huber path: the adaptive-support-weight cost
// (patch_eval_census, pmhstereo.cl:661-736) and the Gauss-Newton plane step
// (patch_census_klt2, :326-410), one thread per pixel, samples in the
// reference's order.
//
// Texel layout.  Each view is stored as four planes of 16-byte texels in rows of W + 8:
// columns -4 .. W+3, the four on either side replicating the edge texel
// (CLK_ADDRESS_CLAMP_TO_EDGE).  Colour (r, g, b, Σw) and gradient (4 components), the
// gradient plane `plane` texels after the colour plane, serve the general loops and the
// centre texel.  The compact plane (r, g, b, the four gradient sign bits as bytes), `plane`
// after the gradient plane, holds all that a first-view window sample needs, in one load.
// The pair plane, `plane` after that, holds all that a bilinear tap of the second view
// between columns i and i + 1 needs, in one load (PairRec).  After the four planes, one int:
// set when the view cannot be read through the pair plane (k_pack_tex): its colours are not
// all k / 255 for a byte k, or a gradient is not finite.
//
// Why pairs.  The loops were bound by the L1 data path: a warp-wide 16-byte gather at any
// texel offset takes 7.3 wavefronts, so 8 gathers of float texels per Gauss-Newton sample
// (4 per cost sample) and one of the first view kept the L1 82-90% busy.  A tap's colours are
// bytes / 255, rebuilt in two instructions per channel, and of its four interpolated
// gradients only the signs are used: each sign is a comparison of the tap weight with a
// threshold fixed by the two texels, so 4 x 16 bits replace 2 x 16 bytes and the four
// interpolations.  3 gathers per Gauss-Newton sample and 1 per cost sample remain.
//
// Blackwell specifics: the bilinear colour mixes, the truncated absolute differences and
// the Gauss-Newton sums run as packed FP32 pairs (sm_100), four gradient signs of a tap
// are compared as 16-bit fields of two integer subtractions, and the three Gauss-Newton
// taps at x'-1, x', x'+1 read three chained pair records.  Every packed operation rounds
// per element exactly like its scalar form, so results equal the scalar restatement bit
// for bit.
#pragma once

#include "pm_device.cuh"

namespace pm {

constexpr int TEX_PAD = 4;     // replicated columns on each side of a texel row
constexpr int TEX_PLANES = 4;  // colour, gradient, compact, pair

struct ViewData {
    const float4* __restrict__ t1;   // first view: colour plane, gradient at + plane, compact at + 2 plane, pair at + 3 plane
    const float4* __restrict__ t2;   // second view
    int W, H, r, P;                  // P = W + 2 * TEX_PAD texels per row
    int plane;                       // H * P
    const int* gen1;                 // the views' flags: read by the general loops (after the planes)
    const int* gen2;
    float2 one;                      // (1, 1), opaque to the compiler (sum2)
    // colour texel (compact texel) of column 0 of row y
    __device__ __forceinline__ const float4* row1(int y) const { return t1 + (size_t)y * P + TEX_PAD; }
    __device__ __forceinline__ const float4* row1c(int y) const { return t1 + 2 * (size_t)plane + (size_t)y * P + TEX_PAD; }
    __device__ __forceinline__ const float4* row2(int y) const { return t2 + (size_t)y * P + TEX_PAD; }
    // pair record of column 0 of row y
    __device__ __forceinline__ const float4* row2p(int y) const { return t2 + 3 * (size_t)plane + (size_t)y * P + TEX_PAD; }
};

// Pair record of columns (i, i + 1), one 16-byte word group:
//   x  bytes r, g, b of texel i; bits 24-27 the signs of its four gradient components
//   y  bytes r, g, b of texel i + 1
//   z  sign thresholds of gradient components 1 (low half) and 3 (high half)
//   w  sign thresholds of components 0 and 2
// With A = a 2^15 the tap weight in units of 2^-15, the interpolated component has the sign
// of texel i for A < threshold and the other sign from there on (pair_threshold).
typedef uint4 PairRec;
constexpr uint32_t PAIR_NEVER = 0x8000u;   // threshold of a component whose sign does not change

struct Counters {
    unsigned long long eval, klt, calls, exits;
};

__device__ __forceinline__ float2 f2(float x, float y) { return make_float2(x, y); }

// bilinear pair: (1-a)*T0 + a*T1 per element; fused contracts a*T1.  The strict form rounds
// the two products (one packed multiply each) and adds them with scalar, explicitly rounded
// adds: packed adds fed by packed multiplies were measured to come out fused, which would
// change the rounding; a packed multiply feeding __fadd_rn does not (the 1280x720 results are
// bit-identical to the all-scalar form, which PM_STRICT_FMUL2=0 selects).
#ifndef PM_STRICT_FMUL2
#define PM_STRICT_FMUL2 1
#endif

template <bool F>
__device__ __forceinline__ float2 lerp2(float2 a2, float2 b2, float2 t0, float2 t1)
{
    if (F) return __ffma2_rn(a2, t1, __fmul2_rn(b2, t0));
#if PM_STRICT_FMUL2
    const float2 p0 = __fmul2_rn(b2, t0), p1 = __fmul2_rn(a2, t1);
    return make_float2(__fadd_rn(p0.x, p1.x), __fadd_rn(p0.y, p1.y));
#else
    return make_float2(__fadd_rn(__fmul_rn(b2.x, t0.x), __fmul_rn(a2.x, t1.x)),
                       __fadd_rn(__fmul_rn(b2.y, t0.y), __fmul_rn(a2.y, t1.y)));
#endif
}

// one texel: colour (r, g, b, w) and gradient (4 components)
struct Texel {
    float4 c, g;
};

__device__ __forceinline__ Texel texel_at(const float4* __restrict__ p, int plane)
{
    Texel t;
    t.c = __ldg(p);
    t.g = __ldg(p + plane);
    return t;
}

template <bool F>
__device__ __forceinline__ Texel lerp_texel(float a, float b, const Texel& t0, const Texel& t1)
{
    const float2 a2 = f2(a, a), b2 = f2(b, b);
    const float2 c01 = lerp2<F>(a2, b2, f2(t0.c.x, t0.c.y), f2(t1.c.x, t1.c.y));
    const float2 c23 = lerp2<F>(a2, b2, f2(t0.c.z, t0.c.w), f2(t1.c.z, t1.c.w));
    const float2 g01 = lerp2<F>(a2, b2, f2(t0.g.x, t0.g.y), f2(t1.g.x, t1.g.y));
    const float2 g23 = lerp2<F>(a2, b2, f2(t0.g.z, t0.g.w), f2(t1.g.z, t1.g.w));
    Texel r;
    r.c = make_float4(c01.x, c01.y, c23.x, c23.y);
    r.g = make_float4(g01.x, g01.y, g23.x, g23.y);
    return r;
}

// SAMPLER_BILINEAR (:71) read at (u, row + 0.5), OpenCL 1.2 s8.2 with the vertical weight
// exactly 0: (1-a)*T[i0] + a*T[i0+1], columns clamped to the edge; a non-finite
// coordinate reads the positive quiet NaN.  General form, for the rare taps the fast
// paths below do not cover.
template <bool F>
__device__ __forceinline__ Texel lerp_texel_at(const float4* __restrict__ row, int plane, int W, float u)
{
    const float t = u - 0.5f;
    if (!fin(t)) {
        const float n = qnan();
        Texel r;
        r.c = f4(n, n, n, n);
        r.g = r.c;
        return r;
    }
    float fl = floorf(t);
    const float a = t - fl;
    fl = fminf(fmaxf(fl, -1.0f), (float)W);
    const int i0 = (int)fl;
    const int j0 = min(max(i0, 0), W - 1), j1 = min(max(i0 + 1, 0), W - 1);
    return lerp_texel<F>(a, 1.0f - a, texel_at(row + j0, plane), texel_at(row + j1, plane));
}

// byte k holds the top byte of component k, so bit 7 of byte k is its sign bit
__device__ __forceinline__ uint32_t sign_bytes(float4 g)
{
    const uint32_t lo = __byte_perm(__float_as_uint(g.x), __float_as_uint(g.y), 0x0073);
    const uint32_t hi = __byte_perm(__float_as_uint(g.z), __float_as_uint(g.w), 0x0073);
    return __byte_perm(lo, hi, 0x5410);
}

// number of gradient components whose signs differ (the census term, :712-715, :367-370)
__device__ __forceinline__ int sign_mismatch(uint32_t a, uint32_t b) { return __popc((a ^ b) & 0x80808080u); }

// x / 0.05f for 0 <= x <= 0.05f, x >= 2^-100 or x = 0: 1 / 0.05f = 20 + D005 (D005 =
// RN(1 / 0.05f - 20)), and RN(20 x + RN(D005 x)) is the correctly rounded quotient
// (Brisebarre and Muller, "Correctly rounded multiplication by arbitrary precision
// constants"; compared with the division for every float of the range).
#define PM_D005 -2.98023224e-07f

// Sum over r, g, b of fmin(|v2 - ref|, 0.05) / 0.05 (:707-709, :364-365), divisions exact.
// Below 2^-100 the division itself is taken (CHK); colours read as k / 255 never give such
// a difference (see tap_cost), so loops over those leave the test out.
template <bool CHK>
__device__ __forceinline__ float ad_sum(float4 v2, float4 ref)
{
    const float2 d01 = __ffma2_rn(f2(ref.x, ref.y), f2(-1.0f, -1.0f), f2(v2.x, v2.y));   // v2 - ref, exact
    const float d2 = v2.z - ref.z;
    const float m0 = fminf(fabsf(d01.x), 0.05f), m1 = fminf(fabsf(d01.y), 0.05f), m2 = fminf(fabsf(d2), 0.05f);
    const float2 m01 = f2(m0, m1);
    float2 c01 = __ffma2_rn(m01, f2(20.0f, 20.0f), __fmul2_rn(m01, f2(PM_D005, PM_D005)));
    float c2 = fmaf(m2, 20.0f, m2 * PM_D005);
    if (CHK && fminf(fminf(m0, m1), m2) < 7.88860905e-31f) {   // below 2^-100 the two-term product is not exact
        c01 = f2(m0 / 0.05f, m1 / 0.05f);
        c2 = m2 / 0.05f;
    }
    return c01.x + c01.y + c2;
}

// (w1 * 0.125f) * 0.33f and 0.125f * (0.33f * S) as one multiply: the product of 0.125 and
// 0.33f is exact, and scaling by a power of two commutes with rounding
#define PM_K033_8 0.04125000163912773f

// Per-sample weights of a Gauss-Newton window sample for klt_cost: k1 = w1 * 0.125 * 0.33
// (one multiply, see PM_K033_8) and the census weight x = w1 * 0.875f.
struct KltWeights {
    float k1, x;
};

template <bool F>
__device__ __forceinline__ KltWeights klt_weights(float w1)
{
    KltWeights k;
    k.k1 = w1 * PM_K033_8;
    k.x = F ? w1 * 0.21875f : w1 * 0.875f;
    return k;
}

// the cost of one Gauss-Newton tap from its interpolated texel (:361-370), general loops.
// `w1 * (1.0f - alpha) * 0.25 * (float)cnt` (:370) carries a double literal, so the sum is a
// double-precision one rounded once: formed exactly in double (strict) or with one fma
// (fused; w1 * 0.875f * 0.25f is one multiply by 0.21875 for the same reason as above).
template <bool F>
__device__ __forceinline__ float klt_cost(const KltWeights& kw, float4 val1, uint32_t sb1, const Texel& t)
{
    float C = kw.k1 * ad_sum<true>(t.c, val1);
    const int n = sign_mismatch(sb1, sign_bytes(t.g));
    if (F) C = fmaf(kw.x, (float)n, C);
    else C = (float)((double)C + (double)kw.x * 0.25 * (double)(float)n);
    return C;
}

// mat3f_lusolve (Matrix3.cl:286-311) on the symmetric 3x3 H = [h00 h01 h02; h01 h11 h12; h02 h12 h22]
__device__ __forceinline__ float3 lusolve(float h00, float h01, float h02, float h11, float h12, float h22, float3 b)
{
    float m10 = h01, m20 = h02, m11 = h11, m12 = h12, m21 = h12, m22 = h22;
    const float m00 = h00, m01 = h01, m02 = h02;
    m10 /= m00;
    m20 /= m00;
    m11 -= m10 * m01;
    m12 -= m10 * m02;
    m21 -= m20 * m01;
    m22 -= m20 * m02;
    m21 /= m11;
    m22 -= m21 * m12;
    b.y -= m10 * b.x;
    b.z -= m20 * b.x + m21 * b.y;
    float3 ret;
    ret.z = b.z / m22;
    ret.y = (b.y - m12 * ret.z) / m11;
    ret.x = (b.x - (m01 * ret.y + m02 * ret.z)) / m00;
    return ret;
}

// Kernels that run the window loops come in two variants launched back to back: the pair-plane
// loops (return at once when a view's flag is set) and the general ones (GEN; return at once
// when none is, if `dual`); a kernel launched alone is the general one with dual = 0.
__device__ __forceinline__ bool views_general(const ViewData& V) { return (__ldg(V.gen1) | __ldg(V.gen2)) != 0; }
template <bool GEN>
__device__ __forceinline__ bool variant_skips(const ViewData& V, int dual)
{
    const bool gen = views_general(V);
    return GEN ? (dual && !gen) : gen;
}

// one window sample of patch_eval_census (:690-722), general loops, at window position (qx, row of q1) of a
// pixel with centre texel `in`, for the plane s (byq = s.y * qy): accumulates the weighted
// cost into census and the weight into wsum, or returns false when the matched column lies
// outside the image (:693-696)
template <bool F>
__device__ __forceinline__ bool eval_sample(const float4* __restrict__ q1, const float4* __restrict__ row2, int plane,
                                            int W, float fW, float4 in, float4 s, float qx, float byq, float& census,
                                            float& wsum)
{
    const float p2x = F ? fmaf(s.x, qx, byq) + s.z : s.x * qx + byq + s.z;
    if (p2x < 0 || p2x >= fW) return false;
    const float4 q = __ldg(q1);   // compact texel
    const float w = support_weight<F>(q.x - in.x, q.y - in.y, q.z - in.z);
    const float t = (p2x + 0.5f) - 0.5f;
    Texel tx;
    if (fin(t)) {
        // p2x in [0, W) gives t in [0, W]: texels i0, i0 + 1 lie in the padded row
        const float fl = floorf(t);
        const float a = t - fl;
        const float4* __restrict__ b = row2 + (int)fl;
        tx = lerp_texel<F>(a, 1.0f - a, texel_at(b, plane), texel_at(b + 1, plane));
    } else {   // a non-finite coordinate reads the positive quiet NaN (lerp_texel_at)
        const float n = qnan();
        tx.c = f4(n, n, n, n);
        tx.g = tx.c;
    }
    float cost = PM_K033_8 * ad_sum<true>(tx.c, q);
    // cost + 0.875f * (0.25f * n): the product 0.21875 n is exact, so one fma rounds the same
    cost = fmaf(0.21875f, (float)sign_mismatch(__float_as_uint(q.w), sign_bytes(tx.g)), cost);
    census = F ? fmaf(w, cost, census) : census + w * cost;
    wsum += w;
    return true;
}

// validity test at the top of patch_eval_census (:675-678): a plane that is not finite,
// too steep, or whose centre matches outside the image costs 1e5 without a window
__device__ __forceinline__ bool plane_usable(float4 s, float cx, float cy, int W)
{
    const float c2x = transform_x(s, cx, cy);
    return fin(s.x) && fin(s.y) && fin(s.z) && !(to_normal(s).z < 1e-4f) && !(c2x < 0) && !(c2x >= (float)W);
}

// patch_eval_census (:661-736).  The early exit `census / bilw >= mincost` (:724) is tested
// as census >= exit_threshold(mincost, bilw), the same predicate without a division.
// Window coordinates run as floats (integers below 2^24 are exact) instead of being
// converted from the loop counters.
template <bool F, bool COUNT>
__device__ __forceinline__ float patch_eval_general(const ViewData& V, int px, int py, float4 s, float mincost, Counters& cnt)
{
    const float cx = (float)px, cy = (float)py;
    if (!plane_usable(s, cx, cy, V.W)) return 1e5f;
    const int W = V.W, plane = V.plane;
    const float4 in = __ldg(V.row1(py) + px);
    const float thr = exit_threshold(mincost, in.w);
    float wsum = 0.0f, census = 0.0f;
    if (COUNT) cnt.calls++;
    const int r = V.r;
    const int dy0 = max(-r, -py), dy1 = min(r, V.H - 1 - py);
    const int dx0 = max(-r, -px), dx1 = min(r, W - 1 - px);
    const float fW = (float)W;
    const float qx0 = cx + (float)dx0;
    float qy = cy + (float)dy0;
    for (int iy = py + dy0; iy <= py + dy1; iy++, qy += 1.0f) {
        const float byq = s.y * qy;
        const float4* __restrict__ q1 = V.row1c(iy) + px + dx0;
        const float4* __restrict__ row2 = V.row2(iy);
        float qx = qx0;
        for (int n = dx1 - dx0; n >= 0; n--, q1++, qx += 1.0f) {
            if (!eval_sample<F>(q1, row2, plane, W, fW, in, s, qx, byq, census, wsum)) continue;
            if (COUNT) cnt.eval++;
            if (census >= thr) {
                if (COUNT) cnt.exits++;
                return 1.0f;
            }
        }
    }
    if (wsum <= 1.0f) return 1.1f;
    return census / wsum;
}

// patch_census_klt2 (:326-410), with the in-bounds test on the window position rather than
// the matched one (:358) and the colour term against the colour difference (:352, :364)
template <bool F, bool COUNT>
__device__ __forceinline__ float4 klt2_general(const ViewData& V, int px, int py, float4 s, Counters& cnt)
{
    const float cxf = (float)px, cyf = (float)py;
    const int W = V.W, plane = V.plane;
    float2 J01 = f2(0.0f, 0.0f);
    float J2 = 0.0f;
    float2 h00_01 = f2(0.0f, 0.0f), h02_11 = f2(0.0f, 0.0f), h12_22 = f2(0.0f, 0.0f);
    const float4 c1 = __ldg(V.row1(py) + px);
    const int r = V.r;
    const int dy0 = max(-r, -py), dy1 = min(r, V.H - 1 - py);
    const int dx0 = max(-r, 1 - px), dx1 = min(r, W - 2 - px);   // the 3-point cost needs 1 <= qx < W - 1
    const float qx0 = cxf + (float)dx0;
    const float fWm2 = (float)(W - 2), fWm1 = (float)(W - 1);
    float qy = cyf + (float)dy0;
    for (int iy = py + dy0; iy <= py + dy1; iy++, qy += 1.0f) {
        const float byq = s.y * qy;
        const float yy = qy * qy;
        const float4* __restrict__ q1 = V.row1c(iy) + px + dx0;
        const float4* __restrict__ row2 = V.row2(iy);
        float qx = qx0;
        for (int n = dx1 - dx0; n >= 0; n--, q1++, qx += 1.0f) {
            const float4 q = __ldg(q1);   // compact texel
            const float4 val1 = make_float4(q.x - c1.x, q.y - c1.y, q.z - c1.z, 0.0f);
            const float w1 = support_weight<F>(val1.x, val1.y, val1.z);
            const uint32_t sb1 = __float_as_uint(q.w);
            const KltWeights kw = klt_weights<F>(w1);
            const float p2x = F ? fmaf(s.x, qx, byq) + s.z : s.x * qx + byq + s.z;
            // The three taps read at t - 1, t, t + 1 (t the tap coordinate minus 0.5, each formed
            // as the source forms it).  Common case: 1 <= p2x < W - 1 and p2x + 1.5 in the binade
            // of p2x; then p2x is a multiple of its ulp (<= 0.5), every +-1 and +-0.5 below is
            // exact, the coordinates are p2x - 1, p2x, p2x + 1 and share the weight
            // p2x - floor(p2x).  Otherwise the coordinates and their floors are formed exactly;
            // when the floors still chain (f0 - 1, f0, f0 + 1) the taps read the same four texels
            // with their own weights, and only then, or off the padded row, each tap is read on
            // its own.  Every path gives the bilinear values lerp_texel_at gives.
            float f0, am, a0, ap;
            bool chain = p2x >= 1.0f && p2x < fWm1 &&
                         ((__float_as_uint(p2x + 1.5f) ^ __float_as_uint(p2x)) < 0x00800000u);
            if (chain) {
                f0 = floorf(p2x);
                a0 = p2x - f0;
                am = a0;
                ap = a0;
            } else {
                const float t0 = (p2x + 0.5f) - 0.5f;
                const float tp = ((p2x + 1.0f) + 0.5f) - 0.5f;
                const float tm = ((p2x + -1.0f) + 0.5f) - 0.5f;
                f0 = floorf(t0);
                const float fp = floorf(tp), fm = floorf(tm);
                a0 = t0 - f0;
                ap = tp - fp;
                am = tm - fm;
                chain = fp == f0 + 1.0f && fm == f0 - 1.0f && f0 >= -1.0f && f0 <= fWm2;
            }
            Texel xm, x0, xp;
            if (chain) {
                // texels f0-1 .. f0+2, inside the padded row
                const float4* __restrict__ b = row2 + ((int)f0 - 1);
                const Texel tA = texel_at(b, plane), tB = texel_at(b + 1, plane);
                const Texel tC = texel_at(b + 2, plane), tD = texel_at(b + 3, plane);
                xm = lerp_texel<F>(am, 1.0f - am, tA, tB);
                x0 = lerp_texel<F>(a0, 1.0f - a0, tB, tC);
                xp = lerp_texel<F>(ap, 1.0f - ap, tC, tD);
            } else {
                xm = lerp_texel_at<F>(row2, plane, W, (p2x + -1.0f) + 0.5f);
                x0 = lerp_texel_at<F>(row2, plane, W, p2x + 0.5f);
                xp = lerp_texel_at<F>(row2, plane, W, (p2x + 1.0f) + 0.5f);
            }
            const float Cxm = klt_cost<F>(kw, val1, sb1, xm);
            const float C = klt_cost<F>(kw, val1, sb1, x0);
            const float Cxp = klt_cost<F>(kw, val1, sb1, xp);
            if (COUNT) cnt.klt++;
            // the update of :394-402 without a branch: a rejected sample adds exact zeros, and
            // no accumulator can be -0, so adding +0 or -0 leaves it unchanged
            const float curv = Cxp + Cxm - 2.0f * C;
            const bool take = curv > 0.0f;
            const float t = take ? w1 * (Cxm - Cxp) * 0.5f : 0.0f;
            const float sc = take ? w1 * curv : 0.0f;
            if (F) {
                const float2 t2 = f2(t, t), s2 = f2(sc, sc);
                J01 = __ffma2_rn(t2, f2(qx, qy), J01);
                J2 = fmaf(t, 1.0f, J2);
                h00_01 = __ffma2_rn(s2, f2(qx * qx, qx * qy), h00_01);
                h02_11 = __ffma2_rn(s2, f2(qx, yy), h02_11);
                h12_22 = __ffma2_rn(s2, f2(qy, 1.0f), h12_22);
            } else {   // scalar, explicitly rounded (see lerp2)
                J01 = f2(__fadd_rn(J01.x, __fmul_rn(t, qx)), __fadd_rn(J01.y, __fmul_rn(t, qy)));
                J2 = J2 + t * 1.0f;
                h00_01 = f2(__fadd_rn(h00_01.x, __fmul_rn(sc, qx * qx)), __fadd_rn(h00_01.y, __fmul_rn(sc, qx * qy)));
                h02_11 = f2(__fadd_rn(h02_11.x, __fmul_rn(sc, qx)), __fadd_rn(h02_11.y, __fmul_rn(sc, yy)));
                h12_22 = f2(__fadd_rn(h12_22.x, __fmul_rn(sc, qy)), __fadd_rn(h12_22.y, __fmul_rn(sc, 1.0f)));
            }
        }
    }
    const float3 d = lusolve(h00_01.x, h00_01.y, h02_11.x, h02_11.y, h12_22.x, h12_22.y, make_float3(J01.x, J01.y, J2));
    return f4(s.x - d.x, s.y - d.y, s.z - d.z, s.w - 1e5f);
}

// ---- pair-plane loops ------------------------------------------------------------------

// p + c per element, each rounded, for p a packed product.  A packed add fed by a packed multiply comes out
// contracted (with .rn on both and with an fma by a literal 1 too); an fma by a kernel argument
// that is 1 cannot.
__device__ __forceinline__ float2 sum2(float2 p, float2 c, float2 one) { return __ffma2_rn(p, one, c); }

// byte k of a record word, as the float byte * 2^-133: bits 16-23 of an otherwise zero word
// (exponent field 0 or 1, one linear scale)
template <int K>
__device__ __forceinline__ float pair_byte(uint32_t w)
{
    return __uint_as_float(__byte_perm(w, 0u, 0x4044 | (K << 8)));
}

// byte / 255 correctly rounded from byte * 2^-133: 2^133 / 255 = RGB_HI + RGB_LO and
// RN(RGB_HI x + RN(RGB_LO x)) (the method of PM_D005; equal to the division for all 256 bytes)
#define PM_RGB_HI 0x1.010102p+125f
#define PM_RGB_LO -0x1.fdfdfep+100f
__device__ __forceinline__ float2 rgb_unit(float2 x)
{
    return __ffma2_rn(x, f2(PM_RGB_HI, PM_RGB_HI), __fmul2_rn(x, f2(PM_RGB_LO, PM_RGB_LO)));
}

// bilinear mix of two texels' colours (rg0, b.x), (rg1, b.y) with weights (1 - a), a
template <bool F>
__device__ __forceinline__ void mix_rgb(float a, float b1, float2 rg0, float2 rg1, float2 b, float2& rg,
                                        float& bl, float2 one)
{
    const float2 p0 = __fmul2_rn(f2(b1, b1), rg0);
    if (F) {
        rg = __ffma2_rn(f2(a, a), rg1, p0);
        bl = fmaf(a, b.y, b1 * b.x);
    } else {
        rg = sum2(p0, __fmul2_rn(f2(a, a), rg1), one);
        const float2 pb = __fmul2_rn(f2(b1, a), b);
        bl = __fadd_rn(pb.x, pb.y);
    }
}

// the interpolated colour of a tap from its pair record
template <bool F>
__device__ __forceinline__ void pair_rgb(const PairRec& R, float a, float2& rg, float& bl, float2 one)
{
    const float2 rg0 = rgb_unit(f2(pair_byte<0>(R.x), pair_byte<1>(R.x)));
    const float2 rg1 = rgb_unit(f2(pair_byte<0>(R.y), pair_byte<1>(R.y)));
    mix_rgb<F>(a, 1.0f - a, rg0, rg1, rgb_unit(f2(pair_byte<2>(R.x), pair_byte<2>(R.y))), rg, bl, one);
}

// ad_sum of an interpolated colour against minus the reference colour
__device__ __forceinline__ float ad_pair(float2 rg, float bl, float2 nref_rg, float nref_b)
{
    const float2 d = __ffma2_rn(nref_rg, f2(1.0f, 1.0f), rg);
    const float m2 = fminf(fabsf(bl + nref_b), 0.05f);
    const float2 m = f2(fminf(fabsf(d.x), 0.05f), fminf(fabsf(d.y), 0.05f));
    const float2 c = __ffma2_rn(m, f2(20.0f, 20.0f), __fmul2_rn(m, f2(PM_D005, PM_D005)));
    return c.x + c.y + fmaf(m2, 20.0f, m2 * PM_D005);
}

// the tap weight 0 <= a < 1 as floor(a 2^15) with bit 15 set, in both halves of a word
__device__ __forceinline__ uint32_t pair_weight(float a)
{
    const uint32_t u = __float_as_uint(__fadd_rd(a, 257.0f));   // ulp(257) = 2^-15
    return __byte_perm(u, u, 0x1010);
}

// The sign comparisons of a tap: each half of the differences has its bit 15 set when the weight has
// reached the threshold (no half borrows: a half of M is >= 0x8000, a threshold <= 0x8000).  With the
// weight rounded down and the threshold up, the answer is certain unless they differ by one
// (a half equal to 0x7fff): sign_unsure.
struct PairSigns {
    uint32_t yw, xz;
};
__device__ __forceinline__ PairSigns pair_signs(uint32_t M, const PairRec& R) { return PairSigns{M - R.z, M - R.w}; }
// max of the signed halves reaches 0x7fff: adding one to it changes its sign (a carry out of a low half
// of -1 can only raise a high half, which at worst asks for the exact signs without need)
__device__ __forceinline__ bool sign_unsure(uint32_t m) { return ((m + 0x00010001u) & ~m & 0x80008000u) != 0; }

// number of gradient components whose sign differs from the first view's (sb1: sign_bytes)
__device__ __forceinline__ int pair_mismatch(const PairSigns& d, uint32_t w0, uint32_t sb1)
{
    const uint32_t flips = __byte_perm(d.xz, d.yw, 0x7351);          // component c's flag at bit 8 c + 7
    const uint32_t s0 = (w0 >> 24) * 0x10204080u;                    // bit c of the four signs to bit 8 c + 7
    return __popc((flips ^ s0 ^ sb1) & 0x80808080u);
}

// the same from the interpolated gradient itself (g: gradient texel i)
template <bool F>
__device__ __forceinline__ int exact_mismatch(const float4* __restrict__ g, float a, uint32_t sb1)
{
    const float4 g0 = __ldg(g), g1 = __ldg(g + 1);
    const float2 a2 = f2(a, a), b2 = f2(1.0f - a, 1.0f - a);
    const float2 u = lerp2<F>(a2, b2, f2(g0.x, g0.y), f2(g1.x, g1.y)), v = lerp2<F>(a2, b2, f2(g0.z, g0.w), f2(g1.z, g1.w));
    return sign_mismatch(sb1, sign_bytes(make_float4(u.x, u.y, v.x, v.y)));
}

// support_weight of two samples
template <bool F>
__device__ __forceinline__ float2 support_weight2(float2 dx, float2 dy, float2 dz, float2 one)
{
    const float2 wr = f2(PM_GW_R, PM_GW_R), wg = f2(PM_GW_G, PM_GW_G), wb = f2(PM_GW_B, PM_GW_B);
    float2 g;
    if (F) g = __ffma2_rn(dz, wb, __ffma2_rn(dy, wg, __fmul2_rn(dx, wr)));
    else g = sum2(__fmul2_rn(dz, wb), sum2(__fmul2_rn(dy, wg), __fmul2_rn(dx, wr), one), one);
    const float2 x = f2(-fabsf(g.x) * 12.0f, -fabsf(g.y) * 12.0f);
    // expf_neg, element by element
    const float M = 12582912.0f;
    const float2 t = sum2(__fmul2_rn(x, f2(1.44269502162933349609375f, 1.44269502162933349609375f)), f2(M, M), one);
    const float2 n = __fadd2_rn(t, f2(-M, -M));
    float2 r = __ffma2_rn(n, f2(-0.693145751953125f, -0.693145751953125f), x);
    r = __ffma2_rn(n, f2(-1.428606765330187045e-06f, -1.428606765330187045e-06f), r);
    float2 p = f2(1.9841270113829523e-4f, 1.9841270113829523e-4f);
    p = __ffma2_rn(p, r, f2(1.3888889e-3f, 1.3888889e-3f));
    p = __ffma2_rn(p, r, f2(8.3333338e-3f, 8.3333338e-3f));
    p = __ffma2_rn(p, r, f2(4.1666668e-2f, 4.1666668e-2f));
    p = __ffma2_rn(p, r, f2(1.6666667e-1f, 1.6666667e-1f));
    p = __ffma2_rn(p, r, f2(0.5f, 0.5f));
    p = __ffma2_rn(p, r, f2(1.0f, 1.0f));
    p = __ffma2_rn(p, r, f2(1.0f, 1.0f));
    return f2(__int_as_float(__float_as_int(p.x) + (__float_as_int(t.x) << 23)),
              __int_as_float(__float_as_int(p.y) + (__float_as_int(t.y) << 23)));
}

// the matched columns s.x * qx + s.y * qy + s.z of two samples (byq = s.y * qy)
template <bool F>
__device__ __forceinline__ float2 match2(float4 s, float2 qx, float byq, float2 one)
{
    const float2 sx = f2(s.x, s.x), by = f2(byq, byq), sz = f2(s.z, s.z);
    return __fadd2_rn(F ? __ffma2_rn(sx, qx, by) : sum2(__fmul2_rn(sx, qx), by, one), sz);
}

// one colour channel (byte K of two words each) of two samples mixed with weights b1 = 1 - a, a
template <bool F, int K>
__device__ __forceinline__ float2 mix_channel2(uint32_t w0, uint32_t w1, uint32_t v0, uint32_t v1, float2 a, float2 b1, float2 one)
{
    const float2 c0 = rgb_unit(f2(pair_byte<K>(w0), pair_byte<K>(w1))), c1 = rgb_unit(f2(pair_byte<K>(v0), pair_byte<K>(v1)));
    const float2 p0 = __fmul2_rn(b1, c0);
    return F ? __ffma2_rn(a, c1, p0) : sum2(__fmul2_rn(a, c1), p0, one);
}

// fmin(|d|, 0.05) / 0.05 of two samples (ad_sum)
__device__ __forceinline__ float2 trunc2(float2 d)
{
    const float2 m = f2(fminf(fabsf(d.x), 0.05f), fminf(fabsf(d.y), 0.05f));
    return __ffma2_rn(m, f2(20.0f, 20.0f), __fmul2_rn(m, f2(PM_D005, PM_D005)));
}

// one window sample of patch_eval_census at (qx, row of q1) whose matched column p2x lies in the image
template <bool F>
__device__ __forceinline__ void eval_one(const ViewData& V, uintptr_t base, const float4* __restrict__ g2, float4 q,
                                         float4 in, float p2x, float& census, float& wsum)
{
    const float w = support_weight<F>(q.x - in.x, q.y - in.y, q.z - in.z);
    // 0 <= t <= W: the floor is the integer part of t + 2^23 rounded down
    const float t = (p2x + 0.5f) - 0.5f;
    const float fm = __fadd_rd(t, 8388608.0f);
    const float a = t - (fm - 8388608.0f);
    const PairRec R = __ldg(reinterpret_cast<const uint4*>(base + (uintptr_t)__float_as_uint(fm) * 16u));
    const PairSigns d = pair_signs(pair_weight(a), R);
    int nm = pair_mismatch(d, R.x, __float_as_uint(q.w));
    if (sign_unsure(__vmaxs2(d.yw, d.xz)))
        nm = exact_mismatch<F>(g2 + (__float_as_int(fm) - 0x4B000000), a, __float_as_uint(q.w));
    float2 rg;
    float bl;
    pair_rgb<F>(R, a, rg, bl, V.one);
    // cost + 0.875f * (0.25f * n): the product 0.21875 n is exact, so one fma rounds the same
    const float cost = fmaf(0.21875f, (float)nm, PM_K033_8 * ad_pair(rg, bl, f2(-q.x, -q.y), -q.z));
    census = F ? fmaf(w, cost, census) : census + w * cost;
    wsum += w;
}

// a row of patch_eval_pair, two samples per packed instruction; IN: every matched column, one past
// the end included, lies in the image (otherwise: is finite; samples outside get weight 0).
// Returns the maximum of the sign comparisons for sign_unsure.
template <bool F, bool IN>
__device__ __forceinline__ uint32_t eval_row(float& census, float& wsum, float2 one, uintptr_t base,
                                             const float4* __restrict__ q1, float4 in, float4 s, float byq, float qx0,
                                             float qx1, float fW)
{
    uint32_t sure = 0x80008000u;
    for (float2 qx = f2(qx0, qx0 + 1.0f); qx.x <= qx1; qx = __fadd2_rn(qx, f2(2.0f, 2.0f)), q1 += 2) {
        const float4 q0 = __ldg(q1), qn = __ldg(q1 + 1);
        const float2 p = match2<F>(s, qx, byq, one);
        float2 t = __fadd2_rn(__fadd2_rn(p, f2(0.5f, 0.5f)), f2(-0.5f, -0.5f));
        if (!IN) t = f2(fminf(fmaxf(t.x, 0.0f), fW), fminf(fmaxf(t.y, 0.0f), fW));
        // 0 <= t <= W: the floor is the integer part of t + 2^23 rounded down
        const float2 fm = __fadd2_rd(t, f2(8388608.0f, 8388608.0f));
        const PairRec R0 = __ldg(reinterpret_cast<const uint4*>(base + (uintptr_t)__float_as_uint(fm.x) * 16u));
        const PairRec R1 = __ldg(reinterpret_cast<const uint4*>(base + (uintptr_t)__float_as_uint(fm.y) * 16u));
        const float2 a = __ffma2_rn(__fadd2_rn(fm, f2(-8388608.0f, -8388608.0f)), f2(-1.0f, -1.0f), t);
        const float2 b1 = __ffma2_rn(a, f2(-1.0f, -1.0f), f2(1.0f, 1.0f));
        float2 w = support_weight2<F>(f2(q0.x - in.x, qn.x - in.x), f2(q0.y - in.y, qn.y - in.y),
                                      f2(q0.z - in.z, qn.z - in.z), one);
        if (!IN && !(p.x >= 0.0f && p.x < fW)) w.x = 0.0f;
        if (!(qx.y <= qx1 && (IN || (p.y >= 0.0f && p.y < fW)))) w.y = 0.0f;   // an odd row's last pair has one sample
        const PairSigns d0 = pair_signs(pair_weight(a.x), R0), d1 = pair_signs(pair_weight(a.y), R1);
        sure = __vimax3_s16x2(__vimax3_s16x2(sure, d0.yw, d0.xz), d1.yw, d1.xz);
        const float2 nm = f2((float)pair_mismatch(d0, R0.x, __float_as_uint(q0.w)),
                             (float)pair_mismatch(d1, R1.x, __float_as_uint(qn.w)));
        float2 v = mix_channel2<F, 0>(R0.x, R1.x, R0.y, R1.y, a, b1, one);
        float2 ad = trunc2(f2(v.x - q0.x, v.y - qn.x));
        v = mix_channel2<F, 1>(R0.x, R1.x, R0.y, R1.y, a, b1, one);
        ad = __fadd2_rn(ad, trunc2(f2(v.x - q0.y, v.y - qn.y)));
        v = mix_channel2<F, 2>(R0.x, R1.x, R0.y, R1.y, a, b1, one);
        ad = __fadd2_rn(ad, trunc2(f2(v.x - q0.z, v.y - qn.z)));
        // cost + 0.875f * (0.25f * n): the product 0.21875 n is exact, so one fma rounds the same
        const float2 cost = __ffma2_rn(f2(0.21875f, 0.21875f), nm, __fmul2_rn(f2(PM_K033_8, PM_K033_8), ad));
        if (F) {
            census = fmaf(w.y, cost.y, fmaf(w.x, cost.x, census));
        } else {
            const float2 wc = __fmul2_rn(w, cost);
            census = __fadd_rn(__fadd_rn(census, wc.x), wc.y);
        }
        wsum = (wsum + w.x) + w.y;
    }
    return sure;
}

// patch_eval_census (:661-736) over pair records.
//
// The census only grows (every term is >= 0), so the source's exit test after each sample,
// `census / bilw >= mincost` with a sample counted (:724), is decided by the census at the row's
// end; it is tested there as census >= exit_threshold(mincost, bilw).
//
// Rows run two samples per packed instruction; p2x is monotone along a row, so its two ends decide for
// the warp whether samples can lie outside the image, or a column can be non-finite.  Such
// rows, and rows where some sign was unsure, run sample by sample.  From column 256 on a tap
// weight is a multiple of 2^-15 and no sign is unsure.
template <bool F>
__device__ __forceinline__ float patch_eval_pair(const ViewData& V, int px, int py, float4 s, float mincost)
{
    const float cx = (float)px, cy = (float)py;
    if (!plane_usable(s, cx, cy, V.W)) return 1e5f;
    const int W = V.W;
    const float2 one = V.one;
    const float4 in = __ldg(V.row1(py) + px);
    const float thr = exit_threshold(mincost, in.w);
    float wsum = 0.0f, census = 0.0f;
    const int r = V.r;
    const int dy0 = max(-r, -py), dy1 = min(r, V.H - 1 - py);
    const int dx0 = max(-r, -px), dx1 = min(r, W - 1 - px);
    const float fW = (float)W;
    const float qx0 = cx + (float)dx0, qx1 = cx + (float)dx1;
    float qy = cy + (float)dy0;
    for (int iy = py + dy0; iy <= py + dy1; iy++, qy += 1.0f) {
        const float byq = s.y * qy;
        const float4* __restrict__ q1 = V.row1c(iy) + px + dx0;
        // column c of the row is at base + 16 * (bits of the float 2^23 + c)
        const uintptr_t base = reinterpret_cast<uintptr_t>(V.row2p(iy)) - (uintptr_t)0x4B000000u * 16u;
        const float2 pe = match2<F>(s, f2(qx0, qx1 + 1.0f), byq, one);
        const float plo = fminf(pe.x, pe.y);
        const float census0 = census, wsum0 = wsum;
        const bool finite = fin(pe.x) && fin(pe.y);
        const unsigned lanes = __activemask();
        bool single = true;
        if (__all_sync(lanes, pe.x >= 0.0f && pe.y >= 0.0f && pe.x < fW && pe.y < fW)) {
            single = sign_unsure(eval_row<F, true>(census, wsum, one, base, q1, in, s, byq, qx0, qx1, fW)) && plo < 256.0f;
        } else if (__all_sync(lanes, finite)) {
            if (!__any_sync(lanes, plo < fW && fmaxf(pe.x, pe.y) >= 0.0f)) continue;
            single = sign_unsure(eval_row<F, false>(census, wsum, one, base, q1, in, s, byq, qx0, qx1, fW)) && plo < 256.0f;
        }
        if (single) {
            census = census0;
            wsum = wsum0;
            const float4* __restrict__ g2 = V.row2(iy) + V.plane;
            for (float qx = qx0; qx <= qx1; qx += 1.0f, q1++) {
                const float p2x = F ? fmaf(s.x, qx, byq) + s.z : s.x * qx + byq + s.z;
                if (p2x < 0 || p2x >= fW) continue;
                const float4 q = __ldg(q1);   // compact texel
                if (p2x == p2x) {
                    eval_one<F>(V, base, g2, q, in, p2x, census, wsum);
                } else {   // a NaN column reads the positive quiet NaN: full colour cost, positive signs
                    const float w = support_weight<F>(q.x - in.x, q.y - in.y, q.z - in.z);
                    const float cost = fmaf(0.21875f, (float)sign_mismatch(__float_as_uint(q.w), 0u), PM_K033_8 * 3.0f);
                    census = F ? fmaf(w, cost, census) : census + w * cost;
                    wsum += w;
                }
            }
        }
        if (census >= thr && wsum > 0.0f) return 1.0f;
    }
    if (wsum <= 1.0f) return 1.1f;
    return census / wsum;
}

// The cost of a Gauss-Newton tap, k1 * ad + x * 0.25 * n (:361-370).  The source's sum is a double
// one rounded to float; here one fma.  They agree for colours k / 255: a nonzero truncated difference is
// then >= 2^-33 (the reference colour is 0 or >= 2^-8 in magnitude, the tap weights are multiples
// of 2^-25), so the colour term is 0 or >= 2^-34 of the weight; the double sum is inexact only when
// the colour term is below 2^-28 of the sum, and then it cannot land on a midpoint of two floats
// unless the colour term is below 2^-53 of it.
__device__ __forceinline__ float tap_cost(float k1, float x, float ad, int n) { return fmaf(x, (float)n, k1 * ad); }

// the sums of a Gauss-Newton step; J holds twice the source's (its factor 0.5 is taken out of the
// loop: scaling by a power of two commutes with rounding).  The sums are never -0, so a sample
// whose terms are +-0 leaves them unchanged.
struct KltSums {
    float J0, J1, J2, h00, h01, h02, h11, h12, h22;
};

// sum + v.x * f.x, then + v.y * f.y
template <bool F>
__device__ __forceinline__ float accum2(float sum, float2 v, float2 f)
{
    if (F) return fmaf(v.y, f.y, fmaf(v.x, f.x, sum));
    const float2 p = __fmul2_rn(v, f);
    return __fadd_rn(__fadd_rn(sum, p.x), p.y);
}

// the costs of one tap of two samples: colour bytes of the texels on its left (l0, l1) and right (r0, r1)
template <bool F>
__device__ __forceinline__ float2 tap2(uint32_t l0, uint32_t l1, uint32_t r0, uint32_t r1, float2 a, float2 b1, float2 nr,
                                       float2 ng, float2 nb, float2 k1, float2 x, int n0, int n1, float2 one)
{
    float2 ad = trunc2(__fadd2_rn(mix_channel2<F, 0>(l0, l1, r0, r1, a, b1, one), nr));
    ad = __fadd2_rn(ad, trunc2(__fadd2_rn(mix_channel2<F, 1>(l0, l1, r0, r1, a, b1, one), ng)));
    ad = __fadd2_rn(ad, trunc2(__fadd2_rn(mix_channel2<F, 2>(l0, l1, r0, r1, a, b1, one), nb)));
    return __ffma2_rn(x, f2((float)n0, (float)n1), __fmul2_rn(k1, ad));
}

// one tap of two samples on its own: the coordinate u + 0.5 and its floor as the source forms them, the
// column clamped to the padded row, where the records hold the edge texels that the source's
// clamp gives, the signs from the gradients themselves
template <bool F>
__device__ __forceinline__ float2 tap_alone2(float2 u, const ViewData& V, const float4* __restrict__ row2,
                                             const float4* __restrict__ g2, float2 nr, float2 ng, float2 nb, uint32_t s0,
                                             uint32_t sn, float2 k1, float2 x)
{
    const float2 t = __fadd2_rn(__fadd2_rn(u, f2(0.5f, 0.5f)), f2(-0.5f, -0.5f));
    const float2 fl = f2(floorf(t.x), floorf(t.y));
    const float2 a = __ffma2_rn(fl, f2(-1.0f, -1.0f), t);
    const float2 b1 = __ffma2_rn(a, f2(-1.0f, -1.0f), f2(1.0f, 1.0f));
    const float fW = (float)V.W;
    const int c0 = (int)fminf(fmaxf(fl.x, -2.0f), fW), cn = (int)fminf(fmaxf(fl.y, -2.0f), fW);
    const uint4* row = reinterpret_cast<const uint4*>(row2);
    const PairRec A = __ldg(row + c0), B = __ldg(row + cn);
    return tap2<F>(A.x, B.x, A.y, B.y, a, b1, nr, ng, nb, k1, x, exact_mismatch<F>(g2 + c0, a.x, s0),
                   exact_mismatch<F>(g2 + cn, a.y, sn), V.one);
}

// patch_census_klt2 (:326-410) over pair records, two samples of a row per packed instruction.
//
// The three taps at t - 1, t, t + 1 (each coordinate formed as the source forms it) mostly have the floors
// f - 1, f, f + 1: they then read three consecutive records, whose four texels are decoded once,
// each with its own weight (the weights differ in the last bit near powers of two).  The weights decide
// whether that holds: t - f in [0, 1) exactly if f is t's floor.  The column f is clamped
// to the padded row, where records beyond the image hold edge texels, as the source's clamp gives.
// Where a weight is out of range (floors that do not chain, a non-finite column) or a sign unsure, each
// tap of the pair is read on its own.
template <bool F>
__device__ __forceinline__ float4 klt2_pair(const ViewData& V, int px, int py, float4 s)
{
    // a NaN plane has no column: no sample counts, the 0 / 0 solution is NaN
    if (s.x != s.x || s.y != s.y || s.z != s.z) return f4(qnan(), qnan(), qnan(), s.w - 1e5f);
    const float cxf = (float)px, cyf = (float)py;
    const float2 one = V.one;
    KltSums A = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    const float4 c1 = __ldg(V.row1(py) + px);
    const int r = V.r;
    const int dy0 = max(-r, -py), dy1 = min(r, V.H - 1 - py);
    const int dx0 = max(-r, 1 - px), dx1 = min(r, V.W - 2 - px);   // the 3-point cost needs 1 <= qx < W - 1
    const float qx0 = cxf + (float)dx0, qx1 = cxf + (float)dx1;
    const float MAGIC = 12582912.0f;   // 1.5 * 2^23: MAGIC + t rounded down is MAGIC + floor(t) for |t| < 2^22
    const float first = MAGIC - 3.0f, last = MAGIC + (float)(V.W + 1);
    float qy = cyf + (float)dy0;
    for (int iy = py + dy0; iy <= py + dy1; iy++, qy += 1.0f) {
        const float byq = s.y * qy;
        const float4* __restrict__ q1 = V.row1c(iy) + px + dx0;
        // column c of the row is at base + 16 * (bits of the float MAGIC + c)
        const uintptr_t base = reinterpret_cast<uintptr_t>(V.row2p(iy)) - (uintptr_t)0x4B400000u * 16u;
        for (float2 qx = f2(qx0, qx0 + 1.0f); qx.x <= qx1; qx = __fadd2_rn(qx, f2(2.0f, 2.0f)), q1 += 2) {
            const float4 q0 = __ldg(q1), qn = __ldg(q1 + 1);
            const float2 p = match2<F>(s, qx, byq, one);
            const float2 h = f2(0.5f, 0.5f), mh = f2(-0.5f, -0.5f);
            const float2 t0 = __fadd2_rn(__fadd2_rn(p, h), mh);
            const float2 tm = __fadd2_rn(__fadd2_rn(__fadd2_rn(p, f2(-1.0f, -1.0f)), h), mh);
            const float2 tp = __fadd2_rn(__fadd2_rn(__fadd2_rn(p, f2(1.0f, 1.0f)), h), mh);
            const float2 fm = __fadd2_rd(t0, f2(MAGIC, MAGIC));
            const uint4* b0 =
                reinterpret_cast<const uint4*>(base + (uintptr_t)__float_as_uint(fminf(fmaxf(fm.x, first), last)) * 16u);
            const uint4* bn =
                reinterpret_cast<const uint4*>(base + (uintptr_t)__float_as_uint(fminf(fmaxf(fm.y, first), last)) * 16u);
            const PairRec Am = __ldg(b0 - 1), A0 = __ldg(b0), Ap = __ldg(b0 + 1);
            const PairRec Bm = __ldg(bn - 1), B0 = __ldg(bn), Bp = __ldg(bn + 1);
            const float2 nf = __ffma2_rn(fm, f2(-1.0f, -1.0f), f2(MAGIC, MAGIC));   // -f
            const float2 a0 = __fadd2_rn(t0, nf), am = __fadd2_rn(tm, __fadd2_rn(nf, f2(1.0f, 1.0f))),
                         ap = __fadd2_rn(tp, __fadd2_rn(nf, f2(-1.0f, -1.0f)));
            const float2 nr = f2(c1.x - q0.x, c1.x - qn.x), ng = f2(c1.y - q0.y, c1.y - qn.y),
                         nb = f2(c1.z - q0.z, c1.z - qn.z);   // minus the colour differences
            const uint32_t s0 = __float_as_uint(q0.w), sn = __float_as_uint(qn.w);
            const PairSigns dm = pair_signs(pair_weight(am.x), Am), d0 = pair_signs(pair_weight(a0.x), A0),
                            dp = pair_signs(pair_weight(ap.x), Ap);
            const PairSigns em = pair_signs(pair_weight(am.y), Bm), e0 = pair_signs(pair_weight(a0.y), B0),
                            ep = pair_signs(pair_weight(ap.y), Bp);
            const int nm0 = pair_mismatch(dm, Am.x, s0), n00 = pair_mismatch(d0, A0.x, s0), np0 = pair_mismatch(dp, Ap.x, s0);
            const int nm1 = pair_mismatch(em, Bm.x, sn), n01 = pair_mismatch(e0, B0.x, sn), np1 = pair_mismatch(ep, Bp.x, sn);
            const uint32_t ma = __vimax3_s16x2(__vimax3_s16x2(dm.yw, dm.xz, d0.yw), __vimax3_s16x2(d0.xz, dp.yw, dp.xz), em.yw);
            const uint32_t mb = __vimax3_s16x2(__vimax3_s16x2(em.xz, e0.yw, e0.xz), ep.yw, ep.xz);
            // a weight in [0, 1) has bits below 1.0f's; a negative one or a NaN has not
            const uint32_t wa = __vimax3_u32(__float_as_uint(am.x), __float_as_uint(a0.x), __float_as_uint(ap.x));
            const uint32_t wb = __vimax3_u32(__float_as_uint(am.y), __float_as_uint(a0.y), __float_as_uint(ap.y));
            const bool alone = sign_unsure(__vmaxs2(ma, mb)) || max(wa, wb) >= 0x3f800000u;
            float2 w = support_weight2<F>(nr, ng, nb, one);
            w.y = qx.y <= qx1 ? w.y : 0.0f;   // an odd row's last pair has one sample
            const float2 k1 = __fmul2_rn(w, f2(PM_K033_8, PM_K033_8));
            const float2 x = __fmul2_rn(w, f2(0.21875f, 0.21875f));   // (w * 0.875f) * 0.25, exact scaling
            float2 Cm = tap2<F>(Am.x, Bm.x, A0.x, B0.x, am, __ffma2_rn(am, f2(-1.0f, -1.0f), f2(1.0f, 1.0f)), nr, ng, nb, k1,
                                x, nm0, nm1, one);
            float2 C = tap2<F>(A0.x, B0.x, A0.y, B0.y, a0, __ffma2_rn(a0, f2(-1.0f, -1.0f), f2(1.0f, 1.0f)), nr, ng, nb, k1,
                               x, n00, n01, one);
            float2 Cp = tap2<F>(A0.y, B0.y, Ap.y, Bp.y, ap, __ffma2_rn(ap, f2(-1.0f, -1.0f), f2(1.0f, 1.0f)), nr, ng, nb, k1,
                                x, np0, np1, one);
            if (alone) {
                const float4* __restrict__ row2 = V.row2p(iy);
                const float4* __restrict__ g2 = V.row2(iy) + V.plane;
                Cm = tap_alone2<F>(__fadd2_rn(p, f2(-1.0f, -1.0f)), V, row2, g2, nr, ng, nb, s0, sn, k1, x);
                C = tap_alone2<F>(p, V, row2, g2, nr, ng, nb, s0, sn, k1, x);
                Cp = tap_alone2<F>(__fadd2_rn(p, f2(1.0f, 1.0f)), V, row2, g2, nr, ng, nb, s0, sn, k1, x);
                // a non-finite column reads NaN texels for all three taps: equal costs, nothing added
                if (!fin(p.x)) w.x = Cm.x = C.x = Cp.x = 0.0f;
                if (!fin(p.y)) w.y = Cm.y = C.y = Cp.y = 0.0f;
            }
            // the update of :394-402 without a branch (KltSums)
            const float2 curv = __ffma2_rn(C, f2(-2.0f, -2.0f), __fadd2_rn(Cp, Cm));   // 2 C is exact
            const float2 wt = f2(curv.x > 0.0f ? w.x : 0.0f, curv.y > 0.0f ? w.y : 0.0f);
            const float2 t = __fmul2_rn(wt, __ffma2_rn(Cp, f2(-1.0f, -1.0f), Cm)), sc = __fmul2_rn(wt, curv);
            const float2 qy2 = f2(qy, qy);
            A.J0 = accum2<F>(A.J0, t, qx);
            A.J1 = accum2<F>(A.J1, t, qy2);
            A.J2 = (A.J2 + t.x) + t.y;
            A.h00 = accum2<F>(A.h00, sc, __fmul2_rn(qx, qx));
            A.h01 = accum2<F>(A.h01, sc, __fmul2_rn(qx, qy2));
            A.h02 = accum2<F>(A.h02, sc, qx);
            A.h11 = accum2<F>(A.h11, sc, f2(qy * qy, qy * qy));
            A.h12 = accum2<F>(A.h12, sc, qy2);
            A.h22 = (A.h22 + sc.x) + sc.y;
        }
    }
    const float3 d = lusolve(A.h00, A.h01, A.h02, A.h11, A.h12, A.h22, make_float3(A.J0 * 0.5f, A.J1 * 0.5f, A.J2 * 0.5f));
    return f4(s.x - d.x, s.y - d.y, s.z - d.z, s.w - 1e5f);
}

// the window functions of a variant: pair-plane loops, or the general ones (GEN, which count)
template <bool F, bool COUNT, bool GEN>
__device__ __forceinline__ float patch_eval(const ViewData& V, int px, int py, float4 s, float mincost, Counters& cnt)
{
    if (GEN) return patch_eval_general<F, COUNT>(V, px, py, s, mincost, cnt);
    return patch_eval_pair<F>(V, px, py, s, mincost);
}

template <bool F, bool COUNT, bool GEN>
__device__ __forceinline__ float4 klt2(const ViewData& V, int px, int py, float4 s, Counters& cnt)
{
    if (GEN) return klt2_general<F, COUNT>(V, px, py, s, cnt);
    return klt2_pair<F>(V, px, py, s);
}

}  // namespace pm
