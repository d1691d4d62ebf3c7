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
// Arithmetic.  The pair loops are bound by instruction issue.  Packed FP32 instructions do
// not help there: measured on B200, FFMA2 / FMUL2 / FADD2 hold the scheduler for 2 cycles (3 when all
// three operands are register pairs), as two scalar instructions do, so the loops are scalar.
// Every operation rounds as the scalar restatement does, so results equal it bit for bit.
#pragma once

#include "pm_device.cuh"

namespace pm {

constexpr int TEX_PAD = 4;     // replicated columns on each side of a texel row
constexpr int TEX_PLANES = 4;  // colour, gradient, compact, pair

// The samples over which a warp walks the windows it shares (pm_warp.cuh), row by row: the 2 r + 1 columns and rows
// from (px - r, py - r), those outside the image with weight 0; or, where the window of every pixel of the
// PW x PH that have one spans the image (at most r + 1 columns or rows), the image's (17x9, r = 32: 153
// samples a window, not 4225).
struct WindowSpan {
    int cols, rows;
    unsigned recip;       // ceil(2^20 / cols): row(e) is exact for e < cols rows, both <= 65
    int xmask, ymask;     // 0: all windows start at column (row) 0, else -1
    __host__ __device__ WindowSpan(int W, int H, int r, int PW, int PH)
        : cols(PW <= r + 1 ? W : 2 * r + 1), rows(PH <= r + 1 ? H : 2 * r + 1), recip(((1u << 20) + cols - 1) / cols),
          xmask(PW <= r + 1 ? 0 : -1), ymask(PH <= r + 1 ? 0 : -1)
    {
    }
    WindowSpan() = default;
    __device__ __forceinline__ int row(int e) const { return (int)(((unsigned)e * recip) >> 20); }
    // first column and row of a pixel's window
    __device__ __forceinline__ int left(int px, int r) const { return (px - r) & xmask; }
    __device__ __forceinline__ int top(int py, int r) const { return (py - r) & ymask; }
};

struct ViewData {
    const float4* __restrict__ t1;   // first view: colour plane, gradient at + plane, compact at + 2 plane, pair at + 3 plane
    const float4* __restrict__ t2;   // second view
    int W, H, r, P;                  // P = W + 2 * TEX_PAD texels per row
    int plane;                       // H * P
    const int* gen1;                 // the views' flags: read by the general loops (after the planes)
    const int* gen2;
    WindowSpan span;
    // colour texel (compact texel) of column 0 of row y
    __device__ __forceinline__ const float4* row1(int y) const { return t1 + (size_t)y * P + TEX_PAD; }
    __device__ __forceinline__ const float4* row1c(int y) const { return t1 + 2 * (size_t)plane + (size_t)y * P + TEX_PAD; }
    __device__ __forceinline__ const float4* row2(int y) const { return t2 + (size_t)y * P + TEX_PAD; }
    // pair record of column 0 of row y
    __device__ __forceinline__ const float4* row2p(int y) const { return t2 + 3 * (size_t)plane + (size_t)y * P + TEX_PAD; }
};

// Pair record of columns (i, i + 1), one 16-byte word group:
//   x  bytes r, g, b of texel i
//   y  bytes r, g, b of texel i + 1
//   z  sign words of gradient components 1 (low half) and 3 (high half)
//   w  sign words of components 0 and 2
// With A = a 2^15 the tap weight in units of 2^-15, the interpolated component has the sign
// of texel i for A < threshold and the other sign from there on (pair_sign_word); bit 15 of
// A + sign word (mod 2^16) is that sign.
typedef uint4 PairRec;

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
    const float w = support_weight_any<F>(q.x - in.x, q.y - in.y, q.z - in.z);
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
            const float w1 = support_weight_any<F>(val1.x, val1.y, val1.z);
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
//
// The loops serve two window models, their last template parameter: PMH, the functions of pmhstereo.cl
// that the comments cite, and VPM, those of VPMStereo.cl (patch_eval_census :200-258, patch_census_klt
// :117-198; pm_vpm.cu), which differ in the support weight, the mix of the two costs, the reference colour
// of a Gauss-Newton tap and in taking every Gauss-Newton sample.
enum Model { PMH, VPM };

// support weight of a colour difference
template <bool F, Model M>
__device__ __forceinline__ float pair_support(float dx, float dy, float dz)
{
    return expf_neg(-fabsf(gray_dot<F>(dx, dy, dz)) * (M == PMH ? 12.0f : 8.0f));
}

// the two parts of a sample's weighted cost, PMH: their sum (one product), VPM: colour and census part
struct SampleTerms {
    float a, b;
};
template <bool F, Model M>
__device__ __forceinline__ SampleTerms sample_terms(float w, float ad, int n)
{
    if (M == VPM) return SampleTerms{w * 0.05f * 0.33f * ad, w * (1.0f - 0.05f) * 0.25f * (float)n};
    // K ad + 0.875f * (0.25f * n): the product 0.21875 n is exact, so one fma rounds the same
    const float cost = fmaf(0.21875f, (float)n, PM_K033_8 * ad);
    return SampleTerms{F ? cost : w * cost, 0.0f};
}
// adds a sample to the sums
template <bool F, Model M>
__device__ __forceinline__ void add_terms(float& census, float& wsum, float w, SampleTerms s)
{
    if (M == VPM) census = (census + s.a) + s.b;
    else census = F ? fmaf(w, s.a, census) : census + s.a;
    wsum += w;
}

// byte K of a record word / 255, correctly rounded, in one permute and one fma: the byte twice, in bits
// 8-23 of an otherwise zero word, is x = 257 byte 2^-141 as a float (exponent field 0 or 1, one
// linear scale).  RN(x RGB) for RGB = RN(2^141 / 65535) is RN(byte / 255) except where x RGB is
// a tie, which rounds up in byte / 255 (its binary expansion goes on); the addend x, 2^125 times
// smaller, decides the ties.  Equal to the division for all 256 bytes.
#define PM_RGB 0x1.0001p+125f
template <int K>
__device__ __forceinline__ float pair_unit(uint32_t w)
{
    const float x = __uint_as_float(__byte_perm(w, 0u, 0x4004 | (K << 4) | (K << 8)));
    return fmaf(x, PM_RGB, x);
}

// T0 b1 + T1 a, the bilinear mix with b1 = 1 - a
template <bool F>
__device__ __forceinline__ float mix(float a, float b1, float t0, float t1)
{
    return F ? fmaf(a, t1, b1 * t0) : b1 * t0 + a * t1;
}

// fmin(|d|, 0.05) / 0.05 (ad_sum)
__device__ __forceinline__ float trunc_ad(float d)
{
    const float m = fminf(fabsf(d), 0.05f);
    return fmaf(m, 20.0f, m * PM_D005);
}

// the tap weight 0 <= a < 1 as floor(a 2^15) in both halves of a word
__device__ __forceinline__ uint32_t pair_weight(float a)
{
    const uint32_t u = __float_as_uint(__fadd_rd(a, 256.0f));   // ulp(256) = 2^-15
    return __byte_perm(u, u, 0x1010);
}

__device__ __forceinline__ uint32_t add_u16x2(uint32_t a, uint32_t b)
{
    uint32_t r;
    asm("add.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// The signs of a tap's interpolated gradient.  With the weight rounded down and the threshold up to
// multiples of 2^-15, a sign is certain unless weight + 1 = threshold, where the low 15 bits of its
// half are all ones.
struct PairSigns {
    uint32_t yw, xz;
};
__device__ __forceinline__ PairSigns pair_signs(uint32_t A, const PairRec& R)
{
    return PairSigns{add_u16x2(A, R.z), add_u16x2(A, R.w)};
}
// number of components whose sign differs from the first view's (sb1: sign_bytes)
__device__ __forceinline__ int pair_mismatch(const PairSigns& d, uint32_t sb1)
{
    return __popc((__byte_perm(d.xz, d.yw, 0x7351) ^ sb1) & 0x80808080u);
}
// the largest half so far, each with its bit 15 set: 0xffff when some sign was unsure
__device__ __forceinline__ uint32_t unsure_max(uint32_t m, const PairSigns& d)
{
    return __vimax3_u16x2(m, d.yw | 0x80008000u, d.xz | 0x80008000u);
}
__device__ __forceinline__ bool unsure(uint32_t m) { return (m >> 16) == 0xffffu || (m & 0xffffu) == 0xffffu; }

// the number of mismatches from the interpolated gradient itself (g: gradient texel i)
template <bool F>
__device__ __forceinline__ int exact_mismatch(const float4* __restrict__ g, float a, uint32_t sb1)
{
    const float4 g0 = __ldg(g), g1 = __ldg(g + 1);
    const float2 a2 = f2(a, a), b2 = f2(1.0f - a, 1.0f - a);
    const float2 u = lerp2<F>(a2, b2, f2(g0.x, g0.y), f2(g1.x, g1.y)), v = lerp2<F>(a2, b2, f2(g0.z, g0.w), f2(g1.z, g1.w));
    return sign_mismatch(sb1, sign_bytes(make_float4(u.x, u.y, v.x, v.y)));
}

// the matched column s.x qx + s.y qy + s.z (byq = s.y qy)
template <bool F>
__device__ __forceinline__ float match(float4 s, float qx, float byq)
{
    return F ? fmaf(s.x, qx, byq) + s.z : s.x * qx + byq + s.z;
}

// One sample of patch_eval_census (:690-722): compact texel q of the first view, matched column p2x whose
// t = (p2x + 0.5) - 0.5 lies in [0, W].  The column's texel is at base + 16 * (bits of the float
// 2^23 + column).  Returns the sample's colour cost (ad_sum) and the signs.
template <bool F>
__device__ __forceinline__ float eval_sample_pair(uintptr_t base, float4 q, float t, PairSigns& d, float& a)
{
    const float fm = __fadd_rd(t, 8388608.0f);   // 2^23 + floor(t)
    a = t - (fm - 8388608.0f);
    const PairRec R = __ldg(reinterpret_cast<const uint4*>(base + (uintptr_t)__float_as_uint(fm) * 16u));
    d = pair_signs(pair_weight(a), R);
    const float b1 = 1.0f - a;
    float ad = trunc_ad(mix<F>(a, b1, pair_unit<0>(R.x), pair_unit<0>(R.y)) - q.x);
    ad = ad + trunc_ad(mix<F>(a, b1, pair_unit<1>(R.x), pair_unit<1>(R.y)) - q.y);
    ad = ad + trunc_ad(mix<F>(a, b1, pair_unit<2>(R.x), pair_unit<2>(R.y)) - q.z);
    return ad;
}

// a row of patch_eval_pair.  IN: every matched column lies in the image; otherwise all are finite and
// samples outside get weight 0.  SURE: no sign can be unsure; otherwise returns unsure_max.
template <bool F, bool IN, bool SURE, Model M>
__device__ __forceinline__ uint32_t eval_row(float& census, float& wsum, uintptr_t base, const float4* __restrict__ q1,
                                             float4 in, float4 s, float byq, float qx0, float qx1, float fW)
{
    uint32_t m = 0;
    for (float qx = qx0; qx <= qx1; qx += 1.0f, q1++) {
        const float4 q = __ldg(q1);
        const float p2x = match<F>(s, qx, byq);
        float t = (p2x + 0.5f) - 0.5f;
        if (!IN) t = fminf(fmaxf(t, 0.0f), fW);
        float w = pair_support<F, M>(q.x - in.x, q.y - in.y, q.z - in.z);
        if (!IN) w = p2x >= 0.0f && p2x < fW ? w : 0.0f;
        PairSigns d;
        float a;
        const float ad = eval_sample_pair<F>(base, q, t, d, a);
        if (!SURE) m = unsure_max(m, d);
        add_terms<F, M>(census, wsum, w, sample_terms<F, M>(w, ad, pair_mismatch(d, __float_as_uint(q.w))));
    }
    return m;
}

// A row iy of patch_eval_pair, for the lanes that call it together.  p2x is monotone along a row, so its
// two ends decide, for the warp, whether samples can lie outside the image or a column be
// non-finite.  From column 256 on a tap weight is a multiple of 2^-15 and no sign is unsure.
// Rows with a non-finite column and rows where some sign was unsure run sample by sample with the
// signs from the gradients.
template <bool F, Model M = PMH>
__device__ __forceinline__ void eval_row_pixel(const ViewData& V, int iy, float4 s, float byq, float4 in, float qx0,
                                               float qx1, float& census, float& wsum)
{
    const float fW = (float)V.W;
    const float4* __restrict__ q1 = V.row1c(iy) + (int)qx0;
    const uintptr_t base = reinterpret_cast<uintptr_t>(V.row2p(iy)) - (uintptr_t)0x4B000000u * 16u;
    const float pa = match<F>(s, qx0, byq), pb = match<F>(s, qx1, byq);
    const float plo = fminf(pa, pb), phi = fmaxf(pa, pb);
    const float census0 = census, wsum0 = wsum;
    const bool in_image = pa >= 0.0f && pb >= 0.0f && phi < fW;
    const bool sure = in_image && plo >= 256.0f;
    const unsigned lanes = __activemask();
    bool single = true;
    if (__all_sync(lanes, sure)) {
        eval_row<F, true, true, M>(census, wsum, base, q1, in, s, byq, qx0, qx1, fW);
        single = false;
    } else if (__all_sync(lanes, in_image)) {
        single = unsure(eval_row<F, true, false, M>(census, wsum, base, q1, in, s, byq, qx0, qx1, fW)) && !sure;
    } else if (__all_sync(lanes, fin(pa) && fin(pb))) {
        if (!__any_sync(lanes, plo < fW && phi >= 0.0f)) return;
        single = unsure(eval_row<F, false, false, M>(census, wsum, base, q1, in, s, byq, qx0, qx1, fW)) && !sure;
    }
    if (!single) return;
    census = census0;
    wsum = wsum0;
    const float4* __restrict__ g2 = V.row2(iy) + V.plane;
    for (float qx = qx0; qx <= qx1; qx += 1.0f, q1++) {
        const float p2x = match<F>(s, qx, byq);
        if (p2x < 0 || p2x >= fW) continue;
        const float4 q = __ldg(q1);
        const float w = pair_support<F, M>(q.x - in.x, q.y - in.y, q.z - in.z);
        float ad = 3.0f;   // a NaN column reads the positive quiet NaN: full colour cost, positive signs
        int nm = sign_mismatch(__float_as_uint(q.w), 0u);
        if (p2x == p2x) {
            PairSigns d;
            float a;
            const float t = (p2x + 0.5f) - 0.5f;
            ad = eval_sample_pair<F>(base, q, t, d, a);
            nm = exact_mismatch<F>(g2 + (int)t, a, __float_as_uint(q.w));
        }
        add_terms<F, M>(census, wsum, w, sample_terms<F, M>(w, ad, nm));
    }
}

// patch_eval_census (:661-736) over pair records.  The census only grows (every term is >= 0), so the
// source's exit test after each sample, `census / bilw >= mincost` with a sample counted (:724), is
// decided by the census at the row's end; it is tested there as
// census >= exit_threshold(mincost, bilw).
template <bool F>
__device__ __forceinline__ float patch_eval_pair(const ViewData& V, int px, int py, float4 s, float mincost)
{
    const float cx = (float)px, cy = (float)py;
    if (!plane_usable(s, cx, cy, V.W)) return 1e5f;
    const float4 in = __ldg(V.row1(py) + px);
    const float thr = exit_threshold(mincost, in.w);
    float wsum = 0.0f, census = 0.0f;
    const int r = V.r;
    const float qx0 = (float)max(px - r, 0), qx1 = (float)min(px + r, V.W - 1);
    for (int iy = max(py - r, 0); iy <= min(py + r, V.H - 1); iy++) {
        eval_row_pixel<F>(V, iy, s, s.y * (float)iy, in, qx0, qx1, census, wsum);
        if (census >= thr && wsum > 0.0f) return 1.0f;
    }
    if (wsum <= 1.0f) return 1.1f;
    return census / wsum;
}

// The cost of a Gauss-Newton tap, k1 * ad + x * 0.25 * n (:361-370; VPMStereo.cl:154-162).  The source's sum is a double
// one rounded to float; here one fma.  They agree for colours k / 255: a nonzero truncated difference is
// then >= 2^-33 (the reference colour is 0 or >= 2^-8 in magnitude, the tap weights are multiples
// of 2^-25), so the colour term is 0 or >= 2^-36 of the weight; the double sum is inexact only when
// the colour term is below 2^-28 of the sum, and then it cannot land on a midpoint of two floats
// unless the colour term is below 2^-53 of it.
__device__ __forceinline__ float tap_cost(float k1, float x, float ad, int n) { return fmaf(x, (float)n, k1 * ad); }

// the sums of a Gauss-Newton step; J holds twice the source's (its factor 0.5 is taken out of the
// loop: scaling by a power of two commutes with rounding).  The sums are never -0, so a sample
// whose terms are +-0 leaves them unchanged.
struct KltSums {
    float J0, J1, J2, h00, h01, h02, h11, h12, h22;
};

// the colour cost of a tap: texels t0, t1 (r, g, b) mixed with weights b1 = 1 - a, a, against minus the
// reference colour
template <bool F>
__device__ __forceinline__ float tap_ad(float3 t0, float3 t1, float a, float b1, float3 nref)
{
    const float c0 = trunc_ad(mix<F>(a, b1, t0.x, t1.x) + nref.x), c1 = trunc_ad(mix<F>(a, b1, t0.y, t1.y) + nref.y),
                c2 = trunc_ad(mix<F>(a, b1, t0.z, t1.z) + nref.z);
    return c0 + c1 + c2;
}

__device__ __forceinline__ float3 pair_rgb(uint32_t w) { return make_float3(pair_unit<0>(w), pair_unit<1>(w), pair_unit<2>(w)); }

// one tap on its own: the coordinate u + 0.5 and its floor as the source forms them, the column
// clamped to the padded row, where the records hold the edge texels that the source's clamp
// gives, the signs from the gradients themselves (row2, g2: column 0 of the rows)
template <bool F>
__device__ __forceinline__ float tap_alone(float u, int W, const float4* __restrict__ row2, const float4* __restrict__ g2,
                                           float3 nref, uint32_t sb1, float k1, float x)
{
    const float t = (u + 0.5f) - 0.5f;
    const float fl = floorf(t);
    const float a = t - fl;
    const int c = (int)fminf(fmaxf(fl, -2.0f), (float)W);
    const PairRec R = __ldg(reinterpret_cast<const uint4*>(row2 + c));
    return tap_cost(k1, x, tap_ad<F>(pair_rgb(R.x), pair_rgb(R.y), a, 1.0f - a, nref), exact_mismatch<F>(g2 + c, a, sb1));
}

// The terms of a window sample of a Gauss-Newton step (:350-402): t = w (Cxm - Cxp), twice the factor of
// J's sums, and sc = w curv, the factor of H's; both +-0 for a rejected sample.  q: compact texel,
// c1: centre colour, p2x: matched column; row2, g2: column 0 of the pair and gradient rows.
// EVEN: p2x is at least 1 with p2x + 1.5 in the same binade, below 2^22.  p2x is then a
// multiple of its ulp <= 0.5, the +-1 and +-0.5 of the source are exact, and the taps at t - 1, t,
// t + 1 share the weight p2x - floor(p2x).  Otherwise each tap's coordinate is formed as the source
// forms it; mostly the floors are still f - 1, f, f + 1 and only the weights differ in the last bit, and the
// weights decide whether that holds: t - f is in [0, 1) exactly if f is t's floor.
// The three taps read three consecutive records, whose four texels are decoded once.  The column f
// is clamped to the padded row, where records beyond the image hold edge texels, as the
// source's clamp gives.  Where a weight is out of range (floors that do not chain, a non-finite column) or,
// not SURE, a sign unsure, each tap is read on its own.
template <bool F, bool EVEN, bool SURE, Model M>
__device__ __forceinline__ void klt_terms(int W, const float4* __restrict__ row2, const float4* __restrict__ g2, float4 q,
                                          float4 c1, float p2x, float& t, float& sc)
{
    const float MAGIC = EVEN ? 8388608.0f : 12582912.0f;   // MAGIC + t rounded down: MAGIC + floor(t), t >= 0 or |t| < 2^22
    // column c of the row is at base + 16 * (bits of the float MAGIC + c)
    const uintptr_t base = reinterpret_cast<uintptr_t>(row2) - (uintptr_t)(EVEN ? 0x4B000000u : 0x4B400000u) * 16u;
    const float first = MAGIC - 3.0f, last = MAGIC + (float)(W + 1);
    const float t0 = EVEN ? p2x : (p2x + 0.5f) - 0.5f;
    const float fm = __fadd_rd(t0, MAGIC);
    const float fc = EVEN ? fminf(fm, last) : fminf(fmaxf(fm, first), last);
    const uint4* b = reinterpret_cast<const uint4*>(base + (uintptr_t)__float_as_uint(fc) * 16u);
    const PairRec Rm = __ldg(b - 1), R0 = __ldg(b), Rp = __ldg(b + 1);
    const float f = fm - MAGIC;
    const float a0 = t0 - f;
    float am = a0, ap = a0;
    if (!EVEN) {
        am = (((p2x + -1.0f) + 0.5f) - 0.5f) - (f - 1.0f);
        ap = (((p2x + 1.0f) + 0.5f) - 0.5f) - (f + 1.0f);
    }
    const uint32_t A0 = pair_weight(a0), Am = EVEN ? A0 : pair_weight(am), Ap = EVEN ? A0 : pair_weight(ap);
    const uint32_t sb1 = __float_as_uint(q.w);
    const PairSigns dm = pair_signs(Am, Rm), d0 = pair_signs(A0, R0), dp = pair_signs(Ap, Rp);
    const float3 df = make_float3(c1.x - q.x, c1.y - q.y, c1.z - q.z);
    float w1 = pair_support<F, M>(df.x, df.y, df.z);
    // minus the reference colour: PMH takes the colour difference (:352, :364), VPM the colour
    const float3 nref = M == PMH ? df : make_float3(-q.x, -q.y, -q.z);
    const float k1 = M == PMH ? w1 * PM_K033_8 : w1 * 0.05f * 0.33f;
    // (w1 * 0.875f) * 0.25, (w1 * 0.95f) * 0.25: exact scaling
    const float x = M == PMH ? w1 * 0.21875f : w1 * (1.0f - 0.05f) * 0.25f;
    const float b0 = 1.0f - a0, bm = EVEN ? b0 : 1.0f - am, bp = EVEN ? b0 : 1.0f - ap;
    const float3 tA = pair_rgb(Rm.x), tB = pair_rgb(R0.x);
    float Cm = tap_cost(k1, x, tap_ad<F>(tA, tB, am, bm, nref), pair_mismatch(dm, sb1));
    const float3 tC = pair_rgb(R0.y);
    float C = tap_cost(k1, x, tap_ad<F>(tB, tC, a0, b0, nref), pair_mismatch(d0, sb1));
    const float3 tD = pair_rgb(Rp.y);
    float Cp = tap_cost(k1, x, tap_ad<F>(tC, tD, ap, bp, nref), pair_mismatch(dp, sb1));
    bool alone = false;
    if (!SURE) alone = unsure(unsure_max(unsure_max(unsure_max(0u, dm), d0), dp));
    // a weight in [0, 1) has bits below 1.0f's; a negative one or a NaN has not
    if (!EVEN) alone |= max(max(__float_as_uint(am), __float_as_uint(a0)), __float_as_uint(ap)) >= 0x3f800000u;
    if (alone) {
        Cm = tap_alone<F>(p2x + -1.0f, W, row2, g2, nref, sb1, k1, x);
        C = tap_alone<F>(p2x, W, row2, g2, nref, sb1, k1, x);
        Cp = tap_alone<F>(p2x + 1.0f, W, row2, g2, nref, sb1, k1, x);
        // a non-finite column reads NaN texels for all three taps: equal costs, nothing added
        if (!fin(p2x)) w1 = Cm = C = Cp = 0.0f;
    }
    // the update of :394-402 without a branch
    const float curv = fmaf(-2.0f, C, Cp + Cm);   // 2 C is exact
    const float wt = M == VPM || curv > 0.0f ? w1 : 0.0f;
    t = wt * (Cm - Cp);
    sc = wt * curv;
}

// a row of klt2_pair
template <bool F, bool EVEN, bool SURE, Model M>
__device__ __forceinline__ void klt_row(KltSums& A, int W, const float4* __restrict__ row2, const float4* __restrict__ g2,
                                        const float4* __restrict__ q1, float4 c1, float4 s, float byq, float qx0, float qx1,
                                        float qy)
{
    const float yy = qy * qy;
    for (float qx = qx0; qx <= qx1; qx += 1.0f, q1++) {
        float t, sc;
        klt_terms<F, EVEN, SURE, M>(W, row2, g2, __ldg(q1), c1, match<F>(s, qx, byq), t, sc);
        if (F) {
            A.J0 = fmaf(t, qx, A.J0);
            A.J1 = fmaf(t, qy, A.J1);
            A.h00 = fmaf(sc, qx * qx, A.h00);
            A.h01 = fmaf(sc, qx * qy, A.h01);
            A.h02 = fmaf(sc, qx, A.h02);
            A.h11 = fmaf(sc, yy, A.h11);
            A.h12 = fmaf(sc, qy, A.h12);
        } else {
            A.J0 = A.J0 + t * qx;
            A.J1 = A.J1 + t * qy;
            A.h00 = A.h00 + sc * (qx * qx);
            A.h01 = A.h01 + sc * (qx * qy);
            A.h02 = A.h02 + sc * qx;
            A.h11 = A.h11 + sc * yy;
            A.h12 = A.h12 + sc * qy;
        }
        A.J2 = A.J2 + t;
        A.h22 = A.h22 + sc;
    }
}

// patch_census_klt2 (:326-410) over pair records.  p2x is monotone along a row, so its two ends decide
// the row's kind (klt_row), for the warp: one whose lanes differ would run several loops.
template <bool F, Model M = PMH>
__device__ __forceinline__ float4 klt2_pair(const ViewData& V, int px, int py, float4 s)
{
    // a NaN plane has no column: no sample counts, the 0 / 0 solution is NaN
    if (s.x != s.x || s.y != s.y || s.z != s.z) return f4(qnan(), qnan(), qnan(), s.w - 1e5f);
    const float cxf = (float)px, cyf = (float)py;
    KltSums A = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    const float4 c1 = __ldg(V.row1(py) + px);
    const int r = V.r;
    const int dy0 = max(-r, -py), dy1 = min(r, V.H - 1 - py);
    const int dx0 = max(-r, 1 - px), dx1 = min(r, V.W - 2 - px);   // the 3-point cost needs 1 <= qx < W - 1
    const float qx0 = cxf + (float)dx0, qx1 = cxf + (float)dx1;
    float qy = cyf + (float)dy0;
    for (int iy = py + dy0; iy <= py + dy1; iy++, qy += 1.0f) {
        const float byq = s.y * qy;
        const float4* __restrict__ q1 = V.row1c(iy) + px + dx0;
        const float4* __restrict__ row2 = V.row2p(iy);
        const float4* __restrict__ g2 = V.row2(iy) + V.plane;
        const float pa = match<F>(s, qx0, byq), pb = match<F>(s, qx1, byq);
        const float plo = fminf(pa, pb), phi = fmaxf(pa, pb);
        const bool even = pa >= 1.0f && pb >= 1.0f && phi < 4194304.0f &&
                          ((__float_as_uint(phi + 1.5f) ^ __float_as_uint(plo)) < 0x00800000u);
        const unsigned lanes = __activemask();
        if (!__all_sync(lanes, even)) klt_row<F, false, false, M>(A, V.W, row2, g2, q1, c1, s, byq, qx0, qx1, qy);
        // from column 256 on the weight is a multiple of 2^-15 and no sign is unsure
        else if (__all_sync(lanes, plo >= 256.0f)) klt_row<F, true, true, M>(A, V.W, row2, g2, q1, c1, s, byq, qx0, qx1, qy);
        else klt_row<F, true, false, M>(A, V.W, row2, g2, q1, c1, s, byq, qx0, qx1, qy);
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
