// Window loops of a warp over the pixels it owns (pm_window.cuh has the loops of one thread).
//
// Every sum of a window must round in sample order, but the terms do not depend on each other: a row's
// terms of all pixels that still need it are spread over the 32 lanes, left in shared memory, and
// added in order by the lanes that own the sums.  Two uses:
//   * the lanes of a warp leave a cost window at different rows (early exit) or do not need it at all (19 of
//     32 lanes active in a converged 640x360 pass): from WARP_TASKS pixels down the rows are shared;
//   * an image too small to fill the chip with a thread per pixel gets fewer pixels per warp (`owners`,
//     prop_owners in pm_propagate.cu), for the cost windows and for the Gauss-Newton steps.
#pragma once

#include "pm_window.cuh"

namespace pm {

// Pixels a warp shares its windows over at most, and terms per pass over them.  A shared sample costs about
// 1.6 times a sample of a thread's own row, so above half of the lanes each runs its own row
// (1280x720, 3 iterations, candidate chain in ms: sharing from 28 pixels down 69.6, 24 65.6, 20 65.1, 16
// 64.1; never 69.2).
constexpr int WARP_TASKS = 16, WARP_TERMS = 16 * 23;

template <Model M = PMH>
struct WarpScratch {
    float4 par[WARP_TASKS][2];   // per pixel: plane and column of the window's left end; centre colour and top row
    float2 term[WARP_TERMS];     // (first part, weight) of a cost term, or (t, sc) of a Gauss-Newton term
    float part[M == VPM ? WARP_TERMS : 1];   // second part of a cost term
};

// The items of a pass: samples e0 .. e0 + len - 1 (row by row) of n windows, item i = (task, sample e0 + i % len)
struct WarpItem {
    int i, task, e, len, e0;
    __device__ __forceinline__ WarpItem(int lane, int e0_, int len_) : i(lane), task(lane / len_), e(lane % len_), len(len_), e0(e0_) {}
    __device__ __forceinline__ void next()
    {
        i += 32;
        e += 32;
        while (e >= len) {
            e -= len;
            task++;
        }
    }
};

// Samples e0 .. e0 + len - 1 of the windows of patch_eval_census of the n pixels whose parameters are in S.par,
// spread over the warp; their terms go to S.term[task * len + sample - e0].  ROW: all windows
// have the top row `top` (a warp along an image row).
template <bool F, bool ROW, Model M>
__device__ __forceinline__ void eval_terms_shared(const ViewData& V, WarpScratch<M>& S, int lane, int n, int e0, int len,
                                                  const WindowSpan& span, int top)
{
    const int W = V.W;
    const float fW = (float)W;
    for (WarpItem it(lane, e0, len); it.i < n * len; it.next()) {
        const float4 A = S.par[it.task][0], B = S.par[it.task][1];   // (s.x, s.y, s.z, left column), (colour, top row)
        const int e = it.e0 + it.e, j = span.row(e);
        const int y = (ROW ? top : __float_as_int(B.w)) + j, x = __float_as_int(A.w) + e - j * span.cols;
        const bool in1 = (unsigned)x < (unsigned)W && (unsigned)y < (unsigned)V.H;
        const int yc = min(max(y, 0), V.H - 1);
        const float qx = (float)x;
        const float4 q = __ldg(V.row1c(yc) + min(max(x, 0), W - 1));
        const float p2x = match<F>(A, qx, A.y * (float)y);
        const float t = fminf(fmaxf((p2x + 0.5f) - 0.5f, 0.0f), fW);   // in [0, W], 0 for a NaN
        float w = pair_support<F, M>(q.x - B.x, q.y - B.y, q.z - B.z);
        const uintptr_t base = reinterpret_cast<uintptr_t>(V.row2p(yc)) - (uintptr_t)0x4B000000u * 16u;
        PairSigns d;
        float a;
        float ad = eval_sample_pair<F>(base, q, t, d, a);
        int nm = pair_mismatch(d, __float_as_uint(q.w));
        // a NaN column reads the positive quiet NaN: full colour cost, positive signs
        const bool nan = p2x != p2x;
        if (unsure(unsure_max(0u, d)) || nan) {
            nm = nan ? sign_mismatch(__float_as_uint(q.w), 0u)
                     : exact_mismatch<F>(V.row2(yc) + V.plane + (int)t, a, __float_as_uint(q.w));
            if (nan) ad = 3.0f;
        }
        if (!in1 || p2x < 0.0f || p2x >= fW) w = 0.0f;
        const SampleTerms c = sample_terms<F, M>(w, ad, nm);
        S.term[it.i] = f2(c.a, w);
        if (M == VPM) S.part[it.i] = c.b;
    }
}

// patch_eval_census (:661-736) for the pixels of a warp whose lanes set `need`; all 32 lanes call.
// S: this warp's scratch.  All windows of the warp are at the same sample e0: rows that the lanes run on
// their own end on a whole row, and once few enough windows are left they stay shared.
//
// VPM (VPMStereo.cl:200-258) has no early exit of its own, but its caller only asks whether the cost is below
// mincost.  The census only grows and the weight sum stays at or below the whole window's
// (in.w; sums of a subset of the terms in the same order round no higher), so once
// census / in.w >= mincost the cost cannot be below mincost any more, and any such value may be returned.
template <bool F, bool ROW, Model M = PMH>
__device__ __forceinline__ float patch_eval_warp(const ViewData& V, WarpScratch<M>& S, int lane, bool need, int px, int py,
                                                 float4 s, float mincost)
{
    const float cx = (float)px, cy = (float)py;
    float ret = M == PMH ? 1e5f : 1.0f, wsum = 0.0f, census = 0.0f, thr = 0.0f;
    float4 in = f4(0.0f, 0.0f, 0.0f, 0.0f);
    bool act = need;
    if (M == PMH) {
        act = act && plane_usable(s, cx, cy, V.W);
    } else {
        const float c2x = transform_x(s, cx, cy);
        act = act && !(c2x < 0 || c2x >= (float)V.W);
    }
    if (act) {
        in = __ldg(V.row1(py) + px);
        thr = exit_threshold(mincost, in.w);
    }
    const int r = V.r;
    const float qx0 = (float)max(px - r, 0), qx1 = (float)min(px + r, V.W - 1);
    // constant operands (V.span) are 0.7% faster in the main path's candidate kernel (320x240, r = 7) and up to
    // 6% slower in VPM's (107x110, r = 10)
    const WindowSpan span = M == PMH ? V.span : WindowSpan(V.W, V.H, r, V.W, V.H);
    const int top = span.top(py, r), left = span.left(px, r), samples = span.cols * span.rows;
    for (int e0 = 0; e0 < samples;) {
        const unsigned m = __ballot_sync(0xffffffffu, act);
        const int n = __popc(m);
        if (n == 0) break;
        if (n > WARP_TASKS) {   // every lane its own row
            const int iy = top + span.row(e0);
            if (act && iy >= 0 && iy < V.H) eval_row_pixel<F, M>(V, iy, s, s.y * (float)iy, in, qx0, qx1, census, wsum);
            e0 += span.cols;
        } else {
            const int rank = __popc(m & ((1u << lane) - 1u));
            const int len = min((WARP_TERMS / n - 1) | 1, samples - e0);   // odd: the ordered sums read with this stride
            if (act) {
                S.par[rank][0] = f4(s.x, s.y, s.z, __int_as_float(left));
                S.par[rank][1] = f4(in.x, in.y, in.z, __int_as_float(top));
            }
            __syncwarp();
            eval_terms_shared<F, ROW, M>(V, S, lane, n, e0, len, span, top);
            __syncwarp();
            if (act) {
                const float2* v = S.term + rank * len;
#pragma unroll 4
                for (int k = 0; k < len; k++) {
                    const float2 c = v[k];
                    add_terms<F, M>(census, wsum, c.y, SampleTerms{c.x, M == VPM ? S.part[rank * len + k] : 0.0f});
                }
            }
            e0 += len;
            __syncwarp();
        }
        if (act && census >= thr && wsum > 0.0f) {   // the exit test, as in patch_eval_pair
            ret = M == PMH ? 1.0f : __int_as_float(0x7f800000);
            act = false;
        }
    }
    if (act) ret = M == PMH && wsum <= 1.0f ? 1.1f : census / wsum;
    return ret;
}

// `steps` steps of patch_census_klt2 (:326-410) for the first `owners` <= WARP_KLT lanes of a warp along an image
// row, those with `need`; all 32 lanes call.  The terms (t, sc) of all owned windows are
// spread over the lanes, pass by pass; each of a window's nine sums belongs to one lane, which
// adds its products in sample order.  The factor of a sum is a product of two of 1, qx, qy, exact.
constexpr int WARP_KLT = 4;
static_assert(WARP_KLT <= WARP_TASKS, "klt2_steps_warp keeps its pixels in the scratch");
template <bool F, Model M = PMH>
__device__ __forceinline__ float4 klt2_steps_warp(const ViewData& V, WarpScratch<M>& S, int lane, int owners, int steps,
                                                  bool need, int px, int py, float4 s)
{
    constexpr int NU = (9 * WARP_KLT + 31) / 32;   // sums per lane, at most
    const int W = V.W, r = V.r;
    const int units = 9 * owners;
    const WindowSpan span(W, V.H, r, W, V.H);   // V.span's constant operands: 1-3% slower (64x48, r = 32)
    const int cols = span.cols, top = span.top(py, r);
    // rows inside the image: samples first .. end - 1
    const int first = max(-top, 0) * cols, end = min(span.rows, V.H - top) * cols;
    float* const sums = reinterpret_cast<float*>(S.term);
    const float4 c1 = need ? __ldg(V.row1(py) + px) : f4(0.0f, 0.0f, 0.0f, 0.0f);
    const int chunk = WARP_TERMS / owners;
    for (int step = 0; step < steps; step++) {
        // a NaN plane has no column: no sample counts, the 0 / 0 solution is NaN
        const bool nan = s.x != s.x || s.y != s.y || s.z != s.z;
        const unsigned m = __ballot_sync(0xffffffffu, need && !nan);
        if (lane < owners) {
            S.par[lane][0] = f4(s.x, s.y, s.z, (float)span.left(px, r));
            S.par[lane][1] = f4(c1.x, c1.y, c1.z, 0.0f);
        }
        float acc[NU];
#pragma unroll
        for (int k = 0; k < NU; k++) acc[k] = 0.0f;
        for (int e0 = first; e0 < end; e0 += chunk) {
            const int len = min(chunk, end - e0);
            __syncwarp();
            for (WarpItem it(lane, e0, len); it.i < owners * len; it.next()) {
                float2 v = f2(0.0f, 0.0f);
                const float4 A = S.par[it.task][0];
                const int e = it.e0 + it.e, j = span.row(e), y = top + j;
                const float qx = A.w + (float)(e - j * cols);
                // the 3-point cost needs 1 <= qx < W - 1
                if (((m >> it.task) & 1u) && qx >= 1.0f && qx < (float)(W - 1)) {
                    const float4 c = S.par[it.task][1];
                    klt_terms<F, false, false, M>(W, V.row2p(y), V.row2(y) + V.plane, __ldg(V.row1c(y) + (int)qx), c,
                                               match<F>(A, qx, A.y * (float)y), v.x, v.y);
                }
                S.term[it.i] = v;
            }
            __syncwarp();
#pragma unroll
            for (int k = 0; k < NU; k++) {
                const int u = lane + 32 * k;
                if (u < units) {
                    const int task = u / 9, j = u - 9 * task;
                    // sum j: J = t (qx, qy, 1), H = sc (qx qx, qx qy, qx, qy qy, qy, 1); factors f and g
                    const bool fx = j == 0 || (j >= 3 && j <= 5), fy = j == 1 || j == 6 || j == 7;
                    const bool gx = j == 3, gy = j == 4 || j == 6;
                    const float* v = reinterpret_cast<const float*>(S.term + task * len) + (j >= 3);
                    const float left = S.par[task][0].w;
                    float sum = acc[k];
                    int row = span.row(e0), dx = e0 - row * cols;
                    for (int d = 0; d < len;) {
                        const float qy = (float)(top + row);
                        const float f1 = fx ? 1.0f : 0.0f, f0 = fx ? 0.0f : fy ? qy : 1.0f;
                        const float g1 = gx ? 1.0f : 0.0f, g0 = gx ? 0.0f : gy ? qy : 1.0f;
                        const int stop = min(len, d + cols - dx);
                        float qx = left + (float)dx;
#pragma unroll 4
                        for (; d < stop; d++, qx += 1.0f) {
                            const float f = fmaf(f1, qx, f0) * fmaf(g1, qx, g0);
                            sum = F ? fmaf(v[2 * d], f, sum) : sum + v[2 * d] * f;
                        }
                        dx = 0;
                        row++;
                    }
                    acc[k] = sum;
                }
            }
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < NU; k++)
            if (lane + 32 * k < units) sums[lane + 32 * k] = acc[k];
        __syncwarp();
        if (need) {
            if (nan) {
                s = f4(qnan(), qnan(), qnan(), s.w - 1e5f);
            } else {
                const float* a = sums + 9 * lane;
                const float3 d = lusolve(a[3], a[4], a[5], a[6], a[7], a[8],
                                         make_float3(a[0] * 0.5f, a[1] * 0.5f, a[2] * 0.5f));
                s = f4(s.x - d.x, s.y - d.y, s.z - d.z, s.w - 1e5f);
            }
        }
        __syncwarp();
    }
    return s;
}

}  // namespace pm
