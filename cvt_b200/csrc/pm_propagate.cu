// pmhstereo_propagate_view (cvt/cl/kernel/pmhstereo.cl:880-1071) on sm_100a, as three
// kernels over the same pixels:
//   k_prop_chain  the candidate chain up to the randomized refinement (:927-1028)
//   k_prop_klt_list  the six Gauss-Newton steps (:1034-1038) of listed pixels; k_prop_klt_warp runs them with few
//                 pixels per warp, k_prop_klt over the general loops
//   k_prop_final  the evaluation of their result, the view scatter and the output (:1039-1070)
// The state between them is `self` and the Gauss-Newton result (two float4 fields).
//
// The candidate chain keeps the source's structure: the lanes of a warp evaluate their
// pixels' k-th candidates together, so that neighbouring lanes read neighbouring texels of
// both views (a per-lane schedule, where each lane moves on to its next candidate as soon as
// its window ends, measured slower: the lanes' windows then diverge in rows and planes and
// the L1 hit rate halves).
#include <cuda_runtime.h>
#include <stdint.h>

#include "pm_kernels.h"
#include "pm_warp.cuh"

namespace pm {

namespace {

// block shape of the single-pair kernels: PROP_BX consecutive threads, one warp, along a row, PM_PROP_BY rows
#ifndef PM_PROP_BY
#define PM_PROP_BY 4
#endif
constexpr int PROP_BX = 32, PROP_BY = PM_PROP_BY, PROP_THREADS = PROP_BX * PROP_BY;
// Resident threads per SM asked of the register allocator for each kernel (640 = 96 registers, no
// spills).  The window loops issue 82-88% of the cycles (640x360), so more threads give nothing: 1280x720,
// r = 10, 3 iterations, ms (chain / Gauss-Newton): 512 threads 75.5 / 89.1, 640 69.2 / 88.9,
// 768 69.2 / 88.7, 1024 (chain) 71.5; unrolling a row's loop by two 75.0 / 89.2 at 512.  The
// block shape does not matter either (32x4, 16x8, 8x16 and 32x2 within 1.5% of each other).
#ifndef PM_CHAIN_THREADS
#define PM_CHAIN_THREADS 640
#endif
#ifndef PM_KLT_THREADS
#define PM_KLT_THREADS 640
#endif
constexpr int PM_CHAIN_BLOCKS = PM_CHAIN_THREADS / PROP_THREADS, PM_KLT_BLOCKS = PM_KLT_THREADS / PROP_THREADS;
// the batched (persistent) forms index each pair's arguments in a parameter block, which takes registers
#ifndef PM_BATCH_THREADS
#define PM_BATCH_THREADS 640
#endif
constexpr int PM_BATCH_BLOCKS = PM_BATCH_THREADS / PROP_THREADS;

inline dim3 grid2d(int W, int H, dim3 b) { return dim3((W + b.x - 1) / b.x, (H + b.y - 1) / b.y); }

template <bool COUNT>
__device__ __forceinline__ void flush_counters(const Counters& cnt, unsigned long long* out)
{
    if (!COUNT) return;
    unsigned long long v[4] = {cnt.eval, cnt.klt, cnt.calls, cnt.exits};
#pragma unroll
    for (int k = 0; k < 4; k++) {
        unsigned long long s = v[k];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if ((threadIdx.x & 31) == 0 && s) atomicAdd(out + k, s);
    }
}

// keep the two smallest source columns of a view-buffer entry (see pm_kernels.h)
__device__ __forceinline__ bool view_insert(unsigned long long* slot, unsigned int x)
{
    unsigned long long cur = *reinterpret_cast<volatile unsigned long long*>(slot);
    for (int guard = 0; guard < 4096; guard++) {
        const unsigned int lo = (unsigned int)cur, hi = (unsigned int)(cur >> 32);
        unsigned long long nv;
        if (x < lo) nv = ((unsigned long long)lo << 32) | x;
        else if (x < hi) nv = ((unsigned long long)x << 32) | lo;
        else return true;
        const unsigned long long prev = atomicCAS(slot, cur, nv);
        if (prev == cur) return true;
        cur = prev;
    }
    return false;
}

// A candidate whose plane (a, b, c) equals the current one bit for bit has the current
// plane's smoothing distance d (smoothDistance reads no cost).  Evaluated without an early
// exit it returns the current cost and is taken, which changes nothing; with an exit it
// returns 1 and is taken only if 1 + theta d <= cost + theta d.  When that comparison fails,
// the candidate leaves the state as it is whatever its window gives, and is not evaluated.
__device__ __forceinline__ bool known_outcome(float4 nb, float4 self, float theta, float sd_self)
{
    return __float_as_uint(nb.x) == __float_as_uint(self.x) && __float_as_uint(nb.y) == __float_as_uint(self.y) &&
           __float_as_uint(nb.z) == __float_as_uint(self.z) && !(1.0f + theta * sd_self <= self.w + theta * sd_self);
}

// one warp's share of the shared memory of the window loops, and the calling lane (the block's warps are 32
// consecutive threads, whatever its shape)
__device__ __forceinline__ WarpScratch<>& warp_scratch(WarpScratch<>* ws, int& lane)
{
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    lane = tid & 31;
    return ws[tid >> 5];
}

// the window cost of the pixels of a warp whose lanes set `need` (all lanes call)
template <bool F, bool COUNT, bool GEN, bool ROW>
__device__ __forceinline__ float eval_pixels(const ViewData& V, WarpScratch<>* ws, bool need, int px, int py, float4 s,
                                             float mincost, Counters& cnt)
{
    if (GEN) return need ? patch_eval_general<F, COUNT>(V, px, py, s, mincost, cnt) : 0.0f;
    int lane;
    WarpScratch<>& S = warp_scratch(ws, lane);
    return patch_eval_warp<F, ROW>(V, S, lane, need, px, py, s, mincost);
}

// pmhstereo_propagate_view (:927-1028): candidates k = 0 (the current plane, re-evaluated,
// :939-940), 1 smooth (:968-976), 2-5 random neighbours with offsets drawn x first, in
// [-4, 5] (:982-991), 6 a random plane (:996-1002), 7-8 cross-view planes (:1007-1016),
// 9 the randomized refinement (:1021-1028).  One loop, so that the window evaluation has a
// single call site, which the lanes of a warp reach together (eval_pixels).  A block covers
// P.owners x BY pixels: the lanes threadIdx.x < P.owners own one each.
//
// Candidate 0, the current plane without an early exit, gives back the cost it was stored with: that is
// the same window sum unless it is the 1 that an early exit returns.  Within a run (P.known) it
// is evaluated only then; it was a sixth of a pass's cost samples (1280x720, 3 iterations:
// chain 64.1 -> 56.0 ms).
template <bool F, bool COUNT, bool GEN, int BX = PROP_BX, int BY = PROP_BY>
__device__ __forceinline__ void chain_tile(const PropParams& P, WarpScratch<>* ws, int bx, int by, Counters& cnt)
{
    const ViewData& V = P.V;
    const int px = bx * P.owners + threadIdx.x, py = by * BY + threadIdx.y;
    const bool own = threadIdx.x < P.owners && px < V.W && py < V.H;
    if (GEN && !own) return;
    const int W = V.W;
    const size_t idx = (size_t)py * W + px;
    const float cx = (float)px, cy = (float)py;
    const int lr = P.lr;
    const float theta = P.theta, dmax = P.dmax;
    float4 smooth = f4(0.0f, 0.0f, 0.0f, 0.0f), self = smooth;
    // cross-view candidates of this pixel; the entry is emptied for the next writer
    int nview = 0;
    unsigned long long vsrc = ~0ULL;
    if (own) {
        smooth = P.smooth[idx];
        smooth.w = clampf(smooth.w, 0.0f, 1.0f) * dmax;   // :927-928
        self = P.old[idx];
        if (P.vin_count) {
            nview = min(P.vin_count[idx], 2);
            vsrc = P.vin_src[idx];
            P.vin_count[idx] = 0;
            P.vin_src[idx] = ~0ULL;
        }
    }

    Rng rng;
    // RNG_init(&rng, lin, ((1*1 - 1) + NUMRNDTRIES) * 3 + 2 * NUMRNDSAMPLE) (:942) expands to
    // (lin) * ((1*1 - 1) + 2) * 3 + 2 * 4 = 6 * lin + 8
    rng.init_skip((py * W + px + P.iter) * 6 + 8);

    float sd_self = 0.0f;   // smoothing distance of `self` (smoothDistance does not read the cost)
    for (int k = 0; k < 10; k++) {
        float4 nb = self;
        bool need = own;
        if (k == 1) {
            nb = from_disparity_normal(cx, cy, smooth.w * (lr ? -1.0f : 1.0f),
                                       normalize3(make_float3(smooth.x, smooth.y, smooth.z)));
            if (!lr) nb = viewprop(nb);
        } else if (k >= 2 && k <= 5) {
            const int ox = (int)((rng.next() - 0.5f) * 2.0f * 5.0f + 0.5f);
            const int oy = (int)((rng.next() - 0.5f) * 2.0f * 5.0f + 0.5f);
            if (own) nb = P.old[(size_t)min(max(py + oy, 0), V.H - 1) * W + min(max(px + ox, 0), W - 1)];
        } else if (k == 6) {
            nb = nd_state_init(rng, cx, cy, lr, dmax);
        } else if (k == 7 || k == 8) {
            need = k - 7 < nview;
            if (need)
                nb = viewprop(P.vin_planes[(size_t)py * W + (k == 7 ? (unsigned int)vsrc : (unsigned int)(vsrc >> 32))]);
        } else if (k == 9) {
            nb = nd_state_refine(rng, self, cx, cy, dmax, lr);
        }
        float sd = 0.0f, mincost = 1e10f;
        if (k == 0) {
            if (!GEN && P.known) need = need && self.w == 1.0f;
        } else {
            need = need && !known_outcome(nb, self, theta, sd_self);
            sd = smooth_dist1(nb, smooth, cx, cy, dmax, lr);
            // minimalCost (:873-877)
            mincost = self.w + theta * sd_self - theta * sd;
        }
        nb.w = eval_pixels<F, COUNT, GEN, BX == 32>(V, ws, need, px, py, nb, mincost, cnt);
        if (k == 0) {
            if (need) self.w = nb.w;
            sd_self = smooth_dist1(self, smooth, cx, cy, dmax, lr);
        } else if (need && nb.w + theta * sd <= self.w + theta * sd_self) {   // :976 etc.
            self = nb;
            sd_self = sd;
        }
    }
    // Within a run (P.known) the Gauss-Newton steps of a plane that the pixel already had after the previous
    // iteration's candidates would give the result that still lies in tmp_nb.  The others are listed, a warp's
    // pixels together (launch_pass; the list's order changes nothing, each pixel is on its own).
    if (!GEN && P.list) {
        bool todo = own;
        if (own && P.known && P.iter > 0) {
            const float4 was = P.tmp_self[idx];
            todo = __float_as_uint(was.x) != __float_as_uint(self.x) || __float_as_uint(was.y) != __float_as_uint(self.y) ||
                   __float_as_uint(was.z) != __float_as_uint(self.z);
        }
        const int lane = (threadIdx.y * blockDim.x + threadIdx.x) & 31;
        const unsigned m = __ballot_sync(0xffffffffu, todo);
        int at = 0;
        if (lane == 0 && m) at = atomicAdd(P.list_count, __popc(m));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (todo) P.list[at + __popc(m & ((1u << lane) - 1u))] = (int)idx;
    }
    if (own) P.tmp_self[idx] = self;
}

template <bool F, bool COUNT, bool GEN>
__global__ void __launch_bounds__(PROP_THREADS, PM_CHAIN_BLOCKS) k_prop_chain(PropParams P)
{
    if (variant_skips<GEN>(P.V, P.dual)) return;
    __shared__ WarpScratch<> ws[GEN ? 1 : PROP_THREADS / 32];
    Counters cnt = {0, 0, 0, 0};
    chain_tile<F, COUNT, GEN>(P, ws, blockIdx.x, blockIdx.y, cnt);
    flush_counters<COUNT>(cnt, P.counters);
}

// Gauss-Newton plane steps (:1034-1038)
template <bool F, bool COUNT, bool GEN, int BX = PROP_BX, int BY = PROP_BY>
__device__ __forceinline__ void klt_tile(const PropParams& P, int bx, int by, Counters& cnt)
{
    const ViewData& V = P.V;
    const int px = bx * BX + threadIdx.x, py = by * BY + threadIdx.y;
    if (px < V.W && py < V.H) {
        const size_t idx = (size_t)py * V.W + px;
        float4 nb = P.tmp_self[idx];
        for (int k = 0; k < 6; k++) nb = klt2<F, COUNT, GEN>(V, px, py, nb, cnt);
        P.tmp_nb[idx] = nb;
    }
}

template <bool F, bool COUNT>
__global__ void __launch_bounds__(PROP_THREADS, PM_KLT_BLOCKS) k_prop_klt(PropParams P)
{
    if (variant_skips<true>(P.V, P.dual)) return;
    Counters cnt = {0, 0, 0, 0};
    klt_tile<F, COUNT, true>(P, blockIdx.x, blockIdx.y, cnt);
    flush_counters<COUNT>(cnt, P.counters);
}

// the same over the pair-plane loops, for the pixels of P.list
template <bool F>
__global__ void __launch_bounds__(PROP_THREADS, PM_KLT_BLOCKS) k_prop_klt_list(PropParams P)
{
    if (variant_skips<false>(P.V, P.dual)) return;
    const int i = blockIdx.x * PROP_THREADS + threadIdx.x;
    if (i >= *P.list_count) return;
    const int idx = P.list[i];
    const int py = idx / P.V.W, px = idx - py * P.V.W;
    float4 nb = P.tmp_self[idx];
    for (int k = 0; k < 6; k++) nb = klt2_pair<F>(P.V, px, py, nb);
    P.tmp_nb[idx] = nb;
}

// the same with P.owners <= WARP_KLT pixels per warp (prop_owners)
template <bool F>
__global__ void __launch_bounds__(PROP_THREADS, PM_KLT_BLOCKS) k_prop_klt_warp(PropParams P)
{
    if (variant_skips<false>(P.V, P.dual)) return;
    __shared__ WarpScratch<> ws[PROP_THREADS / 32];
    const ViewData& V = P.V;
    int lane;
    WarpScratch<>& S = warp_scratch(ws, lane);
    const int px = blockIdx.x * P.owners + threadIdx.x, py = blockIdx.y * PROP_BY + threadIdx.y;
    if (py >= V.H) return;   // a warp is a row of the block
    const bool own = threadIdx.x < P.owners && px < V.W;
    const size_t idx = (size_t)py * V.W + px;
    float4 nb = own ? P.tmp_self[idx] : f4(0.0f, 0.0f, 0.0f, 0.0f);
    nb = klt2_steps_warp<F>(V, S, lane, P.owners, 6, own, px, py, nb);
    if (own) P.tmp_nb[idx] = nb;
}

// evaluation of the Gauss-Newton result (:1039-1052), view scatter (:1060-1067), output (:1070)
template <bool F, bool COUNT, bool GEN, int BX = PROP_BX, int BY = PROP_BY>
__device__ __forceinline__ void final_tile(const PropParams& P, WarpScratch<>* ws, int bx, int by, Counters& cnt)
{
    const ViewData& V = P.V;
    const int px = bx * P.owners + threadIdx.x, py = by * BY + threadIdx.y;
    const bool own = threadIdx.x < P.owners && px < V.W && py < V.H;
    if (GEN && !own) return;
    const int W = V.W;
    const size_t idx = (size_t)py * W + px;
    const float cx = (float)px, cy = (float)py;
    const int lr = P.lr;
    const float dmax = P.dmax, theta = P.theta;
    float4 smooth = f4(0.0f, 0.0f, 0.0f, 0.0f), self = smooth, nb = smooth;
    if (own) {
        smooth = P.smooth[idx];
        smooth.w = clampf(smooth.w, 0.0f, 1.0f) * dmax;
        self = P.tmp_self[idx];
        nb = P.tmp_nb[idx];
    }
    const float2 sd = smooth_distance(nb, self, smooth, cx, cy, dmax, lr);
    const bool need = own && !known_outcome(nb, self, theta, sd.y);
    const float mincost = self.w + theta * sd.y - theta * sd.x;
    nb.w = eval_pixels<F, COUNT, GEN, BX == 32>(V, ws, need, px, py, nb, mincost, cnt);
    if (own) {
        if (need && nb.w + theta * sd.x <= self.w + theta * sd.y) self = nb;

        if (P.vout_count) {
            const float sidesign = lr ? -1.0f : 1.0f;
            const float tx = transform_x(self, cx, cy);
            const int xpv = __float2int_rn(tx);           // convert_int_rte
            const int disp = (int)((tx - cx) * sidesign);  // convert_int
            if (xpv >= 0 && xpv < W && disp > 0) {
                const size_t t = (size_t)py * W + xpv;
                atomicAdd(P.vout_count + t, 1);
                if (!view_insert(P.vout_src + t, (unsigned int)px)) atomicAdd(P.error, 1);
            }
        }
        P.out[idx] = self;
    }
}

template <bool F, bool COUNT, bool GEN>
__global__ void __launch_bounds__(PROP_THREADS) k_prop_final(PropParams P)
{
    if (variant_skips<GEN>(P.V, P.dual)) return;
    __shared__ WarpScratch<> ws[GEN ? 1 : PROP_THREADS / 32];
    Counters cnt = {0, 0, 0, 0};
    if (!GEN && P.list && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && threadIdx.y == 0) *P.list_count = 0;
    final_tile<F, COUNT, GEN>(P, ws, blockIdx.x, blockIdx.y, cnt);
    flush_counters<COUNT>(cnt, P.counters);
}

// Batched propagate passes (a batch of pairs in lockstep): persistent CTAs take tiles of
// any pair of a group from the job list (grab_job) and run the single-pair kernels' tile
// functions on them with that pair's arguments.  The group's arguments travel as one kernel
// parameter block (read through the constant cache, as a single-pair launch reads its own),
// job.x indexing it.  Every pixel runs the same operations on the same fields as in a
// single-pair launch, so the results are the same bit for bit.
template <bool F, bool COUNT, bool GEN, int BX>
__global__ void __launch_bounds__(PROP_THREADS, PM_BATCH_BLOCKS)
    k_prop_chain_b(const __grid_constant__ PropGroup G, const uint2* __restrict__ jobs, int njobs, int* next)
{
    __shared__ WarpScratch<> ws[GEN ? 1 : PROP_THREADS / 32];
    for (;;) {
        const int j = grab_job(next);
        if (j >= njobs) return;
        const uint2 job = jobs[j];
        const PropParams& P = G.p[job.x];
        if (variant_skips<GEN>(P.V, P.dual)) continue;
        Counters cnt = {0, 0, 0, 0};
        chain_tile<F, COUNT, GEN, BX, PROP_THREADS / BX>(P, ws, (int)(job.y & 0xffffu), (int)(job.y >> 16), cnt);
        flush_counters<COUNT>(cnt, P.counters);
    }
}

template <bool F, bool COUNT, bool GEN, int BX>
__global__ void __launch_bounds__(PROP_THREADS, PM_BATCH_BLOCKS)
    k_prop_klt_b(const __grid_constant__ PropGroup G, const uint2* __restrict__ jobs, int njobs, int* next)
{
    for (;;) {
        const int j = grab_job(next);
        if (j >= njobs) return;
        const uint2 job = jobs[j];
        const PropParams& P = G.p[job.x];
        if (variant_skips<GEN>(P.V, P.dual)) continue;
        Counters cnt = {0, 0, 0, 0};
        klt_tile<F, COUNT, GEN, BX, PROP_THREADS / BX>(P, (int)(job.y & 0xffffu), (int)(job.y >> 16), cnt);
        flush_counters<COUNT>(cnt, P.counters);
    }
}

template <bool F, bool COUNT, bool GEN, int BX>
__global__ void __launch_bounds__(PROP_THREADS, PM_BATCH_BLOCKS)
    k_prop_final_b(const __grid_constant__ PropGroup G, const uint2* __restrict__ jobs, int njobs, int* next)
{
    __shared__ WarpScratch<> ws[GEN ? 1 : PROP_THREADS / 32];
    for (;;) {
        const int j = grab_job(next);
        if (j >= njobs) return;
        const uint2 job = jobs[j];
        const PropParams& P = G.p[job.x];
        if (variant_skips<GEN>(P.V, P.dual)) continue;
        Counters cnt = {0, 0, 0, 0};
        final_tile<F, COUNT, GEN, BX, PROP_THREADS / BX>(P, ws, (int)(job.y & 0xffffu), (int)(job.y >> 16), cnt);
        flush_counters<COUNT>(cnt, P.counters);
    }
}

// resident CTAs per SM of a kernel with PROP_THREADS threads (at least 1)
template <class K>
int resident_ctas(K kernel)
{
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, PROP_THREADS, 0) != cudaSuccess) {
        cudaGetLastError();
        n = 1;
    }
    return n < 1 ? 1 : n;
}

template <bool F, bool COUNT, bool GEN, int BX>
void launch_batch_shape(const PropGroup& tab, const JobList& J, int ctas_per_sm, int sms, int* next, cudaStream_t st)
{
    const dim3 b(BX, PROP_THREADS / BX);
    auto grid = [&](int resident) {
        const int per_sm = ctas_per_sm > 0 && ctas_per_sm < resident ? ctas_per_sm : resident;
        const long long g = (long long)per_sm * sms;
        return (unsigned)(g < J.njobs ? g : J.njobs);
    };
    k_prop_chain_b<F, COUNT, GEN, BX><<<grid(resident_ctas(k_prop_chain_b<F, COUNT, GEN, BX>)), b, 0, st>>>(
        tab, J.jobs, J.njobs, next);
    k_prop_klt_b<F, COUNT, GEN, BX><<<grid(resident_ctas(k_prop_klt_b<F, COUNT, GEN, BX>)), b, 0, st>>>(
        tab, J.jobs, J.njobs, next + 1);
    k_prop_final_b<F, COUNT, GEN, BX><<<grid(resident_ctas(k_prop_final_b<F, COUNT, GEN, BX>)), b, 0, st>>>(
        tab, J.jobs, J.njobs, next + 2);
}

// the tile shapes of the batched kernels: 32 x 4 pixels (a warp = 32 pixels of a row) or
// 16 x 8 (a warp = two rows of 16)
template <bool F, bool COUNT, bool GEN>
void launch_batch_variant(const PropGroup& tab, const JobList& J, int tile_w, int ctas_per_sm, int sms, int* next,
                          cudaStream_t st)
{
    if (tile_w == 16) launch_batch_shape<F, COUNT, GEN, 16>(tab, J, ctas_per_sm, sms, next, st);
    else launch_batch_shape<F, COUNT, GEN, 32>(tab, J, ctas_per_sm, sms, next, st);
}

}  // namespace

void prop_tile_shape(int* w, int* h)
{
    *w = PROP_BX;
    *h = PROP_BY;
}

bool prop_batch_tile_shape(int tile_w, int* w, int* h)
{
    if (tile_w != 16 && tile_w != 32) return false;
    *w = tile_w;
    *h = PROP_THREADS / tile_w;
    return true;
}

int propagate_batch_launches(int counting) { return counting ? 3 : 6; }

void launch_propagate_batch(const PropParams* group, int n, const JobList& J, int tile_w, int ctas_per_sm, int fused,
                            int counting, int* next, cudaStream_t st)
{
    if (J.njobs <= 0 || n < 1 || n > PROP_GROUP) return;
    static thread_local PropGroup tab;   // 28 KB: off the stack; copied into the launch
    for (int i = 0; i < n; i++) {
        tab.p[i] = group[i];
        tab.p[i].owners = tile_w;
        tab.p[i].list = nullptr;   // the batched Gauss-Newton kernels run every pixel
    }
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) {
        cudaGetLastError();
        sms = 1;
    }
    // as launch_propagate: uncounted passes run both variants (each table entry has dual = 1),
    // counted ones the general variant alone (dual = 0)
    if (counting) {
        if (fused) launch_batch_variant<true, true, true>(tab, J, tile_w, ctas_per_sm, sms, next, st);
        else launch_batch_variant<false, true, true>(tab, J, tile_w, ctas_per_sm, sms, next, st);
    } else if (fused) {
        launch_batch_variant<true, false, false>(tab, J, tile_w, ctas_per_sm, sms, next, st);
        launch_batch_variant<true, false, true>(tab, J, tile_w, ctas_per_sm, sms, next + 3, st);
    } else {
        launch_batch_variant<false, false, false>(tab, J, tile_w, ctas_per_sm, sms, next, st);
        launch_batch_variant<false, false, true>(tab, J, tile_w, ctas_per_sm, sms, next + 3, st);
    }
}

// Pixels per warp of a pass when `pixels` pixels run at a time, windows of half-width r: a thread per pixel (32)
// unless the pixels are so few that their warps, one thread's serial windows each, leave the chip idle.
// Shared windows take 1.6 times the instructions, and small ones do not fill a warp's rows, so they win only while
// about 20 warps per SM (WARPS) hold the pixels with 2 or 4 each.
// Measured, ms a call with 2 / 4 / 32 pixels, disparity maps of 5 iterations (two views) and VPM of 4:
//            64x48               90x68               107x110             160x120             181x130
//   r = 1    1.40 / 1.42 / 1.58  1.79 / 1.49 / 1.60  2.38 / 2.00 / 1.65  3.13 / 2.39 / 1.73  3.60 / 2.76 / 1.77
//   r = 3    1.69 / 1.81 / 2.60  2.30 / 1.97 / 2.64  3.19 / 2.79 / 2.75  4.42 / 3.58 / 2.85  5.14 / 4.16 / 3.00
//   r = 5    2.12 / 2.49 / 4.36  3.00 / 2.81 / 4.45  4.37 / 4.00 / 4.57  6.22 / 5.45 / 4.81  7.35 / 6.48 / 5.26
//   r = 10   4.12 / 5.36 / 12.2  6.19 / 6.50 / 12.4  9.93 / 9.47 / 13.3  14.8 / 14.0 / 14.0  17.6 / 16.7 / 16.0
//   VPM 1    0.20 / 0.22 / 0.31  0.27 / 0.23 / 0.30  0.38 / 0.32 / 0.31  0.50 / 0.39 / 0.32  0.59 / 0.46 / 0.33
//   VPM 5    0.48 / 0.60 / 1.49  0.72 / 0.67 / 1.47  1.09 / 0.99 / 1.55  1.59 / 1.40 / 1.65  1.89 / 1.63 / 1.74
//   VPM 10   1.26 / 1.66 / 4.67  1.91 / 1.95 / 4.61  3.03 / 2.87 / 4.77  4.53 / 4.24 / 5.36  5.35 / 4.90 / 5.51
// Single runs stop at 4 WARPS, where the windows are large enough: the planes of a depth map settle, and the list
// of changed ones is then worth more than sharing (115x115, 9 iterations, 4 / 32 pixels: r = 5 8.9 / 6.9 ms, r = 10
// 16.7 / 16.2; a disparity map 8.2 / 8.4, 19.5 / 24.4).  Pairs of a batch run side by side (`beside`; pm_api.cu,
// batch_load): 32 pairs of 120x90, r = 7: 139 / 119 / 56.6; 16 of 64x48, r = 5: 13.9 / 12.2 / 7.3; 4: 4.2 / 3.8 / 4.8;
// 2: 2.7 / 2.9 / 4.6; 100x80, r = 10, 4 pairs: 21.8 / 19.6 / 18.1, 2: 11.6 / 11.0 / 13.5.
int prop_owners(long long pixels, int r, Model m, bool beside)
{
    constexpr float WARPS = 2960.0f;
    const float n = (float)pixels / WARPS;
    float four = beside ? fminf(fmaxf(2.2f + 0.48f * r, 4.0f), 10.0f) : 4.0f;
    if (m == PMH) four = fminf(four, 2.0f + 0.75f * r);
    return n <= 2.0f ? 2 : n <= four ? 4 : 32;
}

namespace {

template <bool F>
void launch_pass(const PropParams& Q, cudaStream_t st)
{
    const dim3 b(PROP_BX, PROP_BY);
    const dim3 g = grid2d(Q.V.W, Q.V.H, dim3(Q.owners, PROP_BY)), gg = grid2d(Q.V.W, Q.V.H, b);
    PropParams G = Q;
    G.owners = PROP_BX;
    // both variants; the one that does not apply returns at once (pm_window.cuh).  Each kernel of the
    // pass finishes before the next starts, for either variant.
    k_prop_chain<F, false, false><<<g, b, 0, st>>>(Q);
    k_prop_chain<F, false, true><<<gg, b, 0, st>>>(G);
    if (Q.owners <= WARP_KLT) k_prop_klt_warp<F><<<g, b, 0, st>>>(Q);
    else k_prop_klt_list<F><<<(Q.V.W * Q.V.H + PROP_THREADS - 1) / PROP_THREADS, PROP_THREADS, 0, st>>>(Q);
    k_prop_klt<F, false><<<gg, b, 0, st>>>(G);
    k_prop_final<F, false, false><<<g, b, 0, st>>>(Q);
    k_prop_final<F, false, true><<<gg, b, 0, st>>>(G);
}

// counted passes: the general variant alone, which counts
template <bool F>
void launch_pass_counted(const PropParams& Q, cudaStream_t st)
{
    const dim3 b(PROP_BX, PROP_BY);
    const dim3 g = grid2d(Q.V.W, Q.V.H, b);
    k_prop_chain<F, true, true><<<g, b, 0, st>>>(Q);
    k_prop_klt<F, true><<<g, b, 0, st>>>(Q);
    k_prop_final<F, true, true><<<g, b, 0, st>>>(Q);
}

}  // namespace

void launch_propagate(const PropParams& P, int fused, cudaStream_t st)
{
    PropParams Q = P;
    if (P.counters) {
        Q.dual = 0;
        Q.owners = PROP_BX;
        if (fused) launch_pass_counted<true>(Q, st);
        else launch_pass_counted<false>(Q, st);
    } else {
        Q.dual = 1;
        const long long own = (long long)P.V.W * P.V.H;
        Q.owners = prop_owners(P.load > own ? P.load : own, P.V.r, PMH, P.load > own);
        if (Q.owners <= WARP_KLT) Q.list = nullptr;
        if (fused) launch_pass<true>(Q, st);
        else launch_pass<false>(Q, st);
    }
}

}  // namespace pm
