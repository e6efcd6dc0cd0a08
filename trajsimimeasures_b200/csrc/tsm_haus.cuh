// Pruned Hausdorff: one warp per pair, with exact skipping of segments and
// points that cannot change the result.
//
// Both trajectories are staged in shared memory as segment pairs (SegPair,
// tsm_tile.cuh) with the bounding box of every block of 8 segments.  A
// directed distance max_p min_s d(p, s) takes the points of P in groups of 32,
// one per lane:
//   1. For every group an upper bound on its points' minima: the smallest over
//      the blocks of the largest box-to-box distance.
//   2. The groups in order of that bound, largest first; once it is no larger
//      than the maximum m found so far, the rest cannot raise m.
//   3. In a group, the block that gave the bound is evaluated first; another
//      block only if its box lies closer to the group's box than the largest
//      minimum that still counts, and then closer to some lane's point than
//      that lane's minimum so far, which still exceeds m.
// Every evaluation is p2s_pair's, and a skipped one could not have been the
// minimum or the maximum, so the result is the unpruned kernels' bit for bit:
// the bounds are compared with a margin delta above the rounding error of an
// evaluation.  With M the extent of the two trajectories' common bounding box
// and u = 2^-24, an evaluated foot offset differs from the offset to a point
// of the segment by at most 3 u M per coordinate; delta = max(2^-19 M, 2^-62) is 7
// times the resulting length, and twice what underflow can take: the approximate
// square root of a bound flushes squared distances below 2^-126 (lengths below
// 2^-63) to 0.  A widened bound stays a normal number (2^-124 at least).
// Non-finite coordinates set delta to infinity, which turns every skip off.
//
// What bounds it: issue, and the latency of its warp votes and reductions.  On
// pairs of random walks of 20..200 points, of 8 groups (both directions) 3.8
// are evaluated, 6 blocks of 8 segments for them in all, against 112
// without pruning.  Eight segments per box: 4 need 30 box tests a pair
// where 8 need 16, and 16 evaluate 6.7 blocks of twice the size.  Measured on
// B200, unpruned -> pruned, bit for bit the same: 2000 x 2000 of 20..200
// points 39.9 -> 9.1 ms, 1200 x 1500 18.5 -> 4.2 ms, 600 x 600 of 20..700
// points 55.3 -> 6.2 ms; 200,000 pairs of 20..200 points 6.7 -> 0.94 ms, 50,000
// lognormal pairs (10..2000 points) 8.8 -> 0.59 ms.  64 registers (32 warps
// per SM); 48 (40 warps) spill: 10.9 ms for the first case.  Finishing a group
// with one lane per segment once few of its points count was slower (12.0), and
// so was leaving out a group's tests after three that skipped nothing (2.46 ->
// 2.87 ms for 1000 x 1000, and 13.1 -> 17.4 on points without any order).
//
// A pair with a long trajectory (22 bytes of shared memory a point) is a CTA's,
// so that 8 to 24 warps work on an SM whatever the lengths; its warps take the
// groups side by side and share the maximum, which skips a little less than one
// warp after the other (1.00 ms for 200 x 200 of 300..500 points by CTAs, 0.68 by
// warps, which still fit 16 times there).  From 256 points on (320, 384, 512): 600 x
// 600 of 20..700 points 6.3 ms (6.1, 7.2, 6.2; 5.7 by eight warps an SM), 1,000 of
// 20..200 and one of 1,000 3.2 (4.1, 4.1, 4.1; 7.2), 100 x 100 of 800..1000 0.48
// (0.60, 0.60, 0.60; 0.90).
#pragma once

#include <type_traits>

#include "tsm_tile.cuh"

namespace tsm {

constexpr int kHausBlk = 8;                   // segments per box
constexpr int kHausGrp = 32 / kHausBlk;       // boxes per group of 32 points
constexpr float kHausSlack = 1.f + 0x1p-18f;  // above the rounding of the squared bounds themselves

// Shared memory of one staged trajectory of up to cap points, in floats: the
// segment pairs (A, B float4, C float2) and the boxes of the blocks and of the
// groups (float4).
__host__ __device__ constexpr int haus_pairs(int cap) { return (cap + 1) / 2; }
__host__ __device__ constexpr int haus_blocks(int cap) { return (cap + kHausBlk - 1) / kHausBlk; }
__host__ __device__ constexpr int haus_groups(int cap) { return (cap + 31) / 32; }
__host__ __device__ constexpr int haus_floats(int cap) {
    return 8 * haus_pairs(cap) + 4 * (haus_blocks(cap) + haus_groups(cap)) + 2 * ((haus_pairs(cap) + 1) & ~1);
}

// A staged trajectory: n points (segment k = point k to k + 1; the last
// vertex is a zero-length segment), box = its bounding box (xlo, xhi, ylo,
// yhi), all infinite when a coordinate is not finite.
struct HausTraj {
    float4 *A, *B, *box, *grp;
    float2* C;
    int n;
    float4 bb;
    __device__ __forceinline__ HausTraj(float* base, int cap) {
        A = reinterpret_cast<float4*>(base);
        B = A + haus_pairs(cap);
        box = B + haus_pairs(cap);
        grp = box + haus_blocks(cap);
        C = reinterpret_cast<float2*>(grp + haus_groups(cap));
        n = 0;
    }
    __device__ __forceinline__ float2 pt(int k) const {  // point k negated
        const float* a = reinterpret_cast<const float*>(A + (k >> 1)) + (k & 1);
        return make_float2(a[0], a[2]);
    }
};

__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Who works on a pair: one warp (TEAM false) or all warps of the CTA.
template <bool TEAM>
struct HausGang {
    static __device__ __forceinline__ int rank() { return TEAM ? threadIdx.x : threadIdx.x & 31; }
    static __device__ __forceinline__ int size() { return TEAM ? blockDim.x : 32; }
    static __device__ __forceinline__ void sync() {
        if constexpr (TEAM) __syncthreads();
        else __syncwarp();
    }
    static __device__ __forceinline__ bool all(bool v) {
        if constexpr (TEAM) return __syncthreads_and(v);
        else return __all_sync(0xffffffffu, v);
    }
};

// Stages n points (all threads of the gang); the boxes include both end points
// of every segment of their block.
template <bool EXACT, bool TEAM>
__device__ __forceinline__ void haus_stage(HausTraj& t, const float2* __restrict__ p, int n) {
    using G = HausGang<TEAM>;
    const int rank = G::rank(), size = G::size(), lane = threadIdx.x & 31;
    t.n = n;
    bool fin = true;
    const int npair = (n + 1) >> 1;
    for (int j = rank; j < npair; j += size) {
        const int k0 = 2 * j, k1 = min(k0 + 1, n - 1), k2 = min(k0 + 2, n - 1);
        const float2 v0 = __ldg(p + k0), v1 = __ldg(p + k1), v2 = __ldg(p + k2);
        SegPair g;
        seg_lane<EXACT>(g, 0, v0, v1);
        seg_lane<EXACT>(g, 1, v1, v2);
        t.A[j] = make_float4(g.n1x.x, g.n1x.y, g.n1y.x, g.n1y.y);
        t.B[j] = make_float4(g.nsx.x, g.nsx.y, g.nsy.x, g.nsy.y);
        t.C[j] = g.ninv;
        fin = fin && isfinite(v0.x) && isfinite(v0.y) && isfinite(v1.x) && isfinite(v1.y);
    }
    G::sync();
    float4 u = make_float4(CUDART_INF_F, -CUDART_INF_F, CUDART_INF_F, -CUDART_INF_F);
    auto widen = [&](const float4& v) {
        u.x = fminf(u.x, v.x);
        u.y = fmaxf(u.y, v.y);
        u.z = fminf(u.z, v.z);
        u.w = fmaxf(u.w, v.w);
    };
    for (int b = rank; b < (n + kHausBlk - 1) / kHausBlk; b += size) {
        float4 v = make_float4(CUDART_INF_F, -CUDART_INF_F, CUDART_INF_F, -CUDART_INF_F);
#pragma unroll
        for (int k = 0; k <= kHausBlk; k += 2) {  // vertices 8 b .. 8 b + 8, two per pair
            const int j = min((kHausBlk * b + k) >> 1, npair - 1);
            const float4 a = t.A[j];
            // an odd count repeats the last vertex; the last pair's second vertex lies past the block
            const bool two = k < kHausBlk;
            v.x = min3f(v.x, -a.x, two ? -a.y : -a.x);
            v.y = max3f(v.y, -a.x, two ? -a.y : -a.x);
            v.z = min3f(v.z, -a.z, two ? -a.w : -a.z);
            v.w = max3f(v.w, -a.z, two ? -a.w : -a.z);
        }
        t.box[b] = v;
        if (!TEAM) widen(v);
    }
    G::sync();
    for (int g = rank; g < (n + 31) >> 5; g += size) {
        float4 v = t.box[kHausGrp * g];
        for (int i = 1; i < kHausGrp; ++i) {
            const float4 w = t.box[min(kHausGrp * g + i, haus_blocks(n) - 1)];
            v = make_float4(fminf(v.x, w.x), fmaxf(v.y, w.y), fminf(v.z, w.z), fmaxf(v.w, w.w));
        }
        t.grp[g] = v;
    }
    if constexpr (TEAM) {  // every warp makes the whole box
        G::sync();
        for (int g = lane; g < (n + 31) >> 5; g += 32) widen(t.grp[g]);
    }
    u.x = warp_min(u.x);
    u.y = -warp_min(-u.y);
    u.z = warp_min(u.z);
    u.w = -warp_min(-u.w);
    t.bb = G::all(fin) ? u : make_float4(-CUDART_INF_F, CUDART_INF_F, -CUDART_INF_F, CUDART_INF_F);
    if (!TEAM) G::sync();
}

// Squared smallest and largest distance of two boxes (a point: lo = hi).
__device__ __forceinline__ float box_near2(const float4& a, const float4& b) {
    const float dx = max3f(0.f, a.x - b.y, b.x - a.y), dy = max3f(0.f, a.z - b.w, b.z - a.w);
    return fmaf(dx, dx, dy * dy);
}
__device__ __forceinline__ float box_far2(const float4& a, const float4& b) {
    const float dx = fmaxf(a.y - b.x, b.y - a.x), dy = fmaxf(a.w - b.z, b.w - a.z);
    return fmaf(dx, dx, dy * dy);
}
// (sqrt(d2) + delta)^2, rounded up: a squared bound with the margin.
__device__ __forceinline__ float widen2(float d2, float delta) {
    const float s = tsqrt<false>(d2) + delta;
    return s * s * kHausSlack;
}

// max(m, max over the points of P of the min over the segments of T), by one
// warp (m and the result uniform), or the groups of P shared out to the warps of
// a CTA (TEAM): a warp's result is then the largest that it or, as far as it has
// seen, another one found, and *shared (a float's bits, not below m) the largest
// of all once every warp is through.
template <bool TEAM>
__device__ __forceinline__ float haus_directed(const HausTraj& P, const HausTraj& T, float m, float delta, int lane,
                                               int* shared) {
    constexpr unsigned kFull = 0xffffffffu;
    if (T.n < 2 || P.n <= 0) return m;
    const int w0 = TEAM ? threadIdx.x >> 5 : 0, nw = TEAM ? blockDim.x >> 5 : 1;
    const int ngrp = (P.n + 31) >> 5, nblk = (T.n + kHausBlk - 1) / kHausBlk, npair = (T.n + 1) >> 1;
    for (int g0 = 0; g0 < ngrp; g0 += 32) {
        // lane l keeps the bound of group g0 + l (0: done; a bound is not, see delta) and the block it came from
        const int ng = min(32, ngrp - g0);
        uint32_t ub = 0;
        int ubb = 0;
        for (int g = w0; g < ng; g += nw) {
            const float4 gb = P.grp[g0 + g];
            float far = CUDART_INF_F;
            int fb = 0;
            for (int b = lane; b < nblk; b += 32) {
                const float f = box_far2(gb, T.box[b]);
                if (f < far) {
                    far = f;
                    fb = b;
                }
            }
            const uint32_t best = __reduce_min_sync(kFull, __float_as_uint(far));
            const int src = __ffs(__ballot_sync(kFull, __float_as_uint(far) == best)) - 1;
            fb = __shfl_sync(kFull, fb, src);
            if (lane == g) {
                ub = __float_as_uint(widen2(__uint_as_float(best), delta));
                ubb = fb;
            }
        }
        for (;;) {
            // the remaining group with the largest bound (bounds are not negative: ordered like their bits)
            const uint32_t top = __reduce_max_sync(kFull, ub);
            if constexpr (TEAM) {
                const int seen = lane == 0 ? *reinterpret_cast<volatile int*>(shared) : 0;
                m = fmaxf(m, __int_as_float(__shfl_sync(kFull, seen, 0)));
            }
            if (__uint_as_float(top) <= m || top == 0) break;
            const int g = __ffs(__ballot_sync(kFull, ub == top)) - 1;
            const int first = __shfl_sync(kFull, ubb, g);
            if (lane == g) ub = 0;
            const int k = (g0 + g) * 32 + lane;
            const bool valid = k < P.n;
            const float2 np = P.pt(min(k, P.n - 1));
            const float4 pb = make_float4(-np.x, -np.x, -np.y, -np.y);
            const float2 px = make_float2(-np.x, -np.x), py = make_float2(-np.y, -np.y);
            float best = CUDART_INF_F;
            auto eval = [&](int b) {
                const int j1 = min((b + 1) * (kHausBlk / 2), npair);
                for (int j = b * (kHausBlk / 2); j < j1; ++j) best = p2s_pair(px, py, staged_pair(T.A, T.B, T.C, j), best);
            };
            eval(first);
            float thr = (valid && best > m) ? widen2(best, delta) : -1.f;  // below any bound: this lane needs no more
            const float4 gb = P.grp[g0 + g];
            for (int b0 = 0; b0 < nblk; b0 += 32) {
                const float most = __uint_as_float(__reduce_max_sync(kFull, thr < 0.f ? 0u : __float_as_uint(thr)));
                unsigned todo = __ballot_sync(kFull, b0 + lane < nblk && b0 + lane != first &&
                                                         box_near2(gb, T.box[min(b0 + lane, nblk - 1)]) <= most);
                while (todo) {
                    const int b = b0 + __ffs(todo) - 1;
                    todo &= todo - 1;
                    if (!__any_sync(kFull, box_near2(pb, T.box[b]) <= thr)) continue;
                    eval(b);
                    thr = (valid && best > m) ? widen2(best, delta) : -1.f;
                }
            }
            const uint32_t top_min = __reduce_max_sync(kFull, valid ? __float_as_uint(best) : 0u);
            if (TEAM && lane == 0 && __uint_as_float(top_min) > m) atomicMax(shared, (int)top_min);
            m = fmaxf(m, __uint_as_float(top_min));
        }
    }
    return m;
}

// The squared Hausdorff distance of two staged trajectories.  TEAM: of the CTA's
// pair, *shared 0 before; each warp's part of it, all in *shared once every warp
// is through.
template <bool TEAM>
__device__ __forceinline__ float haus_pair(const HausTraj& a, const HausTraj& b, int lane, int* shared) {
    const float w = fmaxf(a.bb.y, b.bb.y) - fminf(a.bb.x, b.bb.x), h = fmaxf(a.bb.w, b.bb.w) - fminf(a.bb.z, b.bb.z);
    const float delta = fmaxf(0x1p-19f * (w + h), 0x1p-62f);
    const float m = haus_directed<TEAM>(a, b, 0.f, delta, lane, shared);
    return haus_directed<TEAM>(b, a, m, delta, lane, shared);
}

// Matrix kernel: CTA (t, chunk) stages the queries q_order[QB t ..] (QB of
// them, one per warp); its warps take the database slots of the chunk
// (per_cta of them) in turn, each staging the trajectory in its own shared
// memory once for all QB queries.  Query order, symmetric and gather modes as
// in dp_matrix_kernel (gather: QB = 1, since every query has its own slots).
// Dynamic shared memory = QB * haus_floats(q cap) + W * haus_floats(d cap)
// floats, W >= QB.
template <int QB, bool EXACT>
__global__ void __launch_bounds__(256) hausdorff_pruned_matrix_kernel(
    const float2* __restrict__ q_pts, const int64_t* __restrict__ q_off, const int32_t* __restrict__ q_len,
    const int32_t* __restrict__ q_order, int64_t nq, const float2* __restrict__ d_pts,
    const int64_t* __restrict__ d_off, const int32_t* __restrict__ d_len, const int32_t* __restrict__ d_order,
    int64_t nd, int64_t d_total, int chunks, int per_cta, int sym, int q_cap, int d_cap, float* __restrict__ out,
    int64_t ld) {
    extern __shared__ float4 smem4[];
    float* smem = reinterpret_cast<float*>(smem4);
    __shared__ float4 q_bb[QB];
    __shared__ int q_n[QB];  // -1: outside the set or a bad length
    __shared__ int64_t q_id[QB];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const int64_t qs0 = (int64_t)(blockIdx.x / chunks) * QB;
    const int64_t s0 = (int64_t)(blockIdx.x % chunks) * per_cta;
    const int64_t s1 = min(nd, s0 + per_cta);
    if (sym == 1 && s1 <= qs0) return;
    if (warp < QB) {
        const int64_t qs = qs0 + warp;
        const int64_t qi = qs < nq ? (q_order ? (int64_t)q_order[qs] : qs) : 0;
        int n = qs < nq ? q_len[qi] : -1;
        if (n > q_cap) n = -1;
        if (n >= 0) {
            HausTraj q(smem + warp * haus_floats(q_cap), q_cap);
            haus_stage<EXACT, false>(q, q_pts + q_off[qi], n);
            if (lane == 0) q_bb[warp] = q.bb;
        }
        if (lane == 0) {
            q_n[warp] = n;
            q_id[warp] = qi;
        }
    }
    __syncthreads();
    HausTraj d(smem + QB * haus_floats(q_cap) + warp * haus_floats(d_cap), d_cap);
    for (int64_t slot = s0 + warp; slot < s1; slot += nwarp) {
        if (sym == 1 && slot < qs0) continue;
        const int64_t dj = d_order ? (int64_t)d_order[(sym == 2 ? q_id[0] * nd : 0) + slot] : slot;
        const bool dbad = dj < 0 || dj >= d_total;
        int n = dbad ? -1 : d_len[dj];
        if (n > d_cap) n = -1;
        if (n >= 0) haus_stage<EXACT, false>(d, d_pts + d_off[dj], n);
        for (int i = 0; i < QB; ++i) {
            if (qs0 + i >= nq || (sym == 1 && slot < qs0 + i)) break;
            float v = CUDART_NAN_F;
            if (n >= 0 && q_n[i] >= 0) {
                HausTraj q(smem + i * haus_floats(q_cap), q_cap);
                q.n = q_n[i];
                q.bb = q_bb[i];
                v = __fsqrt_rn(haus_pair<false>(q, d, lane, nullptr));
            }
            const int64_t qi = q_id[i];
            if (lane == 0) {
                out[qi * ld + (sym == 2 ? slot : dj)] = v;
                if (sym == 1 && dj != qi) out[dj * ld + qi] = v;
            }
        }
        __syncwarp();  // the staged trajectory is free
    }
}

// The same for a database with long trajectories.  A slot of at most w_cap points
// is one warp's as above; a longer one is the CTA's, staged over the warps' memory,
// with the groups of its pairs shared out to the warps: one long trajectory does
// not leave room for a few warps only.  (Short databases keep the kernel above:
// in this one the CTA's part takes registers from the warps', 2000 x 2000 of
// 20..200 points 5 % slower.)  Dynamic shared memory = QB * haus_floats(q cap) +
// max(W * haus_floats(w cap), haus_floats(d cap)) floats, W >= QB, per_cta <= 64.
template <int QB, bool EXACT>
__global__ void __launch_bounds__(256, 3) hausdorff_long_matrix_kernel(
    const float2* __restrict__ q_pts, const int64_t* __restrict__ q_off, const int32_t* __restrict__ q_len,
    const int32_t* __restrict__ q_order, int64_t nq, const float2* __restrict__ d_pts,
    const int64_t* __restrict__ d_off, const int32_t* __restrict__ d_len, const int32_t* __restrict__ d_order,
    int64_t nd, int64_t d_total, int chunks, int per_cta, int sym, int q_cap, int w_cap, int d_cap,
    float* __restrict__ out, int64_t ld) {
    extern __shared__ float4 smem4[];
    float* smem = reinterpret_cast<float*>(smem4);
    __shared__ float4 q_bb[QB];
    __shared__ int q_n[QB];  // -1: outside the set or a bad length
    __shared__ int64_t q_id[QB];
    __shared__ unsigned longs[2];  // bit s: slot s0 + s of the chunk is longer than w_cap
    __shared__ int found[QB];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const int64_t qs0 = (int64_t)(blockIdx.x / chunks) * QB;
    const int64_t s0 = (int64_t)(blockIdx.x % chunks) * per_cta;
    const int64_t s1 = min(nd, s0 + per_cta);
    if (sym == 1 && s1 <= qs0) return;
    if (threadIdx.x < 2) longs[threadIdx.x] = 0;
    auto stage_query = [&](int i, auto team) {
        const int64_t qs = qs0 + i;
        const int64_t qi = qs < nq ? (q_order ? (int64_t)q_order[qs] : qs) : 0;
        int n = qs < nq ? q_len[qi] : -1;
        if (n > q_cap) n = -1;
        if (n >= 0) {
            HausTraj q(smem + i * haus_floats(q_cap), q_cap);
            haus_stage<EXACT, decltype(team)::value>(q, q_pts + q_off[qi], n);
            if (lane == 0) q_bb[i] = q.bb;  // (TEAM: the same from every warp)
        }
        if (lane == 0) {
            q_n[i] = n;
            q_id[i] = qi;
        }
    };
    if constexpr (QB == 1) stage_query(0, std::true_type{});  // (all warps on the one)
    else if (warp < QB) stage_query(warp, std::false_type{});
    __syncthreads();
    float* area = smem + QB * haus_floats(q_cap);
    // a slot's database index and length (-1: outside the set or a bad length)
    auto slot_of = [&](int64_t slot, int64_t& dj) {
        dj = d_order ? (int64_t)d_order[(sym == 2 ? q_id[0] * nd : 0) + slot] : slot;
        const int n = dj < 0 || dj >= d_total ? -1 : d_len[dj];
        return n > d_cap ? -1 : n;
    };
    // the pairs of a slot, staged as d (n >= 0)
    auto pairs_of = [&](const HausTraj& d, int n, int64_t slot, int64_t dj, auto team) {
        constexpr bool TEAM = decltype(team)::value;
        for (int i = 0; i < QB; ++i) {
            if (qs0 + i >= nq || (sym == 1 && slot < qs0 + i)) break;
            float v = CUDART_NAN_F;
            if (n >= 0 && q_n[i] >= 0) {
                HausTraj q(smem + i * haus_floats(q_cap), q_cap);
                q.n = q_n[i];
                q.bb = q_bb[i];
                v = haus_pair<TEAM>(q, d, lane, found + i);
            }
            if (TEAM) continue;
            const int64_t qi = q_id[i];
            if (lane == 0) {
                v = __fsqrt_rn(v);
                out[qi * ld + (sym == 2 ? slot : dj)] = v;
                if (sym == 1 && dj != qi) out[dj * ld + qi] = v;
            }
        }
    };
    HausTraj d(area + warp * haus_floats(w_cap), w_cap);
    for (int64_t slot = s0 + warp; slot < s1; slot += nwarp) {
        if (sym == 1 && slot < qs0) continue;
        int64_t dj;
        const int n = slot_of(slot, dj);
        if (n > w_cap) {
            if (lane == 0) atomicOr(&longs[(slot - s0) >> 5], 1u << ((slot - s0) & 31));
            continue;
        }
        if (n >= 0) haus_stage<EXACT, false>(d, d_pts + d_off[dj], n);
        pairs_of(d, n, slot, dj, std::false_type{});
        __syncwarp();  // the staged trajectory is free
    }
    __syncthreads();
    HausTraj t(area, d_cap);
    for (int h = 0; h < 2; ++h)
        for (unsigned todo = longs[h]; todo; todo &= todo - 1) {
            const int64_t slot = s0 + 32 * h + __ffs(todo) - 1;
            int64_t dj;
            const int n = slot_of(slot, dj);
            if (threadIdx.x < QB) found[threadIdx.x] = 0;
            haus_stage<EXACT, true>(t, d_pts + d_off[dj], n);
            pairs_of(t, n, slot, dj, std::true_type{});
            __syncthreads();  // every warp is through
            if (threadIdx.x < QB) {
                const int i = threadIdx.x;
                if (qs0 + i < nq && !(sym == 1 && slot < qs0 + i)) {
                    const float v = q_n[i] < 0 ? CUDART_NAN_F : __fsqrt_rn(__int_as_float(found[i]));
                    const int64_t qi = q_id[i];
                    out[qi * ld + (sym == 2 ? slot : dj)] = v;
                    if (sym == 1 && dj != qi) out[dj * ld + qi] = v;
                }
            }
        }
}

// Pairs kernel: the pairs of more than warp_cells point products whose longer
// side is above min_side and at most cap points (the others are another launch's,
// hausdorff_pairs_kernel's or hausdorff_wave_kernel's), one warp each or (TEAM)
// one CTA each.  Persistent, with the pair assignment of dp_wave_kernel.  Dynamic
// shared memory = 2 * haus_floats(cap) floats for each pair in work.
template <bool TEAM, bool EXACT>
__global__ void __launch_bounds__(256) hausdorff_pruned_pairs_kernel(
    const float2* __restrict__ pts, const int64_t* __restrict__ off_a, const int32_t* __restrict__ len_a,
    const int64_t* __restrict__ off_b, const int32_t* __restrict__ len_b, const int32_t* __restrict__ order,
    int64_t n, int min_side, int cap, int64_t warp_cells, float* __restrict__ out) {
    extern __shared__ float4 smem4[];
    __shared__ int found;
    const int lane = threadIdx.x & 31, warp = TEAM ? 0 : threadIdx.x >> 5;
    float* smem = reinterpret_cast<float*>(smem4) + warp * 2 * haus_floats(cap);
    HausTraj a(smem, cap), b(smem + haus_floats(cap), cap);
    const int per = TEAM ? 1 : blockDim.x >> 5;
    const int64_t gw = (int64_t)blockIdx.x * per + warp;
    const int64_t nw = (int64_t)gridDim.x * per;
    for (int64_t i0 = 0; i0 * nw < n; i0 += 32) {
        const int64_t i = i0 + lane;
        const int64_t t = i * nw + ((i & 1) ? nw - 1 - gw : gw);
        int64_t k = 0;
        bool mine = false;
        if (t < n) {
            k = order ? (int64_t)order[t] : t;
            const int na = len_a[k], nb = len_b[k];
            mine = na >= 0 && nb >= 0 && na <= cap && nb <= cap && max(na, nb) > min_side &&
                   (int64_t)na * nb > warp_cells;
        }
        unsigned todo = __ballot_sync(0xffffffffu, mine);  // (TEAM: the same in every warp)
        while (todo) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1;
            const int64_t kk = __shfl_sync(0xffffffffu, k, src);
            if (TEAM && threadIdx.x == 0) found = 0;
            haus_stage<EXACT, TEAM>(a, pts + off_a[kk], len_a[kk]);
            haus_stage<EXACT, TEAM>(b, pts + off_b[kk], len_b[kk]);
            const float v = haus_pair<TEAM>(a, b, lane, &found);
            HausGang<TEAM>::sync();
            if (TEAM) {
                if (threadIdx.x == 0) out[kk] = __fsqrt_rn(__int_as_float(found));
                __syncthreads();  // (read before the next pair clears it)
            } else if (lane == 0) {
                out[kk] = __fsqrt_rn(v);
            }
        }
    }
}

}  // namespace tsm
