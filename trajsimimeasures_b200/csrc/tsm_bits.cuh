// EDR and LCSS counts, 32 DP rows per machine word.
//
// Neighbouring cells of both tables differ by at most one, so a column of 32
// rows is held as bit vectors of its vertical differences and advanced by a
// dozen integer operations: for EDR Myers' block step (JACM 46(3), 1999),
// with the reference's zero borders as zero initial differences, for LCSS the
// addition form of Crochemore et al. (IPL 80(6), 2001) and Hyyro (2004).  The
// count is the sum of the last column's differences, an exact integer, equal
// to the cell-by-cell recurrence's.  What is left per cell is its match test
// d2 < eps2 (d2nr, tsm_device.cuh): a thread holds 32 rows in registers and
// makes the match word of a column point, unless the point lies so far from
// the box of the 32 rows that no row can match.
//
// The far test is exact: with epsr a float whose rounded square is at least
// eps2, a column x at or above the rounded-up sum xhi + epsr has
// fl(c.x - r.x) >= epsr for every row (rounding is monotone), hence a rounded
// d2 of at least eps2.  Points with NaN coordinates match nothing and widen no
// box.
//
// Rows ahead of the first that can match: with no match the EDR table is
// D(i, j) = min(i, j) + 1 and the LCSS table 0, so such a block of rows is not
// swept, and a pair whose boxes are apart costs one test.
//
// What bounds it: issue.  Per 32 cells 26 instructions where no row can match
// and about 220 where one can, against 7.6 (LCSS) and 8.8 (EDR) a cell for the
// cell-by-cell kernels this replaced.  Measured on B200, before -> after, same
// counts: all-pairs 2000 x 2000 random walks of 20..200 points EDR 13.9 ->
// 0.49 ms, LCSS 12.5 -> 0.42 (1.10 and 0.97 with the pairs to sweep left in
// their lanes instead of collected); 400 x 400 of 20..1000 points EDR 56 ->
// 2.2; 200,000 EDR pairs of 20..200 points in any order 2.7 -> 0.29.  1000 x
// 1000 of 20..200 points with everything within reach of everything, where no
// test helps: EDR 3.71 -> 3.74, LCSS 3.35 -> 3.48 (600 x 600 1.68 -> 1.74 and
// 1.51 -> 1.66, 200 x 200 0.46 -> 0.51 and 0.38 -> 0.48, where the launch is as long
// as a lane's longest pairs; 1000 x 1000 of 2..20 points 0.095 -> 0.119 and 0.082 ->
// 0.114).  Tried and slower: eight lanes per pair with four ballots a column (100 x
// 100 as one warp per pair, 600 x 600 4.1 ms), loading a short word's rows only
// (registers: 600 x 600 1.86), a second loop without tests for words near
// everything, match masks by set instead of predicates (2.26).
#pragma once

#include "tsm_device.cuh"

namespace tsm {

// Words of shared memory per lane for the carries of a block of rows into the
// next, nc columns (EDR: two bits a column).
__host__ __device__ constexpr int bits_words(int nc) { return 2 * ((nc + 31) / 32); }

// A box (xlo, xhi, ylo, yhi).
__device__ __forceinline__ float4 empty_box() {
    return make_float4(CUDART_INF_F, -CUDART_INF_F, CUDART_INF_F, -CUDART_INF_F);
}
__device__ __forceinline__ float4 box_add(const float4& b, float2 p) {
    return make_float4(fminf(b.x, p.x), fmaxf(b.y, p.x), fminf(b.z, p.y), fmaxf(b.w, p.y));
}
// The limits at or beyond which a coordinate is far from box b.
__device__ __forceinline__ float4 far_limits(const float4& b, float epsr) {
    return make_float4(__fsub_rd(b.x, epsr), __fadd_ru(b.y, epsr), __fsub_rd(b.z, epsr), __fadd_ru(b.w, epsr));
}
__device__ __forceinline__ bool far_point(const float4& f, float2 c) {
    return c.x <= f.x || c.x >= f.y || c.y <= f.z || c.y >= f.w;
}
__device__ __forceinline__ bool far_box(const float4& f, const float4& c) {
    return c.y <= f.x || c.x >= f.y || c.w <= f.z || c.z >= f.w;
}

// Warp minimum / maximum of floats that are not NaN, through order-preserving integers.
__device__ __forceinline__ int ordered_int(float v) {
    const int k = __float_as_int(v);
    return k ^ ((k >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float ordered_float(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7fffffff)); }
// The box of n points, by one warp (uniform arguments and result).
__device__ __forceinline__ float4 warp_box(const float2* p, int n, int lane) {
    float4 b = empty_box();
    for (int i = lane; i < n; i += 32) b = box_add(b, p[i]);
    return make_float4(ordered_float(__reduce_min_sync(0xffffffffu, ordered_int(b.x))),
                       ordered_float(__reduce_max_sync(0xffffffffu, ordered_int(b.y))),
                       ordered_float(__reduce_min_sync(0xffffffffu, ordered_int(b.z))),
                       ordered_float(__reduce_max_sync(0xffffffffu, ordered_int(b.w))));
}
// The boxes of the lanes' own trajectories (p, n; n <= 0: none): one after the
// other by the whole warp (coalesced loads, but a load's latency each) or, where
// all are short, each by its lane.  All 32 lanes call it.
__device__ __forceinline__ float4 lane_boxes(const float2* p, int n, int lane) {
    float4 mine = empty_box();
    if (__reduce_max_sync(0xffffffffu, n) <= 32) {
#pragma unroll 4
        for (int i = 0; i < n; ++i) mine = box_add(mine, __ldg(p + i));
        return mine;
    }
    unsigned todo = __ballot_sync(0xffffffffu, n > 0);
    while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        const float2* q = reinterpret_cast<const float2*>(
            __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(p), src));
        const float4 b = warp_box(q, __shfl_sync(0xffffffffu, n, src), lane);
        if (lane == src) mine = b;
    }
    return mine;
}

// One column of 32 rows.  EDR: vp, vn the +1 and -1 vertical differences, cp
// and cn the +1 and -1 horizontal differences above the rows (EDR) of the
// columns to come, this one in bit 0; the differences below the rows enter at
// bit 31.  LCSS: v with 0 bits for +1 differences, cp the carries.
template <int M>
__device__ __forceinline__ void bits_column(uint32_t eq, uint32_t& vp, uint32_t& vn, uint32_t& cp, uint32_t& cn) {
    if constexpr (M == EDR) {
        const uint32_t x = eq | (cn & 1u);
        const uint32_t xh = (((x & vp) + vp) ^ vp) | x, xv = eq | vn;
        const uint32_t hp = vn | ~(xh | vp), hn = vp & xh;
        const uint32_t hps = hp + hp + (cp & 1u), hns = hn + hn + (cn & 1u);
        cp = (cp >> 1) | (hp & 0x80000000u);
        cn = (cn >> 1) | (hn & 0x80000000u);
        vp = hns | ~(xv | hps);
        vn = hps & xv;
    } else {
        uint32_t& v = vp;
        const uint32_t u = v & eq;
        const uint32_t s = v + u + (cp & 1u);
        cp = (cp >> 1) | (((v & u) | ((v | u) & ~s)) & 0x80000000u);
        v = s | (v & ~eq);
    }
}
template <int M>
__device__ __forceinline__ int bits_total(uint32_t vp, uint32_t vn, int rows) {
    const uint32_t valid = rows >= 32 ? 0xffffffffu : (1u << rows) - 1u;
    return M == EDR ? __popc(vp & valid) - __popc(vn & valid) : __popc(~vp & valid);
}
template <int M>
__device__ __forceinline__ uint32_t bits_start() {
    return M == EDR ? 0u : 0xffffffffu;
}

// The EDR or LCSS count of one lane's pair (nr, nc >= 1): rows rowp, columns
// cols.pt(j) inside the box cbox; carry: this lane's bits_words(nc) words,
// word w at carry[32 * w].
template <int M, class Cols>
__device__ __forceinline__ int bits_count(const float2* __restrict__ rowp, int nr, const Cols& cols, int nc,
                                          uint32_t* carry, float eps2, float epsr, const float4& cbox) {
    static_assert(M == EDR || M == LCSS, "integer counts");
    bool ahead = true;  // no block of rows swept yet
    int total = M == EDR ? min(nr, nc) : 0;
#pragma unroll 1
    for (int rb = 0; rb < nr; rb += 32) {
        float2 n[32];  // negated, for d2nr; rows past the end repeat the last and are masked at the end
        float4 box = empty_box();
#pragma unroll
        for (int r = 0; r < 32; ++r) {
            const float2 q = __ldg(rowp + min(rb + r, nr - 1));
            box = box_add(box, q);
            n[r] = make_float2(-q.x, -q.y);
        }
        const float4 f = far_limits(box, epsr);
        if (ahead && far_box(f, cbox)) continue;
        uint32_t vp = bits_start<M>(), vn = 0;
#pragma unroll 1
        for (int jb = 0; jb < nc; jb += 32) {
            // carries of columns jb .. jb + 31 from the rows above: bit i is column jb + i.  They are taken from
            // the low end while the carries out enter at the high end.
            uint32_t* cw = carry + 2 * jb;
            uint32_t cp = M == EDR && jb < rb ? 0xffffffffu : 0u, cn = 0;
            if (!ahead) {
                cp = cw[0];
                if (M == EDR) cn = cw[32];
            }
            const int e = min(32, nc - jb);
#pragma unroll 1
            for (int i = 0; i < e; ++i) {
                const float2 c = cols.pt(jb + i);
                uint32_t eq = 0;
                if (!far_point(f, c)) {
                    uint32_t m[4] = {0, 0, 0, 0};
#pragma unroll
                    for (int g = 0; g < 32; g += 8) {  // no tests past the last rows' group of eight
                        if (rb + g >= nr) break;
#pragma unroll
                        for (int r = g; r < g + 8; ++r) {
                            const float d2 = d2nr(n[r], c);
                            asm("{\n\t.reg .pred q;\n\tsetp.lt.f32 q, %1, %2;\n\t@q add.u32 %0, %0, %3;\n\t}"
                                : "+r"(m[r & 3])
                                : "f"(d2), "f"(eps2), "r"(1u << r));
                        }
                    }
                    eq = (m[0] | m[1]) | (m[2] | m[3]);
                }
                bits_column<M>(eq, vp, vn, cp, cn);
            }
            cw[0] = cp >> (32 - e);
            if (M == EDR) cw[32] = cn >> (32 - e);
        }
        if (M == EDR && ahead) total = min(rb, nc);
        total += bits_total<M>(vp, vn, nr - rb);
        ahead = false;
    }
    return total;
}

// The same count by a whole warp (uniform arguments and result): lane l tests
// row l of each block of 32, and a ballot makes the match word.  30
// instructions a word and column whatever matches, so better than one lane
// among idle ones, and a quarter of its time.  carry: bits_words(nc) words,
// contiguous.
template <int M>
__device__ __forceinline__ int bits_count_warp(const float2* __restrict__ rowp, int nr, const float2* cols, int nc,
                                               uint32_t* carry, float eps2, float epsr, const float4& cbox, int lane) {
    constexpr unsigned kFull = 0xffffffffu;
    const float4 f = far_limits(cbox, epsr);
    bool ahead = true;
    int total = M == EDR ? min(nr, nc) : 0;
    for (int rb = 0; rb < nr; rb += 32) {
        const float2 q = __ldg(rowp + min(rb + lane, nr - 1));
        const float2 n = make_float2(-q.x, -q.y);
        if (ahead && __all_sync(kFull, far_point(f, q))) continue;
        uint32_t vp = bits_start<M>(), vn = 0;
        for (int jb = 0; jb < nc; jb += 32) {
            uint32_t* cw = carry + jb / 16;
            uint32_t cp = M == EDR && jb < rb ? 0xffffffffu : 0u, cn = 0;
            if (!ahead) {
                cp = cw[0];
                cn = cw[1];
            }
            __syncwarp();
            const int e = min(32, nc - jb);
#pragma unroll 4
            for (int i = 0; i < e; ++i) {
                const uint32_t eq = __ballot_sync(kFull, d2nr(n, cols[jb + i]) < eps2);
                bits_column<M>(eq, vp, vn, cp, cn);
            }
            if (lane == 0) {
                cw[0] = cp >> (32 - e);
                cw[1] = cn >> (32 - e);
            }
        }
        __syncwarp();
        if (M == EDR && ahead) total = min(rb, nc);
        total += bits_total<M>(vp, vn, nr - rb);
        ahead = false;
    }
    return total;
}

// Output of a pair from its count (edr.py:51, lcss.py:52).
template <int M>
__device__ __forceinline__ float count_value(int count, int n1, int n2) {
    if (M == EDR) return __fdiv_rn((float)count, (float)max(n1, n2));
    return __fsub_rn(1.f, __fdiv_rn((float)count, (float)min(n1, n2)));
}

// Columns in shared memory.
struct BitsSmemCols {
    const float2* p;
    __device__ __forceinline__ float2 pt(int j) const { return p[j]; }
};

// Matrix kernel.  CTA (t, chunk) takes the queries q_order[QG t ..] (QG of
// them, staged in shared memory with their boxes) and blockDim database slots,
// one per thread (FEW, for launches of few pairs: one per warp), whose boxes it
// makes once for all QG queries.  The pairs whose boxes are apart are written at
// once; the others are collected and then taken 32 at a time, one per lane, or,
// when only a few are left over and always with FEW, one per warp.  Query order, symmetric and gather modes as in dp_matrix_kernel
// (gather: QG = 1).  Dynamic shared memory = QG * q_cap float2 + (blockDim /
// 32) * 32 * bits_words(q_cap) words.
constexpr int kBitsQueries = 16;
constexpr int kBitsThreads = 128;
constexpr int kBitsWarpRest = 16;  // a rest of fewer pairs than this goes one per warp
template <int M, bool FEW>
__global__ void __launch_bounds__(kBitsThreads) bits_matrix_kernel(
    const float2* __restrict__ q_pts, const int64_t* __restrict__ q_off, const int32_t* __restrict__ q_len,
    const int32_t* __restrict__ q_order, int64_t nq, const float2* __restrict__ d_pts,
    const int64_t* __restrict__ d_off, const int32_t* __restrict__ d_len, const int32_t* __restrict__ d_order,
    int64_t nd, int64_t d_total, int chunks, int QG, int sym, int q_cap, int d_max_len, KParams p,
    float* __restrict__ out, int64_t ld, int32_t* __restrict__ counts) {
    extern __shared__ __align__(16) float2 bits_smem[];
    __shared__ float4 q_box[kBitsQueries];
    __shared__ int q_n[kBitsQueries];  // -1: a bad length
    __shared__ int64_t q_id[kBitsQueries];
    __shared__ const float2* d_ptr[kBitsThreads];
    __shared__ int d_n[kBitsThreads];
    __shared__ int64_t d_id[kBitsThreads];
    __shared__ uint16_t todo[kBitsQueries * kBitsThreads];  // query * kBitsThreads + slot of the pairs to sweep
    __shared__ int n_todo, next;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t* carry = reinterpret_cast<uint32_t*>(bits_smem + QG * q_cap) + warp * 32 * bits_words(q_cap);
    const int64_t qs0 = (int64_t)(blockIdx.x / chunks) * QG;
    constexpr int kSlots = FEW ? kBitsThreads / 32 : kBitsThreads;
    const int64_t s0 = (int64_t)(blockIdx.x % chunks) * kSlots;
    if (sym == 1 && s0 + kSlots <= qs0) return;  // below the diagonal (uniform per CTA)
    const int ng = (int)min((int64_t)QG, nq - qs0);
    if (threadIdx.x == 0) n_todo = next = 0;
    for (int i = warp; i < ng; i += kBitsThreads / 32) {
        const int64_t qi = q_order ? (int64_t)q_order[qs0 + i] : qs0 + i;
        int n = q_len[qi];
        if (n < 0 || n > q_cap) n = -1;
        const float2* src = q_pts + q_off[qi];
        for (int j = lane; j < n; j += 32) bits_smem[i * q_cap + j] = __ldg(src + j);
        __syncwarp();
        const float4 b = warp_box(bits_smem + i * q_cap, n, lane);
        if (lane == 0) {
            q_box[i] = b;
            q_n[i] = n;
            q_id[i] = qi;
        }
    }
    __syncthreads();
    auto slot_of = [&](int x) { return s0 + (FEW ? x >> 5 : x); };
    const int64_t slot = FEW && lane > 0 ? nd : slot_of(threadIdx.x);  // (nd: none)
    int64_t dj = -1;
    int n = -1;
    const float2* dp = d_pts;
    if (slot < nd) {
        dj = d_order ? (int64_t)d_order[(sym == 2 ? q_id[0] * nd : 0) + slot] : slot;
        n = dj < 0 || dj >= d_total ? -1 : d_len[dj];
        if (n > d_max_len) n = -1;
        if (n > 0) dp += d_off[dj];
    }
    d_ptr[threadIdx.x] = dp;
    d_n[threadIdx.x] = n;
    d_id[threadIdx.x] = dj;
    auto put = [&](int64_t qi, int64_t dj, int64_t s, int m, int n, int c) {
        const float v = c < 0 ? CUDART_NAN_F : count_value<M>(c, m, n);
        const int64_t o = qi * ld + (sym == 2 ? s : dj);
        out[o] = v;
        if (counts) counts[o] = c;
        if (sym == 1 && dj != qi) {
            const int64_t t = dj * ld + qi;
            out[t] = v;
            if (counts) counts[t] = c;
        }
    };
    const float4 f = far_limits(lane_boxes(dp, n, lane), p.epsr);
    for (int i = 0; i < ng; ++i) {
        const int m = q_n[i];
        const bool mine = slot < nd && !(sym == 1 && slot < qs0 + i);
        const bool sweep = mine && n > 0 && m > 0 && !far_box(f, q_box[i]);
        const unsigned w = __ballot_sync(0xffffffffu, sweep);
        if (w) {
            int at = 0;
            if (lane == 0) at = atomicAdd(&n_todo, __popc(w));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(w & ((1u << lane) - 1u));
            if (sweep) todo[at] = (uint16_t)(i * kBitsThreads + threadIdx.x);
        }
        if (mine && !sweep) put(q_id[i], dj, slot, m, n, n < 0 || m < 0 ? -1 : M == EDR ? min(n, m) : 0);
    }
    __syncthreads();
    const int all = n_todo;
    const int full = FEW ? 0 : (all + 32 - kBitsWarpRest) / 32;  // tasks of up to 32 pairs; the rest one by one
    const int tasks = full + max(0, all - 32 * full);
    for (;;) {
        int t = 0;
        if (lane == 0) t = atomicAdd(&next, 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= tasks) break;
        if (!FEW && t < full) {
            const int k = 32 * t + lane;
            if (k < all) {
                const int i = todo[k] / kBitsThreads, x = todo[k] % kBitsThreads;
                const int c = bits_count<M>(d_ptr[x], d_n[x], BitsSmemCols{bits_smem + i * q_cap}, q_n[i], carry + lane,
                                            p.eps2, p.epsr, q_box[i]);
                put(q_id[i], d_id[x], slot_of(x), q_n[i], d_n[x], c);
            }
        } else {
            const int k = 32 * full + t - full;
            const int i = todo[k] / kBitsThreads, x = todo[k] % kBitsThreads;
            const int c = bits_count_warp<M>(d_ptr[x], d_n[x], bits_smem + i * q_cap, q_n[i], carry, p.eps2, p.epsr,
                                             q_box[i], lane);
            if (lane == 0) put(q_id[i], d_id[x], slot_of(x), q_n[i], d_n[x], c);
        }
        __syncwarp();
    }
}

}  // namespace tsm
