// Tile kernels: one thread per trajectory pair, register-blocked DP.
//
// A thread sweeps its pair's DP matrix in horizontal blocks of R rows.  The R
// row points and the R current DP values live in registers; the block walks
// the columns left to right, one column per step, computing R cells per step.
// The bottom row of a block (one value per column) goes to a per-thread
// boundary row in shared memory, laid out [column][lane] so a warp's 32
// accesses hit 32 banks; the next block reads it as its top border.  Only
// the row points, the column points and this one boundary row are touched per
// step, so a cell costs its arithmetic and ~3/R memory operations.
//
// Pairs mode: every thread has its own pair (rows = longer trajectory,
// columns = shorter, which keeps the boundary row short).  Matrix mode: a CTA
// owns one query trajectory Q_i, staged once in shared memory as the columns,
// and two threads (one for short queries) take one database trajectory D_j as
// its rows; database trajectories are visited in the caller's order (sorted by
// length, the lanes of a warp have near-equal row counts and the column loop is
// uniform).
//
// Reference kernels replaced: core/dtw.py:10-53, core/edr.py:10-52,
// core/lcss.py:12-53, core/erp.py:10-91, core/discret_frechet.py:9-50 (one
// CUDA block per pair, 64 threads, an FP64 3-diagonal ring in global memory
// and a __syncthreads per anti-diagonal), core/hausdorff.py:12-93.
#pragma once

#include "tsm_bits.cuh"
#include "tsm_device.cuh"

namespace tsm {

// Column accessors ----------------------------------------------------------

// Columns read from global memory (pairs mode): per-lane trajectories.
struct GlobalCols {
    const float2* __restrict__ p;
    __device__ __forceinline__ float2 pt(int j) const { return __ldg(p + j); }
};

// Columns staged in shared memory as float4 (x, y, gap distance, 0).
struct SmemCols {
    const float4* p;
    __device__ __forceinline__ float2 pt(int j) const {
        float4 v = p[j];
        return make_float2(v.x, v.y);
    }
    __device__ __forceinline__ float4 pt4(int j) const { return p[j]; }
};

// Gap distance of column j (ERP): staged value, or computed on the fly.
template <bool EXACT>
__device__ __forceinline__ float4 col4(const GlobalCols& c, int j, const KParams& p, bool gap) {
    float2 v = c.pt(j);
    return make_float4(v.x, v.y, gap ? gapdist<EXACT>(v.x, v.y, p) : 0.f, 0.f);
}
template <bool EXACT>
__device__ __forceinline__ float4 col4(const SmemCols& c, int j, const KParams&, bool) {
    return c.pt4(j);
}

// R consecutive rows of a pair's DP: their points (negated, for d2nr), their
// ERP gap distances and their current DP values, all in registers.
template <class C, int R, bool EXACT>
struct RowBlock {
    float2 n[R];
    float g[R], D[R];

    // rows i0 .. i0+R-1; rows past the end repeat the last point (their
    // values are never read by a valid cell)
    __device__ __forceinline__ void load(const float2* __restrict__ rowp, int i0, int nr, float srow,
                                         const KParams& p) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float2 q = __ldg(rowp + min(i0 + r, nr - 1));
            n[r] = make_float2(-q.x, -q.y);
            g[r] = C::kGap ? gapdist<EXACT>(q.x, q.y, p) : 0.f;
            D[r] = C::rowb(srow, i0 + r);
        }
    }

    // One column: top = D(i0-1, j), diag = D(i0-1, j-1); D[] holds column j-1
    // on entry and column j on exit.  Returns the block's bottom value.
    __device__ __forceinline__ float step(const float4& c, float top, float diag, float eps2) {
        float up = top, dg = diag;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float left = D[r];
            const float nv = C::cell(dg, up, left, d2nr(n[r], make_float2(c.x, c.y)), g[r], c.z, eps2);
            D[r] = nv;
            dg = left;
            up = nv;
        }
        return up;
    }

    // Same column step, reading the previous column from Din and writing the
    // new one to Dout: alternating two arrays between steps needs no register
    // copies (an in-place update costs one move per row).
    __device__ __forceinline__ float step2(const float (&Din)[R], float (&Dout)[R], const float4& c, float top,
                                           float diag, float eps2) const {
        float up = top, dg = diag;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float left = Din[r];
            const float nv = C::cell(dg, up, left, d2nr(n[r], make_float2(c.x, c.y)), g[r], c.z, eps2);
            Dout[r] = nv;
            dg = left;
            up = nv;
        }
        return up;
    }

    __device__ __forceinline__ float pick(int rr) const {
        float v = 0.f;
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (r == rr) v = D[r];
        return v;
    }
};

// The DP of one pair, prefetching form (dp_pair's default).  rowp/nr: row
// trajectory; cols/nc: column trajectory; buf: this thread's boundary row
// (element j at buf[32*j]); srow/scol: ERP gap totals of the row/column
// trajectory.  Returns D(nr-1, nc-1).
//
// Rows go in passes of 2R: an upper and a lower block of R rows, the lower
// one column behind the upper.  At step j the upper block computes column j
// from the boundary row, the lower block column j-1 from the upper block's
// bottom values of columns j-1 and j-2 (kept in registers), and writes its
// own bottom value of column j-1 to the boundary row.  The two blocks' cell
// chains are independent within a step (two chains for the scheduler), and
// only one boundary-row load and store are paid per 2R cells.  Each block's
// values alternate between two register arrays, two columns per loop trip,
// so no register copies are needed.  A final pass of at most R rows uses one
// block.  (Packing the two blocks into FP32x2 instructions was measured
// slower: assembling the pairs around the scalar min/max costs more than the
// packed arithmetic saves.  Packing only the squared distances, with the row
// points held as (upper, lower) pairs and one column pair per step, was
// measured too: all-pairs 2000 x 2000 DTW 15.25 -> 19.1 ms, Frechet 12.37 ->
// 17.6 ms, ERP 18.86 -> 23.96 ms on B200, bit-identical results.)
template <int M, int R, bool EXACT, class Cols>
__device__ __forceinline__ float dp_pair_prefetch(const float2* __restrict__ rowp, int nr, const Cols& cols,
                                                  int nc, float* buf, const KParams& p, float srow, float scol) {
    using C = typename CellOf<M, EXACT>::type;
    for (int j = 0; j < nc; ++j) buf[32 * j] = C::topb(scol, j);
    float dlast = 0.f;
    int rb = 0;
    for (; nr - rb > R; rb += 2 * R) {
        RowBlock<C, R, EXACT> hi, lo;
        hi.load(rowp, rb, nr, srow, p);
        lo.load(rowp, rb + R, nr, srow, p);
        float HA[R], HB[R], LA[R], LB[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            HA[r] = hi.D[r];
            LA[r] = lo.D[r];
        }
        float top = buf[0];
        float4 c = col4<EXACT>(cols, 0, p, C::kGap);
        const int j1 = min(1, nc - 1);
        float4 cn = col4<EXACT>(cols, j1, p, C::kGap);
        float tn = buf[32 * j1];
        // step 0: the upper block's column 0 (HA -> HB); the lower block waits in LA
        float ub1 = hi.step2(HA, HB, c, top, (rb == 0) ? C::corner() : C::rowb(srow, rb - 1), p.eps2);
        float ub2 = C::rowb(srow, rb + R - 1), udiag = top;
        float4 cprev = c;
        // steps 1 .. nc-1: upper column j, lower column j-1
        auto pair_step = [&](const float (&Hi)[R], float (&Ho)[R], const float (&Li)[R], float (&Lo)[R], int j) {
            c = cn;
            top = tn;
            const int jn = min(j + 1, nc - 1);  // prefetch the next column
            cn = col4<EXACT>(cols, jn, p, C::kGap);
            tn = buf[32 * jn];
            const float nb = hi.step2(Hi, Ho, c, top, udiag, p.eps2);
            const float lb = lo.step2(Li, Lo, cprev, ub1, ub2, p.eps2);
            buf[32 * (j - 1)] = lb;
            udiag = top;
            ub2 = ub1;
            ub1 = nb;
            cprev = c;
        };
        int j = 1;
        for (; j + 1 < nc; j += 2) {
            pair_step(HB, HA, LA, LB, j);
            pair_step(HA, HB, LB, LA, j + 1);
        }
        // the lower block's last column; the final arrays depend on nc's parity
        float lb;
        const int rr = nr - 1 - (rb + R);
        if (j < nc) {
            pair_step(HB, HA, LA, LB, j);
            lb = lo.step2(LB, LA, cprev, ub1, ub2, p.eps2);
            if (rb + 2 * R >= nr) {
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (r == rr) dlast = LA[r];
            }
        } else {
            lb = lo.step2(LA, LB, cprev, ub1, ub2, p.eps2);
            if (rb + 2 * R >= nr) {
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (r == rr) dlast = LB[r];
            }
        }
        buf[32 * (nc - 1)] = lb;
    }
    if (rb < nr) {  // last rows (at most R): one block
        RowBlock<C, R, EXACT> blk;
        blk.load(rowp, rb, nr, srow, p);
        float diag = (rb == 0) ? C::corner() : C::rowb(srow, rb - 1);
        float4 cn = col4<EXACT>(cols, 0, p, C::kGap);
        float tn = buf[0];
        for (int j = 0; j < nc; ++j) {
            const float4 c = cn;
            const float top = tn;
            const int jn = min(j + 1, nc - 1);
            cn = col4<EXACT>(cols, jn, p, C::kGap);
            tn = buf[32 * jn];
            blk.step(c, top, diag, p.eps2);
            diag = top;
        }
        dlast = blk.pick(nr - 1 - rb);
    }
    return dlast;
}

// The DP of one pair (DTW, ERP, discrete Frechet), one lane.
template <int M, int R, bool EXACT, class Cols>
__device__ __forceinline__ float dp_pair(const float2* __restrict__ rowp, int nr, const Cols& cols,
                                         int nc, float* buf, const KParams& p, float srow, float scol) {
    if (nr <= 0 || nc <= 0) return 0.f;
    return dp_pair_prefetch<M, R, EXACT>(rowp, nr, cols, nc, buf, p, srow, scol);
}

// The DP of a pair by two lanes (lanes 2 q and 2 q + 1 of a warp, all 32 lanes
// together; nc uniform, nr the pair's own), columns in shared memory.  Rows go
// in strips of 2 R, lane u = 0, 1 taking rows u R .. u R + R - 1 of a strip and
// column s - u at step s: lane 1's top values come from lane 0 by a shuffle, lane
// 0's from the boundary row, which lane 1 rewrites one column behind.  The
// boundary row is shared by two lanes (element j at ring[16 * j]), half the
// shared memory of a pair per lane, so 16 warps fit an SM where 8 did with a
// pair per lane: on a chain of cells alone 2 warps per scheduler take 11.1
// cycles a cell, 4 take 9.1, against the square root's 8 (its unit's rate).
// Strips are of 2 R rows while more than R are left to some pair of the warp,
// then of R (the sweep of rows that are not there is what long blocks cost).
//
// Measured on B200, all-pairs 2000 x 2000 of 20..200 points, ms, against one
// lane per pair (two, for ERP four, blocks of 8 rows a lane), same bits: DTW 15.2
// -> 13.9, ERP 18.1 -> 17.1, Frechet 12.3 -> 11.6; R = 4: 16.9, 19.7, 14.1.  The
// launch bound of 4 CTAs gives ptxas the registers that the shared memory allows
// (without it DTW 14.1, ERP 19.9; with 6 CTAs 16.6, 20.0, 12.6).  R = 16 has none
// (with 4 ERP spills): 1000 x 1000 DTW 3.81 ms, ERP 4.69, Frechet 3.14 (4.22, 5.71,
// 3.33 with it; one lane per pair 4.22, 5.23, 3.49).  Scalar instead of f32x2
// differences, 2 % faster for Frechet with one lane per pair: 3.39 for 3.17 with two.
// Tried on one
// lane per pair, slower, same bits: the square roots one column ahead of the
// recurrence (DTW 15.2 -> 16.0, ERP 18.1 -> 19.8), the lower block first (25 %),
// the squared distances of two rows packed in f32x2 (19.0, 20.5, Frechet 15.6:
// an f32x2 instruction holds the pipe and the issue port as long as two scalar
// ones).
// cols.p[-1] .. cols.p[nc + 1] and ring[0 .. 16 (nc + 1)] are loaded (the values
// past the ends are not used).  The cells are dp_pair_prefetch's.
__host__ __device__ constexpr int duo_ring(int cap) { return 16 * (cap + 2); }  // floats per warp

// One strip, rows rb .. rb + 2 R - 1.  Sets dlast to D(nr - 1, nc - 1) in the
// lane that holds row nr - 1, and mine there, if the strip has that row.
template <int M, int R, bool EXACT>
__device__ __forceinline__ void duo_strip(const float2* __restrict__ rowp, int nr, const SmemCols& cols, int nc,
                                          float* ring, const KParams& p, float srow, int u, int rb, float& dlast,
                                          bool& mine) {
    using C = typename CellOf<M, EXACT>::type;
    constexpr unsigned kFull = 0xffffffffu;
    const int row0 = rb + u * R;
    const int lr = nr - 1 - row0;  // the last row, if it is in this lane's block
    const bool last = lr >= 0 && lr < R;
    RowBlock<C, R, EXACT> blk;
    if (nr > 0) blk.load(rowp, row0, nr, srow, p);
    float A[R], B[R];
#pragma unroll
    for (int r = 0; r < R; ++r) A[r] = blk.D[r];
    const float diag0 = row0 == 0 ? C::corner() : C::rowb(srow, row0 - 1);
    float diag = diag0, bottom = 0.f;
    const float4* cp = cols.p - u;  // this lane's column of step 0
    float* rp = ring;
    float4 c = cp[0];
    float t = rp[0];
    // step s with cp and rp at step s - k: the next step's column and (for lane 0) top value are loaded first
    auto step = [&](const float (&Di)[R], float (&Do)[R], int k) {
        const float above = __shfl_up_sync(kFull, bottom, 1);
        const float top = u ? above : t;
        const float4 cc = c;
        c = cp[k + 1];
        t = rp[16 * (k + 1)];
        bottom = blk.step2(Di, Do, cc, top, diag, p.eps2);
        diag = top;
    };
    auto pick = [&](const float (&D)[R]) {
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (r == lr) dlast = D[r];
        mine = true;
    };
    step(A, B, 0);
    if (u) {  // lane 1 starts at step 1
        diag = diag0;
#pragma unroll
        for (int r = 0; r < R; ++r) B[r] = A[r];
    }
    int s = 1;
    for (; s + 1 < nc; s += 2, cp += 2, rp += 32) {
        step(B, A, 1);
        if (u) rp[0] = bottom;
        step(A, B, 2);
        if (u) rp[16] = bottom;
    }
    if (s < nc) {
        step(B, A, 1);
        if (u) rp[0] = bottom;
        if (last && u == 0) pick(A);
        step(A, B, 2);
        if (u) rp[16] = bottom;
        if (last && u == 1) pick(B);
    } else {
        if (last && u == 0) pick(B);
        step(B, A, 1);
        if (u) rp[0] = bottom;
        if (last && u == 1) pick(A);
    }
    __syncwarp();
}
template <int M, int R, bool EXACT>
__device__ __forceinline__ float dp_duo(const float2* __restrict__ rowp, int nr, const SmemCols& cols, int nc,
                                        float* ring, const KParams& p, float srow, float scol, int u, bool& mine) {
    using C = typename CellOf<M, EXACT>::type;
    float dlast = 0.f;
    mine = u == 0 && (nr <= 0 || nc <= 0);
    if (nc <= 0) return dlast;
    for (int j = u; j < nc; j += 2) ring[16 * j] = C::topb(scol, j);
    const int most = __reduce_max_sync(0xffffffffu, nr);
    __syncwarp();
    int rb = 0;
    for (; most - rb > (R > 4 ? R : 0); rb += 2 * R)
        duo_strip<M, R, EXACT>(rowp, nr, cols, nc, ring, p, srow, u, rb, dlast, mine);
    if constexpr (R > 4)
        if (rb < most) duo_strip<M, R / 2, EXACT>(rowp, nr, cols, nc, ring, p, srow, u, rb, dlast, mine);
    return dlast;
}

// The EDR or LCSS count of one pair per lane (na, nb < 0: none), the whole
// warp together; a count of 0 for an empty trajectory.
template <int M>
__device__ __forceinline__ int lane_count(const float2* a, int na, const float2* b, int nb, uint32_t* carry,
                                          const KParams& p, int lane) {
    const bool a_rows = na >= nb;
    const float2* rowp = a_rows ? a : b;
    const float2* colp = a_rows ? b : a;
    const int nr = a_rows ? na : nb, nc = a_rows ? nb : na;
    // the columns' boxes cost the warp about 1,400 instructions: for sweeps much longer than that (26 a word and
    // column) only.  200,000 pairs of 2..32 points without this line 0.062 ms, with it 0.043
    const int sweep = __reduce_max_sync(0xffffffffu, nc > 0 ? (nr + 31) / 32 * nc : 0);
    const float4 all = make_float4(-CUDART_INF_F, CUDART_INF_F, -CUDART_INF_F, CUDART_INF_F);
    const float4 cbox = sweep > 128 ? lane_boxes(colp, nc, lane) : all;
    return nc > 0 ? bits_count<M>(rowp, nr, GlobalCols{colp}, nc, carry, p.eps2, p.epsr, cbox) : 0;
}

// Pairs mode ------------------------------------------------------------------

// Block = 32*W threads, dynamic shared memory = W*32*cap floats (EDR, LCSS:
// W*32*bits_words(cap) words, tsm_bits.cuh).
template <int M, int R, bool EXACT>
__global__ void __launch_bounds__(128) dp_pairs_kernel(
    const float2* __restrict__ pts, const int64_t* __restrict__ off_a, const int32_t* __restrict__ len_a,
    const int64_t* __restrict__ off_b, const int32_t* __restrict__ len_b, const int32_t* __restrict__ order,
    int64_t n, int cap, int max_len, KParams p, float* __restrict__ out, int32_t* __restrict__ counts) {
    extern __shared__ float smem[];
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if constexpr (M == EDR || M == LCSS) {
        const int lane = threadIdx.x & 31;
        uint32_t* carry = reinterpret_cast<uint32_t*>(smem) + (threadIdx.x >> 5) * 32 * bits_words(cap) + lane;
        const int64_t k = t < n ? (order ? (int64_t)order[t] : t) : 0;
        int na = -1, nb = -1;
        bool bad = false;
        if (t < n) {
            na = len_a[k];
            nb = len_b[k];
            bad = na < 0 || nb < 0 || na > max_len || nb > max_len;
        }
        // (the wave kernel's pairs are left to it)
        const bool mine = t < n && !bad && min(na, nb) <= cap && !tile_heavy<R>(max(na, nb), min(na, nb));
        int c = lane_count<M>(mine ? pts + off_a[k] : pts, mine ? na : -1, mine ? pts + off_b[k] : pts, mine ? nb : -1,
                              carry, p, lane);
        if (bad) c = -1;
        if (!mine && !bad) return;
        out[k] = bad ? CUDART_NAN_F : count_value<M>(c, na, nb);
        if (counts) counts[k] = c;
        return;
    }
    float* buf = smem + (threadIdx.x >> 5) * (32 * cap) + (threadIdx.x & 31);
    if (t >= n) return;
    const int64_t k = order ? (int64_t)order[t] : t;
    const int na = len_a[k], nb = len_b[k];
    if (na < 0 || nb < 0 || na > max_len || nb > max_len) {
        out[k] = CUDART_NAN_F;
        return;
    }
    const float2* a = pts + off_a[k];
    const float2* b = pts + off_b[k];
    const bool a_rows = na >= nb;
    const float2* rowp = a_rows ? a : b;
    const float2* colp = a_rows ? b : a;
    const int nr = a_rows ? na : nb, nc = a_rows ? nb : na;
    if (nc > cap || tile_heavy<R>(nr, nc)) return;  // the wave kernel's pair
    float srow = 0.f, scol = 0.f;
    if constexpr (M == ERP) {
        srow = gapsum<EXACT>(rowp, nr, p);
        scol = gapsum<EXACT>(colp, nc, p);
    }
    const float dl = dp_pair<M, R, EXACT>(rowp, nr, GlobalCols{colp}, nc, buf, p, srow, scol);
    float o;
    int c;
    finalize<M>(dl, na, nb, o, c);
    out[k] = o;
}

// Matrix mode -----------------------------------------------------------------
// grid.x = nq * chunks; CTA (s, chunk) computes out[i, d_order[chunk * S + t]], t <
// S = blockDim / 2 (two lanes a slot; dp_matrix_lane_kernel: blockDim), for the
// query i = q_order[s] (i = s without an order).
// Symmetric mode (sym == 1; the query set is the database set and q_order ==
// d_order): only the slots at or after the query's own sorted position s are
// computed (the upper triangle in sorted order), and each value is written to
// out[i, j] and out[j, i]; CTAs wholly below the diagonal exit at once.
// Gather mode (sym == 2): d_order holds one row of nd database indices per
// query i (row i, whatever the processing order q_order), and slot t of query i
// goes to out[i, t].  A database index outside 0..d_total-1 gives NaN.
// (EDR and LCSS: bits_matrix_kernel, tsm_bits.cuh.)
// Dynamic shared memory = cap + 3 float4 columns + W * duo_ring(cap) floats.

template <int M, int R, bool EXACT>
__global__ void __launch_bounds__(128, R == 16 ? 1 : 4) dp_matrix_kernel(
    const float2* __restrict__ q_pts, const int64_t* __restrict__ q_off, const int32_t* __restrict__ q_len,
    const int32_t* __restrict__ q_order, const float2* __restrict__ d_pts, const int64_t* __restrict__ d_off,
    const int32_t* __restrict__ d_len, const int32_t* __restrict__ d_order, int64_t nd, int64_t d_total, int chunks,
    int sym, int cap, int d_max_len, KParams p, float* __restrict__ out, int64_t ld) {
    extern __shared__ float smem[];
    __shared__ float s_scol;
    float4* cols = reinterpret_cast<float4*>(smem) + 1;
    const int u = threadIdx.x & 1;
    float* ring = smem + 4 * (cap + 3) + (threadIdx.x >> 5) * duo_ring(cap) + ((threadIdx.x & 31) >> 1);
    const int64_t qs = blockIdx.x / chunks;
    const int chunk = blockIdx.x % chunks;
    const int per = blockDim.x >> 1;  // slots per CTA
    if (sym == 1 && (int64_t)(chunk + 1) * per <= qs) return;  // below the diagonal (uniform per CTA)
    const int64_t qi = q_order ? (int64_t)q_order[qs] : qs;
    const int nq = q_len[qi];
    const bool qbad = nq < 0 || nq > cap;
    if (!qbad) {
        const float2* qp = q_pts + q_off[qi];
        for (int j = threadIdx.x; j < nq; j += blockDim.x) {
            const float2 v = __ldg(qp + j);
            cols[j] = make_float4(v.x, v.y, M == ERP ? gapdist<EXACT>(v.x, v.y, p) : 0.f, 0.f);
        }
    }
    __syncthreads();
    if constexpr (M == ERP) {
        if (threadIdx.x == 0 && !qbad) {
            double s = 0.0;
            for (int j = 0; j < nq; ++j) s = __dadd_rn(s, (double)cols[j].z);
            s_scol = (float)s;
        }
        __syncthreads();
    }
    const int64_t slot = (int64_t)chunk * per + (threadIdx.x >> 1);
    const bool mine = slot < nd && !(sym == 1 && slot < qs);  // (the whole warp runs dp_duo)
    const int64_t dj = !mine ? -1 : d_order ? (int64_t)d_order[(sym == 2 ? qi * nd : 0) + slot] : slot;
    const bool dbad = dj < 0 || dj >= d_total;
    int ndl = dbad ? -1 : d_len[dj];
    const bool bad = qbad || ndl < 0 || ndl > d_max_len;
    if (bad) ndl = 0;
    const float2* dp = bad ? d_pts : d_pts + d_off[dj];
    float srow = 0.f, scol = 0.f;
    if constexpr (M == ERP) {
        srow = gapsum<EXACT>(dp, ndl, p);
        scol = s_scol;
    }
    bool last;  // this lane has the pair's result
    const float dl = dp_duo<M, R, EXACT>(dp, ndl, SmemCols{cols}, qbad ? 0 : nq, ring, p, srow, scol, u, last);
    if (!mine || !last) return;
    float o = CUDART_NAN_F;
    int c;
    if (!bad) finalize<M>(dl, nq, ndl, o, c);
    out[qi * ld + (sym == 2 ? slot : dj)] = o;
    if (sym == 1 && dj != qi) out[dj * ld + qi] = o;
}

// The same with one lane per pair, for short queries (DTW and discrete
// Frechet): a pair's fixed work is then paid in one lane, not two.  Dynamic
// shared memory = cap float4 columns + W*32*cap floats.
template <int M, int R, bool EXACT>
__global__ void __launch_bounds__(128) dp_matrix_lane_kernel(
    const float2* __restrict__ q_pts, const int64_t* __restrict__ q_off, const int32_t* __restrict__ q_len,
    const int32_t* __restrict__ q_order, const float2* __restrict__ d_pts, const int64_t* __restrict__ d_off,
    const int32_t* __restrict__ d_len, const int32_t* __restrict__ d_order, int64_t nd, int64_t d_total, int chunks,
    int sym, int cap, int d_max_len, KParams p, float* __restrict__ out, int64_t ld) {
    extern __shared__ float smem[];
    float4* cols = reinterpret_cast<float4*>(smem);
    float* buf = smem + 4 * cap + (threadIdx.x >> 5) * (32 * cap) + (threadIdx.x & 31);
    const int64_t qs = blockIdx.x / chunks;
    const int chunk = blockIdx.x % chunks;
    if (sym == 1 && (int64_t)(chunk + 1) * blockDim.x <= qs) return;  // below the diagonal (uniform per CTA)
    const int64_t qi = q_order ? (int64_t)q_order[qs] : qs;
    const int nq = q_len[qi];
    const bool qbad = nq < 0 || nq > cap;
    if (!qbad) {
        const float2* qp = q_pts + q_off[qi];
        for (int j = threadIdx.x; j < nq; j += blockDim.x) {
            const float2 v = __ldg(qp + j);
            cols[j] = make_float4(v.x, v.y, 0.f, 0.f);
        }
    }
    __syncthreads();
    const int64_t slot = (int64_t)chunk * blockDim.x + threadIdx.x;
    if (slot >= nd || (sym == 1 && slot < qs)) return;
    const int64_t dj = d_order ? (int64_t)d_order[(sym == 2 ? qi * nd : 0) + slot] : slot;
    const bool dbad = dj < 0 || dj >= d_total;
    const int ndl = dbad ? -1 : d_len[dj];
    const int64_t o_idx = qi * ld + (sym == 2 ? slot : dj), t_idx = dj * ld + qi;
    const bool mirror = sym == 1 && dj != qi;
    if (qbad || dbad || ndl < 0 || ndl > d_max_len) {
        out[o_idx] = CUDART_NAN_F;
        if (mirror) out[t_idx] = CUDART_NAN_F;
        return;
    }
    const float2* dp = d_pts + d_off[dj];
    const float dl = dp_pair<M, R, EXACT>(dp, ndl, SmemCols{cols}, nq, buf, p, 0.f, 0.f);
    float o;
    int c;
    finalize<M>(dl, nq, ndl, o, c);
    out[o_idx] = o;
    if (mirror) out[t_idx] = o;
}

// Hausdorff -------------------------------------------------------------------
// Point-to-segment squared distance (core/hausdorff.py:12-45), restated on
// relative vectors a = p - s1, s = s2 - s1 (no absolute foot point, which
// would cost the FP32 path ~1e-3 relative):
//   u = (a.s) * inv(|s|^2);  t = 0 if u < 1e-5, else min(u, 1);  |a - t s|^2.
// u < 1e-5 -> the reference takes min(|p-s1|^2, |p-s2|^2) = |p-s1|^2 (t = 0);
// u > 1 -> |p-s2|^2 (t = 1).  A zero-length segment has inv = 0, so t = 0 and
// the result is |p - s1|^2 as in hausdorff.py:30-31.  mul.sat clamps u to
// [0, 1] (NaN to 0) in the multiply itself.  This scalar form is the
// definition (and the oracle twin's formula); the kernels use p2s_pair.
__device__ __forceinline__ float p2s(float px, float py, float s1x, float s1y, float sx, float sy,
                                     float inv) {
    const float ax = __fsub_rn(px, s1x), ay = __fsub_rn(py, s1y);
    const float dot = __fmaf_rn(ay, sy, __fmul_rn(ax, sx));
    float u;
    asm("mul.rn.sat.f32 %0, %1, %2;" : "=f"(u) : "f"(dot), "f"(inv));
    const float t = (u < 1e-5f) ? 0.f : u;
    const float ex = __fmaf_rn(-t, sx, ax), ey = __fmaf_rn(-t, sy, ay);
    return __fmaf_rn(ey, ey, __fmul_rn(ex, ex));
}

// The kernels evaluate p2s two segments at a time in FP32x2: for a point p
// and consecutive segments k, k+1 of one trajectory, the vector quantities
// (a, dot, foot offset, squared distance) are f32x2 pairs, while the clamp
// u -> t and the running min stay scalar (f32x2 has no saturation and no
// min).  Segments are kept negated (-s1, -s, -1/|s|^2), so a - b becomes an
// f32x2 add and the foot a - t s an f32x2 fma: every value is bit-identical
// to p2s above, and min(best, d_k, d_k+1) is one three-input min.  Per two
// evaluations: 8 f32x2 + 2 scalar FMA-pipe and 5 ALU instructions, against
// 18 + 6 for two scalar p2s calls.
struct SegPair {
    float2 n1x, n1y;  // -s1 of segments k, k+1
    float2 nsx, nsy;  // -(s2 - s1)
    float2 ninv;      // -1/|s|^2 (0 for a zero-length segment)
};

// p2s of one point (pair-broadcast px2 = (px, px), py2) against segments
// k and k+1, folded into best.
__device__ __forceinline__ float p2s_pair(float2 px2, float2 py2, const SegPair& g, float best) {
    const float2 ax = __fadd2_rn(px2, g.n1x), ay = __fadd2_rn(py2, g.n1y);
    const float2 ndot = __ffma2_rn(ay, g.nsy, __fmul2_rn(ax, g.nsx));  // -(a.s)
    float u0, u1;
    asm("mul.rn.sat.f32 %0, %1, %2;" : "=f"(u0) : "f"(ndot.x), "f"(g.ninv.x));
    asm("mul.rn.sat.f32 %0, %1, %2;" : "=f"(u1) : "f"(ndot.y), "f"(g.ninv.y));
    const float2 t = make_float2((u0 < 1e-5f) ? 0.f : u0, (u1 < 1e-5f) ? 0.f : u1);
    const float2 ex = __ffma2_rn(t, g.nsx, ax), ey = __ffma2_rn(t, g.nsy, ay);
    const float2 d2 = __ffma2_rn(ey, ey, __fmul2_rn(ex, ex));
    return min3f(best, d2.x, d2.y);
}

// Segment k of trajectory T (k = n-1: the last vertex as a zero-length
// segment), negated, into lane `hi` of a SegPair.
template <bool EXACT>
__device__ __forceinline__ void seg_lane(SegPair& g, int hi, float2 s1, float2 s2) {
    const float sx = __fsub_rn(s2.x, s1.x), sy = __fsub_rn(s2.y, s1.y);
    const float len2 = __fmaf_rn(sy, sy, __fmul_rn(sx, sx));
    const float inv = (sx == 0.f && sy == 0.f) ? 0.f : trcp<EXACT>(len2);
    if (hi) {
        g.n1x.y = -s1.x; g.n1y.y = -s1.y; g.nsx.y = -sx; g.nsy.y = -sy; g.ninv.y = -inv;
    } else {
        g.n1x.x = -s1.x; g.n1y.x = -s1.y; g.nsx.x = -sx; g.nsy.x = -sy; g.ninv.x = -inv;
    }
}

// Staged query segments for the packed matrix kernel: pair j holds segments
// 2j and 2j+1 of the query (the last vertex counted as segment nq-1; an odd
// count repeats it), as float4 (n1x, n1y) + float4 (nsx, nsy) + float2 ninv.
__device__ __forceinline__ SegPair staged_pair(const float4* A, const float4* B, const float2* C, int j) {
    const float4 a = A[j], b = B[j];
    SegPair g;
    g.n1x = make_float2(a.x, a.y);
    g.n1y = make_float2(a.z, a.w);
    g.nsx = make_float2(b.x, b.y);
    g.nsy = make_float2(b.z, b.w);
    g.ninv = C[j];
    return g;
}

// directed_max with P from global memory and T staged as segment pairs.
template <int R>
__device__ __forceinline__ float directed_max_staged2(const float2* __restrict__ P, int np, const float4* A,
                                                      const float4* B, const float2* C, int nq) {
    if (nq < 2 || np <= 0) return 0.f;
    const int npair = (nq + 1) >> 1;
    float m = 0.f;
    for (int pb = 0; pb < np; pb += R) {
        float2 px[R], py[R];
        float best[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float2 q = __ldg(P + min(pb + r, np - 1));
            px[r] = make_float2(q.x, q.x);
            py[r] = make_float2(q.y, q.y);
            best[r] = CUDART_INF_F;
        }
        for (int j = 0; j < npair; ++j) {
            const SegPair g = staged_pair(A, B, C, j);
#pragma unroll
            for (int r = 0; r < R; ++r) best[r] = p2s_pair(px[r], py[r], g, best[r]);
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (pb + r < np) m = fmaxf(m, best[r]);
    }
    return m;
}

// max over the points of P of (min over the segments of T), hausdorff.py:48-69
// per point, then the max of the host reduction at :121 over valid points.
// T's segment pairs are built on the fly from global memory.  The loop also
// visits T's last vertex as a zero-length segment: in exact arithmetic that
// distance is never below the last segment's, so the min is the reference's;
// in FP32 it makes a point that coincides with the last vertex come out
// exactly 0 (u = dot * (1/len2) can round to 1-ulp, leaving a ~1e-11
// residue), as every other vertex already does as the first endpoint of its
// outgoing segment.  Points pb0, pb0 + pstride, ... (blocks of R) of P: a
// thread takes all points (pb0 = 0, pstride = R) or, in a warp-per-pair
// task, every 32nd block.
template <int R, bool EXACT, class Pts>
__device__ __forceinline__ float directed_max2(const Pts& P, int np, const float2* __restrict__ T, int nt,
                                               int pb0 = 0, int pstride = R) {
    if (nt < 2 || np <= 0) return 0.f;  // p2t_dist over zero segments is 0.0
    float m = 0.f;
    for (int pb = pb0; pb < np; pb += pstride) {
        float2 px[R], py[R];
        float best[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float2 q = P.pt(min(pb + r, np - 1));
            px[r] = make_float2(q.x, q.x);
            py[r] = make_float2(q.y, q.y);
            best[r] = CUDART_INF_F;
        }
        float2 v0 = __ldg(T);
        float2 v1 = __ldg(T + 1);
        for (int k = 0; k < nt; k += 2) {  // segments k, k+1 (segment nt-1 is the last vertex)
            const float2 v2 = __ldg(T + min(k + 2, nt - 1));
            SegPair g;
            seg_lane<EXACT>(g, 0, v0, v1);
            if (k + 1 < nt) seg_lane<EXACT>(g, 1, v1, v2);
            else seg_lane<EXACT>(g, 1, v0, v0);  // odd count: repeat the last vertex
#pragma unroll
            for (int r = 0; r < R; ++r) best[r] = p2s_pair(px[r], py[r], g, best[r]);
            v0 = v2;
            v1 = __ldg(T + min(k + 3, nt - 1));
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (pb + r < np) m = fmaxf(m, best[r]);
    }
    return m;
}

// The staged query's points, read back from the negated segment starts.
struct StagedNegPts {
    const float4* A;
    __device__ __forceinline__ float2 pt(int k) const {
        const float4 a = A[k >> 1];
        return make_float2(-((k & 1) ? a.y : a.x), -((k & 1) ? a.w : a.z));
    }
};

// Matrix kernel: CTA (s, chunk) stages query i's segment pairs in shared
// memory once; each thread takes one database trajectory.  Query order,
// symmetric and gather modes as in dp_matrix_kernel.  Dynamic shared memory =
// ceil(q_max_len/2) * 40 bytes.
template <int R, bool EXACT>
__global__ void __launch_bounds__(128) hausdorff_matrix_kernel(
    const float2* __restrict__ q_pts, const int64_t* __restrict__ q_off, const int32_t* __restrict__ q_len,
    const int32_t* __restrict__ q_order, const float2* __restrict__ d_pts, const int64_t* __restrict__ d_off,
    const int32_t* __restrict__ d_len, const int32_t* __restrict__ d_order, int64_t nd, int64_t d_total, int chunks,
    int sym, int q_max_len, int d_max_len, float* __restrict__ out, int64_t ld) {
    extern __shared__ float4 smem4[];
    const int cap_pairs = (q_max_len + 1) >> 1;
    float4* A = smem4;
    float4* B = smem4 + cap_pairs;
    float2* C = reinterpret_cast<float2*>(smem4 + 2 * cap_pairs);
    const int64_t qs = blockIdx.x / chunks;
    const int chunk = blockIdx.x % chunks;
    if (sym == 1 && (int64_t)(chunk + 1) * blockDim.x <= qs) return;
    const int64_t qi = q_order ? (int64_t)q_order[qs] : qs;
    const int nq = q_len[qi];
    const bool qbad = nq < 0 || nq > q_max_len;
    if (!qbad && nq > 0) {
        const float2* qp = q_pts + q_off[qi];
        const int npair = (nq + 1) >> 1;
        for (int j = threadIdx.x; j < npair; j += blockDim.x) {
            SegPair g;
            const int k0 = 2 * j, k1 = min(2 * j + 1, nq - 1);
            seg_lane<EXACT>(g, 0, __ldg(qp + k0), __ldg(qp + min(k0 + 1, nq - 1)));
            seg_lane<EXACT>(g, 1, __ldg(qp + k1), __ldg(qp + min(k1 + 1, nq - 1)));
            A[j] = make_float4(g.n1x.x, g.n1x.y, g.n1y.x, g.n1y.y);
            B[j] = make_float4(g.nsx.x, g.nsx.y, g.nsy.x, g.nsy.y);
            C[j] = g.ninv;
        }
    }
    __syncthreads();
    const int64_t slot = (int64_t)chunk * blockDim.x + threadIdx.x;
    if (slot >= nd || (sym == 1 && slot < qs)) return;
    const int64_t dj = d_order ? (int64_t)d_order[(sym == 2 ? qi * nd : 0) + slot] : slot;
    const bool dbad = dj < 0 || dj >= d_total;
    const int ndl = dbad ? -1 : d_len[dj];
    const int64_t o_idx = qi * ld + (sym == 2 ? slot : dj);
    const bool mirror = sym == 1 && dj != qi;
    float v = CUDART_NAN_F;
    if (!(qbad || dbad || ndl < 0 || ndl > d_max_len)) {
        const float2* dp = d_pts + d_off[dj];
        const float m1 = directed_max_staged2<R>(dp, ndl, A, B, C, nq);
        const float m2 = directed_max2<R, EXACT>(StagedNegPts{A}, nq, dp, ndl);
        v = __fsqrt_rn(fmaxf(m1, m2));
    }
    out[o_idx] = v;
    if (mirror) out[dj * ld + qi] = v;
}

// Pairs mode: a pair with more than kHausWarpCells point products (na * nb)
// runs one warp or one CTA per pair (hausdorff_pruned_pairs_kernel, or above
// kHausPrunedMax points hausdorff_wave_kernel): below that line one thread
// per pair costs less than staging a pair (see matrix_launch for both sides).
constexpr int64_t kHausWarpCells = 2048;

// Pairs kernel: one thread per pair, both trajectories from global memory
// (the pairs up to warp_cells point products -- kHausWarpCells, or 0 when a
// small batch runs every non-empty pair on the warp kernels; it also flags
// bad lengths).
template <int R, bool EXACT>
__global__ void __launch_bounds__(128) hausdorff_pairs_kernel(
    const float2* __restrict__ pts, const int64_t* __restrict__ off_a, const int32_t* __restrict__ len_a,
    const int64_t* __restrict__ off_b, const int32_t* __restrict__ len_b, const int32_t* __restrict__ order,
    int64_t n, int max_len, int64_t warp_cells, float* __restrict__ out) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int64_t k = order ? (int64_t)order[t] : t;
    const int na = len_a[k], nb = len_b[k];
    if (na < 0 || nb < 0 || na > max_len || nb > max_len) {
        out[k] = CUDART_NAN_F;
        return;
    }
    if ((int64_t)na * nb > warp_cells) return;  // the warp kernel's pair
    const float2* a = pts + off_a[k];
    const float2* b = pts + off_b[k];
    const float m1 = directed_max2<R, EXACT>(GlobalCols{a}, na, b, nb);
    const float m2 = directed_max2<R, EXACT>(GlobalCols{b}, nb, a, na);
    out[k] = __fsqrt_rn(fmaxf(m1, m2));
}

// Long pairs (more than warp_cells point products and a side of more than
// min_side points), one warp each.  Persistent, with the pair assignment of dp_wave_kernel (rounds of nw
// pairs in snake order, a ballot over 32 pairs at a time).  Lane l takes
// point blocks l, l+32, ... of both directions; the lanes' maxima are
// reduced with one warp max (exact), so the result is the one-thread
// kernel's, bit for bit.
template <int R, bool EXACT>
__global__ void __launch_bounds__(128) hausdorff_wave_kernel(
    const float2* __restrict__ pts, const int64_t* __restrict__ off_a, const int32_t* __restrict__ len_a,
    const int64_t* __restrict__ off_b, const int32_t* __restrict__ len_b, const int32_t* __restrict__ order,
    int64_t n, int max_len, int min_side, int64_t warp_cells, float* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const int64_t gw = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t i0 = 0; i0 * nw < n; i0 += 32) {
        const int64_t i = i0 + lane;
        const int64_t t = i * nw + ((i & 1) ? nw - 1 - gw : gw);
        int64_t k = 0;
        bool mine = false;
        if (t < n) {
            k = order ? (int64_t)order[t] : t;
            const int na = len_a[k], nb = len_b[k];
            mine = na >= 0 && nb >= 0 && na <= max_len && nb <= max_len && max(na, nb) > min_side &&
                   (int64_t)na * nb > warp_cells;
        }
        unsigned todo = __ballot_sync(0xffffffffu, mine);
        while (todo) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1;
            const int64_t kk = __shfl_sync(0xffffffffu, k, src);
            const int na = len_a[kk], nb = len_b[kk];
            const float2* a = pts + off_a[kk];
            const float2* b = pts + off_b[kk];
            float m = fmaxf(directed_max2<R, EXACT>(GlobalCols{a}, na, b, nb, lane * R, 32 * R),
                            directed_max2<R, EXACT>(GlobalCols{b}, nb, a, na, lane * R, 32 * R));
            // non-negative floats order like their bit patterns
            m = __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(m)));
            if (lane == 0) out[kk] = __fsqrt_rn(m);
        }
    }
}

}  // namespace tsm
