// Training recurrences of the encoder on the tensor cores (tcgen05): the GRU
// over time with the values BPTT needs, BPTT itself, and the gradients of the
// conv layer.
//
// Each time step's products are W [gates x features] times the features of 16
// trajectories: the weights are the MMA's A operand (M = 128 gate rows, BF16,
// resident in tensor memory for all steps) and the trajectories its N.  The
// activations are FP32: x = hi + mid + lo, three BF16 parts that hold all 24
// bits, stand side by side as N = 3 x 16 columns, and the epilogue adds the
// three FP32 results.  Products of BF16 values are exact in FP32, so a sum
// differs from an FP32 one only in how it is accumulated.
//
// Threads: 512 of the epilogue, thread (k, q) with k = hidden unit
// (tensor-memory lane) and q = 4 of the block's 16 trajectories, whose h (dh)
// it keeps in registers, and a seventeenth warp that issues copies and MMAs.  An
// operand stands in shared memory as [part][half][k][8 trajectories] (MN-major,
// N group stride 16 K bytes), so each part is also the operand image of the
// weight gradients, whose K runs over (slot, trajectory): the issuing warp
// stores it with one bulk copy and the epilogue never touches it.
//
// Blocks take trajectories of similar length (a counting sort by length), so
// few of a block's 16 rows idle, and time steps are stored compactly.
//
// What bounds it: the chain of steps.  A forward step (1.75 us) is 24 MMAs (M =
// 128, N = 48, K = 16, about 40 cycles each) on the previous step's result, a
// commit, the tensor-memory loads (370 cycles), the gate math (1,300) and the
// operand stores (110); the input products of the next step run under the gate
// math.  A backward step (1.7 us) has 24 MMAs on the chain and 24 (dA) beside it.
// 48 KB leave and 40 KB enter the SM a step, all by bulk copies off the chain.
// Measured, 1,024 pairs of 20..200 points (128 blocks): forward 350 us, backward
// 350 us.  With the weights in shared memory (64 cycles an MMA: bound by reading
// A; 128 for the 64-row dA), eight values a thread and every value stored and
// loaded by the epilogue: about 560 us each.
#include <cstdio>

#include "tsm.h"
#include "tsm_enc.cuh"
#include "tsm_train.h"
#include "tsm_umma.cuh"
#include "tsm_wgrad.h"

int tsm_internal_fail(int code, const char* msg);

namespace enc {

namespace U = tsm::umma;

constexpr int NN = 3 * TB;             // MMA N: three parts of 16 trajectories
constexpr int A_PARTB = C1 * TB * 2;   // bytes of one part of the operands: 2,048
constexpr int H_PARTB = HD * TB * 2;   // 4,096
constexpr int A_OP = 3 * A_PARTB;      // 6,144
constexpr int H_OP = 3 * H_PARTB;      // 12,288
constexpr int EPI = 512;               // epilogue threads
constexpr int THREADS = EPI + 32;      // + the issuing warp
constexpr int NBUF = 3;                // a-operand buffers of the forward
constexpr int C_OP = 5 * HD * TB * 4;  // what BPTT reads of a step: 40,960
constexpr long long WAIT_CYCLES = 2000000000LL;  // ~1 s of SM clocks
// status bits
constexpr int ERR_FWD_COPY = 256, ERR_FWD_MMA = 512, ERR_BWD_MMA = 1024, ERR_HELD = 128;

// Descriptor of an operand of `rows` K rows; a K step of 16 is 256 bytes on.
__device__ __forceinline__ uint64_t op_desc(uint32_t saddr, int rows) { return U::smem_desc(saddr, 128, rows * 16); }

// 1 / (1 + e^-x).  The quotient by the hardware's approximate reciprocal y and one
// Newton step y + y (1 - d y), on a quarter of the denominator so that y stays
// normal (0 for an infinite one): the same bits as 1.f / (1.f + expf(-x)) for
// 2^24 values of x from -87 to 30, the last bit of some subnormal results below.
// A step of 1,024 pairs takes 1.213 ms with the division, 1.168 with this.  (The approximate power of -log2(e) x would save 25 us
// more, but the rounding of the product makes a relative error of 2^-24 |x|: 3e-6
// of a gate closed at x = -70, and of its gradient.)
__device__ __forceinline__ float sigm(float x) {
    const float d = 0.25f * (1.f + expf(-x));
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d));
    return 0.25f * (y > 0.f ? fmaf(y, fmaf(-d, y, 1.f), y) : y);
}

// Two values as three BF16 parts each, x = hi + mid + lo.
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float lo_of(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float hi_of(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }
__device__ __forceinline__ void split2(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
    h = pack2(a, b);
    const float a1 = a - lo_of(h), b1 = b - hi_of(h);
    m = pack2(a1, b1);
    l = pack2(a1 - lo_of(m), b1 - hi_of(m));
}
// The three parts of this thread's four trajectories.
struct Split {
    uint2 part[3];
    __device__ __forceinline__ explicit Split(const float (&v)[4]) {
        split2(v[0], v[1], part[0].x, part[1].x, part[2].x);
        split2(v[2], v[3], part[0].y, part[1].y, part[2].y);
    }
    // to K row k of an operand of HD rows
    __device__ __forceinline__ void put(unsigned char* op, int k, int q) const {
        unsigned char* d = op + (q >> 1) * (HD * 16) + k * 16 + (q & 1) * 8;
#pragma unroll
        for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(d + i * H_PARTB) = part[i];
    }
};
// This thread's zeros in the image [group][HD][8] of one slot.
__device__ __forceinline__ void zero_img(unsigned char* img, int64_t slot, int k, int q) {
    *reinterpret_cast<uint2*>(img + (((2 * slot + (q >> 1)) * HD + k) << 4) + (q & 1) * 8) = make_uint2(0, 0);
}

// The sum of the three parts' results, 4 columns from `col` (this thread's
// lane and trajectories; parts 16 columns apart).
struct Parts {
    uint32_t r[3][4];
    __device__ __forceinline__ void load(uint32_t taddr) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 3; ++i) U::ld4(taddr + 16 * i, r[i]);
    }
    __device__ __forceinline__ void wait() {
#pragma unroll
        for (int i = 0; i < 3; ++i) U::wait_ld4(r[i]);
    }
    __device__ __forceinline__ float sum(int s) const {
        return __uint_as_float(r[0][s]) + (__uint_as_float(r[1][s]) + __uint_as_float(r[2][s]));
    }
};

// Sorts the batch by length, longest first (counting sort over up to 1,024
// length classes; within a class any order), cuts it into blocks and assigns
// the slots.  One CTA of 1,024 threads.
__global__ void __launch_bounds__(1024) train_plan(const int32_t* __restrict__ len, int B, int T, int blocks,
                                                    int32_t* __restrict__ perm, int32_t* __restrict__ slot0) {
    __shared__ int hist[1024];
    __shared__ int tot[32];
    __shared__ int carry;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto n_of = [&](int b) { return min(max(len[b], 0), T); };
    auto cls = [&](int n) { return 1023 - (int)((int64_t)n * 1023 / T); };  // class 0: the longest
    auto scan = [&](int v) {  // exclusive sum over the CTA
        int x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) tot[warp] = x;
        __syncthreads();
        if (warp == 0) {
            int w = tot[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += y;
            }
            tot[lane] = w;
        }
        __syncthreads();
        return x - v + (warp ? tot[warp - 1] : 0);
    };
    hist[tid] = 0;
    __syncthreads();
    for (int b = tid; b < B; b += 1024) atomicAdd(&hist[cls(n_of(b))], 1);
    __syncthreads();
    const int first = scan(hist[tid]);
    __syncthreads();
    hist[tid] = first;
    if (tid == 0) carry = 0;
    __syncthreads();
    for (int b = tid; b < B; b += 1024) perm[atomicAdd(&hist[cls(n_of(b))], 1)] = b;
    for (int r = B + tid; r < blocks * TB; r += 1024) perm[r] = -1;
    __syncthreads();
    for (int k0 = 0; k0 < blocks; k0 += 1024) {
        const int k = k0 + tid;
        int n = 0;
        if (k < blocks)
            for (int s = 0; s < TB; ++s) {
                const int b = perm[k * TB + s];
                if (b >= 0) n = max(n, n_of(b));
            }
        const int slots = (n + 1) & ~1;
        const int before = scan(slots) + carry;
        if (k < blocks) slot0[k] = before;
        __syncthreads();
        if (tid == 1023) carry = before + slots;
        __syncthreads();
    }
    if (tid == 0) slot0[blocks] = carry;
}

// conv + relu of every slot: the operand of the recurrence and of the weight
// gradient, and the relu's sign bits.  CTA = (block, 16 slots); thread (half, c).
// Steps at or past a trajectory's length are zero.
constexpr int CV_T = 16;
__global__ void __launch_bounds__(128) train_conv(const float2* __restrict__ pts, const int64_t* __restrict__ off,
                                                  const int32_t* __restrict__ len, int T, float4 nrm,
                                                  const __nv_bfloat16* __restrict__ wq, const float* __restrict__ p,
                                                  TrainWs w) {
    __shared__ float xs[CV_T + KW - 1][2][TB];  // xs[u][i][s]: input i of trajectory s at step t0 + u - 2
    __shared__ int n_s[TB];
    const int blk = blockIdx.x, t0 = blockIdx.y * CV_T;
    const int u0 = w.slot0[blk], nt = w.slot0[blk + 1] - u0;
    if (t0 >= nt) return;
    for (int e = threadIdx.x; e < (CV_T + KW - 1) * 2 * TB; e += 128) {
        const int s = e % TB, i = (e / TB) % 2, u = e / (2 * TB);
        const int b = w.perm[blk * TB + s];
        xs[u][i][s] = b >= 0 ? xin(pts, off[b], len[b], t0 + u - 2, i, nrm) : 0.f;
        if (u == 0 && i == 0) n_s[s] = b >= 0 ? min(len[b], T) : 0;
    }
    __syncthreads();
    const int c = threadIdx.x % C1, half = threadIdx.x / C1;
    float w1[KW][2];
#pragma unroll
    for (int k = 0; k < KW; ++k)
#pragma unroll
        for (int i = 0; i < 2; ++i) w1[k][i] = __bfloat162float(wq[OFF_W1 + (c * 2 + i) * KW + k]);
    const float b1 = p[OFF_B1 + c];
    for (int t = t0; t < min(t0 + CV_T, nt); ++t) {
        float a[8];
        uint32_t on = 0;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int s = 8 * half + e;
            float acc = b1;
#pragma unroll
            for (int k = 0; k < KW; ++k)
#pragma unroll
                for (int i = 0; i < 2; ++i) acc = fmaf(w1[k][i], xs[t - t0 + k][i][s], acc);
            a[e] = t < n_s[s] ? fmaxf(acc, 0.f) : 0.f;
            on |= (a[e] > 0.f ? 1u : 0u) << e;
        }
        uint32_t part[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) split2(a[2 * e], a[2 * e + 1], part[0][e], part[1][e], part[2][e]);
        const int64_t u = u0 + t, g = 2 * u + half;
#pragma unroll
        for (int i = 0; i < 3; ++i)
            *reinterpret_cast<uint4*>(w.a_op + u * A_OP + i * A_PARTB + (half * C1 + c) * 16) =
                make_uint4(part[i][0], part[i][1], part[i][2], part[i][3]);
        w.a_on[g * C1 + c] = (unsigned char)on;
    }
}

// Shared memory of the forward: h (two buffers), a (NBUF buffers), what BPTT
// reads (three buffers), barriers.  (More than half an SM's: a block needs all
// of tensor memory.)
constexpr int F_H = 0, F_A = F_H + 2 * H_OP, F_C = F_A + NBUF * A_OP, F_BAR = F_C + 3 * C_OP, F_SMEM = F_BAR + 128;
static_assert(F_SMEM + 1024 <= 227 * 1024, "train_gru_fwd shared memory");
// Tensor memory: Whh (3 gates, K = 128), Wih (3 gates, K = 64), accumulators r, z, n (hidden), n (input)
constexpr uint32_t COLS = 512;
constexpr uint32_t F_WHH = 0, F_WIH = F_WHH + 3 * HD / 2, F_ACC = F_WIH + 3 * C1 / 2;
static_assert(F_ACC + 4 * NN <= COLS, "train_gru_fwd tensor memory");

__global__ void __launch_bounds__(THREADS, 1) train_gru_fwd(const int32_t* __restrict__ len, int T,
                                                            const __nv_bfloat16* __restrict__ wq,
                                                            const float* __restrict__ p, TrainWs w,
                                                            float* __restrict__ hl, int* __restrict__ status,
                                                            long long wait_cycles) {
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ int n_s[TB], b_s[TB], busy;
    const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(sm));
    // mbarriers: a step's products done, loaded, its h written, a-buffer i landed, the last products done, the last values written
    const uint32_t hbar = sbase + F_BAR, lbar = hbar + 8, rbar = hbar + 16, abar = hbar + 24, last = abar + 8 * NBUF, fin = last + 8;
    constexpr int SLOT = F_BAR + 24 + 8 * NBUF + 16;
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(sm + SLOT);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int k = 32 * (warp & 3) + lane, q = warp >> 2;
    const int blk = blockIdx.x;
    const int64_t u0 = w.slot0[blk];
    const int nt = w.slot0[blk + 1] - (int)u0;

    for (int e = tid; e < H_OP / 16; e += THREADS) *reinterpret_cast<uint4*>(sm + F_H + 16 * e) = make_uint4(0, 0, 0, 0);
    if (tid < TB) {
        const int b = w.perm[blk * TB + tid];
        b_s[tid] = b;
        n_s[tid] = b >= 0 ? min(max(len[b], 0), T) : 0;
    }
    if (tid == 0) {
        U::mbar_init(hbar, 1);
        U::mbar_init(lbar, EPI / 32);
        U::mbar_init(rbar, EPI / 32);
        U::mbar_init(fin, EPI / 32);
        for (int i = 0; i < NBUF; ++i) U::mbar_init(abar + 8 * i, 1);
        U::mbar_init(last, 1);
        busy = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) U::tmem_alloc(sbase + SLOT, COLS);
    U::fence_smem_async();
    U::fence_before_sync();
    __syncthreads();
    U::fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    if (warp < EPI / 32) {  // the weights: lane = row of a gate, 16 K a write
        const uint32_t tw = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
        constexpr int NH = 3 * HD / 16, NI = 3 * C1 / 16;
        for (int i = q; i < NH + NI; i += 4) {
            const int j = i - NH;
            const __nv_bfloat16* src = i < NH ? wq + OFF_WHH + (i / (HD / 16) * HD + k) * HD + i % (HD / 16) * 16
                                              : wq + OFF_WIH + (j / (C1 / 16) * HD + k) * C1 + j % (C1 / 16) * 16;
            const uint4 x = *reinterpret_cast<const uint4*>(src), y = *reinterpret_cast<const uint4*>(src + 8);
            const uint32_t r[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
            __syncwarp();
            U::st8(tw + F_WHH + 8 * i, r);  // (Wih's columns follow Whh's)
        }
        U::wait_st();
    }
    U::fence_before_sync();
    __syncthreads();
    U::fence_after_sync();
    int tmax = 0;
    for (int s = 0; s < TB; ++s) tmax = max(tmax, n_s[s]);

    if (warp == EPI / 32) {  // copies and MMAs
        if (tmax > 0) {  // the whole warp runs this, its leader issues
            constexpr uint32_t id = U::idesc_bf16_f32_bmn(HD, NN);
            const uint32_t leader = U::elect_leader();
            const uint32_t acc = tmem + F_ACC;
            int loaded = 0;
            auto load_a = [&](int t) {
                const uint32_t bar = abar + 8 * (t % NBUF);
                if (leader) {
                    U::mbar_arrive_expect_tx(bar, A_OP);
                    U::bulk_load(sbase + F_A + (t % NBUF) * A_OP, w.a_op + (u0 + t) * A_OP, A_OP, bar);
                }
                __syncwarp();
                loaded = t + 1;
            };
            auto waited = [&](uint32_t bar, int parity) {
                return (bool)__all_sync(0xffffffffu, U::mbar_wait(bar, (uint32_t)(parity & 1), wait_cycles));
            };
            auto a_landed = [&](int t) { return waited(abar + 8 * (t % NBUF), t / NBUF); };
            auto store_c = [&](int t) {
                U::bulk_store(reinterpret_cast<unsigned char*>(w.cache) + (u0 + t) * C_OP, sbase + F_C + t % 3 * C_OP, C_OP);
            };
            // the input products of step t
            auto input_mmas = [&](int t) {
                const uint64_t a = op_desc(sbase + F_A + (t % NBUF) * A_OP, C1);
#pragma unroll
                for (int ks = 0; ks < C1 / 16; ++ks)
#pragma unroll
                    for (int g = 0; g < 3; ++g)
                        U::mma_bf16_warp_ta(acc + (g == 2 ? 3 : g) * NN, tmem + F_WIH + g * (C1 / 2) + ks * 8, a + ks * 16,
                                            id, ks, leader);
            };
            for (int t = 0; t < min(NBUF - 1, tmax); ++t) load_a(t);
            int err = a_landed(0) ? 0 : ERR_FWD_COPY;
            U::fence_after_sync();
            if (!err) input_mmas(0);
            for (int t = 0; t < tmax && !err; ++t) {
                if (t > 0 && !waited(rbar, t - 1)) {
                    err = ERR_FWD_MMA;
                    break;
                }
                U::fence_smem_async();
                U::fence_after_sync();
                const uint32_t hs = sbase + F_H + (t & 1) * H_OP;
                const uint64_t hop = op_desc(hs, HD);
#pragma unroll
                for (int ks = 0; ks < HD / 16; ++ks)
#pragma unroll
                    for (int g = 0; g < 3; ++g)
                        U::mma_bf16_warp_ta(acc + g * NN, tmem + F_WHH + g * (HD / 2) + ks * 8, hop + ks * 16, id,
                                            (g < 2 || ks > 0) ? 1u : 0u, leader);
                if (leader) {  // the weight gradient's images of h before this step
                    U::bulk_store(w.h_hi + (u0 + t) * H_PARTB, hs, H_PARTB);
                    U::bulk_store(w.h_lo + (u0 + t) * H_PARTB, hs + H_PARTB, H_PARTB);
                    if (t > 1) store_c(t - 2);  // written before h of step t - 1
                    U::bulk_commit();
                    U::bulk_wait_read_but_last();  // (the other buffer, which the epilogue writes next)
                    U::commit(hbar);
                }
                __syncwarp();
                // a free buffer: its last reader, step t - 1, is done (h of that step is written)
                if (t + NBUF - 1 < tmax) load_a(t + NBUF - 1);
                if (t + 1 < tmax) {  // under this step's gate math, once its accumulators are loaded
                    if (waited(lbar, t) && a_landed(t + 1)) {
                        U::fence_after_sync();
                        input_mmas(t + 1);
                    } else {
                        err = ERR_FWD_COPY;
                    }
                }
            }
            if (!err && waited(fin, 0)) {  // the last two steps' values
                U::fence_smem_async();
                if (leader) {
                    if (tmax > 1) store_c(tmax - 2);
                    store_c(tmax - 1);
                    U::bulk_commit();
                }
                __syncwarp();
            } else if (!err) {
                err = ERR_FWD_MMA;
            }
            // nothing of this CTA may be in flight when it exits
            if (err) {
                if (leader) atomicOr(status, err);
                for (int i = max(0, loaded - NBUF); i < loaded; ++i) a_landed(i);
            }
            if (leader) {
                U::bulk_wait();
                U::commit(last);
            }
            __syncwarp();
            if (!waited(last, 0) && leader) {
                atomicOr(status, ERR_HELD);
                busy = 1;
            }
        }
    } else {
        const uint32_t tl = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + F_ACC + 4 * q;
        int n[4];
        float h[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            n[e] = n_s[4 * q + e];
            h[e] = 0.f;
        }
        const float br = p[OFF_BIH + k] + p[OFF_BHH + k], bz = p[OFF_BIH + HD + k] + p[OFF_BHH + HD + k];
        const float bni = p[OFF_BIH + 2 * HD + k], bnh = p[OFF_BHH + 2 * HD + k];
        bool failed = false;
        for (int t = 0; t < tmax; ++t) {
            if (!__all_sync(0xffffffffu, U::mbar_wait(hbar, (uint32_t)(t & 1), wait_cycles))) {
                if (lane == 0) atomicOr(status, ERR_FWD_MMA);
                failed = true;
                break;
            }
            U::fence_after_sync();
            Parts pr, pz, ph, pi;
            pr.load(tl);
            pz.load(tl + NN);
            ph.load(tl + 2 * NN);
            pi.load(tl + 3 * NN);
            pr.wait();
            pz.wait();
            ph.wait();
            pi.wait();
            U::fence_before_sync();
            __syncwarp();
            if (lane == 0) U::mbar_arrive(lbar);
            float vr[4], vz[4], vn[4], vg[4], hp[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                vr[e] = sigm(pr.sum(e) + br);
                vz[e] = sigm(pz.sum(e) + bz);
                vg[e] = ph.sum(e) + bnh;
                vn[e] = tanhf(pi.sum(e) + bni + vr[e] * vg[e]);
                hp[e] = h[e];
                if (t < n[e]) h[e] = (1.f - vz[e]) * vn[e] + vz[e] * h[e];
            }
            Split(h).put(sm + F_H + ((t + 1) & 1) * H_OP, k, q);
            U::fence_before_sync();
            __syncwarp();
            if (lane == 0) U::mbar_arrive(rbar);
            // Off the chain: what BPTT reads, copied out two steps later.  (Stored
            // from here, 40 KB a step stalled the warps for 1,200 cycles.)
            unsigned char* cp = sm + F_C + t % 3 * C_OP + (q * HD + k) * 16;
            auto put4 = [&](int i, const float (&v)[4]) {
                *reinterpret_cast<float4*>(cp + i * (C_OP / 5)) = make_float4(v[0], v[1], v[2], v[3]);
            };
            put4(0, vr);
            put4(1, vz);
            put4(2, vn);
            put4(3, vg);
            put4(4, hp);
        }
        __syncwarp();
        if (lane == 0 && !failed) U::mbar_arrive(fin);  // the last step's values written
        if (tmax < nt) {  // the slot that rounds the block up
            zero_img(w.h_hi, u0 + nt - 1, k, q);
            zero_img(w.h_lo, u0 + nt - 1, k, q);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int b = b_s[4 * q + e];
            if (b >= 0) hl[(int64_t)b * HD + k] = failed ? __int_as_float(0x7fc00000) : h[e];
        }
    }
    U::fence_before_sync();
    __syncthreads();
    if (warp == 0 && !busy) {
        U::fence_after_sync();
        U::tmem_dealloc(tmem, COLS);
    }
}

// Shared memory of the backward: the gate gradients r, z, n (input), n
// (hidden), an operand each, two buffers; the forward's values, two buffers; barriers
constexpr int B_G = 0, B_SET = 4 * H_OP, B_C = B_G + 2 * B_SET, B_BAR = B_C + 2 * C_OP, B_SMEM = B_BAR + 64;
static_assert(B_SMEM + 1024 <= 227 * 1024, "train_gru_bwd shared memory");
// Tensor memory: Whh^T (lane = k, K = gate rows), Wih^T (lanes 0..63 = c; M = 64 would take the tensor cores twice
// as long as M = 128), dh, dA
constexpr uint32_t B_WHH = 0, B_WIH = B_WHH + G3 / 2, B_DH = B_WIH + G3 / 2, B_DA = B_DH + NN;
static_assert(B_DA + NN <= COLS, "train_gru_bwd tensor memory");

__global__ void __launch_bounds__(THREADS, 1) train_gru_bwd(const int32_t* __restrict__ len, int T,
                                                            const __nv_bfloat16* __restrict__ wq,
                                                            const float* __restrict__ dhl, TrainWs w,
                                                            float* __restrict__ gbih, float* __restrict__ gbhh,
                                                            int* __restrict__ status, long long wait_cycles) {
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ int n_s[TB], b_s[TB], busy;
    const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(sm));
    // mbarriers: a step's dh products done, its dA products done, its gate gradients written, the last products done,
    // the forward's values landed (one a buffer)
    const uint32_t hbar = sbase + B_BAR, abar = hbar + 8, rbar = hbar + 16, last = hbar + 24, cbar = hbar + 32;
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(sm + B_BAR + 48);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int k = 32 * (warp & 3) + lane, q = warp >> 2;
    const int blk = blockIdx.x;
    const int64_t u0 = w.slot0[blk];
    const int nt = w.slot0[blk + 1] - (int)u0;

    if (tid < TB) {
        const int b = w.perm[blk * TB + tid];
        b_s[tid] = b;
        n_s[tid] = b >= 0 ? min(max(len[b], 0), T) : 0;
    }
    if (tid == 0) {
        U::mbar_init(hbar, 1);
        U::mbar_init(abar, 1);
        U::mbar_init(rbar, EPI / 32);
        U::mbar_init(last, 1);
        for (int i = 0; i < 2; ++i) U::mbar_init(cbar + 8 * i, 1);
        busy = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) U::tmem_alloc(sbase + B_BAR + 48, COLS);
    U::fence_smem_async();
    U::fence_before_sync();
    __syncthreads();
    U::fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    if (warp < EPI / 32) {  // the weights, transposed: 16 K (gate rows) a write
        const uint32_t tw = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
        const unsigned short* whh = reinterpret_cast<const unsigned short*>(wq + OFF_WHH) + k;
        const unsigned short* wih = reinterpret_cast<const unsigned short*>(wq + OFF_WIH) + k;
        for (int i = q; i < G3 / 16; i += 4) {
            uint32_t r[8], x[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int row = 16 * i + 2 * j;
                r[j] = (uint32_t)whh[row * HD] | (uint32_t)whh[(row + 1) * HD] << 16;
                x[j] = k < C1 ? (uint32_t)wih[row * C1] | (uint32_t)wih[(row + 1) * C1] << 16 : 0u;
            }
            __syncwarp();
            U::st8(tw + B_WHH + 8 * i, r);
            U::st8(tw + B_WIH + 8 * i, x);
        }
        U::wait_st();
    }
    U::fence_before_sync();
    __syncthreads();
    U::fence_after_sync();
    int tmax = 0;
    for (int s = 0; s < TB; ++s) tmax = max(tmax, n_s[s]);

    if (warp == EPI / 32) {  // MMAs
        if (tmax > 0) {  // the whole warp runs this, its leader issues
            constexpr uint32_t id = U::idesc_bf16_f32_bmn(HD, NN);
            const uint32_t leader = U::elect_leader();
            const int64_t img_tile = w.slots * H_PARTB;  // bytes between the images of two gates
            auto waited = [&](uint32_t bar, int parity) {
                return (bool)__all_sync(0xffffffffu, U::mbar_wait(bar, (uint32_t)(parity & 1), wait_cycles));
            };
            int loaded = 0;
            auto load_c = [&]() {  // the next step's values of the forward
                if (loaded == tmax) return;
                const uint32_t bar = cbar + 8 * (loaded & 1);
                if (leader) {
                    U::mbar_arrive_expect_tx(bar, C_OP);
                    U::bulk_load(sbase + B_C + (loaded & 1) * C_OP,
                                 reinterpret_cast<const unsigned char*>(w.cache) + (u0 + tmax - 1 - loaded) * C_OP, C_OP, bar);
                }
                __syncwarp();
                ++loaded;
            };
            load_c();
            load_c();
            for (int i = 0; i < tmax; ++i) {
                if (!waited(rbar, i)) {
                    if (leader) atomicOr(status, ERR_BWD_MMA);
                    for (int j = max(0, loaded - 2); j < loaded; ++j) waited(cbar + 8 * (j & 1), j / 2);
                    break;
                }
                U::fence_smem_async();
                U::fence_after_sync();
                const uint32_t gs = sbase + B_G + (i & 1) * B_SET;
                const uint64_t gop = op_desc(gs, HD);
                auto mma = [&](uint32_t d, uint32_t a, int kg, int n_op) {  // 16 K: rows 16 kg of the gates r, z, n of one side
                    const int g = kg / (HD / 16);
                    U::mma_bf16_warp_ta(d, a + 8 * kg, gop + ((g == 2 ? n_op : g) * H_OP >> 4) + kg % (HD / 16) * 16, id, kg,
                                        leader);
                };
#pragma unroll
                for (int kg = 0; kg < G3 / 16; ++kg) mma(tmem + B_DH, tmem + B_WHH, kg, 3);
                if (leader) U::commit(hbar);
                __syncwarp();
                load_c();  // into this step's buffer
#pragma unroll
                for (int kg = 0; kg < G3 / 16; ++kg) mma(tmem + B_DA, tmem + B_WIH, kg, 2);
                if (leader) {  // the weight gradient's images
                    const int64_t at = (u0 + tmax - 1 - i) * H_PARTB;
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        U::bulk_store(w.g_hi + g * img_tile + at, gs + g * H_OP, H_PARTB);
                        U::bulk_store(w.g_lo + g * img_tile + at, gs + g * H_OP + H_PARTB, H_PARTB);
                    }
                    U::bulk_commit();
                    U::bulk_wait_read_but_last();  // (the other buffer, which the epilogue writes next)
                    U::commit(abar);
                }
                __syncwarp();
            }
            if (leader) {  // nothing of this CTA may be in flight when it exits
                U::bulk_wait();
                U::commit(last);
            }
            __syncwarp();
            if (!waited(last, 0) && leader) {
                atomicOr(status, ERR_HELD);
                busy = 1;
            }
        }
    } else {
        const uint32_t tl = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + 4 * q;
        int n[4];
        float dh[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            n[e] = n_s[4 * q + e];
            const int b = b_s[4 * q + e];
            dh[e] = b >= 0 ? dhl[(int64_t)b * HD + k] : 0.f;
        }
        if (tmax < nt)
            for (int g = 0; g < 4; ++g) {
                zero_img(w.g_hi + g * w.slots * H_PARTB, u0 + nt - 1, k, q);
                zero_img(w.g_lo + g * w.slots * H_PARTB, u0 + nt - 1, k, q);
            }
        // the conv gradient of step t (lanes 0..63), from the loaded accumulators
        const bool has_dA = (warp & 3) < C1 / 32;
        auto signs = [&](int t) { return (uint32_t)__ldg(w.a_on + (2 * (u0 + t) + (q >> 1)) * C1 + k); };
        auto put_dA = [&](int t, const Parts& pa, uint32_t on) {
            const int64_t u = u0 + t;
            float v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = (on >> (4 * (q & 1) + e) & 1u) ? pa.sum(e) : 0.f;
            *reinterpret_cast<float4*>(w.dA + ((4 * u + q) * C1 + k) * 4) = make_float4(v[0], v[1], v[2], v[3]);
        };
        auto waited = [&](uint32_t bar, uint32_t parity) {
            const bool ok = __all_sync(0xffffffffu, U::mbar_wait(bar, parity, wait_cycles));
            if (!ok && lane == 0) atomicOr(status, ERR_BWD_MMA);
            U::fence_after_sync();
            return ok;
        };
        float sr = 0.f, sz = 0.f, sn = 0.f, snh = 0.f;  // bias gradients
        bool ok = true;
        // What a step's gate gradients need besides dh, formed while the previous
        // step's products run: dn = (1 - z)(1 - n^2) dh, dr = (Whn h + bhn) r (1 - r)
        // dn, dz = (h - n) z (1 - z) dh
        float cn[4], cr[4], cz[4], r[4], z[4];
        auto coefficients = [&](uint32_t i) {
            if (!waited(cbar + 8 * (i & 1), (i >> 1) & 1)) return false;
            const float* cp = reinterpret_cast<const float*>(sm + B_C + (i & 1) * C_OP + (q * HD + k) * 16);
            float c[5][4];
#pragma unroll
            for (int j = 0; j < 5; ++j) {
                const float4 x = *reinterpret_cast<const float4*>(cp + j * (C_OP / 20));
                c[j][0] = x.x; c[j][1] = x.y; c[j][2] = x.z; c[j][3] = x.w;
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                r[e] = c[0][e];
                z[e] = c[1][e];
                const float nn = c[2][e];
                cn[e] = (1.f - z[e]) * (1.f - nn * nn);
                cr[e] = c[3][e] * r[e] * (1.f - r[e]);
                cz[e] = (c[4][e] - nn) * z[e] * (1.f - z[e]);
            }
            return true;
        };
        if (tmax > 0) ok = coefficients(0);
        for (int t = tmax - 1; t >= 0 && ok; --t) {
            const uint32_t i = (uint32_t)(tmax - 1 - t);  // steps before this one
            const uint32_t on = i > 0 && has_dA ? signs(t + 1) : 0;
            float gr[4], gz[4], gn[4], gh[4], d[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const bool live = t < n[e];
                const float g = dh[e], vn = g * cn[e];
                gn[e] = live ? vn : 0.f;
                gr[e] = live ? vn * cr[e] : 0.f;
                gz[e] = live ? g * cz[e] : 0.f;
                gh[e] = live ? vn * r[e] : 0.f;
                d[e] = live ? g * z[e] : g;  // past its end a trajectory's dh passes through
                sr += gr[e];
                sz += gz[e];
                sn += gn[e];
                snh += gh[e];
            }
            const Split xr(gr), xz(gz), xn(gn), xh(gh);
            Parts pa;
            if (i > 0) {  // the previous step's dA products are done (and the copies out of this step's buffer)
                if (!(ok = waited(abar, (i - 1) & 1))) break;
                if (has_dA) pa.load(tl + B_DA);
            }
            unsigned char* g_op = sm + B_G + (i & 1) * B_SET;
            xr.put(g_op, k, q);
            xz.put(g_op + H_OP, k, q);
            xn.put(g_op + 2 * H_OP, k, q);
            xh.put(g_op + 3 * H_OP, k, q);
            if (i > 0 && has_dA) pa.wait();
            U::fence_before_sync();
            __syncwarp();
            if (lane == 0) U::mbar_arrive(rbar);
            if (i > 0 && has_dA) put_dA(t + 1, pa, on);
            if (t > 0 && !(ok = coefficients(i + 1))) break;
            if (!(ok = waited(hbar, i & 1))) break;
            Parts pd;
            pd.load(tl + B_DH);
            pd.wait();
#pragma unroll
            for (int e = 0; e < 4; ++e) dh[e] = d[e] + pd.sum(e);
        }
        if (tmax > 0 && ok && waited(abar, (uint32_t)(tmax - 1) & 1) && has_dA) {
            Parts pa;
            pa.load(tl + B_DA);
            pa.wait();
            put_dA(0, pa, signs(0));
        }
        if (tmax > 0) {
            atomicAdd(gbih + k, sr);
            atomicAdd(gbih + HD + k, sz);
            atomicAdd(gbih + 2 * HD + k, sn);
            atomicAdd(gbhh + k, sr);
            atomicAdd(gbhh + HD + k, sz);
            atomicAdd(gbhh + 2 * HD + k, snh);
        }
    }
    U::fence_before_sync();
    __syncthreads();
    if (warp == 0 && !busy) {
        U::fence_after_sync();
        U::tmem_dealloc(tmem, COLS);
    }
}

// Conv weight gradients.  CTA = (block, CB_T steps), 704 threads: thread q
// takes weight (c, i, k) = (q / 10, (q / 5) % 2, q % 5) of the 640, or the bias
// of channel q - 640, summed over the steps and trajectories (one atomic per
// thread).  The normalised inputs are staged in shared memory.  (One CTA per
// block, 128 for a batch of 2,048, was bound by the latency of its gradient
// loads: 0.21 ms.)
constexpr int CB_THREADS = C1 * 2 * KW + C1;  // 704
constexpr int CB_T = 32;
constexpr int CB_I = TB + 4, CB_U = CB_I + TB;  // a warp's 10 (i, k) windows in 8 groups of 4 banks: two wavefronts, not five
__global__ void __launch_bounds__(CB_THREADS) train_conv_bwd(const float2* __restrict__ pts,
                                                            const int64_t* __restrict__ off,
                                                            const int32_t* __restrict__ len, float4 nrm, TrainWs w,
                                                            float* __restrict__ grad) {
    __shared__ __align__(16) float xs[(CB_T + KW - 1) * CB_U];  // input i of trajectory s at step t0 + u - 2: u CB_U + i CB_I + s
    const int blk = blockIdx.x, q = threadIdx.x, t0 = blockIdx.y * CB_T;
    const int64_t u0 = w.slot0[blk];
    int tmax = 0;
    for (int s = 0; s < TB; ++s) {
        const int b = w.perm[blk * TB + s];
        if (b >= 0) tmax = max(tmax, min(len[b], w.slot0[blk + 1] - (int)u0));
    }
    const int t1 = min(tmax, t0 + CB_T);
    if (t0 >= t1) return;
    const bool wt = q < C1 * 2 * KW;
    const int c = wt ? q / (2 * KW) : q - C1 * 2 * KW, i = (q / KW) % 2, k = q % KW;
    for (int e = q; e < (t1 - t0 + KW - 1) * 2 * TB; e += CB_THREADS) {
        const int s = e % TB, ii = (e / TB) % 2, u = e / (2 * TB);
        const int b = w.perm[blk * TB + s];
        xs[u * CB_U + ii * CB_I + s] = b >= 0 ? xin(pts, off[b], len[b], t0 + u - 2, ii, nrm) : 0.f;
    }
    __syncthreads();
    float acc = 0.f;
#pragma unroll 4
    for (int t = t0; t < t1; ++t) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 g = __ldg(reinterpret_cast<const float4*>(w.dA + ((4 * (u0 + t) + j) * C1 + c) * 4));
            if (wt) {
                const float4 x = *reinterpret_cast<const float4*>(xs + (t - t0 + k) * CB_U + i * CB_I + 4 * j);
                acc = fmaf(g.x, x.x, fmaf(g.y, x.y, fmaf(g.z, x.z, fmaf(g.w, x.w, acc))));
            } else {
                acc += (g.x + g.y) + (g.z + g.w);
            }
        }
    }
    atomicAdd(grad + (wt ? OFF_W1 + q : OFF_B1 + c), acc);
}

namespace {
int check(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return TSM_OK;
    char b[256];
    snprintf(b, sizeof(b), "%s: %s", what, cudaGetErrorString(e));
    return tsm_internal_fail(TSM_ECUDA, b);
}
}  // namespace

int64_t train_layout(int B, int T, unsigned char* base, TrainWs* w) {
    int64_t o = 0;
    auto take = [&](int64_t bytes) {
        unsigned char* q = base ? base + o : nullptr;
        o += (bytes + 255) & ~int64_t(255);
        return q;
    };
    TrainWs x;
    x.blocks = (B + TB - 1) / TB;
    x.slots = (int64_t)x.blocks * ((T + 1) & ~1);
    const int64_t groups = 2 * x.slots;
    x.perm = reinterpret_cast<int32_t*>(take((int64_t)x.blocks * TB * 4));
    x.slot0 = reinterpret_cast<int32_t*>(take((int64_t)(x.blocks + 1) * 4));
    x.a_op = take(x.slots * A_OP);
    x.a_on = take(groups * C1);
    x.h_hi = take(groups * HD * 16);
    x.h_lo = take(groups * HD * 16);
    x.cache = reinterpret_cast<float*>(take(x.slots * 5 * 2 * HD * 8 * 4));
    x.g_hi = take(4 * groups * HD * 16);
    x.g_lo = take(4 * groups * HD * 16);
    x.dA = reinterpret_cast<float*>(take(groups * C1 * 8 * 4));
    if (w) *w = x;
    return o;
}

int train_forward(const float2* pts, const int64_t* off, const int32_t* len, int B, int T, float4 nrm,
                  const __nv_bfloat16* wq, const float* p, const TrainWs& w, float* hl, int* status, cudaStream_t s) {
    train_plan<<<1, 1024, 0, s>>>(len, B, T, w.blocks, w.perm, w.slot0);
    const int chunks = (((T + 1) & ~1) + CV_T - 1) / CV_T;
    if (chunks > 65535) return tsm_internal_fail(TSM_EINVAL, "encoder: trajectory too long to train on");
    train_conv<<<dim3(w.blocks, chunks), 128, 0, s>>>(pts, off, len, T, nrm, wq, p, w);
    int rc = check(cudaFuncSetAttribute(train_gru_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, F_SMEM),
                   "cudaFuncSetAttribute(train_gru_fwd)");
    if (rc) return rc;
    train_gru_fwd<<<w.blocks, THREADS, F_SMEM, s>>>(len, T, wq, p, w, hl, status, WAIT_CYCLES);
    return check(cudaGetLastError(), "training forward launch");
}

int train_backward(const float2* pts, const int64_t* off, const int32_t* len, int B, int T, float4 nrm,
                   const __nv_bfloat16* wq, const float* dhl, const TrainWs& w, float* grad, int* status,
                   cudaStream_t s) {
    int rc = check(cudaFuncSetAttribute(train_gru_bwd, cudaFuncAttributeMaxDynamicSharedMemorySize, B_SMEM),
                   "cudaFuncSetAttribute(train_gru_bwd)");
    if (rc) return rc;
    train_gru_bwd<<<w.blocks, THREADS, B_SMEM, s>>>(len, T, wq, dhl, w, grad + OFF_BIH, grad + OFF_BHH, status,
                                                    WAIT_CYCLES);
    if ((rc = tsm_wgrad_tc(w, status, grad + OFF_WIH, grad + OFF_WHH, s))) return rc;
    train_conv_bwd<<<dim3(w.blocks, (((T + 1) & ~1) + CB_T - 1) / CB_T), CB_THREADS, 0, s>>>(pts, off, len, nrm, w, grad);
    return check(cudaGetLastError(), "training backward launch");
}

}  // namespace enc
