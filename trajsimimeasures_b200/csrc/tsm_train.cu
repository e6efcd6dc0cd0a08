// Training recurrences of the encoder on the tensor cores (tcgen05): the GRU
// over time with the values BPTT needs, BPTT itself, and the gradients of the
// conv layer.
//
// Each time step's products are W [gates x features] times the features of 16
// trajectories: the weights are the MMA's A operand (M = 128 gate rows, BF16,
// resident in shared memory for all steps) and the trajectories its N.  The
// activations are FP32: x = hi + mid + lo, three BF16 parts that hold all 24
// bits, stand side by side as N = 3 x 16 columns, and the epilogue adds the
// three FP32 results.  Products of BF16 values are exact in FP32, so a sum
// differs from an FP32 one only in how it is accumulated.
//
// Threads: 256 of the epilogue, thread (k, half) with k = hidden unit
// (tensor-memory lane) and half = 8 of the block's 16 trajectories, whose h
// (dh) it keeps in registers, and a ninth warp that issues copies and MMAs.  Eight values of one unit are eight consecutive N, so the three
// parts go to the operand in shared memory as one 16-byte store each
// (MN-major: element (n, k) at (k / 8) * 768 + (n / 8) * 128 + (k % 8) * 16 +
// (n % 8) * 2), and to the weight gradient's operand images likewise, whose K
// runs over (slot, trajectory).
//
// Blocks take trajectories of similar length (a counting sort by length), so
// few of a block's 16 rows idle, and time steps are stored compactly.
//
// What bounds it: the chain of steps.  A step is 24 MMAs (M = 128, N = 48, K =
// 16) on the previous step's result, a commit, the tensor-memory loads and the
// gate math; the input products of the next step run under the gate math.
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
constexpr int KG = NN * 16;            // bytes of 8 K rows of an operand (the K-group stride): 768
constexpr int A_OP = C1 / 8 * KG;      // 6,144
constexpr int H_OP = HD / 8 * KG;      // 12,288
constexpr int G_OP = G3 / 8 * KG;      // 36,864
constexpr int EPI = 256;               // epilogue threads
constexpr int THREADS = EPI + 32;      // + the issuing warp
constexpr int NBUF = 3;                // a-operand buffers of the forward
constexpr int W_HH = HD * HD * 2;      // one gate's Whh tile: 32 KB
constexpr int W_IH = HD * C1 * 2;      // one gate's Wih tile: 16 KB
constexpr long long WAIT_CYCLES = 2000000000LL;  // ~1 s of SM clocks
// status bits
constexpr int ERR_FWD_COPY = 256, ERR_FWD_MMA = 512, ERR_BWD_MMA = 1024, ERR_HELD = 128;

__device__ __forceinline__ uint64_t op_desc(uint32_t saddr) { return U::smem_desc(saddr, KG, 128); }

__device__ __forceinline__ float sigm(float x) { return 1.f / (1.f + expf(-x)); }

// Eight values as three BF16 parts, x = hi + mid + lo.
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float lo_of(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float hi_of(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }
__device__ __forceinline__ void split8(const float (&v)[8], uint4& hi, uint4& mid, uint4& lo) {
    uint32_t h[4], m[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float a = v[2 * i], b = v[2 * i + 1];
        h[i] = pack2(a, b);
        const float a1 = a - lo_of(h[i]), b1 = b - hi_of(h[i]);
        m[i] = pack2(a1, b1);
        l[i] = pack2(a1 - lo_of(m[i]), b1 - hi_of(m[i]));
    }
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    mid = make_uint4(m[0], m[1], m[2], m[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
}
// K row k of an operand: the three parts of this thread's 8 trajectories.
__device__ __forceinline__ void put_op(unsigned char* op, int k, int half, const uint4& hi, const uint4& mid,
                                       const uint4& lo) {
    unsigned char* d = op + (k >> 3) * KG + half * 128 + (k & 7) * 16;
    *reinterpret_cast<uint4*>(d) = hi;
    *reinterpret_cast<uint4*>(d + 256) = mid;
    *reinterpret_cast<uint4*>(d + 512) = lo;
}
// One group row of an image: [group][rows][8] BF16.
__device__ __forceinline__ void put_img(unsigned char* img, int64_t group, int rows, int r, const uint4& v) {
    *reinterpret_cast<uint4*>(img + ((group * rows + r) << 4)) = v;
}

// The sum of the three parts' results, 8 columns from `col` (this thread's
// lane and half; parts 16 columns apart).
struct Parts {
    uint32_t r[3][8];
    __device__ __forceinline__ void load(uint32_t taddr) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 3; ++i) U::ld8(taddr + 16 * i, r[i]);
    }
    __device__ __forceinline__ void wait() {
#pragma unroll
        for (int i = 0; i < 3; ++i) U::wait_ld8(r[i]);
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

// conv + relu of every slot: the recurrence's operand, the weight gradient's
// images and the relu's sign bits.  CTA = (block, 16 slots); thread (half, c).
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
        uint4 hi, mid, lo;
        split8(a, hi, mid, lo);
        const int64_t u = u0 + t, g = 2 * u + half;
        put_op(w.a_op + u * A_OP, c, half, hi, mid, lo);
        put_img(w.a_hi, g, C1, c, hi);
        put_img(w.a_lo, g, C1, c, mid);
        w.a_on[g * C1 + c] = (unsigned char)on;
    }
}

// Shared memory of the forward: Whh (3 tiles), Wih (3 tiles), h, a (NBUF buffers), barriers
constexpr int F_WHH = 0, F_WIH = F_WHH + 3 * W_HH, F_H = F_WIH + 3 * W_IH, F_A = F_H + H_OP, F_BAR = F_A + NBUF * A_OP,
              F_SMEM = F_BAR + 64;
static_assert(F_SMEM + 1024 <= 227 * 1024, "train_gru_fwd shared memory");
constexpr uint32_t F_COLS = 512;  // two sets of accumulators r, z, n (hidden), n (input), 48 columns each
constexpr uint32_t F_SET = 4 * NN;

__global__ void __launch_bounds__(THREADS, 1) train_gru_fwd(const int32_t* __restrict__ len, int T,
                                                            const __nv_bfloat16* __restrict__ wq,
                                                            const float* __restrict__ p, TrainWs w,
                                                            float* __restrict__ hl, int* __restrict__ status,
                                                            long long wait_cycles) {
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ int n_s[TB], b_s[TB], busy;
    const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(sm));
    // mbarriers: a step's products done, its h written, a-buffer i landed, the last products done
    const uint32_t hbar = sbase + F_BAR, rbar = hbar + 8, abar = hbar + 16, last = abar + 8 * NBUF;
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(sm + F_BAR + 56);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int k = 32 * (warp & 3) + lane, half = warp >> 2;
    const int blk = blockIdx.x;
    const int64_t u0 = w.slot0[blk];
    const int nt = w.slot0[blk + 1] - (int)u0;

    for (int e = tid; e < G3 * (HD / 8); e += THREADS) {
        const int r = e / (HD / 8), c = e % (HD / 8);
        *reinterpret_cast<uint4*>(sm + F_WHH + (r / HD) * W_HH + U::core_offset(r % HD, 8 * c, HD)) =
            *reinterpret_cast<const uint4*>(wq + OFF_WHH + r * HD + 8 * c);
    }
    for (int e = tid; e < G3 * (C1 / 8); e += THREADS) {
        const int r = e / (C1 / 8), c = e % (C1 / 8);
        *reinterpret_cast<uint4*>(sm + F_WIH + (r / HD) * W_IH + U::core_offset(r % HD, 8 * c, HD)) =
            *reinterpret_cast<const uint4*>(wq + OFF_WIH + r * C1 + 8 * c);
    }
    for (int e = tid; e < H_OP / 16; e += THREADS) *reinterpret_cast<uint4*>(sm + F_H + 16 * e) = make_uint4(0, 0, 0, 0);
    if (tid < TB) {
        const int b = w.perm[blk * TB + tid];
        b_s[tid] = b;
        n_s[tid] = b >= 0 ? min(max(len[b], 0), T) : 0;
    }
    if (tid == 0) {
        U::mbar_init(hbar, 1);
        U::mbar_init(rbar, EPI / 32);
        for (int i = 0; i < NBUF; ++i) U::mbar_init(abar + 8 * i, 1);
        U::mbar_init(last, 1);
        busy = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) U::tmem_alloc(sbase + F_BAR + 56, F_COLS);
    U::fence_smem_async();
    U::fence_before_sync();
    __syncthreads();
    U::fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    int tmax = 0;
    for (int s = 0; s < TB; ++s) tmax = max(tmax, n_s[s]);

    if (warp == EPI / 32) {  // copies and MMAs
        if (tmax > 0) {  // the whole warp runs this, its leader issues
            constexpr uint32_t id = U::idesc_bf16_f32_bmn(HD, NN);
            const uint32_t leader = U::elect_leader();
            const uint64_t whh = U::smem_desc(sbase + F_WHH, HD * 16, 128), wih = U::smem_desc(sbase + F_WIH, HD * 16, 128);
            const uint64_t hop = op_desc(sbase + F_H);
            auto step_of = [](int bytes) { return (uint64_t)(bytes >> 4); };  // descriptor increment of a start address
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
            // the input products of step t into its accumulator set
            auto input_mmas = [&](int t) {
                const uint32_t d = tmem + (t & 1) * F_SET;
                const uint64_t a = op_desc(sbase + F_A + (t % NBUF) * A_OP);
#pragma unroll
                for (int g = 0; g < 3; ++g)
#pragma unroll
                    for (int ks = 0; ks < C1 / 16; ++ks)
                        U::mma_bf16_warp(d + (g == 2 ? 3 * NN : g * NN), wih + step_of(g * W_IH + ks * 2 * (HD * 16)),
                                         a + step_of(ks * 2 * KG), id, ks, leader);
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
                U::fence_after_sync();
                const uint32_t d = tmem + (t & 1) * F_SET;
#pragma unroll
                for (int g = 0; g < 3; ++g)
#pragma unroll
                    for (int ks = 0; ks < HD / 16; ++ks)
                        U::mma_bf16_warp(d + g * NN, whh + step_of(g * W_HH + ks * 2 * (HD * 16)),
                                         hop + step_of(ks * 2 * KG), id, (g < 2 || ks > 0) ? 1u : 0u, leader);
                if (leader) U::commit(hbar);
                __syncwarp();
                // a free buffer: its last reader, step t - 1, is done (h of that step is written)
                if (t + NBUF - 1 < tmax) load_a(t + NBUF - 1);
                if (t + 1 < tmax) {  // under this step's gate math
                    if (a_landed(t + 1)) {
                        U::fence_after_sync();
                        input_mmas(t + 1);
                    } else {
                        err = ERR_FWD_COPY;
                    }
                }
            }
            // nothing of this CTA may be in flight when it exits
            if (err) {
                if (leader) atomicOr(status, err);
                for (int i = max(0, loaded - NBUF); i < loaded; ++i) a_landed(i);
            }
            if (leader) U::commit(last);
            __syncwarp();
            if (!waited(last, 0) && leader) {
                atomicOr(status, ERR_HELD);
                busy = 1;
            }
        }
    } else {
        const uint32_t tl = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + 8 * half;
        int n[8];
        float h[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            n[e] = n_s[8 * half + e];
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
            const uint32_t ta = tl + (t & 1) * F_SET;
            Parts pr, pz, ph, pi;
            pr.load(ta);
            pz.load(ta + NN);
            ph.load(ta + 2 * NN);
            pi.load(ta + 3 * NN);
            pr.wait();
            pz.wait();
            ph.wait();
            pi.wait();
            float vr[8], vz[8], vn[8], vg[8], hp[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                vr[e] = sigm(pr.sum(e) + br);
                vz[e] = sigm(pz.sum(e) + bz);
                vg[e] = ph.sum(e) + bnh;
                vn[e] = tanhf(pi.sum(e) + bni + vr[e] * vg[e]);
                hp[e] = h[e];
                if (t < n[e]) h[e] = (1.f - vz[e]) * vn[e] + vz[e] * h[e];
            }
            uint4 hi, mid, lo;
            split8(h, hi, mid, lo);
            put_op(sm + F_H, k, half, hi, mid, lo);
            U::fence_smem_async();
            U::fence_before_sync();
            __syncwarp();
            if (lane == 0) U::mbar_arrive(rbar);
            // off the chain: what BPTT and the weight gradients read
            const int64_t u = u0 + t;
            float* cp = w.cache + ((u * 5 * 2 + half) * HD + k) * 8;
            auto put8 = [&](int i, const float (&v)[8]) {
                float4* q = reinterpret_cast<float4*>(cp + (int64_t)i * 2 * HD * 8);
                q[0] = make_float4(v[0], v[1], v[2], v[3]);
                q[1] = make_float4(v[4], v[5], v[6], v[7]);
            };
            put8(0, vr);
            put8(1, vz);
            put8(2, vn);
            put8(3, vg);
            put8(4, hp);
            split8(hp, hi, mid, lo);
            put_img(w.h_hi, 2 * u + half, HD, k, hi);
            put_img(w.h_lo, 2 * u + half, HD, k, mid);
        }
        if (tmax < nt) {  // the slot that rounds the block up
            put_img(w.h_hi, 2 * (u0 + nt - 1) + half, HD, k, make_uint4(0, 0, 0, 0));
            put_img(w.h_lo, 2 * (u0 + nt - 1) + half, HD, k, make_uint4(0, 0, 0, 0));
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int b = b_s[8 * half + e];
            if (b >= 0) hl[(int64_t)b * HD + k] = failed ? __int_as_float(0x7fc00000) : h[e];
        }
    }
    U::fence_before_sync();
    __syncthreads();
    if (warp == 0 && !busy) {
        U::fence_after_sync();
        U::tmem_dealloc(tmem, F_COLS);
    }
}

// Shared memory of the backward: Whh^T (128 x 384), Wih^T (64 x 384), hidden-side
// gate gradients (K = 384), input-side n gradients (K = 128), barriers
constexpr int B_WHH = 0, B_WIH = B_WHH + HD * G3 * 2, B_G = B_WIH + C1 * G3 * 2, B_N = B_G + G_OP, B_BAR = B_N + H_OP,
              B_SMEM = B_BAR + 64;
static_assert(B_SMEM + 1024 <= 227 * 1024, "train_gru_bwd shared memory");
constexpr uint32_t B_COLS = 128;  // dh at column 0, dA at 64

__global__ void __launch_bounds__(THREADS, 1) train_gru_bwd(const int32_t* __restrict__ len, int T,
                                                            const __nv_bfloat16* __restrict__ wq,
                                                            const float* __restrict__ dhl, TrainWs w,
                                                            float* __restrict__ gbih, float* __restrict__ gbhh,
                                                            int* __restrict__ status, long long wait_cycles) {
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ int n_s[TB], b_s[TB], busy;
    const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(sm));
    // mbarriers: a step's dh products done, its dA products done, its gate gradients written, the last products done
    const uint32_t hbar = sbase + B_BAR, abar = hbar + 8, rbar = hbar + 16, last = hbar + 24;
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(sm + B_BAR + 32);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int k = 32 * (warp & 3) + lane, half = warp >> 2;
    const int blk = blockIdx.x;
    const int64_t u0 = w.slot0[blk];
    const int nt = w.slot0[blk + 1] - (int)u0;

    for (int e = tid; e < G3 * HD / 2; e += THREADS) {  // Whh[j][k] -> row k, K = j
        const int j = 2 * (e / HD), kk = e % HD;
        const __nv_bfloat162 v{wq[OFF_WHH + j * HD + kk], wq[OFF_WHH + (j + 1) * HD + kk]};
        *reinterpret_cast<__nv_bfloat162*>(sm + B_WHH + U::core_offset(kk, j, HD)) = v;
    }
    for (int e = tid; e < G3 * C1 / 2; e += THREADS) {
        const int j = 2 * (e / C1), c = e % C1;
        const __nv_bfloat162 v{wq[OFF_WIH + j * C1 + c], wq[OFF_WIH + (j + 1) * C1 + c]};
        *reinterpret_cast<__nv_bfloat162*>(sm + B_WIH + U::core_offset(c, j, C1)) = v;
    }
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
        busy = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) U::tmem_alloc(sbase + B_BAR + 32, B_COLS);
    U::fence_smem_async();
    U::fence_before_sync();
    __syncthreads();
    U::fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    int tmax = 0;
    for (int s = 0; s < TB; ++s) tmax = max(tmax, n_s[s]);

    if (warp == EPI / 32) {  // MMAs
        if (tmax > 0) {  // the whole warp runs this, its leader issues
            constexpr uint32_t id_h = U::idesc_bf16_f32_bmn(HD, NN), id_a = U::idesc_bf16_f32_bmn(C1, NN);
            const uint32_t leader = U::elect_leader();
            const uint64_t whh = U::smem_desc(sbase + B_WHH, HD * 16, 128), wih = U::smem_desc(sbase + B_WIH, C1 * 16, 128);
            const uint64_t gop = op_desc(sbase + B_G), nop = op_desc(sbase + B_N);
            auto step_of = [](int bytes) { return (uint64_t)(bytes >> 4); };  // descriptor increment of a start address
            auto waited = [&](uint32_t bar, int parity) {
                return (bool)__all_sync(0xffffffffu, U::mbar_wait(bar, (uint32_t)(parity & 1), wait_cycles));
            };
            for (int i = 0; i < tmax; ++i) {
                if (!waited(rbar, i)) {
                    if (leader) atomicOr(status, ERR_BWD_MMA);
                    break;
                }
                U::fence_after_sync();
#pragma unroll
                for (int ks = 0; ks < G3 / 16; ++ks)
                    U::mma_bf16_warp(tmem, whh + step_of(ks * 2 * (HD * 16)), gop + step_of(ks * 2 * KG), id_h, ks, leader);
                if (leader) U::commit(hbar);
                __syncwarp();
#pragma unroll
                for (int ks = 0; ks < G3 / 16; ++ks)
                    U::mma_bf16_warp(tmem + 64, wih + step_of(ks * 2 * (C1 * 16)),
                                     ks < 2 * HD / 16 ? gop + step_of(ks * 2 * KG) : nop + step_of((ks - 2 * HD / 16) * 2 * KG),
                                     id_a, ks, leader);
                if (leader) U::commit(abar);
                __syncwarp();
            }
            if (leader) U::commit(last);  // nothing of this CTA may be in flight when it exits
            __syncwarp();
            if (!waited(last, 0) && leader) {
                atomicOr(status, ERR_HELD);
                busy = 1;
            }
        }
    } else {
        const uint32_t tl = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + 8 * half;
        int n[8];
        float dh[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            n[e] = n_s[8 * half + e];
            const int b = b_s[8 * half + e];
            dh[e] = b >= 0 ? dhl[(int64_t)b * HD + k] : 0.f;
        }
        const int64_t img_tile = w.slots * 2 * HD * 16;  // bytes between the images of two gates
        if (tmax < nt) {
            for (int g = 0; g < 4; ++g) {
                put_img(w.g_hi + g * img_tile, 2 * (u0 + nt - 1) + half, HD, k, make_uint4(0, 0, 0, 0));
                put_img(w.g_lo + g * img_tile, 2 * (u0 + nt - 1) + half, HD, k, make_uint4(0, 0, 0, 0));
            }
        }
        // this thread's cached values of a step, loaded a step ahead
        float c[5][8];
        auto load_c = [&](int t) {
            const float* cp = w.cache + (((u0 + t) * 5 * 2 + half) * HD + k) * 8;
#pragma unroll
            for (int i = 0; i < 5; ++i) {
                const float4* q = reinterpret_cast<const float4*>(cp + (int64_t)i * 2 * HD * 8);
                const float4 x = __ldg(q), y = __ldg(q + 1);
                c[i][0] = x.x; c[i][1] = x.y; c[i][2] = x.z; c[i][3] = x.w;
                c[i][4] = y.x; c[i][5] = y.y; c[i][6] = y.z; c[i][7] = y.w;
            }
        };
        // the conv gradient of step t (M = 64: rows 16 q .. 16 q + 15 in the first 16 lanes of quarter q)
        auto put_dA = [&](int t) {
            Parts pa;
            pa.load(tl + 64);
            pa.wait();
            if (lane < 16) {
                const int ch = 16 * (warp & 3) + lane;
                const int64_t g = 2 * (u0 + t) + half;
                const uint32_t on = w.a_on[g * C1 + ch];
                float v[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] = (on >> e & 1u) ? pa.sum(e) : 0.f;
                float4* q = reinterpret_cast<float4*>(w.dA + (g * C1 + ch) * 8);
                q[0] = make_float4(v[0], v[1], v[2], v[3]);
                q[1] = make_float4(v[4], v[5], v[6], v[7]);
            }
            __syncwarp();
        };
        auto waited = [&](uint32_t bar, uint32_t parity) {
            const bool ok = __all_sync(0xffffffffu, U::mbar_wait(bar, parity, wait_cycles));
            if (!ok && lane == 0) atomicOr(status, ERR_BWD_MMA);
            U::fence_after_sync();
            return ok;
        };
        float sr = 0.f, sz = 0.f, sn = 0.f, snh = 0.f;  // bias gradients
        bool ok = true;
        if (tmax > 0) load_c(tmax - 1);
        for (int t = tmax - 1; t >= 0 && ok; --t) {
            const uint32_t i = (uint32_t)(tmax - 1 - t);  // steps before this one
            float gr[8], gz[8], gn[8], gh[8], d[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const bool live = t < n[e];
                const float r = c[0][e], z = c[1][e], nn = c[2][e], g = dh[e];
                const float dn = g * (1.f - z), dz = g * (c[4][e] - nn);
                const float vn = dn * (1.f - nn * nn);
                gn[e] = live ? vn : 0.f;
                gr[e] = live ? vn * c[3][e] * r * (1.f - r) : 0.f;
                gz[e] = live ? dz * z * (1.f - z) : 0.f;
                gh[e] = live ? vn * r : 0.f;
                d[e] = live ? g * z : g;  // past its end a trajectory's dh passes through
                sr += gr[e];
                sz += gz[e];
                sn += gn[e];
                snh += gh[e];
            }
            if (t > 0) load_c(t - 1);
            uint4 hi[4], mid[4], lo[4];
            split8(gr, hi[0], mid[0], lo[0]);
            split8(gz, hi[1], mid[1], lo[1]);
            split8(gn, hi[2], mid[2], lo[2]);
            split8(gh, hi[3], mid[3], lo[3]);
            if (i > 0) {  // the previous step's dA products have read the operand
                if (!(ok = waited(abar, (i - 1) & 1))) break;
                put_dA(t + 1);
            }
            put_op(sm + B_G, k, half, hi[0], mid[0], lo[0]);
            put_op(sm + B_G, HD + k, half, hi[1], mid[1], lo[1]);
            put_op(sm + B_G, 2 * HD + k, half, hi[3], mid[3], lo[3]);
            put_op(sm + B_N, k, half, hi[2], mid[2], lo[2]);
            U::fence_smem_async();
            U::fence_before_sync();
            __syncwarp();
            if (lane == 0) U::mbar_arrive(rbar);
            // the weight gradient's images, while the products run
            const int64_t g2 = 2 * (u0 + t) + half;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                put_img(w.g_hi + g * img_tile, g2, HD, k, hi[g]);
                put_img(w.g_lo + g * img_tile, g2, HD, k, mid[g]);
            }
            if (!(ok = waited(hbar, i & 1))) break;
            Parts pd;
            pd.load(tl);
            pd.wait();
#pragma unroll
            for (int e = 0; e < 8; ++e) dh[e] = d[e] + pd.sum(e);
        }
        if (tmax > 0 && ok && waited(abar, (uint32_t)(tmax - 1) & 1)) put_dA(0);
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
        U::tmem_dealloc(tmem, B_COLS);
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
        for (int half = 0; half < 2; ++half) {
            const float4* g = reinterpret_cast<const float4*>(w.dA + ((2 * (u0 + t) + half) * C1 + c) * 8);
            const float4 g0 = __ldg(g), g1 = __ldg(g + 1);
            if (wt) {
                const float4* x = reinterpret_cast<const float4*>(xs + (t - t0 + k) * CB_U + i * CB_I + 8 * half);
                const float4 x0 = x[0], x1 = x[1];
                acc = fmaf(g0.x, x0.x, fmaf(g0.y, x0.y, fmaf(g0.z, x0.z, fmaf(g0.w, x0.w, acc))));
                acc = fmaf(g1.x, x1.x, fmaf(g1.y, x1.y, fmaf(g1.z, x1.z, fmaf(g1.w, x1.w, acc))));
            } else {
                acc += ((g0.x + g0.y) + (g0.z + g0.w)) + ((g1.x + g1.y) + (g1.z + g1.w));
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
    x.a_hi = take(groups * C1 * 16);
    x.a_lo = take(groups * C1 * 16);
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
