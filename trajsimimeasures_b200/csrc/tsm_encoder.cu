// Learned candidate filter: a trajectory encoder trained on DTW distances.
//
// Network (per trajectory of n points, coordinates normalised on the host):
//   conv   a_t = relu(b1 + sum_{k<5, i<2} W1[c][i][k] x_{t+k-2,i})   64 channels, zero padding
//   GRU    r = s(Wir a + bir + Whr h + bhr),  z = s(Wiz a + biz + Whz h + bhz),
//          n = tanh(Win a + bin + r * (Whn h + bhn)),  h' = (1-z) n + z h      hidden 128
//   head   e = [Wo h_n + bo | sc_k * r_k]                                       160-d embedding
//          r_k = point round(k (n - 1) / 15) of the trajectory, k < 16, normalised (32 values):
//          a geometric skip around the recurrent branch, with a learned weight sc_k = exp(u_k)
//          per point (u_k stored: Adam then moves the weights by relative steps)
//   pair   d(a, b) = ||e_a - e_b||_2, trained with MSE against DTW / max DTW.
// Conv and GRU weights are used as BF16 values (rounded from FP32 master
// weights before each forward), all accumulation is FP32; the head and the
// skip are FP32 (a BF16 path cannot hold positions to the ~1e-4 of the box
// that separates DTW neighbours among a million trajectories; the skip
// carries them exactly).
// The reference trains its learned measures the same way (MSE on
// distance / max distance, nn/MLP_trajsimi_train.py:74-84,197-200).
//
// Training runs on the tensor cores with FP32-accurate activations (three BF16
// parts, tsm_train.cu; weight gradients tsm_wgrad.cu).  Inference (embedding a
// database or a query batch) takes a_t and h_t as BF16: enc_gru_embed_tc, 128
// trajectories per CTA, each step's products (128 x 384 x 192) tcgen05 MMA
// tiles with the accumulators in tensor memory.
//
//   enc_round_bf16    FP32 master -> BF16 weights
//   train_forward     conv + GRU over time, with the values BPTT needs (tsm_train.cu)
//   enc_head_fwd      e = [Wo h_last + bo | sc_k r_k]
//   enc_pair_loss     distances, MSE loss, dL/de (atomic)
//   enc_head_bwd      dWo, dbo, dh_last; enc_skip_bwd: d sc_k
//   train_backward    BPTT, GRU and conv gradients (tsm_train.cu, tsm_wgrad.cu)
//   enc_adam          Adam step on the FP32 master weights
//   enc_conv_fwd_tc   conv + relu -> BF16 a_t operand images for the tensor-core GRU
//   enc_gru_embed_tc  inference GRU on the tensor cores -> last hidden state
#include <cuda_bf16.h>
#include <cstdio>
#include <cuda_runtime.h>
#include <stdint.h>

#include "tsm.h"
#include "tsm_enc.cuh"
#include "tsm_train.h"
#include "tsm_umma.cuh"

int tsm_internal_fail(int code, const char* msg);

namespace enc {

static_assert(SK == 32, "enc_skip_bwd maps one skip value per lane");

// FP32 master -> BF16 copies of the conv and GRU weights (head stays FP32).
__global__ void enc_round_bf16(const float* __restrict__ p, __nv_bfloat16* __restrict__ q) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < OFF_WO) q[i] = __float2bfloat16_rn(p[i]);
}

// Point index of resampled point k (0 <= k < NS) of a trajectory of n >= 1
// points: round(k (n - 1) / (NS - 1)), halves rounded up, in integers.
__device__ __forceinline__ int skip_index(int k, int n) { return (2 * k * (n - 1) + (NS - 1)) / (2 * (NS - 1)); }

// E[b][EO + 2 k + i] = sc_k * coordinate i of resampled point k (the
// normalised input at skip_index(k, n); 0 for an empty trajectory), the
// geometric skip, written unscaled to X[b][2 k + i] too when X is given (the
// training forward keeps it for the gradients of sc_k).  One thread per value:
// each is a chain of three loads, which inside the head's few CTAs cost 28 us.
__global__ void __launch_bounds__(256) enc_skip_fwd(int B, const float* __restrict__ p, float* __restrict__ E,
                                                    const float2* __restrict__ pts, const int64_t* __restrict__ off,
                                                    const int32_t* __restrict__ len, float4 nrm, float* __restrict__ X) {
    const int64_t g = (int64_t)blockIdx.x * 256 + threadIdx.x;
    const int64_t b = g / SK;
    const int q = g % SK;
    if (b >= B) return;
    const int n = len[b];
    const float x = n > 0 ? xin(pts, off[b], n, skip_index(q >> 1, n), q & 1, nrm) : 0.f;
    E[b * ED + EO + q] = expf(p[OFF_SC + (q >> 1)]) * x;
    if (X) X[b * SK + q] = x;
}

// E[b][o] = bo[o] + sum_k Wo[o][k] hl[b][k] (bias first, k ascending) for o <
// EO.  A CTA keeps W_o transposed in shared memory and takes blocks of HEAD_B
// trajectories in turn, their hidden states staged there too: lane l outputs l,
// l + 32, l + 64, l + 96 of its warp's HEAD_R trajectories, so that a 16-byte
// load of hidden states (4 clocks, broadcast or not) feeds 16 FMAs.  (One
// output a thread, W_o rows read from global memory, 32 lines a load: 0.33 ms
// for 100,000 trajectories.)
constexpr int HEAD_R = 16;
constexpr int HEAD_B = 4 * HEAD_R;
constexpr int HEAD_LD = EO + 1;  // row stride of the transposed W_o: no bank conflicts either way
constexpr int HEAD_SMEM = (HEAD_B * HD + HD * HEAD_LD) * 4;
__global__ void __launch_bounds__(EO) enc_head_fwd(const float* __restrict__ hl, int B, const float* __restrict__ p,
                                                   float* __restrict__ E) {
    extern __shared__ __align__(16) float head_sm[];
    float* hs = head_sm;                 // [HEAD_B][HD]
    float* wt = head_sm + HEAD_B * HD;   // [HD][HEAD_LD]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll 8
    for (int r = 0; r < EO; ++r) wt[tid * HEAD_LD + r] = __ldg(p + OFF_WO + r * HD + tid);
    float bo[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) bo[i] = p[OFF_BO + lane + 32 * i];
    for (int64_t b0 = (int64_t)blockIdx.x * HEAD_B; b0 < B; b0 += (int64_t)gridDim.x * HEAD_B) {
        __syncthreads();  // W_o is staged; the last block's readers are done
#pragma unroll 8
        for (int e = tid; e < HEAD_B * HD; e += EO) {
            const int64_t b = b0 + e / HD;
            hs[e] = b < B ? hl[b * HD + e % HD] : 0.f;
        }
        __syncthreads();
        float acc[4][HEAD_R];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < HEAD_R; ++j) acc[i][j] = bo[i];
        const float* hw = hs + warp * HEAD_R * HD;
        for (int k = 0; k < HD; k += 4) {
            float w[4][4];
#pragma unroll
            for (int d = 0; d < 4; ++d)
#pragma unroll
                for (int i = 0; i < 4; ++i) w[i][d] = wt[(k + d) * HEAD_LD + lane + 32 * i];
#pragma unroll
            for (int j = 0; j < HEAD_R; ++j) {
                const float4 h = *reinterpret_cast<const float4*>(hw + j * HD + k);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    acc[i][j] = fmaf(w[i][3], h.w, fmaf(w[i][2], h.z, fmaf(w[i][1], h.y, fmaf(w[i][0], h.x, acc[i][j]))));
            }
        }
#pragma unroll
        for (int j = 0; j < HEAD_R; ++j) {
            const int64_t b = b0 + warp * HEAD_R + j;
            if (b < B)
#pragma unroll
                for (int i = 0; i < 4; ++i) E[b * ED + lane + 32 * i] = acc[i][j];
        }
    }
}

// One warp per pair: pred = ||E[ia]-E[ib]|| (all ED embedding values), loss += w (pred-y)^2 / P,
// dE[ia] += 2 w (pred-y)/P * (E[ia]-E[ib])/pred, dE[ib] -= the same; w = wt[p] (1 without weights).
__global__ void enc_pair_loss(const float* __restrict__ E, const int32_t* __restrict__ ia,
                              const int32_t* __restrict__ ib, const float* __restrict__ y,
                              const float* __restrict__ wt, int P, float* __restrict__ pred,
                              float* __restrict__ loss, float* __restrict__ dE) {
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= P) return;
    const float* ea = E + (int64_t)ia[w] * ED;
    const float* eb = E + (int64_t)ib[w] * ED;
    float d[ED / 32];
    float ss = 0.f;
#pragma unroll
    for (int q = 0; q < ED / 32; ++q) {
        d[q] = ea[lane + 32 * q] - eb[lane + 32 * q];
        ss = fmaf(d[q], d[q], ss);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float pr = sqrtf(ss);
    const float err = pr - y[w];
    const float wp = wt ? wt[w] : 1.f;
    if (lane == 0) {
        pred[w] = pr;
        if (loss) atomicAdd(loss, wp * err * err / P);
    }
    if (dE && pr > 0.f) {
        const float g = 2.f * wp * err / (P * pr);
#pragma unroll
        for (int q = 0; q < ED / 32; ++q) {
            atomicAdd(dE + (int64_t)ia[w] * ED + lane + 32 * q, g * d[q]);
            atomicAdd(dE + (int64_t)ib[w] * ED + lane + 32 * q, -g * d[q]);
        }
    }
}

// dWo[o][k] += sum_b dE[b][o] hl[b][k]; dbo[o] += sum_b dE[b][o];
// dhl[b][k] = sum_o Wo[o][k] dE[b][o].
// (One CTA per output and HB_B trajectories, added with atomics: with one CTA
// per output the sum over a batch was a chain of 2,048 dependent loads, 0.21 ms.)
constexpr int HB_B = 128;
__global__ void enc_head_bwd_w(const float* __restrict__ dE, const float* __restrict__ hl, int B,
                               float* __restrict__ grad) {
    const int o = blockIdx.x;  // EO blocks
    const int k = threadIdx.x; // 128 threads
    float acc = 0.f, accb = 0.f;
    const int b1 = min(B, ((int)blockIdx.y + 1) * HB_B);
#pragma unroll 8
    for (int b = blockIdx.y * HB_B; b < b1; ++b) {
        const float g = dE[(int64_t)b * ED + o];
        acc = fmaf(g, hl[(int64_t)b * HD + k], acc);
        accb += g;
    }
    atomicAdd(grad + OFF_WO + o * HD + k, acc);
    if (k == 0) atomicAdd(grad + OFF_BO + o, accb);
}

__global__ void enc_head_bwd_h(const float* __restrict__ dE, int B, const float* __restrict__ p, float* __restrict__ dhl) {
    const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= (int64_t)B * HD) return;
    const int k = gid % HD;
    const int64_t b = gid / HD;
    float acc = 0.f;
    for (int o = 0; o < EO; ++o) acc = fmaf(p[OFF_WO + o * HD + k], dE[b * ED + o], acc);
    dhl[gid] = acc;
}

// d u_k += sc_k sum_b sum_i dE[b][EO + 2k + i] X[b][2k + i] (the gradients of
// the skip's log-weights, sc_k = exp(u_k)).  Lane q of every warp takes skip value q of the warp's
// trajectories (blockDim a multiple of 32 = SK); lanes 2k and 2k + 1 are summed
// before one atomic per point and warp.
__global__ void enc_skip_bwd(const float* __restrict__ dE, const float* __restrict__ X, int B,
                             const float* __restrict__ p, float* __restrict__ grad) {
    const int q = threadIdx.x & (SK - 1);
    const int64_t wid = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / SK;
    const int64_t nw = (int64_t)gridDim.x * blockDim.x / SK;
    float acc = 0.f;
    for (int64_t b = wid; b < B; b += nw) acc = fmaf(dE[b * ED + EO + q], X[b * SK + q], acc);
    acc += __shfl_xor_sync(0xffffffffu, acc, 1);
    if ((q & 1) == 0) atomicAdd(grad + OFF_SC + (q >> 1), expf(p[OFF_SC + (q >> 1)]) * acc);
}

__global__ void enc_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                         float* __restrict__ v, int n, float lr, float b1, float b2, float eps, float bc1, float bc2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
}

// ---------------------------------------------------------------------------
// Tensor-core GRU forward for inference (tcgen05).  CTA = 128 trajectories
// (the MMA's M); per time step the operand [a_t | h_t] (128 x 192 BF16, shared
// memory) is multiplied by the BF16 gate weights, resident in shared memory for
// all steps, into FP32 accumulators in tensor memory (all 512 columns).  (n
// needs Whn h apart from Win a: r multiplies only the hidden part.)
//
// The hidden units go in two halves of 64, each with accumulators of its own
// (256 columns: Win a | r | z | Whn h), so that the tensor cores and the gate
// math overlap although a step needs all of the step before: while the gates
// of half 0 are computed the products of half 1 run, and under the gates of
// half 1 the next step's products of half 0 with a and with the new h of half
// 0.  Only the products of half 0 with the h of half 1 wait for the whole step.
// h of half 0 has two buffers (half 1's products of step t read it while step
// t + 1's is written), h of half 1 one.
//
// Threads: a ninth warp issues copies and MMAs (one elected lane); eight warps
// do the gates, warp w the tensor-memory lanes (trajectories) 32 (w % 4) .. +31
// and 32 of a half's 64 units, with the biases in FP32, h in FP32 registers and
// written back to shared memory as BF16.  The a_t part comes from
// enc_conv_fwd_tc as one 16 KB BF16 image per step already in the operand
// layout, bulk-copied a step ahead into the other of two buffers.  a_t and h_t enter the products as BF16
// (the training kernels multiply FP32 a and h by the BF16 weights) and the
// gates use the hardware tanh, so the embeddings agree with the training
// forward to BF16 rounding of the activations.
//
// What bounds it: the gate math.  The hardware tanh, three a unit at 16 a clock
// and SM, takes 3,072 clocks a step; measured 5,100 with the six biases a unit
// (shared-memory loads of 16 bytes, which take 4 clocks though broadcast; without
// them 3,300), 900 for the tensor-memory loads, 700 for writing h back, 1,000
// waiting for the first products: 7,700 a step against 12,500 when products and
// gates took turns.  100,000 trajectories of 20..200 points in three launches:
// 3.76 -> 2.33 ms.  Sixteen gate warps of 16 units spill (96 registers): 8,000.
// The two biases of a gate are added one after the other: their sum would save
// a quarter of the loads but round differently, and a BF16 rounding of h that
// flips shows as 6e-4 of the embedding's size.
constexpr int TC_M = 128;
constexpr int TC_EPI = 256;                                 // gate threads: two warps per 32-lane quarter of tensor memory
constexpr int TC_THREADS = TC_EPI + 32;
constexpr int TC_HH = HD / 2;                               // hidden units of a half
constexpr int TC_HU = TC_HH / (TC_EPI / 128);               // of them per thread (32)
constexpr int TC_N = 3 * TC_HH;                             // MMA N: 192
constexpr int TC_A_BYTES = TC_M * C1 * 2;                   // one a_t image: 16 KB
constexpr int TC_H_BYTES = TC_M * TC_HH * 2;                // one half of h: 16 KB
constexpr int TC_WA_BYTES = TC_N * C1 * 2;                  // a half's weights of a: rows Win | Wir | Wiz, 24 KB
constexpr int TC_WH_BYTES = TC_N * HD * 2;                  // of h: rows Whr | Whz | Whn, 48 KB
constexpr int TC_OFF_A = 0;                                 // a-buffers [128][64] BF16
constexpr int TC_OFF_H = TC_OFF_A + 2 * TC_A_BYTES;         // h: half 0 (two buffers), half 1
constexpr int TC_OFF_WA = TC_OFF_H + 3 * TC_H_BYTES;
constexpr int TC_OFF_WH = TC_OFF_WA + 2 * TC_WA_BYTES;
constexpr int TC_OFF_BIAS = TC_OFF_WH + 2 * TC_WH_BYTES;    // float b_ir, b_hr, b_iz, b_hz, b_in [128], b_hn [112]
constexpr int TC_OFF_BAR = TC_OFF_BIAS + (6 * HD - 16) * 4;        // mbarriers; tensor-memory address
constexpr int TC_SMEM = TC_OFF_BAR + 64;
static_assert(TC_SMEM <= 227 * 1024, "enc_gru_embed_tc shared memory");
constexpr uint32_t TC_TMEM_COLS = 512;
// a wait for the tensor cores or a copy longer than this many SM clocks (~1 s) is an error
constexpr long long TC_WAIT_CYCLES = 2000000000LL;

// Gate nonlinearities of the inference kernel: the hardware tanh (MUFU,
// about 2^-11 relative error, the size of the BF16 rounding the operands
// already carry) and sigma(x) = (1 + tanh(x / 2)) / 2, one MUFU operation each.
__device__ __forceinline__ float tanh_hw(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float sigm_hw(float x) { return fmaf(0.5f, tanh_hw(0.5f * x), 0.5f); }

// Eight BF16 values as one 16-byte store.
__device__ __forceinline__ uint4 pack8_bf16(const float* v) {
    uint4 u;
    u.x = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v[0])) |
          ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v[1])) << 16);
    u.y = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v[2])) |
          ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v[3])) << 16);
    u.z = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v[4])) |
          ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v[5])) << 16);
    u.w = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v[6])) |
          ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v[7])) << 16);
    return u;
}

// Conv output for the tensor-core GRU (same arithmetic as train_conv, then
// rounded to BF16): for block g of 128 trajectories and step t, the 16 KB
// image of the a_t operand (rows = trajectories, k = channels, core-matrix
// layout) at Ab + (g * T + t) * 128 * 64.  Rows past B and steps past a
// trajectory's length are zero.  One thread per (trajectory, CT steps), all 64
// channels: a channel's ten weights (shared memory, 16-byte loads) serve CT
// steps (with one step a thread and a load per weight the images of 100,000
// trajectories of 20..200 steps took 0.75 ms, with four 0.66, with eight 0.79:
// at 1.8 GB written it is near what plain writes reach).  Consecutive threads take
// consecutive rows of one image, so a warp's 16-byte stores are contiguous.
// Bp = B rounded up to a multiple of 128; blockDim = 256.
constexpr int CT = 4;
__global__ void __launch_bounds__(256) enc_conv_fwd_tc(const float2* __restrict__ pts, const int64_t* __restrict__ off,
                                                       const int32_t* __restrict__ len, int B, int Bp, int T,
                                                       float4 nrm, const __nv_bfloat16* __restrict__ wq,
                                                       const float* __restrict__ p, __nv_bfloat16* __restrict__ Ab) {
    __shared__ __align__(16) float w1[C1][12];  // the ten weights of a channel, its bias
    for (int e = threadIdx.x; e < C1 * 2 * KW; e += blockDim.x) {
        const int c = e / (2 * KW), i = e / KW % 2, k = e % KW;
        w1[c][2 * k + i] = __bfloat162float(wq[OFF_W1 + e]);
    }
    for (int e = threadIdx.x; e < C1; e += blockDim.x) w1[e][2 * KW] = p[OFF_B1 + e];
    __syncthreads();
    const int tq = (T + CT - 1) / CT;
    const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= (int64_t)Bp * tq) return;
    const int row = gid % TC_M;
    const int t0 = (int)(gid / TC_M % tq) * CT;
    const int g = (int)(gid / ((int64_t)TC_M * tq));
    const int b = g * TC_M + row;
    const int n = b < B ? len[b] : 0;
    float x[KW - 1 + CT][2];  // the window's normalised points
    if (t0 < n) {
        const int64_t o = off[b];
#pragma unroll
        for (int k = 0; k < KW - 1 + CT; ++k)
#pragma unroll
            for (int i = 0; i < 2; ++i) x[k][i] = xin(pts, o, n, t0 + k - 2, i, nrm);
    }
    unsigned char* img = reinterpret_cast<unsigned char*>(Ab + ((int64_t)g * T + t0) * (TC_M * C1));
#pragma unroll 1
    for (int c8 = 0; c8 < C1 / 8; ++c8) {
        float a[CT][8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float4* w4 = reinterpret_cast<const float4*>(w1[8 * c8 + q]);
            const float4 wa = w4[0], wb = w4[1], wc = w4[2];
            const float w[2 * KW] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w, wc.x, wc.y};
#pragma unroll
            for (int d = 0; d < CT; ++d) {
                float v = 0.f;
                if (t0 + d < n) {
                    float acc = wc.z;
#pragma unroll
                    for (int k = 0; k < KW; ++k)
#pragma unroll
                        for (int i = 0; i < 2; ++i) acc = fmaf(w[2 * k + i], x[d + k][i], acc);
                    v = fmaxf(acc, 0.f);
                }
                a[d][q] = v;
            }
        }
#pragma unroll
        for (int d = 0; d < CT; ++d)
            if (t0 + d < T)
                *reinterpret_cast<uint4*>(img + (int64_t)d * (TC_M * C1 * 2) + tsm::umma::core_offset(row, 8 * c8, TC_M)) =
                    pack8_bf16(a[d]);
    }
}

// Bits of the embedding status word (the first word of the embed workspace).
constexpr int TC_ERR_COPY = 1;      // an a_t copy did not land within the wait limit (no MMA issued for it)
constexpr int TC_ERR_MMA = 2;       // the MMAs of a step did not complete within the wait limit
constexpr int TC_ERR_TMEM_HELD = 4; // ... nor within a second limit: the CTA exited without freeing tensor memory

// hl[b][128] = h after the last valid step of trajectory b.  Ab: the a_t
// images of enc_conv_fwd_tc (T steps per block of 128).  wq: BF16 weights; p:
// FP32 parameters (biases).  If the tensor cores or a copy do not complete
// within wait_cycles, the CTA ORs a TC_ERR_* bit into *status, writes NaN to
// its rows of hl and stops: after waiting (bounded) for its copy in flight,
// and, if MMAs of the failed step were issued, once more for them; tensor
// memory is freed only when no MMA can still write it.  stall_step >= 0 is a
// test hook: the a_t copy of that step is announced on its mbarrier but never
// issued, so that its wait runs out with no MMA in flight (-1 in normal use).
__global__ void __launch_bounds__(TC_THREADS, 1) enc_gru_embed_tc(const __nv_bfloat16* __restrict__ Ab,
                                                                   const int32_t* __restrict__ len, int B, int T,
                                                                   const __nv_bfloat16* __restrict__ wq,
                                                                   const float* __restrict__ p,
                                                                   float* __restrict__ hl, int* __restrict__ status,
                                                                   long long wait_cycles, int stall_step) {
    namespace U = tsm::umma;
    extern __shared__ __align__(1024) unsigned char sm[];
    // (no static shared memory: the dynamic part, aligned to 1 KB, would start behind it and not fit)
    // the CTA's steps; once all have read them, -1: MMAs may still write tensor memory
    volatile int& steps = *reinterpret_cast<volatile int*>(sm + TC_OFF_BAR + 60);
    float* bias = reinterpret_cast<float*>(sm + TC_OFF_BIAS);
    const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(sm));
    // mbarriers: products of half p done, h of half p written, a-buffer i landed, the last products done
    const uint32_t bar = sbase + TC_OFF_BAR;
    auto dbar = [&](int p) { return bar + 8 * p; };
    auto ebar = [&](int p) { return bar + 16 + 8 * p; };
    auto abar = [&](int i) { return bar + 32 + 8 * i; };
    const uint32_t last = bar + 48;
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(sm + TC_OFF_BAR + 56);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int blk = gridDim.x - 1 - blockIdx.x;  // the last block, the longest of a batch in length order, first
    const __nv_bfloat16* img = Ab + (int64_t)blk * T * (TC_M * C1);  // this block's a_t images

    if (tid == 0) steps = 0;
    // weights -> core-matrix layout (16-byte chunks of 8 consecutive k); operand row 64 g + i of half q is unit
    // 64 q + i of the g-th gate of its list (gate rows r 0..127, z 128..255, n 256..383)
    for (int e = tid; e < 2 * TC_N * (C1 / 8); e += TC_THREADS) {  // a: n, r, z
        const int c = e % (C1 / 8), r = e / (C1 / 8) % TC_N, q = e / (TC_N * (C1 / 8)), g = r / TC_HH;
        const int row = (g == 0 ? 2 : g - 1) * HD + TC_HH * q + r % TC_HH;
        *reinterpret_cast<uint4*>(sm + TC_OFF_WA + q * TC_WA_BYTES + U::core_offset(r, 8 * c, TC_N)) =
            *reinterpret_cast<const uint4*>(wq + OFF_WIH + row * C1 + 8 * c);
    }
    for (int e = tid; e < 2 * TC_N * (HD / 8); e += TC_THREADS) {  // h: r, z, n
        const int c = e % (HD / 8), r = e / (HD / 8) % TC_N, q = e / (TC_N * (HD / 8)), g = r / TC_HH;
        const int row = g * HD + TC_HH * q + r % TC_HH;
        *reinterpret_cast<uint4*>(sm + TC_OFF_WH + q * TC_WH_BYTES + U::core_offset(r, 8 * c, TC_N)) =
            *reinterpret_cast<const uint4*>(wq + OFF_WHH + row * HD + 8 * c);
    }
    for (int e = tid; e < HD; e += TC_THREADS) {
        bias[e] = p[OFF_BIH + e];
        bias[HD + e] = p[OFF_BHH + e];
        bias[2 * HD + e] = p[OFF_BIH + HD + e];
        bias[3 * HD + e] = p[OFF_BHH + HD + e];
        bias[4 * HD + e] = p[OFF_BIH + 2 * HD + e];
        if (e < HD - 16) bias[5 * HD + e] = p[OFF_BHH + 2 * HD + e];  // (the last 16 do not fit: registers)
    }
    for (int e = tid; e < 3 * TC_H_BYTES / 16; e += TC_THREADS)  // h_0 = 0
        *reinterpret_cast<uint4*>(sm + TC_OFF_H + 16 * e) = make_uint4(0, 0, 0, 0);
    if (tid == 0) {
        for (int q = 0; q < 2; ++q) {
            U::mbar_init(dbar(q), 1);
            U::mbar_init(ebar(q), TC_EPI / 32);
            U::mbar_init(abar(q), 1);
        }
        U::mbar_init(last, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) U::tmem_alloc(sbase + TC_OFF_BAR + 56, TC_TMEM_COLS);
    U::fence_smem_async();
    U::fence_before_sync();
    __syncthreads();
    U::fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    if (tid < TC_M && blk * TC_M + tid < B) atomicMax(const_cast<int*>(&steps), min(len[blk * TC_M + tid], T));
    __syncthreads();
    const int tmax = steps;

    if (warp == TC_EPI / 32) {
        if (tmax > 0) {  // the whole warp runs this, its leader issues
            constexpr uint32_t kLBO = TC_M * 16, kWL = TC_N * 16;  // K-chunk strides of the operands
            constexpr uint32_t id3 = U::idesc_bf16_f32(TC_M, TC_N), id2 = U::idesc_bf16_f32(TC_M, 2 * TC_HH),
                               id1 = U::idesc_bf16_f32(TC_M, TC_HH);
            const uint32_t leader = U::elect_leader();
            auto step_of = [](int bytes) { return (uint64_t)(bytes >> 4); };  // descriptor increment of a start address
            const uint64_t a_desc = U::smem_desc(sbase + TC_OFF_A, kLBO, 128), h_desc = U::smem_desc(sbase + TC_OFF_H, kLBO, 128);
            const uint64_t wa = U::smem_desc(sbase + TC_OFF_WA, kWL, 128), wh = U::smem_desc(sbase + TC_OFF_WH, kWL, 128);
            auto waited = [&](uint32_t b, int use) {
                return (bool)__all_sync(0xffffffffu, U::mbar_wait(b, (uint32_t)(use & 1), wait_cycles));
            };
            int loaded = 0;
            auto load_a = [&](int t) {
                if (leader) {
                    U::mbar_arrive_expect_tx(abar(t & 1), TC_A_BYTES);
                    if (t != stall_step)
                        U::bulk_load(sbase + TC_OFF_A + (t & 1) * TC_A_BYTES, img + (int64_t)t * (TC_M * C1), TC_A_BYTES,
                                     abar(t & 1));
                }
                __syncwarp();
                loaded = t + 1;
            };
            auto a_products = [&](int t, int q) {
                const uint64_t a = a_desc + step_of((t & 1) * TC_A_BYTES), w = wa + step_of(q * TC_WA_BYTES);
#pragma unroll
                for (int ks = 0; ks < C1 / 16; ++ks)
                    U::mma_bf16_warp(tmem + 256 * q, a + step_of(ks * 2 * kLBO), w + step_of(ks * 2 * kWL), id3, ks, leader);
            };
            auto h_products = [&](int t, int q, int part) {  // part: half of h
                const uint64_t h = h_desc + step_of((part ? 2 : (t & 1)) * TC_H_BYTES);
                const uint64_t w = wh + step_of(q * TC_WH_BYTES + part * (TC_HH / 8) * kWL);
#pragma unroll
                for (int ks = 0; ks < TC_HH / 16; ++ks) {
                    const uint64_t hk = h + step_of(ks * 2 * kLBO), wk = w + step_of(ks * 2 * kWL);
                    if (part == 0 && ks == 0) {  // Whn h starts here; r and z go on from the products with a
                        U::mma_bf16_warp(tmem + 256 * q + TC_HH, hk, wk, id2, 1u, leader);
                        U::mma_bf16_warp(tmem + 256 * q + 3 * TC_HH, hk, wk + step_of(2 * TC_HH * 16), id1, 0u, leader);
                    } else {
                        U::mma_bf16_warp(tmem + 256 * q + TC_HH, hk, wk, id3, 1u, leader);
                    }
                }
            };
            int err = 0;
            load_a(0);
            for (int t = 0; t < tmax && !err; ++t) {
                if (!waited(abar(t & 1), t >> 1)) {
                    err = TC_ERR_COPY;
                    break;
                }
                if (t > 0 && !waited(ebar(0), t - 1)) {
                    err = TC_ERR_MMA;
                    break;
                }
                U::fence_after_sync();
                a_products(t, 0);
                h_products(t, 0, 0);
                if (t > 0 && !waited(ebar(1), t - 1)) {
                    err = TC_ERR_MMA;
                    break;
                }
                U::fence_after_sync();
                h_products(t, 0, 1);
                if (leader) U::commit(dbar(0));
                __syncwarp();
                if (t + 1 < tmax) load_a(t + 1);  // its buffer's readers, step t - 1, are done
                a_products(t, 1);
                h_products(t, 1, 0);
                h_products(t, 1, 1);
                if (leader) U::commit(dbar(1));
                __syncwarp();
            }
            // nothing of this CTA may be in flight when it exits
            if (err) {
                if (leader) atomicOr(status, err);
                for (int i = max(0, loaded - 2); i < loaded; ++i)
                    if (i != stall_step) waited(abar(i & 1), i >> 1);
            }
            if (leader) U::commit(last);
            __syncwarp();
            if (!waited(last, 0) && leader) {
                atomicOr(status, TC_ERR_TMEM_HELD);
                steps = -1;
            }
        }
    } else {
        const int row = 32 * (warp & 3) + lane;  // this thread's trajectory (tensor-memory lane)
        const int sub = warp >> 2;               // units TC_HU sub .. +TC_HU-1 of each half
        const int b = blk * TC_M + row;
        const int n = b < B ? len[b] : 0;
        const uint32_t tl = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
        float h[2 * TC_HU], tail[16];
#pragma unroll
        for (int i = 0; i < 2 * TC_HU; ++i) h[i] = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) tail[i] = __ldg(p + OFF_BHH + 3 * HD - 16 + i);
        bool failed = false;
        for (int t = 0; t < tmax && !failed; ++t) {
            const bool live = t < n;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                if (!__all_sync(0xffffffffu, U::mbar_wait(dbar(q), (uint32_t)(t & 1), wait_cycles))) {
                    if (lane == 0) atomicOr(status, TC_ERR_MMA);
                    failed = true;
                    break;
                }
                U::fence_after_sync();
                __syncwarp();
                unsigned char* H = sm + TC_OFF_H + (q ? 2 : ((t + 1) & 1)) * TC_H_BYTES;
#pragma unroll
                for (int c = 0; c < TC_HU / 16; ++c) {  // 16 hidden units at a time
                    const int u0 = TC_HU * sub + 16 * c, k0 = TC_HH * q + u0;
                    uint32_t rr[16], zz[16], ii[16], hh[16];
                    U::ld16(tl + 256 * q + u0, ii);
                    U::ld16(tl + 256 * q + TC_HH + u0, rr);
                    U::ld16(tl + 256 * q + 2 * TC_HH + u0, zz);
                    U::ld16(tl + 256 * q + 3 * TC_HH + u0, hh);
                    U::wait_ld(ii);
                    U::wait_ld(rr);
                    U::wait_ld(zz);
                    U::wait_ld(hh);
                    float hv[16];
#pragma unroll
                    for (int j4 = 0; j4 < 16; j4 += 4) {
                        auto b4 = [&](int a) { return *reinterpret_cast<const float4*>(bias + a * HD + k0 + j4); };
                        // the two biases of a gate are added one after the other
                        const float4 r1 = b4(0), r2 = b4(1), z1 = b4(2), z2 = b4(3), bi = b4(4);
                        const bool in_regs = q == 1 && c == TC_HU / 16 - 1;  // the last 16 units of the last warps
                        float4 bh = make_float4(tail[j4], tail[j4 + 1], tail[j4 + 2], tail[j4 + 3]);
                        if (!in_regs || sub == 0) bh = b4(5);
                        const float xr1[4] = {r1.x, r1.y, r1.z, r1.w}, xr2[4] = {r2.x, r2.y, r2.z, r2.w};
                        const float xz1[4] = {z1.x, z1.y, z1.z, z1.w}, xz2[4] = {z2.x, z2.y, z2.z, z2.w};
                        const float xi[4] = {bi.x, bi.y, bi.z, bi.w}, xh[4] = {bh.x, bh.y, bh.z, bh.w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int j = j4 + e;
                            const float r = sigm_hw(__uint_as_float(rr[j]) + xr1[e] + xr2[e]);
                            const float z = sigm_hw(__uint_as_float(zz[j]) + xz1[e] + xz2[e]);
                            const float nn = tanh_hw(__uint_as_float(ii[j]) + xi[e] + r * (__uint_as_float(hh[j]) + xh[e]));
                            const float hp = h[TC_HU * q + 16 * c + j];
                            hv[j] = live ? (1.f - z) * nn + z * hp : hp;
                            h[TC_HU * q + 16 * c + j] = hv[j];
                        }
                    }
                    *reinterpret_cast<uint4*>(H + U::core_offset(row, u0, TC_M)) = pack8_bf16(hv);
                    *reinterpret_cast<uint4*>(H + U::core_offset(row, u0 + 8, TC_M)) = pack8_bf16(hv + 8);
                }
                U::fence_smem_async();
                U::fence_before_sync();
                __syncwarp();
                if (lane == 0) U::mbar_arrive(ebar(q));
            }
        }
        if (b < B) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                float* dst = hl + (int64_t)b * HD + TC_HH * q + TC_HU * sub;
#pragma unroll
                for (int i = 0; i < TC_HU; ++i) dst[i] = failed ? __int_as_float(0x7fc00000) : h[TC_HU * q + i];
            }
        }
    }
    U::fence_before_sync();
    __syncthreads();
    if (warp == 0 && steps >= 0) {
        U::fence_after_sync();
        U::tmem_dealloc(tmem, TC_TMEM_COLS);
    }
}

}  // namespace enc

// ---------------------------------------------------------------------------
// Host orchestration (C ABI, declared in include/tsm.h)
// ---------------------------------------------------------------------------
namespace {

struct EncWs {  // views into the caller's workspace
    int* status;  // first word: bits OR-ed in by the tensor-core weight-gradient kernel (zeroed by the caller)
    float *hl, *E, *dE, *dhl, *pred, *loss, *X;
    __nv_bfloat16* wq;
    enc::TrainWs tr;  // the recurrences' buffers (tsm_train.cu)
};

int64_t align64(int64_t n) { return (n + 63) & ~int64_t(63); }

// Lays the workspace out (base != NULL) and returns its size in floats.
int64_t ws_layout(int B, int T, int P, float* base, EncWs* w) {
    int64_t o = 0;
    auto take = [&](float** dst, int64_t n) {
        if (base) *dst = base + o;
        o += align64(n);
    };
    EncWs tmp;
    EncWs* x = w ? w : &tmp;
    float* st = nullptr;
    take(&st, 1);
    if (base) x->status = reinterpret_cast<int*>(st);
    take(&x->hl, (int64_t)B * enc::HD);
    take(&x->E, (int64_t)B * enc::ED);
    take(&x->dE, (int64_t)B * enc::ED);
    take(&x->dhl, (int64_t)B * enc::HD);
    take(&x->X, (int64_t)B * enc::SK);
    take(&x->pred, P > 0 ? P : 1);
    take(&x->loss, 1);
    float* wqf = nullptr;
    take(&wqf, (enc::N_PARAMS + 1) / 2);  // BF16 copy of the weights
    if (base) x->wq = reinterpret_cast<__nv_bfloat16*>(wqf);
    // (align64 keeps every buffer on a 256-byte boundary)
    o += align64((enc::train_layout(B, T, base ? reinterpret_cast<unsigned char*>(base + o) : nullptr, &x->tr) + 3) / 4);
    return o;
}

int enc_check(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return TSM_OK;
    char b[256];
    snprintf(b, sizeof(b), "%s: %s", what, cudaGetErrorString(e));
    return tsm_internal_fail(TSM_ECUDA, b);
}

// The head over B trajectories: at most two CTAs per SM, each over blocks of HEAD_B.
int enc_head(const float* hl, int B, const float* params, float* E, const float2* pts, const int64_t* off,
             const int32_t* len, float4 n4, float* X, cudaStream_t s) {
    using namespace enc;
    int rc = enc_check(cudaFuncSetAttribute(enc_head_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, HEAD_SMEM),
                       "cudaFuncSetAttribute(enc_head_fwd)");
    if (rc) return rc;
    const int blocks = (B + HEAD_B - 1) / HEAD_B;
    enc_skip_fwd<<<(unsigned)(((int64_t)B * SK + 255) / 256), 256, 0, s>>>(B, params, E, pts, off, len, n4, X);
    enc_head_fwd<<<blocks < 296 ? blocks : 296, EO, HEAD_SMEM, s>>>(hl, B, params, E);
    return enc_check(cudaGetLastError(), "enc_head_fwd launch");
}

int enc_args(const void* params, const void* pts, const void* off, const void* len, int B, int T, const float* nrm,
             const void* ws) {
    if (!params || !pts || !off || !len || !nrm || !ws) return tsm_internal_fail(TSM_EINVAL, "encoder: null pointer");
    if (B < 1 || T < 1) return tsm_internal_fail(TSM_EINVAL, "encoder: batch and time must be positive");
    if (reinterpret_cast<uintptr_t>(ws) % 256)
        return tsm_internal_fail(TSM_EINVAL, "encoder: workspace must be 256-byte aligned");
    if ((int64_t)B * T * enc::G3 > (int64_t)1 << 40) return tsm_internal_fail(TSM_EINVAL, "encoder: batch too large");
    return TSM_OK;
}

int enc_forward(const float* params, const float* pts, const int64_t* off, const int32_t* len, int B, int T,
                const float* nrm, EncWs& w, cudaStream_t s) {
    using namespace enc;
    const float4 n4 = make_float4(nrm[0], nrm[1], nrm[2], nrm[3]);
    enc_round_bf16<<<(OFF_WO + 255) / 256, 256, 0, s>>>(params, w.wq);
    const int rc = train_forward(reinterpret_cast<const float2*>(pts), off, len, B, T, n4, w.wq, params, w.tr, w.hl,
                                 w.status, s);
    if (rc) return rc;
    return enc_head(w.hl, B, params, w.E, reinterpret_cast<const float2*>(pts), off, len, n4, w.X, s);
}

int enc_backward(const float* params, const float* pts, const int64_t* off, const int32_t* len, int B, int T,
                 const float* nrm, EncWs& w, float* grad, cudaStream_t s) {
    using namespace enc;
    const float4 n4 = make_float4(nrm[0], nrm[1], nrm[2], nrm[3]);
    if ((B + HB_B - 1) / HB_B > 65535) return tsm_internal_fail(TSM_EINVAL, "encoder: batch too large");
    enc_head_bwd_w<<<dim3(EO, (B + HB_B - 1) / HB_B), HD, 0, s>>>(w.dE, w.hl, B, grad);
    enc_skip_bwd<<<(unsigned)(((int64_t)B * SK + 255) / 256 < 256 ? ((int64_t)B * SK + 255) / 256 : 256), 256, 0, s>>>(
        w.dE, w.X, B, params, grad);
    enc_head_bwd_h<<<(unsigned)(((int64_t)B * HD + 255) / 256), 256, 0, s>>>(w.dE, B, params, w.dhl);
    return train_backward(reinterpret_cast<const float2*>(pts), off, len, B, T, n4, w.wq, w.dhl, w.tr, grad, w.status, s);
}

// Inference workspace: the BF16 a_t images (B rounded up to 128 rows), last
// hidden states, embeddings, BF16 weights.
struct EmbWs {
    int* status;  // first word of the workspace: TC_ERR_* bits of the last call
    __nv_bfloat16* Ab;
    float *hl, *E;
    __nv_bfloat16* wq;
};

int64_t emb_layout(int B, int T, float* base, EmbWs* w) {
    int64_t o = 0;
    auto take = [&](int64_t n) {
        float* q = base ? base + o : nullptr;
        o += align64(n);
        return q;
    };
    float* st = take(1);
    const int64_t Bp = ((int64_t)B + enc::TC_M - 1) / enc::TC_M * enc::TC_M;
    float* Ab = take(Bp * T * enc::C1 / 2);
    float* hl = take((int64_t)B * enc::HD);
    float* E = take((int64_t)B * enc::ED);
    float* wqf = take((enc::N_PARAMS + 1) / 2);
    if (w) {
        w->status = reinterpret_cast<int*>(st);
        w->Ab = reinterpret_cast<__nv_bfloat16*>(Ab);
        w->hl = hl;
        w->E = E;
        w->wq = reinterpret_cast<__nv_bfloat16*>(wqf);
    }
    return o;
}

}  // namespace

extern "C" {

int tsm_enc_param_count(void) { return enc::N_PARAMS; }

int64_t tsm_enc_workspace_bytes(int32_t B, int32_t T, int32_t P) {
    if (B < 1 || T < 1 || P < 0) return -1;
    return ws_layout(B, T, P, nullptr, nullptr) * 4;
}

int tsm_enc_forward(const float* params, const float* pts, const int64_t* off, const int32_t* len, int32_t B,
                    int32_t T, const float* nrm, void* workspace, float* emb, void* stream) {
    int rc = enc_args(params, pts, off, len, B, T, nrm, workspace);
    if (rc) return rc;
    EncWs w;
    ws_layout(B, T, 0, static_cast<float*>(workspace), &w);
    cudaStream_t s = (cudaStream_t)stream;
    rc = enc_forward(params, pts, off, len, B, T, nrm, w, s);
    if (rc) return rc;
    if (emb) rc = enc_check(cudaMemcpyAsync(emb, w.E, (size_t)B * enc::ED * 4, cudaMemcpyDeviceToDevice, s),
                            "copy embeddings");
    return rc;
}

int tsm_enc_loss_grad_w(const float* params, const float* pts, const int64_t* off, const int32_t* len, int32_t B,
                        int32_t T, const float* nrm, const int32_t* ia, const int32_t* ib, const float* y,
                        const float* weights, int32_t P, void* workspace, float* grad, float* loss, float* pred,
                        void* stream) {
    int rc = enc_args(params, pts, off, len, B, T, nrm, workspace);
    if (rc) return rc;
    if (P < 1 || !ia || !ib || !y || !grad) return tsm_internal_fail(TSM_EINVAL, "tsm_enc_loss_grad: bad pairs");
    EncWs w;
    ws_layout(B, T, P, static_cast<float*>(workspace), &w);
    cudaStream_t s = (cudaStream_t)stream;
    rc = enc_forward(params, pts, off, len, B, T, nrm, w, s);
    if (rc) return rc;
    if ((rc = enc_check(cudaMemsetAsync(w.dE, 0, (size_t)B * enc::ED * 4, s), "memset dE"))) return rc;
    if ((rc = enc_check(cudaMemsetAsync(w.loss, 0, 4, s), "memset loss"))) return rc;
    if ((rc = enc_check(cudaMemsetAsync(grad, 0, (size_t)enc::N_PARAMS * 4, s), "memset grad"))) return rc;
    enc::enc_pair_loss<<<(P * 32 + 255) / 256, 256, 0, s>>>(w.E, ia, ib, y, weights, P, w.pred, w.loss, w.dE);
    rc = enc_backward(params, pts, off, len, B, T, nrm, w, grad, s);
    if (rc) return rc;
    if (loss) rc = enc_check(cudaMemcpyAsync(loss, w.loss, 4, cudaMemcpyDeviceToDevice, s), "copy loss");
    if (!rc && pred) rc = enc_check(cudaMemcpyAsync(pred, w.pred, (size_t)P * 4, cudaMemcpyDeviceToDevice, s), "copy pred");
    return rc;
}

int tsm_enc_loss_grad(const float* params, const float* pts, const int64_t* off, const int32_t* len, int32_t B,
                      int32_t T, const float* nrm, const int32_t* ia, const int32_t* ib, const float* y, int32_t P,
                      void* workspace, float* grad, float* loss, float* pred, void* stream) {
    return tsm_enc_loss_grad_w(params, pts, off, len, B, T, nrm, ia, ib, y, nullptr, P, workspace, grad, loss, pred,
                               stream);
}

int tsm_enc_adam(float* params, const float* grad, float* m, float* v, int32_t step, float lr, float beta1,
                 float beta2, float eps, void* stream) {
    if (!params || !grad || !m || !v || step < 1) return tsm_internal_fail(TSM_EINVAL, "tsm_enc_adam: bad arguments");
    const float bc1 = 1.f - powf(beta1, (float)step), bc2 = 1.f - powf(beta2, (float)step);
    enc::enc_adam<<<(enc::N_PARAMS + 255) / 256, 256, 0, (cudaStream_t)stream>>>(params, grad, m, v, enc::N_PARAMS, lr,
                                                                                 beta1, beta2, eps, bc1, bc2);
    return enc_check(cudaGetLastError(), "enc_adam launch");
}

int64_t tsm_enc_embed_workspace_bytes(int32_t B, int32_t T) {
    if (B < 1 || T < 1) return 0;
    return emb_layout(B, T, nullptr, nullptr) * 4;
}

int tsm_enc_embed_opts(const float* params, const float* pts, const int64_t* off, const int32_t* len, int32_t B,
                       int32_t T, const float* nrm, void* workspace, float* emb, int64_t wait_cycles,
                       int32_t stall_step, void* stream) {
    int rc = enc_args(params, pts, off, len, B, T, nrm, workspace);
    if (rc) return rc;
    if (!emb) return tsm_internal_fail(TSM_EINVAL, "tsm_enc_embed: null output");
    if (wait_cycles < 1 || stall_step < -1) return tsm_internal_fail(TSM_EINVAL, "tsm_enc_embed_opts: bad wait limit or stall step");
    using namespace enc;
    EmbWs w;
    emb_layout(B, T, static_cast<float*>(workspace), &w);
    cudaStream_t s = (cudaStream_t)stream;
    const float4 n4 = make_float4(nrm[0], nrm[1], nrm[2], nrm[3]);
    if ((rc = enc_check(cudaMemsetAsync(w.status, 0, 4, s), "memset embed status"))) return rc;
    enc_round_bf16<<<(OFF_WO + 255) / 256, 256, 0, s>>>(params, w.wq);
    const int Bp = (B + TC_M - 1) / TC_M * TC_M;
    const int64_t tot = (int64_t)Bp * ((T + CT - 1) / CT);
    enc_conv_fwd_tc<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(reinterpret_cast<const float2*>(pts), off, len, B,
                                                                   Bp, T, n4, w.wq, params, w.Ab);
    rc = enc_check(cudaFuncSetAttribute(enc_gru_embed_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM),
                   "cudaFuncSetAttribute(enc_gru_embed_tc)");
    if (rc) return rc;
    enc_gru_embed_tc<<<Bp / TC_M, TC_THREADS, TC_SMEM, s>>>(w.Ab, len, B, T, w.wq, params, w.hl, w.status,
                                                            wait_cycles, stall_step);
    return enc_head(w.hl, B, params, emb, reinterpret_cast<const float2*>(pts), off, len, n4, nullptr, s);
}

int tsm_enc_embed(const float* params, const float* pts, const int64_t* off, const int32_t* len, int32_t B,
                  int32_t T, const float* nrm, void* workspace, float* emb, void* stream) {
    return tsm_enc_embed_opts(params, pts, off, len, B, T, nrm, workspace, emb, enc::TC_WAIT_CYCLES, -1, stream);
}

int tsm_enc_train_status(void* workspace, int32_t* status, void* stream) {
    if (!workspace || !status) return tsm_internal_fail(TSM_EINVAL, "tsm_enc_train_status: null argument");
    int rc = enc_check(cudaStreamSynchronize((cudaStream_t)stream), "tsm_enc_train_status: synchronise");
    if (rc) return rc;
    if ((rc = enc_check(cudaMemcpy(status, workspace, 4, cudaMemcpyDeviceToHost), "tsm_enc_train_status: read")))
        return rc;
    if (*status == 0) return TSM_OK;
    if ((rc = enc_check(cudaMemset(workspace, 0, 4), "tsm_enc_train_status: clear"))) return rc;
    char b[256];
    snprintf(b, sizeof(b), "training kernels: a tensor-core or copy wait ran out (status %d%s); "
             "results of the tsm_enc_loss_grad and tsm_enc_forward calls since the last check are incomplete", *status,
             (*status & 128) ? ": tensor memory not freed, reset the device" : "");
    return tsm_internal_fail(TSM_ETIMEOUT, b);
}

int tsm_enc_embed_status(const void* workspace, int32_t* status, void* stream) {
    if (!workspace || !status) return tsm_internal_fail(TSM_EINVAL, "tsm_enc_embed_status: null argument");
    int rc = enc_check(cudaStreamSynchronize((cudaStream_t)stream), "tsm_enc_embed_status: synchronise");
    if (rc) return rc;
    if ((rc = enc_check(cudaMemcpy(status, workspace, 4, cudaMemcpyDeviceToHost), "tsm_enc_embed_status: read")))
        return rc;
    if (*status == 0) return TSM_OK;
    char b[256];
    snprintf(b, sizeof(b), "tsm_enc_embed: a tensor-core wait ran out (status %d: %s%s%s); the affected embeddings are NaN",
             *status, (*status & enc::TC_ERR_COPY) ? "a_t copy " : "", (*status & enc::TC_ERR_MMA) ? "MMA " : "",
             (*status & enc::TC_ERR_TMEM_HELD) ? "tensor memory not freed: reset the device" : "");
    return tsm_internal_fail(TSM_ETIMEOUT, b);
}

}  // extern "C"
