// Weight gradients of the encoder's GRU on the tensor cores (tcgen05):
//     dW_ih[j][c]  = sum_(slot,s) G [j] A[c]       384 x 64
//     dW_hh[j][kk] = sum_(slot,s) GH[j] H[kk]      384 x 128
// over the batch's time slots and the 16 trajectories of each (tsm_train.h; the
// gate gradients of a trajectory past its end are zero), G / GH the gate
// gradients of the input and hidden side, which differ in the n rows only, A
// the conv activations and H the hidden state before the step.
//
// Precision.  The four operands are FP32.  Each is split into BF16 parts,
// x = hi + lo with lo = bf16(x - hi) (BF16 keeps FP32's exponent range, which
// gate gradients of 1e-9 need), and the tensor cores take
//     g . x = g_hi . x_hi + g_lo . x_hi + g_hi . x_lo   (+ g_lo . x_lo, dropped)
// with FP32 accumulation: three MMAs per K step, about 2^-16 relative per
// product (the split-product method of Markidis et al., IPDPSW 2018).
//
// The operands of the recurrences are the hi and lo images (tsm_train.cu),
// K-major core-matrix layout (tsm_umma.cuh), 16 K per slot.  One kernel, split-K over
// the CTAs: CTA (m tile of 128 rows of j, K range) streams both products'
// operands through a four-stage ring (cp.async.bulk, mbarrier transaction
// counts), one thread issues six MMAs per K step into four accumulators, and
// all four warps add the results to the gradient with atomics.  The cross
// products accumulate apart from the hi . hi ones: an accumulation step
// truncates, and 900 instead of 300 of them on the large sums made the error of
// dW_ih half again as large (1,024 pairs: 4.2e-6 of the gradient's norm).  Waits are bounded (about 1 s of SM clocks); one that
// runs out ORs a bit into *status and the CTA adds nothing.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdio>

#include "tsm.h"
#include "tsm_umma.cuh"
#include "tsm_wgrad.h"

int tsm_internal_fail(int code, const char* msg);

namespace tsm {
namespace wgrad {

constexpr int G3 = 384;   // gate rows j (r, z, n)
constexpr int NA = 64;    // conv channels c
constexpr int NH = 128;   // hidden units kk
constexpr int MT = 128;   // rows of j per CTA (MMA M, tensor-memory lanes)
constexpr int SKW = 32;   // K per stage: two MMAs of K = 16 per product
constexpr int NST = 4;    // stages
constexpr int THREADS = 128;
// one stage: [G hi | G lo | GH hi | GH lo | A hi | A lo | H hi | H lo]
constexpr int M_PART = MT * SKW * 2;   // 8,192
constexpr int A_PART = NA * SKW * 2;   // 4,096
constexpr int H_PART = NH * SKW * 2;   // 8,192
constexpr int S_GHI = 0, S_GLO = M_PART, S_GHHI = 2 * M_PART, S_GHLO = 3 * M_PART, S_AHI = 4 * M_PART,
              S_ALO = S_AHI + A_PART, S_HHI = S_ALO + A_PART, S_HLO = S_HHI + H_PART;
constexpr int STAGE = S_HLO + H_PART;  // 57,344
constexpr int OFF_BAR = NST * STAGE;
constexpr int SMEM = OFF_BAR + 128;    // 229,504
// accumulators ih (64 columns) and hh (128) of the hi . hi products at column 0, of the cross products at T_X
constexpr uint32_t TMEM_COLS = 512, T_X = 256;
constexpr long long WAIT_CYCLES = 2000000000LL;
static_assert(SMEM <= 227 * 1024, "shared memory");

// status bits (OR-ed into the caller's word)
constexpr int ERR_COPY = 16, ERR_MMA = 32, ERR_DONE = 64, ERR_TMEM = 128;

__global__ void __launch_bounds__(THREADS, 1) wg_kernel(
    enc::TrainWs w, float* __restrict__ d_ih, float* __restrict__ d_hh, int* __restrict__ status,
    long long wait_cycles) {
    namespace U = tsm::umma;
    extern __shared__ __align__(1024) unsigned char sm[];
    const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(sm));
    const uint32_t bar = sbase + OFF_BAR;
    auto full = [&](int i) { return bar + 8 * i; };
    auto empty = [&](int i) { return bar + 8 * NST + 8 * i; };
    const uint32_t donebar = bar + 16 * NST;
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(sm + OFF_BAR + 16 * NST + 8);
    volatile int* flags = reinterpret_cast<volatile int*>(sm + OFF_BAR + 16 * NST + 12);  // bit 0 failed, 1 busy
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int mt = blockIdx.x;  // tile of j: gate r, z or n
    const bool n_rows = mt == 2;
    // this CTA's stages [s0, s1) of the K range (a stage: two slots of 16), from the device-side slot count
    const int64_t nst_all = w.slot0[w.blocks] / 2;
    const int64_t per = (nst_all + gridDim.y - 1) / gridDim.y;
    const int64_t s0 = (int64_t)blockIdx.y * per;
    const int64_t s1 = min(nst_all, s0 + per);
    const int64_t ns = s1 > s0 ? s1 - s0 : 0;
    if (ns == 0) return;  // uniform over the CTA, before any barrier or allocation

    if (threadIdx.x == 0) {
        for (int i = 0; i < NST; ++i) {
            U::mbar_init(full(i), 1);
            U::mbar_init(empty(i), 1);
        }
        U::mbar_init(donebar, 1);
        *flags = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) U::tmem_alloc(sbase + OFF_BAR + 16 * NST + 8, TMEM_COLS);
    U::fence_before_sync();
    __syncthreads();
    U::fence_after_sync();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0 && lane == 0) {  // copies
        const int64_t tile = w.slots * 2 * MT * 16;  // bytes of one gate's image
        int64_t g = 0;
        for (int64_t s = s0; s < s1; ++s, ++g) {
            const int slot = (int)(g % NST);
            const uint32_t u = (uint32_t)(g / NST);
            if (!U::mbar_wait(empty(slot), (u & 1) ^ 1, wait_cycles)) {
                atomicOr(status, ERR_COPY);
                *flags = 1;
                break;
            }
            const uint32_t st = sbase + slot * STAGE;
            U::mbar_arrive_expect_tx(full(slot), n_rows ? STAGE : STAGE - 2 * M_PART);
            auto load = [&](int at, const unsigned char* src, int part) {
                U::bulk_load(st + at, src + s * part, part, full(slot));
            };
            load(S_GHI, w.g_hi + mt * tile, M_PART);
            load(S_GLO, w.g_lo + mt * tile, M_PART);
            if (n_rows) {  // the hidden side has its own n gradients
                load(S_GHHI, w.g_hi + 3 * tile, M_PART);
                load(S_GHLO, w.g_lo + 3 * tile, M_PART);
            }
            for (int j = 0; j < 2; ++j) {  // a slot's three parts stand together
                const unsigned char* src = w.a_op + (2 * s + j) * (3 * A_PART / 2);
                U::bulk_load(st + S_AHI + j * (A_PART / 2), src, A_PART / 2, full(slot));
                U::bulk_load(st + S_ALO + j * (A_PART / 2), src + A_PART / 2, A_PART / 2, full(slot));
            }
            load(S_HHI, w.h_hi, H_PART);
            load(S_HLO, w.h_lo, H_PART);
        }
        // every copy issued lands before the CTA exits: the last use of each slot
        for (int slot = 0; slot < NST; ++slot)
            if (slot < g) U::mbar_wait(full(slot), (uint32_t)((g - 1 - slot) / NST) & 1, wait_cycles);
    } else if (warp == 1 && lane == 0) {  // MMAs
        constexpr uint32_t id_ih = U::idesc_bf16_f32(MT, NA), id_hh = U::idesc_bf16_f32(MT, NH);
        const uint32_t t_ih = tmem, t_hh = tmem + NA;
        for (int64_t g = 0; g < ns; ++g) {
            const int slot = (int)(g % NST);
            const uint32_t u = (uint32_t)(g / NST);
            if (!U::mbar_wait(full(slot), u & 1, wait_cycles)) {
                atomicOr(status, ERR_MMA);
                *flags = 1;
                break;
            }
            U::fence_after_sync();
            const uint32_t st = sbase + slot * STAGE;
#pragma unroll
            for (int kk = 0; kk < SKW / 16; ++kk) {
                const uint32_t first = (g == 0 && kk == 0) ? 0u : 1u;
                const uint64_t gd_hi = U::smem_desc(st + S_GHI + kk * 2 * (MT * 16), MT * 16, 128);
                const uint64_t gd_lo = U::smem_desc(st + S_GLO + kk * 2 * (MT * 16), MT * 16, 128);
                const uint64_t ghd_hi = n_rows ? U::smem_desc(st + S_GHHI + kk * 2 * (MT * 16), MT * 16, 128) : gd_hi;
                const uint64_t ghd_lo = n_rows ? U::smem_desc(st + S_GHLO + kk * 2 * (MT * 16), MT * 16, 128) : gd_lo;
                const uint64_t ad_hi = U::smem_desc(st + S_AHI + kk * 2 * (NA * 16), NA * 16, 128);
                const uint64_t ad_lo = U::smem_desc(st + S_ALO + kk * 2 * (NA * 16), NA * 16, 128);
                const uint64_t hd_hi = U::smem_desc(st + S_HHI + kk * 2 * (NH * 16), NH * 16, 128);
                const uint64_t hd_lo = U::smem_desc(st + S_HLO + kk * 2 * (NH * 16), NH * 16, 128);
                U::mma_bf16(t_ih, gd_hi, ad_hi, id_ih, first);
                U::mma_bf16(t_ih + T_X, gd_lo, ad_hi, id_ih, first);
                U::mma_bf16(t_ih + T_X, gd_hi, ad_lo, id_ih, 1u);
                U::mma_bf16(t_hh, ghd_hi, hd_hi, id_hh, first);
                U::mma_bf16(t_hh + T_X, ghd_lo, hd_hi, id_hh, first);
                U::mma_bf16(t_hh + T_X, ghd_hi, hd_lo, id_hh, 1u);
            }
            U::commit(empty(slot));
        }
        U::commit(donebar);  // completes when every MMA issued above has
    }
    // epilogue: all four warps; warp w reads tensor-memory lanes 32 w .. 32 w + 31 (rows j of the tile)
    __syncwarp();
    const bool done = __all_sync(0xffffffffu, U::mbar_wait(donebar, 0, wait_cycles));
    if (!done) {
        if (lane == 0) atomicOr(status, ERR_DONE);
        if (lane == 0) *flags = 3;  // MMAs may still write tensor memory: keep it allocated
    }
    U::fence_after_sync();
    __syncthreads();
    const int fl = *flags;
    if (fl == 0) {
        const int64_t j = (int64_t)mt * MT + 32 * warp + lane;
        const uint32_t ta = tmem + ((uint32_t)(32 * warp) << 16);
        for (int c0 = 0; c0 < NA + NH; c0 += 16) {
            uint32_t r[16], x[16];
            U::ld16(ta + c0, r);
            U::ld16(ta + T_X + c0, x);
            U::wait_ld(r);
            U::wait_ld(x);
            float* dst = c0 < NA ? d_ih + j * NA + c0 : d_hh + j * NH + (c0 - NA);
#pragma unroll
            for (int i = 0; i < 16; ++i) atomicAdd(dst + i, __uint_as_float(r[i]) + __uint_as_float(x[i]));
        }
    }
    U::fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        if (fl & 2) {
            if (lane == 0) atomicOr(status, ERR_TMEM);
        } else {
            U::fence_after_sync();
            U::tmem_dealloc(tmem, TMEM_COLS);
        }
    }
}

}  // namespace wgrad
}  // namespace tsm

namespace {

int wg_check(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return TSM_OK;
    char b[256];
    snprintf(b, sizeof(b), "%s: %s", what, cudaGetErrorString(e));
    return tsm_internal_fail(TSM_ECUDA, b);
}

}  // namespace

int tsm_wgrad_tc(const enc::TrainWs& w, int* status, float* d_ih, float* d_hh, cudaStream_t s) {
    using namespace tsm::wgrad;
    int rc = wg_check(cudaFuncSetAttribute(wg_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM),
                      "cudaFuncSetAttribute(wg_kernel)");
    if (rc) return rc;
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // K split: one wave of CTAs over the three j tiles, at most the stages there can be
    int64_t ksplit = sms / (G3 / MT);
    if (ksplit > w.slots / 2) ksplit = w.slots / 2;
    if (ksplit < 1) ksplit = 1;
    wg_kernel<<<dim3(G3 / MT, (unsigned)ksplit), THREADS, SMEM, s>>>(w, d_ih, d_hh, status, WAIT_CYCLES);
    return wg_check(cudaGetLastError(), "wgrad launch");
}
