// Training recurrences of the encoder (tsm_train.cu), called by the training
// entry points of tsm_encoder.cu.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace enc {

constexpr int TB = 16;  // trajectories per block of the recurrences

// Device buffers of one batch.  The batch's trajectories are sorted by length,
// longest first, and cut into blocks of TB; a block of longest length n has
// slots for n time steps rounded up to even, block k's first slot at
// slot0[k].  "half" is 0 for trajectories 0..7 of a block, 1 for 8..15; a
// group is one half of a slot.
struct TrainWs {
    int32_t* perm;   // [blocks * TB] trajectory of each row, -1 past the batch
    int32_t* slot0;  // [blocks + 1]
    unsigned char* a_op;              // [slot][3 parts][half][64][8] BF16: conv output
    unsigned char* a_on;              // [group][64] bit s: conv output of trajectory s positive
    unsigned char *h_hi, *h_lo;       // [group][128][8] BF16: hidden state before the step, first two parts
    float* cache;                     // [slot][5][4][128][4]: r, z, n, Whn h + bhn, h before the step
    unsigned char *g_hi, *g_lo;       // [4][group][128][8] BF16: gate gradients r, z, n (input), n (hidden)
    float* dA;                        // [slot][4][64][4] gradient of the conv output (before the relu)
    int64_t slots;                    // capacity
    int blocks;
};

// Lays the buffers out from `base` (256-byte aligned; nullptr: size only) and
// returns their size in bytes, for B trajectories of at most T steps.
int64_t train_layout(int B, int T, unsigned char* base, TrainWs* w);

// Forward: hl[b][128] = the hidden state after the last point, and what the
// backward needs.  wq: BF16 weights; p: FP32 parameters.  Stream-ordered.  A
// bounded wait that runs out ORs a bit into *status.
int train_forward(const float2* pts, const int64_t* off, const int32_t* len, int B, int T, float4 nrm,
                  const __nv_bfloat16* wq, const float* p, const TrainWs& w, float* hl, int* status, cudaStream_t s);
// Backward from dhl[b][128]: adds the gradients of the conv and GRU
// parameters to grad (flat parameter layout).
int train_backward(const float2* pts, const int64_t* off, const int32_t* len, int B, int T, float4 nrm,
                   const __nv_bfloat16* wq, const float* dhl, const TrainWs& w, float* grad, int* status,
                   cudaStream_t s);

}  // namespace enc
