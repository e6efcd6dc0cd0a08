// Shapes, parameter layout and small helpers shared by the encoder's
// translation units (tsm_encoder.cu, tsm_train.cu).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace enc {

constexpr int C1 = 64;    // conv channels
constexpr int KW = 5;     // conv width
constexpr int HD = 128;   // hidden
constexpr int G3 = 384;   // 3 gates
constexpr int EO = 128;   // learned head outputs
constexpr int NS = 16;    // resampled points of the geometric skip
constexpr int SK = 2 * NS;  // skip features (x, y of each resampled point)
constexpr int ED = EO + SK; // embedding: [head outputs | skip weights * resampled points]

// parameter offsets in the flat FP32 master buffer
constexpr int OFF_W1 = 0;                    // [64][2][5]
constexpr int OFF_B1 = OFF_W1 + C1 * 2 * KW; // [64]
constexpr int OFF_WIH = OFF_B1 + C1;         // [384][64]
constexpr int OFF_BIH = OFF_WIH + G3 * C1;   // [384]
constexpr int OFF_WHH = OFF_BIH + G3;        // [384][128]
constexpr int OFF_BHH = OFF_WHH + G3 * HD;   // [384]
constexpr int OFF_WO = OFF_BHH + G3;         // [128][128]
constexpr int OFF_BO = OFF_WO + EO * HD;     // [128]
constexpr int OFF_SC = OFF_BO + EO;          // [16] u_k: log-weights of the resampled points of the skip
constexpr int N_PARAMS = OFF_SC + NS;

// Normalised input coordinate i of point t of trajectory b (0 outside).
__device__ __forceinline__ float xin(const float2* pts, int64_t off, int len, int t, int i, float4 nrm) {
    if (t < 0 || t >= len) return 0.f;
    const float2 v = pts[off + t];
    return i == 0 ? (v.x - nrm.x) * nrm.z : (v.y - nrm.y) * nrm.w;
}

}  // namespace enc
