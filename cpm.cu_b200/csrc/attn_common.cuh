// Shared by the attention kernel and the stage-1 scores of block selection: tile geometry.
#pragma once
#include "common.cuh"
#include "ptx.cuh"

namespace attn {

constexpr int ROWS = 128;       // query rows per tile (UMMA M)
constexpr int KEYS = 128;       // keys per tile
constexpr int HALF_BYTES = ROWS * 128;        // 64 columns of a tile: 128 rows x 128 B

__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

}  // namespace attn
