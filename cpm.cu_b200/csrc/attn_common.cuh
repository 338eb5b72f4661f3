// Shared by the attention kernel and the stage-1 scores of block selection: tile geometry.
#pragma once
#include "common.cuh"
#include "ptx.cuh"

namespace attn {

constexpr int ROWS = 128;       // query rows per tile (UMMA M)
constexpr int KEYS = 128;       // keys per tile
constexpr int HALF_BYTES = ROWS * 128;        // 64 columns of a tile: 128 rows x 128 B

struct AttnArgs {
    int tq, hq, hkv, grp, tok_per_tile, num_mtiles;
    int heavy_first;  // causal prefill: token tiles are handed out last-to-first, longest key range first
    const int32_t* kv_len;
    int kv_len_add;
    const int32_t* n_valid;
    const uint64_t* mask;
    int mask_k;
    int window;
    int exact_window;    // > 0: per-token sliding window (tokens); BIASED instantiations only
    float bias_exp;      // > 0: distance bias with slopes 2^(-bias_exp * (h + 1) / hq); BIASED instantiations only
    int sink;            // 1: exp(0) is added to every row's sum
    float out_scale;     // factor of the output
    int out_cols;        // value columns that are stored per head (the rest of DV is padding)
    const uint64_t* blockmask;  // [hkv][tq][bm_words] bits over 64-key blocks, or null
    int bm_words, block_window;
    float scale_log2;
    bf16* out;
    int out_ld;
    float* ws_o;
    float* ws_ml;
    int* error;
    long long* prof;  // bench only (-DCPMCU_ATTN_PROFILE): clock counters of CTA 0, or null
};

__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

}  // namespace attn

// Two query tiles per CTA (pair_attn.cu); `a` as for the one-tile kernel.
void launch_pair_attention(const AttnPlan& p, const attn::AttnArgs& a, cudaStream_t s);
