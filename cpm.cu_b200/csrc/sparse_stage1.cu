// Stage-1 scores of InfLLM-v2 block selection for prefill-sized launches on the tensor cores, sm_100a (see sparse_select.cu for
// what is computed and for decode-sized launches).
//
// One CTA has 8 tokens x 16 query heads of a key head as the 128 rows of a tile and walks the compressed keys in chunks of
// 128: first the keys of the log-sum-exp (running maximum and sum per row), then the scored keys, whose exponentials are
// normalised and summed over the 16 heads: lanes of a warp, 15 shuffles per 16 keys leave lane l with key l.  The exponentials bound
// it (16384 per chunk on the MUFU pipe, 1024 cycles; the MMAs take 512); two CTAs per SM hide one another's latencies.
// The blocks of peaked heads are told apart by scores below 2^-126, which ex2.approx.ftz makes equal: a chunk with a sum below 2^-98
// (above, what 16 flushed terms would add is below the last place) is gone through again with exp2f, as in sparse_select.cu,
// from its scores in tensor memory.  Beside the row's largest term of the log-sum-exp, which is one, what is flushed there is below the
// last place as well.
// A 32768-token prompt in chunks of 2048, 32 query heads, 44 us a launch on average; as warp-level fragments in two kernels with
// partial sums through memory 146 + 64 us.
#include "attn_common.cuh"
#include "sparse_select.cuh"

using namespace attn;

namespace {

constexpr int S1_TOKENS = 8, S1_HEADS = 16;
constexpr int SOFT_THREADS = 256;                  // two threads per row, 64 keys of a chunk each
constexpr int S1_UMMA_THREADS = SOFT_THREADS + 32; // + TMA and MMA
constexpr int TILE_BYTES = ROWS * 256;             // 128 rows x 128 columns bf16
constexpr int SMEM_K = TILE_BYTES;                 // 2 stages
constexpr int SMEM_XCH = SMEM_K + 2 * TILE_BYTES;  // [2 halves][128] (max, sum)
constexpr int SMEM_CTRL = SMEM_XCH + 2 * ROWS * 8;
constexpr int SMEM_BYTES = SMEM_CTRL + 128 + 1024;
constexpr int S1_TMEM_COLS = 256;                  // S(i) at 128 (i & 1)

struct Stage1UmmaArgs {
    const int32_t* kv_len;
    int kv_add;
    const int32_t* n_valid;
    int lse_stride, sparse_switch;
    float scale_log2;
    bf16* scores;
    int score_ld, T;
    int* error;
};

__device__ __forceinline__ int entries_of(int L, int stride) { return max((L - stride) / stride, 0); }

__global__ void __launch_bounds__(S1_UMMA_THREADS, 2)
sparse_stage1_umma_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_lse,
                          const __grid_constant__ CUtensorMap tm_c1, const Stage1UmmaArgs a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* q_bar = reinterpret_cast<uint64_t*>(smem + SMEM_CTRL);
    uint64_t* k_full = q_bar + 1;   // [2]
    uint64_t* s_bar = q_bar + 3;    // [2]  S(i) is in TMEM
    uint64_t* s_free = q_bar + 5;   // [2]  S(i) has been read
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(q_bar + 7);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    float2* xch = reinterpret_cast<float2*>(smem + SMEM_XCH);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    grid_dep_trigger();
    const int t0 = blockIdx.x * S1_TOKENS, g = blockIdx.y;
    if (tid == 0) {
        ptx::mbar_init(q_bar, 1);
        for (int i = 0; i < 2; ++i) {
            ptx::mbar_init(&k_full[i], 1);
            ptx::mbar_init(&s_bar[i], 1);
            ptx::mbar_init(&s_free[i], SOFT_THREADS / 32);
        }
        *abort_flag = 0;
        ptx::mbar_fence_init();
    }
    if (warp == 0) {
        ptx::tmem_alloc(tmem_slot, S1_TMEM_COLS);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    grid_dep_wait();

    const int L = *a.kv_len + a.kv_add;
    const int t_end = (a.n_valid != nullptr) ? min(*a.n_valid, a.T) : a.T;
    const bool active = L > 0 && entries_of(L, a.lse_stride) * a.lse_stride >= a.sparse_switch && t0 < t_end;
    const int nl = active ? entries_of(L, a.lse_stride) : 0, n1 = active ? entries_of(L, 16) : 0;
    const int chunks_l = (nl + KEYS - 1) / KEYS, n_it = chunks_l + (n1 + KEYS - 1) / KEYS;

    if (warp == SOFT_THREADS / 32) {
        if (lane == 0 && n_it > 0) {
            constexpr uint32_t idesc = ptx::umma_idesc_bf16(ROWS, KEYS, 0, 0);
            const uint32_t q_addr = ptx::smem_u32(smem);
            auto load = [&](int i) {
                const CUtensorMap* tm = i < chunks_l ? &tm_lse : &tm_c1;
                const int key0 = (i < chunks_l ? i : i - chunks_l) * KEYS;
                uint8_t* dst = smem + SMEM_K + (i & 1) * TILE_BYTES;
                ptx::mbar_arrive_expect_tx(&k_full[i & 1], TILE_BYTES);
                for (int c = 0; c < 2; ++c) ptx::tma_load_2d(dst + c * HALF_BYTES, tm, &k_full[i & 1], g * 128 + c * 64, key0);
            };
            ptx::mbar_arrive_expect_tx(q_bar, TILE_BYTES);
            for (int c = 0; c < 2; ++c) ptx::tma_load_3d(smem + c * HALF_BYTES, &tm_q, q_bar, c * 64, g * S1_HEADS, t0);
            load(0);
            bool ok = ptx::mbar_wait(q_bar, 0, abort_flag);
            for (int i = 0; ok && i < n_it; ++i) {
                const int st = i & 1;
                if (!ptx::mbar_wait(&k_full[st], (i >> 1) & 1, abort_flag)) { ok = false; break; }
                if (!ptx::mbar_wait(&s_free[st], ((i >> 1) & 1) ^ 1, abort_flag)) { ok = false; break; }
                ptx::tc_fence_after();
                const uint32_t k_addr = ptx::smem_u32(smem + SMEM_K + st * TILE_BYTES);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const uint32_t off = (j >> 2) * HALF_BYTES + (j & 3) * 32;
                    ptx::umma_ss(tmem_base + st * KEYS, ptx::umma_desc_sw128(q_addr + off, 16, 1024), ptx::umma_desc_sw128(k_addr + off, 16, 1024), idesc,
                                 j ? 1u : 0u);
                }
                ptx::umma_commit(&s_bar[st]);
                if (i + 1 < n_it) {   // the other stage's keys were read by S(i - 1)
                    if (i > 0 && !ptx::mbar_wait(&s_bar[st ^ 1], ((i - 1) >> 1) & 1, abort_flag)) { ok = false; break; }
                    load(i + 1);
                }
            }
            if (!ok) {
                const long long c0 = clock64();   // copies in flight land before the CTA retires
                while (clock64() - c0 < 2000000LL) {}
            }
        }
    } else {
        const int ch = warp >> 2, row = (warp & 3) * 32 + lane;
        const uint32_t tmem_s = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + ch * 64;
        const float sl2 = a.scale_log2;
        bool ok = true;
        uint32_t sc[64];
        auto fetch = [&](int i) -> bool {
            const int st = i & 1;
            if (!ptx::mbar_wait_warp(&s_bar[st], (i >> 1) & 1, abort_flag)) return false;
            ptx::tc_fence_after();
            ptx::tmem_ld32(tmem_s + st * KEYS, sc);
            ptx::tmem_ld32(tmem_s + st * KEYS + 32, sc + 32);
            ptx::tmem_wait_ld();
            return true;
        };
        auto release = [&](int i) {
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&s_free[i & 1]);
        };
        float m = -INFINITY, sum = 0.f;
        for (int i = 0; ok && i < chunks_l; ++i) {
            ok = fetch(i);
            if (!ok) break;
            release(i);
            const int left = nl - i * KEYS - ch * 64;   // keys of this thread that exist
            if (left < 64) {
#pragma unroll
                for (int c = 0; c < 64; ++c) {
                    if (c >= left) sc[c] = 0xff800000u;
                }
            }
            float mx[4] = {m, m, m, m};
#pragma unroll
            for (int c = 0; c < 64; ++c) mx[c & 3] = fmaxf(mx[c & 3], __uint_as_float(sc[c]));
            const float m_new = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            if (m_new != -INFINITY) {
                float s4[4] = {m == -INFINITY ? 0.f : sum * fast_exp2((m - m_new) * sl2), 0.f, 0.f, 0.f};
#pragma unroll
                for (int c = 0; c < 64; ++c) s4[c & 3] += fast_exp2((__uint_as_float(sc[c]) - m_new) * sl2);
                sum = (s4[0] + s4[1]) + (s4[2] + s4[3]);
                m = m_new;
            }
        }
        // both halves of a row: (max, 1 / sum); every softmax thread gets here, whatever its waits returned
        xch[ch * ROWS + row] = make_float2(m, sum);
        ptx::named_bar_sync(1, SOFT_THREADS);
        const float2 o = xch[(ch ^ 1) * ROWS + row];
        float m_row = fmaxf(m, o.x), inv = 0.f;
        if (m_row == -INFINITY) {
            m_row = 0.f;
        } else {
            const float a0 = m == -INFINITY ? 0.f : sum * fast_exp2((m - m_row) * sl2), a1 = o.x == -INFINITY ? 0.f : o.y * fast_exp2((o.x - m_row) * sl2);
            const float both = a0 + a1;
            inv = both > 0.f ? 1.f / both : 0.f;
        }
        const int t = t0 + row / S1_HEADS;
        bf16* dst = a.scores + (static_cast<size_t>(g) * a.T + (t < t_end ? t : t0)) * a.score_ld + ch * 64 + (lane & 15);
        for (int i = chunks_l; ok && i < n_it; ++i) {
            ok = fetch(i);
            if (!ok) break;
            const int key0 = (i - chunks_l) * KEYS;
            const int left = n1 - key0 - ch * 64;
            // sum over the 16 lanes of a token: each step a lane keeps half of its columns and hands over the rest
            auto store_sums = [&](float (&v)[16], int c0) {
#pragma unroll
                for (int h = 8; h > 0; h >>= 1) {
                    const bool upper = (lane & h) != 0;
#pragma unroll
                    for (int c = 0; c < h; ++c) {
                        const float give = upper ? v[c] : v[c + h], keep = upper ? v[c + h] : v[c];
                        v[c] = keep + __shfl_xor_sync(0xffffffffu, give, h);
                    }
                }
                if (t < t_end) dst[key0 + c0] = __float2bfloat16(v[0]);
            };
            bool small = false;
#pragma unroll
            for (int c0 = 0; c0 < 64; c0 += 16) {
                float v[16];
#pragma unroll
                for (int c = 0; c < 16; ++c) v[c] = c0 + c < left ? fast_exp2((__uint_as_float(sc[c0 + c]) - m_row) * sl2) * inv : 0.f;
                store_sums(v, c0);
                small = small || (v[0] < 0x1p-98f && c0 + (lane & 15) < left);
            }
            if (__any_sync(0xffffffffu, small)) {
#pragma unroll 1
                for (int c0 = 0; c0 < 64; c0 += 16) {
                    uint32_t r[16];
                    float v[16];
                    ptx::tmem_ld16(tmem_s + (i & 1) * KEYS + c0, r);
                    ptx::tmem_wait_ld();
#pragma unroll
                    for (int c = 0; c < 16; ++c) v[c] = c0 + c < left ? exp2f((__uint_as_float(r[c]) - m_row) * sl2) * inv : 0.f;
                    store_sums(v, c0);
                }
            }
            release(i);
        }
    }

    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem_base, S1_TMEM_COLS);
    }
    if (tid == 0 && *abort_flag) atomicOr(a.error, ERR_ATTN_TIMEOUT);
}

}  // namespace

void launch_sparse_stage1_prefill(const SparseBuffers& b, const SparseConfig& cfg, int layer, const bf16* q, int q_ld, int T, int hkv,
                                  const int32_t* kv_len, int kv_add, const int32_t* n_valid, cudaStream_t s) {
    static bool configured = false;
    if (!configured) {
        CUDA_CHECK(cudaFuncSetAttribute(sparse_stage1_umma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        configured = true;
    }
    const uint64_t kv_dim = static_cast<uint64_t>(hkv) * 128;
    const bf16* c1 = b.c1 + layer * b.c1_layer_stride;
    const CUtensorMap tm_q = make_tmap_3d(q, 128, static_cast<uint64_t>(hkv) * S1_HEADS, T, 256, static_cast<uint64_t>(q_ld) * 2, 64, S1_HEADS, S1_TOKENS);
    const CUtensorMap tm_c1 = make_tmap_2d(c1, kv_dim, b.budget / 16, kv_dim * 2, 64, KEYS);
    const CUtensorMap tm_lse = cfg.compress_lse ? make_tmap_2d(b.c2 + layer * b.c2_layer_stride, kv_dim, b.budget / 64, kv_dim * 2, 64, KEYS) : tm_c1;
    Stage1UmmaArgs a;
    a.kv_len = kv_len; a.kv_add = kv_add; a.n_valid = n_valid;
    a.lse_stride = cfg.compress_lse ? 64 : 16;
    a.sparse_switch = cfg.sparse_switch;
    a.scale_log2 = 1.4426950408889634f / sqrtf(128.f);
    a.scores = b.scores; a.score_ld = b.score_ld; a.T = T;
    a.error = runtime().d_error;
    launch_kernel(sparse_stage1_umma_kernel, dim3(ceil_div(T, S1_TOKENS), hkv), dim3(S1_UMMA_THREADS), SMEM_BYTES, s, tm_q, tm_lse, tm_c1, a);
}
