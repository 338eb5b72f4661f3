// Prefill attention with two query tiles per CTA, sm_100a: what tree_attn_kernel computes with one key split, for launches of
// many query tiles (make_biased_attn_plan has the rule).
//
// What bounds it.  A 128-row query tile against 128 keys costs 1024 cycles of tensor pipe (S = Q K^T and P V, 128 x 128 x 128 each)
// and 1024 cycles of exponentials (16384 on the MUFU pipe).  With one tile per CTA the two follow one another with their latencies
// between them (2750 cycles per tile) and every tile fetches its own keys.  Here two tiles A and B share one fetch of the keys
// and the SM's pipes: about 4600 cycles for both, in which either pipe is busy for 2048.  The rest is the softmax's own chain: of a
// softmax thread's cycles by role clocks 1450 are exponentials and their stores, 800 waits for scores, 700 maxima, 300 the exchange of
// maxima, 260 waits for P V, 230 loads of scores; what is left are instructions between them.  576 threads leave 96 registers,
// and beside 64 scores a thread keeps 44 to 116 bytes of addresses and bounds in local memory.
// One tile / two tiles per CTA, 32 query heads on 2 key heads: 4096 causal rows 192 / 149 us, 2048 behind 30000 1330 / 1048
// (1.0 PFLOP/s).
// Probabilities in tensor memory (in the scores' place, tiles taking turns), which spares shared memory a third of its traffic, took the
// same 154 us as P in shared memory then did, and an issuing warp per tile 171: neither the memory nor the order of issue is the bound.
//   S            one buffer per tile in tensor memory; it is free as soon as the softmax holds the scores in registers, so S(i+1) is
//                computed while the softmax of iteration i runs
//   P            bf16 in shared memory, one buffer per tile; PV(i) runs under the next softmax
//   K, V         one stage each: K(i+2) is fetched from the end of S(i+1) on, V(i+1) from the end of PV(i) on, both most of an
//                iteration before they are needed
//   softmax      two threads per row, 64 keys each; the row maximum is exchanged through shared memory, once per iteration, by the two
//                warps of 32 rows alone
// Keys come in blocks of 64: thread half ch of iteration i works on block 2 i + ch.  Block-sparse mode lists the union of the
// two tiles' blocks, so an iteration's two blocks need not be neighbours.  The union of sixteen tokens is nearly all blocks where each
// sees an eighth of them, but a warp's 32 rows are two tokens (of 16 heads) and mostly see nothing: such a warp leaves out scores, maxima and
// exponentials and only keeps zeros in its part of P.  Which tokens of the pair see a listed block is one word in shared memory,
// filled once; read from the block mask in every iteration, the bits' latency stood before the wait for the scores.  Block-sparse, 2048 rows
// behind 30000 keys, 5, 13, 40 and 100 % of the blocks per token, before / now: 771 / 603, 1162 / 914, 1276 / 1159, 1111 / 1031 us;
// behind 9000, 13 %: 396 / 325.  Pairs of more than 32 tokens keep the mask's rows.
// A tile's P V takes only the blocks some row of that tile
// sees: a probability of zero does not hide an infinity or a NaN among the values, so no row meets values that the one-tile
// kernel would not have shown it.
// Tensor memory: S_A [0,128) S_B [128,256) O_A [256,384) O_B [384,512).
#include <algorithm>
#include <type_traits>

#include "attn_common.cuh"

using namespace attn;

namespace {

constexpr int BLK = 64;                       // keys per block
constexpr int BLK_BYTES = BLK * 128;          // 64 rows of a 64-column half
constexpr int TILE_THREADS = 256;             // softmax threads per query tile
constexpr int SOFT_WARPS = 2 * TILE_THREADS / 32;
constexpr int PAIR_THREADS = (SOFT_WARPS + 2) * 32;   // + MMA issuer, TMA producer
constexpr int PAIR_TMEM_COLS = 512, PAIR_TMEM_O = 256;
constexpr int MAX_BLOCKS = 4096;              // 262144 keys (block-sparse mode)
// How a thread learns which blocks its token sees: all, from the token's row of the block mask, or from a word per listed block with
// a bit per token of the pair (at most 32 tokens)
enum { DENSE = 0, BY_ROW = 1, BY_WORD = 2 };

template <int DK, int DV>
struct PairCfg {
    static constexpr int Q_TILE = ROWS * DK * 2, K_TILE = KEYS * DK * 2, V_TILE = KEYS * DV * 2, P_TILE = ROWS * KEYS * 2;
    static constexpr int SMEM_Q = 0;                             // 2 tiles
    static constexpr int SMEM_K = SMEM_Q + 2 * Q_TILE;
    static constexpr int SMEM_V = SMEM_K + K_TILE;
    static constexpr int SMEM_P = SMEM_V + V_TILE;               // 2 tiles
    static constexpr int SMEM_LIST = SMEM_P + 2 * P_TILE;        // block numbers, 16 bits each
    static constexpr int SMEM_UNION = SMEM_LIST + MAX_BLOCKS * 2;    // 64 words of 64 blocks, then 65 prefix counts
    static constexpr int SMEM_SEEN = SMEM_UNION + 64 * 8 + 320;  // [2 tiles] the words of that tile alone
    static constexpr int SMEM_XCH = SMEM_SEEN + 2 * 64 * 8;      // [2 tiles][2 buffers][2 halves][128] floats
    static constexpr int SMEM_WORD = SMEM_XCH + 8 * ROWS * 4;    // BY_WORD: [MAX_BLOCKS] words
    static constexpr int SMEM_CTRL = SMEM_WORD + MAX_BLOCKS * 4;
    static constexpr int SMEM_TOTAL = SMEM_CTRL + 256 + 1024;
    static_assert(SMEM_TOTAL <= 232448, "shared memory budget");
};

template <int DK, int DV, bool BIASED, int SPARSE>
__global__ void __launch_bounds__(PAIR_THREADS, 1)
pair_attn_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                 const __grid_constant__ CUtensorMap tm_v, const AttnArgs a) {
    using C = PairCfg<DK, DV>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::SMEM_CTRL);
    uint64_t* q_bar = bars;
    uint64_t* k_full = bars + 1;
    uint64_t* v_full = bars + 2;
    uint64_t* k_empty = bars + 3;
    uint64_t* v_empty = bars + 4;
    uint64_t* s_bar = bars + 5;     // [2 tiles]  S(i) is in TMEM
    uint64_t* s_free = bars + 7;    // [2 tiles]  S(i) has been read
    uint64_t* p_ready = bars + 9;   // [2 tiles]  P(i) is in shared memory
    uint64_t* o_bar = bars + 11;    // [2 tiles]  PV(i) is done
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 13);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    uint16_t* list = reinterpret_cast<uint16_t*>(smem + C::SMEM_LIST);
    unsigned long long* uni = reinterpret_cast<unsigned long long*>(smem + C::SMEM_UNION);
    int* uni_at = reinterpret_cast<int*>(uni + 64);
    unsigned long long* seen = reinterpret_cast<unsigned long long*>(smem + C::SMEM_SEEN);
    int* run = uni_at + 65;
    uint32_t* words = reinterpret_cast<uint32_t*>(smem + C::SMEM_WORD);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    grid_dep_trigger();
    const int n_pairs = (a.num_mtiles + 1) / 2;
    // longest first over all key heads (tiles that need more keys have higher numbers)
    const int mt0 = 2 * (n_pairs - 1 - static_cast<int>(blockIdx.x) / a.hkv);
    const int h = blockIdx.x % a.hkv;     // kv head

    if (tid == 0) {
        ptx::mbar_init(q_bar, 1);
        ptx::mbar_init(k_full, 1);
        ptx::mbar_init(v_full, 1);
        ptx::mbar_init(k_empty, 1);
        ptx::mbar_init(v_empty, 1);
        for (int i = 0; i < 2; ++i) {
            ptx::mbar_init(&s_bar[i], 1);
            ptx::mbar_init(&o_bar[i], 1);
            ptx::mbar_init(&s_free[i], TILE_THREADS / 32);    // one arrival per softmax warp
            ptx::mbar_init(&p_ready[i], TILE_THREADS / 32);
        }
        *abort_flag = 0;
        ptx::mbar_fence_init();
        ptx::prefetch_tensormap(&tm_q);
        ptx::prefetch_tensormap(&tm_k);
        ptx::prefetch_tensormap(&tm_v);
    }
    if (warp == 0) {
        ptx::tmem_alloc(tmem_slot, PAIR_TMEM_COLS);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    grid_dep_wait();

    // ---- geometry: the pair's tokens [t0, t_end) and the blocks any of its rows may see
    const int kv_total = *a.kv_len + a.kv_len_add;
    const int tq_eff = (a.n_valid != nullptr) ? min(*a.n_valid, a.tq) : a.tq;
    const int causal_base = kv_total - tq_eff;   // token t sees keys < causal_base + t + 1
    const int t0 = mt0 * a.tok_per_tile;
    const int t_end = min(t0 + 2 * a.tok_per_tile, tq_eff);
    int key_hi = (t_end > t0) ? min(kv_total, causal_base + t_end) : 0;
    if (key_hi < 0) key_hi = 0;
    // first key of a tile's rows under the draft layer's block-granular window (see tree_attn_kernel)
    auto tile_lo = [&](int first_token) {
        int lo = 0;
        if (a.window > 0) {
            const int lo_blk = (causal_base + (first_token / 64) * 64 + KEYS - 1) / KEYS - a.window / KEYS;
            if (lo_blk > 0) lo = lo_blk * KEYS;
        }
        return lo;
    };
    int key_lo = tile_lo(t0);
    if (BIASED && a.exact_window > 0) key_lo = max(causal_base + t0 - a.exact_window + 1, 0);
    const int blk_lo = key_lo / BLK;
    const int blk_hi = (key_hi + BLK - 1) / BLK;
    // blocks [lo, hi) that rows of one of the two tiles may see
    auto tile_blocks = [&](int tile, int& lo, int& hi) {
        const int first = t0 + tile * a.tok_per_tile, end = min(first + a.tok_per_tile, tq_eff);
        lo = (BIASED && a.exact_window > 0 ? max(causal_base + first - a.exact_window + 1, 0) : tile_lo(first)) / BLK;
        hi = end > first ? (max(min(kv_total, causal_base + end), 0) + BLK - 1) / BLK : 0;
    };
    int n_blk = max(blk_hi - blk_lo, 0);

    constexpr bool sparse = SPARSE != DENSE;
    if (sparse) {
        if (tid == 0) { run[0] = 0; run[1] = MAX_BLOCKS; }
        if (tid < 128) {   // 64 words of each tile
            const int tile = tid >> 6, word = tid & 63;
            const int first = t0 + tile * a.tok_per_tile, end = min(first + a.tok_per_tile, t_end);
            unsigned long long m = 0ull;
            if (word < a.bm_words) {
                const uint64_t* r = a.blockmask + (static_cast<size_t>(h) * a.tq + first) * a.bm_words + word;
                for (int t = first; t < end; ++t, r += a.bm_words) m |= *r;
            }
            // the trailing window of the tile's first token reaches furthest back
            const int left = max((first + causal_base + 63) / 64 - a.block_window, 0);
            const int b0 = word * 64;
            auto from = [&](int b) -> unsigned long long { return b <= b0 ? ~0ull : b >= b0 + 64 ? 0ull : ~0ull << (b - b0); };
            int lo, hi;
            tile_blocks(tile, lo, hi);
            seen[tid] = (m | from(left)) & from(lo) & ~from(min(hi, MAX_BLOCKS));
        }
        __syncthreads();
        if (tid < 64) uni[tid] = seen[tid] | seen[64 + tid];
        __syncthreads();
        if (warp == 0) {   // exclusive prefix counts of the 64 words, two per lane
            const int c0 = __popcll(uni[2 * lane]), c1 = __popcll(uni[2 * lane + 1]);
            int sum = c0 + c1;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += v;
            }
            uni_at[2 * lane] = sum - c0 - c1;
            uni_at[2 * lane + 1] = sum - c1;
            if (lane == 31) uni_at[64] = sum;
        }
        __syncthreads();
        n_blk = uni_at[64];
        if (tid < 512) {   // eight blocks per thread
            const int word = tid >> 3, bit0 = (tid & 7) * 8;
            const unsigned long long m = uni[word], shared = seen[word] & seen[64 + word];
            int at = uni_at[word] + __popcll(m & ((1ull << bit0) - 1ull));
            int lo = 0, hi = n_blk;
            for (int k = bit0; k < bit0 + 8; ++k) {
                if (!((m >> k) & 1ull)) continue;
                if (!((shared >> k) & 1ull)) {
                    if (2 * at < n_blk) lo = at + 1;
                    else hi = min(hi, at);
                }
                list[at++] = static_cast<uint16_t>(word * 64 + k);
            }
            lo = __reduce_max_sync(0xffffffffu, lo);
            hi = __reduce_min_sync(0xffffffffu, hi);
            if (lane == 0) {
                if (lo > 0) atomicMax(run, lo);
                if (hi < n_blk) atomicMin(run + 1, hi);
            }
        }
        __syncthreads();
        if (SPARSE == BY_WORD) {
            for (int j = tid; j < n_blk; j += PAIR_THREADS) {
                const int b = list[j];
                uint32_t w = 0;
                const uint64_t* r = a.blockmask + (static_cast<size_t>(h) * a.tq + t0) * a.bm_words + (b >> 6);
                for (int t = t0; t < t_end; ++t, r += a.bm_words) {
                    const bool sees = b >= (t + causal_base + 63) / 64 - a.block_window || ((b >> 6) < a.bm_words && ((*r >> (b & 63)) & 1ull));
                    w |= static_cast<uint32_t>(sees) << (t - t0);
                }
                words[j] = w;
            }
            __syncthreads();
        }
    }
    const int n_it = (n_blk + 1) / 2;
    auto block_of = [&](int j) -> int { return sparse ? list[min(j, n_blk - 1)] : blk_lo + j; };

    if (warp == SOFT_WARPS) {
        // ================================================= MMA issue
        if (lane == 0 && n_it > 0) {
            int lo_a, hi_a, lo_b, hi_b;
            tile_blocks(0, lo_a, hi_a);
            tile_blocks(1, lo_b, hi_b);
            auto tile_sees = [&](int tile, int b) -> bool {
                return sparse ? (seen[64 * tile + (b >> 6)] >> (b & 63)) & 1ull : b >= (tile ? lo_b : lo_a) && b < (tile ? hi_b : hi_a);
            };
            // iterations [whole_lo, whole_hi) have two blocks that both tiles see: the longest stretch in the middle of the list
            const int whole_lo = ((sparse ? run[0] : max(lo_b - blk_lo, 0)) + 1) / 2, whole_hi = (sparse ? min(run[1], n_blk) : max(min(hi_a, hi_b) - blk_lo, 0)) / 2;
            constexpr uint32_t idesc_s = ptx::umma_idesc_bf16(ROWS, KEYS, 0, 0);
            constexpr uint32_t idesc_o = ptx::umma_idesc_bf16(ROWS, DV, 0, 1);
            const uint32_t q_addr = ptx::smem_u32(smem + C::SMEM_Q), k_addr = ptx::smem_u32(smem + C::SMEM_K),
                           v_addr = ptx::smem_u32(smem + C::SMEM_V), p_addr = ptx::smem_u32(smem + C::SMEM_P);
            // descriptors of the first 16 columns or rows; one further on is its distance in 16-byte units away
            const uint64_t q_desc = ptx::umma_desc_sw128(q_addr, 16, 1024), k_desc = ptx::umma_desc_sw128(k_addr, 16, 1024),
                           p_desc = ptx::umma_desc_sw128(p_addr, 16, 1024), v_desc = ptx::umma_desc_sw128(v_addr, HALF_BYTES, 1024);
            auto issue_s = [&](int tile) {
#pragma unroll
                for (int j = 0; j < DK / 16; ++j) {
                    const int off = (j >> 2) * HALF_BYTES + (j & 3) * 32;
                    ptx::umma_ss(tmem_base + tile * KEYS, q_desc + (tile * C::Q_TILE + off) / 16, k_desc + off / 16, idesc_s, j ? 1u : 0u);
                }
                ptx::umma_commit(&s_bar[tile]);
            };
            // bit 2 tile + j: some row of the tile sees block j of iteration i
            auto blocks_of = [&](int i) -> uint32_t {
                uint32_t f = 0;
                for (int j = 0; j < 2; ++j) {
                    if (2 * i + j >= n_blk) break;
                    const int b = block_of(2 * i + j);
                    for (int tile = 0; tile < 2; ++tile) f |= static_cast<uint32_t>(tile_sees(tile, b)) << (2 * tile + j);
                }
                return f;
            };
            uint32_t begun = 0;   // tiles whose O holds something
            // O += P V of a tile, for all 128 keys or for one block of 64
            auto issue_pv = [&](int tile, int kk0, int steps, uint32_t acc) {
#pragma unroll
                for (int kk = kk0; kk < kk0 + steps; ++kk) {
                    // A: P, K-major: 64-key half (kk / 4), 32 B per 16-key step inside it;  B: V, N-major: 16 key rows of 128 B per
                    // step, 64-wide halves of the value columns HALF_BYTES apart
                    ptx::umma_ss(tmem_base + PAIR_TMEM_O + tile * 128, p_desc + (tile * C::P_TILE + (kk >> 2) * HALF_BYTES + (kk & 3) * 32) / 16,
                                 v_desc + kk * 16 * 128 / 16, idesc_o, kk > kk0 ? 1u : acc);
                }
            };
            bool w = ptx::mbar_wait(q_bar, 0, abort_flag) && ptx::mbar_wait(k_full, 0, abort_flag);
            if (w) {
                ptx::tc_fence_after();
                issue_s(0);
                issue_s(1);
                ptx::umma_commit(k_empty);
            }
            auto iterate = [&](int i, auto whole) {   // whole: both tiles see both blocks
                if (i + 1 < n_it) {
                    w = ptx::mbar_wait(k_full, (i + 1) & 1, abort_flag);
                    for (int tile = 0; w && tile < 2; ++tile) {
                        w = ptx::mbar_wait(&s_free[tile], i & 1, abort_flag);
                        if (!w) break;
                        ptx::tc_fence_after();
                        issue_s(tile);
                    }
                    if (!w) return;
                    ptx::umma_commit(k_empty);
                }
                const uint32_t blocks = decltype(whole)::value ? 15u : blocks_of(i);
                w = ptx::mbar_wait(v_full, i & 1, abort_flag);
                for (int tile = 0; w && tile < 2; ++tile) {
                    w = ptx::mbar_wait(&p_ready[tile], i & 1, abort_flag);
                    if (!w) break;
                    ptx::tc_fence_after();
                    const uint32_t own = (blocks >> (2 * tile)) & 3u, old = (begun >> tile) & 1u;
                    if (decltype(whole)::value) {
                        issue_pv(tile, 0, KEYS / 16, old);
                    } else {
                        if (own & 1u) issue_pv(tile, 0, BLK / 16, old);
                        if (own & 2u) issue_pv(tile, BLK / 16, BLK / 16, old | (own & 1u));
                    }
                    begun |= own != 0u ? 1u << tile : 0u;
                    ptx::umma_commit(&o_bar[tile]);
                }
                if (w) ptx::umma_commit(v_empty);
            };
            int i = 0;
            for (; w && i < min(whole_lo, n_it); ++i) iterate(i, std::false_type{});
            for (; w && i < whole_hi; ++i) iterate(i, std::true_type{});
            for (; w && i < n_it; ++i) iterate(i, std::false_type{});
        }
    } else if (warp == SOFT_WARPS + 1) {
        // ================================================= TMA producer
        if (lane == 0 && n_it > 0) {
            // rows of a tile beyond grp * tok_per_tile keep whatever shared memory held; nothing of them is stored
            ptx::mbar_arrive_expect_tx(q_bar, 2 * a.grp * a.tok_per_tile * DK * 2);
#pragma unroll
            for (int tile = 0; tile < 2; ++tile) {
#pragma unroll
                for (int c = 0; c < DK / 64; ++c) {
                    ptx::tma_load_3d(smem + C::SMEM_Q + tile * C::Q_TILE + c * HALF_BYTES, &tm_q, q_bar, c * 64, h * a.grp,
                                     t0 + tile * a.tok_per_tile);
                }
            }
            bool w = true;
            auto load = [&](uint64_t* full, uint64_t* empty, uint8_t* dst, const CUtensorMap* tm, int halves, int i, uint32_t bytes) {
                if (!w || i >= n_it) return;
                w = ptx::mbar_wait(empty, (i & 1) ^ 1, abort_flag);
                if (!w) return;
                ptx::mbar_arrive_expect_tx(full, bytes);
                for (int j = 0; j < 2; ++j) {
                    const int key = block_of(2 * i + j) * BLK;
                    for (int c = 0; c < halves; ++c) ptx::tma_load_2d(dst + c * HALF_BYTES + j * BLK_BYTES, tm, full, h * halves * 64 + c * 64, key);
                }
            };
            auto load_k = [&](int i) { load(k_full, k_empty, smem + C::SMEM_K, &tm_k, DK / 64, i, C::K_TILE); };
            auto load_v = [&](int i) { load(v_full, v_empty, smem + C::SMEM_V, &tm_v, DV / 64, i, C::V_TILE); };
            load_k(0);
            load_v(0);
            load_k(1);
            for (int i = 0; w && i < n_it; ++i) {   // in the order their buffers become free: S(i+1) ends before PV(i)
                load_k(i + 2);
                load_v(i + 1);
            }
            if (!w) {
                // give copies already in flight time to land before the CTA retires
                const long long c0 = clock64();
                while (clock64() - c0 < 2000000LL) {}
            }
        }
    } else {
        // ================================================= softmax
        const int tile = warp >> 3;
        const int ch = (warp >> 2) & 1;              // block of the iteration
        const int row = (warp & 3) * 32 + lane;      // query row of the tile == TMEM lane
        const int tt0 = t0 + tile * a.tok_per_tile;
        const int t = tt0 + row / a.grp;             // query token
        const int qh = h * a.grp + row % a.grp;      // query head
        const bool row_in = !BIASED || row < a.grp * a.tok_per_tile;   // 128 need not be a multiple of grp
        const bool row_valid = row_in && (t < tq_eff);
        int limit = row_valid ? min(kv_total, causal_base + t + 1) : 0;
        if (limit < 0) limit = 0;
        const int mbeg = (a.mask != nullptr) ? (kv_total - a.mask_k) : 0x7fffffff;
        const uint64_t mword = (a.mask != nullptr && row_valid) ? a.mask[t] : ~0ull;
        const int row_lo = (BIASED && a.exact_window > 0) ? max(causal_base + t - a.exact_window + 1, 0) : tile_lo(tt0);
        const bool biased = BIASED && a.bias_exp > 0.f;
        const float slope2 =   // log2(e) * slope of this row's head
            biased ? 1.4426950408889634f * exp2f(-a.bias_exp * static_cast<float>(qh + 1) / static_cast<float>(a.hq)) : 0.f;
        const float sl2 = biased ? 1.f : a.scale_log2;   // biased scores are brought to log2 units as they are read
        const int win_left = SPARSE == BY_ROW ? (t + causal_base + 63) / 64 - a.block_window : 0;
        const uint64_t* bm_row = (SPARSE == BY_ROW && row_valid) ? a.blockmask + (static_cast<size_t>(h) * a.tq + t) * a.bm_words : nullptr;
        const uint32_t lane_sel = static_cast<uint32_t>((warp & 3) * 32) << 16;
        const uint32_t tmem_s = tmem_base + lane_sel + tile * KEYS + ch * 64;
        const uint32_t tmem_o = tmem_base + lane_sel + PAIR_TMEM_O + tile * 128 + ch * (DV / 2);
        float* xch = reinterpret_cast<float*>(smem + C::SMEM_XCH) + tile * 4 * ROWS;
        uint8_t* p_half = smem + C::SMEM_P + tile * C::P_TILE + ch * HALF_BYTES + row * 128;
        const int bar_id = 1 + tile * 4 + (warp & 3);   // the two warps of these 32 rows
        float m_run = -INFINITY;  // running max of raw scores (same in both threads of a row)
        float l_run = 0.f;        // this thread's share of the running sum
        // BY_WORD: the tokens of this warp's 32 rows
        const int tok0 = tile * a.tok_per_tile + (warp & 3) * 32 / a.grp;
        const uint32_t warp_tokens = SPARSE == BY_WORD ? ((a.grp < 32 ? (1u << (32 / a.grp)) - 1u : 1u) << tok0) : 0u;
        bool zeros = false;   // BY_WORD: this thread's part of P holds zeros
        bool ok = true;
        for (int i = 0; i < n_it; ++i) {
            const int j = 2 * i + ch;
            const int b = block_of(j);
            const int key0 = b * BLK;
            bool blk_ok = j < n_blk;
            bool any = true;   // some row of this warp sees the block; where none does, neither scores nor exponentials are needed
            if (SPARSE == BY_WORD) {
                const uint32_t w = words[min(j, n_blk - 1)];
                blk_ok = blk_ok && ((w >> (t - t0)) & 1u);
                any = j < n_blk && (w & warp_tokens) != 0u;
            }
            if (SPARSE == BY_ROW) {
                blk_ok = blk_ok && (b >= win_left || (bm_row != nullptr && (b >> 6) < a.bm_words && ((bm_row[b >> 6] >> (b & 63)) & 1ull)));
            }
            ok = ok && ptx::mbar_wait_warp(&s_bar[tile], i & 1, abort_flag);
            if (!ok) {
                for (int k = i; k < n_it; ++k) ptx::named_bar_sync(bar_id, 64);   // every warp arrives equally often
                break;
            }
            ptx::tc_fence_after();
            uint32_t sc[64];
            if (any) {
                ptx::tmem_ld32(tmem_s, sc);
                ptx::tmem_ld32(tmem_s + 32, sc + 32);
                ptx::tmem_wait_ld();
            }
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&s_free[tile]);
            float m_half = -INFINITY;
            if (any) {
                if (biased) {
                    const float b0 = slope2 * static_cast<float>(key0 - (causal_base + t));   // <= 0 where the key is visible
#pragma unroll
                    for (int c = 0; c < 64; ++c) {
                        sc[c] = __float_as_uint(fmaf(__uint_as_float(sc[c]), a.scale_log2, fmaf(slope2, static_cast<float>(c), b0)));
                    }
                }
                // visibility of this thread's 64 keys as one word: causal bound, window bound, tree-mask bits, block selection
                uint64_t vb = ~0ull;
                if (!blk_ok || limit <= key0 || row_lo >= key0 + 64) {
                    vb = 0ull;
                } else {
                    if (limit < key0 + 64) vb &= (1ull << (limit - key0)) - 1ull;
                    if (row_lo > key0) vb &= ~((1ull << (row_lo - key0)) - 1ull);
                    const int mo = mbeg - key0;  // first column the tree mask applies to (mbeg is huge when there is none)
                    if (mo < 64) {
                        const uint64_t tm = (mo >= 0) ? ((mo > 0 ? (mword << mo) : mword) | ((1ull << mo) - 1ull))
                                                      : ((-mo < 64) ? (mword >> (-mo)) : 0ull);
                        vb &= tm;
                    }
                }
                if (vb != ~0ull) {
#pragma unroll
                    for (int c = 0; c < 64; ++c) {
                        if (!((vb >> c) & 1ull)) sc[c] = 0xff800000u;  // -inf
                    }
                }
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int c = 0; c < 64; c += 8) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) mx[e] = fmaxf(mx[e], fmaxf(__uint_as_float(sc[c + e]), __uint_as_float(sc[c + 4 + e])));
                }
                m_half = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            }
            // the buffer of iteration i is written again in i + 2, past the barrier of i + 1
            float* xb = xch + (i & 1) * 2 * ROWS;
            xb[ch * ROWS + row] = m_half;
            ptx::named_bar_sync(bar_id, 64);
            const float m_tile = fmaxf(m_half, xb[(ch ^ 1) * ROWS + row]);
            // lazy running maximum, as in tree_attn_kernel: it moves only for a new one more than 2^8 above it
            float m_new = m_run;
            if (m_tile != -INFINITY && (m_run == -INFINITY || (m_tile - m_run) * sl2 > 8.f)) m_new = m_tile;
            const float m_use = (m_new == -INFINITY) ? 0.f : m_new;
            const float alpha = (m_run == -INFINITY) ? 1.f : fast_exp2((m_run - m_use) * sl2);
            if (i > 0) {   // PV(i-1) is done: O may change, and P may be written
                ok = ptx::mbar_wait_warp(&o_bar[tile], (i - 1) & 1, abort_flag);
                ptx::tc_fence_after();
            }
            if (ok && i > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll 1
                for (int c0 = 0; c0 < DV / 2; c0 += 16) {
                    uint32_t r[16];
                    ptx::tmem_ld16(tmem_o + c0, r);
                    ptx::tmem_wait_ld();
#pragma unroll
                    for (int c = 0; c < 16; ++c) r[c] = __float_as_uint(__uint_as_float(r[c]) * alpha);
                    ptx::tmem_st16(tmem_o + c0, r);
                }
                ptx::tmem_wait_st();
            }
            m_run = m_new;
            if (any) {
                // P = 2^((s - m) * scale) in bf16 into the swizzled A-operand tile; row sums in fp32
                const float m_off = m_use * sl2;
                float ls[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int c8 = 0; c8 < 8; ++c8) {
                    uint4 pk;
                    uint32_t* w = reinterpret_cast<uint32_t*>(&pk);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float p0 = fast_exp2(fmaf(__uint_as_float(sc[c8 * 8 + 2 * e]), sl2, -m_off));
                        const float p1 = fast_exp2(fmaf(__uint_as_float(sc[c8 * 8 + 2 * e + 1]), sl2, -m_off));
                        ls[(2 * e) & 3] += p0;
                        ls[(2 * e + 1) & 3] += p1;
                        const __nv_bfloat162 b2 = __floats2bfloat162_rn(p0, p1);
                        w[e] = *reinterpret_cast<const uint32_t*>(&b2);
                    }
                    *reinterpret_cast<uint4*>(p_half + ((c8 ^ (row & 7)) << 4)) = pk;
                }
                l_run = l_run * alpha + ((ls[0] + ls[1]) + (ls[2] + ls[3]));
            } else {
                l_run *= alpha;
                if (!zeros) {
#pragma unroll
                    for (int c8 = 0; c8 < 8; ++c8) *reinterpret_cast<uint4*>(p_half + ((c8 ^ (row & 7)) << 4)) = make_uint4(0u, 0u, 0u, 0u);
                }
            }
            if (SPARSE == BY_WORD) zeros = !any;
            ptx::fence_proxy_async_smem();  // P stores -> visible to the tensor core's async proxy
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&p_ready[tile]);
        }
        if (ok && n_it > 0) {
            ok = ptx::mbar_wait_warp(&o_bar[tile], (n_it - 1) & 1, abort_flag);
            ptx::tc_fence_after();
        }
        // ---- write-out.  TMEM reads are warp-collective, so every thread runs them and only the stores depend on the row.
        float* xb = xch + (n_it & 1) * 2 * ROWS;   // the last maxima went through the other buffer
        xb[ch * ROWS + row] = l_run;
        ptx::named_bar_sync(bar_id, 64);
        float l_row = l_run + xb[(ch ^ 1) * ROWS + row];
        if (BIASED && a.sink != 0 && m_run != -INFINITY) l_row += exp2f(-m_run * sl2);
        if (ok) {
            const bool store = row_in && (t < a.tq);
            const float inv = (l_row > 0.f) ? (BIASED ? a.out_scale : 1.f) / l_row : 0.f;
            const bool none = l_row == 0.f;   // a row that sees no key: its tile's O may never have been written
            bf16* dst = a.out + static_cast<size_t>(store ? t : 0) * a.out_ld + qh * (BIASED ? a.out_cols : DV) + ch * (DV / 2);
            const int cols = BIASED ? a.out_cols - ch * (DV / 2) : DV / 2;   // real columns of this thread's half
            const bool whole = !BIASED || (a.out_cols % 8 == 0 && a.out_ld % 8 == 0);
#pragma unroll 1
            for (int c0 = 0; c0 < DV / 2; c0 += 32) {
                uint32_t r[32];
                if (n_it > 0) {  // uniform across the CTA
                    ptx::tmem_ld32(tmem_o + c0, r);
                    ptx::tmem_wait_ld();
                }
                if (n_it == 0 || none) {
#pragma unroll
                    for (int c = 0; c < 32; ++c) r[c] = 0;
                }
                if (store) {
#pragma unroll
                    for (int c = 0; c < 32; c += 8) {
                        uint4 pk;
                        uint32_t* w = reinterpret_cast<uint32_t*>(&pk);
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const __nv_bfloat162 b2 = __floats2bfloat162_rn(__uint_as_float(r[c + e * 2]) * inv, __uint_as_float(r[c + e * 2 + 1]) * inv);
                            w[e] = *reinterpret_cast<const uint32_t*>(&b2);
                        }
                        if (!BIASED || (whole && c0 + c < cols)) {
                            *reinterpret_cast<uint4*>(dst + c0 + c) = pk;
                        } else if (!whole) {   // a head width that 16-byte stores do not fit
                            const bf16* e8 = reinterpret_cast<const bf16*>(&pk);
#pragma unroll
                            for (int e = 0; e < 8; ++e) {
                                if (c0 + c + e < cols) dst[c0 + c + e] = e8[e];
                            }
                        }
                    }
                }
            }
        }
    }

    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem_base, PAIR_TMEM_COLS);
    }
    if (tid == 0 && *abort_flag) atomicOr(a.error, ERR_ATTN_TIMEOUT);
}

template <int DK, int DV, bool BIASED, int SPARSE = DENSE>
void launch(const AttnPlan& p, const AttnArgs& a, cudaStream_t s) {
    static bool configured = false;
    if (!configured) {
        CUDA_CHECK(cudaFuncSetAttribute(pair_attn_kernel<DK, DV, BIASED, SPARSE>, cudaFuncAttributeMaxDynamicSharedMemorySize, PairCfg<DK, DV>::SMEM_TOTAL));
        configured = true;
    }
    launch_kernel(pair_attn_kernel<DK, DV, BIASED, SPARSE>, dim3(ceil_div(a.num_mtiles, 2) * p.hkv), dim3(PAIR_THREADS), PairCfg<DK, DV>::SMEM_TOTAL, s,
                  p.tm_q, p.tm_k, p.tm_v, a);
}

}  // namespace

void launch_pair_attention(const AttnPlan& p, const AttnArgs& a, cudaStream_t s) {
    CPM_REQUIRE(!p.biased || p.blockmask == nullptr, "attention: a block mask needs an unbiased plan");
    if (!p.biased && p.blockmask == nullptr) launch<128, 128, false>(p, a, s);
    else if (!p.biased && 2 * a.tok_per_tile <= 32) launch<128, 128, false, BY_WORD>(p, a, s);
    else if (!p.biased) launch<128, 128, false, BY_ROW>(p, a, s);
    else if (p.d == 128 && p.dv == 128) launch<128, 128, true>(p, a, s);
    else if (p.d == 128) launch<128, 64, true>(p, a, s);
    else if (p.dv == 128) launch<64, 128, true>(p, a, s);
    else launch<64, 64, true>(p, a, s);
}
