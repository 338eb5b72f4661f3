// Products of ONE token row with bf16 weights: y[N] = x[K] W[N,K]^T, alone (LinearPlan) or grouped by expert
// (MoeGemmPlan), with the SwiGLU and clamped-gate epilogues of the tensor-core kernels.
//
// Bound: the weights' bytes from HBM, 2 FLOP each, so the tensor cores have nothing to do, and what the tile kernels need
// before the first byte arrives (tensor memory, descriptors, barriers) and after the last one (tensor memory back to
// registers, pieces of split tiles summed through a workspace) is most of a product of a few megabytes.  Here a CTA
// owns R output rows over the whole of K: eight lanes read 128 consecutive bytes of one row (the tile-major
// layout keeps the R rows of a k-block together), the eight warps take k-blocks in turn, and only sums of one CTA
// meet.  A warp keeps eight 16-byte loads per lane in flight, the first of them before the wait for the predecessor.  About
// 20 instructions per 16 bytes leave three quarters of the issue slots free at the HBM rate.
// Back to back, weights from HBM, tensor-core tiles / this: 2048 x 2048 7.0 / 2.6 us, 2048 x 8192 11.0 / 7.4, 4096 x 16384 22.8 / 19.9,
// 73448 x 4096 88 / 83 (7.2 TB/s); 512 x 256 3.7 / 3.3.
#include "common.cuh"
#include "layered.cuh"
#include "row_ops.cuh"

namespace {

constexpr int ONE_WARPS = 8;
constexpr int TILE_ROWS = 128, BLOCK_COLS = 64;           // tile-major layout (linear_weight_elems)
constexpr int BLOCK_ELEMS = TILE_ROWS * BLOCK_COLS;

struct OneRowArgs {
    const bf16 *w, *x, *xs;
    bf16* y;
    const bf16* bias;
    int N, kblocks, ctas;            // one matrix
    int N_s, kblocks_s, ctas_s;      // the shared expert's (or the grouped product's extra one); ctas_s = 0: none
    long long stride, w_s;           // elements from one matrix to the next; the shared one's start
    int ldx, ldy, xs_row, ys_row;
    const int4* entries;             // router's choice: {expert, input row, output row, 1}
    const int32_t* n_entries;
    int uniform;                     // > 0: matrix i has row i of x and y
    int ahead;                       // !EARLY: the shared matrix's CTAs run beside the router (LaunchOrder)
    float gate_limit, gate_alpha;
    RopeRow rope;                    // ROPE
    SideRow side;                    // SIDE
};

// A plain load that the compiler keeps in its place, not a read-only one: with ld.global.nc a product's first loads did not run beside its
// predecessor's end (one token of 8 layers of 2048: 447 us a pass, 418 with plain loads; 6 layers of 4096 with experts 683 and 666).
__device__ __forceinline__ uint4 load_stream(const bf16* p) {
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ f32x2 widen(uint32_t two) { return pair(__uint_as_float(two << 16), __uint_as_float(two & 0xffff0000u)); }

// PLAIN, GATED: the rows are R / 2 gate rows and the R / 2 up rows of the same features (64 + 64 in a tile), ROPE: a tile is a head of 128, the
// rows are R / 2 of its lower half and their partners of the upper half; queries are rotated, keys rotated and values copied into the cache.
// SIDE: the output is gated into the token's side input.
enum Epilogue { PLAIN, GATED, ROPE, SIDE };
// Rotation and append as a launch of their own cost 1.7 us a layer (8 layers of 2048: 418 us a pass, 410 with them here).
// EARLY: the router's choice may be read before the wait for the predecessor.  Without it (gate/up) the launch lets its successor start after its own
// wait, and right behind a router that starts it only when the row exists, the shared matrix's CTAs compute and store beside it, with no wait
// (ahead).  The other CTAs of the launch wait, and so it still ends after the router.  The router is 8 us of latency on five CTAs: 32 tokens of six layers
// of 4096 with a shared expert of 4096 took 24.7 ms, now 22.5.
// HOLD: the successor starts only after this launch's wait; it may then run beside this launch on what was there before it.
template <int R, Epilogue EPI, bool EARLY, bool HOLD>
__global__ void __launch_bounds__(ONE_WARPS * 32, 4)
one_row_kernel(const OneRowArgs a) {
    constexpr bool PAIR = EPI == GATED || EPI == ROPE;
    constexpr int LOADS = R / 4;                       // per lane and k-block
    constexpr int U = 8 / LOADS;                       // k-blocks per batch
    __shared__ float part[ONE_WARPS][R];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (EARLY && !HOLD) grid_dep_trigger();

    const bool shared = static_cast<int>(blockIdx.x) < a.ctas_s;
    const int b = shared ? blockIdx.x : blockIdx.x - a.ctas_s;
    const int g = shared ? 0 : b / a.ctas;
    const int c = b - g * a.ctas;
    int4 e = make_int4(g, g, g, 1);
    bool there = true, waited = false;
    if (!shared && a.uniform == 0) {
        if (!EARLY) {
            grid_dep_wait();
            grid_dep_trigger();
            waited = true;
        }
        there = g < __ldcg(a.n_entries);
        if (there) e = __ldcg(a.entries + g);
    }
    const int N = shared ? a.N_s : a.N, kblocks = shared ? a.kblocks_s : a.kblocks;
    const int first = c * (PAIR ? R / 2 : R);          // output
    const int tile = first / (PAIR ? 64 : TILE_ROWS), r0 = first % (PAIR ? 64 : TILE_ROWS);
    const bf16* w = a.w + (shared ? a.w_s : static_cast<long long>(e.x) * a.stride) + static_cast<size_t>(tile) * kblocks * BLOCK_ELEMS +
                    (r0 + (lane >> 3)) * BLOCK_COLS + (lane & 7) * 8;

    uint4 wv[U][LOADS];
    auto load = [&](int kb0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int kb = kb0 + u * ONE_WARPS;
#pragma unroll
            for (int i = 0; i < LOADS; ++i) {
                const int row = PAIR && i >= LOADS / 2 ? 64 + (i - LOADS / 2) * 4 : i * 4;
                wv[u][i] = there && kb < kblocks ? load_stream(w + static_cast<size_t>(kb) * BLOCK_ELEMS + row * BLOCK_COLS) : make_uint4(0u, 0u, 0u, 0u);
            }
        }
    };
    load(warp);
    const bool ahead = !EARLY && shared && a.ahead != 0;
    if (!waited) {
        if (!ahead) grid_dep_wait();
        if (!EARLY || HOLD) grid_dep_trigger();
    }
    if (!there) return;
    int pos = 0, kv_len = 0, valid = 1;
    if (EPI == ROPE && threadIdx.x < R / 2) {   // here before the sums are
        pos = a.rope.pos != nullptr ? *a.rope.pos : *a.rope.pos_base + a.rope.pos_off;
        kv_len = *a.rope.kv_len;
        if (a.rope.n_valid != nullptr) valid = *a.rope.n_valid;
    }
    const bf16* x = (shared ? a.xs + static_cast<size_t>(a.xs_row) * a.ldx
                            : a.x + static_cast<size_t>(a.uniform > 0 || PAIR ? e.y : e.z) * a.ldx) + (lane & 7) * 8;
    float side = 0.f;
    if (EPI == SIDE && threadIdx.x < R && first + static_cast<int>(threadIdx.x) < N) {
        int id = *a.side.ids;
        if (id < 0 || id >= a.side.vocab) id = 0;   // reported by the embedding
        side = __bfloat162float(a.side.table[static_cast<size_t>(id) * a.side.table_ld + a.side.col0 + first + threadIdx.x]);
    }
    f32x2 acc[LOADS];
#pragma unroll
    for (int i = 0; i < LOADS; ++i) acc[i] = 0;
    for (int kb0 = warp; kb0 < kblocks; kb0 += U * ONE_WARPS) {
        uint4 xv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int kb = kb0 + u * ONE_WARPS;
            // the choice of the load only where there is one: in every kernel, even as a constant, it cost products of long rows
            // (4096 x 16384 21.1 us instead of 19.9, 512 x 16384 10.7 and 9.6, 4096 x 4096 6.26 and 6.06)
            if constexpr (EARLY) {
                xv[u] = kb < kblocks ? *reinterpret_cast<const uint4*>(x + kb * BLOCK_COLS) : make_uint4(0u, 0u, 0u, 0u);
            } else {
                const uint4* px = reinterpret_cast<const uint4*>(x + kb * BLOCK_COLS);
                if (ahead) xv[u] = kb < kblocks ? __ldcg(px) : make_uint4(0u, 0u, 0u, 0u);   // the first-level cache has not been waited for
                else xv[u] = kb < kblocks ? *px : make_uint4(0u, 0u, 0u, 0u);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const f32x2 x0 = widen(xv[u].x), x1 = widen(xv[u].y), x2 = widen(xv[u].z), x3 = widen(xv[u].w);
#pragma unroll
            for (int i = 0; i < LOADS; ++i) {
                acc[i] = fma2(widen(wv[u][i].x), x0, acc[i]);
                acc[i] = fma2(widen(wv[u][i].y), x1, acc[i]);
                acc[i] = fma2(widen(wv[u][i].z), x2, acc[i]);
                acc[i] = fma2(widen(wv[u][i].w), x3, acc[i]);
            }
        }
        if (kb0 + U * ONE_WARPS < kblocks) load(kb0 + U * ONE_WARPS);
    }
#pragma unroll
    for (int i = 0; i < LOADS; ++i) {
        const float2 p = unpair(acc[i]);
        float v = p.x + p.y;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((lane & 7) == 0) part[warp][i * 4 + (lane >> 3)] = v;
    }
    __syncthreads();
    const int t = threadIdx.x;
    if (t >= (PAIR ? R / 2 : R) || first + t >= (EPI == ROPE ? N / 2 : N)) return;
    float sum = 0.f, up = 0.f;
#pragma unroll
    for (int k = 0; k < ONE_WARPS; ++k) {
        sum += part[k][t];
        if (PAIR) up += part[k][(R / 2 + t) % R];
    }
    if (EPI == ROPE) {
        // rounded to bf16 before the rotation, as where the product is stored in between
        const int f = r0 + t;
        const long long kv_row = static_cast<long long>(kv_len) + a.rope.kv_off;
        float lo = __bfloat162float(__float2bfloat16(sum)), hi = __bfloat162float(__float2bfloat16(up));
        if (tile < a.rope.hq + a.rope.hkv) {
            float sn, cs;
            sincosf(pos * a.rope.inv_freq[f], &sn, &cs);
            const float x0 = lo, x1 = hi;
            lo = x0 * cs - x1 * sn;
            hi = x0 * sn + x1 * cs;
        }
        bf16* dst = a.y + tile * 128 + f;
        if (tile >= a.rope.hq) {
            if (valid < 1 || kv_row < 0) return;
            if (kv_row >= a.rope.cache_rows) {   // host-side length checks come first; this only keeps memory intact
                atomicOr(a.rope.error, ERR_KV_OVERFLOW);
                return;
            }
            const int kv_dim = a.rope.hkv * 128, h = tile - a.rope.hq;
            dst = (h < a.rope.hkv ? a.rope.k_cache + h * 128 : a.rope.v_cache + (h - a.rope.hkv) * 128) + kv_row * kv_dim + f;
        }
        dst[0] = __float2bfloat16(lo);
        dst[64] = __float2bfloat16(hi);
        return;
    }
    if (PAIR) {
        // both projections are rounded to bf16 before silu's product, as where they are stored in between
        sum = a.gate_limit > 0.f ? clamped_gate(sum, up, a.gate_limit, a.gate_alpha)
                                 : silu_mul(__bfloat162float(__float2bfloat16(sum)), __bfloat162float(__float2bfloat16(up)));
    } else if (EPI == SIDE) {
        sum = gelu_tanh(__bfloat162float(__float2bfloat16(sum))) * side;
    } else if (a.bias != nullptr) {
        sum += __bfloat162float(a.bias[first + t]);
    }
    a.y[static_cast<size_t>(shared ? a.ys_row : e.z) * a.ldy + first + t] = __float2bfloat16(sum);
}

// Output rows per CTA: 16 make longer bursts and fewer sums, 8 even out the SMs' shares.  The GPU holds four CTAs per SM: 8 rows while
// CTAs of 8 all fit at once, and where those of 16 would leave a second wave less than half full and a CTA has enough to
// read for that to matter.  Rows x K with 8 / 16 rows, us: 4096 x 8192 11.7 / 13.2, 4608 x 13824 20.1 / 21.6; 4864 x 8192 16.4 / 15.0,
// 9216 x 5120 16.4 / 15.3; 9728 x 8192 26.3 / 30.6, 12288 x 13824 50.0 / 53.7, 12288 x 2048 9.8 / 10.1, 12288 x 1024 7.1 / 6.2;
// 16384 x 5120 27.2 / 25.8, 32768 (gated) x 1024 16.7 / 12.0.  4 rows (2048 x 2048 4.0 us against 3.6) and 32 (73448 x 4096 90 us against
// 84) were slower.
int rows_per_cta(long long outputs, int kblocks) {
    static const char* forced = tuning_env("CPMCU_ONE_ROW");   // bench only
    if (forced) return atoi(forced) == 8 ? 8 : 16;
    const long long resident = 4LL * runtime().num_sms;
    const bool short_wave = outputs > 16 * resident && outputs <= 24 * resident && kblocks >= 32;
    return outputs <= 8 * resident || short_wave ? 8 : 16;
}

}  // namespace

// Everywhere but where long rows meet SMs that are dealt three CTAs of 16 rows beside SMs with two: there nothing evens out the SMs'
// shares and the tiles, which cut K, keep up.  N x K, here / tiles, us: 5120 x 13824 26.5 / 24.4, 5632 x 13824 27.7 / 25.8; 4864 x 13824
// 23.7 / 24.2, 5888 x 13824 28.2 / 33.3, 5120 x 8192 16.7 / 19.2, 5632 x 8192 17.3 / 18.9 (11000 is where the lines cross).
bool linear_one_row_fits(int N, int K, int sms) {
    const int ctas = ceil_div(N, 16), extra = ctas - 2 * sms;
    return K < 11000 || extra * 10 < sms || extra * 20 > 9 * sms;
}

namespace {

template <Epilogue EPI, bool EARLY, bool HOLD = false>
void launch(int R, const OneRowArgs& a, int grid, cudaStream_t s) {
    switch (R) {
        case 8: launch_kernel(one_row_kernel<8, EPI, EARLY, HOLD>, dim3(grid), dim3(ONE_WARPS * 32), 0, s, a); break;
        default: launch_kernel(one_row_kernel<16, EPI, EARLY, HOLD>, dim3(grid), dim3(ONE_WARPS * 32), 0, s, a); break;
    }
}

}  // namespace

void launch_linear_one_row(const LinearPlan& p, cudaStream_t s, const RopeRow* rope, const SideRow* side) {
    OneRowArgs a = {};
    a.w = p.w; a.x = p.x; a.y = p.y; a.bias = p.bias;
    a.N = p.N; a.kblocks = p.K / BLOCK_COLS;
    a.ldx = p.K; a.ldy = p.ldy;
    a.uniform = 1;
    a.gate_limit = p.gate_limit; a.gate_alpha = p.gate_alpha;
    const int R = rows_per_cta(p.swiglu ? 2LL * p.N : p.N, a.kblocks);
    a.ctas = ceil_div(p.N, p.swiglu ? R / 2 : R);
    if (rope != nullptr) {
        CPM_REQUIRE(!p.swiglu && p.N == (rope->hq + 2 * rope->hkv) * 128, "one row: a rotated product is that of queries, keys and values of heads of 128");
        a.rope = *rope;
        launch<ROPE, true>(R, a, a.ctas, s);
    } else if (side != nullptr) {
        CPM_REQUIRE(!p.swiglu && p.bias == nullptr, "one row: a side input's gate is a plain product");
        a.side = *side;
        launch<SIDE, true>(R, a, a.ctas, s);
    } else if (p.swiglu) {
        launch<GATED, true>(R, a, a.ctas, s);
    } else {
        launch<PLAIN, true>(R, a, a.ctas, s);
    }
}

void launch_moe_one_row(const MoeGemmPlan& p, cudaStream_t s, bool hold, bool ahead) {
    OneRowArgs a = {};
    a.w = p.w; a.x = p.x; a.xs = p.xs; a.y = p.y;
    a.N = p.N; a.kblocks = p.kblocks; a.N_s = p.N_s; a.kblocks_s = p.kblocks_s;
    a.stride = static_cast<long long>(p.n_tiles) * p.kblocks * BLOCK_ELEMS;
    a.w_s = p.w_row_s * BLOCK_COLS;
    a.ldx = p.ldx; a.ldy = p.ldy; a.xs_row = p.xs_row0; a.ys_row = p.ys_row0;
    a.entries = p.entries; a.n_entries = p.n_entries; a.uniform = p.uniform;
    const int per = p.swiglu ? 2 : 1;
    const int R = rows_per_cta(static_cast<long long>(per) * (static_cast<long long>(p.max_entries) * p.N + (p.n_tiles_s > 0 ? p.N_s : 0)), p.kblocks);
    a.ctas = ceil_div(p.N, R / per);
    a.ctas_s = p.n_tiles_s > 0 ? ceil_div(p.N_s, R / per) : 0;
    const int grid = a.ctas_s + p.max_entries * a.ctas;
    a.ahead = ahead && p.max_entries > 0;   // some CTA waits for the router
    if (hold) launch<PLAIN, true, true>(R, a, grid, s);
    else if (p.swiglu) launch<GATED, false>(R, a, grid, s);
    else launch<PLAIN, true>(R, a, grid, s);
}
