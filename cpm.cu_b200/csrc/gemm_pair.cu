// Prefill-sized linear layers on pairs of CTAs, sm_100a:  Y[M,N] = X[M,K] W[N,K]^T (+ bias), M > 256, bf16 in, fp32 accumulate.
//
// Same operand mapping, work order, split of the last wave and epilogue as linear_umma_kernel<256> (gemm_umma.cu), but a
// cluster of two CTAs shares a tile of 256 features x 256 tokens: each loads 128 weight rows and HALF of the tokens,
// and one tcgen05.mma.cta_group::2 of rank 0 (M = 256, N = 256) multiplies them on both SMs' tensor cores.  What bounds these
// launches is the tensor pipe and, in a warm pass, the power cap: per MMA an SM reads 8 KB of operands from shared memory
// instead of 12, and per k-block 32 KB come in instead of 48, so L2 and shared memory spend less of the power.
// Loads carry no multicast; the barrier that counts both CTAs' copies is rank 0's.
// Back to back on constant data, single CTAs / pairs, both with the former epilogue: 4096 x 4096 x 16384 (rows x N x K) 357 / 283 us,
// 4096 x 4608 x 4096 113 / 107, 2048 x 4096 x 16384 191 / 151; with the present one (gemm_common.cuh) 274, 87 and 144.
#include <algorithm>

#include "common.cuh"
#include "gemm_common.cuh"
#include "gemm_pair.cuh"
#include "ptx.cuh"

using namespace gemm;

namespace {

constexpr int BLOCK_K = 64, UMMA_K = 16, MT = 256;
constexpr int HALF_M = MT / 2;                               // token rows each CTA loads
constexpr int W_BYTES = BLOCK_N * BLOCK_K * 2, X_BYTES = HALF_M * BLOCK_K * 2;
constexpr int STAGE_BYTES = W_BYTES + X_BYTES;
constexpr int STAGES = 6;
constexpr int TMEM_COLS = 2 * MT;
constexpr int CTRL_BYTES = 256;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + CTRL_BYTES + EPI_XCH_BYTES + 1024;
constexpr int NUM_THREADS = 192;   // warp 0 TMA, warp 1 MMA (rank 0) + TMEM, warps 2-5 epilogue
static_assert(SMEM_BYTES <= 232448, "shared memory budget");

__global__ void __launch_bounds__(NUM_THREADS, 1)
linear_umma_pair_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, const LinearArgs a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);   // rank 0's count both CTAs' copies
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;
    uint64_t* acc_empty = acc_full + 2;                                          // rank 0's
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* s_last = abort_flag + 1;
    float* epi_xch = reinterpret_cast<float*>(smem + STAGES * STAGE_BYTES + CTRL_BYTES);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int rank = static_cast<int>(ptx::cluster_ctarank());
    const int G = gridDim.x / 2, g = blockIdx.x / 2;
    grid_dep_trigger();

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            ptx::mbar_init(&full[s], 1);
            ptx::mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            ptx::mbar_init(&acc_full[s], 1);
            ptx::mbar_init(&acc_empty[s], 2 * 128);
        }
        *abort_flag = 0;
        *s_last = 0;
        ptx::mbar_fence_init();
        ptx::prefetch_tensormap(&tm_w);
        ptx::prefetch_tensormap(&tm_x);
    }
    if (warp == 1) ptx::tmem_alloc_pair(tmem_slot, TMEM_COLS);
    ptx::tc_fence_before();
    __syncthreads();
    ptx::cluster_sync();   // both CTAs' barriers are there before either copies or arrives
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    SegIter it = make_seg_iter(a, g, G);
    if (warp != 0) grid_dep_wait();

    if (warp == 0) {
        // ------------------------------------------------ TMA producer (both CTAs)
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            int tile, kb0, kb1;
            bool ok = true;
            auto bar_of = [&](int s) { return ptx::cluster_map(ptx::smem_u32(&full[s]), 0); };
            auto load_w = [&](int s, int kb, int n_tile) {
                if (rank == 0) ptx::mbar_arrive_expect_tx(&full[s], 2 * STAGE_BYTES);
                ptx::tma_load_2d_pair(smem + s * STAGE_BYTES, &tm_w, bar_of(s), 0, ((2 * n_tile + rank) * a.kblocks + kb) * BLOCK_N);
            };
            auto load_x = [&](int s, int kb, int m_tile) {
                ptx::tma_load_2d_pair(smem + s * STAGE_BYTES + W_BYTES, &tm_x, bar_of(s), kb * BLOCK_K, m_tile * MT + rank * HALF_M);
            };
            // weights of the first stages do not depend on the predecessor
            int pre = 0;
            {
                SegIter pit = it;
                while (pre < STAGES && pit.next(tile, kb0, kb1)) {
                    int m_tile, n_tile;
                    tile_to_mn(a, tile, m_tile, n_tile);
                    for (int kb = kb0; kb < kb1 && pre < STAGES; ++kb, ++pre) load_w(pre, kb, n_tile);
                }
            }
            grid_dep_wait();
            int issued = 0;
            while (ok && it.next(tile, kb0, kb1)) {
                int m_tile, n_tile;
                tile_to_mn(a, tile, m_tile, n_tile);
                for (int kb = kb0; kb < kb1; ++kb, ++issued) {
                    if (issued >= pre) {
                        if (!ptx::mbar_wait(&empty[stage], phase ^ 1, abort_flag)) { ok = false; break; }
                        load_w(stage, kb, n_tile);
                    }
                    load_x(stage, kb, m_tile);
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
            }
            if (!ok) {
                // give copies already in flight time to land before the CTA retires
                const long long t0 = clock64();
                while (clock64() - t0 < 2000000LL) {}
            }
        } else {
            grid_dep_wait();
        }
    } else if (warp == 1) {
        // ------------------------------------------------ MMA issuer (rank 0)
        if (lane == 0 && rank == 0) {
            constexpr uint32_t idesc = ptx::umma_idesc_bf16(2 * BLOCK_N, MT, 0, 0);
            int stage = 0;
            uint32_t phase = 0;
            int acc = 0;
            uint32_t acc_phase = 0;
            int tile, kb0, kb1;
            bool ok = true;
            while (ok && it.next(tile, kb0, kb1)) {
                if (!ptx::mbar_wait(&acc_empty[acc], acc_phase ^ 1, abort_flag)) break;
                ptx::tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * MT;
                for (int kb = kb0; kb < kb1; ++kb) {
                    if (!ptx::mbar_wait(&full[stage], phase, abort_flag)) { ok = false; break; }
                    ptx::tc_fence_after();
                    const uint32_t wa = ptx::smem_u32(smem + stage * STAGE_BYTES);
                    const uint32_t xa = wa + W_BYTES;
#pragma unroll
                    for (int j = 0; j < BLOCK_K / UMMA_K; ++j) {
                        const uint64_t da = ptx::umma_desc_sw128(wa + j * UMMA_K * 2, 16, 1024);
                        const uint64_t db = ptx::umma_desc_sw128(xa + j * UMMA_K * 2, 16, 1024);
                        ptx::umma_ss_pair(d_tmem, da, db, idesc, (kb > kb0 || j > 0) ? 1u : 0u);
                    }
                    ptx::umma_commit_pair(&empty[stage]);
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
                if (!ok) break;
                ptx::umma_commit_pair(&acc_full[acc]);
                acc ^= 1;
                if (acc == 0) acc_phase ^= 1;
            }
        }
    } else {
        // ------------------------------------------------ epilogue (128 threads of each CTA, its own 128 features)
        run_epilogue<MT, 32, 2>(a, it, tmem_base, acc_full, acc_empty, abort_flag, s_last, warp, lane, threadIdx.x - 64, g, G, 0, 2,
                                epi_xch, rank);
    }

    ptx::tc_fence_before();
    __syncthreads();
    __syncwarp();
    ptx::cluster_sync();   // neither CTA leaves while the other may still read its memory or arrive at its barriers
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc_pair(tmem_base, TMEM_COLS);
    }
    if (threadIdx.x == 0 && *abort_flag) atomicOr(a.error, ERR_GEMM_TIMEOUT);
}

void configure() {
    static bool configured = false;
    if (!configured) {
        CUDA_CHECK(cudaFuncSetAttribute(linear_umma_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        configured = true;
    }
}

}  // namespace

int linear_pair_capacity() {
    static int cached = -1;
    if (cached < 0) {
        configure();
        cached = max_active_clusters(linear_umma_pair_kernel, dim3(NUM_THREADS), SMEM_BYTES, 2);
    }
    return cached;
}

void launch_linear_pair(const LinearPlan& p, const LinearArgs& a, cudaStream_t s) {
    configure();
    launch_kernel_cluster(linear_umma_pair_kernel, dim3(p.grid), dim3(NUM_THREADS), SMEM_BYTES, s, 2, p.tm_w, p.tm_x, a);
}
