// Plain attention (any head width up to 512) and the fp32 matrix product of layered models (layered.cuh): everything in
// true 32-bit on the SIMT pipes.
#include <algorithm>

#include "ptx.cuh"
#include "row_ops.cuh"

using namespace ptx;

namespace {

// ---------------------------------------------------------------- attention
// A CTA takes up to RG * R query rows of one key head (row r = token r / grp, head r % grp of the group) and stages tiles
// of 32 keys in shared memory; a warp takes R rows and one tile at a time: lanes are keys for the scores and value columns
// for the output.  A prompt has rows enough for eight warps with rows of their own (KS = 1): keys and values are read once
// per 32 rows instead of once per row.  A single token has not: there the warps, and the CTAs of a cluster, take different
// key tiles (KS tiles a CTA at once) and the partial softmaxes meet in (distributed) shared memory.  Latency of the loads
// and the FMA pipe bound it.  12 heads over 4 key heads of 72, fp32: 300 tokens 61 us, one token behind 300 9.4 us; one warp
// per row, each lane walking a key row of its own in memory, took 128 us a launch on average.
constexpr int PA_MAX_D = 512, PA_TILE = 32;

struct PlainShape {
    int rg, ks, cluster;   // row groups and key tiles per CTA (rg * ks of its eight warps compute), CTAs along the keys
    int smem;
};

template <typename T, int R, int NC>
__global__ void __launch_bounds__(256) plain_attention_kernel(const PlainAttnArgs a, const PlainShape sh) {
    grid_dependency_sync();
    extern __shared__ __align__(16) float smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, threads = blockDim.x;
    const int grp = a.hq / a.hkv, g = blockIdx.z, rows = a.tq * grp;
    const int cta_rows = sh.rg * R, row0 = blockIdx.y * cta_rows;
    const int rank = blockIdx.x;   // the cluster spans the x dimension
    const int kst = a.dk + 4, vst = a.dv + 4;   // padded rows: eight lanes' 16-byte reads fall into eight bank groups
    float* sq = smem;                           // [cta_rows][dk]
    float* sp = sq + cta_rows * a.dk;           // [rg * ks][R][32]
    float* sk = sp + sh.rg * sh.ks * R * 32;    // [ks * 32][kst]
    float* sv = sk + sh.ks * PA_TILE * kst;     // [ks * 32][vst]
    const int first = *a.kv_len + a.kv_len_add - a.tq;   // position of token 0
    for (int i = threadIdx.x * 4; i < cta_rows * a.dk; i += threads * 4) {
        const int rr = i / a.dk, c = i - rr * a.dk, r = min(row0 + rr, rows - 1);
        const T* q = static_cast<const T*>(a.q) + (static_cast<size_t>(r / grp) * a.hq + g * grp + r % grp) * a.dk + c;
#pragma unroll
        for (int e = 0; e < 4; ++e) sq[i + e] = to_float<T>(q[e]);
    }
    const int rg = warp % sh.rg, ks = warp / sh.rg;
    int pos[R], low[R];
    float slope[R], m[R], l[R], acc[R][NC];
#pragma unroll
    for (int x = 0; x < R; ++x) {
        const int r = min(row0 + rg * R + x, rows - 1), h = g * grp + r % grp;
        pos[x] = first + r / grp;
        low[x] = a.window > 0 ? max(pos[x] - a.window + 1, 0) : 0;
        slope[x] = a.bias_exp > 0.f ? exp2f(-a.bias_exp * static_cast<float>(h + 1) / static_cast<float>(a.hq)) : 0.f;
        m[x] = -INFINITY;
        l[x] = 0.f;
#pragma unroll
        for (int c = 0; c < NC; ++c) acc[x][c] = 0.f;
    }
    // the CTA's rows see keys [lo, hi)
    const int t_lo = row0 / grp, t_hi = (min(row0 + cta_rows, rows) - 1) / grp;
    const int lo = a.window > 0 ? max(first + t_lo - a.window + 1, 0) : 0, hi = first + t_hi + 1;
    const size_t kld = static_cast<size_t>(a.hkv) * a.dk, vld = static_cast<size_t>(a.hkv) * a.dv;
    const T* kc = static_cast<const T*>(a.k_cache) + static_cast<size_t>(g) * a.dk;
    const T* vc = static_cast<const T*>(a.v_cache) + static_cast<size_t>(g) * a.dv;
    // a short range gives every CTA of the cluster a tile before any of them gets a second
    const int nks = min(sh.ks, max(1, (hi - lo + PA_TILE * sh.cluster - 1) / (PA_TILE * sh.cluster)));
    const int step = nks * PA_TILE;
    // `n` rows of `cols` columns into shared memory rows of `st`, zeros up to `step` rows; four requests in flight per thread
    auto stage = [&](const T* src, size_t ld, int cols, float* dst, int st, int n) {
        float odd[4] = {0.f, 0.f, 0.f, 0.f};   // NaN once an element is not finite
        for (int i0 = threadIdx.x * 8; i0 < step * cols; i0 += threads * 32) {
            float f[4][8];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = i0 + u * threads * 8, j = i / cols, c = i - j * cols;
#pragma unroll
                for (int e = 0; e < 8; ++e) f[u][e] = 0.f;
                if (j < n) load_vec<8>(src + static_cast<size_t>(j) * ld + c, f[u]);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = i0 + u * threads * 8, j = i / cols, c = i - j * cols;
                if (j >= step) break;
                float4* d = reinterpret_cast<float4*>(dst + j * st + c);
                d[0] = make_float4(f[u][0], f[u][1], f[u][2], f[u][3]);
                d[1] = make_float4(f[u][4], f[u][5], f[u][6], f[u][7]);
#pragma unroll
                for (int e = 0; e < 8; ++e) odd[u] = fmaf(f[u][e], 0.f, odd[u]);
            }
        }
        return (odd[0] + odd[1]) + (odd[2] + odd[3]) != 0.f;
    };
    for (int j0 = lo + rank * step; j0 < hi; j0 += sh.cluster * step) {
        const int n = min(step, hi - j0);
        __syncthreads();   // the last tiles have been read
        stage(kc + static_cast<size_t>(j0) * kld, kld, a.dk, sk, kst, n);
        const int not_finite = __syncthreads_or(stage(vc + static_cast<size_t>(j0) * vld, vld, a.dv, sv, vst, n));
        if (ks >= nks || ks * PA_TILE >= n) continue;   // warp-uniform
        const int j = j0 + ks * PA_TILE + lane;
        const float* k = sk + (ks * PA_TILE + lane) * kst;
        const float* q = sq + rg * R * a.dk;
        float s[R];
#pragma unroll
        for (int x = 0; x < R; ++x) s[x] = 0.f;
        for (int c = 0; c < a.dk; c += 4) {
            const float4 kv = *reinterpret_cast<const float4*>(k + c);
#pragma unroll
            for (int x = 0; x < R; ++x) {
                const float4 qv = *reinterpret_cast<const float4*>(q + x * a.dk + c);
                s[x] += qv.x * kv.x;
                s[x] += qv.y * kv.y;
                s[x] += qv.z * kv.z;
                s[x] += qv.w * kv.w;
            }
        }
        float* p_s = sp + warp * R * 32;
#pragma unroll
        for (int x = 0; x < R; ++x) {
            const float score = (j >= low[x] && j <= pos[x]) ? s[x] * a.scale - slope[x] * static_cast<float>(pos[x] - j) : -INFINITY;
            float mx = score;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const float m_new = fmaxf(m[x], mx);
            const float base = m_new == -INFINITY ? 0.f : m_new;   // no key of these for this row
            const float alpha = expf(m[x] - base), p = expf(score - base);
            l[x] = l[x] * alpha + warp_sum(p);
            m[x] = m_new;
            p_s[x * 32 + lane] = p;
#pragma unroll
            for (int c = 0; c < NC; ++c) acc[x][c] *= alpha;
        }
        __syncwarp();
        const float* v = sv + ks * PA_TILE * vst + lane;
        if (not_finite) {
            // A probability of zero does not hide an infinity or a NaN: values are added only to the rows that see their key.
            const int t0 = j0 + ks * PA_TILE;
#pragma unroll 1
            for (int jj = 0; jj < PA_TILE; ++jj) {
#pragma unroll
                for (int x = 0; x < R; ++x) {
                    if (t0 + jj < low[x] || t0 + jj > pos[x]) continue;
                    const float p = p_s[x * 32 + jj];
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        if (c * 32 < a.dv) acc[x][c] += p * v[jj * vst + c * 32];
                    }
                }
            }
            __syncwarp();
            continue;
        }
#pragma unroll 2
        for (int jj = 0; jj < PA_TILE; jj += 4) {
            float4 p[R];
#pragma unroll
            for (int x = 0; x < R; ++x) p[x] = *reinterpret_cast<const float4*>(p_s + x * 32 + jj);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                if (c * 32 < a.dv) {
                    const float* vv = v + jj * vst + c * 32;
                    const float v0 = vv[0], v1 = vv[vst], v2 = vv[2 * vst], v3 = vv[3 * vst];
#pragma unroll
                    for (int x = 0; x < R; ++x) {
                        acc[x][c] += p[x].x * v0;
                        acc[x][c] += p[x].y * v1;
                        acc[x][c] += p[x].z * v2;
                        acc[x][c] += p[x].w * v3;
                    }
                }
            }
        }
        __syncwarp();
    }
    auto out_row = [&](int r) {
        return static_cast<T*>(a.out) + static_cast<size_t>(r / grp) * a.out_ld + static_cast<size_t>(g * grp + r % grp) * a.out_cols;
    };
    if (sh.ks * sh.cluster == 1) {
#pragma unroll
        for (int x = 0; x < R; ++x) {
            const int r = row0 + rg * R + x;
            if (r >= rows || ks > 0) break;
            if (a.sink != 0) l[x] += expf(-m[x]);
            const float inv = l[x] > 0.f ? a.out_scale / l[x] : 0.f;
            T* out = out_row(r);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                if (c * 32 + lane < a.out_cols) out[c * 32 + lane] = from_float<T>(acc[x][c] * inv);
            }
        }
        return;
    }
    // Partial softmaxes meet over the staging area: first the warps' ([nks][cta_rows][dv] outputs and [nks][cta_rows] (m, l)),
    // added up into one per CTA behind them, then the CTAs', whose rows are dealt to the CTAs of the cluster.  Both in key
    // order.
    __syncthreads();
    float* part = sk;
    float2* ml = reinterpret_cast<float2*>(part + nks * cta_rows * a.dv);
    float* one = reinterpret_cast<float*>(ml + nks * cta_rows);
    float2* one_ml = reinterpret_cast<float2*>(one + cta_rows * a.dv);
#pragma unroll
    for (int x = 0; x < R; ++x) {
        if (ks >= nks) break;
        const int e = ks * cta_rows + rg * R + x;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            if (c * 32 < a.dv) part[e * a.dv + c * 32 + lane] = acc[x][c];
        }
        if (lane == 0) ml[e] = make_float2(m[x], l[x]);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < cta_rows * a.dv; i += threads) {
        const int rr = i / a.dv, c = i - rr * a.dv;
        float top = -INFINITY, sum = 0.f, o = 0.f;
        for (int k = 0; k < nks; ++k) top = fmaxf(top, ml[k * cta_rows + rr].x);
        const float base = top == -INFINITY ? 0.f : top;
        for (int k = 0; k < nks; ++k) {
            const float2 p = ml[k * cta_rows + rr];
            const float wk = expf(p.x - base);
            sum += wk * p.y;
            o += wk * part[(k * cta_rows + rr) * a.dv + c];
        }
        one[i] = o;
        if (c == 0) one_ml[rr] = make_float2(top, sum);
    }
    if (sh.cluster > 1) cluster_sync();
    else __syncthreads();
    const uint32_t one_at = smem_u32(one), ml_at = smem_u32(one_ml);
    for (int i = threadIdx.x; i < cta_rows * a.dv; i += threads) {
        const int rr = i / a.dv, c = i - rr * a.dv;
        if (rr % sh.cluster != rank || row0 + rr >= rows || c >= a.out_cols) continue;
        float m_k[8], l_k[8], o_k[8], top = -INFINITY, sum = 0.f, o = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) {   // at most eight CTAs: every request in flight at once
            const bool there = k < sh.cluster;
            const uint32_t at = cluster_map(ml_at + 8 * rr, there ? k : rank);
            m_k[k] = there ? ld_cluster_f32(at) : -INFINITY;
            l_k[k] = there ? ld_cluster_f32(at + 4) : 0.f;
            o_k[k] = there ? ld_cluster_f32(cluster_map(one_at + 4 * i, k)) : 0.f;
            top = fmaxf(top, m_k[k]);
        }
        const float base = top == -INFINITY ? 0.f : top;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float wk = expf(m_k[k] - base);
            sum += wk * l_k[k];
            o += wk * o_k[k];
        }
        if (a.sink != 0) sum += expf(-top);
        out_row(row0 + rr)[c] = from_float<T>(o * (sum > 0.f ? a.out_scale / sum : 0.f));
    }
    if (sh.cluster > 1) cluster_sync();   // the peers have read this CTA's partials
}

template <typename T, int R, int NC>
void run_plain_attention(const PlainAttnArgs& a, cudaStream_t s) {
    const int grp = a.hq / a.hkv, rows = a.tq * grp;
    PlainShape sh;
    sh.rg = 1;
    while (sh.rg < 8 && sh.rg * R < rows) sh.rg *= 2;
    auto bytes = [&](int ks) {
        return 4 * (sh.rg * R * a.dk + sh.rg * ks * R * 32 + std::max(ks * PA_TILE * (a.dk + a.dv + 8), (ks + 1) * sh.rg * R * (a.dv + 2)));
    };
    sh.ks = 1;
    // as many tiles at once as eight warps and the shared memory allow
    while (sh.ks * 2 * sh.rg <= 8 && bytes(sh.ks * 2) <= 200 * 1024) sh.ks *= 2;
    const int ctas = ceil_div(rows, sh.rg * R) * a.hkv;
    // key splits while the row tiles alone leave SMs idle
    sh.cluster = 1;
    while (sh.cluster < 8 && ctas * sh.cluster * 2 <= runtime().num_sms) sh.cluster *= 2;
    sh.smem = bytes(sh.ks);
    CPM_REQUIRE(a.dk % 64 == 0 && a.dv % 64 == 0 && a.dv <= NC * 32 && sh.smem <= 220 * 1024, "attention: head too wide");
    auto kernel = plain_attention_kernel<T, R, NC>;
    static const bool ready = [&] {
        CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
        return true;
    }();
    (void)ready;
    const dim3 grid(sh.cluster, ceil_div(rows, sh.rg * R), a.hkv), block(256);
    if (sh.cluster > 1) launch_kernel_cluster(kernel, grid, block, sh.smem, s, sh.cluster, a, sh);
    else launch_kernel(kernel, grid, block, sh.smem, s, a, sh);
}

// ---------------------------------------------------------------- fp32 products
// {expert, first x row, first y row, rows} of this CTA's row group (layered.cuh), or the whole matrix
struct F32Rows {
    const bf16* w;
    int x0, y0, rows;
};
__device__ __forceinline__ F32Rows f32_rows(const bf16* w, size_t w_stride, int M, const int4* entries, int x_at_y) {
    F32Rows r{w, 0, 0, M};
    if (entries != nullptr) {
        const int4 e = entries[blockIdx.z];
        r.w = w + static_cast<size_t>(e.x) * w_stride;
        r.x0 = x_at_y ? e.z : e.y;
        r.y0 = e.z;
        r.rows = e.w;
    }
    return r;
}

// Up to R rows at a time: a warp owns two output features, its lanes lie along K with 16 bytes of each weight row at a time; all of a
// chunk's weights are requested before the first is used (and, where the row group is known, before the previous kernel is
// waited for).  Bound by the latency of one weight fetch, or for wide matrices by HBM: a 64 x 64 tile with one row in it
// walked K in 32-element steps with two barriers each: 64 us a launch on average over the decoding steps of a model 1000
// wide, 2.9 us now.
template <int R>
__global__ void __launch_bounds__(256) linear_f32_few_kernel(const float* __restrict__ x, int ldx, const bf16* __restrict__ w, size_t w_stride,
                                                             float* __restrict__ y, int ldy, int M, int N, int K,
                                                             const int4* __restrict__ entries, const int32_t* __restrict__ n_entries, int x_at_y) {
    constexpr int U = 4, CHUNK = U * 256;   // elements of K in flight per row
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = (blockIdx.x * 8 + warp) * 2;
    uint4 wv[2][U];
    auto request = [&](const bf16* base, int k0) {
#pragma unroll
        for (int f = 0; f < 2; ++f) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int k = k0 + u * 256 + lane * 8;
                wv[f][u] = (n0 + f < N && k < K) ? __ldg(reinterpret_cast<const uint4*>(base + static_cast<size_t>(n0 + f) * K + k)) : make_uint4(0, 0, 0, 0);
            }
        }
    };
    grid_dep_trigger();
    if (entries == nullptr) request(w, 0);
    grid_dep_wait();
    if (entries != nullptr && static_cast<int>(blockIdx.z) >= *n_entries) return;
    F32Rows g = f32_rows(w, w_stride, M, entries, x_at_y);
    const int r0 = blockIdx.y * R;
    if (r0 >= g.rows) return;
    g.x0 += r0; g.y0 += r0; g.rows -= r0;
    if (entries != nullptr) request(g.w, 0);
    float acc[2][R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[0][r] = acc[1][r] = 0.f;
    for (int k0 = 0; k0 < K; k0 += CHUNK) {
        if (k0 > 0) request(g.w, k0);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = k0 + u * 256 + lane * 8;
            if (k >= K) continue;
            float f0[8], f1[8];
            const bf16 *b0 = reinterpret_cast<const bf16*>(&wv[0][u]), *b1 = reinterpret_cast<const bf16*>(&wv[1][u]);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                f0[e] = __bfloat162float(b0[e]);
                f1[e] = __bfloat162float(b1[e]);
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (r >= g.rows) break;
                float v[8];
                load_vec<8>(x + static_cast<size_t>(g.x0 + r) * ldx + k, v);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    acc[0][r] = fmaf(v[e], f0[e], acc[0][r]);
                    acc[1][r] = fmaf(v[e], f1[e], acc[1][r]);
                }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (r >= g.rows) break;
        const float a = warp_sum(acc[0][r]), b = warp_sum(acc[1][r]);
        float* out = y + static_cast<size_t>(g.y0 + r) * ldy + n0;
        if (lane == 0 && n0 < N) out[0] = a;
        if (lane == 1 && n0 + 1 < N) out[1] = b;
    }
}

// More rows: 32 x 32 output tile; four groups of 64 threads (8 x 8, 4 x 4 outputs each) take a quarter of every 64-element
// step of K and their sums meet at the end, so that the CTA keeps eight warps busy on a tile small enough for a few hundred
// rows of a narrow model to fill the GPU.  Steps arrive by cp.async, two ahead, in the matrices' own layout (rows padded so
// that eight rows' 16-byte reads fall into eight bank groups).  Bound by the FMA pipe and the last wave: 64 x 4096 x 1024 30 us, 32 x 32768 x 1024 67 us (32 TFLOP/s).  A single-buffered tile of 64 x 64
// took 112 us a launch where this takes 37, over the products of 300 tokens in a model 1000 wide.
constexpr int F32_T = 32, F32_KT = 64, F32_STAGES = 3, F32_LDX = F32_KT + 4, F32_LDW = F32_KT + 8;

__global__ void __launch_bounds__(256)
linear_f32_tile_kernel(const float* __restrict__ x, int ldx, const bf16* __restrict__ w, size_t w_stride, float* __restrict__ y, int ldy,
                       int M, int N, int K, const int4* __restrict__ entries, const int32_t* __restrict__ n_entries, int x_at_y) {
    grid_dependency_sync();
    __shared__ __align__(16) float sx[F32_STAGES][F32_T][F32_LDX];
    __shared__ __align__(16) bf16 sw[F32_STAGES][F32_T][F32_LDW];
    if (entries != nullptr && static_cast<int>(blockIdx.z) >= *n_entries) return;
    const F32Rows g = f32_rows(w, w_stride, M, entries, x_at_y);
    const int m0 = blockIdx.y * F32_T, n0 = blockIdx.x * F32_T;
    if (m0 >= g.rows) return;
    const int tid = threadIdx.x, kg = tid >> 6, tx = tid & 7, ty = (tid >> 3) & 7;
    const int steps = K / F32_KT;   // K is a multiple of 64
    auto fetch = [&](int i) {
        if (i < steps) {
            const int st = i % F32_STAGES, k0 = i * F32_KT;
#pragma unroll
            for (int q = 0; q < 2; ++q) {   // 32 rows x 16 pieces of x
                const int r = (tid >> 4) + 16 * q, c = (tid & 15) * 4;
                const bool in = m0 + r < g.rows;
                cp_async16(&sx[st][r][c], x + static_cast<size_t>(g.x0 + (in ? m0 + r : 0)) * ldx + k0 + c, in ? 16 : 0);
            }
            const int r = tid >> 3, c = (tid & 7) * 8;   // 32 rows x 8 pieces of w
            const bool in = n0 + r < N;
            cp_async16(&sw[st][r][c], g.w + static_cast<size_t>(in ? n0 + r : 0) * K + k0 + c, in ? 16 : 0);
        }
        cp_async_commit();
    };
    float acc[4][4] = {};   // rows ty + 8 i, features tx + 8 j
    fetch(0);
    fetch(1);
    for (int i = 0; i < steps; ++i) {
        cp_async_wait<1>();
        __syncthreads();   // step i is here for everyone, and everyone is done with the stage that is filled next
        fetch(i + 2);
        const int st = i % F32_STAGES;
#pragma unroll
        for (int k = kg * (F32_KT / 4); k < (kg + 1) * (F32_KT / 4); k += 4) {
            float4 xv[4];
            float wv[4][4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                xv[e] = *reinterpret_cast<const float4*>(&sx[st][ty + 8 * e][k]);
                const uint2 u = *reinterpret_cast<const uint2*>(&sw[st][tx + 8 * e][k]);
                wv[e][0] = __uint_as_float(u.x << 16);
                wv[e][1] = __uint_as_float(u.x & 0xffff0000u);
                wv[e][2] = __uint_as_float(u.y << 16);
                wv[e][3] = __uint_as_float(u.y & 0xffff0000u);
            }
#pragma unroll
            for (int a = 0; a < 4; ++a) {
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    acc[a][b] = fmaf(xv[a].x, wv[b][0], acc[a][b]);
                    acc[a][b] = fmaf(xv[a].y, wv[b][1], acc[a][b]);
                    acc[a][b] = fmaf(xv[a].z, wv[b][2], acc[a][b]);
                    acc[a][b] = fmaf(xv[a].w, wv[b][3], acc[a][b]);
                }
            }
        }
    }
    __syncthreads();
    float* red = &sx[0][0][0];   // [4][32][32 + 1]
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) red[(kg * F32_T + ty + 8 * i) * (F32_T + 1) + tx + 8 * j] = acc[i][j];
    }
    __syncthreads();
    const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int i = 0; i < F32_T; i += 8) {
        const int r = i + warp;
        float sum = 0.f;
#pragma unroll
        for (int q = 0; q < 4; ++q) sum += red[(q * F32_T + r) * (F32_T + 1) + lane];
        if (m0 + r < g.rows && n0 + lane < N) y[static_cast<size_t>(g.y0 + m0 + r) * ldy + n0 + lane] = sum;
    }
}

}  // namespace

template <typename T>
void launch_plain_attention(const PlainAttnArgs& a, cudaStream_t s) {
    ProfileScope prof(KC_ATTENTION, s);
    CPM_REQUIRE(a.dk % 64 == 0 && a.dk <= PA_MAX_D && a.dv <= PA_MAX_D && a.hq % a.hkv == 0, "attention: head width above 512");
    // accumulators: 16 registers for heads up to 128 wide, 32 above
    if (a.dv <= 128) run_plain_attention<T, 4, 4>(a, s);
    else run_plain_attention<T, 2, 16>(a, s);
}
template void launch_plain_attention<bf16>(const PlainAttnArgs&, cudaStream_t);
template void launch_plain_attention<float>(const PlainAttnArgs&, cudaStream_t);

void launch_linear_f32(const float* x, int ldx, const bf16* w, size_t w_stride, float* y, int ldy, int M, int N, int K,
                       const int4* entries, const int32_t* n_entries, int max_entries, bool x_at_y, cudaStream_t s) {
    ProfileScope prof(entries ? KC_MOE : KC_LINEAR, s);
    CPM_REQUIRE(K % 64 == 0 && ldx % 4 == 0, "linear_f32: K must be a multiple of 64");
    const int z = entries ? max_entries : 1, most = entries ? std::min(M, kF32Rows) : M;
    // Up to eight rows a warp per two features reads every weight once; beyond, while few features make few warps, so do a
    // warp's eight rows of several.  K = 1024, few / tile, us, weights from HBM: 8 rows x 4096 9.4 / 30.4, 24 x 4096 25.5 / 30.7,
    // 32 x 4096 33.5 / 30.7, 8 x 8192 17.8 / 29.9, 16 x 8192 31.5 / 30.0, 8 x 32768 48.8 / 66.6, 12 x 32768 75.9 / 66.8 (the tile waits
    // for each step's weights); a model that fits L2: 16 x 2048 9.3 / 12.9, 32 x 1024 9.3 / 12.9, 32 x 2048 17.4 / 13.3, 64 x 1024 17.3 / 13.0.
    if (most <= 8 || (most <= 32 && ceil_div(most, 8) * N < 16384)) {
        auto kernel = most == 1 ? linear_f32_few_kernel<1> : most == 2 ? linear_f32_few_kernel<2> : most <= 4 ? linear_f32_few_kernel<4> : linear_f32_few_kernel<8>;
        launch_kernel(kernel, dim3(ceil_div(N, 16), ceil_div(most, 8), z), dim3(256), 0, s, x, ldx, w, w_stride, y, ldy, M, N, K, entries, n_entries, x_at_y ? 1 : 0);
        return;
    }
    launch_kernel(linear_f32_tile_kernel, dim3(ceil_div(N, F32_T), ceil_div(most, F32_T), z), dim3(256), 0, s, x, ldx, w, w_stride, y, ldy, M, N, K,
                  entries, n_entries, x_at_y ? 1 : 0);
}
