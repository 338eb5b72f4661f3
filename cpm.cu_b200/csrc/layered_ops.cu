// Row-wise kernels of layered models (layered.cuh).  Norms and the residual sum are fp32 whatever T is.
#include <algorithm>

#include "row_ops.cuh"

namespace {

template <typename T>
__global__ void embed_rows_kernel(const int32_t* __restrict__ ids, const bf16* __restrict__ table, int vocab, float scale, float* __restrict__ x32,
                                  T* __restrict__ xh, int ld, const StateCheck check, int* __restrict__ error) {
    grid_dependency_sync();
    const size_t row = blockIdx.x;
    if (check.state_len != nullptr && row == 0 && threadIdx.x == 0) {
        const int first = *check.kv_len + check.kv_off;
        const bool ok = first == 0 || first == *check.state_len;
        if (!ok) atomicOr(error, ERR_STATE_POS);
        *check.state_len = ok ? first + static_cast<int>(gridDim.x) : -1;
    }
    int id = ids[row];
    if (id < 0 || id >= vocab) {
        if (threadIdx.x == 0) atomicOr(error, ERR_BAD_TOKEN);
        id = 0;
    }
    const bf16* src = table + static_cast<size_t>(id) * ld;
    for (int c = threadIdx.x * 8; c < ld; c += blockDim.x * 8) {
        float f[8];
        load_vec<8>(src + c, f);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] *= scale;
        store_vec<8>(x32 + row * ld + c, f);
        store_vec<8>(xh + row * ld + c, f);
    }
}

// FRESH: past the first-level cache
template <int VEC, bool FRESH, typename T>
__device__ __forceinline__ void load_row(const T* p, float* f) {
    if constexpr (FRESH && VEC == 8 && sizeof(T) == 2) {
        const uint4 v = __ldcg(reinterpret_cast<const uint4*>(p));
        load_vec<8>(reinterpret_cast<const T*>(&v), f);
    } else if constexpr (FRESH && sizeof(T) == 2) {
        static_assert(VEC == 1, "pieces of 16 bytes or single elements");
        f[0] = __bfloat162float(__ushort_as_bfloat16(__ldcg(reinterpret_cast<const unsigned short*>(p))));
    } else {
        load_vec<VEC>(p, f);
    }
}

// One CTA per token row.  BESIDE: the row's writer has ended before this launch starts, and the wait for the predecessor comes at the end, so
// that whatever waits for this launch has waited for both.
template <typename T, int VEC, bool BESIDE>
__global__ void qkv_norm_append_kernel(const QkvNormArgs a) {
    grid_dep_trigger();
    if (!BESIDE) grid_dep_wait();
    __shared__ float sh[64];
    __shared__ float2 turn[256];   // cos, sin of the row's angles
    const int r = blockIdx.x;
    const int nq = a.heads * a.dim, nk = a.kv_heads * a.dim, nv = a.kv_heads * a.vdim;
    const T* row = static_cast<const T*>(a.qkv) + static_cast<size_t>(r) * a.ld;
    const bool own_kv = a.k_cache != nullptr;
    const long long kv_row = own_kv ? static_cast<long long>(__ldcg(a.kv_len)) + a.kv_off + r : 0;
    const bool store_kv = own_kv && kv_row >= 0 && kv_row < a.cache_rows;
    if (own_kv && !store_kv && threadIdx.x == 0) atomicOr(a.error, ERR_KV_OVERFLOW);
    const int half = a.rot_dims / 2;
    if (half > 0) {
        const float pos = static_cast<float>(__ldcg(a.kv_len) + a.kv_off + r);
        for (int i = threadIdx.x; i < half; i += blockDim.x) {
            float sn, cs;
            sincosf(pos * a.inv_freq[i], &sn, &cs);
            turn[i] = make_float2(cs, sn);
        }
        __syncthreads();
    }
    float rq = 1.f, rk = 1.f;
    if (a.wq != nullptr) {
        float sq = 0.f, sk = 0.f, f[VEC];
        for (int c = threadIdx.x * VEC; c < nq; c += blockDim.x * VEC) {
            load_row<VEC, BESIDE>(row + c, f);
#pragma unroll
            for (int e = 0; e < VEC; ++e) sq += f[e] * f[e];
        }
        if (own_kv) {
            for (int c = threadIdx.x * VEC; c < nk; c += blockDim.x * VEC) {
                load_row<VEC, BESIDE>(row + nq + c, f);
#pragma unroll
                for (int e = 0; e < VEC; ++e) sk += f[e] * f[e];
            }
        }
        const float2 t = block_sum2(sq, sk, sh);
        rq = rsqrtf(t.x / nq + a.eps);
        if (own_kv) rk = rsqrtf(t.y / nk + a.eps);
    }
    auto place = [&](const T* src, const bf16* w, float rs, int n_heads, int d, int dp, T* dst, bool pad, int rot) {
        const int per = (pad ? dp : d) / VEC;
        for (int i = threadIdx.x; i < n_heads * per; i += blockDim.x) {
            const int h = i / per, c = (i - h * per) * VEC;
            float f[VEC];
            if (c < d) {
                load_row<VEC, BESIDE>(src + h * d + c, f);
                if (w != nullptr) {
                    float g[VEC];
                    load_vec<VEC>(w + h * d + c, g);
#pragma unroll
                    for (int e = 0; e < VEC; ++e) f[e] = f[e] * rs * g[e];
                }
                if (c < 2 * rot) {   // rot is a multiple of VEC
                    const bool upper = c >= rot;
                    const int other = upper ? c - rot : c + rot, i0 = upper ? c - rot : c;
                    float p[VEC];
                    load_row<VEC, BESIDE>(src + h * d + other, p);
                    if (w != nullptr) {
                        float g[VEC];
                        load_vec<VEC>(w + h * d + other, g);
#pragma unroll
                        for (int e = 0; e < VEC; ++e) p[e] = p[e] * rs * g[e];
                    }
#pragma unroll
                    for (int e = 0; e < VEC; ++e) {
                        const float2 cs = turn[i0 + e];
                        f[e] = upper ? f[e] * cs.x + p[e] * cs.y : f[e] * cs.x - p[e] * cs.y;
                    }
                }
            } else {
#pragma unroll
                for (int e = 0; e < VEC; ++e) f[e] = 0.f;
            }
            store_vec<VEC>(dst + static_cast<size_t>(h) * dp + c, f);
        }
    };
    // the query buffer is shared by layers of different widths, so its padding is written; a cache's padding stays zero
    place(row, a.wq, rq, a.heads, a.dim, a.dim_p, static_cast<T*>(a.q_out) + static_cast<size_t>(r) * a.heads * a.dim_p, true, half);
    if (store_kv) {
        place(row + nq, a.wk, rk, a.kv_heads, a.dim, a.dim_p,
              static_cast<T*>(a.k_cache) + static_cast<size_t>(kv_row) * a.kv_heads * a.dim_p, false, half);
        place(row + nq + nk, nullptr, 1.f, a.kv_heads, a.vdim, a.vdim_p,
              static_cast<T*>(a.v_cache) + static_cast<size_t>(kv_row) * a.kv_heads * a.vdim_p, false, 0);
        (void)nv;
    }
    if (BESIDE) grid_dep_wait();
}

// Eight consecutive elements as they are (2 or 4 bytes each)
template <typename T>
struct Raw8 {
    uint4 q[sizeof(T) / 2];
    __device__ __forceinline__ void load(const T* p) {
#pragma unroll
        for (int i = 0; i < static_cast<int>(sizeof(T) / 2); ++i) q[i] = reinterpret_cast<const uint4*>(p)[i];
    }
    __device__ __forceinline__ void load_l2(const T* p) {
#pragma unroll
        for (int i = 0; i < static_cast<int>(sizeof(T) / 2); ++i) q[i] = __ldcg(reinterpret_cast<const uint4*>(p) + i);
    }
    __device__ __forceinline__ void widen(float* f) const { load_vec<8>(reinterpret_cast<const T*>(q), f); }
};

// Without experts, with them, or with them for one row.  Many rows are bound by memory and hide one another's round trips (4096 rows of 2048 with
// the loads of one row: 45 -> 48.5 us, without experts 18 -> 21); one row is a chain of round trips: the router's choice and the
// stream are asked for before the wait (MoeMix::early), then eight experts' pieces at once.  A token of six layers of 4096 580 -> 571 us.
// Rows wider than 4096 (four pieces a thread) keep the form of many rows; one row of them has not been measured.
enum Mixture { NO_MIX, MIX_ROWS, MIX_ONE };
template <typename T, int VPT, Mixture MIX>
__global__ void __launch_bounds__(512)
out_norm_kernel(float* __restrict__ x32, T* __restrict__ xh, const T* __restrict__ delta, const MoeMix mix, float mult,
                const bf16* __restrict__ w, int width, int ld, float eps) {
    grid_dep_trigger();
    __shared__ float sh[64];
    __shared__ int s_row[kMoeMaxTop];
    __shared__ float s_w[kMoeMaxTop];
    const size_t base = static_cast<size_t>(blockIdx.x) * ld;
    float wv[VPT][8];   // the weights never depend on the previous kernel
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
        const int c = (threadIdx.x + j * blockDim.x) * 8;
        if (c < ld) load_vec<8>(w + c, wv[j]);
    }
    float xv[VPT][8], dv[VPT][8];
    float idw = 0.f;
    // one row: past the first-level cache, which nothing has waited for
    auto stream = [&]() {
#pragma unroll
        for (int j = 0; j < VPT; ++j) {
            const int c = (threadIdx.x + j * blockDim.x) * 8;
            if (c >= ld) continue;
            if constexpr (MIX == MIX_ONE) {
                Raw8<float> raw;
                raw.load_l2(x32 + base + c);
                raw.widen(xv[j]);
            } else {
                load_vec<8>(x32 + base + c, xv[j]);
            }
        }
        auto get = [](const auto* p) {
            if constexpr (MIX == MIX_ONE) return __ldcg(p);
            else return *p;
        };
        if constexpr (MIX != NO_MIX) {
            if (threadIdx.x < mix.top) {
                const size_t i = static_cast<size_t>(blockIdx.x) * mix.top + threadIdx.x;
                const int e = get(mix.expert + i);
                s_row[threadIdx.x] = e < mix.experts ? get(mix.offset + e) + get(mix.rank + i) : -1;
                s_w[threadIdx.x] = get(mix.weight + i);
            }
            if (MIX == MIX_ONE) idw = get(mix.id_weight + blockIdx.x);
        }
    };
    const bool early = MIX == MIX_ONE && mix.early != 0;
    if (early) stream();
    grid_dep_wait();
    if (!early) stream();
    if constexpr (MIX != NO_MIX) {
        __syncthreads();
        if (MIX != MIX_ONE) idw = mix.id_weight[blockIdx.x];
        const T* y = static_cast<const T*>(mix.y);
#pragma unroll
        for (int j = 0; j < VPT; ++j) {
            const int c = (threadIdx.x + j * blockDim.x) * 8;
            if (c >= ld) continue;
#pragma unroll
            for (int e = 0; e < 8; ++e) dv[j][e] = idw * xv[j][e];
            const T* ys = y + (static_cast<size_t>(mix.shared_row0) + blockIdx.x) * ld + c;
            float f[8];
            if constexpr (MIX == MIX_ONE) {
                constexpr int AT_ONCE = 8;
                Raw8<T> shared;
                if (mix.shared_row0 >= 0) shared.load(ys);
                for (int k0 = 0; k0 < mix.top; k0 += AT_ONCE) {
                    Raw8<T> raw[AT_ONCE];
                    int row[AT_ONCE];
#pragma unroll
                    for (int u = 0; u < AT_ONCE; ++u) {
                        row[u] = k0 + u < mix.top ? s_row[k0 + u] : -1;
                        if (row[u] >= 0) raw[u].load(y + static_cast<size_t>(row[u]) * ld + c);
                    }
#pragma unroll
                    for (int u = 0; u < AT_ONCE; ++u) {
                        if (row[u] < 0) continue;
                        raw[u].widen(f);
                        const float wk = s_w[k0 + u];
#pragma unroll
                        for (int e = 0; e < 8; ++e) dv[j][e] += wk * f[e];
                    }
                }
                if (mix.shared_row0 >= 0) shared.widen(f);
            } else {
#pragma unroll 4
                for (int k = 0; k < mix.top; ++k) {
                    if (s_row[k] < 0) continue;
                    load_vec<8>(y + static_cast<size_t>(s_row[k]) * ld + c, f);
                    const float wk = s_w[k];
#pragma unroll
                    for (int e = 0; e < 8; ++e) dv[j][e] += wk * f[e];
                }
                if (mix.shared_row0 >= 0) load_vec<8>(ys, f);
            }
            if (mix.shared_row0 >= 0) {
#pragma unroll
                for (int e = 0; e < 8; ++e) dv[j][e] += f[e];
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < VPT; ++j) {
            const int c = (threadIdx.x + j * blockDim.x) * 8;
            if (c < ld) load_vec<8>(delta + base + c, dv[j]);
        }
    }
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
        const int c = (threadIdx.x + j * blockDim.x) * 8;
        if (c < ld) {
#pragma unroll
            for (int e = 0; e < 8; ++e) ss += dv[j][e] * dv[j][e];   // padding columns are zero
        }
    }
    const float rs = rsqrtf(block_sum2(ss, 0.f, sh).x / width + eps);
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
        const int c = (threadIdx.x + j * blockDim.x) * 8;
        if (c < ld) {
#pragma unroll
            for (int e = 0; e < 8; ++e) xv[j][e] += mult * (dv[j][e] * rs * (1.f + wv[j][e]));
            store_vec<8>(x32 + base + c, xv[j]);
            store_vec<8>(xh + base + c, xv[j]);
        }
    }
}

template <typename T>
__global__ void norm_rows_kernel(const float* __restrict__ x32, const int32_t* __restrict__ rows_idx, const bf16* __restrict__ w,
                                 T* __restrict__ y, int width, int ld, float eps) {
    grid_dependency_sync();
    __shared__ float sh[64];
    const float* x = x32 + static_cast<size_t>(rows_idx ? rows_idx[blockIdx.x] : blockIdx.x) * ld;
    float ss = 0.f, f[8], g[8];
    for (int c = threadIdx.x * 8; c < ld; c += blockDim.x * 8) {
        load_vec<8>(x + c, f);
#pragma unroll
        for (int e = 0; e < 8; ++e) ss += f[e] * f[e];
    }
    const float rs = rsqrtf(block_sum2(ss, 0.f, sh).x / width + eps);
    for (int c = threadIdx.x * 8; c < ld; c += blockDim.x * 8) {
        load_vec<8>(x + c, f);
        load_vec<8>(w + c, g);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = f[e] * rs * (1.f + g[e]);
        store_vec<8>(y + static_cast<size_t>(blockIdx.x) * ld + c, f);
    }
}

__global__ void silu_f32_kernel(const float* __restrict__ gu, int ld_gu, float* __restrict__ act, int ld_act, int ff) {
    grid_dependency_sync();
    const float* g = gu + static_cast<size_t>(blockIdx.x) * ld_gu;
    float* o = act + static_cast<size_t>(blockIdx.x) * ld_act;
    for (int c = threadIdx.x; c < ff; c += blockDim.x) o[c] = g[c] / (1.f + expf(-g[c])) * g[ff + c];
}

}  // namespace

template <typename T>
void launch_embed_rows(const int32_t* ids, const bf16* table, int vocab, float scale, float* x32, T* xh, int ld, int rows,
                       const StateCheck& check, cudaStream_t s) {
    ProfileScope prof(KC_ROW, s);
    launch_kernel(embed_rows_kernel<T>, dim3(rows), dim3(128), 0, s, ids, table, vocab, scale, x32, xh, ld, check, runtime().d_error);
}

template <typename T>
void launch_qkv_norm_append(const QkvNormArgs& a, int rows, cudaStream_t s) {
    ProfileScope prof(KC_ROW, s);
    CPM_REQUIRE(a.rot_dims % 2 == 0 && a.rot_dims <= a.dim && a.rot_dims <= 512, "layered model: bad number of rotated dimensions");
    const bool v8 = a.dim % 8 == 0 && a.vdim % 8 == 0 && a.ld % 8 == 0 && (a.rot_dims / 2) % 8 == 0;
    auto run = [&](auto kernel) { launch_kernel(kernel, dim3(rows), dim3(256), 0, s, a); };
    if constexpr (sizeof(T) == 2) {
        if (runtime().order.ended(a.written_by)) {
            if (v8) run(qkv_norm_append_kernel<T, 8, true>); else run(qkv_norm_append_kernel<T, 1, true>);
            return;
        }
    }
    if (v8) run(qkv_norm_append_kernel<T, 8, false>); else run(qkv_norm_append_kernel<T, 1, false>);
}

template <typename T>
void launch_out_norm(float* x32, T* xh, const T* delta, const MoeMix& mix_, float mult, const bf16* w, int rows, int width, int ld,
                     float eps, cudaStream_t s) {
    ProfileScope prof(KC_ROW, s);
    MoeMix mix = mix_;
    mix.early = runtime().order.ended(mix.routed) ? 1 : 0;
    CPM_REQUIRE(ld % 64 == 0 && ld <= 512 * 8 * 4, "layered model: width above 16384 is not supported");
    CPM_REQUIRE(mix.top <= kMoeMaxTop, "mixture of experts: too many experts per token");
    const int vecs = ld / 8;
    const int threads = vecs >= 512 ? 512 : (vecs + 31) / 32 * 32;
    const bool mixed = mix.y != nullptr;
    auto run = [&](auto kernel) { launch_kernel(kernel, dim3(rows), dim3(threads), 0, s, x32, xh, delta, mix, mult, w, width, ld, eps); };
    if (vecs <= 512) {
        if (mixed && rows == 1) run(out_norm_kernel<T, 1, MIX_ONE>);
        else if (mixed) run(out_norm_kernel<T, 1, MIX_ROWS>);
        else run(out_norm_kernel<T, 1, NO_MIX>);
    } else {
        if (mixed) run(out_norm_kernel<T, 4, MIX_ROWS>); else run(out_norm_kernel<T, 4, NO_MIX>);
    }
}

template <typename T>
void launch_norm_rows(const float* x32, const int32_t* rows_idx, const bf16* w, T* y, int rows, int width, int ld, float eps,
                      cudaStream_t s) {
    ProfileScope prof(KC_ROW, s);
    launch_kernel(norm_rows_kernel<T>, dim3(rows), dim3(256), 0, s, x32, rows_idx, w, y, width, ld, eps);
}

void launch_silu_f32(const float* gu, int ld_gu, float* act, int ld_act, int rows, int ff, cudaStream_t s) {
    ProfileScope prof(KC_ROW, s);
    launch_kernel(silu_f32_kernel, dim3(rows), dim3(256), 0, s, gu, ld_gu, act, ld_act, ff);
}

#define CPM_INSTANTIATE(T)                                                                                                          \
    template void launch_embed_rows<T>(const int32_t*, const bf16*, int, float, float*, T*, int, int, const StateCheck&, cudaStream_t); \
    template void launch_qkv_norm_append<T>(const QkvNormArgs&, int, cudaStream_t);                                                 \
    template void launch_out_norm<T>(float*, T*, const T*, const MoeMix&, float, const bf16*, int, int, int, float, cudaStream_t);  \
    template void launch_norm_rows<T>(const float*, const int32_t*, const bf16*, T*, int, int, int, float, cudaStream_t);
CPM_INSTANTIATE(bf16)
CPM_INSTANTIATE(float)
