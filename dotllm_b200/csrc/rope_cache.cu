// Rotary position encoding of Q and K fused with the write of K and V into the paged cache.
//
// Rotation is the half-split pairing (x[i], x[i + d/2]) -> (x0*cos - x1*sin, x0*sin + x1*cos)
// of the reference's rope_f32 with rope_type == 1 (native/kernels/rope_f32.cu:6-57) and of
// its CPU twin (src/DotLLM.Cpu/Kernels/RoPE.cs:250-256); the reference then copies the K and
// V rows into the cache (src/DotLLM.Cuda/CudaKvCache.cs:64-97).  Here the angles come from a
// float32 cos/sin table built once on the host in float64, the arithmetic is float32, Q is
// rotated in place and rotated K goes straight to its cache page.  V pages are transposed.
//
// Values may have a width of their own (`vd` channels a head against `hd` key channels), and the
// projections' biases may be added here, in float32, before the rotation (`q_bias` [nh*hd], `k_bias`
// [nkv*hd], `v_bias` [nkv*vd], each NULL for none): a projection with biases then needs no pass of its own.
#include "common.cuh"

// The rotation, written with explicit roundings so that both kernels below (and any compiler
// version) produce the same bits: no contraction into fused multiply-adds.
__device__ __forceinline__ float rope_lo(float x0, float x1, float c, float s) { return __fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, s)); }
__device__ __forceinline__ float rope_hi(float x0, float x1, float c, float s) { return __fadd_rn(__fmul_rn(x0, s), __fmul_rn(x1, c)); }

// Grid: (token, head) with the query heads first, then the KV heads; a block's threads each take
// one rotation pair (query heads) or one dimension (KV heads), so a decode step's handful of
// tokens still spreads over hundreds of blocks and no thread loops over dependent loads.
template <typename T>
__global__ void __launch_bounds__(128)
rope_cache_write_kernel(T* __restrict__ q, int q_stride, const T* __restrict__ k, int k_stride,
                        const T* __restrict__ v, int v_stride, const float* __restrict__ cos_t,
                        const float* __restrict__ sin_t, int rotary_dim, int table_rows,
                        const int32_t* __restrict__ token_seq, const int32_t* __restrict__ token_pos,
                        const int32_t* __restrict__ block_table, int bt_stride, T* __restrict__ k_pool,
                        T* __restrict__ v_pool, int n_pages, int nh, int nkv, int hd, int vd,
                        const float* __restrict__ q_bias, const float* __restrict__ k_bias,
                        const float* __restrict__ v_bias, int write_cache) {
    dl_launch_dependents();
    dl_grid_dependency_wait();
    const int t = blockIdx.x;
    const int pos = token_pos[t];
    const int half = rotary_dim / 2;
    if (pos < 0 || (half > 0 && pos >= table_rows)) return;      // host-validated; never index outside
    const float* cs = cos_t + (size_t)pos * half;
    const float* sn = sin_t + (size_t)pos * half;

    if ((int)blockIdx.y < nh) {                                   // a query head: rotate in place
        T* p = q + (size_t)t * q_stride + (size_t)blockIdx.y * hd;
        const float* qb = q_bias != nullptr ? q_bias + (size_t)blockIdx.y * hd : nullptr;
        for (int i = threadIdx.x; i < half; i += blockDim.x) {
            float x0 = dl_to_f32<T>(p[i]), x1 = dl_to_f32<T>(p[i + half]);
            if (qb != nullptr) x0 += qb[i], x1 += qb[i + half];
            const float c = cs[i], s = sn[i];
            p[i] = dl_from_f32<T>(rope_lo(x0, x1, c, s));
            p[i + half] = dl_from_f32<T>(rope_hi(x0, x1, c, s));
        }
        if (qb != nullptr)                                        // the channels beyond the rotation take their bias too
            for (int d = 2 * half + threadIdx.x; d < hd; d += blockDim.x) p[d] = dl_from_f32<T>(dl_to_f32<T>(p[d]) + qb[d]);
        return;
    }
    if (!write_cache) return;
    const int h = blockIdx.y - nh;                                // a KV head: rotate K on its way to the page
    const int seq = token_seq[t];
    const int page = block_table[(size_t)seq * bt_stride + pos / DL_PAGE];
    if (page < 0 || page >= n_pages) return;
    const int in_page = pos % DL_PAGE;
    const T* krow = k + (size_t)t * k_stride + (size_t)h * hd;
    const T* vrow = v + (size_t)t * v_stride + (size_t)h * vd;
    const float* kb = k_bias != nullptr ? k_bias + (size_t)h * hd : nullptr;
    const float* vb = v_bias != nullptr ? v_bias + (size_t)h * vd : nullptr;
    T* kdst = k_pool + dl_k_offset(page, nkv, h, in_page, hd);
    for (int d = threadIdx.x; d < hd; d += blockDim.x) {
        float kv;
        if (d < half) {
            kv = rope_lo(dl_to_f32<T>(krow[d]) + (kb ? kb[d] : 0.f), dl_to_f32<T>(krow[d + half]) + (kb ? kb[d + half] : 0.f), cs[d], sn[d]);
        } else if (d < 2 * half) {
            const int i = d - half;
            kv = rope_hi(dl_to_f32<T>(krow[i]) + (kb ? kb[i] : 0.f), dl_to_f32<T>(krow[d]) + (kb ? kb[d] : 0.f), cs[i], sn[i]);
        } else {
            kv = dl_to_f32<T>(krow[d]) + (kb ? kb[d] : 0.f);
        }
        kdst[d] = dl_from_f32<T>(kv);
    }
    for (int d = threadIdx.x; d < vd; d += blockDim.x)
        v_pool[dl_v_offset(page, nkv, h, d, vd) + in_page] = vb ? dl_from_f32<T>(dl_to_f32<T>(vrow[d]) + vb[d]) : vrow[d];
}

// The same work for steps of many tokens (prefill).  Grid: (tile of 64 packed tokens, head).  A
// block of a KV head stages the tile's V rows in shared memory and writes them transposed, token
// fastest, so that the tokens of one page (consecutive positions of one sequence) fill whole
// 128-byte lines of the transposed V page instead of one 2-byte element each.
#define RT_TOKENS 64
#ifndef RT_THREADS
#define RT_THREADS 256
#endif
template <typename T>
__global__ void __launch_bounds__(RT_THREADS)
rope_cache_write_tile_kernel(T* __restrict__ q, int q_stride, const T* __restrict__ k, int k_stride,
                             const T* __restrict__ v, int v_stride, const float* __restrict__ cos_t,
                             const float* __restrict__ sin_t, int rotary_dim, int table_rows,
                             const int32_t* __restrict__ token_seq, const int32_t* __restrict__ token_pos,
                             const int32_t* __restrict__ block_table, int bt_stride, T* __restrict__ k_pool,
                             T* __restrict__ v_pool, int n_pages, int n_tokens, int nh, int nkv, int hd, int vd,
                             const float* __restrict__ q_bias, const float* __restrict__ k_bias,
                             const float* __restrict__ v_bias, int write_cache) {
    extern __shared__ __align__(16) unsigned char rt_raw[];
    T* tile = reinterpret_cast<T*>(rt_raw);                  // [64 tokens][vd + pad]: V rows of one KV head
    __shared__ int s_pos[RT_TOKENS], s_page[RT_TOKENS];
    dl_launch_dependents();
    dl_grid_dependency_wait();
    const int t0 = blockIdx.x * RT_TOKENS;
    const int nt = min(RT_TOKENS, n_tokens - t0);
    const int half = rotary_dim / 2;
    // KV heads first: their blocks do more (K to its page, V through the transposing tile) and should not start last
    const int kv_first = write_cache ? nkv : 0;
    const bool is_q = (int)blockIdx.y >= kv_first;
    const int pitch = vd + (int)(4 / sizeof(T));             // an odd number of 32-bit words (even vd): no bank conflicts on the transpose
    if (threadIdx.x < RT_TOKENS) {
        int pos = -1, page = -1;
        if ((int)threadIdx.x < nt) {
            pos = token_pos[t0 + threadIdx.x];
            if (pos < 0 || (half > 0 && pos >= table_rows)) pos = -1;    // host-validated; never index outside
            if (pos >= 0 && !is_q && write_cache) {
                page = block_table[(size_t)token_seq[t0 + threadIdx.x] * bt_stride + pos / DL_PAGE];
                if (page < 0 || page >= n_pages) page = -1;
            }
        }
        s_pos[threadIdx.x] = pos;
        s_page[threadIdx.x] = page;
    }
    __syncthreads();
    if (is_q) {                                              // a query head: rotate in place
        for (int idx = threadIdx.x; idx < nt * half; idx += RT_THREADS) {
            const int i = idx / half, p = idx - i * half;
            const int pos = s_pos[i];
            if (pos < 0) continue;
            const int qh = (int)blockIdx.y - kv_first;
            T* row = q + (size_t)(t0 + i) * q_stride + (size_t)qh * hd;
            float x0 = dl_to_f32<T>(row[p]), x1 = dl_to_f32<T>(row[p + half]);
            if (q_bias != nullptr) x0 += q_bias[(size_t)qh * hd + p], x1 += q_bias[(size_t)qh * hd + p + half];
            const float c = cos_t[(size_t)pos * half + p], s = sin_t[(size_t)pos * half + p];
            row[p] = dl_from_f32<T>(rope_lo(x0, x1, c, s));
            row[p + half] = dl_from_f32<T>(rope_hi(x0, x1, c, s));
        }
        const int rest = hd - 2 * half;
        if (q_bias != nullptr && rest > 0) {                 // the channels beyond the rotation take their bias too
            const int qh = (int)blockIdx.y - kv_first;
            for (int idx = threadIdx.x; idx < nt * rest; idx += RT_THREADS) {
                const int i = idx / rest, d = 2 * half + idx - i * rest;
                if (s_pos[i] < 0) continue;
                T* row = q + (size_t)(t0 + i) * q_stride + (size_t)qh * hd;
                row[d] = dl_from_f32<T>(dl_to_f32<T>(row[d]) + q_bias[(size_t)qh * hd + d]);
            }
        }
        return;
    }
    if (!write_cache) return;
    const int h = blockIdx.y;                                // a KV head: rotate K on its way to the page, stage V
    const float* kb = k_bias != nullptr ? k_bias + (size_t)h * hd : nullptr;
    const float* vb = v_bias != nullptr ? v_bias + (size_t)h * vd : nullptr;
    for (int idx = threadIdx.x; idx < nt * vd; idx += RT_THREADS) {
        const int i = idx / vd, d = idx - i * vd;
        const T raw = v[(size_t)(t0 + i) * v_stride + (size_t)h * vd + d];
        tile[i * pitch + d] = vb ? dl_from_f32<T>(dl_to_f32<T>(raw) + vb[d]) : raw;
    }
    for (int idx = threadIdx.x; idx < nt * hd; idx += RT_THREADS) {
        const int i = idx / hd, d = idx - i * hd;
        const int page = s_page[i], pos = s_pos[i];
        if (page < 0) continue;
        const T* krow = k + (size_t)(t0 + i) * k_stride + (size_t)h * hd;
        const float* cs = cos_t + (size_t)pos * half;
        const float* sn = sin_t + (size_t)pos * half;
        float kv;
        if (d < half) {
            kv = rope_lo(dl_to_f32<T>(krow[d]) + (kb ? kb[d] : 0.f), dl_to_f32<T>(krow[d + half]) + (kb ? kb[d + half] : 0.f), cs[d], sn[d]);
        } else if (d < 2 * half) {
            const int j = d - half;
            kv = rope_hi(dl_to_f32<T>(krow[j]) + (kb ? kb[j] : 0.f), dl_to_f32<T>(krow[d]) + (kb ? kb[d] : 0.f), cs[j], sn[j]);
        } else {
            kv = dl_to_f32<T>(krow[d]) + (kb ? kb[d] : 0.f);
        }
        k_pool[dl_k_offset(page, nkv, h, pos % DL_PAGE, hd) + d] = dl_from_f32<T>(kv);
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < RT_TOKENS * vd; idx += RT_THREADS) {    // token fastest
        const int i = idx % RT_TOKENS, d = idx / RT_TOKENS;
        if (i >= nt) continue;
        const int page = s_page[i];
        if (page < 0) continue;
        v_pool[dl_v_offset(page, nkv, h, d, vd) + (s_pos[i] % DL_PAGE)] = tile[i * pitch + d];
    }
}

// The tile kernel for rows that can be moved 16 bytes at a time: E = 8 bfloat16 or 4 float32 elements (hd a multiple of E, the
// rotated part a multiple of 2 E channels, 16-byte aligned rows, values as wide as keys).  A thread moves E rotation pairs of Q
// or K, or E channels beyond the rotation, or E values of V, instead of one element.  Biases (float32, NULL for none) are added
// before the rotation.
//
// The work is a read and a write of every row.  What bounds it is how many loads are in flight: a multiprocessor's blocks of
// float32 prompts are few, with a handful of units a thread, so a thread loads BATCH units (rows, cosines and sines) before it
// rotates and stores the first; stores to Q in place would otherwise hold the next unit's loads back.  bfloat16 rows are half as
// long and come with more tokens (blocks), and a second unit's registers cost more blocks than its loads bring.  Measured: float32,
// 1,000 tokens of 32 + 8 heads of 128, 59 us one element a thread, 14 us here; bfloat16, 9,431 tokens of 32 + 8 heads of 64,
// 33 us with a batch of one (3.5 TB/s of rows read and written), 54 us with two.
template <typename T>
struct RopeUnit {
    static constexpr int E = 16 / (int)sizeof(T);
    static constexpr int BATCH = sizeof(T) == 4 ? 4 : 1;
    alignas(16) T x[E];
};
template <typename T>
__device__ __forceinline__ RopeUnit<T> rope_load(const T* p) {
    RopeUnit<T> u;
    *reinterpret_cast<uint4*>(u.x) = *reinterpret_cast<const uint4*>(p);
    return u;
}
template <typename T>
__device__ __forceinline__ void rope_store(T* p, const RopeUnit<T>& u) { *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(u.x); }

template <typename T>
__device__ __forceinline__ void rope_add(RopeUnit<T>& u, const float* b) {
#pragma unroll
    for (int e = 0; e < RopeUnit<T>::E; ++e) u.x[e] = dl_from_f32<T>(dl_to_f32<T>(u.x[e]) + b[e]);
}

template <typename T>
__device__ __forceinline__ void rope_rotate(RopeUnit<T>& u0, RopeUnit<T>& u1, const float4* c4, const float4* s4, const float* b0, const float* b1) {
#pragma unroll
    for (int e = 0; e < RopeUnit<T>::E; ++e) {
        const float4 cv = c4[e / 4], sv = s4[e / 4];
        const float c = e % 4 == 0 ? cv.x : e % 4 == 1 ? cv.y : e % 4 == 2 ? cv.z : cv.w;
        const float s = e % 4 == 0 ? sv.x : e % 4 == 1 ? sv.y : e % 4 == 2 ? sv.z : sv.w;
        float f0 = dl_to_f32<T>(u0.x[e]), f1 = dl_to_f32<T>(u1.x[e]);
        if (b0 != nullptr) f0 += b0[e], f1 += b1[e];
        u0.x[e] = dl_from_f32<T>(rope_lo(f0, f1, c, s));
        u1.x[e] = dl_from_f32<T>(rope_hi(f0, f1, c, s));
    }
}

// The units of one head's rows in a tile, from `src` to where `dst_of(row)` says (NULL: the row is left out).  `rest` units a row
// beyond the rotation are moved too.
template <typename T, typename Dst>
__device__ __forceinline__ void rope_units(const T* src, int stride, int nt, int pairs, int rest, int half, const int* s_pos, const float* cos_t,
                                           const float* sin_t, const float* bias, Dst dst_of) {
    constexpr int E = RopeUnit<T>::E, BATCH = RopeUnit<T>::BATCH;
    const int per = pairs + rest, n = nt * per;
    for (int base = threadIdx.x; base < n; base += BATCH * RT_THREADS) {
        RopeUnit<T> x0[BATCH], x1[BATCH];
        float4 c[BATCH][E / 4], s[BATCH][E / 4];
        T* dst[BATCH];
        int at[BATCH];
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            const int idx = base + u * RT_THREADS;
            const int i = min(idx, n - 1) / per, g = min(idx, n - 1) - i * per;
            dst[u] = idx < n ? dst_of(i) : nullptr;
            if (dst[u] == nullptr) continue;
            const T* row = src + (size_t)i * stride;
            if (g < pairs) {
                at[u] = g * E;
                const size_t angle = (size_t)s_pos[i] * half + g * E;
                x0[u] = rope_load(row + at[u]);
                x1[u] = rope_load(row + half + at[u]);
#pragma unroll
                for (int e = 0; e < E / 4; ++e) {
                    c[u][e] = *reinterpret_cast<const float4*>(cos_t + angle + 4 * e);
                    s[u][e] = *reinterpret_cast<const float4*>(sin_t + angle + 4 * e);
                }
            } else {
                at[u] = 2 * half + (g - pairs) * E;
                x0[u] = rope_load(row + at[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            if (dst[u] == nullptr) continue;
            if (at[u] < half) {
                rope_rotate(x0[u], x1[u], c[u], s[u], bias ? bias + at[u] : nullptr, bias ? bias + half + at[u] : nullptr);
                rope_store(dst[u] + at[u], x0[u]);
                rope_store(dst[u] + half + at[u], x1[u]);
            } else {
                if (bias != nullptr) rope_add(x0[u], bias + at[u]);
                rope_store(dst[u] + at[u], x0[u]);
            }
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(RT_THREADS)
rope_cache_write_tile_vec_kernel(T* __restrict__ q, int q_stride, const T* __restrict__ k, int k_stride,
                                 const T* __restrict__ v, int v_stride, const float* __restrict__ cos_t,
                                 const float* __restrict__ sin_t, int rotary_dim, int table_rows, const int32_t* __restrict__ token_seq,
                                 const int32_t* __restrict__ token_pos, const int32_t* __restrict__ block_table, int bt_stride,
                                 T* __restrict__ k_pool, T* __restrict__ v_pool, int n_pages,
                                 int n_tokens, int nh, int nkv, int hd, const float* __restrict__ q_bias,
                                 const float* __restrict__ k_bias, const float* __restrict__ v_bias, int write_cache) {
    constexpr int E = RopeUnit<T>::E;
    extern __shared__ __align__(16) unsigned char rt_raw[];
    T* tile = reinterpret_cast<T*>(rt_raw);                  // [64 tokens][hd + a 32-bit word]: V rows of one KV head
    __shared__ int s_pos[RT_TOKENS], s_page[RT_TOKENS];
    dl_launch_dependents();
    dl_grid_dependency_wait();
    const int t0 = blockIdx.x * RT_TOKENS;
    const int nt = min(RT_TOKENS, n_tokens - t0);
    const int half = rotary_dim / 2;
    const int pairs = half / E, rest = (hd - rotary_dim) / E;   // groups of E rotation pairs, and of E channels beyond them, per head
    // KV heads first: their blocks do more (K to its page, V through the transposing tile) and should not start last
    const int kv_first = write_cache ? nkv : 0;
    const bool is_q = (int)blockIdx.y >= kv_first;
    const int pitch = hd + 4 / (int)sizeof(T);
    if (threadIdx.x < RT_TOKENS) {
        int pos = -1, page = -1;
        if ((int)threadIdx.x < nt) {
            pos = token_pos[t0 + threadIdx.x];
            if (pos < 0 || (half > 0 && pos >= table_rows)) pos = -1;      // host-validated; never index outside
            if (pos >= 0 && !is_q && write_cache) {
                page = block_table[(size_t)token_seq[t0 + threadIdx.x] * bt_stride + pos / DL_PAGE];
                if (page < 0 || page >= n_pages) page = -1;
            }
        }
        s_pos[threadIdx.x] = pos;
        s_page[threadIdx.x] = page;
    }
    __syncthreads();
    if (is_q) {                                              // a query head: rotate in place
        const int qh = (int)blockIdx.y - kv_first;
        T* rows = q + (size_t)t0 * q_stride + (size_t)qh * hd;
        // without a bias the channels beyond the rotation stay as they are
        rope_units<T>(rows, q_stride, nt, pairs, q_bias != nullptr ? rest : 0, half, s_pos, cos_t, sin_t,
                      q_bias != nullptr ? q_bias + (size_t)qh * hd : nullptr,
                      [&](int i) { return s_pos[i] < 0 ? nullptr : rows + (size_t)i * q_stride; });
        return;
    }
    if (!write_cache) return;
    const int h = blockIdx.y;                                // a KV head: rotate K on its way to the page, stage V
    const float* vb = v_bias != nullptr ? v_bias + (size_t)h * hd : nullptr;
    const int units = hd / E;
#pragma unroll 4
    for (int idx = threadIdx.x; idx < nt * units; idx += RT_THREADS) {
        const int i = idx / units, d = (idx - i * units) * E;
        RopeUnit<T> x = rope_load(v + (size_t)(t0 + i) * v_stride + (size_t)h * hd + d);
        if (vb != nullptr) rope_add(x, vb + d);
        uint32_t* dst = reinterpret_cast<uint32_t*>(tile + i * pitch + d);          // 4-byte aligned: so are the pitch and d
        const uint32_t* words = reinterpret_cast<const uint32_t*>(x.x);
        dst[0] = words[0]; dst[1] = words[1]; dst[2] = words[2]; dst[3] = words[3];
    }
    rope_units<T>(k + (size_t)t0 * k_stride + (size_t)h * hd, k_stride, nt, pairs, rest, half, s_pos, cos_t, sin_t,
                  k_bias != nullptr ? k_bias + (size_t)h * hd : nullptr,
                  [&](int i) { return s_page[i] < 0 ? nullptr : k_pool + dl_k_offset(s_page[i], nkv, h, s_pos[i] % DL_PAGE, hd); });
    __syncthreads();
#pragma unroll 4
    for (int idx = threadIdx.x; idx < RT_TOKENS * hd; idx += RT_THREADS) {    // token fastest
        const int i = idx % RT_TOKENS, d = idx / RT_TOKENS;
        if (i >= nt) continue;
        const int page = s_page[i];
        if (page < 0) continue;
        v_pool[dl_v_offset(page, nkv, h, d, hd) + (s_pos[i] % DL_PAGE)] = tile[i * pitch + d];
    }
}

extern "C" int dl_rope_cache_write(void* q, int q_stride, const void* k, int k_stride, const void* v, int v_stride,
                                   int dtype, const float* cos_t, const float* sin_t, int rotary_dim,
                                   int table_rows, const int32_t* token_seq, const int32_t* token_pos,
                                   const int32_t* block_table, int bt_stride, void* k_pool, void* v_pool,
                                   int n_pages, int n_tokens, int nh, int nkv, int hd, int vd, const float* q_bias,
                                   const float* k_bias, const float* v_bias, int write_cache, void* stream) {
    DL_REQUIRE(n_tokens >= 0 && nh > 0 && nkv > 0 && hd > 0 && vd > 0, "rope_cache_write: bad sizes");
    DL_REQUIRE(rotary_dim >= 0 && rotary_dim <= hd && rotary_dim % 2 == 0,
               "rope_cache_write: rotary_dim %d must be even and at most head_dim %d", rotary_dim, hd);
    DL_REQUIRE(rotary_dim == 0 || (cos_t && sin_t && table_rows > 0), "rope_cache_write: rotation needs tables");
    DL_REQUIRE(q_stride >= nh * hd && (!write_cache || (k_stride >= nkv * hd && v_stride >= nkv * vd)),
               "rope_cache_write: row strides shorter than the rows");
    DL_REQUIRE(!write_cache || (k && v && k_pool && v_pool && block_table && n_pages > 0),
               "rope_cache_write: cache write needs k, v, pools and a block table");
    if (n_tokens == 0) return DL_OK;
    cudaStream_t s = (cudaStream_t)stream;
    DL_REQUIRE(nh + nkv <= 65535, "rope_cache_write: too many heads");
    cudaError_t e;
    const size_t elem = dtype == DL_F32 ? 4 : 2;
    const size_t tile_smem = (size_t)RT_TOKENS * (vd + 4 / elem) * elem;
    const bool biases_aligned = ((uintptr_t)q_bias % 16) == 0 && ((uintptr_t)k_bias % 16) == 0 && ((uintptr_t)v_bias % 16) == 0;
    if (n_tokens >= RT_TOKENS && tile_smem <= 48 * 1024 && (dtype == DL_F32 || dtype == DL_BF16)) {
        // queries that are neither rotated nor biased stay as they are: no blocks for them
        const int q_blocks = (rotary_dim > 0 || q_bias != nullptr) ? nh : 0;
        if (q_blocks == 0 && !write_cache) return DL_OK;
        dim3 tgrid((n_tokens + RT_TOKENS - 1) / RT_TOKENS, (write_cache ? nkv : 0) + q_blocks);
        const int unit = 16 / (int)elem;                     // elements of 16 bytes
        const bool aligned = ((uintptr_t)q % 16) == 0 && q_stride % unit == 0 && ((uintptr_t)cos_t % 16) == 0 &&
                             ((uintptr_t)sin_t % 16) == 0 &&
                             (!write_cache || (((uintptr_t)k % 16) == 0 && ((uintptr_t)v % 16) == 0 && k_stride % unit == 0 &&
                                               v_stride % unit == 0 && ((uintptr_t)k_pool % 16) == 0));
        if (vd == hd && hd % unit == 0 && rotary_dim % (2 * unit) == 0 && aligned && biases_aligned) {
            if (dtype == DL_F32)
                e = dl_launch_dependent(rope_cache_write_tile_vec_kernel<float>, tgrid, dim3(RT_THREADS), tile_smem, s, (float*)q,
                                        q_stride, (const float*)k, k_stride, (const float*)v, v_stride, cos_t, sin_t, rotary_dim,
                                        table_rows, token_seq, token_pos, block_table, bt_stride, (float*)k_pool, (float*)v_pool,
                                        n_pages, n_tokens, nh, nkv, hd, q_bias, k_bias, v_bias, write_cache);
            else
                e = dl_launch_dependent(rope_cache_write_tile_vec_kernel<__nv_bfloat16>, tgrid, dim3(RT_THREADS), tile_smem, s,
                                        (__nv_bfloat16*)q, q_stride, (const __nv_bfloat16*)k, k_stride, (const __nv_bfloat16*)v,
                                        v_stride, cos_t, sin_t, rotary_dim, table_rows, token_seq, token_pos, block_table, bt_stride,
                                        (__nv_bfloat16*)k_pool, (__nv_bfloat16*)v_pool, n_pages, n_tokens, nh, nkv, hd, q_bias,
                                        k_bias, v_bias, write_cache);
            if (e != cudaSuccess) return dl_fail(DL_ERR_LAUNCH, "rope_cache_write: %s", cudaGetErrorString(e));
            return DL_OK;
        }
        if (dtype == DL_F32)
            e = dl_launch_dependent(rope_cache_write_tile_kernel<float>, tgrid, dim3(RT_THREADS), tile_smem, s, (float*)q, q_stride,
                                    (const float*)k, k_stride, (const float*)v, v_stride, cos_t, sin_t, rotary_dim, table_rows,
                                    token_seq, token_pos, block_table, bt_stride, (float*)k_pool, (float*)v_pool, n_pages,
                                    n_tokens, nh, nkv, hd, vd, q_bias, k_bias, v_bias, write_cache);
        else
            e = dl_launch_dependent(rope_cache_write_tile_kernel<__nv_bfloat16>, tgrid, dim3(RT_THREADS), tile_smem, s,
                                    (__nv_bfloat16*)q, q_stride, (const __nv_bfloat16*)k, k_stride, (const __nv_bfloat16*)v,
                                    v_stride, cos_t, sin_t, rotary_dim, table_rows, token_seq, token_pos, block_table,
                                    bt_stride, (__nv_bfloat16*)k_pool, (__nv_bfloat16*)v_pool, n_pages, n_tokens, nh, nkv, hd,
                                    vd, q_bias, k_bias, v_bias, write_cache);
        if (e != cudaSuccess) return dl_fail(DL_ERR_LAUNCH, "rope_cache_write: %s", cudaGetErrorString(e));
        return DL_OK;
    }
    dim3 grid(n_tokens, write_cache ? nh + nkv : nh);
    if (dtype == DL_F32)
        e = dl_launch_dependent(rope_cache_write_kernel<float>, grid, dim3(128), 0, s, (float*)q, q_stride, (const float*)k,
                                k_stride, (const float*)v, v_stride, cos_t, sin_t, rotary_dim, table_rows, token_seq,
                                token_pos, block_table, bt_stride, (float*)k_pool, (float*)v_pool, n_pages, nh, nkv, hd,
                                vd, q_bias, k_bias, v_bias, write_cache);
    else if (dtype == DL_BF16)
        e = dl_launch_dependent(rope_cache_write_kernel<__nv_bfloat16>, grid, dim3(128), 0, s, (__nv_bfloat16*)q, q_stride,
                                (const __nv_bfloat16*)k, k_stride, (const __nv_bfloat16*)v, v_stride, cos_t, sin_t,
                                rotary_dim, table_rows, token_seq, token_pos, block_table, bt_stride,
                                (__nv_bfloat16*)k_pool, (__nv_bfloat16*)v_pool, n_pages, nh, nkv, hd, vd, q_bias, k_bias,
                                v_bias, write_cache);
    else
        return dl_fail(DL_ERR_UNSUPPORTED, "rope_cache_write: dtype %d", dtype);
    if (e != cudaSuccess) return dl_fail(DL_ERR_LAUNCH, "rope_cache_write: %s", cudaGetErrorString(e));
    return DL_OK;
}

DL_PACKED(dl_rope_cache_write)
