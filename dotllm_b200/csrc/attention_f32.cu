// Float32 attention over the paged cache for heads of 64 or 128 channels (keys and values of one width): a kernel over
// tiles of 64 query rows for prompts and one over (page, KV head, token) for a few new tokens per sequence.
//
// The math is the generic kernel's (attention_generic.cu), all of it float32 with exact exponentials; like there a query's
// result depends on its position alone, never on how its sequence was cut into steps, which the 32-bit path relies on.  So the two
// kernels do the same operations on a query in the same order:
//   * a score is the sum of two chains of fused multiply-adds, over the even and over the odd channels in ascending order (one
//     packed instruction steps both), scaled, capped, biased, masked;
//   * a page of 64 keys (aligned to absolute positions) gives m = max(scores), p = exp(s - m), l = the sum of the 64 p in a fixed
//     tree (keys x, x + 16, x + 32, x + 48 in order, then the sixteen sums in a butterfly) and per channel again two chains, over
//     the page's even and odd keys;
//   * pages are merged in ascending order: M' = max(M, m), both sides scaled by exp(. - M').
// A key that a query does not see has weight 0 and changes no sum; a page is left out where the query sees none of its keys, and
// only there: whether it does follows from positions, never from a score, so that a score that is no number (which a maximum
// ignores) reaches the sums and the result.  Keys beyond the query are read only where a neighbour in the tile sees them.
//
// What bounds it.  Prompts: the FFMA pipes (74 TFLOP/s) and, about as much, the reads of shared memory that feed them; the generic
// kernel ran a warp per (token, head) and brought every tile of keys into shared memory once per token.  Here 64 rows share a
// page, a thread holds 4 rows x 4 scores and 4 rows x hd/16 outputs (128 threads with 8 rows each: 315 us where this takes 291; the
// packed multiply-adds issue half as often at the same rate and leave it there).  One prompt of 1,000 tokens, 32 heads of 128: 1,858 -> 295 us,
// 28 TFLOP/s over the visible scores, issue slots 50 % and shared memory 68 % busy.  Decode: the bytes of K and V; the generic kernel
// walked a sequence's keys one tile after the other, 64 blocks in all.  Here a page is a block's work, for all query heads of
// the KV head (several pages where the machine is full), and a second kernel merges the pages' parts: 8 sequences of up to 1,500 tokens, 8 KV heads of 64: 144 -> 18 us
// (blocks that walked four pages each took 22).
#include "common.cuh"
#include <atomic>

#define AF_ROWS 64                       // query rows per tile
#define AF_TILE_THREADS 256
#define AF_SPLIT_THREADS 256
#define AF_MAX_GROUP 16

struct AfScore {
    float scale, softcap;
    const float* slopes;
    int window, keep_first;
};

// First key of the window of the query at `pos`, and how many of the sequence's first keys stay visible in front of it.
__device__ __forceinline__ void af_range(const AfScore& sc, int pos, int& first, int& kept) {
    first = (sc.window > 0 && pos - sc.window + 1 > 0) ? pos - sc.window + 1 : 0;
    kept = min(sc.keep_first, first);
}
// Does the query see some key of the page at key0?
__device__ __forceinline__ bool af_sees(int key0, int pos, int first, int kept) {
    return key0 <= pos && (key0 < kept || key0 + DL_PAGE > first);
}
// The score of the key at j from the raw dot product; explicit roundings, so that both kernels get the same bits.
__device__ __forceinline__ float af_score(float dot, const AfScore& sc, float slope, int j, int pos) {
    float s = __fmul_rn(dot, sc.scale);
    if (sc.softcap > 0.f) s = __fmul_rn(sc.softcap, tanhf(__fdiv_rn(s, sc.softcap)));
    if (sc.slopes != nullptr) s = __fadd_rn(s, __fmul_rn(slope, (float)(j - pos)));
    return s;
}
// The base that weights' exponents are taken from (0 while no key has been seen: exp(-inf) is 0).
__device__ __forceinline__ float af_base(float m) { return m == -INFINITY ? 0.f : m; }
// A page's (m, l) into the running (M, L): factors of the running and of the page's output.
__device__ __forceinline__ void af_merge(float& M, float& L, float m, float l, float& e1, float& e2) {
    const float mn = fmaxf(M, m), base = af_base(mn);
    e1 = expf(__fsub_rn(M, base));
    e2 = expf(__fsub_rn(m, base));
    L = fmaf(L, e1, __fmul_rn(l, e2));
    M = mn;
}
__device__ __forceinline__ float af_blend(float a, float e1, float b, float e2) { return fmaf(a, e1, __fmul_rn(b, e2)); }
// What the merged output is multiplied by: the sink's term joins the denominator, the gate's sigmoid the result.
__device__ __forceinline__ float af_inverse(float M, float L, const float* sinks, const float* gate, int gate_stride, int t, int h) {
    float inv = 1.0f / (sinks != nullptr ? L + expf(sinks[h] - M) : L);
    if (gate != nullptr) inv *= 1.0f / (1.0f + expf(-gate[(size_t)t * gate_stride + h]));
    return inv;
}

// Two fused multiply-adds in one instruction.
__device__ __forceinline__ void af_fma2(float2& d, float ax, float ay, float bx, float by) {
    asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rd, {%0, %1};\n\t"
        "fma.rn.f32x2 rd, ra, rb, rd;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "+f"(d.x), "+f"(d.y)
        : "f"(ax), "f"(ay), "f"(bx), "f"(by));
}
__device__ __forceinline__ void af_dot4(float2& d, const float4& a, const float4& b) {
    af_fma2(d, a.x, a.y, b.x, b.y);
    af_fma2(d, a.z, a.w, b.z, b.w);
}

__device__ __forceinline__ void af_copy16(float* dst, const float* src, bool real) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int bytes = real ? 16 : 0;                       // 0: sixteen zeros are written and nothing is read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void af_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void af_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Shared-memory tiles: rows of 16-byte chunks, the chunk number exclusive-or-ed with the row's low three bits, so that eight rows' reads of
// one chunk meet different banks.
template <int CH> __device__ __forceinline__ int af_at(int row, int chunk) { return (row * CH + (chunk ^ (row & 7))) * 4; }

// ------------------------------------------------------------------ prompts
// Grid (head, tile): tile i is rows tile_row0[i] .. + 63 of the new tokens of sequence tile_seq[i].  Thread (ty, tx) holds rows
// ty + TY i, scores of keys tx + 16 j and channels tx + 16 c.
template <int HD>
__global__ void __launch_bounds__(AF_TILE_THREADS, 2)
attention_f32_tile_kernel(const float* __restrict__ q, int q_stride, float* __restrict__ out, int out_stride, const float* __restrict__ k_pool,
                          const float* __restrict__ v_pool, int n_pages, const int32_t* __restrict__ tile_seq,
                          const int32_t* __restrict__ tile_row0, const int32_t* __restrict__ seq_start, const int32_t* __restrict__ seq_new,
                          const int32_t* __restrict__ cu_new, const int32_t* __restrict__ block_table, int bt_stride, int nh, int nkv,
                          const AfScore sc, const float* __restrict__ gate, int gate_stride, const float* __restrict__ sinks) {
    constexpr int CH = HD / 4, DIMS = HD / 16, TY = AF_TILE_THREADS / 16, R = AF_ROWS / TY;
    extern __shared__ __align__(16) float af_smem[];
    float* qs = af_smem;                                   // [64][HD]
    float* ks = qs + AF_ROWS * HD;                         // [64 keys][HD]
    float* vs = ks + DL_PAGE * HD;                         // [HD][64 keys]
    float* ps = vs + HD * DL_PAGE;                         // [64][64 keys]
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const int h = blockIdx.x, kvh = h / (nh / nkv), b = tile_seq[blockIdx.y], row0 = tile_row0[blockIdx.y];
    const int n_rows = min(AF_ROWS, seq_new[b] - row0);
    if (n_rows <= 0) return;
    const int pos0 = seq_start[b] + row0, last = pos0 + n_rows - 1, t0 = cu_new[b] + row0;
    const int32_t* pages = block_table + (size_t)b * bt_stride;
    const float slope = sc.slopes != nullptr ? sc.slopes[h] : 0.f;

    int first0, kept0, first1, kept1;
    af_range(sc, pos0, first0, kept0);                     // the earliest row sees the earliest keys,
    af_range(sc, last, first1, kept1);                     // the latest row keeps the most first ones
    const int kept_pages = (kept1 + DL_PAGE - 1) / DL_PAGE, window_page = first0 / DL_PAGE, end_page = min(last / DL_PAGE + 1, bt_stride);
    auto next_page = [&](int p) {                          // the first page from p on that some row may see
        if (p >= kept_pages && p < window_page) p = window_page;
        return p;
    };
    auto page_id = [&](int p) { const int id = pages[p]; return id >= 0 && id < n_pages ? id : -1; };   // -1: given up (no row sees it); never read outside the pool
    auto fetch_k = [&](int p) {
        const int id = page_id(p);
        const float* src = k_pool + dl_k_offset(max(id, 0), nkv, kvh, 0, HD);
        for (int e = tid; e < DL_PAGE * CH; e += AF_TILE_THREADS)
            af_copy16(ks + af_at<CH>(e / CH, e % CH), src + 4 * e, id >= 0 && p * DL_PAGE + e / CH <= last);
    };
    auto fetch_v = [&](int p) {
        const int id = page_id(p);
        const float* src = v_pool + dl_v_offset(max(id, 0), nkv, kvh, 0, HD);
        for (int e = tid; e < HD * 16; e += AF_TILE_THREADS)
            af_copy16(vs + af_at<16>(e / 16, e % 16), src + 4 * e, id >= 0 && p * DL_PAGE + 4 * (e % 16) <= last);
    };
    for (int e = tid; e < AF_ROWS * CH; e += AF_TILE_THREADS) {
        const int r = e / CH, c = e % CH;
        af_copy16(qs + af_at<CH>(r, c), q + (size_t)(t0 + min(r, n_rows - 1)) * q_stride + (size_t)h * HD + 4 * c, r < n_rows);
    }
    int page = next_page(0);
    if (page < end_page) fetch_k(page);
    af_commit();
    if (page < end_page) fetch_v(page);
    af_commit();

    float A[R][DIMS], M[R], L[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        M[i] = -INFINITY, L[i] = 0.f;
#pragma unroll
        for (int c = 0; c < DIMS; ++c) A[i][c] = 0.f;
    }
    while (page < end_page) {
        const int next = next_page(page + 1);
        af_wait<1>();                                      // this page's keys (and the queries) have landed
        __syncthreads();
        float2 pair[R][4];
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) pair[i][j] = make_float2(0.f, 0.f);
#pragma unroll 2
        for (int c = 0; c < CH; ++c) {
            float4 kk[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) kk[j] = *reinterpret_cast<const float4*>(ks + af_at<CH>(tx + 16 * j, c));
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const float4 qq = *reinterpret_cast<const float4*>(qs + af_at<CH>(ty + TY * i, c));
#pragma unroll
                for (int j = 0; j < 4; ++j) af_dot4(pair[i][j], qq, kk[j]);
            }
        }
        float s[R][4];
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = __fadd_rn(pair[i][j].x, pair[i][j].y);
        __syncthreads();                                   // the keys have been used: the next page's may come
        if (next < end_page) fetch_k(next);
        af_commit();
        float e1[R], e2[R];                                // factors of the running output and of the page's
        // a page that every row sees whole needs no mask
        const int key0 = page * DL_PAGE;
        const bool there = page_id(page) >= 0;
        const bool whole = there && key0 + DL_PAGE - 1 <= pos0 && n_rows == AF_ROWS && (key0 >= first1 || key0 + DL_PAGE <= kept0);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int row = ty + TY * i, pos = pos0 + row;
            int first, kept;
            af_range(sc, pos, first, kept);
            float top = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = key0 + tx + 16 * j;
                const bool seen = whole || (there && row < n_rows && key <= pos && (key >= first || key < kept));
                s[i][j] = seen ? af_score(s[i][j], sc, slope, key, pos) : -INFINITY;
                top = fmaxf(top, s[i][j]);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
            const float base = af_base(top);
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                s[i][j] = expf(__fsub_rn(s[i][j], base));
                sum = __fadd_rn(sum, s[i][j]);
                ps[af_at<16>(row, (tx >> 2) + 4 * j) + (tx & 3)] = s[i][j];
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, o));
            e1[i] = 1.f, e2[i] = 0.f;                          // a page without a visible key changes nothing
            if (there && af_sees(key0, pos, first, kept)) af_merge(M[i], L[i], top, sum, e1[i], e2[i]);
        }
        af_wait<1>();                                      // this page's values have landed
        __syncthreads();
        bool careful = false;
        if (!whole) {                                      // 0 times a value that is no number would not be 0: such pages mask value by value
            bool odd = false;
            for (int e = tid; e < HD * DL_PAGE; e += AF_TILE_THREADS) odd = odd || !(fabsf(vs[e]) <= 3.402823466e38f);
            careful = __syncthreads_or(odd);
        }
        constexpr int HALF = DIMS / 2;                     // half of the channels at a time: the chains' registers
#pragma unroll
        for (int c0 = 0; c0 < DIMS; c0 += HALF) {
            float2 acc[R][HALF];
#pragma unroll
            for (int i = 0; i < R; ++i)
#pragma unroll
                for (int c = 0; c < HALF; ++c) acc[i][c] = make_float2(0.f, 0.f);
            if (!careful) {
#pragma unroll 2
                for (int kc = 0; kc < 16; ++kc) {
                    float4 vv[HALF];
#pragma unroll
                    for (int c = 0; c < HALF; ++c) vv[c] = *reinterpret_cast<const float4*>(vs + af_at<16>(tx + 16 * (c0 + c), kc));
#pragma unroll
                    for (int i = 0; i < R; ++i) {
                        const float4 pp = *reinterpret_cast<const float4*>(ps + af_at<16>(ty + TY * i, kc));
#pragma unroll
                        for (int c = 0; c < HALF; ++c) af_dot4(acc[i][c], pp, vv[c]);
                    }
                }
            } else {
#pragma unroll 1
                for (int kk = 0; kk < DL_PAGE; ++kk) {
                    const int key = key0 + kk;
#pragma unroll
                    for (int i = 0; i < R; ++i) {
                        const int row = ty + TY * i, pos = pos0 + row;
                        int first, kept;
                        af_range(sc, pos, first, kept);
                        if (row >= n_rows || key > pos || (key < first && key >= kept)) continue;
                        const float p = ps[af_at<16>(row, kk >> 2) + (kk & 3)];
#pragma unroll
                        for (int c = 0; c < HALF; ++c) {
                            const float v = vs[af_at<16>(tx + 16 * (c0 + c), kk >> 2) + (kk & 3)];
                            if (kk & 1) acc[i][c].y = fmaf(p, v, acc[i][c].y);
                            else acc[i][c].x = fmaf(p, v, acc[i][c].x);
                        }
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < R; ++i)
#pragma unroll
                for (int c = 0; c < HALF; ++c) A[i][c0 + c] = af_blend(A[i][c0 + c], e1[i], __fadd_rn(acc[i][c].x, acc[i][c].y), e2[i]);
        }
        __syncthreads();                                   // values and weights have been used
        if (next < end_page) fetch_v(next);
        af_commit();
        page = next;
    }
    af_wait<0>();
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int row = ty + TY * i;
        if (row >= n_rows) continue;
        const float inv = af_inverse(M[i], L[i], sinks, gate, gate_stride, t0 + row, h);
        float* o = out + (size_t)(t0 + row) * out_stride + (size_t)h * HD;
#pragma unroll
        for (int c = 0; c < DIMS; ++c) o[tx + 16 * c] = __fmul_rn(A[i][c], inv);
    }
}

// ------------------------------------------------------- a few new tokens
// Grid (pages, KV head, token): the token's queries of all G heads of the KV head over page x, then x + the grid's width and so on up to
// the token's own page.  The width is the table's up to the machine filled several times over (a captured step's table is as wide as
// its longest sequence may become: a block for every column would be blocks that find nothing to do).  part_o, part_ml: per (token, head, page)
// the output [HD], m and l (l -1: the token sees nothing of the page).  PAIRS: (head, channel) pairs a thread keeps.
template <int HD, int PAIRS>
__global__ void __launch_bounds__(AF_SPLIT_THREADS, HD == 64 ? 6 : 3)
attention_f32_split_kernel(const float* __restrict__ q, int q_stride, const float* __restrict__ k_pool, const float* __restrict__ v_pool,
                           int n_pages, const int32_t* __restrict__ token_seq, const int32_t* __restrict__ token_pos,
                           const int32_t* __restrict__ block_table, int bt_stride, int nh, int nkv, const AfScore sc,
                           float* __restrict__ part_o, float* __restrict__ part_ml) {
    constexpr int CH = HD / 4;
    extern __shared__ __align__(16) float af_smem[];
    float* ks = af_smem;                                   // [64 keys][HD]
    float* vs = ks + DL_PAGE * HD;                         // [HD][64 keys]
    float* qs = vs + HD * DL_PAGE;                         // [G][HD]
    const int G = nh / nkv;
    float* ps = qs + G * HD;                               // [G][64]
    dl_launch_dependents();
    dl_grid_dependency_wait();
    const int kvh = blockIdx.y, t = blockIdx.z;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int pos = token_pos[t], end = min(pos / DL_PAGE + 1, bt_stride);
    int first, kept;
    af_range(sc, pos, first, kept);
    bool asked = false;                                    // the queries are asked for behind the first page
    for (int page = blockIdx.x; page < end; page += gridDim.x) {
        const int key0 = page * DL_PAGE;
        const size_t part0 = ((size_t)t * nh + kvh * G) * bt_stride + page;      // head g's: + g * bt_stride
        const int id = block_table[(size_t)token_seq[t] * bt_stride + page];
        if (!af_sees(key0, pos, first, kept) || id < 0 || id >= n_pages) {      // nothing here for this token
            for (int g = tid; g < G; g += AF_SPLIT_THREADS) part_ml[(part0 + (size_t)g * bt_stride) * 2 + 1] = -1.f;
            continue;
        }
        auto visible = [&](int key) { return key <= pos && (key >= first || key < kept); };
        const float* ksrc = k_pool + dl_k_offset(id, nkv, kvh, 0, HD);
        for (int e = tid; e < DL_PAGE * CH; e += AF_SPLIT_THREADS) af_copy16(ks + af_at<CH>(e / CH, e % CH), ksrc + 4 * e, visible(key0 + e / CH));
        af_commit();
        const float* vsrc = v_pool + dl_v_offset(id, nkv, kvh, 0, HD);
        for (int e = tid; e < HD * 16; e += AF_SPLIT_THREADS) af_copy16(vs + af_at<16>(e / 16, e % 16), vsrc + 4 * e, key0 + 4 * (e % 16) <= pos);
        af_commit();
        for (int e = asked ? G * HD : tid; e < G * HD; e += AF_SPLIT_THREADS) qs[e] = q[(size_t)t * q_stride + (size_t)kvh * G * HD + e];
        asked = true;
        af_wait<1>();
        __syncthreads();
        for (int e = tid; e < G * DL_PAGE; e += AF_SPLIT_THREADS) {
            const int g = e / DL_PAGE, kk = e % DL_PAGE, key = key0 + kk;
            float2 pair = make_float2(0.f, 0.f);
#pragma unroll 8
            for (int c = 0; c < CH; ++c)
                af_dot4(pair, *reinterpret_cast<const float4*>(qs + g * HD + 4 * c), *reinterpret_cast<const float4*>(ks + af_at<CH>(kk, c)));
            const float dot = __fadd_rn(pair.x, pair.y);
            const float slope = sc.slopes != nullptr ? sc.slopes[kvh * G + g] : 0.f;
            ps[e] = visible(key) ? af_score(dot, sc, slope, key, pos) : -INFINITY;
        }
        __syncthreads();
        // a half warp per head: sixteen lanes with four keys each
        for (int g = warp * 2 + (lane >> 4); g < ((G + 1) & ~1); g += AF_SPLIT_THREADS / 16) {
            const int x = lane & 15, row = min(g, G - 1);
            float s[4], top = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) s[j] = ps[row * DL_PAGE + x + 16 * j], top = fmaxf(top, s[j]);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
            const float base = af_base(top);
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                s[j] = expf(__fsub_rn(s[j], base));
                sum = __fadd_rn(sum, s[j]);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, o));
            __syncwarp();
            if (g < G) {
#pragma unroll
                for (int j = 0; j < 4; ++j) ps[g * DL_PAGE + x + 16 * j] = s[j];
                if (x == 0) {
                    float* ml = part_ml + (part0 + (size_t)g * bt_stride) * 2;
                    ml[0] = top, ml[1] = sum;
                }
            }
        }
        af_wait<0>();
        __syncthreads();
        const bool whole = key0 + DL_PAGE - 1 <= pos && (key0 >= first || key0 + DL_PAGE <= kept);
#pragma unroll
        for (int a = 0; a < PAIRS; ++a) {
            const int e = tid + a * AF_SPLIT_THREADS;
            if (e >= G * HD) continue;
            const int g = e / HD, d = e % HD;
            float2 o = make_float2(0.f, 0.f);
#pragma unroll 8
            for (int kc = 0; kc < 16; ++kc) {
                const float4 vv = *reinterpret_cast<const float4*>(vs + af_at<16>(d, kc));
                const float4 pp = *reinterpret_cast<const float4*>(ps + g * DL_PAGE + 4 * kc);
                if (whole) {
                    af_dot4(o, pp, vv);
                } else {                                       // a value nobody may see may hold anything
                    const int key = key0 + 4 * kc;
                    if (visible(key)) o.x = fmaf(pp.x, vv.x, o.x);
                    if (visible(key + 1)) o.y = fmaf(pp.y, vv.y, o.y);
                    if (visible(key + 2)) o.x = fmaf(pp.z, vv.z, o.x);
                    if (visible(key + 3)) o.y = fmaf(pp.w, vv.w, o.y);
                }
            }
            part_o[(part0 + (size_t)g * bt_stride) * HD + d] = __fadd_rn(o.x, o.y);
        }
        __syncthreads();                                       // the page has been used
    }
}

// A block per (head, token): the pages' parts in ascending order.
#define AF_MERGE_AHEAD 16
template <int HD>
__global__ void __launch_bounds__(HD)
attention_f32_merge_kernel(float* __restrict__ out, int out_stride, const float* __restrict__ part_o, const float* __restrict__ part_ml,
                           int bt_stride, int nh, const int32_t* __restrict__ token_pos, const float* __restrict__ gate, int gate_stride,
                           const float* __restrict__ sinks) {
    dl_launch_dependents();
    dl_grid_dependency_wait();
    const int h = blockIdx.x, t = blockIdx.y, d = threadIdx.x;
    const int end = min(token_pos[t] / DL_PAGE + 1, bt_stride);
    const float2* ml = reinterpret_cast<const float2*>(part_ml) + ((size_t)t * nh + h) * bt_stride;
    const float* po = part_o + ((size_t)t * nh + h) * bt_stride * HD + d;
    float M = -INFINITY, L = 0.f, A = 0.f;
    for (int p0 = 0; p0 < end; p0 += AF_MERGE_AHEAD) {
        float2 x[AF_MERGE_AHEAD];
        float o[AF_MERGE_AHEAD];
#pragma unroll
        for (int i = 0; i < AF_MERGE_AHEAD; ++i) {         // parts that were not written are read and not used
            const int p = min(p0 + i, end - 1);
            x[i] = ml[p];
            o[i] = po[(size_t)p * HD];
        }
#pragma unroll
        for (int i = 0; i < AF_MERGE_AHEAD; ++i) {
            if (p0 + i >= end || x[i].y < 0.f) continue;
            float e1, e2;
            af_merge(M, L, x[i].x, x[i].y, e1, e2);
            A = af_blend(A, e1, o[i], e2);
        }
    }
    out[(size_t)t * out_stride + (size_t)h * HD + d] = __fmul_rn(A, af_inverse(M, L, sinks, gate, gate_stride, t, h));
}

template <typename K>
static cudaError_t af_size(K kernel, std::atomic<unsigned long long>& sized, int smem) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 64 || !(sized.load() >> dev & 1)) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        if (dev < 64) sized.fetch_or(1ull << dev);
    }
    return cudaSuccess;
}

#define AF_CHECK(what)                                                                                                              \
    DL_REQUIRE(nh > 0 && nkv > 0 && n_pages > 0 && nh % nkv == 0, what ": bad sizes");                                              \
    DL_REQUIRE(hd == 64 || hd == 128, what ": heads of %d channels", hd);                                                           \
    DL_REQUIRE(q_stride >= nh * hd && out_stride >= nh * hd, what ": row strides shorter than the rows");                           \
    DL_REQUIRE(q_stride % 4 == 0 && ((uintptr_t)q % 16) == 0 && ((uintptr_t)k_pool % 16) == 0 && ((uintptr_t)v_pool % 16) == 0,     \
               what ": unaligned operands");                                                                                        \
    DL_REQUIRE(window >= 0 && keep_first >= 0 && softcap >= 0.f, what ": negative window, kept tokens or cap");                      \
    DL_REQUIRE(gate == nullptr || gate_stride >= nh, what ": a row of gate logits holds one per query head");

// Prompts: tiles of 64 rows (tile_seq, tile_row0: int32 [n_tiles]).  Pools as in attention_generic.cu, float32.
extern "C" int dl_attention_f32_tile(const float* q, int q_stride, float* out, int out_stride, const float* k_pool, const float* v_pool,
                                     int n_pages, const int32_t* tile_seq, const int32_t* tile_row0, int n_tiles, const int32_t* seq_start,
                                     const int32_t* seq_new, const int32_t* cu_new, const int32_t* block_table, int bt_stride, int nh,
                                     int nkv, int hd, float scale, int window, float softcap, const float* slopes, const float* gate,
                                     int gate_stride, int keep_first, const float* sinks, void* stream) {
    AF_CHECK("attention_f32_tile");
    DL_REQUIRE(n_tiles >= 0 && n_tiles <= 65535, "attention_f32_tile: %d tiles", n_tiles);
    if (n_tiles == 0) return DL_OK;
    const AfScore sc = {scale, softcap, slopes, window, keep_first};
    const dim3 grid(nh, n_tiles), block(AF_TILE_THREADS);
    const int smem = (AF_ROWS * hd + 2 * DL_PAGE * hd + AF_ROWS * DL_PAGE) * 4;
    cudaStream_t s = (cudaStream_t)stream;
#define AF_TILE(HD)                                                                                                                 \
    {                                                                                                                               \
        static std::atomic<unsigned long long> sized{0};                                                                            \
        const cudaError_t e = af_size(attention_f32_tile_kernel<HD>, sized, smem);                                                  \
        if (e != cudaSuccess) return dl_fail(DL_ERR_LAUNCH, "attention_f32_tile: %s", cudaGetErrorString(e));                       \
        attention_f32_tile_kernel<HD><<<grid, block, smem, s>>>(q, q_stride, out, out_stride, k_pool, v_pool, n_pages, tile_seq,    \
                                                                tile_row0, seq_start, seq_new, cu_new, block_table, bt_stride, nh,  \
                                                                nkv, sc, gate, gate_stride, sinks);                                 \
    }
    if (hd == 64) AF_TILE(64) else AF_TILE(128)
#undef AF_TILE
    DL_CHECK_LAUNCH("attention_f32_tile");
    return DL_OK;
}

// A few new tokens per sequence.  part_o: float32 [tokens, nh, bt_stride, hd], part_ml [tokens, nh, bt_stride, 2] (8-byte aligned), scratch.
extern "C" int dl_attention_f32_split(const float* q, int q_stride, float* out, int out_stride, const float* k_pool, const float* v_pool,
                                      int n_pages, const int32_t* token_seq, const int32_t* token_pos, const int32_t* block_table,
                                      int bt_stride, int n_tokens, int nh, int nkv, int hd, float scale, int window, float softcap,
                                      const float* slopes, const float* gate, int gate_stride, int keep_first, const float* sinks,
                                      float* part_o, float* part_ml, void* stream) {
    AF_CHECK("attention_f32_split");
    const int G = nh / nkv;
    DL_REQUIRE(G <= AF_MAX_GROUP, "attention_f32_split: %d query heads a KV head, the kernel takes up to %d", G, AF_MAX_GROUP);
    DL_REQUIRE(n_tokens >= 0 && n_tokens <= 65535 && nkv <= 65535 && bt_stride >= 1, "attention_f32_split: %d tokens", n_tokens);
    DL_REQUIRE(part_o != nullptr && part_ml != nullptr && ((uintptr_t)part_ml % 8) == 0, "attention_f32_split: no room for the pages' parts");
    if (n_tokens == 0) return DL_OK;
    const AfScore sc = {scale, softcap, slopes, window, keep_first};
    const long fill = (16L * dl_sm_count() + (long)nkv * n_tokens - 1) / ((long)nkv * n_tokens);     // some three times what the machine holds at once
    const dim3 grid(bt_stride < fill ? bt_stride : (unsigned)(fill > 1 ? fill : 1), nkv, n_tokens), block(AF_SPLIT_THREADS);
    const int smem = (2 * DL_PAGE * hd + G * hd + G * DL_PAGE) * 4, most = (2 * DL_PAGE * hd + AF_MAX_GROUP * (hd + DL_PAGE)) * 4;
    cudaStream_t s = (cudaStream_t)stream;
    const int pairs = (G * hd + AF_SPLIT_THREADS - 1) / AF_SPLIT_THREADS;
    cudaError_t e = cudaSuccess;
#define AF_SPLIT(HD, P)                                                                                                             \
    {                                                                                                                               \
        static std::atomic<unsigned long long> sized{0};                                                                            \
        e = af_size(attention_f32_split_kernel<HD, P>, sized, most);                                                                \
        if (e == cudaSuccess)                                                                                                       \
            e = dl_launch_dependent(attention_f32_split_kernel<HD, P>, grid, block, (size_t)smem, s, q, q_stride, k_pool, v_pool,   \
                                    n_pages, token_seq, token_pos, block_table, bt_stride, nh, nkv, sc, part_o, part_ml);           \
    }
    if (hd == 64) {
        if (pairs <= 1) AF_SPLIT(64, 1) else if (pairs <= 2) AF_SPLIT(64, 2) else AF_SPLIT(64, 4)
    } else {
        if (pairs <= 1) AF_SPLIT(128, 1) else if (pairs <= 2) AF_SPLIT(128, 2) else if (pairs <= 4) AF_SPLIT(128, 4) else AF_SPLIT(128, 8)
    }
#undef AF_SPLIT
    if (e == cudaSuccess)
        e = hd == 64 ? dl_launch_dependent(attention_f32_merge_kernel<64>, dim3(nh, n_tokens), dim3(64), 0, s, out, out_stride, part_o, part_ml,
                                           bt_stride, nh, token_pos, gate, gate_stride, sinks)
                     : dl_launch_dependent(attention_f32_merge_kernel<128>, dim3(nh, n_tokens), dim3(128), 0, s, out, out_stride, part_o, part_ml,
                                           bt_stride, nh, token_pos, gate, gate_stride, sinks);
    if (e != cudaSuccess) return dl_fail(DL_ERR_LAUNCH, "attention_f32_split: %s", cudaGetErrorString(e));
    return DL_OK;
}

DL_PACKED(dl_attention_f32_tile)
DL_PACKED(dl_attention_f32_split)
