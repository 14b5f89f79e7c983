// The two recurrences with a decay per key channel over prompts, 32 tokens at a time, in float32 throughout (the chunked forms of Yang et
// al., "Gated Linear Attention Transformers with Hardware-Efficient Training" and "Parallelizing Linear Transformers with the Delta
// Rule over Sequence Length", here without divisions by running products of decays):
//
//   gated linear attention (gla.cu)    S_t = diag(a_t) S_(t-1) + k_t v_t^T                        o_t = S_t^T q_t
//   gated delta rule (delta.cu)        S_t = diag(a_t) S_(t-1) + k_t u_t^T,                       o_t = S_t^T q_t
//                                      u_t = b_t (v_t - (diag(a_t) S_(t-1))^T k_t)
//
// The scans of those files walk a sequence token by token: a chain of dependent steps, two warps a scheduler waiting for it (2,048
// tokens of 16 heads 227 us for the first, 320 for the second; at no time is a pipe or the memory busy).  Over a chunk of L tokens that
// starts from S_0, with P_t = a_1 ... a_t (per channel), both are matrix products:
//
//   A[t][j] = sum_c q_t[c] k_j[c] (a_(j+1) ... a_t)[c]  (j <= t),      N[t][j] = b_t sum_c k_t[c] k_j[c] (a_(j+1) ... a_t)[c]  (j < t)
//   U = (I + N)^-1 diag(b) (V - K+ S_0)   (delta; U = V otherwise),    K+_t = P_t k_t
//   O = Q+ S_0 + A U,   Q+_t = P_t q_t;      S_L = diag(P_L) S_0 + K'^T U,   K'_j = (a_(j+1) ... a_L) k_j
//
// Every factor is a running product of decays in [0, 1]: nothing is divided, so nothing can overflow however fast a channel
// forgets.  What does not depend on S_0 is made for all chunks side by side: a lane owns a key token j and steps its decayed key
// through the chunk (A and N); with the delta rule 96 lanes solve (I + N) [W | T] = diag(b) [K+ | I] by forward substitution, a
// column each, and
//
//   S_L = (diag(P_L) - K'^T W) S_0 + K'^T T V,      O = (Q+ - A W) S_0 + A T V
//
// leaves one product a chunk, G [96 x 96] times [S_0; V], for the walk from chunk to chunk (columns of S never mix: a block owns CW
// value channels of one (sequence, head), a thread 6 rows x CW/8 columns).  Without the delta rule the state's part is a diagonal,
// so nothing needs to walk: every chunk's contribution K'^T V, an elementwise pass over the chunks' states, and every chunk's O
// run as three launches.
//
// Measured (bfloat16 rows, kernels alone, state of 64 x 128 a head): gated linear attention, one sequence of 2,048 tokens, 16 heads: 227 ->
// 95 us (46 the states, 14 the pass, 35 the outputs), eight such sequences 1,131 -> 720.  Delta rule, three sequences of 3,743 tokens in all, 32 heads:
// 734 -> 489 us (208 for G, 281 the walk); one of 2,048, 16 heads: 320 -> 199.  What bounds them now is the FFMA pipes' issue
// (18 and 50 million multiply-adds a thousand tokens and head).
//
// A token that is no number (an infinity or a NaN among its inputs) must not reach the outputs of the tokens before it, and 0 times it
// is a NaN: A and T hold nothing but zeros above their diagonals, and an output that is not finite is summed again over its own and
// earlier tokens only (the same sums in the same order, so the bits of the tokens before do not change).
//
// The sums run in another order than the scans': the results agree to float32 rounding, not to the bit.  A float32 run therefore
// keeps the scans (there a sequence may be cut anywhere), and so do steps of few tokens.
#include "common.cuh"
#include <atomic>

#define CK_L 32                          // tokens a chunk
#define CK_DIM 64                        // key channels a head, at most (padded with zeros)
#define CK_X (CK_DIM + CK_L)             // rows of [S_0; V], and rows and columns of G
#define CK_THREADS 128
#define CK_LDT (CK_L + 4)                // rows along tokens, in floats: 16-byte aligned, eight rows' reads meet different banks
#define CK_LDX (CK_X + 4)

__device__ __forceinline__ bool ck_finite(float v) { return fabsf(v) <= 3.402823466e38f; }
__device__ __forceinline__ float ck_silu(float v) { return v / (1.0f + expf(-v)); }
__device__ __forceinline__ void ck_copy16(float* dst, const float* src, bool live) {      // 16 bytes, zeros where not live
    const int bytes = live ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ck_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int K> __device__ __forceinline__ void ck_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(K) : "memory"); }

template <int N> struct CkVec;
template <> struct CkVec<4> { using type = float4; };
template <> struct CkVec<2> { using type = float2; };
template <int N> __device__ __forceinline__ void ck_load(const float* p, float (&v)[N]) {
    const typename CkVec<N>::type x = *reinterpret_cast<const typename CkVec<N>::type*>(p);
    const float* e = reinterpret_cast<const float*>(&x);
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = e[i];
}
template <int N> __device__ __forceinline__ void ck_store(float* p, const float (&v)[N]) {
    typename CkVec<N>::type x;
    float* e = reinterpret_cast<float*>(&x);
#pragma unroll
    for (int i = 0; i < N; ++i) e[i] = v[i];
    *reinterpret_cast<typename CkVec<N>::type*>(p) = x;
}
__device__ __forceinline__ void ck_load(const __nv_bfloat16* p, float (&v)[4]) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&raw.x), b = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
    v[0] = __low2float(a), v[1] = __high2float(a), v[2] = __low2float(b), v[3] = __high2float(b);
}
// acc[i][e] += sum over 4 NK values k of a[(16 i) * LDA + k] * b[k * LDB + e]
template <int RN, int N, int NK, int LDA, int LDB>
__device__ __forceinline__ void ck_product(float (&acc)[RN][N], const float* a, const float* b) {
#pragma unroll 4
    for (int k4 = 0; k4 < NK; ++k4) {
        float bv[4][N];
#pragma unroll
        for (int k = 0; k < 4; ++k) ck_load<N>(b + (4 * k4 + k) * LDB, bv[k]);
#pragma unroll
        for (int i = 0; i < RN; ++i) {
            const float4 av = *reinterpret_cast<const float4*>(a + 16 * i * LDA + 4 * k4);
#pragma unroll
            for (int e = 0; e < N; ++e)
                acc[i][e] = fmaf(av.w, bv[3][e], fmaf(av.z, bv[2][e], fmaf(av.y, bv[1][e], fmaf(av.x, bv[0][e], acc[i][e]))));
        }
    }
}

// One row of a product once more, over its first n values k alone (in ck_product's order), from the sums at `from` (distance `apart`; NULL:
// from 0): for an output that is not finite.  Rare, so one value after the other: it must not cost the kernels registers.
template <int N, int LDB>
__device__ __forceinline__ void ck_row_again(float* dst, const float* a, const float* b, int n, const float* from, int apart) {
#pragma unroll 1
    for (int e = 0; e < N; ++e) {
        float acc = from != nullptr ? from[e * apart] : 0.f;
#pragma unroll 1
        for (int k = 0; k < n; ++k) acc = fmaf(a[k], b[k * LDB + e], acc);
        dst[e] = acc;
    }
}
template <int N>
__device__ __forceinline__ bool ck_all_finite(const float (&v)[N]) {
    bool ok = true;
#pragma unroll
    for (int e = 0; e < N; ++e) ok = ok && ck_finite(v[e]);
    return ok;
}

// What the kernels have of a chunk.
//
// Chunks of all sequences lie one behind the other: chunk c of sequence b is piece ck_piece0(b) + c.  With ck_piece0(b) = floor((cu_new[b] +
// 31 b) / 32) a sequence of n tokens has at least ceil(n / 32) pieces before the next one's, and all have at most floor((tokens +
// 31 sequences) / 32) in all, which the host knows without reading cu_new.  The operands of a window of pieces (`lo` .. `lo` + n - 1)
// lie in the scratch at a time: what it holds follows the tokens, whatever the sequences' lengths.
struct CkRange {
    int t0, n, first, count, slot;       // the sequence's first row, its tokens, the chunk's first of them and how many, the slot
};
__device__ __forceinline__ bool ck_sequence(CkRange& r, const int32_t* cu_new, const int32_t* slots, int n_slots, int b) {
    r.t0 = cu_new[b], r.n = cu_new[b + 1] - r.t0, r.first = 0, r.count = min(CK_L, r.n), r.slot = slots[b];
    return r.n > 0 && r.slot >= 0 && r.slot < n_slots;
}
__device__ __forceinline__ int ck_piece0(int cu, int b) { return (int)(((unsigned)cu + (CK_L - 1) * (unsigned)b) / CK_L); }
// The chunk of a piece (every warp searches for itself: 32 sequences at a time, what it needs of them asked for at once); false where the
// piece holds none.
__device__ __forceinline__ bool ck_find(CkRange& r, const int32_t* cu_new, const int32_t* slots, int n_slots, int n_seqs, int piece, int lane) {
    int b = 0, step = 1;
    while (step * 32 < n_seqs) step *= 32;
    for (;;) {                                             // the last sequence whose first piece is not behind this one
        const int i = b + lane * step, at = min(i, n_seqs - 1);
        const int cu = cu_new[at], cu1 = cu_new[at + 1], slot = slots[at];
        const int w = __popc(__ballot_sync(0xffffffffu, i < n_seqs && ck_piece0(cu, i) <= piece)) - 1;
        b += w * step;
        if (step == 1) {
            r.t0 = __shfl_sync(0xffffffffu, cu, w), r.n = __shfl_sync(0xffffffffu, cu1, w) - r.t0, r.slot = __shfl_sync(0xffffffffu, slot, w);
            r.first = (piece - ck_piece0(r.t0, b)) * CK_L, r.count = min(CK_L, r.n - r.first);
            return r.first < r.n && r.slot >= 0 && r.slot < n_slots;
        }
        step /= 32;
    }
}

// Lane j of a warp: its key, decayed step by step, against every later token's query (aq) and key (ak): sixteen channels a warp.
template <bool DELTA>
__device__ __forceinline__ void ck_pairs(const float* sq, const float* sk, const float* sa, float (&aq)[CK_L], float (&ak)[CK_L], int warp, int lane) {
#pragma unroll
    for (int t = 0; t < CK_L; ++t) aq[t] = 0.f, ak[t] = 0.f;
#pragma unroll 1
    for (int c = warp * (CK_DIM / 4); c < (warp + 1) * (CK_DIM / 4); ++c) {
        const float kj = sk[c * CK_LDT + lane];
        float y = 0.f;
#pragma unroll
        for (int t4 = 0; t4 < CK_L / 4; ++t4) {
            const float4 a4 = *reinterpret_cast<const float4*>(sa + c * CK_LDT + 4 * t4), q4 = *reinterpret_cast<const float4*>(sq + c * CK_LDT + 4 * t4);
            const float4 k4 = DELTA ? *reinterpret_cast<const float4*>(sk + c * CK_LDT + 4 * t4) : q4;
            const float at[4] = {a4.x, a4.y, a4.z, a4.w}, qt[4] = {q4.x, q4.y, q4.z, q4.w}, kt[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int t = 4 * t4 + i;
                y = t == lane ? kj : y * at[i];
                aq[t] = fmaf(qt[i], y, aq[t]);
                if (DELTA) ak[t] = fmaf(kt[i], y, ak[t]);
            }
        }
    }
}

// In place, a channel's row: K'_j = (a_(j+1) ... a_L) k_j; returns P_L.
__device__ __forceinline__ float ck_keys_to_end(float* k, const float* a) {
    float s = 1.f;
#pragma unroll 2
    for (int t4 = CK_L / 4 - 1; t4 >= 0; --t4) {
        float4 k4 = *reinterpret_cast<const float4*>(k + 4 * t4);
        const float4 a4 = *reinterpret_cast<const float4*>(a + 4 * t4);
        k4.w *= s, s *= a4.w;
        k4.z *= s, s *= a4.z;
        k4.y *= s, s *= a4.y;
        k4.x *= s, s *= a4.x;
        *reinterpret_cast<float4*>(k + 4 * t4) = k4;
    }
    return s;
}
// In place, a channel's row: Q+_t = P_t q_t.
__device__ __forceinline__ void ck_queries_from_start(float* q, const float* a) {
    float p = 1.f;
#pragma unroll 2
    for (int t4 = 0; t4 < CK_L / 4; ++t4) {
        float4 q4 = *reinterpret_cast<const float4*>(q + 4 * t4);
        const float4 a4 = *reinterpret_cast<const float4*>(a + 4 * t4);
        p *= a4.x, q4.x *= p;
        p *= a4.y, q4.y *= p;
        p *= a4.z, q4.z *= p;
        p *= a4.w, q4.w *= p;
        *reinterpret_cast<float4*>(q + 4 * t4) = q4;
    }
}

// ------------------------------------------------------------ the delta rule
// A block per (piece of the window, head): G.  q, k [tokens, G*dim] (unit vectors, q scaled), g [tokens, H*dim] the decays, beta [tokens, H].
#define CK_DELTA_SMEM ((3 * CK_DIM * CK_LDT + 4 * CK_L * CK_L + 2 * CK_L * CK_LDT + CK_L + CK_DIM) * 4)
__global__ void __launch_bounds__(CK_THREADS, 4)
delta_chunk_prepare_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ g, const float* __restrict__ beta,
                           const int32_t* __restrict__ cu_new, const int32_t* __restrict__ slots, int n_slots, int n_seqs, float* __restrict__ G, int H,
                           int group, int dim, int lo) {
    extern __shared__ __align__(16) float ck_smem[];
    float* sq = ck_smem;                                   // [64][LDT]: q, then Q+, by channel
    float* sk = sq + CK_DIM * CK_LDT;                      // k, then K'
    float* sa = sk + CK_DIM * CK_LDT;                      // decays
    float* part = sa + CK_DIM * CK_LDT;                    // the warps' shares of A, then of N; then [L][LDX]: -W and T side by side
    float* sA = part + 4 * CK_L * CK_L;                    // [L][LDT]
    float* sn = sA + CK_L * CK_LDT;                        // [L][LDT]
    float* sb = sn + CK_L * CK_LDT;                        // [L]
    float* s_end = sb + CK_L;                              // [64]
    static_assert(CK_L * CK_LDX <= 4 * CK_L * CK_L, "W and T lie where the shares were");
    dl_launch_dependents();
    dl_grid_dependency_wait();
    const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, kvh = h / group;
    CkRange r;
    if (!ck_find(r, cu_new, slots, n_slots, n_seqs, lo + blockIdx.x, lane)) return;
    for (int e = tid; e < CK_L * CK_DIM; e += CK_THREADS) {
        const int t = e / CK_DIM, c = e % CK_DIM;
        float qv = 0.f, kv = 0.f, av = t < r.count ? 0.f : 1.f;    // a token that is not there decays nothing and adds nothing
        if (t < r.count && c < dim) {
            const long row = r.t0 + r.first + t, at = row * (H / group) * dim + (long)kvh * dim + c;
            qv = q[at], kv = k[at], av = g[row * H * dim + (long)h * dim + c];
        }
        sq[c * CK_LDT + t] = qv, sk[c * CK_LDT + t] = kv, sa[c * CK_LDT + t] = av;
    }
    if (tid < CK_L) sb[tid] = tid < r.count ? beta[(long)(r.t0 + r.first + tid) * H + h] : 0.f;
    __syncthreads();
    constexpr int W = CK_L * CK_L;
    {
        float aq[CK_L], ak[CK_L];
        ck_pairs<true>(sq, sk, sa, aq, ak, warp, lane);
#pragma unroll
        for (int t = 0; t < CK_L; ++t) part[(warp * CK_L + t) * CK_L + lane] = aq[t];
        __syncthreads();
        for (int e = tid; e < W; e += CK_THREADS) {
            const int t = e / CK_L, j = e % CK_L;
            sA[t * CK_LDT + j] = j <= t ? (part[e] + part[W + e]) + (part[2 * W + e] + part[3 * W + e]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int t = 0; t < CK_L; ++t) part[(warp * CK_L + t) * CK_L + lane] = ak[t];
        __syncthreads();
        for (int e = tid; e < W; e += CK_THREADS) {
            const int t = e / CK_L, j = e % CK_L;
            sn[t * CK_LDT + j] = j < t ? ((part[e] + part[W + e]) + (part[2 * W + e] + part[3 * W + e])) * sb[t] : 0.f;
        }
        __syncthreads();
    }
    if (tid < CK_X) {                                      // column `tid` of [W | T]
        float x[CK_L], p = 1.f;
#pragma unroll
        for (int t = 0; t < CK_L; ++t) {
            float right;
            if (tid < CK_DIM) {
                p *= sa[tid * CK_LDT + t];
                right = sk[tid * CK_LDT + t] * p;
            } else {
                right = t == tid - CK_DIM ? 1.f : 0.f;
            }
            float acc[4] = {sb[t] * right, 0.f, 0.f, 0.f};
#pragma unroll
            for (int s4 = 0; s4 < (t + 3) / 4; ++s4) {
                const float4 n4 = *reinterpret_cast<const float4*>(sn + t * CK_LDT + 4 * s4);
                acc[0] = fmaf(-n4.x, x[4 * s4], acc[0]);
                if (4 * s4 + 1 < t) acc[1] = fmaf(-n4.y, x[4 * s4 + 1], acc[1]);
                if (4 * s4 + 2 < t) acc[2] = fmaf(-n4.z, x[4 * s4 + 2], acc[2]);
                if (4 * s4 + 3 < t) acc[3] = fmaf(-n4.w, x[4 * s4 + 3], acc[3]);
            }
            x[t] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
            part[t * CK_LDX + tid] = tid < CK_DIM ? -x[t] : x[t];
        }
    }
    __syncthreads();
    if (tid < CK_DIM) s_end[tid] = ck_keys_to_end(sk + tid * CK_LDT, sa + tid * CK_LDT);
    else ck_queries_from_start(sq + (tid - CK_DIM) * CK_LDT, sa + (tid - CK_DIM) * CK_LDT);
    __syncthreads();
    // G = [diag(P_L) | 0; Q+ | 0] + [K'^T; A] [-W | T]: thread (rg, cg) of 16 x 8 takes rows rg + 16 i, columns 4 cg + 32 p
    float* out = G + ((long)blockIdx.x * H + h) * (CK_X * CK_X);
    const int rg = tid >> 3, cg = tid & 7;
#pragma unroll 1
    for (int p = 0; p < 3; ++p) {
        const int col = 32 * p + 4 * cg;
        float top[4][4], low[2][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) top[i][e] = rg + 16 * i == col + e ? s_end[col + e] : 0.f;
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) low[i][e] = col < CK_DIM ? sq[(col + e) * CK_LDT + rg + 16 * i] : 0.f;
        ck_product<4, 4, CK_L / 4, CK_LDT, CK_LDX>(top, sk + rg * CK_LDT, part + col);
        ck_product<2, 4, CK_L / 4, CK_LDT, CK_LDX>(low, sA + rg * CK_LDT, part + col);
#pragma unroll
        for (int i = 0; i < 4; ++i) ck_store<4>(out + (rg + 16 * i) * CK_X + col, top[i]);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int t = rg + 16 * i;
            float* dst = out + (CK_DIM + t) * CK_X + col;
            ck_store<4>(dst, low[i]);
            if (!ck_all_finite(low[i]))
                ck_row_again<4, CK_LDX>(dst, sA + t * CK_LDT, part + col, t + 1, col < CK_DIM ? sq + col * CK_LDT + t : nullptr, CK_LDT);
        }
    }
}

// The walk over the window's chunks of a sequence: thread (rg, cg) of 16 x 8, rows rg + 16 i of G, columns N cg .. of [S_0; V] (N = CW / 8).  G comes in two halves of its
// columns: while one is used the other, or the next chunk's, is under way.
template <int CW>
__global__ void __launch_bounds__(CK_THREADS, 3)
delta_chunk_walk_kernel(const float* __restrict__ v, const float* __restrict__ G, const int32_t* __restrict__ cu_new,
                        const int32_t* __restrict__ slots, float* __restrict__ state, long slot_stride, int n_slots, float* __restrict__ out, int H,
                        int dim, int vdim, int lo, int n_pieces) {
    constexpr int N = CW / 8, HALF = CK_X / 2;
    extern __shared__ __align__(16) float ck_smem[];
    float* s_g = ck_smem;                                  // [96][LDX]
    float* s_x = s_g + CK_X * CK_LDX;                      // two of [96][CW]: S_0, then V
    dl_launch_dependents();
    dl_grid_dependency_wait();
    const int tid = threadIdx.x, rg = tid >> 3, cg = tid & 7, h = blockIdx.y, b = blockIdx.z;
    CkRange r;
    if (!ck_sequence(r, cu_new, slots, n_slots, b)) return;
    const int first = ck_piece0(r.t0, b) - lo;             // the sequence's first piece, from the window's
    const int begin = max(0, -first), end = min((r.n + CK_L - 1) / CK_L, n_pieces - first);      // its chunks in the window
    if (begin >= end) return;
    const int n = r.n, col = blockIdx.x * CW + N * cg;     // vdim is a multiple of 4: a thread's columns are all there or all beyond
    const bool col_ok = col < vdim;
    float* S = state + (long)r.slot * slot_stride + (long)h * dim * vdim;
    auto bring = [&](int chunk, int half) {
        const float* src = G + ((long)(first + chunk) * H + h) * (CK_X * CK_X) + half * HALF;
        for (int e = tid; e < CK_X * (HALF / 4); e += CK_THREADS)
            ck_copy16(s_g + (e / (HALF / 4)) * CK_LDX + half * HALF + 4 * (e % (HALF / 4)), src + (e / (HALF / 4)) * CK_X + 4 * (e % (HALF / 4)), true);
    };
    bring(begin, 0);
    ck_commit();
    bring(begin, 1);
    ck_commit();
    const float* v_at = v + ((long)r.t0 * H + h) * vdim + col;
    float* o_at = out + ((long)r.t0 * H + h) * vdim + col;
    const long step = (long)H * vdim;
    float vv[2][N], acc[6][N];
    auto fetch_v = [&](int chunk) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int t = chunk * CK_L + rg + 16 * i;
            if (t < n && col_ok) ck_load<N>(v_at + t * step, vv[i]);
            else {
#pragma unroll
                for (int e = 0; e < N; ++e) vv[i][e] = 0.f;
            }
        }
    };
    fetch_v(begin);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int c = rg + 16 * i;
#pragma unroll
        for (int e = 0; e < N; ++e) acc[i][e] = c < dim && col_ok ? S[(long)c * vdim + col + e] : 0.f;
    }
    for (int chunk = begin; chunk < end; ++chunk) {
        float* x = s_x + (chunk & 1) * CK_X * CW;
#pragma unroll
        for (int i = 0; i < 4; ++i) ck_store<N>(x + (rg + 16 * i) * CW + N * cg, acc[i]);
#pragma unroll
        for (int i = 0; i < 2; ++i) ck_store<N>(x + (CK_DIM + rg + 16 * i) * CW + N * cg, vv[i]);
        fetch_v(chunk + 1);
#pragma unroll
        for (int i = 0; i < 6; ++i)
#pragma unroll
            for (int e = 0; e < N; ++e) acc[i][e] = 0.f;
        ck_wait<1>();
        __syncthreads();                                   // G's first half, the state and the values are there
        ck_product<6, N, HALF / 4, CK_LDX, CW>(acc, s_g + rg * CK_LDX, x + N * cg);
        __syncthreads();                                   // G's first half has been used
        if (chunk + 1 < end) bring(chunk + 1, 0);
        ck_commit();
        ck_wait<1>();
        __syncthreads();                                   // its second half is there
        float half_o[2][N];                                // the outputs so far
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < N; ++e) half_o[i][e] = acc[4 + i][e];
        ck_product<6, N, HALF / 4, CK_LDX, CW>(acc, s_g + rg * CK_LDX + HALF, x + HALF * CW + N * cg);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int t = rg + 16 * i;
            if (chunk * CK_L + t >= n || !col_ok) continue;
            float* dst = o_at + (chunk * CK_L + t) * step;
            ck_store<N>(dst, acc[4 + i]);
            if (!ck_all_finite(acc[4 + i])) {
                ck_store<N>(dst, half_o[i]);
                ck_row_again<N, CW>(dst, s_g + (CK_DIM + t) * CK_LDX + HALF, x + HALF * CW + N * cg, CK_DIM - HALF + t + 1, dst, 1);
            }
        }
        __syncthreads();                                   // and has been used
        if (chunk + 1 < end) bring(chunk + 1, 1);
        ck_commit();
    }
    ck_wait<0>();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int c = rg + 16 * i;
        if (c < dim && col_ok) {
#pragma unroll
            for (int e = 0; e < N; ++e) S[(long)c * vdim + col + e] = acc[i][e];
        }
    }
}

// --------------------------------------------------- gated linear attention
#define CK_GLA_COLS 64                   // value channels that a block's threads take at a time: (rg, cg) of 16 x 16, four columns each
#define CK_GLA_THREADS 256
struct CkGla {                           // per (piece of the window, head), float32
    float* qa;                           // [L][96]: Q+, then A
    float* end;                          // [64]: P_L
    float* states;                       // [64][vdim]: K'^T V, then the state before the chunk
};

// The chunk's rows of v, columns col0 .. + 63, through silu where asked, zeros beyond, into [L][64].
__device__ __forceinline__ void ck_bring_v(float* s_v, const __nv_bfloat16* v, long v_ld, int v_silu, const CkRange& r, int h, int vdim, int col0, int tid) {
    for (int e = tid; e < CK_L * (CK_GLA_COLS / 4); e += CK_GLA_THREADS) {
        const int t = e / (CK_GLA_COLS / 4), c = (e % (CK_GLA_COLS / 4)) * 4;
        float x[4] = {0.f, 0.f, 0.f, 0.f};
        if (t < r.count && col0 + c < vdim) {
            ck_load(v + (long)(r.t0 + r.first + t) * v_ld + (long)h * vdim + col0 + c, x);
            if (v_silu) {
#pragma unroll
                for (int i = 0; i < 4; ++i) x[i] = ck_silu(x[i]);
            }
        }
        ck_store<4>(s_v + t * CK_GLA_COLS + c, x);
    }
}

// A block per (piece, head): Q+, A, P_L and K'^T V.  z, z_bias as in dl_gla_scan.
__global__ void __launch_bounds__(CK_GLA_THREADS)
gla_chunk_states_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ v, long ld, const float* __restrict__ z, long z_ld,
                        const float* __restrict__ z_bias, const int32_t* __restrict__ cu_new, const int32_t* __restrict__ slots, int n_slots, int n_seqs,
                        CkGla out, int H, int dim, int vdim, float q_scale, float inv_tau, int lo) {
    __shared__ __align__(16) float sq[CK_DIM * CK_LDT], sk[CK_DIM * CK_LDT], sa[CK_DIM * CK_LDT];
    __shared__ __align__(16) float part[4 * CK_L * CK_L];  // the warps' shares of A; then 64 columns of V
    dl_launch_dependents();
    dl_grid_dependency_wait();
    const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    CkRange r;
    if (!ck_find(r, cu_new, slots, n_slots, n_seqs, lo + blockIdx.x, lane)) return;
    const long piece = (long)blockIdx.x * H + h;
    for (int e = tid; e < CK_L * CK_DIM; e += CK_GLA_THREADS) {
        const int t = e / CK_DIM, c = e % CK_DIM;
        float qv = 0.f, kv = 0.f, av = t < r.count ? 0.f : 1.f;    // a token that is not there decays nothing and adds nothing
        if (t < r.count && c < dim) {
            const long row = r.t0 + r.first + t;
            qv = dl_to_f32<__nv_bfloat16>(q[row * ld + (long)h * dim + c]), kv = dl_to_f32<__nv_bfloat16>(k[row * ld + (long)h * dim + c]);
            if (z != nullptr) {
                const float zz = z[row * z_ld + (long)h * dim + c] + z_bias[h * dim + c];
                av = expf((fminf(zz, 0.f) - log1pf(expf(-fabsf(zz)))) * inv_tau);
            } else {
                qv = ck_silu(qv), kv = ck_silu(kv), av = z_bias[h];
            }
            qv *= q_scale;
        }
        sq[c * CK_LDT + t] = qv, sk[c * CK_LDT + t] = kv, sa[c * CK_LDT + t] = av;
    }
    __syncthreads();
    if (warp < 4) {
        float aq[CK_L], ak[CK_L];
        ck_pairs<false>(sq, sk, sa, aq, ak, warp, lane);
#pragma unroll
        for (int t = 0; t < CK_L; ++t) part[(warp * CK_L + t) * CK_L + lane] = aq[t];
    }
    __syncthreads();
    float* qa = out.qa + piece * (CK_L * CK_X);
    constexpr int W = CK_L * CK_L;
    for (int e = tid; e < W; e += CK_GLA_THREADS)
        qa[(e / CK_L) * CK_X + CK_DIM + e % CK_L] =
            e % CK_L <= e / CK_L ? (part[e] + part[W + e]) + (part[2 * W + e] + part[3 * W + e]) : 0.f;
    if (tid < CK_DIM) out.end[piece * CK_DIM + tid] = ck_keys_to_end(sk + tid * CK_LDT, sa + tid * CK_LDT);
    else if (tid < 2 * CK_DIM) ck_queries_from_start(sq + (tid - CK_DIM) * CK_LDT, sa + (tid - CK_DIM) * CK_LDT);
    __syncthreads();
    for (int e = tid; e < CK_L * CK_DIM; e += CK_GLA_THREADS) qa[(e / CK_DIM) * CK_X + e % CK_DIM] = sq[(e % CK_DIM) * CK_LDT + e / CK_DIM];
    const int rg = tid >> 4, cg = tid & 15;
    for (int col0 = 0; col0 < vdim; col0 += CK_GLA_COLS) {
        ck_bring_v(part, v, ld, z == nullptr ? 1 : 0, r, h, vdim, col0, tid);
        __syncthreads();
        float acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;
        ck_product<4, 4, CK_L / 4, CK_LDT, CK_GLA_COLS>(acc, sk + rg * CK_LDT, part + 4 * cg);
        const int col = col0 + 4 * cg;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (col < vdim) ck_store<4>(out.states + (piece * CK_DIM + rg + 16 * i) * vdim + col, acc[i]);
        __syncthreads();
    }
}

// The state before every chunk in place of the chunk's contribution: a thread per four neighbouring values of one (sequence, head).
__global__ void __launch_bounds__(256, 4)
gla_chunk_pass_kernel(CkGla io, const int32_t* __restrict__ cu_new, const int32_t* __restrict__ slots, float* __restrict__ state, int n_slots, int H,
                      int dim, int vdim, int lo, int n_pieces) {
    dl_launch_dependents();
    dl_grid_dependency_wait();
    const int b = blockIdx.z, h = blockIdx.y, at = (blockIdx.x * 256 + threadIdx.x) * 4, c = at / vdim;
    CkRange r;
    if (at >= dim * vdim || !ck_sequence(r, cu_new, slots, n_slots, b)) return;
    const int first = ck_piece0(r.t0, b) - lo;             // the sequence's first piece, from the window's
    const int begin = max(0, -first), end = min((r.n + CK_L - 1) / CK_L, n_pieces - first);      // its chunks in the window
    if (begin >= end) return;
    float4* S = reinterpret_cast<float4*>(state + ((long)r.slot * H + h) * dim * vdim + at);
    float4 s = *S;
    const long piece0 = (long)first * H + h;
    constexpr int AHEAD = 8;                               // chunks whose contributions are asked for together
    for (int c0 = begin; c0 < end; c0 += AHEAD) {
        float4 x[AHEAD];
        float keep[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            const long piece = piece0 + (long)min(c0 + i, end - 1) * H;
            x[i] = *reinterpret_cast<const float4*>(io.states + piece * CK_DIM * vdim + at);
            keep[i] = io.end[piece * CK_DIM + c];
        }
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            if (c0 + i >= end) break;
            *reinterpret_cast<float4*>(io.states + (piece0 + (long)(c0 + i) * H) * CK_DIM * vdim + at) = s;
            s = make_float4(fmaf(keep[i], s.x, x[i].x), fmaf(keep[i], s.y, x[i].y), fmaf(keep[i], s.z, x[i].z), fmaf(keep[i], s.w, x[i].w));
        }
    }
    *S = s;
}

// A block per (piece, head): O = [Q+ | A] [S_0; V].
__global__ void __launch_bounds__(CK_GLA_THREADS)
gla_chunk_out_kernel(const __nv_bfloat16* __restrict__ v, long v_ld, int v_silu, CkGla in, const int32_t* __restrict__ cu_new, const int32_t* __restrict__ slots,
                     int n_slots, int n_seqs, float* __restrict__ out, long out_ld, int H, int dim, int vdim, int lo) {
    __shared__ __align__(16) float s_qa[CK_L * CK_LDX], s_x[CK_X * CK_GLA_COLS];
    dl_launch_dependents();
    dl_grid_dependency_wait();
    const int h = blockIdx.y, tid = threadIdx.x, rg = tid >> 4, cg = tid & 15;
    CkRange r;
    if (!ck_find(r, cu_new, slots, n_slots, n_seqs, lo + blockIdx.x, tid & 31)) return;
    const long piece = (long)blockIdx.x * H + h;
    for (int e = tid; e < CK_L * (CK_X / 4); e += CK_GLA_THREADS)
        ck_copy16(s_qa + (e / (CK_X / 4)) * CK_LDX + 4 * (e % (CK_X / 4)), in.qa + piece * (CK_L * CK_X) + 4 * e, true);
    for (int col0 = 0; col0 < vdim; col0 += CK_GLA_COLS) {
        for (int e = tid; e < CK_DIM * (CK_GLA_COLS / 4); e += CK_GLA_THREADS) {
            const int c = e / (CK_GLA_COLS / 4), col = col0 + (e % (CK_GLA_COLS / 4)) * 4;
            const bool live = c < dim && col < vdim;       // (channels beyond dim have no state: they were not passed)
            ck_copy16(s_x + 4 * e, in.states + (live ? (piece * CK_DIM + c) * vdim + col : 0), live);
        }
        ck_commit();
        ck_bring_v(s_x + CK_DIM * CK_GLA_COLS, v, v_ld, v_silu, r, h, vdim, col0, tid);
        ck_wait<0>();
        __syncthreads();
        float acc[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;
        ck_product<2, 4, CK_X / 4, CK_LDX, CK_GLA_COLS>(acc, s_qa + rg * CK_LDX, s_x + 4 * cg);
        const int col = col0 + 4 * cg;
#pragma unroll
        for (int i = 0; i < 2; ++i)
            if (rg + 16 * i < r.count && col < vdim) {
                float* dst = out + (long)(r.t0 + r.first + rg + 16 * i) * out_ld + (long)h * vdim + col;
                ck_store<4>(dst, acc[i]);
                if (!ck_all_finite(acc[i]))
                    ck_row_again<4, CK_GLA_COLS>(dst, s_qa + (rg + 16 * i) * CK_LDX, s_x + 4 * cg, CK_DIM + rg + 16 * i + 1, nullptr, 0);
            }
        __syncthreads();
    }
}

static cudaError_t ck_size(const void* kernel, std::atomic<unsigned long long>& sized, int smem) {
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

#define CK_CHECK(what)                                                                                                                \
    DL_REQUIRE(n_seqs >= 0 && H > 0 && H <= 65535 && n_seqs <= 65535 && dim > 0 && dim <= CK_DIM && vdim > 0 && vdim % 4 == 0 && n_slots > 0, \
               what ": sizes that the chunks do not take");                                                                           \
    DL_REQUIRE(at_once >= 1 && scratch != nullptr && ((uintptr_t)scratch % 16) == 0, what ": no scratch");                            \
    DL_REQUIRE(out_ld % 4 == 0 && ((uintptr_t)out % 16) == 0, what ": unaligned rows");

// Pieces that the chunks of so many tokens and sequences lie in, and floats of scratch for one of them: for the delta rule, and for gated
// linear attention with values of vdim channels.
extern "C" int dl_chunk_pieces(int n_tokens, int n_seqs) { return (int)(((long long)n_tokens + (CK_L - 1) * (long long)n_seqs) / CK_L); }
extern "C" int dl_delta_chunk_scratch(int H, long long* floats) {
    *floats = (long long)H * (CK_X * CK_X);
    return DL_OK;
}
extern "C" int dl_gla_chunk_scratch(int H, int vdim, long long* floats) {
    *floats = (long long)H * (CK_L * CK_X + CK_DIM + (long long)CK_DIM * vdim);
    return DL_OK;
}

// As dl_gla_scan for bfloat16 rows; v's rows 8-byte aligned, the state's and out's rows 16-byte aligned.  scratch: for `at_once` pieces; where
// there are more, a window of so many after the other (the states wait in `state` in between: the same bits).
extern "C" int dl_gla_chunk(const void* q, const void* k, const void* v, int ld, const float* z, int z_stride, const float* z_bias,
                            const int32_t* cu_new, const int32_t* slots, float* state, int n_slots, float* out, int out_ld, float* scratch,
                            int n_seqs, int n_tokens, int H, int dim, int vdim, float q_scale, float tau, int at_once, void* stream) {
    CK_CHECK("gla_chunk");
    DL_REQUIRE(tau > 0.f && out_ld >= H * vdim && (z == nullptr || z_stride >= H * dim), "gla_chunk: bad arguments");
    DL_REQUIRE(ld % 4 == 0 && ((uintptr_t)v % 8) == 0 && ((uintptr_t)state % 16) == 0, "gla_chunk: unaligned values or states");
    if (n_seqs == 0 || n_tokens == 0) return DL_OK;
    cudaStream_t s = (cudaStream_t)stream;
    const long long pieces = dl_chunk_pieces(n_tokens, n_seqs), in_scratch = (long long)at_once * H;
    CkGla sc;
    sc.qa = scratch;
    sc.end = sc.qa + in_scratch * CK_L * CK_X;
    sc.states = sc.end + in_scratch * CK_DIM;
    cudaError_t e = cudaSuccess;
    for (long long lo = 0; lo < pieces && e == cudaSuccess; lo += at_once) {
        const int n = (int)(pieces - lo < at_once ? pieces - lo : at_once);
        const dim3 grid(n, H);
        e = dl_launch_dependent(gla_chunk_states_kernel, grid, dim3(CK_GLA_THREADS), 0, s, (const __nv_bfloat16*)q, (const __nv_bfloat16*)k, (const __nv_bfloat16*)v, ld, z, z_stride,
                                z_bias, cu_new, slots, n_slots, n_seqs, sc, H, dim, vdim, q_scale, 1.0f / tau, (int)lo);
        if (e == cudaSuccess)
            e = dl_launch_dependent(gla_chunk_pass_kernel, dim3((dim * vdim / 4 + 255) / 256, H, n_seqs), dim3(256), 0, s, sc, cu_new, slots, state,
                                    n_slots, H, dim, vdim, (int)lo, n);
        if (e == cudaSuccess)
            e = dl_launch_dependent(gla_chunk_out_kernel, grid, dim3(CK_GLA_THREADS), 0, s, (const __nv_bfloat16*)v, ld, z == nullptr ? 1 : 0, sc, cu_new, slots,
                                    n_slots, n_seqs, out, out_ld, H, dim, vdim, (int)lo);
    }
    if (e != cudaSuccess) return dl_fail(DL_ERR_LAUNCH, "gla_chunk: %s", cudaGetErrorString(e));
    return DL_OK;
}

template <int CW>
static cudaError_t ck_walk(const float* v, const float* G, const int32_t* cu_new, const int32_t* slots, float* state, long slot_stride, int n_slots,
                           float* out, int n_seqs, int H, int dim, int vdim, int lo, int n_pieces, cudaStream_t s) {
    constexpr int smem = (CK_X * CK_LDX + 2 * CK_X * CW) * 4;
    static std::atomic<unsigned long long> sized{0};
    const cudaError_t e = ck_size((const void*)delta_chunk_walk_kernel<CW>, sized, smem);
    if (e != cudaSuccess) return e;
    // long-running blocks: they start when the kernel before has ended, spread over all multiprocessors
    return dl_launch_dependent_if(false, delta_chunk_walk_kernel<CW>, dim3((vdim + CW - 1) / CW, H, n_seqs), dim3(CK_THREADS), (size_t)smem, s, v, G, cu_new,
                                  slots, state, slot_stride, n_slots, out, H, dim, vdim, lo, n_pieces);
}

// The recurrence of dl_delta_rule from its prepared rows: q, k [tokens, G*dim], v [tokens, H*vdim], g [tokens, H*dim], beta [tokens, H], all float32.  scratch
// and at_once as in dl_gla_chunk.
int dl_delta_chunk(const float* q, const float* k, const float* v, const float* g, const float* beta, const int32_t* cu_new, const int32_t* slots,
                   float* state, long slot_stride, int n_slots, float* out, float* scratch, int n_seqs, int n_tokens, int H, int G, int dim, int vdim,
                   int at_once, cudaStream_t s) {
    const int out_ld = H * vdim;
    CK_CHECK("delta_chunk");
    DL_REQUIRE(((uintptr_t)v % 16) == 0 && n_tokens >= 0, "delta_chunk: unaligned values");
    static std::atomic<unsigned long long> sized{0};
    cudaError_t e = ck_size((const void*)delta_chunk_prepare_kernel, sized, CK_DELTA_SMEM);
    // 32 columns a block read G half as often as 16; 16 where 32 would leave multiprocessors without a block
    const bool wide = (long)((vdim + 31) / 32) * H * n_seqs >= dl_sm_count();
    const long long pieces = dl_chunk_pieces(n_tokens, n_seqs);
    for (long long lo = 0; lo < pieces && e == cudaSuccess; lo += at_once) {
        const int m = (int)(pieces - lo < at_once ? pieces - lo : at_once);
        e = dl_launch_dependent(delta_chunk_prepare_kernel, dim3(m, H), dim3(CK_THREADS), (size_t)CK_DELTA_SMEM, s, q, k, g, beta, cu_new, slots, n_slots,
                                n_seqs, scratch, H, H / G, dim, (int)lo);
        if (e == cudaSuccess)
            e = wide ? ck_walk<32>(v, scratch, cu_new, slots, state, slot_stride, n_slots, out, n_seqs, H, dim, vdim, (int)lo, m, s)
                     : ck_walk<16>(v, scratch, cu_new, slots, state, slot_stride, n_slots, out, n_seqs, H, dim, vdim, (int)lo, m, s);
    }
    if (e != cudaSuccess) return dl_fail(DL_ERR_LAUNCH, "delta_chunk: %s", cudaGetErrorString(e));
    return DL_OK;
}

DL_PACKED(dl_chunk_pieces)
DL_PACKED(dl_delta_chunk_scratch)
DL_PACKED(dl_gla_chunk_scratch)
DL_PACKED(dl_gla_chunk)
