// y = x W^T for float32 matrices on the fifth-generation tensor cores, with float32 accuracy.  (Splitting float32 values into three
// bfloat16 ones: Henry, Tang and Heinecke, "Leveraging the bfloat16 Artificial Intelligence Datatype For Higher-Precision Computations".)
//
// What bounds the product: on the FFMA pipes 74 TFLOP/s (the kernels of gemm_f32.cu reach 24), for a few rows the four
// bytes of every weight.  Here every operand value is split into three bfloat16 values, v = hi + mid + lo, each rounded to
// nearest, which together hold its 24 bits (mid is below 2^-8 v, lo below 2^-17 v), and six of the nine products of
// pieces are summed by bfloat16 MMAs with float32 accumulation:
//
//   x w = hi hi + (hi mid + mid hi) + (mid mid + hi lo + lo hi) + [mid lo + lo mid + lo lo: about 2^-26 x w, left out]
//
// Each product of two pieces is exact in float32.  The tensor core's sum is not rounded to nearest, so it is kept short, and
// pieces of one size are kept together: three accumulators take hi hi, the two products of 2^-9 and the three of 2^-18 of 256 k
// and are then added to a float32 register (rounded to nearest) by the epilogue.  Against float64 the result is closer than one
// chain of fused multiply-adds over k: at K 2,048 / 14,336 a relative error of 2.4e-7 / 2.4e-7 against 8.1e-7 / 2.1e-6.
//
// The order of every sum depends on N and K alone: runs of 256 k in ascending order within a segment (an eighth of K, whole
// blocks of 32), segments in ascending order.  Any number of rows, any tile of tokens and any cut of the segments between blocks
// gives the same bits; the 32-bit path relies on that (a prompt in one step, in portions or token by token).
//
// Values are multiplied by 2^24 as they are split and the sums by 2^-48 at the end, all of it exact: without it the last piece of a
// value below about 1e-33 would be smaller than any bfloat16, now even the smallest float32 keeps its bits.
//
// A result that is not finite - an infinity or a NaN went in, a piece (of a value above 2e31) or a sum (above 1e24) overflowed - is
// computed again as one chain of fused multiply-adds, so those outputs are the FFMA kernels'.  A block does that with all its
// threads, tile by tile through shared memory, once its pipeline has ended (of cut tiles, the blocks that sum them).
//
// Shape: 128 rows of W are the MMA's M and up to 128 tokens its N, so that a step of any number of rows runs the same
// arithmetic and W, four bytes a value, is read once per tile of tokens.  The three pieces of x lie behind one another in shared
// memory, so that one MMA meets a piece of W with up to three of them (N = 3 x tokens): an MMA has a cost of its own whatever
// its N, and with a few tokens that, not the tensor pipe, bounds the kernel (twelve MMAs per 32 k instead of six: 2.7 instead
// of 3.4 TB/s of W).
//   warp 0        one thread issues TMA copies: W [128][32] float32 (128-byte swizzle) into one ring; with more than 32 tokens the
//                 three planes of x, [tokens][32] bfloat16 (64-byte swizzle), that a kernel of its own made, into another; with
//                 fewer x [tokens][32] float32 beside W
//   warp 1        one thread issues the MMAs
//   groups of four warps, two or three of them, take turns at the blocks of 32 k: read W (and a few tokens' x), split it and write
//                 the three operand tiles (64-byte swizzle)
//   eight warps   the epilogue: each warp owns 32 outputs and half of the tokens, keeps a segment's sum in registers and the
//                 sum of the segments in tensor memory
//
// Measured (launched one after the other, FFMA kernel in brackets): 500 x 16,384 x 2,048 in 216 us, 156 TFLOP/s (1,036); 2,048 x
// 28,672 x 4,096 in 2.85 ms, 169 TFLOP/s (12.8); 8 rows x 28,672 x 4,096 in 122 us, 3.8 TB/s of W (528).  With 128 tokens the
// tensor pipe is half used.  Of the 216 us, 209 are left without the splitting of W, 204 without the drain of the accumulators (three tensor-memory ranges of 128
// columns leave no second set: the pipe waits for the epilogue once per run; runs of 128 k instead of 256: 5 % slower), 167 with a third of the MMAs: no one of them
// bounds it alone.  Shared memory, 160 KB per block of 32 k by count, is at 22 % under ncu; the operands' way from the L2, 40 KB per block and
// 9 TB/s over the GPU, is the likely bound.  With a few tokens it is the MMAs' own time, six per 16 KB of W, and the splitting.
#include "common.cuh"
#include "tma.cuh"
#include "tcgen05.cuh"
#include <atomic>

#define FT_BM 128                       // rows of W per tile
#define FT_BK 32                        // k per block: 128 bytes of float32, 64 of bfloat16
#define FT_SEGMENTS 8
#define FT_RUN 8                        // blocks of 32 k that an accumulator takes
#define FT_RAW_BYTES (FT_BM * FT_BK * 4)
#define FT_PLANE_BYTES (FT_BM * FT_BK * 2)
#define FT_SPLIT_BYTES (3 * FT_PLANE_BYTES)
#define FT_GROUP_WARPS 4                // warps that split one block of W; the groups take turns, each with an operand buffer of its own
#define FT_EPI_WARPS 8
#define FT_MAX_RING 12
#define FT_SELF_SPLIT 32                // steps of up to so many rows split x beside W: one launch less (x is read again by every block)

// Ring depths (what fits 224 KB; copies of W run no further ahead than those of x), accumulators, splitting groups.  X 0: x is
// split beside W.  RAW is a multiple of GROUPS: a stage's copies are all awaited by one group, which so sees every phase of the
// stage's barrier (a wait tells phases apart by parity alone, and copies may land out of order).
template <int NT> struct FtRings;
template <> struct FtRings<128> { enum { RAW = 4, X = 4, ACC = 1, GROUPS = 2 }; };
template <> struct FtRings<64> { enum { RAW = 6, X = 4, ACC = 2, GROUPS = 3 }; };
template <> struct FtRings<32> { enum { RAW = 6, X = 0, ACC = 2, GROUPS = 3 }; };
template <> struct FtRings<16> { enum { RAW = 6, X = 0, ACC = 2, GROUPS = 3 }; };
template <int NT> struct FtShape : FtRings<NT> {
    using R = FtRings<NT>;
    enum {
        X_PLANE = NT * FT_BK * 2,
        RAW_STAGE = FT_RAW_BYTES + (R::X ? 0 : NT * FT_BK * 4),
        SPLIT_STAGE = FT_SPLIT_BYTES + (R::X ? 0 : 3 * X_PLANE),
        SMEM = 1024 + R::RAW * RAW_STAGE + R::GROUPS * SPLIT_STAGE + R::X * 3 * X_PLANE,
        THREADS = 32 * (2 + R::GROUPS * FT_GROUP_WARPS + FT_EPI_WARPS)
    };
};

struct FtWork {
    const float* x;
    const float* w;
    float* y;
    float* sums;                        // [segment][M][N], used when parts > 1
    int x_stride, y_stride;
    int M, N, K;
    int row_tiles, token_tiles;
    int blocks, seg_blocks, segments;   // blocks of 32 k in all and per segment
    int parts;                          // runs of segments that a tile is cut into
    int units;                          // row_tiles * token_tiles * parts
};

__device__ __forceinline__ bool ft_finite(float v) { return fabsf(v) <= 3.402823466e38f; }

#define FT_SCALE 16777216.f              // 2^24: of every value that is split
#define FT_UNSCALE 3.5527136788005009e-15f   // 2^-48: of a sum of products of two such values

// Two values (times FT_SCALE) into their three pieces, packed as bfloat16 pairs (first value in the low half).
__device__ __forceinline__ void ft_split2(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    asm("{\n\t.reg .b64 v, s;\n\tmov.b64 v, {%0, %1};\n\tmov.b64 s, {%2, %2};\n\tmul.rn.f32x2 v, v, s;\n\tmov.b64 {%0, %1}, v;\n\t}" : "+f"(a), "+f"(b) : "f"(FT_SCALE));
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    a -= __uint_as_float(hi << 16);
    b -= __uint_as_float(hi & 0xffff0000u);
    const __nv_bfloat162 m = __floats2bfloat162_rn(a, b);
    mid = *reinterpret_cast<const uint32_t*>(&m);
    a -= __uint_as_float(mid << 16);
    b -= __uint_as_float(mid & 0xffff0000u);
    const __nv_bfloat162 l = __floats2bfloat162_rn(a, b);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

// x [M, K] into three planes [3][M][Kp] (Kp: K rounded up to a multiple of 8, zeros behind K): a thread per 8 values.  VEC:
// rows are 16-byte aligned and K is a multiple of 8.
template <bool VEC>
__global__ void __launch_bounds__(256)
ft_split_kernel(const float* __restrict__ x, int x_stride, __nv_bfloat16* __restrict__ planes, int M, int K, int Kp) {
    dl_launch_dependents();
    dl_grid_dependency_wait();
    const int per_row = Kp / 8;
    const long idx = (long)blockIdx.x * 256 + threadIdx.x;
    if (idx >= (long)M * per_row) return;
    const int m = (int)(idx / per_row), k = (int)(idx % per_row) * 8;
    const float* src = x + (size_t)m * x_stride + k;
    float v[8];
    if (VEC) {
        const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = k + i < K ? src[i] : 0.f;
    }
    uint32_t p[3][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) ft_split2(v[2 * i], v[2 * i + 1], p[0][i], p[1][i], p[2][i]);
#pragma unroll
    for (int s = 0; s < 3; ++s)
        *reinterpret_cast<uint4*>(planes + ((size_t)s * M + m) * Kp + k) = make_uint4(p[s][0], p[s][1], p[s][2], p[s][3]);
}

// Rows of `src` (at most `rows` of them, `ld` apart), values k0 .. k0 + 4 `vecs` - 1, into shared memory `pitch` floats apart.
__device__ __forceinline__ void ft_stage(float* dst, int pitch, const float* src, size_t ld, bool aligned, int rows, int live, int k0, int vecs, int tid,
                                         int threads) {
    for (int e = tid; e < rows * vecs; e += threads) {
        const int r = e / vecs, c = 4 * (e - r * vecs);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < live) {
            const float* p = src + r * ld + k0 + c;
            v = aligned ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
        }
        *reinterpret_cast<float4*>(dst + r * pitch + c) = v;
    }
}
__device__ __forceinline__ float ft_chain4(float acc, const float4& a, const float4& b) {
    return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, acc))));
}

// The outputs of a unit's tile (128 rows of W from row0, NT tokens from token0) that are not finite, as chains over k in ascending order.
// All threads of the block; `smem`: 128 rows of 36 floats.
template <int NT>
__device__ __noinline__ void ft_tile_again(const FtWork& wk, float* smem, int row0, int token0, int tid, int threads) {
    constexpr int TM = NT < 64 ? NT : 64, TN = 64, PER = TM / 16, PITCH = FT_BK + 4;       // a thread: 4 x PER outputs
    float* ws = smem;
    float* xs = ws + TN * PITCH;
    const int tx = tid & 15, ty = tid >> 4;                // (256 of the threads multiply, all of them stage)
    const bool aligned = wk.x_stride % 4 == 0 && ((uintptr_t)wk.x % 16) == 0;
#pragma unroll 1
    for (int part = 0; part < (FT_BM / TN) * (NT / TM); ++part) {
        const int n0 = row0 + (part % (FT_BM / TN)) * TN, m0 = token0 + (part / (FT_BM / TN)) * TM;
        auto place = [&](int i, int j, float*& y) {        // the thread's output (i, j), if there is one
            const int n = n0 + tx + 16 * i, m = m0 + ty + 16 * j;
            y = wk.y + (size_t)m * wk.y_stride + n;
            return tid < 256 && n < wk.N && m < wk.M;
        };
        bool fine = true;
        float* y;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < PER; ++j)
                if (place(i, j, y)) fine = fine && ft_finite(*y);
        if (!__syncthreads_or(!fine)) continue;
        float acc[4][PER];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < PER; ++j) acc[i][j] = 0.f;
        for (int k0 = 0; k0 < wk.K; k0 += FT_BK) {         // K is a multiple of 4
            const int vecs = min(FT_BK, wk.K - k0) / 4;
            ft_stage(ws, PITCH, wk.w + (size_t)n0 * wk.K, wk.K, true, TN, wk.N - n0, k0, vecs, tid, threads);
            ft_stage(xs, PITCH, wk.x + (size_t)m0 * wk.x_stride, wk.x_stride, aligned, TM, wk.M - m0, k0, vecs, tid, threads);
            __syncthreads();
            if (tid < 256) {
                for (int c = 0; c < vecs; ++c) {
                    float4 xv[PER];
#pragma unroll
                    for (int j = 0; j < PER; ++j) xv[j] = *reinterpret_cast<const float4*>(xs + (ty + 16 * j) * PITCH + 4 * c);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float4 wv = *reinterpret_cast<const float4*>(ws + (tx + 16 * i) * PITCH + 4 * c);
#pragma unroll
                        for (int j = 0; j < PER; ++j) acc[i][j] = ft_chain4(acc[i][j], xv[j], wv);
                    }
                }
            }
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < PER; ++j)
                if (place(i, j, y) && !ft_finite(*y)) *y = acc[i][j];
    }
}

// One output as a chain over k in ascending order, four values at a time (K is a multiple of 4).  No shared memory: the kernel that calls it
// starts beside the product's blocks, which leave none.
__device__ __noinline__ float ft_chain(const FtWork& wk, int m, int n) {
    const float* a = wk.x + (size_t)m * wk.x_stride;
    const float* b = wk.w + (size_t)n * wk.K;
    float acc = 0.f;
    if (((uintptr_t)a % 16) == 0) {
#pragma unroll 8
        for (int k = 0; k < wk.K; k += 4) acc = ft_chain4(acc, __ldg(reinterpret_cast<const float4*>(a + k)), __ldg(reinterpret_cast<const float4*>(b + k)));
    } else {
        for (int k = 0; k < wk.K; k += 4) acc = ft_chain4(acc, make_float4(a[k], a[k + 1], a[k + 2], a[k + 3]), __ldg(reinterpret_cast<const float4*>(b + k)));
    }
    return acc;
}

// y = the segments' sums in ascending order (the order in which an uncut tile adds them).  A block: 256 / tm outputs of each of tm = 2^log_tm tokens
// (chains of neighbours share the rows they read).
#define FT_REDUCE_THREADS 256
__global__ void __launch_bounds__(FT_REDUCE_THREADS) ft_reduce_kernel(const FtWork wk, int log_tm) {
    dl_launch_dependents();
    dl_grid_dependency_wait();
    const int tid = threadIdx.x, log_tn = 8 - log_tm;      // 256 threads
    const int n = (blockIdx.x << log_tn) + (tid & ((1 << log_tn) - 1));
    for (long m = ((long)blockIdx.y << log_tm) + (tid >> log_tn); m < wk.M && n < wk.N; m += (long)gridDim.y << log_tm) {
        const size_t step = (size_t)wk.M * wk.N, at = (size_t)m * wk.N + n;
        float v[FT_SEGMENTS];
#pragma unroll
        for (int j = 0; j < FT_SEGMENTS; ++j) v[j] = j < wk.segments ? __ldcg(wk.sums + j * step + at) : 0.f;
        float total = v[0];
#pragma unroll
        for (int j = 1; j < FT_SEGMENTS; ++j)
            if (j < wk.segments) total += v[j];
        wk.y[(size_t)m * wk.y_stride + n] = ft_finite(total) ? total * FT_UNSCALE : ft_chain(wk, (int)m, n);
    }
}

// 8 values of a row: read from two 16-byte pieces of a raw tile (128-byte swizzle), written as one 16-byte piece of each operand tile.
__device__ __forceinline__ void ft_load8(const unsigned char* src, int row, int c, float4 (&v)[2]) {
    v[0] = *reinterpret_cast<const float4*>(src + row * 128 + (((2 * c) ^ (row & 7)) << 4));
    v[1] = *reinterpret_cast<const float4*>(src + row * 128 + (((2 * c + 1) ^ (row & 7)) << 4));
}
__device__ __forceinline__ void ft_store8(unsigned char* dst, int plane_bytes, int row, int c, const float4 (&v)[2]) {
    uint4 p[3];
    ft_split2(v[0].x, v[0].y, p[0].x, p[1].x, p[2].x);
    ft_split2(v[0].z, v[0].w, p[0].y, p[1].y, p[2].y);
    ft_split2(v[1].x, v[1].y, p[0].z, p[1].z, p[2].z);
    ft_split2(v[1].z, v[1].w, p[0].w, p[1].w, p[2].w);
    unsigned char* at = dst + row * 64 + ((c ^ ((row >> 1) & 3)) << 4);
#pragma unroll
    for (int s = 0; s < 3; ++s) *reinterpret_cast<uint4*>(at + s * plane_bytes) = p[s];
}
// 8 columns of the three accumulators as one float32 each: the large one plus the sum of the small ones.
template <int NT>
__device__ __forceinline__ void ft_acc8(uint32_t at, float (&v)[8]) {
    uint32_t r[3][8];
#pragma unroll
    for (int s = 0; s < 3; ++s)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(r[s][0]), "=r"(r[s][1]), "=r"(r[s][2]), "=r"(r[s][3]), "=r"(r[s][4]), "=r"(r[s][5]), "=r"(r[s][6]), "=r"(r[s][7])
                     : "r"(at + s * NT)
                     : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[0][i]) + (__uint_as_float(r[1][i]) + __uint_as_float(r[2][i]));
}

template <int NT>
__global__ void __launch_bounds__(FtShape<NT>::THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const FtWork wk,
                   int early_weights, int* __restrict__ status) {
    constexpr int RAW = FtShape<NT>::RAW, ACC = FtShape<NT>::ACC, GROUPS = FtShape<NT>::GROUPS;
    constexpr bool PLANES = FtShape<NT>::X > 0;               // x comes split
    constexpr int XR = PLANES ? (int)FtShape<NT>::X : 1;
    constexpr int EPI_WARP0 = 2 + GROUPS * FT_GROUP_WARPS;    // any four warps in a row cover the four quarters of tensor memory
    constexpr int X_PLANE = FtShape<NT>::X_PLANE, RAW_STAGE = FtShape<NT>::RAW_STAGE, SPLIT_STAGE = FtShape<NT>::SPLIT_STAGE;
    constexpr int COLS = NT / 2;                              // tokens an epilogue warp owns
    constexpr uint32_t ACC_COLS = 3 * NT;
    constexpr uint32_t TOTAL_AT = ACC * ACC_COLS;             // the sums of the segments so far
    constexpr uint32_t NEED = TOTAL_AT + NT, TMEM_COLS = NEED <= 128 ? 128 : NEED <= 256 ? 256 : 512;
    static_assert(NEED <= 512, "tensor memory");
    static_assert(RAW % GROUPS == 0, "a stage of the copies' ring belongs to one splitting group");
    extern __shared__ unsigned char ft_smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)ft_smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* raw = base;
    unsigned char* split = raw + RAW * RAW_STAGE;
    unsigned char* xs = split + GROUPS * SPLIT_STAGE;
    __shared__ uint64_t raw_full[FT_MAX_RING], raw_empty[FT_MAX_RING], x_full[FT_MAX_RING], x_empty[FT_MAX_RING];
    __shared__ uint64_t split_full[3], split_empty[3], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_holder;
    __shared__ volatile int gave_up, odd;                     // odd: an output is not finite
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        gave_up = 0, odd = 0;
        for (int s = 0; s < RAW; ++s) tc_mbar_init(&raw_full[s], 1), tc_mbar_init(&raw_empty[s], FT_GROUP_WARPS);
        for (int s = 0; s < XR; ++s) tc_mbar_init(&x_full[s], 1), tc_mbar_init(&x_empty[s], 1);
        for (int s = 0; s < GROUPS; ++s) tc_mbar_init(&split_full[s], FT_GROUP_WARPS), tc_mbar_init(&split_empty[s], 1);
        for (int s = 0; s < ACC; ++s) tc_mbar_init(&acc_full[s], 1), tc_mbar_init(&acc_empty[s], FT_EPI_WARPS);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tc_tmem_alloc(&tmem_holder, TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    dl_launch_dependents();
    const uint32_t tmem = tmem_holder;

    // A unit: (tile of rows of W, part of the segments, tile of tokens), tokens fastest: the blocks that read one tile of W run side by side.
    auto unit_of = [&](int u, int& row0, int& token0, int& seg0, int& seg1, int& b0, int& b1) {
        const int tt = u % wk.token_tiles, rest = u / wk.token_tiles;
        const int part = rest % wk.parts;
        row0 = (rest / wk.parts) * FT_BM;
        token0 = tt * NT;
        seg0 = part * wk.segments / wk.parts, seg1 = (part + 1) * wk.segments / wk.parts;
        b0 = seg0 * wk.seg_blocks, b1 = min(wk.blocks, seg1 * wk.seg_blocks);
    };

    if (warp == 0) {
        // ------------------------------------------------------------ copies
        if (lane == 0) {
            const uint64_t policy = dl_stream_policy();
            const bool reread = wk.token_tiles > 1;           // W is read by several blocks: keep it in the L2
            int it = 0;                                       // blocks of k
            int w_issued = 0, x_issued = 0;
            bool stop = false;
            auto load_w = [&](int row0, int b, int i) {
                const int s = i % RAW;
                tc_mbar_expect(&raw_full[s], RAW_STAGE);
                if (reread) dl_tma_load_2d(raw + s * RAW_STAGE, &tmap_w, b * FT_BK, row0, &raw_full[s]);
                else dl_tma_load_2d_hint(raw + s * RAW_STAGE, &tmap_w, b * FT_BK, row0, &raw_full[s], policy);
                ++w_issued;
            };
            // while the kernel before this one finishes, the ring fills with weights
            int ahead = 0;
            if (early_weights && (int)blockIdx.x < wk.units) {
                int row0, token0, s0, s1, b0, b1;
                unit_of(blockIdx.x, row0, token0, s0, s1, b0, b1);
                for (; ahead < RAW && b0 + ahead < b1; ++ahead) load_w(row0, b0 + ahead, ahead);
            }
            dl_grid_dependency_wait();
            for (int u = blockIdx.x; u < wk.units && !stop; u += gridDim.x) {
                int row0, token0, s0, s1, b0, b1;
                unit_of(u, row0, token0, s0, s1, b0, b1);
                for (int b = b0; b < b1; ++b, ++it) {
                    const int sx = it % XR, sr = it % RAW;
                    if (it >= ahead) {
                        if (it >= RAW && !tc_mbar_wait(&raw_empty[sr], ((it / RAW) - 1) & 1, &gave_up)) { stop = true; break; }
                        load_w(row0, b, it);
                    }
                    if (PLANES) {
                        if (it >= XR && !tc_mbar_wait(&x_empty[sx], ((it / XR) - 1) & 1, &gave_up)) { stop = true; break; }
                        tc_mbar_expect(&x_full[sx], 3 * X_PLANE);
                        for (int p = 0; p < 3; ++p)
                            dl_tma_load_2d(xs + (sx * 3 + p) * X_PLANE, &tmap_x, b * FT_BK, p * wk.M + token0, &x_full[sx]);
                    } else {
                        dl_tma_load_2d(raw + sr * RAW_STAGE + FT_RAW_BYTES, &tmap_x, b * FT_BK, token0, &raw_full[sr]);
                    }
                    ++x_issued;
                }
            }
            if (stop) {
                if (!gave_up) atomicExch(status, 61);
                gave_up = 1;
                // copies already issued must land before the block's shared memory is released
                for (int i = max(0, w_issued - RAW); i < (PLANES ? w_issued : min(w_issued, x_issued)); ++i) {
                    const long long t0 = clock64();
                    while (!tc_mbar_try(&raw_full[i % RAW], (i / RAW) & 1) && clock64() - t0 < TC_WAIT_CYCLES / 16) {}
                }
                for (int i = max(0, x_issued - XR); PLANES && i < x_issued; ++i) {
                    const long long t0 = clock64();
                    while (!tc_mbar_try(&x_full[i % XR], (i / XR) & 1) && clock64() - t0 < TC_WAIT_CYCLES / 16) {}
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ tensor-core issue
        if (lane == 0) {
            constexpr uint32_t ID1 = tc_idesc_bf16(FT_BM, NT), ID2 = tc_idesc_bf16(FT_BM, 2 * NT), ID3 = tc_idesc_bf16(FT_BM, NT <= 64 ? 3 * NT : NT);
            int it = 0, run = 0;
            bool ok = true;
            for (int u = blockIdx.x; u < wk.units && ok; u += gridDim.x) {
                int row0, token0, s0, s1, b0, b1;
                unit_of(u, row0, token0, s0, s1, b0, b1);
                int in_seg = 0;                               // blocks of the segment so far
                for (int b = b0; b < b1; ++b, ++it) {
                    const int ss = it % GROUPS, sx = it % XR, sa = run % ACC;
                    const bool first = in_seg % FT_RUN == 0;
                    ok = (!first || run < ACC || tc_mbar_wait(&acc_empty[sa], ((run / ACC) - 1) & 1, &gave_up)) &&
                         (!PLANES || tc_mbar_wait(&x_full[sx], (it / XR) & 1, &gave_up)) &&
                         tc_mbar_wait(&split_full[ss], (it / GROUPS) & 1, &gave_up);
                    if (!ok) {
                        if (!gave_up) atomicExch(status, 62);
                        gave_up = 1;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a_addr = tc_smem(split + ss * SPLIT_STAGE);
                    const uint32_t b_addr = PLANES ? tc_smem(xs + sx * 3 * X_PLANE) : a_addr + FT_SPLIT_BYTES;
                    const uint64_t hi = tc_operand_desc_64(a_addr), mid = tc_operand_desc_64(a_addr + FT_PLANE_BYTES);
                    const uint64_t lo = tc_operand_desc_64(a_addr + 2 * FT_PLANE_BYTES), xd = tc_operand_desc_64(b_addr);
                    const uint32_t d = tmem + sa * ACC_COLS;
#pragma unroll
                    for (int k = 0; k < 2; ++k) {             // 16 k = 32 bytes further along the swizzled rows
                        const uint64_t at = 2 * k;
                        const uint32_t acc = (first && k == 0) ? 0u : 1u;
                        if (NT <= 64) {
                            tc_mma(d, hi + at, xd + at, ID3, acc);
                        } else {
                            tc_mma(d, hi + at, xd + at, ID2, acc);
                            tc_mma(d + 2 * NT, hi + at, tc_operand_desc_64(b_addr + 2 * X_PLANE) + at, ID1, acc);
                        }
                        tc_mma(d + NT, mid + at, xd + at, ID2, 1u);
                        tc_mma(d + 2 * NT, lo + at, xd + at, ID1, 1u);
                    }
                    tc_commit(&split_empty[ss]);
                    if (PLANES) tc_commit(&x_empty[sx]);
                    ++in_seg;
                    const bool seg_ends = in_seg == wk.seg_blocks || b + 1 == b1;
                    if (seg_ends || in_seg % FT_RUN == 0) {
                        tc_commit(&acc_full[sa]);
                        ++run;
                    }
                    if (seg_ends) in_seg = 0;
                }
            }
        }
    } else if (warp < EPI_WARP0) {
        // ------------------------------------------------------------ W (and a few tokens' x) into pieces
        const int cw = (warp - 2) % FT_GROUP_WARPS, group = (warp - 2) / FT_GROUP_WARPS;
        int it = 0;
        bool ok = true;
        for (int u = blockIdx.x; u < wk.units && ok; u += gridDim.x) {
            int row0, token0, s0, s1, b0, b1;
            unit_of(u, row0, token0, s0, s1, b0, b1);
            for (int b = b0; b < b1; ++b, ++it) {
                const int sr = it % RAW, ss = it % GROUPS;
                if (ss != group) continue;
                ok = tc_mbar_wait(&raw_full[sr], (it / RAW) & 1, &gave_up) &&
                     (it < GROUPS || tc_mbar_wait(&split_empty[ss], ((it / GROUPS) - 1) & 1, &gave_up));
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) {
                    if (lane == 0 && !gave_up) atomicExch(status, 63);
                    gave_up = 1;
                    break;
                }
                const unsigned char* src = raw + sr * RAW_STAGE;
                unsigned char* dst = split + ss * SPLIT_STAGE;
                const int row = cw * 32 + (lane >> 2), c = lane & 3;      // a lane takes 8 values of each of four rows
                float4 v[4][2], xv[2];
                constexpr int X_PIECES = NT * 4;                          // of 8 values of x
                const int xp = cw * 32 + lane;
#pragma unroll
                for (int i = 0; i < 4; ++i) ft_load8(src, row + 8 * i, c, v[i]);
                if (!PLANES && xp < X_PIECES) ft_load8(src + FT_RAW_BYTES, xp >> 2, xp & 3, xv);
#pragma unroll
                for (int i = 0; i < 4; ++i) ft_store8(dst, FT_PLANE_BYTES, row + 8 * i, c, v[i]);
                if (!PLANES && xp < X_PIECES) ft_store8(dst + FT_SPLIT_BYTES, X_PLANE, xp >> 2, xp & 3, xv);
                tc_fence_async_smem();                        // the operand tiles, before the tensor core reads them
                __threadfence_block();                        // the raw tile has been read before the copy engine refills it
                __syncwarp();
                if (lane == 0) {
                    tc_mbar_arrive(&raw_empty[sr]);
                    tc_mbar_arrive(&split_full[ss]);
                }
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue
        dl_grid_dependency_wait();                            // y and the sums may still be in use by the kernel before this one
        const int quarter = warp & 3, half = (warp - EPI_WARP0) >> 2;
        const uint32_t lane_at = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * COLS);
        int run = 0;
        bool ok = true;
        for (int u = blockIdx.x; u < wk.units && ok; u += gridDim.x) {
            int row0, token0, s0, s1, b0, b1;
            unit_of(u, row0, token0, s0, s1, b0, b1);
            const int n = row0 + quarter * 32 + lane, m0 = token0 + half * COLS;
            for (int seg = s0; seg < s1 && ok; ++seg) {
                const int seg_end = min(b1, (seg + 1) * wk.seg_blocks);
                float sum[COLS];
#pragma unroll
                for (int i = 0; i < COLS; ++i) sum[i] = 0.f;
                for (int b = seg * wk.seg_blocks; b < seg_end; b += FT_RUN, ++run) {
                    const int sa = run % ACC;
                    ok = __all_sync(0xffffffffu, tc_mbar_wait(&acc_full[sa], (run / ACC) & 1, &gave_up));
                    if (!ok) {
                        if (lane == 0 && !gave_up) atomicExch(status, 64);
                        gave_up = 1;
                        break;
                    }
                    tc_fence_after();
#pragma unroll
                    for (int c = 0; c < COLS; c += 8) {
                        float v[8];
                        ft_acc8<NT>(lane_at + sa * ACC_COLS + c, v);
#pragma unroll
                        for (int i = 0; i < 8; ++i) sum[c + i] += v[i];
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) tc_mbar_arrive(&acc_empty[sa]);
                }
                if (!ok) break;
                if (wk.parts > 1) {
                    float* dst = wk.sums + ((size_t)seg * wk.M + m0) * wk.N + n;
#pragma unroll
                    for (int i = 0; i < COLS; ++i)
                        if (n < wk.N && m0 + i < wk.M) dst[(size_t)i * wk.N] = sum[i];
                    continue;
                }
                // the sum of the segments: in tensor memory between two of them
                if (seg > s0) {
#pragma unroll
                    for (int c = 0; c < COLS; c += 8) {
                        float v[8];
                        tc_tmem_load8(lane_at + TOTAL_AT + c, v);
#pragma unroll
                        for (int i = 0; i < 8; ++i) sum[c + i] = v[i] + sum[c + i];
                    }
                }
                if (seg + 1 < s1) {
#pragma unroll
                    for (int c = 0; c < COLS; c += 8) {
                        const float v[8] = {sum[c], sum[c + 1], sum[c + 2], sum[c + 3], sum[c + 4], sum[c + 5], sum[c + 6], sum[c + 7]};
                        tc_tmem_store8(lane_at + TOTAL_AT + c, v);
                    }
                    tc_tmem_store_wait();
                } else {
                    float* dst = wk.y + (size_t)m0 * wk.y_stride + n;
                    bool fine = true;
#pragma unroll
                    for (int i = 0; i < COLS; ++i) {
                        fine = fine && ft_finite(sum[i]);
                        if (n < wk.N && m0 + i < wk.M) dst[(size_t)i * wk.y_stride] = sum[i] * FT_UNSCALE;
                    }
                    if (!fine) odd = 1;                       // (or a column beyond M, which may hold anything: then nothing is found)
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tc_tmem_free(tmem, TMEM_COLS);
    if (odd && !gave_up) {
        static_assert(RAW * RAW_STAGE >= 128 * (FT_BK + 4) * 4, "ft_tile_again's rows lie where the copies' ring was");
#pragma unroll 1
        for (int u = blockIdx.x; u < wk.units; u += gridDim.x) {
            int row0, token0, s0, s1, b0, b1;
            unit_of(u, row0, token0, s0, s1, b0, b1);
            ft_tile_again<NT>(wk, reinterpret_cast<float*>(base), row0, token0, threadIdx.x, FtShape<NT>::THREADS);
        }
    }
}

static int ft_tokens(int M) { return M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128; }

static void ft_plan(int M, int N, int K, int sms, FtWork* wk) {
    wk->M = M, wk->N = N, wk->K = K;
    const int nt = ft_tokens(M);
    wk->row_tiles = (N + FT_BM - 1) / FT_BM;
    wk->token_tiles = (M + nt - 1) / nt;
    wk->blocks = (K + FT_BK - 1) / FT_BK;
    wk->seg_blocks = (wk->blocks + FT_SEGMENTS - 1) / FT_SEGMENTS;
    wk->segments = (wk->blocks + wk->seg_blocks - 1) / wk->seg_blocks;
    // The cut of a tile's segments between blocks: what the slowest multiprocessor works through (measured: a block of 32 k takes
    // 0.65 us with up to 32 tokens, 0.75 with 64, 0.95 with 128), and for cut tiles a second launch and the sums' trip through memory.
    const double tb = nt == 128 ? 0.95 : nt == 64 ? 0.75 : 0.65;
    double best = 0.0;
    wk->parts = 1;
    for (int p = 1; p <= wk->segments; ++p) {
        const long units = (long)wk->row_tiles * wk->token_tiles * p;
        const long waves = (units + sms - 1) / sms;
        double cost = (double)waves * ((wk->segments + p - 1) / p) * wk->seg_blocks * tb;
        if (p > 1) cost += 2.0 + 8.0 * wk->segments * (double)M * N / 5.0e6;
        if (p == 1 || cost < best) best = cost, wk->parts = p;
    }
    wk->units = wk->row_tiles * wk->token_tiles * wk->parts;
}

// Scratch the product of these sizes needs: `planes` bfloat16 values and `sums` floats.
extern "C" int dl_gemm_f32_tc_scratch(int M, int N, int K, int sms, long long* planes, long long* sums) {
    FtWork wk;
    ft_plan(M, N, K, sms, &wk);
    *planes = M > FT_SELF_SPLIT ? 3ll * M * ((K + 7) / 8 * 8) : 0;
    *sums = wk.parts > 1 ? (long long)wk.segments * M * N : 0;
    return DL_OK;
}

template <int NT>
static cudaError_t ft_launch(const CUtensorMap& mw, const CUtensorMap& mx, const FtWork& wk, int early, int grid, int* status, cudaStream_t s) {
    static std::atomic<unsigned long long> sized{0};          // devices (by number, up to 64) whose kernel has its shared memory
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 64 || !(sized.load() >> dev & 1)) {
        e = cudaFuncSetAttribute(gemm_f32_tc_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, FtShape<NT>::SMEM);
        if (e != cudaSuccess) return e;
        if (dev < 64) sized.fetch_or(1ull << dev);
    }
    return dl_launch_dependent(gemm_f32_tc_kernel<NT>, dim3(grid), dim3(FtShape<NT>::THREADS), (size_t)FtShape<NT>::SMEM, s, mw, mx, wk, early, status);
}

// x: [M, K] rows x_stride apart (up to FT_SELF_SPLIT rows: 16-byte aligned); w: contiguous [N, K], 16-byte aligned, K a multiple of 4;
// y: [M, N] rows y_stride apart; planes and sums: scratch of at least what dl_gemm_f32_tc_scratch says for the device's
// multiprocessors.  `resident`: nothing still pending on the stream writes w.
extern "C" int dl_gemm_f32_tc(const float* x, int x_stride, const float* w, float* y, int y_stride, int M, int N, int K, void* planes,
                              long long planes_len, float* sums, long long sums_len, int resident, int* status, void* stream) {
    DL_REQUIRE(M >= 0 && N > 0 && K > 0 && x_stride >= K && y_stride >= N, "gemm_f32_tc: bad sizes M=%d N=%d K=%d", M, N, K);
    DL_REQUIRE(K % 4 == 0 && ((uintptr_t)w % 16) == 0 && ((uintptr_t)planes % 16) == 0, "gemm_f32_tc: unaligned operands");
    DL_REQUIRE(M > FT_SELF_SPLIT || (x_stride % 4 == 0 && ((uintptr_t)x % 16) == 0), "gemm_f32_tc: a few rows of x must be 16-byte aligned");
    if (M == 0) return DL_OK;
    const int sms = dl_sm_count() > 0 ? dl_sm_count() : 148;
    FtWork wk;
    ft_plan(M, N, K, sms, &wk);
    wk.x = x, wk.w = w, wk.y = y, wk.sums = sums, wk.x_stride = x_stride, wk.y_stride = y_stride;
    const int Kp = (K + 7) / 8 * 8;
    DL_REQUIRE(M <= FT_SELF_SPLIT || planes_len >= 3ll * M * Kp, "gemm_f32_tc: %lld values of planes, %lld needed", planes_len, 3ll * M * Kp);
    DL_REQUIRE(wk.parts == 1 || sums_len >= (long long)wk.segments * M * N, "gemm_f32_tc: %lld sums, %lld needed", sums_len,
               (long long)wk.segments * M * N);
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e;
    const int nt = ft_tokens(M);
    CUtensorMap mw, mx;
    if (dl_tmap_cached_2d_f32(&mw, w, N, K, (unsigned long long)K * 4, FT_BM, FT_BK, DL_TMAP_SWIZZLE_128B) != 0) return DL_ERR_LAUNCH;
    if (M > FT_SELF_SPLIT) {
        const long items = (long)M * (Kp / 8);
        const bool vec = K % 8 == 0 && x_stride % 4 == 0 && ((uintptr_t)x % 16) == 0;
        e = dl_launch_dependent(vec ? ft_split_kernel<true> : ft_split_kernel<false>, dim3((unsigned)((items + 255) / 256)), dim3(256), 0, s, x, x_stride,
                                (__nv_bfloat16*)planes, M, K, Kp);
        if (e != cudaSuccess) return dl_fail(DL_ERR_LAUNCH, "gemm_f32_tc: %s", cudaGetErrorString(e));
        if (dl_tmap_cached_2d_bf16(&mx, planes, 3ull * M, Kp, (unsigned long long)Kp * 2, nt, FT_BK, DL_TMAP_SWIZZLE_64B) != 0) return DL_ERR_LAUNCH;
    } else if (dl_tmap_cached_2d_f32(&mx, x, M, K, (unsigned long long)x_stride * 4, nt, FT_BK, DL_TMAP_SWIZZLE_128B) != 0) {
        return DL_ERR_LAUNCH;
    }
    const int grid = wk.units < sms ? wk.units : sms;
    if (nt == 16) e = ft_launch<16>(mw, mx, wk, resident, grid, status, s);
    else if (nt == 32) e = ft_launch<32>(mw, mx, wk, resident, grid, status, s);
    else if (nt == 64) e = ft_launch<64>(mw, mx, wk, resident, grid, status, s);
    else e = ft_launch<128>(mw, mx, wk, resident, grid, status, s);
    if (e != cudaSuccess) return dl_fail(DL_ERR_LAUNCH, "gemm_f32_tc: %s", cudaGetErrorString(e));
    if (wk.parts > 1) {
        const int log_tm = M >= 16 ? 4 : M >= 8 ? 3 : M >= 4 ? 2 : M >= 2 ? 1 : 0, tm = 1 << log_tm, tn = FT_REDUCE_THREADS / tm;
        const int rows = (M + tm - 1) / tm;
        e = dl_launch_dependent(ft_reduce_kernel, dim3((N + tn - 1) / tn, rows < 65535 ? rows : 65535), dim3(FT_REDUCE_THREADS), 0, s, wk, log_tm);
        if (e != cudaSuccess) return dl_fail(DL_ERR_LAUNCH, "gemm_f32_tc: %s", cudaGetErrorString(e));
    }
    return DL_OK;
}

DL_PACKED(dl_gemm_f32_tc_scratch)
DL_PACKED(dl_gemm_f32_tc)
