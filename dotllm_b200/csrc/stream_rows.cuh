// What the kernels that stream matrices by rows share (gemm_skinny.cu, experts_rows.cu): the barriers of their rings, the tensor-core
// instruction, and how rows are cut into blocks, passes and tiles.
#pragma once
#include "common.cuh"
#include <stdint.h>

#ifndef GS_CONSUMERS
#define GS_CONSUMERS 8
#endif
#define GR_MOST 48                         // rows of a pass, at most (gated: 16 pairs)
#define GR_MAX_SLOTS 8                     // ring stages per consumer warp, at most
#define GR_THREADS(TILES) (32 * (GS_CONSUMERS + 1 + (TILES)))   // consumers, the producer warp, a warp a tile that adds
#define GR_SMEM 231168                     // bytes of shared memory for the rings and the sums, at most: what a block can have less the barriers
#define GR_CHAINS(TILES) ((TILES) == 1 ? 2 : 1)     // by TILES alone: a row's bits do not depend on NT (more cost registers and time)
#define GS_WAIT_CYCLES (1ll << 31)

__device__ __forceinline__ void gs_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                       uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// A chunk's products where the sums keep float32's accuracy: every instruction starts from zero, and what they leave is added up as a binary tree of
// rounded additions.  (The tensor core cuts an accumulator's low bits off with every instruction that adds to it, so a chain of them drifts.)
// S steps of 32 k, a power of two; the last one adds the chunk's sum to acc.
template <int S> struct GsTree {
    float level[4][4];
    __device__ __forceinline__ void add(int s, float (&acc)[4], const uint4& lo, const uint4& hi, const uint4& x) {
        static_assert(S >= 1 && S <= 16 && (S & (S - 1)) == 0, "a power of two");
        float u[4] = {0.f, 0.f, 0.f, 0.f}, v[4] = {0.f, 0.f, 0.f, 0.f};
        gs_mma(u, lo.x, hi.x, lo.y, hi.y, x.x, x.y);
        gs_mma(v, lo.z, hi.z, lo.w, hi.w, x.z, x.w);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            float sum = u[e] + v[e];
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                if (!(s >> l & 1)) break;                    // (constants once the caller's loop over s is unrolled)
                sum += level[l][e];
            }
            if (s == S - 1) acc[e] += sum;
            else level[s & 1 ? (s & 2 ? (s & 4 ? 3 : 2) : 1) : 0][e] = sum;
        }
    }
};

__device__ __forceinline__ uint32_t gs_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void gs_mbar_init(uint64_t* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(gs_smem(bar)), "r"(count));
}
__device__ __forceinline__ void gs_mbar_expect(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(gs_smem(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void gs_mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(gs_smem(bar)) : "memory");
}
__device__ __forceinline__ bool gs_mbar_try(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(gs_smem(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool gs_mbar_wait(uint64_t* bar, uint32_t parity, volatile int* gave_up) {
    if (gs_mbar_try(bar, parity)) return true;
    const long long t0 = clock64();
    while (!gs_mbar_try(bar, parity)) {
        if (*gave_up || clock64() - t0 > GS_WAIT_CYCLES) return false;
    }
    return true;
}
__device__ __forceinline__ uint4 gs_lds128(uint32_t addr) {     // 16 bytes from a shared-space byte address
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}

// Rows of a stage (gated: the up rows lie behind room for all tiles' gate rows), and bytes of a block's rings with what a read of the missing
// rows of the last tile reaches beyond them.
__host__ __device__ static inline int GR_stage_rows(int rows, bool gated, int tiles) { return gated ? 8 * tiles + rows : rows; }
__host__ __device__ static inline int GR_ring_bytes(int rows, int slots, bool gated, int tiles, int bk) {
    const int stage = GR_stage_rows(rows, gated, tiles);
    return (GS_CONSUMERS * slots * stage + 16 * tiles - stage) * bk * 2;
}

// How rows are shared out: rows of a block, passes of a block, rows of a pass, blocks.  By N and the device alone, so that the parts of a row's
// sum of squares lie the same for every product of that width.
struct GsRowsPlan {
    int block_rows, passes, rows, blocks;
};
static inline GsRowsPlan gs_rows_plan(int N, bool gated, int sms) {
    const int most = gated ? 16 : GR_MOST;
    GsRowsPlan p;
    p.block_rows = (N + sms - 1) / sms;
    p.passes = (p.block_rows + most - 1) / most;
    p.rows = (p.block_rows + p.passes - 1) / p.passes;
    p.blocks = (N + p.block_rows - 1) / p.block_rows;
    return p;
}
