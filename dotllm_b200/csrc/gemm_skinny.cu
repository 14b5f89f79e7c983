// y = x W^T for a handful of rows of x (decode steps): a weight-streaming product.
//
// With M <= 16 rows every projection is bound by the bytes of W, read once.  The reference runs
// these through cuBLAS or one-block-per-output-row GEMV kernels
// (src/DotLLM.Cuda/CudaTransformerModel.cs:317-349, native/kernels/quantized_gemv.cu:13-63).
// Here W is the 16-row operand of mma.sync.m16n8k16 and the tokens are its 8 columns: within a
// 32-wide slice of k, lane (g, t) holds k = 8t..8t+7 of rows g and g+8 and the same slice of token
// g's activations, which is a consistent permutation of k for both operands of two MMAs.
//
// Shape: persistent, warp-specialised, in two forms.  One producer warp per block (lane c serving consumer warp c) copies chunks of W as tiled
// boxes of a tensor map (cp.async.bulk.tensor.2d) into a private ring of shared-memory stages for each of eight consumer warps, signalling an
// mbarrier per stage; copies run ahead of the arithmetic by the depth of the ring.  Either way a result does not depend on the number of rows of x and
// is the same on every launch.  With FUSE_SWIGLU a tile's rows 0-7 are gate rows and rows 8-15 the matching up rows, and the epilogue
// writes silu(gate) * up (native/kernels/swiglu.cu:7-41).
//
// * By rows (gemm_skinny_rows_kernel; most sizes): every multiprocessor owns the same number of rows of W over all of k.  The consumer warps split k,
//   their sums meet in shared memory, and warps of their own add them in a fixed order and run the epilogue.  Nothing passes between blocks: no
//   partial sums through global memory, no counters.  A pass holds up to 48 rows, so a chunk's slice of x is read once for all of them (x is 8 / 48 of what
//   W is; with 16-row tiles it was half, and its loads' latency set the pace).
// * By shares (gemm_skinny_kernel; few rows a block and K > 4,096, see gs_by_rows): the list of (16-row tile, 256-wide chunk of k) pairs in
//   tile-major order is cut into equal contiguous shares, one per consumer warp of the whole grid.  A tile cut between shares is summed, in share
//   order, by whichever of its warps arrives last.
//
// By rows against by shares, each product in a graph of many, 8 rows: 3,072 x 2,048 5.5 -> 5.0 us, 2,048 x 2,048 5.1 -> 4.2, 64 x 2,048 3.8 -> 2.7, gated
// 8,192 x 2,048 15.4 -> 13.3, 6,144 x 4,096 12.7 -> 11.1, 4,096 x 14,336 22.1 -> 20.9, gated 14,336 x 4,096 40.3 -> 38.5, 128,256 x 2,048
// 87.0 -> 80.6 (6.5 TB/s); the small ones are a chain of latencies (start, rows of x, sums).  One tile a block leaves x at half the bytes of W again.
// A decode step of 16 layers of the smaller widths, 8 sequences at 2,000 tokens: 905 -> 849 us.  Tried: rings of half the size, so that the next product's first weights arrive under this one
// (941 us), x asked for three chunks ahead (2,048 x 2,048 4.3 -> 4.7), passes of 32 rows (5,120 x 13,824, 35 rows a block: 25.5 -> 30.1).
//
// Two optional fusions take the add + RMSNorm between two products of a decode step into the products
// themselves (the reference's fused_add_rmsnorm, native/kernels/fused_add_rmsnorm.cu:9-72, is a kernel
// of its own).  A float32 product with `gain` set adds its result into the float32 residual stream it
// is given as `out`, writes the sum times the norm's gain as bfloat16 (`scaled`) and the sum of squares
// of every tile and row (`sumsq_out`, a part of 16 floats a tile).  The product that follows takes `scaled` as its x
// and `sumsq_in`: a warp of its own adds the tiles' sums in tile order, and every output row is
// multiplied by rsqrt(sum / n + eps) in the epilogue - x W^T of the normalised row, since the
// normalisation is one factor per row.  All of it in float32 and in a fixed order.
//
// Every wait on an mbarrier is bounded (about a second of clock cycles); on expiry the kernel records
// a code in `status` and returns after waiting (bounded) for copies in flight.
#include "common.cuh"
#include "gating.cuh"
#include "stream_rows.cuh"
#include "tma.cuh"
#include <atomic>
#include <mutex>
#include <type_traits>
#include <unordered_map>

#ifndef GS_SLOTS
#define GS_SLOTS 3                         // ring stages per consumer warp
#endif
#define GS_BK 256                          // k per chunk
#define GS_STAGE_ELEMS (16 * GS_BK)         // a stage is the dense box the copy engine writes: [16 rows][256 k]
#define GS_THREADS (32 * (GS_CONSUMERS + 2))   // consumers, the producer warp, the row-statistics warp
#define GS_MAX_ROWS 16
template <typename TOut> __device__ __forceinline__ void gs_store(TOut* p, float v);
template <> __device__ __forceinline__ void gs_store<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void gs_store<__nv_bfloat16>(__nv_bfloat16* p, float v) {
    *p = __float2bfloat16_rn(v);
}

// The optional fusions of a launch (all pointers null: a plain product).
struct GsFuse {
    const float* gain;          // set: out is the float32 residual stream, out += x W^T in place, and ...
    __nv_bfloat16* scaled;      // ... scaled[m][n] = bf16(out[m][n] * gain[n]), rows scaled_stride apart,
    int scaled_stride;
    float* sumsq_out;           // ... sumsq_out[tile * 16 + m] = sum over the tile's 16 columns of out[m][n]^2
    const float* sumsq_in;      // set: output row m is multiplied by rsqrt(sum_p sumsq_in[p * 16 + m] * inv_n + eps)
    int n_parts;
    float inv_n, eps;
    int gate_kind;              // gated products: 0 = SwiGLU, else a gating of gating.cuh with ...
    float gate_limit, gate_alpha;   // ... its constants
    const float* gate_bias;     // gated products: set: [2N], added to the gate and the up rows' products before the gating
};

// acc[j] = {(row g, tok 2t), (row g, tok 2t+1), (row g+8, tok 2t), (row g+8, tok 2t+1)} of 8-token group j
// `row_scale`: null, or the factor of every output row (token).  `fuse.gain` (float32 plain products
// only): add into `out` and leave the scaled copy and the tile's sums of squares for the next product.
// The tile's rows of W are `base` .. `end` - 1 (at most 16, gated: pairs, at most 8); its sums of squares are part `part`.
template <int NT, typename TOut, bool FUSE_SWIGLU>
__device__ __forceinline__ void gs_epilogue(const float (&acc_in)[NT][4], TOut* out, int out_stride, int part, int base, int end, int M,
                                            int N, int g, int t, const float* row_scale, const GsFuse& fuse,
                                            const float (&stream_in)[NT][4], const float (&gain_in)[2]) {
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        const int tok0 = j * 8 + 2 * t;
        float acc[4] = {acc_in[j][0], acc_in[j][1], acc_in[j][2], acc_in[j][3]};
        if (row_scale != nullptr) {
            const float s0 = row_scale[tok0], s1 = row_scale[tok0 + 1];
            acc[0] *= s0, acc[1] *= s1, acc[2] *= s0, acc[3] *= s1;
        }
        if (FUSE_SWIGLU) {
            const int col = base + g;
            if (col < end) {
                if (fuse.gate_bias != nullptr) {
                    const float bg = __ldg(fuse.gate_bias + col), bu = __ldg(fuse.gate_bias + N + col);
                    acc[0] += bg, acc[1] += bg, acc[2] += bu, acc[3] += bu;
                }
                const float g0 = acc[0], g1 = acc[1];
                if (fuse.gate_kind != GATE_SILU) {
                    if (tok0 < M)
                        gs_store<TOut>(out + (size_t)tok0 * out_stride + col, dl_gate_value(fuse.gate_kind, g0, acc[2], fuse.gate_limit, fuse.gate_alpha));
                    if (tok0 + 1 < M)
                        gs_store<TOut>(out + (size_t)(tok0 + 1) * out_stride + col, dl_gate_value(fuse.gate_kind, g1, acc[3], fuse.gate_limit, fuse.gate_alpha));
                } else {
                    if (tok0 < M) gs_store<TOut>(out + (size_t)tok0 * out_stride + col, g0 * (1.0f / (1.0f + expf(-g0))) * acc[2]);
                    if (tok0 + 1 < M) gs_store<TOut>(out + (size_t)(tok0 + 1) * out_stride + col, g1 * (1.0f / (1.0f + expf(-g1))) * acc[3]);
                }
            }
        } else if (std::is_same<TOut, float>::value && fuse.gain != nullptr) {
            float* stream = reinterpret_cast<float*>(out);
            float ss[2] = {0.f, 0.f};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int row = base + g + (e >> 1) * 8, tok = tok0 + (e & 1);
                if (row < end && tok < M) {
                    const float h = stream_in[j][e] + acc[e];
                    stream[(size_t)tok * out_stride + row] = h;
                    fuse.scaled[(size_t)tok * fuse.scaled_stride + row] = __float2bfloat16_rn(h * gain_in[e >> 1]);
                    ss[e & 1] = fmaf(h, h, ss[e & 1]);
                }
            }
            // the tile's columns of a token lie in the 8 lanes that share t: add them in a fixed order
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                ss[e] += __shfl_xor_sync(0xffffffffu, ss[e], 4);
                ss[e] += __shfl_xor_sync(0xffffffffu, ss[e], 8);
                ss[e] += __shfl_xor_sync(0xffffffffu, ss[e], 16);
                if (g == 0 && tok0 + e < M) fuse.sumsq_out[(size_t)part * 16 + tok0 + e] = ss[e];
            }
        } else {
            if (!dl_gate_is_gated(fuse.gate_kind)) {         // an activation of the one product
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[e] = dl_unary_value(fuse.gate_kind, acc[e]);
            }
            const int row_lo = base + g, row_hi = row_lo + 8;
            if (row_lo < end) {
                if (tok0 < M) gs_store<TOut>(out + (size_t)tok0 * out_stride + row_lo, acc[0]);
                if (tok0 + 1 < M) gs_store<TOut>(out + (size_t)(tok0 + 1) * out_stride + row_lo, acc[1]);
            }
            if (row_hi < end) {
                if (tok0 < M) gs_store<TOut>(out + (size_t)tok0 * out_stride + row_hi, acc[2]);
                if (tok0 + 1 < M) gs_store<TOut>(out + (size_t)(tok0 + 1) * out_stride + row_hi, acc[3]);
            }
        }
    }
}

// Built with -DGS_TIMELINE (DOTLLM_NVCC_EXTRA), every warp of a product stamps the global nanosecond timer at six
// points of a launch into gs_timeline, which dl_gemm_skinny_timeline copies out
// (`python -m dotllm_b200.kernels.microbench gemm_skinny --timeline` prints the spread over the grid).
#define GS_TIMELINE_WARPS 12                     // of a block, at most (GR_THREADS(3) / 32)
#ifdef GS_TIMELINE
__device__ long long gs_timeline[6][2048];       // [event][block * GS_TIMELINE_WARPS + warp]
__device__ __forceinline__ long long gs_now() {
    long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
#define GS_STAMP(ev)                                                                                                     \
    do {                                                                                                                 \
        const int slot__ = blockIdx.x * GS_TIMELINE_WARPS + (threadIdx.x >> 5);                                             \
        if ((threadIdx.x & 31) == 0 && slot__ < 2048) gs_timeline[ev][slot__] = gs_now();                                 \
    } while (0)
extern "C" int dl_gemm_skinny_timeline(long long* out) {
    return cudaMemcpyFromSymbol(out, gs_timeline, sizeof(gs_timeline)) == cudaSuccess ? DL_OK : DL_ERR_LAUNCH;
}
#else
#define GS_STAMP(ev)
#endif

// The product of a launch: its operands and how its chunks are cut (see GsPlan below).
struct GsWork {
    const __nv_bfloat16* x;
    int x_stride;
    void* out;
    int out_stride;
    int M, N, K, up_offset, cpt, total_chunks, active, share;      // active: consumer warps of a block that have a share
    GsFuse fuse;
};

// The rings of a block: a private ring of GS_SLOTS stages per consumer warp.
struct GsRings {
    __nv_bfloat16* stage_mem;                               // [consumer][slot][16][GS_BK]
    uint64_t (*full_bar)[GS_SLOTS];
    uint64_t (*empty_bar)[GS_SLOTS];
    volatile int* gave_up;
    int* status;
    uint64_t* scale_bar;                                    // completes when row_scale is written
    const float* row_scale;                                 // [16] factors of the output rows (sumsq_in)
};

// Producer lane `lane` (< GS_CONSUMERS) feeds consumer warp `lane`: it walks that warp's share chunk
// by chunk, waits for the ring slot to be free, and issues one tiled copy (two for gate + up) per
// chunk.  `cnt` counts the chunks of this ring.  False: gave up.
template <bool FUSE_SWIGLU>
__device__ __forceinline__ bool gs_produce(const CUtensorMap* tmap, const GsWork& w, const GsRings& r, int lane, int& cnt) {
    const int gw = blockIdx.x * w.active + lane;
    int cur = min(w.total_chunks, gw * w.share);
    const int end = min(w.total_chunks, (gw + 1) * w.share);
    const uint64_t policy = dl_stream_policy();             // W is read once a step: first out of the L2
    // Every lane whose slot is free issues its next chunk; none waits inside for another lane's slot.
    long long t0 = clock64();
    while (cur < end) {
        const int slot = cnt % GS_SLOTS;
        if (cnt < GS_SLOTS || gs_mbar_try(&r.empty_bar[lane][slot], ((cnt / GS_SLOTS) - 1) & 1)) {
            const int tile = cur / w.cpt, kc = cur - tile * w.cpt;
            __nv_bfloat16* dst = r.stage_mem + (size_t)(lane * GS_SLOTS + slot) * GS_STAGE_ELEMS;
            // a box is always written whole: parts outside the matrix arrive as zeros
            gs_mbar_expect(&r.full_bar[lane][slot], GS_STAGE_ELEMS * 2);
            if (FUSE_SWIGLU) {
                dl_tma_load_2d_hint(dst, tmap, kc * GS_BK, tile * 8, &r.full_bar[lane][slot], policy);
                dl_tma_load_2d_hint(dst + 8 * GS_BK, tmap, kc * GS_BK, w.up_offset + tile * 8, &r.full_bar[lane][slot], policy);
            } else {
                dl_tma_load_2d_hint(dst, tmap, kc * GS_BK, tile * 16, &r.full_bar[lane][slot], policy);
            }
            ++cur, ++cnt;
            t0 = clock64();
        } else if (*r.gave_up || clock64() - t0 > GS_WAIT_CYCLES) {
            if (!*r.gave_up) atomicExch(r.status, 1);
            *r.gave_up = 1;
            return false;
        }
    }
    return true;
}

// After giving up: copies already issued must land before the block's shared memory is released.
__device__ __forceinline__ void gs_drain(const GsRings& r, int lane, int cnt) {
    for (int i = max(0, cnt - GS_SLOTS); i < cnt; ++i) {
        const long long t0 = clock64();
        while (!gs_mbar_try(&r.full_bar[lane][i % GS_SLOTS], (i / GS_SLOTS) & 1) && clock64() - t0 < GS_WAIT_CYCLES) {}
    }
}

// Consumer warp `warp` works through its share of the product.  `cnt` counts the chunks of its ring;
// `dead` is set when a wait expired.
template <int NT, typename TOut, bool FUSE_SWIGLU>
__device__ __forceinline__ void gs_consume(const GsWork& w, const GsRings& r, float* __restrict__ partials,
                                           int* __restrict__ counters, int warp, int lane, int& cnt, bool& dead) {
    const int g = lane >> 2, t = lane & 3;
    const int gw = blockIdx.x * w.active + warp;
    const int begin = min(w.total_chunks, gw * w.share), end = min(w.total_chunks, (gw + 1) * w.share);
    const int cpt = w.cpt, share = w.share, M = w.M, N = w.N, K = w.K;
    const __nv_bfloat16* x = w.x;
    TOut* out = reinterpret_cast<TOut*>(w.out);
    float acc[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
    const float* row_scale = nullptr;                    // set once the statistics warp has written the factors
    // The stream's values and the gains of the tile at hand, asked for when the tile begins so that the
    // epilogue does not wait for them (only this tile's finishing warp ever writes them).
    float stream_in[NT][4], gain_in[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) stream_in[j][e] = 0.f;
    int stream_tile = -1;
    int seg_begin = begin;                               // first chunk of the current tile's segment
    for (int cur = begin; cur < end; ++cur, ++cnt) {
        const int slot = cnt % GS_SLOTS;
        const int tile = cur / cpt, kc = cur - tile * cpt;
        const int k0 = kc * GS_BK;
        if (std::is_same<TOut, float>::value && !FUSE_SWIGLU && w.fuse.gain != nullptr && tile != stream_tile) {
            stream_tile = tile;
            const float* stream = reinterpret_cast<const float*>(w.out);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int row = tile * 16 + g + 8 * h;
                gain_in[h] = row < N ? __ldg(w.fuse.gain + row) : 0.f;
#pragma unroll
                for (int j = 0; j < NT; ++j)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int tok = j * 8 + 2 * t + e;
                        stream_in[j][2 * h + e] = (row < N && tok < M) ? __ldcg(stream + (size_t)tok * w.out_stride + row) : 0.f;
                    }
            }
        }
        // activations of this chunk, asked for before waiting on the weights
        uint4 xf[GS_BK / 32][NT];
#pragma unroll
        for (int s = 0; s < GS_BK / 32; ++s)
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                const int tok = j * 8 + g, k = k0 + 32 * s + 8 * t;
                xf[s][j] = make_uint4(0u, 0u, 0u, 0u);
                if (tok < M && k < K) xf[s][j] = __ldg(reinterpret_cast<const uint4*>(x + (size_t)tok * w.x_stride + k));
            }
        if (!dead && !gs_mbar_wait(&r.full_bar[warp][slot], (cnt / GS_SLOTS) & 1, r.gave_up)) {
            if (!*r.gave_up) atomicExch(r.status, 3);
            *r.gave_up = 1;
            dead = true;
        }
        if (cur == begin) GS_STAMP(2);                        // the first chunk of the share has landed
        if (!dead) {
            // this lane's byte address in shared space; the loads below are constant offsets away.
            // Rows beyond the matrix and k beyond K arrived as zeros, so nothing needs guarding.
            const uint32_t st = gs_smem(r.stage_mem + (size_t)(warp * GS_SLOTS + slot) * GS_STAGE_ELEMS) +
                                (uint32_t)(g * GS_BK + 8 * t) * 2u;
#pragma unroll
            for (int s = 0; s < GS_BK / 32; ++s) {
                const uint4 a_lo = gs_lds128(st + (uint32_t)(32 * s * 2));
                const uint4 a_hi = gs_lds128(st + (uint32_t)((8 * GS_BK + 32 * s) * 2));
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    gs_mma(acc[j], a_lo.x, a_hi.x, a_lo.y, a_hi.y, xf[s][j].x, xf[s][j].y);
                    gs_mma(acc[j], a_lo.z, a_hi.z, a_lo.w, a_hi.w, xf[s][j].z, xf[s][j].w);
                }
            }
            // The slot may be released only after every MMA fed from it has been issued (an MMA issues
            // when its operands have arrived from shared memory; a released slot is overwritten by the
            // next copy at once).  The MMAs are not volatile, so pin their results here: the compiler
            // cannot sink them below this point.
#pragma unroll
            for (int j = 0; j < NT; ++j) asm volatile("" : "+f"(acc[j][0]), "+f"(acc[j][1]), "+f"(acc[j][2]), "+f"(acc[j][3]));
            // ... and the reads themselves must be done before the copy engine may overwrite the stage:
            // without this fence a slot that was refilled at once showed rows of the new chunk to the old reads.
            __threadfence_block();
            __syncwarp();
            if (lane == 0) gs_mbar_arrive(&r.empty_bar[warp][slot]);
        }
        if (cur == end - 1) GS_STAMP(3);                      // the last chunk of the share is consumed
        if (kc == cpt - 1 || cur == end - 1) {
            // ---- the segment [seg_begin, cur] of this tile is done
            const bool whole = (seg_begin == tile * cpt) && (kc == cpt - 1);
            if (w.fuse.sumsq_in != nullptr && row_scale == nullptr && !dead) {
                // the factors of the rows: written by the statistics warp long before the first tile ends
                if (!gs_mbar_wait(r.scale_bar, 0, r.gave_up)) {
                    if (!*r.gave_up) atomicExch(r.status, 5);
                    *r.gave_up = 1;
                    dead = true;
                } else {
                    row_scale = r.row_scale;
                }
            }
            if (whole) {
                gs_epilogue<NT, TOut, FUSE_SWIGLU>(acc, out, w.out_stride, tile, tile * (FUSE_SWIGLU ? 8 : 16), N, M, N, g, t, row_scale, w.fuse, stream_in, gain_in);
            } else {
                // a warp's first tile may be shared with the share before, its last with the share after
                const int which = (tile == begin / cpt) ? 0 : 1;
                float* mine = partials + ((size_t)gw * 2 + which) * (NT * 4 * 32);
#pragma unroll
                for (int j = 0; j < NT; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) mine[(j * 4 + e) * 32 + lane] = acc[j][e];
                __syncwarp();
                const int g_lo = (tile * cpt) / share, g_hi = ((tile + 1) * cpt - 1) / share;
                int last = 0;
                if (lane == 0) {
                    // One read-modify-write that releases this warp's part (the lanes' stores are ordered
                    // before it by the __syncwarp above) and acquires the parts of the warps counted before.
                    int seen;
                    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(seen) : "l"(counters + tile) : "memory");
                    last = (seen == g_hi - g_lo) ? 1 : 0;
                    if (last) counters[tile] = 0;        // ready for the next product or launch
                }
                last = __shfl_sync(0xffffffffu, last, 0);
                __syncwarp();                            // the other lanes' reads below come after lane 0's acquire
                if (last) {
#pragma unroll
                    for (int j = 0; j < NT; ++j)
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
                    for (int gg = g_lo; gg <= g_hi; ++gg) {          // share order: fixed
                        const int wh = (tile == (gg * share) / cpt) ? 0 : 1;
                        const float* theirs = partials + ((size_t)gg * 2 + wh) * (NT * 4 * 32);
#pragma unroll
                        for (int j = 0; j < NT; ++j)
#pragma unroll
                            for (int e = 0; e < 4; ++e) acc[j][e] += __ldcg(theirs + (j * 4 + e) * 32 + lane);
                    }
                    gs_epilogue<NT, TOut, FUSE_SWIGLU>(acc, out, w.out_stride, tile, tile * (FUSE_SWIGLU ? 8 : 16), N, M, N, g, t, row_scale, w.fuse, stream_in, gain_in);
                }
            }
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
            seg_begin = cur + 1;
        }
    }
}

#define GS_INIT_RINGS()                                                                                  \
    extern __shared__ __align__(128) unsigned char gs_smem_raw[];                                        \
    __shared__ uint64_t full_bar[GS_CONSUMERS][GS_SLOTS], empty_bar[GS_CONSUMERS][GS_SLOTS];             \
    __shared__ volatile int gave_up;                                                                     \
    __shared__ uint64_t scale_bar;                                                                       \
    __shared__ float row_scale_smem[GS_MAX_ROWS];                                                        \
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;                                          \
    if (threadIdx.x == 0) {                                                                              \
        gave_up = 0;                                                                                     \
        gs_mbar_init(&scale_bar, 1);                                                                     \
        for (int c = 0; c < GS_CONSUMERS; ++c)                                                           \
            for (int s = 0; s < GS_SLOTS; ++s) {                                                         \
                gs_mbar_init(&full_bar[c][s], 1);                                                        \
                gs_mbar_init(&empty_bar[c][s], 1);                                                       \
            }                                                                                            \
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");                               \
    }                                                                                                    \
    __syncthreads();                                                                                     \
    dl_launch_dependents();                                                                              \
    const GsRings rings{reinterpret_cast<__nv_bfloat16*>(gs_smem_raw), full_bar, empty_bar, &gave_up, status, &scale_bar,  \
                        row_scale_smem}

// The row-statistics warp: the factors of the output rows from the sums that the product before left (`scale_bar` completes when they are written).
__device__ __forceinline__ void gs_row_factors(const GsFuse& fuse, float* factors, uint64_t* scale_bar, int lane) {
    if (fuse.sumsq_in == nullptr) return;
    dl_grid_dependency_wait();   // the sums come from the kernel before this one
    // A warp-wide float4 load covers 8 parts x 16 rows: lane -> (rows 4q .. 4q+3, part l/4 of
    // every 8).  All loads of a batch are in flight together; a lane adds its parts in part
    // order, then the 8 lanes of a row group are added in a fixed order: the same bits on
    // every launch.
    const int q = lane & 3, sub = lane >> 2;
    const float4* in = reinterpret_cast<const float4*>(fuse.sumsq_in) + q;
    float4 acc4 = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int p0 = 0; p0 < fuse.n_parts; p0 += 8 * 16) {
        float4 v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int p = p0 + 8 * i + sub;
            v[i] = p < fuse.n_parts ? __ldcg(in + (size_t)p * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) acc4.x += v[i].x, acc4.y += v[i].y, acc4.z += v[i].z, acc4.w += v[i].w;
    }
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
        // both partners add (lower lane's value) + (higher lane's value)
        const float4 other = make_float4(__shfl_xor_sync(0xffffffffu, acc4.x, o), __shfl_xor_sync(0xffffffffu, acc4.y, o),
                                         __shfl_xor_sync(0xffffffffu, acc4.z, o), __shfl_xor_sync(0xffffffffu, acc4.w, o));
        const bool low = (lane & o) == 0;
        acc4.x = low ? acc4.x + other.x : other.x + acc4.x;
        acc4.y = low ? acc4.y + other.y : other.y + acc4.y;
        acc4.z = low ? acc4.z + other.z : other.z + acc4.z;
        acc4.w = low ? acc4.w + other.w : other.w + acc4.w;
    }
    if (lane < 4) {
        factors[4 * lane + 0] = rsqrtf(acc4.x * fuse.inv_n + fuse.eps);
        factors[4 * lane + 1] = rsqrtf(acc4.y * fuse.inv_n + fuse.eps);
        factors[4 * lane + 2] = rsqrtf(acc4.z * fuse.inv_n + fuse.eps);
        factors[4 * lane + 3] = rsqrtf(acc4.w * fuse.inv_n + fuse.eps);
    }
    __threadfence_block();
    __syncwarp();
    if (lane == 0) gs_mbar_arrive(scale_bar);
}

template <int NT, typename TOut, bool FUSE_SWIGLU>
__global__ void __launch_bounds__(GS_THREADS, 1)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmap, const GsWork work, int early_weights,
                   float* __restrict__ partials, int* __restrict__ counters, int* __restrict__ status) {
    GS_STAMP(0);                                              // block started
    GS_INIT_RINGS();
    GS_STAMP(1);                                              // barriers ready
    if (warp == GS_CONSUMERS) {
        // ------------------------------------------------------------ producer warp
        // When the caller vouches that no pending work writes the weights (early_weights), the
        // producer does not wait for the kernel before this one: while that kernel finishes, the
        // rings fill.
        if (!early_weights) dl_grid_dependency_wait();
        if (lane < work.active) {
            int cnt = 0;
            if (!gs_produce<FUSE_SWIGLU>(&tmap, work, rings, lane, cnt)) gs_drain(rings, lane, cnt);
        }
    } else if (warp == GS_CONSUMERS + 1) {
        // ------------------------------------------------------------ row-statistics warp
        gs_row_factors(work.fuse, row_scale_smem, &scale_bar, lane);
    } else if (warp < work.active) {
        // ------------------------------------------------------------ consumer warp
        dl_grid_dependency_wait();       // x comes from the kernel before this one; out, partials and counters may be in use by it
        int cnt = 0;
        bool dead = false;
        gs_consume<NT, TOut, FUSE_SWIGLU>(work, rings, partials, counters, warp, lane, cnt, dead);
        GS_STAMP(4);                                          // share done, hand-over of cut tiles included
    }
    __syncthreads();                                         // nobody leaves while copies may still land
    GS_STAMP(5);
}

// ---------------------------------------------------------------------------------------------
// Rows shared out evenly: block b owns rows R b .. R (b + 1) - 1 of W (R = ceil(N / multiprocessors)) over all of k, in `passes` passes of `rows` <= 48
// of them (gated: pairs, <= 16), TILES tiles of 16 (8 pairs) at most.  A pass's chunks of BK k go round the block's eight consumer warps; at its end the warps' sums meet in
// shared memory, where a warp a tile adds them in warp order while the others go on with the next pass.  Nothing passes between blocks.
struct GsRowsWork {
    const __nv_bfloat16* x;
    int x_stride;
    void* out;
    int out_stride;
    int M, N, K, up_offset, cpt, block_rows, rows, passes, slots, sums;     // ring stages of a consumer warp; passes whose sums have room
    GsFuse fuse;
};

// Tiles of 16 rows that n rows make in passes of `rows`.
__host__ __device__ static inline int gs_rows_tiles(int n, int rows) {
    const int full = n / rows, rest = n - full * rows;
    return full * ((rows + 15) / 16) + (rest + 15) / 16;
}

// A lane's values of the tokens: a step of 32 k, a chunk.
template <int NT>
__device__ __forceinline__ void gs_rows_x(uint4 (&xf)[NT], const GsRowsWork& w, int k0, int g, int t) {
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        const int tok = j * 8 + g, k = k0 + 8 * t;
        xf[j] = make_uint4(0u, 0u, 0u, 0u);
        if (tok < w.M && k < w.K) xf[j] = __ldg(reinterpret_cast<const uint4*>(w.x + (size_t)tok * w.x_stride + k));
    }
}
template <int NT, int S>
__device__ __forceinline__ void gs_rows_x(uint4 (&xf)[S][NT], const GsRowsWork& w, int k0, int g, int t) {
#pragma unroll
    for (int s = 0; s < S; ++s) gs_rows_x<NT>(xf[s], w, k0 + 32 * s, g, t);
}

template <int NT, typename TOut, bool FUSE_SWIGLU, int TILES, int BK>
__global__ void __launch_bounds__(GR_THREADS(TILES), 1)
gemm_skinny_rows_kernel(const __grid_constant__ CUtensorMap tmap, const GsRowsWork w, int early_weights, int* __restrict__ status) {
    constexpr int TILE = FUSE_SWIGLU ? 8 : 16;               // rows (gated: pairs) of a tile
    constexpr int CHAINS = GR_CHAINS(TILES);                 // accumulators that a chunk's instructions go round: they wait for one another otherwise
    // The next chunk's values of x are asked for before this one's arithmetic, into registers of their own.  Chunks of 256 k ask behind every step, into the
    // registers that it has left: two sets of 16 tokens spilled, and a spilled load is waited for (2,048 x 14,336, 10 rows: 25.8 us, this way 15.8; 8 rows
    // 13.9 both ways; 2,048 x 4,096, 8 rows 6.0 and 5.9).  Chunks of 128 lose by it (4,096 x 8,192, 8 rows: 14.3 and 14.7).
    constexpr bool IN_PLACE = BK == 256;
    extern __shared__ __align__(128) unsigned char gs_smem_raw[];
    __shared__ uint64_t full_bar[GS_CONSUMERS][GR_MAX_SLOTS], empty_bar[GS_CONSUMERS][GR_MAX_SLOTS], scale_bar, sums_full[2], sums_empty[2];
    __shared__ volatile int gave_up;
    __shared__ float row_scale_smem[GS_MAX_ROWS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    GS_STAMP(0);                                             // block started
    if (threadIdx.x == 0) {
        gave_up = 0;
        gs_mbar_init(&scale_bar, 1);
        for (int h = 0; h < 2; ++h) gs_mbar_init(&sums_full[h], GS_CONSUMERS), gs_mbar_init(&sums_empty[h], TILES);
        for (int c = 0; c < GS_CONSUMERS; ++c)
            for (int s = 0; s < w.slots; ++s) {
                gs_mbar_init(&full_bar[c][s], 1);
                gs_mbar_init(&empty_bar[c][s], 1);
            }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    dl_launch_dependents();
    GS_STAMP(1);                                             // barriers ready
    const int first = blockIdx.x * w.block_rows, end_row = min(w.N, first + w.block_rows);      // this block's rows
    const int passes = (end_row - first + w.rows - 1) / w.rows, total = passes * w.cpt;
    const uint32_t box_bytes = w.rows * (BK * 2), stage_bytes = GR_stage_rows(w.rows, FUSE_SWIGLU, TILES) * (BK * 2);
    // the sums of a pass, or of two passes in turn: [sums][warp][tile][NT][lane]
    float4* sums = reinterpret_cast<float4*>(gs_smem_raw + GR_ring_bytes(w.rows, w.slots, FUSE_SWIGLU, TILES, BK));
    if (warp < GS_CONSUMERS) {
        // ------------------------------------------------------------ consumer warp
        dl_grid_dependency_wait();       // x comes from the kernel before this one
        uint4 xf[BK / 32][NT];
        int cur = warp, slot = 0, phase = 0;
        bool dead = false;
        auto gave = [&](int code) {
            if (!gave_up) atomicExch(status, code);
            gave_up = 1;
            dead = true;
        };
        if (cur < total) gs_rows_x<NT>(xf, w, (cur % w.cpt) * BK, g, t);
        for (int p = 0; p < passes; ++p) {
            float acc[TILES][NT][CHAINS][4];
#pragma unroll
            for (int i = 0; i < TILES; ++i)
#pragma unroll
                for (int j = 0; j < NT; ++j)
#pragma unroll
                    for (int e = 0; e < 4 * CHAINS; ++e) acc[i][j][e / 4][e % 4] = 0.f;
            for (const int pass_end = (p + 1) * w.cpt; cur < pass_end; cur += GS_CONSUMERS) {
                if (!dead && !gs_mbar_wait(&full_bar[warp][slot], phase, &gave_up)) gave(3);
                if (cur == warp) GS_STAMP(2);                // the warp's first chunk has landed
                const int next = cur + GS_CONSUMERS, k_next = next < total ? (next % w.cpt) * BK : w.K;
                uint4 xn[BK / 32][NT];
                if (!IN_PLACE) gs_rows_x<NT>(xn, w, k_next, g, t);
                if (!dead) {
                    // rows beyond the box are whatever lies behind it: they reach output rows that are not stored
                    const uint32_t st = gs_smem(gs_smem_raw + (size_t)(warp * w.slots + slot) * stage_bytes) + (uint32_t)(g * BK + 8 * t) * 2u;
                    const int tiles = (w.rows + TILE - 1) / TILE;
#pragma unroll
                    for (int s = 0; s < BK / 32; ++s) {
#pragma unroll
                        for (int i = 0; i < TILES; ++i) {
                            if (i >= tiles) break;
                            // a plain tile's upper eight rows lie behind its lower eight, a gated one's behind all gate rows
                            const uint4 a_lo = gs_lds128(st + (uint32_t)((TILE * i * BK + 32 * s) * 2));
                            const uint4 a_hi = gs_lds128(st + (uint32_t)(((FUSE_SWIGLU ? TILE * TILES + TILE * i : TILE * i + 8) * BK + 32 * s) * 2));
#pragma unroll
                            for (int j = 0; j < NT; ++j) {
                                gs_mma(acc[i][j][2 * s % CHAINS], a_lo.x, a_hi.x, a_lo.y, a_hi.y, xf[s][j].x, xf[s][j].y);
                                gs_mma(acc[i][j][(2 * s + 1) % CHAINS], a_lo.z, a_hi.z, a_lo.w, a_hi.w, xf[s][j].z, xf[s][j].w);
                            }
                        }
                        if (IN_PLACE) gs_rows_x<NT>(xf[s], w, k_next + 32 * s, g, t);
                    }
                    // as in gs_consume: the slot is released when every read of it is done
#pragma unroll
                    for (int i = 0; i < TILES; ++i)
#pragma unroll
                        for (int j = 0; j < NT; ++j)
#pragma unroll
                            for (int c = 0; c < CHAINS; ++c)
                                asm volatile("" : "+f"(acc[i][j][c][0]), "+f"(acc[i][j][c][1]), "+f"(acc[i][j][c][2]), "+f"(acc[i][j][c][3]));
                    __threadfence_block();
                    __syncwarp();
                    if (lane == 0) gs_mbar_arrive(&empty_bar[warp][slot]);
                }
                if (++slot == w.slots) slot = 0, phase ^= 1;
                if (next >= total) GS_STAMP(3);              // the warp's last chunk is consumed
                if (!IN_PLACE) {
#pragma unroll
                    for (int s = 0; s < BK / 32; ++s)
#pragma unroll
                        for (int j = 0; j < NT; ++j) xf[s][j] = xn[s][j];
                }
            }
            const int h = w.sums == 2 ? p & 1 : 0, turn = w.sums == 2 ? p >> 1 : p;      // whose turn it is with sums h
            if (turn >= 1 && !dead && !gs_mbar_wait(&sums_empty[h], (turn - 1) & 1, &gave_up)) gave(6);
            float4* mine = sums + (size_t)(h * GS_CONSUMERS + warp) * TILES * NT * 32 + lane;
            if (!dead) {
#pragma unroll
                for (int i = 0; i < TILES; ++i)
#pragma unroll
                    for (int j = 0; j < NT; ++j) {
                        float (&a)[4] = acc[i][j][0];
#pragma unroll
                        for (int c = 1; c < CHAINS; ++c)
#pragma unroll
                            for (int e = 0; e < 4; ++e) a[e] += acc[i][j][c][e];
                        mine[(i * NT + j) * 32] = make_float4(a[0], a[1], a[2], a[3]);
                    }
            }
            __threadfence_block();
            __syncwarp();
            if (lane == 0) gs_mbar_arrive(&sums_full[h]);
        }
        GS_STAMP(4);                                         // its sums are handed over
    } else if (warp == GS_CONSUMERS) {
        // ------------------------------------------------------------ producer warp: lane c serves consumer warp c
        // When the caller vouches that no pending work writes the weights (early_weights), the rings fill while the kernel before this one finishes.
        if (!early_weights) dl_grid_dependency_wait();
        if (lane < GS_CONSUMERS) {
            const uint64_t policy = dl_stream_policy();      // W is read once a step: first out of the L2
            int cnt = 0, cur = lane, slot = 0, phase = 1;
            bool ok = true;
            long long t0 = clock64();
            while (cur < total) {
                if (cnt < w.slots || gs_mbar_try(&empty_bar[lane][slot], phase)) {
                    const int pass = cur / w.cpt, kc = cur - pass * w.cpt, row = first + pass * w.rows;
                    unsigned char* dst = gs_smem_raw + (size_t)(lane * w.slots + slot) * stage_bytes;
                    // a box is always written whole: parts outside the matrix arrive as zeros
                    gs_mbar_expect(&full_bar[lane][slot], FUSE_SWIGLU ? 2 * box_bytes : box_bytes);
                    dl_tma_load_2d_hint(dst, &tmap, kc * BK, row, &full_bar[lane][slot], policy);
                    if (FUSE_SWIGLU) dl_tma_load_2d_hint(dst + TILES * TILE * BK * 2, &tmap, kc * BK, w.up_offset + row, &full_bar[lane][slot], policy);
                    cur += GS_CONSUMERS, ++cnt;
                    if (++slot == w.slots) slot = 0, phase ^= 1;
                    t0 = clock64();
                } else if (gave_up || clock64() - t0 > GS_WAIT_CYCLES) {
                    if (!gave_up) atomicExch(status, 1);
                    gave_up = 1;
                    ok = false;
                    break;
                }
            }
            if (!ok)                                         // copies already issued must land before the block's shared memory is released
                for (int i = max(0, cnt - w.slots); i < cnt; ++i) {
                    const long long t1 = clock64();
                    while (!gs_mbar_try(&full_bar[lane][i % w.slots], (i / w.slots) & 1) && clock64() - t1 < GS_WAIT_CYCLES) {}
                }
        }
    } else {
        // ------------------------------------------------------------ adding warps: one a tile of a pass; the first makes the row factors before that
        const int tile = warp - GS_CONSUMERS - 1, N = w.N, M = w.M;
        if (tile == 0) gs_row_factors(w.fuse, row_scale_smem, &scale_bar, lane);
        dl_grid_dependency_wait();                           // out may be in use by the kernel before this one
        TOut* out = reinterpret_cast<TOut*>(w.out);
        const bool into = std::is_same<TOut, float>::value && !FUSE_SWIGLU && w.fuse.gain != nullptr;
        const float* row_scale = nullptr;
        bool dead = false;
        for (int p = 0; p < passes && !dead; ++p) {
            const int h = w.sums == 2 ? p & 1 : 0, turn = w.sums == 2 ? p >> 1 : p, pass_end = min(end_row, first + (p + 1) * w.rows);
            const int base = first + p * w.rows + tile * TILE;
            // the stream's values and the gains, asked for early so that the epilogue does not wait for them (only this warp ever writes them)
            float stream_in[NT][4], gain_in[2] = {0.f, 0.f};
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) stream_in[j][e] = 0.f;
            if (into) {
                const float* stream = reinterpret_cast<const float*>(w.out);
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const int row = base + g + 8 * r;
                    gain_in[r] = row < pass_end ? __ldg(w.fuse.gain + row) : 0.f;
#pragma unroll
                    for (int j = 0; j < NT; ++j)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int tok = j * 8 + 2 * t + e;
                            stream_in[j][2 * r + e] = (row < pass_end && tok < M) ? __ldcg(stream + (size_t)tok * w.out_stride + row) : 0.f;
                        }
                }
            }
            if (!gs_mbar_wait(&sums_full[h], turn & 1, &gave_up) ||
                (w.fuse.sumsq_in != nullptr && row_scale == nullptr && !gs_mbar_wait(&scale_bar, 0, &gave_up))) {
                if (!gave_up) atomicExch(status, 5);
                gave_up = 1;
                dead = true;
                continue;
            }
            if (w.fuse.sumsq_in != nullptr) row_scale = row_scale_smem;
            float acc[NT][4];
            const float4* theirs = sums + (size_t)(h * GS_CONSUMERS * TILES + tile) * NT * 32 + lane;
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                float4 v[GS_CONSUMERS];
#pragma unroll
                for (int c = 0; c < GS_CONSUMERS; ++c) v[c] = theirs[(c * TILES * NT + j) * 32];
                acc[j][0] = v[0].x, acc[j][1] = v[0].y, acc[j][2] = v[0].z, acc[j][3] = v[0].w;
#pragma unroll
                for (int c = 1; c < GS_CONSUMERS; ++c) acc[j][0] += v[c].x, acc[j][1] += v[c].y, acc[j][2] += v[c].z, acc[j][3] += v[c].w;
            }
            __syncwarp();
            if (lane == 0) gs_mbar_arrive(&sums_empty[h]);
            if (base < pass_end)
                gs_epilogue<NT, TOut, FUSE_SWIGLU>(acc, out, w.out_stride, blockIdx.x * gs_rows_tiles(w.block_rows, w.rows) + p * ((w.rows + 15) / 16) + tile, base, pass_end, M, N, g, t, row_scale, w.fuse, stream_in, gain_in);
        }
    }
    __syncthreads();                                         // nobody leaves while copies may still land
    GS_STAMP(5);
}

// Which products go that way; the others by shares.  By rows every block reads all of x, by shares what passes between blocks takes its time: rows
// for short k and where a block has many rows, shares for a few rows of long k.  By the sizes alone, so that a row's bits do not depend on the
// number of rows of x.  Measured at 8 and at 10 rows of x, by rows / by shares, us (2,048 columns: 14 rows of W a block of 148; 1,536: 11; 2,400: 17):
//   2,048 x 4,096   6.0 6.7 / 6.3 6.7      2,048 x 8,192   9.7 11.1 / 9.3 10.0      2,048 x 14,336  13.9 15.8 / 13.4 14.3
//   2,048 x 5,120   7.3 8.2 / 8.0 8.6      2,048 x 12,288 12.6 14.2 / 11.8 12.8     2,048 x 16,384  15.1 17.6 / 15.9 16.6
//   1,536 x 14,336 12.6 14.5 / 11.1 12.2   512 x 4,096      4.5  5.3 / 5.1  5.8      512 x 14,336   10.2 12.6 / 8.0 9.1
//   2,400 x 4,096 and less as 2,048        2,400 x 8,192  12.6 14.3 / 11.4 12.2     3,072 x 8,192   13.4 14.2 / 13.2 13.9
//   2,368 x 12,288 13.5 15.5 / 14.3 14.8   2,368 x 16,384 16.4 18.6 / 17.3 17.8      (14 to 16 rows a block and K >= 12,288: level, 5 % either way)
// Gated: 1,024 x 14,336 (14 rows: 7 pairs) 13.9 15.8 / 13.1 13.9, 512 x 8,192 7.6 9.0 / 6.9 8.0, 512 x 14,336 10.8 13.5 / 9.4 10.6, 64 x 14,336 9.5 12.2 / 7.7 8.8.
static bool gs_by_rows(int N, int K, bool gated, int sms) {
    const int rows = (gated ? 2 : 1) * ((N + sms - 1) / sms);     // of W a block
    if (K <= 4096 || rows > 20) return true;
    if (gated) return rows >= 14;
    return rows >= 14 && rows <= 16 && (K <= 5120 || K >= 12288);
}

// Parts of the sums of squares (16 floats each) that a product of N output columns over K leaves.
extern "C" int dl_gemm_skinny_parts(int N, int K) {
    const int sms = dl_sm_count();
    if (!gs_by_rows(N, K, false, sms)) return (N + 15) / 16;
    const GsRowsPlan p = gs_rows_plan(N, false, sms);
    const int last = N - (p.blocks - 1) * p.block_rows;      // the last block may have fewer rows
    return (p.blocks - 1) * gs_rows_tiles(p.block_rows, p.rows) + gs_rows_tiles(last, p.rows);
}

// How the work of an (N, K) matrix is cut: tiles of 16 rows (8 gate + 8 up when gated), chunks per
// tile, consumer warps of a block with a share, chunks of a share, blocks.  Depends on the matrix and the device only, never on M.
struct GsPlan {
    int tiles, cpt, total, active, share, blocks;
};

static GsPlan gs_plan(int N, int K, int fuse_swiglu, int sms) {
    GsPlan p;
    p.tiles = fuse_swiglu ? (N + 7) / 8 : (N + 15) / 16;
    p.cpt = (K + GS_BK - 1) / GS_BK;
    p.total = p.tiles * p.cpt;
    // A share is a whole number of chunks, so the last multiprocessors get less, or nothing: the number of warps, and the share, that leave the busiest
    // multiprocessor the fewest chunks.  Shares that do not divide a tile's chunks count six more: their warps end one tile and begin another, about 1 us
    // (1,536 x 8,192, 8 rows: seven warps of 3 of 32 chunks 8.75 us, six of 4 7.9; 1,024 x 10,240: six of 3 of 40 8.9, six of 4 8.1).  And a tile is cut
    // into 31 parts at most, or fewer where k is long, since one warp adds them all (512 x 8,192: 32 parts 7.3 us, 16 6.3; 512 x 12,288: 24
    // parts 7.3, 12 7.2; 16 x 16,384: 64 parts 9.0, 32 7.1, 16 6.7).  Of equals the one with more warps: they have more of the ring.
    const int least = p.cpt >= 48 ? 4 : p.cpt >= 32 ? 2 : 1;
    int best = 0;
    for (int c = GS_CONSUMERS; c >= GS_CONSUMERS / 2; --c) {
        const int even = (p.total + sms * c - 1) / (sms * c), first = even > least ? even : least;
        for (int share = first; share <= first + 1; ++share) {
            const int cost = 2 * (c * share + (p.cpt % share != 0 ? 6 : 0)) + (p.cpt % share != 0 ? 1 : 0);
            if (best == 0 || cost < best) best = cost, p.active = c, p.share = share;
        }
    }
    p.blocks = (p.total + p.active * p.share - 1) / (p.active * p.share);
    if (p.blocks < 1) p.blocks = 1;
    return p;
}

// The form and the cut of a product on a device of `sms` multiprocessors: by rows (1) or by shares (0), and by shares the warps of a block that have one,
// its chunks, blocks.
extern "C" int dl_gemm_skinny_plan(int N, int K, int gated, int sms, int* by_rows, int* active, int* share, int* blocks) {
    DL_REQUIRE(N > 0 && K > 0 && sms > 0, "gemm_skinny_plan: bad sizes");
    const GsPlan p = gs_plan(N, K, gated, sms);
    *by_rows = gs_by_rows(N, K, gated != 0, sms) ? 1 : 0, *active = p.active, *share = p.share, *blocks = p.blocks;
    return DL_OK;
}

// Scratch the product needs: float32 partial sums and int32 arrival counters (zero before the first
// launch; every launch leaves them zero).
extern "C" int dl_gemm_skinny_scratch(int M, int N, int K, int fuse_swiglu, int sms, int* partial_floats,
                                      int* n_counters) {
    const GsPlan p = gs_plan(N, K, fuse_swiglu, sms);
    const int nt = M <= 8 ? 1 : 2;
    *partial_floats = p.blocks * GS_CONSUMERS * 2 * nt * 4 * 32;
    *n_counters = p.tiles;
    return DL_OK;
}

// Tensor map of W: `rows` rows of K bfloat16, boxes of `box` rows by `bk` columns.  Encoding
// costs a driver call, so maps are kept per (matrix, shape).
struct GsMapKey {
    const void* w;
    int rows, k, box, bk;
    bool operator==(const GsMapKey& o) const { return w == o.w && rows == o.rows && k == o.k && box == o.box && bk == o.bk; }
};
struct GsMapKeyHash {
    size_t operator()(const GsMapKey& k) const {
        return std::hash<const void*>()(k.w) ^ ((size_t)k.rows * 1000003u) ^ ((size_t)k.k * 10007u) ^ (size_t)(k.box + 32 * k.bk);
    }
};

static int gs_weight_map(CUtensorMap* out, const void* w, int rows, int K, int box, int bk) {
    static std::unordered_map<GsMapKey, CUtensorMap, GsMapKeyHash> maps;
    static std::mutex maps_mutex;
    std::lock_guard<std::mutex> lock(maps_mutex);
    const GsMapKey key{w, rows, K, box, bk};
    auto it = maps.find(key);
    if (it == maps.end()) {
        CUtensorMap fresh;
        if (dl_tmap_encode_2d_bf16(&fresh, w, (uint64_t)rows, (uint64_t)K, (uint64_t)K * 2, box, bk, DL_TMAP_SWIZZLE_NONE) != 0)
            return DL_ERR_LAUNCH;
        if (maps.size() > 4096) maps.clear();
        it = maps.emplace(key, fresh).first;
    }
    *out = it->second;
    return DL_OK;
}

template <int NT, typename TOut, bool FUSE>
static int gs_launch(const GsPlan& p, cudaStream_t s, const __nv_bfloat16* x, int x_stride, const __nv_bfloat16* w,
                     void* out, int out_stride, int M, int N, int K, int up_offset, int early_weights, float* partials,
                     int* counters, int* status, const GsFuse& fuse) {
    const size_t smem = (size_t)GS_CONSUMERS * GS_SLOTS * GS_STAGE_ELEMS * 2;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(gemm_skinny_kernel<NT, TOut, FUSE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return dl_fail(DL_ERR_LAUNCH, "gemm_skinny: shared memory %zu: %s", smem, cudaGetErrorString(e));
        configured = true;
    }
    CUtensorMap tmap;
    const int rc = gs_weight_map(&tmap, w, FUSE ? 2 * N : N, K, FUSE ? 8 : 16, GS_BK);
    if (rc != DL_OK) return rc;
    const GsWork work{x, x_stride, out, out_stride, M, N, K, up_offset, p.cpt, p.total, p.active, p.share, fuse};
    cudaError_t le = dl_launch_dependent(gemm_skinny_kernel<NT, TOut, FUSE>, dim3(p.blocks), dim3(GS_THREADS), smem, s, tmap, work,
                                         early_weights, partials, counters, status);
    if (le != cudaSuccess) return dl_fail(DL_ERR_LAUNCH, "gemm_skinny: %s", cudaGetErrorString(le));
    return DL_OK;
}

template <int NT, typename TOut, bool FUSE, int TILES, int BK>
static int gs_launch_rows_of(const GsRowsPlan& p, cudaStream_t s, const __nv_bfloat16* x, int x_stride, const __nv_bfloat16* w, void* out, int out_stride, int M,
                          int N, int K, int early_weights, int* status, const GsFuse& fuse) {
    const int cpt = (K + BK - 1) / BK;
    const int a_warp = (p.passes * cpt + GS_CONSUMERS - 1) / GS_CONSUMERS;     // the busiest warp's chunks: no stages beyond them
    const int a_pass = GS_CONSUMERS * TILES * NT * 512;      // bytes of a pass's sums
    auto stages = [&](int sums) {
        int slots = a_warp < GR_MAX_SLOTS ? a_warp : GR_MAX_SLOTS;
        while (slots > 1 && GR_ring_bytes(p.rows, slots, FUSE, TILES, BK) + sums * a_pass > GR_SMEM) --slots;
        return slots;
    };
    // Sums of two passes, unless that leaves the rings a single stage where one pass's leave two (48 rows and 16 tokens: 128,256 x 2,048 of 10 rows
    // 95.7 us with one stage, 80 with two).
    const int sums = p.passes > 1 && (stages(2) > 1 || stages(1) == 1) ? 2 : 1, slots = stages(sums);
    const int smem = GR_ring_bytes(p.rows, slots, FUSE, TILES, BK) + sums * a_pass;
    static std::atomic<unsigned long long> sized{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess && (dev >= 64 || !(sized.load() >> dev & 1))) {
        e = cudaFuncSetAttribute(gemm_skinny_rows_kernel<NT, TOut, FUSE, TILES, BK>, cudaFuncAttributeMaxDynamicSharedMemorySize, GR_SMEM);
        if (e == cudaSuccess && dev < 64) sized.fetch_or(1ull << dev);
    }
    if (e != cudaSuccess) return dl_fail(DL_ERR_LAUNCH, "gemm_skinny: shared memory %d: %s", smem, cudaGetErrorString(e));
    CUtensorMap tmap;
    const int rc = gs_weight_map(&tmap, w, FUSE ? 2 * N : N, K, p.rows, BK);
    if (rc != DL_OK) return rc;
    const GsRowsWork work{x, x_stride, out, out_stride, M, N, K, N, cpt, p.block_rows, p.rows, p.passes, slots, sums, fuse};
    e = dl_launch_dependent(gemm_skinny_rows_kernel<NT, TOut, FUSE, TILES, BK>, dim3(p.blocks), dim3(GR_THREADS(TILES)), (size_t)smem, s, tmap, work, early_weights, status);
    if (e != cudaSuccess) return dl_fail(DL_ERR_LAUNCH, "gemm_skinny: %s", cudaGetErrorString(e));
    return DL_OK;
}

template <int NT, typename TOut, bool FUSE>
static int gs_launch_rows(int sms, cudaStream_t s, const __nv_bfloat16* x, int x_stride, const __nv_bfloat16* w, void* out, int out_stride, int M,
                          int N, int K, int early_weights, int* status, const GsFuse& fuse) {
    const GsRowsPlan p = gs_rows_plan(N, FUSE, sms);
#define GR_OF(TILES, BK) gs_launch_rows_of<NT, TOut, FUSE, TILES, BK>(p, s, x, x_stride, w, out, out_stride, M, N, K, early_weights, status, fuse)
    const int tiles = (p.rows + (FUSE ? 7 : 15)) / (FUSE ? 8 : 16);
    if (tiles == 1) return GR_OF(1, 256);
    if (FUSE || tiles == 2) return GR_OF(2, 128);
    if constexpr (!FUSE) return GR_OF(3, 128);
#undef GR_OF
}

// x: bf16 [M, K] rows x_stride apart, M <= 16.  w: bf16, contiguous rows of K.
// flags bit 0 (gated) clear: w is [N, K], out [M, N].  Set: w is [2N, K] (N gate rows, then N up
// rows), out [M, N] = silu(x Wg^T) * (x Wu^T).
// flags bit 1 (resident weights): the caller vouches that nothing still pending on the stream
// writes w, so the kernel may start reading w before the kernel launched before it has finished.
// partials / counters: scratch of the sizes dl_gemm_skinny_scratch gives; status: int32, set
// non-zero if a wait expired.
static int gs_run(const void* x, int x_stride, const void* w, void* out, int out_dtype, int out_stride, int M, int N, int K,
                  int flags, float* partials, int partial_floats, int* counters, int n_counters, int* status, void* stream,
                  const GsFuse& fuse) {
    const int fuse_swiglu = flags & 1, early = (flags >> 1) & 1;
    DL_REQUIRE((flags & ~3) == 0, "gemm_skinny: unknown flags %d", flags);
    DL_REQUIRE(M >= 1 && M <= GS_MAX_ROWS, "gemm_skinny: takes 1 to %d rows, got %d", GS_MAX_ROWS, M);
    DL_REQUIRE(N > 0 && K > 0 && K % 8 == 0, "gemm_skinny: K=%d must be a positive multiple of 8", K);
    DL_REQUIRE(x_stride % 8 == 0 && x_stride >= K, "gemm_skinny: row stride of x (%d) must be a multiple of 8", x_stride);
    DL_REQUIRE(((uintptr_t)x % 16) == 0 && ((uintptr_t)w % 16) == 0, "gemm_skinny: x and W must be 16-byte aligned");
    DL_REQUIRE(out_stride >= N, "gemm_skinny: out stride shorter than N");
    DL_REQUIRE(out_dtype == DL_F32 || out_dtype == DL_BF16, "gemm_skinny: out dtype %d", out_dtype);
    DL_REQUIRE(status != nullptr && partials != nullptr && counters != nullptr, "gemm_skinny: needs scratch and a status word");
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return dl_fail(DL_ERR_LAUNCH, "gemm_skinny: cannot query the device");
    const int nt = M <= 8 ? 1 : 2;
    if (gs_by_rows(N, K, fuse_swiglu != 0, sms)) {
        cudaStream_t s = (cudaStream_t)stream;
        const __nv_bfloat16 *xb = (const __nv_bfloat16*)x, *wb = (const __nv_bfloat16*)w;
#define GR_CASE(NTV)                                                                                                                               \
    if (nt == NTV) {                                                                                                                               \
        if (fuse_swiglu && out_dtype == DL_F32) return gs_launch_rows<NTV, float, true>(sms, s, xb, x_stride, wb, out, out_stride, M, N, K, early, status, fuse);        \
        if (fuse_swiglu) return gs_launch_rows<NTV, __nv_bfloat16, true>(sms, s, xb, x_stride, wb, out, out_stride, M, N, K, early, status, fuse); \
        if (out_dtype == DL_F32) return gs_launch_rows<NTV, float, false>(sms, s, xb, x_stride, wb, out, out_stride, M, N, K, early, status, fuse); \
        return gs_launch_rows<NTV, __nv_bfloat16, false>(sms, s, xb, x_stride, wb, out, out_stride, M, N, K, early, status, fuse);                 \
    }
        GR_CASE(1) GR_CASE(2)
#undef GR_CASE
    }
    const GsPlan p = gs_plan(N, K, fuse_swiglu, sms);
    DL_REQUIRE(partial_floats >= p.blocks * GS_CONSUMERS * 2 * nt * 4 * 32 && n_counters >= p.tiles,
               "gemm_skinny: scratch too small (%d floats, %d counters)", partial_floats, n_counters);
    cudaStream_t s = (cudaStream_t)stream;
    const __nv_bfloat16* xb = (const __nv_bfloat16*)x;
    const __nv_bfloat16* wb = (const __nv_bfloat16*)w;
#define GS_CASE(NTV)                                                                                                   \
    if (nt == NTV) {                                                                                                   \
        if (fuse_swiglu) {                                                                                             \
            if (out_dtype == DL_F32) return gs_launch<NTV, float, true>(p, s, xb, x_stride, wb, out, out_stride, M, N, K, N, early, partials, counters, status, fuse); \
            return gs_launch<NTV, __nv_bfloat16, true>(p, s, xb, x_stride, wb, out, out_stride, M, N, K, N, early, partials, counters, status, fuse);                \
        }                                                                                                              \
        if (out_dtype == DL_F32) return gs_launch<NTV, float, false>(p, s, xb, x_stride, wb, out, out_stride, M, N, K, 0, early, partials, counters, status, fuse);    \
        return gs_launch<NTV, __nv_bfloat16, false>(p, s, xb, x_stride, wb, out, out_stride, M, N, K, 0, early, partials, counters, status, fuse);                   \
    }
    GS_CASE(1) GS_CASE(2)
#undef GS_CASE
    return dl_fail(DL_ERR_UNSUPPORTED, "gemm_skinny: %d rows", M);
}

extern "C" int dl_gemm_skinny_bf16(const void* x, int x_stride, const void* w, void* out, int out_dtype,
                                   int out_stride, int M, int N, int K, int flags, float* partials,
                                   int partial_floats, int* counters, int n_counters, int* status, void* stream) {
    return gs_run(x, x_stride, w, out, out_dtype, out_stride, M, N, K, flags, partials, partial_floats, counters, n_counters,
                  status, stream, GsFuse{});
}

// The gated product with another gating than SwiGLU (gating.cuh) in its epilogue; arguments as dl_gemm_skinny_bf16
// with the gated flag set.  With a `gate_kind` that is an activation of ONE product (relu^2) the gated flag is clear,
// w is [N, K] and out = act(x W^T).  bias: float32 [2N] (the gate rows', then the up rows') or NULL, added before the gating.
extern "C" int dl_gemm_skinny_gated_bf16(const void* x, int x_stride, const void* w, void* out, int out_dtype,
                                         int out_stride, int M, int N, int K, int flags, int gate_kind, float limit, float alpha,
                                         const float* bias, float* partials, int partial_floats, int* counters, int n_counters, int* status,
                                         void* stream) {
    DL_REQUIRE(gate_kind >= 0 && gate_kind < GATE_KINDS && ((flags & 1) == 1) == dl_gate_is_gated(gate_kind),
               "gemm_skinny_gated: a known gating, and the gated flag exactly where it reads two products");
    DL_REQUIRE(bias == nullptr || (flags & 1) == 1, "gemm_skinny_gated: biases go with two products");
    GsFuse fuse{};
    fuse.gate_kind = gate_kind, fuse.gate_limit = limit, fuse.gate_alpha = alpha, fuse.gate_bias = bias;
    return gs_run(x, x_stride, w, out, out_dtype, out_stride, M, N, K, flags, partials, partial_floats, counters, n_counters,
                  status, stream, fuse);
}

// The same with the fusions of an add + RMSNorm between two products (either, both or neither):
// gain set (float32 [N]; out must be float32 and the product plain): out is the float32 residual
//   stream and is added to in place; scaled bf16 [M, N] (rows scaled_stride apart) receives
//   out * gain, sumsq_out float32 [dl_gemm_skinny_parts(N, K) * 16] the sum of squares per tile and row.
// sumsq_in set (float32 [n_parts * 16], as a product before this one left it): every output row m
//   is multiplied by rsqrt(sum_p sumsq_in[p * 16 + m] / n + eps), n = 1 / inv_n the width of x's norm.
extern "C" int dl_gemm_skinny_fused_bf16(const void* x, int x_stride, const void* w, void* out, int out_dtype,
                                         int out_stride, int M, int N, int K, int flags, const float* gain, void* scaled,
                                         int scaled_stride, float* sumsq_out, const float* sumsq_in, int n_parts, float inv_n,
                                         float eps, float* partials, int partial_floats, int* counters, int n_counters,
                                         int* status, void* stream) {
    GsFuse fuse{};
    if (gain != nullptr) {
        DL_REQUIRE(out_dtype == DL_F32 && (flags & 1) == 0, "gemm_skinny: adding into the stream needs a plain float32 product");
        DL_REQUIRE(scaled != nullptr && sumsq_out != nullptr && scaled_stride >= N, "gemm_skinny: the scaled copy and the sums need a place");
        fuse.gain = gain, fuse.scaled = (__nv_bfloat16*)scaled, fuse.scaled_stride = scaled_stride, fuse.sumsq_out = sumsq_out;
    }
    if (sumsq_in != nullptr) {
        DL_REQUIRE(n_parts > 0 && inv_n > 0.f && eps >= 0.f, "gemm_skinny: row factors need parts, a width and an eps");
        fuse.sumsq_in = sumsq_in, fuse.n_parts = n_parts, fuse.inv_n = inv_n, fuse.eps = eps;
    }
    return gs_run(x, x_stride, w, out, out_dtype, out_stride, M, N, K, flags, partials, partial_floats, counters, n_counters,
                  status, stream, fuse);
}

// ---------------------------------------------------------------------------------------------
// The same product for callers that must not allocate (declared in gemm_skinny_static.h).
//
// dl_gemm_skinny_bf16 above takes its scratch from the caller, who normally gets it from an
// allocator.  Some callers have no allocator to ask: code that runs between a framework's
// allocation phases, a host process whose device memory is handed out once at start-up and then
// frozen, a real-time loop that may not take the allocator's lock.  For them the scratch lives in
// this library's own image: a file-scope __device__ array of a fixed, modest size that every GPU
// loading the library holds until the process exits.
//
// The array's name is only a host-side handle for the device object; its device address is asked
// for once per device, with that device current, through cudaGetSymbolAddress.
#include "gemm_skinny_static.h"

#define GS_STATIC_PARTIAL_FLOATS ((DL_GEMM_SKINNY_STATIC_SCRATCH_BYTES - 256) / 4 - DL_GEMM_SKINNY_STATIC_MAX_TILES)

struct GsStaticScratch {
    int status;
    int pad[63];
    int counters[DL_GEMM_SKINNY_STATIC_MAX_TILES];
    float partials[GS_STATIC_PARTIAL_FLOATS];
};
static __device__ __align__(256) GsStaticScratch gs_static_scratch;

#define GS_MAX_DEVICES 64
static GsStaticScratch* gs_static_ptr[GS_MAX_DEVICES];      // device address of the array, per device
static std::mutex gs_static_mutex;

// The device address of the scratch on the current device (looked up on the first call there).
static int gs_static_address(GsStaticScratch** out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return dl_fail(DL_ERR_LAUNCH, "gemm_skinny_static: cudaGetDevice: %s", cudaGetErrorString(e));
    if (dev < 0 || dev >= GS_MAX_DEVICES) return dl_fail(DL_ERR_UNSUPPORTED, "gemm_skinny_static: device %d out of range", dev);
    std::lock_guard<std::mutex> lock(gs_static_mutex);
    if (gs_static_ptr[dev] == nullptr) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, gs_static_scratch);
        if (e != cudaSuccess || p == nullptr)
            return dl_fail(DL_ERR_LAUNCH, "gemm_skinny_static: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
        gs_static_ptr[dev] = static_cast<GsStaticScratch*>(p);
    }
    *out = gs_static_ptr[dev];
    return DL_OK;
}

extern "C" int dl_gemm_skinny_bf16_static(const void* x, int x_stride, const void* w, void* out, int out_dtype,
                                          int out_stride, int M, int N, int K, int fuse_swiglu, void* stream) {
    DL_REQUIRE(M >= 1 && M <= GS_MAX_ROWS && N > 0 && K > 0, "gemm_skinny_static: bad sizes M=%d N=%d K=%d (1 to %d rows)", M, N,
               K, GS_MAX_ROWS);
    int sms = 0, dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return dl_fail(DL_ERR_LAUNCH, "gemm_skinny_static: cannot query the device");
    int need_floats = 0, need_counters = 0;
    dl_gemm_skinny_scratch(M, N, K, fuse_swiglu, sms, &need_floats, &need_counters);
    if (need_counters > DL_GEMM_SKINNY_STATIC_MAX_TILES || need_floats > (int)GS_STATIC_PARTIAL_FLOATS)
        return dl_fail(DL_ERR_UNSUPPORTED,
                       "gemm_skinny_static: M=%d N=%d K=%d needs %d row tiles and %d scratch floats; the built-in "
                       "scratch holds %d tiles and %d floats - use dl_gemm_skinny_bf16 with your own scratch",
                       M, N, K, need_counters, need_floats, DL_GEMM_SKINNY_STATIC_MAX_TILES, (int)GS_STATIC_PARTIAL_FLOATS);
    GsStaticScratch* scratch = nullptr;
    const int rc = gs_static_address(&scratch);
    if (rc != DL_OK) return rc;
    // The array keeps whatever the last call left; the arrival counters must start at zero.
    cudaError_t e = cudaMemsetAsync(scratch->counters, 0, sizeof(int) * need_counters, (cudaStream_t)stream);
    if (e != cudaSuccess) return dl_fail(DL_ERR_LAUNCH, "gemm_skinny_static: memset: %s", cudaGetErrorString(e));
    return dl_gemm_skinny_bf16(x, x_stride, w, out, out_dtype, out_stride, M, N, K, fuse_swiglu ? 1 : 0, scratch->partials,
                               need_floats, scratch->counters, need_counters, &scratch->status, stream);
}

// The give-up word of the static calls on the current device: copies it to *code (0: every wait so
// far was served) and clears it.  Waits for `stream` to drain, so that it speaks for every static
// call queued there before it; allocates nothing.
extern "C" int dl_gemm_skinny_static_status(int* code, void* stream) {
    DL_REQUIRE(code != nullptr, "gemm_skinny_static_status: needs a place for the code");
    GsStaticScratch* scratch = nullptr;
    const int rc = gs_static_address(&scratch);
    if (rc != DL_OK) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e = cudaMemcpyAsync(code, &scratch->status, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess && *code != 0) e = cudaMemsetAsync(&scratch->status, 0, sizeof(int), s);
    if (e != cudaSuccess) return dl_fail(DL_ERR_LAUNCH, "gemm_skinny_static_status: %s", cudaGetErrorString(e));
    return DL_OK;
}

DL_PACKED(dl_gemm_skinny_scratch)
DL_PACKED(dl_gemm_skinny_parts)
DL_PACKED(dl_gemm_skinny_plan)
DL_PACKED(dl_gemm_skinny_bf16)
DL_PACKED(dl_gemm_skinny_gated_bf16)
DL_PACKED(dl_gemm_skinny_fused_bf16)
