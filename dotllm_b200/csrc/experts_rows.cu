// Routed experts for steps of a few tokens (bfloat16), every chosen expert's matrices read once.
//
// The same results as expert_gate_up_kernel and expert_down_kernel (experts.cu), which read an expert's matrices once for every (token, choice) row
// that chose it.  Here every multiprocessor owns the same rows of every expert's matrix (as gemm_skinny.cu's products by rows, whose rings
// and tiles these are) and walks the list of experts that any row chose; an expert's (token, choice) rows are the columns of the
// tensor-core instruction.  A block makes the list for itself from the ids: experts in order, an expert's rows in order, at most 8 NT rows an
// entry (an expert of more has several entries).  Nothing passes between blocks, and k is cut the same way for every
// entry, so a row's result does not depend on what else is in the step.
//
// Sums keep the accuracy of float32 additions (GsTree in stream_rows.cuh): accumulators that live on in the tensor core left the down product's float32 results
// 1.3e-7 (rows of 1,408 values) to 1.8e-6 (14,336) off, relative to float64, where chains of multiply-adds row by row are 0.8e-7 to 1.3e-7 off; these
// are 0.8e-7 to 1.0e-7 off (rows of 704 to 1,408 values 1.02 to 1.05 of row by row's, longer ones 0.75 to 1), in the same time.
//
// The down product's block keeps its columns of every (token, choice) row in shared memory and at the end sums each token's choices in their order,
// with weights, identity experts and addend, as the kernel of experts.cu does.
//
// What bounds it: the bytes of the chosen experts' matrices, and for small experts about 1.25 us an entry and product (1.8 with 16 columns): a chain of
// the rows of x, a chunk's instructions and the hand-over of its sums.  Both products, against row by row: 8 tokens of 16 experts of 25 MB, two choices
// each (11 distinct) 84 -> 49 us (5.6 TB/s); 32 experts of 50 MB, four choices (about 21 distinct) 280 -> 151.  Which steps go this way: kernels/ops.py.
//
// Every wait on an mbarrier is bounded; on expiry the kernel records a code in `status` and returns after waiting (bounded) for copies in flight.
//
// Rings, hand-over and producer are gemm_skinny_rows_kernel's with entries around the passes: a change to a wait or to the release of a slot belongs in both.
#include "common.cuh"
#include "gating.cuh"
#include "stream_rows.cuh"
#include "tma.cuh"
#include <atomic>

#define XR_ROWS 128                        // (token, choice) rows of a step, at most
#define XR_EXPERTS 512                     // experts, at most
#define XR_Y 6144                          // float32 results of a block that wait in shared memory (down), at most
#define XR_SMEM 222208                     // bytes of shared memory for rings, sums and results: what a block can have less the lists

struct XrWork {
    const __nv_bfloat16* x;                // gate/up: [tokens, K]; down: h [rows, K]
    int x_stride;
    const int32_t* ids;
    int rows, top, E, K, N;                // N: pairs (gate/up) or output columns (down) of an expert
    int expert_rows;                       // rows of an expert in the stacked matrices: 2 N or N
    int cpt, block_rows, pass_rows, slots;
    int kind;                              // gate/up
    float limit, alpha;
    __nv_bfloat16* h;                      // gate/up: [rows, N]
    const float* weights;                  // down: as in dl_expert_down
    const float* addend;
    int addend_stride;
    float* out;
    const float* addend_gate;
    int addend_gate_stride;
    const __nv_bfloat16* identity;
    int identity_stride, n_identity;
};

struct XrLists {
    int id[XR_ROWS];                       // a row's expert, -1: none with matrices
    int order[XR_ROWS];                    // rows by expert
    int count[XR_EXPERTS], start[XR_EXPERTS];
    int expert[XR_ROWS], from[XR_ROWS], n[XR_ROWS];      // the entries: an expert, its first row in `order`, how many
    int entries;
};

// All threads of the block; ids are there.
template <int NT>
__device__ __forceinline__ void xr_make_lists(XrLists& l, const XrWork& w) {
    const int tid = threadIdx.x, lane = tid & 31;
    for (int e = tid; e < w.E; e += blockDim.x) l.count[e] = 0;
    for (int r = tid; r < w.rows; r += blockDim.x) {
        const int e = w.ids[r];
        l.id[r] = e >= 0 && e < w.E ? e : -1;
    }
    __syncthreads();
    int rank = 0;                                            // of row `tid` among its expert's (blocks have more threads than rows)
    const int e_mine = tid < w.rows ? l.id[tid] : -1;
    if (e_mine >= 0) {
        for (int r = 0; r < tid; ++r) rank += l.id[r] == e_mine ? 1 : 0;
        atomicAdd(&l.count[e_mine], 1);
    }
    __syncthreads();
    if (tid < 32) {
        int at = 0, entries = 0;
        for (int e0 = 0; e0 < w.E; e0 += 32) {
            const int c = e0 + lane < w.E ? l.count[e0 + lane] : 0, k = (c + 8 * NT - 1) / (8 * NT);
            int ci = c, ki = k;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int cu = __shfl_up_sync(0xffffffffu, ci, o), ku = __shfl_up_sync(0xffffffffu, ki, o);
                if (lane >= o) ci += cu, ki += ku;
            }
            if (e0 + lane < w.E) l.start[e0 + lane] = at + ci - c;
            for (int i = 0; i < k; ++i) {                    // (entries are at most as many as rows)
                const int to = entries + ki - k + i;
                l.expert[to] = e0 + lane, l.from[to] = at + ci - c + 8 * NT * i, l.n[to] = min(8 * NT, c - 8 * NT * i);
            }
            at += __shfl_sync(0xffffffffu, ci, 31), entries += __shfl_sync(0xffffffffu, ki, 31);
        }
        if (lane == 0) l.entries = entries;
    }
    __syncthreads();
    if (e_mine >= 0) l.order[l.start[e_mine] + rank] = tid;
    __syncthreads();
}

// A lane's values of an instruction's columns, 32 k from k0 on.
template <int NT>
__device__ __forceinline__ void xr_load_x(uint4 (&xf)[NT], const __nv_bfloat16* const (&rows)[NT], int K, int k0, int t) {
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        const int k = k0 + 8 * t;
        xf[j] = make_uint4(0u, 0u, 0u, 0u);
        if (rows[j] != nullptr && k < K) xf[j] = __ldg(reinterpret_cast<const uint4*>(rows[j] + k));
    }
}

// tmap: the experts' stacked matrices [E * expert_rows, K], boxes of pass_rows x BK.
template <int NT, bool DOWN, int TILES, int BK>
__global__ void __launch_bounds__(GR_THREADS(TILES), 1)
expert_rows_kernel(const __grid_constant__ CUtensorMap tmap, const XrWork w, int* __restrict__ status) {
    constexpr int TILE = DOWN ? 16 : 8;                      // rows (pairs) of a tile
    // The next chunk's values of x are asked for before this one's arithmetic, into registers of their own; where that would spill (two groups of
    // columns and chunks of 256), behind every step into the registers that it has left, which asks a little later (5 to 10 % slower where both fit).
    constexpr bool IN_PLACE = NT == 2 && BK == 256;
    extern __shared__ __align__(128) unsigned char xr_smem[];
    __shared__ uint64_t full_bar[GS_CONSUMERS][GR_MAX_SLOTS], empty_bar[GS_CONSUMERS][GR_MAX_SLOTS], sums_full[2], sums_empty[2];
    __shared__ volatile int gave_up;
    __shared__ XrLists l;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    if (threadIdx.x == 0) {
        gave_up = 0;
        for (int h = 0; h < 2; ++h) gs_mbar_init(&sums_full[h], GS_CONSUMERS), gs_mbar_init(&sums_empty[h], TILES);
        for (int c = 0; c < GS_CONSUMERS; ++c)
            for (int s = 0; s < w.slots; ++s) {
                gs_mbar_init(&full_bar[c][s], 1);
                gs_mbar_init(&empty_bar[c][s], 1);
            }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    dl_launch_dependents();
    dl_grid_dependency_wait();                               // which matrices are read is what the kernels before this one decided
    __syncthreads();
    xr_make_lists<NT>(l, w);
    const int first = blockIdx.x * w.block_rows, end_row = min(w.N, first + w.block_rows);      // this block's rows of every expert
    const int passes = (end_row - first + w.pass_rows - 1) / w.pass_rows, chunks = passes * w.cpt, entries = l.entries;
    const uint32_t box_bytes = w.pass_rows * (BK * 2), stage_bytes = GR_stage_rows(w.pass_rows, !DOWN, TILES) * (BK * 2);
    float4* sums = reinterpret_cast<float4*>(xr_smem + GR_ring_bytes(w.pass_rows, w.slots, !DOWN, TILES, BK));      // [2][warp][tile][NT][lane]
    float* y = reinterpret_cast<float*>(sums + 2 * GS_CONSUMERS * TILES * NT * 32);              // [rows][block_rows], down
    if (warp < GS_CONSUMERS) {
        // ------------------------------------------------------------ consumer warp: chunks warp, warp + 8, ... of every entry
        uint4 xf[BK / 32][NT];
        const __nv_bfloat16* xr[NT];
        auto rows_of = [&](int d) {
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                const int i = j * 8 + g;
                xr[j] = nullptr;
                if (d < entries && i < l.n[d]) {
                    const int r = l.order[l.from[d] + i];
                    xr[j] = w.x + (size_t)(DOWN ? r : r / w.top) * w.x_stride;
                }
            }
        };
        int slot = 0, phase = 0;
        bool dead = false;
        auto gave = [&](int code) {
            if (!gave_up) atomicExch(status, code);
            gave_up = 1;
            dead = true;
        };
        rows_of(0);
        if (warp < chunks) {
#pragma unroll
            for (int s = 0; s < BK / 32; ++s) xr_load_x<NT>(xf[s], xr, w.K, (warp % w.cpt) * BK + 32 * s, t);
        }
        const int tiles = (w.pass_rows + TILE - 1) / TILE;
        for (int d = 0, q = 0; d < entries; ++d) {
            int cur = warp;
            for (int p = 0; p < passes; ++p, ++q) {
                float acc[TILES][NT][4];
#pragma unroll
                for (int i = 0; i < TILES; ++i)
#pragma unroll
                    for (int j = 0; j < NT; ++j)
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
                for (const int pass_end = (p + 1) * w.cpt; cur < pass_end; cur += GS_CONSUMERS) {
                    if (!dead && !gs_mbar_wait(&full_bar[warp][slot], phase, &gave_up)) gave(3);
                    int next = cur + GS_CONSUMERS;
                    if (next >= chunks) rows_of(d + 1), next = warp;
                    next = (next % w.cpt) * BK;
                    uint4 xn[IN_PLACE ? 1 : BK / 32][NT];
                    if (!IN_PLACE)
#pragma unroll
                        for (int s = 0; s < BK / 32; ++s) xr_load_x<NT>(xn[IN_PLACE ? 0 : s], xr, w.K, next + 32 * s, t);
                    if (!dead) {
                        // rows beyond the box are whatever lies behind it: they reach results that are not stored
                        const uint32_t st = gs_smem(xr_smem + (size_t)(warp * w.slots + slot) * stage_bytes) + (uint32_t)(g * BK + 8 * t) * 2u;
#pragma unroll
                        for (int i = 0; i < TILES; ++i) {
                            if (i >= tiles) break;
                            GsTree<BK / 32> tree[NT];
#pragma unroll
                            for (int s = 0; s < BK / 32; ++s) {
                                const uint4 a_lo = gs_lds128(st + (uint32_t)((TILE * i * BK + 32 * s) * 2));
                                const uint4 a_hi = gs_lds128(st + (uint32_t)(((DOWN ? TILE * i + 8 : TILE * TILES + TILE * i) * BK + 32 * s) * 2));
#pragma unroll
                                for (int j = 0; j < NT; ++j) tree[j].add(s, acc[i][j], a_lo, a_hi, xf[s][j]);
                                if (IN_PLACE && i == tiles - 1) xr_load_x<NT>(xf[s], xr, w.K, next + 32 * s, t);
                            }
                        }
                        // the slot is released when every read of it is done (gs_consume in gemm_skinny.cu)
#pragma unroll
                        for (int i = 0; i < TILES; ++i)
#pragma unroll
                            for (int j = 0; j < NT; ++j)
                                asm volatile("" : "+f"(acc[i][j][0]), "+f"(acc[i][j][1]), "+f"(acc[i][j][2]), "+f"(acc[i][j][3]));
                        __threadfence_block();
                        __syncwarp();
                        if (lane == 0) gs_mbar_arrive(&empty_bar[warp][slot]);
                    }
                    if (++slot == w.slots) slot = 0, phase ^= 1;
                    if (!IN_PLACE)
#pragma unroll
                        for (int s = 0; s < BK / 32; ++s)
#pragma unroll
                            for (int j = 0; j < NT; ++j) xf[s][j] = xn[IN_PLACE ? 0 : s][j];
                }
                const int h = q & 1;
                if (q >= 2 && !dead && !gs_mbar_wait(&sums_empty[h], ((q >> 1) - 1) & 1, &gave_up)) gave(6);
                float4* mine = sums + (size_t)(h * GS_CONSUMERS + warp) * TILES * NT * 32 + lane;
                if (!dead) {
#pragma unroll
                    for (int i = 0; i < TILES; ++i)
#pragma unroll
                        for (int j = 0; j < NT; ++j) mine[(i * NT + j) * 32] = make_float4(acc[i][j][0], acc[i][j][1], acc[i][j][2], acc[i][j][3]);
                }
                __threadfence_block();
                __syncwarp();
                if (lane == 0) gs_mbar_arrive(&sums_full[h]);
            }
        }
    } else if (warp == GS_CONSUMERS) {
        // ------------------------------------------------------------ producer warp: lane c serves consumer warp c
        if (lane < GS_CONSUMERS) {
            const uint64_t policy = dl_stream_policy();
            int cnt = 0, cur = lane, slot = 0, phase = 1, d = lane < chunks ? 0 : entries;
            bool ok = true;
            long long t0 = clock64();
            while (d < entries) {
                if (cnt < w.slots || gs_mbar_try(&empty_bar[lane][slot], phase)) {
                    const int pass = cur / w.cpt, kc = cur - pass * w.cpt, row = l.expert[d] * w.expert_rows + first + pass * w.pass_rows;
                    unsigned char* dst = xr_smem + (size_t)(lane * w.slots + slot) * stage_bytes;
                    gs_mbar_expect(&full_bar[lane][slot], DOWN ? box_bytes : 2 * box_bytes);
                    dl_tma_load_2d_hint(dst, &tmap, kc * BK, row, &full_bar[lane][slot], policy);
                    if (!DOWN) dl_tma_load_2d_hint(dst + TILES * TILE * BK * 2, &tmap, kc * BK, w.N + row, &full_bar[lane][slot], policy);
                    cur += GS_CONSUMERS, ++cnt;
                    if (cur >= chunks) cur = lane, ++d;
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
        // ------------------------------------------------------------ adding warps: one a tile of a pass
        const int tile = warp - GS_CONSUMERS - 1, mine = tile * 32 + lane, n_cols = end_row - first;
        if (!DOWN)                                           // rows without an expert
            for (int r = 0; r < w.rows; ++r)
                if (l.id[r] < 0)
                    for (int c = mine; c < n_cols; c += 32 * TILES) w.h[(size_t)r * w.N + first + c] = __float2bfloat16_rn(0.f);
        bool dead = false;
        for (int d = 0, q = 0; d < entries && !dead; ++d)
            for (int p = 0; p < passes && !dead; ++p, ++q) {
                const int h = q & 1, pass_end = min(end_row, first + (p + 1) * w.pass_rows), base = first + p * w.pass_rows + tile * TILE;
                if (!gs_mbar_wait(&sums_full[h], (q >> 1) & 1, &gave_up)) {
                    if (!gave_up) atomicExch(status, 5);
                    gave_up = 1;
                    dead = true;
                    continue;
                }
                float acc[NT][4];
                const float4* theirs = sums + (size_t)(h * GS_CONSUMERS * TILES + tile) * NT * 32 + lane;
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    float4 v[GS_CONSUMERS];
#pragma unroll
                    for (int c = 0; c < GS_CONSUMERS; ++c) v[c] = theirs[(c * TILES * NT + j) * 32];
#pragma unroll
                    for (int half = GS_CONSUMERS / 2; half > 0; half /= 2)
#pragma unroll
                        for (int c = 0; c < half; ++c) v[c].x += v[c + half].x, v[c].y += v[c + half].y, v[c].z += v[c + half].z, v[c].w += v[c + half].w;
                    acc[j][0] = v[0].x, acc[j][1] = v[0].y, acc[j][2] = v[0].z, acc[j][3] = v[0].w;
                }
                __syncwarp();
                if (lane == 0) gs_mbar_arrive(&sums_empty[h]);
#pragma unroll
                for (int j = 0; j < NT; ++j)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int i = j * 8 + 2 * t + e;
                        if (i >= l.n[d]) continue;
                        const int r = l.order[l.from[d] + i];
                        if (DOWN) {
                            if (base + g < pass_end) y[r * w.block_rows + base + g - first] = acc[j][e];
                            if (base + g + 8 < pass_end) y[r * w.block_rows + base + g + 8 - first] = acc[j][2 + e];
                        } else if (base + g < pass_end) {
                            w.h[(size_t)r * w.N + base + g] = __float2bfloat16_rn(dl_gate_value(w.kind, acc[j][e], acc[j][2 + e], w.limit, w.alpha));
                        }
                    }
            }
        if (DOWN) {
            asm volatile("bar.sync 1, %0;" ::"n"(32 * TILES) : "memory");        // every column of every row is there
            const int tokens = w.rows / w.top;
            for (int i = mine; i < tokens * n_cols && !gave_up; i += 32 * TILES) {
                const int token = i / n_cols, c = i - token * n_cols, n = first + c;
                float total = 0.f;
                for (int j = 0; j < w.top; ++j) {
                    const int r = token * w.top + j, e = l.id[r];
                    const float weight = w.weights != nullptr ? w.weights[r] : 1.0f;
                    if (e >= 0) total += weight * y[r * w.block_rows + c];
                    else if (w.identity != nullptr && w.ids[r] >= w.E && w.ids[r] < w.E + w.n_identity)
                        total += weight * __bfloat162float(w.identity[(size_t)token * w.identity_stride + n]);
                }
                if (w.addend != nullptr) {
                    const float ag = w.addend_gate != nullptr ? 1.0f / (1.0f + expf(-w.addend_gate[(size_t)token * w.addend_gate_stride])) : 1.0f;
                    total += ag * w.addend[(size_t)token * w.addend_stride + n];
                }
                w.out[(size_t)token * w.N + n] = total;
            }
        }
    }
    __syncthreads();                                         // nobody leaves while copies may still land
}

template <int NT, bool DOWN, int TILES, int BK>
static cudaError_t xr_launch(XrWork& w, const GsRowsPlan& p, const void* matrices, int* status, cudaStream_t s) {
    w.cpt = (w.K + BK - 1) / BK;
    const int fixed = 2 * GS_CONSUMERS * TILES * NT * 512 + (DOWN ? w.rows * p.block_rows * 4 : 0);
    w.slots = GR_MAX_SLOTS;
    while (w.slots > 1 && GR_ring_bytes(p.rows, w.slots, !DOWN, TILES, BK) + fixed > XR_SMEM) --w.slots;
    const int smem = GR_ring_bytes(p.rows, w.slots, !DOWN, TILES, BK) + fixed;
    static std::atomic<unsigned long long> sized{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess && (dev >= 64 || !(sized.load() >> dev & 1))) {
        e = cudaFuncSetAttribute(expert_rows_kernel<NT, DOWN, TILES, BK>, cudaFuncAttributeMaxDynamicSharedMemorySize, XR_SMEM);
        if (e == cudaSuccess && dev < 64) sized.fetch_or(1ull << dev);
    }
    if (e != cudaSuccess) return e;
    CUtensorMap tmap;
    if (dl_tmap_cached_2d_bf16(&tmap, matrices, (unsigned long long)w.E * w.expert_rows, w.K, (unsigned long long)w.K * 2, p.rows, BK,
                               DL_TMAP_SWIZZLE_NONE) != 0)
        return cudaErrorInvalidValue;
    return dl_launch_dependent(expert_rows_kernel<NT, DOWN, TILES, BK>, dim3(p.blocks), dim3(GR_THREADS(TILES)), (size_t)smem, s, tmap, w, status);
}

template <int NT, bool DOWN>
static cudaError_t xr_launch(XrWork& w, const void* matrices, int* status, cudaStream_t s) {
    const GsRowsPlan p = gs_rows_plan(w.N, !DOWN, dl_sm_count());
    w.block_rows = p.block_rows, w.pass_rows = p.rows;
    const int tiles = (p.rows + (DOWN ? 15 : 7)) / (DOWN ? 16 : 8);
    if (tiles == 1) return xr_launch<NT, DOWN, 1, 256>(w, p, matrices, status, s);
    if (!DOWN || tiles == 2) return xr_launch<NT, DOWN, 2, 128>(w, p, matrices, status, s);
    if constexpr (DOWN) return xr_launch<NT, DOWN, 3, 128>(w, p, matrices, status, s);
    return cudaErrorInvalidValue;
}

#define XR_CHECK(what, width)                                                                                                                   \
    DL_REQUIRE(tokens >= 0 && top > 0 && K > 0 && (width) > 0 && E > 0, what ": bad sizes");                                                    \
    DL_REQUIRE(tokens <= 16 && (long long)tokens * top <= XR_ROWS && E <= XR_EXPERTS, what ": %d tokens of %d choices among %d experts", tokens, top, E); \
    DL_REQUIRE(K % 8 == 0 && ((uintptr_t)w % 16) == 0 && status != nullptr, what ": rows of a multiple of 8 values, 16-byte aligned")

// Arguments as dl_expert_gate_up for bfloat16 and gatings of two products, without a row scale; x's rows 16-byte aligned.  status: int32, set
// non-zero if a wait expired.
extern "C" int dl_expert_gate_up_rows(const void* x, int x_stride, const int32_t* ids, const void* w, void* out, int tokens, int top, int K, int ff,
                                      int E, int kind, float limit, float alpha, int* status, void* stream) {
    XR_CHECK("expert_gate_up_rows", ff);
    DL_REQUIRE(kind >= 0 && kind < GATE_KINDS && dl_gate_is_gated(kind) && x_stride >= K && x_stride % 8 == 0 && ((uintptr_t)x % 16) == 0,
               "expert_gate_up_rows: a gating of two products, rows of x 16-byte aligned");
    if (tokens == 0) return DL_OK;
    XrWork k{};
    k.x = (const __nv_bfloat16*)x, k.x_stride = x_stride, k.ids = ids, k.rows = tokens * top, k.top = top, k.E = E, k.K = K, k.N = ff;
    k.expert_rows = 2 * ff, k.kind = kind, k.limit = limit, k.alpha = alpha, k.h = (__nv_bfloat16*)out;
    const cudaError_t e = tokens <= 8 ? xr_launch<1, false>(k, w, status, (cudaStream_t)stream) : xr_launch<2, false>(k, w, status, (cudaStream_t)stream);
    if (e != cudaSuccess) return dl_fail(DL_ERR_LAUNCH, "expert_gate_up_rows: %s", cudaGetErrorString(e));
    return DL_OK;
}

// May the down product of these sizes go by rows?  (Its block keeps its columns of every row in shared memory.)
extern "C" int dl_expert_down_rows_takes(int rows, int N) { return (long long)rows * ((N + dl_sm_count() - 1) / dl_sm_count()) <= XR_Y ? 1 : 0; }

// Arguments as dl_expert_down for bfloat16, h's address a multiple of 16 bytes.
extern "C" int dl_expert_down_rows(const void* h, const int32_t* ids, const float* weights, const void* w, const float* addend, int addend_stride,
                                   float* out, int tokens, int top, int ff, int N, int E, const float* addend_gate, int addend_gate_stride,
                                   const void* identity, int identity_stride, int n_identity, int* status, void* stream) {
    const int K = ff;
    XR_CHECK("expert_down_rows", N);
    DL_REQUIRE(identity == nullptr || (n_identity > 0 && identity_stride >= N), "expert_down_rows: identity experts give back rows of the output's width");
    DL_REQUIRE(((uintptr_t)h % 16) == 0 && dl_expert_down_rows_takes(tokens * top, N), "expert_down_rows: %d rows of %d columns", tokens * top, N);
    if (tokens == 0) return DL_OK;
    XrWork k{};
    k.x = (const __nv_bfloat16*)h, k.x_stride = ff, k.ids = ids, k.rows = tokens * top, k.top = top, k.E = E, k.K = K, k.N = N, k.expert_rows = N;
    k.weights = weights, k.addend = addend, k.addend_stride = addend_stride, k.out = out, k.addend_gate = addend_gate;
    k.addend_gate_stride = addend_gate_stride, k.identity = (const __nv_bfloat16*)identity, k.identity_stride = identity_stride, k.n_identity = n_identity;
    const cudaError_t e = tokens <= 8 ? xr_launch<1, true>(k, w, status, (cudaStream_t)stream) : xr_launch<2, true>(k, w, status, (cudaStream_t)stream);
    if (e != cudaSuccess) return dl_fail(DL_ERR_LAUNCH, "expert_down_rows: %s", cudaGetErrorString(e));
    return DL_OK;
}

DL_PACKED(dl_expert_gate_up_rows)
DL_PACKED(dl_expert_down_rows_takes)
DL_PACKED(dl_expert_down_rows)
