// Routed experts over many tokens: every expert runs for the tokens that chose it and for no others.
//
// The tokens of each expert are gathered into rows of their own (row tiles of 128, so that no tile holds two experts),
// the gated product of a row tile with its expert's weights leaves the hidden activations, already multiplied by the
// token's weight for that expert, the down product stores each row's result, and a token's few results are added up in
// the order of the experts and then to its row of the output: in one order, so that the same step gives the same bits.
// A further expert may take every token with weight one (the shared expert); it is one more segment of rows, the tokens
// as they lie, with hidden activations of its own size, whose results go to the output at once (one per element of it,
// before the others).
// How many rows each expert has is known on the device only: the products walk a list of tiles that every CTA derives
// from the counts, and the grids depend on the host's bounds alone, so a step with experts has no host decision.
//
//   expert_list_kernel    a block per expert: the tokens that chose it, in order, and their number
//   expert_gather_kernel  rows of the input side by side, expert after expert; token and weight of every row, and the rows
//                         of every token
//   expert_gemm_kernel    persistent tcgen05 product over the list of tiles, gated (up) or storing float32 rows (down)
//   expert_sum_kernel     a block per token: its rows into the output
//
// Before, every token passed through every expert: 2048 tokens, width 2048, 8 experts of 2048 and a shared one, 2 chosen,
// B200: gated product 230 us, scaling of the hidden values about 25, down product 117; now list 6, gather 9, gated product
// 79 (1.3 PFLOP/s, bound by the tensor cores with their last wave), down product 54 (0.96 PFLOP/s; its epilogue writes 50 MB of
// float32 in 16-byte pieces), sums 12. The whole feed-forward: 443 -> 217 us. Adding into the tokens' rows with atomics instead
// takes 11 us less, in an order that changes from run to run.
//
// Every wait on an mbarrier is bounded, as in gemm_tcgen05.cu.
#include "tcgen05_utils.cuh"

namespace {

constexpr int ROWS = 128;            // rows of a tile = MMA M
constexpr int COLS = 256;            // weight rows of a tile = MMA N: 128 gated features, or 256 plain ones
constexpr int UMMA_K = 16;
constexpr int MAX_EXPERTS = 256;

// ---------------------------------------------------------------- which tokens chose which expert
// weights [T, ldw]: a token's weight per expert, zero where it did not choose it. list[e * T ..]: the tokens of expert e.
// place[e * T + t] becomes -1: no row yet.
__global__ void __launch_bounds__(1024)
expert_list_kernel(const float* __restrict__ weights, int ldw, int T, int* __restrict__ counts, int* __restrict__ list,
                   int* __restrict__ place) {
    __shared__ int warp_count[32];
    lp_grid_release();
    lp_grid_wait();
    const int e = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int base = 0;
    for (int t0 = 0; t0 < T; t0 += 1024) {
        const int t = t0 + threadIdx.x;
        const bool chosen = t < T && !(weights[(long long)t * ldw + e] == 0.f);     // a weight that is no number counts as chosen
        const unsigned votes = __ballot_sync(0xffffffffu, chosen);
        if (t < T) place[(long long)e * T + t] = -1;
        __syncthreads();
        if (lane == 0) warp_count[warp] = __popc(votes);
        __syncthreads();
        int before = base, all = 0;
#pragma unroll
        for (int w = 0; w < 32; ++w) {
            const int c = warp_count[w];
            if (w < warp) before += c;
            all += c;
        }
        if (chosen) list[(long long)e * T + before + __popc(votes & ((1u << lane) - 1u))] = t;
        base += all;
    }
    if (threadIdx.x == 0) counts[e] = base;
}

// First row of every routed expert's segment and the end, in `start` (E + 1 integers of shared memory). Called by all threads of a
// block. More choices than there is room for (weights that no router made) are cut off at the room and reported by the gather kernel.
__device__ __forceinline__ int segment_starts(const int* counts, int E, int room, int* start) {
    for (int e = threadIdx.x; e < E; e += blockDim.x) start[e + 1] = (counts[e] + ROWS - 1) / ROWS * ROWS;
    __syncthreads();
    if (threadIdx.x == 0) {
        start[0] = 0;
        for (int e = 0; e < E; ++e) start[e + 1] += start[e];
    }
    __syncthreads();
    const int end = start[E];
    if (end > room) {
        __syncthreads();
        for (int e = threadIdx.x; e < E + 1; e += blockDim.x) start[e] = min(start[e], room);
        __syncthreads();
    }
    return end;
}

// x [T, d] -> rows [R, d] (16 bytes per thread and step), row_token (-1: padding) and row_weight, and place [E, T]: the row
// of every token and expert that belong together. A block per four rows.
__global__ void __launch_bounds__(256)
expert_gather_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ weights, int ldw, const int* __restrict__ counts,
                     const int* __restrict__ list, int T, int d, int E, __nv_bfloat16* __restrict__ rows, int* __restrict__ row_token,
                     float* __restrict__ row_weight, int* __restrict__ place, int* __restrict__ status) {
    __shared__ int start[MAX_EXPERTS + 1];
    lp_grid_release();
    lp_grid_wait();
    const int room = gridDim.x * 4;
    if (segment_starts(counts, E, room, start) > room && blockIdx.x == 0 && threadIdx.x == 0) atomicExch(status, 55);
    const int r0 = blockIdx.x * 4;
    if (r0 >= start[E]) return;
    int e = 0;
    while (r0 >= start[e + 1]) ++e;                       // four rows never belong to two segments
    int token[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int at = r0 + i - start[e];
        token[i] = at < counts[e] ? list[(long long)e * T + at] : -1;
    }
    if (threadIdx.x < 4) {
        int mine = -1;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (threadIdx.x == i) mine = token[i];
        row_token[r0 + threadIdx.x] = mine;
        if (mine >= 0) place[(long long)e * T + mine] = r0 + threadIdx.x;
        row_weight[r0 + threadIdx.x] = mine < 0 ? 0.f : weights[(long long)mine * ldw + e];
    }
    for (int c = threadIdx.x * 8; c < d; c += 256 * 8) {
        uint4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = token[i] >= 0 ? *(const uint4*)(x + (long long)token[i] * d + c) : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int i = 0; i < 4; ++i) *(uint4*)(rows + (long long)(r0 + i) * d + c) = v[i];
    }
}

// ---------------------------------------------------------------- the products
constexpr int W_BYTES = COLS * BLOCK_K * 2, X_BYTES = ROWS * BLOCK_K * 2, STAGE_BYTES = W_BYTES + X_BYTES;
constexpr int STAGES = (196 * 1024) / STAGE_BYTES;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
constexpr int THREADS = 64 + 32 * 8;

struct Experts {
    const int* counts;
    const int* row_token;
    const float* row_weight;
    int E, shared_rows;          // routed experts; rows of the shared one (the tokens; 0: none)
    int ff, shared_ff;           // hidden size of a routed expert and of the shared one, multiples of 128
    int d;                       // width of the stream
    int room;                    // routed rows that the buffers hold
    int col0, cols;              // columns of the stream that the down product forms
};
// Where the shared expert's rows go: the hidden activations, or the stream.
struct Shared {
    void* at;                    // [T, ld]
    int ld, overwrite;
};
__device__ __forceinline__ void add4(float4* to, const float4& v) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(to), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

// UP: out[row, f] = silu(gate) * up * weight of the row, bfloat16; W is the interleaved gate / up matrix of all experts.
// Else: out[row, f] = hidden[row] . W[col0 + f, columns of the row's expert], float32, f < cols; the shared expert's rows go to
// the stream at col0 + f, added to it (the only addition to an element in this launch) or stored.
// map_x: the routed rows, map_s: the shared expert's.
// One CTA per SM walks the tiles (row tile first within an expert, so that the CTAs at work share weight tiles in L2) with
// two accumulators in tensor memory: one tile's epilogue runs under the next one's MMAs. Rows are the MMA's M, so a thread
// of the epilogue holds one row: its weight and its token are read once.
template <bool UP>
__global__ void __launch_bounds__(THREADS, 1)
expert_gemm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                   const __grid_constant__ CUtensorMap map_s, void* __restrict__ out, int ldo, Experts ex, Shared shared,
                   int* __restrict__ status) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ int start[MAX_EXPERTS + 1];           // first row of a routed expert's segment
    __shared__ int first_tile[MAX_EXPERTS + 2];      // first tile of a segment
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = (uint64_t*)(smem + STAGES * STAGE_BYTES);
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;             // [2]
    uint64_t* acc_empty = acc_full + 2;              // [2]
    uint32_t* tmem_slot = (uint32_t*)(acc_empty + 2);
    volatile uint32_t* failed = tmem_slot + 1;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    lp_grid_release();
    if (threadIdx.x == 0) {
        *failed = 0;
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_s) : "memory");
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int k = 0; k < 2; ++k) { mbar_init(&acc_full[k], 1); mbar_init(&acc_empty[k], 8); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    lp_grid_wait();
    segment_starts(ex.counts, ex.E, ex.room, start);
    auto row_tiles_of = [&](int e) { return e < ex.E ? (start[e + 1] - start[e]) / ROWS : (ex.shared_rows + ROWS - 1) / ROWS; };
    if (threadIdx.x == 0) {
        int at = 0;
        for (int e = 0; e <= ex.E; ++e) {
            first_tile[e] = at;
            const int cols = UP ? (e < ex.E ? ex.ff : ex.shared_ff) / 128 : (ex.cols + COLS - 1) / COLS;
            at += row_tiles_of(e) * cols;
        }
        first_tile[ex.E + 1] = at;
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const int num_tiles = first_tile[ex.E + 1];
    // tile -> (segment, column tile, first row: of the routed rows, or of the shared expert's)
    auto tile_at = [&](int tile, int& e, int& f, int& row0) {
        while (tile >= first_tile[e + 1]) ++e;       // tiles only grow, and so does e
        const int row_tiles = row_tiles_of(e), r = tile - first_tile[e];
        f = r / row_tiles;
        row0 = (e < ex.E ? start[e] : 0) + (r - f * row_tiles) * ROWS;
    };
    auto k_blocks_of = [&](int e) { return (UP ? ex.d + BLOCK_K - 1 : e < ex.E ? ex.ff : ex.shared_ff) / BLOCK_K; };

    if (warp == 0) {
        if (lane == 0) {
            int it = 0, e = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
                int f, row0;
                tile_at(tile, e, f, row0);
                const int k_blocks = k_blocks_of(e);
                const int w_row = UP ? 2 * e * ex.ff + f * COLS : ex.col0 + f * COLS, w_col = UP ? 0 : e * ex.ff;
                for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (!mbar_wait(&empty[s], ((it / STAGES) & 1) ^ 1)) { atomicExch(status, 51); *failed = 1; ok = false; break; }
                    uint8_t* stage = smem + s * STAGE_BYTES;
                    mbar_expect_tx(&full[s], STAGE_BYTES);
                    tma_load_2d(stage, &map_w, w_col + kb * BLOCK_K, w_row, &full[s]);
                    tma_load_2d(stage + W_BYTES, e < ex.E ? &map_x : &map_s, kb * BLOCK_K, row0, &full[s]);
                }
            }
            if (!ok) {
                for (int i = max(0, it - STAGES); i < it; ++i) mbar_wait(&full[i % STAGES], (i / STAGES) & 1);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc =
                (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(COLS >> 3) << 17) | ((uint32_t)(ROWS >> 4) << 24);
            int it = 0, j = 0, e = 0;
            bool ok = true;
            for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++j) {
                int f, row0;
                tile_at(tile, e, f, row0);
                const int k_blocks = k_blocks_of(e);
                const int ab = j & 1;
                if (!mbar_wait(&acc_empty[ab], ((j >> 1) & 1) ^ 1)) { atomicExch(status, 52); *failed = 1; ok = false; break; }
                tcgen05_fence_after();
                const uint32_t acc = tmem_base + ab * COLS;
                for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (!mbar_wait(&full[s], (it / STAGES) & 1)) { atomicExch(status, 53); *failed = 1; ok = false; break; }
                    tcgen05_fence_after();
                    const uint32_t w_addr = smem_u32(smem + s * STAGE_BYTES);
                    const uint64_t dw = smem_desc(w_addr), dx = smem_desc(w_addr + W_BYTES);
#pragma unroll
                    for (int k = 0; k < BLOCK_K / UMMA_K; ++k) {
                        const uint64_t step = (uint64_t)((k * UMMA_K * 2) >> 4);
                        tcgen05_mma(acc, dx + step, dw + step, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    }
                    tcgen05_commit(&empty[s]);
                }
                tcgen05_commit(&acc_full[ab]);
            }
        }
        __syncwarp();
    } else {
        const int quarter = warp & 3, ehalf = (warp - 2) >> 2;      // 32 rows of the tile; which half of the columns
        int j = 0, e = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x, ++j) {
            const int ab = j & 1;
            int f, row0;
            tile_at(tile, e, f, row0);
            const int row = row0 + quarter * 32 + lane;
            const bool routed = e < ex.E;
            const int token = routed ? ex.row_token[row] : row < ex.shared_rows ? row : -1;
            const float weight = !routed ? 1.f : UP ? ex.row_weight[row] : 0.f;
            void* to_rows = routed ? out : shared.at;
            const int ld = routed ? ldo : shared.ld;
            if (ok && !mbar_wait(&acc_full[ab], (j >> 1) & 1)) { if (lane == 0) atomicExch(status, 54); *failed = 1; ok = false; }
            tcgen05_fence_after();
            const bool go = __all_sync(0xffffffffu, ok && *failed == 0);
            const uint32_t lane_addr = tmem_base + ab * COLS + ((uint32_t)(quarter * 32) << 16);
            if (go && UP) {
                // columns 0..63 gate, 64..127 up of 64 features, 128..255 the same of the next 64
#pragma unroll 1
                for (int part = 2 * ehalf; part < 2 * ehalf + 2; ++part) {
                    const int half = part >> 1, c0 = (part & 1) * 32;
                    uint32_t g[32], u[32];
                    tmem_ld32(lane_addr + half * 128 + c0, g);
                    tmem_ld32(lane_addr + half * 128 + 64 + c0, u);
                    tmem_ld_wait();
                    uint32_t packed[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        float v[2];
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            const float gate = __uint_as_float(g[2 * i + k]);
                            v[k] = __fdividef(gate, 1.0f + __expf(-gate)) * __uint_as_float(u[2 * i + k]) * weight;
                        }
                        __nv_bfloat162 p = __floats2bfloat162_rn(v[0], v[1]);
                        packed[i] = *reinterpret_cast<uint32_t*>(&p);
                    }
                    if (token >= 0) {
                        uint4* to = reinterpret_cast<uint4*>((__nv_bfloat16*)to_rows + (size_t)row * ld + f * 128 + half * 64 + c0);
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            to[q] = make_uint4(packed[4 * q], packed[4 * q + 1], packed[4 * q + 2], packed[4 * q + 3]);
                    }
                }
            } else if (go) {
#pragma unroll 1
                for (int c0 = ehalf * (COLS / 2); c0 < (ehalf + 1) * (COLS / 2); c0 += 32) {
                    uint32_t g[32];
                    tmem_ld32(lane_addr + c0, g);
                    tmem_ld_wait();
                    const int f0 = f * COLS + c0;
                    if (token >= 0) {
                        float4* to = (float4*)((float*)to_rows + (size_t)row * ld + (routed ? 0 : ex.col0) + f0);
                        const bool adds = !routed && !shared.overwrite;
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            if (f0 + 4 * q >= ex.cols) break;          // (widths are multiples of 8)
                            const float4 v = make_float4(__uint_as_float(g[4 * q]), __uint_as_float(g[4 * q + 1]), __uint_as_float(g[4 * q + 2]),
                                                         __uint_as_float(g[4 * q + 3]));
                            if (adds) add4(to + q, v); else to[q] = v;
                        }
                    }
                }
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[ab])) : "memory");
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) {
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u));
    }
}

// out[t, col0 + c] (+)= the rows of token t, added in the order of the experts, c < cols. Bound by its bytes (the rows come from L2
// where they fit) and by the two reads that wait for one another.
template <bool OVERWRITE>
__global__ void __launch_bounds__(256)
expert_sum_kernel(const float* __restrict__ results, const int* __restrict__ place, int T, int E, float* __restrict__ out, int ldo, int col0,
                  int cols) {
    __shared__ int rows[MAX_EXPERTS];
    __shared__ int held;
    lp_grid_release();
    lp_grid_wait();
    const int t = blockIdx.x, lane = threadIdx.x & 31;
    if (threadIdx.x < 32) {
        int n = 0;
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int row = e0 + lane < E ? place[(long long)(e0 + lane) * T + t] : -1;
            const unsigned votes = __ballot_sync(0xffffffffu, row >= 0);
            if (row >= 0) rows[n + __popc(votes & ((1u << lane) - 1u))] = row;
            n += __popc(votes);
        }
        if (lane == 0) held = n;
    }
    __syncthreads();
    const int n = held;
    for (int c = threadIdx.x * 4; c < cols; c += 256 * 4) {
        float4* to = (float4*)(out + (size_t)t * ldo + col0 + c);
        const float4 old = OVERWRITE ? make_float4(0.f, 0.f, 0.f, 0.f) : *to;
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
        for (int i = 0; i < n; ++i) {
            const float4 v = *(const float4*)(results + (size_t)rows[i] * cols + c);
            sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
        }
        *to = OVERWRITE ? sum : make_float4(old.x + sum.x, old.y + sum.y, old.z + sum.z, old.w + sum.w);
    }
}

int failed_launch(cudaError_t err, const char* what) {
    snprintf(lp_error_text, sizeof(lp_error_text), "experts (%s): %s", what, cudaGetErrorString(err));
    return (int)err;
}

template <bool UP>
int launch_gemm(const CUtensorMap& mw, const CUtensorMap& mx, const CUtensorMap& ms, void* out, int ldo, const Experts& ex,
                const Shared& shared, int* status, cudaStream_t stream) {
    auto kernel = expert_gemm_kernel<UP>;
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        if (e != cudaSuccess) return failed_launch(e, "shared memory");
        configured = true;
    }
    const long long shared_tiles = (ex.shared_rows + ROWS - 1) / ROWS, cols = (ex.cols + COLS - 1) / COLS;
    const long long most_tiles = UP ? (long long)ex.room / ROWS * (ex.ff / 128) + shared_tiles * (ex.shared_ff / 128)
                                    : ((long long)ex.room / ROWS + shared_tiles) * cols;
    const int grid = most_tiles < lp_sm_count() ? (int)most_tiles : lp_sm_count();
    const cudaError_t err = lp_launch(kernel, dim3(grid), THREADS, SMEM_BYTES, stream, mw, mx, ms, out, ldo, ex, shared, status);
    return err == cudaSuccess ? lp_check_launch("experts (product)") : failed_launch(err, "product");
}

}  // namespace

// rows: the host's bound on the routed rows, a multiple of 128 (checked against T * top + ...: every expert's segment is rounded up
// to 128). x: bfloat16 [T, d]. weights: float32 [T, ldw], its first E columns. w_up: bfloat16 [2 * (E * ff + shared_ff), d], gate
// and up rows interleaved in blocks of 64. w_down: bfloat16 [d, E * ff + shared_ff]. Scratch: counts [E], list [E * T], place [E * T],
// gathered: 16-byte aligned, room for [rows, d] bfloat16 and, once those have been used, for [rows, slice] float32: the down product
// forms `slice` columns at a time (a multiple of 256, or d). hidden: [rows, ff] and behind it [T, shared_ff]. row_token, row_weight
// [rows]. out: float32 [T, ldo], added to, or (overwrite) stored. Launches 3 + 2 ceil(d / slice) kernels.
extern "C" int lp_experts(const void* x, const float* weights, int ldw, const void* w_up, const void* w_down, float* out, int ldo, int T,
                          int d, int E, int top, int ff, int shared_ff, int rows, int* counts, int* list, int* place, void* gathered,
                          int slice, void* hidden, int* row_token, float* row_weight, int overwrite, int* status, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (E <= 0 || E > MAX_EXPERTS || top <= 0 || ldw < E) LP_REFUSE("experts: %d experts (at most %d), %d chosen, weights of %d", E, MAX_EXPERTS, top, ldw);
    if (ff <= 0 || ff % 128 || shared_ff < 0 || shared_ff % 128) LP_REFUSE("experts: hidden sizes %d and %d must be multiples of 128", ff, shared_ff);
    if (d <= 0 || d % 8 || ldo < d || ldo % 4) LP_REFUSE("experts: width %d (a multiple of 8), rows of %d", d, ldo);
    if (slice <= 0 || (slice < d && slice % COLS)) LP_REFUSE("experts: slices of %d columns (a multiple of %d)", slice, COLS);
    if (((uintptr_t)x | (uintptr_t)w_up | (uintptr_t)w_down | (uintptr_t)gathered | (uintptr_t)hidden | (uintptr_t)out) & 15)
        LP_REFUSE("experts: operands must be 16-byte aligned");
    // at most T * top choices, and every expert's last tile may hold a single row
    long long need = (T * (long long)(top < E ? top : E) + (long long)E * (ROWS - 1)) / ROWS * ROWS;
    const long long most = (long long)E * ((T + ROWS - 1) / ROWS) * ROWS;
    if (need > most) need = most;
    if (rows % ROWS || rows < need) LP_REFUSE("experts: room for %d rows, %lld may be needed", rows, need);
    const int shared_rows = shared_ff > 0 ? T : 0;
    __nv_bfloat16* hidden_s = (__nv_bfloat16*)hidden + (size_t)rows * ff;
    CUtensorMap m_up, m_x, m_xs, m_down, m_h, m_hs;
    int rc = make_map(&m_up, w_up, 2LL * ((long long)E * ff + shared_ff), d, d, COLS);
    if (!rc) rc = make_map(&m_x, gathered, rows, d, d, ROWS);
    if (!rc) rc = make_map(&m_down, w_down, d, (long long)E * ff + shared_ff, (long long)E * ff + shared_ff, COLS);
    if (!rc) rc = make_map(&m_h, hidden, rows, ff, ff, ROWS);
    m_xs = m_x;                                               // (not read without a shared expert)
    m_hs = m_h;
    if (!rc && shared_ff > 0) rc = make_map(&m_xs, x, T, d, d, ROWS);
    if (!rc && shared_ff > 0) rc = make_map(&m_hs, hidden_s, T, shared_ff, shared_ff, ROWS);
    if (rc) return rc;
    cudaError_t err = lp_launch(expert_list_kernel, dim3(E), dim3(1024), 0, stream, weights, ldw, T, counts, list, place);
    if (err != cudaSuccess) return failed_launch(err, "list");
    err = lp_launch(expert_gather_kernel, dim3(rows / 4), dim3(256), 0, stream, (const __nv_bfloat16*)x, weights, ldw, (const int*)counts,
                    (const int*)list, T, d, E, (__nv_bfloat16*)gathered, row_token, row_weight, place, status);
    if (err != cudaSuccess) return failed_launch(err, "gather");
    Experts ex = {counts, row_token, row_weight, E, shared_rows, ff, shared_ff, d, rows, 0, d};
    const Shared to_hidden = {hidden_s, shared_ff, 1}, to_stream = {out, ldo, overwrite};
    const bool stores = overwrite && shared_ff == 0;          // (the shared expert's rows have been stored by then)
    rc = launch_gemm<true>(m_up, m_x, m_xs, hidden, ff, ex, to_hidden, status, stream);
    for (int c = 0; c < d && !rc; c += slice) {
        ex.col0 = c;
        ex.cols = d - c < slice ? d - c : slice;
        rc = launch_gemm<false>(m_down, m_h, m_hs, gathered, ex.cols, ex, to_stream, status, stream);
        if (rc) break;
        err = lp_launch(stores ? expert_sum_kernel<true> : expert_sum_kernel<false>, dim3(T), dim3(256), 0, stream, (const float*)gathered,
                        (const int*)place, T, E, out, ldo, c, ex.cols);
        if (err != cudaSuccess) return failed_launch(err, "sum");
        rc = lp_check_launch("experts (sum)");
    }
    return rc;
}
