// Plain matrix product for weights stored [out, in]:  C[M, N] = A[M, K] * W[N, K]^T.
// No tensor cores, float32 multiply-add only. Every output element is summed in one fixed way whatever M is and
// whichever kernel below forms it: K is cut into eighths (rounded up to 32 products), each eighth is a chain of
// multiply-adds in increasing k that starts at zero, and the eighths' sums are added in increasing order. So a
// row's result does not depend on which other rows share the launch, the eighths can be formed side by side where
// a launch would otherwise leave the chip idle, and the chains are an eighth as long as one over all of K would
// be (which makes the rounding error smaller, not larger). It is the product of the float32 path and the
// comparison twin of the tensor-core kernels.
//
// Counterparts in the reference (src/main/resources/kernels/cuda/): matmul_f32.cu:6-39,
// matmul_bf16.cu:6-37 (one warp per output row, one input vector), silu_mul.cu:6-15,
// and the add-to-output mode the reference uses for the residual
// (java21 inference/CudaForwardPass.java:1012-1017).
#include <cooperative_groups.h>

#include "common.cuh"

#define LP_GEMM_STORE 0      // C = A W^T
#define LP_GEMM_ACCUMULATE 1 // C += A W^T         (C float32: the residual stream)
#define LP_GEMM_SWIGLU 2     // C = silu(A Wg^T) * (A Wu^T), W = [gate rows | up rows], N = rows of each

namespace {

constexpr int PARTS = 8;     // chains per output element

// products per chain: an eighth of K, rounded up to 32
__host__ __device__ __forceinline__ int part_length(int K) { return ((K + 32 * PARTS - 1) / (32 * PARTS)) * 32; }

__device__ __forceinline__ float silu_mul(float g, float u) { return g / (1.0f + expf(-g)) * u; }

// ---------------------------------------------------------------- any types, sizes and alignments
constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

template <typename TA, typename TW, typename TC, int MODE>
__global__ void __launch_bounds__(256)
gemm_plain_kernel(const TA* __restrict__ A, const TW* __restrict__ W, TC* __restrict__ C, int M, int N, int K,
                  int lda, int ldw, int ldc) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    __shared__ float Us[MODE == LP_GEMM_SWIGLU ? BK : 1][BN + 4];

    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;

    float acc[TM][TN], sum[TM][TN];
    float acu[MODE == LP_GEMM_SWIGLU ? TM : 1][TN], sumu[MODE == LP_GEMM_SWIGLU ? TM : 1][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            acc[i][j] = sum[i][j] = 0.f;
            if (MODE == LP_GEMM_SWIGLU) acu[i][j] = sumu[i][j] = 0.f;
        }

    // each thread loads 4 elements of each 64x16 tile: row = tid / 4, k = (tid % 4) * 4 .. +3
    const int lr = tid >> 2, lk = (tid & 3) * 4;
    const int part = part_length(K);
    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = k0 + lk + j;
            const int am = m0 + lr, wn = n0 + lr;
            As[lk + j][lr] = (am < M && k < K) ? lp_to_float(A[(long long)am * lda + k]) : 0.f;
            Ws[lk + j][lr] = (wn < N && k < K) ? lp_to_float(W[(long long)wn * ldw + k]) : 0.f;
            if (MODE == LP_GEMM_SWIGLU)
                Us[lk + j][lr] = (wn < N && k < K) ? lp_to_float(W[(long long)(wn + N) * ldw + k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float a[TM], w[TN], u[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[k][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                w[j] = Ws[k][tx * TN + j];
                if (MODE == LP_GEMM_SWIGLU) u[j] = Us[k][tx * TN + j];
            }
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
                    if (MODE == LP_GEMM_SWIGLU) acu[i][j] = fmaf(a[i], u[j], acu[i][j]);
                }
        }
        __syncthreads();
        if ((k0 + BK) % part == 0 || k0 + BK >= K) {        // a chain ends here
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    sum[i][j] += acc[i][j];
                    acc[i][j] = 0.f;
                    if (MODE == LP_GEMM_SWIGLU) {
                        sumu[i][j] += acu[i][j];
                        acu[i][j] = 0.f;
                    }
                }
        }
    }

#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty * TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx * TN + j;
            if (n >= N) continue;
            TC* c = C + (long long)m * ldc + n;
            if (MODE == LP_GEMM_STORE)
                *c = lp_from_float<TC>(sum[i][j]);
            else if (MODE == LP_GEMM_ACCUMULATE)
                *c = lp_from_float<TC>(lp_to_float(*c) + sum[i][j]);
            else
                *c = lp_from_float<TC>(silu_mul(sum[i][j], sumu[i][j]));
        }
    }
}

// ---------------------------------------------------------------- float32, a handful of rows
__device__ __forceinline__ void copy16(void* smem, const void* gmem, bool real) {
    const unsigned to = (unsigned)__cvta_generic_to_shared(smem);
    const int bytes = real ? 16 : 0;       // the rest of the 16 bytes is zero
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

constexpr int ROW_FEATURES = 8;          // output features of a CTA (in the gated form as many gate and up rows)
constexpr int ROW_CHUNK = 32;            // products of a chain per stage
constexpr int ROW_STRIDE = ROW_CHUNK + 4;   // 144 bytes from one chain's chunk to the next: eight lanes' 16-byte reads hit all banks

// DEEP: a ring of up to eight stages, two CTAs per SM (for grids that have no more); else four stages, of which two (16 rows) to five (one
// row) CTAs fit an SM, in the gated form two, and one at 16 rows (147 KB)
template <int MR, int MODE, bool DEEP> struct RowsShape {
    static constexpr int WROWS = MODE == LP_GEMM_SWIGLU ? 2 * ROW_FEATURES : ROW_FEATURES;
    static constexpr int THREADS = WROWS * PARTS;
    static constexpr int STAGE = (WROWS + MR) * PARTS * ROW_STRIDE;       // floats
    static constexpr int ROOM = 113 * 1024 / 4 / STAGE;
    static constexpr int STAGES = !DEEP || ROOM < 4 ? 4 : ROOM < 8 ? ROOM : 8;
    static constexpr size_t SMEM = (size_t)STAGE * STAGES * sizeof(float);
};

template <int MR, int MODE, bool DEEP>
__global__ void __launch_bounds__(RowsShape<MR, MODE, DEEP>::THREADS, 1)
gemm_f32_rows_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K,
                     int lda, int ldw, int ldc) {
    // A step of a few sequences reads every weight once and is bound by that. A thread owns one chain of one weight row
    // for all MR rows of A: the chains of a CTA's rows run side by side, so N / 8 CTAs of 64 threads are enough to keep
    // the memory busy, and the order of every sum stays the one named above. 4 rows, B200: 16384 x 2048 (gated) 229 -> 30 us
    // (4.5 TB/s), 2048 x 8192 about 700 -> 19 us (3.5 TB/s) against the 64 x 64 tiles of the kernel above, which left most of
    // the chip idle. What is left is issue: about 60 instructions per warp and 4 KB of weights, and the launch itself.
    using S = RowsShape<MR, MODE, DEEP>;
    extern __shared__ __align__(16) float ring[];
    const int tid = threadIdx.x;
    const int n0 = blockIdx.x * ROW_FEATURES, m0 = blockIdx.y * MR;
    const int row = tid % S::WROWS, chain = tid / S::WROWS;
    const int part = part_length(K);
    const int steps = part / ROW_CHUNK;

    // Copies go in pieces of 16 bytes, eight to a chunk, chunks ordered [chain][row]: thread tid always copies piece
    // tid % 8 of weight row tid / 8, for every chain, so only the step moves its addresses.
    const int piece = (tid & 7) * 4, copy_row = tid >> 3;
    const int feature = n0 + (copy_row % ROW_FEATURES);
    const bool feature_ok = feature < N;
    const float* from_w = W + (feature_ok ? (long long)(copy_row < ROW_FEATURES ? feature : N + feature) * ldw + piece : 0);
    float* to_w = ring + copy_row * ROW_STRIDE + piece;
    auto fetch_w = [&](int step, int slot) {
        if (step >= steps) return;
        float* to = to_w + slot * S::STAGE;
        const float* from = from_w + step * ROW_CHUNK;
        const int limit = feature_ok ? K - piece - step * ROW_CHUNK : 0;
#pragma unroll
        for (int c = 0; c < PARTS; ++c) copy16(to + c * S::WROWS * ROW_STRIDE, c * part < limit ? from + c * part : W, c * part < limit);
    };
    constexpr int A_COPIES = MR * PARTS * 8 / S::THREADS > 0 ? MR * PARTS * 8 / S::THREADS : 1;     // per thread
    auto fetch_a = [&](int step, int slot) {
        if (step >= steps) return;
        float* base = ring + slot * S::STAGE + PARTS * S::WROWS * ROW_STRIDE;
#pragma unroll
        for (int i = 0; i < A_COPIES; ++i) {
            const int p = (i * S::THREADS + tid) >> 3, r = p % MR, c = p / MR;
            if (c >= PARTS) break;
            const int k = c * part + step * ROW_CHUNK + piece;
            const bool real = k < K && m0 + r < M;
            copy16(base + (c * MR + r) * ROW_STRIDE + piece, real ? A + (long long)(m0 + r) * lda + k : A, real);
        }
    };

    // weights are written by no kernel of a step: the first stages of them are asked for before the wait
#pragma unroll
    for (int s = 0; s < S::STAGES - 1; ++s) fetch_w(s, s);
    lp_grid_wait();
    lp_grid_release();
#pragma unroll
    for (int s = 0; s < S::STAGES - 1; ++s) {
        fetch_a(s, s);
        copies_commit();       // the first group also holds all weights asked for above
    }
    float acc[MR];
#pragma unroll
    for (int m = 0; m < MR; ++m) acc[m] = 0.f;
    int slot = 0;
    for (int step = 0; step < steps; ++step) {
        copies_wait<S::STAGES - 2>();
        __syncthreads();
        {
            const int next = step + S::STAGES - 1, to = slot == 0 ? S::STAGES - 1 : slot - 1;
            fetch_w(next, to);
            fetch_a(next, to);
            copies_commit();
        }
        const float* w = ring + slot * S::STAGE + (chain * S::WROWS + row) * ROW_STRIDE;
        const float* a = ring + slot * S::STAGE + PARTS * S::WROWS * ROW_STRIDE + chain * MR * ROW_STRIDE;
#pragma unroll
        for (int c = 0; c < ROW_CHUNK / 4; ++c) {
            const float4 wv = *(const float4*)(w + c * 4);
#pragma unroll
            for (int m = 0; m < MR; ++m) {
                const float4 av = *(const float4*)(a + m * ROW_STRIDE + c * 4);
                acc[m] = fmaf(av.x, wv.x, acc[m]);
                acc[m] = fmaf(av.y, wv.y, acc[m]);
                acc[m] = fmaf(av.z, wv.z, acc[m]);
                acc[m] = fmaf(av.w, wv.w, acc[m]);
            }
        }
        slot = slot + 1 == S::STAGES ? 0 : slot + 1;
    }
    copies_wait<0>();
    __syncthreads();
    float* sums = ring;                                   // [chain][m][weight row]
#pragma unroll
    for (int m = 0; m < MR; ++m) sums[(chain * MR + m) * S::WROWS + row] = acc[m];
    __syncthreads();
    const int chains = (K + part - 1) / part;
    for (int i = tid; i < MR * ROW_FEATURES; i += S::THREADS) {
        const int m = i / ROW_FEATURES, f = i % ROW_FEATURES;
        if (m0 + m >= M || n0 + f >= N) continue;
        float s = 0.f, u = 0.f;
        for (int c = 0; c < chains; ++c) {
            s += sums[(c * MR + m) * S::WROWS + f];
            if (MODE == LP_GEMM_SWIGLU) u += sums[(c * MR + m) * S::WROWS + ROW_FEATURES + f];
        }
        float* out = C + (long long)(m0 + m) * ldc + n0 + f;
        if (MODE == LP_GEMM_STORE) *out = s;
        else if (MODE == LP_GEMM_ACCUMULATE) *out += s;
        else *out = silu_mul(s, u);
    }
}

// ---------------------------------------------------------------- float32, many rows
// Two multiply-adds in one instruction, each rounded like fmaf: a plain fmaf per product leaves half of the units idle.
typedef unsigned long long pair_t;
__device__ __forceinline__ pair_t make_pair(float lo, float hi) {
    pair_t p;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(lo), "f"(hi));
    return p;
}
__device__ __forceinline__ float2 from_pair(pair_t p) {
    float2 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ pair_t fma_pair(pair_t a, pair_t b, pair_t c) {
    pair_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

constexpr int TILE_N = 128, TILE_K = 16;

template <int ROWS> struct TileShape {
    static constexpr int THREADS = ROWS * 2;              // 8 x 8 outputs each
    static constexpr int LDA = ROWS + 4, LDW = TILE_N + 4;
    static constexpr int STAGE = TILE_K * (LDA + LDW);    // floats; two stages
    static constexpr int HELD = 64 * THREADS;             // floats: every thread's outputs, [16 groups of 4][thread]
    static constexpr size_t SMEM = (size_t)(2 * STAGE + HELD) * sizeof(float);
};

// A thread forms rows {ty*4.., ROWS/2 + ty*4..} x columns {tx*4.., 64 + tx*4..} of a ROWS x 128 tile; in the gated form
// the first 64 columns are gate rows of W and the last 64 the up rows of the same features, so a thread holds both.
// SPLIT: the eight CTAs of a cluster form one chain each and add them up through distributed shared memory.
// Bound by the multiply-add units (71 TFLOP/s measured for multiply-adds alone). B200, 509 rows: 16384 x 2048 (gated) 1272 ->
// 821 us, 2048 x 8192 about 900 -> 407 us, 3072 x 2048 307 -> 164 us (42 TFLOP/s; 50 at 2048 rows, where the last wave is
// fuller). The kernel above reads shared memory four bytes at a time and reaches 27.
template <int ROWS, int MODE, bool SPLIT>
__global__ void __launch_bounds__(ROWS * 2, ROWS == 128 ? 2 : 4)
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K,
                     int lda, int ldw, int ldc) {
    using S = TileShape<ROWS>;
    extern __shared__ __align__(16) float smem[];
    float* held = smem + 2 * S::STAGE;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = (warp & 1) * 8 + (lane & 7), ty = (warp >> 1) * 4 + (lane >> 3);
    constexpr int FEATURES = MODE == LP_GEMM_SWIGLU ? TILE_N / 2 : TILE_N;
    const int n0 = blockIdx.x * FEATURES, m0 = blockIdx.y * ROWS;
    const int part = part_length(K);
    const int k_begin = SPLIT ? (int)blockIdx.z * part : 0;
    const int k_end = SPLIT ? min(K, k_begin + part) : K;

    // loads: 4 values along k of one row; lanes cover 8 rows x 16 k, so a row's 64 bytes are read together
    constexpr int PASS = S::THREADS / 4;                  // rows per pass
    constexpr int PA = ROWS / PASS, PW = TILE_N / PASS;
    const int lr = tid >> 2, lk = (tid & 3) * 4;
    const float* wrow[PW];
    bool wok[PW];
#pragma unroll
    for (int i = 0; i < PW; ++i) {
        const int c = lr + i * PASS;
        const int f = MODE == LP_GEMM_SWIGLU ? n0 + (c & 63) : n0 + c;
        wok[i] = f < N;
        wrow[i] = W + (long long)(MODE == LP_GEMM_SWIGLU && c >= 64 ? N + f : f) * ldw;
    }
    float4 ra[PA], rw[PW];
    const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
    auto fetch = [&](int k0) {
        const int k = k0 + lk;
#pragma unroll
        for (int i = 0; i < PW; ++i) rw[i] = wok[i] && k < k_end ? *(const float4*)(wrow[i] + k) : none;
#pragma unroll
        for (int i = 0; i < PA; ++i) {
            const int m = m0 + lr + i * PASS;
            ra[i] = m < M && k < k_end ? *(const float4*)(A + (long long)m * lda + k) : none;
        }
    };
    auto put = [&](int stage) {
        float* as = smem + stage * S::STAGE;
        float* ws = as + TILE_K * S::LDA;
#pragma unroll
        for (int i = 0; i < PA; ++i) {
            const int r = lr + i * PASS;
            as[(lk + 0) * S::LDA + r] = ra[i].x;
            as[(lk + 1) * S::LDA + r] = ra[i].y;
            as[(lk + 2) * S::LDA + r] = ra[i].z;
            as[(lk + 3) * S::LDA + r] = ra[i].w;
        }
#pragma unroll
        for (int i = 0; i < PW; ++i) {
            const int c = lr + i * PASS;
            ws[(lk + 0) * S::LDW + c] = rw[i].x;
            ws[(lk + 1) * S::LDW + c] = rw[i].y;
            ws[(lk + 2) * S::LDW + c] = rw[i].z;
            ws[(lk + 3) * S::LDW + c] = rw[i].w;
        }
    };

    pair_t acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;

    lp_grid_wait();
    lp_grid_release();
    fetch(k_begin);
    put(0);
    __syncthreads();
    int stage = 0;
    bool first_part = true;
    for (int k0 = k_begin; k0 < k_end; k0 += TILE_K) {
        const bool more = k0 + TILE_K < k_end;
        if (more) fetch(k0 + TILE_K);
        const float* as = smem + stage * S::STAGE + ty * 4;
        const float* ws = smem + stage * S::STAGE + TILE_K * S::LDA + tx * 4;
#pragma unroll
        for (int k = 0; k < TILE_K; ++k) {
            const float4 a0 = *(const float4*)(as + k * S::LDA), a1 = *(const float4*)(as + k * S::LDA + ROWS / 2);
            const ulonglong2 w0 = *(const ulonglong2*)(ws + k * S::LDW), w1 = *(const ulonglong2*)(ws + k * S::LDW + 64);
            const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const pair_t a = make_pair(av[i], av[i]);
                acc[i][0] = fma_pair(a, w0.x, acc[i][0]);
                acc[i][1] = fma_pair(a, w0.y, acc[i][1]);
                acc[i][2] = fma_pair(a, w1.x, acc[i][2]);
                acc[i][3] = fma_pair(a, w1.y, acc[i][3]);
            }
        }
        if (!SPLIT && more && (k0 + TILE_K) % part == 0) {        // a chain ends: its sums join those held
            float4* h = (float4*)held + tid;
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const float2 lo = from_pair(acc[i][2 * j]), hi = from_pair(acc[i][2 * j + 1]);
                    float4 v = first_part ? none : h[(i * 2 + j) * S::THREADS];
                    v.x += lo.x; v.y += lo.y; v.z += hi.x; v.w += hi.y;
                    h[(i * 2 + j) * S::THREADS] = v;
                    acc[i][2 * j] = acc[i][2 * j + 1] = 0ull;
                }
            first_part = false;
        }
        if (more) {
            put(stage ^ 1);
            __syncthreads();
            stage ^= 1;
        }
    }

    auto finish = [&](int i, float4 s0, float4 s1) {
        const int m = m0 + (i < 4 ? ty * 4 + i : ROWS / 2 + ty * 4 + i - 4);
        if (m >= M) return;
        float* c = C + (long long)m * ldc;
        auto store4 = [&](int n, const float4& v) {
            const float x[4] = {v.x, v.y, v.z, v.w};
            if (n + 3 < N && (ldc & 3) == 0 && ((size_t)C & 15) == 0) {
                float4* to = (float4*)(c + n);
                if (MODE == LP_GEMM_ACCUMULATE) {
                    const float4 old = *to;
                    *to = make_float4(old.x + x[0], old.y + x[1], old.z + x[2], old.w + x[3]);
                } else {
                    *to = v;
                }
                return;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (n + j < N) c[n + j] = MODE == LP_GEMM_ACCUMULATE ? c[n + j] + x[j] : x[j];
        };
        if (MODE == LP_GEMM_SWIGLU) {
            store4(n0 + tx * 4, make_float4(silu_mul(s0.x, s1.x), silu_mul(s0.y, s1.y), silu_mul(s0.z, s1.z), silu_mul(s0.w, s1.w)));
        } else {
            store4(n0 + tx * 4, s0);
            store4(n0 + 64 + tx * 4, s1);
        }
    };
    float4* h = (float4*)held + tid;
    if (SPLIT) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float2 lo = from_pair(acc[i][2 * j]), hi = from_pair(acc[i][2 * j + 1]);
                h[(i * 2 + j) * S::THREADS] = make_float4(lo.x, lo.y, hi.x, hi.y);
            }
        cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
        cluster.sync();
        const int i = blockIdx.z;                        // this CTA adds up one of the eight rows of every thread
        float4 s[2] = {none, none};
#pragma unroll
        for (int c = 0; c < PARTS; ++c) {
            const float4* from = (const float4*)cluster.map_shared_rank(held, c) + tid;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float4 v = from[(i * 2 + j) * S::THREADS];
                s[j].x += v.x; s[j].y += v.y; s[j].z += v.z; s[j].w += v.w;
            }
        }
        finish(i, s[0], s[1]);
        cluster.sync();                                  // nobody leaves while its sums are still read
        return;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float4 s[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float2 lo = from_pair(acc[i][2 * j]), hi = from_pair(acc[i][2 * j + 1]);
            s[j] = first_part ? none : h[(i * 2 + j) * S::THREADS];
            s[j].x += lo.x; s[j].y += lo.y; s[j].z += hi.x; s[j].w += hi.y;
        }
        finish(i, s[0], s[1]);
    }
}

// ---------------------------------------------------------------- choice and launch
int failed(cudaError_t err, const char* what) {
    snprintf(lp_error_text, sizeof(lp_error_text), "gemm_plain (%s): %s", what, cudaGetErrorString(err));
    return (int)err;
}

template <int MR, int MODE, bool DEEP>
int launch_rows_as(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t stream) {
    using S = RowsShape<MR, MODE, DEEP>;
    auto kernel = gemm_f32_rows_kernel<MR, MODE, DEEP>;
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
    if (err != cudaSuccess) return failed(err, "rows");
    dim3 grid((N + ROW_FEATURES - 1) / ROW_FEATURES, (M + MR - 1) / MR);
    err = lp_launch(kernel, grid, dim3(S::THREADS), S::SMEM, stream, A, W, C, M, N, K, lda, ldw, ldc);
    return err == cudaSuccess ? lp_check_launch("gemm_plain (rows)") : failed(err, "rows");
}

template <int MR, int MODE>
int launch_rows(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t stream) {
    const long long ctas = (long long)((N + ROW_FEATURES - 1) / ROW_FEATURES) * ((M + MR - 1) / MR);
    if (MODE != LP_GEMM_SWIGLU && ctas <= 2 * lp_sm_count())
        return launch_rows_as<MR, MODE, true>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    return launch_rows_as<MR, MODE, false>(A, W, C, M, N, K, lda, ldw, ldc, stream);
}

template <int ROWS, int MODE, bool SPLIT>
int launch_tile(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t stream) {
    using S = TileShape<ROWS>;
    auto kernel = gemm_f32_tile_kernel<ROWS, MODE, SPLIT>;
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
    if (err != cudaSuccess) return failed(err, "tile");
    constexpr int FEATURES = MODE == LP_GEMM_SWIGLU ? TILE_N / 2 : TILE_N;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((N + FEATURES - 1) / FEATURES, (M + ROWS - 1) / ROWS, SPLIT ? PARTS : 1);
    cfg.blockDim = dim3(S::THREADS);
    cfg.dynamicSmemBytes = S::SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int attrs = 0;
    if (lp_pdl_enabled()) {
        attr[attrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[attrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (SPLIT) {
        attr[attrs].id = cudaLaunchAttributeClusterDimension;
        attr[attrs].val.clusterDim.x = 1;
        attr[attrs].val.clusterDim.y = 1;
        attr[attrs++].val.clusterDim.z = PARTS;
    }
    cfg.attrs = attr;
    cfg.numAttrs = attrs;
    err = cudaLaunchKernelEx(&cfg, kernel, A, W, C, M, N, K, lda, ldw, ldc);
    return err == cudaSuccess ? lp_check_launch("gemm_plain (tile)") : failed(err, "tile");
}

template <int MODE>
int launch_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t s) {
    // up to 32 rows the weights' bytes bound the product (16 rows at a time; from 33 rows on the tile of 64 is faster:
    // 16384 x 2048 gated, 32 / 48 rows: 130 / 129 us)
    if (M <= 1) return launch_rows<1, MODE>(A, W, C, M, N, K, lda, ldw, ldc, s);
    if (M <= 2) return launch_rows<2, MODE>(A, W, C, M, N, K, lda, ldw, ldc, s);
    if (M <= 4) return launch_rows<4, MODE>(A, W, C, M, N, K, lda, ldw, ldc, s);
    if (M <= 8) return launch_rows<8, MODE>(A, W, C, M, N, K, lda, ldw, ldc, s);
    if (M <= 32) return launch_rows<16, MODE>(A, W, C, M, N, K, lda, ldw, ldc, s);
    constexpr int FEATURES = MODE == LP_GEMM_SWIGLU ? TILE_N / 2 : TILE_N;
    const bool tall = (M + 127) / 128 * 2 == (M + 63) / 64;       // the 128-row tile wastes no more rows than the 64-row one
    const long long tiles = (long long)((N + FEATURES - 1) / FEATURES) * ((M + (tall ? 127 : 63)) / (tall ? 128 : 64));
    // fewer tiles than two per SM: the chains side by side (64 tiles, 2048 x 2048 at 509 rows: 111 us in clusters)
    const bool split = K > 32 * PARTS && tiles < 2 * lp_sm_count();
    if (tall)
        return split ? launch_tile<128, MODE, true>(A, W, C, M, N, K, lda, ldw, ldc, s)
                     : launch_tile<128, MODE, false>(A, W, C, M, N, K, lda, ldw, ldc, s);
    return split ? launch_tile<64, MODE, true>(A, W, C, M, N, K, lda, ldw, ldc, s)
                 : launch_tile<64, MODE, false>(A, W, C, M, N, K, lda, ldw, ldc, s);
}

template <typename TA, typename TW, typename TC>
int launch_mode(const void* A, const void* W, void* C, int M, int N, int K, int lda, int ldw, int ldc, int mode,
                cudaStream_t stream) {
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (mode == LP_GEMM_STORE)
        gemm_plain_kernel<TA, TW, TC, LP_GEMM_STORE><<<grid, 256, 0, stream>>>(
            (const TA*)A, (const TW*)W, (TC*)C, M, N, K, lda, ldw, ldc);
    else if (mode == LP_GEMM_ACCUMULATE)
        gemm_plain_kernel<TA, TW, TC, LP_GEMM_ACCUMULATE><<<grid, 256, 0, stream>>>(
            (const TA*)A, (const TW*)W, (TC*)C, M, N, K, lda, ldw, ldc);
    else
        gemm_plain_kernel<TA, TW, TC, LP_GEMM_SWIGLU><<<grid, 256, 0, stream>>>(
            (const TA*)A, (const TW*)W, (TC*)C, M, N, K, lda, ldw, ldc);
    return lp_check_launch("gemm_plain");
}

template <typename TA, typename TW>
int launch_out(const void* A, const void* W, void* C, int c_dtype, int M, int N, int K, int lda, int ldw, int ldc,
               int mode, cudaStream_t stream) {
    if (c_dtype == LP_F32) return launch_mode<TA, TW, float>(A, W, C, M, N, K, lda, ldw, ldc, mode, stream);
    return launch_mode<TA, TW, __nv_bfloat16>(A, W, C, M, N, K, lda, ldw, ldc, mode, stream);
}

}  // namespace

// A: [M, K] row stride lda; W: [N, K] (or [2N, K] in SWIGLU mode) row stride ldw; C: [M, N] row stride ldc.
extern "C" int lp_gemm_plain(const void* A, int a_dtype, const void* W, int w_dtype, void* C, int c_dtype, int M,
                             int N, int K, int lda, int ldw, int ldc, int mode, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) LP_REFUSE("gemm_plain: inner size %d", K);
    if (mode < 0 || mode > 2) LP_REFUSE("gemm_plain: mode %d", mode);
    if (c_dtype != LP_F32 && c_dtype != LP_BF16) LP_REFUSE("gemm_plain: output dtype code %d", c_dtype);
    if (mode == LP_GEMM_ACCUMULATE && c_dtype != LP_F32)
        LP_REFUSE("gemm_plain: accumulation needs a float32 output");
    if ((N + BN - 1) / BN > 2147483647 || (M + BM - 1) / BM > 65535)
        LP_REFUSE("gemm_plain: %d rows exceed the grid", M);
    // rows of float32 that can be read 16 bytes at a time: the kernels made for that, others: the one for everything
    const bool wide = a_dtype == LP_F32 && w_dtype == LP_F32 && c_dtype == LP_F32 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0
                      && (size_t)A % 16 == 0 && (size_t)W % 16 == 0;
    if (wide) {
        const float *a = (const float*)A, *w = (const float*)W;
        if (mode == LP_GEMM_STORE) return launch_f32<LP_GEMM_STORE>(a, w, (float*)C, M, N, K, lda, ldw, ldc, stream);
        if (mode == LP_GEMM_ACCUMULATE) return launch_f32<LP_GEMM_ACCUMULATE>(a, w, (float*)C, M, N, K, lda, ldw, ldc, stream);
        return launch_f32<LP_GEMM_SWIGLU>(a, w, (float*)C, M, N, K, lda, ldw, ldc, stream);
    }
    if (a_dtype == LP_F32 && w_dtype == LP_F32)
        return launch_out<float, float>(A, W, C, c_dtype, M, N, K, lda, ldw, ldc, mode, stream);
    if (a_dtype == LP_BF16 && w_dtype == LP_BF16)
        return launch_out<__nv_bfloat16, __nv_bfloat16>(A, W, C, c_dtype, M, N, K, lda, ldw, ldc, mode, stream);
    if (a_dtype == LP_BF16 && w_dtype == LP_F32)
        return launch_out<__nv_bfloat16, float>(A, W, C, c_dtype, M, N, K, lda, ldw, ldc, mode, stream);
    if (a_dtype == LP_F32 && w_dtype == LP_BF16)
        return launch_out<float, __nv_bfloat16>(A, W, C, c_dtype, M, N, K, lda, ldw, ldc, mode, stream);
    LP_REFUSE("gemm_plain: dtype codes a=%d w=%d", a_dtype, w_dtype);
}
