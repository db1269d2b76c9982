// Plain matrix product for weights stored [out, in]:  C[M, N] = A[M, K] * W[N, K]^T.
// Every output element is summed in one fixed way whatever M is, so a row's result does not depend on which other rows share the
// launch: K is cut into eighths (rounded up to 32 products), each eighth is a sum of its own, the eighths of each half are
// added in increasing order, then the halves. Two ways of forming an eighth:
//   * rows of 32 float32 and more that can be read 16 bytes at a time: on the tensor cores, float32 numbers as three bfloat16 parts
//     (gemm_f32_few_kernel and gemm_f32_rows_kernel up to 16 rows, gemm_f32_split_kernel from 17 on: the same bits);
//   * any other types, sizes and alignments: a chain of multiply-adds in increasing k that starts at zero (gemm_plain_kernel, which
//     adds all eighths in order).
// Errors against 64 bits, root mean square in units of 2^-24 of the sum of the products' magnitudes, in parts / by multiply-adds, at
// K = 32, 64, 256, 2048, 8192: normal numbers 0.20 / 0.47, 0.17 / 0.35, 0.11 / 0.19, 0.05 / 0.17, 0.04 / 0.17; numbers in [1, 2) 0.65 / 1.46, 0.82 / 1.21,
// 0.90 / 0.96, 0.92 / 1.62, 1.02 / 2.94; numbers of very different sizes (normal times e^(2 normal)) 0.61 / 1.08, 0.62 / 1.02, 0.62 / 0.92, 0.54 / 1.58,
// 0.55 / 2.30; mantissas of ones 1.25 / 1.89, 1.16 / 1.63, 1.22 / 2.22, 1.43 / 2.38, 1.64 / 115, but 1.16 / 0.87 at K = 16: hence the line at 32 (behind it
// these alone came out worse, at 40: 1.59 / 1.11). A product that stands alone in its sum is off by 0.63 (3.7 at most) where a rounded one is by 0.42 (1.0).
// It is the product of the float32 path and the comparison twin of the bfloat16 kernels.
//
// Counterparts in the reference (src/main/resources/kernels/cuda/): matmul_f32.cu:6-39,
// matmul_bf16.cu:6-37 (one warp per output row, one input vector), silu_mul.cu:6-15,
// and the add-to-output mode the reference uses for the residual
// (java21 inference/CudaForwardPass.java:1012-1017).
#include <cooperative_groups.h>

#include "tcgen05_utils.cuh"

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

// ---------------------------------------------------------------- float32 on the tensor cores
// A float32 number is the sum of three bfloat16 ones (3 x 8 bits), and a product of two such parts is exact in float32. So a
// product of float32 numbers is six products on the tensor cores: all pairs of parts but the three smallest (together at most 3 x 2^-24 of
// the whole, of either sign: split_tokens). What would lose bits is their sum: the tensor cores cut every partial sum off instead of rounding it. So
// the sums in tensor memory are short: 32 products of K, the small pairs first, the two steps of the leading parts last
// (a step is 16 products); such a block's sum is added to those before it in registers, rounded to nearest, as fmaf would.
// The exponents of float32 and bfloat16 end at the same place, parts and products of parts do not: operands are taken times 2^24, so that
// every part of every float32 number has room and no product that a float32 result could hold vanishes, and sums times 2^-48 at the end; sums beyond 2^80
// are formed again one by one, like those that are not finite.
//
// Per CTA: 128 weight rows (in the gated form 64 gate and the 64 up rows of the same features) x TOK tokens.
//   warp 0       TMA: float32 boxes of 32 columns of the weights into a ring of stages
//   warp 2       the tokens' parts, made beforehand by split_rows_kernel, into a ring of their own
//   warps 1, 3   issue the MMAs of every second block: 12 of 128 x TOK x 16
//   warps 4-     a weight row per thread: its 32 values in three parts, into tensor memory (the row operand of the MMAs); two groups
//                of four warps, for every second block each, or one
//   the last 4 or 8   a block's sums from tensor memory into registers, chains of an eighth of K, the output
// Two buffers of operands and two of sums, so that all of these work at the same time on neighbouring blocks. Bound by the way round one
// buffer (sums fetched, weights split, MMAs of about 80 cycles each beside the traffic to tensor memory): about 1,100 cycles per block
// against 790 for its MMAs alone. B200, each product back to back with itself (weights partly in L2), against register tiles of paired multiply-adds, 509
// rows: 16384 x 2048 (gated) 820 -> 222 us, 2048 x 8192 407 -> 105, 3072 x 2048 163 -> 53, 2048 x 2048 111 -> 39; the four one behind the other
// (243 MB of weights, cold) 1499 -> 420. 64 rows: 130 -> 60, 121 -> 53, 34 -> 22, 34 -> 26; together 359 -> 177. 17 rows: together 301 -> 170.
constexpr int SPLIT_K = 32;                     // products of a block
constexpr int SPLIT_MIN_K = 32;                 // shorter sums run on gemm_plain_kernel (300 x 2048, K = 16: 4.7 us, 9.8 in parts)
constexpr float SPLIT_SCALE = 16777216.f, SUM_SCALE = 1.f / (SPLIT_SCALE * SPLIT_SCALE);      // 2^24 of an operand, 2^-48 of a sum

template <int TOK> struct SplitTile {
    static constexpr int ADDERS = TOK == 128 ? 8 : 4;             // warps that add blocks up
    static constexpr int GROUPS = TOK == 128 ? 1 : 2;             // of four warps that split weights (registers allow 16 warps in all)
    static constexpr int FIRST_ADDER = 4 + 4 * GROUPS;
    static constexpr int THREADS = (FIRST_ADDER + ADDERS) * 32;
    static constexpr int COLS = 64;                               // columns (tokens) of an adding thread
    static constexpr int PART = TOK * 64;                         // bytes of one part of the tokens' block: rows of 32 bfloat16
    static constexpr int W_BYTES = 128 * 128, STAGES = TOK == 128 ? 4 : 5;
    static constexpr int X_STAGE = 3 * PART, X_STAGES = TOK == 128 ? 4 : 6;
    static constexpr int RING = STAGES * W_BYTES + X_STAGES * X_STAGE;
    static constexpr int TMEM_COLS = 512;
    static constexpr int SUMS = 0, WEIGHTS = 2 * TOK, HELD = WEIGHTS + 2 * 48;      // columns of tensor memory
    static constexpr int SLOTS = TOK == 128 ? 1 : 2;              // sums of chains that tensor memory has room for
    static constexpr int HALF = TOK == 128 ? TOK * 128 * 4 : 0;   // bytes for the sums of the first half of K, where that room is one slot
    static constexpr size_t SMEM = 1024 + (size_t)RING + HALF + 256;
    static_assert(HELD + SLOTS * TOK <= TMEM_COLS, "tensor memory");
    static_assert(RING >= SLOTS * TOK * 128 * 4, "the ring also holds the sums that a cluster adds up");
    static_assert(X_STAGE % 1024 == 0 && PART % 512 == 0, "swizzled boxes");
};

__device__ __forceinline__ void split_mma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// K-major tile of rows of 64 bytes, swizzled in groups of 8 rows (512 bytes): 16-byte piece c of row r lies at piece c ^ (r / 2 % 4)
__device__ __forceinline__ uint64_t smem_desc_rows64(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFF) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)4 << 61;
}
// Neighbouring values, times 2^24, in three parts each: leading eight bits, the next eight, the rest. An infinity or a NaN, or a value
// that the factor or the rounding takes beyond the range, makes sums that are no numbers, which the epilogue forms again one by one.
__device__ __forceinline__ void scale_pair(float& x, float& y) {
    asm("{\n\t.reg .b64 v, f;\n\tmov.b64 v, {%0, %1};\n\tmov.b64 f, {%2, %2};\n\tmul.rn.f32x2 v, v, f;\n\tmov.b64 {%0, %1}, v;\n\t}"
        : "+f"(x), "+f"(y) : "f"(SPLIT_SCALE));
}
template <bool ROUND>
__device__ __forceinline__ uint32_t leading_pair(float& x, float& y) {       // x and y keep what is behind their leading bits
    const uint32_t p = __float_as_uint(x) + (ROUND ? 0x8000u : 0u), q = __float_as_uint(y) + (ROUND ? 0x8000u : 0u);
    asm("{\n\t.reg .b64 v, h;\n\tmov.b64 v, {%0, %1};\n\tmov.b64 h, {%2, %3};\n\tsub.rn.f32x2 v, v, h;\n\tmov.b64 {%0, %1}, v;\n\t}"
        : "+f"(x), "+f"(y) : "r"(p & 0xffff0000u), "r"(q & 0xffff0000u));
    return __byte_perm(p, q, 0x7632);
}
__device__ __forceinline__ uint32_t cut_pair(float x, float y) { return __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632); }

// Weights: cut off (byte moves and masks; the conversion to bfloat16 issues at a quarter of their rate).
__device__ __forceinline__ void split_weights(float x, float y, uint32_t& a, uint32_t& b, uint32_t& c) {
    scale_pair(x, y);
    a = leading_pair<false>(x, y);
    b = leading_pair<false>(x, y);
    c = cut_pair(x, y);
}
// Tokens, four values of a row at a time (k, k + 1 in the first of two words): the first two parts rounded to nearest (a tie away from
// zero), so that what is left out of a product has either sign. Where one of the four has a third part, 2^-25 of each is added to
// it, against the two cuts of a block's leading sum, which take off some 0.9 x 2^-24 of numbers of one sign: as much as leaves sums that are
// exact as they are (with 3/4 of 2^-24 numbers just below a power of two came back a last bit larger from a product with one).
__device__ __forceinline__ void split_tokens(const float4& v, uint32_t* a, uint32_t* b, uint32_t* c) {
    float x[4] = {v.x, v.y, v.z, v.w}, whole[4];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        scale_pair(x[2 * i], x[2 * i + 1]);
        whole[2 * i] = x[2 * i];
        whole[2 * i + 1] = x[2 * i + 1];
        a[i] = leading_pair<true>(x[2 * i], x[2 * i + 1]);
        b[i] = leading_pair<true>(x[2 * i], x[2 * i + 1]);
    }
    const uint32_t any = (__float_as_uint(x[0]) | __float_as_uint(x[1])) | (__float_as_uint(x[2]) | __float_as_uint(x[3]));
    const float share = any ? 0x1p-25f : 0.f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        asm("{\n\t.reg .b64 v, h, f;\n\tmov.b64 v, {%0, %1};\n\tmov.b64 h, {%2, %3};\n\tmov.b64 f, {%4, %4};\n\tfma.rn.f32x2 v, h, f, v;\n\t"
            "mov.b64 {%0, %1}, v;\n\t}" : "+f"(x[2 * i]), "+f"(x[2 * i + 1]) : "f"(whole[2 * i]), "f"(whole[2 * i + 1]), "f"(share));
        c[i] = cut_pair(x[2 * i], x[2 * i + 1]);
    }
}

// The values are formed here and not where they are used, behind a wait: the time from the end of a block's MMAs to the buffer's next
// ones is what bounds the kernel.
__device__ __forceinline__ void keep_here(uint32_t* v, int n) {
#pragma unroll
    for (int j = 0; j < n; ++j) asm volatile("" : "+r"(v[j]));
}

// The rows of A in three parts [3][M][K rounded up to 8] of bfloat16, once for all the tiles that read them.
__global__ void __launch_bounds__(256)
split_rows_kernel(const float* __restrict__ A, uint16_t* __restrict__ parts, int M, int K, int lda, int ldp) {
    lp_grid_wait();
    lp_grid_release();
    const long long pieces = (long long)M * (K / 4);
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < pieces; i += (long long)gridDim.x * 256) {
        const int m = (int)(i / (K / 4)), k = (int)(i % (K / 4)) * 4;
        const float4 v = *(const float4*)(A + (long long)m * lda + k);
        uint32_t p[3][2];
        split_tokens(v, p[0], p[1], p[2]);
#pragma unroll
        for (int q = 0; q < 3; ++q) *(uint2*)(parts + ((long long)q * M + m) * ldp + k) = make_uint2(p[q][0], p[q][1]);
    }
}

// The product of two rows by multiply-adds, in the order of gemm_plain_kernel: for outputs that are no finite numbers in parts.
__device__ __noinline__ float row_product(const float* a, const float* w, int K) {
    const int part = part_length(K);
    float total = 0.f;
    for (int k0 = 0; k0 < K; k0 += part) {
        float s = 0.f;
        for (int k = k0; k < min(K, k0 + part); ++k) s = fmaf(a[k], w[k], s);
        total += s;
    }
    return total;
}

// SPLIT: the gridDim.z CTAs of a cluster form PARTS / gridDim.z chains each and add them up through distributed shared memory: two
// CTAs a half's sum each, four or eight CTAs the single chains.
template <int TOK, int MODE, bool SPLIT>
__global__ void __launch_bounds__(SplitTile<TOK>::THREADS, 1)
gemm_f32_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const float* __restrict__ A,
                      const float* __restrict__ W, float* __restrict__ C, int M, int N, int K, int lda, int ldw, int ldc,
                      int* __restrict__ status) {
    using T = SplitTile<TOK>;
    constexpr bool GATED = MODE == LP_GEMM_SWIGLU;
    constexpr int FEATURES = GATED ? 64 : 128;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* token_ring = smem + T::STAGES * T::W_BYTES;
    float* first_half = (float*)(smem + T::RING);
    uint64_t* full = (uint64_t*)(smem + T::RING + T::HALF);
    uint64_t* empty = full + T::STAGES;
    uint64_t* x_full = empty + T::STAGES;          // the tokens' ring
    uint64_t* x_empty = x_full + T::X_STAGES;
    uint64_t* ready = x_empty + T::X_STAGES;       // [2] a block's operands are made, and the sums before it are fetched
    uint64_t* formed = ready + 2;                  // [2] its MMAs have ended: the operands may go, the sums are there
    uint64_t* turn = formed + 2;                   // [2] whose MMAs are issued next
    uint32_t* tmem_slot = (uint32_t*)(turn + 2);
    volatile uint32_t* failed = tmem_slot + 1;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int token_tiles = (M + TOK - 1) / TOK;                 // token tile first: a weight tile's readers run together
    const int m0 = (int)(blockIdx.x % token_tiles) * TOK, n0 = (int)(blockIdx.x / token_tiles) * FEATURES;
    const int part = part_length(K);
    const int share = SPLIT ? PARTS / (int)gridDim.z : PARTS;    // chains of this CTA
    const int k_begin = SPLIT ? min(K, (int)blockIdx.z * share * part) : 0;
    const int k_end = SPLIT ? min(K, k_begin + share * part) : K;
    const int blocks = (k_end - k_begin + SPLIT_K - 1) / SPLIT_K;
    const int chain_blocks = part / SPLIT_K;

    lp_grid_release();
    if (tid == 0) {
        *failed = 0;
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
        for (int s = 0; s < T::STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 4); }
        for (int s = 0; s < T::X_STAGES; ++s) { mbar_init(&x_full[s], 1); mbar_init(&x_empty[s], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&ready[i], 4 + T::ADDERS); mbar_init(&formed[i], 1); mbar_init(&turn[i], 1); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)T::TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem = *tmem_slot;
    if (warp != 0) lp_grid_wait();
    bool done = false;                               // this adding thread's sums are whole
    float sum[T::COLS];                              // of the chain that is being formed, at the end (of one chain, or not SPLIT) the whole

    auto all_wait = [&](uint64_t* bar, int parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity)); };
    auto give_up = [&](int code) {
        if (lane == 0) atomicExch(status, code);
        *failed = 1;
    };

    if (warp == 0) {
        if (lane == 0) {
            auto weights = [&](int b) {
                const int s = b % T::STAGES;
                mbar_expect_tx(&full[s], T::W_BYTES);
                uint8_t* to = smem + s * T::W_BYTES;
                tma_load_2d(to, &map_w, k_begin + b * SPLIT_K, n0, &full[s]);
                if (GATED) tma_load_2d(to + T::W_BYTES / 2, &map_w, k_begin + b * SPLIT_K, N + n0, &full[s]);
            };
            // this thread reads nothing but weights, and split_rows_kernel lets this kernel start only when all before it has ended: no wait
            int b = 0;
            for (; b < blocks; ++b) {
                if (!mbar_wait(&empty[b % T::STAGES], ((b / T::STAGES) & 1) ^ 1)) { atomicExch(status, 71); *failed = 1; break; }
                weights(b);
            }
            if (b < blocks)                          // gave up: no copy may be in flight when the CTA ends
                for (int i = max(0, b - T::STAGES); i < b; ++i) mbar_wait(&full[i % T::STAGES], (i / T::STAGES) & 1);
        }
        __syncwarp();
    } else if (warp == 2) {
        if (lane == 0) {
            constexpr int RING = T::X_STAGES;
            int b = 0;
            for (; b < blocks; ++b) {
                const int s = b % RING;
                if (!mbar_wait(&x_empty[s], ((b / RING) & 1) ^ 1)) { atomicExch(status, 70); *failed = 1; break; }
                mbar_expect_tx(&x_full[s], T::X_STAGE);
                uint8_t* to = token_ring + s * T::X_STAGE;
#pragma unroll
                for (int q = 0; q < 3; ++q) tma_load_2d(to + q * T::PART, &map_x, k_begin + b * SPLIT_K, q * M + m0, &x_full[s]);
            }
            if (b < blocks)
                for (int i = max(0, b - RING); i < b; ++i) mbar_wait(&x_full[i % RING], (i / RING) & 1);
        }
        __syncwarp();
    } else if (warp == 1 || warp == 3) {
        // Two warps issue, one block each in turn: behind its MMAs a warp's next wait takes some 400 cycles to return. They take turns,
        // or the MMAs of two blocks would mix and both blocks end late.
        constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TOK >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        constexpr int RING = T::X_STAGES;
        const int i = warp >> 1;
        const uint32_t d = tmem + T::SUMS + i * TOK, a = tmem + T::WEIGHTS + i * 48;
        for (int b = i; b < blocks; b += 2) {
            const int s = b % RING;
            bool ok = true;
            if (lane == 0) {
                ok = mbar_wait(&x_full[s], (b / RING) & 1);
                if (ok) ok = mbar_wait(&ready[i], (b >> 1) & 1);
                if (ok && b > 0) ok = mbar_wait(&turn[i], ((b - 1) >> 1) & 1);
                if (ok) {
                    tcgen05_fence_after();
                    const uint64_t x = smem_desc_rows64(smem_u32(token_ring + s * T::X_STAGE));
                    constexpr uint64_t P = T::PART >> 4;
                    uint32_t more = 0;
#pragma unroll
                    for (int k = 0; k < 2; ++k) {    // parts 0 (leading) to 2 of 16 products: 8 columns of weights, 32 bytes of tokens
                        const uint32_t w = a + k * 8;
                        const uint64_t t = x + k * 2;
                        split_mma(d, w + 16, t + P, idesc, more);
                        more = 1;
                        split_mma(d, w, t + 2 * P, idesc, 1);
                        split_mma(d, w + 32, t, idesc, 1);
                        if (k == 1) mbar_arrive(&turn[i ^ 1]);       // it arrives behind the MMAs issued so far
                        split_mma(d, w, t + P, idesc, 1);
                        split_mma(d, w + 16, t, idesc, 1);
                    }
#pragma unroll
                    for (int k = 0; k < 2; ++k) split_mma(d, a + k * 8, x + k * 2, idesc, 1);
                    tcgen05_commit(&formed[i]);
                    tcgen05_commit(&x_empty[s]);
                }
            }
            if (!ok) { give_up(72); break; }
        }
        __syncwarp();
    } else if (warp >= 4 && warp < T::FIRST_ADDER) {
        const uint32_t row_addr = (uint32_t)((warp & 3) * 32) << 16;
        const int row = (warp & 3) * 32 + lane;
        const int begin = T::GROUPS == 2 ? (warp - 4) >> 2 : 0;
        constexpr bool AHEAD = T::GROUPS == 1;       // the next block's values are asked for before the wait for the last one's MMAs
        float4 v[8];
        auto fetch = [&](int b) {
            const int s = b % T::STAGES;
            if (!all_wait(&full[s], (b / T::STAGES) & 1)) return false;
            const uint8_t* from = smem + s * T::W_BYTES;
#pragma unroll
            for (int c = 0; c < 8; ++c) v[c] = *(const float4*)(from + row * 128 + ((c ^ (row & 7)) << 4));
            return true;
        };
        if (AHEAD && begin < blocks && !fetch(begin)) give_up(74);
        for (int b = begin; b < blocks; b += T::GROUPS) {
            const int s = b % T::STAGES, i = b & 1;
            if (!AHEAD && !fetch(b)) { give_up(74); break; }
            uint32_t p[3][16];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                split_weights(v[c].x, v[c].y, p[0][2 * c], p[1][2 * c], p[2][2 * c]);
                split_weights(v[c].z, v[c].w, p[0][2 * c + 1], p[1][2 * c + 1], p[2][2 * c + 1]);
            }
            keep_here(&p[0][0], 48);
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[s]);
            if (AHEAD && b + 1 < blocks && !fetch(b + 1)) { give_up(74); break; }
            if (!all_wait(&formed[i], ((b >> 1) & 1) ^ 1)) { give_up(75); break; }
            tcgen05_fence_after();
#pragma unroll
            for (int q = 0; q < 3; ++q) tmem_st16(tmem + T::WEIGHTS + i * 48 + q * 16 + row_addr, p[q]);
            tmem_st_wait();
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ready[i]);
        }
    } else if (warp >= T::FIRST_ADDER) {
        // a thread: one weight row (its lane of tensor memory), COLS tokens
        const int half = (warp - T::FIRST_ADDER) >> 2;
        const uint32_t lane_addr = ((uint32_t)((warp & 3) * 32) << 16) + half * T::COLS;
        if (lane == 0) { mbar_arrive(&ready[0]); mbar_arrive(&ready[1]); }         // nothing to fetch before the first two blocks
        int in_chain = 0, chain = 0;
        bool ok = true;
        for (int b = 0; b < blocks; ++b) {
            const int i = b & 1;
            if (!all_wait(&formed[i], (b >> 1) & 1)) { give_up(78); ok = false; break; }
            tcgen05_fence_after();
#pragma unroll
            for (int c = 0; c < T::COLS; c += 32) {
                uint32_t r[32];
                tmem_ld32(tmem + T::SUMS + i * TOK + lane_addr + c, r);
                tmem_ld_wait();
                if (in_chain == 0) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) sum[c + j] = __uint_as_float(r[j]);
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j) sum[c + j] += __uint_as_float(r[j]);
                }
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0 && b + 2 < blocks) mbar_arrive(&ready[i]);
            if (++in_chain < chain_blocks && b + 1 < blocks) continue;
            in_chain = 0;                            // a chain ends
            const bool apart = SPLIT && share < PARTS / 2, again = !SPLIT && chain == PARTS / 2 - 1;
            if (!apart && chain % (PARTS / 2) > 0) { // it joins those of its half
#pragma unroll
                for (int c = 0; c < T::COLS; c += 16) {
                    uint32_t r[16];
                    tmem_ld16(tmem + T::HELD + lane_addr + c, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) sum[c + j] = __uint_as_float(r[j]) + sum[c + j];
                }
            }
            const bool last = b + 1 == blocks;
            if (T::HALF && again && !last) {         // the first half is whole
#pragma unroll
                for (int j = 0; j < T::COLS; ++j) first_half[(half * T::COLS + j) * 128 + (warp & 3) * 32 + lane] = sum[j];
            } else if (!last || (apart && T::SLOTS > 1)) {
                const int slot = apart ? chain : again ? 1 : 0;
#pragma unroll
                for (int c = 0; c < T::COLS; c += 16) {
                    uint32_t r[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(sum[c + j]);
                    tmem_st16(tmem + T::HELD + slot * TOK + lane_addr + c, r);
                }
                tmem_st_wait();
            }
            ++chain;
        }
        if (!SPLIT && chain > PARTS / 2) {           // both halves
#pragma unroll
            for (int c = 0; c < T::COLS; c += 16) {
                uint32_t r[16];
                if (T::HALF) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(first_half[(half * T::COLS + c + j) * 128 + (warp & 3) * 32 + lane]);
                } else {
                    tmem_ld16(tmem + T::HELD + TOK + lane_addr + c, r);
                    tmem_ld_wait();
                }
#pragma unroll
                for (int j = 0; j < 16; ++j) sum[c + j] = __uint_as_float(r[j]) + sum[c + j];
            }
        }
        done = ok;
    }

    const int quarter = warp & 3, column0 = (warp - T::FIRST_ADDER) / 4 * T::COLS;      // of an adding warp
    const bool adder = warp >= T::FIRST_ADDER;
    auto weight_row = [&](int f) { return W + (long long)f * ldw; };
    auto whole = [&](float v, int m, int f) {       // a sum that is no finite number is formed again
        return fabsf(v) < INFINITY ? v * SUM_SCALE : row_product(A + (long long)m * lda, weight_row(f), K);
    };
    auto store = [&](int m, int f, float v) {
        float* c = C + (long long)m * ldc + f;
        *c = MODE == LP_GEMM_ACCUMULATE ? *c + v : v;
    };
    if constexpr (SPLIT) {
        cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
        const int chains = (K + part - 1) / part;    // of the whole
        const bool apart = share < PARTS / 2;
        float* sums = (float*)smem;                  // [slot][token][weight row]; every copy and MMA that used this memory has ended
        if (adder && done && blocks > 0) {
            if (apart && T::SLOTS > 1) {
                const int here = min(share, chains - (int)blockIdx.z * share);
                for (int q = 0; q < here; ++q) {
#pragma unroll
                    for (int c = 0; c < T::COLS; c += 16) {
                        uint32_t r[16];
                        tmem_ld16(tmem + T::HELD + q * TOK + ((uint32_t)(quarter * 32) << 16) + column0 + c, r);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; ++j) sums[((size_t)q * TOK + column0 + c + j) * 128 + quarter * 32 + lane] = __uint_as_float(r[j]);
                    }
                }
            } else {
#pragma unroll
                for (int j = 0; j < T::COLS; ++j) sums[(column0 + j) * 128 + quarter * 32 + lane] = sum[j];
            }
        }
        __syncthreads();
        cluster.sync();
        const int tokens = TOK / (int)gridDim.z;     // of the tile, finished by this CTA
        uint32_t bad = 0;
        for (int c = 0; c < (int)gridDim.z; ++c) bad |= *(volatile uint32_t*)cluster.map_shared_rank((uint32_t*)failed, c);
        if (!bad) {
            for (int e = tid; e < tokens * FEATURES; e += T::THREADS) {
                const int t = (int)blockIdx.z * tokens + e / FEATURES, f = e % FEATURES;
                const int m = m0 + t, n = n0 + f;
                if (m >= M || n >= N) continue;
                float g = 0.f, u = 0.f, g0 = 0.f, u0 = 0.f;
                const int step = apart ? 1 : share;  // chains per sum
                for (int c = 0; c < chains; c += step) {
                    const float* from = cluster.map_shared_rank(sums, c / share) + ((apart ? c % share : 0) * TOK + t) * 128 + f;
                    const bool starts = c % (PARTS / 2) == 0;
                    if (starts) { g0 = g; u0 = u; }
                    g = starts ? from[0] : g + from[0];
                    if (GATED) u = starts ? from[64] : u + from[64];
                }
                if (chains > PARTS / 2) { g = g0 + g; u = u0 + u; }
                if (GATED) C[(long long)m * ldc + n] = silu_mul(whole(g, m, n), whole(u, m, N + n));
                else store(m, n, whole(g, m, n));
            }
        }
        cluster.sync();                              // nobody leaves while its sums are still read
    } else if constexpr (GATED) {
        float* up = (float*)smem;                    // [token][feature]
        if (adder && quarter >= 2) {
#pragma unroll
            for (int j = 0; j < T::COLS; ++j) up[(column0 + j) * 64 + (quarter - 2) * 32 + lane] = sum[j];
        }
        __syncthreads();
        const int f = quarter * 32 + lane, n = n0 + f;
        if (adder && quarter < 2 && n < N && !*failed) {
#pragma unroll
            for (int j = 0; j < T::COLS; ++j) {
                const int m = m0 + column0 + j;
                if (m < M) C[(long long)m * ldc + n] = silu_mul(whole(sum[j], m, n), whole(up[(column0 + j) * 64 + f], m, N + n));
            }
        }
    } else {
        __syncthreads();
        const int n = n0 + quarter * 32 + lane;
        if (adder && n < N && !*failed) {
#pragma unroll
            for (int j = 0; j < T::COLS; ++j) {
                const int m = m0 + column0 + j;
                if (m < M) store(m, n, whole(sum[j], m, n));
            }
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) {
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)T::TMEM_COLS));
    }
}

// ---------------------------------------------------------------- float32, a handful of rows
// A step of a few sequences reads every weight once and is bound by that: 16 weight rows (in the gated form 8 gate and 8 up rows) x
// 8 or 16 tokens per CTA and turn, a warp per chain of K. A warp copies its own stages, splits them in
// registers and multiplies them with mma.sync, whose sums of 16 products are those of tcgen05.mma bit for bit: same steps, same
// order, so a row's result is the same as in the tiles above. Nothing but the chains' sums crosses warps. Bound by the copies in flight,
// the splitting (100 of some 170 instructions per warp and block of 2 KB) and the chain of twelve MMAs per block. B200, the four products of a layer of width
// 2048 one behind the other (243 MB), by a thread per chain and weight row with multiply-adds / in parts, us: 1 row 53 / 54, 2 rows 55 / 56, 4 rows 62 / 56, 8 rows
// 93 / 60, 16 rows 165 / 85.
constexpr int ROW_FEATURES = 16;

template <int TOK, bool DEEP> struct RowsShape {
    static constexpr int THREADS = PARTS * 32;
    static constexpr int STAGE = (ROW_FEATURES + TOK) * 128;      // bytes of a warp's stage: rows of 32 values
    // two CTAs per SM; DEEP: one, for grids that have no more (four products of 16 rows: 85 us, 106 with the short ring everywhere)
    static constexpr int STAGES = (DEEP ? 200 : 96) * 1024 / (PARTS * STAGE);
    static constexpr int TOGETHER = DEEP && TOK == 8 ? 2 : 1;     // blocks whose MMAs (a chain of twelve) run side by side
    static constexpr size_t SMEM = (size_t)PARTS * STAGES * STAGE;
};

__device__ __forceinline__ void copy16(void* smem, const void* gmem, bool real) {
    const unsigned to = (unsigned)__cvta_generic_to_shared(smem);
    const int bytes = real ? 16 : 0;       // the rest of the 16 bytes is zero
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void mma_16x8(float* c, const uint32_t* a, const uint32_t* b) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

template <int TOK, int MODE, bool DEEP>
__global__ void __launch_bounds__(PARTS * 32, DEEP ? 1 : 2)
gemm_f32_rows_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K,
                     int lda, int ldw, int ldc) {
    using S = RowsShape<TOK, DEEP>;
    constexpr bool GATED = MODE == LP_GEMM_SWIGLU;
    constexpr int FEATURES = GATED ? ROW_FEATURES / 2 : ROW_FEATURES, TILES = TOK / 8;
    extern __shared__ __align__(128) uint8_t rows_smem[];
    __shared__ float sums[PARTS][TOK][ROW_FEATURES];
    const int tid = threadIdx.x, chain = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int n0 = blockIdx.x * FEATURES;
    const int part = part_length(K);
    const int k_begin = min(K, chain * part), k_end = min(K, k_begin + part);
    const int blocks = (k_end - k_begin + SPLIT_K - 1) / SPLIT_K;
    uint8_t* ring = rows_smem + chain * S::STAGES * S::STAGE;

    // 16-byte piece c of row r lies at piece c ^ 4 (r % 2): the eight lanes that are served together read two rows
    const int piece = lane & 7, copy_row = lane >> 3;             // rows copy_row, + 4, + 8, ...
    auto weight_row = [&](int r) { return GATED ? (r < FEATURES ? n0 + r : N + n0 + r - FEATURES) : n0 + r; };
    auto feature_real = [&](int r) { return n0 + (GATED ? r % FEATURES : r) < N; };
    const float* from_w[4];                          // (rows that there are not repeat the first: their sums go nowhere)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = copy_row + i * 4;
        from_w[i] = W + (feature_real(r) ? (long long)weight_row(r) * ldw : 0);
    }
    const uint32_t to = copy_row * 128 + ((piece ^ ((copy_row & 1) * 4)) << 4);
    auto fetch_w = [&](int b) {
        if (b >= blocks) return;
        uint8_t* stage = ring + (unsigned)b % S::STAGES * S::STAGE + to;
        const int k = k_begin + b * SPLIT_K + piece * 4;
        const bool inside = k < k_end;
        const int at = inside ? k : 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) copy16(stage + i * 512, from_w[i] + at, inside);
    };
    auto fetch_x = [&](int b) {
        if (b >= blocks) return;
        uint8_t* stage = ring + (unsigned)b % S::STAGES * S::STAGE + ROW_FEATURES * 128 + to;
        const int k = k_begin + b * SPLIT_K + piece * 4;
#pragma unroll
        for (int i = 0; i < TOK / 4; ++i) {
            const int m = copy_row + i * 4;
            const bool real = m < M && k < k_end;
            copy16(stage + i * 512, real ? A + (long long)m * lda + k : A, real);
        }
    };

    // no kernel of a step writes weights: the first stages of them are asked for before the wait
#pragma unroll
    for (int b = 0; b < S::STAGES - S::TOGETHER; ++b) fetch_w(b);
    lp_grid_wait();
    lp_grid_release();
#pragma unroll
    for (int b = 0; b < S::STAGES - S::TOGETHER; ++b) {
        fetch_x(b);
        copies_commit();       // the first group also holds all weights asked for above
    }
    float sum[TILES][4];
#pragma unroll
    for (int n = 0; n < TILES; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) sum[n][i] = 0.f;
    constexpr int U = S::TOGETHER;
    for (int b = 0; b < blocks; b += U) {
        copies_wait<S::STAGES - 2 * U>();
        __syncwarp();
        // parts [part][register]: a lane's four neighbouring values of 16 are its two pairs of an operand, so products 4 t .. 4 t + 3 of a
        // step stand where the instruction counts 2 t, 2 t + 1, 2 t + 8, 2 t + 9; which of the 16 comes where does not matter to their sum
        uint32_t w[U][2][3][4], x[U][TILES][2][3][2];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint8_t* stage = ring + (unsigned)(b + u) % S::STAGES * S::STAGE;
            auto at = [&](int row, int step) { return *(const float4*)(stage + row * 128 + (((step * 4 + t) ^ ((row & 1) * 4)) << 4)); };
#pragma unroll
            for (int s = 0; s < 2; ++s) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float4 v = at(g + h * 8, s);
                    split_weights(v.x, v.y, w[u][s][0][h], w[u][s][1][h], w[u][s][2][h]);
                    split_weights(v.z, v.w, w[u][s][0][h + 2], w[u][s][1][h + 2], w[u][s][2][h + 2]);
                }
#pragma unroll
                for (int n = 0; n < TILES; ++n) {
                    const float4 v = at(ROW_FEATURES + n * 8 + g, s);
                    split_tokens(v, x[u][n][s][0], x[u][n][s][1], x[u][n][s][2]);
                }
            }
        }
        __syncwarp();                                // the stages before these are free
#pragma unroll
        for (int u = 0; u < U; ++u) {
            fetch_w(b + u + S::STAGES - U);
            fetch_x(b + u + S::STAGES - U);
            copies_commit();
        }
        float d[U][TILES][4];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int n = 0; n < TILES; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) d[u][n][i] = 0.f;
        auto product = [&](int s, int p, int q) {
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int n = 0; n < TILES; ++n) mma_16x8(d[u][n], w[u][s][p], x[u][n][s][q]);
        };
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            product(s, 1, 1);
            product(s, 0, 2);
            product(s, 2, 0);
            product(s, 0, 1);
            product(s, 1, 0);
        }
        product(0, 0, 0);
        product(1, 0, 0);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (b + u >= blocks) break;
#pragma unroll
            for (int n = 0; n < TILES; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) sum[n][i] = b + u == 0 ? d[u][n][i] : sum[n][i] + d[u][n][i];
        }
    }
    copies_wait<0>();
#pragma unroll
    for (int n = 0; n < TILES; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) sums[chain][n * 8 + t * 2 + (i & 1)][g + (i >> 1) * 8] = sum[n][i];
    __syncthreads();
    const int chains = (K + part - 1) / part;
    for (int e = tid; e < TOK * FEATURES; e += S::THREADS) {
        const int m = e / FEATURES, f = e % FEATURES;
        if (m >= M || n0 + f >= N) continue;
        auto whole = [&](int r) {
            float v = 0.f, first = 0.f;
            for (int c = 0; c < chains; ++c) {
                if (c == PARTS / 2) first = v;
                v = c % (PARTS / 2) == 0 ? sums[c][m][r] : v + sums[c][m][r];
            }
            if (chains > PARTS / 2) v = first + v;
            // a sum that is no finite number is formed again
            return fabsf(v) < INFINITY ? v * SUM_SCALE : row_product(A + (long long)m * lda, W + (long long)weight_row(r) * ldw, K);
        };
        float* out = C + (long long)m * ldc + n0 + f;
        if (GATED) *out = silu_mul(whole(f), whole(FEATURES + f));
        else if (MODE == LP_GEMM_ACCUMULATE) *out += whole(f);
        else *out = whole(f);
    }
}

// Up to 8 tokens whose parts fit shared memory: a CTA per SM walks over the tiles of features and splits the tokens once, and its weights' ring
// runs on from tile to tile. With a CTA per tile, which splits the tokens that it multiplies with again, the four products above take 61 us (1 row) to 62
// (8 rows). GROUPS of eight warps walk over tiles of their own.
template <int GROUPS_, int STAGES_, int TOGETHER_> struct FewShape {
    static constexpr int GROUPS = GROUPS_, STAGES = STAGES_, TOGETHER = TOGETHER_, THREADS = GROUPS * PARTS * 32;
    static constexpr int STAGE = ROW_FEATURES * 128;
    static constexpr int RING = GROUPS * PARTS * STAGES * STAGE, SUMS = GROUPS * 2 * PARTS * 8 * ROW_FEATURES * 4;
    static constexpr int ROOM = 225 * 1024 - RING - SUMS;            // for the tokens' parts
};
__host__ __device__ __forceinline__ int token_bytes(int K) { return part_length(K) * 6 + 32; }       // of one chain; tokens 32 bytes apart in the banks
__host__ __device__ __forceinline__ int tokens_bytes(int M, int K) { return PARTS * M * token_bytes(K) + 64; }      // (a last pair of blocks reads on)

template <int MODE, class S>
__global__ void __launch_bounds__(S::THREADS, 1)
gemm_f32_few_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K, int lda, int ldw,
                    int ldc) {
    constexpr bool GATED = MODE == LP_GEMM_SWIGLU;
    constexpr int FEATURES = GATED ? ROW_FEATURES / 2 : ROW_FEATURES, U = S::TOGETHER;
    extern __shared__ __align__(128) uint8_t few_smem[];
    const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int group = tid / (PARTS * 32), chain = (tid >> 5) % PARTS;
    const int part = part_length(K);
    const int k_begin = min(K, chain * part), k_end = min(K, k_begin + part);
    const int blocks = (k_end - k_begin + SPLIT_K - 1) / SPLIT_K, steps = (blocks + U - 1) / U * U;
    uint8_t* ring = few_smem + (group * PARTS + chain) * S::STAGES * S::STAGE;
    float* sums = (float*)(few_smem + S::RING) + group * 2 * PARTS * 8 * ROW_FEATURES;       // [2][chain][token][weight row]
    uint8_t* parts = few_smem + S::RING + S::SUMS;
    const int x_row = token_bytes(K);
    uint8_t* xs = parts + chain * M * x_row;                        // [token][part][value] of this chain
    const int tiles = (N + FEATURES - 1) / FEATURES, stride = (int)gridDim.x * S::GROUPS;
    const int first = (int)blockIdx.x + group * (int)gridDim.x;

    // copies: 16-byte piece c of row r lies at piece c ^ 4 (r % 2): the eight lanes that are served together read two rows
    const int piece = lane & 7, copy_row = lane >> 3;
    const uint32_t to = copy_row * 128 + ((piece ^ ((copy_row & 1) * 4)) << 4);
    auto weight_row = [&](int n0, int r) { return GATED ? (r < FEATURES ? n0 + r : N + n0 + r - FEATURES) : n0 + r; };
    const float* from_w[4];
    int next_tile = first, next_block = 0, next_slot = 0;
    auto fetch = [&]() {                                            // the next block of this chain, of this tile or the one behind it
        if (next_tile < tiles) {
            if (next_block == 0) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int r = copy_row + i * 4, n0 = next_tile * FEATURES;      // (rows that there are not repeat the first: their sums go nowhere)
                    from_w[i] = W + (n0 + (GATED ? r % FEATURES : r) < N ? (long long)weight_row(n0, r) * ldw : 0);
                }
            }
            const int k = k_begin + next_block * SPLIT_K + piece * 4;
            const bool inside = k < k_end;
            const int at = inside ? k : 0;
            uint8_t* stage = ring + next_slot * S::STAGE + to;
#pragma unroll
            for (int i = 0; i < 4; ++i) copy16(stage + i * 512, from_w[i] + at, inside);
            if (++next_block == steps) {
                next_block = 0;
                next_tile += stride;
            }
        }
        next_slot = next_slot + 1 == S::STAGES ? 0 : next_slot + 1;
        copies_commit();
    };
    // no kernel of a step writes weights: the first stages of them are asked for before the wait
    if (steps > 0)
#pragma unroll
        for (int b = 0; b < S::STAGES - U; ++b) fetch();
    lp_grid_wait();
    lp_grid_release();
    const int quads = part / 4;
#pragma unroll 4
    for (int e = lane + group * 32; e < M * quads; e += 32 * S::GROUPS) {
        const int m = e / quads, k = (e - m * quads) * 4;
        const float4 v = k_begin + k < k_end ? *(const float4*)(A + (long long)m * lda + k_begin + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        uint32_t p[3][2];
        split_tokens(v, p[0], p[1], p[2]);
#pragma unroll
        for (int q = 0; q < 3; ++q) *(uint2*)(xs + m * x_row + (q * part + k) * 2) = make_uint2(p[q][0], p[q][1]);
    }
    __syncthreads();
    const bool x_real = g < M;                                      // columns of tokens that there are not go nowhere
    const uint8_t* x_from = xs + (x_real ? g : 0) * x_row + t * 8;
    const int chains = (K + part - 1) / part;
    int slot = 0, turn = 0;
    for (int tile = first; tile < tiles; tile += stride, turn ^= 1) {
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
        for (int b = 0; b < steps; b += U) {
            copies_wait<S::STAGES - 2 * U>();
            __syncwarp();
            // parts [part][register]: a lane's four neighbouring values of 16 are its two pairs of an operand, so products 4 t .. 4 t + 3 of a
            // step stand where the instruction counts 2 t, 2 t + 1, 2 t + 8, 2 t + 9; which of the 16 comes where does not matter to their sum
            uint32_t w[U][2][3][4];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const uint8_t* stage = ring + slot * S::STAGE;
                auto at = [&](int row, int step) { return *(const float4*)(stage + row * 128 + (((step * 4 + t) ^ ((row & 1) * 4)) << 4)); };
#pragma unroll
                for (int s = 0; s < 2; ++s)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const float4 v = at(g + h * 8, s);
                        split_weights(v.x, v.y, w[u][s][0][h], w[u][s][1][h], w[u][s][2][h]);
                        split_weights(v.z, v.w, w[u][s][0][h + 2], w[u][s][1][h + 2], w[u][s][2][h + 2]);
                    }
                slot = slot + 1 == S::STAGES ? 0 : slot + 1;
            }
            __syncwarp();                                           // the stages are free
#pragma unroll
            for (int u = 0; u < U; ++u) fetch();
            uint2 x[U][2][3];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int s = 0; s < 2; ++s)
#pragma unroll
                    for (int q = 0; q < 3; ++q)
                        x[u][s][q] = x_real ? *(const uint2*)(x_from + (q * part + (b + u) * SPLIT_K + s * 16) * 2) : make_uint2(0, 0);
            float d[U][4] = {};
            auto product = [&](int s, int p, int q) {
#pragma unroll
                for (int u = 0; u < U; ++u) mma_16x8(d[u], w[u][s][p], (const uint32_t*)&x[u][s][q]);
            };
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                product(s, 1, 1);
                product(s, 0, 2);
                product(s, 2, 0);
                product(s, 0, 1);
                product(s, 1, 0);
            }
            product(0, 0, 0);
            product(1, 0, 0);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (b + u >= blocks) break;
#pragma unroll
                for (int i = 0; i < 4; ++i) sum[i] = b + u == 0 ? d[u][i] : sum[i] + d[u][i];
            }
        }
        float* mine = sums + turn * PARTS * 8 * ROW_FEATURES;       // the other half may still be read for the tile before
#pragma unroll
        for (int i = 0; i < 4; ++i) mine[(chain * 8 + t * 2 + (i & 1)) * ROW_FEATURES + g + (i >> 1) * 8] = sum[i];
        if (S::GROUPS == 1) __syncthreads();
        else asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(PARTS * 32) : "memory");
        const int e = tid % (PARTS * 32), m = e / FEATURES, f = e % FEATURES, n0 = tile * FEATURES;
        if (m >= M || n0 + f >= N) continue;
        auto whole = [&](int r) {
            const float* from = mine + m * ROW_FEATURES + r;
            float v = 0.f, half = 0.f;
            for (int c = 0; c < chains; ++c) {
                const float s = from[c * 8 * ROW_FEATURES];
                if (c == PARTS / 2) half = v;
                v = c % (PARTS / 2) == 0 ? s : v + s;
            }
            if (chains > PARTS / 2) v = half + v;
            // a sum that is no finite number is formed again
            return fabsf(v) < INFINITY ? v * SUM_SCALE : row_product(A + (long long)m * lda, W + (long long)weight_row(n0, r) * ldw, K);
        };
        float* out = C + (long long)m * ldc + n0 + f;
        if (GATED) *out = silu_mul(whole(f), whole(FEATURES + f));
        else if (MODE == LP_GEMM_ACCUMULATE) *out += whole(f);
        else *out = whole(f);
    }
    copies_wait<0>();
}

// ---------------------------------------------------------------- choice and launch
int failed(cudaError_t err, const char* what) {
    snprintf(lp_error_text, sizeof(lp_error_text), "gemm_plain (%s): %s", what, cudaGetErrorString(err));
    return (int)err;
}

// [rows, K] bfloat16, row stride ld, boxes of box_rows x 32 (64 bytes, swizzled)
int make_map_rows64(CUtensorMap* map, const void* base, long long rows, long long K, long long ld, int box_rows) {
    EncodeTiled enc = encode_fn();
    if (!enc) LP_REFUSE("gemm: the driver does not offer cuTensorMapEncodeTiled");
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {(cuuint32_t)SPLIT_K, (cuuint32_t)box_rows};
    cuuint32_t elem[2] = {1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) LP_REFUSE("gemm: cuTensorMapEncodeTiled failed with code %d for a [%lld, %lld] matrix of parts",
                                     (int)r, rows, K);
    return 0;
}

struct F32Call {
    const float *A, *W;
    float* C;
    int M, N, K, lda, ldw, ldc;
    uint16_t* parts;           // room for the parts of A (lp_gemm_plain), or null
    int* status;
    cudaStream_t stream;
};

template <int TOK, int MODE, bool SPLIT>
int launch_split(const F32Call& c, int ctas) {
    using T = SplitTile<TOK>;
    constexpr int FEATURES = MODE == LP_GEMM_SWIGLU ? 64 : 128;
    CUtensorMap mw, mx;
    int rc = make_map_f32(&mw, c.W, MODE == LP_GEMM_SWIGLU ? 2ll * c.N : c.N, c.K, c.ldw, FEATURES);
    if (!rc) rc = make_map_rows64(&mx, c.parts, 3ll * c.M, c.K, (c.K + 7) / 8 * 8, TOK);
    if (rc) return rc;
    const long long pieces = (long long)c.M * (c.K / 4);
    cudaError_t err = lp_launch(split_rows_kernel, (unsigned)min((pieces + 255) / 256, (long long)lp_sm_count() * 8), 256, 0, c.stream,
                                c.A, c.parts, c.M, c.K, c.lda, (c.K + 7) / 8 * 8);
    if (err != cudaSuccess) return failed(err, "parts");
    auto kernel = gemm_f32_split_kernel<TOK, MODE, SPLIT>;
    err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::SMEM);
    if (err != cudaSuccess) return failed(err, "float32");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((c.M + TOK - 1) / TOK) * ((c.N + FEATURES - 1) / FEATURES), 1, ctas);
    cfg.blockDim = dim3(T::THREADS);
    cfg.dynamicSmemBytes = T::SMEM;
    cfg.stream = c.stream;
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
        attr[attrs++].val.clusterDim.z = ctas;
    }
    cfg.attrs = attr;
    cfg.numAttrs = attrs;
    err = cudaLaunchKernelEx(&cfg, kernel, mw, mx, c.A, c.W, c.C, c.M, c.N, c.K, c.lda, c.ldw, c.ldc, c.status);
    return err == cudaSuccess ? lp_check_launch("gemm_plain (float32)") : failed(err, "float32");
}

template <int TOK, int MODE>
int launch_tokens(const F32Call& c) {
    using T = SplitTile<TOK>;
    constexpr int FEATURES = MODE == LP_GEMM_SWIGLU ? 64 : 128;
    const long long tiles = (long long)((c.N + FEATURES - 1) / FEATURES) * ((c.M + TOK - 1) / TOK);
    const long long blocks = (c.K + SPLIT_K - 1) / SPLIT_K;
    // how many CTAs share a tile's chains: the number whose busiest SM has least to do, a CTA's beginning and end counted as eight blocks (as none, the
    // four products take 480 us for 509 rows and 213 for 17, as four 420 and 170, as eight 420 and 170, as sixteen 441 and 169)
    int best = 1;
    long long least = 0;
    for (int ctas = 1; ctas <= PARTS; ctas *= 2) {
        if (ctas > 1 && (c.K <= SPLIT_K * PARTS || (ctas > 2 && PARTS / ctas > T::SLOTS))) continue;
        const long long each = (tiles * ctas + lp_sm_count() - 1) / lp_sm_count();            // CTAs of the busiest SM
        const long long cost = each * ((blocks + ctas - 1) / ctas + 8);
        if (ctas == 1 || cost < least) { best = ctas; least = cost; }
    }
    return best > 1 ? launch_split<TOK, MODE, true>(c, best) : launch_split<TOK, MODE, false>(c, 1);
}

template <int TOK, int MODE, bool DEEP>
int launch_rows_as(const F32Call& c) {
    using S = RowsShape<TOK, DEEP>;
    constexpr int FEATURES = MODE == LP_GEMM_SWIGLU ? ROW_FEATURES / 2 : ROW_FEATURES;
    auto kernel = gemm_f32_rows_kernel<TOK, MODE, DEEP>;
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
    if (err == cudaSuccess)
        err = lp_launch(kernel, dim3((c.N + FEATURES - 1) / FEATURES), dim3(S::THREADS), S::SMEM, c.stream, c.A, c.W, c.C, c.M, c.N, c.K,
                        c.lda, c.ldw, c.ldc);
    return err == cudaSuccess ? lp_check_launch("gemm_plain (rows)") : failed(err, "rows");
}

template <int TOK, int MODE>
int launch_rows(const F32Call& c) {
    constexpr int FEATURES = MODE == LP_GEMM_SWIGLU ? ROW_FEATURES / 2 : ROW_FEATURES;
    return (c.N + FEATURES - 1) / FEATURES <= lp_sm_count() ? launch_rows_as<TOK, MODE, true>(c) : launch_rows_as<TOK, MODE, false>(c);
}

template <int MODE, class S>
int launch_few_as(const F32Call& c) {
    constexpr int FEATURES = MODE == LP_GEMM_SWIGLU ? ROW_FEATURES / 2 : ROW_FEATURES;
    auto kernel = gemm_f32_few_kernel<MODE, S>;
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::RING + S::SUMS + S::ROOM);
    const int tiles = (c.N + FEATURES - 1) / FEATURES;
    if (err == cudaSuccess)
        err = lp_launch(kernel, dim3(min(tiles, lp_sm_count())), dim3(S::THREADS), S::RING + S::SUMS + tokens_bytes(c.M, c.K), c.stream, c.A,
                        c.W, c.C, c.M, c.N, c.K, c.lda, c.ldw, c.ldc);
    return err == cudaSuccess ? lp_check_launch("gemm_plain (few)") : failed(err, "few");
}

template <int MODE>
int launch_few(const F32Call& c) {
    constexpr int FEATURES = MODE == LP_GEMM_SWIGLU ? ROW_FEATURES / 2 : ROW_FEATURES;
    const int tokens = c.K <= 65536 ? tokens_bytes(c.M, c.K) : 1 << 30;
    // with a tile per SM or fewer a second group would have nothing to do, and two blocks' MMAs run side by side instead (four products of one row
    // with two groups everywhere: 55 us, so 54); the ring gives way to the tokens (8 rows of 2048: 60 us, 62 with gemm_f32_rows_kernel)
    using Alone = FewShape<1, 6, 2>;
    using Wide = FewShape<2, 4, 1>;
    using Tight = FewShape<2, 3, 1>;
    if ((c.N + FEATURES - 1) / FEATURES <= lp_sm_count() && tokens <= Alone::ROOM) return launch_few_as<MODE, Alone>(c);
    if (tokens <= Wide::ROOM) return launch_few_as<MODE, Wide>(c);
    if (tokens <= Tight::ROOM) return launch_few_as<MODE, Tight>(c);
    return launch_rows<8, MODE>(c);
}

template <int MODE>
int launch_f32(const F32Call& c) {
    // up to 16 rows the weights' bytes bound the product; four products (above), us: 16 rows 85, 17 rows in a tile of 64 170, as two launches of 16
    // would take, 32 rows 172
    if (c.M <= 8) return launch_few<MODE>(c);
    if (c.M <= 16) return launch_rows<16, MODE>(c);
    // from 65 rows on a tile of 128 splits the weights half as often (the four, tiles of 64 / 128: 65 rows 221 / 206, 96 rows 225 / 210, 130 rows
    // 323 / 293, 190 rows 339 / 311, 256 rows 373 / 322, 509 rows 630 / 420)
    if (c.M <= 64) return launch_tokens<64, MODE>(c);
    return launch_tokens<128, MODE>(c);
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

// rows of float32 that can be read 16 bytes at a time go to the tensor cores, everything else (and short sums) to the kernel for any types
bool wide_f32(const void* A, int a_dtype, const void* W, int w_dtype, int c_dtype, int K, int lda, int ldw) {
    return a_dtype == LP_F32 && w_dtype == LP_F32 && c_dtype == LP_F32 && K >= SPLIT_MIN_K && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0
           && (size_t)A % 16 == 0 && (size_t)W % 16 == 0;
}

}  // namespace

// scratch: room for 3 x M x (K rounded up to 8) bfloat16, 16-byte aligned, for float32 products of more than 16 rows on the tensor
// cores (may be null: they then run on the kernel for any types).
// A: [M, K] row stride lda; W: [N, K] (or [2N, K] in SWIGLU mode) row stride ldw; C: [M, N] row stride ldc.
extern "C" int lp_gemm_plain(const void* A, int a_dtype, const void* W, int w_dtype, void* C, int c_dtype, int M,
                             int N, int K, int lda, int ldw, int ldc, int mode, void* scratch, int* status, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) LP_REFUSE("gemm_plain: inner size %d", K);
    if (mode < 0 || mode > 2) LP_REFUSE("gemm_plain: mode %d", mode);
    if (c_dtype != LP_F32 && c_dtype != LP_BF16) LP_REFUSE("gemm_plain: output dtype code %d", c_dtype);
    if (mode == LP_GEMM_ACCUMULATE && c_dtype != LP_F32)
        LP_REFUSE("gemm_plain: accumulation needs a float32 output");
    if ((N + BN - 1) / BN > 2147483647 || (M + BM - 1) / BM > 65535)
        LP_REFUSE("gemm_plain: %d rows exceed the grid", M);
    if (wide_f32(A, a_dtype, W, w_dtype, c_dtype, K, lda, ldw) && (M <= 16 || scratch)) {
        const F32Call c{(const float*)A, (const float*)W, (float*)C, M, N, K, lda, ldw, ldc, (uint16_t*)scratch, status, stream};
        if (mode == LP_GEMM_STORE) return launch_f32<LP_GEMM_STORE>(c);
        if (mode == LP_GEMM_ACCUMULATE) return launch_f32<LP_GEMM_ACCUMULATE>(c);
        return launch_f32<LP_GEMM_SWIGLU>(c);
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
