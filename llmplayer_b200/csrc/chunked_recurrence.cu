// Linear-attention recurrences over prompts in chunks of 32 tokens, with the sums inside and between chunks as matrix
// products (the recurrences of linear_attention.cu for steps with many tokens; the same state, the same results up to
// rounding):
//
//     plain:       S_t = diag(a_t) S_(t-1) + k_t v_t^T                                                o_t = S_t^T q_t
//     delta rule:  S <- diag(a_t) S;  u_t = b_t (v_t - S^T k_t);  S <- S + k_t u_t^T                  o_t = S^T q_t
//
// With S the state that enters a chunk, P_i the product of the decays of tokens 1 .. i of the chunk (a vector over the key
// channels) and P_(j,i] that of tokens j + 1 .. i,
//
//     A_ij = sum_c k_ic k_jc P_(j,i],c  (j < i)          B_ij = sum_c q_ic k_jc P_(j,i],c  (j <= i)
//     (I + diag(b) A) U = diag(b) (V - (P k) S),  so  U = U0 - W S  with U0, W the solutions for diag(b) V and diag(b) (P k)
//     o_i = (P_i q_i)^T S + sum_j B_ij u_j               S' = P_32 S + sum_j (P_(j,32] k_j) u_j^T
//
// (the plain recurrence has U = V). Decays enter as running products only, forwards or backwards from a token or a block
// border, so nothing is divided by a product of decays and no logarithm is taken: strong decays (down to zero) are exact.
//
//   prepare   one CTA per (chunk, head, sequence): products of decays, A and B (blocks of 4 tokens: between two blocks as sums
//             over factored decays, inside a block with the decays multiplied token by token), the triangular solve with a
//             thread per column, all in float32 arithmetic; the results go to a record per chunk and head, laid out as the
//             operand fragments of the second kernel's products.
//   carry     one CTA per (16 value columns, head, sequence) walks the sequence's chunks in order; the state's columns stay in
//             registers, 16 key channels per warp. The products run on the tensor cores (mma.sync m16n8k8) at float32
//             precision: every operand is split into two TF32 parts, x = hi + lo with 22 bits of mantissa together, and
//             hi hi + hi lo + lo hi are summed in float32. Records come by bulk copies, up to two chunks ahead.
#include "tcgen05_utils.cuh"

namespace {

constexpr int CT = 32;                  // tokens per chunk
constexpr int HB = 4;                   // tokens per block inside a chunk
constexpr int BLOCKS = CT / HB, BLOCK_PAIRS = BLOCKS * (BLOCKS - 1) / 2;
constexpr int NC = 16;                  // value columns per CTA of the second kernel
constexpr int THREADS = 256;            // of the first kernel
constexpr int JOINERS = CT / 8;         // warps of the second kernel beside one per 16 key channels: one per 8 tokens
constexpr int MAX_DK = 256;
constexpr int CARRY_THREADS = 32 * (MAX_DK / 16 + JOINERS);      // at most
constexpr int NARROW_DK = 128, CARRY_THREADS_NARROW = 32 * (NARROW_DK / 16 + JOINERS);
constexpr size_t MAX_SMEM = 227 * 1024 - 64;      // beside the barriers

constexpr int DECAY_CHANNEL = 0, DECAY_HEAD = 1, DECAY_FIXED = 2;

// Floats of a record: [W][Q][K^T][B][P_32], fragments of 8 x 16 values each (128 floats: a lane's four values together).
__host__ __device__ __forceinline__ int padded(int dk) { return (dk + 15) / 16 * 16; }
__host__ __device__ __forceinline__ int record_floats(int dkp, bool delta) { return CT * dkp * (delta ? 3 : 2) + CT * CT + dkp; }
__host__ __device__ __forceinline__ int value_floats(int dv) { return (dv + NC - 1) / NC * NC * CT; }

// Where element (r, c) of a matrix with `ksteps` = columns / 8 lies as the column operand of m16n8k8, two steps together. The
// columns of a step are taken in the order 0, 2, 4, 6, 1, 3, 5, 7: a lane holds two neighbouring ones, as it does of a product's
// results, which so are the other operand of the next product as they lie.
__device__ __forceinline__ int fragment_at(int r, int c, int ksteps) {
    const int lane = (r & 7) * 4 + ((c & 7) >> 1), reg = (c & 1) + ((c >> 3) & 1) * 2;
    return (((r >> 3) * (ksteps >> 1) + (c >> 4)) * 32 + lane) * 4 + reg;
}

__device__ __forceinline__ float rotated_channel(const float* head, int c, int rd, int interleaved, const float2* cs) {
    const float val = __ldg(head + c);
    if (c >= rd) return val;
    const int half = rd >> 1;
    const bool first = interleaved ? (c & 1) == 0 : c < half;
    const int pair = interleaved ? c >> 1 : (first ? c : c - half);
    const float other = __ldg(head + (interleaved ? (c ^ 1) : (first ? c + half : c - half)));
    const float2 a = __ldg(cs + pair);
    return first ? val * a.x - other * a.y : val * a.x + other * a.y;
}

struct Inputs {
    const float* proj;            // [T, ld]: queries at q_off, keys at k_off ([qk heads, dk]), values at v_off ([H, dv])
    int ld, q_off, k_off, v_off;
    const float* decay;           // by `decay_form`: [T, H * dk], [T, H] or [H]
    int decay_form;
    const float* key_gain;        // [T, H] or null
    const float* beta;            // [T, H] or null: the delta rule
    const float2* angles;         // [T, rd / 2] or null
    int rd, interleaved;
    float q_scale;
    int H, dk, dv, qk_group;
    int wide;                     // no rotation, and rows of queries, keys and decays that take reads of four channels
};

// ---------------------------------------------------------------- prepare
// two float32 sums in one register pair
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ float both(uint64_t a) { return __uint_as_float((uint32_t)a) + __uint_as_float((uint32_t)(a >> 32)); }
__device__ __forceinline__ float4 four(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }

// Bound by its instructions and the latencies between its barriers (two blocks per SM): rows read four
// channels at a time, and the sums inside and between blocks as pairs of channels in one instruction, took 2048 tokens of 8
// heads of 128 x 256 from 54 to 44 us on a B200 (three prompts of 518 to 777 tokens, 128 x 128, delta rule: 57 -> 47). Stamped inside,
// 17,000 of a block's 38,000 cycles went into the sums inside blocks of 16 (a half-warp per pair of keys, whose sums met in
// shuffles for every row), 9,900 into the products of decays (the keys' record stored four bytes at a time, 64 apart). Blocks of
// 4 whose pairs are plain sums of a thread, a tile of 2 x 2 per thread between blocks, and a key's record stored 16 bytes at a
// time: the layer of 2048 tokens 219.5 -> 209.5 us, the delta rule's 231.6 -> 222.1.
// NARROW: at most 128 key channels (two blocks per SM).
template <bool NARROW>
__global__ void __launch_bounds__(THREADS, NARROW ? 2 : 1)
prepare_kernel(Inputs in, const int* __restrict__ q_start, int first_chunk, int chunks, float* __restrict__ records,
               float* __restrict__ values) {
    extern __shared__ __align__(16) float sm[];
    const int dk = in.dk, dv = in.dv, H = in.H, dkp = padded(dk), ks = dkp + 4;      // rows padded against bank conflicts
    float* qs = sm;                        // [CT][ks]: queries; later times the decays since their block's start
    float* kk = qs + CT * ks;              // [CT][ks]: keys
    float* gs = kk + CT * ks;              // [CT][ks]: decays
    float* kf = gs + CT * ks;              // [CT][ks]: keys times the decays since their block's start (their own included)
    float* ke = kf + CT * ks;              // [CT][ks]: keys times the decays up to their block's end
    float* between = ke + CT * ks;         // [BLOCK_PAIRS][ks]: products of the decays of the blocks between two
    float* L = between + BLOCK_PAIRS * ks; // [CT][CT]: b_i A_ij
    float* Bm = L + CT * CT;               // [CT][CT]
    float* bs = Bm + CT * CT;              // [CT]
    lp_grid_release();
    lp_grid_wait();
    const int h = blockIdx.y, b = blockIdx.z, tid = threadIdx.x;
    const int t0 = q_start[b] + (first_chunk + blockIdx.x) * CT, t1 = q_start[b + 1];
    if (t0 >= t1) return;
    const int n = min(CT, t1 - t0);
    const bool delta = in.beta != nullptr;
    const size_t slot = ((size_t)b * chunks + blockIdx.x) * H + h;
    float* rec = records + slot * record_floats(dkp, delta);
    float* val = values + slot * value_floats(dv);
    float* rec_w = rec;
    float* rec_q = rec + (delta ? CT * dkp : 0);
    float* rec_k = rec_q + CT * dkp;
    float* rec_b = rec_k + CT * dkp;
    float* rec_p = rec_b + CT * CT;
    const int hq = h / in.qk_group;
    // four elements per thread and turn (four times four channels where the rows allow it), so that their loads are in flight
    // together
    if (in.wide) {
        const int groups = dkp >> 2;
        for (int e0 = tid; e0 < CT * groups; e0 += 4 * THREADS) {
            float4 q[4], k[4], g[4];
            int at[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int e = e0 + u * THREADS;
                const int i = e / groups, c = (e - i * groups) * 4;
                at[u] = e < CT * groups ? i * ks + c : -1;
                q[u] = k[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                g[u] = make_float4(1.f, 1.f, 1.f, 1.f);
                if (i < n && c < dk) {
                    const size_t t = t0 + i;
                    const float* row = in.proj + t * in.ld;
                    q[u] = four(row + in.q_off + hq * dk + c);
                    k[u] = four(row + in.k_off + hq * dk + c);
                    if (in.decay_form == DECAY_CHANNEL) {
                        g[u] = four(in.decay + (t * H + h) * dk + c);
                    } else {
                        const float one = __ldg(in.decay + (in.decay_form == DECAY_FIXED ? (size_t)h : t * H + h));
                        g[u] = make_float4(one, one, one, one);
                    }
                    if (in.key_gain) {
                        const float gain = __ldg(in.key_gain + t * H + h);
                        k[u].x *= gain; k[u].y *= gain; k[u].z *= gain; k[u].w *= gain;
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (at[u] >= 0) {
                    *reinterpret_cast<float4*>(qs + at[u]) =
                        make_float4(q[u].x * in.q_scale, q[u].y * in.q_scale, q[u].z * in.q_scale, q[u].w * in.q_scale);
                    *reinterpret_cast<float4*>(kk + at[u]) = k[u];
                    *reinterpret_cast<float4*>(gs + at[u]) = g[u];
                }
        }
    } else {
        for (int e0 = tid; e0 < CT * dkp; e0 += 4 * THREADS) {
            float q[4], k[4], g[4];
            int at[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int e = e0 + u * THREADS;
                const int i = e / dkp, c = e - i * dkp;
                at[u] = e < CT * dkp ? i * ks + c : -1;
                q[u] = k[u] = 0.f;
                g[u] = 1.f;
                if (i < n && c < dk) {
                    const float* row = in.proj + (size_t)(t0 + i) * in.ld;
                    const float* qh = row + in.q_off + hq * dk;
                    const float* kh = row + in.k_off + hq * dk;
                    if (in.rd > 0) {
                        const float2* cs = in.angles + (size_t)(t0 + i) * (in.rd >> 1);
                        q[u] = rotated_channel(qh, c, in.rd, in.interleaved, cs);
                        k[u] = rotated_channel(kh, c, in.rd, in.interleaved, cs);
                    } else {
                        q[u] = __ldg(qh + c);
                        k[u] = __ldg(kh + c);
                    }
                    g[u] = in.decay_form == DECAY_FIXED ? __ldg(in.decay + h)
                           : in.decay_form == DECAY_HEAD ? __ldg(in.decay + (size_t)(t0 + i) * H + h)
                                                         : __ldg(in.decay + ((size_t)(t0 + i) * H + h) * dk + c);
                    if (in.key_gain) k[u] *= __ldg(in.key_gain + (size_t)(t0 + i) * H + h);
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (at[u] >= 0) {
                    qs[at[u]] = q[u] * in.q_scale;
                    kk[at[u]] = k[u];
                    gs[at[u]] = g[u];
                }
        }
    }
    for (int i = tid; i < CT; i += THREADS) bs[i] = delta && i < n ? in.beta[(size_t)(t0 + i) * H + h] : 0.f;
    for (int e = tid; e < CT * CT; e += THREADS) L[e] = Bm[e] = 0.f;
    __syncthreads();

    // pairs (i, j) of one block: a pair, or a token with itself (B alone), per two threads, which take every other four channels
    {
        const int item = tid >> 1, half = tid & 1;
        constexpr int INSIDE = HB * (HB - 1) / 2, PAIRS = BLOCKS * INSIDE;
        int i = 0, j = 0;
        if (item < PAIRS) {
            const int pair = item % INSIDE;
            const int r = pair < 1 ? 1 : pair < 3 ? 2 : 3;
            i = item / INSIDE * HB + r;
            j = item / INSIDE * HB + pair - r * (r - 1) / 2;
        } else if (item < PAIRS + CT) i = j = item - PAIRS;
        uint64_t sa = 0, sb = 0;
        if (item < PAIRS + CT)
            for (int c = half; c < dkp >> 2; c += 2) {
                auto row = [&](const float* x, int r) { return reinterpret_cast<const ulonglong2*>(x + r * ks)[c]; };
                const ulonglong2 k = row(kk, i), q = row(qs, i);
                ulonglong2 m = row(kk, j);
                for (int t = j + 1; t <= i; ++t) {
                    const ulonglong2 g = row(gs, t);
                    m.x = mul2(m.x, g.x);
                    m.y = mul2(m.y, g.y);
                }
                sa = fma2(k.x, m.x, fma2(k.y, m.y, sa));
                sb = fma2(q.x, m.x, fma2(q.y, m.y, sb));
            }
        float a = both(sa), bsum = both(sb);
        a += __shfl_xor_sync(0xffffffffu, a, 1);
        bsum += __shfl_xor_sync(0xffffffffu, bsum, 1);
        if (half == 0 && item < PAIRS + CT) {
            Bm[i * CT + j] = bsum;
            if (i > j) L[i * CT + j] = bs[i] * a;
        }
    }
    __syncthreads();

    // products of decays, a thread per key channel (forwards; its column of diag(b) (P k) stays in registers for the solve) and
    // one backwards (other threads where there are enough)
    float col[CT];
    const int back = dkp <= THREADS / 2 ? THREADS / 2 : 0;
    if (tid < dkp) {
        const int c = tid;
        float p = 1.f, pb = 1.f, block[BLOCKS];
#pragma unroll
        for (int i = 0; i < CT; ++i) {
            const float g = gs[i * ks + c], k = kk[i * ks + c], q = qs[i * ks + c];
            p *= g;
            rec_q[fragment_at(i, c, dkp >> 3)] = q * p;
            col[i] = bs[i] * k * p;
            pb = i % HB ? pb * g : g;
            kf[i * ks + c] = k * pb;
            qs[i * ks + c] = q * pb;
            if (i % HB == HB - 1) block[i / HB] = pb;
        }
        rec_p[c] = p;
#pragma unroll
        for (int from = 0; from < BLOCKS - 1; ++from) {
            float gap = 1.f;
#pragma unroll
            for (int to = from + 1; to < BLOCKS; ++to) {
                between[(to * (to - 1) / 2 + from) * ks + c] = gap;
                gap *= block[to];
            }
        }
    }
    if (tid >= back && tid - back < dkp) {
        const int c = tid - back;
        float p = 1.f, pb = 1.f;
#pragma unroll
        for (int i0 = CT - 16; i0 >= 0; i0 -= 16) {
            float x[16];
#pragma unroll
            for (int u = 15; u >= 0; --u) {
                const int i = i0 + u;
                const float g = gs[i * ks + c], k = kk[i * ks + c];
                x[u] = k * p;
                p *= g;
                if (u % HB == HB - 1) pb = 1.f;
                ke[i * ks + c] = k * pb;
                pb *= g;
            }
            float4* at = reinterpret_cast<float4*>(rec_k + fragment_at(c, i0, CT >> 3));
#pragma unroll
            for (int u = 0; u < 4; ++u) at[u] = make_float4(x[2 * u], x[2 * u + 1], x[2 * u + 8], x[2 * u + 9]);
        }
    }
    __syncthreads();

    // between the blocks: a tile of two rows and two keys per two threads, which take every other four channels
    {
        const int item = tid >> 1, half = tid & 1, pair = item >> 2;
        int to = 1;
        while (to * (to + 1) / 2 <= pair) ++to;
        const int from = pair - to * (to - 1) / 2;
        const bool real = pair < BLOCK_PAIRS;
        const int i = real ? to * HB + (item >> 1 & 1) * 2 : 0, j = real ? from * HB + (item & 1) * 2 : 0;
        uint64_t sa[2][2] = {}, sb[2][2] = {};
        if (real)
            for (int c = half; c < dkp >> 2; c += 2) {
                auto row = [&](const float* x, int r) { return reinterpret_cast<const ulonglong2*>(x + r * ks)[c]; };
                const ulonglong2 g = row(between, pair);
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    ulonglong2 e = row(ke, j + v);
                    e.x = mul2(e.x, g.x);
                    e.y = mul2(e.y, g.y);
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const ulonglong2 k = row(kf, i + u), q = row(qs, i + u);
                        sa[u][v] = fma2(k.x, e.x, fma2(k.y, e.y, sa[u][v]));
                        sb[u][v] = fma2(q.x, e.x, fma2(q.y, e.y, sb[u][v]));
                    }
                }
            }
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                const float a = both(sa[u][v]), bsum = both(sb[u][v]);
                // the first thread of the two finishes A, the other B
                const float sum = (half ? bsum : a) + __shfl_xor_sync(0xffffffffu, half ? a : bsum, 1);
                if (!real) continue;
                if (half) Bm[(i + u) * CT + j + v] = sum;
                else L[(i + u) * CT + j + v] = bs[i + u] * sum;
            }
    }
    __syncthreads();
    for (int e = tid; e < CT * CT; e += THREADS) rec_b[fragment_at(e / CT, e % CT, CT >> 3)] = Bm[e];

    // the solve: x_i = r_i - sum_(j<i) L_ij x_j, a thread per column of [diag(b) (P k) | diag(b) V]
    const int columns = dkp + (dv + NC - 1) / NC * NC;
    for (int item = delta ? tid : tid + dkp; item < columns; item += THREADS) {      // (the plain recurrence needs no keys here)
        const bool key = item < dkp;
        const int c = item - dkp;
        if (!key) {
#pragma unroll
            for (int i = 0; i < CT; ++i) {
                const float v = (i < n && c < dv) ? __ldg(in.proj + (size_t)(t0 + i) * in.ld + in.v_off + h * dv + c) : 0.f;
                col[i] = delta ? bs[i] * v : v;
            }
        }
        if (delta) {
#pragma unroll
            for (int i = 1; i < CT; ++i) {
                float acc = col[i];
#pragma unroll
                for (int j = 0; j < i; j += 4) {
                    const float4 l = *reinterpret_cast<const float4*>(L + i * CT + j);      // zero from the diagonal on
                    acc = fmaf(-l.x, col[j], acc);
                    if (j + 1 < i) acc = fmaf(-l.y, col[j + 1], acc);
                    if (j + 2 < i) acc = fmaf(-l.z, col[j + 2], acc);
                    if (j + 3 < i) acc = fmaf(-l.w, col[j + 3], acc);
                }
                col[i] = acc;
            }
        }
        if (key) {
#pragma unroll
            for (int i = 0; i < CT; ++i) rec_w[fragment_at(i, item, dkp >> 3)] = col[i];
        } else {
            float* at = val + (c / NC) * (CT * NC) + c % NC;
#pragma unroll
            for (int i = 0; i < CT; ++i) at[i * NC] = col[i];
        }
    }
}

// ---------------------------------------------------------------- carry
// x = hi + lo with two TF32 values: hi is x with its last 13 bits cut off, lo the remainder rounded to TF32 (by integer
// operations: the conversion instruction runs at a fraction of their rate)
__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
    hi = __float_as_uint(x) & 0xffffe000u;
    lo = (__float_as_uint(x - __uint_as_float(hi)) + 0x1000u) & 0xffffe000u;
}
__device__ __forceinline__ void mma_tf32(float* c, const uint32_t* a, const uint32_t* b) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// A fragment of a record, split as the column operand of two steps of 8
struct Columns {
    uint32_t hi[4], lo[4];
    __device__ __forceinline__ explicit Columns(float4 y) {
        split_tf32(y.x, hi[0], lo[0]);
        split_tf32(y.y, hi[1], lo[1]);
        split_tf32(y.z, hi[2], lo[2]);
        split_tf32(y.w, hi[3], lo[3]);
    }
};
template <int N> struct Count { static constexpr int value = N; };
// acc += step w of X Y, X [16 x 16] split as row operands (xh, xl), Y [16 x 8]; three chains of sums
__device__ __forceinline__ void product(float (*acc)[4], const uint32_t (*xh)[4], const uint32_t (*xl)[4], const Columns& y, int w) {
    mma_tf32(acc[0], xh[w], y.hi + 2 * w);
    mma_tf32(acc[1], xh[w], y.lo + 2 * w);
    mma_tf32(acc[2], xl[w], y.hi + 2 * w);
}
__device__ __forceinline__ float4 chains(const float (*acc)[4]) {
    return make_float4(acc[0][0] + (acc[1][0] + acc[2][0]), acc[0][1] + (acc[1][1] + acc[2][1]), acc[0][2] + (acc[1][2] + acc[2][2]),
                       acc[0][3] + (acc[1][3] + acc[2][3]));
}

// All products are taken transposed (value columns are their 16 rows). Worker m holds S^T for the key channels 16 m .. 16 m + 15
// in registers, which are the row operand of its share of (W S)^T and (Q S)^T as they lie; the shares meet in shared memory.
// Joiner n has the tokens 8 n .. 8 n + 7: it requests the records, makes U^T = (U0 - W S)^T (split, as the row operand of what
// follows) and the outputs of its tokens from the shares of (Q S)^T and (B U)^T.
// The plain recurrence's chain is the state alone (U is V), with one barrier per chunk: behind it the workers take their shares
// of Q S and go on to the next state, while the joiners write the chunk before (its shares lie in the other half of a double
// buffer), form B U and split the next chunk's values (likewise). The delta rule's chain goes through U, with two barriers: the
// workers' shares of W S; U^T from them, while the workers take their shares of Q S; the next state, while the outputs are
// written, which may last into the next chunk's shares of W S.
// 2048 tokens of 8 heads of 128 x 256, B200: 114 us with the state split in shared memory, read as column operands and stored again
// in every chunk; 97 with it in registers; 90 with bulk copies in place of 16 bytes per thread and request, which went through the
// load unit that the fragments come through; 82 with one barrier in place of two and a warp's reads, splits and products of a
// chunk side by side (three prompts of 518 to 777 tokens, 8 heads of 128 x 128, delta rule: 88, -, 71, 68 with two barriers in
// place of three). What is left, per chunk of 1.28 us: 864 cycles of the tensor cores (8 per product and quarter SM), some 1,180
// of shared memory and 780 issue slots, partly one behind the other in the two workers of a quarter SM; with the records not
// copied at all it takes 74 us, so neither L2 nor the copies bound it.
// STAGES: records in flight (three, or fewer where they do not fit shared memory; with fewer the delta rule frees a stage by a
// barrier at a chunk's end).
// WIDE: more than 128 key channels, and more warps with fewer registers each.
template <int STAGES, bool DELTA, bool WIDE>
__global__ void __launch_bounds__(WIDE ? CARRY_THREADS : CARRY_THREADS_NARROW)
carry_kernel(float* __restrict__ state, const int* __restrict__ slots, const int* __restrict__ q_start, int first_chunk, int chunks,
             const float* __restrict__ records, const float* __restrict__ values, float* __restrict__ out, int H, int dk, int dv,
             int* __restrict__ status) {
    static_assert(DELTA || STAGES >= 2, "the plain recurrence reads the next chunk's values during a chunk");
    extern __shared__ __align__(16) float sm[];
    __shared__ uint64_t full[STAGES];                   // a stage's record is there
    const int dkp = padded(dk), rec_n = record_floats(dkp, DELTA), kt = dkp >> 4;
    uint4* Us = reinterpret_cast<uint4*>(sm);            // [2 unless DELTA][JOINERS][32 lanes] twice: U^T as row operands, its two parts
    float4* parts_q = reinterpret_cast<float4*>(Us + (DELTA ? 2 : 4) * JOINERS * 32);      // [kt][JOINERS][32 lanes], and again
    float4* parts_w = parts_q + kt * JOINERS * 32;       // for W, or for the odd chunks
    float* ring = reinterpret_cast<float*>(parts_w + kt * JOINERS * 32);      // STAGES records, each followed by the chunk's
                                                         // 32 x 16 values
    const int stage = rec_n + CT * NC;
    lp_grid_release();
    lp_grid_wait();
    const int h = blockIdx.y, b = blockIdx.z, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int j0 = blockIdx.x * NC;
    const int begin = q_start[b] + first_chunk * CT, t1 = q_start[b + 1];
    if (begin >= t1) return;
    const int used = min(chunks, (t1 - begin + CT - 1) / CT);
    float* row = state + ((size_t)slots[b] * H + h) * dv * dk;

    const bool joins = warp >= kt;
    const int n = warp - kt;                        // of a joiner
    auto request = [&](int p) {                     // one thread: chunk p's record and values into stage p % STAGES
        if (tid != 32 * kt || p >= used) return;
        const size_t slot = ((size_t)b * chunks + p) * H + h;
        float* dst = ring + (p % STAGES) * stage;
        uint64_t* bar = &full[p % STAGES];
        mbar_expect_tx(bar, stage * 4);
        bulk_load(dst, records + slot * rec_n, rec_n * 4, bar);
        bulk_load(dst + rec_n, values + slot * value_floats(dv) + blockIdx.x * (CT * NC), CT * NC * 4, bar);
    };
    if (tid == 32 * kt) {
#pragma unroll
        for (int i = 0; i < STAGES; ++i) mbar_init(&full[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // a stage that every warp has left takes the next record during a chunk; with fewer than three stages the delta rule's own
    // stage does when the chunk ends
    constexpr bool EARLY = !DELTA || STAGES >= 3;
    if (joins) {
#pragma unroll
        for (int p = 0; p < (EARLY ? STAGES - 1 : STAGES); ++p) request(p);
    }
    const int g8 = lane >> 2, t4 = lane & 3;
    // s[w]: value columns g8 and g8 + 8 (entries 0, 1 and 2, 3) of two neighbouring channels
    auto channel = [&](int w, int e) { return warp * 16 + w * 8 + t4 * 2 + (e & 1); };
    auto column = [&](int e) { return j0 + g8 + (e >> 1) * 8; };
    float s[2][4];
#pragma unroll
    for (int w = 0; w < 2; ++w)
#pragma unroll
        for (int e = 0; e < 4; ++e)
            s[w][e] = (!joins && column(e) < dv && channel(w, e) < dk) ? row[(size_t)column(e) * dk + channel(w, e)] : 0.f;
    uint32_t sh[2][4], sl[2][4];
    auto split_state = [&] {
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            split_tf32(s[w][0], sh[w][0], sl[w][0]);
            split_tf32(s[w][2], sh[w][1], sl[w][1]);
            split_tf32(s[w][1], sh[w][2], sl[w][2]);
            split_tf32(s[w][3], sh[w][3], sl[w][3]);
        }
    };
    constexpr int TOGETHER = WIDE ? 1 : JOINERS;     // of a worker's products: their reads, splits and sums overlap
    // a worker's share of (X S)^T for the matrix X of a record
    auto share = [&](const float* x, float4* parts) {
        const float4* at = reinterpret_cast<const float4*>(x) + warp * 32 + lane;
#pragma unroll
        for (int i0 = 0; i0 < JOINERS; i0 += TOGETHER) {
            float4 y[TOGETHER];
#pragma unroll
            for (int i = 0; i < TOGETHER; ++i) y[i] = at[(i0 + i) * kt * 32];
            float acc[TOGETHER][3][4] = {};
#pragma unroll
            for (int w = 0; w < 2; ++w)
#pragma unroll
                for (int i = 0; i < TOGETHER; ++i) product(acc[i], sh, sl, Columns(y[i]), w);
#pragma unroll
            for (int i = 0; i < TOGETHER; ++i) parts[(warp * JOINERS + i0 + i) * 32 + lane] = chains(acc[i]);
        }
    };
    // the shares of 8 tokens, added in order
    auto gather = [&](const float4* parts) {
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4* at = parts + n * 32 + lane;
#pragma unroll 8
        for (int m = 0; m < kt; ++m) {
            const float4 v = at[m * JOINERS * 32];
            sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
        }
        return sum;
    };
    // a joiner's 8 tokens of U^T: the values less `sum`
    auto join = [&](const float* val, float4 sum, uint4* u) {
        const float* at = val + (n * 8 + t4 * 2) * NC + g8;
        uint4 hi, lo;
        split_tf32(at[0] - sum.x, hi.x, lo.x);
        split_tf32(at[NC] - sum.y, hi.z, lo.z);
        split_tf32(at[8] - sum.z, hi.y, lo.y);
        split_tf32(at[NC + 8] - sum.w, hi.w, lo.w);
        u[n * 32 + lane] = hi;
        u[(JOINERS + n) * 32 + lane] = lo;
    };
    // acc[i] += U^T Y_i over the tokens 16 q .. 16 q + 15, for `count` fragment columns Y_i
    auto times_u = [&](auto count, float (*acc)[3][4], const uint4* u, const float* frag, int q) {
        constexpr int COUNT = decltype(count)::value;
        uint32_t uh[2][4], ul[2][4];
        float4 y[COUNT];
#pragma unroll
        for (int i = 0; i < COUNT; ++i) y[i] = reinterpret_cast<const float4*>(frag)[(2 * i + q) * 32 + lane];
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            const uint4 hi = u[(2 * q + w) * 32 + lane], lo = u[(JOINERS + 2 * q + w) * 32 + lane];
            uh[w][0] = hi.x; uh[w][1] = hi.y; uh[w][2] = hi.z; uh[w][3] = hi.w;
            ul[w][0] = lo.x; ul[w][1] = lo.y; ul[w][2] = lo.z; ul[w][3] = lo.w;
        }
#pragma unroll
        for (int w = 0; w < 2; ++w)
#pragma unroll
            for (int i = 0; i < COUNT; ++i) product(acc[i], uh, ul, Columns(y[i]), w);
    };
    auto move_state = [&](const uint4* u, const float* rec_k, const float* rec_p) {
        float up[2][3][4] = {};
#pragma unroll
        for (int q = 0; q < 2; ++q) times_u(Count<2>{}, up, u, rec_k + warp * 4 * 128, q);
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            const float2 decay = *reinterpret_cast<const float2*>(rec_p + channel(w, 0));
#pragma unroll
            for (int e = 0; e < 4; ++e)
                s[w][e] = fmaf(e & 1 ? decay.y : decay.x, s[w][e], up[w][0][e] + (up[w][1][e] + up[w][2][e]));
        }
    };
    // a joiner's 8 tokens of chunk p's outputs: the shares of Q S and B U
    auto write_out = [&](int p, float4 o, float4 u) {
        const float x[4] = {o.x + u.x, o.y + u.y, o.z + u.z, o.w + u.w};
        const int t = begin + p * CT + n * 8 + t4 * 2;
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (t + (e & 1) < t1 && column(e) < dv) out[((size_t)(t + (e & 1)) * H + h) * dv + column(e)] = x[e];
    };
    // a wait that ran out ends the block: its own copies in flight are waited for first
    auto give_up = [&](int p) {
        if (tid != 32 * kt) return;
        atomicExch(status, 61);
        for (int i = p + 1; i < min(used, p + (EARLY ? STAGES - 1 : STAGES)); ++i) mbar_wait(&full[i % STAGES], (i / STAGES) & 1);
    };
    auto wait = [&](int p) { return mbar_wait(&full[p % STAGES], (p / STAGES) & 1); };
    auto record = [&](int p) { return ring + (p % STAGES) * stage; };
    constexpr int U_CHUNK = 2 * JOINERS * 32;
    if constexpr (!DELTA) {
        const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
        bool there = true;
        float4 held = none;                          // a joiner's share of B U until the chunk's shares of Q S are there
        if (joins) {
            there = wait(0);
            join(record(0) + rec_n, none, Us);
        }
        for (int p = 0; p < used; ++p) {
            there = wait(p) && there;
            if (!__syncthreads_and(there)) {         // the chunk before is done, this one's values are split
                give_up(p);
                return;
            }
            const float* rec_k = record(p) + CT * dkp;
            const float* rec_b = rec_k + CT * dkp;
            const uint4* u = Us + (p & 1) * U_CHUNK;
            if (!joins) {
                split_state();
                share(record(p), p & 1 ? parts_w : parts_q);
                move_state(u, rec_k, rec_b + CT * CT);
            } else {
                request(p + STAGES - 1);
                if (p > 0) write_out(p - 1, gather(p & 1 ? parts_q : parts_w), held);
                float acc[1][3][4] = {};
#pragma unroll
                for (int q = 0; q < 2; ++q) times_u(Count<1>{}, acc, u, rec_b + n * 2 * 128, q);
                held = chains(acc[0]);
                if (p + 1 < used) {
                    there = wait(p + 1);
                    join(record(p + 1) + rec_n, none, Us + ((p + 1) & 1) * U_CHUNK);
                }
            }
        }
        __syncthreads();
        if (joins) write_out(used - 1, gather((used - 1) & 1 ? parts_w : parts_q), held);
    } else {
        for (int p = 0; p < used; ++p) {
            const bool there = wait(p);
            const float* rec_q = record(p) + CT * dkp;
            const float* rec_k = rec_q + CT * dkp;
            const float* rec_b = rec_k + CT * dkp;
            if (!joins) {
                split_state();
                if (there) share(record(p), parts_w);
            }
            if (!__syncthreads_and(there)) {         // the shares of W S are there, and the chunk before is done
                give_up(p);
                return;
            }
            if (!joins) {
                share(rec_q, parts_q);
            } else {
                join(record(p) + rec_n, gather(parts_w), Us);
                if (EARLY) request(p + STAGES - 1);
            }
            __syncthreads();                         // U and the shares of Q S are there
            if (!joins) {
                move_state(Us, rec_k, rec_b + CT * CT);
            } else {
                float acc[1][3][4] = {};
#pragma unroll
                for (int q = 0; q < 2; ++q) times_u(Count<1>{}, acc, Us, rec_b + n * 2 * 128, q);
                write_out(p, gather(parts_q), chains(acc[0]));
            }
            if (!EARLY) {
                __syncthreads();                     // the stage is free
                if (joins) request(p + STAGES);
            }
        }
    }
#pragma unroll
    for (int w = 0; w < 2; ++w)
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (!joins && column(e) < dv && channel(w, e) < dk) row[(size_t)column(e) * dk + channel(w, e)] = s[w][e];
}

template <typename K> int reserve(K kernel, size_t bytes, size_t& granted) {
    if (bytes <= 40 * 1024 || bytes <= granted) return 0;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) LP_REFUSE("chunked_recurrence: cannot reserve %zu bytes of shared memory: %s", bytes, cudaGetErrorString(e));
    granted = bytes;
    return 0;
}

}  // namespace

extern "C" int lp_chunked_tokens() { return CT; }
// Floats that one chunk of one head needs: a record for the second kernel, and the columns of U.
extern "C" int lp_chunked_record_floats(int dk, int delta) { return record_floats(padded(dk), delta != 0); }
extern "C" int lp_chunked_value_floats(int dv) { return value_floats(dv); }

// The recurrence over a step's tokens of B sequences, from and into `state` (float32 [slots, H, dv, dk]). See Inputs for the
// operands. records: float32 [B, chunks, H, record floats], values: float32 [B, chunks, H, value floats]: room for `chunks`
// chunks of every sequence; a step with longer sequences (max_new: the most new tokens of one) runs in several rounds.
extern "C" int lp_chunked_recurrence(const float* proj, int ld, int q_off, int k_off, int v_off, const float* decay, int decay_form,
                                     const float* key_gain, const float* beta, const float* angles, int rd, int interleaved,
                                     float q_scale, float* state, const int* slots, const int* q_start, float* out, int B, int H,
                                     int dk, int dv, int qk_heads, int max_new, int chunks, float* records, float* values, int* status,
                                     cudaStream_t stream) {
    if (B <= 0 || max_new <= 0) return 0;
    if (H <= 0 || H > 65535 || B > 65535 || dk <= 0 || dk > MAX_DK || dv <= 0) LP_REFUSE("chunked_recurrence: %d sequences, %d heads of %d x %d (at most %d key channels)", B, H, dk, dv, MAX_DK);
    if (qk_heads <= 0) qk_heads = H;
    if (H % qk_heads) LP_REFUSE("chunked_recurrence: %d heads over %d query / key heads", H, qk_heads);
    if (q_off < 0 || k_off < 0 || v_off < 0 || q_off + qk_heads * dk > ld || k_off + qk_heads * dk > ld || v_off + H * dv > ld)
        LP_REFUSE("chunked_recurrence: slices at %d, %d, %d do not fit rows of %d", q_off, k_off, v_off, ld);
    if (decay_form < DECAY_CHANNEL || decay_form > DECAY_FIXED) LP_REFUSE("chunked_recurrence: decay form %d", decay_form);
    if (rd < 0 || rd > dk || (rd & 1) || (rd > 0 && !angles)) LP_REFUSE("chunked_recurrence: a rotation over %d of %d channels", rd, dk);
    if (chunks <= 0 || !records || !values || !status) LP_REFUSE("chunked_recurrence: room for %d chunks", chunks);
    if ((((uintptr_t)records | (uintptr_t)values) & 15) != 0) LP_REFUSE("chunked_recurrence: buffers must be aligned to 16 bytes");
    const Inputs in{proj, ld, q_off, k_off, v_off, decay, decay_form, key_gain, beta, (const float2*)angles, rd, interleaved, q_scale,
                    H, dk, dv, H / qk_heads,
                    rd == 0 && (dk & 3) == 0 && (ld & 3) == 0 && (q_off & 3) == 0 && (k_off & 3) == 0 && ((uintptr_t)proj & 15) == 0 &&
                        (decay_form != DECAY_CHANNEL || ((uintptr_t)decay & 15) == 0)};
    const int dkp = padded(dk), delta = beta ? 1 : 0;
    const size_t smem_p = ((size_t)(5 * CT + BLOCK_PAIRS) * (dkp + 4) + 2 * CT * CT + CT) * sizeof(float);
    const size_t stage = (size_t)(record_floats(dkp, delta) + CT * NC) * sizeof(float);
    const int kt = dkp / 16;
    const size_t kept = (size_t)((delta ? 2 : 4) + kt * 2) * JOINERS * 32 * sizeof(float4);
    const int stages = kept + 3 * stage <= MAX_SMEM ? 3 : kept + 2 * stage <= MAX_SMEM ? 2 : 1;      // (plain: two at least)
    const size_t smem_c = kept + stages * stage;
    auto prepare = dkp <= NARROW_DK ? prepare_kernel<true> : prepare_kernel<false>;
    const bool wide = dkp > NARROW_DK;                        // (narrow: three stages always fit)
    auto carry = delta ? (!wide ? carry_kernel<3, true, false> : stages == 3 ? carry_kernel<3, true, true>
                          : stages == 2 ? carry_kernel<2, true, true> : carry_kernel<1, true, true>)
                       : (!wide ? carry_kernel<3, false, false> : stages == 3 ? carry_kernel<3, false, true>
                                                                              : carry_kernel<2, false, true>);
    static size_t granted_p[2] = {}, granted_c[2][4] = {};       // what each kernel has been allowed so far
    int rc = reserve(prepare, smem_p, granted_p[dkp <= NARROW_DK]);
    if (rc) return rc;
    rc = reserve(carry, smem_c, granted_c[delta][wide ? stages : 0]);
    if (rc) return rc;
    const int total = (max_new + CT - 1) / CT;
    for (int first = 0; first < total; first += chunks) {
        const int here = total - first < chunks ? total - first : chunks;
        lp_launch(prepare, dim3(here, H, B), THREADS, smem_p, stream, in, q_start, first, chunks, records, values);
        rc = lp_check_launch("chunked_recurrence (prepare)");
        if (rc) return rc;
        lp_launch(carry, dim3((dv + NC - 1) / NC, H, B), 32 * (kt + JOINERS), smem_c, stream, state, slots, q_start, first, chunks,
                  (const float*)records, (const float*)values, out, H, dk, dv, status);
        rc = lp_check_launch("chunked_recurrence (carry)");
        if (rc) return rc;
    }
    return 0;
}
