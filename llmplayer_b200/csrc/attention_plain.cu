// Plain attention of a batch of query tokens over the paged key/value cache.
//
// Float32 queries over a float32 cache take the kernels further down, which finish blocks of 128 keys one by one. Other
// types and odd head sizes take the first kernel: one block per (query token, query head). Keys are visited in blocks of 128
// aligned to absolute positions; within a block one thread scores one key, the
// running maximum and sum are updated (online softmax, all float32), then each
// thread owns output features and adds the block's weighted values in increasing
// key order. The order of every sum depends only on the query's position and the
// window, never on how tokens were cut into steps or batched.
//
// Counterpart in the reference: src/main/resources/kernels/cuda/attention.cu:10-108
// (one query, scores in shared memory) and the online-softmax variant
// inference/Attention.java:161-207.
#include "common.cuh"

namespace {

constexpr int KB = 128;       // keys per block = threads per block
constexpr int MAX_HD = 256;

template <typename TQ, typename TKV>
__global__ void __launch_bounds__(KB)
attention_plain_kernel(const TQ* __restrict__ q, TQ* __restrict__ out, const TKV* __restrict__ pages,
                       const int* __restrict__ page_table, int pt_stride, const int* __restrict__ seq_ids,
                       const int* __restrict__ positions, int H, int G, int hd, int page_size, float scale,
                       int window, float softcap, const float* __restrict__ sinks, int keep, int chunk,
                       const float* __restrict__ dist_scale, const float* __restrict__ dist_rate,
                       const float* __restrict__ gate, int gate_ld) {
    __shared__ float qs[MAX_HD];
    __shared__ float prob[KB];
    __shared__ long long row_off[KB];
    __shared__ float scratch[32];

    const int t = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
    const int g = h / (H / G);
    const int seq = seq_ids[t];
    const int pos = positions[t];
    int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
    if (chunk > 0) lo = max(lo, pos / chunk * chunk);         // keys of the query's own chunk of positions only
    const float ds = dist_scale ? dist_scale[h] : 0.f, dr = dist_scale ? dist_rate[h] : 0.f;
    // a window may keep a sequence's first `keep` tokens visible as well: keys [0, keep_end) besides [lo, pos]
    const int keep_end = keep < lo ? (keep > 0 ? keep : 0) : lo;
    const int c_lo = (lo / KB) * KB;

    const TQ* qr = q + ((long long)t * H + h) * hd;
    for (int i = tid; i < hd; i += KB) qs[i] = lp_to_float(qr[i]);
    __syncthreads();

    float m = -INFINITY, l = 0.f;
    float acc0 = 0.f, acc1 = 0.f;   // features tid and tid + 128
    const int* pt = page_table + (long long)seq * pt_stride;

    for (int c0 = 0;; c0 += KB) {
        if (c0 >= keep_end && c0 < c_lo) c0 = c_lo;      // the blocks between the kept tokens and the window are not seen
        if (c0 > pos) break;
        const int key = c0 + tid;
        const bool valid = key <= pos && (key >= lo || key < keep_end);
        float sc = -INFINITY;
        if (valid) {
            const int page = pt[key / page_size];
            const long long off = (((long long)page * 2 * G + g) * page_size + (key % page_size)) * hd;
            row_off[tid] = off;
            const TKV* kr = pages + off;
            float dot = 0.f;
            for (int i = 0; i < hd; ++i) dot = fmaf(qs[i], lp_to_float(kr[i]), dot);
            sc = dot * scale;
            if (softcap > 0.f) sc = softcap * tanhf(sc / softcap);
            if (dist_scale) sc -= ds * log1pf(dr * (float)(pos - key));
        }
        const float cmax = lp_block_max(sc, scratch);
        const float m_new = fmaxf(m, cmax);
        const float pr = valid ? expf(sc - m_new) : 0.f;
        prob[tid] = pr;
        const float csum = lp_block_sum(pr, scratch);   // also publishes prob[] and row_off[]
        const float alpha = (m == -INFINITY) ? 0.f : expf(m - m_new);
        l = l * alpha + csum;
        acc0 *= alpha;
        acc1 *= alpha;
        const int nk = (pos - c0 + 1 < KB) ? pos - c0 + 1 : KB;
        const int first = c0 < keep_end ? 0 : (lo > c0 ? lo - c0 : 0);
        const long long v_shift = (long long)G * page_size * hd;    // from a K row to its V row
        if (tid < hd) {
            for (int j = first; j < nk; ++j)
                if (prob[j] > 0.f) acc0 = fmaf(prob[j], lp_to_float(pages[row_off[j] + v_shift + tid]), acc0);
        }
        if (tid + KB < hd) {
            for (int j = first; j < nk; ++j)
                if (prob[j] > 0.f) acc1 = fmaf(prob[j], lp_to_float(pages[row_off[j] + v_shift + tid + KB]), acc1);
        }
        m = m_new;
        __syncthreads();
    }
    // a sink: a learned logit per head that takes part in the softmax's denominator only, once
    if (sinks) {
        const float sk = sinks[h];
        const float m_new = fmaxf(m, sk);
        const float alpha = expf(m - m_new);
        l = l * alpha + expf(sk - m_new);
        acc0 *= alpha;
        acc1 *= alpha;
    }
    // a gate per query token and head multiplies the head's finished output
    const float inv = gate ? 1.0f / (l * (1.0f + expf(-gate[(long long)t * gate_ld + h]))) : 1.0f / l;
    TQ* o = out + ((long long)t * H + h) * hd;
    if (tid < hd) o[tid] = lp_from_float<TQ>(acc0 * inv);
    if (tid + KB < hd) o[tid + KB] = lp_from_float<TQ>(acc1 * inv);
}

// ---------------------------------------------------------------- float32, keys in blocks that are finished one by one
// A query's result is put together from blocks of 128 keys aligned to absolute positions. Within a block: scores (each a
// chain of multiply-adds over the head's features), the block's maximum, exponentials against it, their sum (lane l
// adds keys l, l + 32, l + 64, l + 96, then a butterfly) and the weighted values (a chain over the keys). The blocks join
// in increasing order. Every step of that depends on the query's position and mask alone, so the two kernels below (a tile
// of queries walking its blocks; a CTA per block, joined by a third kernel) give the same bits, and a position's result
// does not depend on how its sequence was cut into steps or batched.
struct Mask {
    int window, keep, chunk;
    // keys [0, keep_end) and [lo, pos] are seen
    __device__ __forceinline__ int first(int pos) const {
        int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
        return chunk > 0 ? max(lo, pos / chunk * chunk) : lo;
    }
    __device__ __forceinline__ int kept(int lo) const { return keep < lo ? (keep > 0 ? keep : 0) : lo; }
};
__device__ __forceinline__ bool block_seen(int c0, int lo, int keep_end, int pos) {
    return c0 < keep_end || (c0 <= pos && c0 + KB > lo);
}
struct Scoring {
    float scale, softcap;
    const float *dist_scale, *dist_rate;
    __device__ __forceinline__ float operator()(float dot, int h, int distance) const {
        float sc = dot * scale;
        if (softcap > 0.f) sc = softcap * tanhf(sc / softcap);
        if (dist_scale) sc -= dist_scale[h] * log1pf(dist_rate[h] * (float)distance);
        return sc;
    }
};
// Whether a block takes no part in a row's sum: none of its keys is seen, or all that are have a weight of zero. Scores that are no
// number leave no maximum either, but a sum that is none: they join, and the row's result is no number.
__device__ __forceinline__ bool block_empty(float mb, float lb) { return mb == -INFINITY && lb == lb; }
// What a block's exponentials are taken against: scores of minus infinity weigh nothing also where there are no others.
__device__ __forceinline__ float block_base(float mb) { return mb == -INFINITY ? 0.f : mb; }
// the factors by which what is held and a further block enter their sum
__device__ __forceinline__ void join(float& m, float& l, float mb, float lb, float& held, float& fresh) {
    const float m_new = fmaxf(m, mb);
    held = m == -INFINITY ? 0.f : expf(m - m_new);
    fresh = expf(mb - m_new);
    l = fmaf(l, held, __fmul_rn(lb, fresh));
    m = m_new;
}
__device__ __forceinline__ float join_value(float acc, float held, float block, float fresh) {
    return fmaf(acc, held, __fmul_rn(block, fresh));
}
// the sink and the gate: returns the factor of the finished output
__device__ __forceinline__ float finish_factor(float& m, float& l, const float* sinks, int h, const float* gate, int gate_ld, int t,
                                               float& held) {
    held = 1.f;
    if (sinks) {
        const float sk = sinks[h];
        const float m_new = fmaxf(m, sk);
        held = expf(m - m_new);
        l = l * held + expf(sk - m_new);
    }
    return gate ? 1.0f / (l * (1.0f + expf(-gate[(long long)t * gate_ld + h]))) : 1.0f / l;
}

__device__ __forceinline__ void copy16(void* smem, const void* gmem, bool real) {
    const unsigned to = (unsigned)__cvta_generic_to_shared(smem);
    const int bytes = real ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(gmem), "r"(bytes) : "memory");
}

// Where the 128 keys of a block begin (keys of key head g; values lie G * page_size * hd further), -1 for those that nobody sees: worked out
// once per block, so that the copies need neither the page table nor a division.
template <typename Seen>
__device__ __forceinline__ void find_rows(long long* rows, int c0, const int* pt, int page_size, int G, int g, int hd, Seen seen) {
    if ((int)threadIdx.x < KB) {
        const int key = c0 + threadIdx.x;
        long long at = -1;
        if (seen(key)) {
            const int page = pt[key / page_size];
            if (page >= 0) at = (((long long)page * 2 * G + g) * page_size + key % page_size) * hd;
        }
        rows[threadIdx.x] = at;
    }
}
// rows of hd values (hd a multiple of 4) to shared memory, `stride` floats apart, by all THREADS threads
template <int THREADS>
__device__ __forceinline__ void copy_rows(float* to, int stride, const float* from, const long long* rows, int hd) {
    const int n4 = hd / 4, step_row = THREADS / n4, step_piece = THREADS % n4;
    int j = threadIdx.x / n4, c = threadIdx.x % n4;
    while (j < KB) {
        const long long at = rows[j];
        copy16(to + j * stride + c * 4, at >= 0 ? from + at + c * 4 : from, at >= 0);
        j += step_row;
        c += step_piece;
        if (c >= n4) { c -= n4; ++j; }
    }
}

constexpr int TILE_WARPS = 8;

// Prompts: a tile of 8 * RW consecutive tokens and one head per CTA; a warp owns RW of its rows, a lane four keys of a
// block for the scores and features lane, lane + 32, ... for the values. Bound by the multiply-adds and the reads of shared
// memory that feed them (RW x 4 scores per lane: RW + 4 reads of 16 bytes for 16 RW multiply-adds). Four rows per warp and
// two CTAs per SM: 509 tokens, 32 heads of 64, B200: 1143 us with a block per query (above) -> 220 us with eight rows per
// warp and one CTA per SM -> 107 us -> 90 us with the keys' places worked out once per block and, for heads of up to 64, the values
// asked for together with the keys.
template <int NI, int RW>
__global__ void __launch_bounds__(TILE_WARPS * 32, NI <= 4 ? 2 : 1)
attention_f32_tile_kernel(const float* __restrict__ q, float* __restrict__ out, const float* __restrict__ pages,
                          const int* __restrict__ page_table, int pt_stride, const int* __restrict__ seq_ids,
                          const int* __restrict__ positions, int T, int H, int G, int hd, int page_size, Scoring scoring, Mask mask,
                          const float* __restrict__ sinks, const float* __restrict__ gate, int gate_ld) {
    constexpr int ROWS = TILE_WARPS * RW;
    extern __shared__ __align__(16) float smem[];
    const int stride = hd + 4;                    // a multiple of 4 floats that walks through the banks
    float* qs = smem;                             // [ROWS][stride]
    float* kv = qs + ROWS * stride;               // [KB][stride]: keys, then values unless these have room of their own
    constexpr bool BOTH = NI <= 2;                // there is room for the values beside the keys: asked for together
    float* vals = BOTH ? kv + KB * stride : kv;
    float* probs = vals + KB * stride;            // [warp][KB][RW]
    __shared__ int row_seq[ROWS], row_pos[ROWS];
    __shared__ long long key_rows[KB];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // the last tiles of a sequence have the most keys: they start first
    const int t0 = (int)(gridDim.y - 1 - blockIdx.y) * ROWS, h = blockIdx.x, g = h / (H / G);
    const int n4 = hd / 4;
    lp_grid_wait();
    lp_grid_release();
    for (int r = tid; r < ROWS; r += TILE_WARPS * 32) {
        row_seq[r] = t0 + r < T ? seq_ids[t0 + r] : -1;
        row_pos[r] = t0 + r < T ? positions[t0 + r] : -1;
    }
    for (int i = tid; i < ROWS * n4; i += TILE_WARPS * 32) {
        const int r = i / n4, c = i % n4 * 4;
        *(float4*)(qs + r * stride + c) = t0 + r < T ? *(const float4*)(q + ((long long)(t0 + r) * H + h) * hd + c)
                                                       : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();

    float m[RW], l[RW], acc[RW][NI];
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        m[r] = -INFINITY;
        l[r] = 0.f;
#pragma unroll
        for (int i = 0; i < NI; ++i) acc[r][i] = 0.f;
    }
    float* mine = probs + warp * KB * RW;
    // rows of one sequence after another (a tile of a prompt holds one or two)
    for (int first = 0; first < ROWS && row_seq[first] >= 0;) {
        const int seq = row_seq[first];
        int last = first, seg_pos = -1, seg_lo = 0x7fffffff, seg_kept = 0;
        for (; last < ROWS && row_seq[last] == seq; ++last) {
            const int lo = mask.first(row_pos[last]);
            seg_pos = max(seg_pos, row_pos[last]);
            seg_lo = min(seg_lo, lo);
            seg_kept = max(seg_kept, mask.kept(lo));
        }
        const int* pt = page_table + (long long)seq * pt_stride;
        for (int c0 = 0; c0 <= seg_pos; c0 += KB) {
            if (!block_seen(c0, seg_lo, seg_kept, seg_pos)) continue;
            find_rows(key_rows, c0, pt, page_size, G, g, hd,
                      [&](int key) { return key <= seg_pos && (key >= seg_lo || key < seg_kept); });      // other pages may be gone
            __syncthreads();
            copy_rows<TILE_WARPS * 32>(kv, stride, pages, key_rows, hd);
            asm volatile("cp.async.commit_group;" ::: "memory");
            if (BOTH) {
                copy_rows<TILE_WARPS * 32>(vals, stride, pages + (long long)G * page_size * hd, key_rows, hd);
                asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 1;" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            __syncthreads();
            bool active = false;
#pragma unroll
            for (int r = 0; r < RW; ++r) {
                const int row = warp * RW + r;
                if (row < first || row >= last) continue;
                const int lo = mask.first(row_pos[row]);
                active |= block_seen(c0, lo, mask.kept(lo), row_pos[row]);
            }
            float mb[RW], lb[RW];
            if (active) {
                float s[RW][4];
#pragma unroll
                for (int r = 0; r < RW; ++r)
#pragma unroll
                    for (int j = 0; j < 4; ++j) s[r][j] = 0.f;
                const float* qw = qs + warp * RW * stride;
                for (int c = 0; c < hd; c += 4) {
                    float4 k[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) k[j] = *(const float4*)(kv + (lane + 32 * j) * stride + c);
#pragma unroll
                    for (int r = 0; r < RW; ++r) {
                        const float4 a = *(const float4*)(qw + r * stride + c);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            s[r][j] = fmaf(a.x, k[j].x, s[r][j]);
                            s[r][j] = fmaf(a.y, k[j].y, s[r][j]);
                            s[r][j] = fmaf(a.z, k[j].z, s[r][j]);
                            s[r][j] = fmaf(a.w, k[j].w, s[r][j]);
                        }
                    }
                }
#pragma unroll
                for (int r = 0; r < RW; ++r) {
                    const int row = warp * RW + r, pos = row_pos[row];
                    const int lo = mask.first(pos), keep_end = mask.kept(lo);
                    const bool in_segment = row >= first && row < last;
                    float top = -INFINITY;
                    bool seen[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int key = c0 + lane + 32 * j;
                        seen[j] = in_segment && key <= pos && (key >= lo || key < keep_end);
                        s[r][j] = seen[j] ? scoring(s[r][j], h, pos - key) : -INFINITY;
                        top = fmaxf(top, s[r][j]);
                    }
                    mb[r] = lp_warp_max(top);
                    const float base = block_base(mb[r]);
                    float sum = 0.f;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float p = seen[j] ? expf(s[r][j] - base) : 0.f;
                        mine[(lane + 32 * j) * RW + r] = p;
                        sum += p;
                    }
                    lb[r] = lp_warp_sum(sum);
                }
            }
            if (!BOTH) {
                __syncthreads();                   // all warps are through with the keys
                copy_rows<TILE_WARPS * 32>(vals, stride, pages + (long long)G * page_size * hd, key_rows, hd);
                asm volatile("cp.async.commit_group;" ::: "memory");
            }
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            if (active) {
                float part[RW][NI];
#pragma unroll
                for (int r = 0; r < RW; ++r)
#pragma unroll
                    for (int i = 0; i < NI; ++i) part[r][i] = 0.f;
                const int count = min(KB, seg_pos - c0 + 1);
#pragma unroll 4
                for (int j = 0; j < count; ++j) {
                    float p[RW], v[NI];
#pragma unroll
                    for (int r = 0; r < RW; r += 4) {
                        const float4 four = *(const float4*)(mine + j * RW + r);
                        p[r] = four.x; p[r + 1] = four.y; p[r + 2] = four.z; p[r + 3] = four.w;
                    }
#pragma unroll
                    for (int i = 0; i < NI; ++i) v[i] = lane + 32 * i < hd ? vals[j * stride + lane + 32 * i] : 0.f;
#pragma unroll
                    for (int r = 0; r < RW; ++r)
                        if (p[r] > 0.f) {          // a weight of zero takes nothing from a row, whatever it holds
#pragma unroll
                            for (int i = 0; i < NI; ++i) part[r][i] = fmaf(p[r], v[i], part[r][i]);
                        }
                }
#pragma unroll
                for (int r = 0; r < RW; ++r) {
                    if (block_empty(mb[r], lb[r])) continue;
                    float held, fresh;
                    join(m[r], l[r], mb[r], lb[r], held, fresh);
#pragma unroll
                    for (int i = 0; i < NI; ++i) acc[r][i] = join_value(acc[r][i], held, part[r][i], fresh);
                }
            }
            __syncthreads();                       // all warps are through with the values
        }
        first = last;
    }
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        const int t = t0 + warp * RW + r;
        if (t >= T) continue;
        float held;
        const float inv = finish_factor(m[r], l[r], sinks, h, gate, gate_ld, t, held);
#pragma unroll
        for (int i = 0; i < NI; ++i)
            if (lane + 32 * i < hd) out[((long long)t * H + h) * hd + lane + 32 * i] = acc[r][i] * held * inv;
    }
}

// Steps of a few tokens per sequence: a CTA per (block of keys, key head, token) serves all query heads that share the key
// head (SHARE_HEADS at a time) and leaves maximum, sum and weighted values of its block; the blocks of long sequences lie side by
// side on the chip instead of one behind the other. Bound by the latency of one block's reads. 4 sequences of up to 700, 32 heads of 64 on
// 8, B200: 19.1 us with a division and a look into the page table per 16 bytes and a chain per head, now 10.4.
template <int SHARE_HEADS>
__global__ void __launch_bounds__(KB)
attention_f32_share_kernel(const float* __restrict__ q, float* __restrict__ parts, const float* __restrict__ pages,
                           const int* __restrict__ page_table, int pt_stride, const int* __restrict__ seq_ids,
                           const int* __restrict__ positions, int H, int G, int hd, int page_size, int blocks, Scoring scoring,
                           Mask mask) {
    extern __shared__ __align__(16) float smem[];
    const int stride = hd + 4;
    float* ks = smem;                             // [KB][stride]
    float* vs = ks + KB * stride;                 // [KB][hd]
    float* qs = vs + KB * hd;                     // [SHARE_HEADS][hd]
    __shared__ __align__(16) float probs[KB][SHARE_HEADS];
    __shared__ long long key_rows[KB];
    __shared__ float warp_max[SHARE_HEADS][KB / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b = blockIdx.x, g = blockIdx.y, t = blockIdx.z;
    lp_grid_wait();
    lp_grid_release();
    const int pos = positions[t], c0 = b * KB;
    const int lo = mask.first(pos), keep_end = mask.kept(lo);
    if (!block_seen(c0, lo, keep_end, pos)) return;
    const int* pt = page_table + (long long)seq_ids[t] * pt_stride;
    const int rep = H / G;
    find_rows(key_rows, c0, pt, page_size, G, g, hd, [&](int key) { return key <= pos && (key >= lo || key < keep_end); });
    __syncthreads();
    copy_rows<KB>(ks, stride, pages, key_rows, hd);
    asm volatile("cp.async.commit_group;" ::: "memory");
    copy_rows<KB>(vs, hd, pages + (long long)G * page_size * hd, key_rows, hd);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const int key = c0 + tid;
    const bool seen = key <= pos && (key >= lo || key < keep_end);
    for (int h0 = 0; h0 < rep; h0 += SHARE_HEADS) {
        const int heads = min(SHARE_HEADS, rep - h0);
        const float* from = q + ((long long)t * H + g * rep + h0) * hd;
        for (int i = tid; i < SHARE_HEADS * hd; i += KB) qs[i] = i < heads * hd ? from[i] : 0.f;
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        float s[SHARE_HEADS];
#pragma unroll
        for (int r = 0; r < SHARE_HEADS; ++r) s[r] = 0.f;
#pragma unroll 4
        for (int c = 0; c < hd; c += 4) {
            const float4 k = *(const float4*)(ks + tid * stride + c);
#pragma unroll
            for (int r = 0; r < SHARE_HEADS; ++r) {
                const float4 a = *(const float4*)(qs + r * hd + c);
                s[r] = fmaf(a.x, k.x, s[r]);
                s[r] = fmaf(a.y, k.y, s[r]);
                s[r] = fmaf(a.z, k.z, s[r]);
                s[r] = fmaf(a.w, k.w, s[r]);
            }
        }
#pragma unroll
        for (int r = 0; r < SHARE_HEADS; ++r) {
            s[r] = seen && r < heads ? scoring(s[r], g * rep + h0 + r, pos - key) : -INFINITY;
            const float top = lp_warp_max(s[r]);
            if (lane == 0) warp_max[r][warp] = top;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < SHARE_HEADS; ++r) {
            const float top = fmaxf(fmaxf(warp_max[r][0], warp_max[r][1]), fmaxf(warp_max[r][2], warp_max[r][3]));
            probs[tid][r] = seen && r < heads ? expf(s[r] - block_base(top)) : 0.f;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        const int count = min(KB, pos - c0 + 1);
        // neighbouring threads: neighbouring features; two heads' chains at a time where there are two
        constexpr int PAIR = SHARE_HEADS > 1 ? 2 : 1;
        for (int i = tid; i < hd * (SHARE_HEADS / PAIR); i += KB) {
            const int r = i / hd * PAIR, d = i % hd;
            if (r >= heads) break;
            float part[PAIR];
#pragma unroll
            for (int k = 0; k < PAIR; ++k) part[k] = 0.f;
#pragma unroll 16
            for (int j = 0; j < count; ++j) {
                const float v = vs[j * hd + d];
#pragma unroll
                for (int k = 0; k < PAIR; ++k) {
                    const float p = probs[j][r + k];
                    part[k] = p > 0.f ? fmaf(p, v, part[k]) : part[k];
                }
            }
#pragma unroll
            for (int k = 0; k < PAIR; ++k)
                if (r + k < heads) parts[(((long long)t * H + g * rep + h0 + r + k) * blocks + b) * (hd + 2) + 2 + d] = part[k];
        }
        for (int r = warp; r < heads; r += KB / 32) {
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) sum += probs[lane + 32 * j][r];
            sum = lp_warp_sum(sum);
            if (lane == 0) {
                float* to = parts + (((long long)t * H + g * rep + h0 + r) * blocks + b) * (hd + 2);
                to[0] = fmaxf(fmaxf(warp_max[r][0], warp_max[r][1]), fmaxf(warp_max[r][2], warp_max[r][3]));
                to[1] = sum;
            }
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(MAX_HD)
attention_f32_join_kernel(const float* __restrict__ parts, float* __restrict__ out, const int* __restrict__ positions, int H, int hd,
                          int blocks, Mask mask, const float* __restrict__ sinks, const float* __restrict__ gate, int gate_ld) {
    const int t = blockIdx.x, h = blockIdx.y, d = threadIdx.x;
    lp_grid_wait();
    lp_grid_release();
    const int pos = positions[t];
    const int lo = mask.first(pos), keep_end = mask.kept(lo);
    float m = -INFINITY, l = 0.f, acc = 0.f;
    const float* from = parts + ((long long)t * H + h) * blocks * (hd + 2);
    constexpr int AHEAD = 8;                       // blocks asked for before the first of them is used
    for (int b0 = 0; b0 < blocks && b0 * KB <= pos; b0 += AHEAD) {
        float mb[AHEAD], lb[AHEAD], vb[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            const int c0 = (b0 + i) * KB;
            const bool seen = b0 + i < blocks && c0 <= pos && block_seen(c0, lo, keep_end, pos);
            const float* p = from + (long long)(b0 + i) * (hd + 2);
            mb[i] = seen ? p[0] : -INFINITY;
            lb[i] = seen ? p[1] : 0.f;
            vb[i] = seen && d < hd ? p[2 + d] : 0.f;
        }
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            if (block_empty(mb[i], lb[i])) continue;
            float held, fresh;
            join(m, l, mb[i], lb[i], held, fresh);
            acc = join_value(acc, held, vb[i], fresh);
        }
    }
    float held;
    const float inv = finish_factor(m, l, sinks, h, gate, gate_ld, t, held);
    if (d < hd) out[((long long)t * H + h) * hd + d] = acc * held * inv;
}

int failed(cudaError_t err) {
    snprintf(lp_error_text, sizeof(lp_error_text), "attention_plain: %s", cudaGetErrorString(err));
    return (int)err;
}

template <int NI, int RW>
int launch_tile(const float* q, float* out, const float* pages, const int* page_table, int pt_stride, const int* seq_ids,
                const int* positions, int T, int H, int G, int hd, int page_size, Scoring scoring, Mask mask, const float* sinks,
                const float* gate, int gate_ld, cudaStream_t stream) {
    constexpr int ROWS = TILE_WARPS * RW;
    const size_t smem = ((size_t)(ROWS + (NI <= 2 ? 2 : 1) * KB) * (hd + 4) + (size_t)KB * ROWS) * sizeof(float);
    auto kernel = attention_f32_tile_kernel<NI, RW>;
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err == cudaSuccess)
        err = lp_launch(kernel, dim3(H, (T + ROWS - 1) / ROWS), dim3(TILE_WARPS * 32), smem, stream, q, out, pages, page_table,
                        pt_stride, seq_ids, positions, T, H, G, hd, page_size, scoring, mask, sinks, gate, gate_ld);
    return err == cudaSuccess ? lp_check_launch("attention_plain (tile)") : failed(err);
}

template <int HEADS>
int launch_shares(const float* q, float* parts, float* out, const float* pages, const int* page_table, int pt_stride, const int* seq_ids,
                  const int* positions, int T, int H, int G, int hd, int page_size, int blocks, Scoring scoring, Mask mask,
                  const float* sinks, const float* gate, int gate_ld, cudaStream_t stream) {
    const size_t smem = ((size_t)KB * (hd + 4) + (size_t)KB * hd + (size_t)HEADS * hd) * sizeof(float);
    auto kernel = attention_f32_share_kernel<HEADS>;
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err == cudaSuccess)
        err = lp_launch(kernel, dim3(blocks, G, T), dim3(KB), smem, stream, q, parts, pages, page_table, pt_stride, seq_ids, positions, H,
                        G, hd, page_size, blocks, scoring, mask);
    if (err == cudaSuccess)
        err = lp_launch(attention_f32_join_kernel, dim3(T, H), dim3((hd + 31) / 32 * 32), 0, stream, parts, out, positions, H, hd, blocks,
                        mask, sinks, gate, gate_ld);
    return err == cudaSuccess ? lp_check_launch("attention_plain (blocks)") : failed(err);
}

}  // namespace

// q, out: [T, H, hd]; pages: [num_pages, 2, G, page_size, hd]; page_table: [B, pt_stride];
// seq_ids, positions: [T]. window <= 0: all keys up to the query's position. softcap > 0: a score s becomes
// softcap * tanh(s / softcap) after the scale. sinks (optional): float32 [H], see the kernel. keep > 0 (with a window):
// the sequence's first `keep` tokens stay visible to every later query, at their true positions. chunk > 0: a query at p
// sees keys from p / chunk * chunk on only. dist_scale, dist_rate (optional, float32 [H] each): a key n positions back
// loses dist_scale[h] * ln(1 + dist_rate[h] * n) of its score. gate (optional, float32, rows of gate_ld values): head h's
// output of query token t is multiplied by sigmoid(gate[t, h]).
// parts (optional, float32): room for T * H * blocks * (hd + 2) values, blocks * 128 > every position: given it, float32
// queries over a float32 cache run with a CTA per block of keys (for steps of a few tokens per sequence).
extern "C" int lp_attention_plain(const void* q, void* out, int q_dtype, const void* pages, int kv_dtype,
                                  const int* page_table, int pt_stride, const int* seq_ids, const int* positions,
                                  int T, int H, int G, int hd, int page_size, float scale, int window,
                                  float softcap, const float* sinks, int keep, int chunk, const float* dist_scale,
                                  const float* dist_rate, const float* gate, int gate_ld, float* parts, int blocks, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (gate && gate_ld < H) LP_REFUSE("attention_plain: rows of %d gates for %d heads", gate_ld, H);
    if ((dist_scale == nullptr) != (dist_rate == nullptr)) LP_REFUSE("attention_plain: a distance bias has a scale and a rate per head");
    if (keep > 0 && window > 0 && chunk > 0) LP_REFUSE("attention_plain: kept first tokens (%d) and chunks (%d) exclude each other", keep, chunk);
    if (H <= 0 || G <= 0 || H % G) LP_REFUSE("attention_plain: %d query heads over %d key heads", H, G);
    if (hd <= 0 || hd > MAX_HD) LP_REFUSE("attention_plain: head size %d (supported: 1..%d)", hd, MAX_HD);
    if (page_size <= 0) LP_REFUSE("attention_plain: page size %d", page_size);
    if (H > 65535) LP_REFUSE("attention_plain: %d heads exceed the grid", H);
    if (parts && blocks <= 0) LP_REFUSE("attention_plain: room for %d blocks of keys", blocks);
    // rows that can be read 16 bytes at a time: the kernels made for that, others: the one for everything
    if (q_dtype == LP_F32 && kv_dtype == LP_F32 && hd % 4 == 0 && (size_t)q % 16 == 0 && (size_t)pages % 16 == 0
        && (T + 31) / 32 <= 65535) {
        const float *qf = (const float*)q, *pf = (const float*)pages;
        const Scoring scoring = {scale, softcap, dist_scale, dist_rate};
        const Mask mask = {window, keep, chunk};
        if (parts && T <= 65535 && G <= 65535) {
            const int rep = H / G;
            if (((size_t)KB * (hd + 4) + (size_t)KB * hd + 8 * (size_t)hd) * sizeof(float) <= 200 * 1024) {
                if (rep == 1)
                    return launch_shares<1>(qf, parts, (float*)out, pf, page_table, pt_stride, seq_ids, positions, T, H, G, hd, page_size,
                                            blocks, scoring, mask, sinks, gate, gate_ld, stream);
                if (rep <= 4)
                    return launch_shares<4>(qf, parts, (float*)out, pf, page_table, pt_stride, seq_ids, positions, T, H, G, hd, page_size,
                                            blocks, scoring, mask, sinks, gate, gate_ld, stream);
                return launch_shares<8>(qf, parts, (float*)out, pf, page_table, pt_stride, seq_ids, positions, T, H, G, hd, page_size,
                                        blocks, scoring, mask, sinks, gate, gate_ld, stream);
            }
        }
        if (hd <= 64)
            return launch_tile<2, 4>(qf, (float*)out, pf, page_table, pt_stride, seq_ids, positions, T, H, G, hd, page_size, scoring, mask,
                                     sinks, gate, gate_ld, stream);
        if (hd <= 128)
            return launch_tile<4, 4>(qf, (float*)out, pf, page_table, pt_stride, seq_ids, positions, T, H, G, hd, page_size, scoring, mask,
                                     sinks, gate, gate_ld, stream);
        return launch_tile<8, 4>(qf, (float*)out, pf, page_table, pt_stride, seq_ids, positions, T, H, G, hd, page_size, scoring, mask,
                                 sinks, gate, gate_ld, stream);
    }
    dim3 grid(T, H);
#define LP_LAUNCH_ATT(TQ, TKV)                                                                                 \
    attention_plain_kernel<TQ, TKV><<<grid, KB, 0, stream>>>((const TQ*)q, (TQ*)out, (const TKV*)pages,          \
                                                             page_table, pt_stride, seq_ids, positions, H, G,  \
                                                             hd, page_size, scale, window, softcap, sinks, keep, \
                                                             chunk, dist_scale, dist_rate, gate, gate_ld)
    if (q_dtype == LP_F32 && kv_dtype == LP_F32) LP_LAUNCH_ATT(float, float);
    else if (q_dtype == LP_BF16 && kv_dtype == LP_BF16) LP_LAUNCH_ATT(__nv_bfloat16, __nv_bfloat16);
    else if (q_dtype == LP_F32 && kv_dtype == LP_BF16) LP_LAUNCH_ATT(float, __nv_bfloat16);
    else if (q_dtype == LP_BF16 && kv_dtype == LP_F32) LP_LAUNCH_ATT(__nv_bfloat16, float);
    else LP_REFUSE("attention_plain: dtype codes q=%d kv=%d", q_dtype, kv_dtype);
#undef LP_LAUNCH_ATT
    return lp_check_launch("attention_plain");
}
