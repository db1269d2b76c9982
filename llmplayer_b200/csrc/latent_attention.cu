// Attention over a cache of low-rank latents ("latent attention").
//
// Every position of a sequence keeps one row [rank + dr]: the normed latent c (rank values) from which
// each head's keys and values are linear maps (K_h = U_h c, V_h = W_h c), and one rotated key part (dr
// values) that all heads share. A head's score against a position is
//     (q_n . U_h c + q_r . k_r) * scale  =  ((U_h^T q_n) . c + q_r . k_r) * scale,
// so the key map is applied to the query once ("absorbed") and every head attends over the same rows,
// and the head's output W_h (sum_j p_j c_j) applies the value map once to the weighted latent sum.
//
//   lp_latent_prepare   per token: RMS norm of the latent, rotation of the shared key part and of the
//                       queries' rotated parts, write of the row into the paged cache
//   lp_latent_absorb    q'[t, h] = [U_h^T q_n | q_r]
//   lp_latent_attend    online-softmax attention of q' over the rows of the pages (float32 scores,
//                       weights and sums), the keys of a sequence optionally shared out over several CTAs;
//                       over a bfloat16 cache the products run on the tensor cores, the queries and the
//                       weights as sums of three bfloat16 numbers (24 bits), the rows as they are
//   lp_latent_expand    merge of the shares, value map, output gate
//
// All arithmetic is float32 (or products of its exact parts); the cache and the weights may be bfloat16 or float32. Keys
// are visited in blocks of 32 (64 on the tensor cores) aligned to absolute positions, so a position's result does not depend on how its
// sequence was cut into steps or batched (the number of shares changes only the last merge).
#include "bf16_parts.cuh"
#include "tcgen05_utils.cuh"

namespace {

constexpr int KEYS = 32;            // keys per block: one per lane
constexpr int WARPS = 8;

// ---------------------------------------------------------------- prepare
template <typename TKV>
__global__ void __launch_bounds__(256)
latent_prepare_kernel(const float* __restrict__ proj, int ld, int q_off, int kv_off, const float* __restrict__ gain,
                      float eps, const float* __restrict__ inv_freq, int rot, const int* __restrict__ positions,
                      const int* __restrict__ seq_ids, const int* __restrict__ page_table, int pt_stride,
                      float* __restrict__ q_out, TKV* __restrict__ pages, int H, int dn, int dr, int rank,
                      int page_size, __nv_bfloat16* __restrict__ latent_out, __nv_bfloat16* __restrict__ shared_out,
                      __nv_bfloat16* __restrict__ q_half, int q_half_hd, const float* __restrict__ q_sep, int ldq,
                      int interleaved, float magnitude) {
    __shared__ float cs[128], sn[128];
    __shared__ float scratch[32];
    lp_grid_release();
    lp_grid_wait();
    const int t = blockIdx.x, tid = threadIdx.x;
    const int pos = positions[t];
    const int half = rot >> 1;
    for (int i = tid; i < half; i += blockDim.x) {
        float sv, cv;
        sincosf((float)pos * inv_freq[i], &sv, &cv);
        // a rotation may come with a factor on both cosine and sine (wavelength-stretched encodings)
        sn[i] = magnitude != 1.0f ? sv * magnitude : sv;
        cs[i] = magnitude != 1.0f ? cv * magnitude : cv;
    }
    const float* row = proj + (long long)t * ld;
    const float* kv = row + kv_off;
    float ss = 0.f;
    for (int i = tid; i < rank; i += blockDim.x) ss += kv[i] * kv[i];
    ss = lp_block_sum(ss, scratch);                       // also publishes cs / sn
    const float factor = 1.0f / sqrtf(ss / (float)rank + eps);
    const int page = page_table[(long long)seq_ids[t] * pt_stride + pos / page_size];
    const int Dk = rank + dr;
    TKV* dst = pages + ((long long)page * page_size + pos % page_size) * Dk;
    for (int i = tid; i < rank; i += blockDim.x) {
        const float c = kv[i] * factor * gain[i];
        dst[i] = lp_from_float<TKV>(c);
        if (latent_out) latent_out[(long long)t * rank + i] = __float2bfloat16_rn(c);
    }
    // the shared key part: pairs (i, i + half), or neighbours (2i, 2i + 1), of its first `rot` values turn, the rest pass
    const float* kr = kv + rank;
    for (int i = tid; i < dr; i += blockDim.x) {
        float v = kr[i];
        if (interleaved) {
            if (i < rot) {
                const int pr = i >> 1;
                v = (i & 1) ? __fadd_rn(__fmul_rn(kr[i], cs[pr]), __fmul_rn(kr[i - 1], sn[pr]))
                            : __fsub_rn(__fmul_rn(kr[i], cs[pr]), __fmul_rn(kr[i + 1], sn[pr]));
            }
        } else if (i < half) v = __fsub_rn(__fmul_rn(kr[i], cs[i]), __fmul_rn(kr[i + half], sn[i]));
        else if (i < rot) v = __fadd_rn(__fmul_rn(kr[i], cs[i - half]), __fmul_rn(kr[i - half], sn[i - half]));
        dst[rank + i] = lp_from_float<TKV>(v);
        if (shared_out) shared_out[(long long)t * dr + i] = __float2bfloat16_rn(v);
    }
    // queries: head by head [dn as projected | dr with the same rotation]
    const int hd = dn + dr;
    const float* q = q_sep ? q_sep + (long long)t * ldq : row + q_off;      // queries may come from a product of their own
    float* qo = q_out + (long long)t * H * hd;
    for (int e = tid; e < H * hd; e += blockDim.x) {
        const int i = e % hd - dn;
        float v = q[e];
        if (i >= 0) {
            if (interleaved) {
                if (i < rot) {
                    const int pr = i >> 1;
                    v = (i & 1) ? __fadd_rn(__fmul_rn(q[e], cs[pr]), __fmul_rn(q[e - 1], sn[pr]))
                                : __fsub_rn(__fmul_rn(q[e], cs[pr]), __fmul_rn(q[e + 1], sn[pr]));
                }
            } else if (i < half) v = __fsub_rn(__fmul_rn(q[e], cs[i]), __fmul_rn(q[e + half], sn[i]));
            else if (i < rot) v = __fadd_rn(__fmul_rn(q[e], cs[i - half]), __fmul_rn(q[e - half], sn[i - half]));
        }
        if (q_out) qo[e] = v;
        if (q_half) q_half[((long long)t * H + e / hd) * q_half_hd + e % hd] = __float2bfloat16_rn(v);
    }
    if (q_half && q_half_hd > hd) {                       // heads padded with zeros to a size the attention kernels take
        const int pad = q_half_hd - hd;
        for (int e = tid; e < H * pad; e += blockDim.x)
            q_half[((long long)t * H + e / pad) * q_half_hd + hd + e % pad] = __float2bfloat16_rn(0.f);
    }
}

// The same four values at a time (sizes, offsets and row lengths of a multiple of four, rotary halves as well; 16-byte
// aligned rows): a warp per head instead of a division per value, in steps of few tokens with CTAs of their own for the heads
// (8 tokens: 8.7 -> 6.8 us). Bound by its bytes and the latency of one token's steps: 1925 tokens, 16 heads of 192, rank 512, B200: 29 us value by
// value with the float32 queries -> 19 without them.
__device__ __forceinline__ void store4(float* to, const float* v) { *(float4*)to = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void store4(__nv_bfloat16* to, const float* v) {
    __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
    *(uint2*)to = make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
}
// values i .. i + 3 of a row part whose first `rot` values turn
__device__ __forceinline__ void rotate4(const float* x, int i, int rot, int interleaved, const float* cs, const float* sn, float* v) {
    const float4 a = *(const float4*)(x + i);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    const int half = rot >> 1;
    if (i >= rot) return;
    if (interleaved) {
#pragma unroll
        for (int k = 0; k < 4; k += 2) {
            const int pr = (i + k) >> 1;
            const float lo = v[k], hi = v[k + 1];
            v[k] = __fsub_rn(__fmul_rn(lo, cs[pr]), __fmul_rn(hi, sn[pr]));
            v[k + 1] = __fadd_rn(__fmul_rn(hi, cs[pr]), __fmul_rn(lo, sn[pr]));
        }
        return;
    }
    const bool first = i < half;
    const int at = first ? i : i - half;
    const float4 b = *(const float4*)(x + (first ? i + half : i - half));
    const float other[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int k = 0; k < 4; ++k)
        v[k] = first ? __fsub_rn(__fmul_rn(v[k], cs[at + k]), __fmul_rn(other[k], sn[at + k]))
                     : __fadd_rn(__fmul_rn(v[k], cs[at + k]), __fmul_rn(other[k], sn[at + k]));
}

template <typename TKV>
__global__ void __launch_bounds__(256)
latent_prepare_vec4_kernel(const float* __restrict__ proj, int ld, int q_off, int kv_off, const float* __restrict__ gain,
                           float eps, const float* __restrict__ inv_freq, int rot, const int* __restrict__ positions,
                           const int* __restrict__ seq_ids, const int* __restrict__ page_table, int pt_stride,
                           float* __restrict__ q_out, TKV* __restrict__ pages, int H, int dn, int dr, int rank,
                           int page_size, __nv_bfloat16* __restrict__ latent_out, __nv_bfloat16* __restrict__ shared_out,
                           __nv_bfloat16* __restrict__ q_half, int q_half_hd, const float* __restrict__ q_sep, int ldq,
                           int interleaved, float magnitude) {
    __shared__ float cs[128], sn[128];
    __shared__ float scratch[32];
    lp_grid_release();
    lp_grid_wait();
    const int t = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int pos = positions[t];
    const int half = rot >> 1;
    for (int i = tid; i < half; i += blockDim.x) {
        float sv, cv;
        sincosf((float)pos * inv_freq[i], &sv, &cv);
        sn[i] = magnitude != 1.0f ? sv * magnitude : sv;
        cs[i] = magnitude != 1.0f ? cv * magnitude : cv;
    }
    const float* row = proj + (long long)t * ld;
    const float* kv = row + kv_off;
    float ss = 0.f;
    // a grid of several CTAs per token: the first takes the latent and the shared key part, the others eight heads each
    const bool whole = gridDim.y == 1, takes_row = blockIdx.y == 0;
    for (int i = tid * 4; i < rank && takes_row; i += blockDim.x * 4) {
        const float4 v = *(const float4*)(kv + i);
        ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    }
    ss = lp_block_sum(ss, scratch);                       // also publishes cs / sn
    const float factor = 1.0f / sqrtf(ss / (float)rank + eps);
    const int page = page_table[(long long)seq_ids[t] * pt_stride + pos / page_size];
    const int Dk = rank + dr;
    TKV* dst = pages + ((long long)page * page_size + pos % page_size) * Dk;
    for (int i = tid * 4; i < rank && takes_row; i += blockDim.x * 4) {
        const float4 x = *(const float4*)(kv + i), g = *(const float4*)(gain + i);
        const float v[4] = {x.x * factor * g.x, x.y * factor * g.y, x.z * factor * g.z, x.w * factor * g.w};
        store4(dst + i, v);
        if (latent_out) store4(latent_out + (long long)t * rank + i, v);
    }
    for (int i = tid * 4; i < dr && takes_row; i += blockDim.x * 4) {
        float v[4];
        rotate4(kv + rank, i, rot, interleaved, cs, sn, v);
        store4(dst + rank + i, v);
        if (shared_out) store4(shared_out + (long long)t * dr + i, v);
    }
    if (takes_row && !whole) return;
    const int hd = dn + dr;
    const float* q = q_sep ? q_sep + (long long)t * ldq : row + q_off;
    for (int h = (whole ? 0 : ((int)blockIdx.y - 1) * 8) + warp; h < H; h += whole ? 8 : H) {
        const float* qh = q + h * hd;
        for (int i = lane * 4; i < max(hd, q_half ? q_half_hd : 0); i += 128) {
            float v[4] = {0.f, 0.f, 0.f, 0.f};            // heads padded with zeros to a size the attention kernels take
            if (i < dn) {
                const float4 x = *(const float4*)(qh + i);
                v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
            } else if (i < hd) {
                rotate4(qh + dn, i - dn, rot, interleaved, cs, sn, v);
            }
            if (q_out && i < hd) store4(q_out + ((long long)t * H + h) * hd + i, v);
            if (q_half) store4(q_half + ((long long)t * H + h) * q_half_hd + i, v);
        }
    }
}

// ---------------------------------------------------------------- per-head keys and values of a prompt
// For steps whose sequences all start at their first token, the heads' keys and values are formed outright
// (one product with the stacked key and value maps) and laid out as pages of keys and values, so that the
// tensor-core attention of ordinary heads serves: key of head h = [its unrotated part | the shared rotated
// part], both padded with zeros to heads of hd >= dn + dr (a size the attention kernels are built for), value of
// head h likewise. kv: bfloat16 [T, H * dn + H * dv].
__global__ void __launch_bounds__(256)
latent_heads_to_pages_kernel(const __nv_bfloat16* __restrict__ kv, const __nv_bfloat16* __restrict__ shared_part,
                             const int* __restrict__ positions, const int* __restrict__ seq_ids,
                             const int* __restrict__ table, int pt_stride, const int* __restrict__ kv_len,
                             __nv_bfloat16* __restrict__ pages, int H, int dn, int dr, int dv, int page_size, int hd) {
    lp_grid_release();
    lp_grid_wait();
    const int t = blockIdx.x;
    const int pos = positions[t];
    const int seq = seq_ids[t];
    const long long page = table[(long long)seq * pt_stride + pos / page_size];
    __nv_bfloat16* kdst = pages + page * 2 * H * page_size * hd + (long long)(pos % page_size) * hd;
    __nv_bfloat16* vdst = kdst + (long long)H * page_size * hd;
    const __nv_bfloat16* row = kv + (long long)t * H * (dn + dv);
    const __nv_bfloat16 zero = __float2bfloat16_rn(0.f);
    for (int e = threadIdx.x; e < H * hd; e += blockDim.x) {
        const int h = e / hd, i = e - h * hd;
        const long long at = (long long)h * page_size * hd + i;
        kdst[at] = i < dn ? row[h * dn + i] : (i < dn + dr ? shared_part[(long long)t * dr + i - dn] : zero);
        vdst[at] = i < dv ? row[H * dn + h * dv + i] : zero;
    }
    // the sequence's last token also clears the rest of its last page: the attention kernel multiplies those rows
    // by weights of zero, which only gives zero if the rows are finite
    if (pos == kv_len[seq] - 1) {
        const int rest = page_size - 1 - pos % page_size;
        for (long long e = threadIdx.x; e < (long long)H * rest * hd; e += blockDim.x) {
            const int h = (int)(e / ((long long)rest * hd));
            const long long at = (long long)h * page_size * hd + hd + (e - (long long)h * rest * hd);
            kdst[at] = zero;
            vdst[at] = zero;
        }
    }
}

// The same eight values at a time (sizes of a multiple of eight, 16-byte aligned buffers), the rows behind a sequence's last
// token shared out over its tokens: token n from the end clears rows n, n + length, ... Bound by its bytes: 1925 tokens, 16
// heads of 192, B200: 106 us with one block clearing them -> 14.
__global__ void __launch_bounds__(256)
latent_heads_to_pages_vec8_kernel(const __nv_bfloat16* __restrict__ kv, const __nv_bfloat16* __restrict__ shared_part,
                                  const int* __restrict__ positions, const int* __restrict__ seq_ids,
                                  const int* __restrict__ table, int pt_stride, const int* __restrict__ kv_len,
                                  __nv_bfloat16* __restrict__ pages, int H, int dn, int dr, int dv, int page_size, int hd) {
    lp_grid_release();
    lp_grid_wait();
    const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int pos = positions[t], seq = seq_ids[t], len = kv_len[seq];
    const long long page = table[(long long)seq * pt_stride + pos / page_size];
    __nv_bfloat16* kdst = pages + page * 2 * H * page_size * hd + (long long)(pos % page_size) * hd;
    __nv_bfloat16* vdst = kdst + (long long)H * page_size * hd;
    const __nv_bfloat16* row = kv + (long long)t * H * (dn + dv);
    const uint4 zero = make_uint4(0, 0, 0, 0);
    for (int h = warp; h < H; h += 8) {
        const long long at = (long long)h * page_size * hd;
        for (int i = lane * 8; i < hd; i += 256) {
            *(uint4*)(kdst + at + i) = i < dn ? *(const uint4*)(row + h * dn + i)
                                              : i < dn + dr ? *(const uint4*)(shared_part + (long long)t * dr + i - dn) : zero;
            *(uint4*)(vdst + at + i) = i < dv ? *(const uint4*)(row + H * dn + h * dv + i) : zero;
        }
    }
    const int used = (len - 1) % page_size + 1;           // rows of the last page that hold tokens
    const long long last = table[(long long)seq * pt_stride + (len - 1) / page_size];
    __nv_bfloat16* base = pages + last * 2 * H * page_size * hd;
    for (int r = used + len - 1 - pos; r < page_size; r += len)
        for (int e = threadIdx.x; e < 2 * H * (hd / 8); e += blockDim.x) {
            const int h = e / (hd / 8);                   // keys' heads, then values'
            *(uint4*)(base + ((long long)h * page_size + r) * hd + (e - h * (hd / 8)) * 8) = zero;
        }
}

// out[t, h * dv + v] = heads[t, h * hd + v] * sigmoid(gate[t, h]): the first dv features of each head, gated.
__global__ void __launch_bounds__(256)
latent_gate_heads_kernel(const __nv_bfloat16* __restrict__ heads, const float* __restrict__ gate, int ldg,
                         __nv_bfloat16* __restrict__ out, int T, int H, int hd, int dv, float* __restrict__ zero,
                         long long zero_count) {
    lp_grid_release();
    lp_grid_wait();
    clear_on_the_side(zero, zero_count);
    const long long n = (long long)T * H * dv;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const long long th = i / dv;
        const int v = (int)(i - th * dv);
        const long long t = th / H;
        const int h = (int)(th - t * H);
        float x = __bfloat162float(heads[th * hd + v]);
        if (gate) x *= 1.0f / (1.0f + expf(-gate[t * ldg + h]));
        out[i] = __float2bfloat16_rn(x);
    }
}

// The same, a warp per token and head, eight values per lane and step (head sizes of a multiple of eight, aligned buffers):
// the gate once per head instead of once per value. 1925 tokens, 16 heads of 192 / 128, B200: 21 us -> 7.
__global__ void __launch_bounds__(256)
latent_gate_heads_vec8_kernel(const __nv_bfloat16* __restrict__ heads, const float* __restrict__ gate, int ldg,
                              __nv_bfloat16* __restrict__ out, int rows, int H, int hd, int dv, float* __restrict__ zero,
                              long long zero_count) {
    lp_grid_release();
    lp_grid_wait();
    clear_on_the_side(zero, zero_count);
    const int lanes = dv / 8;                              // lanes that a row needs, at most 32
    const int per_warp = 32 / lanes, lane = threadIdx.x & 31;
    const int in_row = lane % lanes, sub = lane / lanes;
    if (sub >= per_warp) return;
    const int warps = gridDim.x * (blockDim.x >> 5);
    for (long long th = (long long)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * per_warp + sub; th < rows;
         th += (long long)warps * per_warp) {
        uint4 v = *(const uint4*)(heads + th * hd + in_row * 8);
        if (gate) {
            const long long t = th / H;
            const float g = 1.0f / (1.0f + expf(-gate[t * ldg + (th - t * H)]));
            __nv_bfloat162* pairs = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float2 f = __bfloat1622float2(pairs[k]);
                pairs[k] = __floats2bfloat162_rn(f.x * g, f.y * g);
            }
        }
        *(uint4*)(out + th * dv + in_row * 8) = v;
    }
}

// ---------------------------------------------------------------- absorb
constexpr int TOK_TILE = 8;

template <typename TW>
__global__ void __launch_bounds__(128)
latent_absorb_kernel(const float* __restrict__ q, const TW* __restrict__ uk, float* __restrict__ qa, int T, int H,
                     int dn, int dr, int rank) {
    extern __shared__ float qs[];                         // [TOK_TILE][dn]
    lp_grid_release();
    lp_grid_wait();
    const int t0 = blockIdx.x * TOK_TILE, h = blockIdx.y, tid = threadIdx.x;
    const int hd = dn + dr, Dk = rank + dr;
    const int nt = min(TOK_TILE, T - t0);
    for (int e = tid; e < TOK_TILE * dn; e += blockDim.x) {
        const int i = e / dn, d = e - i * dn;
        qs[e] = i < nt ? q[((long long)(t0 + i) * H + h) * hd + d] : 0.f;
    }
    __syncthreads();
    const TW* u = uk + (long long)h * dn * rank;
    for (int r = blockIdx.z * blockDim.x + tid; r < rank; r += gridDim.z * blockDim.x) {
        float acc[TOK_TILE];
#pragma unroll
        for (int i = 0; i < TOK_TILE; ++i) acc[i] = 0.f;
#pragma unroll 16
        for (int d = 0; d < dn; ++d) {
            const float w = lp_to_float(u[(long long)d * rank + r]);
#pragma unroll
            for (int i = 0; i < TOK_TILE; ++i) acc[i] = fmaf(qs[i * dn + d], w, acc[i]);
        }
#pragma unroll
        for (int i = 0; i < TOK_TILE; ++i)
            if (i < nt) qa[((long long)(t0 + i) * H + h) * Dk + r] = acc[i];
    }
    for (int e = blockIdx.z * blockDim.x + tid; e < nt * dr; e += gridDim.z * blockDim.x) {
        const int i = e / dr, d = e - i * dr;
        qa[((long long)(t0 + i) * H + h) * Dk + rank + d] = q[((long long)(t0 + i) * H + h) * hd + dn + d];
    }
}

// ---------------------------------------------------------------- attend
// A CTA takes ROWS = WARPS * RW consecutive (token, head) rows of one sequence (heads of a token lie
// together, so a warp's rows mostly share their causal limit) and one share of the sequence's key blocks.
// Per block of 32 keys: the rows of the block go to shared memory as float32; lane j scores key j for the
// warp's RW rows; maximum and sum are updated per row across the warp; then lane c owns columns c, c + 32,
// ... of the latent sum and adds the 32 weighted rows in increasing key order.
template <typename TKV, int RW, int NC>
__global__ void __launch_bounds__(WARPS * 32)
latent_attend_kernel(const float* __restrict__ qa, const TKV* __restrict__ pages, const int* __restrict__ page_table,
                     int pt_stride, const int* __restrict__ q_start, const int* __restrict__ kv_len,
                     float* __restrict__ part, int H, int rank, int dr, int page_size, float scale, int shares,
                     int window) {
    extern __shared__ __align__(16) float smem[];
    constexpr int ROWS = WARPS * RW;
    // rows of a multiple of 4 values are read four at a time (a key row's stride of Dk + 4 floats keeps the lanes'
    // 16-byte reads on distinct banks); other widths one value at a time with a stride of Dk + 1
    const int Dk = rank + dr;
    const bool vec = (Dk & 3) == 0;
    const int KS = vec ? Dk + 4 : Dk + 1;
    float* Qs = smem;                       // [ROWS][Dk]
    float* Ks = smem + ROWS * Dk;           // [KEYS][KS]
    lp_grid_release();
    lp_grid_wait();
    const int b = blockIdx.y, share = blockIdx.z;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int first_tok = q_start[b], n_new = q_start[b + 1] - first_tok;
    const int len = kv_len[b];
    const int rows_total = n_new * H;
    const int r0 = blockIdx.x * ROWS;
    if (r0 >= rows_total) return;
    const int n_rows = min(ROWS, rows_total - r0);
    const int first_pos = len - n_new;                    // position of the sequence's first new token
    // queries of this CTA
    for (int r = warp; r < ROWS; r += WARPS) {
        const float* src = qa + ((long long)first_tok * H + r0 + r) * Dk;
        for (int e = lane; e < Dk; e += 32) Qs[r * Dk + e] = r < n_rows ? src[e] : 0.f;
    }
    int pos_r[RW];
    float m[RW], l[RW], o[RW][NC];
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        const int row = r0 + warp * RW + r;
        pos_r[r] = row < rows_total ? first_pos + row / H : -1;
        m[r] = -INFINITY;
        l[r] = 0.f;
#pragma unroll
        for (int c = 0; c < NC; ++c) o[r][c] = 0.f;
    }
    const int last_pos = first_pos + (r0 + n_rows - 1) / H;          // the CTA's largest causal limit
    // the key blocks that some row of the CTA can see (up to the largest causal limit, and from the start of the
    // first row's window on) are cut into the shares
    const int cta_first_pos = first_pos + r0 / H;
    const int blk_first = window > 0 ? max(0, cta_first_pos - window + 1) / KEYS : 0;
    const int blk_end = last_pos / KEYS + 1;
    const int per = (blk_end - blk_first + shares - 1) / shares;
    const int blk_lo = blk_first + share * per;
    const int blk_hi = min(blk_lo + per, blk_end);
    const int* pt = page_table + (long long)b * pt_stride;
    for (int blk = blk_lo; blk < blk_hi; ++blk) {
        const int k0 = blk * KEYS;
        __syncthreads();                                  // the previous block has been used (and Qs is written)
        {
            // a warp brings keys warp, warp + 8, warp + 16, warp + 24 together, so that four loads are in flight per lane
            constexpr int PER = KEYS / WARPS;
            const TKV* src[PER];
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                const int kp = k0 + warp + u * WARPS;
                src[u] = kp <= last_pos ? pages + ((long long)pt[kp / page_size] * page_size + kp % page_size) * Dk : nullptr;
            }
#pragma unroll 2
            for (int e = lane; e < Dk; e += 32) {
                float v[PER];
#pragma unroll
                for (int u = 0; u < PER; ++u) v[u] = src[u] ? lp_to_float(src[u][e]) : 0.f;
#pragma unroll
                for (int u = 0; u < PER; ++u) Ks[(warp + u * WARPS) * KS + e] = v[u];
            }
        }
        __syncthreads();
        int warp_last = pos_r[0];
#pragma unroll
        for (int r = 1; r < RW; ++r) warp_last = max(warp_last, pos_r[r]);
        if (warp_last < k0) continue;                                 // nothing of this block is visible to the warp
        float dot[RW];
#pragma unroll
        for (int r = 0; r < RW; ++r) dot[r] = 0.f;
        const float* kr = Ks + lane * KS;
        const float* qw = Qs + warp * RW * Dk;
        if (vec) {
#pragma unroll 2
            for (int d = 0; d < Dk; d += 4) {
                const float4 kv = *reinterpret_cast<const float4*>(kr + d);
#pragma unroll
                for (int r = 0; r < RW; ++r) {
                    const float4 qv = *reinterpret_cast<const float4*>(qw + r * Dk + d);
                    dot[r] = fmaf(qv.x, kv.x, dot[r]);
                    dot[r] = fmaf(qv.y, kv.y, dot[r]);
                    dot[r] = fmaf(qv.z, kv.z, dot[r]);
                    dot[r] = fmaf(qv.w, kv.w, dot[r]);
                }
            }
        } else {
            for (int d = 0; d < Dk; ++d) {
                const float kv = kr[d];
#pragma unroll
                for (int r = 0; r < RW; ++r) dot[r] = fmaf(qw[r * Dk + d], kv, dot[r]);
            }
        }
        float p[RW];
#pragma unroll
        for (int r = 0; r < RW; ++r) {
            const bool seen = k0 + lane <= pos_r[r] && (window <= 0 || k0 + lane > pos_r[r] - window);
            const float sc = seen ? dot[r] * scale : -INFINITY;
            const float m_new = fmaxf(m[r], lp_warp_max(sc));
            float alpha = 1.f;
            p[r] = 0.f;
            if (m_new != -INFINITY) {
                p[r] = seen ? expf(sc - m_new) : 0.f;
                alpha = (m[r] == -INFINITY) ? 0.f : expf(m[r] - m_new);
            }
            l[r] = l[r] * alpha + lp_warp_sum(p[r]);
            m[r] = m_new;
#pragma unroll
            for (int c = 0; c < NC; ++c) o[r][c] *= alpha;
        }
        for (int j = 0; j < KEYS; ++j) {
            float pj[RW];
#pragma unroll
            for (int r = 0; r < RW; ++r) pj[r] = __shfl_sync(0xffffffffu, p[r], j);
            const float* cj = Ks + j * KS;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const int col = lane + 32 * c;
                if (col < rank) {
                    const float cv = cj[col];
#pragma unroll
                    for (int r = 0; r < RW; ++r) o[r][c] = fmaf(pj[r], cv, o[r][c]);
                }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < RW; ++r) {
        const int row = r0 + warp * RW + r;
        if (row >= rows_total) continue;
        float* dst = part + (((long long)first_tok * H + row) * shares + share) * (rank + 2);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int col = lane + 32 * c;
            if (col < rank) dst[col] = o[r][c];
        }
        if (lane == 0) {
            dst[rank] = m[r];
            dst[rank + 1] = l[r];
        }
    }
}

// ---------------------------------------------------------------- attend, on the tensor cores
// A bfloat16 row of the cache is an exact operand; a float32 query (or softmax weight) is the sum of three bfloat16
// numbers: 3 x 8 bits. So three mma.sync products per tile give the float32 scores and sums without rounding the query or
// the weights to fewer than 24 bits.
constexpr int TC_ROWS = 16;          // (token, head) rows of a CTA = MMA M
constexpr int TC_KEYS = 64;          // keys per block
constexpr int TC_PSTRIDE = TC_KEYS + 8, TC_SSTRIDE = TC_KEYS + 4;

constexpr int TC_BOX = TC_KEYS * 128;      // bytes of a block's 64 columns: rows of 128 bytes whose 16-byte pieces lie at piece ^ (row & 7)

__host__ __device__ constexpr int tc_stage(int Dk) { return (Dk + 63) / 64 * TC_BOX; }
__host__ __device__ constexpr size_t tc_smem(int Dk) {
    return 1024 + 2 * (size_t)tc_stage(Dk) + (size_t)3 * TC_ROWS * (Dk + 8) * 2 + (size_t)4 * TC_ROWS * TC_SSTRIDE * 4 +
           (size_t)3 * TC_ROWS * TC_PSTRIDE * 2;
}

// A CTA takes 16 (token, head) rows of one sequence and one share of its blocks of 64 keys; the next block's rows are on
// their way while a block is worked on, by TMA in boxes of 64 columns. Scores: a warp takes 32 keys and a quarter of the row's width, the
// quarters meet in shared memory; softmax: half a warp per row; sums: a warp takes an eighth of the latent's columns (NT tiles of
// 8). The boxes' swizzle, and row strides of an odd multiple of 16 bytes elsewhere, keep ldmatrix free of bank conflicts.
// Bound by the tensor instructions (3 x 72 + 3 x 64 per 16 keys and CTA at rank 512, rows of 576; 3,260 cycles of a block's 5,100)
// and the latency of a block's steps: 32 sequences of 750 to 1500 rows of 576, 16 heads, B200: 210 us with a lane per key
// (above) -> 32 (39 with cold caches) -> 26. Of the 32, stamped inside, the threads' own copies of 16 bytes took 2,230 cycles per block
// (a bulk copy per row is no better: 64 of them take one warp as long), the softmax with a warp per row and two rows behind one another 1,540, and reading the queries one
// round trip at a time 6,000 per CTA.
template <int NT>
__global__ void __launch_bounds__(WARPS * 32, 1)
latent_attend_tc_kernel(const __grid_constant__ CUtensorMap rows_map, const float* __restrict__ qa, const int* __restrict__ page_table,
                        int pt_stride, const int* __restrict__ q_start, const int* __restrict__ kv_len, float* __restrict__ part, int H,
                        int dr, int page_size, float scale, int shares, int window, int* __restrict__ status) {
    extern __shared__ __align__(16) uint8_t raw[];
    constexpr int rank = NT * 64;
    const int Dk = rank + dr, stride = Dk + 8;
    const uint32_t stage_bytes = tc_stage(Dk);
    uint8_t* Ks = raw + (1024 - (smem_at(raw) & 1023) & 1023);               // two stages of boxes, each box at a multiple of 1024
    __nv_bfloat16* Qs = (__nv_bfloat16*)(Ks + 2 * stage_bytes);               // [3][TC_ROWS][stride]
    float* Ss = (float*)(Qs + 3 * TC_ROWS * stride);                          // [4][TC_ROWS][TC_SSTRIDE]
    __nv_bfloat16* Ps = (__nv_bfloat16*)(Ss + 4 * TC_ROWS * TC_SSTRIDE);      // [3][TC_ROWS][TC_PSTRIDE]
    __shared__ float alphas[TC_ROWS];
    __shared__ uint64_t full[2];                                              // a stage's rows are there
    const int b = blockIdx.y, share = blockIdx.z;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        mbar_init(&full[0], 1);
        mbar_init(&full[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    lp_grid_release();
    lp_grid_wait();
    const int first_tok = q_start[b], n_new = q_start[b + 1] - first_tok;
    const int rows_total = n_new * H, r0 = blockIdx.x * TC_ROWS;
    if (r0 >= rows_total) return;
    const int n_rows = min(TC_ROWS, rows_total - r0);
    const int first_pos = kv_len[b] - n_new;
    const int last_pos = first_pos + (r0 + n_rows - 1) / H;
    const int blk_first = window > 0 ? max(0, first_pos + r0 / H - window + 1) / TC_KEYS : 0;
    const int blk_end = last_pos / TC_KEYS + 1;
    const int per = (blk_end - blk_first + shares - 1) / shares;
    const int blk_lo = blk_first + share * per, blk_hi = min(blk_lo + per, blk_end);
    const int* pt = page_table + (long long)b * pt_stride;
    // one lane of every warp asks for its share of a block's boxes (a box takes some 150 cycles to ask for)
    int page = lane == 0 && blk_lo < blk_hi ? pt[blk_lo * TC_KEYS / page_size] : 0;      // of the block to fetch next
    auto fetch = [&](int blk) {
        if (lane != 0 || blk >= blk_hi) return;
        const int k0 = blk * TC_KEYS, st = (blk - blk_lo) & 1;
        if (warp == 0) mbar_expect_tx(&full[st], stage_bytes);
        for (uint32_t c = warp; c * TC_BOX < stage_bytes; c += WARPS)
            tma_load_2d(Ks + st * stage_bytes + c * TC_BOX, &rows_map, c * 64, page * page_size + k0 % page_size, &full[st]);
        if (blk + 1 < blk_hi) page = pt[(k0 + TC_KEYS) / page_size];
    };
    __syncthreads();                                      // the barriers are set up
    fetch(blk_lo);
    constexpr int Q_LOADS = NT / 2 + 1;                   // float4s of a row per lane and turn
    for (int e0 = lane * 4; e0 < Dk; e0 += Q_LOADS * 128) {
        float4 x[2][Q_LOADS];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int u = 0; u < Q_LOADS; ++u) {
                const int r = warp + i * WARPS, e = e0 + u * 128;
                x[i][u] = r < n_rows && e < Dk ? *(const float4*)(qa + ((long long)first_tok * H + r0 + r) * Dk + e) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int u = 0; u < Q_LOADS; ++u) {
                const int r = warp + i * WARPS, e = e0 + u * 128;
                if (e >= Dk) continue;
                const float v[4] = {x[i][u].x, x[i][u].y, x[i][u].z, x[i][u].w};
                __nv_bfloat16 p[4][3];
#pragma unroll
                for (int j = 0; j < 4; ++j) three_parts(v[j], p[j]);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    __nv_bfloat162* to = (__nv_bfloat162*)(Qs + (k * TC_ROWS + r) * stride + e);
                    to[0] = __halves2bfloat162(p[0][k], p[1][k]);
                    to[1] = __halves2bfloat162(p[2][k], p[3][k]);
                }
            }
    }
    const int my_row = 2 * warp + (lane >> 4);            // of the softmax: half a warp per row
    const int my_pos = my_row < n_rows ? first_pos + (r0 + my_row) / H : -1;
    float m = -INFINITY, l = 0.f;
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[n][k] = 0.f;
    const int key_group = warp & 1, quarter = warp >> 1;
    const int k_steps = Dk / 16, step_lo = quarter * k_steps / 4, step_hi = (quarter + 1) * k_steps / 4;
    for (int blk = blk_lo; blk < blk_hi; ++blk) {
        fetch(blk + 1);
        const int turn = blk - blk_lo;
        const bool there = mbar_wait(&full[turn & 1], (turn >> 1) & 1);
        if (!__syncthreads_and(there)) {                  // a wait that ran out ends the block; its other copies are waited for first
            if (tid == 0) {
                atomicExch(status, 62);
                if (blk + 1 < blk_hi) mbar_wait(&full[(turn + 1) & 1], ((turn + 1) >> 1) & 1);
            }
            return;
        }
        uint8_t* K = Ks + (turn & 1) * stage_bytes;
        const int held = last_pos + 1 - blk * TC_KEYS;
        if (held < TC_KEYS) {                             // what lies behind the last position is no row: zeros
            const int per_row = stage_bytes / (TC_KEYS * 16);
            for (int e = tid; e < (TC_KEYS - held) * per_row; e += WARPS * 32) {
                const int r = held + e / per_row, c = e % per_row;
                *(uint4*)(K + (c >> 3) * TC_BOX + r * 128 + (c & 7) * 16) = make_uint4(0, 0, 0, 0);
            }
            __syncthreads();
        }
        {
            // a chain of products per part and tile of 8 keys: none waits for another
            float s[3][4][4];
#pragma unroll
            for (int p = 0; p < 3; ++p)
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int k = 0; k < 4; ++k) s[p][n][k] = 0.f;
            const uint32_t a_at = smem_at(Qs + (lane & 15) * stride + (lane >> 4) * 8);
            const uint32_t b_at = smem_at(K + (key_group * 32 + (lane >> 4) * 8 + (lane & 7)) * 128);
#pragma unroll 3
            for (int step = step_lo; step < step_hi; ++step) {
                uint32_t kf[2][4];
                const uint32_t at = b_at + (step >> 2) * TC_BOX + ((((step & 3) * 2 + ((lane >> 3) & 1)) ^ (lane & 7)) << 4);
                ldmatrix4(at, kf[0]);
                ldmatrix4(at + 16 * 128, kf[1]);
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    uint32_t qf[4];
                    ldmatrix4(a_at + p * TC_ROWS * stride * 2 + step * 32, qf);
#pragma unroll
                    for (int n = 0; n < 4; ++n) mma_bf16(s[p][n], qf, kf[n >> 1][(n & 1) * 2], kf[n >> 1][(n & 1) * 2 + 1]);
                }
            }
            float* to = Ss + (quarter * TC_ROWS + (lane >> 2)) * TC_SSTRIDE + key_group * 32 + (lane & 3) * 2;
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                float v[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] = s[0][n][k] + (s[1][n][k] + s[2][n][k]);
                *(float2*)(to + n * 8) = make_float2(v[0], v[1]);
                *(float2*)(to + 8 * TC_SSTRIDE + n * 8) = make_float2(v[2], v[3]);
            }
        }
        __syncthreads();
        {
            const int c = (lane & 15) * 4, key0 = blk * TC_KEYS + c;       // four neighbouring keys per lane
            const float* from = Ss + my_row * TC_SSTRIDE + c;
            float4 quarter4[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) quarter4[k] = *(const float4*)(from + k * TC_ROWS * TC_SSTRIDE);
            const float dot[4] = {(quarter4[0].x + quarter4[1].x) + (quarter4[2].x + quarter4[3].x),
                                  (quarter4[0].y + quarter4[1].y) + (quarter4[2].y + quarter4[3].y),
                                  (quarter4[0].z + quarter4[1].z) + (quarter4[2].z + quarter4[3].z),
                                  (quarter4[0].w + quarter4[1].w) + (quarter4[2].w + quarter4[3].w)};
            float sc[4];
            bool seen[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                seen[k] = key0 + k <= my_pos && (window <= 0 || key0 + k > my_pos - window);
                sc[k] = seen[k] ? dot[k] * scale : -INFINITY;
            }
            float top = fmaxf(fmaxf(sc[0], sc[1]), fmaxf(sc[2], sc[3]));
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
            const float m_new = fmaxf(m, top);
            float alpha = 1.f, p[4] = {0.f, 0.f, 0.f, 0.f};
            if (m_new != -INFINITY) {
#pragma unroll
                for (int k = 0; k < 4; ++k) p[k] = seen[k] ? expf(sc[k] - m_new) : 0.f;
                alpha = m == -INFINITY ? 0.f : expf(m - m_new);
            }
            float sum = (p[0] + p[1]) + (p[2] + p[3]);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            l = l * alpha + sum;
            m = m_new;
            if ((lane & 15) == 0) alphas[my_row] = alpha;
            __nv_bfloat16 parts[4][3];
#pragma unroll
            for (int k = 0; k < 4; ++k) three_parts(p[k], parts[k]);
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                __nv_bfloat162* to = (__nv_bfloat162*)(Ps + (q * TC_ROWS + my_row) * TC_PSTRIDE + c);
                to[0] = __halves2bfloat162(parts[0][q], parts[1][q]);
                to[1] = __halves2bfloat162(parts[2][q], parts[3][q]);
            }
        }
        __syncthreads();
        const float f0 = alphas[lane >> 2], f1 = alphas[(lane >> 2) + 8];
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            acc[n][0] *= f0;
            acc[n][1] *= f0;
            acc[n][2] *= f1;
            acc[n][3] *= f1;
        }
        const uint32_t p_at = smem_at(Ps + (lane & 15) * TC_PSTRIDE + (lane >> 4) * 8);
        const uint32_t c_at = smem_at(K + (lane & 15) * 128);
#pragma unroll
        for (int step = 0; step < TC_KEYS / 16; ++step) {
            uint32_t pf[3][4];
#pragma unroll
            for (int p = 0; p < 3; ++p) ldmatrix4(p_at + p * TC_ROWS * TC_PSTRIDE * 2 + step * 32, pf[p]);
#pragma unroll
            for (int n = 0; n < NT; n += 2) {
                uint32_t cf[4];
                // (NT = 1: the second tile belongs to the next warp or to the key part; it is read and not used)
                const int piece = warp * NT + n + (lane >> 4);
                ldmatrix4_trans(c_at + step * 16 * 128 + (piece >> 3) * TC_BOX + (((piece & 7) ^ (lane & 7)) << 4), cf);
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    mma_bf16(acc[n], pf[p], cf[0], cf[1]);
                    if (n + 1 < NT) mma_bf16(acc[n + 1 < NT ? n + 1 : n], pf[p], cf[2], cf[3]);
                }
            }
        }
        __syncthreads();                                  // the block's rows may be overwritten
    }
    const int row_a = lane >> 2, col = warp * (NT * 8) + (lane & 3) * 2;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int r = row_a + 8 * i;
        if (r >= n_rows) continue;
        float* dst = part + (((long long)first_tok * H + r0 + r) * shares + share) * (rank + 2) + col;
#pragma unroll
        for (int n = 0; n < NT; ++n) *(float2*)(dst + n * 8) = make_float2(acc[n][2 * i], acc[n][2 * i + 1]);
    }
    if ((lane & 15) == 0 && my_row < n_rows)
        *(float2*)(part + (((long long)first_tok * H + r0 + my_row) * shares + share) * (rank + 2) + rank) = make_float2(m, l);
}

// Whether the tensor-core kernel serves these sizes: a rank of 64, 128, 256 or 512, rows of a multiple of 16 values that
// fit shared memory, pages of whole blocks.
inline bool attend_on_tensor_cores(int kv_dtype, int rank, int dr, int page_size) {
    return kv_dtype == LP_BF16 && (rank == 64 || rank == 128 || rank == 256 || rank == 512) && dr % 16 == 0 &&
           page_size % TC_KEYS == 0 && tc_smem(rank + dr) <= 227 * 1024 - 256;
}

// ---------------------------------------------------------------- merge
// The shares of one (token, head) row become one: out = [sum_s o_s e^(m_s - M) / sum_s l_s e^(m_s - M) | 0 | 1],
// the form of a single share whose sum of weights is one. One CTA per row; every warp forms the weights.
__global__ void __launch_bounds__(128)
latent_merge_kernel(const float* __restrict__ part, int shares, float* __restrict__ out, int rank) {
    extern __shared__ float ws[];                         // [shares]
    lp_grid_release();
    lp_grid_wait();
    const int tid = threadIdx.x, lane = tid & 31;
    const int width = rank + 2;
    const float* p = part + (long long)blockIdx.x * shares * width;
    float M = -INFINITY;
    for (int s = lane; s < shares; s += 32) M = fmaxf(M, p[s * width + rank]);
    M = lp_warp_max(M);
    float L = 0.f;
    for (int s = lane; s < shares; s += 32) {
        const float ms = p[s * width + rank];
        L += ms == -INFINITY ? 0.f : p[s * width + rank + 1] * expf(ms - M);
    }
    L = lp_warp_sum(L);
    const float inv = 1.0f / L;
    if (tid < 32)
        for (int s = lane; s < shares; s += 32) {
            const float ms = p[s * width + rank];
            ws[s] = ms == -INFINITY ? 0.f : expf(ms - M) * inv;
        }
    __syncthreads();
    float* dst = out + (long long)blockIdx.x * width;
    for (int r = tid; r < rank; r += blockDim.x) {
        float acc = 0.f;
#pragma unroll 8
        for (int s = 0; s < shares; ++s) acc = fmaf(p[(long long)s * width + r], ws[s], acc);
        dst[r] = acc;
    }
    if (tid == 0) {
        dst[rank] = 0.f;
        dst[rank + 1] = 1.f;
    }
}

// ---------------------------------------------------------------- expand
// out[t, h * dv + v] = gate(t, h) * sum_r W[h * dv + v, r] * latent[t, h, r], where latent is the merge of
// the shares: sum_s o_s e^(m_s - M) / sum_s l_s e^(m_s - M). One warp per output feature, lanes over r.
template <typename TW, typename TOut>
__global__ void __launch_bounds__(128)
latent_expand_kernel(const float* __restrict__ part, int shares, const TW* __restrict__ uv,
                     const float* __restrict__ gate, int ldg, TOut* __restrict__ out, int T, int H, int rank, int dv,
                     float* __restrict__ zero, long long zero_count) {
    extern __shared__ float ls[];                         // [TOK_TILE][rank], then [TOK_TILE][shares] weights
    __shared__ float gs[TOK_TILE];
    float* ws = ls + TOK_TILE * rank;
    lp_grid_release();
    lp_grid_wait();
    clear_on_the_side(zero, zero_count);
    const int t0 = blockIdx.x * TOK_TILE, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nt = min(TOK_TILE, T - t0);
    const int width = rank + 2;
    // each share's weight e^(m_s - M) / sum_s l_s e^(m_s - M): a warp per token, lanes over shares
    for (int i = warp; i < nt; i += 4) {
        const float* p = part + ((long long)(t0 + i) * H + h) * shares * width;
        float M = -INFINITY;
        for (int s = lane; s < shares; s += 32) M = fmaxf(M, p[s * width + rank]);
        M = lp_warp_max(M);
        float L = 0.f;
        for (int s = lane; s < shares; s += 32) {
            const float ms = p[s * width + rank];
            const float e = ms == -INFINITY ? 0.f : expf(ms - M);
            ws[i * shares + s] = e;
            L += p[s * width + rank + 1] * e;
        }
        L = lp_warp_sum(L);
        const float inv = 1.0f / L;
        for (int s = lane; s < shares; s += 32) ws[i * shares + s] *= inv;
        if (lane == 0) gs[i] = gate ? 1.0f / (1.0f + expf(-gate[(long long)(t0 + i) * ldg + h])) : 1.0f;
    }
    __syncthreads();
    for (int e = tid; e < TOK_TILE * rank; e += blockDim.x) {
        const int i = e / rank, r = e - i * rank;
        float acc = 0.f;
        if (i < nt) {
            const float* p = part + ((long long)(t0 + i) * H + h) * shares * width + r;
            const float* wi = ws + i * shares;
#pragma unroll 4
            for (int s = 0; s < shares; ++s) acc = fmaf(p[(long long)s * width], wi[s], acc);
        }
        ls[e] = acc;
    }
    __syncthreads();
    for (int v = blockIdx.z * 4 + warp; v < dv; v += gridDim.z * 4) {
        const TW* w = uv + ((long long)h * dv + v) * rank;
        float acc[TOK_TILE];
#pragma unroll
        for (int i = 0; i < TOK_TILE; ++i) acc[i] = 0.f;
#pragma unroll 8
        for (int r = lane; r < rank; r += 32) {
            const float wv = lp_to_float(w[r]);
#pragma unroll
            for (int i = 0; i < TOK_TILE; ++i) acc[i] = fmaf(ls[i * rank + r], wv, acc[i]);
        }
#pragma unroll
        for (int i = 0; i < TOK_TILE; ++i) {
            const float s = lp_warp_sum(acc[i]);
            if (lane == 0 && i < nt) out[((long long)(t0 + i) * H + h) * dv + v] = lp_from_float<TOut>(s * gs[i]);
        }
    }
}

// The same for a step of few tokens, one CTA per (token, head) row: the row's shares are merged by all threads,
// then each warp forms value features of the row (lanes over the latent).
template <typename TW, typename TOut>
__global__ void __launch_bounds__(256)
latent_expand_rows_kernel(const float* __restrict__ part, int shares, const TW* __restrict__ uv,
                          const float* __restrict__ gate, int ldg, TOut* __restrict__ out, int H, int rank, int dv,
                          float* __restrict__ zero, long long zero_count) {
    extern __shared__ float ls[];                         // [rank] merged latent, then [shares] weights
    float* ws = ls + rank;
    lp_grid_release();
    lp_grid_wait();
    clear_on_the_side(zero, zero_count);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row = blockIdx.x, t = row / H, h = row - t * H;
    const int width = rank + 2;
    const float* p = part + (long long)row * shares * width;
    float M = -INFINITY;
    for (int s = lane; s < shares; s += 32) M = fmaxf(M, p[s * width + rank]);
    M = lp_warp_max(M);
    float L = 0.f;
    for (int s = lane; s < shares; s += 32) {
        const float ms = p[s * width + rank];
        L += ms == -INFINITY ? 0.f : p[s * width + rank + 1] * expf(ms - M);
    }
    L = lp_warp_sum(L);
    const float inv = 1.0f / L;
    if (warp == 0)
        for (int s = lane; s < shares; s += 32) {
            const float ms = p[s * width + rank];
            ws[s] = ms == -INFINITY ? 0.f : expf(ms - M) * inv;
        }
    __syncthreads();
    for (int r = tid; r < rank; r += blockDim.x) {
        float acc = 0.f;
#pragma unroll 8
        for (int s = 0; s < shares; ++s) acc = fmaf(p[(long long)s * width + r], ws[s], acc);
        ls[r] = acc;
    }
    __syncthreads();
    const float g = gate ? 1.0f / (1.0f + expf(-gate[(long long)t * ldg + h])) : 1.0f;
    for (int v = warp; v < dv; v += 8) {
        const TW* w = uv + ((long long)h * dv + v) * rank;
        float acc = 0.f;
#pragma unroll 8
        for (int r = lane; r < rank; r += 32) acc = fmaf(ls[r], lp_to_float(w[r]), acc);
        acc = lp_warp_sum(acc);
        if (lane == 0) out[(long long)row * dv + v] = lp_from_float<TOut>(acc * g);
    }
}

// ---------------------------------------------------------------- absorb and expand on the tensor cores
// Both maps are products per head with bfloat16 weights and a float32 operand: the weights are exact operands, the other is
// split into three bfloat16 parts (24 bits), sums are float32. 16 tokens per CTA, so a head's weights are read once per 16
// tokens, from L2.

// qa[t, h, r] = sum over d of uk[h, d, r] q[t, h, d]: 64 columns of the latent per CTA, 16 per warp. Bound by latency: 32
// tokens, 16 heads of 128, rank 512, B200: 28 us with a thread per column (above) -> 12 (cold caches).
// With `k.pages` the same launch does what latent_prepare does in front of it: the queries come as the projection leaves them
// (their rope parts are rotated on the way), and CTAs of their own (blockIdx.y == H) norm the tokens' latents, rotate the shared
// key parts and write both into the cache. A decode step's chain loses
// a kernel: a layer with 32 sequences, captured, B200: 59.6 -> 56.1 us; a request of 8 x 300 tokens and 16 steps to a hybrid of 4
// layers 5330 -> 5174. Queries read four values at a time, all in flight, took the absorb alone from 5.9 to 5.0 us (8 tokens 4.5 -> 3.4).
struct KeyRows {
    const float* kv;                // [T, ld]: the latent and the shared key part of a token, rank + dr values
    int ld;
    const float* gain;
    float eps;
    const float* inv_freq;
    int rot, interleaved;
    float magnitude;
    const int *positions, *seq_ids, *page_table;
    int pt_stride, page_size;
    __nv_bfloat16* pages;           // null: no keys, and queries whose rope parts are rotated already
};
// unit u of a part of dr values whose first `rot` turn: a pair of them, or one that passes
template <typename F>
__device__ __forceinline__ void rope_unit(const KeyRows& k, const float* x, int u, int pos, F store) {
    const int half = k.rot >> 1;
    if (u >= half) {
        store(u + half, x[u + half]);
        return;
    }
    float sn, cs;
    sincosf((float)pos * k.inv_freq[u], &sn, &cs);
    if (k.magnitude != 1.0f) {
        sn *= k.magnitude;
        cs *= k.magnitude;
    }
    const int i = k.interleaved ? 2 * u : u, j = k.interleaved ? 2 * u + 1 : u + half;
    const float lo = x[i], hi = x[j];
    store(i, __fsub_rn(__fmul_rn(lo, cs), __fmul_rn(hi, sn)));
    store(j, __fadd_rn(__fmul_rn(hi, cs), __fmul_rn(lo, sn)));
}

constexpr int AB_COLS = 64, AB_WARPS = 4;
__global__ void __launch_bounds__(AB_WARPS * 32)
latent_absorb_tc_kernel(const float* __restrict__ q, int ldq, const __nv_bfloat16* __restrict__ uk, float* __restrict__ qa, int T, int H,
                        int dn, int dr, int rank, const KeyRows k) {
    extern __shared__ __align__(16) uint8_t raw[];
    const int stride = dn + 8;
    constexpr int WSTRIDE = AB_COLS + 8;
    __nv_bfloat16* Qs = (__nv_bfloat16*)raw;                  // [3][16][stride]
    __nv_bfloat16* Ws = Qs + 3 * TC_ROWS * stride;            // [dn][WSTRIDE]
    const int t0 = blockIdx.x * TC_ROWS, h = blockIdx.y, c0 = blockIdx.z * AB_COLS;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int hd = dn + dr, Dk = rank + dr, nt = min(TC_ROWS, T - t0), units = dr - (k.rot >> 1);
    if (h == H) {                                             // the tokens' rows of the cache, shared out over blockIdx.z
        __shared__ float scratch[32];
        lp_grid_release();
        lp_grid_wait();
        for (int i = blockIdx.z; i < nt; i += gridDim.z) {
            const int t = t0 + i, pos = k.positions[t];
            const float* kv = k.kv + (long long)t * k.ld;
            const int page = k.page_table[(long long)k.seq_ids[t] * k.pt_stride + pos / k.page_size];
            __nv_bfloat16* dst = k.pages + ((long long)page * k.page_size + pos % k.page_size) * Dk;
            for (int u = tid; u < units; u += AB_WARPS * 32)
                rope_unit(k, kv + rank, u, pos, [&](int c, float v) { dst[rank + c] = __float2bfloat16_rn(v); });
            float ss = 0.f;
            for (int c = tid * 4; c < rank; c += AB_WARPS * 128) {
                const float4 v = *(const float4*)(kv + c);
                ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;      // (in the order of latent_prepare_vec4_kernel: the same bits)
            }
            const float factor = 1.0f / sqrtf(lp_block_sum(ss, scratch) / (float)rank + k.eps);
            for (int c = tid * 4; c < rank; c += AB_WARPS * 128) {
                const float4 v = *(const float4*)(kv + c), g = *(const float4*)(k.gain + c);
                const float normed[4] = {v.x * factor * g.x, v.y * factor * g.y, v.z * factor * g.z, v.w * factor * g.w};
                store4(dst + c, normed);
            }
        }
        return;
    }
    // weights are written by no kernel of a step: asked for before the wait
    for (int i = tid; i < dn * (AB_COLS / 8); i += AB_WARPS * 32) {
        const int d = i / (AB_COLS / 8), c = i % (AB_COLS / 8) * 8;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                     ::"r"(smem_at(Ws + d * WSTRIDE + c)), "l"(uk + ((long long)h * dn + d) * rank + c0 + c) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    lp_grid_release();
    lp_grid_wait();
    const float* first = q + (long long)t0 * ldq + h * hd;    // of the tile's first token
    const int quads = dn >> 2;
#pragma unroll 4
    for (int e = tid; e < TC_ROWS * quads; e += AB_WARPS * 32) {
        const int i = e / quads, d = (e - i * quads) * 4;
        const float4 x = i < nt ? *(const float4*)(first + (long long)i * ldq + d) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float v[4] = {x.x, x.y, x.z, x.w};
        __nv_bfloat16 p[4][3];
#pragma unroll
        for (int j = 0; j < 4; ++j) three_parts(v[j], p[j]);
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            __nv_bfloat162* to = (__nv_bfloat162*)(Qs + (m * TC_ROWS + i) * stride + d);
            to[0] = __halves2bfloat162(p[0][m], p[1][m]);
            to[1] = __halves2bfloat162(p[2][m], p[3][m]);
        }
    }
    if (blockIdx.z == 0)
        for (int e = tid; e < nt * units; e += AB_WARPS * 32) {
            const int i = e / units;
            float* to = qa + ((long long)(t0 + i) * H + h) * Dk + rank;
            rope_unit(k, first + (long long)i * ldq + dn, e - i * units, k.pages ? k.positions[t0 + i] : 0, [&](int c, float v) { to[c] = v; });
        }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    const uint32_t a_at = smem_at(Qs + (lane & 15) * stride + (lane >> 4) * 8);
    const uint32_t b_at = smem_at(Ws + (lane & 15) * WSTRIDE + warp * 16 + (lane >> 4) * 8);
    for (int step = 0; step < dn / 16; ++step) {
        uint32_t wf[4];
        ldmatrix4_trans(b_at + step * 16 * WSTRIDE * 2, wf);
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            uint32_t qf[4];
            ldmatrix4(a_at + p * TC_ROWS * stride * 2 + step * 32, qf);
            mma_bf16(acc[0], qf, wf[0], wf[1]);
            mma_bf16(acc[1], qf, wf[2], wf[3]);
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int r = (lane >> 2) + 8 * i;
        if (r >= nt) continue;
        float* to = qa + ((long long)(t0 + r) * H + h) * Dk + c0 + warp * 16 + (lane & 3) * 2;
#pragma unroll
        for (int n = 0; n < 2; ++n) *(float2*)(to + n * 8) = make_float2(acc[n][2 * i], acc[n][2 * i + 1]);
    }
}

// out[t, h * dv + v] = gate * sum over r of uv[h, v, r] latent[t, h, r], the latent being the merge of the shares: 32 value
// features per CTA, 8 per pair of warps, each with half of the rank; the halves meet in shared memory. The CL CTAs of a cluster
// have the same rows: each merges the shares of 1 / CL of the latent's columns and leaves them in all of them. Bound by latency: 32 tokens,
// 16 heads of 128, rank 512, 4 shares, B200: 26 us with a CTA per row (above) -> 19 (cold caches; 38 with one row's shares asked for at a
// time). Warm, one launch behind the other, every CTA merging all columns / clusters of 4: 64 tokens of 2 shares 14.4 / 9.7, 32 of 4 11.8 / 8.6,
// 8 of 8 9.4 / 5.9, 4 of 16 9.2 / 6.7, 2 of 16 7.0 / 6.0, 1 of 16 5.9 / 6.3: one token goes without.
constexpr int EX_FEATURES = 32, EX_WARPS = 8;
template <typename TOut, int CL>
__global__ void __cluster_dims__(1, 1, CL) __launch_bounds__(EX_WARPS * 32, 2)
latent_expand_tc_kernel(const float* __restrict__ part, int shares, const __nv_bfloat16* __restrict__ uv, const float* __restrict__ gate,
                        int ldg, TOut* __restrict__ out, int T, int H, int rank, int dv, float* __restrict__ zero, long long zero_count) {
    extern __shared__ __align__(16) uint8_t raw[];
    const int stride = rank + 8;
    __nv_bfloat16* Ls = (__nv_bfloat16*)raw;                  // [3][16][stride]
    __nv_bfloat16* Ws = Ls + 3 * TC_ROWS * stride;            // [EX_FEATURES][stride]
    float* ws = (float*)(Ws + EX_FEATURES * stride);          // [16][shares]
    __shared__ float gs[TC_ROWS];
    __shared__ float halves[TC_ROWS][EX_FEATURES];
    const int t0 = blockIdx.x * TC_ROWS, h = blockIdx.y, v0 = blockIdx.z * EX_FEATURES;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nt = min(TC_ROWS, T - t0), width = rank + 2, nv = min(EX_FEATURES, dv - v0);
    // a CTA stores into the others' shared memory only when all have started
    if (CL > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    for (int i = tid; i < EX_FEATURES * (rank / 8); i += EX_WARPS * 32) {
        const int v = i / (rank / 8), c = i % (rank / 8) * 8;
        const int bytes = v < nv ? 16 : 0;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                     ::"r"(smem_at(Ws + v * stride + c)), "l"(v < nv ? uv + ((long long)h * dv + v0 + v) * rank + c : uv), "r"(bytes) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    lp_grid_release();
    lp_grid_wait();
    clear_on_the_side(zero, zero_count);
    for (int i = warp; i < nt; i += EX_WARPS) {
        const float* p = part + ((long long)(t0 + i) * H + h) * shares * width + rank;
        const float g = gate ? gate[(long long)(t0 + i) * ldg + h] : 0.f;
        const float2 own = lane < shares ? *(const float2*)(p + (long long)lane * width) : make_float2(-INFINITY, 0.f);      // maximum, sum
        float M = own.x;
        for (int s = lane + 32; s < shares; s += 32) M = fmaxf(M, p[(long long)s * width]);
        M = lp_warp_max(M);
        const float e_own = own.x == -INFINITY ? 0.f : expf(own.x - M);
        float L = own.y * e_own;
        for (int s = lane + 32; s < shares; s += 32) {
            const float2 other = *(const float2*)(p + (long long)s * width);
            const float e = other.x == -INFINITY ? 0.f : expf(other.x - M);
            ws[i * shares + s] = e;
            L += other.y * e;
        }
        L = lp_warp_sum(L);
        const float inv = 1.0f / L;
        if (lane < shares) ws[i * shares + lane] = e_own * inv;
        for (int s = lane + 32; s < shares; s += 32) ws[i * shares + s] *= inv;
        if (lane == 0) gs[i] = gate ? 1.0f / (1.0f + expf(-g)) : 1.0f;
    }
    __syncthreads();
    if (CL > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    const int quads = rank / CL / 4, first = (blockIdx.z % CL) * (rank / CL);
#pragma unroll 2
    for (int e = tid; e < TC_ROWS * quads; e += EX_WARPS * 32) {
        const int i = e / quads, r = first + (e - i * quads) * 4;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (i < nt) {
            const float* p = part + ((long long)(t0 + i) * H + h) * shares * width + r;
            const float* wi = ws + i * shares;
#pragma unroll 4
            for (int s = 0; s < shares; ++s) {
                const float2 x = *(const float2*)(p + (long long)s * width), y = *(const float2*)(p + (long long)s * width + 2);
                v[0] = fmaf(x.x, wi[s], v[0]);
                v[1] = fmaf(x.y, wi[s], v[1]);
                v[2] = fmaf(y.x, wi[s], v[2]);
                v[3] = fmaf(y.y, wi[s], v[3]);
            }
        }
        __nv_bfloat16 parts[4][3];
#pragma unroll
        for (int j = 0; j < 4; ++j) three_parts(v[j], parts[j]);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const __nv_bfloat162 lo = __halves2bfloat162(parts[0][k], parts[1][k]), hi = __halves2bfloat162(parts[2][k], parts[3][k]);
            __nv_bfloat162* to = (__nv_bfloat162*)(Ls + (k * TC_ROWS + i) * stride + r);
            if (CL == 1) {
                to[0] = lo;
                to[1] = hi;
            } else {
#pragma unroll
                for (int peer = 0; peer < CL; ++peer) {
                    uint32_t at;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_at(to)), "r"(peer));
                    asm volatile("st.shared::cluster.v2.b32 [%0], {%1, %2};"
                                 ::"r"(at), "r"(*reinterpret_cast<const uint32_t*>(&lo)), "r"(*reinterpret_cast<const uint32_t*>(&hi)) : "memory");
                }
            }
        }
    }
    if (CL > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const int group = warp & 3, half = warp >> 2;             // 8 features; half of the rank
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    const int pairs = rank / 32;                              // steps of 32: two MMA steps per ldmatrix of the weights
    const uint32_t a_at = smem_at(Ls + (lane & 15) * stride + (lane >> 4) * 8);
    const uint32_t b_at = smem_at(Ws + (group * 8 + (lane & 7)) * stride + (lane >> 3) * 8);
#pragma unroll 2
    for (int step = half * pairs / 2; step < (half + 1) * pairs / 2; ++step) {
        uint32_t wf[4];
        ldmatrix4(b_at + step * 64, wf);
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                uint32_t lf[4];
                ldmatrix4(a_at + p * TC_ROWS * stride * 2 + step * 64 + k * 32, lf);
                mma_bf16(acc, lf, wf[2 * k], wf[2 * k + 1]);
            }
    }
    const int row = lane >> 2, col = group * 8 + (lane & 3) * 2;
    if (half) {
#pragma unroll
        for (int i = 0; i < 4; ++i) halves[row + (i >> 1) * 8][col + (i & 1)] = acc[i];
    }
    __syncthreads();
    if (!half) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = row + (i >> 1) * 8, v = col + (i & 1);
            if (r < nt && v < nv)
                out[((long long)(t0 + r) * H + h) * dv + v0 + v] = lp_from_float<TOut>((acc[i] + halves[r][v]) * gs[r]);
        }
    }
}

template <typename K>
int grant_shared(K kernel, size_t bytes, const char* what) {
    if (bytes > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e != cudaSuccess) {
            snprintf(lp_error_text, sizeof(lp_error_text), "%s: cannot reserve %zu bytes of shared memory: %s", what, bytes,
                     cudaGetErrorString(e));
            return -1;
        }
    }
    return 0;
}


// ---------------------------------------------------------------- the queries' own latent
// out[t, i] = x[t, off + i] / sqrt(mean_i x^2 + eps) * gain[i] for the `rank` columns from `off` of the float32
// projection: where queries go through a latent of their own, its RMS norm in front of the queries' map.
template <typename TOut>
__global__ void __launch_bounds__(256)
latent_query_norm_kernel(const float* __restrict__ proj, int ld, int off, int rank, const float* __restrict__ gain, float eps,
                         TOut* __restrict__ out) {
    __shared__ float scratch[32];
    lp_grid_release();
    lp_grid_wait();
    const float* x = proj + (long long)blockIdx.x * ld + off;
    float ss = 0.f;
    for (int i = threadIdx.x; i < rank; i += blockDim.x) ss = fmaf(x[i], x[i], ss);
    ss = lp_block_sum(ss, scratch);
    const float f = 1.0f / sqrtf(ss / (float)rank + eps);
    TOut* o = out + (long long)blockIdx.x * rank;
    for (int i = threadIdx.x; i < rank; i += blockDim.x) o[i] = lp_from_float<TOut>(x[i] * f * gain[i]);
}

}  // namespace

// proj: float32 [T, ld] with the queries at q_off ([H, dn + dr]) and the latent and shared key part at kv_off
// ([rank + dr]); pages: [num_pages, page_size, rank + dr]; q_out: float32 [T, H, dn + dr]. Optional bfloat16
// copies that lie together: latent_out [T, rank], shared_out [T, dr], q_half [T, H, q_half_hd] (heads padded with
// zeros from dn + dr to q_half_hd).
extern "C" int lp_latent_prepare(const float* proj, int ld, int q_off, int kv_off, const float* gain, float eps,
                                 const float* inv_freq, int rot, const int* positions, const int* seq_ids,
                                 const int* page_table, int pt_stride, float* q_out, void* pages, int kv_dtype, int T,
                                 int H, int dn, int dr, int rank, int page_size, void* latent_out, void* shared_out,
                                 void* q_half, int q_half_hd, const float* q_sep, int ldq, int interleaved,
                                 float magnitude, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (q_sep && ldq < H * (dn + dr)) LP_REFUSE("latent_prepare: query rows of %d for %d heads of %d", ldq, H, dn + dr);
    if (H <= 0 || dn < 0 || dr < 0 || rank <= 0 || dn + dr <= 0) LP_REFUSE("latent_prepare: %d heads of %d + %d over rank %d", H, dn, dr, rank);
    if (rot < 0 || (rot & 1) || rot > dr || rot > 256) LP_REFUSE("latent_prepare: rotary width %d of %d (even, at most 256)", rot, dr);
    if (rot > 0 && !inv_freq) LP_REFUSE("latent_prepare: rotation without frequencies");
    if (page_size <= 0) LP_REFUSE("latent_prepare: page size %d", page_size);
    if (q_half && q_half_hd < dn + dr) LP_REFUSE("latent_prepare: padded heads of %d for heads of %d", q_half_hd, dn + dr);
    if (q_off < 0 || kv_off < 0 || (!q_sep && q_off + H * (dn + dr) > ld) || kv_off + rank + dr > ld)
        LP_REFUSE("latent_prepare: slices at %d and %d do not fit rows of %d", q_off, kv_off, ld);
    const bool vec = ld % 4 == 0 && q_off % 4 == 0 && kv_off % 4 == 0 && dn % 4 == 0 && dr % 4 == 0 && rank % 4 == 0 && rot % 8 == 0 &&
                     (!q_sep || ldq % 4 == 0) && (!q_half || q_half_hd % 4 == 0) &&
                     (((uintptr_t)proj | (uintptr_t)gain | (uintptr_t)q_out | (uintptr_t)pages | (uintptr_t)latent_out | (uintptr_t)shared_out |
                       (uintptr_t)q_half | (uintptr_t)q_sep) & 15) == 0;
    if (!q_out && !q_half) LP_REFUSE("latent_prepare: nowhere to write the queries");
    const int shares = vec && T * (1 + (H + 7) / 8) <= 2 * lp_sm_count() ? 1 + (H + 7) / 8 : 1;
#define LP_LAUNCH_PREP(TKV)                                                                                       \
    lp_launch(vec ? latent_prepare_vec4_kernel<TKV> : latent_prepare_kernel<TKV>, dim3(T, shares), 256, 0, stream, proj, ld, q_off, kv_off, gain, eps, inv_freq, rot,    \
              positions, seq_ids, page_table, pt_stride, q_out, (TKV*)pages, H, dn, dr, rank, page_size,                   \
              (__nv_bfloat16*)latent_out, (__nv_bfloat16*)shared_out, (__nv_bfloat16*)q_half, q_half_hd, q_sep, ldq,    \
              interleaved, magnitude)
    if (kv_dtype == LP_F32) LP_LAUNCH_PREP(float);
    else if (kv_dtype == LP_BF16) LP_LAUNCH_PREP(__nv_bfloat16);
    else LP_REFUSE("latent_prepare: cache dtype code %d", kv_dtype);
#undef LP_LAUNCH_PREP
    return lp_check_launch("latent_prepare");
}

namespace {
size_t absorb_bytes(int dn) { return ((size_t)3 * TC_ROWS * (dn + 8) + (size_t)dn * (AB_COLS + 8)) * 2; }
// Whether the tensor-core kernel serves the map: 16-bit weights whose tiles can be read 16 bytes at a time.
bool absorb_on_tensor_cores(int w_dtype, int dn, int dr, int rank, const void* uk, const float* qa) {
    return w_dtype == LP_BF16 && dn > 0 && dn % 16 == 0 && rank % AB_COLS == 0 && dr % 2 == 0 && (uintptr_t)uk % 16 == 0 &&
           (uintptr_t)qa % 8 == 0 && absorb_bytes(dn) <= 200 * 1024;
}
}  // namespace

// What lp_latent_prepare and lp_latent_absorb do one after the other, in one launch, for a 16-bit cache and 16-bit weights; see there for
// the operands. Returns LP_NOT_SERVED for sizes and addresses that it does not take: those that lp_latent_prepare refuses or serves value by
// value are left to it, so that a cached row has the same bits whichever wrote it (a rank of up to 512, as the cache's readers take).
extern "C" int lp_latent_queries(const float* proj, int ld, int q_off, int kv_off, const float* gain, float eps, const float* inv_freq,
                                 int rot, const int* positions, const int* seq_ids, const int* page_table, int pt_stride, void* pages,
                                 int kv_dtype, int T, int H, int dn, int dr, int rank, int page_size, const float* q_sep, int ldq,
                                 int interleaved, float magnitude, const void* uk, int w_dtype, float* qa, cudaStream_t stream) {
    if (T <= 0) return 0;
    const float* q = q_sep ? q_sep : proj + q_off;
    if (!q_sep) ldq = ld;
    if (H <= 0 || H >= 65535 || page_size <= 0 || kv_dtype != LP_BF16 || rot < 0 || rot % 8 || rot > dr || rot > 256 || (rot > 0 && !inv_freq) || q_off < 0 ||
        kv_off < 0 || kv_off + rank + dr > ld || (q_sep ? 0 : q_off) + H * (dn + dr) > ldq || !absorb_on_tensor_cores(w_dtype, dn, dr, rank, uk, qa) ||
        ld % 4 || ldq % 4 || kv_off % 4 || dr % 4 || (((uintptr_t)q | (uintptr_t)proj | (uintptr_t)gain | (uintptr_t)pages) & 15) != 0)
        return LP_NOT_SERVED;
    const KeyRows k{proj + kv_off, ld, gain, eps, inv_freq, rot, interleaved, magnitude, positions, seq_ids, page_table, pt_stride, page_size,
                    (__nv_bfloat16*)pages};
    const size_t bytes = absorb_bytes(dn);
    if (grant_shared(latent_absorb_tc_kernel, bytes, "latent_queries")) return -1;
    lp_launch(latent_absorb_tc_kernel, dim3((T + TC_ROWS - 1) / TC_ROWS, H + 1, rank / AB_COLS), AB_WARPS * 32, bytes, stream, q, ldq,
              (const __nv_bfloat16*)uk, qa, T, H, dn, dr, rank, k);
    return lp_check_launch("latent_queries");
}

// q: float32 [T, H, dn + dr]; uk: [H * dn, rank]; qa: float32 [T, H, rank + dr].
extern "C" int lp_latent_absorb(const float* q, const void* uk, int w_dtype, float* qa, int T, int H, int dn, int dr,
                                int rank, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (H <= 0 || H > 65535 || dn < 0 || dr < 0 || rank <= 0) LP_REFUSE("latent_absorb: %d heads of %d + %d over rank %d", H, dn, dr, rank);
    // bfloat16 weights whose tiles can be read 16 bytes at a time go to the tensor cores
    if (absorb_on_tensor_cores(w_dtype, dn, dr, rank, uk, qa) && (dn + dr) % 4 == 0 && (uintptr_t)q % 16 == 0) {
        const size_t bytes = absorb_bytes(dn);
        if (grant_shared(latent_absorb_tc_kernel, bytes, "latent_absorb")) return -1;
        lp_launch(latent_absorb_tc_kernel, dim3((T + TC_ROWS - 1) / TC_ROWS, H, rank / AB_COLS), AB_WARPS * 32, bytes, stream, q,
                  H * (dn + dr), (const __nv_bfloat16*)uk, qa, T, H, dn, dr, rank, KeyRows{});
        return lp_check_launch("latent_absorb");
    }
    dim3 grid((T + TOK_TILE - 1) / TOK_TILE, H, (rank + 127) / 128);
    const size_t smem = (size_t)TOK_TILE * (dn > 0 ? dn : 1) * sizeof(float);
    if (w_dtype == LP_F32) {
        if (grant_shared(latent_absorb_kernel<float>, smem, "latent_absorb")) return -1;
        lp_launch(latent_absorb_kernel<float>, grid, 128, smem, stream, q, (const float*)uk, qa, T, H, dn, dr, rank);
    } else if (w_dtype == LP_BF16) {
        if (grant_shared(latent_absorb_kernel<__nv_bfloat16>, smem, "latent_absorb")) return -1;
        lp_launch(latent_absorb_kernel<__nv_bfloat16>, grid, 128, smem, stream, q, (const __nv_bfloat16*)uk, qa, T, H, dn, dr, rank);
    } else LP_REFUSE("latent_absorb: weight dtype code %d", w_dtype);
    return lp_check_launch("latent_absorb");
}

constexpr int ATTEND_RW = 4;

// How many (token, head) rows one CTA of lp_latent_attend takes, and how many keys a block holds.
extern "C" int lp_latent_attend_rows(int kv_dtype, int rank, int dr, int page_size) {
    return attend_on_tensor_cores(kv_dtype, rank, dr, page_size) ? TC_ROWS : WARPS * ATTEND_RW;
}
extern "C" int lp_latent_attend_keys(int kv_dtype, int rank, int dr, int page_size) {
    return attend_on_tensor_cores(kv_dtype, rank, dr, page_size) ? TC_KEYS : KEYS;
}

// qa: float32 [T, H, rank + dr]; part: float32 [T, H, shares, rank + 2] (unnormalised sums, maximum, sum of
// weights); q_start [B + 1], kv_len [B] (lengths after the step); max_new: most new tokens of a sequence.
extern "C" int lp_latent_attend(const float* qa, const void* pages, int kv_dtype, const int* page_table, int pt_stride,
                                const int* q_start, const int* kv_len, float* part, int B, int max_new, int H,
                                int rank, int dr, int page_size, long long num_pages, float scale, int shares, int window, int* status,
                                cudaStream_t stream) {
    if (B <= 0 || max_new <= 0) return 0;
    if (!status) LP_REFUSE("latent_attend: nowhere to report a wait that ran out%s", "");
    if (H <= 0 || rank <= 0 || dr < 0) LP_REFUSE("latent_attend: %d heads over rank %d + %d", H, rank, dr);
    if (rank > 512) LP_REFUSE("latent_attend: rank %d (supported: up to 512)", rank);
    if (page_size <= 0 || page_size % KEYS) LP_REFUSE("latent_attend: page size %d must be a multiple of %d", page_size, KEYS);
    if (shares <= 0 || shares > 65535 || B > 65535) LP_REFUSE("latent_attend: %d shares, %d sequences", shares, B);
    if (attend_on_tensor_cores(kv_dtype, rank, dr, page_size) && (uintptr_t)pages % 16 == 0 && (uintptr_t)qa % 16 == 0 &&
        (uintptr_t)part % 8 == 0) {
        const size_t bytes = tc_smem(rank + dr);
        CUtensorMap rows_map;
        if (make_map(&rows_map, pages, num_pages * page_size, rank + dr, rank + dr, TC_KEYS)) return -1;
        const dim3 tc_grid((unsigned)(((long long)max_new * H + TC_ROWS - 1) / TC_ROWS), B, shares);
#define LP_LAUNCH_TC(NT)                                                                                                     \
    do {                                                                                                                     \
        if (grant_shared(latent_attend_tc_kernel<NT>, bytes, "latent_attend")) return -1;                                    \
        lp_launch(latent_attend_tc_kernel<NT>, tc_grid, WARPS * 32, bytes, stream, rows_map, qa, page_table, pt_stride,      \
                  q_start, kv_len, part, H, dr, page_size, scale, shares, window, status);                    \
    } while (0)
        if (rank == 64) LP_LAUNCH_TC(1);
        else if (rank == 128) LP_LAUNCH_TC(2);
        else if (rank == 256) LP_LAUNCH_TC(4);
        else LP_LAUNCH_TC(8);
#undef LP_LAUNCH_TC
        return lp_check_launch("latent_attend");
    }
    constexpr int ROWS = WARPS * ATTEND_RW;
    const int Dk = rank + dr;
    const size_t smem = ((size_t)ROWS * Dk + (size_t)KEYS * (Dk + 4)) * sizeof(float);
    if (smem > 227 * 1024) LP_REFUSE("latent_attend: rows of %d values need %zu bytes of shared memory", Dk, smem);
    dim3 grid((unsigned)(((long long)max_new * H + ROWS - 1) / ROWS), B, shares);
#define LP_LAUNCH_ATTEND(TKV, NC)                                                                                    \
    do {                                                                                                             \
        if (grant_shared(latent_attend_kernel<TKV, ATTEND_RW, NC>, smem, "latent_attend")) return -1;                \
        lp_launch(latent_attend_kernel<TKV, ATTEND_RW, NC>, grid, WARPS * 32, smem, stream, qa, (const TKV*)pages,   \
                  page_table, pt_stride, q_start, kv_len, part, H, rank, dr, page_size, scale, shares, window);      \
    } while (0)
#define LP_PICK_NC(TKV)                                  \
    do {                                                 \
        if (rank <= 32) LP_LAUNCH_ATTEND(TKV, 1);        \
        else if (rank <= 64) LP_LAUNCH_ATTEND(TKV, 2);   \
        else if (rank <= 128) LP_LAUNCH_ATTEND(TKV, 4);  \
        else if (rank <= 256) LP_LAUNCH_ATTEND(TKV, 8);  \
        else LP_LAUNCH_ATTEND(TKV, 16);                  \
    } while (0)
    if (kv_dtype == LP_F32) LP_PICK_NC(float);
    else if (kv_dtype == LP_BF16) LP_PICK_NC(__nv_bfloat16);
    else LP_REFUSE("latent_attend: cache dtype code %d", kv_dtype);
#undef LP_PICK_NC
#undef LP_LAUNCH_ATTEND
    return lp_check_launch("latent_attend");
}

// part: float32 [rows, shares, rank + 2] as lp_latent_attend leaves it; out: float32 [rows, 1, rank + 2], one share.
extern "C" int lp_latent_merge(const float* part, int shares, float* out, int rows, int rank, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (shares <= 0 || rank <= 0) LP_REFUSE("latent_merge: %d shares of rank %d", shares, rank);
    lp_launch(latent_merge_kernel, rows, 128, (size_t)shares * sizeof(float), stream, part, shares, out, rank);
    return lp_check_launch("latent_merge");
}

// part: as lp_latent_attend leaves it; uv: [H * dv, rank]; gate: float32 [T, ldg] with one value per head
// (or null); out: [T, H * dv].
// zero (optional): a float32 buffer cleared on the side. Steps of at most ROWS_FORM_TOKENS tokens take the form with one
// CTA per (token, head) row.
constexpr int ROWS_FORM_TOKENS = 64;
extern "C" int lp_latent_expand(const float* part, int shares, const void* uv, int w_dtype, const float* gate, int ldg,
                                void* out, int out_dtype, int T, int H, int rank, int dv, float* zero, long long zero_count,
                                cudaStream_t stream) {
    if (T <= 0) return 0;
    if (H <= 0 || H > 65535 || rank <= 0 || dv <= 0 || shares <= 0) LP_REFUSE("latent_expand: %d heads, rank %d, values of %d, %d shares", H, rank, dv, shares);
    const size_t tc_bytes = ((size_t)3 * TC_ROWS + EX_FEATURES) * (rank + 8) * 2 + (size_t)TC_ROWS * shares * sizeof(float);
    if (w_dtype == LP_BF16 && rank % 64 == 0 && (uintptr_t)uv % 16 == 0 && (uintptr_t)part % 8 == 0 && tc_bytes <= 200 * 1024 &&
        (out_dtype == LP_BF16 || out_dtype == LP_F32)) {
        const dim3 tc_grid((T + TC_ROWS - 1) / TC_ROWS, H, (dv + EX_FEATURES - 1) / EX_FEATURES);
#define LP_LAUNCH_TC(TOut)                                                                                           \
    do {                                                                                                             \
        auto kernel = T > 1 && tc_grid.z % 4 == 0 ? latent_expand_tc_kernel<TOut, 4>                                          \
                      : T > 1 && tc_grid.z % 2 == 0 ? latent_expand_tc_kernel<TOut, 2>                               \
                                                    : latent_expand_tc_kernel<TOut, 1>;                              \
        if (grant_shared(kernel, tc_bytes, "latent_expand")) return -1;                                              \
        lp_launch(kernel, tc_grid, EX_WARPS * 32, tc_bytes, stream, part, shares, (const __nv_bfloat16*)uv, gate,    \
                  ldg, (TOut*)out, T, H, rank, dv, zero, zero_count);                                                \
    } while (0)
        if (out_dtype == LP_BF16) LP_LAUNCH_TC(__nv_bfloat16);
        else LP_LAUNCH_TC(float);
#undef LP_LAUNCH_TC
        return lp_check_launch("latent_expand");
    }
    if (T <= ROWS_FORM_TOKENS) {
        const size_t bytes = (size_t)(rank + shares) * sizeof(float);
#define LP_LAUNCH_ROWS(TW, TOut)                                                                                     \
    do {                                                                                                             \
        if (grant_shared(latent_expand_rows_kernel<TW, TOut>, bytes, "latent_expand")) return -1;                    \
        lp_launch(latent_expand_rows_kernel<TW, TOut>, T * H, 256, bytes, stream, part, shares, (const TW*)uv, gate,  \
                  ldg, (TOut*)out, H, rank, dv, zero, zero_count);                                                   \
    } while (0)
        if (w_dtype == LP_F32 && out_dtype == LP_F32) LP_LAUNCH_ROWS(float, float);
        else if (w_dtype == LP_BF16 && out_dtype == LP_BF16) LP_LAUNCH_ROWS(__nv_bfloat16, __nv_bfloat16);
        else if (w_dtype == LP_BF16 && out_dtype == LP_F32) LP_LAUNCH_ROWS(__nv_bfloat16, float);
        else if (w_dtype == LP_F32 && out_dtype == LP_BF16) LP_LAUNCH_ROWS(float, __nv_bfloat16);
        else LP_REFUSE("latent_expand: dtype codes w=%d out=%d", w_dtype, out_dtype);
#undef LP_LAUNCH_ROWS
        return lp_check_launch("latent_expand");
    }
    // few tokens: the value columns of a head are shared out over CTAs as well (each merges the shares itself)
    const int tiles = (T + TOK_TILE - 1) / TOK_TILE;
    int vparts = 1;
    if (tiles * H < 2 * lp_sm_count()) vparts = min((dv + 15) / 16, max(1, 2 * lp_sm_count() / (tiles * H)));
    dim3 grid(tiles, H, vparts);
    const size_t smem = (size_t)TOK_TILE * (rank + shares) * sizeof(float);
#define LP_LAUNCH_EXPAND(TW, TOut)                                                                                \
    do {                                                                                                          \
        if (grant_shared(latent_expand_kernel<TW, TOut>, smem, "latent_expand")) return -1;                       \
        lp_launch(latent_expand_kernel<TW, TOut>, grid, 128, smem, stream, part, shares, (const TW*)uv, gate, ldg, \
                  (TOut*)out, T, H, rank, dv, zero, zero_count);                                                  \
    } while (0)
    if (w_dtype == LP_F32 && out_dtype == LP_F32) LP_LAUNCH_EXPAND(float, float);
    else if (w_dtype == LP_BF16 && out_dtype == LP_BF16) LP_LAUNCH_EXPAND(__nv_bfloat16, __nv_bfloat16);
    else if (w_dtype == LP_BF16 && out_dtype == LP_F32) LP_LAUNCH_EXPAND(__nv_bfloat16, float);
    else if (w_dtype == LP_F32 && out_dtype == LP_BF16) LP_LAUNCH_EXPAND(float, __nv_bfloat16);
    else LP_REFUSE("latent_expand: dtype codes w=%d out=%d", w_dtype, out_dtype);
#undef LP_LAUNCH_EXPAND
    return lp_check_launch("latent_expand");
}

// kv: bfloat16 [T, H * dn + H * dv] (every head's unrotated keys, then every head's values); shared_part: bfloat16
// [T, dr]; pages: bfloat16 [num_pages, 2, H, page_size, hd]; table: [B, pt_stride]; kv_len [B]: the sequences'
// lengths, all of whose positions are in this step.
extern "C" int lp_latent_heads_to_pages(const void* kv, const void* shared_part, const int* positions, const int* seq_ids,
                                        const int* table, int pt_stride, const int* kv_len, void* pages, int T, int H,
                                        int dn, int dr, int dv, int page_size, int hd, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (H <= 0 || dn < 0 || dr < 0 || dv <= 0 || hd < dn + dr || dv > hd)
        LP_REFUSE("latent_heads_to_pages: %d heads of %d + %d in %d, values of %d", H, dn, dr, hd, dv);
    if (page_size <= 0) LP_REFUSE("latent_heads_to_pages: page size %d", page_size);
    const bool vec = dn % 8 == 0 && dr % 8 == 0 && dv % 8 == 0 && hd % 8 == 0 &&
                     (((uintptr_t)kv | (uintptr_t)shared_part | (uintptr_t)pages) & 15) == 0;
    lp_launch(vec ? latent_heads_to_pages_vec8_kernel : latent_heads_to_pages_kernel, T, 256, 0, stream, (const __nv_bfloat16*)kv, (const __nv_bfloat16*)shared_part,
              positions, seq_ids, table, pt_stride, kv_len, (__nv_bfloat16*)pages, H, dn, dr, dv, page_size, hd);
    return lp_check_launch("latent_heads_to_pages");
}

extern "C" int lp_latent_gate_heads(const void* heads, const float* gate, int ldg, void* out, int T, int H, int hd, int dv,
                                    float* zero, long long zero_count, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (H <= 0 || dv <= 0 || dv > hd) LP_REFUSE("latent_gate_heads: %d heads of %d, values of %d", H, hd, dv);
    const long long n = (long long)T * H * dv;
    if (dv % 8 == 0 && dv <= 256 && hd % 8 == 0 && (((uintptr_t)heads | (uintptr_t)out) & 15) == 0 && (long long)T * H <= 0x7fffffff) {
        long long wide = (n / 8 + 255) / 256;
        if (wide > 148 * 16) wide = 148 * 16;
        lp_launch(latent_gate_heads_vec8_kernel, (unsigned)wide, 256, 0, stream, (const __nv_bfloat16*)heads, gate, ldg,
                  (__nv_bfloat16*)out, T * H, H, hd, dv, zero, zero_count);
        return lp_check_launch("latent_gate_heads");
    }
    long long blocks = (n + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    lp_launch(latent_gate_heads_kernel, (unsigned)blocks, 256, 0, stream, (const __nv_bfloat16*)heads, gate, ldg,
              (__nv_bfloat16*)out, T, H, hd, dv, zero, zero_count);
    return lp_check_launch("latent_gate_heads");
}

// proj: float32 [T, ld]; the latent's `rank` columns start at `off`; gain: float32 [rank]; out: [T, rank].
extern "C" int lp_latent_query_norm(const float* proj, int ld, int off, int rank, const float* gain, float eps, void* out,
                                    int dtype, int T, cudaStream_t stream) {
    if (T <= 0) return 0;
    if (rank <= 0 || off < 0 || off + rank > ld) LP_REFUSE("latent_query_norm: %d columns at %d of rows of %d", rank, off, ld);
    if (dtype == LP_F32) lp_launch(latent_query_norm_kernel<float>, T, 256, 0, stream, proj, ld, off, rank, gain, eps, (float*)out);
    else if (dtype == LP_BF16) lp_launch(latent_query_norm_kernel<__nv_bfloat16>, T, 256, 0, stream, proj, ld, off, rank, gain, eps, (__nv_bfloat16*)out);
    else LP_REFUSE("latent_query_norm: dtype code %d", dtype);
    return lp_check_launch("latent_query_norm");
}
