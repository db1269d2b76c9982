// Products of a float32 operand with a bfloat16 one on the tensor cores (mma.sync m16n8k16) without rounding the former: it
// enters as the sum of three bfloat16 numbers, 3 x 8 bits of mantissa, and every product of parts is exact in float32.
#pragma once

#include "common.cuh"

namespace {

__device__ __forceinline__ uint32_t smem_at(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldmatrix4(uint32_t addr, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t addr, uint32_t* r) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// x = part[0] + part[1] + part[2] to 24 bits; an infinity or a NaN stays in the first part alone
__device__ __forceinline__ void three_parts(float x, __nv_bfloat16* part) {
    part[0] = __float2bfloat16_rn(x);
    const float head = __bfloat162float(part[0]);
    const bool finite = fabsf(head) < INFINITY;
    const float rest = finite ? x - head : 0.f;
    part[1] = __float2bfloat16_rn(rest);
    part[2] = __float2bfloat16_rn(rest - __bfloat162float(part[1]));
}

}  // namespace
