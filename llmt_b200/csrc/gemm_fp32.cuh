// What the two fp32 GEMM kernels share: reads of a cluster's shared memory and the finishing of one value.
#pragma once

#include <cuda_bf16.h>

#include "common.h"

namespace llmt_b200 {

__device__ __forceinline__ float4 ld_dsmem16(uint32_t addr, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ float ld_dsmem4(uint32_t addr, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}

__device__ __forceinline__ float f32_finish(const Fp32GemmParams& p, float acc, const float* dst, int64_t col) {
    float v = p.alpha * acc;
    if (p.beta != 0.0f) v += p.beta * *dst;
    if (p.epi_flags & kEpiBias)
        v += p.bias_is_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p.bias)[col]) : static_cast<const float*>(p.bias)[col];
    if (p.epi_flags & kEpiGelu) v = gelu_tanh_precise(v);
    return v;
}

}  // namespace llmt_b200
