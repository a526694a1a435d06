// Snapshot storage shared by the step kernels, and the flags of a step.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include "engine.h"

namespace fwi2d {

enum StepFlags { F_STORE = 1, F_EXTRACT = 2, F_AMAX = 4, F_GRAD = 8 };

// ---------------------------------------------------------------------------
// Snapshot storage: fp32, or bf16/fp16 scaled by a per-snapshot power of two
// chosen from the snapshot's max |u| (so |u*scale| < 2^14).
// ---------------------------------------------------------------------------
__device__ __forceinline__ float snap_scale(const unsigned *amax, int slot)
{
    float m = __uint_as_float(__ldcg(amax + slot));   // earlier steps of the same launch may have set it
    if (!(m > 0.f)) return 1.f;
    int e = ilogbf(m) + 1;                 // m < 2^e
    return ldexpf(1.f, min(14 - e, 126));   // a field below 2^-112 must not push the factor to infinity
}

__device__ __forceinline__ void snap_store(void *base, long long idx, int prec, float v, float scale)
{
    if (prec == SNAP_FP32) ((float *)base)[idx] = v;
    else if (prec == SNAP_BF16) ((__nv_bfloat16 *)base)[idx] = __float2bfloat16_rn(v * scale);
    else ((__half *)base)[idx] = __float2half_rn(v * scale);
}

__device__ __forceinline__ float snap_load(const void *base, long long idx, int prec, float inv)
{
    if (prec == SNAP_FP32) return ((const float *)base)[idx];
    if (prec == SNAP_BF16) return __bfloat162float(((const __nv_bfloat16 *)base)[idx]) * inv;
    return __half2float(((const __half *)base)[idx]) * inv;
}

// pair of samples at an even index
__device__ __forceinline__ float2 ld2(const float *base, int idx)
{
    return *reinterpret_cast<const float2 *>(base + idx);
}

// Two-sample snapshot loads for the lean path (even index).
__device__ __forceinline__ float2 snap_load2(const void *base, long long idx, int prec, float inv)
{
    if (prec == SNAP_FP32) return *reinterpret_cast<const float2 *>((const float *)base + idx);
    if (prec == SNAP_BF16) {
        const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>((const __nv_bfloat16 *)base + idx));
        return make_float2(v.x * inv, v.y * inv);
    }
    const float2 v = __half22float2(*reinterpret_cast<const __half2 *>((const __half *)base + idx));
    return make_float2(v.x * inv, v.y * inv);
}

}  // namespace fwi2d
