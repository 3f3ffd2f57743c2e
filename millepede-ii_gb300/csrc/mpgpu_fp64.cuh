// mpgpu_fp64.cuh -- FP64 helpers of the factorisations' pivot chains.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

// Reciprocal by Newton's iteration from an FP32 seed (relative error below
// 2^-21, squared twice: what is left is the last step's rounding, half an ulp;
// equal to 1 / d in all of 2^30 random d),
// d within 2^+-120; the conversions in integers, as a conversion costs a slot of
// the FP64 pipe.
__device__ __forceinline__ double newton_rcp(double d) {
    const uint32_t hi = (uint32_t)__double2hiint(d), lo = (uint32_t)__double2loint(d);
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float((hi - (896u << 20)) << 3 | lo >> 29)));
    const uint32_t f = __float_as_uint(y);
    double z = __hiloint2double((int)((f >> 3) + (896u << 20)), (int)(f << 29));
    z = fma(z, fma(-d, z, 1.0), z);
    return fma(z, fma(-d, z, 1.0), z);
}
