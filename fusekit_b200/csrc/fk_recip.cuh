// 1 / x, x from 1 to below 2^126, in three instructions without a branch: an approximation and one Newton step in fused multiply-adds (P. Markstein, IBM J. Res. Dev. 34,
// 1990).  The bits of a division for every such float on this hardware: tests/test_gpu_reciprocal.py looks at all of them.
#pragma once
#define FK_RECIP_END 0x1p126f

__device__ __forceinline__ float recip_from_one(float x) {
    float r; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return fmaf(r, fmaf(-x, r, 1.0f), r);
}
