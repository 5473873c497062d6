// tvg_inv_sqrt.cuh -- the plain walk's rounded 1 / sqrt(r2) in FP32.
#pragma once

// 1 / sqrt(r2) as the reference rounds it, both operations to nearest, without
// the branches of the general operations, for r2 in [2^-60, 2^60]. The root: a
// Goldschmidt step from the approximate reciprocal root with Markstein's
// correction (IBM J. Res. Dev. 34, 1990). The reciprocal: two Newton steps from
// the same approximation, the first rounded up so that the last one never
// starts below a result that lies next to a tie. Equal to the two rounded
// operations for every significand and exponent parity; powers of four only
// scale it (tests/inv_sqrt_check.cu compares all of them).
__device__ __forceinline__ float inv_sqrt(float r2)
{
	float y;
	asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(r2));
	const float g = __fmul_rn(r2, y), h = __fmul_rn(0.5f, y);
	const float s = __fmaf_rn(__fmaf_rn(-g, g, r2), h, g);
	const float y1 = __fmaf_ru(y, __fmaf_rn(-s, y, 1.0f), y);
	return __fmaf_rn(__fmaf_rn(-s, y1, 1.0f), y1, y1);
}
