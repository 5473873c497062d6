// Compares the plain walk's rounded 1 / sqrt (tvg_inv_sqrt.cuh) with the two
// rounded operations for every FP32 significand and exponent parity, at the
// smallest, the middle and the largest exponents of its range. Prints the number
// of differences.
#include <cstdio>

#include "../tandav_b200/csrc/tvg_inv_sqrt.cuh"

__global__ void k_check(unsigned long long *bad)
{
	const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;      // 2^24: significand and parity
	const int e0[3] = { 67, 127, 185 };                            // biased: 2^-60, 1, 2^58
	for (int k = 0; k < 3; k++) {
		const float x = __uint_as_float(((unsigned) e0[k] << 23) + i);
		if (inv_sqrt(x) != __frcp_rn(__fsqrt_rn(x))) atomicAdd(bad, 1ull);
	}
}

int main()
{
	unsigned long long *d = nullptr, h = 1;
	if (cudaMalloc(&d, 8) != cudaSuccess || cudaMemset(d, 0, 8) != cudaSuccess) return 1;
	k_check<<<(1 << 24) / 256, 256>>>(d);
	if (cudaMemcpy(&h, d, 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
	printf("%llu\n", h);
	cudaFree(d);
	return 0;
}
