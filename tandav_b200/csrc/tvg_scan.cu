// tvg_scan.cu -- device-wide exclusive prefix sum of int32 (reduce, apply; for
// many blocks a scan of their sums between), 4096 items per block, warp-shuffle
// block scans. No inter-block waits: every phase is its own launch.
#include "tvg_internal.cuh"

#define SCAN_THREADS 512
#define SCAN_IPT 8
#define SCAN_TILE (SCAN_THREADS * SCAN_IPT)

__device__ __forceinline__ int32_t warp_incl_scan(int32_t v)
{
	const int lane = threadIdx.x & 31;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		int32_t u = __shfl_up_sync(0xFFFFFFFFu, v, o);
		if (lane >= o) v += u;
	}
	return v;
}

// exclusive scan of one value per thread across the block; returns the block total
__device__ __forceinline__ int32_t block_excl_scan(int32_t v, int32_t *excl, int32_t *s_warp)
{
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
	int32_t inc = warp_incl_scan(v);
	if (lane == 31) s_warp[w] = inc;
	__syncthreads();
	if (w == 0) {
		int32_t t = lane < nw ? s_warp[lane] : 0;
		int32_t ti = warp_incl_scan(t);
		if (lane < nw) s_warp[lane] = ti - t;
		if (lane == nw - 1) s_warp[32] = ti;
	}
	__syncthreads();
	*excl = inc - v + s_warp[w];
	int32_t total = s_warp[32];
	__syncthreads();
	return total;
}

// the eight items from base on, zero past n
__device__ __forceinline__ void load_items(const int32_t *__restrict__ in, int64_t n, int64_t base, int32_t (&v)[SCAN_IPT])
{
	if (((uintptr_t) in & 15) == 0 && base + SCAN_IPT <= n) {
		const int4 a = *(const int4 *) (in + base), b = *(const int4 *) (in + base + 4);
		v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
		v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
	} else {
#pragma unroll
		for (int k = 0; k < SCAN_IPT; k++) v[k] = base + k < n ? in[base + k] : 0;
	}
}

__global__ void __launch_bounds__(SCAN_THREADS)
k_scan_reduce(const int32_t *__restrict__ in, int64_t n, int32_t *__restrict__ sums)
{
	__shared__ int32_t s_warp[SCAN_THREADS / 32];
	int32_t v[SCAN_IPT], acc = 0;
	load_items(in, n, (int64_t) blockIdx.x * SCAN_TILE + (int64_t) threadIdx.x * SCAN_IPT, v);
#pragma unroll
	for (int k = 0; k < SCAN_IPT; k++) acc += v[k];
	acc = __reduce_add_sync(0xFFFFFFFFu, acc);
	if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = acc;
	__syncthreads();
	if (threadIdx.x == 0) {
		int32_t t = 0;
#pragma unroll
		for (int k = 0; k < SCAN_THREADS / 32; k++) t += s_warp[k];
		sums[blockIdx.x] = t;
	}
}

// What precedes a block: nothing or the scanned offset offs[b] (OFFSETS), the
// sum of offs[0 .. b) (SUMS), or of the items of the tiles before it (ITEMS; in
// and out are then different arrays).
enum { SCAN_OFFSETS, SCAN_SUMS, SCAN_ITEMS };

template <int BEFORE>
__global__ void __launch_bounds__(SCAN_THREADS)
k_scan_apply(const int32_t *in, int32_t *out, int64_t n, const int32_t *__restrict__ offs, int64_t *total_out)
{
	__shared__ int32_t s_warp[33], s_before[SCAN_THREADS / 32];
	const int64_t base = (int64_t) blockIdx.x * SCAN_TILE + (int64_t) threadIdx.x * SCAN_IPT;
	int32_t v[SCAN_IPT];
	int32_t acc = 0, before = 0;
	load_items(in, n, base, v);
#pragma unroll
	for (int k = 0; k < SCAN_IPT; k++) acc += v[k];
	if (BEFORE == SCAN_SUMS)
		for (unsigned b = threadIdx.x; b < blockIdx.x; b += SCAN_THREADS) before += offs[b];
	if (BEFORE == SCAN_ITEMS) {
#pragma unroll 4
		for (unsigned b = 0; b < blockIdx.x; b++) {
			int32_t u[SCAN_IPT];
			load_items(in, n, (int64_t) b * SCAN_TILE + (int64_t) threadIdx.x * SCAN_IPT, u);
#pragma unroll
			for (int k = 0; k < SCAN_IPT; k++) before += u[k];
		}
	}
	if (BEFORE != SCAN_OFFSETS) {
		before = __reduce_add_sync(0xFFFFFFFFu, before);
		if ((threadIdx.x & 31) == 0) s_before[threadIdx.x >> 5] = before;
	}
	int32_t ex;
	block_excl_scan(acc, &ex, s_warp);
	int32_t run = ex;
	if (BEFORE == SCAN_OFFSETS) {
		run += offs ? offs[blockIdx.x] : 0;
	} else {
#pragma unroll
		for (int k = 0; k < SCAN_THREADS / 32; k++) run += s_before[k];
	}
	if (((uintptr_t) out & 15) == 0 && base + SCAN_IPT <= n) {
		int32_t o[SCAN_IPT];
#pragma unroll
		for (int k = 0; k < SCAN_IPT; k++) {
			o[k] = run;
			run += v[k];
		}
		*(int4 *) (out + base) = make_int4(o[0], o[1], o[2], o[3]);
		*(int4 *) (out + base + 4) = make_int4(o[4], o[5], o[6], o[7]);
	} else {
#pragma unroll
		for (int k = 0; k < SCAN_IPT; k++) {
			if (base + k < n) out[base + k] = run;
			run += v[k];
		}
	}
	// the thread holding the last element: the inclusive sum of everything
	if (total_out && base <= n - 1 && n - 1 < base + SCAN_IPT) *total_out = run;
}

// A scan of few items is as long as its launches. Up to SCAN_FEW tiles every block
// adds up the tiles before its own again (one launch, where in and out differ), up
// to SCAN_MANY the sums before its own (two); beyond, the sums are scanned by
// launches of their own (`tmp` must hold the block sums of every level).
// With three launches for everything past one tile the build of 3001 particles
// took 0.155 ms, so 0.130; of 32,768 0.150 / 0.125; of 16.7M, where loads and stores
// of four items count, 3.03 / 2.77.
#define SCAN_FEW 16
#define SCAN_MANY 2048
static int scan_rec(tvg_context *ctx, const int32_t *in, int32_t *out, int64_t n, int32_t *tmp,
                    size_t tmp_elems, int64_t *total_dev)
{
	const int64_t nb = (n + SCAN_TILE - 1) / SCAN_TILE;
	cudaStream_t s = ctx->stream;
	if (nb <= 1 || (nb <= SCAN_FEW && in != out)) {
		k_scan_apply<SCAN_ITEMS><<<TVG_CNT(ctx, (unsigned) nb), SCAN_THREADS, 0, s>>>(in, out, n, nullptr, total_dev);
		TVG_CUDA(ctx, cudaGetLastError());
		return TVG_OK;
	}
	if ((size_t) (2 * nb) > tmp_elems)
		return tvg_fail(ctx, TVG_E_NOMEM, "scan scratch too small (%lld blocks)", (long long) nb);
	int32_t *sums = tmp, *offs = tmp + nb;
	k_scan_reduce<<<TVG_CNT(ctx, (unsigned) nb), SCAN_THREADS, 0, s>>>(in, n, sums);
	TVG_CUDA(ctx, cudaGetLastError());
	if (nb <= SCAN_MANY) {
		k_scan_apply<SCAN_SUMS><<<TVG_CNT(ctx, (unsigned) nb), SCAN_THREADS, 0, s>>>(in, out, n, sums, total_dev);
	} else {
		TVG_CHECK(scan_rec(ctx, sums, offs, nb, tmp + 2 * nb, tmp_elems - 2 * nb, nullptr));
		k_scan_apply<SCAN_OFFSETS><<<TVG_CNT(ctx, (unsigned) nb), SCAN_THREADS, 0, s>>>(in, out, n, offs, total_dev);
	}
	TVG_CUDA(ctx, cudaGetLastError());
	return TVG_OK;
}

// out[i] = sum(in[0..i)); *total (if not NULL) receives the full sum, read
// back synchronously. in and out may alias.
int tvg_device_scan_i32(tvg_context *ctx, const int32_t *in, int32_t *out, int64_t n,
                        int64_t *total)
{
	if (n <= 0) {
		if (total) *total = 0;
		return TVG_OK;
	}
	int32_t last_in = 0;
	if (total)
		TVG_CUDA(ctx, cudaMemcpyAsync(&last_in, in + n - 1, 4, cudaMemcpyDeviceToHost, ctx->stream));
	TVG_CHECK(scan_rec(ctx, in, out, n, (int32_t *) ctx->scan_tmp, ctx->scan_tmp_bytes / 4, nullptr));
	if (total) {
		int32_t last_out = 0;
		TVG_CUDA(ctx, cudaMemcpyAsync(&last_out, out + n - 1, 4, cudaMemcpyDeviceToHost, ctx->stream));
		TVG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
		*total = (int64_t) last_out + last_in;
	}
	return TVG_OK;
}

// the total stays on the device (int64 at total_dev); no synchronisation
int tvg_device_scan_i32_dev(tvg_context *ctx, const int32_t *in, int32_t *out, int64_t n,
                            int64_t *total_dev)
{
	if (n <= 0) {
		TVG_CUDA(ctx, cudaMemsetAsync(total_dev, 0, 8, ctx->stream));
		return TVG_OK;
	}
	return scan_rec(ctx, in, out, n, (int32_t *) ctx->scan_tmp, ctx->scan_tmp_bytes / 4, total_dev);
}
