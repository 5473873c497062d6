// tvg_domain.cu -- set_computational_domain (src/domain.c:732-847): the cube
// the keys and node sizes refer to.
//
// Periodic: origin 0, size the box. Isolated: the centre is the median of
// each coordinate (find_domain_center, domain.c:763-801), the size 2.001
// times the largest |x - centre| over all particles and axes, in double
// (find_largest_particle_distance, :805-835), and origin = centre - size / 2.
//
// Median (select.c:95-107) is Select(n >> 1, n, data), the Numerical Recipes
// selection written for arrays indexed from 1 (l = 1, ir = n - 1) and run on
// an array indexed from 0: it returns the (n >> 1)-th smallest of
// data[1 .. n-1] (the first particle in the current order takes no part),
// and data[0] for n = 1. Here that order statistic is found exactly by a
// radix select over the coordinates mapped to ordered unsigned integers: one
// histogram pass per byte, most significant first, each keeping the bucket
// that holds the wanted rank. The centre is kept in Float, as the reference
// keeps it. The three axes go together, and the last block of a pass picks the
// buckets on the device, so a pass is one launch and the host waits once, for
// the result (with a launch and a wait per byte and axis: 0.30 ms for 200,000
// particles in FP32; so: 0.05 ms).
// Roofline: HBM bound, one read of the positions per byte of the Float (4 or 8
// passes) plus one for the distance.
#include <stddef.h>

#include "tvg_internal.cuh"

namespace {

__device__ __forceinline__ uint32_t ordered(float v)
{
	const uint32_t u = __float_as_uint(v);
	return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ uint64_t ordered(double v)
{
	const uint64_t u = (uint64_t) __double_as_longlong(v);
	return (u & 0x8000000000000000ull) ? ~u : (u | 0x8000000000000000ull);
}

template <typename F> struct Bits;
template <> struct Bits<float> { typedef uint32_t U; };
template <> struct Bits<double> { typedef uint64_t U; };

__device__ __forceinline__ float unordered(uint32_t u)
{
	return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

__device__ __forceinline__ double unordered(uint64_t u)
{
	return __longlong_as_double((long long) ((u & 0x8000000000000000ull) ? (u & 0x7FFFFFFFFFFFFFFFull) : ~u));
}

// selection state on the device; zero but for the ranks at the start
struct DomainState {
	uint32_t hist[2][3][256];      // byte counts per axis, of the even and the odd passes
	uint64_t prefix[3];            // the bytes chosen so far (ordered bits)
	uint64_t rank[3];              // 0-based rank among the values with that prefix
	uint32_t done;                 // blocks that have finished the pass
	uint32_t lost;                 // the rank fell outside the counts
	unsigned long long max_bits;   // largest |x - centre|, as bits
	double center[3];
};

#define DS_THREADS 256
// Few particles a thread, loaded together: a pass is as long as one thread's chain.
// 400,000 particles in FP64, whole search with 16 one by one / 8 / 4: 165 / 95 / 94
// us (200,000 in FP32: 75 / 64 / 54; 4M in FP64 with one block a SM 437, two 264,
// four 203).
#define DS_IPT 4
#define DS_BLOCKS 4

// One byte of the three selections: counts the byte at `shift` of the ordered
// values of particles 1 .. n-1 that have the prefix; the last block picks the
// bucket with the wanted rank (warp per axis) and clears the other histogram.
template <typename F>
__global__ void __launch_bounds__(DS_THREADS)
k_select(int64_t n, const F *__restrict__ x, const F *__restrict__ y, const F *__restrict__ z, int shift, int pass,
         DomainState *st)
{
	typedef typename Bits<F>::U U;
	__shared__ uint32_t h[3][256];
	__shared__ bool s_last;
	for (int b = threadIdx.x; b < 768; b += DS_THREADS) (&h[0][0])[b] = 0;
	__syncthreads();
	const U mask = pass == 0 ? (U) 0 : (U) ~(U) 0 << (shift + 8);
	const F *X[3] = { x, y, z };
	U prefix[3];
#pragma unroll
	for (int d = 0; d < 3; d++) prefix[d] = (U) st->prefix[d];
	const unsigned lane_bit = 1u << (threadIdx.x & 31);
	for (int64_t base = 1 + blockIdx.x * (int64_t) (DS_IPT * DS_THREADS); base < n;
	     base += (int64_t) gridDim.x * (DS_IPT * DS_THREADS)) {
		F v[3][DS_IPT];
#pragma unroll
		for (int r = 0; r < DS_IPT; r++) {
			const int64_t i = base + r * DS_THREADS + threadIdx.x;
#pragma unroll
			for (int d = 0; d < 3; d++) v[d][r] = i < n ? X[d][i] : (F) 0;
		}
#pragma unroll
		for (int r = 0; r < DS_IPT; r++) {
			const bool have = base + r * DS_THREADS + threadIdx.x < n;
#pragma unroll
			for (int d = 0; d < 3; d++) {
				const U u = ordered(v[d][r]);
				const bool in = have && (u & mask) == prefix[d];
				const unsigned m = __ballot_sync(0xFFFFFFFFu, in);
				if (m == 0) continue;
				// the lanes with the first lane's byte count once, together:
				// the top bytes are nearly all the same
				const uint32_t byte = (uint32_t) (u >> shift) & 0xFF;
				const int first = __ffs(m) - 1;
				const uint32_t lead = __shfl_sync(0xFFFFFFFFu, byte, first);
				const unsigned same = __ballot_sync(0xFFFFFFFFu, in && byte == lead);
				if (lane_bit == 1u << first) atomicAdd(&h[d][lead], (uint32_t) __popc(same));
				else if (in && byte != lead) atomicAdd(&h[d][byte], 1u);
			}
		}
	}
	__syncthreads();
	uint32_t *g = &st->hist[pass & 1][0][0];
	for (int b = threadIdx.x; b < 768; b += DS_THREADS)
		if ((&h[0][0])[b]) atomicAdd(&g[b], (&h[0][0])[b]);
	__threadfence();
	__syncthreads();
	if (threadIdx.x == 0) s_last = atomicAdd(&st->done, 1u) == gridDim.x - 1;
	__syncthreads();
	if (!s_last) return;
	__threadfence();
	for (int b = threadIdx.x; b < 768; b += DS_THREADS) (&st->hist[(pass & 1) ^ 1][0][0])[b] = 0;
	const int lane = threadIdx.x & 31, d = threadIdx.x >> 5;
	if (d < 3) {
		// lane l holds the counts of bytes 8 l .. 8 l + 7
		uint32_t c[8], sum = 0;
#pragma unroll
		for (int k = 0; k < 8; k++) {
			c[k] = __ldcg(&g[d * 256 + 8 * lane + k]);
			sum += c[k];
		}
		uint32_t inc = sum;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, inc, o);
			if (lane >= o) inc += u;
		}
		const uint64_t rank = st->rank[d];
		const bool here = rank >= inc - sum && rank < inc;
		if (__ballot_sync(0xFFFFFFFFu, here) == 0 && lane == 0) st->lost = 1;
		if (here) {
			uint64_t r = rank - (inc - sum);
			int k = 0;
			while (r >= c[k]) r -= c[k++];
			const uint64_t p = st->prefix[d] | (uint64_t) (8 * lane + k) << shift;
			st->prefix[d] = p;
			st->rank[d] = r;
			if (shift == 0) st->center[d] = (double) unordered((U) p);
		}
	}
	if (threadIdx.x == 0) st->done = 0;
}

// largest |x - c| over the particles and the three axes, in double; the
// non-negative doubles order like their bit patterns
template <typename F>
__global__ void k_max_distance(int64_t n, const F *__restrict__ x, const F *__restrict__ y,
                               const F *__restrict__ z, DomainState *st)
{
	const double cx = st->center[0], cy = st->center[1], cz = st->center[2];
	double m = 0;
	for (int64_t i = blockIdx.x * (int64_t) blockDim.x + threadIdx.x; i < n;
	     i += (int64_t) gridDim.x * blockDim.x) {
		m = fmax(m, fabs((double) x[i] - cx));
		m = fmax(m, fabs((double) y[i] - cy));
		m = fmax(m, fabs((double) z[i] - cz));
	}
#pragma unroll
	for (int o = 16; o; o >>= 1) m = fmax(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
	if ((threadIdx.x & 31) == 0) atomicMax(&st->max_bits, (unsigned long long) __double_as_longlong(m));
}

// the state's start: the ranks, and for one particle its position (data[0])
template <typename F>
__global__ void k_select_start(int64_t n, const F *x, const F *y, const F *z, DomainState *st)
{
	const int t = threadIdx.x;
	for (int b = t; b < 1536; b += blockDim.x) (&st->hist[0][0][0])[b] = 0;
	if (t < 3) {
		st->prefix[t] = 0;
		st->rank[t] = n > 1 ? (uint64_t) (n >> 1) - 1 : 0;      // 0-based among x[1 .. n-1]
		st->center[t] = (double) (t == 0 ? x[0] : t == 1 ? y[0] : z[0]);
	}
	if (t == 0) {
		st->done = 0;
		st->lost = 0;
		st->max_bits = 0;
	}
}

template <typename F>
int find_domain_typed(tvg_context *ctx, double origin[3], double *size)
{
	const int64_t n = ctx->n;
	cudaStream_t s = ctx->stream;
	const F *x = (const F *) ctx->f[FS_POS0], *y = (const F *) ctx->f[FS_POS1], *z = (const F *) ctx->f[FS_POS2];
	if (!ctx->domain_state) TVG_CHECK(tvg_alloc(ctx, &ctx->domain_state, sizeof(DomainState)));
	DomainState *st = (DomainState *) ctx->domain_state;
	// up to DS_BLOCKS blocks a SM
	const unsigned need = tvg_blocks(n, DS_IPT * DS_THREADS), grid = need < 148u * DS_BLOCKS ? need : 148u * DS_BLOCKS;
	k_select_start<F><<<TVG_CNT(ctx, 1), DS_THREADS, 0, s>>>(n, x, y, z, st);
	if (n > 1)
		for (int pass = 0; pass < (int) sizeof(F); pass++)
			k_select<F><<<TVG_CNT(ctx, grid), DS_THREADS, 0, s>>>(n, x, y, z, 8 * (int) sizeof(F) - 8 - 8 * pass,
			                                                      pass, st);
	k_max_distance<F><<<TVG_CNT(ctx, grid), DS_THREADS, 0, s>>>(n, x, y, z, st);
	TVG_CUDA(ctx, cudaGetLastError());
	DomainState h;
	const size_t from = offsetof(DomainState, lost);
	TVG_CUDA(ctx, cudaMemcpyAsync((char *) &h + from, (char *) st + from, sizeof(h) - from, cudaMemcpyDeviceToHost, s));
	TVG_CUDA(ctx, cudaStreamSynchronize(s));
	if (h.lost) return tvg_fail(ctx, TVG_E_CUDA, "find_domain: selection lost the rank");
	double maxd;
	memcpy(&maxd, &h.max_bits, 8);
	*size = 2.001 * maxd;                               // domain.c:832
	for (int d = 0; d < 3; d++) origin[d] = h.center[d] - 0.5 * *size;   // Float center[3] (domain.c:767)
	return TVG_OK;
}

} // namespace

extern "C" int tvg_find_domain(tvg_context *ctx, double origin[3], double *size)
{
	if (!ctx || !origin || !size) return TVG_E_BADINPUT;
	if (ctx->n <= 0) return tvg_fail(ctx, TVG_E_STATE, "find_domain: no particles");
	TVG_CUDA(ctx, cudaSetDevice(ctx->device));
	double o[3], sz = 0;
	if (ctx->cfg.periodic) {                            // domain.c:732-747
		sz = ctx->cfg.boxsize;
		o[0] = o[1] = o[2] = 0;
	} else {
		const int rc = ctx->cfg.float_bytes == 4 ? find_domain_typed<float>(ctx, o, &sz)
		                                         : find_domain_typed<double>(ctx, o, &sz);
		if (rc != TVG_OK) return rc;
	}
	for (int d = 0; d < 3; d++) origin[d] = o[d];
	*size = sz;
	return tvg_set_domain(ctx, o, sz);
}
