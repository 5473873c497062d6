// tvg_sort.cu -- PH-order sort of all particle fields.
//
// Replaces Qsort_Index on the 128-bit keys (sort.c:90-341, cmp_peanoKeys at
// peano.c:6-12) and reorder_collisionless_particles (peano.c:50-82).
//  1. LSD radix sort of (key_hi, index) on the 64-bit high key word: 8-bit
//     digits, one kernel per digit (k_radix_pass), the published one-sweep form
//     (Adinets and Merrill 2022) with decoupled look-back over the tiles' counts
//     (Merrill and Garland 2016). All eight digit histograms are
//     counted in one pass over the keys beforehand; a pass takes tiles of 4096 keys
//     (few keys: 1024) in the order of a device counter, ranks a tile's keys
//     stably with warp ballots, finds the tile's place among the equal digits of
//     earlier tiles by looking back over their published counts, four tiles at a
//     time, and writes through a shared-memory staging sort (coalesced runs per
//     digit). A digit that is
//     equal for every key (decided on the device) is not ranked: its pass copies
//     the keys through, so the number of passes, and with it the buffer a step
//     ends in, never depends on the data. Up to one tile of keys is sorted by one
//     block in shared memory (k_sort_tile).
//  2. Runs of equal high words are ordered by the low word (k_tie_rank: a thread
//     per key of a run counts the run's keys that precede it, r loads each in a
//     run of r; runs are rare and short unless positions coincide).
//  3. Every particle field is gathered through the permutation in one launch,
//     four particles per thread with 128-bit stores (and 128-bit loads where
//     the permutation keeps an aligned run of four in place).
// The resulting order is the ascending 128-bit key order, equal keys in
// input order (the reference's quicksort leaves equal keys in an
// unspecified order).
// Roofline: HBM bound; per pass 12 B read + 12 B write per key. Histogram, scan
// and scatter kernels per digit (three to five launches, 20 B read) took, with
// the gather of the fields, 4.65 ms for 16.7M particles, 0.47 ms for 400,000,
// 0.27 ms for 32,768 and 0.28 ms for 3001; this 2.44, 0.20, 0.10 and 0.06 ms. A
// pass over many keys waits on memory (of 15 stall cycles an instruction 4.3 on
// global loads, keys and look-back, and 2.1 on shared memory) at 29 of the 32 warps
// an SM holds (4M keys: 56 us, 0.95 TB/s of DRAM traffic, as the L2 holds much of
// both buffers).
#include <mutex>

#include "tvg_internal.cuh"

#define RS_THREADS 256
#define RS_TILE (RS_THREADS * 16)
#define RS_WARPS (RS_THREADS / 32)

// global histogram of all 8 digits of key_hi (to skip constant digits)
__global__ void k_digit_counts(int64_t n, const uint64_t *__restrict__ key, uint32_t *count)
{
	__shared__ uint32_t h[8 * 256];
	for (int i = threadIdx.x; i < 8 * 256; i += blockDim.x) h[i] = 0;
	__syncthreads();
	for (int64_t i = blockIdx.x * (int64_t) blockDim.x + threadIdx.x; i < n;
	     i += (int64_t) gridDim.x * blockDim.x) {
		uint64_t k = key[i];
#pragma unroll
		for (int d = 0; d < 8; d++) atomicAdd(&h[d * 256 + ((k >> (8 * d)) & 0xFF)], 1u);
	}
	__syncthreads();
	for (int i = threadIdx.x; i < 8 * 256; i += blockDim.x)
		if (h[i]) atomicAdd(&count[i], h[i]);
}

// A block per digit: its counts to exclusive offsets, skip[d] = 1 when the digit
// has the same value in all n keys, and the pass's tile counter to zero.
__global__ void __launch_bounds__(256) k_digit_offsets(int64_t n, uint32_t *count, int32_t *skip, uint32_t *tiles)
{
	__shared__ uint32_t s_warp[8];
	const int d = blockIdx.x, t = threadIdx.x, lane = t & 31, w = t >> 5;
	const uint32_t c = count[d * 256 + t];
	const int all = __syncthreads_or(c == (uint32_t) n);
	uint32_t inc = c;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, inc, o);
		if (lane >= o) inc += u;
	}
	if (lane == 31) s_warp[w] = inc;
	__syncthreads();
	for (int k = 0; k < w; k++) inc += s_warp[k];
	count[d * 256 + t] = inc - c;
	if (t == 0) {
		skip[d] = all;
		tiles[d] = 0;
	}
}

// exclusive prefix sum of one value per thread of a 256-thread block
__device__ __forceinline__ uint32_t scan256(uint32_t v, uint32_t *s_warp)
{
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	uint32_t inc = v;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, inc, o);
		if (lane >= o) inc += u;
	}
	if (lane == 31) s_warp[w] = inc;
	__syncthreads();
	uint32_t base = 0;
#pragma unroll
	for (int k = 0; k < RS_WARPS; k++) base += k < w ? s_warp[k] : 0u;
	return base + inc - v;
}

// lanes that hold the digit d of this one (256: none), by a ballot per bit (with
// a match instruction the sort of 16.7M keys took 2.80 ms instead of 2.48)
__device__ __forceinline__ unsigned equal_digits(uint32_t d)
{
	unsigned peers = __ballot_sync(0xFFFFFFFFu, d < 256);
#pragma unroll
	for (int b = 0; b < 8; b++) {
		const bool one = (d >> b) & 1;
		const unsigned m = __ballot_sync(0xFFFFFFFFu, one);
		peers &= one ? m : ~m;
	}
	return peers;
}

// Ranks a tile's digits: a warp holds IPT x 32 consecutive keys, key r of
// lane l at r * 32 + l; whist[w][d] counts digit d of warp w as it goes, so that
// rank[r] is the key's place among the equal digits of its warp. Returns with
// whist holding, per digit, the offset of each warp among the tile's equal
// digits, and in thread t the tile's count of digit t.
template <int IPT>
__device__ __forceinline__ uint32_t rank_tile(const uint32_t (&d)[IPT], uint32_t (&rank)[IPT],
                                              uint32_t (*whist)[256])
{
	const int t = threadIdx.x, lane = t & 31, w = t >> 5;
	const unsigned lt = (1u << lane) - 1u;
#pragma unroll
	for (int k = 0; k < RS_WARPS; k++) whist[k][t] = 0;
	__syncthreads();
#pragma unroll
	for (int r = 0; r < IPT; r++) {
		const unsigned peers = equal_digits(d[r]);
		const int leader = __ffs(peers) - 1;
		uint32_t old = 0;
		if (lane == leader && d[r] < 256) {
			old = whist[w][d[r]];
			whist[w][d[r]] = old + (uint32_t) __popc(peers);
		}
		old = __shfl_sync(0xFFFFFFFFu, old, leader);
		rank[r] = old + (uint32_t) __popc(peers & lt);
		__syncwarp();
	}
	__syncthreads();
	uint32_t run = 0;
#pragma unroll
	for (int k = 0; k < RS_WARPS; k++) {
		const uint32_t c = whist[k][t];
		whist[k][t] = run;
		run += c;
	}
	return run;
}

// published state of (tile, digit): the tile's count, or the count of all tiles
// up to it; 0: not published yet
#define RS_COUNT 0x40000000u
#define RS_TOTAL 0x80000000u
#define RS_VALUE 0x3FFFFFFFu
// polls of one predecessor's state before the pass gives up (about a second);
// tiles are taken in order, so the predecessors run or have run
#define RS_SPIN (1 << 21)
// predecessors looked at together
#define RS_LOOK 4

// One digit's pass. state: ntiles x 256 words of this pass, zero at its start;
// next: those of the next pass, zeroed here. vin null: the values are the
// indices.
template <int IPT>
__global__ void __launch_bounds__(RS_THREADS, IPT > 4 ? 4 : 6)
k_radix_pass(int64_t n, int shift, const uint64_t *__restrict__ kin, const uint32_t *__restrict__ vin,
             uint64_t *__restrict__ kout, uint32_t *__restrict__ vout, const uint32_t *__restrict__ offsets,
             volatile uint32_t *state, uint32_t *__restrict__ next, uint32_t *tiles,
             const int32_t *__restrict__ skip, int *status)
{
	constexpr int TILE = RS_THREADS * IPT;
	__shared__ __align__(16) uint64_t skey[TILE];     // keys, then values
	__shared__ uint32_t whist[RS_WARPS][256];
	__shared__ uint32_t dstart[256], gstart[256], s_warp[RS_WARPS], s_tile;
	const int t = threadIdx.x, lane = t & 31, w = t >> 5;
	next[(int64_t) blockIdx.x * 256 + t] = 0;
	if (skip[shift >> 3]) {                              // constant digit: the order stays
		const int64_t b0 = (int64_t) blockIdx.x * TILE;
		const int c0 = (int) min((int64_t) TILE, n - b0);
		for (int p = t; p < c0; p += RS_THREADS) {
			kout[b0 + p] = kin[b0 + p];
			vout[b0 + p] = vin ? vin[b0 + p] : (uint32_t) (b0 + p);
		}
		return;
	}
	if (t == 0) s_tile = atomicAdd(&tiles[shift >> 3], 1u);
	__syncthreads();
	const int64_t tile = s_tile, base = tile * TILE;
	const int cnt = (int) min((int64_t) TILE, n - base);
	uint64_t k[IPT];
	uint32_t d[IPT], rank[IPT];
	const int first = w * (32 * IPT) + lane;
#pragma unroll
	for (int r = 0; r < IPT; r++) {
		const int idx = first + 32 * r;
		k[r] = idx < cnt ? kin[base + idx] : 0;
		d[r] = idx < cnt ? (uint32_t) (k[r] >> shift) & 0xFF : 256u;
	}
	const uint32_t count = rank_tile(d, rank, whist);
	state[tile * 256 + t] = (tile == 0 ? RS_TOTAL : RS_COUNT) | count;
	dstart[t] = scan256(count, s_warp);
	// look back: thread t sums digit t's counts of the earlier tiles
	uint32_t before = 0;
	for (int64_t q = tile - 1; q >= 0; q -= RS_LOOK) {
		uint32_t v[RS_LOOK];
#pragma unroll
		for (int j = 0; j < RS_LOOK; j++) v[j] = q - j >= 0 ? state[(q - j) * 256 + t] : RS_TOTAL;
		bool done = false;
#pragma unroll
		for (int j = 0; j < RS_LOOK; j++) {
			if (done) continue;
			for (int spin = 0; v[j] == 0; spin++) {
				if (spin > RS_SPIN) {
					atomicOr(status, TVG_ST_TIMEOUT);
					v[j] = RS_TOTAL;
					break;
				}
				v[j] = state[(q - j) * 256 + t];
			}
			before += v[j] & RS_VALUE;
			done = v[j] & RS_TOTAL;
		}
		if (done) break;
	}
	if (tile > 0) state[tile * 256 + t] = RS_TOTAL | ((before + count) & RS_VALUE);
	gstart[t] = offsets[t] + before - dstart[t];
	__syncthreads();
#pragma unroll
	for (int r = 0; r < IPT; r++) {
		if (d[r] < 256) {
			rank[r] += dstart[d[r]] + whist[w][d[r]];
			skey[rank[r]] = k[r];
		}
	}
	__syncthreads();
	uint32_t dest[IPT];
#pragma unroll
	for (int r = 0; r < IPT; r++) {
		const int p = t + RS_THREADS * r;
		dest[r] = 0xFFFFFFFFu;
		if (p < cnt) {
			const uint64_t key = skey[p];
			dest[r] = gstart[(uint32_t) (key >> shift) & 0xFF] + (uint32_t) p;
			if (dest[r] < n) kout[dest[r]] = key;
		}
	}
	__syncthreads();
	uint32_t *sval = (uint32_t *) skey;
#pragma unroll
	for (int r = 0; r < IPT; r++) {
		const int idx = first + 32 * r;
		if (idx < cnt) sval[rank[r]] = vin ? vin[base + idx] : (uint32_t) (base + idx);
	}
	__syncthreads();
#pragma unroll
	for (int r = 0; r < IPT; r++) {
		const int p = t + RS_THREADS * r;
		if (dest[r] < n) vout[dest[r]] = sval[p];
	}
}

// up to RS_TILE keys in one block: all eight digits in shared memory; key is
// sorted in place, perm receives the input indices
__global__ void __launch_bounds__(RS_THREADS)
k_sort_tile(int n, uint64_t *__restrict__ key, uint32_t *__restrict__ perm)
{
	constexpr int IPT = RS_TILE / RS_THREADS;
	__shared__ __align__(16) uint64_t skey[RS_TILE];
	__shared__ uint32_t whist[RS_WARPS][256];
	__shared__ uint32_t dstart[256], s_warp[RS_WARPS];
	uint32_t *sval = (uint32_t *) skey;
	const int t = threadIdx.x, lane = t & 31, w = t >> 5, first = w * (32 * IPT) + lane;
	uint64_t k[IPT];
	uint32_t v[IPT], d[IPT], rank[IPT];
#pragma unroll
	for (int r = 0; r < IPT; r++) {
		const int idx = first + 32 * r;
		k[r] = idx < n ? key[idx] : 0;
		v[r] = (uint32_t) idx;
	}
	for (int shift = 0; shift < 64; shift += 8) {
#pragma unroll
		for (int r = 0; r < IPT; r++) d[r] = first + 32 * r < n ? (uint32_t) (k[r] >> shift) & 0xFF : 256u;
		const uint32_t count = rank_tile(d, rank, whist);
		if (__syncthreads_or(count == (uint32_t) n)) continue;
		dstart[t] = scan256(count, s_warp);
		__syncthreads();
#pragma unroll
		for (int r = 0; r < IPT; r++)
			if (d[r] < 256) {
				rank[r] += dstart[d[r]] + whist[w][d[r]];
				skey[rank[r]] = k[r];
			}
		__syncthreads();
#pragma unroll
		for (int r = 0; r < IPT; r++)
			if (d[r] < 256) k[r] = skey[first + 32 * r];
		__syncthreads();
#pragma unroll
		for (int r = 0; r < IPT; r++)
			if (d[r] < 256) sval[rank[r]] = v[r];
		__syncthreads();
#pragma unroll
		for (int r = 0; r < IPT; r++)
			if (d[r] < 256) v[r] = sval[first + 32 * r];
		__syncthreads();
	}
#pragma unroll
	for (int r = 0; r < IPT; r++) {
		const int idx = first + 32 * r;
		if (idx < n) {
			key[idx] = k[r];
			perm[idx] = v[r];
		}
	}
}

// Orders runs of equal key_hi by the low key word, stably (the radix passes
// sort the high words only): out = perm with each run reordered. Every
// element of a run finds the run's ends and its rank by one pass over the run,
// in parallel, so a run of r equal high words costs O(r) time on r threads;
// elements outside runs are copied.
__global__ void k_tie_rank(int64_t n, const uint64_t *__restrict__ hi, const uint64_t *__restrict__ lo_orig,
                           const uint32_t *__restrict__ perm, uint32_t *__restrict__ out)
{
	const int64_t i = blockIdx.x * (int64_t) blockDim.x + threadIdx.x;
	if (i >= n) return;
	const uint64_t h = hi[i];
	// (a pass that gave up leaves places unwritten: keep every index inside)
	const uint32_t last = (uint32_t) (n - 1), pv = min(perm[i], last);
	if (!((i > 0 && hi[i - 1] == h) || (i + 1 < n && hi[i + 1] == h))) {
		out[i] = pv;
		return;
	}
	int64_t a = i, e = i + 1;
	while (a > 0 && hi[a - 1] == h) a--;
	while (e < n && hi[e] == h) e++;
	const uint64_t kv = lo_orig[pv];
	int64_t r = 0;
	for (int64_t j = a; j < e; j++) {
		const uint64_t kj = lo_orig[min(perm[j], last)];
		r += (kj < kv || (kj == kv && j < i)) ? 1 : 0;
	}
	out[a + r] = pv;
}

// the particle fields and the low key words
struct GatherList {
	const void *in[FS_NFIELDS + 1];
	void *out[FS_NFIELDS + 1];
	int bytes[FS_NFIELDS + 1];
	int nf;
};

// All particle fields through the permutation in one pass (perm read once).
// A thread moves four consecutive particles i .. i+3 (i a multiple of 4):
// their permutation entries come in one 128-bit load, and every field is
// written with 128-bit stores (one per 4-byte field, two per 8-byte field).
// Where the four sources are one aligned run (perm[i] a multiple of 4 and
// perm[i+k] = perm[i] + k: particles that kept their place in the order,
// nearly all of them between the steps of a run) the loads are 128-bit too;
// elsewhere the four elements are gathered one by one. Buffers start
// 256-byte aligned, so every vector access is aligned.
__global__ void k_gather_fields(int64_t n, const uint32_t *__restrict__ perm, GatherList g)
{
	const int64_t i = 4 * (blockIdx.x * (int64_t) blockDim.x + threadIdx.x);
	if (i >= n) return;
	if (i + 4 > n) {                               // ragged end: scalar
		for (int64_t j = i; j < n; j++) {
			const uint32_t src = perm[j];
			for (int f = 0; f < g.nf; f++) {
				if (g.bytes[f] == 8) ((uint64_t *) g.out[f])[j] = ((const uint64_t *) g.in[f])[src];
				else ((uint32_t *) g.out[f])[j] = ((const uint32_t *) g.in[f])[src];
			}
		}
		return;
	}
	const uint4 p = *(const uint4 *) (perm + i);
	const bool run = (p.x & 3u) == 0 && p.y == p.x + 1 && p.z == p.x + 2 && p.w == p.x + 3;
	for (int f = 0; f < g.nf; f++) {
		if (g.bytes[f] == 8) {
			const uint64_t *in = (const uint64_t *) g.in[f];
			uint4 *out = (uint4 *) ((uint64_t *) g.out[f] + i);
			if (run) {
				const uint4 *v = (const uint4 *) (in + p.x);
				out[0] = __ldg(v);
				out[1] = __ldg(v + 1);
			} else {
				const uint64_t a = in[p.x], b = in[p.y], c = in[p.z], d = in[p.w];
				out[0] = make_uint4((uint32_t) a, (uint32_t) (a >> 32), (uint32_t) b, (uint32_t) (b >> 32));
				out[1] = make_uint4((uint32_t) c, (uint32_t) (c >> 32), (uint32_t) d, (uint32_t) (d >> 32));
			}
		} else {
			const uint32_t *in = (const uint32_t *) g.in[f];
			uint4 *out = (uint4 *) ((uint32_t *) g.out[f] + i);
			if (run) *out = __ldg((const uint4 *) (in + p.x));
			else *out = make_uint4(in[p.x], in[p.y], in[p.z], in[p.w]);
		}
	}
}

// The eight passes over n keys: kin / kout and the two value buffers alternate,
// and after the eighth pass the result is back in kin and vb. count: 8 x 256
// words; st[2]: tile states; tiles: 8 words.
template <int IPT>
static cudaError_t radix_passes(cudaStream_t s, int64_t n, const uint64_t *key, uint64_t *kin, uint64_t *kout,
                                uint32_t *va, uint32_t *vb, uint32_t *count, int32_t *skip,
                                uint32_t *const st[2], uint32_t *tiles, int *status)
{
	constexpr int TILE = RS_THREADS * IPT;
	const int64_t ntiles = (n + TILE - 1) / TILE, ncount = (n + RS_TILE - 1) / RS_TILE;
	cudaError_t e = cudaMemsetAsync(count, 0, 4 * 8 * 256, s);
	if (e == cudaSuccess) e = cudaMemsetAsync(st[0], 0, 4 * 256 * (size_t) ntiles, s);
	if (e != cudaSuccess) return e;
	const unsigned nb = (unsigned) (ncount < 296 ? ncount : 296);
	k_digit_counts<<<nb, 512, 0, s>>>(n, key, count);
	k_digit_offsets<<<8, 256, 0, s>>>(n, count, skip, tiles);
	const uint32_t *vin = nullptr;
	const uint64_t *in = key;
	for (int d = 0; d < 8; d++) {
		uint64_t *out = d & 1 ? kin : kout;
		uint32_t *vout = d & 1 ? vb : va;
		k_radix_pass<IPT><<<(unsigned) ntiles, RS_THREADS, 0, s>>>(n, 8 * d, in, vin, out, vout, count + 256 * d,
		                                                      st[d & 1], st[(d & 1) ^ 1], tiles, skip, status);
		in = out;
		vin = vout;
	}
	return cudaGetLastError();
}
#define RS_LAUNCHES 10

// Up to this many keys the tiles are of 1024 keys instead of 4096: a pass is then
// one wave of blocks, as long as one block's chain of loads, ranks and look-back.
// Sort and gather, tiles of 4096 / 1024: 5000 keys 156 / 109 us, 32768 172 / 126,
// 200,000 212 / 176, 400,000 224 / 214, 700,000 288 / 291, 1,000,000 333 / 360.
#define RS_SMALL_KEYS (1 << 19)

// words of one pass's tile states for up to n keys
size_t tvg_sort_state_words(int64_t n)
{
	const int64_t large = (n + RS_TILE - 1) / RS_TILE, few = n < RS_SMALL_KEYS ? n : RS_SMALL_KEYS;
	const int64_t small = (few + RS_THREADS * 4 - 1) / (RS_THREADS * 4);
	return 256 * (size_t) ((large > small ? large : small) + 1);
}

int tvg_impl_sort(tvg_context *ctx, uint32_t *perm_out)
{
	const int64_t n = ctx->n;
	if (n == 0) return TVG_OK;
	cudaStream_t s = ctx->stream;
	uint64_t *kin = ctx->key_hi;
	uint32_t *vin = ctx->perm, *vout = ctx->perm_tmp;
	if (n <= RS_TILE) {
		k_sort_tile<<<TVG_CNT(ctx, 1), RS_THREADS, 0, s>>>((int) n, kin, vin);
		TVG_CUDA(ctx, cudaGetLastError());
	} else {
		uint32_t *const st[2] = { ctx->sort_hist, ctx->sort_off };
		ctx->launches += RS_LAUNCHES;
		const auto passes = n <= RS_SMALL_KEYS ? radix_passes<4> : radix_passes<16>;
		TVG_CUDA(ctx, passes(s, n, kin, kin, ctx->key_tmp, vout, vin, ctx->digit_count, ctx->dc->sort_skip, st,
		                     ctx->dc->sort_tiles, ctx->status));
	}
	// runs of equal high words by the low words, into the other buffer
	k_tie_rank<<<TVG_CNT(ctx, tvg_blocks(n, 256)), 256, 0, s>>>(n, kin, ctx->key_lo, vin, vout);
	ctx->perm = vout; ctx->perm_tmp = vin;
	GatherList g;
	g.in[0] = ctx->key_lo;
	g.out[0] = ctx->key_tmp;
	g.bytes[0] = 8;
	g.nf = 1;
	{ uint64_t *t = ctx->key_lo; ctx->key_lo = ctx->key_tmp; ctx->key_tmp = t; }
	for (int f = 0; f < FS_NFIELDS; f++) {
		g.in[g.nf] = ctx->f[f];
		g.out[g.nf] = ctx->falt[f];
		g.bytes[g.nf] = (int) tvg_field_bytes(ctx, f);
		g.nf++;
	}
	if (ctx->gather_wait) TVG_CUDA(ctx, cudaStreamWaitEvent(s, ctx->gather_wait, 0));
	k_gather_fields<<<TVG_CNT(ctx, tvg_blocks((n + 3) / 4, 256)), 256, 0, s>>>(n, ctx->perm, g);
	TVG_CUDA(ctx, cudaGetLastError());
	for (int f = 0; f < FS_NFIELDS; f++) { void *t = ctx->f[f]; ctx->f[f] = ctx->falt[f]; ctx->falt[f] = t; }
	if (perm_out)
		TVG_CUDA(ctx, cudaMemcpyAsync(perm_out, ctx->perm, 4 * n, cudaMemcpyDeviceToHost, s));
	return TVG_OK;
}

// ------------------------------------------------------------------------
// Sort without any allocation (tvg_sort_keys_noalloc).
//
// Some callers cannot allocate device memory: a host code whose own memory
// manager reserves the GPU's memory up front and forbids allocations behind
// its back, or a latency-bound step loop that cannot pay the device-wide
// synchronisation that cudaMalloc and cudaFree imply. For them this variant
// of the sort keeps its scratch (the
// key and index ping-pong buffers and the digit histograms) in one file-scope
// device array of fixed size, so a call allocates nothing; the caller passes
// the keys and receives the permutation in its own device buffers.
//
// The array belongs to every GPU that loads this library, for the life of the
// process (about 6.4 MB). All calls on a device share it and it keeps the
// last call's contents: a call zeroes the counts and states it starts from. Two
// calls that overlap on the same GPU (from two host threads, or on two streams)
// corrupt each other's scratch.
// ------------------------------------------------------------------------

#define NOALLOC_TILES (TVG_NOALLOC_MAX_KEYS / RS_TILE)

struct NoallocScratch {
	uint64_t key[2][TVG_NOALLOC_MAX_KEYS];   // sorted high words, ping-pong
	uint32_t idx[2][TVG_NOALLOC_MAX_KEYS];   // permutation, ping-pong
	uint32_t state[2][256 * NOALLOC_TILES];  // the passes' tile states
	uint32_t count[8 * 256];                 // digit counts, then offsets
	int32_t skip[8];
	uint32_t tiles[8];
	int status;
};

static __device__ __align__(256) unsigned char g_noalloc_scratch[sizeof(NoallocScratch)];

// Device address of the scratch array, looked up once per device with that
// device current (the host-side symbol is not a device address).
static NoallocScratch *noalloc_scratch(int device)
{
	static std::mutex mu;
	static NoallocScratch *addr[64] = { nullptr };
	if (device < 0 || device >= 64) return nullptr;
	std::lock_guard<std::mutex> lock(mu);
	if (!addr[device]) {
		void *p = nullptr;
		if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess) {
			cudaGetLastError();
			return nullptr;
		}
		addr[device] = (NoallocScratch *) p;
	}
	return addr[device];
}

extern "C" int tvg_sort_keys_noalloc(const uint64_t *key_hi, const uint64_t *key_lo, int64_t n,
                                     uint32_t *perm)
{
	if (n < 0 || n > TVG_NOALLOC_MAX_KEYS) return TVG_E_BADINPUT;
	if (n == 0) return TVG_OK;
	if (!key_hi || !key_lo || !perm) return TVG_E_BADINPUT;
	int device = 0;
	if (cudaGetDevice(&device) != cudaSuccess) { cudaGetLastError(); return TVG_E_CUDA; }
	NoallocScratch *S = noalloc_scratch(device);
	if (!S) return TVG_E_CUDA;
	cudaStream_t s = 0;
	cudaError_t e = cudaMemsetAsync(&S->status, 0, sizeof(int), s);
	if (e == cudaSuccess) {
		uint32_t *const st[2] = { S->state[0], S->state[1] };
		e = radix_passes<16>(s, n, key_hi, S->key[0], S->key[1], S->idx[0], S->idx[1], S->count, S->skip, st, S->tiles,
		                 &S->status);
	}
	if (e == cudaSuccess) {
		k_tie_rank<<<tvg_blocks(n, 256), 256, 0, s>>>(n, S->key[0], key_lo, S->idx[1], perm);
		e = cudaGetLastError();
	}
	int status = 0;
	if (e == cudaSuccess) e = cudaMemcpyAsync(&status, &S->status, sizeof(int), cudaMemcpyDeviceToHost, s);
	if (e == cudaSuccess) e = cudaStreamSynchronize(s);
	if (e == cudaSuccess && status) return TVG_E_TIMEOUT;
	return e == cudaSuccess ? TVG_OK : TVG_E_CUDA;
}
