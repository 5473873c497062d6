// tvg_ewald_mlp.cu -- the learned Ewald correction: a 3 -> 64 -> 64 -> 3
// network (tanh) on the symmetry-folded octant that stands in for the
// interpolation of the lattice-minus-image force T(x) (the quantity of the
// reference's Ewald table, Gravity/periodic.c:35-113, 352-461).
//
// Model: x in [0, 1/2]^3 (box units, the folded octant; the other octants
// follow from the symmetries T_a(.., -x_b, ..) = -T_a if a = b, +T_a
// otherwise), v = 4 x - 1, and
//     T(x) = 4 pi x / 3 + S(x) + C . m(v) + s N(v)
// (tvg_ewald_mlp.cuh): the linear background term, the seven nearest lattice
// images, a cubic least-squares fit, and the network N on what is left,
// scaled by that rest's rms s. Without S and the fit the same network reached
// 5.6e-3 rms in T; with them, 1.4e-4 (FP64 fits of 2^15 points, 6000 Adam
// steps). Parameters, 4672 floats:
//     W1[64][3] @0, b1[64] @192, W2[64][64] @256, b2[64] @4352,
//     W3[3][64] @4416, b3[3] @4608 (the network, 4611, trained);
//     C[3][20] @4611, s @4671 (fitted).
//
// Training (own kernels): 2^20 seeded points uniform on the octant, FP64
// targets T(x) by the Ewald sum of the table generator (tvg_ewald_sum.cuh)
// minus the analytic part; the normal equations of the cubic fit summed in
// FP64 (fixed-order block sums) and solved on the host (Cholesky); then the
// network's FP32 minibatch mean-square loss on the normalised rest: tiles of 64
// samples run forward and backward in shared memory, the gradients summed as
// matrix products into one slot per block, then over the slots in fixed order
// (deterministic), then Adam.
//
// Inference: BF16 weights (rounded once after training), FP32 arithmetic and
// accumulation. The exact FP64 table (the reference's 65^3 nodes) validates
// it: tvg_ewald_mlp_validate measures the max and rms error there, and the
// walk refuses the learned correction when the max error is above the limit
// the caller gives.
#include <math.h>

#include <algorithm>
#include <cmath>
#include <stdlib.h>

#include <vector>

#include "tvg_internal.cuh"
#include "tvg_ewald_sum.cuh"
#include "tvg_ewald_mlp.cuh"

// ------------------------------------------------------------ data

__device__ __forceinline__ uint64_t splitmix64(uint64_t z)
{
	z += 0x9E3779B97F4A7C15ull;
	z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
	z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
	return z ^ (z >> 31);
}

__device__ __forceinline__ double u01(uint64_t r) { return (double) (r >> 11) * (1.0 / 9007199254740992.0); }

// points uniform on [0, 1/2]^3 (FP32-representable) and, in FP64, what the
// analytic part leaves of T there
__global__ void k_mlp_data(int64_t n, uint64_t seed, float *x, double *yraw)
{
	const int64_t i = blockIdx.x * (int64_t) blockDim.x + threadIdx.x;
	if (i >= n) return;
	double p[3], f[3], a[3], pot;
	for (int d = 0; d < 3; d++)
		p[d] = (double) (float) (0.5 * u01(splitmix64(seed ^ (uint64_t) (3 * i + d) * 0x2545F4914F6CDD1Dull)));
	ewald_point(p, f, &pot);
	mlp_analytic(p, a);
	for (int d = 0; d < 3; d++) {
		x[3 * i + d] = (float) p[d];
		yraw[3 * i + d] = f[d] - a[d];
	}
}

// normal equations of the cubic fit: entry e < 210 is G_ij = sum m_i m_j
// (i <= j, row by row), e < 270 is b_ai = sum y_a m_i, e < 273 is sum y_a^2;
// block (e, c) sums the samples of chunk c in a fixed order
#define LSQ_NE 273
#define LSQ_CHUNKS 64
__global__ void __launch_bounds__(128)
k_mlp_lsq(int64_t n, const float *__restrict__ x, const double *__restrict__ yraw, double *part)
{
	const int e = blockIdx.x, c = blockIdx.y;
	int kind, i = 0, j = 0, a = 0;
	if (e < 210) {
		kind = 0;
		int r = e;
		while (r >= MLP_NMONO - i) { r -= MLP_NMONO - i; i++; }
		j = i + r;
	} else if (e < 270) {
		kind = 1;
		a = (e - 210) / MLP_NMONO;
		i = (e - 210) % MLP_NMONO;
	} else {
		kind = 2;
		a = e - 270;
	}
	const int64_t lo = n * c / LSQ_CHUNKS, hi = n * (c + 1) / LSQ_CHUNKS;
	double acc = 0;
	for (int64_t q = lo + threadIdx.x; q < hi; q += blockDim.x) {
		const double v[3] = { 4.0 * x[3 * q] - 1.0, 4.0 * x[3 * q + 1] - 1.0, 4.0 * x[3 * q + 2] - 1.0 };
		double m[MLP_NMONO];
		mlp_monomials<double>(v, m);
		if (kind == 0) acc += m[i] * m[j];
		else if (kind == 1) acc += yraw[3 * q + a] * m[i];
		else acc += yraw[3 * q + a] * yraw[3 * q + a];
	}
#pragma unroll
	for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
	__shared__ double ws[4];
	if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = acc;
	__syncthreads();
	if (threadIdx.x == 0) part[(int64_t) e * LSQ_CHUNKS + c] = ((ws[0] + ws[1]) + ws[2]) + ws[3];
}

// network targets: (what the analytic part and the fit leave) / s, with the
// FP32 coefficients inference uses
__global__ void k_mlp_target(int64_t n, const float *__restrict__ x, const double *__restrict__ yraw,
                             const float *__restrict__ prm, float *y)
{
	const int64_t q = blockIdx.x * (int64_t) blockDim.x + threadIdx.x;
	if (q >= n) return;
	const double v[3] = { 4.0 * x[3 * q] - 1.0, 4.0 * x[3 * q + 1] - 1.0, 4.0 * x[3 * q + 2] - 1.0 };
	double m[MLP_NMONO];
	mlp_monomials<double>(v, m);
	const double inv_s = 1.0 / (double) prm[MLP_SCALE];
	for (int a = 0; a < 3; a++) {
		double r = yraw[3 * q + a];
		for (int k = 0; k < MLP_NMONO; k++) r -= (double) prm[MLP_POLY + MLP_NMONO * a + k] * m[k];
		y[3 * q + a] = (float) (r * inv_s);
	}
}

// ------------------------------------------------------------ training

__device__ __forceinline__ float warp_sum(float v)
{
#pragma unroll
	for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
	return v;
}

// Forward and backward of tiles of MT samples, gradients summed over a block's
// tiles in registers and written to the block's slot. Per sample the network is
// three 64 x 64 products (W2 a1, W2^T dz2 and the outer product dz2 a1^T), FP32 FMA
// bound: two threads share a sample (32 neurons each) for the first two, and
// the outer products of a tile are one 64 x 64 x MT product with an 8 x 4 tile of
// dW2 a thread, so that a weight gradient costs one FMA a sample (a warp's
// butterfly sum of every parameter took 10 instructions: 123 us for 16,384
// samples, 26 us now). Samples past n contribute zero.
#define MT 64
#define MT_THREADS 128
#define MT_LD 68                // row stride: 16-byte rows, conflict-free by quarter warps
struct MlpTile {
	float w2[MLP_H * MLP_H];
	float a1[MT * MT_LD], a2[MT * MT_LD], dz2[MT * MT_LD], dz1[MT * MT_LD];
	float w1[3 * MLP_H], b1[MLP_H], b2[MLP_H], w3[3 * MLP_H], b3[4];
	float v[MT][4], dy[MT][4], out[2][MT][4];
};

__global__ void __launch_bounds__(MT_THREADS)
k_mlp_grad(int64_t n, const float *__restrict__ x, const float *__restrict__ y,
           const float *__restrict__ prm, float inv_norm, float *slots, float *loss_slots)
{
	extern __shared__ __align__(16) unsigned char mlp_smem[];
	MlpTile &T = *(MlpTile *) mlp_smem;
	const int tid = threadIdx.x, s = tid & (MT - 1), half = tid / MT, j0 = half * (MLP_H / 2);
	for (int e = tid; e < MLP_H * MLP_H; e += MT_THREADS) T.w2[e] = prm[MLP_W2 + e];
	for (int e = tid; e < 3 * MLP_H; e += MT_THREADS) {
		T.w1[e] = prm[MLP_W1 + e];
		T.w3[e] = prm[MLP_W3 + e];
	}
	if (tid < MLP_H) {
		T.b1[tid] = prm[MLP_B1 + tid];
		T.b2[tid] = prm[MLP_B2 + tid];
	}
	if (tid < 3) T.b3[tid] = prm[MLP_B3 + tid];
	// this thread's parameters: an 8 x 4 tile of dW2; of neuron `s` of layer 2
	// (half 0) or 1 (half 1) the bias and three weights; db3 of component tid
	const int tj = 8 * (tid / 16), ti = 4 * (tid % 16);
	float g2[8][4], gs[4] = { 0.f, 0.f, 0.f, 0.f }, g3 = 0.f, loss = 0.f;
#pragma unroll
	for (int a = 0; a < 8; a++)
#pragma unroll
		for (int b = 0; b < 4; b++) g2[a][b] = 0.f;
	const int64_t ntile = (n + MT - 1) / MT;
	for (int64_t tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
		const int64_t q = tile * MT + s;
		const bool have = q < n;
		float v[3], t[3];
#pragma unroll
		for (int d = 0; d < 3; d++) {
			v[d] = have ? 4.f * x[3 * q + d] - 1.f : 0.f;
			t[d] = have ? y[3 * q + d] : 0.f;
		}
		__syncthreads();          // the weights, and the previous tile's last readers
		if (half == 0)
#pragma unroll
			for (int d = 0; d < 3; d++) T.v[s][d] = v[d];
#pragma unroll 8
		for (int j = j0; j < j0 + MLP_H / 2; j += 4) {
			float a[4];
#pragma unroll
			for (int k = 0; k < 4; k++)
				a[k] = tanhf(T.b1[j + k] + T.w1[3 * (j + k)] * v[0] + T.w1[3 * (j + k) + 1] * v[1]
				             + T.w1[3 * (j + k) + 2] * v[2]);
			*(float4 *) &T.a1[s * MT_LD + j] = make_float4(a[0], a[1], a[2], a[3]);
		}
		__syncthreads();
		float a1[MLP_H];
#pragma unroll
		for (int i = 0; i < MLP_H; i += 4) {
			const float4 f = *(const float4 *) &T.a1[s * MT_LD + i];
			a1[i] = f.x; a1[i + 1] = f.y; a1[i + 2] = f.z; a1[i + 3] = f.w;
		}
		float o[3] = { 0.f, 0.f, 0.f };
		for (int j = j0; j < j0 + MLP_H / 2; j += 4) {
			float z[4];
#pragma unroll
			for (int k = 0; k < 4; k++) z[k] = T.b2[j + k];
#pragma unroll
			for (int i = 0; i < MLP_H; i += 4)
#pragma unroll
				for (int k = 0; k < 4; k++) {
					const float4 w = *(const float4 *) &T.w2[MLP_H * (j + k) + i];
					z[k] = fmaf(w.x, a1[i], z[k]);
					z[k] = fmaf(w.y, a1[i + 1], z[k]);
					z[k] = fmaf(w.z, a1[i + 2], z[k]);
					z[k] = fmaf(w.w, a1[i + 3], z[k]);
				}
#pragma unroll
			for (int k = 0; k < 4; k++) {
				z[k] = tanhf(z[k]);
				o[0] = fmaf(T.w3[j + k], z[k], o[0]);
				o[1] = fmaf(T.w3[MLP_H + j + k], z[k], o[1]);
				o[2] = fmaf(T.w3[2 * MLP_H + j + k], z[k], o[2]);
			}
			*(float4 *) &T.a2[s * MT_LD + j] = make_float4(z[0], z[1], z[2], z[3]);
		}
#pragma unroll
		for (int d = 0; d < 3; d++) T.out[half][s][d] = o[d];
		__syncthreads();
		float dy[3];
#pragma unroll
		for (int d = 0; d < 3; d++) {
			const float r = have ? T.b3[d] + T.out[0][s][d] + T.out[1][s][d] - t[d] : 0.f;
			if (half == 0) loss = fmaf(r, r, loss);
			dy[d] = 2.f * r * inv_norm;
			if (half == 0) T.dy[s][d] = dy[d];
		}
		for (int j = j0; j < j0 + MLP_H / 2; j += 4) {
			const float4 f = *(const float4 *) &T.a2[s * MT_LD + j];
			const float a2[4] = { f.x, f.y, f.z, f.w };
			float dz[4];
#pragma unroll
			for (int k = 0; k < 4; k++)
				dz[k] = (T.w3[j + k] * dy[0] + T.w3[MLP_H + j + k] * dy[1] + T.w3[2 * MLP_H + j + k] * dy[2])
				      * (1.f - a2[k] * a2[k]);
			*(float4 *) &T.dz2[s * MT_LD + j] = make_float4(dz[0], dz[1], dz[2], dz[3]);
		}
		__syncthreads();
		// dz1 of this half's neurons: W2^T dz2
		float dh[MLP_H / 2];
#pragma unroll
		for (int i = 0; i < MLP_H / 2; i++) dh[i] = 0.f;
#pragma unroll 2
		for (int j = 0; j < MLP_H; j++) {
			const float d = T.dz2[s * MT_LD + j];
#pragma unroll
			for (int i = 0; i < MLP_H / 2; i += 4) {
				const float4 w = *(const float4 *) &T.w2[MLP_H * j + j0 + i];
				dh[i] = fmaf(w.x, d, dh[i]);
				dh[i + 1] = fmaf(w.y, d, dh[i + 1]);
				dh[i + 2] = fmaf(w.z, d, dh[i + 2]);
				dh[i + 3] = fmaf(w.w, d, dh[i + 3]);
			}
		}
#pragma unroll
		for (int i = 0; i < MLP_H / 2; i += 4) {
			const float4 f = *(const float4 *) &T.a1[s * MT_LD + j0 + i];
			*(float4 *) &T.dz1[s * MT_LD + j0 + i] =
			    make_float4(dh[i] * (1.f - f.x * f.x), dh[i + 1] * (1.f - f.y * f.y),
			                dh[i + 2] * (1.f - f.z * f.z), dh[i + 3] * (1.f - f.w * f.w));
		}
		__syncthreads();
		// the tile's gradients
#pragma unroll 2
		for (int k = 0; k < MT; k++) {
			const float4 d0 = *(const float4 *) &T.dz2[k * MT_LD + tj], d1 = *(const float4 *) &T.dz2[k * MT_LD + tj + 4],
			             a = *(const float4 *) &T.a1[k * MT_LD + ti];
			const float d[8] = { d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w };
#pragma unroll
			for (int e = 0; e < 8; e++) {
				g2[e][0] = fmaf(d[e], a.x, g2[e][0]);
				g2[e][1] = fmaf(d[e], a.y, g2[e][1]);
				g2[e][2] = fmaf(d[e], a.z, g2[e][2]);
				g2[e][3] = fmaf(d[e], a.w, g2[e][3]);
			}
		}
		if (half == 0) {
			for (int k = 0; k < MT; k++) {
				const float a = T.a2[k * MT_LD + s];
				gs[0] += T.dz2[k * MT_LD + s];
#pragma unroll
				for (int d = 0; d < 3; d++) gs[1 + d] = fmaf(T.dy[k][d], a, gs[1 + d]);
			}
		} else {
			for (int k = 0; k < MT; k++) {
				const float a = T.dz1[k * MT_LD + s];
				gs[0] += a;
#pragma unroll
				for (int d = 0; d < 3; d++) gs[1 + d] = fmaf(a, T.v[k][d], gs[1 + d]);
			}
		}
		if (tid < 3)
			for (int k = 0; k < MT; k++) g3 += T.dy[k][tid];
	}
	float *slot = slots + (int64_t) blockIdx.x * MLP_NNET;
#pragma unroll
	for (int e = 0; e < 8; e++)
#pragma unroll
		for (int k = 0; k < 4; k++) slot[MLP_W2 + MLP_H * (tj + e) + ti + k] = g2[e][k];
	if (half == 0) {
		slot[MLP_B2 + s] = gs[0];
#pragma unroll
		for (int d = 0; d < 3; d++) slot[MLP_W3 + d * MLP_H + s] = gs[1 + d];
	} else {
		slot[MLP_B1 + s] = gs[0];
#pragma unroll
		for (int d = 0; d < 3; d++) slot[MLP_W1 + 3 * s + d] = gs[1 + d];
	}
	if (tid < 3) slot[MLP_B3 + tid] = g3;
	// half 0 is warps 0 and 1
	loss = warp_sum(loss);
	if (tid == 0 || tid == 32) T.out[0][tid / 32][0] = loss;
	__syncthreads();
	if (tid == 0) loss_slots[blockIdx.x] = T.out[0][0][0] + T.out[0][1][0];
}

// sums of the blocks' slots in FP64, each parameter over four interleaved
// parts that are added in order (deterministic)
__global__ void __launch_bounds__(256)
k_mlp_sum(int nslots, const float *__restrict__ slots, const float *__restrict__ lslots,
          float *grad, float *loss)
{
	__shared__ double part[4][64];
	const int c = threadIdx.x & 63, w = threadIdx.x >> 6, e = blockIdx.x * 64 + c;
	double g = 0;
	if (e < MLP_NNET) {
#pragma unroll 4
		for (int k = w; k < nslots; k += 4) g += (double) slots[(int64_t) k * MLP_NNET + e];
	} else if (e == MLP_NNET) {
		for (int k = w; k < nslots; k += 4) g += (double) lslots[k];
	}
	part[w][c] = g;
	__syncthreads();
	if (w > 0 || e > MLP_NNET) return;
	g = ((part[0][c] + part[1][c]) + part[2][c]) + part[3][c];
	if (e < MLP_NNET) grad[e] = (float) g;
	else *loss = (float) g;
}

// Adam (Kingma & Ba 2015)
__global__ void k_mlp_adam(float *prm, const float *__restrict__ grad, float *m, float *v, float lr,
                           float c1, float c2)
{
	const int e = blockIdx.x * blockDim.x + threadIdx.x;
	if (e >= MLP_NNET) return;
	const float g = grad[e];
	m[e] = 0.9f * m[e] + 0.1f * g;
	v[e] = 0.999f * v[e] + 0.001f * g * g;
	prm[e] -= lr * (m[e] * c1) / (sqrtf(v[e] * c2) + 1e-8f);
}

__global__ void k_mlp_to_bf16(const float *__restrict__ prm, __nv_bfloat16 *out)
{
	const int e = blockIdx.x * blockDim.x + threadIdx.x;
	if (e < MLP_NPARAM) out[e] = __float2bfloat16_rn(prm[e]);
}

// forward only: per-warp sums of the network's squared residual (in units
// of s^2)
__global__ void __launch_bounds__(128)
k_mlp_loss(int64_t n, const float *__restrict__ x, const float *__restrict__ y,
           const float *__restrict__ prm, float *loss_slots)
{
	__shared__ float P[MLP_NPARAM];
	for (int e = threadIdx.x; e < MLP_NPARAM; e += blockDim.x) P[e] = prm[e];
	__syncthreads();
	const int64_t s = blockIdx.x * (int64_t) blockDim.x + threadIdx.x;
	float l = 0.f;
	if (s < n) {
		float v[3], out[3];
		for (int d = 0; d < 3; d++) v[d] = 4.f * x[3 * s + d] - 1.f;
		mlp_net(P, v, out);
		for (int d = 0; d < 3; d++) {
			const float r = out[d] - y[3 * s + d];
			l += r * r;
		}
	}
	l = warp_sum(l);
	if ((threadIdx.x & 31) == 0) loss_slots[s >> 5] = l;
}

// ------------------------------------------------------------ inference

// T(x) for points of the octant by the walk's evaluation (mlp_forward_warp:
// BF16 network on the tensor cores, FP32 elsewhere)
__global__ void __launch_bounds__(128)
k_mlp_eval(int64_t n, const double *__restrict__ x, const __nv_bfloat16 *__restrict__ w,
           const float *__restrict__ f32, double *t)
{
	__shared__ float P[MLP_NPARAM];
	__shared__ uint32_t W2b[MLP_H * MLP_H / 2];
	mlp_load_shared(w, f32, P, W2b);
	__syncthreads();
	const int64_t s = blockIdx.x * (int64_t) blockDim.x + threadIdx.x;
	const bool have = s < n;          // every lane of a warp takes part
	float xs[3] = { 0.f, 0.f, 0.f }, out[3];
	if (have)
		for (int d = 0; d < 3; d++) xs[d] = (float) x[3 * s + d];
	mlp_forward_warp(P, W2b, xs, out);
	if (have)
		for (int d = 0; d < 3; d++) t[3 * s + d] = (double) out[d];
}

// ------------------------------------------------------------ host

// blocks of the gradient kernel, and its slots: two tiles on an SM at a time
static inline int grad_blocks(int64_t n) { return (int) std::min<int64_t>((n + MT - 1) / MT, 2 * 148); }

// a loss slot per warp of the forward kernel (blocks of 128 threads)
static inline int64_t loss_slots(int64_t n) { return ((n + 127) / 128) * 4; }

static int dmalloc(tvg_context *ctx, void **p, size_t b)
{
	if (*p) return TVG_OK;
	TVG_CUDA(ctx, cudaMalloc(p, b));
	return TVG_OK;
}

static void init_params(std::vector<float> &p, uint64_t seed)
{
	// Glorot-uniform weights, zero biases, from a seeded host generator
	uint64_t st = seed * 0x9E3779B97F4A7C15ull + 1;
	auto next = [&]() {
		st ^= st << 13; st ^= st >> 7; st ^= st << 17;
		return (double) (st >> 11) * (1.0 / 9007199254740992.0);
	};
	p.assign(MLP_NPARAM, 0.f);
	const double l1 = sqrt(6.0 / (3 + MLP_H)), l2 = sqrt(6.0 / (2 * MLP_H)), l3 = sqrt(6.0 / (MLP_H + 3));
	for (int e = 0; e < 3 * MLP_H; e++) p[MLP_W1 + e] = (float) ((2 * next() - 1) * l1);
	for (int e = 0; e < MLP_H * MLP_H; e++) p[MLP_W2 + e] = (float) ((2 * next() - 1) * l2);
	for (int e = 0; e < 3 * MLP_H; e++) p[MLP_W3 + e] = (float) ((2 * next() - 1) * l3);
}

// the cubic fit from the summed normal equations (k_mlp_lsq): Cholesky in
// FP64 for the three components; the coefficients are stored as FP32 and s is
// the rms of what they leave (evaluated with the FP32 coefficients)
static int fit_cubic(tvg_context *ctx, const std::vector<double> &part, int64_t ns,
                     std::vector<float> &p0)
{
	const int M = MLP_NMONO;
	double sum[LSQ_NE];
	for (int e = 0; e < LSQ_NE; e++) {
		double t = 0;
		for (int c = 0; c < LSQ_CHUNKS; c++) t += part[(size_t) e * LSQ_CHUNKS + c];
		sum[e] = t;
	}
	double G[M][M], L[M][M] = {};
	int e = 0;
	for (int i = 0; i < M; i++)
		for (int j = i; j < M; j++, e++) G[i][j] = G[j][i] = sum[e];
	for (int i = 0; i < M; i++) {
		for (int j = 0; j <= i; j++) {
			double t = G[i][j];
			for (int k = 0; k < j; k++) t -= L[i][k] * L[j][k];
			if (i == j) {
				if (!(t > 0)) return tvg_fail(ctx, TVG_E_CUDA, "mlp fit: normal equations not positive definite");
				L[i][i] = sqrt(t);
			} else {
				L[i][j] = t / L[j][j];
			}
		}
	}
	double r2 = 0;
	for (int a = 0; a < 3; a++) {
		double z[M], c[M];
		for (int i = 0; i < M; i++) {
			double t = sum[210 + M * a + i];
			for (int k = 0; k < i; k++) t -= L[i][k] * z[k];
			z[i] = t / L[i][i];
		}
		for (int i = M - 1; i >= 0; i--) {
			double t = z[i];
			for (int k = i + 1; k < M; k++) t -= L[k][i] * c[k];
			c[i] = t / L[i][i];
		}
		double cf[M], gc = 0, bc = 0;
		for (int i = 0; i < M; i++) {
			p0[MLP_POLY + M * a + i] = (float) c[i];
			cf[i] = (double) (float) c[i];
		}
		for (int i = 0; i < M; i++) {
			bc += cf[i] * sum[210 + M * a + i];
			for (int j = 0; j < M; j++) gc += cf[i] * G[i][j] * cf[j];
		}
		r2 += sum[270 + a] - 2 * bc + gc;
	}
	const double sc = sqrt(r2 / (3.0 * (double) ns));
	p0[MLP_SCALE] = (sc > 1e-30 && std::isfinite(sc)) ? (float) sc : 1.f;
	return TVG_OK;
}

static int ensure_mlp(tvg_context *ctx)
{
	TVG_CHECK(dmalloc(ctx, (void **) &ctx->mlp_prm, 4 * MLP_NPARAM));
	TVG_CHECK(dmalloc(ctx, (void **) &ctx->mlp_bf16, 2 * MLP_NPARAM));
	return TVG_OK;
}

static int refresh_bf16(tvg_context *ctx)
{
	k_mlp_to_bf16<<<TVG_CNT(ctx, (MLP_NPARAM + 255) / 256), 256, 0, ctx->stream>>>(ctx->mlp_prm, (__nv_bfloat16 *) ctx->mlp_bf16);
	TVG_CUDA(ctx, cudaGetLastError());
	ctx->have_mlp = true;
	ctx->mlp_ok = false;          // until validated
	return TVG_OK;
}

// one gradient of the mean-square loss over n samples (device arrays)
static int grad_batch(tvg_context *ctx, int64_t n, const float *x, const float *y, float *grad,
                      float *loss, float *slots, float *lslots)
{
	const int nb = grad_blocks(n);
	TVG_CUDA(ctx, cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize,
	                                   (int) sizeof(MlpTile)));
	k_mlp_grad<<<TVG_CNT(ctx, nb), MT_THREADS, sizeof(MlpTile), ctx->stream>>>(
	    n, x, y, ctx->mlp_prm, 1.f / (3.f * (float) n), slots, lslots);
	TVG_CUDA(ctx, cudaGetLastError());
	k_mlp_sum<<<TVG_CNT(ctx, (MLP_NNET + 1 + 63) / 64), 256, 0, ctx->stream>>>(nb, slots, lslots, grad, loss);
	TVG_CUDA(ctx, cudaGetLastError());
	return TVG_OK;
}

extern "C" int tvg_ewald_mlp_train(tvg_context *ctx, const tvg_mlp_train_config *cfg,
                                   float *final_loss)
{
	if (!ctx || !cfg) return TVG_E_BADINPUT;
	if (cfg->n_samples < 32 || cfg->batch < 32 || cfg->batch > cfg->n_samples || cfg->steps < 0)
		return tvg_fail(ctx, TVG_E_BADINPUT, "mlp train: need 32 <= batch <= n_samples, steps >= 0");
	TVG_CUDA(ctx, cudaSetDevice(ctx->device));
	cudaStream_t s = ctx->stream;
	TVG_CHECK(ensure_mlp(ctx));
	const int64_t ns = cfg->n_samples, nb = cfg->batch;
	float *x = nullptr, *y = nullptr, *slots = nullptr, *lslots = nullptr, *grad = nullptr,
	      *m = nullptr, *v = nullptr, *loss = nullptr, *yraw_f = nullptr, *part_f = nullptr;
	std::vector<void *> bufs;
	auto alloc = [&](float **p, size_t b) -> int {
		cudaError_t e = cudaMalloc((void **) p, b);
		if (e != cudaSuccess) {
			cudaGetLastError();
			return tvg_fail(ctx, TVG_E_NOMEM, "mlp train: cudaMalloc(%zu) failed", b);
		}
		bufs.push_back(*p);
		return TVG_OK;
	};
	int rc = TVG_OK;
	const int nslots = grad_blocks(nb);
	if ((rc = alloc(&x, 12 * (size_t) ns)) || (rc = alloc(&y, 12 * (size_t) ns))
	    || (rc = alloc(&slots, 4 * (size_t) nslots * MLP_NPARAM)) || (rc = alloc(&lslots, 4 * (size_t) nslots))
	    || (rc = alloc(&grad, 4 * MLP_NPARAM)) || (rc = alloc(&m, 4 * MLP_NPARAM))
	    || (rc = alloc(&v, 4 * MLP_NPARAM)) || (rc = alloc(&loss, 4))
	    || (rc = alloc(&yraw_f, 24 * (size_t) ns)) || (rc = alloc(&part_f, 8 * LSQ_NE * LSQ_CHUNKS))) {
		for (void *b : bufs) cudaFree(b);
		return rc;
	}
	double *yraw = (double *) yraw_f, *part = (double *) part_f;
	auto done = [&](int r) {
		cudaStreamSynchronize(s);
		for (void *b : bufs) cudaFree(b);
		return r;
	};
	k_mlp_data<<<TVG_CNT(ctx, tvg_blocks(ns, 128)), 128, 0, s>>>(ns, cfg->seed, x, yraw);
	if (cudaGetLastError() != cudaSuccess) return done(tvg_fail(ctx, TVG_E_CUDA, "mlp data launch"));
	if (!cfg->resume) {
		// the cubic fit of what the analytic part leaves, then the network's
		// initial weights (a resumed training keeps both)
		std::vector<float> p0;
		init_params(p0, cfg->seed);
		k_mlp_lsq<<<TVG_CNT(ctx, dim3(LSQ_NE, LSQ_CHUNKS)), 128, 0, s>>>(ns, x, yraw, part);
		if (cudaGetLastError() != cudaSuccess) return done(tvg_fail(ctx, TVG_E_CUDA, "mlp lsq launch"));
		std::vector<double> hp((size_t) LSQ_NE * LSQ_CHUNKS);
		if (cudaMemcpyAsync(hp.data(), part, 8 * hp.size(), cudaMemcpyDeviceToHost, s) != cudaSuccess
		    || cudaStreamSynchronize(s) != cudaSuccess)
			return done(tvg_fail(ctx, TVG_E_CUDA, "mlp lsq copy"));
		if ((rc = fit_cubic(ctx, hp, ns, p0))) return done(rc);
		if (cudaMemcpyAsync(ctx->mlp_prm, p0.data(), 4 * MLP_NPARAM, cudaMemcpyHostToDevice, s) != cudaSuccess)
			return done(tvg_fail(ctx, TVG_E_CUDA, "mlp train: upload failed"));
	}
	k_mlp_target<<<TVG_CNT(ctx, tvg_blocks(ns, 128)), 128, 0, s>>>(ns, x, yraw, ctx->mlp_prm, y);
	if (cudaGetLastError() != cudaSuccess) return done(tvg_fail(ctx, TVG_E_CUDA, "mlp target launch"));
	cudaMemsetAsync(m, 0, 4 * MLP_NPARAM, s);
	cudaMemsetAsync(v, 0, 4 * MLP_NPARAM, s);
	const int64_t nbatches = ns / nb;
	for (int st = 0; st < cfg->steps; st++) {
		// cosine decay from lr to lr_final
		const double f = cfg->steps > 1 ? (double) st / (cfg->steps - 1) : 0.0;
		const float lr = (float) (cfg->lr_final + 0.5 * (cfg->lr - cfg->lr_final) * (1.0 + cos(M_PI * f)));
		const int64_t off = (st % nbatches) * nb;
		rc = grad_batch(ctx, nb, x + 3 * off, y + 3 * off, grad, loss, slots, lslots);
		if (rc) return done(rc);
		const float c1 = (float) (1.0 / (1.0 - pow(0.9, st + 1))), c2 = (float) (1.0 / (1.0 - pow(0.999, st + 1)));
		k_mlp_adam<<<TVG_CNT(ctx, (MLP_NNET + 255) / 256), 256, 0, s>>>(ctx->mlp_prm, grad, m, v, lr, c1, c2);
		if (cudaGetLastError() != cudaSuccess) return done(tvg_fail(ctx, TVG_E_CUDA, "mlp adam launch"));
	}
	// mean-square residual of the trained FP32 weights over all samples
	float *lall = nullptr;
	if ((rc = alloc(&lall, 4 * (size_t) loss_slots(ns)))) return done(rc);
	k_mlp_loss<<<TVG_CNT(ctx, tvg_blocks(ns, 128)), 128, 0, s>>>(ns, x, y, ctx->mlp_prm, lall);
	if (cudaGetLastError() != cudaSuccess) return done(tvg_fail(ctx, TVG_E_CUDA, "mlp loss launch"));
	std::vector<float> lw((size_t) loss_slots(ns));
	float sc = 1.f;
	if (cudaMemcpyAsync(lw.data(), lall, 4 * lw.size(), cudaMemcpyDeviceToHost, s) != cudaSuccess
	    || cudaMemcpyAsync(&sc, ctx->mlp_prm + MLP_SCALE, 4, cudaMemcpyDeviceToHost, s) != cudaSuccess)
		return done(tvg_fail(ctx, TVG_E_CUDA, "mlp loss copy"));
	cudaStreamSynchronize(s);
	double tot = 0;
	for (float q : lw) tot += q;
	// in units of T^2
	if (final_loss) *final_loss = (float) (tot / (3.0 * (double) ns) * (double) sc * (double) sc);
	rc = refresh_bf16(ctx);
	return done(rc);
}

extern "C" int tvg_ewald_mlp_weights(tvg_context *ctx, float *params, int32_t set)
{
	if (!ctx || !params) return TVG_E_BADINPUT;
	TVG_CUDA(ctx, cudaSetDevice(ctx->device));
	if (set) {
		TVG_CHECK(ensure_mlp(ctx));
		TVG_CUDA(ctx, cudaMemcpy(ctx->mlp_prm, params, 4 * MLP_NPARAM, cudaMemcpyHostToDevice));
		TVG_CHECK(refresh_bf16(ctx));
		TVG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
		return TVG_OK;
	}
	if (!ctx->have_mlp) return tvg_fail(ctx, TVG_E_STATE, "mlp: no weights");
	TVG_CUDA(ctx, cudaMemcpy(params, ctx->mlp_prm, 4 * MLP_NPARAM, cudaMemcpyDeviceToHost));
	return TVG_OK;
}

// device memory kept between gradient calls (released with the context)
#define MLP_KEEP ((size_t) 64 << 20)

extern "C" int tvg_ewald_mlp_grad(tvg_context *ctx, int64_t n, const float *x, const float *y,
                                  float *grad, float *loss)
{
	if (!ctx || !x || !y || !grad || n < 1) return TVG_E_BADINPUT;
	if (!ctx->have_mlp) return tvg_fail(ctx, TVG_E_STATE, "mlp: no weights");
	TVG_CUDA(ctx, cudaSetDevice(ctx->device));
	cudaStream_t s = ctx->stream;
	// samples, slots, gradient and loss in one block of device memory, kept in
	// the context up to MLP_KEEP bytes (the five allocations and their frees took
	// 1.1 ms of a call with 16,384 samples)
	const int nslots = grad_blocks(n);
	const size_t b_xy = ((size_t) 12 * n + 255) & ~(size_t) 255, b_sl = 4 * (size_t) nslots * MLP_NNET,
	             bytes = 2 * b_xy + b_sl + 4 * (size_t) nslots + 4 * MLP_NPARAM + 4;
	char *ws = (char *) ctx->mlp_ws;
	if (bytes > ctx->mlp_ws_bytes) {
		if (bytes <= MLP_KEEP && ctx->mlp_ws) {
			cudaFree(ctx->mlp_ws);
			ctx->mlp_ws = nullptr;
			ctx->mlp_ws_bytes = 0;
		}
		TVG_CUDA(ctx, cudaMalloc((void **) &ws, bytes));
		if (bytes <= MLP_KEEP) {
			ctx->mlp_ws = ws;
			ctx->mlp_ws_bytes = bytes;
		}
	}
	float *dx = (float *) ws, *dy = (float *) (ws + b_xy), *g = (float *) (ws + 2 * b_xy),
	      *l = g + MLP_NPARAM, *ll = l + 1, *sl = ll + nslots;
	cudaMemsetAsync(g, 0, 4 * MLP_NPARAM + 4, s);      // the fitted entries have no gradient
	cudaMemcpyAsync(dx, x, 12 * (size_t) n, cudaMemcpyHostToDevice, s);
	cudaMemcpyAsync(dy, y, 12 * (size_t) n, cudaMemcpyHostToDevice, s);
	int rc = grad_batch(ctx, n, dx, dy, g, l, sl, ll);
	if (rc == TVG_OK) {
		cudaMemcpyAsync(grad, g, 4 * MLP_NPARAM, cudaMemcpyDeviceToHost, s);
		if (loss) cudaMemcpyAsync(loss, l, 4, cudaMemcpyDeviceToHost, s);
		if (cudaStreamSynchronize(s) != cudaSuccess) rc = tvg_fail(ctx, TVG_E_CUDA, "mlp grad copy");
	}
	if (ws != ctx->mlp_ws) cudaFree(ws);
	return rc;
}

extern "C" int tvg_ewald_mlp_eval(tvg_context *ctx, int64_t n, const double *x, double *t)
{
	if (!ctx || !x || !t || n < 1) return TVG_E_BADINPUT;
	if (!ctx->have_mlp) return tvg_fail(ctx, TVG_E_STATE, "mlp: no weights");
	TVG_CUDA(ctx, cudaSetDevice(ctx->device));
	double *dx, *dt;
	TVG_CUDA(ctx, cudaMalloc((void **) &dx, 24 * (size_t) n));
	TVG_CUDA(ctx, cudaMalloc((void **) &dt, 24 * (size_t) n));
	cudaMemcpyAsync(dx, x, 24 * (size_t) n, cudaMemcpyHostToDevice, ctx->stream);
	k_mlp_eval<<<TVG_CNT(ctx, tvg_blocks(n, 128)), 128, 0, ctx->stream>>>(n, dx, (const __nv_bfloat16 *) ctx->mlp_bf16,
	                                                                      ctx->mlp_prm, dt);
	cudaError_t e = cudaGetLastError();
	if (e == cudaSuccess) e = cudaMemcpyAsync(t, dt, 24 * (size_t) n, cudaMemcpyDeviceToHost, ctx->stream);
	if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
	cudaFree(dx);
	cudaFree(dt);
	if (e != cudaSuccess) return tvg_fail(ctx, TVG_E_CUDA, "mlp eval: %s", cudaGetErrorString(e));
	return TVG_OK;
}

// errors of the walk's evaluation of the model at the 65^3 nodes of the
// exact FP64 table
__global__ void __launch_bounds__(128)
k_mlp_validate(const double *__restrict__ raw, const __nv_bfloat16 *__restrict__ w,
            const float *__restrict__ f32, double *err)
{
	__shared__ float P[MLP_NPARAM];
	__shared__ uint32_t W2b[MLP_H * MLP_H / 2];
	mlp_load_shared(w, f32, P, W2b);
	__syncthreads();
	const int idx = blockIdx.x * blockDim.x + threadIdx.x;
	const bool have = idx < 65 * 65 * 65;      // every lane of a warp takes part
	const int id = have ? idx : 0;
	const int i = id / (65 * 65), j = (id / 65) % 65, k = id % 65;
	const float xs[3] = { 0.5f * i / 64.f, 0.5f * j / 64.f, 0.5f * k / 64.f };
	float out[3];
	mlp_forward_warp(P, W2b, xs, out);
	if (!have) return;
	double e2 = 0;
	for (int d = 0; d < 3; d++) {
		const double r = (double) out[d] - raw[4 * idx + d];
		e2 += r * r;
	}
	err[idx] = sqrt(e2);
}

extern "C" int tvg_ewald_mlp_validate(tvg_context *ctx, double max_allowed, double *max_err,
                                   double *rms_err)
{
	if (!ctx) return TVG_E_BADINPUT;
	if (!ctx->have_mlp) return tvg_fail(ctx, TVG_E_STATE, "mlp: no weights");
	if (!ctx->have_ewald || !ctx->ewald_raw)
		return tvg_fail(ctx, TVG_E_STATE, "mlp validate: exact Ewald table not initialised");
	TVG_CUDA(ctx, cudaSetDevice(ctx->device));
	const int npt = 65 * 65 * 65;
	double *d;
	TVG_CUDA(ctx, cudaMalloc((void **) &d, 8 * (size_t) npt));
	k_mlp_validate<<<TVG_CNT(ctx, (npt + 127) / 128), 128, 0, ctx->stream>>>(ctx->ewald_raw, (const __nv_bfloat16 *) ctx->mlp_bf16,
	                                                                       ctx->mlp_prm, d);
	std::vector<double> h(npt);
	cudaError_t e = cudaGetLastError();
	if (e == cudaSuccess) e = cudaMemcpyAsync(h.data(), d, 8 * (size_t) npt, cudaMemcpyDeviceToHost, ctx->stream);
	if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
	cudaFree(d);
	if (e != cudaSuccess) return tvg_fail(ctx, TVG_E_CUDA, "mlp validate: %s", cudaGetErrorString(e));
	double mx = 0, s2 = 0;
	for (double q : h) { mx = q > mx ? q : mx; s2 += q * q; }
	if (max_err) *max_err = mx;
	if (rms_err) *rms_err = sqrt(s2 / npt);
	ctx->mlp_max_err = mx;
	ctx->mlp_ok = mx <= max_allowed;
	return TVG_OK;
}
