// tvg_forcetest.cu -- Gravity_Forcetest (Gravity/forcetest.c:25-172) on the GPU.
//
// FP64 direct summation over all resident particles for a list of target
// particles, with the reference's softened kernel (h = -41/32 eps, the same
// branch and polynomial as forcetest.c:81-99 and tree_accel.c:362-394) on the
// nearest image. In a periodic box the sum is Ewald-summed, not tabulated:
//
//   a_i = sum_j [ K_soft(d_ij) - G m_j d_ij / r^3 (erf(a r) - 2 a r / sqrt(pi) e^{-a^2 r^2}) ]
//       + (4 G / L^2) sum_{h in half space} h / |h|^2 e^{-pi^2 |h|^2 / (a L)^2}
//                     [cos(k.x_i) S_s(k) - sin(k.x_i) S_c(k)],   k = 2 pi h / L
//
// with d_ij the nearest-image separation (source minus target), S_c + i S_s
// = sum_j m_j e^{i k.x_j} the structure factor, and a L = 12: the real-space
// terms of all further images are below erfc(6) ~ 2e-17 of their Newtonian
// value, and the k-space sum is cut at |h|^2 <= 576 where its terms fall
// below e^{-39} ~ 1e-17. Softened Newton on the nearest image plus this sum is
// exactly what the reference's tree adds up (nearest image + Ewald_Correction,
// whose table is the same sum at a L = 2 with images to |n|, |h| <= 4,
// Gravity/periodic.c:368-411), minus the table's interpolation error.
//
// parts selects the sum: TVG_WALK_GRAVITY alone is the nearest-image softened
// sum (what the gravity walk approximates), with TVG_WALK_EWALD the Ewald sum
// (what gravity + Ewald walks approximate together).
//
// Error statistics compare the resident Grav_Acc (the walk's output) with the
// direct sum: e = |a_tree - a_direct| / |a_direct| per target; rms, 99th
// percentile (nearest rank), mean and max.
//
// Cost: ~75 FP64 instructions for a real-space pair (exp, erfcx, rsqrt). The
// structure factor is a product of matrices: with A = m e^{i (h_x x + h_y y)} for
// the 930 pairs (h_x, h_y) of the half space and the cosines and sines of
// h_z z, h_z = 0 .. 24, four real sums over the sources per (pair, h_z) give
// both signs of h_z, 2 FMA for a source and a wave (one product of phases a
// wave took ~10). For 262,144 sources and
// 1000 targets (ms): structure factor 12.6 -> 2.3, k-space sum of the targets
// 5.2 -> 0.08 (one thread walked all 28,000 waves of a target, a sincospi
// each), real space 3.5 -> 2.2.
#include <math.h>
#include <stdlib.h>

#include <algorithm>
#include <vector>

#include "tvg_internal.cuh"

#define FT_THREADS 128
#define FT_ALPHA_L 12.0
#define FT_HMAX 24
#define FT_NH (FT_HMAX + 1)
#define FT_H2 576

struct FtParams {
	int64_t n, nt, chunk;
	int tpb;                   // targets per block of the real-space sum (a power of two)
	int periodic, ewald;
	double box, half_box, inv_box;
	double G, h2, c16;         // softening: h^2 and 1/(16 h^3), h = -41/32 eps
	double alpha, c2a;         // Ewald alpha and 2 alpha / sqrt(pi)
};

template <typename F>
__global__ void k_ft_gather(int64_t nt, const int64_t *__restrict__ idx, const F *x, const F *y,
                            const F *z, const F *gx, const F *gy, const F *gz, double *tp,
                            double *ta)
{
	const int64_t t = blockIdx.x * (int64_t) blockDim.x + threadIdx.x;
	if (t >= nt) return;
	const int64_t i = idx[t];
	tp[t] = (double) x[i];
	tp[nt + t] = (double) y[i];
	tp[2 * nt + t] = (double) z[i];
	ta[t] = (double) gx[i];
	ta[nt + t] = (double) gy[i];
	ta[2 * nt + t] = (double) gz[i];
}

// Real-space part: the sources of one chunk staged in shared memory tile by
// tile; a thread has one target, and when there are fewer targets than threads
// the spare threads share the targets' sources. Partial sums per chunk, added in
// chunk order later.
template <typename F>
__global__ void __launch_bounds__(FT_THREADS)
k_ft_direct(FtParams p, const F *__restrict__ x, const F *__restrict__ y, const F *__restrict__ z,
            const F *__restrict__ m, const double *__restrict__ tp, double *part)
{
	__shared__ double sx[FT_THREADS], sy[FT_THREADS], sz[FT_THREADS], sm[FT_THREADS];
	const int lt = threadIdx.x & (p.tpb - 1), share = threadIdx.x / p.tpb, nshare = FT_THREADS / p.tpb;
	const int64_t t = blockIdx.x * (int64_t) p.tpb + lt;
	const bool have = t < p.nt;
	const double xi = have ? tp[t] : 0.0, yi = have ? tp[p.nt + t] : 0.0,
	             zi = have ? tp[2 * p.nt + t] : 0.0;
	const int64_t j0 = blockIdx.y * p.chunk, j1 = min(p.n, j0 + p.chunk);
	double ax = 0, ay = 0, az = 0;
	for (int64_t b = j0; b < j1; b += FT_THREADS) {
		const int64_t j = b + threadIdx.x;
		__syncthreads();
		if (j < j1) {
			sx[threadIdx.x] = (double) x[j];
			sy[threadIdx.x] = (double) y[j];
			sz[threadIdx.x] = (double) z[j];
			sm[threadIdx.x] = p.G * (double) m[j];
		}
		__syncthreads();
		const int nb = (int) min((int64_t) FT_THREADS, j1 - b);
		for (int s = share; s < nb; s += nshare) {
			double dx = sx[s] - xi, dy = sy[s] - yi, dz = sz[s] - zi;
			if (p.ewald) {
				// the nearest image by rounding d / L (through 1.5 2^52: three FP64
				// instructions a component). Which of two images half a box away is
				// taken does not matter here: either is erfc(6) of its Newtonian value.
				const double big = 6755399441055744.0;
				dx = fma(-p.box, fma(dx, p.inv_box, big) - big, dx);
				dy = fma(-p.box, fma(dy, p.inv_box, big) - big, dy);
				dz = fma(-p.box, fma(dz, p.inv_box, big) - big, dz);
			} else if (p.periodic) {       // Periodic_Nearest (periodic.c:62-80)
				dx = dx > p.half_box ? dx - p.box : (dx < -p.half_box ? dx + p.box : dx);
				dy = dy > p.half_box ? dy - p.box : (dy < -p.half_box ? dy + p.box : dy);
				dz = dz > p.half_box ? dz - p.box : (dz < -p.half_box ? dz + p.box : dz);
			}
			const double r2 = dx * dx + dy * dy + dz * dz;
			if (!(r2 > 0)) continue;        // forcetest.c:79
			const double ri = rsqrt(r2);
			const double ri3 = ri * ri * ri;
			double fac;
			if (r2 < p.h2) {
				const double u2 = r2 / p.h2;
				fac = (175.0 - u2 * (294.0 - u2 * 135.0)) * p.c16;
				if (p.ewald) {
					const double r = r2 * ri, a = p.alpha * r;
					fac -= ri3 * (erf(a) - p.c2a * r * exp(-a * a));
				}
			} else if (p.ewald) {
				// erfc(a) + c2a r e^{-a^2}, with erfc(a) = e^{-a^2} erfcx(a)
				const double r = r2 * ri, a = p.alpha * r;
				fac = ri3 * (exp(-a * a) * fma(p.c2a, r, erfcx(a)));
			} else {
				fac = ri3;
			}
			fac *= sm[s];
			ax += fac * dx;
			ay += fac * dy;
			az += fac * dz;
		}
	}
	if (nshare > 1) {
		__syncthreads();
		sx[threadIdx.x] = ax;
		sy[threadIdx.x] = ay;
		sz[threadIdx.x] = az;
		__syncthreads();
		for (int q = 1; q < nshare && share == 0; q++) {
			ax += sx[q * p.tpb + lt];
			ay += sy[q * p.tpb + lt];
			az += sz[q * p.tpb + lt];
		}
	}
	if (have && share == 0) {
		double *o = part + (int64_t) blockIdx.y * 3 * p.nt;
		o[t] = ax;
		o[p.nt + t] = ay;
		o[2 * p.nt + t] = az;
	}
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
	return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// e[h] = e^{2 pi i h u}, h = 0..FT_HMAX: the odd and even powers from e^{2 pi
// i u} and its square, two chains of 12 products (round-off ~12 eps)
__device__ __forceinline__ void phases(double two_u, double2 *e)
{
	double2 a;
	sincospi(two_u, &a.y, &a.x);
	const double2 sq = cmul(a, a);
	double2 even = make_double2(1, 0), odd = a;
	e[0] = even;
	e[1] = odd;
#pragma unroll 4
	for (int h = 2; h <= FT_HMAX; h += 2) {
		even = cmul(even, sq);
		e[h] = even;
		if (h + 1 <= FT_HMAX) {
			odd = cmul(odd, sq);
			e[h + 1] = odd;
		}
	}
}

// Structure factor S(k) = sum_j m_j e^{i k.x_j} of one source chunk, for one
// tile of FT_MP pairs (h_x, h_y) and all h_z: the product of the real matrices
// with rows Re A, Im A of each pair and columns cos, sin of each h_z on the FP64
// matrix instruction (8 x 8 x 4). A warp keeps 8 pairs (16 rows) times all
// columns in registers, 9 8-byte shared loads for 14 instructions; with plain
// FMAs on register tiles the shared loads were the bound (3.8 ms at 262,144
// sources). Pairs are sorted by h_x^2 + h_y^2, so a tile's pairs end at about the
// same h_z and it leaves out the columns past it. Output: S for +h_z and -h_z.
#define FT_MP 32
#define FT_KT 24               // sources per stage
#define FT_LDA (2 * FT_MP + 4) // row strides that spread a fragment over the banks
#define FT_LDZ 60
#define FT_NT 7                // column tiles: 2 * 25 columns of 8
struct FtStage {
	double2 ex[FT_KT][FT_NH], ey[FT_KT][FT_NH];
	double z[FT_KT][FT_LDZ];   // cos, sin of h_z = 0, 1, ...
	double a[FT_KT][FT_LDA];   // Re, Im of the pairs
	char4 pairs[FT_MP];
};

__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b)
{
	asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
	    : "+d"(c[0]), "+d"(c[1])
	    : "d"(a), "d"(b));
}

template <typename F>
__global__ void __launch_bounds__(FT_THREADS)
k_ft_structure(int64_t n, int64_t chunk, int np, const char4 *__restrict__ pairs, const F *x,
               const F *y, const F *z, const F *m, double two_over_box, double2 *partS)
{
	extern __shared__ __align__(16) unsigned char ft_smem[];
	FtStage &S = *(FtStage *) ft_smem;
	const int p0 = blockIdx.x * FT_MP;
	// the first pair of the tile reaches the largest h_z
	const int nz = (int) pairs[p0].z + 1, ntile = (nz + 3) / 4;
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, q4 = lane & 3;
	double c[2][FT_NT][2];
#pragma unroll
	for (int i = 0; i < 2; i++)
#pragma unroll
		for (int t = 0; t < FT_NT; t++) c[i][t][0] = c[i][t][1] = 0;
	for (int k = threadIdx.x; k < FT_KT * (FT_LDZ - 2 * FT_NH); k += FT_THREADS)
		S.z[k / (FT_LDZ - 2 * FT_NH)][2 * FT_NH + k % (FT_LDZ - 2 * FT_NH)] = 0;     // padding columns
	if (threadIdx.x < FT_MP) S.pairs[threadIdx.x] = pairs[min(p0 + (int) threadIdx.x, np - 1)];
	const int64_t j0 = blockIdx.y * chunk, j1 = min(n, j0 + chunk);
	for (int64_t b = j0; b < j1; b += FT_KT) {
		__syncthreads();
		if (threadIdx.x < 3 * FT_KT) {
			const int ax = threadIdx.x / FT_KT, k = threadIdx.x % FT_KT;
			const int64_t j = b + k;
			const F *X = ax == 0 ? x : ax == 1 ? y : z;
			phases(j < j1 ? (double) X[j] * two_over_box : 0.0,
			       ax == 0 ? S.ex[k] : ax == 1 ? S.ey[k] : (double2 *) S.z[k]);
		}
		__syncthreads();
		for (int e = threadIdx.x; e < FT_MP * FT_KT; e += FT_THREADS) {
			const int k = e / FT_MP, q = e % FT_MP;
			const int64_t j = b + k;
			const char4 pr = S.pairs[q];
			const double mj = j < j1 ? (double) m[j] : 0.0;
			double2 ey = S.ey[k][abs((int) pr.y)];
			if (pr.y < 0) ey.y = -ey.y;
			double2 v = cmul(S.ex[k][(int) pr.x], ey);
			v.x *= mj;
			v.y *= mj;
			*(double2 *) &S.a[k][2 * q] = v;
		}
		__syncthreads();
#pragma unroll 2
		for (int k = 0; k < FT_KT; k += 4) {
			const double a0 = S.a[k + q4][16 * w + g], a1 = S.a[k + q4][16 * w + 8 + g];
#pragma unroll
			for (int t = 0; t < FT_NT; t++) {
				if (t >= ntile) break;
				const double bz = S.z[k + q4][8 * t + g];
				mma_f64(c[0][t], a0, bz);
				mma_f64(c[1][t], a1, bz);
			}
		}
	}
	// a lane of an even row holds (sum Re cos, sum Re sin) of pair g / 2 and h_z
	// 4 t + q4, the lane four further on (sum Im cos, sum Im sin)
	double2 *o = partS + (int64_t) blockIdx.y * 2 * FT_NH * np;
#pragma unroll
	for (int i = 0; i < 2; i++)
#pragma unroll
		for (int t = 0; t < FT_NT; t++) {
			const double ic = __shfl_xor_sync(0xFFFFFFFFu, c[i][t][0], 4);
			const double is = __shfl_xor_sync(0xFFFFFFFFu, c[i][t][1], 4);
			const int p = p0 + 8 * w + 4 * i + (g >> 1), hz = 4 * t + q4;
			if ((g & 1) || p >= np || hz >= nz) continue;
			o[(2 * hz) * np + p] = make_double2(c[i][t][0] - is, ic + c[i][t][1]);
			o[(2 * hz + 1) * np + p] = make_double2(c[i][t][0] + is, ic - c[i][t][1]);
		}
}

// the chunks' structure factors in order, times the wave's weight
// 4 G / L^2 e^{-pi^2 h^2 / (alpha L)^2} / h^2; 0 outside the half space and past
// the cutoff. Layout [h_z][+, -][pair].
__global__ void k_ft_sum_structure(int np, int nchunks, double fac, const char4 *__restrict__ pairs,
                                   const double2 *__restrict__ partS, double2 *__restrict__ S)
{
	const int e = blockIdx.x * blockDim.x + threadIdx.x;
	if (e >= 2 * FT_NH * np) return;
	const char4 pr = pairs[e % np];
	const int hz = e / np >> 1, minus = (e / np) & 1;
	const int h2 = pr.x * pr.x + pr.y * pr.y + hz * hz;
	double2 a = make_double2(0, 0);
	// one of h and -h: h_x > 0, or h_x = 0 and (h_y > 0, or h_y = 0 and h_z > 0)
	const bool have = hz <= pr.z && h2 <= FT_H2 && h2 > 0 && !(minus && (hz == 0 || (pr.x == 0 && pr.y == 0)));
	if (have) {
		for (int c = 0; c < nchunks; c++) {
			const double2 v = partS[(int64_t) c * 2 * FT_NH * np + e];
			a.x += v.x;
			a.y += v.y;
		}
		const double w = fac * exp(-M_PI * M_PI * h2 / (FT_ALPHA_L * FT_ALPHA_L)) / h2;
		a.x *= w;
		a.y *= w;
	}
	S[e] = a;
}

// A block for TB targets: the partial real-space sums, and the k-space sum with
// the threads dealt over the pairs (every S is read once for TB targets); the
// threads' sums are added in a fixed order.
template <int TB>
__global__ void __launch_bounds__(FT_THREADS)
k_ft_final(int64_t nt, int nchunks, const double *__restrict__ part, const double *__restrict__ tp, int np,
           const char4 *__restrict__ pairs, const double2 *__restrict__ S, double two_over_box, double *acc)
{
	__shared__ double2 e[TB][3][FT_NH];
	__shared__ double red[FT_THREADS / 32][TB][3];
	const int64_t t0 = blockIdx.x * (int64_t) TB;
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	double v[TB][3];
#pragma unroll
	for (int i = 0; i < TB; i++) {
		v[i][0] = v[i][1] = v[i][2] = 0;
		for (int c = threadIdx.x; c < nchunks && t0 + i < nt; c += FT_THREADS) {
			const double *o = part + (int64_t) c * 3 * nt + t0 + i;
			v[i][0] += o[0];
			v[i][1] += o[nt];
			v[i][2] += o[2 * nt];
		}
	}
	if (np > 0) {
		for (int k = threadIdx.x; k < TB * 3 * FT_NH; k += FT_THREADS) {
			const int i = k / (3 * FT_NH), d = (k / FT_NH) % 3, h = k % FT_NH;
			const double u = t0 + i < nt ? tp[d * nt + t0 + i] : 0.0;
			double2 q;
			sincospi(u * two_over_box * h, &q.y, &q.x);
			e[i][d][h] = q;
		}
		__syncthreads();
		for (int q = threadIdx.x; q < np; q += FT_THREADS) {
			const char4 pr = pairs[q];
			double2 a[TB];
			double sum[TB], sz[TB];
#pragma unroll
			for (int i = 0; i < TB; i++) {
				double2 ey = e[i][1][abs((int) pr.y)];
				if (pr.y < 0) ey.y = -ey.y;
				a[i] = cmul(e[i][0][(int) pr.x], ey);
				sum[i] = sz[i] = 0;
			}
			for (int hz = 0; hz <= pr.z; hz++) {
				const double2 sp = S[(2 * hz) * np + q], sn = S[(2 * hz + 1) * np + q];
#pragma unroll
				for (int i = 0; i < TB; i++) {
					const double2 c = e[i][2][hz];
					const double rc = a[i].x * c.x, is = a[i].y * c.y, ic = a[i].y * c.x, rs = a[i].x * c.y;
					const double vp = (rc - is) * sp.y - (ic + rs) * sp.x;
					const double vn = (rc + is) * sn.y - (ic - rs) * sn.x;
					sum[i] += vp + vn;
					sz[i] += (double) hz * (vp - vn);
				}
			}
#pragma unroll
			for (int i = 0; i < TB; i++) {
				v[i][0] += sum[i] * pr.x;
				v[i][1] += sum[i] * pr.y;
				v[i][2] += sz[i];
			}
		}
	}
#pragma unroll
	for (int i = 0; i < TB; i++)
#pragma unroll
		for (int d = 0; d < 3; d++) {
#pragma unroll
			for (int o = 16; o; o >>= 1) v[i][d] += __shfl_xor_sync(0xFFFFFFFFu, v[i][d], o);
			if (lane == 0) red[w][i][d] = v[i][d];
		}
	__syncthreads();
	if (threadIdx.x < TB * 3) {
		const int i = threadIdx.x / 3, d = threadIdx.x % 3;
		double s = 0;
		for (int k = 0; k < FT_THREADS / 32; k++) s += red[k][i][d];
		if (t0 + i < nt) acc[d * nt + t0 + i] = s;
	}
}

namespace {

// The call's device memory: one block, the context's own up to FT_KEEP bytes
// (kept for the next call, released with the context), else one that is freed
// when the call ends.
#define FT_KEEP ((size_t) 64 << 20)
struct Scratch {
	char *p = nullptr;
	size_t used = 0, size = 0;
	bool own = false;
	~Scratch() { if (own) cudaFree(p); }
	int get(tvg_context *ctx, size_t bytes)
	{
		size = bytes;
		if (bytes <= ctx->ft_bytes) {
			p = (char *) ctx->ft_ws;
			return TVG_OK;
		}
		if (bytes <= FT_KEEP && ctx->ft_ws) {
			cudaFree(ctx->ft_ws);
			ctx->ft_ws = nullptr;
			ctx->ft_bytes = 0;
		}
		cudaError_t e = cudaMalloc((void **) &p, bytes);
		if (e != cudaSuccess) {
			cudaGetLastError();
			p = nullptr;
			return tvg_fail(ctx, TVG_E_NOMEM, "forcetest: cudaMalloc(%zu) failed: %s", bytes,
			                cudaGetErrorString(e));
		}
		if (bytes <= FT_KEEP) {
			ctx->ft_ws = p;
			ctx->ft_bytes = bytes;
		} else {
			own = true;
		}
		return TVG_OK;
	}
	static size_t round(size_t b) { return (b + 255) & ~(size_t) 255; }
	template <typename T> T *take(size_t count)
	{
		T *q = (T *) (p + used);
		used += round(sizeof(T) * count);
		return q;
	}
};

// the pairs (h_x, h_y) of the half space, h_x^2 + h_y^2 ascending, and the
// largest |h_z| each has
const std::vector<char4> &wave_pairs()
{
	static const std::vector<char4> table = [] {
		std::vector<char4> v;
		for (int hx = 0; hx <= FT_HMAX; hx++)
			for (int hy = hx ? -FT_HMAX : 0; hy <= FT_HMAX; hy++) {
				const int r2 = FT_H2 - hx * hx - hy * hy;
				if (r2 < 0) continue;
				int hz = 0;
				while ((hz + 1) * (hz + 1) <= r2) hz++;
				v.push_back(make_char4((signed char) hx, (signed char) hy, (signed char) hz, 0));
			}
		std::stable_sort(v.begin(), v.end(), [](const char4 &a, const char4 &b) {
			return a.x * a.x + a.y * a.y < b.x * b.x + b.y * b.y;
		});
		return v;
	}();
	return table;
}

}   // namespace

template <typename F>
static int forcetest_typed(tvg_context *ctx, bool ewald, int64_t nt, const int64_t *targets,
                           double *acc_direct, double *acc_tree, double *err)
{
	const int64_t n = ctx->n;
	cudaStream_t s = ctx->stream;
	const tvg_config &cf = ctx->cfg;
	int nsm = 148;
	TVG_CUDA(ctx, cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, ctx->device));
	// real space: 16 blocks of FT_THREADS for every SM, whatever the number of
	// targets (a chunk has at least one tile of sources)
	int tpb = FT_THREADS;
	while (tpb > 1 && tpb / 2 >= nt) tpb /= 2;
	const int64_t tblocks = (nt + tpb - 1) / tpb;
	int64_t dchunks = std::max<int64_t>(1, 16 * (int64_t) nsm / tblocks);
	dchunks = std::max<int64_t>(1, std::min(dchunks, std::min<int64_t>((n + FT_THREADS - 1) / FT_THREADS, 1024)));
	// structure factor: 12 blocks for every SM (5 resident; the tiles differ in
	// work. 4 / 8 / 12 / 24 blocks: 4.84 / 4.80 / 4.62 / 5.14 ms for the call at
	// 262,144 sources and 1000 targets)
	const std::vector<char4> &pairs = wave_pairs();
	const int np = ewald ? (int) pairs.size() : 0, ntile = (np + FT_MP - 1) / FT_MP;
	int64_t schunks = ewald ? std::max(1, 12 * nsm / ntile) : 0;
	if (ewald) schunks = std::max<int64_t>(1, std::min(schunks, (n + FT_KT - 1) / FT_KT));
	const size_t nS = (size_t) 2 * FT_NH * np;
	Scratch W;
	TVG_CHECK(W.get(ctx, Scratch::round(8 * (size_t) nt) + 3 * Scratch::round(24 * (size_t) nt)
	                         + Scratch::round(24 * (size_t) nt * dchunks) + Scratch::round(4 * (size_t) np)
	                         + Scratch::round(16 * nS) + Scratch::round(16 * nS * schunks)));
	int64_t *d_idx = W.take<int64_t>(nt);
	double *tp = W.take<double>(3 * nt), *ta = W.take<double>(3 * nt), *acc = W.take<double>(3 * nt),
	       *part = W.take<double>(3 * nt * dchunks);
	char4 *d_pairs = W.take<char4>(np);
	double2 *d_S = W.take<double2>(nS), *partS = W.take<double2>(nS * schunks);
	TVG_CUDA(ctx, cudaMemcpyAsync(d_idx, targets, 8 * (size_t) nt, cudaMemcpyHostToDevice, s));
	const F *X = (const F *) ctx->f[FS_POS0], *Y = (const F *) ctx->f[FS_POS1],
	        *Z = (const F *) ctx->f[FS_POS2], *M = (const F *) ctx->f[FS_MASS];
	k_ft_gather<F><<<TVG_CNT(ctx, tvg_blocks(nt, 256)), 256, 0, s>>>(
	    nt, d_idx, X, Y, Z, (const F *) ctx->f[FS_GACC0], (const F *) ctx->f[FS_GACC1],
	    (const F *) ctx->f[FS_GACC2], tp, ta);
	TVG_CUDA(ctx, cudaGetLastError());

	FtParams p;
	p.n = n;
	p.nt = nt;
	p.chunk = (n + dchunks - 1) / dchunks;
	p.tpb = tpb;
	p.periodic = cf.periodic;      // nearest image
	p.ewald = ewald;
	p.box = cf.periodic ? cf.boxsize : 0.0;
	p.half_box = 0.5 * p.box;
	p.inv_box = cf.periodic ? 1.0 / cf.boxsize : 0.0;
	p.G = cf.gravity;
	const double h = -41.0 / 32.0 * cf.softening;      // tree_build.c:136
	p.h2 = h * h;
	p.c16 = 1.0 / (16.0 * h * h * h);
	p.alpha = ewald ? FT_ALPHA_L / cf.boxsize : 0.0;
	p.c2a = 2.0 * p.alpha / sqrt(M_PI);
	const dim3 gd((unsigned) tblocks, (unsigned) dchunks);
	k_ft_direct<F><<<TVG_CNT(ctx, gd), FT_THREADS, 0, s>>>(p, X, Y, Z, M, tp, part);
	TVG_CUDA(ctx, cudaGetLastError());

	const double two_over_box = ewald ? 2.0 / cf.boxsize : 0.0;
	if (ewald) {
		TVG_CUDA(ctx, cudaMemcpyAsync(d_pairs, pairs.data(), sizeof(char4) * np, cudaMemcpyHostToDevice, s));
		const size_t smem = sizeof(FtStage);
		TVG_CUDA(ctx, cudaFuncSetAttribute(k_ft_structure<F>, cudaFuncAttributeMaxDynamicSharedMemorySize,
		                                   (int) smem));
		const dim3 gs(ntile, (unsigned) schunks);
		k_ft_structure<F><<<TVG_CNT(ctx, gs), FT_THREADS, smem, s>>>(
		    n, (n + schunks - 1) / schunks, np, d_pairs, X, Y, Z, M, two_over_box, partS);
		TVG_CUDA(ctx, cudaGetLastError());
		k_ft_sum_structure<<<TVG_CNT(ctx, tvg_blocks((int64_t) nS, 256)), 256, 0, s>>>(
		    np, (int) schunks, 4.0 * cf.gravity / (cf.boxsize * cf.boxsize), d_pairs, partS, d_S);
		TVG_CUDA(ctx, cudaGetLastError());
	}
	if (nt >= 4 * nsm)
		k_ft_final<4><<<TVG_CNT(ctx, tvg_blocks(nt, 4)), FT_THREADS, 0, s>>>(nt, (int) dchunks, part, tp, np,
		                                                                     d_pairs, d_S, two_over_box, acc);
	else
		k_ft_final<1><<<TVG_CNT(ctx, (unsigned) nt), FT_THREADS, 0, s>>>(nt, (int) dchunks, part, tp, np,
		                                                                 d_pairs, d_S, two_over_box, acc);
	TVG_CUDA(ctx, cudaGetLastError());
	std::vector<double> ad(3 * nt), at(3 * nt);
	TVG_CUDA(ctx, cudaMemcpyAsync(ad.data(), acc, 24 * (size_t) nt, cudaMemcpyDeviceToHost, s));
	TVG_CUDA(ctx, cudaMemcpyAsync(at.data(), ta, 24 * (size_t) nt, cudaMemcpyDeviceToHost, s));
	TVG_CUDA(ctx, cudaStreamSynchronize(s));
	if (acc_direct) memcpy(acc_direct, ad.data(), 24 * (size_t) nt);
	if (acc_tree) memcpy(acc_tree, at.data(), 24 * (size_t) nt);
	if (err) {
		std::vector<double> e(nt);
		double sum2 = 0, sum = 0, mx = 0;
		for (int64_t t = 0; t < nt; t++) {
			double d2 = 0, a2 = 0;
			for (int k = 0; k < 3; k++) {
				const double d = at[k * nt + t] - ad[k * nt + t];
				d2 += d * d;
				a2 += ad[k * nt + t] * ad[k * nt + t];
			}
			e[t] = a2 > 0 ? sqrt(d2 / a2) : 0.0;
			sum2 += e[t] * e[t];
			sum += e[t];
			mx = std::max(mx, e[t]);
		}
		std::sort(e.begin(), e.end());
		const int64_t r99 = (int64_t) ceil(0.99 * (double) nt) - 1;
		err[0] = sqrt(sum2 / nt);
		err[1] = e[std::max<int64_t>(r99, 0)];
		err[2] = sum / nt;
		err[3] = mx;
	}
	return TVG_OK;
}

extern "C" int tvg_forcetest(tvg_context *ctx, uint32_t parts, int64_t n_targets,
                             const int64_t *targets, double *acc_direct, double *acc_tree,
                             double *err)
{
	if (!ctx) return TVG_E_BADINPUT;
	if (!(parts & TVG_WALK_GRAVITY))
		return tvg_fail(ctx, TVG_E_BADINPUT, "forcetest: parts must include TVG_WALK_GRAVITY");
	if ((parts & TVG_WALK_EWALD) && !ctx->cfg.periodic)
		return tvg_fail(ctx, TVG_E_STATE, "forcetest: Ewald part needs a periodic box");
	const bool ewald = (parts & TVG_WALK_EWALD) != 0;
	if (n_targets <= 0 || n_targets > TVG_FORCETEST_MAX_TARGETS || !targets)
		return tvg_fail(ctx, TVG_E_BADINPUT, "forcetest: n_targets must be in 1..%d",
		                TVG_FORCETEST_MAX_TARGETS);
	for (int64_t t = 0; t < n_targets; t++)
		if (targets[t] < 0 || targets[t] >= ctx->n)
			return tvg_fail(ctx, TVG_E_BADINPUT, "forcetest: target %lld out of range",
			                (long long) targets[t]);
	TVG_CUDA(ctx, cudaSetDevice(ctx->device));
	if (ctx->cfg.float_bytes == 4)
		return forcetest_typed<float>(ctx, ewald, n_targets, targets, acc_direct, acc_tree, err);
	return forcetest_typed<double>(ctx, ewald, n_targets, targets, acc_direct, acc_tree, err);
}
