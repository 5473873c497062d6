// tvg_ewald.cu -- Ewald correction tables on the GPU (Gravity_Periodic_Init,
// Gravity/periodic.c:180-300).
//
// compute_ewald_force / compute_ewald_potential (Gravity/periodic.c:352-461):
// the force of the periodic lattice minus the nearest image, after Hernquist,
// Bouchet & Suto (1991, eqs. 2.14-2.16), alpha = 2, real-space images and
// k-space vectors with |n|, |h| <= 4 per axis, evaluated in FP64 at the
// (64+1)^3 points of the folded octant [0, L/2]^3 (box units), one thread per
// point and axis-sum. Stored as Float, then divided by Boxsize^2 (force) and
// Boxsize (potential) as the reference does after loading (periodic.c:215-228).
// The raw FP64 values stay on the device as the training target and max-error
// reference for validating the learned correction.
#include "tvg_internal.cuh"
#include "tvg_ewald_sum.cuh"

#define N_EWALD 64
#define N_EW1 (N_EWALD + 1)

template <typename F>
__global__ void k_ewald_table(double box, F *fx, F *fy, F *fz, F *fp, double *raw)
{
	const int idx = blockIdx.x * blockDim.x + threadIdx.x;
	if (idx >= N_EW1 * N_EW1 * N_EW1) return;
	const int i = idx / (N_EW1 * N_EW1), j = (idx / N_EW1) % N_EW1, k = idx % N_EW1;
	const double x[3] = { (0.5 * i) / N_EWALD, (0.5 * j) / N_EWALD, (0.5 * k) / N_EWALD };
	double f[3], pot;
	ewald_point(x, f, &pot);
	raw[4 * idx + 0] = f[0];
	raw[4 * idx + 1] = f[1];
	raw[4 * idx + 2] = f[2];
	raw[4 * idx + 3] = pot;
	// Float storage, then the division after the load (periodic.c:215-228)
	fx[idx] = (F) ((double) (F) f[0] / (box * box));
	fy[idx] = (F) ((double) (F) f[1] / (box * box));
	fz[idx] = (F) ((double) (F) f[2] / (box * box));
	fp[idx] = (F) ((double) (F) pot / box);
}

int tvg_impl_ewald_init(tvg_context *ctx)
{
	const size_t npt = (size_t) N_EW1 * N_EW1 * N_EW1;
	for (int t = 0; t < 4; t++)
		if (!ctx->ewald_f[t]) TVG_CUDA(ctx, cudaMalloc(&ctx->ewald_f[t], tvg_fsize(ctx) * npt));
	if (!ctx->ewald_raw) TVG_CUDA(ctx, cudaMalloc((void **) &ctx->ewald_raw, 4 * 8 * npt));
	const unsigned nb = tvg_blocks((int64_t) npt, 128);
	if (ctx->cfg.float_bytes == 4)
		k_ewald_table<float><<<TVG_CNT(ctx, nb), 128, 0, ctx->stream>>>(
		    ctx->cfg.boxsize, (float *) ctx->ewald_f[0], (float *) ctx->ewald_f[1],
		    (float *) ctx->ewald_f[2], (float *) ctx->ewald_f[3], ctx->ewald_raw);
	else
		k_ewald_table<double><<<TVG_CNT(ctx, nb), 128, 0, ctx->stream>>>(
		    ctx->cfg.boxsize, (double *) ctx->ewald_f[0], (double *) ctx->ewald_f[1],
		    (double *) ctx->ewald_f[2], (double *) ctx->ewald_f[3], ctx->ewald_raw);
	TVG_CUDA(ctx, cudaGetLastError());
	TVG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
	return TVG_OK;
}

// Lattice force T (the periodic lattice minus the image at the origin, box
// units, unit G m) on the grid of half the node spacing of a table of `nodes`
// nodes per axis, with two ghost points beyond each end (the analytic
// continuation beyond L/2 and below 0). Evaluated for sorted coordinates only; the
// others are their permutations.
__host__ __device__ __forceinline__ int fine_points(int nodes) { return 2 * (nodes - 1) + 1 + 4; }

__global__ void k_ewald_fine(int nodes, double *fine)
{
	const int nf = fine_points(nodes);
	const int idx = blockIdx.x * blockDim.x + threadIdx.x;
	if (idx >= nf * nf * nf) return;
	const int i[3] = { idx / (nf * nf), (idx / nf) % nf, idx % nf };
	if (i[0] > i[1] || i[1] > i[2]) return;
	const double d = 1.0 / (4.0 * (nodes - 1));
	const double x[3] = { (i[0] - 2) * d, (i[1] - 2) * d, (i[2] - 2) * d };
	double f[3], pot;
	ewald_point(x, f, &pot);
	const int perm[6][3] = { { 0, 1, 2 }, { 0, 2, 1 }, { 1, 0, 2 }, { 1, 2, 0 }, { 2, 0, 1 }, { 2, 1, 0 } };
	for (int q = 0; q < 6; q++) {
		const int *o = perm[q];
		double *w = fine + 3 * (((int64_t) i[o[0]] * nf + i[o[1]]) * nf + i[o[2]]);
		for (int a = 0; a < 3; a++) w[a] = f[o[a]];
	}
}

// Finite differences of T_a at fine point (ci, cj, ck), in node units (fine
// spacing 1/2): fourth-order central differences for the first and pure second
// derivatives, second-order ones for the mixed and third derivatives (small
// correction terms); FP64 round-off enters as ~1e-16 / delta^3, below 1e-8.
struct FineDiff {
	const double *fine;
	int nf, c[3];
	__device__ double f(int a, int di, int dj, int dk) const
	{
		return fine[3 * (((int64_t) (c[0] + di) * nf + (c[1] + dj)) * nf + (c[2] + dk)) + a];
	}
	__device__ double g(int a, int b, int s) const
	{
		return b == 0 ? f(a, s, 0, 0) : b == 1 ? f(a, 0, s, 0) : f(a, 0, 0, s);
	}
	__device__ double g2(int a, int b, int sb, int e, int se) const
	{
		int d[3] = { 0, 0, 0 };
		d[b] += sb;
		d[e] += se;
		return f(a, d[0], d[1], d[2]);
	}
	__device__ double d1(int a, int b) const
	{
		return (-g(a, b, 2) + 8 * g(a, b, 1) - 8 * g(a, b, -1) + g(a, b, -2)) / 6;
	}
	__device__ double d2(int a, int b) const
	{
		return (-g(a, b, 2) + 16 * g(a, b, 1) - 30 * f(a, 0, 0, 0) + 16 * g(a, b, -1) - g(a, b, -2)) / 3;
	}
	__device__ double d2m(int a, int b, int e) const
	{
		return g2(a, b, 1, e, 1) - g2(a, b, 1, e, -1) - g2(a, b, -1, e, 1) + g2(a, b, -1, e, -1);
	}
	__device__ double d3(int a, int b) const
	{
		return (g(a, b, 2) - 2 * g(a, b, 1) + 2 * g(a, b, -1) - g(a, b, -2)) * 4;
	}
	// d3 T_a / db db de: the difference along e of the second differences along b
	__device__ double d3m(int a, int b, int e) const
	{
		const double up = g2(a, b, 1, e, 1) - 2 * g2(a, b, 0, e, 1) + g2(a, b, -1, e, 1);
		const double dn = g2(a, b, 1, e, -1) - 2 * g2(a, b, 0, e, -1) + g2(a, b, -1, e, -1);
		return (up - dn) * 4;
	}
	__device__ double d3xyz(int a) const
	{
		double s3 = 0;
		for (int sx = -1; sx <= 1; sx += 2)
			for (int sy = -1; sy <= 1; sy += 2)
				for (int sz = -1; sz <= 1; sz += 2) s3 += sx * sy * sz * f(a, sx, sy, sz);
		return s3;
	}
};

__device__ __forceinline__ FineDiff fine_diff(const double *fine, int nodes, int idx)
{
	return { fine, fine_points(nodes),
	         { 2 * (idx / (nodes * nodes)) + 2, 2 * ((idx / nodes) % nodes) + 2, 2 * (idx % nodes) + 2 } };
}

// Taylor table of the group form: at each node x = i / (2 (N - 1)) (box units, i
// = 0..N-1 per axis, N = TVG_TAYLOR_NODES) of the octant, T and its first three
// derivatives, the k-th with respect to the node coordinate u = 2 (N - 1) x. T is a
// gradient, so the derivative tensors are symmetric: each entry is the mean of
// the finite differences that approximate it. Record of 32 floats:
//   Tx Ty Tz, dT xx yy zz xy xz yz, d2T xxx xxy xxz xyy xyz xzz yyy yyz yzz zzz,
//   d3T xxxx yyyy zzzz xxyy xxzz yyzz xxxy xxxz xyyy yyyz xxyz xyyz (xyzz, xzzz and yzzz
//   from the zero trace), 0.
// A lookup expands T about the nearest node (|du| <= 1/2 per axis): T to third
// order, dT to second, d2T to first. With 33 nodes (spacing 1/64), at 400 random
// points of the octant against direct lattice sums: the value within 4.8e-7 of |T|,
// the gradient within 4.2e-5 of its largest component (the derivatives component by
// component, 60 floats: 5.8e-7 and 4.2e-5).
__global__ void k_ewald_taylor(const double *__restrict__ fine, float *tay)
{
	const int idx = blockIdx.x * blockDim.x + threadIdx.x;
	if (idx >= TVG_TAYLOR_NODES * TVG_TAYLOR_NODES * TVG_TAYLOR_NODES) return;
	const FineDiff F = fine_diff(fine, TVG_TAYLOR_NODES, idx);
	// the components that approximate d2T_bbe (b != e) and d3T_bbbe, d3T_bbee
	auto c2 = [&](int b, int e) { return (F.d2(e, b) + 2 * F.d2m(b, b, e)) / 3; };
	auto d31 = [&](int b, int e) { return (F.d3(e, b) + 3 * F.d3m(b, b, e)) / 4; };
	auto d22 = [&](int b, int e) { return 0.5 * (F.d3m(b, e, b) + F.d3m(e, b, e)); };
	auto d211 = [&](int b, int e, int f) {
		return (F.d3m(f, b, e) + F.d3m(e, b, f) + 2 * F.d3xyz(b)) / 4;
	};
	const double v[32] = {
		F.f(0, 0, 0, 0), F.f(1, 0, 0, 0), F.f(2, 0, 0, 0),
		F.d1(0, 0), F.d1(1, 1), F.d1(2, 2), 0.5 * (F.d1(0, 1) + F.d1(1, 0)), 0.5 * (F.d1(0, 2) + F.d1(2, 0)),
		0.5 * (F.d1(1, 2) + F.d1(2, 1)),
		F.d2(0, 0), c2(0, 1), c2(0, 2), c2(1, 0), (F.d2m(0, 1, 2) + F.d2m(1, 0, 2) + F.d2m(2, 0, 1)) / 3,
		c2(2, 0), F.d2(1, 1), c2(1, 2), c2(2, 1), F.d2(2, 2),
		F.d3(0, 0), F.d3(1, 1), F.d3(2, 2), d22(0, 1), d22(0, 2), d22(1, 2), d31(0, 1), d31(0, 2), d31(1, 0),
		d31(1, 2), d211(0, 1, 2), d211(1, 0, 2), 0
	};
	float *r = tay + 32 * (int64_t) idx;
	for (int q = 0; q < 32; q++) r[q] = (float) v[q];
}

// Table of the lattice force for single points (the group form's wide groups,
// k_ewald_wide): at each node x = i / (2 (N - 1)), N = TVG_WIDE_NODES, of the
// octant, T and its first three derivatives in node units. T is a gradient and
// its divergence is 4 pi, so the derivative tensors are symmetric and
// traceless (but for that constant) and 24 numbers hold them all: 96 bytes,
// three 32-byte loads, where a tricubic lookup of a 68^3 value table took 64
// loads. Record:
//   Tx Ty Tz, d2 phi xx yy xy xz yz -> dT;
//   d2T as xxx xxy xxz xyy xyz yyy yyz, d3T as xxxx;
//   xxxy xxxz yyyy xyyy yyyz xxyy xxyz xyyz.
// With 41 nodes the third-order expansion about the nearest node is within
// 5e-8 rms of direct lattice sums over the octant (tricubic: 8e-8, and 1.2e-7
// with its FP32 sums).
__global__ void k_ewald_wide_table(const double *__restrict__ fine, float *tab)
{
	const int idx = blockIdx.x * blockDim.x + threadIdx.x;
	if (idx >= TVG_WIDE_NODES * TVG_WIDE_NODES * TVG_WIDE_NODES) return;
	const FineDiff F = fine_diff(fine, TVG_WIDE_NODES, idx);
	const double v[24] = {
		F.f(0, 0, 0, 0), F.f(1, 0, 0, 0), F.f(2, 0, 0, 0), F.d1(0, 0), F.d1(1, 1), F.d1(0, 1), F.d1(0, 2),
		F.d1(1, 2),
		F.d2(0, 0), F.d2(1, 0), F.d2(2, 0), F.d2(0, 1), (F.d2m(0, 1, 2) + F.d2m(1, 0, 2) + F.d2m(2, 0, 1)) / 3,
		F.d2(1, 1), F.d2(2, 1), F.d3(0, 0),
		F.d3(1, 0), F.d3(2, 0), F.d3(1, 1), F.d3(0, 1), F.d3(2, 1), 0.5 * (F.d3m(1, 0, 1) + F.d3m(0, 1, 0)),
		F.d3m(2, 0, 1), F.d3m(2, 1, 0)
	};
	float *r = tab + 24 * (int64_t) idx;
	for (int q = 0; q < 24; q++) r[q] = (float) v[q];
}

// one of the two tables: the fine grid, then the records
static int make_table(tvg_context *ctx, int nodes, size_t record, void (*kernel)(const double *, float *), float **out)
{
	const int nf = fine_points(nodes);
	const int64_t n = (int64_t) nodes * nodes * nodes, nfine = (int64_t) nf * nf * nf;
	double *fine = nullptr;
	float *tab = nullptr;
	TVG_CHECK(tvg_alloc(ctx, (void **) &fine, 24 * (size_t) nfine));
	const int rc = tvg_alloc(ctx, (void **) &tab, record * (size_t) n);
	if (rc != TVG_OK) {
		cudaFree(fine);
		return rc;
	}
	k_ewald_fine<<<TVG_CNT(ctx, tvg_blocks(nfine, 128)), 128, 0, ctx->stream>>>(nodes, fine);
	kernel<<<TVG_CNT(ctx, tvg_blocks(n, 128)), 128, 0, ctx->stream>>>(fine, tab);
	cudaError_t e = cudaGetLastError();
	const cudaError_t es = cudaStreamSynchronize(ctx->stream);
	if (e == cudaSuccess) e = es;
	cudaFree(fine);
	if (e != cudaSuccess) {
		cudaFree(tab);
		return tvg_fail(ctx, TVG_E_CUDA, "ewald taylor table: %s", cudaGetErrorString(e));
	}
	*out = tab;
	return TVG_OK;
}

int tvg_impl_ewald_taylor(tvg_context *ctx)
{
	return make_table(ctx, TVG_TAYLOR_NODES, 128, k_ewald_taylor, &ctx->ewald_taylor);
}

int tvg_impl_ewald_wide(tvg_context *ctx)
{
	return make_table(ctx, TVG_WIDE_NODES, 96, k_ewald_wide_table, &ctx->ewald_wide);
}

// raw Float tables (box units) -> device tables, as after
// read_ewald_correction_table + the division at periodic.c:215-228
template <typename F>
__global__ void k_ewald_from_raw(double box, const F *rx, const F *ry, const F *rz, const F *rp,
                                 F *fx, F *fy, F *fz, F *fp, double *raw)
{
	const int idx = blockIdx.x * blockDim.x + threadIdx.x;
	if (idx >= N_EW1 * N_EW1 * N_EW1) return;
	raw[4 * idx + 0] = (double) rx[idx];
	raw[4 * idx + 1] = (double) ry[idx];
	raw[4 * idx + 2] = (double) rz[idx];
	raw[4 * idx + 3] = (double) rp[idx];
	fx[idx] = (F) ((double) rx[idx] / (box * box));
	fy[idx] = (F) ((double) ry[idx] / (box * box));
	fz[idx] = (F) ((double) rz[idx] / (box * box));
	fp[idx] = (F) ((double) rp[idx] / box);
}

extern "C" int tvg_upload_ewald_table(tvg_context *ctx, const void *fx, const void *fy,
                                      const void *fz, const void *fp)
{
	if (!ctx || !fx || !fy || !fz || !fp) return TVG_E_BADINPUT;
	if (!ctx->cfg.periodic) return tvg_fail(ctx, TVG_E_STATE, "upload_ewald_table: not periodic");
	TVG_CUDA(ctx, cudaSetDevice(ctx->device));
	const size_t npt = (size_t) N_EW1 * N_EW1 * N_EW1, b = tvg_fsize(ctx) * npt;
	for (int t = 0; t < 4; t++)
		if (!ctx->ewald_f[t]) TVG_CUDA(ctx, cudaMalloc(&ctx->ewald_f[t], b));
	if (!ctx->ewald_raw) TVG_CUDA(ctx, cudaMalloc((void **) &ctx->ewald_raw, 4 * 8 * npt));
	void *tmp = nullptr;
	TVG_CUDA(ctx, cudaMalloc(&tmp, 4 * b));
	const void *src[4] = { fx, fy, fz, fp };
	for (int t = 0; t < 4; t++)
		TVG_CUDA(ctx, cudaMemcpyAsync((char *) tmp + t * b, src[t], b, cudaMemcpyHostToDevice, ctx->stream));
	const unsigned nb = tvg_blocks((int64_t) npt, 256);
	if (ctx->cfg.float_bytes == 4) {
		const float *r = (const float *) tmp;
		k_ewald_from_raw<float><<<TVG_CNT(ctx, nb), 256, 0, ctx->stream>>>(
		    ctx->cfg.boxsize, r, r + npt, r + 2 * npt, r + 3 * npt, (float *) ctx->ewald_f[0],
		    (float *) ctx->ewald_f[1], (float *) ctx->ewald_f[2], (float *) ctx->ewald_f[3], ctx->ewald_raw);
	} else {
		const double *r = (const double *) tmp;
		k_ewald_from_raw<double><<<TVG_CNT(ctx, nb), 256, 0, ctx->stream>>>(
		    ctx->cfg.boxsize, r, r + npt, r + 2 * npt, r + 3 * npt, (double *) ctx->ewald_f[0],
		    (double *) ctx->ewald_f[1], (double *) ctx->ewald_f[2], (double *) ctx->ewald_f[3],
		    ctx->ewald_raw);
	}
	cudaError_t e = cudaGetLastError();
	if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
	cudaFree(tmp);
	TVG_CUDA(ctx, e);
	ctx->have_ewald = true;
	return TVG_OK;
}

template <typename F>
__global__ void k_ewald_raw_float(const double *raw, F *out, int comp, int n)
{
	int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) out[i] = (F) raw[4 * i + comp];
}

extern "C" int tvg_download_ewald_table(tvg_context *ctx, void *fx, void *fy, void *fz, void *fp)
{
	if (!ctx) return TVG_E_BADINPUT;
	if (!ctx->have_ewald) return tvg_fail(ctx, TVG_E_STATE, "ewald table not initialised");
	TVG_CUDA(ctx, cudaSetDevice(ctx->device));
	const int npt = N_EW1 * N_EW1 * N_EW1;
	void *outs[4] = { fx, fy, fz, fp };
	void *tmp = nullptr;
	TVG_CUDA(ctx, cudaMalloc(&tmp, tvg_fsize(ctx) * npt));
	for (int c = 0; c < 4; c++) {
		if (!outs[c]) continue;
		if (ctx->cfg.float_bytes == 4)
			k_ewald_raw_float<float><<<TVG_CNT(ctx, tvg_blocks(npt, 256)), 256, 0, ctx->stream>>>(ctx->ewald_raw,
			                                                                          (float *) tmp, c, npt);
		else
			k_ewald_raw_float<double><<<TVG_CNT(ctx, tvg_blocks(npt, 256)), 256, 0, ctx->stream>>>(ctx->ewald_raw,
			                                                                           (double *) tmp, c, npt);
		cudaError_t e = cudaMemcpyAsync(outs[c], tmp, tvg_fsize(ctx) * npt, cudaMemcpyDeviceToHost,
		                                ctx->stream);
		if (e != cudaSuccess) { cudaFree(tmp); TVG_CUDA(ctx, e); }
	}
	cudaError_t e = cudaStreamSynchronize(ctx->stream);
	cudaFree(tmp);
	TVG_CUDA(ctx, e);
	return TVG_OK;
}
