// tvg_walk_plain.cu -- the plain GPU form: the reference tree walk of each
// active particle, in the host's Float width.
//
// Gravity part: Gravity_Tree_Acceleration (tree_accel.c:32-394) -- every top
// node (interact_with_topnode), then the subtree walk with the BH or the
// relative criterion over the DNext skip pointers; softened monopole
// interact() with the Dehnen K1 kernel at h = -41/32 eps (tree_build.c:136,
// kept as in the reference: the sign flip of quirk Q1).
// Ewald part: Gravity_Tree_Periodic (tree_periodic.c:23-450) with the
// trilinear table lookup of Ewald_Correction (Gravity/periodic.c:35-113).
// With TVG_CFG_POTENTIAL (GRAVITY_POTENTIAL) the potential of interact()
// (tree_accel.c:362-389) and of interact_with_ewald_cube (tree_periodic.c:
// 425-447, Ewald_Potential at Gravity/periodic.c:115-170) are summed in double
// as the reference's Recv.Grav_Potential.
// This file is compiled with -fmad=false: every expression rounds in the
// reference's order (float/double promotion as in C), so given the same tree
// the accelerations are the reference's bit for bit.
//
// What bounds it is the arithmetic that replays the reference (per
// interaction an IEEE square root and reciprocal, three conversions to double
// and three double additions). So whatever does not depend on the target is
// computed once per walk and the same values are read back: a particle is one
// packed load (position and the rounded G m), a node one record (the left side
// of its test, its thresholds), a comparison of a float with a double
// threshold is one of floats (the threshold rounded so that every float
// compares alike), and the Ewald tables are interleaved so that one load
// brings the components of a corner (FP32: of two).
//
// A warp's 32 targets walk the tree together: every lane keeps the node it
// goes to next, the warp visits the smallest of them, and the lanes that are
// there take part. A lane so makes exactly its own walk in its own order, while
// nodes and the particles of opened bundles are loaded once for the warp and
// no lane waits while another is inside a bundle. Targets far apart in the
// particle order share few nodes: a warp of such targets (a sparse active
// list) walks lane by lane instead (PLAIN_SPREAD).
//
// Box of 50^3, FP32, gravity and Ewald part: 101 and 123 ms with a walk per
// thread over the reference's records, 33 and 76 ms so (the Ewald part then
// bound by L1: 82 % of its wavefronts, one per lane and 32-byte table load).
// Halo of 30,011, FP64 with the potential: 6.4 ms before, 2.8 ms.
#include "tvg_internal.cuh"
#include "tvg_inv_sqrt.cuh"

template <typename F> struct WNode {
	int32_t DNext;
	uint32_t Bitfield;
	int32_t DUp;
	int32_t Npart;
	F Pos[3];
	F Mass;
	F CoM[3];
	F Dp[3];
};

struct PlainParams {
	double gravity, domain_size, boxsize, open_bh, open_rel;
	double eps, eps2, eps3, box2grid;
	int periodic, use_bh, vsize, ntop, fix_small;
};

// four Floats in one (FP32) or two (FP64) 16-byte loads
template <typename F> struct __align__(16) Float4 {
	F x, y, z, w;
};

// What the tests of a node need, in the walk's criterion (48 B in FP32).
template <typename F> struct __align__(16) PNode {
	F com[3];
	F gm;          // (F) (G Mass), interact()
	F crit;        // nsize^2 (Barnes-Hut) or Mass nsize nsize
	F pos[3];
	F lim;         // |x| < 0.6 nsize for every Float x: |x| < lim
	F dl;          // Ewald, |x| > (box - nsize) / 2: |x| > dl; -1 when nsize > 0.2 box
	int32_t dnext, npart;
};

template <typename F> struct PlainCtx {
	const F *x, *y, *z, *m;
	const Float4<F> *src;      // x, y, z and (F) (G m)
	const F *ew;               // the Ewald tables, interleaved (k_plain_ewald)
	const tvg_topnode *top;
	const WNode<F> *tree;
	const PNode<float> *pn;    // FP32 builds: the node records
	F boxhalf;
	F eps2;                    // r2 < eps^2 for every Float r2: r2 < eps2
	F r2min, r2max;            // FP32: range of the branch-free root (inv_sqrt)
	F box;                     // FP32: boxsize as a float, 0 if it is not one
	int64_t tree_cap;          // node capacity: the walks never read past it
	int64_t n;                 // particles
	PlainParams p;
};

// the smallest float >= v (x < v for a float x exactly when x < it), and the
// largest <= v (x > v exactly when x > it)
template <typename F> __device__ __forceinline__ F up(double v);
template <> __device__ __forceinline__ float up<float>(double v) { return __double2float_ru(v); }
template <> __device__ __forceinline__ double up<double>(double v) { return v; }
template <typename F> __device__ __forceinline__ F down(double v);
template <> __device__ __forceinline__ float down<float>(double v) { return __double2float_rd(v); }
template <> __device__ __forceinline__ double down<double>(double v) { return v; }

template <typename F> __device__ __forceinline__ F fabs_(F v);
template <> __device__ __forceinline__ float fabs_<float>(float v) { return fabsf(v); }
template <> __device__ __forceinline__ double fabs_<double>(double v) { return fabs(v); }

template <typename F> __device__ __forceinline__ F fsqrt(F v);
template <> __device__ __forceinline__ float fsqrt<float>(float v) { return __fsqrt_rn(v); }
template <> __device__ __forceinline__ double fsqrt<double>(double v) { return __dsqrt_rn(v); }

template <typename F>
__device__ __forceinline__ void nearest(const PlainCtx<F> &c, F dr[3])
{
	if (!c.p.periodic) return;
	// one test for the common case of no wrap
	if (!(fabs_(dr[0]) > c.boxhalf || fabs_(dr[1]) > c.boxhalf || fabs_(dr[2]) > c.boxhalf)) return;
#pragma unroll
	for (int k = 0; k < 3; k++) {
		if (dr[k] > c.boxhalf) dr[k] = (F) (dr[k] - c.p.boxsize);
		else if (dr[k] < -c.boxhalf) dr[k] = (F) (dr[k] + c.p.boxsize);
	}
}

// domain_size / (1UL << level): the reference's division by an exact power of
// two (a negative level, a top node between a tree kick and its drift, shifts
// to 0: infinite, so opened)
__device__ __forceinline__ double level_size(double domain_size, int lvl)
{
	return domain_size * __hiloint2double(lvl < 0 ? 0x7FF00000 : (1023 - lvl) << 20, 0);
}

template <typename F>
__device__ __forceinline__ PNode<F> make_node(const PlainParams &p, const WNode<F> &nd)
{
	const F nsz = (F) level_size(p.domain_size, (int) (nd.Bitfield & 0x3F));
	PNode<F> r;
	r.com[0] = nd.CoM[0];
	r.com[1] = nd.CoM[1];
	r.com[2] = nd.CoM[2];
	r.gm = (F) (p.gravity * nd.Mass);
	r.crit = p.use_bh ? nsz * nsz : nd.Mass * nsz * nsz;
	r.pos[0] = nd.Pos[0];
	r.pos[1] = nd.Pos[1];
	r.pos[2] = nd.Pos[2];
	r.lim = up<F>(0.6 * nsz);
	r.dl = nsz > 0.2 * p.boxsize ? (F) -1 : down<F>(0.5 * (p.boxsize - nsz));
	r.dnext = nd.DNext;
	r.npart = nd.Npart;
	return r;
}

__device__ __forceinline__ PNode<float> load_node(const PlainCtx<float> &c, int node)
{
	const float4 *q = (const float4 *) (c.pn + node);
	const float4 a = __ldg(q), b = __ldg(q + 1), d = __ldg(q + 2);
	PNode<float> r;
	r.com[0] = a.x; r.com[1] = a.y; r.com[2] = a.z; r.gm = a.w;
	r.crit = b.x; r.pos[0] = b.y; r.pos[1] = b.z; r.pos[2] = b.w;
	r.lim = d.x; r.dl = d.y;
	r.dnext = __float_as_int(d.z);
	r.npart = __float_as_int(d.w);
	return r;
}

// FP64: the few products cost less than a second copy of the tree
__device__ __forceinline__ PNode<double> load_node(const PlainCtx<double> &c, int node)
{
	return make_node<double>(c.p, c.tree[node]);
}

__device__ __forceinline__ Float4<float> load4(const Float4<float> *p)
{
	const float4 v = __ldg((const float4 *) p);
	return { v.x, v.y, v.z, v.w };
}

__device__ __forceinline__ Float4<double> load4(const Float4<double> *p)
{
	const double2 a = __ldg((const double2 *) p), b = __ldg((const double2 *) p + 1);
	return { a.x, a.y, b.x, b.y };
}

// A target's sums, kept alike by the S lanes that share it (Lanes<S>)
struct Sums {
	double a[3];
	double pot;
	int32_t n;                 // interactions counted by every lane of the target
	int32_t own;               // interactions of this lane's particles
};

// one interaction's addends (adding +0 leaves a sum as it is: none is ever -0)
template <typename F> struct Term {
	F x, y, z, pot;
};

// S consecutive lanes walk for one target: a node is tested by all of them, the
// particles of a bundle are dealt out in turn, and the addends are exchanged
// so that every lane sums all of them in particle order.
template <int S> struct Lanes {
	unsigned mask;             // the target's lanes
	int sub;                   // this lane's place among them
	int base;                  // the first of them
};

template <int S> __device__ __forceinline__ Lanes<S> lanes()
{
	const int lane = threadIdx.x & 31;
	Lanes<S> l;
	l.sub = lane & (S - 1);
	l.base = lane & ~(S - 1);
	l.mask = S == 32 ? 0xFFFFFFFFu : ((1u << (S & 31)) - 1u) << l.base;
	return l;
}

template <bool POT, int S, typename F>
__device__ __forceinline__ void add_terms(const Lanes<S> &l, const Term<F> &t, Sums &s)
{
	if (S == 1) {
		s.a[0] += t.x;
		s.a[1] += t.y;
		s.a[2] += t.z;
		if (POT) s.pot += t.pot;
		return;
	}
#pragma unroll
	for (int q = 0; q < S; q++) {
		s.a[0] += __shfl_sync(l.mask, t.x, l.base + q);
		s.a[1] += __shfl_sync(l.mask, t.y, l.base + q);
		s.a[2] += __shfl_sync(l.mask, t.z, l.base + q);
		if (POT) s.pot += __shfl_sync(l.mask, t.pot, l.base + q);
	}
}

// interact(), tree_accel.c:362-394; with POT the potential fac_pot, whose
// inner polynomial is the reference's (u2 * (175 - (u2 * 147 - u2 * 45))
// - 105) / (32 Epsilon). gm is the reference's (Float) (Const.Gravity * mass)
template <bool POT, typename F>
__device__ __forceinline__ Term<F> interact(const PlainCtx<F> &c, F gm, const F dr[3], F r2)
{
	F fac = gm;
	F fac_pot = gm;
	if (r2 < c.eps2) {
		F u2 = (F) (r2 / c.p.eps2);
		F poly = (F) 175 - u2 * ((F) 294 - u2 * (F) 135);
		fac = (F) (fac * (poly / (16 * c.p.eps3)));
		if (POT) {
			const F ppoly = u2 * ((F) 175 - (u2 * (F) 147 - u2 * (F) 45)) - (F) 105;
			fac_pot = (F) (fac_pot * (ppoly / (32 * c.p.eps)));
		}
	} else {
		F r_inv = (F) 1 / fsqrt<F>(r2);
		fac *= r_inv * r_inv * r_inv;
		if (POT) fac_pot *= r_inv;
	}
	return { fac * dr[0], fac * dr[1], fac * dr[2], fac_pot };
}

// a node's (or top node's) interaction, made by all lanes of the target
template <bool POT, typename F>
__device__ __forceinline__ void add_node(const PlainCtx<F> &c, F gm, const F dr[3], F r2, Sums &s)
{
	const Term<F> t = interact<POT>(c, gm, dr, r2);
	s.a[0] += t.x;
	s.a[1] += t.y;
	s.a[2] += t.z;
	if (POT) s.pot += t.pot;
	s.n++;
}

// particle jp for a target at sp; have: the bundle has it
template <bool POT, typename F>
__device__ __forceinline__ Term<F> particle(const PlainCtx<F> &c, bool have, int64_t jp, const F sp[3], Sums &s)
{
	Term<F> t = { 0, 0, 0, 0 };
	if (have) {
		const Float4<F> q = load4(c.src + jp);
		F d[3] = { q.x - sp[0], q.y - sp[1], q.z - sp[2] };
		nearest(c, d);
		const F r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
		if (r2 != 0) {
			t = interact<POT>(c, q.w, d, r2);
			s.own++;
		}
	}
	return t;
}

// U particles of a bundle, FP32. Without a special one (all
// r2 inside [r2min, r2max], so neither softened nor the target itself) they run
// straight-line, U independent chains that meet in the ordered double sums; a
// bundle that reaches the half-box plane wraps its separations by the same
// subtraction in float (exact when the box side is a float). Everything else
// takes the general form.
template <bool POT, int U>
__device__ __forceinline__ void gravity_run(const PlainCtx<float> &c, int64_t jp, const float sp[3], Sums &s)
{
	float d[U][3], gm[U], r2[U];
	Term<float> t[U];
	bool wrap = false, plain = true;
#pragma unroll
	for (int u = 0; u < U; u++) {
		const Float4<float> q = load4(c.src + jp + u);
		d[u][0] = q.x - sp[0];
		d[u][1] = q.y - sp[1];
		d[u][2] = q.z - sp[2];
		gm[u] = q.w;
		if (fmaxf(fmaxf(fabsf(d[u][0]), fabsf(d[u][1])), fabsf(d[u][2])) > c.boxhalf) wrap = true;
	}
	if (c.p.periodic && wrap) {
		if (c.box == 0) plain = false;
#pragma unroll
		for (int u = 0; u < U; u++)
#pragma unroll
			for (int k = 0; k < 3; k++)
				if (fabsf(d[u][k]) > c.boxhalf) d[u][k] = d[u][k] - copysignf(c.box, d[u][k]);
	}
#pragma unroll
	for (int u = 0; u < U; u++) {
		r2[u] = d[u][0] * d[u][0] + d[u][1] * d[u][1] + d[u][2] * d[u][2];
		if (!(r2[u] >= c.r2min && r2[u] <= c.r2max)) plain = false;
	}
	if (plain) {
#pragma unroll
		for (int u = 0; u < U; u++) {
			const float ri = inv_sqrt(r2[u]);
			const float fac = gm[u] * (ri * ri * ri);
			t[u] = { fac * d[u][0], fac * d[u][1], fac * d[u][2], gm[u] * ri };
		}
		s.own += U;
	} else {
#pragma unroll
		for (int u = 0; u < U; u++) t[u] = particle<POT>(c, true, jp + u, sp, s);
	}
#pragma unroll
	for (int u = 0; u < U; u++) add_terms<POT>(Lanes<1>(), t[u], s);
}

// the particles [f, f + np) of a bundle
template <bool POT, int S>
__device__ __forceinline__ void gravity_bundle(const PlainCtx<float> &c, const Lanes<S> &l, int64_t f, int np,
                                               const float sp[3], Sums &s)
{
	static_assert(S == 1, "FP32 gravity takes one lane per target");
	constexpr int U = 4;
	int k = 0;
	for (; k + U <= np; k += U) gravity_run<POT, U>(c, f + k, sp, s);
	for (; k < np; k++) gravity_run<POT, 1>(c, f + k, sp, s);
}

template <bool POT, int S>
__device__ __forceinline__ void gravity_bundle(const PlainCtx<double> &c, const Lanes<S> &l, int64_t f, int np,
                                               const double sp[3], Sums &s)
{
	for (int k = 0; k < np; k += S) {
		const Term<double> t = particle<POT>(c, k + l.sub < np, f + k + l.sub, sp, s);
		if (S > 1) __syncwarp(l.mask);
		add_terms<POT>(l, t, s);
	}
}

// The particles of an opened small top node: the reference takes them from
// Target on, a running node count, which passes the last particle when nodes
// outnumber particles (bundles of one). add(f, np) takes those that exist;
// past(d) says whether a particle at the origin, d from the target, counts: what
// lies past the last particle is such a particle without mass, which adds nothing
// but its count.
template <typename F, typename Add, typename Past>
__device__ __forceinline__ void small_top(const PlainCtx<F> &c, const tvg_topnode &t, const F sp[3], Sums &s,
                                          Add add, Past past)
{
	const int64_t f = c.p.fix_small ? t.first_part : t.target;
	const int np = (int) max((int64_t) 0, min((int64_t) t.npart, c.n - f));
	add(f, np);
	if (np < t.npart) {
		F d[3] = { -sp[0], -sp[1], -sp[2] };
		nearest(c, d);
		if (past(d)) s.n += t.npart - np;
	}
}

// one node of a subtree for one target; returns the node it goes to next
// (INT_MAX at the subtree's terminator, DNext = 0; a valid tree ends every
// subtree with one well inside the capacity, the bound keeps a damaged one in
// memory)
template <bool POT, int S, typename F>
__device__ __forceinline__ int gravity_node(const PlainCtx<F> &c, const Lanes<S> &l, int node, const F sp[3],
                                            F fac, Sums &s)
{
	if (node >= c.tree_cap) return INT32_MAX;
	const PNode<F> nd = load_node(c, node);
	if (nd.dnext == 0) return INT32_MAX;
	if (nd.dnext < 0) {
		gravity_bundle<POT, S>(c, l, -(int64_t) nd.dnext - 1, nd.npart, sp, s);
		return node + 1;
	}
	F d[3] = { nd.com[0] - sp[0], nd.com[1] - sp[1], nd.com[2] - sp[2] };
	nearest(c, d);
	const F r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
	if (c.p.use_bh) {
		if ((double) nd.crit > r2 * c.p.open_bh) return node + 1;
	} else {
		if (nd.crit > r2 * r2 * fac) return node + 1;
		F ds[3] = { nd.pos[0] - sp[0], nd.pos[1] - sp[1], nd.pos[2] - sp[2] };
		nearest(c, ds);
		if (fabs_(ds[0]) < nd.lim && fabs_(ds[1]) < nd.lim && fabs_(ds[2]) < nd.lim) return node + 1;
	}
	add_node<POT>(c, nd.gm, d, r2, s);
	return node + nd.dnext;
}

// COH: the lanes of the warp together (all of them call; have: this lane has a
// target), else each target on its own
template <bool POT, bool COH, int S, typename F>
__device__ void walk_gravity(const PlainCtx<F> &c, const Lanes<S> &l, bool have, const F sp[3], F sacc, Sums &s)
{
	const F fac = (F) (sacc / c.p.gravity * c.p.open_rel);
	for (int j = 0; j < c.p.ntop; j++) {
		const tvg_topnode &t = c.top[j];
		const F nsize = (F) level_size(c.p.domain_size, t.level);
		bool open = have;
		if (have) {
			F dr[3] = { (F) t.pos[0] - sp[0], (F) t.pos[1] - sp[1], (F) t.pos[2] - sp[2] };
			const bool inside = fabs((double) dr[0]) < 0.6 * nsize && fabs((double) dr[1]) < 0.6 * nsize
			                 && fabs((double) dr[2]) < 0.6 * nsize;
			if (!inside) {
				dr[0] = (F) t.com[0] - sp[0];
				dr[1] = (F) t.com[1] - sp[1];
				dr[2] = (F) t.com[2] - sp[2];
				nearest(c, dr);
				const F r2 = dr[0] * dr[0] + dr[1] * dr[1] + dr[2] * dr[2];
				const F nmass = (F) t.mass;
				if (c.p.use_bh) open = (double) (nsize * nsize) > r2 * c.p.open_bh;
				else open = nmass * nsize * nsize > r2 * r2 * fac;
				if (!open) add_node<POT>(c, (F) (c.p.gravity * nmass), dr, r2, s);
			}
		}
		if (t.npart <= c.p.vsize) {
			if (open)
				small_top(
				    c, t, sp, s, [&](int64_t f, int np) { gravity_bundle<POT, S>(c, l, f, np, sp, s); },
				    [](const F d[3]) { return d[0] * d[0] + d[1] * d[1] + d[2] * d[2] != 0; });
			if (COH) __syncwarp();
			continue;
		}
		const int start = t.target;
		int cur = open ? start : INT32_MAX;
		if (COH) {
			for (;;) {
				const int node = __reduce_min_sync(0xFFFFFFFFu, cur);
				if (node == INT32_MAX) break;
				if (cur == node) cur = gravity_node<POT, S>(c, l, node, sp, fac, s);
				__syncwarp();
			}
		} else {
			while (cur != INT32_MAX) cur = gravity_node<POT, S>(c, l, cur, sp, fac, s);
		}
	}
}

// The corners of an Ewald table cell, fx, fy, fz and the potential of each, in
// the order (i, j, k), (i, j, k + 1), (i, j + 1, k), ... of the reference's
// sums. The lanes of a warp sit in as many cells, so the gather is bound by
// the cache lines it touches, not by its bytes: FP32 entries hold two
// neighbours along k (8 floats, one 32-byte load; 4 loads a cell instead of
// 24), FP64 entries one corner (4 doubles, one 32-byte load).
__device__ __forceinline__ void load_cell(const float *ew, int i, int j, int k, Float4<float> t[8])
{
#pragma unroll
	for (int q = 0; q < 4; q++) {
		const float *e = ew + 8 * (((i + (q >> 1)) * 65 + j + (q & 1)) * 64 + k);
		Float4<float> &a = t[2 * q], &b = t[2 * q + 1];
		asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
		    : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
		    : "l"(e));
	}
}

__device__ __forceinline__ void load_cell(const double *ew, int i, int j, int k, Float4<double> t[8])
{
#pragma unroll
	for (int q = 0; q < 8; q++) {
		const double *e = ew + 4 * (((i + (q >> 2)) * 65 + j + ((q >> 1) & 1)) * 65 + k + (q & 1));
		asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
		    : "=d"(t[q].x), "=d"(t[q].y), "=d"(t[q].z), "=d"(t[q].w)
		    : "l"(e));
	}
}

// Ewald_Correction, Gravity/periodic.c:35-113, and with POT Ewald_Potential,
// Gravity/periodic.c:115-170: trilinear in double on the potential table at
// |dr|, the result stored as Float
template <bool POT, typename F>
__device__ __forceinline__ void ewald_corr(const PlainCtx<F> &c, const F dr[3], F f[3], F &fpot)
{
	const F dx = fabs_(dr[0]), dy = fabs_(dr[1]), dz = fabs_(dr[2]);
	const double ud = dx * c.p.box2grid, vd = dy * c.p.box2grid, wd = dz * c.p.box2grid;
	F u = (F) ud, v = (F) vd, w = (F) wd;
	const int i = min((int) u, 63), j = min((int) v, 63), k = min((int) w, 63);
	Float4<F> t[8];
	load_cell(c.ew, i, j, k, t);
	u -= i; v -= j; w -= k;
	const F one = 1;
	const F wt[8] = { (one - u) * (one - v) * (one - w), (one - u) * (one - v) * w,
	                  (one - u) * v * (one - w), (one - u) * v * w,
	                  u * (one - v) * (one - w), u * (one - v) * w,
	                  u * v * (one - w), u * v * w };
	f[0] = wt[0] * t[0].x + wt[1] * t[1].x + wt[2] * t[2].x + wt[3] * t[3].x + wt[4] * t[4].x + wt[5] * t[5].x
	     + wt[6] * t[6].x + wt[7] * t[7].x;
	f[1] = wt[0] * t[0].y + wt[1] * t[1].y + wt[2] * t[2].y + wt[3] * t[3].y + wt[4] * t[4].y + wt[5] * t[5].y
	     + wt[6] * t[6].y + wt[7] * t[7].y;
	f[2] = wt[0] * t[0].z + wt[1] * t[1].z + wt[2] * t[2].z + wt[3] * t[3].z + wt[4] * t[4].z + wt[5] * t[5].z
	     + wt[6] * t[6].z + wt[7] * t[7].z;
	// the sign rule: -1 for dr >= 0, else +1
	if (!(dr[0] < 0)) f[0] = -f[0];
	if (!(dr[1] < 0)) f[1] = -f[1];
	if (!(dr[2] < 0)) f[2] = -f[2];
	if (POT) {
		// the cell from the double coordinate, which may round up into the next
		// one as a Float
		const int ip = min((int) ud, 63), jp = min((int) vd, 63), kp = min((int) wd, 63);
		if (ip != i || jp != j || kp != k) load_cell(c.ew, ip, jp, kp, t);
		const double a = ud - ip, b = vd - jp, g = wd - kp;
		const double wp[8] = { (1 - a) * (1 - b) * (1 - g), (1 - a) * (1 - b) * g,
		                       (1 - a) * b * (1 - g), (1 - a) * b * g,
		                       a * (1 - b) * (1 - g), a * (1 - b) * g,
		                       a * b * (1 - g), a * b * g };
		fpot = (F) (wp[0] * t[0].w + wp[1] * t[1].w + wp[2] * t[2].w + wp[3] * t[3].w + wp[4] * t[4].w
		            + wp[5] * t[5].w + wp[6] * t[6].w + wp[7] * t[7].w);
	}
}

// interact_with_ewald_cube, tree_periodic.c:425-447 (its addends in double)
template <bool POT, typename F>
__device__ __forceinline__ Term<double> ewald_cube(const PlainCtx<F> &c, const F dr[3], F mass)
{
	F r[3], rpot = 0;
	ewald_corr<POT>(c, dr, r, rpot);
	const double gm = c.p.gravity * mass;
	return { gm * r[0], gm * r[1], gm * r[2], POT ? gm * rpot : 0.0 };
}

template <bool POT, typename F>
__device__ __forceinline__ void ewald_add_node(const PlainCtx<F> &c, const F dr[3], F mass, Sums &s)
{
	const Term<double> t = ewald_cube<POT>(c, dr, mass);
	s.a[0] += t.x;
	s.a[1] += t.y;
	s.a[2] += t.z;
	if (POT) s.pot += t.pot;
	s.n++;
}

// U particles of a bundle a lane, jp + S u, U lookups in flight; have: the
// bundle has them (U = 1)
template <bool POT, int S, int U, typename F>
__device__ __forceinline__ void ewald_run(const PlainCtx<F> &c, const Lanes<S> &l, bool have, int64_t jp,
                                          const F sp[3], Sums &s)
{
	F d[U][3], m[U];
	Term<double> t[U];
#pragma unroll
	for (int u = 0; u < U; u++) {
		t[u] = { 0, 0, 0, 0 };
		if (!have) continue;
		const Float4<F> q = load4(c.src + jp + S * u);
		m[u] = c.m[jp + S * u];
		d[u][0] = q.x - sp[0];
		d[u][1] = q.y - sp[1];
		d[u][2] = q.z - sp[2];
		nearest(c, d[u]);
	}
	if (have) {
#pragma unroll
		for (int u = 0; u < U; u++) t[u] = ewald_cube<POT>(c, d[u], m[u]);
#pragma unroll
		for (int u = 0; u < U; u++) {
			if (d[u][0] != 0 && d[u][1] != 0 && d[u][2] != 0) s.own++;
			else t[u] = { 0, 0, 0, 0 };
		}
	}
	if (S > 1) __syncwarp(l.mask);
#pragma unroll
	for (int u = 0; u < U; u++) add_terms<POT>(l, t[u], s);
}

template <bool POT, int S, typename F>
__device__ __forceinline__ void ewald_bundle(const PlainCtx<F> &c, const Lanes<S> &l, int64_t f, int np,
                                             const F sp[3], Sums &s)
{
	constexpr int U = sizeof(F) == 4 && S == 1 ? 2 : 1;
	int k = 0;
	if (U > 1)
		for (; k + S * U <= np; k += S * U) ewald_run<POT, S, U>(c, l, true, f + k + l.sub, sp, s);
	for (; k < np; k += S) ewald_run<POT, S, 1>(c, l, k + l.sub < np, f + k + l.sub, sp, s);
}

template <bool POT, int S, typename F>
__device__ __forceinline__ int ewald_node(const PlainCtx<F> &c, const Lanes<S> &l, int node, int end,
                                          const F sp[3], F fac, double bh2, Sums &s)
{
	if (node >= end || node >= c.tree_cap) return INT32_MAX;
	const PNode<F> nd = load_node(c, node);
	if (nd.dnext < 0) {
		ewald_bundle<POT, S>(c, l, -(int64_t) nd.dnext - 1, nd.npart, sp, s);
		return node + 1;
	}
	F d[3] = { nd.com[0] - sp[0], nd.com[1] - sp[1], nd.com[2] - sp[2] };
	nearest(c, d);
	const F rr = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
	F ds[3] = { nd.pos[0] - sp[0], nd.pos[1] - sp[1], nd.pos[2] - sp[2] };
	bool wo = c.p.use_bh ? (double) nd.crit > rr * bh2 : nd.crit > rr * rr * fac;
	if (!wo && fabs_(ds[0]) < nd.lim && fabs_(ds[1]) < nd.lim && fabs_(ds[2]) < nd.lim) wo = true;
	if (wo) {
		nearest(c, ds);
		if (fabs_(ds[0]) > nd.dl || fabs_(ds[1]) > nd.dl || fabs_(ds[2]) > nd.dl) return node + 1;
	}
	ewald_add_node<POT>(c, d, c.tree[node].Mass, s);
	return node + nd.dnext;
}

template <bool POT, bool COH, int S, typename F>
__device__ void walk_ewald(const PlainCtx<F> &c, const Lanes<S> &l, bool have, const F sp[3], F sacc, Sums &s)
{
	const double box = c.p.boxsize;
	const F fac = (F) (sacc / c.p.gravity * c.p.open_rel);
	const double bh2 = c.p.open_bh * c.p.open_bh;
	for (int j = 0; j < c.p.ntop; j++) {
		const tvg_topnode &t = c.top[j];
		const F nsize = (F) level_size(c.p.domain_size, t.level);
		bool open = false;
		if (have) {
			bool want = false;
			F dr[3] = { (F) t.com[0] - sp[0], (F) t.com[1] - sp[1], (F) t.com[2] - sp[2] };
			nearest(c, dr);
			const F r2 = dr[0] * dr[0] + dr[1] * dr[1] + dr[2] * dr[2];
			if (c.p.use_bh) {
				if ((double) (nsize * nsize) > r2 * c.p.open_bh) want = true;
			} else {
				const F nmass = (F) t.mass;
				if (nmass * nsize * nsize > r2 * r2 * fac) want = true;
			}
			const double dx = fabs((double) (F) (sp[0] - (F) t.pos[0]));
			if (dx < 0.6 * nsize) {
				const double dy = fabs((double) (F) (sp[1] - (F) t.pos[1]));
				if (dy < 0.6 * nsize) {
					const double dz = fabs((double) (F) (sp[2] - (F) t.pos[2]));
					if (dz < 0.6 * nsize) want = true;
				}
			}
			if (want) {
				const double lim = 0.5 * (box - nsize);
				if (fabs((double) dr[0]) > lim || fabs((double) dr[1]) > lim || fabs((double) dr[2]) > lim
				    || nsize > 0.2 * box)
					open = true;
			}
			if (!open) ewald_add_node<POT>(c, dr, (F) t.mass, s);
		}
		if (t.npart <= c.p.vsize) {
			if (open)
				small_top(
				    c, t, sp, s, [&](int64_t f, int np) { ewald_bundle<POT, S>(c, l, f, np, sp, s); },
				    [](const F d[3]) { return d[0] != 0 && d[1] != 0 && d[2] != 0; });
			if (COH) __syncwarp();
			continue;
		}
		const int start = t.target;
		const int end = start + c.tree[start].DNext;
		int cur = open ? start : INT32_MAX;
		if (COH) {
			for (;;) {
				const int node = __reduce_min_sync(0xFFFFFFFFu, cur);
				if (node == INT32_MAX) break;
				if (cur == node) cur = ewald_node<POT, S>(c, l, node, end, sp, fac, bh2, s);
				__syncwarp();
			}
		} else {
			while (cur != INT32_MAX) cur = ewald_node<POT, S>(c, l, cur, end, sp, fac, bh2, s);
		}
	}
}

// A warp walks together when its targets lie within this many particles of
// the order. Walked together, every 8th particle of a 50^3 box (FP32 gravity)
// takes 16 ms against 80 ms of the walk per thread; lane by lane, every 64th
// takes 21 against 80 ms, and of a halo of 400,000 (FP64) 2.1 against 14 ms.
#ifndef PLAIN_SPREAD
#define PLAIN_SPREAD 512
#endif

template <bool POT, bool EW, int S, typename F>
__global__ void __launch_bounds__(128)
k_walk_plain(int64_t n_act, const int32_t *__restrict__ active, PlainCtx<F> c,
             const F *__restrict__ last_acc, F *acc0, F *acc1, F *acc2, F *gacc0, F *gacc1,
             F *gacc2, F *cost_out, F *pot_out, double *counter)
{
	// every thread reads every top node: staged in shared memory when they
	// fit (one target: <= 64 level-2 cells), else read through L1
	__shared__ tvg_topnode s_top[64];
	PlainCtx<F> cc = c;
	if (c.p.ntop <= 64) {
		for (int j = threadIdx.x; j < c.p.ntop; j += blockDim.x) s_top[j] = c.top[j];
		__syncthreads();
		cc.top = s_top;
	}
	const Lanes<S> l = lanes<S>();
	const int64_t t = (blockIdx.x * (int64_t) blockDim.x + threadIdx.x) / S;
	const bool have = t < n_act;
	const int64_t tt = have ? t : n_act - 1;
	const int64_t i = active ? active[tt] : tt;     // Active_Particle_List[t]
	const F sp[3] = { c.x[i], c.y[i], c.z[i] };
	Sums s = { { 0, 0, 0 }, 0, 0, 0 };
	const int first = __reduce_min_sync(0xFFFFFFFFu, (int) i), last = __reduce_max_sync(0xFFFFFFFFu, (int) i);
	if (last - first < PLAIN_SPREAD) {
		if constexpr (EW) walk_ewald<POT, true, S>(cc, l, have, sp, last_acc[i], s);
		else walk_gravity<POT, true, S>(cc, l, have, sp, last_acc[i], s);
	} else {
		if constexpr (EW) walk_ewald<POT, false, S>(cc, l, have, sp, last_acc[i], s);
		else walk_gravity<POT, false, S>(cc, l, have, sp, last_acc[i], s);
	}
	__syncwarp();
#pragma unroll
	for (int o = 1; o < S; o <<= 1) s.own += __shfl_xor_sync(0xFFFFFFFFu, s.own, o);
	const int n = s.n + s.own;
	// the reference counts in Float, where adding 1 stops at 2^24
	const F cost = sizeof(F) == 4 ? (F) min(n, 1 << 24) : (F) n;
	const bool write = have && l.sub == 0;
	if (write) {
		// add_recv_to (tree_accel.c:110-129, tree_periodic.c:91-110)
		acc0[i] += s.a[0];
		acc1[i] += s.a[1];
		acc2[i] += s.a[2];
		if (EW) {
			gacc0[i] += s.a[0];
			gacc1[i] += s.a[1];
			gacc2[i] += s.a[2];
			cost_out[i] += cost;
			if (POT) pot_out[i] += s.pot;
		} else {
			gacc0[i] = (F) s.a[0];
			gacc1[i] = (F) s.a[1];
			gacc2[i] = (F) s.a[2];
			cost_out[i] = cost;
			if (POT) pot_out[i] = (F) s.pot;
		}
	}
	// interaction count for the roofline accounting
	double cw = write ? (double) cost : 0.0;
#pragma unroll
	for (int o = 16; o; o >>= 1) cw += __shfl_xor_sync(0xFFFFFFFFu, cw, o);
	if ((threadIdx.x & 31) == 0 && cw != 0) atomicAdd(counter, cw);
}

// the packed particles of the walks
template <typename F>
__global__ void k_plain_src(int64_t n, double gravity, const F *__restrict__ x, const F *__restrict__ y,
                            const F *__restrict__ z, const F *__restrict__ m, Float4<F> *__restrict__ src)
{
	const int64_t i = blockIdx.x * (int64_t) blockDim.x + threadIdx.x;
	if (i < n) src[i] = { x[i], y[i], z[i], (F) (gravity * m[i]) };
}

__global__ void k_plain_nodes(const tvg_devcount *__restrict__ dc, int64_t tcap, PlainParams p,
                              const WNode<float> *__restrict__ tree, PNode<float> *__restrict__ out)
{
	const int64_t nn = min(dc->nnodes, tcap);
	for (int64_t g = blockIdx.x * (int64_t) blockDim.x + threadIdx.x; g < nn; g += (int64_t) gridDim.x * blockDim.x)
		out[g] = make_node<float>(p, tree[g]);
}

// entries of load_cell
__global__ void k_plain_ewald(const float *__restrict__ fx, const float *__restrict__ fy,
                              const float *__restrict__ fz, const float *__restrict__ fp, float *__restrict__ out)
{
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= 65 * 65 * 64) return;
	const int g = (i >> 6) * 65 + (i & 63);
	float4 *o = (float4 *) out + 2 * i;
	o[0] = make_float4(fx[g], fy[g], fz[g], fp[g]);
	o[1] = make_float4(fx[g + 1], fy[g + 1], fz[g + 1], fp[g + 1]);
}

__global__ void k_plain_ewald(const double *__restrict__ fx, const double *__restrict__ fy,
                              const double *__restrict__ fz, const double *__restrict__ fp,
                              double *__restrict__ out)
{
	const int g = blockIdx.x * blockDim.x + threadIdx.x;
	if (g >= 65 * 65 * 65) return;
	double2 *o = (double2 *) out + 2 * g;
	o[0] = make_double2(fx[g], fy[g]);
	o[1] = make_double2(fz[g], fp[g]);
}

template <bool POT, bool EW, int S, typename F>
static void launch(tvg_context *ctx, int64_t n_act, const PlainCtx<F> &c)
{
	k_walk_plain<POT, EW, S, F><<<TVG_CNT(ctx, tvg_blocks(n_act * S, 128)), 128, 0, ctx->stream>>>(
	    n_act, ctx->use_active ? ctx->active : nullptr, c, (const F *) ctx->f[FS_LAST_ACC],
	    (F *) ctx->f[FS_ACC0], (F *) ctx->f[FS_ACC1], (F *) ctx->f[FS_ACC2], (F *) ctx->f[FS_GACC0],
	    (F *) ctx->f[FS_GACC1], (F *) ctx->f[FS_GACC2], (F *) ctx->f[FS_COST],
	    (F *) ctx->f[FS_GRAV_POT], ctx->counters + (EW ? 1 : 0));
}

// Lanes per target: one, while there are targets enough to fill the SMs. Below
// that FP64 and the Ewald part are bound by the latency of one particle (the
// FP64 root and reciprocal, the table lookup), and sharing a target's particles
// between lanes gives the SMs more of them in flight, at the price of the
// exchange. Measured, ms by lanes per target 1 / 2 / 4 / 8: FP64 gravity with
// the potential, halo of 60,000: 5.07 / 4.71 / 5.05 / 6.63; of 30,011: 5.14 /
// 3.78 / 2.84 / 3.90; of 3500: 1.51 / 1.21 / 0.76 / 0.62. FP32 Ewald, box of
// 125,000: 75.6 / 78.9 / 77.5 / 94.2; of 64,000: 29.3 / 25.8 / 28.6 / 34.3; of
// 21,952: 16.5 / 12.6 / 10.2 / 12.4; of 5832: 3.8 / 2.9 / 1.9 / 1.6. FP32
// gravity has four particles in flight by itself (33 / 52 / 65 ms at 125,000,
// 3.3 / 3.7 / 3.0 at 21,952, 1.3 / 1.6 / 1.3 at 5832) and keeps one.
template <bool POT, bool EW, typename F>
static void launch_lanes(tvg_context *ctx, int64_t n_act, const PlainCtx<F> &c)
{
	if constexpr (!EW && sizeof(F) == 4) {
		launch<POT, EW, 1, F>(ctx, n_act, c);
	} else {
		if (n_act >= 100000) launch<POT, EW, 1, F>(ctx, n_act, c);
		else if (n_act >= 45000) launch<POT, EW, 2, F>(ctx, n_act, c);
		else if (n_act >= 8000) launch<POT, EW, 4, F>(ctx, n_act, c);
		else launch<POT, EW, 8, F>(ctx, n_act, c);
	}
}

template <typename F>
static int walk_typed(tvg_context *ctx, int use_bh, uint32_t parts)
{
	const int64_t n = ctx->n;
	if (n == 0) return TVG_OK;
	static_assert(sizeof(PNode<float>) == sizeof(tvg_wnode), "the node records use the walk tree's memory");
	PlainCtx<F> c;
	c.x = (const F *) ctx->f[FS_POS0];
	c.y = (const F *) ctx->f[FS_POS1];
	c.z = (const F *) ctx->f[FS_POS2];
	c.m = (const F *) ctx->f[FS_MASS];
	c.top = ctx->d_top;
	c.tree = (const WNode<F> *) ctx->tree;
	c.tree_cap = ctx->tcap;
	c.n = n;
	const tvg_config &cf = ctx->cfg;
	c.p.gravity = cf.gravity;
	c.p.domain_size = ctx->dsize;
	c.p.boxsize = cf.periodic ? cf.boxsize : 0;
	c.p.open_bh = cf.open_bh;
	c.p.open_rel = cf.open_rel;
	const double eps = -41.0 / 32.0 * cf.softening;    // tree_build.c:136-138
	c.p.eps = eps;
	c.p.eps2 = eps * eps;
	c.p.eps3 = eps * eps * eps;
	c.p.box2grid = cf.periodic ? 2 * 64 / cf.boxsize : 0;
	c.p.periodic = cf.periodic;
	c.p.use_bh = use_bh;
	c.p.vsize = cf.vector_size;
	c.p.ntop = ctx->ntop;
	c.p.fix_small = (cf.flags & TVG_CFG_FIX_SMALL_TOPNODES) ? 1 : 0;
	c.boxhalf = (F) (c.p.boxsize / 2.0);
	c.eps2 = (F) c.p.eps2;
	if ((double) c.eps2 < c.p.eps2) c.eps2 = (F) nextafterf((float) c.eps2, 3.0e38f);
	c.r2min = c.eps2 > (F) 8.7e-19 ? c.eps2 : (F) 8.7e-19;      // above 2^-60
	c.r2max = (F) 1.15e18;                                      // below 2^60
	c.box = c.p.boxsize == (double) (float) c.p.boxsize ? (F) c.p.boxsize : (F) 0;
	cudaStream_t s = ctx->stream;
	TVG_CUDA(ctx, cudaMemsetAsync(ctx->counters, 0, 16, s));
	TVG_CUDA(ctx, cudaEventRecord(ctx->ev[0], s));
	// packed particles in the key staging buffer (32 B per particle), node
	// records in the group form's walk tree, which its next walk then rebuilds
	Float4<F> *src = (Float4<F> *) ctx->pref;
	k_plain_src<F><<<TVG_CNT(ctx, tvg_blocks(n, 256)), 256, 0, s>>>(n, cf.gravity, c.x, c.y, c.z, c.m, src);
	c.src = src;
	c.pn = nullptr;
	if (sizeof(F) == 4) {
		PNode<float> *pn = (PNode<float> *) ctx->wtree;
		ctx->have_walktree = false;
		k_plain_nodes<<<TVG_CNT(ctx, 148 * 8), 256, 0, s>>>(ctx->dc, ctx->tcap, c.p,
		                                                    (const WNode<float> *) ctx->tree, pn);
		c.pn = pn;
	}
	c.ew = nullptr;
	if (parts & TVG_WALK_EWALD) {
		const int npt = 65 * 65 * 65;
		if (!ctx->ewald_xyz) TVG_CHECK(tvg_alloc(ctx, &ctx->ewald_xyz, 32 * (size_t) npt));
		F *const *f = (F *const *) ctx->ewald_f;
		k_plain_ewald<<<TVG_CNT(ctx, tvg_blocks(npt, 256)), 256, 0, s>>>(f[0], f[1], f[2], f[3],
		                                                                 (F *) ctx->ewald_xyz);
		c.ew = (const F *) ctx->ewald_xyz;
	}
	TVG_CUDA(ctx, cudaGetLastError());
	for (int part = 0; part < 2; part++) {
		const bool ew = part == 1;
		if (!(parts & (ew ? TVG_WALK_EWALD : TVG_WALK_GRAVITY))) continue;
		if (ew) TVG_CUDA(ctx, cudaEventRecord(ctx->ev[0], s));
		const int64_t n_act = ctx->use_active ? ctx->n_active : n;
		if (n_act > 0) {
			const bool pot = (cf.flags & TVG_CFG_POTENTIAL) != 0;
			if (ew && pot) launch_lanes<true, true, F>(ctx, n_act, c);
			else if (ew) launch_lanes<false, true, F>(ctx, n_act, c);
			else if (pot) launch_lanes<true, false, F>(ctx, n_act, c);
			else launch_lanes<false, false, F>(ctx, n_act, c);
			TVG_CUDA(ctx, cudaGetLastError());
		}
		TVG_CUDA(ctx, cudaEventRecord(ctx->ev[1], s));
		TVG_CUDA(ctx, cudaEventSynchronize(ctx->ev[1]));
		float ms = 0;
		TVG_CUDA(ctx, cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]));
		ctx->phase_ms[ew ? 5 : 4] = ms;
	}
	double cnt[2];
	TVG_CUDA(ctx, cudaMemcpy(cnt, ctx->counters, 16, cudaMemcpyDeviceToHost));
	ctx->last_counts[0] = cnt[0];
	ctx->last_counts[1] = cnt[1];
	return TVG_OK;
}

int tvg_impl_walk_plain(tvg_context *ctx, int use_bh, uint32_t parts)
{
	if (ctx->cfg.float_bytes == 4) return walk_typed<float>(ctx, use_bh, parts);
	return walk_typed<double>(ctx, use_bh, parts);
}

// accel.c:28-43: Last_Acc_Mag = |Acc|, Acc = 0 (the active particles; their
// number from the device when n_dev is given, n bounds it)
template <typename F>
__global__ void k_save_last(int64_t n, const int64_t *__restrict__ n_dev, const int32_t *__restrict__ active,
                            F *a0, F *a1, F *a2, F *last)
{
	const int64_t k = blockIdx.x * (int64_t) blockDim.x + threadIdx.x;
	if (k >= n || (n_dev && k >= *n_dev)) return;
	const int64_t i = active ? active[k] : k;
	last[i] = fsqrt<F>(a0[i] * a0[i] + a1[i] * a1[i] + a2[i] * a2[i]);
	a0[i] = a1[i] = a2[i] = 0;
}

int tvg_impl_save_last_accel(tvg_context *ctx)
{
	// with an active list its length is read on the device (the list may be
	// built in the same captured step)
	const int64_t n = ctx->n;
	const int32_t *act = ctx->use_active ? ctx->active : nullptr;
	const int64_t *nd = ctx->use_active ? &ctx->dc->n_active : nullptr;
	if (!n) return TVG_OK;
	if (ctx->cfg.float_bytes == 4)
		k_save_last<float><<<TVG_CNT(ctx, tvg_blocks(n, 256)), 256, 0, ctx->stream>>>(
		    n, nd, act, (float *) ctx->f[FS_ACC0], (float *) ctx->f[FS_ACC1], (float *) ctx->f[FS_ACC2],
		    (float *) ctx->f[FS_LAST_ACC]);
	else
		k_save_last<double><<<TVG_CNT(ctx, tvg_blocks(n, 256)), 256, 0, ctx->stream>>>(
		    n, nd, act, (double *) ctx->f[FS_ACC0], (double *) ctx->f[FS_ACC1], (double *) ctx->f[FS_ACC2],
		    (double *) ctx->f[FS_LAST_ACC]);
	TVG_CUDA(ctx, cudaGetLastError());
	return TVG_OK;
}

template <typename F>
__global__ void k_zero_active(int64_t n, const int32_t *__restrict__ active, F *a0, F *a1, F *a2,
                              F *g0, F *g1, F *g2, F *cost)
{
	const int64_t k = blockIdx.x * (int64_t) blockDim.x + threadIdx.x;
	if (k >= n) return;
	const int64_t i = active[k];
	a0[i] = a1[i] = a2[i] = 0;
	g0[i] = g1[i] = g2[i] = 0;
	cost[i] = 0;
}

// Acc, Grav_Acc and Cost of the active particles (all when no list is set)
int tvg_impl_zero_accel(tvg_context *ctx)
{
	if (ctx->use_active) {
		const int64_t n = ctx->n_active;
		if (!n) return TVG_OK;
		void **f = ctx->f;
		if (ctx->cfg.float_bytes == 4)
			k_zero_active<float><<<TVG_CNT(ctx, tvg_blocks(n, 256)), 256, 0, ctx->stream>>>(
			    n, ctx->active, (float *) f[FS_ACC0], (float *) f[FS_ACC1], (float *) f[FS_ACC2],
			    (float *) f[FS_GACC0], (float *) f[FS_GACC1], (float *) f[FS_GACC2], (float *) f[FS_COST]);
		else
			k_zero_active<double><<<TVG_CNT(ctx, tvg_blocks(n, 256)), 256, 0, ctx->stream>>>(
			    n, ctx->active, (double *) f[FS_ACC0], (double *) f[FS_ACC1], (double *) f[FS_ACC2],
			    (double *) f[FS_GACC0], (double *) f[FS_GACC1], (double *) f[FS_GACC2],
			    (double *) f[FS_COST]);
		TVG_CUDA(ctx, cudaGetLastError());
		return TVG_OK;
	}
	const size_t b = tvg_fsize(ctx) * ctx->n;
	const int slots[] = { FS_ACC0, FS_ACC1, FS_ACC2, FS_GACC0, FS_GACC1, FS_GACC2, FS_COST, FS_GRAV_POT };
	for (int s : slots) TVG_CUDA(ctx, cudaMemsetAsync(ctx->f[s], 0, b, ctx->stream));
	return TVG_OK;
}
