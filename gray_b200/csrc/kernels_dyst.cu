/*
 * Mixed-precision persistent kernel for numerical spacetimes (interp.cl +
 * dyst.cl): several lanes per ray, the ray's cell held in registers.
 *
 * A ray moves at most 0.01 M per stage through cells of up to 2 M, so the same
 * 8 corners mostly serve dozens to hundreds of RHS evaluations.  (The fisheye
 * nodes crowd at the coordinate planes: at 256^3 cells are thinner than a
 * stage's 0.01 M within 0.13 M of one, and a ray that crosses them searches and
 * reads at every RHS while its warp waits.  A strip of 300 x 200 rays along a
 * plane takes 28.7 ms there, one across it 26.1.)
 * Lane m of a ray's
 * four lanes owns x^m, u^m and row m of the Christoffel symbols: the ten
 * Gamma^m_ab of the cell's 8 corners stay in 80 of its registers and are
 * read from memory only when the ray enters another cell.  An RHS is then 40
 * packed FMAs per lane (two corners each) and about ten shuffles, with no
 * loads.  With one ray per thread the 40 symbols of 8 corners (320 floats)
 * fit no thread, so every RHS fetched 1,280 bytes per ray through L1, and
 * that latency bound the kernel.
 *
 * What bounds it: the FP32 pipe and issue, about evenly (512^2 rays inside the
 * box: FMA pipe 57% of its cycles, issue 60%, 141 instructions per warp and
 * RHS against 105 counted from the algorithm; 12 warps per SM at 168
 * registers).  Measured, B200 at
 * 1965 MHz, one ray per thread before and four lanes now: 512^2 rays at 200 M
 * on a 128^3 grid 530 -> 197 ms (1.48e10 -> 3.99e10 ray-steps/s), 97 x 72
 * rays on a 256^3 grid 243 -> 22.8 ms, 160 x 120 rays between two levels
 * with four frequencies 47.3 -> 14.3 ms; outputs bit-identical.  The pairs
 * are kept as 64-bit values: as float2 the compiler repacked the cell at
 * every RHS (247 instructions, 301 ms).  At 128 registers and 16 warps the
 * large render took 196 ms but the spills cost small ones 17% (20.3 ms
 * against 17.3 at 64^2 rays).
 *
 * Where rays run between the two time levels (LV = 2) a ray has eight lanes,
 * four per level.
 *
 * Thermal transfer: lanes 0 and 3 also hold their rows of g (for k_t and
 * k_z), lane 1 rho.  Emission and absorption at a stage depend on the
 * geodesic alone, so the four stages are walked first and then lane m
 * evaluates stage m, one frequency per pass (two with eight lanes); only
 * e^-tau chains the stages, through one shuffle.  With a frequency per lane
 * instead, 200 x 160 rays between two levels took 28.1 ms for one frequency
 * (now 19.0) and 160 x 120 rays 17.5 ms for four (14.3); eight frequencies in
 * one level, where no lane idled, 14.7 (18.0).  At 168 registers these forms
 * spill (244 to 310 bytes of stores).
 *
 * Grid layout: per time level float [nz][ny][nx][GRAY_NSTRIDE] with the
 * fields of one grid point contiguous (Gamma 0..39, g 40..49, rho 50, pad).
 * The fisheye node coordinates come from a per-axis table (n + 1 entries)
 * instead of sinh((A i + B)^3) per field and call (interp.cl:99-121), and the
 * cell search runs once per RHS for all fields instead of once per field
 * (102 times in the reference).
 */
#include <cfloat>
#include <climits>

#include "dyst64.cuh"
#include "mixed_table.h"

namespace {

using dyst64::dyst_getuu64;
using dyst64::dyst_getdt64;

/* ---------------------------------------------------------------- mixed */

__device__ __forceinline__ float
rcp_a(float x)
{
	float r;
	asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
	return r;
}

__device__ __forceinline__ float
ex2_a(float x)
{
	float r;
	asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
	return r;
}

__device__ __forceinline__ float
lg2_a(float x)
{
	float r;
	asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
	return r;
}

__device__ __forceinline__ float
sqrt_a(float x)
{
	float r;
	asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
	return r;
}

struct DystConst {
	float B[3], iA[3];
};

/* Fractional logical coordinate on a fisheye axis, with the cell found
 * exactly against the node table: the FP32 map only gives the first guess,
 * node comparisons settle it (the answer depends on x and the table alone).
 * cell: x0, x1, 1/(x1 - x0), i of the cell; past either end the range in
 * which x is clamped there, with 0 for 1/(x1 - x0). */
__device__ __forceinline__ float
axis_search(const float *nd, int n, float x, float Bf, float iAf, float4 &cell)
{
	const float first = __ldg(nd), last = __ldg(nd + n - 1);
	if(!(x >= first)) {               /* before the first node (or NaN): clamp-to-edge */
		cell = make_float4(-INFINITY, first, 0.0f, 0.0f);
		return 0.0f;
	}
	if(x >= last) {                   /* at or past the last node */
		cell = make_float4(last, INFINITY, 0.0f, (float)(n - 1));
		return (float)(n - 1);
	}
	float ax = fabsf(x);
	float as = 0.69314718f * lg2_a(ax + sqrt_a(fmaf(ax, ax, 1.0f)));   /* asinh|x| */
	float cb = as > 0.0f ? ex2_a(0.33333334f * lg2_a(as)) : 0.0f;       /* cbrt     */
	cb = copysignf(cb, x);
	float xi = floorf((cb - Bf) * iAf);
	int i = xi >= 0.0f ? (xi <= (float)(n - 2) ? (int)xi : n - 2) : 0;
	float x0 = __ldg(nd + i), x1 = __ldg(nd + i + 1);
	/* nd[0] <= x < nd[n-1] keeps both walks inside [0, n-2] */
	for(int it = 0; it < 2 && x < x0; ++it) {
		--i;
		x1 = x0;
		x0 = __ldg(nd + i);
	}
	for(int it = 0; it < 2 && x >= x1; ++it) {
		++i;
		x0 = x1;
		x1 = __ldg(nd + i + 1);
	}
	const float inv = rcp_a(x1 - x0);
	cell = make_float4(x0, x1, inv, (float)i);
	return fmaf(x - x0, inv, (float)i);
}

/* ------------------------------------------------ thermal transfer island */

/* 1/b to ~1e-14 relative: the FP32 approximate reciprocal refined by one
 * FP64 Newton step (b within the FP32 normal range) */
__device__ __forceinline__ double
rcp64(double b)
{
	const double r = (double)rcp_a((float)b);
	return fma(r, fma(-b, r, 1.0), r);
}

/* e^x for |x| within the FP32 range, ~1e-7 relative */
__device__ __forceinline__ float
exp_f(float x)
{
	return ex2_a(x * 1.4426950408889634f);
}

/* rt.cl:80-198 for the mixed kernel: the magnitudes (1e-47 .. 1e+39 in CGS)
 * stay FP64, the special functions of O(1) arguments (exp, log, cbrt,
 * sqrt) take the FP32 approximate instructions, and everything that
 * depends only on the render is a ThermalFast constant.  Same formulas and
 * branches as the FP64 kernels; agreement to ~1e-6 relative. */
struct RayFrame { /* what the frequencies of a ray at one event share */
	double shift, ish2, nus, inus, ne;
	bool syn;
};

__device__ __forceinline__ RayFrame
ray_frame(const ThermalFast &t, double kt, double kz, double ne)
{
	const double EPS = GRAY_EPSILON;
	RayFrame r;
	r.ne = ne;
	r.shift = -kt;
	const float bkcos = (float)(kz * t.b) * rcp_a((float)(r.shift * t.b + EPS));
	r.ish2 = rcp64(fma(r.shift, r.shift, EPS));
	/* synchrotron frequency: nu_s = knus sin(theta), zero along the field */
	r.nus = r.inus = 0.0;
	r.syn = t.syn && bkcos > -1.0f && bkcos < 1.0f;
	if(r.syn) {
		r.nus = t.knus * (double)sqrt_a(fmaf(-bkcos, bkcos, 1.0f));
		r.inus = rcp64(r.nus + EPS);
	}
	return r;
}

/* L_nu at the event, and B_nu */
__device__ __forceinline__ double
emissivity(const ThermalFast &t, const RayFrame &r, double nu_hz, double &B)
{
	const double EPS = GRAY_EPSILON;
	const double nu = nu_hz * r.shift;
	/* rt.cl:80-93 */
	const double f2 = nu * t.kf2;
	if(f2 > 1e-5) {
		double em1;
		if(f2 < 0.3) /* e^f2 - 1 by its series: no cancellation */
			em1 = f2 * fma(f2, fma(f2, fma(f2, fma(f2, fma(f2, fma(f2,
			      1.0 / 5040, 1.0 / 720), 1.0 / 120), 1.0 / 24), 1.0 / 6), 0.5), 1.0);
		else if(f2 < 80.0)
			em1 = (double)exp_f((float)f2) - 1.0;
		else
			em1 = exp(f2);
		B = t.kB * (nu * nu) * nu / em1;
	} else {
		B = t.kB2 * (nu * nu) * rcp64(fma(f2, fma(f2, 1.0 / 6, 0.5), 1.0));
	}
	/* rt.cl:95-143 bremsstrahlung */
	const double y = nu * t.ky;
	double Lff = 0.0;
	if(y < 80.0) {
		const float yf = (float)(y + EPS);
		const float sy = sqrt_a((float)y);
		double G;
		if(t.xg > 1.0)
			G = y > 1.0 ? t.g1 / (double)sy
			            : t.g2 * (t.g3 - 0.6931471805599453 * (double)lg2_a(yf));
		else if(t.xg * y > 1.0)
			G = t.g5 * rcp64(t.sxg * (double)sy);
		else if(y > t.sxg)
			G = 1.0;
		else {
			G = t.g2 * (t.g4 + 0.6931471805599453 *
			                      (double)(lg2_a((float)t.sxg) - lg2_a(yf)));
			G = G > EPS ? G : EPS;
		}
		Lff = (t.kff * (r.ne * r.ne)) * G * rcp64(fma(t.sqte, (double)exp_f((float)y), EPS));
	}
	/* rt.cl:145-170 synchrotron */
	double Lsyn = 0.0;
	if(r.syn) {
		double x = nu * r.inus;
		x = x < 1e30 ? x : 1e30; /* e^-cbrt(x) is 0 long before */
		const float xf = (float)x;
		const float cx = ex2_a(0.33333334f * lg2_a(xf));
		const double xx = (double)sqrt_a(xf) + 1.88774862536 * (double)sqrt_a(cx);
		Lsyn = t.ksyn * (xx * xx) * (double)exp_f(-cx) * (r.ne * r.nus);
	}
	return Lsyn + Lff;
}

/* ------------------------------------------------------------ the kernel */

/* The cell a lane holds: rows of ten (of Gamma^m_ab, a <= b) and, with the
 * transfer, four more (row m of g, or rho), as pairs of corners (c, c + 1)
 * along x, so that one packed FMA serves two corners. */
typedef unsigned long long pair_t; /* two FP32 in one 64-bit register pair */

__device__ __forceinline__ pair_t
pair(float a, float b)
{
	pair_t r;
	asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
	return r;
}

__device__ __forceinline__ float2
unpair(pair_t a)
{
	float2 r;
	asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
	return r;
}

__device__ __forceinline__ pair_t
fma2(pair_t a, pair_t b, pair_t c)
{
	pair_t r;
	asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
	return r;
}

__device__ __forceinline__ pair_t
mul2(pair_t a, pair_t b)
{
	pair_t r;
	asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
	return r;
}

template <bool RT>
struct Cell {
	pair_t G[4][10];
	pair_t W[RT ? 4 : 1][RT ? 4 : 1];
};

/* the fields of lane m's extra row: row m of g (dyst.cl:55-81; g_zz from
 * g_yz where the flag says so, dyst.cl:78) on lanes 0 and 3, rho on lane 1 */
__device__ __forceinline__ int
extra_field(int m, int k, int bug_gzz)
{
	if(m == 0)
		return 40 + k;
	if(m == 1)
		return k == 0 ? 50 : -1;
	if(m == 3)
		return k == 0 ? 43 : k == 1 ? 46 : k == 2 ? 48 : bug_gzz ? 48 : 49;
	return -1;
}

template <bool RT>
__device__ __forceinline__ void
load_cell(const GridParams &g, const float *lvl, int m, int ix, int iy, int iz, Cell<RT> &C)
{
	const int jx = min(ix + 1, g.nx - 1), jy = min(iy + 1, g.ny - 1), jz = min(iz + 1, g.nz - 1);
#pragma unroll
	for(int j = 0; j < 4; ++j) {
		const long long yz = (long long)((j & 2) ? jz : iz) * g.ny + ((j & 1) ? jy : iy);
		const float *a = lvl + (yz * g.nx + ix) * GRAY_NSTRIDE;
		const float *b = lvl + (yz * g.nx + jx) * GRAY_NSTRIDE;
		/* 10 m floats into a 224-byte row: 8-byte aligned */
		const float2 *ga = (const float2 *)(a + 10 * m), *gb = (const float2 *)(b + 10 * m);
#pragma unroll
		for(int k = 0; k < 5; ++k) {
			const float2 va = __ldg(ga + k), vb = __ldg(gb + k);
			C.G[j][2 * k] = pair(va.x, vb.x);
			C.G[j][2 * k + 1] = pair(va.y, vb.y);
		}
		if constexpr(RT) {
#pragma unroll
			for(int k = 0; k < 4; ++k) {
				const int f = extra_field(m, k, g.bug_gzz);
				C.W[j][k] = f >= 0 ? pair(__ldg(a + f), __ldg(b + f)) : 0;
			}
		}
	}
}

/* What a lane keeps of its axis (lanes 1-3) or of time (lane 0).  While x^m
 * stays in [xa, xb) the cell held is the right one, so the RHS needs no
 * search: w = (x - x0) inv + ci - ci.  The range is the cell cut to the box
 * (lane 0: the times with the same levels in use), or empty. */
struct Axis {
	float x0, inv, ci; /* the cell's first node, 1/width and index       */
	float xa, xb;
	int tag;           /* the cell index (lane 0: level code) in Cell    */
};

/* the levels in use: bit 0 level 0, bit 1 level 1.  In physics mode the time
 * factor is clamped to [0, 1] and a level of weight zero is not read; in
 * reference semantics, which two levels always run with LV = 2, the fields
 * extrapolate (interp.cl:183-205): both at any time, none at a NaN */
template <int LV>
__device__ __forceinline__ int
level_code(const GridParams &g, float ft)
{
	const int both = LV == 2 && !g.physics ? 3 : 0;
	return g.single ? 1 : (ft < 1.0f ? 1 | both : 0) | (ft > 0.0f ? 2 | both : 0);
}

template <bool RT>
__device__ __forceinline__ void
forget(Axis &A, Cell<RT> &C)
{
	A.tag = -1;
	A.xa = INFINITY; /* empty */
#pragma unroll
	for(int j = 0; j < 4; ++j) {
#pragma unroll
		for(int k = 0; k < 10; ++k)
			C.G[j][k] = 0;
		if constexpr(RT)
#pragma unroll
			for(int k = 0; k < 4; ++k)
				C.W[j][k] = 0;
	}
}

/* Contraction of both levels straight from memory, for a ray between the
 * levels in a one-level launch (LV = 1): rare there by the launch rule. */
template <bool RT>
__device__ __noinline__ float2
contract_both(const GridParams &g, int m, int ix, int iy, int iz, float4 w4, float4 u4)
{
	const float w[4] = {w4.x, w4.y, w4.z, w4.w}, u[4] = {u4.x, u4.y, u4.z, u4.w};
	float G = 0.0f, K = 0.0f;
#pragma unroll 1
	for(int c = 0; c < 8; ++c) {
		const float wc = ((c & 1) ? w[0] : 1.0f - w[0]) * ((c & 2) ? w[1] : 1.0f - w[1]) *
		                 ((c & 4) ? w[2] : 1.0f - w[2]);
		const int x = (c & 1) ? min(ix + 1, g.nx - 1) : ix;
		const int y = (c & 2) ? min(iy + 1, g.ny - 1) : iy;
		const int z = (c & 4) ? min(iz + 1, g.nz - 1) : iz;
		const long long row = (((long long)z * g.ny + y) * g.nx + x) * GRAY_NSTRIDE;
#pragma unroll 1
		for(int l = 0; l < 2; ++l) {
			const float wl = wc * (l ? w[3] : 1.0f - w[3]);
			const float *src = g.lvl[l] + row;
			const float2 *gs = (const float2 *)(src + 10 * m);
			float s = 0.0f;
			int k = 0;
#pragma unroll
			for(int i = 0; i < 4; ++i)
#pragma unroll
				for(int j = i; j < 4; ++j) {
					const float uu = u[i] * u[j];
					const float2 v = __ldg(gs + k / 2);
					s = fmaf((k & 1) ? v.y : v.x, i == j ? uu : 2.0f * uu, s);
					++k;
				}
			G = fmaf(wl, s, G);
			if(RT) {
				const float v1[4] = {1.0f, 0.0f, 0.0f, 0.0f};
				const float *v = m == 1 ? v1 : u;
				float e[4];
#pragma unroll
				for(int q = 0; q < 4; ++q) {
					const int f = extra_field(m, q, g.bug_gzz);
					e[q] = f >= 0 ? __ldg(src + f) : 0.0f;
				}
				const float kk = fmaf(e[3], v[3], fmaf(e[2], v[2], fmaf(e[1], v[1], e[0] * v[0])));
				K = fmaf(wl, kk, K);
			}
		}
	}
	return make_float2(G, K);
}

/* The ray left its cell, entered or left the box, or changed levels:
 * search, load what is missing, and set the range in which none of this is
 * needed.  Returns w (lane 0: the time factor); in: inside the box. */
template <int LV, bool RT>
__device__ __forceinline__ float
enter_cell(const GridParams &g, const DystConst &dc, Axis &A, Cell<RT> &C, int lane, bool on,
           float xs, bool &in)
{
	constexpr int L = 4 * LV;
	const unsigned FULL = 0xffffffffu;
	const int m = lane & 3, l = (lane & (L - 1)) >> 2, first = lane & ~(L - 1);
	const float lo = g.box[m], hi = g.box[m + 4];
	in = true;
	if(g.physics) {
		const unsigned out = __ballot_sync(FULL, m > 0 && !(xs >= lo && xs <= hi));
		in = ((out >> first) & ((1u << L) - 1u)) == 0;
	}
	const bool need = on && in;
	float w = 0.0f;
	int i0 = 0;
	if(need) {
		if(m == 0) {
			if(!g.single) {
				A.x0 = lo;
				A.inv = rcp_a(hi - lo);
				w = (xs - lo) * A.inv;
				if(g.physics)
					w = fminf(fmaxf(w, 0.0f), 1.0f);
			}
			i0 = level_code<LV>(g, w);
			/* times at which the rounded factor surely gives the same code */
			const float mg = LV == 2 && !g.physics ? -INFINITY : 1e-5f * (fabsf(lo) + fabsf(hi));
			A.xa = i0 == 2 ? hi + mg : i0 == 3 ? lo + mg : -INFINITY;
			A.xb = i0 == 1 ? (g.single ? INFINITY : lo) : i0 == 3 ? hi - mg : INFINITY;
			/* a level that holds alone: no factor, which may be above 1 and
			 * would then send every stage here */
			if(LV == 1)
				A.inv = 0.0f;
			if(i0 == 0 || (LV == 1 && i0 == 3))
				A.xa = INFINITY;
		} else {
			float uu;
			if(xs >= A.xa && xs < A.xb) {
				uu = fmaf(xs - A.x0, A.inv, A.ci);
			} else {
				const int n = m == 1 ? g.nx : m == 2 ? g.ny : g.nz;
				float4 cell;
				uu = axis_search(g.nodes_f[m - 1], n, xs, dc.B[m - 1], dc.iA[m - 1], cell);
				A.x0 = cell.z > 0.0f ? cell.x : 0.0f;
				A.inv = cell.z;
				A.ci = cell.w;
				A.xa = cell.x;
				A.xb = cell.y;
				if(g.physics) {
					A.xa = fmaxf(A.xa, lo);
					A.xb = fminf(A.xb, hi);
				}
			}
			const float fl = floorf(uu);
			i0 = (int)fl;
			w = uu - fl;
			if(fl != A.ci) /* rounded up to the next node: that cell, this once */
				A.xa = INFINITY;
		}
	}
	const unsigned moved = __ballot_sync(FULL, need && A.tag != i0);
	if(moved) {
		const int ix = __shfl_sync(FULL, i0, 1, 4), iy = __shfl_sync(FULL, i0, 2, 4),
		          iz = __shfl_sync(FULL, i0, 3, 4), code = __shfl_sync(FULL, i0, 0, 4);
		if((moved >> first) & ((1u << L) - 1u)) {
			A.tag = i0;
			if(LV == 1 ? code == 1 || code == 2 : (code >> l) & 1)
				load_cell<RT>(g, g.lvl[LV == 1 ? code - 1 : l], m, ix, iy, iz, C);
		}
	}
	return w;
}

/* Gamma^m_ab u^a u^b on lane m, and the acceleration du^m of dyst.cl:112-194
 * from it.  All lanes of the warp take part; `on` marks the lanes whose ray
 * steps.  Corners are summed in the order 000, 100, 010, ... with the levels
 * of each corner in turn.  With RT also kn = {k_t, k_z, n_e}.  in: inside
 * the box (or no box); all: so are all rays, in the cells they hold. */
template <int LV, bool RT>
__device__ __forceinline__ float
dyst_accel(const GridParams &g, const DystConst &dc, Axis &A, Cell<RT> &C, int lane, bool on,
           float xs, float us, float *kn, bool &in, bool &all)
{
	constexpr int L = 4 * LV;
	const unsigned FULL = 0xffffffffu;
	const int m = lane & 3, first = lane & ~(L - 1);
	const float u0 = __shfl_sync(FULL, us, 0, 4), u1 = __shfl_sync(FULL, us, 1, 4),
	            u2 = __shfl_sync(FULL, us, 2, 4), u3 = __shfl_sync(FULL, us, 3, 4);
	float w = fmaf(xs - A.x0, A.inv, A.ci) - A.ci;
	in = true;
	all = __all_sync(FULL, !on || (xs >= A.xa && xs < A.xb && (w < 1.0f || (LV == 2 && m == 0))));
	if(!all)
		w = enter_cell<LV, RT>(g, dc, A, C, lane, on, xs, in);
	else if(LV == 2 && m == 0 && g.physics)
		w = fminf(fmaxf(w, 0.0f), 1.0f);
	const bool need = on && in;
	const float wx = __shfl_sync(FULL, w, 1, 4), wy = __shfl_sync(FULL, w, 2, 4),
	            wz = __shfl_sync(FULL, w, 3, 4);

	pair_t S2[4] = {0, 0, 0, 0};
	{
		const float u[4] = {u0, u1, u2, u3};
		int k = 0;
#pragma unroll
		for(int i = 0; i < 4; ++i)
#pragma unroll
			for(int j = i; j < 4; ++j) {
				const float uu = u[i] * u[j];
				const float p = i == j ? uu : 2.0f * uu;
				const pair_t p2 = pair(p, p);
#pragma unroll
				for(int q = 0; q < 4; ++q)
					S2[q] = fma2(C.G[q][k], p2, S2[q]);
				++k;
			}
	}
	float2 S[4], K[4];
#pragma unroll
	for(int q = 0; q < 4; ++q)
		S[q] = unpair(S2[q]);
	if constexpr(RT) {
		const bool rho = m == 1;
		const float v0 = rho ? 1.0f : u0, v1 = rho ? 0.0f : u1, v2 = rho ? 0.0f : u2,
		            v3 = rho ? 0.0f : u3;
#pragma unroll
		for(int q = 0; q < 4; ++q)
			K[q] = unpair(fma2(C.W[q][3], pair(v3, v3),
			              fma2(C.W[q][2], pair(v2, v2),
			              fma2(C.W[q][1], pair(v1, v1), mul2(C.W[q][0], pair(v0, v0))))));
	}
	const float ax = 1.0f - wx, ay = 1.0f - wy, az = 1.0f - wz;
	float G = 0.0f, Km = 0.0f;
	if constexpr(LV == 1) {
		/* one level in use: its time weight is exactly 1 (a single level, or
		 * the clamped factor of physics mode) */
#pragma unroll
		for(int j = 0; j < 4; ++j) {
			const float wy_ = (j & 1) ? wy : ay, wz_ = (j & 2) ? wz : az;
			const float2 wc = unpair(mul2(mul2(pair(ax, wx), pair(wy_, wy_)), pair(wz_, wz_)));
			G = fmaf(wc.x, S[j].x, G);
			G = fmaf(wc.y, S[j].y, G);
			if(RT) {
				Km = fmaf(wc.x, K[j].x, Km);
				Km = fmaf(wc.y, K[j].y, Km);
			}
		}
		if(!all && !g.single) {
			const int code = __shfl_sync(FULL, A.tag, 0, 4);
			if(need && code != 1 && code != 2) {
				G = Km = 0.0f;
				if(code == 3) {
					const unsigned gm = 0xfu << first;
					const float ft = __shfl_sync(gm, w, 0, 4);
					const float2 r = contract_both<RT>(g, m, __shfl_sync(gm, A.tag, 1, 4),
					                                   __shfl_sync(gm, A.tag, 2, 4),
					                                   __shfl_sync(gm, A.tag, 3, 4),
					                                   make_float4(wx, wy, wz, ft),
					                                   make_float4(u0, u1, u2, u3));
					G = r.x;
					Km = r.y;
					forget(A, C); /* nothing of the cell is live across the call */
				}
			}
		}
	} else {
		const float ft = __shfl_sync(FULL, w, 0, 4);
		const int code = __shfl_sync(FULL, A.tag, 0, 4);
		/* the other level's sums come from the ray's other four lanes; the
		 * lanes of level 0 add both up */
		const bool use0 = code & 1, use1 = code & 2;
#pragma unroll
		for(int c = 0; c < 8; ++c) {
			const float wc = ((c & 1) ? wx : ax) * ((c & 2) ? wy : ay) * ((c & 4) ? wz : az);
			const float s0 = (c & 1) ? S[c >> 1].y : S[c >> 1].x;
			const float s1 = __shfl_xor_sync(FULL, s0, 4);
			const float w0 = wc * (1.0f - ft), w1 = wc * ft;
			G = use0 ? fmaf(w0, s0, G) : G;
			G = use1 ? fmaf(w1, s1, G) : G;
			if(RT) {
				const float k0 = (c & 1) ? K[c >> 1].y : K[c >> 1].x;
				const float k1 = __shfl_xor_sync(FULL, k0, 4);
				Km = use0 ? fmaf(w0, k0, Km) : Km;
				Km = use1 ? fmaf(w1, k1, Km) : Km;
			}
		}
		G = __shfl_sync(FULL, G, m, L);
	}
	const float G0 = __shfl_sync(FULL, G, 0, L);
	if constexpr(RT) {
		kn[0] = __shfl_sync(FULL, Km, 0, L);
		kn[1] = __shfl_sync(FULL, Km, 3, L);
		kn[2] = __shfl_sync(FULL, Km, 1, L);
	}
	return fmaf(G0, us, -G);
}

/* Far from the box (physics mode): u is constant and a step is the
 * compensated update of x alone, so a chunk of steps runs as one loop of
 * four operations each: as many as every ray of the warp surely stays
 * outside (by its distance to the box on some axis, less 1% for rounding
 * and two steps for the stage positions) and short of its interval's last
 * step.  k: the sum of the stages' slopes, dx: the size of one step.  False:
 * no step was taken. */
__device__ __forceinline__ bool
flat_steps(const GridParams &g, int m, bool step, int &h, int n, int dh_step,
           float h6, float k, float dx, float &xh, float &xl, float uh, float ul, unsigned &cnt)
{
	const unsigned FULL = 0xffffffffu;
	/* steps until this lane's axis may reach the box; 0: it is inside */
	const float lo = g.box[m], hi = g.box[m + 4];
	const float d = m ? fmaxf(lo - xh, xh - hi) : 0.0f;
	float far = d > 0.0f ? fminf(0.99f * d * rcp_a(dx + 1e-30f), 1e6f) - 2.0f : 0.0f;
	far = fmaxf(far, __shfl_xor_sync(FULL, far, 1));
	far = fmaxf(far, __shfl_xor_sync(FULL, far, 2));
	/* u's own update must be a fixed point, and x may not overflow on the way
	 * (a ray whose state does, or is not finite, ends at that step) */
	const float tu = uh - ul;
	const bool still = tu == uh && (tu - uh) + ul == ul && fabsf(xh) <= 1e30f && dx <= 1e24f;
	int todo = far >= 1.0f ? (int)far : 0;
	const int left = step ? (n - h - 1) / dh_step : INT_MAX; /* not the last step */
	todo = !step ? INT_MAX : still ? min(todo, left) : 0;
	todo = __reduce_min_sync(FULL, todo);
	if(todo <= 0 || todo == INT_MAX)
		return false;
	if(step) {
		for(int i = 0; i < todo; ++i) {
			const float yx = fmaf(h6, k, -xl);
			const float tx = xh + yx;
			xl = (tx - xh) - yx;
			xh = tx;
		}
		h += todo * dh_step;
		cnt += todo;
	}
	__syncwarp();
	return true;
}

/* the null-constraint diagnostic of a finished ray, out of line so that its
 * FP64 temporaries do not add to the registers of the stepping loop */
__device__ __noinline__ double
final_uu(const GridParams &g, double q0, double q1, double q2, double q3, double v0, double v1,
         double v2, double v3)
{
	const double s[8] = {q0, q1, q2, q3, v0, v1, v2, v3};
	return dyst_getuu64(g, s);
}

/* RK4 of a ray's (I, tau) over a step of hs, given on lane m the frame of
 * stage m.  Frequency f is kept by lane (f / LV) % 4 of half f % LV. */
template <int LV, int FPL>
__device__ __forceinline__ void
transfer(const MixedRender &c, int nf, unsigned gmask, int lane, double hs, float kt, float kz,
         float ne, double *I, double *tau)
{
	const int m = lane & 3, l = LV == 2 ? (lane >> 2) & 1 : 0;
	const ThermalFast &t = c.tf;
	const RayFrame r = ray_frame(t, kt, kz, ne);
	const double h6 = hs / 6.0, cd = m == 3 ? hs : 0.5 * hs;
#pragma unroll
	for(int i = 0; i < FPL; ++i)
#pragma unroll 1
		for(int q = 0; q < 4; ++q) {
			const int f = LV * (4 * i + q) + l;
			if(LV * (4 * i + q) >= nf)
				break;
			double B;
			const double nL = -emissivity(t, r, c.nu_hz[f < nf ? f : 0], B);
			const double dt = nL * r.shift * rcp64(B + GRAY_EPSILON);
			const double t0 = __shfl_sync(gmask, tau[i], q, 4);
			const double before = __shfl_up_sync(gmask, dt, 1, 4);
			const double st = m ? fma(cd, before, t0) : t0;
			const double dI = nL * (double)exp_f(-(float)st) * r.ish2;
			double sI = __shfl_sync(gmask, dI, 0, 4), sT = __shfl_sync(gmask, dt, 0, 4);
#pragma unroll
			for(int k = 1; k < 4; ++k) {
				const double w = k < 3 ? 2.0 : 1.0;
				sI = fma(w, __shfl_sync(gmask, dI, k, 4), sI);
				sT = fma(w, __shfl_sync(gmask, dt, k, 4), sT);
			}
			if(m == q && f < nf) {
				I[i] = fma(h6, sI, I[i]);
				tau[i] = fma(h6, sT, tau[i]);
			}
		}
}

constexpr int DYST_BLOCK = 128, DYST_PER_SM = 3;

/* LV: the time levels a ray's lanes hold; FPL: frequencies
 * per lane (0: geodesics alone).  The transfer pairs (I, tau) are FP64 and
 * ride along in the same RK4 stages. */
template <int LV, int FPL>
__global__ void __launch_bounds__(DYST_BLOCK, DYST_PER_SM)
dyst_mixed_kernel(const MixedTable T, const __grid_constant__ GridParams g, const DystConst dc,
                  const int nf, unsigned int *__restrict__ queue,
                  unsigned long long *__restrict__ steps, unsigned long long *__restrict__ inbox)
{
	constexpr int L = 4 * LV;   /* lanes per ray */
	constexpr bool RT = FPL > 0;
	/* stages unrolled: 197 ms against 225 on the 512^2 render; beside the
	 * transfer one body (its registers are short) */
	constexpr int STAGES = RT ? 1 : 4;
	constexpr int NR = RT ? FPL : 1;
	const unsigned FULL = 0xffffffffu;
	const int lane = threadIdx.x & 31, sub = lane & (L - 1), m = lane & 3;
	const int first = lane & ~(L - 1);
	const unsigned gmask = ((L == 32 ? 0u : (1u << L)) - 1u) << first;

	Axis A;
	Cell<RT> C;
	forget(A, C);
	A.x0 = A.inv = A.ci = A.xb = 0.0f;

	float xh = 0.0f, xl = 0.0f, uh = 0.0f, ul = 0.0f; /* x^m, u^m: high and low parts */
	/* (I, tau) of the frequencies this lane keeps: own(0), own(1) */
	auto own = [&](int i) { return LV * (4 * i + m) + (sub >> 2); };
	double I[NR], tau[NR];
#pragma unroll
	for(int i = 0; i < NR; ++i)
		I[i] = tau[i] = 0.0;
	unsigned ray = 0;
	int dump = 0, h = 0, dh_step = 0, n = 0;
	float dtn = 0.0f;
	double dtnd = 0.0; /* the FP64 substep unit of the transfer */
	bool active = false, exhausted = false, bad = false;
	bool quiet = false; /* every ray of the warp stayed in its cell and the box */
	/* steps of the rays this lane leads, flushed at dump boundaries once a
	 * count reaches 2^31: an interval takes fewer than 2^31 steps */
	unsigned cnt = 0, cnt_in = 0;
	const MixedRender *c = nullptr;

	for(;;) {
		if(!__all_sync(FULL, active)) {
			const bool need = !active && !exhausted;
			const unsigned mask = __ballot_sync(FULL, need && sub == 0);
			if(mask) {
				const int leader = __ffs(mask) - 1;
				unsigned base = 0;
				if(lane == leader)
					base = atomicAdd(queue, (unsigned)__popc(mask));
				base = __shfl_sync(FULL, base, leader);
				if(need) {
					const unsigned long long gidx = (unsigned long long)base +
					                                __popc(mask & ((1u << first) - 1u));
					if(gidx < T.total) {
						int rr = 0;
						while(rr + 1 < T.n_renders && T.prefix[rr + 1] <= gidx)
							++rr;
						c = &T.renders[rr];
						ray = (unsigned)(gidx - T.prefix[rr]);
						n = (int)((INT_MAX / c->n_sub) * c->n_sub);
						const double vx = c->data[m * c->n_rays + ray];
						const double vu = c->data[(4 + m) * c->n_rays + ray];
						xh = (float)vx;
						xl = (float)((double)xh - vx);
						uh = (float)vu;
						ul = (float)((double)uh - vu);
						if constexpr(RT) {
#pragma unroll
							for(int i = 0; i < FPL; ++i) {
								const int f = own(i) < nf ? own(i) : 0;
								I[i] = c->data[(8 + f) * c->n_rays + ray];
								tau[i] = c->data[(8 + nf + f) * c->n_rays + ray];
							}
						}
						dump = c->dump_begin - 1;
						h = n; /* forces the first dump set-up below */
						active = true;
					} else {
						exhausted = true;
					}
				}
				__syncwarp();
			}
			if(!__any_sync(FULL, active))
				break;
		}
		bool step = active;
		if(active && h >= n) { /* next dump interval: constants of driver.cl:93 */
			step = false;
			if(cnt >= 0x80000000u) {
				if(sub == 0)
					atomicAdd(steps, (unsigned long long)cnt);
				cnt = 0;
			}
			if(cnt_in >= 0x80000000u) {
				if(sub == 0 && inbox)
					atomicAdd(inbox, (unsigned long long)cnt_in);
				cnt_in = 0;
			}
			if(bad || ++dump >= c->dump_end) { /* done: write the ray back */
				const double x = (double)xh - (double)xl, u = (double)uh - (double)ul;
				double q[4], v[4];
#pragma unroll
				for(int k = 0; k < 4; ++k) {
					q[k] = __shfl_sync(gmask, x, k, 4);
					v[k] = __shfl_sync(gmask, u, k, 4);
				}
				if(sub < 4) {
					c->data[m * c->n_rays + ray] = x;
					c->data[(4 + m) * c->n_rays + ray] = u;
				}
				if constexpr(RT) {
#pragma unroll
					for(int i = 0; i < FPL; ++i)
						if(own(i) < nf) {
							c->data[(8 + own(i)) * c->n_rays + ray] = I[i];
							c->data[(8 + nf + own(i)) * c->n_rays + ray] = tau[i];
						}
				}
				if(sub == 0)
					c->info[ray] = bad ? q[0] - q[0] /* NaN marks the ray */
					                   : final_uu(g, q[0], q[1], q[2], q[3], v[0], v[1], v[2], v[3]);
				active = bad = false;
				forget(A, C); /* nothing of the cell is live across the call */
			} else {
				double t0 = c->t_init + (double)dump * c->dt_dump;
				double t1 = c->t_init + (double)(dump + 1) * c->dt_dump;
				double dt = t1 - t0;
				const double ticks = dyst_getdt64(dt / (double)c->n_sub) / dt * (double)n;
				dh_step = ticks >= 1.0 ? (int)ticks : 0;
				dtnd = dt / (double)n;
				dtn = (float)dtnd;
				h = 0;
				if(dh_step == 0) /* zero-length interval: nothing to integrate */
					h = n;
				else
					step = true;
			}
		}
		__syncwarp();
		const int dh = step ? (dh_step < n - h ? dh_step : n - h) : 0;
		const float hs = (float)dh * dtn, hh = 0.5f * hs;
		const float h6 = hs * (1.0f / 6.0f);

		/* flat space through the whole step (physics mode outside the box):
		 * no field enters, u is constant, nothing emits.  Not asked where the
		 * last step found every ray inside. */
		bool out = false, in0 = true, in = true; /* out: this ray, all step long */
		bool flat = false;
		if(g.physics && !quiet) {
			const float lo = g.box[m], hi = g.box[m + 4];
			auto outside = [&](float x) {
				unsigned b = __ballot_sync(FULL, m > 0 && !(x >= lo && x <= hi));
				return ((b >> first) & ((1u << L) - 1u)) != 0;
			};
			const bool o1 = outside(xh), o2 = outside(fmaf(hh, uh, xh)), o4 = outside(fmaf(hs, uh, xh));
			out = o1 && o2 && o4;
			flat = __all_sync(FULL, !step || out);
		}
		float sx, su, kx, ku;
		if(flat) {
			sx = fmaf(2.0f, uh, fmaf(2.0f, uh, uh));
			kx = uh;
			su = ku = 0.0f;
			in0 = false;
			if(flat_steps(g, m, step, h, n, dh_step, h6, sx + kx, fabsf(hs * uh), xh, xl, uh, ul,
			              cnt))
				continue;
		} else {
			float kn[3], kt = 0.0f, kz = 0.0f, ne = 0.0f; /* stage m's */
			bool all = true;
			quiet = true;
			sx = su = 0.0f;
			float x = xh, u = uh;
#pragma unroll STAGES
			for(int s = 0; s < 4; ++s) {
				kx = u;
				ku = dyst_accel<LV, RT>(g, dc, A, C, lane, step && !out, x, u, kn, in, all);
				in = in && !out;
				quiet = quiet && all;
				in0 = s == 0 ? in : in0;
				ku = in ? ku : 0.0f;
				if(RT && s == m) {
					/* flat space, empty, outside */
					kt = in ? kn[0] : -1.0f;
					kz = in ? kn[1] : 0.0f;
					ne = in ? kn[2] : 0.0f;
				}
				const float wg = (s == 1 || s == 2) ? 2.0f : 1.0f;
				const float cg = s < 2 ? hh : hs;
				if(s < 3) { /* k4 stays in kx, ku for the update */
					sx = s == 0 ? kx : fmaf(wg, kx, sx);
					su = s == 0 ? ku : fmaf(wg, ku, su);
				}
				x = fmaf(cg, kx, xh);
				u = fmaf(cg, ku, uh);
			}
			quiet = quiet && __all_sync(FULL, !out);
			if constexpr(RT) {
				const double hsd = (double)dh * dtnd;
				if(step) /* uniform over a ray's lanes */
					transfer<LV, FPL>(*c, nf, gmask, lane, hsd, kt, kz, ne, I, tau);
			}
		}
		/* compensated update, value = hi - lo */
		const float yx = fmaf(h6, sx + kx, -xl), yu = fmaf(h6, su + ku, -ul);
		const float tx = xh + yx, tu = uh + yu;
		const bool badl = !(fabsf(tx) <= FLT_MAX) || !(fabsf(tu) <= FLT_MAX);
		if(step) {
			xl = (tx - xh) - yx;
			xh = tx;
			ul = (tu - uh) - yu;
			uh = tu;
			++cnt;
			cnt_in += in0 ? 1 : 0;
			h += dh;
		}
		const unsigned badm = __ballot_sync(FULL, step && badl);
		if(badm & gmask) { /* NaN/Inf (inside the singular region): ray done */
			bad = true;
			h = n;
		}
		__syncwarp();
	}
	unsigned long long total = sub == 0 ? cnt : 0, total_in = sub == 0 ? cnt_in : 0;
#pragma unroll
	for(int o = 16; o > 0; o >>= 1) {
		total += __shfl_xor_sync(FULL, total, o);
		total_in += __shfl_xor_sync(FULL, total_in, o);
	}
	if(lane == 0 && total)
		atomicAdd(steps, total);
	if(lane == 0 && total_in && inbox)
		atomicAdd(inbox, total_in);
}

template <int LV, int FPL>
cudaError_t
launch_dyst(const MixedTable &T, const GridParams &g, const DystConst &dc, int nf,
            unsigned int *queue, unsigned long long *steps, cudaStream_t st,
            const MixedLaunch &cfg, unsigned long long *inbox)
{
	const int sms = cfg.sms > 0 ? cfg.sms : 148;
	const int max_block = cfg.block > 0 && cfg.block < DYST_BLOCK ? cfg.block : DYST_BLOCK;
	/* few rays: one warp per block until every SM has a warp, so that a
	 * small render's warps do not share an SM while others idle */
	const unsigned long long warps = (T.total + 32 / (4 * LV) - 1) / (32 / (4 * LV));
	int block = max_block;
	if(warps < (unsigned long long)sms * (max_block / 32))
		block = 32 * (int)((warps + sms - 1) / sms);
	int occ = 0;
	cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
		&occ, dyst_mixed_kernel<LV, FPL>, block, 0);
	if(e != cudaSuccess)
		return e;
	/* a plan's blocks may be larger: as many warps per SM in these */
	int per_sm = cfg.blocks_per_sm;
	if(cfg.block > DYST_BLOCK)
		per_sm *= (cfg.block + DYST_BLOCK - 1) / DYST_BLOCK;
	if(per_sm <= 0 || per_sm > occ)
		per_sm = occ > 0 ? occ : 1;
	const long long want = (long long)per_sm * sms;
	const long long need = (long long)((warps + block / 32 - 1) / (block / 32));
	unsigned grid = (unsigned)(want < need ? want : need);
	if(grid == 0)
		grid = 1;
	dyst_mixed_kernel<LV, FPL><<<grid, block, 0, st>>>(T, g, dc, nf, queue, steps, inbox);
	return cudaGetLastError();
}

} /* namespace */

/* Whether any ray of the renders may run between the two time levels, where
 * both have weight: always in reference semantics (time extrapolates), and
 * in physics mode if a window overlaps the levels' times.  A ray's time is its
 * affine parameter counted from the camera (dyst.cl:106), whatever affine time
 * the render starts at; t0 is that of dump 0.  It only chooses the launch: a
 * ray that was written to another time is right in either, and slow in the
 * wrong one (300 x 200 rays between the levels 15 ms with two levels' lanes,
 * 71 with one's; on one level 6.5 and 15). */
bool
dyst_between(const GridParams &g, const MixedRender *r, int n, double t0)
{
	if(g.single)
		return false;
	if(!g.physics)
		return true;
	for(int i = 0; i < n; ++i) {
		const double a = t0 + (double)r[i].dump_begin * r[i].dt_dump;
		const double b = t0 + (double)r[i].dump_end * r[i].dt_dump;
		if((a < b ? a : b) < (double)g.box[4] && (a < b ? b : a) > (double)g.box[0])
			return true;
	}
	return false;
}

int
dyst_rays_per_sm(bool between)
{
	return DYST_BLOCK * DYST_PER_SM / (between ? 8 : 4);
}

cudaError_t
launch_dyst_mixed_table(const MixedTable &T, const GridParams &g, int n_freq,
                        unsigned int *queue, unsigned long long *steps, cudaStream_t st,
                        const MixedLaunch &cfg, bool between, unsigned long long *inbox)
{
	static_assert(GRAY_MAX_FREQ == 8, "two frequencies per lane at most");
	DystConst dc;
	for(int a = 0; a < 3; ++a) {
		dc.B[a] = (float)g.B[a];
		dc.iA[a] = (float)(1.0 / g.A[a]);
	}
	if(n_freq < 0 || n_freq > GRAY_MAX_FREQ)
		return cudaErrorInvalidValue;
	if(cfg.block > 256)
		return cudaErrorInvalidValue;
	cudaError_t e = cudaMemsetAsync(queue, 0, sizeof(unsigned int), st);
	if(e != cudaSuccess)
		return e;
	if(between)
		return n_freq == 0 ? launch_dyst<2, 0>(T, g, dc, n_freq, queue, steps, st, cfg, inbox)
		                   : launch_dyst<2, 1>(T, g, dc, n_freq, queue, steps, st, cfg, inbox);
	return n_freq == 0   ? launch_dyst<1, 0>(T, g, dc, n_freq, queue, steps, st, cfg, inbox)
	       : n_freq <= 4 ? launch_dyst<1, 1>(T, g, dc, n_freq, queue, steps, st, cfg, inbox)
	                     : launch_dyst<1, 2>(T, g, dc, n_freq, queue, steps, st, cfg, inbox);
}
