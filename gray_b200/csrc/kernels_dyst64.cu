/*
 * FP64 numerical-spacetime kernels and the boosted Kerr-Schild grid
 * generator.  Compiled with -fmad=false: the only fused multiply-adds are
 * the explicit fma() calls that mirror the CPU oracle.
 *
 *  - dyst_icond_kernel, dyst_evolve64_kernel: dyst.cl:89-110 camera rays
 *    and driver.cl:69-108 substepping on the interpolated spacetime, one
 *    launch per dump (the reference structure).
 *  - boosted_ks_kernel: samples boosted Kerr-Schild on the grid (the
 *    generator of tools/generate_data.py:87-160 with tools/boosted_ks.py's
 *    dual-number derivatives), one grid point per thread.
 */
#include <climits>

#include "dyst64.cuh"

namespace {

using namespace dyst64;

/* dyst.cl:89-110: camera ray, not null-normalised */
__global__ void __launch_bounds__(128)
dyst_icond_kernel(const RenderParams p, const GridParams g, double *__restrict__ data,
                  double *__restrict__ info)
{
	const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if(r >= p.n_rays)
		return;
	const long long gi = r % p.w_rays;
	const long long gj = p.row0 + r / p.w_rays;
	double alpha = (((double)gi + 0.5) / (double)p.w_rays - 0.5) * p.w_img;
	double beta  = (((double)gj + 0.5) / (double)p.h_rays - 0.5) * p.h_img;
	double R0 = fma(p.r_obs, p.si, -(beta * p.ci));
	double z  = fma(p.r_obs, p.ci, beta * p.si);
	double y  = fma(R0, p.sj, alpha * p.cj);
	double x  = fma(R0, p.cj, -(alpha * p.sj));
	double s[8] = {0.0, x, y, z, 1.0, p.si * p.cj, p.si * p.sj, p.ci};
	const long long n = p.n_rays;
#pragma unroll
	for(int c = 0; c < 8; ++c)
		data[c * n + r] = s[c];
	for(int c = 8; c < p.n_data; ++c)
		data[c * n + r] = 0.0; /* rt_icond(), rt.cl:179-183 */
	info[r] = dyst_getuu64(g, s);
}

/* ------------------------------------------ the evolution, lanes per ray */

/* Lane m of a ray's four lanes (eight with two time levels, four per level)
 * owns x^m, u^m and row m of Gamma: the ten Gamma^m_ab of the cell's 8
 * corners stay in 160 registers as doubles until the ray enters another
 * cell; with transfer also, as floats, the four fields of extra_field().
 * Every value is computed by the operations of interp.cl and dyst.cl in the
 * oracle's order, so results are bit-identical to one ray per thread. */
template <bool RT>
struct Cell64L {
	double G[8][10];
	float W[RT ? 8 : 1][RT ? 4 : 1];
};

/* row m of g on lanes 0 and 3 (k_t, k_z: all the transfer reads; g_zz from
 * g_yz where the flag says so, dyst.cl:78), rho on lane 1 */
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
load_cell64(const GridParams &g, const float *lvl, int m, int ix, int iy, int iz, Cell64L<RT> &C)
{
#pragma unroll
	for(int c = 0; c < 8; ++c) {
		const int x = (c & 1) ? min(ix + 1, g.nx - 1) : ix;
		const int y = (c & 2) ? min(iy + 1, g.ny - 1) : iy;
		const int z = (c & 4) ? min(iz + 1, g.nz - 1) : iz;
		const float *a = lvl + (((long long)z * g.ny + y) * g.nx + x) * GRAY_NSTRIDE;
		/* 10 m floats into a 224-byte row: 8-byte aligned */
		const float2 *ga = (const float2 *)(a + 10 * m);
#pragma unroll
		for(int k = 0; k < 5; ++k) {
			const float2 v = __ldg(ga + k);
			C.G[c][2 * k] = (double)v.x;
			C.G[c][2 * k + 1] = (double)v.y;
		}
		if constexpr(RT) {
#pragma unroll
			for(int k = 0; k < 4; ++k) {
				const int f = extra_field(m, k, g.bug_gzz);
				C.W[c][k] = f >= 0 ? __ldg(a + f) : 0.0f;
			}
		}
	}
}

/* A lane's axis (lane 0: time).  While x^m is in [xa, xb) the cell held is
 * the one axis_uvw64() finds: the cell less a millionth of its width at each
 * end (its own rounding is below 1e-10 of it), cut to the box. */
struct Axis64 {
	double x0, dx, ci; /* first node, width, index; lane 0: t1, t2 - t1, 0 */
	double xa, xb;
	int tag;           /* the cell index loaded; lane 0: unused (0)      */
};

/* The ray left its cell, or entered or left the box.  Returns w. */
template <int LV, bool RT>
__device__ __forceinline__ double
enter_cell64(const GridParams &g, Axis64 &A, Cell64L<RT> &C, int lane, bool on, double xs, bool &in)
{
	constexpr int L = 4 * LV;
	const unsigned FULL = 0xffffffffu;
	const int m = lane & 3, l = (lane & (L - 1)) >> 2, first = lane & ~(L - 1);
	const double lo = (double)g.box[m], hi = (double)g.box[m + 4];
	in = true;
	if(g.physics) {
		const unsigned out = __ballot_sync(FULL, m > 0 && !(xs >= lo && xs <= hi));
		in = ((out >> first) & ((1u << L) - 1u)) == 0;
	}
	const bool need = on && in;
	double w = 0.0;
	int i0 = 0;
	if(need && m > 0) {
		const int n = m == 1 ? g.nx : m == 2 ? g.ny : g.nz;
		const double u = axis_uvw64(g, m - 1, xs);
		const double fl = floor(u);
		i0 = (int)fl;
		w = u - fl;
		const int i = min(i0, n - 2);
		const double x0 = g.nodes[m - 1][i], x1 = g.nodes[m - 1][i + 1];
		const double mg = 1e-6 * (x1 - x0);
		A.x0 = x0;
		A.dx = x1 - x0;
		A.ci = fl;
		A.xa = x0 + mg;
		A.xb = x1 - mg;
		if(!(xs >= x0) || i0 > i) { /* clamped to the first or last node: w = 0 */
			A.x0 = 0.0;
			A.dx = INFINITY;
			A.xa = i0 > i ? x1 + mg : -INFINITY;
			A.xb = i0 > i ? INFINITY : i0 == 0 ? x0 - mg : -INFINITY;
		}
		if(g.physics) {
			A.xa = fmax(A.xa, lo);
			A.xb = fmin(A.xb, hi);
		}
	} else if(need) {
		A.xa = -INFINITY; /* a NaN time still takes this way */
		A.xb = INFINITY;
	}
	const unsigned moved = __ballot_sync(FULL, need && A.tag != i0);
	if(moved) {
		const int ix = __shfl_sync(FULL, i0, 1, 4), iy = __shfl_sync(FULL, i0, 2, 4),
		          iz = __shfl_sync(FULL, i0, 3, 4);
		if((moved >> first) & ((1u << L) - 1u)) {
			A.tag = i0;
			load_cell64<RT>(g, g.lvl[l], m, ix, iy, iz, C);
		}
	}
	return w;
}

/* du^m of dyst.cl:112-194 on lane m, and with RT kn = {k_t, k_z, n_e}
 * (dyst.cl:55-81).  All lanes take part; `on` marks the rays that step, in:
 * inside the box (or no box), all: so are all of them, in the cells held. */
template <int LV, bool RT>
__device__ __forceinline__ double
dyst_accel64(const GridParams &g, Axis64 &A, Cell64L<RT> &C, int lane, bool on, double xs,
             double us, double *kn, bool &in, bool &all)
{
	constexpr int L = 4 * LV;
	const unsigned FULL = 0xffffffffu;
	const int m = lane & 3;
	double u[4];
#pragma unroll
	for(int k = 0; k < 4; ++k)
		u[k] = __shfl_sync(FULL, us, k, 4);
	in = true;
	all = __all_sync(FULL, !on || (xs >= A.xa && xs < A.xb));
	double w = 0.0;
	if(LV == 2 || m > 0) {
		/* interp.cl:123-164 within the cell; lane 0: the time factor */
		const double q = (xs - A.x0) / A.dx;
		w = m > 0 ? (A.ci + q) - A.ci : q;
	}
	if(!all) {
		const double we = enter_cell64<LV, RT>(g, A, C, lane, on, xs, in);
		w = m > 0 ? we : w;
	}
	double ft = 0.0;
	if(LV == 2) {
		ft = __shfl_sync(FULL, w, 0, 4);
		if(g.physics) {
			if(!(ft >= 0.0))
				ft = 0.0;
			if(ft > 1.0)
				ft = 1.0;
		}
	}
	const double wx = __shfl_sync(FULL, w, 1, 4), wy = __shfl_sync(FULL, w, 2, 4),
	             wz = __shfl_sync(FULL, w, 3, 4);
	const double ax = 1.0 - wx, ay = 1.0 - wy, az = 1.0 - wz;
	double wc[8];
#pragma unroll
	for(int c = 0; c < 8; ++c)
		wc[c] = (((c & 1) ? wx : ax) * ((c & 2) ? wy : ay)) * ((c & 4) ? wz : az);
	/* trilinear (corner order 000, 100, 010, ...), then linear in time, then
	 * the contraction; with two levels the other level's value comes from
	 * the ray's other four lanes, and level 0's lanes go on */
	auto in_time = [&](double y) {
		if(LV == 1)
			return y;
		const double y2 = __shfl_xor_sync(FULL, y, 4);
		return fma(ft, y2 - y, y);
	};
	double G = 0.0;
	int k = 0;
#pragma unroll
	for(int i = 0; i < 4; ++i)
#pragma unroll
		for(int j = i; j < 4; ++j) {
			const double uu = u[i] * u[j];
			const double p = i == j ? uu : 2.0 * uu;
			double v = wc[0] * C.G[0][k];
#pragma unroll
			for(int c = 1; c < 8; ++c)
				v = fma(wc[c], C.G[c][k], v);
			v = in_time(v);
			G = k ? fma(v, p, G) : v * p;
			++k;
		}
	if constexpr(RT) {
		double e[4];
#pragma unroll
		for(int q = 0; q < 4; ++q) {
			double v = wc[0] * (double)C.W[0][q];
#pragma unroll
			for(int c = 1; c < 8; ++c)
				v = fma(wc[c], (double)C.W[c][q], v);
			e[q] = in_time(v);
		}
		const double kk = fma(e[3], u[3], fma(e[2], u[2], fma(e[1], u[1], e[0] * u[0])));
		kn[0] = __shfl_sync(FULL, kk, 0, L);
		kn[1] = __shfl_sync(FULL, kk, 3, L);
		kn[2] = __shfl_sync(FULL, e[0], 1, L);
	}
	if(LV == 2)
		G = __shfl_sync(FULL, G, m, L);
	const double G0 = __shfl_sync(FULL, G, 0, L);
	return fma(G0, us, -G);
}

/* Outside the box (physics mode) u is constant and a step only moves x: a
 * chunk of steps as one loop, as many as every ray of the warp surely stays
 * outside (its distance to the box on some axis less 1%, and two steps for
 * the stage positions) and short of the interval's last step. */
__device__ __forceinline__ int
flat_chunk64(const GridParams &g, int m, bool step, double x, double dx, int left)
{
	const unsigned FULL = 0xffffffffu;
	const double lo = (double)g.box[m], hi = (double)g.box[m + 4];
	const float d = m ? (float)fmax(lo - x, x - hi) : 0.0f;
	float far = d > 0.0f ? fminf(0.99f * d / ((float)fabs(dx) + 1e-30f), 1e6f) - 2.0f : 0.0f;
	far = fmaxf(far, __shfl_xor_sync(FULL, far, 1));
	far = fmaxf(far, __shfl_xor_sync(FULL, far, 2));
	/* NaN or infinite slopes take the general step */
	int todo = far >= 1.0f && fabs(dx) < 1e30 ? min((int)far, left) : 0;
	todo = __reduce_min_sync(FULL, step ? todo : INT_MAX);
	return todo == INT_MAX ? 0 : todo;
}

/* RK4 of a ray's (I, tau) over a step of hs (rt.cl:185-198 with getflow() of
 * flow.cl:36-58), given on lane m k_t, k_z and n_e at stage m: what a stage
 * emits and absorbs depends on the geodesic alone, so lane m evaluates stage
 * m, a frequency per pass (two with eight lanes), and only e^-tau chains the
 * stages.  Frequency f is kept by lane (f / LV) % 4 of half f % LV. */
template <int LV, int FPL>
__device__ __forceinline__ void
transfer64(const RenderParams &p, int lane, double hs, double h6, double kt, double kz, double ne,
           double *I, double *tau)
{
	const unsigned FULL = 0xffffffffu;
	const int m = lane & 3, l = LV == 2 ? (lane >> 2) & 1 : 0;
	const double shift = -kt;
	const double bkcos = (kz * p.flow_b) / (shift * p.flow_b + thermal::EPS);
	const double cd = m == 3 ? hs : 0.5 * hs;
#pragma unroll
	for(int i = 0; i < FPL; ++i)
#pragma unroll 1
		for(int q = 0; q < 4; ++q) {
			const int f = LV * (4 * i + q) + l;
			if(LV * (4 * i + q) >= p.n_freq)
				break;
			const double nu = p.nu[f < p.n_freq ? f : 0] * shift;
			const double B = thermal::B_Planck(nu, p.flow_te);
			const double nL = -(thermal::L_j_syn(p.th, p.m_adm, nu, p.flow_te, ne, p.flow_b, bkcos) +
			                    thermal::L_j_ff(p.th, p.m_adm, nu, p.flow_te, ne));
			const double dt = nL * shift / (B + thermal::EPS);
			const double t0 = __shfl_sync(FULL, tau[i], q, 4);
			const double before = __shfl_up_sync(FULL, dt, 1, 4);
			const double st = m ? fma(cd, before, t0) : t0;
			const double dI = nL * exp(-st) / (shift * shift + thermal::EPS);
			double kI[4], kT[4];
#pragma unroll
			for(int k = 0; k < 4; ++k) {
				kI[k] = __shfl_sync(FULL, dI, k, 4);
				kT[k] = __shfl_sync(FULL, dt, k, 4);
			}
			if(m == q && f < p.n_freq) {
				I[i] = fma(h6, fma(2.0, kI[1] + kI[2], kI[0]) + kI[3], I[i]);
				tau[i] = fma(h6, fma(2.0, kT[1] + kT[2], kT[0]) + kT[3], tau[i]);
			}
		}
}

constexpr int BLOCK64 = 64;

/* driver.cl:69-108 on the numerical spacetime over one dump interval of
 * length dt; FPL: frequencies per lane (0: geodesics alone).
 *
 * What bounds it: the FP64 pipe (126 operations per lane and RHS, 80 of them
 * the interpolation of a lane's ten Gamma) at 8 warps per SM, and with
 * transfer the emissivities' exp, log and cbrt.  Measured, one ray per thread
 * before and four (two levels: eight) lanes now: 256 x 200 rays in one level
 * 65.5 -> 13.0 ms, 64 x 48 rays between two levels 92.1 -> 2.8 ms, with one
 * frequency 130.5 -> 8.5 ms (14.6 with a frequency per lane).  Before, every RHS converted 320 floats a ray
 * to double and searched each axis with cbrt and asinh. */
template <int LV, int FPL>
__global__ void __launch_bounds__(BLOCK64, 4)
dyst_evolve64_kernel(const __grid_constant__ RenderParams p, const __grid_constant__ GridParams g,
                     double *__restrict__ data, double *__restrict__ info, const double dt,
                     const long long n_sub, unsigned long long *__restrict__ steps)
{
	constexpr int L = 4 * LV;
	constexpr bool RT = FPL > 0;
	constexpr int STAGES = RT ? 1 : 4;
	constexpr int NR = RT ? FPL : 1;
	const unsigned FULL = 0xffffffffu;
	const int lane = threadIdx.x & 31, sub = lane & (L - 1), m = lane & 3;
	const int first = lane & ~(L - 1);
	const long long nr = p.n_rays;
	const long long r = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / L;
	const bool mine = r < nr;

	Cell64L<RT> C;
	Axis64 A;
	A.tag = -1;
	A.xa = INFINITY; /* empty */
	A.xb = A.ci = 0.0;
	A.x0 = (double)g.box[0];
	A.dx = (double)g.box[4] - (double)g.box[0];
#pragma unroll
	for(int c = 0; c < 8; ++c) {
#pragma unroll
		for(int k = 0; k < 10; ++k)
			C.G[c][k] = 0.0;
		if constexpr(RT)
#pragma unroll
			for(int k = 0; k < 4; ++k)
				C.W[c][k] = 0.0f;
	}
	/* (I, tau) of the frequencies this lane keeps: own(0), own(1) */
	auto own = [&](int i) { return LV * (4 * i + m) + (sub >> 2); };
	double x = 0.0, u = 0.0, I[NR], tau[NR];
	if(mine) {
		x = data[m * nr + r];
		u = data[(4 + m) * nr + r];
	}
#pragma unroll
	for(int i = 0; i < NR; ++i) {
		const int f = own(i) < p.n_freq ? own(i) : 0;
		I[i] = tau[i] = 0.0;
		if(RT && mine) {
			I[i] = data[(8 + f) * nr + r];
			tau[i] = data[(8 + p.n_freq + f) * nr + r];
		}
	}
	const int n = (int)((INT_MAX / n_sub) * n_sub);
	const double dts = dt / (double)n_sub;
	const int dh_step = (int)(dyst_getdt64(dts) / dt * (double)n);
	unsigned cnt = 0;
	bool quiet = false; /* every ray of the warp stayed in its cell and the box */
	for(int h = 0; h < n && dh_step != 0;) {
		const int dh = dh_step > n - h ? n - h : dh_step;
		const double hs = ((double)dh * dt) / (double)n, hh = 0.5 * hs;
		const double h6 = hs / 6.0;
		bool out = false; /* in flat space all step long */
		if(g.physics && !quiet) {
			const double lo = (double)g.box[m], hi = (double)g.box[m + 4];
			auto outside = [&](double q) {
				const unsigned b = __ballot_sync(FULL, m > 0 && !(q >= lo && q <= hi));
				return ((b >> first) & ((1u << L) - 1u)) != 0;
			};
			const bool o1 = outside(x), o2 = outside(fma(hh, u, x)), o4 = outside(fma(hs, u, x));
			out = o1 && o2 && o4;
			if(__all_sync(FULL, !mine || out)) {
				const double k = fma(2.0, u + u, u) + u;
				const int todo = flat_chunk64(g, m, mine, x, hs * u,
				                              dh == dh_step ? (n - h - 1) / dh_step : 0);
				for(int i = 0; i < todo; ++i)
					x = fma(h6, k, x);
				cnt += todo;
				h += todo * dh_step;
				if(todo)
					continue;
			}
		}
		double xq = x, uq = u, kx1 = 0.0, ku1 = 0.0, kx2 = 0.0, ku2 = 0.0, kx = 0.0, ku = 0.0;
		double kt = 0.0, kz = 0.0, ne = 0.0; /* stage m's */
		quiet = true;
#pragma unroll STAGES
		for(int s = 0; s < 4; ++s) {
			double kn[3];
			bool in = true, all = true;
			kx = uq;
			ku = dyst_accel64<LV, RT>(g, A, C, lane, mine && !out, xq, uq, kn, in, all);
			in = in && !out;
			quiet = quiet && all;
			ku = in ? ku : 0.0;
			if(RT && s == m) {
				/* flat space, empty, outside */
				kt = in ? kn[0] : -1.0;
				kz = in ? kn[1] : 0.0;
				ne = in ? kn[2] : 0.0;
			}
			const double cg = s < 2 ? hh : hs;
			if(s == 0) {
				kx1 = kx;
				ku1 = ku;
			} else if(s < 3) { /* k2 + k3 */
				kx2 = s == 1 ? kx : kx2 + kx;
				ku2 = s == 1 ? ku : ku2 + ku;
			}
			xq = fma(cg, kx, x);
			uq = fma(cg, ku, u);
		}
		quiet = quiet && __all_sync(FULL, !out);
		/* RK4.cl:37-47 */
		x = fma(h6, fma(2.0, kx2, kx1) + kx, x);
		u = fma(h6, fma(2.0, ku2, ku1) + ku, u);
		if constexpr(RT)
			transfer64<LV, FPL>(p, lane, hs, h6, kt, kz, ne, I, tau);
		++cnt;
		h += dh;
	}
	double s[8];
#pragma unroll
	for(int k = 0; k < 4; ++k) {
		s[k] = __shfl_sync(FULL, x, k, 4);
		s[4 + k] = __shfl_sync(FULL, u, k, 4);
	}
	if(mine) {
		if(sub < 4) {
			data[m * nr + r] = x;
			data[(4 + m) * nr + r] = u;
		}
		if constexpr(RT) {
#pragma unroll
			for(int i = 0; i < NR; ++i)
				if(own(i) < p.n_freq) {
					data[(8 + own(i)) * nr + r] = I[i];
					data[(8 + p.n_freq + own(i)) * nr + r] = tau[i];
				}
		}
		if(sub == 0)
			info[r] = dyst_getuu64(g, s);
	}
	unsigned long long total = mine && sub == 0 ? cnt : 0;
#pragma unroll
	for(int o = 16; o > 0; o >>= 1)
		total += __shfl_xor_sync(FULL, total, o);
	if(lane == 0 && total)
		atomicAdd(steps, total);
}

/* ------------------------------------------------------- boosted KS grid */

struct Dual {
	double f, s;
};
__device__ __forceinline__ Dual D(double f, double s) { Dual r = {f, s}; return r; }
__device__ __forceinline__ Dual operator+(Dual a, Dual b) { return D(a.f + b.f, a.s + b.s); }
__device__ __forceinline__ Dual operator-(Dual a, Dual b) { return D(a.f - b.f, a.s - b.s); }
__device__ __forceinline__ Dual operator*(Dual a, Dual b) { return D(a.f * b.f, a.s * b.f + a.f * b.s); }
__device__ __forceinline__ Dual operator*(Dual a, double c) { return D(a.f * c, a.s * c); }
__device__ __forceinline__ Dual operator/(Dual a, Dual b)
{
	return D(a.f / b.f, (a.s * b.f - a.f * b.s) / (b.f * b.f));
}
__device__ __forceinline__ Dual dsqrt(Dual a)
{
	double r = sqrt(a.f);
	return D(r, a.s * 0.5 / r);
}

/* boosted_ks.py:120-186: h and covariant l_mu at X (dual numbers) */
__device__ void
bks_hl(double m, double a, double v, int axis, const Dual *X, Dual &h, Dual *l)
{
	double gam = 1.0 / sqrt(1.0 - v * v);
	Dual x0[4] = {X[0], X[1], X[2], X[3]};
	x0[0]    = (X[0] - X[axis] * v) * gam;
	x0[axis] = (X[axis] - X[0] * v) * gam;
	Dual xx = x0[1], yy = x0[2], zz = x0[3];
	Dual rho2 = xx * xx + yy * yy + zz * zz;
	Dual w = rho2 - D(a * a, 0.0);
	Dual r2 = w * 0.5 + dsqrt(w * w * 0.25 + zz * zz * (a * a));
	Dual r = dsqrt(r2);
	Dual ct = zz / r;
	h = (r * m) / (r2 + ct * ct * (a * a));
	Dual ra2 = r2 + D(a * a, 0.0);
	Dual l0[4] = {D(1.0, 0.0), (r * xx + yy * a) / ra2, (r * yy - xx * a) / ra2, zz / r};
	for(int c = 0; c < 4; ++c)
		l[c] = l0[c];
	l[0]    = (l0[0] - l0[axis] * v) * gam;
	l[axis] = (l0[axis] - l0[0] * v) * gam;
}

/* numpy.nan_to_num then float32 (tools/generate_data.py:143-144) */
__device__ __forceinline__ float
to_f32(double x)
{
	if(x != x)
		return 0.0f;
	return (float)x;
}

__global__ void __launch_bounds__(128)
boosted_ks_kernel(const GridParams g, float *__restrict__ lvl, double m, double a,
                  double v, int axis, double t)
{
	const long long npts = (long long)g.nx * g.ny * g.nz;
	const long long pt = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if(pt >= npts)
		return;
	const int ix = (int)(pt % g.nx);
	const int iy = (int)((pt / g.nx) % g.ny);
	const int iz = (int)(pt / ((long long)g.nx * g.ny));
	const double q[4] = {t, g.nodes[0][ix], g.nodes[1][iy], g.nodes[2][iz]};
	const double ETA[4] = {-1.0, 1.0, 1.0, 1.0};
	double dg[4][4][4], gd[4][4], gu[4][4];
	for(int w = 0; w < 4; ++w) {
		Dual X[4], h, l[4];
		for(int c = 0; c < 4; ++c)
			X[c] = D(q[c], c == w ? 1.0 : 0.0);
		bks_hl(m, a, v, axis, X, h, l);
		for(int i = 0; i < 4; ++i)
			for(int j = 0; j < 4; ++j) {
				Dual gij = h * (l[i] * l[j]) * 2.0;
				dg[w][i][j] = gij.s;
				if(w == 0) {
					gd[i][j] = (i == j ? ETA[i] : 0.0) + gij.f;
					double li = i == 0 ? -l[0].f : l[i].f;
					double lj = j == 0 ? -l[0].f : l[j].f;
					gu[i][j] = (i == j ? ETA[i] : 0.0) - 2.0 * h.f * li * lj;
				}
			}
	}
	float *out = lvl + pt * GRAY_NSTRIDE;
	int k = 0;
	for(int i = 0; i < 4; ++i)
		for(int b = 0; b < 4; ++b)
			for(int c = b; c < 4; ++c) {
				double s = 0.0;
				for(int mm = 0; mm < 4; ++mm)
					s += gu[i][mm] * (dg[c][mm][b] + dg[b][mm][c] - dg[mm][b][c]);
				out[k++] = to_f32(0.5 * s);
			}
	for(int i = 0; i < 4; ++i)
		for(int j = i; j < 4; ++j)
			out[k++] = to_f32(gd[i][j]);
	/* generate_data.py:124-128: rho = 1 / r */
	out[50] = to_f32(1.0 / sqrt(q[1] * q[1] + q[2] * q[2] + q[3] * q[3]));
	for(int pad = GRAY_NCOMP; pad < GRAY_NSTRIDE; ++pad)
		out[pad] = 0.0f;
}

inline unsigned
blocks_for(long long n, int block)
{
	return (unsigned)((n + block - 1) / block);
}

} /* namespace */

cudaError_t
launch_dyst_icond(const RenderParams &p, const GridParams &g, double *data, double *info,
                  cudaStream_t st)
{
	dyst_icond_kernel<<<blocks_for(p.n_rays, 128), 128, 0, st>>>(p, g, data, info);
	return cudaGetLastError();
}

cudaError_t
launch_dyst_evolve64(const RenderParams &p, const GridParams &g, double *data, double *info,
                     double dt, long long n_sub, unsigned long long *steps, cudaStream_t st)
{
	if(p.n_freq < 0 || p.n_freq > GRAY_MAX_FREQ)
		return cudaErrorInvalidValue;
	/* an interval whose ends round to the same time has no step count
	 * (driver.cl:93 divides by its length) and leaves the state as it is */
	if(!(fabs(dt) > 0.0))
		return cudaSuccess;
	const int lanes = g.single ? 4 : 8;
	/* one warp per block: a small render's warps spread over every SM */
	const int block = p.n_rays * lanes > 148 * 4 * 32 ? BLOCK64 : 32;
	const unsigned nb = blocks_for(p.n_rays * lanes, block);
#define GRAY_DYST64(LV, FPL) \
	dyst_evolve64_kernel<LV, FPL><<<nb, block, 0, st>>>(p, g, data, info, dt, n_sub, steps)
	if(!g.single) {
		if(p.n_freq == 0)
			GRAY_DYST64(2, 0);
		else
			GRAY_DYST64(2, 1);
	} else if(p.n_freq == 0) {
		GRAY_DYST64(1, 0);
	} else if(p.n_freq <= 4) {
		GRAY_DYST64(1, 1);
	} else {
		GRAY_DYST64(1, 2);
	}
#undef GRAY_DYST64
	return cudaGetLastError();
}

cudaError_t
launch_boosted_ks(const GridParams &g, float *lvl, double a, double v, int axis, double t,
                  cudaStream_t st)
{
	const long long npts = (long long)g.nx * g.ny * g.nz;
	boosted_ks_kernel<<<blocks_for(npts, 128), 128, 0, st>>>(g, lvl, 1.0, a, v, axis, t);
	return cudaGetLastError();
}
