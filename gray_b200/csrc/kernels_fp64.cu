/*
 * Plain FP64 kernels: one ray per thread, SoA state, the substep loop of the
 * reference's evolve_drv (driver.cl:69-108) over one dump interval or all of
 * them.  This is the FP64 baseline the mixed-precision path is measured
 * against, and the kernel that must agree with the CPU oracle to 1e-10.
 *
 * Rounding contract: this translation unit is compiled with -fmad=false,
 * so the only fused multiply-adds are the explicit fma() calls below; they
 * sit exactly where the oracle (oracle/gray_oracle.c) places its fma()
 * calls.  FP64 '/' and sqrt() are IEEE round-to-nearest on sm_100, as in
 * the oracle, so the geodesic agrees bit for bit; the stepping loop's own
 * quotients and roots (round64.cuh) round the same.
 */
#include <climits>

#include "gray_internal.h"
#include "round64.cuh"

namespace {

using namespace round64;

constexpr int EVOLVE64_BLOCK = 64;

/* KS.cl:48-55 getrr() */
__device__ __forceinline__ double
getrr64(const RenderParams &p, double x, double y, double z)
{
	double zz = z * z;
	double kk = 0.5 * (fma(x, x, fma(y, y, zz)) - p.aa);
	return sqrt(fma(kk, kk, p.aa * zz)) + kk;
}

/* The radius at an event (KS.cl:48-55, 289-295): what the step rule and the
 * first RHS of a step share.  Valid where in_range(). */
struct Rad64 {
	double zz, dd, rr, r;
	double hd, yr, yq; /* about 1/(2 dd), 1/r; within 2^-18 of 1/rr */
	bool ones;         /* all_ones() of a radicand           */
};

/* where every operand of the loop's quotients and roots is normal with room
 * to spare: r^2/2 <= sqrt(k^2 + a^2 z^2) <= r^2 + 1 and r^2 <= r^2 + a^2
 * (rays outside the horizon have r > 1).  k >= 0 (r^2 >= dd; everywhere
 * outside the sphere r = |a|) keeps dd + k from cancelling. */
__device__ __forceinline__ bool
in_range(const Rad64 &R)
{
	return R.rr > 1e-6 && R.rr < 1e60 && R.rr >= R.dd && !R.ones;
}

/* A lone warp's step is one chain of dependent operations, and the seeds of
 * r's root and of 1/r^2 stood in it: both come from r^2 to 2^-19, known
 * before its own root is refined.  With 1/(r^2 + a^2 z^2 / r^2) from the
 * root's own 1/(2 dd): 64^2 rays dump by dump 140.4 -> 129.8 ms (other
 * cameras 124.6 -> 115.1), 251 x 190 rays with 4 frequencies 96.7 -> 93.5
 * (bit-identical). */
__device__ __forceinline__ Rad64
radius64(const RenderParams &p, double x, double y, double z)
{
	Rad64 R;
	R.zz = z * z;
	const double kk = 0.5 * (fma(x, x, fma(y, y, R.zz)) - p.aa);
	const double d2 = fma(kk, kk, p.aa * R.zz), y0 = seed_rsqrt(d2);
	const double about = fma(d2, y0, kk);
	const double yr = seed_rsqrt(about);
	R.yq = seed_rcp(about);
	R.dd = sqrt_from(d2, y0, R.hd);
	R.rr = R.dd + kk;
	double hr;
	R.r = sqrt_from(R.rr, yr, hr);
	R.yr = hr + hr;
	R.ones = all_ones(d2) | all_ones(R.rr);
	return R;
}

struct Aux64 {
	double r, f, lx, ly, lz, flu, iss, ir;
	bool ones; /* all_ones() of a divisor */
};

/* KS.cl:263-378 gr_rhs(), Chan et al. form; returns f, l and f l.u for the
 * transfer step (phys.cl:70 down() reuses them). */
template <bool ANY>
__device__ __forceinline__ void
ks_rhs64(const RenderParams &p, const Rad64 &R, const double *s, double *ds, Aux64 &aux)
{
	const double a = p.a;
	const double x = s[1], y = s[2], z = s[3];
	const double ut = s[4], ux = s[5], uy = s[6], uz = s[7];

	double f, dx_f, dy_f, dz_f;
	double lx, dx_lx, dy_lx, dz_lx;
	double ly, dx_ly, dy_ly, dz_ly;
	double lz, dx_lz, dy_lz, dz_lz;
	double dx_r, dy_r, dz_r, ir, iss, tmp;
	const double r = R.r;
	{
		const double aa = p.aa, zz = R.zz, dd = R.dd, rr = R.rr;
		const double ss = rr + aa, rd = r * dd, az = aa * zz;
		double hrd, t2; /* 0.5 / (r dd), 2 / (rr + aa zz / rr) */
		if constexpr(ANY) {
			ir  = 1.0 / r;
			iss = 1.0 / ss;
			hrd = 0.5 / rd;
			t2  = 2.0 / (rr + az / rr);
			aux.ones = false;
		} else {
			/* a power of 2 over b is that power of 1/b, exactly; 1/rr from
			 * its own seed, so that it does not wait for the root; and
			 * rr + az / rr is 2 dd but for rounding (az = dd^2 - kk^2) */
			ir  = rcp_near(r, R.yr);
			iss = rcp_rn(ss);
			hrd = 0.5 * rcp_near(rd, rcp_near(rd, R.yr * (R.hd + R.hd)));
			const double den = rr + div_rn(az, rr, rcp_near(rr, rcp_from(rr, R.yq)));
			t2  = 2.0 * rcp_near(den, rcp_near(den, R.hd));
			aux.ones = all_ones(ss) | all_ones(rd) | all_ones(den);
		}
		tmp  = hrd;
		dz_r = (tmp * ss) * z;
		tmp  = tmp * rr;
		dy_r = tmp * y;
		dx_r = tmp * x;
		tmp  = t2;
		double tmp2 = fma(-2.0 * rr, tmp, 3.0);
		f    = tmp * r;
		dx_f = (tmp * dx_r) * tmp2;
		dy_f = (tmp * dy_r) * tmp2;
		dz_f = tmp * fma(dz_r, tmp2, -(((tmp * aa) * z) * ir));
	}
	{
		double m2r  = -2.0 * r;
		double issr = iss * r;
		double issa = iss * a;

		lx    = iss * fma(x, r, y * a);
		tmp   = iss * fma(m2r, lx, x);
		dx_lx = fma(tmp, dx_r, issr);
		dy_lx = fma(tmp, dy_r, issa);
		dz_lx = tmp * dz_r;

		ly    = iss * fma(y, r, -(x * a));
		tmp   = iss * fma(m2r, ly, y);
		dx_ly = fma(tmp, dx_r, -issa);
		dy_ly = fma(tmp, dy_r, issr);
		dz_ly = tmp * dz_r;

		lz    = z * ir;
		tmp   = -lz * ir;
		dx_lz = tmp * dx_r;
		dy_lz = tmp * dy_r;
		dz_lz = fma(tmp, dz_r, ir);
	}
	double lu  = fma(lz, uz, fma(ly, uy, fma(lx, ux, ut)));
	double flu = f * lu;
	double Dx0 = fma(dx_f, lu, f * fma(dx_lz, uz, fma(dx_ly, uy, dx_lx * ux)));
	double Dy0 = fma(dy_f, lu, f * fma(dy_lz, uz, fma(dy_ly, uy, dy_lx * ux)));
	double Dz0 = fma(dz_f, lu, f * fma(dz_lz, uz, fma(dz_ly, uy, dz_lx * ux)));

	double Dx1 = fma(Dx0, lx, flu * dx_lx);
	double Dx2 = fma(Dx0, ly, flu * dx_ly);
	double Dx3 = fma(Dx0, lz, flu * dx_lz);

	double Dy1 = fma(Dy0, lx, flu * dy_lx);
	double Dy2 = fma(Dy0, ly, flu * dy_ly);
	double Dy3 = fma(Dy0, lz, flu * dy_lz);

	double Dz1 = fma(Dz0, lx, flu * dz_lx);
	double Dz2 = fma(Dz0, ly, flu * dz_ly);
	double Dz3 = fma(Dz0, lz, flu * dz_lz);

	double hDxu = 0.5 * fma(Dx3, uz, fma(Dx2, uy, fma(Dx1, ux, Dx0 * ut)));
	double hDyu = 0.5 * fma(Dy3, uz, fma(Dy2, uy, fma(Dy1, ux, Dy0 * ut)));
	double hDzu = 0.5 * fma(Dz3, uz, fma(Dz2, uy, fma(Dz1, ux, Dz0 * ut)));

	double uD0 = fma(uz, Dz0, fma(uy, Dy0, ux * Dx0));
	double uD1 = fma(uz, Dz1, fma(uy, Dy1, ux * Dx1));
	double uD2 = fma(uz, Dz2, fma(uy, Dy2, ux * Dx2));
	double uD3 = fma(uz, Dz3, fma(uy, Dy3, ux * Dx3));

	tmp = f * fma(lz, uD3 - hDzu, fma(ly, uD2 - hDyu, fma(lx, uD1 - hDxu, -uD0)));

	ds[0] = ut;
	ds[1] = ux;
	ds[2] = uy;
	ds[3] = uz;
	ds[4] = uD0 - tmp;
	ds[5] = fma(lx, tmp, hDxu - uD1);
	ds[6] = fma(ly, tmp, hDyu - uD2);
	ds[7] = fma(lz, tmp, hDzu - uD3);

	aux.r = r; aux.f = f; aux.lx = lx; aux.ly = ly; aux.lz = lz;
	aux.flu = flu; aux.iss = iss; aux.ir = ir;
}

/* Torus flow + transfer in the rt.cl:185-198 form (see the oracle's
 * torus_rt() for the model): any operands. */
template <int NF>
__device__ __noinline__ void
torus_any64(const RenderParams &p, const double *s, const Aux64 &x, double *ds)
{
	double n = 0.0, shift = 1.0;
	if(x.r > p.risco && p.flow == GRAY_FLOW_TORUS) {
		const double q1 = s[1], q2 = s[2], q3 = s[3];
		double kt = x.flu - s[4];
		double kx = fma(x.flu, x.lx, s[5]);
		double ky = fma(x.flu, x.ly, s[6]);
		double R2 = fma(q1, q1, q2 * q2);
		double Om = 1.0 / fma(x.r, sqrt(x.r), p.a);
		double vv = fma(Om * Om, R2, -1.0);
		double lv = fma(-((p.a * Om) * R2), x.iss, 1.0);
		double D  = -fma(x.f * lv, lv, vv);
		if(D > 0.0) {
			double utf = 1.0 / sqrt(D);
			shift = -utf * fma(Om, fma(q1, ky, -(q2 * kx)), kt);
			if(shift > 0.0) {
				double qr = p.rp / x.r;
				double hz = p.torus_hr * x.r;
				n = ((p.torus_n0 * qr) * sqrt(qr)) *
				    exp(-((q3 * q3) / ((2.0 * hz) * hz)));
			}
		}
	}
	if(n == 0.0) {
		for(int i = 0; i < 2 * NF; ++i)
			ds[i] = 0.0;
		return;
	}
	double ish  = 1.0 / shift;
	double jfac = n * pow(shift, -0.7);
	double tfac = (p.torus_kappa * n) * ish;
	double is2  = 1.0 / fma(shift, shift, GRAY_EPSILON);
	for(int i = 0; i < NF; ++i) {
		double j = jfac * p.nupow[i];
		ds[i]      = -(j * exp(-s[8 + NF + i])) * is2;
		ds[NF + i] = -(tfac * p.nuinv2[i]);
	}
}

/* The same transfer with 1/r and its root shared: the density is n0 r_+^1.5
 * r^-1.5 e^-g, g = (z/r)^2 / (2 h_r^2).  What the shared factors add to the
 * rounding is carried along where it costs an operation or two (z/r rounded
 * to nearest, r^-1.5 and the render's constants with their low parts), so that
 * the mean error is not above that of the operators, pow and exp; one
 * exponential per frequency of the three exponents' sum had up to 1.3 times
 * theirs, as its error grows with its argument.  Returns whether its operands
 * were in the ranges this holds in, given ok of the RHS.  (With the operators,
 * transfer took three quarters of a step's time at four frequencies.) */
template <int NF>
__device__ __forceinline__ bool
torus_rt64(const RenderParams &p, bool ok, const double *s, const Aux64 &x, double *ds)
{
	bool emits = false;
	double shift = 1.0, n = 0.0, pw = 0.0, is2 = 0.0, ish = 0.0;
	if(x.r > p.risco && p.flow == GRAY_FLOW_TORUS) {
		const double q1 = s[1], q2 = s[2];
		const double kt = x.flu - s[4];
		const double kx = fma(x.flu, x.lx, s[5]);
		const double ky = fma(x.flu, x.ly, s[6]);
		const double R2 = fma(q1, q1, q2 * q2);
		double irs;
		const double sr = sqrt_rn(x.r, irs);
		const double Om = rcp_fast(fma(x.r, sr, p.a));
		const double vv = fma(Om * Om, R2, -1.0);
		const double lv = fma(-((p.a * Om) * R2), x.iss, 1.0);
		const double D = -fma(x.f * lv, lv, vv);
		double utf;
		sqrt_rn(D, utf);
		shift = -utf * fma(Om, fma(q1, ky, -(q2 * kx)), kt);
		emits = D > 0.0 && !(shift <= 0.0);
		ok = ok && (!emits || (D > 1e-30 && shift > 1e-9 && shift < 1e9));
		pw = pow_m07(shift);
		is2 = rcp_fast(fma(shift, shift, GRAY_EPSILON));
		ish = rcp_fast(shift);
		const double v = div_rn(s[3], x.r, x.ir), v2 = v * v;
		const double w = x.ir * irs, wl = fma(x.ir, irs, -w);
		const double g = fma(v2, p.torus_ig, v2 * p.torus_igl);
		n = fma(w, p.torus_n15, fma(w, p.torus_n15l, wl * p.torus_n15)) * exp(-g);
		emits = emits && n != 0.0;
	}
	if(!emits || !ok) {
#pragma unroll
		for(int i = 0; i < 2 * NF; ++i)
			ds[8 + i] = 0.0;
		return ok;
	}
	const double tfac = (p.torus_kappa * n) * ish;
	const double jfac = (n * is2) * pw;
#pragma unroll
	for(int i = 0; i < NF; ++i) {
		ds[8 + i]      = -((jfac * p.nupow[i]) * exp(-s[8 + NF + i]));
		ds[8 + NF + i] = -(tfac * p.nuinv2[i]);
	}
	return true;
}

/* phys.cl:66-74 rhs() at operands outside in_range(): the operators */
template <int NF>
__device__ __noinline__ void
rhs_any64(const RenderParams &p, const double *s, double *ds)
{
	Rad64 R;
	Aux64 aux;
	R.zz = s[3] * s[3];
	const double kk = 0.5 * (fma(s[1], s[1], fma(s[2], s[2], R.zz)) - p.aa);
	R.dd = sqrt(fma(kk, kk, p.aa * R.zz));
	R.rr = R.dd + kk;
	R.r = sqrt(R.rr);
	R.hd = R.yr = R.yq = 0.0;
	R.ones = false;
	ks_rhs64<true>(p, R, s, ds, aux);
	if constexpr(NF > 0)
		torus_any64<NF>(p, s, aux, ds + 8);
}

/* RK4.cl:37-47 integrate() by dt, h6 = dt / 6, with the operators */
template <int NF>
__device__ __noinline__ void
rk4_any64(const RenderParams &p, double *s, double dt, double h6)
{
	constexpr int ND = 8 + 2 * NF;
	double k1[ND], k2[ND], k[ND], t[ND];
	const double hdt = 0.5 * dt;
	rhs_any64<NF>(p, s, k1);
	for(int i = 0; i < ND; ++i) t[i] = fma(hdt, k1[i], s[i]);
	rhs_any64<NF>(p, t, k2);
	for(int i = 0; i < ND; ++i) t[i] = fma(hdt, k2[i], s[i]);
	rhs_any64<NF>(p, t, k);
	for(int i = 0; i < ND; ++i) {
		t[i] = fma(dt, k[i], s[i]);
		k2[i] = k2[i] + k[i];
	}
	rhs_any64<NF>(p, t, k);
	for(int i = 0; i < ND; ++i)
		s[i] = fma(h6, fma(2.0, k2[i], k1[i]) + k[i], s[i]);
}

/* phys.cl:66-74 rhs(); false: operands that the loop's own quotients and
 * roots do not hold for */
template <int NF>
__device__ __forceinline__ bool
rhs64(const RenderParams &p, const Rad64 &R, const double *s, double *ds)
{
	Aux64 aux;
	bool ok = in_range(R) && !all_ones(R.r);
	ks_rhs64<false>(p, R, s, ds, aux);
	if constexpr(NF > 0)
		ok = torus_rt64<NF>(p, ok, s, aux, ds);
	return ok && !aux.ones;
}

/* RK4.cl:37-47 integrate() by dt, h6 = dt / 6; R: the radius at s.  A step
 * that met such operands is taken again with the operators: asked once per
 * step, the question does not stand between the stages. */
template <int NF>
__device__ __forceinline__ void
rk4_64(const RenderParams &p, const Rad64 &R, double *s, double dt, double h6)
{
	constexpr int ND = 8 + 2 * NF;
	double k1[ND], k2[ND], k[ND], t[ND];
	const double hdt = 0.5 * dt;
	bool ok = rhs64<NF>(p, R, s, k1);
#pragma unroll
	for(int i = 0; i < ND; ++i) t[i] = fma(hdt, k1[i], s[i]);
	ok &= rhs64<NF>(p, radius64(p, t[1], t[2], t[3]), t, k2);
#pragma unroll
	for(int i = 0; i < ND; ++i) t[i] = fma(hdt, k2[i], s[i]);
	ok &= rhs64<NF>(p, radius64(p, t[1], t[2], t[3]), t, k);
#pragma unroll
	for(int i = 0; i < ND; ++i) {
		t[i] = fma(dt, k[i], s[i]);
		k2[i] = k2[i] + k[i]; /* k2 + k3 */
	}
	ok &= rhs64<NF>(p, radius64(p, t[1], t[2], t[3]), t, k);
	if(ok) {
#pragma unroll
		for(int i = 0; i < ND; ++i)
			s[i] = fma(h6, fma(2.0, k2[i], k1[i]) + k[i], s[i]);
	} else {
		/* a copy: what a call is given by address lives in memory */
		double any[ND];
#pragma unroll
		for(int i = 0; i < ND; ++i)
			any[i] = s[i];
		rk4_any64<NF>(p, any, dt, h6);
#pragma unroll
		for(int i = 0; i < ND; ++i)
			s[i] = any[i];
	}
}

/* f and l_mu at q with the operation sequence of ks_rhs64() */
__device__ __forceinline__ void
ks_fl64(const RenderParams &p, const double *q, double &r_, double &f_,
        double &lx_, double &ly_, double &lz_)
{
	double aa  = p.aa;
	double zz  = q[3] * q[3];
	double kk  = 0.5 * (fma(q[1], q[1], fma(q[2], q[2], zz)) - aa);
	double dd  = sqrt(fma(kk, kk, aa * zz));
	double rr  = dd + kk;
	double r   = sqrt(rr);
	double ir  = 1.0 / r;
	double ss  = rr + aa;
	double iss = 1.0 / ss;
	double tmp = 2.0 / (rr + (aa * zz) / rr);
	r_  = r;
	f_  = tmp * r;
	lx_ = iss * fma(q[1], r, q[2] * p.a);
	ly_ = iss * fma(q[2], r, -(q[1] * p.a));
	lz_ = q[3] * ir;
}

/* KS.cl:91-114 down() */
__device__ __forceinline__ void
down64(const RenderParams &p, const double *q, const double *u, double *k)
{
	double r, f, lx, ly, lz;
	ks_fl64(p, q, r, f, lx, ly, lz);
	double lu  = fma(lz, u[3], fma(ly, u[2], fma(lx, u[1], u[0])));
	double flu = f * lu;
	k[0] = flu - u[0];
	k[1] = fma(flu, lx, u[1]);
	k[2] = fma(flu, ly, u[2]);
	k[3] = fma(flu, lz, u[3]);
}

/* KS.cl:164-168 getuu() */
__device__ __forceinline__ double
getuu64(const RenderParams &p, const double *s)
{
	double k[4];
	down64(p, s, s + 4, k);
	return fma(k[3], s[7], fma(k[2], s[6], fma(k[1], s[5], k[0] * s[4])));
}

__device__ __forceinline__ void
warp_add_steps(unsigned long long *steps, unsigned long long v)
{
#pragma unroll
	for(int o = 16; o > 0; o >>= 1)
		v += __shfl_xor_sync(0xffffffffu, v, o);
	if((threadIdx.x & 31) == 0 && v)
		atomicAdd(steps, v);
}

/* driver.cl:36-67 icond_drv(), KS.cl:188-232 gr_icond(), rt.cl:179-183 */
__global__ void __launch_bounds__(128)
icond64_kernel(const RenderParams p, double *__restrict__ data,
               double *__restrict__ info)
{
	const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if(g >= p.n_rays)
		return;
	const long long gi = g % p.w_rays;
	const long long gj = p.row0 + g / p.w_rays;
	double alpha = (((double)gi + 0.5) / (double)p.w_rays - 0.5) * p.w_img;
	double beta  = (((double)gj + 0.5) / (double)p.h_rays - 0.5) * p.h_img;

	double R0 = fma(p.r_obs, p.si, -(beta * p.ci));
	double z  = fma(p.r_obs, p.ci, beta * p.si);
	double y  = fma(R0, p.sj, alpha * p.cj);
	double x  = fma(R0, p.cj, -(alpha * p.sj));
	double s[8] = {0.0, x, y, z, 1.0, p.si * p.cj, p.si * p.sj, p.ci};

	double r, f, lx, ly, lz;
	ks_fl64(p, s, r, f, lx, ly, lz);
	const double ux = s[5], uy = s[6], uz = s[7];
	double flx = f * lx, fly = f * ly, flz = f * lz;
	double A  = f - 1.0;
	double B  = 2.0 * fma(flz, uz, fma(fly, uy, flx * ux));
	double Cx = fma(flx * lz, uz, fma(flx * ly, uy, fma(flx, lx, 1.0) * ux));
	double Cy = fma(fly * lz, uz, fma(fma(fly, ly, 1.0), uy, (fly * lx) * ux));
	double Cz = fma(fma(flz, lz, 1.0), uz, fma(flz * ly, uy, (flz * lx) * ux));
	double C  = fma(Cz, uz, fma(Cy, uy, Cx * ux));
	double den = -(B + sqrt(fma(B, B, -((4.0 * A) * C)))) / (2.0 * A);
	s[5] = ux / den;
	s[6] = uy / den;
	s[7] = uz / den;

	const long long n = p.n_rays;
#pragma unroll
	for(int c = 0; c < 8; ++c)
		data[c * n + g] = s[c];
	for(int c = 8; c < p.n_data; ++c)
		data[c * n + g] = 0.0;
	info[g] = getuu64(p, s);
}

/* driver.cl:69-108 evolve_drv(): integer-tick substepping over n_dump dump
 * intervals of n_sub substeps.  One interval has length dt; of several,
 * interval i runs from t_init + i dt to t_init + (i + 1) dt, as the host
 * loop computes it (sim-org/gray.c:251-252).  Each ray walks its intervals by
 * itself: launched one by one, every interval waited for the rays that take
 * 10^4 short steps to the horizon in one of them.
 *
 * What bounds it: the FP64 pipe (82% of its rate without transfer and 70% with
 * four frequencies at 512 x 384 rays), and where few rays run, or few are left,
 * the latency of a step: 1.33 us alone (3.28 where four frequencies emit), of
 * dependent FP64 operations.  Measured with the operators and one launch per
 * interval, and now, B200 at 1965 MHz: 160 x 120 rays through the hole's
 * region, 4 frequencies, 126.3 -> 58.1 ms, 1 frequency 123.2 -> 51.1, none
 * 97.2 -> 40.2; 512 x 384 rays over one interval, 4 frequencies, 46.9 -> 25.0,
 * none 12.4 -> 11.0; 24 x 16 rays 40.2 -> 23.1.
 * One warp more per scheduler (168 registers) gained 8% on the 512 x 384
 * render, but the rays that end last step slower: 251 x 190 rays lost 8%. */
template <int NF>
__global__ void __launch_bounds__(EVOLVE64_BLOCK)
evolve64_kernel(const __grid_constant__ RenderParams p, double *__restrict__ data,
                double *__restrict__ info, const double t_init, const double dt_dump,
                const int n_dump, const long long n_sub, unsigned long long *__restrict__ steps)
{
	constexpr int ND = 8 + 2 * NF;
	const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	const long long nr = p.n_rays;
	unsigned long long cnt = 0;
	if(g < nr) {
		double s[ND];
#pragma unroll
		for(int c = 0; c < ND; ++c)
			s[c] = data[c * nr + g];

		const int n = (int)((INT_MAX / n_sub) * n_sub);
		const double nd = (double)n, in = 1.0 / nd, i6 = 1.0 / 6.0;
		double dt = 0.0, dts = 0.0, idt = 0.0;
		bool plain = false; /* dt near the ends of the exponent range */
		int h = n, dump = 0, cap = 0;
		for(;;) {
			if(h >= n) { /* next interval */
				if(dump >= n_dump)
					break;
				dt = dt_dump;
				if(n_dump > 1)
					dt = (t_init + (double)(dump + 1) * dt_dump) -
					     (t_init + (double)dump * dt_dump);
				++dump;
				h = 0;
				dts = dt / (double)n_sub;
				idt = 1.0 / dt;
				plain = !(fabs(dt) > 1e-60 && fabs(dt) < 1e60);
				/* no steps where the interval's ends round to the same time */
				const double c = dts / dt * nd;
				cap = c >= 1.0 ? (int)c : 0;
			}
			/* phys.cl:48-64 getdt() in ticks */
			const Rad64 R = radius64(p, s[1], s[2], s[3]);
			const double r = in_range(R) ? R.r : sqrt(getrr64(p, s[1], s[2], s[3]));
			const double eps = r - p.rp, lim = (0.01 * eps) * eps;
			const double q = copysign(lim, dts);
			int dh = (int)((plain ? q / dt : div_rn(q, dt, idt)) * nd);
			dh = fabs(dts) > lim ? dh : cap;
			dh = eps < p.eps_stop ? 0 : dh;
			if(!dh) { /* the ray rests for the rest of the interval */
				h = n;
				continue;
			}
			if(dh > n - h)
				dh = n - h;
			const double a = (double)dh * dt;
			const double hs = plain ? a / nd : div_rn(a, nd, in);
			rk4_64<NF>(p, R, s, hs, plain ? hs / 6.0 : div_rn(hs, 6.0, i6));
			h += dh;
			++cnt;
		}
#pragma unroll
		for(int c = 0; c < ND; ++c)
			data[c * nr + g] = s[c];
		info[g] = getuu64(p, s);
	}
	warp_add_steps(steps, cnt);
}

__global__ void
kdown64_kernel(const RenderParams p, const double *__restrict__ data,
               double *__restrict__ k)
{
	const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	const long long n = p.n_rays;
	if(g >= n)
		return;
	double s[8], kk[4];
#pragma unroll
	for(int c = 0; c < 8; ++c)
		s[c] = data[c * n + g];
	down64(p, s, s + 4, kk);
#pragma unroll
	for(int c = 0; c < 4; ++c)
		k[c * n + g] = kk[c];
}

/* KS.cl:63-153 output coordinates, in the oracle's operation order.  The
 * event of down()'s metric is x + i y = (r + i a) e^(i phi) sin(theta);
 * KS.cl:68-69 and 130 use (r - i a), and KS.cl:148-151 put u^phi and u^t
 * where u^r belongs: as_written reproduces both. */
__device__ __forceinline__ void
sph_ks64(const RenderParams &p, const double *q, int as_written, double *out)
{
	double r = sqrt(getrr64(p, q[1], q[2], q[3]));
	double sa = as_written ? p.a : -p.a;
	out[0] = q[0];
	out[1] = r;
	out[2] = acos(q[3] / r);
	out[3] = atan2(fma(q[2], r, q[1] * sa), fma(q[1], r, -(q[2] * sa)));
}

__device__ __forceinline__ void
sph_ks_u64(const RenderParams &p, const double *q, const double *u, int as_written,
           double *out)
{
	const double aa = p.aa;
	double RR = fma(q[1], q[1], q[2] * q[2]);
	double zz = q[3] * q[3];
	double kk = 0.5 * (RR + zz - aa);
	double dd = sqrt(fma(kk, kk, aa * zz));
	double rr = dd + kk;
	double r  = sqrt(rr);
	double den = 2.0 * r * dd;
	double J1[4] = {0.0, rr * q[1] / den, rr * q[2] / den, (rr + aa) * q[3] / den};
	double zr = q[3] / r, sq = sqrt(rr - zz);
	double J2[4] = {0.0, zr * J1[1] / sq, zr * J1[2] / sq, (zr * J1[3] - 1.0) / sq};
	double c = (as_written ? -p.a : p.a) / (rr + aa);
	double J3[4] = {0.0, fma(c, J1[1], -q[2] / RR), fma(c, J1[2], q[1] / RR), c * J1[3]};
	out[0] = u[0];
	out[1] = fma(J1[3], u[3], fma(J1[2], u[2], J1[1] * u[1]));
	out[2] = fma(J2[3], u[3], fma(J2[2], u[2], J2[1] * u[1]));
	out[3] = fma(J3[3], u[3], fma(J3[2], u[2], J3[1] * u[1]));
}

/* system 0: spherical KS; 1: Boyer-Lindquist with t matched at r_match */
__global__ void
coords64_kernel(const RenderParams p, const double *__restrict__ data,
                double *__restrict__ out, int system, double r_match, int as_written)
{
	const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	const long long n = p.n_rays;
	if(g >= n)
		return;
	double s[8], x[4], v[4];
#pragma unroll
	for(int c = 0; c < 8; ++c)
		s[c] = data[c * n + g];
	const double *q = s, *u = s + 4;
	sph_ks64(p, q, as_written, x);
	sph_ks_u64(p, q, u, as_written, v);
	if(system == 1) {
		double h  = sqrt(1.0 - p.aa);
		double rp = 1.0 + h, rm = 1.0 - h, r = x[1];
		x[0] = x[0] + (rm * log((r - rm) / (r_match - rm)) -
		               rp * log((r - rp) / (r_match - rp))) / h;
		x[3] = x[3] + 0.5 * p.a * log((r - rm) / (r - rp)) / h;
		double rr = getrr64(p, q[1], q[2], q[3]);
		double rq = sqrt(rr);
		double D  = rr - 2.0 * rq + p.aa;
		double ut = as_written ? v[3] : v[1];
		double up = as_written ? v[0] : v[1];
		v[0] = v[0] - ut * 2.0 * rq / D;
		v[3] = v[3] - up * p.a / D;
	}
#pragma unroll
	for(int c = 0; c < 4; ++c) {
		out[c * n + g] = x[c];
		out[(4 + c) * n + g] = v[c];
	}
}

__global__ void
getuu64_kernel(const RenderParams p, const double *__restrict__ data,
               double *__restrict__ info)
{
	const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	const long long n = p.n_rays;
	if(g >= n)
		return;
	double s[8];
#pragma unroll
	for(int c = 0; c < 8; ++c)
		s[c] = data[c * n + g];
	info[g] = getuu64(p, s);
}

/* SoA <-> AoS (sim-org/SoA.cl:29 vs AoS.cl:29) through a tile in shared
 * memory so both sides stay coalesced. */
__global__ void
transpose_kernel(const double *__restrict__ src, double *__restrict__ dst,
                 long long n_rays, int n_data, int to_aos)
{
	extern __shared__ double tile[]; /* [n_data][64] */
	const long long base = (long long)blockIdx.x * 64;
	const int tid = threadIdx.x;
	const int total = 64 * n_data;
	for(int e = tid; e < total; e += blockDim.x) {
		if(to_aos) {
			int c = e / 64, r = e % 64;
			long long g = base + r;
			if(g < n_rays)
				tile[c * 64 + r] = src[(long long)c * n_rays + g];
		} else {
			int r = e / n_data, c = e % n_data;
			long long g = base + r;
			if(g < n_rays)
				tile[c * 64 + r] = src[g * n_data + c];
		}
	}
	__syncthreads();
	for(int e = tid; e < total; e += blockDim.x) {
		if(to_aos) {
			int r = e / n_data, c = e % n_data;
			long long g = base + r;
			if(g < n_rays)
				dst[g * n_data + c] = tile[c * 64 + r];
		} else {
			int c = e / 64, r = e % 64;
			long long g = base + r;
			if(g < n_rays)
				dst[(long long)c * n_rays + g] = tile[c * 64 + r];
		}
	}
}

inline unsigned
blocks_for(long long n, int block)
{
	return (unsigned)((n + block - 1) / block);
}

} /* namespace */

cudaError_t
launch_icond64(const RenderParams &p, double *data, double *info, cudaStream_t st)
{
	icond64_kernel<<<blocks_for(p.n_rays, 128), 128, 0, st>>>(p, data, info);
	return cudaGetLastError();
}

cudaError_t
launch_evolve64(const RenderParams &p, double *data, double *info, double t_init,
                double dt_dump, long long n_dump, long long n_sub, unsigned long long *steps,
                cudaStream_t st)
{
	/* one warp per block while the warps do not fill the SMs' schedulers */
	const int block = p.n_rays > 148 * 4 * 32 ? EVOLVE64_BLOCK : 32;
	const unsigned grid = blocks_for(p.n_rays, block);
	switch(p.n_freq) {
#define CASE(NF) case NF: evolve64_kernel<NF><<<grid, block, 0, st>>>(p, data, info, t_init, dt_dump, (int)n_dump, n_sub, steps); break;
	CASE(0) CASE(1) CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(7) CASE(8)
#undef CASE
	default:
		return cudaErrorInvalidValue;
	}
	return cudaGetLastError();
}

cudaError_t
launch_kdown64(const RenderParams &p, const double *data, double *k, cudaStream_t st)
{
	kdown64_kernel<<<blocks_for(p.n_rays, 128), 128, 0, st>>>(p, data, k);
	return cudaGetLastError();
}

cudaError_t
launch_coords64(const RenderParams &p, const double *data, double *out, int system,
                double r_match, int as_written, cudaStream_t st)
{
	coords64_kernel<<<blocks_for(p.n_rays, 128), 128, 0, st>>>(p, data, out, system, r_match,
	                                                           as_written);
	return cudaGetLastError();
}

cudaError_t
launch_getuu64(const RenderParams &p, const double *data, double *info, cudaStream_t st)
{
	getuu64_kernel<<<blocks_for(p.n_rays, 128), 128, 0, st>>>(p, data, info);
	return cudaGetLastError();
}

cudaError_t
launch_transpose(const double *src, double *dst, long long n_rays, int n_data,
                 int to_aos, cudaStream_t st)
{
	size_t smem = sizeof(double) * 64 * (size_t)n_data;
	transpose_kernel<<<blocks_for(n_rays, 64), 256, smem, st>>>(src, dst, n_rays,
	                                                            n_data, to_aos);
	return cudaGetLastError();
}
