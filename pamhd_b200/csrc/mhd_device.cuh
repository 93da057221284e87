/*
FP64 device physics of the finite-volume MHD step (sm_100a).

The four Riemann solvers of the reference (mhd/rusanov.hpp:67,
mhd/hll_athena.hpp:65, mhd/hlld_athena.hpp:62, mhd/roe_athena.hpp:575) and
the MHD primitives they use (mhd/common.hpp), written for the GPU:

  - Each cell's derived quantities (1/rho, velocity, thermal pressure,
    magnetic pressure and the fast magnetosonic speed along each axis) are
    computed once per cell and shared by the six faces of the cell.  The
    reference recomputes them in every solver call.
  - Divisions by the same denominator are done once as a reciprocal,
    products added are fused multiply-adds, and HLLD and Roe are rearranged
    (see flux_hlld, flux_roe).  Results therefore differ from the reference
    by round-off (the parity tests hold them to 1e-12).
  - Branches (supersonic upwinding, HLLD degeneracy thresholds, region
    selection, Roe's positivity check) are the reference's, with its
    epsilon thresholds.
  - Where the reference throws std::domain_error, the device code raises a
    PAMHD_FLAG_* bit for that face instead (include/pamhd_gpu.h).

Conventions: a face is solved in its own frame, x = face normal; Side holds
one cell's state rotated into that frame (get_rotated_vector,
mhd/common.hpp:612).  Flux order: rho, mom x/y/z, E, B x/y/z.
*/
#ifndef PAMHD_B200_MHD_DEVICE_CUH
#define PAMHD_B200_MHD_DEVICE_CUH

#include <cstdint>

#include "../../include/pamhd_gpu.h"

namespace pamhd_b200 {

constexpr double DBL_EPS = 2.220446049250313080847e-16;  // numeric_limits<double>::epsilon()

/*
Checks on the high word (sign, exponent, top of the mantissa): one or two
integer instructions, where comparisons of doubles would take the FP64
pipe that bounds these kernels.
*/
__device__ __forceinline__ bool is_normal(const double x)
{
	return ((unsigned int)__double2hiint(x) & 0x7fffffffu) - 0x00100000u < 0x7fe00000u;
}

// x > 0 and normal
__device__ __forceinline__ bool is_positive_normal(const double x)
{
	return (unsigned int)__double2hiint(x) - 0x00100000u < 0x7fe00000u;
}

__device__ __forceinline__ bool is_finite(const double x)
{
	return ((unsigned int)__double2hiint(x) & 0x7fffffffu) < 0x7ff00000u;
}

// the sign bit: x < 0 for any number but -0
__device__ __forceinline__ bool is_negative(const double x)
{
	return __double2hiint(x) < 0;
}

// zero, negative or not a number (an infinite x counts too: its timestep is 0 as well)
__device__ __forceinline__ bool no_speed(const double x)
{
	return (unsigned int)__double2hiint(x) - 1u >= 0x7ff00000u - 1u;
}

// the larger of two numbers (fmax() also sorts out NaN, which takes twice the instructions)
__device__ __forceinline__ double larger(const double a, const double b)
{
	return a > b ? a : b;
}

// physical constants of one run
struct Gas {
	double gamma;     // adiabatic index
	double mu0;       // vacuum permeability
	double inv_mu0;   // 1 / mu0
	double sqrt_mu0;
	double inv_sqrt_mu0;
};

/*
Derived quantities of one cell (mhd/common.hpp:79 get_pressure,
:327 get_sound_speed, :381 get_alfven_speed, :418
get_fast_magnetosonic_speed), computed once per cell.  cf[d] is the fast
magnetosonic speed along axis d.  bad holds the PAMHD_FLAG_* bits the
reference would raise for any face touching this cell, in its order of
checks: density, then pressure, then wave speed.
*/
struct Derived {
	double rinv, vx, vy, vz, p, pt, cf[3];  // pt: thermal plus magnetic pressure
	uint32_t bad;
};

// in Derived::bad, alone: round-off decides whether the reference takes the cell's fast speed
// (reference_wave), and derive was told to leave that to the caller
constexpr uint32_t OPEN_WAVE = 1u << 7;

#ifdef __CUDACC__
// the hardware's estimates of 1/x and 1/sqrt(x), which take a subnormal x for zero (a host build of
// these solvers brings its own)
__device__ __forceinline__ double rcp_estimate(const double x)
{
	double r;
	asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
	return r;
}

__device__ __forceinline__ double rsqrt_estimate(const double x)
{
	double r;
	asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
	return r;
}
#endif

/*
Reciprocal of a non-zero normal double: one third-order step of the
Householder family for f(r) = 1/r - x, r <- r (1 + e + e^2) with
e = 1 - x r, from the hardware estimate of PTX rcp.approx.ftz.f64.  The
step cubes the estimate's relative error (at most 2^-19.9, measured over
2^26 mantissas), so the result is within one unit in the last place of
1/x, with three dependent operations where two Newton steps take four.
Used where the operand is a normal, non-zero number by construction.
*/
__device__ __forceinline__ double recip(const double x)
{
	const double r = rcp_estimate(x);
	const double e = __fma_rn(-x, r, 1.0);
	return __fma_rn(r, __fma_rn(e, e, e), r);
}

/*
One third-order step for f(r) = 1/r^2 - x from an estimate r:
r <- r (1 + e/2 + 3 e^2 / 8) with e = 1 - x r^2.
*/
__device__ __forceinline__ double rsqrt_step(const double x, const double r)
{
	const double e = __fma_rn(__dmul_rn(-x, r), r, 1.0);
	return __fma_rn(__dmul_rn(r, e), __fma_rn(0.375, e, 0.5), r);
}

/*
Reciprocal square root of a positive normal double, from the hardware
estimate of PTX rsqrt.approx.ftz.f64.
*/
__device__ __forceinline__ double rsqrt_nr(const double x)
{
	return rsqrt_step(x, rsqrt_estimate(x));
}

// x raised to the smallest normal number (an integer maximum of the high word)
__device__ __forceinline__ double raised(const double x)
{
	return __hiloint2double(max(__double2hiint(x), 0x00100000), __double2loint(x));
}

/*
Square root of a non-negative finite double as x rsqrt(x); the estimate is
taken of x raised, so that 0 gives 0.
*/
__device__ __forceinline__ double sqrt_nr(const double x)
{
	return __dmul_rn(x, rsqrt_step(x, rsqrt_estimate(raised(x))));
}

/*
Correctly rounded reciprocals, quotients and roots of normal numbers by
Markstein's final step (IBM J. Res. Dev. 34, 1990): a result y within an ulp
is corrected by its remainder, which a fused multiply-add gives exactly,
times the (rounded) reciprocal.  Straight code where the IEEE functions are
calls; only a divisor whose mantissa is all ones can miss the last bit.
*/
__device__ __forceinline__ double recip_rn(const double x)
{
	const double r = recip(x);
	return __fma_rn(__fma_rn(-x, r, 1.0), r, r);
}

// a / x, with r = recip_rn(x)
__device__ __forceinline__ double quotient_rn(const double a, const double x, const double r)
{
	const double q = __dmul_rn(a, r);
	return __fma_rn(__fma_rn(-q, x, a), r, q);
}

// 0 gives 0
__device__ __forceinline__ double sqrt_rn(const double x)
{
	const double r = rsqrt_nr(raised(x)), s = __dmul_rn(x, r);
	return __fma_rn(__fma_rn(-s, s, x), __dmul_rn(0.5, r), s);
}

/*
Whether get_fast_magnetosonic_speed (mhd/common.hpp:418-491) takes a cell, in
the frame of the face: the argument of its inner root,
a^4 + v_A^4 + 2 a^2 v_A^2 (1 - 2 cos^2), cancels to round-off, of either
sign, where the sound and Alfven speeds are equal and the field is along the
normal.  Its operations one for one, each rounded on its own.
*/
__device__ __forceinline__ bool reference_wave(
	const double rho, const double m0, const double m1, const double m2, const double E,
	const double b0, const double b1, const double b2, const Gas& g
) {
	const auto mul = [](const double x, const double y) { return __dmul_rn(x, y); };
	const auto add = [](const double x, const double y) { return __dadd_rn(x, y); };
	const auto sub = [](const double x, const double y) { return __dsub_rn(x, y); };
	const double i = recip_rn(rho);
	const double bsq = add(add(mul(b0, b0), mul(b1, b1)), mul(b2, b2));
	const double kinetic = mul(mul(0.5, i), add(add(mul(m0, m0), mul(m1, m1)), mul(m2, m2)));
	const double p = mul(sub(sub(E, kinetic), mul(mul(0.5, g.inv_mu0), bsq)), g.gamma - 1.0);
	const double sound = sqrt_rn(quotient_rn(mul(g.gamma, p), rho, i)), b = sqrt_rn(bsq);
	const double mass = sqrt_rn(mul(g.mu0, rho));
	const double alfven = quotient_rn(b, mass, recip_rn(mass)), cosine = quotient_rn(b0, b, recip_rn(b));
	const double s2 = mul(sound, sound), a2 = mul(alfven, alfven);
	const double part = sub(1.0, mul(2.0, mul(cosine, cosine)));
	return is_positive_normal(add(add(mul(s2, s2), mul(a2, a2)), mul(mul(mul(2.0, s2), a2), part)));
}

/*
Every operation below is an explicitly rounded intrinsic, so that every
inlined copy of this function computes the same bits for the same cell
(the halo of one tile is the interior of the next).

The fast speed: c_f^2 = (a^2 + v_A^2 + root) / 2 with
root^2 = (a^2 + v_A^2)^2 - 4 a^2 v_A,n^2, written as
(a^2 - v_A^2)^2 + 4 a^2 v_A,t^2 (v_A,t from the field across the axis):
no division by B^2 and no cancellation.

RECORD: for the cell-centred steps' records.  Without it both roots are
correctly rounded, three operations more each (with it the speed's error is
8 % larger, rms), and a cell whose wave speed round-off decides is judged
here, for the axes asked for; with it that is left open (OPEN_WAVE) and the
speeds are given: the judgement, though it is hardly ever made, took 1.8 %
of a 256^3 step here.
*/
template <bool NEED_X, bool NEED_Y, bool NEED_Z, bool RECORD = false>
__device__ __forceinline__ Derived derive(
	const double rho, const double mx, const double my, const double mz,
	const double E, const double bx, const double by, const double bz, const Gas& g
) {
	Derived d;
	d.rinv = recip(rho);
	d.vx = __dmul_rn(mx, d.rinv);
	d.vy = __dmul_rn(my, d.rinv);
	d.vz = __dmul_rn(mz, d.rinv);
	const double bb[3] = {__dmul_rn(bx, bx), __dmul_rn(by, by), __dmul_rn(bz, bz)};
	const double b2 = __dadd_rn(__dadd_rn(bb[0], bb[1]), bb[2]);
	const double m2 = __fma_rn(mz, mz, __fma_rn(my, my, __dmul_rn(mx, mx)));
	const double kinetic = __dmul_rn(__dmul_rn(0.5, d.rinv), m2);
	const double magnetic = __dmul_rn(__dmul_rn(0.5, g.inv_mu0), b2);
	d.p = __dmul_rn(__dsub_rn(__dsub_rn(E, kinetic), magnetic), g.gamma - 1.0);
	d.pt = __dadd_rn(d.p, magnetic);
	d.bad = 0;
	if (not is_positive_normal(rho)) {
		d.bad = PAMHD_FLAG_DENSITY;
	} else if (not is_positive_normal(d.p)) {
		d.bad = PAMHD_FLAG_PRESSURE;
	}
	const double cs2 = __dmul_rn(__dmul_rn(g.gamma, d.p), d.rinv);
	const auto root = [](const double x) { return RECORD ? sqrt_nr(x) : sqrt_rn(x); };
	const bool need[3] = {NEED_X, NEED_Y, NEED_Z};
	if (b2 > 0.0) {
		const double im = __dmul_rn(g.inv_mu0, d.rinv);
		const double va2 = __dmul_rn(b2, im);
		const double sum2 = __dadd_rn(cs2, va2), diff2 = __dsub_rn(cs2, va2);
		const double base = __dmul_rn(diff2, diff2);
		const double cross = __dmul_rn(__dmul_rn(4.0, cs2), im);
		const bool sum_ok = is_positive_normal(sum2) and is_finite(b2);
		bool wave_ok = sum_ok;
		// the high word of some 2^-40 (a^2 + v_A^2)^2 (twice a logarithm, in integers): where the root's
		// argument is smaller, round-off decides whether the reference takes the cell
		const int low = int(2u * ((unsigned int)__double2hiint(sum2) - (0x1ff80000u + (20u << 20))));
		bool open[3] = {false, false, false};
		#pragma unroll
		for (int a = 0; a < 3; a++) {
			if (not need[a]) {
				d.cf[a] = 0.0;
				continue;
			}
			const double to_sqrt = __fma_rn(cross, __dadd_rn(bb[(a + 1) % 3], bb[(a + 2) % 3]), base);
			open[a] = __double2hiint(to_sqrt) < low;
			wave_ok = wave_ok and is_positive_normal(to_sqrt);
			d.cf[a] = root(__dmul_rn(0.5, __dadd_rn(sum2, root(to_sqrt))));
		}
		const bool undecided = (open[0] or open[1] or open[2]) and sum_ok;
		if (d.bad == 0) d.bad = undecided ? OPEN_WAVE : (wave_ok ? 0u : (uint32_t)PAMHD_FLAG_WAVE_SPEED);
		if (not RECORD and d.bad == OPEN_WAVE) {
			d.bad = 0;
			#pragma unroll 1
			for (int a = 0; a < 3; a++) {
				const auto turn = [a](const double x, const double y, const double z) { return a == 0 ? x : (a == 1 ? y : z); };
				if ((a == 0 ? open[0] : (a == 1 ? open[1] : open[2]))
					and not reference_wave(rho, turn(mx, my, mz), turn(my, mz, mx), turn(mz, mx, my), E,
					                       turn(bx, by, bz), turn(by, bz, bx), turn(bz, bx, by), g)) {
					d.bad = PAMHD_FLAG_WAVE_SPEED;
				}
			}
		}
	} else {
		d.cf[0] = d.cf[1] = d.cf[2] = root(cs2);
		if (d.bad == 0 and not is_finite(b2)) d.bad = PAMHD_FLAG_WAVE_SPEED;
	}
	// a refused cell: no face of it counts, its speeds stay numbers
	if (d.bad != 0 and d.bad != OPEN_WAVE) d.cf[0] = d.cf[1] = d.cf[2] = 0.0;
	return d;
}

// in the frame of faces normal to axis a (known at run time): cf[0] is the fast speed along it
__device__ __forceinline__ Derived derive_along(const int a, const double U[8], const Gas& g)
{
	const auto turn = [a](const double x, const double y, const double z) { return a == 0 ? x : (a == 1 ? y : z); };
	return derive<true, false, false>(
		U[0], turn(U[1], U[2], U[3]), turn(U[2], U[3], U[1]), turn(U[3], U[1], U[2]), U[4],
		turn(U[5], U[6], U[7]), turn(U[6], U[7], U[5]), turn(U[7], U[5], U[6]), g);
}

// one cell seen from a face, rotated into the face frame
struct Side {
	double rho, m0, m1, m2, E, b0, b1, b2;
	double rinv, v0, v1, v2, cf;
	double pt;   // thermal plus magnetic pressure
	double p;    // thermal pressure, for the fluxes with a background field only
	uint32_t bad;
};

/*
Rotation into the frame of a face normal to axis `axis` (0, 1, 2):
get_rotated_vector(v, axis + 1), mhd/common.hpp:612-648:
  x: (v0, v1, v2)   y: (v1, v2, v0)   z: (v2, v0, v1)
*/
template <int AXIS>
__device__ __forceinline__ void rotate(const double a, const double b, const double c,
                                       double& r0, double& r1, double& r2)
{
	if (AXIS == 0) { r0 = a; r1 = b; r2 = c; }
	if (AXIS == 1) { r0 = b; r1 = c; r2 = a; }
	if (AXIS == 2) { r0 = c; r1 = a; r2 = b; }
}

// and back: get_rotated_vector(r, -(axis + 1))
template <int AXIS>
__device__ __forceinline__ void unrotate(const double r0, const double r1, const double r2,
                                         double& a, double& b, double& c)
{
	if (AXIS == 0) { a = r0; b = r1; c = r2; }
	if (AXIS == 1) { a = r2; b = r0; c = r1; }
	if (AXIS == 2) { a = r1; b = r2; c = r0; }
}

// a cell's state (8 values, xyz frame) and derived quantities seen from a face normal to axis A
template <int A>
__device__ __forceinline__ Side side_of(const double U[8], const Derived& d)
{
	Side s;
	s.rho = U[0];
	rotate<A>(U[1], U[2], U[3], s.m0, s.m1, s.m2);
	s.E = U[4];
	rotate<A>(U[5], U[6], U[7], s.b0, s.b1, s.b2);
	s.rinv = d.rinv;
	s.pt = d.pt;
	s.p = d.p;
	s.cf = d.cf[A];
	s.v0 = s.m0 * s.rinv;
	s.v1 = s.m1 * s.rinv;
	s.v2 = s.m2 * s.rinv;
	s.bad = d.bad;
	return s;
}

/*
Arithmetic of the face solvers (Rusanov, HLL, HLLD): every operation an
explicitly rounded intrinsic, a fused multiply-add where the formula has a
product added, so that every kernel computes the same bits for the same
face, whatever other code it is inlined beside and whichever flags its
file is compiled with.
*/
struct Ar {
	static __device__ __forceinline__ double mul(const double a, const double b) { return __dmul_rn(a, b); }
	static __device__ __forceinline__ double add(const double a, const double b) { return __dadd_rn(a, b); }
	static __device__ __forceinline__ double sub(const double a, const double b) { return __dsub_rn(a, b); }
	static __device__ __forceinline__ double fma(const double a, const double b, const double c)
	{
		return __fma_rn(a, b, c);
	}
};

/*
Ideal-MHD flux along the face normal, mhd/common.hpp:146-244, with the
background field zero (every configuration of the fused step).
*/
__device__ __forceinline__ void physical_flux(const Side& s, const Gas& g, double F[8])
{
	using A = Ar;
	const double b0m = A::mul(s.b0, g.inv_mu0);
	F[0] = s.m0;
	F[1] = A::fma(s.m0, s.v0, A::fma(-b0m, s.b0, s.pt));
	F[2] = A::fma(s.m1, s.v0, -A::mul(b0m, s.b1));
	F[3] = A::fma(s.m2, s.v0, -A::mul(b0m, s.b2));
	const double vb = A::fma(s.v2, s.b2, A::fma(s.v1, s.b1, A::mul(s.v0, s.b0)));
	F[4] = A::fma(s.v0, A::add(s.E, s.pt), -A::mul(b0m, vb));
	F[5] = 0.0;
	F[6] = A::fma(s.v0, s.b1, -A::mul(s.b0, s.v1));
	F[7] = A::fma(s.v0, s.b2, -A::mul(s.b0, s.v2));
}

/*
The same with a background face field bg (in the face frame), for the
solver-level entry point: mhd/common.hpp:174-241 splits the field into the
cell's own part B and the background part.
*/
__device__ __forceinline__ void physical_flux_bg(
	const Side& s, const double bg0, const double bg1, const double bg2, const Gas& g, double F[8]
) {
	const double t0 = s.b0 + bg0, t1 = s.b1 + bg1, t2 = s.b2 + bg2;
	const double p_bg = 0.5 * g.inv_mu0 * (bg0 * bg0 + bg1 * bg1 + bg2 * bg2);
	const double p_b1 = 0.5 * g.inv_mu0 * (s.b0 * s.b0 + s.b1 * s.b1 + s.b2 * s.b2);
	const double p_tot = 0.5 * g.inv_mu0 * (t0 * t0 + t1 * t1 + t2 * t2);
	F[0] = s.m0;
	F[1] = s.m0 * s.v0 - g.inv_mu0 * (t0 * t0 - bg0 * bg0) + (s.p + p_tot - p_bg);
	F[2] = s.m1 * s.v0 - g.inv_mu0 * (t0 * t1 - bg0 * bg1);
	F[3] = s.m2 * s.v0 - g.inv_mu0 * (t0 * t2 - bg0 * bg2);
	const double vb = s.v0 * s.b0 + s.v1 * s.b1 + s.v2 * s.b2;
	F[4] = s.v0 * (s.E + s.p + p_b1) - s.b0 * vb * g.inv_mu0
		+ g.inv_mu0 * (s.b1 * (s.v0 * bg1 - s.v1 * bg0) + s.b2 * (s.v0 * bg2 - s.v2 * bg0));
	F[5] = 0.0;
	F[6] = s.v0 * t1 - t0 * s.v1;
	F[7] = s.v0 * t2 - t0 * s.v2;
}

/*
Rusanov (local Lax-Friedrichs), mhd/rusanov.hpp:67-179:
F = (F_L + F_R)/2 - s/2 (U_R - U_L), s = max(|u_L|, |u_R|) + max(c_f,L, c_f,R).
The field's normal component is diffused like the rest (the reference
does not zero it).
*/
template <bool BG>
__device__ __forceinline__ double flux_rusanov(const Side& L, const Side& R, const Gas& g, double F[8],
                                               uint32_t& flag, const double* bg = nullptr)
{
	using A = Ar;
	const double fast = larger(L.cf, R.cf);
	const double s = A::add(larger(fabs(L.v0), fabs(R.v0)), fast);
	double FL[8], FR[8];
	if (BG) {
		physical_flux_bg(L, bg[0], bg[1], bg[2], g, FL);
		physical_flux_bg(R, bg[0], bg[1], bg[2], g, FR);
	} else {
		physical_flux(L, g, FL);
		physical_flux(R, g, FR);
	}
	const double h = A::mul(0.5, s);
	const double UL[8] = {L.rho, L.m0, L.m1, L.m2, L.E, L.b0, L.b1, L.b2};
	const double UR[8] = {R.rho, R.m0, R.m1, R.m2, R.E, R.b0, R.b1, R.b2};
	#pragma unroll
	for (int v = 0; v < 8; v++) {
		F[v] = A::fma(-A::sub(UR[v], UL[v]), h, A::mul(0.5, A::add(FL[v], FR[v])));
	}
	if (flag == 0 and (not is_finite(F[0]) or not is_finite(s))) flag = PAMHD_FLAG_FLUX;
	return s;
}

/*
HLL with Davis wave-speed estimates, mhd/hll_athena.hpp:65-275:
S_L = min(u_L, u_R) - max c_f, S_R = max(u_L, u_R) + max c_f,
bm = min(S_L, 0), bp = max(S_R, 0); a degenerate fan (bp - bm not a
positive normal number) gives zero flux and zero speed.
*/
template <bool BG>
__device__ __forceinline__ double flux_hll(const Side& L, const Side& R, const Gas& g, double F[8],
                                           uint32_t& /*flag*/, const double* bg = nullptr)
{
	using A = Ar;
	const double fast = larger(L.cf, R.cf);
	const bool order = L.v0 <= R.v0;
	const double s_neg = A::sub(order ? L.v0 : R.v0, fast);
	const double s_pos = A::add(order ? R.v0 : L.v0, fast);
	const double bm = is_negative(s_neg) ? s_neg : 0.0, bp = is_negative(s_pos) ? 0.0 : s_pos;
	const double width = A::sub(bp, bm);
	if (not is_positive_normal(width)) {
		#pragma unroll
		for (int v = 0; v < 8; v++) F[v] = 0.0;
		return 0.0;
	}
	double FL[8], FR[8];
	if (BG) {
		physical_flux_bg(L, bg[0], bg[1], bg[2], g, FL);
		physical_flux_bg(R, bg[0], bg[1], bg[2], g, FR);
	} else {
		physical_flux(L, g, FL);
		physical_flux(R, g, FR);
	}
	const double UL[8] = {L.rho, L.m0, L.m1, L.m2, L.E, L.b0, L.b1, L.b2};
	const double UR[8] = {R.rho, R.m0, R.m1, R.m2, R.E, R.b0, R.b1, R.b2};
	// as a mean and a difference, in which both sides round alike: equal states at rest give exactly
	// their pressure, mirrored faces mirrored fluxes (weights on the sides, two operations less per
	// row, leave a mass flux of up to 1e-9 of the row between equal states at rest)
	const double w = A::mul(A::mul(0.5, A::add(bp, bm)), recip(width));
	#pragma unroll
	for (int v = 0; v < 8; v++) {
		const double a = A::fma(-bm, UL[v], FL[v]), b = A::fma(-bp, UR[v], FR[v]);
		F[v] = v == 5 ? 0.0 : A::fma(A::sub(a, b), w, A::mul(0.5, A::add(a, b)));
	}
	return larger(bp, -bm);
}

// transverse velocity and field of one side's star state (Miyoshi & Kusano eqns 44-47): v - b t1
// and b t2, with t1 = 0 and t2 = 1 in the degenerate case (keep)
struct Star_T {
	double w1, w2, b1, b2;
	bool keep;
};

__device__ __forceinline__ Star_T star_transverse(const Side& X, const double rho_sd, const double sd,
                                                  const double sm, const double s_mid, const double bxm,
                                                  const double bx2_mu, const double thr)
{
	using A = Ar;
	const double tmp = A::fma(rho_sd, sm, -bx2_mu);
	const double it = recip(tmp);
	Star_T t;
	t.keep = fabs(tmp) < thr;
	const double t1 = t.keep ? 0.0 : A::mul(A::mul(bxm, A::sub(s_mid, X.v0)), it);
	const double t2 = t.keep ? 1.0 : A::mul(A::fma(rho_sd, sd, -bx2_mu), it);
	t.w1 = A::fma(-X.b1, t1, X.v1);
	t.w2 = A::fma(-X.b2, t1, X.v2);
	t.b1 = A::mul(X.b1, t2);
	t.b2 = A::mul(X.b2, t2);
	return t;
}

/*
The two sides a face is solved between, when both are held in registers.
*/
struct Held_Sides {
	const Side& L;
	const Side& R;
	__device__ __forceinline__ Side operator()(const bool left) const { return left ? L : R; }
};

/*
HLLD of Miyoshi & Kusano (J. Comput. Phys. 208, 2005), as
mhd/hlld_athena.hpp:62-559; the background field is ignored there (:77)
and here.  Past the supersonic cases every region's ingredients are
computed in one straight run (both sides' transverse star states, the
step across the Alfven wave) and the reference's region choice (:475-552)
selects among them, so that the compiler can overlap the two sides'
dependency chains; values of regions not taken are discarded by selects,
never multiplied in.

The reference sums the flux up from the outer state, F + S_out (U* - U) +
S_in (U** - U*).  The jump conditions that define the star states make
that sum, in exact arithmetic, the flux of the intermediate state itself
with the star total pressure,
  rho* S_M,  rho* S_M^2 + p_t*,  rho* S_M v_t - B_x B_t / mu0,
  (E + p_t*) S_M - B_x (v . B) / mu0,  S_M B_t - B_x v_t,
plus what the reference's use of the side's own normal field B_n in F (and
in v . B of the outer state), where the star states have the mean B_x,
leaves over:
  -B_n^2 / mu0 in the normal momentum (the formula has no B_x^2 there),
  -(B_n - B_x) B_t / mu0, -(B_n - B_x) (v . B) / mu0, -(B_n - B_x) v_t
of the outer state in the others; in the degenerate case, where the star
state keeps the outer B_t and v_t, also (v_n - S_M) B_t in the field.
That is some 60 operations less per face, and the double-star state needs
only the velocity step across its Alfven wave: v** = v* + dv,
B** = B* +- sqrt(mu0 rho*) sign(B_x) dv, dv = 0 where there is no such
wave.  The step is bound by the latency of these FP64 chains: this form, the
third-order reciprocals and the fast speed of derive() took a 256^3 step
from 2.14 to 1.73 ms, a 150 x 99 x 67 step from 180 to 148 us.

The side the flux is taken from comes from pick(left): a caller that holds
the sides' records in shared memory reads that side again instead of
selecting all of its fields between the two sides held in registers.
*/
template <class PICK>
__device__ __forceinline__ double flux_hlld(const Side& L, const Side& R, const Gas& g, double F[8],
                                            const PICK& pick)
{
	using A = Ar;
	const double fast = larger(L.cf, R.cf);
	const bool order = L.v0 <= R.v0;
	const double s_neg = A::sub(order ? L.v0 : R.v0, fast);  // eqn 67
	const double s_pos = A::add(order ? R.v0 : L.v0, fast);
	const double speed = larger(fabs(s_neg), fabs(s_pos));

	if (not is_negative(s_neg) or is_negative(s_pos)) {
		physical_flux(pick(not is_negative(s_neg)), g, F);
		return speed;
	}

	const double bx = A::mul(0.5, A::add(L.b0, R.b0));
	const double bxm = A::mul(bx, g.inv_mu0), bx2_mu = A::mul(bx, bxm);
	const double sdL = A::sub(s_neg, L.v0), sdR = A::sub(s_pos, R.v0);       // < 0 and > 0 here
	const double rsdL = A::mul(L.rho, sdL), rsdR = A::mul(R.rho, sdR);
	// eqn 38; the denominator is sdR rho_R - sdL rho_L > 0
	const double s_mid = A::mul(A::add(A::sub(A::mul(sdR, R.m0), A::mul(sdL, L.m0)), A::sub(L.pt, R.pt)),
	                            recip(A::sub(rsdR, rsdL)));
	const double smL = A::sub(s_neg, s_mid), smR = A::sub(s_pos, s_mid);     // < 0 and > 0 for physical states
	const double ismL = recip(smL), ismR = recip(smR);
	// eqn 43, and the square roots of the star densities with their reciprocals
	const double rsL = A::mul(rsdL, ismL), rsR = A::mul(rsdR, ismR);
	const double irL = rsqrt_nr(rsL), irR = rsqrt_nr(rsR);
	const double sqL = A::mul(rsL, irL), sqR = A::mul(rsR, irR);
	// eqn 51
	const double abx = A::mul(fabs(bx), g.inv_sqrt_mu0);
	const double ssL = A::fma(-abx, irL, s_mid), ssR = A::fma(abx, irR, s_mid);
	const double thr = A::mul(DBL_EPS, A::fma(rsdL, A::sub(s_mid, L.v0), L.pt));
	// transverse star velocity and field of both sides, eqns 44-47
	const Star_T tl = star_transverse(L, rsdL, sdL, smL, s_mid, bxm, bx2_mu, thr);
	const Star_T tr = star_transverse(R, rsdR, sdR, smR, s_mid, bxm, bx2_mu, thr);

	// region order of hlld_athena.hpp:475-552: S*_L >= 0, S_M >= 0, S*_R > 0, else
	const bool left = not is_negative(s_mid);
	const bool star_l = not is_negative(ssL);
	const bool star_r = not star_l and not left and is_negative(ssR);
	const bool useL = star_l or (not star_r and left);   // the side the flux is taken from
	// the double-star region (the star state itself when Bx ~ 0)
	const bool two = not star_l and not star_r and not (A::mul(A::mul(0.5, bx), bx) < thr);
	const Side S = pick(useL);
	const Star_T ts = useL ? tl : tr;
	const double ism = useL ? ismL : ismR, rs = useL ? rsL : rsR;
	// the star total pressure, equal on both sides but for round-off, from the side the flux is taken
	// from, so that a mirrored face has the mirrored flux
	const double ptst = A::fma(useL ? rsdL : rsdR, A::sub(s_mid, S.v0), S.pt);

	// the step across that side's Alfven wave, eqns 59-62 less the star state
	const double inv_sum = recip(A::add(sqL, sqR));
	const double sgn = (bx > 0.0) ? 1.0 : -1.0;
	const double cv = A::mul(sgn, g.inv_sqrt_mu0);
	const double near = useL ? sqL : -sqR, far = useL ? sqR : -sqL;
	const double d1 = A::mul(inv_sum, A::fma(cv, A::sub(tr.b1, tl.b1), A::mul(far, A::sub(tr.w1, tl.w1))));
	const double d2 = A::mul(inv_sum, A::fma(cv, A::sub(tr.b2, tl.b2), A::mul(far, A::sub(tr.w2, tl.w2))));
	const double dv1 = two ? d1 : 0.0, dv2 = two ? d2 : 0.0;
	const double db = A::mul(A::mul(sgn, g.sqrt_mu0), near);
	const double w1 = A::add(ts.w1, dv1), w2 = A::add(ts.w2, dv2);
	const double b1 = A::fma(db, dv1, ts.b1), b2 = A::fma(db, dv2, ts.b2);

	// energy of the star state, eqn 48, and of the double-star state, eqn 63
	const double vb = A::fma(S.v2, S.b2, A::fma(S.v1, S.b1, A::mul(S.v0, S.b0)));
	const double smb = A::mul(s_mid, bx);
	const double vb_star = A::fma(ts.w2, ts.b2, A::fma(ts.w1, ts.b1, smb));
	const double vb2 = A::fma(w2, b2, A::fma(w1, b1, smb));
	double e = A::fma(A::sub(useL ? s_neg : s_pos, S.v0), S.E, -A::mul(S.pt, S.v0));
	e = A::fma(ptst, s_mid, e);
	e = A::fma(bxm, A::sub(vb, vb_star), e);
	e = A::fma(A::mul(cv, near), A::sub(vb2, vb_star), A::mul(e, ism));

	// the flux
	const double b0m = A::mul(S.b0, g.inv_mu0);
	const double over = A::sub(S.b0, bx), overm = A::sub(b0m, bxm);
	F[0] = A::mul(rs, s_mid);
	F[1] = A::fma(F[0], s_mid, A::fma(-b0m, S.b0, ptst));
	F[2] = A::fma(F[0], w1, A::fma(-bxm, b1, -A::mul(overm, S.b1)));
	F[3] = A::fma(F[0], w2, A::fma(-bxm, b2, -A::mul(overm, S.b2)));
	F[4] = A::fma(A::add(e, ptst), s_mid, A::fma(-bxm, vb2, -A::mul(overm, vb)));
	F[5] = 0.0;
	const double kv = ts.keep ? A::sub(S.v0, s_mid) : 0.0;
	F[6] = A::fma(kv, S.b1, A::fma(s_mid, b1, A::fma(-bx, w1, -A::mul(over, S.v1))));
	F[7] = A::fma(kv, S.b2, A::fma(s_mid, b2, A::fma(-bx, w2, -A::mul(over, S.v2))));
	return speed;
}

// a double whose operators round explicitly (as Ar), for formulas that read better with operators
struct Rd {
	double v;
	__device__ __forceinline__ Rd(const double x = 0.0) : v(x) {}
	__device__ __forceinline__ operator double() const { return v; }
};
__device__ __forceinline__ Rd operator*(const Rd a, const Rd b) { return __dmul_rn(a.v, b.v); }
__device__ __forceinline__ Rd operator*(const double a, const Rd b) { return __dmul_rn(a, b.v); }
__device__ __forceinline__ Rd operator*(const Rd a, const double b) { return __dmul_rn(a.v, b); }
__device__ __forceinline__ Rd operator+(const Rd a, const Rd b) { return __dadd_rn(a.v, b.v); }
__device__ __forceinline__ Rd operator-(const Rd a, const Rd b) { return __dsub_rn(a.v, b.v); }
__device__ __forceinline__ Rd operator-(const Rd a) { return -a.v; }
__device__ __forceinline__ Rd mad(const Rd a, const Rd b, const Rd c) { return __fma_rn(a.v, b.v, c.v); }

/*
alpha_f and alpha_s of Roe's eigensystem (B17-B29 of Stone et al.) for an
almost aligned average field (a small transverse component).  One of the
reference's numerators a^2 - c_s^2 and c_f^2 - a^2 is then all or partly
round-off, some 1e-16, whose root weighs in at up to 1e-8 where the
transverse velocity or field jumps: its operations are repeated here one for
one, each rounded on its own (mhd/roe_athena.hpp:56-559), so that such faces
agree with it too.
*/
__device__ __forceinline__ void near_aligned_alphas(const Side& L, const Side& R, const Gas& g, double& alpha_f,
                                                    double& alpha_s)
{
	const auto mul = [](const double a, const double b) { return __dmul_rn(a, b); };
	const auto add = [](const double a, const double b) { return __dadd_rn(a, b); };
	const auto sub = [](const double a, const double b) { return __dsub_rn(a, b); };
	const auto sq3 = [&](const double a, const double b, const double c) {
		return add(add(mul(a, a), mul(b, b)), mul(c, c));
	};
	const double gm1 = g.gamma - 1.0, gm2 = g.gamma - 2.0;
	const auto field = [&](const double b) { return quotient_rn(b, g.sqrt_mu0, g.inv_sqrt_mu0); };
	const double bx = mul(0.5, field(add(L.b0, R.b0))), bx2 = mul(bx, bx);
	const double byl = field(L.b1), bzl = field(L.b2), byr = field(R.b1), bzr = field(R.b2);
	const double il = recip_rn(L.rho), ir = recip_rn(R.rho);
	const double sl = sqrt_rn(L.rho), sr = sqrt_rn(R.rho), sum = add(sl, sr);
	const double isd = recip_rn(sum), rho = mul(sl, sr), di = recip_rn(rho);
	const auto enthalpy = [&](const Side& s, const double i, const double by, const double bz, const double root) {
		const double p = mul(sub(sub(s.E, mul(mul(0.5, i), sq3(s.m0, s.m1, s.m2))),
		                         mul(0.5, sq3(s.b0, s.b1, s.b2))), gm1);
		const double H = add(add(s.E, p), mul(0.5, add(add(bx2, mul(by, by)), mul(bz, bz))));
		return quotient_rn(H, root, recip_rn(root));
	};
	const double h = mul(add(enthalpy(L, il, byl, bzl, sl), enthalpy(R, ir, byr, bzr, sr)), isd);
	const auto mean = [&](const double l, const double r) {
		return mul(add(mul(sl, mul(l, il)), mul(sr, mul(r, ir))), isd);
	};
	const double vsq = sq3(mean(L.m0, R.m0), mean(L.m1, R.m1), mean(L.m2, R.m2));
	const double by = mul(add(mul(sr, byl), mul(sl, byr)), isd), bz = mul(add(mul(sr, bzl), mul(sl, bzr)), isd);
	const double dy = sub(byl, byr), dz = sub(bzl, bzr), sum2 = mul(sum, sum);
	const double x = quotient_rn(mul(0.5, add(mul(dy, dy), mul(dz, dz))), sum2, recip_rn(sum2));
	const double y = quotient_rn(mul(0.5, add(L.rho, R.rho)), rho, di);
	const double btsq = add(mul(by, by), mul(bz, bz));
	const double ct2 = mul(mul(sub(gm1, mul(gm2, y)), btsq), di), va2 = mul(bx2, di);
	const double hp = sub(h, add(va2, mul(btsq, di)));
	const double a2 = fmax(sub(mul(gm1, sub(hp, mul(0.5, vsq))), mul(gm2, x)), DBL_EPS);
	const double vat2 = add(va2, ct2), tdif = sub(vat2, a2);
	const double root = sqrt_rn(add(mul(tdif, tdif), mul(mul(4.0, a2), ct2)));
	const double cf2 = mul(0.5, add(add(vat2, a2), root));
	const double cs2 = quotient_rn(mul(a2, va2), cf2, recip_rn(cf2));
	const double q = sub(cf2, cs2), f = sub(a2, cs2), s = sub(cf2, a2);
	alpha_f = 1.0;
	alpha_s = 0.0;
	if (q == 0.0) return;
	if (f <= 0.0) {
		alpha_f = 0.0;
		alpha_s = 1.0;
	} else if (s > 0.0) {
		const double iq = recip_rn(q);
		alpha_f = sqrt_rn(quotient_rn(f, q, iq));
		alpha_s = sqrt_rn(quotient_rn(s, q, iq));
	}
}

/*
Roe solver for adiabatic MHD, after Athena's esys_roe_adb_mhd and fluxes
(mhd/roe_athena.hpp:56-559; eigensystem eqns B17-B29 of Stone et al.,
ApJS 178, 2008), in units where the field is B / sqrt(mu0).  The signal
speed is the one of mhd/roe_athena.hpp:763-815.

The seven waves come as v - c, v + c pairs (fast 0 and 6, slow 2 and 4,
Alfven 1 and 5) whose eigenvectors differ only in the sign of one part:
each pair's strengths are a sum and a difference of two shared
projections, and its contribution to the flux takes the sum and the
difference of the pair's weights.  No 7 x 7 matrix is formed, and no
product with one of its zeros computed; every root and quotient comes from
the reciprocal steps above.  Bound by FP64 work (1798 flops per 2-D
cell-update, 3026 as dense matrices with IEEE roots and quotients): a 512^2
step went from 107 to 65 us (67 with the almost aligned faces' alphas).

alpha_f^2 = (a^2 - c_s^2) / (c_f^2 - c_s^2) and alpha_s^2 = (c_f^2 - a^2) /
(c_f^2 - c_s^2), whose numerators cancel, are taken from the quadratic's
roots: with q = c_f^2 - c_s^2 its discriminant's root and
t = v_A^2 - a^2 (v_A with the starred transverse field), the larger of the
two numerators is (q + |t|) / 2 and the smaller a^2 c_t^2 over that, so
that nothing cancels; where the reference's own cancellation shows, in an
almost aligned field, they are the reference's (near_aligned_alphas).
*/
__device__ __forceinline__ double flux_roe(const Side& L, const Side& R, const Gas& g, double F[8],
                                           uint32_t& flag)
{
	const Rd gm1 = g.gamma - 1.0, gm2 = g.gamma - 2.0, half = 0.5;
	const Rd ism = g.inv_sqrt_mu0;
	const Rd bxi = half * (Rd(L.b0) + Rd(R.b0)) * ism;
	const Rd byl = Rd(L.b1) * ism, bzl = Rd(L.b2) * ism, byr = Rd(R.b1) * ism, bzr = Rd(R.b2) * ism;
	// pressure with mu0 = 1, as the reference's get_primitive call (roe_athena.hpp:706-721)
	const auto thermal = [&](const Side& s) -> Rd {
		const Rd m2 = mad(s.m2, s.m2, mad(s.m1, s.m1, Rd(s.m0) * Rd(s.m0)));
		const Rd b2 = mad(s.b2, s.b2, mad(s.b1, s.b1, Rd(s.b0) * Rd(s.b0)));
		return gm1 * mad(-half, b2, mad(-(half * Rd(s.rinv)), m2, s.E));
	};
	const Rd pl = thermal(L), pr = thermal(R);
	const Rd bx2 = bxi * bxi;
	const Rd pbl = half * mad(bzl, bzl, mad(byl, byl, bx2)), pbr = half * mad(bzr, bzr, mad(byr, byr, bx2));
	const Rd ptl = pl + pbl, ptr = pr + pbr;

	// Roe averages
	const Rd il = rsqrt_nr(L.rho), ir = rsqrt_nr(R.rho);
	const Rd sdl = Rd(L.rho) * il, sdr = Rd(R.rho) * ir;
	const Rd isd = recip(sdl + sdr);
	const Rd wl = sdl * isd, wr = sdr * isd;
	const Rd droe = sdl * sdr, di = il * ir;
	const Rd isqrtd = rsqrt_nr(droe), sqrtd = droe * isqrtd;
	const Rd v1 = mad(wl, L.v0, wr * Rd(R.v0)), v2 = mad(wl, L.v1, wr * Rd(R.v1)), v3 = mad(wl, L.v2, wr * Rd(R.v2));
	// products rounded: opposite fields at equal densities average to exactly 0
	const Rd b2 = wr * byl + wl * byr, b3 = wr * bzl + wl * bzr;
	const Rd dby = byl - byr, dbz = bzl - bzr;
	const Rd x = half * mad(dby, dby, dbz * dbz) * (isd * isd);
	const Rd y = half * (Rd(L.rho) + Rd(R.rho)) * di;
	const Rd h = mad(Rd(L.E) + ptl, il, (Rd(R.E) + ptr) * ir) * isd;

	// wave speeds
	const Rd vsq = mad(v3, v3, mad(v2, v2, v1 * v1));
	const Rd btsq = mad(b3, b3, b2 * b2);
	const Rd ystar = mad(-gm2, y, gm1);
	const Rd vaxsq = bx2 * di;
	const Rd hp = h - mad(btsq, di, vaxsq);
	const Rd asq = fmax(double(mad(gm1, mad(-half, vsq, hp), -(gm2 * x))), DBL_EPS);
	const Rd ct2 = ystar * btsq * di;
	const Rd va2 = vaxsq + ct2;
	const Rd tdif = va2 - asq, a2ct2 = asq * ct2;
	const Rd root = sqrt_nr(mad(tdif, tdif, Rd(4.0) * a2ct2));
	const Rd cfsq = half * (va2 + asq + root);
	const Rd icf = rsqrt_nr(cfsq), cf = cfsq * icf;
	const Rd ia = rsqrt_nr(asq), a = asq * ia;
	const Rd vax = fabs(bxi.v) * isqrtd;
	const Rd cs = a * vax * icf;
	const double ev[7] = {v1 - cf, v1 - vax, v1 - cs, v1, v1 + cs, v1 + vax, v1 + cf};

	// flux of each side, and the conserved difference
	const double Fl[7] = {
		L.m0, mad(L.m0, L.v0, ptl - bx2), mad(L.m0, L.v1, -(bxi * byl)), mad(L.m0, L.v2, -(bxi * bzl)),
		mad(Rd(L.E) + ptl, L.v0, -(bxi * mad(bzl, L.v2, mad(byl, L.v1, bxi * Rd(L.v0))))),
		mad(byl, L.v0, -(bxi * Rd(L.v1))), mad(bzl, L.v0, -(bxi * Rd(L.v2)))};
	const double Fr[7] = {
		R.m0, mad(R.m0, R.v0, ptr - bx2), mad(R.m0, R.v1, -(bxi * byr)), mad(R.m0, R.v2, -(bxi * bzr)),
		mad(Rd(R.E) + ptr, R.v0, -(bxi * mad(bzr, R.v2, mad(byr, R.v1, bxi * Rd(R.v0))))),
		mad(byr, R.v0, -(bxi * Rd(R.v1))), mad(bzr, R.v0, -(bxi * Rd(R.v2)))};

	double Fo[7];
	if (ev[0] >= 0.0) {
		#pragma unroll
		for (int r = 0; r < 7; r++) Fo[r] = Fl[r];
	} else if (ev[6] <= 0.0) {
		#pragma unroll
		for (int r = 0; r < 7; r++) Fo[r] = Fr[r];
	} else {
		// the fast and slow normalisations and the transverse direction
		const Rd big = half * (root + Rd(fabs(tdif.v)));
		const Rd iroot = recip(root);
		const Rd large = big * iroot, small = a2ct2 * recip(big) * iroot;
		const bool slow_field = tdif < 0.0;
		const Rd one = 1.0, none = 0.0;
		Rd af = sqrt_nr(slow_field ? large : small), as = sqrt_nr(slow_field ? small : large);
		const Rd ibt = rsqrt_nr(btsq);
		Rd bt = btsq * ibt, bet2 = b2 * ibt, bet3 = b3 * ibt;
		// below 1e-5 the reference's round-off in the smaller alpha weighs more than some 2e-13 of the flux
		// (1e5 random faces; 6e-13 at 1e-6).  NaN, where the root is 0, too
		if (not (small > 1e-5)) near_aligned_alphas(L, R, g, af.v, as.v);
		if (not is_positive_normal(btsq)) {
			// no field, or one whose square is subnormal, which the estimate of the root takes for 0:
			// its direction from the field times 2^600
			const Rd s2 = b2 * 0x1p600, s3 = b3 * 0x1p600;
			const double s = __dsqrt_rn(mad(s3, s3, s2 * s2));
			bt = s * 0x1p-600;
			bet2 = btsq > 0.0 ? __ddiv_rn(s2, s) : 1.0;
			bet3 = btsq > 0.0 ? __ddiv_rn(s3, s) : 0.0;
		}
		const Rd iys = rsqrt_nr(ystar), sys = ystar * iys;
		const Rd sg = bxi > 0.0 ? one : -one;
		const Rd qf = cf * af * sg, qs = cs * as * sg;
		const Rd afp = a * af * isqrtd, asp = a * as * isqrtd;   // alpha' of B17-B29
		const Rd vb = mad(v2, bet2, v3 * bet3), vx = mad(v2, bet3, -(v3 * bet2));

		// wave strengths: projections of the difference on the left eigenvectors
		const Rd d0 = Rd(R.rho) - Rd(L.rho), d1 = Rd(R.m0) - Rd(L.m0), d2 = Rd(R.m1) - Rd(L.m1);
		const Rd d3 = Rd(R.m2) - Rd(L.m2), d4 = Rd(R.E) - Rd(L.E), d5 = byr - byl, d6 = bzr - bzl;
		const Rd norm = half * ia * ia;
		const Rd e2 = mad(-v2, d0, d2), e3 = mad(-v3, d0, d3);   // rho times the transverse velocity step
		const Rd X = mad(v1, d0, -d1);
		const Rd Y = sys * mad(bet2, e2, bet3 * e3);
		const Rd Z = sys * mad(bet2, d5, bet3 * d6) * droe - bt * sys * d0;
		const Rd P = mad(vsq - hp, d0, mad(-v1, d1, mad(-v2, d2, mad(-v3, d3, mad(-b2, d5, mad(-b3, d6, d4))))));
		const Rd Pn = gm1 * P;
		const Rd sf = norm * mad(af, mad(cf * cf, d0, Pn), asp * Z), df = norm * mad(cf * af, X, qs * Y);
		const Rd ss = norm * mad(as, mad(cs * cs, d0, Pn), -(afp * Z)), ds = norm * mad(cs * as, X, -(qf * Y));
		const Rd al = half * mad(bet2, e3, -(bet3 * e2)), be = half * sqrtd * sg * mad(bet2, d6, -(bet3 * d5));
		const Rd k = gm2 * x * recip(gm1);
		const Rd half_vsq = half * vsq;
		const Rd a3 = mad(-(norm + norm) * gm1, mad(hp - half_vsq - k, d0, P), d0);
		const double am[7] = {sf + df, al + be, ss + ds, a3, ss - ds, be - al, sf - df};

		// right eigenvectors: the parts a pair shares (s) and the parts that change sign (d)
		const Rd qsb = qs * iys, qfb = qf * iys;
		const Rd fv2 = af * v2, fv3 = af * v3, sv2 = as * v2, sv3 = as * v3;
		const Rd fe = mad(af, hp, asp * bt * iys), se = mad(as, hp, -(afp * bt * iys));
		const Rd fde = mad(qsb, vb, -(af * v1 * cf)), sde = -mad(qfb, vb, as * v1 * cs);
		const Rd fb2 = asp * bet2 * iys, fb3 = asp * bet3 * iys, sb2 = -(afp * bet2 * iys), sb3 = -(afp * bet3 * iys);
		const Rd sgi = sg * isqrtd;
		const Rd ab2 = -(bet3 * sgi), ab3 = bet2 * sgi;
		const Rd ee = half_vsq + k;

		// positivity of the intermediate states: the reference throws at the first failing one between
		// two distinct waves.  p < 0 as (E - b^2 / 2) rho < m^2 / 2, without a division
		{
			Rd u[7] = {L.rho, L.m0, L.m1, L.m2, L.E, byl, bzl};
			uint32_t roe_fail = 0;
			const auto after = [&](const int n, const Rd r0, const Rd r1, const Rd r2, const Rd r3, const Rd r4,
			                       const Rd r5, const Rd r6) {
				const Rd w = am[n];
				u[0] = mad(w, r0, u[0]); u[1] = mad(w, r1, u[1]); u[2] = mad(w, r2, u[2]); u[3] = mad(w, r3, u[3]);
				u[4] = mad(w, r4, u[4]); u[5] = mad(w, r5, u[5]); u[6] = mad(w, r6, u[6]);
				const Rd m2 = mad(u[3], u[3], mad(u[2], u[2], u[1] * u[1]));
				const Rd e = mad(-half, mad(u[6], u[6], mad(u[5], u[5], bx2)), u[4]);
				const uint32_t bad = u[0] <= 0.0 ? PAMHD_FLAG_ROE_DENSITY
					: (mad(e, u[0], -(half * m2)) < 0.0 ? PAMHD_FLAG_ROE_PRESSURE : 0u);
				if (ev[n + 1] > ev[n] and roe_fail == 0) roe_fail = bad;
			};
			after(0, af, af * Rd(ev[0]), mad(qsb, bet2, fv2), mad(qsb, bet3, fv3), fe + fde, fb2, fb3);
			after(1, none, none, -bet3, bet2, -vx, ab2, ab3);
			after(2, as, as * Rd(ev[2]), mad(-qfb, bet2, sv2), mad(-qfb, bet3, sv3), se + sde, sb2, sb3);
			after(3, one, v1, v2, v3, ee, none, none);
			after(4, as, as * Rd(ev[4]), mad(qfb, bet2, sv2), mad(qfb, bet3, sv3), se - sde, sb2, sb3);
			after(5, none, none, bet3, -bet2, vx, ab2, ab3);
			if (flag == 0) flag = roe_fail;
		}

		// flux: the mean less half the sum of the strengths times |speed| times the right eigenvectors
		Rd c[7];
		#pragma unroll
		for (int m = 0; m < 7; m++) c[m] = Rd(am[m]) * Rd(fabs(ev[m]));
		const Rd f = c[0] + c[6], fd = c[0] - c[6], s = c[2] + c[4], sd = c[2] - c[4], t = c[1] + c[5], td = c[1] - c[5];
		const Rd T = mad(af, f, mad(as, s, c[3]));
		const Rd Q = mad(qsb, fd, -(qfb * sd));
		const Rd B = mad(asp, f, -(afp * s)) * iys;
		const double D[7] = {
			T,
			mad(v1, T, -mad(af * cf, fd, as * cs * sd)),
			mad(v2, T, mad(bet2, Q, -(bet3 * td))),
			mad(v3, T, mad(bet3, Q, bet2 * td)),
			mad(fe, f, mad(se, s, mad(ee, c[3], mad(fde, fd, mad(sde, sd, -(vx * td)))))),
			mad(bet2, B, ab2 * t),
			mad(bet3, B, ab3 * t)};
		#pragma unroll
		for (int r = 0; r < 7; r++) Fo[r] = half * (Rd(Fl[r]) + Rd(Fr[r]) - Rd(D[r]));
	}
	F[0] = Fo[0]; F[1] = Fo[1]; F[2] = Fo[2]; F[3] = Fo[3]; F[4] = Fo[4];
	F[5] = 0.0;
	F[6] = Rd(Fo[5]) * Rd(g.sqrt_mu0);
	F[7] = Rd(Fo[6]) * Rd(g.sqrt_mu0);

	// signal speed (roe_athena.hpp:763-815)
	const double fast = fmax(L.cf, R.cf);
	const bool order = L.v0 <= R.v0;
	const double s_neg = Rd(order ? L.v0 : R.v0) - Rd(fast);
	const double s_pos = Rd(order ? R.v0 : L.v0) + Rd(fast);
	if (s_neg >= 0.0) return fabs(s_pos);
	if (s_pos <= 0.0) return fabs(s_neg);
	return fmax(fabs(s_neg), fabs(s_pos));
}

// pick: see flux_hlld (the other solvers use the sides held)
template <int SOLVER, class PICK>
__device__ __forceinline__ double solve_face(const Side& L, const Side& R, const Gas& g, double F[8],
                                             uint32_t& flag, const PICK& pick)
{
	flag = L.bad | R.bad;
	if (flag & PAMHD_FLAG_DENSITY) flag = PAMHD_FLAG_DENSITY;
	else if (flag & PAMHD_FLAG_PRESSURE) flag = PAMHD_FLAG_PRESSURE;
	if (SOLVER == PAMHD_RUSANOV) return flux_rusanov<false>(L, R, g, F, flag);
	if (SOLVER == PAMHD_HLL_ATHENA) return flux_hll<false>(L, R, g, F, flag);
	if (SOLVER == PAMHD_HLLD_ATHENA) return flux_hlld(L, R, g, F, pick);
	return flux_roe(L, R, g, F, flag);
}

template <int SOLVER>
__device__ __forceinline__ double solve_face(const Side& L, const Side& R, const Gas& g, double F[8],
                                             uint32_t& flag)
{
	return solve_face<SOLVER>(L, R, g, F, flag, Held_Sides{L, R});
}

} // namespace pamhd_b200

#endif
