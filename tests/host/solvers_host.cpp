/*
Host build of the face solvers (pamhd_b200/csrc/mhd_device.cuh) and of the
step's tile shapes (grid_setup.cuh) for the CPU tests: the same source the GPU kernels inline, compiled by g++ with the
device intrinsics it uses written out as the IEEE operations they are, and
stand-ins for the two hardware estimates: 20 good bits, a subnormal operand
taken for zero (the .ftz of the instructions).  Test infrastructure; not
part of the library.
*/
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

#define __host__
#define __device__
#define __forceinline__ inline

using std::max;

// of the CUDA runtime, in declarations only
typedef struct CUstream_st* cudaStream_t;
struct int4;

static inline double __fma_rn(const double a, const double b, const double c) { return std::fma(a, b, c); }
static inline double __dmul_rn(const double a, const double b) { return a * b; }
static inline double __dadd_rn(const double a, const double b) { return a + b; }
static inline double __dsub_rn(const double a, const double b) { return a - b; }
static inline double __ddiv_rn(const double a, const double b) { return a / b; }
static inline double __drcp_rn(const double a) { return 1.0 / a; }
static inline double __dsqrt_rn(const double a) { return std::sqrt(a); }

static inline int64_t bits(const double x)
{
	int64_t v;
	std::memcpy(&v, &x, 8);
	return v;
}

static inline double from_bits(const int64_t v)
{
	double x;
	std::memcpy(&x, &v, 8);
	return x;
}

static inline int __double2hiint(const double x) { return int(bits(x) >> 32); }
static inline int __double2loint(const double x) { return int(bits(x)); }
static inline double __hiloint2double(const int hi, const int lo)
{
	return from_bits(int64_t(uint64_t(uint32_t(hi)) << 32 | uint32_t(lo)));
}

namespace pamhd_b200 {

static inline double flushed(const double x) { return std::fpclassify(x) == FP_SUBNORMAL ? std::copysign(0.0, x) : x; }
// the mantissa's first 20 bits
static inline double short_of(const double x) { return from_bits(bits(x) & ~((int64_t(1) << 32) - 1)); }
static inline double rcp_estimate(const double x) { return flushed(short_of(1.0 / flushed(x))); }
static inline double rsqrt_estimate(const double x) { return short_of(1.0 / std::sqrt(flushed(x))); }

} // namespace pamhd_b200

#include "../../pamhd_b200/csrc/grid_setup.cuh"

using namespace pamhd_b200;

template <int SOLVER>
static void solve(const int64_t n, const double* neg, const double* pos, const Gas& g, double* flux, double* speed,
                  uint32_t* flags)
{
	const auto side = [&](const double* s) {
		double U[8];
		std::copy(s, s + 8, U);
		return side_of<0>(U, derive<true, false, false>(U[0], U[1], U[2], U[3], U[4], U[5], U[6], U[7], g));
	};
	for (int64_t i = 0; i < n; i++) {
		double F[8];
		speed[i] = solve_face<SOLVER>(side(neg + 8 * i), side(pos + 8 * i), g, F, flags[i]);
		if (flags[i] != 0) speed[i] = 0.0;
		for (int v = 0; v < 8; v++) flux[8 * i + v] = flags[i] != 0 ? 0.0 : F[v];
	}
}

// as pamhd_gpu_face_flux without a background field
extern "C" void host_face_flux(const int32_t solver, const int64_t n, const double* neg, const double* pos,
                               const double gamma, const double mu0, double* flux, double* speed, uint32_t* flags)
{
	Gas g;
	g.gamma = gamma;
	g.mu0 = mu0;
	g.inv_mu0 = 1.0 / mu0;
	g.sqrt_mu0 = std::sqrt(mu0);
	g.inv_sqrt_mu0 = 1.0 / g.sqrt_mu0;
	switch (solver) {
	case PAMHD_RUSANOV: solve<PAMHD_RUSANOV>(n, neg, pos, g, flux, speed, flags); break;
	case PAMHD_HLL_ATHENA: solve<PAMHD_HLL_ATHENA>(n, neg, pos, g, flux, speed, flags); break;
	case PAMHD_HLLD_ATHENA: solve<PAMHD_HLLD_ATHENA>(n, neg, pos, g, flux, speed, flags); break;
	default: solve<PAMHD_ROE_ATHENA>(n, neg, pos, g, flux, speed, flags); break;
	}
}

// the correctly rounded helpers: 1 / x, a / x, sqrt(x)
extern "C" void host_rounded(const int64_t n, const double* a, const double* x, double* inverse, double* quotient,
                             double* root)
{
	for (int64_t i = 0; i < n; i++) {
		inverse[i] = recip_rn(x[i]);
		quotient[i] = quotient_rn(a[i], x[i], inverse[i]);
		root[i] = sqrt_rn(x[i]);
	}
}

// columns along x and y of the tiles of a step with 32 x rows threads and z faces, and its z planes per block
extern "C" void host_tile_shape(const int32_t solver, const int32_t rows, const int32_t n[3], int32_t shape[3])
{
	const Tile_Kind kind{solver, rows, true};
	tile_shape(kind, n[0], n[1], shape[0], shape[1]);
	const long long tiles = (long long)((n[0] + shape[0] - 1) / shape[0]) * ((n[1] + shape[1] - 1) / shape[1]);
	shape[2] = planes_per_block(tiles, n[2], kind.resident());
}
