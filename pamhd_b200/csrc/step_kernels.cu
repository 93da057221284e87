/*
Kernels of the fused finite-volume MHD step (sm_100a, FP64 CUDA cores).

step_kernel<SOLVER, TY, ZACT> - one launch = one whole step (the reference's
  get_all_fluxes + update_mhd_state + minimize_timestep, mhd/solve.hpp:
  1702-1811, :1518-1614, :1933-2014, in their cell-centred form):
  * a block of 32 TY threads owns a tile of about as many columns and
    marches along z through a chunk of planes ("2.5-D blocking");
  * each plane of the tile plus a one-cell halo in x and y is read once
    from HBM (coalesced along x), its derived quantities (1/rho, pressure,
    fast speeds along x, y, z) computed once per cell into shared memory;
  * every x and y face of the tile is solved once from shared memory and
    its dt-scaled flux kept in shared memory; the z face between the
    previous and the current plane is solved by the thread owning the
    column and kept in registers, so every z face is solved once;
  * the new state of a cell is written as soon as its last (+z) face is
    known, plus its periodic image or COPY ghost (so no separate ghost
    fill pass is needed);
  * the face signal speeds are max-reduced per axis (warp shuffles, then
    one atomicMax per block on the bits of the non-negative double) into a
    three-slot ring; the next step's dt is computed from that ring by
    every block at kernel start, so consecutive steps never wait on the
    host and can be replayed from a CUDA graph.
Only the redundant halo faces of each tile (with 32 x 8 columns, 1/32 + 1/8
of the x/y faces) and one z plane per chunk are solved twice.
*/
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "step.cuh"

namespace pamhd_b200 {

constexpr int TX = 32;
constexpr int TY_3D = 4;     // the smaller tile: 32 x 4
constexpr int TY_WIDE = 8;   // the larger: 32 x 8

// record of a cell in shared memory: rho, mom xyz, E, B xyz, 1/rho, thermal plus magnetic
// pressure, cf x, cf y (the fast speed along z is needed by the column's owner only, which keeps
// it in a register)
constexpr int NV = 12;
enum { R_RINV = 8, R_PT = 9, R_CF = 10 };

/*
Rows of a face flux kept in shared memory, in the face frame: rho, the
normal and the two tangential momenta, E, the two tangential field
components, and the normal field component only for Rusanov, the one
solver whose flux of it is not zero (mhd/rusanov.hpp diffuses it).
*/
template <int SOLVER> struct Flux_Rows { static constexpr int N = SOLVER == PAMHD_RUSANOV ? 8 : 7; };

template <int TY, bool ZACT, int NF = 8> struct Tile {
	static constexpr int JO = (TY > 1) ? 1 : 0;            // halo rows exist when y is active
	static constexpr int CELLS = Tile_Kind::records_of(TY);  // records of a plane, halo included
	static constexpr int FLAT = Tile_Kind::flat_width_of(TY);
	static constexpr int REC = NV * CELLS;                 // doubles per plane slot
	static constexpr int SLOTS = ZACT ? 2 : 1;             // planes whose records are held
	// the record slots; the x and the y face fluxes of a plane, indexed as the record of the cell on
	// the face's positive side, so that one index per thread serves records and fluxes; one
	// validity byte per cell and slot
	static constexpr size_t BYTES = size_t(SLOTS * REC + NF * CELLS * (1 + JO)) * 8 + size_t(SLOTS * CELLS);
};

template <int SOLVER, int TY, bool ZACT> constexpr size_t tile_bytes()
{
	return Tile<TY, ZACT, Flux_Rows<SOLVER>::N>::BYTES;
}

int batch_tile_rows()
{
	return TY_3D;
}

// ------------------------------------------------------------------ helpers

__device__ __forceinline__ double warp_max(double v)
{
	#pragma unroll
	for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
	return v;
}

/*
dt of the step from the previous step's face speeds: the minimum over
faces of CFL * d_len / s (solve.hpp:1983-2003), which equals
CFL * d_len / max(s) per axis because rounding is monotonic; 0 when any
face speed was <= 0; replaced by the cap when cap <= that minimum
(substepping.hpp:331-338).
*/
__device__ __forceinline__ double step_dt(const Step_Params& P)
{
	if (P.forced_dt >= 0.0) return P.forced_dt;
	// read at L2 (ld.global.cg): a persistent launch reads what other blocks wrote a step before
	const Speed_Max& r = P.red[P.phase];
	bool zero = __ldcg(&r.zero) != 0;
	double smallest = 1.7976931348623157e308;
	#pragma unroll
	for (int d = 0; d < 3; d++) {
		if (not P.active[d]) continue;
		const double s = __longlong_as_double((long long)__ldcg(&r.smax[d]));
		if (not (s > 0.0)) {
			zero = true;
		} else {
			smallest = fmin(smallest, (P.cfl * P.len[d]) / s);
		}
	}
	if (zero) smallest = 0.0;
	const double t = __ldcg(&P.clock[P.phase].t);
	const double cap = P.control->max_dt >= 0.0 ? P.control->max_dt : P.control->t_end - t;
	return (cap <= smallest) ? cap : smallest;
}

/*
Whether the grid stopped in an earlier step: a face failed there (the
reference aborts at that step, mhd/solve.hpp:156-181).  Such a step leaves
the state as it is and the clock where it is.  The failing step itself is
completed (every block of it sees the same answer: the failure is dated by
the clock's step count).
*/
__device__ __forceinline__ bool stopped_before(const Step_Params& P)
{
	const unsigned int at = __ldcg(&P.status->fail_step);
	return at != 0u and (long long)(at - 1u) < __ldcg(&P.clock[P.phase].steps);
}

/*
A block barrier in two halves (an mbarrier in shared memory, one arrival
per warp): what a warp does between its arrival and its wait overlaps the
other warps' way to theirs.  phase counts the block's uses, from 0.
*/
struct Split_Barrier {
	uint32_t addr;   // shared-memory address
	uint32_t phase;

	// by one thread, before a __syncthreads()
	__device__ __forceinline__ void init(const uint32_t warps) const
	{
		asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(addr), "r"(warps) : "memory");
	}

	__device__ __forceinline__ void arrive() const
	{
		__syncwarp();
		if ((threadIdx.x & 31) == 0) {
			asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(addr) : "memory");
		}
	}

	// false when the other warps did not arrive within the poll limit.  The step has then failed: it is
	// dated, as a failing face's (record_failure), so that the grid or box holds its later steps.  The
	// warp goes on to the block's next barrier, which it reaches like the others: this use is then
	// complete, and the phase in step again
	__device__ __forceinline__ bool wait(const Step_Params& P)
	{
		const uint32_t parity = phase & 1u;
		phase++;
		#pragma unroll 1
		for (int poll = 0; poll < P.barrier_polls; poll++) {
			uint32_t done;
			asm volatile("{\n\t.reg .pred p;\n\t"
			             "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
			             "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(addr), "r"(parity) : "memory");
			if (done) return true;
		}
		atomicOr(&P.status->flags, (unsigned int)PAMHD_FLAG_TIMEOUT);
		P.status->fail_step = (unsigned int)(__ldcg(&P.clock[P.phase].steps) + 1);
		return false;
	}
};

__device__ __forceinline__ Split_Barrier split_barrier(unsigned long long* const word)
{
	return Split_Barrier{uint32_t(__cvta_generic_to_shared(word)), 0u};
}

/*
The start of a step, by one thread of the block: the step's dt to *s_dt and
whether the grid stopped in an earlier step to *s_stop (dt 0, the clock
held); the first block's thread advances the clock ring.
*/
__device__ __forceinline__ void find_dt(const Step_Params& P, double* s_dt, const bool first_block, int* s_stop)
{
	const bool stop = stopped_before(P);
	const double dt = stop ? 0.0 : step_dt(P);
	*s_dt = dt;
	*s_stop = stop ? 1 : 0;
	if (first_block) {
		Clock c;
		c.t = __ldcg(&P.clock[P.phase].t);
		c.steps = __ldcg(&P.clock[P.phase].steps);
		Clock& next = P.clock[(P.phase + 1) % 3];
		next.t = c.t + dt;
		next.dt = dt;
		next.steps = stop ? c.steps : c.steps + 1;
		if (P.dt_hist != nullptr and not stop) P.dt_hist[c.steps % P.hist_len] = dt;
		Speed_Max& z = P.red[(P.phase + 2) % 3];
		z.smax[0] = z.smax[1] = z.smax[2] = 0ull;
		z.zero = 0u;
		if (stop) {
			// no face is solved: the failing step's maxima stay the latest
			const Speed_Max& r = P.red[P.phase];
			Speed_Max& o = P.red[(P.phase + 1) % 3];
			o.smax[0] = __ldcg(&r.smax[0]);
			o.smax[1] = __ldcg(&r.smax[1]);
			o.smax[2] = __ldcg(&r.smax[2]);
			o.zero = __ldcg(&r.zero);
		}
	}
}

// the same for the whole block, which knows both when it returns
__device__ __forceinline__ double begin_step(const Step_Params& P, double* s_dt, const bool first_block,
                                             int* s_stop)
{
	if (threadIdx.x == 0) find_dt(P, s_dt, first_block, s_stop);
	__syncthreads();
	return *s_dt;
}

// the first failing face, numbered as the oracle's extended grid (x fastest)
__device__ void record_failure(const Step_Params& P, const uint32_t flag, const int i, const int j,
                               const int k, const int dir)
{
	int c[3] = {i, j, k};
	#pragma unroll
	for (int d = 0; d < 3; d++) {
		if (P.periodic[d] and c[d] < 0) c[d] += P.L.n[d];
	}
	const unsigned long long nx = P.L.n[0] + 2 * P.ext[0], ny = P.L.n[1] + 2 * P.ext[1];
	const unsigned long long lin = (unsigned long long)(c[0] + P.ext[0])
		+ nx * ((unsigned long long)(c[1] + P.ext[1]) + ny * (unsigned long long)(c[2] + P.ext[2]));
	atomicOr(&P.status->flags, flag);
	atomicMin(&P.status->first, ((lin * 4ull + (unsigned long long)dir) << 8) | flag);
	// every failure of a step writes the same date
	P.status->fail_step = (unsigned int)(__ldcg(&P.clock[P.phase].steps) + 1);
}

// folds a block's speeds into the step's reduction; returns whether any of its threads has `open` set
__device__ __forceinline__ bool flush_speeds(const Step_Params& P, double smax[3], bool zero, bool open = false)
{
	__shared__ double part[3][32];
	__shared__ int part_zero[32];
	const int tid = threadIdx.y * blockDim.x + threadIdx.x;
	const int warp = tid >> 5, lane = tid & 31, warps = (blockDim.x * blockDim.y + 31) >> 5;
	#pragma unroll
	for (int d = 0; d < 3; d++) smax[d] = warp_max(smax[d]);
	const int z = (__any_sync(0xffffffffu, zero) ? 1 : 0) | (__any_sync(0xffffffffu, open) ? 2 : 0);
	if (lane == 0) {
		part[0][warp] = smax[0];
		part[1][warp] = smax[1];
		part[2][warp] = smax[2];
		part_zero[warp] = z;
	}
	__syncthreads();
	int any = 0;
	for (int w = 0; w < warps; w++) any |= part_zero[w];
	if (tid == 0) {
		Speed_Max& r = P.red[(P.phase + 1) % 3];
		#pragma unroll
		for (int d = 0; d < 3; d++) {
			double m = 0.0;
			for (int w = 0; w < warps; w++) m = fmax(m, part[d][w]);
			if (P.active[d] and m > 0.0) {
				atomicMax(&r.smax[d], (unsigned long long)__double_as_longlong(m));
			}
		}
		if ((any & 1) != 0) atomicOr(&r.zero, 1u);
	}
	return (any & 2) != 0;
}

__device__ __forceinline__ void store_cell(double* out, const Layout& L, const int i, const int j,
                                           const int k, const double U[8])
{
	const long long off = L.offset(i, j, k);
	#pragma unroll
	for (int v = 0; v < 8; v++) out[v * L.var + off] = U[v];
}

// the state of a time-stamped inflow at time t
__device__ __forceinline__ const double* inflow_at(const Inflow_Table& T, const double t)
{
	int i = 0;
	while (i < T.count and t >= T.times[i]) i++;
	return T.states + 8 * i;
}

/*
New state of an interior cell plus its periodic image / COPY ghost (the
neighbour's density, velocity, pressure and field, mhd/boundaries.hpp:
818-1030, which is its state: taking the energy apart and together again
cost every warp at an open side two IEEE divisions per cell), and the
ghost of a time-stamped VALUE side at the time the new state holds: the
step's start time plus dt, as begin_step advances the clock.
*/
__device__ void write_cell(const Step_Params& P, const int i, const int j, const int k, const double U[8],
                           const double dt)
{
	store_cell(P.out, P.L, i, j, k, U);
	const int c[3] = {i, j, k};
	#pragma unroll
	for (int d = 0; d < 3; d++) {
		if (not P.active[d]) continue;
		const int n = P.L.n[d];
		int t[3] = {i, j, k};
		if (c[d] == 0) {
			if (P.periodic[d]) {
				t[d] = n;
				store_cell(P.out, P.L, t[0], t[1], t[2], U);
			} else if (P.bc_lo[d] == PAMHD_BC_COPY) {
				t[d] = -1;
				store_cell(P.out, P.L, t[0], t[1], t[2], U);
			} else if (P.bc_lo[d] == PAMHD_BC_VALUE and P.inflow != nullptr and P.inflow[2 * d].states != nullptr) {
				t[d] = -1;
				store_cell(P.out, P.L, t[0], t[1], t[2], inflow_at(P.inflow[2 * d], __ldcg(&P.clock[P.phase].t) + dt));
			}
		}
		if (c[d] == n - 1) {
			t[0] = i; t[1] = j; t[2] = k;
			if (P.periodic[d]) {
				t[d] = -1;
				store_cell(P.out, P.L, t[0], t[1], t[2], U);
			} else if (P.bc_hi[d] == PAMHD_BC_COPY) {
				t[d] = n;
				store_cell(P.out, P.L, t[0], t[1], t[2], U);
			} else if (P.bc_hi[d] == PAMHD_BC_VALUE and P.inflow != nullptr and P.inflow[2 * d + 1].states != nullptr) {
				t[d] = n;
				store_cell(P.out, P.L, t[0], t[1], t[2], inflow_at(P.inflow[2 * d + 1], __ldcg(&P.clock[P.phase].t) + dt));
			}
		}
	}
}

/*
Read a cell from HBM, derive its per-cell quantities into a record slot.
CO: loads at L2 (ld.global.cg) instead of through the read-only cache, for a
persistent launch whose later steps read what other blocks wrote (the
non-coherent L1 could hold a line of the same buffer from two steps before).
A cell whose wave speed round-off decides is taken for now, and open set
(settle_tile).
*/
template <bool CX, bool CY, bool CZ, bool CO, class Meanwhile>
__device__ __forceinline__ double load_record(const Step_Params& P, double* rec, uint8_t* bad, const int cells,
                                              const int ri, const long long off, bool& open,
                                              const Meanwhile& meanwhile)
{
	double U[8];
	#pragma unroll
	for (int v = 0; v < 8; v++) U[v] = CO ? __ldcg(P.in + v * P.L.var + off) : __ldg(P.in + v * P.L.var + off);
	meanwhile();   // while the loads are on their way
	const Derived d = derive<CX, CY, CZ, true>(U[0], U[1], U[2], U[3], U[4], U[5], U[6], U[7], P.gas);
	#pragma unroll
	for (int v = 0; v < 8; v++) rec[v * cells + ri] = U[v];
	rec[R_RINV * cells + ri] = d.rinv;
	rec[R_PT * cells + ri] = d.pt;
	if (CX) rec[(R_CF + 0) * cells + ri] = d.cf[0];
	if (CY) rec[(R_CF + 1) * cells + ri] = d.cf[1];
	bad[ri] = uint8_t(d.bad & ~OPEN_WAVE);
	open = open or d.bad == OPEN_WAVE;
	// the fast speed along z, for the caller's z faces
	return CZ ? d.cf[2] : 0.0;
}

// one cell of a record slot seen from a face normal to axis A (rotation by index permutation),
// with its fast speed along A
template <int A>
__device__ __forceinline__ Side side_at(const double* rec, const uint8_t* bad, const int cells, const int ri,
                                        const double cf)
{
	Side s;
	s.rho = rec[ri];
	rotate<A>(rec[1 * cells + ri], rec[2 * cells + ri], rec[3 * cells + ri], s.m0, s.m1, s.m2);
	s.E = rec[4 * cells + ri];
	rotate<A>(rec[5 * cells + ri], rec[6 * cells + ri], rec[7 * cells + ri], s.b0, s.b1, s.b2);
	s.rinv = rec[R_RINV * cells + ri];
	s.pt = rec[R_PT * cells + ri];
	s.p = 0.0;  // not read without a background field
	s.cf = cf;
	s.v0 = s.m0 * s.rinv;
	s.v1 = s.m1 * s.rinv;
	s.v2 = s.m2 * s.rinv;
	s.bad = bad[ri];
	return s;
}

/*
Solves one z face, folds its speed into the running max and returns the
unscaled flux in the xyz frame (the update multiplies by dt / dz once per
cell).  Each kernel inlines this once, so a z face is computed by the same
instructions wherever it lies in the tiling.
*/
template <int SOLVER, int CELLS>
__device__ __forceinline__ void solve_z(const Step_Params& P, const double* rec_l, const uint8_t* bad_l,
                                        const double* rec_r, const uint8_t* bad_r, const int ri, const double cf_l,
                                        const double cf_r, double d[8], double& smax, bool& zero, const int i,
                                        const int j, const int k)
{
	const Side L = side_at<2>(rec_l, bad_l, CELLS, ri, cf_l);
	const Side R = side_at<2>(rec_r, bad_r, CELLS, ri, cf_r);
	double F[8];
	uint32_t flag = 0;
	// the side an HLLD flux is taken from, read again from the records (see flux_hlld)
	const auto pick = [&](const bool left) {
		return side_at<2>(left ? rec_l : rec_r, left ? bad_l : bad_r, CELLS, ri, left ? cf_l : cf_r);
	};
	const double s = solve_face<SOLVER>(L, R, P.gas, F, flag, pick);
	if (flag != 0) record_failure(P, flag, i, j, k, 3);
	smax = larger(s, smax);
	zero = zero or no_speed(s);
	d[0] = F[0];
	unrotate<2>(F[1], F[2], F[3], d[1], d[2], d[3]);
	d[4] = F[4];
	unrotate<2>(F[5], F[6], F[7], d[5], d[6], d[7]);
}

/*
One x or y face (axis a, 0 or 1, known only at run time) between record
positions rl and rr of a slot.  The x and y faces of a plane share
this one inlined solver instance (half the code of one instance per axis,
which the instruction cache rewards).  The rotation into the face frame is
a choice of record rows to read, two offsets per side: x reads rows m_x,
m_y, m_z; y reads m_y, m_z (one row on) and m_x.  The unscaled flux goes to
out[r][rr] in the face frame, Flux_Rows<SOLVER>::N rows (the caller rotates
it back).  Returns the face's signal speed.
*/
template <int SOLVER, bool ZACT, class T>
__device__ __forceinline__ double solve_xy(const Step_Params& P, const double* rec, const uint8_t* bad,
                                           const int rl, const int rr, const int a, double* const out,
                                           const int gx0, const int gy0, const int k)
{
	constexpr int C = T::CELLS;
	const int near = a * C, far = a == 0 ? 2 * C : 0;
	auto side = [&](const int r) {
		const double* const c = rec + r;
		const double* const n = c + near;
		const double* const f = c + far;
		Side s;
		s.rho = c[0];
		s.m0 = n[C];
		s.m1 = n[2 * C];
		s.m2 = f[C];
		s.E = c[4 * C];
		s.b0 = n[5 * C];
		s.b1 = n[6 * C];
		s.b2 = f[5 * C];
		s.rinv = c[R_RINV * C];
		s.pt = c[R_PT * C];
		s.p = 0.0;  // not read without a background field
		s.cf = n[R_CF * C];
		s.v0 = s.m0 * s.rinv;
		s.v1 = s.m1 * s.rinv;
		s.v2 = s.m2 * s.rinv;
		s.bad = bad[r];
		return s;
	};
	const Side L = side(rl);
	const Side R = side(rr);
	double F[8];
	uint32_t flag = 0;
	const auto pick = [&](const bool left) { return side(left ? rl : rr); };
	const double sp = solve_face<SOLVER>(L, R, P.gas, F, flag, pick);
	if (flag != 0) {
		// the face's negative cell: one of the tile's rows (the first the halo row below), or the column
		// left of it
		const int tw = ZACT ? P.tw : T::FLAT + 2, columns = ZACT ? (P.th + 2 * T::JO) * tw : 1 << 30;
		const int i = rl < columns ? rl % tw - (ZACT ? 0 : 1) : -1, j = rl < columns ? rl / tw - T::JO : rl - columns;
		record_failure(P, flag, gx0 + i, gy0 + j, k, a + 1);
	}
	out[rr] = F[0];
	out[C + rr] = F[1];
	out[2 * C + rr] = F[2];
	out[3 * C + rr] = F[3];
	out[4 * C + rr] = F[4];
	out[5 * C + rr] = F[6];
	out[6 * C + rr] = F[7];
	if (Flux_Rows<SOLVER>::N == 8) out[7 * C + rr] = F[5];
	return sp;
}

// ------------------------------------------------------------------ the step

// a step's dt and stop found within tile_step (shared memory); first: this block advances the clock
struct Late_Start {
	double dt;
	int stop;
	int first;
};

// the planes [kb, ke) of block row bz: a z chunk, or with kpart 1 the first (bz 0) or the last
// (bz 1) plane alone, or with kpart 2 a chunk of the planes between them
__device__ __forceinline__ void tile_planes(const Step_Params& P, const int bz, int& kb, int& ke)
{
	const int nz = P.L.n[2];
	const int kbase = P.kpart == 2 ? 1 : 0, ktop = P.kpart == 2 ? nz - 1 : nz;
	kb = P.kpart == 1 ? (bz == 0 ? 0 : nz - 1) : kbase + bz * P.kchunk;
	ke = P.kpart == 1 ? kb + 1 : min(ktop, kb + P.kchunk);
}

/*
A step of a grid that stopped: the tile's cells are copied into the new
state unchanged, with the ghosts a step writes, so that both states hold
the failing step's result.  CO: loads at L2 (see load_record).
*/
template <bool CO>
__device__ void tile_hold(const Step_Params& P, const int bx, const int by, const int bz)
{
	int kb, ke;
	tile_planes(P, bz, kb, ke);
	const int ty = threadIdx.x / P.tw, tx = threadIdx.x - ty * P.tw;
	const int gx = bx * P.tw + tx, gy = by * P.th + ty;
	if (ty >= P.th or gx >= P.L.n[0] or gy >= P.L.n[1]) return;
	for (int k = kb; k < ke; k++) {
		const long long off = P.L.offset(gx, gy, k);
		double U[8];
		#pragma unroll
		for (int v = 0; v < 8; v++) U[v] = CO ? __ldcg(P.in + v * P.L.var + off) : P.in[v * P.L.var + off];
		write_cell(P, gx, gy, k, U, 0.0);
	}
}

/*
Judges the cells of a tile whose wave speed round-off decides, as the
reference judges them at each face they have: along its normal, and the face
is named by the cell before it.  An own cell has two faces along each axis; a
ghost of a side that is not periodic has one, along the side's axis.  By
blocks that met such a cell, after their planes (in the planes' loop the
judgement took 1.4 % of a 256^3 step, unused: registers and code).
*/
__device__ void settle_tile(const Step_Params& P, const int bx, const int by, const int bz)
{
	int kb, ke;
	tile_planes(P, bz, kb, ke);
	const int ty = threadIdx.x / P.tw, tx = threadIdx.x - ty * P.tw;
	const int gx = bx * P.tw + tx, gy = by * P.th + ty;
	if (ty >= P.th or gx >= P.L.n[0] or gy >= P.L.n[1]) return;
	// axis a, of the cell at (i, j, k): whether the reference refuses it
	const auto refused = [&](const int a, const int i, const int j, const int k) {
		const long long off = P.L.offset(i, j, k);
		double U[8];
		#pragma unroll
		for (int v = 0; v < 8; v++) U[v] = __ldcg(P.in + v * P.L.var + off);
		return derive_along(a, U, P.gas).bad == PAMHD_FLAG_WAVE_SPEED;
	};
	#pragma unroll 1
	for (int k = kb; k < ke; k++) {
		#pragma unroll 1
		for (int a = 0; a < 3; a++) {
			if (not P.active[a]) continue;
			const int di = a == 0 ? 1 : 0, dj = a == 1 ? 1 : 0, dk = a == 2 ? 1 : 0;
			const int at = a == 0 ? gx : (a == 1 ? gy : k);
			const bool own = refused(a, gx, gy, k);
			if (own or (not P.periodic[a] and at == 0 and refused(a, gx - di, gy - dj, k - dk))) {
				record_failure(P, PAMHD_FLAG_WAVE_SPEED, gx - di, gy - dj, k - dk, a + 1);
			}
			if (own or (not P.periodic[a] and at == P.L.n[a] - 1 and refused(a, gx + di, gy + dj, k + dk))) {
				record_failure(P, PAMHD_FLAG_WAVE_SPEED, gx, gy, k, a + 1);
			}
		}
	}
}

/*
One work item of a step: the tile (bx, by) of tw x th columns over the z
chunk bz, marched plane by plane; the face speeds are folded into
s0, s1, s2 and zero (flushed by the caller).  Shared by the single-grid
and the batched kernels, so that both compute the same bits.

The records of plane k (two slots alternate, so that the z face between
planes k and k + 1 can read both) are staged an iteration ahead; per plane:
  (a) a block barrier: the plane's records are there, and the fluxes of the
      plane before were used;
  (b) every x and y face of the plane into shared memory, then the arrival
      at the split barrier;
  (c) what needs no other warp: the next plane's records, and the z face
      above each own cell, whose two sides the thread staged itself;
  (d) the wait for the other warps' x and y fluxes, then the own cell:
      state plus x and y flux differences plus its two z fluxes, written.
Stage and z face between arrival and wait leave a warp that has an extra
pass in (b) two thirds of a plane's work to catch up in: with one barrier
before and one after (b) warps spent 18 % of their time at the two, and a
256^3 HLLD step took 1.73 ms; split, 1.56 ms.
A grid without z faces (ZACT false) has one plane and nothing to overlap:
one record slot and two block barriers.  There a block finds the step's dt
late: thread 0 while its first loads are under way, the block behind its
first barrier, instead of before the loads (512^2 HLLD 33.1 -> 32.0 us per
step; the 3-D tiles, which start once per chunk of planes, lost 1.6 % that way and
Roe's 4 % to registers).
*/
template <int SOLVER, int TY, bool ZACT, bool CO = false, bool LATE = false>
__device__ __forceinline__ void tile_step(const Step_Params& P, double* const smem, Split_Barrier& bar,
                                          double dt, const int bx, const int by, const int bz,
                                          double& s0, double& s1, double& s2, bool& zero, bool& open,
                                          Late_Start* const late = nullptr)
{
	constexpr int NF = Flux_Rows<SOLVER>::N;
	using T = Tile<TY, ZACT, NF>;
	double* const rec_base = smem;
	double* const fx = smem + T::SLOTS * T::REC;   // [NF][CELLS]
	double* const fy = fx + NF * T::CELLS;         // [NF][CELLS] (y active)
	uint8_t* const bad_base = reinterpret_cast<uint8_t*>(fx + NF * T::CELLS * (1 + T::JO));

	constexpr bool YACT = TY > 1;
	const int nx = P.L.n[0], ny = P.L.n[1];
	constexpr int THREADS = TX * TY;
	// the tile's columns one per thread, x fastest; the threads past them (tw th <= THREADS) own none
	// (grids without z faces keep 32 x TY, or 31 x 1 columns, known at compile time)
	const int tw = ZACT ? P.tw : T::FLAT, th = ZACT ? P.th : TY, t = threadIdx.x;
	const int ty = t / tw, tx = t - ty * tw;
	const int gx0 = bx * tw, gy0 = by * th;
	const int gx = gx0 + tx, gy = gy0 + ty;
	const bool own = ty < th and gx < nx and gy < ny;
	// the +x / +y ghost of a partial tile lies inside the tile's own columns / rows
	const bool stage = ty < th and gx <= nx and (TY == 1 ? gy == 0 : gy <= ny);
	// the planes of this block
	int kb, ke;
	tile_planes(P, bz, kb, ke);
	const int kfirst = ZACT ? kb - 1 : kb;
	const int klast = ZACT ? ke : ke - 1;
	// record positions.  Tiles that march in z: the rows of columns, the halo rows first and last, tw
	// apart, so that a warp's own cells are 32 consecutive doubles whatever tw is (a row pitch of
	// tw + 2 makes two-way bank conflicts wherever a warp crosses a row's end); then the halo columns
	// left and right.  Others, whose rows are warps: the halo columns at their rows' ends.
	const int pitch = ZACT ? tw : T::FLAT + 2;
	const int left_column = (th + 2 * T::JO) * tw, right_column = left_column + th;
	const auto at = [&](const int row, const int x) { return (row + T::JO) * pitch + x + (ZACT ? 0 : 1); };
	const auto left_of_row = [&](const int row) { return ZACT ? left_column + row : at(row, -1); };
	const auto right_of_row = [&](const int row) { return ZACT ? right_column + row : at(row, tw); };
	const int ri = at(ty, tx);
	const int r_east = ZACT and tx == tw - 1 ? right_of_row(ty) : ri + 1;
	// the flux terms are dt F / dx: dt / dx once per axis and cell
	double cx = dt * P.inv_len[0], cy = dt * P.inv_len[1], cz = dt * P.inv_len[2];

	// this thread's halo cell of planes with x / y faces, if any: first the rows below and above the
	// tile, then the columns left and right of it
	int hri = -1;
	long long hoff = 0;
	{
		const int rows = YACT ? 2 * tw : 0;
		if (t < rows) {
			const bool top = t >= tw;
			const int x = top ? t - tw : t, hy = top ? gy0 + th : gy0 - 1;
			if (gx0 + x < nx and hy <= ny) {
				hri = at(top ? th : -1, x);
				hoff = P.L.offset(gx0 + x, hy, 0);
			}
		} else if (t < rows + 2 * th) {
			const bool right = t >= rows + th;
			const int y = t - rows - (right ? th : 0), hx = right ? gx0 + tw : gx0 - 1;
			if (gy0 + y < ny and hx <= nx) {
				hri = right ? right_of_row(y) : left_of_row(y);
				hoff = P.L.offset(hx, gy0 + y, 0);
			}
		}
	}
	const long long col = P.L.offset(gx, gy, 0);
	// a plane's records: own cells, and the halo.  Returns the own column's fast speed along z.
	const auto stage_plane = [&](const int k) -> double {
		const int slot = ZACT ? (k - kfirst) & 1 : 0;
		double* const rec = rec_base + slot * T::REC;
		uint8_t* const bad = bad_base + slot * T::CELLS;
		double cfz = 0.0;
		if (stage) {
			cfz = load_record<true, YACT, ZACT, CO>(P, rec, bad, T::CELLS, ri, col + k * P.L.plane, open, [&]() {
				if (LATE and t == 0) find_dt(P, &late->dt, late->first, &late->stop);
				// the plane after this one on its way to L2, a plane's time before its loads: they waited
				// for DRAM a seventh of the warps' time (256^3 HLLD 1.46 -> 1.41 ms per step; copying it
				// into the record slot with cp.async, 8 bytes a lane, cost 8 %)
				if (ZACT and k < klast) {
					const double* const next = P.in + col + (k + 1) * P.L.plane;
					#pragma unroll
					for (int v = 0; v < 8; v++) asm volatile("prefetch.global.L2 [%0];" :: "l"(next + v * P.L.var));
				}
			});
		}
		if (k >= kb and k < ke and hri >= 0) {
			load_record<true, YACT, false, CO>(P, rec, bad, T::CELLS, hri, hoff + k * P.L.plane, open, []() {});
		}
		return cfz;
	};

	// the x and y faces this thread solves, at most one per pass, as positive record position |
	// (ZACT) negative one << 10 | axis << 20, or -1: an owner its -x and its -y face; the tile's +x and
	// +y faces (numbered in this order) go to the threads without a cell, two each, and what they
	// leave to a further pass of the last warps.  32 x TY tiles of one plane (every thread owns a
	// column) give the last two warps a pass each for the +x and the +y faces, so that a pass has one
	// axis, known to the whole warp (512^2 Roe: 66 us per step, 70 with mixed axes)
	constexpr int NONE = -1;
	const auto face_of = [](const int rr, const int rl, const int a) { return rr | (ZACT ? rl << 10 : 0) | (a << 20); };
	const auto extra = [&](const int e) -> int {
		if (e < th) return (gx0 + tw <= nx and gy0 + e < ny) ? face_of(right_of_row(e), at(e, tw - 1), 0) : NONE;
		const int x = e - th;
		return (YACT and x < tw and gy0 + th <= ny and gx0 + x < nx) ? face_of(at(th, x), at(th - 1, x), 1) : NONE;
	};
	const int spare = THREADS - tw * th;
	int face0 = NONE, face1 = NONE;
	if (ty < th) {
		if (gx <= nx and gy < ny) face0 = face_of(ri, tx == 0 ? left_of_row(ty) : ri - 1, 0);
		if (YACT and gy <= ny and gx < nx) face1 = face_of(ri, ri - pitch, 1);
	} else {
		face0 = extra(t - tw * th);
		if (YACT) face1 = extra(t - tw * th + spare);
	}
	const int last = THREADS - 1 - t;
	const int face2 = ZACT ? extra(2 * spare + last)
	                : (YACT and last >= 32 and last - 32 < th ? extra(last - 32) : NONE);
	const int face3 = not ZACT and YACT and last < tw ? extra(th + last) : NONE;
	// a cell on the grid's x or y edge also writes a ghost
	const bool edge = gx == 0 or gx == nx - 1 or gy == 0 or gy == ny - 1;

	// the scaled flux of the -z face of the own cell of plane k
	double low[8];
	#pragma unroll
	for (int v = 0; v < 8; v++) low[v] = 0.0;
	// the own column's fast speed along z in plane k
	double cfz = 0.0;

	#pragma unroll 1
	for (int k = kfirst - 1; k < ke; k++) {
		const int slot = ZACT ? (k - kfirst) & 1 : 0;
		double* const rec = rec_base + slot * T::REC;
		uint8_t* const bad = bad_base + slot * T::CELLS;
		double* const next = rec_base + (slot ^ 1) * T::REC;
		uint8_t* const next_bad = bad_base + (slot ^ 1) * T::CELLS;
		const bool inner = k >= kb;

		if (inner) {
			__syncthreads();
			if (LATE) {
				if (late->stop) {
					tile_hold<CO>(P, bx, by, bz);
					return;
				}
				dt = late->dt;
				cx = dt * P.inv_len[0];
				cy = dt * P.inv_len[1];
			}
			// (b) x and y faces, all through one call site
			#pragma unroll 1
			for (int pass = 0; pass < (ZACT ? 3 : (YACT ? 4 : 1)); pass++) {
				// own x, own y, further ones; or (one plane) own x, further x, own y, further y
				const int face = pass == 0 ? face0 : (pass == (ZACT ? 1 : 2) ? face1 : (pass == 3 ? face3 : face2));
				if (face >= 0) {
					const int a = ZACT ? face >> 20 : pass >> 1;
					const int rr = face & 1023, rl = ZACT ? (face >> 10) & 1023 : rr - (a == 0 ? 1 : pitch);
					const double sp = solve_xy<SOLVER, ZACT, T>(P, rec, bad, rl, rr, a, fx + a * NF * T::CELLS, gx0, gy0, k);
					const double m = larger(sp, a == 0 ? s0 : s1);
					if (a == 0) s0 = m; else s1 = m;
					zero = zero or no_speed(sp);
				}
			}
			if (ZACT) bar.arrive();
			else __syncthreads();
		}
		// (c) the next plane's records (their slot's plane k - 1 was last read before this plane's
		// barrier, but for own cells), and the z face between the planes
		const double cfz_below = cfz;
		if (k < klast) cfz = stage_plane(k + 1);
		double high[8];
		#pragma unroll
		for (int v = 0; v < 8; v++) high[v] = 0.0;
		if (ZACT and k >= kfirst and own) {
			solve_z<SOLVER, T::CELLS>(P, rec, bad, next, next_bad, ri, cfz_below, cfz, high, s2, zero, gx, gy, k);
			#pragma unroll
			for (int v = 0; v < 8; v++) high[v] = __dmul_rn(high[v], cz);
		}
		// (d) the own cell: U += (F- - F+) dt/dx, then y, then z (solve.hpp:1551-1587)
		if (inner) {
			// without the other warps' fluxes (a wait that gave up) the cell stays unwritten
			const bool arrived = not ZACT or bar.wait(P);
			if (own and arrived) {
				// the flux row of each xyz variable in the x and the y face frames; -1: the normal
				// field component, whose flux is zero unless the solver keeps an eighth row
				constexpr int XROW[8] = {0, 1, 2, 3, 4, NF == 8 ? 7 : -1, 5, 6};
				constexpr int YROW[8] = {0, 3, 1, 2, 4, 6, NF == 8 ? 7 : -1, 5};
				double Un[8];
				#pragma unroll
				for (int v = 0; v < 8; v++) {
					Un[v] = rec[v * T::CELLS + ri];
					if (XROW[v] >= 0) {
						const double* f = fx + XROW[v] * T::CELLS;
						Un[v] = __fma_rn(__dsub_rn(f[ri], f[r_east]), cx, Un[v]);
					}
				}
				if (YACT) {
					#pragma unroll
					for (int v = 0; v < 8; v++) {
						if (YROW[v] >= 0) {
							const double* f = fy + YROW[v] * T::CELLS + ri;
							Un[v] = __fma_rn(__dsub_rn(f[0], f[pitch]), cy, Un[v]);
						}
					}
				}
				if (ZACT) {
					#pragma unroll
					for (int v = 0; v < 8; v++) Un[v] = __dadd_rn(Un[v], __dsub_rn(low[v], high[v]));
				}
				if (edge or (ZACT and (k == 0 or k == P.L.n[2] - 1))) {
					write_cell(P, gx, gy, k, Un, dt);
				} else {
					double* const to = P.out + col + k * P.L.plane;
					#pragma unroll
					for (int v = 0; v < 8; v++) to[v * P.L.var] = Un[v];
				}
			}
		}
		#pragma unroll
		for (int v = 0; v < 8; v++) low[v] = high[v];
	}
}

/*
The batched step: every box of an ensemble advances one step in one launch.
Blocks walk the work-item table (box, tile x, tile y, z chunk) with a grid
stride; each box has its own parameters (state buffers, layout, boundary
kinds, reduction ring, clock, status), so each advances with its own dt.
The block holding a box's first item advances that box's clock.
*/
template <int SOLVER, int TY, bool ZACT>
__global__ void __launch_bounds__(TX * TY, Tile_Kind::resident_of(SOLVER, TY, ZACT)) batch_step_kernel(const Step_Params* __restrict__ boxes,
                                                                  const int4* __restrict__ items,
                                                                  const int nitems, const int phase,
                                                                  const int barrier_polls)
{
	extern __shared__ __align__(16) double smem[];
	__shared__ Step_Params sp;
	__shared__ double s_dt;
	__shared__ int s_stop;
	__shared__ unsigned long long s_bar;
	const int tid = threadIdx.y * blockDim.x + threadIdx.x;
	Split_Barrier bar = split_barrier(&s_bar);
	if (tid == 0) bar.init(TY);
	for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
		const int4 w = items[item];
		__syncthreads();  // the previous item is done with sp
		if (tid == 0) {
			sp = boxes[w.x];
			sp.phase = phase;
			sp.barrier_polls = barrier_polls;
		}
		__syncthreads();
		const bool first = w.y == 0 and w.z == 0 and w.w == 0;
		const double dt = begin_step(sp, &s_dt, first, &s_stop);
		const int tiles_x = (sp.L.n[0] + sp.tw - 1) / sp.tw;
		if (s_stop) {
			tile_hold<false>(sp, w.y % tiles_x, w.y / tiles_x, w.z);
			continue;
		}
		double s0 = 0.0, s1 = 0.0, s2 = 0.0;
		bool zero = false, open = false;
		tile_step<SOLVER, TY, ZACT>(sp, smem, bar, dt, w.y % tiles_x, w.y / tiles_x, w.z, s0, s1, s2, zero, open);
		double smax[3] = {s0, s1, s2};
		if (flush_speeds(sp, smax, zero, open)) settle_tile(sp, w.y % tiles_x, w.y / tiles_x, w.z);
	}
}

// the (ghost dimension d, side, tangential axis e) combinations with ghost-ghost faces
__device__ __forceinline__ int boundary_combos(const Step_Params& P, int combos[12][3])
{
	int nc = 0;
	for (int d = 0; d < 3; d++) {
		if (not P.active[d] or P.periodic[d]) continue;
		for (int side = 0; side < 2; side++) {
			// the ghost layer of a slab cut is the neighbouring slab's interior: its faces are counted there
			if ((side ? P.bc_hi[d] : P.bc_lo[d]) == PAMHD_BC_EXTERNAL) continue;
			for (int e = 0; e < 3; e++) {
				if (e == d or not P.active[e]) continue;
				combos[nc][0] = d; combos[nc][1] = side; combos[nc][2] = e;
				nc++;
			}
		}
	}
	return nc;
}

// faces of one combination: along a slab cut at the high side, the face into the ghost plane is
// this slab's (the one into the low ghost plane is the lower neighbour's)
__device__ __forceinline__ long long boundary_count(const Step_Params& P, const int d, const int e)
{
	const int f = 3 - d - e;
	const int ne = (P.periodic[e] or P.bc_hi[e] == PAMHD_BC_EXTERNAL) ? P.L.n[e] : P.L.n[e] - 1;
	return (long long)ne * P.L.n[f];
}

// face t of combination (d, side, e): solved for its speed only (CO: loads at L2, see load_record)
template <int SOLVER, bool CO>
__device__ __forceinline__ void boundary_face(const Step_Params& P, const int d, const int side, const int e,
                                              const long long t, double smax[3], bool& zero)
{
	const int f = 3 - d - e;
	const int ne = (P.periodic[e] or P.bc_hi[e] == PAMHD_BC_EXTERNAL) ? P.L.n[e] : P.L.n[e] - 1;
	int a[3], b[3];
	a[d] = b[d] = side ? P.L.n[d] : -1;
	a[e] = int(t % ne);
	b[e] = (a[e] + 1 == P.L.n[e] and P.periodic[e]) ? 0 : a[e] + 1;
	a[f] = b[f] = int(t / ne);
	double UA[8], UB[8];
	const long long oa = P.L.offset(a[0], a[1], a[2]), ob = P.L.offset(b[0], b[1], b[2]);
	#pragma unroll
	for (int v = 0; v < 8; v++) {
		UA[v] = CO ? __ldcg(P.in + v * P.L.var + oa) : P.in[v * P.L.var + oa];
		UB[v] = CO ? __ldcg(P.in + v * P.L.var + ob) : P.in[v * P.L.var + ob];
	}
	const Derived da = derive_along(e, UA, P.gas), db = derive_along(e, UB, P.gas);
	Side L, R;
	auto fill = [e](Side& s, const double U[8], const Derived& dd) {
		s.rho = U[0];
		s.E = U[4];
		double m[3] = {U[1], U[2], U[3]}, B[3] = {U[5], U[6], U[7]};
		const int i0 = e, i1 = (e + 1) % 3, i2 = (e + 2) % 3;
		s.m0 = m[i0]; s.m1 = m[i1]; s.m2 = m[i2];
		s.b0 = B[i0]; s.b1 = B[i1]; s.b2 = B[i2];
		s.rinv = dd.rinv;
		s.v0 = s.m0 * s.rinv; s.v1 = s.m1 * s.rinv; s.v2 = s.m2 * s.rinv;
		s.p = dd.p;
		s.pt = dd.pt;
		s.cf = dd.cf[0];
		s.bad = dd.bad;
	};
	fill(L, UA, da);
	fill(R, UB, db);
	double F[8];
	uint32_t flag = 0;
	const double sp = solve_face<SOLVER>(L, R, P.gas, F, flag);
	if (flag != 0) record_failure(P, flag, a[0], a[1], a[2], e + 1);
	smax[e] = fmax(smax[e], sp);
	zero = zero or not (sp > 0.0);
}

/*
Speeds of the faces between two boundary ghosts of a non-periodic side
(cells of class 0 on both sides), by threads first, first + stride, ...
The reference solves those faces too (mhd/solve.hpp:254-311 visits every
cell of class >= 0) and their speeds enter the timestep (:1965-2005); their
fluxes change nothing.
*/
template <int SOLVER, bool CO>
__device__ __forceinline__ void boundary_faces(const Step_Params& P, const long long first, const long long stride,
                                               double smax[3], bool& zero)
{
	int combos[12][3];
	const int nc = boundary_combos(P, combos);
	#pragma unroll 1
	for (int c = 0; c < nc; c++) {
		const long long count = boundary_count(P, combos[c][0], combos[c][2]);
		#pragma unroll 1
		for (long long t = first; t < count; t += stride) {
			boundary_face<SOLVER, CO>(P, combos[c][0], combos[c][1], combos[c][2], t, smax, zero);
		}
	}
}

/*
One step of a grid.  The last P.boundary layers of blocks solve the
ghost-ghost faces of non-periodic sides: they read and reduce what the
tiles do, and fill the SMs as the tiles' last wave drains (as a launch of
its own before the step they took 12 of 110 us on a 96 x 64 x 50 grid).
*/
template <int SOLVER, int TY, bool ZACT>
__global__ void __launch_bounds__(TX * TY, Tile_Kind::resident_of(SOLVER, TY, ZACT)) step_kernel(const Step_Params P)
{
	extern __shared__ __align__(16) double smem[];
	constexpr bool LATE = not ZACT and SOLVER != PAMHD_ROE_ATHENA;
	__shared__ Late_Start start;
	__shared__ unsigned long long s_bar;
	Split_Barrier bar = split_barrier(&s_bar);
	const bool first_block = blockIdx.x == 0 and blockIdx.y == 0 and blockIdx.z == 0;
	if (threadIdx.x == 0) {
		bar.init(TY);
		start.first = first_block ? 1 : 0;
	}
	double dt = 0.0;
	if (not LATE or blockIdx.z >= gridDim.z - P.boundary) {
		dt = begin_step(P, &start.dt, first_block, &start.stop);
		if (start.stop) {
			if (blockIdx.z < gridDim.z - P.boundary) tile_hold<false>(P, blockIdx.x, blockIdx.y, blockIdx.z);
			return;
		}
	}
	double s0 = 0.0, s1 = 0.0, s2 = 0.0;
	bool zero = false;
	const int chunks = gridDim.z - P.boundary;
	if ((int)blockIdx.z >= chunks) {
		double smax[3] = {0.0, 0.0, 0.0};
		const long long block = (blockIdx.z - chunks) * (long long)gridDim.x * gridDim.y + blockIdx.y * gridDim.x + blockIdx.x;
		boundary_faces<SOLVER, false>(P, block * (TX * TY) + threadIdx.x,
		                              P.boundary * (long long)gridDim.x * gridDim.y * (TX * TY), smax, zero);
		flush_speeds(P, smax, zero);
		return;
	}
	bool open = false;
	tile_step<SOLVER, TY, ZACT, false, LATE>(P, smem, bar, dt, blockIdx.x, blockIdx.y, blockIdx.z, s0, s1, s2, zero, open, &start);
	if (LATE and start.stop) return;
	double smax[3] = {s0, s1, s2};
	if (flush_speeds(P, smax, zero, open)) settle_tile(P, blockIdx.x, blockIdx.y, blockIdx.z);
}

// the ghost-ghost faces of every box of a batch, blockIdx.y the box
template <int SOLVER>
__global__ void batch_boundary_speed_kernel(const Step_Params* __restrict__ boxes, const int phase)
{
	__shared__ Step_Params sp;
	if (threadIdx.x == 0) {
		sp = boxes[blockIdx.y];
		sp.phase = phase;
	}
	__syncthreads();
	// a box that stopped solves no face (the value is the same for every thread)
	if (stopped_before(sp)) return;
	double smax[3] = {0.0, 0.0, 0.0};
	bool zero = false;
	boundary_faces<SOLVER, false>(sp, blockIdx.x * (long long)blockDim.x + threadIdx.x,
	                              (long long)gridDim.x * blockDim.x, smax, zero);
	flush_speeds(sp, smax, zero);
}

// ------------------------------------------------------------------ layout and ghosts

// the padded offset of interior cell t of n (x fastest), with 32-bit quotients where n allows: three
// 64-bit ones per cell took longer than the cell's 16 bytes
__device__ __forceinline__ long long cell_offset(const Layout& L, const long long t, const long long n)
{
	if (n <= 0xffffffffll) {
		const unsigned int u = (unsigned int)t, n0 = (unsigned int)L.n[0], n1 = (unsigned int)L.n[1];
		const unsigned int q = u / n0, k = q / n1;
		return L.offset(int(u - q * n0), int(q - k * n1), int(k));
	}
	return L.offset(int(t % L.n[0]), int((t / L.n[0]) % L.n[1]), int(t / ((long long)L.n[0] * L.n[1])));
}

__global__ void scatter_kernel(const double* __restrict__ packed, double* __restrict__ var, const Layout L)
{
	const long long n = (long long)L.n[0] * L.n[1] * L.n[2];
	for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
		var[cell_offset(L, t, n)] = packed[t];
	}
}

__global__ void gather_kernel(const double* __restrict__ var, double* __restrict__ packed, const Layout L)
{
	const long long n = (long long)L.n[0] * L.n[1] * L.n[2];
	for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
		packed[t] = var[cell_offset(L, t, n)];
	}
}

/*
Fills every face ghost of `state` from its interior (periodic image, COPY)
or the configured VALUE state (apply_boundaries, mhd/boundaries.hpp:1261).
value_lo/hi are passed through the params of the host context.
*/
struct Ghost_Values {
	double lo[3][8];
	double hi[3][8];
};

__global__ void fill_ghosts_kernel(const Step_Params P, double* state, const Ghost_Values V)
{
	for (int d = 0; d < 3; d++) {
		if (not P.active[d]) continue;
		const int e = (d + 1) % 3, f = (d + 2) % 3;
		const long long count = (long long)P.L.n[e] * P.L.n[f];
		for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < 2 * count;
		     t += (long long)gridDim.x * blockDim.x) {
			const int side = int(t / count);
			const long long r = t % count;
			int c[3];
			c[e] = int(r % P.L.n[e]);
			c[f] = int(r / P.L.n[e]);
			c[d] = side ? P.L.n[d] : -1;
			int s[3] = {c[0], c[1], c[2]};
			double U[8];
			const int kind = side ? P.bc_hi[d] : P.bc_lo[d];
			if (kind == PAMHD_BC_EXTERNAL) continue;  // written by the halo exchange
			if (P.periodic[d]) {
				s[d] = side ? 0 : P.L.n[d] - 1;
				const long long o = P.L.offset(s[0], s[1], s[2]);
				for (int v = 0; v < 8; v++) U[v] = state[v * P.L.var + o];
			} else if (kind == PAMHD_BC_COPY) {
				s[d] = side ? P.L.n[d] - 1 : 0;
				const long long o = P.L.offset(s[0], s[1], s[2]);
				for (int v = 0; v < 8; v++) U[v] = state[v * P.L.var + o];
			} else {
				for (int v = 0; v < 8; v++) U[v] = side ? V.hi[d][v] : V.lo[d][v];
			}
			store_cell(state, P.L, c[0], c[1], c[2], U);
		}
	}
}

// ------------------------------------------------------------------ the persistent batched run

// marks every box's status with PAMHD_FLAG_TIMEOUT, once per launch
__device__ void run_timeout(Run_Sync* sync, const Step_Params* boxes, const int nboxes)
{
	if (atomicExch(&sync->error, 1u) == 0u) {
		for (int b = 0; b < nboxes; b++) atomicOr(&boxes[b].status->flags, (unsigned int)PAMHD_FLAG_TIMEOUT);
	}
}

/*
The batched ensemble advanced nsteps steps in one launch.  The grid is the
resident capacity of the SMs (a cooperative launch, so that every block
runs at once).  The work is the sequence of (step, work item) pairs, the
items of a step being the boxes' tiles as in batch_step_kernel, largest
boxes first, then, for boxes with non-periodic sides, chunks of their
ghost-ghost faces, whose speeds enter the timestep.  Blocks take the pairs
one at a time from a shared counter.  An item of step s of box b first
waits until all items of step s - 1 of box b are done (done[b] counts the
box's finished items): the only dependency of a box's step, since each box
has its own state, reduction ring and clock.  Boxes therefore advance at
their own pace, without a grid-wide barrier, and a block that finishes
early takes the next item, of this step or the next.  The pairs are handed
out in order and all blocks are resident, so the earliest unfinished item
has its dependency met: the run always progresses.  A wait gives up after
wait_limit polls: it sets the error word and PAMHD_FLAG_TIMEOUT on every
box, and every block stops at its next item.  boxes_even / boxes_odd are
the boxes' parameters of the two state parities, the first used by step
step0.  Loads that read what another block wrote before go through L2 (CO).
*/
template <int SOLVER, int TY, bool ZACT>
__global__ void __launch_bounds__(TX * TY, Tile_Kind::resident_of(SOLVER, TY, ZACT)) batch_run_kernel(
	const Step_Params* __restrict__ boxes_even, const Step_Params* __restrict__ boxes_odd,
	const int4* __restrict__ items, const int nitems, const int* __restrict__ box_items, unsigned int* done,
	const int nboxes, const long long step0, const int nsteps, Run_Sync* sync, const long long wait_limit)
{
	extern __shared__ __align__(16) double smem[];
	__shared__ Step_Params sp;
	__shared__ double s_dt;
	__shared__ unsigned int s_q;
	__shared__ int s_go;
	__shared__ int s_stop;
	__shared__ unsigned long long s_bar;
	const int tid = threadIdx.y * blockDim.x + threadIdx.x;
	Split_Barrier bar = split_barrier(&s_bar);
	if (tid == 0) bar.init(TY);
	const int nthreads = blockDim.x * blockDim.y;
	const unsigned int total = (unsigned int)nsteps * (unsigned int)nitems;
	for (;;) {
		__syncthreads();  // the previous item is done with sp and the shared words
		if (tid == 0) {
			volatile unsigned int* verr = &sync->error;
			s_q = *verr != 0u ? total : atomicAdd(&sync->next, 1u);
		}
		__syncthreads();
		const unsigned int q = s_q;
		if (q >= total) return;
		const int s = int(q / (unsigned int)nitems);
		const int4 w = items[q % (unsigned int)nitems];
		const Step_Params* boxes = (s & 1) ? boxes_odd : boxes_even;
		if (tid == 0) {
			// the box's previous step: all its items done
			const unsigned int need = (unsigned int)s * (unsigned int)box_items[w.x];
			volatile unsigned int* vdone = done + w.x;
			volatile unsigned int* verr = &sync->error;
			long long polls = 0;
			int go = 1;
			while (*vdone < need) {
				if (*verr != 0u) {
					go = 0;
					break;
				}
				if (polls >= wait_limit) {
					run_timeout(sync, boxes, nboxes);
					go = 0;
					break;
				}
				polls++;
				__nanosleep(100);
			}
			__threadfence();
			s_go = go;
			sp = boxes[w.x];
			sp.phase = int((step0 + s) % 3);
			sp.barrier_polls = int(min(wait_limit, (long long)BARRIER_POLLS));
		}
		__syncthreads();
		if (not s_go) return;
		double smax[3] = {0.0, 0.0, 0.0};
		bool zero = false, open = false;
		if (w.w == 0) {
			const bool first = w.y == 0 and w.z == 0;
			const double dt = begin_step(sp, &s_dt, first, &s_stop);
			const int tiles_x = (sp.L.n[0] + sp.tw - 1) / sp.tw;
			if (s_stop) {
				tile_hold<true>(sp, w.y % tiles_x, w.y / tiles_x, w.z);
			} else {
				tile_step<SOLVER, TY, ZACT, true>(sp, smem, bar, dt, w.y % tiles_x, w.y / tiles_x, w.z, smax[0], smax[1],
				                            smax[2], zero, open);
			}
		} else if (not stopped_before(sp)) {
			// ghost-ghost faces: combination w.y, faces [w.z BOUNDARY_CHUNK, (w.z + 1) BOUNDARY_CHUNK)
			int combos[12][3];
			const int nc = boundary_combos(sp, combos);
			if (w.y < nc) {
				const int d = combos[w.y][0], side = combos[w.y][1], e = combos[w.y][2];
				const long long count = boundary_count(sp, d, e);
				const long long t1 = min(count, (long long)(w.z + 1) * BOUNDARY_CHUNK);
				for (long long t = (long long)w.z * BOUNDARY_CHUNK + tid; t < t1; t += nthreads) {
					boundary_face<SOLVER, true>(sp, d, side, e, t, smax, zero);
				}
			}
		}
		if (flush_speeds(sp, smax, zero, open)) {
			const int tiles_x = (sp.L.n[0] + sp.tw - 1) / sp.tw;
			settle_tile(sp, w.y % tiles_x, w.y / tiles_x, w.z);
		}
		// publish the item's writes (every thread's), then count it done
		__threadfence();
		__syncthreads();
		if (tid == 0) atomicAdd(done + w.x, 1u);
	}
}

// ------------------------------------------------------------------ a 1-D grid's steps in one launch

/*
nsteps steps of a small 1-D grid in one launch of one thread-block cluster:
a thread per cell, its state in registers from the first step to the last.
A step is bound by latency (one face's solve, some 2 us with the barrier),
where a launch per step spends most of its time starting up, reading the
state and the last step's speeds back and draining: 1000 cells HLLD took
7.1 us per step as graph-replayed launches and take 3.0 us here.

Per step every thread derives its cell's record into shared memory (two
buffers alternate), the tile's end cells also into the neighbouring block's
halo (distributed shared memory), and one cluster barrier makes them, and
the blocks' speed maxima of the step before, visible; then a thread solves
its cell's -x face (one thread more the last +x face) and, after a block
barrier, updates its cell.  The arithmetic is the step kernel's, bit for
bit.  A step after a failing one is not taken (see stopped_before).
*/
template <int SOLVER> struct Line { static constexpr int THREADS = SOLVER == PAMHD_ROE_ATHENA ? 256 : 512; };
constexpr int LINE_REC = 11;   // rho, mom xyz, E, B xyz, 1/rho, total pressure, cf x
constexpr int LINE_BLOCKS = 8;

struct Line_Slot {
	double smax;
	int zero;
	int fail;
};

static size_t line_bytes(const int threads)
{
	return (size_t(2 * LINE_REC) * (threads + 2) + size_t(8) * (threads + 1)) * sizeof(double) + size_t(2) * (threads + 2);
}

template <int SOLVER>
__global__ void __launch_bounds__(Line<SOLVER>::THREADS) line_run_kernel(const Step_Params P, double* const other,
                                                                        const int nsteps, const int cells)
{
	namespace cg = cooperative_groups;
	extern __shared__ __align__(16) double smem[];
	__shared__ Line_Slot slots[2][LINE_BLOCKS];
	__shared__ double warp_speed[Line<SOLVER>::THREADS / 32];
	__shared__ int warp_zero[Line<SOLVER>::THREADS / 32];
	__shared__ int block_fail;
	const cg::cluster_group cluster = cg::this_cluster();
	const int rank = cluster.block_rank(), blocks = cluster.num_blocks(), T = blockDim.x, t = threadIdx.x;
	const int n = P.L.n[0], C = T + 2;
	const int mine = min(cells, n - rank * cells), last_mine = n - (blocks - 1) * cells;
	const int i = rank * cells + t;
	const bool own = t < mine;
	double* const flux = smem + 2 * LINE_REC * C;
	uint8_t* const bad = reinterpret_cast<uint8_t*>(flux + 8 * (T + 1));

	// a record at position pos of buffer b in block `to`
	const auto put = [&](const int to, const int b, const int pos, const double U[8], const Derived& d) {
		double* const r = cluster.map_shared_rank(smem, to) + b * LINE_REC * C + pos;
		#pragma unroll
		for (int v = 0; v < 8; v++) r[v * C] = U[v];
		r[8 * C] = d.rinv;
		r[9 * C] = d.pt;
		r[10 * C] = d.cf[0];
		cluster.map_shared_rank(bad, to)[b * C + pos] = uint8_t(d.bad);
	};
	const auto side = [&](const int b, const int pos) {
		const double* const r = smem + b * LINE_REC * C + pos;
		Side s;
		s.rho = r[0];
		s.m0 = r[C]; s.m1 = r[2 * C]; s.m2 = r[3 * C];
		s.E = r[4 * C];
		s.b0 = r[5 * C]; s.b1 = r[6 * C]; s.b2 = r[7 * C];
		s.rinv = r[8 * C];
		s.pt = r[9 * C];
		s.p = 0.0;  // not read without a background field
		s.cf = r[10 * C];
		s.v0 = s.m0 * s.rinv;
		s.v1 = s.m1 * s.rinv;
		s.v2 = s.m2 * s.rinv;
		s.bad = bad[b * C + pos];
		return s;
	};
	const auto load = [&](const int cell, double U[8]) {
		const long long off = P.L.offset(cell, 0, 0);
		#pragma unroll
		for (int v = 0; v < 8; v++) U[v] = P.in[v * P.L.var + off];
	};

	// a wave speed that round-off decides
	const auto settle = [&](Derived& d, const double U[8]) {
		if (d.bad == OPEN_WAVE) {
			d.bad = reference_wave(U[0], U[1], U[2], U[3], U[4], U[5], U[6], U[7], P.gas) ? 0u : (uint32_t)PAMHD_FLAG_WAVE_SPEED;
		}
	};

	double U[8] = {};
	if (own) load(i, U);
	// constant ghosts
	if (t == 0) {
		double G[8];
		if (rank == 0 and not P.periodic[0] and P.bc_lo[0] == PAMHD_BC_VALUE) {
			load(-1, G);
			Derived d = derive<true, false, false, true>(G[0], G[1], G[2], G[3], G[4], G[5], G[6], G[7], P.gas);
			settle(d, G);
			put(rank, 0, 0, G, d);
			put(rank, 1, 0, G, d);
		}
		if (rank == blocks - 1 and not P.periodic[0] and P.bc_hi[0] == PAMHD_BC_VALUE) {
			load(n, G);
			Derived d = derive<true, false, false, true>(G[0], G[1], G[2], G[3], G[4], G[5], G[6], G[7], P.gas);
			settle(d, G);
			put(rank, 0, mine + 1, G, d);
			put(rank, 1, mine + 1, G, d);
		}
		block_fail = 0;
	}
	double time = P.clock[P.phase].t, dt = P.clock[P.phase].dt;
	long long steps = P.clock[P.phase].steps;
	const double max_dt = P.control->max_dt, t_end = P.control->t_end;
	double smax = __longlong_as_double((long long)P.red[P.phase].smax[0]);
	bool zero = P.red[P.phase].zero != 0u, stop = stopped_before(P);
	cluster.sync();   // every block runs; its flags are set

	int s = 0;
	for (; s < nsteps; s++) {
		const int b = s & 1;
		if (own) {
			Derived d = derive<true, false, false, true>(U[0], U[1], U[2], U[3], U[4], U[5], U[6], U[7], P.gas);
			settle(d, U);
			put(rank, b, t + 1, U, d);
			if (t == 0) {
				if (rank > 0) put(rank - 1, b, cells + 1, U, d);
				else if (P.periodic[0]) put(blocks - 1, b, last_mine + 1, U, d);
				else if (P.bc_lo[0] == PAMHD_BC_COPY) put(rank, b, 0, U, d);
			}
			if (t == mine - 1) {
				if (rank < blocks - 1) put(rank + 1, b, 0, U, d);
				else if (P.periodic[0]) put(0, b, 0, U, d);
				else if (P.bc_hi[0] == PAMHD_BC_COPY) put(rank, b, mine + 1, U, d);
			}
		}
		cluster.sync();
		if (s > 0) {
			smax = 0.0;
			zero = stop = false;
			for (int r = 0; r < blocks; r++) {
				const Line_Slot& o = slots[b][r];
				smax = larger(o.smax, smax);
				zero = zero or o.zero != 0;
				stop = stop or o.fail != 0;
			}
		}
		if (stop) break;   // the same in every thread of the cluster
		// the step's dt (step_dt with one active dimension)
		double smallest = 0.0;
		if (not zero and smax > 0.0) smallest = fmin(1.7976931348623157e308, (P.cfl * P.len[0]) / smax);
		const double cap = max_dt >= 0.0 ? max_dt : t_end - time;
		dt = cap <= smallest ? cap : smallest;
		const double cx = dt * P.inv_len[0];

		double speed = 0.0;
		bool no = false;
		if (t <= mine) {
			const Side L = side(b, t), R = side(b, t + 1);
			double F[8];
			uint32_t flag = 0;
			const auto pick = [&](const bool left) { return side(b, left ? t : t + 1); };
			speed = solve_face<SOLVER>(L, R, P.gas, F, flag, pick);
			no = no_speed(speed);
			if (flag != 0) {
				block_fail = 1;
				int c = i - 1;
				if (P.periodic[0] and c < 0) c += n;
				atomicOr(&P.status->flags, flag);
				atomicMin(&P.status->first, (((unsigned long long)(c + P.ext[0]) * 4ull + 1ull) << 8) | flag);
				P.status->fail_step = (unsigned int)(steps + 1);
			}
			#pragma unroll
			for (int v = 0; v < 8; v++) {
				if (v != 5 or SOLVER == PAMHD_RUSANOV) flux[v * (T + 1) + t] = F[v];
			}
		}
		speed = warp_max(larger(speed, 0.0));
		no = __any_sync(0xffffffffu, no);
		if ((t & 31) == 0) {
			warp_speed[t >> 5] = speed;
			warp_zero[t >> 5] = no ? 1 : 0;
		}
		__syncthreads();
		if (own) {
			#pragma unroll
			for (int v = 0; v < 8; v++) {
				if (v != 5 or SOLVER == PAMHD_RUSANOV) {
					const double* const f = flux + v * (T + 1) + t;
					U[v] = __fma_rn(__dsub_rn(f[0], f[1]), cx, U[v]);
				}
			}
		}
		if (t < blocks) {
			Line_Slot o{0.0, 0, block_fail};
			for (int w = 0; w < (T + 31) / 32; w++) {
				o.smax = larger(warp_speed[w], o.smax);
				o.zero |= warp_zero[w];
			}
			cluster.map_shared_rank(&slots[b ^ 1][rank], t)[0] = o;
		}
		if (rank == 0 and t == 0 and P.dt_hist != nullptr) P.dt_hist[steps % P.hist_len] = dt;
		time += dt;
		steps++;
	}
	cluster.sync();   // the last step's maxima; no block leaves while another writes to it
	if (rank == 0 and t == 0) {
		if (s > 0 and s == nsteps) {
			smax = 0.0;
			zero = false;
			for (int r = 0; r < blocks; r++) {
				smax = larger(slots[s & 1][r].smax, smax);
				zero = zero or slots[s & 1][r].zero != 0;
			}
		}
		const int end = (P.phase + nsteps) % 3;
		Clock& c = P.clock[end];
		c.t = time;
		c.dt = s < nsteps ? 0.0 : dt;   // held steps have none
		c.steps = steps;
		Speed_Max& r = P.red[end];
		r.smax[0] = smax > 0.0 ? (unsigned long long)__double_as_longlong(smax) : 0ull;
		r.smax[1] = r.smax[2] = 0ull;
		r.zero = zero ? 1u : 0u;
		Speed_Max& next = P.red[(end + 1) % 3];
		next.smax[0] = next.smax[1] = next.smax[2] = 0ull;
		next.zero = 0u;
	}
	if (own) {
		// a grid that stopped holds the failing step's result in both state buffers
		for (int k = 0; k < (s < nsteps ? 2 : 1); k++) {
			double* const out = k == 0 ? P.out : other;
			store_cell(out, P.L, i, 0, 0, U);
			if (i == 0) {
				if (P.periodic[0]) store_cell(out, P.L, n, 0, 0, U);
				else if (P.bc_lo[0] == PAMHD_BC_COPY) store_cell(out, P.L, -1, 0, 0, U);
			}
			if (i == n - 1) {
				if (P.periodic[0]) store_cell(out, P.L, -1, 0, 0, U);
				else if (P.bc_hi[0] == PAMHD_BC_COPY) store_cell(out, P.L, n, 0, 0, U);
			}
		}
	}
}

// ------------------------------------------------------------------ solver-level entry

__device__ __forceinline__ Side face_side(const double* s, const double* bg, const bool use_bg, const Gas& g)
{
	Side out;
	out.rho = s[0]; out.m0 = s[1]; out.m1 = s[2]; out.m2 = s[3]; out.E = s[4];
	out.b0 = s[5]; out.b1 = s[6]; out.b2 = s[7];
	const Derived d = derive<true, false, false>(s[0], s[1], s[2], s[3], s[4], s[5], s[6], s[7], g);
	out.rinv = d.rinv;
	out.v0 = d.vx; out.v1 = d.vy; out.v2 = d.vz;
	out.p = d.p;
	out.pt = d.pt;
	out.cf = d.cf[0];
	out.bad = d.bad;
	if (use_bg) {
		// fast speed with the total field (get_fast_magnetosonic_speed, mhd/common.hpp:433-490)
		const double t0 = s[5] + bg[0], t1 = s[6] + bg[1], t2 = s[7] + bg[2];
		const double t2s = t0 * t0 + t1 * t1 + t2 * t2;
		const double cs2 = g.gamma * d.p * d.rinv;
		if (t2s > 0.0) {
			const double va2 = t2s * g.inv_mu0 * d.rinv;
			const double sum2 = cs2 + va2;
			const double to_sqrt = cs2 * cs2 + va2 * va2 + 2.0 * cs2 * va2 * (1.0 - 2.0 * (t0 * t0 / t2s));
			if (out.bad == 0 and not (is_normal(sum2) and to_sqrt > 0.0 and is_normal(to_sqrt))) {
				out.bad = PAMHD_FLAG_WAVE_SPEED;
			}
			out.cf = sqrt(0.5 * (sum2 + sqrt(fmax(to_sqrt, 0.0))));
		} else {
			out.cf = sqrt(fmax(cs2, 0.0));
		}
	}
	return out;
}

template <int SOLVER>
__global__ void face_flux_kernel(long long n, const double* __restrict__ neg, const double* __restrict__ pos,
                                 const double* __restrict__ bg, const Gas g, double* __restrict__ flux,
                                 double* __restrict__ speed, uint32_t* __restrict__ flags)
{
	for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
		const bool use_bg = bg != nullptr and (SOLVER == PAMHD_RUSANOV or SOLVER == PAMHD_HLL_ATHENA);
		const double zero3[3] = {0.0, 0.0, 0.0};
		const double* b = use_bg ? bg + 3 * t : zero3;
		const Side L = face_side(neg + 8 * t, b, use_bg, g);
		const Side R = face_side(pos + 8 * t, b, use_bg, g);
		double F[8];
		uint32_t flag = L.bad | R.bad;
		if (flag & PAMHD_FLAG_DENSITY) flag = PAMHD_FLAG_DENSITY;
		else if (flag & PAMHD_FLAG_PRESSURE) flag = PAMHD_FLAG_PRESSURE;
		double s;
		if (SOLVER == PAMHD_RUSANOV) s = use_bg ? flux_rusanov<true>(L, R, g, F, flag, b) : flux_rusanov<false>(L, R, g, F, flag);
		else if (SOLVER == PAMHD_HLL_ATHENA) s = use_bg ? flux_hll<true>(L, R, g, F, flag, b) : flux_hll<false>(L, R, g, F, flag);
		else if (SOLVER == PAMHD_HLLD_ATHENA) s = flux_hlld(L, R, g, F, Held_Sides{L, R});
		else s = flux_roe(L, R, g, F, flag);
		for (int v = 0; v < 8; v++) flux[8 * t + v] = flag ? 0.0 : F[v];
		speed[t] = flag ? 0.0 : s;
		flags[t] = flag;
	}
}

// ------------------------------------------------------------------ conserved totals

/*
Per-block partial sums of the eight conserved variables over interior
cells (compensated summation inside a thread, a fixed-order tree across
the block), so that totals are deterministic run to run.
*/
__global__ void totals_kernel(const double* __restrict__ state, const Layout L, double* __restrict__ partial)
{
	__shared__ double red[8][256];
	const long long n = (long long)L.n[0] * L.n[1] * L.n[2];
	const long long per = (n + gridDim.x - 1) / gridDim.x;
	const long long a = blockIdx.x * per, b = min(n, a + per);
	double sum[8], comp[8];
	for (int v = 0; v < 8; v++) sum[v] = comp[v] = 0.0;
	for (long long t = a + threadIdx.x; t < b; t += blockDim.x) {
		const int i = int(t % L.n[0]);
		const int j = int((t / L.n[0]) % L.n[1]);
		const int k = int(t / ((long long)L.n[0] * L.n[1]));
		const long long o = L.offset(i, j, k);
		for (int v = 0; v < 8; v++) {
			const double y = state[v * L.var + o] - comp[v];
			const double s = sum[v] + y;
			comp[v] = (s - sum[v]) - y;
			sum[v] = s;
		}
	}
	for (int v = 0; v < 8; v++) red[v][threadIdx.x] = sum[v];
	__syncthreads();
	for (int w = blockDim.x / 2; w > 0; w >>= 1) {
		if ((int)threadIdx.x < w) {
			for (int v = 0; v < 8; v++) red[v][threadIdx.x] += red[v][threadIdx.x + w];
		}
		__syncthreads();
	}
	if (threadIdx.x == 0) {
		for (int v = 0; v < 8; v++) partial[8 * blockIdx.x + v] = red[v][0];
	}
}

// ------------------------------------------------------------------ launchers

/*
Calls body(solver, rows, zact) with the values of kind as integral
constants: the solver, the tile rows (1 where y is inactive) and whether
there are z faces (only with y active).
*/
template <int N> using Const = std::integral_constant<int, N>;

template <int SOLVER, class Body> static int with_rows(const Tile_Kind& kind, const Body& body)
{
	if (kind.rows == 1 and not kind.zact) return body(Const<SOLVER>{}, Const<1>{}, std::false_type{});
	if (kind.rows == TY_3D) {
		return kind.zact ? body(Const<SOLVER>{}, Const<TY_3D>{}, std::true_type{})
		                 : body(Const<SOLVER>{}, Const<TY_3D>{}, std::false_type{});
	}
	if (kind.rows == TY_WIDE) {
		return kind.zact ? body(Const<SOLVER>{}, Const<TY_WIDE>{}, std::true_type{})
		                 : body(Const<SOLVER>{}, Const<TY_WIDE>{}, std::false_type{});
	}
	return PAMHD_ERR_ARGUMENT;
}

template <class Body> static int with_kind(const Tile_Kind& kind, const Body& body)
{
	switch (kind.solver) {
	case PAMHD_RUSANOV: return with_rows<PAMHD_RUSANOV>(kind, body);
	case PAMHD_HLL_ATHENA: return with_rows<PAMHD_HLL_ATHENA>(kind, body);
	case PAMHD_HLLD_ATHENA: return with_rows<PAMHD_HLLD_ATHENA>(kind, body);
	case PAMHD_ROE_ATHENA: return with_rows<PAMHD_ROE_ATHENA>(kind, body);
	default: return PAMHD_ERR_ARGUMENT;
	}
}

static int status_of(const cudaError_t e)
{
	return e == cudaSuccess ? PAMHD_OK : PAMHD_ERR_CUDA;
}

/*
The single-grid step's tile (its size; tile_shape() lays it out).  3-D
grids: 32 x 8, two blocks of 256 threads
per SM (a taller tile solves fewer halo faces and records per cell).  2-D
grids: 32 x 4, four blocks of 128 threads per SM: the same 16 warps in
blocks that wait for fewer others, and twice the blocks on small grids
(HLLD against 32 x 8 tiles: 257 x 180 cells 10.1 us per step, was 11.2;
512^2 33.8, was 34.4; 1024^2 118, was 128), but for grids with more rows than
a launch has 32 x 4 tiles for.  Roe's solver needs more
registers than either leaves, so it keeps 32 x 4 tiles at three blocks per
SM (at four, 512^2 took 72 us instead of 66).
*/
Tile_Kind step_tile(const int solver, const int ny, const bool zact)
{
	const bool small = solver == PAMHD_ROE_ATHENA or (not zact and ny <= TY_3D * MAX_TILE_ROWS);
	return Tile_Kind{solver, ny <= 1 ? 1 : (small ? TY_3D : TY_WIDE), zact};
}

int prepare_step_kernels(const Tile_Kind& kind)
{
	return with_kind(kind, [](auto solver, auto rows, auto zact) {
		const auto kernel = step_kernel<solver(), rows(), zact()>;
		cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
		                                     int(tile_bytes<solver(), rows(), zact()>()));
		// all of the SM's memory as shared memory, so that the blocks the registers allow fit
		if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
		return status_of(e);
	});
}

int launch_step(const Step_Params& P, const int solver, cudaStream_t stream)
{
	const int nz = P.L.n[2];
	const int chunks = P.kpart == 1 ? (nz > 1 ? 2 : 1)
	                 : P.kpart == 2 ? (nz - 2 + P.kchunk - 1) / P.kchunk
	                 : (nz + P.kchunk - 1) / P.kchunk;
	if (chunks < 1) return PAMHD_OK;  // no planes between the first and the last
	return with_kind(step_tile(solver, P.L.n[1], P.active[2] != 0), [&](auto solver_, auto rows, auto zact) {
		const dim3 grid((P.L.n[0] + P.tw - 1) / P.tw, (P.L.n[1] + P.th - 1) / P.th, chunks + P.boundary);
		step_kernel<solver_(), rows(), zact()>
			<<<grid, TX * rows(), tile_bytes<solver_(), rows(), zact()>(), stream>>>(P);
		return status_of(cudaGetLastError());
	});
}

// calls body with the solver as an integral constant
template <class Body> static int with_solver(const int solver, const Body& body)
{
	switch (solver) {
	case PAMHD_RUSANOV: return body(Const<PAMHD_RUSANOV>{});
	case PAMHD_HLL_ATHENA: return body(Const<PAMHD_HLL_ATHENA>{});
	case PAMHD_HLLD_ATHENA: return body(Const<PAMHD_HLLD_ATHENA>{});
	case PAMHD_ROE_ATHENA: return body(Const<PAMHD_ROE_ATHENA>{});
	default: return PAMHD_ERR_ARGUMENT;
	}
}

/*
Whether a grid's steps run as line_run_kernel: 1-D, cells enough for one per
thread of eight blocks (a thread more per block for the last face), and no
side whose state changes with time.
*/
bool line_run_fits(const Step_Params& P, const int solver)
{
	const int most = LINE_BLOCKS * ((solver == PAMHD_ROE_ATHENA ? 256 : 512) - 1);
	return P.active[0] and not P.active[1] and not P.active[2] and P.L.n[0] <= most and P.inflow == nullptr
		and P.forced_dt < 0.0;
}

int prepare_line_run(const int solver)
{
	return with_solver(solver, [](auto s) {
		return status_of(cudaFuncSetAttribute(line_run_kernel<s()>, cudaFuncAttributeMaxDynamicSharedMemorySize,
		                                      int(line_bytes(Line<s()>::THREADS))));
	});
}

int launch_line_run(const Step_Params& P, double* other, const int nsteps, const int solver, cudaStream_t stream)
{
	// 1, 2, 4 or 8 blocks of up to 127 cells (four warps, one per scheduler), then 8 larger ones
	const int n = P.L.n[0];
	int blocks = 1;
	while (blocks < LINE_BLOCKS and n > 127 * blocks) blocks *= 2;
	const int cells = (n + blocks - 1) / blocks;
	return with_solver(solver, [&](auto s) {
		cudaLaunchConfig_t c = {};
		c.gridDim = dim3(blocks);
		c.blockDim = dim3((cells + 1 + 31) / 32 * 32);
		c.dynamicSmemBytes = line_bytes(int(c.blockDim.x));
		c.stream = stream;
		cudaLaunchAttribute a[1];
		a[0].id = cudaLaunchAttributeClusterDimension;
		a[0].val.clusterDim.x = c.gridDim.x;
		a[0].val.clusterDim.y = 1;
		a[0].val.clusterDim.z = 1;
		c.attrs = a;
		c.numAttrs = 1;
		return status_of(cudaLaunchKernelEx(&c, line_run_kernel<s()>, P, other, nsteps, cells));
	});
}

int prepare_batch_kernels(const Tile_Kind& kind)
{
	return with_kind(kind, [](auto solver, auto rows, auto zact) {
		return status_of(cudaFuncSetAttribute(batch_step_kernel<solver(), rows(), zact()>,
		                                      cudaFuncAttributeMaxDynamicSharedMemorySize,
		                                      int(tile_bytes<solver(), rows(), zact()>())));
	});
}

int batch_blocks_per_sm(const Tile_Kind& kind, int* blocks)
{
	return with_kind(kind, [&](auto solver, auto rows, auto zact) {
		return status_of(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
			blocks, batch_step_kernel<solver(), rows(), zact()>, TX * rows(),
			tile_bytes<solver(), rows(), zact()>()));
	});
}

int prepare_batch_run_kernels(const Tile_Kind& kind)
{
	return with_kind(kind, [](auto solver, auto rows, auto zact) {
		return status_of(cudaFuncSetAttribute(batch_run_kernel<solver(), rows(), zact()>,
		                                      cudaFuncAttributeMaxDynamicSharedMemorySize,
		                                      int(tile_bytes<solver(), rows(), zact()>())));
	});
}

int batch_run_blocks_per_sm(const Tile_Kind& kind, int* blocks)
{
	return with_kind(kind, [&](auto solver, auto rows, auto zact) {
		return status_of(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
			blocks, batch_run_kernel<solver(), rows(), zact()>, TX * rows(),
			tile_bytes<solver(), rows(), zact()>()));
	});
}

int launch_batch_run(const Step_Params* even, const Step_Params* odd, const int4* items, const int nitems,
                     const int* box_items, unsigned int* done, const int nboxes, const long long step0,
                     const int nsteps, Run_Sync* sync, const long long wait_limit, const int grid,
                     const Tile_Kind& kind, cudaStream_t stream)
{
	return with_kind(kind, [&](auto solver, auto rows, auto zact) {
		cudaLaunchConfig_t c = {};
		c.gridDim = dim3(grid);
		c.blockDim = TX * rows();
		c.dynamicSmemBytes = tile_bytes<solver(), rows(), zact()>();
		c.stream = stream;
		cudaLaunchAttribute a[1];
		a[0].id = cudaLaunchAttributeCooperative;
		a[0].val.cooperative = 1;
		c.attrs = a;
		c.numAttrs = 1;
		return status_of(cudaLaunchKernelEx(&c, batch_run_kernel<solver(), rows(), zact()>,
		                                    even, odd, items, nitems, box_items, done, nboxes, step0, nsteps, sync,
		                                    wait_limit));
	});
}

int launch_batch_step(const Step_Params* boxes, const int4* items, const int nitems, const int phase,
                      const int barrier_polls, const int grid, const Tile_Kind& kind, cudaStream_t stream)
{
	return with_kind(kind, [&](auto solver, auto rows, auto zact) {
		batch_step_kernel<solver(), rows(), zact()>
			<<<grid, TX * rows(), tile_bytes<solver(), rows(), zact()>(), stream>>>(boxes, items, nitems, phase, barrier_polls);
		return status_of(cudaGetLastError());
	});
}

int launch_batch_boundary_speeds(const Step_Params* boxes, const int nboxes, const int largest, const int phase,
                                 const int solver, cudaStream_t stream)
{
	const dim3 grid(min(1024, (largest + 255) / 256), nboxes);
	switch (solver) {
	case PAMHD_RUSANOV: batch_boundary_speed_kernel<PAMHD_RUSANOV><<<grid, 256, 0, stream>>>(boxes, phase); break;
	case PAMHD_HLL_ATHENA: batch_boundary_speed_kernel<PAMHD_HLL_ATHENA><<<grid, 256, 0, stream>>>(boxes, phase); break;
	case PAMHD_HLLD_ATHENA: batch_boundary_speed_kernel<PAMHD_HLLD_ATHENA><<<grid, 256, 0, stream>>>(boxes, phase); break;
	case PAMHD_ROE_ATHENA: batch_boundary_speed_kernel<PAMHD_ROE_ATHENA><<<grid, 256, 0, stream>>>(boxes, phase); break;
	default: return PAMHD_ERR_ARGUMENT;
	}
	return cudaGetLastError() == cudaSuccess ? PAMHD_OK : PAMHD_ERR_CUDA;
}

int boundary_layers(const Step_Params& P, const int solver)
{
	long long faces = 0;
	for (int d = 0; d < 3; d++) {
		if (not P.active[d] or P.periodic[d]) continue;
		for (int e = 0; e < 3; e++) {
			if (e != d and P.active[e]) faces += 2LL * P.L.n[e] * P.L.n[3 - d - e];
		}
	}
	// about a face per thread
	const int rows = step_tile(solver, P.L.n[1], P.active[2] != 0).rows;
	const long long layer = (long long)((P.L.n[0] + P.tw - 1) / P.tw) * ((P.L.n[1] + P.th - 1) / P.th) * TX * rows;
	return int(min(1024LL, (faces + layer - 1) / layer));
}

int launch_scatter(const double* packed, double* var_base, const Layout& L, cudaStream_t stream)
{
	scatter_kernel<<<1184, 256, 0, stream>>>(packed, var_base, L);
	return cudaGetLastError() == cudaSuccess ? PAMHD_OK : PAMHD_ERR_CUDA;
}

int launch_gather(const double* var_base, double* packed, const Layout& L, cudaStream_t stream)
{
	gather_kernel<<<1184, 256, 0, stream>>>(var_base, packed, L);
	return cudaGetLastError() == cudaSuccess ? PAMHD_OK : PAMHD_ERR_CUDA;
}

int launch_fill_ghosts_values(const Step_Params& P, double* state, const double lo[3][8], const double hi[3][8],
                              cudaStream_t stream)
{
	Ghost_Values V;
	for (int d = 0; d < 3; d++) {
		for (int v = 0; v < 8; v++) {
			V.lo[d][v] = lo[d][v];
			V.hi[d][v] = hi[d][v];
		}
	}
	fill_ghosts_kernel<<<296, 256, 0, stream>>>(P, state, V);
	return cudaGetLastError() == cudaSuccess ? PAMHD_OK : PAMHD_ERR_CUDA;
}

int launch_face_flux(const int solver, const long long n, const double* neg, const double* pos, const double* bg,
                     const Gas& gas, double* flux, double* speed, uint32_t* flags, cudaStream_t stream)
{
	const int blocks = int(min(4096LL, (n + 127) / 128));
	if (blocks == 0) return PAMHD_OK;
	switch (solver) {
	case PAMHD_RUSANOV: face_flux_kernel<PAMHD_RUSANOV><<<blocks, 128, 0, stream>>>(n, neg, pos, bg, gas, flux, speed, flags); break;
	case PAMHD_HLL_ATHENA: face_flux_kernel<PAMHD_HLL_ATHENA><<<blocks, 128, 0, stream>>>(n, neg, pos, bg, gas, flux, speed, flags); break;
	case PAMHD_HLLD_ATHENA: face_flux_kernel<PAMHD_HLLD_ATHENA><<<blocks, 128, 0, stream>>>(n, neg, pos, bg, gas, flux, speed, flags); break;
	case PAMHD_ROE_ATHENA: face_flux_kernel<PAMHD_ROE_ATHENA><<<blocks, 128, 0, stream>>>(n, neg, pos, bg, gas, flux, speed, flags); break;
	default: return PAMHD_ERR_ARGUMENT;
	}
	return cudaGetLastError() == cudaSuccess ? PAMHD_OK : PAMHD_ERR_CUDA;
}

int launch_totals(const double* state, const Layout& L, const double /*volume*/, double* partial, const int nblocks,
                  cudaStream_t stream)
{
	totals_kernel<<<nblocks, 256, 0, stream>>>(state, L, partial);
	return cudaGetLastError() == cudaSuccess ? PAMHD_OK : PAMHD_ERR_CUDA;
}

} // namespace pamhd_b200
