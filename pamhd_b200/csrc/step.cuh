/*
Device-side data structures of the fused MHD step, shared by the kernels
(step_kernels.cu) and the host context (context.cu).
*/
#ifndef PAMHD_B200_STEP_CUH
#define PAMHD_B200_STEP_CUH

#include <cstdint>

#include "mhd_device.cuh"

namespace pamhd_b200 {

/*
Layout of one state copy in HBM: eight FP64 arrays (rho, mom xyz, E,
B xyz), each a padded 3-D block with one ghost layer on every active
dimension.  Rows are padded so that the first interior cell of every row
sits on a 32-byte boundary (a full DRAM sector); periodic dimensions have
ghosts too, refreshed by the step kernel itself.
*/
struct Layout {
	int n[3];        // interior cells
	int g[3];        // ghost width (1 on active dimensions, else 0)
	int xoff;        // column of interior x = 0
	int pitch;       // doubles per row
	int rows;        // rows per plane: n[1] + 2 g[1]
	int planes;      // n[2] + 2 g[2]
	long long plane; // doubles per plane
	long long var;   // doubles per variable array

	__host__ __device__ long long offset(const int i, const int j, const int k) const
	{
		return (long long)(k + g[2]) * plane + (long long)(j + g[1]) * pitch + (i + xoff);
	}
};

// per-step reduction of face signal speeds (bit patterns of non-negative doubles)
struct Speed_Max {
	unsigned long long smax[3];
	unsigned int zero;   // some face had speed <= 0 (or no reduction yet)
	unsigned int pad;
};

// simulation clock, one slot per step phase
struct Clock {
	double t;
	double dt;
	long long steps;
	double pad;
};

// error state: OR of flags and the first failing face ((key << 8) | flag)
struct Status {
	unsigned int flags;
	unsigned int fail_step;        // the cell-centred steps: 1 + the clock's step count of the failing step (0: none)
	unsigned long long first;
};

// what a call returns for it
inline int status_code(const Status& s)
{
	if (s.flags & PAMHD_FLAG_TIMEOUT) return PAMHD_ERR_TIMEOUT;
	return s.flags != 0 ? PAMHD_ERR_PHYSICS : PAMHD_OK;
}

// limits read by the step kernel from device memory (so graphs need no re-capture)
struct Control {
	double max_dt;   // >= 0: cap of dt; < 0: cap is t_end - t
	double t_end;
};

/*
Time-stamped inflow of a VALUE side (the solar-wind boundary of
mhd/solar_wind_box.hpp:227-268): states[i] (8 conservative values) holds
while i of the count timestamps are <= the simulation time.  Device
memory; states == nullptr: the side keeps its constant ghost values.
*/
struct Inflow_Table {
	const double* times;
	const double* states;   // (count + 1) x 8
	int count;
};

/*
Scheduler state of the persistent batched run: the next (step, work item)
to hand out, and an error word set by a block whose bounded wait ran out.
*/
struct Run_Sync {
	unsigned int next;
	unsigned int error;
	unsigned int pad[2];
};

struct Step_Params {
	const double* __restrict__ in;
	double* __restrict__ out;
	Layout L;
	Gas gas;
	double len[3];
	double inv_len[3];
	double cfl;
	int active[3];
	int periodic[3];
	int bc_lo[3];
	int bc_hi[3];
	int ext[3];          // ghost extent of the failure numbering (1 on non-periodic active dims)
	Speed_Max* red;      // [3], ring by step phase
	Clock* clock;        // [3]
	Status* status;
	const Control* control;
	double* dt_hist;
	int hist_len;
	int phase;           // step index mod 3
	int tw, th;          // columns of a tile along x and y
	int kchunk;          // z planes per block
	double forced_dt;    // >= 0: the step's dt (a prescribed schedule); < 0: the CFL rule
	int kpart;           // z planes a launch computes: 0 all, 1 the first and last only, 2 the others
	int boundary;        // block layers of the step's launch that solve ghost-ghost faces (0: none)
	int barrier_polls;   // polls a block's split barrier makes before it gives up
	const Inflow_Table* inflow;  // [3][2] by dimension and side (lo, hi) in device memory, or nullptr
};

// the kernel instance a grid or batch runs: solver, tile size (32 x rows threads; rows 1: y
// inactive), whether there are z faces
struct Tile_Kind {
	int solver;
	int rows;
	bool zact;
	// resident blocks per SM asked of the register allocator: 16 warps of at most 128 registers with
	// 32 x 8 tiles and with 32 x 4 tiles of one plane, 12 warps of at most 168 with 32 x 4 tiles that
	// march in z, with Roe's solver and with one-row tiles
	static constexpr int resident_of(const int solver, const int rows, const bool zact)
	{
		return rows == 8 ? 2 : (rows == 4 and not zact and solver != PAMHD_ROE_ATHENA ? 4 : 3);
	}
	int resident() const { return resident_of(solver, rows, zact); }
	// columns along x of a tile without z faces: 32, or 31 with one row, whose last thread then takes
	// the tile's +x face in the same pass
	static constexpr int flat_width_of(const int rows) { return rows == 1 ? 31 : 32; }
	// records of a plane of a tile and its halo, the most its shared memory holds: 32 x 8 columns need
	// 336, 22 x 11 308; 32 x 4 need 200, 42 x 3 216; 31 x 1 33
	static constexpr int records_of(const int rows) { return rows == 8 ? 352 : (rows == 4 ? 216 : 33); }
};

// launchers (step_kernels.cu)
int launch_step(const Step_Params& P, int solver, cudaStream_t stream);
// nsteps steps of a small 1-D grid in one launch; P.out: the buffer of the last step, other: the other
bool line_run_fits(const Step_Params& P, int solver);
int prepare_line_run(int solver);
int launch_line_run(const Step_Params& P, double* other, int nsteps, int solver, cudaStream_t stream);
// block layers for the ghost-ghost faces of a grid with non-periodic sides (Step_Params::boundary)
int boundary_layers(const Step_Params& P, int solver);
int launch_scatter(const double* packed, double* var_base, const Layout& L, cudaStream_t stream);
int launch_gather(const double* var_base, double* packed, const Layout& L, cudaStream_t stream);
int launch_fill_ghosts_values(const Step_Params& P, double* state, const double lo[3][8], const double hi[3][8],
                              cudaStream_t stream);
int prepare_step_kernels(const Tile_Kind& kind);
int launch_face_flux(int solver, long long n, const double* neg, const double* pos, const double* bg,
                     const Gas& gas, double* flux, double* speed, uint32_t* flags, cudaStream_t stream);
int launch_totals(const double* state, const Layout& L, double volume, double* partial, int nblocks,
                  cudaStream_t stream);
constexpr int MAX_TILE_ROWS = 65535;   // of a launch: tiles along y are its grid's y dimension
Tile_Kind step_tile(int solver, int ny, bool zact);
int batch_tile_rows();
int prepare_batch_kernels(const Tile_Kind& kind);
int batch_blocks_per_sm(const Tile_Kind& kind, int* blocks);
int launch_batch_step(const Step_Params* boxes, const int4* items, int nitems, int phase, int barrier_polls, int grid,
                      const Tile_Kind& kind, cudaStream_t stream);
int launch_batch_boundary_speeds(const Step_Params* boxes, int nboxes, int largest, int phase, int solver,
                                 cudaStream_t stream);
// the persistent batched run: nsteps steps of every box in one cooperative launch (see batch_run_kernel)
int prepare_batch_run_kernels(const Tile_Kind& kind);
int batch_run_blocks_per_sm(const Tile_Kind& kind, int* blocks);
int launch_batch_run(const Step_Params* boxes_even, const Step_Params* boxes_odd, const int4* items, int nitems,
                     const int* box_items, unsigned int* done, int nboxes, long long step0, int nsteps,
                     Run_Sync* sync, long long wait_limit, int grid, const Tile_Kind& kind,
                     cudaStream_t stream);
// polls of a block's split barrier where the caller set no limit (its warps all arrive: never reached)
constexpr int BARRIER_POLLS = 1 << 20;
constexpr int BOUNDARY_CHUNK = 4096;  // ghost-ghost faces per boundary work item of the persistent run

} // namespace pamhd_b200

#endif
