"""Parity of the CUDA path (through the C ABI) with the CPU oracle.

Tolerance: the GPU computes in FP64 with FMA contraction and reciprocals,
the oracle in the reference's exact operation order, so results agree to
round-off.  Per step the bar is a relative state error <= 1e-12: for every
variable, |gpu - oracle| <= 1e-12 * max(|oracle| over that variable's
field) per cell (a field-normwise relative error; momentum and field
components pass through zero, where a cellwise ratio is meaningless).
Face fluxes use the same bar per face: |gpu - oracle| <= 1e-12 * max over
the face's eight flux components.
"""
import numpy as np
import pytest

import pamhd_b200 as pg
from oracle import pyoracle as po
import states

pytestmark = pytest.mark.gpu

STEP_TOL = 1e-12


def field_err(a, b):
    """max over variables of max|a - b| / max|b| (b = oracle)."""
    a = a.reshape(8, -1)
    b = b.reshape(8, -1)
    scale = np.abs(b).max(axis=1)
    scale[scale == 0] = 1.0
    return float((np.abs(a - b).max(axis=1) / scale).max())


def pair(port, n, solver, lengths, gamma, mu0, cfl, bc_lo=(0, 0, 0), bc_hi=(0, 0, 0),
         value_lo=None, value_hi=None):
    cfg = pg.Config(n=n, solver=solver, cell_length=lengths, adiabatic_index=gamma, vacuum_permeability=mu0,
                    time_step_factor=cfl, bc_lo=bc_lo, bc_hi=bc_hi,
                    value_lo=value_lo or [None] * 3, value_hi=value_hi or [None] * 3)
    ocfg = po.make_cfg(n, solver, lengths, gamma, mu0, cfl, bc_lo, bc_hi, value_lo, value_hi)
    return pg.Context(cfg), port.grid(ocfg, threads=8)


# ---------------------------------------------------------------- solver level

@pytest.mark.parametrize("bc", ["periodic", "copy", "value"])
@pytest.mark.parametrize("solver", ["rusanov", "hll_athena", "hlld_athena", "roe_athena"])
@pytest.mark.parametrize("n", [2, 31, 127, 128, 255, 1000, 1017, 2040, 2041, 4088, 4089])
def test_line_run_equals_single_steps(n, solver, bc):
    """A 1-D grid's steps in one launch (up to 4088 cells, 2040 with Roe) against the same steps made
    one by one: state, every dt and the clock bit for bit, after an odd and an even number of steps;
    n at the edges of one, two, four and eight blocks and just past the largest."""
    kind = {"periodic": pg.BC_PERIODIC, "copy": pg.BC_COPY, "value": pg.BC_VALUE}[bc]
    U = states.smooth_3d((1, 1, n), np.random.default_rng(n))
    cfg = pg.Config(n=(n, 1, 1), solver=po.SOLVERS[solver], cell_length=(1.0 / n, 1.0, 1.0), time_step_factor=0.4,
                    bc_lo=(kind, 0, 0), bc_hi=(kind, 0, 0), value_lo=[U[:, 0, 0, 0], None, None],
                    value_hi=[U[:, 0, 0, -1], None, None])
    a, b = pg.Context(cfg), pg.Context(cfg)
    for g in (a, b):
        g.set_state(U)
    for count in (5, 8, 2):
        a.steps(count, 1e300)
        for _ in range(count):
            b.step(1e300)
        np.testing.assert_array_equal(a.get_state(), b.get_state())
        assert a.time() == b.time()
        np.testing.assert_array_equal(a.dt_history(20), b.dt_history(20))
    a.sync()


def test_line_run_stops_at_a_failure():
    """A 1-D run that loses positivity (a timestep factor of 3, far beyond stability): the one-launch
    steps stop at the step, cell and flag of the steps made one by one and hold that step's result,
    in both state buffers."""
    n = 300
    U = states.smooth_3d((1, 1, n), np.random.default_rng(1))
    cfg = pg.Config(n=(n, 1, 1), solver=pg.HLLD, cell_length=(1.0 / n, 1.0, 1.0), time_step_factor=3.0)
    a, b = pg.Context(cfg), pg.Context(cfg)
    for g in (a, b):
        g.set_state(U)
    failed = None
    for s in range(80):
        try:
            b.step(1e300)
        except pg.PhysicsError as e:
            failed = (e.flags, e.cell, e.direction)
            break
    assert failed is not None and s > 0
    held = b.get_state()
    for count in (s + 1, 3, 2):   # the failing step last, then held steps
        a.steps(count, 1e300)
        with pytest.raises(pg.PhysicsError) as e:
            a.sync()
        assert (e.value.flags, e.value.cell, e.value.direction) == failed
        np.testing.assert_array_equal(a.get_state(), held)
    assert a.time()[:2] == b.time()[:2]


@pytest.mark.parametrize("bc", ["periodic", "copy"])
@pytest.mark.parametrize("solver", list(po.SOLVERS))
@pytest.mark.parametrize("n", list(states.SHORT_GRIDS))
def test_short_z_chunks_match_oracle(port, n, solver, bc):
    """Small 3-D grids, whose blocks take a few planes each, in tiles of 32 x 8 and of other columns (the
    sizes and what they are for: states.SHORT_GRIDS; Roe's tiles, of half as many threads, are others);
    on open sides the step's own blocks solve the ghost-ghost faces.  Per step, the bar of this file."""
    kinds = ((pg.BC_COPY,) * 3 if bc == "copy" else (pg.BC_PERIODIC,) * 3,) * 2
    L = (0.1, 0.12, 0.09)
    U = states.smooth_3d((n[2], n[1], n[0]), np.random.default_rng(3))
    gpu, ora = pair(port, n, po.SOLVERS[solver], L, states.GAMMA_53, 1.0, 0.4, *kinds)
    gpu.set_state(U)
    ora.set_state(U)
    for s in range(4):
        dg = gpu.step(0.0 if s == 0 else 1.0)
        do, flag, _, _ = ora.step(0.0 if s == 0 else 1.0)
        assert flag == 0
        assert abs(dg - do) <= 1e-13 * max(do, 1e-300), s
        assert field_err(gpu.get_state(), ora.get_state()) <= STEP_TOL, s


@pytest.mark.parametrize("solver", list(po.SOLVERS))
def test_block_barrier_timeout_is_reported(solver):
    """A block barrier that gives up (a limit of 0 polls) ends in PAMHD_ERR_TIMEOUT and
    PAMHD_FLAG_TIMEOUT, in a single step and in replayed ones; later steps hold the grid and its clock;
    after set_state with the limit restored the grid steps as a new one."""
    n = (40, 21, 33)
    U = states.smooth_3d(n[::-1], np.random.default_rng(2))
    cfg = pg.Config(n=n, solver=po.SOLVERS[solver], cell_length=(0.1, 0.12, 0.09), time_step_factor=0.4)
    a, b = pg.Context(cfg), pg.Context(cfg)
    a.set_state(U)
    a.steps(13, 1e300)   # a captured graph holds the old limit
    a.sync()
    a.set_wait_limit(0)
    with pytest.raises(pg.PamhdError) as e:
        a.step(1.0)
    assert e.value.code == pg.ERR_TIMEOUT
    assert a.status()[0] & pg.FLAG_TIMEOUT
    held, clock = a.get_state(), a.time()[:2]
    a.steps(13, 1e300)
    with pytest.raises(pg.PamhdError) as e:
        a.sync()
    assert e.value.code == pg.ERR_TIMEOUT
    np.testing.assert_array_equal(a.get_state(), held)
    assert a.time()[:2] == clock
    a.set_state(U)
    a.steps(13, 1e300)   # fails in its first step
    with pytest.raises(pg.PamhdError) as e:
        a.sync()
    assert e.value.code == pg.ERR_TIMEOUT and a.time()[1] == 1
    a.set_wait_limit(1 << 20)
    for g in (a, b):
        g.set_state(U)
        g.steps(13, 1e300)
        g.sync()
    np.testing.assert_array_equal(a.get_state(), b.get_state())
    assert a.time() == b.time()


@pytest.mark.parametrize("ny,solver", [(4 * 65535, "hlld_athena"), (4 * 65535 + 1, "hlld_athena"),
                                       (300000, "rusanov"), (300000, "hll_athena"), (8 * 65535, "hlld_athena")])
def test_many_rows_match_oracle(port, ny, solver):
    """2-D grids of as many rows as a launch has 32 x 4 tiles for, one more (then 32 x 8 tiles), and the
    most accepted, with COPY sides along y, whose ghost-ghost faces are solved.  Per step, the bar of
    this file."""
    n, kinds = (2, ny, 1), (0, pg.BC_COPY, 0)
    U = states.smooth_3d((1, ny, 2), np.random.default_rng(3))
    gpu, ora = pair(port, n, po.SOLVERS[solver], (0.5, 1.0 / ny, 1.0), states.GAMMA_53, 1.0, 0.4, kinds, kinds)
    gpu.set_state(U)
    ora.set_state(U)
    for s in range(3):
        dg = gpu.step(0.0 if s == 0 else 1.0)
        do, flag, _, _ = ora.step(0.0 if s == 0 else 1.0)
        assert flag == 0
        assert abs(dg - do) <= 1e-13 * max(do, 1e-300), s
        assert field_err(gpu.get_state(), ora.get_state()) <= STEP_TOL, s


@pytest.mark.parametrize("normal", ["field", "none"])
def test_roe_aligned_faces_match_oracle(port, normal):
    """Faces without a transverse field in the Roe average (no transverse field at all, or opposite
    ones at equal densities, with and without a normal field): the solver's branch for them repeats
    the reference's round-off in alpha_f and alpha_s.  Bar: the face bar of 1e-12 of the flux row."""
    rng = np.random.default_rng(12)
    a, b = states.random_face_states(4000, rng, spread=0.3), states.random_face_states(4000, rng, spread=0.3)
    for s in (a, b):
        s[:, 4] -= 0.5 * (s[:, 5:8] ** 2).sum(1)
        s[:, 6:8] = 0.0
        if normal == "none":
            s[:, 5] = 0.0
        s[:, 4] += 0.5 * s[:, 5] ** 2
    half = len(a) // 2   # opposite transverse fields at equal densities
    b[:half, 1:4] *= (a[:half, 0] / b[:half, 0])[:, None]
    b[:half, 4] += 0.5 * (b[:half, 1:4] ** 2).sum(1) * (1 / a[:half, 0] - b[:half, 0] / a[:half, 0] ** 2)
    b[:half, 0] = a[:half, 0]
    t = rng.normal(0.0, 0.3, (half, 2))
    a[:half, 6:8], b[:half, 6:8] = t, -t
    for s in (a, b):
        s[:half, 4] += 0.5 * (t ** 2).sum(1)
    fo, so, go = port.face_flux(po.SOLVERS["roe_athena"], a, b, None, 5 / 3, 1.0)
    fg, sg, gg = pg.face_flux(po.SOLVERS["roe_athena"], a, b, None, 5 / 3, 1.0)
    assert np.array_equal(gg, go)
    ok = go == 0
    assert ok.sum() > 1000
    assert (np.abs(fg[ok] - fo[ok]) / np.abs(fo[ok]).max(axis=1, keepdims=True)).max() <= STEP_TOL


def test_hll_uniform_states_at_rest():
    """HLL in SI units: no mass, energy or field flux between equal states at rest, and a uniform grid
    at rest stays as it is, bit for bit."""
    mu0 = 4e-7 * np.pi
    s = states.states_at_rest(2000, np.random.default_rng(6), mu0)
    flux, speed, flags = pg.face_flux(pg.HLL, s, s, None, 5 / 3, mu0)
    assert not flags.any() and (speed > 0).all()
    assert np.array_equal(flux[:, [0, 4, 5, 6, 7]], np.zeros((len(s), 5)))
    U = np.tile(s[0].reshape(8, 1, 1, 1), (1, 9, 12, 40))
    grid = pg.Context(pg.Config(n=(40, 12, 9), solver=pg.HLL, cell_length=(1e7,) * 3, vacuum_permeability=mu0,
                                time_step_factor=0.4))
    grid.set_state(U)
    grid.steps(8, 1e300)
    grid.sync()
    np.testing.assert_array_equal(grid.get_state(), U)


@pytest.mark.parametrize("solver", list(po.SOLVERS))
def test_equal_wave_speeds_are_refused_like_the_oracle(port, solver):
    """Cells whose sound and Alfven speeds are equal to rounding, the field along the face normal, which
    the reference takes or refuses by the sign of its round-off: the oracle's flags, face by face."""
    s = states.equal_speed_states(5000, np.random.default_rng(10))
    go = port.face_flux(po.SOLVERS[solver], s, s, None, 5 / 3, 1.0)[2]
    assert np.array_equal(pg.face_flux(po.SOLVERS[solver], s, s, None, 5 / 3, 1.0)[2], go)


@pytest.mark.parametrize("solver", list(po.SOLVERS))
@pytest.mark.parametrize("n", [(9, 1, 1), (9, 6, 1), (7, 6, 5), (34, 9, 3)])
def test_a_cell_of_equal_wave_speeds_is_refused_like_the_oracle(port, n, solver):
    """One such cell in a grid at rest, at its corners, on its sides and inside, the field along each
    axis, the sides periodic, COPY or (the cell a ghost state) VALUE: the step takes or refuses it as the
    oracle, with its flag and at its face; in one step, in a run of two and in an ensemble."""
    rng = np.random.default_rng(10)
    cells = states.equal_speed_states(48, rng)
    cells[:, 4] -= 0.5 * (cells[:, 1:4] ** 2).sum(1) / cells[:, 0]
    cells[:, 1:4] = 0.0
    refused = 0
    for i, U in enumerate(cells):
        axis = i % sum(m > 1 for m in n)
        U[5:] = np.roll(U[5:], axis)
        around = U.copy()
        around[4] *= 1.1   # another sound speed
        grid = np.tile(around.reshape(8, 1, 1, 1), (1,) + n[::-1])
        value = i % 3 == 2
        at = [(0, m // 2, m - 1)[rng.integers(3)] for m in n]
        if not value:
            grid[:, at[2], at[1], at[0]] = U
        lo, hi, vlo, vhi = [0] * 3, [0] * 3, [None] * 3, [None] * 3
        if i % 3 > 0:
            lo = hi = [pg.BC_COPY if m > 1 else 0 for m in n]
        if value:
            lo = list(lo)
            lo[axis], vlo[axis] = pg.BC_VALUE, U
        gpu, ora = pair(port, n, po.SOLVERS[solver], (0.1, 0.1, 0.1), 5 / 3, 1.0, 0.4, lo, hi, vlo, vhi)
        ora.set_state(grid)
        _, flag, cell, direction = ora.step(0.0)
        refused += flag != 0
        batch = pg.Batch([gpu.cfg])
        batch.set_state(0, grid)
        for run in (lambda: gpu.step(0.0), lambda: (gpu.steps(2, 0.0), gpu.sync()),
                    lambda: (batch.steps(1, 0.0), batch.sync()), lambda: (batch.run(1, 0.0), batch.sync())):
            gpu.set_state(grid)
            batch.set_state(0, grid)
            if flag == 0:
                run()
                continue
            with pytest.raises(pg.PhysicsError) as e:
                run()
            assert (e.value.flags, tuple(e.value.cell), e.value.direction) == (flag, tuple(cell), direction), i
    assert 0 < refused < len(cells)


@pytest.mark.parametrize("solver", list(po.SOLVERS))
def test_sound_speed_is_correctly_rounded(solver):
    """The face speed between equal states at rest without a field: the sound speed, correctly rounded."""
    s, speed = states.unit_density_gas(5000, np.random.default_rng(9))
    assert np.array_equal(pg.face_flux(po.SOLVERS[solver], s, s, None, 5 / 3, 1.0)[1], speed)


def test_roe_small_transverse_field():
    """Roe faces whose transverse field's square is zero, subnormal or a small normal number: finite."""
    a, b = states.small_transverse_field_states(4000, np.random.default_rng(5), -165, -150)
    flux, _, _ = pg.face_flux(po.SOLVERS["roe_athena"], a, b, None, 5 / 3, 1.0)
    assert np.isfinite(flux).all()


@pytest.mark.parametrize("exponent", [-400, -14, -10, -6, -4, -2])
def test_roe_almost_aligned_faces_match_oracle(port, exponent):
    """Roe faces with a transverse field of size 10^exponent (0 at -400), where the smaller of the
    reference's alphas is all or partly a root of round-off.  Bar: the face bar."""
    a, b = states.small_transverse_field_states(4000, np.random.default_rng(4), exponent, exponent)
    fo, so, go = port.face_flux(po.SOLVERS["roe_athena"], a, b, None, 5 / 3, 1.0)
    fg, sg, gg = pg.face_flux(po.SOLVERS["roe_athena"], a, b, None, 5 / 3, 1.0)
    assert np.array_equal(gg, go)
    ok = go == 0
    assert ok.sum() > 1000
    assert (np.abs(fg[ok] - fo[ok]) / np.abs(fo[ok]).max(axis=1, keepdims=True)).max() <= STEP_TOL


def test_roe_field_tail_matches_oracle(port):
    """A narrow transverse field on 1000 periodic cells, 320 Roe steps: its tail falls by a factor per
    cell and reaches 1e-154 (whose square is subnormal) at step 239.  Bar: STEP_TOL per step."""
    n, steps = 1000, 320
    x = (np.arange(n) + 0.5) / n
    U = np.zeros((8, 1, 1, n))
    U[0] = 1.0
    U[5] = 0.75
    U[6] = np.where(np.abs(x - 0.5) < 0.03, 0.2, 0.0)
    U[4] = 1.0 / (5 / 3 - 1) + 0.5 * (U[5:] ** 2).sum(0)
    gpu, ora = pair(port, (n, 1, 1), po.SOLVERS["roe_athena"], (1 / n, 1.0, 1.0), 5 / 3, 1.0, 0.4)
    gpu.set_state(U)
    ora.set_state(U)
    gpu.steps(steps, 1e300)
    gpu.sync()
    for s in range(steps):
        _, flag, _, _ = ora.step(0.0 if s == 0 else 1e300)
        assert flag == 0
    small = np.abs(ora.get_state()[6])
    assert ((small > 1e-162) & (small < 1.5e-154)).any()
    assert field_err(gpu.get_state(), ora.get_state()) <= steps * STEP_TOL


@pytest.mark.parametrize("solver", list(po.SOLVERS))
def test_face_flux_matches_oracle(port, solver):
    rng = np.random.default_rng(11)
    a, b = states.nearby_face_states(20000, rng)
    c = states.random_face_states(20000, rng)
    d = states.random_face_states(20000, rng)
    e, f = states.edge_case_face_states()
    neg = np.vstack([a, c, e])
    pos = np.vstack([b, d, f])
    sid = po.SOLVERS[solver]
    for mu0, bg in ((1.0, None), (1.0, rng.normal(0, 0.3, (neg.shape[0], 3))), (4e-7 * np.pi, None)):
        scale = np.ones(8)
        if mu0 != 1.0:
            scale[5:8] = np.sqrt(mu0)
        n_, p_ = neg * scale, pos * scale
        fo, so, go = port.face_flux(sid, n_, p_, bg, 5 / 3, mu0)
        fg, sg, gg = pg.face_flux(sid, n_, p_, bg, 5 / 3, mu0)
        # every face the reference rejects is rejected with the same class of error
        assert np.array_equal(gg != 0, go != 0)
        assert np.array_equal(gg[go != 0], go[go != 0])
        ok = go == 0
        row = np.abs(fo[ok]).max(axis=1, keepdims=True)
        row[row == 0] = 1.0
        assert (np.abs(fg[ok] - fo[ok]) / row).max() <= STEP_TOL
        assert (np.abs(sg[ok] - so[ok]) / np.maximum(so[ok], 1e-300)).max() <= STEP_TOL


# ---------------------------------------------------------------- one step from identical inputs

CASES = {
    "periodic3d": dict(n=(12, 10, 9), lengths=(1 / 12, 1 / 10, 1 / 9), gamma=5 / 3, mu0=1.0, cfl=0.4),
    "periodic3d_wide": dict(n=(70, 19, 11), lengths=(0.01, 0.02, 0.03), gamma=5 / 3, mu0=1.0, cfl=0.4),
    "orszag_tang64": dict(n=(64, 64, 1), lengths=(1 / 64, 1 / 64, 1.0), gamma=5 / 3, mu0=1.0, cfl=0.4),
    "briowu200": dict(n=(200, 1, 1), lengths=(1 / 200, 1.0, 1.0), gamma=2.0, mu0=1.0, cfl=0.5,
                      bc_lo=(1, 0, 0), bc_hi=(1, 0, 0)),
}


def initial_state(key, rng):
    c = CASES[key]
    nx, ny, nz = c["n"]
    if key.startswith("orszag"):
        return states.orszag_tang(nx)
    if key.startswith("briowu"):
        return states.brio_wu(nx)
    return states.smooth_3d((nz, ny, nx), rng, amp=0.15)


@pytest.mark.parametrize("solver", list(po.SOLVERS))
@pytest.mark.parametrize("key", list(CASES))
def test_one_step_matches_oracle(port, key, solver):
    rng = np.random.default_rng(21)
    U0 = initial_state(key, rng)
    c = dict(CASES[key])
    gpu, ora = pair(port, c.pop("n"), po.SOLVERS[solver], c.pop("lengths"), c.pop("gamma"), c.pop("mu0"),
                    c.pop("cfl"), **c)
    gpu.set_state(U0)
    ora.set_state(U0)
    # priming step: dt = 0, state unchanged, speeds recorded (tests/mhd/test.cpp:462)
    assert gpu.step(1.0) == 0.0
    assert ora.step(1.0)[0] == 0.0
    np.testing.assert_array_equal(gpu.get_state(), U0)
    # one real step from identical inputs
    dg = gpu.step(1.0)
    do, flag, _, _ = ora.step(1.0)
    assert flag == 0
    assert abs(dg - do) <= STEP_TOL * do
    assert field_err(gpu.get_state(), ora.get_state()) <= STEP_TOL


@pytest.mark.parametrize("solver", list(po.SOLVERS))
def test_bounded_grid_matches_oracle(port, solver):
    """COPY and VALUE sides plus a periodic one: ghost refresh and the boundary-layer speeds."""
    rng = np.random.default_rng(5)
    U0 = states.smooth_3d((7, 9, 11), rng, amp=0.1)
    inflow = np.array([1.2, 0.3 * 1.2, 0.2 * 1.2, 0.0,
                       states.energy(1.2, np.array([[0.3], [0.2], [0.0]]), 0.7,
                                     np.array([[0.4], [0.1], [-0.2]]), 5 / 3)[0], 0.4, 0.1, -0.2])
    gpu, ora = pair(port, (11, 9, 7), po.SOLVERS[solver], (0.09, 0.11, 0.13), 5 / 3, 1.0, 0.4,
                    bc_lo=(po.BC_VALUE, po.BC_COPY, po.BC_PERIODIC), bc_hi=(po.BC_COPY, po.BC_COPY, po.BC_PERIODIC),
                    value_lo=[inflow, None, None])
    gpu.set_state(U0)
    ora.set_state(U0)
    for step in range(6):
        dg = gpu.step(1.0)
        do, flag, _, _ = ora.step(1.0)
        assert flag == 0
        assert abs(dg - do) <= 1e-12 * max(do, 1e-300) or dg == do == 0.0
        assert field_err(gpu.get_state(), ora.get_state()) <= STEP_TOL * (1 + step)


@pytest.mark.parametrize("solver", list(po.SOLVERS))
@pytest.mark.parametrize("layout", ["bounded3d", "yz_plane"])
def test_max_signal_matches_oracle(port, layout, solver):
    """pamhd_gpu_step's max_signal output: per dimension the largest face speed of the step (the
    maxima of the reference's Max_v, ghost-ghost faces of non-periodic sides included), equal to
    the oracle's to round-off, and the next step's dt follows from it by the CFL rule."""
    rng = np.random.default_rng(13)
    if layout == "bounded3d":
        n, lengths = (11, 9, 7), (0.09, 0.11, 0.13)
        U0 = states.smooth_3d((7, 9, 11), rng, amp=0.1)
        bc = dict(bc_lo=(po.BC_COPY, po.BC_COPY, po.BC_PERIODIC), bc_hi=(po.BC_COPY, po.BC_COPY, po.BC_PERIODIC))
    else:  # a y-z grid: the context relabels its axes, max_signal stays in the caller's axes
        n, lengths = (1, 16, 12), (1.0, 1 / 16, 1 / 12)
        U0 = states.smooth_3d((12, 16, 1), rng, amp=0.1)
        bc = {}
    gpu, ora = pair(port, n, po.SOLVERS[solver], lengths, 5 / 3, 1.0, 0.4, **bc)
    gpu.set_state(U0)
    ora.set_state(U0)
    prev = None
    for step in range(4):
        dg, sig = gpu.step_signal(1.0)
        do, flag, _, _ = ora.step(1.0)
        assert flag == 0
        so = ora.max_signal()
        assert np.all((sig == 0) == (so == 0))
        assert np.abs(sig - so).max() <= 1e-12 * so.max()
        if prev is not None:
            # the lagged rule: dt = min over dimensions of CFL * dx_d / max_signal_d of the last step
            expect = min(0.4 * lengths[d] / prev[d] for d in range(3) if prev[d] > 0)
            assert dg == min(expect, 1.0)
        prev = sig


# ---------------------------------------------------------------- trajectories

@pytest.mark.parametrize("solver", ["rusanov", "hll_athena", "hlld_athena"])
def test_orszag_tang_trajectory(port, solver):
    """50 steps of Orszag-Tang 64^2: dt history and state stay within round-off growth."""
    U0 = states.orszag_tang(64)
    c = dict(CASES["orszag_tang64"])
    gpu, ora = pair(port, c.pop("n"), po.SOLVERS[solver], c.pop("lengths"), c.pop("gamma"), c.pop("mu0"),
                    c.pop("cfl"))
    gpu.set_state(U0)
    ora.set_state(U0)
    t_o, dts_o = ora.run(0.0, 10.0, 50)
    gpu.steps(50, 10.0)
    gpu.sync()
    t_g, n_g, _ = gpu.time()
    dts_g = gpu.dt_history(50)
    assert n_g == 50
    np.testing.assert_allclose(dts_g, dts_o, rtol=1e-10, atol=0)
    assert abs(t_g - t_o) <= 1e-10 * t_o
    assert field_err(gpu.get_state(), ora.get_state()) <= 1e-9


def test_brio_wu_to_t_end(port):
    """Brio-Wu, 1000 cells, gamma 2, HLLD, CFL 0.5, copy boundaries, to t = 0.1."""
    U0 = states.brio_wu(1000)
    gpu, ora = pair(port, (1000, 1, 1), po.HLLD, (1e-3, 1.0, 1.0), 2.0, 1.0, 0.5,
                    bc_lo=(po.BC_COPY, 0, 0), bc_hi=(po.BC_COPY, 0, 0))
    gpu.set_state(U0)
    ora.set_state(U0)
    t_o, dts_o = ora.run(0.0, 0.1, 100000)
    gpu.steps(len(dts_o) + 5, 0.1)
    t_g, n_g, _ = gpu.time()
    assert t_o == pytest.approx(0.1, abs=0) or abs(t_o - 0.1) < 1e-15
    assert abs(t_g - t_o) <= 1e-13
    dts_g = gpu.dt_history(n_g)
    np.testing.assert_allclose(dts_g[: len(dts_o)], dts_o, rtol=1e-9)
    assert field_err(gpu.get_state(), ora.get_state()) <= 1e-8


# ---------------------------------------------------------------- properties at any size

def test_graph_steps_equal_single_steps():
    rng = np.random.default_rng(8)
    U0 = states.smooth_3d((20, 24, 40), rng)
    cfg = pg.Config(n=(40, 24, 20), solver=pg.HLLD, cell_length=(0.025, 0.04, 0.05), time_step_factor=0.4)
    a, b = pg.Context(cfg), pg.Context(cfg)
    a.set_state(U0)
    b.set_state(U0)
    for _ in range(14):
        a.step(1e9)
    b.steps(14, 1e9)
    b.sync()
    np.testing.assert_array_equal(a.get_state(), b.get_state())
    np.testing.assert_array_equal(a.dt_history(14), b.dt_history(14))


def test_translation_invariance_bitwise():
    """Shifting a periodic initial state by whole cells shifts the solution bit for bit:
    every face is solved by the same arithmetic wherever it sits in the tiling."""
    rng = np.random.default_rng(9)
    U0 = states.smooth_3d((16, 20, 72), rng)
    cfg = pg.Config(n=(72, 20, 16), solver=pg.HLLD, cell_length=(0.02, 0.05, 0.06), time_step_factor=0.4)
    a, b = pg.Context(cfg), pg.Context(cfg)
    shift = (5, 7, 13)  # z, y, x
    a.set_state(U0)
    b.set_state(np.roll(U0, shift, axis=(1, 2, 3)))
    a.steps(7, 1e9)
    b.steps(7, 1e9)
    np.testing.assert_array_equal(np.roll(a.get_state(), shift, axis=(1, 2, 3)), b.get_state())


@pytest.mark.parametrize("solver", list(po.SOLVERS))
def test_conservation_on_periodic_grid(solver):
    rng = np.random.default_rng(10)
    U0 = states.smooth_3d((24, 32, 40), rng)
    cfg = pg.Config(n=(40, 32, 24), solver=po.SOLVERS[solver], cell_length=(0.025, 0.03, 0.04),
                    time_step_factor=0.4)
    g = pg.Context(cfg)
    g.set_state(U0)
    t0 = g.totals()
    g.steps(20, 1e9)
    t1 = g.totals()
    absum = np.abs(U0).reshape(8, -1).sum(axis=1) * 0.025 * 0.03 * 0.04
    assert np.all(np.abs(t1 - t0) <= 1e-13 * absum)


def test_invalid_state_reported_like_oracle(port):
    rng = np.random.default_rng(5)
    U0 = states.smooth_3d((6, 5, 40), rng)
    U0[4, 3, 2, 17] = 0.0  # negative pressure in cell x=17, y=2, z=3
    gpu, ora = pair(port, (40, 5, 6), po.HLLD, (0.025, 0.2, 0.16), 5 / 3, 1.0, 0.4)
    gpu.set_state(U0)
    ora.set_state(U0)
    _, flag, cell, d = ora.step(0.0)
    with pytest.raises(pg.PhysicsError) as e:
        gpu.step(0.0)
    assert e.value.flags == flag == pg.FLAG_PRESSURE
    assert e.value.cell == cell and e.value.direction == d


def test_time_capped_at_t_end():
    U0 = states.orszag_tang(32)
    cfg = pg.Config(n=(32, 32, 1), solver=pg.HLL, cell_length=(1 / 32, 1 / 32, 1.0), time_step_factor=0.4)
    g = pg.Context(cfg)
    g.set_state(U0)
    g.steps(400, 0.05)
    t, n, _ = g.time()
    assert t == 0.05 and n == 400


def test_blast_positivity_failure_matches_oracle(port):
    """The 64^3 magnetised blast loses positivity in the reference scheme (first-order HLLD, cell-
    centred field): the GPU must stop at the same step, on the same face, with the same error."""
    n = 64
    U0 = states.blast_wave(n)
    gpu, ora = pair(port, (n, n, n), po.HLLD, (1 / n,) * 3, 5 / 3, 1.0, 0.4)
    gpu.set_state(U0)
    ora.set_state(U0)
    fail_o = fail_g = None
    for step in range(120):
        do, flag, cell, d = ora.step(1e30)
        if flag:
            fail_o = (step, flag, cell, d)
            break
        dg = gpu.step(1e30)
        assert abs(dg - do) <= 1e-10 * max(do, 1e-300) or dg == do == 0.0
    assert fail_o is not None
    try:
        gpu.step(1e30)
    except pg.PhysicsError as e:
        fail_g = (fail_o[0], e.flags, e.cell, e.direction)
    assert fail_g == fail_o


def test_steps_after_a_failure_hold_the_grid():
    """The reference aborts in the step whose face fails (mhd/solve.hpp:156-181): here that step
    completes and every later one leaves the grid as it left it.  The 64^3 blast loses positivity
    after some steps; then steps one at a time, in a CUDA graph and split in two parts keep the
    state, the time, the step count and the dt history, and report the error again; set_state
    starts over."""
    n = 64
    U0 = states.blast_wave(n)
    cfg = pg.Config(n=(n, n, n), solver=pg.HLLD, cell_length=(1 / n,) * 3, time_step_factor=0.4)
    g = pg.Context(cfg)
    g.set_state(U0)
    failed = None
    for step in range(120):
        try:
            g.step(1e30)
        except pg.PhysicsError as e:
            failed = (step, e.flags, e.cell, e.direction)
            break
    assert failed is not None and failed[0] > 5
    held = g.get_state()
    t, count, _ = g.time()
    assert count == failed[0] + 1
    history = g.dt_history(200)
    assert len(history) == count and history[-1] > 0.0
    for _ in range(2):
        with pytest.raises(pg.PhysicsError) as e:
            g.step(1e30)
        assert (e.value.flags, e.value.cell, e.value.direction) == failed[1:]
    g.steps(13, 1e30)
    with pytest.raises(pg.PhysicsError):
        g.sync()
    g.step_part(1, 1e30)
    g.step_part(2, 1e30)
    with pytest.raises(pg.PhysicsError):
        g.sync()
    np.testing.assert_array_equal(g.get_state(), held)
    assert g.time() == (t, count, 0.0)
    np.testing.assert_array_equal(g.dt_history(200), history)
    g.set_state(U0)
    assert g.step(1e30) == 0.0 and g.step(1e30) == history[1]
    assert g.status()[0] == 0


@pytest.mark.parametrize("count", [0, 1, 33, 257])
def test_face_flux_empty_and_ragged_batches(port, count):
    """Batches of no face, one face and counts that leave partial blocks: the same results as
    the oracle face by face (an empty batch is a valid call that does nothing)."""
    rng = np.random.default_rng(12)
    a, b = states.nearby_face_states(max(count, 1), rng)
    a, b = a[:count], b[:count]
    fo, so, go = port.face_flux(po.HLLD, a, b, None, 5 / 3, 1.0)
    fg, sg, gg = pg.face_flux(po.HLLD, a, b, None, 5 / 3, 1.0)
    assert fg.shape == (count, 8) and sg.shape == (count,) and gg.shape == (count,)
    assert np.array_equal(gg, go)
    if count:
        row = np.maximum(np.abs(fo).max(axis=1, keepdims=True), 1e-300)
        assert (np.abs(fg - fo) / row).max() <= STEP_TOL
        assert (np.abs(sg - so) / np.maximum(so, 1e-300)).max() <= STEP_TOL


# ---------------------------------------------------------------- the configured workloads

def test_blast_256_configured(port):
    """The headline workload at its size: the 256^3 magnetised blast, HLLD, CFL 0.4, periodic.
    The priming step and two steps against the oracle (on every host thread) at the per-step bar;
    then size-independent properties over 20 more steps: the conserved totals stay within
    round-off, and a copy of the state shifted by whole cells stays the shifted solution bit for
    bit."""
    import os
    n = 256
    U0 = states.blast_wave(n)
    gpu, _ = pair(port, (n, n, n), po.HLLD, (1 / n,) * 3, 5 / 3, 1.0, 0.4)
    ora = port.grid(po.make_cfg((n, n, n), po.HLLD, (1 / n,) * 3, 5 / 3, 1.0, 0.4),
                    threads=max(1, len(os.sched_getaffinity(0))))
    gpu.set_state(U0)
    ora.set_state(U0)
    for s in range(3):
        cap = 0.0 if s == 0 else 1.0
        do, flag, _, _ = ora.step(cap)
        dg = gpu.step(cap)
        assert flag == 0
        assert abs(dg - do) <= 1e-13 * max(do, 1e-300)
        assert field_err(gpu.get_state(), ora.get_state()) <= STEP_TOL, s
    del ora
    shift = (17, 5, 200)   # z, y, x
    b = pg.Context(gpu.cfg)
    U3 = gpu.get_state()
    b.set_state(np.roll(U3, shift, axis=(1, 2, 3)))
    gpu.set_state(U3)
    t0 = gpu.totals()
    gpu.steps(20, 1e9)
    b.steps(20, 1e9)
    t1 = gpu.totals()
    Uf = gpu.get_state()
    # round-off of 16.7 M cell updates a step (random signs): about sqrt(N) eps of the sum of |U|
    absum = np.maximum(np.abs(U3).reshape(8, -1).sum(axis=1), np.abs(Uf).reshape(8, -1).sum(axis=1)) / n ** 3
    assert np.all(np.abs(t1 - t0) <= 1e-11 * absum)
    np.testing.assert_array_equal(np.roll(Uf, shift, axis=(1, 2, 3)), b.get_state())


@pytest.mark.parametrize("solver", list(po.SOLVERS))
def test_brio_wu_configured_every_solver(port, solver):
    """The shock-tube workload with each solver: 1000 cells on [0, 1], gamma 2, CFL 0.5, copy
    boundaries, to t = 0.1; same step count, dt history within 1e-9, state within 1e-8."""
    U0 = states.brio_wu(1000)
    gpu, ora = pair(port, (1000, 1, 1), po.SOLVERS[solver], (1e-3, 1.0, 1.0), 2.0, 1.0, 0.5,
                    bc_lo=(po.BC_COPY, 0, 0), bc_hi=(po.BC_COPY, 0, 0))
    gpu.set_state(U0)
    ora.set_state(U0)
    t_o, dts_o = ora.run(0.0, 0.1, 100000)
    gpu.steps(len(dts_o) + 5, 0.1)
    gpu.sync()
    t_g, n_g, _ = gpu.time()
    assert abs(t_g - t_o) <= 1e-13
    dts_g = gpu.dt_history(n_g)
    np.testing.assert_allclose(dts_g[: len(dts_o)], dts_o, rtol=1e-9)
    assert np.all(dts_g[len(dts_o):] == 0.0)
    assert field_err(gpu.get_state(), ora.get_state()) <= 1e-8


@pytest.mark.parametrize("solver", list(po.SOLVERS))
def test_orszag_tang_512_configured(port, solver):
    """The 2-D workload at its size: Orszag-Tang 512^2, periodic, gamma 5/3, CFL 0.4, up to 1000
    steps with each solver.  Every 50 steps both are restarted from the GPU's state (a priming
    step, then one step from identical inputs must agree to 1e-12, the per-step bar); in between
    they run independently (dt within 1e-9).  The reference scheme loses positivity on this
    problem near t = 0.104 for some solvers: the GPU must stop at the same step and face, with
    the same error class, as the oracle, or both run all the steps."""
    n = 512
    U0 = states.orszag_tang(n)
    gpu, ora = pair(port, (n, n, 1), po.SOLVERS[solver], (1 / n, 1 / n, 1.0), 5 / 3, 1.0, 0.4)
    gpu.set_state(U0)
    ora.set_state(U0)
    fail_g = fail_o = None
    for s in range(1001):
        if s % 50 == 0 and s > 0:
            U = gpu.get_state()
            gpu.set_state(U)
            ora.set_state(U)
            assert gpu.step(1.0) == 0.0 and ora.step(1.0)[0] == 0.0
            checked = True
        else:
            checked = False
        try:
            dg = gpu.step(1.0)
        except pg.PhysicsError as e:
            fail_g = (s, tuple(e.cell), e.direction, e.flags)
        do, flag, cell, d = ora.step(1.0)
        if flag:
            fail_o = (s, tuple(cell), d, flag)
        if fail_g or fail_o:
            break
        assert abs(dg - do) <= 1e-9 * max(do, 1e-300) or dg == do == 0.0
        if checked:
            assert abs(dg - do) <= STEP_TOL * do, s
            assert field_err(gpu.get_state(), ora.get_state()) <= STEP_TOL, s
    # the same step and first failing face; the GPU's flags (all failures of the step, OR-ed)
    # include the oracle's (the first face's)
    assert (fail_g is None) == (fail_o is None), (fail_g, fail_o)
    if fail_g is not None:
        assert fail_g[:3] == fail_o[:3], (fail_g, fail_o)
        assert fail_g[3] & fail_o[3], (fail_g, fail_o)


@pytest.mark.parametrize("case,vx", [("da_px", 1.0), ("da_mx", -1.0)])
def test_reproduces_reference_program_output(case, vx):
    """The reference program's own output (tests/mhd/reference/hydrodynamic/density_advection/1d/
    {+x,-x}/rusanov/mhd_000000917.dc, via tests/golden/dc_goldens.npz): density advection, 200
    periodic cells, Rusanov, CFL 0.5, t = 0 .. 1.  Same 917 steps and final time, state within
    1e-12 of the reference's."""
    import os
    g = np.load(os.path.join(os.path.dirname(__file__), "golden", "dc_goldens.npz"))
    gamma = float(g[case + "_gamma"])
    n = int(g[case + "_cells"][0])
    U0 = states.density_advection(n, gamma, vx, float(g[case + "_proton_mass"]))
    cfg = pg.Config(n=(n, 1, 1), solver=pg.RUSANOV, cell_length=tuple(g[case + "_cell_length"]),
                    adiabatic_index=gamma, vacuum_permeability=float(g[case + "_mu0"]), time_step_factor=0.5)
    ctx = pg.Context(cfg)
    ctx.set_state(U0)
    t_end = float(g[case + "_time"])
    ctx.steps(int(g[case + "_step"]) + 10, t_end)
    ctx.sync()
    t, steps, _ = ctx.time()
    dts = ctx.dt_history(steps)
    assert abs(t - t_end) <= 1e-14
    assert int((dts > 0).sum()) == int(g[case + "_step"])
    out = ctx.get_state().reshape(8, n)
    ref = g[case + "_state"]
    scale = np.maximum(np.abs(ref).max(axis=1), 1e-300)
    assert (np.abs(out - ref).max(axis=1) / scale).max() <= STEP_TOL
    # the same state through the reference's file format, and back into a context
    import tempfile
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "mhd_000000917.dc")
        ctx.save_dc(path, step=int(g[case + "_step"]), time=t, proton_mass=float(g[case + "_proton_mass"]))
        info, U = pg.read_dc(path)
        assert info["step"] == int(g[case + "_step"]) and info["periodic"] == (True, True, True)
        assert np.array_equal(U.reshape(8, n), out)
        ctx2 = pg.Context(cfg)
        ctx2.load_dc(path)
        assert np.array_equal(ctx2.get_state().reshape(8, n), out)


# ---------------------------------------------------------------- other active dimensions

RELABEL_CASES = {
    "yz_periodic": dict(n=(1, 12, 10), lengths=(1.0, 0.08, 0.1), bc_lo=(0, 0, 0), bc_hi=(0, 0, 0)),
    "xz_copy": dict(n=(14, 1, 10), lengths=(0.07, 1.0, 0.1), bc_lo=(po.BC_COPY, 0, po.BC_COPY),
                    bc_hi=(po.BC_COPY, 0, po.BC_COPY)),
    "z_copy": dict(n=(1, 1, 40), lengths=(1.0, 1.0, 0.025), bc_lo=(0, 0, po.BC_COPY), bc_hi=(0, 0, po.BC_COPY)),
    "y_periodic": dict(n=(1, 36, 1), lengths=(1.0, 0.03, 1.0), bc_lo=(0, 0, 0), bc_hi=(0, 0, 0)),
}


@pytest.mark.parametrize("solver", ["hll_athena", "hlld_athena", "roe_athena"])
@pytest.mark.parametrize("key", list(RELABEL_CASES))
def test_other_active_dimensions_match_oracle(port, key, solver):
    """Grids that are not x, x-y or x-y-z run with relabelled axes on the GPU; the oracle steps
    them as they are.  Per step within 1e-12."""
    c = RELABEL_CASES[key]
    nx, ny, nz = c["n"]
    rng = np.random.default_rng(41)
    U0 = states.smooth_3d((nz, ny, nx), rng, amp=0.1)
    gpu, ora = pair(port, c["n"], po.SOLVERS[solver], c["lengths"], 5 / 3, 1.0, 0.4, bc_lo=c["bc_lo"],
                    bc_hi=c["bc_hi"])
    gpu.set_state(U0)
    ora.set_state(U0)
    for step in range(6):
        dg = gpu.step(1.0)
        do, flag, _, _ = ora.step(1.0)
        assert flag == 0
        assert abs(dg - do) <= STEP_TOL * max(do, 1e-300) or dg == do == 0.0
        assert field_err(gpu.get_state(), ora.get_state()) <= STEP_TOL * (1 + step), step


def test_yz_grid_equals_xy_grid_bitwise():
    """A y-z grid runs as the x-y grid with its axes rotated: the same bits."""
    rng = np.random.default_rng(43)
    ny, nz = 20, 16
    U_yz = states.smooth_3d((nz, ny, 1), rng, amp=0.1)            # (8, nz, ny, 1)
    # the rotated problem: x' = y, y' = z, z' = x; momentum and field components rotate with the axes
    U_xy = np.empty((8, 1, nz, ny))
    for v, u in enumerate((0, 2, 3, 1, 4, 6, 7, 5)):
        U_xy[v, 0] = U_yz[u, :, :, 0]
    a = pg.Context(pg.Config(n=(1, ny, nz), solver=pg.HLLD, cell_length=(1.0, 0.05, 0.0625), time_step_factor=0.4))
    b = pg.Context(pg.Config(n=(ny, nz, 1), solver=pg.HLLD, cell_length=(0.05, 0.0625, 1.0), time_step_factor=0.4))
    a.set_state(U_yz)
    b.set_state(U_xy)
    a.steps(12, 1e9)
    b.steps(12, 1e9)
    a.sync()
    b.sync()
    Ya, Xb = a.get_state(), b.get_state()
    for v, u in enumerate((0, 2, 3, 1, 4, 6, 7, 5)):
        np.testing.assert_array_equal(Xb[v, 0], Ya[u, :, :, 0])
    np.testing.assert_array_equal(a.dt_history(12), b.dt_history(12))
    np.testing.assert_array_equal(a.totals()[[0, 2, 3, 1, 4, 6, 7, 5]], b.totals())


@pytest.mark.parametrize("solver", ["rusanov", "hll_athena", "hlld_athena", "roe_athena"])
@pytest.mark.parametrize("name", ["blast_3d", "smooth_3d", "orszag_tang_2d", "smooth_1d"])
def test_steps_match_reference_step_functions(name, solver):
    """The GPU step against the reference's own step functions (minimize_timestep, the substep
    plan, get_all_fluxes, update_mhd_state, compiled unchanged; committed outputs, see
    test_cell_centred_ref_pin.py): the priming step and nine steps, every dt within 1e-13 and the
    state within 1e-12 of each field's largest magnitude."""
    import test_cell_centred_ref_pin as R
    U, dts = R.golden(name, solver)
    n, lengths = R.CASES[name]
    cfg = pg.Config(n=n, solver=R.SOLVERS[solver], cell_length=lengths, adiabatic_index=states.GAMMA_53,
                    time_step_factor=0.4)
    ctx = pg.Context(cfg)
    try:
        ctx.set_state(R.case_input(name))
        got = [ctx.step(0.0 if s == 0 else 1e300) for s in range(R.STEPS)]
        Ug = ctx.get_state()
    finally:
        ctx.close()
    assert np.abs(np.array(got) - dts).max() <= 1e-13 * dts.max()
    for rows in ([0], [1, 2, 3], [4], [5, 6, 7]):
        assert np.abs(Ug[rows] - U[rows]).max() <= 1e-12 * np.abs(U[rows]).max(), rows
