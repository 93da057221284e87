"""The face solvers of the GPU step (pamhd_b200/csrc/mhd_device.cuh), compiled for the host
(tests/host/solvers_host.cpp), against the oracle's on states where rearranged arithmetic can go
wrong, and the tile shapes of the step (CPU only)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from oracle import pyoracle as po
import states

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "host", "solvers_host.cpp")
LIB = os.path.join(HERE, "host", "_build", "libsolvers_host.so")
D = ctypes.POINTER(ctypes.c_double)


@pytest.fixture(scope="module")
def host():
    """face_flux(solver, neg, pos, mu0) -> flux, speed, flags of the host build; .lib, the build."""
    os.makedirs(os.path.dirname(LIB), exist_ok=True)
    csrc = os.path.join(os.path.dirname(HERE), "pamhd_b200", "csrc")
    deps = [SRC] + [os.path.join(csrc, f) for f in ("mhd_device.cuh", "step.cuh", "grid_setup.cuh")]
    if not os.path.exists(LIB) or any(os.path.getmtime(d) > os.path.getmtime(LIB) for d in deps):
        subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-o", LIB, SRC],
                       check=True)
    L = ctypes.CDLL(LIB)
    L.host_face_flux.argtypes = [ctypes.c_int32, ctypes.c_int64, D, D, ctypes.c_double, ctypes.c_double, D, D,
                                 ctypes.POINTER(ctypes.c_uint32)]
    L.host_face_flux.restype = None

    def face_flux(solver, neg, pos, mu0=1.0):
        neg, pos = np.ascontiguousarray(neg), np.ascontiguousarray(pos)
        flux, speed, flags = np.zeros((len(neg), 8)), np.zeros(len(neg)), np.zeros(len(neg), np.uint32)
        c = lambda a: a.ctypes.data_as(D)
        L.host_face_flux(solver, len(neg), c(neg), c(pos), 5 / 3, mu0, c(flux), c(speed),
                         flags.ctypes.data_as(ctypes.POINTER(ctypes.c_uint32)))
        return flux, speed, flags

    face_flux.lib = L
    return face_flux


@pytest.mark.parametrize("low,high", [(-165, -153), (-153, -3)])
def test_roe_small_transverse_field(host, port, low, high):
    """Roe faces whose transverse field is 1e-165 to 1e-3: its square is zero, subnormal (below some
    1.5e-154) or normal.  The flux is finite wherever the oracle's is.  Except between 1e-163 and
    1e-157, where that square keeps too few bits for the oracle's field direction to have length 1, the
    flags are the oracle's and the flux is at most 1e-6 of the row away (alphas that are a root of
    round-off, some 1e-8)."""
    a, b = states.small_transverse_field_states(20000, np.random.default_rng(5), low, high)
    fo, so, go = port.face_flux(po.SOLVERS["roe_athena"], a, b, None, 5 / 3, 1.0)
    fh, sh, gh = host(po.SOLVERS["roe_athena"], a, b)
    assert (go == 0).sum() > 10000 and np.isfinite(fo).all()
    assert np.isfinite(fh).all()
    size = np.maximum(np.abs(a[:, 6:8]).max(1), np.abs(b[:, 6:8]).max(1))
    clear = (size < 1e-163) | (size > 1e-157)
    assert np.array_equal(gh[clear], go[clear])
    ok = clear & (go == 0)
    assert (np.abs(fh[ok] - fo[ok]) / np.abs(fo[ok]).max(axis=1, keepdims=True)).max() <= 1e-6


@pytest.mark.parametrize("exponent", [-400, -14, -12, -10, -8, -6, -5, -4, -3, -2, -1])
def test_roe_almost_aligned_field_matches_oracle(host, port, exponent):
    """Roe faces with a transverse field of size 10^exponent (0 at -400): the smaller of the reference's
    alphas is a root of round-off below some 1e-8, partly so up to 1e-3.  Bar: 1e-12 of the flux row."""
    a, b = states.small_transverse_field_states(20000, np.random.default_rng(4), exponent, exponent)
    fo, so, go = port.face_flux(po.SOLVERS["roe_athena"], a, b, None, 5 / 3, 1.0)
    fh, sh, gh = host(po.SOLVERS["roe_athena"], a, b)
    assert np.array_equal(gh, go)
    ok = go == 0
    assert ok.sum() > 10000
    assert (np.abs(fh[ok] - fo[ok]) / np.abs(fo[ok]).max(axis=1, keepdims=True)).max() <= 1e-12


def test_hll_equal_states_at_rest(host):
    """HLL between equal states at rest, SI units: no mass, energy or field flux at all."""
    mu0 = 4e-7 * np.pi
    s = states.states_at_rest(2000, np.random.default_rng(6), mu0)
    flux, speed, flags = host(po.SOLVERS["hll_athena"], s, s, mu0)
    assert not flags.any() and (speed > 0).all()
    assert np.array_equal(flux[:, [0, 4, 5, 6, 7]], np.zeros((len(s), 5)))


@pytest.mark.parametrize("solver", ["rusanov", "hll_athena", "hlld_athena"])
def test_mirrored_faces(host, solver):
    """A face mirrored along its normal has the mirrored flux, bit for bit."""
    rng = np.random.default_rng(7)
    a, b = states.random_face_states(5000, rng), states.random_face_states(5000, rng)
    f, s, g = host(po.SOLVERS[solver], a, b)
    fm, sm, gm = host(po.SOLVERS[solver], b * states.MIRROR_STATE, a * states.MIRROR_STATE)
    assert np.array_equal(g, gm) and np.array_equal(s, sm)
    assert np.array_equal(fm, np.where(g[:, None] == 0, f * states.MIRROR_FLUX, 0.0))


def test_rounded_helpers(host):
    """recip_rn, quotient_rn and sqrt_rn against IEEE division and square root, bit for bit."""
    rng = np.random.default_rng(8)
    n = 200000
    x = rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-500, 500, n)
    a = rng.uniform(-2.0, 2.0, n) * 2.0 ** rng.integers(-200, 200, n)
    x[:3] = 1.0, 2.0 ** -700, 2.0 ** 1000
    inverse, quotient, root = np.zeros(n), np.zeros(n), np.zeros(n)
    host.lib.host_rounded(ctypes.c_int64(n), *(v.ctypes.data_as(D) for v in (a, x, inverse, quotient, root)))
    assert np.array_equal(inverse, 1.0 / x)
    assert np.array_equal(quotient, a / x)
    assert np.array_equal(root, np.sqrt(x))
    zero = np.zeros(1)
    host.lib.host_rounded(ctypes.c_int64(1), *(v.ctypes.data_as(D) for v in (zero, zero, inverse, quotient, root)))
    assert root[0] == 0.0


def test_sound_speed_is_correctly_rounded(host):
    """The speed of a face between equal states at rest without a field is the sound speed, whose root is
    correctly rounded in the face fluxes (as in the staggered and local-time-stepping steps)."""
    s, speed = states.unit_density_gas(5000, np.random.default_rng(9))
    for solver in ("rusanov", "hll_athena", "hlld_athena", "roe_athena"):
        assert np.array_equal(host(po.SOLVERS[solver], s, s)[1], speed), solver


@pytest.mark.parametrize("mu0", [1.0, 4e-7 * np.pi])
def test_equal_wave_speeds_are_refused_like_the_oracle(host, port, mu0):
    """Cells whose sound and Alfven speeds are equal to rounding, the field along the face normal: the
    reference's fast speed is the root of round-off, of either sign or zero, and it refuses the cell
    unless that is positive.  The same flags as the oracle."""
    s = states.equal_speed_states(5000, np.random.default_rng(10), mu0=mu0)
    for solver in ("rusanov", "hll_athena", "hlld_athena", "roe_athena"):
        go = port.face_flux(po.SOLVERS[solver], s, s, None, 5 / 3, mu0)[2]
        assert (go == 0).sum() > 500 and (go != 0).sum() > 500
        assert np.array_equal(host(po.SOLVERS[solver], s, s, mu0)[2], go), solver


def test_short_grids_have_the_tiles_they_are_named_for(host):
    """The grids of the GPU test of short z chunks and shaped tiles take the tiles listed with them."""
    I3 = ctypes.c_int32 * 3
    for n, tiles in states.SHORT_GRIDS.items():
        shape = I3()
        host.lib.host_tile_shape(po.SOLVERS["hlld_athena"], 8, I3(*n), shape)
        assert tuple(shape) == tiles, n
