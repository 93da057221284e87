"""What the framework's speed is measured on: runs of its steps as a simulation program makes them.

A pass is one whole run through the public API: the initial state in, the dt = 0 priming step, the
steps, the final state out (the cell-centred context on device arrays, the others, whose API takes
host arrays, on pinned host memory).  The same state can be run again: every pass starts from the
initial state.  The states are the workloads of the tests and of bench.py (Brio-Wu tube,
Orszag-Tang vortex, magnetised blast, solar-wind boxes, smooth 3-D states) with a seeded
perturbation, so that another seed gives another run.

exact() computes the same runs with torch in 64 bits from the schemes' formulas alone.
"""
import ctypes
import math

import numpy as np
import torch

import pamhd_b200 as pg

GAMMA = 5.0 / 3.0
MU0_SI = 4e-7 * math.pi
PROTON = 1.672621777e-27
BOLTZMANN = 1.380649e-23
BOX_CELL = 6.371e5          # cell size of the solar-wind boxes, m
T_END = 1e300
DEV = "cuda"

# flops of a cell's update: per face solved, and per cell (derived quantities and update)
FACE_FLOPS = {"rusanov": 110, "hll_athena": 120, "hlld_athena": 260, "roe_athena": 450}
CELL_FLOPS = 110


def listed():
    return [
        # the smallest call: the shock tube every MHD code starts with; launches and latency
        {"name": "tube_hlld_1000", "kind": "tube", "solver": "hlld_athena", "nx": 1000, "ny": 1, "nz": 1, "steps": 200},
        # a small ragged 2-D vortex with the cheapest solver: less than one wave of tiles
        {"name": "vortex_rusanov_257x180", "kind": "vortex", "solver": "rusanov", "nx": 257, "ny": 180, "nz": 1,
         "steps": 60},
        # the 2-D vortex at its configured size with the most accurate solver
        {"name": "vortex_roe_512", "kind": "vortex", "solver": "roe_athena", "nx": 512, "ny": 512, "nz": 1, "steps": 30},
        # a 3-D blast of odd sizes, partial tiles along x and y
        {"name": "blast_hlld_150x99x67", "kind": "blast", "solver": "hlld_athena", "nx": 150, "ny": 99, "nz": 67,
         "steps": 20},
        # the largest: the 3-D magnetised blast at its configured size
        {"name": "blast_hlld_256", "kind": "blast", "solver": "hlld_athena", "nx": 256, "ny": 256, "nz": 256,
         "steps": 20},
        # one solar-wind box: inflow on -x, open sides elsewhere
        {"name": "wind_hll_96x64x50", "kind": "wind", "solver": "hll_athena", "nx": 96, "ny": 64, "nz": 50, "steps": 40},
        # an ensemble of solar-wind boxes, each with its own timestep, in one persistent run
        {"name": "ensemble_hll_16", "kind": "ensemble", "solver": "hll_athena", "boxes": 16, "smallest": 32,
         "largest": 96, "steps": 60},
        # a gradient of a 2-D run (checkpointed discrete adjoint): the backward direction
        {"name": "adjoint_hlld_256", "kind": "adjoint", "solver": "hlld_athena", "nx": 256, "ny": 256, "nz": 1,
         "steps": 60, "every": 10},
        # the production step with the face field, periodic
        {"name": "staggered_hlld_128", "kind": "staggered", "solver": "hlld_athena", "nx": 128, "ny": 128, "nz": 128,
         "steps": 60},
        # the same in a solar-wind box: inflow on -x, open sides, odd sizes
        {"name": "staggered_box_hlld_100x75x50", "kind": "staggered_box", "solver": "hlld_athena", "nx": 100,
         "ny": 75, "nz": 50, "steps": 40},
        # two populations sharing one field
        {"name": "two_population_128", "kind": "two_population", "solver": "rusanov", "nx": 128, "ny": 128, "nz": 128,
         "steps": 40},
        # local time stepping, two period regions, planned every step
        {"name": "substep_hlld_96", "kind": "substep", "solver": "hlld_athena", "nx": 96, "ny": 96, "nz": 96,
         "steps": 12},
    ]


def _size(rng, lo, hi):
    """An edge between lo and hi, spread over its logarithm; any remainder."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tube", "vortex", "vortex", "blast", "blast", "wind", "ensemble", "adjoint", "staggered",
                       "staggered_box", "two_population", "substep"])
    solver = rng.choice(["rusanov", "hll_athena", "hlld_athena", "hlld_athena", "roe_athena"])
    if kind == "tube":
        return {"kind": kind, "solver": solver, "nx": _size(rng, 100, 8000), "ny": 1, "nz": 1,
                "steps": rng.randint(60, 200)}
    if kind == "vortex":
        return {"kind": kind, "solver": solver, "nx": _size(rng, 64, 1024), "ny": _size(rng, 64, 1024), "nz": 1,
                "steps": rng.randint(20, 60)}
    if kind == "blast":
        return {"kind": kind, "solver": "hlld_athena" if solver == "roe_athena" else solver, "nx": _size(rng, 32, 256),
                "ny": _size(rng, 32, 256), "nz": _size(rng, 32, 256), "steps": rng.randint(10, 20)}
    if kind == "wind":
        return {"kind": kind, "solver": "hll_athena", "nx": _size(rng, 32, 160), "ny": _size(rng, 24, 128),
                "nz": _size(rng, 24, 128), "steps": rng.randint(20, 50)}
    if kind == "ensemble":
        lo = _size(rng, 24, 40)
        return {"kind": kind, "solver": "hll_athena", "boxes": rng.randint(6, 20), "smallest": lo,
                "largest": lo + _size(rng, 16, 64), "steps": rng.randint(30, 60)}
    if kind == "adjoint":
        n = rng.randint(30, 60)
        return {"kind": kind, "solver": rng.choice(["rusanov", "hll_athena", "hlld_athena"]),
                "nx": _size(rng, 64, 300), "ny": _size(rng, 64, 300), "nz": 1, "steps": n,
                "every": rng.choice([7, 10, 15])}
    steps = rng.randint(10, 50)
    if kind == "staggered" or kind == "staggered_box":
        return {"kind": kind, "solver": rng.choice(["hll_athena", "hlld_athena", "hlld_athena"]),
                "nx": _size(rng, 32, 144), "ny": _size(rng, 32, 144), "nz": _size(rng, 32, 144), "steps": steps}
    if kind == "two_population":
        return {"kind": kind, "solver": "rusanov", "nx": _size(rng, 32, 144), "ny": _size(rng, 32, 144),
                "nz": _size(rng, 32, 144), "steps": steps}
    return {"kind": kind, "solver": rng.choice(["hll_athena", "hlld_athena"]), "nx": _size(rng, 32, 110),
            "ny": _size(rng, 32, 110), "nz": _size(rng, 32, 110), "steps": rng.randint(6, 12)}


# ------------------------------------------------------------------ initial states

def _energy(rho, v, p, B, gamma, mu0=1.0):
    return p / (gamma - 1) + 0.5 * rho * (v * v).sum(0) + 0.5 / mu0 * (B * B).sum(0)


def _pack(rho, v, p, B, gamma, mu0=1.0):
    return torch.cat([rho[None], rho * v, _energy(rho, v, p, B, gamma, mu0)[None], B]).contiguous()


def _grid(case):
    """Cell centres in units of the edges, shaped to broadcast over (nz, ny, nx)."""
    c = [(torch.arange(case[a], device=DEV, dtype=torch.float64) + 0.5) / case[a] for a in ("nx", "ny", "nz")]
    return c[0][None, None, :], c[1][None, :, None], c[2][:, None, None]


def _noise(case, rng, amp, modes=4, kmax=2):
    """A smooth periodic field of zero mean: a few random Fourier modes."""
    x, y, z = _grid(case)
    f = torch.zeros((case["nz"], case["ny"], case["nx"]), device=DEV, dtype=torch.float64)
    for _ in range(modes):
        k = [int(v) for v in rng.integers(-kmax, kmax + 1, 3)]
        ph, a = float(rng.uniform(0, 2 * math.pi)), float(rng.normal()) * amp
        f += a * torch.cos(2 * math.pi * (k[0] * x + k[1] * y + k[2] * z) + ph)
    return f


def _smooth(case, rng, amp):
    rho = 1.0 + _noise(case, rng, amp)
    p = 0.6 + _noise(case, rng, amp)
    v = torch.stack([base + _noise(case, rng, amp) for base in (0.1, -0.05, 0.02)])
    B = torch.stack([base + _noise(case, rng, amp) for base in (0.5, 0.3, -0.2)])
    return rho, v, p, B


def _tube(case, rng):
    x, _, _ = _grid(case)
    left = x < 0.5
    s = 1 + 0.02 * rng.uniform(-1, 1, 4)
    left = left.to(torch.float64)
    rho = left * s[0] + (1 - left) * 0.125 * s[1]
    p = left * s[2] + (1 - left) * 0.1 * s[3]
    B = torch.stack([torch.full_like(rho, 0.75), 2 * left - 1, torch.zeros_like(rho)])
    return _pack(rho, torch.zeros_like(B), p, B, 2.0)


def _vortex(case, rng):
    x, y, _ = _grid(case)
    x, y = x + float(rng.uniform()), y + float(rng.uniform())
    tau = 2 * math.pi
    one = torch.ones((1, case["ny"], case["nx"]), device=DEV, dtype=torch.float64)
    rho = 25.0 / (36.0 * math.pi) * (1 + _noise(case, rng, 0.01))
    p = 5.0 / (12.0 * math.pi) * (1 + _noise(case, rng, 0.01))
    v = torch.stack([-torch.sin(tau * y) * one + _noise(case, rng, 0.01),
                     torch.sin(tau * x) * one + _noise(case, rng, 0.01), _noise(case, rng, 0.01)])
    B = torch.stack([-torch.sin(tau * y) * one, torch.sin(2 * tau * x) * one,
                     0.02 + _noise(case, rng, 0.01)]) / math.sqrt(4 * math.pi)
    return _pack(rho, v, p, B, GAMMA)


def _blast(case, rng):
    n = max(case["nx"], case["ny"], case["nz"])
    x, y, z = _grid(case)
    r2 = sum((g - 0.5) ** 2 * (case[a] / n) ** 2 for g, a in ((x, "nx"), (y, "ny"), (z, "nz")))
    p = 0.1 + 9.9 * (r2 < 0.01).to(torch.float64)
    rho = torch.ones_like(p)
    # B0 plus modes transverse to their wave vectors
    B = torch.zeros((3,) + p.shape, device=DEV, dtype=torch.float64)
    B[0:2] += 1 / math.sqrt(2)
    for _ in range(6):
        m = rng.integers(1, 5, 3) * rng.choice([-1, 1], 3)
        k = m * n / np.array([case["nx"], case["ny"], case["nz"]])
        a = np.cross(k, rng.normal(size=3)) * 0.002
        c = torch.cos(2 * math.pi * (int(m[0]) * x + int(m[1]) * y + int(m[2]) * z) + float(rng.uniform(0, 6)))
        for d in range(3):
            B[d] += float(a[d]) * c
    return _pack(rho, torch.zeros_like(B), p, B, GAMMA)


def _wind_states(rng):
    """Inflow (8 values) and interior (8 values) of a solar-wind box, SI units."""
    dens = rng.uniform(2.0, 10.0) * 1e6
    speed = rng.uniform(300.0, 500.0) * 1e3
    d = rng.normal(size=3)
    B = rng.uniform(2.0, 8.0) * 1e-9 * d / np.linalg.norm(d)
    T = 10 ** rng.uniform(5.3, 6.3)
    out = []
    for f, v in ((1.0, speed), (0.25, 0.0)):
        rho, p = f * dens * PROTON, f * dens * BOLTZMANN * T
        e = p / (GAMMA - 1) + 0.5 * rho * v * v + 0.5 / MU0_SI * float(B @ B)
        out.append(np.array([rho, rho * v, 0.0, 0.0, e, *B]))
    return out


def _fill(values, n):
    return torch.tensor(values, device=DEV)[:, None, None, None].expand(8, n[2], n[1], n[0]).contiguous()


def _boxes(case, rng):
    """(edge, inflow, interior) of every box: the edges spread evenly over the range, large and small
    ones mixed; each box with a wind of its own."""
    k, lo, hi = case["boxes"], case["smallest"], case["largest"]
    edges = [lo + (hi - lo) * i // (k - 1) for i in range(k)]
    return [(n,) + tuple(_wind_states(rng)) for n in edges[::2] + edges[1::2]]


def _up(a, d, shift=-1):
    """The value one cell up along axis d (0 x, 1 y, 2 z) on a periodic grid."""
    return torch.roll(a, shift, dims=-1 - d)


def _staggered(case, rng):
    """A smooth state with a divergence-free face field: uniform plus the curl of a potential."""
    L = _lengths(case)
    A = [_noise(case, rng, 0.01) for _ in range(3)]
    faces = []
    for d, base in enumerate((0.3, -0.2, 0.1)):
        a, b = (d + 1) % 3, (d + 2) % 3
        faces.append(base + (_up(A[b], a) - A[b]) / L[a] - (_up(A[a], b) - A[a]) / L[b])
    faces = torch.stack(faces)
    B = torch.stack([0.5 * (faces[d] + _up(faces[d], d)) for d in range(3)])
    rho, v, p, _ = _smooth(case, rng, 0.03)
    return _pack(rho, v, p, B, GAMMA), faces


def _two_population(case, rng):
    rho1, v1, p1, B = _smooth(case, rng, 0.03)
    rho2, v2, _, _ = _smooth(case, rng, 0.03)
    rho2 = 0.5 * rho2
    pb = 0.5 * (B * B).sum(0)
    out = []
    for rho, v, p in ((rho1, v1, p1), (rho2, v2, 0.5 * p1)):
        out += [rho[None], rho * v, (p / (GAMMA - 1) + 0.5 * rho * (v * v).sum(0) + rho / (rho1 + rho2) * pb)[None]]
    return torch.cat(out + [B]).contiguous()


def _lengths(case):
    if case["kind"] in ("wind", "ensemble"):
        return (BOX_CELL,) * 3
    if case["kind"] in ("tube", "vortex", "adjoint"):
        return (1.0 / case["nx"], 1.0 / case["ny"] if case["ny"] > 1 else 1.0, 1.0)
    n = max(case["nx"], case["ny"], case["nz"])
    return (1.0 / n,) * 3


CFL = {"tube": 0.5, "adjoint": 0.25, "wind": 0.5, "ensemble": 0.5}


def _initial(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "wind":
        inflow, interior = _wind_states(rng)
        return inflow, _fill(interior, (case["nx"], case["ny"], case["nz"]))
    make = {"tube": _tube, "vortex": _vortex, "adjoint": _vortex, "blast": _blast, "ensemble": _boxes,
            "staggered": _staggered, "staggered_box": _staggered, "two_population": _two_population,
            "substep": lambda c, r: _pack(*_smooth(c, r, 0.03), GAMMA)}
    return make[kind](case, rng)


def _seed_field(case, seed):
    """The cotangent of the final state of an adjoint run."""
    return np.random.default_rng(seed + 7).normal(size=(8, 1, case["ny"], case["nx"]))


def _exponents(case):
    """Period exponents 0 in the lower half along y, 1 in the upper."""
    e = (torch.arange(case["ny"]) >= case["ny"] // 2).to(torch.int32)
    return e[None, :, None].expand(case["nz"], case["ny"], case["nx"]).contiguous()


def _wall_faces(U, faces, kind):
    """Face arrays with the high walls of a bounded grid (the face that wraps around)."""
    out = []
    for d in range(3):
        f = faces[d]
        out.append(torch.cat([f, f.narrow(2 - d, 0, 1)], dim=2 - d) if kind == "staggered_box" else f)
    return out


def _host(t):
    """A copy in pinned host memory."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h


# ------------------------------------------------------------------ the runs

def _config(case, n, bounds=None, value=None):
    lo, hi = bounds or ((pg.BC_PERIODIC,) * 3, (pg.BC_PERIODIC,) * 3)
    si = case["kind"] in ("wind", "ensemble")
    return pg.Config(n=n, solver=pg.SOLVERS[case["solver"]], cell_length=_lengths(case),
                     adiabatic_index=2.0 if case["kind"] == "tube" else GAMMA,
                     vacuum_permeability=MU0_SI if si else 1.0, time_step_factor=CFL.get(case["kind"], 0.4),
                     bc_lo=lo, bc_hi=hi, value_lo=[value, None, None])


WIND = ((pg.BC_VALUE, pg.BC_COPY, pg.BC_COPY), (pg.BC_COPY,) * 3)
OPEN_X = ((pg.BC_COPY, pg.BC_PERIODIC, pg.BC_PERIODIC), (pg.BC_COPY, pg.BC_PERIODIC, pg.BC_PERIODIC))


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    init = _initial(case, seed)
    if kind == "ensemble":
        s["handle"] = pg.Batch([_config(case, (n,) * 3, WIND, inflow) for n, inflow, _ in init])
        s["in"] = [_host(_fill(interior, (n,) * 3)) for n, _, interior in init]
        s["out"] = [torch.empty(u.shape, dtype=u.dtype, pin_memory=True) for u in s["in"]]
        s["pointers"] = [(ctypes.c_void_p * 8)(*[u[k].data_ptr() for k in range(8)]) for u in s["out"]]
        return s
    n = (case["nx"], case["ny"], case["nz"])
    if kind in ("tube", "vortex", "blast", "wind", "adjoint"):
        value, U = init if kind == "wind" else (None, init)
        s["handle"] = pg.Context(_config(case, n, {"tube": OPEN_X, "wind": WIND}.get(kind), value))
        s["in"] = U
        s["in_ptrs"] = [U[k].data_ptr() for k in range(8)]
        if kind == "adjoint":
            s["seed"] = _seed_field(case, seed)
        else:
            s["out"] = torch.empty_like(U)
            s["out_ptrs"] = [s["out"][k].data_ptr() for k in range(8)]
        return s
    if kind in ("staggered", "staggered_box"):
        U, faces = init
        value = U[:, 0, 0, 0].cpu().numpy() * np.array([1.3, 1.3, 1.3, 1.3, 1, 1, 1, 1])
        box = kind == "staggered_box"
        s["handle"] = pg.StaggeredContext(_config(case, n, WIND if box else None, value if box else None))
        s["in"] = [_host(U)] + [_host(f) for f in _wall_faces(U, faces, kind)]
        s["out"] = [torch.empty(t.shape, dtype=t.dtype, pin_memory=True) for t in s["in"]]
        return s
    s["in"] = _host(init)
    s["out"] = torch.empty(init.shape, dtype=init.dtype, pin_memory=True)
    if kind == "two_population":
        s["handle"] = pg.TwoPopulationContext(n, _lengths(case), solver=pg.SOLVERS[case["solver"]],
                                              adiabatic_index=GAMMA)
        return s
    s["handle"] = pg.SubstepContext(_config(case, n))
    s["handle"].set_state(s["in"].numpy())
    e = _exponents(case).numpy()
    s["handle"].set_exponents(e, e)
    return s


def run(s):
    case, h = s["case"], s["handle"]
    kind, steps = case["kind"], case["steps"]
    if kind in ("tube", "vortex", "blast", "wind"):
        h.set_state_device(s["in_ptrs"])
        h.step(0.0)
        h.steps(steps, T_END)
        h.get_state_device(s["out_ptrs"])
        return s["out"]
    if kind == "ensemble":
        for i, u in enumerate(s["in"]):
            h.set_state(i, u.numpy())
        h.run(steps + 1)
        for i, p in enumerate(s["pointers"]):
            h.L.pamhd_gpu_batch_get_state(h.h, i, p)
        return s["out"]
    if kind == "adjoint":
        h.set_state_device(s["in_ptrs"])
        h.step(0.0)
        grad, _, dts = h.adjoint(steps, case["every"], s["seed"])
        return {"grad": grad, "dt": dts}
    if kind in ("staggered", "staggered_box"):
        h.set_state(s["in"][0].numpy(), [f.numpy() for f in s["in"][1:]])
        h.step(0.0)
        h.steps(steps, T_END)
        h.get_state(out=(s["out"][0].numpy(), [f.numpy() for f in s["out"][1:]]))
        return s["out"]
    if kind == "two_population":
        h.set_state(s["in"].numpy())
        h.run(steps + 1, 0.4, T_END)
        h.get_state(out=s["out"].numpy())
        return s["out"]
    h.set_state(s["in"].numpy())
    h.step(0.0)
    dts = [h.step(T_END)[0] for _ in range(steps)]
    h.get_state(out=s["out"].numpy())
    return {"U": s["out"], "dt": np.array(dts)}


def work(case):
    """Bytes and flops of a pass: every step reads and writes the state once (a step's state does not
    fit on the chip but for the smallest grids), plus the input and the output.  The faces of a step
    are one per cell and active dimension."""
    kind, steps = case["kind"], case["steps"]
    if kind == "ensemble":
        cells = case["boxes"] * ((case["smallest"] + case["largest"]) / 2) ** 3
        dims = 3
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
        dims = sum(1 for a in ("nx", "ny", "nz") if case[a] > 1)
    words = {"staggered": 11, "staggered_box": 11, "two_population": 13}.get(kind, 8)
    flops = dims * FACE_FLOPS[case["solver"]] + CELL_FLOPS
    if kind == "adjoint":
        # forward, then the reverse of every step: states and cotangents read, cotangents written
        return {"bytes": cells * 8.0 * (steps * 5 * words + 3 * words), "flops": cells * steps * 4.0 * flops}
    updates = steps * (1.5 if kind == "substep" else 1.0)
    return {"bytes": cells * 16.0 * words * (updates + 1), "flops": cells * updates * flops}


# ------------------------------------------------------------------ the same runs in plain torch

def _cell(U, d, gamma, mu0):
    """A state seen from a face normal to axis d: conservative values in the face frame, velocity,
    pressure, magnetic pressure and the fast magnetosonic speed."""
    o = [d, (d + 1) % 3, (d + 2) % 3]
    m, b = [U[1 + i] for i in o], [U[5 + i] for i in o]
    rho, E = U[0], U[4]
    v = [x / rho for x in m]
    b2 = b[0] ** 2 + b[1] ** 2 + b[2] ** 2
    pb = b2 / (2 * mu0)
    p = (gamma - 1) * (E - 0.5 * (m[0] * v[0] + m[1] * v[1] + m[2] * v[2]) - pb)
    a2, va2 = gamma * p / rho, b2 / (mu0 * rho)
    root = torch.sqrt((a2 - va2) ** 2 + 4 * a2 * (b[1] ** 2 + b[2] ** 2) / (mu0 * rho))
    return {"rho": rho, "m": m, "E": E, "b": b, "v": v, "p": p, "pb": pb, "cf": torch.sqrt(0.5 * (a2 + va2 + root)),
            "U": [rho] + m + [E] + b}


def _flux(s, mu0):
    b, v, m = s["b"], s["v"], s["m"]
    pt, vb = s["p"] + s["pb"], s["v"][0] * b[0] + s["v"][1] * b[1] + s["v"][2] * b[2]
    return [m[0], m[0] * v[0] + pt - b[0] ** 2 / mu0, m[1] * v[0] - b[0] * b[1] / mu0, m[2] * v[0] - b[0] * b[2] / mu0,
            v[0] * (s["E"] + pt) - b[0] * vb / mu0, torch.zeros_like(pt), v[0] * b[1] - b[0] * v[1],
            v[0] * b[2] - b[0] * v[2]]


def _rusanov(L, R, gamma, mu0):
    s = torch.maximum(L["v"][0].abs(), R["v"][0].abs()) + torch.maximum(L["cf"], R["cf"])
    return [0.5 * (fl + fr) - 0.5 * s * (ur - ul)
            for fl, fr, ul, ur in zip(_flux(L, mu0), _flux(R, mu0), L["U"], R["U"])], s


def _fan(L, R):
    c = torch.maximum(L["cf"], R["cf"])
    return torch.minimum(L["v"][0], R["v"][0]) - c, torch.maximum(L["v"][0], R["v"][0]) + c


def _hll(L, R, gamma, mu0):
    lo, hi = _fan(L, R)
    bm, bp = lo.clamp(max=0.0), hi.clamp(min=0.0)
    F = [(bp * fl - bm * fr + bp * bm * (ur - ul)) / (bp - bm)
         for fl, fr, ul, ur in zip(_flux(L, mu0), _flux(R, mu0), L["U"], R["U"])]
    F[5] = torch.zeros_like(F[5])
    return F, torch.maximum(bm.abs(), bp.abs())


def _hlld(L, R, gamma, mu0):
    """Miyoshi and Kusano, J. Comput. Phys. 208 (2005); the normal field the mean of both sides'."""
    lo, hi = _fan(L, R)
    sub = (lo < 0) & (hi > 0)
    one = torch.ones_like(lo)
    S = [torch.where(sub, lo, -one - L["v"][0].abs() - R["v"][0].abs()),
         torch.where(sub, hi, one + L["v"][0].abs() + R["v"][0].abs())]
    X = [L, R]
    pt = [x["p"] + x["pb"] for x in X]
    sd = [S[i] - X[i]["v"][0] for i in (0, 1)]
    rd = [X[i]["rho"] * sd[i] for i in (0, 1)]
    sm = (sd[1] * R["m"][0] - sd[0] * L["m"][0] - pt[1] + pt[0]) / (rd[1] - rd[0])
    bx = 0.5 * (L["b"][0] + R["b"][0])
    ps = pt[0] + rd[0] * (sm - L["v"][0])
    small = torch.finfo(torch.float64).eps * ps
    rs, w, bs, Us, ss = [], [], [], [], []
    for i in (0, 1):
        x = X[i]
        d = S[i] - sm
        r = torch.where(sub, rd[i] / d, one)
        den = rd[i] * d - bx * bx / mu0
        keep = den.abs() < small
        den = torch.where(keep, one, den)
        t1, t2 = bx * (sm - x["v"][0]) / (mu0 * den), (rd[i] * sd[i] - bx * bx / mu0) / den
        wi = [torch.where(keep, x["v"][j], x["v"][j] - x["b"][j] * t1) for j in (1, 2)]
        bi = [torch.where(keep, x["b"][j], x["b"][j] * t2) for j in (1, 2)]
        vb = x["v"][0] * x["b"][0] + x["v"][1] * x["b"][1] + x["v"][2] * x["b"][2]
        e = (sd[i] * x["E"] - pt[i] * x["v"][0] + ps * sm
             + bx / mu0 * (vb - sm * bx - wi[0] * bi[0] - wi[1] * bi[1])) / d
        rs.append(r); w.append(wi); bs.append(bi)
        Us.append([r, r * sm, r * wi[0], r * wi[1], e, bx, bi[0], bi[1]])
        ss.append(sm + (2 * i - 1) * bx.abs() / torch.sqrt(mu0 * r))
    q = [torch.sqrt(r) for r in rs]
    sg, rm = torch.where(bx > 0, 1.0, -1.0), math.sqrt(mu0)
    vv = [(q[0] * w[0][j] + q[1] * w[1][j] + sg / rm * (bs[1][j] - bs[0][j])) / (q[0] + q[1]) for j in (0, 1)]
    bb = [(q[0] * bs[1][j] + q[1] * bs[0][j] + sg * rm * q[0] * q[1] * (w[1][j] - w[0][j])) / (q[0] + q[1])
          for j in (0, 1)]
    vb2 = sm * bx + vv[0] * bb[0] + vv[1] * bb[1]
    two = 0.5 * bx * bx >= small
    out = []
    for i in (0, 1):
        vb1 = sm * bx + w[i][0] * bs[i][0] + w[i][1] * bs[i][1]
        e2 = Us[i][4] + (2 * i - 1) * q[i] * sg / rm * (vb1 - vb2)
        U2 = [rs[i], rs[i] * sm, rs[i] * vv[0], rs[i] * vv[1], e2, bx, bb[0], bb[1]]
        F = _flux(X[i], mu0)
        star = [f + S[i] * (a - u) for f, a, u in zip(F, Us[i], X[i]["U"])]
        dbl = [f + ss[i] * (torch.where(two, c, a) - a) for f, a, c in zip(star, Us[i], U2)]
        out.append((F, star, dbl))
    FL, FR = out
    left = sm >= 0
    F = []
    for v in range(8):
        inner = torch.where(ss[0] >= 0, FL[1][v], torch.where(left, FL[2][v],
                            torch.where(ss[1] > 0, FR[2][v], FR[1][v])))
        F.append(torch.where(lo >= 0, FL[0][v], torch.where(hi <= 0, FR[0][v], inner)))
    F[5] = torch.zeros_like(F[5])
    return F, torch.maximum(lo.abs(), hi.abs())


def _roe(L, R, gamma, mu0):
    """Roe's solver with the eigenvectors of Stone et al., ApJS 178 (2008), B17-B29 (mu0 1)."""
    g1, g2 = gamma - 1, gamma - 2
    bx = 0.5 * (L["b"][0] + R["b"][0])
    ql, qr = torch.sqrt(L["rho"]), torch.sqrt(R["rho"])
    i = 1 / (ql + qr)
    v = [(ql * a + qr * b) * i for a, b in zip(L["v"], R["v"])]
    b2, b3 = ((qr * L["b"][j] + ql * R["b"][j]) * i for j in (1, 2))
    rho = ql * qr
    x = 0.5 * ((L["b"][1] - R["b"][1]) ** 2 + (L["b"][2] - R["b"][2]) ** 2) * i * i
    y = 0.5 * (L["rho"] + R["rho"]) / rho
    U, F, pb = [], [], []
    for s in (L, R):
        m, b, w = s["m"], s["b"], s["v"]
        pm = 0.5 * (bx * bx + b[1] ** 2 + b[2] ** 2)
        pb.append(pm)
        U.append([s["rho"], *m, s["E"], b[1], b[2]])
        F.append([m[0], m[0] * w[0] + s["p"] + pm - bx * bx, m[0] * w[1] - bx * b[1], m[0] * w[2] - bx * b[2],
                  (s["E"] + s["p"] + pm) * w[0] - bx * (bx * w[0] + b[1] * w[1] + b[2] * w[2]),
                  b[1] * w[0] - bx * w[1], b[2] * w[0] - bx * w[2]])
    h = ((L["E"] + L["p"] + pb[0]) / ql + (R["E"] + R["p"] + pb[1]) / qr) * i
    vsq, bt2 = v[0] ** 2 + v[1] ** 2 + v[2] ** 2, b2 * b2 + b3 * b3
    ys = g1 - g2 * y
    va2, ct2 = bx * bx / rho, ys * bt2 / rho
    hp = h - va2 - bt2 / rho
    a2 = (g1 * (hp - 0.5 * vsq) - g2 * x).clamp(min=torch.finfo(torch.float64).eps)
    root = torch.sqrt((va2 + ct2 - a2) ** 2 + 4 * a2 * ct2)
    cf2 = 0.5 * (va2 + ct2 + a2 + root)
    cs2 = a2 * va2 / cf2
    cf, cs, a, va, bt = (torch.sqrt(t) for t in (cf2, cs2, a2, va2, bt2))
    n2, n3 = torch.where(bt > 0, b2 / bt, 1.0), torch.where(bt > 0, b3 / bt, 0.0)
    n2, n3 = torch.nan_to_num(n2, nan=1.0), torch.nan_to_num(n3, nan=0.0)
    rys = torch.sqrt(ys)
    s2, s3 = n2 / rys, n3 / rys
    d = torch.where(cf2 > cs2, cf2 - cs2, torch.ones_like(cf2))
    af = torch.sqrt(((a2 - cs2) / d).clamp(min=0.0, max=1.0))
    as_ = torch.sqrt(((cf2 - a2) / d).clamp(min=0.0, max=1.0))
    sg, rq = torch.where(bx > 0, 1.0, -1.0), torch.sqrt(rho)
    qf, qs = cf * af * sg, cs * as_ * sg
    pf, ps = a * af / rq, a * as_ / rq
    bts = torch.sqrt(ys) * bt
    bsq = s2 * s2 + s3 * s3
    vbet = v[1] * s2 + v[2] * s3
    zero, one = torch.zeros_like(rho), torch.ones_like(rho)
    lam = [v[0] - cf, v[0] - va, v[0] - cs, v[0], v[0] + cs, v[0] + va, v[0] + cf]
    Rm = {}
    for w, sgn in ((0, -1), (6, 1)):
        Rm[w] = [af, af * lam[w], af * v[1] - sgn * qs * s2, af * v[2] - sgn * qs * s3,
                 af * (hp + sgn * v[0] * cf) - sgn * qs * vbet + ps * bts * bsq, ps * s2, ps * s3]
    for w, sgn in ((2, -1), (4, 1)):
        Rm[w] = [as_, as_ * lam[w], as_ * v[1] + sgn * qf * s2, as_ * v[2] + sgn * qf * s3,
                 as_ * (hp + sgn * v[0] * cs) + sgn * qf * vbet - pf * bts * bsq, -pf * s2, -pf * s3]
    for w, sgn in ((1, -1), (5, 1)):
        Rm[w] = [zero, zero, sgn * n3, -sgn * n2, sgn * (v[1] * n3 - v[2] * n2), -n3 * sg / rq, n2 * sg / rq]
    Rm[3] = [one, v[0], v[1], v[2], 0.5 * vsq + g2 * x / g1, zero, zero]
    N = 0.5 / a2
    t2, t3 = s2 / bsq, s3 / bsq
    vq = v[1] * t2 + v[2] * t3
    Lm = {}
    for w, sgn in ((0, -1), (6, 1)):
        Lm[w] = [N * (af * g1 * (vsq - hp) + af * cf * (cf - sgn * v[0]) + sgn * qs * vq - ps * bts),
                 N * (-af * g1 * v[0] + sgn * af * cf), N * (-af * g1 * v[1] - sgn * qs * t2),
                 N * (-af * g1 * v[2] - sgn * qs * t3), N * af * g1, N * (ps * rho * t2 - af * g1 * b2),
                 N * (ps * rho * t3 - af * g1 * b3)]
    for w, sgn in ((2, -1), (4, 1)):
        Lm[w] = [N * (as_ * g1 * (vsq - hp) + as_ * cs * (cs - sgn * v[0]) - sgn * qf * vq + pf * bts),
                 N * (-as_ * g1 * v[0] + sgn * as_ * cs), N * (-as_ * g1 * v[1] + sgn * qf * t2),
                 N * (-as_ * g1 * v[2] + sgn * qf * t3), N * as_ * g1, N * (-pf * rho * t2 - as_ * g1 * b2),
                 N * (-pf * rho * t3 - as_ * g1 * b3)]
    for w, sgn in ((1, -1), (5, 1)):
        Lm[w] = [-sgn * 0.5 * (v[1] * n3 - v[2] * n2), zero, sgn * 0.5 * n3, -sgn * 0.5 * n2, zero,
                 -0.5 * rq * n3 * sg, 0.5 * rq * n2 * sg]
    M = 2 * N * g1
    Lm[3] = [1 - M * (0.5 * vsq - g2 * x / g1), M * v[0], M * v[1], M * v[2], -M, M * b2, M * b3]
    out = [0.5 * (p + q) for p, q in zip(*F)]
    for w in range(7):
        strength = sum(Lm[w][r] * (U[1][r] - U[0][r]) for r in range(7))
        out = [o - 0.5 * strength * lam[w].abs() * Rm[w][r] for r, o in enumerate(out)]
    out = [torch.where(lam[0] >= 0, p, torch.where(lam[6] <= 0, q, o)) for o, p, q in zip(out, *F)]
    lo, hi = _fan(L, R)
    return out[:5] + [torch.zeros_like(rho)] + out[5:], torch.maximum(lo.abs(), hi.abs())


SOLVE = {"rusanov": _rusanov, "hll_athena": _hll, "hlld_athena": _hlld, "roe_athena": _roe}


def _face(case, UL, UR, d):
    """Flux (xyz components) and signal speed of the faces between two arrays of states."""
    g = 2.0 if case["kind"] == "tube" else GAMMA
    mu0 = MU0_SI if case["kind"] in ("wind", "ensemble") else 1.0
    F, s = SOLVE[case["solver"]](_cell(UL, d, g, mu0), _cell(UR, d, g, mu0), g, mu0)
    o = [d, (d + 1) % 3, (d + 2) % 3]
    out = [None] * 8
    out[0], out[4] = F[0], F[4]
    for i in range(3):
        out[1 + o[i]], out[5 + o[i]] = F[1 + i], F[5 + i]
    return torch.stack(out), s


def _padded(U, d, kind, inflow):
    ax = 3 - d
    lo, hi = U.narrow(ax, U.shape[ax] - 1, 1), U.narrow(ax, 0, 1)
    if kind in ("wind", "ensemble") or (kind == "tube" and d == 0):
        lo, hi = hi, lo
        if inflow is not None and d == 0:
            lo = inflow[:, None, None, None].expand(lo.shape)
    return torch.cat([lo, U, hi], dim=ax)


def _advance(case, U, dt, inflow=None):
    """One cell-centred step; returns the new state and the next step's limit."""
    L, new, limit = _lengths(case), U, None
    for d in range(3):
        if U.shape[3 - d] == 1:
            continue
        P = _padded(U, d, case["kind"], inflow)
        n = P.shape[3 - d] - 1
        F, s = _face(case, P.narrow(3 - d, 0, n), P.narrow(3 - d, 1, n), d)
        new = new + dt / L[d] * (F.narrow(3 - d, 0, n - 1) - F.narrow(3 - d, 1, n - 1))
        top = s.max()
        if inflow is not None and d > 0:   # faces between the inflow ghosts
            w = inflow[:, None]
            top = torch.maximum(top, _face(case, w, w, d)[1].max())
        lim = CFL.get(case["kind"], 0.4) * L[d] / top
        limit = lim if limit is None else torch.minimum(limit, lim)
    return new, limit


def _march(case, U, steps, inflow=None):
    dt, states, dts = torch.zeros((), device=DEV, dtype=torch.float64), [U], []
    for n in range(steps + 1):
        dts.append(dt)
        U, dt = _advance(case, U, dt, inflow)
        if case["kind"] == "adjoint":
            states.append(U)
    return U, states, dts


def _adjoint(case, U, seed):
    _, states, dts = _march(case, U, case["steps"])
    lam = torch.from_numpy(_seed_field(case, seed)).to(DEV)
    for n in range(case["steps"], 0, -1):
        V = states[n].detach().requires_grad_(True)
        with torch.enable_grad():
            W, _ = _advance(case, V, dts[n])
        lam, = torch.autograd.grad(W, V, lam)
    return {"grad": lam, "dt": torch.stack(dts[1:])}


def _march_staggered(case, U, Bf, steps):
    L = _lengths(case)
    area = (L[1] * L[2], L[0] * L[2], L[0] * L[1])
    dt = torch.zeros((), device=DEV, dtype=torch.float64)
    for _ in range(steps + 1):
        F, limit = [], None
        for d in range(3):
            f, s = _face(case, _up(U, d, 1), U, d)
            F.append(f)
            lim = 0.4 * L[d] / s.max()
            limit = lim if limit is None else torch.minimum(limit, lim)
        for d in range(3):
            U = U + dt / L[d] * (F[d] - _up(F[d], d))
        new = []
        for d in range(3):
            # a quarter of each edge's electric field from each of the four fluxes around it
            a, b = (d + 1) % 3, (d + 2) % 3
            fa, fb = F[d][5 + a], F[d][5 + b]
            ga, gb = F[a][5 + d], F[b][5 + d]
            ga, gb = ga + _up(ga, d, 1), gb + _up(gb, d, 1)
            change = L[b] * (_up(fa, a) - _up(fa, a, 1) - _up(ga, a) + ga) \
                + L[a] * (_up(fb, b) - _up(fb, b, 1) - _up(gb, b) + gb)
            new.append(Bf[d] + dt / 4 * change / area[d])
        Bf = torch.stack(new)
        B = torch.stack([0.5 * (Bf[d] + _up(Bf[d], d)) for d in range(3)])
        E = U[4] + 0.5 * ((B * B).sum(0) - (U[5:8] ** 2).sum(0))
        U = torch.cat([U[:4], E[None], B])
        dt = limit
    return [U] + [Bf[d] for d in range(3)]


def _march_two(case, U, steps):
    L = _lengths(case)
    limit = 0.0
    for _ in range(steps + 1):
        dt = 0.4 * limit
        T = torch.cat([U[:5] + U[5:10], U[10:13]])
        f1 = U[0] / T[0]
        new, limit = U, None
        for d in range(3):
            TL = _up(T, d, 1)
            a, b = _cell(TL, d, GAMMA, 1.0), _cell(T, d, GAMMA, 1.0)
            c = torch.maximum(a["cf"], b["cf"])
            s = torch.maximum(a["v"][0].abs() + c, b["v"][0].abs() + c)
            o = [d, (d + 1) % 3, (d + 2) % 3]

            def xyz(F):
                r = [None] * 8
                r[0], r[4] = F[0], F[4]
                for i in range(3):
                    r[1 + o[i]], r[5 + o[i]] = F[1 + i], F[5 + i]
                return torch.stack(r)

            neg = 0.5 * (xyz(_flux(a, 1.0)) + s * TL)
            pos = 0.5 * (xyz(_flux(b, 1.0)) - s * T)
            g1 = _up(f1, d, 1)
            G = torch.cat([g1 * neg[:5] + f1 * pos[:5], (1 - g1) * neg[:5] + (1 - f1) * pos[:5], neg[5:] + pos[5:]])
            new = new + dt / L[d] * (G - _up(G, d))
            lim = L[d] / s.max()
            limit = lim if limit is None else torch.minimum(limit, lim)
        U = new
    return U


def _march_substeps(case, U, steps):
    L = _lengths(case)
    e = _exponents(case).to(DEV)
    period = 2 ** e
    M = period.clone()
    for off in [(x, y, z) for x in (-1, 0, 1) for y in (-1, 0, 1) for z in (-1, 0, 1)]:
        if sum(1 for v in off if v) in (1, 2):
            M = torch.minimum(M, torch.roll(period, off, dims=(-1, -2, -3)))
    dts, speed = [], None
    for n in range(steps + 1):
        if n == 0:
            sub, last = torch.zeros((), device=DEV, dtype=torch.float64), 1
        else:
            limit = torch.stack([torch.minimum(0.4 * L[d] / speed[d], 0.4 * L[d] / _up(speed[d], d, 1))
                                 for d in range(3)]).amin(0)
            sub, last = (limit / period).min(), int(period.max())
        acc = torch.zeros_like(U)
        per, reach = (torch.ones_like(period), torch.ones_like(M)) if n == 0 else (period, M)
        for s in range(1, last + 1):
            on = (s % reach == 0)
            speed = [] if speed is None or len(speed) < 3 else speed
            for d in range(3):
                F, v = _face(case, U, _up(U, d), d)   # the cell's +d face
                F = torch.where(on, sub * reach * F, 0.0) / L[d]
                acc = acc - F + _up(F, d, 1)
                if len(speed) < 3:
                    speed.append(v)
                else:
                    speed[d] = torch.where(on, v, speed[d])
            due = (s % per == 0)
            U = torch.where(due, U + acc, U)
            acc = torch.where(due, 0.0, acc)
        dts.append(sub * last)
    return {"U": U, "dt": torch.stack(dts[1:])}


@torch.no_grad()
def exact(case, seed):
    kind, steps = case["kind"], case["steps"]
    init = _initial(case, seed)
    if kind == "ensemble":
        # the persistent run's first step is the priming step
        return [_march(case, _fill(u, (n,) * 3), steps, torch.tensor(v, device=DEV))[0] for n, v, u in init]
    if kind == "wind":
        return _march(case, init[1], steps, torch.tensor(init[0], device=DEV))[0]
    if kind == "adjoint":
        return _adjoint(case, init, seed)
    if kind == "staggered":
        return _march_staggered(case, init[0], init[1], steps)
    if kind == "staggered_box":
        return None     # its layer of boundary cells and wall faces: several hundred cell-by-cell rules
    if kind == "two_population":
        return _march_two(case, init, steps)
    if kind == "substep":
        return _march_substeps(case, init, steps)
    return _march(case, init, steps)[0]
