"""Performance cases: what a program built on this library has it do, through
the C ABI (include/bcg.h, by its ctypes binding) and the Python classes over
it, from a colony of a thousand cells to the 1M-cell workload.

  steps        the host time loop (bcg_sim_run, the benchmark cadence): a
               colony enters as host records, is stepped (MoveCell, GrowCell,
               divisions and, with vcycles > 0, one agar solve a step) and
               goes back to the host
  python_steps the same mechanics through the Colony class, a call a phase
  update       the reference's UpdateFlag block on a standing colony: density
               chain, nutrient update ([agar solve + 200 sweeps] x units),
               neighbour rebuild, height chain, and the fields read back
  agar         agar time steps alone (fixed V-cycles, or to a tolerance in
               FP64 or mixed precision), and the solution read back
  steady       the steady glucose field and the gradients of a loss on it
  ensemble     several colonies of uneven size stepped together

Colonies are "packed" (layers of touching cells, as a grown colony is) or
"loose" (random sequential placement).  Grids are the named workloads' or
the ensemble member's grid for the colony's size with a chosen agar depth.
"""
import ctypes
import math

import numpy as np
import torch

from baccolonygrowth_b200 import _abi, params as _params
from baccolonygrowth_b200.colony import Colony, Rng, depleted_wall, packed_colony, synth_colony
from baccolonygrowth_b200.steady import Steady, synthetic_problem

F = _abi.FIELDS
WALLS = ("WALLF_CARBON", "WALLF_OXYGEN", "WALLF_ACETATE")
ENV = ("ENV_CARBON", "ENV_OXYGEN", "ENV_ACETATE", "ENV_WASTE", "ENV_GROWTH1", "ENV_PH")
SURFACE = ("ROUGH_DENSITY", "DENSITY_SHIFT", "HEIGHT", "NORMAL_X", "NORMAL_Z")
AGAR = ("AGARF_CARBON", "AGARF_OXYGEN", "AGARF_ACETATE")
SOLUTION = ("MG_SOL_CARBON", "MG_SOL_OXYGEN", "MG_SOL_ACETATE")
RECORD = ("p", "q", "length", "ldiv", "growth_rate", "velocity", "angular_velocity", "dyn_fric", "sta_fric",
          "time_p", "time_q", "age_p", "age_q", "type", "ancestor")
THETA = (0.8, 0.3, 1.0, 0.05)      # d_agar, d_colony, vmax, km of the steady field


def listed():
    return [
        # a young colony stepped from Python, a call a phase: the smallest
        # calls, latency alone
        {"name": "python_1k", "kind": "python_steps", "n": 1000, "colony": "loose", "grid": "small_4k", "steps": 10},
        # the shipped small simulation's size in the host loop: launches and
        # host round trips count
        {"name": "steps_4k", "kind": "steps", "n": 4096, "colony": "loose", "grid": "small_4k", "steps": 20,
         "vcycles": 1, "tuned": False, "stress": False},
        # an ordinary colony of an odd size on a grid made for it, left at
        # the library's own kernel shapes
        {"name": "steps_50k", "kind": "steps", "n": 50021, "colony": "packed", "grid": "member", "rows": 128, "levels": 2,
         "steps": 20, "vcycles": 1, "tuned": False, "stress": False},
        # the 1M-cell workload, tuned once as bench.py does: the largest
        {"name": "steps_1m", "kind": "steps", "n": 1048576, "colony": "packed", "grid": "mixed_1m", "steps": 20,
         "vcycles": 1, "tuned": True, "stress": False},
        # mechanics between two field updates of a dense mid-size colony, and
        # the stress diagnostics of its output step
        {"name": "mechanics_262k", "kind": "steps", "n": 262144, "colony": "packed", "grid": "scale_262k", "steps": 20,
         "vcycles": 0, "tuned": False, "stress": True},
        # the field update of the small simulation
        {"name": "update_4k", "kind": "update", "n": 4096, "colony": "loose", "grid": "small_4k", "units": 8, "agar": True},
        # ... of an ordinary colony of an odd size
        {"name": "update_33k", "kind": "update", "n": 33333, "colony": "packed", "grid": "member", "rows": 64, "levels": 2,
         "units": 4, "agar": True},
        # ... of the 1M-cell workload, whose agar stays on the device until an
        # output step
        {"name": "update_1m", "kind": "update", "n": 1048576, "colony": "packed", "grid": "mixed_1m", "units": 1,
         "agar": False},
        # the agar field on the 262k grid stepped to a tolerance in mixed
        # precision, and read
        {"name": "agar_262k", "kind": "agar", "n": 65536, "colony": "packed", "grid": "scale_262k", "solves": 4,
         "precision": 32},
        # the inverse problem's inner loop at its configured size: forward
        # solve and gradients
        {"name": "steady_129", "kind": "steady", "nx": 129, "nz": 65, "n": 50000},
        # ... on a finer grid
        {"name": "steady_513", "kind": "steady", "nx": 513, "nz": 257, "n": 200000},
        # parameter sweeps: colonies of uneven size advanced together
        {"name": "ensemble_16", "kind": "ensemble", "members": 16, "lo": 1000, "hi": 30000, "steps": 5, "vcycles": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("python_steps", "steps", "steps", "update", "update", "agar", "steady", "ensemble"))
    if kind == "python_steps":
        return {"kind": kind, "n": _log(rng, 200, 4096), "colony": "loose", "grid": "small_4k", "steps": rng.randint(3, 12)}
    if kind == "steps":
        n = _log(rng, 500, 1000000)
        return {"kind": kind, "n": n, "colony": "packed" if n > 20000 else rng.choice(("packed", "loose")),
                "grid": "member", "rows": rng.choice((32, 64, 128, 256)), "levels": rng.choice((2, 3)),
                "steps": rng.randint(5, 20), "vcycles": rng.choice((0, 1, 1, 2)), "tuned": rng.random() < 0.3,
                "stress": rng.random() < 0.4}
    if kind == "update":
        n = _log(rng, 500, 400000)
        return {"kind": kind, "n": n, "colony": "packed" if n > 20000 else rng.choice(("packed", "loose")),
                "grid": "member", "rows": rng.choice((32, 64, 128)), "levels": rng.choice((2, 3)),
                "units": rng.randint(1, 8 if n < 50000 else 2), "agar": n < 50000}
    if kind == "agar":
        return {"kind": kind, "n": _log(rng, 1000, 60000), "colony": "packed", "grid": "member",
                "rows": rng.choice((32, 64, 128, 256)), "levels": rng.choice((2, 3)), "solves": rng.randint(1, 6),
                "precision": rng.choice((0, 32, 64))}
    if kind == "steady":
        a = rng.randint(5, 9)
        return {"kind": kind, "nx": 2 ** a + 1, "nz": 2 ** rng.randint(4, a) + 1, "n": _log(rng, 100, 200000)}
    lo = _log(rng, 500, 2000)
    return {"kind": kind, "members": rng.randint(2, 20), "lo": lo, "hi": _log(rng, 4000, 30000), "steps": rng.randint(2, 6),
            "vcycles": rng.choice((0, 1))}


# ---------------------------------------------------------------------------
def _check(rc, what):
    _abi.check(rc, what)


def _member(n, rows, levels):
    p = _params.ensemble_member(n)
    p.box_z_agar, p.max_levels_mg = rows, levels
    return _params.finalize(p)


def _problem(c, seed):
    """Params and cell records of a case."""
    n = c["n"]
    if c["grid"] == "member":
        aspect, p = 1.0 / 20.0, _member(n, c["rows"], c["levels"])
    else:
        aspect, p = _params.WORKLOADS[c["grid"]][1], _params.workload_params(c["grid"])
    if c["colony"] == "packed":
        w, h = _params.dome_size(n, aspect, 0.9)
        return p, packed_colony(n, w, h, seed=seed)
    w, h = _params.dome_size(n, aspect)
    return p, synth_colony(n, w, h, seed=seed, div_phase_spread=1.0)


def _depletion(seed):
    """How far the colony has used up the nutrients under it."""
    r = np.random.default_rng(seed)
    return {"depth_c": r.uniform(0.3, 0.9), "depth_o": r.uniform(0.3, 0.9), "acetate": r.uniform(0.5, 4.0)}


def _pinned(shape, dtype):
    dtype = np.dtype(dtype)
    count = int(np.prod(shape))
    t = torch.empty(max(count, 1) * dtype.itemsize, dtype=torch.uint8, pin_memory=True)
    return t.numpy()[: count * dtype.itemsize].view(dtype).reshape(shape)


class _Fields:
    """Field reads of a context into buffers kept for them."""

    def __init__(self, ctx, wanted):
        self.lib, self.ctx, self.buf = _abi.load(), ctx, {}
        for name, level in wanted:
            n = ctypes.c_size_t()
            _check(self.lib.bcg_field_size(ctx, F[name], level, ctypes.byref(n)), name)
            self.buf[name, level] = _pinned((n.value,), np.float64)

    def read(self):
        out = {}
        for (name, level), b in self.buf.items():
            _check(self.lib.bcg_get_field(self.ctx, F[name], level, _abi.ptr(b, ctypes.c_double), b.size), name)
            out["%s_%d" % (name, level)] = b
        return out


class _Sim:
    """A bcg_sim in the benchmark cadence with its host records."""

    def __init__(self, p, cells, seed, vcycles, tuned):
        self.lib, self.p = _abi.load(), p
        self.h = ctypes.c_void_p()
        self.cells = _pinned((len(cells),), _abi.CELL_DTYPE)
        self.cells[:] = cells
        self.out = _pinned((p.max_cells,), _abi.CELL_DTYPE)      # room for the divisions to come
        self.out[:] = np.zeros((), _abi.CELL_DTYPE)
        _check(self.lib.bcg_sim_create(ctypes.byref(p), _abi.ptr(self.cells), len(cells), seed & 0x7fffffff, 0,
                                       ctypes.byref(self.h)), "bcg_sim_create")
        _check(self.lib.bcg_sim_set_step_mode(self.h, 0, vcycles), "bcg_sim_set_step_mode")
        self.ctx = self.lib.bcg_sim_ctx(self.h)
        growth = np.full(p.box_x * p.box_z, 0.9)      # a colony in steady supply
        self.set("ENV_GROWTH1", growth)
        _check(self.lib.bcg_update_density(self.ctx), "bcg_update_density")
        inside = np.zeros(p.box_x * p.box_z)
        _check(self.lib.bcg_get_field(self.ctx, F["INSIDE"], 0, _abi.ptr(inside, ctypes.c_double), inside.size), "INSIDE")
        for name, v in zip(WALLS, depleted_wall(p, inside, **_depletion(seed))):
            self.set(name, v)
        _check(self.lib.bcg_rebuild_neighbours(self.ctx), "bcg_rebuild_neighbours")
        if tuned:
            for what in ("SMOOTHER", "FORCE_GROUP"):
                _check(self.lib.bcg_autotune(self.ctx, _abi.TUNE[what], None), "bcg_autotune")
        self.walls = _Fields(self.ctx, [(w, l) for w in WALLS for l in range(p.max_levels_mg)]) if vcycles else None

    def set(self, name, values):
        v = np.ascontiguousarray(values, dtype=np.float64)
        _check(self.lib.bcg_set_field(self.ctx, F[name], 0, _abi.ptr(v, ctypes.c_double), v.size), name)

    def load(self):
        """The colony as host records to the device, and its lists."""
        _check(self.lib.bcg_upload_cells(self.ctx, _abi.ptr(self.cells), len(self.cells)), "bcg_upload_cells")
        _check(self.lib.bcg_rebuild_neighbours(self.ctx), "bcg_rebuild_neighbours")

    def records(self):
        n = ctypes.c_int()
        _check(self.lib.bcg_download_cells(self.ctx, _abi.ptr(self.out), len(self.out), ctypes.byref(n)), "bcg_download_cells")
        out = {k: self.out[k] for k in RECORD}
        out["cells"] = n.value
        if self.walls:
            out.update(self.walls.read())
        return out

    def __del__(self):
        if self.h:
            self.lib.bcg_sim_destroy(self.h)
            self.h = ctypes.c_void_p()


class _State:
    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        e = self.__dict__.get("ensemble")
        if e:
            _abi.load().bcg_ensemble_destroy(e)


def _ensemble_sizes(c, seed):
    """Sizes of the members: fixed by the case, spread over their logarithm."""
    m = c["members"]
    return [int(round(c["lo"] * (c["hi"] / c["lo"]) ** (j / max(1, m - 1)))) | 1 for j in range(m)]


def _steady_problem(c, seed):
    nx, nz = c["nx"], c["nz"]
    nz_agar = (nz + 1) // 2
    cells, w, _ = synthetic_problem(nx, nz, nz_agar, 2.0, c["n"], seed)
    g = np.random.default_rng(seed + 1).standard_normal((nz, nx)) / (nx * nz)
    return dict(nx=nx, nz=nz, nz_agar=nz_agar, h=2.0, c0=20.0), cells, w, g


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "steady":
        grid, cells, w, g = _steady_problem(c, seed)
        s = Steady(max_cells=len(cells), **grid)
        s.set_cells(cells)
        return _State(case=c, solver=s, w=w, g=g)
    if kind == "ensemble":
        sims = []
        for j, n in enumerate(_ensemble_sizes(c, seed)):
            p, cells = _problem({"n": n, "grid": "member", "rows": 64, "levels": 2, "colony": "packed"}, seed + 1000 * j)
            sims.append(_Sim(p, cells, seed + j, c["vcycles"], False))
        e = ctypes.c_void_p()
        arr = (ctypes.c_void_p * len(sims))(*[s.h.value for s in sims])
        _check(_abi.load().bcg_ensemble_create(arr, len(sims), ctypes.byref(e)), "bcg_ensemble_create")
        return _State(case=c, sims=sims, ensemble=e)
    p, cells = _problem(c, seed)
    if kind == "steps":
        s = _Sim(p, cells, seed, c["vcycles"], c["tuned"])
        stress = _pinned((p.max_cells, 5), np.float64) if c["stress"] else None
        if stress is not None:
            stress[:] = 0.0
        return _State(case=c, sim=s, stress=stress)
    col = Colony(p, cells)
    if kind == "python_steps":
        col.set_field("ENV_GROWTH1", np.full(p.box_x * p.box_z, 0.9))
        col.update_density()
        return _State(case=c, col=col, cells=cells, rng=Rng(seed & 0x7fffffff), out=np.zeros(p.max_cells, _abi.CELL_DTYPE))
    levels = range(p.max_levels_mg)
    if kind == "update":
        col.initial_density()
        col.nutrient_update(2)                 # the fields of a running simulation
        wanted = [(f, 0) for f in ENV + SURFACE] + [(f, l) for f in WALLS + (AGAR if c["agar"] else ()) for l in levels]
        return _State(case=c, col=col, fields=_Fields(col.h, wanted))
    col.update_density()
    col.deplete_wall(**_depletion(seed))
    return _State(case=c, col=col, fields=_Fields(col.h, [(f, l) for f in SOLUTION + WALLS for l in levels]))


def run(state):
    c, kind = state.case, state.case["kind"]
    lib = _abi.load()
    if kind == "steps":
        s = state.sim
        s.load()
        _check(lib.bcg_sim_run(s.h, c["steps"]), "bcg_sim_run")
        out = s.records()
        if state.stress is not None:
            _check(lib.bcg_mean_stress(s.ctx, _abi.ptr(state.stress, ctypes.c_double), None, None), "bcg_mean_stress")
            out["stress"] = state.stress
        return out
    if kind == "python_steps":
        col = state.col
        col.upload(state.cells)
        col.rebuild_neighbours()
        dt = col.params.dt
        for k in range(c["steps"]):
            col.step(dt, k * dt, state.rng)
        cells = col.cells()
        state.out[: len(cells)] = cells
        return dict({k: state.out[k] for k in RECORD}, cells=len(cells))
    if kind == "update":
        col = state.col
        col.update_density()
        col.nutrient_update(c["units"])
        col.rebuild_neighbours()
        col.update_height()
        return state.fields.read()
    if kind == "agar":
        for _ in range(c["solves"]):
            if c["precision"]:
                state.col.mg_solve_tol(1e-8, c["precision"], 50)
            else:
                state.col.mg_solve()
        return state.fields.read()
    if kind == "steady":
        C = state.solver.solve(THETA, state.w)
        grad_theta, grad_w = state.solver.vjp(state.g)
        return {"C": C, "grad_theta": grad_theta, "grad_w": grad_w}
    for s in state.sims:
        s.load()
    _check(lib.bcg_ensemble_run(state.ensemble, c["steps"]), "bcg_ensemble_run")
    out = {}
    for j, s in enumerate(state.sims):
        r = s.records()
        out["%d" % j] = {k: r[k] for k in ("p", "q", "velocity")}
    return out


# ---------------------------------------------------------------------------
def _solve_bytes(p, vcycles):
    """Bytes one Multigrid::solve cannot do without, FP64: per point and
    species the right-hand side and the correction read and the correction
    written once before and once after the coarse correction (48), the
    transfers (24), and per solve the residual and the update (56)."""
    d0, total = 1 << p.max_levels_mg, 0.0
    for l in range(p.mg_levels):
        nx = min(p.box_x * d0 // (1 << l) // 2, p.box_x)
        nz = min(p.box_z_agar * d0 // (1 << l) // 2, p.box_z_agar)
        pts = 3 * (nx + 1) * (nz + 1)
        total += vcycles * 72.0 * pts + (56.0 * pts if l < p.max_levels_mg else 16.0 * pts)
    return total


def _work_params(c):
    if c["grid"] == "member":
        return _member(c["n"], c["rows"], c["levels"])
    return _params.workload_params(c["grid"])


def work(case):
    c, kind = case, case["kind"]
    n = c.get("n", 0)
    if kind == "steady":
        pts = c["nx"] * c["nz"]
        # about 6 Newton steps of 10 preconditioned CG iterations, then the
        # adjoint's: the iterates, right-hand side and coefficients per cycle
        return {"bytes": 70 * 200.0 * pts + 48.0 * n, "flops": 70 * 150.0 * pts}
    if kind == "ensemble":
        b = f = 0.0
        for m in _ensemble_sizes(c, 0):
            p = _member(m, 64, 2)
            b += m * (2 * 208 + 144.0) + c["steps"] * (m * 300.0 + (_solve_bytes(p, c["vcycles"]) if c["vcycles"] else 0))
            f += c["steps"] * m * 1500.0
        return {"bytes": b, "flops": f}
    p = _work_params(c)
    if kind in ("steps", "python_steps"):
        v = c.get("vcycles", 0)
        return {"bytes": n * (2 * 208 + 144.0) + c["steps"] * (n * 300.0 + (_solve_bytes(p, v) if v else 0)),
                "flops": c["steps"] * n * 1500.0}
    if kind == "update":
        points = n * 4.0 / 0.6 / p.box_length ** 2        # boxes the colony covers
        sweeps = c["units"] * 200 * (points * 73.0 + 100.0 * p.box_x)
        return {"bytes": sweeps + c["units"] * _solve_bytes(p, 3) + n * (2 * 144.0) + 88.0 * p.box_x * p.box_z,
                "flops": c["units"] * 200 * points * 150.0}
    cycles = 8 if c["precision"] else 3
    return {"bytes": c["solves"] * _solve_bytes(p, cycles), "flops": c["solves"] * _solve_bytes(p, cycles) / 4}


# ---------------------------------------------------------------------------
def exact(case, seed):
    """What run() returns, in 64 bits by other means.  The steady field and
    its gradients: Newton with a direct block-tridiagonal solve.  Of an
    update, the deposited density; its nutrient fields are the state after a
    fixed number of V-cycles and sweeps, and the steps' records a trajectory
    through rand()'s draws, which have no value apart from that schedule."""
    if case["kind"] == "update":
        return _exact_update(case, seed)
    if case["kind"] == "steady":
        return _exact_steady(case, seed)
    return None


def _exact_update(c, seed):
    p, cells = _problem(c, seed)
    out = {"%s_0" % f: None for f in ENV + SURFACE}
    out.update({"%s_%d" % (f, l): None for f in WALLS + (AGAR if c["agar"] else ()) for l in range(p.max_levels_mg)})
    x, z = 0.5 * (cells["p"][:, 0] + cells["q"][:, 0]), 0.5 * (cells["p"][:, 2] + cells["q"][:, 2])
    xi, zi = (x / p.box_length + p.box_x // 2).astype(int), (z / p.box_length).astype(int)
    rough = np.bincount(xi * p.box_z + zi, weights=cells["length"] * cells["radius"], minlength=p.box_x * p.box_z)
    out["ROUGH_DENSITY_0"] = rough / p.box_length ** 2
    return out


class _Tridiagonal:
    """A = -dF/dC on rows 1.., factored: row blocks coupled by multiples of
    the identity (a row's diffusivity is constant along it)."""

    def __init__(self, d, face, h, sig):
        nz, nx = sig.shape
        ih2 = 1.0 / (h * h)
        self.up = [face[k] * ih2 for k in range(nz - 1)]          # between rows k and k+1
        side = torch.full((nx,), 2.0, dtype=torch.float64, device=sig.device)
        side[0] = side[-1] = 1.0
        off = torch.ones(nx - 1, dtype=torch.float64, device=sig.device)
        self.inv, prev = [None], None
        for k in range(1, nz):
            v = self.up[k - 1] + (self.up[k] if k + 1 < nz else 0.0)
            m = torch.diag(side * d[k] * ih2 + sig[k] + v) - torch.diag(off * d[k] * ih2, 1) - torch.diag(off * d[k] * ih2, -1)
            if prev is not None:
                m = m - self.up[k - 1] ** 2 * prev
            prev = torch.cholesky_inverse(torch.linalg.cholesky(m))
            self.inv.append(prev)

    def solve(self, b):
        nz = b.shape[0]
        y = [None] * nz
        for k in range(1, nz):
            y[k] = b[k] if k == 1 else b[k] + self.up[k - 1] * (self.inv[k - 1] @ y[k - 1])
        x = torch.zeros_like(b)
        for k in range(nz - 1, 0, -1):
            x[k] = self.inv[k] @ (y[k] if k == nz - 1 else y[k] + self.up[k] * x[k + 1])
        return x


def _exact_steady(c, seed):
    grid, cells, w, g = _steady_problem(c, seed)
    nx, nz, na, h, c0 = (grid[k] for k in ("nx", "nz", "nz_agar", "h", "c0"))
    da, dc, vmax, km = THETA
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    i, k = np.rint(cells[:, 0] / h).astype(int), np.rint(cells[:, 1] / h).astype(int)
    ok = (i >= 0) & (i < nx) & (k >= na) & (k < nz)
    pt = np.where(ok, k * nx + i, 0)
    lr = cells[:, 2] * cells[:, 3] / (h * h) * ok
    q = torch.from_numpy(np.bincount(pt, weights=w * lr, minlength=nx * nz).reshape(nz, nx)).to(dev)
    d = [da if r < na else dc for r in range(nz)]
    face = [d[r] if d[r] == d[r + 1] else 2 * d[r] * d[r + 1] / (d[r] + d[r + 1]) for r in range(nz - 1)]
    rowd = torch.tensor(d, dtype=torch.float64, device=dev)[:, None]
    fz = torch.tensor(face, dtype=torch.float64, device=dev)[:, None]
    ih2 = 1.0 / (h * h)

    def parts(C):
        """Differences to the row below/above and to the side neighbours."""
        dz = (C[1:] - C[:-1]) * ih2
        dx = (C[:, 1:] - C[:, :-1]) * ih2
        side = torch.zeros_like(C)
        side[:, :-1] += dx
        side[:, 1:] -= dx
        return dz, side

    def residual(C):
        dz, side = parts(C)
        f = rowd * side
        f[:-1] += fz * dz
        f[1:] -= fz * dz
        f = f - q * vmax * C / (km + C)
        f[0] = 0.0
        return f

    C = torch.full((nz, nx), c0, dtype=torch.float64, device=dev)
    for _ in range(12):
        f = residual(C)
        A = _Tridiagonal(d, face, h, q * vmax * km / (km + C) ** 2)
        step = A.solve(f)
        C = C + step
        if float(step.abs().max()) < 1e-14 * c0:
            break
    A = _Tridiagonal(d, face, h, q * vmax * km / (km + C) ** 2)
    gt = torch.from_numpy(g).to(dev)
    rhs = -gt
    rhs[0] = 0.0
    lam = A.solve(rhs)
    # dF/dd on rows 1..: agar and colony faces, the interface's harmonic mean
    dz, side = parts(C)
    wa = torch.tensor([1.0 if r + 1 < na else (2 * dc * dc / (da + dc) ** 2 if r < na else 0.0) for r in range(nz - 1)],
                      dtype=torch.float64, device=dev)[:, None]
    wc = torch.tensor([0.0 if r + 1 < na else (2 * da * da / (da + dc) ** 2 if r < na else 1.0) for r in range(nz - 1)],
                      dtype=torch.float64, device=dev)[:, None]
    rows_a = torch.tensor([1.0 if r < na else 0.0 for r in range(nz)], dtype=torch.float64, device=dev)[:, None]
    grads = []
    for wz, rows in ((wa, rows_a), (wc, 1.0 - rows_a)):
        df = rows * side
        df[:-1] += wz * dz
        df[1:] -= wz * dz
        grads.append(-float((lam * df)[1:].sum()))
    grads.append(float((lam * q * C / (km + C))[1:].sum()))
    grads.append(-float((lam * q * vmax * C / (km + C) ** 2)[1:].sum()))
    lc = (lam * vmax * C / (km + C)).cpu().numpy().reshape(-1)
    return {"C": C.cpu().numpy(), "grad_theta": np.array(grads), "grad_w": lc[pt] * lr}
