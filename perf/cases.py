"""Timed cases of the fractional-step path: what a user's program hands to the library and calls.

Four kinds of work, each through the package's public entry points:

* ``step``    -- one RK3 time step of a vessel case resident on the GPU (``Case.step``): the call a time
                 loop makes, from a developed flow;
* ``batch``   -- the same step of several uneven cases at once (``Batch.step``), as the batched and the
                 serving workloads make it;
* ``poisson`` -- one pressure solve on resident fields from zero (``Case.poisson``);
* ``ops``     -- the explicit part of one substep through the reference's launcher FFI, operator by
                 operator, as the Fortran wrappers call it (FP64 and the ``_sp_`` FP32 launchers);
* ``jor``     -- 50 JOR sweeps through the launcher FFI (the reference's own pressure relaxation).

Sizes are cells per axis.  They span the configurations of this repository: 32 x 32 x 64 (the smallest
batched case) to 384 x 384 x 768 (the benchmark case), with the operator microbench's stretched grid, the
plain step's JOR solver and ragged sizes whose rows hold no whole 16-byte vectors.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpu-impact-ct_b200"))
import impact_b200 as I  # noqa: E402

VELOCITY = ("vel1", "vel2", "vel3")


def _step(name, n, precision, precond=1, stretch=0, cheb=0):
    return {"name": name, "kind": "step", "n1": n[0], "n2": n[1], "n3": n[2], "precision": precision, "precond": precond,
            "stretch": stretch, "cheb": cheb}


def listed():
    return [
        # the benchmark case of the repository: one large stenosed vessel, mixed precision
        _step("step_mixed_384", (384, 384, 768), 1),
        # an ordinary single case, mixed precision
        _step("step_mixed_128", (128, 128, 256), 1),
        # the smallest case that the batched and serving workloads admit, stepped alone: latency
        _step("step_mixed_32", (32, 32, 64), 1),
        # the drop-in's precision with the multigrid preconditioner, medium size
        _step("step_fp64_192", (192, 192, 384), 0),
        # the plain drop-in step: FP64, JOR-preconditioned BiCGstab, 64 x 64 x 128
        _step("step_jor_64", (64, 64, 128), 0, precond=0),
        # a grid refined in x and y around the vessel (per-row weights in every operator)
        _step("step_mixed_stretched", (112, 96, 168), 1, stretch=1),
        # a CT volume with its own odd extents: no coarsening, no whole vectors in a row
        _step("step_jor_ragged", (59, 47, 83), 1, precond=0),
        # uneven cases advanced together (continuous batching), Chebyshev bottom as the workloads run it
        {"name": "batch_mixed_12", "kind": "batch", "cases": 12, "lo": 32, "hi": 152, "precision": 1, "pick": 7},
        # a pressure solve by itself
        {"name": "poisson_mixed_256", "kind": "poisson", "n1": 256, "n2": 256, "n3": 512, "precision": 1, "cheb": 0},
        # the operator microbench: 256 x 256 x 512, x and y stretched, FP64 fields far above the L2
        {"name": "ops_fp64_256", "kind": "ops", "n1": 256, "n2": 256, "n3": 512, "fp32": 0, "stretch": 1},
        # FP32 launchers on a ragged grid
        {"name": "ops_fp32_ragged", "kind": "ops", "n1": 187, "n2": 131, "n3": 157, "fp32": 1, "stretch": 0},
        # the reference's relaxation on a small grid: short kernels, one after another
        {"name": "jor_fp64_64", "kind": "jor", "n1": 64, "n2": 64, "n3": 128, "fp32": 0, "stretch": 0},
    ]


def draw(rng):
    def log_size(lo, hi, multiple=1):
        v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        return int(max(lo, min(hi, round(v / multiple) * multiple)))

    kind = rng.choice(("step", "step", "step", "batch", "poisson", "ops", "ops", "jor"))
    if kind == "step" and rng.random() < 0.3:  # JOR: any extents
        n = log_size(24, 72)
        side = [max(9, n + rng.randint(-8, 8)) for _ in range(2)]
        return {k: v for k, v in _step("", (*side, n + rng.randint(0, n)), rng.randint(0, 1), precond=0).items() if k != "name"}
    if kind in ("step", "poisson"):
        precision = rng.randint(0, 1)
        n = log_size(32, 224 if precision else 160, 8)
        n1, n2 = (max(32, n + 8 * rng.randint(-2, 2)) for _ in range(2))
        n3 = max(32, int(n * rng.uniform(1.0, 2.2) / 8) * 8)
        cheb = rng.choice((0, 32))
        if kind == "poisson":
            return {"kind": kind, "n1": n1, "n2": n2, "n3": n3, "precision": precision, "cheb": cheb}
        c = _step("", (n1, n2, n3), precision, stretch=int(rng.random() < 0.25), cheb=cheb)
        return {k: v for k, v in c.items() if k != "name"}
    if kind == "batch":
        lo = 8 * rng.randint(4, 8)
        return {"kind": kind, "cases": rng.randint(2, 12), "lo": lo, "hi": 8 * rng.randint(lo // 8 + 1, 18),
                "precision": rng.randint(0, 1), "pick": rng.randint(0, 10**6)}
    fp32, stretch = rng.randint(0, 1), rng.randint(0, 1)
    n = log_size(16, 288 if kind == "ops" else 208)
    if rng.random() < 0.5:
        n = max(16, n // 8 * 8)
        sizes = (n, max(16, n + 8 * rng.randint(-1, 1)), max(16, n + 8 * rng.randint(0, n // 8)))
    else:
        sizes = tuple(max(9, int(n * rng.uniform(0.6, 1.4))) for _ in range(3))
    return {"kind": kind, "n1": sizes[0], "n2": sizes[1], "n3": sizes[2], "fp32": fp32, "stretch": stretch}


# ---------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------
def _grid(case):
    n = (case["n1"], case["n2"], case["n3"])
    kinds = (1, 1, 0) if case.get("stretch") else (0, 0, 0)
    h = 1.0 / max(n[0], n[1])
    return I.Grid(tuple(m + 1 for m in n), tuple(m * h for m in n), kinds)


def _coords(grid):
    """Pressure points 1..n of the axes on the GPU, shaped to broadcast over (k, j, i)."""
    x = [torch.from_numpy(grid.xp[a][4:grid.N[a] + 3].copy()).cuda() for a in range(3)]
    return x[0][None, None, :], x[1][None, :, None], x[2][:, None, None]


class _Resident:
    """A field of a case as an array of the device (the case lives as long as a tensor of it)."""

    def __init__(self, case, field):
        self.case = case
        self.__cuda_array_interface__ = {"shape": case.grid.shape, "typestr": "<f8", "version": 3, "strides": None,
                                         "data": (case.field_ptr(field), False)}


def _inner(t, grid):
    n = [m - 1 for m in grid.N]
    return t[..., 4:4 + n[2], 4:4 + n[1], 4:4 + n[0]]


def _field(case, field):
    return _inner(torch.as_tensor(_Resident(case, field), device="cuda"), case.grid)


def _modes(grid, gen, count=6):
    """A smooth periodic field: a few Fourier modes with random phases."""
    X = _coords(grid)
    out = torch.zeros([m - 1 for m in reversed(grid.N)], dtype=torch.float64, device="cuda")
    for _ in range(count):
        k = torch.randint(1, 5, (3,), generator=gen).tolist()
        ph = (2 * math.pi * torch.rand(3, generator=gen, dtype=torch.float64)).tolist()
        a = float(torch.rand(1, generator=gen, dtype=torch.float64)) + 0.2
        f = [torch.sin(2 * math.pi * k[q] * X[q] / grid.L[q] + ph[q]) for q in range(3)]
        out += a * f[0] * f[1] * f[2]
    return out / math.sqrt(count)


def _vessel(grid, gen, radius):
    """Labels (k, j, i) of a stenosed cylinder along z and the normalised distance from its axis."""
    x, y, z = _coords(grid)
    z0 = grid.L[2] * (0.3 + 0.4 * float(torch.rand(1, generator=gen)))
    side = min(grid.L[0], grid.L[1])
    r = radius * side * (1.0 - 0.37 * torch.exp(-((z - z0) ** 2) / (2 * (0.5 * radius * side) ** 2)))
    s = torch.sqrt((x - 0.5 * grid.L[0]) ** 2 + (y - 0.5 * grid.L[1]) ** 2) / r
    lab = (s <= 1.0).to(torch.uint8)
    ends = max(2, min(10, lab.shape[0] // 8))
    lab[:ends] *= 5
    lab[-ends:] *= 9
    return lab, s


def _vessel_case(case, gen, radius=0.25, U0=1.0):
    """A case stepped for a while: a parabolic jet through the vessel with disturbances, no pressure yet."""
    grid = _grid(case)
    c = I.Case(grid, precision=case["precision"])
    lab, s = _vessel(grid, gen, radius)
    full = torch.zeros(grid.shape, dtype=torch.uint8, device="cuda")
    _inner(full, grid)[...] = lab
    c.set_labels(full.cpu().numpy())
    solid = lab == 0
    for m, f in enumerate(VELOCITY):
        v = 0.05 * U0 * _modes(grid, gen)
        if m == 2:
            v += U0 * (1.0 - s * s).clamp_min(0.0)
        v[solid] = 0.0
        _field(c, f)[...] = v
    torch.cuda.synchronize()
    return c, lab


def _solver(case, init_yes=0):
    jor = case.get("precond", 1) == 0
    if case["precision"] == 0:
        max_it, inner = (2000 if jor else 200), 0
    else:
        max_it, inner = 40, (4000 if jor else 400)
    return dict(tol_rel=1e-8, max_it=max_it, inner_max_it=inner, inner_tol_rel=3e-3, n_sweeps=4, omega=0.8, init_yes=init_yes,
                check_every=4 if jor else 2, precond=0 if jor else 1, mg_down=3, mg_up=3, mg_bottom=3, tile_kc=0 if jor else 64,
                bottom_cheb=case.get("cheb", 0))


def _params(case, Re=400.0, U0=1.0):
    return I.step_params(Re=Re, CFL=0.2, dtime_max=1.0, U0=U0, T_pulse=1.0, level_pressure=1, **_solver(case))


def _batch_members(case):
    rng = np.random.default_rng(case["pick"])
    out = []
    for _ in range(case["cases"]):
        n = int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]))) / 8)) * 8
        out.append({"n1": n, "n2": n, "n3": 2 * n, "precision": case["precision"], "cheb": 32,
                    "radius": float(rng.uniform(0.15, 0.3)), "Re": float(rng.uniform(100, 800)), "U0": float(rng.uniform(0.5, 1.5))})
    return out


def _generator(seed):
    gen = torch.Generator()
    gen.manual_seed(int(seed))
    return gen


def _ops_inputs(case, seed):
    grid = _grid(case)
    dt = torch.float32 if case["fp32"] else torch.float64
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))

    def field(count):
        t = torch.zeros((count,) + grid.shape, dtype=dt, device="cuda")
        v = _inner(t, grid)
        v[...] = torch.rand(v.shape, dtype=dt, device="cuda", generator=gen) * 2 - 1
        return t

    tab = {k: [torch.from_numpy(a).cuda().to(dt) for a in v] for k, v in grid.tab.items()}
    return grid, dt, tab, field


class _Calls:
    """Launcher calls with their arguments by reference, as the Fortran wrappers hold them."""

    def __init__(self, grid, fp32):
        self.sfx, self.real = ("_sp_", ctypes.c_float) if fp32 else ("_", ctypes.c_double)
        self.dims = [m + 7 for m in grid.N]
        self.calls = []

    def add(self, name, ints, reals, arrays):
        keep = [ctypes.c_int(v) for v in ints] + [self.real(v) for v in reals]
        keep += [ctypes.cast(ctypes.c_void_p(t.data_ptr()), ctypes.POINTER(ctypes.c_double)) for t in arrays]
        self.calls.append((getattr(I.lib(), name + self.sfx), [ctypes.byref(v) for v in keep], keep, list(arrays)))

    def run(self):
        for f, args, _, _ in self.calls:
            f(*args)


RE, DT = 400.0, 2e-3
A_RK = 8.0 / 15.0


def _prepare_ops(case, seed):
    """interpolate_vel, the advection and diffusion terms and the update of the three components,
    divergence2 of the provisional velocity, projection with a given pressure: 34 launcher calls."""
    grid, dt, tab, field = _ops_inputs(case, seed)
    vel, pre = field(3), field(1)
    zero = lambda n: torch.zeros((n,) + grid.shape, dtype=dt, device="cuda")  # noqa: E731
    work, nl, rhs, new = zero(3), zero(3), zero(3), zero(3)
    pp, grad, div = zero(1), zero(1), zero(1)
    k = _Calls(grid, case["fp32"])
    d = k.dims
    for m in range(3):
        k.add("interpolate2_vel_pre_launcher", [m + 1, *d, 6, grid.N[m] + 1], [], [vel[m], tab["cIup"][m], work[m]])
    for m in range(3):
        for a in range(3):
            k.add("interpolate2_pre_vel_launcher", [m + 1, *d, 6, grid.N[m] + 1], [], [work[a], tab["cIpu"][m], pp])
            up, dn = ("cNuU", "cNuD") if a == m else ("cNpU", "cNpD")
            k.add("nonlinear_upwind_launcher", [3 * m + a + 1, *d, 7, grid.N[a] + 1], [],
                  [pp, vel[m], nl[m], tab[up][a], tab[dn][a]])
        c = [tab["cuu" if a == m else "cpp"][a] for a in range(3)]
        k.add("helmholtz_explicit_launcher", [m + 1, *d, 7, 7, 7], [1.0 / RE], [vel[m], nl[m], *c])
        k.add("axpby_launcher", d, [1.0, -DT * A_RK], [vel[m], nl[m], rhs[m]])
    k.add("divergence2_launcher", [*d, 6, 6, 6], [], [rhs, div, *tab["cD"]])
    for m in range(3):
        k.add("gradient_launcher", [m + 1, *d, 6, grid.N[m] + 1], [], [pre, tab["cG"][m], grad])
        k.add("axpby_launcher", d, [1.0, -1.0], [rhs[m], grad, new[m]])
    return {"calls": k, "out": {"nl": nl, "rhs": rhs, "div": div, "new": new}, "keep": (work, pre, vel, tab)}


def _prepare_jor(case, seed):
    grid, dt, tab, field = _ops_inputs(case, seed)
    rel, bb, comp = field(1), field(1), torch.zeros((1,) + grid.shape, dtype=dt, device="cuda")
    k = _Calls(grid, case["fp32"])
    src, dst = rel, comp
    for _ in range(50):
        # (grid id, extents, table extents, table width), omega, tables, iterate, right-hand side, result
        k.add("jacobi_launcher", [1, *k.dims, *grid.N, 3], [0.8], [*tab["cdg"], src, bb, dst])
        src, dst = dst, src
    return {"calls": k, "out": {"rel": rel}, "keep": (bb, comp, tab)}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ops":
        return _prepare_ops(case, seed)
    if kind == "jor":
        return _prepare_jor(case, seed)
    gen = _generator(seed)
    if kind == "poisson":
        c = I.Case(_grid(case), precision=case["precision"])
        b = _modes(c.grid, gen)
        noise = torch.Generator(device="cuda")
        noise.manual_seed(int(seed))
        b += 0.1 * torch.randn(b.shape, dtype=b.dtype, device="cuda", generator=noise)
        _field(c, "res")[...] = b - b.mean()
        torch.cuda.synchronize()
        return {"case": c, "params": I.solver_params(**_solver(case, init_yes=1))}
    if kind == "step":
        c, _ = _vessel_case(case, gen)
        return {"case": c, "params": _params(case)}
    members = _batch_members(case)
    cases = [_vessel_case(m, gen, m["radius"], m["U0"])[0] for m in members]
    return {"batch": I.Batch(cases), "cases": cases, "params": [_params(m, m["Re"], m["U0"]) for m in members]}


def _state_of(c):
    return {f: _field(c, f) for f in VELOCITY + ("pre",)}


def run(state):
    if "calls" in state:
        state["calls"].run()
        return state["out"]
    if "batch" in state:
        st = state["batch"].step(state["params"], 1)
        return {"dt": [s.dtime for s in st][0], "cases": [_state_of(c) for c in state["cases"]]}
    c = state["case"]
    if isinstance(state["params"], I.SolverParams):
        c.poisson("res", "pre", state["params"])
        p = _field(c, "pre")
        return {"pre": p - p.mean()}  # the pressure is defined up to a constant
    return dict(_state_of(c), dt=c.step(state["params"], 1).dtime)


# ---------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------
def work(case):
    """Inputs once in, outputs once out; the operations of one evaluation of every formula (one operator
    application for a solve, whose iteration count is the solver's affair)."""
    if case["kind"] == "batch":
        cells = sum(m["n1"] * m["n2"] * m["n3"] for m in _batch_members(case))
        return {"bytes": 65.0 * cells, "flops": 1600.0 * cells}
    cells = float(case["n1"] * case["n2"] * case["n3"])
    if case["kind"] == "step":  # velocity and pressure in and out, labels in
        return {"bytes": 65.0 * cells, "flops": 1600.0 * cells}
    if case["kind"] == "poisson":
        return {"bytes": 16.0 * cells, "flops": 66.0 * cells}
    size = 4.0 if case["fp32"] else 8.0
    if case["kind"] == "jor":
        return {"bytes": 3 * size * cells, "flops": 50 * 16.0 * cells}
    return {"bytes": 14 * size * cells, "flops": 470.0 * cells}


# ---------------------------------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------------------------------


def _s(f, table, a, low):
    """sum_l c(l, q) f(q + low + l) along axis a, periodic; table rows 0..N."""
    n = f.shape[2 - a]
    c = table.double().reshape(n + 2, -1)[1:n + 1]
    shape = [1, 1, 1]
    shape[2 - a] = n
    out = torch.zeros_like(f)
    for l in range(c.shape[1]):
        out += c[:, l].reshape(shape) * torch.roll(f, -(low + l), 2 - a)
    return out


def _advect(m, vel, work, tab, Re):
    nl = torch.zeros_like(vel)
    for a in range(3):
        pp = _s(work[a], tab["cIpu"][m], m, -2)
        up, dn = ("cNuU", "cNuD") if a == m else ("cNpU", "cNpD")
        nl += pp * torch.where(pp >= 0, _s(vel, tab[up][a], a, -3), _s(vel, tab[dn][a], a, -3))
    for a in range(3):
        nl -= _s(vel, tab["cuu" if a == m else "cpp"][a], a, -3) / Re
    return nl


def _solve(b, tab):
    """A x = b of an equidistant periodic grid by Fourier transform, zero mean."""
    total = torch.zeros(b.shape[0], b.shape[1], b.shape[2] // 2 + 1, dtype=torch.complex128, device="cuda")
    for a in range(3):
        n = b.shape[2 - a]
        cD, cG = (tab[t][a].double().reshape(n + 2, 6)[n // 2].cpu() for t in ("cD", "cG"))
        th = 2 * math.pi * torch.arange(n // 2 + 1 if a == 0 else n, dtype=torch.float64) / n
        e = lambda o: torch.exp(1j * th * o)  # noqa: E731
        sym = sum(cD[l] * e(l - 3) for l in range(6)) * sum(cG[l] * e(l - 2) for l in range(6))
        shape = [1, 1, 1]
        shape[2 - a] = sym.numel()
        total += sym.cuda().reshape(shape)
    total[0, 0, 0] = 1.0
    x = torch.fft.rfftn(b) / total
    x[0, 0, 0] = 0.0
    return torch.fft.irfftn(x, s=b.shape)


def _limits():
    """Radius of the RK3 stability region along the 41 rays of get_dtime."""
    lim = []
    for q in range(41):
        z1 = complex(-math.sin(q * math.pi / 80), math.cos(q * math.pi / 80))
        g = lambda r: abs(1 + r * z1 + (r * z1) ** 2 / 2 + (r * z1) ** 3 / 6) - 1.0  # noqa: E731
        lo = hi = 1e-3
        while g(hi) < 0 and hi < 10:
            lo, hi = hi, hi + 1e-3
        for _ in range(100):
            mid = 0.5 * (lo + hi)
            lo, hi = (mid, hi) if g(mid) < 0 else (lo, mid)
        lim.append(0.5 * (lo + hi))
    return torch.tensor(lim, dtype=torch.float64, device="cuda")


def _time_step(vel, work_of, tab, Re, CFL):
    are, aim = 0.0, 0.0
    for a in range(3):
        n = vel[0].shape[2 - a]
        shape = [1, 1, 1]
        shape[2 - a] = n
        rows = lambda t: tab[t][a].reshape(n + 2, 7)[1:n + 1].abs().sum(1).reshape(shape)  # noqa: E731
        are = are + rows("cpp") / Re
        aim = aim + rows("cp1") * work_of[a].abs()
    angle = torch.where(aim < 1e-16, torch.full_like(aim, math.pi / 2), torch.atan(are / aim.clamp_min(1e-300)))
    ray = torch.floor(80 * angle / math.pi + 0.5).long().clamp(0, 40)
    beta = float((torch.sqrt(are * are + aim * aim) / _limits()[ray]).max()) / CFL
    return min(1.0, 1.0 / beta)


def _exact_step(case, gen, radius=0.25, Re=400.0, U0=1.0):
    c, lab = _vessel_case(case, gen, radius, U0)
    tab = {k: [torch.from_numpy(a).cuda() for a in v] for k, v in c.grid.tab.items()}
    vel = [_field(c, f).clone() for f in VELOCITY]
    c.close()
    dt, old, pre = None, [None] * 3, None
    for sub, (aRK, bRK) in enumerate(((8 / 15, 0.0), (5 / 12, -17 / 60), (3 / 4, -5 / 12))):
        w = [_s(vel[a], tab["cIup"][a], a, -3) for a in range(3)]
        if sub == 0:
            dt = _time_step(vel, w, tab, Re, 0.2)
        rhs = []
        for m in range(3):
            nl = _advect(m, vel[m], w, tab, Re)
            rhs.append(vel[m] - dt * aRK * nl - (dt * bRK * old[m] if sub else 0.0))
            old[m] = nl
        x = _solve(sum(_s(rhs[a], tab["cD"][a], a, -3) for a in range(3)), tab)
        vel = [rhs[a] - _s(x, tab["cG"][a], a, -2) for a in range(3)]
        pre = x / (aRK + bRK) / dt
    solid, inflow = lab == 0, lab == 5
    for m in range(3):
        vel[m][solid] = 0.0
        vel[m][inflow] = U0 * (1 + 0.5 * math.sin(2 * math.pi * dt)) if m == 2 else 0.0
    return dict(zip(VELOCITY + ("pre",), vel + [pre - pre.mean()])), dt


def _padded(v, grid):
    out = torch.zeros((len(v),) + grid.shape, dtype=torch.float64, device="cuda")
    for m, x in enumerate(v):
        _inner(out[m], grid)[...] = x
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":  # the first case's time step for all, and every case's fields
        gen, out = _generator(seed), []
        for m in _batch_members(case):
            out.append(_exact_step(m, gen, m["radius"], m["Re"], m["U0"]))
        return {"dt": out[0][1], "cases": [f for f, _ in out]}
    if kind == "step":
        if case["stretch"]:  # no Fourier solve on a stretched grid
            return None
        f, dt = _exact_step(case, _generator(seed))
        return dict(f, dt=dt)
    if kind == "poisson":
        state = prepare(case, seed)
        c = state["case"]
        return {"pre": _solve(_field(c, "res").clone(), {k: [torch.from_numpy(a) for a in c.grid.tab[k]] for k in ("cD", "cG")})}
    state = prepare(case, seed)
    grid = _grid(case)
    if kind == "jor":
        bb, _, tab = state["keep"]
        x, b = (_inner(t[0], grid).double() for t in (state["out"]["rel"], bb))
        c = []
        for a in range(3):
            shape = [1, 1, 1]
            shape[2 - a] = x.shape[2 - a]
            c.append([tab["cdg"][a].double().reshape(-1, 3)[:x.shape[2 - a], l].reshape(shape) for l in range(3)])
        diag = c[0][1] + c[1][1] + c[2][1]
        for _ in range(50):
            r = b - sum(c[a][0] * torch.roll(x, 1, 2 - a) + c[a][2] * torch.roll(x, -1, 2 - a) for a in range(3))
            x = 0.8 * r / diag + 0.2 * x
        return {"rel": _padded([x], grid)}
    _, pre, vel, tab = state["keep"]
    vel, pre = [_inner(v, grid).double() for v in vel], _inner(pre[0], grid).double()
    w = [_s(vel[a], tab["cIup"][a], a, -3) for a in range(3)]
    nl = [_advect(m, vel[m], w, tab, RE) for m in range(3)]
    rhs = [vel[m] - DT * A_RK * nl[m] for m in range(3)]
    div = sum(_s(rhs[a], tab["cD"][a], a, -3) for a in range(3))
    new = [rhs[a] - _s(pre, tab["cG"][a], a, -2) for a in range(3)]
    return {"nl": _padded(nl, grid), "rhs": _padded(rhs, grid), "div": _padded([div], grid), "new": _padded(new, grid)}
