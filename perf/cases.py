"""Performance cases of the framework: the calls a user's program makes, over the sizes, precisions and
directions it makes them in.

Each case is a dict of plain values; `prepare` builds what the program has in hand before the call, `run` makes
one pass through the public entry points, `exact` evaluates the same result in plain 64-bit torch where that is
a formula and not a long iteration.  Kinds:

  operator   one operator of one level (residual with norms, Jacobian product, transposed product): what hosts
             that drive their own solver, and convergence checks, call
  forward    one implicit time step (u, v, H at t + dt) from a given state
  gradient   the adjoint solve at a solved state and the gradients for bed, beta, H_prev and smb
  step       one autograd step of an inversion: GlideStep forward, misfit, backward
  group      forward and adjoint solves of several equal members in grouped launches (ensembles)
  thermal    the thermal half of a coupled step: omega, heating, column sweeps, rate factor
  columns    enthalpy column sweeps with layer-dependent velocities (polythermal ice, several sweeps)

Solver forms: "reference" is the reference algorithm (10/20/50/200 FASCD sweeps, 30 local Newton iterations) at a
fixed number of V-cycles; "fast" is the Newton form with the tangent multigrid, solved to a relative residual
of 1e-8, with the short adjoint schedule.
"""
from __future__ import annotations

import math

import torch

RHO_G = 910.0 * 9.81
B0 = (1e-16 ** (-1.0 / 3.0)) / RHO_G
FLOT = float(torch.tensor(0.917, dtype=torch.float32))  # a binary32 literal of the operator
YEAR = 365.25 * 86400.0
THKLIM = 0.1


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # one residual evaluation with its norms on the 64^2 slab level: the smallest call, all latency
        dict(name="residual_64", kind="operator", op="residual", ny=64, nx=64, dx=1000.0, dt=10.0, precision="fp64"),
        # a binary32 Jacobian product of a ragged level: matrix-free solvers and sensitivity studies
        dict(name="jvp_1000x760_fp32", kind="operator", op="jvp", ny=1000, nx=760, dx=1500.0, dt=10.0,
             precision="fp32"),
        # the ISMIP-HOM-like slab step: 4 levels, 3 V-cycles of the reference algorithm; launches and latency count
        dict(name="slab_64_forward", kind="forward", ny=64, nx=64, levels=4, dx=1000.0, dt=10.0, precision="fp64",
             form="reference", vcycles=3, quirks=True, shape="slab"),
        # a regional, non-square domain in binary32 with corrected transfers
        dict(name="region_600x424_fp32_forward", kind="forward", ny=600, nx=424, levels=3, dx=2000.0, dt=5.0,
             precision="fp32", form="reference", vcycles=2, quirks=False, shape="dome", radius=0.4),
        # the continental dome, plain binary64 reference algorithm, 3 V-cycles a step
        dict(name="dome_512_forward", kind="forward", ny=512, nx=512, levels=5, dx=1500.0, dt=10.0,
             precision="fp64", form="reference", vcycles=3, quirks=True, shape="dome", radius=0.78),
        # its adjoint with the reference's schedule and the four gradients
        dict(name="dome_512_gradient", kind="gradient", ny=512, nx=512, levels=5, dx=1500.0, dt=10.0,
             precision="fp64", form="reference", vcycles=2, quirks=True, shape="dome", radius=0.78),
        # one inversion step on the same dome: mixed precision, solved to 1e-8 both ways through autograd
        dict(name="dome_512_mixed_step", kind="step", ny=512, nx=512, levels=5, dx=1500.0, dt=10.0,
             precision="mixed", form="fast", vcycles=40, quirks=False, shape="dome", radius=0.78),
        # the large dome's time step to 1e-8 in mixed precision: the headline workload
        dict(name="dome_2048_mixed_forward", kind="forward", ny=2048, nx=2048, levels=7, dx=750.0, dt=5.0,
             precision="mixed", form="fast", vcycles=40, quirks=False, shape="dome", radius=0.78),
        # and its gradient
        dict(name="dome_2048_mixed_gradient", kind="gradient", ny=2048, nx=2048, levels=7, dx=750.0, dt=5.0,
             precision="mixed", form="fast", vcycles=40, quirks=False, shape="dome", radius=0.78),
        # eight ensemble members solved in grouped launches
        dict(name="group_8x192", kind="group", ny=192, nx=192, levels=4, dx=3000.0, dt=10.0, precision="fp64",
             form="fast", vcycles=3, quirks=False, shape="dome", radius=0.4, members=8),
        # the thermal half of a coupled step: 41 sigma levels, depth-independent velocity, default stop test
        dict(name="thermal_1024x41", kind="thermal", ny=1024, nx=1024, nz=41, dx=1500.0, dt=5.0),
        # polythermal columns on a ragged grid with layer velocities: three full sweeps
        dict(name="columns_250x190x21", kind="columns", ny=250, nx=190, nz=21, dx=2000.0, dt=10.0, sweeps=3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["operator", "operator", "forward", "forward", "gradient", "step", "group", "thermal",
                       "columns", "columns"])
    if kind == "operator":
        return dict(kind=kind, op=rng.choice(["residual", "jvp", "vjp"]), ny=_log_int(rng, 64, 2048),
                    nx=_log_int(rng, 64, 2048), dx=rng.choice([750.0, 1000.0, 1500.0, 3000.0]),
                    dt=rng.choice([1.0, 5.0, 10.0]), precision=rng.choice(["fp64", "fp32"]))
    if kind == "thermal":
        return dict(kind=kind, ny=_log_int(rng, 64, 1024), nx=_log_int(rng, 64, 1024), nz=rng.choice([11, 21, 31, 41]),
                    dx=rng.choice([1000.0, 1500.0, 3000.0]), dt=rng.choice([1.0, 5.0, 10.0]))
    if kind == "columns":
        return dict(kind=kind, ny=_log_int(rng, 32, 512), nx=_log_int(rng, 32, 512),
                    nz=rng.choice([3, 11, 17, 21, 41, 64]), dx=rng.choice([1000.0, 2000.0, 5000.0]),
                    dt=rng.choice([5.0, 10.0]), sweeps=rng.choice([1, 2, 3, 5]))
    if kind == "group":
        n = 16 * rng.choice([4, 6, 8, 10, 12])
        return dict(kind=kind, ny=n, nx=n, levels=3, dx=3000.0, dt=rng.choice([5.0, 10.0]), precision="fp64",
                    form="fast", vcycles=rng.choice([2, 3]), quirks=False, shape="dome", radius=0.4, members=rng.choice([2, 5, 8]))
    # solves: a coarsest grid times a power of two per direction
    levels = rng.choice([3, 4, 5])
    unit = 2 ** (levels - 1)
    square = rng.random() < 0.5
    form = "fast" if kind == "step" else rng.choice(["reference", "fast"])
    most = 1024 if form == "fast" else 640
    ny = unit * max(16, _log_int(rng, 64, most) // unit)
    nx = ny if square else unit * max(16, _log_int(rng, 64, most) // unit)
    # binary64 and mixed hold for every form; the plain binary32 handle is used with the reference algorithm
    precision = rng.choice(["fp64", "mixed"]) if form == "fast" or kind == "gradient" else rng.choice(["fp64", "fp32"])
    return dict(kind=kind, ny=ny, nx=nx, levels=levels, dx=1536000.0 / max(ny, nx), dt=rng.choice([5.0, 10.0]),
                precision=precision, form=form, vcycles=40 if form == "fast" else rng.choice([1, 2, 3]),
                quirks=square and form == "reference", shape="dome",
                radius=0.78 if form == "fast" else rng.choice([0.4, 0.78]))


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 13)
    return g


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _smooth(f, cells):
    """Gaussian smoothing by a periodic FFT."""
    ky = torch.fft.fftfreq(f.shape[0], device="cuda", dtype=torch.float64)[:, None]
    kx = torch.fft.fftfreq(f.shape[1], device="cuda", dtype=torch.float64)[None, :]
    w = torch.exp(-2 * (math.pi * cells) ** 2 * (kx * kx + ky * ky))
    return torch.fft.ifft2(torch.fft.fft2(f) * w).real


def _centres(ny, nx, dx):
    y = (torch.arange(ny, device="cuda", dtype=torch.float64) + 0.5) * dx - ny * dx / 2
    x = (torch.arange(nx, device="cuda", dtype=torch.float64) + 0.5) * dx - nx * dx / 2
    return y[:, None], x[None, :]


def _fields(case, g):
    """Geometry and parameters: a Vialov-like dome on a Gaussian random bed (spectral slope -3, std 400 m, mean
    200 m) with log-normal smoothed beta and an elevation-dependent smb, or the tilted slab with a bump."""
    ny, nx, dx = case["ny"], case["nx"], case["dx"]
    Y, X = _centres(ny, nx, dx)
    ones = torch.ones(ny, nx, device="cuda", dtype=torch.float64)
    if case.get("shape") == "slab":
        L = nx * dx
        ph = 2 * math.pi * torch.rand(2, generator=g, device="cuda", dtype=torch.float64)
        px, py = 2 * math.pi * (X + L / 2) / L, 2 * math.pi * (Y + ny * dx / 2) / (ny * dx)
        bed = -(X + L / 2) * math.tan(math.radians(0.5)) + 500.0 * torch.sin(px + ph[0]) * torch.sin(py + ph[1])
        beta = (1000.0 + 500.0 * torch.sin(px + ph[0])) / RHO_G * ones
        H, smb = 1000.0 * ones, 0.3 * ones
    else:
        R = case.get("radius", 0.4) * max(ny, nx) * dx  # 0.78 covers the domain with ice, 0.4 leaves margins
        r = torch.sqrt(X * X + Y * Y)
        H = (3000.0 * torch.clamp(1.0 - (r / R) ** (4.0 / 3.0), min=0.0) ** (3.0 / 8.0)).clamp(min=THKLIM)
        ky = torch.fft.fftfreq(ny, device="cuda", dtype=torch.float64)[:, None]
        kx = torch.fft.fftfreq(nx, device="cuda", dtype=torch.float64)[None, :]
        k = torch.sqrt(kx * kx + ky * ky)
        k[0, 0] = 1.0
        w = torch.fft.ifft2(torch.fft.fft2(_randn(g, ny, nx)) * k ** -1.5).real
        bed = 200.0 + 400.0 * (w - w.mean()) / w.std()
        beta = _smooth(torch.exp(math.log(2000.0) + 0.8 * _randn(g, ny, nx)), 10e3 / dx) / RHO_G
        s = torch.maximum(bed + H, (1.0 - 0.917) * H)
        smb = 0.5 - 2e-3 * (s - 1500.0)
    return dict(bed=bed, beta=beta, smb=smb, B=B0 * ones, H=H, H_prev=H.clone())


def _velocity(case, g, H):
    """A radial outflow with noise (m/a), on the u and v faces."""
    ny, nx, dx = case["ny"], case["nx"], case["dx"]
    Y, X = _centres(ny, nx, dx)
    R = 0.4 * max(ny, nx) * dx
    uc = (200.0 * X / R) * (H > 1.0) * (1.0 + 0.2 * _smooth(_randn(g, ny, nx), 3.0))
    vc = (-200.0 * Y / R) * (H > 1.0) * (1.0 + 0.2 * _smooth(_randn(g, ny, nx), 3.0))
    u = torch.zeros(ny, nx + 1, device="cuda", dtype=torch.float64)
    v = torch.zeros(ny + 1, nx, device="cuda", dtype=torch.float64)
    u[:, 1:-1] = 0.5 * (uc[:, 1:] + uc[:, :-1])
    v[1:-1, :] = 0.5 * (vc[1:, :] + vc[:-1, :])
    return u, v


def _operator_inputs(case, seed):
    g = _gen(seed)
    f = _fields(case, g)
    f["u"], f["v"] = _velocity(case, g, f["H"])
    f["mask"] = (f["H"] <= THKLIM).to(torch.float64)
    f["H"] = f["H"] * (1.0 + 0.01 * _smooth(_randn(g, case["ny"], case["nx"]), 2.0))
    # the direction of the products: smooth with grid-scale noise, zero on the Dirichlet faces
    f["e_u"], f["e_v"] = _randn(g, *f["u"].shape), _randn(g, *f["v"].shape)
    f["e_H"] = _randn(g, *f["H"].shape)
    f["e_u"][:, 0] = f["e_u"][:, -1] = 0.0
    f["e_v"][0, :] = f["e_v"][-1, :] = 0.0
    if case["precision"] == "fp32":
        f = {k: t.float() for k, t in f.items()}
    return f


def _thermal_inputs(case, seed):
    g = _gen(seed)
    ny, nx = case["ny"], case["nx"]
    f = _fields(case, g)
    f["H"] = f["H"] * (1.0 + 0.05 * _smooth(_randn(g, ny, nx), 4.0))
    f["u"], f["v"] = _velocity(case, g, f["H"])
    f["H1"] = f["H"] * (1.0 + 1e-3 * _randn(g, ny, nx))
    s = torch.maximum(f["bed"] + f["H"], (1.0 - 0.917) * f["H"])
    f["T_s"] = 273.15 + (-30.0 + 6e-3 * (2000.0 - s))
    # cold at the surface, warming towards the pressure melting point at the bed
    sig = torch.linspace(0.0, 1.0, case["nz"], device="cuda", dtype=torch.float64)
    Tb = 272.0 + 1.5 * torch.rand(ny, nx, generator=g, device="cuda", dtype=torch.float64)
    f["T"] = f["T_s"][:, :, None] + (Tb - f["T_s"])[:, :, None] * (1.0 - sig) ** 2
    return f


def _column_inputs(case, seed):
    """Cold and temperate nodes on both sides of the melting point, thin columns, layer velocities (m/s)."""
    g = _gen(seed)
    ny, nx, nz = case["ny"], case["nx"], case["nz"]

    def rnd(lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)

    H = torch.where(rnd(0, 1, ny, nx) < 0.1, rnd(1.0, 20.0, ny, nx), rnd(500.0, 3000.0, ny, nx))
    sig = torch.linspace(0.0, 1.0, nz, device="cuda", dtype=torch.float64)
    Ep = _e_pmp(sig, H[:, :, None])
    E = Ep + rnd(-0.5, 0.02, ny, nx, nz)
    return dict(H=H, E=E, E_prev=E + 0.01 * _randn(g, ny, nx, nz), H_prev=H * rnd(0.98, 1.02, ny, nx),
                u3d=100.0 / YEAR * _randn(g, nz, ny, nx + 1), v3d=100.0 / YEAR * _randn(g, nz, ny + 1, nx),
                omega=0.3 / YEAR * _randn(g, ny, nx, nz), f_E=1e-6 * _randn(g, ny, nx, nz) * (sig < 1.0),
                E_s=Ep[:, :, -1] - rnd(0.1, 0.4, ny, nx))


# ------------------------------------------------------------------------------------------------ prepare
PARAMS = (("bed", "geometry"), ("B", "rheology"), ("beta", "sliding"), ("smb", "forcing"))


def _model(case, f):
    from glide_b200.model import IceDynamics
    m = IceDynamics(n_levels=case["levels"], ny=case["ny"], nx=case["nx"], dx=case["dx"], precision=case["precision"],
                    reference_quirks=case["quirks"])
    for k, group in PARAMS:
        getattr(getattr(m.mg, group), k).set(f[k])
    m.mg.state.H.set(f["H"])
    m.mg.state.H_prev.set(f["H_prev"])
    fast = case["form"] == "fast"
    rtol = 1e-8 if fast and case["kind"] != "group" else 0.0
    for solver in (m.forward_solver, m.adjoint_solver):
        solver.fas_options.set(maximum_vcycles=case["vcycles"], relative_tolerance=rtol, absolute_tolerance=0.0,
                               report_norms=False)
    if fast:
        from glide_b200.ensemble import CANDIDATES, apply_schedule
        apply_schedule(m, CANDIDATES["fast"])
        m.mg.hierarchy.set_tuning(mixed_inner_vcycles=2)
        m.adjoint_solver.fas_options.set(pre_steps=4, post_steps=4, finest_steps=0, coarsest_steps=50)
        m.adjoint_solver.vanka_options.set(omega=0.8)
    return m


def _start(m, f, case):
    """The state a step starts from.  A dome has taken two steps from rest, as in a time loop."""
    if case["shape"] == "dome":
        for _ in range(2):
            m.forward(0.0, case["dt"])
    s = m.mg[0].state
    return {k: getattr(s, k).data.clone() for k in ("u", "v", "H", "mask")}


def _set_start(m, s):
    for k in ("u", "v", "H", "mask"):
        getattr(m.mg.state, k).set(s[k])
    m.mg.state.H_prev.set(s["H"])


class _State(dict):
    """What a program keeps between calls.  The tensors that alias a solver's memory keep its handle alive, and the
    handle keeps them: dropping the state drops them, so that the memory goes back."""

    def __del__(self):
        for owner in self.get("owners", ()):
            owner._views.clear()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "operator":
        from glide_b200.multigrid import Multigrid
        f = _operator_inputs(case, seed)
        mg = Multigrid(1, ny=case["ny"], nx=case["nx"], dx=case["dx"],
                       dtype=torch.float32 if case["precision"] == "fp32" else torch.float64)
        for k, group in PARAMS:
            getattr(getattr(mg, group), k).set(f[k])
        for k in ("u", "v", "H", "H_prev", "mask"):
            getattr(mg.state, k).set(f[k])
        ops = mg[0].forward_operators
        ops.set_rhs(case["dt"])
        if case["op"] == "jvp":
            for k in "uvH":
                getattr(ops, "var_" + k).copy_(f["e_" + k])
        elif case["op"] == "vjp":
            ops.compute_phi()
            for k in "uvH":
                getattr(mg.adjoint, "lambda_" + k).set(f["e_" + k])
        return _State(case=case, mg=mg, owners=[mg.hierarchy])
    if kind == "thermal":
        from glide_b200.grid import Grid
        from glide_b200.model import ThermalModel
        f = _thermal_inputs(case, seed)
        grid = Grid(case["ny"], case["nx"], case["dx"])
        for owner, k in ((grid.state, "u"), (grid.state, "v"), (grid.state, "H"), (grid.geometry, "bed"),
                         (grid.sliding, "beta"), (grid.rheology, "B")):
            getattr(owner, k).set(f[k])
        tm = ThermalModel(grid, nz=case["nz"])
        tm.initialize(f["T_s"], T_field=f["T"], Q_geo=0.05)
        return _State(case=case, tm=tm, grid=grid, H0=f["H"], H1=f["H1"], T_s=f["T_s"], E0=tm.enthalpy.clone(),
                      owners=[grid._hier, tm.ops])
    if kind == "columns":
        from glide_b200.enthalpy import EnthalpyOperators
        from glide_b200.grid import Grid
        f = _column_inputs(case, seed)
        grid = Grid(case["ny"], case["nx"], case["dx"])
        grid.state.H.set(f["H"])
        ops = EnthalpyOperators(grid, nz=case["nz"])
        ops.enthalpy_state.E_prev[:] = f["E_prev"]
        ops.f_E[:] = f["f_E"]
        ops.H_prev[:] = f["H_prev"]
        ops.enthalpy_velocity.u3d[:] = f["u3d"]
        ops.enthalpy_velocity.v3d[:] = f["v3d"]
        ops.enthalpy_velocity.omega[:] = f["omega"]
        ops.enthalpy_forcing.E_surface[:] = f["E_s"]
        ops.smoother_config.relative_tolerance = 1e-30
        ops.smoother_config.absolute_tolerance = 0.0
        return _State(case=case, ops=ops, E0=ops.enthalpy_state.E.copy_(f["E"]).clone(), owners=[grid._hier, ops])
    if kind == "group":
        from glide_b200.group import HierarchyGroup
        members = []
        for q in range(case["members"]):
            f = _fields(case, _gen(seed * 131 + q))
            m = _model(case, f)
            members.append((m, _start(m, f, case)))
        owners = [m.mg.hierarchy for m, _ in members]
        return _State(case=case, members=members, group=HierarchyGroup(owners), owners=owners)
    g = _gen(seed)
    f = _fields(case, g)
    m = _model(case, f)
    start = _start(m, f, case)
    state = _State(case=case, model=m, start=start, owners=[m.mg.hierarchy])
    if kind in ("gradient", "step"):
        u, v = start["u"], start["v"]
        state["obs"] = (u * (1.0 + 0.1 * _randn(g, *u.shape)), v * (1.0 + 0.1 * _randn(g, *v.shape)))
    if kind == "gradient":
        if case["shape"] != "dome":
            m.forward(0.0, case["dt"])
        state["dJ"] = tuple(x.data - o for x, o in zip((m.mg[0].state.u, m.mg[0].state.v), state["obs"]))
    if kind == "step":
        state["inputs"] = [t.clone().requires_grad_() for t in (start["H"], f["bed"], f["beta"], f["smb"])]
    return state


# ------------------------------------------------------------------------------------------------ run
def run(state):
    case = state["case"]
    kind, dt = case["kind"], case["dt"]
    if kind == "operator":
        mg = state["mg"]
        ops = mg[0].forward_operators
        if case["op"] == "residual":
            norms = ops.compute_residual(dt, return_norms=True)
            return dict(u=ops.r_u, v=ops.r_v, H=ops.r_H, norms=list(norms))
        if case["op"] == "jvp":
            ops.compute_jvp(dt)
            return dict(u=ops.jvp_u, v=ops.jvp_v, H=ops.jvp_H)
        adj = mg[0].adjoint_operators
        adj.compute_vjp(dt)
        return dict(u=adj.vjp_u, v=adj.vjp_v, H=adj.vjp_H)
    if kind == "thermal":
        tm, grid = state["tm"], state["grid"]
        grid.state.H.set(state["H0"])
        tm.enthalpy.copy_(state["E0"])
        tm.pre_momentum()
        grid.state.H.set(state["H1"])  # what the momentum step between them returns
        tm.ops.set_surface_enthalpy_from_temperature(state["T_s"])
        tm.step(dt * YEAR)
        return dict(E=tm.enthalpy, B=grid.rheology.B.data)
    if kind == "columns":
        ops = state["ops"]
        ops.enthalpy_state.E.copy_(state["E0"])
        ops.column_sweep(dt * YEAR, case["sweeps"])
        return ops.enthalpy_state.E
    if kind == "group":
        from glide_b200 import _lib
        for m, s in state["members"]:
            _set_start(m, s)
        state["group"].forward(dt)
        for m, _ in state["members"]:
            st = m.mg[0].state
            m.prepare_backward(0.05 * st.u.data, 0.05 * st.v.data)
        state["group"].backward(dt, mask=_lib.GRAD_ALL)
        return [dict(u=m.mg[0].state.u.data, v=m.mg[0].state.v.data, H=m.mg[0].state.H.data,
                     beta=m.mg[0].sliding.beta.grad, bed=m.mg[0].geometry.bed.grad) for m, _ in state["members"]]
    m = state["model"]
    lev = m.mg[0]
    if kind == "forward":
        _set_start(m, state["start"])
        m.forward(0.0, dt, update_geometry=False)
        return dict(u=lev.state.u.data, v=lev.state.v.data, H=lev.state.H.data)
    if kind == "gradient":
        for k in ("lambda_u", "lambda_v", "lambda_H"):
            getattr(m.mg.adjoint, k).set(0.0)
        m.backward(0.0, dt, dJdu=state["dJ"][0], dJdv=state["dJ"][1])
        return dict(beta=lev.sliding.beta.grad, bed=lev.geometry.bed.grad, H_prev=lev.state.H_prev.grad,
                    smb=lev.forcing.smb.grad)
    from glide_b200.torch import GlideStep
    for k in ("u", "v", "mask"):
        getattr(m.mg.state, k).set(state["start"][k])
    u, v, H = GlideStep.apply(0.0, dt, m, 0, *state["inputs"])
    uo, vo = state["obs"]
    loss = 0.5 * ((u - uo).square().sum() + (v - vo).square().sum())
    grads = torch.autograd.grad(loss, state["inputs"])
    return dict(u=u.detach(), v=v.detach(), H=H.detach(), H_prev=grads[0], bed=grads[1], beta=grads[2], smb=grads[3])


# ------------------------------------------------------------------------------------------------ work
def _cells(case, all_levels=False):
    n = case["ny"] * case["nx"]
    return n * (4.0 / 3.0) if all_levels else float(n)


def work(case):
    """Bytes: each input and output once.  Flops: one evaluation of the operator per row, node or smoother
    application that the options ask for (about 250 a cell for the residual, 450 for a Jacobian product or its
    transpose, 100 a node and pass for the enthalpy rows, 700 a cell for a Vanka block with its local solve)."""
    n, kind = _cells(case), case["kind"]
    s = 4 if case.get("precision") == "fp32" else 8
    if kind == "operator":
        arrays, flops = {"residual": (13, 250), "jvp": (14, 450), "vjp": (14, 450)}[case["op"]]
        return dict(bytes=arrays * n * s, flops=flops * n)
    if kind == "thermal":
        return dict(bytes=8 * n * (3 * case["nz"] + 8), flops=100 * 6 * n * case["nz"])
    if kind == "columns":
        return dict(bytes=8 * n * (7 * case["nz"] + 4), flops=100 * (5 * case["sweeps"] + 1) * n * case["nz"])
    arrays = dict(forward=5 + 5 + 3, gradient=10 + 2 + 4, step=5 + 5 + 2 + 7, group=5 + 5 + 5)[kind]
    members = case.get("members", 1)
    # fine-level smoother applications: fixed by the schedule; a solve to tolerance takes about seven cycles
    if case["form"] == "reference":
        sweeps, each = 80 * case["vcycles"], 700 if kind == "forward" else 500
        flops = each * sweeps * n + each * 30 * case["vcycles"] * (_cells(case, True) - n)
    else:
        cycles = case["vcycles"] if kind == "group" else 7
        flops = 500 * 8 * cycles * _cells(case, True) * (2 if kind in ("step", "group", "gradient") else 1)
    return dict(bytes=arrays * n * s * members, flops=flops * members)


# ------------------------------------------------------------------------------------------------ tolerance
def tolerance(case):
    """About four times what was seen: operators and columns against `exact`, fixed numbers of cycles with inputs
    moved by a rounding error, solves to 1e-8 against the same solve to 1e-11."""
    kind, precision = case["kind"], case.get("precision", "fp64")
    if kind == "operator":  # the residual's rows cancel, the more the finer the grid
        if precision == "fp64":
            return dict(rel=1e-13, max=1e-12)
        return dict(rel=1e-5, max=1e-4) if case["op"] == "residual" else dict(rel=5e-7, max=5e-6)
    if kind == "thermal":
        return dict(rel=1e-14, max=5e-13)
    if kind == "columns":
        return dict(rel=5e-14, max=4e-11)
    if case["form"] == "fast" and kind != "group":
        return dict(rel=1e-8, max=4e-7) if kind == "forward" else dict(rel=1e-7, max=4e-6)
    if precision == "fp32":
        return dict(rel=8e-5, max=2e-3)
    if precision == "mixed":  # binary32 corrections of a fixed number of cycles
        return dict(rel=1e-7, max=4e-6)
    return dict(rel=1e-12, max=1e-11)


# ------------------------------------------------------------------------------------------------ exact
def exact(case, seed):
    kind = case["kind"]
    if kind == "operator":
        f = {k: t.double() for k, t in _operator_inputs(case, seed).items()}
        return _exact_operator(case, f)
    if kind == "thermal":
        return _exact_thermal(case, _thermal_inputs(case, seed))
    if kind == "columns":
        f = _column_inputs(case, seed)
        p = _Columns(case["dx"], case["dt"] * YEAR, f["H"], f["H_prev"], f["E_prev"], f["f_E"], f["omega"], f["E_s"],
                     f["u3d"], f["v3d"])
        return p.sweeps(f["E"], case["sweeps"], 1e-30, 0.0)
    return None  # iterative solves: minutes in plain torch


def _ssa_rows(case, f, u, v, H, phi):
    """(viscous momentum rows, other momentum rows, mass row) of the coupled operator without forcing; the
    interior faces only."""
    dxi = 1.0 / case["dx"]
    ux, vy = (u[:, 1:] - u[:, :-1]) * dxi, (v[:-1] - v[1:]) * dxi
    pad = torch.nn.functional.pad
    shear = pad(0.5 * ((u[:-1, 1:-1] - u[1:, 1:-1]) + (v[1:-1, 1:] - v[1:-1, :-1])) * dxi, (1, 1, 1, 1))
    s2 = shear * shear
    eII = ux * ux + vy * vy + ux * vy + 0.25 * (s2[:-1, :-1] + s2[:-1, 1:] + s2[1:, :-1] + s2[1:, 1:]) + 1e-6
    etaH = 0.5 * f["B"] * eII ** (-1.0 / 3.0) * H

    def visc(etaH):
        sx, sy = 2 * etaH * (2 * ux + vy), 2 * etaH * (ux + 2 * vy)
        eHv = pad(0.25 * (etaH[:-1, :-1] + etaH[:-1, 1:] + etaH[1:, :-1] + etaH[1:, 1:]), (1, 1, 1, 1))
        t = 2 * eHv * shear
        return (dxi * (sx[:, 1:] - sx[:, :-1] + t[:-1, 1:-1] - t[1:, 1:-1]),
                dxi * (sy[:-1] - sy[1:] - t[1:-1, :-1] + t[1:-1, 1:]))

    bp = f["beta"] * phi
    S = phi * f["bed"] - (1.0 - phi) * FLOT * H + H
    ru = -(0.5 * (bp[:, :-1] + bp[:, 1:]) + 1e-5) * u[:, 1:-1] \
        - 0.5 * (H[:, :-1] + H[:, 1:]) * (S[:, 1:] - S[:, :-1]) * dxi
    rv = -(0.5 * (bp[:-1] + bp[1:]) + 1e-5) * v[1:-1] - 0.5 * (H[:-1] + H[1:]) * (S[:-1] - S[1:]) * dxi
    w = u[:, 1:-1]
    qu = pad(0.5 * (H[:, :-1] + H[:, 1:]) * w - 0.5 * torch.sqrt(w * w + 10.0) * (H[:, 1:] - H[:, :-1]), (1, 1, 0, 0))
    w = v[1:-1]
    qv = pad(0.5 * (H[:-1] + H[1:]) * w - 0.5 * torch.sqrt(w * w + 10.0) * (H[:-1] - H[1:]), (0, 0, 1, 1))
    rH = H / case["dt"] + dxi * (qu[:, 1:] - qu[:, :-1] + qv[:-1] - qv[1:])
    return visc, etaH, (ru, rv), rH


def _exact_operator(case, f):
    phi = torch.sigmoid(torch.clamp(0.1 * (f["bed"] + FLOT * f["H"]), -20.0, 20.0))
    mask = f["mask"]

    def rows(u, v, H):
        visc, etaH, (ru, rv), rH = _ssa_rows(case, f, u, v, H, phi)
        a, b = visc(etaH)
        return a + ru, b + rv, rH

    x = (f["u"], f["v"], f["H"])
    e = (f["e_u"], f["e_v"], f["e_H"])
    if case["op"] == "residual":
        ru, rv, rH = rows(*x)
        o_u, o_v = f["u"].clone(), f["v"].clone()
        o_u[:, 1:-1], o_v[1:-1] = ru, rv
        o_H = rH - f["H_prev"] / case["dt"] - f["smb"]
        o_H = (1.0 - mask) * o_H + mask * (f["H"] - THKLIM)
        return dict(u=o_u, v=o_v, H=o_H, norms=[float(t.square().sum().sqrt()) for t in (o_u, o_v, o_H)])
    o_u, o_v = torch.zeros_like(f["u"]), torch.zeros_like(f["v"])
    if case["op"] == "jvp":
        _, (ru, rv, rH) = torch.func.jvp(rows, x, e)
        o_u[:, 1:-1], o_v[1:-1] = ru, rv
        return dict(u=o_u, v=o_v, H=(1.0 - mask) * rH)

    # The transposed product as the operator defines it: the viscous block is its forward derivative along
    # lambda (the block is symmetric), everything else is transposed.
    def viscous(u, v):
        visc, etaH, _, _ = _ssa_rows(case, f, u, v, f["H"], phi)
        return visc(etaH)

    lu, lv, lH = e[0][:, 1:-1], e[1][1:-1], e[2] * (1.0 - mask)
    _, (vu, vv) = torch.func.jvp(viscous, x[:2], e[:2])
    u, v, H = (t.clone().requires_grad_() for t in x)
    visc, etaH, (ru, rv), rH = _ssa_rows(case, f, u, v, H, phi)
    eta = (etaH / H).detach()
    su, sv = _ssa_rows(case, f, f["u"], f["v"], f["H"], phi)[0](eta * H)
    dot = (ru * lu).sum() + (rv * lv).sum() + (rH * lH).sum() + (su * lu).sum() + (sv * lv).sum()
    gu, gv, gH = torch.autograd.grad(dot, (u, v, H))
    o_u[:, 1:-1] = gu[:, 1:-1] + vu
    o_v[1:-1] = gv[1:-1] + vv
    return dict(u=o_u, v=o_v, H=torch.where(mask > 0, torch.zeros_like(gH), gH))


# Enthalpy columns: the constants are binary32 literals of the operator, their products formed in binary32.
def _f32(x):
    return float(torch.tensor(x, dtype=torch.float32))


_RHO, _CI, _L, _KTF, _SHARP = 910.0, 2009.0, 334000.0, _f32(0.1), _f32(0.01)
_TR, _TM, _REG = _f32(223.15), _f32(273.15), _f32(1.00413490930961e-14)
_ESC = float(torch.tensor(2009.0, dtype=torch.float32) * (torch.tensor(273.15) - torch.tensor(223.15)))
_KC = float(torch.tensor(2.1) / torch.tensor(2009.0))
_CC = float(torch.tensor(7.9e-08) * torch.tensor(910.0) * torch.tensor(9.81))


def _e_pmp(sig, H):
    return (_TM - _CC * (1.0 - sig) * H - _TR) * (_CI / _ESC)


def _switch(z):
    return 1.0 / (1.0 + torch.exp(-z.clamp(-20.0, 20.0)))


class _Columns:
    """Residual, column Newton/Thomas and layer smoothers of the enthalpy equation on (ny, nx, nz) arrays."""

    def __init__(self, dx, dt, H, H_prev, E_prev, f_E, omega, E_s, u3d, v3d):
        self.dt, self.H, self.Hp, self.Ep, self.f, self.E_s = dt, H, H_prev, E_prev, f_E, E_s
        self.nz = E_prev.shape[2]
        self.ds = 1.0 / (self.nz - 1)
        self.dxi, self.drain = 1.0 / dx, 0.01 / YEAR
        self.om = omega
        sig = torch.linspace(0.0, 1.0, self.nz, device="cuda", dtype=torch.float64)
        self.pmp = _e_pmp(sig, H[:, :, None])
        self.thin = H < 25.0
        pad = torch.nn.functional.pad
        u, v = u3d[:, :, 1:-1].permute(1, 2, 0), v3d[:, 1:-1, :].permute(1, 2, 0)
        Hc = H[:, :, None]
        qx = 0.5 * (Hc[:, :-1] + Hc[:, 1:]) * u - 0.5 * torch.sqrt(u * u + _REG) * (Hc[:, 1:] - Hc[:, :-1])
        qy = 0.5 * (Hc[:-1] + Hc[1:]) * v - 0.5 * torch.sqrt(v * v + _REG) * (Hc[:-1] - Hc[1:])
        self.qx, self.qy = pad(qx, (0, 0, 1, 1)), pad(qy, (0, 0, 0, 0, 1, 1))  # zero on the domain edge
        self.sq = math.sqrt(1.0 + 1e-12)

    def _horiz(self, E, frozen):
        """Horizontal advection with centre values E and neighbours `frozen`, and its diagonal."""
        def flux(q, a, b):
            return 0.5 * q * (a + b) - 0.5 * q.abs() * self.sq * (b - a)
        pad = torch.nn.functional.pad
        F = pad(frozen.permute(2, 0, 1)[None], (1, 1, 1, 1), mode="replicate")[0].permute(1, 2, 0)
        ql, qr, qt, qb = self.qx[:, :-1], self.qx[:, 1:], self.qy[:-1], self.qy[1:]
        fl, fr = flux(ql, F[1:-1, :-2], E), flux(qr, E, F[1:-1, 2:])
        ft, fb = flux(qt, E, F[:-2, 1:-1]), flux(qb, F[2:, 1:-1], E)
        a = [q.abs() * self.sq for q in (ql, qr, qt, qb)]
        diag = 0.5 * ((qr + a[1]) - (ql - a[0]) + (qt + a[2]) - (qb - a[3]))
        return _RHO * (fr - fl + ft - fb) * self.dxi, _RHO * diag * self.dxi

    def rows(self, E, frozen):
        """Residual of rows 0..nz-2 and their tridiagonal coefficients."""
        H, h_inv, ds = self.H[:, :, None], 1.0 / self.H[:, :, None], self.ds
        k0, k1 = E[:, :, :-1], E[:, :, 1:]
        x = (0.5 * (k0 + k1) - 0.5 * (self.pmp[:, :, :-1] + self.pmp[:, :, 1:])) * _ESC * _SHARP
        s = _switch(x)
        K = _KC * (1.0 - s + _KTF * s)
        w = 0.5 * (self.om[:, :, :-1] + self.om[:, :, 1:])
        wp, wn = w.clamp(min=0.0), w.clamp(max=0.0)
        zero = torch.zeros_like(K[:, :, :1])
        below = lambda t, first: torch.cat([first, t[:, :, :-1]], 2)  # noqa: E731
        cell = torch.full((self.nz - 1,), ds, device="cuda", dtype=torch.float64)
        cell[0] = 0.5 * ds
        F = wp * k0 + wn * k1
        adv = _RHO * (F - below(F, self.om[:, :, :1] * E[:, :, :1])) / cell
        D = h_inv * K * (k1 - k0) / ds
        dif = -(D - below(D, zero)) / cell
        up, lo = h_inv * K / (ds * cell), below(h_inv * K, zero) / (ds * cell)
        a = -_RHO * below(wp, zero) / cell - lo
        c = _RHO * wn / cell - up
        b = up + lo + _RHO * (wp - below(wn, self.om[:, :, :1])) / cell
        xd = (k0 - self.pmp[:, :, :-1]) * _ESC
        ax = _SHARP * xd
        sp = torch.where(ax > 10.0, xd, torch.log1p(torch.exp(ax.clamp(-20.0, 10.0))) / _SHARP)
        drn = H * 1000.0 * _L * (self.drain * (sp / _L)) / _ESC
        b = b + H * 1000.0 * _L * self.drain * (_switch(ax) / _L)
        hr, hd = self._horiz(E, frozen)
        r = _RHO * (H * E - self.Hp[:, :, None] * self.Ep)[:, :, :-1] / self.dt + hr[:, :, :-1] + adv + dif + drn \
            - self.f[:, :, :-1]
        return r, a, b + hd[:, :, :-1] + _RHO * H / self.dt, c

    def norm(self, E):
        r = self.rows(E, E)[0].abs()
        return float(torch.where(self.thin[:, :, None], torch.zeros_like(r), r).max())

    def column(self, E):
        X = E.clone()
        for _ in range(3):
            r, a, b, c = self.rows(X, E)
            cp, dp = [], []
            for k in range(self.nz - 1):
                den = b[:, :, k] - (a[:, :, k] * cp[-1] if k else 0.0)
                cp.append(c[:, :, k] / den)
                dp.append((-r[:, :, k] - (a[:, :, k] * dp[-1] if k else 0.0)) / den)
            x = self.E_s - X[:, :, -1]
            X[:, :, -1] += x
            for k in range(self.nz - 2, -1, -1):
                x = dp[k] - cp[k] * x
                X[:, :, k] += x
        clamped = torch.minimum(self.E_s[:, :, None], self.pmp)
        return torch.where(self.thin[:, :, None], clamped, X)

    def layer(self, E):
        r, _, b, _ = self.rows(E, E)
        X = E.clone()
        X[:, :, :-1] -= r / b
        return torch.where(self.thin[:, :, None], E, X)

    def sweeps(self, E, n, rtol, atol):
        r0 = self.norm(E)
        for _ in range(n):
            E = self.layer(self.column(E))
            r = self.norm(E)
            if (r0 > 0 and r / r0 < rtol) or r < atol:
                break
        return E


def _exact_thermal(case, f):
    nz, esc = case["nz"], 2009.0 * 50.0
    H, u, v = f["H1"], f["u"], f["v"]
    sig = torch.linspace(0.0, 1.0, nz, device="cuda", dtype=torch.float64)
    melt = lambda h: 273.15 - 7.9e-8 * RHO_G * (1.0 - sig) * h[:, :, None]  # noqa: E731
    E = 2009.0 * (torch.minimum(f["T"], melt(f["H"])) - 223.15) / esc
    E_s = 2009.0 * (f["T_s"].clamp(max=273.15) - 223.15) / esc
    pad = torch.nn.functional.pad

    def flux(w, a, b):
        return 0.5 * (a + b) * w - 0.5 * torch.sqrt(w * w + 10.0) * (b - a)

    qx = pad(flux(u[:, 1:-1], H[:, :-1], H[:, 1:]), (1, 1, 0, 0))
    qy = pad(flux(v[1:-1], H[1:], H[:-1]), (0, 0, 1, 1))
    div = (qx[:, 1:] - qx[:, :-1] + qy[:-1] - qy[1:]) / case["dx"]
    rate = ((H - f["H"]) / case["dt"] + div)[:, :, None]
    omega = -rate * sig / YEAR
    omega = torch.where((H < 1e-3)[:, :, None], torch.zeros_like(omega), omega)
    us, vs = u / YEAR, v / YEAR
    uc, vc = 0.5 * (us[:, 1:] + us[:, :-1]), 0.5 * (vs[1:] + vs[:-1])
    Q = 0.05 + f["beta"] * (uc * uc + vc * vc + 1.0)
    f_E = torch.zeros_like(E)
    f_E[:, :, 0] = Q / (0.5 / (nz - 1) * esc)
    p = _Columns(case["dx"], case["dt"] * YEAR, H, f["H"], E, f_E, omega, E_s, us[None].expand(nz, -1, -1),
                 vs[None].expand(nz, -1, -1))
    E = p.sweeps(E, 10, 1e-5, 1e-2)
    T_m = melt(H)
    T = torch.minimum(E * esc / 2009.0 + 223.15, T_m)
    cold = T < 263.15
    A = torch.where(cold, 3.985e-13 * torch.exp(-60e3 / (8.314 * T)), 1.916e3 * torch.exp(-139e3 / (8.314 * T)))
    A = A * (1.0 + 181.25 * (E * esc - 2009.0 * (T_m - 223.15)).clamp(min=0.0) / 334000.0)
    return dict(E=E, B=A.mean(2) ** (-1.0 / 3.0) / (917.0 * 9.81 * YEAR ** (1.0 / 3.0)))
