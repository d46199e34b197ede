"""The marched linear operator (glide_b200/csrc/strip.cuh) where its strips and
chunks can go wrong: widths around the 27 and 28 owned columns and the 32 lanes, the
smallest levels, chunks of 2 to 32 rows at ragged heights, linear and nonlinear
sliding, calving on, both precisions.

- J^T lambda and the adjoint sweeps against the oracle (binary64 1e-12 for one
  product, 1e-10 for sweeps); J e against the oracle's residual by Richardson
  -extrapolated central differences: with steps h and h/2 of the relative size 1e-4
  their truncation is O(h^4) and their rounding eps / h = 1e-12 of the residual's
  terms, which the thin columns amplify; 1e-6 as for the solver tests.
- Binary32 against binary64 on inputs that are binary32 numbers.
- The tangent sweeps against their formula, block solves in numpy.
- Longer chunks (one row a warp more with every 2400 or 4800 warps the grid has)
  against two-row ones, bit for bit: the rows of a large grid and of one cut from it.
"""
from __future__ import annotations

import numpy as np
import pytest

from cases import random_state
from util import oracle_single_level, rel_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

DX, DT = 1500.0, 5.0
SIZES = [(2, 2), (3, 26), (4, 27), (5, 28), (9, 31), (17, 33), (34, 55), (66, 57)]
PHYS = [dict(calving_rate=2.0), dict(m=1.0 / 3.0)]


def _setup(ny, nx, phys, seed=0):
    from glide_b200.hierarchy import Hierarchy
    f = random_state(ny, nx, seed=7 * ny + nx + seed)
    rng = np.random.default_rng(ny + nx)
    lam = [rng.standard_normal(s) for s in ((ny, nx + 1), (ny + 1, nx), (ny, nx))]
    h = Hierarchy(ny, nx, DX, 1)
    for k in ("u", "v", "H", "H_prev", "mask", "bed", "B", "beta", "smb", "f_u", "f_v"):
        h.set(k, 0, torch.as_tensor(f[k]))
    o = oracle_single_level({f"in_{k}": a for k, a in f.items()}, DX)
    h.set_phys(-1, **phys)
    o.set_phys(**phys)
    h.compute_phi(0)
    o.levels[0].compute_phi()
    return h, o.levels[0], lam


@pytest.mark.parametrize("phys", PHYS)
@pytest.mark.parametrize("ny,nx", SIZES)
def test_transposed_product_and_sweeps_match_oracle(ny, nx, phys):
    h, lev, lam = _setup(ny, nx, phys)
    rng = np.random.default_rng(5)
    for q, k in enumerate("uvH"):
        rhs = rng.standard_normal(lam[q].shape)
        h.set("lambda_" + k, 0, torch.as_tensor(lam[q]))
        h.set("adj_f_" + k, 0, torch.as_tensor(rhs))
        getattr(lev, "l_" + k)[...] = lam[q]
        getattr(lev, "af_" + k)[...] = rhs
    h.vjp(0, DT)
    for a in (lev.vjp_u, lev.vjp_v, lev.vjp_H):
        a.fill(0)
    lev.adj_vjp(DT)
    for k in "uvH":
        assert rel_err(h.view("vjp_" + k, 0).cpu().numpy(), getattr(lev, "vjp_" + k)) <= 1e-12, k
    for n in (3, 2, 1):  # fused in pairs; the last of an odd count is a product and a block solve
        h.adjoint_sweep(0, DT, n)
        lev.adj_sweep(DT, n)
        for k in "uvH":
            assert rel_err(h.view("lambda_" + k, 0).cpu().numpy(), getattr(lev, "l_" + k)) <= 1e-10, (n, k)
            # the residual the last sweep started from stays readable
            assert rel_err(h.view("adj_r_" + k, 0).cpu().numpy(), getattr(lev, "ar_" + k)) <= 1e-10, (n, k)


@pytest.mark.parametrize("phys", PHYS)
@pytest.mark.parametrize("ny,nx", SIZES)
def test_jacobian_product_matches_differences(ny, nx, phys):
    h, lev, e = _setup(ny, nx, phys, seed=1)
    e[0][:, [0, -1]] = 0.0
    e[1][[0, -1]] = 0.0
    for q, k in enumerate("uvH"):
        h.set("var_" + k, 0, torch.as_tensor(e[q]))
    h.jvp(0, DT, reference_rows=True, flags=0)
    base = [lev.u.copy(), lev.v.copy(), lev.H.copy()]
    phi = lev.phi.copy()

    def rows(s):
        lev.u[...], lev.v[...], lev.H[...] = (b + s * d for b, d in zip(base, e))
        lev.phi[...] = phi
        return [a.copy() for a in lev.residual(DT, use_mask=False, operator_only=True, freeze_phi=True)]

    def diff(s):
        return [(a - b) / (2 * s) for a, b in zip(rows(s), rows(-s))]

    s = 2e-3
    want = [(4 * b - a) / 3 for a, b in zip(diff(s), diff(s / 2))]
    want[0][:, [0, -1]] = 0.0  # pinned rows are zero in the reference's convention
    want[1][[0, -1]] = 0.0
    for k, w in zip("uvH", want):
        assert rel_err(h.view("jvp_" + k, 0).cpu().numpy(), w) <= 1e-6, k


@pytest.mark.parametrize("m", [0.2, 2.9, 4.0])
def test_sliding_exponents(m):
    """The power of the sliding law on both sides of |e| = |m - 1| / 2 = 1, where its evaluation changes, at velocities
    of 1e-4 to 1e4 m/a.  J^T lambda against the oracle; J e without ice (H = e_H = 0 leaves the drag alone) against its
    formula in extended precision: 1e-14 of the terms' sizes, a dozen binary64 roundings and the power's 2.4e-16."""
    ny, nx = 17, 33
    h, lev, lam = _setup(ny, nx, dict(m=m))
    rng = np.random.default_rng(9)
    vel = {}
    for q, (k, s) in enumerate((("u", (ny, nx + 1)), ("v", (ny + 1, nx)), ("H", (ny, nx)))):
        if k != "H":
            vel[k] = rng.choice([-1.0, 1.0], s) * 10.0 ** rng.uniform(-4, 4, s)
            h.set(k, 0, torch.as_tensor(vel[k]))
            getattr(lev, k)[...] = vel[k]
        h.set("lambda_" + k, 0, torch.as_tensor(lam[q]))
        getattr(lev, "l_" + k)[...] = lam[q]
    h.vjp(0, DT)
    for a in (lev.vjp_u, lev.vjp_v, lev.vjp_H):
        a.fill(0)
    lev.adj_vjp(DT)
    for k in "uvH":
        assert rel_err(h.view("vjp_" + k, 0).cpu().numpy(), getattr(lev, "vjp_" + k)) <= 1e-12, k

    h.set("H", 0, 0.0)
    h.set("var_u", 0, torch.as_tensor(lam[0]))
    h.set("var_v", 0, torch.as_tensor(lam[1]))
    h.set("var_H", 0, 0.0)
    h.jvp(0, DT, reference_rows=True, flags=0)
    X = np.longdouble
    u, v, eu, ev = (X(a) for a in (vel["u"], vel["v"], lam[0], lam[1]))
    bp = X(h.get("beta", 0).cpu().numpy() * h.get("phi", 0).cpu().numpy())
    ph = h.get_phys(0)
    e, reg, wd = (X(m) - 1) / 2, X(ph["u_reg"]), X(ph["water_drag"])

    def drag(w, c, dw, dc, be):  # face velocity, the four corners, their directions
        q = w * w + sum(x * x for x in c) / 4 + reg
        p, s = q ** e, e * q ** (e - 1)
        t = [be * 2 * s * w * w * dw, be * p * dw, wd * dw] + [be * s / 2 * w * x * d for x, d in zip(c, dc)]
        return -sum(t), sum(abs(x) for x in t)

    def corners(a):
        return a[:-1, :-1], a[:-1, 1:], a[1:, :-1], a[1:, 1:]

    want, size = drag(u[:, 1:-1], corners(v), eu[:, 1:-1], corners(ev), (bp[:, :-1] + bp[:, 1:]) / 2)
    assert np.all(abs(h.get("jvp_u", 0).cpu().numpy()[:, 1:-1] - want) <= 1e-14 * size)
    want, size = drag(v[1:-1], corners(u), ev[1:-1], corners(eu), (bp[:-1] + bp[1:]) / 2)
    assert np.all(abs(h.get("jvp_v", 0).cpu().numpy()[1:-1] - want) <= 1e-14 * size)


def test_sliding_power_at_rest():
    """u = v = 0 and u_reg = 0 with m = 3: the drag and its derivative are zero, as if there were no drag at all."""
    out = []
    for m, beta in ((3.0, None), (1.0, 0.0)):
        h, lev, e = _setup(9, 31, dict(m=m, u_reg=0.0))
        if beta is not None:
            h.set("beta", 0, beta)
        h.set("u", 0, 0.0)
        h.set("v", 0, 0.0)
        for q, k in enumerate("uvH"):
            h.set("var_" + k, 0, torch.as_tensor(e[q]))
        h.jvp(0, DT, reference_rows=True, flags=0)
        out.append([h.get("jvp_" + k, 0).cpu().numpy() for k in "uvH"])
    for a, b in zip(*out):
        assert rel_err(a, b) <= 1e-14


def _load(f, dtype, phys, lam, rhs=None, mask=None):
    from glide_b200.hierarchy import Hierarchy
    h = Hierarchy(*f["H"].shape, DX, 1, dtype=dtype)
    for k in ("u", "v", "H", "H_prev", "mask", "bed", "B", "beta", "smb", "f_u", "f_v"):
        h.set(k, 0, torch.as_tensor(f[k]))
    h.set_phys(-1, **phys)
    h.compute_phi(0)
    for q, k in enumerate("uvH"):
        h.set("var_" + k, 0, torch.as_tensor(lam[q]))
        h.set("lambda_" + k, 0, torch.as_tensor(lam[q]))
        if rhs is not None:
            h.set("adj_f_" + k, 0, torch.as_tensor(rhs[q]))
    return h


def _inputs(ny, nx, seed=0):
    """State, direction and right-hand side, all of them binary32 numbers; velocities of 5 m/a."""
    f = random_state(ny, nx, seed=7 * ny + nx + seed)
    f["u"], f["v"] = 0.1 * f["u"], 0.1 * f["v"]
    rng = np.random.default_rng(ny + nx)
    shapes = ((ny, nx + 1), (ny + 1, nx), (ny, nx))
    r32 = lambda a: np.asarray(a, np.float32).astype(np.float64)
    return ({k: r32(a) for k, a in f.items()}, [r32(rng.standard_normal(s)) for s in shapes],
            [r32(rng.standard_normal(s)) for s in shapes])


def _get(h, prefix):
    return [h.get(prefix + k, 0).double().cpu().numpy() for k in "uvH"]


@pytest.mark.parametrize("phys", PHYS)
@pytest.mark.parametrize("ny,nx", SIZES + [(701, 611)])
def test_binary32_matches_binary64(ny, nx, phys):
    """Products: sums of a few dozen binary32 terms, 5e-6 of the largest value as for the operator cases (the rows cancel);
    two sweeps: the factors' and the block solves' rounding on top, 2e-4, the bar of the binary32 solves."""
    f, lam, rhs = _inputs(ny, nx)
    a, b = (_load(f, t, phys, lam, rhs) for t in (torch.float32, torch.float64))
    a.set("phi", 0, b.get("phi", 0))
    b.set("phi", 0, a.get("phi", 0).double())
    for rows in (True, False):
        for h in (a, b):
            h.jvp(0, DT, reference_rows=rows)
        for x, y in zip(_get(a, "jvp_"), _get(b, "jvp_")):
            assert rel_err(x, y) <= 5e-6, rows
    for h in (a, b):
        h.vjp(0, DT)
    for x, y in zip(_get(a, "vjp_"), _get(b, "vjp_")):
        assert rel_err(x, y) <= 5e-6
    for h in (a, b):
        h.set_vanka(True, -1, omega=0.5)
        h.adjoint_sweep(0, DT, 2)
    for x, y in zip(_get(a, "lambda_"), _get(b, "lambda_")):
        assert np.isfinite(x).all() and rel_err(x, y) <= 2e-4


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("ny,nx", SIZES)
def test_pinned_rows_of_the_tangent(ny, nx, dtype):
    """J e with the solver's rows: e itself on the Dirichlet faces and the active cells, the unmasked product elsewhere;
    with the reference's rows: zero on them."""
    f, lam, _ = _inputs(ny, nx, seed=2)
    h = _load(f, dtype, PHYS[0], lam)
    h.jvp(0, DT, reference_rows=True, flags=0)
    free = _get(h, "jvp_")
    on = f["mask"] > 0.5
    for rows in (False, True):
        h.jvp(0, DT, reference_rows=rows)
        got = _get(h, "jvp_")
        want = [a.copy() for a in free]
        want[0][:, [0, -1]] = 0.0 if rows else lam[0][:, [0, -1]]
        want[1][[0, -1]] = 0.0 if rows else lam[1][[0, -1]]
        want[2][on] = 0.0 if rows else lam[2][on]
        for g, w in zip(got, want):
            np.testing.assert_array_equal(g, w)


@pytest.mark.parametrize("ny,nx", SIZES + [(463, 451), (701, 611)])
def test_norms_are_those_of_the_rows(ny, nx):
    f, lam, rhs = _inputs(ny, nx)
    for dtype in (torch.float64, torch.float32):
        h = _load(f, dtype, PHYS[0], lam, rhs)
        norms = h.adjoint_residual(0, DT, norms=True)
        for n, r in zip(norms, _get(h, "adj_r_")):
            assert abs(n - np.linalg.norm(r)) <= 1e-12 * n  # the same numbers, summed in another order


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("ny,nx,rows64,rows32", [(463, 451, 3, 2), (701, 611, 6, 3), (1501, 1403, 31, 15)])
def test_long_chunks_equal_short_ones(ny, nx, rows64, rows32, dtype):
    cols = (nx + 28) // 28
    for r, warps in ((rows64, 2400), (rows32, 4800)):
        assert min(32, max(2, ny * cols // warps)) == r  # what the launches below take
    f, lam, rhs = _inputs(ny, nx)
    my, mx = 150, 170
    cut = lambda q, a: a[:my + (q == 1), :mx + (q == 0)].copy()
    side = lambda k: dict(u=0, f_u=0, v=1, f_v=1).get(k, 2)
    small = ({k: cut(side(k), a) for k, a in f.items()}, [cut(q, a) for q, a in enumerate(lam)],
             [cut(q, a) for q, a in enumerate(rhs)])
    out = []
    for g, l, r in ((f, lam, rhs), small):
        h = _load(g, dtype, PHYS[0], l, r)
        h.jvp(0, DT, reference_rows=False)
        h.vjp(0, DT)
        got = _get(h, "jvp_") + _get(h, "vjp_")
        h.adjoint_sweep(0, DT, 4)
        out.append(got + _get(h, "lambda_"))
    for a, b in zip(*out):
        # two cells from the cut for a product, three a sweep
        np.testing.assert_array_equal(a[:my - 13, :mx - 13], b[:my - 13, :mx - 13])


def _tangent_reference(h, f, n, omega, bf16):
    """e after n block-smoother sweeps of J e = -r from e = 0 at the state of `f`, as Solver::newton_cycle solves it:
    e -= omega (the two cells' mean of B^-1 (J e + r)), B the damped local Newton matrix with pinned rows."""
    ny, nx = f["H"].shape
    h.set_rhs(0, DT)
    h.residual(0, DT, 0)
    r = [h.get("r_" + k, 0).cpu().numpy() for k in "uvH"]
    gamma, H = h.get("gamma", 0).cpu().numpy(), f["H"]
    on = H - DT * r[2] <= gamma
    h.set("mask", 0, torch.as_tensor(on.astype(float)))
    rhs = [-r[0], -r[1], np.where(on, -(H - gamma), -r[2])]
    J = h.vanka_dump(0, DT)[0].cpu().numpy().reshape(ny, nx, 5, 5)
    c = h.get_vanka(2, 0)
    pin = np.zeros((ny, nx, 5), bool)
    pin[:, 0, 0] = pin[:, -1, 1] = pin[0, :, 2] = pin[-1, :, 3] = True
    pin[..., 4] = on
    for k, d in enumerate([-c["ssa_damping"]] * 4 + [c["mc_damping"]]):
        J[..., k, k] += np.where(pin[..., k], 0.0, d)
    M = J.copy()  # L below the diagonal, U above it, pivot reciprocals on it
    for k in range(5):
        inv = 1.0 / M[..., k, k]
        for q in range(k + 1, 5):
            M[..., q, k] *= inv
            M[..., q, k + 1:] -= M[..., q, k, None] * M[..., k, k + 1:]
        M[..., k, k] = inv
    if bf16:
        M = torch.as_tensor(M).float().bfloat16().double().numpy()
    e = [np.zeros((ny, nx + 1)), np.zeros((ny + 1, nx)), np.zeros((ny, nx))]
    for _ in range(n):
        for q, k in enumerate("uvH"):
            h.set("var_" + k, 0, torch.as_tensor(e[q]))
        h.jvp(0, DT, reference_rows=False)
        ru, rv, rH = (a - b for a, b in zip([h.get("jvp_" + k, 0).cpu().numpy() for k in "uvH"], rhs))
        x = np.stack([ru[:, :-1], ru[:, 1:], rv[:-1], rv[1:], rH], -1)
        for q in range(5):
            for p in range(q):
                x[..., q] -= M[..., q, p] * x[..., p]
        for q in range(4, -1, -1):
            for p in range(q + 1, 5):
                x[..., q] -= M[..., q, p] * x[..., p]
            x[..., q] *= M[..., q, q]
        e[0][:, :-1] -= omega * 0.5 * x[..., 0]
        e[0][:, 1:] -= omega * 0.5 * x[..., 1]
        e[1][:-1] -= omega * 0.5 * x[..., 2]
        e[1][1:] -= omega * 0.5 * x[..., 3]
        e[2] -= omega * x[..., 4]
    return e, gamma


@pytest.mark.parametrize("sweeps", [2, 3])
@pytest.mark.parametrize("precision,bar", [("fp64", 1e-12), ("fp32", 5e-5)])
@pytest.mark.parametrize("ny,nx", [(5, 28), (17, 33), (34, 55), (66, 57), (130, 84)])
def test_tangent_sweeps_match_block_solves(ny, nx, precision, bar, sweeps):
    """One Newton step of a one-level handle is `sweeps` tangent sweeps: two fused, a third unfused.  Bars of the largest
    correction: binary64 1e-12 (measured 2e-14), binary32 5e-5 (1e-5: its residual's cancelled terms).  Binary32 stores
    the factors as bfloat16, and so does the reference."""
    from glide_b200.hierarchy import Hierarchy
    f, _, _ = _inputs(ny, nx, seed=3)
    omega = 0.3
    # thick ice on a rough bed with an ice-free corner (active cells), a few nonlinear sweeps from rest
    rng = np.random.default_rng(ny * nx)
    f["H"] = np.float32(800.0 + 40.0 * rng.random((ny, nx))).astype(float)
    f["bed"] = np.float32(100.0 + 40.0 * rng.random((ny, nx))).astype(float)
    f["H"][:ny // 4, :nx // 3] = np.float32(0.1)
    f["smb"][:ny // 4, :nx // 3] = -1.0
    f["H_prev"] = f["H"].copy()
    settle = Hierarchy(ny, nx, DX, 1, dtype=torch.float32)
    for k in ("H", "H_prev", "bed", "B", "beta", "smb"):
        settle.set(k, 0, torch.as_tensor(f[k]))
    settle.set_rhs(0, DT)
    settle.vanka_sweep(0, DT, 10)
    for k in ("u", "v", "H"):
        f[k] = settle.get(k, 0).double().cpu().numpy()
    f["f_u"], f["f_v"] = np.zeros_like(f["f_u"]), np.zeros_like(f["f_v"])

    h = Hierarchy(ny, nx, DX, 1, precision=precision)
    for k in ("u", "v", "H", "H_prev", "mask", "bed", "B", "beta", "smb"):
        h.set(k, 0, torch.as_tensor(f[k]))
    h.set_tuning(forward_method="newton", newton_switch_exp10=0)
    h.set_fas(False, maximum_vcycles=1, relative_tolerance=1e-30, absolute_tolerance=0.0)
    h.set_fas(2, coarsest_steps=sweeps)
    h.set_vanka(2, -1, omega=omega)
    h.forward(DT, 0)
    ref = _load(f, torch.float64, {}, [np.zeros_like(f[k]) for k in "uvH"])
    ref.set_vanka(2, -1, omega=omega)
    e, gamma = _tangent_reference(ref, f, sweeps, omega, precision == "fp32")
    want = [f["u"] + e[0], f["v"] + e[1], np.maximum(f["H"] + e[2], gamma)]
    for k, w, step in zip("uvH", want, e):
        got = h.get(k, 0).double().cpu().numpy()
        assert np.abs(got - f[k]).max() > 0, "the step was undone"
        assert np.abs(got - w).max() <= bar * np.abs(step).max(), (k, np.abs(got - w).max() / np.abs(step).max())
