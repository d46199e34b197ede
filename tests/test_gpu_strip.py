"""The marched linear operator (glide_b200/csrc/strip.cuh) where its strips and
chunks can go wrong: widths around the 27 and 28 owned columns and the 32 lanes,
heights around a chunk, the smallest levels, linear and nonlinear sliding,
calving on.

J^T lambda and the fused adjoint sweeps against the oracle (binary64 1e-12 for
one product, 1e-10 for sweeps); J e against the oracle's residual by Richardson
-extrapolated central differences: with steps h and h/2 of the relative size
1e-4 their truncation is O(h^4) and their rounding eps / h = 1e-12 of the
residual's terms, which the thin columns amplify; 1e-6 as for the solver tests.
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
