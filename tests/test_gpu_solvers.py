"""GPU tests of the solver variants beyond the reference's own algorithm:
the Jacobian-vector product, the Newton outer iteration with the tangent
linear multigrid (binary64 and mixed binary64/binary32), the tuned FASCD
schedule -- all must reach the same discrete solution as the reference
method -- and the transpose consistency of J and J^T.

Tolerances: single operators against the reference 1e-12 (binary64);
finite differences 1e-6; converged solutions of different methods at a
relative residual of 1e-11: 1e-8 relative in u, v, H.
"""
from __future__ import annotations

import numpy as np
import pytest

from util import load_golden, rel_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

DT = 5.0


def _np(t):
    return t.detach().cpu().numpy()


def _hier(ny, nx, dx, levels=1, precision="fp64", quirks=True):
    from glide_b200.hierarchy import Hierarchy
    return Hierarchy(ny, nx, dx, levels, precision=precision, reference_quirks=quirks)


def _load_random(h, g):
    for k in ("u", "v", "H", "H_prev", "mask", "bed", "B", "beta", "smb", "f_u", "f_v"):
        h.set(k, 0, torch.as_tensor(g[f"in_{k}"]))


def test_jvp_matches_reference():
    g = load_golden("random_jvp_f64")
    ny, nx = g["in_H"].shape
    h = _hier(ny, nx, 1500.0)
    _load_random(h, g)
    for k in ("var_u", "var_v", "var_H"):
        h.set(k, 0, torch.as_tensor(g[f"in_{k}"]))
    h.compute_phi(0)
    h.jvp(0, DT, reference_rows=True)
    for k in ("jvp_u", "jvp_v", "jvp_H"):
        assert rel_err(_np(h.view(k, 0)), g[f"out_{k}"]) <= 1e-12, k


@pytest.mark.parametrize("tag,kw", [("", {}), ("_nomask", dict(use_mask=False)),
                                    ("_frozen", dict(freeze_calving=True))])
def test_compute_jvp_flags_match_reference(tag, kw):
    """ForwardOperators.compute_jvp's use_mask and freeze_calving, through
    the reference-facing Grid API, against the reference's own compute_jvp
    run with the same keywords (calving rate 2, so freezing it matters)."""
    from glide_b200.grid import Grid
    g = load_golden("random_jvp_flags_f64")
    ny, nx = g["in_H"].shape
    gr = Grid(ny, nx, 1500.0)
    for k in ("u", "v", "H", "H_prev", "mask"):
        getattr(gr.state, k).set(torch.as_tensor(g[f"in_{k}"]))
    gr.geometry.bed.set(torch.as_tensor(g["in_bed"]))
    gr.rheology.B.set(torch.as_tensor(g["in_B"]))
    gr.sliding.beta.set(torch.as_tensor(g["in_beta"]))
    gr.forcing.smb.set(torch.as_tensor(g["in_smb"]))
    gr.calving.calving_rate.set(float(g["in_calving_rate"]))
    ops = gr.forward_operators
    ops.f_u[:, :] = torch.as_tensor(g["in_f_u"])
    ops.f_v[:, :] = torch.as_tensor(g["in_f_v"])
    ops.set_rhs(DT)
    for k in ("var_u", "var_v", "var_H"):
        getattr(ops, k)[:, :] = torch.as_tensor(g[f"in_{k}"])
    assert ops.compute_jvp(DT, return_norms=True, **kw) is None
    for k in ("jvp_u", "jvp_v", "jvp_H"):
        assert rel_err(_np(getattr(ops, k)), g[f"out_{k}{tag}"]) <= 1e-12, (tag, k)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_jvp_tma_staging_equals_scalar_staging(precision):
    """The product is marched from global memory and does not depend on how
    other kernels stage their tiles (the tiled product of fixed-cycle mixed
    solves does: tests/test_gpu_fixed_cycles.py)."""
    from cases import random_state
    st = random_state(88, 70, seed=21)
    out = []
    for tma in (1, 0):
        h = _hier(88, 70, 900.0, precision=precision)
        h.set_tuning(tma_staging=tma)
        for k in ("u", "v", "H", "H_prev", "mask", "bed", "B", "beta", "smb"):
            h.set(k, 0, torch.as_tensor(st[k]))
        rng = np.random.default_rng(3)
        for k, shape in (("var_u", (88, 71)), ("var_v", (89, 70)), ("var_H", (88, 70))):
            h.set(k, 0, torch.as_tensor(rng.standard_normal(shape)))
        h.compute_phi(0)
        for rows in (True, False):
            h.jvp(0, DT, reference_rows=rows)
            out.append({k: _np(h.view(k, 0)).copy() for k in ("jvp_u", "jvp_v", "jvp_H")})
    for a, b in zip(out[:2], out[2:]):
        for k in a:
            assert np.array_equal(a[k], b[k]), k
            assert np.abs(a[k]).max() > 0


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_vjp_tma_staging_equals_scalar_staging(precision):
    """As above for the transposed product; its 24- and 22-row boxes are staged
    both ways in the fixed-cycle mixed solves."""
    from cases import random_state
    st = random_state(88, 70, seed=22)
    out = []
    for tma in (1, 0):
        h = _hier(88, 70, 900.0, precision=precision)
        h.set_tuning(tma_staging=tma)
        for k in ("u", "v", "H", "H_prev", "mask", "bed", "B", "beta", "smb"):
            h.set(k, 0, torch.as_tensor(st[k]))
        rng = np.random.default_rng(4)
        for k, shape in (("lambda_u", (88, 71)), ("lambda_v", (89, 70)), ("lambda_H", (88, 70))):
            h.set(k, 0, torch.as_tensor(rng.standard_normal(shape)))
        h.compute_phi(0)
        h.vjp(0, DT)
        out.append({k: _np(h.view(k, 0)).copy() for k in ("vjp_u", "vjp_v", "vjp_H")})
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k
        assert np.abs(out[0][k]).max() > 0


def test_tangent_jvp_matches_finite_differences():
    from cases import random_state
    st = random_state(24, 40, seed=3, thin_frac=0.0)
    st["mask"][:] = 0.0
    h = _hier(24, 40, 1500.0)
    for k in ("u", "v", "H", "H_prev", "mask", "bed", "B", "beta", "smb"):
        h.set(k, 0, torch.as_tensor(st[k]))
    h.compute_phi(0)
    rng = np.random.default_rng(9)
    e = dict(var_u=rng.normal(0, 1, st["u"].shape), var_v=rng.normal(0, 1, st["v"].shape),
             var_H=rng.normal(0, 10, st["H"].shape))
    for k, v in e.items():
        h.set(k, 0, torch.as_tensor(v))
    h.jvp(0, DT, reference_rows=False)
    jv = {k: _np(h.view(f"jvp_{k}", 0)).copy() for k in ("u", "v", "H")}
    eps = 1e-5
    res = {}
    for sgn in (1, -1):
        for k in ("u", "v", "H"):
            h.set(k, 0, torch.as_tensor(st[k] + sgn * eps * e[f"var_{k}"]))
        h.residual(0, DT, 8)  # FREEZE_PHI, no mask, forcing on
        res[sgn] = {k: _np(h.view(f"r_{k}", 0)).copy() for k in ("u", "v", "H")}
    for k in ("u", "v", "H"):
        fd = (res[1][k] - res[-1][k]) / (2 * eps)
        assert rel_err(jv[k], fd) <= 1e-6, k


def test_reference_dot_product_identity():
    """<J e, lam> vs <e, J^T lam> with the reference's conventions (e and lam
    zero on Dirichlet faces and masked cells), the check of tests/adjoint_test.py."""
    from cases import random_state
    st = random_state(32, 32, seed=21)
    h = _hier(32, 32, 1000.0)
    for k in ("u", "v", "H", "H_prev", "mask", "bed", "B", "beta", "smb"):
        h.set(k, 0, torch.as_tensor(st[k]))
    h.compute_phi(0)
    rng = np.random.default_rng(4)
    m = st["mask"] > 0.5

    def field(shape, kind):
        a = rng.normal(0, 1, shape)
        if kind == "u":
            a[:, 0] = a[:, -1] = 0
        elif kind == "v":
            a[0] = a[-1] = 0
        else:
            a[m] = 0
        return a

    e = {k: field(st[k].shape, k) for k in ("u", "v", "H")}
    lam = {k: field(st[k].shape, k) for k in ("u", "v", "H")}
    for k in ("u", "v", "H"):
        h.set(f"var_{k}", 0, torch.as_tensor(e[k]))
        h.set(f"lambda_{k}", 0, torch.as_tensor(lam[k]))
    h.jvp(0, DT, reference_rows=True)
    h.vjp(0, DT)
    t1 = sum(float((_np(h.view(f"vjp_{k}", 0)) * e[k]).sum()) for k in ("u", "v", "H"))
    t2 = sum(float((_np(h.view(f"jvp_{k}", 0)) * lam[k]).sum()) for k in ("u", "v", "H"))
    # the reference applies the viscous block's forward derivative in its
    # transpose (symmetric only up to the discrete eta coupling): measured,
    # not exact; the mismatch stays a small fraction of the product
    assert abs(t1 - t2) <= 2e-2 * 0.5 * (abs(t1) + abs(t2)), (t1, t2)


def _solve_c1(precision="fp64", quirks=True, method=None, schedule=None, relax=None, omega=None, rtol=1e-11,
              newton_steps=None, switch=None):
    from cases import slab_c1
    f = slab_c1()
    h = _hier(64, 64, 1000.0, levels=4, precision=precision, quirks=quirks)
    for k in ("bed", "B", "beta", "smb", "H", "H_prev"):
        h.set(k, 0, torch.as_tensor(f[k]), restrict_down=True)
    h.set_fas(False, maximum_vcycles=200, relative_tolerance=rtol, absolute_tolerance=0.0)
    if schedule:
        h.set_fas(False, pre_steps=schedule[0], post_steps=schedule[1], finest_steps=schedule[2],
                  coarsest_steps=schedule[3])
    kw = {}
    if relax is not None:
        kw["relaxation"] = relax
    if newton_steps is not None:
        kw["newton_steps"] = newton_steps
    if omega is not None:
        kw["omega"] = omega
    if kw:
        h.set_vanka(False, -1, **kw)
    if method:
        h.set_tuning(forward_method=method)
    if switch is not None:
        h.set_tuning(newton_switch_exp10=switch)
    st = h.forward(10.0, 0)
    return h, st


@pytest.fixture(scope="module")
def c1_reference_solution():
    h, st = _solve_c1()
    assert st["final_norm"] <= 1e-11 * st["initial_norm"], st
    return {k: _np(h.view(k, 0)).copy() for k in ("u", "v", "H")}


def test_tuned_schedule_reaches_reference_solution(c1_reference_solution):
    h, st = _solve_c1(quirks=False, relax=1.0)
    assert st["final_norm"] <= 1e-11 * st["initial_norm"]
    for k, ref in c1_reference_solution.items():
        assert rel_err(_np(h.view(k, 0)), ref) <= 1e-8, k


def test_newton_binary64_reaches_reference_solution(c1_reference_solution):
    h, st = _solve_c1(quirks=False, schedule=(4, 4, 0, 200), method="newton")
    assert st["final_norm"] <= 1e-11 * st["initial_norm"]
    for k, ref in c1_reference_solution.items():
        assert rel_err(_np(h.view(k, 0)), ref) <= 1e-8, k


def test_mixed_precision_reaches_reference_solution(c1_reference_solution):
    h, st = _solve_c1(precision="mixed", quirks=False, schedule=(4, 4, 0, 200))
    assert st["final_norm"] <= 1e-11 * st["initial_norm"]
    for k, ref in c1_reference_solution.items():
        assert rel_err(_np(h.view(k, 0)), ref) <= 1e-8, k


@pytest.mark.parametrize("switch", [0, 2])
def test_fast_form_reaches_reference_solution(c1_reference_solution, switch):
    """The benchmark's fast form: mixed precision, corrected transfers,
    guarded Newton from the start (switch 0) or after FASCD (4/4/0/50, local
    Newton capped at 3) has reached 1e-2 (switch 2).  Its binary32 tangent
    smoother keeps the block factors in bfloat16 pairs; the solution still
    meets the binary64 reference form at 1e-8."""
    h, st = _solve_c1(precision="mixed", quirks=False, schedule=(4, 4, 0, 50), method="newton",
                      newton_steps=3, switch=switch)
    assert st["final_norm"] <= 1e-11 * st["initial_norm"]
    for k, ref in c1_reference_solution.items():
        assert rel_err(_np(h.view(k, 0)), ref) <= 1e-8, k


def test_rejected_newton_step_is_undone():
    """Newton from a cold start on a steep dome makes the residual grow at
    first; the guard undoes those steps and the solve still converges."""
    from cases import dome
    from glide_b200.hierarchy import Hierarchy
    f = dome(128, 1500.0, 86e3, seed=3)
    h = Hierarchy(128, 128, 1500.0, 4, precision="mixed", reference_quirks=False)
    for k in ("bed", "B", "beta", "smb", "H", "H_prev"):
        h.set(k, 0, torch.as_tensor(f[k]), restrict_down=True)
    h.set_fas(False, maximum_vcycles=80, relative_tolerance=1e-9, absolute_tolerance=0.0,
              pre_steps=4, post_steps=4, finest_steps=0, coarsest_steps=50)
    h.set_vanka(False, -1, newton_steps=3)
    h.set_tuning(forward_method="newton", newton_switch_exp10=0)
    st = h.forward(5.0, 0)
    assert np.isfinite(st["final_norm"]) and st["final_norm"] <= 1e-9 * st["initial_norm"], st


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_adjoint_converges_to_reference_adjoint(precision):
    """Converged adjoint of C1 (binary64 reference form) against the fast
    forms: lambda to 1e-8 relative, gradients to 1e-7.  The mixed adjoint
    smoother keeps binary32 block factors: in reference mode the converged
    adjoint depends on the cycle's path (the reference's v-face prolongation
    writes into the pinned v faces), and with bfloat16 factors it moved
    2.4e-6 from binary64."""
    def run(prec, quirks):
        h, st = _solve_c1(precision=prec, quirks=quirks)
        u, v = h.get("u", 0), h.get("v", 0)
        h.set("adj_f_u", 0, -(u - 1.1 * u))
        h.set("adj_f_v", 0, -(v - 0.9 * v))
        h.set("adj_f_H", 0, 0.0)
        h.set_fas(True, maximum_vcycles=100, relative_tolerance=1e-11, absolute_tolerance=0.0)
        ast = h.backward(10.0, 0)
        assert ast["final_norm"] <= 1e-11 * ast["initial_norm"], ast
        return {k: _np(h.view(k, 0)).copy() for k in ("lambda_u", "lambda_v", "lambda_H", "grad_beta", "grad_bed")}
    ref = run("fp64", True)
    got = run(precision, True)
    for k in ("lambda_u", "lambda_v", "lambda_H"):
        assert rel_err(got[k], ref[k]) <= 1e-8, k
    for k in ("grad_beta", "grad_bed"):
        assert rel_err(got[k], ref[k]) <= 1e-7, k


def test_vanka_dump_matches_reference():
    """ForwardOperators.vanka_dump: the local 5x5 Vanka systems of every cell."""
    g = load_golden("random_vanka_dump_f64")
    ny, nx = g["in_H"].shape
    h = _hier(ny, nx, 1500.0)
    for k in ("u", "v", "H", "H_prev", "bed", "B", "beta", "smb", "phi", "gamma", "f_u", "f_v"):
        h.set(k, 0, torch.as_tensor(g[f"in_{k}"]))
    h.set_phys(0, calving_rate=1.0)
    h.set_rhs(0, DT)
    J, r = h.vanka_dump(0, DT)
    assert rel_err(_np(J), g["out_J"]) <= 1e-12
    assert rel_err(_np(r), g["out_r"]) <= 1e-12


def test_binary32_operators_against_binary64():
    """The binary32 fast-math operators the mixed form runs against their
    binary64 versions on the same state, at the operator level: the JVP and
    VJP at a solved dome state, and the residual operator F(x) at that state
    with u and v perturbed (at the solution F(x) balances the forcing, the
    small difference of large terms, below binary32 resolution).  Relative
    max-norm differences at the binary32 rounding level, stated here as
    5e-5."""
    from cases import dome
    n, dx = 256, 6000.0
    f = dome(n, dx, 1200e3, seed=1)
    h64 = _hier(n, n, dx, levels=4, quirks=False)
    for k in ("bed", "B", "beta", "smb", "H", "H_prev"):
        h64.set(k, 0, torch.as_tensor(f[k]), restrict_down=True)
    h64.set_fas(False, maximum_vcycles=4, relative_tolerance=0.0, absolute_tolerance=0.0)
    h64.forward(DT, 0)
    h32 = _hier(n, n, dx, precision="fp32", quirks=False)
    rng = np.random.default_rng(8)
    fields = ("u", "v", "H", "H_prev", "mask", "bed", "B", "beta", "smb")
    extra = {"var_u": 50.0 * rng.standard_normal((n, n + 1)), "var_v": 50.0 * rng.standard_normal((n + 1, n)),
             "var_H": 10.0 * rng.standard_normal((n, n)), "lambda_u": rng.standard_normal((n, n + 1)),
             "lambda_v": rng.standard_normal((n + 1, n)), "lambda_H": rng.standard_normal((n, n))}
    for k, v in extra.items():
        h64.set(k, 0, torch.as_tensor(v))
    for k in fields + tuple(extra):
        h32.set(k, 0, h64.get(k, 0).to(torch.float32))
    errs = {}
    for h in (h64, h32):
        h.set_rhs(0, DT)
        h.compute_phi(0)
        h.jvp(0, DT, reference_rows=False)
        h.vjp(0, DT)
    pu = h64.get("u", 0) + 20.0 * torch.as_tensor(rng.standard_normal((n, n + 1)), device="cuda")
    pv = h64.get("v", 0) + 20.0 * torch.as_tensor(rng.standard_normal((n + 1, n)), device="cuda")
    for h in (h64, h32):
        h.set("u", 0, pu.to(h.dtype))
        h.set("v", 0, pv.to(h.dtype))
        h.residual(0, DT, 1 | 2 | 8)  # USE_MASK | OPERATOR_ONLY | FREEZE_PHI: F(x) into F_*
    for k in ("F_u", "F_v", "F_H", "jvp_u", "jvp_v", "jvp_H", "vjp_u", "vjp_v", "vjp_H"):
        errs[k] = rel_err(_np(h32.view(k, 0)).astype(np.float64), _np(h64.view(k, 0)))
    print("binary32 vs binary64 operators:", {k: f"{e:.1e}" for k, e in errs.items()})
    for k, e in errs.items():
        assert e <= 5e-5, (k, e)
