"""Mixed-precision solves of a fixed number of cycles (both tolerances zero): the
iterates follow the reference's row order in the linear operators of both halves
(glide_b200/csrc/adjoint_tile.cuh, tangent_tile.cuh).

golden/mixed_fixed_cycles.npz holds the iterates of those kernels when they were
the only ones (two forward steps, then an adjoint solve, on every third node).
The same sums in the same order leave equality; 1e-12 is far below what another
order of the binary32 sums does to these iterates (1e-9 to 1e-5).

    python tests/test_gpu_fixed_cycles.py   (writes the fixture from the library in use)
"""
from __future__ import annotations

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

DT = 10.0
CASES = {"square": (96, True, 3, 2), "native": (80, False, 2, 3)}  # n, quirks, forward and adjoint cycles
STATE = ("u", "v", "H", "mask", "phi")
ADJOINT = ("lambda_u", "lambda_v", "lambda_H", "grad_beta", "grad_bed")


def _hier(name, n=None):
    from cases import dome
    from glide_b200.hierarchy import Hierarchy
    size, quirks, fwd, adj = CASES[name]
    n = n or size
    f = dome(n, 4000.0, R=0.4 * n * 4000.0, seed=n)
    h = Hierarchy(n, n, 4000.0, 3, precision="mixed", reference_quirks=quirks)
    for k in ("bed", "B", "beta", "smb", "H", "H_prev"):
        h.set(k, 0, torch.as_tensor(f[k]), restrict_down=True)
    h.set_fas(False, maximum_vcycles=fwd, relative_tolerance=0.0, absolute_tolerance=0.0)
    h.set_fas(True, maximum_vcycles=adj, relative_tolerance=0.0, absolute_tolerance=0.0)
    return h


def _forward(h):
    for _ in range(2):
        h.forward(DT, 0)
        h.set("H_prev", 0, h.get("H", 0))
    return {k: h.get(k, 0).cpu().numpy() for k in STATE}


def _adjoint(h, state):
    for k in STATE:
        h.set(k, 0, torch.as_tensor(state[k]))
    for k in "uvH":
        h.set("lambda_" + k, 0, 0.0)
    h.set("adj_f_u", 0, -0.05 * h.get("u", 0))
    h.set("adj_f_v", 0, -0.05 * h.get("v", 0))
    h.set("adj_f_H", 0, 0.0)
    h.backward(DT, 0)
    return {k: h.get(k, 0).cpu().numpy() for k in ADJOINT}


def _golden():
    from util import load_golden
    return load_golden("mixed_fixed_cycles")


def _close(a, want, what):
    assert np.abs(a[::3, ::3] - want).max() <= 1e-12 * np.abs(want).max(), what


@pytest.mark.parametrize("name", CASES)
def test_fixed_cycle_iterates_keep_their_order(name):
    g = _golden()
    h = _hier(name)
    state = _forward(h)
    for k in ("u", "v", "H"):
        _close(state[k], g[f"{name}_{k}"], k)
    lam = _adjoint(h, state)
    for k in ADJOINT:
        _close(lam[k], g[f"{name}_{k}"], k)


def test_fixed_cycle_iterates_do_not_depend_on_staging():
    """The tiles staged by TMA (24-row boxes in binary32, 22-row in binary64, edge tiles fixed up) or by clamped loads
    hold the same values, on levels whose tiles are ragged."""
    out = []
    for tma in (1, 0):
        h = _hier("native", n=88)
        h.set_tuning(tma_staging=tma)
        s = _forward(h)
        out.append({**s, **_adjoint(h, s)})
    for k in out[0]:
        np.testing.assert_array_equal(out[0][k], out[1][k], err_msg=k)


def test_operator_calls_do_not_depend_on_the_solve_before():
    """A fixed-cycle adjoint solve leaves the handle's own products as they were."""
    h = _hier("native")
    s = _forward(h)
    _adjoint(h, s)
    h.vjp(0, DT)
    a = {k: h.get("vjp_" + k, 0) for k in "uvH"}
    h.set_fas(True, relative_tolerance=1e-8)
    h.vjp(0, DT)
    for k in "uvH":
        assert torch.equal(a[k], h.get("vjp_" + k, 0)), k


if __name__ == "__main__":
    import sys
    from pathlib import Path
    here = Path(__file__).resolve().parent
    sys.path[:0] = [str(here), str(here.parent)]
    out = {}
    for name in CASES:
        h = _hier(name)
        s = _forward(h)
        for k, a in {**s, **_adjoint(h, s)}.items():
            out[f"{name}_{k}"] = a[::3, ::3]
    np.savez_compressed(sys.argv[1] if len(sys.argv) > 1 else here / "golden" / "mixed_fixed_cycles.npz", **out)
