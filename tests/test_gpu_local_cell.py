"""The Vanka sweep's linear-sliding form (glide_b200/csrc/local_cell.cuh) and
its general form against the oracle's sweeps, at the edges of the blocks' 7 x 15
owned cells and on the smallest levels.

binary64: 1e-10, the multi-sweep parity bar.  binary32: 2e-4, the bar of the
binary32 solves, for all but a few values: a cell whose H - dt r_H lies within
binary32 rounding of gamma may take the other active-set decision.  With
|H - dt r_H| up to 1e5 spread over about 1e3 that is 6e-6 of the decisions, 60
of them per cell in two sweeps -- about one cell at the largest size here --
and one such cell reaches the 5 x 5 around it in the two sweeps: two cells' worth,
50 values, may differ.
"""
from __future__ import annotations

import numpy as np
import pytest

from cases import random_state
from util import oracle_single_level, rel_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

DX, DT = 1500.0, 5.0
SIZES = [(2, 2), (7, 15), (8, 16), (6, 14), (15, 31), (22, 9), (33, 61)]


def _run(ny, nx, dtype, phys=None, sweeps=2):
    from glide_b200.hierarchy import Hierarchy
    f = random_state(ny, nx, seed=100 * ny + nx)
    h = Hierarchy(ny, nx, DX, 1, dtype=torch.float64 if dtype == np.float64 else torch.float32)
    for k in ("u", "v", "H", "H_prev", "mask", "bed", "B", "beta", "smb", "f_u", "f_v"):
        h.set(k, 0, torch.as_tensor(f[k]))
    o = oracle_single_level({f"in_{k}": a for k, a in f.items()}, DX, dtype=dtype)
    lev = o.levels[0]
    if phys:
        h.set_phys(-1, **phys)
        o.set_phys(**phys)
    h.set_rhs(0, DT)
    lev.f_H[...] = lev.H_prev / dtype(DT) + lev.smb
    h.vanka_sweep(0, DT, sweeps)
    lev.vanka_sweep(DT, sweeps)
    return {k: (h.view(k, 0).cpu().numpy(), getattr(lev, k)) for k in ("u", "v", "H", "mask")}


@pytest.mark.parametrize("dtype,tol", [(np.float64, 1e-10), (np.float32, 2e-4)])
@pytest.mark.parametrize("ny,nx", SIZES)
def test_linear_sliding_sweeps_match_oracle(ny, nx, dtype, tol):
    got = _run(ny, nx, dtype, phys=dict(calving_rate=2.0))
    for k in ("u", "v", "H"):
        a, b = got[k]
        off = np.abs(a - b) > tol * np.abs(b).max()
        assert off.sum() <= (0 if dtype == np.float64 else 50), k
    if dtype == np.float64:
        assert (got["mask"][0] == got["mask"][1]).mean() >= 0.998


@pytest.mark.parametrize("phys", [dict(m=1.0 / 3.0), dict(water_drag=-0.02)])
def test_general_form_matches_oracle(phys):
    """Nonlinear sliding, or a drag that leaves the diagonals unbounded below, runs the general form."""
    for ny, nx in ((8, 16), (31, 16)):
        got = _run(ny, nx, np.float64, phys=phys)
        for k in ("u", "v", "H"):
            assert rel_err(*got[k]) <= 1e-10, (k, ny, nx)
