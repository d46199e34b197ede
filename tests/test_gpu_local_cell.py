"""The Vanka sweep's forms against the oracle's sweeps in binary64, at the edges of
their blocks and on the smallest levels: the linear-sliding local iteration
(glide_b200/csrc/local_cell.cuh: m = 1, damping + drag > 0, binary32) and the
general one, whose block shape depends on the size, the precision and m.

The inputs are binary32 numbers, so both sides solve the same cells.  Velocities of
5 m/a keep |H - dt r_H - gamma| above the binary32 rounding of its terms (1e-4 m)
in every cell used here, so no active-set decision may differ and no value is
excused.  Bars: binary64 1e-10, the multi-sweep parity bar.  Binary32, of the
largest value: one sweep ends within a few roundings of the local solution
(measured 3e-7 linear, 6e-7 general: 2e-6 and 4e-6); the second starts from that
and multiplies it by the local conditioning (2e-6, 1.2e-5: 1e-5 and 5e-5).
"""
from __future__ import annotations

import numpy as np
import pytest

from cases import random_state
from util import oracle_single_level

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

DX, DT = 1500.0, 5.0
SIZES = [(2, 2), (3, 2), (2, 40), (7, 15), (8, 16), (6, 14), (15, 31), (22, 9), (33, 61), (120, 150)]
LINEAR_BAR = {1: 2e-6, 2: 1e-5}
GENERAL_BAR = {1: 4e-6, 2: 5e-5}


def _state(ny, nx, thin=0.0):
    f = random_state(ny, nx, seed=100 * ny + nx, thin_frac=thin)
    f["u"], f["v"] = 0.1 * f["u"], 0.1 * f["v"]
    return {k: np.asarray(a, np.float32).astype(np.float64) for k, a in f.items()}


def _sweep(f, dtype, phys, sweeps):
    from glide_b200.hierarchy import Hierarchy
    h = Hierarchy(*f["H"].shape, DX, 1, dtype=dtype)
    for k in ("u", "v", "H", "H_prev", "mask", "bed", "B", "beta", "smb", "f_u", "f_v"):
        h.set(k, 0, torch.as_tensor(f[k]))
    h.set_phys(-1, **phys)
    h.set_rhs(0, DT)
    h.vanka_sweep(0, DT, sweeps)
    return {k: h.get(k, 0).cpu().numpy() for k in ("u", "v", "H", "mask")}


def _check(f, dtype, phys, sweeps, bar):
    got = _sweep(f, dtype, phys, sweeps)
    o = oracle_single_level({f"in_{k}": a for k, a in f.items()}, DX)
    o.set_phys(**phys)
    lev = o.levels[0]
    lev.f_H[...] = lev.H_prev / DT + lev.smb
    lev.vanka_sweep(DT, sweeps)
    for k in ("u", "v", "H"):
        want = getattr(lev, k)
        assert np.isfinite(got[k]).all(), k
        assert np.abs(got[k] - want).max() <= bar * np.abs(want).max(), (k, np.abs(got[k] - want).max())
    np.testing.assert_array_equal(got["mask"], lev.mask)


@pytest.mark.parametrize("sweeps,thin", [(1, 0.0), (1, 0.2), (2, 0.0)])
@pytest.mark.parametrize("ny,nx", SIZES)
def test_linear_sliding_in_binary32(ny, nx, sweeps, thin):
    _check(_state(ny, nx, thin), torch.float32, dict(calving_rate=2.0), sweeps, LINEAR_BAR[sweeps])


@pytest.mark.parametrize("phys", [dict(calving_rate=2.0), dict(m=1.0 / 3.0), dict(water_drag=-0.02)])
@pytest.mark.parametrize("ny,nx", SIZES)
def test_general_form_in_binary64(ny, nx, phys):
    # thin cells have nothing but the drag on their diagonals, and a negative one makes some nearly singular
    _check(_state(ny, nx, 0.0 if "water_drag" in phys else 0.2), torch.float64, phys, 2, 1e-10)


@pytest.mark.parametrize("phys", [dict(m=1.0 / 3.0), dict(water_drag=-0.02), dict(m=1.0 + 2.0 ** -22)])
@pytest.mark.parametrize("ny,nx", SIZES)
def test_general_form_in_binary32(ny, nx, phys):
    """Nonlinear sliding (as little as one step from m = 1: the linear form ignores the power law), or a drag that
    leaves the diagonals unbounded, is solved by the general form."""
    for sweeps in (1, 2):
        _check(_state(ny, nx), torch.float32, phys, sweeps, GENERAL_BAR[sweeps])


@pytest.mark.parametrize("m", [1.0, 1.0 / 3.0])
@pytest.mark.parametrize("size", [(434, 470), (441, 470)])
def test_wide_blocks_match_oracle(m, size):
    """On both sides of the size from which the general form takes its larger blocks in binary64 (2000 small ones),
    ragged in both directions."""
    _check(_state(*size), torch.float64, dict(m=m), 1, 1e-10)


@pytest.mark.parametrize("m", [1.0, 1.0 / 3.0])
def test_block_shape_changes_no_bit(m):
    """Three sweeps of the upper left cells of a large grid and of a grid cut there agree bit for bit where the cut is
    out of reach (three cells a sweep), on a rough state whose cells stop at every count of local iterations."""
    f = random_state(460, 470, seed=5)
    ny, nx = 200, 210
    cut = {k: a[:ny + (k in ("v", "f_v")), :nx + (k in ("u", "f_u"))].copy() for k, a in f.items()}
    a, b = (_sweep(s, torch.float64, dict(m=m), 3) for s in (f, cut))
    for k in ("u", "v", "H", "mask"):
        np.testing.assert_array_equal(a[k][:ny - 10, :nx - 10], b[k][:ny - 10, :nx - 10], err_msg=k)
