"""The fused z pass of the inelastic sweeps (mat3d_b200/csrc/passes_zmid.cuh)
against the separate z passes, which the oracle pins: J2 and damage, both stop
rules, both transform types, grids whose lines do and do not fill its tiles.
The same sweeps in another summation order: the same sweep counts, FP64 states
within a few hundred roundings (1e-11 allows 1e5), FP32 transforms within the
rounding of the increments they carry (1e-5)."""
import numpy as np
import pytest

import mat3d_b200 as m3d
from mat3d_b200 import rve as R

pytestmark = pytest.mark.gpu

J2 = np.array([[400e9, 0.2, 1e30, 0.0, 1.0, 0.0, 1e30], [70e9, 0.33, 100e6, 1e9, 1.0, 0.0, 1e30]])
POWER = np.array([[400e9, 0.2, 1e30, 0.0, 1.0, 0.0, 1e30], [70e9, 0.33, 100e6, 1e8, 0.5, 0.0, 1e30]])
DAMAGE = np.array([[20e9, 0.2, 1e30, 0.0, 1.0, 1e-4, 8e2], [3e9, 0.35, 1e30, 0.0, 1.0, 5e-4, 30.0]])
X0 = np.array([1.0, 0, 0, 0, 0, 0])


def rel(a, b):
    return np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(b)


def solve(shape, behav, mat, prec, crit, fused, monkeypatch, batch=1):
    monkeypatch.setenv("M3D_NO_SLAB", "0" if fused else "1")
    g, _ = R.penetrable_spheres(shape, radius=3.0, vf=0.2, seed=4)
    s = m3d.Solver(m3d.KIND_MECH, *shape, behav, prec, batch)
    s.set_material_mech(mat, g)
    for b in range(batch):
        s.set_load(np.array([2.4e-3 / (b + 1), 0, 0, 0, 0, 0]), X0, b)
    s.run(1e-4, 1e-4, 3, crit)
    out = [s.field(w, b).copy() for b in range(batch) for w in (m3d.FIELD_STRAIN, m3d.FIELD_STRESS)]
    out.append(s.field(m3d.FIELD_EPS_P if behav == m3d.J2 else m3d.FIELD_DAMAGE).copy())
    out.append(s.increments())
    st = s.stats()
    s.close()
    return out, st["sweeps"]


@pytest.mark.parametrize("prec,bound", [("fp64", 1e-11), ("fp32", 1e-5)])
@pytest.mark.parametrize("crit", [m3d.CRIT_REFERENCE, m3d.CRIT_RESIDUAL])
@pytest.mark.parametrize("shape,behav,mat", [((32, 32, 32), m3d.J2, J2), ((16, 15, 48), m3d.J2, J2), ((12, 12, 64), m3d.DAMAGE, DAMAGE),
                                             ((8, 10, 96), m3d.J2, POWER), ((6, 7, 128), m3d.DAMAGE, DAMAGE),
                                             ((5, 6, 256), m3d.J2, J2), ((5, 7, 64), m3d.J2, J2)])
def test_matches_separate_passes(shape, behav, mat, crit, prec, bound, monkeypatch):
    a, na = solve(shape, behav, mat, prec, crit, True, monkeypatch)
    b, nb = solve(shape, behav, mat, prec, crit, False, monkeypatch)
    assert na == nb
    for x, y in zip(a, b):
        assert rel(x, y) < bound


def test_batch_entries(monkeypatch):
    """Entries that stop at different sweeps keep their own converged stress."""
    a, _ = solve((16, 16, 32), m3d.J2, J2, "fp64", m3d.CRIT_RESIDUAL, True, monkeypatch, batch=2)
    b, _ = solve((16, 16, 32), m3d.J2, J2, "fp64", m3d.CRIT_RESIDUAL, False, monkeypatch, batch=2)
    for x, y in zip(a, b):
        assert rel(x, y) < 1e-11
