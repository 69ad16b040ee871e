"""Two-pass elastic sweeps (the kz-plane pass and the z-mid pass,
mat3d_b200/csrc/passes_plane.cuh) against the five-pass sweeps, which the
oracle pins, at every length that has the kernels.

Tolerances, for the same stop rule and sweep count: both sweeps evaluate the
same sums in another order, so FP64 fields agree to a few hundred roundings
(1e-10 allows a million), FP32 fields to 1e-5 (the rounding of ~30 sweeps of
six 1-D transforms of up to 96 points, 30 * 6 * 7 * 6e-8 = 8e-5 worst case, a
tenth of it in practice for independent roundings), refined fields to the
residual they are refined to."""
import numpy as np
import pytest

import mat3d_b200 as m3d
from mat3d_b200 import rve as R
from oracle import mat3d_oracle as O

pytestmark = pytest.mark.gpu

STIFF = np.array([[60e9, 0.2, 1e30, 0, 1, 0, 1e30], [3e9, 0.35, 1e30, 0, 1, 0, 1e30]])   # stress-based
SOFT = np.array([[0.15e9, 0.3, 1e30, 0, 1, 0, 1e30], [3e9, 0.35, 1e30, 0, 1, 0, 1e30]])  # strain-based
THREE = np.vstack([STIFF, [[20e9, 0.25, 1e30, 0, 1, 0, 1e30]]])


def rel(a, b):
    return np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(b)


def phases(N, seed, three=False):
    g, _ = R.penetrable_spheres(N, radius=max(2.0, N / 10.0), vf=0.2, seed=seed)
    if three:
        h, _ = R.penetrable_spheres(N, radius=max(2.0, N / 12.0), vf=0.1, seed=seed + 50)
        g = np.where(h == 0, 2, g).astype(np.int32)
    return g


def solve(N, mat, ph, E, prec, tol, monkeypatch, two_pass, nrve=None, graph=True):
    monkeypatch.setenv("M3D_NO_SLAB", "0" if two_pass else "1")
    monkeypatch.setenv("M3D_NO_GRAPH", "0" if graph else "1")
    s = m3d.Solver(m3d.KIND_MECH, N, N, N, precision=prec)
    s.set_material_mech(mat, ph)
    s.set_load(E)
    s.run(tol)
    st = s.stats()
    assert st["passes_per_sweep"] == (2 if two_pass else 5)
    f = s.field(m3d.FIELD_STRAIN).copy()
    s.close()
    return f, st


LOAD = {"stiff": np.array([1e6, -2e5, 3e5, 1e5, 2e5, -1e5]), "soft": np.array([1e-3, -2e-4, 0, 1e-4, 2e-4, 3e-4])}


@pytest.mark.parametrize("name,mat", [("stiff", STIFF), ("soft", SOFT)])
@pytest.mark.parametrize("prec,tol,bound", [("fp64", 1e-9, 1e-10), ("fp32", 1e-5, 1e-5), ("fp32_refine", 1e-9, 1e-8)])
@pytest.mark.parametrize("N", [32, 48, 64, 96])
def test_matches_five_passes(N, prec, tol, bound, name, mat, monkeypatch):
    if prec == "fp64" and N == 96:
        pytest.skip("no FP64 plane kernel at 96")
    ph = phases(N, 7)
    a, sa = solve(N, mat, ph, LOAD[name], prec, tol, monkeypatch, True)
    b, sb = solve(N, mat, ph, LOAD[name], prec, tol, monkeypatch, False)
    assert sa["sweeps_fp64"] == sb["sweeps_fp64"] and abs(sa["sweeps_fp32"] - sb["sweeps_fp32"]) <= 2
    assert rel(a, b) < bound


def test_oracle_three_phases(monkeypatch):
    N = 32
    ph = phases(N, 11, three=True)
    a, st = solve(N, THREE, ph, LOAD["stiff"], "fp64", 1e-9, monkeypatch, True)
    o = O.MechOracle(N, N, N)
    o.material(THREE, ph)
    o.set_load(LOAD["stiff"])
    o.run(1e-9, 0.0, criterion=O.CRIT_RESIDUAL)
    assert st["iters"] == o.iters_per_inc[-1]
    assert rel(a, o.eps.reshape(6, -1)) < 1e-10


@pytest.mark.parametrize("N", [32, 96])
def test_many_rves_equal_single_solves(N, monkeypatch):
    """Entries that converge at different sweeps, each RVE with its own scheme:
    bitwise the tensors of the RVEs alone; graph and host loops bitwise too."""
    monkeypatch.setenv("M3D_NO_SLAB", "0")
    mats, maps = [STIFF, SOFT, STIFF * np.array([[0.2], [1.0]]) + np.array([[0, 0.16, 0, 0, 0.8, 0, 0], [0] * 7])], []
    m = m3d.Solver(m3d.KIND_MECH, N, N, N, precision="fp32_refine", nrve=3)
    for r, mat in enumerate(mats):
        maps.append(phases(N, 20 + r))
        m.set_material_mech(mat, maps[r], rve=r)
    C = m.homogenize(1e-8)[0]
    monkeypatch.setenv("M3D_NO_GRAPH", "1")
    for r, mat in enumerate(mats):
        s = m3d.Solver(m3d.KIND_MECH, N, N, N, precision="fp32_refine", batch=6)
        s.set_material_mech(mat, maps[r])
        assert np.array_equal(s.homogenize(1e-8)[0], C[r])
