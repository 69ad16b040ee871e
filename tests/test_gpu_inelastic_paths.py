"""The fused z pass of J2 and damage solves on lines without a compile-time
transform (k_zmid_gen of mat3d_b200/csrc/passes_zmid.cuh): radix variants 5, 13
and 31, a partly filled last tile, both transform types, both stop rules,
against the separate z passes; and the launches a sweep reports, which name the
path that ran.  Tolerances of the compile-time lengths' test: FP64 states within
a few hundred roundings (1e-11 allows 1e5), FP32 transforms within the rounding
of the increments they carry (1e-5)."""
import numpy as np
import pytest

import mat3d_b200 as m3d
from mat3d_b200 import rve as R

pytestmark = pytest.mark.gpu

J2 = np.array([[400e9, 0.2, 1e30, 0.0, 1.0, 0.0, 1e30], [70e9, 0.33, 100e6, 1e9, 1.0, 0.0, 1e30]])
DAMAGE = np.array([[20e9, 0.2, 1e30, 0.0, 1.0, 1e-4, 8e2], [3e9, 0.35, 1e30, 0.0, 1.0, 5e-4, 30.0]])
X0 = np.array([1.0, 0, 0, 0, 0, 0])


def rel(a, b):
    return np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(b)


def solve(shape, behav, prec, crit, fused, monkeypatch):
    monkeypatch.setenv("M3D_NO_SLAB", "0" if fused else "1")
    g, _ = R.penetrable_spheres(shape, radius=3.0, vf=0.2, seed=4)
    s = m3d.Solver(m3d.KIND_MECH, *shape, behav, prec)
    s.set_material_mech(J2 if behav == m3d.J2 else DAMAGE, g)
    s.set_load(np.array([2.4e-3, 0, 0, 0, 0, 0]), X0)
    s.run(1e-4, 1e-4, 3, crit)
    out = [s.field(w).copy() for w in (m3d.FIELD_STRAIN, m3d.FIELD_STRESS)]
    out.append(s.field(m3d.FIELD_EPS_P if behav == m3d.J2 else m3d.FIELD_DAMAGE).copy())
    out.append(s.increments())
    st = s.stats()
    s.close()
    return out, st


@pytest.mark.parametrize("prec,bound", [("fp64", 1e-11), ("fp32", 1e-5)])
@pytest.mark.parametrize("crit", [m3d.CRIT_REFERENCE, m3d.CRIT_RESIDUAL])
@pytest.mark.parametrize("behav", [m3d.J2, m3d.DAMAGE])
@pytest.mark.parametrize("shape", [(7, 9, 25), (5, 7, 26), (6, 5, 38), (16, 16, 16)])
def test_generic_lines_match_separate_passes(shape, behav, crit, prec, bound, monkeypatch):
    a, sa = solve(shape, behav, prec, crit, True, monkeypatch)
    b, sb = solve(shape, behav, prec, crit, False, monkeypatch)
    assert (sa["passes_per_sweep"], sb["passes_per_sweep"]) == (4, 5)
    assert sa["sweeps"] == sb["sweeps"]
    for x, y in zip(a, b):
        assert rel(x, y) < bound


@pytest.mark.parametrize("shape,passes", [((32, 32, 32), 4), ((12, 12, 64), 4), ((8, 10, 96), 4), ((5, 6, 256), 4),
                                          ((5, 7, 64), 5)])  # 35 lines: no whole tiles of four
def test_reported_passes(shape, passes, monkeypatch):
    _, st = solve(shape, m3d.J2, "fp64", m3d.CRIT_RESIDUAL, True, monkeypatch)
    assert st["passes_per_sweep"] == passes


def linear(kind, shape, prec, fused, monkeypatch):
    monkeypatch.setenv("M3D_NO_SLAB", "0" if fused else "1")
    g, _ = R.penetrable_spheres(shape, radius=3.0, vf=0.2, seed=9)
    s = m3d.Solver(kind, *shape, precision=prec)
    if kind == m3d.KIND_THERMAL:
        s.set_material_thermal(1.0, 20.0, g)
        s.set_load(np.array([0.3, -0.2, 1.0]))
    else:
        s.set_material_mech(np.array([[60e9, 0.2, 1e30, 0, 1, 0, 1e30], [3e9, 0.35, 1e30, 0, 1, 0, 1e30]]), g)
        s.set_load(np.array([1e6, 2e5, 0, 3e5, 0, -1e5]))
    s.run(1e-5 if prec == "fp32" else 1e-9)
    f, st = s.field(m3d.FIELD_STRAIN).copy(), s.stats()
    s.close()
    return f, st


# FP64 and FP32 fields: the same sums in another order; refined ones stop at a residual of 1e-9
@pytest.mark.parametrize("kind,shape,prec", [(m3d.KIND_THERMAL, (6, 8, 128), "fp64"), (m3d.KIND_THERMAL, (4, 8, 96), "fp64"),
                                             (m3d.KIND_MECH, (4, 8, 96), "fp64")] +
                         [(k, (16, 16, 16), p) for k in (m3d.KIND_THERMAL, m3d.KIND_MECH) for p in ("fp64", "fp32", "fp32_refine")])
def test_linear_fused_pass(kind, shape, prec, monkeypatch):
    a, sa = linear(kind, shape, prec, True, monkeypatch)
    b, sb = linear(kind, shape, prec, False, monkeypatch)
    assert (sa["passes_per_sweep"], sb["passes_per_sweep"]) == (4, 5)
    assert sa["sweeps_fp64"] == sb["sweeps_fp64"] and abs(sa["sweeps_fp32"] - sb["sweeps_fp32"]) <= 2
    assert rel(a, b) < {"fp64": 1e-10, "fp32": 1e-5, "fp32_refine": 1e-8}[prec]
