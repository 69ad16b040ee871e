"""The generic line transforms' odd radices (7 ... 31) against the oracle, on
grids whose three lengths hold one of each and lengths that mix them.  Every
solve is FP64 to residual 1e-10 with the oracle's own sweep count, so fields
differ by rounding only: an R-point butterfly adds at most R terms of one ulp
to each of the ~40 sweeps' six transforms, 31 * 6 * 40 * 1.1e-16 < 1e-12 of
the field; 1e-11 allows a factor ten."""
import numpy as np
import pytest

import mat3d_b200 as m3d
from oracle import mat3d_oracle as O

pytestmark = pytest.mark.gpu

MAT = np.array([[40e9, 0.2, 1e30, 0, 1, 0, 1e30], [3e9, 0.35, 1e30, 0, 1, 0, 1e30]])


def rve(shape, seed):
    g = np.ones(shape, np.int32)
    g[np.random.default_rng(seed).random(shape) < 0.25] = 0
    return g.ravel()


def rel(a, b):
    return np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(b)


@pytest.mark.parametrize("shape", [(7, 11, 13), (14, 17, 19), (23, 9, 29), (31, 26, 21)])
def test_thermal_and_elastic(shape):
    g = rve(shape, 3)
    E = np.array([0.4, -0.3, 1.0])
    s = m3d.Solver(m3d.KIND_THERMAL, *shape)
    s.set_material_thermal(1.0, 20.0, g)
    s.set_load(E)
    s.run(1e-10, 0.0)
    o = O.ThermOracle(*shape)
    o.material(1.0, 20.0, g)
    o.set_load(E)
    o.run(1e-10, 0.0, criterion=O.CRIT_RESIDUAL)
    assert s.stats()["iters"] == o.iters
    assert rel(s.field(m3d.FIELD_STRAIN), o.grad.reshape(3, -1)) < 1e-11
    E = np.array([1e6, 0, 2e5, 0, 3e5, 0.0])
    s = m3d.Solver(m3d.KIND_MECH, *shape)
    s.set_material_mech(MAT, g)
    s.set_load(E)
    s.run(1e-10, 0.0)
    o = O.MechOracle(*shape)
    o.material(MAT, g)
    o.set_load(E)
    o.run(1e-10, 0.0, criterion=O.CRIT_RESIDUAL)
    assert s.stats()["iters"] == o.iters_per_inc[-1]
    assert rel(s.field(m3d.FIELD_STRESS), o.sig.reshape(6, -1)) < 1e-11


@pytest.mark.parametrize("N", [11, 26, 51, 57, 62])
def test_plane(N):
    g = rve((N, N), 5)
    E = np.array([0.002, -0.001, 0.004])
    o = O.Mech2DOracle(N, N)
    props = [3e9, 0.35, 70e9, 0.2]
    o.material(props, g)
    o.setLoad(E)
    o.runAnalysis(25)
    s = m3d.Solver2D(N, N)
    s.material(props, g)
    s.set_load(E)
    s.run(25)
    eps, sig = s.fields()
    assert rel(eps, o.eps) < 1e-11
    assert rel(sig, o.sig) < 1e-11
