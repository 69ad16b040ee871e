"""The thermal x turnaround of few column groups (a warp per component,
`k_xturn_cp`) against the rank-one and register kernels (`M3D_XTURN_CP=0`), on
grids and batches on both sides of the rule's line (740 groups), in each precision
and both stop rules.  Per mode the two differ by the rounding of a dozen
operations, at most a few 1e-7 of the field in FP32 and 1e-15 in FP64 a sweep, and
a converging sweep damps what the one before left: rel-L2 below 1e-5 for FP32
sweeps (1e-9 with refinement, which solves to 1e-10) and 1e-12 for FP64.
Reference: src/3dTherm/FFT_thermal3D.cpp:200-266."""
import numpy as np
import pytest

import mat3d_b200 as m3d

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("criterion", [m3d.CRIT_RESIDUAL, m3d.CRIT_REFERENCE])
@pytest.mark.parametrize("prec,tol,bound", [("fp32", 1e-4, 1e-5), ("fp32_refine", 1e-10, 1e-9), ("fp64", 1e-6, 1e-12)])
@pytest.mark.parametrize("N,nrve", [(32, 1), (48, 1), (64, 1), (32, 2), (32, 3), (96, 1)])
def test_few_columns(N, nrve, prec, tol, bound, criterion, monkeypatch):
    if prec == "fp32_refine" and criterion == m3d.CRIT_REFERENCE:
        pytest.skip("refinement runs under the residual rule")
    rng = np.random.default_rng(N + nrve)
    rve = (rng.random((nrve, N ** 3)) < 0.3).astype(np.int32)
    out = []
    for cp in ("1", "0"):
        monkeypatch.setenv("M3D_XTURN_CP", cp)
        nload = 1 if nrve == 1 else 3
        s = m3d.Solver(m3d.KIND_THERMAL, N, N, N, m3d.ELASTIC, prec, nrve=nrve, nload=nload)
        for r in range(nrve):
            s.set_material_thermal(1.0, 12.0, rve[r], rve=r)
        if nload == 1:
            s.set_load(np.array([0.01, 0.003, -0.002]))
            s.run(tol, tol, 1, criterion)
            out.append((s.stats()["sweeps"], s.field(m3d.FIELD_STRAIN, 0)))
        else:
            C, *_ = s.homogenize(tol, tol, criterion)
            out.append((s.stats()["sweeps"], C))
        s.close()
    assert out[0][0] == out[1][0]
    assert rel(out[0][1], out[1][1]) < bound
