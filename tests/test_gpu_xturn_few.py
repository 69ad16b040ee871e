"""The thermal x turnaround of few column groups (a warp per component,
`k_xturn_r1cp`) against the kernel that gives a warp all three
(`M3D_XTURN_CP=0`), on grids and batches on both sides of the rule's line (740
groups), in each precision.  Under the residual rule both do the same arithmetic:
equal bits and sweep counts, also of an entry alone and the same entry in a batch
of the other kernel.  Under the reference rule the switch picks other kernels,
which sum the check in another order: the fields agree to rounding, rel-L2 below
1e-5 in FP32 and 1e-12 in FP64.
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
    if criterion == m3d.CRIT_RESIDUAL:
        assert np.array_equal(out[0][1], out[1][1])
    assert rel(out[0][1], out[1][1]) < bound


@pytest.mark.parametrize("prec,tol", [("fp32", 1e-4), ("fp32_refine", 1e-9), ("fp64", 1e-6)])
@pytest.mark.parametrize("contrast", [12.0, 0.08])  # gradient- and flux-based
def test_entry_alone_and_in_a_batch(contrast, prec, tol):
    N, nrve = 32, 9  # 96 and 864 column groups
    rng = np.random.default_rng(5)
    rve = (rng.random((nrve, N ** 3)) < 0.3).astype(np.int32)
    E = np.array([0.01, 0.003, -0.002])
    fields = []
    for which in (range(nrve), [4]):
        s = m3d.Solver(m3d.KIND_THERMAL, N, N, N, m3d.ELASTIC, prec, nrve=len(which), nload=1)
        for i, r in enumerate(which):
            s.set_material_thermal(1.0, contrast, rve[r], rve=i)
            s.set_load(E, b=i)
        s.run(tol, tol, 1, m3d.CRIT_RESIDUAL)
        fields.append(s.field(m3d.FIELD_STRAIN, list(which).index(4)))
        s.close()
    assert np.array_equal(*fields)
