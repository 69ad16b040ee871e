"""Rounding of the fused J2 update: its FP64 strains and plastic strains are no
further from those of plain 64-bit torch (perf/cases.py) than the separate
passes' are, over ten RVEs.  (An update that adds the terms of C e in another
order was 15% and 20% further.)  The ratio of the two errors scatters by 4% from
RVE to RVE, so the mean of ten stays within 3% of 1 where the updates round
alike."""
import numpy as np
import pytest

from perf import cases

pytestmark = pytest.mark.gpu

CASE = {"kind": "j2", "n": 32, "precision": "fp64", "tol": 1e-4, "increments": 1, "strain": 3e-3}


def errors(seed, exact, fused, monkeypatch):
    monkeypatch.setenv("M3D_NO_SLAB", "0" if fused else "1")
    s = cases.prepare(CASE, seed)
    got = cases.run(s)
    s["solver"].close()
    return [float((got[k].double().cpu().ravel() - exact[k].double().cpu().ravel()).norm() / exact[k].double().norm().cpu())
            for k in ("strain", "plastic")]


def test_no_further_from_64_bits(monkeypatch):
    ratios = []
    for seed in range(1, 11):
        exact = cases.exact(CASE, seed)
        err = [errors(seed, exact, fused, monkeypatch) for fused in (True, False)]
        assert np.max(err) < 1e-12
        ratios.append(np.log(err[0]) - np.log(err[1]))
    strain, plastic = np.exp(np.mean(ratios, axis=0))
    print("strain %.3f plastic %.3f" % (strain, plastic))
    assert strain < 1.03 and plastic < 1.03
