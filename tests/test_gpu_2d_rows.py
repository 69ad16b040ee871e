"""The 2-D solver's fused row kernels and column tiles (`k2d_mid`, `k2d_cols`)
against the numpy restatement: one and two iterations (the stress is stored by
the first kernel of a run of one, by a later one of a longer run), the shortest lines,
the primes the register DFTs end at, one and two columns a tile, more rows a CTA
than one with a last CTA part full, and rows too long for the fused kernel.
Tolerance: the fields are sums of terms of the size of the load, so rel-L2 is
that of two FP64 transforms an iteration, (iterations) 2 log2(Nx Ny) 2^-53
< 1e-14; 1e-12 leaves two digits for the Green operator's cancellation.
Reference: src/2d/FFT_analysis2D.cpp."""
import numpy as np
import pytest

import mat3d_b200 as m3d
from oracle import mat3d_oracle as O

pytestmark = pytest.mark.gpu

PROPS = np.array([68.9e9, 0.35, 400e9, 0.23])


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("iterations", [1, 2])
@pytest.mark.parametrize("Nx,Ny", [(2, 8), (8, 2), (29, 31), (26, 62), (6, 16), (1040, 6),
                                   (1100, 3), (1000, 10), (899, 12), (5, 1280), (3, 2002), (3, 2048)])
def test_2d_rows_and_columns(Nx, Ny, iterations):
    rng = np.random.default_rng(Nx * 10007 + Ny)
    rve = (rng.random(Nx * Ny) < 0.4).astype(np.int32)
    E = np.array([0.002, -0.001, 0.004 + 0.0005j])
    o = O.Mech2DOracle(Nx, Ny)
    o.material(PROPS, rve)
    o.setLoad(E)
    o.runAnalysis(iterations)
    assert np.isfinite(o.eps).all()
    s = m3d.Solver2D(Nx, Ny)
    s.material(PROPS, rve)
    s.set_load(E)
    s.run(iterations)
    eps, sig = s.fields()
    s.close()
    assert rel(eps, o.eps) < 1e-12 and rel(sig, o.sig) < 1e-12
