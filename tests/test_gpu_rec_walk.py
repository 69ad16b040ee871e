"""The threshold walk of the reconstruction (`krec_thr_hist`, `krec_thr_walk`, and
the count per try where too many voxels lie on the cuts): fields with none, some,
as many as are listed and more voxels within rounding of the cuts 0.5 - 0.001 k,
beyond the first and last cut, infinite, and walks that run out of tries in either
direction.  Integer counts and exact double steps: equal bit for bit.
Reference: src/rec/reconstruction.cpp:370-395."""
import numpy as np
import pytest

import mat3d_b200 as m3d
from oracle import mat3d_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,hi", [(-0.1, 1.1), (0.31, 0.52), (0.72, 0.9), (0.1, 0.28)])
@pytest.mark.parametrize("shape,on_cuts", [((1, 1, 1), 1), ((3, 5, 7), 0), ((13, 13, 13), 40), ((13, 13, 13), 1024),
                                           ((13, 13, 13), 1025), ((13, 13, 13), 2197), ((64, 25, 9), 700)])
def test_walk(shape, on_cuts, lo, hi):
    n = int(np.prod(shape))
    rng = np.random.default_rng(n + on_cuts)
    T = (0.3 * n) ** 2 / n * np.ones(n)  # normC[0] / n = 0.3
    f = lo + (hi - lo) * rng.random(n)
    at = rng.permutation(n)[:on_cuts]
    # the cuts as the walk makes them, one step at a time, and their neighbours
    up = 0.5 - np.cumsum(np.r_[0.0, np.full(203, 0.001)])
    down = 0.5 - np.cumsum(np.r_[0.0, np.full(203, -0.001)])
    cuts = np.concatenate([up, down])
    cuts = cuts[(cuts >= lo) & (cuts <= hi)] if on_cuts < 2197 and ((cuts >= lo) & (cuts <= hi)).any() else cuts
    f[at] = np.nextafter(rng.choice(cuts, at.size), rng.choice((-9.0, 9.0), at.size))
    f[at[::2]] = rng.choice(cuts, at[::2].size)
    if n > 1:
        f[rng.integers(n, size=2)] = np.inf, -np.inf
    r = m3d.Reconstruction(T, *shape)
    r.set_state(f.astype(np.complex128), 0, 0, 1)
    r.threshold()
    got = r.get_state()["field"].real
    r.close()
    assert np.array_equal(got, O.RecOracle(T, *shape).threshold(f))
