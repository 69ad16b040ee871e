"""The benchmark's record names the passes of the sweep that ran and counts their
bytes (bench.py: sweep_of, pass_names, pass_bytes)."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402


@pytest.mark.parametrize("passes,kind,sweep,last", [(5, "thermal", "five", "z_inverse"), (4, "mech", "four", "z_fused"),
                                                    (2, "thermal", "slab", "yz_slab"), (2, "mech", "plane", "z_fused")])
def test_names(passes, kind, sweep, last):
    assert bench.sweep_of(passes, kind) == sweep
    names = bench.pass_names(sweep)
    assert len(names) == 5 and names[4] == last and sum(n is not None for n in names) == passes


def test_bytes():
    N, c, w = 64, 6, 8
    V, rows, plane = N ** 3, 6 * N * N * 34 * 16, 6 * N * N * 33 * 16  # half spectra of 34 (row layout) and 33 planes
    state = c * V * w
    assert bench.pass_bytes(c, w, N, False, "five") == (state + V + rows, 2 * rows, 2 * rows, 2 * rows, rows + 2 * state + V)
    assert bench.pass_bytes(c, w, N, False, "four") == (0, 2 * rows, 2 * rows, 2 * rows, 2 * rows + 2 * state + V)
    assert bench.pass_bytes(c, w, N, False, "plane") == (0, 0, 2 * plane, 0, 2 * plane + 2 * state + V)
    rows3, state3 = 3 * N * N * 34 * 8, 3 * V * 4
    assert bench.pass_bytes(3, 4, N, True, "slab") == (0, 0, 2 * rows3, 0, 2 * rows3 + 2 * state3 + 3 * V + 3 * V * 4)
