"""The library is built for sm_100a with line tables, and its device images are
not compressed: unpacking them costs a process up to 20 ms at the first use of each
source file's kernels."""
import os

from mat3d_b200 import build


def test_flags():
    flags = build.NVCC_FLAGS
    assert "arch=compute_100a,code=sm_100a" in flags and "-lineinfo" in flags
    assert "--compress-mode=none" in flags


def test_every_source_is_built():
    csrc = set(f for f in os.listdir(build.CSRC) if f.endswith((".cu", ".cpp")))
    assert csrc == set(os.path.basename(s) for s in build.SOURCES)
