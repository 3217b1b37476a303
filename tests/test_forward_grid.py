"""The triangles of the forward warp's vertex grid (csrc/forward_grid.h, the code the kernels run), built for the
host: the vertices' pixels of frames from 2 x 2 up to more than 2^32 pixels, whose kernels read them from arrays
of that size."""
import ctypes
import subprocess

import pytest

from twixtor_b200 import buildlib

SOURCE = """
#include "forward_grid.h"
extern "C" int grid(long t, int w, int h, long* out) {
    tw::GridTriangle g;
    if (!tw::grid_triangle_at(t, w, h, g)) return 0;
    for (int k = 0; k < 3; k++) out[k] = g.first + g.at[k];
    return 1;
}
"""


@pytest.fixture(scope="module")
def grid(tmp_path_factory):
    d = tmp_path_factory.mktemp("grid")
    (d / "grid.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-I", buildlib.CSRC, "-o", str(d / "grid.so"), str(d / "grid.cpp")],
                   check=True)
    f = ctypes.CDLL(str(d / "grid.so")).grid
    f.argtypes = [ctypes.c_long, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
    return f


@pytest.mark.parametrize("w,h", [(2, 2), (2, 5), (7, 3), (46341, 46341), (46342, 46342), (65537, 65537), (2, 2 ** 31 - 1),
                                 (2 ** 30, 5)])
def test_vertices_of_a_triangle(grid, w, h):
    out = (ctypes.c_long * 3)()
    cells = (w - 1) * (h - 1)
    for cell in sorted({c for c in (0, 1, w - 2, w - 1, w, cells // 2, 2 ** 31 - 1, 2 ** 31, 2 ** 32, cells - 1) if c < cells}):
        r, c = divmod(cell, w - 1)
        first = r * w + c
        assert grid(2 * cell, w, h, out) and list(out) == [first, first + 1, first + w]
        assert grid(2 * cell + 1, w, h, out) and list(out) == [first + w + 1, first + 1, first + w]
        assert max(out) < w * h
    assert not grid(2 * cells, w, h, out)
