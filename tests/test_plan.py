"""CPU tests of the index maps and launch plans that the kernels and the engine share
(fire_b200/csrc/fx_plan.h), compiled here by the host compiler alone."""
from __future__ import annotations

import ctypes as C
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

SHIM = r"""
#include "fx_plan.h"
extern "C" {
int zs_input_row(int q, int Y) { return fx_zs_input_row(q, Y); }
int zs_reflect(int q, int n) { return fx_zs_reflect(q, n); }
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "shim.cpp").write_text(SHIM)
    so = d / "plan.so"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-Wall", "-Werror", "-I",
                    str(ROOT / "fire_b200" / "csrc"), "-o", str(so), str(d / "shim.cpp")], check=True)
    return C.CDLL(str(so))


def test_strip_tiles_copy_rows_and_planes_of_the_grid(plan):
    """Every input row of every tile of 14 rows (two above and two below it) and every plane that a
    chunk requests lies in the grid, from the flattest grid on; the ones beside it are their
    reflections at the floor and, above, the top row."""
    for Y in [*range(4, 64, 4), 508, 2048]:
        for y0 in range(0, Y, 14):
            for q in range(y0 - 2, y0 + 16):
                r = plan.zs_input_row(q, Y)
                assert 0 <= r < Y, (Y, y0, q, r)
                assert r == (q if 0 <= q < Y else -1 - q if q < 0 else Y - 1), (Y, q, r)
    for Z in (4, 8, 12, 508):
        for q in range(-2, Z + 2):
            assert 0 <= plan.zs_reflect(q, Z) < Z, (Z, q)
