"""CPU tests of the index maps and launch plans that the kernels and the engine share
(fire_b200/csrc/fx_plan.h), compiled here by the host compiler alone."""
from __future__ import annotations

import ctypes as C
import subprocess
from pathlib import Path

import pytest

from fire_b200 import _abi as A

ROOT = Path(__file__).resolve().parent.parent

SHIM = r"""
#include "fx_plan.h"
extern "C" {
int zs_input_row(int q, int Y) { return fx_zs_input_row(q, Y); }
int zs_reflect(int q, int n) { return fx_zs_reflect(q, n); }
static std::vector<std::array<int, 3>> grids(int n, const int* d) {
    std::vector<std::array<int, 3>> v;
    for (int i = 0; i < n; ++i) v.push_back({d[3 * i], d[3 * i + 1], d[3 * i + 2]});
    return v;
}
int default_kernel(int n, const int* d, int half) {
    const auto v = grids(n, d);
    long long cells = 0;
    for (const auto& g : v) cells += (long long)g[0] * g[1] * g[2];
    int kernel, k, zc;
    fx_default_jacobi(cells, fx_zs_fill(v), half != 0, &kernel, &k, &zc);
    return kernel;
}
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


def flat(grids):
    return len(grids), (C.c_int * (3 * len(grids)))(*[v for g in grids for v in g])


@pytest.mark.parametrize("grids,half,kernel", [
    # narrow and flat: the strips' tiles would stay empty (unblocked measured faster)
    ([(4, 1024, 1024)], 0, A.JACOBI_UNBLOCKED), ([(4, 1024, 1024)], 1, A.JACOBI_UNBLOCKED),
    ([(8, 512, 1024)], 0, A.JACOBI_UNBLOCKED), ([(2048, 4, 512)], 0, A.JACOBI_UNBLOCKED),
    ([(36, 16, 36)] * 200, 0, A.JACOBI_UNBLOCKED), ([(36, 16, 36)] * 450, 0, A.JACOBI_UNBLOCKED),
    ([(4, 64, 64)] * 200, 0, A.JACOBI_UNBLOCKED), ([(4, 2048, 1024)], 0, A.JACOBI_UNBLOCKED),
    ([(36, 60, 36)] * 60, 1, A.JACOBI_UNBLOCKED), ([(36, 400, 300)], 1, A.JACOBI_UNBLOCKED),
    # and those on which the strips are the faster
    ([(16, 512, 512)], 0, A.JACOBI_FUSED), ([(36, 60, 36)] * 60, 0, A.JACOBI_FUSED),
    ([(36, 60, 36)] * 120, 1, A.JACOBI_FUSED), ([(512, 8, 1024)], 1, A.JACOBI_FUSED),
    ([(160, 240, 160)], 0, A.JACOBI_FUSED), ([(160, 240, 160)], 1, A.JACOBI_FUSED),
    ([(36, 44, 28)] * 128, 0, A.JACOBI_FUSED), ([(508, 508, 508)], 0, A.JACOBI_FUSED),
    ([(64, 96, 64), (160, 240, 160), (128, 192, 128)], 0, A.JACOBI_FUSED),
    # below 2 Mi cells
    ([(128, 128, 96)], 0, A.JACOBI_UNBLOCKED),
])
def test_default_kernel_by_fill_of_the_strip_tiles(plan, grids, half, kernel):
    assert plan.default_kernel(*flat(grids), half) == kernel
