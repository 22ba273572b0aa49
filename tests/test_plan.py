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
#include <cstdint>
#include <cstring>
static float of(uint32_t b) { float x; std::memcpy(&x, &b, 4); return x; }
// floats x of the binade 2^e for which RN(x rh + RN(x rl)) is not RN(x / d)
static int wrong(float d, float rh, float rl, int e) {
    int n = 0;
    for (uint32_t m = 0; m < 1u << 23; ++m) {
        const float x = std::ldexp(of(0x3f800000u | m), e);
        n += std::fmaf(x, rh, x * rl) != x / d;
    }
    return n;
}
extern "C" {
// the candidate that one binade accepts (-1: none), and what it gets wrong in the binade 2^e (e >= 1000:
// in the lowest binade it is used in)
int two_op_choice(float d) {
    const FxTwoOp t = fx_two_op_candidates(d);
    for (int k = 0; k < 5; ++k)
        if (wrong(d, t.rh, t.rl[k], 0) == 0) return k;
    return -1;
}
int two_op_wrong(float d, int k, int e) {
    const FxTwoOp t = fx_two_op_candidates(d);
    return wrong(d, t.rh, t.rl[k], e >= 1000 ? std::ilogb(t.lo) + e - 1000 : e);
}
float two_op_lo(float d) { return fx_two_op_candidates(d).lo; }
float denominator(const int* dims, const float* extent) {  // of the Jacobi (the engine's refresh_params)
    float w[3];
    for (int i = 0; i < 3; ++i) {
        const float m = (float)dims[i] / extent[i];
        w[i] = m * m;
    }
    return 2.0f * (w[0] + w[1] + w[2]);
}
int fixed_wrong(int slot, int e) {
    const FxDivTwo c = fx_div_two_of(slot);
    return wrong(c.d, c.rh, c.rl, e);
}
int fixed_specials(int slot) {  // zeros, infinities and NaN
    const FxDivTwo c = fx_div_two_of(slot);
    int n = 0;
    for (float x : {0.0f, -0.0f, INFINITY, -INFINITY}) {
        const float r = std::fmaf(x, c.rh, x * c.rl), q = x / c.d;
        n += std::memcmp(&r, &q, 4) != 0;
    }
    const float r = std::fmaf(NAN, c.rh, NAN * c.rl);
    return n + (r == r);
}
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
    lib = C.CDLL(str(so))
    for f in (lib.two_op_lo, lib.denominator):
        f.restype = C.c_float
    for f in (lib.two_op_choice, lib.two_op_lo):
        f.argtypes = [C.c_float]
    lib.two_op_wrong.argtypes = [C.c_float, C.c_int, C.c_int]
    return lib


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


DEFAULT_EXTENT = (1.15, 1.35, 1.15)


def denominator(plan, dims, extent=DEFAULT_EXTENT):
    return plan.denominator((C.c_int * 3)(*dims), (C.c_float * 3)(*extent))


@pytest.mark.parametrize("dims,extent", [((128, 192, 128), DEFAULT_EXTENT), ((4, 4, 4), (4.0, 6.0, 4.0)), ((2048, 2048, 2048), (0.5, 0.5, 0.5)),
                                         ((64, 96, 64), (1.0, 1.0, 1.0)), ((508, 508, 508), DEFAULT_EXTENT)])
def test_one_binade_decides_the_two_operation_quotient(plan, dims, extent):
    """A reciprocal that is exact over [1, 2) is exact in the lowest binades it is used in, in the
    highest, and in between: the engine checks the one binade on the device."""
    d = denominator(plan, dims, extent)
    k = plan.two_op_choice(d)
    assert k >= 0 and 0.0 < plan.two_op_lo(d) <= 2.0 ** -60
    for e in (1000, 1001, -40, 1, 60, 127):
        assert plan.two_op_wrong(d, k, e) == 0, (d, k, e)


def test_fixed_divisors_of_the_source_pass(plan):
    """The literals of fx_div_two_of, from the smallest magnitude they are used for (slot 0 divides sums
    down to 2^-100, the others differences from a constant of at least 0.3); from 2^-98 on the
    products by both parts of slot 0's reciprocal are normal, so the binades between repeat [1, 2)."""
    for slot in range(8):
        for e in ((-100, -99, -98) if slot == 0 else (-27, -26)) + (0, 1, 24, 127 if slot != 1 else 125):
            assert plan.fixed_wrong(slot, e) == 0, (slot, e)
        assert plan.fixed_specials(slot) == 0, slot
