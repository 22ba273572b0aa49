"""CPU tests of the index maps and launch plans that the kernels and the engine share
(fire_b200/csrc/fx_plan.h), compiled here by the host compiler alone."""
from __future__ import annotations

import ctypes as C
import subprocess
import time
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
// smem of a plan over every box (-1: one does not fit), as fx_reg_smem has it from four of them
long long reg_smem_all(int X, int Y, int Z, int by, int nby, int nbz) {
    const FxResBox bx{by, (Z + nbz - 1) / nbz, nby, nbz};
    long long most = 0;
    for (int b = 0; b < nby * nbz; ++b) {
        const FxRegGeom g = fx_reg_geom(X, Y, Z, bx, b);
        if (g.cols > FX_REG_THREADS || g.len > FX_REG_MAXZ || g.cols * g.parts > FX_REG_THREADS ||
            2 * (g.ny + g.nz) * (X / 4) > FX_REG_MAXH * FX_REG_THREADS)
            return -1;
        most = std::max(most, fx_reg_smem_bytes(X, g));
    }
    return most;
}
long long reg_smem(int X, int Y, int Z, int by, int nby, int nbz) {
    return fx_reg_smem(X, Y, Z, FxResBox{by, (Z + nbz - 1) / nbz, nby, nbz});
}
int reg_plan(int n, const int* d, int cap, int* boxes) {  // by, nby, nbz of each member; 0: does not fit
    std::vector<FxResBox> b;
    int smem;
    if (!fx_res_assign(grids(n, d), cap, FX_RES_REGISTERS, &b, &smem)) return 0;
    for (int i = 0; i < n; ++i) {
        boxes[3 * i] = b[i].by;
        boxes[3 * i + 1] = b[i].nby;
        boxes[3 * i + 2] = b[i].nbz;
    }
    return smem;
}
long long reg_exchange(int X, int by, int bz, int nby, int nbz) {
    return FX_REG_EXCHANGE_HEAD + 16 * (long long)fx_reg_packets(X, FxResBox{by, bz, nby, nbz});
}
long long reg_exchange_most(int cap) { return fx_reg_exchange_most(cap); }
int reg_min_ctas(int X, int Y, int Z, int cap) { return fx_reg_min_ctas(X, Y, Z, cap); }
// every cell of the grid is stored by one thread of one box
int reg_covers(int X, int Y, int Z, int by, int nby, int nbz) {
    const FxResBox bx{by, (Z + nbz - 1) / nbz, nby, nbz};
    std::vector<int> owners((size_t)Y * Z);
    for (int b = 0; b < nby * nbz; ++b) {
        const FxRegGeom g = fx_reg_geom(X, Y, Z, bx, b);
        if (g.ny % 2 || g.len > FX_REG_MAXZ) return 0;
        auto start = [&](int r) { return g.parts > 1 ? r * (g.nz - g.len) / (g.parts - 1) : 0; };
        for (int r = 0; r < g.parts; ++r)
            for (int k = r > 0 ? start(r - 1) + g.len - start(r) : 0; k < g.len; ++k)
                for (int y = 0; y < g.ny; ++y) ++owners[(size_t)(g.z0 + start(r) + k) * Y + g.y0 + y];
    }
    for (int n : owners)
        if (n != 1) return 0;
    return 1;
}
int auto_tma(int n, const int* d) { return fx_zs_auto_tma(grids(n, d)); }
int reg_crowded(int X, int Y, int Z, int cap) {
    FxResBox bx;
    return fx_reg_box(X, Y, Z, cap, &bx) ? fx_reg_crowded(X, bx) : -1;
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
    for f in (lib.reg_smem, lib.reg_smem_all, lib.reg_exchange, lib.reg_exchange_most):
        f.restype = C.c_longlong
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
    ([(36, 60, 36)] * 60, 1, A.JACOBI_UNBLOCKED), ([(16, 512, 512)], 1, A.JACOBI_UNBLOCKED),
    # and those on which the strips are the faster
    ([(16, 512, 512)], 0, A.JACOBI_FUSED), ([(36, 60, 36)] * 60, 0, A.JACOBI_FUSED),
    ([(20, 48, 24)] * 256, 1, A.JACOBI_FUSED), ([(40, 60, 40)] * 48, 1, A.JACOBI_FUSED), ([(36, 60, 36)] * 120, 1, A.JACOBI_FUSED), ([(512, 8, 1024)], 1, A.JACOBI_FUSED),
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


CTAS = 148


def test_register_boxes_are_judged_by_their_largest(plan):
    """Four boxes of a plan stand for all of them, whatever the remainders."""
    fits = 0
    for X, Y, Z in [(4, 4, 4), (16, 24, 20), (32, 48, 32), (36, 44, 28), (64, 96, 64), (100, 148, 92), (20, 400, 200), (128, 8, 148)]:
        for by in range(2, min(Y, 40) + 1, 2):
            nby = -(-Y // by)
            for nbz in {n for n in (1, 2, 3, 5, 7, Z // 4, Z // 2, Z - 1) if 0 < n <= Z} | {Z}:
                want = plan.reg_smem_all(X, Y, Z, by, nby, nbz)
                assert plan.reg_smem(X, Y, Z, by, nby, nbz) == want, (X, Y, Z, by, nbz)
                fits += want >= 0
    assert fits > 100


@pytest.mark.parametrize("grids", [[(4, 4, 4)], [(16, 24, 16)], [(32, 48, 32)], [(36, 44, 28)], [(100, 148, 92)], [(96, 144, 96)],
                                   [(260, 12, 16)], [(64, 96, 64)] * 4, [(48, 72, 48), (32, 48, 32), (64, 96, 64)], [(16, 24, 16)] * 64])
def test_register_plans_cover_every_cell_once(plan, grids):
    boxes = (C.c_int * (3 * len(grids)))()
    assert plan.reg_plan(*flat(grids), CTAS, boxes)
    assert sum(boxes[3 * i + 1] * boxes[3 * i + 2] for i in range(len(grids))) <= CTAS
    for i, (X, Y, Z) in enumerate(grids):
        assert plan.reg_covers(X, Y, Z, *boxes[3 * i:3 * i + 3])


def test_a_plan_costs_less_than_the_step_it_prepares(plan):
    """The register plan of a preview grid, whose step takes 90 us on the device, made in the first step
    of a handle: 17 us when four boxes are judged per row height, 109 when all of them were."""
    grids, boxes = flat([(32, 48, 32)]), (C.c_int * 3)()
    best = min(_timed(lambda: plan.reg_plan(*grids, CTAS, boxes)) for _ in range(200))
    assert best < 50e-6, best


def _timed(f):
    t = time.perf_counter()
    f()
    return time.perf_counter() - t


@pytest.mark.parametrize("grids", [[(32, 48, 32)], [(100, 148, 92)], [(256, 64, 64)], [(64, 96, 64)] * 4, [(256, 32, 32)] * 4,
                                   [(48, 72, 48), (32, 48, 32), (64, 96, 64)], [(16, 24, 16)] * 64, [(128, 192, 128), (32, 48, 32)],
                                   [(64, 96, 64)] * 5, [(4, 4, 4)] * 148])
def test_a_batchs_exchange_buffer_serves_every_plan(plan, grids):
    """The batch reserves it when its members' fewest CTAs fit together, which is when a plan exists."""
    boxes = (C.c_int * (3 * len(grids)))()
    least = [plan.reg_min_ctas(*g, CTAS) for g in grids]
    fits = plan.reg_plan(*flat(grids), CTAS, boxes) != 0
    assert fits == (0 not in least and sum(least) <= CTAS)
    need = 0
    for i, (X, Y, Z) in enumerate(grids if fits else []):
        by, nby, nbz = boxes[3 * i:3 * i + 3]
        need += plan.reg_exchange(X, by, -(-Z // nbz), nby, nbz)
    assert need <= plan.reg_exchange_most(CTAS) + 128 * len(grids) and plan.reg_exchange_most(CTAS) < 15 << 20


@pytest.mark.parametrize("grids,tma", [([(32, 48, 32)] * 60, 0), ([(32, 48, 32)] * 200, 0), ([(28, 48, 32)] * 150, 0), ([(32, 96, 32)] * 90, 0),
                                       ([(20, 48, 24)] * 256, 0), ([(36, 48, 32)] * 150, 1), ([(16, 24, 16)] * 500, 1), ([(32, 512, 256)], 1),
                                       ([(160, 240, 160)], 1), ([(64, 96, 64)] * 16, 1), ([(32, 48, 32), (160, 240, 160)], 1)])
def test_auto_staging(plan, grids, tma):
    assert plan.auto_tma(*flat(grids)) == tma


@pytest.mark.parametrize("dims,crowded", [((256, 64, 64), 1), ((256, 60, 64), 1), ((252, 80, 44), 1), ((240, 96, 48), 0), ((240, 40, 100), 0),
                                          ((200, 80, 72), 0), ((256, 64, 48), 0), ((256, 48, 48), 0), ((304, 208, 16), 0), ((512, 32, 32), 0),
                                          ((96, 144, 96), 0), ((128, 128, 96), 0), ((60, 184, 144), 0)])
def test_where_the_copy_warp_is_faster_than_registers(plan, dims, crowded):
    assert plan.reg_crowded(*dims, CTAS) == crowded
