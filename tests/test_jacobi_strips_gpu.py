"""GPU tests of the two-sweep Jacobi pass by strips (fx_jacobi_zs.cuh) where it can go wrong: grids
one tile (32 x 14 cells) wide and high and one group or row beside it, single-group rows, chunks
of one plane and of the whole grid, both stagings, FP16 pressure, sweep counts that leave one to
three single sweeps, and solves that start from rest, whose fronts are below the range of the
two-operation quotient. Every case must equal single sweeps bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from fire_b200 import _abi as A
from fire_b200.sim import FireXSim
from oracle.oracle import OracleSim
from tests.helpers import DT, sphere_options

pytestmark = pytest.mark.gpu

FIELDS = ("flow", "species", "pressure", "reaction", "divergence", "correction")


def same(a, b):
    assert a.state == b.state
    for f in FIELDS:
        x, y = a.read(f), b.read(f)
        assert np.array_equal(x, y), (f, float(np.abs(x.astype(np.float64) - y).max()))


def pair(dims, steps=2, zc=0, staging=A.STAGING_AUTO, **kw):
    one, two = FireXSim(dims, sphere_options(dims, **kw)), FireXSim(dims, sphere_options(dims, **kw))
    one.set_jacobi("unblocked")
    two.set_jacobi("fused", 2, zc)
    two.set_staging(staging)
    one.step(steps, DT)
    two.step(steps, DT)
    assert two.diagnostics["jacobi_block"] == 2
    same(one, two)
    one.close()
    two.close()


@pytest.mark.parametrize("staging", [A.STAGING_CPASYNC, A.STAGING_TMA])
@pytest.mark.parametrize("dims", [(4, 12, 4), (8, 16, 4), (28, 28, 8), (32, 12, 8), (32, 28, 12), (36, 32, 8), (68, 16, 20)])
def test_tile_edges(dims, staging):
    for zc in (1, 7, 64):
        pair(dims, zc=zc, staging=staging, P=8, R=8)


@pytest.mark.parametrize("dims", [(4, 12, 4), (36, 16, 12), (100, 44, 8)])
def test_tile_edges_fp16_pressure(dims):
    pair(dims, zc=5, P=8, R=8, pressure_mode=A.PRESSURE_F16)


@pytest.mark.parametrize("P,R", [(4, 5), (6, 7), (13, 10)])
def test_remaining_single_sweeps(P, R):
    pair((36, 32, 20), P=P, R=R)


@pytest.mark.parametrize("mode", [A.PRESSURE_WARM_F32, A.PRESSURE_COLD_F32])
def test_fronts_of_a_solve_from_rest(mode):
    # no noise: the pressure spreads from the emitter through cells at rest and decays by about a
    # factor of six a cell, below the smallest float within the grid
    for staging in (A.STAGING_CPASYNC, A.STAGING_TMA):
        pair((64, 96, 64), zc=16, staging=staging, P=48, R=40, noise=0.0, pressure_mode=mode)


def test_auto_on_a_grid_beyond_the_chip_equals_single_sweeps_and_the_oracle():
    dims = (256, 144, 128)
    opts = sphere_options(dims, P=8, R=9)
    auto, one, o = FireXSim(dims, opts), FireXSim(dims, opts), OracleSim(dims, opts)
    one.set_jacobi("unblocked")
    for s in (auto, one, o):
        s.step(2, 0.0)
    d = auto.diagnostics
    assert d["jacobi_kernel"] == A.JACOBI_FUSED and d["jacobi_staging"] == A.STAGING_TMA, d
    same(auto, one)
    same(auto, o)


# ---- the resident variant with the pressure in registers (fx_jacobi_reg.cuh) -------------------

@pytest.mark.parametrize("dims", [(4, 12, 8), (8, 28, 4), (36, 20, 44), (100, 36, 20), (128, 8, 148), (260, 12, 16), (64, 96, 64)])
@pytest.mark.parametrize("P,R", [(1, 1), (7, 4)])
def test_registers_equal_single_sweeps(dims, P, R):
    """Rows of one group and of 25 and 65 (rows across warps), columns in overlapping parts, more boxes
    than planes or rows, and the slots of one to seven sweeps over three steps."""
    opts = sphere_options(dims, P=P, R=R)
    one, reg = FireXSim(dims, opts), FireXSim(dims, opts)
    one.set_jacobi("unblocked")
    one.step(3, DT)
    reg.step(3, DT)
    d = reg.diagnostics
    assert d["jacobi_kernel"] == A.JACOBI_RESIDENT and d["jacobi_variant"] == 4, d
    same(one, reg)


def test_registers_from_rest_and_cold():
    dims = (48, 64, 48)
    for mode in (A.PRESSURE_WARM_F32, A.PRESSURE_COLD_F32):
        opts = sphere_options(dims, P=40, R=24, noise=0.0, pressure_mode=mode)
        one, reg = FireXSim(dims, opts), FireXSim(dims, opts)
        one.set_jacobi("unblocked")
        one.step(2, DT)
        reg.step(2, DT)
        same(one, reg)


def test_registers_survive_a_change_of_members():
    """The exchange buffer is kept, regrown and cleared as the batch's members change."""
    from fire_b200.sim import FireXBatch
    dims = [(32, 48, 32), (48, 64, 48), (36, 44, 28)]
    alone = [FireXSim(d, sphere_options(d, P=6, R=5, seed=i)) for i, d in enumerate(dims)]
    sims = [FireXSim(d, sphere_options(d, P=6, R=5, seed=i)) for i, d in enumerate(dims)]
    for s in alone:
        s.set_jacobi("unblocked")
        s.step(4, DT)
    with FireXBatch() as b:
        b.add(sims[0])
        b.step(1, DT)
        b.add(sims[1])
        b.step(2, DT)
        b.remove(sims[0])
        b.add(sims[2])
        b.step(1, DT)
        b.remove(sims[1])
        b.step(3, DT)
        b.remove(sims[2])
    for s in sims[:2]:  # the fourth step of these, alone
        s.step(1, DT)
    for a, m in zip(alone, sims):
        same(a, m)


# ---- the copy-warp kernel's two-operation quotient (fx_jacobi_res.cuh, long columns) ------------

@pytest.mark.parametrize("P,R,noise,mode", [(40, 24, 0.0, A.PRESSURE_WARM_F32), (40, 24, 0.0, A.PRESSURE_COLD_F32),
                                            (1, 2, 0.18, A.PRESSURE_WARM_F32)])
def test_copy_warp_from_rest(P, R, noise, mode):
    dims = (128, 192, 128)
    opts = sphere_options(dims, P=P, R=R, noise=noise, pressure_mode=mode)
    one, res = FireXSim(dims, opts), FireXSim(dims, opts)
    one.set_jacobi("unblocked")
    one.step(2, DT)
    res.step(2, DT)
    d = res.diagnostics
    assert d["jacobi_kernel"] == A.JACOBI_RESIDENT and d["jacobi_variant"] == 4, d
    same(one, res)


# ---- the flattest grids: a tile's rows reach far above the top --------------------------------

@pytest.mark.parametrize("staging", [A.STAGING_CPASYNC, A.STAGING_TMA])
@pytest.mark.parametrize("dims", [(4, 4, 4), (36, 4, 12), (64, 4, 20), (36, 8, 12)])
def test_flat_grids(dims, staging):
    for zc in (1, 7, 64):
        pair(dims, zc=zc, staging=staging, P=8, R=8)


@pytest.mark.parametrize("dims", [(4, 4, 4), (36, 4, 12), (64, 8, 20)])
def test_flat_grids_fp16_pressure(dims):
    for zc in (1, 7):
        pair(dims, zc=zc, P=8, R=8, pressure_mode=A.PRESSURE_F16)


# ---- a wait on tensor loads that runs out -------------------------------------------------------

def test_unfinished_tensor_loads_expire_the_wait():
    """Chunk 0's first wait counts as run out: its CTA waits once more for its loads, reports and
    returns, the host answers with a timeout, and a fresh handle steps exactly."""
    from fire_b200.sim import FireXError
    dims = (36, 32, 20)
    opts = sphere_options(dims, P=4, R=4)

    def handle():
        s = FireXSim(dims, opts)
        s.set_jacobi("fused", 2, 7)
        s.set_staging(A.STAGING_TMA)
        return s

    g = handle()
    g.step(1, DT)
    g.sync()
    assert g.diagnostics["jacobi_staging"] == A.STAGING_TMA
    g.test_hold_face(0, 1)
    g.step(1, DT)
    with pytest.raises(FireXError) as e:
        g.sync()
    assert e.value.code == A.ERR_TIMEOUT
    with pytest.raises(FireXError) as e:
        g.step(1, DT)
    assert e.value.code == A.ERR_STATE
    g.close()
    h, o = handle(), OracleSim(dims, opts)
    h.step(2, 0.0)
    o.step(2, 0.0)
    same(h, o)
    h.close()


# ---- phases that AUTO does not fuse ----------------------------------------------------------------

def test_auto_runs_unblocked_sweeps_where_no_phase_fuses():
    """Beyond the chip and within L2: fewer than four sweeps, and members of different sweep counts."""
    from fire_b200.sim import FireXBatch
    s = FireXSim((160, 240, 160), sphere_options((160, 240, 160), P=2, R=3))
    s.step(1, DT)
    s.sync()
    assert s.diagnostics["jacobi_kernel"] == A.JACOBI_UNBLOCKED, s.diagnostics
    s.close()
    dims = (96, 144, 96)
    alone = [FireXSim(dims, sphere_options(dims, P=6 + i, R=9 - i, seed=i)) for i in range(4)]
    members = [FireXSim(dims, sphere_options(dims, P=6 + i, R=9 - i, seed=i)) for i in range(4)]
    for a in alone:
        a.set_jacobi("unblocked")
        a.step(2, DT)
    with FireXBatch() as b:
        for m in members:
            b.add(m)
        b.step(2, DT)
        b.sync()
        assert members[0].diagnostics["jacobi_kernel"] == A.JACOBI_UNBLOCKED, members[0].diagnostics
    for a, m in zip(alone, members):
        same(a, m)


# ---- a cold start's shared buffers -----------------------------------------------------------------

@pytest.mark.parametrize("P,R", [(13, 8), (5, 4), (7, 12), (8, 9), (6, 11), (13, 10), (8, 8)])
@pytest.mark.parametrize("staging", [A.STAGING_CPASYNC, A.STAGING_TMA])
def test_cold_start_leaves_the_last_two_sweeps(P, R, staging):
    """The pressure is read from buffer P mod 2, which both solves of a cold start share: with R of the
    other parity it holds the residual solve's last sweep but one."""
    pair((36, 32, 20), P=P, R=R, staging=staging, pressure_mode=A.PRESSURE_COLD_F32)


def test_auto_with_a_cold_start_beyond_the_chip():
    dims = (160, 216, 152)
    opts = sphere_options(dims, P=5, R=8, pressure_mode=A.PRESSURE_COLD_F32)
    auto, one = FireXSim(dims, opts), FireXSim(dims, opts)
    one.set_jacobi("unblocked")
    auto.step(2, DT)
    one.step(2, DT)
    assert auto.diagnostics["jacobi_kernel"] == A.JACOBI_FUSED
    same(auto, one)


# ---- the fitted chunk is kept with the members -----------------------------------------------------

def test_the_fitted_chunk_follows_the_members():
    """A batch's chunk is that of its present members: as in a batch that never had others."""
    from fire_b200.sim import FireXBatch
    dims = [(160, 216, 152), (128, 128, 96), (96, 144, 96)]

    def chunk(sims, b):
        b.step(1, DT)
        b.sync()
        d = sims[0].diagnostics
        assert d["jacobi_kernel"] == A.JACOBI_FUSED, d
        return d["jacobi_zrun"]

    want = {}
    for n in (1, 2, 3):
        sims = [FireXSim(d, sphere_options(d, P=8, R=8)) for d in dims[:n]]
        with FireXBatch() as b:
            for s in sims:
                b.add(s)
            want[n] = chunk(sims, b)
        for s in sims:
            s.close()
    assert len(set(want.values())) > 1, want
    sims = [FireXSim(d, sphere_options(d, P=8, R=8)) for d in dims]
    with FireXBatch() as b:
        for n, s in enumerate(sims, 1):
            b.add(s)
            assert chunk(sims, b) == want[n]
            assert chunk(sims, b) == want[n]
        b.remove(sims[2])
        assert chunk(sims, b) == want[2]
        b.set_jacobi("fused", 2, 9)
        assert chunk(sims, b) == 9
        b.set_jacobi("auto")
        assert chunk(sims, b) == want[2]


def test_a_step_call_makes_no_plan_anew():
    """The host's part of a step of 48 uneven members: a graph launch and a look at the members."""
    import statistics
    import time
    from fire_b200.sim import FireXBatch
    grids = [(64, 96, 64), (96, 144, 96), (128, 192, 128), (160, 240, 160)]
    sims = [FireXSim(grids[i % 4], sphere_options(grids[i % 4], P=4, R=4, precision=A.PRECISION_MIXED)) for i in range(48)]
    one = FireXSim(grids[0], sphere_options(grids[0], P=4, R=4))
    with FireXBatch() as b:
        for s in sims:
            b.add(s)

        def call(stepper):
            times = []
            for _ in range(25):
                stepper.sync()
                t = time.perf_counter()
                stepper.step(1, DT)
                times.append(time.perf_counter() - t)
            stepper.sync()
            return statistics.median(times[5:])

        batch, alone = call(b), call(one)
    assert batch < alone + 20e-6, (batch, alone)


@pytest.mark.parametrize("P,R,launches", [(6, 8, 4 + 4), (13, 10, 7 + 6), (4, 3, 2 + 3), (3, 2, 3 + 2), (16, 1, 8 + 1)])
def test_launches_of_a_fused_solve(P, R, launches):
    """An even number of two-sweep launches and up to three single sweeps, beside the step's own seven."""
    dims = (36, 32, 20)
    s = FireXSim(dims, sphere_options(dims, P=P, R=R))
    s.set_jacobi("fused", 2)
    s.step(1, DT)
    s.sync()
    assert s.diagnostics["launches_per_step"] == 7 + launches, s.diagnostics
    s.close()
