"""GPU tests that tell the two forms of the resident Jacobi's variant 4 apart. The planner takes
the pressure in registers (fx_jacobi_reg.cuh) where columns are short; asked for by number,
variant 4 is the copy warp (fx_jacobi_res.cuh, fx_res_copier) on every grid it fits. Each runs
here where it is certain which ran: bit for bit like one sweep per launch, in a batch, and
its bounded waits expiring when a box withholds its faces."""
from __future__ import annotations

import numpy as np
import pytest

from fire_b200 import _abi as A
from fire_b200.sim import FireXBatch, FireXError, FireXSim
from oracle.oracle import OracleSim
from tests.helpers import DT, sphere_options

pytestmark = pytest.mark.gpu

FIELDS = ("flow", "species", "pressure", "reaction", "divergence", "correction")


def same(a, b):
    assert a.state == b.state
    for f in FIELDS:
        x, y = a.read(f), b.read(f)
        assert np.array_equal(x, y), (f, float(np.abs(x.astype(np.float64) - y).max()))


def variant4(s, registers):
    d = s.diagnostics
    assert d["jacobi_kernel"] == A.JACOBI_RESIDENT and d["jacobi_variant"] == 4, d
    assert d["jacobi_registers"] == registers, d


@pytest.mark.parametrize("mode", [A.PRESSURE_WARM_F32, A.PRESSURE_COLD_F32])
@pytest.mark.parametrize("dims,P,R", [((96, 144, 96), 12, 9), ((80, 120, 80), 1, 2), ((132, 96, 64), 7, 4),
                                      ((100, 120, 88), 2, 1), ((64, 96, 128), 5, 6)])
def test_variant4_by_number_is_the_copy_warp(dims, P, R, mode):
    """Grids on which the pressure would also fit in registers."""
    opts = sphere_options(dims, P=P, R=R, pressure_mode=mode)
    one, copy = FireXSim(dims, opts), FireXSim(dims, opts)
    one.set_jacobi("unblocked")
    copy.set_jacobi("resident", 5)
    one.step(3, DT)
    copy.step(3, DT)
    variant4(copy, registers=0)
    same(one, copy)
    one.close()
    copy.close()


def test_the_planner_takes_registers_for_short_columns():
    for dims in ((32, 48, 32), (64, 96, 64), (96, 144, 96)):
        g = FireXSim(dims, sphere_options(dims, P=6, R=5))
        g.step(1, DT)
        variant4(g, registers=1)
        g.set_jacobi("resident")
        g.step(1, DT)
        variant4(g, registers=1)
        g.close()


def test_the_planner_takes_the_copy_warp_for_crowded_boxes_of_wide_rows():
    dims = (256, 64, 64)
    opts = sphere_options(dims, P=6, R=5)
    one, g = FireXSim(dims, opts), FireXSim(dims, opts)
    one.set_jacobi("unblocked")
    one.step(2, DT)
    g.step(2, DT)
    variant4(g, registers=0)
    same(one, g)


def test_a_batch_of_small_members_shares_one_register_launch():
    dims = [(32, 48, 32), (36, 44, 28), (48, 64, 48), (32, 48, 32)]
    alone = [FireXSim(d, sphere_options(d, P=7 + i, R=6 - i, seed=i)) for i, d in enumerate(dims)]
    members = [FireXSim(d, sphere_options(d, P=7 + i, R=6 - i, seed=i)) for i, d in enumerate(dims)]
    for s in alone:
        s.set_jacobi("unblocked")
        s.step(4, DT)
    with FireXBatch() as b:
        for m in members:
            b.add(m)
        b.step(4, DT)
        b.sync()
        variant4(members[0], registers=1)
        assert members[0].diagnostics["jacobi_kernel"] == A.JACOBI_RESIDENT
    for a, m in zip(alone, members):
        same(a, m)


@pytest.mark.parametrize("registers,dims", [(1, (64, 96, 64)), (0, (80, 120, 80))])
@pytest.mark.parametrize("sweep", [3, 11])
def test_withheld_face_expires_the_waits(registers, dims, sweep):
    """Sweep 11 of 12 is the last: only the residual phase's projection waits for its faces."""
    opts = sphere_options(dims, P=12, R=12)

    def handle():
        s = FireXSim(dims, opts)
        s.set_jacobi("resident", 0 if registers else 5)
        return s

    g = handle()
    g.step(1, DT)
    g.sync()
    variant4(g, registers)
    assert g.diagnostics["project_resident"] == 1
    g.set_wait_limit(4096)
    g.test_hold_face(0, sweep)
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
    variant4(h, registers)
    same(h, o)
    h.close()
