"""GPU tests of the register Jacobi's exchange buffer: it comes with the handle, so that no step
allocates device memory; it counts in device_bytes, is left out under a memory budget without room
for it; a batch of small members has its own from the call on that completed it."""
from __future__ import annotations

import numpy as np
import pytest

from fire_b200 import _abi as A
from fire_b200.serve import FireXServer, Request
from fire_b200.sim import FireXBatch, FireXSim, planned_device_bytes
from tests.helpers import DT, sphere_options

pytestmark = pytest.mark.gpu

FIELDS = ("flow", "species", "pressure", "reaction", "divergence", "correction")
DIMS = (64, 96, 64)


def same(a, b):
    assert a.state == b.state
    for f in FIELDS:
        x, y = a.read(f), b.read(f)
        assert np.array_equal(x, y), (f, float(np.abs(x.astype(np.float64) - y).max()))


def free_bytes():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_a_handles_first_step_allocates_nothing():
    def run():
        s = FireXSim(DIMS, sphere_options(DIMS))
        s.set_graphs(False)
        before = free_bytes()
        s.step(1, DT)
        s.sync()
        taken = before - free_bytes()
        assert s.diagnostics["jacobi_registers"] == 1
        s.close()
        return taken

    run()  # loads the kernels
    assert run() == 0


def test_the_buffer_counts_and_a_budget_without_room_goes_without():
    opts = sphere_options(DIMS, P=7, R=5)
    planned = planned_device_bytes(DIMS, opts)
    free, tight = FireXSim(DIMS, opts), None
    opts.memory_budget_bytes = planned
    tight = FireXSim(DIMS, opts)
    for s in (free, tight):
        s.step(2, DT)
        s.sync()
    assert free.diagnostics["jacobi_registers"] == 1 and tight.diagnostics["jacobi_registers"] == 0
    assert tight.device_bytes <= planned < free.device_bytes
    opts.memory_budget_bytes = free.device_bytes + (1 << 20)
    roomy = FireXSim(DIMS, opts)
    roomy.step(2, DT)
    roomy.sync()
    assert roomy.diagnostics["jacobi_registers"] == 1 and roomy.device_bytes <= opts.memory_budget_bytes
    same(free, tight)
    same(free, roomy)


def test_batches_have_their_own_buffer():
    """Boxes change with the company: alone, in three batches, alone again; tags of other boxes never match."""
    dims = [(32, 48, 32), (48, 64, 48), (36, 44, 28)]
    ref = [FireXSim(d, sphere_options(d, P=5, R=4, seed=i)) for i, d in enumerate(dims)]
    sims = [FireXSim(d, sphere_options(d, P=5, R=4, seed=i)) for i, d in enumerate(dims)]
    held = [s.device_bytes for s in sims]
    for r in ref:
        r.set_jacobi("unblocked")
        r.step(9, DT)
    for s in sims:
        s.step(2, DT)
    for group in (sims, sims[::-1], sims[:2]):
        with FireXBatch() as b:
            for s in group:
                b.add(s)
            b.step(2, DT)
            b.sync()
            assert group[0].diagnostics["jacobi_registers"] == 1
            for s in group:
                b.remove(s)
    for s, done in zip(sims, (8, 8, 6)):
        s.step(9 - done, DT)
        s.sync()
        assert s.diagnostics["jacobi_registers"] == 1
    for r, s in zip(ref, sims):
        same(r, s)
    assert [s.device_bytes for s in sims] == held


def test_a_batch_that_loses_its_large_member_runs_in_registers():
    small, large = (48, 64, 48), (128, 192, 128)
    opts = [sphere_options(d, P=5, R=4, seed=i) for i, d in enumerate((small, large, small))]
    sims = [FireXSim(d, o) for d, o in zip((small, large, small), opts)]
    ref = [FireXSim(small, opts[0]), FireXSim(small, opts[2])]
    for r in ref:
        r.set_jacobi("unblocked")
        r.step(4, DT)
    with FireXBatch() as b:
        for s in sims:
            b.add(s)
        b.step(2, DT)
        b.remove(sims[1])
        b.step(2, DT)
        b.sync()
        assert sims[0].diagnostics["jacobi_registers"] == 1
    same(sims[0], ref[0])
    same(sims[2], ref[1])


def test_the_server_stays_within_its_budget():
    opts = dict(pressure_iterations=4, correction_iterations=4)
    need = planned_device_bytes(DIMS, sphere_options(DIMS, P=4, R=4, precision=A.PRECISION_MIXED))
    for room in (need, int(2.05 * need), int(3.5 * need)):
        srv = FireXServer(budget_bytes=room, tick_target_ms=None)
        ids = [srv.submit(Request(dims=DIMS, steps=2, options=dict(opts, seed=i))) for i in range(3)]
        most = 0
        while True:
            srv._admit()
            held = sum(s.sim.device_bytes for s in srv.slots.values())
            assert held <= room and srv.used <= room, (held, srv.used, room)
            most = max(most, len(srv.slots))
            if not srv.tick():
                break
        assert most == room // need
        assert all(srv.poll(i)["status"] == "done" for i in ids) and srv.used == 0
        srv.close()
