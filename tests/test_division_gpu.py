"""GPU tests of the Jacobi's division by its denominator (fx_div_two, fx_step_math.cuh): grids whose
denominator has no two-operation quotient run every kernel's other instance, and must equal
single sweeps bit for bit; a change of the domain costs no exhaustive check of that quotient."""
from __future__ import annotations

import statistics
import time

import numpy as np
import pytest

from fire_b200 import _abi as A
from fire_b200.sim import FireXSim
from tests.helpers import DT, sphere_options

pytestmark = pytest.mark.gpu

FIELDS = ("flow", "species", "pressure", "reaction", "divergence", "correction")


def same(a, b):
    assert a.state == b.state
    for f in FIELDS:
        x, y = a.read(f), b.read(f)
        assert np.array_equal(x, y), (f, float(np.abs(x.astype(np.float64) - y).max()))


def run(dims, opts, jacobi, staging=A.STAGING_AUTO, steps=2):
    one, other = FireXSim(dims, opts), FireXSim(dims, opts)
    one.set_jacobi("unblocked")
    other.set_jacobi(*jacobi)
    other.set_staging(staging)
    one.step(steps, DT)
    other.step(steps, DT)
    d = other.diagnostics
    assert d["jacobi_two_op"] == 0, d
    same(one, other)
    one.close()
    other.close()
    return d


# none of the five roundings of the reciprocal is exact for these grids (default domain)
@pytest.mark.parametrize("noise", [0.05, 0.0])
@pytest.mark.parametrize("dims", [(84, 32, 20), (36, 100, 20), (92, 12, 68)])
def test_strips_without_the_two_operation_quotient(dims, noise):
    for mode, staging in ((A.PRESSURE_WARM_F32, A.STAGING_CPASYNC), (A.PRESSURE_COLD_F32, A.STAGING_TMA),
                          (A.PRESSURE_F16, A.STAGING_CPASYNC)):
        d = run(dims, sphere_options(dims, P=13, R=8, noise=noise, pressure_mode=mode), ("fused", 2, 7), staging)
        assert d["jacobi_block"] == 2 and d["jacobi_staging"] == staging, d


@pytest.mark.parametrize("noise", [0.05, 0.0])
@pytest.mark.parametrize("dims,registers", [((84, 32, 20), 1), ((36, 88, 100), 1), ((68, 136, 128), 0), ((100, 152, 76), 0)])
def test_resident_without_the_two_operation_quotient(dims, registers, noise):
    for R in (6, 0):  # with and without the projection inside the launch
        d = run(dims, sphere_options(dims, P=9, R=R, noise=noise), ("resident", 0 if registers else 5, 0))
        assert d["jacobi_variant"] == 4 and d["jacobi_registers"] == registers, d


def test_a_changed_domain_takes_its_own_quotient():
    dims = (64, 96, 64)
    opts = sphere_options(dims, P=9, R=6)
    one, reg = FireXSim(dims, opts), FireXSim(dims, opts)
    one.set_jacobi("unblocked")
    for width in (1.15, 1.97, 0.83, 1.15):
        for s in (one, reg):
            s.set_parameter("domainWidth", width)
            s.step(1, DT)
    same(one, reg)


def test_a_changed_domain_costs_no_exhaustive_check_of_the_quotient():
    """Every divisor has one check over all floats (a new oxygen rate makes one, a new domain one, the
    Jacobi denominator's); the two-operation quotient adds microseconds to it."""
    s = FireXSim((64, 96, 64), sphere_options((64, 96, 64)))

    def cost(name, values):
        times = []
        for v in values:
            t = time.perf_counter()
            s.set_parameter(name, v)
            times.append(time.perf_counter() - t)
        return statistics.median(times)

    cost("domainWidth", (1.31,))
    cost("oxygenRate", (0.71,))
    domain = cost("domainWidth", [1.32 + 0.013 * i for i in range(9)])
    oxygen = cost("oxygenRate", [0.72 + 0.013 * i for i in range(9)])
    assert oxygen > 1e-3, "each oxygen rate is new: it is checked"
    assert domain < 1.35 * oxygen, (domain, oxygen)
    s.close()


def test_fluid_at_rest_divides_as_fast_as_moving_fluid():
    """Once the fronts of a solve from rest have passed, zeros and small numerators take no slow path:
    steps 9 to 16 of a plume in still air cost the Jacobi what they cost in noise."""
    dims = (128, 192, 128)
    ms = {}
    for noise in (0.0, 0.05):
        best = float("inf")
        for _ in range(3):
            s = FireXSim(dims, sphere_options(dims, P=64, R=64, noise=noise))
            s.step(8, DT)
            s.set_profiling(True)
            s.pass_times()
            s.step(8, DT)
            best = min(best, s.pass_times()["jacobi"][0])
            s.close()
        ms[noise] = best
    assert ms[0.0] < 1.05 * ms[0.05], ms
