"""GPU test of a value that a program should not write but may: NaN in the oxygen of cells where nothing
burns, by the field itself or by a NaN velocity that advects it, reaches their products in a
step as it does in the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from fire_b200 import _abi as A
from fire_b200.sim import FireXSim
from oracle.oracle import OracleSim
from tests.helpers import DT, sphere_options

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [A.PRECISION_F32, A.PRECISION_MIXED])
@pytest.mark.parametrize("field,component", [("species", 1), ("flow", 0)])
@pytest.mark.parametrize("dt", [DT, 0.0])
def test_nan_oxygen_reaches_the_products_of_cold_cells(field, component, dt, precision):
    dims = (36, 44, 28)
    opts = sphere_options(dims, P=4, R=4, noise=0.0, precision=precision)
    g, o = FireXSim(dims, opts), OracleSim(dims, opts)
    o.step(2, DT)
    f = o.read(field)
    for cell in ((20, 30, 8), (0, 0, 0), (5, 40, 33)):
        f[cell + (component,)] = np.nan
    for name in ("flow", "species", "pressure"):
        x = f if name == field else o.read(name)
        g.write(name, x)
        o.write(name, x)
    st = o.state
    g.set_state(st["simulation_time"], st["frame_index"], st["species_index"], st["pressure_index"])
    g.step(1, dt)
    o.step(1, dt)
    a, b = np.isnan(g.read("species")[..., 2]), np.isnan(o.read("species")[..., 2])
    assert b.sum() >= 3
    assert np.array_equal(a, b), np.argwhere(a != b)[:8]


KERNELS = [("zmarch", 0, A.STAGING_AUTO), ("fused", 2, A.STAGING_CPASYNC), ("fused", 2, A.STAGING_TMA), ("resident", 0, A.STAGING_AUTO),
           ("resident", 5, A.STAGING_AUTO), ("resident", 4, A.STAGING_AUTO), ("resident", 2, A.STAGING_AUTO), ("resident", 1, A.STAGING_AUTO)]


@pytest.mark.parametrize("mode", [A.PRESSURE_WARM_F32, A.PRESSURE_F16])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 3e38, -0.0, 1e-44, 1e-30])
def test_odd_pressures_spread_alike_in_every_jacobi_kernel(value, mode):
    """One step with the value in a few cells of the pressure equals single unblocked sweeps, on a grid
    that every kernel takes; 84x32x20 has no two-operation quotient."""
    for dims in ((80, 120, 80), (84, 32, 20)):
        opts = sphere_options(dims, P=5, R=5, pressure_mode=mode)
        X, Y, Z = dims
        odd = None
        want = None
        for kernel in [("unblocked", 0, A.STAGING_AUTO)] + KERNELS:
            if mode == A.PRESSURE_F16 and kernel[2] == A.STAGING_TMA:
                continue
            s = FireXSim(dims, opts)
            s.set_jacobi("unblocked")
            s.step(1, DT)
            if odd is None:
                odd = s.read("pressure")
                for z, y, x in ((Z // 2, Y // 2, X // 2), (0, 0, 0), (Z - 1, Y - 2, X - 1), (3, 1, 30), (5, Y - 1, 7)):
                    odd[z, y, x] = value
            s.write("pressure", odd)
            s.set_jacobi(*kernel[:2])
            s.set_staging(kernel[2])
            s.step(1, DT)
            got = {f: s.read(f) for f in ("pressure", "flow", "divergence", "correction")}
            s.close()
            if want is None:
                want = got
            for f in want:
                assert np.array_equal(got[f], want[f], equal_nan=True), (dims, kernel, f)
