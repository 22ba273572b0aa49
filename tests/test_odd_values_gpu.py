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
