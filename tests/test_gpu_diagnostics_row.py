"""The diagnostic row's sums over one to three block groups (65,536 points each), against the
fields they sum."""
import numpy as np
import pytest

import vpd
from vpd.case import DIAG, tensile_bar

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("shape", [(9, 4, 4), (64, 32, 32), (65, 32, 32), (131, 32, 32)])
def test_row_sums_are_the_fields_sums(shape, precision):
    nx, ny, nz = shape
    case = tensile_bar(3, nx=nx, ny=ny, nz=nz, precision=precision, damage_mode=0)
    with vpd.Simulation(case) as sim:
        row = sim.step(4)[-1]
        v, f = sim.field("velocity"), sim.field("force_density")
        vol, eqps = sim.field("volume")[:, 0], sim.field("state")[:, 1]
    n, eps = len(vol), 2.0 ** -52
    kinetic = float((0.5 * case.density * vol * (v * v).sum(1)).sum())
    net = np.linalg.norm((f * vol[:, None]).sum(0))
    # a sum of n terms: n roundings of the sum of their absolute values at most, here and in the row
    assert abs(row[DIAG["kinetic_energy_Nmm"]] - kinetic) <= 2 * n * eps * kinetic
    assert abs(row[DIAG["net_internal_force_N"]] - net) <= 4 * n * eps * (np.abs(f) * vol[:, None]).sum()
    assert row[DIAG["max_eqps"]] == eqps.max()
    assert row[DIAG["step"]] == 4 and row[DIAG["finite"]] == 1.0
