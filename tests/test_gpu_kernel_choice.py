"""The rules that choose a kernel by size, held to the time of the other kernels over forms far from the sizes that
they were set at. The limits are wide (a factor of two and more): they catch a rule that takes the wrong
kernel, not a slow machine."""
import time

import numpy as np
import pytest

import vpd
from vpd.case import PRECISION_FP64, tensile_bar

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# small lattices with a long reach: a box's staged region has no room for more than a few points beside it
@pytest.mark.parametrize("dims,ratio", [((17, 17, 17), 5.015), ((40, 10, 10), 5.515), ((101, 21, 5), 5.015),
                                        ((12, 12, 12), 5.015), ((22, 22, 22), 4.015)])
@pytest.mark.parametrize("damage", [0, 1])
def test_small_lattice_increment_takes_at_most_half_as_long_again_as_the_tiles(monkeypatch, dims, ratio, damage):
    nx, ny, nz = dims
    case = tensile_bar(3, nx=nx, ny=ny, nz=nz, horizon=ratio * 0.1, damage_mode=damage, precision=PRECISION_FP64)
    best = {}
    for kind in ("tiles", ""):
        monkeypatch.setenv("VPD_BOND_KERNEL", kind)
        with vpd.Simulation(case) as sim:
            sim.step(32)
            best[kind] = min((sim.step(32), sim.last_step_ms())[1] for _ in range(5))
    assert best[""] <= 1.5 * best["tiles"]
