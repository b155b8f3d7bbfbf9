"""The bond kernels' shapes by lattice size against one another, bit for bit. FP64 against the per-slot kernels:
both sum every point's bonds in slot order with the same operations."""
import numpy as np
import pytest

import vpd
from vpd.case import PRECISION_FP64, PRECISION_MIXED, tensile_bar

pytestmark = pytest.mark.gpu

FIELDS = ("displacement", "velocity", "stress_corotational", "state", "damage_index", "force_density")


# boxes of 32, 64 and 128 points, ragged in every direction; lattices thinner than the stencil; the longest
# reach whose region fits (6) and the first that does not (7: the tiled kernels); beyond the default's range
@pytest.mark.parametrize("dims,ratio", [((9, 2, 3), 3.015), ((13, 5, 7), 4.015), ((41, 10, 11), 3.0), ((31, 13, 17), 4.015),
                                        ((40, 17, 19), 3.015), ((12, 37, 70), 4.015), ((17, 9, 8), 6.015),
                                        ((17, 9, 8), 7.015)])
@pytest.mark.parametrize("damage", [0, 1])
def test_box_kernels_match_slot_kernels_bitwise(monkeypatch, dims, ratio, damage):
    nx, ny, nz = dims
    case = tensile_bar(3, nx=nx, ny=ny, nz=nz, horizon=ratio * 0.1, damage_mode=damage, damage_initiation=0.004,
                       precision=PRECISION_FP64)
    out = {}
    for kind in ("slot", "box", "tiles", ""):
        monkeypatch.setenv("VPD_BOND_KERNEL", kind)
        with vpd.Simulation(case) as sim:
            rows = sim.step(150)
            out[kind] = {f: sim.field(f) for f in FIELDS} | {"rows": rows}
    for kind in ("box", "tiles", ""):
        for f, want in out["slot"].items():
            assert np.array_equal(out[kind][f], want), (kind, f)


# the tile shapes of larger lattices: one point per thread in both kernels (20k points), two and three in small blocks
# (98k), three in the deformation too, one wave of it (155k), two again (210k)
@pytest.mark.parametrize("dims", [(33, 25, 24), (61, 41, 40), (80, 45, 43), (103, 46, 45)])
@pytest.mark.parametrize("damage", [0, 1])
def test_tile_shapes_match_slot_kernels_bitwise(monkeypatch, dims, damage):
    nx, ny, nz = dims
    case = tensile_bar(3, nx=nx, ny=ny, nz=nz, horizon=0.3015, damage_mode=damage, damage_initiation=0.002,
                       precision=PRECISION_FP64)
    out = {}
    for kind in ("slot", "tiles"):
        monkeypatch.setenv("VPD_BOND_KERNEL", kind)
        with vpd.Simulation(case) as sim:
            rows = sim.step(60)
            out[kind] = {f: sim.field(f) for f in FIELDS} | {"rows": rows}
    for f, want in out["slot"].items():
        assert np.array_equal(out["tiles"][f], want), f
    if damage:
        assert out["slot"]["damage_index"].max() > 0


# a warp per stencil plane (seven, nine and eleven planes; a lattice thinner than the stencil; ragged columns) and a
# thread per tile against each other in mixed precision: the plane partials are folded in the same order
@pytest.mark.parametrize("dims,ratio", [((8, 3, 5), 4.0), ((13, 5, 7), 3.015), ((24, 21, 17), 4.015), ((19, 12, 13), 5.015),
                                        ((41, 10, 11), 3.0)])
@pytest.mark.parametrize("damage", [0, 1])
def test_plane_split_mixed_kernels_match_bitwise(monkeypatch, dims, ratio, damage):
    nx, ny, nz = dims
    case = tensile_bar(3, nx=nx, ny=ny, nz=nz, horizon=ratio * 0.1, damage_mode=damage, damage_initiation=0.004,
                       precision=PRECISION_MIXED)
    out = {}
    for kind in ("pair", "planes", ""):
        monkeypatch.setenv("VPD_BOND_KERNEL", kind)
        with vpd.Simulation(case) as sim:
            rows = sim.step(150)
            out[kind] = {f: sim.field(f) for f in FIELDS} | {"rows": rows}
    for kind in ("planes", ""):
        for f, want in out["pair"].items():
            assert np.array_equal(out[kind][f], want), (kind, f)


# the thread-per-tile mixed kernels' block shapes against the plane split: one wave of 128 threads, one of 192, between two
# and three waves, above three (192 threads for the force, 256 for the damaged deformation)
@pytest.mark.parametrize("dims", [(500, 16, 16), (97, 43, 37), (200, 40, 45), (260, 50, 50)])
@pytest.mark.parametrize("damage", [0, 1])
def test_pair_shapes_match_plane_split_bitwise(monkeypatch, dims, damage):
    nx, ny, nz = dims
    case = tensile_bar(3, nx=nx, ny=ny, nz=nz, damage_mode=damage, damage_initiation=0.004, precision=PRECISION_MIXED)
    out = {}
    for kind in ("pair", "planes"):
        monkeypatch.setenv("VPD_BOND_KERNEL", kind)
        with vpd.Simulation(case) as sim:
            sim.step(60)
            out[kind] = {f: sim.field(f) for f in ("displacement", "force_density", "damage_index")}
    for f, want in out["pair"].items():
        assert np.array_equal(out["planes"][f], want), f
