"""The bond kernels' shapes by lattice size against one another, bit for bit, on bars that are coming apart: bonds break
in the deformation kernel and leave the force sum, and some hold."""
import numpy as np
import pytest

import vpd
from vpd.case import PRECISION_FP64, PRECISION_MIXED, tensile_bar

pytestmark = pytest.mark.gpu

FIELDS = ("displacement", "velocity", "stress_corotational", "state", "damage_index", "force_density")


def run(case, monkeypatch, kinds, steps):
    out = {}
    for kind in kinds:
        monkeypatch.setenv("VPD_BOND_KERNEL", kind)
        with vpd.Simulation(case) as sim:
            rows = sim.step(steps)
            out[kind] = {f: sim.field(f) for f in FIELDS} | {"rows": rows}
    index = out[kinds[0]]["damage_index"]
    assert index.max() > 0.0, "no bond broke"
    assert np.count_nonzero((index > 0.0) & (index < 1.0)) > 0, "no damaged point kept a bond"
    assert index.min() < 1.0
    for kind in kinds[1:]:
        for f, want in out[kinds[0]].items():
            assert np.array_equal(out[kind][f], want), (kind, f)


# boxes of 32, 64 and 128 points; the tiled kernels beyond
@pytest.mark.parametrize("dims,ratio", [((9, 2, 3), 3.015), ((13, 5, 7), 4.015), ((41, 10, 11), 3.0), ((31, 13, 17), 4.015),
                                        ((40, 17, 19), 3.015), ((17, 9, 8), 6.015)])
def test_boxes_and_tiles_fp64(monkeypatch, dims, ratio):
    nx, ny, nz = dims
    case = tensile_bar(3, nx=nx, ny=ny, nz=nz, horizon=ratio * 0.1, damage_mode=1, damage_initiation=0.001,
                       precision=PRECISION_FP64)
    run(case, monkeypatch, ("slot", "box", "tiles", ""), 150)


# a warp per stencil plane and a thread per tile
@pytest.mark.parametrize("dims,ratio", [((8, 3, 5), 4.0), ((13, 5, 7), 3.015), ((24, 21, 17), 4.015), ((19, 12, 13), 5.015),
                                        ((41, 10, 11), 3.0)])
def test_planes_and_pairs_mixed(monkeypatch, dims, ratio):
    nx, ny, nz = dims
    case = tensile_bar(3, nx=nx, ny=ny, nz=nz, horizon=ratio * 0.1, damage_mode=1, damage_initiation=0.001,
                       precision=PRECISION_MIXED)
    run(case, monkeypatch, ("pair", "planes", ""), 150)


# block shapes of the thread-per-tile mixed kernels: 128, 192 and 256 threads
@pytest.mark.parametrize("dims", [(500, 16, 16), (97, 43, 37), (200, 40, 45), (260, 50, 50)])
def test_pair_block_shapes_mixed(monkeypatch, dims):
    nx, ny, nz = dims
    case = tensile_bar(3, nx=nx, ny=ny, nz=nz, damage_mode=1, damage_initiation=0.001, precision=PRECISION_MIXED)
    run(case, monkeypatch, ("planes", "pair"), 60)


# stencils on either side of 16 and 22 mask words, from where on the blocks are larger
@pytest.mark.parametrize("ratio", [4.4, 4.515, 4.9, 5.015])
def test_pair_block_shapes_of_long_stencils_mixed(monkeypatch, ratio):
    case = tensile_bar(3, nx=1000, ny=20, nz=10, horizon=ratio * 0.1, damage_mode=1, damage_initiation=0.001,
                       precision=PRECISION_MIXED)
    run(case, monkeypatch, ("planes", "pair"), 60)


# wide cross-sections: last waves of the deformation blocks filled by 0.37, 0.58 and 0.26
@pytest.mark.parametrize("dims", [(100, 45, 45), (150, 40, 40), (70, 70, 70)])
@pytest.mark.parametrize("ratio", [3.015, 4.015, 5.015])
def test_block_shapes_of_wide_cross_sections(monkeypatch, dims, ratio):
    nx, ny, nz = dims
    for precision, kinds in ((PRECISION_MIXED, ("planes", "pair")), (PRECISION_FP64, ("slot", "tiles"))):
        case = tensile_bar(3, nx=nx, ny=ny, nz=nz, horizon=ratio * 0.1, damage_mode=1, damage_initiation=0.001,
                           precision=precision)
        run(case, monkeypatch, kinds, 60)
