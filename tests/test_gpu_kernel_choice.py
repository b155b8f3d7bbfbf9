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


def seconds(call, count=20):
    for _ in range(3):
        call()
    best = float("inf")
    for _ in range(5):
        torch.cuda.synchronize()
        start = time.perf_counter()
        for _ in range(count):
            call()
        torch.cuda.synchronize()
        best = min(best, (time.perf_counter() - start) / count)
    return best


# a large body with a few bonds a point: all but the row's lengths and indices is a pass over memory
@pytest.mark.parametrize("bonds", [4, 8, 18])
def test_bond_sums_over_short_rows_take_at_most_four_times_a_copy(bonds):
    n = 1_000_000
    pos, disp = (torch.randn((n, 3), dtype=torch.float64, device="cuda") for _ in range(2))
    vol = torch.rand(n, dtype=torch.float64, device="cuda") + 0.5
    row_ptr = bonds * torch.arange(n + 1, dtype=torch.int64, device="cuda")
    col = (torch.arange(n, dtype=torch.int32, device="cuda")[:, None] +
           torch.arange(1, bonds + 1, dtype=torch.int32, device="cuda")).remainder(n).to(torch.int32).reshape(-1).contiguous()
    kinv = torch.randn((n, 9), dtype=torch.float64, device="cuda")
    bond = torch.zeros(bonds * n, dtype=torch.float64, device="cuda")
    # read: rows and their indices, points and displacements; K^-1, F or the bonds' damage and the index
    deformation = 8 * n + 4 * bonds * n + 56 * n + 144 * n
    damage = 8 * n + 4 * bonds * n + 56 * n + 8 * bonds * n + 8 * n
    for moved, call in ((deformation, lambda: vpd.deformation_gradients(pos, disp, vol, row_ptr, col, kinv)),
                        (damage, lambda: vpd.damage_update(pos, disp, vol, row_ptr, col, 0.5, 0.0, bond))):
        a = torch.empty(moved // 2, dtype=torch.uint8, device="cuda")
        b = torch.empty_like(a)
        assert seconds(call) <= 4.0 * seconds(lambda: b.copy_(a))


def test_neighbour_lists_of_one_cell_take_at_most_six_times_those_of_many():
    """All points in one cell (3,374 bonds each) against the same body in 125 cells (96 bonds)."""
    pos = np.stack(np.meshgrid(*[np.arange(15.0)] * 3, indexing="ij"), -1).reshape(-1, 3)
    x = torch.as_tensor(pos).cuda()
    assert seconds(lambda: vpd.build_neighbor_list(x, 30.0)) <= 6.0 * seconds(lambda: vpd.build_neighbor_list(x, 3.015))


def test_neighbour_lists_of_plates_and_lines_take_less_time_than_those_of_a_body():
    """1M points at two spacings: 12 bonds and nine cells to look into in a plate, 4 and 3 in a line, 31 and 27 in a body."""
    x, y, z = (torch.as_tensor(np.stack(np.meshgrid(*[np.arange(float(k)) for k in shape], indexing="ij"), -1).reshape(-1, 3)).cuda()
               for shape in ((1000, 1000, 1), (100, 100, 100), (1000000, 1, 1)))
    body = seconds(lambda: vpd.build_neighbor_list(y, 2.015), 5)
    assert seconds(lambda: vpd.build_neighbor_list(x, 2.015), 5) <= 0.95 * body
    assert seconds(lambda: vpd.build_neighbor_list(z, 2.015), 5) <= 0.95 * body
