"""The neighbour search by cell against the oracle's lists, element for element: bodies with few and many points
a cell, cells too sparse or too crowded for it (the per-point search), coincident points, distances on the threshold,
and coordinates far from the origin or far from one in size."""
import numpy as np
import pytest

import oracle as O
import vpd

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def lattice(nx, ny, nz):
    return np.stack(np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij"), -1).reshape(-1, 3) * 1.0


def cloud(kind):
    rng = np.random.default_rng(5)
    if kind == "one":
        return np.zeros((1, 3)), 1.0
    if kind == "pair":
        return np.array([[0.0, 0.0, 0.0], [1.0, 0.0, 0.0]]), 1.0
    if kind == "lattice_threshold":          # 24 of a point's bonds lie exactly on the horizon
        return lattice(17, 9, 11) * 0.1, 0.3
    if kind == "lattice_jitter":
        p = lattice(19, 13, 10)
        return (p + rng.uniform(-0.05, 0.05, p.shape)) * 0.1, 0.4015
    if kind == "shuffled":                   # no index order to rely on
        return rng.permutation(lattice(15, 14, 9)) * 0.1 + 3.0, 0.3015
    if kind == "random":
        return rng.uniform(0, 1, (4000, 3)), 0.17
    if kind == "sparse":                     # under one point a cell
        return rng.uniform(0, 1, (3000, 3)), 0.03
    if kind == "crowded":                    # more candidates around a cell than shared memory holds
        return rng.normal(0, 1, (6000, 3)) * 0.2, 0.5
    if kind == "coincident":
        return np.repeat(rng.uniform(0, 1, (300, 3)), 3, axis=0), 0.3
    if kind == "far":
        return lattice(12, 9, 9) + 1.0e9, 3.0
    if kind == "tiny":
        return lattice(12, 9, 9) * 1.0e-40, 3.015e-40
    if kind == "full_cells":                 # 4096 candidates at most: the largest sort of the search by cell
        return lattice(18, 18, 18), 5.01
    raise ValueError(kind)


@pytest.mark.parametrize("kind", ["one", "pair", "lattice_threshold", "lattice_jitter", "shuffled", "random", "sparse",
                                  "crowded", "coincident", "far", "tiny", "full_cells"])
def test_lists_equal_the_oracle(kind):
    pos, horizon = cloud(kind)
    want_ptr, want_col = O.neighbor_list(np.ascontiguousarray(pos), horizon)
    row_ptr, col = vpd.build_neighbor_list(torch.as_tensor(np.ascontiguousarray(pos)).cuda(), horizon)
    assert np.array_equal(row_ptr.cpu().numpy(), want_ptr)
    assert np.array_equal(col.cpu().numpy(), want_col[:len(col)])
