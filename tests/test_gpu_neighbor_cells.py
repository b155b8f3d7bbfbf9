"""The neighbour search where several blocks share a cell's points, against the oracle's lists, element for element."""
import numpy as np
import pytest

import oracle as O
import vpd

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def cloud(kind):
    rng = np.random.default_rng(7)
    if kind.startswith("one_cell"):          # every point a candidate of every other
        return rng.uniform(0.0, 1.0, (int(kind.split()[1]), 3)), 30.0
    if kind == "few_cells":
        return rng.uniform(0.0, 1.0, (2744, 3)), 0.7
    if kind == "cluster":                    # one crowded cell among sparse ones
        sparse = rng.uniform(0.0, 8.0, (2500, 3))
        return np.concatenate([sparse, 4.5 + 0.3 * rng.uniform(0.0, 1.0, (3001, 3))]), 1.0
    raise ValueError(kind)


@pytest.mark.parametrize("kind", ["one_cell 2", "one_cell 32", "one_cell 33", "one_cell 65", "one_cell 1000", "one_cell 3375",
                                  "one_cell 4096", "one_cell 4097", "few_cells", "cluster"])
def test_lists_equal_the_oracle(kind):
    pos, horizon = cloud(kind)
    want_ptr, want_col = O.neighbor_list(np.ascontiguousarray(pos), horizon)
    row_ptr, col = vpd.build_neighbor_list(torch.as_tensor(np.ascontiguousarray(pos)).cuda(), horizon)
    assert np.array_equal(row_ptr.cpu().numpy(), want_ptr)
    assert np.array_equal(col.cpu().numpy(), want_col[:len(col)])


# points a cell on either side of where the search by cell begins, in bodies, plates and lines
@pytest.mark.parametrize("shape,horizon", [((14, 14, 14), 1.7), ((14, 14, 14), 1.72), ((14, 14, 14), 2.015),
                                           ((60, 40, 1), 2.8), ((60, 40, 1), 2.9), ((60, 40, 1), 3.015),
                                           ((1, 3000, 1), 13.5), ((1, 3000, 1), 14.5), ((4, 4, 4), 9.0)])
def test_lists_on_either_side_of_the_search_by_cell(shape, horizon):
    pos = np.stack(np.meshgrid(*[np.arange(float(k)) for k in shape], indexing="ij"), -1).reshape(-1, 3)
    want_ptr, want_col = O.neighbor_list(np.ascontiguousarray(pos), horizon)
    row_ptr, col = vpd.build_neighbor_list(torch.as_tensor(pos).cuda(), horizon)
    assert np.array_equal(row_ptr.cpu().numpy(), want_ptr)
    assert np.array_equal(col.cpu().numpy(), want_col[:len(col)])
