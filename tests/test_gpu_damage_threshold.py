"""Bond breaking in compression where the threshold lies close to a bond of no length, against the reference's
formula bit for bit: there the formula's own rounding of the stretch, 1e-16 of the initial length, is far more than
1e-16 of the current one."""
import numpy as np
import pytest

import vpd

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def cuda(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a)).to(dtype=dtype, device="cuda").contiguous()


@pytest.mark.parametrize("left", [0.5, 0.011, 0.0099, 1e-4, 1e-6, 1e-8, 1e-10, 3e-16])
def test_compression_decisions_match_the_reference_formula(left):
    """Point 0 at the origin and bonds from it to the others, pressed to about `left` of their lengths."""
    rng = np.random.default_rng(11)
    n = 4000
    failure = 1.0 - left
    pos = rng.standard_normal((n, 3))
    pos[0] = 0.0
    target = pos * (1.0 - failure) * (1.0 + 4e-16 / left * rng.uniform(-1, 1, (n, 1)))
    disp = target - pos
    want = np.zeros(n - 1)
    e, y = pos[1:] - pos[0], (pos[1:] + disp[1:]) - (pos[0] + disp[0])
    first = np.sqrt((e[:, 0] * e[:, 0] + e[:, 1] * e[:, 1]) + e[:, 2] * e[:, 2])
    now = np.sqrt((y[:, 0] * y[:, 0] + y[:, 1] * y[:, 1]) + y[:, 2] * y[:, 2])
    want[(now - first) / first < -failure] = 1.0
    assert 0 < want.sum() < n - 1
    row_ptr = np.concatenate([[0], np.full(n, n - 1)])
    bond = cuda(np.zeros(n - 1))
    vpd.damage_update(cuda(pos), cuda(disp), cuda(np.ones(n)), cuda(row_ptr, torch.int64),
                      cuda(np.arange(1, n), torch.int32), 10.0, failure, bond)
    assert np.array_equal(bond.cpu().numpy(), want)
