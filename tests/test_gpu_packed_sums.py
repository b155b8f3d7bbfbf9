"""The module functions' CSR sums at the sizes and mean row lengths where their lanes per row change and where they
take packed point records, against plain NumPy in float64: rows in no order, of another length each."""
import numpy as np
import pytest

import vpd

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def cuda(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a)).to(dtype=dtype, device="cuda").contiguous()


def body(n, bonds=8):
    """Rows of about `bonds` neighbours, some three fewer or more."""
    rng = np.random.default_rng(n)
    pos, vol = rng.standard_normal((n, 3)), 0.5 + rng.random(n)
    length = rng.integers(bonds - 3, bonds + 4, n)
    row_ptr = np.concatenate([[0], np.cumsum(length)])
    owner = np.repeat(np.arange(n), length)
    col = (owner + rng.integers(1, n, len(owner))) % n
    return rng, pos, vol, row_ptr, owner, col


def row_sums(values, row_ptr):
    return np.add.reduceat(values, row_ptr[:-1], axis=0)


@pytest.mark.parametrize("n,bonds", [(59_999, 8), (60_000, 8), (60_000, 23), (60_001, 25), (149_999, 8), (150_000, 8),
                                     (150_001, 19), (150_000, 21), (150_001, 63), (150_000, 65),
                                     (499_999, 8), (500_001, 8), (500_000, 66)])
def test_sums_match_numpy(n, bonds):
    rng, pos, vol, row_ptr, owner, col = body(n, bonds)
    disp = 0.01 * rng.standard_normal((n, 3))
    xi = pos[col] - pos[owner]
    X, V, P, C = cuda(pos), cuda(vol), cuda(row_ptr, torch.int64), cuda(col, torch.int32)
    K = row_sums(vol[col, None, None] * xi[:, :, None] * xi[:, None, :], row_ptr)
    cond = np.linalg.cond(K)
    ok = cond < 100.0
    assert ok.mean() > 0.5
    got = vpd.shape_tensor_inverse(X, V, P, C).cpu().numpy().reshape(n, 3, 3)
    want = np.linalg.inv(K[ok])
    # a determinant and cofactors of sums of at most 68 terms: roundings of some 50 ulp, grown by the condition number twice
    bound = 50 * 2.0 ** -52 * cond[ok] ** 2 * np.abs(want).max(axis=(1, 2))
    assert (np.abs(got[ok] - want).max(axis=(1, 2)) <= bound).all()
    kinv = rng.standard_normal((n, 9))
    G = row_sums((vol[col, None] * (disp[col] - disp[owner]))[:, :, None] * xi[:, None, :], row_ptr)
    want = np.eye(3) + G @ kinv.reshape(n, 3, 3)
    got = vpd.deformation_gradients(X, cuda(disp), V, P, C, cuda(kinv)).cpu().numpy().reshape(n, 3, 3)
    assert np.abs(got - want).max() <= 1e-12 * max(1.0, np.abs(want).max())
    F = np.eye(3) + 0.1 * rng.standard_normal((n, 3, 3))
    sigma = rng.standard_normal((n, 3, 3))
    bond = np.where(rng.random(len(col)) < 0.3, rng.choice([1.0, 0.25, -1.0, 2.0], len(col)), 0.0)
    M = np.linalg.det(F)[:, None, None] * sigma @ np.linalg.inv(F).transpose(0, 2, 1) @ kinv.reshape(n, 3, 3)
    w = (1.0 - np.clip(bond, 0, 1)) * vol[col]
    want = row_sums(w[:, None] * np.einsum("qab,qb->qa", M[owner] + M[col], xi), row_ptr)
    got = vpd.force_density(X, V, P, C, cuda(kinv), cuda(F.reshape(n, 9)), cuda(sigma.reshape(n, 9)), cuda(bond))
    # (a few of the random F are nearly singular: their M is large)
    assert np.abs(got.cpu().numpy() - want).max() <= 1e-12 * max(1.0, np.abs(M).max() * 70)


@pytest.mark.parametrize("n,bonds", [(15_999, 30), (16_000, 23), (16_000, 25), (16_001, 30), (60_000, 8), (60_001, 30),
                                     (99_999, 30), (100_000, 30),
                                     (150_001, 8), (150_000, 21), (150_001, 66)])
@pytest.mark.parametrize("failure", [0.0, 0.01])
def test_damage_decisions_match_the_reference_formula(n, bonds, failure):
    rng, pos, vol, row_ptr, owner, col = body(n, bonds)
    eps = 0.02
    # points scaled about the origin, so that stretches straddle the thresholds, some to the last bits
    disp = pos * (eps * (1.0 + 1e-12 * rng.standard_normal((n, 1)))) * rng.choice([1.0, 0.0, -0.6], (n, 1))
    bond = np.where(rng.random(len(col)) < 0.1, 0.5, 0.0)
    e, y = pos[col] - pos[owner], (pos[col] + disp[col]) - (pos[owner] + disp[owner])
    first = np.sqrt((e[:, 0] * e[:, 0] + e[:, 1] * e[:, 1]) + e[:, 2] * e[:, 2])
    now = np.sqrt((y[:, 0] * y[:, 0] + y[:, 1] * y[:, 1]) + y[:, 2] * y[:, 2])
    s = (now - first) / first
    want = np.where((s > eps) | ((failure > 0) & (s < -failure)), 1.0, bond)
    index = row_sums(want * vol[col], row_ptr) / row_sums(vol[col], row_ptr)
    B = cuda(bond)
    got = vpd.damage_update(cuda(pos), cuda(disp), cuda(vol), cuda(row_ptr, torch.int64), cuda(col, torch.int32), eps,
                            failure, B).cpu().numpy()
    assert np.array_equal(B.cpu().numpy(), want)
    assert np.abs(got - index).max() <= 1e-14
