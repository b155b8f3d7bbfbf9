"""The module functions' CSR bond sums (eight lanes per row) against plain NumPy in float64, on rows of every
length from empty through several passes of the lanes, in no lattice order, with bonds near the
critical-stretch thresholds."""
import numpy as np
import pytest

import vpd

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def cuda(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a)).to(dtype=dtype, device="cuda").contiguous()


def body(n, longest, seed):
    rng = np.random.default_rng(seed)
    pos, vol = rng.standard_normal((n, 3)), 0.5 + rng.random(n)
    rows = [rng.permutation(np.delete(np.arange(n), i))[: min(n - 1, (i * 7) % (longest + 1))] for i in range(n)]
    row_ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
    return rng, pos, vol, rows, row_ptr, np.concatenate(rows + [np.zeros(0, int)])


@pytest.mark.parametrize("n,longest", [(1, 0), (5, 3), (33, 8), (257, 9), (300, 70)])
def test_bond_sums_match_numpy(n, longest):
    rng, pos, vol, rows, row_ptr, col = body(n, longest, n)
    disp = 0.01 * rng.standard_normal((n, 3))
    kinv = rng.standard_normal((n, 9))
    F = np.eye(3).reshape(1, 9) + 0.1 * rng.standard_normal((n, 9))
    sigma = rng.standard_normal((n, 9))
    bond = np.where(rng.random(len(col)) < 0.3, rng.choice([1.0, 0.25, -1.0, 2.0], len(col)), 0.0)
    M = np.stack([np.linalg.det(f) * s @ np.linalg.inv(f).T @ k for f, s, k in
                  zip(F.reshape(-1, 3, 3), sigma.reshape(-1, 3, 3), kinv.reshape(-1, 3, 3))])
    wantF, wantf = np.empty((n, 9)), np.empty((n, 3))
    for i, r in enumerate(rows):
        xi, v = pos[r] - pos[i], vol[r]
        wantF[i] = (np.eye(3) + ((v[:, None] * (disp[r] - disp[i])).T @ xi) @ kinv[i].reshape(3, 3)).ravel()
        w = (1.0 - np.clip(bond[row_ptr[i]:row_ptr[i + 1]], 0, 1)) * v
        wantf[i] = np.einsum("j,jab,jb->a", w, M[i] + M[r], xi)
    X, V, P = cuda(pos), cuda(vol), cuda(row_ptr, torch.int64)
    C = cuda(col if len(col) else np.zeros(1), torch.int32)
    args = (X, V, P, C)
    got = vpd.deformation_gradients(X, cuda(disp), V, P, C, cuda(kinv)).cpu().numpy()
    # sums of at most 70 terms: roundings of a few hundred ulp of the largest term
    assert np.abs(got - wantF).max() <= 1e-12 * max(1.0, np.abs(wantF).max())
    scale = 1e-12 * max(1.0, np.abs(M).max() * 70)
    B = cuda(bond if len(bond) else np.zeros(1))
    assert np.abs(vpd.force_density(*args, cuda(kinv), cuda(F), cuda(sigma), B).cpu().numpy() - wantf).max() <= scale
    out = torch.empty((n, 3), dtype=torch.float64, device="cuda")
    vpd.force_density_noalloc(*args, cuda(kinv), cuda(F), cuda(sigma), out, B)
    assert np.abs(out.cpu().numpy() - wantf).max() <= scale


@pytest.mark.parametrize("failure", [0.0, 0.01, 1.0])
@pytest.mark.parametrize("n,longest", [(5, 3), (257, 9), (300, 70)])
def test_damage_decisions_match_the_reference_formula(n, longest, failure):
    rng, pos, vol, rows, row_ptr, col = body(n, longest, n + 1)
    eps = 0.02
    # each point scaled about the origin so that stretches straddle the thresholds, some to the last bits; some
    # bonds of zero length (coincident points) and some that do not change
    disp = pos * (eps * (1.0 + 1e-12 * rng.standard_normal((n, 1)))) * rng.choice([1.0, 0.0, -0.6], (n, 1))
    pos[n // 2], disp[n // 2] = pos[0], disp[0]
    bond = np.where(rng.random(len(col)) < 0.1, 0.5, 0.0)
    want, index = bond.copy(), np.zeros(n)
    for i, r in enumerate(rows):
        if not len(r):
            continue
        e, yy = pos[r] - pos[i], (pos[r] + disp[r]) - (pos[i] + disp[i])
        with np.errstate(all="ignore"):
            ln = np.sqrt((e[:, 0] * e[:, 0] + e[:, 1] * e[:, 1]) + e[:, 2] * e[:, 2])
            cur = np.sqrt((yy[:, 0] * yy[:, 0] + yy[:, 1] * yy[:, 1]) + yy[:, 2] * yy[:, 2])
            s = (cur - ln) / ln
        s_ = slice(row_ptr[i], row_ptr[i + 1])
        want[s_][(s > eps) | ((failure > 0) & (s < -failure))] = 1.0
        index[i] = (want[s_] * vol[r]).sum() / vol[r].sum()
    B = cuda(bond)
    got = vpd.damage_update(cuda(pos), cuda(disp), cuda(vol), cuda(row_ptr, torch.int64), cuda(col, torch.int32), eps,
                            failure, B).cpu().numpy()
    assert np.array_equal(B.cpu().numpy(), want)
    assert np.abs(got - index).max() <= 1e-14
