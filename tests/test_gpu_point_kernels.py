"""The pointwise module kernels (tensors copied through shared memory a block at a time): ragged last blocks, arrays
whose tensors are not on 16-byte boundaries, and points with singular kinematics."""
import numpy as np
import pytest

import vpd
from vpd.case import steel_props

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
NAMES = ("defgrad_old", "left_stretch", "rotation", "strain", "stress_corotational", "state", "temperature",
         "energy_internal", "energy_inelastic")


def inputs(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(s, generator=g, dtype=torch.float64, device="cuda")  # noqa: E731
    eye = torch.eye(3, dtype=torch.float64, device="cuda").reshape(1, 9)
    state = dict(defgrad_old=eye + 1e-3 * r(n, 9), left_stretch=eye + 0.0 * r(n, 9), rotation=eye + 0.0 * r(n, 9),
                 strain=r(n, 9), stress_corotational=200.0 * r(n, 9), state=torch.zeros((n, 6), dtype=torch.float64, device="cuda"),
                 temperature=r(n), energy_internal=r(n), energy_inelastic=r(n))
    s = state["stress_corotational"].reshape(n, 3, 3)
    state["stress_corotational"] = (0.5 * (s + s.mT)).reshape(n, 9).contiguous()
    state["state"][:, 0], state["state"][:, 2], state["state"][:, 3] = 1.0, 293.0, 350.0
    return eye + 4e-3 * r(n, 9), state


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 385])
def test_slices_give_the_same_bits(n):
    F, state = inputs(n + 1, n)
    whole = {k: v.clone() for k, v in state.items()}
    part = {k: v.clone()[1:] for k, v in state.items()}  # its tensors start 72 bytes on
    assert part["strain"].data_ptr() % 16 == 8 and part["strain"].is_contiguous()
    a = vpd.material_update(steel_props(), 1e-3, F, whole)
    b = vpd.material_update(steel_props(), 1e-3, F[1:], part)
    assert torch.equal(a[1:], b) and bool((whole["state"][:, 4] > 0).any() or n < 8)
    for k in NAMES:
        assert torch.equal(whole[k][1:], part[k]), k
    c = vpd.corotational_update(state["defgrad_old"], F, state["left_stretch"], state["rotation"], 1e-3)
    d = vpd.corotational_update(state["defgrad_old"][1:], F[1:], state["left_stretch"][1:], state["rotation"][1:], 1e-3)
    for k in c:
        assert torch.equal(c[k][1:], d[k]), k
        assert bool(torch.isfinite(c[k]).all())


@pytest.mark.parametrize("n", [1, 130])
def test_a_singular_point_keeps_its_fields(n):
    F, state = inputs(n, 3)
    bad = n // 2
    state["defgrad_old"][bad] = 0.0
    good = {k: v.clone() for k, v in state.items()}
    with pytest.raises(vpd.VpdError):
        vpd.material_update(steel_props(), 1e-3, F, good)
    for k in NAMES:
        assert torch.equal(good[k][bad], state[k][bad]), k
        if n > 1 and k in ("defgrad_old", "left_stretch", "strain", "energy_internal"):
            keep = torch.arange(n, device="cuda") != bad
            assert not bool((good[k][keep] == state[k][keep]).all()), k
    assert np.isfinite(good["strain"].cpu().numpy()).all()
