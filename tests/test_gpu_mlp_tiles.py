"""The network kernels' tiles: batches around multiples of 128 rows and of the persistent forward kernel's
148 x 4 tiles, and arrays that start between 16-byte boundaries."""
import numpy as np
import pytest

import mlp as M
import vpd

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def rows(batch, seed, offset):
    """[batch][16] normals with 10 live columns, starting `offset` floats into an aligned buffer."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    flat = torch.zeros(batch * 16 + 4, device="cuda")
    x = flat[offset:offset + batch * 16].view(batch, 16)
    x[:, :10] = torch.randn((batch, 10), generator=g, device="cuda")
    return x


def network(seed):
    w, b = M.init_params(seed)
    wt = torch.as_tensor(np.asarray(w).view(np.int16)).cuda()
    return w, b, wt, torch.as_tensor(np.asarray(b, np.float32)).cuda()


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("batch", [1, 127, 128, 129, 592 * 128 - 1, 592 * 128 + 1])
def test_forward_rows_do_not_depend_on_their_tile(batch, offset):
    w, b, wt, bt = network(11)
    x = rows(batch, batch, offset)
    got = vpd.mlp_forward(wt, bt, x)
    pick = sorted({0, batch // 2, max(0, batch - 129), batch - 1})
    alone = torch.cat([vpd.mlp_forward(wt, bt, x[k:k + 1]) for k in pick])
    assert torch.equal(got[pick], alone)
    want = M.forward(w, b, x[pick].cpu().numpy())
    # BF16 rounding flips of single activations (the tolerance of tests/test_mlp.py, per row instead of per batch)
    assert np.linalg.norm(alone.cpu().numpy() - want) <= 1e-2 * np.linalg.norm(want)


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("batch", [1, 127, 129, 700])
def test_gradients_of_ragged_batches(batch, offset):
    w, b, wt, bt = network(12)
    x, g = rows(batch, batch, offset), rows(batch, batch + 1, offset) / batch
    g[:, 7:] = 0.0
    got = vpd.mlp_gradients(wt, bt, x, g.contiguous()).cpu().numpy()
    want = M.gradients(w, b, x.cpu().numpy(), g.cpu().numpy())
    assert np.linalg.norm(got - want) <= 5e-3 * np.linalg.norm(want)
    # the rows past the batch in the last tile contribute nothing: the same rows in a batch of one tile more
    pad = torch.cat([x, torch.ones((128, 16), device="cuda")]), torch.cat([g, torch.zeros((128, 16), device="cuda")])
    padded = vpd.mlp_gradients(wt, bt, *pad).cpu().numpy()
    assert np.linalg.norm(got - padded) <= 1e-6 * np.linalg.norm(got)
