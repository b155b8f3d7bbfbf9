"""Device memory of the module functions: what allocates and what does not, under capture too, and how much of it
stays with the library."""
import ctypes

import numpy as np
import pytest

import vpd

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

def cuda(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a)).to(dtype=dtype, device="cuda").contiguous()


class Step:
    """A ring of n points, each bonded to the next six, and the calls of an increment on it into buffers of its own."""

    def __init__(self, n):
        rng = np.random.default_rng(n)
        self.n = n
        self.pos, self.disp = cuda(rng.standard_normal((n, 3))), cuda(0.01 * rng.standard_normal((n, 3)))
        self.vol = cuda(0.5 + rng.random(n))
        self.row_ptr = cuda(6 * np.arange(n + 1), torch.int64)
        self.col = cuda((np.arange(n)[:, None] + np.arange(1, 7)) % n, torch.int32)
        self.kinv, self.F = torch.empty((n, 9), dtype=torch.float64, device="cuda"), cuda(np.tile(np.eye(3).ravel(), (n, 1)))
        self.sigma = cuda(rng.standard_normal((n, 9)))
        self.bond = torch.zeros(6 * n, dtype=torch.float64, device="cuda")
        self.index = torch.zeros(n, dtype=torch.float64, device="cuda")
        self.force = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()

    def call(self, name, *args):
        a = [vpd._ptr(v) if torch.is_tensor(v) else v for v in args]
        vpd._check(getattr(vpd.library(), name)(*a, vpd._stream()))

    def shape(self):
        self.call("vpd_shape_tensor_inverse", self.pos, self.vol, self.n, self.row_ptr, self.col, self.kinv)

    def deformation(self):
        self.call("vpd_deformation_gradients", self.pos, self.disp, self.vol, self.n, self.row_ptr, self.col, self.kinv,
                  self.F)

    def damage(self):
        self.call("vpd_damage_update", self.pos, self.disp, self.vol, self.n, self.row_ptr, self.col, 0.005, 0.0,
                  self.bond, self.index)

    def noalloc_force(self):
        self.call("vpd_force_density_noalloc", self.pos, self.vol, self.n, self.row_ptr, self.col, self.kinv, self.F,
                  self.sigma, self.bond, self.force)


def free_bytes():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def loaded():
    """Every kernel of the step's calls loaded (CUDA loads them lazily)."""
    for n in (64, 65_000):
        body = Step(n)
        body.shape(), body.deformation(), body.damage(), body.noalloc_force()


@pytest.mark.parametrize("n", [65536, 151_000])
def test_the_calls_of_an_increment_allocate_nothing(n):
    """For hosts that hand all device memory to their own pool (vpd_force_density_noalloc: up to 65,536 points)."""
    loaded()
    body = Step(n)
    before = free_bytes()
    body.shape(), body.deformation(), body.damage()
    if n <= 65536:
        body.noalloc_force()
    assert before - free_bytes() < 1 << 20  # (the pool grows by 32 MiB)


def test_captured_calls_hold_kernels_only():
    """The two calls that do not synchronise, at a size where packed records pay."""
    body = Step(151_000)
    body.shape(), body.deformation(), body.damage()
    torch.cuda.synchronize()
    want = body.F.clone(), body.bond.clone(), body.index.clone()
    body.F.zero_(), body.bond.zero_(), body.index.zero_()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        body.deformation(), body.damage()
    driver = ctypes.CDLL("libcuda.so.1")
    count = ctypes.c_size_t()
    raw = ctypes.c_void_p(graph.raw_cuda_graph())
    assert driver.cuGraphGetNodes(raw, None, ctypes.byref(count)) == 0
    nodes = (ctypes.c_void_p * count.value)()
    assert driver.cuGraphGetNodes(raw, nodes, ctypes.byref(count)) == 0
    kinds = []
    for node in nodes:
        kind = ctypes.c_int()
        assert driver.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        kinds.append(kind.value)
    graph.instantiate()
    graph.replay()
    torch.cuda.synchronize()
    for got, expected in zip((body.F, body.bond, body.index), want):
        assert torch.equal(got, expected)
    assert kinds and set(kinds) == {0}  # CU_GRAPH_NODE_TYPE_KERNEL


def test_records_must_lie_on_a_32_byte_boundary():
    body = Step(64)
    records = torch.empty(8 * body.n + 4, dtype=torch.float64, device="cuda")
    for bad in (None, ctypes.c_void_p(records.data_ptr() + 8)):
        with pytest.raises(vpd.VpdError) as e:
            body.call("vpd_shape_tensor_inverse_packed", body.pos, body.vol, body.n, body.row_ptr, body.col, body.kinv, bad)
        assert e.value.status == 1


def test_idle_memory_is_bounded_when_a_call_returns():
    w = torch.zeros(vpd.MLP_WEIGHTS, dtype=torch.int16, device="cuda")
    b = torch.zeros(vpd.MLP_PARAMS - vpd.MLP_WEIGHTS, dtype=torch.float32, device="cuda")
    x = torch.randn((400_000, 16), dtype=torch.float32, device="cuda")
    first = vpd.mlp_gradients(w, b, x[:128], x[:128])
    before = free_bytes()
    second = vpd.mlp_gradients(w, b, x, x)  # 466 MB of partial gradients in all
    # (not free_bytes(): its synchronisation would give memory back too)
    assert before - torch.cuda.mem_get_info()[0] <= 256 << 20
    del first, second


def test_idle_memory_is_given_back_on_request_and_with_a_handle():
    from vpd.case import tensile_bar
    w = torch.zeros(vpd.MLP_WEIGHTS, dtype=torch.int16, device="cuda")
    b = torch.zeros(vpd.MLP_PARAMS - vpd.MLP_WEIGHTS, dtype=torch.float32, device="cuda")
    x = torch.randn((100_000, 16), dtype=torch.float32, device="cuda")
    vpd.mlp_gradients(w, b, x[:128], x[:128])
    vpd.Simulation(tensile_bar(1)).close()  # every kernel loaded
    vpd.release_workspace()
    before = free_bytes()
    for give_back, left in ((vpd.release_workspace, 0), (lambda: vpd.Simulation(tensile_bar(1)).close(), 32 << 20)):
        vpd.mlp_gradients(w, b, x, x)  # 117 MB of partial gradients
        assert before - free_bytes() > 100_000_000
        give_back()
        assert before - free_bytes() <= left


def test_gradients_in_parts_sum_in_the_same_order():
    """A batch beyond the rows whose partial gradients are held at once (7 x 148 blocks of 128 rows): the rows after them
    add to the sum of those before, block by block, so a zero output gradient leaves it as it was."""
    rows = 7 * 148 * 128
    g = torch.Generator(device="cuda").manual_seed(5)
    w = (0.1 * torch.randn(vpd.MLP_WEIGHTS, generator=g, device="cuda")).to(torch.bfloat16).view(torch.int16)
    b = 0.1 * torch.randn(vpd.MLP_PARAMS - vpd.MLP_WEIGHTS, generator=g, device="cuda")
    x, gout = (torch.randn((rows + 129, 16), generator=g, device="cuda") for _ in range(2))
    first, rest = vpd.mlp_gradients(w, b, x[:rows], gout[:rows]), vpd.mlp_gradients(w, b, x[rows:], gout[rows:])
    both = vpd.mlp_gradients(w, b, x, gout)
    # one float addition against another order of the last 129 rows' sum
    assert (both - (first + rest)).abs().max() <= 4 * 2.0 ** -23 * (first.abs() + rest.abs()).max()
    assert rest.abs().max() > 0
    gout[rows:] = 0.0
    assert torch.equal(vpd.mlp_gradients(w, b, x, gout), first)
