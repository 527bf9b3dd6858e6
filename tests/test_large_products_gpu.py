"""GPU: products whose operands are too large to copy as a whole, devices without room for the copies, and
first calls under stream capture."""
import pytest
import torch

import autograph_b200 as ag

pytestmark = pytest.mark.gpu


def _check(c, a, b, rows, cols):
    """Rows and columns of c = a . b against float64; the bounds are those of test_gemm_tcx_gpu.py."""
    k = a.shape[1]
    for ai, bi, ci in ((a[rows], b, c[rows]), (a, b[:, cols], c[:, cols])):
        err = torch.zeros(ci.shape, dtype=torch.float64, device=ci.device)
        s, ref = err.clone(), err.clone()
        for k0 in range(0, k, 4096):   # the operands do not fit in float64
            x, y = ai[:, k0:k0 + 4096].double(), bi[k0:k0 + 4096].double()
            ref += x @ y
            s += x.abs() @ y.abs()
        bound = s * (5 * 2.0 ** -23 + 2.0 ** -24 + 2 * (k / 64 + 1) * 2.0 ** -24)
        if c.dtype == torch.bfloat16:
            bound = ref.abs() * 2.0 ** -8 + s * (66 * 2.0 ** -23 + 2 * (k / 1024 + 1) * 2.0 ** -24)
        assert ((ci.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("layout", ["nn", "tt"])
def test_operand_beyond_2_32_elements(dev, dtype, layout):
    m, k, n = 70001, 65537, 131
    gen = torch.Generator(device=dev.torch_device).manual_seed(1)

    def operand(r, c, l):
        shape = (r, c) if l == "n" else (c, r)
        t = torch.empty(shape, dtype=dtype, device=dev.torch_device).uniform_(-1, 1, generator=gen)
        return t if l == "n" else t.t()

    a, b = operand(m, k, layout[0]), operand(k, n, layout[1])
    assert a.numel() > 2 ** 32
    rows = torch.tensor([0, 1, m // 2 - 200, 35071, 35072, m - 130, m - 1], device=dev.torch_device)
    _check(dev.dot(a, b), a, b, rows, torch.tensor([], dtype=torch.long, device=dev.torch_device))
    dev.wait()


@pytest.fixture
def fresh():
    """A device object that has not allocated scratch yet."""
    d = ag.Device(0)
    yield d
    d.wait()
    d.close()
    torch.cuda.empty_cache()


def test_planes_are_bounded(dev, fresh):
    """30,000 x 16,400 x 30,001 in f32 has 3 GB of planes an operand: the product is cut and the scratch stays
    below 5.5 GB (4 GiB, the slices' sums and a quarter of it for growth)."""
    m, k, n = 30000, 16400, 30001
    a = torch.empty((m, k), device=fresh.torch_device).uniform_(-1, 1)
    b = torch.empty((k, n), device=fresh.torch_device).uniform_(-1, 1)
    c = torch.empty((m, n), device=fresh.torch_device)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    fresh.gemm(1.0, a, b, 0.0, c)
    fresh.wait()
    assert free - torch.cuda.mem_get_info()[0] < 5.5e9
    at = lambda size: torch.tensor([0, size // 2 - 240, size // 2 + 1, size - 1], device=fresh.torch_device)
    _check(c, a, b, at(m), at(n))
    torch.cuda.set_stream(dev.stream)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_no_room_for_planes(dev, fresh, dtype):
    """With no memory left for the copies the product runs on the engine that needs none."""
    m, k, n = 8191, 8193, 8189
    rnd = lambda r, c: (torch.rand((r, c), device=fresh.torch_device) * 2 - 1).to(dtype)
    a, b, c = rnd(m, k), rnd(k, n), torch.empty((m, n), dtype=dtype, device=fresh.torch_device)
    at = torch.tensor([0, 4000, 8188], device=fresh.torch_device)
    _check(c.copy_(a[:m, :1]), a[:, :1], torch.ones_like(b[:1]), at, at)   # room for the comparison's temporaries
    torch.cuda.synchronize()
    planes = 2 * m * k * (6 if dtype == torch.float32 else 2)
    hog = torch.empty(torch.cuda.mem_get_info()[0] - planes // 2, dtype=torch.uint8, device=fresh.torch_device)
    fresh.gemm(1.0, a, b, 0.0, c)
    fresh.wait()
    del hog
    torch.cuda.empty_cache()
    _check(c, a, b, at, at)
    torch.cuda.set_stream(dev.stream)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(1001, 1003, 777), (2049, 2051, 2047)])
def test_first_call_under_capture(dev, fresh, dtype, shape):
    """Scratch that a call needs may be allocated while the stream is being captured."""
    m, k, n = shape
    rnd = lambda r, c: (torch.rand((r, c), device=fresh.torch_device) * 2 - 1).to(dtype)
    a, b, c = rnd(m, k), rnd(k, n), torch.zeros((m, n), dtype=dtype, device=fresh.torch_device)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=fresh.stream):
        fresh.gemm(1.0, a, b, 0.0, c)
    at = torch.tensor([0, m // 2, n - 1], device=fresh.torch_device)
    for _ in range(2):
        c.zero_()
        graph.replay()
        torch.cuda.synchronize()
        _check(c, a, b, at, at)
        a.mul_(-0.5)
    del graph
    torch.cuda.set_stream(dev.stream)
