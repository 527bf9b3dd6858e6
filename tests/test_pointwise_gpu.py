"""GPU: relu, max-pool, scaled_add, bias and SGD kernels; bit-exact against the oracle."""
import numpy as np
import pytest
import torch

import oracle
from conftest import cycle

pytestmark = pytest.mark.gpu
DTYPES = [torch.float32, torch.bfloat16]


def _prep(a, dtype):
    return oracle.round_bf16(a) if dtype == torch.bfloat16 else a.astype(np.float32)


def _np(t):
    return t.float().cpu().numpy()


@pytest.mark.parametrize("dtype", DTYPES)
def test_relu_golden_and_random(dev, golden, dtype):
    for c in golden.meta["relu"]:
        shape = tuple(c["shape"])
        n = shape[0] * shape[1]
        x = dev.tensor(cycle(-10, 10, n).reshape(shape), dtype)
        assert np.array_equal(_np(dev.relu(x)), golden[c["name"] + "_y"])
        xb = dev.tensor(cycle(-1, 1, n).reshape(shape), dtype)
        dy = np.arange(n, dtype=np.float32).reshape(shape)
        if dtype == torch.bfloat16:
            dy = oracle.round_bf16(dy)
        want = np.where(cycle(-1, 1, n).reshape(shape) >= 0, dy, 0)
        dyd = dev.tensor(dy, dtype)
        assert np.array_equal(_np(dev.relu_backward(xb, dyd)), want)          # relu_backward
        assert np.array_equal(_np(dev.relu_backward(xb, dyd, inplace=True)), want)  # _mut
    rng = np.random.default_rng(1)
    for n in [1, 7, 1000, 100003]:
        x = _prep(rng.standard_normal(n), dtype)
        x[::5] = 0.0
        x[1::7] = -0.0
        dy = _prep(rng.standard_normal(n), dtype)
        xd = dev.tensor(x, dtype)
        y = dev.relu(xd)
        assert np.array_equal(_np(y).view(np.uint32), oracle.relu(x).view(np.uint32))
        dx = dev.relu_backward(xd, dev.tensor(dy, dtype))
        assert np.array_equal(_np(dx).view(np.uint32), oracle.relu_backward(x, dy).view(np.uint32))
        y2 = dev.relu(xd.clone(), inplace=True)
        assert torch.equal(y, y2)
    # NaN -> 0, like x >= 0 ? x : 0
    y = dev.relu(dev.tensor(np.array([np.nan, -np.inf, np.inf], np.float32), dtype))
    assert _np(y).tolist() == [0.0, 0.0, float("inf")]


@pytest.mark.parametrize("dtype", DTYPES)
def test_max_pool2_golden(dev, golden, dtype):
    for c in golden.meta["pool"]:
        shape = tuple(c["shape"])
        x = cycle(0, 10, int(np.prod(shape))).reshape(shape)
        xd = dev.tensor(x, dtype)
        y = dev.max_pool2(xd)
        assert np.array_equal(_np(y), golden[c["name"] + "_y"])
        dy = np.arange(y.numel(), dtype=np.float32).reshape(tuple(y.shape))
        want = golden[c["name"] + "_dx"]
        if dtype == torch.bfloat16:
            dy = oracle.round_bf16(dy)
            want = oracle.max_pool2_backward(x, dy)
        assert np.array_equal(_np(dev.max_pool2_backward(xd, dev.tensor(dy, dtype))), want)
        assert np.array_equal(_np(dev.max_pool2_backward_from_input(xd, dev.tensor(dy, dtype))), want)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("case", [((3, 6, 24, 24), (2, 2), None), ((2, 16, 8, 8), (2, 2), None),
                                  ((2, 4, 62, 62), (2, 2), None), ((2, 3, 29, 29), (2, 2), None),
                                  ((2, 2, 13, 17), (3, 2), None), ((1, 2, 20, 21), (2, 3), (3, 4)),
                                  # a last row no window covers (keeps x), vector / staged paths
                                  ((2, 3, 9, 16), (2, 2), None), ((2, 3, 7, 10), (2, 2), None),
                                  ((2, 3, 10, 10), (2, 2), None), ((700, 5, 12, 14), (2, 2), None)])
def test_max_pool2_random(dev, dtype, case):
    shape, size, strides = case
    rng = np.random.default_rng(2)
    x = _prep(rng.integers(-4, 5, shape).astype(np.float32) * 0.5, dtype)  # many ties
    xd = dev.tensor(x, dtype)
    y = dev.max_pool2(xd, size, strides)
    want = oracle.max_pool2(x, size, strides)
    assert np.array_equal(_np(y), want)
    dy = _prep(rng.standard_normal(want.shape), dtype)
    dx = dev.max_pool2_backward(xd, dev.tensor(dy, dtype), size, strides)
    assert np.array_equal(_np(dx), oracle.max_pool2_backward(x, dy, size, strides))
    dx = dev.max_pool2_backward_from_input(xd, dev.tensor(dy, dtype), size, strides)
    assert np.array_equal(_np(dx), oracle.max_pool2_backward(x, dy, size, strides))
    # an input that does not start on a 16-byte boundary (the staged copy keeps the source phase)
    flat = dev.empty((x.size + 3,), dtype)
    flat[3:].copy_(xd.reshape(-1))
    dx = dev.max_pool2_backward_from_input(flat[3:].reshape(xd.shape), dev.tensor(dy, dtype), size, strides)
    assert np.array_equal(_np(dx), oracle.max_pool2_backward(x, dy, size, strides))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("shape", [(100, 6, 24, 24), (100, 16, 8, 8), (3, 5, 2, 2), (2, 3, 6, 10),
                                   (0, 4, 8, 8)])
def test_relu_max_pool2_equals_the_two_layers(dev, dtype, shape):
    """One pass gives what Relu then MaxPool2 give, forward and backward (ties, zeros, -0.0)."""
    rng = np.random.default_rng(21)
    x = _prep(rng.integers(-3, 4, shape).astype(np.float32) * 0.5, dtype)
    if x.size:
        x.reshape(-1)[::7] = -0.0
    xd = dev.tensor(x, dtype)
    y = dev.relu_max_pool2(xd)
    want = oracle.max_pool2(oracle.relu(x)) if x.size else np.zeros(y.shape, np.float32)
    assert np.array_equal(_np(y), want)
    dy = _prep(rng.standard_normal(want.shape), dtype)
    dx = dev.relu_max_pool2_backward(xd, dev.tensor(dy, dtype))
    if x.size:
        want_dx = oracle.relu_backward(x, oracle.max_pool2_backward(oracle.relu(x), dy))
        assert np.array_equal(_np(dx), want_dx)
        # and bit for bit what the separate kernels give
        r = dev.relu(xd)
        sep = dev.relu_backward(xd, dev.max_pool2_backward_from_input(r, dev.tensor(dy, dtype)))
        assert np.array_equal(_np(dx).view(np.uint32), _np(sep).view(np.uint32))


def test_relu_max_pool2_rejects_odd_planes(dev):
    import autograph_b200 as ag
    with pytest.raises(ag.AgError, match="even"):
        dev.relu_max_pool2(dev.empty((1, 1, 5, 4), torch.float32))


def test_max_pool2_errors(dev):
    import autograph_b200 as ag
    with pytest.raises(ag.AgError):
        dev.max_pool2(dev.empty((1, 1, 1, 4), torch.float32))
    x = dev.empty((1, 1, 6, 6), torch.float32)
    with pytest.raises(ag.AgError, match="non-overlapping"):
        dev.max_pool2_backward(x, dev.empty((1, 1, 5, 5), torch.float32), (2, 2), (1, 1))


@pytest.mark.parametrize("dtype", DTYPES)
def test_scaled_add(dev, golden, dtype):
    for c in golden.meta["axpy"]:  # scaled_add_<T> (tests/integration_tests.rs:425-452)
        n = c["n"]
        y = dev.tensor(cycle(11, 20, n), dtype)
        dev.scaled_add(y, 2.0, dev.tensor(cycle(1, 10, n), dtype))
        assert np.array_equal(_np(y), golden[c["name"]])
    rng = np.random.default_rng(3)
    for n in [5, 4096, 46920, 1000001]:
        x = _prep(rng.standard_normal(n), dtype)
        y = _prep(rng.standard_normal(n), dtype)
        yd = dev.tensor(y, dtype)
        dev.scaled_add(yd, -0.01, dev.tensor(x, dtype))
        want = oracle.scaled_add(oracle.round_bf16(np.float32([-0.01]))[0]
                                 if dtype == torch.bfloat16 else -0.01, x, y,
                                 bf16=dtype == torch.bfloat16)
        assert np.array_equal(_np(yd), want)
    # unaligned views take the scalar path
    base = dev.tensor(np.zeros(1003, np.float32))
    src = dev.tensor(np.arange(1003, dtype=np.float32))
    dev.scaled_add(base[1:1002], 3.0, src[2:1003])
    assert np.array_equal(_np(base)[1:1002], 3.0 * np.arange(2, 1003, dtype=np.float32))
    assert _np(base)[0] == 0 and _np(base)[1002] == 0


@pytest.mark.parametrize("dtype", DTYPES)
def test_bias_add_and_grad(dev, golden, dtype):
    for c in golden.meta["colsum"]:
        x = cycle(1, 16, c["rows"] * c["cols"] * c["inner"]).reshape(c["rows"], c["cols"], c["inner"])
        got = _np(dev.bias_grad(dev.tensor(x, dtype)))
        want = golden[c["name"]]
        assert np.array_equal(got, oracle.round_bf16(want) if dtype == torch.bfloat16 else want)
    rng = np.random.default_rng(4)
    for shape in [(100, 10), (7, 6, 24, 24), (1000, 84)]:
        y = _prep(rng.standard_normal(shape), dtype)
        b = _prep(rng.standard_normal(shape[1]), dtype)
        yd = dev.tensor(y, dtype)
        dev.bias_add(yd, dev.tensor(b, dtype))
        assert np.array_equal(_np(yd), oracle.bias_add(y, b, bf16=dtype == torch.bfloat16))
        g = _np(dev.bias_grad(dev.tensor(y, dtype)))
        ref = y.astype(np.float64).sum(axis=tuple(i for i in range(len(shape)) if i != 1))
        tol = 1e-2 if dtype == torch.bfloat16 else 1e-5
        assert np.abs(g - ref).max() <= tol * max(np.abs(ref).max(), 1.0)
    acc = dev.tensor(np.ones(10, np.float32))
    dev.bias_grad(dev.tensor(np.ones((100, 10), np.float32)), beta=2.0, out=acc)
    assert np.array_equal(_np(acc), np.full(10, 102.0, np.float32))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("shape,offset", [((1, 1, 3, 3), 0), ((2, 3, 2, 5), 1), ((2, 3, 5, 2), 0), ((5, 7, 11, 6), 1),
                                          ((1, 2, 1301, 2777), 0),   # more windows than one round of the grid holds
                                          ((1, 1, 1902, 2782), 2)])
def test_windows_of_two_by_two(dev, dtype, shape, offset):
    """Odd planes, starts off 16 bytes, in and out of place: exact, and the cells no window covers are kept."""
    rng = np.random.default_rng(31)
    x = _prep(rng.integers(-4, 5, shape).astype(np.float32) * 0.5, dtype)
    flat = dev.empty((x.size + offset,), dtype)
    flat[offset:].copy_(dev.tensor(x, dtype).reshape(-1))
    xd = flat[offset:].reshape(shape)
    want = oracle.max_pool2(x, (2, 2), None)
    assert np.array_equal(_np(dev.max_pool2(xd)), want)
    dy = _prep(rng.standard_normal(want.shape), dtype)
    want = oracle.max_pool2_backward(x, dy, (2, 2), None)
    assert np.array_equal(_np(dev.max_pool2_backward_from_input(xd, dev.tensor(dy, dtype))), want)
    assert np.array_equal(_np(dev.max_pool2_backward(xd, dev.tensor(dy, dtype))), want)


def _pool_2x2(x, dy=None, relu=False):
    """Torch, window by window in order: the first maximum wins, a NaN never after the first cell.  Output, or the
    gradient with the cells no window covers kept."""
    oh, ow = x.shape[2] // 2, x.shape[3] // 2
    cells = [x[:, :, i:2 * oh:2, j:2 * ow:2] for i in (0, 1) for j in (0, 1)]
    gates = [c >= 0 for c in cells]
    if relu:
        cells = [torch.where(g, c, torch.zeros_like(c)) for c, g in zip(cells, gates)]
    best, at = cells[0].clone(), torch.zeros(cells[0].shape, dtype=torch.uint8, device=x.device)
    for k in (1, 2, 3):
        at[cells[k] > best] = k
        best = torch.where(cells[k] > best, cells[k], best)
    if dy is None:
        return best
    dx = x.clone()
    for k, gate in enumerate(gates):
        won = (at == k) & gate if relu else at == k
        dx[:, :, k // 2:2 * oh:2, k % 2:2 * ow:2] = torch.where(won, dy + 0, torch.zeros_like(dy))
    return dx


def _same(a, b):
    """Equal, NaNs and signs of zeros included."""
    return bool((((a == b) & (torch.signbit(a) == torch.signbit(b))) | (a.isnan() & b.isnan())).all())


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("shape", [(9, 16, 14, 14), (9, 16, 13, 13), (5, 3, 37, 62), (2, 3, 301, 203),
                                   (300, 64, 7, 7), (195, 64, 7, 7), (700, 64, 9, 9), (700, 64, 9, 11), (2000, 64, 3, 3),
                                   (600, 64, 3, 3)])
def test_windows_of_two_by_two_with_special_values(dev, dtype, shape):
    """NaN, infinities, both zeros and the largest values, at the sizes where a rule chooses the kernel."""
    gen = torch.Generator(device=dev.torch_device).manual_seed(sum(shape))
    big = torch.finfo(dtype).max
    pick = torch.tensor([float("nan"), float("inf"), -float("inf"), 0.0, -0.0, big, -big, 1.0], dtype=dtype, device=dev.torch_device)

    def values(s):
        t = torch.randn(s, generator=gen, device=dev.torch_device).to(dtype)
        special = pick[torch.randint(0, 8, s, generator=gen, device=dev.torch_device)]
        return torch.where(torch.rand(s, generator=gen, device=dev.torch_device) < 0.4, special, t)

    x, dy = values(shape), values((*shape[:2], shape[2] // 2, shape[3] // 2))
    assert _same(dev.max_pool2(x), _pool_2x2(x))
    want = _pool_2x2(x, dy)
    assert _same(dev.max_pool2_backward_from_input(x, dy), want)
    assert _same(dev.max_pool2_backward(x, dy), want)
    if shape[2] % 2 == 0 and shape[3] % 2 == 0:
        assert _same(dev.relu_max_pool2(x), _pool_2x2(x, relu=True))
        assert _same(dev.relu_max_pool2_backward(x, dy), _pool_2x2(x, dy, relu=True))


@pytest.mark.parametrize("shape", [(70001, 1, 250, 251), (1, 1, 65537, 65539), (1, 1, 65538, 65540)])
def test_windows_of_two_by_two_beyond_2_32_cells(dev, shape):
    """Sets of planes, and single planes, that take several launches."""
    dev.set_guards(False)   # their checks would need another 20 GB
    assert shape[0] * shape[2] * shape[3] > 2 ** 32
    x = torch.empty(shape, dtype=torch.bfloat16, device=dev.torch_device).normal_()
    y = dev.max_pool2(x)
    dx = dev.max_pool2_backward_from_input(x, y)
    for part in range(16):   # by planes, or by pairs of rows
        if shape[0] > 1:
            at = slice(part * shape[0] // 16, (part + 1) * shape[0] // 16)
            xs, ys, dxs = x[at], y[at], dx[at]
        else:
            r0, r1 = (y.shape[2] * p // 16 for p in (part, part + 1))
            rows = slice(2 * r0, 2 * r1 if part < 15 else shape[2])
            xs, ys, dxs = x[:, :, rows], y[:, :, r0:r1], dx[:, :, rows]
        assert torch.equal(ys, _pool_2x2(xs)) and torch.equal(dxs, _pool_2x2(xs, ys))
    del x, y, dx, xs, ys, dxs
    torch.cuda.empty_cache()
    dev.set_guards(True)


def test_gradient_of_two_by_two_windows_keeps_up(dev):
    """16384 planes of 62 x 62 bf16 take less than 1.7 times as long as a copy that moves as many bytes (1.35 with a
    window per thread, 2.0 with four)."""
    dev.set_guards(False)
    x = torch.randn((256, 64, 62, 62), device=dev.torch_device).bfloat16()
    dy = torch.randn((256, 64, 31, 31), device=dev.torch_device).bfloat16()
    n = x.numel() + dy.numel() // 2
    a, b = torch.empty(n, dtype=x.dtype, device=dev.torch_device), torch.empty(n, dtype=x.dtype, device=dev.torch_device)

    def us(f):
        best = float("inf")
        for _ in range(10):
            t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda._sleep(500_000)   # the launches queue up behind it
            t0.record(dev.stream)
            for _ in range(10):
                f()
            t1.record(dev.stream)
            t1.synchronize()
            best = min(best, t0.elapsed_time(t1) * 100)
        return best

    assert us(lambda: dev.max_pool2_backward_from_input(x, dy)) < 1.7 * us(lambda: b.copy_(a))
    dev.set_guards(True)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("shape,offset", [((1, 1, 2), 0), ((3, 2, 2, 2), 1), ((2, 3, 7), 0), ((9, 5, 511), 1), ((4, 3, 512), 0),
                                          ((2, 2, 1023), 1), ((70, 33, 1025), 0), ((2, 1500, 6), 0), ((1, 1, 70001), 3)])
def test_bias_grad_of_planes(dev, dtype, shape, offset):
    """Planes that start and end anywhere in a 16-byte vector, one unit of loads or several, one launch or two.
    An f32 sum of n values of size one, added in at most n / 32 + 32 steps per lane and tree, is off by less than
    (n / 32 + 32) * 2^-24 * sum |x|."""
    rng = np.random.default_rng(32)
    x = _prep(rng.standard_normal(shape), dtype)
    flat = dev.empty((x.size + offset,), dtype)
    flat[offset:].copy_(dev.tensor(x, dtype).reshape(-1))
    axes = tuple(i for i in range(len(shape)) if i != 1)
    got = _np(dev.bias_grad(flat[offset:].reshape(shape)))
    want, size = x.astype(np.float64).sum(axis=axes), np.abs(x).sum(axis=axes)
    bound = (x.size / shape[1] / 32 + 32) * 2.0 ** -24 * size
    if dtype == torch.bfloat16:
        bound += 2.0 ** -8 * (np.abs(want) + bound)
    assert (np.abs(got - want) <= bound).all()


@pytest.mark.parametrize("dtype", DTYPES)
def test_bias_grad_of_planes_accumulates(dev, dtype):
    """beta and a given output, where the last chunk of a channel finishes it and where a second launch does (1024
    channels and more), with other numbers of chunks in between: a call leaves every counter as it found it.  The bound
    is that of the sums above, and two roundings of f32 for beta."""
    gen = torch.Generator(device=dev.torch_device).manual_seed(33)
    rnd = lambda *s: torch.randn(s, generator=gen, device=dev.torch_device).to(dtype)
    cases = [(rnd(*s), rnd(s[1]), beta) for s, beta in
             (((9, 5, 511), 1.0), ((70, 33, 1025), 0.5), ((2, 1500, 6), -2.0), ((1, 1, 70001), 1.0), ((300, 1023, 9), 0.25),
              ((40, 1024, 33), 1.0), ((5, 7, 2), 1.0))]
    first = []
    for again in range(3):
        for i, (x, y, beta) in enumerate(cases):
            out = y.clone()
            assert dev.bias_grad(x, beta, out) is out
            if again == 0:
                first.append(out)
            assert torch.equal(out, first[i])
    for (x, y, beta), got in zip(cases, first):
        want = x.double().sum(dim=(0, 2)) + beta * y.double()
        size = x.double().abs().sum(dim=(0, 2)) + abs(beta) * y.double().abs()
        bound = (x.numel() / x.shape[1] / 32 + 34) * 2.0 ** -24 * size
        if dtype == torch.bfloat16:
            bound += 2.0 ** -8 * (want.abs() + bound)
        assert ((got.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("dtype", DTYPES)
def test_sgd(dev, dtype):
    rng = np.random.default_rng(5)
    n = 46920
    bf = dtype == torch.bfloat16
    w, g, v = (_prep(rng.standard_normal(n) * s, dtype) for s in (0.1, 0.01, 0.001))
    wd = dev.tensor(w, dtype)
    dev.sgd_update(wd, dev.tensor(g, dtype), 0.01)
    assert np.array_equal(_np(wd), oracle.sgd_update(w, g, 0.01, bf16=bf))
    wd, vd = dev.tensor(w, dtype), dev.tensor(v, dtype)
    dev.sgd_update_momentum(wd, dev.tensor(g, dtype), vd, 0.01, 0.01)
    w2, v2 = oracle.sgd_update_momentum(w, g, v, 0.01, 0.01, bf16=bf)
    assert np.array_equal(_np(wd), w2) and np.array_equal(_np(vd), v2)
