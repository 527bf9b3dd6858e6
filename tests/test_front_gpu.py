"""GPU: the native front end gives what the Python form of every method gives, raises the same errors,
and leaves anything but the plain case to it."""
import pytest
import torch

import autograph_b200 as ag

pytestmark = pytest.mark.gpu


@pytest.fixture
def plain(dev):
    """The device without output guards (with them every call takes the Python form)."""
    dev.set_guards(False)
    yield dev
    dev.set_guards(True)


def _calls(d, dtype):
    gen = torch.Generator(device=d.torch_device).manual_seed(1)
    r = lambda *s: torch.randn(s, generator=gen, device=d.torch_device).to(dtype)
    a, b, bias = r(40, 24), r(24, 33), r(33)
    x, w, cb, dy = r(3, 5, 12, 11), r(7, 5, 3, 3), r(7), r(3, 7, 6, 6)
    o = dict(padding=(1, 1), stride=(2, 2))
    z = r(3, 7, 12, 11)
    return [
        ("dot", (a, b), {}), ("dot", (b.T, a.T), {}), ("dot", (a[::2], b[:, ::3]), {}),
        ("gemm", (0.5, a, b, 2.0, r(40, 33)), {}),
        ("dense_forward", (a, b), dict(bias=bias, relu=True)), ("dense_forward", (a, b, None), {}),
        ("conv2_forward", (x, w), {}), ("conv2_forward", (x, w, cb), dict(relu=True, **o)),
        ("conv2_backward_input", (w, dy, (12, 11)), o), ("conv2_backward_weight", (x, dy, (3, 3)), o),
        ("conv2_backward_weight", (x, dy, (3, 3)), dict(beta=1.0, dw=w.clone(), **o)),
        ("max_pool2", (x,), {}), ("max_pool2", (x, (3, 2), (3, 2)), {}),
        ("max_pool2_backward_from_input", (x, r(3, 5, 6, 5)), {}),
        ("relu", (x,), {}), ("relu", (x.clone(), True), {}), ("relu", (x.transpose(0, 1),), {}),
        ("relu_backward", (z, r(3, 7, 12, 11)), {}), ("relu_backward", (a, r(40, 24)), dict(inplace=True)),
        ("bias_add", (r(3, 7, 12, 11), cb), {}), ("bias_grad", (z,), {}), ("bias_grad", (a,), dict(beta=1.0, out=r(24))),
    ]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_same_results_as_the_python_form(plain, dtype):
    for (name, args, kw), (_, args2, kw2) in zip(_calls(plain, dtype), _calls(plain, dtype)):
        got = getattr(plain, name)(*args, **kw)
        want = getattr(ag._PyDevice, name)(plain, *args2, **kw2)
        assert got.dtype == want.dtype and torch.equal(got, want), name
        for v, v2 in zip(list(args) + list(kw.values()), list(args2) + list(kw2.values())):
            if isinstance(v, torch.Tensor):
                assert torch.equal(v, v2), name   # in-place arguments too


def test_same_errors(plain):
    x = plain.empty((4, 5), torch.float32)
    bad = [("dot", (x, plain.empty((4, 3), torch.float32)), {}, "a_cols != b_rows"),
           ("dot", (x, plain.empty((5, 3), torch.bfloat16)), {}, "different types"),
           ("dot", (x.double(), x.double().T), {}, "unimplemented"),
           ("dense_forward", (x, x), {}, "a_cols"),
           ("conv2_forward", (plain.empty((1, 2, 4, 4), torch.float32), plain.empty((3, 2, 5, 5), torch.float32)), {}, "fit"),
           ("max_pool2", (plain.empty((1, 1, 2, 2), torch.float32), (3, 3)), {}, "does not fit")]
    for name, args, kw, text in bad:
        with pytest.raises(ag.AgError, match=text):
            getattr(plain, name)(*args, **kw)
    with pytest.raises(TypeError):
        plain.dot(x)


def test_host_tensors_are_refused(plain):
    """One tensor in host memory, whichever argument: an error before anything is launched."""
    for name, args, kw in _calls(plain, torch.float32):
        for key in [*range(len(args)), *kw]:
            a, w = list(args), dict(kw)
            at = a if isinstance(key, int) else w
            if not isinstance(at[key], torch.Tensor):
                continue
            at[key] = at[key].cpu()
            with pytest.raises(ag.AgError, match="must be in device memory"):
                getattr(plain, name)(*a, **w)


def test_page_locked_operands_are_read(plain):
    a, b = torch.randn(40, 24).pin_memory(), torch.randn(24, 33).pin_memory()
    assert torch.equal(plain.dense_forward(a, b), plain.dense_forward(a.cuda(), b.cuda()))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_a_default_device_changes_nothing(plain, dtype):
    """Outputs come on the device's GPU, whatever tensors are made on by default."""
    for name, args, kw in _calls(plain, dtype):
        if kw.get("inplace") or "out" in kw or "dw" in kw or name in ("gemm", "bias_add") or any(a is True for a in args):
            continue   # called twice below
        want = getattr(plain, name)(*args, **kw)
        with torch.device("cpu"):
            got = getattr(plain, name)(*args, **kw)
        assert got.device == want.device and torch.equal(got, want), name


def _strided(t):
    if t.dim() == 1:
        return torch.stack((t, t + 1), 1)[:, 0]
    back = tuple(reversed(range(t.dim())))
    return t.permute(back).contiguous().permute(back)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_strided_operands(plain, dtype):
    """Every operand strided at once, of equal sizes too: a copy freed early would be the next one's memory."""
    sq = lambda k: torch.randn((64, 64), generator=torch.Generator("cuda").manual_seed(k), device="cuda").to(dtype)
    calls = _calls(plain, dtype) + [("dense_forward", (sq(1), sq(2)), {}), ("dense_chain_forward", (sq(1), [sq(2), sq(3)]), {}),
                                    ("relu_backward", (sq(1), sq(2)), {})]
    for name, args, kw in calls:
        if name in ("gemm", "bias_add") or kw.get("inplace") or "out" in kw or "dw" in kw or any(a is True for a in args):
            continue
        as_strided = lambda v: _strided(v) if isinstance(v, torch.Tensor) else [_strided(t) for t in v] if isinstance(v, list) else v
        want = getattr(plain, name)(*args, **kw)
        got = getattr(plain, name)(*map(as_strided, args), **{k: as_strided(v) for k, v in kw.items()})
        assert torch.equal(got, want), name
    other = torch.cuda.Stream()
    a, b = sq(4), sq(5)
    want = plain.dense_forward(a, b)
    plain.wait()
    with torch.cuda.stream(other):
        got = [plain.dense_forward(_strided(a), _strided(b)) for _ in range(50)]
    other.synchronize()
    plain.wait()
    assert all(torch.equal(g, want) for g in got)


def test_another_current_stream_is_ordered(plain):
    """Inputs produced on another current stream: the call waits for that stream."""
    a = torch.zeros((512, 512), device=plain.torch_device)
    plain.wait()
    other = torch.cuda.Stream()
    with torch.cuda.stream(other):
        torch.cuda._sleep(2_000_000)
        a.fill_(1.0)
        c = plain.dot(a, a)
    plain.wait()
    assert bool((c == 512).all())


def test_model_calls(plain):
    m = ag.Model(plain, seed=3)
    x = torch.rand((5, 1, 28, 28))
    out = torch.empty((5, 10))
    assert m.infer(x, out) is out
    assert torch.equal(m.infer(x), out)
    assert torch.equal(m.forward_device(x.cuda(), torch.empty((5, 10), device="cuda")).cpu(), out)
    with pytest.raises(ag.AgError, match="expected"):
        m.infer(x.double(), out)
    with pytest.raises(ag.AgError, match="expected shape"):
        m.infer(x, torch.empty((4, 10)))
    with pytest.raises(ag.AgError, match="device memory"):
        m.forward_device(x)
    t = torch.zeros(5, dtype=torch.uint8)
    loss, ptr, n = m.train_forward_backward(x.cuda(), t.cuda())
    assert loss > 0 and ptr and n >= sum(m.parameter_lens)
    before = m.get_parameter(0)
    m.apply_update(0.1)
    assert (m.get_parameter(0) != before).any()
    assert abs(m.train_step(x, t, lr=0.0) - m.train_step(x, t, 0.0)) < 1e-6
    with pytest.raises(ag.AgError):
        m.train_step(x, t[:3], 0.1)
    m.close()
