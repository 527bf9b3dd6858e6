"""Kernels that start before their predecessor in the stream has ended."""
import re
from pathlib import Path

import pytest
import torch

CSRC = Path(__file__).resolve().parent.parent / "autograph_b200" / "csrc"


def _kernels():
    for path in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        for body in re.split(r"\b__global__\b", path.read_text())[1:]:
            body = re.sub(r"//[^\n]*", "", body.split("\n}\n")[0])
            yield path.name, re.search(r"(\w+)\(", re.sub(r"__launch_bounds__\([^)]*\)", "", body)).group(1), body


def test_tensor_memory_comes_before_dependents():
    """A dependent that came first could hold columns that this kernel still waits for: every kernel with tensor
    memory allocates it, and meets at a barrier, before one of its threads lets dependents launch."""
    seen = 0
    for file, name, body in _kernels():
        trigger = re.search(r"let_dependents_launch\(|griddepcontrol\.launch_dependents", body)
        alloc = max(body.find("tmem_alloc("), body.rfind("tmem_alloc2("))
        if trigger is None or alloc < 0:
            continue
        seen += 1
        assert alloc < trigger.start(), f"{file}: {name} lets dependents launch before it allocates tensor memory"
        assert "__syncthreads()" in body[alloc:trigger.start()], f"{file}: {name}: no barrier between the two"
    assert seen >= 9


def test_pairs_meet_before_they_allocate():
    """Tensor memory of a pair of CTAs is allocated by both: a barrier of the cluster comes before the first allocation,
    with no barrier of one CTA alone between the two."""
    seen = 0
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for body in re.split(r"\b__global__\b", text)[1:]:
            alloc = body.split("\n}\n")[0].find("tmem_alloc2(")
            if alloc < 0:
                continue
            seen += 1
            barriers = re.findall(r"cluster_sync\(\)|__syncthreads\(\)", body[:alloc])
            assert barriers and barriers[-1] == "cluster_sync()", path.name
    assert seen == 2


@pytest.fixture
def plain(dev):
    """The device without output guards, whose fills would come between the kernels."""
    dev.set_guards(False)
    yield dev
    dev.set_guards(True)


def _stage(dev, x, w, dw_filter, step):
    """Forward and backward of a convolution stage and two dense layers: every kind of dependent kernel in a row."""
    out = []
    def op(name, *args, **kw):
        out.append(getattr(dev, name)(*args, **kw))
        step()
        return out[-1]
    pad = dict(padding=(1, 1))
    y = op("conv2_forward", x, w, relu=True, **pad)
    p = op("max_pool2", y)
    g = op("max_pool2_backward_from_input", y, p)
    g = op("relu_backward", y, g)
    op("bias_grad", g)
    op("conv2_backward_weight", x, g, dw_filter, **pad)
    op("conv2_backward_input", w, g, tuple(x.shape[2:]), **pad)
    flat = p.reshape(p.shape[0], -1)
    d = op("dense_forward", flat[:, :400].contiguous(), flat[:1, :4000].reshape(400, 10).contiguous())
    op("dot", flat.t(), d)
    op("dot", flat, flat.t())
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("bs,ic,oc,hw", [(3, 16, 40, 21), (20, 64, 96, 30), (70, 3, 32, 25)])
def test_operators_in_a_row_and_replayed(plain, dtype, bs, ic, oc, hw):
    """The bits of calls that are each waited for, from calls that are not and from a graph of them, twice over inputs
    that change."""
    dev = plain
    gen = torch.Generator(device=dev.torch_device).manual_seed(hw)
    rnd = lambda *s: torch.randn(s, generator=gen, device=dev.torch_device).mul_(0.1).to(dtype)
    x, w = rnd(bs, ic, hw, hw), rnd(oc, ic, 3, 3)
    _stage(dev, x, w, (3, 3), dev.wait)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=dev.stream):
        replayed = _stage(dev, x, w, (3, 3), lambda: None)
    for _ in range(2):
        x.copy_(rnd(bs, ic, hw, hw))
        want = _stage(dev, x, w, (3, 3), dev.wait)
        for _ in range(3):
            for a, b in zip(_stage(dev, x, w, (3, 3), lambda: None), want):
                assert torch.equal(a, b)
            graph.replay()
            graph.replay()
            for a, b in zip(replayed, want):
                assert torch.equal(a, b)
    del graph


def _replay_us(dev, calls, n=20):
    for f in calls:
        f()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=dev.stream):
        for _ in range(n):
            for f in calls:
                f()
    best = float("inf")
    for _ in range(20):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(dev.stream)
        graph.replay()
        b.record(dev.stream)
        b.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3 / n)
    del graph
    return best


@pytest.mark.gpu
@pytest.mark.parametrize("call", ["product", "narrow", "convolution"])
def test_early_launches_cost_nothing(plain, call):
    """A kernel that follows itself at once is no slower than one that a launch of torch's, which waits for all of
    it, comes between: dependents that crowd on the first free SMs made these 13.0, 34.8 and 24.2 us of 8.3, 21.6
    and 14.9, and the launch between takes one or two."""
    dev = plain
    rnd = lambda *s, dt=torch.float32: torch.randn(s, device=dev.torch_device).to(dt)
    if call == "product":
        a, b = rnd(256, 256), rnd(256, 256)
        f = lambda: dev.dot(a, b)
    elif call == "narrow":
        a, b = rnd(16384, 512), rnd(512, 10)
        f = lambda: dev.dense_forward(a, b)
    else:
        x, w = rnd(16, 64, 31, 31, dt=torch.bfloat16), rnd(128, 64, 3, 3, dt=torch.bfloat16)
        f = lambda: dev.conv2_forward(x, w)
    one = torch.zeros(1, device=dev.torch_device)
    assert _replay_us(dev, [f]) <= _replay_us(dev, [f, lambda: one.add_(1)])
