"""GPU: two devices of one GPU, each driven by a thread of its own."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _in_threads(calls, times):
    """Runs every call `times` times in a thread of its own, all at once; returns what they raised."""
    raised, start = [], threading.Barrier(len(calls))

    def work(call):
        start.wait()
        try:
            for _ in range(times):
                call()
        except Exception as e:   # noqa: BLE001 - reported by the caller
            raised.append(e)

    threads = [threading.Thread(target=work, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return raised


def test_pools_to_nchw_of_several_sizes(dev, monkeypatch):
    """The pools that write NCHW stage 64 channels of a plane in shared memory, here 400 and 961 windows: more than a kernel
    has without an attribute, which the two devices share.  With the attribute set to each call's size one of these
    threads lowered it under the other every few hundred calls."""
    import autograph_b200 as ag
    monkeypatch.setenv("AG_GRAPH", "0")   # every pass launches its kernels itself
    calls, devices = [], []
    for pooled in (20, 31):
        d = ag.Device(0)
        model = ag.Model(d, [("conv", 16, 64, (1, 1), False), ("relu",), ("pool", (2, 2)), ("flatten",),
                             ("dense", 64 * pooled ** 2, 1, False)], torch.bfloat16, seed=3)
        x = torch.rand((300, 16, 2 * pooled, 2 * pooled), device=d.torch_device).to(torch.bfloat16)
        out = torch.empty((300, 1), dtype=torch.bfloat16, device=d.torch_device)
        torch.cuda.synchronize()
        model.forward_device(x, out)
        devices.append(d)
        calls.append(lambda model=model, x=x, out=out: model.forward_device(x, out))
    raised = _in_threads(calls, 3000)
    for d in devices:
        d.wait()
    assert not raised, raised


def test_convolutions_on_pixel_rows_of_several_sizes(dev):
    """The first calls of the kernels on pixel rows, 16 channels into 32, in two threads: boxes of 224 rows and of 160, filters
    of 27 KB and of 9 KB, whose shared memory differs."""
    import autograph_b200 as ag
    cases = []
    for hw, f in ((32, (3, 3)), (24, (1, 3))):
        x = torch.randn((64, 16, hw, hw), device=dev.torch_device)
        w = torch.randn((32, 16, *f), device=dev.torch_device)
        dy = torch.randn((64, 32, hw, hw), device=dev.torch_device)
        cases.append((ag.Device(0), x, w, dy, dict(padding=(f[0] // 2, f[1] // 2))))
    torch.cuda.synchronize()

    def call(d, x, w, dy, opt):
        d.conv2_forward(x, w, **opt)
        d.conv2_backward_weight(x, dy, tuple(w.shape[2:]), **opt)
        d.conv2_backward_input(w, dy, tuple(x.shape[2:]), **opt)

    raised = _in_threads([lambda c=c: call(*c) for c in cases], 200)
    for d, *_ in cases:
        d.wait()
    assert not raised, raised
