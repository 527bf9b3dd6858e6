"""GPU: convolutions whose index arithmetic is near the ends of 32 bits, and scratch that is bounded or not to be
had."""
import pytest
import torch
import torch.nn.functional as F

import autograph_b200 as ag

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_weight_gradient_of_one_long_row(dev, dtype):
    """A row of 2^25 pixels: the taps that meet it lie two rows into the padding, at offsets of 2^26."""
    n, oc = 2 ** 25, 6
    gen = torch.Generator(device=dev.torch_device).manual_seed(1)
    x = torch.randint(-2, 3, (1, 1, 1, n), generator=gen, device=dev.torch_device).to(dtype)
    dy = (torch.rand((1, oc, 1, n - 4), generator=gen, device=dev.torch_device) < 1e-4).to(dtype)
    dw = dev.conv2_backward_weight(x, dy, (5, 5), padding=(2, 0))
    want = torch.zeros((oc, 1, 5, 5), dtype=torch.float64, device=dev.torch_device)
    for j in range(5):
        want[:, 0, 2, j] = dy[0, :, 0].double() @ x[0, 0, 0, j:j + n - 4].double()
    # at most 2^25 * 1e-4 * 2 in a sum: exact in f32
    assert torch.equal(dw, want.to(dtype))
    dev.wait()


def test_filters_beyond_2_31_elements(dev):
    """A filter bank of 2.4e9 values: forward and both gradients."""
    oc, ic = 65536, 4096
    gen = torch.Generator(device=dev.torch_device).manual_seed(2)
    w = torch.empty((oc, ic, 3, 3), device=dev.torch_device)
    for i in range(0, oc, 4096):
        w[i:i + 4096] = torch.randint(-2, 3, (4096, ic, 3, 3), generator=gen, device=dev.torch_device)
    x = torch.randint(-2, 3, (1, ic, 3, 3), generator=gen, device=dev.torch_device).float()
    dy = torch.randint(-2, 3, (1, oc, 1, 1), generator=gen, device=dev.torch_device).float()
    flat, xv, dv = w.view(oc, -1), x.view(-1).double(), dy.view(-1).double()
    want = torch.cat([flat[i:i + 4096].double() @ xv for i in range(0, oc, 4096)])
    assert torch.equal(dev.conv2_forward(x, w).view(-1), want.float())
    want = sum(dv[i:i + 4096] @ flat[i:i + 4096].double() for i in range(0, oc, 4096))
    assert torch.equal(dev.conv2_backward_input(w, dy, (3, 3)).view(-1), want.float())
    del w, flat
    dw = dev.conv2_backward_weight(x, dy, (3, 3)).view(oc, -1)
    for i in (0, 1, oc // 2, 58254, 58255, oc - 1):   # 2^31 lies in row 58,254
        assert torch.equal(dw[i], x.view(-1) * dy[0, i, 0, 0])
    dev.wait()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_input_gradient_in_batch_slices(dev, dtype):
    """Sums per tap beyond 1 GiB are made for some of the images at a time, the last slice short."""
    bs, ic, oc, hw = 2271, 6, 64, 50   # 2157 images and 114
    gen = torch.Generator(device=dev.torch_device).manual_seed(3)
    ints = lambda *s: torch.randint(-2, 3, s, generator=gen, device=dev.torch_device).to(dtype)
    w, dy = ints(oc, ic, 3, 3), ints(bs, oc, hw - 2, hw - 2)
    dx = dev.conv2_backward_input(w, dy, (hw, hw))
    at = torch.tensor([0, 1000, 2156, 2157, 2270], device=dev.torch_device)
    want = F.conv_transpose2d(dy[at].double(), w.double())
    assert torch.equal(dx[at], want.to(dtype))   # sums of 576 products of at most 4 in absolute value
    assert torch.equal(dx[2200:], dev.conv2_backward_input(w, dy[2200:], (hw, hw)))
    dev.wait()


@pytest.mark.parametrize("channels", [(6, 128), (512, 512)])
def test_no_room_for_scratch(dev, channels):
    """With no memory for the sums per tap (few input channels) or for the copy of the filters the other forms
    run."""
    ic, oc = channels
    bs, hw = (512, 40) if ic == 6 else (64, 32)
    gen = torch.Generator(device=dev.torch_device).manual_seed(4)
    ints = lambda *s: torch.randint(-2, 3, s, generator=gen, device=dev.torch_device).float()
    x, w = ints(bs, ic, hw, hw), ints(oc, ic, 3, 3)
    dy = ints(bs, oc, hw - 2, hw - 2)

    def run(d):
        return d.conv2_forward(x, w), d.conv2_backward_input(w, dy, (hw, hw))

    want = run(dev)   # and the kernels are loaded
    dev.wait()
    fresh = ag.Device(0)
    torch.cuda.set_stream(fresh.stream)
    room = [torch.empty_like(t) for t in want]
    torch.cuda.synchronize()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (40 << 20 if ic == 6 else 6 << 20), dtype=torch.uint8,
                      device=dev.torch_device)
    del room   # the outputs' memory
    got = run(fresh)
    fresh.wait()
    del hog
    torch.cuda.empty_cache()
    assert all(torch.equal(g, t) for g, t in zip(got, want))
    fresh.close()
    torch.cuda.set_stream(dev.stream)
