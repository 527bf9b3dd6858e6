"""GPU: convolutions whose tensors are split into channels-last bf16 planes ahead of the product (split_worth in
csrc/conv_tcx_impl.cuh; csrc/conv_halo_f32.cu, whose filters stay in shared memory): every direction against float64, and sums
that are not finite."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

# bs, ic, h, w, oc, filter, padding, stride, dilation: 3e8 multiply-adds in every direction
CASES = [
    (27, 40, 31, 28, 48, (3, 3), (1, 1), (1, 1), (1, 1)),    # channels in eights that are no sixteens
    (14, 45, 33, 30, 70, (3, 3), (0, 1), (1, 1), (1, 1)),    # channels and columns padded, 128-column tiles with a rest
    (33, 36, 29, 41, 33, (3, 5), (1, 2), (2, 1), (1, 1)),   # strides, columns beyond 32
    (36, 64, 27, 25, 20, (3, 3), (2, 2), (1, 1), (2, 2)),    # dilation: masks of taps, fewer columns than a tile
    (60, 32, 9, 9, 96, (5, 5), (2, 2), (1, 1), (1, 1)),     # few tiles: slices of k
    (6, 72, 50, 22, 130, (5, 3), (4, 0), (1, 2), (1, 1)),   # taps that leave the image on most sides
]
# The same for the engine with resident filters, f32, 8e7 multiply-adds forward and in the input gradient: pixel rows of 32, 64
# and 128 bytes both ways, 16, 32 and 64 columns with a rest, padding none, "same" and full, k groups with a rest
RESIDENT = [
    (64, 16, 32, 32, 32, (3, 3), (1, 1), (1, 1), (1, 1)),
    (90, 12, 29, 23, 20, (3, 3), (0, 0), (1, 1), (1, 1)),
    (30, 30, 41, 35, 62, (3, 3), (2, 2), (1, 1), (1, 1)),
    (40, 60, 30, 27, 15, (3, 3), (1, 0), (1, 1), (1, 1)),
    (70, 16, 26, 31, 6, (5, 5), (2, 2), (1, 1), (1, 1)),
    (150, 6, 33, 34, 33, (3, 3), (1, 1), (1, 1), (1, 1)),
    (50, 33, 25, 26, 13, (1, 5), (0, 2), (1, 1), (1, 1)),
    (1500, 20, 12, 11, 40, (2, 3), (1, 1), (1, 1), (1, 1)),   # several images per tile, tiles in every accumulator
    (1500, 20, 12, 11, 30, (2, 3), (1, 1), (1, 1), (1, 1)),
    (200, 40, 24, 23, 31, (3, 3), (1, 1), (1, 1), (1, 1)),    # weight gradients: two products a filter row, one accumulator of each
    (41, 3, 20, 21, 10, (3, 3), (0, 1), (1, 1), (1, 1)),
    (17, 33, 9, 57, 16, (1, 7), (0, 3), (1, 1), (1, 1)),      # four of them
    (9, 1, 40, 31, 5, (5, 4), (4, 3), (1, 1), (1, 1)),        # padding of all but a pixel
    (33, 16, 20, 22, 6, (3, 3), (0, 0), (1, 1), (1, 1)),      # where the direct kernels could be
    (60, 12, 24, 26, 16, (5, 5), (0, 0), (1, 1), (1, 1)),
]


def _reference(x, w, dy, p, s, d):
    x, w, dy = x.double(), w.double(), dy.double()
    kw = dict(padding=p, stride=s, dilation=d)
    y = F.conv2d(x, w, **kw)
    dx = torch.nn.grad.conv2d_input(x.shape, w, dy, **kw)
    dw = torch.nn.grad.conv2d_weight(x, w.shape, dy, **kw)
    return y, dw, dx


def _inputs(dev, case, dtype):
    bs, ic, h, w, oc, f, p, s, d = case
    gen = torch.Generator(device=dev.torch_device).manual_seed(ic * oc)
    rnd = lambda *shape: torch.randn(shape, generator=gen, device=dev.torch_device).to(dtype)
    out = [(n + 2 * p[i] - d[i] * (f[i] - 1) - 1) // s[i] + 1 for i, n in enumerate((h, w))]
    return rnd(bs, ic, h, w), rnd(oc, ic, *f), rnd(bs, oc, *out), dict(padding=p, stride=s, dilation=d)


@pytest.mark.parametrize("case,dtype", [(c, t) for c in CASES for t in (torch.float32, torch.bfloat16)] +
                         [(c, torch.float32) for c in RESIDENT])
def test_split_convolutions(dev, case, dtype):
    x, w, dy, opt = _inputs(dev, case, dtype)
    bias = torch.randn(w.shape[0], generator=torch.Generator().manual_seed(1)).to(dtype).to(x.device)
    biased = dev.conv2_forward(x, w, bias, relu=True, **opt)
    got = (dev.conv2_forward(x, w, **opt), dev.conv2_backward_weight(x, dy, tuple(w.shape[2:]), **opt),
           dev.conv2_backward_input(w, dy, tuple(x.shape[2:]), **opt))
    ref = _reference(x, w, dy, opt["padding"], opt["stride"], opt["dilation"])
    size = _reference(x.abs(), w.abs(), dy.abs(), opt["padding"], opt["stride"], opt["dilation"])
    dev.wait()
    for g, r, m in zip(got, ref, size):
        # an f32 rounding per 64 products and slice, on sums that grow as a walk: 2^-20 of the sum of magnitudes is a
        # hundred of them in a row; bf16's store on top
        bound = 2.0 ** -20 * m + (2.0 ** -8 * r.abs() if dtype == torch.bfloat16 else 0.0)
        assert bool(((g.double() - r).abs() <= bound).all())
    assert torch.equal(biased, (got[0] + bias[:, None, None]).clamp(min=0))
    if dtype == torch.float32:
        added = dev.conv2_backward_weight(x, dy, tuple(w.shape[2:]), beta=1.0, dw=torch.ones_like(got[1]), **opt)
        dev.wait()
        assert torch.equal(added, got[1] + 1)


@pytest.mark.parametrize("case", [CASES[1], RESIDENT[1]])
def test_split_convolutions_with_infinities(dev, case):
    """An infinity and a NaN of the input reach the outputs that they reach in float64.  Their blocks of 32 x 32 are computed
    again with FMAs one after another, so the others there have other roundings, within the same bound."""
    x, w, dy, opt = _inputs(dev, case, torch.float32)
    clean = x.clone()
    x[2, 7, 11, 13], x[5, -1, 0, 22] = float("inf"), float("nan")
    got = dev.conv2_forward(x, w, **opt), dev.conv2_backward_weight(x, dy, (3, 3), **opt)
    ref = _reference(x, w, dy, opt["padding"], opt["stride"], opt["dilation"])
    size = _reference(clean.abs(), w.abs(), dy.abs(), opt["padding"], opt["stride"], opt["dilation"])
    dev.wait()
    for g, r, m in zip(got, ref, size):
        assert torch.equal(g.isnan(), r.isnan()) and torch.equal(g.isinf(), r.isinf())
        assert bool((g[r.isinf()].sign() == r[r.isinf()].sign()).all())
        ok = r.isfinite()
        assert bool(((g.double() - r).abs()[ok] <= 2.0 ** -20 * m[ok]).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("case", [
    (9, 16, 10, 11, 64, (5, 5), (0, 0), (1, 1), (1, 1)),     # a few slices of one wave of tiles
    (24, 64, 13, 13, 100, (5, 5), (2, 2), (1, 1), (1, 1)),   # columns with a rest, shares of them that differ
    (50, 64, 12, 13, 33, (3, 3), (0, 0), (2, 2), (1, 1)),    # a last tile of 33 - 32 columns' share, strides
    (4, 40, 20, 24, 17, (3, 3), (1, 1), (1, 1), (1, 1)),
])
def test_slices_added_by_clusters(dev, case, dtype):
    """Convolutions whose k slices are added through the shared memory of a cluster, and one with a NaN in a slice."""
    x, w, dy, opt = _inputs(dev, case, dtype)
    for bad in (False, True):
        if bad:
            x[1, 3, 4, 5] = float("nan")
        got = dev.conv2_forward(x, w, **opt), dev.conv2_backward_weight(x, dy, tuple(w.shape[2:]), **opt)
        ref = _reference(x, w, dy, opt["padding"], opt["stride"], opt["dilation"])
        size = _reference(x.abs().nan_to_num(), w.abs(), dy.abs(), opt["padding"], opt["stride"], opt["dilation"])
        dev.wait()
        for g, r, m in zip(got, ref, size):
            ok = r.isfinite()
            assert torch.equal(g.isnan(), r.isnan())
            bound = 2.0 ** -20 * m + (2.0 ** -8 * r.abs() if dtype == torch.bfloat16 else 0.0)
            assert bool(((g.double() - r).abs()[ok] <= bound[ok]).all())
