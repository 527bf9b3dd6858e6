"""GPU: convolutions whose tensors are split into channels-last bf16 planes ahead of the product (split_worth in
csrc/conv_tcx_impl.cuh; csrc/conv_halo_f32.cu, whose filters stay in shared memory): every direction against float64, and sums
that are not finite."""
import json
import re
import subprocess
import sys
from pathlib import Path

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

# bs, ic, h, w, oc, filter, padding, stride, dilation: 3e8 multiply-adds in every direction.
CASES = [
    (27, 40, 31, 28, 48, (3, 3), (1, 1), (1, 1), (1, 1)),    # channels in eights that are no sixteens
    (14, 45, 33, 30, 70, (3, 3), (0, 1), (1, 1), (1, 1)),    # channels and columns padded, 128-column tiles with a rest
    (33, 36, 29, 41, 33, (3, 5), (1, 2), (2, 1), (1, 1)),   # strides, columns beyond 32
    (36, 64, 27, 25, 20, (3, 3), (2, 2), (1, 1), (2, 2)),    # dilation: masks of taps, fewer columns than a tile
    (60, 32, 9, 9, 96, (5, 5), (2, 2), (1, 1), (1, 1)),     # few tiles: slices of k
    (6, 72, 50, 22, 130, (5, 3), (4, 0), (1, 2), (1, 1)),   # taps that leave the image on most sides
    (36, 72, 27, 25, 90, (3, 3), (2, 2), (1, 1), (2, 2)),    # dilation and more than 64 channels both ways
]
# The same for the engine with resident filters, f32: pixel rows of 32, 64 and 128 bytes both ways, 16, 32 and 64 columns with a
# rest, padding none, "same" and full, k groups with a rest.  Beside each case, what its forward pass, weight gradient and
# input gradient run on: r pixel rows, s split tensors, . neither.
RESIDENT = {
    (64, 16, 32, 32, 32, (3, 3), (1, 1), (1, 1), (1, 1)): "rrr",
    (90, 12, 29, 23, 20, (3, 3), (0, 0), (1, 1), (1, 1)): "rrr",
    (30, 30, 41, 35, 62, (3, 3), (2, 2), (1, 1), (1, 1)): "rss",
    (40, 60, 30, 27, 15, (3, 3), (1, 0), (1, 1), (1, 1)): "rrr",
    (70, 16, 26, 31, 6, (5, 5), (2, 2), (1, 1), (1, 1)): "srs",
    (150, 6, 33, 34, 33, (3, 3), (1, 1), (1, 1), (1, 1)): "r..",
    (50, 33, 25, 26, 13, (1, 5), (0, 2), (1, 1), (1, 1)): ".rr",
    (1500, 20, 12, 11, 40, (2, 3), (1, 1), (1, 1), (1, 1)): "r..",   # several images per tile, tiles in every accumulator
    (1500, 20, 12, 11, 30, (2, 3), (1, 1), (1, 1), (1, 1)): "rrr",
    (200, 40, 24, 23, 31, (3, 3), (1, 1), (1, 1), (1, 1)): "srr",    # weight gradients: two products a filter row, one accumulator of each
    (41, 3, 20, 21, 10, (3, 3), (0, 1), (1, 1), (1, 1)): ".rr",
    (17, 33, 9, 57, 16, (1, 7), (0, 3), (1, 1), (1, 1)): ".r.",      # four of them
    (9, 1, 40, 31, 5, (5, 4), (4, 3), (1, 1), (1, 1)): ".r.",        # padding of all but a pixel
    (33, 16, 20, 22, 6, (3, 3), (0, 0), (1, 1), (1, 1)): ".r.",      # where the direct kernels could be
    (60, 12, 24, 26, 16, (5, 5), (0, 0), (1, 1), (1, 1)): ".rr",
}
# Work enough to split, but each element is read too few times for the pass: splitting these took 1.2, 1.4 and 1.07 of their time
# forward.  The last two: weight gradients that pixel rows take 1.06 and 1.1 of their time for.
GATHERED = {
    (107, 32, 47, 47, 64, (3, 3), (0, 0), (2, 2), (1, 1)): "..s",
    (153, 64, 30, 30, 6, (3, 3), (0, 0), (2, 2), (1, 1)): "...",
    (42, 6, 57, 57, 32, (5, 5), (2, 2), (1, 1), (1, 1)): ".rs",
    (100, 1, 46, 46, 16, (5, 5), (2, 2), (1, 1), (1, 1)): "...",
    (50, 64, 12, 12, 16, (3, 3), (0, 0), (1, 1), (1, 1)): "...",
}
# bf16 runs here where the convolutions on TMA boxes do not take it.
ALL = [(c, torch.float32, e) for c, e in zip(CASES, ("sss", "sss", "sss", "ss.", "sss", "sss", "sss"))] + [(c, torch.float32, e) for c, e in RESIDENT.items()]
ALL += [(c, torch.bfloat16, e) for c, e in zip(CASES, ("...", "...", "sss", "ss.", "...", "sss", "sss"))]
ALL += [(c, torch.float32, e) for c, e in GATHERED.items()]


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


def _passes(dev, x, w, dy, opt):
    return (lambda: dev.conv2_forward(x, w, **opt), lambda: dev.conv2_backward_weight(x, dy, tuple(w.shape[2:]), **opt),
            lambda: dev.conv2_backward_input(w, dy, tuple(x.shape[2:]), **opt))


def _engines_seen():
    """For every case, the kernels of its three passes as the profiler names them; run in a process of its own."""
    sys.path.insert(0, str(Path(__file__).resolve().parent.parent))
    from torch.profiler import ProfilerActivity, profile

    import autograph_b200 as ag
    dev = ag.Device(0)
    torch.cuda.set_stream(dev.stream)
    seen = []
    for case, dtype, _ in ALL:
        got = ""
        for call in _passes(dev, *_inputs(dev, case, dtype)):
            dev.wait()
            with profile(activities=[ProfilerActivity.CUDA]) as prof:
                call()
                dev.wait()
            names = " ".join(e.name for e in prof.events())
            got += ("?" if not re.search(r"\w+_kernel\b", names) else "r" if "conv_halo_" in names else
                    "s" if re.search(r"\bsplit_kernel\b", names) else ".")
        seen.append(got)
    return seen


def test_engines_of_the_cases(dev):
    """The cases are where their tables say: a change to the lines between the engines moves them elsewhere otherwise, and the
    tests here pass without a launch of the kernels that they are for."""
    dev.wait()
    out = subprocess.run([sys.executable, __file__], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    seen = json.loads(out.stdout.splitlines()[-1])
    if any("?" in e for e in seen):
        pytest.skip("no kernel names from the profiler")
    assert {c: e for c, e in zip(ALL, seen) if e != c[2]} == {}


@pytest.mark.parametrize("case,dtype,engines", ALL)
def test_split_convolutions(dev, case, dtype, engines):
    x, w, dy, opt = _inputs(dev, case, dtype)
    bias = torch.randn(w.shape[0], generator=torch.Generator().manual_seed(1)).to(dtype).to(x.device)
    biased = dev.conv2_forward(x, w, bias, relu=True, **opt)
    got = [call() for call in _passes(dev, x, w, dy, opt)]
    ref = _reference(x, w, dy, opt["padding"], opt["stride"], opt["dilation"])
    size = _reference(x.abs(), w.abs(), dy.abs(), opt["padding"], opt["stride"], opt["dilation"])
    dev.wait()
    for g, r, m, engine in zip(got, ref, size, engines):
        # an f32 rounding per 64 products and slice, on sums that grow as a walk: 2^-20 of the sum of magnitudes is a
        # hundred of them in a row; bf16's store on top
        bound = 2.0 ** -20 * m + (2.0 ** -8 * r.abs() if dtype == torch.bfloat16 else 0.0)
        assert bool(((g.double() - r).abs() <= bound).all())
        if dtype == torch.float32 and engine != ".":
            # Of all values together: six products that leave out 2^-24 of a term (its square root's share of a sum), up to
            # a hundred roundings of 2^-25 on the way of a sum that grows as their walk does.  Three products instead of the
            # six, or planes of two, are 4e-6 off.
            error = ((g.double() - r).norm() / r.norm()).item()
            assert error <= 5e-7, error
    assert torch.equal(biased, (got[0] + bias[:, None, None]).clamp(min=0))
    if dtype == torch.float32:
        added = dev.conv2_backward_weight(x, dy, tuple(w.shape[2:]), beta=1.0, dw=torch.ones_like(got[1]), **opt)
        dev.wait()
        assert torch.equal(added, got[1] + 1)


@pytest.mark.parametrize("case", [CASES[1], list(RESIDENT)[1], list(RESIDENT)[3]])
def test_split_convolutions_with_infinities(dev, case):
    """An infinity and a NaN of an operand reach the outputs that they reach in float64.  Their blocks of 32 x 32 are computed
    again with FMAs one after another, so the others there have other roundings, within the same bound."""
    x, w, dy, opt = _inputs(dev, case, torch.float32)
    bad_x, bad_dy = x.clone(), dy.clone()
    bad_x[2, 7, 11, 13], bad_x[5, -1, 0, 22] = float("inf"), float("nan")
    bad_dy[3, 4, 10, 9], bad_dy[1, 0, 5, 6] = float("-inf"), float("nan")   # where all taps meet pixels
    opts = opt["padding"], opt["stride"], opt["dilation"]
    passes = _passes(dev, bad_x, w, dy, opt)[:2] + _passes(dev, x, w, bad_dy, opt)[1:]
    got = [call() for call in passes]
    ref = _reference(bad_x, w, dy, *opts)[:2] + _reference(x, w, bad_dy, *opts)[1:]
    size = _reference(x.abs(), w.abs(), dy.abs(), *opts)
    dev.wait()
    for g, r, m in zip(got, ref, size[:2] + size[1:]):
        assert torch.equal(g.isnan(), r.isnan()) and torch.equal(g.isinf(), r.isinf())
        assert bool(r.isnan().any()) and bool(r.isinf().any())
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


@pytest.mark.parametrize("bs,ic,hw,oc,pad", [(9, 61, 27, 1, 1), (3, 29, 39, 3, 0), (16, 46, 30, 15, 1)])
def test_weight_gradients_on_pixel_rows_add_as_a_tree(dev, bs, ic, hw, oc, pad):
    """Few rows a CTA and sums of many CTAs: a thread adds at most five, and the 32 threads' sums go through five additions, so
    that roundings (2^-24 of a partial sum) stay below what the products themselves leave, 1e-7 in 2-norm.  With the 32 added
    in a row the errors were above 1.3e-7."""
    gen = torch.Generator(device=dev.torch_device).manual_seed(bs)
    error = 0.0
    for _ in range(3):
        x = torch.randn((bs, ic, hw, hw), generator=gen, device=dev.torch_device)
        dy = torch.randn((bs, oc, hw + 2 * pad - 2, hw + 2 * pad - 2), generator=gen, device=dev.torch_device)
        ref = torch.nn.grad.conv2d_weight(x.double(), (oc, ic, 3, 3), dy.double(), padding=pad)
        got = dev.conv2_backward_weight(x, dy, (3, 3), padding=(pad, pad)).double()
        error += ((got - ref).norm() / ref.norm()).item() / 3
    assert error <= 1.25e-7, error


if __name__ == "__main__":
    print(json.dumps(_engines_seen()))
