"""GPU: the tensor-core engines for operands TMA cannot read as they are (f32 split into bf16
planes, unaligned bf16, convolutions with any options) against float64."""
import numpy as np
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _views(a, b, layout):
    return (a.T if layout[0] == "t" else a), (b.T if layout[1] == "t" else b)


def _f32_bound(av, bv, k):
    """Per-element bound, S = sum |a||b|: in every 64-k block four additions of full-size terms and
    twenty of terms 2^-8 of that truncate to 24 bits (below 5 * 2^-23 S), the partial products left
    out are below 2^-24 S, and the k / 64 block sums are added with a rounding of 2^-24 each; k
    slices add at most as many roundings again."""
    s = av.double().abs() @ bv.double().abs()
    return s * (5 * 2.0 ** -23 + 2.0 ** -24 + 2 * (k / 64 + 1) * 2.0 ** -24)


def _bf16_bound(s, ref, k):
    """S = sum |a||b| again: in every 1024-k block 64 additions that truncate to 24 bits (2 more for those
    within one instruction), the block sums and k slices added with a rounding each, one bf16 store."""
    return ref.abs() * 2.0 ** -8 + s * (66 * 2.0 ** -23 + 2 * (k / 1024 + 1) * 2.0 ** -24)


@pytest.mark.parametrize("layout", ["nn", "nt", "tn", "tt"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [
    # gathered engine: one 32 / 64 / 128 column tile with ragged edges, k not a multiple of 8 or 64
    (2049, 513, 31), (4001, 165, 63), (257, 1030, 129), (1300, 333, 1301),
    # k slices, the last one short
    (130, 8003, 33),
    # packed engine: slices of k, whole tiles, tiles of a partial wave cut in two
    (1000, 5001, 130), (1537, 1601, 1703), (2560, 321, 2050),
    (1000, 20001, 130), (2560, 641, 2050),
])
def test_product_vs_f64(dev, dtype, layout, shape):
    m, k, n = shape
    gen = torch.Generator(device=dev.torch_device).manual_seed(m + k + n)
    mk = lambda r, c: (torch.rand((r, c), generator=gen, device=dev.torch_device) * 2 - 1).to(dtype)
    a = mk(*((m, k) if layout[0] == "n" else (k, m)))
    b = mk(*((k, n) if layout[1] == "n" else (n, k)))
    av, bv = _views(a, b, layout)
    c = dev.dot(av, bv)
    assert torch.equal(c, dev.dot(av, bv))
    ref = av.double() @ bv.double()
    err = (c.double() - ref).abs()
    bound = _f32_bound(av, bv, k)
    if dtype == torch.bfloat16:
        bound = _bf16_bound(av.double().abs() @ bv.double().abs(), ref, k)
    assert (err <= bound).all()
    # alpha, beta and a view of C, exact on small integers
    ai, bi = (torch.randint(-2, 3, t.shape, generator=gen, device=dev.torch_device).to(dtype) for t in (a, b))
    c0 = torch.randint(-4, 5, (m, n + 3), generator=gen, device=dev.torch_device).to(dtype)
    want = c0.double()
    want[:, 1:n + 1] = 0.5 * (_views(ai, bi, layout)[0].double() @ _views(ai, bi, layout)[1].double()) + 2 * want[:, 1:n + 1]
    dev.gemm(0.5, *_views(ai, bi, layout), 2.0, c0[:, 1:n + 1])
    assert torch.equal(c0, want.to(dtype))
    dev.wait()


@pytest.mark.parametrize("shape", [(700, 300, 200), (1100, 700, 1300), (1100, 1500, 1300)])
def test_f32_special_values(dev, shape):
    """Infinities, NaNs and values that round up to infinity in bf16 give what f32 gives; the rest
    of the product is not disturbed."""
    m, k, n = shape
    rng = np.random.default_rng(3)
    a = rng.integers(-3, 4, (m, k)).astype(np.float32)
    b = rng.integers(1, 4, (k, n)).astype(np.float32)
    a[3, 5], a[7, 9], a[11, 2], b[4, 6] = np.inf, np.nan, np.finfo(np.float32).max, -np.inf
    a[11, :] = np.where(np.arange(k) == 2, a[11, 2], 0)
    b[2, :] = np.where(np.arange(n) % 2, 1.0, 2.0)     # 2 * max overflows, 1 * max does not
    with np.errstate(all="ignore"):
        want = (a.astype(np.float64) @ b.astype(np.float64)).astype(np.float32)
    got = dev.dot(dev.tensor(a), dev.tensor(b)).cpu().numpy()
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(got[~np.isnan(got)], want[~np.isnan(want)])


CONVS = [
    # bs, ic, ih, iw, oc, f, padding, stride, dilation
    (9, 5, 31, 27, 33, 3, 1, 1, 1), (6, 16, 32, 32, 70, 3, 1, 2, 1), (5, 24, 29, 30, 130, 5, 2, 1, 1),
    (4, 33, 23, 41, 7, 3, 2, 2, 2), (7, 6, 40, 17, 96, (5, 3), (2, 0), (3, 1), (1, 2)),
]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("case", CONVS)
def test_convolution_vs_f64(dev, dtype, case):
    bs, ic, ih, iw, oc, f, pad, st, dil = case
    pair = lambda v: v if isinstance(v, tuple) else (v, v)
    f = pair(f)
    kw = dict(padding=pair(pad), stride=pair(st), dilation=pair(dil))
    gen = torch.Generator(device=dev.torch_device).manual_seed(ic * oc)
    rnd = lambda s: torch.randn(s, generator=gen, device=dev.torch_device).to(dtype)
    x, w = rnd((bs, ic, ih, iw)), rnd((oc, ic) + f)
    xd, wd = x.double().requires_grad_(), w.double().requires_grad_()
    y = F.conv2d(xd, wd, **kw)
    dy = rnd(tuple(y.shape))
    dx, dw = torch.autograd.grad(y, (xd, wd), dy.double())
    xa, wa = x.double().abs().requires_grad_(), w.double().abs().requires_grad_()
    ya = F.conv2d(xa, wa, **kw)
    dxa, dwa = torch.autograd.grad(ya, (xa, wa), dy.double().abs())
    got = (dev.conv2_forward(x, w, **kw), dev.conv2_backward_input(w, dy, (ih, iw), **kw),
           dev.conv2_backward_weight(x, dy, f, **kw))
    ks = (ic * f[0] * f[1], oc * f[0] * f[1], bs * y.shape[2] * y.shape[3])
    for g, ref, s, k in zip(got, (y, dx, dw), (ya, dxa, dwa), ks):
        bound = s * (5 * 2.0 ** -23 + 2.0 ** -24 + 2 * (k / 64 + 1) * 2.0 ** -24)   # as in _f32_bound
        if dtype == torch.bfloat16:
            bound = _bf16_bound(s, ref, k)
        assert ((g.double() - ref).abs() <= bound).all()
    dw2 = dev.conv2_backward_weight(x, dy, f, beta=1.0, dw=torch.ones_like(w), **kw)
    assert ((dw2.double() - dw - 1).abs() <= (bound * 1.01 + (dw.abs() + 1) * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23))).all()
    # the fused bias + relu equals the separate calls bit for bit
    b = rnd((oc,))
    assert torch.equal(dev.conv2_forward(x, w, bias=b, relu=True, **kw), dev.relu(dev.bias_add(got[0].clone(), b)))
    dev.wait()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(777, 333, 129), (5001, 260, 131), (1500, 1001, 900), (1500, 1601, 900)])
def test_dense_epilogue(dev, dtype, shape):
    """Bias and relu in either engine's epilogue equal the product and the separate calls."""
    bs, ins, outs = shape
    gen = torch.Generator(device=dev.torch_device).manual_seed(bs)
    rnd = lambda s: (torch.rand(s, generator=gen, device=dev.torch_device) - 0.5).to(dtype)
    x, w, b = rnd((bs, ins)), rnd((ins, outs)), rnd((outs,))
    assert torch.equal(dev.dense_forward(x, w, bias=b, relu=True),
                       dev.relu(dev.bias_add(dev.dot(x, w), b), inplace=True))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(1, 40, 33), (3, 512, 256), (75, 129, 64), (149, 17, 200), (600, 84, 10),
                                   (1200, 300, 100), (7, 8, 32)])
def test_small_products(dev, dtype, shape):
    """Every split of rows over CTAs of the latency-oriented kernel, ragged in all dimensions."""
    m, k, n = shape
    gen = torch.Generator(device=dev.torch_device).manual_seed(m)
    rnd = lambda s: (torch.rand(s, generator=gen, device=dev.torch_device) * 2 - 1).to(dtype)
    x, w, b = rnd((m, k)), rnd((k, n)), rnd((n,))
    ref = x.double() @ w.double()
    bound = x.double().abs() @ w.double().abs() * (k + 2) * 2.0 ** -24   # any order of k f32 roundings
    if dtype == torch.bfloat16:
        bound = bound + ref.abs() * 2.0 ** -8
    c = dev.dot(x, w)
    assert ((c.double() - ref).abs() <= bound).all()
    assert torch.equal(dev.dense_forward(x, w, bias=b, relu=True), dev.relu(dev.bias_add(c, b)))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(1, 25003, 515), (15, 700, 1201), (4999, 1030, 3),
                                   (208, 1328, 144), (384, 2864, 336), (160, 416, 432),
                                   (17, 333, 401), (40, 1436, 36)])
def test_few_rows_or_columns(dev, dtype, shape):
    """Long products with fewer rows or columns than an MMA tile has; aligned ones of a few tiles."""
    m, k, n = shape
    gen = torch.Generator(device=dev.torch_device).manual_seed(k)
    rnd = lambda s: (torch.rand(s, generator=gen, device=dev.torch_device) * 2 - 1).to(dtype)
    a, b = rnd((m, k)), rnd((k, n))
    ref = a.double() @ b.double()
    bound = _f32_bound(a, b, k)
    if dtype == torch.bfloat16:
        bound = _bf16_bound(a.double().abs() @ b.double().abs(), ref, k)
    assert ((dev.dot(a, b).double() - ref).abs() <= bound).all()
    dev.wait()


def _same_specials(got, want):
    """want in float64 of small integers: finite values equal, infinities and NaNs in their places."""
    want = want.to(torch.float32)
    nan = torch.isnan(want)
    assert torch.equal(torch.isnan(got), nan)
    assert torch.equal(got[~nan], want[~nan])


@pytest.mark.parametrize("layout", ["nn", "nt", "tn", "tt"])
@pytest.mark.parametrize("shape", [
    # gathered engine: several tiles per CTA; slices of k.  Packed: several tiles per pair, some cut in two; slices of k
    (2561, 100, 2049), (130, 8003, 33), (3300, 1501, 3333), (1000, 20001, 130),
])
def test_f32_not_finite_blocks(dev, layout, shape):
    """Sums that are not finite leave the pipeline of tiles alone: their blocks are computed after it, with
    C's old values read once."""
    m, k, n = shape
    gen = torch.Generator(device=dev.torch_device).manual_seed(m)
    ints = lambda r, c: torch.randint(-2, 3, (r, c), generator=gen, device=dev.torch_device).float()
    a, b = ints(m, k), ints(k, n)
    a[5, 7], a[m // 2, k - 1], a[m - 1, 0] = float("inf"), float("nan"), torch.finfo(torch.float32).max
    b[k // 3, n - 1] = float("-inf")
    b[0].clamp_(-1, 1)   # no overflow with the largest value
    strided = lambda t, l: t if l == "n" else t.t().contiguous().t()
    av, bv = strided(a, layout[0]), strided(b, layout[1])
    want = a.double() @ b.double()
    _same_specials(dev.dot(av, bv), want)
    c = ints(m, n + 1)
    want2 = 2 * want + 3 * c[:, 1:].double()
    dev.gemm(2.0, av, bv, 3.0, c[:, 1:])
    _same_specials(c[:, 1:], want2)
    # every output at once
    av[:, k // 2] = float("nan")
    assert torch.isnan(dev.dot(av, bv)).all()
    dev.wait()


def test_f32_not_finite_weight_gradient(dev):
    """180 tiles of 23,328 positions each on 148 SMs, without slices."""
    bs, ic, hw, oc = 8, 512, 56, 640
    gen = torch.Generator(device=dev.torch_device).manual_seed(1)
    ints = lambda *s: torch.randint(-2, 3, s, generator=gen, device=dev.torch_device).float()
    x, dy = ints(bs, ic, hw, hw), ints(bs, oc, hw - 2, hw - 2)

    def want():
        d = dy.double().transpose(0, 1).reshape(oc, -1)
        taps = [d @ x[:, :, i:i + hw - 2, j:j + hw - 2].double().transpose(0, 1).reshape(ic, -1).t()
                for i in range(3) for j in range(3)]
        return torch.stack(taps, 2).view(oc, ic, 3, 3)

    x[3, 100, 20, 20], x[0, 511, 55, 55], dy[1, 639, 0, 0] = float("nan"), float("inf"), float("-inf")
    _same_specials(dev.conv2_backward_weight(x, dy, (3, 3)), want())
    x.fill_(float("nan"))
    assert torch.isnan(dev.conv2_backward_weight(x, dy, (3, 3))).all()
    dev.wait()


@pytest.mark.parametrize("shape", [(700, 300, 200), (2561, 100, 2049), (1000, 5001, 130), (2560, 641, 2050)])
@pytest.mark.parametrize("layout", ["nn", "tn"])
@pytest.mark.parametrize("tiny", [-100, -112, -120, -126, -135, -145])
def test_f32_small_magnitudes(dev, shape, layout, tiny):
    """Operands down to f32's smallest normal number keep all their bits when the other operand brings the
    product back into range, whichever of the two is small; subnormal ones and sums count with an error of
    one unit of 2^-149 (the products left out are below 2^-24 of a product only while the first eight bits
    of an operand are a bf16 number)."""
    m, k, n = shape
    gen = torch.Generator(device=dev.torch_device).manual_seed(m)
    rnd = lambda r, c, e: torch.ldexp(torch.rand((r, c), generator=gen, device=dev.torch_device) * 2 - 1,
                                      torch.tensor(float(e), device=dev.torch_device))
    strided = lambda t, l: t if l == "n" else t.t().contiguous().t()
    for ea, eb in ((tiny, 100), (100, tiny)):
        a, b = strided(rnd(m, k, ea), layout[0]), strided(rnd(k, n, eb), layout[1])
        if tiny == -112:   # among ordinary values too
            a[::3], b[:, ::5] = torch.ldexp(a[::3], torch.tensor(-20.0, device=dev.torch_device)), 2.0 ** -10
        assert a.abs().max() > 0 and b.abs().max() > 0
        err = (dev.dot(a, b).double() - a.double() @ b.double()).abs()
        units = a.double().abs().sum(1, keepdim=True) + b.double().abs().sum(0, keepdim=True) + k
        assert (err <= _f32_bound(a, b, k) + units * 2.0 ** -149).all()
    dev.wait()


def _mean_signed(got, ref):
    return float(((got.double() - ref) / ref).mean())


@pytest.mark.parametrize("shape", [(1601, 100001, 1603), (1601, 3001, 1603), (130, 100001, 67)])
def test_bf16_long_positive_sums(dev, shape):
    """Sums of one sign over a long k: the truncating additions of an accumulator (64, half an ulp of 2^-23
    each on average) leave no more than 4e-6 towards zero; the rest of the limit is what the stores' roundings,
    whose spacing the sums' spread does not average out, show with FP32 arithmetic (2e-5)."""
    m, k, n = shape
    gen = torch.Generator(device=dev.torch_device).manual_seed(k)
    rnd = lambda r, c: torch.rand((r, c), generator=gen, device=dev.torch_device)
    a, b = (rnd(m, k) * (1 + rnd(m, 1))).bfloat16(), rnd(k, n).bfloat16()
    assert abs(_mean_signed(dev.dot(a, b), a.double() @ b.double())) <= 4e-5
    dev.wait()


def test_bf16_long_positive_weight_gradient(dev):
    """135 tiles of 147,456 positions each, without slices."""
    bs, ic, o, oc = 64, 128, 48, 640
    gen = torch.Generator(device=dev.torch_device).manual_seed(7)
    rnd = lambda *s: torch.rand(s, generator=gen, device=dev.torch_device)
    x, dy = rnd(bs, ic, 2 * o + 1, 2 * o + 1).bfloat16(), (rnd(bs, oc, o, o) * (1 + rnd(1, oc, 1, 1))).bfloat16()
    dw = dev.conv2_backward_weight(x, dy, (3, 3), stride=(2, 2))
    d = dy.double().transpose(0, 1).reshape(oc, -1)
    for i in range(3):
        for j in range(3):
            tap = x[:, :, i:i + 2 * o - 1:2, j:j + 2 * o - 1:2].double().transpose(0, 1).reshape(ic, -1)
            assert abs(_mean_signed(dw[:, :, i, j], d @ tap.t())) <= 4e-5
    dev.wait()
