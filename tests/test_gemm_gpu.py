"""GPU: ag_gemm / dot against the reference's tensor_dot vectors and the oracle."""
import itertools

import numpy as np
import pytest
import torch

import oracle
from conftest import cycle

pytestmark = pytest.mark.gpu


def _views(a, b, ta, tb):
    return (a.T if ta == "t" else a), (b.T if tb == "t" else b)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_tensor_dot_golden(dev, golden, dtype):
    """tensor_dot_<T>_m{n}_k{n}_n{n}_{nn,tn,nt,tt} (tests/integration_tests.rs:272-376)."""
    for n in [2, 4, 5, 8, 16, 32, 64, 128]:
        a = dev.tensor(cycle(1, 10, n * n).reshape(n, n), dtype)
        b = dev.tensor(cycle(1, 10, n * n).reshape(n, n), dtype)
        for ta, tb in itertools.product("nt", "nt"):
            av, bv = _views(a, b, ta, tb)
            c = dev.dot(av, bv).float().cpu().numpy()
            want = golden[f"dot_n{n}_{ta}{tb}"]
            if dtype == torch.bfloat16:
                want = oracle.round_bf16(want)  # f32 accumulation is exact here; one rounding
            assert np.array_equal(c, want), (n, ta, tb, dtype)


def _rel_err(c, ref):
    return float(np.abs(c.astype(np.float64) - ref).max() / max(np.abs(ref).max(), 1e-30))


@pytest.mark.parametrize("n", [256, 1024])
@pytest.mark.parametrize("layout", ["nn", "tn", "nt", "tt"])
def test_f32_random_vs_oracle(dev, n, layout):
    """Uniform [-1,1) operands; max error relative to max|C| within 1e-5*sqrt(K)."""
    rng = np.random.default_rng(3000 + n)
    a = rng.uniform(-1, 1, (n, n)).astype(np.float32)
    b = rng.uniform(-1, 1, (n, n)).astype(np.float32)
    av, bv = _views(a, b, *layout)
    ref = av.astype(np.float64) @ bv.astype(np.float64)
    if n <= 256:
        ref_o = oracle.gemm(av, bv, acc="f64")
        assert _rel_err(ref_o, ref) < 1e-6
    ad, bd = dev.tensor(a), dev.tensor(b)
    c = dev.dot(*_views(ad, bd, *layout)).cpu().numpy()
    assert _rel_err(c, ref) <= 1e-5 * np.sqrt(n)


def test_f32_4096_sampled_rows(dev):
    n = 4096
    rng = np.random.default_rng(3012)
    a = rng.uniform(-1, 1, (n, n)).astype(np.float32)
    b = rng.uniform(-1, 1, (n, n)).astype(np.float32)
    ad, bd = dev.tensor(a), dev.tensor(b)
    rows = rng.choice(n, 48, replace=False)
    for layout in ["nn", "tn", "nt"]:
        av, bv = _views(a, b, *layout)
        c = dev.dot(*_views(ad, bd, *layout)).cpu().numpy()
        ref = av[rows].astype(np.float64) @ bv.astype(np.float64)
        assert _rel_err(c[rows], ref) <= 1e-5 * np.sqrt(n), layout
        # linearity: column checksum of C equals (1^T A) B
        chk = (av.astype(np.float64).sum(0) @ bv.astype(np.float64))
        assert np.abs(c.astype(np.float64).sum(0) - chk).max() <= 1e-5 * np.sqrt(n) * n


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_alpha_beta_strides_offsets(dev, dtype):
    rng = np.random.default_rng(5)
    big_a = rng.integers(-3, 4, (40, 70)).astype(np.float32)
    big_b = rng.integers(-3, 4, (70, 50)).astype(np.float32)
    big_c = rng.integers(-3, 4, (45, 60)).astype(np.float32)
    ad, bd, cd = dev.tensor(big_a, dtype), dev.tensor(big_b, dtype), dev.tensor(big_c, dtype)
    # sub-views with offsets and non-unit column strides
    av, bv = ad[3:33, 5:65:2], bd[4:64:2, 1:49:3]       # 30x30, 30x16
    cv = cd[2:32, 7:39:2]                                # 30x16
    want = 2.0 * (big_a[3:33, 5:65:2] @ big_b[4:64:2, 1:49:3]) - 1.0 * big_c[2:32, 7:39:2]
    dev.gemm(2.0, av, bv, -1.0, cv)
    got = cd.float().cpu().numpy()
    expect = big_c.copy()
    expect[2:32, 7:39:2] = want
    assert np.array_equal(got, expect)  # small integers: exact in both types


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_split_k_and_skinny_shapes(dev, dtype):
    """The LeNet5 products the reference's author benchmarks (src/tensor/linalg.rs:507-519)."""
    rng = np.random.default_rng(6)
    shapes = [(57600, 25, 6, "nt"), (6400, 150, 16, "nt"), (100, 256, 128, "nn"),
              (100, 128, 84, "nn"), (100, 84, 10, "nn"), (100, 10, 84, "nt"), (84, 100, 10, "tn"),
              (128, 100, 84, "tn"), (256, 100, 128, "tn"), (16, 6400, 150, "tn"),
              (6, 57600, 25, "tn"), (3, 5000, 2, "nn")]
    for m, k, n, layout in shapes:
        a = rng.uniform(-1, 1, (m, k) if layout[0] == "n" else (k, m)).astype(np.float32)
        b = rng.uniform(-1, 1, (k, n) if layout[1] == "n" else (n, k)).astype(np.float32)
        if dtype == torch.bfloat16:
            a, b = oracle.round_bf16(a), oracle.round_bf16(b)
        av, bv = _views(a, b, *layout)
        ref = av.astype(np.float64) @ bv.astype(np.float64)
        c = dev.dot(*_views(dev.tensor(a, dtype), dev.tensor(b, dtype), *layout))
        c = c.float().cpu().numpy()
        tol = 1e-5 * np.sqrt(k) if dtype == torch.float32 else 1e-2
        assert _rel_err(c, ref) <= tol, (m, k, n, layout)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("layout", ["nn", "tn", "nt", "tt"])
def test_short_reductions_all_layouts(dev, dtype, layout):
    """k <= 128 with few output tiles takes the kernel that stages the whole k range."""
    rng = np.random.default_rng(61)
    for m, k, n in [(1, 1, 1), (33, 7, 5), (100, 8, 84), (97, 33, 130), (84, 100, 10),
                    (256, 128, 128), (130, 127, 31)]:
        a = rng.uniform(-1, 1, (m, k) if layout[0] == "n" else (k, m)).astype(np.float32)
        b = rng.uniform(-1, 1, (k, n) if layout[1] == "n" else (n, k)).astype(np.float32)
        if dtype == torch.bfloat16:
            a, b = oracle.round_bf16(a), oracle.round_bf16(b)
        av, bv = _views(a, b, *layout)
        ref = av.astype(np.float64) @ bv.astype(np.float64)
        ad, bd = dev.tensor(a, dtype), dev.tensor(b, dtype)
        c1 = dev.dot(*_views(ad, bd, *layout)).float().cpu().numpy()
        c2 = dev.dot(*_views(ad, bd, *layout)).float().cpu().numpy()
        tol = 1e-5 * np.sqrt(k) if dtype == torch.float32 else 1e-2
        assert _rel_err(c1, ref) <= tol, (m, k, n)
        assert np.array_equal(c1, c2)


def test_split_k_is_deterministic(dev):
    rng = np.random.default_rng(7)
    a = dev.tensor(rng.uniform(-1, 1, (16, 6400)).astype(np.float32))
    b = dev.tensor(rng.uniform(-1, 1, (6400, 150)).astype(np.float32))
    c1 = dev.dot(a, b).cpu().numpy()
    c2 = dev.dot(a, b).cpu().numpy()
    assert np.array_equal(c1, c2)


def test_empty_and_k_zero(dev):
    a = dev.empty((0, 5), torch.float32)
    b = dev.empty((5, 3), torch.float32)
    assert dev.dot(a, b).shape == (0, 3)
    a = dev.empty((4, 0), torch.float32)
    b = dev.empty((0, 3), torch.float32)
    c = dev.tensor(np.ones((4, 3), np.float32))
    dev.gemm(1.0, a, b, 2.0, c)
    assert np.array_equal(c.cpu().numpy(), 2 * np.ones((4, 3), np.float32))
    assert np.array_equal(dev.dot(a, b).cpu().numpy(), np.zeros((4, 3), np.float32))


def test_errors_like_reference(dev):
    import autograph_b200 as ag
    a = dev.empty((4, 5), torch.float32)
    with pytest.raises(ag.AgError, match="a_cols != b_rows"):
        dev.dot(a, dev.empty((4, 3), torch.float32))
    with pytest.raises(ag.AgError, match="different types"):
        dev.dot(a, dev.empty((5, 3), torch.bfloat16))
    with pytest.raises(ag.AgError):
        dev.gemm(1.0, a, dev.empty((5, 3), torch.float32), 0.0, dev.empty((4, 4), torch.float32))
    with pytest.raises(ag.AgError, match="unimplemented"):
        dev.dot(dev.empty((2, 2), torch.float64), dev.empty((2, 2), torch.float64))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (3, 512, 16), (5, 511, 10), (149, 84, 10), (600, 7, 3), (4096, 84, 10)])
def test_dense_with_few_outputs(dev, dtype, m, k, n):
    """One, two and four rows per CTA with ragged ends, against float64: k products and additions of f32 are within
    (k + 2) * 2^-24 of the sum of magnitudes, and bf16 rounds twice more."""
    gen = torch.Generator(device=dev.torch_device).manual_seed(m + n)
    x, w, b = (torch.rand(s, generator=gen, device=dev.torch_device).sub_(0.5).to(dtype) for s in ((m, k), (k, n), (n,)))
    got = dev.dense_forward(x, w, bias=b, relu=True).double()
    want = (x.double() @ w.double() + b.double()).clamp(min=0)
    bound = (k + 2) * 2.0 ** -24 * (x.double().abs() @ w.double().abs() + b.double().abs())
    if dtype == torch.bfloat16:
        bound += 2.0 ** -7 * (want.abs() + b.double().abs() + bound)
    assert ((got - want).abs() <= bound).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("m", [5, 300, 1000])   # one, two and four rows per CTA on their own
@pytest.mark.parametrize("k,n", [(84, 10), (83, 16), (130, 3), (256, 10), (7, 1)])
def test_dense_with_few_outputs_gives_the_bits_of_the_chain(dev, dtype, m, k, n):
    """The layer alone, as a dot, and as the last one of a run."""
    gen = torch.Generator(device=dev.torch_device).manual_seed(m + k + n)
    x, w0, w1, b = (torch.rand(s, generator=gen, device=dev.torch_device).sub_(0.5).to(dtype)
                    for s in ((m, 24), (24, k), (k, n), (n,)))
    h = dev.dense_forward(x, w0, relu=True)
    for bias, relu in ((b, False), (None, True)):
        chain = dev.dense_chain_forward(x, [w0, w1], [None, bias], [True, relu])
        assert torch.equal(dev.dense_forward(h, w1, bias=bias, relu=relu), chain)
    assert torch.equal(dev.dot(h, w1).clamp(min=0), chain)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("m,k,n", [(1, 129, 1), (31, 512, 16), (33, 511, 5), (64, 130, 8), (70, 256, 9), (512, 256, 10),
                                   (100, 300, 13), (5000, 150, 3), (129, 513, 12)])
def test_products_with_few_columns(dev, dtype, m, k, n):
    """a^T . b with up to 16 columns, rows of either operand and of the result further apart than they are long, against
    float64: the sums' roundings, at most k / 16 + 16 in a row of 2^-24 of the sum of magnitudes each, and bf16's store."""
    rng = torch.Generator().manual_seed(m * 1000 + k + n)
    a = torch.empty((k, m + 3)).uniform_(-1, 1, generator=rng).to(dtype).cuda(dev.torch_device)
    b = torch.empty((k, n + 2)).uniform_(-1, 1, generator=rng).to(dtype).cuda(dev.torch_device)
    c = torch.full((m, n + 1), 7.0, dtype=dtype, device=dev.torch_device)
    av, bv, cv = a[:, 1:m + 1], b[:, 2:], c[:, :n]
    from autograph_b200 import _capi, lib
    code = _capi.AG_F32 if dtype == torch.float32 else _capi.AG_BF16
    _capi.check(lib().ag_gemm(dev._h, code, m, k, n, 1.0, av.data_ptr(), 0, 1, m + 3, bv.data_ptr(), 0, n + 2, 1, 0.0,
                              cv.data_ptr(), 0, n + 1, 1))
    dev.wait()
    a64, b64 = av.double(), bv.double()
    bound = (k / 16 + 16) * 2.0 ** -24 * (a64.abs().t() @ b64.abs())
    ref = a64.t() @ b64
    if dtype == torch.bfloat16:
        bound = bound + 2.0 ** -8 * ref.abs()
    assert bool(((cv.double() - ref).abs() <= bound).all())
    assert bool((c[:, n] == 7.0).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("m,k,n", [(33, 511, 5), (512, 256, 10), (31, 512, 12)])
def test_products_with_few_columns_and_values_that_are_not_finite(dev, dtype, m, k, n):
    """One launch, and infinities and NaNs reach the outputs that they reach in float64 and no others: column 0 of b is zero, and
    what a warp's last group of eight k has beyond k multiplies nothing."""
    import autograph_b200 as ag
    rng = torch.Generator().manual_seed(m * 1000 + k + n)
    a = torch.empty((k, m)).uniform_(-1, 1, generator=rng).to(dtype).cuda(dev.torch_device)
    b = torch.empty((k, n)).uniform_(-1, 1, generator=rng).to(dtype).cuda(dev.torch_device)
    b[:, 0] = 0
    a[7, 3], a[k - 1, 20], a[k // 2, 11] = float("inf"), float("-inf"), float("nan")
    b[k - 2, n - 1] = float("inf")
    launches = ag.kernel_launch_count()
    c = dev.dot(a.t(), b).double()
    assert ag.kernel_launch_count() - launches == 1
    ref = a.double().t() @ b.double()
    dev.wait()
    assert torch.equal(c.isnan(), ref.isnan()) and torch.equal(c.isposinf(), ref.isposinf()) and torch.equal(c.isneginf(), ref.isneginf())
    ok = ref.isfinite()
    assert bool(((c - ref).abs()[ok] <= (2.0 ** -8 if dtype == torch.bfloat16 else 1e-5) * (1 + ref.abs()[ok])).all())
