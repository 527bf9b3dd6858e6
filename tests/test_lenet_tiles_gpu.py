"""GPU: the tensor-core tile kernel of LeNet5 (bf16, large batches) against the kernels on the FP32 pipe, at
the smallest batch it takes, with a ragged last tile and with several tiles per SM."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("tiles,extra", [(0.5, 0), (1, 1), (2, -127), (3.3, 64)])
def test_tiles_against_fp32_pipe(dev, monkeypatch, tiles, extra, bias):
    sms = torch.cuda.get_device_properties(dev.torch_device).multi_processor_count
    bs = int(tiles * sms) * 128 + extra
    g = torch.Generator(device=dev.torch_device).manual_seed(bs)
    u = lambda *s: (torch.rand(s, device=dev.torch_device, generator=g) * 2 - 1)
    x = u(bs, 1, 28, 28).abs().to(torch.bfloat16)
    x[3, 0, 5, 6] = float("inf")       # its window only, and only this image
    x[bs - 1, 0, 27, 27] = float("nan")
    P = [(u(*s) * (2.0 / f) ** 0.5).to(torch.bfloat16) for s, f in
         [((6, 1, 5, 5), 25), ((16, 6, 5, 5), 150), ((256, 128), 256), ((128, 84), 128), ((84, 10), 84)]]
    biases = [u(n).mul(0.1).to(torch.bfloat16) for n in (128, 84, 10)] if bias else None
    run = lambda: dev.conv_dense_chain_forward(x, [(P[0], None, True, (2, 2)), (P[1], None, True, (2, 2))], P[2:],
                                               biases, [True, True, False])
    got = run().float().cpu().numpy()
    monkeypatch.setenv("AG_LENET_TILES", "0")
    ref = run().float().cpu().numpy()
    dev.wait()
    odd = [3, bs - 1]
    plain = np.setdiff1d(np.arange(bs), odd)
    assert np.isfinite(got[plain]).all()
    # sums in another order: a value now and then rounds the other way (2^-8), five layers deep
    err = got[plain].astype(np.float64) - ref[plain]
    assert np.linalg.norm(err) <= 5e-3 * np.linalg.norm(ref[plain])
    assert np.abs(err).max() <= 4e-2 * np.abs(ref[plain]).max()
    np.testing.assert_allclose(got[odd], ref[odd], rtol=4e-2, atol=4e-2 * np.abs(ref[plain]).max())
