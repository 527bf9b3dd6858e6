"""GPU: the fused LeNet5 training step against the layers run one by one, at the batch sizes where its
image groups (1, 2, 4), its parts of the batch and the last ragged group change."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("bs", [1, 7, 148, 149, 257, 299, 1003, 2501])
def test_fused_step_against_layers(dev, monkeypatch, dtype, bs):
    import autograph_b200 as ag
    momentum = 0.9 if bs % 2 else None
    fused = ag.Model(dev, ag.LENET5_SPEC, dtype, seed=11)
    monkeypatch.setenv("AG_FUSE_NET", "0")
    layers = ag.Model(dev, ag.LENET5_SPEC, dtype, seed=11)
    monkeypatch.delenv("AG_FUSE_NET")
    rng = np.random.default_rng(bs)
    buf = torch.empty(bs * 784 + 1, dtype=dtype).pin_memory()
    images = torch.from_numpy(rng.uniform(0, 1, (bs, 1, 28, 28)).astype(np.float32)).to(dtype)
    labels = torch.from_numpy(rng.integers(0, 10, bs).astype(np.uint8)).pin_memory()
    buf[1:] = images.reshape(-1)
    sources = [images.pin_memory(), buf[1:].reshape(bs, 1, 28, 28)]  # aligned, and a view that is not
    for m in (fused, layers):
        m.set_sgd(momentum)
    for step in range(2):
        before = [fused.get_parameter(i) for i in range(6)]
        x = sources[step]
        lf, ll = fused.train_step(x, labels, 0.01), layers.train_step(x, labels, 0.01)
        # f32: the sums differ in order only (about 1e-6); a relu or pool gate that turns on the last
        # bit moves one window's row of a gradient.  bf16: some values round the other way, 2^-8 each.
        tol = 1e-3 if dtype == torch.float32 else 2e-2
        assert abs(lf - ll) <= tol * 0.1 * abs(ll)
        for i in range(6):
            gf, gl = (m.get_gradient(i).astype(np.float64).ravel() for m in (fused, layers))
            assert np.linalg.norm(gf - gl) <= tol * np.linalg.norm(gl), (i, step)
            if momentum is None and dtype == torch.float32:
                assert np.array_equal(fused.get_parameter(i).ravel(),
                                      oracle.sgd_update(before[i].ravel(), fused.get_gradient(i).ravel(), 0.01))
        layers.set_parameters([fused.get_parameter(i) for i in range(6)])  # the next step starts equal again
    # the gradients alone, from device buffers, and the update as a call of its own: the same bits
    again = ag.Model(dev, ag.LENET5_SPEC, dtype, seed=11)
    again.set_sgd(momentum)
    xd, td = images.to(dev.torch_device), labels.to(dev.torch_device)
    for _ in range(2):
        again.train_forward_backward(xd, td, sync=False)
        again.apply_update(0.01)
    for i in range(6):
        assert np.array_equal(again.get_parameter(i), fused.get_parameter(i)), i
    for m in (fused, layers, again):
        m.close()
