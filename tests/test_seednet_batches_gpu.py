"""The seed net's gradients at the sizes where their launches change (partial 64-pixel and 128-row chunks, one and several
chunks per CTA, odd grids): the gradient of a batch is the mean of its images' gradients. With a power-of-two batch the
loss' 1 / blocks scales every bf16 operand exactly, so the two differ by float32 summation order alone: at most 2^13
accumulations of relative error 2^-22, 2e-3 of the norm."""
import numpy as np
import pytest
import torch

import framegen as fg
import seednet_train

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import build
    build.build()


@pytest.mark.parametrize("B,h,w", [(2, 1, 1), (16, 9, 7), (8, 33, 17), (32, 24, 40), (64, 64, 64), (4, 130, 250)])
def test_batch_gradient_is_the_mean_of_its_images(B, h, w):
    g = torch.Generator(device="cuda")
    g.manual_seed(B * h + w)
    luma = torch.rand((2, B, h, w), generator=g, device="cuda") * 255
    x = fg.SeedNet.pack(luma[0], luma[1])
    tgt = torch.randn((B, (h + 7) // 8, (w + 7) // 8, 6), generator=g, device="cuda")
    tgt[..., 4] = 1.0
    net = fg.SeedNet(B, h, w)
    net.set_params(seednet_train.init_params(3))
    loss = torch.zeros(1, device="cuda")
    net.backward(x, tgt, loss)
    whole, whole_loss = net.grads().astype(np.float64), float(loss)
    again = []
    for _ in range(2):   # a fixed summation order: the same bits every time
        net.zero_grads()
        net.backward(x, tgt, loss)
        again.append(net.grads())
    assert np.array_equal(again[0], again[1]) and np.array_equal(again[0], whole.astype(np.float32))
    mean, mean_loss = np.zeros_like(whole), 0.0
    for i in range(B):
        net.zero_grads()
        net.backward(x[i:i + 1], tgt[i:i + 1], loss)
        mean += net.grads() / B
        mean_loss += float(loss) / B
    assert net.fused_errors() == 0
    assert np.linalg.norm(whole) > 0 and np.linalg.norm(whole - mean) <= 2e-3 * np.linalg.norm(mean)
    assert abs(whole_loss - mean_loss) <= 1e-5 * abs(mean_loss)
    net.close()
