"""Weight and bias gradients of the U-Net's full-resolution layers against 64
bits, where the operands are known exactly: with zero weights and unit biases every
activation of the last two layers is 1, the output is 0, and the gradient that
enters the last layer is the target, scaled by powers of two.

Tolerances, of the sum of absolute terms.  Weights: the tensor cores' FP32 sums
truncate at each step of 16 pixels, half a unit in the last place (at most 2^-23)
on average, and with positive terms the sum is half its final value on average: n
steps lose at most n * 2^-25.  A part of the rows, one per SM, has rows / SMs rows of
128 pixels, 8 steps each.  Biases: chains of as many additions as a part has rows,
then one atomic per SM, rounding to nearest: 2^-25 * sqrt(n) on average, four times
that at most."""
import math

import numpy as np
import pytest
import torch

from synkrotomo_gb300.unet import UNet, param_shapes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [16, 32])
def test_last_layer_against_64_bits(gpu, batch):
    size, at, pos = 256, {}, 0
    for name, shape in param_shapes():
        at[name] = slice(pos, pos + int(np.prod(shape)))
        pos += int(np.prod(shape))
    flat = torch.zeros(pos)
    flat[at["conv12.b"]] = 1.0
    flat[at["conv13.b"]] = 1.0
    head = torch.full((32,), 0.25)
    head[1::2] = -0.25
    flat[at["head.w"]] = head
    gen = torch.Generator(device="cuda").manual_seed(batch)
    v = torch.randn(batch, size, size, device="cuda", generator=gen).abs().bfloat16().float()
    net = UNet(size, batch, seed=1)
    net.load(flat)
    net.train_step(torch.zeros_like(v), -v, apply=False)
    grads = net.gradients().double().cpu()
    scale, vd = 2.0 / v.numel(), v.double()
    total = float(vd.sum()) * scale * 0.25
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    part = batch * 2 * size / sms
    tol_w, tol_b = 8.0 * part * 2.0 ** -25, 4.0 * math.sqrt(part + sms) * 2.0 ** -25
    sign = torch.sign(head).double()
    dw = grads[at["conv13.w"]].view(32, 3, 3, 32)
    for ky in range(3):
        for kx in range(3):
            rows, cols = slice(max(0, 1 - ky), min(size, size + 1 - ky)), slice(max(0, 1 - kx), min(size, size + 1 - kx))
            want = float(vd[:, rows, cols].sum()) * scale * 0.25
            assert float((dw[:, ky, kx] - want * sign[:, None]).abs().max()) < tol_w * total, (ky, kx)
    assert float((grads[at["conv13.b"]] - total * sign).abs().max()) < tol_b * total
