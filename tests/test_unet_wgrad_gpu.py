"""Weight and bias gradients of the U-Net's 3x3 layers at other splits of their
pixel rows: the gradient of a batch is the mean of its images' gradients.  With a
power of two of images the factor is exact in every format on the way, so only
the order of FP32 sums differs (relative L2 2e-5 per tensor, over sums of up to
2^20 terms that round to 2^-24).  Sides 256 and 512 have rows of 512 down to 32
pixels; a net of one image has fewer rows than CTAs at its lowest level.  At 512 the FP64 oracle judges as well, at the BF16 tolerance of the
other gradient tests."""
import numpy as np
import pytest
import torch

from oracle import unet_ref
from synkrotomo_gb300 import phantom
from synkrotomo_gb300.unet import UNet, param_shapes

pytestmark = pytest.mark.gpu


def _grads(net, x, t):
    net.train_step(x, t, apply=False)
    return net.gradients().cpu().double()


def _check(a, b, tol):
    off = 0
    for name, shape in param_shapes():
        n = int(np.prod(shape))
        u, v = a[off:off + n], b[off:off + n]
        off += n
        if float(v.norm()) > 1e-12:
            assert float((u - v).norm() / v.norm()) < tol, name


@pytest.mark.parametrize("size,batch", [(256, 2), (256, 8), (512, 2)])
def test_batch_gradient_is_the_mean_of_its_images(gpu, size, batch):
    t = torch.stack([torch.from_numpy(phantom.ellipse_phantom(size, 5 + b)).reshape(size, size) for b in range(batch)])
    g = torch.Generator().manual_seed(size + batch)
    x = (0.6 * t + 0.05 * torch.randn(t.shape, generator=g)).float()
    t = t.float()
    p = None
    single = 0.0
    for b in range(batch):
        net = UNet(size, 1, seed=4)   # gradients add up within a net
        if p is None:
            p = net.params()
            p[-33:-1] = torch.linspace(-0.5, 0.5, 32, device="cuda")
        net.load(p)
        single = single + _grads(net, x[b:b + 1], t[b:b + 1]) / batch
    net = UNet(size, batch, seed=4)
    net.load(p)
    whole = _grads(net, x, t)
    _check(whole, single, 2e-5)
    if size == 512:
        ref = unet_ref.loss_and_grads(p.cpu(), x.numpy()[:1], t.numpy()[:1])[2]
        net = UNet(size, 1, seed=4)
        net.load(p)
        _check(_grads(net, x[:1], t[:1]), ref, 5e-2)
