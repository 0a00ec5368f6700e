"""The row-streaming 3x3 convolution (image rows of 128k pixels, weights of all
taps in shared memory) against plain PyTorch FP32 at its edges: images of one,
two and three rows, runs of rows that cross columns and images, fewer rows than
SMs and many more, 64- and 32-channel strips with a half-filled last one, one
and several n tiles, channel slices, and weights at an address that needs a copy.
BF16 outputs round to 2^-9 of each element, so the relative L2 error of an exact
FP32 accumulation stays below that."""
import pytest
import torch
import torch.nn.functional as Fnn

from synkrotomo_gb300 import runtime as rt

pytestmark = pytest.mark.gpu
TOL = 1.01 * 2.0 ** -9


def _conv(x, w, b=None):
    cin = x.shape[-1]
    wk = w.reshape(w.shape[0], 3, 3, cin).permute(0, 3, 1, 2).double()
    y = Fnn.conv2d(x.double().permute(0, 3, 1, 2), wk, None if b is None else b.double(), padding=1)
    return y.permute(0, 2, 3, 1)


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm().clamp_min(1e-30))


CASES = [(1, 1, 128, 32, 32), (2, 2, 128, 32, 64), (3, 3, 256, 64, 32), (1, 5, 384, 96, 32), (2, 40, 256, 32, 96),
         (3, 17, 128, 64, 64), (1, 9, 128, 64, 192), (1, 7, 256, 64, 128), (5, 64, 128, 160, 32), (2, 130, 256, 32, 128)]


@pytest.mark.parametrize("B,H,W,Cin,Cout", CASES)
@pytest.mark.parametrize("off", [0, 1])
def test_rows_forward_and_backward_data(gpu, B, H, W, Cin, Cout, off):
    g = torch.Generator(device="cuda").manual_seed(B * H + W + Cin * Cout)
    ldx, xoff, ldy, yoff = Cin + 40, 8, Cout + 24, 16
    xbuf = torch.randn(B, H, W, ldx, device="cuda", generator=g).to(torch.bfloat16)
    store = (0.1 * torch.randn(Cout * 9 * Cin + 8, device="cuda", generator=g)).to(torch.bfloat16)
    w = store[off:off + Cout * 9 * Cin]           # off 1: two bytes past a 16-byte boundary
    bias = torch.randn(Cout, device="cuda", generator=g)
    x, wm = xbuf[..., xoff:xoff + Cin], w.reshape(Cout, 9 * Cin)
    mask = torch.randn(B, H, W, ldy, device="cuda", generator=g).to(torch.bfloat16)
    mask[..., 1::3] = 0.0
    want = _conv(x, wm)
    ctx = rt.context()
    for epi, ref in ((1, torch.relu(want + bias.double())), (4, want + bias.double()),
                     (2, want * (mask[..., yoff:yoff + Cout].double() > 0))):
        y = torch.full((B, H, W, ldy), 7.0, dtype=torch.bfloat16, device="cuda")
        rc = ctx.lib.synk_conv3x3_bf16(ctx.handle, rt._ptr(xbuf), ldx, xoff, Cin, B, H, W, w.data_ptr(),
                                       rt._ptr(bias), rt._ptr(y), ldy, yoff, Cout, epi,
                                       rt._ptr(mask) if epi == 2 else None, ldy, yoff)
        ctx.check(rc, "conv")
        ctx.sync()
        assert _rel(y[..., yoff:yoff + Cout], ref) < TOL
        assert bool((y[..., :yoff] == 7.0).all()) and bool((y[..., yoff + Cout:] == 7.0).all())
