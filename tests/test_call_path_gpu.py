"""The drop-in classes' argument path: a flat contiguous tensor on the device is
taken as it is, any other form gives the same result, and each call runs on the
caller's current stream.  Equal inputs give equal bits."""
import numpy as np
import pytest
import torch

from futhark import backprojection, forwardprojection
from synkrotomo_gb300 import phantom

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["flat", "square", "strided", "host"])
def test_input_forms_and_streams(gpu, form):
    g = phantom.geometry(64, 40)
    img = torch.from_numpy(phantom.ellipse_phantom(64, seed=5))
    ang = torch.from_numpy(g.angles).cuda()
    ref = forwardprojection.forwardprojection().main(ang, g.rhozero, g.deltarho, g.numrhos, img.cuda()).torch()
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        x = torch.zeros(64 * 64, device="cuda")
        torch.cuda._sleep(20_000_000)                 # the image arrives late on this stream
        x.copy_(img.cuda())
        arg = {"flat": x, "square": x.view(64, 64), "strided": torch.stack([x, x], 1)[:, 0],
               "host": img.numpy()}[form]
        out = forwardprojection.forwardprojection().main(ang, g.rhozero, g.deltarho, g.numrhos, arg).torch()
        back = backprojection.backprojection().main(ang, g.rhozero, g.deltarho, 64, out).torch()
    s.synchronize()
    assert torch.equal(out, ref)
    assert torch.equal(back, backprojection.backprojection().main(ang, g.rhozero, g.deltarho, 64, ref).torch())
    assert np.array_equal(img.numpy(), phantom.ellipse_phantom(64, seed=5))
