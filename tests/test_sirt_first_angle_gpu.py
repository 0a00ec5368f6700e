"""SIRT in one cooperative launch (csrc/sirt_small.cu) from a first angle off the
axes, against the FP32 restatement: detector rows short of the image and full
rows whose windows leave them past the last column (N off the 32-wide units).

Tolerance: 1e-5 relative L2, the parity bar of the SIRT path.  The restatement
is within 1.2e-6 of 64 bits on these geometries."""
import math

import numpy as np
import pytest
import torch

from oracle import cpu_ref
from synkrotomo_gb300 import phantom
from synkrotomo_gb300 import runtime as rt
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


def _dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


@pytest.mark.parametrize("first,step", [(0.3, 1), (math.radians(135.0), 1), (math.radians(179.0), -1)])
@pytest.mark.parametrize("size,angles,det", [(100, 91, 142), (200, 60, 283), (128, 90, 100)])
@pytest.mark.parametrize("ns", [1, 3])
def test_first_angle_off_the_axes(gpu, size, angles, det, first, step, ns):
    ang = (first + step * math.pi / angles * np.arange(angles)).astype(np.float32)
    rhozero, its = -(det - 1) / 2.0, 5
    b = np.stack([phantom.add_noise(cpu_ref.forwardprojection(ang, rhozero, 1.0, det,
                                                              phantom.ellipse_phantom(size, 60 + s)), s)
                  for s in range(ns)])
    start = np.stack([0.1 * phantom.ellipse_phantom(size, 70 + s) for s in range(ns)]).astype(np.float32)
    x, _, _ = rt.sirt_slices(_dev(ang), rhozero, 1.0, det, size, ns, _dev(start).reshape(-1), _dev(b).reshape(-1), its)
    x = x.cpu().numpy().reshape(ns, -1)
    for s in range(ns):
        ref = cpu_ref.sirt(ang, rhozero, 1.0, start[s], b[s], its)
        assert rel_l2(x[s], ref) < 1e-5, s
