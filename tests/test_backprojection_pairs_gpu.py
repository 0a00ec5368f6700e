"""The packed detector-pair backprojection (csrc/bp_tile.cuh, bp_chunk_pair) at
the edges of its chunks and tiles, against the FP32 restatement: one angle past
a 256-angle chunk, an odd last angle, the smallest image side that takes it,
and single-slice SIRT on both of its register variants.

Tolerances: the projectors' and SIRT's parity bar, 1e-5 relative L2."""
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


@pytest.mark.parametrize("size,a,extra", [
    (1184, 257, 100),       # 37 x 19 tiles, a second chunk of one angle, N = 32 mod 64
    (1216, 259, 90),        # an odd number of angles in the last chunk, axes among them
])
def test_dense_backprojection(gpu, size, a, extra):
    g = phantom.geometry(size, a, numrhos=phantom.default_detectors(size) + extra)
    y = np.random.default_rng(size + a).random(g.n_rays).astype(np.float32)
    out = rt.backprojection(_dev(g.angles), g.rhozero, g.deltarho, size, _dev(y)).cpu().numpy()
    ref = cpu_ref.backprojection(g.angles, g.rhozero, g.deltarho, size, y)
    assert rel_l2(out, ref) < 1e-5


@pytest.mark.parametrize("size,a,extra", [
    (448, 257, 60),         # 14 x 7 tiles: three blocks per SM
    (992, 260, 100),        # 31 x 16 tiles fit four blocks per SM of 152 SMs, not three
])
def test_single_slice_sirt(gpu, size, a, extra):
    g = phantom.geometry(size, a, numrhos=phantom.default_detectors(size) + extra)
    img = phantom.ellipse_phantom(size, 5)
    b = phantom.add_noise(cpu_ref.forwardprojection(g.angles, g.rhozero, g.deltarho, g.numrhos, img), 1)
    x = rt.sirt(_dev(g.angles), g.rhozero, g.deltarho, _dev(np.zeros(size * size, np.float32)), _dev(b), 2)
    ref = cpu_ref.sirt(g.angles, g.rhozero, g.deltarho, np.zeros(size * size, np.float32), b, 2)
    assert rel_l2(x.cpu().numpy(), ref) < 1e-5
