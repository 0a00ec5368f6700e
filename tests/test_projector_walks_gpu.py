"""The forward projector's packed walk and its two kernels (csrc/fp_tile.cuh,
csrc/project.cu) at the edges of their ranges: angle counts around the
detector/lane kernel threshold, image sides whose rows leave a remainder of
two, detectors past and short of the image, and the largest side, whose two
pair images take one launch per class.

Tolerances: the projector's parity bar, 1e-5 relative L2 against the FP32
restatement, and 1e-4 of the largest value per ray."""
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


def _check(g, img):
    out = rt.forwardprojection(_dev(g.angles), g.rhozero, g.deltarho, g.numrhos, _dev(img)).cpu().numpy()
    ref = cpu_ref.forwardprojection(g.angles, g.rhozero, g.deltarho, g.numrhos, img)
    assert rel_l2(out, ref) < 1e-5
    assert np.max(np.abs(out - ref)) <= 1e-4 * max(1.0, float(np.max(np.abs(ref))))


@pytest.mark.parametrize("size,a,nr,dr,arc", [
    (2, 40, 5, 1.0, math.pi),               # smallest image
    (6, 200, 9, 1.0, 2 * math.pi),
    (66, 159, None, 1.0, math.pi),          # detector kernel, rows 4n + 2
    (66, 160, None, 1.0, math.pi),          # lane kernel
    (130, 161, 300, 1.0, 2 * math.pi),      # detectors far past the image
    (258, 33, 97, 1.0, math.pi),            # detectors short of the image
    (322, 650, 463, 0.7, math.pi),          # several chunks of rows, one row part
    (600, 257, None, 1.0, 2 * math.pi / 3),
])
def test_walk_edges(gpu, size, a, nr, dr, arc):
    g = phantom.geometry(size, a, numrhos=nr, deltarho=dr, arc=arc)
    rng = np.random.default_rng(size + a)
    _check(g, rng.random(size * size).astype(np.float32))


@pytest.mark.parametrize("a", [3, 165])
def test_largest_side(gpu, a):
    """N = 16384: the pair images span more than 4 GB, so each class is its own launch."""
    size, nr = 16384, 24
    g = phantom.geometry(size, a, numrhos=nr, deltarho=600.0)
    rng = np.random.default_rng(a)
    img = rng.random(size * size, dtype=np.float32)
    _check(g, img)


def test_non_finite_angle_stays_in_its_row(gpu):
    """A NaN angle leaves the other angles' rows as they are without it."""
    g = phantom.geometry(96, 200)
    img = phantom.ellipse_phantom(96, 3)
    ang = g.angles.copy()
    ref = rt.forwardprojection(_dev(ang), g.rhozero, 1.0, g.numrhos, _dev(img)).cpu().numpy().reshape(200, -1)
    ang[70] = np.float32("nan")
    out = rt.forwardprojection(_dev(ang), g.rhozero, 1.0, g.numrhos, _dev(img)).cpu().numpy().reshape(200, -1)
    keep = np.arange(200) != 70
    assert rel_l2(out[keep], ref[keep]) < 1e-6
