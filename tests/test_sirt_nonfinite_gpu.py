"""NaN in the start image or the measured data reaches the same pixels from every
SIRT engine: a ray that misses a pixel takes nothing from it, and a pixel takes
nothing from detectors outside its window (a candidate inside it counts, with
weight zero too).  One iteration from each engine; the patterns of NaN must be
those of the phase kernels or the persistent kernel, whose gathers are bounded
ray by ray and window by window, and the other pixels must agree to 1e-5, the
parity bar.

The angles start off the axes and the sizes are small, so no detector coordinate
lies within rounding of a window's end."""
import math

import numpy as np
import pytest
import torch

from synkrotomo_gb300 import phantom
from synkrotomo_gb300 import runtime as rt
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


def _solve(ang, det, size, ns, image, b, grid):
    x, _, _ = rt.sirt_slices(torch.from_numpy(ang).cuda(), -(det - 1) / 2.0, 1.0, det, size, ns,
                             None if image is None else torch.from_numpy(image).cuda(), torch.from_numpy(b).cuda(), 1,
                             grid_blocks=grid)
    return x.cpu().numpy()


def _same(got, want):
    bad = np.isnan(want)
    assert bad.any() and not bad.all()
    assert np.array_equal(np.isnan(got), bad)
    assert rel_l2(got[~bad], want[~bad]) < 1e-5


@pytest.mark.parametrize("size,angles,row,col", [(64, 8, 20, 32), (130, 6, 100, 65), (66, 10, 3, 33),
                                                 (64, 7, 20, 32)])
def test_rays_that_miss_a_nan_pixel(gpu, size, angles, row, col):
    """The centre column is where lanes without a ray walk."""
    det = phantom.default_detectors(size)
    ang = (0.31 + math.pi / angles * np.arange(angles)).astype(np.float32)
    b = np.random.default_rng(size).random(angles * det).astype(np.float32)
    image = np.zeros((size, size), np.float32)
    image[row, col] = np.nan
    _same(_solve(ang, det, size, 1, image.ravel(), b, 0), _solve(ang, det, size, 1, image.ravel(), b, -1))


@pytest.mark.parametrize("size,angles", [(64, 7), (130, 33), (66, 1)])
def test_odd_angle_count_and_a_nan_detector(gpu, size, angles):
    """The last angle of an odd count is read by the filler of its pair too."""
    det = phantom.default_detectors(size)
    ang = (0.31 + math.pi / angles * np.arange(angles)).astype(np.float32)
    b = np.random.default_rng(size).random((angles, det)).astype(np.float32)
    b[-1, det // 2] = np.nan
    _same(_solve(ang, det, size, 1, None, b.ravel(), 0), _solve(ang, det, size, 1, None, b.ravel(), -1))


@pytest.mark.parametrize("size,angles,ns", [(256, 45, 12), (250, 45, 13), (160, 271, 6)])
def test_stack_with_a_nan_detector(gpu, size, angles, ns):
    """Neighbouring pixels of the interleaved slices share a window of three
    detectors, of which a pixel's own are two."""
    det = phantom.default_detectors(size)
    assert ns * angles * size * (size + det) > 6.5e7
    ang = (0.31 + math.pi / angles * np.arange(angles)).astype(np.float32)
    b = np.random.default_rng(size).random((ns, angles, det)).astype(np.float32)
    b[1, 3, det // 3] = np.nan
    b[-1, 7, det // 2 + 11] = np.nan
    _same(_solve(ang, det, size, ns, None, b.ravel(), 0),
          _solve(ang, det, size, ns, None, b.ravel(), rt.resident_blocks()))
