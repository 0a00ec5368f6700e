"""Row parts of the forward projector's detector kernel (csrc/project.cu,
launch_fp_rays), by the kernel names that the profiler records, and its values
against the FP32 restatement: the parts shrink from 32 to 8 as the rays grow.
And the lane kernel's warps whose detectors lie past the image.

Tolerances: the projector's parity bar, 1e-5 relative L2, and 1e-4 of the largest
value per ray."""
import numpy as np
import pytest
import torch

from oracle import cpu_ref
from synkrotomo_gb300 import phantom
from synkrotomo_gb300 import runtime as rt
from tests.conftest import rel_l2
from tests.test_sirt_routes_gpu import _kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,angles,deltarho,kernel", [
    (512, 4, 1.0, "fp_det_kernel<32>"),
    (512, 30, 1.0, "fp_det_kernel<16>"),
    (512, 96, 0.25, "fp_det_kernel<8>"),      # 91 groups of 32 detectors, 96 angles
    (1026, 33, 1.0, "fp_det_kernel<8>"),
    (258, 31, 1.0, "fp_det_kernel<16>"),      # parts of 16 rows at most
    (66, 40, 0.5, "fp_det_kernel<4>"),
])
def test_row_parts(gpu, size, angles, deltarho, kernel):
    det = int(np.ceil(size * np.sqrt(2.0) / deltarho))
    g = phantom.geometry(size, angles, numrhos=det, deltarho=deltarho)
    img = np.random.default_rng(size + angles).random(size * size).astype(np.float32)
    args = (torch.from_numpy(g.angles).cuda(), g.rhozero, g.deltarho, g.numrhos, torch.from_numpy(img).cuda())
    out = rt.forwardprojection(*args).cpu().numpy()
    ref = cpu_ref.forwardprojection(g.angles, g.rhozero, g.deltarho, g.numrhos, img)
    assert rel_l2(out, ref) < 1e-5
    assert np.max(np.abs(out - ref)) <= 1e-4 * max(1.0, float(np.max(np.abs(ref))))
    assert any(kernel in n for n in _kernels(lambda: rt.forwardprojection(*args)))


@pytest.mark.parametrize("size,angles,det,first", [(16, 200, 300, -150.0), (34, 161, 90, 20.0), (66, 170, 47, -800.0)])
def test_detectors_past_the_image(gpu, size, angles, det, first):
    """Rows that reach far past the image on both sides, on one, and not to it at all
    (those rays must be zero)."""
    ang = phantom.geometry(size, angles).angles
    img = np.random.default_rng(size).random(size * size).astype(np.float32)
    out = rt.forwardprojection(torch.from_numpy(ang).cuda(), first, 1.0, det, torch.from_numpy(img).cuda()).cpu().numpy()
    ref = cpu_ref.forwardprojection(ang, first, 1.0, det, img)
    if first == -800.0:
        assert not ref.any() and not out.any()
    else:
        assert rel_l2(out, ref) < 1e-5
        assert np.max(np.abs(out - ref)) <= 1e-4 * max(1.0, float(np.max(np.abs(ref))))
