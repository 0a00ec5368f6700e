"""Which kernels run a SIRT solve (csrc/capi.cu, sirt_batch), by the names that the
profiler records, and the same solves against the FP32 restatement: stacks and
single slices with too few tiles for the tile kernels, rests of one and two slices,
and each kernel that a moved threshold would leave untested.

Tolerance: 1e-5 relative L2 per slice, the parity bar of the SIRT path."""
import math

import numpy as np
import pytest
import torch

from oracle import cpu_ref
from synkrotomo_gb300 import phantom
from synkrotomo_gb300 import runtime as rt
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

SLICES4, SLICES2 = "sirt_bp_slices_kernel<4>", "sirt_bp_slices_kernel<2>"
GENERIC, SMALL = "sirt_bp_phase_kernel", "sirt_small_kernel"
TILES3, TILES4 = "sirt_bp_stack_kernel<3>", "sirt_bp_stack_kernel<4>"
BACKWARD = (SLICES4, SLICES2, GENERIC, SMALL, TILES3, TILES4, "sirt_persistent_kernel")


def _kernels(f):
    """Names of the kernels that f launches."""
    from torch.profiler import ProfilerActivity, profile
    for _ in range(3):                      # the first session of a process may come back empty
        with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
            f()
            torch.cuda.synchronize()
        names = [e.key for e in p.key_averages()]
        if any("synk::" in n for n in names):
            return names
    pytest.fail("the profiler recorded no kernel")


def _dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


@pytest.mark.parametrize("size,angles,ns,extra,kernels", [
    (96, 600, 8, 0, [GENERIC]),             # 18 tiles of 32 x 32 in two groups: the angles are split instead
    (128, 400, 4, 60, [GENERIC]),           # the same where the 64-row tiles' windows are in range
    (256, 400, 1, 30, [GENERIC]),           # one slice, 32 tiles of 32 x 64
    (160, 257, 10, 0, [SLICES4]),           # a rest of two beside two groups: one wave, one launch
    (320, 257, 2, 0, [SLICES2]),            # one pair; two chunks of angles, the second of one
    (512, 40, 9, 0, [SLICES4, SLICES2]),    # a rest of one after a wave of groups: launches of its own
    (32, 64, 250, 0, [SLICES4]),            # narrow slices below the other stacks' threshold
    (768, 361, 1, 40, [TILES3]),            # 288 blocks of 32 x 64, two chunks of angles
    (992, 261, 1, 100, [TILES4]),           # 496 blocks: four per SM fit 152 SMs, three do not
    (96, 90, 3, 0, [SMALL]),
])
def test_kernels_and_values(gpu, size, angles, ns, extra, kernels):
    g = phantom.geometry(size, angles, numrhos=phantom.default_detectors(size) + extra)
    some = sorted({0, ns // 2, ns - 1})     # the slices that are compared
    b = np.stack([phantom.add_noise(cpu_ref.forwardprojection(g.angles, g.rhozero, g.deltarho, g.numrhos,
                                                              phantom.ellipse_phantom(size, 20 + s % 12)), s)
                  for s in range(ns)])
    args = (_dev(g.angles), g.rhozero, g.deltarho, g.numrhos, size, ns, None, _dev(b).reshape(-1), 2)
    x, _, done = rt.sirt_slices(*args)
    x = x.cpu().numpy().reshape(ns, -1)
    for s in some:
        ref = cpu_ref.sirt(g.angles, g.rhozero, g.deltarho, np.zeros(size * size, np.float32), b[s], 2)
        assert rel_l2(x[s], ref) < 1e-5, s
    assert np.all(done.cpu().numpy() == 2)
    names = _kernels(lambda: rt.sirt_slices(*args))
    assert [k for k in BACKWARD if any(k in n for n in names)] == sorted(kernels, key=BACKWARD.index)


@pytest.mark.parametrize("size,angles,ns,deltarho,extra,forward,backward", [
    (768, 361, 1, 1.0, 40, "sirt_fp_stack_kernel", TILES3),     # one large slice
    (128, 200, 8, 0.75, 0, "sirt_fp_stack_kernel", GENERIC),    # a stack of another spacing: one slice per blockIdx.z
    (320, 257, 3, 1.0, 0, "sirt_fp_slices_kernel", SLICES4),    # a group of three slices, two chunks of angles
])
def test_history_and_stops_match_persistent(gpu, size, angles, ns, deltarho, extra, forward, backward):
    """Residual history and stopping iterations of the launched phases against the
    persistent kernel's (1e-5, as between the other engines: the same sums in other
    orders), the iterates against the FP32 restatement."""
    g = phantom.geometry(size, angles, numrhos=int(math.ceil(size * math.sqrt(2.0) / deltarho)) + extra,
                         deltarho=deltarho)
    vol = [phantom.ellipse_phantom(size, 3 + s) for s in range(ns)]
    b = np.stack([phantom.add_noise(cpu_ref.forwardprojection(g.angles, g.rhozero, g.deltarho, g.numrhos, v), s)
                  for s, v in enumerate(vol)])
    assert ns * angles * size * (size + g.numrhos) > 6e7
    its = 8
    args = (_dev(g.angles), g.rhozero, g.deltarho, g.numrhos, size, ns, None, _dev(b).reshape(-1), its)
    full = rt.resident_blocks()
    _, rp, _ = rt.sirt_slices(*args, residuals=True, grid_blocks=full)
    xs, rs, _ = rt.sirt_slices(*args, residuals=True)
    for x, bs in zip(xs.cpu().numpy().reshape(ns, -1), b):
        ref = cpu_ref.sirt(g.angles, g.rhozero, g.deltarho, np.zeros(size * size, np.float32), bs, its)
        assert rel_l2(x, ref) < 1e-5
    np.testing.assert_allclose(rs.cpu().numpy(), rp.cpu().numpy(), rtol=1e-5)
    tol = float(np.median(rp.cpu().numpy()[:, 4])) * 1.003
    _, _, dp = rt.sirt_slices(*args, tol=tol, grid_blocks=full)
    _, _, ds = rt.sirt_slices(*args, tol=tol)
    assert torch.equal(dp, ds) and int(ds.min()) < its
    names = _kernels(lambda: rt.sirt_slices(*args, tol=tol))
    assert any(forward in n for n in names) and any(backward in n for n in names)
