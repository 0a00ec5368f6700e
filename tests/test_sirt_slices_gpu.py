"""SIRT of slice stacks on slice-pair planes (csrc/sirt_slices.cu): every
slice against the FP32 restatement, over even and odd slice counts, angle
counts around the 256-angle chunk, image sides off the 32-pixel tiles and
several row splits.

Tolerance: 1e-5 relative L2 per slice, the parity bar of the SIRT path; both
sides round in float32 in different orders.
"""
import math

import numpy as np
import pytest
import torch

from oracle import cpu_ref
from synkrotomo_gb300 import phantom
from synkrotomo_gb300 import runtime as rt
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

# size, angles, detectors, slices, iterations, arc: all above 6e7 ray-row
# steps plus pixel-angle pairs per iteration, where stacks take these kernels
CASES = [
    (160, 180, None, 7, 6, math.pi),            # two slice groups of 4, the last padded
    (160, 180, None, 9, 3, math.pi),            # two groups and a last pair of one slice
    (130, 257, 184, 6, 4, math.pi),             # two chunks of angles, the second of one; a last pair
    (98, 520, 142, 8, 3, 2 * math.pi),          # three chunks, all four axes, N = 2 mod 32
    (256, 256, None, 2, 3, math.pi),            # one pair only
    (512, 45, 730, 3, 2, 2 * math.pi / 3),      # few angles: lanes of one warp far apart
]


def _problem(size, a, nr, ns, arc):
    g = phantom.geometry(size, a, numrhos=nr, arc=arc)
    b = []
    for s in range(ns):
        img = phantom.ellipse_phantom(size, 40 + s)
        b.append(phantom.add_noise(cpu_ref.forwardprojection(g.angles, g.rhozero, g.deltarho, g.numrhos, img), s))
    return g, np.stack(b)


def _dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


@pytest.mark.parametrize("size,a,nr,ns,its,arc", CASES)
def test_stack_matches_oracle(gpu, size, a, nr, ns, its, arc):
    g, b = _problem(size, a, nr, ns, arc)
    start = np.stack([0.1 * phantom.ellipse_phantom(size, 90 + s) for s in range(ns)]).astype(np.float32)
    for image in (None, start):
        ref = [cpu_ref.sirt(g.angles, g.rhozero, g.deltarho,
                            np.zeros(size * size, np.float32) if image is None else image[s], b[s], its)
               for s in range(ns)]
        for split in (0, 4):
            x, res, done = rt.sirt_slices(_dev(g.angles), g.rhozero, g.deltarho, g.numrhos, size, ns,
                                          None if image is None else _dev(image).reshape(-1), _dev(b).reshape(-1),
                                          its, residuals=True, fp_split=split)
            x = x.cpu().numpy().reshape(ns, -1)
            for s in range(ns):
                assert rel_l2(x[s], ref[s]) < 1e-5, (s, split)
            r = res.cpu().numpy()
            last = [cpu_ref.forwardprojection(g.angles, g.rhozero, g.deltarho, g.numrhos, ref[s]) for s in range(ns)]
            want = [np.linalg.norm(last[s].astype(np.float64) - b[s]) / np.linalg.norm(b[s].astype(np.float64))
                    for s in range(ns)]
            np.testing.assert_allclose(r[:, its], want, rtol=1e-4)
            assert np.all(done.cpu().numpy() == its)


def test_stack_without_history_is_the_same(gpu):
    size, a, ns, its = 160, 180, 7, 5
    g, b = _problem(size, a, None, ns, math.pi)
    args = (_dev(g.angles), g.rhozero, g.deltarho, g.numrhos, size, ns, None, _dev(b).reshape(-1), its)
    x1, _, _ = rt.sirt_slices(*args, residuals=True)
    x2, _, _ = rt.sirt_slices(*args)
    assert torch.equal(x1, x2)


def test_stack_stopping_rule_per_slice(gpu):
    """Slices of one group stop at their own iterations and keep the iterate they had there."""
    size, a, ns, its = 160, 180, 6, 30
    g, b = _problem(size, a, None, ns, math.pi)
    b[1] *= 0.0
    b[1, 5] = 1.0
    args = (_dev(g.angles), g.rhozero, g.deltarho, g.numrhos, size, ns, None, _dev(b).reshape(-1))
    _, res, _ = rt.sirt_slices(*args, its, residuals=True)
    hist = res.cpu().numpy()
    tol = float(np.sort(hist[:, 12])[2]) * 1.0001
    x, _, done = rt.sirt_slices(*args, its, tol=tol, residuals=True)
    x = x.cpu().numpy().reshape(ns, -1)
    stops = [next((i for i in range(its) if hist[s, i] <= tol), its) for s in range(ns)]
    assert len(set(stops)) > 1
    assert done.cpu().numpy().tolist() == stops
    for s in range(ns):
        y, _, _ = rt.sirt_slices(*args, stops[s])
        assert np.array_equal(x[s], y.cpu().numpy().reshape(ns, -1)[s])
