"""SIRT of small problems in one cooperative launch (csrc/sirt_small.cu) against
the FP32 restatement: image sides and detector counts off the 32-wide units,
odd angle counts, the largest angle count it takes and one more, detectors
short of the image, only near-axis angles, several slices, the stopping rule
and the barrier's time limit.

Tolerance: 1e-5 relative L2, the parity bar of the SIRT path."""
import math

import numpy as np
import pytest
import torch

from oracle import cpu_ref
from synkrotomo_gb300 import phantom
from synkrotomo_gb300 import runtime as rt
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

CASES = [
    # size, angles, detectors, slices, iterations, arc
    (2, 1, 3, 1, 4, math.pi),                  # one near-axis angle, one unit
    (16, 2, 24, 1, 6, math.pi),                # both axes only: no fast-path unit
    (34, 33, 49, 1, 12, math.pi),              # two detector groups, odd angles, N = 2 mod 32
    (64, 5, 91, 3, 8, 2 * math.pi / 3),        # fewer angles than parts, several slices
    (66, 360, 95, 1, 5, 2 * math.pi),          # the most angles, all four axes
    (66, 361, 95, 1, 5, 2 * math.pi),          # one more: the launched phases
    (96, 90, 60, 1, 6, math.pi),               # detectors short of the image: bounds tests
    (128, 128, 182, 2, 10, math.pi),
    (320, 200, 453, 1, 4, math.pi),            # several rounds of units per block
]


def _dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def _problem(size, a, nr, ns, arc):
    g = phantom.geometry(size, a, numrhos=nr, arc=arc)
    b = [phantom.add_noise(cpu_ref.forwardprojection(g.angles, g.rhozero, g.deltarho, g.numrhos,
                                                     phantom.ellipse_phantom(size, 60 + s)), s) for s in range(ns)]
    return g, np.stack(b)


@pytest.mark.parametrize("size,a,nr,ns,its,arc", CASES)
def test_small_matches_oracle(gpu, size, a, nr, ns, its, arc):
    g, b = _problem(size, a, nr, ns, arc)
    start = np.stack([0.1 * phantom.ellipse_phantom(size, 70 + s) for s in range(ns)]).astype(np.float32)
    ref = [cpu_ref.sirt(g.angles, g.rhozero, g.deltarho, start[s], b[s], its) for s in range(ns)]
    for splits in ((0, 0), (1, 1), (2, 4)):
        x, res, done = rt.sirt_slices(_dev(g.angles), g.rhozero, g.deltarho, g.numrhos, size, ns,
                                      _dev(start).reshape(-1), _dev(b).reshape(-1), its, residuals=True,
                                      fp_split=splits[0], bp_split=splits[1])
        x = x.cpu().numpy().reshape(ns, -1)
        r = res.cpu().numpy()
        for s in range(ns):
            assert rel_l2(x[s], ref[s]) < 1e-5, splits
            fp = cpu_ref.forwardprojection(g.angles, g.rhozero, g.deltarho, g.numrhos, ref[s])
            want = np.linalg.norm(fp.astype(np.float64) - b[s]) / np.linalg.norm(b[s].astype(np.float64))
            np.testing.assert_allclose(r[s, its], want, rtol=1e-4)
        assert np.all(done.cpu().numpy() == its)


def test_small_stopping_rule(gpu):
    size, a, ns, its = 64, 60, 4, 40
    g, b = _problem(size, a, None, ns, math.pi)
    args = (_dev(g.angles), g.rhozero, g.deltarho, g.numrhos, size, ns, None, _dev(b).reshape(-1))
    _, res, _ = rt.sirt_slices(*args, its, residuals=True)
    hist = res.cpu().numpy()
    tol = float(np.sort(hist[:, 15])[1]) * 1.0001
    x, _, done = rt.sirt_slices(*args, its, tol=tol)
    stops = [next((i for i in range(its) if hist[s, i] <= tol), its) for s in range(ns)]
    assert done.cpu().numpy().tolist() == stops and len(set(stops)) > 1
    x = x.cpu().numpy().reshape(ns, -1)
    for s in range(ns):
        y, _, _ = rt.sirt_slices(*args, stops[s])
        assert np.array_equal(x[s], y.cpu().numpy().reshape(ns, -1)[s])


def test_small_barrier_timeout_is_reported(gpu):
    """A barrier that waits for a block that never comes gives up after the limit
    and the next sync reports it; the context then solves as before."""
    g, b = _problem(64, 60, None, 1, math.pi)
    args = (_dev(g.angles), g.rhozero, g.deltarho, _dev(np.zeros(64 * 64, np.float32)), _dev(b[0]), 6)
    want = rt.sirt(*args).cpu().numpy()
    ctx = rt.context()
    ctx.set_barrier_limit(timeout_ns=20_000_000, missing_blocks=1)
    try:
        rt.sirt(*args)
        with pytest.raises(rt.SynkError) as e:
            ctx.sync()
        assert e.value.code == 3
    finally:
        ctx.set_barrier_limit()
    assert np.array_equal(rt.sirt(*args).cpu().numpy(), want)
    ctx.sync()
