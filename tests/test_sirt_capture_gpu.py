"""SIRT calls captured by the caller into a CUDA graph: every engine, replayed after
other host work and with other measured data, gives what a direct call gives, bit for
bit (the same kernels on the same data)."""
import gc
import math

import numpy as np
import pytest
import torch

from synkrotomo_gb300 import phantom
from synkrotomo_gb300 import runtime as rt

pytestmark = pytest.mark.gpu


def _data(size, angles, ns, seed):
    g = phantom.geometry(size, angles)
    ang = torch.from_numpy(g.angles).cuda()
    b = torch.cat([rt.forwardprojection(ang, g.rhozero, 1.0, g.numrhos,
                                        torch.from_numpy(phantom.ellipse_phantom(size, seed + s)).cuda())
                   for s in range(ns)])
    return g, ang, b


def _churn():
    """Host memory of the capturing call is used for something else."""
    gc.collect()
    return [np.random.default_rng(i).random(int(2 ** (5 + i % 12))) for i in range(400)]


@pytest.mark.parametrize("size,angles,ns,tol", [
    (64, 60, 1, 0.0),           # one cooperative launch
    (160, 180, 8, 0.0),         # interleaved slices
    (128, 400, 2, 1e-3),        # launched phases with a stopping rule
])
def test_captured_call(gpu, size, angles, ns, tol):
    g, ang, b = _data(size, angles, ns, 1)
    out = torch.empty(ns * size * size, device="cuda")
    args = (ang, g.rhozero, 1.0, g.numrhos, size, ns, None, b, 6)
    rt.sirt_slices(*args, tol=tol, out=out)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _, _, done = rt.sirt_slices(*args, tol=tol, out=out)
    for seed in (1, 5):
        keep = _churn()
        b.copy_(_data(size, angles, ns, seed)[2])
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        want, _, want_done = rt.sirt_slices(*args, tol=tol)
        assert torch.equal(out, want) and torch.equal(done, want_done)
        del keep
    rt.context().sync()


def test_captured_batch(gpu):
    probs = []
    for size, angles in ((96, 40), (64, 33), (48, 17)):
        g, ang, b = _data(size, angles, 1, size)
        probs.append(rt.Problem(ang, g.rhozero, 1.0, g.numrhos, size, b, 5))
    for grid in (0, rt.resident_blocks()):
        rt.sirt_batch(probs, grid_blocks=grid)
        want = [p.out.clone() for p in probs]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            rt.sirt_batch(probs, grid_blocks=grid)
        keep = _churn()
        for p in probs:
            p.out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(p.out, w) for p, w in zip(probs, want))
        del keep
    rt.context().sync()
