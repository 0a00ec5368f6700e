"""The word that the stopping rule's host check reads back (csrc/poll_word.cuh): a
call ends early on its own count only, not on one that a call on another stream of
the same context left in the pinned word."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def done(tmp_path_factory):
    d = tmp_path_factory.mktemp("word")
    src, so = d / "word.cpp", d / "word.so"
    src.write_text('#include "poll_word.cuh"\n'
                   'extern "C" int done(unsigned long long w, int call) { return synk::poll_done(w, call); }\n')
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "synkrotomo_gb300", "csrc"), str(src), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    return lambda count, by, call: bool(lib.done(ctypes.c_ulonglong((count << 32) | by), call))


def test_own_count(done):
    assert done(0, 7, 7)
    assert not done(3, 7, 7)
    assert done(0, 0x7fffffff, 0x7fffffff)


def test_another_calls_count(done):
    assert not done(0, 6, 7)
    assert not done(0, 0, 7)
    assert not done(1, 6, 7)


@pytest.mark.gpu
def test_two_streams_with_their_own_stops(gpu):
    """A stack that stops early and one that never does, in turn on two streams of one
    context: both are what they are alone."""
    import torch

    from synkrotomo_gb300 import phantom
    from synkrotomo_gb300 import runtime as rt
    calls = []
    for size, angles, ns, its, tol in ((256, 400, 1, 60, 0.2), (128, 400, 4, 80, 1e-30)):
        g = phantom.geometry(size, angles)
        ang = torch.from_numpy(g.angles).cuda()
        b = torch.cat([rt.forwardprojection(ang, g.rhozero, 1.0, g.numrhos,
                                            torch.from_numpy(phantom.ellipse_phantom(size, s)).cuda())
                       for s in range(ns)])
        calls.append(((ang, g.rhozero, 1.0, g.numrhos, size, ns, None, b, its), tol))
    alone = [rt.sirt_slices(*a, tol=t) for a, t in calls]
    torch.cuda.synchronize()
    assert int(alone[0][2].max()) < 60 and int(alone[1][2].min()) == 80
    streams = [torch.cuda.Stream() for _ in calls]
    for _ in range(5):
        got = []
        for s, (a, t) in zip(streams, calls):
            with torch.cuda.stream(s):
                got.append(rt.sirt_slices(*a, tol=t))
        torch.cuda.synchronize()
        for (x, _, d), (y, _, e) in zip(got, alone):
            assert torch.equal(x, y) and torch.equal(d, e)
