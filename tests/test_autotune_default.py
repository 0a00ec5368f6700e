"""The autotuner times the library's own choice beside the shapes: a tuned solve is
never one that measured slower than an untuned one."""
import json

import numpy as np
import pytest

from synkrotomo_gb300 import autotune

SHAPE = dict(fp_split=2, bp_split=4, grid_blocks=-1)


def _measure(times):
    def f(c):
        f.calls.append(c)
        return times["default" if c["grid_blocks"] == 0 else "shape"]
    f.calls = []
    return f


@pytest.mark.parametrize("default,want", [(1.0, autotune.DEFAULT), (3.0, SHAPE)])
def test_the_faster_is_used(tmp_path, default, want):
    path = str(tmp_path / "t.json")
    m = _measure({"default": default, "shape": 2.0})
    c = autotune.with_default("k", autotune.choose("k", [dict(SHAPE)], m, path=path), m, path)
    assert autotune.launch_kwargs(c) == want
    assert {k: c[k] for k in SHAPE} == SHAPE and c["default_ms"] == default * 1e3
    assert autotune.load_cache(path)["k"] == c
    n = len(m.calls)
    assert autotune.with_default("k", autotune.choose("k", [dict(SHAPE)], m, path=path), m, path) == c
    assert len(m.calls) == n                       # both times came from the cache


def test_an_entry_without_the_default_is_completed(tmp_path):
    """A cache written before the default was timed."""
    path = tmp_path / "t.json"
    path.write_text(json.dumps({"k": dict(SHAPE, ms=2.0), "other": dict(SHAPE, ms=1.0)}))
    m = _measure({"default": 0.5e-3, "shape": 2.0e-3})
    c = autotune.with_default("k", autotune.choose("k", [dict(SHAPE)], m, path=str(path)), m, str(path))
    assert autotune.launch_kwargs(c) == autotune.DEFAULT and len(m.calls) == 1
    assert autotune.load_cache(str(path))["other"] == dict(SHAPE, ms=1.0)


def test_a_bare_shape_stays_a_shape():
    assert autotune.launch_kwargs(dict(SHAPE, ms=2.0)) == SHAPE


@pytest.mark.gpu
def test_tuned_solve(gpu, tmp_path):
    import torch

    from oracle import cpu_ref
    from synkrotomo_gb300 import phantom
    from synkrotomo_gb300 import runtime as rt
    g = phantom.geometry(64, 48)
    b = phantom.add_noise(cpu_ref.forwardprojection(g.angles, g.rhozero, g.deltarho, g.numrhos,
                                                    phantom.ellipse_phantom(64, 1)), 1)
    ang, bd = torch.from_numpy(g.angles).cuda(), torch.from_numpy(b).cuda()
    c = autotune.tune_sirt(ang, g.rhozero, g.deltarho, g.numrhos, 64, bd, path=str(tmp_path / "t.json"))
    x, _, _ = rt.sirt_slices(ang, g.rhozero, g.deltarho, g.numrhos, 64, 1, None, bd, 20, **autotune.launch_kwargs(c))
    ref = cpu_ref.sirt(g.angles, g.rhozero, g.deltarho, np.zeros(64 * 64, np.float32), b, 20)
    assert np.linalg.norm(x.cpu().numpy() - ref) < 1e-5 * np.linalg.norm(ref)
    assert c["default_ms"] > 0.0
