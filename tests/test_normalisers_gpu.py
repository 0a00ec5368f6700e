"""The SIRT normalisers (csrc/project.cu) where their splits end: sides that are
no multiple of a block's four rows or 32 columns, one angle over a group of 32 and
over eight groups, near-axis angles in several places of a block, one to three
candidates per pixel, a detector row that misses part of the image.  One update from zero is
C * A^T (R * b), so it shows every entry of both.

Tolerance: SIRT's parity bar against the FP32 restatement, 1e-5 relative L2."""
import math

import numpy as np
import pytest
import torch

from oracle import cpu_ref
from synkrotomo_gb300 import runtime as rt
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,a,dr,extra,turns", [
    (2, 1, 1.0, 0, 0.5),
    (34, 33, 1.0, 0, 0.5),
    (66, 257, 1.0, 1, 0.5),
    (98, 24, 1.0, 0, 3.0),       # every eighth angle along an axis
    (130, 40, 1.0, -40, 0.5),
    (62, 65, 0.5, 0, 0.5),
    (62, 31, 1.5, 2, 0.5),
])
def test_one_update(gpu, size, a, dr, extra, turns):
    det = int(math.ceil(size * math.sqrt(2.0) / dr)) + extra
    ang = np.linspace(0.0, 2.0 * math.pi * turns, a, endpoint=False).astype(np.float32)
    rz, d = float(np.float32(-(det - 1) / 2.0 * dr)), float(np.float32(dr))
    b = (1.0 + np.random.default_rng(size + a).random(a * det)).astype(np.float32)
    zero = np.zeros(size * size, np.float32)
    x = rt.sirt(torch.from_numpy(ang).cuda(), rz, d, torch.from_numpy(zero).cuda(), torch.from_numpy(b).cuda(), 1)
    assert rel_l2(x.cpu().numpy(), cpu_ref.sirt(ang, rz, d, zero, b, 1)) < 1e-5
