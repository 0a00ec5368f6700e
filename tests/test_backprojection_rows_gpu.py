"""The backprojector's rows of detector pairs (csrc/bp_tile.cuh, PairRows and
bp_chunk_pair) over the forms that choose its variants: one to four candidates
per pixel, split and whole angle sets, padded and clamped windows, an angle
without a direction, more angles than a grid's second dimension.

Tolerance: the projectors' parity bar, 1e-5 relative L2, against the 64-bit
oracle (few angles at deltarho 0.5 and 1186 x 1186 pixels take the FP32
restatement itself 1.07e-5 away from it); every 37th row of the large images."""
import math

import numpy as np
import pytest
import torch

from oracle import cpu_ref
from oracle import fut_ref as F
from synkrotomo_gb300 import runtime as rt
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


def _case(size, a, dr, extra, shift):
    det = int(math.ceil(size * math.sqrt(2.0) / dr)) + extra
    ang = (0.01 + np.linspace(0.0, math.pi, a, endpoint=False)).astype(np.float32)
    rz = float(np.float32((-(det - 1) / 2.0 + shift) * dr))
    y = np.random.default_rng(size * a + det).random(a * det).astype(np.float32)
    return ang, rz, float(np.float32(dr)), y


def _run(ang, rz, dr, size, y):
    return rt.backprojection(torch.from_numpy(ang).cuda(), rz, dr, size, torch.from_numpy(y).cuda()).cpu().numpy()


@pytest.mark.parametrize("size,a,dr,extra,shift", [
    (2, 1, 1.0, 0, 0),          # the smallest call: all but four pixels of a tile lie outside
    (34, 17, 1.0, 0, 0),        # two angle parts, an odd angle over, padding of 29 pixels
    (130, 71, 1.0, 1, 0),       # eight parts, 32-row tiles
    (226, 257, 1.0, 0, 0),      # eight pixels per thread, a second chunk of one angle
    (1186, 258, 1.0, 0, 0),     # whole angle sets
    (130, 71, 1.0, -60, 0),     # detectors that miss the corners: padding
    (322, 40, 1.0, -300, 0),    # more than the padding: clamped
    (322, 40, 1.0, 0, 400.25),  # the row beside the image, off the grid
    (98, 260, 1.5, 0, 0),       # one candidate
    (98, 33, 0.8, 7, 0),        # two
    (1186, 20, 0.5, 0, 0.3),    # three, whole angle sets
    (98, 61, 0.5, -120, 0),     # three, clamped
    (98, 300, 0.4, 0, 0),       # four
    (98, 61, 0.3, 0, 0),        # five: the plain rows
])
def test_against_oracle(gpu, size, a, dr, extra, shift):
    ang, rz, d, y = _case(size, a, dr, extra, shift)
    rows = np.arange(0, size, 37 if size > 1000 else 1)
    out = _run(ang, rz, d, size, y).reshape(size, size)[rows]
    assert rel_l2(out.reshape(-1), np.asarray(F.backprojection_rows(ang, rz, d, size, y, rows)).reshape(-1)) < 1e-5


@pytest.mark.parametrize("dr", [1.0, 0.5])
def test_angle_without_direction_adds_nothing(gpu, dr):
    ang, rz, d, y = _case(66, 40, dr, 0, 0)
    bad = np.insert(ang, 20, np.float32(np.nan))
    rows = np.insert(y.reshape(40, -1), 20, 1.0, axis=0).reshape(-1)
    assert rel_l2(_run(bad, rz, d, 66, rows), _run(ang, rz, d, 66, y)) < 1e-6


def test_more_angles_than_a_grid_dimension(gpu):
    ang, rz, d, y = _case(16, 65537, 1.0, 0, 0)
    assert rel_l2(_run(ang, rz, d, 16, y), cpu_ref.backprojection(ang, rz, d, 16, y)) < 1e-5
