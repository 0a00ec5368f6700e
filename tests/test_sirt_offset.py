"""Gather offsets of the one-launch SIRT engine (csrc/sirt_offset.cuh), evaluated
on the host over every angle and pixel of geometries whose first angle lies off
the axes: the entry of detector s of angle k is 4*(k*D + s) bytes from the
residual, also for s = -1, whose neighbour, detector 0, the kernel reads.  The
kernel's base lies kSmallLead entries before the residual."""
import ctypes
import math
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# 0x4B400000: the bits of 1.5 * 2^23
SOURCE = """
#include "sirt_offset.cuh"
extern "C" void offsets(const int *k, const int *s, int n, int D, int zi, long long *out) {
    for (int i = 0; i < n; ++i)
        out[i] = (long long)synk::small_gather_offset(0x4B400000u + (unsigned)(s[i] - zi),
                                                      synk::small_row_offset(k[i], D, zi, 0x4B400000)) -
                 4 * synk::kSmallLead;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("offset")
    src, so = d / "offset.cpp", d / "offset.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "synkrotomo_gb300", "csrc"), str(src), "-o", str(so)], check=True)
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize("size,angles,det,first", [
    (128, 90, 100, 0.3),                    # detectors short of the image
    (100, 91, 142, math.radians(179.0)),    # full rows, a descending scan: lanes past the last column
    (100, 60, 142, math.radians(135.0)),
    (68, 45, 97, math.radians(179.0)),
])
def test_every_gathered_entry_is_its_detectors(lib, size, angles, det, first):
    step = -math.pi / angles if first > 3.0 else math.pi / angles
    th = first + step * np.arange(angles)
    rhozero = -(det - 1) / 2.0
    zi = int(np.rint(-rhozero))
    col = np.arange((size + 31) // 32 * 32) - size // 2 + 0.5
    row = np.arange(size) - size // 2 + 0.5
    rho = col[None, None, :] * np.cos(th)[:, None, None] - row[None, :, None] * np.sin(th)[:, None, None]
    s = np.ceil(rho - math.sqrt(0.5) - rhozero).astype(np.int32)
    k = np.broadcast_to(np.arange(angles, dtype=np.int32)[:, None, None], s.shape)
    read = (s >= -1) & (s < det)            # a candidate inside the row
    k, s = np.ascontiguousarray(k[read]), np.ascontiguousarray(s[read])
    assert np.any((k == 0) & (s == -1))
    out = np.empty(k.size, np.int64)
    ip = ctypes.POINTER(ctypes.c_int)
    lib.offsets(k.ctypes.data_as(ip), s.ctypes.data_as(ip), k.size, det, zi,
                out.ctypes.data_as(ctypes.POINTER(ctypes.c_longlong)))
    np.testing.assert_array_equal(out, 4 * (k.astype(np.int64) * det + s))
