"""The TMEM loads and stores of the tensor-core kernels are .sync.aligned: all 32
lanes execute them together.  Read from the sources: between such a call and the
last warp-wide meeting before it no lane may have gone its own way (a wait that
each lane leaves by itself, a branch on the lane, a copy issued by one lane), nor
after it in the same loop body without a meeting on the way back to it."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "synkrotomo_gb300", "csrc")
CALL = re.compile(r"\b(tmem_ld_32x32|tmem_ld_32x8|tmem_zero32)\(")
MEET = re.compile(r"__syncwarp\(\)|__all_sync\(|__syncthreads\(\)")
APART = re.compile(r"mbar_wait\(|\blane == 0\b|\bmover\b|elect_one\(\)|!rvalid")


def _kernels(src):
    """Bodies of the __global__ functions, comments removed and waits whose result
    the whole warp shares (__all_sync) folded into the meeting."""
    src = re.sub(r"//[^\n]*", "", src)
    out, pos = [], 0
    while (i := src.find("__all_sync(", pos)) >= 0:
        depth, j = 1, i + len("__all_sync(")
        while depth:
            depth += {"(": 1, ")": -1}.get(src[j], 0)
            j += 1
        out.append(src[pos:i] + "__all_sync()")
        pos = j
    src = "".join(out) + src[pos:]
    for m in re.finditer(r"__global__", src):
        i = src.index("{", m.end())
        depth, j = 0, i
        while True:
            depth += {"{": 1, "}": -1}.get(src[j], 0)
            j += 1
            if depth == 0:
                break
        yield src[i:j]


def _loop_body(body, at):
    """The innermost braced for body around `at`, as (start, end), else the kernel's."""
    depth, i = 0, at
    while i > 0:
        i -= 1
        depth += {"}": 1, "{": -1}.get(body[i], 0)
        if depth < 0:
            if re.search(r"for \([^{}]*\)\s*$", body[:i]):
                break
            depth = 0
    else:
        return 0, len(body)
    depth, j = 0, i
    while True:
        depth += {"{": 1, "}": -1}.get(body[j], 0)
        j += 1
        if depth == 0:
            return i, j


@pytest.mark.parametrize("name", ["conv_rows.cu", "conv_wgrad.cu", "umma_gemm.cu"])
def test_tmem_accesses_follow_a_meeting_of_the_warp(name):
    with open(os.path.join(CSRC, name)) as f:
        bodies = list(_kernels(f.read()))
    seen = 0
    for body in bodies:
        for m in CALL.finditer(body):
            seen += 1
            meets = [x.end() for x in MEET.finditer(body, 0, m.start())]
            assert meets, (name, m.group(1))
            apart = APART.search(body, meets[-1], m.start())
            assert apart is None, (name, m.group(1), body[apart.start():m.end()])
            beg, end = _loop_body(body, m.start())
            last = max((x.end() for x in APART.finditer(body, m.end(), end)), default=None)
            if last is not None:         # on the way back to the call: a meeting after it, or before the call in the body
                assert MEET.search(body, last, end) or MEET.search(body, beg, m.start()), (name, m.group(1), body[beg:end])
    assert seen
