"""The time limit of the one-launch SIRT engine's grid barrier (csrc/poll_limit.cuh),
evaluated on the host: polling uses it up, time in which the GPU ran another process
does not."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = """
#include "poll_limit.cuh"
// the look at which a wait of `limit` ns gives up, -1: never within n looks
extern "C" int gives_up(const unsigned long long *now, int n, unsigned long long limit) {
    synk::PollLimit l;
    l.start(now[0]);
    for (int i = 1; i < n; ++i)
        if (l.over(now[i], limit)) return i;
    return -1;
}
"""


@pytest.fixture(scope="module")
def gives_up(tmp_path_factory):
    d = tmp_path_factory.mktemp("poll")
    src, so = d / "poll.cpp", d / "poll.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "synkrotomo_gb300", "csrc"), str(src), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))

    def call(now, limit):
        return lib.gives_up((ctypes.c_ulonglong * len(now))(*now), len(now), ctypes.c_ulonglong(limit))
    return call


LOOK = 45_000           # ns between two looks: 64 polls


def test_polling_runs_out_at_the_limit(gives_up):
    now = [LOOK * i for i in range(1000)]
    assert gives_up(now, 20_000_000) == 20_000_000 // LOOK + 1
    assert gives_up(now, 1_000) == 1
    assert gives_up(now, 60_000_000) == -1


@pytest.mark.parametrize("gap", [3_000_000_000, 60_000_000_000])
def test_a_preempted_wait_goes_on(gives_up, gap):
    """A few looks, a gap longer than the limit, a few more looks."""
    now = [LOOK * i for i in range(10)] + [gap + LOOK * i for i in range(10, 20)]
    assert gives_up(now, 2_000_000_000) == -1


def test_many_slices_count_as_what_was_polled(gives_up):
    """Alternating 2 ms of polling and 2 ms away: 20 ms polled are over after 40 ms at the latest."""
    now, t = [0], 0
    for _ in range(40):
        for _ in range(2_000_000 // LOOK):
            t += LOOK
            now.append(t)
        t += 2_000_000
        now.append(t)
    i = gives_up(now, 20_000_000)
    assert i > 0 and 20_000_000 < now[i] <= 40_000_000
