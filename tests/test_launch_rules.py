"""The particle loops' waits by batch size (launch_rules.h, compiled for the
host): the rules apply while a tuning key is at its default, and any other
value is taken as it is at every size."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "xdg_gb300", "csrc")
SMS = 152
FULL = SMS * 16 * 32

WRAP = r"""
#include "launch_rules.h"
extern "C" int flush_wait(int key, int event_wait, int mixed, int64_t n, int sms) {
  return xdgcu::particle_flush_wait(key, event_wait, mixed != 0, n, sms);
}
extern "C" int event_wait(int key, int mixed, int64_t n, int sms) {
  return xdgcu::transport_event_wait(key, mixed != 0, n, sms);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = str(tmp_path_factory.mktemp("rules"))
    src, so = os.path.join(d, "w.cpp"), os.path.join(d, "librules.so")
    with open(src, "w") as f:
        f.write(WRAP)
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-fPIC", "-shared", "-I", CSRC,
                        src, "-o", so], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    L = ctypes.CDLL(so)
    L.flush_wait.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_int64, ctypes.c_int]
    L.event_wait.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_int64, ctypes.c_int]
    return L


SIZES = [1, 6000, FULL - 1, FULL, 8 * FULL - 1, 8 * FULL, 10_000_000]


def test_set_values_are_kept(lib):
    for n in SIZES:
        for mixed in (0, 1):
            for v in [1, 2, 3, 5, 11, 16, 32]:
                assert lib.flush_wait(v, 20, mixed, n, SMS) == v
                assert lib.event_wait(v, mixed, n, SMS) == v


def test_defaults_by_batch(lib):
    assert [lib.event_wait(4, 1, n, SMS) for n in SIZES] == [1, 1, 1, 4, 4, 8, 8]
    assert [lib.event_wait(4, 0, n, SMS) for n in SIZES] == [1, 1, 1, 4, 4, 4, 4]
    assert [lib.flush_wait(4, 20, 1, n, SMS) for n in SIZES] == [4, 4, 4, 12, 12, 12, 12]
    assert [lib.flush_wait(4, 20, 0, n, SMS) for n in SIZES] == [4] * 7


def test_waits_leave_a_lane(lib):
    """Lanes that wait for their event and for a drain are at most a warp."""
    for e in range(1, 33):
        w = lib.flush_wait(4, e, 1, FULL, SMS)
        assert w == 4 or (e + w <= 32 and w <= 12)
