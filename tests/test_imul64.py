"""The integer product of imul64.cuh equals the IEEE product bit for bit on its
domain (operands zero or normal, product zero or normal), and in_range() is
what its comment says.  The header is the product's own, compiled for the
host; the IEEE products are the host's.  Both sides are exact roundings of the
same real number, so nothing but equality is accepted."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "xdg_gb300", "csrc")

WRAP = r"""
#include "imul64.cuh"
extern "C" void products(const double* a, const double* b, int64_t n, double* out) {
  for (int64_t i = 0; i < n; ++i) out[i] = xdgcu::mul_int(a[i], b[i]);
}
extern "C" void ranges(const double* a, int64_t n, uint8_t* out) {
  for (int64_t i = 0; i < n; ++i) out[i] = xdgcu::in_range(a[i]) ? 1 : 0;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = str(tmp_path_factory.mktemp("imul"))
    src, so = os.path.join(d, "w.cpp"), os.path.join(d, "libimul.so")
    with open(src, "w") as f:
        f.write(WRAP)
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-ffp-contract=off", "-fPIC",
                        "-shared", "-I", CSRC, src, "-o", so], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(so)


def _operands(rng, n, kind):
    b = rng.integers(0, 2**63, n, dtype=np.uint64) << np.uint64(1)
    b |= rng.integers(0, 2, n, dtype=np.uint64)
    mant = b & np.uint64((1 << 52) - 1)
    spread = 300 if kind == "wide" else 3
    e = (1023 + rng.integers(-spread, spread + 1, n)).astype(np.uint64)
    if kind == "short":      # short significands: exact products and ties
        keep = rng.integers(0, 53, n).astype(np.uint64)
        mant = (mant >> keep) << keep
    if kind == "edge":       # long runs of ones or zeros: carries across the words
        run = rng.integers(0, 52, n).astype(np.uint64)
        ones = ((np.uint64(1) << np.uint64(52)) - np.uint64(1)) ^ ((np.uint64(1) << run) - np.uint64(1))
        mant = np.where(rng.random(n) < 0.5, ones, (np.uint64(1) << run) - np.uint64(1))
        mant ^= rng.integers(0, 2, n, dtype=np.uint64)
    x = ((b >> np.uint64(63) << np.uint64(63)) | (e << np.uint64(52)) | mant).view(np.float64).copy()
    zero = rng.random(n) < 0.02
    x[zero] = np.where(rng.random(zero.sum()) < 0.5, 0.0, -0.0)
    return x


@pytest.mark.parametrize("ka", ["wide", "near", "short", "edge"])
@pytest.mark.parametrize("kb", ["wide", "near", "short", "edge"])
def test_products(lib, ka, kb):
    rng = np.random.default_rng([ord(ka[0]), ord(kb[0])])
    n = 300_000
    a, b = _operands(rng, n, ka), _operands(rng, n, kb)
    out = np.empty(n)
    lib.products(a.ctypes.data_as(ctypes.c_void_p), b.ctypes.data_as(ctypes.c_void_p),
                 ctypes.c_int64(n), out.ctypes.data_as(ctypes.c_void_p))
    want = a * b
    bad = np.nonzero(out.view(np.uint64) != want.view(np.uint64))[0]
    assert len(bad) == 0, [(a[k].hex(), b[k].hex(), want[k].hex(), out[k].hex()) for k in bad[:3]]


def test_in_range(lib):
    lo, hi = 2.0 ** -150, 2.0 ** 150
    x = np.array([0.0, -0.0, lo, -lo, np.nextafter(lo, 0), np.nextafter(hi, 0), hi, -hi, 1.0, 5e-324,
                  1e-310, np.inf, -np.inf, np.nan, 1e300])
    want = np.array([1, 1, 1, 1, 0, 1, 0, 0, 1, 0, 0, 0, 0, 0, 0], dtype=np.uint8)
    out = np.empty(len(x), dtype=np.uint8)
    lib.ranges(x.ctypes.data_as(ctypes.c_void_p), ctypes.c_int64(len(x)),
               out.ctypes.data_as(ctypes.c_void_p))
    assert np.array_equal(out, want)
