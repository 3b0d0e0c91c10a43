"""The oriented boxes of closest's tree nodes (cobb.h): the FP32 lower bound
`closest_children` takes from a child's three slabs never exceeds the distance
from the point to a triangle of the cluster (closest.cpp:54-183 through the
oracle).  The rows, slabs and roundings come from the product's own header,
compiled for the host; the kernel's FP32 evaluation (point rounded, three
FMAs a row, squares, root) is restated in numpy.  Clusters: flat and curved
patches, soups, needles and single degenerate triangles, sizes 1e-4..1e2 up to
1e6 from the origin; points near, on and far from them.  The bound is proved
in the header and the kernel's comment, so no tolerance is allowed."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from fp32_emul import U, fma32

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "xdg_gb300", "csrc")

WRAP = r"""
#include <cstdint>
#include "cobb.h"
using namespace xdgcu;
// v: 9 doubles per triangle; out: 3 x (row, middle, half width)
extern "C" void obb(const double* v, int64_t n, float* out) {
  float ns[3] = {0, 0, 0}, area = 0, vm[3] = {0, 0, 0};
  double vmax = 0;
  for (int64_t j = 0; j < n; ++j) {
    float w[9], a[3], b[3];
    for (int k = 0; k < 9; ++k) {
      w[k] = (float)v[9 * j + k] - (float)v[k % 3];
      vmax = fmax(vmax, fabs(v[9 * j + k]));
    }
    for (int k = 0; k < 3; ++k) { a[k] = w[3 + k] - w[k]; b[k] = w[6 + k] - w[k]; }
    const float c[3] = {a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]};
    for (int k = 0; k < 3; ++k) ns[k] += c[k];
    area += sqrtf(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]);
    for (int k = 0; k < 9; ++k) vm[k % 3] += w[k] / (3.0f * n);
  }
  float row[3][3], s[3] = {0, 0, 0}, a[3][3];
  obb_axes(ns, area, row);
  for (int64_t k = 0; k < 3 * n; ++k) {
    float x = 0, y = 0;
    for (int i = 0; i < 3; ++i) {
      const float w = (float)v[3 * k + i] - (float)v[i] - vm[i];
      x += w * row[1][i];
      y += w * row[2][i];
    }
    s[0] += x * x; s[1] += x * y; s[2] += y * y;
  }
  obb_turn(s[0], s[1], s[2], row[1], row[2]);
  obb_rows32(row, a);
  for (int i = 0; i < 3; ++i) {
    double lo = INFINITY, hi = -INFINITY;
    for (int64_t k = 0; k < 3 * n; ++k) {
      const double x = obb_dot(a[i], v + 3 * k);
      lo = fmin(lo, x);
      hi = fmax(hi, x);
    }
    for (int k = 0; k < 3; ++k) out[5 * i + k] = a[i][k];
    obb_slab(lo, hi, vmax, out + 5 * i + 3, out + 5 * i + 4);
  }
}
"""
F = np.float32


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = str(tmp_path_factory.mktemp("obb"))
    src, so = os.path.join(d, "w.cpp"), os.path.join(d, "libobb.so")
    with open(src, "w") as f:
        f.write(WRAP)
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-ffp-contract=off", "-fPIC",
                        "-shared", "-I", CSRC, src, "-o", so], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(so)


def _cluster(rng, kind):
    scale, size = 10.0 ** rng.choice([0.0, 2.0, 4.0, 6.0]), 10.0 ** rng.uniform(-4, 2)
    c = rng.uniform(-1, 1, 3) * scale
    n = int(rng.choice([1, 2, 3, 7, 30]))
    if kind == "patch":  # triangles of a curved patch with a random frame
        q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        xy = rng.uniform(-1, 1, (n, 1, 2)) + 0.3 * rng.normal(size=(n, 3, 2))
        z = rng.choice([0.0, 0.01, 0.3]) * (xy ** 2).sum(2)
        t = np.concatenate([xy, z[:, :, None]], 2) @ q.T
    elif kind == "soup":
        t = rng.normal(size=(n, 3, 3))
    else:                # needles, some of them degenerate
        d = rng.normal(size=(n, 1, 3))
        t = rng.normal(size=(n, 1, 3)) + rng.normal(size=(n, 3, 1)) * d
        t = t + rng.choice([0.0, 1e-12, 1e-6]) * rng.normal(size=(n, 3, 3))
    return c + size * t, size


@pytest.mark.parametrize("kind", ["patch", "soup", "needle"])
def test_lower_bound(lib, oracle, kind):
    rng = np.random.default_rng(len(kind))
    used = 0
    for _ in range(400):
        tri, size = _cluster(rng, kind)
        v = np.ascontiguousarray(tri.reshape(-1, 9))
        out = np.zeros((3, 5), dtype=np.float32)
        lib.obb(v.ctypes.data_as(ctypes.c_void_p), ctypes.c_int64(len(v)),
                out.ctypes.data_as(ctypes.c_void_p))
        w = rng.dirichlet([1, 1, 1], 12)
        p = (w[:, :, None] * tri[rng.integers(0, len(tri), 12)]).sum(1)
        p += rng.normal(size=p.shape) * size * 10.0 ** rng.uniform(-9, 2, (12, 1))
        M = F(np.abs(v).max() * (1 + 1e-6))
        p32 = p.astype(np.float32)
        margin = F(48) * F(U) * (np.abs(p32).max(1) + M)
        s2 = np.zeros(12, dtype=np.float32)
        for r in out:
            one = np.ones(12, dtype=np.float32)
            s = fma32(one * r[2], p32[:, 2], -one * r[3])
            s = fma32(one * r[0], p32[:, 0], fma32(one * r[1], p32[:, 1], s))
            e = np.maximum(np.abs(s) - r[4], F(0))
            s2 = fma32(e, e, s2)
        lb = np.sqrt(s2) * F(1 - 8 * U) - margin
        foot = np.array([[oracle.closest_on_tri(t, q) for t in v] for q in p])
        d = np.linalg.norm(foot - p[:, None], axis=2)
        d = np.where(np.isfinite(d), d, np.inf).min(1)
        assert (lb.astype(np.float64) <= d).all()
        used += int((lb > 0.5 * d).sum())
    # the bound has to be worth having: within a factor two of the distance for
    # many of the points that are not on the triangles
    assert used > 400
