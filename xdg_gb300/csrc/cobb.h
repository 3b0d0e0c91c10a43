// cobb.h -- oriented boxes of closest's tree nodes.
//
// A child of an inner node gets three slabs  |a_i . x - d_i| <= h_i  that hold
// every triangle below it.  With the rows a_i as a matrix A of spectral norm
// at most 1, any x inside them and any point p satisfy
//   |p - x| >= |A (p - x)| >= sqrt(sum_i max(|a_i . p - d_i| - h_i, 0)^2),
// a lower bound of the distance that follows the surface: along a smooth
// surface the box is as thin as the patch is flat, where an axis-aligned box
// reaches out by the patch's size times its tilt.  From outside a sphere of
// 81,920 triangles 87 axis-aligned leaf boxes are within the distance of the
// nearest triangle, most of them far from it.
//
// The rows are any orthonormal triple (to FP64 rounding), scaled by 1 - 16 u and rounded
// to FP32 (u = 2^-24; the rounding adds at most 2 u to the norm, so it stays
// below 1); d_i and h_i are taken against the rounded row, from FP64 dot
// products of the vertices (each within 4 eps |a_i||v|), with h_i rounded up.
// So the slabs hold whatever the choice of the axes; the axes only decide
// how tight they are.
#pragma once

#include <math.h>

#ifndef __CUDACC__
#define XDG_COBB_HD inline
#else
#define XDG_COBB_HD __host__ __device__ inline
#endif

namespace xdgcu {

// Two axes normal to the unit vector n and to each other.
XDG_COBB_HD void obb_tangents(const float n[3], float t[3], float b[3]) {
  const float ax = fabsf(n[0]), ay = fabsf(n[1]), az = fabsf(n[2]);
  float e[3] = {0.0f, 0.0f, 0.0f};
  e[ax <= ay ? (ax <= az ? 0 : 2) : (ay <= az ? 1 : 2)] = 1.0f;
  t[0] = n[1] * e[2] - n[2] * e[1];
  t[1] = n[2] * e[0] - n[0] * e[2];
  t[2] = n[0] * e[1] - n[1] * e[0];
  const float l = 1.0f / sqrtf(t[0] * t[0] + t[1] * t[1] + t[2] * t[2]);
  for (int k = 0; k < 3; ++k) t[k] *= l;
  b[0] = n[1] * t[2] - n[2] * t[1];
  b[1] = n[2] * t[0] - n[0] * t[2];
  b[2] = n[0] * t[1] - n[1] * t[0];
}

// The axes of a cluster from the sum `nsum` of its triangles' area normals
// and the sum `area` of their lengths: the mean normal and two tangents, or
// the coordinate axes where the normals cancel (a closed or folded patch).
XDG_COBB_HD void obb_axes(const float nsum[3], float area, float row[3][3]) {
  const float l = sqrtf(nsum[0] * nsum[0] + nsum[1] * nsum[1] + nsum[2] * nsum[2]);
  for (int i = 0; i < 3; ++i)
    for (int k = 0; k < 3; ++k) row[i][k] = i == k ? 1.0f : 0.0f;
  if (l > 0.5f * area && l > 1e-30f && l < 1e18f) {
    for (int k = 0; k < 3; ++k) row[0][k] = nsum[k] / l;
    obb_tangents(row[0], row[1], row[2]);
  }
}

// Turns the two tangents so that the cluster's vertices are uncorrelated in
// their plane (sxx, sxy, syy: second moments along t, b): the half angle of
// (sxx - syy, 2 sxy).
XDG_COBB_HD void obb_turn(float sxx, float sxy, float syy, float t[3], float b[3]) {
  const float x = sxx - syy, y = 2.0f * sxy, l = sqrtf(x * x + y * y);
  if (!(l > 1e-30f && l < 1e30f)) return;
  const float c = sqrtf(fmaxf(0.5f * (1.0f + x / l), 0.0f));
  const float s = copysignf(sqrtf(fmaxf(0.5f * (1.0f - x / l), 0.0f)), y);
  for (int k = 0; k < 3; ++k) {
    const float p = c * t[k] + s * b[k], q = c * b[k] - s * t[k];
    t[k] = p;
    b[k] = q;
  }
}

// The rows a_i: the axes made orthonormal in FP64 (Gram-Schmidt), scaled by
// 1 - 16 u and rounded; the coordinate axes where that fails.
XDG_COBB_HD void obb_rows32(const float axes[3][3], float out[3][3]) {
  const double u = 5.9604644775390625e-08;
  double r[3][3];
  bool ok = true;
  for (int i = 0; i < 2; ++i) {
    for (int k = 0; k < 3; ++k) r[i][k] = axes[i][k];
    if (i == 1) {
      const double p = r[0][0] * r[1][0] + r[0][1] * r[1][1] + r[0][2] * r[1][2];
      for (int k = 0; k < 3; ++k) r[1][k] -= p * r[0][k];
    }
    const double l = sqrt(r[i][0] * r[i][0] + r[i][1] * r[i][1] + r[i][2] * r[i][2]);
    ok = ok && l > 0.5 && l < 2.0;
    for (int k = 0; k < 3; ++k) r[i][k] /= l;
  }
  r[2][0] = r[0][1] * r[1][2] - r[0][2] * r[1][1];
  r[2][1] = r[0][2] * r[1][0] - r[0][0] * r[1][2];
  r[2][2] = r[0][0] * r[1][1] - r[0][1] * r[1][0];
  for (int i = 0; i < 3; ++i)
    for (int k = 0; k < 3; ++k)
      out[i][k] = (float)((ok ? r[i][k] : (i == k ? 1.0 : 0.0)) * (1.0 - 16.0 * u));
}

// a . v for the rounded row
XDG_COBB_HD double obb_dot(const float a[3], const double* v) {
  return (double)a[0] * v[0] + (double)a[1] * v[1] + (double)a[2] * v[2];
}

// The slab of the products lo .. hi: its middle d and half width h, rounded
// so that it holds them.  vmax bounds the vertices' coordinates.
XDG_COBB_HD void obb_slab(double lo, double hi, double vmax, float* d, float* h) {
  const float mid = (float)(0.5 * (lo + hi));
  const double w = fmax(hi - (double)mid, (double)mid - lo) + 1e-14 * vmax;
  float up = (float)w;
  if ((double)up < w) up = nextafterf(up, INFINITY);
  *d = mid;
  *h = up;
}

}  // namespace xdgcu
