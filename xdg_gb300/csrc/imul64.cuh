// imul64.cuh -- binary64 products on the integer pipes.
//
// GB300 runs FP64 at 1/64 of its FP32 rate: one FP64 warp instruction holds a
// scheduler's FP64 unit for 39 ns, whatever the number of active lanes (1 to
// 32 the same), and a predicated-off one costs as much.  The integer pipes
// beside it are all but idle in the kernels that wait for it.  mul_int is the
// IEEE product, rounded to nearest even, in about thirty integer
// instructions: 29 ns per warp and scheduler, issued beside the FP64 unit
// (measured with 8 independent products and 8 FP64 additions per iteration,
// 4 warps per scheduler: 314 ns against 623 with the FP64 product).  A chain
// of products and sums in which the products run here and the sums on the
// FP64 unit so takes half the time, bit for bit the same.
//
// Domain: each operand is zero or normal, and the product is zero or a
// normal number (it neither overflows nor underflows).  in_range() is the test
// the callers make on their inputs: for values that are zero or of magnitude
// 2^-150 .. 2^150, every product in the Plucker coordinates, barycentric
// weights and hit distances of plucker.h:45-161 stays inside (the smallest
// non-zero intermediate is above 2^-900: a difference of two doubles is zero
// or a multiple of the smaller one's last place, and a coordinate that is
// not snapped to zero is at least 20 eps).
//
// Host-compilable, so that it can be checked against the host's own products.
#pragma once

#include <cstdint>
#include <cstring>

#ifndef __CUDACC__
#define XDG_HD inline
#else
#define XDG_HD __host__ __device__ __forceinline__
#endif

namespace xdgcu {

struct W64 {
  uint32_t lo, hi;
};

XDG_HD W64 words(double x) {
  W64 w;
#ifdef __CUDA_ARCH__
  w.lo = (uint32_t)__double2loint(x);
  w.hi = (uint32_t)__double2hiint(x);
#else
  uint64_t b;
  std::memcpy(&b, &x, 8);
  w.lo = (uint32_t)b;
  w.hi = (uint32_t)(b >> 32);
#endif
  return w;
}

XDG_HD double from_words(uint32_t lo, uint32_t hi) {
#ifdef __CUDA_ARCH__
  return __hiloint2double((int)hi, (int)lo);
#else
  const uint64_t b = ((uint64_t)hi << 32) | lo;
  double x;
  std::memcpy(&x, &b, 8);
  return x;
#endif
}

// upper word of (hi:lo) << s, s in 0..31
XDG_HD uint32_t shl_hi(uint32_t lo, uint32_t hi, uint32_t s) {
#ifdef __CUDA_ARCH__
  return __funnelshift_l(lo, hi, s);
#else
  return s ? (hi << s) | (lo >> (32u - s)) : hi;
#endif
}

// a * b rounded to nearest even (see the domain above).  The significand of a
// is shifted to 64 bits and b's left at 53, so the product's upper 64 bits
// hold the result's 52 or 53 leading bits, and the word below them its
// round bit and, with the lowest word, the sticky bits.
XDG_HD double mul_int(double a, double b) {
  const W64 x = words(a), y = words(b);
  const uint32_t ex = x.hi & 0x7ff00000u, ey = y.hi & 0x7ff00000u;
  const uint32_t ah = shl_hi(x.lo, x.hi, 11) | 0x80000000u, al = x.lo << 11;
  const uint32_t bh = (y.hi & 0xfffffu) | 0x100000u, bl = y.lo;
  const uint64_t p0 = (uint64_t)al * bl;
  const uint64_t p1 = (uint64_t)al * bh + (p0 >> 32);
  const uint64_t p2 = (uint64_t)ah * bl + (uint32_t)p1;
  const uint64_t hi = (uint64_t)ah * bh + ((p1 >> 32) + (p2 >> 32));
  const uint32_t h1 = (uint32_t)(hi >> 32), h0 = (uint32_t)hi, l1 = (uint32_t)p2;
  const uint32_t n = ((h1 >> 20) & 1u) ^ 1u;  // 1: only 52 bits, shift left once
  const uint32_t m1 = shl_hi(h0, h1, n), m0 = shl_hi(l1, h0, n), rest = l1 << n;
  // rounds up when rest > half, or at half when a lower bit or the last place
  // is set: the carry of rest + (half, or half - 1)
  const uint32_t half = ((uint32_t)p0 | (m0 & 1u)) != 0u ? 0x80000000u : 0x7fffffffu;
  const uint64_t carry = ((uint64_t)rest + half) >> 32;
  const uint32_t sign = (x.hi ^ y.hi) & 0x80000000u;
  // m1 carries the leading bit, which adds one to the exponent field
  const uint32_t e = ex + ey - ((1023u + n) << 20) + sign;
  const uint64_t r = (((uint64_t)(m1 + e) << 32) | m0) + carry;
  const bool zero = ex == 0u || ey == 0u;
  return from_words(zero ? 0u : (uint32_t)r, zero ? sign : (uint32_t)(r >> 32));
}

// x is +-0 or 2^-P <= |x| < 2^P
template <int P>
XDG_HD bool in_range_of(double x) {
  const W64 w = words(x);
  const uint32_t h = w.hi & 0x7fffffffu;
  return h - ((1023u - P) << 20) < ((2u * P) << 20) || (h | w.lo) == 0u;
}
XDG_HD bool in_range(double x) { return in_range_of<150>(x); }

}  // namespace xdgcu
