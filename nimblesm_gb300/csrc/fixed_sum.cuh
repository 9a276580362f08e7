// The sum of up to eight FP64 numbers in 64-bit fixed point.
//
// An FP64 addition takes a warp 64 clocks of a quarter of an SM, an integer
// instruction one or two.  Aligned to the largest of them, with the leading
// bit of that at bit 59, eight numbers add up without overflow, each cut below
// 2^-59 of the largest's power of two, and the sum is rounded once: the error is
// below 8 2^-59 of that power of two plus half a unit of the sum.  FP64 additions
// round every partial sum at 2^-53 of it and are up to 80 times further off,
// also where the large terms nearly cancel, as they do at a node near
// equilibrium (tests/fixed_sum_bound_check.cc).  They are the closer ones where
// large terms cancel exactly and before smaller ones are added: of 1, -1 and
// 1e-3 they leave 1e-3, the fixed point 1e-3 (1 - 8.5e-16).  About 14 integer
// instructions per number and one conversion in place of seven additions.
#pragma once

#include <cmath>
#include <cstring>

#include "hex_fixed.cuh"

namespace nsm {
namespace fx {

#define NSM_HD __host__ __device__ __forceinline__

NSM_HD unsigned high_word(double x)
{
#ifdef __CUDA_ARCH__
  return (unsigned)__double2hiint(x);
#else
  u64 b;
  memcpy(&b, &x, 8);
  return (unsigned)(b >> 32);
#endif
}
NSM_HD unsigned low_word(double x)
{
#ifdef __CUDA_ARCH__
  return (unsigned)__double2loint(x);
#else
  u64 b;
  memcpy(&b, &x, 8);
  return (unsigned)b;
#endif
}

// x[0] + ... + x[7], zeros for the ones that are not there.  An infinity, a
// NaN, or nothing above 2^-959: FP64 additions in order (all of them zero: +0).
NSM_HD double sum8(const double x[8])
{
  unsigned most = 0;
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const unsigned h = high_word(x[j]) & 0x7fffffffu;
    most             = h > most ? h : most;
  }
  const unsigned E = most >> 20;  // biased exponent of the largest
  if (E - 64u > 0x7f0u - 64u) {
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < 8; j++) s += x[j];
    return s;
  }
  u64 s = 0;
#pragma unroll
  for (int j = 0; j < 8; j++) s += (u64)to_fixed(high_word(x[j]), low_word(x[j]), (int)E + 4);
  const double d = (double)(i64)s;  // * 2^(E - 1082)
#ifdef __CUDA_ARCH__
  return s == 0 ? 0.0 : __hiloint2double(__double2hiint(d) + (((int)E - 1082) << 20), __double2loint(d));
#else
  return ldexp(d, (int)E - 1082);
#endif
}

#undef NSM_HD

}  // namespace fx
}  // namespace nsm
