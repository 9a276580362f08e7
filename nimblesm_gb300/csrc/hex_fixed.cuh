// The hex8 element in 64-bit fixed point: the arithmetic of the FP64 form's
// fast path (element_fixed.cu).
//
// The chip's FP64 pipe takes one warp instruction per 16 clocks and SM; its
// integer pipes take one wide product (32 x 32 bits to 64) and up to four
// additions per clock (measured: DFMA 0.0625, mul.wide 1.0, IADD3 2.0 on one
// of its two pipes).  A 64 x 64 bit product kept to 64 bits is three wide
// products, so a dot product of three terms costs 9 of them and two more
// instructions (10 clocks) where three FP64 instructions cost 48, and an
// addition 2 instructions instead of 16 clocks.  Elements are well suited to fixed
// point: H = F - I, the cofactors and J are numbers near 0 or 1, and what has
// a dimension (displacement, geometry, moduli) is scaled per element or per
// material by a power of two.  Numbers carry 56 to 61 bits below the largest
// value of their kind, against FP64's 53 bits.
//
// Accuracy.  The sums and differences of the modal transforms are exact, the
// terms linear in H enter cofactors, J and stress exactly, and products are
// cut at 2^-60 (H, cofactors, J) and 2^-59 (stress over modulus) absolute.
// An FP64 evaluation rounds J at 2^-53 absolute.  Measured against extended
// precision (tests/fixed_check.cc), at a strain of 1e-3 the stress is off by
// 7e-15 of itself (FP64: 1.5e-13), the forces by 1.8e-14 (7e-14), and the same
// factors at strains from 1e-9 to 3e-2; beside a rigid displacement of the
// element's size both are 10 to 100 times closer than in FP64.
//
// That is against an FP64 evaluation's J, an error of K 2^-53: neo-Hookean
// elements of K < G / 2 (where it would be the smaller one) are not evaluated
// here.  An FP64 evaluation of an elastic element has no such absolute error;
// how its bits are kept here is said at elastic_scale.
//
// Domain.  |H| < 1/2 (Frobenius; a rotation by 20 degrees) at every point; for
// neo-Hookean elements also displacement modes below 1.375 2^60, which end at
// |H| between 0.1 and 0.3, stresses below the larger modulus past |H| = 1/8, and
// displacements within 2^26 of the element's scale; finite inputs.  The functions
// report what leaves it; the caller then evaluates the element in FP64 as a
// whole, so each element's result depends on its own inputs alone.
//
// One element is shared by four lanes, each with one edge along xi: the two
// points and two corners on its side along eta and zeta.  A lane works in
// coordinates mirrored along eta and zeta so that its side is "+" (the rows
// eta and zeta of its points' G0 are stored negated where it is "-"): all
// lanes then run the same code without a sign, and every sum over a pair of
// lanes is "own + other" or "own - other".
#pragma once

#include "nsm_common.cuh"

namespace nsm {
namespace fx {

using i64 = long long;
using u64 = unsigned long long;

#define NSM_HD __host__ __device__ __forceinline__

// A fixed-point number as two signed limbs: hi * 2^32 + lo.
struct Limbs {
  int hi, lo;
};
NSM_HD Limbs split(i64 x)
{
  const int lo = (int)x;
  return Limbs{(int)(x >> 32) + (int)((unsigned)lo >> 31), lo};
}

// a b (spelled out: the compiler takes the C++ form apart into 64-bit products
// of the limbs' parts, five times the work).  The product alone, not mad.wide:
// sums in C++ let the compiler put the additions into the products (a sum of
// three 64 x 64 bit products is 9 + 2 instructions), which it does not do for
// a chain of mad.wide: 1,513 instructions per point became 1,190 and the
// element kernel 1,105 us instead of 1,240 at 2,097,152 elements; the funnel
// shifts below gave 14 us more.  (A third addend of zero in additions of two,
// to keep them off the multiplier's pipe: 1,103 to 1,193 us.)
NSM_HD u64 mul_wide(int a, int b)
{
#ifdef __CUDA_ARCH__
  u64 d;
  asm("mul.wide.s32 %0, %1, %2;" : "=l"(d) : "r"(a), "r"(b));
  return d;
#else
  return (u64)((i64)a * b);
#endif
}

// Sum of products / 2^(64 - k), truncated: the products of high limbs and the
// mixed ones (the product of low limbs is below a quarter of the last place
// for k = 0).  Both sums start from the zero register; a rounding constant
// would cost two moves a sum.
template <int k>
struct Acc {
  u64 hh, mid;
  NSM_HD Acc() : hh(0), mid(0) {}
  NSM_HD void add(Limbs a, Limbs b)
  {
    hh += mul_wide(a.hi, b.hi);
    mid += mul_wide(a.hi, b.lo);
    mid += mul_wide(a.lo, b.hi);
  }
  NSM_HD void sub(Limbs a, Limbs b)
  {
    hh -= mul_wide(a.hi, b.hi);
    mid -= mul_wide(a.hi, b.lo);
    mid -= mul_wide(a.lo, b.hi);
  }
  NSM_HD i64 value() const
  {
    const u64 t = hh + (u64)((i64)mid >> 32);
    if (k == 0) return (i64)t;
#ifdef __CUDA_ARCH__
    return (i64)((u64)__funnelshift_l((unsigned)t, (unsigned)(t >> 32), k) << 32 |
                 __funnelshift_l((unsigned)mid, (unsigned)t, k));
#else
    return (i64)((t << k) | ((unsigned)mid >> (32 - k)));
#endif
  }
};
template <int k>
NSM_HD i64 mul(Limbs a, Limbs b)
{
  Acc<k> s;
  s.add(a, b);
  return s.value();
}

// The same to the nearest.
template <int k>
NSM_HD i64 mul_rounded(Limbs a, Limbs b)
{
  Acc<k> s;
  s.mid = 1ull << (31 - k);
  s.add(a, b);
  return s.value();
}

constexpr i64 kOne = 1ll << 60;  // 1.0 of H, F, the cofactors, J

// Powers and constants.
constexpr double kTwo61 = 2305843009213693952.0, kTwo62 = 4611686018427387904.0;
NSM_HD constexpr i64 q62(double v) { return (i64)(v * kTwo62); }
// g - 1 and g^2 at 2^64 (g the Gauss coordinate: x g = x + x (g - 1)), 1/3 at
// 2^64, 5/3 at 2^61
constexpr i64 kGm1_64 = 4 * q62(kGauss - 1.0), kGG64 = 4 * q62(kGauss * kGauss), kThird64 = 4 * (q62(1.0) / 3),
              kFiveThirds61 = q62(1.0) / 6 * 5;

NSM_HD i64 times_g(i64 x) { return x + mul<0>(split(x), split(kGm1_64)); }

// Whether |x| < 2^(32 + bits): zero in `mask` bits of the result otherwise.
template <int bits>
NSM_HD unsigned outside(i64 x)
{
  return (unsigned)((int)(x >> 32) + (1 << bits)) & ~((2u << bits) - 1u);
}

// |u| * 2^sc truncated, with the sign of u; R = 1086 - sc.  The biased
// exponent's shift leaves nothing of zeros and denormals.
NSM_HD i64 to_fixed(unsigned hi, unsigned lo, int R)
{
  const u64      m = ((u64)((hi & 0xfffffu) | 0x100000u) << 43) | ((u64)lo << 11);
  const unsigned r = (unsigned)(R - (int)((hi >> 20) & 0x7ffu));
  u64            a;
#ifdef __CUDA_ARCH__
  asm("shr.u64 %0, %1, %2;" : "=l"(a) : "l"(m), "r"(r));
#else
  a = r > 63u ? 0ull : m >> r;
#endif
  return (int)hi < 0 ? -(i64)a : (i64)a;
}

// ---- nodal displacements to gradients ----

// The modes of one component that the gradient needs, in a lane's mirrored
// coordinates, from its own modes q[my][mx] along xi and eta (m = 0 the sum, 1
// the difference along the axis) and those o of the lane across zeta.
enum Mode { kX, kXZ, kY, kYZ, kXY, kXYZ, kZ };
NSM_HD void lane_modes(const i64 q[2][2], const i64 o[2][2], i64 v[7])
{
  v[kX]   = q[0][1] + o[0][1];
  v[kXZ]  = q[0][1] - o[0][1];
  v[kY]   = q[1][0] + o[1][0];
  v[kYZ]  = q[1][0] - o[1][0];
  v[kXY]  = q[1][1] + o[1][1];
  v[kXYZ] = q[1][1] - o[1][1];
  v[kZ]   = q[0][0] - o[0][0];
}

// Shift from the displacements' scale to the element's (0 <= sh <= 26): the
// modes stay below 1.375 2^60, the gradients below 2^61.8, and |H|^2, of at most
// nine squares of 1.29, in 64 bits.
NSM_HD unsigned lane_shift(i64 v[7], int sh)
{
  unsigned  bad = 0;
  const int lim = (11 << 25) >> sh;
#pragma unroll
  for (int k = 0; k < 7; k++) {
    bad |= (unsigned)((int)(v[k] >> 32) + lim) >= 2u * (unsigned)lim;
    v[k] = (i64)((u64)v[k] << sh);
  }
  return bad;
}

// The gradient of one component at the lane's points: 8 du/dxi = x, and
// 8 du/deta = y, 8 du/dzeta = z at the first point (the - side along xi), y1
// and z1 more at the second.
struct Gradient {
  i64 x, y, y1, z, z1;
};
NSM_HD void lane_gradient(const i64 v[7], Gradient& G)
{
  const i64 xy = times_g(v[kXY]), xz = times_g(v[kXZ]), yz = times_g(v[kYZ]), xyz = mul<0>(split(v[kXYZ]), split(kGG64));
  const i64 hy = xy + xyz, hz = xz + xyz;
  G.x  = v[kX] + xy + hz;
  G.y  = v[kY] + yz - hy;
  G.y1 = hy + hy;
  G.z  = v[kZ] + yz - hz;
  G.z1 = hz + hz;
}

// ---- one point ----

// Moduli over 2^exponent, at 2^62 (at most 1/8), and lambda = K - 2 G / 3 for
// the elastic material.
struct Moduli {
  i64 half_k, g, lambda;
  int exponent;  // out of [-400, 400]: not representable
  int model;
};

struct Point {
  i64      H[3][3];  // 2^60
  Limbs    h[3][3];  // 2^62
  i64      C[3][3];  // cofactors of F, 2^60
  i64      t;        // J - 1, 2^60
  i64      n2;       // |H|^2, 2^60
  i64      sig[6];   // stress over 2^exponent, 2^62 (elastic 2^(62 + e); when asked for)
};

// H = Du G0 (Du at 2^su, G0 at 2^sG, su + sG = 124 + e: H at 2^(60 + e)), cut
// or rounded.
template <bool kRound = false>
NSM_HD void displacement_gradient(const i64 Du[3][3], const Limbs G0[3][3], i64 H[3][3])
{
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const Limbs d0 = split(Du[i][0]), d1 = split(Du[i][1]), d2 = split(Du[i][2]);
#pragma unroll
    for (int J = 0; J < 3; J++) {
      Acc<0> s;
      if (kRound) s.mid = 1ull << 31;
      s.add(d0, G0[0][J]);
      s.add(d1, G0[1][J]);
      s.add(d2, G0[2][J]);
      H[i][J] = s.value();
    }
  }
}

// From H: |H|^2, the cofactors of F = I + H and t = J - 1.  Reports |H| >= 1/2:
// up to there the high limbs of H at 2^62, of the cofactors and of F at 2^60 are
// below 2^29.3, and the sums of mixed products keep within 63 bits.  (|H|^2 is
// right to 2^33 for any H that Du G0 can give, entries below 1.29.)
NSM_HD unsigned kinematics(Point& p)
{
  u64 sq = 0, mid = 0;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      p.h[i][j] = split((i64)((u64)p.H[i][j] << 2));
      sq += mul_wide(p.h[i][j].hi, p.h[i][j].hi);
      mid += mul_wide(p.h[i][j].hi, p.h[i][j].lo);
    }
  p.n2 = (i64)sq + ((i64)mid >> 31);
#pragma unroll
  for (int r = 0; r < 3; r++)
#pragma unroll
    for (int c = 0; c < 3; c++) {
      // cofactor of entry (r, c): the minor of rows r1, r2 and columns c1, c2 in cyclic order
      const int r1 = (r + 1) % 3, r2 = (r + 2) % 3, c1 = (c + 1) % 3, c2 = (c + 2) % 3;
      Acc<0>    s;
      s.add(p.h[r1][c1], p.h[r2][c2]);
      s.sub(p.h[r1][c2], p.h[r2][c1]);
      p.C[r][c] = r == c ? s.value() + (p.H[r1][r1] + p.H[r2][r2] + kOne) : s.value() - p.H[c][r];
    }
  Acc<2> s;
  s.add(p.h[0][0], split(p.C[0][0]));
  s.add(p.h[0][1], split(p.C[0][1]));
  s.add(p.h[0][2], split(p.C[0][2]));
  p.t = (p.C[0][0] - kOne) + s.value();
  return (unsigned)((u64)p.n2 >> 58 != 0);
}

// J^(-5/3) and 1/J at 2^60 from t = J - 1.  y, J^(-1/3) to about 20 bits, is
// rounded to the integer Y = y 2^20, whose powers up to the third are exact;
// with e = 1 - J Y^3 (below 2^-18), 1/J = Y^3 (1 - e)^-1 and J^(-5/3) = Y^5
// (1 - e)^(-5/3), the binomial series to third order.  Their second-order
// terms are below 2^-35, where FP32 gives them to 2^-59.
NSM_HD void powers(i64 t, i64& r5, i64& rj)
{
  const i64   J  = kOne + t;
  const float jf = (float)(int)(J >> 32) * (1.0f / 268435456.0f);
#ifdef __CUDA_ARCH__
  const float y = exp2f(__log2f(jf) * (-1.0f / 3.0f));
#else
  const float y = exp2f(log2f(jf) * (-1.0f / 3.0f));
#endif
  const int   Y  = (int)(y * 1048576.0f + 0.5f);
  const i64   Y2 = (i64)mul_wide(Y, Y);  // 2^40
  const i64   Y3 = Y2 * Y;                     // 2^60
  const Limbs y3 = split(Y3);
  const i64   e  = kOne - mul<4>(split(J), y3);
  const float ef = (float)(int)(e >> 16) * (1.0f / 17592186044416.0f);
  const float e2 = ef * ef;
  const i64   c1 = e + (i64)(int)(e2 * (1.0f + ef) * 1.152921504606846976e18f);
  rj             = Y3 + (mul<0>(y3, split((i64)((u64)c1 << 20))) >> 16);
  const i64 Y5   = mul<4>(y3, split(Y2 << 20));
  const i64 c5   = (mul<0>(split((i64)((u64)e << 20)), split(kFiveThirds61)) >> 17) +
                 (i64)(int)(e2 * ((20.0f / 9.0f) + (220.0f / 81.0f) * ef) * 1.152921504606846976e18f);
  r5 = Y5 + (mul<0>(split(Y5), split((i64)((u64)c5 << 20))) >> 16);
}

// The scale of an elastic element.  Its stress is linear in H, and FP64 gives
// it to a relative 2^-52 however small H is, which 2^-60 absolute is not below
// strains of 1e-3.  Its displacement modes are therefore shifted up until the
// largest has 60 bits, e places beyond the scale of H at 2^60, and H, the
// stress and the forces are at 2^(60 + e), ...  (`bits` the length of the
// largest mode of the element, at 2^sc.)  e below -3: strains above the domain.
//
// The rows of its G0 are each scaled to their own largest entry (Rows), and the
// modes to match, so that a flat element loses few places: forces to 1.0e-16 of
// themselves for cubes (FP64 1.9e-16) and 1.3e-16 at an aspect ratio of 4 (FP64
// 3.9e-16; tests/fixed_domain_check.cc).  Flatter elements than kMaxRow says,
// and materials of K > 4 G (their shear modulus has fewer bits), are left to
// FP64: where it has nothing to round but the result (shear along the axes of an
// unjittered mesh, 1.1e-16; plane stress, 1.6e-16) the forces of cubes with
// K = 2 G are off by 1.6e-16 and 1.3e-16 here, at K = 4 G and an aspect ratio of
// 4 by 6e-16 and 5e-16, and more beyond.
//
// The forces at the points keep kElasticForce further places: with more, their
// sums could leave 63 bits, and one element left to the FP64 code makes a launch
// wait 45 us for it.  Products are rounded, not cut.
constexpr int kElasticForce = 3;
NSM_HD void elastic_scale(int bits, int sc, int su, int& sh, int& e)
{
  sh = 60 - bits;
  e  = sc + sh - su;
}

// Binary places by which the rows xi, eta, zeta of an elastic element's G0 lie
// below the largest (0) and are stored scaled up.
constexpr int kMaxRow = 2;
struct Rows {
  int x, y, z;
};
NSM_HD int lower(int a, int b) { return a < b ? a : b; }

// A mode belongs to the rows of its axes and is kept at the scale of the
// largest of them (Du of a row at 2^(su - its places)).
NSM_HD void mode_places(const Rows& r, int places[7])
{
  places[kX]   = r.x;
  places[kY]   = r.y;
  places[kZ]   = r.z;
  places[kXY]  = lower(r.x, r.y);
  places[kXZ]  = lower(r.x, r.z);
  places[kYZ]  = lower(r.y, r.z);
  places[kXYZ] = 0;
}

// The bits of one component's modes, each at its scale and kMaxRow places more:
// the longest of an element gives `bits` of elastic_scale, kMaxRow less.  (Zero
// for zeros alone.)
NSM_HD u64 mode_bits(const i64 v[7], const Rows& r)
{
  int places[7];
  mode_places(r, places);
  u64 m = 0;
#pragma unroll
  for (int k = 0; k < 7; k++) m |= ((u64)(v[k] ^ (v[k] >> 63)) | (u64)(v[k] & 1)) << (kMaxRow - places[k]);
  return m;
}

// Shift of the modes to the element's scale (0 <= sh < 60; below 2^62 on the way).
NSM_HD void elastic_shift(i64 v[7], const Rows& r, int sh)
{
  int places[7];
  mode_places(r, places);
#pragma unroll
  for (int k = 0; k < 7; k++) v[k] = (i64)((u64)v[k] << sh) >> places[k];
}

// lane_gradient with each row's values at the row's scale.
NSM_HD void elastic_gradient(const i64 v[7], const Rows& r, Gradient& G)
{
  int places[7];
  mode_places(r, places);
  const i64 xy = times_g(v[kXY]), xz = times_g(v[kXZ]), yz = times_g(v[kYZ]), xyz = mul<0>(split(v[kXYZ]), split(kGG64));
  const i64 hy = (xy >> (r.y - places[kXY])) + (xyz >> r.y), hz = (xz >> (r.z - places[kXZ])) + (xyz >> r.z);
  G.x  = v[kX] + (xy >> (r.x - places[kXY])) + (xz >> (r.x - places[kXZ])) + (xyz >> r.x);
  G.y  = v[kY] + (yz >> (r.y - places[kYZ])) - hy;
  G.y1 = hy + hy;
  G.z  = v[kZ] + (yz >> (r.z - places[kYZ])) - hz;
  G.z1 = hz + hz;
}

// P[J][i] = det' adj(F) sigma at 2^62 over 2^exponent of the moduli, det' the
// point's reference volume over the element's power of two (2^62).
//
// Neo-Hookean: sigma = q0 I + g (b - I) with g = G J^(-5/3) and
// q0 = K/2 (J - 1/J) - g tr(b - I) / 3, and adj(F) b = J F^T, so
// adj(F) sigma = g J F^T + (q0 - g) adj(F): the stress itself is formed only
// where it is stored.  With |H| < 1/8 and moduli of at most 1/8, |P| < 2^58.4
// and the forces stay below 2^62.2.  Up to |H| = 1/2 (J in [0.35, 2.2], J^(-5/3)
// below 5.8, |P| < 2^62.5) that is checked, and larger P reported.
template <bool kStress>
NSM_HD unsigned neohookean_force(const Moduli& m, i64 det, Point& p, i64 P[3][3])
{
  const Limbs d  = split(det);
  const i64   tr = p.H[0][0] + p.H[1][1] + p.H[2][2];
  i64         r5, rj;
  powers(p.t, r5, rj);
  const i64   g  = mul<4>(split(r5), split(m.g));  // 2^62
  const Limbs gl = split(g);
  const i64   gm = mul<4>(split(mul<0>(split(2 * tr + p.n2), split(kThird64))), gl);  // tr(b - I) = 2 tr H + |H|^2
  const i64   pr = mul<4>(split(p.t + (kOne - rj)), split(m.half_k));                 // K/2 (J - 1/J)
  const i64   q0 = pr - gm;
  const i64   a  = g + mul<4>(gl, split(p.t));
  const i64   b  = q0 - g;
  if (kStress) {
#pragma unroll
    for (int q = 0; q < 6; q++) {
      const int i = q < 3 ? q : (q == 3 ? 0 : (q == 4 ? 1 : 2)), j = q < 3 ? q : (q == 3 ? 1 : (q == 4 ? 2 : 0));
      Acc<0>    s;
      s.add(p.h[i][0], p.h[j][0]);
      s.add(p.h[i][1], p.h[j][1]);
      s.add(p.h[i][2], p.h[j][2]);
      p.sig[q] = mul<4>(split(s.value() + p.H[i][j] + p.H[j][i]), gl) + (q < 3 ? q0 : 0);
    }
  }
  const Limbs ad = split(mul<2>(split(a), d)), bd = split(mul<2>(split(b), d));
#pragma unroll
  for (int J = 0; J < 3; J++)
#pragma unroll
    for (int i = 0; i < 3; i++) {
      Acc<4> s;
      s.add(ad, split(p.H[i][J] + (i == J ? kOne : 0)));
      s.add(bd, split(p.C[i][J]));
      P[J][i] = s.value();
    }
  unsigned bad = 0;
  if ((p.n2 >> 54) != 0) {
#pragma unroll
    for (int q = 0; q < 9; q++) bad |= outside<26>(P[q / 3][q % 3]);
  }
  return bad;
}

// The same for the elastic material, sigma = G (H + H^T) + lambda tr(H) I, with
// H at 2^(60 + e) as He: P at 2^(62 + e + kElasticForce).  adj(F) sigma is
// formed as sigma + (adj(F) - I) sigma: the first term loses nothing, and the
// products of the second have two places more.
template <bool kStress>
NSM_HD unsigned elastic_force(const Moduli& m, i64 det, const i64 He[3][3], Point& p, i64 P[3][3])
{
  unsigned    bad = 0;
  const Limbs d = split(det), g = split(m.g);
  const i64   l = mul_rounded<4>(split(He[0][0] + He[1][1] + He[2][2]), split(m.lambda));
  i64         s[6];
#pragma unroll
  for (int q = 0; q < 6; q++) {
    const int i = q < 3 ? q : (q == 3 ? 0 : (q == 4 ? 1 : 2)), j = q < 3 ? q : (q == 3 ? 1 : (q == 4 ? 2 : 0));
    const i64 v = mul_rounded<4>(split(He[i][j] + He[j][i]), g) + (q < 3 ? l : 0);
    if (kStress) p.sig[q] = v;
    s[q] = mul_rounded<2>(split(v), d);
    bad |= outside<26>(s[q]);  // (P below 2^62.2)
  }
#pragma unroll
  for (int J = 0; J < 3; J++) {
    Limbs c[3];
#pragma unroll
    for (int k = 0; k < 3; k++) c[k] = split((i64)((u64)(p.C[k][J] - (k == J ? kOne : 0)) << 2));
#pragma unroll
    for (int i = 0; i < 3; i++) {
      Acc<2 + kElasticForce> a;
      a.mid = 1ull << (31 - (2 + kElasticForce));
#pragma unroll
      for (int k = 0; k < 3; k++) a.add(c[k], split(s[sym_slot(k, i)]));
      P[J][i] = a.value() + (i64)((u64)s[sym_slot(J, i)] << kElasticForce);
    }
  }
  return bad;
}

// Q[d][i] = sum_J G0[d][J] P[J][i].
NSM_HD void point_force(const Limbs G0[3][3], const i64 P[3][3], i64 Q[3][3])
{
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const Limbs p0 = split(P[0][i]), p1 = split(P[1][i]), p2 = split(P[2][i]);
#pragma unroll
    for (int d = 0; d < 3; d++) {
      Acc<0> s;
      s.mid = 1ull << 31;  // rounded: the eight points' forces add up
      s.add(G0[d][0], p0);
      s.add(G0[d][1], p1);
      s.add(G0[d][2], p2);
      Q[d][i] = s.value();
    }
  }
}

// ---- point sums to nodal forces ----

// Sums of one component over the lane's points (sides - and + along xi); y1
// and z1 with the side's sign.
struct Sums {
  i64 x, y, y1, z, z1;
};

// An elastic element's sums from the scales of their rows to a common one,
// kElasticSum places below that of the forces at the points (one place: 7 to 14
// of 20,000 unjittered cubes would be too large without it, none with it).
constexpr int kElasticSum = 1;
NSM_HD i64 rounded_down(i64 x, int places) { return (x + (1ll << (places - 1))) >> places; }
NSM_HD void common_scale(Sums& S, const Rows& r)
{
  S.x  = rounded_down(S.x, r.x + kElasticSum);
  S.y  = rounded_down(S.y, r.y + kElasticSum);
  S.y1 = rounded_down(S.y1, r.y + kElasticSum);
  S.z  = rounded_down(S.z, r.z + kElasticSum);
  S.z1 = rounded_down(S.z1, r.z + kElasticSum);
}

// Whether the forces of sums this large may leave 63 bits: a force is at most
// 29.8 of the largest sum (lane_adjoint: 3.15 even and 4.31 odd in xi, four
// lanes), and those of 2^58 and less stay below 2^62.9.
NSM_HD unsigned too_large(const Sums& S)
{
  return outside<26>(S.x) | outside<26>(S.y) | outside<26>(S.y1) | outside<26>(S.z) | outside<26>(S.z1);
}

// A lane's part of the forces in one component, even and odd in xi, with and
// without a factor of the side along eta: for its own side along zeta (keep)
// and for the other (send).
struct Parts {
  i64 e0, e1, o0, o1;
};
NSM_HD void lane_adjoint(const Sums& S, Parts& keep, Parts& send)
{
  const i64 xy = times_g(S.x + S.y1), xz = times_g(S.x + S.z1), yz = times_g(S.y + S.z);
  const i64 xyz = mul<0>(split(S.x + S.y1 + S.z1), split(kGG64));
  keep = Parts{S.z, S.y + yz, S.x + xz, xy + xyz};
  send = Parts{-S.z, S.y - yz, S.x - xz, xy - xyz};
}

#undef NSM_HD

}  // namespace fx
}  // namespace nsm
