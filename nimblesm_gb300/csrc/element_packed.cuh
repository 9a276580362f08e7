// The FP32 form's element with two integration points per operation.
//
// The element kernel is bound by issue: 2,290 instructions per element, 1,750 of
// them on the FMA pipe, which was busy half the time.  A packed operation
// (add/mul/fma.rn.f32x2) issues once for two values and takes the pipe twice
// as long, so the points x = 0 and x = 1 of each (y, z) are evaluated together:
// 1,810 instructions, 194 -> 172 us for 2,097,152 elements.  What the two
// points share along x is one sum per point pair and stays scalar, as do
// J^(-1/3), the reciprocals and the transforms before and after (packed over u
// and X, those would have to be taken apart again for the points).
//
// The operations and their order are those that element_work<float> compiles
// to, products fused into sums included (minor, dot3), so the bits are the
// same.  Neo-Hookean elements, no records: steps inside an advance.  H is dead
// once b - I is formed, without which the registers of 3 blocks per SM do not
// suffice (with records 200 us, 1 KB of spills per warp; 2 blocks per SM 240).
#pragma once

#include "element_work.cuh"

namespace nsm {
namespace p2 {

// Two FP32 values in a register pair, the low half first; every operation is
// the IEEE one of each half.
using f2 = unsigned long long;
__device__ __forceinline__ f2 pack(float x, float y)
{
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float half(f2 v, int h)
{
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
  return h ? y : x;
}
__device__ __forceinline__ f2 add(f2 a, f2 b)
{
  f2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 mul(f2 a, f2 b)
{
  f2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 fma(f2 a, f2 b, f2 c)
{
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f2 neg(f2 a) { return a ^ 0x8000000080000000ull; }

// a b - c d with nc = -c, and a0 b0 + a1 b1 + a2 b2.
__device__ __forceinline__ f2 minor(f2 a, f2 b, f2 nc, f2 d) { return fma(a, b, mul(nc, d)); }
__device__ __forceinline__ f2 dot3(f2 a0, f2 b0, f2 a1, f2 b1, f2 a2, f2 b2)
{
  return fma(a2, b2, fma(a0, b0, mul(a1, b1)));
}

// hex_math.cuh's invert3 and cofactor3.
__device__ __forceinline__ void invert3(const f2 A[3][3], f2 inv[3][3], float det[2])
{
  f2 N[3][3];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) N[i][j] = neg(A[i][j]);
  const f2 c00 = minor(A[1][1], A[2][2], N[1][2], A[2][1]);
  const f2 c01 = minor(A[1][2], A[2][0], N[1][0], A[2][2]);
  const f2 c02 = minor(A[1][0], A[2][1], N[1][1], A[2][0]);
  const f2 d   = dot3(A[0][0], c00, A[0][1], c01, A[0][2], c02);
  det[0]       = half(d, 0);
  det[1]       = half(d, 1);
  const f2 r   = pack(reciprocal(det[0]), reciprocal(det[1]));
  inv[0][0]    = mul(c00, r);
  inv[1][0]    = mul(c01, r);
  inv[2][0]    = mul(c02, r);
  inv[0][1]    = mul(minor(A[0][2], A[2][1], N[0][1], A[2][2]), r);
  inv[1][1]    = mul(minor(A[0][0], A[2][2], N[0][2], A[2][0]), r);
  inv[2][1]    = mul(minor(A[0][1], A[2][0], N[0][0], A[2][1]), r);
  inv[0][2]    = mul(minor(A[0][1], A[1][2], N[0][2], A[1][1]), r);
  inv[1][2]    = mul(minor(A[0][2], A[1][0], N[0][0], A[1][2]), r);
  inv[2][2]    = mul(minor(A[0][0], A[1][1], N[0][1], A[1][0]), r);
}
__device__ __forceinline__ f2 cofactor3(const f2 M[3][3], f2 C[3][3])
{
  f2 N[3][3];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) N[i][j] = neg(M[i][j]);
  C[0][0] = minor(M[1][1], M[2][2], N[1][2], M[2][1]);
  C[0][1] = minor(M[1][2], M[2][0], N[1][0], M[2][2]);
  C[0][2] = minor(M[1][0], M[2][1], N[1][1], M[2][0]);
  C[1][0] = minor(M[0][2], M[2][1], N[0][1], M[2][2]);
  C[1][1] = minor(M[0][0], M[2][2], N[0][2], M[2][0]);
  C[1][2] = minor(M[0][1], M[2][0], N[0][0], M[2][1]);
  C[2][0] = minor(M[0][1], M[1][2], N[0][2], M[1][1]);
  C[2][1] = minor(M[0][2], M[1][0], N[0][0], M[1][2]);
  C[2][2] = minor(M[0][0], M[1][1], N[0][1], M[1][0]);
  return dot3(M[0][0], C[0][0], M[0][1], C[0][1], M[0][2], C[0][2]);
}

// hex_math.cuh's neohookean_stress: b - I, then the stress.
__device__ __forceinline__ void strain(const f2 H[3][3], f2 B[6])
{
#pragma unroll
  for (int q = 0; q < 6; q++) {
    const int i = q < 3 ? q : (q == 3 ? 0 : (q == 4 ? 1 : 2));
    const int j = q < 3 ? q : (q == 3 ? 1 : (q == 4 ? 2 : 0));
    B[q]        = fma(H[i][0], H[j][0], fma(H[i][1], H[j][1], fma(H[i][2], H[j][2], add(H[i][j], H[j][i]))));
  }
}
__device__ __forceinline__ void neohookean_stress(const f2 B[6], const float J[2], float K, float G, f2 sig[6])
{
  float pr[2], Gr5[2];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const float r  = rcbrt_refined(J[h]);
    const float r2 = r * r;
    const float r3 = r2 * r;
    const float r5 = r3 * r2;
    pr[h]          = 0.5f * K * (J[h] - r3);
    Gr5[h]         = G * r5;
  }
  const f2 third = pack(float(1.0 / 3.0), float(1.0 / 3.0));
  const f2 g     = pack(Gr5[0], Gr5[1]);
  const f2 m     = mul(add(add(B[0], B[1]), B[2]), third);
  const f2 q0    = fma(neg(g), m, pack(pr[0], pr[1]));
#pragma unroll
  for (int q = 0; q < 6; q++) sig[q] = q < 3 ? fma(g, B[q], q0) : mul(g, B[q]);
}

}  // namespace p2

// element_work<float, false> (neo-Hookean, no records) with two points (x = 0,
// 1) at a time.
template <class Nodes>
__device__ __forceinline__ void element_work_packed(const ElementArgs& a, const int e, const Nodes& nodes)
{
  using p2::f2;
  float Gu[3][3][2][2], GX[3][3][2][2];
  {
    float x[8][3];
#pragma unroll
    for (int n = 0; n < 8; n++) nodes.u(n, x[n]);
    nodal_gradient<float>(x, Gu);
  }
  {
    float x[8][3];
#pragma unroll
    for (int n = 0; n < 8; n++) nodes.X(n, x[n]);
    nodal_gradient<float>(x, GX);
  }
  f2    S2[2][3][2];     // d - 1, i, the bit along the other of eta and zeta
  float S0[3][2][2];
  float K = (float)a.bulk, Gm = (float)a.shear;
  if (a.elem_group) {
    const GroupMaterial& m = a.mats[__ldg(&a.elem_group[e])];
    K                      = (float)m.bulk;
    Gm                     = (float)m.shear;
  }
  bool bad = false;

#pragma unroll
  for (int z = 0; z < 2; z++)
#pragma unroll
    for (int y = 0; y < 2; y++) {
      f2 JX[3][3], G0[3][3], Du[3][3], H[3][3], Jx[3][3], Cx[3][3], sig[6];
#pragma unroll
      for (int i = 0; i < 3; i++) {
        JX[i][0] = p2::pack(GX[0][i][y][z], GX[0][i][y][z]);
        JX[i][1] = p2::pack(GX[1][i][0][z], GX[1][i][1][z]);
        JX[i][2] = p2::pack(GX[2][i][0][y], GX[2][i][1][y]);
        Du[i][0] = p2::pack(Gu[0][i][y][z], Gu[0][i][y][z]);
        Du[i][1] = p2::pack(Gu[1][i][0][z], Gu[1][i][1][z]);
        Du[i][2] = p2::pack(Gu[2][i][0][y], Gu[2][i][1][y]);
      }
      float det0[2], J[2];
      p2::invert3(JX, G0, det0);
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int d = 0; d < 3; d++) Jx[i][d] = p2::add(JX[i][d], Du[i][d]);
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int k = 0; k < 3; k++)
          H[i][k] = p2::fma(Du[i][0], G0[0][k], p2::fma(Du[i][1], G0[1][k], p2::mul(Du[i][2], G0[2][k])));
      f2 B[6];
      p2::strain(H, B);
      const f2 det = p2::cofactor3(Jx, Cx);
#pragma unroll
      for (int h = 0; h < 2; h++) {
        if (!(det0[h] > 0.0f)) bad = true;
        J[h] = p2::half(det, h) * reciprocal(det0[h]);
        if (!positive(J[h])) bad = true;
      }
      p2::neohookean_stress(B, J, K, Gm, sig);
      // the lower-numbered point of a pair along an axis is the first of its sum
#pragma unroll
      for (int d = 1; d < 3; d++)
#pragma unroll
        for (int i = 0; i < 3; i++) {
          f2&      acc  = S2[d - 1][i][d == 1 ? z : y];
          const f2 s0 = sig[sym_slot(0, i)], s1 = sig[sym_slot(1, i)], s2 = sig[sym_slot(2, i)];
          const f2 tail = (d == 1 ? y : z) == 0 ? p2::mul(Cx[2][d], s2) : p2::fma(Cx[2][d], s2, acc);
          acc           = p2::fma(Cx[0][d], s0, p2::fma(Cx[1][d], s1, tail));
        }
#pragma unroll
      for (int i = 0; i < 3; i++) {
        float acc = 0.0f;
#pragma unroll
        for (int n = 0; n < 2; n++) {
          const int   h  = n == 0 ? y : 1 - y;  // y = 0: x = 0 first, y = 1: x = 1
          const float c0 = p2::half(Cx[0][0], h), c1 = p2::half(Cx[1][0], h), c2 = p2::half(Cx[2][0], h);
          const float s0 = p2::half(sig[sym_slot(0, i)], h), s1 = p2::half(sig[sym_slot(1, i)], h),
                      s2 = p2::half(sig[sym_slot(2, i)], h);
          const float tail = n == 0 ? c2 * s2 : fmaf(c2, s2, acc);
          acc              = fmaf(c0, s0, fmaf(c1, s1, tail));
        }
        S0[i][y][z] = acc;
      }
    }
  float S[3][3][2][2], f[8][3];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int s = 0; s < 2; s++)
#pragma unroll
      for (int t = 0; t < 2; t++) {
        S[0][i][s][t] = S0[i][s][t];
        S[1][i][s][t] = p2::half(S2[0][i][t], s);
        S[2][i][s][t] = p2::half(S2[1][i][t], s);
      }
  nodal_adjoint<float>(S, -1.0f / 512.0f, f);
  store_forces<float>(a, e, f, bad);
}

}  // namespace nsm
