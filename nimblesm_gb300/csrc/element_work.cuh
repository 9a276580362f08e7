// One element's work on floating point (gather -> deformation gradient ->
// neo-Hookean or elastic Cauchy stress -> B^T sigma), T = double / float, with
// what it needs to load nodal values and to store records.  The element math
// and the reasons for its form are in hex_math.cuh.
#pragma once

#include <type_traits>

#include "hex_math.cuh"
#include "nsm_kernels.cuh"

namespace nsm {

// Vector stores of a thread's contiguous values (16-byte aligned).
__device__ __forceinline__ void store_vec(float* dst, const float* v, int n)
{
#pragma unroll
  for (int k = 0; k < n; k += 4)
    *reinterpret_cast<float4*>(dst + k) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
}
__device__ __forceinline__ void store_vec(double* dst, const double* v, int n)
{
#pragma unroll
  for (int k = 0; k < n; k += 2) *reinterpret_cast<double2*>(dst + k) = make_double2(v[k], v[k + 1]);
}

// Warp-cooperative stores.  A thread's point record (64 or 128 B) is
// contiguous, and so are those of the 32 consecutive elements of a warp;
// stored lane by lane, each store instruction would scatter 16-byte pieces a
// record apart, which HBM takes at half the rate of contiguous writes.
// Instead the warp passes its 32 records through a shared-memory tile and
// each instruction writes 512 contiguous bytes.  The tile slots are swizzled
// (4 and 8 chunks per record) so that neither the per-lane writes nor the
// transposed reads conflict on banks.
template <int kChunks>
__device__ __forceinline__ int tile_slot(int row, int c)
{
  if constexpr (kChunks == 4) return row * 4 + (c ^ ((row >> 1) & 3));
  else if constexpr (kChunks == 8) return row * 8 + (c ^ (row & 7));
  else return row * (kChunks + 1) + c;
}
template <int kChunks>
__host__ __device__ constexpr int tile_chunks() { return 32 * (kChunks == 4 || kChunks == 8 ? kChunks : kChunks + 1); }

__device__ __forceinline__ uint4 pack16(const float* v, int c)
{
  return make_uint4(__float_as_uint(v[4 * c]), __float_as_uint(v[4 * c + 1]), __float_as_uint(v[4 * c + 2]),
                    __float_as_uint(v[4 * c + 3]));
}
__device__ __forceinline__ uint4 pack16(const double* v, int c)
{
  const unsigned long long a = __double_as_longlong(v[2 * c]), b = __double_as_longlong(v[2 * c + 1]);
  return make_uint4((unsigned)a, (unsigned)(a >> 32), (unsigned)b, (unsigned)(b >> 32));
}

// A warp's tile: contiguous, or rows of 32 chunks `row` chunks apart.
struct Tile {
  uint4* p;
  int    row;
  __device__ __forceinline__ uint4& operator[](int i) const { return p[(i >> 5) * row + (i & 31)]; }
};

// dst: the first lane's block; all 32 lanes of the warp take part.
template <int kChunks, typename T>
__device__ __forceinline__ void warp_store(uint4* __restrict__ dst, const T* v, const Tile& tile, int lane)
{
  __syncwarp();  // the tile's previous contents have been read
#pragma unroll
  for (int c = 0; c < kChunks; c++) tile[tile_slot<kChunks>(lane, c)] = pack16(v, c);
  __syncwarp();
#pragma unroll
  for (int k = 0; k < kChunks; k++) {
    const int j = k * 32 + lane;
    dst[j]      = tile[tile_slot<kChunks>(j / kChunks, j % kChunks)];
  }
}

// Finiteness without the FP64 pipe: an exponent field of all ones is an
// infinity or a NaN.
__device__ __forceinline__ bool finite_bits(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }
__device__ __forceinline__ bool finite_bits(float x) { return isfinite(x); }

// J > 0 without the FP64 pipe: the sign and magnitude bits of an IEEE number
// order like a signed integer (a NaN J passes here and is caught as a
// non-finite force).
__device__ __forceinline__ bool positive(double x) { return __double_as_longlong(x) > 0; }
__device__ __forceinline__ bool positive(float x) { return x > 0.0f; }

// Where an element's nodal values come from.  GlobalNodes: gathered through
// the connectivity, from the FP64 field's planes or, in the FP32 form, from
// the FP32 copies (no FP64 conversions, which would run on the FP64 pipe), one
// 16-byte record per node and field.  StagedNodes: this thread's slots of a
// shared-memory stage that cp.async filled one element ahead (FP32 form).
template <typename T>
struct GlobalNodes {
  const ElementArgs& a;
  int                id[8];
  __device__ __forceinline__ GlobalNodes(const ElementArgs& args, int e) : a(args)
  {
#pragma unroll
    for (int n = 0; n < 8; n++) id[n] = __ldg(&a.conn[n * a.ld_e + e]);
  }
  __device__ __forceinline__ void u(int n, T x[3]) const
  {
    if constexpr (sizeof(T) == 8) {
#pragma unroll
      for (int k = 0; k < 3; k++) x[k] = a.u[k * a.ld_n + id[n]];  // (an overlapped launch's: ordinary loads)
    } else {
      const float4 v = a.uf[id[n]];
      x[0] = v.x, x[1] = v.y, x[2] = v.z;
    }
  }
  __device__ __forceinline__ void X(int n, T x[3]) const
  {
    const float4 v = __ldg(&a.Xf[id[n]]);
    x[0] = v.x, x[1] = v.y, x[2] = v.z;
  }
  __device__ __forceinline__ Tile tile(uint4* own) const { return Tile{own, 32}; }
};

// Stage layout: [16][blockDim] float4 per element slot, 0..7 the nodes' u,
// 8..15 X; thread t owns column t, so the lanes of a warp read consecutive
// chunks.  Once the values are read the first rows serve as the warp's tile.
constexpr int kStageValues = 16;
struct StagedNodes {
  float4* s;  // this thread's column of the stage
  int     B;  // column stride (threads per block)
  __device__ __forceinline__ void u(int n, float x[3]) const
  {
    const float4 v = s[n * B];
    x[0] = v.x, x[1] = v.y, x[2] = v.z;
  }
  __device__ __forceinline__ void X(int n, float x[3]) const
  {
    const float4 v = s[(8 + n) * B];
    x[0] = v.x, x[1] = v.y, x[2] = v.z;
  }
  __device__ __forceinline__ Tile tile(uint4*) const { return Tile{reinterpret_cast<uint4*>(s - (threadIdx.x & 31)), B}; }
};

// An element's nodal forces, and what they report.
template <typename T>
__device__ __forceinline__ void store_forces(const ElementArgs& a, const int e, const T f[8][3], bool bad)
{
  const long ld_e = a.ld_e;
  T    fv[24];
  bool finite = true;
#pragma unroll
  for (int n = 0; n < 8; n++)
#pragma unroll
    for (int i = 0; i < 3; i++) {
      fv[n * 3 + i] = f[n][i];
      finite        = finite & finite_bits(f[n][i]);
    }
  bool planes = true;
  if constexpr (sizeof(T) == 4) {
    planes = a.fe_slot == nullptr;
    if (!planes) {
#pragma unroll
      for (int n = 0; n < 8; n++)
        reinterpret_cast<float4*>(a.fe)[__ldg(&a.fe_slot[n * ld_e + e])] =
            make_float4(fv[3 * n], fv[3 * n + 1], fv[3 * n + 2], 0.0f);
    }
  }
  if (planes) {
    T* fe = reinterpret_cast<T*>(a.fe) + e;
#pragma unroll
    for (int q = 0; q < 24; q++) fe[(size_t)q * ld_e] = fv[q];
  }
  if (bad || !finite) atomicOr(a.status, (bad ? NSM_STATUS_BAD_JACOBIAN : 0) | (finite ? 0 : NSM_STATUS_NONFINITE));
}

// FP64 form: reference geometry precomputed (geo planes).  FP32 form: the
// reference Jacobian is rebuilt from X each step with the same transform.
// kPass: 0 the fused step (F, sigma, records, forces); with a block-material
// callback the step is split as the reference's plugin path splits it,
// 1 kinematics (F and the built-in materials' sigma into the records; zero
// sigma where the callback computes it), 2 forces from the recorded sigma.
template <typename T, bool kPrecomputedGeo, class Nodes, int kPass = 0, bool kWarp = true>
__device__ __forceinline__ void element_work(const ElementArgs& a, const int e, const Nodes& nodes)
{
  const long ld_e = a.ld_e;

  // displacement gradient at the points (36 distinct values)
  T Gu[3][3][2][2];
  {
    T x[8][3];
#pragma unroll
    for (int n = 0; n < 8; n++) nodes.u(n, x[n]);
    nodal_gradient<T>(x, Gu);
  }
  T GX[3][3][2][2];
  if constexpr (!kPrecomputedGeo) {
    T x[8][3];
#pragma unroll
    for (int n = 0; n < 8; n++) nodes.X(n, x[n]);
    nodal_gradient<T>(x, GX);
  }

  T S[3][3][2][2];  // point sums of Q[d][i] grouped by the other-axis sign pairs
#pragma unroll
  for (int d = 0; d < 3; d++)
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int s = 0; s < 2; s++)
#pragma unroll
        for (int t = 0; t < 2; t++) S[d][i][s][t] = T(0);

  T   K = T(a.bulk), Gm = T(a.shear);
  int model = a.model;
  if (a.elem_group) {
    const GroupMaterial& m = a.mats[__ldg(&a.elem_group[e])];
    K                      = T(m.bulk);
    Gm                     = T(m.shear);
    model                  = m.model;
  }
  bool    bad = false;
  T*      rec = reinterpret_cast<T*>(a.ip) + (size_t)e * kIpRecord;
  const bool store =
      kPass == 1 ||
      (kPass == 0 && (a.store_ip == kStoreAlways ||
                      (a.store_ip == kStoreOutput && a.sched != nullptr &&
                       a.sched[(long)(*a.step_base + a.k) * a.num_groups].is_output)));
  // a warp of 32 consecutive elements (kWarp) stores through its tile; a
  // partial warp or a single lane by itself
  constexpr int kRecChunks = kIpRecord * (int)sizeof(T) / 16;
  constexpr int kTile      = tile_chunks<kRecChunks>();
  constexpr bool   kOwnTile = kWarp && !std::is_same<Nodes, StagedNodes>::value;
  __shared__ uint4 tiles[kOwnTile ? 4 : 1][kOwnTile ? kTile : 1];  // blocks of at most 128 threads
  const int        lane   = threadIdx.x & 31;
  const long       e0     = (long)e - lane;  // the warp's elements are e0 .. e0 + 31
  const bool       whole  = kWarp && e0 + 32 <= a.E;
  const Tile       tile   = nodes.tile(tiles[kOwnTile ? (threadIdx.x >> 5) & 3 : 0]);

#pragma unroll
  for (int p = 0; p < 8; p++) {
    const int bit[3] = {sx_of(p), sy_of(p), sz_of(p)};
    T         G0[3][3], JX[3][3], idet0;  // J_X^{-1} / 8, 8 J_X, 1 / (512 det J_X)
    if (kPrecomputedGeo) {
#pragma unroll
      for (int q = 0; q < 9; q++) {
        G0[q / 3][q % 3] = T(__ldg(&a.geo[(p * kGeoPerPoint + q) * ld_e + e]));
        JX[q / 3][q % 3] = T(__ldg(&a.geo[(p * kGeoPerPoint + 10 + q) * ld_e + e]));
      }
      idet0 = T(__ldg(&a.geo[(p * kGeoPerPoint + 19) * ld_e + e]));
    } else {
      T det0;
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int d = 0; d < 3; d++) JX[i][d] = GX[d][i][bit[other1(d)]][bit[other2(d)]];
      invert3<T>(JX, G0, det0);
      if (!(det0 > T(0))) bad = true;  // (checked once at setup in the FP64 form)
      idet0 = reciprocal(det0);
    }
    // Du[i][d] = 8 du_i/dxi_d;  H = Du G0;  8 J_x = 8 J_X + Du, J_x the current Jacobian
    T Du[3][3], H[3][3], Jx[3][3];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int d = 0; d < 3; d++) {
        Du[i][d] = Gu[d][i][bit[other1(d)]][bit[other2(d)]];
        Jx[i][d] = JX[i][d] + Du[i][d];
      }
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int J = 0; J < 3; J++) H[i][J] = fma(Du[i][0], G0[0][J], fma(Du[i][1], G0[1][J], Du[i][2] * G0[2][J]));
    // det J_x = J det J_X, and the force term det(J_x) J_x^{-1} sigma = adj(J_x) sigma
    T       Cx[3][3];
    const T J = cofactor3<T>(Jx, Cx) * idet0;
    T sig[6];
    if constexpr (kPass == 2) {  // the stress the kinematics pass and the callback recorded
#pragma unroll
      for (int q = 0; q < 6; q++) sig[q] = rec[(size_t)p * ld_e * kIpRecord + 9 + q];
    } else {
      material_stress_j<T>(model, H, J, K, Gm, sig);
    }
    if (!positive(J)) bad = true;  // inverted element
    if (store) {
      T r[kIpRecord];
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int k = 0; k < 3; k++) r[full_slot(i, k)] = (i == k) ? one_plus(H[i][k]) : H[i][k];
#pragma unroll
      for (int q = 0; q < 6; q++) r[9 + q] = sig[q];
      r[15] = T(0);
      if (whole)
        warp_store<kRecChunks>(reinterpret_cast<uint4*>(reinterpret_cast<T*>(a.ip) + ((size_t)p * ld_e + e0) * kIpRecord),
                               r, tile, lane);
      else
        store_vec(rec + (size_t)p * ld_e * kIpRecord, r, kIpRecord);
    }
    // Q[d][i] = sum_k adj(J_x)[d][k] sigma[k][i] = sum_k cof(J_x)[k][d] sigma[k][i],
    // summed over the two points of each sign pair (the first assigns)
    if constexpr (kPass != 1) {
#pragma unroll
      for (int d = 0; d < 3; d++)
#pragma unroll
        for (int i = 0; i < 3; i++) {
          T&      acc  = S[d][i][bit[other1(d)]][bit[other2(d)]];
          const T tail = first_of_pair(d, p) ? Cx[2][d] * sym(sig, 2, i) : fma(Cx[2][d], sym(sig, 2, i), acc);
          acc          = fma(Cx[0][d], sym(sig, 0, i), fma(Cx[1][d], sym(sig, 1, i), tail));
        }
    }
  }
  if constexpr (kPass == 1) {  // kinematics only: the records are written
    if (bad) atomicOr(a.status, NSM_STATUS_BAD_JACOBIAN);
    return;
  }

  // f_a,i = - sum_p sum_d dN_a/dxi_d(p) Q_p[d][i].  J_x and hence Q carry
  // the factor 8^2 of the modal gradient, dN/dxi another 8: scale -1/512.
  T f[8][3];
  nodal_adjoint<T>(S, T(-1.0 / 512.0), f);
  store_forces<T>(a, e, f, bad);
}

}  // namespace nsm
