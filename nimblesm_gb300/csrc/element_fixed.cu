// The FP64 form's element kernel in 64-bit fixed point (hex_fixed.cuh): gather
// -> deformation gradient -> neo-Hookean or elastic Cauchy stress -> B^T
// sigma, from FP64 displacements to FP64 element forces and records.
//
// Bound: the integer pipes and issue.  On the FP64 pipe the same work is 170
// FP64 instructions per point at 16 clocks each per SM: 5.08 ms for 128^3
// elements, pipe 89% busy.  Here it is 1,190 instructions per point, 374 of
// them wide products (one per clock and SM; 530 on the multiplier's pipe), the
// others at two to four per clock: 1.10 ms (issue 46%), 1.56 ms with F and sigma
// stored; one launch on 4,096 elements 11 us against 60 us.
//
// Four lanes per element (lanes j, j + 8, j + 16, j + 24 of a warp hold the
// j-th of 8 consecutive elements; in small meshes eight, with a point each), two
// points each, in a loop that is not unrolled: the code of one point stays in
// the instruction cache (four points unrolled, two lanes per element, ran at 25%
// issue with instruction fetch the largest stall), and a small mesh waits for
// two points in a row, not eight.
// The lanes exchange 18 numbers before and 18 after.  Everything an element's
// result depends on is its own, so any launch shape gives the same bits.
//
// The warps are persistent and independent of one another: each walks groups
// of 8 elements with the next group's geometry (one 5 KB bulk copy),
// displacements (cp.async) and connectivity in flight.
//
// An element outside the fixed-point domain is evaluated by the FP64 code
// (element_work), records included, and where (nearly) all are, or the device has
// no room for this geometry, every element is (launch_element_plain).
#include <algorithm>
#include <cmath>

#include "element_work.cuh"
#include "hex_fixed.cuh"
#include "tc05.cuh"

namespace nsm {

using fx::i64;
using fx::Limbs;
using fx::u64;

// Geometry of 8 elements in fixed point, one block of kGeoRows rows of 32
// lanes (row (side along xi, value), lane [side along (zeta, eta)][element]):
// per point G0 (9 values, row-major, as limbs) and the reference volume; the
// last row holds each element's exponents and, of elastic elements, fx::Rows
// (bits 16-27).  A warp's working set is this one block, which a bulk copy
// brings to shared memory while the previous one is computed on.
constexpr int kGeoPoint = 10, kGeoRows = 2 * kGeoPoint + 1, kGeoBlock = kGeoRows * 32;  // words
constexpr int kGeoBytes = kGeoBlock * 8;

// A material that fixed_material leaves to the FP64 code.
__device__ __forceinline__ bool unfit(const FixedMaterial& m) { return (unsigned)(m.exponent + 400) > 800u; }

// From the FP64 planes: G0 scaled by 2^sG so that its largest entry over the
// points is in [2^60, 2^61) (of elastic elements each row's), the volume det J_X
// over 2^Ed (the largest in [1/2, 1)) at 2^62, and the exponents su = 124 - sG
// and Ed - sG + 2.  `never`: counts the elements that their geometry or material
// keeps out of the domain whatever their displacements.
__global__ void k_fixed_geometry(int E, long ld_e, const double* __restrict__ geo, const int* __restrict__ elem_group,
                                 const FixedMaterial* __restrict__ mats, i64* __restrict__ out, int* __restrict__ never)
{
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= E) return;
  const FixedMaterial mat     = mats[elem_group ? elem_group[e] : 0];
  const bool          elastic = mat.model == kElastic;
  double     row[3] = {0.0, 0.0, 0.0}, dmax = 0.0;
  for (int p = 0; p < 8; p++) {
    for (int q = 0; q < 9; q++) row[q / 3] = fmax(row[q / 3], fabs(geo[(p * kGeoPerPoint + q) * ld_e + e]));
    dmax = fmax(dmax, geo[(p * kGeoPerPoint + 9) * ld_e + e]);
  }
  const double gmax = fmax(row[0], fmax(row[1], row[2])), gmin = fmin(row[0], fmin(row[1], row[2]));
  int          eg = 0, ed = 0, places[3] = {0, 0, 0};
  frexp(gmax, &eg);
  frexp(dmax, &ed);
  // (values far from 1 leave the element to the FP64 code)
  bool fits = gmax > 1e-90 && gmax < 1e90 && gmin > 0.0 && dmax > 1e-60 && dmax < 1e60;
  if (elastic && fits)
    for (int d = 0; d < 3; d++) {
      int er;
      frexp(row[d], &er);
      places[d] = eg - er;
      if (places[d] > fx::kMaxRow) fits = false;
    }
  if (!fits || unfit(mat)) atomicAdd(never, 1);
  const int  sG = 61 - eg, su = fits ? 124 - sG : 1 << 20, ef = fits ? ed - sG + 2 : 0;
  const int  low = elastic && fits ? (places[0] | places[1] << 4 | places[2] << 8) << 16 | (ef & 0xffff) : ef;
  i64* const base = out + (size_t)(e >> 3) * kGeoBlock + (e & 7);
  for (int p = 0; p < 8; p++) {
    const int  y = sy_of(p), z = sz_of(p), lane = (2 * z + y) * 8;
    i64* const dst = base + sx_of(p) * kGeoPoint * 32 + lane;
    for (int q = 0; q < 9; q++) {
      const double g    = geo[(p * kGeoPerPoint + q) * ld_e + e];
      const bool   flip = (q / 3 == 1 && y == 0) || (q / 3 == 2 && z == 0);  // mirrored rows
      const Limbs  l    = fx::split(fits ? __double2ll_rn(scalbn(flip ? -g : g, sG + places[q / 3])) : 0);
      dst[q * 32]       = (i64)(((u64)(unsigned)l.hi << 32) | (unsigned)l.lo);
    }
    dst[9 * 32] = fits ? __double2ll_rn(scalbn(geo[(p * kGeoPerPoint + 9) * ld_e + e], 62 - ed)) : 0;
    if (sx_of(p) == 0) base[2 * kGeoPoint * 32 + lane] = (i64)(((u64)(unsigned)su << 32) | (unsigned)low);
  }
}

size_t fixed_geometry_words(long ld_e) { return (size_t)((ld_e + 7) / 8) * kGeoBlock; }

cudaError_t launch_fixed_geometry(int E, long ld_e, const double* geo, const int* elem_group, const FixedMaterial* mats,
                                  long long* out, int* never, cudaStream_t stream)
{
  if (E == 0) return cudaSuccess;
  k_fixed_geometry<<<grid_for(E, 128), 128, 0, stream>>>(E, ld_e, geo, elem_group, mats, out, never);
  return cudaGetLastError();
}

FixedMaterial fixed_material(const GroupMaterial& m)
{
  FixedMaterial f{0, 0, 0, 1 << 20, m.model};
  const double  most = std::fmax(m.bulk, m.shear);
  if (!std::isfinite(most) || !(most > 1e-90) || !(most < 1e90)) return f;  // left to the FP64 code
  // as are ratios of the moduli at which that is the more exact one (hex_fixed.cuh)
  if (m.model == kElastic ? m.bulk > 4.0 * m.shear : 2.0 * m.bulk < m.shear) return f;
  f.exponent = std::ilogb(most) + 4;
  f.half_k   = std::llrint(std::ldexp(m.bulk, 61 - f.exponent));
  f.shear    = std::llrint(std::ldexp(m.shear, 62 - f.exponent));
  f.lambda   = std::llrint(std::ldexp(m.bulk - 2.0 * m.shear / 3.0, 62 - f.exponent));
  return f;
}

// Largest scale of an elastic element's displacements: down to 2^-844 they have
// 57 bits, and zeros convert to zero (fx::to_fixed; at 1079 they would not).
// Smaller ones are left to the FP64 code.
constexpr int kMaxScale = 900;

template <int kXor>
__device__ __forceinline__ i64 other(i64 x)
{
  return __shfl_xor_sync(0xffffffffu, x, kXor);
}
constexpr int kAcrossXi = 4, kAcrossEta = 8, kAcrossZeta = 16;  // lane masks (xi: one point per lane)

// x 2^e, the scale added to the exponent (a product is one more instruction of
// 64 clocks a warp on the FP64 pipe, as the conversion is).
__device__ __forceinline__ double scaled(i64 x, int e)
{
  const double d = (double)x;
  return x == 0 ? 0.0 : __hiloint2double(__double2hiint(d) + (e << 20), __double2loint(d));
}

// The element as a whole on the FP64 pipe, by one lane.
__device__ __noinline__ void fallback_fp64(const ElementArgs& a, int e)
{
  element_work<double, true, GlobalNodes<double>, 0, false>(a, e, GlobalNodes<double>(a, e));
}

// The records of one point per lane: 8 consecutive records in each of four
// planes, through the warp's tile (warp_store's slots: rows of 8 chunks), 512
// contiguous bytes per instruction.  Elements outside [e_begin, E) are not
// this launch's.
__device__ __forceinline__ void store_records(const ElementArgs& a, long eb, int sx, const double* r, uint4* tile, int lane)
{
  __syncwarp();
#pragma unroll
  for (int c = 0; c < 8; c++) tile[tile_slot<8>(lane, c)] = pack16(r, c);
  __syncwarp();
  uint4* const ip = reinterpret_cast<uint4*>(a.ip);
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int  yz = k >> 1, j = (k & 1) * 32 + lane;  // chunk j of the plane's 8 records
    const int  p  = corner_of(sx, yz & 1, yz >> 1);
    const long e  = eb + (j >> 3);
    if (e >= a.e_begin && e < a.E) ip[((size_t)p * a.ld_e + eb) * 8 + j] = tile[tile_slot<8>(yz * 8 + (j >> 3), j & 7)];
  }
}

// A warp's shared memory: two geometry blocks, two sets of the lanes' nodal
// displacements, the barriers of the blocks' copies; then, where records are
// stored, their tile.
constexpr int kStageU     = 2 * kGeoBytes;
constexpr int kStageBar   = kStageU + 2 * 6 * 32 * 8;
constexpr int kStageTile  = kStageBar + 128;
constexpr int kStageBytes = kStageTile, kStageBytesStore = kStageTile + 32 * 128;
static_assert(kStageTile % 128 == 0 && kGeoBytes % 16 == 0, "alignment");

__device__ __forceinline__ void load_g0(const i64* gp, Limbs g0[3][3])
{
#pragma unroll
  for (int q = 0; q < 9; q++) {
    const i64 w      = gp[q * 32];
    g0[q / 3][q % 3] = Limbs{(int)(w >> 32), (int)w};
  }
}

// Whether each of a warp's elements has a lane that reports it.
template <int kElems>
__device__ __forceinline__ bool none_inside(unsigned bad)
{
  unsigned b = __ballot_sync(0xffffffffu, bad != 0);
  if (kElems == 4) b |= b >> 4;
  b |= b >> 8;
  b |= b >> 16;
  return (~b & ((1u << kElems) - 1)) == 0;
}

// The block's elements that are left to the FP64 code, collected in the staging
// (`room` ints per warp) and evaluated 32 to a warp: the FP64 pipe takes a warp
// instruction as long for 8 lanes as for 32.  A block's warps have neighbouring
// groups, so a round of its loop is `span` consecutive elements.  The first
// batch falls to another warp, another scheduler, in every quarter of the grid,
// since a small mesh has one batch per block and four blocks on an SM.  A mesh
// turned by 0.6 takes 57 to 63 us a step up to 8,000 elements, 85 at 21,952, 756
// at 262,144 and 5,690 at 2,097,152 (by one lane per element, 8 to a warp, 58 to
// 154, 255, 2,770 and 21,730 us; without the fixed-point code, every element in
// FP64, 58 to 64, 104, 697 and 5,260): the pipe 85% busy, after 0.35 ms in which
// the fixed-point code finds them outside.  A quarter of 2,097,152 elements beyond
// the domain: 2.4 ms.  (Evaluated between rounds, beside other blocks' fixed-point
// work: 5.6 ms, but 9% more for meshes inside the domain, whose loop loses the
// registers of the call.)
template <int kElems>
__device__ __noinline__ void left_to_fp64(const ElementArgs& a, int* queue, int room)
{
  const int  lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5, span = warps * kElems;
  const int  rounds = (warps * room - 1) / span;  // that the queue holds; queue[0]: its length
  const long step   = (long)gridDim.x * span;
  for (long e0 = (long)(a.e_begin / kElems) * kElems + (long)blockIdx.x * span; e0 < a.E; e0 += rounds * step) {
    __syncthreads();
    if (threadIdx.x == 0) queue[0] = 0;
    __syncthreads();
    for (int r = warp; r < rounds && e0 + r * step < a.E; r += warps) {
      const long     e    = e0 + r * step + lane;
      const bool     left = lane < span && e >= a.e_begin && e < a.E && a.elem_left[e];
      const unsigned m    = __ballot_sync(0xffffffffu, left);
      if (m == 0) continue;
      int at = lane == 0 ? atomicAdd(queue, __popc(m)) : 0;
      at     = __shfl_sync(0xffffffffu, at, 0);
      if (left) queue[1 + at + __popc(m & ((1u << lane) - 1))] = (int)e;
    }
    __syncthreads();
    const int n = queue[0], turn = (int)(4u * blockIdx.x / gridDim.x);
    __syncthreads();
    if (threadIdx.x == 0) queue[0] = warps;  // the next batch that no warp has
    __syncthreads();
    for (int b = (warp + turn) % warps; b * 32 < n;) {
      if (b * 32 + lane < n) fallback_fp64(a, queue[1 + b * 32 + lane]);
      __syncwarp();
      if (lane == 0) b = atomicAdd(queue, 1);
      b = __shfl_sync(0xffffffffu, b, 0);
    }
  }
}

// kStore: F and sigma are formed and stored when the launch asks for it.
// kHasElastic: some material of the model is elastic.
// kPoints: points per lane.  1 (small meshes; without records): two lanes share
// what a lane does otherwise, each with one of the two points; the transforms
// before and after are done by both.
template <bool kStore, bool kHasElastic>
constexpr int kBlocks = kStore || kHasElastic ? 3 : 4;  // per SM
template <bool kStore, bool kHasElastic, int kPoints>
__global__ void __launch_bounds__(128, kBlocks<kStore, kHasElastic>) k_element_fixed(ElementArgs a)
{
  static_assert(kPoints == 2 || (kPoints == 1 && !kStore), "points per lane");
  constexpr int  kElems = 4 * kPoints;  // of a warp, half a geometry block or a whole one
  extern __shared__ __align__(128) uint8_t stage_all[];
  const int      lane = threadIdx.x & 31, warp = threadIdx.x >> 5, j = lane & (kElems - 1), y = (lane >> 3) & 1, z = lane >> 4;
  const int      side = kPoints == 1 ? (lane >> 2) & 1 : 0;  // of this lane's point along xi
  const long     ld_e = a.ld_e, ld_n = a.ld_n;
  uint8_t* const stage = stage_all + warp * (kStore ? kStageBytesStore : kStageBytes);
  double* const  us    = reinterpret_cast<double*>(stage + kStageU) + lane;  // [2][6][32]
  i64* const     us_i  = reinterpret_cast<i64*>(us);
  uint64_t*      bar   = reinterpret_cast<uint64_t*>(stage + kStageBar);
  const bool     store =
      kStore && (a.store_ip == kStoreAlways || (a.sched != nullptr && a.sched[(long)(*a.step_base + a.k) * a.num_groups].is_output));
  const int* const conn = a.conn + (long)(corner_of(0, y, 0) + 4 * z) * ld_e;
  const long       next_corner = (corner_of(1, y, 0) - corner_of(0, y, 0)) * ld_e;

  // groups of kElems elements; those at the ends of [e_begin, E) may be partial
  const long g_end = (a.E + kElems - 1) / kElems, g_step = (long)gridDim.x * (blockDim.x >> 5);
  long       g     = a.e_begin / kElems + (long)blockIdx.x * (blockDim.x >> 5) + warp;
  auto load_ids = [&](long gr, int id[2]) {
    const long e = min(gr * kElems + j, (long)a.E - 1);  // (spare lanes repeat the last element)
    id[0]        = __ldg(&conn[e]);
    id[1]        = __ldg(&conn[e + next_corner]);
  };
  auto stage_u = [&](int buf, const int id[2]) {
#pragma unroll
    for (int bx = 0; bx < 2; bx++)
#pragma unroll
      for (int i = 0; i < 3; i++) cp_async8(us + (buf * 6 + i * 2 + bx) * 32, a.u + i * ld_n + id[bx]);
  };
  auto stage_geo = [&](int buf, long gr) {
    if (lane == 0) tc::bulk_load(stage + buf * kGeoBytes, a.geo_fixed + gr * kElems / 8 * kGeoBlock, kGeoBytes, &bar[buf]);
  };
  if (lane == 0) {
    tc::mbar_init(&bar[0], 1);
    tc::mbar_init(&bar[1], 1);
    tc::fence_mbar_init();
  }
  __syncwarp();
  int id[2];
  if (g < g_end) {
    load_ids(g, id);
    stage_geo(0, g);
  }
  wait_prerequisites();  // the node kernel that writes u
  launch_dependents();
  if (g < g_end) stage_u(0, id);
  cp_async_commit();
  if (g + g_step < g_end) load_ids(g + g_step, id);

  unsigned any_bad = 0;
  bool     gave_up = false;
  uint32_t phase = 0;  // bit b: parity of block b's next copy
  for (int buf = 0; g < g_end; g += g_step, buf ^= 1) {
    cp_async_wait_all();
    if (!tc::mbar_wait_warp(&bar[buf], (phase >> buf) & 1u)) {
      // Given up, as a warp.  Once more for the late copy, so that it does not
      // land in another block's memory; nothing else of this warp is in flight.
      tc::mbar_wait_warp(&bar[buf], (phase >> buf) & 1u);
      if (lane == 0) atomicOr(a.status, NSM_STATUS_COPY_TIMEOUT);
      gave_up = true;
      break;
    }
    phase ^= 1u << buf;
    if (g + g_step < g_end) {
      stage_geo(buf ^ 1, g + g_step);
      stage_u(buf ^ 1, id);
      cp_async_commit();
      if (g + 2 * g_step < g_end) load_ids(g + 2 * g_step, id);
    }
    const long       eb    = g * kElems;
    const int        e     = (int)min(eb + j, (long)a.E - 1);
    const bool       valid = eb + j >= a.e_begin && eb + j < a.E;
    // the lane's column of the block
    i64* const       gs    = reinterpret_cast<i64*>(stage + buf * kGeoBytes) + (kPoints == 2 ? lane : (lane & 24) + (eb & 4) + j);

    // ---- displacements of the lane's two corners, at 2^sc ----
    u64      u[3][2];
    int      exm = 0;
    unsigned low = 0;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int bx = 0; bx < 2; bx++) {
        u[i][bx] = (u64)__double_as_longlong(us[(buf * 6 + i * 2 + bx) * 32]);
        exm      = max(exm, (int)((unsigned)(u[i][bx] >> 32) & 0x7fffffffu));
        low |= (unsigned)u[i][bx];
      }
    if (kHasElastic) exm = max(exm, low != 0);
    exm = max(exm, __shfl_xor_sync(0xffffffffu, exm, kAcrossEta));
    exm = max(exm, __shfl_xor_sync(0xffffffffu, exm, kAcrossZeta));
    // (of all 24 numbers: none but zeros, or the largest one's exponent)
    const bool at_rest = exm == 0;
    exm >>= 20;
    const i64           ge      = gs[2 * kGeoPoint * 32];
    const FixedMaterial mat     = a.fixed_mats[a.elem_group ? __ldg(&a.elem_group[e]) : 0];
    const bool          elastic = kHasElastic && mat.model == kElastic;
    const int           su      = (int)(ge >> 32);
    int                 sc      = min(1079 - exm, elastic ? kMaxScale : su);
    int                 ef      = (int)ge;
    fx::Rows            rows    = {0, 0, 0};
    int                 sh = su - sc, ee = 0;
    unsigned bad = unfit(mat);
    // An infinity or a NaN, or numbers whose sums may become one (2^1017 and
    // more): an elastic element's modes do not show it, as the same value at all
    // corners leaves nothing in any difference.
    if (kHasElastic) bad |= exm > 0x7f7;
    if (kHasElastic && elastic) {
      bad |= exm < 1079 - kMaxScale && !at_rest;  // (shorter than 57 bits at the largest scale)
      rows = fx::Rows{ef >> 16 & 15, ef >> 20 & 15, ef >> 24 & 15};
      ef   = (int)(short)ef;
    }

    // ---- modes and gradients ----
    fx::Gradient G[3];
    {
      i64 v[3][7];
#pragma unroll
      for (int i = 0; i < 3; i++) {
        const i64 c0 = fx::to_fixed((unsigned)(u[i][0] >> 32), (unsigned)u[i][0], 1086 - sc);
        const i64 c1 = fx::to_fixed((unsigned)(u[i][1] >> 32), (unsigned)u[i][1], 1086 - sc);
        const i64 s = c1 + c0, d = c1 - c0;
        const i64 so = other<kAcrossEta>(s), dn = other<kAcrossEta>(d);
        i64       q[2][2] = {{s + so, d + dn}, {s - so, d - dn}}, o[2][2];
#pragma unroll
        for (int k = 0; k < 4; k++) o[k >> 1][k & 1] = other<kAcrossZeta>(q[k >> 1][k & 1]);
        fx::lane_modes(q, o, v[i]);
      }
      if (kHasElastic && __any_sync(0xffffffffu, elastic)) {
        u64 m = 0;
#pragma unroll
        for (int i = 0; i < 3; i++) m |= fx::mode_bits(v[i], rows);
        m |= (u64)other<kAcrossEta>((i64)m);
        m |= (u64)other<kAcrossZeta>((i64)m);
        if (elastic) {
          if (m == 0) sh = 0;
          else fx::elastic_scale(64 - fx::kMaxRow - __clzll((i64)m), sc, su, sh, ee);
          // strains above the domain; forces or stresses that are not normal numbers
          if (ee < -3 || min(ef, 0) + mat.exponent - ee < -900) bad = 1, sh = 0, ee = 0;
#pragma unroll
          for (int i = 0; i < 3; i++) fx::elastic_shift(v[i], rows, sh);
        }
      }
      if (!elastic && sh != 0) {
        if (sh > 26) bad = 1, sh = 26;
#pragma unroll
        for (int i = 0; i < 3; i++) bad |= fx::lane_shift(v[i], sh);
      }
#pragma unroll
      for (int i = 0; i < 3; i++) {
        if (kHasElastic) fx::elastic_gradient(v[i], rows, G[i]);
        else fx::lane_gradient(v[i], G[i]);
        if (kPoints == 2) {  // the second point's increments wait where the displacements were
          us_i[(buf * 6 + i) * 32]     = G[i].y1;
          us_i[(buf * 6 + 3 + i) * 32] = G[i].z1;
        }
      }
    }

    // ---- the lane's two points ----
    // What a point does not need while it is computed waits in shared memory
    // (registers spilled to local memory would miss the small L1 that the
    // staging leaves): G0 is read twice, and the first point's forces are kept
    // in its own geometry rows.
    i64              Q[3][3];
    const fx::Moduli mod{mat.half_k, mat.shear, mat.lambda, mat.exponent, mat.model};
    i64*             gp = gs + side * kGeoPoint * 32;
    // All of the warp's elements outside by their modes already: only that is left
    // to say.  (From the second round on: small meshes wait for the vote.)
    const bool none = kPoints == 2 && g >= a.e_begin / kElems + g_step && none_inside<kElems>(bad);
    if (side) {
#pragma unroll
      for (int i = 0; i < 3; i++) G[i].y += G[i].y1, G[i].z += G[i].z1;
    }
#pragma unroll 1
    for (int sx = 0; sx < (none ? 0 : kPoints); sx++, gp += kGeoPoint * 32) {
      i64 P[3][3];
      {
        Limbs g0[3][3];
        load_g0(gp, g0);
        i64 Du[3][3];
#pragma unroll
        for (int i = 0; i < 3; i++) Du[i][0] = G[i].x, Du[i][1] = G[i].y, Du[i][2] = G[i].z;
        const i64 det = gp[9 * 32];
        fx::Point pt;
        i64       He[3][3];
        if (kHasElastic && elastic) {
          const int up = max(-ee, 0), down = min(max(ee, 0), 63);
          fx::displacement_gradient<true>(Du, g0, He);
#pragma unroll
          for (int q = 0; q < 9; q++) {
            pt.H[q / 3][q % 3] = (i64)((u64)He[q / 3][q % 3] << up) >> down;
            bad |= fx::outside<27>(pt.H[q / 3][q % 3]);  // (|H|^2 below would not show it)
          }
        } else {
          fx::displacement_gradient(Du, g0, pt.H);
        }
        bad |= fx::kinematics(pt);
        if (kHasElastic && elastic) bad |= fx::elastic_force<kStore>(mod, det, He, pt, P);
        else bad |= fx::neohookean_force<kStore>(mod, det, pt, P);
        if (store) {
          double       r[kIpRecord];
#pragma unroll
          for (int i = 0; i < 3; i++)
#pragma unroll
            for (int k = 0; k < 3; k++)
              r[full_slot(i, k)] = scaled(pt.H[i][k] + (i == k ? fx::kOne : 0), -60);
#pragma unroll
          for (int q = 0; q < 6; q++) r[9 + q] = scaled(pt.sig[q], mat.exponent - ee - 62);
          r[15] = 0.0;
          store_records(a, eb, sx, r, reinterpret_cast<uint4*>(stage + kStageTile), lane);
        }
      }
      asm volatile("" ::: "memory");  // G0 is read again rather than kept
      Limbs g0[3][3];
      load_g0(gp, g0);
      fx::point_force(g0, P, Q);
      if (kPoints == 1) {
#pragma unroll
        for (int q = 0; q < 9; q++) gp[q * 32] = Q[q / 3][q % 3];
      } else if (sx == 0) {
#pragma unroll
        for (int q = 0; q < 9; q++) gp[q * 32] = Q[q / 3][q % 3];
#pragma unroll
        for (int i = 0; i < 3; i++) {
          G[i].y += us_i[(buf * 6 + i) * 32];
          G[i].z += us_i[(buf * 6 + 3 + i) * 32];
        }
      }
    }

    if (none) {
      bad = 1;
    } else {
      // ---- nodal forces of the lane's corners ----
      ef += mat.exponent - ee - (elastic ? fx::kElasticForce - fx::kElasticSum : 0);
      const double scale = __longlong_as_double((i64)(1023 + ef) << 52);
      double       f[2][3];
      if (kPoints == 1) {  // both lanes' forces
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 9; q++) Q[q / 3][q % 3] = gs[(kGeoPoint + q) * 32];
      }
#pragma unroll
      for (int i = 0; i < 3; i++) {
        const i64      qx = gs[i * 32], qy = gs[(3 + i) * 32], qz = gs[(6 + i) * 32];
        fx::Sums       S{Q[0][i] + qx, Q[1][i] + qy, Q[1][i] - qy, Q[2][i] + qz, Q[2][i] - qz};
        fx::Parts      keep, send;
        if (elastic) {
          fx::common_scale(S, rows);
          bad |= fx::too_large(S);
        }
        fx::lane_adjoint(S, keep, send);
        const i64 e0 = keep.e0 + other<kAcrossZeta>(send.e0), e1 = keep.e1 + other<kAcrossZeta>(send.e1);
        const i64 o0 = keep.o0 + other<kAcrossZeta>(send.o0), o1 = keep.o1 + other<kAcrossZeta>(send.o1);
        const i64 ev = (e0 + e1) + other<kAcrossEta>(e0 - e1), od = (o0 + o1) + other<kAcrossEta>(o0 - o1);
        f[0][i] = (double)(od - ev) * scale;
        f[1][i] = (double)(-od - ev) * scale;
      }
      if (kPoints == 1) bad |= __shfl_xor_sync(0xffffffffu, bad, kAcrossXi);
      bad |= __shfl_xor_sync(0xffffffffu, bad, kAcrossEta);
      bad |= __shfl_xor_sync(0xffffffffu, bad, kAcrossZeta);
      if (bad == 0 && valid) {
        double* const fe = reinterpret_cast<double*>(a.fe) + e;
#pragma unroll
        for (int bx = 0; bx < 2; bx++)
          if (kPoints == 2 || bx == side) {
#pragma unroll
            for (int i = 0; i < 3; i++) fe[(size_t)(3 * (corner_of(bx, y, 0) + 4 * z) + i) * ld_e] = f[bx][i];
          }
      }
    }
    // which elements are left to the FP64 code
    any_bad |= bad;
    if (y == 0 && z == 0 && side == 0 && valid) a.elem_left[e] = bad != 0;
    tc::fence_proxy_async();  // this lane's writes to the block come before the next copy into it
    __syncwarp();             // this group's staged data are read, its records written
  }
  // (after the loop: a call inside it would spill the loop's state)
  if (!__syncthreads_or(any_bad != 0)) return;
  if (__syncthreads_or(gave_up)) return;  // a late copy may still change the staging
  if (lane == 0) {  // which is used otherwise from here on
    tc::mbar_inval(&bar[0]);
    tc::mbar_inval(&bar[1]);
  }
  left_to_fp64<kElems>(a, reinterpret_cast<int*>(stage_all), (kStore ? kStageBytesStore : kStageBytes) / 4);
}

// Blocks of 128 threads, four warps, four blocks per SM: 16 warps of 128
// registers and 14 KB of staging.  Three where records are stored or elastic
// elements would spill: 64,000 of them 53.9 us a step, 58.6 with four.
template <bool kStore, bool kHasElastic, int kPoints>
static cudaError_t launch_fixed(const ElementArgs& a, const ElementLaunch& l, cudaStream_t stream)
{
  constexpr int     bytes = kStore ? kStageBytesStore : kStageBytes;
  static std::atomic<unsigned long long> configured{0};
  cudaError_t err = once_per_device(configured, [] {
    cudaError_t e =
        cudaFuncSetAttribute(k_element_fixed<kStore, kHasElastic, kPoints>, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * bytes);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_element_fixed<kStore, kHasElastic, kPoints>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    return e;
  });
  if (err != cudaSuccess) return err;
  const int  warps  = l.block == 64 ? 2 : 4;
  constexpr int kElems = 4 * kPoints;
  const long groups = (a.E + kElems - 1L) / kElems - a.e_begin / kElems;
  const int  per_sm = l.persistent ? l.blocks_per_sm : kBlocks<kStore, kHasElastic> * (4 / warps);
  const long blocks = (groups + warps - 1) / warps, fit = (long)per_sm * num_sms();
  // One block fewer past eight rounds: its 32 elements a round are then a stretch
  // of the mesh elsewhere in each (608 blocks of 32 come back to the same quarter
  // of a row of 128), and elements outside the domain are spread over all blocks.
  const long grid   = blocks <= 8 * fit ? std::min(blocks, fit) : std::max(1L, fit - 1);
  return launch_overlapped(k_element_fixed<kStore, kHasElastic, kPoints>, (int)grid, 32 * warps, warps * bytes, stream, a.overlap != 0, a);
}

// One point per lane as long as that gives none of the chip's schedulers (four
// per SM) a second warp of 4 elements: a step of 100 elements 7.6 us with two
// points per lane, 6.4 with one; 1,728 elements 8.8 and 7.7 (elastic blocks
// beside neo-Hookean ones 11.6 and 10.6); 4,096 9.7 and 9.9 (13.0 and 12.6);
// 8,000 12.0 and 13.2.
cudaError_t launch_element_fp64(const ElementArgs& a, const ElementLaunch& l, cudaStream_t stream)
{
  if (a.E <= a.e_begin) return cudaSuccess;
  if (!a.geo_fixed) return launch_element_plain(a, stream);
  if (a.store_ip != kStoreNever)
    return a.has_elastic ? launch_fixed<true, true, 2>(a, l, stream) : launch_fixed<true, false, 2>(a, l, stream);
  if (a.E - a.e_begin <= 4 * 4 * num_sms())
    return a.has_elastic ? launch_fixed<false, true, 1>(a, l, stream) : launch_fixed<false, false, 1>(a, l, stream);
  return a.has_elastic ? launch_fixed<false, true, 2>(a, l, stream) : launch_fixed<false, false, 2>(a, l, stream);
}

}  // namespace nsm
