// Fused hex8 element kernel of the FP32-mixed form: gather -> deformation
// gradient -> neo-Hookean or elastic Cauchy stress -> B^T sigma, one thread per
// element; the two passes of models with block-material callbacks (FP32 and
// FP64); the FP64 form without its fixed-point geometry; energies and the layout
// conversions.  The FP64 form's fused kernel is element_fixed.cu; the element
// math and the reasons for its form are in hex_math.cuh.
#include <algorithm>

#include "element_packed.cuh"
#include "element_work.cuh"

namespace nsm {

// One thread per element, or (persistent form) a fixed grid of blocks walking
// the elements of all samples in tiles of blockDim.x.
template <typename T, bool kPrecomputedGeo, bool kPersistent, int kMinBlocks = 1, int kPass = 0>
__global__ void __launch_bounds__(128, kMinBlocks) k_element(ElementArgs a)
{
  if constexpr (!kPersistent) {
    const int e = a.e_begin + blockIdx.x * blockDim.x + threadIdx.x;
    if (e < a.E) element_work<T, kPrecomputedGeo, GlobalNodes<T>, kPass>(a, e, GlobalNodes<T>(a, e));
  } else {
    for (long e = a.e_begin + blockIdx.x * (long)blockDim.x + threadIdx.x; e < a.E;
         e += (long)gridDim.x * blockDim.x)
      element_work<T, kPrecomputedGeo>(a, (int)e, GlobalNodes<T>(a, (int)e));
  }
}

// Staged FP32 form: a persistent grid in which each thread walks the elements
// e, e + stride, ... with the next element's 48 nodal values (u and X) and the
// connectivity of the one after in flight as cp.async copies into its own
// shared-memory columns while it computes the current element.  Neither the
// connectivity load nor the gather it addresses stalls the element math, and
// nothing staged is held in registers.  Copy groups are per thread and each
// thread reads only its own columns: no block barrier is needed.

// Per thread and slot: kStageValues 16-byte records (0..7 u, 8..15 X), then 8
// connectivity entries; column stride B.  Two slots, for the element being
// computed and the next one.  One record per node and field: in a mesh without
// locality every gathered value is a 32-byte sector of its own, and three
// 4-byte planes per field made that three times as many.
constexpr int kStageBytes = kStageValues * 16 + 8 * 4;

__device__ __forceinline__ void stage_conn(const ElementArgs& a, long e, int* col, int B)
{
#pragma unroll
  for (int n = 0; n < 8; n++) cp_async4(col + n * B, a.conn + n * a.ld_e + e);
}

__device__ __forceinline__ void stage_nodes(const ElementArgs& a, const int* conn_col, float4* col, int B)
{
#pragma unroll
  for (int n = 0; n < 8; n++) {
    const int id = conn_col[n * B];
    cp_async16(col + n * B, a.uf + id);
    cp_async16(col + (8 + n) * B, a.Xf + id);
  }
}

// kPacked: two points per operation (element_packed.cuh).
template <bool kPacked>
__global__ void __launch_bounds__(128, 3) k_element_staged(ElementArgs a)
{
  extern __shared__ __align__(16) uint8_t stage_mem[];  // [2][16][blockDim.x] float4, then [2][8][blockDim.x] int
  const int  B      = blockDim.x;
  const long stride = (long)gridDim.x * B;
  float4*    cur    = reinterpret_cast<float4*>(stage_mem) + threadIdx.x;  // the element being computed
  float4*    nxt    = cur + kStageValues * B;                              // the next one
  int*       ccur   = reinterpret_cast<int*>(stage_mem + 2 * kStageValues * 16 * B) + threadIdx.x;
  int*       cnxt   = ccur + 8 * B;
  long       e      = a.e_begin + blockIdx.x * (long)B + threadIdx.x;
  // prologue: connectivity of e (waited for), its nodal values and the
  // connectivity of e + stride in flight
  if (e < a.E) stage_conn(a, e, ccur, B);
  cp_async_commit();
  cp_async_wait_all();
  wait_prerequisites();  // the node kernel that writes u
  launch_dependents();
  if (e < a.E) stage_nodes(a, ccur, cur, B);
  if (e + stride < a.E) stage_conn(a, e + stride, cnxt, B);
  cp_async_commit();
  for (; e < a.E; e += stride) {
    cp_async_wait_all();  // this element's values and the next one's connectivity
    if (e + stride < a.E) stage_nodes(a, cnxt, nxt, B);
    if (e + 2 * stride < a.E) stage_conn(a, e + 2 * stride, ccur, B);
    cp_async_commit();
    if constexpr (kPacked) element_work_packed(a, (int)e, StagedNodes{cur, B});
    else element_work<float, false>(a, (int)e, StagedNodes{cur, B});
    // a whole warp's tile has been read before a lane's next copies arrive in it
    if (a.store_ip != kStoreNever && e - (threadIdx.x & 31) + 32 <= a.E) __syncwarp();
    float4* t = cur;
    cur       = nxt;
    nxt       = t;
    int* c    = ccur;
    ccur      = cnxt;
    cnxt      = c;
  }
  cp_async_wait_all();
}

// Point records before the first evaluation: F = I, sigma = 0, as the
// reference initialises its element data.
template <typename T>
__global__ void k_ip_identity(int E, long ld_e, T* __restrict__ ip)
{
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= E) return;
  for (int p = 0; p < 8; p++) {
    T* rec = ip + ((size_t)p * ld_e + e) * kIpRecord;
#pragma unroll
    for (int i = 0; i < 3; i++) rec[full_slot(i, i)] = T(1);
  }
}

cudaError_t launch_ip_identity(int E, long ld_e, void* ip, int ip_is_float, cudaStream_t stream)
{
  if (E == 0) return cudaSuccess;
  if (ip_is_float)
    k_ip_identity<float><<<grid_for(E, 128), 128, 0, stream>>>(E, ld_e, (float*)ip);
  else
    k_ip_identity<double><<<grid_for(E, 128), 128, 0, stream>>>(E, ld_e, (double*)ip);
  return cudaGetLastError();
}

int num_sms()
{
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 1;
  }
  return n;
}

cudaError_t launch_element_pass(const ElementArgs& a, int is_float, int pass, cudaStream_t stream)
{
  if (a.E <= a.e_begin) return cudaSuccess;
  const int grid = grid_for(a.E - a.e_begin, 128);
  if (pass != 1 && pass != 2) return cudaErrorInvalidValue;
  if (is_float) {
    if (pass == 1)
      k_element<float, false, false, 3, 1><<<grid, 128, 0, stream>>>(a);
    else
      k_element<float, false, false, 3, 2><<<grid, 128, 0, stream>>>(a);
  } else {
    if (pass == 1)
      k_element<double, true, false, 1, 1><<<grid, 128, 0, stream>>>(a);
    else
      k_element<double, true, false, 1, 2><<<grid, 128, 0, stream>>>(a);
  }
  return cudaGetLastError();
}

cudaError_t launch_element_plain(const ElementArgs& a, cudaStream_t stream)
{
  k_element<double, true, false, 3><<<grid_for(a.E - a.e_begin, 128), 128, 0, stream>>>(a);
  return cudaGetLastError();
}

template <bool kPacked>
static cudaError_t launch_staged(const ElementArgs& a, const ElementLaunch& l, int block, cudaStream_t stream)
{
  static std::atomic<unsigned long long> configured{0};
  cudaError_t err = once_per_device(configured, [] {  // 72 KB at 128 threads: above the default 48 KB of dynamic shared memory
    cudaError_t e = cudaFuncSetAttribute(k_element_staged<kPacked>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         2 * kStageBytes * 128);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_element_staged<kPacked>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    return e;
  });
  if (err != cudaSuccess) return err;
  ElementArgs b    = a;
  b.persistent     = 1;
  const int   grid = std::min(grid_for(a.E - a.e_begin, block), (l.blocks_per_sm > 0 ? l.blocks_per_sm : 1) * num_sms());
  return launch_overlapped(k_element_staged<kPacked>, grid, block, 2 * kStageBytes * block, stream, a.overlap != 0, b);
}

cudaError_t launch_element_fp32(const ElementArgs& a, const ElementLaunch& l, cudaStream_t stream)
{
  if (a.E <= a.e_begin) return cudaSuccess;
  const int block = (l.block == 64 || l.block == 128) ? l.block : 128;
  if (!l.staged) {  // registers bounded for 3 blocks of 128 per SM (measured fastest)
    const int grid = grid_for(a.E - a.e_begin, block);
    if (l.persistent) {
      ElementArgs b = a;
      b.persistent  = 1;
      k_element<float, false, true, 3><<<std::min(grid, l.blocks_per_sm * num_sms()), block, 0, stream>>>(b);
    } else {
      k_element<float, false, false, 3><<<grid, block, 0, stream>>>(a);
    }
    return cudaGetLastError();
  }
  return a.store_ip == kStoreNever && !a.has_elastic ? launch_staged<true>(a, l, block, stream)
                                                     : launch_staged<false>(a, l, block, stream);
}

// Energies of the current state, FP64 whatever the element precision:
// kinetic 1/2 m v.v per node and internal det J_X W(F) per point, with H
// rebuilt from u (so an FP32 F store does not limit the energy's accuracy).
// Per-block partial sums in a fixed order, then one block: deterministic.
__global__ void __launch_bounds__(128) k_energy_partials(int N, long ld_n, const double* __restrict__ mass,
                                                         const double* __restrict__ v, int E, long ld_e,
                                                         const int* __restrict__ conn, const double* __restrict__ u,
                                                         const double* __restrict__ geo,
                                                         const int* __restrict__ elem_group,
                                                         const GroupMaterial* __restrict__ mats,
                                                         double* __restrict__ partial)
{
  __shared__ double s_ke[128], s_ie[128];
  double            ke = 0.0, ie = 0.0;
  for (long n = blockIdx.x * (long)blockDim.x + threadIdx.x; n < N; n += (long)gridDim.x * blockDim.x) {
    double vx = v[n], vy = v[ld_n + n], vz = v[2 * ld_n + n];
    ke += 0.5 * mass[n] * (vx * vx + vy * vy + vz * vz);
  }
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < E; e += (long)gridDim.x * blockDim.x) {
    double x[8][3];
#pragma unroll
    for (int c = 0; c < 8; c++) {
      int id = conn[c * ld_e + e];
#pragma unroll
      for (int k = 0; k < 3; k++) x[c][k] = u[k * ld_n + id];
    }
    double Gu[3][3][2][2];
    nodal_gradient<double>(x, Gu);
    const GroupMaterial& mat = mats[elem_group ? elem_group[e] : 0];
    const double         K = mat.bulk, Gm = mat.shear;
    const bool           elastic_model = mat.model == kElastic;
#pragma unroll 1
    for (int p = 0; p < 8; p++) {
      const int bit[3] = {sx_of(p), sy_of(p), sz_of(p)};
      double    G0[3][3];
      for (int q = 0; q < 9; q++) G0[q / 3][q % 3] = geo[(p * kGeoPerPoint + q) * ld_e + e];
      double H[3][3];
      for (int i = 0; i < 3; i++)
        for (int J = 0; J < 3; J++) {
          double h = 0.0;
          for (int d = 0; d < 3; d++) {
            const int o1 = other1(d), o2 = other2(d);
            h += Gu[d][i][bit[o1]][bit[o2]] * G0[d][J];
          }
          H[i][J] = h;
        }
      // (a block whose stress a callback computes has no energy density here)
      if (mat.model != kExternal)
        ie += geo[(p * kGeoPerPoint + 9) * ld_e + e] *
              (elastic_model ? energy_density_elastic(H, K, Gm) : energy_density(H, K, Gm));
    }
  }
  s_ke[threadIdx.x] = ke;
  s_ie[threadIdx.x] = ie;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      s_ke[threadIdx.x] += s_ke[threadIdx.x + w];
      s_ie[threadIdx.x] += s_ie[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    partial[2 * blockIdx.x]     = s_ke[0];
    partial[2 * blockIdx.x + 1] = s_ie[0];
  }
}

__global__ void k_energy_final(int nblocks, const double* __restrict__ partial, double* __restrict__ out)
{
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  double ke = 0.0, ie = 0.0;
  for (int b = 0; b < nblocks; b++) {
    ke += partial[2 * b];
    ie += partial[2 * b + 1];
  }
  out[0] = ke;
  out[1] = ie;
}

cudaError_t launch_energies(int N, long ld_n, const double* mass, const double* v, int E, long ld_e,
                            const int* conn, const double* u, const double* geo, const int* elem_group,
                            const GroupMaterial* mats, double* partial, double* out, cudaStream_t stream)
{
  const int blocks = kEnergyBlocks;
  k_energy_partials<<<blocks, 128, 0, stream>>>(N, ld_n, mass, v, E, ld_e, conn, u, geo, elem_group, mats, partial);
  k_energy_final<<<1, 32, 0, stream>>>(blocks, partial, out);
  return cudaGetLastError();
}

// Per-point records ip[(p*ld_e + e)*16 + slot] -> reference layout
// dst[(e*8 + p)*comps + c] in doubles (F: slots 0..8, sigma: slots 9..14).
template <typename T>
__global__ void k_ip_to_aos(int E, long ld_e, const T* __restrict__ ip, int which, double* __restrict__ dst)
{
  const int comps = which == 0 ? 9 : 6, first = which == 0 ? 0 : 9;
  long      i     = blockIdx.x * (long)blockDim.x + threadIdx.x;
  long      total = (long)E * 8 * comps;
  if (i >= total) return;
  int  c = (int)(i % comps);
  long r = i / comps;
  int  p = (int)(r % 8);
  long e = r / 8;
  dst[i] = (double)ip[((size_t)p * ld_e + e) * kIpRecord + first + c];
}

cudaError_t launch_ip_to_aos(int E, long ld_e, const void* ip, int src_is_float, int which, double* dst,
                             cudaStream_t stream)
{
  long total = (long)E * 8 * (which == 0 ? 9 : 6);
  if (total == 0) return cudaSuccess;
  if (src_is_float)
    k_ip_to_aos<float><<<grid_for(total, 256), 256, 0, stream>>>(E, ld_e, (const float*)ip, which, dst);
  else
    k_ip_to_aos<double><<<grid_for(total, 256), 256, 0, stream>>>(E, ld_e, (const double*)ip, which, dst);
  return cudaGetLastError();
}

// Per-sample max |x| over listed nodes; values are non-negative doubles, so
// their bit patterns order like 64-bit integers and atomicMax on the bits is
// an exact, order-independent maximum.
__global__ void k_group_max_abs(int count, const int* __restrict__ nodes, const double* __restrict__ field, long ld_n,
                                int component, const int* __restrict__ node_group, unsigned long long* out)
{
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  int    n = nodes[i];
  double v = fabs(field[component * ld_n + n]);
  int    g = node_group ? node_group[n] : 0;
  atomicMax(&out[g], (unsigned long long)__double_as_longlong(v));
}

cudaError_t launch_group_max_abs(int count, const int* nodes, const double* field, long ld_n, int component,
                                 const int* node_group, int num_groups, double* out, cudaStream_t stream)
{
  cudaError_t e = cudaMemsetAsync(out, 0, sizeof(double) * num_groups, stream);
  if (e != cudaSuccess || count == 0) return e;
  k_group_max_abs<<<grid_for(count, 256), 256, 0, stream>>>(count, nodes, field, ld_n, component, node_group,
                                                            reinterpret_cast<unsigned long long*>(out));
  return cudaGetLastError();
}

// FP64 planes to the FP32 form's records {x, y, z, 0} of the nodes.
__global__ void k_to_records(int N, long ld_n, const double* __restrict__ src, float4* __restrict__ dst)
{
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n < N) dst[n] = make_float4((float)src[n], (float)src[ld_n + n], (float)src[2 * ld_n + n], 0.0f);
}

cudaError_t launch_to_records(int N, long ld_n, const double* src, float4* dst, cudaStream_t stream)
{
  if (N == 0) return cudaSuccess;
  k_to_records<<<grid_for(N, 256), 256, 0, stream>>>(N, ld_n, src, dst);
  return cudaGetLastError();
}

__global__ void k_node_soa_to_aos(int N, long ld_n, const double* __restrict__ src, double* __restrict__ dst)
{
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= 3L * N) return;
  dst[i] = src[(i % 3) * ld_n + i / 3];
}

__global__ void k_node_aos_to_soa(int N, long ld_n, const double* __restrict__ src, double* __restrict__ dst,
                                  float4* __restrict__ dstf)
{
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= 3L * N) return;
  const double x = src[i];
  dst[(i % 3) * ld_n + i / 3] = x;
  if (dstf) reinterpret_cast<float*>(dstf + i / 3)[i % 3] = (float)x;
}

cudaError_t launch_node_soa_to_aos(int N, long ld_n, const double* src, double* dst, cudaStream_t stream)
{
  if (N == 0) return cudaSuccess;
  k_node_soa_to_aos<<<grid_for(3L * N, 256), 256, 0, stream>>>(N, ld_n, src, dst);
  return cudaGetLastError();
}

cudaError_t launch_node_aos_to_soa(int N, long ld_n, const double* src, double* dst, float4* dstf,
                                   cudaStream_t stream)
{
  if (N == 0) return cudaSuccess;
  k_node_aos_to_soa<<<grid_for(3L * N, 256), 256, 0, stream>>>(N, ld_n, src, dst, dstf);
  return cudaGetLastError();
}

}  // namespace nsm
