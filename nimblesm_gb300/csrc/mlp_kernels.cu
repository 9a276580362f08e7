// Kernels of the learned constitutive closure (network and layouts in
// mlp_common.cuh): training-set generation from the neo-Hookean material,
// the training step (forward + backward, all GEMMs on the 5th-generation
// tensor cores), a deterministic gradient reduction with Adam, the BF16
// operand images, and batched inference.
#include <cuda_runtime.h>

#include "hex_math.cuh"
#include "mlp_common.cuh"
#include "mlp_kernels.cuh"
#include "nsm_kernels.cuh"

namespace nsm {
namespace mlp {

using namespace tc;

// ---------------------------------------------------------------------------
// Training set: F = I + N(0, s^2) per entry, rejected while det F < min_det,
// sigma from the engine's FP64 neo-Hookean (the same function the FP64 element
// kernel uses, parity-checked against the reference); stored as H = F - I
// (row-major) and sigma / G (symmetric order), FP32.

__device__ __forceinline__ uint64_t splitmix64(uint64_t& s)
{
  uint64_t z = (s += 0x9E3779B97F4A7C15ull);
  z          = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z          = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__device__ __forceinline__ double uniform01(uint64_t& s) { return ((splitmix64(s) >> 11) + 0.5) * (1.0 / 9007199254740992.0); }

__global__ void k_generate(long n, unsigned long long seed, double sd, double min_det, double K, double G,
                           float* __restrict__ X, float* __restrict__ Y, int* __restrict__ status)
{
  long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint64_t s = seed ^ (0x632BE59BD9B4E019ull * (uint64_t)(i + 1));
  double   H[3][3];
  bool     ok = false;
  for (int attempt = 0; attempt < 64 && !ok; attempt++) {
    for (int q = 0; q < 9; q += 2) {  // Box-Muller pairs
      double u1 = uniform01(s), u2 = uniform01(s);
      double r = sqrt(-2.0 * log(u1)), t = 6.283185307179586 * u2;
      H[q / 3][q % 3] = sd * r * cos(t);
      if (q + 1 < 9) H[(q + 1) / 3][(q + 1) % 3] = sd * r * sin(t);
    }
    double F00 = 1 + H[0][0], F11 = 1 + H[1][1], F22 = 1 + H[2][2];
    double det = F00 * (F11 * F22 - H[1][2] * H[2][1]) - H[0][1] * (H[1][0] * F22 - H[1][2] * H[2][0]) +
                 H[0][2] * (H[1][0] * H[2][1] - F11 * H[2][0]);
    ok = det >= min_det;
  }
  if (!ok) atomicOr(status, NSM_STATUS_BAD_JACOBIAN);
  double sig[6], C[3][3], J;
  neohookean<double>(H, K, G, sig, C, J);
  for (int q = 0; q < 9; q++) X[9 * i + q] = (float)H[q / 3][q % 3];
  for (int q = 0; q < 6; q++) Y[6 * i + q] = (float)(sig[q] / G);
}

// Sum over the training set of |(sigma/G - B(H)) / |x|^3|^2 (per-block
// partials, summed in block order on the host): sets the residual scale.
__global__ void k_residual_moment(long n, const float* __restrict__ X, const float* __restrict__ Y, float k_over_g,
                                  float in_scale, double* __restrict__ partial)
{
  __shared__ double s[256];
  double            acc = 0.0;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    float x[9], xs[9], L[6];
    for (int q = 0; q < 9; q++) {
      x[q]  = X[9 * i + q];
      xs[q] = x[q] * in_scale;
    }
    base_part(x, k_over_g, L);
    const double g = gate(xs);
    for (int q = 0; q < 6; q++) {
      double r = ((double)Y[6 * i + q] - (double)L[q]) / g;
      acc += r * r;
    }
  }
  s[threadIdx.x] = acc;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = s[0];
}

// ---------------------------------------------------------------------------
// BF16 operand images from the FP32 master parameters.
__global__ void k_images(const float* __restrict__ P, uint8_t* __restrict__ img)
{
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  // W1x [64][32]
  if (t < kHid * kInX) {
    int   n = t / kInX, k = t % kInX;
    float w = 0.0f;
    if (k < 9) w = P[oW1 + n * 9 + k];
    else if (k == 9) w = P[ob1 + n];
    else if (k >= 16 && k < 25) w = P[oW1 + n * 9 + (k - 16)];
    store_bf16(img + kOffW1, n, k, kInX, w);
  }
  // W2 [64][64] and W2t [64][64]
  if (t < kHid * kHid) {
    int n = t / kHid, k = t % kHid;
    store_bf16(img + kOffW2, n, k, kHid, P[oW2 + n * kHid + k]);
    store_bf16(img + kOffW2t, n, k, kHid, P[oW2 + k * kHid + n]);
  }
  // W3x [16][64] and W3t [64][16]
  if (t < kOutX * kHid) {
    int n = t / kHid, k = t % kHid;
    store_bf16(img + kOffW3, n, k, kHid, n < kOut ? P[oW3 + n * kHid + k] : 0.0f);
    int n2 = t / kOutX, k2 = t % kOutX;
    store_bf16(img + kOffW3t, n2, k2, kOutX, k2 < kOut ? P[oW3 + k2 * kHid + n2] : 0.0f);
  }
}

// ---------------------------------------------------------------------------
// Training step: one tile of 128 points per CTA (thread r <-> point r, whose
// accumulator row is tensor-memory lane r).  Writes this CTA's gradient of
// the mean-squared residual loss and its loss sum.
//
// Bound: the serial chain of six dependent MMA rounds and the two launches of
// a step; the tensor pipe is busy a few percent of the time.  The rounds are
// therefore kept short:
//   * Every activation and gradient is written once, as rows [point][feature].
//     The forward and data-gradient products read the rows K-major (K =
//     features), the weight gradients read the same bytes MN-major (K =
//     points): an 8 x 8 core matrix of one layout is a core matrix of the
//     other.  (Separate transposed copies were 2-byte stores four lanes to a
//     bank, and a 130 KB region to clear first.)
//   * Weight gradients are formed transposed, D[input][neuron], so that the 32
//     lanes of a warp store 32 consecutive parameters.
//   * A weight gradient is issued behind the data gradient that the chain
//     waits for, and stored while a later round runs.
//   * The pairs are gathered before the wait for the previous step's Adam
//     launch (programmatic dependent launch).
namespace tr {
// rows [128][kF]: A1 at columns 0-63, the extended input X at 64-95, A2 at
// 96-159; and [128][kD]: dZ2 at 0-63, dZ1 at 64-127, dZ3 at 128-143
constexpr int kF = 160, cA1 = 0, cX = 64, cA2 = 96;
constexpr int kD = 144, cD2 = 0, cD1 = 64, cD3 = 128;
constexpr int F    = 0;
constexpr int D    = F + 128 * kF * 2;
constexpr int W    = D + 128 * kD * 2;         // operand images
constexpr int B    = W + kImgBytes;            // b2[64], b3[6]
constexpr int SMEM = B + 512;
// tensor-memory columns; the weight gradients take over columns whose values
// have been read (W2's those of Z2, W1's those of Z1, W3's those of Z3)
constexpr uint32_t cZ1 = 0, cZ2 = 64, cDA = 128, cZ3 = 192, kCols = 256;
constexpr uint32_t cGW1 = cZ1, cGW2 = cZ2, cGW3 = cZ3;
constexpr int      kOnes = cX + 9;             // column of F that is 1 (the bias column of X)
}  // namespace tr

struct Sync {
  uint64_t* mbar;
  uint32_t  phase;
  int*      err;
};

// Issue-side: make operand writes visible to the tensor core and order them
// before the MMAs thread 0 is about to issue.
__device__ __forceinline__ void publish_operands()
{
  fence_proxy_async();
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
}

// Wait for the last commit; false (and the CTA-wide error flag) on timeout.
__device__ __forceinline__ bool await_mma(Sync& s)
{
  const bool ok = mbar_wait(s.mbar, s.phase);
  s.phase ^= 1u;
  if (!ok) atomicOr(s.err, 1);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  return *s.err == 0;
}

__device__ __forceinline__ void ld_row(uint32_t tbase, uint32_t col, int n16, float* v)
{
  const uint32_t lane_base = (uint32_t)(((threadIdx.x >> 5) & 3) * 32) << 16;  // the warp's lane quarter
  for (int c = 0; c < n16; c++) tmem_ld16(tbase + lane_base + col + 16 * c, v + 16 * c);
  tmem_wait_ld();
}

__device__ __forceinline__ void gemm(uint32_t d, const uint8_t* a, int a_rows_k, const uint8_t* b, int b_rows_k,
                                     int N, int K, bool accumulate_first)
{
  // a, b: K-major tiles whose row pitch per 8-row group is 16*K bytes
  const uint32_t idesc = idesc_bf16_f32(128, N);
  for (int ks = 0; ks < K / 16; ks++) {
    uint64_t ad = smem_desc(smem_addr(a) + ks * 2 * kLBO, kLBO, 16 * a_rows_k);
    uint64_t bd = smem_desc(smem_addr(b) + ks * 2 * kLBO, kLBO, 16 * b_rows_k);
    mma_bf16(d, ad, bd, idesc, accumulate_first || ks > 0);
  }
}

// D[128][N] = A^T B over the 128 points of two row tiles [128][a_width],
// [128][b_width]: both operands MN-major, a and b at the first of their 128
// and N columns.  A's columns may run past its rows' end (into the next rows,
// or what follows the tile): they give rows of D that nobody reads.
__device__ __forceinline__ void gemm_points(uint32_t d, const uint8_t* a, int a_width, const uint8_t* b, int b_width, int N)
{
  const uint32_t idesc = idesc_bf16_f32(128, N) | kIdescMnMajor;
  for (int ks = 0; ks < 128 / 16; ks++)
    mma_bf16(d, smem_desc(smem_addr(a) + ks * 2 * 16 * a_width, 16 * a_width, 128),
             smem_desc(smem_addr(b) + ks * 2 * 16 * b_width, 16 * b_width, 128), idesc, ks > 0);
}

// Two warpgroups per tile: thread t owns row r = t % 128 (tensor-memory lane r)
// and, in the 64-column epilogues, the columns [32 h, 32 h + 32) of half
// h = t / 128, so each thread's share of the activation and gradient work is
// half a row and the tile's dependent MMA rounds wait on half as much
// epilogue each.
constexpr int kTrainThreads = 256;

__global__ void __launch_bounds__(kTrainThreads) k_train(const float* __restrict__ X, const float* __restrict__ Y,
                                                         long n, long first, long stride_a, long offset_b,
                                                         const uint8_t* img, const float* P,
                                                         Scales sc, float inv_batch, float* __restrict__ grad_partial,
                                                         float* __restrict__ loss_partial, int* __restrict__ status)
{
  extern __shared__ __align__(1024) uint8_t sm[];
  __shared__ uint64_t mbar, mbar_w3, mbar_w2;
  __shared__ uint32_t tslot;
  __shared__ int      err;
  __shared__ float    red[128];
  const int           tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = tid & 127, half = tid >> 7;
  const int           c0  = 32 * half;  // this thread's first column in the 64-column epilogues

  // The point's pair (half 0), from its row of the epoch's visiting order.
  const long j     = first + (long)blockIdx.x * 128 + r;
  const bool valid = j < n;
  float      x[9], y[6];
  if (half == 0) {
    const long idx = valid ? (long)((stride_a * j + offset_b) % n) : 0;
#pragma unroll
    for (int q = 0; q < 9; q++) x[q] = __ldg(&X[9 * idx + q]);
#pragma unroll
    for (int q = 0; q < 6; q++) y[q] = __ldg(&Y[6 * idx + q]);
  }
  if (warp == 0) {
    tmem_alloc(&tslot, tr::kCols);
    tmem_relinquish();
  }
  if (tid == 0) {
    mbar_init(&mbar, 1);
    mbar_init(&mbar_w3, 1);
    mbar_init(&mbar_w2, 1);
    err = 0;
  }
  // ---- the point (half 0: its input row and target) ----
  float t[6];
  if (half == 0) {
    float xs[9];
    for (int q = 0; q < 9; q++) xs[q] = x[q] * sc.in_scale;
    {
      float L[6];
      base_part(x, sc.k_over_g, L);
      const float g = gate(xs) * sc.res_scale;
      for (int q = 0; q < 6; q++) t[q] = (y[q] - L[q]) / g;
    }
    float row[kInX];
    input_row(xs, row);
    for (int k0 = 0; k0 < kInX; k0 += 8) store_chunk(sm + tr::F, r, tr::cX + k0, tr::kF, row + k0);
  }
  // ---- what the previous step's Adam launch wrote: weight images, biases ----
  wait_prerequisites();
  launch_dependents();  // (not before the wait: this step's Adam launch reads the state that the previous one wrote)
  {
    const uint4* src = reinterpret_cast<const uint4*>(img);
    for (int i = tid; i < kImgBytes / 16; i += kTrainThreads) reinterpret_cast<uint4*>(sm + tr::W)[i] = __ldcg(src + i);
    float* bias = reinterpret_cast<float*>(sm + tr::B);
    if (tid < kHid) bias[tid] = __ldcg(&P[ob2 + tid]);
    if (tid < kOut) bias[64 + tid] = __ldcg(&P[ob3 + tid]);
  }
  publish_operands();
  const float*   b2 = reinterpret_cast<const float*>(sm + tr::B);
  const float*   b3 = b2 + 64;
  const uint32_t tb = tslot;
  Sync           sy{&mbar, 0u, &err};
  float* const   G  = grad_partial + (long)blockIdx.x * kParams;
  const uint8_t* Xop = sm + tr::F + tr::cX * 16;  // column c of a row tile starts 16 c bytes in
  const uint8_t* A1op = sm + tr::F + tr::cA1 * 16;
  const uint8_t* A2op = sm + tr::F + tr::cA2 * 16;
  const uint8_t* D1op = sm + tr::D + tr::cD1 * 16;
  const uint8_t* D2op = sm + tr::D + tr::cD2 * 16;
  const uint8_t* D3op = sm + tr::D + tr::cD3 * 16;

  // ---- forward ----
  if (tid == 0) {
    gemm(tb + tr::cZ1, Xop, tr::kF, sm + tr::W + kOffW1, kInX, kHid, kInX, false);
    mma_commit(&mbar);
  }
  if (!await_mma(sy)) goto cleanup;
  {
    float z[32];
    ld_row(tb, tr::cZ1 + c0, 2, z);
    for (int q = 0; q < 32; q++) z[q] = act(z[q]);
    for (int k0 = 0; k0 < 32; k0 += 8) store_chunk(sm + tr::F, r, tr::cA1 + c0 + k0, tr::kF, z + k0);
  }
  publish_operands();
  if (tid == 0) {
    gemm(tb + tr::cZ2, A1op, tr::kF, sm + tr::W + kOffW2, kHid, kHid, kHid, false);
    mma_commit(&mbar);
  }
  if (!await_mma(sy)) goto cleanup;
  {
    float z[32];
    ld_row(tb, tr::cZ2 + c0, 2, z);
    for (int q = 0; q < 32; q++) z[q] = act(z[q] + b2[c0 + q]);
    for (int k0 = 0; k0 < 32; k0 += 8) store_chunk(sm + tr::F, r, tr::cA2 + c0 + k0, tr::kF, z + k0);
  }
  publish_operands();
  if (tid == 0) {
    gemm(tb + tr::cZ3, A2op, tr::kF, sm + tr::W + kOffW3, kHid, kOutX, kHid, false);
    mma_commit(&mbar);
  }
  if (!await_mma(sy)) goto cleanup;
  if (half == 0) {
    float z[16], g[16];
    ld_row(tb, tr::cZ3, 1, z);
    float lsum = 0.0f;
    for (int q = 0; q < 16; q++) g[q] = 0.0f;
    for (int q = 0; q < kOut; q++) {
      float d = valid ? (z[q] + b3[q] - t[q]) : 0.0f;
      lsum += d * d;
      g[q] = 2.0f * d * inv_batch;
    }
    red[r] = lsum;
    for (int k0 = 0; k0 < 16; k0 += 8) store_chunk(sm + tr::D, r, tr::cD3 + k0, tr::kD, g + k0);
  }
  publish_operands();
  // ---- backward ----
  if (tid == 0) {
    gemm(tb + tr::cDA, D3op, tr::kD, sm + tr::W + kOffW3t, kOutX, kHid, kOutX, false);
    mma_commit(&mbar);
    gemm_points(tb + tr::cGW3, Xop, tr::kF, D3op, tr::kD, kOutX);  // rows 0-31 X (its ones: b3), 32-95 A2
    mma_commit(&mbar_w3);
  }
  if (!await_mma(sy)) goto cleanup;
  {
    float da[32], z[32];
    ld_row(tb, tr::cDA + c0, 2, da);
    ld_row(tb, tr::cZ2 + c0, 2, z);
    for (int q = 0; q < 32; q++) da[q] *= act_grad(z[q] + b2[c0 + q]);
    for (int k0 = 0; k0 < 32; k0 += 8) store_chunk(sm + tr::D, r, tr::cD2 + c0 + k0, tr::kD, da + k0);
  }
  publish_operands();
  if (tid == 0) {
    gemm(tb + tr::cDA, D2op, tr::kD, sm + tr::W + kOffW2t, kHid, kHid, kHid, false);
    mma_commit(&mbar);
    gemm_points(tb + tr::cGW2, A1op, tr::kF, D2op, tr::kD, kHid);  // rows 0-63 A1, 64-95 X (its ones: b2)
    mma_commit(&mbar_w2);
  }
  // W3's gradient, while the data gradient is formed
  if (!mbar_wait(&mbar_w3, 0u)) atomicOr(&err, 1);
  fence_after_sync();
  if (half == 1 && warp < 7) {
    float w[16];
    ld_row(tb, tr::cGW3, 1, w);
    if (warp == 4) {
      if (lane == tr::kOnes - tr::cX)
        for (int o = 0; o < kOut; o++) G[ob3 + o] = w[o];
    } else {
      for (int o = 0; o < kOut; o++) G[oW3 + o * kHid + (r - 32)] = w[o];
    }
  }
  if (!await_mma(sy)) goto cleanup;
  {
    float da[32], z[32];
    ld_row(tb, tr::cDA + c0, 2, da);
    ld_row(tb, tr::cZ1 + c0, 2, z);
    for (int q = 0; q < 32; q++) da[q] *= act_grad(z[q]);
    for (int k0 = 0; k0 < 32; k0 += 8) store_chunk(sm + tr::D, r, tr::cD1 + c0 + k0, tr::kD, da + k0);
  }
  publish_operands();
  if (tid == 0) {
    gemm_points(tb + tr::cGW1, A1op, tr::kF, D1op, tr::kD, kHid);  // rows 64-95 X
    mma_commit(&mbar);
  }
  // W2's gradient, while W1's is formed: this half's 32 neurons
  if (!mbar_wait(&mbar_w2, 0u)) atomicOr(&err, 1);
  fence_after_sync();
  if ((warp & 3) < 3) {
    float w[32];
    ld_row(tb, tr::cGW2 + c0, 2, w);
    if (r < 64) {
      for (int q = 0; q < 32; q++) G[oW2 + (c0 + q) * kHid + r] = w[q];
    } else if (r == tr::kOnes) {
      for (int q = 0; q < 32; q++) G[ob2 + c0 + q] = w[q];
    }
  }
  if (half == 1 && tid < 192) {  // the tile's loss, summed in a fixed order by two warps
    float l = red[tid - 128] + red[tid - 64];
    red[tid - 128] = l;
  }
  if (!await_mma(sy)) goto cleanup;
  if ((warp & 3) == 2) {  // rows 64-95: inputs X; the input's two terms are lanes q and 16 + q
    float w[32];
    ld_row(tb, tr::cGW1 + c0, 2, w);
    for (int q = 0; q < 32; q++) {
      const float lo = __shfl_down_sync(0xffffffffu, w[q], 16);
      if (lane < kIn) G[oW1 + (c0 + q) * kIn + lane] = w[q] + lo;
      else if (lane == 9) G[ob1 + c0 + q] = w[q];
    }
  } else if (warp == 0) {
    float l = red[lane] + red[lane + 32];
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) l += __shfl_down_sync(0xffffffffu, l, w);
    if (lane == 0) loss_partial[blockIdx.x] = l;
  }

cleanup:
  if (tid == 0 && err) {
    mbar_wait(sy.mbar, sy.phase ^ 1u);  // bounded: let a timed-out MMA drain before the columns are freed
    atomicOr(status, NSM_STATUS_TIMEOUT);
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tb, tr::kCols);
}

// The operand-image entries of parameter i (the layout k_images writes), from
// its value w.  The biases b2 and b3 have none (the kernels read them in
// FP32), nor do the images' zero padding entries, which k_images wrote.
__device__ __forceinline__ void store_images(int i, float w, uint8_t* __restrict__ img)
{
  if (i < ob1) {
    const int n = (i - oW1) / kIn, k = (i - oW1) % kIn;
    store_bf16(img + kOffW1, n, k, kInX, w);
    store_bf16(img + kOffW1, n, k + 16, kInX, w);
  } else if (i < oW2) {
    store_bf16(img + kOffW1, i - ob1, 9, kInX, w);
  } else if (i < ob2) {
    const int n = (i - oW2) / kHid, k = (i - oW2) % kHid;
    store_bf16(img + kOffW2, n, k, kHid, w);
    store_bf16(img + kOffW2t, k, n, kHid, w);
  } else if (i >= oW3 && i < ob3) {
    const int n = (i - oW3) / kHid, k = (i - oW3) % kHid;
    store_bf16(img + kOffW3, n, k, kHid, w);
    store_bf16(img + kOffW3t, k, n, kOutX, w);
  }
}

// Deterministic reduction of the per-CTA gradients, an Adam step on the FP32
// master parameters, and the new parameters' BF16 operand-image entries.
// Bound: the latency of the partials' loads.  Eight warps share 32 parameters:
// warp j sums the partials of CTAs j, j + 8, ... in order (a 128-byte row per
// load, up to 20 in flight ahead of the in-order sum), and the eight sums are
// combined in a fixed order, so every run gives the same bits.
constexpr int kAdamWarps = 8, kAdamAhead = 20;
__global__ void __launch_bounds__(32 * kAdamWarps) k_adam(int ncta, const float* grad_partial, float* __restrict__ P,
                                                          float* __restrict__ m1, float* __restrict__ m2, float lr,
                                                          float beta1, float beta2, float eps, float bc1, float bc2,
                                                          uint8_t* __restrict__ img)
{
  __shared__ float sums[kAdamWarps][32];
  const int        lane = threadIdx.x & 31, sub = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
  const bool       own = i < kParams;
  launch_dependents();
  // (the state is the previous Adam launch's, which had ended when this step's training launch let this one start)
  float a0 = 0.0f, b0 = 0.0f, p0 = 0.0f;
  if (sub == 0 && own) a0 = m1[i], b0 = m2[i], p0 = P[i];
  wait_prerequisites();
  float g = 0.0f;
  if (own) {
    const float* gp = grad_partial + i;
    for (int c = sub; c < ncta; c += kAdamAhead * kAdamWarps) {
      float v[kAdamAhead];
#pragma unroll
      for (int k = 0; k < kAdamAhead; k++)
        if (c + k * kAdamWarps < ncta) v[k] = __ldcg(&gp[(long)(c + k * kAdamWarps) * kParams]);
#pragma unroll
      for (int k = 0; k < kAdamAhead; k++)
        if (c + k * kAdamWarps < ncta) g += v[k];
    }
  }
  sums[sub][lane] = g;
  __syncthreads();
  if (sub != 0 || !own) return;
  float s[kAdamWarps];
#pragma unroll
  for (int k = 0; k < kAdamWarps; k++) s[k] = sums[k][lane];
  g = ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
  const float a = fmaf(1.0f - beta1, g, beta1 * a0);
  const float b = fmaf((1.0f - beta2) * g, g, beta2 * b0);
  m1[i]         = a;
  m2[i]         = b;
  const float w = p0 - lr * (a / bc1) / (sqrtf(b / bc2) + eps);
  P[i]          = w;
  store_images(i, w, img);
}

__global__ void k_sum_gradient(int ncta, const float* __restrict__ grad_partial, float* __restrict__ g)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kParams) return;
  float s = 0.0f;
  for (int c = 0; c < ncta; c++) s += grad_partial[(long)c * kParams + i];
  g[i] = s;
}

// ---------------------------------------------------------------------------
// Inference on a batch of points: H (row-major, FP32) -> sigma / G.  Points
// outside the training envelope take the plain neo-Hookean stress and are
// counted.
namespace inf {
constexpr int X    = 0;                     // [128][32]
constexpr int A1   = X + 128 * kInX * 2;    // [128][64]
constexpr int A2   = A1 + 128 * kHid * 2;   // [128][64]
constexpr int W    = A2 + 128 * kHid * 2;   // W1x, W2, W3x images
constexpr int B    = W + kOffW2t;           // b2[64], b3[6]
constexpr int END  = B + 512;
constexpr int SMEM = END + 16384;
constexpr uint32_t cZ1 = 0, cZ2 = 64, cZ3 = 128, kCols = 256;
}  // namespace inf

__global__ void __launch_bounds__(128) k_predict(long n, const float* __restrict__ H, const uint8_t* __restrict__ img,
                                                 const float* __restrict__ P, Scales sc, double K, double G,
                                                 double* __restrict__ sigma, int* __restrict__ fallback,
                                                 int* __restrict__ status)
{
  extern __shared__ __align__(1024) uint8_t sm[];
  __shared__ uint64_t mbar;
  __shared__ uint32_t tslot;
  __shared__ int      err;
  const int           r = threadIdx.x, warp = r >> 5;
  if (warp == 0) {
    tmem_alloc(&tslot, inf::kCols);
    tmem_relinquish();
  }
  if (r == 0) {
    mbar_init(&mbar, 1);
    err = 0;
  }
  {
    const uint4* src = reinterpret_cast<const uint4*>(img);
    for (int i = r; i < kOffW2t / 16; i += 128) reinterpret_cast<uint4*>(sm + inf::W)[i] = src[i];
    float* bias = reinterpret_cast<float*>(sm + inf::B);
    if (r < kHid) bias[r] = P[ob2 + r];
    if (r < kOut) bias[64 + r] = P[ob3 + r];
  }
  const float* b2 = reinterpret_cast<const float*>(sm + inf::B);
  const float* b3 = b2 + 64;
  const long   i  = (long)blockIdx.x * 128 + r;
  const bool   valid = i < n;
  float        h[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  if (valid)
    for (int q = 0; q < 9; q++) h[q] = H[9 * i + q];
  float xs[9], row[kInX];
  for (int q = 0; q < 9; q++) xs[q] = h[q] * sc.in_scale;
  input_row(xs, row);
  for (int k0 = 0; k0 < kInX; k0 += 8) store_chunk(sm + inf::X, r, k0, kInX, row + k0);
  publish_operands();
  Sync           sy{&mbar, 0u, &err};
  const uint32_t tb = tslot;
  if (r == 0) {
    gemm(tb + inf::cZ1, sm + inf::X, kInX, sm + inf::W + kOffW1, kInX, kHid, kInX, false);
    mma_commit(&mbar);
  }
  if (!await_mma(sy)) goto cleanup;
  {
    float z[64];
    ld_row(tb, inf::cZ1, 4, z);
    for (int q = 0; q < 64; q++) z[q] = act(z[q]);
    for (int k0 = 0; k0 < 64; k0 += 8) store_chunk(sm + inf::A1, r, k0, kHid, z + k0);
  }
  publish_operands();
  if (r == 0) {
    gemm(tb + inf::cZ2, sm + inf::A1, kHid, sm + inf::W + kOffW2, kHid, kHid, kHid, false);
    mma_commit(&mbar);
  }
  if (!await_mma(sy)) goto cleanup;
  {
    float z[64];
    ld_row(tb, inf::cZ2, 4, z);
    for (int q = 0; q < 64; q++) z[q] = act(z[q] + b2[q]);
    for (int k0 = 0; k0 < 64; k0 += 8) store_chunk(sm + inf::A2, r, k0, kHid, z + k0);
  }
  publish_operands();
  if (r == 0) {
    gemm(tb + inf::cZ3, sm + inf::A2, kHid, sm + inf::W + kOffW3, kHid, kOutX, kHid, false);
    mma_commit(&mbar);
  }
  if (!await_mma(sy)) goto cleanup;
  {
    float z[16];
    ld_row(tb, inf::cZ3, 1, z);
    if (valid) {
      if (in_envelope(h, sc)) {
        float L[6];
        base_part(h, sc.k_over_g, L);
        const float g = gate(xs) * sc.res_scale;
        for (int q = 0; q < kOut; q++) sigma[6 * i + q] = G * (double)(L[q] + g * (z[q] + b3[q]));
      } else {
        double Hd[3][3], s6[6], C[3][3], J;
        for (int q = 0; q < 9; q++) Hd[q / 3][q % 3] = h[q];
        neohookean<double>(Hd, K, G, s6, C, J);
        for (int q = 0; q < kOut; q++) sigma[6 * i + q] = s6[q];
        atomicAdd(fallback, 1);
      }
    }
  }
cleanup:
  if (r == 0 && err) {
    mbar_wait(sy.mbar, sy.phase ^ 1u);  // bounded: let a timed-out MMA drain before the columns are freed
    atomicOr(status, NSM_STATUS_TIMEOUT);
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tslot, inf::kCols);
}

// ---------------------------------------------------------------------------
cudaError_t launch_generate(long n, unsigned long long seed, double sd, double min_det, double K, double G, float* X,
                            float* Y, int* status, cudaStream_t s)
{
  if (n <= 0) return cudaSuccess;
  k_generate<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, seed, sd, min_det, K, G, X, Y, status);
  return cudaGetLastError();
}

cudaError_t launch_residual_moment(long n, const float* X, const float* Y, float k_over_g, float in_scale,
                                   double* partial, int blocks, cudaStream_t s)
{
  k_residual_moment<<<blocks, 256, 0, s>>>(n, X, Y, k_over_g, in_scale, partial);
  return cudaGetLastError();
}

cudaError_t launch_images(const float* P, uint8_t* img, cudaStream_t s)
{
  k_images<<<(kHid * kHid + 127) / 128, 128, 0, s>>>(P, img);
  return cudaGetLastError();
}

cudaError_t setup_kernels()
{
  cudaError_t e = cudaFuncSetAttribute(k_train, cudaFuncAttributeMaxDynamicSharedMemorySize, tr::SMEM);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(k_predict, cudaFuncAttributeMaxDynamicSharedMemorySize, inf::SMEM);
}

cudaError_t launch_train(int tiles, const float* X, const float* Y, long n, long first, long stride_a, long offset_b,
                         const uint8_t* img, const float* P, const Scales& sc, float inv_batch, float* grad_partial,
                         float* loss_partial, int* status, bool after_adam, cudaStream_t s)
{
  return launch_overlapped(k_train, tiles, kTrainThreads, tr::SMEM, s, after_adam, X, Y, n, first, stride_a, offset_b, img, P,
                           sc, inv_batch, grad_partial, loss_partial, status);
}

cudaError_t launch_adam(int ncta, const float* grad_partial, float* P, float* m1, float* m2, float lr, float beta1,
                        float beta2, float eps, float bc1, float bc2, uint8_t* img, cudaStream_t s)
{
  return launch_overlapped(k_adam, (kParams + 31) / 32, 32 * kAdamWarps, 0, s, true, ncta, grad_partial, P, m1, m2, lr, beta1,
                           beta2, eps, bc1, bc2, img);
}

cudaError_t launch_sum_gradient(int ncta, const float* grad_partial, float* g, cudaStream_t s)
{
  k_sum_gradient<<<(kParams + 255) / 256, 256, 0, s>>>(ncta, grad_partial, g);
  return cudaGetLastError();
}

cudaError_t launch_predict(long n, const float* H, const uint8_t* img, const float* P, const Scales& sc, double K,
                           double G, double* sigma, int* fallback, int* status, cudaStream_t s)
{
  if (n <= 0) return cudaSuccess;
  k_predict<<<(unsigned)((n + 127) / 128), 128, inf::SMEM, s>>>(n, H, img, P, sc, K, G, sigma, fallback, status);
  return cudaGetLastError();
}

}  // namespace mlp
}  // namespace nsm
