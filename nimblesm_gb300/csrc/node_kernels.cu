// Node kernels: assembly of the element forces and the central-difference
// update.
//
// FP64 form: a node's first eight element forces are one sum in fixed point
// (fixed_sum.cuh), and every product and sum after that an explicit
// round-to-nearest intrinsic (__dmul_rn / __dadd_rn are never fused), so given
// the same assembled force the nodal state equals the reference's bit for bit.
// FP32-mixed form: the FP32 element forces are assembled in FP32 and the FP64
// update uses fused multiply-adds -- on this chip FP64 operations, not bytes,
// bound a node update, and the exact rounding of the reference buys nothing when
// the forces themselves are FP32.
#include "fixed_sum.cuh"
#include "nsm_kernels.cuh"

namespace nsm {

// Value of expression program `prog` at node n and time t: the postfix
// program on an operand stack, one double-precision operation at a time (no
// contraction across operations).  The host refuses programs deeper than the
// stack; a malformed one gives NaN rather than an access outside it.
__device__ __noinline__ double eval_bc_expression(const BcExprTable& ex, int prog, int n, double t)
{
  const double x = ex.X[n], y = ex.X[ex.ld_n + n], z = ex.X[2 * ex.ld_n + n];
  double       st[kExprStack];
  int          sp = 0;
  for (int i = ex.start[prog]; i < ex.start[prog + 1]; i++) {
    const ExprOp o = ex.code[i];
    if (o.code <= kExT) {
      if (sp >= kExprStack) return NAN;
      st[sp++] = o.code == kExConst ? o.c : (o.code == kExX ? x : (o.code == kExY ? y : (o.code == kExZ ? z : t)));
      continue;
    }
    if (o.code == kExSelect) {
      if (sp < 3) return NAN;
      sp -= 2;
      st[sp - 1] = st[sp - 1] != 0.0 ? st[sp] : st[sp + 1];
      continue;
    }
    if (expr_is_unary(o.code)) {
      if (sp < 1) return NAN;
      const double a = st[sp - 1];
      double       r;
      switch (o.code) {
        case kExNeg: r = -a; break;
        case kExSin: r = sin(a); break;
        case kExCos: r = cos(a); break;
        case kExTan: r = tan(a); break;
        case kExErf: r = erf(a); break;
        case kExExp: r = exp(a); break;
        case kExLog: r = log(a); break;
        case kExAbs: r = fabs(a); break;
        case kExAsin: r = asin(a); break;
        case kExAcos: r = acos(a); break;
        case kExAtan: r = atan(a); break;
        case kExSqrt: r = sqrt(a); break;
        case kExCbrt: r = cbrt(a); break;
        case kExErfc: r = erfc(a); break;
        case kExCeil: r = ceil(a); break;
        case kExRound: r = round(a); break;
        case kExFloor: r = floor(a); break;
        case kExLog10: r = log10(a); break;
        default: r = a != 0.0 ? 0.0 : 1.0; break;  // kExNot
      }
      st[sp - 1] = r;
      continue;
    }
    if (sp < 2) return NAN;
    const double a = st[sp - 2], b = st[sp - 1];
    double       r;
    switch (o.code) {
      case kExAdd: r = __dadd_rn(a, b); break;
      case kExSub: r = __dsub_rn(a, b); break;
      case kExMul: r = __dmul_rn(a, b); break;
      case kExDiv: r = __ddiv_rn(a, b); break;
      case kExMod: r = fmod(a, b); break;
      case kExPow: r = pow(a, b); break;
      case kExGt: r = a > b ? 1.0 : 0.0; break;
      case kExGe: r = a >= b ? 1.0 : 0.0; break;
      case kExLt: r = a < b ? 1.0 : 0.0; break;
      case kExLe: r = a <= b ? 1.0 : 0.0; break;
      case kExEq: r = a == b ? 1.0 : 0.0; break;
      case kExAnd: r = (a != 0.0 && b != 0.0) ? 1.0 : 0.0; break;
      case kExOr: r = (a != 0.0 || b != 0.0) ? 1.0 : 0.0; break;
      case kExXor: r = ((a != 0.0) != (b != 0.0)) ? 1.0 : 0.0; break;
      default: return NAN;
    }
    st[--sp - 1] = r;
  }
  return sp == 1 ? st[0] : NAN;
}

// ApplyKinematicBC for the explicit scheme
// (src/nimble_boundary_condition_manager.h:136-217): prescribed velocity sets
// v; prescribed displacement sets v = (d - u) / delta when delta > 0.  The
// magnitude is the line's constant or its expression's value at the node's
// reference coordinates and time_current (`ev`, evaluated beforehand).
// Components c0 .. c0 + kComps - 1.
template <int kComps>
__device__ __forceinline__ void apply_bc(const NodeBC& bc, double delta, const double* ev, int c0, const double u[kComps],
                                         double v[kComps])
{
#pragma unroll
  for (int i = 0; i < kComps; i++) {
    const int k = c0 + i;
    if (bc.kind[k] == 0 || (bc.kind[k] == 2 && !(delta > 0.0))) continue;
    const double value = bc.expr[k] < 0 ? bc.value[k] : ev[k];
    if (bc.kind[k] == 1) {
      v[i] = value;
    } else {
      v[i] = __ddiv_rn(__dadd_rn(value, -u[i]), delta);
    }
  }
}

// f + 0.0, the zero external force added as the reference adds it, without
// the FP64 pipe: the sum is f itself except for -0.0, which becomes +0.0.
__device__ __forceinline__ double plus_zero(double f)
{
  return __double_as_longlong(f) == (long long)0x8000000000000000ULL ? 0.0 : f;
}

// y + s*x, rounded as the reference's two operations or fused.
template <bool kExact>
__device__ __forceinline__ double axpy(double s, double x, double y)
{
  return kExact ? __dadd_rn(y, __dmul_rn(s, x)) : fma(s, x, y);
}

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// The first incidences of node n (all of them at a hex mesh's interior node),
// -1 past its last, and whether it has more: 8 e + corner from the slot-major
// copy, or (kRecords) the place of the force record.
constexpr int kFirst = 8;
template <bool kRecords>
__device__ __forceinline__ bool load_incidences(const NodeArgs& a, int n, int at[kFirst])
{
  if constexpr (kRecords) {
    const int count = __ldg(&a.node_ptr[n + 1]) - __ldg(&a.node_ptr[n]);
#pragma unroll
    for (int j = 0; j < kFirst; j++) at[j] = j < count ? j * (int)a.ld_n + n : -1;
    return count > kFirst;
  } else {
#pragma unroll
    for (int j = 0; j < kFirst; j++) at[j] = __ldg(&a.node_slots[(long)j * a.ld_n + n]);
    return (__ldg(&a.node_more[n >> 5]) >> (n & 31)) & 1u;
  }
}

// Components c0 ... of force record `at`.
template <int kComps>
__device__ __forceinline__ void load_record(const NodeArgs& a, int at, int c0, float x[kComps])
{
  const float4* row = reinterpret_cast<const float4*>(a.fe) + at;
  if constexpr (kComps == 1) {
    x[0] = reinterpret_cast<const float*>(row)[c0];
  } else {
    const float4 v = *row;
    x[0] = v.x, x[1] = v.y, x[2] = v.z;
  }
}

// The assembled element force of node n, components c0 ...: in the FP64 form the
// first eight contributions as one sum in fixed point, which has no order (sum8;
// on the FP64 pipe their additions were half of the launch's: 128^3 elements
// 183 -> 130 us, 15,625 nodes of 11 samples 24.5 -> 22), then, and in the FP32
// form from the first, additions in increasing element order.
template <typename TF, bool kExact, int kComps, bool kRecords>
__device__ __forceinline__ void gather_force(const NodeArgs& a, int n, const int ec[kFirst], bool more, int c0,
                                             double f[kComps])
{
  const TF* fe = reinterpret_cast<const TF*>(a.fe) + c0 * a.ld_e;  // planes
  TF        fs[kComps];
  // every load issued before the first sum
  TF x[kFirst][kComps];
#pragma unroll
  for (int j = 0; j < kFirst; j++)
    if constexpr (kRecords) {
      if (ec[j] >= 0) load_record<kComps>(a, ec[j], c0, x[j]);
    } else {
#pragma unroll
      for (int i = 0; i < kComps; i++)
        x[j][i] = ec[j] >= 0 ? fe[((ec[j] & 7) * 3 + i) * a.ld_e + (ec[j] >> 3)] : TF(0);
    }
  if constexpr (kExact) {
#pragma unroll
    for (int i = 0; i < kComps; i++) {
      double y[kFirst];
#pragma unroll
      for (int j = 0; j < kFirst; j++) y[j] = x[j][i];
      fs[i] = fx::sum8(y);
    }
  } else {
#pragma unroll
    for (int i = 0; i < kComps; i++) fs[i] = TF(0);
#pragma unroll
    for (int j = 0; j < kFirst; j++)
      if (ec[j] >= 0) {
#pragma unroll
        for (int i = 0; i < kComps; i++) fs[i] += x[j][i];
      }
  }
  const int k1 = more ? __ldg(&a.node_ptr[n + 1]) : 0;
  for (int k = more ? __ldg(&a.node_ptr[n]) + kFirst : 0; k < k1; k++) {
    const int  ec = __ldg(&a.node_inc[k]);
    const long e  = ec >> 3;
    const int  c  = ec & 7;
    TF         xk[kComps];
    if constexpr (kRecords) load_record<kComps>(a, __ldg(&a.fe_slot[c * a.ld_e + e]), c0, xk);
#pragma unroll
    for (int i = 0; i < kComps; i++) {
      const TF xi = kRecords ? xk[i] : fe[(c * 3 + i) * a.ld_e + e];
      fs[i]       = kExact ? TF(__dadd_rn(double(fs[i]), double(xi))) : fs[i] + xi;
    }
  }
#pragma unroll
  for (int i = 0; i < kComps; i++) f[i] = double(fs[i]);
}

// UqModel::ApplyClosure (src/uq/nimble_uq.cc:327-345) for a node of an
// approximate sample: f = f_0 c_0, then f += f_k c_k over the exact samples,
// force(k) being sample k's at the same local node.
template <bool kExact, typename Force>
__device__ __forceinline__ double close_force(const NodeArgs& a, int group, Force force)
{
  const double* c  = a.closure + (long)(group - a.closure_first) * (a.num_exact + 1);
  double        fk = force(0);
  double        f  = kExact ? __dmul_rn(fk, c[0]) : fk * c[0];
  for (int k = 1; k <= a.num_exact; k++) {
    fk = force(k);
    f  = kExact ? __dadd_rn(f, __dmul_rn(fk, c[k])) : fma(fk, c[k], f);
  }
  return f;
}

// What a node's update reads besides its force, components c0 ....
template <int kComps>
struct NodeState {
  double    u[kComps], v[kComps];
  double    im = 0.0;
  StepSched post, pre;

  __device__ __forceinline__ void load(const NodeArgs& a, int n, int c0, int group)
  {
    if (a.k_post >= 0) {
      post = a.sched[(long)(*a.step_base + a.k_post) * a.num_groups + group];
      im   = a.inv_mass[n];
    }
#pragma unroll
    for (int i = 0; i < kComps; i++) {
      v[i] = a.v[(c0 + i) * a.ld_n + n];
      u[i] = a.u[(c0 + i) * a.ld_n + n];
    }
  }
  __device__ __forceinline__ void load_pre(const NodeArgs& a, int group)
  {
    if (a.k_pre >= 0) pre = a.sched[(long)(*a.step_base + a.k_pre) * a.num_groups + group];
  }
};

// The end of the step finished, from its assembled forces.
template <bool kExact, int kComps>
__device__ __forceinline__ void end_step(const NodeArgs& a, int n, int c0, int slot, const NodeBC& bc,
                                         const double f[kComps], NodeState<kComps>& s, double acc[kComps])
{
#pragma unroll
  for (int i = 0; i < kComps; i++) {
    // a = (1/m) (f_int + f_ext), f_ext = 0 (src/integrators/explicit_time_integrator.cc:250-257)
    acc[i] = kExact ? __dmul_rn(s.im, plus_zero(f[i])) : s.im * f[i];
    s.v[i] = axpy<kExact>(s.post.half, acc[i], s.v[i]);
  }
  if (s.post.is_output && slot >= 0)
    apply_bc<kComps>(bc, s.post.delta, a.bc_expr_post ? a.bc_expr_post + (long)slot * 3 : nullptr, c0, s.u, s.v);
}

// The beginning of the step started, and the stores of the state.
template <typename TF, bool kExact, int kComps>
__device__ __forceinline__ void begin_step(const NodeArgs& a, int n, int c0, int slot, const NodeBC& bc,
                                           NodeState<kComps>& s, const double acc[kComps])
{
  const long ld = a.ld_n;
  if (a.k_pre >= 0) {
    // v^{n+1/2} = v^n + dt/2 a^n; BCs; u^{n+1} = u^n + dt v^{n+1/2}; BCs
    // (src/integrators/explicit_time_integrator.cc:200-223)
#pragma unroll
    for (int i = 0; i < kComps; i++) s.v[i] = axpy<kExact>(s.pre.half, acc[i], s.v[i]);
    const double* ev = a.bc_expr_pre ? a.bc_expr_pre + (long)slot * 3 : nullptr;
    if (slot >= 0) apply_bc<kComps>(bc, s.pre.delta, ev, c0, s.u, s.v);
#pragma unroll
    for (int i = 0; i < kComps; i++) s.u[i] = axpy<kExact>(s.pre.delta, s.v[i], s.u[i]);
    if (slot >= 0) apply_bc<kComps>(bc, s.pre.delta, ev, c0, s.u, s.v);
  }
#pragma unroll
  for (int i = 0; i < kComps; i++) {
    a.u[(c0 + i) * ld + n] = s.u[i];
    a.v[(c0 + i) * ld + n] = s.v[i];
    if (a.k_post >= 0 && a.k_pre < 0) a.a[(c0 + i) * ld + n] = acc[i];
  }
  if (sizeof(TF) == 4 && a.uf != nullptr) {  // FP32 forms only
    if constexpr (kComps == 3) a.uf[n] = make_float4((float)s.u[0], (float)s.u[1], (float)s.u[2], 0.0f);
    else reinterpret_cast<float*>(a.uf + n)[c0] = (float)s.u[0];
  }
}

// kComps = 3: a thread per node.  kComps = 1: a thread per node and component
// (blockIdx.y), with everything that the element kernel does not write read
// ahead of the wait for it; for meshes that one wave of blocks covers, where a
// step waits for latency: a third of the serial FP64 operations (64 clocks
// each for a warp by itself), and the loads of state and schedule overlap the
// element kernel's end.  (Three components that far ahead would spill.)
// kBlocks per SM: FP32 meshes beyond L2 wait for memory, 128^3 96.3 us with 5
// (48 registers), 92.1 with 6 (40, 52 bytes spilled), 105 with 7 (32); within it
// the spills cost more, 64^3 37.6 us a step with 5, 38.2 with 6 (90^3 101.5 and
// 100).  FP64 122 us with 4, 133 with 5, 138 with 3; FP32 records 15.2 with 4,
// 16.3 with 5.
template <typename TF, bool kExact, int kComps, bool kRecords, int kBlocks>
__global__ void __launch_bounds__(256, kBlocks) k_node_update(NodeArgs a)
{
  constexpr bool kAhead = kComps == 1;
  const int      n      = a.n_begin + blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= a.N) return;
  const int  c0    = kComps == 1 ? blockIdx.y : 0;
  const long ld    = a.ld_n;
  const int  slot  = a.bc_slot[n];
  const int  group = a.node_group ? __ldg(&a.node_group[n]) : 0;
  NodeBC     bc;
  if (slot >= 0) bc = a.bcs[slot];
  int               ec[kFirst];
  bool              more = false;
  double            acc[kComps];
  NodeState<kComps> s;
  // under the UQ closure a thread of a small mesh assembles the forces that it
  // needs by itself
  const bool closes = kComps == 1 && a.closure && group >= a.closure_first;
  if ((a.k_post >= 0 || a.gather_only) && !closes) more = load_incidences<kRecords>(a, n, ec);
  // The state, read after the gather (registers), is on its way to L2 meanwhile,
  // asked for by one lane per 128 bytes: 128^3 elements, FP64, 130.6 -> 121.9 us
  // (by every lane 127.4), FP32 97.8 -> 96.9.
  if (kComps == 3 && !a.gather_only && (threadIdx.x & 15) == 0) {
#pragma unroll
    for (int i = 0; i < 3; i++) {
      prefetch_l2(a.u + i * ld + n);
      prefetch_l2(a.v + i * ld + n);
    }
    prefetch_l2(a.inv_mass + n);
  }
  // (u and v are the previous node launch's, which had ended when the element
  // kernel let this one start)
  if (kAhead && !a.gather_only) {
    s.load(a, n, c0, group);
    s.load_pre(a, group);
  }
  wait_prerequisites();
  launch_dependents();

  if (a.k_post >= 0 || a.gather_only) {
    // ModelData::ComputeInternalForce: the sum of the element contributions
    // (src/nimble_model_data.cc:620-667, src/nimble_block.cc:373-383), which the
    // reference adds in increasing element order, as the FP32 form does.
    double f[kComps];
    if (closes) {
      f[0] = close_force<kExact>(a, group, [&](int k) {
        const int exact = a.node_off[k] + n - a.node_off[group];
        double    fk[1];
        more = load_incidences<kRecords>(a, exact, ec);
        gather_force<TF, kExact, 1, kRecords>(a, exact, ec, more, c0, fk);
        return fk[0];
      });
    } else {
      gather_force<TF, kExact, kComps, kRecords>(a, n, ec, more, c0, f);
    }
    // f_int (and a, below) are read by nothing inside a launch sequence: the
    // sequence's last launch (k_pre < 0) leaves them for the host's queries
    if (a.gather_only || a.k_pre < 0) {
#pragma unroll
      for (int i = 0; i < kComps; i++) a.f_int[(c0 + i) * ld + n] = f[i];
    }
    if (a.gather_only) {
      if (a.f_rows) {
#pragma unroll
        for (int i = 0; i < kComps; i++) a.f_rows[3L * n + c0 + i] = f[i];
      }
      return;
    }
    if (!kAhead) s.load(a, n, c0, group);
    end_step<kExact, kComps>(a, n, c0, slot, bc, f, s, acc);
  } else {
    if (!kAhead) s.load(a, n, c0, group);
#pragma unroll
    for (int i = 0; i < kComps; i++) acc[i] = a.a[(c0 + i) * ld + n];
  }
  if (!kAhead) s.load_pre(a, group);
  begin_step<TF, kExact, kComps>(a, n, c0, slot, bc, s, acc);
}

// The samples of one mesh under the UQ closure, past small meshes: a block takes
// 32 local nodes of all samples, a warp one sample and component of them at a
// time.  First the nominal and exact samples' forces are assembled, into f_int
// (read back through L1), then every node is updated.  Bound by the FP64 pipe,
// 64 clocks per warp and instruction on a quarter of an SM; a thread per node
// with each approximate node assembling the full samples' forces again is
// three times as many of its instructions with two exact samples.  15,625
// nodes of 11 samples (8 approximate): 41 -> 25 us, 35,937 of 12: 96 -> 48;
// 15,625 of 5 (1 approximate): 24.5 -> 16.3 (with FP64 additions in the
// assembly; 22, 43 and 14.5 without).  At most 12 warps: 6 or 8 and 16 took 26
// and 49 to 54 us for the first two.  Small meshes wait for latency
// instead, and this order lengthens the chain of a step: 216 nodes of 8
// samples 12.8 us a step against 11.3, 4,913 of 10 21.6 against 19.3.
constexpr int kUqWarps = 12;
template <typename TF, bool kExact, bool kRecords>
__global__ void __launch_bounds__(32 * kUqWarps, 3) k_node_update_uq(NodeArgs a)
{
  const int  local = blockIdx.x * 32 + (threadIdx.x & 31);
  const int  warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const bool in = local < a.local_nodes;
  const long ld = a.ld_n;
  wait_prerequisites();
  launch_dependents();
  for (int t = warp; t < 3 * (a.num_exact + 1) && in; t += warps) {
    const int  n = __ldg(&a.node_off[t / 3]) + local;
    int        ec[kFirst];
    const bool more = load_incidences<kRecords>(a, n, ec);
    double     f[1];
    gather_force<TF, kExact, 1, kRecords>(a, n, ec, more, t % 3, f);
    a.f_int[(t % 3) * ld + n] = f[0];
  }
  __syncthreads();
  for (int t = warp; t < 3 * a.num_groups && in; t += warps) {
    const int    group = t / 3, c0 = t % 3;
    const int    n    = __ldg(&a.node_off[group]) + local;
    const int    slot = a.bc_slot[n];
    NodeBC       bc;
    NodeState<1> s;
    if (slot >= 0) bc = a.bcs[slot];
    if (!a.gather_only) {
      s.load(a, n, c0, group);
      s.load_pre(a, group);
    }
    double f[1], acc[1];
    if (group < a.closure_first) {
      f[0] = a.f_int[c0 * ld + n];
    } else {
      f[0] = close_force<kExact>(a, group, [&](int k) { return a.f_int[c0 * ld + __ldg(&a.node_off[k]) + local]; });
      if (a.gather_only || a.k_pre < 0) a.f_int[c0 * ld + n] = f[0];
    }
    if (a.gather_only) continue;
    end_step<kExact, 1>(a, n, c0, slot, bc, f, s, acc);
    begin_step<TF, kExact, 1>(a, n, c0, slot, bc, s, acc);
  }
}

template <typename TF, bool kExact, bool kRecords>
static cudaError_t launch_small(const NodeArgs& a, int count, cudaStream_t stream)
{
  // The element kernels take all of an SM's shared memory; with the same split
  // of L1 here, an SM need not drain to change it between the two (a 4,096
  // element step with overlapped launches: 16.5 us with differing splits).
  static std::atomic<unsigned long long> configured{0};
  cudaError_t err = once_per_device(configured, [] {
    return cudaFuncSetAttribute(k_node_update<TF, kExact, 1, kRecords, 4>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  });
  if (err != cudaSuccess) return err;
  const int block = count <= 64 * 152 ? 64 : 256;  // the smallest meshes over more SMs
  return launch_overlapped(k_node_update<TF, kExact, 1, kRecords, 4>, dim3(grid_for(count, block), 3), block, 0, stream, a.overlap != 0, a);
}

// Nodes whose step (250 bytes each in the FP32 form) does not stay in L2.
constexpr int kBeyondL2 = 500000;

template <typename TF, bool kExact, bool kRecords>
static cudaError_t launch_nodes(const NodeArgs& a, cudaStream_t stream)
{
  const int count = a.N - a.n_begin;
  if (count <= 0) return cudaSuccess;
  if (a.closure && count > kSmallNodes && (a.k_post >= 0 || a.gather_only)) {
    const int tasks = 3 * a.num_groups, rounds = (tasks + kUqWarps - 1) / kUqWarps;
    const int warps = (tasks + rounds - 1) / rounds;
    return launch_overlapped(k_node_update_uq<TF, kExact, kRecords>, dim3(grid_for(a.local_nodes, 32)), 32 * warps, 0, stream,
                             a.overlap != 0, a);
  }
  if (count <= kSmallNodes) return launch_small<TF, kExact, kRecords>(a, count, stream);
  constexpr int kFew = sizeof(TF) == 4 && !kRecords ? 5 : 4, kMore = sizeof(TF) == 4 && !kRecords ? 6 : 4;
  return launch_overlapped(count > kBeyondL2 ? k_node_update<TF, kExact, 3, kRecords, kMore>
                                             : k_node_update<TF, kExact, 3, kRecords, kFew>,
                           dim3(grid_for(count, 256)), 256, 0, stream, a.overlap != 0, a);
}

cudaError_t launch_node_update(const NodeArgs& a, cudaStream_t stream)
{
  if (a.fe_is_float)
    return a.fe_slot ? launch_nodes<float, false, true>(a, stream) : launch_nodes<float, false, false>(a, stream);
  return launch_nodes<double, true, false>(a, stream);
}

// The place of each element corner's force record: the node's j-th incidence at
// j ld_n + n, the ones past its eighth in any order after all of those.
__global__ void k_force_slots(int N, long ld_n, long ld_e, const int* __restrict__ node_ptr,
                              const int* __restrict__ node_inc, int* __restrict__ counter, int* __restrict__ fe_slot)
{
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  const int k0 = node_ptr[n], count = node_ptr[n + 1] - k0;
  int       past = count > kFirst ? 8 * (int)ld_n + atomicAdd(counter, count - kFirst) : 0;
  for (int j = 0; j < count; j++) {
    const int ec                         = node_inc[k0 + j];
    fe_slot[(ec & 7) * ld_e + (ec >> 3)] = j < kFirst ? j * (int)ld_n + n : past++;
  }
}

cudaError_t launch_force_slots(int N, long ld_n, long ld_e, const int* node_ptr, const int* node_inc, int* counter,
                               int* fe_slot, cudaStream_t stream)
{
  if (N == 0) return cudaSuccess;
  k_force_slots<<<grid_for(N, 256), 256, 0, stream>>>(N, ld_n, ld_e, node_ptr, node_inc, counter, fe_slot);
  const cudaError_t err = cudaGetLastError();
  return err != cudaSuccess ? err : cudaMemsetAsync(counter, 0, sizeof(int), stream);
}

// One thread per (slot, component) and step (grid row): a program's latency on
// the FP64 pipe (a sine takes about 15 us) is that of one evaluation however
// many steps are evaluated at once.
__global__ void k_bc_expr_values(BcExprSteps q, BcExprTable ex, double* __restrict__ out)
{
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 3 * q.num_slots) return;
  const int s = t / 3, c = t % 3, prog = q.bcs[s].expr[c];
  if (prog < 0) return;
  const int    n     = q.slot_node[s];
  const int    group = q.node_group ? q.node_group[n] : 0;
  const double time  = q.sched[(long)(*q.step_base + q.k + blockIdx.y) * q.num_groups + group].time;
  out[(long)blockIdx.y * 3 * q.num_slots + t] = eval_bc_expression(ex, prog, n, time);
}

cudaError_t launch_bc_expr_values(const BcExprSteps& q, int steps, const BcExprTable& ex, double* out, cudaStream_t stream)
{
  if (q.num_slots == 0 || steps == 0) return cudaSuccess;
  k_bc_expr_values<<<dim3(grid_for(3L * q.num_slots, 128), steps), 128, 0, stream>>>(q, ex, out);
  return cudaGetLastError();
}

__global__ void k_advance_base(int* base, int k) { *base += k; }

cudaError_t launch_advance_base(int* step_base, int k, cudaStream_t stream)
{
  k_advance_base<<<1, 1, 0, stream>>>(step_base, k);
  return cudaGetLastError();
}

__global__ void k_apply_bc(int N, long ld_n, const int* __restrict__ bc_slot, const NodeBC* __restrict__ bcs,
                           double delta, double time, BcExprTable ex, const double* __restrict__ u,
                           double* __restrict__ v)
{
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  const int slot = bc_slot[n];
  if (slot < 0) return;
  double uu[3], vv[3];
#pragma unroll
  for (int i = 0; i < 3; i++) {
    uu[i] = u[i * ld_n + n];
    vv[i] = v[i * ld_n + n];
  }
  const NodeBC& bc = bcs[slot];
  double        ev[3];
#pragma unroll
  for (int k = 0; k < 3; k++) ev[k] = bc.expr[k] >= 0 ? eval_bc_expression(ex, bc.expr[k], n, time) : 0.0;
  apply_bc<3>(bc, delta, ev, 0, uu, vv);
#pragma unroll
  for (int i = 0; i < 3; i++) v[i * ld_n + n] = vv[i];
}

cudaError_t launch_apply_bc(int N, long ld_n, const int* bc_slot, const NodeBC* bcs, double delta, double time,
                            const BcExprTable& ex, const double* u, double* v, cudaStream_t stream)
{
  if (N == 0) return cudaSuccess;
  k_apply_bc<<<grid_for(N, 256), 256, 0, stream>>>(N, ld_n, bc_slot, bcs, delta, time, ex, u, v);
  return cudaGetLastError();
}

}  // namespace nsm
