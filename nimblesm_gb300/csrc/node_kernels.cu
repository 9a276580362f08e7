// Node kernels: assembly of the element forces and the central-difference
// update.
//
// FP64 form: every product and sum is an explicit round-to-nearest intrinsic
// (__dmul_rn / __dadd_rn are never fused), so given the same element forces
// the nodal state equals the reference's bit for bit.  FP32-mixed form: the
// FP32 element forces are assembled in FP32 and the FP64 update uses fused
// multiply-adds -- on this chip FP64 operations, not bytes, bound a node
// update, and the exact rounding of the reference buys nothing when the forces
// themselves are FP32.
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

// The assembled element force of node n, components c0 ...: element
// contributions in increasing element order.
template <typename TF, bool kExact, int kComps, bool kRecords>
__device__ __forceinline__ void gather_force(const NodeArgs& a, int n, const int ec[kFirst], bool more, int c0,
                                             double f[kComps])
{
  const TF* fe = reinterpret_cast<const TF*>(a.fe) + c0 * a.ld_e;  // planes
  TF        fs[kComps];
  // every load issued before the first sum, the sums in the same order as the
  // rest from the CSR below
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
#pragma unroll
  for (int i = 0; i < kComps; i++) fs[i] = TF(0);
  // the first sum is 0 + x: x itself but for -0.0 (+0.0), an integer select
  // rather than an FP64 add in the exact form
  if (ec[0] >= 0) {
#pragma unroll
    for (int i = 0; i < kComps; i++) fs[i] = kExact ? TF(plus_zero(double(x[0][i]))) : fs[i] + x[0][i];
  }
#pragma unroll
  for (int j = 1; j < kFirst; j++)
    if (ec[j] >= 0) {
#pragma unroll
      for (int i = 0; i < kComps; i++) fs[i] = kExact ? TF(__dadd_rn(double(fs[i]), double(x[j][i]))) : fs[i] + x[j][i];
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

// kComps = 3: a thread per node.  kComps = 1: a thread per node and component
// (blockIdx.y), with everything that the element kernel does not write read
// ahead of the wait for it; for meshes that one wave of blocks covers, where a
// step waits for latency: a third of the serial FP64 operations (64 clocks
// each for a warp by itself), and the loads of state and schedule overlap the
// element kernel's end.  (Three components that far ahead would spill.)
template <typename TF, bool kExact, int kComps, bool kRecords>
__global__ void __launch_bounds__(256, kComps == 3 && sizeof(TF) == 4 && !kRecords ? 5 : 4) k_node_update(NodeArgs a)
{
  constexpr bool kAhead = kComps == 1;
  const int      n      = a.n_begin + blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= a.N) return;
  const int  c0 = kComps == 1 ? blockIdx.y : 0;
  const long ld = a.ld_n;
  double     u[kComps], v[kComps], acc[kComps];
  const int  slot  = a.bc_slot[n];
  const int  group = a.node_group ? __ldg(&a.node_group[n]) : 0;
  NodeBC     bc;
  if (slot >= 0) bc = a.bcs[slot];
  const bool closes = a.closure && group >= a.closure_first;
  int        ec[kFirst];
  bool       more = false;
  StepSched  post, pre;
  double     im = 0.0;
  auto       load_state = [&] {
    if (a.k_post >= 0) {
      post = a.sched[(long)(*a.step_base + a.k_post) * a.num_groups + group];
      im   = a.inv_mass[n];
    }
#pragma unroll
    for (int i = 0; i < kComps; i++) {
      v[i] = a.v[(c0 + i) * ld + n];
      u[i] = a.u[(c0 + i) * ld + n];
    }
  };
  if ((a.k_post >= 0 || a.gather_only) && !closes) more = load_incidences<kRecords>(a, n, ec);
  // (u and v are the previous node launch's, which had ended when the element
  // kernel let this one start)
  if (kAhead && !a.gather_only) {
    load_state();
    if (a.k_pre >= 0) pre = a.sched[(long)(*a.step_base + a.k_pre) * a.num_groups + group];
  }
  wait_prerequisites();
  launch_dependents();

  if (a.k_post >= 0 || a.gather_only) {
    // ModelData::ComputeInternalForce: zero, then element contributions in
    // increasing element order (src/nimble_model_data.cc:620-667,
    // src/nimble_block.cc:373-383).
    double f[kComps];
    if (closes) {
      // UqModel::ApplyClosure (src/uq/nimble_uq.cc:327-345): f = f_0 c_0, then
      // f += f_k c_k over the exact samples, from the same assembled forces
      // the nominal and exact samples' own nodes compute
      const int     local = n - a.node_off[group];
      const double* c     = a.closure + (long)(group - a.closure_first) * (a.num_exact + 1);
      double        fk[kComps];
      more = load_incidences<kRecords>(a, a.node_off[0] + local, ec);
      gather_force<TF, kExact, kComps, kRecords>(a, a.node_off[0] + local, ec, more, c0, fk);
#pragma unroll
      for (int i = 0; i < kComps; i++) f[i] = kExact ? __dmul_rn(fk[i], c[0]) : fk[i] * c[0];
      for (int k = 1; k <= a.num_exact; k++) {
        more = load_incidences<kRecords>(a, a.node_off[k] + local, ec);
        gather_force<TF, kExact, kComps, kRecords>(a, a.node_off[k] + local, ec, more, c0, fk);
#pragma unroll
        for (int i = 0; i < kComps; i++)
          f[i] = kExact ? __dadd_rn(f[i], __dmul_rn(fk[i], c[k])) : fma(fk[i], c[k], f[i]);
      }
    } else {
      gather_force<TF, kExact, kComps, kRecords>(a, n, ec, more, c0, f);
    }
    // f_int (and a, below) are read by nothing inside a launch sequence: the
    // sequence's last launch (k_pre < 0) leaves them for the host's queries
    if (a.gather_only || a.k_pre < 0) {
#pragma unroll
      for (int i = 0; i < kComps; i++) a.f_int[(c0 + i) * ld + n] = f[i];
    }
    if (a.gather_only) return;
    if (!kAhead) load_state();
#pragma unroll
    for (int i = 0; i < kComps; i++) {
      // a = (1/m) (f_int + f_ext), f_ext = 0 (src/integrators/explicit_time_integrator.cc:250-257)
      acc[i] = kExact ? __dmul_rn(im, plus_zero(f[i])) : im * f[i];
      v[i]   = axpy<kExact>(post.half, acc[i], v[i]);
    }
    if (post.is_output && slot >= 0)
      apply_bc<kComps>(bc, post.delta, a.bc_expr_post ? a.bc_expr_post + (long)slot * 3 : nullptr, c0, u, v);
  } else {
    if (!kAhead) load_state();
#pragma unroll
    for (int i = 0; i < kComps; i++) acc[i] = a.a[(c0 + i) * ld + n];
  }
  if (a.k_pre >= 0) {
    // v^{n+1/2} = v^n + dt/2 a^n; BCs; u^{n+1} = u^n + dt v^{n+1/2}; BCs
    // (src/integrators/explicit_time_integrator.cc:200-223)
    if (!kAhead) pre = a.sched[(long)(*a.step_base + a.k_pre) * a.num_groups + group];
#pragma unroll
    for (int i = 0; i < kComps; i++) v[i] = axpy<kExact>(pre.half, acc[i], v[i]);
    const double* ev = a.bc_expr_pre ? a.bc_expr_pre + (long)slot * 3 : nullptr;
    if (slot >= 0) apply_bc<kComps>(bc, pre.delta, ev, c0, u, v);
#pragma unroll
    for (int i = 0; i < kComps; i++) u[i] = axpy<kExact>(pre.delta, v[i], u[i]);
    if (slot >= 0) apply_bc<kComps>(bc, pre.delta, ev, c0, u, v);
  }
#pragma unroll
  for (int i = 0; i < kComps; i++) {
    a.u[(c0 + i) * ld + n] = u[i];
    a.v[(c0 + i) * ld + n] = v[i];
    if (a.k_post >= 0 && a.k_pre < 0) a.a[(c0 + i) * ld + n] = acc[i];
  }
  if (sizeof(TF) == 4 && a.uf != nullptr) {  // FP32 forms only
    if constexpr (kComps == 3) a.uf[n] = make_float4((float)u[0], (float)u[1], (float)u[2], 0.0f);
    else reinterpret_cast<float*>(a.uf + n)[c0] = (float)u[0];
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
    return cudaFuncSetAttribute(k_node_update<TF, kExact, 1, kRecords>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  });
  if (err != cudaSuccess) return err;
  const int block = count <= 64 * 152 ? 64 : 256;  // the smallest meshes over more SMs
  return launch_overlapped(k_node_update<TF, kExact, 1, kRecords>, dim3(grid_for(count, block), 3), block, 0, stream, a.overlap != 0, a);
}

template <typename TF, bool kExact, bool kRecords>
static cudaError_t launch_nodes(const NodeArgs& a, cudaStream_t stream)
{
  const int count = a.N - a.n_begin;
  if (count <= 0) return cudaSuccess;
  if (count <= kSmallNodes) return launch_small<TF, kExact, kRecords>(a, count, stream);
  return launch_overlapped(k_node_update<TF, kExact, 3, kRecords>, dim3(grid_for(count, 256)), 256, 0, stream,
                           a.overlap != 0, a);
}

cudaError_t launch_node_update(const NodeArgs& a, cudaStream_t stream)
{
  if (a.fe_is_float)
    return a.fe_slot ? launch_nodes<float, false, true>(a, stream) : launch_nodes<float, false, false>(a, stream);
  return launch_nodes<double, true, false>(a, stream);
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
