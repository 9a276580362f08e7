// Host check of which elements the fixed-point arithmetic (hex_fixed.cuh) takes
// and how exact it is there: elements of several aspect ratios, moduli, strains
// and rotations, as the kernel's four lanes evaluate them, and the same in FP64
// by the FP64 code's own functions (hex_math.cuh), both against the formulas in
// extended precision.  Prints per kind: model, kind, elements outside, and the
// relative errors of forces and stresses of both (root of the mean square over
// the elements inside).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <random>
#include <vector>

// What hex_math.cuh takes from CUDA.
static int      __double2hiint(double d) { long long b; std::memcpy(&b, &d, 8); return (int)(b >> 32); }
static int      __double2loint(double d) { long long b; std::memcpy(&b, &d, 8); return (int)b; }
static double   __longlong_as_double(long long b) { double d; std::memcpy(&d, &b, 8); return d; }
static long long __double_as_longlong(double d) { long long b; std::memcpy(&b, &d, 8); return b; }
static double   __hiloint2double(int h, int l) { return __longlong_as_double((long long)((unsigned long long)(unsigned)h << 32 | (unsigned)l)); }
static unsigned __float_as_uint(float f) { unsigned u; std::memcpy(&u, &f, 4); return u; }
static float    __uint_as_float(unsigned u) { float f; std::memcpy(&f, &u, 4); return f; }
static float    rcbrtf(float x) { return 1.0f / std::cbrt(x); }
static float    __frcp_rn(float x) { return 1.0f / x; }
#define __log2f std::log2
using std::fma;
#include "../nimblesm_gb300/csrc/hex_math.cuh"
#undef __log2f
#include "../nimblesm_gb300/csrc/hex_fixed.cuh"

using namespace nsm;
using namespace nsm::fx;
using Real = long double;

template <class T>
void shape(int p, int n, T d[3])
{
  const T g = (T)kGauss;
  const T sx = sx_of(n) ? 1 : -1, sy = sy_of(n) ? 1 : -1, sz = sz_of(n) ? 1 : -1;
  const T x = 1 + sx * (sx_of(p) ? g : -g), y = 1 + sy * (sy_of(p) ? g : -g), z = 1 + sz * (sz_of(p) ? g : -g);
  d[0] = sx * y * z / 8, d[1] = sy * x * z / 8, d[2] = sz * x * y / 8;
}
template <class T>
T cofactors(const T M[3][3], T C[3][3])
{
  for (int r = 0; r < 3; r++)
    for (int c = 0; c < 3; c++) {
      const int r1 = (r + 1) % 3, r2 = (r + 2) % 3, c1 = (c + 1) % 3, c2 = (c + 2) % 3;
      C[r][c] = M[r1][c1] * M[r2][c2] - M[r1][c2] * M[r2][c1];
    }
  return M[0][0] * C[0][0] + M[0][1] * C[0][1] + M[0][2] * C[0][2];
}

struct Element {
  double u[8][3], G0[8][3][3], det[8], JX8[8][3][3], idet[8];
};

void exact(const Element& e, int model, Real K, Real G, Real f[8][3], Real sig[8][6])
{
  std::memset(f, 0, sizeof(Real) * 24);
  for (int p = 0; p < 8; p++) {
    Real Du[3][3] = {}, dn[8][3], H[3][3], C[3][3], s[3][3], B[3][3];
    for (int n = 0; n < 8; n++) {
      shape<Real>(p, n, dn[n]);
      for (int i = 0; i < 3; i++)
        for (int d = 0; d < 3; d++) Du[i][d] += 8 * dn[n][d] * (Real)e.u[n][i];
    }
    for (int i = 0; i < 3; i++)
      for (int J = 0; J < 3; J++) {
        H[i][J] = 0;
        for (int d = 0; d < 3; d++) H[i][J] += Du[i][d] * (Real)e.G0[p][d][J];
      }
    // cofactors of I + H and J - 1 without the cancellation
    for (int r = 0; r < 3; r++)
      for (int c = 0; c < 3; c++) {
        const int r1 = (r + 1) % 3, r2 = (r + 2) % 3, c1 = (c + 1) % 3, c2 = (c + 2) % 3;
        C[r][c] = (r == c ? 1 + H[r1][r1] + H[r2][r2] : -H[c][r]) + H[r1][c1] * H[r2][c2] - H[r1][c2] * H[r2][c1];
      }
    const Real tr = H[0][0] + H[1][1] + H[2][2];
    const Real t  = tr + H[0][0] * (H[1][1] + H[2][2]) + H[1][1] * H[2][2] - H[0][1] * H[1][0] - H[0][2] * H[2][0] -
                   H[1][2] * H[2][1] + H[0][0] * (H[1][1] * H[2][2] - H[1][2] * H[2][1]) +
                   H[0][1] * (H[1][2] * H[2][0] - H[1][0] * H[2][2]) + H[0][2] * (H[1][0] * H[2][1] - H[1][1] * H[2][0]);
    for (int i = 0; i < 3; i++)
      for (int j = 0; j < 3; j++) B[i][j] = H[i][j] + H[j][i] + H[i][0] * H[j][0] + H[i][1] * H[j][1] + H[i][2] * H[j][2];
    const Real g = G * std::exp(-std::log1p(t) * 5 / 3), m = (B[0][0] + B[1][1] + B[2][2]) / 3, pr = K / 2 * (t + t / (1 + t));
    for (int i = 0; i < 3; i++)
      for (int j = 0; j < 3; j++)
        s[i][j] = model == kElastic ? G * (H[i][j] + H[j][i]) + (i == j ? (K - 2 * G / 3) * tr : 0)
                                    : g * (B[i][j] - (i == j ? m : 0)) + (i == j ? pr : 0);
    const Real o[6] = {s[0][0], s[1][1], s[2][2], s[0][1], s[1][2], s[2][0]};
    for (int q = 0; q < 6; q++) sig[p][q] = o[q];
    for (int n = 0; n < 8; n++)
      for (int i = 0; i < 3; i++)
        for (int d = 0; d < 3; d++) {
          Real Q = 0;
          for (int k = 0; k < 3; k++)
            for (int J = 0; J < 3; J++) Q += 8 * (Real)e.det[p] * (Real)e.G0[p][d][J] * C[k][J] * s[k][i];
          f[n][i] -= dn[n][d] * Q;
        }
  }
}

// The FP64 code (element_work).
void in_fp64(const Element& e, int model, double K, double G, double f[8][3], double sig[8][6])
{
  double x[8][3], Gu[3][3][2][2], S[3][3][2][2] = {};
  std::memcpy(x, e.u, sizeof x);
  nodal_gradient<double>(x, Gu);
  for (int p = 0; p < 8; p++) {
    const int bit[3] = {sx_of(p), sy_of(p), sz_of(p)};
    double    Du[3][3], H[3][3], Jx[3][3], Cx[3][3];
    for (int i = 0; i < 3; i++)
      for (int d = 0; d < 3; d++) {
        Du[i][d] = Gu[d][i][bit[other1(d)]][bit[other2(d)]];
        Jx[i][d] = e.JX8[p][i][d] + Du[i][d];
      }
    for (int i = 0; i < 3; i++)
      for (int J = 0; J < 3; J++) H[i][J] = fma(Du[i][0], e.G0[p][0][J], fma(Du[i][1], e.G0[p][1][J], Du[i][2] * e.G0[p][2][J]));
    const double J = cofactor3<double>(Jx, Cx) * e.idet[p];
    material_stress_j<double>(model, H, J, K, G, sig[p]);
    for (int d = 0; d < 3; d++)
      for (int i = 0; i < 3; i++) {
        double&      acc  = S[d][i][bit[other1(d)]][bit[other2(d)]];
        const double tail = first_of_pair(d, p) ? Cx[2][d] * sym(sig[p], 2, i) : fma(Cx[2][d], sym(sig[p], 2, i), acc);
        acc               = fma(Cx[0][d], sym(sig[p], 0, i), fma(Cx[1][d], sym(sig[p], 1, i), tail));
      }
  }
  nodal_adjoint<double>(S, -1.0 / 512.0, f);
}

int length(u64 m)
{
  int bits = 0;
  while (bits < 64 && (m >> bits)) bits++;
  return bits;
}

// The kernel's evaluation (k_fixed_geometry, fixed_material and k_element_fixed
// of element_fixed.cu), its four lanes in turn; false outside the domain.
bool fixed_point(const Element& el, int model, double K, double G, double f[8][3], double sig[8][6])
{
  const bool elastic = model == kElastic;
  if (elastic ? K > 4 * G : 2 * K < G) return false;
  double row[3] = {}, dmax = 0;
  for (int p = 0; p < 8; p++) {
    for (int q = 0; q < 9; q++) row[q / 3] = std::fmax(row[q / 3], std::fabs(el.G0[p][q / 3][q % 3]));
    dmax = std::fmax(dmax, el.det[p]);
  }
  const int eg = std::max({std::ilogb(row[0]), std::ilogb(row[1]), std::ilogb(row[2])});
  int       places[3] = {};
  for (int d = 0; d < 3 && elastic; d++) {
    places[d] = eg - std::ilogb(row[d]);
    if (places[d] > kMaxRow) return false;
  }
  const Rows r{places[0], places[1], places[2]};
  const int  sG = 60 - eg, ed = std::ilogb(dmax) + 1, su = 124 - sG, EM = std::ilogb(std::fmax(K, G)) + 4;
  const Moduli m{std::llrint(std::ldexp(K, 61 - EM)), std::llrint(std::ldexp(G, 62 - EM)),
                 std::llrint(std::ldexp(K - 2 * G / 3, 62 - EM)), EM, model};
  int  exm  = 0;
  bool zero = true;
  for (int n = 0; n < 24; n++) {
    exm  = std::max(exm, (__double2hiint(el.u[n / 3][n % 3]) >> 20) & 0x7ff);
    zero = zero && el.u[n / 3][n % 3] == 0.0;
  }
  if (elastic && (exm > 0x7f7 || (exm < 179 && !zero))) return false;
  const int sc = std::min(1079 - exm, elastic ? 900 : su);
  int       sh = su - sc, e = 0;
  unsigned  bad = 0;
  i64       c[4][3][2], q[4][3][2][2], v[4][3][7];
  for (int l = 0; l < 4; l++)  // lane l: sides l & 1 along eta, l >> 1 along zeta
    for (int k = 0; k < 6; k++) {
      const double u = el.u[corner_of(k & 1, l & 1, l >> 1)][k >> 1];
      c[l][k >> 1][k & 1] = to_fixed((unsigned)__double2hiint(u), (unsigned)__double2loint(u), 1086 - sc);
    }
  for (int l = 0; l < 4; l++)
    for (int i = 0; i < 3; i++) {
      const i64 s = c[l][i][1] + c[l][i][0], d = c[l][i][1] - c[l][i][0];
      const i64 so = c[l ^ 1][i][1] + c[l ^ 1][i][0], dn = c[l ^ 1][i][1] - c[l ^ 1][i][0];
      q[l][i][0][0] = s + so, q[l][i][0][1] = d + dn, q[l][i][1][0] = s - so, q[l][i][1][1] = d - dn;
    }
  u64 most = 0;
  for (int l = 0; l < 4; l++)
    for (int i = 0; i < 3; i++) {
      lane_modes(q[l][i], q[l ^ 2][i], v[l][i]);
      if (elastic) most |= mode_bits(v[l][i], r);
    }
  int ef = ed - sG + 2;
  if (elastic) {
    if (most == 0) sh = 0;
    else elastic_scale(length(most) - kMaxRow, sc, su, sh, e);
    if (e < -3 || std::min(ef, 0) + EM - e < -900) return false;
  } else if (sh > 26) {
    return false;
  }
  Parts keep[4][3], send[4][3];
  for (int l = 0; l < 4; l++) {
    Gradient gr[3];
    Sums     S[3] = {};
    for (int i = 0; i < 3; i++) {
      if (elastic) {
        elastic_shift(v[l][i], r, sh);
        elastic_gradient(v[l][i], r, gr[i]);
      } else {
        if (sh != 0) bad |= lane_shift(v[l][i], sh);
        lane_gradient(v[l][i], gr[i]);
      }
    }
    for (int bx = 0; bx < 2; bx++) {
      const int p = corner_of(bx, l & 1, l >> 1);
      i64       Du[3][3], He[3][3], P[3][3], Q[3][3];
      Limbs     g0[3][3];
      Point     pt;
      for (int i = 0; i < 3; i++)
        Du[i][0] = gr[i].x, Du[i][1] = gr[i].y + (bx ? gr[i].y1 : 0), Du[i][2] = gr[i].z + (bx ? gr[i].z1 : 0);
      for (int d = 0; d < 3; d++)
        for (int J = 0; J < 3; J++) {
          const bool flip = (d == 1 && !(l & 1)) || (d == 2 && !(l >> 1));
          g0[d][J]        = split(std::llrint(std::ldexp(flip ? -el.G0[p][d][J] : el.G0[p][d][J], sG + places[d])));
        }
      const i64 det = std::llrint(std::ldexp(el.det[p], 62 - ed));
      if (elastic) {
        displacement_gradient<true>(Du, g0, He);
        for (int k = 0; k < 9; k++) {
          pt.H[k / 3][k % 3] = e > 0 ? He[k / 3][k % 3] >> std::min(e, 63) : (i64)((u64)He[k / 3][k % 3] << -e);
          bad |= outside<27>(pt.H[k / 3][k % 3]);
        }
      } else {
        displacement_gradient(Du, g0, pt.H);
      }
      bad |= kinematics(pt);
      if (elastic) bad |= elastic_force<true>(m, det, He, pt, P);
      else bad |= neohookean_force<true>(m, det, pt, P);
      for (int k = 0; k < 6; k++) sig[p][k] = std::ldexp((double)pt.sig[k], EM - 62 - e);
      point_force(g0, P, Q);
      for (int i = 0; i < 3; i++) {
        S[i].x += Q[0][i];
        S[i].y += Q[1][i], S[i].y1 += bx ? Q[1][i] : -Q[1][i];
        S[i].z += Q[2][i], S[i].z1 += bx ? Q[2][i] : -Q[2][i];
      }
    }
    for (int i = 0; i < 3; i++) {
      if (elastic) {
        common_scale(S[i], r);
        bad |= too_large(S[i]);
      }
      lane_adjoint(S[i], keep[l][i], send[l][i]);
    }
  }
  if (bad) return false;
  ef += EM - e - (elastic ? kElasticForce - kElasticSum : 0);
  for (int i = 0; i < 3; i++) {
    Parts t[4];
    for (int l = 0; l < 4; l++) {
      const Parts &a = keep[l][i], &b = send[l ^ 2][i];
      t[l] = Parts{a.e0 + b.e0, a.e1 + b.e1, a.o0 + b.o0, a.o1 + b.o1};
    }
    for (int l = 0; l < 4; l++) {
      const i64 ev = t[l].e0 + t[l].e1 + (t[l ^ 1].e0 - t[l ^ 1].e1), od = t[l].o0 + t[l].o1 + (t[l ^ 1].o0 - t[l ^ 1].o1);
      f[corner_of(0, l & 1, l >> 1)][i] = std::ldexp((double)(od - ev), ef);
      f[corner_of(1, l & 1, l >> 1)][i] = std::ldexp((double)(-od - ev), ef);
    }
  }
  return true;
}

struct Kind {
  const char* name;
  double      thin[3] = {1, 1, 1}, jitter = 0.1, strain = 1e-3, rotation = 0, ratio = 2, rigid = 0;
  double      all = 0;  // this value at every corner instead (in x alone: `component`)
  bool        component = false;
  bool        swelling = false;  // the same strain in all directions, axes aligned
};

void rotation(double w, double x, double y, double z, double R[3][3])
{
  const double n = std::sqrt(w * w + x * x + y * y + z * z);
  w /= n, x /= n, y /= n, z /= n;
  const double M[3][3] = {{1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)},
                          {2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)},
                          {2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)}};
  std::memcpy(R, M, sizeof M);
}

int main(int argc, char** argv)
{
  const int count = argc > 1 ? std::atoi(argv[1]) : 300;
  const double inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
  std::vector<Kind> kinds;
  auto add = [&](const char* name) -> Kind& {
    kinds.push_back(Kind{});
    kinds.back().name = name;
    return kinds.back();
  };
  add("plain");
  for (double a : {1.5, 2.0, 3.0, 4.0}) add("flat").thin[2] = a;
  for (double a : {2.0, 3.5}) {
    Kind& k = add("needle");
    k.thin[1] = k.thin[2] = a;
  }
  for (double a : {30.0, 1000.0}) add("very_flat").thin[2] = a;
  for (double j : {0.0, 0.2, 0.3}) add("jitter").jitter = j;
  for (double r : {0.6, 1.0, 2.5, 3.6}) add("moduli").ratio = r;
  for (double r : {0.05, 0.3}) add("soft_in_volume").ratio = r;
  for (double r : {5.0, 20.0, 1e6}) add("soft_in_shear").ratio = r;
  for (double s : {1e-12, 1e-9, 1e-6, 1e-4, 1e-2, 3e-2, 5e-2}) add("strain").strain = s;
  for (double s : {1e-240, 1e-100, 1e-30, 1e-20, 1e-15}) add("tiny_strain").strain = s;
  for (double s : {1e-270, 5e-322}) add("below_the_scales").strain = s;
  for (double s : {0.08, 0.12, 0.2, 0.3}) add("large_strain").strain = s;
  for (double a : {0.01, 0.03, 0.05, 0.1, 0.2, 0.34}) add("turned").rotation = a;
  for (double a : {0.1, 0.3}) {
    Kind& k    = add("turned_and_strained");
    k.rotation = a, k.strain = 0.03;
  }
  for (double a : {1.0, 3.0}) {
    Kind& k    = add("swelling");
    k.swelling = true, k.jitter = 0, k.thin[2] = a;
  }
  add("turned_far").rotation = 0.6;
  for (double t : {1e-2, 1.0, 1e3}) add("moved").rigid = t;
  for (double x : {inf, -inf, nan, 1e307})
    for (bool c : {false, true}) {
      Kind& k     = add("not_numbers");
      k.all       = x;
      k.component = c;
    }
  for (int model = 0; model < 2; model++)
    for (const Kind& k : kinds) {
      std::mt19937_64 rng(7);
      auto        uniform = [&](double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); };
      long double sum[4] = {};
      int         outside = 0;
      for (int it = 0; it < count; it++) {
        const double h = std::pow(10.0, uniform(-3, 0.5)), G = 79.3e9 * uniform(0.5, 2), K = G * k.ratio * uniform(0.9, 1.1);
        Element      e;
        double       X[8][3], R[3][3], W[3][3], A[3][3], t[3];
        rotation(uniform(-1, 1), uniform(-1, 1), uniform(-1, 1), uniform(-1, 1), R);
        rotation(std::cos(k.rotation / 2), std::sin(k.rotation / 2), 0, 0, W);
        for (int i = 0; i < 3; i++) {
          t[i] = k.rigid * h * uniform(-1, 1);
          for (int j = 0; j < 3; j++) A[i][j] = k.strain * uniform(-1, 1) + (W[i][j] - (i == j));
          for (int j = 0; j < 3 && k.swelling; j++) A[i][j] = i == j ? k.strain : 0, R[i][j] = i == j;
        }
        for (int n = 0; n < 8; n++) {
          const int b[3] = {sx_of(n), sy_of(n), sz_of(n)};
          double    x[3];
          for (int i = 0; i < 3; i++) x[i] = h / k.thin[i] * (b[i] + uniform(-k.jitter, k.jitter));
          for (int i = 0; i < 3; i++) X[n][i] = R[i][0] * x[0] + R[i][1] * x[1] + R[i][2] * x[2];
        }
        const double least = h / std::max({k.thin[0], k.thin[1], k.thin[2]});
        for (int n = 0; n < 8; n++)
          for (int i = 0; i < 3; i++) {
            e.u[n][i] = t[i] + A[i][0] * X[n][0] + A[i][1] * X[n][1] + A[i][2] * X[n][2] + (k.swelling ? 0 : k.strain) * 0.1 * least * uniform(-1, 1);
            if (k.all != 0 && (i == 0 || !k.component)) e.u[n][i] = k.all;
          }
        for (int p = 0; p < 8; p++) {
          double JX[3][3] = {}, C[3][3];
          for (int n = 0; n < 8; n++) {
            double d[3];
            shape<double>(p, n, d);
            for (int i = 0; i < 3; i++)
              for (int j = 0; j < 3; j++) JX[i][j] += X[n][i] * d[j];
          }
          e.det[p]  = cofactors(JX, C);
          e.idet[p] = 1 / e.det[p] / 512;
          for (int i = 0; i < 3; i++)
            for (int J = 0; J < 3; J++) e.G0[p][i][J] = C[J][i] / e.det[p] / 8, e.JX8[p][i][J] = 8 * JX[i][J];
        }
        Real   f[8][3], s[8][6];
        double ff[8][3], sf[8][6], fd[8][3], sd[8][6];
        if (!fixed_point(e, model, K, G, ff, sf)) {
          outside++;
          continue;
        }
        exact(e, model, K, G, f, s);
        in_fp64(e, model, K, G, fd, sd);
        Real d[4] = {}, nf = 0, ns = 0;
        for (int n = 0; n < 24; n++) {
          const Real x = f[n / 3][n % 3], a = ff[n / 3][n % 3] - x, b = fd[n / 3][n % 3] - x;
          nf += x * x, d[0] += a * a, d[1] += b * b;
        }
        for (int n = 0; n < 48; n++) {
          const Real x = s[n / 6][n % 6], a = sf[n / 6][n % 6] - x, b = sd[n / 6][n % 6] - x;
          ns += x * x, d[2] += a * a, d[3] += b * b;
        }
        for (int j = 0; j < 4; j++) sum[j] += (j < 2 ? nf : ns) > 0 ? d[j] / (j < 2 ? nf : ns) : 0;
      }
      const int in = std::max(1, count - outside);
      std::printf("%d %s %d %.3e %.3e %.3e %.3e\n", model, k.name, outside, (double)std::sqrt(sum[0] / in),
                  (double)std::sqrt(sum[1] / in), (double)std::sqrt(sum[2] / in), (double)std::sqrt(sum[3] / in));
    }
}
