// Host check of the fixed-point element arithmetic (hex_fixed.cuh): random
// elements, each evaluated as the kernel's four lanes evaluate it, against the
// same formulas in extended precision, and beside them in FP64 as the FP64
// code forms them (J from the cofactors of the current Jacobian).  Prints, per
// material, rigid displacement and strain scale, the relative errors of forces
// and stresses of both and the number of elements outside the domain.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

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

template <class T>
void evaluate(const Element& e, int model, T K, T G, bool current_jacobian, T f[8][3], T sig[8][6])
{
  std::memset(f, 0, sizeof(T) * 24);
  for (int p = 0; p < 8; p++) {
    T Du[3][3] = {}, dn[8][3], H[3][3], F[3][3], C[3][3], Cx[3][3];
    for (int n = 0; n < 8; n++) {
      shape<T>(p, n, dn[n]);
      for (int i = 0; i < 3; i++)
        for (int d = 0; d < 3; d++) Du[i][d] += 8 * dn[n][d] * (T)e.u[n][i];
    }
    for (int i = 0; i < 3; i++)
      for (int J = 0; J < 3; J++) {
        H[i][J] = Du[i][0] * (T)e.G0[p][0][J] + Du[i][1] * (T)e.G0[p][1][J] + Du[i][2] * (T)e.G0[p][2][J];
        F[i][J] = H[i][J] + (i == J ? 1 : 0);
      }
    T J = cofactors(F, C);
    if (current_jacobian) {
      T Jx[3][3];
      for (int i = 0; i < 3; i++)
        for (int d = 0; d < 3; d++) Jx[i][d] = (T)e.JX8[p][i][d] + Du[i][d];
      J = cofactors(Jx, Cx) * (T)e.idet[p];
    }
    const T tr = H[0][0] + H[1][1] + H[2][2];
    T       s[3][3], B[3][3];
    for (int i = 0; i < 3; i++)
      for (int j = 0; j < 3; j++) B[i][j] = H[i][j] + H[j][i] + H[i][0] * H[j][0] + H[i][1] * H[j][1] + H[i][2] * H[j][2];
    const T g = G * std::pow(J, T(-5) / T(3)), m = (B[0][0] + B[1][1] + B[2][2]) / 3, pr = K / 2 * (J - 1 / J);
    for (int i = 0; i < 3; i++)
      for (int j = 0; j < 3; j++)
        s[i][j] = model == kElastic ? G * (H[i][j] + H[j][i]) + (i == j ? (K - 2 * G / 3) * tr : 0)
                                    : g * (B[i][j] - (i == j ? m : 0)) + (i == j ? pr : 0);
    const T o[6] = {s[0][0], s[1][1], s[2][2], s[0][1], s[1][2], s[2][0]};
    for (int q = 0; q < 6; q++) sig[p][q] = o[q];
    for (int n = 0; n < 8; n++)
      for (int i = 0; i < 3; i++)
        for (int d = 0; d < 3; d++) {
          T Q = 0;
          for (int k = 0; k < 3; k++) {
            if (current_jacobian) Q += Cx[k][d] * s[k][i] / 64;
            else
              for (int Jc = 0; Jc < 3; Jc++) Q += 8 * (T)e.det[p] * (T)e.G0[p][d][Jc] * C[k][Jc] * s[k][i];
          }
          f[n][i] -= dn[n][d] * Q;
        }
  }
}

// The kernel's evaluation, its four lanes in turn; false outside the domain.
bool fixed_point(const Element& el, int model, double K, double G, double f[8][3], double sig[8][6])
{
  double gmax = 0, dmax = 0;
  for (int p = 0; p < 8; p++) {
    for (int q = 0; q < 9; q++) gmax = std::fmax(gmax, std::fabs(el.G0[p][q / 3][q % 3]));
    dmax = std::fmax(dmax, el.det[p]);
  }
  const int sG = 60 - std::ilogb(gmax), ed = std::ilogb(dmax) + 1, su = 124 - sG, EM = std::ilogb(std::fmax(K, G)) + 4;
  const Moduli m{std::llrint(std::ldexp(K / 2, 62 - EM)), std::llrint(std::ldexp(G, 62 - EM)),
                 std::llrint(std::ldexp(K - 2 * G / 3, 62 - EM)), EM, model};
  int exm = 0;
  for (int n = 0; n < 24; n++) {
    u64 b;
    std::memcpy(&b, &el.u[n / 3][n % 3], 8);
    exm = std::max(exm, (int)((b >> 52) & 0x7ff));
  }
  const bool elastic = model == kElastic;
  const int  sc = elastic ? 1079 - exm : std::min(su, 1079 - exm);
  int        sh = su - sc, e = 0;
  unsigned   bad = 0;
  i64        c[4][3][2], q[4][3][2][2], v[4][3][7];
  for (int l = 0; l < 4; l++)  // lane l: sides l & 1 along eta, l >> 1 along zeta
    for (int k = 0; k < 6; k++) {
      u64 b;
      std::memcpy(&b, &el.u[corner_of(k & 1, l & 1, l >> 1)][k >> 1], 8);
      c[l][k >> 1][k & 1] = to_fixed((unsigned)(b >> 32), (unsigned)b, 1086 - sc);
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
      for (int k = 0; k < 7; k++) most |= (u64)(v[l][i][k] ^ (v[l][i][k] >> 63));
    }
  if (elastic) {
    int bits = 0;
    while (bits < 64 && (most >> bits)) bits++;
    if (bits == 0) sh = 0;
    else elastic_scale(bits, sc, su, sh, e);
    if (e < -3) return false;
  } else if (sh > 26) {
    return false;
  }
  Parts keep[4][3], send[4][3];
  for (int l = 0; l < 4; l++) {
    Gradient gr[3];
    Sums     S[3] = {};
    for (int i = 0; i < 3; i++) {
      if (elastic)
        for (int k = 0; k < 7; k++) v[l][i][k] = sh >= 0 ? (i64)((u64)v[l][i][k] << sh) : v[l][i][k] >> std::min(-sh, 63);
      else if (sh != 0) bad |= lane_shift(v[l][i], sh);
      lane_gradient(v[l][i], gr[i]);
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
          g0[d][J]        = split(std::llrint(std::ldexp(flip ? -el.G0[p][d][J] : el.G0[p][d][J], sG)));
        }
      const i64 det = std::llrint(std::ldexp(el.det[p], 62 - ed));
      displacement_gradient(Du, g0, He);
      for (int k = 0; k < 9; k++) pt.H[k / 3][k % 3] = e > 0 ? He[k / 3][k % 3] >> e : (i64)((u64)He[k / 3][k % 3] << -e);
      if (elastic)
        for (int k = 0; k < 9; k++) bad |= outside<27>(pt.H[k / 3][k % 3]);
      bad |= kinematics(pt);
      if (elastic) bad |= elastic_force<true>(m, det, He, pt, P);
      else neohookean_force<true>(m, det, pt, P);
      for (int k = 0; k < 6; k++) sig[p][k] = std::ldexp((double)pt.sig[k], EM - 62 - e);
      point_force(g0, P, Q);
      for (int i = 0; i < 3; i++) {
        S[i].x += Q[0][i];
        S[i].y += Q[1][i], S[i].y1 += bx ? Q[1][i] : -Q[1][i];
        S[i].z += Q[2][i], S[i].z1 += bx ? Q[2][i] : -Q[2][i];
      }
    }
    for (int i = 0; i < 3; i++) {
      if (elastic) bad |= too_large(S[i]);
      lane_adjoint(S[i], keep[l][i], send[l][i]);
    }
  }
  if (bad) return false;
  const int ef = ed - sG + 2 + EM - e - (elastic ? kElasticForce : 0);
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

int main(int argc, char** argv)
{
  const int       count = argc > 1 ? std::atoi(argv[1]) : 300;
  std::mt19937_64 rng(argc > 2 ? std::atoi(argv[2]) : 1);
  auto            uniform = [&](double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); };
  for (int model = 0; model < 2; model++)
    for (double rigid : {0.0, 1e-2, 1.0})
      for (double strain : {1e-9, 1e-6, 1e-5, 1e-4, 1e-3, 1e-2, 3e-2, 1.0}) {
        long double ef = 0, ed = 0, nf = 0, es = 0, esd = 0, ns = 0;
        int         outside = 0;
        for (int it = 0; it < count; it++) {
          const double h = std::pow(10.0, uniform(-3, 0.5)), K = 160e9 * uniform(0.5, 2), G = 79.3e9 * uniform(0.05, 2);
          Element      e;
          double       X[8][3], A[3][3], t[3];
          for (int i = 0; i < 3; i++) {
            t[i] = rigid * uniform(-1, 1);
            for (int j = 0; j < 3; j++) A[i][j] = strain * uniform(-1, 1);
          }
          for (int n = 0; n < 8; n++) {
            const int b[3] = {sx_of(n), sy_of(n), sz_of(n)};
            for (int i = 0; i < 3; i++) X[n][i] = h * (b[i] + uniform(-0.2, 0.2));
          }
          for (int n = 0; n < 8; n++)
            for (int i = 0; i < 3; i++)
              e.u[n][i] = t[i] + A[i][0] * X[n][0] + A[i][1] * X[n][1] + A[i][2] * X[n][2] + strain * 0.1 * h * uniform(-1, 1);
          for (int p = 0; p < 8; p++) {
            double JX[3][3] = {}, C[3][3];
            for (int n = 0; n < 8; n++) {
              double d[3];
              shape<double>(p, n, d);
              for (int i = 0; i < 3; i++)
                for (int k = 0; k < 3; k++) JX[i][k] += X[n][i] * d[k];
            }
            e.det[p]  = cofactors(JX, C);
            e.idet[p] = 1 / e.det[p] / 512;
            for (int k = 0; k < 3; k++)
              for (int J = 0; J < 3; J++) e.G0[p][k][J] = C[J][k] / e.det[p] / 8, e.JX8[p][k][J] = 8 * JX[k][J];
          }
          Real   f[8][3], s[8][6];
          double fd[8][3], sd[8][6], ff[8][3], sf[8][6];
          if (!fixed_point(e, model, K, G, ff, sf)) {
            outside++;
            continue;
          }
          evaluate<Real>(e, model, K, G, false, f, s);
          evaluate<double>(e, model, K, G, true, fd, sd);
          const Real w = 1 / (h * h * K * strain), ws = 1 / (K * strain);
          for (int n = 0; n < 24; n++) {
            const Real x = f[n / 3][n % 3], a = ff[n / 3][n % 3] - x, b = fd[n / 3][n % 3] - x;
            ef += a * a * w * w, ed += b * b * w * w, nf += x * x * w * w;
          }
          for (int n = 0; n < 48; n++) {
            const Real x = s[n / 6][n % 6], a = sf[n / 6][n % 6] - x, b = sd[n / 6][n % 6] - x;
            es += a * a * ws * ws, esd += b * b * ws * ws, ns += x * x * ws * ws;
          }
        }
        auto rel = [](Real a, Real b) { return b > 0 ? (double)std::sqrt(a / b) : 0.0; };
        std::printf("%d %g %g %.3e %.3e %.3e %.3e %d\n", model, rigid, strain, rel(ef, nf), rel(ed, nf), rel(es, ns),
                    rel(esd, ns), outside);
      }
}
