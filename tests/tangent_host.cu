/* Host check of the element algebra (biofem-ia_gb300/csrc/element.cuh) for
   tests/test_tangent_host.py.  argv: nq, corrector steps, prism normal (0/1).
   For a seeded element state and seeded reference constants of the sizes that
   occur, prints
     1. the largest difference of the analytic tangent (tangent_coefs,
        tangent_block) from central differences of the element forces, both in
        long double, relative to the largest entry;
     2. the largest difference of the double tangent from the long-double one;
     3. the largest error of FFAcc's sums of nine products over 24 decades
        against long double, relative to the sum of the magnitudes;
     4. the status bits that any evaluation raised. */
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <vector>

namespace biofem {
inline long double dsqrt(long double a) { return sqrtl(a); }
inline long double dabs(long double a) { return fabsl(a); }
}
#include "../biofem-ia_gb300/csrc/element.cuh"

using namespace biofem;
typedef long double L;

static uint64_t g_state = 0x9e3779b97f4a7c15ull;
static double urand()
{
  g_state = g_state * 6364136223846793005ull + 1442695040888963407ull;
  return (double)(g_state >> 11) * (1.0 / 9007199254740992.0);
}
static double rnd() { return 2.0 * urand() - 1.0; }

template <class R> static void tangent(const R y[15], const EPar<R> &p, const R *ref, R D[15][15], int &st)
{
  const ElemGeom<R> g = elem_geom<R>(y, p);
  R N[3], M[3];
  TanMoments<R> mo;
  mo.clear();
  elem_resultants<R>(g, p, RefCol<R>{ref, 1}, N, M, st, true, true,
                     [&](int, R w, R th, const R(*C)[5]) { mo.add(w, th, C); });
  R c[kTanCoefs];
  tangent_coefs(g, N, M, mo, p.tnormal, [&](int k, R v) { c[k] = v; });
  for (int s = 0; s < 5; s++) {
    R B[15][3];
    tangent_block<R>(s, [&](int k) { return c[k]; }, B);
    for (int i = 0; i < 15; i++)
      for (int j = 0; j < 3; j++) D[i][3 * s + j] = B[i][j];
  }
}

template <class R> static EPar<R> params(int nq, int iters, int tnormal)
{
  EPar<R> p;
  p.nq = nq; p.iters = iters; p.tnormal = tnormal;
  p.mu = (R)0.3846; p.K = (R)0.8333; p.hhalf = (R)0.005;
  for (int q = 0; q < nq; q++) {
    p.theta[q] = (R)(-0.9 + 0.37 * q);
    p.w[q] = (R)(0.3 + 0.05 * q);
  }
  return p;
}

int main(int argc, char **argv)
{
  const int nq = std::atoi(argv[1]), iters = std::atoi(argv[2]), tn = std::atoi(argv[3]);
  const L h = 0.03L;
  int st = 0;
  L e_fd = 0, e_double = 0;
  for (int trial = 0; trial < 8; trial++) {
    const EPar<L> p = params<L>(nq, iters, tn);
    /* edges h e1, h (0.5, 0.85), second derivatives of size 5 h^2 */
    L y[15] = {h * (1 + 0.1L * rnd()), h * 0.2L * rnd(), h * 0.1L * rnd(),
               h * 0.5L * (1 + 0.1L * rnd()), h * 0.85L * (1 + 0.1L * rnd()), h * 0.1L * rnd()};
    for (int k = 6; k < 15; k++) y[k] = h * h * 5 * rnd();
    std::vector<L> ref((size_t)kRefPerQp * nq + 1);
    const L g00 = h * h, g11 = h * h * 0.9L, g01 = h * h * 0.45L, det = g00 * g11 - g01 * g01;
    for (int q = 0; q < nq; q++) {
      L *o = &ref[(size_t)kRefPerQp * q];
      o[0] = p.mu; o[1] = p.mu * g11 / det * 1.3L; o[2] = p.mu * g00 / det; o[3] = -p.mu * g01 / det;
      for (int f = 0; f < 10; f++) {
        L *u = o + 4 + 4 * f;
        for (int m = 0; m < 3; m++) u[m] = 0.02L * h * h * rnd();
        u[3] = f == 0 ? 2.0L : f < 4 ? 0.01L * rnd() / (h * h) : 1.0L + 0.05L * rnd();
      }
      o[kRfB00] += 2; o[kRfB11 + 1] += 2; o[kRfB01 + 2] += 2;
      o[kRfRho] = 1 / (det * 0.81L);
    }
    ref[(size_t)kRefPerQp * nq] = 0.005L * h * h / 2;
    L D[15][15], mx = 0, err = 0;
    tangent<L>(y, p, ref.data(), D, st);
    for (int k = 0; k < 15; k++) {
      const L d = (k < 6 ? h : h * h * 5) * 1e-6L;
      L z[15], f1[15], f2[15];
      for (int i = 0; i < 15; i++) z[i] = y[i];
      z[k] = y[k] + d;
      elem_forces<L>(z, p, RefCol<L>{ref.data(), 1}, f1, st);
      z[k] = y[k] - d;
      elem_forces<L>(z, p, RefCol<L>{ref.data(), 1}, f2, st);
      for (int i = 0; i < 15; i++) {
        const L v = (f1[i] - f2[i]) / (2 * d);
        mx = fmaxl(mx, fabsl(v));
        err = fmaxl(err, fabsl(v - D[i][k]));
      }
    }
    e_fd = fmaxl(e_fd, err / mx);
    const EPar<double> pd = params<double>(nq, iters, tn);
    const std::vector<double> rd(ref.begin(), ref.end());
    double yd[15], Dd[15][15];
    L ed = 0;
    for (int i = 0; i < 15; i++) yd[i] = (double)y[i];
    tangent<double>(yd, pd, rd.data(), Dd, st);
    for (int i = 0; i < 15; i++)
      for (int j = 0; j < 15; j++) ed = fmaxl(ed, fabsl(Dd[i][j] - D[i][j]));
    e_double = fmaxl(e_double, ed / mx);
  }
  L e_acc = 0;
  for (int k = 0; k < 20000; k++) {
    const auto operand = [] { return FF((urand() < 0.5 ? -1.0 : 1.0) * std::pow(10.0, -6.0 + 12.0 * urand()) * (1.0 + urand())); };
    const auto ld = [](FF a) { return (L)a.hi + (L)a.lo; };
    FF a = operand(), b = operand();
    FFAcc s(a, b);
    L exact = ld(a) * ld(b), mag = fabsl(exact);
    for (int t = 1; t < 9; t++) {
      a = operand(); b = operand();
      s.add(a, b);
      exact += ld(a) * ld(b);
      mag += fabsl(ld(a) * ld(b));
    }
    e_acc = fmaxl(e_acc, fabsl(ld(s.get()) - exact) / mag);
  }
  std::printf("%.3Le %.3Le %.3Le %d\n", e_fd, e_double, e_acc, st);
  return 0;
}
