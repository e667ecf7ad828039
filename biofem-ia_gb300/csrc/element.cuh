/*
 * Element physics of the active-strain Kirchhoff-Love shell, written once for
 * double, float and float-float: the internal force, the gradient of the
 * stress along the metric, and from it the force's derivative.
 *
 * The element is reduced to 15 "generalised coordinates"
 *   y = (a1, a2, Aaa, Abb, Aab) = N x_patch,
 * the centroid tangents and second derivatives of the Loop-subdivision patch
 * (active_strain.c:514-540 regular, :668-694 irregular).  The internal force
 * of the reference (ElemUpdFint, active_strain.c:1762-1995) is exactly
 *   Fb_a = sum_r N[r][a] f_r(y)   (r over the 5 rows of N, 3 components each)
 * with five force vectors f_r built from the membrane and bending resultants
 *   N^ab = pref0 sum_q w_q S_q^ab,  M^ab = pref0 sum_q w_q theta3_q S_q^ab:
 *   f1 = N11 a1 + N12 a2 - (gc1.Q) n,  f2 = N22 a2 + N12 a1 - (gc2.Q) n,
 *   f3 = -M11 n,  f4 = -M22 n,  f5 = -2 M12 n,   Q = M11 Aaa + M22 Abb + 2 M12 Aab.
 * The element stiffness is therefore K_e = N^T (df/dy) N.
 *
 * The stress S_q (ElemCGDefTens .. ModElemC33, active_strain.c:1332-1707,
 * 2048-2138) is evaluated in closed form.  With the reference-configuration
 * covariant fibre components t_i = g0_i . f, s = G^-1 t, phi = f.f, and the
 * active gradient Fa_cart = I - gamma f f^T:
 *   Fa.Cont = G^-1 - gamma s s^T,   Fa_inv.Cov = G + gamma' t t^T,
 *   gamma' = gamma / (1 - gamma phi);
 *   A = Fa.Cont G = I - gamma s t^T,  H = Fa_inv.Cov G^-1 = I + gamma' t s^T,
 *   A^T H = I.
 * Hence, for the "C_inv.Cont" matrix Ci of each C33 sub-iteration:
 *   Ce_inv = A Ci A^T,  Je = sqrt(rho / det Ci),  rho = 1 / (det G (1-gamma phi)^2),
 *   S  = mu (G^-1 + c1 s s^T) + alpha/2 (Ci + A Ci H),   c1 = 2 gamma' + gamma'^2 phi,
 *   CC3333 = 1/4 [2(beta-alpha) Qvv^2 + 4 beta Qvv Qwe - 4 alpha Qvw Qve
 *                 + (2beta-alpha) Qwe^2 - alpha Qww Qee],
 *   Qxy = (A^T x)^T Ci (A^T y),  v = Fa_inv.Cov G^-1 e3,  w = H v,
 *   alpha = K (Je^2 - Je) - mu,  beta = K Je (2 Je - 1) / 2,
 * which is the contraction the reference evaluates with its 3^6 and 3^8 loops
 * (active_strain.c:1381-1434, 1494-1532, 1592-1651).  All of it is linear in
 * Ci but for alpha, beta and the products of the Q's, so the per-(element, qp)
 * reference constants are the linear forms' coefficients, computed once per
 * mesh.
 */
#ifndef BIOFEM_ELEMENT_CUH
#define BIOFEM_ELEMENT_CUH

#include "biofem_host.h"
#include "ff.cuh"

namespace biofem {

/* ---------------- scalar types ---------------- */
__host__ __device__ __forceinline__ double dsqrt(double a) { return sqrt(a); }
__host__ __device__ __forceinline__ float dsqrt(float a) { return sqrtf(a); }
/* 1 / sqrt(a): one instruction sequence for double instead of two */
template <class R> __host__ __device__ __forceinline__ R drsqrt(R a) { return R(1) / dsqrt(a); }
#ifdef __CUDA_ARCH__
template <> __device__ __forceinline__ double drsqrt(double a) { return rsqrt(a); }
#endif
__host__ __device__ __forceinline__ double dabs(double a) { return fabs(a); }
__host__ __device__ __forceinline__ float dabs(float a) { return fabsf(a); }

template <class T> struct V3 { T x, y, z; };
template <class T> __host__ __device__ __forceinline__ V3<T> operator+(const V3<T> &a, const V3<T> &b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
template <class T> __host__ __device__ __forceinline__ V3<T> operator-(const V3<T> &a, const V3<T> &b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
template <class T, class S> __host__ __device__ __forceinline__ V3<T> scl(const S &s, const V3<T> &a) { return {s * a.x, s * a.y, s * a.z}; }

/* A sum of products: one chain of fused multiply-adds, or its float-float form. */
template <class R> struct Acc {
  R v;
  __host__ __device__ __forceinline__ Acc(R c) : v(c) {}
  __host__ __device__ __forceinline__ Acc(R a, R b) : v(a * b) {}
  __host__ __device__ __forceinline__ void add(R a, R b) { v = v + a * b; }
  __host__ __device__ __forceinline__ R get() const { return v; }
};
template <> struct Acc<FF> : FFAcc { using FFAcc::FFAcc; };
template <class R> __host__ __device__ __forceinline__ R pow2(R x, float c) { return x * R(c); }

/* a b + c d (+ e f) */
template <class R> __host__ __device__ __forceinline__ R sop(R a, R b, R c, R d) { Acc<R> s(a, b); s.add(c, d); return s.get(); }
template <class R> __host__ __device__ __forceinline__ R sop(R a, R b, R c, R d, R e, R f)
{
  Acc<R> s(a, b);
  s.add(c, d); s.add(e, f);
  return s.get();
}
/* c + a b */
template <class R> __host__ __device__ __forceinline__ R mad(R a, R b, R c) { Acc<R> s(c); s.add(a, b); return s.get(); }

template <class T> __host__ __device__ __forceinline__ T dot(const V3<T> &a, const V3<T> &b) { return sop(a.x, b.x, a.y, b.y, a.z, b.z); }
template <class T> __host__ __device__ __forceinline__ V3<T> cross(const V3<T> &a, const V3<T> &b)
{
  return {sop(a.y, b.z, -b.y, a.z), sop(b.x, a.z, -a.x, b.z), sop(a.x, b.y, -b.x, a.y)};
}
/* c + s a */
template <class T> __host__ __device__ __forceinline__ V3<T> mad(const T &s, const V3<T> &a, const V3<T> &c)
{
  return {mad(s, a.x, c.x), mad(s, a.y, c.y), mad(s, a.z, c.z)};
}
/* r a + s b + t c */
template <class T>
__host__ __device__ __forceinline__ V3<T> lin3(const T &r, const V3<T> &a, const T &s, const V3<T> &b, const T &t, const V3<T> &c)
{
  return {sop(r, a.x, s, b.x, t, c.x), sop(r, a.y, s, b.y, t, c.y), sop(r, a.z, s, b.z, t, c.z)};
}
/* a x b + c x d */
template <class T>
__host__ __device__ __forceinline__ V3<T> cross2(const V3<T> &a, const V3<T> &b, const V3<T> &c, const V3<T> &d)
{
  Acc<T> x(a.y, b.z), y(b.x, a.z), z(a.x, b.y);
  x.add(-b.y, a.z); x.add(c.y, d.z); x.add(-d.y, c.z);
  y.add(-a.x, b.z); y.add(d.x, c.z); y.add(-c.x, d.z);
  z.add(-b.x, a.y); z.add(c.x, d.y); z.add(-d.x, c.y);
  return {x.get(), y.get(), z.get()};
}

/* Reference constants of one (element, thickness point), kRefPerQp values.
   Everything the stress contracts the in-plane inverse metric with is linear
   in c = (c00, c11, c01, c22), so the constants are the forms' coefficients,
   four each, computed once per mesh (k_ref_prep in kernels.cu):
     S^33 etc. = S.. + alpha/2 B..(c),  Q_xy(c) of v, w, e3.
   A form costs 3 + 1 multiply-adds against the 5 to 9 of evaluating it from
   s, t, A^T v, ..., at 25 more loads a point, and FP64 is the bound: residual
   0.39 -> 0.31 ms on the 98,304-triangle sheet (0.28 now, 0.58 with gradients). */
enum {
  kRfS33 = 0, kRfS00, kRfS11, kRfS01,                       /* mu (G^-1 + c1 s s^T) */
  kRfB33 = 4, kRfB00 = 8, kRfB11 = 12, kRfB01 = 16,         /* Ci + A Ci H */
  kRfQvv = 20, kRfQww = 24, kRfQee = 28, kRfQvw = 32, kRfQve = 36, kRfQwe = 40,
  kRfRho = 44
};
static_assert(kRefPerQp == kRfRho + 1, "reference constants");

/* One element's column of the reference constants (SoA, stride = ne).  The
   float-float form keeps the heads and the tails as two float planes, the
   heads being the FP32 tangent's constants. */
template <class R> struct RefCol {
  const R *p;
  size_t stride;
  __host__ __device__ __forceinline__ R operator()(int k) const { return p[(size_t)k * stride]; }
  __host__ __device__ __forceinline__ RefCol at(int k) const { return {p + (size_t)k * stride, stride}; }
};
template <> struct RefCol<FF> {
  const float *p;
  size_t stride, tail;          /* distance of the tails' plane */
  __host__ __device__ __forceinline__ FF operator()(int k) const
  {
    return FF(p[(size_t)k * stride], p[tail + (size_t)k * stride]);
  }
  __host__ __device__ __forceinline__ RefCol at(int k) const { return {p + (size_t)k * stride, stride, tail}; }
};

/* One thickness point's constants in registers, loaded together (the FP32
   tangent waits for memory, not for arithmetic). */
template <class R> struct RefRegs {
  R v[kRefPerQp];
  __host__ __device__ __forceinline__ explicit RefRegs(const RefCol<R> &r)
  {
#pragma unroll
    for (int k = 0; k < kRefPerQp; k++) v[k] = r(k);
  }
  __host__ __device__ __forceinline__ R operator()(int k) const { return v[k]; }
};

/* Material / quadrature constants in the working precision R. */
template <class R> struct EPar {
  R mu, K, hhalf;
  R theta[kMaxQp], w[kMaxQp];
  int nq, iters;
  int tnormal;   /* 1: thickness metric from the tangential part of a3,alpha (extension) */
};

template <class R> __host__ __device__ __forceinline__ EPar<R> epar(const KParams &p);
template <> __host__ __device__ __forceinline__ EPar<double> epar<double>(const KParams &p)
{
  EPar<double> e;
  e.mu = p.mu; e.K = p.K; e.hhalf = p.hhalf; e.nq = p.nq; e.iters = p.iters; e.tnormal = p.tnormal;
  for (int q = 0; q < kMaxQp; q++) { e.theta[q] = p.theta[q]; e.w[q] = p.w[q]; }
  return e;
}
/* Float-float parameters (the FP32-bulk residual) */
/* float-float parameters were split on the host */
template <> __host__ __device__ __forceinline__ EPar<FF> epar<FF>(const KParams &p)
{
  EPar<FF> e;
  e.mu = FF(p.mu2[0], p.mu2[1]); e.K = FF(p.K2[0], p.K2[1]); e.hhalf = FF(p.hhalf2[0], p.hhalf2[1]);
  e.nq = p.nq; e.iters = p.iters; e.tnormal = p.tnormal;
  for (int q = 0; q < kMaxQp; q++) {
    e.theta[q] = FF(p.theta2[q][0], p.theta2[q][1]);
    e.w[q] = FF(p.w2[q][0], p.w2[q][1]);
  }
  return e;
}
/* FP32 parameters were converted on the host: no FP64 work in FP32 kernels */
template <> __host__ __device__ __forceinline__ EPar<float> epar<float>(const KParams &p)
{
  EPar<float> e;
  e.mu = p.muf; e.K = p.Kf; e.hhalf = p.hhalff; e.nq = p.nq; e.iters = p.iters; e.tnormal = p.tnormal;
  for (int q = 0; q < kMaxQp; q++) { e.theta[q] = p.thetaf[q]; e.w[q] = p.wf[q]; }
  return e;
}

/* d/dg of a symmetric inverse c = g^-1, restricted to the in-plane block:
   L[m][k] = d c_m / d g_k for c_m = c00, c11, c01 and the metric components
   g_k = 00, 11, 01, 02, 12 (dc = -c dg c; c02 = c12 = 0 for a 2x2 inverse). */
template <class R>
__host__ __device__ __forceinline__ void inverse_rows(R c00, R c11, R c01, R c02, R c12, R L[3][5])
{
  const R two = R(2);
  L[0][0] = -(c00 * c00); L[0][1] = -(c01 * c01); L[0][2] = -(two * c00 * c01);
  L[0][3] = -(two * c00 * c02); L[0][4] = -(two * c01 * c02);
  L[1][0] = L[0][1]; L[1][1] = -(c11 * c11); L[1][2] = -(two * c01 * c11);
  L[1][3] = -(two * c01 * c12); L[1][4] = -(two * c11 * c12);
  L[2][0] = -(c00 * c01); L[2][1] = -(c01 * c11); L[2][2] = -(c00 * c11 + c01 * c01);
  L[2][3] = -(c00 * c12 + c01 * c02); L[2][4] = -(c01 * c12 + c11 * c02);
}

/* Stress of one thickness point after the C33 sub-iterations:
   returns S^11, S^22, S^12 in sv[0..2]; status bit 1 on a vanishing CC3333.
   Every sub-iteration ends with the C33 update (ModElemC33); the stress is
   taken before the last one, so final_update = false skips that update
   (CC3333 and its check included) when only the stress is wanted and another
   kernel of the same call performs the check.  c33_out receives C33 after
   the last update.

   grad: C[i][k] = d sv_i / d g_k for the metric components g_k = 00, 11, 01,
   02, 12 (the sixth, g33 = n.n, is 1 for every state).  The stress depends on
   the metric only through c(0), the in-plane block of the first
   sub-iteration's inverse, c(1), the in-plane 2x2 inverse of all later ones,
   and the scalar C33, whose update of each sub-iteration depends on four
   numbers (c00, c11, c01, c22 = 1/C33).  So one gradient of that scalar per
   sub-iteration replaces a forward derivative along each of the five
   components: X, Y carry dC33 as a combination of dc(0) and dc(1) (XJ, YJ of
   the determinants in Je), and the metric enters once at the end through
   dc = -c dg c and d ln det = c:dg.  The damping factor of a bisected update
   is constant, as in the update itself.  About 0.3 of the arithmetic of five
   forward directions. */
template <class R, class Ref>
__host__ __device__ __forceinline__ void qp_stress(const R gm[5] /* 00 11 01 02 12 */, const Ref &r, R mu, R K,
                                                   int iters, R sv[3], int &status, R *c33_out = nullptr,
                                                   bool final_update = true, bool grad = false, R C[3][5] = nullptr)
{
  const R one = R(1), two = R(2), half = R(0.5), four = R(4);
  const R half_K = pow2(K, 0.5f), quarter_K = pow2(K, 0.25f), half_mu = pow2(mu, 0.5f);
  const R g00 = gm[0], g11 = gm[1], g01 = gm[2], g02 = gm[3], g12 = gm[4];
  /* ElemCGDefTens: C_inv in-plane = in-plane block of gm^-1 (g33 = n.n = 1), C33 = 1 */
  const R cof00 = mad(-g12, g12, g11);
  const R cof11 = mad(-g02, g02, g00);
  const R cof01 = mad(g02, g12, -g01);
  const R cofx = sop(g01, g12, -g11, g02);
  const R det = sop(g00, cof00, g01, cof01, g02, cofx);
  const R idet = one / det;
  R c00 = cof00 * idet, c11 = cof11 * idet, c01 = cof01 * idet;
  R c22 = one;
  R C33 = one;
  R X[3], Y[3], XJ = R(0), YJ = R(0);        /* grad: dC33 = X.dc(0) + XJ d ln det(0) + Y.dc(1) + YJ d ln det(1) */
  const R k00 = c00, k11 = c11, k01 = c01;   /* c(0) */
  const R den = sop(g00, g11, -g01, g01);
  /* 1 / (c00 c11 - c01^2), the determinant the in-plane inverse was divided
     by: det for c(0), the 2x2 determinant for c(1).  Je takes it from here,
     1 / det Ci = ipre C33, rather than from the rounded inverse: one division
     less a sub-iteration and about half the rounding error. */
  R ipre = det;
  /* the in-plane parts of the seven forms of c every sub-iteration needs; c
     changes in the plane once, after the first */
  constexpr int kForm[7] = {kRfB33, kRfQvv, kRfQww, kRfQee, kRfQvw, kRfQve, kRfQwe};
  R ip[7];
  auto in_plane = [&]() {
#pragma unroll
    for (int f = 0; f < 7; f++) ip[f] = sop(r(kForm[f]), c00, r(kForm[f] + 1), c11, r(kForm[f] + 2), c01);
  };
  in_plane();
  if (grad) {
#pragma unroll
    for (int m = 0; m < 3; m++) X[m] = Y[m] = R(0);
  }
  for (int it = 0; it < iters; it++) {
    const bool last = it == iters - 1;
    const R J2 = r(kRfRho) * ipre * C33;
    const R Je = dsqrt(J2);
    const R half_a = mad(half_K, J2 - Je, -half_mu);
    if (last) {
      R Bi[3];
#pragma unroll
      for (int i = 0; i < 3; i++) {
        const int o = kRfB00 + 4 * i;
        Acc<R> b(r(o), c00);
        b.add(r(o + 1), c11); b.add(r(o + 2), c01); b.add(r(o + 3), c22);
        Bi[i] = b.get();
        sv[i] = mad(half_a, Bi[i], r(kRfS00 + i));
      }
      if (grad) {
        /* dJe = Je/2 (d ln ipre + dC33/C33), d ln ipre = c:dg */
        const R sJ = (half * K) * (two * Je - one) * (half * Je);
        if (it > 0) {
          /* v = dC33/dg: the rows of dc and d ln det at c(0) (cofactor (1, 2)
             of the 3x3 inverse is g01 g02 - g00 g12), then at c(1) */
          R L[3][5], v[5];
          const R k02 = cofx * idet, k12 = (g01 * g02 - g00 * g12) * idet;
          const R ln0[5] = {k00, k11, two * k01, two * k02, two * k12};
          inverse_rows<R>(k00, k11, k01, k02, k12, L);
#pragma unroll
          for (int k = 0; k < 5; k++) v[k] = X[0] * L[0][k] + X[1] * L[1][k] + X[2] * L[2][k] + XJ * ln0[k];
          inverse_rows<R>(c00, c11, c01, R(0), R(0), L);
          const R ln1[3] = {c00, c11, two * c01};
#pragma unroll
          for (int k = 0; k < 3; k++) v[k] = v[k] + (Y[0] * L[0][k] + Y[1] * L[1][k] + Y[2] * L[2][k] + YJ * ln1[k]);
          const R hc = half_a * (c22 * c22);
#pragma unroll
          for (int i = 0; i < 3; i++) {
            const int o = kRfB00 + 4 * i;
            const R a = sJ * Bi[i], d00 = half_a * r(o), d11 = half_a * r(o + 1), d01 = half_a * r(o + 2);
            const R z = a * c22 - hc * r(o + 3);                 /* along C33 (dc22 = -c22^2 dC33) */
#pragma unroll
            for (int k = 0; k < 3; k++) C[i][k] = d00 * L[0][k] + d11 * L[1][k] + d01 * L[2][k] + a * ln1[k] + z * v[k];
            C[i][3] = z * v[3]; C[i][4] = z * v[4];
          }
        } else {
          R L[3][5];
          const R k02 = cofx * idet, k12 = (g01 * g02 - g00 * g12) * idet;
          const R ln0[5] = {k00, k11, two * k01, two * k02, two * k12};
          inverse_rows<R>(k00, k11, k01, k02, k12, L);
#pragma unroll
          for (int i = 0; i < 3; i++) {
            const int o = kRfB00 + 4 * i;
            const R a = sJ * Bi[i], d00 = half_a * r(o), d11 = half_a * r(o + 1), d01 = half_a * r(o + 2);
#pragma unroll
            for (int k = 0; k < 5; k++) C[i][k] = d00 * L[0][k] + d11 * L[1][k] + d01 * L[2][k] + a * ln0[k];
          }
        }
      }
      if (!final_update) break;
    }
    /* S^33 and CC3333 */
    const R B33 = mad(r(kRfB33 + 3), c22, ip[0]);
    const R S33 = mad(half_a, B33, r(kRfS33));
    const R qvv = mad(r(kRfQvv + 3), c22, ip[1]), qww = mad(r(kRfQww + 3), c22, ip[2]);
    const R qee = mad(r(kRfQee + 3), c22, ip[3]), qvw = mad(r(kRfQvw + 3), c22, ip[4]);
    const R qve = mad(r(kRfQve + 3), c22, ip[5]), qwe = mad(r(kRfQwe + 3), c22, ip[6]);
    /* 4 CC3333 = Qvv (2 (beta - alpha) Qvv + 4 beta Qwe) + Qwe (2 beta - alpha) Qwe - alpha (4 Qvw Qve + Qww Qee),
       with alpha = 2 half_a, beta = 2 b and the constants holding 2 Qvw and Qww / 2:
       CC3333 = b (Qvv + Qwe)^2 - half_a (Qvv^2 + Qwe^2 / 2 + Qvw Qve + Qww Qee) */
    const R b = half_K * sop(Je, Je, -half, Je);
    const R sum = qvv + qwe, sum2 = sum * sum;
    Acc<R> quad(qvv, qvv);
    quad.add(pow2(qwe, 0.5f), qwe); quad.add(qvw, qve); quad.add(qww, qee);
    const R Mq = quad.get();
    const R CC = sop(b, sum2, -half_a, Mq);
    /* ModElemC33 (active_strain.c:1654-1707) */
    if (!(dabs(CC) > R(1e-14))) { status |= 1; return; }
    const R iCC = one / CC;
    R dC = -(S33 * iCC);
    const R dC0 = dC;
    R damp = one;
    R Ct = C33 + dC;
    if (den * Ct <= R(0)) {
      R lo = R(0), hi = one;
      for (int bk = 0; bk < 16; bk++) {
        const R mid = half * (lo + hi);
        const R ct = C33 + mid * dC;
        if (den * ct > R(0)) lo = mid; else hi = mid;
      }
      dC = dC * lo;
      Ct = C33 + dC;
      damp = lo;
    }
    if (grad && !last) {
      /* d dC = damp (-(dS33 + dC0 dCC) / CC) through Je (coefficient wJ on
         d ln ipre + dC33/C33), B33 (wB) and the quadratic forms (p..) */
      const R e = -(damp * iCC);
      const R kj = K * (two * Je - one);
      const R wJ = e * (half * kj * (B33 - dC0 * Mq) + dC0 * sum2 * (quarter_K * (four * Je - one))) * (half * Je);
      const R wQ = e * dC0, wh = wQ * half_a, wb = two * wQ * b * sum;
      const R w[7] = {e * half_a, wb - two * wh * qvv, -(wh * qee), -(wh * qww), -(wh * qve), -(wh * qvw), wb - wh * qwe};
      R d[4];
#pragma unroll
      for (int m = 0; m < 4; m++) {
        d[m] = w[0] * r(kForm[0] + m);
#pragma unroll
        for (int f = 1; f < 7; f++) d[m] = d[m] + w[f] * r(kForm[f] + m);
      }
      if (it == 0) {
        X[0] = d[0]; X[1] = d[1]; X[2] = d[2]; XJ = wJ;
      } else {
        const R f = one + wJ * c22 - d[3] * (c22 * c22);
#pragma unroll
        for (int m = 0; m < 3; m++) { X[m] = f * X[m]; Y[m] = f * Y[m] + d[m]; }
        XJ = f * XJ; YJ = f * YJ + wJ;
      }
    }
    C33 = Ct;
    if (!last) {
      /* C_inv = INV([[gm00 gm01 0][gm01 gm11 0][0 0 C33]]): the in-plane block
         is the same in every later sub-iteration */
      if (it == 0) {
        const R id2 = one / den;
        c00 = g11 * id2; c11 = g00 * id2; c01 = -g01 * id2;
        ipre = den;
        in_plane();
      }
      c22 = one / C33;
    }
  }
  if (c33_out) *c33_out = C33;
}

/* Mid-surface geometry of the element from y = (a1, a2, Aaa, Abb, Aab). */
template <class T> struct ElemGeom {
  V3<T> a1, a2, Aaa, Abb, Aab, n, gc1, gc2, a31, a32;
};

template <class T>
__host__ __device__ __forceinline__ ElemGeom<T> elem_geom(const T y[15], const EPar<T> &p)
{
  const T one = T(1);
  ElemGeom<T> g;
  g.a1 = {y[0], y[1], y[2]}; g.a2 = {y[3], y[4], y[5]};
  g.Aaa = {y[6], y[7], y[8]}; g.Abb = {y[9], y[10], y[11]}; g.Aab = {y[12], y[13], y[14]};
  const V3<T> cr = cross(g.a1, g.a2);
  const T icn = drsqrt(dot(cr, cr));
  g.n = scl(icn, cr);
  g.gc1 = scl(icn, cross(g.a2, g.n));       /* a1.(a2 x n) = a2.(n x a1) = |a1 x a2| */
  g.gc2 = scl(icn, cross(g.n, g.a1));
  g.a31 = scl(icn, cross2(g.Aaa, g.a2, g.a1, g.Aab));
  g.a32 = scl(icn, cross2(g.Aab, g.a2, g.a1, g.Abb));
  if (p.tnormal) {   /* n_,alpha: drop the J_,alpha / J n part of the unnormalised derivative */
    g.a31 = mad(-dot(g.a31, g.n), g.n, g.a31);
    g.a32 = mad(-dot(g.a32, g.n), g.n, g.a32);
  }
  return g;
}

/* Metric (00 11 01 02 12; the sixth, n.n, is 1) of the thickness point theta3 (ElemUpdateG). */
template <class T>
__host__ __device__ __forceinline__ void qp_metric(const ElemGeom<T> &g, T th3, T gm[5])
{
  const V3<T> g1 = mad(th3, g.a31, g.a1), g2 = mad(th3, g.a32, g.a2);
  gm[0] = dot(g1, g1); gm[1] = dot(g2, g2); gm[2] = dot(g1, g2);
  gm[3] = dot(g1, g.n); gm[4] = dot(g2, g.n);
}

/* The 15 force components from the resultants (ElemUpdFint, Nᵀ applied by the caller). */
template <class R>
__host__ __device__ __forceinline__ void elem_out(const ElemGeom<R> &g, const R N[3], const R M[3], R f[15])
{
  const R twoM2 = pow2(M[2], 2.f);
  const V3<R> Q = lin3(M[0], g.Aaa, M[1], g.Abb, twoM2, g.Aab);
  const V3<R> f1 = lin3(N[0], g.a1, N[2], g.a2, -dot(g.gc1, Q), g.n);
  const V3<R> f2 = lin3(N[1], g.a2, N[2], g.a1, -dot(g.gc2, Q), g.n);
  f[0] = f1.x; f[1] = f1.y; f[2] = f1.z;
  f[3] = f2.x; f[4] = f2.y; f[5] = f2.z;
  f[6] = -(M[0] * g.n.x); f[7] = -(M[0] * g.n.y); f[8] = -(M[0] * g.n.z);
  f[9] = -(M[1] * g.n.x); f[10] = -(M[1] * g.n.y); f[11] = -(M[1] * g.n.z);
  f[12] = -(twoM2 * g.n.x); f[13] = -(twoM2 * g.n.y); f[14] = -(twoM2 * g.n.z);
}

/* The thickness-integrated resultants N = (N11, N22, N12) and M, scaled by
   pref0; ref is the element's column of constants.  With
   `grad`, out(q, w, th3, C) receives each thickness point's stress gradient
   (qp_stress), w the point's weight times pref0.  Points q0, q0 + dq, ... only. */
template <class R, class Grad>
__host__ __device__ __forceinline__ void elem_resultants(const ElemGeom<R> &g, const EPar<R> &p, const RefCol<R> &ref,
                                                         R N[3], R M[3], int &status, bool final_update,
                                                         bool grad, Grad out, int q0 = 0, int dq = 1)
{
  const int nq = p.nq;
  const R pref0 = ref(kRefPerQp * nq);
  for (int i = 0; i < 3; i++) N[i] = M[i] = R(0);
  for (int q = q0; q < nq; q += dq) {
    const R th3 = p.hhalf * p.theta[q];
    R gm[5], sv[3] = {R(0), R(0), R(0)};
    qp_metric(g, th3, gm);
    R C[3][5] = {};
    if constexpr (sizeof(R) == 4)
      qp_stress<R>(gm, RefRegs<R>(ref.at(kRefPerQp * q)), p.mu, p.K, p.iters, sv, status, nullptr, final_update, grad, C);
    else
      qp_stress<R>(gm, ref.at(kRefPerQp * q), p.mu, p.K, p.iters, sv, status, nullptr, final_update, grad, C);
    if (grad) out(q, pref0 * p.w[q], th3, C);
    const R wq = p.w[q], wt = p.w[q] * th3;
    for (int i = 0; i < 3; i++) { N[i] = mad(wq, sv[i], N[i]); M[i] = mad(wt, sv[i], M[i]); }
  }
  for (int i = 0; i < 3; i++) { N[i] = pref0 * N[i]; M[i] = pref0 * M[i]; }
}

/* f(y): the 15 force components of the element. */
template <class R>
__host__ __device__ __forceinline__ void elem_forces(const R y[15], const EPar<R> &p, const RefCol<R> &ref, R f[15],
                                                     int &status)
{
  const ElemGeom<R> g = elem_geom<R>(y, p);
  R N[3], M[3];
  elem_resultants<R>(g, p, ref, N, M, status, true, false, [](int, R, R, R(*)[5]) {});
  elem_out(g, N, M, f);
}

/* UpdateElementThickness (active_strain.c:2198-2224): h0 sqrt(C33) with C33
   the mean over the thickness points of C33 after the sub-iterations (1 when
   that mean is not positive). */
template <class R>
__host__ __device__ __forceinline__ R elem_thickness(const R y[15], const EPar<R> &p, const RefCol<R> &ref, R h0,
                                                     int &status)
{
  const ElemGeom<R> g = elem_geom<R>(y, p);
  const int nq = p.nq;
  R sum = R(0);
  for (int q = 0; q < nq; q++) {
    R gm[5], sv[3], c33 = R(1);
    qp_metric(g, p.hhalf * p.theta[q], gm);
    qp_stress<R>(gm, ref.at(kRefPerQp * q), p.mu, p.K, p.iters, sv, status, &c33);
    sum += c33;
  }
  const R C33 = nq > 0 ? sum / (R)nq : R(1);
  return h0 * (C33 > R(0) ? sqrt(C33) : R(1));
}

/* ---------------- element tangent D = df/dy ---------------- */
/* The stress of every thickness point depends on y only through eight
   scalars: the mid-surface metric a11, a22, a12, the curvature components
   b11 = n.Aaa, b22 = n.Abb, b12 = n.Aab and kappa1, kappa2, the normal parts
   of a3,alpha:
     a3,1 = kappa1 n - b11 gc1 - b12 gc2,  a3,2 = kappa2 n - b12 gc1 - b22 gc2,
     kappa1 = G^1_11 + G^2_12,  kappa2 = G^1_12 + G^2_22,  G^c_ab = gc_c . A_ab
   (kappa = 0 with the tangential thickness metric), so that
     g00 = a11 - 2 th b11 + th^2 h11 (g11, g01 alike),  g02 = th kappa1,
     g12 = th kappa2,  h_ab = kappa_a kappa_b + b_ac a^cd b_db,
   and the force is f.dy = N:da/2 - M:db, i.e. f1 = N11 a1 + N12 a2 - q1 n,
   f3 = -M11 n, ..., q_c = M:G^c.  Hence D needs the 6 x 8 derivative H of the
   resultants along the eight scalars, whose y-derivatives are short
   combinations of a1, a2, n, gc1, gc2 (dn = -gc_c (n.da_c),
   dgc_c = -gc_d (gc_c.da_d) + a^cd n (n.da_d)), and rank-one terms:
     D = sum_m phi_m (x) dR_m  +  terms with the resultants held fixed.
   tangent_coefs forms H and the combination coefficients once per element
   (one thread), tangent_block the 15 x 3 block of columns of one of
   a1, a2, Aaa, Abb, Aab (one lane each).  About 1,300 + 5 x 245 operations
   at three thickness points; the forward-mode form this replaced took 16
   lanes of 600 instructions per element. */
enum {   /* per resultant m = N11, N22, N12, M11, M22, 2 M12 (base kTcRow m) */
  kTcA1 = 0, kTcA2, kTcA12, kTcZ1, kTcZ2, kTcX11, kTcX12, kTcX21, kTcX22, kTcB11, kTcB22, kTcB12, kTcK1, kTcK2
};
constexpr int kTcRow = 14;
constexpr int kTcVec = 6 * kTcRow;       /* a1, a2, n, gc1, gc2 */
constexpr int kTcRes = kTcVec + 15;      /* N11 N22 N12 M11 M22 2M12 */
constexpr int kTcQ = kTcRes + 6;         /* q1 q2 */
constexpr int kTcGam = kTcQ + 2;         /* G^1_11 G^1_22 G^1_12, G^2_11 G^2_22 G^2_12 */
constexpr int kTcE = kTcGam + 6;         /* (M:b) times a^11, a^12, a^22 */
static_assert(kTcE + 3 == kTanCoefs, "tangent coefficient block");

/* Moments of the stress gradients over the thickness points:
   T[k][3 i + c] = sum w th^k C_i,c (c = 00, 11, 01), U[k][2 i + c] the same
   of the 02 and 12 columns for th^1 and th^2. */
template <class R> struct TanMoments {
  R T[4][9], U[2][6];
  __host__ __device__ __forceinline__ void clear()
  {
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
      for (int i = 0; i < 9; i++) T[k][i] = R(0);
#pragma unroll
    for (int k = 0; k < 2; k++)
#pragma unroll
      for (int i = 0; i < 6; i++) U[k][i] = R(0);
  }
  __host__ __device__ __forceinline__ void add(R w, R th, const R C[3][5])
  {
    const R w1 = w * th, w2 = w1 * th, w3 = w2 * th;
#pragma unroll
    for (int i = 0; i < 3; i++) {
#pragma unroll
      for (int c = 0; c < 3; c++) {
        T[0][3 * i + c] += w * C[i][c]; T[1][3 * i + c] += w1 * C[i][c];
        T[2][3 * i + c] += w2 * C[i][c]; T[3][3 * i + c] += w3 * C[i][c];
      }
#pragma unroll
      for (int c = 0; c < 2; c++) { U[0][2 * i + c] += w1 * C[i][3 + c]; U[1][2 * i + c] += w2 * C[i][3 + c]; }
    }
  }
};

/* What the tangent coefficients of every resultant share. */
template <class R> struct TanShape {
  R b11, b22, b12, G11, G22, G12;
  R s111, s122, s112, s211, s222, s212;    /* G^1_11 G^1_22 G^1_12, G^2_.. */
  R k1, k2;
  R m11, m21, m12, m22;                    /* b^c_a = a^cd b_da */
  int tnormal;

  __host__ __device__ __forceinline__ TanShape(const ElemGeom<R> &g, int tn) : tnormal(tn)
  {
    b11 = dot(g.n, g.Aaa); b22 = dot(g.n, g.Abb); b12 = dot(g.n, g.Aab);
    G11 = dot(g.gc1, g.gc1); G22 = dot(g.gc2, g.gc2); G12 = dot(g.gc1, g.gc2);
    s111 = dot(g.gc1, g.Aaa); s122 = dot(g.gc1, g.Abb); s112 = dot(g.gc1, g.Aab);
    s211 = dot(g.gc2, g.Aaa); s222 = dot(g.gc2, g.Abb); s212 = dot(g.gc2, g.Aab);
    k1 = tn ? R(0) : s111 + s212; k2 = tn ? R(0) : s112 + s222;
    m11 = G11 * b11 + G12 * b12; m21 = G12 * b11 + G22 * b12;
    m12 = G11 * b12 + G12 * b22; m22 = G12 * b12 + G22 * b22;
  }

  /* the coefficients of resultant m = 3 t + i: T0..T2 the moments t .. t + 2 of
     the i-th stress's 00, 11, 01 columns, U the moment t + 1 of 02, 12 */
  template <class Store>
  __host__ __device__ __forceinline__ void row(int m, const R T0[3], const R T1[3], const R T2[3], const R U[2], Store st) const
  {
    const R two = R(2);
    /* dh along (a11, a22, a12) and (b11, b22, b12), rows h11, h22, h12 */
    const R ha[3][3] = {{-(m11 * m11), -(m21 * m21), -(two * m11 * m21)},
                        {-(m12 * m12), -(m22 * m22), -(two * m12 * m22)},
                        {-(m11 * m12), -(m21 * m22), -(m11 * m22 + m21 * m12)}};
    const R hb[3][3] = {{two * m11, R(0), two * m21}, {R(0), two * m22, two * m12}, {m12, m21, m11 + m22}};
    const R sc = m == 5 ? two : R(1);
    R Ha[3], Hb[3];
    const R h0 = T2[0], h1 = T2[1], h2 = T2[2];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      Ha[c] = sc * (T0[c] + (h0 * ha[0][c] + h1 * ha[1][c] + h2 * ha[2][c]));
      Hb[c] = sc * ((h0 * hb[0][c] + h1 * hb[1][c] + h2 * hb[2][c]) - two * T1[c]);
    }
    const R Hk1 = tnormal ? R(0) : sc * (U[0] + two * k1 * h0 + k2 * h2);
    const R Hk2 = tnormal ? R(0) : sc * (U[1] + two * k2 * h1 + k1 * h2);
    const int o = kTcRow * m;
    st(o + kTcA1, two * Ha[0]); st(o + kTcA2, two * Ha[1]); st(o + kTcA12, Ha[2]);
    st(o + kTcZ1, (Hk1 * m11 + Hk2 * m12) - (Hb[0] * s111 + Hb[1] * s122 + Hb[2] * s112));
    st(o + kTcZ2, (Hk1 * m21 + Hk2 * m22) - (Hb[0] * s211 + Hb[1] * s222 + Hb[2] * s212));
    st(o + kTcX11, -(Hk1 * s111 + Hk2 * s112)); st(o + kTcX12, -(Hk1 * s112 + Hk2 * s122));
    st(o + kTcX21, -(Hk1 * s211 + Hk2 * s212)); st(o + kTcX22, -(Hk1 * s212 + Hk2 * s222));
    st(o + kTcB11, Hb[0]); st(o + kTcB22, Hb[1]); st(o + kTcB12, Hb[2]);
    st(o + kTcK1, Hk1); st(o + kTcK2, Hk2);
  }

  /* the rest: vectors, resultants and what is formed from them */
  template <class Store>
  __host__ __device__ __forceinline__ void rest(const ElemGeom<R> &g, const R N[3], const R M[3], Store st) const
  {
    const V3<R> v[5] = {g.a1, g.a2, g.n, g.gc1, g.gc2};
#pragma unroll
    for (int k = 0; k < 5; k++) { st(kTcVec + 3 * k, v[k].x); st(kTcVec + 3 * k + 1, v[k].y); st(kTcVec + 3 * k + 2, v[k].z); }
    const R M2 = R(2) * M[2];
    st(kTcRes, N[0]); st(kTcRes + 1, N[1]); st(kTcRes + 2, N[2]);
    st(kTcRes + 3, M[0]); st(kTcRes + 4, M[1]); st(kTcRes + 5, M2);
    st(kTcQ, M[0] * s111 + M[1] * s122 + M2 * s112); st(kTcQ + 1, M[0] * s211 + M[1] * s222 + M2 * s212);
    st(kTcGam, s111); st(kTcGam + 1, s122); st(kTcGam + 2, s112);
    st(kTcGam + 3, s211); st(kTcGam + 4, s222); st(kTcGam + 5, s212);
    const R mb = M[0] * b11 + M[1] * b22 + M2 * b12;
    st(kTcE, mb * G11); st(kTcE + 1, mb * G12); st(kTcE + 2, mb * G22);
  }
};

/* st(k, value) for every k < kTanCoefs */
template <class R, class Store>
__host__ __device__ __forceinline__ void tangent_coefs(const ElemGeom<R> &g, const R N[3], const R M[3],
                                                       const TanMoments<R> &mo, int tnormal, Store st)
{
  const TanShape<R> sh(g, tnormal);
#pragma unroll
  for (int m = 0; m < 6; m++) {
    const int i = m % 3, t = m / 3;                 /* N rows take th^0..2, M rows th^1..3 */
    sh.row(m, mo.T[t] + 3 * i, mo.T[t + 1] + 3 * i, mo.T[t + 2] + 3 * i, mo.U[t] + 2 * i, st);
  }
  sh.rest(g, N, M, st);
}

/* Columns 3 s .. 3 s + 2 of D (s = 0..4: a1, a2, Aaa, Abb, Aab) from the
   coefficients ld(k): D[row][j]. */
template <class R, class Load>
__host__ __device__ __forceinline__ void tangent_block(int s, Load ld, R D[15][3])
{
  auto vec = [&](int k) { return V3<R>{ld(kTcVec + 3 * k), ld(kTcVec + 3 * k + 1), ld(kTcVec + 3 * k + 2)}; };
  const V3<R> a1 = vec(0), a2 = vec(1), n = vec(2), g1 = vec(3), g2 = vec(4);
  const R zero = R(0);
  const bool t = s < 2;                              /* a tangent's columns */
  /* dR_m along the columns = c1 a1 + c2 a2 + c3 n + c4 gc1 + c5 gc2 */
  const int i1 = s == 0 ? kTcA1 : kTcA12, i2 = s == 0 ? kTcA12 : kTcA2;
  const int i3 = s == 0 ? kTcZ1 : s == 1 ? kTcZ2 : s == 2 ? kTcB11 : s == 3 ? kTcB22 : kTcB12;
  const int i4 = s == 0 ? kTcX11 : s == 1 ? kTcX21 : s == 2 ? kTcK1 : kTcK2;
  const int i5 = s == 0 ? kTcX12 : s == 1 ? kTcX22 : s == 3 ? kTcK2 : kTcK1;
  V3<R> dR[6];
#pragma unroll
  for (int m = 0; m < 6; m++) {
    const int o = kTcRow * m;
    const R c1 = t ? ld(o + i1) : zero, c2 = t ? ld(o + i2) : zero, c3 = ld(o + i3);
    const R c4 = s == 3 ? zero : ld(o + i4), c5 = s == 2 ? zero : ld(o + i5);
    dR[m] = scl(c1, a1) + scl(c2, a2) + scl(c3, n) + scl(c4, g1) + scl(c5, g2);
  }
  const R q1 = ld(kTcQ), q2 = ld(kTcQ + 1);
  /* dq_c = sum_m G^c_m dM_m, plus M:dG^c: -q_s gc_c + (M:b) a^cs n for a tangent, M_m gc_c for A_m */
  const R kg = s == 0 ? -q1 : s == 1 ? -q2 : ld(kTcRes + 1 + s);
  const R n1 = t ? ld(kTcE + s) : zero, n2 = t ? ld(kTcE + 1 + s) : zero;
  V3<R> dq1 = scl(kg, g1) + scl(n1, n), dq2 = scl(kg, g2) + scl(n2, n);
#pragma unroll
  for (int m = 0; m < 3; m++) {
    dq1 = dq1 + scl(ld(kTcGam + m), dR[3 + m]);
    dq2 = dq2 + scl(ld(kTcGam + 3 + m), dR[3 + m]);
  }
  const V3<R> gs = t ? (s == 0 ? g1 : g2) : V3<R>{zero, zero, zero};
  const R a1c[3] = {a1.x, a1.y, a1.z}, a2c[3] = {a2.x, a2.y, a2.z}, nc[3] = {n.x, n.y, n.z}, gc[3] = {gs.x, gs.y, gs.z};
  auto row = [&](const V3<R> &v, int j) { return j == 0 ? v.x : j == 1 ? v.y : v.z; };
  const R N0 = ld(kTcRes), N1 = ld(kTcRes + 1), N2 = ld(kTcRes + 2);
  const R M0 = ld(kTcRes + 3), M1 = ld(kTcRes + 4), M2 = ld(kTcRes + 5);
  const R e1 = s == 0 ? N0 : s == 1 ? N2 : zero, e2 = s == 0 ? N2 : s == 1 ? N1 : zero;
#pragma unroll
  for (int j = 0; j < 3; j++) {
    /* minus the coefficient of n_i, and of gc_s,i */
    const R nj = row(n, j);
    const R p1 = row(dq1, j), p2 = row(dq2, j), p3 = row(dR[3], j), p4 = row(dR[4], j), p5 = row(dR[5], j);
    const R w1 = q1 * nj, w2 = q2 * nj, w3 = M0 * nj, w4 = M1 * nj, w5 = M2 * nj;
    const R v0 = row(dR[0], j), v1 = row(dR[1], j), v2 = row(dR[2], j);
#pragma unroll
    for (int i = 0; i < 3; i++) {
      D[i][j] = a1c[i] * v0 + a2c[i] * v2 + gc[i] * w1 - nc[i] * p1 + (i == j ? e1 : zero);
      D[3 + i][j] = a2c[i] * v1 + a1c[i] * v2 + gc[i] * w2 - nc[i] * p2 + (i == j ? e2 : zero);
      D[6 + i][j] = gc[i] * w3 - nc[i] * p3;
      D[9 + i][j] = gc[i] * w4 - nc[i] * p4;
      D[12 + i][j] = gc[i] * w5 - nc[i] * p5;
    }
  }
}

/* ---------------- tangent contraction ---------------- */
/* The element stiffness is K_e = N^T D N with D = df/dy (15 x 15) and N the
   5 x nen basis table acting on each Cartesian component; one block row a at a
   time:
     w = (N[:,a] (x) I3)^T D          (3 x 15, w[15 i + k] = sum_r N[r][a] D[3r+i][k]),
     K_ab[i][j] = sum_s N[s][b] w[15 i + 3 s + j],
   plus, when a and b are corner slots of the triangle, the follower-pressure
   block: the cross-product matrix of sc v_b, v_b the corner's vector.
   This is the plain form, for the host tests alone; the row assemblies of
   kernels.cu take the same sums in their own number formats and layouts (the
   FP64 one's are tested on the host through fx.cuh).
   Both sums run over the five basis rows, so the operands are kept with that
   index innermost, padded to 8: the table as tabT[8 b + s] = N[s][b] and w as
   wT[8 (3 i + j) + s] = w[15 i + 3 s + j]. */
constexpr int kRowPad = 8;

/* five consecutive values from a 16-byte aligned address */
template <class R>
__host__ __device__ __forceinline__ void load5(const R *p, R v[5])
{
#ifdef __CUDA_ARCH__
  if constexpr (sizeof(R) == 4) {
    const float4 a = *reinterpret_cast<const float4 *>(p);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = p[4];
  } else {
    const double2 a = *reinterpret_cast<const double2 *>(p), b = *reinterpret_cast<const double2 *>(p + 2);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = p[4];
  }
#else
  for (int k = 0; k < 5; k++) v[k] = p[k];
#endif
}

/* Entry t < 45 of w for the row slot whose table column is tabT_a (= tabT +
   8 a); *pos receives its place in wT. */
template <class R>
__host__ __device__ __forceinline__ R row_wt_entry(const R *D, const R *tabT_a, int t, int *pos)
{
  const int i = t / 15, k = t - 15 * i, s = k / 3, j = k - 3 * s;
  R n[5];
  load5(tabT_a, n);
  R acc = R(0);
#pragma unroll
  for (int r = 0; r < 5; r++) acc = fma(n[r], D[(3 * r + i) * 15 + k], acc);
  *pos = kRowPad * (3 * i + j) + s;
  return acc;
}

/* acc + K_ab[i][j], q = 3 i + j, from wT_q = wT + 8 q and tabT_b = tabT + 8 b,
   as one chain of fused multiply-adds. */
template <class R>
__host__ __device__ __forceinline__ R row_block_accum(const R *wT_q, const R *tabT_b, R acc)
{
  R w[5], n[5];
  load5(wT_q, w);
  load5(tabT_b, n);
#pragma unroll
  for (int s = 0; s < 5; s++) acc = fma(n[s], w[s], acc);
  return acc;
}

/* Entry (i, j) of the follower-pressure block d c / d x_k = [s v]x (the cross
   product matrix of s v), for runtime i, j. */
template <class R>
__host__ __device__ __forceinline__ R skew_entry(int i, int j, const R v[3], R s)
{
  if (i == j) return R(0);
  const int m3 = 3 - i - j;
  const R vm = m3 == 0 ? v[0] : (m3 == 1 ? v[1] : v[2]);
  const R t = s * vm;
  return (j - i + 3) % 3 == 1 ? -t : t;
}

} /* namespace biofem */
#endif
