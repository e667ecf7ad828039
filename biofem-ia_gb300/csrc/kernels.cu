/*
 * sm_103a kernels of the element residual / tangent / assembly path.
 *
 *   k_positions      x (Vec layout) -> padded node positions; ghost nodes
 *                    x_g = x_nv2 + x_nv1 - x_nv3 (GlobalGhost, bending.c:1763-1814)
 *   k_ref_prep       one-time reference geometry per element (geom0 + the
 *                    reference half of ElemUpdateG and ElemActDefGrad)
 *   k_elem_residual  one thread, or three lanes, per element: geometry, stress,
 *                    element forces Fb (ElemUpdFint) and the follower-pressure
 *                    corner force (SurfaceNormalPressure, external.c:589-624)
 *                    (and, for the FP64 tangent, the stress gradients and the
 *                    coefficients k_elem_tangent combines)
 *   k_elem_tangent   five lanes per element, one per column block of
 *                    D = df/dy, combined from the element's coefficients
 *                    (element.cuh, tangent_block) and stored, with the
 *                    follower-pressure corner vectors, for the row assembly
 *   k_elem_tangent_f32  the FP32-bulk tangent, one thread per element
 *   k_elem_residual_ff  the FP32-bulk residual: k_elem_residual's element math
 *                    in float-float numbers on the FP32 pipe
 *   k_node_gather    one thread per node and component: Fint / Fext (and FDynamic's Fdyn)
 *                    summed over the node's element contributions in element
 *                    order (the order FInternalAct's VecSetValues loop adds
 *                    them), R = Fint - Fext + Fdyn, clamp rows R = x - X,
 *                    ghost rows 0 (main.c:844-1016)
 *   k_row_assemble_* one warp per row node: for every element holding the
 *                    node, K_e's block row N_a^T D N (and the pressure blocks)
 *                    added into the row's blocks in shared memory in a fixed
 *                    order, then the row written once; FP64 K in fixed point
 *                    on the integer pipe (fx.cuh)
 *   k_scale          R *= 1 / max(|Fext|_inf, 1) (main.c:1020-1026); the row
 *                    assembly applies the same factor to K as it writes it
 *   k_elem_thickness UpdateElementThickness (output); k_dyn_diag / k_dyn_update
 *                    the dynamic term's tangent diagonal and xAccVel
 *
 * Assembly is deterministic: every sum runs in a fixed order given by the
 * precomputed node-to-element lists, independent of the launch
 * configuration; nothing is accumulated with atomics.
 */
#include <cuda_runtime.h>

#include <algorithm>

#include "element.cuh"
#include "fx.cuh"

namespace biofem {

/* ---------------- helpers ---------------- */
__device__ __forceinline__ void load_node(const double *pos, int node, double &x, double &y, double &z)
{
  const double2 a = __ldg(reinterpret_cast<const double2 *>(pos) + 2 * (size_t)node);
  const double b = __ldg(pos + 4 * (size_t)node + 2);
  x = a.x; y = a.y; z = b;
}

__device__ __forceinline__ void set_status(int *status, int bits)
{
  if (bits) atomicOr(status, bits);
}

/* y = N x over the element patch (regular table or IN arrays of valence v). */
__device__ __forceinline__ void gather_y(const double *pos, const int *patch, int e, int nen, const double *tab,
                                         double y[15])
{
  for (int k = 0; k < 15; k++) y[k] = 0.0;
  const int4 *p4 = reinterpret_cast<const int4 *>(patch + 16 * (size_t)e);
  int nodes[16];
  const int4 q0 = __ldg(p4), q1 = __ldg(p4 + 1), q2 = __ldg(p4 + 2), q3 = __ldg(p4 + 3);
  nodes[0] = q0.x; nodes[1] = q0.y; nodes[2] = q0.z; nodes[3] = q0.w;
  nodes[4] = q1.x; nodes[5] = q1.y; nodes[6] = q1.z; nodes[7] = q1.w;
  nodes[8] = q2.x; nodes[9] = q2.y; nodes[10] = q2.z; nodes[11] = q2.w;
  nodes[12] = q3.x; nodes[13] = q3.y; nodes[14] = q3.z; nodes[15] = q3.w;
#pragma unroll 4
  for (int i = 0; i < nen; i++) {
    double x, yy, z;
    load_node(pos, nodes[i], x, yy, z);
#pragma unroll
    for (int r = 0; r < 5; r++) {
      const double c = tab[r * 16 + i];
      y[3 * r] += c * x; y[3 * r + 1] += c * yy; y[3 * r + 2] += c * z;
    }
  }
}

/* ---------------- positions / ghosts ---------------- */
__global__ void k_positions(int nv, int ng, const double *__restrict__ x, const int *__restrict__ ghost3,
                            double *__restrict__ pos, unsigned long long *__restrict__ fmax)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) *fmax = 0ull;          /* k_node_gather's maximum, of the same pass */
  double o[4] = {0.0, 0.0, 0.0, 0.0};
  if (i < nv) {
    o[0] = x[3 * (size_t)i]; o[1] = x[3 * (size_t)i + 1]; o[2] = x[3 * (size_t)i + 2];
  } else if (i < nv + ng) {
    const int g = i - nv;
    const int n1 = ghost3[3 * g], n2 = ghost3[3 * g + 1], n3 = ghost3[3 * g + 2];
    for (int d = 0; d < 3; d++) o[d] = x[3 * (size_t)n2 + d] + x[3 * (size_t)n1 + d] - x[3 * (size_t)n3 + d];
  } else {
    return;
  }
  double2 *dst = reinterpret_cast<double2 *>(pos) + 2 * (size_t)i;
  dst[0] = make_double2(o[0], o[1]);
  dst[1] = make_double2(o[2], o[3]);
}

/* ---------------- reference preparation ---------------- */
/* 3x3 inverse by cofactors (math.c:75-89 form). */
__device__ __forceinline__ void inv3(const double A[3][3], double B[3][3])
{
  const double det = A[0][0] * (A[2][2] * A[1][1] - A[2][1] * A[1][2]) - A[1][0] * (A[2][2] * A[0][1] - A[2][1] * A[0][2])
                   + A[2][0] * (A[1][2] * A[0][1] - A[1][1] * A[0][2]);
  const double c = 1.0 / det;
  B[0][0] = c * (A[2][2] * A[1][1] - A[2][1] * A[1][2]);
  B[0][1] = -c * (A[2][2] * A[0][1] - A[2][1] * A[0][2]);
  B[0][2] = c * (A[1][2] * A[0][1] - A[1][1] * A[0][2]);
  B[1][0] = -c * (A[2][2] * A[1][0] - A[2][0] * A[1][2]);
  B[1][1] = c * (A[2][2] * A[0][0] - A[2][0] * A[0][2]);
  B[1][2] = -c * (A[1][2] * A[0][0] - A[1][0] * A[0][2]);
  B[2][0] = c * (A[2][1] * A[1][0] - A[2][0] * A[1][1]);
  B[2][1] = -c * (A[2][1] * A[0][0] - A[2][0] * A[0][1]);
  B[2][2] = c * (A[1][1] * A[0][0] - A[1][0] * A[0][1]);
}

__device__ __forceinline__ double det3(const double A[3][3])
{
  return A[0][0] * (A[1][1] * A[2][2] - A[1][2] * A[2][1]) - A[0][1] * (A[1][0] * A[2][2] - A[1][2] * A[2][0])
       + A[0][2] * (A[1][0] * A[2][1] - A[1][1] * A[2][0]);
}

__global__ void k_ref_prep(DevMesh m, KParams p, const double *__restrict__ fib, const double *__restrict__ gscale,
                           double *__restrict__ eref)
{
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= p.ne) return;
  const int info = m.einfo[e];
  const int nen = info & 0xff, tabi = info >> 8;
  double y[15];
  gather_y(m.pos, m.patch, e, nen, m.ntab + tabi * 80, y);
  const V3<double> a1 = {y[0], y[1], y[2]}, a2 = {y[3], y[4], y[5]};
  const V3<double> Aaa = {y[6], y[7], y[8]}, Abb = {y[9], y[10], y[11]}, Aab = {y[12], y[13], y[14]};
  const V3<double> cr = cross(a1, a2);
  const double cn = sqrt(dot(cr, cr));
  const V3<double> n = {cr.x / cn, cr.y / cn, cr.z / cn};
  V3<double> a31 = cross(Aaa, a2) + cross(a1, Aab), a32 = cross(Aab, a2) + cross(a1, Abb);
  a31 = {a31.x / cn, a31.y / cn, a31.z / cn};
  a32 = {a32.x / cn, a32.y / cn, a32.z / cn};
  if (p.tnormal) {
    a31 = a31 - scl(dot(a31, n), n);
    a32 = a32 - scl(dot(a32, n), n);
  }
  /* Fa_cart = afac (I - gam f f^T): the fibre activation (-cart_fib_act 1)
     has afac = 1; the isotropic one (-cart_fib_act 0,
     active_strain.c:1238-1255), diag(a, a, 1/a^2) with a = 1 - gamma, is
     a (I - (1 - 1/a^3) e3 e3^T).  The scale afac divides the mu part of the
     stress by afac^2 and rho by afac^6 (det Fa_cart = afac^3 (1 - gam phi));
     Ci + A Ci H, CC3333 and the quadratic forms do not depend on it. */
  double afac = 1.0, gam;
  V3<double> f;
  if (!p.iso_act) {
    f = {fib[3 * (size_t)e], fib[3 * (size_t)e + 1], fib[3 * (size_t)e + 2]};
    gam = p.gamma * gscale[e];
  } else {
    afac = 1.0 - p.gamma * gscale[e];
    f = {0.0, 0.0, 1.0};
    gam = 1.0 - 1.0 / (afac * afac * afac);
  }
  const double ia2 = 1.0 / (afac * afac);
  const double phi = dot(f, f);
  const double gamp = gam / (1.0 - gam * phi);
  const double c1 = (2.0 * gamp + gamp * gamp * phi) * ia2;
  /* flat reference triangle area (AreaNormal, io.c:1646-1669) */
  double X[3][3];
  for (int k = 0; k < 3; k++) load_node(m.pos, m.etri[3 * (size_t)e + k], X[k][0], X[k][1], X[k][2]);
  const V3<double> d21 = {X[1][0] - X[0][0], X[1][1] - X[0][1], X[1][2] - X[0][2]};
  const V3<double> d31 = {X[2][0] - X[0][0], X[2][1] - X[0][1], X[2][2] - X[0][2]};
  const V3<double> ca = cross(d21, d31);
  const double dA0 = 0.5 * sqrt(ca.x * ca.x + ca.y * ca.y + ca.z * ca.z);
  const size_t ne = p.ne;
  for (int q = 0; q < p.nq; q++) {
    const double th3 = p.hhalf * p.theta[q];
    const V3<double> g[3] = {a1 + scl(th3, a31), a2 + scl(th3, a32), n};
    double G[3][3], Gi[3][3];
    for (int i = 0; i < 3; i++) for (int j = 0; j < 3; j++) G[i][j] = dot(g[i], g[j]);
    inv3(G, Gi);
    double t[3], s[3];
    for (int i = 0; i < 3; i++) t[i] = dot(g[i], f);
    for (int i = 0; i < 3; i++) s[i] = Gi[i][0] * t[0] + Gi[i][1] * t[1] + Gi[i][2] * t[2];
    const double omg = 1.0 - gam * phi;
    const double a3 = afac * afac * afac;
    const double rho = 1.0 / (det3(G) * omg * omg * (a3 * a3));
    /* v = Fa_inv.Cov G^-1 e3, w = Fa_inv.Cov G^-1 v, A^T x = G (Fa.Cont x) */
    double u[3] = {Gi[0][2], Gi[1][2], Gi[2][2]};
    double v[3], gv[3], w[3];
    const double tu = t[0] * u[0] + t[1] * u[1] + t[2] * u[2];
    for (int i = 0; i < 3; i++) v[i] = G[i][0] * u[0] + G[i][1] * u[1] + G[i][2] * u[2] + gamp * t[i] * tu;
    for (int i = 0; i < 3; i++) gv[i] = Gi[i][0] * v[0] + Gi[i][1] * v[1] + Gi[i][2] * v[2];
    const double tgv = t[0] * gv[0] + t[1] * gv[1] + t[2] * gv[2];
    for (int i = 0; i < 3; i++) w[i] = G[i][0] * gv[0] + G[i][1] * gv[1] + G[i][2] * gv[2] + gamp * t[i] * tgv;
    auto aT = [&](const double xin[3], double out[3]) {
      double fa[3];
      const double sx = s[0] * xin[0] + s[1] * xin[1] + s[2] * xin[2];
      for (int i = 0; i < 3; i++) fa[i] = Gi[i][0] * xin[0] + Gi[i][1] * xin[1] + Gi[i][2] * xin[2] - gam * s[i] * sx;
      for (int i = 0; i < 3; i++) out[i] = G[i][0] * fa[0] + G[i][1] * fa[1] + G[i][2] * fa[2];
    };
    double av[3], aw[3], ae[3];
    const double e3[3] = {0.0, 0.0, 1.0};
    aT(v, av); aT(w, aw); aT(e3, ae);
    /* the stress's forms in (c00, c11, c01, c22): S^ij = mu (G^ij + c1 s_i s_j)
       + alpha/2 (Ci + A Ci H)^ij with A = I - gam s t^T, H = I + gam' t s^T,
       and Q_xy = (A^T x)^T Ci (A^T y); 2 Q_vw and Q_ww / 2, as CC3333 takes them */
    double *o = eref + (size_t)kRefPerQp * q * ne + e;
    auto form = [&](int k, double f00, double f11, double f01, double f22) {
      o[(size_t)k * ne] = f00; o[(size_t)(k + 1) * ne] = f11; o[(size_t)(k + 2) * ne] = f01; o[(size_t)(k + 3) * ne] = f22;
    };
    auto quad = [&](int k, const double x[3], const double y[3], double sc = 1.0) {
      form(k, sc * (x[0] * y[0]), sc * (x[1] * y[1]), sc * (x[0] * y[1] + x[1] * y[0]), sc * (x[2] * y[2]));
    };
    const double gg = gam * gamp, dg = gamp - gam;
    const double t00 = t[0] * t[0], t11 = t[1] * t[1], t01 = 2.0 * t[0] * t[1], t22 = t[2] * t[2];
    const double g33 = gg * s[2] * s[2], g00 = gg * s[0] * s[0], g11 = gg * s[1] * s[1], g01 = gg * s[0] * s[1];
    o[(size_t)kRfS33 * ne] = p.mu * (Gi[2][2] * ia2 + c1 * s[2] * s[2]);
    o[(size_t)kRfS00 * ne] = p.mu * (Gi[0][0] * ia2 + c1 * s[0] * s[0]);
    o[(size_t)kRfS11 * ne] = p.mu * (Gi[1][1] * ia2 + c1 * s[1] * s[1]);
    o[(size_t)kRfS01 * ne] = p.mu * (0.5 * (Gi[0][1] + Gi[1][0]) * ia2 + c1 * s[0] * s[1]);
    form(kRfB33, -g33 * t00, -g33 * t11, -g33 * t01, 2.0 + dg * s[2] * t[2] - g33 * t22);
    form(kRfB00, 2.0 + dg * s[0] * t[0] - g00 * t00, -g00 * t11, dg * s[0] * t[1] - g00 * t01, -g00 * t22);
    form(kRfB11, -g11 * t00, 2.0 + dg * s[1] * t[1] - g11 * t11, dg * s[1] * t[0] - g11 * t01, -g11 * t22);
    form(kRfB01, gamp * s[1] * t[0] - g01 * t00, -gam * s[0] * t[1] - g01 * t11,
         2.0 + gamp * s[1] * t[1] - gam * s[0] * t[0] - g01 * t01, -g01 * t22);
    quad(kRfQvv, av, av); quad(kRfQww, aw, aw, 0.5); quad(kRfQee, ae, ae);
    quad(kRfQvw, av, aw, 2.0); quad(kRfQve, av, ae); quad(kRfQwe, aw, ae);
    o[(size_t)kRfRho * ne] = rho;
  }
  eref[(size_t)kRefPerQp * p.nq * ne + e] = 0.5 * (2.0 * p.hhalf) * dA0;   /* pref0 */
}

/* ---------------- residual element kernel ---------------- */
/* Pressure corner force of element e: each corner receives n P dA / 3 =
   P (x2-x1)x(x3-x1) / 6 (SurfaceNormalPressure, external.c:589-624); the dead
   load takes the same expression on the reference corners
   (SurfaceConstNormalPressure, Nf and dA0 of Init, external.c:699-730). */
__device__ __forceinline__ void elem_pressure_force(const DevMesh &m, const KParams &p, int e)
{
  const size_t ne = p.ne;
  double X[3][3];
  for (int k = 0; k < 3; k++) {
    const size_t c = (size_t)m.etri[3 * (size_t)e + k];
    if (p.pres_dead) { X[k][0] = m.X[3 * c]; X[k][1] = m.X[3 * c + 1]; X[k][2] = m.X[3 * c + 2]; }
    else load_node(m.pos, (int)c, X[k][0], X[k][1], X[k][2]);
  }
  const V3<double> d21 = {X[1][0] - X[0][0], X[1][1] - X[0][1], X[1][2] - X[0][2]};
  const V3<double> d31 = {X[2][0] - X[0][0], X[2][1] - X[0][1], X[2][2] - X[0][2]};
  const V3<double> ca = cross(d21, d31);
  const double n2 = dot(ca, ca);
  if (n2 > 1e-280 && n2 < 1e280) {   /* |ca| cancels; a square root and three divisions less */
    const double sc = p.pressure * (1.0 / 6.0);
    m.fp[e] = ca.x * sc; m.fp[ne + e] = ca.y * sc; m.fp[2 * ne + e] = ca.z * sc;
    return;
  }
  const double nrm = sqrt(n2);       /* a triangle without area gives NaN */
  const double dA = 0.5 * nrm;
  m.fp[e] = (ca.x / nrm) * p.pressure * dA / 3.;
  m.fp[ne + e] = (ca.y / nrm) * p.pressure * dA / 3.;
  m.fp[2 * ne + e] = (ca.z / nrm) * p.pressure * dA / 3.;
}

/* The pressure block vectors of one element (follower-pressure load
   stiffness): every corner carries P/6 (x2-x1)x(x3-x1), so d/dx1 = [b-a]x,
   d/dx2 = -[b]x, d/dx3 = [a]x with a = x2-x1, b = x3-x1, times psc = -P/6 (R
   subtracts the load); stored after D in the element's block for the row
   assembly. */
template <class R>
__device__ __forceinline__ void store_pressure_vectors(const R av[3], const R bv[3], R psc, R *dst)
{
#pragma unroll
  for (int d = 0; d < 3; d++) {
    dst[d] = psc * (bv[d] - av[d]);
    dst[3 + d] = -(psc * bv[d]);
    dst[6 + d] = psc * av[d];
  }
}

/* L = 1: one thread per element.  For the R + K call (tan) it also evaluates the
   stress gradients (about 280 FP64 operations a thickness point beside the
   370 of the stress itself), keeps them in cq between the thickness loop and
   the moments (its own column: 15 values a point would not fit in registers
   beside the stress), and stores the kTanCoefs tangent coefficients
   k_elem_tangent reads.  One kernel serves both calls, so that R is bit for
   bit the same: two instances would contract multiply-adds differently.

   L = 3: three lanes per element (ten elements a warp), for meshes that leave
   FP64 units idle (residual_lanes).  Lane s gathers Cartesian component s of
   y, takes thickness points s, s + 3, .., forms the tangent coefficients of
   the two resultants of stress s (N11 and M11, ..) from their moments alone, and
   scatters component s of the force; the geometry in between is formed by all
   three.  A chain of some 700 FP64 operations (1,200 with gradients) in place of
   1,760 (3,560), at 64 cycles each. */
template <int L> constexpr int kResElems = 32 / L;      /* elements a warp */
constexpr int kResBlock = 128;

/* lane s's component of the three lanes' doubles, in every lane */
__device__ __forceinline__ double lane3(double v, int base, int s) { return __shfl_sync(0xffffffffu, v, base + s); }

template <int L>
__global__ void __launch_bounds__(kResBlock) k_elem_residual(DevMesh m, KParams p, bool tan)
{
  static_assert(L == 1 || L == 3, "one thread, or one lane per Cartesian component");
  __shared__ double tabs[kNumTables * 80];
  for (int i = threadIdx.x; i < kNumTables * 80; i += blockDim.x) tabs[i] = m.ntab[i];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int e0 = L == 1 ? blockIdx.x * kResBlock + threadIdx.x
                        : (blockIdx.x * (kResBlock / 32) + (threadIdx.x >> 5)) * kResElems<L> + min(lane / L, kResElems<L> - 1);
  if (L == 1 ? e0 >= p.ne : __all_sync(0xffffffffu, e0 >= p.ne)) return;
  const int e = min(e0, p.ne - 1), s = lane % L, base = L * min(lane / L, kResElems<L> - 1);
  const bool live = e0 < p.ne && lane < L * kResElems<L>;     /* the others repeat an element */
  const int info = m.einfo[e];
  const int nen = info & 0xff, tabi = info >> 8;
  const double *tab = tabs + tabi * 80;
  double y[15];
  if constexpr (L == 1) {
    gather_y(m.pos, m.patch, e, nen, tab, y);
  } else {
    double ys[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    const int *pe = m.patch + 16 * (size_t)e;
#pragma unroll 4
    for (int i = 0; i < nen; i++) {
      const double x = __ldg(m.pos + 4 * (size_t)__ldg(pe + i) + s);
#pragma unroll
      for (int r = 0; r < 5; r++) ys[r] += tab[r * 16 + i] * x;
    }
#pragma unroll
    for (int r = 0; r < 5; r++)
#pragma unroll
      for (int d = 0; d < 3; d++) y[3 * r + d] = lane3(ys[r], base, d);
  }
  double f[15];
  int st = 0;
  const EPar<double> ep = epar<double>(p);
  const size_t ne = p.ne;
  const ElemGeom<double> g = elem_geom<double>(y, ep);
  double N[3], M[3];
  const double pref0 = m.eref[(size_t)kRefPerQp * ep.nq * ne + e];
  elem_resultants<double>(g, ep, RefCol<double>{m.eref + e, ne}, N, M, st, true, tan, [&](int q, double, double, double C[3][5]) {
    double *cq = m.cq + e;
    if (live)
      for (int i = 0; i < 3; i++)
        for (int k = 0; k < 5; k++) cq[(size_t)(15 * q + 5 * i + k) * ne] = C[i][k];
  }, s, L);
  if constexpr (L == 3) {
#pragma unroll
    for (int i = 0; i < 3; i++) {
      N[i] = lane3(N[i], base, 0) + lane3(N[i], base, 1) + lane3(N[i], base, 2);
      M[i] = lane3(M[i], base, 0) + lane3(M[i], base, 1) + lane3(M[i], base, 2);
    }
  }
  elem_out(g, N, M, f);
  set_status(m.status, st);
  /* Fb_a = sum_r N[r][a] f_r, stored slot-major: fb[(3a+d)*ne + e] */
  if constexpr (L == 1) {
    for (int a = 0; a < nen; a++) {
      double fx = 0.0, fy = 0.0, fz = 0.0;
#pragma unroll
      for (int r = 0; r < 5; r++) {
        const double c = tab[r * 16 + a];
        fx += c * f[3 * r]; fy += c * f[3 * r + 1]; fz += c * f[3 * r + 2];
      }
      m.fb[(3 * a) * ne + e] = fx;
      m.fb[(3 * a + 1) * ne + e] = fy;
      m.fb[(3 * a + 2) * ne + e] = fz;
    }
  } else {
    double fs[5];
#pragma unroll
    for (int r = 0; r < 5; r++) fs[r] = s == 0 ? f[3 * r] : s == 1 ? f[3 * r + 1] : f[3 * r + 2];
    for (int a = 0; a < nen; a++) {
      double v = 0.0;
#pragma unroll
      for (int r = 0; r < 5; r++) v += tab[r * 16 + a] * fs[r];
      if (live) m.fb[(3 * a + s) * ne + e] = v;
    }
  }
  if (live && s == 0 && p.pressure != 0.0) elem_pressure_force(m, p, e);
  if (!tan) return;
  double *tc = m.tcoef + e;
  if constexpr (L == 1) {
    TanMoments<double> mo;
    mo.clear();
    for (int q = 0; q < ep.nq; q++) {
      double C[3][5];
      for (int i = 0; i < 3; i++)
        for (int k = 0; k < 5; k++) C[i][k] = m.cq[(size_t)(15 * q + 5 * i + k) * ne + e];
      mo.add(pref0 * ep.w[q], ep.hhalf * ep.theta[q], C);
    }
    tangent_coefs<double>(g, N, M, mo, ep.tnormal, [&](int k, double v) { tc[(size_t)k * ne] = v; });
  } else {
    __syncwarp();                                  /* the other lanes' gradients */
    double T[4][3] = {}, U[2][2] = {};             /* TanMoments of stress s */
    for (int q = 0; q < ep.nq; q++) {
      const double th = ep.hhalf * ep.theta[q], w0 = pref0 * ep.w[q], w1 = w0 * th, w2 = w1 * th, w3 = w2 * th;
      const double *C = m.cq + (size_t)(15 * q + 5 * s) * ne + e;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const double v = C[(size_t)c * ne];
        T[0][c] += w0 * v; T[1][c] += w1 * v; T[2][c] += w2 * v; T[3][c] += w3 * v;
      }
#pragma unroll
      for (int c = 0; c < 2; c++) { const double v = C[(size_t)(3 + c) * ne]; U[0][c] += w1 * v; U[1][c] += w2 * v; }
    }
    const TanShape<double> sh(g, ep.tnormal);
    auto put = [&](int k, double v) { if (live) tc[(size_t)k * ne] = v; };
    sh.row(s, T[0], T[1], T[2], U[0], put);
    sh.row(3 + s, T[1], T[2], T[3], U[1], put);
    if (live && s == 0) sh.rest(g, N, M, put);
  }
  if (live && s == 0 && p.pressure != 0.0 && !p.pres_dead) {
    double X[3][3];
    for (int k = 0; k < 3; k++) load_node(m.pos, m.etri[3 * (size_t)e + k], X[k][0], X[k][1], X[k][2]);
    const double av[3] = {X[1][0] - X[0][0], X[1][1] - X[0][1], X[1][2] - X[0][2]};
    const double bv[3] = {X[2][0] - X[0][0], X[2][1] - X[0][1], X[2][2] - X[0][2]};
    store_pressure_vectors<double>(av, bv, -p.pressure / 6.0, m.De + (size_t)kDeStride * e + kDePres);
  }
}

/* ---------------- FP32-bulk residual (float-float) ---------------- */
/* The residual of the FP32-bulk form, on the FP32 pipe with float-float
   numbers (ff.cuh, about 48 significant bits): one thread per element, the
   element math of k_elem_residual.  Plain FP32 does not keep the residual's
   1e-6 budget on these meshes: rounding y = N x alone to FP32 moves R by
   ~1e-6 relative (C1, C2) and the FP32 stress by ~5e-6, so the residual takes
   float-float, whose error sits near 1e-13.  Node positions are taken
   relative to the element's first corner in FP64 before the split, the shift
   is put back through (sum_i N_r[i]) x_c; the element forces leave as
   doubles (hi + lo is exact in FP64) for the FP64 node sums.

   L = 3 shares an element among three lanes, as k_elem_residual does. */
__device__ __forceinline__ FF lane3(FF v, int base, int s)
{
  return FF(__shfl_sync(0xffffffffu, v.hi, base + s), __shfl_sync(0xffffffffu, v.lo, base + s));
}

template <int L>
__global__ void __launch_bounds__(kResBlock, 3) k_elem_residual_ff(DevMesh m, KParams p)
{
  __shared__ FF tabs[kNumTables * 85];   /* tables, then their row sums */
  const FF *ntab = static_cast<const FF *>(m.ntabFF);
  for (int i = threadIdx.x; i < kNumTables * 85; i += blockDim.x) tabs[i] = ntab[i];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int e0 = L == 1 ? blockIdx.x * kResBlock + threadIdx.x
                        : (blockIdx.x * (kResBlock / 32) + (threadIdx.x >> 5)) * kResElems<L> + min(lane / L, kResElems<L> - 1);
  if (L == 1 ? e0 >= p.ne : __all_sync(0xffffffffu, e0 >= p.ne)) return;
  const int e = min(e0, p.ne - 1), s = lane % L, base = L * min(lane / L, kResElems<L> - 1);
  const bool live = e0 < p.ne && lane < L * kResElems<L>;     /* the others repeat an element */
  const int info = m.einfo[e];
  const int nen = info & 0xff, tabi = info >> 8;
  const FF *tab = tabs + tabi * 80, *tsum = tabs + kNumTables * 80 + tabi * 5;
  const int *pe = m.patch + 16 * (size_t)e;
  FF y[15];
  if constexpr (L == 1) {
    double xc[3];
    load_node(m.pos, m.etri[3 * (size_t)e], xc[0], xc[1], xc[2]);
    FFAcc acc[15] = {
#define BIOFEM_Y0(r) FFAcc(tsum[r], ff_split(xc[0])), FFAcc(tsum[r], ff_split(xc[1])), FFAcc(tsum[r], ff_split(xc[2]))
        BIOFEM_Y0(0), BIOFEM_Y0(1), BIOFEM_Y0(2), BIOFEM_Y0(3), BIOFEM_Y0(4)
#undef BIOFEM_Y0
    };
    for (int i = 0; i < nen; i++) {
      double X, Y, Z;
      load_node(m.pos, __ldg(pe + i), X, Y, Z);
      const FF d[3] = {ff_split(X - xc[0]), ff_split(Y - xc[1]), ff_split(Z - xc[2])};
#pragma unroll
      for (int r = 0; r < 5; r++) {
        const FF c = tab[r * 16 + i];
#pragma unroll
        for (int k = 0; k < 3; k++) acc[3 * r + k].add(c, d[k]);
      }
    }
#pragma unroll
    for (int k = 0; k < 15; k++) y[k] = acc[k].get();
  } else {
    const double xc = __ldg(m.pos + 4 * (size_t)m.etri[3 * (size_t)e] + s);
    const FF c0 = ff_split(xc);
    FFAcc acc[5] = {FFAcc(tsum[0], c0), FFAcc(tsum[1], c0), FFAcc(tsum[2], c0), FFAcc(tsum[3], c0), FFAcc(tsum[4], c0)};
#pragma unroll 4
    for (int i = 0; i < nen; i++) {
      const FF d = ff_split(__ldg(m.pos + 4 * (size_t)__ldg(pe + i) + s) - xc);
#pragma unroll
      for (int r = 0; r < 5; r++) acc[r].add(tab[r * 16 + i], d);
    }
#pragma unroll
    for (int r = 0; r < 5; r++) {
      const FF v = acc[r].get();
#pragma unroll
      for (int d = 0; d < 3; d++) y[3 * r + d] = lane3(v, base, d);
    }
  }
  FF f[15];
  int st = 0;
  const EPar<FF> ep = epar<FF>(p);
  const RefCol<FF> ref{m.erefF + e, (size_t)p.ne, (size_t)p.ne * (kRefPerQp * p.nq + kRefPerElem)};
  const ElemGeom<FF> g = elem_geom<FF>(y, ep);
  FF N[3], M[3];
  elem_resultants<FF>(g, ep, ref, N, M, st, true, false, [](int, FF, FF, FF(*)[5]) {}, s, L);
  if constexpr (L == 3) {
#pragma unroll
    for (int i = 0; i < 3; i++) {
      N[i] = lane3(N[i], base, 0) + lane3(N[i], base, 1) + lane3(N[i], base, 2);
      M[i] = lane3(M[i], base, 0) + lane3(M[i], base, 1) + lane3(M[i], base, 2);
    }
  }
  elem_out(g, N, M, f);
  set_status(m.status, st);
  const size_t ne = p.ne;
  if constexpr (L == 1) {
    for (int a = 0; a < nen; a++) {
      const FF c0 = tab[a];
      FFAcc fx(c0, f[0]), fy(c0, f[1]), fz(c0, f[2]);
#pragma unroll
      for (int r = 1; r < 5; r++) {
        const FF c = tab[r * 16 + a];
        fx.add(c, f[3 * r]); fy.add(c, f[3 * r + 1]); fz.add(c, f[3 * r + 2]);
      }
      m.fb[(3 * a) * ne + e] = ff_to_double_bits(fx.get());
      m.fb[(3 * a + 1) * ne + e] = ff_to_double_bits(fy.get());
      m.fb[(3 * a + 2) * ne + e] = ff_to_double_bits(fz.get());
    }
  } else {
    FF fs[5];
#pragma unroll
    for (int r = 0; r < 5; r++) fs[r] = s == 0 ? f[3 * r] : s == 1 ? f[3 * r + 1] : f[3 * r + 2];
    for (int a = 0; a < nen; a++) {
      FFAcc v(tab[a], fs[0]);
#pragma unroll
      for (int r = 1; r < 5; r++) v.add(tab[r * 16 + a], fs[r]);
      if (live) m.fb[(3 * a + s) * ne + e] = ff_to_double_bits(v.get());
    }
  }
  if (live && s == 0 && p.pressure != 0.0) elem_pressure_force(m, p, e);
}

/* heads, then tails, of the float-float form of a */
__global__ void k_to_ff(const double *__restrict__ a, float *__restrict__ b, long long n)
{
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const FF f(a[t]);
  b[t] = f.hi;
  b[n + t] = f.lo;
}

/* ---------------- tangent element kernel ---------------- */
/* Five lanes per element (six elements a warp), lane s forming the 15 x 3
   block of columns of D along the s-th of a1, a2, Aaa, Abb, Aab from the
   element's coefficients (tangent_block).  FP64-pipe bound: 245 FP64
   instructions a lane, 0.27 ms on the 98,304-triangle sheet (with the
   residual kernel's 0.30 ms of gradients and coefficients: 0.57 ms; the
   16-lane forward-mode form took 1.99 ms).  D leaves in the row assembly's fixed-point form
   (fx.cuh): per Cartesian pair (i, j) the largest exponent over the element's
   25 entries, then every entry as two 32-bit words; an element with an
   infinity or NaN, or with a pair near underflow, keeps its doubles and is
   marked kFxRaw.  The pressure vectors' exponents go beside D's (fx_pack), so
   that a load larger than D does not take D's digits. */
constexpr int kTanElems = 6;         /* elements per warp */

/* place of entry (k = 5 r + s, q = 3 i + j) of D in an FP64 element block, see the
   row assembly.  FP32 blocks hold float4s of rows r = 0..3: (s, q) at 9 s + q;
   then, row 4, a float4 of s = 0..3 for each q (45 + q) and s = 4 (float 216 + q). */
__host__ __device__ __forceinline__ int fx_place(int k, int q) { return (k / 2) * 18 + 2 * q + k % 2; }

__global__ void __launch_bounds__(128) k_elem_tangent(DevMesh m, KParams p)
{
  const int lane = threadIdx.x & 31;
  const int g = lane < 5 * kTanElems ? lane / 5 : kTanElems - 1, s = lane % 5;
  const int e = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kTanElems + g;
  const bool live = lane < 5 * kTanElems && e < p.ne;
  const int ee = min(e, p.ne - 1);
  const size_t ne = p.ne;
  const double *tc = m.tcoef + ee;
  double D[15][3];
  tangent_block<double>(s, [&](int k) { return __ldg(tc + (size_t)k * ne); }, D);
  const bool pres_live = p.pressure != 0.0 && !p.pres_dead;
  const double *pv = m.De + (size_t)kDeStride * ee + kDePres + 3 * min(s, 2);
  /* exponent of each (i, j) over this lane's five rows, then of the pressure vectors' components (one corner
     read here), two to a register, then over the element's five lanes */
  unsigned eb[6] = {0u, 0u, 0u, 0u, 0u, 0u};
#pragma unroll
  for (int q = 0; q < 12; q++) {
    int h = 0;
    if (q < 9) {
#pragma unroll
      for (int r = 0; r < 5; r++) h = max(h, __double2hiint(D[3 * r + q / 3][q % 3]) & 0x7fffffff);
    } else if (pres_live && s < 3) {
      h = __double2hiint(pv[q - 9]) & 0x7fffffff;
    }
    h >>= 20;
    eb[q / 2] |= (unsigned)h << (q % 2 * 16);
  }
#pragma unroll
  for (int k = 1; k < 5; k++) {
    const int src = lane < 5 * kTanElems ? 5 * g + (s + k) % 5 : lane;
#pragma unroll
    for (int q = 0; q < 6; q++) eb[q] = __vmaxu2(eb[q], __shfl_sync(0xffffffffu, eb[q], src));
  }
  auto field = [&](int q) { return (int)(q % 2 ? eb[q / 2] >> 16 : eb[q / 2] & 0xffffu); };
  /* the pressure block's entry (i, j) is component 3 - i - j of the corner vectors */
  auto load = [&](int q) { return q % 4 ? field(12 - q / 3 - q % 3) : 0; };
  bool raw = false;
  int most = 0;
#pragma unroll
  for (int q = 0; q < 9; q++) {
    raw |= field(q) == kFxRaw || load(q) == kFxRaw ||
           (field(q) && (field(q) < kFxMinExp || load(q) > field(q) + kFxMaxExcess));
    most = max(most, field(q));
  }
  if (!live) return;
  if (s == 0) {
    unsigned *dst = m.dexp + kFxExps * (size_t)e;
#pragma unroll
    for (int q = 0; q < 9; q++) dst[q] = raw ? fx_pack(kFxRaw, 0, kFxRaw) : fx_pack(field(q), load(q), most);
  }
  double *De = m.De + (size_t)kDeStride * e;
#pragma unroll
  for (int r = 0; r < 5; r++)
#pragma unroll
    for (int q = 0; q < 9; q++) {
      const double d = D[3 * r + q / 3][q % 3];
      const Fx v = fx_split(fx_from_double(d, field(q)));
      const int2 w = raw ? make_int2(__double2loint(d), __double2hiint(d)) : make_int2(v.lo, v.hi);
      *reinterpret_cast<int2 *>(De + fx_place(5 * r + s, q)) = w;
    }
}

/* ---------------- FP32-bulk tangent ---------------- */
/* The element tangent in single precision, one thread per element: stress
   gradients, coefficients and the five column blocks in registers, each block
   leaving through shared memory as the row assembly's 16-byte pieces, nine
   neighbouring lanes an element.  Node positions
   are shifted to the element's first corner in FP64 and rounded to FP32, so
   the FP32 values carry the element-size digits; the shift is put back through
   (sum_i N_r[i]) * x_c, which is not zero for the truncated second-derivative
   rows (their rows sum to -1e-4 / -1e-4 / +2e-4).
   Bound by the loads of the constants and the stores of D (1.1 KB an element):
   0.18 -> 0.08 ms on the 98,304-triangle sheet; staging all of D in one go
   took 0.09, a thread storing its own 0.10. */
constexpr int kTanF32Block = 64;

__global__ void __launch_bounds__(kTanF32Block, 6) k_elem_tangent_f32(DevMesh m, KParams p)
{
  __shared__ float stage[kTanF32Block * 37];       /* rows r = 0..3 of one column block, [q][r], an odd stride */
  __shared__ float row4[kTanF32Block * 45];        /* row r = 4 of the blocks, [q][s], until all five are known */
  const int lane = threadIdx.x & 31, w0 = threadIdx.x & ~31;
  const int e0 = blockIdx.x * kTanF32Block + w0;   /* the warp's elements e0 .. e0 + 31 */
  if (e0 >= p.ne) return;
  const int nw = min(32, p.ne - e0);
  const int e = e0 + min(lane, nw - 1);            /* the last warp's spare lanes repeat its last element */
  const int info = m.einfo[e];
  const int nen = info & 0xff, tabi = info >> 8;
  const float *tab = m.ntabF + tabi * 80, *tsum = m.ntabF + kNumTables * 80 + tabi * 5;
  int corner[3];
  for (int k = 0; k < 3; k++) corner[k] = m.etri[3 * (size_t)e + k];
  double xc, yc, zc;
  load_node(m.pos, corner[0], xc, yc, zc);
  float y[15];
#pragma unroll
  for (int r = 0; r < 5; r++) {
    const float sr = __ldg(tsum + r);
    y[3 * r] = sr * (float)xc; y[3 * r + 1] = sr * (float)yc; y[3 * r + 2] = sr * (float)zc;
  }
  const int *pe = m.patch + 16 * (size_t)e;
#pragma unroll 4
  for (int i = 0; i < nen; i++) {
    double X, Y, Z;
    load_node(m.pos, __ldg(pe + i), X, Y, Z);
    const float ax = (float)(X - xc), ay = (float)(Y - yc), az = (float)(Z - zc);
#pragma unroll
    for (int r = 0; r < 5; r++) {
      const float c = __ldg(tab + r * 16 + i);
      y[3 * r] = fmaf(c, ax, y[3 * r]); y[3 * r + 1] = fmaf(c, ay, y[3 * r + 1]); y[3 * r + 2] = fmaf(c, az, y[3 * r + 2]);
    }
  }
  const EPar<float> ep = epar<float>(p);
  const ElemGeom<float> g = elem_geom<float>(y, ep);
  float N[3], M[3];
  int st = 0;
  TanMoments<float> mo;
  mo.clear();
  /* the stress only: the residual kernel of the same call checks the last CC3333 */
  elem_resultants<float>(g, ep, RefCol<float>{m.erefF + e, (size_t)p.ne}, N, M, st, false, true,
                         [&](int, float w, float th, float C[3][5]) { mo.add(w, th, C); });
  if (lane < nw) set_status(m.status, st);
  float tc[kTanCoefs];
  tangent_coefs<float>(g, N, M, mo, ep.tnormal, [&](int k, float v) { tc[k] = v; });
  float4 *out = reinterpret_cast<float4 *>(m.DeF + (size_t)kDeStride * e0);
  float *sd = stage + 37 * threadIdx.x, *r4 = row4 + 45 * threadIdx.x;
#pragma unroll
  for (int s = 0; s < 5; s++) {
    float D[15][3];
    tangent_block<float>(s, [&](int k) { return tc[k]; }, D);
#pragma unroll
    for (int q = 0; q < 9; q++) {
#pragma unroll
      for (int r = 0; r < 4; r++) sd[4 * q + r] = D[3 * r + q / 3][q % 3];
      r4[5 * q + s] = D[12 + q / 3][q % 3];
    }
    __syncwarp();
    for (int t = lane; t < 9 * nw; t += 32) {
      const int g = t / 9, q = t - 9 * g;
      const float *v = stage + 37 * (w0 + g) + 4 * q;
      out[(kDeStride / 4) * g + 9 * s + q] = make_float4(v[0], v[1], v[2], v[3]);
    }
    __syncwarp();
  }
  for (int t = lane; t < 9 * nw; t += 32) {
    const int g = t / 9, q = t - 9 * g;
    const float *v = row4 + 45 * (w0 + g) + 5 * q;
    out[(kDeStride / 4) * g + 45 + q] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float *>(out + (kDeStride / 4) * g)[216 + q] = v[4];
  }
  if (p.pres6f != 0.f && !p.pres_dead && lane < nw) {
    double X[3][3];
    for (int k = 0; k < 3; k++) load_node(m.pos, corner[k], X[k][0], X[k][1], X[k][2]);
    const float av[3] = {(float)(X[1][0] - xc), (float)(X[1][1] - yc), (float)(X[1][2] - zc)};
    const float bv[3] = {(float)(X[2][0] - xc), (float)(X[2][1] - yc), (float)(X[2][2] - zc)};
    store_pressure_vectors<float>(av, bv, -p.pres6f, m.DeF + (size_t)kDeStride * e + kDePres);
  }
}

/* ---------------- node gather (residual assembly) ---------------- */
__device__ __forceinline__ unsigned long long abs_bits(double v)
{
  return (unsigned long long)__double_as_longlong(fabs(v));
}

/* v[idx(c)] over c in [c0, c1), in order; eight loads in flight at a time (one
   after another, the 24 dependent pairs of loads of an inner node were the
   kernel's time: 27 us on the 98,304-triangle sheet, 17 on the smallest ones) */
template <class Index>
__device__ __forceinline__ double ordered_sum(const double *__restrict__ v, int c0, int c1, Index idx)
{
  double s = 0.0;
  for (; c0 < c1; c0 += 8) {
    double x[8];
#pragma unroll
    for (int u = 0; u < 8; u++) x[u] = c0 + u < c1 ? __ldg(v + idx(c0 + u)) : 0.0;
#pragma unroll
    for (int u = 0; u < 8; u++)
      if (c0 + u < c1) s += x[u];
  }
  return s;
}

/* one thread per node and Cartesian component d = blockIdx.y */
__global__ void __launch_bounds__(128) k_node_gather(DevMesh m, KParams p, const double *__restrict__ x,
                                                     double *__restrict__ R, double *__restrict__ parts)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x, d = blockIdx.y;
  unsigned long long lmax = 0ull;
  if (i < p.nt) {
    const size_t ne = p.ne, o = 3 * (size_t)i + d;
    /* ridx: 3*slot*ne + e */
    const double fi = ordered_sum(m.fb + d * ne, m.rptr[i], m.rptr[i + 1], [&](int c) { return (size_t)__ldg(m.ridx + c); });
    const double fe = p.pressure != 0.0 ? ordered_sum(m.fp + d * ne, m.pptr[i], m.pptr[i + 1],
                                                      [&](int c) { return (size_t)__ldg(m.pidx + c); })
                                        : 0.0;
    const int kind = m.rowkind[i];
    /* FDynamic (main.c:1178-1270, the path of an active-strain run):
       triangle-order sum of the node's inertial (and damping) force over the
       real triangles with this corner */
    double fd = 0.0;
    if (p.dyn && (kind == 0 || (parts && i < p.nv))) {
      for (int c = m.dptr[i]; c < m.dptr[i + 1]; c++) {
        const double M = p.dyn_rhoh0 * m.dA0[m.didx[c]] / 3;
        const double C = p.dyn_damp ? p.dyn_dampf * M : 0.0;
        double f;
        if (!p.dyn_central) {
          const double facc = M * (p.dyn_M1 * m.xn[o] + p.dyn_M2 * m.xd[o] + p.dyn_M3 * m.xdd[o]);
          const double fvel = C * (p.dyn_C1 * m.xn[o] + p.dyn_C2 * m.xd[o] + p.dyn_C3 * m.xdd[o]);
          f = M * p.dyn_M1 * x[o] + C * p.dyn_C1 * x[o] - facc - fvel;
        } else {
          f = M * (x[o] - 2 * m.xn[o] + m.xnm1[o]) / (p.dyn_dt * p.dyn_dt) + C * (x[o] - m.xn[o]) / p.dyn_dt;
        }
        fd += f;
      }
    }
    double r;
    if (kind == 2) r = 0.0;
    else if (kind == 1) r = x[o] - m.X[o];
    else if (p.dyn) r = (-1.0 * fe + fi) + 1. * fd;
    else r = -1.0 * fe + fi;
    R[o] = r;
    if (parts) {   /* unscaled Fint, Fext, Fdyn of the real nodes (ghost entries 0) */
      const size_t n3 = 3 * (size_t)p.nt;
      const bool real = i < p.nv;
      parts[o] = real ? fi : 0.0;
      parts[n3 + o] = real ? fe : 0.0;
      parts[2 * n3 + o] = real ? fd : 0.0;
    }
    lmax = abs_bits(fe);
  }
  /* warp max then one atomic per warp */
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long v = __shfl_down_sync(0xffffffffu, lmax, o);
    lmax = v > lmax ? v : lmax;
  }
  if ((threadIdx.x & 31) == 0 && lmax) atomicMax(m.fmax, lmax);
}

/* ---------------- row assembly (tangent) ---------------- */
/* One warp per row node i.  For every element e whose patch holds i at slot a
   (the row's contribution list, element order) and every slot b of that
   patch, K_ib += (N[:,a] (x) I3)^T D_e (N[:,b] (x) I3), with D_e = df/dy the
   element kernel stored, plus the follower-pressure block when a and b are
   corner slots; a ghost slot b adds to the blocks of its parents with signs
   +, +, - (x_g = x_nv2 + x_nv1 - x_nv3).  Clamped and ghost rows are identity
   rows.  K is scaled by 1/max(|Fext|_inf, 1) as it is written
   (main.c:1020-1026; k_node_gather, launched before, found the max); with
   colmajor each 3x3 block is stored column by column.

   Three contributions at a time, lane (c, q) = (contribution, entry q = 3 i + j
   of the 3x3 blocks), 27 lanes: the lane forms its five values
   w_s = sum_r N[r][a] D_rs[q] (D is stored so that the nine lanes of a
   contribution read neighbouring 16-byte pieces: two values (5 r + s, 5 r + s
   + 1) of an entry in FP64, four in FP32), then for every slot b its
   entry sum_s N[s][b] w_s, and adds it to block target(b) of the
   contribution's own copy of the row in shared memory (three copies: two
   contributions may share a block; their sum is taken at the write-out).  Block
   t's three copies lie in 32 consecutive words, entry (c, q) at 32 t + lane, so
   every access is free of bank conflicts whatever the targets.
   Nothing is exchanged between lanes, and on a regular patch N[s][b] is a
   constant-bank operand of the multiply (the kernel parameter `reg`), its
   eight zeros left out: shared memory sees one read and one write an entry.  Forms that shared w through
   shared memory were bound by it (FP64: 0.75 ms, FP32: 0.34 ms on the
   98,304-triangle sheet).  The order of every sum is fixed, so K is
   deterministic. */
constexpr int kRowCopies = 3;
constexpr int kRowWords = 32;        /* words of one block: 3 x 9 entries and padding */
/* N[s][b] = 0 on the regular patch (both kinds of tables; regular_tables checks it) */
__host__ __device__ constexpr bool row_reg_zero(int s, int b)
{
  return (s == 0 && (b == 2 || b == 7)) || (s == 1 && (b == 4 || b == 6)) || (s == 2 && (b == 8 || b == 11)) ||
         (s == 3 && (b == 5 || b == 9));
}

__device__ __forceinline__ int row_find(const int *cols, int nb, int node)
{
  int lo = 0, hi = nb - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (cols[mid] < node) lo = mid + 1; else hi = mid;
  }
  return lo;
}

/* FP64 row assembly in fixed point (fx.cuh); the follower-pressure vectors
   are converted to the row's units and added with it.

   Why integers: the FP64 form of this sum ran at 93 % of the FP64 pipe
   (1.94 ms on the 98,304-triangle sheet, q = 3).  Now 0.49 ms,
   bound by the integer multiplies (IMAD.WIDE, four cycles a warp).  Fetching
   the next contributions' D early, as the FP32 form does, needs 126 registers
   and halves the warps: 0.58 ms.

   A sum of integers has one unit, 2^-57.6 of the row's largest element of the
   Cartesian pair, so a far smaller element would keep fewer bits than a
   double.  A row takes integers only while none lies too far below (fx_pack);
   the others (elements of very different size or stiffness side by side, a load
   far above D), and rows with infinities, NaN or magnitudes near the ends of
   the exponent range, are summed in double (row_assemble_wide). */
struct FxRowBuf {
  long long *acc;     /* kRowWords maxblk */
  int *rec;           /* kRowCopies records */
  double *sc;         /* 9 units of K */
  int *eb;            /* 9 exponents */
};
constexpr int kFxTab = 6;            /* table column: 5 values and fx_column_sum, 48 bytes */

__host__ __device__ __forceinline__ size_t fx_row_bytes(int maxblk)
{
  return (size_t)kRowWords * maxblk * 8 + kRowCopies * kRowRec * 4 + 80 + 48;
}

__device__ __forceinline__ FxRowBuf fx_row_buf(unsigned char *q, int maxblk)
{
  FxRowBuf b;
  b.acc = reinterpret_cast<long long *>(q);
  q += (size_t)kRowWords * maxblk * 8;
  b.rec = reinterpret_cast<int *>(q);
  q += kRowCopies * kRowRec * 4;
  b.sc = reinterpret_cast<double *>(q);
  q += 80;
  b.eb = reinterpret_cast<int *>(q);
  return b;
}

/* fx_entry of the regular table's column B, whose values are small integers over a common denominator */
template <int B>
__device__ __forceinline__ long long fx_entry_reg(const FxRegular &reg, const Fx w[5])
{
  FxIntSum<15> sum;
#pragma unroll
  for (int s = 0; s < 5; s++)
    if (!row_reg_zero(s, B)) sum.add(reg.n[B][s], w[s]);
  return sum.value();
}

/* The row's sum in double over the same lanes and copies, in units of
   1 / reg.wide: an element's sums stay integers in its own units and are added
   as doubles (fx_wide), so that elements of any size keep their digits; one
   that holds doubles, or is near overflow, takes FP64 throughout. */
__device__ __noinline__ void row_assemble_wide(const DevMesh &m, const FxRegular &reg, int c0, int c1, bool pres_live,
                                               double *racc, int nb, int lane)
{
  double *acc = racc + lane;
  for (int t = 0; t < nb; t++) acc[kRowWords * t] = 0.0;
  const int pc = lane / 9, q = lane - 9 * pc;
  for (int cb = c0; cb < c1; cb += kRowCopies) {
    const bool on = pc < min(kRowCopies, c1 - cb);
    const int *rc = m.rrec + (size_t)kRowRec * (on ? cb + pc : cb);
    const int e = rc[0] & ((1 << 27) - 1), a = rc[0] >> 27, info = rc[1];
    const double *De = m.De + (size_t)kDeStride * e;
    if (on) {
      const int nen = info & 0xff, eb = fx_d_exp(m.dexp[kFxExps * (size_t)e + q]);
      const bool f64 = eb > kFxMaxWide;
      const int2 *tab = reinterpret_cast<const int2 *>(m.ntabFx) + (info >> 8) * 16 * kFxTab;
      const double *tabd = m.ntab + (info >> 8) * 80;
      Fx w[5];
      double wd[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
      if (!f64) {
        FxSum<62> sum[5];
#pragma unroll
        for (int k = 0; k < 25; k++) {
          const int2 n = __ldg(tab + a * kFxTab + k / 5), d = __ldg(reinterpret_cast<const int2 *>(De + fx_place(k, q)));
          sum[k % 5].add(Fx{n.x, n.y}, Fx{d.x, d.y});
        }
#pragma unroll
        for (int s = 0; s < 5; s++) w[s] = fx_split(sum[s].value());
      } else {
        for (int r = 0; r < 5; r++)
#pragma unroll
          for (int s = 0; s < 5; s++) {
            const double d = De[fx_place(5 * r + s, q)];
            wd[s] = fma(__ldg(tabd + 16 * r + a), eb == kFxRaw ? d : fx_to_double(Fx{__double2loint(d), __double2hiint(d)}, eb), wd[s]);
          }
#pragma unroll
        for (int s = 0; s < 5; s++) wd[s] *= reg.wide;
      }
      for (int b = 0; b < nen; b++) {
        const unsigned sl = (unsigned)rc[4 + b];
        double v = 0.0;
        if (!f64) {
          Fx n[5];
#pragma unroll
          for (int s = 0; s < 5; s++) {
            const int2 x = __ldg(tab + b * kFxTab + s);
            n[s] = Fx{x.x, x.y};
          }
          v = fx_wide(fx_entry(n, w), eb);
        } else {
#pragma unroll
          for (int s = 0; s < 5; s++) v = fma(__ldg(tabd + 16 * s + b), wd[s], v);
        }
        acc[kRowWords * (int)(sl & 1023u)] += v;
        if ((sl & kRowSlotGhost) && !(sl & kRowSlotDup)) {   /* a repeated real node has one target */
          acc[kRowWords * (int)((sl >> 10) & 1023u)] += v;
          acc[kRowWords * (int)((sl >> 20) & 1023u)] -= v;
        }
      }
    }
    if (!pres_live) continue;
    __syncwarp();                                    /* the contributions' own adds are done */
    const int cs = rc[2], s0 = cs & 31, s1 = (cs >> 5) & 31, s2 = (cs >> 10) & 31;
    if (on && (a == s0 || a == s1 || a == s2)) {     /* lanes as in the integer form below */
      const int k = q / 3, d = q - 3 * k;
      const unsigned sl = (unsigned)rc[4 + (k == 0 ? s0 : k == 1 ? s1 : s2)];
      const double v = De[kDePres + q] * reg.wide;
      double *dst = acc - q + kRowWords * (int)(sl & 1023u);
      dst[d == 0 ? 5 : d == 1 ? 6 : 1] -= v;
      dst[d == 0 ? 7 : d == 1 ? 2 : 3] += v;
    }
    __syncwarp();
  }
}

__global__ void __launch_bounds__(256, 3) k_row_assemble_fx(DevMesh m, KParams p, FxRegular reg, double *__restrict__ K,
                                                            int maxblk, int colmajor)
{
  extern __shared__ __align__(16) unsigned char row_smem[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int i = blockIdx.x * (blockDim.x >> 5) + wid;
  if (i >= p.nt) return;
  const FxRowBuf B = fx_row_buf(row_smem + (size_t)wid * fx_row_bytes(maxblk), maxblk);
  const int k0 = m.rowptr[i], nb = m.rowptr[i + 1] - k0;
  double *Kr = K + 9 * (size_t)k0;
  if (m.rowkind[i] != 0) {   /* clamped (R = x - X) and ghost (R = 0) rows: identity */
    for (int t = lane; t < 9 * nb; t += 32) {
      const int q = t % 9;
      Kr[t] = (m.colind[k0 + t / 9] == i && (q == 0 || q == 4 || q == 8)) ? 1.0 : 0.0;
    }
    return;
  }
  const int c0 = m.rptr[i], c1 = m.rptr[i + 1];
  const int4 *rrec4 = reinterpret_cast<const int4 *>(m.rrec);
  const bool pres_live = p.pressure != 0.0 && !p.pres_dead;
  const int pc = lane / 9, q = lane - 9 * pc;       /* contribution and entry; lanes 27..31 idle */
  int4 nrec = make_int4(0, 0, 0, 0);
  if (lane < (kRowRec / 4) * min(kRowCopies, c1 - c0)) nrec = __ldg(rrec4 + (size_t)(kRowRec / 4) * c0 + lane);
  /* the row's exponent of entry q over all contributions, and the largest that each of them allows */
  int eb = 0, most = kFxRaw;
  for (int c = c0 + pc; c < c1; c += kRowCopies)
    if (pc < kRowCopies) {
      const unsigned x = m.dexp[kFxExps * (size_t)(__ldg(m.rrec + (size_t)kRowRec * c) & ((1 << 27) - 1)) + q];
      eb = max(eb, fx_row_exp(x));
      most = min(most, fx_most_exp(x));
    }
  {
    const int l1 = lane >= 27 ? lane : (lane + 9) % 27, l2 = lane >= 27 ? lane : (lane + 18) % 27;
    const int x1 = __shfl_sync(0xffffffffu, eb, l1), x2 = __shfl_sync(0xffffffffu, eb, l2);
    eb = max(eb, max(x1, x2));
  }
  const int grow = m.rgrow[i];
  const bool wide = __any_sync(0xffffffffu, (eb > 0 && eb < kFxMinExp) || eb > kFxMaxExp || eb + grow > most);
  if (wide) {
    row_assemble_wide(m, reg, c0, c1, pres_live, reinterpret_cast<double *>(B.acc), nb, lane);
  } else {
    eb += grow;
    if (lane < 9) { B.sc[lane] = ldexp(reg.unit, eb - 1022); B.eb[lane] = eb; }
    long long *acc = B.acc + lane;
    for (int t = 0; t < nb; t++) acc[kRowWords * t] = 0;
    for (int cb = c0; cb < c1; cb += kRowCopies) {
      const int np = min(kRowCopies, c1 - cb);
      if (lane < (kRowRec / 4) * np) reinterpret_cast<int4 *>(B.rec)[lane] = nrec;
      if (lane < (kRowRec / 4) * min(kRowCopies, c1 - cb - kRowCopies))
        nrec = __ldg(rrec4 + (size_t)(kRowRec / 4) * (cb + kRowCopies) + lane);
      __syncwarp();   /* also orders the set-up */
      const bool on = pc < np;
      const int *rc = B.rec + kRowRec * (on ? pc : 0);
      const int e = rc[0] & ((1 << 27) - 1), a = rc[0] >> 27, info = rc[1];
      const int2 *tab = reinterpret_cast<const int2 *>(m.ntabFx) + (info >> 8) * 16 * kFxTab;
      Fx w[5];
      if (on) {
        const int4 *D = reinterpret_cast<const int4 *>(m.De + (size_t)kDeStride * e) + q;
        const int sh = eb - fx_d_exp(m.dexp[kFxExps * (size_t)e + q]);
        if ((info >> 8) == 0) {
          const int *nr = reg.n[a];
          const int n[5] = {nr[0], nr[1], nr[2], nr[3], nr[4]};
          FxIntSum<14> sum[5];
#pragma unroll
          for (int g = 0; g < 13; g++) {
            const int4 d = __ldg(D + 9 * g);
            sum[(2 * g) % 5].add(n[(2 * g) / 5], Fx{d.x, d.y});
            if (2 * g + 1 < 25) sum[(2 * g + 1) % 5].add(n[(2 * g + 1) / 5], Fx{d.z, d.w});
          }
#pragma unroll
          for (int s = 0; s < 5; s++) w[s] = fx_split(fx_shift(sum[s].value(), sh));
        } else {
          Fx n[5];
#pragma unroll
          for (int r = 0; r < 5; r++) {
            const int2 x = __ldg(tab + a * kFxTab + r);
            n[r] = Fx{x.x, x.y};
          }
          FxSum<62> sum[5];
#pragma unroll
          for (int g = 0; g < 13; g++) {
            const int4 d = __ldg(D + 9 * g);
            sum[(2 * g) % 5].add(n[(2 * g) / 5], Fx{d.x, d.y});
            if (2 * g + 1 < 25) sum[(2 * g + 1) % 5].add(n[(2 * g + 1) / 5], Fx{d.z, d.w});
          }
#pragma unroll
          for (int s = 0; s < 5; s++) w[s] = fx_split(fx_shift(sum[s].value(), sh));
        }
      }
      if (__all_sync(0xffffffffu, rc[3] == 0)) {    /* regular patches without ghost or repeated slots */
        if (on) {
          const int4 *sl4 = reinterpret_cast<const int4 *>(rc + 4);
          const int4 t0 = sl4[0], t1 = sl4[1], t2 = sl4[2];
          acc[kRowWords * t0.x] += fx_entry_reg<0>(reg, w);
          acc[kRowWords * t0.y] += fx_entry_reg<1>(reg, w);
          acc[kRowWords * t0.z] += fx_entry_reg<2>(reg, w);
          acc[kRowWords * t0.w] += fx_entry_reg<3>(reg, w);
          acc[kRowWords * t1.x] += fx_entry_reg<4>(reg, w);
          acc[kRowWords * t1.y] += fx_entry_reg<5>(reg, w);
          acc[kRowWords * t1.z] += fx_entry_reg<6>(reg, w);
          acc[kRowWords * t1.w] += fx_entry_reg<7>(reg, w);
          acc[kRowWords * t2.x] += fx_entry_reg<8>(reg, w);
          acc[kRowWords * t2.y] += fx_entry_reg<9>(reg, w);
          acc[kRowWords * t2.z] += fx_entry_reg<10>(reg, w);
          acc[kRowWords * t2.w] += fx_entry_reg<11>(reg, w);
        }
      } else if (on) {
        const int nen = info & 0xff;
        for (int b = 0; b < nen; b++) {
          const unsigned sl = (unsigned)rc[4 + b];
          Fx n[5];
#pragma unroll
          for (int s = 0; s < 5; s++) {
            const int2 x = __ldg(tab + b * kFxTab + s);
            n[s] = Fx{x.x, x.y};
          }
          const long long v = fx_entry(n, w);
          acc[kRowWords * (int)(sl & 1023u)] += v;
          if ((sl & kRowSlotGhost) && !(sl & kRowSlotDup)) {   /* a repeated real node has one target */
            acc[kRowWords * (int)((sl >> 10) & 1023u)] += v;
            acc[kRowWords * (int)((sl >> 20) & 1023u)] -= v;
          }
        }
      }
      if (pres_live) __syncwarp();                   /* the contributions' own adds are done */
      if (pres_live && on) {
        /* lane (c, 3 k + d): component d of corner k's vector, entries (i, j) and (j, i) of its cross-product matrix */
        const int cs = rc[2], s0 = cs & 31, s1 = (cs >> 5) & 31, s2 = (cs >> 10) & 31;
        if (a == s0 || a == s1 || a == s2) {
          const int k = q / 3, d = q - 3 * k;
          const unsigned sl = (unsigned)rc[4 + (k == 0 ? s0 : k == 1 ? s1 : s2)];
          const double v = m.De[(size_t)kDeStride * e + kDePres + q];
          const int qm = d == 0 ? 5 : d == 1 ? 6 : 1, qp = d == 0 ? 7 : d == 1 ? 2 : 3;
          long long *dst = acc - q + kRowWords * (int)(sl & 1023u);
          dst[qm] -= fx_load(v * reg.den2, B.eb[qm]);
          dst[qp] += fx_load(v * reg.den2, B.eb[qp]);
        }
      }
      __syncwarp();   /* the records are rewritten by the next three */
    }
  }
  __syncwarp();
  /* dynamic term diagonal, scale, write-out */
  const double fmax = __longlong_as_double((long long)*m.fmax);
  const double sc = fmax > 1.0 ? 1.0 / fmax : 1.0;
  const int pd = p.dyn ? row_find(m.colind + k0, nb, i) : -1;
  const double dd = p.dyn ? m.dyn_diag[i] : 0.0;
  int blk = lane / 9, qq = lane - 9 * blk;
  for (int t = lane; t < 9 * nb; t += 32) {
    const long long *c = B.acc + kRowWords * blk + qq;
    double v;
    if (wide) {
      const double *f = reinterpret_cast<const double *>(c);
      v = ((f[0] + f[9]) + f[18]) * reg.unwide;
    } else {
      v = (double)(c[0] + c[9] + c[18]) * B.sc[qq];
    }
    if (blk == pd && qq % 4 == 0) v += dd;
    if (fmax > 1.0) v *= sc;
    Kr[colmajor ? t - qq + 3 * (qq % 3) + qq / 3 : t] = v;
    blk += 3; qq += 5;
    if (qq >= 9) { qq -= 9; blk++; }
  }
}

/* FP32 row assembly, the same way in single precision, each entry with its
   Kahan compensation beside it.  Latency and the L1 data path bound it:
   0.38 -> 0.26 ms on the 98,304-triangle sheet (0.31 without the early loads
   of D). */
constexpr int kRowF32Max = 64;       /* longest row that an FP32-bulk handle accepts */

__host__ __device__ __forceinline__ size_t row_f32_bytes(int maxblk)
{
  return (size_t)kRowWords * maxblk * 8 + kRowCopies * kRowRec * 4;
}

__device__ __forceinline__ void kahan_add(float2 &a, float v)
{
  const float2 s = a;
  const float y = v - s.y;
  const float t = s.x + y;
  a = make_float2(t, (t - s.x) - y);
}

template <int B> __device__ __forceinline__ float row_entry_reg(const RowTableF &reg, const float w[5])
{
  float v = 0.f;
#pragma unroll
  for (int s = 0; s < 5; s++)
    if (!row_reg_zero(s, B)) v = fmaf(reg.n[B][s], w[s], v);
  return v;
}

__device__ __forceinline__ float row_entry(const float n[5], const float w[5])
{
  float v = 0.f;
#pragma unroll
  for (int s = 0; s < 5; s++) v = fmaf(n[s], w[s], v);
  return v;
}

__global__ void __launch_bounds__(256, 2) k_row_assemble_f32(DevMesh m, KParams p, RowTableF reg,
                                                             float *__restrict__ K, int maxblk, int colmajor)
{
  extern __shared__ __align__(16) unsigned char row_smem[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int i = blockIdx.x * (blockDim.x >> 5) + wid;
  if (i >= p.nt) return;
  unsigned char *base = row_smem + (size_t)wid * row_f32_bytes(maxblk);
  float2 *racc = reinterpret_cast<float2 *>(base);                       /* kRowWords maxblk */
  int *rec = reinterpret_cast<int *>(base + (size_t)kRowWords * maxblk * 8);
  const int k0 = m.rowptr[i], nb = m.rowptr[i + 1] - k0;
  float *Kr = K + 9 * (size_t)k0;
  if (m.rowkind[i] != 0) {   /* clamped and ghost rows: identity */
    for (int t = lane; t < 9 * nb; t += 32) {
      const int q = t % 9;
      Kr[t] = (m.colind[k0 + t / 9] == i && (q == 0 || q == 4 || q == 8)) ? 1.f : 0.f;
    }
    return;
  }
  const int c0 = m.rptr[i], c1 = m.rptr[i + 1];
  const int4 *rrec4 = reinterpret_cast<const int4 *>(m.rrec);
  const bool pres_live = p.pressure != 0.0 && !p.pres_dead;
  const int pc = lane / 9, q = lane - 9 * pc;       /* contribution and entry; lanes 27..31 idle */
  int4 nrec = make_int4(0, 0, 0, 0);
  if (lane < (kRowRec / 4) * min(kRowCopies, c1 - c0)) nrec = __ldg(rrec4 + (size_t)(kRowRec / 4) * c0 + lane);
  float2 *acc = racc + lane;
  for (int t = 0; t < nb; t++) acc[kRowWords * t] = make_float2(0.f, 0.f);
  /* D of the next three contributions is in flight while three are added */
  float4 dn[6];
  float dn24 = 0.f;
  auto load_d = [&](int c) {
    if (pc >= kRowCopies || c >= c1) return;
    const int e = __ldg(m.rrec + (size_t)kRowRec * c) & ((1 << 27) - 1);
    const float4 *D = reinterpret_cast<const float4 *>(m.DeF + (size_t)kDeStride * e) + q;
#pragma unroll
    for (int s = 0; s < 6; s++) dn[s] = __ldg(D + 9 * s);
    dn24 = __ldg(m.DeF + (size_t)kDeStride * e + 216 + q);
  };
  load_d(c0 + pc);
  for (int cb = c0; cb < c1; cb += kRowCopies) {
    const int np = min(kRowCopies, c1 - cb);
    if (lane < (kRowRec / 4) * np) reinterpret_cast<int4 *>(rec)[lane] = nrec;
    if (lane < (kRowRec / 4) * min(kRowCopies, c1 - cb - kRowCopies))
      nrec = __ldg(rrec4 + (size_t)(kRowRec / 4) * (cb + kRowCopies) + lane);
    __syncwarp();   /* also orders the set-up */
    const bool on = pc < np;
    const int *rc = rec + kRowRec * (on ? pc : 0);
    const int e = rc[0] & ((1 << 27) - 1), a = rc[0] >> 27, info = rc[1];
    const float *tab = m.ntabF + (info >> 8) * 80;
    float w[5];
    if (on) {
      float n[5];
#pragma unroll
      for (int r = 0; r < 5; r++) n[r] = (info >> 8) == 0 ? reg.n[a][r] : __ldg(tab + 16 * r + a);
#pragma unroll
      for (int s = 0; s < 5; s++) w[s] = fmaf(n[3], dn[s].w, fmaf(n[2], dn[s].z, fmaf(n[1], dn[s].y, n[0] * dn[s].x)));
      w[0] = fmaf(n[4], dn[5].x, w[0]); w[1] = fmaf(n[4], dn[5].y, w[1]);
      w[2] = fmaf(n[4], dn[5].z, w[2]); w[3] = fmaf(n[4], dn[5].w, w[3]);
      w[4] = fmaf(n[4], dn24, w[4]);
    }
    load_d(cb + kRowCopies + pc);
    if (__all_sync(0xffffffffu, rc[3] == 0)) {    /* regular patches without ghost or repeated slots */
      if (on) {
        const int4 *sl4 = reinterpret_cast<const int4 *>(rc + 4);
        const int4 t0 = sl4[0], t1 = sl4[1], t2 = sl4[2];
        kahan_add(acc[kRowWords * t0.x], row_entry_reg<0>(reg, w));
        kahan_add(acc[kRowWords * t0.y], row_entry_reg<1>(reg, w));
        kahan_add(acc[kRowWords * t0.z], row_entry_reg<2>(reg, w));
        kahan_add(acc[kRowWords * t0.w], row_entry_reg<3>(reg, w));
        kahan_add(acc[kRowWords * t1.x], row_entry_reg<4>(reg, w));
        kahan_add(acc[kRowWords * t1.y], row_entry_reg<5>(reg, w));
        kahan_add(acc[kRowWords * t1.z], row_entry_reg<6>(reg, w));
        kahan_add(acc[kRowWords * t1.w], row_entry_reg<7>(reg, w));
        kahan_add(acc[kRowWords * t2.x], row_entry_reg<8>(reg, w));
        kahan_add(acc[kRowWords * t2.y], row_entry_reg<9>(reg, w));
        kahan_add(acc[kRowWords * t2.z], row_entry_reg<10>(reg, w));
        kahan_add(acc[kRowWords * t2.w], row_entry_reg<11>(reg, w));
      }
    } else if (on) {
      const int nen = info & 0xff;
      for (int b = 0; b < nen; b++) {
        const unsigned sl = (unsigned)rc[4 + b];
        float n[5];
#pragma unroll
        for (int s = 0; s < 5; s++) n[s] = __ldg(tab + 16 * s + b);
        const float v = row_entry(n, w);
        kahan_add(acc[kRowWords * (int)(sl & 1023u)], v);
        if ((sl & kRowSlotGhost) && !(sl & kRowSlotDup)) {   /* a repeated real node has one target */
          kahan_add(acc[kRowWords * (int)((sl >> 10) & 1023u)], v);
          kahan_add(acc[kRowWords * (int)((sl >> 20) & 1023u)], -v);
        }
      }
    }
    if (pres_live) __syncwarp();                     /* the contributions' own adds are done */
    if (pres_live && on) {
      /* lane (c, 3 k + d): component d of corner k's vector, entries (i, j) and (j, i) of its cross-product matrix */
      const int cs = rc[2], s0 = cs & 31, s1 = (cs >> 5) & 31, s2 = (cs >> 10) & 31;
      if (a == s0 || a == s1 || a == s2) {
        const int k = q / 3, d = q - 3 * k;
        const unsigned sl = (unsigned)rc[4 + (k == 0 ? s0 : k == 1 ? s1 : s2)];
        const float v = m.DeF[(size_t)kDeStride * e + kDePres + q];
        float2 *dst = acc - q + kRowWords * (int)(sl & 1023u);
        kahan_add(dst[d == 0 ? 5 : d == 1 ? 6 : 1], -v);
        kahan_add(dst[d == 0 ? 7 : d == 1 ? 2 : 3], v);
      }
    }
    __syncwarp();   /* the records are rewritten by the next three */
  }
  __syncwarp();
  /* dynamic term diagonal, scale, block layout */
  const double fmax = __longlong_as_double((long long)*m.fmax);
  const int pd = p.dyn ? row_find(m.colind + k0, nb, i) : -1;
  const float dd = p.dyn ? (float)m.dyn_diag[i] : 0.f;
  int blk = lane / 9, qq = lane - 9 * blk;
  for (int t = lane; t < 9 * nb; t += 32) {
    const float2 *c = racc + kRowWords * blk + qq;
    const float2 s0 = c[0], s1 = c[9], s2 = c[18];
    float v = ((s0.x + s1.x) + s2.x) - ((s0.y + s1.y) + s2.y);
    if (blk == pd && qq % 4 == 0) v += dd;
    if (fmax > 1.0) v = (float)((double)v * (1.0 / fmax));
    Kr[colmajor ? t - qq + 3 * (qq % 3) + qq / 3 : t] = v;
    blk += 3; qq += 5;
    if (qq >= 9) { qq -= 9; blk++; }
  }
}

/* Row-assembly records (see DevMesh::rrec), built on the device once per
   mesh: one warp per row, lanes over (contribution, patch slot); the slot's
   target is its node's position in the row's sorted columns (a lower-bound
   search), a ghost slot packs its parents nv2, nv1, nv3 at 10 bits each with
   kRowSlotGhost, and a slot repeating an earlier slot's real node is marked
   kRowSlotGhost | kRowSlotDup with its one target (it then takes the ghost
   slots' serial path).  Rows with an identity block get zero records. */
__device__ __forceinline__ unsigned col_lower_bound(const int *cols, int nb, int node)
{
  int lo = 0, hi = nb;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (cols[mid] < node) lo = mid + 1; else hi = mid;
  }
  return (unsigned)lo;
}

__global__ void k_row_records(DevMesh m, KParams p, int *__restrict__ rrec)
{
  const int lane = threadIdx.x & 31;
  const int i = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (i >= p.nt) return;
  const int c0 = m.rptr[i], c1 = m.rptr[i + 1];
  const bool live = m.rowkind[i] == 0;
  const int k0 = m.rowptr[i], nb = m.rowptr[i + 1] - k0;
  const int *cols = m.colind + k0;
  for (int u = lane; u < 16 * (c1 - c0); u += 32) {
    const int c = c0 + (u >> 4), b = u & 15;
    int *r = rrec + (size_t)kRowRec * c;
    const int code = m.ridx[c];                  /* 3 a ne + e */
    const int e = code % p.ne, a = code / (3 * p.ne);
    const int info = m.einfo[e], nen = info & 0xff;
    if (b == 0) {
      r[0] = live ? (e | (a << 27)) : 0;
      r[1] = live ? info : 0;
      r[2] = live ? m.ecorner[e] : 0;
      /* 0: a regular patch of real, distinct nodes */
      const int *pe = m.patch + 16 * (size_t)e;
      int general = info != 12;
      for (int b1 = 0; b1 < nen; b1++) {
        general |= pe[b1] >= p.nv;
        for (int b2 = 0; b2 < b1; b2++) general |= pe[b2] == pe[b1];
      }
      r[3] = live ? general : 0;
    }
    unsigned sl = 0;
    if (live && b < nen) {
      const int *pe = m.patch + 16 * (size_t)e;
      const int node = pe[b];
      if (node < p.nv) {
        sl = col_lower_bound(cols, nb, node);
        for (int b2 = 0; b2 < b; b2++)
          if (pe[b2] == node) { sl |= kRowSlotGhost | kRowSlotDup | (sl << 10) | (1023u << 20); break; }
      } else {
        const int g = node - p.nv;
        sl = kRowSlotGhost | col_lower_bound(cols, nb, m.ghost3[3 * g + 1]) |
             (col_lower_bound(cols, nb, m.ghost3[3 * g]) << 10) | (col_lower_bound(cols, nb, m.ghost3[3 * g + 2]) << 20);
      }
    }
    r[4 + b] = (int)sl;
  }
}

/* The growth bits of every row of the fixed-point assembly (fx_growth), once
   per mesh: one warp per row, lane t the bound of block t. */
__global__ void k_row_growth(DevMesh m, KParams p, unsigned char *__restrict__ rgrow)
{
  const int lane = threadIdx.x & 31;
  const int i = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (i >= p.nt) return;
  const int nb = m.rowptr[i + 1] - m.rowptr[i];
  const int c0 = m.rptr[i], c1 = m.rowkind[i] == 0 ? m.rptr[i + 1] : c0;
  long long most = 0;
  for (int t = lane; t < nb; t += 32) {
    long long sum = 0;
    for (int c = c0; c < c1; c++) {
      const int *rc = m.rrec + (size_t)kRowRec * c;
      const int *tab = m.ntabFx + (rc[1] >> 8) * 16 * 2 * kFxTab + 2 * kFxTab - 2;   /* the columns' sums */
      const int nen = rc[1] & 0xff, a = rc[0] >> 27, cs = rc[2];
      auto corner = [&](int b) { return b == (cs & 31) || b == ((cs >> 5) & 31) || b == ((cs >> 10) & 31); };
      int s = 0;
      for (int b = 0; b < nen; b++) {
        const unsigned sl = (unsigned)rc[4 + b];
        const unsigned u = t;
        const bool hit = (sl & 1023u) == u ||
                         ((sl & kRowSlotGhost) && !(sl & kRowSlotDup) && (((sl >> 10) & 1023u) == u || ((sl >> 20) & 1023u) == u));
        if (hit) s += tab[2 * kFxTab * b];
        if (hit && corner(a) && corner(b)) sum += 64 * 64;      /* the pressure block */
      }
      sum += (long long)s * tab[2 * kFxTab * a];
    }
    most = max(most, sum);
  }
  for (int o = 16; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
  if (lane == 0) rgrow[i] = (unsigned char)fx_growth(most);
}

int launch_row_growth(const DevMesh &m, const KParams &p, unsigned char *rgrow, void *stream)
{
  const long long threads = 32LL * p.nt;
  k_row_growth<<<(unsigned)((threads + 255) / 256), 256, 0, (cudaStream_t)stream>>>(m, p, rgrow);
  return (int)cudaGetLastError();
}

int launch_row_records(const DevMesh &m, const KParams &p, int *rrec, void *stream)
{
  const long long threads = 32LL * p.nt;
  k_row_records<<<(unsigned)((threads + 255) / 256), 256, 0, (cudaStream_t)stream>>>(m, p, rrec);
  return (int)cudaGetLastError();
}

/* ---------------- scaling ---------------- */
__global__ void k_scale(DevMesh m, KParams p, double *__restrict__ R)
{
  const double fmax = __longlong_as_double((long long)*m.fmax);
  if (!(fmax > 1.0)) return;
  const double sc = 1.0 / fmax;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < 3LL * p.nt) R[t] = R[t] * sc;
}

/* ---------------- launchers ---------------- */
static inline int blocks_for(long long n, int bs) { return (int)((n + bs - 1) / bs); }

int launch_ref_prep(const DevMesh &m, const KParams &p, const double *fib, const double *gscale, double *eref_out, void *stream)
{
  k_ref_prep<<<blocks_for(p.ne, 128), 128, 0, (cudaStream_t)stream>>>(m, p, fib, gscale, eref_out);
  return (int)cudaGetLastError();
}

int launch_positions(const DevMesh &m, const KParams &p, const double *x, void *stream)
{
  k_positions<<<blocks_for(p.nt, 256), 256, 0, (cudaStream_t)stream>>>(p.nv, p.ng, x, m.ghost3, m.pos, m.fmax);
  return (int)cudaGetLastError();
}

/* Lanes an element of k_elem_residual.  Its time is a warp's FP64 chain times
   the warps each of the 608 FP64 units gets.  Three lanes up to two rounds of
   ten elements a unit: 1,536 triangles 62 -> 33 us (123 -> 55 with gradients),
   6,144 triangles 62 -> 47 (115 -> 86), 12,160 triangles 63 -> 49 (115 -> 87).
   From there one lane's single round of 32 elements a unit is the shorter:
   13,774 triangles 64 us against 85 (115 against 131). */
static int residual_lanes(int ne)
{
  constexpr int units = 4 * 152;
  return ne <= 2 * kResElems<3> * units ? 3 : 1;
}

int launch_elem_residual(const DevMesh &m, const KParams &p, void *stream, bool tangent)
{
  if (residual_lanes(p.ne) == 3)
    k_elem_residual<3><<<blocks_for(p.ne, kResElems<3> * (kResBlock / 32)), kResBlock, 0, (cudaStream_t)stream>>>(m, p, tangent);
  else
    k_elem_residual<1><<<blocks_for(p.ne, kResBlock), kResBlock, 0, (cudaStream_t)stream>>>(m, p, tangent);
  return (int)cudaGetLastError();
}

/* The same of k_elem_residual_ff, three CTAs an SM: a wave of 18,240 elements
   takes 31 to 35 us with three lanes (1,536 and 13,774 triangles), a wave of
   58,368 takes 52 to 58 with one (to 38,400 triangles). */
static int residual_ff_lanes(int ne)
{
  constexpr int warps = 3 * 152 * (kResBlock / 32);
  const int w3 = (ne - 1) / (kResElems<3> * warps) + 1, w1 = (ne - 1) / (kResElems<1> * warps) + 1;
  return 5 * w3 < 8 * w1 ? 3 : 1;
}

int launch_elem_residual_ff(const DevMesh &m, const KParams &p, void *stream)
{
  if (residual_ff_lanes(p.ne) == 3)
    k_elem_residual_ff<3><<<blocks_for(p.ne, kResElems<3> * (kResBlock / 32)), kResBlock, 0, (cudaStream_t)stream>>>(m, p);
  else
    k_elem_residual_ff<1><<<blocks_for(p.ne, kResBlock), kResBlock, 0, (cudaStream_t)stream>>>(m, p);
  return (int)cudaGetLastError();
}

int launch_to_ff(const double *a, float *b, long long n, void *stream)
{
  k_to_ff<<<blocks_for(n, 256), 256, 0, (cudaStream_t)stream>>>(a, b, n);
  return (int)cudaGetLastError();
}

int launch_elem_tangent(const DevMesh &m, const KParams &p, void *stream)
{
  k_elem_tangent<<<blocks_for(p.ne, 4 * kTanElems), 128, 0, (cudaStream_t)stream>>>(m, p);
  return (int)cudaGetLastError();
}

int launch_elem_tangent_f32(const DevMesh &m, const KParams &p, void *stream)
{
  k_elem_tangent_f32<<<blocks_for(p.ne, kTanF32Block), kTanF32Block, 0, (cudaStream_t)stream>>>(m, p);
  return (int)cudaGetLastError();
}

/* UpdateElementThickness (active_strain.c:2198-2224): one thread per element,
   the residual kernel's geometry and stress with C33 of every thickness point
   kept; thickness = h0 sqrt(mean C33). */
__global__ void __launch_bounds__(128) k_elem_thickness(DevMesh m, KParams p, double h0, double *__restrict__ th)
{
  __shared__ double tabs[kNumTables * 80];
  for (int i = threadIdx.x; i < kNumTables * 80; i += blockDim.x) tabs[i] = m.ntab[i];
  __syncthreads();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= p.ne) return;
  const int info = m.einfo[e];
  const int nen = info & 0xff, tabi = info >> 8;
  double y[15];
  gather_y(m.pos, m.patch, e, nen, tabs + tabi * 80, y);
  int st = 0;
  const EPar<double> ep = epar<double>(p);
  th[e] = elem_thickness<double>(y, ep, RefCol<double>{m.eref + e, (size_t)p.ne}, h0, st);
  set_status(m.status, st);
}

int launch_elem_thickness(const DevMesh &m, const KParams &p, double h0, double *th, void *stream)
{
  k_elem_thickness<<<blocks_for(p.ne, 128), 128, 0, (cudaStream_t)stream>>>(m, p, h0, th);
  return (int)cudaGetLastError();
}

/* d Fdyn / d x: per free node, the triangle-order sum over its corner
   triangles of M M1 + C C1 (Newmark) or M / dt^2 + C / dt (central) */
__global__ void k_dyn_diag(DevMesh m, KParams p)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.nt) return;
  double s = 0.0;
  if (m.rowkind[i] == 0) {
    for (int c = m.dptr[i]; c < m.dptr[i + 1]; c++) {
      const double M = p.dyn_rhoh0 * m.dA0[m.didx[c]] / 3;
      const double C = p.dyn_damp ? p.dyn_dampf * M : 0.0;
      s += p.dyn_central ? M / (p.dyn_dt * p.dyn_dt) + C / p.dyn_dt : M * p.dyn_M1 + C * p.dyn_C1;
    }
  }
  m.dyn_diag[i] = s;
}

/* xAccVel (main.c:1367-1412; with the DMPlex context the n_v real nodes),
   then xnm1 <- xn, xn <- x over every entry (main.c:571-572) */
__global__ void k_dyn_update(DevMesh m, KParams p, const double *__restrict__ x)
{
  const size_t j = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (j >= 3 * (size_t)p.nt) return;
  if (j < 3 * (size_t)p.nv) {
    const double xddn = m.xdd[j];
    const double a = p.dyn_M1 * (x[j] - m.xn[j]) - p.dyn_M2 * m.xd[j] - p.dyn_M3 * m.xdd[j];
    m.xdd[j] = a;
    m.xd[j] = m.xd[j] + p.dyn_U2 * xddn + p.dyn_U3 * a;
  }
  m.xnm1[j] = m.xn[j];
  m.xn[j] = x[j];
}

int launch_dyn_diag(const DevMesh &m, const KParams &p, void *stream)
{
  k_dyn_diag<<<blocks_for(p.nt, 256), 256, 0, (cudaStream_t)stream>>>(m, p);
  return (int)cudaGetLastError();
}

int launch_dyn_update(const DevMesh &m, const KParams &p, const double *x, void *stream)
{
  k_dyn_update<<<blocks_for(3LL * p.nt, 256), 256, 0, (cudaStream_t)stream>>>(m, p, x);
  return (int)cudaGetLastError();
}

int launch_node_gather(const DevMesh &m, const KParams &p, const double *x, double *R, void *stream, double *parts)
{
  k_node_gather<<<dim3(blocks_for(p.nt, 128), 3), 128, 0, (cudaStream_t)stream>>>(m, p, x, R, parts);
  return (int)cudaGetLastError();
}

/* Warps a CTA: of 8, 4, 2, 1 the one that keeps most warps on an SM (24 by
   registers at most for FP64, 32 for FP32; 227 KB shared, 1 KB of it reserved per CTA). */
static size_t row_bytes(int maxblk, bool f32) { return f32 ? row_f32_bytes(maxblk) : fx_row_bytes(maxblk); }

static int row_warps(int maxblk, bool f32)
{
  int best = 1, most = 0;
  for (int w = 8; w >= 1; w /= 2) {
    const int ctas = (int)(228 * 1024 / (w * row_bytes(maxblk, f32) + 1024));
    const int warps = std::min(w * ctas, f32 ? 32 : 24);
    if (warps > most) { most = warps; best = w; }
  }
  return best;
}

size_t row_assemble_smem(int maxblk, bool f32) { return row_warps(maxblk, f32) * row_bytes(maxblk, f32); }

/* The regular table for the row assemblies; false when it does not have the
   zeros or (FP64) the common denominator that they rely on. */
bool regular_tables(const double *tab0, int den, RowTables &t)
{
  bool ok = true;
  for (int b = 0; b < 12; b++)
    for (int s = 0; s < 5; s++) {
      const double v = tab0[16 * s + b];
      const int k = (int)llrint(v * den);
      ok &= (double)k / den == v && (!row_reg_zero(s, b) || k == 0);
      t.x.n[b][s] = k;
      t.f.n[b][s] = (float)v;
    }
  t.x.den2 = (double)den * den;
  t.x.unit = ldexp(1.0 / t.x.den2, -kFxUnit);
  t.x.wide = ldexp(t.x.den2, -kFxDenBits);
  t.x.unwide = ldexp(1.0 / t.x.den2, kFxDenBits);
  return ok;
}

int row_assemble_max_blocks(bool f32) { return f32 ? kRowF32Max : kMaxRowBlocks; }

int launch_row_assemble(const DevMesh &m, const KParams &p, const RowTables &t, void *K, bool f32, bool colmajor, void *stream)
{
  const int warps = row_warps(m.maxblk, f32);
  const int grid = blocks_for(p.nt, warps);
  const size_t smem = row_assemble_smem(m.maxblk, f32);
  if (f32)
    k_row_assemble_f32<<<grid, 32 * warps, smem, (cudaStream_t)stream>>>(
        m, p, t.f, static_cast<float *>(K), m.maxblk, (int)colmajor);
  else
    k_row_assemble_fx<<<grid, 32 * warps, smem, (cudaStream_t)stream>>>(
        m, p, t.x, static_cast<double *>(K), m.maxblk, (int)colmajor);
  return (int)cudaGetLastError();
}

/* The kernels' dynamic shared-memory limit is raised to the device's, once and
   for every handle (a limit set to one handle's need would fail another's
   larger launch); a row buffer that does not fit is refused here. */
int row_assemble_configure(int maxblk, bool f32)
{
  int dev = 0, optin = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e == cudaSuccess && row_assemble_smem(maxblk, f32) > (size_t)optin) e = cudaErrorInvalidValue;
  if (e == cudaSuccess)
    e = f32 ? cudaFuncSetAttribute(k_row_assemble_f32, cudaFuncAttributeMaxDynamicSharedMemorySize, optin)
            : cudaFuncSetAttribute(k_row_assemble_fx, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
  return (int)e;
}

int launch_scale(const DevMesh &m, const KParams &p, double *R, void *stream)
{
  k_scale<<<blocks_for(3LL * p.nt, 256), 256, 0, (cudaStream_t)stream>>>(m, p, R);
  return (int)cudaGetLastError();
}

} /* namespace biofem */
