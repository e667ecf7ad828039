/*
 * Device Newton solve of R(x) = 0 with the assembled tangent: replaces the
 * reference's matrix-free PETSc SNES (newtonls + MFFD + GMRES, main.c:461-551)
 * for one quasi-static load step.
 *
 *   Newton:   x <- x + alpha dx,  K(x) dx = -R(x),  backtracking on ||R||
 *             (sufficient decrease 1e-4, halving up to 12 times), stop at
 *             ||R|| <= rtol ||R0|| (or atol); linear solves to a fixed
 *             relative tolerance or to Eisenstat-Walker forcing terms.
 *   Linear:   restarted flexible GMRES(m) (the preconditioned directions are
 *             kept), preconditioned by smoothed-aggregation multigrid (FP32
 *             V-cycle, amg.cu) or by block-Jacobi(3x3); classical
 *             Gram-Schmidt applied twice, Givens rotations and the small
 *             triangular solve on the device; all Krylov vectors and the
 *             dot products in FP64; the BSR matvec in FP64, or, with the FP32
 *             tangent of an FP32-bulk handle, in float-float arithmetic on
 *             the FP32 pipe (about 47 bits, against K's own 24).  One
 *             iteration: preconditioner, matvec with the first dot products,
 *             projection with the second ones and the Givens step, and the
 *             normalised update, which also starts the next V-cycle.
 * Ghost rows of K are identity and their residual is zero, so ghost entries
 * of x never move.
 */
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <string>
#include <vector>

#include "amg.h"
#include "arena.h"
#include "biofem_host.h"
#include "ff.cuh"

namespace biofem {

int noalloc_fail(int code, const std::string &msg);   /* error reporting (bridge.cu) */

/* ---------------- kernels ---------------- */
/* ---------------- device-resident GMRES state ---------------- */
struct GmState {
  int done;        /* 1 once the cycle has converged, broken down or reached its length */
  int jdone;       /* iterations completed in this cycle: the column the next one works on */
  double bnorm, tol, resid, hn, inv_hn;
};
__device__ __forceinline__ bool gm_done(const GmState *gs) { return gs->done != 0; }

/* A float as a double by its bits: the conversion instruction runs on the FP64
   pipe, at the cost of a multiply-add each (40 % of the FP64 matvec's). */
__device__ __forceinline__ double widen(float x) { return ff_widen(x); }
__device__ __forceinline__ double widen(double x) { return x; }

/* One block row of y = K x over a warp: lane l < 30 on row l % 3 of the 3x3
   blocks l / 3, l / 3 + 10, .., so that neighbouring lanes read neighbouring K;
   S is the stride of a node in x (3, or 4: the V-cycle's padded FP32 result,
   then one 16-byte load).  s[0..2], the three sums, in every lane. */
template <int S, class XT> __device__ __forceinline__ void load_x(const XT *__restrict__ x, int c, XT v[3])
{
  if constexpr (S == 4) {
    const float4 w = *reinterpret_cast<const float4 *>(x + 4 * (size_t)c);
    v[0] = w.x; v[1] = w.y; v[2] = w.z;
  } else {
#pragma unroll
    for (int d = 0; d < 3; d++) v[d] = x[3 * (size_t)c + d];
  }
}

/* a lane's next blocks k, k + 10, .. below k1, all asked for before one is used */
constexpr int kRowBatch = 4;         /* 40 blocks: a regular row's 37 */
template <int S, class KT, class XT>
__device__ __forceinline__ void load_row_batch(const int *__restrict__ colind, const KT *__restrict__ Kr,
                                               const XT *__restrict__ x, int k, int k1, KT b[kRowBatch][3],
                                               XT xv[kRowBatch][3])
{
  int c[kRowBatch];
#pragma unroll
  for (int t = 0; t < kRowBatch; t++) {
    const int kk = min(k + 10 * t, k1 - 1);      /* past the end: the row's last block again, not used */
    c[t] = __ldg(colind + kk);
#pragma unroll
    for (int d = 0; d < 3; d++) b[t][d] = __ldg(Kr + 9 * (size_t)kk + d);
  }
#pragma unroll
  for (int t = 0; t < kRowBatch; t++) load_x<S>(x, c[t], xv[t]);
}

template <int S, class XT>
__device__ __forceinline__ void bsr_row(int k0, int k1, const int *__restrict__ colind, const double *__restrict__ K,
                                        const XT *__restrict__ x, int lane, double s[3])
{
  double v = 0.0;
  if (lane < 30) {
    const double *Kr = K + 3 * (lane % 3);
    for (int k = k0 + lane / 3; k < k1; k += 10 * kRowBatch) {
      double b[kRowBatch][3];
      XT xv[kRowBatch][3];
      load_row_batch<S>(colind, Kr, x, k, k1, b, xv);
#pragma unroll
      for (int t = 0; t < kRowBatch; t++)
        if (k + 10 * t < k1) v += b[t][0] * widen(xv[t][0]) + b[t][1] * widen(xv[t][1]) + b[t][2] * widen(xv[t][2]);
    }
  }
  v += __shfl_down_sync(0xffffffffu, v, 15);
  const double a = __shfl_down_sync(0xffffffffu, v, 3), b = __shfl_down_sync(0xffffffffu, v, 6);
  const double c = __shfl_down_sync(0xffffffffu, v, 9), d = __shfl_down_sync(0xffffffffu, v, 12);
  v = ((v + a) + (b + c)) + d;
#pragma unroll
  for (int r = 0; r < 3; r++) s[r] = __shfl_sync(0xffffffffu, v, r);
}

/* The same for FP32 K, on the FP32 pipe (GB300's FP64 pipe runs at 1/64 of its
   rate): each product K x.hi is formed exactly (two-product) and summed with
   two-sum, the tails and K x.lo go to the low word (ff_axpy); about 47
   significant bits, where K itself carries 24.  The V-cycle's result is FP32,
   so x has no low part there; an FP64 x is split where it is read. */
__device__ __forceinline__ FF ff_of(float x) { return FF(x, 0.f); }
__device__ __forceinline__ FF ff_of(double x) { return ff_split(x); }
/* v += the lane's d further down, the tails' sum left to be normalised */
__device__ __forceinline__ void ff_add_down(FF &v, int d)
{
  const FF s = ff_two_sum(v.hi, __shfl_down_sync(0xffffffffu, v.hi, d));
  v.lo += __shfl_down_sync(0xffffffffu, v.lo, d) + s.lo;
  v.hi = s.hi;
}
template <int S, class XT>
__device__ __forceinline__ void bsr_row(int k0, int k1, const int *__restrict__ colind, const float *__restrict__ K,
                                        const XT *__restrict__ x, int lane, double s[3])
{
  FF v(0.f, 0.f);
  if (lane < 30) {
    const float *Kr = K + 3 * (lane % 3);
    for (int k = k0 + lane / 3; k < k1; k += 10 * kRowBatch) {
      float b[kRowBatch][3];
      XT xv[kRowBatch][3];
      load_row_batch<S>(colind, Kr, x, k, k1, b, xv);
#pragma unroll
      for (int t = 0; t < kRowBatch; t++)
        if (k + 10 * t < k1) {
          ff_axpy(v, b[t][0], ff_of(xv[t][0])); ff_axpy(v, b[t][1], ff_of(xv[t][1])); ff_axpy(v, b[t][2], ff_of(xv[t][2]));
        }
    }
  }
  ff_add_down(v, 15);
  FF a = v;
  ff_add_down(a, 3);          /* lanes 0 .. 2: blocks 0 + 1 (mod 5) */
  const FF f = FF(__shfl_down_sync(0xffffffffu, v.hi, 12), __shfl_down_sync(0xffffffffu, v.lo, 12));
  ff_add_down(a, 6);          /* + 2 + 3 */
  const FF u = ff_two_sum(a.hi, f.hi);
  const double t = ff_to_double_bits(ff_two_sum(u.hi, a.lo + f.lo + u.lo));
#pragma unroll
  for (int r = 0; r < 3; r++) s[r] = __shfl_sync(0xffffffffu, t, r);
}

/* y = b - K x (a cycle's start) */
template <class KT>
__global__ void __launch_bounds__(256) k_bsr_resid(int nb, const int *__restrict__ rowptr, const int *__restrict__ colind,
                                                   const KT *__restrict__ K, const double *__restrict__ x,
                                                   const double *__restrict__ b, double *__restrict__ y)
{
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= nb) return;
  double s[3];
  bsr_row<3>(rowptr[row], rowptr[row + 1], colind, K, x, lane, s);
  if (lane < 3) {
    const size_t o = 3 * (size_t)row + lane;
    y[o] = b[o] - (lane == 0 ? s[0] : lane == 1 ? s[1] : s[2]);
  }
}

/* inverse of every diagonal block (block-Jacobi) */
template <class KT>
__global__ void k_bj_setup(int nb, const int *__restrict__ rowptr, const int *__restrict__ colind,
                           const KT *__restrict__ K, double *__restrict__ Dinv, int *__restrict__ status)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nb) return;
  double a[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
  for (int k = rowptr[i]; k < rowptr[i + 1]; k++)
    if (colind[k] == i) { for (int v = 0; v < 9; v++) a[v] = (double)K[9 * (size_t)k + v]; break; }
  const double c00 = a[4] * a[8] - a[5] * a[7], c01 = a[5] * a[6] - a[3] * a[8], c02 = a[3] * a[7] - a[4] * a[6];
  const double det = a[0] * c00 + a[1] * c01 + a[2] * c02;
  double *o = Dinv + 9 * (size_t)i;
  if (!(fabs(det) > 0.0) || !isfinite(det)) {
    atomicOr(status, 2);
    for (int v = 0; v < 9; v++) o[v] = (v % 4 == 0) ? 1.0 : 0.0;
    return;
  }
  const double id = 1.0 / det;
  o[0] = c00 * id; o[1] = (a[2] * a[7] - a[1] * a[8]) * id; o[2] = (a[1] * a[5] - a[2] * a[4]) * id;
  o[3] = c01 * id; o[4] = (a[0] * a[8] - a[2] * a[6]) * id; o[5] = (a[2] * a[3] - a[0] * a[5]) * id;
  o[6] = c02 * id; o[7] = (a[1] * a[6] - a[0] * a[7]) * id; o[8] = (a[0] * a[4] - a[1] * a[3]) * id;
}

/* z_j = D^-1 v_j, columns j = gs->jdone of V and Z */
__global__ void k_bj_apply(int nb, const double *__restrict__ Dinv, const double *V, double *Z, const GmState *gs, bool check)
{
  if (check && gm_done(gs)) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nb) return;
  const size_t col = 3 * (size_t)nb * gs->jdone;
  const double *d = Dinv + 9 * (size_t)i, *r = V + col;
  double *z = Z + col;
  const double r0 = r[3 * (size_t)i], r1 = r[3 * (size_t)i + 1], r2 = r[3 * (size_t)i + 2];
  z[3 * (size_t)i] = d[0] * r0 + d[1] * r1 + d[2] * r2;
  z[3 * (size_t)i + 1] = d[3] * r0 + d[4] * r1 + d[5] * r2;
  z[3 * (size_t)i + 2] = d[6] * r0 + d[7] * r1 + d[8] * r2;
}

/* partial dot products of w with the first nv basis vectors (column stride
   ld): block (c, j) reduces column j over the c-th strided chunk */
constexpr int kDotBlocks = 128;
__global__ void k_multidot(int n, int nv, const double *__restrict__ V, size_t ld, const double *__restrict__ w,
                           double *__restrict__ part)
{
  __shared__ double red[8];
  const int j = blockIdx.y;
  const double *v = V + (size_t)j * ld;
  double acc = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) acc += v[i] * w[i];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); k++) t += red[k];
    part[(size_t)j * gridDim.x + blockIdx.x] = t;
  }
}

__global__ void k_reduce_parts(int nv, int nparts, const double *__restrict__ part, double *__restrict__ out)
{
  const int j = blockIdx.x;
  double v = 0.0;
  for (int k = threadIdx.x; k < nparts; k += blockDim.x) v += part[(size_t)j * nparts + k];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  __shared__ double s[32];
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); k++) t += s[k];
    out[j] = t;
  }
}

__global__ void k_scale_copy(int n, const double *__restrict__ a, double s, double *__restrict__ b)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = a[i] * s;
}

__global__ void k_axpby(int n, double a, const double *__restrict__ x, double b, double *__restrict__ y)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = a * x[i] + b * y[i];
}

__global__ void k_zero_ghost(int nv, int nt, double *__restrict__ v)
{
  const int i = nv * 3 + blockIdx.x * blockDim.x + threadIdx.x;
  if (i < 3 * nt) v[i] = 0.0;
}

/* Gram-Schmidt, applied twice, in three launches an iteration, each block
   owning a contiguous chunk of block rows throughout:
     k_gs_matvec   w = K z on the chunk, then the chunk's dot products with the
                   columns of V
     k_gs_project  w1 = w - V h1, then its dot products with V and itself
     k_gs_update   v = (w1 - V h2) / h_{j+1,j}, with the V-cycle's start and,
                   in a block of its own, the rest of the Arnoldi column
   A warp sums one column over the chunk before it reduces across lanes (the
   reduction is 5 of some 20 FP64 additions; reducing 8 columns every 2
   entries, it was most of them and the kernel took 32 us on the 98,304-triangle
   sheet).  The last block to finish (counted on an atomic ticket, the
   partials made visible by a fence) adds the partials of every column in a
   fixed order, so the result does not depend on block scheduling. */
constexpr int kGsBlocks = 304, kGsThreads = 512;      /* 2 x 152 SMs, 32 warps each */
constexpr int kMaxRestart = 200;

static inline int gs_rows(int nb) { return std::max(8, (nb + kGsBlocks - 1) / kGsBlocks); }   /* block rows a chunk */
static inline int gs_grid(int nb) { return (nb + gs_rows(nb) - 1) / gs_rows(nb); }

/* The dot products of w, `len` entries from i0 on, with columns 0..nv-1 of V
   (and with itself as column nv when `self`) to part; true in the last block,
   once hs holds every column's total (also written to out).  wl: the chunk's w,
   in shared memory where it fits (kGsLocal), so that it does not come back from
   L2.  One thread fences for the block: what the barrier ordered before it is
   covered. */
constexpr int kGsLocal = 1024;
__device__ __forceinline__ bool gs_chunk_dots(int nv, bool self, const double *V, size_t ld, const double *wl, int i0, int len,
                                              double *part, unsigned *ticket, double *out, double *hs)
{
  __shared__ int last;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int ncol = nv + (self ? 1 : 0);
  for (int c = wid; c < ncol; c += nw) {
    const double *v = c < nv ? V + (size_t)c * ld + i0 : wl;
    double s = 0.0;
#pragma unroll 4
    for (int i = lane; i < len; i += 32) s += v[i] * wl[i];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) part[(size_t)c * gridDim.x + blockIdx.x] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last) return false;
  for (int c = wid; c < ncol; c += nw) {
    double s = 0.0;
    for (int p = lane; p < (int)gridDim.x; p += 32) s += __ldcg(part + (size_t)c * gridDim.x + p);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) { hs[c] = s; out[c] = s; }
  }
  if (threadIdx.x == 0) *ticket = 0u;
  __syncthreads();
  return true;
}

/* w = K z_j over the chunk, then h1 = V^T w (columns 0..j), j = gs->jdone and
   w column j + 1 of V.  z_j is column j of Z, or, from the V-cycle, the FP32
   vector x (four values a node), which is copied to column j on the way. */
template <class KT, class XT>
__global__ void __launch_bounds__(kGsThreads) k_gs_matvec(int nb, int rows, const int *__restrict__ rowptr,
                                                          const int *__restrict__ colind, const KT *__restrict__ K,
                                                          const XT *x, XT *Z, double *V, double *__restrict__ part,
                                                          unsigned *__restrict__ ticket, double *__restrict__ h1,
                                                          const GmState *__restrict__ gs, bool check)
{
  if (check && gm_done(gs)) return;
  __shared__ double hs[kMaxRestart + 2], ws[kGsLocal];
  constexpr int S = sizeof(XT) == 4 ? 4 : 3;
  const int j = gs->jdone, nv = j + 1;
  const size_t ld = 3 * (size_t)nb;
  XT *zj = Z + j * ld;
  const XT *z = S == 4 ? x : zj;
  double *w = V + nv * ld;
  const int r0 = blockIdx.x * rows, r1 = min(nb, r0 + rows), lane = threadIdx.x & 31;
  const bool local = 3 * rows <= kGsLocal;
  int row = r0 + (threadIdx.x >> 5), k0 = 0, k1 = 0;
  if (row < r1) { k0 = rowptr[row]; k1 = rowptr[row + 1]; }
  for (; row < r1; row += kGsThreads / 32) {
    double s[3];
    const int b0 = k0, b1 = k1, next = row + kGsThreads / 32;
    if (next < r1) { k0 = rowptr[next]; k1 = rowptr[next + 1]; }      /* ahead of the row's own loads */
    bsr_row<S>(b0, b1, colind, K, z, lane, s);
    if (lane < 3) {
      const size_t o = 3 * (size_t)row + lane;
      const double v = lane == 0 ? s[0] : lane == 1 ? s[1] : s[2];
      w[o] = v;
      if (local) ws[o - 3 * (size_t)r0] = v;
      if (S == 4) zj[o] = z[S * (size_t)row + lane];
    }
  }
  __syncthreads();
  gs_chunk_dots(nv, false, V, ld, local ? ws : w + 3 * (size_t)r0, 3 * r0, 3 * (r1 - r0), part, ticket, h1, hs);
}

/* w -= V h1 on the chunk, h2 = V^T w and w.w; the last block: |w2|, the next
   vector's scale and the iteration count.  A chunk shorter than the block
   shares each entry's columns among several threads. */
__global__ void __launch_bounds__(kGsThreads) k_gs_project(int nb, int rows, double *V, const double *__restrict__ h1,
                                                           double *__restrict__ part, unsigned *__restrict__ ticket,
                                                           double *__restrict__ h2, GmState *__restrict__ gs, bool check)
{
  if (check && gm_done(gs)) return;
  __shared__ double hs[kMaxRestart + 2], h1s[kMaxRestart + 2], sum[kGsThreads], ws[kGsLocal];
  const int j = gs->jdone, nv = j + 1;
  const size_t ld = 3 * (size_t)nb;
  double *w = V + nv * ld;
  for (int c = threadIdx.x; c < nv; c += blockDim.x) h1s[c] = h1[c];
  __syncthreads();
  const int i0 = 3 * blockIdx.x * rows, i1 = min(3 * nb, i0 + 3 * rows), len = i1 - i0;
  const bool local = 3 * rows <= kGsLocal;
  if (len <= kGsThreads / 2) {
    const int ng = kGsThreads / len, g = threadIdx.x / len, i = i0 + threadIdx.x - g * len;
    double s = 0.0;
    if (g < ng) {
#pragma unroll 4
      for (int c = g; c < nv; c += ng) s += V[(size_t)c * ld + i] * h1s[c];
    }
    sum[threadIdx.x] = s;
    __syncthreads();
    if (g == 0) {
      for (int k = 1; k < min(ng, nv); k++) s += sum[threadIdx.x + k * len];
      const double v = w[i] - s;
      w[i] = v;
      if (local) ws[i - i0] = v;
    }
  } else {
    for (int i = i0 + threadIdx.x; i < i1; i += kGsThreads) {
      double s = 0.0;
#pragma unroll 8
      for (int c = 0; c < nv; c++) s += V[(size_t)c * ld + i] * h1s[c];
      const double v = w[i] - s;
      w[i] = v;
      if (local) ws[i - i0] = v;
    }
  }
  __syncthreads();
  if (!gs_chunk_dots(nv, true, V, ld, local ? ws : w + i0, i0, len, part, ticket, h2, hs)) return;
  if (threadIdx.x < 32) {
    double h2sq = 0.0;
    for (int i = threadIdx.x; i <= j; i += 32) h2sq += hs[i] * hs[i];
    for (int o = 16; o > 0; o >>= 1) h2sq += __shfl_xor_sync(0xffffffffu, h2sq, o);
    if (threadIdx.x == 0) {
      const double hn2 = hs[j + 1] - h2sq;       /* w1.w1 - |h2|^2 = |w2|^2 */
      const double hn = hn2 > 0.0 ? sqrt(hn2) : 0.0;
      gs->hn = hn;
      gs->inv_hn = hn > 0.0 ? 1.0 / hn : 0.0;
      gs->jdone = j + 1;
    }
  }
}

/* Second projection and normalisation, v = (w - V h2) / h_{j+1,j} in place in
   column j + 1 = gs->jdone of V, 64 nodes a block; with r0 given it starts a
   cycle: v0 = r0 / beta.  The preconditioner starts from the new v: b = v in
   FP32, r = D^-1 b, d = r / theta (pc.b null: block-Jacobi, nothing to do).
   The block behind those (not at a start) completes the Arnoldi column
   meanwhile: H[:, j] = h1 + h2 through the previous Givens rotations, a new
   rotation, the residual estimate, and whether the cycle is done. */
constexpr int kUpdNodes = 64;
struct Arnoldi {
  int m;
  const double *h1, *h2;
  double *H, *cs, *sn, *g;
};

/* One FP64 operation depends on the next at some 70 cycles here, so only what
   must is a chain: a_{i+1} = -s_i a_i + c_i col_{i+1}, the products before and
   after it formed by a thread each. */
__device__ __forceinline__ void givens_step(const Arnoldi &A, GmState *gs)
{
  __shared__ double col[kMaxRestart + 2], css[kMaxRestart], sns[kMaxRestart], cb[kMaxRestart], run[kMaxRestart + 2];
  const int j = gs->jdone - 1;
  const double hn = gs->hn, gj = A.g[j];
  for (int i = threadIdx.x; i <= j; i += blockDim.x) col[i] = A.h1[i] + A.h2[i];
  for (int i = threadIdx.x; i < j; i += blockDim.x) { css[i] = A.cs[i]; sns[i] = A.sn[i]; }
  __syncthreads();
  for (int i = threadIdx.x; i < j; i += blockDim.x) cb[i] = css[i] * col[i + 1];
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = col[0];
    run[0] = a;
    for (int i = 0; i < j; i++) { a = fma(-sns[i], a, cb[i]); run[i + 1] = a; }
    const double b = hn, sq = a * a + b * b;
    double r, c, s;
    if (sq > 1e-280 && sq < 1e280) {
      const double ri = rsqrt(sq);
      r = sq * ri; c = a * ri; s = b * ri;
    } else {                            /* zero, or squares out of range */
      r = hypot(a, b);
      c = r > 0 ? a / r : 1.0;
      s = r > 0 ? b / r : 0.0;
    }
    A.cs[j] = c;
    A.sn[j] = s;
    A.H[(size_t)j * A.m + j] = r;
    const double gn = -s * gj, resid = fabs(gn);
    A.g[j + 1] = gn;
    A.g[j] = c * gj;
    gs->resid = resid;
    if (resid <= gs->tol * gs->bnorm || hn == 0.0 || !(hn == hn) || j + 1 == A.m) gs->done = 1;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < j; i += blockDim.x) A.H[(size_t)i * A.m + j] = css[i] * run[i] + sns[i] * col[i + 1];
}

__global__ void __launch_bounds__(3 * kUpdNodes) k_gs_update(int n, double *V, const double *__restrict__ r0, AmgStart pc,
                                                             Arnoldi A, GmState *gs, bool check)
{
  __shared__ float vs[3 * kUpdNodes];
  const int i = blockIdx.x * (3 * kUpdNodes) + threadIdx.x;
  if (check) {
    __shared__ int skip;
    if (threadIdx.x == 0) skip = gs->done;         /* one answer for the block: the last one may set it meanwhile */
    __syncthreads();
    if (skip) return;
  }
  if (!r0 && blockIdx.x == gridDim.x - 1) { givens_step(A, gs); return; }
  if (i < n) {
    const int nv = r0 ? 0 : gs->jdone;
    double *v = V + (size_t)nv * n;
    double s = 0.0;
#pragma unroll 4
    for (int k = 0; k < nv; k++) s += V[(size_t)k * n + i] * A.h2[k];
    const double x = ((r0 ? r0[i] : v[i]) - s) * gs->inv_hn;
    v[i] = x;
    vs[threadIdx.x] = (float)x;
  }
  if (!pc.b) return;
  __syncthreads();
  if (i >= n) return;
  const int node = i / 3, t3 = threadIdx.x - threadIdx.x % 3;
  const float *D = pc.Dinv + 3 * (size_t)i;      /* row i % 3 of the node's inverse */
  const float rv = fmaf(D[2], vs[t3 + 2], fmaf(D[1], vs[t3 + 1], D[0] * vs[t3]));
  pc.b[i] = vs[threadIdx.x];
  pc.r[i] = rv;
  pc.d[4 * (size_t)node + i - 3 * node] = rv * *pc.theta_inv;
}

/* whether the graph's loop of iterations goes on */
__global__ void k_gs_loop(cudaGraphConditionalHandle loop, const GmState *gs)
{
  cudaGraphSetConditional(loop, gm_done(gs) ? 0u : 1u);
}

/* y = H^-1 g over the completed iterations: one warp, the column of the solved
   unknown taken out of every remaining right-hand side at once */
__global__ void k_backsolve(int m, const double *__restrict__ H, const double *__restrict__ g, double *__restrict__ y,
                            const GmState *__restrict__ gs)
{
  __shared__ double rhs[kMaxRestart];
  const int k = gs->jdone;
  for (int i = threadIdx.x; i < k; i += 32) rhs[i] = g[i];
  __syncwarp();
  for (int c = k - 1; c >= 0; c--) {
    const double yc = rhs[c] / H[(size_t)c * m + c];
    __syncwarp();
    for (int i = threadIdx.x; i < c; i += 32) rhs[i] -= H[(size_t)i * m + c] * yc;
    if (threadIdx.x == 0) y[c] = yc;
    __syncwarp();
  }
}

/* dx += Z y over the completed iterations (flexible GMRES keeps the
   preconditioned directions Z) */
template <class ZT>
__global__ void k_combine(int n, const ZT *__restrict__ Z, size_t ld, const double *__restrict__ y,
                          double *__restrict__ dx, const GmState *__restrict__ gs)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int k = gs->jdone;
  double s = 0.0;
  for (int j = 0; j < k; j++) s += widen(Z[(size_t)j * ld + i]) * y[j];
  dx[i] += s;
}

/* cycle start: beta = sqrt(rr), v0 = r / beta, g = (beta, 0, ...), flags reset */
__global__ void k_cycle_start(int m, const double *__restrict__ rr, double *__restrict__ g, GmState *__restrict__ gs)
{
  if (threadIdx.x != 0) return;
  const double beta = sqrt(rr[0]);
  if (gs->bnorm < 0.0) gs->bnorm = beta;       /* first cycle: dx = 0, r = b */
  gs->resid = beta;
  gs->jdone = 0;
  gs->inv_hn = beta > 0.0 ? 1.0 / beta : 0.0;
  gs->done = (beta <= gs->tol * gs->bnorm || beta == 0.0) ? 1 : 0;
  for (int i = 0; i <= m; i++) g[i] = 0.0;
  g[0] = beta;
}

/* solve start: tolerance in, ||b|| unknown until the first cycle */
__global__ void k_solve_begin(double tol, GmState *__restrict__ gs)
{
  if (threadIdx.x != 0) return;
  gs->tol = tol;
  gs->bnorm = -1.0;
  gs->done = 0;
  gs->jdone = 0;
}

/* ---------------- host side ---------------- */
static inline int nblk(long long n, int bs) { return (int)((n + bs - 1) / bs); }

/* Host waits of the solver.  A serving worker sets t_blocking_waits so that
   its thread sleeps on a blocking-sync event instead of spinning in
   cudaStreamSynchronize: with one worker per core the spinning threads took
   the cores the other requests' host preparation needed. */
thread_local bool t_blocking_waits = false;

static cudaError_t host_wait(cudaStream_t st, cudaEvent_t evb)
{
  if (t_blocking_waits && evb) {
    cudaError_t e = cudaEventRecord(evb, st);
    return e != cudaSuccess ? e : cudaEventSynchronize(evb);
  }
  return cudaStreamSynchronize(st);
}

/* Page-locked scalars a solver reads back (its GMRES state, one dot product,
   the element status word), from a process-wide free list: freeing
   page-locked memory can synchronise the whole device, which would make
   every request that finishes wait for all the others. */
struct PinnedScalars {
  GmState gs;
  double scal;
  int stat;
};
static std::mutex g_pin_mu;
static std::vector<PinnedScalars *> g_pin_free;

static PinnedScalars *pin_acquire()
{
  {
    std::lock_guard<std::mutex> lk(g_pin_mu);
    if (!g_pin_free.empty()) {
      PinnedScalars *p = g_pin_free.back();
      g_pin_free.pop_back();
      return p;
    }
  }
  void *p = nullptr;
  return cudaMallocHost(&p, sizeof(PinnedScalars)) == cudaSuccess ? static_cast<PinnedScalars *>(p) : nullptr;
}

static void pin_release(PinnedScalars *p)
{
  if (!p) return;
  std::lock_guard<std::mutex> lk(g_pin_mu);
  g_pin_free.push_back(p);
}

struct SolverWork {
  int n = 0, nb = 0, m = 0;
  double *V = nullptr, *Z = nullptr, *w = nullptr, *dinv = nullptr, *part = nullptr;
  double *h1 = nullptr, *h2 = nullptr, *H = nullptr, *cs = nullptr, *sn = nullptr, *g = nullptr, *y = nullptr;
  double *dx = nullptr, *xt = nullptr, *Rt = nullptr, *xh = nullptr;
  GmState *gs = nullptr;
  unsigned *ticket = nullptr;  /* last-block counter of k_gs_matvec / k_gs_project (returns to 0 after each launch) */
  PinnedScalars *pin = nullptr;   /* the page-locked block of the three below */
  GmState *hgs = nullptr;    /* pinned host copy */
  double *hscal = nullptr;   /* pinned host scalar */
  int *hstat = nullptr;      /* pinned host copy of the element status word */
  cudaEvent_t ev = nullptr;
  cudaEvent_t evb = nullptr; /* blocking-sync event for host_wait */
  /* the captured restart cycle and the arguments it was captured for */
  std::vector<cudaGraphExec_t> gexec;
  const double *g_b = nullptr;
  double *g_dx = nullptr;
  const void *g_K = nullptr;
  const void *g_pc = nullptr;   /* preconditioner the graph was captured with (null: block-Jacobi) */
  cudaStream_t st = nullptr;   /* allocation stream */
  Arena mem;
};

/* Restarted flexible GMRES(m), right-preconditioned (multigrid V-cycle or
   block-Jacobi); the Arnoldi process, the Givens rotations and the small
   triangular solve all run on the device.  Kernels skip their work once the
   cycle has converged. */
class Gmres {
 public:
  Gmres(const DevMesh &dm, const KParams &kp, bool f32, const void *K, SolverWork &w, AmgHier *amg, cudaStream_t st)
      : dm_(dm), kp_(kp), f32_(f32), K_(K), w_(w), amg_(amg), st_(st) {}

  /* z = M^-1 v_j: smoothed-aggregation V-cycle (started by k_gs_update), or
     block-Jacobi; then w = K z and h1 = V^T w */
  template <class KT> void precond_matvec(const KT *K, bool check)
  {
    const int rows = gs_rows(w_.nb), grid = gs_grid(w_.nb);
    if (amg_) {
      amg_apply(amg_, check ? &w_.gs->done : nullptr, st_);
      k_gs_matvec<<<grid, kGsThreads, 0, st_>>>(w_.nb, rows, dm_.rowptr, dm_.colind, K, amg_start(amg_).x, (float *)w_.Z, w_.V,
                                                w_.part, w_.ticket, w_.h1, w_.gs, check);
    } else {
      k_bj_apply<<<nblk(w_.nb, 256), 256, 0, st_>>>(w_.nb, w_.dinv, w_.V, w_.Z, w_.gs, check);
      k_gs_matvec<<<grid, kGsThreads, 0, st_>>>(w_.nb, rows, dm_.rowptr, dm_.colind, K, (const double *)nullptr, w_.Z, w_.V,
                                                w_.part, w_.ticket, w_.h1, w_.gs, check);
    }
  }
  /* a . b into a host double (synchronous) */
  int dot2(const double *a, const double *b, double &out)
  {
    k_multidot<<<dim3(kDotBlocks, 1), 256, 0, st_>>>(w_.n, 1, a, (size_t)w_.n, b, w_.part);
    k_reduce_parts<<<1, 128, 0, st_>>>(1, kDotBlocks, w_.part, w_.h1);
    cudaMemcpyAsync(w_.hscal, w_.h1, sizeof(double), cudaMemcpyDeviceToHost, st_);
    cudaError_t e = host_wait(st_, w_.evb);
    if (e != cudaSuccess) return (int)e;
    out = *w_.hscal;
    return 0;
  }

  /* A restart cycle: the start (r = b - K dx, ||r||, v_0), iterations until
     the state says done (converged, broken down, or m of them), the end (the
     triangular solve and dx += Z y), then the state to the host.  Every kernel
     takes its column from the state, so what is captured once serves all
     iterations, and, the tolerance and ||b|| being in the state too, every
     later cycle of the same buffers.
       one graph with a loop node around an iteration, launched and waited for
       once;
       or, for a serving worker, three graphs, the middle one kChunk iterations
       launched until the state says done: the loops of several streams hold
       each other up (24 served load steps 43.7 ms with loops, 39.5 with
       chunks; a solve alone, 64 x 48: 6.5 ms with the loop, 7.0 with chunks);
       or the same enqueued directly, on the legacy default stream, which
       cannot be captured. */
  static constexpr int kChunk = 3;

  void enqueue_start(const double *b, double *dx)
  {
    const int n = w_.n, m = w_.m;
    GmState *gs = w_.gs;
    if (f32_) k_bsr_resid<<<nblk(w_.nb, 8), 256, 0, st_>>>(w_.nb, dm_.rowptr, dm_.colind, (const float *)K_, dx, b, w_.w);
    else k_bsr_resid<<<nblk(w_.nb, 8), 256, 0, st_>>>(w_.nb, dm_.rowptr, dm_.colind, (const double *)K_, dx, b, w_.w);
    k_multidot<<<dim3(kDotBlocks, 1), 256, 0, st_>>>(n, 1, w_.w, (size_t)n, w_.w, w_.part);
    k_reduce_parts<<<1, 128, 0, st_>>>(1, kDotBlocks, w_.part, w_.h1);
    k_cycle_start<<<1, 32, 0, st_>>>(m, w_.h1, w_.g, gs);
    k_gs_update<<<nblk(n, 3 * kUpdNodes), 3 * kUpdNodes, 0, st_>>>(n, w_.V, w_.w, pc(), arnoldi(), gs, true);
  }

  /* check: kernels look at the state first and do nothing once it says done (a
     load that all others would wait for; the graph's loop ends with the iteration) */
  void enqueue_iteration(bool check)
  {
    const int rows = gs_rows(w_.nb), grid = gs_grid(w_.nb);
    if (f32_) precond_matvec((const float *)K_, check);
    else precond_matvec((const double *)K_, check);
    k_gs_project<<<grid, kGsThreads, 0, st_>>>(w_.nb, rows, w_.V, w_.h1, w_.part, w_.ticket, w_.h2, w_.gs, check);
    k_gs_update<<<nblk(w_.n, 3 * kUpdNodes) + 1, 3 * kUpdNodes, 0, st_>>>(w_.n, w_.V, nullptr, pc(), arnoldi(), w_.gs, check);
  }

  void enqueue_end(double *dx)
  {
    const int n = w_.n, m = w_.m;
    k_backsolve<<<1, 32, 0, st_>>>(m, w_.H, w_.g, w_.y, w_.gs);
    if (amg_) k_combine<<<nblk(n, 256), 256, 0, st_>>>(n, (const float *)w_.Z, (size_t)n, w_.y, dx, w_.gs);
    else k_combine<<<nblk(n, 256), 256, 0, st_>>>(n, w_.Z, (size_t)n, w_.y, dx, w_.gs);
    cudaMemcpyAsync(w_.hgs, w_.gs, sizeof(GmState), cudaMemcpyDeviceToHost, st_);
  }

  void enqueue_chunk()
  {
    for (int k = 0; k < kChunk; k++) enqueue_iteration(true);
    cudaMemcpyAsync(w_.hgs, w_.gs, sizeof(GmState), cudaMemcpyDeviceToHost, st_);
  }

  /* the cycle's graph: start -> while (not done) iterations -> end */
  cudaError_t capture_loop(const double *b, double *dx)
  {
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaGraphCreate(&graph, 0);
    if (e != cudaSuccess) return e;
    cudaGraphConditionalHandle loop;
    cudaGraphNodeParams np{};
    cudaGraphNode_t node = nullptr;
    std::vector<cudaGraphNode_t> tail;
    auto capture = [&](cudaGraph_t g, const std::vector<cudaGraphNode_t> &deps, auto &&enqueue) {
      cudaError_t c = cudaStreamBeginCaptureToGraph(st_, g, deps.data(), nullptr, deps.size(), cudaStreamCaptureModeThreadLocal);
      if (c != cudaSuccess) return c;
      enqueue();
      cudaStreamCaptureStatus status;
      const cudaGraphNode_t *d = nullptr;
      size_t nd = 0;
      c = cudaStreamGetCaptureInfo(st_, &status, nullptr, nullptr, &d, nullptr, &nd);
      if (c == cudaSuccess) tail.assign(d, d + nd);
      cudaGraph_t out = nullptr;
      const cudaError_t c2 = cudaStreamEndCapture(st_, &out);
      return c != cudaSuccess ? c : c2;
    };
    e = cudaGraphConditionalHandleCreate(&loop, graph, 1, cudaGraphCondAssignDefault);
    if (e == cudaSuccess)
      e = capture(graph, {}, [&] { enqueue_start(b, dx); k_gs_loop<<<1, 1, 0, st_>>>(loop, w_.gs); });
    if (e == cudaSuccess) {
      np.type = cudaGraphNodeTypeConditional;
      np.conditional.handle = loop;
      np.conditional.type = cudaGraphCondTypeWhile;
      np.conditional.size = 1;
      e = cudaGraphAddNode(&node, graph, tail.data(), nullptr, tail.size(), &np);
    }
    if (e == cudaSuccess)
      e = capture(np.conditional.phGraph_out[0], {}, [&] {
        enqueue_iteration(false);
        k_gs_loop<<<1, 1, 0, st_>>>(loop, w_.gs);
      });
    if (e == cudaSuccess) e = capture(graph, {node}, [&] { enqueue_end(dx); });
    if (e == cudaSuccess) e = instantiate(graph);
    cudaGraphDestroy(graph);
    return e;
  }

  cudaError_t instantiate(cudaGraph_t graph)
  {
    cudaGraphExec_t x = nullptr;
    const cudaError_t e = cudaGraphInstantiate(&x, graph, 0);
    if (e == cudaSuccess) w_.gexec.push_back(x);
    return e;
  }

  template <class F> cudaError_t capture_piece(F &&enqueue)
  {
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamBeginCapture(st_, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return e;
    enqueue();
    e = cudaStreamEndCapture(st_, &graph);
    if (e != cudaSuccess) return e;
    e = instantiate(graph);
    cudaGraphDestroy(graph);
    return e;
  }

  cudaError_t capture_cycle(const double *b, double *dx, size_t pieces)
  {
    for (cudaGraphExec_t g : w_.gexec) cudaGraphExecDestroy(g);
    w_.gexec.clear();
    w_.g_b = b; w_.g_dx = dx; w_.g_K = K_; w_.g_pc = amg_;
    if (pieces == 1) return capture_loop(b, dx);
    cudaError_t e = capture_piece([&] { enqueue_start(b, dx); });
    if (e == cudaSuccess) e = capture_piece([&] { enqueue_chunk(); });
    if (e == cudaSuccess) e = capture_piece([&] { enqueue_end(dx); });
    return e;
  }

  /* one cycle, and its state on the host */
  int run_cycle(const double *b, double *dx)
  {
    const bool direct = st_ == nullptr;
    const size_t pieces = t_blocking_waits ? 3 : 1;
    cudaError_t e = cudaSuccess;
    if (!direct && (w_.gexec.size() != pieces || w_.g_b != b || w_.g_dx != dx || w_.g_K != K_ || w_.g_pc != (const void *)amg_))
      e = capture_cycle(b, dx, pieces);
    if (e == cudaSuccess && !direct && pieces == 1) {
      e = cudaGraphLaunch(w_.gexec[0], st_);
    } else if (e == cudaSuccess) {
      auto piece = [&](int p) {
        if (!direct) return cudaGraphLaunch(w_.gexec[p], st_);
        if (p == 0) enqueue_start(b, dx);
        else if (p == 1) enqueue_chunk();
        else enqueue_end(dx);
        return cudaGetLastError();
      };
      e = piece(0);
      for (int j = 0; j < w_.m && e == cudaSuccess; j += kChunk) {
        e = piece(1);
        if (e == cudaSuccess) e = host_wait(st_, w_.evb);
        if (w_.hgs->done) break;
      }
      if (e == cudaSuccess) e = piece(2);
    }
    return (int)(e == cudaSuccess ? host_wait(st_, w_.evb) : e);
  }

  /* solve K dx = b from dx = 0; iterations in *its */
  int solve(const double *b, double *dx, double rtol, int maxit, int *its, double *relres)
  {
    *its = 0;
    *relres = 0.0;
    cudaMemsetAsync(dx, 0, w_.n * sizeof(double), st_);
    k_solve_begin<<<1, 32, 0, st_>>>(rtol, w_.gs);
    return resume(b, dx, rtol, maxit, its, relres);
  }

  /* the same solve, from the dx, *its and state that it was left with */
  int resume(const double *b, double *dx, double rtol, int maxit, int *its, double *relres)
  {
    int rc = 0;
    while (*its < maxit) {
      if ((rc = run_cycle(b, dx))) return rc;
      const GmState &h = *w_.hgs;
      *its += h.jdone;
      *relres = h.bnorm > 0.0 ? h.resid / h.bnorm : 0.0;
      if (h.bnorm == 0.0 || h.resid <= rtol * h.bnorm || h.jdone == 0) break;
    }
    return (int)cudaGetLastError();
  }

 private:
  AmgStart pc() const { return amg_ ? amg_start(amg_) : AmgStart{}; }
  Arnoldi arnoldi() const { return {w_.m, w_.h1, w_.h2, w_.H, w_.cs, w_.sn, w_.g}; }

  const DevMesh &dm_;
  const KParams &kp_;
  bool f32_;
  const void *K_;
  SolverWork &w_;
  AmgHier *amg_;
  cudaStream_t st_;
};

SolverWork *solver_create(int n, int nb, int m, void *stream, int *rc)
{
  SolverWork *w = new SolverWork();
  w->n = n; w->nb = nb; w->m = m;
  w->st = (cudaStream_t)stream;
  cudaError_t e = cudaSuccess;
  const size_t dn = sizeof(double) * (size_t)n;
  auto A = [&](void **p, size_t bytes) {
    if (e == cudaSuccess) e = w->mem.get(p, bytes, w->st);
  };
  A((void **)&w->V, dn * (size_t)(m + 1));
  A((void **)&w->Z, dn * (size_t)m); A((void **)&w->w, dn); A((void **)&w->dx, dn); A((void **)&w->xt, dn);
  A((void **)&w->Rt, dn); A((void **)&w->xh, dn);
  A((void **)&w->dinv, sizeof(double) * 9 * (size_t)nb);
  A((void **)&w->part, sizeof(double) * (size_t)(m + 2) * std::max(kDotBlocks, kGsBlocks));
  A((void **)&w->h1, sizeof(double) * (m + 2)); A((void **)&w->h2, sizeof(double) * (m + 2));
  A((void **)&w->H, sizeof(double) * (size_t)(m + 1) * m);
  A((void **)&w->cs, sizeof(double) * m); A((void **)&w->sn, sizeof(double) * m);
  A((void **)&w->g, sizeof(double) * (m + 1)); A((void **)&w->y, sizeof(double) * m);
  A((void **)&w->gs, sizeof(GmState));
  A((void **)&w->ticket, sizeof(unsigned));
  if (e == cudaSuccess) e = cudaMemsetAsync(w->ticket, 0, sizeof(unsigned), w->st);
  if (e == cudaSuccess) {
    w->pin = pin_acquire();
    if (!w->pin) e = cudaErrorMemoryAllocation;
    else { w->hgs = &w->pin->gs; w->hscal = &w->pin->scal; w->hstat = &w->pin->stat; }
  }
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&w->ev, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&w->evb, cudaEventDisableTiming | cudaEventBlockingSync);
  if (e == cudaSuccess) e = cudaStreamSynchronize(w->st);
  *rc = (int)e;
  if (e != cudaSuccess) { solver_destroy(w); return nullptr; }
  return w;
}

void solver_destroy(SolverWork *w)
{
  if (!w) return;
  cudaStream_t st = w->st;
  cudaStreamSynchronize(st);
  w->mem.release(st);
  cudaStreamSynchronize(st);
  if (w->ev) cudaEventDestroy(w->ev);
  if (w->evb) cudaEventDestroy(w->evb);
  for (cudaGraphExec_t g : w->gexec) cudaGraphExecDestroy(g);
  pin_release(w->pin);    /* after the graphs that write into it */
  delete w;
}

double *solver_xbuf(SolverWork *w) { return w->xh; }
int solver_m(const SolverWork *w) { return w->m; }
long long solver_device_bytes(const SolverWork *w) { return w ? (long long)w->mem.held() : 0; }

/* Newton on device data; x is a device vector (updated in place). */
int newton_device(const DevMesh &dm, const KParams &kp, bool f32, void *dK, double *dR, double *x,
                  const BiofemNewtonOptions &o, BiofemNewtonStats &s, SolverWork *wp, AmgHier *amg, cudaStream_t st,
                  ResidualFn residual, JacobianFn jacobian, void *ctx,
                  std::string &err)
{
  const int n = 3 * kp.nt, nb = kp.nt;
  SolverWork &w = *wp;
  Gmres gm(dm, kp, f32, dK, w, amg, st);
  int rc;
  auto norm = [&](const double *v, double &out) -> int {
    double d2 = 0.0;
    int r = gm.dot2(v, v, d2);
    out = std::sqrt(d2);
    return r;
  };
  /* ||R|| of the residual just evaluated, and whether every element's C33
     solve stayed in its domain (status bit 1 clear).  The word is cleared
     after reading; bit 2 (a singular diagonal block, replaced by the
     identity in the preconditioner) needs no action. */
  auto checked_norm = [&](const double *v, double &out, bool &in_domain) -> int {
    cudaMemcpyAsync(w.hstat, dm.status, sizeof(int), cudaMemcpyDeviceToHost, st);
    int r = norm(v, out);                 /* synchronises the stream */
    in_domain = (*w.hstat & 1) == 0;
    if (*w.hstat) cudaMemsetAsync(dm.status, 0, sizeof(int), st);
    return r;
  };
  s = BiofemNewtonStats();
  if ((rc = residual(ctx, x, dR, (void *)st))) { err = "residual"; return rc; }
  s.residual_evals++;
  double rn;
  bool ok = true;
  if ((rc = checked_norm(dR, rn, ok))) { err = "norm"; return rc; }
  if (!ok) { err = "CC3333 too small in the C33 solve at the initial state (ModElemC33, active_strain.c:1676)"; return 72; }
  s.r0 = rn;
  s.rhist[0] = rn;
  const double target = std::max(o.rtol * s.r0, o.atol);
  double eta = 0.3, rn_prev = rn;
  /* A Newton step that took the residual down by three orders left the tangent
     nearly as it was, and the multigrid hierarchy with it: the next step keeps
     it (a setup costs as much as six iterations: 64 x 48 310 us of 50 each,
     98,304 triangles 1.7 ms of 270).  Iterations with the last step's hierarchy
     against its own, by the residual's drop: 6e6 7 / 7, 2e4 15 / 15, 9e3 41 / 41, 100
     42 / 42, but 283 22 / 16 and 62 above 110 / 42.  A solve that needs more than
     twice the iterations that the last setup's rate promises for its tolerance,
     and a cycle, goes on from where it is with a new one.
     An FP64 handle keeps its FP32 copy of the tangent with the hierarchy; on an
     FP32 handle the finest level's operator is the tangent itself, the new one,
     with the old P and P^T A P: a fixed preconditioner all the same, and under
     this rule as good (load steps of 32 x 24 to 256 x 192 cells, fixed and
     adaptive tolerances, both precisions: the iterations of a setup every step). */
  constexpr double kKeepHierarchy = 1e-3;
  double rate = 0.0;       /* log of the residual's factor an iteration, since the last setup */
  for (int it = 0; it < o.max_newton; it++) {
    if (rn <= o.rtol * s.r0 || rn <= o.atol) { s.converged = 1; break; }
    double ksp_rtol = o.gmres_rtol;
    if (o.forcing == 1) {            /* Eisenstat-Walker, version 2 */
      const double alpha = 1.6180339887498949, gamma = 1.0;
      if (it > 0) {
        double e = gamma * std::pow(rn / rn_prev, alpha);
        const double guard = gamma * std::pow(eta, alpha);
        if (guard > 0.1) e = std::max(e, guard);
        eta = e;
      }
      eta = std::min(eta, 0.9);
      ksp_rtol = std::max(std::max(eta, o.gmres_rtol), std::min(0.9, 0.5 * target / rn));
    }
    const bool keep = amg && it > 0 && rn <= kKeepHierarchy * rn_prev;
    rn_prev = rn;
    if ((rc = jacobian(ctx, x, dR, dK, (void *)st))) { err = "jacobian"; return rc; }
    s.jacobian_evals++;
    if (amg) {
      if (!keep && (rc = amg_numeric(amg, dK, f32, st))) { err = "multigrid setup"; return rc; }
    } else if (f32) {
      k_bj_setup<float><<<nblk(nb, 256), 256, 0, st>>>(nb, dm.rowptr, dm.colind, (const float *)dK, w.dinv, dm.status);
    } else {
      k_bj_setup<double><<<nblk(nb, 256), 256, 0, st>>>(nb, dm.rowptr, dm.colind, (const double *)dK, w.dinv, dm.status);
    }
    /* rhs = -R */
    k_scale_copy<<<nblk(n, 256), 256, 0, st>>>(n, dR, -1.0, w.Rt);
    int its = 0;
    double relres = 0.0;
    int most = o.gmres_max_it;
    if (keep && rate < 0.0) most = (int)std::min((double)most, 2.0 * std::ceil(std::log(ksp_rtol) / rate) + w.m);
    if ((rc = gm.solve(w.Rt, w.dx, ksp_rtol, most, &its, &relres))) { err = "gmres"; return rc; }
    int its0 = 0;
    double relres0 = 1.0;
    bool set_up = !keep;
    if (keep && !(relres <= ksp_rtol) && its < o.gmres_max_it) {
      its0 = its;
      relres0 = relres;
      set_up = true;
      if ((rc = amg_numeric(amg, dK, f32, st))) { err = "multigrid setup"; return rc; }
      if (!std::isfinite(relres)) {          /* nothing to go on from */
        s.gmres_its_total += its;
        its0 = 0;
        relres0 = 1.0;
        rc = gm.solve(w.Rt, w.dx, ksp_rtol, o.gmres_max_it - its, &its, &relres);
      } else {
        rc = gm.resume(w.Rt, w.dx, ksp_rtol, o.gmres_max_it, &its, &relres);
      }
      if (rc) { err = "gmres"; return rc; }
    }
    if (set_up && its > its0) rate = std::log(std::max(relres / relres0, 1e-300)) / (its - its0);
    s.gmres_its_total += its;
    s.gmres_its_last = its;
    s.gmres_relres_last = relres;
    if (kp.nt > kp.nv) k_zero_ghost<<<nblk(3LL * (kp.nt - kp.nv), 256), 256, 0, st>>>(kp.nv, kp.nt, w.dx);
    /* backtracking on ||R|| */
    double alpha = 1.0, rnew = 0.0;
    for (int ls = 0; ls < 12; ls++) {
      k_scale_copy<<<nblk(n, 256), 256, 0, st>>>(n, x, 1.0, w.xt);
      k_axpby<<<nblk(n, 256), 256, 0, st>>>(n, alpha, w.dx, 1.0, w.xt);
      if ((rc = residual(ctx, w.xt, dR, (void *)st))) { err = "residual"; return rc; }
      s.residual_evals++;
      if ((rc = checked_norm(dR, rnew, ok))) { err = "norm"; return rc; }
      /* a trial state outside the C33 solve's domain is a failed step:
         shorten it, as a line search does on a function-domain error */
      if (!ok) { rnew = INFINITY; alpha *= 0.5; continue; }
      if (!o.line_search || rnew <= (1.0 - 1e-4 * alpha) * rn || !std::isfinite(rn)) break;
      alpha *= 0.5;
    }
    if (!ok) { err = "CC3333 too small in the C33 solve on every trial step (ModElemC33, active_strain.c:1676)"; return 72; }
    k_scale_copy<<<nblk(n, 256), 256, 0, st>>>(n, w.xt, 1.0, x);
    rn = rnew;
    s.newton_its++;
    if (s.newton_its < 64) s.rhist[s.newton_its] = rn;
  }
  if (rn <= o.rtol * s.r0 || rn <= o.atol) s.converged = 1;
  s.rfinal = rn;
  return (int)cudaStreamSynchronize(st);
}

} /* namespace biofem */
