/*
 * Device part of the smoothed-aggregation preconditioner (see amg.h): the
 * numeric setup from the current tangent and the FP32 V-cycle.
 *
 * Vectors on a level are node-major.  Operator-style kernels give each block
 * row to a warp (or four, on small levels), a lane a row of a block.  Every value
 * is produced by exactly one thread in a fixed order, so the preconditioner is
 * deterministic.  Given the Krylov cycle's "done" flag, the cycle's kernels do
 * nothing once it is set, so that they can be enqueued past its convergence.
 */
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <type_traits>
#include <vector>

#include "amg.h"
#include "arena.h"

namespace biofem {
namespace {

constexpr int kPowerIts = 12;
/* The power iterations whose norm is taken (the next one's iterate is divided
   by it): the last two give the estimate.  A norm is a reduction over the whole
   launch, half of a small level's time.  The iterate before a norm is divided by
   the power of two of its largest entry (an atomic a CTA), so
   that the sum of squares meets one factor of the eigenvalue, not four; the
   iterates between hold three.  That serves to 1e12, more than a nearly singular
   diagonal block gives (k_dinv takes 1e-12 of a block for zero). */
constexpr bool power_norm(int it) { return it == 3 || it == 7 || it >= kPowerIts - 2; }
constexpr bool power_largest(int it) { return !power_norm(it) && power_norm(it + 1); }
constexpr int kPowerBlocks = 912;    /* 6 x 152 SMs; the norm's partial sums */

inline int nblk(long long n, int bs) { return (int)((n + bs - 1) / bs); }

struct LevelPar {        /* device, per level */
  float lambda, theta_inv, c1, c2, omega;
};

/* ---------------- small dense helpers ---------------- */
/* Node vectors that are gathered (x and d of a level, the power iterations'
   iterates) hold four floats a node where a node has three values, so that a
   node is one 16-byte load. */
template <int BS> constexpr int kStride = BS == 3 ? 4 : BS;

template <int BS> __device__ __forceinline__ void load_node(const float *x, int c, float v[BS])
{
  if constexpr (BS == 3) {
    const float4 w = *reinterpret_cast<const float4 *>(x + 4 * (size_t)c);
    v[0] = w.x; v[1] = w.y; v[2] = w.z;
  } else {      /* 24 bytes, 8-byte aligned */
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const float2 w = reinterpret_cast<const float2 *>(x + (size_t)c * BS)[j];
      v[2 * j] = w.x; v[2 * j + 1] = w.y;
    }
  }
}

/* Rows of block vectors M x, blocks of BS x CW floats: a warp a block row, lane
   l on row l % BS of blocks l / BS, l / BS + kLaneBlocks, ..  Neighbouring lanes read
   neighbouring 12 or 24 bytes, and a lane asks for kBatch blocks and their columns
   before it uses one: the loads in flight bound these kernels, not their number. */
template <int BS> constexpr int kLaneBlocks = 30 / BS;      /* 10 or 5; lanes 30 and 31 idle */
template <int BS, int CW> constexpr int kBatch = BS == 3 && CW == 3 ? 4 : 3;
constexpr int kRowCta = 8;          /* warps a CTA */

/* lane's partial sum of its row over blocks [k0, k1), shared by nw warps of
   which this is number w; get(c, xv): the CW values of column c */
template <int BS, int CW, class Get>
__device__ __forceinline__ float row_partial(const float *__restrict__ M, const int *__restrict__ col, int k0, int k1,
                                             int lane, int w, int nw, Get get)
{
  constexpr int NB = kBatch<BS, CW>;
  float v = 0.f;
  if (lane >= BS * kLaneBlocks<BS>) return v;
  const int LB = kLaneBlocks<BS> * nw;
  const float *row = M + (size_t)(lane % BS) * CW;
  for (int k = k0 + kLaneBlocks<BS> * w + lane / BS; k < k1; k += NB * LB) {
    float m[NB][CW], xv[NB][CW];
    int c[NB];
#pragma unroll
    for (int b = 0; b < NB; b++) {
      const int kk = k + b * LB;
      c[b] = kk < k1 ? __ldg(col + kk) : -1;
      if constexpr (CW == 6) {      /* 24 bytes, 8-byte aligned */
#pragma unroll
        for (int j = 0; j < 3; j++) {
          const float2 w = kk < k1 ? __ldg(reinterpret_cast<const float2 *>(row + (size_t)kk * BS * CW) + j) : make_float2(0.f, 0.f);
          m[b][2 * j] = w.x; m[b][2 * j + 1] = w.y;
        }
      } else {
#pragma unroll
        for (int j = 0; j < CW; j++) m[b][j] = kk < k1 ? __ldg(row + (size_t)kk * BS * CW + j) : 0.f;
      }
    }
#pragma unroll
    for (int b = 0; b < NB; b++) {
#pragma unroll
      for (int j = 0; j < CW; j++) xv[b][j] = 0.f;
      if (c[b] >= 0) get(c[b], xv[b]);
    }
#pragma unroll
    for (int b = 0; b < NB; b++)
#pragma unroll
      for (int j = 0; j < CW; j++) v = fmaf(m[b][j], xv[b][j], v);
  }
  return v;
}

/* the lanes' sums by row, in lanes 0 .. BS - 1 (every lane calls) */
template <int BS> __device__ __forceinline__ float row_sum(float v)
{
  if constexpr (BS == 3) v += __shfl_down_sync(0xffffffffu, v, 15);
  const float a = __shfl_down_sync(0xffffffffu, v, BS), b = __shfl_down_sync(0xffffffffu, v, 2 * BS);
  const float c = __shfl_down_sync(0xffffffffu, v, 3 * BS), d = __shfl_down_sync(0xffffffffu, v, 4 * BS);
  return ((v + a) + (b + c)) + d;
}

/* The same over the NW warps that share the row, in all of their lanes (for
   NW > 1 every thread of the CTA calls, once) */
template <int BS, int NW> __device__ __forceinline__ void row_sums(float v, float acc[BS])
{
  v = row_sum<BS>(v);
  if constexpr (NW == 1) {
#pragma unroll
    for (int r = 0; r < BS; r++) acc[r] = __shfl_sync(0xffffffffu, v, r);
  } else {
    __shared__ float part[kRowCta][BS];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane < BS) part[wid][lane] = v;
    __syncthreads();
    const int w0 = wid / NW * NW;
#pragma unroll
    for (int r = 0; r < BS; r++) {
      acc[r] = part[w0][r];
#pragma unroll
      for (int w = 1; w < NW; w++) acc[r] += part[w0 + w][r];
    }
  }
}

/* A warp's place: row, number among the row's NW warps, lane */
template <int NW> struct RowPlace {
  int row, w, lane;
  bool live;
  __device__ __forceinline__ explicit RowPlace(int n)
  {
    const int wid = threadIdx.x >> 5;
    row = (blockIdx.x * kRowCta + wid) / NW;
    w = wid % NW;
    lane = threadIdx.x & 31;
    live = row < n;
    if (!live) row = n - 1;          /* takes part in the CTA's barrier */
  }
};

/* acc[BS] = row of A x, in every lane of the row's warps */
template <int BS, int NW>
__device__ __forceinline__ void row_apply(const int *__restrict__ rowptr, const int *__restrict__ colind,
                                          const float *__restrict__ A, const float *__restrict__ x, const RowPlace<NW> &at,
                                          float acc[BS])
{
  row_sums<BS, NW>(row_partial<BS, BS>(A, colind, rowptr[at.row], rowptr[at.row + 1], at.lane, at.w, NW,
                                       [x](int c, float xv[BS]) { load_node<BS>(x, c, xv); }), acc);
}

/* f(NW): four warps a row where that leaves every warp of a launch on the chip
   at once and the rows are long (the coarse levels' 6 x 6 blocks): a level of
   351 rows of 42 blocks took 5.1 us a product with a warp each */
template <int BS, class F> inline void by_warps(int n, F f)
{
  if constexpr (BS == 6) {
    if (n <= 1024) return f(std::integral_constant<int, 4>());
  }
  f(std::integral_constant<int, 1>());
}

__device__ __forceinline__ bool is_done(const int *done) { return done && *(volatile const int *)done; }

__global__ void k_to_f32(long long n, const double *__restrict__ a, float *__restrict__ b)
{
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < n) b[i] = (float)a[i];
}

/* inverse of each diagonal block by Gauss-Jordan with partial pivoting; a
   vanishing pivot leaves that unknown as identity */
template <int BS>
__global__ void k_dinv(int n, const int *__restrict__ diag, const float *__restrict__ A, float *__restrict__ Dinv,
                       unsigned *__restrict__ largest)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < kPowerIts) largest[i] = 0u;      /* the power iterations', which follow */
  if (i >= n) return;
  float a[BS][BS], v[BS][BS];
  const int k = diag[i];
  float scale = 0.f;
#pragma unroll
  for (int r = 0; r < BS; r++)
#pragma unroll
    for (int c = 0; c < BS; c++) {
      a[r][c] = k >= 0 ? A[(size_t)k * BS * BS + r * BS + c] : (r == c ? 1.f : 0.f);
      v[r][c] = r == c ? 1.f : 0.f;
      scale = fmaxf(scale, fabsf(a[r][c]));
    }
  if (!(scale > 0.f)) scale = 1.f;
#pragma unroll
  for (int p = 0; p < BS; p++) {
    int piv = p;
    float best = fabsf(a[p][p]);
#pragma unroll
    for (int r = p + 1; r < BS; r++)
      if (fabsf(a[r][p]) > best) { best = fabsf(a[r][p]); piv = r; }
    if (piv != p) {
#pragma unroll
      for (int c = 0; c < BS; c++) {
        float t = a[p][c]; a[p][c] = a[piv][c]; a[piv][c] = t;
        t = v[p][c]; v[p][c] = v[piv][c]; v[piv][c] = t;
      }
    }
    if (!(best > 1e-12f * scale)) {             /* singular direction: identity */
#pragma unroll
      for (int c = 0; c < BS; c++) { a[p][c] = c == p ? 1.f : 0.f; }
    }
    const float inv = 1.f / a[p][p];
#pragma unroll
    for (int c = 0; c < BS; c++) { a[p][c] *= inv; v[p][c] *= inv; }
#pragma unroll
    for (int r = 0; r < BS; r++) {
      if (r == p) continue;
      const float f = a[r][p];
#pragma unroll
      for (int c = 0; c < BS; c++) { a[r][c] = fmaf(-f, a[p][c], a[r][c]); v[r][c] = fmaf(-f, v[p][c], v[r][c]); }
    }
  }
  float *o = Dinv + (size_t)i * BS * BS;
#pragma unroll
  for (int r = 0; r < BS; r++)
#pragma unroll
    for (int c = 0; c < BS; c++) o[r * BS + c] = v[r][c];
}

/* 1 / 2^floor(log2 v) of a positive float's bits; 1 for zero, infinity and NaN */
__device__ __forceinline__ float inverse_power_of_two(unsigned v)
{
  const unsigned f = v >> 23;
  return f == 0u || f == 255u ? 1.f : __uint_as_float((254u - min(f, 253u)) << 23);
}

/* one power-iteration step on D^-1 A: y = D^-1 A x over the last norm (s_prev), or
   the power of two of the last step's largest entry (big_prev); x = a fixed
   pseudo-random vector on the first step.  Then ||y|| into norm_out via a
   fixed-order last-block reduction, or y's largest entry into big_out. */
__device__ __forceinline__ float start_vec(unsigned i)
{
  unsigned h = i * 2654435761u;
  h ^= h >> 15; h *= 2246822519u; h ^= h >> 13;
  return (float)(h & 0xffffu) * (1.f / 32768.f) - 1.f;
}

template <int BS, int NW>
__global__ void __launch_bounds__(256) k_power(int n, const int *__restrict__ rowptr, const int *__restrict__ colind,
                                               const float *__restrict__ A, const float *__restrict__ Dinv,
                                               const float *__restrict__ x, const float *__restrict__ s_prev,
                                               const unsigned *__restrict__ big_prev, float *__restrict__ y,
                                               float *__restrict__ part, unsigned *__restrict__ ticket,
                                               float *__restrict__ norm_out, unsigned *__restrict__ big_out)
{
  __shared__ float red[8];
  __shared__ int last;
  const int lane = threadIdx.x & 31;
  const float s = s_prev ? 1.f / fmaxf(*s_prev, 1e-30f) : big_prev ? inverse_power_of_two(*big_prev) : 1.f;
  float local = 0.f;
  unsigned big = 0u;
  for (int r0 = 0; r0 < n; r0 += kRowCta / NW * gridDim.x) {     /* one turn where NW > 1 (host) */
    RowPlace<NW> at(n - r0);
    const int row = r0 + at.row;
    const auto start = [](int c, float xv[BS]) {
#pragma unroll
      for (int t = 0; t < BS; t++) xv[t] = start_vec((unsigned)(c * BS + t));
    };
    const auto from = [x](int c, float xv[BS]) { load_node<BS>(x, c, xv); };
    float acc[BS];
    const int k0 = rowptr[row], k1 = rowptr[row + 1];
    row_sums<BS, NW>(x ? row_partial<BS, BS>(A, colind, k0, k1, lane, at.w, NW, from)
                       : row_partial<BS, BS>(A, colind, k0, k1, lane, at.w, NW, start), acc);
    if (at.live && at.w == 0 && lane < BS) {
      const float *D = Dinv + ((size_t)row * BS + lane) * BS;
      float v = 0.f;
#pragma unroll
      for (int c = 0; c < BS; c++) v = fmaf(D[c], acc[c], v);
      v *= s;
      y[(size_t)row * kStride<BS> + lane] = v;
      local = fmaf(v, v, local);
      big = max(big, __float_as_uint(fabsf(v)));
    }
  }
  if (!norm_out) {
    if (big_out) {
      __shared__ unsigned most[8];
      big = __reduce_max_sync(0xffffffffu, big);
      if (lane == 0) most[threadIdx.x >> 5] = big;
      __syncthreads();
      if (threadIdx.x < 8) {
        big = __reduce_max_sync(0xffu, most[threadIdx.x]);
        if (threadIdx.x == 0) atomicMax(big_out, big);
      }
    }
    return;
  }
  for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
  if (lane == 0) red[threadIdx.x >> 5] = local;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
    part[blockIdx.x] = t;
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  if (threadIdx.x < 32) {
    float t = 0.f;
    for (int p = threadIdx.x; p < (int)gridDim.x; p += 32) t += __ldcg(part + p);
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (threadIdx.x == 0) { *norm_out = sqrtf(t); *ticket = 0u; }
  }
}

/* Chebyshev interval [lambda/30, 1.1 lambda] for degree 2, and the
   prolongator damping omega = 4 / (3 lambda) */
__global__ void k_level_params(const float *__restrict__ lam_in, LevelPar *__restrict__ par)
{
  if (threadIdx.x != 0) return;
  const float lam = fmaxf(*lam_in, 1e-20f);
  const float hi = 1.1f * lam, lo = lam / 30.f;
  const float theta = 0.5f * (hi + lo), delta = 0.5f * (hi - lo), sigma = theta / delta;
  const float rho0 = 1.f / sigma, rho1 = 1.f / (2.f * sigma - rho0);
  par->lambda = lam;
  par->theta_inv = 1.f / theta;
  par->c1 = rho1 * rho0;
  par->c2 = 2.f * rho1 / delta;
  par->omega = 4.f / (3.f * lam);
}

/* Block rows of P, T = A P and Ac = P^T T.  A warp walks the block products of
   an output row (or of its share of one), adding each into the row's
   accumulators in shared memory.  32 products at a time: every lane works out
   one (operand indices, target), which keeps the dependent index loads and the
   search for the target's column off the products' path.  Then up to ten
   products side by side (five of 6 x 6 results), a lane for each row of a
   result, the next step's operands loaded before this one's are used.  A step
   holds products of one operand block, whose targets differ, so one copy of the
   row serves (P: neighbouring columns may share a target, and each place in a step
   has its own copy); the order is fixed.  A row too long for shared memory is
   accumulated in place, a product at a time.
   One thread per output block, searching per operator block, was a chain of
   dependent loads (T on the second level of a 64 x 48 sheet: 170 us for 351
   rows, now 13).  On large levels the issue of loads and shuffles bounds it: a
   lane a row of a result needs about ten instructions a product, nine lanes
   with a pair or 2 x 2 of it each needed twice that (T of the
   98,304-triangle sheet 493 us). */
template <int BS> constexpr int kRowOut = BS * kAmgCoarseBs;

__device__ __forceinline__ int find_col(const int *__restrict__ col, int lo, int hi, int key)
{
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    const int v = col[mid];
    if (v == key) return mid;
    if (v < key) lo = mid + 1; else hi = mid;
  }
  return -1;
}

__device__ __forceinline__ float2 ldg2(const float *p) { return __ldg(reinterpret_cast<const float2 *>(p)); }
__device__ __forceinline__ void fma2(float2 &acc, float f, float2 v) { acc.x = fmaf(f, v.x, acc.x); acc.y = fmaf(f, v.y, acc.y); }

/* For k in [k0, k1), in order: outer(k, a, p, c) gives an operand block a and
   the range [p, p + c) of the others, whose columns col[..] are looked up in
   the row's sorted cols[0, n); for each that is there, by lane group
   0 .. width - 1 of a step, ops.load(a, p) and, a step later (the next operands are
   on their way meanwhile), ops.add(its place among the accumulators). */
template <bool COPIES, class Ops, class Outer>
__device__ __forceinline__ void walk_products(int k0, int k1, int lane, int width, const int *__restrict__ col,
                                              const int *__restrict__ cols, int n, Outer outer, Ops ops)
{
  const int grp = lane / Ops::kLanes;
  for (int kb = k0; kb < k1; kb += 32) {
    int a = 0, p = 0, cnt = 0;
    if (kb + lane < k1) outer(kb + lane, a, p, cnt);
    int incl = cnt;                                /* products up to and with lane's */
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    for (int base = 0; base < total; base += 32) {
      const int idx = base + lane;
      int own = 0;                                 /* the lane whose range holds product idx */
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        if (__shfl_sync(0xffffffffu, incl, own + o - 1) <= idx) own += o;
      const int before = __shfl_sync(0xffffffffu, incl - cnt, own);
      const int ma = __shfl_sync(0xffffffffu, a, own), mp = __shfl_sync(0xffffffffu, p, own) + idx - before;
      const int at = idx < total ? find_col(cols, 0, n, __ldg(col + mp)) : -1;
      /* bit m: product m starts another operand block (or is past the end) */
      unsigned starts = 0u;
      if constexpr (!COPIES) {
        const int prev = __shfl_up_sync(0xffffffffu, own, 1);
        starts = __ballot_sync(0xffffffffu, lane == 0 || own != prev || idx >= total);
      }
      const int nm = min(32, total - base);
      int m0 = 0, len = 0, xt = -1;
      auto fetch = [&]() {                         /* the step at m0: its operands and targets */
        const int m = (m0 + grp) & 31;
        const int xa = __shfl_sync(0xffffffffu, ma, m), xp = __shfl_sync(0xffffffffu, mp, m);
        xt = __shfl_sync(0xffffffffu, at, m);
        const int run = COPIES ? 0 : __ffs((starts >> m0) >> 1);      /* to the next start; 0: none */
        len = min(run ? run : nm - m0, width);
        if (grp >= len) xt = -1;
        if (xt >= 0) ops.load(xa, xp);
      };
      fetch();
      while (m0 < nm) {
        const Ops now = ops;
        const int to = xt;
        m0 += len;
        if (m0 < nm) fetch();
        if (to >= 0) now.add(to);
        __syncwarp();
      }
    }
  }
}

/* acc (BS x 6) += A (BS x BS) Q (BS x 6), lane r of BS on row r */
template <int BS> struct RowProduct {
  static constexpr int C = kAmgCoarseBs, kLanes = BS, kWidth = 30 / BS;
  const float *A, *Q;
  float *acc;
  float av[BS];
  float2 qv[BS][3];
  __device__ __forceinline__ RowProduct(const float *a, const float *q, float *out, int lane)
      : A(a + lane % BS * BS), Q(q), acc(out + lane % BS * C) {}
  __device__ __forceinline__ void load(int a, int q)
  {
    const float *ap = A + (size_t)a * (BS * BS), *qp = Q + (size_t)q * (BS * C);
    if constexpr (BS == 6) {
#pragma unroll
      for (int s = 0; s < 3; s++) {
        const float2 w = ldg2(ap + 2 * s);
        av[2 * s] = w.x; av[2 * s + 1] = w.y;
      }
    } else {
#pragma unroll
      for (int s = 0; s < BS; s++) av[s] = __ldg(ap + s);
    }
#pragma unroll
    for (int s = 0; s < BS; s++)
#pragma unroll
      for (int c = 0; c < 3; c++) qv[s][c] = ldg2(qp + s * C + 2 * c);
  }
  __device__ __forceinline__ void add(int at) const
  {
    float2 *o = reinterpret_cast<float2 *>(acc + at * (BS * C));
#pragma unroll
    for (int c = 0; c < 3; c++) {
      float2 v = o[c];
#pragma unroll
      for (int s = 0; s < BS; s++) fma2(v, av[s], qv[s][c]);
      o[c] = v;
    }
  }
};

/* acc (6 x 6) += P^T (6 x BS) T (BS x 6), lane r of 6 on row r */
template <int BS> struct ColProduct {
  static constexpr int C = kAmgCoarseBs, kLanes = C, kWidth = 30 / C;
  const float *P, *T;
  float *acc;
  float pv[BS];
  float2 tv[BS][3];
  __device__ __forceinline__ ColProduct(const float *p, const float *t, float *out, int lane)
      : P(p + lane % C), T(t), acc(out + lane % C * C) {}
  __device__ __forceinline__ void load(int p, int t)
  {
    const float *pp = P + (size_t)p * (BS * C), *tp = T + (size_t)t * (BS * C);
#pragma unroll
    for (int s = 0; s < BS; s++) {
      pv[s] = __ldg(pp + s * C);
#pragma unroll
      for (int c = 0; c < 3; c++) tv[s][c] = ldg2(tp + s * C + 2 * c);
    }
  }
  __device__ __forceinline__ void add(int at) const
  {
    float2 *o = reinterpret_cast<float2 *>(acc + at * (C * C));
#pragma unroll
    for (int c = 0; c < 3; c++) {
      float2 v = o[c];
#pragma unroll
      for (int s = 0; s < BS; s++) fma2(v, pv[s], tv[s][c]);
      o[c] = v;
    }
  }
};

/* The warps of a CTA and their rows: nw warps share a row (kProdWarps / nw rows
   a CTA), each with its share of the row's outer list [k0, k1) and its own
   accumulators, ncopies of `maxsize` floats in shared memory; with maxsize 0 one
   warp a row, and the output itself (out(row)).  The copies' sum: total(t). */
constexpr int kProdWarps = 8, kProdCopies = 4;
struct ProdRow {
  float *first, *acc;        /* the row's copies, this warp's */
  int row, w, nw, lane, k0, k1, size, copies;
  bool live;
  template <class Out>
  __device__ __forceinline__ ProdRow(float *smem, int n, int nwarps, int maxsize, int ncopies, const int *__restrict__ ptr,
                                     Out out)
  {
    const int wid = threadIdx.x >> 5;
    lane = threadIdx.x & 31;
    nw = nwarps; size = maxsize; copies = maxsize ? ncopies : 1;
    row = (blockIdx.x * (blockDim.x >> 5) + wid) / nw;
    w = wid % nw;
    live = row < n;
    k0 = k1 = 0;
    if (live) {
      const int p0 = ptr[row], cnt = ptr[row + 1] - p0, share = (cnt + nw - 1) / nw;
      k0 = p0 + min(w * share, cnt);
      k1 = p0 + min((w + 1) * share, cnt);
    }
    first = size ? smem + (size_t)(wid - w) * copies * size : live ? out(row) : nullptr;
    acc = first + (size_t)w * copies * size;
  }
  __device__ __forceinline__ void clear(int values) const
  {
    for (int c = 0; c < copies; c++)
      for (int t = lane; t < values; t += 32) acc[c * size + t] = 0.f;
    __syncwarp();
  }
  __device__ __forceinline__ float total(int t) const
  {
    float v = first[t];
    for (int k = 1; k < nw * copies; k++) v += first[k * size + t];
    return v;
  }
};

/* P_iJ = [agg(i) = J] Q_i - omega D_i^-1 sum_{j in row i, agg(j) = J} A_ij Q_j */
template <int BS>
__global__ void __launch_bounds__(32 * kProdWarps) k_pvals(int n, int nw, const int *__restrict__ prow, const int *__restrict__ pcol,
                                                           const int *__restrict__ rowptr, const int *__restrict__ colind,
                                                           const float *__restrict__ A, const float *__restrict__ Dinv,
                                                           const int *__restrict__ agg, const float *__restrict__ Q,
                                                           const LevelPar *__restrict__ par, float *P, int maxsize)
{
  extern __shared__ __align__(16) float row_acc[];
  constexpr int C = kAmgCoarseBs, O = kRowOut<BS>;
  const ProdRow R(row_acc, n, nw, maxsize, kProdCopies, rowptr, [&](int i) { return P + (size_t)prow[i] * O; });
  const int p0 = R.live ? prow[R.row] : 0, np = R.live ? prow[R.row + 1] - p0 : 0;
  if (np) {
    R.clear(np * O);
    walk_products<true>(R.k0, R.k1, R.lane, R.copies, agg, pcol + p0, np,
                        [&](int k, int &a, int &p, int &cnt) { a = k; p = colind[k]; cnt = agg[p] >= 0; },
                        RowProduct<BS>(A, Q, R.acc + min(R.lane / BS, R.copies - 1) * R.size, R.lane));
  }
  __syncthreads();
  if (!np) return;
  const float om = par->omega;
  const float *d = Dinv + (size_t)R.row * BS * BS, *qi = Q + (size_t)R.row * O;
  const int own = agg[R.row];
  for (int b = R.w; b < np; b += nw) {
    const bool mine = pcol[p0 + b] == own;
    float v[(O + 31) / 32];
#pragma unroll
    for (int g = 0; g < (O + 31) / 32; g++) {
      const int o = R.lane + 32 * g, r = o / C, c = o - C * r;
      v[g] = 0.f;
      if (o < O)
#pragma unroll
        for (int s = 0; s < BS; s++) v[g] = fmaf(d[r * BS + s], R.total(b * O + s * C + c), v[g]);
    }
    __syncwarp();                     /* the accumulators may be P itself */
#pragma unroll
    for (int g = 0; g < (O + 31) / 32; g++) {
      const int o = R.lane + 32 * g;
      if (o < O) P[(size_t)(p0 + b) * O + o] = (mine ? qi[o] : 0.f) - om * v[g];
    }
  }
}

/* T_iJ = sum_k A_ik P_kJ */
template <int BS>
__global__ void __launch_bounds__(32 * kProdWarps) k_tvals(int n, int nw, const int *__restrict__ trow, const int *__restrict__ tcol,
                                                           const int *__restrict__ rowptr, const int *__restrict__ colind,
                                                           const float *__restrict__ A, const int *__restrict__ prow,
                                                           const int *__restrict__ pcol, const float *__restrict__ P,
                                                           float *T, int maxsize)
{
  extern __shared__ __align__(16) float row_acc[];
  constexpr int O = kRowOut<BS>;
  const ProdRow R(row_acc, n, nw, maxsize, 1, rowptr, [&](int i) { return T + (size_t)trow[i] * O; });
  const int t0 = R.live ? trow[R.row] : 0, nt = R.live ? trow[R.row + 1] - t0 : 0;
  if (nt) {
    R.clear(nt * O);
    walk_products<false>(R.k0, R.k1, R.lane, maxsize ? RowProduct<BS>::kWidth : 1, pcol, tcol + t0, nt,
                         [&](int k, int &a, int &p, int &cnt) { const int j = colind[k]; a = k; p = prow[j]; cnt = prow[j + 1] - p; },
                         RowProduct<BS>(A, P, R.acc, R.lane));
  }
  __syncthreads();
  if (maxsize)
    for (int t = R.lane + 32 * R.w; t < nt * O; t += 32 * nw) T[(size_t)t0 * O + t] = R.total(t);
}

/* Ac_IJ = sum_{i in P^T row I} P_iI^T T_iJ, plus 1 on the diagonal of dead coarse unknowns */
template <int BS>
__global__ void __launch_bounds__(32 * kProdWarps) k_cvals(int na, int nw, const int *__restrict__ crow, const int *__restrict__ ccol,
                                                           const int *__restrict__ rrow, const int *__restrict__ rcol,
                                                           const int *__restrict__ rmap, const float *__restrict__ P,
                                                           const int *__restrict__ trow, const int *__restrict__ tcol,
                                                           const float *__restrict__ T, const unsigned char *__restrict__ dead,
                                                           float *Ac, int maxsize)
{
  extern __shared__ __align__(16) float row_acc[];
  constexpr int C = kAmgCoarseBs, O = C * C;
  const ProdRow R(row_acc, na, nw, maxsize, 1, rrow, [&](int I) { return Ac + (size_t)crow[I] * O; });
  const int c0 = R.live ? crow[R.row] : 0, nc = R.live ? crow[R.row + 1] - c0 : 0;
  if (nc) {
    R.clear(nc * O);
    walk_products<false>(R.k0, R.k1, R.lane, maxsize ? ColProduct<BS>::kWidth : 1, tcol, ccol + c0, nc,
                         [&](int k, int &a, int &p, int &cnt) { const int i = rcol[k]; a = rmap[k]; p = trow[i]; cnt = trow[i + 1] - p; },
                         ColProduct<BS>(P, T, R.acc, R.lane));
  }
  __syncthreads();
  for (int t = R.lane + 32 * R.w; t < nc * O; t += 32 * nw) {
    float v = R.total(t);
    const int b = t / O, o = t - O * b;
    if (o % (C + 1) == 0 && ccol[c0 + b] == R.row && dead[(size_t)R.row * C + o / (C + 1)]) v += 1.f;
    Ac[(size_t)c0 * O + t] = v;
  }
}

/* The coarsest operator as a dense N x N matrix in shared memory and its
   in-place Gauss-Jordan inverse with partial pivoting (one block,
   N <= kAmgMaxDense); a vanishing pivot is replaced by 1.  Three barriers a
   pivot: the pivot row (one warp searches its column), its scaled copy, the
   other rows, a warp each, the two exchanged rows in the same warp. */
template <int BS>
__global__ void __launch_bounds__(1024) k_dense_invert(int n, const int *__restrict__ rowptr, const int *__restrict__ colind,
                                                       const float *__restrict__ A, float *__restrict__ D)
{
  extern __shared__ float sm[];
  const int N = n * BS, lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  float *a = sm;                       /* N*N */
  float *prow = sm + N * N;            /* max(N, 32): the scaled pivot row */
  __shared__ int perm[kAmgMaxDense];
  __shared__ int piv_s;
  __shared__ float scale_s;
  for (int t = threadIdx.x; t < N * N; t += blockDim.x) a[t] = 0.f;
  __syncthreads();
  float s = 0.f;
  for (int i = wid; i < n; i += nw) {
    const int k0 = rowptr[i] * BS * BS, k1 = rowptr[i + 1] * BS * BS;
    for (int t = k0 + lane; t < k1; t += 32) {
      const int k = t / (BS * BS), o = t - BS * BS * k, r = o / BS, c = o - BS * r;
      const float v = A[t];
      a[(i * BS + r) * N + colind[k] * BS + c] = v;
      s = fmaxf(s, fabsf(v));
    }
  }
  for (int o = 16; o > 0; o >>= 1) s = fmaxf(s, __shfl_xor_sync(0xffffffffu, s, o));
  if (lane == 0) prow[wid] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < nw; w++) s = fmaxf(s, prow[w]);
    scale_s = s > 0.f ? s : 1.f;
  }
  for (int k = 0; k < N; k++) {
    __syncthreads();
    if (wid == 0) {
      /* the largest |a_rk|, r >= k, the smallest r of equal ones */
      unsigned best = 0u;
      int p = k;
      for (int r = k + lane; r < N; r += 32) {
        const unsigned v = __float_as_uint(fabsf(a[r * N + k]));
        if (v > best) { best = v; p = r; }
      }
      const unsigned top = __reduce_max_sync(0xffffffffu, best);
      p = __reduce_min_sync(0xffffffffu, best == top ? p : N);
      if (lane == 0) { perm[k] = p; piv_s = p; }
    }
    __syncthreads();
    const int p = piv_s;
    float pv = a[p * N + k];
    if (!(fabsf(pv) > 1e-12f * scale_s)) pv = 1.f;
    const float inv = 1.f / pv;
    for (int c = threadIdx.x; c < N; c += blockDim.x) prow[c] = (c == k ? 1.f : a[p * N + c]) * inv;
    __syncthreads();
    for (int r = wid; r < N; r += nw) {
      if (r == k && r != p) continue;                /* written with row p below */
      if (r == p) {
        const float f = a[k * N + k];                /* row k moves to p, the scaled pivot row to k */
        __syncwarp();
        for (int c = lane; c < N; c += 32) {
          if (p != k) a[p * N + c] = fmaf(-f, prow[c], c == k ? 0.f : a[k * N + c]);
          a[k * N + c] = prow[c];
        }
      } else {
        const float f = a[r * N + k];
        __syncwarp();
        for (int c = lane; c < N; c += 32) a[r * N + c] = fmaf(-f, prow[c], c == k ? 0.f : a[r * N + c]);
      }
    }
  }
  __syncthreads();
  for (int k = N - 1; k >= 0; k--) {
    const int p = perm[k];
    if (p != k)
      for (int r = threadIdx.x; r < N; r += blockDim.x) {
        const float t = a[r * N + k]; a[r * N + k] = a[r * N + p]; a[r * N + p] = t;
      }
    __syncthreads();
  }
  /* transposed, for k_dense_apply */
  for (int t = threadIdx.x; t < N * N; t += blockDim.x) D[t] = a[(t % N) * N + t / N];
}

/* ---------------- V-cycle kernels ---------------- */
/* One level of the cycle is five launches.  Down: the Chebyshev start
   r = D^-1 b, d = r / theta comes with b from whoever writes it (the Krylov
   update on level 0, the restriction below), k_sm_step finishes the smoothing,
   k_resid leaves res = b - A x, k_restrict its restriction.  Up: the residual
   after the coarse correction is res - T xc with T = A P, which the Galerkin
   product keeps, so k_post_start adds P xc to x and starts the smoothing in one
   launch, or k_prolong and k_sm_start do without T (kCycleL2); k_sm_step
   finishes.
   On a 64 x 48 sheet every kernel is a chain of three dependent loads (row,
   column, value): 3.1 to 4.3 us each.  On 98,304 triangles the loads in flight
   bound them: a product with K (65 MB) takes 14 to 17 us from L2, 10 being the
   DRAM rate's. */

/* Level 0 takes T in only while the cycle's operators stay in L2 (126 MB) with
   it, beside K's copy and the vectors; coarse levels, whose T is a fraction of A,
   always.  98,304 triangles (A 65 MB, T 71, P 27): a solve of 165 iterations 46.9
   ms with T, 45.3 without, every kernel of level 0 slower for the lines T
   displaces; 64 x 48: 4.3 us in one launch, 5.8 in two. */
constexpr long long kCycleL2 = 96 << 20;

/* r = D^-1 b and d = r / theta of one node, lane s < BS its component s */
template <int BS>
__device__ __forceinline__ void cheb_start(const float *__restrict__ Dinv, int i, int s, const float b[BS], float ti,
                                           float *__restrict__ r, float *__restrict__ d)
{
  const float *D = Dinv + ((size_t)i * BS + s) * BS;
  float v = 0.f;
#pragma unroll
  for (int c = 0; c < BS; c++) v = fmaf(D[c], b[c], v);
  r[(size_t)i * BS + s] = v;
  d[(size_t)i * kStride<BS> + s] = v * ti;
}

/* smoothing start from x: r = D^-1 (b - A x), d = r / theta */
template <int BS, int NW>
__global__ void __launch_bounds__(32 * kRowCta) k_sm_start(int n, const int *__restrict__ rowptr, const int *__restrict__ colind,
                                                  const float *__restrict__ A, const float *__restrict__ Dinv,
                                                  const float *__restrict__ b, const float *__restrict__ x,
                                                  float *__restrict__ r, float *__restrict__ d,
                                                  const LevelPar *__restrict__ par, const int *done)
{
  const RowPlace<NW> at(n);
  if (is_done(done) || (NW == 1 && !at.live)) return;
  const int row = at.row, lane = at.lane;
  float acc[BS];
  row_apply<BS, NW>(rowptr, colind, A, x, at, acc);
  if (lane >= BS || at.w || !at.live) return;
#pragma unroll
  for (int s = 0; s < BS; s++) acc[s] = b[(size_t)row * BS + s] - acc[s];
  cheb_start<BS>(Dinv, row, lane, acc, par->theta_inv, r, d);
}

/* second Chebyshev step: r1 = r - D^-1 A d, d1 = c1 d + c2 r1,
   x = (init ? 0 : x) + d + d1; lane s < BS of the row's warp finishes
   component s */
template <int BS, int NW>
__global__ void __launch_bounds__(32 * kRowCta) k_sm_step(int n, const int *__restrict__ rowptr, const int *__restrict__ colind,
                                                 const float *__restrict__ A, const float *__restrict__ Dinv,
                                                 const float *__restrict__ r, const float *__restrict__ d,
                                                 float *__restrict__ x, int init, const LevelPar *__restrict__ par,
                                                 const int *done)
{
  const RowPlace<NW> at(n);
  if (is_done(done) || (NW == 1 && !at.live)) return;
  const int row = at.row, lane = at.lane;
  const size_t o = (size_t)row * kStride<BS> + lane;
  float D[BS], d0 = 0.f, r0 = 0.f, x0 = 0.f, c1 = 0.f, c2 = 0.f;
  const bool own = lane < BS && at.w == 0 && at.live;
  if (own) {                               /* in flight beside the row's loads */
#pragma unroll
    for (int c = 0; c < BS; c++) D[c] = __ldg(Dinv + ((size_t)row * BS + lane) * BS + c);
    d0 = d[o]; r0 = r[(size_t)row * BS + lane];
    if (!init) x0 = x[o];
    c1 = par->c1; c2 = par->c2;
  }
  float acc[BS];
  row_apply<BS, NW>(rowptr, colind, A, d, at, acc);
  if (!own) return;
  float u = 0.f;
#pragma unroll
  for (int c = 0; c < BS; c++) u = fmaf(D[c], acc[c], u);
  const float d1 = c1 * d0 + c2 * (r0 - u);
  x[o] = x0 + d0 + d1;
}

/* res = b - A x */
template <int BS, int NW>
__global__ void __launch_bounds__(32 * kRowCta) k_resid(int n, const int *__restrict__ rowptr, const int *__restrict__ colind,
                                               const float *__restrict__ A, const float *__restrict__ b,
                                               const float *__restrict__ x, float *__restrict__ res, const int *done)
{
  const RowPlace<NW> at(n);
  if (is_done(done) || (NW == 1 && !at.live)) return;
  const int row = at.row, lane = at.lane;
  const bool own = lane < BS && at.w == 0 && at.live;
  const float b0 = own ? b[(size_t)row * BS + lane] : 0.f;
  float acc[BS];
  row_apply<BS, NW>(rowptr, colind, A, x, at, acc);
  if (!own) return;
  float v = acc[0];
#pragma unroll
  for (int s = 1; s < BS; s++) if (lane == s) v = acc[s];
  res[(size_t)row * BS + lane] = b0 - v;
}

/* bc_I = sum_{i in P^T row I} P_iI^T res_i: NW warps per coarse node, three
   lanes a block of P with two columns each, ten blocks a warp at a time, four
   of a lane's asked for together, the warps' sums added in order; then, unless
   the coarse level is solved densely (Dinv null), its smoothing start.  A CTA a
   node for few nodes (their rows are hundreds of blocks long there), four warps
   up to half the chip's. */
constexpr int kRestrictBatch = 4;
template <int BS, int NW>
__global__ void __launch_bounds__(32 * (NW > 4 ? NW : 4)) k_restrict(
    int na, const int *__restrict__ rrow, const int *__restrict__ rcol, const int *__restrict__ rmap,
    const float *__restrict__ P, const float *__restrict__ res, float *__restrict__ bc, const float *__restrict__ Dinv,
    float *__restrict__ rc, float *__restrict__ dc, const LevelPar *__restrict__ par, const int *done)
{
  if (is_done(done)) return;
  constexpr int C = kAmgCoarseBs, NB = kRestrictBatch;
  __shared__ float part[NW > 4 ? NW : 4][C];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int I = (blockIdx.x * (blockDim.x >> 5) + wid) / NW;
  float2 acc = make_float2(0.f, 0.f);
  if (I < na && lane < 30) {
    const int t1 = rrow[I + 1], c = 2 * (lane % 3);
    for (int t = rrow[I] + 10 * (wid % NW) + lane / 3; t < t1; t += 10 * NW * NB) {
      int ip[NB], ir[NB];
      float2 p[NB][BS];
      float rv[NB][BS];
#pragma unroll
      for (int b = 0; b < NB; b++) {
        const int tt = t + 10 * NW * b;
        ip[b] = tt < t1 ? __ldg(rmap + tt) : -1;
        ir[b] = tt < t1 ? __ldg(rcol + tt) : 0;
      }
#pragma unroll
      for (int b = 0; b < NB; b++)
#pragma unroll
        for (int s = 0; s < BS; s++) {
          p[b][s] = ip[b] >= 0 ? ldg2(P + (size_t)ip[b] * BS * C + s * C + c) : make_float2(0.f, 0.f);
          rv[b][s] = ip[b] >= 0 ? res[(size_t)ir[b] * BS + s] : 0.f;
        }
#pragma unroll
      for (int b = 0; b < NB; b++)
#pragma unroll
        for (int s = 0; s < BS; s++) fma2(acc, rv[b][s], p[b][s]);
    }
  }
  acc.x = row_sum<3>(acc.x);
  acc.y = row_sum<3>(acc.y);
  if constexpr (NW > 1) {
    if (lane < 3) { part[wid][2 * lane] = acc.x; part[wid][2 * lane + 1] = acc.y; }
    __syncthreads();
    if (wid % NW) return;
    if (lane < 3)
#pragma unroll
      for (int w = 1; w < NW; w++) { acc.x += part[wid + w][2 * lane]; acc.y += part[wid + w][2 * lane + 1]; }
  }
  float v[C];
#pragma unroll
  for (int c = 0; c < C; c++) v[c] = __shfl_sync(0xffffffffu, c % 2 ? acc.y : acc.x, c / 2);
  if (lane >= C || I >= na) return;
  float mine = v[0];
#pragma unroll
  for (int c = 1; c < C; c++) if (lane == c) mine = v[c];
  bc[(size_t)I * C + lane] = mine;
  if (Dinv) cheb_start<C>(Dinv, I, lane, v, par->theta_inv, rc, dc);
}

/* after the coarse solve: x_i += sum_J P_iJ xc_J, then the smoothing start
   r = D^-1 (res - T xc), d = r / theta */
template <int BS, int NW>
__global__ void __launch_bounds__(32 * kRowCta) k_post_start(int n, const int *__restrict__ trow, const int *__restrict__ tcol,
                                                    const float *__restrict__ T, const int *__restrict__ prow,
                                                    const int *__restrict__ pcol, const float *__restrict__ P,
                                                    const float *__restrict__ xc, const float *__restrict__ res,
                                                    const float *__restrict__ Dinv, float *__restrict__ x,
                                                    float *__restrict__ r, float *__restrict__ d,
                                                    const LevelPar *__restrict__ par, const int *done)
{
  const RowPlace<NW> at(n);
  if (is_done(done) || (NW == 1 && !at.live)) return;
  const int row = at.row, lane = at.lane;
  constexpr int C = kAmgCoarseBs;
  auto coarse = [xc](int c, float xv[C]) { load_node<C>(xc, c, xv); };
  const int t0 = trow[row], t1 = trow[row + 1], p0 = prow[row], p1 = prow[row + 1];
  const bool own = lane < BS && at.w == 0 && at.live;
  float *xo = x + (size_t)row * kStride<BS> + lane;
  const float x0 = own ? *xo : 0.f;
  const float te = row_partial<BS, C>(T, tcol, t0, t1, lane, at.w, NW, coarse);
  /* the short rows of P in the row's last warp, whose share of T is the smallest, on its way to the first */
  float px = at.w == NW - 1 ? row_sum<BS>(row_partial<BS, C>(P, pcol, p0, p1, lane, 0, 1, coarse)) : 0.f;
  if constexpr (NW > 1) {
    __shared__ float ps[kRowCta][BS];
    if (at.w == NW - 1 && lane < BS) ps[threadIdx.x >> 5][lane] = px;
    __syncthreads();
    if (own) px = ps[(threadIdx.x >> 5) + NW - 1][lane];
  }
  float e[BS];
  row_sums<BS, NW>(te, e);
  if (!own) return;
  *xo = x0 + px;
#pragma unroll
  for (int s = 0; s < BS; s++) e[s] = res[(size_t)row * BS + s] - e[s];
  cheb_start<BS>(Dinv, row, lane, e, par->theta_inv, r, d);
}

/* x_i += sum_J P_iJ xc_J (then k_sm_start, where T is too large for k_post_start) */
template <int BS>
__global__ void __launch_bounds__(32 * kRowCta) k_prolong(int n, const int *__restrict__ prow, const int *__restrict__ pcol,
                                                          const float *__restrict__ P, const float *__restrict__ xc,
                                                          float *__restrict__ x, const int *done)
{
  const RowPlace<1> at(n);
  if (is_done(done) || !at.live) return;
  constexpr int C = kAmgCoarseBs;
  float *xo = x + (size_t)at.row * kStride<BS> + at.lane;
  const float x0 = at.lane < BS ? *xo : 0.f;
  const float v = row_sum<BS>(row_partial<BS, C>(P, pcol, prow[at.row], prow[at.row + 1], at.lane, 0, 1,
                                                 [xc](int c, float xv[C]) { load_node<C>(xc, c, xv); }));
  if (at.lane < BS) *xo = x0 + v;
}

/* x = D^-1 b for the dense coarsest inverse, stored transposed so that the
   threads of a warp read neighbouring values: one block, thread (row i, slice
   g of the columns), the slices' sums added in order.  bs: values a node of x. */
constexpr int kDenseThreads = 768;
__global__ void __launch_bounds__(kDenseThreads) k_dense_apply(int N, int bs, const float *__restrict__ Dt,
                                                               const float *__restrict__ b, float *__restrict__ x,
                                                               const int *done)
{
  if (is_done(done)) return;
  __shared__ float bv[kAmgMaxDense], part[kDenseThreads];
  for (int i = threadIdx.x; i < N; i += blockDim.x) bv[i] = b[i];
  __syncthreads();
  const int ng = kDenseThreads / N, g = threadIdx.x / N, i = threadIdx.x - g * N;
  const int len = (N + ng - 1) / ng;
  if (g < ng) {
    float s = 0.f;
    const int j1 = min(N, (g + 1) * len);
#pragma unroll 8
    for (int j = g * len; j < j1; j++) s = fmaf(Dt[(size_t)j * N + i], bv[j], s);
    part[threadIdx.x] = s;
  }
  __syncthreads();
  if (threadIdx.x < N) {
    float s = part[threadIdx.x];
    for (int k = 1; k < ng; k++) s += part[k * N + threadIdx.x];
    x[bs == 3 ? i / 3 * 4 + i % 3 : i] = s;
  }
}

}  // namespace

/* ---------------- host side ---------------- */
/* How a product kernel divides n rows whose accumulators take up to `values`
   floats: eight warps a CTA, sharing a row where there are too few rows for the
   chip, within kProdSmem; rows too long for that are accumulated in place. */
constexpr size_t kProdSmem = 96 * 1024;
struct ProdPlan {
  int nw = 1, warps = 1, size = 0, copies = 1;
  ProdPlan() = default;
  ProdPlan(int n, int values, int ncopies) : warps(kProdWarps), size(values), copies(ncopies)
  {
    while (warps > 1 && bytes() > kProdSmem) warps /= 2;
    if (bytes() > kProdSmem) size = 0;
    while (size && nw < warps && (long long)n * nw < 152 * 16) nw *= 2;
  }
  size_t bytes() const { return sizeof(float) * warps * copies * size; }
  int threads() const { return 32 * warps; }
  int grid(int n) const { return (int)(((long long)n * nw + warps - 1) / warps); }
};

struct AmgLevelDev {
  int n = 0, bs = 0, na = 0;
  long long nnzA = 0, nnzP = 0, nnzT = 0;
  bool post_by_t = true;    /* k_post_start; else k_prolong and k_sm_start (kCycleL2) */
  ProdPlan pp, pt, pc;        /* of P, T, Ac */
  const int *rowptr = nullptr, *colind = nullptr;
  int *diag = nullptr, *agg = nullptr;
  const float *A = nullptr;
  float *Aown = nullptr, *Dinv = nullptr, *Q = nullptr, *P = nullptr, *T = nullptr;
  int *prow = nullptr, *pcol = nullptr;
  int *rrow = nullptr, *rcol = nullptr, *rmap = nullptr;
  int *trow = nullptr, *tcol = nullptr;
  unsigned char *dead = nullptr;
  float *b = nullptr, *x = nullptr, *r = nullptr, *d = nullptr, *y = nullptr;
  LevelPar *par = nullptr;
  float *norms = nullptr;     /* kPowerIts power-iteration norms */
  unsigned *largest = nullptr;   /* and largest entries */
};

struct AmgHier {
  int nt = 0, nl = 0;
  AmgLevelDev L[kAmgMaxLevels];
  bool dense = false;
  int N = 0;
  float *Ad = nullptr;
  float *A0f = nullptr;      /* FP32 copy of an FP64 tangent */
  float *part = nullptr;
  unsigned *ticket = nullptr;
  Arena mem;
  cudaStream_t st = nullptr;
  cudaGraph_t num_graph = nullptr;      /* numeric setup, captured for one tangent buffer */
  cudaGraphExec_t num_exec = nullptr;
  const void *num_K = nullptr;
};

namespace {

template <class T>
int dalloc_(AmgHier *h, T **p, size_t count)
{
  *p = nullptr;
  if (count == 0) count = 1;
  cudaError_t e = h->mem.get((void **)p, count * sizeof(T), h->st);
  if (e != cudaSuccess) return (int)e;
  return 0;
}

template <class T>
int dup_(AmgHier *h, T **p, const std::vector<T> &v)
{
  int rc = dalloc_(h, p, v.size());
  if (rc || v.empty()) return rc;
  return (int)cudaMemcpyAsync(*p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, h->st);
}

template <int BS>
void numeric_level(AmgHier *h, int l, cudaStream_t st)
{
  AmgLevelDev &L = h->L[l];
  k_dinv<BS><<<nblk(L.n, 128), 128, 0, st>>>(L.n, L.diag, L.A, L.Dinv, L.largest);
  by_warps<BS>(L.n, [&](auto nw) {
    constexpr int NW = decltype(nw)::value;
    const int ctas = nblk((long long)NW * L.n, kRowCta), grid = NW > 1 ? ctas : std::min(kPowerBlocks, ctas);
    const float *s_prev = nullptr;
    const unsigned *big_prev = nullptr;
    for (int it = 0; it < kPowerIts; it++) {
      float *norm = power_norm(it) ? L.norms + it : nullptr;
      unsigned *big = power_largest(it) ? L.largest + it : nullptr;
      k_power<BS, NW><<<grid, 32 * kRowCta, 0, st>>>(L.n, L.rowptr, L.colind, L.A, L.Dinv,
                                                     it == 0 ? nullptr : (it & 1 ? L.x : L.d), s_prev, big_prev,
                                                     it & 1 ? L.d : L.x, h->part, h->ticket, norm, big);
      s_prev = norm;
      big_prev = big;
    }
  });
  k_level_params<<<1, 32, 0, st>>>(L.norms + kPowerIts - 1, L.par);
  if (l == h->nl - 1) return;
  AmgLevelDev &Cn = h->L[l + 1];
  k_pvals<BS><<<L.pp.grid(L.n), L.pp.threads(), L.pp.bytes(), st>>>(L.n, L.pp.nw, L.prow, L.pcol, L.rowptr, L.colind, L.A, L.Dinv,
                                                                    L.agg, L.Q, L.par, L.P, L.pp.size);
  k_tvals<BS><<<L.pt.grid(L.n), L.pt.threads(), L.pt.bytes(), st>>>(L.n, L.pt.nw, L.trow, L.tcol, L.rowptr, L.colind, L.A, L.prow,
                                                                    L.pcol, L.P, L.T, L.pt.size);
  k_cvals<BS><<<L.pc.grid(Cn.n), L.pc.threads(), L.pc.bytes(), st>>>(Cn.n, L.pc.nw, Cn.rowptr, Cn.colind, L.rrow, L.rcol, L.rmap,
                                                                     L.P, L.trow, L.tcol, L.T, L.dead, Cn.Aown, L.pc.size);
}

/* the smoothing start of level l from x */
template <int BS>
void smooth_start(AmgHier *h, int l, const int *done, cudaStream_t st)
{
  AmgLevelDev &L = h->L[l];
  by_warps<BS>(L.n, [&](auto nw) {
    constexpr int NW = decltype(nw)::value;
    k_sm_start<BS, NW><<<nblk((long long)NW * L.n, kRowCta), 32 * kRowCta, 0, st>>>(L.n, L.rowptr, L.colind, L.A, L.Dinv, L.b,
                                                                                    L.x, L.r, L.d, L.par, done);
  });
}

/* the second Chebyshev step of level l, from zero (init) or from x */
template <int BS>
void smooth_step(AmgHier *h, int l, int init, const int *done, cudaStream_t st)
{
  AmgLevelDev &L = h->L[l];
  by_warps<BS>(L.n, [&](auto nw) {
    constexpr int NW = decltype(nw)::value;
    k_sm_step<BS, NW><<<nblk((long long)NW * L.n, kRowCta), 32 * kRowCta, 0, st>>>(L.n, L.rowptr, L.colind, L.A, L.Dinv, L.r,
                                                                                   L.d, L.x, init, L.par, done);
  });
}

template <int BS>
void down_to_coarse(AmgHier *h, int l, const int *done, cudaStream_t st)
{
  AmgLevelDev &L = h->L[l];
  AmgLevelDev &Cn = h->L[l + 1];
  const bool dense = h->dense && l + 1 == h->nl - 1;
  smooth_step<BS>(h, l, 1, done, st);
  by_warps<BS>(L.n, [&](auto nw) {
    constexpr int NW = decltype(nw)::value;
    k_resid<BS, NW><<<nblk((long long)NW * L.n, kRowCta), 32 * kRowCta, 0, st>>>(L.n, L.rowptr, L.colind, L.A, L.b, L.x, L.y,
                                                                                 done);
  });
  auto restrict_by = [&](auto nw) {
    constexpr int NW = decltype(nw)::value;
    constexpr int warps = NW > 4 ? NW : 4;
    k_restrict<BS, NW><<<nblk((long long)NW * L.na, warps), 32 * warps, 0, st>>>(
        L.na, L.rrow, L.rcol, L.rmap, L.P, L.y, Cn.b, dense ? nullptr : Cn.Dinv, Cn.r, Cn.d, Cn.par, done);
  };
  if (L.na <= 152) restrict_by(std::integral_constant<int, 16>());
  else if (L.na <= 152 * 8) restrict_by(std::integral_constant<int, 4>());
  else restrict_by(std::integral_constant<int, 1>());
}

template <int BS>
void up_from_coarse(AmgHier *h, int l, const int *done, cudaStream_t st)
{
  AmgLevelDev &L = h->L[l];
  AmgLevelDev &Cn = h->L[l + 1];
  if (L.post_by_t) {
    by_warps<BS>(L.n, [&](auto nw) {
      constexpr int NW = decltype(nw)::value;
      k_post_start<BS, NW><<<nblk((long long)NW * L.n, kRowCta), 32 * kRowCta, 0, st>>>(
          L.n, L.trow, L.tcol, L.T, L.prow, L.pcol, L.P, Cn.x, L.y, L.Dinv, L.x, L.r, L.d, L.par, done);
    });
  } else {
    k_prolong<BS><<<nblk(L.n, kRowCta), 32 * kRowCta, 0, st>>>(L.n, L.prow, L.pcol, L.P, Cn.x, L.x, done);
    smooth_start<BS>(h, l, done, st);
  }
  smooth_step<BS>(h, l, 0, done, st);
}

}  // namespace

/* most blocks in a row of a block CSR pattern */
static int longest_row(const std::vector<int> &row)
{
  int m = 1;
  for (size_t i = 0; i + 1 < row.size(); i++) m = std::max(m, row[i + 1] - row[i]);
  return m;
}

AmgHier *amg_create(int nt, const std::vector<int> &rowptr, const std::vector<int> &colind,
                    const std::vector<unsigned char> &rowkind, const std::vector<double> &X, const int *tri, int ntri,
                    const int *d_rowptr, const int *d_colind, bool k_is_f32, cudaStream_t st, int *rc)
{
  std::vector<AmgLevelHost> H;
  const int nl = amg_symbolic(nt, rowptr, colind, rowkind, X, tri, ntri, H);
  AmgHier *h = new AmgHier();
  h->nt = nt;
  h->nl = nl;
  h->st = st;
  int e = 0;
  for (int l = 0; l < nl && !e; l++) {
    const AmgLevelHost &S = H[l];
    AmgLevelDev &L = h->L[l];
    L.n = S.n; L.bs = S.bs; L.na = (l < nl - 1) ? S.na : 0;
    L.nnzA = (long long)S.colind.size();
    if (l == 0) { L.rowptr = d_rowptr; L.colind = d_colind; }
    const size_t nv = (size_t)S.n * S.bs;
    if (!e) e = dup_(h, &L.diag, S.diag);
    if (!e) e = dalloc_(h, &L.Dinv, (size_t)S.n * S.bs * S.bs);
    if (!e) e = dalloc_(h, &L.b, nv);
    const size_t ns = (size_t)S.n * (S.bs == 3 ? kStride<3> : S.bs);
    if (!e) e = dalloc_(h, &L.x, ns);
    if (!e) e = dalloc_(h, &L.r, nv);
    if (!e) e = dalloc_(h, &L.d, ns);
    if (!e) e = dalloc_(h, &L.y, nv);
    if (!e) e = dalloc_(h, &L.par, 1);
    if (!e) e = dalloc_(h, &L.norms, kPowerIts);
    if (!e) e = dalloc_(h, &L.largest, kPowerIts);
    if (l < nl - 1) {
      L.nnzP = (long long)S.pcol.size();
      L.nnzT = (long long)S.tcol.size();
      const long long bA = 4LL * S.bs * S.bs * L.nnzA, bT = 24LL * S.bs * L.nnzT, bP = 24LL * S.bs * L.nnzP;
      L.post_by_t = 2 * bT <= bA || bA + bT + bP <= kCycleL2;
      L.pp = ProdPlan(S.n, longest_row(S.prow) * S.bs * kAmgCoarseBs, kProdCopies);
      L.pt = ProdPlan(S.n, longest_row(S.trow) * S.bs * kAmgCoarseBs, 1);
      L.pc = ProdPlan(H[l + 1].n, longest_row(H[l + 1].rowptr) * kAmgCoarseBs * kAmgCoarseBs, 1);
      if (!e) e = dup_(h, &L.agg, S.agg);
      if (!e) e = dup_(h, &L.Q, S.Q);
      if (!e) e = dup_(h, &L.prow, S.prow);
      if (!e) e = dup_(h, &L.pcol, S.pcol);
      if (!e) e = dup_(h, &L.rrow, S.rrow);
      if (!e) e = dup_(h, &L.rcol, S.rcol);
      if (!e) e = dup_(h, &L.rmap, S.rmap);
      if (!e) e = dup_(h, &L.trow, S.trow);
      if (!e) e = dup_(h, &L.tcol, S.tcol);
      if (!e) e = dup_(h, &L.dead, S.dead);
      if (!e) e = dalloc_(h, &L.P, (size_t)L.nnzP * S.bs * kAmgCoarseBs);
      if (!e) e = dalloc_(h, &L.T, (size_t)L.nnzT * S.bs * kAmgCoarseBs);
    }
    if (l > 0) {
      int *rp = nullptr, *ci = nullptr;
      if (!e) e = dup_(h, &rp, S.rowptr);
      if (!e) e = dup_(h, &ci, S.colind);
      L.rowptr = rp; L.colind = ci;
      if (!e) e = dalloc_(h, &L.Aown, (size_t)L.nnzA * S.bs * S.bs);
      L.A = L.Aown;
    }
  }
  const AmgLevelDev &Lc = h->L[nl - 1];
  h->N = Lc.n * Lc.bs;
  h->dense = h->N <= kAmgMaxDense;
  if (!e && h->dense) e = dalloc_(h, &h->Ad, (size_t)h->N * h->N);
  if (!e && !k_is_f32) e = dalloc_(h, &h->A0f, (size_t)h->L[0].nnzA * 9);
  if (!e) e = dalloc_(h, &h->part, kPowerBlocks);
  if (!e) e = dalloc_(h, &h->ticket, 1);
  if (!e) e = (int)cudaMemsetAsync(h->ticket, 0, sizeof(unsigned), st);
  for (const void *k : {(const void *)k_pvals<3>, (const void *)k_pvals<6>, (const void *)k_tvals<3>, (const void *)k_tvals<6>,
                        (const void *)k_cvals<3>, (const void *)k_cvals<6>})
    if (!e) e = (int)cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kProdSmem);
  if (!e && h->dense) {
    /* one limit for every hierarchy (handles on other threads launch the
       same kernel): the largest dense size */
    const size_t smem = ((size_t)kAmgMaxDense * kAmgMaxDense + kAmgMaxDense) * sizeof(float);
    e = (int)cudaFuncSetAttribute(k_dense_invert<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (!e) e = (int)cudaFuncSetAttribute(k_dense_invert<6>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  }
  if (!e) e = (int)cudaStreamSynchronize(st);
  *rc = e;
  if (e) { amg_destroy(h); return nullptr; }
  return h;
}

void amg_destroy(AmgHier *h)
{
  if (!h) return;
  cudaStreamSynchronize(h->st);
  if (h->num_exec) cudaGraphExecDestroy(h->num_exec);
  if (h->num_graph) cudaGraphDestroy(h->num_graph);
  h->mem.release(h->st);
  cudaStreamSynchronize(h->st);
  delete h;
}

int amg_levels(const AmgHier *h) { return h ? h->nl : 0; }
long long amg_device_bytes(const AmgHier *h) { return h ? (long long)h->mem.held() : 0; }

static void enqueue_numeric(AmgHier *h, const void *K, bool k_is_f32, cudaStream_t st)
{
  AmgLevelDev &L0 = h->L[0];
  if (k_is_f32) {
    L0.A = (const float *)K;
  } else {
    const long long nv = L0.nnzA * 9;
    k_to_f32<<<nblk(nv, 256), 256, 0, st>>>(nv, (const double *)K, h->A0f);
    L0.A = h->A0f;
  }
  for (int l = 0; l < h->nl; l++) {
    if (h->dense && l == h->nl - 1) break;       /* the dense inverse needs no smoother */
    if (h->L[l].bs == 3) numeric_level<3>(h, l, st);
    else numeric_level<6>(h, l, st);
  }
  if (h->dense) {
    const AmgLevelDev &Lc = h->L[h->nl - 1];
    const size_t smem = ((size_t)h->N * h->N + std::max(h->N, 32)) * sizeof(float);
    const int threads = 1024;
    if (Lc.bs == 3) k_dense_invert<3><<<1, threads, smem, st>>>(Lc.n, Lc.rowptr, Lc.colind, Lc.A, h->Ad);
    else k_dense_invert<6><<<1, threads, smem, st>>>(Lc.n, Lc.rowptr, Lc.colind, Lc.A, h->Ad);
  }
}

/* The numeric setup is a fixed launch sequence over fixed buffers, so it is
   captured once per tangent buffer and replayed for every new tangent. */
int amg_numeric(AmgHier *h, const void *K, bool k_is_f32, cudaStream_t st)
{
  if (!k_is_f32 && !h->A0f) return (int)cudaErrorInvalidValue;
  if (st == nullptr) {                         /* the legacy default stream cannot be captured */
    enqueue_numeric(h, K, k_is_f32, st);
    return (int)cudaGetLastError();
  }
  if (!h->num_exec || h->num_K != K) {
    if (h->num_exec) { cudaGraphExecDestroy(h->num_exec); h->num_exec = nullptr; }
    if (h->num_graph) { cudaGraphDestroy(h->num_graph); h->num_graph = nullptr; }
    cudaError_t e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return (int)e;
    enqueue_numeric(h, K, k_is_f32, st);
    e = cudaStreamEndCapture(st, &h->num_graph);
    if (e != cudaSuccess) return (int)e;
    e = cudaGraphInstantiate(&h->num_exec, h->num_graph, 0);
    if (e != cudaSuccess) return (int)e;
    h->num_K = K;
  }
  return (int)cudaGraphLaunch(h->num_exec, st);
}

AmgStart amg_start(const AmgHier *h)
{
  const AmgLevelDev &L = h->L[0];
  return {L.b, L.r, L.d, L.Dinv, &L.par->theta_inv, L.x};
}

void amg_apply(AmgHier *h, const int *done, cudaStream_t st)
{
  const int nl = h->nl;
  for (int l = 0; l < nl - 1; l++) {
    if (h->L[l].bs == 3) down_to_coarse<3>(h, l, done, st);
    else down_to_coarse<6>(h, l, done, st);
  }
  AmgLevelDev &Lc = h->L[nl - 1];
  if (h->dense) {
    k_dense_apply<<<1, kDenseThreads, 0, st>>>(h->N, Lc.bs, h->Ad, Lc.b, Lc.x, done);
  } else {
    /* no dense solve: smooth from zero and once more */
    auto coarsest = [&](auto bs) {
      constexpr int BS = decltype(bs)::value;
      smooth_step<BS>(h, nl - 1, 1, done, st);
      smooth_start<BS>(h, nl - 1, done, st);
      smooth_step<BS>(h, nl - 1, 0, done, st);
    };
    if (Lc.bs == 3) coarsest(std::integral_constant<int, 3>());
    else coarsest(std::integral_constant<int, 6>());
  }
  for (int l = nl - 2; l >= 0; l--) {
    if (h->L[l].bs == 3) up_from_coarse<3>(h, l, done, st);
    else up_from_coarse<6>(h, l, done, st);
  }
}

}  // namespace biofem
