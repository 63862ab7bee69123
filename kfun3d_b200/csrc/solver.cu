// kfun3d_b200: BLAS-1 reductions, wall forces, the reference's C entry points
// and the device-resident pseudo-transient Newton / GMRES(30) driver.
//
// Compiled with -fmad=false: in exact mode every reduction sums in index
// order (as the reference at one OpenMP thread) and every scalar update keeps
// its operation order; fast mode uses explicit fma() and fixed-shape tree
// reductions (deterministic run to run).
#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <thread>
#include <vector>

#include "internal.h"

extern int g_kf_verbose;

namespace {

constexpr double JV_EPS = 1.490116119384766e-08;   // src/kernel.c:12
constexpr int RED_BLOCKS = 296;                    // 2 x 148 SMs
constexpr int S_XN = 40, S_QN = 42, S_FN = 43, S_T0 = 44, S_VN = 48, S_CMP = 52;

inline unsigned nblk(size_t n, unsigned t) { return (unsigned)((n + t - 1) / t); }

// ------------------------------------------------------------------ reductions

// Sum of a[i]*b[i] in index order (src/utils.c:53-67, src/kernel.c:131-134),
// one CTA: seven warps form the products of one tile in shared memory while
// one thread adds those of the tile before, in order.  Bound by the chain of
// dependent additions (8.2 cycles each).  16 projections and a norm at 10^3
// (4,000 elements): 1,281 us with one warp that passed the products around by
// shuffles, 402 us so (their chains alone: 284 us).
constexpr int SEQ_TILE = 896;   // 4 products for each of the 224 threads
// s plus the tile's first cnt products, one after the other; eight
// shared-memory loads ahead of the additions that use them
__device__ __forceinline__ double add_in_order(double s, const double *tile, int cnt)
{
  const double2 *p = reinterpret_cast<const double2 *>(tile);
  double2 cur[8];
#pragma unroll
  for (int q = 0; q < 8; q++) cur[q] = p[q];
  int i = 0;
  for (; i + 16 <= cnt; i += 16) {
    const int nx = i + 32 <= SEQ_TILE ? i / 2 + 8 : 0;
    double2 nxt[8];
#pragma unroll
    for (int q = 0; q < 8; q++) nxt[q] = p[nx + q];
#pragma unroll
    for (int q = 0; q < 8; q++) {
      s += cur[q].x;
      s += cur[q].y;
      cur[q] = nxt[q];
    }
  }
  for (; i < cnt; i++) s += tile[i];
  return s;
}

__global__ void __launch_bounds__(256) k_dot_seq(size_t n, const double *__restrict__ a, const double *__restrict__ b,
                                                 double *__restrict__ out, int op)
{
  __shared__ __align__(16) double tile[2][SEQ_TILE];
  const size_t nt = (n + SEQ_TILE - 1) / SEQ_TILE;
  double s = 0.0;
  for (size_t t = 0; t <= nt; t++) {
    if (threadIdx.x >= 32) {
      if (t < nt) {
        double u[4], v[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const size_t g = t * SEQ_TILE + (threadIdx.x - 32) + 224 * q;
          u[q] = g < n ? a[g] : 0.0;
          v[q] = g < n ? b[g] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) tile[t & 1][threadIdx.x - 32 + 224 * q] = u[q] * v[q];
      }
    } else if (threadIdx.x == 0 && t > 0) {
      const size_t left = n - (t - 1) * SEQ_TILE;
      s = add_in_order(s, tile[(t - 1) & 1], left < SEQ_TILE ? (int)left : SEQ_TILE);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    if (op == 0) *out = s;
    else if (op == 1) *out = sqrt(s);
    else *out = sqrt(1.0 + sqrt(s));   // src/kernel.c:95
  }
}

__device__ __forceinline__ double warp_sum(double v)
{
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// The last CTA of a grid to arrive (its partial sums written before): true in
// every thread of that CTA, which then sees all partial sums.  Resets *cnt.
__device__ __forceinline__ bool last_cta(unsigned *cnt)
{
  __shared__ bool last_s;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last_s = atomicAdd(cnt, 1u) == gridDim.x - 1;
    if (last_s) *cnt = 0;
  }
  __syncthreads();
  if (last_s) __threadfence();
  return last_s;
}

// Fast form: fixed grid, fixed tree, so the result is run-to-run identical.
// The last CTA adds the CTAs' sums.
__global__ void __launch_bounds__(256) k_dot_fast(size_t n, const double *__restrict__ a,
                                                  const double *__restrict__ b, double *__restrict__ part,
                                                  double *__restrict__ out, int op, unsigned *cnt)
{
  __shared__ double sm[8];
  double s = 0.0;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const size_t n2 = n / 2;
  const double2 *a2 = reinterpret_cast<const double2 *>(a), *b2 = reinterpret_cast<const double2 *>(b);
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n2; i += stride) {
    const double2 x = a2[i], y = b2[i];
    s = fma(x.x, y.x, s);
    s = fma(x.y, y.y, s);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && (n & 1)) s = fma(a[n - 1], b[n - 1], s);
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    double v = threadIdx.x < 8 ? sm[threadIdx.x] : 0.0;
    v = warp_sum(v);
    if (threadIdx.x == 0) part[blockIdx.x] = v;
  }
  if (!last_cta(cnt)) return;
  s = 0.0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) s += __ldcg(part + i);
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double v = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) v += sm[w];
    if (op == 0) *out = v;
    else if (op == 1) *out = sqrt(v);
    else *out = sqrt(1.0 + sqrt(v));
  }
}

__device__ __forceinline__ double block_sum(double v, double *sm)
{
  v = warp_sum(v);
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) sm[w] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x < 32) {
    t = threadIdx.x < (blockDim.x >> 5) ? sm[threadIdx.x] : 0.0;
    t = warp_sum(t);
  }
  __syncthreads();
  return t;   // valid in thread 0
}

__device__ __forceinline__ double grid_total(const double *part, int np, double *sm)
{
  double v = 0.0;
  for (int i = threadIdx.x; i < np; i += blockDim.x) v += __ldcg(part + i);   // written by other blocks
  v = block_sum(v, sm);
  if (threadIdx.x == 0) sm[32] = v;
  __syncthreads();
  const double t = sm[32];
  __syncthreads();
  return t;
}

// Fast-mode modified Gram-Schmidt of w = V[k+1] against V[0..k] and its
// normalisation (src/kernel.c:129-141) with two reductions instead of k + 2:
// the coefficients h_v = V_v . (w - sum_{j<v} h_j V_j) of the sequential sweep
// are h_v = V_v . w - sum_{j<v} h_j (V_v . V_j), so all the products V_v . w are
// formed in one pass (k_gs_dots), with those of V_k against V_0..V_{k-1}, which
// complete the strictly lower triangle L of the basis' Gram matrix (one row a
// step); (I + L) h = V^T w is solved by substitution, and w -= V h takes one
// more pass (k_gs_update).  The basis is not assumed orthonormal, as in the
// sequential sweep.  Every sum has a fixed shape: run-to-run deterministic.
//
// Bound by memory on large meshes (the basis is read twice, once in groups of
// GS_GROUP with w and V_k read again per group: (k+1)(2 + 2/8) + 4 vectors) and
// by three launches on small ones, where the sequential sweep paid a grid
// barrier of about 6 us per projection.  At Arnoldi index 15, sweep with the
// vector kept on chip / now: 25^3 102 / 21 us, 40^3 107 / 27, 70^3 138 / 72,
// 120^3 426 / 342 us (2.2 GB, 6.4 TB/s).
constexpr int GS_BLOCKS = 296;   // 2 x 148 SMs
constexpr int GS_GROUP = 8;      // basis vectors a pass over w takes at once

// part: [2 (k + 1)][GS_BLOCKS] partial sums (w, then V_k, against each vector);
// L: [KF_NBASIS][32], row v = V_v . V_j for j < v
__global__ void __launch_bounds__(256, 2) k_gs_dots(size_t n, const double *__restrict__ V, int k,
                                                    double *__restrict__ h, double *__restrict__ part,
                                                    double *__restrict__ L, unsigned *cnt)
{
  __shared__ double sm[8][2 * GS_GROUP];
  __shared__ double tot[2 * 32];
  const size_t n2 = n / 2, stride = (size_t)gridDim.x * blockDim.x;
  const size_t i0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const double2 *w = reinterpret_cast<const double2 *>(V + (size_t)(k + 1) * n);
  const double2 *vk = reinterpret_cast<const double2 *>(V + (size_t)k * n);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int g0 = 0; g0 <= k; g0 += GS_GROUP) {
    double s[2 * GS_GROUP];
#pragma unroll
    for (int u = 0; u < 2 * GS_GROUP; u++) s[u] = 0.0;
    for (size_t i = i0; i < n2; i += stride) {
      const double2 a = w[i], b = vk[i];
      double2 c[GS_GROUP];
#pragma unroll
      for (int u = 0; u < GS_GROUP; u++) {
        c[u] = b;   // V_k itself (and a filler beyond it)
        if (g0 + u < k) c[u] = __ldcs(reinterpret_cast<const double2 *>(V + (size_t)(g0 + u) * n) + i);
      }
#pragma unroll
      for (int u = 0; u < GS_GROUP; u++) {
        s[u] = fma(a.x, c[u].x, s[u]);
        s[u] = fma(a.y, c[u].y, s[u]);
        s[GS_GROUP + u] = fma(b.x, c[u].x, s[GS_GROUP + u]);
        s[GS_GROUP + u] = fma(b.y, c[u].y, s[GS_GROUP + u]);
      }
    }
#pragma unroll
    for (int u = 0; u < 2 * GS_GROUP; u++) {
      const double v = warp_sum(s[u]);
      if (lane == 0) sm[warp][u] = v;
    }
    __syncthreads();
    if (threadIdx.x < 2 * GS_GROUP) {
      const int u = threadIdx.x % GS_GROUP, which = threadIdx.x / GS_GROUP;
      if (g0 + u <= k) {
        double v = 0.0;
        for (int x = 0; x < 8; x++) v += sm[x][threadIdx.x];
        part[(size_t)(2 * (g0 + u) + which) * GS_BLOCKS + blockIdx.x] = v;
      }
    }
    __syncthreads();
  }
  if (!last_cta(cnt)) return;
  for (int q = warp; q < 2 * (k + 1); q += 8) {
    double v = 0.0;
    for (int x = lane; x < (int)gridDim.x; x += 32) v += __ldcg(part + (size_t)q * GS_BLOCKS + x);
    v = warp_sum(v);
    if (lane == 0) tot[q] = v;
  }
  __syncthreads();
  if (warp == 0) {
    // forward substitution, lane v = coefficient v
    if (lane < k) L[32 * k + lane] = tot[2 * lane + 1];
    double hv = lane <= k ? tot[2 * lane] : 0.0;
    for (int j = 0; j < k; j++) {
      const double hj = __shfl_sync(0xffffffffu, hv, j);
      const double l = lane > j && lane <= k ? (lane == k ? tot[2 * j + 1] : L[32 * lane + j]) : 0.0;
      if (lane > j) hv = fma(-l, hj, hv);
    }
    if (lane <= k) h[lane] = hv;
  }
}

// w -= sum_v h[v] V[v] (in that order) and h[k+1] = |w|.  The last CTA also
// writes the column to the host's pinned memory and then counts it in
// host_seq, so that the host reads it while the vector is still being scaled
// (a copy node and a stream synchronisation an iteration before: 25^3 167 ->
// 153 us an iteration, 40^3 236 -> 215).  Elements from the last to the first:
// those k_gs_dots read last may still be in L2.
__global__ void __launch_bounds__(256, 3) k_gs_update(size_t n, double *__restrict__ V, int k,
                                                      double *__restrict__ h, double *__restrict__ part,
                                                      unsigned *cnt, double *host_h, unsigned *seq,
                                                      volatile unsigned *host_seq)
{
  asm volatile("griddepcontrol.wait;" ::: "memory");
  __shared__ double sm[40];
  __shared__ double hs[32];
  if (threadIdx.x <= k) hs[threadIdx.x] = h[threadIdx.x];
  __syncthreads();
  const size_t n2 = n / 2, stride = (size_t)gridDim.x * blockDim.x;
  const size_t i0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  double2 *w = reinterpret_cast<double2 *>(V + (size_t)(k + 1) * n);
  double s = 0.0;
  for (size_t j = i0; j < n2; j += stride) {
    const size_t i = n2 - 1 - j;
    double2 a = w[i];
    int v = 0;
    for (; v + 8 <= k + 1; v += 8) {
      double2 c[8];
#pragma unroll
      for (int u = 0; u < 8; u++) c[u] = reinterpret_cast<const double2 *>(V + (size_t)(v + u) * n)[i];
#pragma unroll
      for (int u = 0; u < 8; u++) {
        a.x = fma(-hs[v + u], c[u].x, a.x);
        a.y = fma(-hs[v + u], c[u].y, a.y);
      }
    }
    for (; v <= k; v++) {
      const double2 c = reinterpret_cast<const double2 *>(V + (size_t)v * n)[i];
      a.x = fma(-hs[v], c.x, a.x);
      a.y = fma(-hs[v], c.y, a.y);
    }
    w[i] = a;
    s = fma(a.x, a.x, s);
    s = fma(a.y, a.y, s);
  }
  const double bs = block_sum(s, sm);
  if (threadIdx.x == 0) part[blockIdx.x] = bs;
  if (!last_cta(cnt)) return;
  const double t = grid_total(part, gridDim.x, sm);
  if (threadIdx.x <= k) host_h[threadIdx.x] = hs[threadIdx.x];
  if (threadIdx.x == 0) {
    h[k + 1] = sqrt(t);
    host_h[k + 1] = sqrt(t);
  }
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned s = *seq + 1;
    *seq = s;
    *host_seq = s;
  }
}

// w /= |w|, and *xn = |w| of the result: what the next step's difference
// quotient divides by, without a launch and a pass of its own over the vector
// (an Arnoldi step at 25^3 130 -> 125 us, 120^3 FP32 1810 -> 1790).  At most
// eight CTAs an SM, so that few sums are left for the last one.
__global__ void __launch_bounds__(256) k_gs_scale(size_t n, double *__restrict__ V, int k, const double *__restrict__ h,
                                                  double *__restrict__ part, unsigned *cnt, double *__restrict__ xn)
{
  asm volatile("griddepcontrol.wait;" ::: "memory");
  __shared__ double sm[40];
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  double2 *w = reinterpret_cast<double2 *>(V + (size_t)(k + 1) * n);
  const double sc = 1.0 / h[k + 1];
  double s = 0.0;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n / 2; i += stride) {
    double2 a = w[i];
    a.x *= sc;
    a.y *= sc;
    w[i] = a;
    s = fma(a.x, a.x, s);
    s = fma(a.y, a.y, s);
  }
  const double bs = block_sum(s, sm);
  if (threadIdx.x == 0) part[blockIdx.x] = bs;
  if (!last_cta(cnt)) return;
  const double t = grid_total(part, gridDim.x, sm);
  if (threadIdx.x == 0) *xn = sqrt(t);
}

// Exact-mode modified Gram-Schmidt of V[k+1] against V[0..k] and its
// normalisation (src/kernel.c:129-141) in one launch of one CTA: every dot
// product's additions form one chain in index order, and the chains follow one
// another, so one thread adds and the others apply the projection before it
// and form the products a tile ahead.  At Arnoldi index 15 on the 10^3 mesh the
// chains alone take 284 us; a launch for each dot product and each projection
// took 402 us, this one takes 319.
__global__ void __launch_bounds__(256) k_mgs_seq(size_t n, double *V, int k, double *__restrict__ h)
{
  __shared__ __align__(16) double tile[2][SEQ_TILE];
  __shared__ double hs;
  const size_t nt = (n + SEQ_TILE - 1) / SEQ_TILE;
  double *w = V + (size_t)(k + 1) * n;
  for (int v = 0; v <= k + 1; v++) {
    const double *prev = v > 0 ? V + (size_t)(v - 1) * n : nullptr, *cur = v <= k ? V + (size_t)v * n : nullptr;
    const double a = v > 0 ? -1.0 * hs : 0.0;
    double s = 0.0;
    for (size_t t = 0; t <= nt; t++) {
      if (threadIdx.x >= 32) {
        if (t < nt) {
          double x[4], y[4], z[4];
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const size_t g = t * SEQ_TILE + (threadIdx.x - 32) + 224 * q;
            x[q] = g < n ? w[g] : 0.0;
            y[q] = prev && g < n ? prev[g] : 0.0;
            z[q] = cur && g < n ? cur[g] : 0.0;
          }
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const size_t g = t * SEQ_TILE + (threadIdx.x - 32) + 224 * q;
            if (prev) {
              x[q] = a * y[q] + x[q];
              if (g < n) w[g] = x[q];
            }
            tile[t & 1][threadIdx.x - 32 + 224 * q] = x[q] * (cur ? z[q] : x[q]);
          }
        }
      } else if (threadIdx.x == 0 && t > 0) {
        const size_t left = n - (t - 1) * SEQ_TILE;
        s = add_in_order(s, tile[(t - 1) & 1], left < SEQ_TILE ? (int)left : SEQ_TILE);
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) {
      hs = v <= k ? s : sqrt(s);
      h[v] = hs;
    }
    __syncthreads();
  }
  const double nrm = hs;
  for (size_t i = threadIdx.x; i < n; i += blockDim.x) w[i] *= (1.0 / nrm);
}

// y = a x + y (src/utils.c:69-87)
__global__ void k_axpy(size_t n, double a, const double *__restrict__ x, double *__restrict__ y, int fast)
{
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  y[i] = fast ? fma(a, x[i], y[i]) : a * x[i] + y[i];
}

// y = a[0] v[0] + y, then a[1] v[1] + y, ... (k_axpy's arithmetic, vector
// after vector in that order) in one pass: y and every v read once
struct AxpyList {
  const double *v[KF_NBASIS];
  double a[KF_NBASIS];
};
__global__ void k_axpy_multi(size_t n, int k, AxpyList L, double *__restrict__ y, int fast)
{
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double acc = y[i];
  for (int v = 0; v < k; v++) acc = fast ? fma(L.a[v], L.v[v][i], acc) : L.a[v] * L.v[v][i] + acc;
  y[i] = acc;
}

// w = a x + y (src/utils.c:89-107)
__global__ void k_waxpy(size_t n, double a, const double *__restrict__ x, const double *__restrict__ y,
                        double *__restrict__ w, int fast)
{
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  w[i] = fast ? fma(a, x[i], y[i]) : a * x[i] + y[i];
}

// x *= 1/|x| with |x| on the device (src/utils.c:109-122)
__global__ void k_scale_inv(size_t n, const double *__restrict__ nrm, double *__restrict__ x)
{
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  x[i] *= (1.0 / nrm[0]);
}

// J.v set-up, src/kernel.c:27-30: h = eps * qnorm; w = (h/|x|) x + q
__global__ void k_jv_shift(size_t n, const double *__restrict__ xn, const double *__restrict__ qn,
                           const double *__restrict__ x, const double *__restrict__ q, double *__restrict__ w, int fast)
{
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double h = JV_EPS * qn[0];
  const double a = h / xn[0];
  w[i] = fast ? fma(a, x[i], q[i]) : a * x[i] + q[i];
}

// k_jv_shift with the visit-order copy of w written alongside: node i's w in
// the mesh's order (coalesced, like x and q) and at its visit position
// rowof[i] in qv (the same arithmetic)
__global__ void k_jv_shift_visit(uint32_t N, const uint32_t *__restrict__ rowof, const double *__restrict__ xn,
                                 const double *__restrict__ qn,
                                 const double *__restrict__ x, const double *__restrict__ q, double *__restrict__ w,
                                 double4 *__restrict__ qv, int fast)
{
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const double h = JV_EPS * qn[0];
  const double a = h / xn[0];
  const double4 xx = reinterpret_cast<const double4 *>(x)[i], qq = reinterpret_cast<const double4 *>(q)[i];
  double4 o;
  o.x = fast ? fma(a, xx.x, qq.x) : a * xx.x + qq.x;
  o.y = fast ? fma(a, xx.y, qq.y) : a * xx.y + qq.y;
  o.z = fast ? fma(a, xx.z, qq.z) : a * xx.z + qq.z;
  o.w = fast ? fma(a, xx.w, qq.w) : a * xx.w + qq.w;
  reinterpret_cast<double4 *>(w)[i] = o;
  qv[rowof[i]] = o;
}

// src/forces.c:8-120 in the reference's order: per colour an OpenMP
// reduction from zero over the colour's faces in face order, each colour's sum
// then added to the running total.  One warp per colour: the lanes form 32
// faces' products at once, then every lane applies them to the running sums
// in face order (lift = (lift - dcx V) + dcy U, drag = (drag + dcx U) + dcy V,
// momn = (momn + (xmid - 1/4) dcy) - ymid dcx), so the arithmetic is the
// reference's.  The colour sums are added in colour order by one thread.
__global__ void __launch_bounds__(1024) k_forces(uint32_t ncol, const uint32_t *__restrict__ col,
                                                 const uint32_t *__restrict__ wf, const double4 *__restrict__ xyz,
                                                 const double4 *__restrict__ q, double U, double V,
                                                 double *__restrict__ out)
{
  __shared__ double part[3 * 1024];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (uint32_t c = warp; c < ncol; c += nw) {
    double l = 0.0, d = 0.0, m = 0.0;
    for (uint32_t base = col[c]; base < col[c + 1]; base += 32) {
      const uint32_t j = base + lane;
      double a1 = 0, a2 = 0, b1 = 0, b2 = 0, c1 = 0, c2 = 0;
      if (j < col[c + 1]) {
        const uint32_t a = wf[3 * j], b = wf[3 * j + 1], e = wf[3 * j + 2];
        const double4 pa = xyz[a], pb = xyz[b], pe = xyz[e];
        const double ax = pb.x - pa.x, ay = pb.y - pa.y, az = pb.z - pa.z;
        const double bx = pe.x - pa.x, by = pe.y - pa.y, bz = pe.z - pa.z;
        double xnorm = ay * bz; xnorm -= az * by; xnorm = -0.5 * xnorm;
        double ynorm = ax * bz; ynorm -= az * bx; ynorm = 0.5 * ynorm;
        const double press = (q[a].x + q[b].x + q[e].x) / 3.0;
        const double cp = 2.0 * (press - 1.0);
        const double dcx = cp * xnorm, dcy = cp * ynorm;
        const double xmid = pa.x + pb.x + pe.x;
        const double ymid = pa.y + pb.y + pe.y;
        a1 = dcx * V; a2 = dcy * U;
        b1 = dcx * U; b2 = dcy * V;
        c1 = (xmid - 0.25) * dcy; c2 = ymid * dcx;
      }
      const uint32_t cnt = min(32u, col[c + 1] - base);
      for (uint32_t k = 0; k < cnt; k++) {
        l = l - __shfl_sync(0xffffffffu, a1, k);
        l = l + __shfl_sync(0xffffffffu, a2, k);
        d = d + __shfl_sync(0xffffffffu, b1, k);
        d = d + __shfl_sync(0xffffffffu, b2, k);
        m = m + __shfl_sync(0xffffffffu, c1, k);
        m = m - __shfl_sync(0xffffffffu, c2, k);
      }
    }
    if (lane == 0 && c < 1024) {
      part[3 * c] = l;
      part[3 * c + 1] = d;
      part[3 * c + 2] = m;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double lift = 0.0, drag = 0.0, momn = 0.0;
    for (uint32_t c = 0; c < ncol && c < 1024; c++) {
      lift += part[3 * c];
      drag += part[3 * c + 1];
      momn += part[3 * c + 2];
    }
    out[0] = lift;
    out[1] = drag;
    out[2] = momn;
  }
}

// ------------------------------------------------------------------ helpers

unsigned forces_threads(uint32_t ncol) { return 32u * std::min<uint32_t>(std::max<uint32_t>(ncol, 1u), 32u); }

bool check_cuda(const char *what)
{
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    std::string s = std::string(what) + ": " + cudaGetErrorString(e);
    kf_set_error(KFUN3D_ERR_CUDA, s.c_str());
    return false;
  }
  return true;
}

#define CK(call)                                                                   \
  do {                                                                             \
    cudaError_t e_ = (call);                                                       \
    if (e_ != cudaSuccess) {                                                       \
      std::string s_ = std::string(#call) + ": " + cudaGetErrorString(e_);        \
      kf_set_error(KFUN3D_ERR_CUDA, s_.c_str());                                   \
    }                                                                              \
  } while (0)

// Rows between the mesh numbering and the spatial ILU numbering:
// to_spatial: dst[rank[i]] = src[i]; from_spatial: dst[i] = src[rank[i]].
__global__ void k_rows_permute(uint32_t N, const uint32_t *__restrict__ rank, const double4 *__restrict__ src,
                               double4 *__restrict__ dst, int to_spatial)
{
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const uint32_t r = rank[i];
  if (to_spatial) dst[r] = src[i];
  else dst[i] = src[r];
}

// Kernel set of the current arithmetic mode.
struct Ops {
  bool fast;
  void gradient(DevMesh &m, const double *q) const { fast ? kf_fast::gradient(m, q) : kf_exact::gradient(m, q); }
  void residual(DevMesh &m, const double *q, double *r, int fo, double u, double v) const
  {
    fast ? kf_fast::residual(m, q, r, fo, u, v) : kf_exact::residual(m, q, r, fo, u, v);
  }
  void timestep(DevMesh &m, const double *q, double cfl) const
  {
    fast ? kf_fast::timestep(m, q, cfl) : kf_exact::timestep(m, q, cfl);
  }
  void fill(DevMesh &m, const double *q, double u, double v, int p) const
  {
    fast ? kf_fast::fill(m, q, u, v, p) : kf_exact::fill(m, q, u, v, p);
  }
  void ilu(DevMesh &m, int p) const { fast ? kf_fast::ilu(m, p) : kf_exact::ilu(m, p); }
  void sptrsv(DevMesh &m, const double *b, double *x, int p) const
  {
    if (m.ilu_active) {
      // spatial ILU(0): x = P^T (LU)^-1 P b, the permutations folded into the
      // packed sweeps where that schedule runs
      if (fast ? kf_fast::sptrsv_permuted(m, b, x, p) : kf_exact::sptrsv_permuted(m, b, x, p)) return;
      const unsigned nb = (m.N + 255) / 256;
      k_rows_permute<<<nb, 256, 0, m.stream>>>(m.N, m.ilu_rank, (const double4 *)b, (double4 *)m.pb, 1);
      fast ? kf_fast::sptrsv(m, m.pb, m.px, p) : kf_exact::sptrsv(m, m.pb, m.px, p);
      k_rows_permute<<<nb, 256, 0, m.stream>>>(m.N, m.ilu_rank, (const double4 *)m.px, (double4 *)x, 0);
      kf_count_launch(2);
      return;
    }
    fast ? kf_fast::sptrsv(m, b, x, p) : kf_exact::sptrsv(m, b, x, p);
  }
  void residual_jv(DevMesh &m, const double *w, double *y, int fo, double u, double v, const JvArgs &jv) const
  {
    fast ? kf_fast::residual_jv(m, w, y, fo, u, v, jv) : kf_exact::residual_jv(m, w, y, fo, u, v, jv);
  }
};

Ops ops() { return Ops{kf_mode() == KFUN3D_MODE_FAST}; }

// dot / norm into a device scalar: op 0 = sum, 1 = sqrt(sum), 2 = sqrt(1 + sqrt(sum))
void dev_reduce(DevMesh &m, const double *a, const double *b, double *out, int op, bool fast)
{
  const size_t n = 4 * (size_t)m.N;
  if (fast) {
    k_dot_fast<<<RED_BLOCKS, 256, 0, m.stream>>>(n, a, b, m.red, out, op, m.bar + 5);
    kf_count_launch();
  } else {
    k_dot_seq<<<1, 256, 0, m.stream>>>(n, a, b, out, op);
    kf_count_launch();
  }
}

void fetch(DevMesh &m, int first, int count)
{
  CK(cudaMemcpyAsync(m.h_scal + first, m.scal + first, count * sizeof(double), cudaMemcpyDeviceToHost, m.stream));
  CK(cudaStreamSynchronize(m.stream));
}

// Residual of state q into r (gradient first unless first order).
void dev_residual(DevMesh &m, const Ops &o, const double *q, double *r)
{
  double u, v;
  kfun3d_get_freestream(&u, &v);
  const int fo = kf_first_order();
  if (!fo) o.gradient(m, q);
  o.residual(m, q, r, fo, u, v);
}

// iJacVec, src/kernel.c:24-45: y = (F(q + h x/|x|) - r + cdt (w - q)) |x| / h;
// vnorm: x is the basis vector that the last gram_schmidt normalised, its norm
// is in S_VN.
void dev_jacvec(DevMesh &m, const Ops &o, const double *x, double *y, bool vnorm = false)
{
  const size_t n = 4 * (size_t)m.N;
  const double *xn = m.scal + (vnorm ? S_VN : S_XN), *qn = m.scal + S_QN;
  if (!vnorm) dev_reduce(m, x, x, m.scal + S_XN, 1, o.fast);
  if (m.visit) {
    // the shifted state and its visit-order copy in one pass
    k_jv_shift_visit<<<nblk(m.N, 256), 256, 0, m.stream>>>(m.N, m.rowof, xn, qn, x, m.q, m.w, m.qv, o.fast);
    m.qv_of = m.w;
  } else {
    k_jv_shift<<<nblk(n, 256), 256, 0, m.stream>>>(n, xn, qn, x, m.q, m.w, o.fast);
  }
  kf_count_launch();
  double u, v;
  kfun3d_get_freestream(&u, &v);
  const int fo = kf_first_order();
  if (!fo) o.gradient(m, m.w);
  o.residual_jv(m, m.w, y, fo, u, v, JvArgs{m.r, m.q, xn, qn, JV_EPS});
}

void dev_axpy(DevMesh &m, double a, const double *x, double *y, bool fast)
{
  const size_t n = 4 * (size_t)m.N;
  k_axpy<<<nblk(n, 256), 256, 0, m.stream>>>(n, a, x, y, fast);
  kf_count_launch();
}

double *Vb(DevMesh &m, int k) { return m.V + (size_t)k * 4 * m.N; }

// y += sum over v < k of a[v] x[v], one launch (the sum of k dev_axpy calls,
// in their order)
void dev_axpy_multi(DevMesh &m, int k, const double *a, const double *const *x, double *y, bool fast)
{
  if (k <= 0) return;
  const size_t n = 4 * (size_t)m.N;
  AxpyList L{};
  for (int v = 0; v < k && v < KF_NBASIS; v++) { L.v[v] = x[v]; L.a[v] = a[v]; }
  k_axpy_multi<<<nblk(n, 256), 256, 0, m.stream>>>(n, std::min(k, (int)KF_NBASIS), L, y, fast);
  kf_count_launch();
}

void dev_normalize(DevMesh &m, double *x, double *nrm, bool fast)
{
  const size_t n = 4 * (size_t)m.N;
  dev_reduce(m, x, x, nrm, 1, fast);
  k_scale_inv<<<nblk(n, 256), 256, 0, m.stream>>>(n, nrm, x);
  kf_count_launch();
}

template <class... P, class... A>
void launch_dependent(void (*kern)(P...), unsigned grid, cudaStream_t st, A... args)
{
  // starts while the kernel before it ends (it waits for it with griddepcontrol.wait)
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(256);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  CK(cudaLaunchKernelEx(&cfg, kern, args...));
}

void gram_schmidt(DevMesh &m, int k)
{
  const size_t n = 4 * (size_t)m.N;
  const unsigned grid = std::min((unsigned)GS_BLOCKS, std::max(1u, nblk(n / 2, 256)));
  k_gs_dots<<<grid, 256, 0, m.stream>>>(n, m.V, k, m.scal, m.gs_part, m.gs_part + 64 * GS_BLOCKS, m.bar + 2);
  launch_dependent(k_gs_update, grid, m.stream, n, m.V, k, m.scal, m.gs_part, m.bar + 3, m.h_scal, m.gs_seq_d,
                   (volatile unsigned *)m.h_seq);
  m.gs_seq++;
  launch_dependent(k_gs_scale, std::min(1184u, std::max(1u, nblk(n / 2, 256))), m.stream, n, m.V, k,
                   (const double *)m.scal, m.gs_part, m.bar + 6, m.scal + S_VN);
  kf_count_launch(3);
}

// Modified Gram-Schmidt of V[k+1] against V[0..k], normalised; h in scal[0..k+1].
void orthogonalize(DevMesh &m, const Ops &o, int k)
{
  if (o.fast) {
    gram_schmidt(m, k);
    return;
  }
  k_mgs_seq<<<1, 256, 0, m.stream>>>(4 * (size_t)m.N, m.V, k, m.scal);
  kf_count_launch();
}

// One Arnoldi step k (src/kernel.c:123-141): V[k+1] = M^-1 J V[k],
// orthogonalised and normalised; h in scal[0..k+1].
void arnoldi_step(DevMesh &m, const Ops &o, int k, int prec)
{
  dev_jacvec(m, o, Vb(m, k), m.t, o.fast && k > 0);   // (V[0]: normalised by dev_normalize)
  o.sptrsv(m, m.t, Vb(m, k + 1), prec);
  orthogonalize(m, o, k);
}

// Waits for the Hessenberg column of the last gram_schmidt in h_scal[0..k+1]:
// it is there when the kernel's count reaches the host's.  The stream's own
// state ends the wait when the kernel did not get that far.
void wait_column(DevMesh &m, int k)
{
  volatile unsigned *seq = m.h_seq;
  for (unsigned spin = 1; *seq != m.gs_seq; spin++) {
    if (spin % 1024) continue;
    const cudaError_t e = cudaStreamQuery(m.stream);
    if (e == cudaErrorNotReady) continue;
    CK(e);
    if (*seq != m.gs_seq) {   // idle without it: read back what there is, and count from here
      m.gs_seq = *seq;
      fetch(m, 0, k + 2);
    }
    break;
  }
  std::atomic_thread_fence(std::memory_order_acquire);
}

// Fast mode: the Arnoldi step (its Hessenberg column written to the host) as
// one CUDA graph per (precision, first order, k), captured on first use.
void arnoldi_step_graph(DevMesh &m, const Ops &o, int k, int prec)
{
  const int fo = kf_first_order();
  double u, v;
  kfun3d_get_freestream(&u, &v);
  if (m.graph_aoa != kfun3d_get_aoa() || m.graph_ilu != m.ilu_active) {
    for (auto &a : m.arnoldi)
      for (auto &b : a)
        for (auto &g : b)
          if (g) { cudaGraphExecDestroy(g); g = nullptr; }
    m.graph_aoa = kfun3d_get_aoa();
    m.graph_ilu = m.ilu_active;
  }
  cudaGraphExec_t &ge = m.arnoldi[prec][fo][k];
  if (!ge) {
    const unsigned long long before = kfun3d_launch_count();
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamBeginCapture(m.stream, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
      const unsigned seq = m.gs_seq;
      arnoldi_step(m, o, k, prec);
      m.gs_seq = seq;
      e = cudaStreamEndCapture(m.stream, &graph);
    }
    const unsigned nodes = (unsigned)(kfun3d_launch_count() - before);
    kfun3d_reset_launch_count_by(nodes);
    if (e == cudaSuccess) e = cudaGraphInstantiate(&ge, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    if (e != cudaSuccess) {
      // capture not available: run this solve without graphs
      cudaGetLastError();
      ge = nullptr;
      m.use_graphs = false;
      arnoldi_step(m, o, k, prec);
      fetch(m, 0, k + 2);
      return;
    }
    m.arnoldi_nodes[prec][fo][k] = nodes;
  }
  CK(cudaGraphLaunch(ge, m.stream));
  m.gs_seq++;
  kf_count_launch(m.arnoldi_nodes[prec][fo][k]);
  wait_column(m, k);
}

// Device status words: [0] pivot failure in ILU(0), [1] a bounded wait gave up.
int device_status(DevMesh &m)
{
  int st[2] = {0, 0};
  CK(cudaMemcpyAsync(st, m.status, 2 * sizeof(int), cudaMemcpyDeviceToHost, m.stream));
  CK(cudaStreamSynchronize(m.stream));
  if (st[0] || st[1]) {
    CK(cudaMemsetAsync(m.status, 0, 2 * sizeof(int), m.stream));
    // a wait that gave up may leave a grid barrier half-counted
    if (st[1] && m.bar) CK(cudaMemsetAsync(m.bar, 0, 8 * sizeof(unsigned), m.stream));
    if (st[1] && m.flow_buf) CK(kf_flow_reset(m));
  }
  if (st[1]) return KFUN3D_ERR_TIMEOUT;
  return st[0];
}

}  // namespace

// ------------------------------------------------------------------ solve

extern "C" void kfun3d_default_params(kfun3d_solver_params *p)
{
  p->ts_max = 15;
  p->stop_ratio = 10000000.0;
  p->gmres_rtol = 0.01;
  p->gmres_restart = 30;
  p->gmres_max_it = 10000;
  p->cfl_init = 50.0;
  p->cfl_max = 100000.0;
}

// The device-resident solve of src/kernel.c:47-232 (parameters as data).
// The state stays on the device; the host keeps the small GMRES scalars and
// reads one column of the Hessenberg matrix per Arnoldi step.
static int solve_device(DevMesh &m, const GEOMETRY *g, const kfun3d_solver_params *p, kfun3d_step *hist,
                        int max_hist, bool print)
{
  const Ops o = ops();
  const int prec = kf_precision();
  const size_t n = 4 * (size_t)m.N;
  const int restart = std::min(std::max(p->gmres_restart, 1), 30);
  double u, v;
  kfun3d_get_freestream(&u, &v);
  double ghh[KF_NBASIS * (KF_NBASIS + 1)] = {0};
  double cs[KF_NBASIS], sn[KF_NBASIS], rs[KF_NBASIS];
  double fnorm0 = 0.0, cfl = p->cfl_init;
  int nrec = 0, steps = 0;
  cudaEvent_t ev0, ev1;
  CK(cudaEventCreate(&ev0));
  CK(cudaEventCreate(&ev1));
  for (int its = 0; its < p->ts_max; its++) {
    CK(cudaEventRecord(ev0, m.stream));
    dev_residual(m, o, m.q, m.r);
    dev_reduce(m, m.r, m.r, m.scal + S_FN, 1, o.fast);
    fetch(m, S_FN, 1);
    const double fnorm = m.h_scal[S_FN];
    if (!std::isfinite(fnorm)) {
      kf_set_error(KFUN3D_ERR_NONFINITE, "residual norm is not finite");
      steps = -1;
      break;
    }
    if (its == 0) fnorm0 = fnorm;
    else {
      double cfl0 = 1.1 * p->cfl_init * fnorm0;   // src/kernel.c:86-88
      cfl0 /= fnorm;
      cfl = (cfl0 < p->cfl_max) ? cfl0 : p->cfl_max;
    }
    o.timestep(m, m.q, cfl);
    o.fill(m, m.q, u, v, prec);
    dev_reduce(m, m.q, m.q, m.scal + S_QN, 2, o.fast);
    CK(cudaMemsetAsync(m.x, 0, n * sizeof(double), m.stream));
    o.ilu(m, prec);
    o.sptrsv(m, m.r, Vb(m, 0), prec);
    {
      const int st = device_status(m);
      if (st == KFUN3D_ERR_PIVOT) {
        kf_set_error(KFUN3D_ERR_PIVOT, "singular or non-finite pivot block in ILU(0)");
        steps = -1;
        break;
      }
      if (st == KFUN3D_ERR_TIMEOUT) {
        kf_set_error(KFUN3D_ERR_TIMEOUT, "a triangular-solve wait exceeded its bound");
        steps = -1;
        break;
      }
    }

    double tol = 0.0;
    unsigned int total = 0;
    bool done = false;
    while (total <= (unsigned)p->gmres_max_it) {     // src/kernel.c:107-196
      if (total > 0) {
        dev_jacvec(m, o, m.x, m.t);
        k_waxpy<<<nblk(n, 256), 256, 0, m.stream>>>(n, -1.0, m.t, m.r, m.w, o.fast);
        kf_count_launch();
        o.sptrsv(m, m.w, Vb(m, 0), prec);
      }
      dev_normalize(m, Vb(m, 0), m.scal + S_T0, o.fast);
      fetch(m, S_T0, 1);
      rs[0] = m.h_scal[S_T0];
      if (!std::isfinite(rs[0])) {
        kf_set_error(KFUN3D_ERR_NONFINITE, "preconditioned residual is not finite");
        done = false;
        steps = -1;
        break;
      }
      if (total == 0) tol = p->gmres_rtol * rs[0];
      int k = 0;
      while (k < restart) {
        if (o.fast && m.use_graphs) {
          arnoldi_step_graph(m, o, k, prec);
        } else {
          arnoldi_step(m, o, k, prec);
          fetch(m, 0, k + 2);
        }
        double *hh = ghh + k * (KF_NBASIS + 1);
        for (int i = 0; i <= k + 1; i++) hh[i] = m.h_scal[i];
        for (int i = 0; i < k; i++) {               // src/kernel.c:143-149
          const double tt = hh[i];
          hh[i] = cs[i] * hh[i] + sn[i] * hh[i + 1];
          hh[i + 1] = cs[i] * hh[i + 1] - sn[i] * tt;
        }
        const double tt = sqrt(hh[k] * hh[k] + hh[k + 1] * hh[k + 1]);
        const double c = hh[k] / tt, s = hh[k + 1] / tt;
        cs[k] = c;
        sn[k] = s;
        rs[k + 1] = -(s * rs[k]);
        rs[k] = c * rs[k];
        hh[k] = c * hh[k] + s * hh[k + 1];
        const double res = fabs(rs[k + 1]);
        k++;
        if (res <= tol) { done = true; break; }
        if (!std::isfinite(res)) break;
      }
      total += k;
      rs[k - 1] /= ghh[(k - 1) * (KF_NBASIS + 1) + (k - 1)];   // src/kernel.c:178-188
      for (int i = 1; i <= k - 1; i++) {
        const int mm = (k - 1) - i;
        double tt = rs[mm];
        for (int j = mm + 1; j <= k - 1; j++) tt -= ghh[j * (KF_NBASIS + 1) + mm] * rs[j];
        rs[mm] = tt / ghh[mm * (KF_NBASIS + 1) + mm];
      }
      {
        const double *vs[KF_NBASIS];
        for (int vv = 0; vv < k; vv++) vs[vv] = Vb(m, vv);
        dev_axpy_multi(m, k, rs, vs, m.x, o.fast);
      }
      if (print && k == restart) fun3d_printf(5, ">> GMRES: COMPLETED ONE CYCLE\n");
      if (done) break;
    }
    if (steps < 0) break;
    if (print) fun3d_printf(5, ">> GMRES: TOTAL ITERATIONS %d\n", total);
    dev_axpy(m, -1.0, m.x, m.q, o.fast);                           // src/kernel.c:200
    k_forces<<<1, forces_threads(m.ncol), 0, m.stream>>>(m.ncol, m.col, m.wf_nodes, m.xyz, (const double4 *)m.q, u, v, m.forces);
    kf_count_launch();
    CK(cudaEventRecord(ev1, m.stream));
    CK(cudaMemcpyAsync(m.h_scal + 48, m.forces, 3 * sizeof(double), cudaMemcpyDeviceToHost, m.stream));
    CK(cudaStreamSynchronize(m.stream));
    if (!check_cuda("solve")) { steps = -1; break; }
    if (device_status(m) == KFUN3D_ERR_TIMEOUT) {
      kf_set_error(KFUN3D_ERR_TIMEOUT, "a triangular-solve wait exceeded its bound");
      steps = -1;
      break;
    }
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ev0, ev1);
    const double lift = m.h_scal[48], drag = m.h_scal[49], momn = m.h_scal[50];
    if (print) {
      printf("STEP: %d ", its);
      printf("CFL: %g ", cfl);
      printf("NORM: %g\n", fnorm);
      printf("LIFT: %g DRAG: %g MOMN: %g\n", lift, drag, momn);
    }
    if (hist && nrec < max_hist) {
      hist[nrec] = kfun3d_step{its, (int)total, cfl, fnorm, lift, drag, momn, ms * 1e-3};
      nrec++;
    }
    steps = its + 1;
    if (round(fnorm0 / fnorm) >= p->stop_ratio) break;   // src/kernel.c:214
  }
  cudaEventDestroy(ev0);
  cudaEventDestroy(ev1);
  return steps < 0 ? -1 : nrec;
}

// ------------------------------------------------------------------ flexible GMRES

namespace {

// Training pairs written by the ILU(0)-FGMRES solve: slot i holds x0 at
// x0 + i * 16N bytes (BF16 [N x 8]) and the target at tgt + i * 4N floats.
struct PairSink {
  int stride = 0;
  unsigned char *x0 = nullptr;
  float *tgt = nullptr;
  int cap = 0;
  int count = 0;
};

// Givens update of Hessenberg column k (host, src/kernel.c:143-160 arithmetic);
// returns |rs[k+1]|.
double givens(double *hh, double *cs, double *sn, double *rs, int k)
{
  for (int i = 0; i < k; i++) {
    const double tt = hh[i];
    hh[i] = cs[i] * hh[i] + sn[i] * hh[i + 1];
    hh[i + 1] = cs[i] * hh[i + 1] - sn[i] * tt;
  }
  const double tt = sqrt(hh[k] * hh[k] + hh[k + 1] * hh[k + 1]);
  const double c = hh[k] / tt, s = hh[k + 1] / tt;
  cs[k] = c;
  sn[k] = s;
  rs[k + 1] = -(s * rs[k]);
  rs[k] = c * rs[k];
  hh[k] = c * hh[k] + s * hh[k + 1];
  return fabs(rs[k + 1]);
}

// y[0..k-1] from the rotated Hessenberg columns and right-hand side
void back_substitute(const double *ghh, const double *rs, int k, double *y)
{
  for (int i = 0; i < k; i++) y[i] = rs[i];
  y[k - 1] /= ghh[(k - 1) * (KF_NBASIS + 1) + (k - 1)];
  for (int i = 1; i <= k - 1; i++) {
    const int mm = (k - 1) - i;
    double tt = y[mm];
    for (int j = mm + 1; j <= k - 1; j++) tt -= ghh[j * (KF_NBASIS + 1) + mm] * y[j];
    y[mm] = tt / ghh[mm * (KF_NBASIS + 1) + mm];
  }
}

double *Zb(DevMesh &m, int k) { return m.Z + (size_t)k * 4 * m.N; }

bool ensure_flex(DevMesh &m)
{
  const size_t n = 4 * (size_t)m.N;
  if (!m.Z && cudaMalloc(&m.Z, 30 * n * sizeof(double)) != cudaSuccess) return false;
  if (!m.qold && cudaMalloc(&m.qold, n * sizeof(double)) != cudaSuccess) return false;
  if (!m.fy && cudaMalloc(&m.fy, n * sizeof(double)) != cudaSuccess) return false;
  if (!m.fx && cudaMalloc(&m.fx, n * sizeof(double)) != cudaSuccess) return false;
  if (!m.pscr && cudaMalloc(&m.pscr, 264 * sizeof(double)) != cudaSuccess) return false;
  return true;
}

// Pair of the correction x (device, 4N): v = J x, y = ILU(0)^-1 v,
// x0 = BF16([y/s, q]), target = (x - y)/s.
void write_pair(DevMesh &m, const Ops &o, int prec, const double *x, PairSink &ps)
{
  if (ps.count >= ps.cap) return;
  dev_jacvec(m, o, x, m.t);
  o.sptrsv(m, m.t, m.fy, prec);
  kf_mpnn_pair_async(m.N, m.fy, m.q, x, ps.x0 + (size_t)ps.count * 16 * m.N,
                     ps.tgt + (size_t)ps.count * 4 * m.N, m.pscr, m.stream);
  ps.count++;
}

}  // namespace

// The pseudo-transient Newton loop of src/kernel.c:47-232 with its linear
// solves done by flexible GMRES on the reference's left-preconditioned
// system: Arnoldi on ILU(0)^-1 J, residual measured as |ILU(0)^-1 (b - J x)|
// exactly as the reference does, and a right preconditioner allowed to
// change from one iteration to the next,
//   z_k = N_k(v_k),  w = ILU(0)^-1 J z_k orthogonalised against v_0..v_k,
//   x = Z y after each cycle.
// N_k is the identity -- the reference's GMRES, iteration for iteration -- or
// the network's correction v + s N([v/s, q]), which maps an ILU(0)-
// preconditioned residual to an approximation of the correction x with
// ILU(0)^-1 J x = v.  The network is a guest: each linear solve starts with
// both candidate first directions and keeps the network only if its image
// under ILU(0)^-1 J lies closer to v0 (one extra product per Newton step);
// it keeps its place only while the residual falls at least half as fast
// (per iteration, in log) as in the previous step's solve, and for at most
// 1.5x that solve's iterations, after which the solve goes on without it;
// Newton step 0 runs without it to set the pace; three fallbacks in a row
// switch it off for good; and an update after which
// the FP64 nonlinear residual is non-finite or grows tenfold is undone and
// redone without it.
static int solve_flexible(DevMesh &m, const GEOMETRY *g, const kfun3d_solver_params *p, kfun3d_mpnn *net,
                          PairSink *ps, kfun3d_step *hist, int max_hist, kfun3d_flex_stats *st)
{
  const Ops o = ops();
  const int prec = kf_precision();
  const size_t n = 4 * (size_t)m.N;
  const int restart = std::min(std::max(p->gmres_restart, 1), 30);
  double u, v;
  kfun3d_get_freestream(&u, &v);
  kfun3d_flex_stats S{};
  if (!ensure_flex(m)) {
    kf_set_error(KFUN3D_ERR_CUDA, "flexible solve: out of device memory");
    return -1;
  }
  if (net) {
    if (!m.mgraph) m.mgraph = kfun3d_mpnn_graph_create(g);
    if (!m.mgraph || kf_mpnn_prepare(net, m.mgraph) != KFUN3D_OK) return -1;
  }
  double ghh[KF_NBASIS * (KF_NBASIS + 1)] = {0};
  double cs[KF_NBASIS], sn[KF_NBASIS], rs[KF_NBASIS], yk[KF_NBASIS];
  double fnorm0 = 0.0, fnorm_prev = 0.0, cfl = p->cfl_init;
  bool use_net = net != nullptr, last_used_net = false;
  int misses = 0, prev_total = -1;
  double rate_prev = 0.0;   // log residual reduction per iteration of the previous linear solve
  int nrec = 0, steps = 0;
  cudaEvent_t ev0, ev1, es0, es1;
  CK(cudaEventCreate(&ev0));
  CK(cudaEventCreate(&ev1));
  CK(cudaEventCreate(&es0));
  CK(cudaEventCreate(&es1));
  CK(cudaEventRecord(es0, m.stream));
  for (int its = 0; its < p->ts_max; its++) {
    CK(cudaEventRecord(ev0, m.stream));
    dev_residual(m, o, m.q, m.r);
    dev_reduce(m, m.r, m.r, m.scal + S_FN, 1, o.fast);
    fetch(m, S_FN, 1);
    double fnorm = m.h_scal[S_FN];
    if (last_used_net && (!std::isfinite(fnorm) || fnorm > 10.0 * fnorm_prev)) {
      // the nonlinear residual rejects the learned update: undo it, go on without the network
      CK(cudaMemcpyAsync(m.q, m.qold, n * sizeof(double), cudaMemcpyDeviceToDevice, m.stream));
      dev_residual(m, o, m.q, m.r);
      dev_reduce(m, m.r, m.r, m.scal + S_FN, 1, o.fast);
      fetch(m, S_FN, 1);
      fnorm = m.h_scal[S_FN];
      use_net = false;
      S.disabled = 1;
      S.rejected_steps++;
    }
    if (!std::isfinite(fnorm)) {
      kf_set_error(KFUN3D_ERR_NONFINITE, "residual norm is not finite");
      steps = -1;
      break;
    }
    if (its == 0) fnorm0 = fnorm;
    else {
      double cfl0 = 1.1 * p->cfl_init * fnorm0;   // src/kernel.c:86-88
      cfl0 /= fnorm;
      cfl = (cfl0 < p->cfl_max) ? cfl0 : p->cfl_max;
    }
    fnorm_prev = fnorm;
    o.timestep(m, m.q, cfl);
    o.fill(m, m.q, u, v, prec);
    dev_reduce(m, m.q, m.q, m.scal + S_QN, 2, o.fast);
    CK(cudaMemsetAsync(m.x, 0, n * sizeof(double), m.stream));
    o.ilu(m, prec);
    o.sptrsv(m, m.r, Vb(m, 0), prec);                            // src/kernel.c:103
    {
      const int sd = device_status(m);
      if (sd == KFUN3D_ERR_PIVOT) {
        kf_set_error(KFUN3D_ERR_PIVOT, "singular or non-finite pivot block in ILU(0)");
        steps = -1;
        break;
      }
    }
    // Newton step 0 runs without the network: it measures the rate the
    // network then has to beat
    bool step_net = use_net && prev_total > 0;
    // iterations the network may use in this solve: 1.5 x the previous step's
    const int budget = prev_total > 0 ? (3 * prev_total + 1) / 2 : 2 * restart;
    double rs_first = 0.0, res_last = 0.0;
    bool usez[KF_NBASIS] = {false};
    double tol = 0.0;
    unsigned int total = 0;
    bool done = false, failed = false;
    for (int cycle = 0; total <= (unsigned)p->gmres_max_it; cycle++) {   // src/kernel.c:107-196
      if (total > 0) {
        dev_jacvec(m, o, m.x, m.t);
        k_waxpy<<<nblk(n, 256), 256, 0, m.stream>>>(n, -1.0, m.t, m.r, m.w, o.fast);
        kf_count_launch();
        o.sptrsv(m, m.w, Vb(m, 0), prec);
      }
      dev_normalize(m, Vb(m, 0), m.scal + S_T0, o.fast);
      fetch(m, S_T0, 1);
      rs[0] = m.h_scal[S_T0];
      if (!std::isfinite(rs[0])) { failed = true; break; }
      if (total == 0) {
        tol = p->gmres_rtol * rs[0];
        rs_first = rs[0];
        if (rs[0] == 0.0) { done = true; break; }
      }
      int k = 0;
      while (k < restart) {
        bool stepped = false;   // the step ran as a captured graph (its Gram-Schmidt and read-back too)
        if (step_net && cycle == 0 && k == 0) {
          // the network earns this solve on its first direction: both
          // candidates, z = v0 and the network's z, are mapped by
          // ILU(0)^-1 J; the one whose image comes closer to v0
          // (1 - (v0.w)^2 / w.w, the least-squares residual along w) is kept
          if (kf_mpnn_apply_async(net, m.mgraph, Vb(m, 0), m.q, Zb(m, 0), m.stream) != KFUN3D_OK) {
            failed = true;
            break;
          }
          dev_jacvec(m, o, Zb(m, 0), m.t);
          o.sptrsv(m, m.t, Vb(m, 1), prec);
          dev_jacvec(m, o, Vb(m, 0), m.t);
          o.sptrsv(m, m.t, m.fy, prec);
          dev_reduce(m, Vb(m, 0), Vb(m, 1), m.scal + S_CMP, 0, o.fast);
          dev_reduce(m, Vb(m, 1), Vb(m, 1), m.scal + S_CMP + 1, 0, o.fast);
          dev_reduce(m, Vb(m, 0), m.fy, m.scal + S_CMP + 2, 0, o.fast);
          dev_reduce(m, m.fy, m.fy, m.scal + S_CMP + 3, 0, o.fast);
          fetch(m, S_CMP, 4);
          const double *c = m.h_scal + S_CMP;
          const double rho_net = 1.0 - c[0] * c[0] / c[1], rho_plain = 1.0 - c[2] * c[2] / c[3];
          if (!(rho_net < rho_plain)) {
            CK(cudaMemcpyAsync(Vb(m, 1), m.fy, n * sizeof(double), cudaMemcpyDeviceToDevice, m.stream));
            step_net = false;
            usez[0] = false;
            S.fallback_solves++;
            if (++misses >= 3) {   // three solves in a row: off for the rest of the solve
              use_net = false;
              S.disabled = 1;
            }
          } else {
            misses = 0;
            usez[0] = true;
            S.learned_its++;
          }
        } else if (step_net) {
          if (kf_mpnn_apply_async(net, m.mgraph, Vb(m, k), m.q, Zb(m, k), m.stream) != KFUN3D_OK) {
            failed = true;
            break;
          }
          dev_jacvec(m, o, Zb(m, k), m.t);
          o.sptrsv(m, m.t, Vb(m, k + 1), prec);
          usez[k] = true;
          S.learned_its++;
        } else {
          const bool pair = ps && ps->stride < 0 && (k % -ps->stride) == 0 && ps->count < ps->cap;
          usez[k] = false;
          if (o.fast && m.use_graphs && !pair) {
            // without the network the step is the plain Arnoldi step: its
            // captured graph (Gram-Schmidt and the column's read-back included)
            arnoldi_step_graph(m, o, k, prec);
            stepped = true;
          } else {
            dev_jacvec(m, o, Vb(m, k), m.t);                             // src/kernel.c:123-130
            o.sptrsv(m, m.t, Vb(m, k + 1), prec);
            if (pair) {
              // basis pair: x = v_k, y = ILU(0)^-1 J v_k (before Gram-Schmidt)
              kf_mpnn_pair_async(m.N, Vb(m, k + 1), m.q, Vb(m, k), ps->x0 + (size_t)ps->count * 16 * m.N,
                                 ps->tgt + (size_t)ps->count * 4 * m.N, m.pscr, m.stream);
              ps->count++;
            }
          }
        }
        if (!stepped) {
          orthogonalize(m, o, k);
          fetch(m, 0, k + 2);
        }
        double *hh = ghh + k * (KF_NBASIS + 1);
        for (int i = 0; i <= k + 1; i++) hh[i] = m.h_scal[i];
        const double res = givens(hh, cs, sn, rs, k);
        k++;
        if (res <= tol) { done = true; break; }
        if (!std::isfinite(res)) { failed = true; break; }
        res_last = res;
        // the network must keep at least half the previous solve's rate (log
        // residual per iteration) and stay within its iteration budget
        if (step_net && (((int)total + k >= 6 && rate_prev < 0.0 &&
                          log(res / rs_first) > 0.5 * ((int)total + k) * rate_prev) ||
                         (int)total + k > budget)) {
          step_net = false;
          S.fallback_solves++;
          if (++misses >= 3) {
            use_net = false;
            S.disabled = 1;
          }
        }
        if (ps && ps->stride > 0 && cycle == 0 && k < restart && (k % ps->stride) == 0 && ps->count < ps->cap) {
          back_substitute(ghh, rs, k, yk);
          CK(cudaMemsetAsync(m.fx, 0, n * sizeof(double), m.stream));
          {
            const double *vs[KF_NBASIS];
            for (int vv = 0; vv < k; vv++) vs[vv] = Vb(m, vv);
            dev_axpy_multi(m, k, yk, vs, m.fx, o.fast);
          }
          write_pair(m, o, prec, m.fx, *ps);
        }
      }
      if (failed || k == 0) break;
      total += k;
      back_substitute(ghh, rs, k, yk);                                  // src/kernel.c:178-190
      {
        const double *vs[KF_NBASIS];
        for (int vv = 0; vv < k; vv++) vs[vv] = usez[vv] ? Zb(m, vv) : Vb(m, vv);
        dev_axpy_multi(m, k, yk, vs, m.x, o.fast);
      }
      if (done) break;
    }
    if (failed || !done) {
      if (!failed && total > (unsigned)p->gmres_max_it) {
        // iteration limit: keep the iterate, as the reference does
      } else {
        kf_set_error(KFUN3D_ERR_NONFINITE, "flexible GMRES: non-finite residual");
        steps = -1;
        break;
      }
    }
    if (net && kf_mpnn_status(net, m.stream) != KFUN3D_OK) { steps = -1; break; }
    S.gmres_its += (int)total;
    prev_total = (int)total;
    if (total > 0 && rs_first > 0.0 && res_last > 0.0) rate_prev = log(res_last / rs_first) / total;
    if (ps && ps->count < ps->cap) write_pair(m, o, prec, m.x, *ps);
    if (step_net) CK(cudaMemcpyAsync(m.qold, m.q, n * sizeof(double), cudaMemcpyDeviceToDevice, m.stream));
    last_used_net = step_net;
    dev_axpy(m, -1.0, m.x, m.q, o.fast);                           // src/kernel.c:200
    k_forces<<<1, forces_threads(m.ncol), 0, m.stream>>>(m.ncol, m.col, m.wf_nodes, m.xyz, (const double4 *)m.q, u, v,
                                                         m.forces);
    kf_count_launch();
    CK(cudaEventRecord(ev1, m.stream));
    CK(cudaMemcpyAsync(m.h_scal + 48, m.forces, 3 * sizeof(double), cudaMemcpyDeviceToHost, m.stream));
    CK(cudaStreamSynchronize(m.stream));
    if (!check_cuda("flexible solve")) { steps = -1; break; }
    if (device_status(m) == KFUN3D_ERR_TIMEOUT) {
      kf_set_error(KFUN3D_ERR_TIMEOUT, "a triangular-solve wait exceeded its bound");
      steps = -1;
      break;
    }
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ev0, ev1);
    if (hist && nrec < max_hist) {
      hist[nrec] = kfun3d_step{its, (int)total, cfl, fnorm, m.h_scal[48], m.h_scal[49], m.h_scal[50], ms * 1e-3};
      nrec++;
    }
    steps = its + 1;
    if (round(fnorm0 / fnorm) >= p->stop_ratio) break;   // src/kernel.c:214
  }
  CK(cudaEventRecord(es1, m.stream));
  CK(cudaEventSynchronize(es1));
  float tot = 0.f;
  cudaEventElapsedTime(&tot, es0, es1);
  S.newton_steps = steps < 0 ? 0 : steps;
  S.seconds = tot * 1e-3;
  S.pairs = ps ? ps->count : 0;
  if (st) *st = S;
  for (cudaEvent_t e : {ev0, ev1, es0, es1}) cudaEventDestroy(e);
  return steps < 0 ? -1 : nrec;
}

// ------------------------------------------------------------------ entry points

namespace {

DevMesh *dev_or_fail(const GEOMETRY *g)
{
  DevMesh *m = kf_device(g);
  if (m && kf_ilu_select(*m, g, kf_ilu_order()) != KFUN3D_OK) return nullptr;
  if (m && kf_schwarz_select(*m, g, kf_schwarz()) != KFUN3D_OK) return nullptr;
  return m;
}

// One host array and its device copy.
struct HostCopy {
  double *dev;
  double *host;
  size_t n;
};

// Large copies between pageable host arrays and the device go through pinned
// buffers that several host threads fill (or empty) while the copies of the
// others run: the driver's own path for pageable memory is one thread's memcpy
// (about 5 GB/s into pages not yet touched; one residual of the 70^3 mesh, 11 MB
// in, copied directly, and 44 MB out, staged: 9.8 -> 5.2 ms, on a state not passed
// before 6.7 -> 5.0).  To the host, the arrays are written when the call returns;
// to the device, the copies are queued on the mesh's stream.  A chunk a buffer,
// two buffers a thread; the threads take chunks in turn.  The buffers (16 MB) are
// the mesh's and go with it.
// From 32 MB, where one array to the device breaks even; shorter copies do not
// repay the threads' start.  A call directly / staged, one array to the device:
// 8 MB 0.58 / 0.77 ms, 17 MB 1.09 / 1.29, 34 MB 2.03 / 2.03, 55 MB 3.7 / 2.65;
// gradients and residual to the host, into pages not yet touched (and a quarter
// as much to the device): 8 MB 1.45 / 1.52, 16 MB 2.67 / 2.76, 25 MB 3.80 / 3.42,
// 34 MB 4.89 / 3.90, 44 MB 6.67 / 4.90.
constexpr size_t STAGE_MIN = 32u << 20, STAGE_CHUNK = 1u << 20;

bool stage_ready(DevMesh &m)
{
  if (m.stage_failed) return false;
  if (m.stage_buf) return true;
  bool ok = cudaMallocHost(&m.stage_buf, KF_STAGE_SLOTS * STAGE_CHUNK) == cudaSuccess;
  for (int s = 0; s < KF_STAGE_SLOTS && ok; s++)
    ok = cudaEventCreateWithFlags(&m.stage_ev[s], cudaEventDisableTiming) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    m.stage_failed = true;   // without them: plain copies
  }
  return ok;
}

cudaError_t copy_staged(DevMesh &m, const HostCopy *list, int nlist, bool to_host)
{
  struct Chunk {
    unsigned char *dev, *host;
    size_t bytes;
  };
  size_t nchunks = 0;
  for (int i = 0; i < nlist; i++) nchunks += (list[i].n * sizeof(double) + STAGE_CHUNK - 1) / STAGE_CHUNK;
  auto chunk = [&](size_t c) {
    int i = 0;
    for (size_t k; c >= (k = (list[i].n * sizeof(double) + STAGE_CHUNK - 1) / STAGE_CHUNK); i++) c -= k;
    const size_t o = c * STAGE_CHUNK;
    return Chunk{(unsigned char *)list[i].dev + o, (unsigned char *)list[i].host + o,
                 std::min(STAGE_CHUNK, list[i].n * sizeof(double) - o)};
  };
  std::atomic<size_t> next{0};
  std::atomic<int> failed{cudaSuccess};
  auto ok = [&](cudaError_t e) {
    if (e != cudaSuccess) failed = e;
    return e == cudaSuccess;
  };
  auto work = [&](int t) {
    if (!ok(cudaSetDevice(m.device))) return;
    Chunk held[2] = {};   // chunks on their way to the host in the thread's two buffers
    for (int s = 0, last = 0; last < 2; s ^= 1) {
      const int slot = 2 * t + s;
      unsigned char *buf = (unsigned char *)m.stage_buf + slot * STAGE_CHUNK;
      if (m.stage_used[slot]) {
        if (!ok(cudaEventSynchronize(m.stage_ev[slot]))) return;
        m.stage_used[slot] = false;
        if (held[s].bytes) memcpy(held[s].host, buf, held[s].bytes);
        held[s].bytes = 0;
      }
      const size_t c = last ? nchunks : next.fetch_add(1);
      if (c >= nchunks) {
        last += to_host ? 1 : 2;   // this buffer is empty; to the host, the other one has to be too
        continue;
      }
      const Chunk ch = chunk(c);
      if (to_host) {
        if (!ok(cudaMemcpyAsync(buf, ch.dev, ch.bytes, cudaMemcpyDeviceToHost, m.stream))) return;
        held[s] = ch;
      } else {
        memcpy(buf, ch.host, ch.bytes);
        if (!ok(cudaMemcpyAsync(ch.dev, buf, ch.bytes, cudaMemcpyHostToDevice, m.stream))) return;
      }
      if (!ok(cudaEventRecord(m.stage_ev[slot], m.stream))) return;
      m.stage_used[slot] = true;
    }
  };
  const int T = std::min<int>({KF_STAGE_SLOTS / 2, (int)std::max(1u, std::thread::hardware_concurrency()),
                               (int)((nchunks + 1) / 2)});
  std::thread th[KF_STAGE_SLOTS / 2];
  try {
    for (int t = 1; t < T; t++) th[t] = std::thread(work, t);
  } catch (...) {   // no more threads: those that run take all chunks
  }
  work(0);
  for (std::thread &x : th)
    if (x.joinable()) x.join();
  return (cudaError_t)failed.load();
}

void host_copies(DevMesh &m, const HostCopy *list, int nlist, bool to_host)
{
  // pinned, managed and device arrays are copied directly
  size_t bytes = 0;
  bool pageable = true;
  for (int i = 0; i < nlist; i++) bytes += list[i].n * sizeof(double);
  for (int i = 0; i < nlist && bytes >= STAGE_MIN; i++) {
    cudaPointerAttributes at;
    pageable &= cudaPointerGetAttributes(&at, list[i].host) == cudaSuccess && at.type == cudaMemoryTypeUnregistered;
  }
  if (bytes >= STAGE_MIN && pageable && stage_ready(m)) {
    CK(copy_staged(m, list, nlist, to_host));
    return;
  }
  for (int i = 0; i < nlist; i++) {
    if (to_host)
      CK(cudaMemcpyAsync(list[i].host, list[i].dev, list[i].n * sizeof(double), cudaMemcpyDeviceToHost, m.stream));
    else
      CK(cudaMemcpyAsync(list[i].dev, list[i].host, list[i].n * sizeof(double), cudaMemcpyHostToDevice, m.stream));
  }
}

void h2d(DevMesh &m, double *dst, const double *src, size_t n)
{
  const HostCopy c{dst, const_cast<double *>(src), n};
  host_copies(m, &c, 1, false);
}

void d2h(DevMesh &m, double *dst, const double *src, size_t n)
{
  const HostCopy c{const_cast<double *>(src), dst, n};
  host_copies(m, &c, 1, true);
}

bool finish(DevMesh &m, const char *what)
{
  CK(cudaStreamSynchronize(m.stream));
  return check_cuda(what);
}

}  // namespace

extern "C" void ComputeFlux(const GEOMETRY *g, const double *q, GRADIENT *grad, double *r)
{
  DevMesh *m = dev_or_fail(g);
  if (!m) return;
  const size_t n = 4 * (size_t)m->N;
  h2d(*m, m->w, q, n);
  const Ops o = ops();
  if (kf_first_order()) {
    CK(cudaMemsetAsync(m->gx, 0, n * sizeof(double), m->stream));
    CK(cudaMemsetAsync(m->gy, 0, n * sizeof(double), m->stream));
    CK(cudaMemsetAsync(m->gz, 0, n * sizeof(double), m->stream));
  }
  dev_residual(*m, o, m->w, m->t);
  if (!kf_first_order()) {
    if (o.fast) kf_fast::gradient_to_mesh_order(*m);
    else kf_exact::gradient_to_mesh_order(*m);
  }
  const HostCopy out[4] = {{m->gx, grad->x0, n}, {m->gy, grad->x1, n}, {m->gz, grad->x2, n}, {m->t, r, n}};
  host_copies(*m, out, 4, true);
  finish(*m, "ComputeFlux");
}

extern "C" void ComputeTimeStep(const double cfl, GEOMETRY *g)
{
  DevMesh *m = dev_or_fail(g);
  if (!m) return;
  h2d(*m, m->q, g->q->q, 4 * (size_t)m->N);
  ops().timestep(*m, m->q, cfl);
  d2h(*m, g->n->cdt, m->cdt, m->N);
  finish(*m, "ComputeTimeStep");
}

extern "C" void ComputeA(GEOMETRY *g)
{
  DevMesh *m = dev_or_fail(g);
  if (!m) return;
  double u, v;
  kfun3d_get_freestream(&u, &v);
  h2d(*m, m->q, g->q->q, 4 * (size_t)m->N);
  h2d(*m, m->cdt, g->n->cdt, m->N);
  ops().fill(*m, m->q, u, v, kf_precision());
  m->a_valid = true;
  m->factored = false;
  finish(*m, "ComputeA");
}

extern "C" void ComputeNumericalILU(GEOMETRY *g)
{
  DevMesh *m = dev_or_fail(g);
  if (!m) return;
  ops().ilu(*m, kf_precision());
  m->factored = true;
  m->factor_precision = kf_precision();
  if (!finish(*m, "ComputeNumericalILU")) return;
  if (device_status(*m) == KFUN3D_ERR_PIVOT)
    kf_set_error(KFUN3D_ERR_PIVOT, "singular or non-finite pivot block in ILU(0)");
}

extern "C" void ComputeSparseTriangularSolve(const GEOMETRY *g, const double *b, double *x)
{
  DevMesh *m = dev_or_fail(g);
  if (!m) return;
  const size_t n = 4 * (size_t)m->N;
  h2d(*m, m->rhs, b, n);
  ops().sptrsv(*m, m->rhs, m->t, kf_precision());
  d2h(*m, x, m->t, n);
  if (!finish(*m, "ComputeSparseTriangularSolve")) return;
  if (device_status(*m) == KFUN3D_ERR_TIMEOUT)
    kf_set_error(KFUN3D_ERR_TIMEOUT, "a triangular-solve wait exceeded its bound");
}

extern "C" void ComputeForces(const GEOMETRY *g, double *forces)
{
  DevMesh *m = dev_or_fail(g);
  if (!m) return;
  double u, v;
  kfun3d_get_freestream(&u, &v);
  h2d(*m, m->q, g->q->q, 4 * (size_t)m->N);
  k_forces<<<1, forces_threads(m->ncol), 0, m->stream>>>(m->ncol, m->col, m->wf_nodes, m->xyz, (const double4 *)m->q, u, v, m->forces);
  kf_count_launch();
  d2h(*m, forces, m->forces, 3);
  finish(*m, "ComputeForces");
}

// ---- BLAS-1 on host arrays (inc/utils.h): staged through a device buffer

namespace {

struct Scratch {
  double *buf = nullptr;
  size_t cap = 0;
  cudaStream_t stream = nullptr;
  unsigned *cnt = nullptr;   // CTAs of a reduction that have arrived
  double *ensure(size_t n)
  {
    if (!stream) {
      CK(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
      CK(cudaMalloc(&cnt, sizeof(unsigned)));
      CK(cudaMemsetAsync(cnt, 0, sizeof(unsigned), stream));
    }
    if (n > cap) {
      if (buf) cudaFree(buf);
      cap = std::max(n, (size_t)1 << 16);
      CK(cudaMalloc(&buf, (3 * cap + 4096) * sizeof(double)));
    }
    return buf;
  }
} g_scr;

double blas_reduce(size_t sz, const double *hv, int op)
{
  double *d = g_scr.ensure(sz);
  if (!d) return NAN;
  cudaStream_t s = g_scr.stream;
  double *red = d + 3 * g_scr.cap, out = 0.0;
  CK(cudaMemcpyAsync(d, hv, sz * sizeof(double), cudaMemcpyHostToDevice, s));
  if (kf_mode() == KFUN3D_MODE_FAST) {
    k_dot_fast<<<RED_BLOCKS, 256, 0, s>>>(sz, d, d, red + 8, red, op, g_scr.cnt);
    kf_count_launch();
  } else {
    k_dot_seq<<<1, 256, 0, s>>>(sz, d, d, red, op);
    kf_count_launch();
  }
  CK(cudaMemcpyAsync(&out, red, sizeof(double), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  check_cuda("Compute2ndNorm");
  return out;
}

}  // namespace

extern "C" double Compute2ndNorm(const size_t sz, const double *v) { return blas_reduce(sz, v, 1); }

extern "C" void ComputeAXPY(const size_t sz, const double a, const double *x, double *y)
{
  double *d = g_scr.ensure(sz);
  if (!d) return;
  cudaStream_t s = g_scr.stream;
  CK(cudaMemcpyAsync(d, x, sz * sizeof(double), cudaMemcpyHostToDevice, s));
  CK(cudaMemcpyAsync(d + g_scr.cap, y, sz * sizeof(double), cudaMemcpyHostToDevice, s));
  k_axpy<<<nblk(sz, 256), 256, 0, s>>>(sz, a, d, d + g_scr.cap, kf_mode() == KFUN3D_MODE_FAST);
  kf_count_launch();
  CK(cudaMemcpyAsync(y, d + g_scr.cap, sz * sizeof(double), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  check_cuda("ComputeAXPY");
}

extern "C" void ComputeNewAXPY(const size_t sz, const double a, const double *x, const double *y, double *w)
{
  double *d = g_scr.ensure(sz);
  if (!d) return;
  cudaStream_t s = g_scr.stream;
  CK(cudaMemcpyAsync(d, x, sz * sizeof(double), cudaMemcpyHostToDevice, s));
  CK(cudaMemcpyAsync(d + g_scr.cap, y, sz * sizeof(double), cudaMemcpyHostToDevice, s));
  k_waxpy<<<nblk(sz, 256), 256, 0, s>>>(sz, a, d, d + g_scr.cap, d + 2 * g_scr.cap, kf_mode() == KFUN3D_MODE_FAST);
  kf_count_launch();
  CK(cudaMemcpyAsync(w, d + 2 * g_scr.cap, sz * sizeof(double), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  check_cuda("ComputeNewAXPY");
}

extern "C" double Normalize(const size_t sz, double *x)
{
  double *d = g_scr.ensure(sz);
  if (!d) return NAN;
  cudaStream_t s = g_scr.stream;
  double *red = d + 3 * g_scr.cap, nrm = 0.0;
  CK(cudaMemcpyAsync(d, x, sz * sizeof(double), cudaMemcpyHostToDevice, s));
  if (kf_mode() == KFUN3D_MODE_FAST) {
    k_dot_fast<<<RED_BLOCKS, 256, 0, s>>>(sz, d, d, red + 8, red, 1, g_scr.cnt);
    kf_count_launch();
  } else {
    k_dot_seq<<<1, 256, 0, s>>>(sz, d, d, red, 1);
    kf_count_launch();
  }
  k_scale_inv<<<nblk(sz, 256), 256, 0, s>>>(sz, red, d);
  kf_count_launch();
  CK(cudaMemcpyAsync(x, d, sz * sizeof(double), cudaMemcpyDeviceToHost, s));
  CK(cudaMemcpyAsync(&nrm, red, sizeof(double), cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  check_cuda("Normalize");
  return nrm;
}

// ---- whole solves

extern "C" int kfun3d_solve(GEOMETRY *g, const kfun3d_solver_params *p, kfun3d_step *hist, int max_hist)
{
  DevMesh *m = dev_or_fail(g);
  if (!m) return -1;
  kfun3d_solver_params def;
  if (!p) { kfun3d_default_params(&def); p = &def; }
  h2d(*m, m->q, g->q->q, 4 * (size_t)m->N);
  CK(cudaMemsetAsync(m->lslot, 0, (16 * (size_t)m->nlower + 16) * sizeof(double), m->stream));
  const int n = solve_device(*m, g, p, hist, max_hist, false);
  d2h(*m, g->q->q, m->q, 4 * (size_t)m->N);
  d2h(*m, g->n->cdt, m->cdt, m->N);
  finish(*m, "kfun3d_solve");
  return n;
}

extern "C" void Kernel(GEOMETRY *g)
{
  DevMesh *m = dev_or_fail(g);
  if (!m) return;
  kfun3d_solver_params p;
  kfun3d_default_params(&p);
  h2d(*m, m->q, g->q->q, 4 * (size_t)m->N);
  solve_device(*m, g, &p, nullptr, 0, g_kf_verbose != 0);
  d2h(*m, g->q->q, m->q, 4 * (size_t)m->N);
  d2h(*m, g->n->cdt, m->cdt, m->N);
  finish(*m, "Kernel");
}

// ---- device-resident timing

extern "C" double kfun3d_time_kernel(GEOMETRY *g, int which, int reps)
{
  DevMesh *m = dev_or_fail(g);
  if (!m || reps < 1) return -1.0;
  const Ops o = ops();
  const int prec = kf_precision();
  const size_t n = 4 * (size_t)m->N;
  double u, v;
  kfun3d_get_freestream(&u, &v);
  h2d(*m, m->q, g->q->q, n);
  // a consistent state for the preconditioner and the Krylov vectors
  dev_residual(*m, o, m->q, m->r);
  o.timestep(*m, m->q, 50.0);
  o.fill(*m, m->q, u, v, prec);
  o.ilu(*m, prec);
  dev_reduce(*m, m->q, m->q, m->scal + S_QN, 2, o.fast);
  for (int k = 0; k <= 16; k++) {
    CK(cudaMemcpyAsync(Vb(*m, k), m->r, n * sizeof(double), cudaMemcpyDeviceToDevice, m->stream));
    dev_normalize(*m, Vb(*m, k), m->scal + S_T0, o.fast);
  }
  dev_reduce(*m, Vb(*m, 15), Vb(*m, 15), m->scal + S_VN, 1, o.fast);   // for arnoldi_step
  auto run = [&]() {
    switch (which) {
      case 0: dev_residual(*m, o, m->q, m->r); break;
      case 1: o.timestep(*m, m->q, 50.0); break;
      case 2: o.fill(*m, m->q, u, v, prec); break;
      case 3: o.fill(*m, m->q, u, v, prec); o.ilu(*m, prec); break;
      case 4: o.sptrsv(*m, m->r, m->t, prec); break;
      case 5: arnoldi_step(*m, o, 15, prec); break;
      case 6: orthogonalize(*m, o, 15); break;
      case 7: o.gradient(*m, m->q); break;
      case 8: o.residual(*m, m->q, m->r, kf_first_order(), u, v); break;
      default: break;
    }
  };
  for (int i = 0; i < 2; i++) run();
  cudaEvent_t e0, e1;
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  CK(cudaEventRecord(e0, m->stream));
  for (int i = 0; i < reps; i++) run();
  CK(cudaEventRecord(e1, m->stream));
  CK(cudaEventSynchronize(e1));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (!finish(*m, "kfun3d_time_kernel")) return -1.0;
  return (double)ms / reps;
}

extern "C" int kfun3d_gram_schmidt(const GEOMETRY *g, int k, double *V, double *h)
{
  if (k < 0 || k > KF_NBASIS - 2 || !V || !h) {
    kf_set_error(KFUN3D_ERR_ARG, "kfun3d_gram_schmidt: bad arguments");
    return KFUN3D_ERR_ARG;
  }
  DevMesh *m = dev_or_fail(g);
  if (!m) return kfun3d_gpu_last_status();
  const size_t n = 4 * (size_t)m->N;
  h2d(*m, m->V, V, (k + 2) * n);
  orthogonalize(*m, ops(), k);
  d2h(*m, V + (k + 1) * n, Vb(*m, k + 1), n);
  d2h(*m, h, m->scal, k + 2);
  return finish(*m, "kfun3d_gram_schmidt") ? KFUN3D_OK : kfun3d_gpu_last_status();
}

extern "C" int kfun3d_check_bounded_wait(void)
{
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    kf_set_error(KFUN3D_ERR_NO_DEVICE, "no CUDA device");
    return KFUN3D_ERR_NO_DEVICE;
  }
  return kf_fast::bounded_wait_check(0);
}

extern "C" long kfun3d_matrix_read(const GEOMETRY *g, unsigned int *ia, unsigned int *ja, double *blocks)
{
  MatrixHandle *h = kf_handle(g);
  if (!h) {
    kf_set_error(KFUN3D_ERR_ARG, "GEOMETRY::matrix is not a kfun3d_b200 handle");
    return -1;
  }
  const HostPattern &p = kf_host_pattern(h);
  if (ia) memcpy(ia, p.ia.data(), p.ia.size() * sizeof(unsigned int));
  if (ja) memcpy(ja, p.ja.data(), p.ja.size() * sizeof(unsigned int));
  if (blocks) {
    DevMesh *m = dev_or_fail(g);
    if (!m) return -1;
    if (m->ilu_active) {
      kf_set_error(KFUN3D_ERR_ARG, "kfun3d_matrix_read: the blocks are stored in the spatial ILU order; "
                                   "select the mesh order (kfun3d_set_ilu_order(0)) first");
      return -1;
    }
    const size_t nv = 16 * p.nnz;
    if (kf_precision() == 0) {
      d2h(*m, blocks, m->A, nv);
    } else {
      std::vector<float> tmp(nv);
      CK(cudaMemcpyAsync(tmp.data(), m->Af, nv * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
      CK(cudaStreamSynchronize(m->stream));
      for (size_t i = 0; i < nv; i++) blocks[i] = tmp[i];
    }
    if (!finish(*m, "kfun3d_matrix_read")) return -1;
  }
  return (long)p.nnz;
}

extern "C" double kfun3d_time_solve(GEOMETRY *g, const kfun3d_solver_params *p, int reps, kfun3d_step *hist,
                                    int max_hist, int *nsteps)
{
  DevMesh *m = dev_or_fail(g);
  if (!m || reps < 1) return -1.0;
  kfun3d_solver_params def;
  if (!p) { kfun3d_default_params(&def); p = &def; }
  const size_t n = 4 * (size_t)m->N;
  double *q0 = nullptr;
  CK(cudaMalloc(&q0, n * sizeof(double)));
  if (!q0) return -1.0;
  h2d(*m, q0, g->q->q, n);
  cudaEvent_t e0, e1;
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  double total = 0.0;
  int ns = 0;
  for (int r = 0; r < reps; r++) {
    CK(cudaMemcpyAsync(m->q, q0, n * sizeof(double), cudaMemcpyDeviceToDevice, m->stream));
    CK(cudaMemsetAsync(m->lslot, 0, (16 * (size_t)m->nlower + 16) * sizeof(double), m->stream));
    CK(cudaStreamSynchronize(m->stream));
    CK(cudaEventRecord(e0, m->stream));
    ns = solve_device(*m, g, p, hist, max_hist, false);
    CK(cudaEventRecord(e1, m->stream));
    CK(cudaEventSynchronize(e1));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    total += ms * 1e-3;
    if (ns < 0) break;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(q0);
  if (nsteps) *nsteps = ns;
  if (!finish(*m, "kfun3d_time_solve") || ns < 0) return -1.0;
  return total / reps;
}

// ---- flexible GMRES and the learned preconditioner

extern "C" int kfun3d_solve_flexible(GEOMETRY *g, const kfun3d_solver_params *p, kfun3d_mpnn *net,
                                     kfun3d_step *hist, int max_hist, kfun3d_flex_stats *stats)
{
  DevMesh *m = dev_or_fail(g);
  if (!m) return -1;
  kfun3d_solver_params def;
  if (!p) { kfun3d_default_params(&def); p = &def; }
  h2d(*m, m->q, g->q->q, 4 * (size_t)m->N);
  const int n = solve_flexible(*m, g, p, net, nullptr, hist, max_hist, stats);
  d2h(*m, g->q->q, m->q, 4 * (size_t)m->N);
  d2h(*m, g->n->cdt, m->cdt, m->N);
  if (!finish(*m, "kfun3d_solve_flexible")) return -1;
  return n;
}

extern "C" int kfun3d_collect_pairs(GEOMETRY *g, const kfun3d_solver_params *p, int stride, void *d_x0,
                                    float *d_target, int cap, kfun3d_flex_stats *stats)
{
  if (!d_x0 || !d_target || cap < 0) {
    kf_set_error(KFUN3D_ERR_ARG, "kfun3d_collect_pairs: bad arguments");
    return -1;
  }
  DevMesh *m = dev_or_fail(g);
  if (!m) return -1;
  kfun3d_solver_params def;
  if (!p) { kfun3d_default_params(&def); p = &def; }
  PairSink ps;
  ps.stride = stride;
  ps.x0 = (unsigned char *)d_x0;
  ps.tgt = d_target;
  ps.cap = cap;
  h2d(*m, m->q, g->q->q, 4 * (size_t)m->N);
  const int n = solve_flexible(*m, g, p, nullptr, &ps, nullptr, 0, stats);
  d2h(*m, g->q->q, m->q, 4 * (size_t)m->N);
  d2h(*m, g->n->cdt, m->cdt, m->N);
  if (!finish(*m, "kfun3d_collect_pairs")) return -1;
  return n < 0 ? -1 : ps.count;
}

extern "C" double kfun3d_time_solve_flexible(GEOMETRY *g, const kfun3d_solver_params *p, kfun3d_mpnn *net,
                                             int reps, kfun3d_step *hist, int max_hist, int *nsteps,
                                             kfun3d_flex_stats *stats)
{
  DevMesh *m = dev_or_fail(g);
  if (!m || reps < 1) return -1.0;
  kfun3d_solver_params def;
  if (!p) { kfun3d_default_params(&def); p = &def; }
  const size_t n = 4 * (size_t)m->N;
  double *q0 = nullptr;
  CK(cudaMalloc(&q0, n * sizeof(double)));
  if (!q0) return -1.0;
  h2d(*m, q0, g->q->q, n);
  double total = 0.0;
  int ns = 0;
  for (int r = 0; r < reps; r++) {
    CK(cudaMemcpyAsync(m->q, q0, n * sizeof(double), cudaMemcpyDeviceToDevice, m->stream));
    CK(cudaStreamSynchronize(m->stream));
    kfun3d_flex_stats st{};
    ns = solve_flexible(*m, g, p, net, nullptr, hist, max_hist, &st);
    total += st.seconds;
    if (stats) *stats = st;
    if (ns < 0) break;
  }
  cudaFree(q0);
  if (nsteps) *nsteps = ns;
  if (!finish(*m, "kfun3d_time_solve_flexible") || ns < 0) return -1.0;
  return total / reps;
}

extern "C" double kfun3d_time_learned_apply(GEOMETRY *g, kfun3d_mpnn *net, int reps)
{
  DevMesh *m = dev_or_fail(g);
  if (!m || !net || reps < 1) return -1.0;
  if (!ensure_flex(*m)) return -1.0;
  if (!m->mgraph) m->mgraph = kfun3d_mpnn_graph_create(g);
  if (!m->mgraph || kf_mpnn_prepare(net, m->mgraph) != KFUN3D_OK) return -1.0;
  const Ops o = ops();
  const size_t n = 4 * (size_t)m->N;
  h2d(*m, m->q, g->q->q, n);
  dev_residual(*m, o, m->q, m->fy);   // a residual-like input
  cudaEvent_t e0, e1;
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  kf_mpnn_apply_async(net, m->mgraph, m->fy, m->q, m->t, m->stream);   // warm-up
  CK(cudaEventRecord(e0, m->stream));
  for (int r = 0; r < reps; r++) kf_mpnn_apply_async(net, m->mgraph, m->fy, m->q, m->t, m->stream);
  CK(cudaEventRecord(e1, m->stream));
  CK(cudaEventSynchronize(e1));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (kf_mpnn_status(net, m->stream) != KFUN3D_OK || !finish(*m, "kfun3d_time_learned_apply")) return -1.0;
  return ms / reps;
}
