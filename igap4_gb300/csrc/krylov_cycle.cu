// One GMRES restart cycle as one cooperative kernel: residual, the Arnoldi
// steps (preconditioner, multiply, orthogonalisation, Givens rotation,
// convergence test) and the update of x, the stages separated by grid
// barriers instead of kernel launches (role of KSPSolve with
// KSPGMRESModifiedGramSchmidtOrthogonalization, src/interface.c:228-241).
//
// A lattice of a few thousand control points keeps the GPU busy for a few
// microseconds per stage, so launches bound the cycle: modified Gram-Schmidt
// as a dot product and an update per basis vector took three launches a
// vector, 15,150 in a cycle of 100 steps (85 ms launched one by one at
// 32x8x8, 29 ms as a graph of the 16x4x4 system).  Here
//  * modified Gram-Schmidt runs in its inverse compact WY form (Swirydowicz,
//    Langou, Ananthan, Yang, Thomas, Numer. Linear Algebra Appl. 28 (2021)):
//    the sequential projections (I - v_j v_j^T) ... (I - v_0 v_0^T) w equal
//    w - V h with (I + L) h = V^T w, L the strictly lower triangle of V^T V,
//    so one pass over V gives every dot product with w and, beside it, the
//    new row of L (dot products with v_j); T = (I + L)^-1 grows by one row per
//    step and is kept in every block's shared memory, and h = T V^T w;
//  * opts.orth = 1 (classical Gram-Schmidt twice) runs the same two passes
//    twice with T = I;
//  * the convergence test needs only the last rotated entry of a column, a
//    dot product of the column with one row of the accumulated rotations,
//    which every block carries; the rotations themselves are applied to all
//    columns at once at the end of the cycle.  One warp does the test while
//    the others multiply for the next step; the cycle stops one multiply later
//    than the test, with the same iterate (the chain of rotations per step
//    held up every barrier by 14 k clocks);
//  * three grid barriers a step (3.5 k clocks each): the vector is normalised
//    while the multiply gathers it, the preconditioned copy (Jacobi) having
//    been written beside the update; the block preconditioners take a fourth;
//  * the FP64 pipe (2 FMA per clock and SM) bounds the stages, so cross-lane
//    sums are merged: a warp of the multiply owns the three rows of a control
//    point (one gather of x for three products), a warp of the projection
//    four basis vectors, and the partial sums of several rows or vectors are
//    folded together (9 instead of 40 additions for 8 sums).
//
// Measured: 100 iterations at 32x8x8 (10,200 rows, Jacobi) 86.2 ms as separate
// launches, 3.3 ms here; figures over sizes and restarts at cycle_applies.
//
// One block of 1024 threads per SM (cooperative launch: all blocks resident).
// Data that other blocks wrote are read with plain or L2 loads after the
// barrier (release/acquire at GPU scope), never through the read-only path.
// Every barrier wait is bounded; a block that gives up sets the error word
// and returns, the others see the word and return.
#include <cuda_runtime.h>
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include "common.cuh"
#include "spmv.cuh"
#include "asm_pc.cuh"

namespace igap {

namespace {
constexpr int CY_THREADS = 1024, CY_WARPS = CY_THREADS / 32;
constexpr int CY_VB = 4;             // basis vectors per item of the projection
constexpr int CY_RMAX = 256;         // row chunks per group of vectors
constexpr int CY_MAX_RESTART = 200;  // T (m (m - 1) / 2 doubles) in shared memory
constexpr uint32_t CY_WAIT_LIMIT = 1u << 24;

struct CycleState {
  int its;        // Arnoldi steps of this cycle
  double beta;    // |r| at the start of the cycle
  double rnorm;   // residual estimate
  double rnorm0;  // |r| of the first cycle (negative before it)
  double tol;
};

struct CycleArgs {  // w: two buffers, one the current vector, the other its product
  const int64_t *rowptr;
  const int32_t *cols;
  const double *vals;
  const double *b;
  double *x, *w, *wd, *V, *Z;  // wd: the current vector times the reciprocal diagonal (no or scalar preconditioner)
  const double *pcd;   // Jacobi: reciprocal diagonal; block preconditioners: their blocks
  double *H;           // [m][m + 1] columns
  double *y;
  double *part;        // projection partial sums [2][vectors][CY_RMAX]
  double *npart;       // norm partial sums [2][blocks]
  CycleState *st;
  unsigned *bar;       // arrivals at the grid barrier
  int *err;
  CellGeom cg;
  int64_t n;
  int m, steps, pc, orth;
  double rtol, abstol, dtol;
};

struct CycleSmem {
  double red[CY_THREADS];
  double r[CY_MAX_RESTART + 1], l[CY_MAX_RESTART + 1], h[CY_MAX_RESTART + 1];
  // rotations, their diagonal, the rotated right-hand side, the last row of the accumulated rotations
  double cs[CY_MAX_RESTART + 1], sn[CY_MAX_RESTART + 1], den[CY_MAX_RESTART + 1], g[CY_MAX_RESTART + 2],
      q[CY_MAX_RESTART + 2];
  double bc;           // a broadcast sum
  int ok, stop;
  // packed rows of T (row i: entries c < i at i (i - 1) / 2) follow; at the end
  // of the cycle packed columns of H (column c: entries i <= c at c (c + 1) / 2)
};

// All blocks arrive and wait.  Fences at GPU scope by thread 0 (one before the
// arrival, one after the relaxed polls), the block barriers around them order
// the other threads.
__device__ __forceinline__ bool grid_sync(const CycleArgs &a, CycleSmem &S, unsigned &target)
{
  __syncthreads();
  target += gridDim.x;
  if (threadIdx.x == 0) {
    asm volatile("fence.acq_rel.gpu;\n\tred.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
    int ok = 0;
    for (uint32_t it = 0; it < CY_WAIT_LIMIT; it++) {
      unsigned v;
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.bar) : "memory");
      if ((int)(v - target) >= 0) {
        ok = 1;
        break;
      }
      if ((it & 1023u) == 1023u && *(volatile int *)a.err) break;
    }
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    if (!ok) atomicExch(a.err, 4);
    S.ok = ok;
  }
  __syncthreads();
  return S.ok != 0;
}

// Sum of s over the first `warps` warps of the block (the others hold none) in
// a fixed order: through shared memory, then one warp.  Valid in thread 0.
__device__ __forceinline__ double block_sum(CycleSmem &S, double s, int warps)
{
  if (threadIdx.x < 32 * warps) S.red[threadIdx.x] = s;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x < 32) {
#pragma unroll 4
    for (int k = 0; k < warps; k++) t += S.red[threadIdx.x + 32 * k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  }
  return t;
}

// Square root of the sum of the blocks' partial sums, by every block in the
// same order.
__device__ __forceinline__ double total_norm(const CycleArgs &a, CycleSmem &S, int slot)
{
  if (threadIdx.x < 32) {
    double t = 0.0;
    for (unsigned k = threadIdx.x; k < gridDim.x; k += 32) t += __ldcg(a.npart + slot * gridDim.x + k);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (threadIdx.x == 0) S.bc = sqrt(t);
  }
  __syncthreads();
  return S.bc;
}

// Three sums over the lanes of a group of G lanes (16 or 32): the first two
// steps exchange, so that the quarters of the group carry different sums (6
// instead of 15 additions at G = 32).  Returns this lane's sum; `which` tells
// which of the three it is (3: none).
template <int G>
__device__ __forceinline__ double fold3(double s0, double s1, double s2, int sub, int &which)
{
  constexpr int A = G / 2, B = G / 4;
  const bool up = sub & A;
  // upper half keeps s2 (and an empty slot), lower half s0 and s1
  double k0 = up ? s2 : s0, k1 = up ? 0.0 : s1;
  const double g0 = up ? s0 : s2, g1 = up ? s1 : 0.0;
  k0 += __shfl_xor_sync(0xffffffffu, g0, A);
  k1 += __shfl_xor_sync(0xffffffffu, g1, A);
  const bool up2 = sub & B;
  double v = up2 ? k1 : k0;
  v += __shfl_xor_sync(0xffffffffu, up2 ? k0 : k1, B);
#pragma unroll
  for (int o = G / 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  which = up ? (up2 ? 3 : 2) : (up2 ? 1 : 0);
  return v;
}

// w = scale A x (or w = b - A x and wd = M^-1 w with RES) over this grid's
// groups of G lanes, one control point (three rows sharing their columns) per
// group; returns this thread's part of |w|^2 with RES.
template <int G, bool RES>
__device__ __forceinline__ double multiply(const CycleArgs &a, const double *x, double *w, double scale)
{
  const int64_t ncp = a.n / 3;
  const int sub = threadIdx.x % G;
  const int64_t ng = (int64_t)gridDim.x * (CY_THREADS / G);
  double nn = 0.0;
  // consecutive groups of one block take control points a grid apart: every
  // SM gets the same share when there are fewer points than groups
  for (int64_t c0 = blockIdx.x + (int64_t)gridDim.x * (threadIdx.x / 32 * (32 / G)); c0 < ncp; c0 += ng) {
    const int64_t cp = c0 + (int64_t)gridDim.x * ((threadIdx.x % 32) / G);
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    if (cp < ncp) {
      const int64_t r0 = __ldg(a.rowptr + 3 * cp), r1 = __ldg(a.rowptr + 3 * cp + 1);
      const int len = (int)(r1 - r0);
      const double *v0 = a.vals + r0, *v1 = v0 + len, *v2 = v1 + len;
      const int32_t *col = a.cols + r0;
#pragma unroll 4
      for (int k = sub; k < len; k += G) {
        const double xv = x[__ldg(col + k)];
        s0 = fma(__ldg(v0 + k), xv, s0);
        s1 = fma(__ldg(v1 + k), xv, s1);
        s2 = fma(__ldg(v2 + k), xv, s2);
      }
    }
    int which;
    double v = fold3<G>(s0, s1, s2, sub, which);
    if (cp < ncp && which < 3 && (sub & (G / 4 - 1)) == 0) {
      const int64_t row = 3 * cp + which;
      if (RES) {
        v = a.b[row] - v;
        nn = fma(v, v, nn);
        if (a.pc <= 1) a.wd[row] = a.pc ? v * __ldg(a.pcd + row) : v;
      } else {
        v *= scale;
      }
      w[row] = v;
    }
  }
  return nn;
}

template <bool RES>
__device__ __forceinline__ double multiply_any(const CycleArgs &a, const double *x, double *w, double scale)
{
  // 32 lanes a control point while there are fewer points than groups of 16
  return a.n / 3 < (int64_t)gridDim.x * CY_WARPS * 2 ? multiply<32, RES>(a, x, w, scale)
                                                     : multiply<16, RES>(a, x, w, scale);
}

// Folds NS sums (4 or 8) over the lanes of a warp: each exchange halves the
// number of sums a lane carries (NS - 1 additions, then one per remaining
// step).  s[0] becomes sum number `id` in every lane; the lanes with
// (lane & (32 / NS - 1)) == 0 name each once.
template <int NS>
__device__ __forceinline__ int fold(double (&s)[2 * CY_VB], int lane)
{
  int id = 0;
#pragma unroll
  for (int o = 16, cnt = NS; o > 0; o >>= 1) {
    if (cnt > 1) {
      const bool up = lane & o;
#pragma unroll
      for (int q = 0; q < cnt / 2; q++) {
        const double keep = up ? s[q + cnt / 2] : s[q], give = up ? s[q] : s[q + cnt / 2];
        s[q] = keep + __shfl_xor_sync(0xffffffffu, give, o);
      }
      if (up) id += cnt / 2;
      cnt /= 2;
    } else {
      s[0] += __shfl_xor_sync(0xffffffffu, s[0], o);
    }
  }
  return id;
}

// Partial dot products of the basis vectors 0..j with w (and, with LROW, with
// v_j): item (group of CY_VB vectors, row chunk) per warp.
template <bool LROW>
__device__ __forceinline__ void project_partial(const CycleArgs &a, const double *w, int j, int R)
{
  const int lane = threadIdx.x & 31;
  const int ngroup = (j + CY_VB) / CY_VB;
  const int64_t chunk = (a.n + R - 1) / R;
  const double *vj = a.V + (size_t)j * a.n;
  for (int it = blockIdx.x + gridDim.x * (threadIdx.x >> 5); it < ngroup * R; it += gridDim.x * CY_WARPS) {
    const int i0 = (it / R) * CY_VB, r = it % R;
    const int64_t lo = r * chunk, hi = lo + chunk < a.n ? lo + chunk : a.n;
    const double *v[CY_VB];
#pragma unroll
    for (int q = 0; q < CY_VB; q++) v[q] = a.V + (size_t)min(i0 + q, j) * a.n;
    double s[2 * CY_VB];
#pragma unroll
    for (int q = 0; q < 2 * CY_VB; q++) s[q] = 0.0;
#pragma unroll 2
    for (int64_t k = lo + lane; k < hi; k += 32) {
      const double wk = __ldcg(w + k);
      const double vk = LROW ? __ldcg(vj + k) : 0.0;
#pragma unroll
      for (int q = 0; q < CY_VB; q++) {
        const double u = __ldcg(v[q] + k);
        s[q] = fma(u, wk, s[q]);
        if (LROW) s[CY_VB + q] = fma(u, vk, s[CY_VB + q]);
      }
    }
    constexpr int NS = LROW ? 8 : 4;
    const int id = fold<NS>(s, lane);
    const int q = id % CY_VB, kind = id / CY_VB;
    if ((lane & (32 / NS - 1)) == 0 && i0 + q <= j)
      a.part[((size_t)kind * (a.m + 1) + i0 + q) * CY_RMAX + r] = s[0];
  }
}

// Sums the partial dot products into S.r (with w) and S.l (with v_j).
template <bool LROW>
__device__ __forceinline__ void project_total(const CycleArgs &a, CycleSmem &S, int j, int R)
{
  const int lane = threadIdx.x & 31;
  constexpr int NS = LROW ? 8 : 4;
  for (int g = threadIdx.x >> 5; g * CY_VB <= j; g += CY_WARPS) {
    double s[2 * CY_VB];
#pragma unroll
    for (int q = 0; q < 2 * CY_VB; q++) s[q] = 0.0;
    const double *p[NS];
#pragma unroll
    for (int q = 0; q < NS; q++)
      p[q] = a.part + ((size_t)(q / CY_VB) * (a.m + 1) + min(g * CY_VB + q % CY_VB, j)) * CY_RMAX;
    for (int r = lane; r < R; r += 32) {
      double t[NS];  // every sum's load in flight at once
#pragma unroll
      for (int q = 0; q < NS; q++) t[q] = __ldcg(p[q] + r);
#pragma unroll
      for (int q = 0; q < NS; q++) s[q] += t[q];
    }
    const int id = fold<NS>(s, lane), i = g * CY_VB + id % CY_VB;
    if ((lane & (32 / NS - 1)) == 0 && i <= j) (id < CY_VB ? S.r : S.l)[i] = s[0];
  }
  __syncthreads();
}

__device__ __forceinline__ double *t_row(CycleSmem &S, int i)
{
  return reinterpret_cast<double *>(&S + 1) + (size_t)i * (i - 1) / 2;
}

// Row j of T = (I + L)^-1 and h = T r, redundantly in every block.
__device__ __forceinline__ void solve_t(CycleSmem &S, int j)
{
  const int width = (j + 32) & ~31;             // threads per slice of the sums
  const int ns = min(8, CY_THREADS / width);    // slices: their sums are a serial chain
  const int c = threadIdx.x % width, sl = threadIdx.x / width;
  // t_j[c] = -(l_c + sum_{c < k < j} l_k T[k][c])
  double s = 0.0;
  if (sl < ns && c < j)
    for (int k = c + 1 + sl; k < j; k += ns) s = fma(S.l[k], t_row(S, k)[c], s);
  if (sl < ns) S.red[sl * width + c] = s;
  __syncthreads();
  if (threadIdx.x < j) {
    double t = S.l[threadIdx.x];
    for (int q = 0; q < ns; q++) t += S.red[q * width + threadIdx.x];
    t_row(S, j)[threadIdx.x] = -t;
  }
  __syncthreads();
  // h_i = r_i + sum_{c < i} T[i][c] r_c
  s = 0.0;
  if (sl < ns && c <= j)
    for (int k = sl; k < c; k += ns) s = fma(t_row(S, c)[k], S.r[k], s);
  if (sl < ns) S.red[sl * width + c] = s;
  __syncthreads();
  if (threadIdx.x <= j) {
    double t = S.r[threadIdx.x];
    for (int q = 0; q < ns; q++) t += S.red[q * width + threadIdx.x];
    S.h[threadIdx.x] = t;
  }
  __syncthreads();
}

// w -= V h on this block's rows (h = hs) and wd = M^-1 w; returns this thread's
// part of |w|^2, held by the first `warps` warps.  With fewer rows than threads
// the basis vectors are split over ns threads a row and their sums joined
// through shared memory.
__device__ __forceinline__ double update_w(const CycleArgs &a, CycleSmem &S, double *w, const double *hs, int j,
                                           int &warps)
{
  const int64_t per = (a.n + gridDim.x - 1) / gridDim.x;
  const int64_t lo = (int64_t)blockIdx.x * per, hi = lo + per < a.n ? lo + per : a.n;
  double nn = 0.0;
  int width = 32;
  while (width < per && width < CY_THREADS) width *= 2;
  warps = width / 32;
  const int ns = CY_THREADS / width < 8 ? CY_THREADS / width : 8;
  if (ns == 1) {
    for (int64_t r = lo + threadIdx.x; r < hi; r += CY_THREADS) {
      double s = __ldcg(w + r);
#pragma unroll 8
      for (int i = 0; i <= j; i++) s = fma(-hs[i], __ldcg(a.V + (size_t)i * a.n + r), s);
      w[r] = s;
      if (a.pc <= 1) a.wd[r] = a.pc ? s * __ldg(a.pcd + r) : s;
      nn = fma(s, s, nn);
    }
    return nn;
  }
  const int c = threadIdx.x % width, sl = threadIdx.x / width;
  const int64_t r = lo + c;
  if (sl < ns) {
    double s = 0.0;
    if (r < hi) {
#pragma unroll 4
      for (int i = sl; i <= j; i += ns) s = fma(hs[i], __ldcg(a.V + (size_t)i * a.n + r), s);
    }
    S.red[sl * width + c] = s;
  }
  __syncthreads();
  if (sl == 0 && r < hi) {
    double s = __ldcg(w + r);
    for (int q = 0; q < ns; q++) s -= S.red[q * width + c];
    w[r] = s;
    if (a.pc <= 1) a.wd[r] = a.pc ? s * __ldg(a.pcd + r) : s;
    nn = s * s;
  }
  __syncthreads();
  return nn;
}

// v = inv w on this block's rows.
__device__ __forceinline__ void normalise(const CycleArgs &a, const double *w, double inv, double *v)
{
  const int64_t per = (a.n + gridDim.x - 1) / gridDim.x;
  const int64_t lo = (int64_t)blockIdx.x * per, hi = lo + per < a.n ? lo + per : a.n;
  for (int64_t r = lo + threadIdx.x; r < hi; r += CY_THREADS) v[r] = __ldcg(w + r) * inv;
}

__device__ __forceinline__ void block_precondition(const CycleArgs &a, const double *v, double *z, double scale)
{
  if (a.pc == 2) bdiag_apply(z, v, a.pcd, a.n / 3, scale);
  else if (a.pc == 3) cblock_apply(z, v, a.pcd, a.cg, cell_count(a.cg), scale);
  else asm_apply(z, v, reinterpret_cast<const float *>(a.pcd), a.cg, cell_count(a.cg), scale);
}

// Rotation of Hessenberg column j (S.h, norm hn below it) and the convergence
// test, by one warp of every block: the column's last rotated entry is
// q . h with q the last row of the accumulated rotations.
__device__ __forceinline__ void rotate(CycleSmem &S, int j, double hn, double tol)
{
  const int lane = threadIdx.x & 31;
  double hi = 0.0;
  for (int i = lane; i <= j; i += 32) hi = fma(S.q[i], S.h[i], hi);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) hi += __shfl_xor_sync(0xffffffffu, hi, o);
  double den = hypot(hi, hn);
  const bool breakdown = !(den > 0.0) || !isfinite(den);
  if (breakdown) den = 1e-300;
  const double c = hi / den, s = hn / den;
  for (int i = lane; i <= j; i += 32) S.q[i] *= -s;
  if (lane == 0) {
    S.q[j + 1] = c;
    S.cs[j] = c;
    S.sn[j] = s;
    S.den[j] = den;
    const double gj = S.g[j], gn = -s * gj;
    S.g[j] = c * gj;
    S.g[j + 1] = gn;
    S.stop = (fabs(gn) <= tol || breakdown || !isfinite(gn)) ? 1 : 0;
  }
}

// y = R^-1 g of the k columns by one block: the columns of H to shared memory,
// every thread rotates one, one warp substitutes backwards.
__device__ void backsolve(const CycleArgs &a, CycleSmem &S, int k)
{
  double *R = reinterpret_cast<double *>(&S + 1);
  __syncthreads();
  for (int c = threadIdx.x >> 5; c < k; c += CY_WARPS)
    for (int i = threadIdx.x & 31; i <= c; i += 32) R[c * (c + 1) / 2 + i] = __ldcg(a.H + (size_t)c * (a.m + 1) + i);
  __syncthreads();
  if (threadIdx.x < k) {
    const int c = threadIdx.x;
    double *col = R + c * (c + 1) / 2, hi = col[0];
    for (int i = 0; i < c; i++) {
      const double hn = col[i + 1];
      col[i] = fma(S.sn[i], hn, S.cs[i] * hi);
      hi = fma(-S.sn[i], hi, S.cs[i] * hn);
    }
    S.den[c] = 1.0 / S.den[c];
    S.h[c] = S.g[c];
  }
  __syncthreads();
  if (threadIdx.x < 32)
    for (int c = k - 1; c >= 0; c--) {
      const double *col = R + c * (c + 1) / 2;
      const double y = S.h[c] * S.den[c];
      __syncwarp();
      for (int i = threadIdx.x; i < c; i += 32) S.h[i] = fma(-col[i], y, S.h[i]);
      if (threadIdx.x == 0) a.y[c] = y;
      __syncwarp();
    }
}

__global__ void __launch_bounds__(CY_THREADS, 1) gmres_cycle_kernel(CycleArgs a)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  CycleSmem &S = *reinterpret_cast<CycleSmem *>(smem_raw);
  unsigned target = 0;
  const int tid = threadIdx.x, warp = tid >> 5;
  const bool last_block = blockIdx.x == gridDim.x - 1;
  CycleState *st = a.st;
  double *wcur = a.w, *wnext = a.w + a.n;
  // r = b - A x, beta = |r|
  {
    const double nn = block_sum(S, multiply_any<true>(a, a.x, wcur, 1.0), CY_WARPS);
    if (tid == 0) a.npart[blockIdx.x] = nn;
  }
  if (!grid_sync(a, S, target)) return;
  const double beta = total_norm(a, S, 0);
  const double rnorm0 = st->rnorm0 < 0.0 ? beta : st->rnorm0;
  const double tol = st->rnorm0 < 0.0 ? fmax(a.rtol * beta, a.abstol) : st->tol;
  const bool go = beta > tol && isfinite(beta) && !(beta > a.dtol * rnorm0) && a.steps > 0;
  if (!grid_sync(a, S, target)) return;  // every block has read rnorm0 and tol
  if (last_block && tid == 0) {
    st->rnorm0 = rnorm0;
    st->tol = tol;
    st->beta = st->rnorm = beta;
    st->its = 0;
  }
  if (!go) return;
  if (tid == 0) {
    S.g[0] = beta;
    S.q[0] = 1.0;
    S.stop = 0;
  }
  int k = 0;
  double den = beta;
  for (int j = 0; j < a.steps; j++) {
    double *vj = a.V + (size_t)j * a.n, *zj = a.Z + (size_t)j * a.n;
    const double inv = 1.0 / den;
    if (a.pc >= 2) {
      block_precondition(a, wcur, zj, inv);
      normalise(a, wcur, inv, vj);
      if (!grid_sync(a, S, target)) return;
    } else {
      normalise(a, wcur, inv, vj);
    }
    // the previous column's test beside the multiply
    if (j > 0 && warp == CY_WARPS - 1) rotate(S, j - 1, den, tol);
    multiply_any<false>(a, a.pc >= 2 ? zj : a.wd, wnext, a.pc >= 2 ? 1.0 : inv);
    if (!grid_sync(a, S, target)) return;
    if (S.stop) {
      k = j;
      break;
    }
    // orthogonalise
    const int ngroup = (j + CY_VB) / CY_VB;
    int R = (int)(gridDim.x * CY_WARPS) / ngroup;
    const int64_t rmax = (a.n + 159) / 160;  // at least five rows a lane: fewer partial sums for every block to add
    R = R < CY_RMAX ? R : CY_RMAX;
    R = R < rmax ? R : (int)rmax;
    R = R > 0 ? R : 1;
    double nn;
    int warps;
    if (a.orth == 1) {
      project_partial<false>(a, wnext, j, R);
      if (!grid_sync(a, S, target)) return;
      project_total<false>(a, S, j, R);
      update_w(a, S, wnext, S.r, j, warps);
      if (tid <= j) S.h[tid] = S.r[tid];
      if (!grid_sync(a, S, target)) return;
      project_partial<false>(a, wnext, j, R);
      if (!grid_sync(a, S, target)) return;
      project_total<false>(a, S, j, R);
      nn = update_w(a, S, wnext, S.r, j, warps);
      if (tid <= j) S.h[tid] += S.r[tid];
    } else {
      project_partial<true>(a, wnext, j, R);
      if (!grid_sync(a, S, target)) return;
      project_total<true>(a, S, j, R);
      solve_t(S, j);
      nn = update_w(a, S, wnext, S.h, j, warps);
    }
    nn = block_sum(S, nn, warps);
    if (tid == 0) a.npart[gridDim.x * (1 + (j & 1)) + blockIdx.x] = nn;
    if (last_block && tid <= j) a.H[(size_t)j * (a.m + 1) + tid] = S.h[tid];
    if (!grid_sync(a, S, target)) return;
    den = total_norm(a, S, 1 + (j & 1));
    double *t = wcur;
    wcur = wnext;
    wnext = t;
    k = j + 1;
  }
  // the last column of a full cycle has not been rotated yet
  if (!S.stop && warp == CY_WARPS - 1) rotate(S, k - 1, den, tol);
  __syncthreads();
  // x += M^-1 V y
  if (last_block) {
    backsolve(a, S, k);
    if (tid == 0) {
      st->its = k;
      st->rnorm = fabs(S.g[k]);
    }
  }
  if (!isfinite(S.g[k])) return;  // breakdown: every block holds this value; x stays as the last cycle left it
  if (!grid_sync(a, S, target)) return;
  for (int i = tid; i < k; i += CY_THREADS) S.h[i] = __ldcg(a.y + i);
  __syncthreads();
  const double *B = a.pc >= 2 ? a.Z : a.V;
  for (int64_t r = (int64_t)blockIdx.x + (int64_t)gridDim.x * tid; r < a.n; r += (int64_t)gridDim.x * CY_THREADS) {
    double s = 0.0;
#pragma unroll 4
    for (int i = 0; i < k; i++) s = fma(S.h[i], __ldcg(B + (size_t)i * a.n + r), s);
    a.x[r] += a.pc == 1 ? s * __ldg(a.pcd + r) : s;
  }
}

__global__ void diag_reciprocal_kernel(const int64_t *rowptr, const int32_t *cols, const double *vals, double *inv,
                                       int64_t n)
{
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  int64_t lo = rowptr[r], hi = rowptr[r + 1];
  const int64_t end = hi;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (cols[mid] < r) lo = mid + 1;
    else hi = mid;
  }
  const double d = (lo < end && cols[lo] == r) ? vals[lo] : 0.0;
  inv[r] = d != 0.0 ? 1.0 / d : 1.0;  // a zero diagonal counts as 1, as PCJACOBI
}
}  // namespace

struct CycleWork {
  int m = 0, grid = 0;
  double *buf = nullptr;      // H, y, partial sums
  unsigned *ctl = nullptr;    // barrier counter, error word (128 B apart), state
  CycleState *h_st = nullptr; // pinned: state and error word
};

void cycle_release(Context *c)
{
  CycleWork *cw = c->cycle;
  if (!cw) return;
  if (cw->buf) cudaFree(cw->buf);
  if (cw->ctl) cudaFree(cw->ctl);
  if (cw->h_st) cudaFreeHost(cw->h_st);
  delete cw;
  c->cycle = nullptr;
}

constexpr size_t CY_CTL_BYTES = 256 + sizeof(CycleState);

static int ensure_cycle(Context *c, int m)
{
  if (c->cycle && c->cycle->m >= m) return IGAPGPU_OK;
  cycle_release(c);
  CycleWork *cw = new CycleWork();
  c->cycle = cw;
  int dev = 0, grid = 0;
  IGAP_CUDA(cudaGetDevice(&dev));
  IGAP_CUDA(cudaDeviceGetAttribute(&grid, cudaDevAttrMultiProcessorCount, dev));
  const char *env = getenv("IGAPGPU_GMRES_CYCLE");
  if (env && atoi(env) > 0) grid = atoi(env);
  const size_t cnt = (size_t)(m + 1) * m + (size_t)(m + 1) + 2 * (size_t)(m + 1) * CY_RMAX + 3 * (size_t)grid;
  if (room_malloc(c, &cw->buf, sizeof(double) * cnt) != cudaSuccess || room_malloc(c, &cw->ctl, CY_CTL_BYTES) != cudaSuccess ||
      cudaMallocHost(&cw->h_st, CY_CTL_BYTES) != cudaSuccess) {
    cudaGetLastError();
    cycle_release(c);
    set_error("GMRES cycle workspace (restart %d) does not fit", m);
    return IGAPGPU_ERR_NOMEM;
  }
  cw->m = m;
  cw->grid = grid;
  return IGAPGPU_OK;
}

static size_t cycle_smem(int m) { return sizeof(CycleSmem) + sizeof(double) * ((size_t)m * (m + 1) / 2); }

// Whether the cycle kernel takes this solve: T fits in shared memory, the
// multiply is in FP64 (IGAPGPU_SPMV_DF keeps the separate kernels), and the grid
// can be resident at once (a process limited to part of the SMs falls back, or
// names its blocks: IGAPGPU_GMRES_CYCLE=blocks; 0 keeps the separate kernels).
//
// Size and restart: the cycle saves launches and passes over the basis, both
// growing with the step number, and loses on the multiply once the matrix is far
// beyond L2 (every stage waits for the slowest SM, where the separate multiply's
// blocks are handed out as SMs come free).  Separate / cycle, ms:
//   one lattice   64x16x16 (64 k rows)    restart 5   1.02 /  0.68, 30  10.6 /  2.9, 100   88 /  11
//                 128x32x32 (451 k)                   3.27 /  3.01,     21.5 / 13.9,      132 /  51
//                 192x48x48 (1.46 M)                  8.90 /  8.99,     48.1 / 42.6,      227 / 157
//                 256x64x64 (3.37 M)      10  34.5 / 36.3, 20  66.3 / 67.6, 30  101 / 99, 100  431 / 364
//   batches       88 k rows               faster at every restart
//   (generic      366 k                   5   2.39 /  2.33, 30  16.6 / 10.9
//    multiply)    821 k, graphs           10  saves -0.5 of 6, 30  1.6 of 23
//                 4.56 M                  10  37.7 / 45.1, 60  249 / 256, 100  483 / 461
//   batches with CGS2 (graphs, whose two block passes are cheap):
//                 366 k                   10 -0.16 of 3.8, 30 -0.05 of 11, 60  0.7 of 24
//                 821 k                   30 -1.5 of 21, 60 -1.4 of 48
// so the shortest restart it takes grows with the rows.  IGAPGPU_GMRES_CYCLE=blocks
// overrides the line.
bool cycle_applies(const Context *c, int m, int orth)
{
  const char *env = getenv("IGAPGPU_GMRES_CYCLE");
  if (m > CY_MAX_RESTART || spmv_df(c) || c->cycle_unfit || (env && env[0] == '0')) return false;
  if (c->ndof < 200000 || (env && atoi(env) > 0)) return true;
  const double rows = 1e-6 * (double)c->ndof;
  const double line = c->batch ? (orth == 1 ? 110.0 * rows : fmin(22.0 * rows, 75.0)) : fmin(3.0 * rows * rows, 75.0);
  return m >= line;
}

// GMRES cycles on the context matrix; b, x device vectors, pcd the
// preconditioner's data, V and Z the basis buffers, w 2 n and wd n scratch.  `cap`: stop at ksp_max_it
// inside a cycle and return the true residual norm (else whole cycles and the
// recurrence's estimate).
int ksp_cycles(Context *c, const double *b, double *x, const igapgpu_solver_opts *o, int m, int pc, const double *pcd,
               double *V, double *Z, double *w, double *wd, bool cap, int *its_out, double *rnorm_out)
{
  int r = ensure_cycle(c, m);
  if (r) return r;
  CycleWork *cw = c->cycle;
  CycleArgs a;
  memset(&a, 0, sizeof a);
  a.rowptr = c->d_rowptr;
  a.cols = c->d_cols;
  a.vals = c->d_vals;
  a.b = b;
  a.x = x;
  a.w = w;
  a.wd = wd;
  a.V = V;
  a.Z = Z;
  a.pcd = pcd;
  a.H = cw->buf;
  a.y = a.H + (size_t)(cw->m + 1) * cw->m;
  a.part = a.y + cw->m + 1;
  a.npart = a.part + 2 * (size_t)(cw->m + 1) * CY_RMAX;
  a.bar = cw->ctl;
  a.err = reinterpret_cast<int *>(cw->ctl + 32);
  a.st = reinterpret_cast<CycleState *>(cw->ctl + 64);
  a.cg = cell_geom(c);
  a.n = c->ndof;
  a.m = m;
  a.pc = pc;
  a.orth = !cap && o->orth == 1 ? 1 : 0;
  a.rtol = o->ksp_rtol;
  a.abstol = o->ksp_abstol;
  a.dtol = o->ksp_dtol;
  const size_t smem = cycle_smem(m);
  IGAP_CUDA(cudaFuncSetAttribute(gmres_cycle_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cycle_smem(CY_MAX_RESTART)));
  CycleState h0;
  memset(&h0, 0, sizeof h0);
  h0.rnorm0 = -1.0;
  IGAP_CUDA(cudaMemcpyAsync(a.st, &h0, sizeof h0, cudaMemcpyHostToDevice, c->stream));
  int its = 0;
  double rnorm = 0.0;
  for (;;) {
    a.steps = m;
    if (cap && o->ksp_max_it - its < m) a.steps = o->ksp_max_it - its > 0 ? o->ksp_max_it - its : 0;
    IGAP_CUDA(cudaMemsetAsync(cw->ctl, 0, 256, c->stream));
    void *params[] = {&a};
    const cudaError_t e = cudaLaunchCooperativeKernel((const void *)gmres_cycle_kernel, dim3(cw->grid), dim3(CY_THREADS),
                                                      params, smem, c->stream);
    if (its == 0 && (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported)) {
      cudaGetLastError();
      c->cycle_unfit = true;
      return CYCLE_UNFIT;
    }
    IGAP_CUDA(e);
    count_launch();
    IGAP_CUDA(cudaMemcpyAsync(cw->h_st, cw->ctl, CY_CTL_BYTES, cudaMemcpyDeviceToHost, c->stream));
    IGAP_CUDA(cudaStreamSynchronize(c->stream));
    const unsigned *ctl = reinterpret_cast<const unsigned *>(cw->h_st);
    if (ctl[32]) {
      set_error("GMRES: a bounded grid barrier wait expired (code %u)", ctl[32]);
      return IGAPGPU_ERR_TIMEOUT;
    }
    CycleState st;
    memcpy(&st, ctl + 64, sizeof st);
    its += st.its;
    rnorm = st.rnorm;
    if (!isfinite(rnorm) || !isfinite(st.beta)) {
      set_error("GMRES: non-finite residual norm");
      return IGAPGPU_ERR_NUMERIC;
    }
    const bool met = rnorm <= st.tol, out_of_its = its >= o->ksp_max_it;
    // the step limit and the tolerance are looked at before the divergence
    // test when the limit is exact, after it in whole cycles
    if (cap && st.its == 0 && (met || out_of_its)) break;
    if (st.rnorm0 > 0 && st.beta > o->ksp_dtol * st.rnorm0) {
      set_error("GMRES diverged (dtol)");
      return IGAPGPU_ERR_NUMERIC;
    }
    if (met || out_of_its || st.its == 0) {
      if (cap) {  // true residual of the final iterate
        if ((r = spmv(c, c->d_vals, x, w))) return r;
        if ((r = dev_diff_norm2(c, b, w, &rnorm))) return r;
      }
      break;
    }
  }
  if (its_out) *its_out = its;
  if (rnorm_out) *rnorm_out = rnorm;
  return IGAPGPU_OK;
}

int launch_diag_reciprocal(Context *c, double *inv)
{
  diag_reciprocal_kernel<<<(unsigned)((c->ndof + 255) / 256), 256, 0, c->stream>>>(c->d_rowptr, c->d_cols, c->d_vals, inv,
                                                                                   c->ndof);
  count_launch();
  IGAP_CHECK_LAUNCH();
  return IGAPGPU_OK;
}

}  // namespace igap
