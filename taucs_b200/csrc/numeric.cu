// FP64 multifrontal numeric factorization on sm_100a.
//
// The reference factors one front at a time in a depth-first recursion
// (src/taucs_sn_llt.c:1829-1977): calloc F1/F2/U, extend-add each child
// (:1200-1240), assemble A's columns (:1099-1119), then LAPACK/BLAS POTRF
// (:1131), TRSM (:1150) and SYRK (:1180).  Here every front of one level of
// the supernodal tree is processed by the same launches:
//
//   k_small_persistent  the small fronts with only small fronts below them,
//                   all levels in one launch from a device-side queue;
//   k_small_front   the other fronts of order <= SMALL_F_MAX: one CTA builds the whole
//                   front in shared memory (zero + assemble + extend-add),
//                   factors it (right-looking partial Cholesky of the first s
//                   columns, i.e. POTRF+TRSM+SYRK fused) and writes the panel
//                   and the update matrix once;
//   k_build         larger fronts: one CTA per 128x32 tile of the front's lower
//                   part gathers A's entries (shared-memory atomic adds:
//                   duplicate entries are summed) and the children's update
//                   matrices in a fixed child order into shared memory and
//                   writes the tile once;
//   k_panel         blocked partial Cholesky, step kb: one launch factors
//                   the 128x128 diagonal block (one CTA per front) and applies
//                   it to every row below it (a CTA per 64 to 256 rows,
//                   following it piece by piece);
//   k_gemm          C -= A B^T on DMMA (mma.sync m16n8k8 f64) tiles: the
//                   panel updates of a recursive (left half, GEMM, right
//                   half) panel factorization, and the update matrix
//                   U -= L21 L21^T with k = s at the end;
//   k_dinv          after all levels, the inverses of every big front's
//                   64x64 diagonal blocks (used by the solve).
//
// Every kernel first reads the status word and returns when an earlier front
// hit a nonpositive pivot; the smallest failing global column is recorded
// with atomicMin (the reference reports the failing column, :1139-1145).
#include <algorithm>
#include <climits>
#include <cstdio>
#include <type_traits>
#include <cuda_fp16.h>

#include "kernels.h"
#include "launch.h"

namespace tb {

namespace {

__device__ __forceinline__ double rsqrt_t(double x) { return rsqrt(x); }
__device__ __forceinline__ float rsqrt_t(float x) { return rsqrtf(x); }

__device__ __forceinline__ bool failed(const int* status) {
  return *(volatile const int*) status != INT_MAX;
}

// the status word, the panels' counters and the persistent launches' pending
// counts and queue heads
__global__ void k_init_status(int* status, int* done, int n, const int* __restrict__ pending0, int* work, int np) {
  grid_wait_then_trigger();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) *status = INT_MAX;
  if (i < n) done[i] = 0;
  if (i < np) work[i] = pending0[i];
  if (np > 0 && i < 2) work[np + i] = 0;
}

// ------------------------------------------------------------ small fronts

// One small front by one CTA (128 threads) in shared memory W (f x f): zero,
// assemble A's columns, extend-add the children's update matrices in child
// order, partial Cholesky of the first s columns, then write the panel and
// the update matrix.  Every thread returns together; on a nonpositive pivot
// the front's global column is recorded and it returns early.
template <typename T>
__device__ void small_front(const FrontDesc& F, const FrontDesc* __restrict__ fronts, T* W,
                            const int* __restrict__ children,
                            const int* __restrict__ maps, const int* __restrict__ rows,
                            const int* __restrict__ acol_ptr, const int* __restrict__ a_rows,
                            const int* __restrict__ a_idx, const T* __restrict__ vals, T* __restrict__ L,
                            T* __restrict__ U, int* status) {
  const int f = F.f, s = F.s, m = f - s;
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;

  for (int k = tid; k < f * f; k += nt) W[k] = 0.0;
  __syncthreads();
  // A's columns, one thread per column (duplicate rows add in order), the
  // entries four at a time with their loads issued together
  for (int c = tid; c < s; c += nt) {
    int e = __ldg(acol_ptr + F.acol_off + c);
    const int e1 = __ldg(acol_ptr + F.acol_off + c + 1);
    for (; e < e1; e += 4) {
      int r[4];
      T v[4];
#pragma unroll
      for (int q = 0; q < 4; q++) r[q] = e + q < e1 ? __ldg(a_rows + e + q) : -1;
#pragma unroll
      for (int q = 0; q < 4; q++) v[q] = e + q < e1 ? __ldg(vals + __ldg(a_idx + e + q)) : T(0);
#pragma unroll
      for (int q = 0; q < 4; q++)
        if (r[q] >= 0) W[r[q] + c * f] += v[q];
    }
  }
  __syncthreads();
  // the children's update matrices in child order: warp w takes the child's
  // columns w + nw u (eight per pass), lane l its rows l + 32 v; a pass
  // issues all its loads before its adds
  constexpr int SJ = 8, SV = (SMALL_F_MAX + 31) / 32;
  for (int ci = F.child_begin; ci < F.child_end; ci++) {
    const FrontDesc C = fronts[children[ci]];
    const int mc = C.f - C.s;
    const int* mp = maps + C.map_off;
    const T* Uc = U + C.u_off;
    int pi[SV];
#pragma unroll
    for (int v = 0; v < SV; v++) pi[v] = lane + 32 * v < mc ? __ldg(mp + lane + 32 * v) : -1;
    for (int j0 = warp; j0 < mc; j0 += nw * SJ) {
      int pj[SJ];
      T val[SJ][SV];
#pragma unroll
      for (int u = 0; u < SJ; u++) {
        const int j = j0 + nw * u;
        pj[u] = j < mc ? __ldg(mp + j) * f : -1;
#pragma unroll
        for (int v = 0; v < SV; v++) {
          const int i = lane + 32 * v;
          val[u][v] = (j < mc && i >= j && i < mc) ? __ldcg(Uc + i + (size_t) j * mc) : T(0);
        }
      }
#pragma unroll
      for (int u = 0; u < SJ; u++) {
        const int j = j0 + nw * u;
#pragma unroll
        for (int v = 0; v < SV; v++) {
          const int i = lane + 32 * v;
          if (pj[u] >= 0 && i >= j && i < mc) W[pi[v] + pj[u]] += val[u][v];
        }
      }
    }
    __syncthreads();
  }
  // column j stays unscaled in W: its multipliers W[i][j] rj are formed
  // where they are used (the same products as scaling it in place), and the
  // panel is scaled by rjs[] on its way out -- one barrier per column
  __shared__ T rjs[SMALL_F_MAX];
  constexpr int KU = 4;
  for (int j = 0; j < s; j++) {
    const T d = W[j + j * f];
    if (!(d > 0.0)) {
      if (tid == 0) atomicMin(status, rows[F.rows_off + j]);
      return;
    }
    const T rj = rsqrt_t(d);
    if (tid == 0) rjs[j] = rj;
    // warp w takes columns k0 + nw u (u < KU) of the trailing part, lane l
    // the rows from k0 + l; each pass loads before it stores
    const T* wj = W + j * f;
    for (int k0 = j + 1 + warp; k0 < f; k0 += nw * KU) {
      T lk[KU];
#pragma unroll
      for (int u = 0; u < KU; u++) {
        const int k = k0 + nw * u;
        lk[u] = k < f ? wj[k] * rj : T(0);
      }
      for (int i = k0 + lane; i < f; i += 32) {
        const T li = wj[i] * rj;
        T w[KU];
#pragma unroll
        for (int u = 0; u < KU; u++) {
          const int k = k0 + nw * u;
          w[u] = (k < f && i >= k) ? W[i + k * f] : T(0);
        }
#pragma unroll
        for (int u = 0; u < KU; u++) {
          const int k = k0 + nw * u;
          if (k < f && i >= k) W[i + k * f] = w[u] - li * lk[u];
        }
      }
    }
    __syncthreads();
  }
  T* Lp = L + F.l_off;
  for (int k = tid; k < f * s; k += nt) Lp[k] = W[k] * rjs[k / f];
  if (m > 0) {
    T* Up = U + F.u_off;
    for (int k = tid; k < m * m; k += nt) {
      const int i = k % m, c = k / m;
      Up[k] = W[(s + i) + (s + c) * f];
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(128)
k_small_front(const int* __restrict__ list, const FrontDesc* __restrict__ fronts,
              const int* __restrict__ children, const int* __restrict__ maps,
              const int* __restrict__ rows, const int* __restrict__ acol_ptr,
              const int* __restrict__ a_rows, const int* __restrict__ a_idx,
              const T* __restrict__ vals, T* __restrict__ L, T* __restrict__ U,
              int* status) {
  grid_wait();
  extern __shared__ __align__(16) unsigned char smraw[];
  if (failed(status)) return;
  small_front<T>(fronts[list[blockIdx.x]], fronts, reinterpret_cast<T*>(smraw), children, maps, rows, acol_ptr, a_rows,
                 a_idx, vals, L, U, status);
}

__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Waits (bounded) until *p is zero.  Every lane of the warp polls, and the
// loop ends by a vote: a loop that one lane alone runs leaves the warp split,
// and the shuffles after it then issue once per part of the warp (a pivot of
// the one-warp factor below took ~16,000 cycles after such a wait against
// ~900 without one; the launch over a 100 x 100 grid's fronts, FP64, 443 us
// with one lane polling, 68 us with the whole warp).
__device__ __forceinline__ void warp_wait_zero(const int* p, int* status, int ns) {
  int it = 0;
  while (!__all_sync(0xffffffffu, ld_acquire_gpu(p) == 0)) {
    if (++it > (1 << 22)) {
      atomicMin(status, NUMERIC_TIMEOUT);
      break;
    }
    __nanosleep(ns);
  }
}

// The same until *p is at least v, or the factorization has failed (then without
// a timeout of its own: the failing column stays in the status word).  Returns
// the value that lane 0 saw, on every lane (the lanes' loads may see different
// ones, and callers branch on it around votes).
__device__ __forceinline__ int warp_wait_at_least(const int* p, int v, int* status) {
  int it = 0, x;
  while (!__all_sync(0xffffffffu, (x = ld_acquire_gpu(p)) >= v)) {
    ++it;
    if ((it & 63) == 0 && __any_sync(0xffffffffu, failed(status))) break;
    if (it > (1 << 22)) {
      atomicMin(status, NUMERIC_TIMEOUT);
      break;
    }
    __nanosleep(20);
  }
  return __shfl_sync(0xffffffffu, x, 0);
}

// One front of order f <= SMALL_WARP_F by one warp: the front is assembled
// in the warp's shared rows Ws (row-major, one padded row per front row),
// then lane i holds row i in registers for the partial Cholesky of the first
// s columns (column j's multipliers passed by shuffles; the same operations
// as small_front), and writes the panel and the update matrix with zeros
// above the diagonal.  On a nonpositive pivot the front's global column is
// recorded and the warp returns early.
template <typename T>
__device__ void warp_front(const FrontDesc& F, const FrontDesc* __restrict__ fronts, T (*Ws)[SMALL_WARP_F + 1],
                           const int* __restrict__ children, const int* __restrict__ maps,
                           const int* __restrict__ rows, const int* __restrict__ acol_ptr,
                           const int* __restrict__ a_rows, const int* __restrict__ a_idx,
                           const T* __restrict__ vals, T* __restrict__ L, T* __restrict__ U, int* status) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int WF = SMALL_WARP_F;
  const int f = F.f, s = F.s, m = f - s;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int c = 0; c < WF; c++) Ws[lane][c] = T(0);
  __syncwarp();
  // A's column `lane` (one lane per column: duplicate rows add in order)
  if (lane < s) {
    int e = __ldg(acol_ptr + F.acol_off + lane);
    const int e1 = __ldg(acol_ptr + F.acol_off + lane + 1);
    for (; e + 4 <= e1; e += 4) {
      int r[4];
      T v[4];
#pragma unroll
      for (int q = 0; q < 4; q++) r[q] = __ldg(a_rows + e + q);
#pragma unroll
      for (int q = 0; q < 4; q++) v[q] = __ldg(vals + __ldg(a_idx + e + q));
#pragma unroll
      for (int q = 0; q < 4; q++) Ws[r[q]][lane] += v[q];
    }
    for (; e < e1; e++) Ws[__ldg(a_rows + e)][lane] += __ldg(vals + __ldg(a_idx + e));
  }
  // the children's update matrices in child order: lane i takes the child's
  // row i, all its loads before its adds (distinct rows: no conflicts)
  for (int ci = F.child_begin; ci < F.child_end; ci++) {
    const FrontDesc C = fronts[children[ci]];
    const int mc = C.f - C.s;
    const T* Uc = U + C.u_off;
    const int pi = lane < mc ? __ldg(maps + C.map_off + lane) : 0;
    T v[WF];
#pragma unroll
    for (int j = 0; j < WF; j++) v[j] = (j <= lane && lane < mc) ? __ldcg(Uc + lane + (size_t) j * mc) : T(0);
    __syncwarp();
#pragma unroll
    for (int j = 0; j < WF; j++) {
      if (j >= mc) break;
      const int pj = __shfl_sync(FULL, pi, j);
      if (j <= lane && lane < mc) Ws[pi][pj] += v[j];
    }
  }
  __syncwarp();
  T w[WF];
#pragma unroll
  for (int c = 0; c < WF; c++) w[c] = Ws[lane][c];
  __syncwarp();
  // pivot j in a rolled loop: the row is rotated left by one entry per
  // pivot, so column j is always w[0] and column j + k is w[k] (one body of
  // row code instead of one per pivot keeps the kernel cache-resident); the
  // finished column goes straight to the panel
  T* Lp = L + F.l_off;
#pragma unroll 1
  for (int j = 0; j < s; j++) {
    const T d = __shfl_sync(FULL, w[0], j);
    if (!(d > T(0))) {
      if (lane == 0) atomicMin(status, rows[F.rows_off + j]);
      return;
    }
    const T rj = rsqrt_t(d);
    const T lij = lane > j ? w[0] * rj : (lane == j ? d * rj : T(0));
    if (lane < f) Lp[lane + (size_t) j * f] = lij;
#pragma unroll
    for (int k = 1; k < WF; k++) {
      const T lkj = __shfl_sync(FULL, lij, (j + k) & (WF - 1));
      if (lane >= j + k && j + k < f) w[k] -= lij * lkj;
    }
#pragma unroll
    for (int k = 0; k < WF - 1; k++) w[k] = w[k + 1];
    w[WF - 1] = T(0);
  }
  // after s rotations w[k] is the row's column s + k
  if (lane < f && lane >= s) {
    T* Up = U + F.u_off;
#pragma unroll
    for (int k = 0; k < WF; k++)
      if (k < m) Up[(lane - s) + (size_t) k * m] = k <= lane - s ? w[k] : T(0);
  }
}

// The first part of the persistent set (fronts whose subtree has only
// fronts of order <= SMALL_WARP_F), in one launch of resident CTAs of four
// warps: each warp takes the next front from a device-side queue (tasks
// t0 .. t1-1 in level order), waits until the front's children are done
// (pending count), factors it (warp_front) and counts itself off at its
// parent -- also when the parent is in the second part, whose launch runs
// after this one.  Waits are bounded (NUMERIC_TIMEOUT); after a nonpositive
// pivot anywhere the remaining fronts are only counted off.
template <typename T>
__global__ void __launch_bounds__(128, sizeof(T) == 4 ? 6 : 4)
k_small_warp(const int* __restrict__ tasks, int t0, int t1, const int* __restrict__ parent_task, int* pending,
             int* next, const FrontDesc* __restrict__ fronts, const int* __restrict__ children,
             const int* __restrict__ maps, const int* __restrict__ rows, const int* __restrict__ acol_ptr,
             const int* __restrict__ a_rows, const int* __restrict__ a_idx, const T* __restrict__ vals,
             T* __restrict__ L, T* __restrict__ U, int* status) {
  grid_wait();
  __shared__ T Ws_all[4][SMALL_WARP_F][SMALL_WARP_F + 1];
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  for (;;) {
    int t = 0;
    if (lane == 0) t = t0 + atomicAdd(next, 1);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= t1) break;
    warp_wait_zero(pending + t, status, 32);
    if (!__any_sync(0xffffffffu, failed(status)))
      warp_front<T>(fronts[tasks[t]], fronts, Ws_all[wi], children, maps, rows, acol_ptr, a_rows, a_idx, vals, L,
                    U, status);
    __syncwarp();
    if (lane == 0) {
      __threadfence();
      const int pt = parent_task[t];
      if (pt >= 0) atomicSub(pending + pt, 1);
    }
  }
}

// The small fronts whose whole subtree is small (Plan::pers_fronts), in one
// launch of resident CTAs: each CTA takes the next front from a device-side
// queue (an atomic counter over the fronts in level order), waits until the
// front's children are done (its pending count, decremented by each child's
// CTA after its update matrix is written), factors it, and marks it done
// for its parent.  A front is only taken after all fronts before it in level
// order were taken by running CTAs, so every wait ends; the waits are bounded
// all the same (NUMERIC_TIMEOUT).  After a nonpositive pivot anywhere the
// remaining fronts are only marked done.
template <typename T>
__global__ void __launch_bounds__(128)
k_small_persistent(const int* __restrict__ tasks, int t0, int t1, const int* __restrict__ parent_task, int* pending,
                   int* next, const FrontDesc* __restrict__ fronts, const int* __restrict__ children,
                   const int* __restrict__ maps, const int* __restrict__ rows, const int* __restrict__ acol_ptr,
                   const int* __restrict__ a_rows, const int* __restrict__ a_idx, const T* __restrict__ vals,
                   T* __restrict__ L, T* __restrict__ U, int* status) {
  grid_wait();
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ int t_s, skip_s;
  T* W = reinterpret_cast<T*>(smraw);
  for (;;) {
    if (threadIdx.x == 0) t_s = t0 + atomicAdd(next, 1);
    __syncthreads();
    const int t = t_s;
    if (t >= t1) break;
    if (threadIdx.x < 32) {
      warp_wait_zero(pending + t, status, 64);
      if (threadIdx.x == 0) skip_s = failed(status);
    }
    __syncthreads();
    if (!skip_s)
      small_front<T>(fronts[tasks[t]], fronts, W, children, maps, rows, acol_ptr, a_rows, a_idx, vals, L, U, status);
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      const int pt = parent_task[t];
      if (pt >= 0) atomicSub(pending + pt, 1);
    }
  }
}

// --------------------------------------------------------------- front build

// threads of a build CTA: four warps, sixteen CTAs resident per SM
constexpr int BUILD_THREADS = 128;

// The child records of the build tiles, once per plan: CTA t (four warps)
// finds for each child of tile t's front the child's columns and rows that
// land in the tile, the four bounds searched at once (32-ary warp searches
// of the child's increasing map).
__global__ void __launch_bounds__(128)
k_tile_ranges(const Tile* __restrict__ tiles, const FrontDesc* __restrict__ fronts, const int* __restrict__ children,
              const int* __restrict__ maps, TileChild* __restrict__ rec) {
  grid_wait();
  const Tile tl = tiles[blockIdx.x];
  const FrontDesc F = fronts[tl.front];
  const int f = F.f, s = F.s, m = f - s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int R0, C0, nr, nc;
  if (tl.c0 >= 0) {
    R0 = tl.r0; C0 = tl.c0;
    nr = min(BUILD_TR, f - R0); nc = min(BUILD_TC, s - C0);
  } else {
    const int uc0 = -1 - tl.c0;
    R0 = s + tl.r0; C0 = s + uc0;
    nr = min(BUILD_TR, m - tl.r0); nc = min(BUILD_TC, m - uc0);
  }
  for (int ci = F.child_begin; ci < F.child_end; ci++) {
    const FrontDesc C = fronts[children[ci]];
    const int mc = C.f - C.s;
    const int key = warp == 0 ? C0 : warp == 1 ? C0 + nc : warp == 2 ? R0 : R0 + nr;
    const int r = warp_lower_bound(maps + C.map_off, mc, key);
    TileChild* out = rec + tl.ch_off + (ci - F.child_begin);
    if (lane == 0) {
      int* o = &out->ja;
      o[warp] = r;   // ja, jb, ia, ib in warp order
      if (warp == 0) {
        out->map_off = C.map_off;
        out->mc = mc;
        out->u_off = C.u_off;
      }
    }
  }
}


template <typename T>
__global__ void __launch_bounds__(BUILD_THREADS)
k_build(const Tile* __restrict__ tiles, const TileChild* __restrict__ tile_ch, const FrontDesc* __restrict__ fronts,
        const int* __restrict__ maps,
        const int* __restrict__ acol_ptr, const int* __restrict__ a_rows,
        const int* __restrict__ a_idx, const T* __restrict__ vals,
        T* __restrict__ L, T* __restrict__ U, const int* status) {
  __shared__ T W[BUILD_TR * BUILD_TC];
  const Tile tl = tiles[blockIdx.x];
  const FrontDesc F = fronts[tl.front];
  const int f = F.f, s = F.s, m = f - s;
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5;
  const bool panel = tl.c0 >= 0;
  int R0, C0, nr, nc;
  if (panel) {
    R0 = tl.r0; C0 = tl.c0;
    nr = min(BUILD_TR, f - R0); nc = min(BUILD_TC, s - C0);
  } else {
    const int uc0 = -1 - tl.c0;
    R0 = s + tl.r0; C0 = s + uc0;
    nr = min(BUILD_TR, m - tl.r0); nc = min(BUILD_TC, m - uc0);
  }
  for (int k = tid; k < BUILD_TR * BUILD_TC; k += nt) W[k] = 0.0;
  __syncthreads();
  if (panel) {
    // A's entries of the tile's columns: thread (column c, slot q) takes the
    // column's entries q, q + 8, ... -- the loads of all slots in flight at
    // once; the adds are atomic, as a column may list a row more than once
    // (duplicates are summed)
    const int c = tid % BUILD_TC, q = tid / BUILD_TC;
    constexpr int NQS = BUILD_THREADS / BUILD_TC;
    int e = 0, e1 = 0;
    if (c < nc) {
      e = __ldg(acol_ptr + F.acol_off + C0 + c) + q;
      e1 = __ldg(acol_ptr + F.acol_off + C0 + c + 1);
    }
    for (; e < e1; e += NQS) {
      const int r = __ldg(a_rows + e) - R0;
      if (r >= 0 && r < nr) atomicAdd(&W[r + c * BUILD_TR], __ldg(vals + __ldg(a_idx + e)));
    }
    __syncthreads();
  }
  // (above: nothing that a kernel of this factorization writes)
  grid_wait();
  if (failed(status)) return;
  // the children's shares, in child order, from the tile's records (found
  // once per plan); every load of a child's share is issued before the
  // first add (the children's update matrices were written by earlier
  // launches)
  const int nch = F.child_end - F.child_begin;
  for (int c = 0; c < nch; c++) {
    const TileChild R = tile_ch[tl.ch_off + c];
    const int ja = R.ja, jb = R.jb, ia = R.ia, ib = R.ib;
    if (ja >= jb || ia >= ib) continue;
    const int mc = R.mc;
    const int* mp = maps + R.map_off;
    const T* Uc = U + R.u_off;
    // warp w takes the child's columns ja + w + NW u, lane l its rows
    // ia + l + 32v
    constexpr int NW = BUILD_THREADS / 32, JU = (BUILD_TC + NW - 1) / NW, IU = BUILD_TR / 32;
    int pi[IU], pj[JU];
    T val[JU][IU];
#pragma unroll
    for (int v = 0; v < IU; v++) {
      const int i = ia + lane + 32 * v;
      pi[v] = (i < ib) ? __ldg(mp + i) - R0 : -1;
    }
#pragma unroll
    for (int u = 0; u < JU; u++) {
      const int j = ja + warp + NW * u;
      const bool jv = j < jb;
      pj[u] = jv ? (__ldg(mp + j) - C0) * BUILD_TR : -1;
#pragma unroll
      for (int v = 0; v < IU; v++) {
        const int i = ia + lane + 32 * v;
        val[u][v] = (jv && i < ib && i >= j) ? __ldcg(Uc + (size_t) j * mc + i) : T(0);
      }
    }
#pragma unroll
    for (int u = 0; u < JU; u++)
#pragma unroll
      for (int v = 0; v < IU; v++) {
        const int i = ia + lane + 32 * v, j = ja + warp + NW * u;
        if (pj[u] >= 0 && pi[v] >= 0 && i >= j) W[pi[v] + pj[u]] += val[u][v];
      }
    __syncthreads();
  }
  grid_trigger();
  if (panel) {
    T* dst = L + F.l_off;
    for (int k = tid; k < BUILD_TR * BUILD_TC; k += nt) {
      const int r = k % BUILD_TR, c = k / BUILD_TR;
      if (r < nr && c < nc) dst[(R0 + r) + (size_t) (C0 + c) * f] = W[k];
    }
  } else {
    T* dst = U + F.u_off;
    for (int k = tid; k < BUILD_TR * BUILD_TC; k += nt) {
      const int r = k % BUILD_TR, c = k / BUILD_TR;
      if (r < nr && c < nc) dst[(R0 - s + r) + (size_t) (C0 - s + c) * m] = W[k];
    }
  }
}

// -------------------------------------------- inverses of the diagonal blocks

constexpr int LLD = PANEL_NB + 4;   // padded column stride of k_dinv's blocks in shared memory
constexpr int LQ = 16;              // its pieces
constexpr int LYD = LQ + 1;         // column stride of a 16x16 inverse

template <typename T>
constexpr size_t dinv_smem() { return (2 * PANEL_NB * LLD + (PANEL_NB / LQ) * LQ * LYD) * sizeof(T); }

// Inverse of the lower-triangular 16x16 factor held one row per lane (a[k] =
// L[i][k], i = lane & 15, k <= i) into Y (column-major, ld LYD): lane t forms
// column t by forward substitution, reading L[r][k] by broadcast shuffles.
template <typename T>
__device__ __forceinline__ void warp_inv16_rows(const T (&a)[LQ], T* Y) {
  const int i = threadIdx.x & 15;
  T y[LQ];
#pragma unroll
  for (int r = 0; r < LQ; r++) {
    T acc = (r == i) ? T(1) : T(0);
#pragma unroll
    for (int k = 0; k < r; k++) acc -= __shfl_sync(0xffffffffu, a[k], r) * y[k];
    const T lrr = __shfl_sync(0xffffffffu, a[r], r);
    y[r] = (r >= i) ? acc * (T(1) / lrr) : T(0);
  }
  if ((threadIdx.x & 31) < LQ) {
#pragma unroll
    for (int r = 0; r < LQ; r++) Y[r + i * LYD] = y[r];
  }
}

// After the factorization, one CTA per 64x64 diagonal block L_kk of every big
// front: its inverse (lower, zero beyond the block's width), which the solve
// applies, into the block's slot of Dinv.  Warp q inverts the 16x16 diagonal
// piece q; then warp b forms block column b below the diagonal, X_cb = -X_cc
// sum_{b<=k<c} L_ck X_kb.
template <typename T>
__global__ void __launch_bounds__(128)
k_dinv(const int2_* __restrict__ blocks, const FrontDesc* __restrict__ fronts, const T* L,
       T* __restrict__ Dinv, const int* status) {
  grid_wait();
  extern __shared__ __align__(16) unsigned char smraw[];
  T* S = reinterpret_cast<T*>(smraw);   // L_kk, 64 x 64, ld LLD (identity beyond w)
  T* X = S + PANEL_NB * LLD;            // its inverse, ld LLD
  T* Tm = X + PANEL_NB * LLD;           // per warp: a 16x16 partial sum, ld LYD
  if (failed(status)) return;
  const int2_ bl = blocks[blockIdx.x];
  const FrontDesc F = fronts[bl.a];
  const int f = F.f, kb = bl.b * PANEL_NB;
  const int w = min(PANEL_NB, F.s - kb);
  const T* P = L + F.l_off;
  T* Di = Dinv + F.dinv_off + (size_t) bl.b * PANEL_NB * PANEL_NB;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
#pragma unroll 8
  for (int t = 0; t < PANEL_NB * PANEL_NB / 128; t++) {
    const int e = tid + 128 * t, i = e % PANEL_NB, j = e / PANEL_NB;
    const T v = (i < w && j < w && i >= j) ? P[(kb + i) + (size_t) (kb + j) * f] : (i == j ? T(1) : T(0));
    S[i + j * LLD] = v;
    X[i + j * LLD] = T(0);
  }
  __syncthreads();
  {
    const int q0 = warp * LQ, i = lane & 15;
    T a[LQ];
#pragma unroll
    for (int k = 0; k < LQ; k++) a[k] = (k <= i) ? S[(q0 + i) + (q0 + k) * LLD] : T(0);
    T* Yq = Tm + warp * LQ * LYD;
    warp_inv16_rows(a, Yq);
    __syncwarp();
    if (lane < LQ)
      for (int r = 0; r < LQ; r++) X[(q0 + r) + (q0 + lane) * LLD] = Yq[r + lane * LYD];
  }
  __syncthreads();
  if (warp < PANEL_NB / LQ - 1) {
    const int b0 = warp * LQ, t = lane & 15;
    T* Tw = Tm + warp * LQ * LYD;
    for (int c = warp + 1; c < PANEL_NB / LQ; c++) {
      const int c0 = c * LQ;
      // Tw[:, t] = sum_{k=b}^{c-1} L_ck X_kb[:, t]
      T acc[LQ];
#pragma unroll
      for (int r = 0; r < LQ; r++) acc[r] = T(0);
      for (int j = b0; j < c0; j++) {
        const T xj = X[j + (b0 + t) * LLD];
#pragma unroll
        for (int r = 0; r < LQ; r++) acc[r] += S[(c0 + r) + j * LLD] * xj;
      }
      __syncwarp();
      if (lane < LQ)
#pragma unroll
        for (int r = 0; r < LQ; r++) Tw[r + t * LYD] = acc[r];
      __syncwarp();
      // X_cb[:, t] = -X_cc Tw[:, t]
#pragma unroll
      for (int r = 0; r < LQ; r++) acc[r] = T(0);
      for (int j = 0; j < LQ; j++) {
        const T tj = Tw[j + t * LYD];
#pragma unroll
        for (int r = 0; r < LQ; r++) acc[r] += X[(c0 + r) + (c0 + j) * LLD] * tj;
      }
      if (lane < LQ)
#pragma unroll
        for (int r = 0; r < LQ; r++) X[(c0 + r) + (b0 + t) * LLD] = -acc[r];
      __syncwarp();
    }
  }
  __syncthreads();
  for (int e = tid; e < PANEL_NB * PANEL_NB; e += 128) {
    const int i = e % PANEL_NB, j = e / PANEL_NB;
    Di[e] = (i < w && j < w) ? X[i + j * LLD] : T(0);
  }
}

// ------------------------------------------------------------- DMMA GEMM

__device__ __forceinline__ void cp_async8(double* smem, const double* gmem, bool pred) {
  const unsigned saddr = (unsigned) __cvta_generic_to_shared(smem);
  const int sz = pred ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(saddr), "l"(gmem), "r"(sz));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void dmma16888(double (&c)[4], const double (&a)[4], const double (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

__device__ __forceinline__ void cp_async_t(double* smem, const double* gmem, bool pred) { cp_async8(smem, gmem, pred); }
__device__ __forceinline__ void cp_async_t(float* smem, const float* gmem, bool pred) {
  const unsigned saddr = (unsigned) __cvta_generic_to_shared(smem);
  const int sz = pred ? 4 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(saddr), "l"(gmem), "r"(sz));
}

// ---------------------------------------------------------------- panels

// A panel step: the columns [kb, kb + w) of the level's big fronts, w = min(128,
// s - kb), factored and applied to every row below them in ONE launch (the
// reference's POTRF :1131 and TRSM :1150 on a 128-column piece).  What bounds
// it is the chain of pivots, so one CTA per front (the first nb of the launch)
// holds the w x w diagonal block in shared memory and does nothing but that
// chain, in 16-column pieces: the first warp brings the next piece's diagonal
// rows up to date and factors it while the others update the rest.  Each
// finished piece goes to the panel behind a counter (release/acquire); the
// other CTAs hold PROWS rows below the block each, follow the counter, solve their
// rows against the piece and update their columns to the right.  They have
// higher indices than every diagonal CTA and wait for nothing else, so each
// wait ends; the waits are bounded all the same.
//
// The code is kept small: the kernel that this one replaced held rows in
// registers (64 columns a launch) and ran as straight-line code, 4 warps of it
// on an SM, which instruction fetch bounded (the 136 multiply-adds of a
// piece's substitution took 4600 cycles, 700 when they were still in the
// instruction cache).  Here a piece's Cholesky is a loop over pivots, products
// are small tile loops (FP64: DMMA fragments; FP32: multiply-adds in FP32).
// Panel steps and the products between them per factorization, before (64
// columns a launch) and now: 64^3 FP64 10.3 + 17.2 ms -> 7.1 + 10.8, 40x41x39
// FP64 2.96 + 2.82 -> 2.20 + 0.93, 80^3 FP32 13.3 + 11.8 -> 10.9 + 8.3,
// 139x142 FP32 0.59 + 0.13 -> 0.44 + 0.01.  A step takes 35 us while its CTAs
// have an SM each, of which the eight pieces' own pivots are about 16.
constexpr int PW = 128;              // columns of a panel step
constexpr int PB = 16;               // columns of a piece
constexpr int PLDB = PW + 4;         // column stride of a piece that a row CTA reads
// The diagonal block: piece p holds its 16 columns from row 16 p on, column
// stride PLDD - 16 p (a multiple of four elements, and no two rows of a FP64
// fragment in the same bank); FP32 leaves room for the rows of a 32-row unit
// that are past the block's last
template <typename T>
constexpr int PLDD = PW + (sizeof(T) == 4 ? 20 : 4);
template <typename T>
__host__ __device__ constexpr int diag_base(int p) { return PB * (PLDD<T> * p - 8 * p * (p - 1)); }
// column stride of the entries of a row CTA of ROWS rows
template <int ROWS>
constexpr int PLDR = ROWS + 4;
// shared memory of a launch whose widest step has wmax columns
template <typename T, int ROWS>
constexpr size_t panel_smem(int wmax) {
  const int np = (wmax + PB - 1) / PB;
  const size_t d = (size_t) diag_base<T>(np) + 2 * (PB * (PB + 1) + PB);
  const size_t r = (size_t) np * PB * PLDR<ROWS> + 2 * (PB * PLDB + PB);
  return (d > r ? d : r) * sizeof(T);
}

// Pivots J0 .. J1-1 of a piece with at most NC columns right of them.  Lane i
// holds row i, moved one entry to the left per pivot (column J is always
// a[0]).  The scaled column goes to the other lanes through shared memory
// (written relative to the pivot, read back as vectors): with a shuffle per
// column a piece took 4700 cycles in FP32 and 8000 in FP64, this way 2700 and
// 3300.  The next pivot comes from lane J + 1's own entries by one shuffle, and
// its reciprocal square root is on its way before the other columns are
// updated.
template <typename T, int NC>
__device__ __forceinline__ void chol_pivots(T (&a)[PB], int J0, int J1, int i, T& d, T& r, T& rown, int& bad, T* buf,
                                            T* Lp, T* col, int ldc) {
  constexpr int V = 16 / (int) sizeof(T);
  struct alignas(16) Vec { T v[V]; };
#pragma unroll 1
  for (int J = J0; J < J1; J++) {
    if (!(d > T(0)) && bad < 0) bad = J;
    const T l = (i == J) ? d * r : a[0] * r;
    if (i == J) rown = r;
    T* b = buf + (J & 1) * 32;
    b[(i - J - 1) & 31] = l;
    if (i >= J && i < PB) {
      Lp[i * (PB + 1) + J] = l;
      col[J * ldc + i] = l;
    }
    d = __shfl_sync(0xffffffffu, a[1] - l * l, J + 1);
    r = rsqrt_t(d);
    __syncwarp();
    Vec x[(NC + 1) / V];
#pragma unroll
    for (int k = 0; k < (NC + 1) / V; k++) x[k] = reinterpret_cast<const Vec*>(b)[k];
#pragma unroll
    for (int k = 1; k <= NC; k++) a[k - 1] = a[k] - l * x[(k - 1) / V].v[(k - 1) % V];
  }
}
// Cholesky factor of a 16x16 piece by one warp, lane i < 16 with row i (col:
// its columns, stride ldc; what lies above the diagonal and in the next 16 rows
// is read but reaches no result), into Lp
// (row stride 17), the reciprocal diagonal into rinv and back into col; bad:
// the first nonpositive pivot, or -1.  buf: 64 entries of the warp's own.
template <typename T>
__device__ __forceinline__ void chol_piece(T* col, int ldc, T* Lp, T* rinv, int* bad_out, T* buf) {
  const int i = threadIdx.x & 31;
  T a[PB];
#pragma unroll
  for (int k = 0; k < PB; k++) a[k] = col[k * ldc + i];
  int bad = -1;
  T d = __shfl_sync(0xffffffffu, a[0], 0), r = rsqrt_t(d), rown = T(1);
  chol_pivots<T, PB - 1>(a, 0, PB / 2, i, d, r, rown, bad, buf, Lp, col, ldc);
  chol_pivots<T, PB / 2 - 1>(a, PB / 2, PB, i, d, r, rown, bad, buf, Lp, col, ldc);
  if (i < PB) rinv[i] = rown;
  if (i == 0) *bad_out = bad;
}

// x L_p^T = m for one row of 16 entries (stride ld); Lp[i sr + k sc] the piece
template <typename T>
__device__ __forceinline__ void solve_row(T* m, int ld, const T* Lp, int sr, int sc, const T* rinv) {
  T x[PB];
#pragma unroll
  for (int c = 0; c < PB; c++) x[c] = m[c * ld];
#pragma unroll
  for (int c = 0; c < PB; c++) {
    x[c] *= rinv[c];
#pragma unroll
    for (int c2 = c + 1; c2 < PB; c2++) x[c2] -= x[c] * Lp[c2 * sr + c * sc];
  }
  // (stores between the columns would hold back the loads of the next one)
#pragma unroll
  for (int c = 0; c < PB; c++) m[c * ld] = x[c];
}

// C[0..RU) x [0..16) -= A B^T by one warp, K = 16: C and A column-major (row 0 of
// the unit first), B[c + k ldb] the row c of the other operand.  run: the units
// of the trailing updates; diag: a 16 x 16 piece.  FP64: DMMA fragments; FP32:
// multiply-adds, four by four (a diagonal piece four by two) entries a lane.
template <typename T>
struct PanelUnit;
template <>
struct PanelUnit<double> {
  static constexpr int RU = 16;
  __device__ __forceinline__ static void run(double* C, int ldc, const double* A, int lda, const double* B, int ldb) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    double acc[2][4], *c0 = C + g + (2 * t) * ldc;
#pragma unroll
    for (int ni = 0; ni < 2; ni++) {
      const double* c = c0 + 8 * ni * ldc;
      acc[ni][0] = -c[0]; acc[ni][1] = -c[ldc]; acc[ni][2] = -c[8]; acc[ni][3] = -c[ldc + 8];
    }
#pragma unroll
    for (int kk = 0; kk < PB; kk += 8) {
      const double* a = A + g + (kk + t) * lda;
      const double* b = B + g + (kk + t) * ldb;
      const double av[4] = {a[0], a[8], a[4 * lda], a[4 * lda + 8]};
#pragma unroll
      for (int ni = 0; ni < 2; ni++) {
        const double bv[2] = {b[8 * ni], b[4 * ldb + 8 * ni]};
        dmma16888(acc[ni], av, bv);
      }
    }
#pragma unroll
    for (int ni = 0; ni < 2; ni++) {
      double* c = c0 + 8 * ni * ldc;
      c[0] = -acc[ni][0]; c[ldc] = -acc[ni][1]; c[8] = -acc[ni][2]; c[ldc + 8] = -acc[ni][3];
    }
  }
  __device__ __forceinline__ static void diag(double* C, int ldc, const double* A, int lda) {
    run(C, ldc, A, lda, A, lda);
  }
};
template <>
struct PanelUnit<float> {
  static constexpr int RU = 32;
  // R x CC entries a lane, K8 columns of both operands loaded at a time
  template <int CC>
  __device__ __forceinline__ static void unit(float* C, int ldc, const float* A, int lda, const float* B, int ldb, int r,
                                              int c) {
    float acc[CC][4] = {};
#pragma unroll 1
    for (int k0 = 0; k0 < PB; k0 += 8) {
      float4 a[8];
      float b[8][CC];
#pragma unroll
      for (int k = 0; k < 8; k++) a[k] = *reinterpret_cast<const float4*>(A + r + (k0 + k) * lda);
#pragma unroll
      for (int k = 0; k < 8; k++) {
        struct alignas(4 * CC) Vec { float v[CC]; };
        const Vec x = *reinterpret_cast<const Vec*>(B + c + (k0 + k) * ldb);
#pragma unroll
        for (int j = 0; j < CC; j++) b[k][j] = x.v[j];
      }
#pragma unroll
      for (int k = 0; k < 8; k++)
#pragma unroll
        for (int j = 0; j < CC; j++) {
          acc[j][0] += a[k].x * b[k][j];
          acc[j][1] += a[k].y * b[k][j];
          acc[j][2] += a[k].z * b[k][j];
          acc[j][3] += a[k].w * b[k][j];
        }
    }
#pragma unroll
    for (int j = 0; j < CC; j++) {
      float4* p = reinterpret_cast<float4*>(C + r + (c + j) * ldc);
      float4 v = *p;
      v.x -= acc[j][0]; v.y -= acc[j][1]; v.z -= acc[j][2]; v.w -= acc[j][3];
      *p = v;
    }
  }
  __device__ __forceinline__ static void run(float* C, int ldc, const float* A, int lda, const float* B, int ldb) {
    const int lane = threadIdx.x & 31;
    unit<4>(C, ldc, A, lda, B, ldb, 4 * (lane & 7), 4 * (lane >> 3));
  }
  __device__ __forceinline__ static void diag(float* C, int ldc, const float* A, int lda) {
    const int lane = threadIdx.x & 31;
    unit<2>(C, ldc, A, lda, A, lda, 4 * (lane & 3), 2 * (lane >> 2));
  }
};

// The split copy of one slab row for the tensor-core products (FP32): chunk c
// of CW columns of row r, hi and lo parts; x: the row's entries (stride ld),
// zero from column w on.
template <int FMT>
__device__ __forceinline__ void split_chunk(const float* x, int ld, int c, int w, unsigned char* dst, int64_t part) {
  if (FMT == 0) {
    unsigned h[4], l[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int k = c * 4 + q;
      const float v = k < w ? x[k * ld] : 0.0f;
      h[q] = __float_as_uint(v) & 0xffffe000u;
      l[q] = __float_as_uint(v - __uint_as_float(h[q]));
    }
    *reinterpret_cast<uint4*>(dst) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4*>(dst + part) = make_uint4(l[0], l[1], l[2], l[3]);
  } else {
    unsigned h[4], l[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      unsigned hh = 0, ll = 0;
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int k = c * 8 + 2 * q + e;
        const float v = k < w ? x[k * ld] : 0.0f;
        const __half hv = __float2half_rn(v);
        hh |= (unsigned) __half_as_ushort(hv) << (16 * e);
        ll |= (unsigned) __half_as_ushort(__float2half_rn((v - __half2float(hv)) * 2048.0f)) << (16 * e);
      }
      h[q] = hh;
      l[q] = ll;
    }
    *reinterpret_cast<uint4*>(dst) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4*>(dst + part) = make_uint4(l[0], l[1], l[2], l[3]);
  }
}

template <typename T, int FMT, int NT, int PROWS>
__global__ void __launch_bounds__(NT, 512 / NT)
k_panel(const int* __restrict__ cum, int nb, const int* __restrict__ list, const FrontDesc* __restrict__ fronts,
        const int* __restrict__ rows, T* __restrict__ L, float* __restrict__ sp, int kb, int* __restrict__ done,
        double* __restrict__ rdiag_all, int* status) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ __align__(16) T buf_s[64];
  __shared__ int bad_s[2];
  T* S = reinterpret_cast<T*>(smraw);
  const bool is_diag = (int) blockIdx.x < nb;
  int idx = 0;
  const FrontDesc F = fronts[list[is_diag ? (int) blockIdx.x : front_of(cum, nb, (int) blockIdx.x - nb, idx)]];
  const int f = F.f, s = F.s;
  if (kb >= s) return;
  grid_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int* cnt = done + F.blk_off;          // pieces of the front finished so far
  // the row CTAs leave on the status; a diagonal CTA that does not come to its
  // pieces releases those of them that are past this check (another front of the
  // launch may fail between their look at the status and its own)
  auto release = [&]() {
    if (tid == 0) {
      __threadfence();
      atomicExch(cnt, INT_MAX);
    }
  };
  if (__syncthreads_or(failed(status))) {   // all threads together
    if (is_diag) release();
    return;
  }
  const int w = min(PW, s - kb), np = (w + PB - 1) / PB;
  T* P = L + F.l_off;
  constexpr int NW = NT / 32, RU = PanelUnit<T>::RU, PLDR = tb::PLDR<PROWS>;
  T* rdiag = reinterpret_cast<T*>(rdiag_all) + (size_t) F.blk_off * PANEL_NB;   // 1 / L_jj
  const int first = kb / PB;            // of them before this step

  if (is_diag) {
    // -------------------------------------------------------- diagonal block
    T* Lp0 = S + diag_base<T>(np);     // two factored pieces, by parity
    T* rinv0 = Lp0 + 2 * PB * (PB + 1);
    auto at = [&](int p) { return S + diag_base<T>(p); };   // row 16 p of piece p's first column
    auto ldp = [&](int p) { return PLDD<T> - PB * p; };
    // lower part of the block, rows and columns past w as the identity
    const int w16 = np * PB;
    const int crew = (warp >> 2) * 3 + (warp & 3) - 1;   // of the warps that solve and update
    for (int j = warp; j < w16; j += NW) {
      const int p = j / PB;
      T* c = at(p) + (j - PB * p) * ldp(p) - PB * p;
      for (int i = PB * p + lane; i < w16; i += 32) {
        if (i < w && j < w) cp_async_t(c + i, P + (kb + i) + (size_t) (kb + j) * f, true);
        else c[i] = i == j ? T(1) : T(0);
      }
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    if (warp == 0) chol_piece<T>(at(0), ldp(0), Lp0, rinv0, &bad_s[0], buf_s);
    __syncthreads();
    for (int p = 0; p < np; p++) {
      const T* Lp = Lp0 + (p & 1) * PB * (PB + 1);
      const T* rinv = rinv0 + (p & 1) * PB;
      const int t0 = (p + 1) * PB;
      if (bad_s[p & 1] >= 0) {
        if (tid == 0) atomicMin(status, rows[F.rows_off + kb + p * PB + bad_s[p & 1]]);
        release();
        return;
      }
      T* cp = at(p) - PB * p;   // piece p by block row
      if ((warp & 3) != 0) {
        const int r = t0 + crew * 32 + lane;
        if (r < w16) solve_row<T>(cp + r, ldp(p), Lp, PB + 1, 1, rinv);
      }
      __syncthreads();
      // the first warp: the next piece, and nothing else.  The other warps of
      // its scheduler do nothing (their instructions would take the chain's
      // issue slots: with the write-out there a step was 5 % slower)
      auto unit = [&](int r0, int q0) {   // rows r0.., the columns of the piece at q0
        const int q = q0 / PB;
        PanelUnit<T>::run(at(q) - q0 + r0, ldp(q), cp + r0, ldp(p), cp + q0, ldp(p));
      };
      if (warp == 0) {
        if (t0 < w16) {
          PanelUnit<T>::diag(at(p + 1), ldp(p + 1), cp + t0, ldp(p));
          __syncwarp();
          chol_piece<T>(at(p + 1), ldp(p + 1), Lp0 + ((p + 1) & 1) * PB * (PB + 1), rinv0 + ((p + 1) & 1) * PB,
                        &bad_s[(p + 1) & 1], buf_s);
        }
      } else {
        if ((warp & 3) != 0) {
          // the last three of them write this piece out first
          constexpr int PT = 96, CREW = NW / 4 * 3;
          const int t = (crew - (CREW - 3)) * 32 + lane;
          if (t >= 0) {
            for (int e = t; e < PB * PW / 4; e += PT) {
              // four rows apart: every load before the first store
              T v[4];
              const int j = e / (PW / 4), i = e % (PW / 4);
#pragma unroll
              for (int q = 0; q < 4; q++) v[q] = p * PB + j <= i + 32 * q ? cp[i + 32 * q + j * ldp(p)] : T(0);
#pragma unroll
              for (int q = 0; q < 4; q++) {
                const int r = i + 32 * q, c = p * PB + j;
                if (r >= c && r < w && c < w) P[(kb + r) + (size_t) (kb + c) * f] = v[q];
              }
            }
            if (t < PB && p * PB + t < w) rdiag[(first + p) * PB + t] = rinv[t];
            asm volatile("bar.sync 1, %0;" ::"n"(PT) : "memory");
            if (t == 0) {
              __threadfence();
              asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(cnt), "r"(first + p + 1) : "memory");
            }
          }
          // the other units of the trailing lower part
          int turn = crew;
          for (int c = t0; c < w16; c += PB)
            for (int r0 = c == t0 ? t0 + PB : c; r0 < w16; r0 += RU) {
              if (turn == 0) {
                unit(r0, c);
                turn = CREW;
              }
              turn--;
            }
        }
      }
      __syncthreads();
    }
    return;
  }
  // ------------------------------------------------------------ rows below
  const int r0 = kb + w + idx * PROWS;
  const int nr = min(PROWS, f - r0);
  if (nr <= 0) return;
  for (int j = warp; j < np * PB; j += NW)
    for (int i = lane; i < PROWS; i += 32) {
      const bool in = i < nr && j < w;   // zero elsewhere
      cp_async_t(S + i + j * PLDR, P + r0 + (in ? i : 0) + (size_t) (kb + (in ? j : 0)) * f, in);
    }
  cp_async_commit();
  // pieces of the diagonal block, [column][row] and the reciprocal diagonal, in
  // two buffers: the next piece's loads (from L2: the block was written during
  // this launch) are on their way, when it is finished, during this one's work
  constexpr int NPRE = PB * PW / NT;
  T pre[NPRE], pri = T(0);
  auto fetch = [&](int p) {
    const int j0 = p * PB, i = tid % PW;
#pragma unroll
    for (int e = 0; e < NPRE; e++) {
      const int j = tid / PW + e * (NT / PW);
      pre[e] = (i < w && j0 + j < w && i >= j0 + j) ? __ldcg(P + (kb + i) + (size_t) (kb + j0 + j) * f) : T(0);
    }
    if (tid < PB) pri = j0 + tid < w ? __ldcg(rdiag + first * PB + j0 + tid) : T(1);
  };
  int have = 0;             // pieces known to be finished (the first warp: lane 0's load on every
                            // lane, since the waits that it guards vote over the whole warp)
  bool fetched = false;     // the same on every thread: bad_s carries it
  for (int p = 0; p < np; p++) {
    T* Bp = S + np * PB * PLDR + (p & 1) * (PB * PLDB + PB);
    T* rinv = Bp + PB * PLDB;
    if (!fetched) {
      if (warp == 0 && have <= p) have = warp_wait_at_least(cnt, first + p + 1, status) - first;
      __syncthreads();
      fetch(p);
    }
#pragma unroll
    for (int e = 0; e < NPRE; e++) Bp[tid % PW + (tid / PW + e * (NT / PW)) * PLDB] = pre[e];
    if (tid < PB) rinv[tid] = pri;
    if (warp == 0 && p + 1 < np) {
      if (have <= p + 1) have = __shfl_sync(0xffffffffu, ld_acquire_gpu(cnt), 0) - first;
      if (lane == 0) bad_s[p & 1] = have > p + 1;
    }
    cp_async_wait<0>();
    __syncthreads();
    fetched = p + 1 < np && bad_s[p & 1];
    if (fetched) fetch(p + 1);
    const int j0 = p * PB;
    T* Sp = S + j0 * PLDR;
    if (tid < PROWS) solve_row<T>(Sp + tid, PLDR, Bp + j0, 1, PLDB, rinv);
    __syncthreads();
    // one unit after the other, row groups first
    constexpr int NR = PROWS / RU;
    for (int u = warp; u < (np - 1 - p) * NR; u += NW) {
      const int c = j0 + PB + u / NR * PB, r = u % NR * RU;
      PanelUnit<T>::run(S + r + c * PLDR, PLDR, Sp + r, PLDR, Bp + c, PLDB);
    }
  }
  if (__syncthreads_or(failed(status))) return;
  grid_trigger();
  for (int j = warp; j < w; j += NW)
    for (int i = lane; i < nr; i += 32) P[r0 + i + (size_t) (kb + j) * f] = S[i + j * PLDR];
  if constexpr (sizeof(T) == 4) {
    if (sp != nullptr && F.sp_off >= 0) {
      // the rows' final values, split, into the split arena for the tensor-
      // core products; the front's last step also writes the zero columns
      // that pad K to the products' stage width
      const int64_t rg = sp_rgroups(f), part = sp_part_bytes(F, FMT);
      unsigned char* base = reinterpret_cast<unsigned char*>(sp + F.sp_off);
      constexpr int CW = FMT ? 8 : 4;
      const int kc0 = kb / CW, kc_end = (kb + w == s) ? (int) sp_kchunks(s, FMT) : (kb + w) / CW;
      const int i = tid % PROWS;
      if (i < nr)
        for (int c = tid / PROWS; c < kc_end - kc0; c += NT / PROWS)
          split_chunk<FMT>(S + i, PLDR, c, w,
                           base + ((int64_t) (kc0 + c) * rg + ((r0 + i) >> 3)) * 128 + ((r0 + i) & 7) * 16, part);
    }
  }
}

// FP64 fronts: one DMMA per fragment pair
// FP32 fronts: three TF32 products per fragment pair (hi*hi + hi*lo + lo*hi,
// the operands split as x = tf32(x) + tf32(x - tf32(x))), which keeps close
// to FP32 accuracy on the TF32 tensor path (same m16n8k8 fragment layout as
// the FP64 DMMA)
__device__ __forceinline__ void split_tf32(float x, unsigned& hi, unsigned& lo) {
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(x));
  const float r = x - __uint_as_float(hi);
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(r));
}

__device__ __forceinline__ void mma_tf32(float (&c)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// MI x NI fragment products of one k8 step.  FP32: every A and B fragment is
// split into TF32 hi/lo parts once, then three products per pair.
template <int MI, int NI>
__device__ __forceinline__ void mma_block(double (&acc)[MI][NI][4], const double (&a)[MI][4], const double (&b)[NI][2]) {
#pragma unroll
  for (int mi = 0; mi < MI; mi++)
#pragma unroll
    for (int ni = 0; ni < NI; ni++) dmma16888(acc[mi][ni], a[mi], b[ni]);
}

template <int MI, int NI>
__device__ __forceinline__ void mma_block(float (&acc)[MI][NI][4], const float (&a)[MI][4], const float (&b)[NI][2]) {
  unsigned ah[MI][4], al[MI][4], bh[NI][2], bl[NI][2];
#pragma unroll
  for (int mi = 0; mi < MI; mi++)
#pragma unroll
    for (int i = 0; i < 4; i++) split_tf32(a[mi][i], ah[mi][i], al[mi][i]);
#pragma unroll
  for (int ni = 0; ni < NI; ni++)
#pragma unroll
    for (int i = 0; i < 2; i++) split_tf32(b[ni][i], bh[ni][i], bl[ni][i]);
#pragma unroll
  for (int mi = 0; mi < MI; mi++)
#pragma unroll
    for (int ni = 0; ni < NI; ni++) {
      mma_tf32(acc[mi][ni], al[mi], bh[ni]);
      mma_tf32(acc[mi][ni], ah[mi], bl[ni]);
      mma_tf32(acc[mi][ni], ah[mi], bh[ni]);
    }
}

// number of lower-trapezoid tiles of a region with `rows` rows and `cols`
// columns whose column tile c covers rows [c*BN, rows)
__host__ __device__ inline int trap_tiles(int rows, int cols, int bm, int bn) {
  int t = 0;
  for (int c0 = 0; c0 < cols; c0 += bn) t += (rows - c0 + bm - 1) / bm;
  return t;
}

template <int BM, int BN>
struct GemmCfg {
  static constexpr int WM = 2;                     // warps along M
  static constexpr int WN = BN > 64 ? BN / 32 : 2; // warps along N
  static constexpr int THREADS = 32 * WM * WN;
  static constexpr int MI = BM / WM / 16;          // m16 tiles per warp
  static constexpr int NI = BN / WN / 8;           // n8 tiles per warp
  // no more shared memory than it takes: what is left caches the operand columns
  // that the SM's other tiles read too (64^3 update matrices with 2 / 3 / 4 stages
  // of 64x64 tiles: 21.4 / 22.1 / 23.0 ms)
  static constexpr int STAGES = BM == 64 ? 2 : 3;
  // k-row stride (BM >= BN): a FP64 fragment's 4 x 8 entries fill the banks
  // exactly (with BM + 8 every fragment load took two passes)
  static constexpr int LD = BM + 4;
  template <typename T>
  static constexpr size_t smem() { return (size_t) STAGES * 2 * GEMM_BK * LD * sizeof(T); }
};

// C -= A B^T on DMMA m16n8k8 tiles of BM x BN (32x32 and 64x64: 4 warps, 128x128:
// 8 warps), STAGES-deep cp.async pipeline, accumulators preloaded with -C.
// mode 0: panel update of columns [c_lo, min(c_hi, s)) and all rows below
//         c_lo by the panel columns [k_lo, k_hi) (one node of the recursive
//         panel factorization);
// mode 1: U -= L21 L21^T (K = [0, s))
template <typename T, int BM, int BN>
__global__ void __launch_bounds__(GemmCfg<BM, BN>::THREADS, sizeof(T) == 4 || BM == 128 ? 1 : BM == 64 ? 4 : 6)
k_gemm(const int* __restrict__ cum, int nb, const int* __restrict__ list, const FrontDesc* __restrict__ fronts, T* __restrict__ L,
       T* __restrict__ U, int c_lo, int c_hi, int k_lo, int k_hi, int mode, const int* status) {
  using Cfg = GemmCfg<BM, BN>;
  constexpr int MI = Cfg::MI, NI = Cfg::NI, LD = Cfg::LD, NT = Cfg::THREADS, STAGES = Cfg::STAGES;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* gsm = reinterpret_cast<T*>(smraw);   // STAGES x {A, B} x GEMM_BK x LD
  int idx;
  const FrontDesc F = fronts[list[front_of(cum, nb, blockIdx.x, idx)]];
  const int f = F.f, s = F.s, m = f - s;
  int rows, cols, roff, kbeg, kend, ldc;
  const T* P = L + F.l_off;
  T* Cbase;
  if (mode == 0) {
    const int cb = c_lo, ce = min(c_hi, s);
    if (cb >= ce) return;
    rows = f - cb; cols = ce - cb; roff = cb;
    kbeg = k_lo; kend = k_hi;
    Cbase = L + F.l_off + cb + (size_t) cb * f;
    ldc = f;
  } else {
    if (m <= 0 || s <= 0) return;
    rows = m; cols = m; roff = s;
    kbeg = 0; kend = s;
    Cbase = U + F.u_off;
    ldc = m;
  }
  // decode the lower-trapezoid tile
  int c0 = 0;
  for (;;) {
    if (c0 >= cols) return;
    const int nt_c = (rows - c0 + BM - 1) / BM;
    if (idx < nt_c) break;
    idx -= nt_c;
    c0 += BN;
  }
  const int r0 = c0 + idx * BM;
  const int nr = min(BM, rows - r0), nc = min(BN, cols - c0);
  const T* Ag = P + (roff + r0);
  const T* Bg = P + (roff + c0);
  T* C = Cbase + r0 + (size_t) c0 * ldc;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp % Cfg::WM, wn = warp / Cfg::WM, g = lane >> 2, t = lane & 3;
  const int wrow = wm * (BM / Cfg::WM), wcol = wn * (BN / Cfg::WN);
  grid_wait();
  if (failed(status)) return;
  // accumulators start at -C, so acc = A B^T - C and the result is -acc
  T acc[MI][NI][4];
#pragma unroll
  for (int mi = 0; mi < MI; mi++)
#pragma unroll
    for (int ni = 0; ni < NI; ni++)
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int r = wrow + mi * 16 + g + ((q & 2) ? 8 : 0);
        const int c = wcol + ni * 8 + 2 * t + (q & 1);
        acc[mi][ni][q] = (r < nr && c < nc && r0 + r >= c0 + c) ? -C[r + (size_t) c * ldc] : 0.0;
      }

  auto load = [&](int st, int k0) {
    T* As = gsm + (size_t) (st * 2) * GEMM_BK * LD;
    T* Bs = As + GEMM_BK * LD;
#pragma unroll
    for (int q = 0; q < (BM * GEMM_BK) / NT; q++) {
      const int e = tid + q * NT;
      const int r = e % BM, k = e / BM;
      const bool kv = (k0 + k) < kend;
      const bool pa = kv && r < nr;
      const size_t col = (size_t) (kv ? k0 + k : kbeg) * f;
      cp_async_t(As + k * LD + r, Ag + (pa ? r : 0) + col, pa);
    }
#pragma unroll
    for (int q = 0; q < (BN * GEMM_BK) / NT; q++) {
      const int e = tid + q * NT;
      const int r = e % BN, k = e / BN;
      const bool kv = (k0 + k) < kend;
      const bool pb = kv && r < nc;
      const size_t col = (size_t) (kv ? k0 + k : kbeg) * f;
      cp_async_t(Bs + k * LD + r, Bg + (pb ? r : 0) + col, pb);
    }
  };

  const int nk = (kend - kbeg + GEMM_BK - 1) / GEMM_BK;
#pragma unroll
  for (int st = 0; st < STAGES - 1; st++) {
    if (st < nk) load(st, kbeg + st * GEMM_BK);
    cp_async_commit();
  }
  for (int kt = 0; kt < nk; kt++) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    const int kn = kt + STAGES - 1;
    if (kn < nk) load(kn % STAGES, kbeg + kn * GEMM_BK);
    cp_async_commit();
    const T* As = gsm + (size_t) ((kt % STAGES) * 2) * GEMM_BK * LD;
    const T* Bs = As + GEMM_BK * LD;
#pragma unroll
    for (int kk = 0; kk < GEMM_BK; kk += 8) {
      T a[MI][4], b[NI][2];
#pragma unroll
      for (int mi = 0; mi < MI; mi++) {
        const int r = wrow + mi * 16 + g;
        a[mi][0] = As[(kk + t) * LD + r];
        a[mi][1] = As[(kk + t) * LD + r + 8];
        a[mi][2] = As[(kk + t + 4) * LD + r];
        a[mi][3] = As[(kk + t + 4) * LD + r + 8];
      }
#pragma unroll
      for (int ni = 0; ni < NI; ni++) {
        const int c = wcol + ni * 8 + g;
        b[ni][0] = Bs[(kk + t) * LD + c];
        b[ni][1] = Bs[(kk + t + 4) * LD + c];
      }
      mma_block<MI, NI>(acc, a, b);
    }
  }
  cp_async_wait<0>();
  grid_trigger();
#pragma unroll
  for (int mi = 0; mi < MI; mi++)
#pragma unroll
    for (int ni = 0; ni < NI; ni++)
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int r = wrow + mi * 16 + g + ((q & 2) ? 8 : 0);
        const int c = wcol + ni * 8 + 2 * t + (q & 1);
        if (r < nr && c < nc && r0 + r >= c0 + c) C[r + (size_t) c * ldc] = -acc[mi][ni][q];
      }
}

}  // namespace

// algorithmic work of a whole front (the reference's flop count,
// src/taucs_sn_llt.c:3957-3965) and of its assembly / extend-add traffic
static double front_flops(const FrontDesc& F) {
  double fl = 0.0;
  for (int k = 0, c = F.f; k < F.s; k++, c--) fl += 1.0 + (double) c * (double) c;
  return fl;
}

// algorithmic bytes of building one front, values of esz bytes: children's U
// read once (plus their maps), panel and U written once, A entries (value +
// row index)
static double build_bytes(const Plan& P, const FrontDesc& F, double esz) {
  double by = 0.0;
  for (int ci = F.child_begin; ci < F.child_end; ci++) {
    const FrontDesc& C = P.fronts[P.children[ci]];
    const double mc = C.f - C.s;
    by += esz * mc * (mc + 1.0) / 2.0 + 4.0 * mc;
  }
  const double m = F.f - F.s;
  by += esz * ((double) F.f * F.s - (double) F.s * (F.s - 1) / 2.0) + esz * m * (m + 1.0) / 2.0;
  by += (esz + 4.0) * (P.acol_ptr[F.acol_off + F.s] - P.acol_ptr[F.acol_off]);
  return by;
}

// small fronts: read children's U and A once, write panel and U once
static double front_bytes(const Plan& P, const FrontDesc& F, double esz) {
  return build_bytes(P, F, esz);
}

// GEMM variant of level h for the panel updates (kind 0) or the update
// matrix (kind 1): FP64 fronts choose between 64x64 tiles (4 warps, 4 CTAs
// per SM; the default, 28-30 TF/s on the large 64^3 update matrices; 32x32 on
// small launches) and 128x128 tiles (8 warps, one CTA per SM; 19 TF/s there), FP32 fronts between the
// two tcgen05 variants.  The choice comes from the autotuner's measurements
// (Plan::gemm_choice), the default variant otherwise.
template <typename T>
static bool gemm_alt(const Plan& P, int h, int kind) {
  const std::vector<uint8_t>& c = P.gemm_choice[sizeof(T) == 4 ? 1 : 0];
  return (size_t) (2 * h + kind) < c.size() && c[2 * h + kind] != 0;
}

// A launch of up to this many 64x64 tiles (three waves of four CTAs an SM) takes
// 32x32 tiles: four times the CTAs, so that every SM has several of them from the
// first to the last wave; beyond it the larger tile's reuse is worth more.  Panel
// products and update matrices of a 40x41x39 grid without and with them 3.44 and
// 2.64 ms; of 64^3, panel products 13.2 and 11.7, update matrices 27.3 instead of
// 22.9 if all took them.  Factor and solve with the line at 1184, 1776, 2368 and 3552
// tiles: 40x41x39 5.35, 5.32, 5.33, 5.33 ms; 64^3 42.8, 42.8, 42.8, 43.0.
constexpr int SMALL_TILES = 4 * 3 * GPU_SMS;
template <typename T>
static void launch_gemm(bool big, const LaunchWork& w128, const LaunchWork& w64, const LaunchWork& w32, const int* blst,
                        const DevPlan& D, T* L, T* U, int c_lo, int c_hi, int k_lo, int k_hi, int mode, int* status,
                        cudaStream_t st) {
  auto run = [&](auto k, const LaunchWork& w, int threads, size_t smem) {
    launch(k, w.total, threads, smem, st, D.work + w.off, w.nb, blst, D.fronts, L, U, c_lo, c_hi, k_lo, k_hi, mode,
           status);
  };
  using C32 = GemmCfg<32, 32>;
  using C64 = GemmCfg<64, 64>;
  using C128 = GemmCfg<128, 128>;
  if (big) run(k_gemm<T, 128, 128>, w128, C128::THREADS, C128::smem<T>());
  else if (w64.total <= SMALL_TILES) run(k_gemm<T, 32, 32>, w32, C32::THREADS, C32::smem<T>());
  else run(k_gemm<T, 64, 64>, w64, C64::THREADS, C64::smem<T>());
}

// FP32 fronts take the tcgen05 kernels (gemm_tc.cu): by default the one fed
// from the split arena (wsp), with `alt` the one whose producer warps split the
// operands as they load them
static void launch_gemm32(bool alt, const LaunchWork& wsp, const LaunchWork& w128, const LaunchWork& w64,
                          const LaunchWork& w32, const int* blst, const DevPlan& D, float* L, float* U, int c_lo,
                          int c_hi, int k_lo, int k_hi, int mode, int* status, cudaStream_t st, const float* sp,
                          int sp_fmt) {
  if (!alt && sp && gemm_sp_init())
    launch_gemm_sp(sp_fmt, wsp, D.work, blst, D.fronts, sp, L, U, c_lo, c_hi, k_lo, k_hi, mode, status, st);
  else if (gemm_tc_init())
    launch_gemm_tc(w128, D.work, blst, D.fronts, L, U, c_lo, c_hi, k_lo, k_hi, mode, status, st);
  else
    launch_gemm<float>(false, w128, w64, w32, blst, D, L, U, c_lo, c_hi, k_lo, k_hi, mode, status, st);
}

void plan_launches(const Plan& P, DevPlan* D, std::vector<int>& step_list, std::vector<int>& work) {
  D->level_work.clear();
  step_list.clear();
  work.clear();
  for (const LevelPlan& LP : P.levels) {
    LevelWork W;
    std::vector<int> order = LP.big_fronts;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return P.fronts[a].s > P.fronts[b].s; });
    step_list.insert(step_list.end(), order.begin(), order.end());
    // the fronts with more than c0 columns; n(F): CTAs of front F
    auto add = [&](int c0, auto n) {
      LaunchWork w;
      w.off = (int) work.size();
      for (int fi : order) {
        const FrontDesc& F = P.fronts[fi];
        if (F.s <= c0) break;
        w.total += n(F);
        work.push_back(w.total);
        w.nb++;
      }
      return w;
    };
    const int S = LP.max_s_big;
    for (int c = 0; c < S; c += PW) {
      auto below = [&](int rows) {
        return add(c, [&](const FrontDesc& F) { return (F.f - c - std::min(PW, F.s - c) + rows - 1) / rows; });
      };
      W.rows64.push_back(below(64));
      W.rows128.push_back(below(128));
      W.rows256.push_back(below(256));
      // the product into [c, c + lowest set bit of c), of the recursion below
      const int ce = c + (c & -c);
      auto tiles = [&](int b) {
        return c == 0 ? LaunchWork()
                      : add(c, [&](const FrontDesc& F) { return trap_tiles(F.f - c, std::min(ce, F.s) - c, b, b); });
      };
      W.u32.push_back(tiles(32));
      W.u64.push_back(tiles(64));
      W.u128.push_back(tiles(128));
    }
    auto update = [&](int b) {
      return add(0, [&](const FrontDesc& F) { return trap_tiles(F.f - F.s, F.f - F.s, b, b); });
    };
    W.m32 = update(32);
    W.m64 = update(64);
    W.m128 = update(128);
    W.msp = add(0, [&](const FrontDesc& F) { return F.f > F.s ? gemm_sp_tiles_u(F.s, F.f) : 0; });
    D->level_work.push_back(std::move(W));
  }
}

// CTAs of the persistent small-front launch: all that fit on the device at
// once with `smem` bytes each (the shared memory of the largest front in the
// persistent set: a set of small fronts fits many more CTAs per SM)
template <typename T>
static int pers_grid(size_t smem) {
  static PerDeviceOnce pd;
  static int sms[MAX_DEVICES];
  per_device_once(pd, [] {
    int d = 0;
    cudaGetDevice(&d);
    cudaDeviceGetAttribute(&sms[d], cudaDevAttrMultiProcessorCount, d);
    return true;
  });
  int d = 0;
  cudaGetDevice(&d);
  int b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_small_persistent<T>, 128, smem) != cudaSuccess) b = 1;
  return std::max(1, std::max(b, 1) * sms[d]);
}

// CTAs (four warps) of the one-warp-per-front persistent launch: all that
// fit on the device at once
template <typename T>
static int warp_grid() {
  static PerDeviceOnce pd;
  static int grid[MAX_DEVICES];
  per_device_once(pd, [] {
    int d = 0, sms = 0, b = 0;
    cudaGetDevice(&d);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, d);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_small_warp<T>, 128, 0) != cudaSuccess) b = 1;
    grid[d] = std::max(1, std::max(b, 1) * sms);
    return true;
  });
  int d = 0;
  cudaGetDevice(&d);
  return grid[d];
}

template <int N>
using Int = std::integral_constant<int, N>;

template <typename T>
static void set_smem_attrs() {
  // once per device and type (request-server workers reach this concurrently)
  static PerDeviceOnce pd;
  per_device_once(pd, [] {
    cudaFuncSetAttribute(k_small_front<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         SMALL_F_MAX * SMALL_F_MAX * (int) sizeof(T));
    cudaFuncSetAttribute(k_small_persistent<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         SMALL_F_MAX * SMALL_F_MAX * (int) sizeof(T));
    auto panel = [](auto fmt, auto nt, auto rows) {
      constexpr int NT = decltype(nt)::value, ROWS = decltype(rows)::value;
      cudaFuncSetAttribute(k_panel<T, decltype(fmt)::value, NT, ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int) panel_smem<T, ROWS>(PW));
    };
    panel(Int<0>(), Int<256>(), Int<64>());
    panel(Int<0>(), Int<512>(), Int<128>());
    if constexpr (sizeof(T) == 4) {
      panel(Int<0>(), Int<512>(), Int<256>());
      panel(Int<1>(), Int<256>(), Int<64>());
      panel(Int<1>(), Int<512>(), Int<128>());
      panel(Int<1>(), Int<512>(), Int<256>());
    }
    cudaFuncSetAttribute(k_dinv<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) dinv_smem<T>());
    cudaFuncSetAttribute(k_gemm<T, 32, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int) GemmCfg<32, 32>::smem<T>());
    cudaFuncSetAttribute(k_gemm<T, 64, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int) GemmCfg<64, 64>::smem<T>());
    cudaFuncSetAttribute(k_gemm<T, 128, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int) GemmCfg<128, 128>::smem<T>());
    return true;
  });
}

template <typename T>
static int launch_numeric(const Plan& P, const DevPlan& D, const T* vals, T* L, T* U, T* Dinv, float* sp,
                          int sp_fmt, int* status, cudaStream_t st) {
  set_smem_attrs<T>();
  {
    const int n = std::max(std::max(P.n_blk, D.n_pers), 2);
    launch(k_init_status, (n + 255) / 256, 256, 0, st, status, D.panel_done, P.n_blk, D.pers_pending0, D.pers_work,
        D.n_pers);
  }
  count_launch();
  if (D.n_pers > 0) {
    // every small front with only small fronts below it, in two launches:
    // one warp per front for the subtrees of fronts of order <= SMALL_WARP_F
    // (tasks 0 .. nw-1), then one CTA per front for the rest (their children
    // in the first part counted themselves off in the first launch)
    const int nw = P.pers_nwarp, np = D.n_pers;
    auto prof_range = [&](int t0, int t1, double& fl, double& by) {
      fl = by = 0.0;
      if (prof_enabled())
        for (int t = t0; t < t1; t++) {
          fl += front_flops(P.fronts[P.pers_fronts[t]]);
          by += front_bytes(P, P.fronts[P.pers_fronts[t]], sizeof(T));
        }
    };
    double fl, by;
    if (nw > 0) {
      const int grid = std::min((nw + 3) / 4, warp_grid<T>());
      prof_range(0, nw, fl, by);
      prof_begin(KC_SMALL, st);
      launch(k_small_warp<T>, grid, 128, 0, st, D.pers_list, 0, nw, D.pers_parent, D.pers_work, D.pers_work + np,
                                            D.fronts, D.children, D.maps, D.rows, D.acol_ptr, D.a_rows, D.a_idx,
                                            vals, L, U, status);
      prof_end(KC_SMALL, st, fl, by);
      count_launch();
    }
    if (np > nw) {
      const size_t smem = (size_t) P.pers_fmax * P.pers_fmax * sizeof(T);
      const int grid = std::min(np - nw, pers_grid<T>(smem));
      prof_range(nw, np, fl, by);
      prof_begin(KC_SMALL, st);
      launch(k_small_persistent<T>, grid, 128, smem, st, D.pers_list, nw, np, D.pers_parent, D.pers_work,
                                                     D.pers_work + np + 1, D.fronts, D.children, D.maps, D.rows,
                                                     D.acol_ptr, D.a_rows, D.a_idx, vals, L, U, status);
      prof_end(KC_SMALL, st, fl, by);
      count_launch();
    }
  }
  for (int h = 0; h < P.n_levels; h++) {
    const LevelPlan& LP = P.levels[h];
    prof_tag(h);
    // small fronts above a big one (the rest went through the persistent
    // launch), in size classes so that the shared-memory request fits the class
    const int ns = (int) LP.small_numeric.size();
    if (ns > 0) {
      const int* lst = D.small_num + D.small_num_off[h];
      int b = 0;
      const int classes[3] = {32, 64, SMALL_F_MAX};
      for (int cl = 0; cl < 3 && b < ns; cl++) {
        int e = b;
        while (e < ns && P.fronts[LP.small_numeric[e]].f <= classes[cl]) e++;
        if (e > b) {
          const size_t smem = (size_t) classes[cl] * classes[cl] * sizeof(T);
          double fl = 0.0, by = 0.0;
          if (prof_enabled())
            for (int q = b; q < e; q++) {
              const FrontDesc& F = P.fronts[LP.small_numeric[q]];
              fl += front_flops(F);
              by += front_bytes(P, F, sizeof(T));
            }
          prof_begin(KC_SMALL, st);
          launch(k_small_front<T>, e - b, 128, smem, st, lst + b, D.fronts, D.children, D.maps, D.rows,
                                                   D.acol_ptr, D.a_rows, D.a_idx, vals, L, U, status);
          prof_end(KC_SMALL, st, fl, by);
          count_launch();
        }
        b = e;
      }
    }
    if (LP.big_fronts.empty()) continue;
    const int ntiles = (int) LP.build_tiles.size();
    {
      double by = 0.0;
      if (prof_enabled())
        for (int fi : LP.big_fronts) by += build_bytes(P, P.fronts[fi], sizeof(T));
      prof_begin(KC_BUILD, st);
      launch(k_build<T>, ntiles, BUILD_THREADS, 0, st, D.tiles + D.tile_off[h], D.tile_ch, D.fronts, D.maps, D.acol_ptr,
                                      D.a_rows, D.a_idx, vals, L, U, status);
      prof_end(KC_BUILD, st, 0.0, by);
      count_launch();
    }
    // recursive panel factorization over aligned column intervals: factor
    // the left half, update the right half with one GEMM (K = half width),
    // factor the right half; the intervals of PW columns are panel steps
    const int S = LP.max_s_big;
    int span = PW;
    while (span < S) span *= 2;
    const LevelWork& LW = D.level_work[h];
    const int* slst = D.step_list + D.big_off[h];
    auto panel = [&](int kb) {
      const int k = kb / PW, nsteps = LW.rows64[k].nb;
      int wmax = 0;
      double fl = 0.0, by = 0.0;
      for (int fi : LP.big_fronts) {
        const FrontDesc& F = P.fronts[fi];
        if (kb >= F.s) continue;
        const int w = std::min(PW, F.s - kb);
        wmax = std::max(wmax, w);
        if (prof_enabled()) {
          const double ww = w, below = F.f - kb - w;
          fl += ww * ww * ww / 3.0 + below * ww * ww;
          by += 2.0 * sizeof(T) * (ww * (ww + 1.0) / 2.0 + below * ww);
        }
      }
      prof_begin(KC_LEAF, st);
      auto run = [&](auto fmt, auto nt, auto rows) {
        constexpr int NT = decltype(nt)::value, ROWS = decltype(rows)::value;
        const LaunchWork& w = ROWS == 64 ? LW.rows64[k] : ROWS == 128 ? LW.rows128[k] : LW.rows256[k];
        launch(k_panel<T, decltype(fmt)::value, NT, ROWS>, nsteps + w.total, NT, panel_smem<T, ROWS>(wmax), st,
               D.work + w.off, nsteps, slst, D.fronts, D.rows, L, sp, kb, D.panel_done, D.panel_rdiag, status);
      };
      // 16 warps a CTA and 128 rows while every CTA has an SM to itself (29x24x26
      // FP32: 0.80 ms of panels -> 0.72); on fuller launches 8 warps and 64 rows,
      // where two CTAs share an SM and one's updates fill the other's waits, or
      // (FP32: they fit) 16 warps and 256 rows.  64 rows take 35 us for the first
      // wave, which ends with the chain of pivots, and 28 for each further one; 256
      // rows 43 a wave.  80^3 FP32: panel steps 12.3 -> 10.9 ms
      auto size = [&](auto fmt) {
        if (nsteps + LW.rows128[k].total <= GPU_SMS) return run(fmt, Int<512>(), Int<128>());
        if constexpr (sizeof(T) == 4)
        {
          auto waves = [&](const LaunchWork& w, int at_once) { return (nsteps + w.total + at_once - 1) / at_once; };
          if (43 * waves(LW.rows256[k], GPU_SMS) < 7 + 28 * waves(LW.rows64[k], 2 * GPU_SMS))
            return run(fmt, Int<512>(), Int<256>());
        }
        run(fmt, Int<256>(), Int<64>());
      };
      if constexpr (sizeof(T) == 4) {
        if (sp_fmt) size(Int<1>());
        else size(Int<0>());
      } else {
        size(Int<0>());
      }
      prof_end(KC_LEAF, st, fl, by);
      count_launch();
    };
    // the product with the columns [k_lo, k_hi) into [c_lo, c_hi); c_hi - c_lo is
    // c_lo's lowest set bit
    auto update = [&](int c_lo, int c_hi, int k_lo, int k_hi) {
      double fg = 0.0, bg = 0.0;
      if (prof_enabled())
        for (int fi : LP.big_fronts) {
          const FrontDesc& F = P.fronts[fi];
          const int ce = std::min(c_hi, F.s);
          if (c_lo >= ce) continue;
          const double c = ce - c_lo, below = F.f - ce, k = k_hi - k_lo;
          const double entries = c * (c + 1.0) / 2.0 + below * c;
          fg += 2.0 * k * entries;
          bg += 2.0 * sizeof(T) * entries + sizeof(T) * k * (F.f - c_lo);
        }
      const int k = c_lo / PW;
      prof_begin(KC_GEMM_PANEL, st);
      if constexpr (sizeof(T) == 4)
        launch_gemm32(gemm_alt<T>(P, h, 0), LW.u128[k], LW.u128[k], LW.u64[k], LW.u32[k], slst, D, L, U, c_lo, c_hi,
                      k_lo, k_hi, 0, status, st, sp, sp_fmt);
      else
        launch_gemm(gemm_alt<T>(P, h, 0), LW.u128[k], LW.u64[k], LW.u32[k], slst, D, L, U, c_lo, c_hi, k_lo, k_hi, 0,
                    status, st);
      prof_end(KC_GEMM_PANEL, st, fg, bg);
      count_launch();
    };
    struct Rec {
      static void run(int a, int b, int S_, const decltype(panel)& lf, const decltype(update)& up) {
        if (a >= S_) return;
        if (b - a <= PW) { lf(a); return; }
        const int mid = (a + b) / 2;
        run(a, mid, S_, lf, up);
        if (mid < S_) up(mid, b, a, mid);
        run(mid, b, S_, lf, up);
      }
    };
    Rec::run(0, span, S, panel, update);
    if (LW.m64.total > 0) {
      double fu = 0.0, bu = 0.0;
      if (prof_enabled())
        for (int fi : LP.big_fronts) {
          const FrontDesc& F = P.fronts[fi];
          const double m = F.f - F.s;
          fu += 2.0 * F.s * m * (m + 1.0) / 2.0;
          bu += 2.0 * sizeof(T) * m * (m + 1.0) / 2.0 + sizeof(T) * m * F.s;
        }
      prof_begin(KC_GEMM_U, st);
      if constexpr (sizeof(T) == 4)
        launch_gemm32(gemm_alt<T>(P, h, 1), LW.msp, LW.m128, LW.m64, LW.m32, slst, D, L, U, 0, 0, 0, 0, 1, status, st,
                      sp, sp_fmt);
      else
        launch_gemm(gemm_alt<T>(P, h, 1), LW.m128, LW.m64, LW.m32, slst, D, L, U, 0, 0, 0, 0, 1, status, st);
      prof_end(KC_GEMM_U, st, fu, bu);
      count_launch();
    }
  }
  prof_tag(-1);
  if (D.n_dblk > 0) {
    prof_begin(KC_DINV, st);
    launch(k_dinv<T>, D.n_dblk, 128, dinv_smem<T>(), st, D.dblk, D.fronts, L, Dinv, status);
    prof_end(KC_DINV, st, (double) D.n_dblk * PANEL_NB * PANEL_NB * PANEL_NB / 3.0,
             2.0 * sizeof(T) * D.n_dblk * PANEL_NB * PANEL_NB);
    count_launch();
  }
  return (int) cudaGetLastError();
}

int launch_tile_ranges(const DevPlan& D, int ntiles, cudaStream_t st) {
  launch(k_tile_ranges, ntiles, 128, 0, st, D.tiles, D.fronts, D.children, D.maps, D.tile_ch);
  return (int) cudaGetLastError();
}

int launch_numeric_fp64(const Plan& P, const DevPlan& D, const double* vals, double* L, double* U, double* Dinv,
                        int* status, cudaStream_t st) {
  return launch_numeric<double>(P, D, vals, L, U, Dinv, nullptr, 0, status, st);
}

int launch_numeric_fp32(const Plan& P, const DevPlan& D, const float* vals, float* L, float* U, float* Dinv,
                        float* sp, int sp_fmt, int* status, cudaStream_t st) {
  return launch_numeric<float>(P, D, vals, L, U, Dinv, sp, sp_fmt, status, st);
}

}  // namespace tb
