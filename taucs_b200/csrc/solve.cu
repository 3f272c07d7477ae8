// FP64 supernodal triangular solve on sm_100a, level scheduled.
//
// The reference solves one right-hand side per call by recursion
// (src/taucs_sn_llt.c:2596-2885): forward in postorder -- gather b at the
// supernode's columns, TRSM with L11, GEMM with L21, scatter-subtract into b
// at the update rows -- and backward in preorder with L21^T and L11^T.
//
// Here the forward pass is written multifrontally so that no two CTAs ever
// write the same vector entry: each front owns a work vector of f entries
// per right-hand side (W, at the front's row offset).  A front's forward step
// gathers b at its columns, adds its children's update vectors (their W rows
// s..f-1) through the child->parent maps in the fixed child order, solves
// with L11 and leaves y in W[0..s) and the update vector u = w2 - L21 y in
// W[s..f).  The backward pass runs the levels in reverse: gather x at the
// update rows (written by ancestors in earlier launches), r = y - L21^T x2,
// then the L11^T substitution, and scatter x at the columns.  Up to
// SOLVE_NRHS right-hand sides share every read of L.
#include <climits>
#include <mutex>
#include <type_traits>

#include "factor.h"
#include "kernels.h"
#include "launch.h"

namespace tb {

namespace {

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

constexpr int SB = 32;   // substitution block (one warp)

// ------------------------------------------------------------- small fronts
// Fronts of order f <= SMALL_F_MAX, one warp each.  What bounds them is
// latency (a 33 x 33 grid is a chain of 8 dependent fronts each way), so a
// front's data are on their way before its dependency is waited for: the
// task's record (SolveTask: one 32-byte load instead of list entry, then
// descriptor), its panel (element-wise asynchronous copies into the warp's
// slot of shared memory, column stride f | 1 so that both the row reads of
// the forward pass and the column reads of the backward pass are free of bank
// conflicts), its right-hand side entries and its children's records.  After
// the wait one round of loads fetches the neighbours' vectors, and the
// substitution runs from shared memory and registers: lane l holds rows l,
// l + 32, l + 64, and a step costs a shuffle and a multiply-add (the column
// is divided by its pivot off the chain).  A panel larger than the slot goes
// through it in column pieces.  Both persistent launches together, one
// right-hand side: 33 x 33 grid, FP64, 140 -> 54 us forward and 72 -> 50 us
// backward; 512 grids at once, FP32, a refined solution's three passes 12.5 ->
// 8.7 ms.
constexpr int SF_SLOTS = (SMALL_F_MAX + 31) / 32;   // rows per lane

__device__ __forceinline__ void cp_async_elem(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned) __cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void cp_async_elem(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned) __cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void cp_async_wait_warp() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
}

// the lower part of columns [ja, je) of a panel (ld f) into pan (ld f | 1)
template <typename T>
__device__ __forceinline__ void stage_columns(const T* P, int f, int ja, int je, T* pan) {
  const int lane = threadIdx.x & 31, ld = f | 1;
  for (int j = ja; j < je; j++)
    for (int r = (j & ~31) + lane; r < f; r += 32)
      if (r >= j) cp_async_elem(pan + (size_t) (j - ja) * ld + r, P + r + (size_t) j * f);
}

// columns a slot of `slot` elements holds of a panel of order f
__device__ __forceinline__ int slot_columns(int slot, int f) { return slot / (f | 1); }

// what a warp holds of its front before the dependency wait of the forward
// step: the first piece of the panel on its way, b at its columns in ws (zero
// in the other rows), and the records of the first 32 children in the lanes
template <typename T, int NQ>
__device__ __forceinline__ int4 fwd_front_begin(const SolveTask& K, const int4* __restrict__ child_rec,
                                                const int* __restrict__ rows, const T* __restrict__ L,
                                                const T* __restrict__ B, int ldb, int nrhs, T* pan, int slot, T* ws,
                                                int wld) {
  const int lane = threadIdx.x & 31, f = K.f, s = K.s;
  stage_columns(L + K.l_off, f, 0, min(s, slot_columns(slot, f)), pan);
  int g[SF_SLOTS];
#pragma unroll
  for (int k = 0; k < SF_SLOTS; k++) g[k] = lane + 32 * k < s ? __ldg(rows + K.rows_off + lane + 32 * k) : -1;
  const int4 rec = lane < K.child_end - K.child_begin ? __ldg(child_rec + K.child_begin + lane) : make_int4(0, 0, 0, 0);
#pragma unroll
  for (int k = 0; k < SF_SLOTS; k++)
    if (32 * k < f) {
#pragma unroll
      for (int q = 0; q < NQ; q++)
        if (lane + 32 * k < f)
          ws[q * wld + lane + 32 * k] = (g[k] >= 0 && q < nrhs) ? B[g[k] + (size_t) q * ldb] : T(0);
    }
  return rec;
}

// the forward step itself, once the children are done: their update vectors
// added in child order, then y = L11^-1 w and u = w2 - L21 y into W
template <typename T, int NQ, int WS>
__device__ __forceinline__ void fwd_front(const SolveTask& K, int4 rec, const int4* __restrict__ child_rec,
                                          const int* __restrict__ maps, const T* __restrict__ L, T* __restrict__ W,
                                          int nrhs, T* pan, int slot, T* ws, int wld) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, f = K.f, s = K.s, ld = f | 1;
  const int nch = K.child_end - K.child_begin;
  for (int c0 = 0; c0 < nch; c0 += 32) {
    if (c0 > 0) rec = c0 + lane < nch ? __ldg(child_rec + K.child_begin + c0 + lane) : make_int4(0, 0, 0, 0);
    // CB children per round: all their loads before the first add
    constexpr int CB = NQ == 1 ? 4 : NQ <= 4 ? 2 : 1;
    const int ce = min(32, nch - c0);
    for (int c = 0; c < ce; c += CB) {
      int pi[CB][SF_SLOTS];
      T val[CB][SF_SLOTS][NQ];
#pragma unroll
      for (int u = 0; u < CB; u++) {
        const int src = (c + u) & 31;
        const int voff = __shfl_sync(FULL, rec.x, src), cs = __shfl_sync(FULL, rec.y, src),
                  cf = __shfl_sync(FULL, rec.z, src), mo = __shfl_sync(FULL, rec.w, src);
        const int mc = c + u < ce ? cf - cs : 0;
        const T* Wc = W + (int64_t) voff * WS + cs;
#pragma unroll
        for (int k = 0; k < SF_SLOTS; k++) {
          const int i = lane + 32 * k;
          pi[u][k] = i < mc ? __ldg(maps + mo + i) : -1;
#pragma unroll
          for (int q = 0; q < NQ; q++) val[u][k][q] = (i < mc && q < nrhs) ? __ldcg(Wc + i + (size_t) q * cf) : T(0);
        }
      }
#pragma unroll
      for (int u = 0; u < CB; u++) {
        __syncwarp();
#pragma unroll
        for (int k = 0; k < SF_SLOTS; k++)
          if (pi[u][k] >= 0) {
#pragma unroll
            for (int q = 0; q < NQ; q++) ws[q * wld + pi[u][k]] += val[u][k][q];
          }
      }
    }
  }
  __syncwarp();
  T v[SF_SLOTS][NQ], rd[SF_SLOTS];
#pragma unroll
  for (int k = 0; k < SF_SLOTS; k++)
#pragma unroll
    for (int q = 0; q < NQ; q++) v[k][q] = lane + 32 * k < f ? ws[q * wld + lane + 32 * k] : T(0);
  const int cw = slot_columns(slot, f);
#pragma unroll
  for (int k = 0; k < SF_SLOTS; k++) rd[k] = T(0);
  int staged = 0;   // first column of the staged piece
  cp_async_wait_warp();
  for (int ja = 0; ja < s;) {
    if (ja >= staged + cw) {   // the next piece of a panel larger than the slot
      __syncwarp();
      stage_columns(L + K.l_off, f, ja, min(s, ja + cw), pan);
      staged = ja;
      cp_async_wait_warp();
    }
    const int je = min(min(s, staged + cw), (ja & ~31) + 32), kb = ja >> 5;
    const T* pc = pan - (size_t) staged * ld;
    // columns [ja, je), all in row slot kb
#pragma unroll
    for (int b = 0; b < SF_SLOTS; b++) {
      if (b != kb) continue;
      const int own = 32 * b + lane;
      if (own >= ja && own < je) rd[b] = T(1) / pc[own + own * ld];
      // lane l holds 1 / L_ll for the columns of this piece
#pragma unroll 4
      for (int j = ja; j < je; j++) {
        const T rj = __shfl_sync(FULL, rd[b], j & 31);
        T l[SF_SLOTS];
#pragma unroll
        for (int k = b; k < SF_SLOTS; k++) {
          const int r = lane + 32 * k;
          l[k] = (r > j && r < f) ? pc[r + j * ld] * rj : T(0);
        }
#pragma unroll
        for (int q = 0; q < NQ; q++) {
          const T vj = __shfl_sync(FULL, v[b][q], j & 31);
#pragma unroll
          for (int k = b; k < SF_SLOTS; k++) v[k][q] -= l[k] * vj;
        }
      }
    }
    ja = je;
  }
  T* Wf = W + (int64_t) K.rows_off * WS;
#pragma unroll
  for (int k = 0; k < SF_SLOTS; k++) {
    const int r = lane + 32 * k;
    if (r < f) {
#pragma unroll
      for (int q = 0; q < NQ; q++)
        if (q < nrhs) Wf[r + (size_t) q * f] = r < s ? v[k][q] * rd[k] : v[k][q];
    }
  }
}

// columns of one piece of the backward step: a block of 32, or fewer when the
// slot does not hold the whole panel
__device__ __forceinline__ int bwd_piece(int slot, int f, int s) {
  const int cw = slot_columns(slot, f);
  return cw >= s ? SB : min(SB, cw);
}

// the backward step before the wait for the parent: the last piece of the
// panel (the whole panel when the slot holds it) on its way, y in ws, and the
// global rows of the lane's local rows
template <typename T, int NQ, int WS>
__device__ __forceinline__ void bwd_front_begin(const SolveTask& K, const int* __restrict__ rows,
                                                const T* __restrict__ L, const T* W, int nrhs, T* pan,
                                                int slot, T* ws, int wld, int (&g)[SF_SLOTS]) {
  const int lane = threadIdx.x & 31, f = K.f, s = K.s;
  const int ja = slot_columns(slot, f) >= s ? 0 : max(0, s - bwd_piece(slot, f, s));
  stage_columns(L + K.l_off, f, ja, s, pan);
  const T* Wf = W + (int64_t) K.rows_off * WS;
#pragma unroll
  for (int k = 0; k < SF_SLOTS; k++) {
    const int r = lane + 32 * k;
    g[k] = r < f ? __ldg(rows + K.rows_off + r) : -1;
    if (r < s) {
#pragma unroll
      for (int q = 0; q < NQ; q++) ws[q * wld + r] = q < nrhs ? Wf[r + (size_t) q * f] : T(0);
    }
  }
}

// the backward step once x at the update rows is final: per piece of columns
// from the last, r = y - L[below, piece]^T x_below (lane (column c, part p)
// sums every 32 / columns-th row; the parts are added by shuffles), then the
// L11^T substitution
template <typename T, int NQ>
__device__ __forceinline__ void bwd_front(const SolveTask& K, const T* __restrict__ L, T* __restrict__ X, int ldx,
                                          int nrhs, T* pan, int slot, T* ws, int wld, const int (&g)[SF_SLOTS]) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, f = K.f, s = K.s, ld = f | 1;
  {
    T x[SF_SLOTS][NQ];
#pragma unroll
    for (int k = 0; k < SF_SLOTS; k++)
#pragma unroll
      for (int q = 0; q < NQ; q++)
        x[k][q] = (g[k] >= 0 && lane + 32 * k >= s && q < nrhs) ? __ldcg(X + g[k] + (size_t) q * ldx) : T(0);
#pragma unroll
    for (int k = 0; k < SF_SLOTS; k++)
      if (g[k] >= 0 && lane + 32 * k >= s) {
#pragma unroll
        for (int q = 0; q < NQ; q++) ws[q * wld + lane + 32 * k] = x[k][q];
      }
  }
  const int pw = bwd_piece(slot, f, s);
  const bool whole = slot_columns(slot, f) >= s;
  cp_async_wait_warp();
  for (int je = s; je > 0;) {
    // the last piece is the ragged one when the panel goes block by block
    const int ja = whole ? (je - 1) & ~31 : max(0, je - pw), bw = je - ja;
    if (!whole && je < s) {
      __syncwarp();
      stage_columns(L + K.l_off, f, ja, je, pan);
      cp_async_wait_warp();
    }
    const T* pc = whole ? pan : pan - (size_t) ja * ld;
    int cwp = 1;
    while (cwp < bw) cwp <<= 1;
    const int c = lane & (cwp - 1), part = lane / cwp, np = 32 / cwp;
    const bool own = c < bw;
    const T* pj = pc + (ja + (own ? c : 0)) * ld;
    T acc[NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) acc[q] = T(0);
#pragma unroll 4
    for (int i = je + part; i < f; i += np) {
      const T l = pj[i];
#pragma unroll
      for (int q = 0; q < NQ; q++) acc[q] += l * ws[q * wld + i];
    }
    for (int o = cwp; o < 32; o <<= 1)
#pragma unroll
      for (int q = 0; q < NQ; q++) acc[q] += __shfl_xor_sync(FULL, acc[q], o);
    const T rd = own ? T(1) / pj[ja + c] : T(0);
    T v[NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) v[q] = own ? ws[q * wld + ja + c] - acc[q] : T(0);
#pragma unroll 4
    for (int k = bw - 1; k > 0; k--) {
      const T rk = __shfl_sync(FULL, rd, k);
      const T l = (own && c < k) ? pj[ja + k] * rk : T(0);
#pragma unroll
      for (int q = 0; q < NQ; q++) v[q] -= l * __shfl_sync(FULL, v[q], k);
    }
    __syncwarp();
    if (own && part == 0) {
#pragma unroll
      for (int q = 0; q < NQ; q++) ws[q * wld + ja + c] = v[q] * rd;
    }
    __syncwarp();
    je = ja;
  }
#pragma unroll
  for (int k = 0; k < SF_SLOTS; k++)
    if (lane + 32 * k < s) {
#pragma unroll
      for (int q = 0; q < NQ; q++)
        if (q < nrhs) X[g[k] + (size_t) q * ldx] = ws[q * wld + lane + 32 * k];
    }
}

// elements of a warp's slot and vectors in the dynamic shared memory of the
// small-front kernels: wld is the largest order among the launch's fronts
template <typename T, int NQ>
__host__ __device__ constexpr size_t sf_warp_smem(int slot, int wld) {
  return ((size_t) slot + (size_t) NQ * wld) * sizeof(T);
}

__device__ __forceinline__ SolveTask task_of(const FrontDesc& F) {
  return SolveTask{F.l_off, F.rows_off, F.s, F.f, F.child_begin, F.child_end, -1};
}

// level launches: the small fronts with a big front below them (and every
// small front of the allocation-free solve), a warp each, no waits
template <typename T, int NQ, int WS>
__global__ void __launch_bounds__(128)
k_fwd(const int* __restrict__ list, int count, const FrontDesc* __restrict__ fronts, const int4* __restrict__ child_rec,
      const int* __restrict__ maps, const int* __restrict__ rows, const T* __restrict__ L, const T* __restrict__ B,
      int ldb, T* __restrict__ W, int nrhs, int slot, int wld) {
  extern __shared__ __align__(16) unsigned char sfm[];
  const int wi = threadIdx.x >> 5, li = blockIdx.x * (blockDim.x >> 5) + wi;
  if (li >= count) return;
  T* pan = reinterpret_cast<T*>(sfm + wi * sf_warp_smem<T, NQ>(slot, wld));
  const SolveTask K = task_of(fronts[list[li]]);
  const int4 rec = fwd_front_begin<T, NQ>(K, child_rec, rows, L, B, ldb, nrhs, pan, slot, pan + slot, wld);
  grid_wait();
  fwd_front<T, NQ, WS>(K, rec, child_rec, maps, L, W, nrhs, pan, slot, pan + slot, wld);
}

template <typename T, int NQ, int WS>
__global__ void __launch_bounds__(128)
k_bwd(const int* __restrict__ list, int count, const FrontDesc* __restrict__ fronts, const int* __restrict__ rows,
      const T* __restrict__ L, T* __restrict__ X, int ldx, const T* W, int nrhs, int slot, int wld) {
  grid_wait();
  extern __shared__ __align__(16) unsigned char sfm[];
  const int wi = threadIdx.x >> 5, li = blockIdx.x * (blockDim.x >> 5) + wi;
  if (li >= count) return;
  T* pan = reinterpret_cast<T*>(sfm + wi * sf_warp_smem<T, NQ>(slot, wld));
  const SolveTask K = task_of(fronts[list[li]]);
  int g[SF_SLOTS];
  bwd_front_begin<T, NQ, WS>(K, rows, L, W, nrhs, pan, slot, pan + slot, wld, g);
  __syncwarp();
  bwd_front<T, NQ>(K, L, X, ldx, nrhs, pan, slot, pan + slot, wld, g);
}

// Waits (bounded) until *p holds v.  Every lane of the warp polls and the loop
// ends by a vote: after a loop run by one lane alone the warp stays split, and
// the shuffles of the substitution that follows issue once per part of it
// (backward launch over a 33 x 33 grid's fronts, FP64, one right-hand side:
// 148 us with one lane polling, 72 us with the whole warp).
__device__ __forceinline__ void warp_wait_value(const int* p, int v, int* status) {
  int it = 0;
  while (!__all_sync(0xffffffffu, ld_acquire(p) == v)) {
    if (++it > (1 << 22)) {
      atomicExch(status, SOLVE_TIMEOUT);
      break;
    }
    __nanosleep(20);
  }
}

// The small fronts with only small fronts below them (Plan::pers_fronts),
// tasks [t0, t1) of their queue in one launch: each warp takes the next front
// from a device-side queue.  Forward, in level order: a front waits until its
// children's update vectors are in place (pending count), and counts itself
// off at its parent.  Backward, in reverse level order: a front waits until
// its parent has written x at its update rows (done flag = epoch; parents
// outside the set ran in the level launches before this one).  A warp claims
// its next task before it works on the current one; the oldest unfinished
// task is always the current one of its warp, so every wait ends.  Every wait
// is bounded all the same (SOLVE_TIMEOUT).
template <typename T, int NQ, int WS>
__global__ void __launch_bounds__(256, NQ == 1 ? 4 : sizeof(T) == 4 ? 3 : 2)
k_fwd_pers(const SolveTask* __restrict__ tasks, int t0, int t1, int* pending, int* next,
           const int4* __restrict__ child_rec, const int* __restrict__ maps, const int* __restrict__ rows,
           const T* __restrict__ L, const T* __restrict__ B, int ldb, T* __restrict__ W, int nrhs, int* status,
           int slot, int wld) {
  grid_wait();
  extern __shared__ __align__(16) unsigned char sfm[];
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  T* pan = reinterpret_cast<T*>(sfm + wi * sf_warp_smem<T, NQ>(slot, wld));
  T* ws = pan + slot;
  int t = 0;
  if (lane == 0) t = t0 + atomicAdd(next, 1);
  t = __shfl_sync(0xffffffffu, t, 0);
  while (t < t1) {
    int tn = 0;
    if (lane == 0) tn = t0 + atomicAdd(next, 1);
    const SolveTask K = tasks[t];
    const int4 rec = fwd_front_begin<T, NQ>(K, child_rec, rows, L, B, ldb, nrhs, pan, slot, ws, wld);
    if (K.child_end > K.child_begin) warp_wait_value(pending + t, 0, status);
    fwd_front<T, NQ, WS>(K, rec, child_rec, maps, L, W, nrhs, pan, slot, ws, wld);
    __syncwarp();
    if (lane == 0 && K.parent >= 0) {
      __threadfence();
      atomicSub(pending + K.parent, 1);
    }
    t = __shfl_sync(0xffffffffu, tn, 0);
  }
}

template <typename T, int NQ, int WS>
__global__ void __launch_bounds__(256, NQ == 1 ? 4 : sizeof(T) == 4 ? 3 : 2)
k_bwd_pers(const SolveTask* __restrict__ tasks, int t0, int t1, int* done, int* next, int epoch,
           const int* __restrict__ rows, const T* __restrict__ L, T* __restrict__ X, int ldx, const T* W,
           int nrhs, int* status, int slot, int wld) {
  grid_wait();
  extern __shared__ __align__(16) unsigned char sfm[];
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  T* pan = reinterpret_cast<T*>(sfm + wi * sf_warp_smem<T, NQ>(slot, wld));
  T* ws = pan + slot;
  int t = 0;
  if (lane == 0) t = t1 - 1 - atomicAdd(next, 1);
  t = __shfl_sync(0xffffffffu, t, 0);
  while (t >= t0) {
    int tn = 0;
    if (lane == 0) tn = t1 - 1 - atomicAdd(next, 1);
    const SolveTask K = tasks[t];
    int g[SF_SLOTS];
    bwd_front_begin<T, NQ, WS>(K, rows, L, W, nrhs, pan, slot, ws, wld, g);
    if (K.parent >= 0) warp_wait_value(done + K.parent, epoch, status);
    else __syncwarp();
    bwd_front<T, NQ>(K, L, X, ldx, nrhs, pan, slot, ws, wld, g);
    __syncwarp();
    if (lane == 0 && K.child_end > K.child_begin) {
      __threadfence();
      atomicExch(done + t, epoch);
    }
    t = __shfl_sync(0xffffffffu, tn, 0);
  }
}


// ---------------------------------------------------------------- big fronts
// 64-row blocks.  Forward: block r needs the solved blocks k < r of L11,
// accumulates L[r,k] y_k and applies the inverse of its diagonal block.
// Backward: blocks run from the last one; block k needs x_j, j > k.  Waits are
// bounded: on timeout a CTA records SOLVE_TIMEOUT in the status word and
// carries on, so no launch can hang.

constexpr int BR = PANEL_NB;   // rows per block
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

}  // namespace

// Controls of the handshake waits through global memory on this device: the
// polling limit, and an offset added to the flag value waited for (0; any other
// value makes every wait run out -- a testing aid for the timeout reporting, set
// through taucs_b200_debug_waits).
__device__ int g_solve_wait_limit = 1 << 22;
__device__ int g_solve_wait_skew = 0;

int solve_set_wait_controls(int limit, int skew) {
  cudaError_t e = cudaMemcpyToSymbol(g_solve_wait_limit, &limit, sizeof(int));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_solve_wait_skew, &skew, sizeof(int));
  return (int) e;
}

namespace {

// polls flag until it holds epoch (plus the wait offset); on giving up,
// records SOLVE_TIMEOUT.  Called by whole warps: every lane polls and the loop
// ends by a vote, so the warp leaves it undivided (a loop run by one lane
// leaves the warp split through the code that follows).
__device__ __forceinline__ void poll_epoch(const int* flag, int epoch, int* status) {
  const int want = epoch + g_solve_wait_skew, limit = g_solve_wait_limit;
  int it = 0;
  while (!__all_sync(0xffffffffu, ld_acquire(flag) == want)) {
    // a wait that gave up anywhere ends the others at once, so a broken
    // chain costs one polling limit, not one per wait
    ++it;
    if (__any_sync(0xffffffffu, it > limit || ((it & 1023) == 0 && *(volatile int*) status == SOLVE_TIMEOUT))) {
      atomicExch(status, SOLVE_TIMEOUT);
      break;
    }
    __nanosleep(32);
  }
}

// the same wait for every warp of a CTA: the first warp polls
__device__ void wait_epoch(const int* flag, int epoch, int* status) {
  if (threadIdx.x < 32) poll_epoch(flag, epoch, status);
  __syncthreads();
}


// The children's update rows that land in a 64-row block, added into wv in
// child order (the order of the block's records, found once per plan: the
// kernels used to look each child's descriptor and range up, some 3 us a
// child: forward solve at 29x24x26, FP32, three passes, 1030 -> 805 us; at
// 64^3, FP64, 1425 -> 1285 us).  NT threads, thread t on row t % 64 of every
// record; the loads of GC children are issued before the first add, those of
// the first group by load(), ahead of whatever else the block loads.
template <typename T, int NQ, int WS, int NT>
struct ChildGather {
  static constexpr int GC = 4, QS = NT / BR, QN = (NQ + QS - 1) / QS;
  int pi[GC];
  T val[GC][QN];
  __device__ __forceinline__ void load(const int4* __restrict__ rec, int n, const int* __restrict__ maps,
                                       const T* W, int nrhs) {
    const int i = threadIdx.x % BR, q0 = threadIdx.x / BR;
#pragma unroll
    for (int u = 0; u < GC; u++) {
      const int4 R = u < n ? __ldg(rec + u) : make_int4(0, 0, 0, 0);
      const bool in = i < (R.z & 127) && q0 < QS;   // threads past NT take no row
      pi[u] = in ? __ldg(maps + R.w + i) : -1;
      const T* Wc = W + (int64_t) R.x * WS + R.y + i;
#pragma unroll
      for (int t = 0; t < QN; t++) {
        const int q = q0 + QS * t;
        val[u][t] = (in && q < nrhs) ? Wc[(size_t) q * (R.z >> 7)] : T(0);
      }
    }
  }
  // adds the loaded group (already begun) and the later ones into wv rows
  // pi - r0; every thread of the block calls it, before a barrier of its own
  template <int LD>
  __device__ __forceinline__ void add(const int4* __restrict__ rec, int n, const int* __restrict__ maps,
                                      const T* W, int nrhs, int r0, T (*wv)[LD]) {
    const int q0 = threadIdx.x / BR;
    for (int c = 0; c < n; c += GC) {
      if (c > 0) load(rec + c, n - c, maps, W, nrhs);
#pragma unroll
      for (int u = 0; u < GC; u++) {
        if (c + u >= n) break;
        if (pi[u] >= 0)
#pragma unroll
          for (int t = 0; t < QN; t++)
            if (q0 + QS * t < NQ) wv[pi[u] - r0][q0 + QS * t] += val[u][t];
        __syncthreads();
      }
    }
  }
};

constexpr int CH_C = 8;                       // CTAs of a cluster, and the near distance
constexpr int CH_RING = 2 * CH_C;
constexpr int CH_THREADS = 256;
constexpr int CH_VALUES = BR * SOLVE_NRHS;    // values per block and array of published words
constexpr int DLD = BR + 4;                   // column stride of a staged inverse
constexpr int CH_HB = 2;                      // blocks per round of a helper's far terms
// Levels with at least CHAIN_MIN_S columns in their largest big front and at
// most chain_max_fronts() big fronts run as chains.  The number of fronts is
// bounded by residency: walkers wait for helpers of the same launch, and 16
// clusters of 8 are 128 of the 296 CTAs that the GPU holds at two an SM.  Within
// that the lines lie on flat ground.  ms with chains from 128, 256 and 512
// columns on, on no level, and with half the fronts: solve with 64^3's factor 2.00,
// 2.00, 2.00, 2.15, 2.02; 32 columns at 45x47x44 4.50, 4.50, 4.48, 4.56, 4.44; refined
// solution at 56^3 5.27, 5.27, 5.22, 5.56, 5.22; mixed step at 80^3 46.0, 46.0, 46.0,
// 46.5, 46.0, at 29x24x26 2.14, 2.16, 2.16, 2.16, 2.16.  FP64 with 16 fronts: 45x47x44
// 4.55.
constexpr int CHAIN_MIN_S = 256;
template <typename T>
constexpr int chain_max_fronts() { return sizeof(T) == 4 ? 16 : 8; }

template <typename T>
__host__ __device__ constexpr int ch_words() { return (int) sizeof(T) / 4; }   // words per published value

// one published value
template <typename T>
struct Tagged;
template <>
struct Tagged<float> {
  unsigned long long x;
  __device__ __forceinline__ void load(const unsigned long long* p) {
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(x) : "l"(p) : "memory");
  }
  __device__ __forceinline__ bool ok(unsigned tag) const { return (unsigned) (x >> 32) == tag; }
  __device__ __forceinline__ float value() const { return __uint_as_float((unsigned) x); }
  __device__ __forceinline__ static void put(unsigned long long* p, unsigned tag, float v) {
    const unsigned long long w = ((unsigned long long) tag << 32) | __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
  }
};
template <>
struct Tagged<double> {
  unsigned long long x, y;   // high and low half of the value
  __device__ __forceinline__ void load(const unsigned long long* p) {
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "l"(p) : "memory");
  }
  __device__ __forceinline__ bool ok(unsigned tag) const {
    return (unsigned) (x >> 32) == tag && (unsigned) (y >> 32) == tag;
  }
  __device__ __forceinline__ double value() const { return __hiloint2double((int) (unsigned) x, (int) (unsigned) y); }
  __device__ __forceinline__ static void put(unsigned long long* p, unsigned tag, double v) {
    const unsigned long long t = (unsigned long long) tag << 32;
    const unsigned long long a = t | (unsigned) __double2hiint(v), b = t | (unsigned) __double2loint(v);
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
  }
};

// waits (bounded) until the lanes' values all carry the tag, reloading them;
// called by whole warps and left together; lanes with need = false take part
// without a value
template <typename T>
__device__ __forceinline__ void wait_tagged(const unsigned long long* p, Tagged<T>& v, bool need, unsigned tag,
                                            int* status) {
  const int limit = g_solve_wait_limit;
  const unsigned want = tag + (unsigned) (g_solve_wait_skew << 12);
  int it = 0;
  while (!__all_sync(0xffffffffu, !need || v.ok(want))) {
    ++it;
    if (__any_sync(0xffffffffu, it > limit || ((it & 1023) == 0 && *(volatile int*) status == SOLVE_TIMEOUT))) {
      atomicExch(status, SOLVE_TIMEOUT);
      break;
    }
    if (it > 4) __nanosleep(20);
    if (need) v.load(p);
  }
}

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned) __cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned map_rank(unsigned addr, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// QL values of a lane into another CTA's shared memory, counted there
__device__ __forceinline__ void st_async(unsigned addr, unsigned bar, const float (&v)[1]) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr),
               "r"(__float_as_uint(v[0])), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void st_async(unsigned addr, unsigned bar, const float (&v)[2]) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(addr),
               "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void st_async(unsigned addr, unsigned bar, const double (&v)[1]) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
               "l"(__double_as_longlong(v[0])), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void st_async(unsigned addr, unsigned bar, const double (&v)[2]) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(addr),
               "l"(__double_as_longlong(v[0])), "l"(__double_as_longlong(v[1])), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait of a whole warp for a phase of a z's barrier; false when it gave
// up.  Neither the polling limit above nor the status word ends it: every z is
// sent, also after other waits ran out (their values are then wrong, and the
// status says so), and a CTA that did not wait for one would leave with stores
// to its shared memory still on their way.  Its own limit, some 30 seconds, is
// far above what the waits of the CTAs that it depends on can add up to.
constexpr int BAR_SPIN = 4096;          // before the warp sleeps between its tries
constexpr int BAR_LIMIT = 1 << 25;
__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned parity, int* status) {
  for (int it = 0; !__all_sync(0xffffffffu, bar_try(bar, parity)); it++) {
    if (it < BAR_SPIN) continue;
    if (it > BAR_LIMIT) {
      atomicExch(status, SOLVE_TIMEOUT);
      return false;
    }
    __nanosleep(1000);
  }
  return true;
}
// about a millisecond, for stores from other CTAs that nothing counts any more
__device__ __forceinline__ void settle() {
  const long long t0 = clock64();
  for (int it = 0; it < (1 << 16) && clock64() - t0 < (1 << 21); it++) __nanosleep(1000);
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// (a, b) += l (x, y): two FP32 multiply-adds in one packed instruction
__device__ __forceinline__ void fma2(float& a, float& b, float l, float x, float y) {
  asm("{\n\t.reg .b64 p, q, r;\n\t"
      "mov.b64 p, {%2, %2};\n\tmov.b64 q, {%3, %4};\n\tmov.b64 r, {%0, %1};\n\t"
      "fma.rn.f32x2 r, p, q, r;\n\tmov.b64 {%0, %1}, r;\n\t}"
      : "+f"(a), "+f"(b)
      : "f"(l), "f"(x), "f"(y));
}
// A 64-row product by the CTA's eight warps, warp w the rows 8 w .. 8 w + 7.
// Its cost is the bytes of z that the lanes take from shared memory (128 a
// clock), so with several right-hand sides a lane covers R = 2 rows: lane
// (i, j), j < J = 4 R, holds rows 8 w + i + (8 / R) h, h < R, and columns J t +
// j -- a warp's loads cover whole sectors, its reads of z ([column][right-hand
// side]) are neighbouring rows -- and the row's lanes are summed by shuffles.
// FP64 with eight columns runs on DMMA m8n8k4 instead: its A fragment is the
// R = 1 layout, its B fragment one value of z a lane, and its C fragment
// leaves each lane with two columns of its row, with nothing to sum.
// Afterwards a lane owns QL right-hand sides qb .. of row `own` (qact: of
// several lanes with the same values only one).
template <typename T, int NQ>
struct ChainRow {
  static constexpr bool DMMA = sizeof(T) == 8 && NQ == 8;
  static constexpr int R = NQ == 1 || DMMA ? 1 : 2, J = 4 * R, NT = 16 / R;
  static constexpr int NACC = DMMA ? 2 : R * NQ, QL = NQ >= 4 ? NQ / 4 : 1;
  static_assert(NQ == 1 || NQ == 4 || NQ == 8, "the solve's instantiations");
  T acc[NACC];
  __device__ __forceinline__ static int lane() { return threadIdx.x & 31; }
  __device__ __forceinline__ static int jq() { return lane() % J; }
  __device__ __forceinline__ static int row(int h) { return (threadIdx.x >> 5) * 8 + lane() / J + (8 / R) * h; }
  __device__ __forceinline__ static int own() { return row(R == 2 ? jq() >> 2 : 0); }
  __device__ __forceinline__ static int qb() { return NQ >= 4 ? QL * (jq() & 3) : 0; }
  __device__ __forceinline__ static bool qact() { return NQ >= 4 || jq() == 0; }
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int a = 0; a < NACC; a++) acc[a] = T(0);
  }
  // acc += l z, l[h * NT + t] the entry of row(h), column J t + j
  __device__ __forceinline__ void add(const T (&l)[16], const T* z) {
    const int j = jq();
    if constexpr (DMMA) {
#pragma unroll
      for (int t = 0; t < 16; t++) {
        const double b = z[(4 * t + j) * NQ + (lane() >> 2)];
        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                     : "+d"(acc[0]), "+d"(acc[1])
                     : "d"(l[t]), "d"(b));
      }
    } else {
#pragma unroll
      for (int t = 0; t < NT; t++) {
        const T* zr = z + (J * t + j) * NQ;
        T x[NQ];
        if constexpr (NQ * sizeof(T) >= 16) {
          constexpr int V = 16 / (int) sizeof(T);
          struct alignas(16) Vec { T v[V]; };
#pragma unroll
          for (int q = 0; q < NQ; q += V) {
            const Vec y = *reinterpret_cast<const Vec*>(zr + q);
#pragma unroll
            for (int c = 0; c < V; c++) x[q + c] = y.v[c];
          }
        } else {
#pragma unroll
          for (int q = 0; q < NQ; q++) x[q] = zr[q];
        }
#pragma unroll
        for (int h = 0; h < R; h++) {
          if constexpr (std::is_same<T, float>::value && NQ % 2 == 0) {
#pragma unroll
            for (int q = 0; q < NQ; q += 2) fma2(acc[h * NQ + q], acc[h * NQ + q + 1], l[h * NT + t], x[q], x[q + 1]);
          } else {
#pragma unroll
            for (int q = 0; q < NQ; q++) acc[h * NQ + q] += l[h * NT + t] * x[q];
          }
        }
      }
    }
  }
  // the sums over the row's lanes that this lane owns
  __device__ __forceinline__ void sum(T (&out)[QL]) const {
    constexpr unsigned FULL = 0xffffffffu;
    if constexpr (DMMA) {
      out[0] = acc[0];
      out[1] = acc[1];
    } else if constexpr (NQ == 1) {
      T v = acc[0];
      v += __shfl_xor_sync(FULL, v, 2);
      out[0] = v + __shfl_xor_sync(FULL, v, 1);
    } else {
      // at each offset a lane keeps one half of its sums and adds its
      // partner's copy of it: first by row (offset 4), then by column
      T v[NACC];
#pragma unroll
      for (int a = 0; a < NACC; a++) v[a] = acc[a];
#pragma unroll
      for (int o = J / 2, h = NACC / 2; o >= 1; o >>= 1, h >>= 1) {
        const bool up = (threadIdx.x & o) != 0;
#pragma unroll
        for (int a = 0; a < h; a++) v[a] = (up ? v[a + h] : v[a]) + __shfl_xor_sync(FULL, up ? v[a] : v[a + h], o);
      }
#pragma unroll
      for (int q = 0; q < QL; q++) out[q] = v[q];
    }
  }
};

// Backward solve, L21^T x2 over a 64-column block and a chunk of 512 update
// rows by a CTA of NTH threads.  The chunk of x2 is gathered into shared
// memory once ([column][row], conflict-free across lanes).  A warp takes G = 32
// / NQ columns (16 with one right-hand side) over one of RP row parts, 16
// loads of the panel in flight a lane, so that the G x NQ sums of a pass
// finish with one warp reduce-scatter (31 shuffles; lane t ends with sum t =
// column t / NQ, right-hand side t % NQ).  A round of loads is a memory
// latency, which is what bounds a small launch: 4 warps take 16 rounds for a
// chunk (40 us, FP64, one right-hand side, from 72 to 394 CTAs), 16 warps 4.
// sink(column, right-hand side, row part, sum) takes the sums.
template <int NQ, int NTH>
struct L21Split {
  static constexpr int G = NQ >= 2 ? 32 / NQ : 16, SUMS = G * NQ, NW = NTH / 32;
  static constexpr int CG = BR / G;                        // column groups
  static constexpr int RP = NW >= CG ? NW / CG : 1;        // row parts
  static_assert((SUMS == 32 || SUMS == 16) && G <= 16, "a pass holds 32 (one right-hand side: 16) sums");
};
template <typename T, int NQ, int NTH, typename Sink>
__device__ __forceinline__ void l21_chunk(const FrontDesc& F, const T* __restrict__ L, const int* __restrict__ rows,
                                          const T* X, int ldx, int k, int ch, int nrhs, T (*zs)[SOLVE_RCH],
                                          Sink sink) {
  using S = L21Split<NQ, NTH>;
  constexpr int G = S::G, SUMS = S::SUMS, RP = S::RP;
  const int f = F.f, s = F.s, m = f - s;
  const int c0 = k * BR, bw = min(BR, s - c0);
  const int i0 = ch * SOLVE_RCH, nr = min(m - i0, SOLVE_RCH);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const T* P = L + F.l_off + s + i0;
  // all of this thread's loads in flight before its first store
  {
    constexpr int NI = SOLVE_RCH / NTH;
    const int* rw = rows + F.rows_off + s + i0;
    int g[NI];
    T zv[NQ][NI];
#pragma unroll
    for (int t = 0; t < NI; t++) g[t] = (int) threadIdx.x + NTH * t < nr ? __ldg(rw + threadIdx.x + NTH * t) : -1;
#pragma unroll
    for (int q = 0; q < NQ; q++)
#pragma unroll
      for (int t = 0; t < NI; t++) zv[q][t] = (g[t] >= 0 && q < nrhs) ? __ldcg(X + g[t] + (size_t) q * ldx) : T(0);
#pragma unroll
    for (int q = 0; q < NQ; q++)
#pragma unroll
      for (int t = 0; t < NI; t++) zs[q][threadIdx.x + NTH * t] = zv[q][t];
  }
  __syncthreads();
  const int part = warp / S::CG % RP;
  for (int cg = warp % S::CG * G; cg < bw; cg += S::NW >= S::CG ? BR : S::NW * G) {
    T v[SUMS];   // v[a * NQ + q]: column cg + a, right-hand side q
#pragma unroll
    for (int j = 0; j < SUMS; j++) v[j] = T(0);
    constexpr int RU = G >= 16 ? 1 : 16 / G;   // rows per lane per round
    for (int i1 = lane + 32 * RU * part; i1 < nr; i1 += 32 * RU * RP) {
      T lv[RU][G];
#pragma unroll
      for (int u = 0; u < RU; u++)
#pragma unroll
        for (int a = 0; a < G; a++) {
          const int i = i1 + 32 * u;
          lv[u][a] = (i < nr && cg + a < bw) ? P[i + (size_t) (c0 + cg + a) * f] : T(0);
        }
#pragma unroll
      for (int u = 0; u < RU; u++) {
        const int i = i1 + 32 * u;
        if (i < nr) {
          T zi[NQ];
#pragma unroll
          for (int q = 0; q < NQ; q++) zi[q] = zs[q][i];
#pragma unroll
          for (int a = 0; a < G; a++)
#pragma unroll
            for (int q = 0; q < NQ; q++) v[a * NQ + q] += lv[u][a] * zi[q];
        }
      }
    }
    // reduce-scatter: at offset o a lane keeps the half of its remaining
    // sums that matches its bit o and adds the partner's copy of that half
#pragma unroll
    for (int o = 16, h = SUMS / 2; o >= 1; o >>= 1, h >>= 1) {
      if (h == 0) {   // 16 sums: the last pair of lanes holds the same one
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        continue;
      }
      const bool up = (lane & o) != 0;
#pragma unroll
      for (int j = 0; j < h; j++) {
        const T send = up ? v[j] : v[j + h];
        const T keep = up ? v[j + h] : v[j];
        v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
    const int t = SUMS == 32 ? lane : lane >> 1;
    const int a = t / NQ, q = t % NQ;
    if (cg + a < bw && q < nrhs && (SUMS == 32 || (lane & 1) == 0)) sink(cg + a, q, part, v[0]);
  }
}

// the sums of (column block, 512-row chunk) tasks, so that the whole GPU
// streams L21; the chain and block kernels add them in chunk order
template <typename T, int NQ, int NTH>
__global__ void __launch_bounds__(NTH)
k_bwd_l21(const int2_* __restrict__ tasks, const FrontDesc* __restrict__ fronts, const int* __restrict__ rows,
          const T* __restrict__ L, const T* X, int ldx, T* __restrict__ part, int nrhs) {
  constexpr int RP = L21Split<NQ, NTH>::RP;
  __shared__ T zs[NQ][SOLVE_RCH];
  __shared__ T red[RP][BR][NQ];
  const int2_ tk = tasks[blockIdx.x];
  const FrontDesc F = fronts[tk.a];
  const int k = tk.b >> 16, ch = tk.b & 0xffff;
  grid_wait();
  l21_chunk<T, NQ, NTH>(F, L, rows, X, ldx, k, ch, nrhs, zs, [&](int c, int q, int p, T v) { red[p][c][q] = v; });
  __syncthreads();
  T* out = part + F.part_off + ((size_t) ch * F.s + k * BR) * SOLVE_NRHS;
  const int bw = min(BR, F.s - k * BR);
  for (int e = threadIdx.x; e < bw * NQ; e += NTH) {
    const int c = e / NQ, q = e % NQ;
    T v = red[0][c][q];
#pragma unroll
    for (int p = 1; p < RP; p++) v += red[p][c][q];
    if (q < nrhs) out[c * SOLVE_NRHS + q] = v;
  }
}

// What the kernels of the big fronts' blocks share.  zp, pp: published z's and
// p's; forward reads B and writes W, backward reads W (y) and, for fronts of at
// least part_min chunks of update rows, the sums in part (L21^T x2; the other
// fronts form it themselves), and writes X.
template <typename T>
struct SolveArgs {
  const int* walk_fronts;
  int nwalk;
  const int2_* blocks;
  int nblocks;
  const int2_* blk_ch;
  const int4* blk_child;
  const FrontDesc* fronts;
  const int *maps, *rows;
  const T *L, *Dinv, *B;
  T* X;
  int ldx;
  T* W;
  const T* part;
  int part_min;
  unsigned long long *zp, *pp;
  int* flags;
  int nrhs;
  const int* counter;
  int epoch;
  int* status;
};

// a load of the factor that is issued where it stands (a plain read-only load
// may be moved down to its use, past the wait that it is meant to overlap);
// zero, and no access, without in
__device__ __forceinline__ double load_now(const double* p, bool in) {
  double v;
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.f64 %0, 0d0000000000000000;\n\t"
               "@q ld.global.nc.f64 %0, [%1];\n\t}"
               : "=d"(v)
               : "l"(p), "r"((unsigned) in));
  return v;
}
__device__ __forceinline__ float load_now(const float* p, bool in) {
  float v;
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.f32 %0, 0f00000000;\n\t"
               "@q ld.global.nc.f32 %0, [%1];\n\t}"
               : "=f"(v)
               : "l"(p), "r"((unsigned) in));
  return v;
}

// One front's 64-row blocks as the kernels below work on them.  Chain
// position t <-> block (backward: the last block first).  TAGS: the z's between
// CTAs are published values; else (the allocation-free solve, which has no
// room for them) they are in the work vector behind release/acquire flags.
template <typename T, int NQ, int WS, bool BWD, bool TAGS>
struct BigBlock {
  using Row = ChainRow<T, NQ>;
  static constexpr int QL = Row::QL, WPV = ch_words<T>();
  const SolveArgs<T>& A;
  const FrontDesc F;
  const int f, s, nbs;
  const T* const P;
  T* const Wf;
  const int* const rw;
  unsigned long long* const zf;
  unsigned tag = 0;
  __device__ __forceinline__ BigBlock(const SolveArgs<T>& a, int front)
      : A(a), F(a.fronts[front]), f(F.f), s(F.s), nbs((F.s + BR - 1) / BR), P(a.L + F.l_off), Wf(a.W + F.v_off * WS),
        rw(a.rows + F.rows_off), zf(a.zp + (size_t) F.blk_off * CH_VALUES * WPV) {}
  // the launches before this one have finished (a solve's first one waited for
  // the factorization: L and the inverses may be read ahead of this)
  __device__ __forceinline__ void begin() {
    grid_wait();
    if (TAGS) tag = ((unsigned) *(volatile const int*) A.counter << 12) | (unsigned) A.epoch;
  }
  __device__ __forceinline__ int block_of(int t) const { return BWD ? nbs - 1 - t : t; }
  // this lane's 16 entries of A_tu (block row bt: rows below s may belong to
  // the update rows of the last diagonal block, or be an update block)
  __device__ __forceinline__ void tile(int bt, int bu, T (&l)[16]) const {
    const int jq = Row::jq();
#pragma unroll
    for (int h = 0; h < Row::R; h++) {
      const int r = bt * BR + Row::row(h), c = bu * BR + jq;
      const bool rv = r < (BWD ? s : f);
      const T* a = BWD ? P + c + (size_t) r * f : P + r + (size_t) c * f;
#pragma unroll
      for (int t = 0; t < Row::NT; t++)
        l[h * Row::NT + t] = load_now(a + (BWD ? Row::J * t : (size_t) (Row::J * t) * f), rv && c + Row::J * t < s);
    }
  }
  // the inverse of diagonal block b on its way into ds (column stride DLD:
  // the products' reads are free of bank conflicts)
  __device__ __forceinline__ void stage_inverse(int b, T* ds) const {
    const T* Di = A.Dinv + F.dinv_off + (size_t) b * BR * BR;
    constexpr int V = 16 / (int) sizeof(T), PER = BR / V;
#pragma unroll
    for (int e = threadIdx.x; e < BR * PER; e += CH_THREADS) {
      const int c = e / PER, r = e % PER * V;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(ds + c * DLD + r)), "l"(Di + c * BR + r));
    }
  }
  // the right-hand side of block b into vs, with a barrier after it; scr:
  // scratch (backward: a chunk of x2 and its sums, with SUMS)
  template <bool SUMS>
  __device__ __forceinline__ void own_rhs(int b, const int2_ cr, T (*vs)[NQ], T* scr) const {
    const int tid = threadIdx.x, r0 = b * BR, nr = min(BR, f - r0);
    if constexpr (!BWD) {
      ChildGather<T, NQ, WS, CH_THREADS> cg;
      cg.load(A.blk_child + cr.a, cr.b - cr.a, A.maps, A.W, A.nrhs);
      for (int e = tid; e < BR * NQ; e += CH_THREADS) {
        const int i = e % BR, q = e / BR;
        vs[i][q] = (i < nr && q < A.nrhs && r0 + i < s) ? A.B[rw[r0 + i] + (size_t) q * A.ldx] : T(0);
      }
      __syncthreads();
      cg.add(A.blk_child + cr.a, cr.b - cr.a, A.maps, A.W, A.nrhs, r0, vs);
    } else {
      const bool parts = !SUMS || F.nchunk >= A.part_min;
      for (int e = tid; e < BR * NQ; e += CH_THREADS) {
        const int i = e % BR, q = e / BR;
        T v = T(0);
        if (r0 + i < s && q < A.nrhs) {
          v = Wf[r0 + i + (size_t) q * f];
          T acc = T(0);
          if (parts) {
#pragma unroll 4
            for (int ch = 0; ch < F.nchunk; ch++)
              acc += A.part[F.part_off + ((size_t) ch * s + r0 + i) * SOLVE_NRHS + q];
          }
          v -= acc;
        }
        vs[i][q] = v;
      }
      if (SUMS && !parts) {
        constexpr int RP = L21Split<NQ, CH_THREADS>::RP;
        T (*zs)[SOLVE_RCH] = reinterpret_cast<T (*)[SOLVE_RCH]>(scr);
        T (*red)[BR][NQ] = reinterpret_cast<T (*)[BR][NQ]>(scr + NQ * SOLVE_RCH);
        const int nch = (f - s + SOLVE_RCH - 1) / SOLVE_RCH, bw = min(BR, s - r0);
        for (int ch = 0; ch < nch; ch++) {
          l21_chunk<T, NQ, CH_THREADS>(F, A.L, A.rows, A.X, A.ldx, b, ch, A.nrhs, zs,
                                       [&](int c, int q, int p, T v) { red[p][c][q] = v; });
          __syncthreads();
          for (int e = tid; e < bw * NQ; e += CH_THREADS) {
            const int c = e / NQ, q = e % NQ;
            T v = red[0][c][q];
#pragma unroll
            for (int p = 1; p < RP; p++) v += red[p][c][q];
            if (q < A.nrhs) vs[c][q] -= v;
          }
        }
      }
      __syncthreads();
    }
  }
  // acc += sum_{u<n} A_bu z_u as the z's appear.  A round takes up to HB blocks
  // with every load in flight: the leading blocks whose values are all current
  // are used, or the first is waited for.  l: the first round's tiles, already
  // loaded.  zst: HB staged z's.
  template <int HB>
  __device__ __forceinline__ void terms(int b, int n, T (&l)[HB][16], Row& acc, T* zst, unsigned* bad_s) const {
    const int tid = threadIdx.x;
    constexpr int NV = (HB * BR * NQ + CH_THREADS - 1) / CH_THREADS;
    for (int u = 0; u < n;) {
      int ok = min(n - u, HB);
      if constexpr (TAGS) {
        const int nb = ok;
        if (HB > 1 && tid == 0) *bad_s = 0;
        if (HB > 1) __syncthreads();
        Tagged<T> zv[NV];
        auto src = [&](int e) {
          return zf + ((size_t) block_of(u + e / (BR * NQ)) * CH_VALUES + e % (BR * NQ)) * WPV;
        };
#pragma unroll
        for (int i = 0; i < NV; i++) {
          const int e = tid + CH_THREADS * i;
          if (e < nb * BR * NQ) zv[i].load(src(e));
        }
        if constexpr (HB > 1) {
          unsigned bad = 0;
#pragma unroll
          for (int i = 0; i < NV; i++) {
            const int e = tid + CH_THREADS * i;
            if (e < nb * BR * NQ && !zv[i].ok(tag)) bad |= 1u << (e / (BR * NQ));
          }
          if (bad) atomicOr(bad_s, bad);
          __syncthreads();
          ok = __ffs(*bad_s | (1u << nb)) - 1;
        } else {
          ok = 0;
        }
        if (ok == 0) {
#pragma unroll
          for (int i = 0; i < NV; i++) {
            const int e = tid + CH_THREADS * i;
            if (CH_THREADS * i < BR * NQ) wait_tagged<T>(src(e < BR * NQ ? e : 0), zv[i], e < BR * NQ, tag, A.status);
          }
          ok = 1;
        }
#pragma unroll
        for (int i = 0; i < NV; i++) {
          const int e = tid + CH_THREADS * i;
          if (e < ok * BR * NQ) zst[e] = zv[i].value();
        }
      } else {
        ok = 1;
        const int bu = block_of(u);
        wait_epoch(A.flags + F.blk_off + bu, A.epoch, A.status);
        for (int e = tid; e < BR * NQ; e += CH_THREADS) {
          const int i = e / NQ, q = e % NQ;
          zst[e] = (bu * BR + i < s && q < A.nrhs) ? __ldcg(Wf + bu * BR + i + (size_t) q * f) : T(0);
        }
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < HB; i++)
        if (i < ok) acc.add(l[i], zst + i * BR * NQ);
      u += ok;
#pragma unroll
      for (int i = 0; i < HB; i++)
        if (u + i < n) tile(b, block_of(u + i), l[i]);
      __syncthreads();
    }
  }
  // this lane's 16 entries of the staged inverse, once it is complete
  __device__ __forceinline__ static void inverse(const T* ds, T (&d)[16]) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int h = 0; h < Row::R; h++)
#pragma unroll
      for (int i = 0; i < Row::NT; i++) {
        const int r = Row::row(h), c = Row::J * i + Row::jq();
        d[h * Row::NT + i] = ds[BWD ? c + r * DLD : r + c * DLD];
      }
  }
  // z = D v, v (this lane's share pv) in rows of vs; in the last diagonal block
  // the update rows get w_i - L[i, block] y (forward)
  __device__ __forceinline__ void diagonal(int b, const T (&d)[16], const T (&pv)[QL], T (*vs)[NQ], T (&z)[QL]) const {
    const int rho = Row::own(), qb = Row::qb();
    const int r0 = b * BR, nr = min(BR, f - r0), bw = min(BR, s - r0);
    if (Row::qact())
#pragma unroll
      for (int q = 0; q < QL; q++) vs[rho][qb + q] = pv[q];
    __syncthreads();
    Row acc;
    acc.clear();
    acc.add(d, &vs[0][0]);
    acc.sum(z);
    if (!BWD && bw < nr) {
      // the inverse is zero in the update rows: y is in place first
      __syncthreads();
      if (Row::qact() && rho < bw)
#pragma unroll
        for (int q = 0; q < QL; q++) vs[rho][qb + q] = z[q];
      __syncthreads();
      T l[16], uq[QL];
      tile(b, b, l);
      acc.clear();
      acc.add(l, &vs[0][0]);
      acc.sum(uq);
      if (rho >= bw)
#pragma unroll
        for (int q = 0; q < QL; q++) z[q] = pv[q] - uq[q];
    }
  }
  // the result of block b: forward into the work vector, backward into X
  __device__ __forceinline__ void result(int b, const T (&z)[QL]) const {
    const int r = b * BR + Row::own(), qb = Row::qb();
    if (!Row::qact() || r >= (BWD ? s : f)) return;
    if (!BWD || !TAGS) {
#pragma unroll
      for (int q = 0; q < QL; q++)
        if (qb + q < A.nrhs) Wf[r + (size_t) (qb + q) * f] = z[q];
    }
    if (BWD) {
      const int g = __ldg(rw + r);
#pragma unroll
      for (int q = 0; q < QL; q++)
        if (qb + q < A.nrhs) A.X[g + (size_t) (qb + q) * A.ldx] = z[q];
    }
  }
  // a published value array's slot of this lane in block b
  __device__ __forceinline__ unsigned long long* slot(unsigned long long* base, int b) const {
    return base + ((size_t) b * CH_VALUES + Row::own() * NQ + Row::qb()) * WPV;
  }
  __device__ __forceinline__ void publish(unsigned long long* base, int b, const T (&z)[QL]) const {
    if (!Row::qact()) return;
    unsigned long long* dst = slot(base, b);
#pragma unroll
    for (int q = 0; q < QL; q++) Tagged<T>::put(dst + q * WPV, tag, z[q]);
  }
};

// elements of the scratch of own_rhs and terms
template <int NQ, bool BWD, int HB>
__host__ __device__ constexpr int block_scratch() {
  const int rhs = BWD ? NQ * SOLVE_RCH + L21Split<NQ, CH_THREADS>::RP * BR * NQ : 0, z = HB * BR * NQ;
  return rhs > z ? rhs : z;
}

// Forward and backward solve of a level's big fronts as chains, for levels
// with few fronts and several 64-row blocks each.  What bounds such a level
// is the chain of its blocks -- z_t = D_t (p_t - sum_{u<t} A_tu z_u), D_t the
// inverse of a diagonal block (forward: blocks first to last; backward: last
// to first, transposed) -- so the chain runs inside one cluster of CH_C CTAs:
// CTA t mod CH_C computes block t and writes z_t into the shared memory of
// all of them (st.async, counted by the receivers' mbarriers), one to two
// orders faster than a hand-over through global memory.  Between its turns a
// CTA adds the terms of the last CH_C blocks to its next one as they arrive,
// with the tiles of L loaded into registers two terms ahead and into L2 a
// turn ahead: per step the chain waits for one 64x64 product, one product
// with the inverse and one hand-over.  The far terms (u < t - CH_C) and the
// right-hand side of block t are the work of a helper CTA per block, which
// follows the published z_u and publishes p_t about CH_C steps ahead;
// forward, the update rows' blocks are helpers too and stream L21 while the
// chain runs.  Values published between CTAs travel as tagged words (tag in
// the high half, 32 bits of the value in the low half; a double takes two),
// each one relaxed 8-byte access: a reader knows a value is current when its
// tag is, so nothing fences or polls a flag.  The tag is (call counter <<
// 12) | epoch, the counter being advanced on the device at the start of every
// solve call, so recorded launch sequences stay valid.  No stale word can carry
// a pass's tag: forward epochs are odd and backward ones even, in bit 0 also
// when an epoch outgrows its 12 bits or the counter wraps; a pass writes every
// word that it reads, in both directions; so its forward step finds even tags
// everywhere, and its backward step nothing but its own forward tags.  A ring
// of 2 CH_C z's needs no release: block t's CTA has consumed z_{t-CH_C} ..
// z_{t-1}, so when z_{u+2 CH_C} is produced every CTA is past its last use of
// z_u.  Walkers have the lowest CTA indices and helper t waits only for blocks
// whose helpers come before it, so in-order dispatch keeps every wait finite;
// the waits are bounded all the same.  No CTA of a cluster leaves before every
// z has arrived in its shared memory, also when the waits for published values
// give up: the walkers carry on with what they have and send every z.  In the
// last diagonal block rows >= s are update rows of the same front; its CTA
// finishes them too (forward).
// Measured, per 64-row step of the root level's forward chain: FP64, one right-
// hand side (64^3) 2.3 us with flags between CTAs, 1.2 us here; FP64, eight
// (45x47x44) 4.7 -> 1.7 us; FP32, eight (56^3) 4.2 us with one walker CTA per
// front, 2.0 us here.
// dynamic shared memory: the block's inverse, the ring of z's (walker) or a
// round's staged z's and x2 (helper), and the block's vector
template <typename T, int NQ>
constexpr size_t chain_smem() { return (size_t) (BR * DLD + (CH_RING + 1) * BR * NQ) * sizeof(T); }

template <typename T, int NQ, int WS, bool BWD>
__global__ void __cluster_dims__(CH_C, 1, 1) __launch_bounds__(CH_THREADS, 2)
k_chain(const __grid_constant__ SolveArgs<T> A) {
  using BB = BigBlock<T, NQ, WS, BWD, true>;
  using Row = ChainRow<T, NQ>;
  constexpr int QL = Row::QL, WPV = ch_words<T>();
  extern __shared__ __align__(16) unsigned char chm[];
  __shared__ __align__(8) unsigned long long bars[CH_RING];
  __shared__ unsigned bad_s;
  const int tid = threadIdx.x;
  const int rho = Row::own(), qb = Row::qb();
  const bool walker = blockIdx.x < (unsigned) (A.nwalk * CH_C);
  const int h = (int) blockIdx.x - A.nwalk * CH_C;
  if (!walker && h >= A.nblocks) return;
  const int2_ bk = walker ? int2_{A.walk_fronts[blockIdx.x / CH_C], 0} : A.blocks[h];
  BB M(A, bk.a);
  const int f = M.f, s = M.s, nbs = M.nbs;
  unsigned long long* pf = A.pp + (size_t) M.F.blk_off * CH_VALUES * WPV;
  T* ds = reinterpret_cast<T*>(chm);
  T* zs = ds + BR * DLD;                          // [CH_RING][BR][NQ]
  T (*vs)[NQ] = reinterpret_cast<T (*)[NQ]>(zs + CH_RING * BR * NQ);

  if (walker) {
    // ---------------------------------------------------------------- walker
    const unsigned rank = blockIdx.x % CH_C;
    constexpr unsigned ZBYTES = BR * NQ * sizeof(T);
    if (tid == 0) {
      for (int i = 0; i < CH_RING; i++)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&bars[i])) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      for (int i = 0; i < min(CH_RING, nbs); i++) bar_expect(smem_addr(&bars[i]), ZBYTES);
    }
    __syncthreads();
    cluster_sync_all();
    // z_u has arrived (each CTA waits for every u once, in order); its
    // barrier is armed for the z that takes the slot next.  A warp whose wait
    // gave up waits, arms and sends no more: its z's stay incomplete, so that
    // no slot is written, and no barrier armed, a second time within a phase
    bool alive = true;
    auto wait_z = [&](int u) {
      if (alive) alive = bar_wait(smem_addr(&bars[u % CH_RING]), (u / CH_RING) & 1, A.status);
      if (tid == 0 && alive && u + CH_RING < nbs) bar_expect(smem_addr(&bars[u % CH_RING]), ZBYTES);
    };
    if ((int) rank >= nbs) {
      M.begin();
      grid_trigger();
    }
    unsigned peer[CH_C];   // offsets of the others' shared memory, the next CTA of the chain first
#pragma unroll
    for (int r = 0; r < CH_C; r++) peer[r] = map_rank(smem_addr(bars), (rank + 1 + r) % CH_C) - smem_addr(bars);
    for (int t = rank; t < nbs; t += CH_C) {
      const int b = M.block_of(t);
      const int u0 = max(0, t - CH_C);
      T la[16], lb[16], d[16];
      if (u0 < t) M.tile(b, M.block_of(u0), la);
      if (u0 + 1 < t) M.tile(b, M.block_of(u0 + 1), lb);
      __syncthreads();   // every warp is done with the last turn's inverse
      M.stage_inverse(b, ds);
      // the next turn's tiles into L2
      if (t + CH_C < nbs) {
        const int bn = M.block_of(t + CH_C);
        constexpr int LPC = BR * (int) sizeof(T) / 128 + 1;   // lines a 64-entry column piece touches
        for (int e = tid; e < CH_C * BR * LPC; e += CH_THREADS) {
          const int li = e % LPC, c = e / LPC;
          const int bu = M.block_of(t + c / BR);
          const int row = (BWD ? bu : bn) * BR + min(li * (128 / (int) sizeof(T)), BR - 1);
          const int col = (BWD ? bn : bu) * BR + c % BR;
          if (row < f && col < s) prefetch_l2(M.P + row + (size_t) col * f);
        }
        for (int e = tid; e < BR * BR * (int) sizeof(T) / 128; e += CH_THREADS)
          prefetch_l2(reinterpret_cast<const unsigned char*>(A.Dinv + M.F.dinv_off + (size_t) bn * BR * BR) + 128 * e);
      }
      if (t == (int) rank) M.begin();
      if (t + CH_C >= nbs) grid_trigger();
      Row acc;
      acc.clear();
      Tagged<T> pt[QL];
      const unsigned long long* pq = M.slot(pf, b);
      auto load_p = [&]() {
#pragma unroll
        for (int q = 0; q < QL; q++) pt[q].load(pq + q * WPV);
      };
      if (t == 0) {
        load_p();
        M.inverse(ds, d);
      }
      for (int u = u0; u < t; u += 2) {
        if (u + 2 >= t) {   // ahead of the waits that are on the chain
          load_p();
          M.inverse(ds, d);
        }
        wait_z(u);
        acc.add(la, zs + (u % CH_RING) * BR * NQ);
        if (u + 2 < t) M.tile(b, M.block_of(u + 2), la);
        if (u + 1 < t) {
          wait_z(u + 1);
          acc.add(lb, zs + ((u + 1) % CH_RING) * BR * NQ);
          if (u + 3 < t) M.tile(b, M.block_of(u + 3), lb);
        }
      }
      T z[QL], pv[QL];
      acc.sum(z);
#pragma unroll
      for (int q = 0; q < QL; q++) {
        wait_tagged<T>(pq + q * WPV, pt[q], true, M.tag, A.status);
        pv[q] = pt[q].value() - z[q];
      }
      M.diagonal(b, d, pv, vs, z);
      // z_t: into every CTA of the cluster, the next of the chain first, then
      // published for the helpers, then the result
      if (alive && Row::qact()) {
        const unsigned za = smem_addr(zs + ((t % CH_RING) * BR + rho) * NQ + qb), ba = smem_addr(&bars[t % CH_RING]);
#pragma unroll
        for (int r = 0; r < CH_C; r++) st_async(za + peer[r], ba + peer[r], z);
      }
      M.publish(M.zf, b, z);
      M.result(b, z);
    }
    // every z that is still on its way to this CTA's shared memory
    for (int u = (int) rank < nbs ? (int) rank + (nbs - 1 - (int) rank) / CH_C * CH_C : 0; u < nbs; u++) wait_z(u);
    cluster_sync_all();
    // (a z that was cut short completes no phase: what was sent of it)
    if (!alive) settle();
    return;
  }
  // ------------------------------------------------------------------ helper
  const bool upd = !BWD && bk.b >= nbs;                  // an update-row block
  const int b = bk.b, n = upd ? nbs : max(0, (BWD ? nbs - 1 - b : b) - CH_C);
  T l[CH_HB][16];
#pragma unroll
  for (int i = 0; i < CH_HB; i++)
    if (i < n) M.tile(b, M.block_of(i), l[i]);
  M.begin();
  M.template own_rhs<false>(b, BWD ? int2_{0, 0} : A.blk_ch[h], vs, zs);
  Row acc;
  acc.clear();
  M.template terms<CH_HB>(b, n, l, acc, zs, &bad_s);
  grid_trigger();
  T p[QL];
  acc.sum(p);
#pragma unroll
  for (int q = 0; q < QL; q++) p[q] = vs[rho][qb + q] - p[q];
  if (upd) M.result(b, p);
  else M.publish(pf, b, p);
}

// The big fronts of the other levels: one CTA per 64-row block, which adds the
// terms of the blocks before it as they are published, applies its inverse and
// publishes its own result (forward, blocks of update rows stop at the terms).
// Blocks wait only for blocks of lower index.
constexpr int BLK_HB = 1;
template <typename T, int NQ, bool BWD>
constexpr size_t block_smem() { return (size_t) (BR * DLD + block_scratch<NQ, BWD, BLK_HB>() + BR * NQ) * sizeof(T); }

template <typename T, int NQ, int WS, bool BWD, bool TAGS>
__global__ void __launch_bounds__(CH_THREADS, (sizeof(T) == 4 ? 4 : 3) - BWD)
k_block(const __grid_constant__ SolveArgs<T> A) {
  using BB = BigBlock<T, NQ, WS, BWD, TAGS>;
  using Row = ChainRow<T, NQ>;
  constexpr int QL = Row::QL;
  extern __shared__ __align__(16) unsigned char chm[];
  __shared__ unsigned bad_s;
  T* ds = reinterpret_cast<T*>(chm);
  T* scr = ds + BR * DLD;
  T (*vs)[NQ] = reinterpret_cast<T (*)[NQ]>(scr + block_scratch<NQ, BWD, BLK_HB>());
  const int2_ bk = A.blocks[blockIdx.x];
  const int2_ cr = BWD ? int2_{0, 0} : A.blk_ch[blockIdx.x];
  BB M(A, bk.a);
  const int b = bk.b, nbs = M.nbs;
  const bool diag = BWD || b < nbs;
  const int n = !diag ? nbs : BWD ? nbs - 1 - b : b;
  T l[BLK_HB][16];
  // forward, the first tile is on its way before the children's rows are
  // added; backward the sums over x2 need the registers
  auto first = [&]() {
#pragma unroll
    for (int i = 0; i < BLK_HB; i++)
      if (i < n) M.tile(b, M.block_of(i), l[i]);
  };
  if (diag) M.stage_inverse(b, ds);
  if (!BWD) first();
  M.begin();
  M.template own_rhs<true>(b, cr, vs, scr);
  if (BWD) first();
  Row acc;
  acc.clear();
  M.template terms<BLK_HB>(b, n, l, acc, scr, &bad_s);
  grid_trigger();
  T z[QL], pv[QL];
  acc.sum(z);
#pragma unroll
  for (int q = 0; q < QL; q++) pv[q] = vs[Row::own()][Row::qb() + q] - z[q];
  if (!diag) {
    M.result(b, pv);
    return;
  }
  T d[16];
  M.inverse(ds, d);
  M.diagonal(b, d, pv, vs, z);
  if constexpr (TAGS) {
    M.publish(M.zf, b, z);
    M.result(b, z);
  } else {
    M.result(b, z);
    __syncthreads();
    // the barrier orders every thread's writes before thread 0's release store
    if (threadIdx.x == 0) st_release(A.flags + M.F.blk_off + b, A.epoch);
  }
}

// the start of a pass: the persistent queues' pending counts and heads; with
// the first pass of a call also the persistent set's done flags and the call
// counter of the published values
__global__ void k_solve_reset(int first, const int* __restrict__ pending0, int* pers, int np, int* counter) {
  grid_wait_then_trigger();
  const int i0 = blockIdx.x * blockDim.x + threadIdx.x, n = gridDim.x * blockDim.x;
  for (int i = i0; i < np; i += n) {
    pers[i] = pending0[i];
    if (first) pers[np + i] = 0;
  }
  if (i0 < 4) pers[2 * np + i0] = 0;
  if (first && i0 == 0) *counter += 1;
}

}  // namespace

// algorithmic bytes of one solve pass over a front, values of esz bytes: the
// lower panel read once, its row list, the work vector read and written
static double solve_pass_bytes(const FrontDesc& F, int nrhs, double esz) {
  const double s = F.s, m = F.f - F.s;
  return esz * (s * (s + 1.0) / 2.0 + m * s) + 4.0 * F.f + 2.0 * esz * nrhs * F.f;
}

// TAUCS_B200_NO_SOLVE_WALK=1 selects the block kernels (k_block) on every level
// instead of the cluster chains
static bool walk_enabled() {
  static const bool on = [] {
    const char* e = getenv("TAUCS_B200_NO_SOLVE_WALK");
    return !(e && *e && strcmp(e, "0") != 0);
  }();
  return on;
}

// the columns of the instantiation that a pass of nq right-hand sides takes
template <typename F>
static void sf_dispatch(int nq, F run) {
  if (nq <= 1) run(std::integral_constant<int, 1>());
  else if (nq <= 4) run(std::integral_constant<int, 4>());
  else run(std::integral_constant<int, SOLVE_NRHS>());
}

// the same for the chains: FP64 has no four-column form (DMMA takes eight)
template <typename T, typename F>
static void chain_dispatch(int nq, F run) {
  if (nq <= 1) run(std::integral_constant<int, 1>());
  else if (nq <= 4 && sizeof(T) == 4) run(std::integral_constant<int, sizeof(T) == 4 ? 4 : SOLVE_NRHS>());
  else run(std::integral_constant<int, SOLVE_NRHS>());
}

template <typename T>
static void solve_attrs() {
  // once per device and type (request-server workers reach this concurrently)
  static PerDeviceOnce pd;
  per_device_once(pd, [] {
    // static + dynamic shared memory of these kernels can exceed the default
    // 48 KB (8 columns in FP64)
    auto sf = [](auto nqc) {
      constexpr int Q = decltype(nqc)::value;
      // the most any launch asks for: 8 warps of fronts of order <= 32, or 4
      // warps with a full slot
      const size_t most = std::max(8 * sf_warp_smem<T, Q>(SMALL_WARP_F * (SMALL_WARP_F + 1), SMALL_WARP_F),
                                   4 * sf_warp_smem<T, Q>(SOLVE_SLOT_BYTES / sizeof(T), SMALL_F_MAX));
      cudaFuncSetAttribute(k_fwd_pers<T, Q, SOLVE_NRHS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) most);
      cudaFuncSetAttribute(k_bwd_pers<T, Q, SOLVE_NRHS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) most);
      cudaFuncSetAttribute(k_fwd<T, Q, SOLVE_NRHS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) most);
      cudaFuncSetAttribute(k_bwd<T, Q, SOLVE_NRHS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) most);
    };
    auto chain = [](auto nqc) {
      constexpr int Q = decltype(nqc)::value;
      cudaFuncSetAttribute(k_chain<T, Q, SOLVE_NRHS, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int) chain_smem<T, Q>());
      cudaFuncSetAttribute(k_chain<T, Q, SOLVE_NRHS, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int) chain_smem<T, Q>());
      cudaFuncSetAttribute(k_block<T, Q, SOLVE_NRHS, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int) block_smem<T, Q, false>());
      cudaFuncSetAttribute(k_block<T, Q, SOLVE_NRHS, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int) block_smem<T, Q, true>());
    };
    for (int nq : {1, 4, 8}) chain_dispatch<T>(nq, chain);
    sf(std::integral_constant<int, 1>());
    sf(std::integral_constant<int, 4>());
    sf(std::integral_constant<int, SOLVE_NRHS>());
    if constexpr (std::is_same<T, double>::value) {
      const int most = (int) (4 * sf_warp_smem<T, 1>(SOLVE_SLOT_BYTES / sizeof(T), SMALL_F_MAX));
      cudaFuncSetAttribute(k_fwd<T, 1, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
      cudaFuncSetAttribute(k_bwd<T, 1, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    }
    return true;
  });
}

// resident CTAs of a small-front kernel on the current device
template <typename K>
static int sf_resident(K kernel, int threads, size_t smem) {
  static PerDeviceOnce pd;
  static int sms[MAX_DEVICES];
  per_device_once(pd, [] {
    int d = 0;
    cudaGetDevice(&d);
    cudaDeviceGetAttribute(&sms[d], cudaDevAttrMultiProcessorCount, d);
    return true;
  });
  int d = 0, b = 0;
  cudaGetDevice(&d);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, threads, smem) != cudaSuccess) b = 1;
  return std::max(b, 1) * std::max(sms[d], 1);
}

// slot (elements) of a small-front launch whose largest panel has `need`
template <typename T>
static int sf_slot(int need) {
  return std::min((need + 3) & ~3, (int) (SOLVE_SLOT_BYTES / sizeof(T)));
}

// the queue part `part` of the persistent set: its tasks, and the warps per
// CTA (the second part's fronts take up to 16 KB of shared memory a warp:
// smaller CTAs fill an SM better)
static void sf_part(const Plan& P, int np, int part, int* t0, int* t1, int* threads) {
  *t0 = part ? P.pers_nwarp : 0;
  *t1 = part ? np : P.pers_nwarp;
  *threads = part ? 128 : 256;
}

template <typename T>
static int launch_solve(const Plan& P, const DevPlan& D, const T* L, const T* Dinv, int nrhs, T* X, const T* B, int ld, T* W,
                        T* part, int* counter, int* status, cudaStream_t st) {
  solve_attrs<T>();
  // the blocks' published values
  unsigned long long* zpub = reinterpret_cast<unsigned long long*>(part + P.fpart_off);
  unsigned long long* ppub = zpub + (size_t) P.n_blk * CH_VALUES * ch_words<T>();
  auto chain_level = [&](const LevelPlan& LP) {
    return walk_enabled() && LP.max_s_big >= CHAIN_MIN_S && (int) LP.big_fronts.size() <= chain_max_fronts<T>();
  };
  auto chain_grid = [](int nbig, int nblocks) { return nbig * CH_C + (nblocks + CH_C - 1) / CH_C * CH_C; };
  auto args = [&](int h, int nb, const int2_* bl, const int2_* bc, const T* Bq, T* Xq, int nq, int ep, int part_min) {
    return SolveArgs<T>{D.big_list + D.big_off[h], (int) P.levels[h].big_fronts.size(), bl, nb, bc, D.blk_child, D.fronts,
                        D.maps, D.rows, L, Dinv, Bq, Xq, ld, W, part, part_min, zpub, ppub, nullptr, nq, counter, ep, status};
  };
  const int np = D.n_pers;
  // the epochs of a call are always 1, 2, ... and the counter advances on the
  // device, so a recorded launch sequence stays valid
  auto reset = [&](bool first) {
    const int grid = std::max(1, std::min(GPU_SMS, (np + 255) / 256));
    launch(k_solve_reset, grid, 256, 0, st, first, D.pers_pending0, D.pers_solve, np, counter);
    count_launch();
  };
  auto small_list = [&](int h, int nq, auto launch) {
    const int ns = (int) P.levels[h].small_numeric.size();
    if (ns > 0) sf_dispatch(nq, [&](auto nqc) { launch(nqc, D.small_num + D.small_num_off[h], ns); });
  };
  int ep = 0;
  for (int q0 = 0; q0 < nrhs; q0 += SOLVE_NRHS) {
    const int nq = std::min(SOLVE_NRHS, nrhs - q0);
    const T* Bq = B + (size_t) q0 * ld;
    T* Xq = X + (size_t) q0 * ld;
    const int ef = ++ep;
    reset(q0 == 0);
    // every small front with only small fronts below it, a launch per part
    for (int pt = 0; pt < 2; pt++) {
      int t0, t1, th;
      sf_part(P, np, pt, &t0, &t1, &th);
      if (t1 <= t0) continue;
      double by = 0.0;
      if (prof_enabled())
        for (int t = t0; t < t1; t++) by += solve_pass_bytes(P.fronts[P.pers_fronts[t]], nq, sizeof(T));
      prof_begin(KC_SOLVE_FWD, st);
      sf_dispatch(nq, [&](auto nqc) {
        constexpr int Q = decltype(nqc)::value;
        const int slot = sf_slot<T>(P.pers_slot[pt]), wld = P.pers_wld[pt], nw = th / 32;
        const size_t smem = nw * sf_warp_smem<T, Q>(slot, wld);
        const int grid = std::min((t1 - t0 + nw - 1) / nw, sf_resident(k_fwd_pers<T, Q, SOLVE_NRHS>, th, smem));
        launch(k_fwd_pers<T, Q, SOLVE_NRHS>, grid, th, smem, st, D.solve_tasks, t0, t1, D.pers_solve,
                                                             D.pers_solve + 2 * np + pt, D.child_rec, D.maps, D.rows,
                                                             L, Bq, ld, W, nq, status, slot, wld);
      });
      prof_end(KC_SOLVE_FWD, st, 0.0, by);
      count_launch();
    }
    for (int h = 0; h < P.n_levels; h++) {
      const LevelPlan& LP = P.levels[h];
      double by = 0.0;
      if (prof_enabled())
        for (int i = LP.front_begin; i < LP.front_end; i++) by += solve_pass_bytes(P.fronts[i], nq, sizeof(T));
      prof_begin(KC_SOLVE_FWD, st);
      small_list(h, nq, [&](auto nqc, const int* sl, int ns) {
        constexpr int Q = decltype(nqc)::value;
        const int slot = sf_slot<T>(SMALL_F_MAX * (SMALL_F_MAX + 1));
        launch(k_fwd<T, Q, SOLVE_NRHS>, (ns + 3) / 4, 128, 4 * sf_warp_smem<T, Q>(slot, SMALL_F_MAX), st, sl, ns,
            D.fronts, D.child_rec, D.maps, D.rows, L, Bq, ld, W, nq, slot, SMALL_F_MAX);
        count_launch();
      });
      const int nb = (int) LP.solve_fwd_blocks.size();
      if (nb > 0) {
        const int2_ *bl = D.sfwd + D.sfwd_off[h], *bc = D.sfwd_ch + D.sfwd_off[h];
        const SolveArgs<T> A = args(h, nb, bl, bc, Bq, Xq, nq, ef, 1);
        chain_dispatch<T>(nq, [&](auto nqc) {
          constexpr int Q = decltype(nqc)::value;
          if (chain_level(LP))
            launch(k_chain<T, Q, SOLVE_NRHS, false>, chain_grid(A.nwalk, nb), CH_THREADS, chain_smem<T, Q>(), st, A);
          else
            launch(k_block<T, Q, SOLVE_NRHS, false, true>, nb, CH_THREADS, block_smem<T, Q, false>(), st, A);
        });
        count_launch();
      }
      prof_end(KC_SOLVE_FWD, st, 0.0, by);
    }
    const int eb = ++ep;
    for (int h = P.n_levels - 1; h >= 0; h--) {
      const LevelPlan& LP = P.levels[h];
      double by = 0.0;
      if (prof_enabled())
        for (int i = LP.front_begin; i < LP.front_end; i++) by += solve_pass_bytes(P.fronts[i], nq, sizeof(T));
      prof_begin(KC_SOLVE_BWD, st);
      const int nb = (int) LP.solve_bwd_blocks.size();
      if (nb > 0) {
        // chains take all their L21^T x2 from k_bwd_l21, the block kernel
        // that of fronts with more than one chunk of update rows
        const bool chain = chain_level(LP);
        const int nt = chain ? (int) LP.solve_l21_tasks.size() : LP.n_l21_multi;
        const int2_ *tl = D.sl21 + D.sl21_off[h], *bl = D.sbwd + D.sbwd_off[h];
        if (nt > 0) {
          sf_dispatch(nq, [&](auto nqc) {
            constexpr int Q = decltype(nqc)::value;
            // one CTA or less per SM: 16 warps each; the more CTAs, the
            // fewer warps each, down to 4 (solve at 64^3, FP64, backward: 4
            // warps always 1538 us, 16 always 1446, so 1380; mixed step at
            // 80^3, backward: 6509, 7333, 6441)
            if (nt <= GPU_SMS) launch(k_bwd_l21<T, Q, 512>, nt, 512, 0, st, tl, D.fronts, D.rows, L, Xq, ld, part, nq);
            else if (nt <= 4 * GPU_SMS) launch(k_bwd_l21<T, Q, 256>, nt, 256, 0, st, tl, D.fronts, D.rows, L, Xq, ld,
                                        part, nq);
            else launch(k_bwd_l21<T, Q, 128>, nt, 128, 0, st, tl, D.fronts, D.rows, L, Xq, ld, part, nq);
          });
          count_launch();
        }
        const SolveArgs<T> A = args(h, nb, bl, nullptr, nullptr, Xq, nq, eb, chain ? 1 : 2);
        chain_dispatch<T>(nq, [&](auto nqc) {
          constexpr int Q = decltype(nqc)::value;
          if (chain)
            launch(k_chain<T, Q, SOLVE_NRHS, true>, chain_grid(A.nwalk, nb), CH_THREADS, chain_smem<T, Q>(), st, A);
          else
            launch(k_block<T, Q, SOLVE_NRHS, true, true>, nb, CH_THREADS, block_smem<T, Q, true>(), st, A);
        });
        count_launch();
      }
      small_list(h, nq, [&](auto nqc, const int* sl, int ns) {
        constexpr int Q = decltype(nqc)::value;
        const int slot = sf_slot<T>(SMALL_F_MAX * (SMALL_F_MAX + 1));
        launch(k_bwd<T, Q, SOLVE_NRHS>, (ns + 3) / 4, 128, 4 * sf_warp_smem<T, Q>(slot, SMALL_F_MAX), st, sl, ns,
            D.fronts, D.rows, L, Xq, ld, W, nq, slot, SMALL_F_MAX);
        count_launch();
      });
      prof_end(KC_SOLVE_BWD, st, 0.0, by);
    }
    for (int pt = 1; pt >= 0; pt--) {
      int t0, t1, th;
      sf_part(P, np, pt, &t0, &t1, &th);
      if (t1 <= t0) continue;
      double by = 0.0;
      if (prof_enabled())
        for (int t = t0; t < t1; t++) by += solve_pass_bytes(P.fronts[P.pers_fronts[t]], nq, sizeof(T));
      prof_begin(KC_SOLVE_BWD, st);
      sf_dispatch(nq, [&](auto nqc) {
        constexpr int Q = decltype(nqc)::value;
        const int slot = sf_slot<T>(P.pers_slot[pt]), wld = P.pers_wld[pt], nw = th / 32;
        const size_t smem = nw * sf_warp_smem<T, Q>(slot, wld);
        const int grid = std::min((t1 - t0 + nw - 1) / nw, sf_resident(k_bwd_pers<T, Q, SOLVE_NRHS>, th, smem));
        launch(k_bwd_pers<T, Q, SOLVE_NRHS>, grid, th, smem, st, D.solve_tasks, t0, t1, D.pers_solve + np,
                                                             D.pers_solve + 2 * np + 2 + pt, eb, D.rows, L, Xq, ld, W,
                                                             nq, status, slot, wld);
      });
      prof_end(KC_SOLVE_BWD, st, 0.0, by);
      count_launch();
    }
  }
  return (int) cudaGetLastError();
}

int launch_solve_fp64(const Plan& P, const DevPlan& D, const double* L, const double* Dinv, int nrhs, double* X,
                      const double* B, int ld, double* W, double* part, int* calls, int* status,
                      cudaStream_t st) {
  return launch_solve<double>(P, D, L, Dinv, nrhs, X, B, ld, W, part, calls, status, st);
}

int launch_solve_fp32(const Plan& P, const DevPlan& D, const float* L, const float* Dinv, int nrhs, float* X,
                      const float* B, int ld, float* W, float* part, int* calls, int* status,
                      cudaStream_t st) {
  return launch_solve<float>(P, D, L, Dinv, nrhs, X, B, ld, W, part, calls, status, st);
}

}  // namespace tb

// ------------------------------------------------------------------------
// Solve without any allocation.
//
// Some callers must not allocate device memory: a serving thread that works
// inside a fixed, pre-reserved memory budget it may not grow; a latency-
// critical thread that may not call cudaMalloc/cudaFree because they can
// synchronise the device and stall every other stream; a host framework whose
// caching allocator already holds the rest of the GPU's memory.  They can
// still solve with an existing factor: taucs_b200_solve_device_noalloc keeps
// the solve's work vectors, handshake flags and status word in the one static
// device array below instead of the factor's own buffers.  It is the same
// level-scheduled solve as taucs_b200_solve_device, run one right-hand side
// per pass.  taucs_b200_solve_device_noalloc_status reads the status word.
// ------------------------------------------------------------------------

namespace tb {

constexpr size_t NOALLOC_W_DOUBLES = size_t(4) << 20;   // work vectors: 4 Mi doubles (32 MiB)
constexpr size_t NOALLOC_FLAGS = 16384;                 // handshake flags of the big fronts
constexpr size_t NOALLOC_DOUBLES = NOALLOC_W_DOUBLES + NOALLOC_FLAGS / 2 + 32;

// Every GPU that loads this library holds this array (about 32 MiB) until
// the process exits; all calls on a device share it.
static __device__ __align__(256) double g_noalloc_scratch[NOALLOC_DOUBLES];

static std::mutex g_noalloc_mu;
static double* g_noalloc_ptr[256];

// Device address of the static array on the current device, looked up once
// per device (the name is only a host-side stand-in for it).
static int noalloc_scratch(double** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 256) {
    set_error(std::string("taucs_b200_solve_device_noalloc: cudaGetDevice: ") + cudaGetErrorString(e));
    return -1;
  }
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_ptr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p) {
      set_error(std::string("taucs_b200_solve_device_noalloc: cudaGetSymbolAddress: ") + cudaGetErrorString(e));
      return -1;
    }
    g_noalloc_ptr[dev] = (double*) p;
  }
  *out = g_noalloc_ptr[dev];
  return 0;
}

// one right-hand side, work vectors at stride 1 (f doubles per front)
static int launch_solve_noalloc(const Plan& P, const DevPlan& D, const double* L, const double* Dinv, double* X,
                                const double* B,
                                int ld, double* W, int* flags, int* epoch, int* status, cudaStream_t st) {
  solve_attrs<double>();
  const int slot = sf_slot<double>(SMALL_F_MAX * (SMALL_F_MAX + 1));
  const int ef = ++*epoch;
  for (int h = 0; h < P.n_levels; h++) {
    const LevelPlan& LP = P.levels[h];
    const int ns = (int) LP.small_fronts.size();
    if (ns > 0) {
      launch(k_fwd<double, 1, 1>, (ns + 3) / 4, 128, 4 * sf_warp_smem<double, 1>(slot, SMALL_F_MAX), st,
          D.small_list + D.small_off[h], ns, D.fronts, D.child_rec, D.maps, D.rows, L, B, ld, W, 1, slot,
          SMALL_F_MAX);
      count_launch();
    }
    const int nb = (int) LP.solve_fwd_blocks.size();
    if (nb > 0) {
      const SolveArgs<double> A{nullptr, 0, D.sfwd + D.sfwd_off[h], nb, D.sfwd_ch + D.sfwd_off[h], D.blk_child, D.fronts,
                                D.maps, D.rows, L, Dinv, B, X, ld, W, nullptr, INT_MAX, nullptr, nullptr, flags, 1, nullptr,
                                ef, status};
      launch(k_block<double, 1, 1, false, false>, nb, CH_THREADS, block_smem<double, 1, false>(), st, A);
      count_launch();
    }
  }
  const int eb = ++*epoch;
  for (int h = P.n_levels - 1; h >= 0; h--) {
    const LevelPlan& LP = P.levels[h];
    const int nb = (int) LP.solve_bwd_blocks.size();
    if (nb > 0) {
      const SolveArgs<double> A{nullptr, 0, D.sbwd + D.sbwd_off[h], nb, nullptr, nullptr, D.fronts, D.maps, D.rows, L, Dinv,
                                nullptr, X, ld, W, nullptr, INT_MAX, nullptr, nullptr, flags, 1, nullptr, eb, status};
      launch(k_block<double, 1, 1, true, false>, nb, CH_THREADS, block_smem<double, 1, true>(), st, A);
      count_launch();
    }
    const int ns = (int) LP.small_fronts.size();
    if (ns > 0) {
      launch(k_bwd<double, 1, 1>, (ns + 3) / 4, 128, 4 * sf_warp_smem<double, 1>(slot, SMALL_F_MAX), st,
          D.small_list + D.small_off[h], ns, D.fronts, D.rows, L, X, ld, W, 1, slot, SMALL_F_MAX);
      count_launch();
    }
  }
  return (int) cudaGetLastError();
}

}  // namespace tb

extern "C" int taucs_b200_solve_device_noalloc(void* vL, int nrhs, double* d_X, const double* d_B, int ld) {
  using namespace tb;
  Factor* F = (Factor*) vL;
  if (!F || nrhs < 0 || ld < F->n || (nrhs > 0 && (!d_X || !d_B))) {
    set_error("taucs_b200_solve_device_noalloc: bad arguments");
    return -1;
  }
  const Plan& P = F->plan;
  if ((size_t) P.v_len > NOALLOC_W_DOUBLES || (size_t) P.n_blk > NOALLOC_FLAGS) {
    char msg[320];
    snprintf(msg, sizeof msg,
             "taucs_b200_solve_device_noalloc: this factor needs %lld doubles of work vectors and %d flags; "
             "the static scratch holds %zu doubles and %zu flags (use taucs_b200_solve_device)",
             (long long) P.v_len, P.n_blk, NOALLOC_W_DOUBLES, NOALLOC_FLAGS);
    set_error(msg);
    return -1;
  }
  if (!F->has_numeric || !F->dev_ready) {
    set_error("taucs_b200_solve_device_noalloc: the factor has no numeric part");
    return -1;
  }
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev != F->device) {
    set_error("taucs_b200_solve_device_noalloc: the current device is not the one the factor lives on");
    return -1;
  }
  if (nrhs == 0) return 0;
  double* base = nullptr;
  if (noalloc_scratch(&base)) return -1;
  double* W = base;
  int* flags = (int*) (base + NOALLOC_W_DOUBLES);
  int* status = flags + NOALLOC_FLAGS;
  cudaStream_t st = current_stream();
  // the array keeps whatever the previous call left: the flags and the status
  // word must start at zero, the work vectors are written before being read
  cudaError_t e = cudaMemsetAsync(flags, 0, sizeof(int) * (size_t) P.n_blk, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(status, 0, sizeof(int), st);
  if (e != cudaSuccess) {
    set_error(std::string("taucs_b200_solve_device_noalloc: ") + cudaGetErrorString(e));
    return -1;
  }
  int epoch = 0;
  for (int q = 0; q < nrhs; q++) {
    e = (cudaError_t) launch_solve_noalloc(P, F->dp, F->dL, F->dDinv, d_X + (size_t) q * ld, d_B + (size_t) q * ld, ld, W,
                                           flags, &epoch, status, st);
    if (e != cudaSuccess) {
      set_error(std::string("taucs_b200_solve_device_noalloc: ") + cudaGetErrorString(e));
      return -1;
    }
  }
  return 0;
}

// Status of the no-alloc solves issued on the current device: waits for the
// current stream, then reads the status word that those solves share.
extern "C" int taucs_b200_solve_device_noalloc_status(void) {
  using namespace tb;
  double* base = nullptr;
  if (noalloc_scratch(&base)) return -1;
  const int* status = (const int*) (base + NOALLOC_W_DOUBLES) + NOALLOC_FLAGS;
  cudaError_t e = cudaStreamSynchronize(current_stream());
  int h = 0;
  if (e == cudaSuccess) e = cudaMemcpy(&h, status, sizeof(int), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) {
    set_error(std::string("taucs_b200_solve_device_noalloc_status: ") + cudaGetErrorString(e));
    return -1;
  }
  if (h != 0) {
    set_error("taucs_b200_solve_device_noalloc: a bounded wait between thread blocks timed out; "
              "the solution is not valid");
    return -1;
  }
  return 0;
}
