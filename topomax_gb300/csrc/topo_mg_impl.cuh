// Kernels and host orchestration of the multigrid-preconditioned CG.
// Included by topo_mg_f32.cu / topo_mg_f64.cu, which instantiate MG<T>.
#pragma once

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdlib>
#include <cstdio>
#include <cstring>
#include <type_traits>
#include <utility>

#include "topo_kclock.h"
#include "topo_mg.h"
#include "topo_p1.cuh"
#include "topo_p1level.cuh"
#include "topo_p1march.cuh"
#include "topo_p2.cuh"
#include "topo_vec.cuh"

namespace topo {

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------
// Lattice kernels use a 2D grid: blockIdx.y is the row, x covers the columns.
constexpr int kRowThreads = 128;
// P1 levels keep an assembled stencil up to a node count: elasticity levels
// up to 2^18 nodes (a larger one streams 112 B per node and sweep, more than
// building the rows from its triangles' coefficients costs: level_row_free; at 126 k nodes stored
// rows and built ones measured the same, 10 and 11 us a sweep, at 31 k 3.2 and 4.8), filter levels
// always (32 B per node).  TOPO_STENCIL_NODES overrides both limits.
inline size_t stencil_max_nodes(int NC) {
  if (const char* e = std::getenv("TOPO_STENCIL_NODES")) return size_t(std::strtoull(e, nullptr, 10));
  return NC == 2 ? (size_t(1) << 18) : (size_t(1) << 40);
}
#define kRowThreads_ 128
inline dim3 row_grid(int NX, int NY) { return dim3((NX + kRowThreads - 1) / kRowThreads, NY); }

// The column-march P2 kernel (see P2March): each warp marches over one
// segment of cell rows; operand, density and element results move between
// lanes by shuffles.
template <class T>
__device__ __forceinline__ T shfl_down1(T v) { return __shfl_down_sync(0xffffffffu, v, 1); }
template <class T>
__device__ __forceinline__ T shfl_up1(T v) { return __shfl_up_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ dd shfl_down1(dd v) { return dd(shfl_down1(v.hi), shfl_down1(v.lo)); }
__device__ __forceinline__ dd shfl_up1(dd v) { return dd(shfl_up1(v.hi), shfl_up1(v.lo)); }

// column 2 of rows R0..2 (operand) and of density rows from lane L+1
template <class T, int R0, bool OPERAND>
__device__ __forceinline__ void p2m_exchange_down(P2Lane<T>& L) {
  if (OPERAND) {
#pragma unroll
    for (int r = R0; r <= 2; ++r)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const T v = shfl_down1(L.U[r][0][c]);
        if (!L.edge) L.U[r][2][c] = v;
      }
  }
#pragma unroll
  for (int r = (R0 == 0 ? 0 : 1); r <= 1; ++r) {
    const T v = shfl_down1(L.X[r][0]);
    if (!L.edge) L.X[r][1] = v;
  }
}

// element results of column 2 to lane L+1's column 0
template <class T>
__device__ __forceinline__ void p2m_exchange_up(P2Lane<T>& L, int lane) {
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const T v = shfl_up1(L.A[r][2][c]);
      if (lane > 0) L.A[r][0][c] += v;
    }
}

// End of one CG iteration: convergence / cap / breakdown test and beta (run by
// one thread: the reduction's last block, or k_pcg_check).
__device__ inline void pcg_check_dev(PcgDev* dv, cudaGraphConditionalHandle h, int use_cond) {
  dv->it += 1;
  const double pq = dv->pq, rr = dv->rr, rzn = dv->rz_new;
  int st = 1;
  if (!isfinite(pq) || !isfinite(rr) || !isfinite(rzn)) st = 4;
  else if (!(pq > 0.0) || !(dv->rz > 0.0)) st = 3;
  else if (rr <= dv->tol2) st = 0;
  else if (dv->it >= dv->maxit) st = 2;
  // (a chain of FP64 divisions and a root takes this one thread over 1 us: only what is needed)
  if (st == 1) {
    dv->beta = rzn / dv->rz;
  } else {
    dv->beta = 0.0;
    dv->relres = sqrt(rr / dv->bb);
  }
  dv->rz = rzn;
  dv->status = st;
  if (use_cond) cudaGraphSetConditional(h, st == 1 ? 1u : 0u);
}

// One warp's march over cell rows js .. je-1 (see P2March).  LEAN: the warp's
// region passed P2March::lean_region, so the phases make no per-node tests.
template <class T, int MODE, bool LEAN>
__device__ __forceinline__ void p2_march_run(const P2Params<T>& P, const T* xi, const P2Io<T>& io,
                                             int lane, int js, int je, T (&acc)[2]) {
  constexpr bool OPERAND = MODE != kP2Diag;
  P2Lane<T> L;
  P2March<T>::begin(P, L, int(blockIdx.x) * P2M_OWN - 1 + lane, lane == 31);
  const bool owner = lane > 0 && L.i <= P.nx;
  int j = js > 0 ? js - 1 : 0;
  P2March<T>::template load<0, LEAN>(P, io, xi, L, j);
  P2March<T>::template load_mass<LEAN>(P, L.K, L.i, j, L.M);
  p2m_exchange_down<T, 0, OPERAND>(L);
  P2Next<T> N;
  for (;;) {
    const bool more = j + 1 < je;
    if (more) P2March<T>::template prefetch<LEAN>(P, io, xi, L, j + 1, N);  // in flight during this step's arithmetic
    const bool fin = owner && j >= js;
    typename P2March<T>::Fin F;
    if (MODE != kP2Apply && MODE != kP2Diag && fin) P2March<T>::template fin_load<LEAN>(P, io, L, j, F);
    // the pair type keeps no prefetched mass matrices (registers): they are loaded here
    if constexpr (IsDD<T>::value) P2March<T>::template load_mass<LEAN>(P, L.K, L.i, j, L.M);
    P2March<T>::template compute<LEAN>(P, L, j, MODE);
    p2m_exchange_up<T>(L, lane);
    if (fin) P2March<T>::template finish<LEAN>(P, io, L, j, j == P.ny - 1 ? 3 : 2, F, acc);
    if (!more) break;
    ++j;
    P2March<T>::advance(L);
    P2March<T>::take(L, N);
    p2m_exchange_down<T, 1, OPERAND>(L);
  }
}

// resident blocks the register budget is sized for: FP32 4, pair-of-FP32 3, FP64 2
template <class T>
constexpr int p2_march_min_blocks() {
  return IsDD<T>::value ? 3 : sizeof(T) == 4 ? 4 : 2;
}

// the CG's reductions fused into a launch (P2Io::fuse)
template <class T, int MODE>
__device__ __forceinline__ void p2_reduce(const P2Io<T>& io, const T (&acc)[2]) {
  if constexpr ((MODE == kP2Apply || MODE == kP2Post2) && !IsDD<T>::value) {
    if (io.fuse == kFuseNone) return;
    double tot[2];
    if (!finish_reduction<2>(acc, io.partials, io.counter, tot)) return;
    if (io.fuse == kFusePQ) {
      io.pcg->pq = tot[0];
    } else {
      io.pcg->rr = tot[0];
      io.pcg->rz_new = tot[1];
      pcg_check_dev(io.pcg, cudaGraphConditionalHandle(io.cond), io.use_cond);
    }
  }
}

template <class T, int MODE>
__global__ void __launch_bounds__(P2M_THREADS, p2_march_min_blocks<T>())
    k_p2_march(P2Params<T> P, const T* xi, P2Io<T> io, int seg) {
  TOPO_PDL_ENTRY();
  io.mode = MODE;  // compile-time mode: the per-node switches fold
  P2March<T>::prepare(io);
  const int lane = threadIdx.x & 31;
  const int js = (blockIdx.y * P2M_WARPS + (threadIdx.x >> 5)) * seg;
  T acc[2] = {T(0), T(0)};  // fused CG reductions (P2Io::fuse)
  if (js < P.ny) {  // whole warp: warps past the last segment only join the reduction
    const int je = min(js + seg, P.ny);
    // warp-uniform: the same cell columns and rows for all lanes
    if constexpr (IsDD<T>::value) {
      // pair-of-FP32: issue-bound on a long element body; one copy of it (the masked
      // phases) keeps the code within reach of the instruction caches
      p2_march_run<T, MODE, false>(P, xi, io, lane, js, je, acc);
    } else if (P2March<T>::lean_region(P, int(blockIdx.x) * P2M_OWN - 1, js > 0 ? js - 1 : 0, je)) {
      p2_march_run<T, MODE, true>(P, xi, io, lane, js, je, acc);
    } else {
      p2_march_run<T, MODE, false>(P, xi, io, lane, js, je, acc);
    }
  }
  p2_reduce<T, MODE>(io, acc);
}

// One cell row of the short form: warp 0 of a block takes the row below its own P2R_ROWS, for
// what that row adds to their lowest node row; each warp hands its top node row's sums to the
// next through shared memory.  top: 4 values per thread.
template <class T, int MODE, bool LEAN>
__device__ __forceinline__ void p2_rows_run(const P2Params<T>& P, const T* xi, P2Io<T>& io, int lane, int j, bool own,
                                            T* top, T (&acc)[2]) {
  P2Lane<T> L;
  P2March<T>::begin(P, L, int(blockIdx.x) * P2M_OWN - 1 + lane, lane == 31);
  const bool row = j >= 0 && j < P.ny;
  const bool fin = own && row && lane > 0 && L.i <= P.nx;
  if (io.early) {
    P2March<T>::prepare(io);
    if (row) P2March<T>::template load_mass<LEAN>(P, L.K, L.i, j, L.M);
  }
  TOPO_PDL_WAIT();
  TOPO_PDL_LAUNCH();
  if (!io.early) {
    P2March<T>::prepare(io);
    if (row) P2March<T>::template load_mass<LEAN>(P, L.K, L.i, j, L.M);
  }
  typename P2March<T>::Fin F;
  if (row) {  // (the whole warp)
    P2March<T>::template load<0, LEAN>(P, io, xi, L, j);
    if (MODE != kP2Apply && MODE != kP2Diag && fin) P2March<T>::template fin_load<LEAN>(P, io, L, j, F);
    p2m_exchange_down<T, 0, MODE != kP2Diag>(L);
    P2March<T>::template compute<LEAN>(P, L, j, MODE);
    p2m_exchange_up<T>(L, lane);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) top[k * P2R_THREADS + threadIdx.x] = L.A[2][k >> 1][k & 1];
  __syncthreads();
  if (!fin) return;
  if (j > 0)
#pragma unroll
    for (int k = 0; k < 4; ++k) L.A[0][k >> 1][k & 1] += top[k * P2R_THREADS + threadIdx.x - 32];
  P2March<T>::template finish<LEAN>(P, io, L, j, j == P.ny - 1 ? 3 : 2, F, acc);
}

// A march with segments of one row computes each row twice and, in FP64, is bound by the pipe that
// a block's warps share: 160x80 has 480 warps' rows, five row steps per SM here against eight.
template <class T, int MODE>
__global__ void __launch_bounds__(P2R_THREADS, sizeof(T) == 4 ? 3 : 2)
    k_p2_rows(P2Params<T> P, const T* xi, P2Io<T> io) {
  __shared__ T top[4 * P2R_THREADS];
  io.mode = MODE;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, J0 = blockIdx.y * P2R_ROWS, j = J0 - 1 + w;
  T acc[2] = {T(0), T(0)};
  // block-uniform
  if (!IsDD<T>::value &&
      P2March<T>::lean_region(P, int(blockIdx.x) * P2M_OWN - 1, J0 > 0 ? J0 - 1 : 0, J0 + P2R_ROWS))
    p2_rows_run<T, MODE, true>(P, xi, io, lane, j, w > 0, top, acc);
  else
    p2_rows_run<T, MODE, false>(P, xi, io, lane, j, w > 0, top, acc);
  p2_reduce<T, MODE>(io, acc);
}

// The column-march kernel of the large P1 levels (see P1March).
template <class T, int NC, int MODE>
__global__ void __launch_bounds__(P2M_THREADS) k_p1_march(P1Params<T, NC> P, P1Io<T> io, int seg) {
  TOPO_PDL_ENTRY();
  io.mode = MODE;
  P1March<T, NC>::prepare(io);
  const int lane = threadIdx.x & 31;
  const int js = (blockIdx.y * P2M_WARPS + (threadIdx.x >> 5)) * seg;
  if (js >= P.ny) return;  // whole warp
  const int je = min(js + seg, P.ny);
  P1Lane<T, NC> L;
  P1March<T, NC>::begin(L, int(blockIdx.x) * P2M_OWN - 1 + lane, lane == 31);
  const bool owner = lane > 0 && L.i <= P.nx;
  int j = js > 0 ? js - 1 : 0;
  auto down = [&](int r0) {
#pragma unroll
    for (int r = 0; r <= 1; ++r) {
      if (r < r0) continue;
#pragma unroll
      for (int d = 0; d < NC; ++d) {
        const T v = shfl_down1(L.U[r][0][d]);
        if (!L.edge) L.U[r][1][d] = v;
      }
    }
  };
  P1March<T, NC>::template load<0>(P, io, L, j);
  P1March<T, NC>::load_coef(P, L.i, j, L.kk, L.km);
  down(0);
  P1Next<T, NC> N;
  for (;;) {
    const bool more = j + 1 < je;
    if (more) P1March<T, NC>::prefetch(P, io, L, j + 1, N);  // in flight during this step's arithmetic
    const bool fin = owner && j >= js;
    typename P1March<T, NC>::Fin F;
    if (MODE != kP2Apply && fin) P1March<T, NC>::fin_load(P, io, L.i, j, F);
    P1March<T, NC>::compute(P, L, j);
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int d = 0; d < NC; ++d) {
        const T v = shfl_up1(L.A[r][1][d]);
        if (lane > 0) L.A[r][0][d] += v;
      }
    if (fin) P1March<T, NC>::finish(P, io, L, j, j == P.ny - 1 ? 2 : 1, F);
    if (!more) break;
    ++j;
    P1March<T, NC>::advance(L);
    P1March<T, NC>::take(L, N);
    down(1);
  }
}

// The sweeps of a stencil level (see topo_p1level.cuh).  The rows, inverse diagonals and
// smoothing coefficients are fixed during a solve, so they are read before the wait for
// the predecessor; the successor may start its own such reads at once.
//
// Against six launches a level (smoothing steps, residual, transfers) a design evaluation went from
// 11.4 to 7.7 ms at 320x160 and from 22.1 to 17.8 at 1000x500.
// Tile: 10 x 4 coarse nodes, 253 threads for 160 fine nodes of its own down, 220 up (two steps); on
// the 1000x500 evaluation 14 x 6 measured 18.8 ms against 18.6, 6 x 6 19.2, 14 x 2 18.9.  It is
// a constant in FP32 (index arithmetic without divisions).  FP64 tiles: see level_sweep (a tile's
// recomputed ring costs FP64-pipe time, a large tile leaves SMs without a block).
// Levels with built rows fill the chip many times over and take 14 x 6 (31 x 15 nodes for 28 x 12)
// at two steps: 67.9 us down against 70.9 at two million nodes; their loads are issued together
// before the row is built (59.4).  Level 1 of 1000x500 takes 17 + 16 us, of 2000x1000 59 + 64
// (as column marches and transfers 59 and 160).
constexpr int kSweepTileX = 10, kSweepTileY = 4;
// ROWS: StoredRows, or the P1Params that the rows are built from.
struct StoredRows {};
template <class ROWS, int D>
constexpr int sweep_tile_x() {
  return std::is_same<ROWS, StoredRows>::value || D > 2 ? kSweepTileX : 14;
}
template <class ROWS, int D>
constexpr int sweep_tile_y() {
  return std::is_same<ROWS, StoredRows>::value || D > 2 ? kSweepTileY : 6;
}
template <class ROWS, int D>
constexpr int sweep_threads() {  // the down sweep's region, the larger one
  return ((2 * sweep_tile_x<ROWS, D>() + 2 * D - 1) * (2 * sweep_tile_y<ROWS, D>() + 2 * D - 1) + 31) / 32 * 32;
}

template <class T, int NC>
__device__ __forceinline__ const P1Params<T, NC>* row_source(const P1Params<T, NC>& Q) { return &Q; }
template <class T, int NC>
__device__ __forceinline__ const P1Params<T, NC>* row_source(const StoredRows&) { return nullptr; }

// FP32 blocks have one tile (level_sweep), so their index arithmetic divides by constants.
template <class T, int NC, int D, class ROWS>
__global__ void __launch_bounds__(sweep_threads<ROWS, D>())
    k_level_down(LevelSweep<T, NC> P, const ROWS Q, const T* b, T* x, T* bc) {
  using Ph = LevelPhases<T, NC>;
  extern __shared__ __align__(16) unsigned char sweep_raw[];
  constexpr bool F = sizeof(T) == 4, stored = std::is_same<ROWS, StoredRows>::value;
  const int cx = F ? sweep_tile_x<ROWS, D>() : P.cx, cy = F ? sweep_tile_y<ROWS, D>() : P.cy, w = 2 * cx + 2 * D - 1, h = 2 * cy + 2 * D - 1;
  T* s = reinterpret_cast<T*>(sweep_raw);
  T* sn = s + NC * (w + 2) * (h + 2);
  const int tid = threadIdx.x, nt = blockDim.x, I0 = blockIdx.x * cx, J0 = blockIdx.y * cy;
  b += blockIdx.z * size_t(NC) * P.NX * P.NY;  // the batch's vectors
  x += blockIdx.z * size_t(NC) * P.NX * P.NY;
  bc += blockIdx.z * size_t(NC) * P.NXc * P.NYc;
  TOPO_PDL_LAUNCH();
  const int a0 = 2 * I0 - D, b0 = 2 * J0 - D;
  typename Ph::Node N;
  const bool on = Ph::template start<D>(P, a0, b0, w, h, tid, N);
  if (on && stored) N.load(P);
  TOPO_PDL_WAIT();
  if (on) N.load_b(P, b);
  if (on && !stored) N.load(P, row_source<T, NC>(Q));
  Ph::down_first(P, a0, b0, w, h, tid, nt, b, s, on, N);
  __syncthreads();
#pragma unroll
  for (int k = 1; k < D; ++k) {
    if (on && k + 1 < D) Ph::step(P, k, w, s, sn, N);
    if (on && k + 1 == D) Ph::last(P, k, w, s, sn, N);
    T* const t = s;
    s = sn;
    sn = t;
    __syncthreads();
  }
  if (on) {
    Ph::store(P, a0, b0, D, N, x);
    Ph::down_residual(w, s, sn, N);
  }
  __syncthreads();
  Ph::restrict_to(P, cx, cy, I0, J0, w, D, tid, nt, sn, bc);
}

template <class T, int NC, int D, class ROWS>
__global__ void __launch_bounds__(sweep_threads<ROWS, D>())
    k_level_up(LevelSweep<T, NC> P, const ROWS Q, const T* b, const T* xin, const T* xc, T* x) {
  using Ph = LevelPhases<T, NC>;
  extern __shared__ __align__(16) unsigned char sweep_raw[];
  constexpr bool F = sizeof(T) == 4, stored = std::is_same<ROWS, StoredRows>::value;
  const int cx = F ? sweep_tile_x<ROWS, D>() : P.cx, cy = F ? sweep_tile_y<ROWS, D>() : P.cy, w = 2 * cx + 2 * D - 2, h = 2 * cy + 2 * D - 2;
  T* s = reinterpret_cast<T*>(sweep_raw);
  T* sn = s + NC * (w + 2) * (h + 2);
  const int tid = threadIdx.x, nt = blockDim.x, I0 = blockIdx.x * cx, J0 = blockIdx.y * cy;
  b += blockIdx.z * size_t(NC) * P.NX * P.NY;
  x += blockIdx.z * size_t(NC) * P.NX * P.NY;
  xin += blockIdx.z * size_t(NC) * P.NX * P.NY;
  xc += blockIdx.z * size_t(NC) * P.NXc * P.NYc;
  TOPO_PDL_LAUNCH();
  const int a0 = 2 * I0 - (D - 1), b0 = 2 * J0 - (D - 1);
  typename Ph::Node N;
  const bool on = Ph::template start<D>(P, a0, b0, w, h, tid, N);
  if (on && stored) N.load(P);
  TOPO_PDL_WAIT();
  if (on) {
    N.load_b(P, b);
    Ph::up_own(P, xin, xc, N);
    if (!stored) N.load(P, row_source<T, NC>(Q));
  }
  Ph::up_first(P, a0, b0, w, h, tid, nt, xin, xc, s, on, N);
  __syncthreads();
  if (on) Ph::up_residual(P, w, s, sn, N);
#pragma unroll
  for (int k = 1; k < D; ++k) {
    T* const t = s;
    s = sn;
    sn = t;
    __syncthreads();
    if (on && k + 1 < D) Ph::step(P, k, w, s, sn, N);
    if (on && k + 1 == D) Ph::last(P, k, w, s, static_cast<T*>(nullptr), N);
  }
  if (on) Ph::store(P, a0, b0, D - 1, N, x);
}

template <class T, int NC>
__global__ void __launch_bounds__(kRowThreads_) k_prolong_add(Transfer X, const T* xc, T* xf) {
  TOPO_PDL_ENTRY();
  const int a = blockIdx.x * kRowThreads_ + threadIdx.x, b = blockIdx.y;
  if (a < X.NXf) TransferKern<T, NC>::node_prolong_add(a, b, X, xc, xf);
}

template <class T, int NC, class PP>
__global__ void __launch_bounds__(kRowThreads) k_p1_apply(PP P, const T* u, T* y) {
  TOPO_PDL_ENTRY();
  const int a = blockIdx.x * kRowThreads + threadIdx.x, b = blockIdx.y;
  if (a <= P.nx) p1_node_apply<T, NC>(a, b, P, u, y);
}

template <class T, int NC>
__global__ void __launch_bounds__(kRowThreads) k_p1_diag(P1Params<T, NC> P, T* __restrict__ d) {
  const int a = blockIdx.x * kRowThreads + threadIdx.x, b = blockIdx.y;
  if (a <= P.nx) P1Kern<T, NC>::node_diag(a, b, P, d);
}

template <class T, int NC>
__global__ void __launch_bounds__(kRowThreads) k_p1_stencil(P1Params<T, NC> P, T* __restrict__ st) {
  const int a = blockIdx.x * kRowThreads + threadIdx.x, b = blockIdx.y;
  if (a <= P.nx) p1_stencil_node<T, NC>(a, b, P, st + (size_t(b) * (P.nx + 1) + a) * StencilLayout<NC>::stride);
}

template <class T, int NC>
__global__ void __launch_bounds__(kRowThreads) k_restrict(Transfer X, const T* rf, T* bc, const T* tf) {
  TOPO_PDL_ENTRY();
  const int I = blockIdx.x * kRowThreads + threadIdx.x, J = blockIdx.y;
  if (I < X.NXc) TransferKern<T, NC>::node_restrict(I, J, X, rf, bc, tf);
}


// deterministic pseudo-random start vector for the power iteration
template <class T>
__global__ void k_power_start(T* x, size_t n) {
  TOPO_GRID_STRIDE(i, n) {
    unsigned h = unsigned(i) * 2654435761u + 0x9e3779b9u;
    h ^= h >> 15;
    h *= 2246822519u;
    h ^= h >> 13;
    x[i] = T(0.5) + T(h & 0xffffu) / T(65536.0);
  }
}

// Dense inverse of the coarsest operator (n <= kCoarseMaxDofs), assembled from
// the FP64 coefficient masters, Gauss-Jordan (SPD, no pivoting) by ONE warp:
// lane j owns column j in shared memory, so a step needs no block barrier and
// one reciprocal of the pivot.
template <class T, int NC>
__global__ void __launch_bounds__(32) k_coarse_inverse(int nx, int ny, Dir dir, ElemRefs R,
                                                       const double* __restrict__ kK, const double* __restrict__ kM,
                                                       T* __restrict__ inv, int* status) {
  __shared__ double A[kCoarseMaxDofs * kCoarseMaxDofs];
  const int NX = nx + 1, NY = ny + 1, n = NX * NY * NC;
  const int j = threadIdx.x;
  for (int i = j; i < n * n; i += 32) A[i] = 0.0;
  __syncwarp();
  if (j == 0) {
    for (int cj = 0; cj < ny; ++cj)
      for (int ci = 0; ci < nx; ++ci)
        for (int o = 0; o < 2; ++o) {
          const size_t t = (size_t(cj) * nx + ci) * 2 + o;
          const double kk = kK[t];
          const double km = (NC == 1 && kM) ? kM[t] : 0.0;
          for (int k = 0; k < 3; ++k) {
            const int nk = (cj + p1_off_b(o, k)) * NX + ci + p1_off_a(o, k);
            for (int l = 0; l < 3; ++l) {
              const int nl = (cj + p1_off_b(o, l)) * NX + ci + p1_off_a(o, l);
              for (int c = 0; c < NC; ++c)
                for (int d = 0; d < NC; ++d) {
                  double v;
                  if (NC == 2) v = kk * R.K2[o][k * 2 + c][l * 2 + d];
                  else v = kk * R.K1[o][k][l] + km * R.M1[o][k][l];
                  A[(NC * nk + c) * n + NC * nl + d] += v;
                }
            }
          }
        }
  }
  __syncwarp();
  for (int i = j; i < n * n; i += 32) {
    const int r = i / n, c = i % n;
    const int nr = r / NC, nc = c / NC;
    const bool cr = is_clamped(dir, nr % NX, nr / NX), cc = is_clamped(dir, nc % NX, nc / NX);
    if (cr || cc) A[i] = (r == c) ? 1.0 : 0.0;
  }
  __syncwarp();
  int bad = 0;
  for (int k = 0; k < n; ++k) {
    const double p = A[k * n + k];
    if (!(p > 0.0) || !isfinite(p)) {  // the same value in every lane: a uniform exit
      bad = 1;
      break;
    }
    const double ip = 1.0 / p;
    double f[kCoarseMaxDofs];  // column k before this step
#pragma unroll
    for (int i = 0; i < kCoarseMaxDofs; ++i) f[i] = i < n ? A[i * n + k] : 0.0;
    __syncwarp();
    if (j < n) {
      if (j == k) {
#pragma unroll
        for (int i = 0; i < kCoarseMaxDofs; ++i)
          if (i < n) A[i * n + k] = (i == k) ? ip : -f[i] * ip;
      } else {
        const double c = A[k * n + j] * ip;
#pragma unroll
        for (int i = 0; i < kCoarseMaxDofs; ++i)
          if (i < n) A[i * n + j] = (i == k) ? c : A[i * n + j] - f[i] * c;
      }
    }
    __syncwarp();
  }
  for (int i = j; i < n * n; i += 32) {
    const int r = i / n, c = i % n;
    inv[i] = T(0.5 * (A[r * n + c] + A[c * n + r]));
  }
  if (j == 0) *status = bad;
}

// x = Ainv b on the coarsest level, n <= kCoarseMaxDofs (Ainv symmetric: column reads)
constexpr int kDenseThreads = 256;
template <class T>
__global__ void __launch_bounds__(kDenseThreads) k_dense_matvec(const T* Ainv, const T* b, T* x, int n) {
  __shared__ T A[kCoarseMaxDofs * kCoarseMaxDofs], v[kCoarseMaxDofs];
  TOPO_PDL_LAUNCH();
  const int i = threadIdx.x;
  for (int k = i; k < n * n; k += kDenseThreads) A[k] = Ainv[k];
  TOPO_PDL_WAIT();
  if (i < n) v[i] = b[blockIdx.x * size_t(n) + i];
  __syncthreads();
  if (i >= n) return;
  T s = T(0);
  for (int j = 0; j < n; ++j) s = fma_t(A[j * n + i], v[j], s);
  x[blockIdx.x * size_t(n) + i] = s;
}

constexpr int kCoarseThreads = 1024;                   // one-CTA coarse Chebyshev solve
constexpr size_t kCoarseSharedBudget = 196 * 1024;

// Phases of the tail.  A thread's node of a level: its row, inverse diagonal, right-hand side.
template <class T, int NC>
struct TailNode {
  __align__(16) T st[StencilLayout<NC>::stride];
  T di[NC], b[NC];
};

// D - 1 steps from the direction d in shared vector s; the direction goes to sn and back in turn,
// r and v are the residual and the iterate.  The last step stores the iterate instead.
// Returns its vector (the stores followed by a barrier).
template <class T, int NC, int D>
__device__ __forceinline__ T* tail_steps(const T* cheb, bool on, int w, int p, const TailNode<T, NC>& N, T (&r)[NC],
                                         T (&v)[NC], T (&d)[NC], T* s, T* sn) {
#pragma unroll
  for (int k = 1; k < D; ++k) {
    if (on) {
      T t[NC];
      level_apply<T, NC>(N.st, s, w, p, t);
      const T c1 = cheb[2 * k - 1], c2 = cheb[2 * k];
      for (int c = 0; c < NC; ++c) {
        if (k + 1 < D) {
          r[c] -= t[c];
          d[c] = level_direction(c1, d[c], c2, N.di[c], r[c]);
          v[c] += d[c];
          sn[NC * p + c] = d[c];
        } else {
          v[c] = level_last(v[c], c1, d[c], c2, N.di[c], r[c] - t[c]);
          sn[NC * p + c] = v[c];
        }
      }
    }
    T* const q = s;
    s = sn;
    sn = q;
    __syncthreads();
  }
  return s;
}

// Level l from its right-hand side to the next level's; leaves x in L.x.
template <class T, int NC, int D>
__device__ __forceinline__ void tail_down(const TailSweep<T, NC>& P, int l, int tid, T* sm, const TailNode<T, NC>& N) {
  const auto& L = P.lv[l];
  const auto& K = P.lv[l + 1];
  const bool on = tid < L.NX * L.NY;
  const int j = tid / L.NX, i = tid - j * L.NX, w = L.NX + 2, p = on ? (j + 1) * w + i + 1 : 0;
  T r[NC], v[NC], d[NC], t[NC];
  const T c0 = L.cheb[0];
  for (int c = 0; c < NC; ++c) {
    r[c] = N.b[c];
    v[c] = d[c] = (c0 * N.di[c]) * N.b[c];
    if (on) sm[L.d + NC * p + c] = d[c];
  }
  __syncthreads();
  const T* s = tail_steps<T, NC, D>(L.cheb, on, w, p, N, r, v, d, sm + L.d, sm + L.x);
  if (on) level_apply<T, NC>(N.st, s, w, p, t);
  __syncthreads();  // the iterate has been read
  if (on)
    for (int c = 0; c < NC; ++c) {
      sm[L.d + NC * p + c] = N.b[c] - t[c];
      sm[L.x + NC * p + c] = v[c];
    }
  __syncthreads();
  if (tid < K.NX * K.NY) {
    const int J = tid / K.NX, I = tid - J * K.NX;
    const bool zero = is_clamped(K.dir, I, J);
    const T* q = sm + L.d + NC * ((2 * J + 1) * w + 2 * I + 1);
    for (int c = 0; c < NC; ++c) sm[K.b + NC * tid + c] = zero ? T(0) : level_restrict<T, NC>(q + c, w);
  }
  __syncthreads();
}

// Level l from x and the next level's correction to its solution: to xg (level 0) or L.x.
template <class T, int NC, int D>
__device__ __forceinline__ void tail_up(const TailSweep<T, NC>& P, int l, int tid, T* sm, const TailNode<T, NC>& N,
                                        T* xg) {
  const auto& L = P.lv[l];
  const auto& K = P.lv[l + 1];
  const bool on = tid < L.NX * L.NY;
  const int j = tid / L.NX, i = tid - j * L.NX, w = L.NX + 2, p = on ? (j + 1) * w + i + 1 : 0;
  T r[NC], v[NC], d[NC];
  for (int c = 0; c < NC; ++c) r[c] = v[c] = d[c] = T(0);
  if (on && !is_clamped(L.dir, i, j)) {
    const int wc = K.NX + 2;
    const int m0 = ((j >> 1) + 1) * wc + (i >> 1) + 1, m1 = (((j + 1) >> 1) + 1) * wc + ((i + 1) >> 1) + 1;
    for (int c = 0; c < NC; ++c) {
      const T u = sm[K.x + NC * m0 + c], q = sm[K.x + NC * m1 + c];
      sm[L.x + NC * p + c] += m0 == m1 ? u : T(0.5) * (u + q);
    }
  }
  __syncthreads();
  if (on) {
    T t[NC];
    level_apply<T, NC>(N.st, sm + L.x, w, p, t);
    const T c0 = L.cheb[0];
    for (int c = 0; c < NC; ++c) {
      r[c] = N.b[c] - t[c];
      d[c] = (c0 * N.di[c]) * r[c];
      v[c] = sm[L.x + NC * p + c] + d[c];
      sm[L.d + NC * p + c] = d[c];
    }
  }
  __syncthreads();
  tail_steps<T, NC, D>(L.cheb, on, w, p, N, r, v, d, sm + L.d, sm + L.x);
  if (on)
    for (int c = 0; c < NC; ++c) {
      if (l == 0) xg[NC * tid + c] = v[c];
      else sm[L.x + NC * p + c] = v[c];
    }
  if (l) __syncthreads();
}

// a level >= 1's node from shared memory
template <class T, int NC>
__device__ __forceinline__ void tail_node(const TailSweep<T, NC>& P, int l, int tid, const T* sm, TailNode<T, NC>& N) {
  const auto& L = P.lv[l];
  const int n = tid < L.NX * L.NY ? tid : 0;
  copy_row<T, StencilLayout<NC>::stride>(sm + L.row + n * StencilLayout<NC>::stride, N.st);
  for (int c = 0; c < NC; ++c) {
    N.di[c] = sm[L.di + NC * n + c];
    N.b[c] = sm[L.b + NC * n + c];
  }
}

// The last levels of the V-cycle (see TailSweep): x = V-cycle(b) from its level 0 down, D
// Chebyshev steps each way.  Latency-bound: 2 D + 4 barriers a level.  TRACE: SM cycles of every phase
// in execution order, summed in P.trace (TOPO_PROFILE), and the launches after them.
template <class T, int NC, int D, bool TRACE>
__global__ void __launch_bounds__(kTailNodes)
    k_level_tail(const __grid_constant__ TailSweep<T, NC> P, const T* b, T* x) {
  constexpr int SW = StencilLayout<NC>::stride;
  extern __shared__ __align__(16) unsigned char sweep_raw[];
  T* sm = reinterpret_cast<T*>(sweep_raw);
  const int tid = threadIdx.x, nt = blockDim.x;
  b += blockIdx.x * size_t(NC) * P.lv[0].NX * P.lv[0].NY;
  x += blockIdx.x * size_t(NC) * P.lv[0].NX * P.lv[0].NY;
  TOPO_PDL_LAUNCH();
  // what no solve changes: rows, inverse diagonals, the coarsest inverse
  for (int i = tid; i < P.vectors; i += nt) sm[i] = T(0);
  for (int l = 1; l < P.nlev; ++l) {
    const auto& L = P.lv[l];
    for (int n = tid; n < L.NX * L.NY; n += nt) {
      __align__(16) T st[SW];
      load_row(L.st + size_t(n) * SW, st);
      level_row<T, NC>(st);
      copy_row<T, SW>(st, sm + L.row + n * SW);
      for (int c = 0; c < NC; ++c) sm[L.di + NC * n + c] = L.dinv[NC * n + c];
    }
  }
  const auto& C = P.lv[P.nlev];
  const int m = C.NX * C.NY * NC;
  for (int i = tid; i < m * m; i += nt) sm[P.inv + i] = P.cinv[i];
  const auto& L0 = P.lv[0];
  const int n0 = tid < L0.NX * L0.NY ? tid : 0;
  TailNode<T, NC> N0;
  load_row(L0.st + size_t(n0) * SW, N0.st);
  level_row<T, NC>(N0.st);
  for (int c = 0; c < NC; ++c) N0.di[c] = L0.dinv[NC * n0 + c];
  TOPO_PDL_WAIT();
  long long* trace = TRACE && tid == 0 && blockIdx.x == 0 ? P.trace : nullptr;
  long long before = TRACE ? clock64() : 0;
  auto mark = [&]() {
    if (!TRACE || !trace) return;
    const long long now = clock64();
    *trace++ += now - before;
    before = now;
  };
  for (int c = 0; c < NC; ++c) N0.b[c] = b[NC * n0 + c];
  __syncthreads();  // the zeros are in place
  tail_down<T, NC, D>(P, 0, tid, sm, N0);
  mark();
  for (int l = 1; l < P.nlev; ++l) {
    TailNode<T, NC> N;
    tail_node(P, l, tid, sm, N);
    tail_down<T, NC, D>(P, l, tid, sm, N);
    mark();
  }
  if (tid < m) {  // the inverse is symmetric: column reads, one line per step
    T s = T(0);
    for (int k = 0; k < m; ++k) s = fma_t(sm[P.inv + k * m + tid], sm[C.b + k], s);
    const int n = tid / NC, j = n / C.NX, i = n - j * C.NX;
    sm[C.x + NC * ((j + 1) * (C.NX + 2) + i + 1) + tid % NC] = s;
  }
  __syncthreads();
  mark();
  for (int l = P.nlev - 1; l >= 1; --l) {
    TailNode<T, NC> N;
    tail_node(P, l, tid, sm, N);
    tail_up<T, NC, D>(P, l, tid, sm, N, x);
    mark();
  }
  tail_up<T, NC, D>(P, 0, tid, sm, N0, x);
  mark();
  if (TRACE && trace) *trace += 1;
}

template <class T, int NC>
struct CoarseChebDesc {
  P1Stencil<T, NC> S;  // the level's stencil (global memory; staged into shared)
  const T* dinv;
  int NX, nn;
  CoarseCheb<T> C;
};

// The whole Chebyshev solve of a truncated hierarchy's last level in one CTA
// (scalar levels, at most coarse_cheb_npt<T>() nodes per thread).  A
// thread keeps its nodes' stencil rows, inverse diagonal, residual and
// iterate in registers; only the direction, which the neighbours read, goes
// through shared memory (two buffers, one barrier per step).  A neighbour
// outside the lattice has a zero coupling, so its index is only clamped into
// the array.  A step is ~30 instructions per node (the arithmetic of
// CoarseChebNode::step in the stencil's difference form).
// nodes per thread: what the registers of a 1024-thread block hold without spilling
template <class T>
constexpr int coarse_cheb_npt() {
  return sizeof(T) == 4 ? 3 : 1;
}
// most nodes of the level: an FP64 step of a block issues at two products a clock, so above
// 512 nodes a level's own sweeps over all SMs cost less (861 nodes: 37 us)
template <class T>
constexpr size_t coarse_cheb_nodes() {
  return sizeof(T) == 4 ? size_t(kCoarseThreads) * coarse_cheb_npt<T>() : 512;
}

template <class T>
__global__ void __launch_bounds__(kCoarseThreads)
    k_coarse_cheb(const CoarseChebDesc<T, 1>* D, const T* b, T* x_out) {
  TOPO_PDL_LAUNCH();
  constexpr int NP = coarse_cheb_npt<T>(), SW = StencilLayout<1>::stride;
  extern __shared__ __align__(16) unsigned char cc_raw[];
  T* d0 = reinterpret_cast<T*>(cc_raw);
  const int tid = threadIdx.x, nt = blockDim.x;
  const int nn = D->nn, NX = D->NX;
  T* d1 = d0 + nn;
  __shared__ CoarseCheb<T> C;
  if (tid == 0) C = D->C;
  const T* sg = D->S.s;
  b += blockIdx.x * size_t(nn);
  x_out += blockIdx.x * size_t(nn);
  T st[NP][7], dv[NP], r[NP], x[NP];
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    const int n = tid + q * nt;
    const bool on = n < nn;
#pragma unroll
    for (int k = 0; k < 7; ++k) st[q][k] = on ? sg[size_t(n) * SW + k] : T(0);
    if constexpr (sizeof(T) == 8) {  // plain rows for FP64 (level_row)
#pragma unroll
      for (int k = 1; k < 7; ++k) st[q][0] -= st[q][k];
    }
    dv[q] = on ? D->dinv[n] : T(0);
  }
  __syncthreads();
  TOPO_PDL_WAIT();  // the rows above are fixed during a solve
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    const int n = tid + q * nt;
    const bool on = n < nn;
    r[q] = on ? b[n] : T(0);
    x[q] = T(0);
    if (on) d0[n] = C.c0 * dv[q] * r[q];
  }
  __syncthreads();
  T* dc = d0;
  T* dn = d1;
  const int deg = C.deg;
  for (int k = 0; k + 1 < deg; ++k) {
    const T c1 = C.c1[k], c2 = C.c2[k];
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      const int n = tid + q * nt;
      if (n < nn) {
        const T dn0 = dc[n];
        T t = st[q][0] * dn0;
#pragma unroll
        for (int e = 1; e < 7; ++e) {
          const int m = min(max(n + st_da(e) + st_db(e) * NX, 0), nn - 1);
          t += st[q][e] * (sizeof(T) == 8 ? dc[m] : dc[m] - dn0);
        }
        x[q] += dn0;
        r[q] -= t;
        dn[n] = c1 * dn0 + c2 * dv[q] * r[q];
      }
    }
    __syncthreads();
    T* tmp = dc;
    dc = dn;
    dn = tmp;
  }
#pragma unroll
  for (int q = 0; q < NP; ++q) {
    const int n = tid + q * nt;
    if (n < nn) x_out[n] = x[q] + dc[n];
  }
}

// ---------------------------------------------------------------------------
// host helpers
// ---------------------------------------------------------------------------
inline int device_sms() {
  static int cached[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (!cached[dev]) {
    int n = 0;
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    cached[dev] = n > 0 ? n : 1;
  }
  return cached[dev];
}

// Kernels of the solve chain are launched with programmatic stream
// serialization (they begin with TOPO_PDL_ENTRY): a launch overlaps the
// predecessor's drain instead of following its completion.  TOPO_PDL=0
// launches them plainly.
inline bool pdl_enabled() {
  static const bool on = [] {
    const char* e = std::getenv("TOPO_PDL");
    return !(e && e[0] == '0');
  }();
  return on;
}

template <class... KP, class... A>
inline void launch_pdl(void (*k)(KP...), dim3 g, dim3 b, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = g;
  cfg.blockDim = b;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  cudaLaunchKernelEx(&cfg, k, std::forward<A>(args)...);
}

// resident blocks per SM of a march kernel at P2M_THREADS threads (its
// registers decide: the grid is sized to one wave of them)
template <class K>
inline int march_blocks_per_sm(K kernel) {
  int b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, P2M_THREADS, 0) != cudaSuccess) {
    (void)cudaGetLastError();
    b = 0;
  }
  return b > 0 ? b : 1;
}

template <class T, int MODE>
inline int p2_march_bps() {
  static const int b = march_blocks_per_sm(k_p2_march<T, MODE>);
  return b;
}

template <class T, int NC, int MODE>
inline int p1_march_bps() {
  static const int b = march_blocks_per_sm(k_p1_march<T, NC, MODE>);
  return b;
}

// seg_force > 0: that segment length; else the tuned one for `family` (when tuned), else
// the one-wave rule
inline dim3 march_grid(int nx, int ny, int blocks_per_sm, int& seg, int family = -1, int seg_force = 0) {
  const int tuned = seg_force > 0 ? seg_force : (family >= 0 ? tuned_segment(family, nx, ny) : 0);
  seg = tuned > 0 ? std::min(tuned, ny) : p2_march_segment(nx, ny, device_sms(), blocks_per_sm);
  const int nseg = (ny + seg - 1) / seg;
  return dim3((nx + 1 + P2M_OWN - 1) / P2M_OWN, (nseg + P2M_WARPS - 1) / P2M_WARPS);
}

// The grid of a P2 launch: its short form (seg = kRowsSegment) up to three blocks per SM (one wave
// in FP32), else the march.  The rule looks at sizes only: the two forms add a node row's sums in a
// different order, and which one runs must not depend on a timing.
// Short form against the march of its best segment, us: 80x40 Apply 5.8 / 6.6, First 6.0 / 6.7,
// Res 4.1 / 5.2; 320x160 (440 blocks) 7.5 / 8.1, 6.7 / 7.4, 4.9 / 6.0; 303x101 pair-of-FP32 13.6 /
// 44.4; FP64 160x80 18.1 / 25.4, 22.0 / 29.4, 18.0 / 24.5; 1000x500 34.0 / 24.3, 34.0 / 26.4,
// 17.4 / 16.6.
inline bool p2_short_form(int nx, int ny) {
  const long blocks = long((nx + 1 + P2M_OWN - 1) / P2M_OWN) * ((ny + P2R_ROWS - 1) / P2R_ROWS);
  return blocks <= 3l * device_sms();
}
inline dim3 p2_grid(int nx, int ny, int blocks_per_sm, int& seg, int family = -1, int seg_force = 0) {
  if (seg_force > 0 || !p2_short_form(nx, ny)) return march_grid(nx, ny, blocks_per_sm, seg, family, seg_force);
  seg = kRowsSegment;
  return dim3((nx + 1 + P2M_OWN - 1) / P2M_OWN, (ny + P2R_ROWS - 1) / P2R_ROWS);
}

// occupancy queries happen outside any stream capture
template <class T>
inline void prime_march_occupancy() {
  (void)p2_march_bps<T, kP2Apply>();
  (void)p2_march_bps<T, kP2Diag>();
  (void)p2_march_bps<T, kP2Pre>();
  (void)p2_march_bps<T, kP2Res>();
  (void)p2_march_bps<T, kP2First>();
  (void)p2_march_bps<T, kP2Post2>();
  (void)p1_march_bps<T, 1, kP2Apply>();
  if constexpr (sizeof(T) == 8) {  // (FP32 levels are smoothed by the sweeps)
    (void)p1_march_bps<T, 2, kP2Apply>();
    (void)p1_march_bps<T, 1, kP2Pre>();
    (void)p1_march_bps<T, 1, kP2Res>();
    (void)p1_march_bps<T, 1, kP2First>();
    (void)p1_march_bps<T, 1, kP2Post2>();
    (void)p1_march_bps<T, 2, kP2Pre>();
    (void)p1_march_bps<T, 2, kP2Res>();
    (void)p1_march_bps<T, 2, kP2First>();
    (void)p1_march_bps<T, 2, kP2Post2>();
  }
}

// Kernel-clock names and algorithmic bytes of one launch (topo_kclock.h).  A mode
// reads and writes whole level vectors: `vecs` of them, each of n values.
inline const char* mode_name(int mode) {
  switch (mode) {
    case kP2Apply: return "Apply";
    case kP2Diag: return "Diag";
    case kP2Pre: return "Pre";
    case kP2Res: return "Res";
    case kP2First: return "First";
    default: return "Post2";
  }
}
template <class T>
inline const char* p2_family(int mode) {
  static const char* f32[6] = {"P2 march FP32 Apply", "P2 march FP32 Diag", "P2 march FP32 Pre",
                               "P2 march FP32 Res", "P2 march FP32 First", "P2 march FP32 Post2"};
  static const char* f64[6] = {"P2 march FP64 Apply", "P2 march FP64 Diag", "P2 march FP64 Pre",
                               "P2 march FP64 Res", "P2 march FP64 First", "P2 march FP64 Post2"};
  return (sizeof(T) == 4 ? f32 : f64)[mode];
}
// vectors of the level a smoothing or operator mode moves: operand(s) read, results written
// (P2: Pre reads b, D^-1 and writes x; First also writes w; Post2 reads d, w, D^-1 (+ b when
// it reduces r.r, r.z); P1 modes keep r between steps)
inline int mode_vectors(int mode, bool p2, bool fused_rz) {
  switch (mode) {
    case kP2Apply: return 2;
    case kP2Diag: return 1;
    case kP2Pre: return 3;
    case kP2Res: return 3;
    case kP2First: return 5;
    default: return p2 ? (fused_rz ? 5 : 4) : 5;
  }
}

template <class T, int MODE>
inline void launch_p2_mode(const P2Params<T>& P, const T* xi, const P2Io<T>& io, cudaStream_t s, int seg_force = 0) {
  int seg = 0;
  const dim3 g = p2_grid(P.nx, P.ny, p2_march_bps<T, MODE>(), seg, march_family(true, sizeof(T), 2), seg_force);
  const double n = 2.0 * (2 * P.nx + 1) * (2 * P.ny + 1), nv = double(P.nx + 1) * (P.ny + 1);
  // the design (one value per vertex) plus, for First, the coarse correction (2 per vertex)
  const double bytes = (mode_vectors(MODE, true, io.fuse == kFuseRZ) * n + nv + (MODE == kP2First ? 2 * nv : 0)) *
                       sizeof(T);
  KClock kc(s, p2_family<T>(MODE), 0, bytes);
  if (seg == kRowsSegment) launch_pdl(k_p2_rows<T, MODE>, g, P2R_THREADS, 0, s, P, xi, io);
  else launch_pdl(k_p2_march<T, MODE>, g, P2M_THREADS, 0, s, P, xi, io, seg);
}

template <class T>
inline void launch_p2_tile(const P2Params<T>& P, const T* xi, const P2Io<T>& io, cudaStream_t s) {
  switch (io.mode) {
    case kP2Apply: launch_p2_mode<T, kP2Apply>(P, xi, io, s); break;
    case kP2Diag: launch_p2_mode<T, kP2Diag>(P, xi, io, s); break;
    case kP2Pre: launch_p2_mode<T, kP2Pre>(P, xi, io, s); break;
    case kP2Res: launch_p2_mode<T, kP2Res>(P, xi, io, s); break;
    case kP2First: launch_p2_mode<T, kP2First>(P, xi, io, s); break;
    default: launch_p2_mode<T, kP2Post2>(P, xi, io, s); break;
  }
}

template <class T, int NC, int MODE>
inline void launch_p1_mode(const P1Params<T, NC>& P, const P1Io<T>& io, cudaStream_t s, int seg_force = 0) {
  int seg = 0;
  const dim3 g = march_grid(P.nx, P.ny, p1_march_bps<T, NC, MODE>(), seg, march_family(false, sizeof(T), NC), seg_force);
  static const char* fam[6] = {"P1 march Apply", "P1 march Diag", "P1 march Pre", "P1 march Res", "P1 march First",
                               "P1 march Post2"};
  const double n = double(NC) * (P.nx + 1) * (P.ny + 1), ntri = 2.0 * P.nx * P.ny;
  const double bytes = (mode_vectors(MODE, false, false) * n + ntri * ((P.kK ? 1 : 0) + (P.kM ? 1 : 0))) * sizeof(T);
  KClock kc(s, fam[MODE], 1, bytes);
  launch_pdl(k_p1_march<T, NC, MODE>, g, P2M_THREADS, 0, s, P, io, seg);
}

template <class T, int NC>
inline void launch_p1_march(const P1Params<T, NC>& P, const P1Io<T>& io, cudaStream_t s) {
  switch (io.mode) {
    case kP2Apply: launch_p1_mode<T, NC, kP2Apply>(P, io, s); break;
    case kP2Pre: launch_p1_mode<T, NC, kP2Pre>(P, io, s); break;
    case kP2Res: launch_p1_mode<T, NC, kP2Res>(P, io, s); break;
    case kP2First: launch_p1_mode<T, NC, kP2First>(P, io, s); break;
    default: launch_p1_mode<T, NC, kP2Post2>(P, io, s); break;
  }
}

template <class T>
inline void launch_p2_apply(const P2Params<T>& P, const T* xi, const T* x, T* y, cudaStream_t s) {
  P2Io<T> io;
  std::memset(&io, 0, sizeof(io));
  io.mode = kP2Apply;
  io.u = x;
  io.y = y;
  launch_p2_tile<T>(P, xi, io, s);
}

// y = A x with the pair-of-FP32 operator: x, y FP64, P.rmass the mass matrices as
// (hi, lo) pairs (the design is not read)
inline void launch_p2_apply_dd(const P2Params<dd>& P, const double* x, double* y, cudaStream_t s) {
  P2Io<dd> io;
  std::memset(&io, 0, sizeof(io));
  io.mode = kP2Apply;
  io.u = reinterpret_cast<const dd*>(x);
  io.y = reinterpret_cast<dd*>(y);
  int seg = 0;
  const dim3 g = p2_grid(P.nx, P.ny, p2_march_bps<dd, kP2Apply>(), seg);
  // x read and y written in FP64, the mass matrices (12 pairs per cell)
  const double n = 2.0 * (2 * P.nx + 1) * (2 * P.ny + 1), nc = double(P.nx) * P.ny;
  KClock kc(s, "P2 march pair-of-FP32 Apply", 0, 2.0 * n * 8.0 + 12.0 * nc * 8.0);
  if (seg == kRowsSegment)
    launch_pdl(k_p2_rows<dd, kP2Apply>, g, P2R_THREADS, 0, s, P, static_cast<const dd*>(nullptr), io);
  else
    launch_pdl(k_p2_march<dd, kP2Apply>, g, P2M_THREADS, 0, s, P, static_cast<const dd*>(nullptr), io, seg);
}

template <class T, int NC>
inline P1Params<T, NC> make_p1(const LevelSpec& L, const ElemRefs& R, const T* kK, const T* kM) {
  P1Params<T, NC> P;
  std::memset(&P, 0, sizeof(P));
  P.nx = L.nx;
  P.ny = L.ny;
  P.dir = L.dir;
  for (int o = 0; o < 2; ++o) {
    for (int a = 0; a < 3 * NC; ++a)
      for (int b = 0; b < 3 * NC; ++b) P.K[o][a][b] = T(NC == 2 ? R.K2[o][a][b] : R.K1[o][a][b]);
    for (int a = 0; a < 3; ++a)
      for (int b = 0; b < 3; ++b) P.Mm[o][a][b] = T(R.M1[o][a][b]);
  }
  P.kK = kK;
  P.kM = kM;
  P.kK_c = T(0);
  P.kM_c = T(0);
  return P;
}

static inline Transfer make_transfer(const LevelSpec& f, const LevelSpec& c) {
  Transfer X;
  X.NXf = f.NX;
  X.NYf = f.NY;
  X.NXc = c.NX;
  X.NYc = c.NY;
  X.dirf = f.dir;
  X.dirc = c.dir;
  return X;
}

template <class T, int NC>
inline LevelSweep<T, NC> level_sweep(const LevelSpec& S, const Transfer& X, const T* st, const T* inner, const T* dinv,
                                     const T* cheb) {
  LevelSweep<T, NC> P;
  std::memset(&P, 0, sizeof(P));
  P.NX = S.NX;
  P.NY = S.NY;
  P.NXc = X.NXc;
  P.NYc = X.NYc;
  P.cx = kSweepTileX;
  P.cy = kSweepTileY;
  if (sizeof(T) == 8) {
    // FP64: a block's time is its warps' (the SM's FP64 pipe takes two products a clock), so
    // the tile is the one whose waves of blocks hold the fewest warps per SM
    const int tiles[][2] = {{10, 4}, {9, 3}, {6, 4}, {6, 3}, {4, 3}, {6, 2}, {4, 2}, {3, 2}, {2, 2}, {2, 1}};
    int best = 1 << 30;
    for (const auto& t : tiles) {
      const int blocks = ((X.NXc + t[0] - 1) / t[0]) * ((X.NYc + t[1] - 1) / t[1]), sms = device_sms();
      const int warps = ((2 * t[0] + 3) * (2 * t[1] + 3) + 31) / 32, cost = (blocks + sms - 1) / sms * warps;
      if (cost < best) {
        best = cost;
        P.cx = t[0];
        P.cy = t[1];
      }
    }
  }
  P.st = st;
  P.inner = inner;
  P.dinv = dinv;
  P.cheb = cheb;
  P.dirf = X.dirf;
  P.dirc = X.dirc;
  return P;
}

// ---------------------------------------------------------------------------
// graph-resident CG scalars
// ---------------------------------------------------------------------------
// x += alpha p ; r -= alpha q with alpha = rz / pq read from device memory
// (evaluated once per block: an FP64 division per thread is not free here)
// x in T or FP64 (TX = double: the product of two FP32 numbers is exact in FP64)
// r -= alpha q with alpha = rz / pq; block 0 records the alpha it applied
// (the solution update happens in k_pcg_p, which reads p anyway)
template <class T>
__global__ void k_pcg_r(T* r, const T* q, PcgDev* dv, size_t n) {
  TOPO_PDL_ENTRY();
  __shared__ T alpha_s;
  __shared__ bool ok_s;
  // the first values are on their way while thread 0 divides
  const size_t step = size_t(gridDim.x) * blockDim.x;
  size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  T ri = T(0), qi = T(0);
  if (i < n) {
    ri = r[i];
    qi = q[i];
  }
  if (threadIdx.x == 0) {
    const double pq = dv->pq;
    ok_s = (pq > 0.0) && isfinite(pq);
    alpha_s = ok_s ? T(dv->rz / pq) : T(0);
    if (blockIdx.x == 0) dv->alpha = double(alpha_s);
  }
  __syncthreads();
  if (!ok_s) return;
  const T alpha = alpha_s;
  if (i < n) r[i] = ri - alpha * qi;
  for (i += step; i < n; i += step) r[i] -= alpha * q[i];
}

// x += alpha p (x in T or FP64: the product of two FP32 numbers is exact in
// FP64), then p = z + beta p
template <class T, class TX>
__global__ void k_pcg_p(T* p, const T* z, TX* x, const PcgDev* dv, size_t n) {
  TOPO_PDL_ENTRY();
  const T beta = T(dv->beta), alpha = T(dv->alpha);
  TOPO_GRID_STRIDE(i, n) {
    const T pi = p[i], zi = z[i];
    const TX xi = x[i];
    x[i] = xi + TX(alpha) * TX(pi);
    p[i] = zi + beta * pi;
  }
}

// after the prologue: decide whether the loop runs at all.  On entry dv->tol2
// holds rtol^2 and dv->maxit the iteration cap (both written by the host).
static __global__ void k_pcg_start(PcgDev* dv, cudaGraphConditionalHandle h, int use_cond) {
  TOPO_PDL_ENTRY();
  const double bb = dv->bb, rr = dv->rr;
  dv->tol2 = dv->tol2 * bb;
  dv->it = 0;
  dv->relres = bb > 0 ? sqrt(rr / bb) : 0.0;
  int st = 1;
  if (!isfinite(bb) || !isfinite(rr) || !isfinite(dv->rz)) st = 4;
  else if (bb == 0.0) st = 5;
  else if (rr <= dv->tol2) st = 0;
  dv->status = st;
  if (use_cond) cudaGraphSetConditional(h, st == 1 ? 1u : 0u);
}

// end of one iteration: convergence / cap / breakdown test and beta
static __global__ void k_pcg_check(PcgDev* dv, cudaGraphConditionalHandle h, int use_cond) {
  TOPO_PDL_ENTRY();
  pcg_check_dev(dv, h, use_cond);
}

// ---------------------------------------------------------------------------
// MG<T>
// ---------------------------------------------------------------------------
template <class T>
MG<T>::~MG() {
  for (auto& g : graph_)
    if (g.exec) cudaGraphExecDestroy(g.exec);
  for (auto c : cap_)
    if (c) cudaStreamDestroy(c);
  for (auto e : ev_)
    if (e) cudaEventDestroy(e);
  if (hdev_) cudaFreeHost(hdev_);
}

template <class T>
void MG<T>::init(const std::vector<LevelSpec>& specs, const ElemRefs* refs, double lmbda, double mu,
                 Arena& arena, Reducer* red) {
  specs_ = specs;
  refs_ = refs;
  lmbda_ = lmbda;
  mu_ = mu;
  red_ = red;
  sms_ = red->sms;
  prime_march_occupancy<T>();
  if (const char* e = std::getenv("TOPO_POWER_WARM")) {  // warm-started power-iteration steps
    const int v = std::atoi(e);
    if (v >= 1 && v <= 50) power_iters_warm = v;
  }
  lv_.assign(specs.size(), Lev{});
  for (size_t l = 0; l < specs.size(); ++l) {
    const size_t n = specs[l].ndof(), nb = n * batch;
    Lev& v = lv_[l];
    if (l > 0) {
      v.x = arena.alloc_n<T>(nb);
      v.b = arena.alloc_n<T>(nb);
    }
    v.r = arena.alloc_n<T>(n);
    v.d = arena.alloc_n<T>(n);
    v.t = arena.alloc_n<T>(n);
    v.x2 = arena.alloc_n<T>(nb);
    v.diag = arena.alloc_n<T>(n);
    v.dinv = arena.alloc_n<T>(n);
    if (!specs[l].p2) {
      v.kK = arena.alloc_n<T>(specs[l].ntri());
      if (specs[l].NC == 1) v.kM = arena.alloc_n<T>(specs[l].ntri());
      if (specs[l].nn() <= stencil_max_nodes(specs[l].NC))
        v.st = arena.alloc_n<T>(specs[l].nn() * (specs[l].NC == 2 ? StencilLayout<2>::stride : StencilLayout<1>::stride));
    }
  }
  const size_t n0 = specs[0].ndof();
  for (int k = 0; k < kScratch; ++k) pcg_[k] = arena.alloc_n<T>(n0);
  if (fp64_solution) xacc_ = arena.alloc_n<double>(n0);
  if (specs[0].p2) pw_ = arena.alloc_n<T>(n0);  // power-iteration vector kept between set-ups
  const int nc = int(specs.back().ndof());
  cinv_ = arena.alloc_n<T>(size_t(nc) * nc);
  cstat_ = arena.alloc_n<int>(1);
  cheb_ = arena.alloc_n<T>(8 * specs.size());
  dev_ = arena.alloc_n<PcgDev>(1);
  if (!hdev_) cudaMallocHost(&hdev_, sizeof(PcgDev));
  for (auto& c : cap_)
    if (!c) cudaStreamCreateWithFlags(&c, cudaStreamNonBlocking);
  for (auto& e : ev_)
    if (!e) cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
  graph_valid_ = false;
  build_tail(arena);
  cc_buf_ = arena.alloc(sizeof(CoarseChebDesc<T, 1>));
  inner_buf_ = arena.alloc_n<T>(specs.size() * StencilLayout<1>::stride);
}

// Levels with a mass term (the filter), no clamped nodes and the same stencil
// row at every interior node (constant coefficients on the uniform lattice,
// checked on the rows themselves) read that row once instead of per node.
template <class T>
void MG<T>::detect_uniform_levels(cudaStream_t s) {
  const int L = levels();
  for (int l = 0; l < L; ++l) {
    const LevelSpec& S = specs_[l];
    Lev& v = lv_[l];
    v.inner = nullptr;
    if (S.p2 || S.NC != 1 || !v.st || !kM64_[l] || !inner_buf_) continue;
    const Dir& d = S.dir;
    if (d.x_lo || d.y_lo || d.npts || d.x_hi_from < S.NX || d.y_hi_from < S.NY || S.NX < 3 || S.NY < 3) continue;
    constexpr int SW = StencilLayout<1>::stride;
    std::vector<T> st(S.nn() * SW);
    if (cudaMemcpyAsync(st.data(), v.st, st.size() * sizeof(T), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess) {
      cudaGetLastError();
      return;
    }
    const T* ref = st.data() + (size_t(1) * S.NX + 1) * SW;
    bool same = true;
    for (int b = 1; same && b + 1 < S.NY; ++b)
      for (int a = 1; same && a + 1 < S.NX; ++a)
        same = std::memcmp(st.data() + (size_t(b) * S.NX + a) * SW, ref, SW * sizeof(T)) == 0;
    if (!same) continue;
    T* dst = inner_buf_ + size_t(l) * SW;
    // on s: the kernels that read the row run there (a pageable copy is staged before
    // the call returns, so `st` may go out of scope)
    if (cudaMemcpyAsync(dst, ref, SW * sizeof(T), cudaMemcpyHostToDevice, s) != cudaSuccess) {
      cudaGetLastError();
      return;
    }
    v.inner = dst;
  }
  invalidate();
}

// Picks the truncation level (see CoarseCheb): the finest level l >= 1 with a
// scalar assembled stencil that fits one CTA's shared memory and whose Dinv A
// spectrum -- bounded element by element from the coefficient ratios kK/kM
// of the level's triangles -- needs at most coarse_cheb_max_degree steps for
// a residual reduction of 1e-2.  Levels past it are no longer visited.
template <class T>
void MG<T>::select_coarse_cheb(cudaStream_t s) {
  const int prev = cheb_coarse_;
  cheb_coarse_ = -1;
  cc_desc_ = nullptr;
  coarse_cheb_deg = 0;
  const int L = levels();
  for (int l = 1; use_coarse_cheb && cc_buf_ && l < L; ++l) {
    const LevelSpec& S = specs_[l];
    if (S.p2 || S.NC != 1 || !lv_[l].st || !kK64_[l] || !kM64_[l]) continue;
    const size_t smem = 2 * S.nn() * sizeof(T);  // the two direction buffers
    if (S.nn() > coarse_cheb_nodes<T>() || smem > kCoarseSharedBudget) continue;
    const size_t nt = S.ntri();
    std::vector<double> kk(nt), km(nt);
    if (cudaMemcpyAsync(kk.data(), kK64_[l], nt * sizeof(double), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaMemcpyAsync(km.data(), kM64_[l], nt * sizeof(double), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess) {
      cudaGetLastError();
      return;
    }
    double tmin = 1e300, tmax = 0.0;
    bool ok = nt > 0;
    for (size_t t = 0; t < nt && ok; ++t) {
      if (!(km[t] > 0.0) || !(kk[t] >= 0.0) || !std::isfinite(kk[t] / km[t])) ok = false;
      else {
        tmin = std::min(tmin, kk[t] / km[t]);
        tmax = std::max(tmax, kk[t] / km[t]);
      }
    }
    if (!ok) continue;
    double lo, hi;
    const int deg = coarse_cheb_plan(refs_[l], tmin, tmax, 1e-2, lo, hi);
    if (deg > coarse_cheb_max_degree || deg > kCoarseChebMax) continue;
    CoarseChebDesc<T, 1> h;
    std::memset(&h, 0, sizeof(h));
    h.S = P1Stencil<T, 1>{S.nx, S.ny, S.dir, lv_[l].st};
    h.dinv = lv_[l].dinv;
    h.NX = S.NX;
    h.nn = int(S.nn());
    double c0, c1[kCoarseChebMax], c2[kCoarseChebMax];
    coarse_cheb_coefficients(lo, hi, deg, c0, c1, c2);
    h.C.deg = deg;
    h.C.c0 = T(c0);
    for (int k = 0; k + 1 < deg; ++k) {
      h.C.c1[k] = T(c1[k]);
      h.C.c2[k] = T(c2[k]);
    }
    const int limit = int(kCoarseSharedBudget);
    if (cudaMemcpyAsync(cc_buf_, &h, sizeof(h), cudaMemcpyHostToDevice, s) != cudaSuccess ||
        cudaFuncSetAttribute(k_coarse_cheb<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, limit) != cudaSuccess) {
      cudaGetLastError();
      return;
    }
    cheb_coarse_ = l;
    cc_desc_ = cc_buf_;
    cc_smem_ = smem;
    coarse_cheb_deg = deg;
    break;
  }
  if (cheb_coarse_ != prev) invalidate();
}

// Chooses the levels of k_level_tail (FP32): from the first level with at most kTailNodes
// nodes (never level 0) whose shared memory fits, down to the coarsest.
template <class T>
void MG<T>::build_tail(Arena& arena) {
  tail_ = -1;
  const int L = levels();
  auto plan = [&](auto& P, int first) {
    std::memset(&P, 0, sizeof(P));
    P.nlev = L - 1 - first;
    P.cinv = cinv_;
    for (int l = first; l < L; ++l) {
      auto& d = P.lv[l - first];
      d.NX = specs_[l].NX;
      d.NY = specs_[l].NY;
      d.st = lv_[l].st;
      d.dinv = lv_[l].dinv;
      d.cheb = cheb_ + 8 * l;
      d.dir = specs_[l].dir;
    }
    P.plan();
    P.trace = tail_trace_;
    return size_t(P.shared) * sizeof(T) <= kTailShared;
  };
  if (sizeof(T) == 8) return;
  if (profile_levels) {
    tail_trace_ = static_cast<long long*>(arena.alloc(kTailPhases * sizeof(long long)));
    if (tail_trace_) cudaMemset(tail_trace_, 0, kTailPhases * sizeof(long long));
  }
  for (int l = std::max(1, L - 1 - kTailMaxLevels); l + 1 < L && tail_ < 0; ++l) {
    if (specs_[l].nn() > size_t(kTailNodes) || level_degree(l) != level_degree(L - 1)) continue;
    bool ok = true;
    for (int k = l; k < L; ++k) ok &= !specs_[k].p2 && lv_[k].st;
    if (ok && (specs_[l].NC == 2 ? plan(tail2_, l) : plan(tail1_, l))) tail_ = l;
  }
}

template <class T>
void MG<T>::apply(int l, const T* x, T* y, cudaStream_t s, bool op) {
  const LevelSpec& L = specs_[l];
  ++launches;
  if (L.p2) {
    launch_p2_apply<T>(op ? p2_op_ : p2_, xi_, x, y, s);
    return;
  }
  const dim3 g = row_grid(L.NX, L.NY);
  const Lev& v = lv_[l];
  // stencil operator: x read, y written, the stencil rows (unless one row is shared)
  const double abytes = 2.0 * L.ndof() * sizeof(T) +
                        (v.inner ? 0.0 : double((7 * L.NC * L.NC * sizeof(T) + 15) / 16 * 16) * L.nn());
  KClock kc(s, (v.st && stencils_ready_) ? "P1 stencil Apply" : "P1 march Apply (operator)", l,
            (v.st && stencils_ready_) ? abytes : 0.0);
  // (elasticity hierarchies start with a P2 level; nothing applies their P1 levels' operators)
  if (v.st && stencils_ready_) {
    launch_pdl(k_p1_apply<T, 1, P1Stencil<T, 1>>, g, kRowThreads, 0, s, P1Stencil<T, 1>{L.nx, L.ny, L.dir, v.st, v.inner}, x, y);
  } else {
    P1Io<T> io;
    std::memset(&io, 0, sizeof(io));
    io.mode = kP2Apply;
    io.u = x;
    io.y = y;
    launch_p1_mode<T, 1, kP2Apply>(make_p1<T, 1>(L, refs_[l], v.kK, v.kM), io, s);
  }
}

template <class T>
void MG<T>::diag_of(int l, T* d, cudaStream_t s) {
  const LevelSpec& L = specs_[l];
  ++launches;
  if (L.p2) {
    P2Io<T> io;
    std::memset(&io, 0, sizeof(io));
    io.mode = kP2Diag;
    io.y = d;
    launch_p2_tile<T>(p2_, xi_, io, s);
    return;
  }
  const dim3 g = row_grid(L.NX, L.NY);
  if (L.NC == 2) {
    auto P = make_p1<T, 2>(L, refs_[l], lv_[l].kK, nullptr);
    k_p1_diag<T, 2><<<g, kRowThreads, 0, s>>>(P, d);
  } else {
    auto P = make_p1<T, 1>(L, refs_[l], lv_[l].kK, lv_[l].kM);
    k_p1_diag<T, 1><<<g, kRowThreads, 0, s>>>(P, d);
  }
}

template <class T>
double MG<T>::dot(const T* a, const T* b, size_t n, cudaStream_t s) {
  ++launches;
  k_dot<T, T><<<red_->blocks_for(n), kVecThreads, 0, s>>>(a, b, n, red_->partials, red_->counter, red_->out);
  cudaMemcpyAsync(red_->host, red_->out, sizeof(double), cudaMemcpyDeviceToHost, s);
  cudaStreamSynchronize(s);
  return red_->host[0];
}

// Power iteration for lambda_max(D^-1 A) on level l (Rayleigh quotient
// x'Ax / x'Dx).  On the state hierarchy's level 0 the iterate is kept between
// set-ups: consecutive designs differ little, so a warm start needs fewer
// steps.  Normalisation happens on the device; one host read at the end.
template <class T>
double MG<T>::estimate_lmax(int l, cudaStream_t s) {
  const size_t n = specs_[l].ndof();
  const int g = vec_grid(n, sms_);
  Lev& v = lv_[l];
  const bool keep = (l == 0 && pw_);
  T* x = keep ? pw_ : v.r;
  T* y = v.d;
  const bool warm = keep && pw_ready_;
  const int iters = warm ? power_iters_warm : power_iters;
  if (!warm) {
    k_power_start<T><<<g, kVecThreads, 0, s>>>(x, n);
    launches += 1;
  }
  for (int it = 0; it < iters; ++it) {
    apply(l, x, y, s);
    k_mul<T><<<g, kVecThreads, 0, s>>>(x, v.dinv, y, n);
    launches += 1;
    if (it % 4 == 3 || it + 1 == iters) {  // rescale to unit length (on the device)
      k_dot<T, T><<<red_->blocks_for(n), kVecThreads, 0, s>>>(x, x, n, red_->partials, red_->counter, red_->out);
      k_scale_unit<T><<<g, kVecThreads, 0, s>>>(x, red_->out, n);
      launches += 2;
    }
  }
  apply(l, x, y, s);
  k_mul<T><<<g, kVecThreads, 0, s>>>(v.t, v.diag, x, n);
  k_dot2<T><<<red_->blocks_for(n), kVecThreads, 0, s>>>(x, y, x, v.t, n, red_->partials, red_->counter, red_->out);
  launches += 2;
  cudaMemcpyAsync(red_->host, red_->out, 2 * sizeof(double), cudaMemcpyDeviceToHost, s);
  cudaStreamSynchronize(s);
  const double num = red_->host[0], den = red_->host[1];
  double lam = (den > 0) ? num / den : 4.0;
  const bool ok = std::isfinite(lam) && lam > 0;
  if (!ok) lam = 4.0;
  if (keep) pw_ready_ = ok;  // a failed estimate restarts from the fixed start vector
  return lam;
}

template <class T>
int MG<T>::setup(cudaStream_t s) {
  const int L = levels();
  auto t_last = std::chrono::steady_clock::now();
  auto mark = [&](const char* what) {  // trace_setup: synchronised phase times
    if (!trace_setup) return;
    cudaStreamSynchronize(s);
    const auto now = std::chrono::steady_clock::now();
    std::fprintf(stderr, "[topo setup] %-22s %.3f ms\n", what, std::chrono::duration<double, std::milli>(now - t_last).count());
    t_last = now;
  };
  mark("(queued before)");
  // Three independent chains once the coefficient masters (written on s) are
  // ready: level 0's diagonal and eigenvalue estimate on s (the only user of
  // the shared reduction scratch); the P1 levels' coefficients, stencils and
  // diagonals on one owned stream; the coarsest inverse (one warp, long
  // latency) on the other.  s waits for both before it reads levels >= 1.
  cudaStream_t side = cap_[1], side2 = cap_[0];
  cudaEventRecord(ev_[0], s);
  cudaStreamWaitEvent(side, ev_[0], 0);
  cudaStreamWaitEvent(side2, ev_[0], 0);
  auto prep = [&](int l, cudaStream_t q) {
    const LevelSpec& S = specs_[l];
    Lev& v = lv_[l];
    if (!S.p2) {
      const int g = vec_grid(S.ntri(), sms_);
      k_convert<T, double><<<g, kVecThreads, 0, q>>>(v.kK, kK64_[l], 1.0, S.ntri());
      if (v.kM) k_convert<T, double><<<g, kVecThreads, 0, q>>>(v.kM, kM64_[l], 1.0, S.ntri());
      launches += v.kM ? 2 : 1;
      if (v.st) {
        const dim3 gr = row_grid(S.NX, S.NY);
        if (S.NC == 2) k_p1_stencil<T, 2><<<gr, kRowThreads, 0, q>>>(make_p1<T, 2>(S, refs_[l], v.kK, nullptr), v.st);
        else k_p1_stencil<T, 1><<<gr, kRowThreads, 0, q>>>(make_p1<T, 1>(S, refs_[l], v.kK, v.kM), v.st);
        launches += 1;
      }
    }
    stencils_ready_ = true;  // the operator of level l is chosen at launch time
    const size_t n = S.ndof();
    diag_of(l, v.diag, q);
    k_inverse<T><<<vec_grid(n, sms_), kVecThreads, 0, q>>>(v.dinv, v.diag, n);
    launches += 1;
  };
  const LevelSpec& C = specs_[L - 1];
  if (C.NC == 2)
    k_coarse_inverse<T, 2><<<1, 32, 0, side2>>>(C.nx, C.ny, C.dir, refs_[L - 1], kK64_[L - 1], nullptr, cinv_, cstat_);
  else
    k_coarse_inverse<T, 1><<<1, 32, 0, side2>>>(C.nx, C.ny, C.dir, refs_[L - 1], kK64_[L - 1], kM64_[L - 1], cinv_,
                                                cstat_);
  launches += 1;
  cudaEventRecord(ev_[2], side2);
  for (int l = 1; l < L; ++l) prep(l, side);
  cudaEventRecord(ev_[1], side);
  prep(0, s);
  mark("level 0 diagonal");
  std::vector<double> cc(8 * L, 0.0);
  auto bounds = [&](int l) {
    const LevelSpec& S = specs_[l];
    if (!S.p2 && S.NC == 2) {
      lv_[l].lmax = p1_elasticity_bound(refs_[l]);
      lv_[l].bound = true;
    } else if (!S.p2 && element_bounds) {
      lv_[l].lmax = p1_scalar_bound(refs_[l]);
      lv_[l].bound = true;
    } else {
      lv_[l].lmax = estimate_lmax(l, s);
      lv_[l].bound = false;
    }
    const int degree = level_degree(l);
    const double hi = (lv_[l].bound ? 1.0 : 1.1) * lv_[l].lmax;
    const double lo = (degree > 2 ? cheb_lo_deep : cheb_lo_frac) * lv_[l].lmax;
    const double theta = 0.5 * (hi + lo), delta = 0.5 * (hi - lo), sigma = theta / delta;
    double* c = cc.data() + 8 * l;
    c[0] = 1.0 / theta;
    double rho_old = 1.0 / sigma;
    for (int k = 1; k < degree; ++k) {
      const double rho_new = 1.0 / (2.0 * sigma - rho_old);
      c[2 * k - 1] = rho_new * rho_old;
      c[2 * k] = 2.0 * rho_new / delta;
      rho_old = rho_new;
    }
  };
  if (L > 1) bounds(0);
  mark("level 0 eigenvalue bound");
  cudaStreamWaitEvent(s, ev_[1], 0);
  if (!cc_selected_) {  // the coefficients of a hierarchy with a mass term do not change
    cudaStreamSynchronize(s);
    select_coarse_cheb(s);
    if (!element_bounds) detect_uniform_levels(s);
    cc_selected_ = true;
  }
  for (int l = 1; l + 1 < L; ++l) bounds(l);
  mark("levels >= 1 (side stream)");
  // stored in the levels' precision: the kernels use them without conversion
  // (an FP64 load and convert per node costs FP64-pipe time on this GPU)
  cheb_host_.assign(cc.begin(), cc.end());
  cudaMemcpyAsync(cheb_, cheb_host_.data(), cheb_host_.size() * sizeof(T), cudaMemcpyHostToDevice, s);
  cudaStreamWaitEvent(s, ev_[2], 0);
  int st = 0;
  cudaMemcpyAsync(&st, cstat_, sizeof(int), cudaMemcpyDeviceToHost, s);
  cudaError_t e = cudaStreamSynchronize(s);
  mark("coarse inverse");
  if (e != cudaSuccess) return -5;
  if (st) return -2;
  tune_marches(s);
  return cudaStreamSynchronize(s) == cudaSuccess ? 0 : -5;
}

template <class T>
void MG<T>::flush_level_profile() {
  if (prof_events_.empty()) return;
  cudaDeviceSynchronize();
  if (level_ms.size() < specs_.size()) {
    level_ms.assign(specs_.size(), 0.0);
    level_calls.assign(specs_.size(), 0);
  }
  for (auto& pe : prof_events_) {
    float ms = 0.f;
    cudaEventElapsedTime(&ms, pe.second.first, pe.second.second);
    level_ms[pe.first] += ms;
    level_calls[pe.first] += 1;
    cudaEventDestroy(pe.second.first);
    cudaEventDestroy(pe.second.second);
  }
  prof_events_.clear();
}

template <class T>
void MG<T>::tail_profile(std::vector<long long>& cycles) const {
  cycles.clear();
  if (!tail_trace_ || tail_ < 0) return;
  cycles.resize(2 * (levels() - 1 - tail_) + 2);
  if (cudaMemcpy(cycles.data(), tail_trace_, cycles.size() * sizeof(long long), cudaMemcpyDeviceToHost) != cudaSuccess)
    cycles.clear();
}

template <class T>
void MG<T>::vcycle_level(int l, const T* b, T* x, cudaStream_t s) {
  if (profile_levels && !use_graphs) {
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, s);
    prof_depth_ += 1;
    vcycle_level_body(l, b, x, s);
    prof_depth_ -= 1;
    cudaEventRecord(e1, s);
    prof_events_.push_back({l, {e0, e1}});
    if (prof_events_.size() > 4096) flush_level_profile();
    return;
  }
  vcycle_level_body(l, b, x, s);
}

// Both sweeps of level l with D Chebyshev steps, the coarser levels between them.
template <class T>
template <int NC, int D, class ROWS>
void MG<T>::sweep_level(int l, const ROWS& Q, const T* b, T* x, cudaStream_t s) {
  Lev& v = lv_[l];
  Lev& c = lv_[l + 1];
  const LevelSpec& S = specs_[l];
  const Transfer X = make_transfer(S, specs_[l + 1]);
  const double nf = double(S.nn()) * NC, ncrs = double(X.NXc) * X.NYc * NC;
  // the stencil row of every node (7 NC x NC blocks, padded to 16 bytes; one row where the
  // level shares it; the triangles' coefficients where the rows are built from them); down b, D^-1
  // read, x and the coarse residual written; up b, D^-1, x and the coarse correction read, x written
  const double row = !v.st ? double(S.ntri() * sizeof(T) * (NC == 1 ? 2 : 1))
                     : v.inner ? 0.0
                               : double((7 * NC * NC * sizeof(T) + 15) / 16 * 16) * double(S.nn());
  LevelSweep<T, NC> P = level_sweep<T, NC>(S, X, v.st, v.inner, v.dinv, cheb_ + 8 * l);
  if (sizeof(T) == 4) {
    P.cx = sweep_tile_x<ROWS, D>();
    P.cy = sweep_tile_y<ROWS, D>();
  }
  const dim3 g((X.NXc + P.cx - 1) / P.cx, (X.NYc + P.cy - 1) / P.cy, batch);
  const int dw = down_w<D>(P), dh = down_h<D>(P), uw = up_w<D>(P), uh = up_h<D>(P);
  {
    KClock kc(s, "P1 level down", l, row + (3 * nf + ncrs) * sizeof(T));
    launch_pdl(k_level_down<T, NC, D, ROWS>, g, dim3(unsigned(dw * dh + 31) / 32 * 32),
               sweep_shared(dw, dh, NC) * sizeof(T), s, P, Q, b, v.x2, c.b);
  }
  vcycle_level(l + 1, c.b, c.x, s);
  {
    KClock kc(s, "P1 level up", l, row + (4 * nf + ncrs) * sizeof(T));
    launch_pdl(k_level_up<T, NC, D, ROWS>, g, dim3(unsigned(uw * uh + 31) / 32 * 32),
               sweep_shared(uw, uh, NC) * sizeof(T), s, P, Q, b, static_cast<const T*>(v.x2),
               static_cast<const T*>(c.x), x);
  }
  launches += 2;
}

template <class T>
template <int NC>
void MG<T>::sweep_level(int l, const T* b, T* x, cudaStream_t s) {
  // (the degrees in use: see level_degree)
  if constexpr (sizeof(T) == 4) {
    if (!lv_[l].st) {
      const P1Params<T, NC> Q = make_p1<T, NC>(specs_[l], refs_[l], lv_[l].kK, lv_[l].kM);
      if constexpr (NC == 2)
        if (level_degree(l) == kCoarseDegree) return sweep_level<NC, kCoarseDegree>(l, Q, b, x, s);
      return sweep_level<NC, 2>(l, Q, b, x, s);
    }
    if constexpr (NC == 2)
      if (level_degree(l) == kCoarseDegree) return sweep_level<NC, kCoarseDegree>(l, StoredRows{}, b, x, s);
  }
  sweep_level<NC, 2>(l, StoredRows{}, b, x, s);
}

template <class T>
template <int NC, int D>
void MG<T>::launch_tail(const TailSweep<T, NC>& P, int nodes, const T* b, T* x, cudaStream_t s) {
  const dim3 threads(unsigned(nodes + 31) / 32 * 32);
  if (P.trace) launch_pdl(k_level_tail<T, NC, D, true>, batch, threads, P.shared * sizeof(T), s, P, b, x);
  else launch_pdl(k_level_tail<T, NC, D, false>, batch, threads, P.shared * sizeof(T), s, P, b, x);
}

template <class T>
template <int NC>
void MG<T>::launch_tail(const TailSweep<T, NC>& P, int l, const T* b, T* x, cudaStream_t s) {
  const int nodes = int(specs_[l].nn());
  if constexpr (NC == 2)
    if (level_degree(l) == kCoarseDegree) return launch_tail<NC, kCoarseDegree>(P, nodes, b, x, s);
  launch_tail<NC, 2>(P, nodes, b, x, s);
}

// One V-cycle from level l down: Chebyshev steps (level_degree) from x = 0, restriction of the
// residual, coarse correction, the same steps again.
template <class T>
void MG<T>::vcycle_level_body(int l, const T* b, T* x, cudaStream_t s) {
  Lev& v = lv_[l];
  const int L = levels();
  const LevelSpec& S = specs_[l];
  if (l == cheb_coarse_ && cc_desc_) {
    KClock kc(s, "coarse Chebyshev (one CTA)", l, 0.0);
    launch_pdl(k_coarse_cheb<T>, batch, sizeof(T) == 4 ? kCoarseThreads : 512, cc_smem_, s, static_cast<const CoarseChebDesc<T, 1>*>(cc_desc_), b, x);
    ++launches;
    return;
  }
  if constexpr (sizeof(T) == 4) {
    if (l == tail_ && use_tail) {
      KClock kc(s, "V-cycle tail (one CTA)", l, 0.0);
      if (S.NC == 2) launch_tail<2>(tail2_, l, b, x, s);
      else launch_tail<1>(tail1_, l, b, x, s);
      ++launches;
      return;
    }
  }
  if (l == L - 1) {
    launch_pdl(k_dense_matvec<T>, batch, kDenseThreads, 0, s, static_cast<const T*>(cinv_), b, x, int(S.ndof()));
    ++launches;
    return;
  }
  SmoothBufs<T> B{b, v.dinv, x, v.x2, v.r, v.d, cheb_ + 8 * l};
  const Transfer X = make_transfer(S, specs_[l + 1]);
  Lev& c = lv_[l + 1];
  const dim3 gf = row_grid(S.NX, S.NY), gc = row_grid(X.NXc, X.NYc);
  if (S.p2) {
    P2Io<T> io;
    std::memset(&io, 0, sizeof(io));
    io.B = B;
    io.u = x;
    io.early = 1;  // (a solve's launches all follow the set-up's last synchronisation)
    io.mode = kP2Pre;
    launch_p2_tile<T>(p2_, xi_, io, s);
    io.mode = kP2Res;
    launch_p2_tile<T>(p2_, xi_, io, s);
    {
      KClock kc(s, "restriction", l, 2.0 * (double(S.nn()) + double(X.NXc) * X.NYc) * sizeof(T));
      launch_pdl(k_restrict<T, 2>, gc, kRowThreads, 0, s, X, static_cast<const T*>(v.r), c.b, static_cast<const T*>(nullptr));
    }
    launches += 3;
    vcycle_level(l + 1, c.b, c.x, s);
    io.mode = kP2First;  // adds the prolonged coarse correction to its operand on the fly
    io.xc = c.x;
    launch_p2_tile<T>(p2_, xi_, io, s);
    io.mode = kP2Post2;
    if (l == 0 && fuse_rz_) {  // the CG's r.r, r.z and test (see pcg_body)
      io.fuse = kFuseRZ;
      io.partials = red_->partials;
      io.counter = red_->counter;
      io.pcg = dev_;
      io.cond = fuse_cond_;
      io.use_cond = fuse_use_cond_;
    }
    launch_p2_tile<T>(p2_, xi_, io, s);
    launches += 2;
    return;
  }
  if (sizeof(T) == 4 || v.st) {
    if (S.NC == 2) sweep_level<2>(l, b, x, s);
    else sweep_level<1>(l, b, x, s);
    return;
  }
  // FP64 levels without a stencil: the column march (element products per cell; the ring that a
  // sweep's blocks recompute would cost FP64-pipe time)
  if constexpr (sizeof(T) == 8) {
    const double nf = double(S.nn()) * S.NC, ncrs = double(X.NXc) * X.NYc * S.NC;
    const double rbytes = (nf + ncrs) * sizeof(T), pbytes = (2 * nf + ncrs) * sizeof(T);
    auto run_march = [&](auto nc_tag, const auto& P) {
      constexpr int NC = decltype(nc_tag)::value;
      P1Io<T> io;
      std::memset(&io, 0, sizeof(io));
      io.B = B;
      io.u = x;
      io.mode = kP2Pre;
      launch_p1_march<T, NC>(P, io, s);
      io.mode = kP2Res;
      launch_p1_march<T, NC>(P, io, s);
      {
        KClock kc(s, "restriction", l, rbytes);
        launch_pdl(k_restrict<T, NC>, gc, kRowThreads, 0, s, X, static_cast<const T*>(v.r), c.b, static_cast<const T*>(nullptr));
      }
      launches += 3;
      vcycle_level(l + 1, c.b, c.x, s);
      { KClock kc(s, "prolongation", l, pbytes); launch_pdl(k_prolong_add<T, NC>, gf, kRowThreads, 0, s, X, static_cast<const T*>(c.x), x); }
      io.mode = kP2First;
      launch_p1_march<T, NC>(P, io, s);
      io.mode = kP2Post2;
      launch_p1_march<T, NC>(P, io, s);
      launches += 3;
    };
    if (S.NC == 2) run_march(std::integral_constant<int, 2>{}, make_p1<T, 2>(S, refs_[l], v.kK, nullptr));
    else run_march(std::integral_constant<int, 1>{}, make_p1<T, 1>(S, refs_[l], v.kK, v.kM));
  }
}

template <class T>
void MG<T>::vcycle(const T* b, T* x, cudaStream_t s) {
  vcycle_level(0, b, x, s);
}

// Autotuner of the column-march kernels' tile, the cell rows one warp marches:
// candidate segment lengths are timed on the Apply mode with CUDA events (R
// launches back to back per sample, best of two samples: the events resolve
// about 2 us) and the one-wave rule of p2_march_segment is kept unless a
// candidate is more than 5 % faster.  Once per kernel family and grid in the
// process, after set-up and before the first graph recording (graphs keep the
// segment they were recorded with).  Every segment length gives the same node
// values; only the grid, and with it the fused reductions' block partials, changes,
// so two processes may round a CG scalar differently (TOPO_AUTOTUNE=0 keeps the
// one-wave rule and with it bitwise reproducible runs).
template <class T>
void MG<T>::tune_marches(cudaStream_t s) {
  if (!autotune || !autotune_enabled()) return;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (cudaEventCreate(&e0) != cudaSuccess) return;
  if (cudaEventCreate(&e1) != cudaSuccess) {
    cudaEventDestroy(e0);
    return;
  }
  constexpr int R = 6;
  auto time_it = [&](const auto& launch) -> float {
    float best = 1e30f;
    for (int rep = 0; rep < 2; ++rep) {
      launch();  // warm
      cudaEventRecord(e0, s);
      for (int k = 0; k < R; ++k) launch();
      cudaEventRecord(e1, s);
      float ms = 0.f;
      if (cudaEventSynchronize(e1) != cudaSuccess || cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess) return 1e30f;
      best = std::min(best, ms / R);
    }
    return best;
  };
  // max_blocks > 0: a candidate whose grid exceeds it is skipped
  auto choose = [&](int family, int nx, int ny, int blocks_per_sm, size_t max_blocks, const auto& launch_with) {
    if (tuned_segment(family, nx, ny) > 0) return;
    // one tuner per key: a context set up concurrently for the same grid waits here and
    // then uses the same segment, so all contexts of a grid in the process agree
    std::lock_guard<std::recursive_mutex> lock(device_lock());
    if (tuned_segment(family, nx, ny) > 0) return;
    const int heur = p2_march_segment(nx, ny, device_sms(), blocks_per_sm);
    const float t_heur = time_it([&] { launch_with(heur); });
    int best = heur;
    float t_best = t_heur;
    for (int c : {1, 2, 3, 4, 6, 8, 12}) {
      if (c == heur || c > ny) continue;
      int sg = 0;
      const dim3 g = march_grid(nx, ny, blocks_per_sm, sg, -1, c);
      if (max_blocks && size_t(g.x) * g.y > max_blocks) continue;
      const float t = time_it([&] { launch_with(c); });
      if (t < t_best) {
        t_best = t;
        best = c;
      }
    }
    set_tuned_segment(family, nx, ny, t_best < 0.95f * t_heur ? best : heur);
  };
  const int L = levels();
  for (int l = 0; l < L; ++l) {
    const LevelSpec& S = specs_[l];
    Lev& v = lv_[l];
    if (l == tail_ && use_tail) break;  // the tail runs the rest
    if (l == cheb_coarse_ && cc_desc_) break;
    if (S.p2) {
      if (p2_short_form(S.nx, S.ny)) continue;
      const size_t n = S.ndof();
      T *x = pcg_[8], *y = pcg_[9];
      cudaMemsetAsync(x, 0, n * sizeof(T), s);
      P2Io<T> io;
      std::memset(&io, 0, sizeof(io));
      io.mode = kP2Apply;
      io.u = x;
      io.y = y;
      // the fused CG reductions keep 2 partials per block in red_->blocks * 16 slots
      const size_t max_blocks = red_ ? size_t(red_->blocks) * 8 : 0;
      choose(march_family(true, sizeof(T), 2), S.nx, S.ny, p2_march_bps<T, kP2Apply>(), max_blocks,
             [&](int seg) { launch_p2_mode<T, kP2Apply>(p2_op_, xi_, io, s, seg); });
    } else if (!v.st && l + 1 < L && (sizeof(T) == 8 || S.NC == 1)) {
      // (FP32 elasticity levels run no march: the sweeps smooth them, their bound is the elements')
      T* x = l > 0 ? v.x : pcg_[8];  // level 0 works on its caller's vector and owns none
      cudaMemsetAsync(x, 0, S.ndof() * sizeof(T), s);
      P1Io<T> io;
      std::memset(&io, 0, sizeof(io));
      io.mode = kP2Apply;
      io.u = x;
      io.y = v.t;
      if (S.NC == 1) {
        const auto P = make_p1<T, 1>(S, refs_[l], v.kK, v.kM);
        choose(march_family(false, sizeof(T), 1), S.nx, S.ny, p1_march_bps<T, 1, kP2Apply>(), 0,
               [&](int seg) { launch_p1_mode<T, 1, kP2Apply>(P, io, s, seg); });
      } else if constexpr (sizeof(T) == 8) {
        const auto P = make_p1<T, 2>(S, refs_[l], v.kK, nullptr);
        choose(march_family(false, sizeof(T), 2), S.nx, S.ny, p1_march_bps<T, 2, kP2Apply>(), 0,
               [&](int seg) { launch_p1_mode<T, 2, kP2Apply>(P, io, s, seg); });
      }
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
}

// Records the CG solve into a graph: a prologue (initial residual, first
// preconditioned direction, start test) followed by a WHILE conditional node
// whose body is one CG iteration; the body's last kernel decides whether the
// loop continues, so the solve runs without host round trips.  The loop is
// bounded by maxit (checked on the device).  Recording happens on two streams
// owned by this object (capture is not possible on the legacy default stream);
// every graph call is checked and nothing is launched unless all succeeded.
template <class T>
void MG<T>::pcg_prologue(bool warm, cudaStream_t s) {
  const size_t n = specs_[0].ndof();
  const int g = vec_grid(n, sms_);
  T *r = pcg_[0], *z = pcg_[1], *p = pcg_[2], *q = pcg_[3], *bi = pcg_[5], *xi = pcg_[6];
  if (warm) {
    apply(0, xi, q, s, true);
    k_sub<T><<<g, kVecThreads, 0, s>>>(r, bi, q, n);
    // the FP64 solution starts exactly at the guess the residual belongs to
    if (xacc_) k_convert<double, T><<<g, kVecThreads, 0, s>>>(xacc_, xi, 1.0, n);
  } else {
    k_fill<T><<<g, kVecThreads, 0, s>>>(xi, T(0), n);
    if (xacc_) k_fill<double><<<g, kVecThreads, 0, s>>>(xacc_, 0.0, n);
    cudaMemcpyAsync(r, bi, n * sizeof(T), cudaMemcpyDeviceToDevice, s);
  }
  if (xacc_) launches += 1;
  k_dot<T, T><<<red_->blocks_for(n), kVecThreads, 0, s>>>(bi, bi, n, red_->partials, red_->counter, &dev_->bb);
  k_dot<T, T><<<red_->blocks_for(n), kVecThreads, 0, s>>>(r, r, n, red_->partials, red_->counter, &dev_->rr);
  vcycle(r, z, s);
  k_dot<T, T><<<red_->blocks_for(n), kVecThreads, 0, s>>>(r, z, n, red_->partials, red_->counter, &dev_->rz);
  cudaMemcpyAsync(p, z, n * sizeof(T), cudaMemcpyDeviceToDevice, s);
  launches += 5;
}

template <class T>
void MG<T>::pcg_xr(int g, cudaStream_t s) {
  const size_t n = specs_[0].ndof();
  T *r = pcg_[0], *q = pcg_[3];
  KClock kc(s, "CG r -= alpha q", 0, 3.0 * n * sizeof(T));
  launch_pdl(k_pcg_r<T>, g, kVecThreads, 0, s, r, static_cast<const T*>(q), dev_, n);
}

template <class T>
void MG<T>::pcg_p(int g, cudaStream_t s) {
  const size_t n = specs_[0].ndof();
  T *z = pcg_[1], *p = pcg_[2], *xi = pcg_[6];
  const PcgDev* dv = dev_;
  // p read and written, z read, x (FP64 when accumulated so) read and written
  KClock kc(s, "CG x += alpha p, p = z + beta p", 0, n * (3.0 * sizeof(T) + 2.0 * (xacc_ ? 8 : sizeof(T))));
  if (xacc_) launch_pdl(k_pcg_p<T, double>, g, kVecThreads, 0, s, p, static_cast<const T*>(z), xacc_, dv, n);
  else launch_pdl(k_pcg_p<T, T>, g, kVecThreads, 0, s, p, static_cast<const T*>(z), xi, dv, n);
}

template <class T>
void MG<T>::pcg_body(cudaStream_t s, cudaGraphConditionalHandle h, int use_cond) {
  const size_t n = specs_[0].ndof();
  const int g = vec_grid(n, sms_);
  T *r = pcg_[0], *z = pcg_[1], *p = pcg_[2], *q = pcg_[3];
  // both fused launches (operator and last post-smoothing) must fit the partial slots
  int seg = 0;
  const int fam = march_family(true, sizeof(T), 2);
  const dim3 ga = p2_grid(specs_[0].nx, specs_[0].ny, p2_march_bps<T, kP2Apply>(), seg, fam);
  const dim3 gp = p2_grid(specs_[0].nx, specs_[0].ny, p2_march_bps<T, kP2Post2>(), seg, fam);
  const size_t mblocks = std::max(size_t(ga.x) * ga.y, size_t(gp.x) * gp.y);
  if (specs_[0].p2 && mblocks * 2 <= size_t(red_->blocks) * 16) {
    // P2 level 0: p.q is reduced inside the operator launch, r.r / r.z and the
    // iteration's test inside the V-cycle's last post-smoothing launch
    P2Io<T> io;
    std::memset(&io, 0, sizeof(io));
    io.mode = kP2Apply;
    io.u = p;
    io.y = q;
    io.fuse = kFusePQ;
    io.early = 1;
    io.partials = red_->partials;
    io.counter = red_->counter;
    io.pcg = dev_;
    launch_p2_tile<T>(p2_op_, xi_, io, s);
    pcg_xr(g, s);
    fuse_rz_ = true;
    fuse_cond_ = (unsigned long long)h;
    fuse_use_cond_ = use_cond;
    vcycle(r, z, s);
    fuse_rz_ = false;
    pcg_p(g, s);
    launches += 3;
    return;
  }
  apply(0, p, q, s, true);
  {
    KClock kc(s, "CG dot p.q", 0, 2.0 * n * sizeof(T));
    launch_pdl(k_dot<T, T>, red_->blocks_for(n), kVecThreads, 0, s, static_cast<const T*>(p), static_cast<const T*>(q), n,
               red_->partials, red_->counter, &dev_->pq);
  }
  pcg_xr(g, s);
  vcycle(r, z, s);
  {
    KClock kc(s, "CG dots r.r, r.z", 0, 2.0 * n * sizeof(T));
    launch_pdl(k_dot2<T>, red_->blocks_for(n), kVecThreads, 0, s, static_cast<const T*>(r), static_cast<const T*>(r),
               static_cast<const T*>(r), static_cast<const T*>(z), n, red_->partials, red_->counter, &dev_->rr);
  }
  launch_pdl(k_pcg_check, 1, 1, 0, s, dev_, h, use_cond);
  pcg_p(g, s);
  launches += 5;
}

// Captures a solve on s, which must be capturing: the prologue, then a WHILE node (its body on
// sb) running the iterations.  l1, l2: the launch counter before and after the body.
template <class T>
bool MG<T>::record_solve(bool warm, cudaStream_t s, cudaStream_t sb, long long& l1, long long& l2) {
  bool ok = true;
  cudaGraphNode_t wnode = nullptr;
  pcg_prologue(warm, s);
  cudaStreamCaptureStatus cst = cudaStreamCaptureStatusNone;
  cudaGraph_t cg = nullptr;
  const cudaGraphNode_t* deps = nullptr;
  size_t ndeps = 0;
  ok &= cudaStreamGetCaptureInfo(s, &cst, nullptr, &cg, &deps, nullptr, &ndeps) == cudaSuccess;
  ok &= (cst == cudaStreamCaptureStatusActive) && cg != nullptr;
  cudaGraphConditionalHandle h = 0;
  if (ok) ok &= cudaGraphConditionalHandleCreate(&h, cg, 1, cudaGraphCondAssignDefault) == cudaSuccess;
  if (ok) {
    k_pcg_start<<<1, 1, 0, s>>>(dev_, h, 1);
    ok &= cudaStreamGetCaptureInfo(s, &cst, nullptr, &cg, &deps, nullptr, &ndeps) == cudaSuccess;
    ok &= (cst == cudaStreamCaptureStatusActive);
  }
  cudaGraphNodeParams cp = {};
  if (ok) {
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    ok &= cudaGraphAddNode(&wnode, cg, deps, nullptr, ndeps, &cp) == cudaSuccess;
    ok &= cp.conditional.phGraph_out != nullptr;
  }
  if (ok) {
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    l1 = launches;
    ok &= cudaStreamBeginCaptureToGraph(sb, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed) ==
          cudaSuccess;
    if (ok) {
      pcg_body(sb, h, 1);
      ok &= cudaStreamEndCapture(sb, &body) == cudaSuccess;
    }
    l2 = launches;
    if (ok) ok &= cudaStreamUpdateCaptureDependencies(s, &wnode, nullptr, 1, cudaStreamSetCaptureDependencies) ==
                  cudaSuccess;
  }
  return ok;
}

// Records the CG solve into a graph: a prologue (initial residual, first
// preconditioned direction, start test) followed by a WHILE conditional node
// whose body is one CG iteration; the body's last kernel decides whether the
// loop continues, so the solve runs without host round trips.  The loop is
// bounded by maxit (checked on the device).  Recording happens on two streams
// owned by this object (capture is not possible on the legacy default stream);
// every graph call is checked and nothing is launched unless all succeeded.
template <class T>
int MG<T>::capture_pcg(bool warm) {
  std::lock_guard<std::recursive_mutex> lock(device_lock());
  cudaStream_t s = cap_[0], sb = cap_[1];
  if (!s || !sb) return -5;
  Graph& G = graph_[warm ? 1 : 0];
  if (G.exec) {
    cudaGraphExecDestroy(G.exec);
    G.exec = nullptr;
  }
  cudaGetLastError();
  const long long l0 = launches;
  if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) return -5;
  long long l1 = 0, l2 = 0;
  bool ok = record_solve(warm, s, sb, l1, l2);
  cudaGraph_t graph = nullptr;
  const cudaError_t ee = cudaStreamEndCapture(s, &graph);
  ok &= (ee == cudaSuccess) && graph != nullptr;
  if (ok) ok &= cudaGraphInstantiate(&G.exec, graph, 0) == cudaSuccess;
  if (graph) cudaGraphDestroy(graph);
  ok &= cudaGetLastError() == cudaSuccess;
  launches = l0;  // recording is not execution
  if (!ok) {
    if (G.exec) cudaGraphExecDestroy(G.exec);
    G.exec = nullptr;
    return -5;
  }
  G.prologue_nodes = (l1 - l0) + 1;
  G.body_nodes = (l2 - l1);
  return 0;
}

// The recorded solve's kernels launched one by one (a round trip per iteration).
template <class T>
bool MG<T>::solve_from_host(bool warm, cudaStream_t s) {
  pcg_prologue(warm, s);
  k_pcg_start<<<1, 1, 0, s>>>(dev_, 0, 0);
  ++launches;
  for (;;) {
    cudaMemcpyAsync(hdev_, dev_, sizeof(PcgDev), cudaMemcpyDeviceToHost, s);
    if (cudaStreamSynchronize(s) != cudaSuccess) return false;
    if (hdev_->status != 1) return true;
    pcg_body(s, 0, 0);
  }
}

// Runs the captured solve: inputs are copied into the graph's fixed buffers,
// rtol^2 and the iteration cap are written to the device scalars the start
// kernel reads, and the result and the scalars come back after one sync.
template <class T>
int MG<T>::graph_pcg(const T* b, T* x, double* x64, bool warm, double rtol, int maxit, SolveStats& st,
                     cudaStream_t s) {
  const size_t n = specs_[0].ndof();
  T* bi = pcg_[5];
  T* xi = pcg_[6];
  if (!graph_valid_) {
    for (auto& G : graph_)
      if (G.exec) {
        cudaGraphExecDestroy(G.exec);
        G.exec = nullptr;
      }
    graph_valid_ = true;
  }
  Graph& G = graph_[warm ? 1 : 0];
  if (use_graphs && !G.exec) {
    // the recording streams must not see work still queued on s
    if (cudaStreamSynchronize(s) != cudaSuccess) return -5;
    if (capture_pcg(warm) != 0) {
      // a recording can fail when another thread's work synchronises the device
      // meanwhile (first use of a kernel, a free); this solve then runs the same
      // kernels from the host and the next one records again
      cudaGetLastError();
      ++capture_failures;
    }
  }
  const bool graphs = use_graphs && G.exec;
  hdev_->tol2 = rtol * rtol;
  hdev_->maxit = maxit;
  cudaMemcpyAsync(bi, b, n * sizeof(T), cudaMemcpyDeviceToDevice, s);
  if (warm) {
    if (x64) k_convert<T, double><<<vec_grid(n, sms_), kVecThreads, 0, s>>>(xi, x64, 1.0, n);
    else cudaMemcpyAsync(xi, x, n * sizeof(T), cudaMemcpyDeviceToDevice, s);
  }
  cudaMemcpyAsync(&dev_->tol2, &hdev_->tol2, sizeof(double), cudaMemcpyHostToDevice, s);
  cudaMemcpyAsync(&dev_->maxit, &hdev_->maxit, sizeof(int), cudaMemcpyHostToDevice, s);
  if (graphs) {
    cudaGraphLaunch(G.exec, s);
    launches += G.prologue_nodes;
  } else {
    if (!solve_from_host(warm, s)) return -5;
  }
  if (x64) cudaMemcpyAsync(x64, xacc_, n * sizeof(double), cudaMemcpyDeviceToDevice, s);
  else cudaMemcpyAsync(x, xi, n * sizeof(T), cudaMemcpyDeviceToDevice, s);
  cudaMemcpyAsync(hdev_, dev_, sizeof(PcgDev), cudaMemcpyDeviceToHost, s);
  if (cudaStreamSynchronize(s) != cudaSuccess) return -5;
  st.iterations = hdev_->it;
  st.relres = hdev_->relres;
  if (graphs) launches += (long long)hdev_->it * G.body_nodes;
  switch (hdev_->status) {
    case 0: return 0;
    case 5:
      if (x64) k_fill<double><<<vec_grid(n, sms_), kVecThreads, 0, s>>>(x64, 0.0, n);
      else k_fill<T><<<vec_grid(n, sms_), kVecThreads, 0, s>>>(x, T(0), n);
      return 0;
    case 4: return -4;
    case 3: return -3;  // breakdown: caller falls back
    default: return -2;
  }
}

template <class T>
int MG<T>::pcg(const T* b, T* x, bool x_nonzero, double rtol, int maxit, SolveStats& st, cudaStream_t s) {
  st = SolveStats{};
  int rc = graph_pcg(b, x, nullptr, x_nonzero, rtol, maxit, st, s);
  if (rc == -3) {
    // p.Ap <= 0: the operator is indefinite here; continue with MINRES from x
    SolveStats ms;
    rc = minres(b, x, rtol, std::max(1, maxit - st.iterations), ms, s);
    st.iterations += ms.iterations;
    st.relres = ms.relres;
    st.minres = 1;
  }
  return rc;
}

template <class T>
int MG<T>::pcg_x64(const T* b, double* x64, bool x_nonzero, double rtol, int maxit, SolveStats& st,
                   cudaStream_t s) {
  st = SolveStats{};
  if (!xacc_) return -5;
  int rc = graph_pcg(b, nullptr, x64, x_nonzero, rtol, maxit, st, s);
  if (rc == -3) {
    // MINRES continues in T from the iterate rounded to T (pcg_[9]: neither
    // MINRES's work vectors nor the callers' scratch0(4))
    const size_t n = specs_[0].ndof();
    const int g = vec_grid(n, sms_);
    T* xt = pcg_[9];
    k_convert<T, double><<<g, kVecThreads, 0, s>>>(xt, x64, 1.0, n);
    SolveStats ms;
    rc = minres(b, xt, rtol, std::max(1, maxit - st.iterations), ms, s);
    k_convert<double, T><<<g, kVecThreads, 0, s>>>(x64, xt, 1.0, n);
    launches += 2;
    st.iterations += ms.iterations;
    st.relres = ms.relres;
    st.minres = 1;
  }
  return rc;
}
// Preconditioned MINRES (Paige & Saunders) with the SPD V-cycle as M, started
// from x.  The recurrence's residual estimate (in the M^-1 norm) steers the
// iteration; the true 2-norm residual is checked before returning.
template <class T>
int MG<T>::minres(const T* b, T* x, double rtol, int maxit, SolveStats& st, cudaStream_t s) {
  const size_t n = specs_[0].ndof();
  const int g = vec_grid(n, sms_);
  T* r1 = pcg_[0];
  T* r2 = pcg_[1];
  T* y = pcg_[2];
  T* v = pcg_[3];
  T* w = pcg_[5];
  T* w1 = pcg_[6];
  T* w2 = pcg_[7];
  T* t = pcg_[8];
  st = SolveStats{};
  const double bn = std::sqrt(dot(b, b, n, s));
  if (!std::isfinite(bn)) return -4;
  int total = 0;
  for (int restart = 0; restart < 4 && total < maxit; ++restart) {
    apply(0, x, t, s, true);
    k_sub<T><<<g, kVecThreads, 0, s>>>(r1, b, t, n);
    const double rn0 = std::sqrt(dot(r1, r1, n, s));
    st.relres = rn0 / bn;
    if (!std::isfinite(rn0)) return -4;
    if (rn0 <= rtol * bn) return 0;
    vcycle(r1, y, s);
    double beta1 = dot(r1, y, n, s);
    if (!(beta1 > 0.0)) return -2;
    beta1 = std::sqrt(beta1);
    cudaMemcpyAsync(r2, r1, n * sizeof(T), cudaMemcpyDeviceToDevice, s);
    k_fill<T><<<g, kVecThreads, 0, s>>>(w, T(0), n);
    k_fill<T><<<g, kVecThreads, 0, s>>>(w2, T(0), n);
    double beta = beta1, oldb = 0.0, dbar = 0.0, epsln = 0.0, phibar = beta1, cs = -1.0, sn = 0.0;
    // the M^-1-norm estimate is compared against the same ratio of the 2-norms
    const double target = rtol * bn / rn0;
    for (int it = 1; it <= maxit - total; ++it) {
      // v = y / beta ; y = A v - (beta/oldb) r1
      k_convert<T, T><<<g, kVecThreads, 0, s>>>(v, y, 1.0 / beta, n);
      apply(0, v, y, s, true);
      if (it >= 2) k_axpy<T><<<g, kVecThreads, 0, s>>>(y, T(-beta / oldb), r1, n);
      const double alpha = dot(v, y, n, s);
      k_axpy<T><<<g, kVecThreads, 0, s>>>(y, T(-alpha / beta), r2, n);
      std::swap(r1, r2);  // r1 <- r2, r2 <- y
      cudaMemcpyAsync(r2, y, n * sizeof(T), cudaMemcpyDeviceToDevice, s);
      vcycle(r2, y, s);
      oldb = beta;
      const double bb = dot(r2, y, n, s);
      if (!std::isfinite(alpha) || !std::isfinite(bb)) return -4;
      if (!(bb > 0.0)) {
        total += it;
        break;
      }
      beta = std::sqrt(bb);
      const double oldeps = epsln;
      const double delta = cs * dbar + sn * alpha;
      const double gbar = sn * dbar - cs * alpha;
      epsln = sn * beta;
      dbar = -cs * beta;
      double gamma = std::sqrt(gbar * gbar + beta * beta);
      if (gamma < 1e-300) gamma = 1e-300;
      cs = gbar / gamma;
      sn = beta / gamma;
      const double phi = cs * phibar;
      phibar = sn * phibar;
      // w1 <- w2, w2 <- w, w = (v - oldeps w1 - delta w2) / gamma ; x += phi w
      std::swap(w1, w2);  // w1 <- old w2
      std::swap(w2, w);   // w2 <- old w ; w now holds the stale w1 (overwritten below)
      k_fill<T><<<g, kVecThreads, 0, s>>>(w, T(0), n);
      k_axpy<T><<<g, kVecThreads, 0, s>>>(w, T(1.0 / gamma), v, n);
      k_axpy<T><<<g, kVecThreads, 0, s>>>(w, T(-oldeps / gamma), w1, n);
      k_axpy<T><<<g, kVecThreads, 0, s>>>(w, T(-delta / gamma), w2, n);
      k_axpy<T><<<g, kVecThreads, 0, s>>>(x, T(phi), w, n);
      st.iterations = total + it;
      if (phibar / beta1 <= 0.5 * target) {
        total += it;
        break;
      }
      if (it == maxit - total) total = maxit;
    }
    st.minres = 1;
  }
  apply(0, x, t, s, true);
  k_sub<T><<<g, kVecThreads, 0, s>>>(r1, b, t, n);
  const double rn = std::sqrt(dot(r1, r1, n, s));
  st.relres = rn / bn;
  if (!std::isfinite(rn)) return -4;
  return rn <= rtol * bn ? 0 : -2;
}

}  // namespace topo
