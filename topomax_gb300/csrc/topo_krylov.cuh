// Flexible GMRES on the device: the Gram-Schmidt, rotation and update kernels of one restart
// cycle, whose iterations a caller records into the body of a WHILE graph node together with
// its preconditioner and operator (topo_fluid.cu, and the mixed-precision refinement of
// topo_capi.cu).  The basis and all sums are FP64.
#pragma once

#include <cuda_runtime.h>

#include "topo_mg_impl.cuh"
#include "topo_vec.cuh"

namespace topo {

constexpr int kKrylovMax = 60;  // longest restart
// A column is orthogonalised again where less than this share of |w|^2 is left (Kahan's "twice is
// enough").  A vector keeps what the basis before it has lost, times the norm that its own
// products took, so a lower share does not only cost a few roundings: with 0.01 no column of the
// fluid solve was repeated, max |V^T V - I| grew to 0.015 .. 0.25 over 60 vectors (16x16 to 128x128)
// and the residual's estimate was off by up to a third; with 0.5 the loss is 2e-15.  The
// second passes cost 10.4 to 12.5 ms at 40x40, 20.7 to 25.2 at 128x128.
constexpr double kReorthogonalise = 0.5;
constexpr int kDotGroup = 8;  // basis vectors of one block of the Gram-Schmidt products
constexpr int kDotGroups = (kKrylovMax + kDotGroup) / kDotGroup;

// Device-side state of one restart cycle.  v_0 .. v_j are the basis so far, column j of the
// Hessenberg matrix is being formed.
struct KrylovDev {
  int j, it, maxit, status;  // status: 1 running, 0 done, 3 inner breakdown,
                             // 4 non-finite
  int second;                // the column needs a second Gram-Schmidt pass
  int inner, bad;            // inner iterations so far; an inner solve broke down (3) or met NaN (4)
  int inner_maxit;
  double res;                // residual norm of the least-squares problem so far
  double target;             // residual norm to reach
  double inner_tol, inner_floor;  // the inner solve's tolerance: inner_tol / residual, at least the floor
  double psum, zsum;         // (fluid) sums of the pressure parts of v_j and of z_j
  double ww, hn;             // |w|^2 before and |w| after the orthogonalisation
  double h[kKrylovMax + 1], hp[kKrylovMax + 1];  // the column, and a pass's products
  double cs[kKrylovMax], sn[kKrylovMax], gv[kKrylovMax + 1], y[kKrylovMax];
  double H[(kKrylovMax + 1) * kKrylovMax];
};

// sums of v_k . w over C vectors and, where ww is asked for, of w . w.  Two entries at a time for few
// vectors: one entry's loads do not fill the memory pipe.
template <int C>
__device__ __forceinline__ void krylov_products(const double* v, const double* w, size_t n, bool ww, double* s) {
  constexpr int E = C <= 4 ? 2 : 1;
  const size_t step = size_t(gridDim.x) * blockDim.x;
  for (size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += E * step) {
    double wi[E], vi[E][C];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const bool on = e == 0 || i + e * step < n;
      wi[e] = on ? w[i + e * step] : 0.0;
#pragma unroll
      for (int k = 0; k < C; ++k) vi[e][k] = on ? v[size_t(k) * n + i + e * step] : 0.0;
    }
#pragma unroll
    for (int e = 0; e < E; ++e) {
#pragma unroll
      for (int k = 0; k < C; ++k) s[k] += vi[e][k] * wi[e];
      if (ww) s[kDotGroup] += wi[e] * wi[e];
    }
  }
}

// a + sum_k c_k v_k at one entry
template <int C>
__device__ __forceinline__ double krylov_combine(double a, const double* v, size_t n, const double* c) {
  double x[C];
#pragma unroll
  for (int k = 0; k < C; ++k) x[k] = v[size_t(k) * n];
#pragma unroll
  for (int k = 0; k < C; ++k) a += c[k] * x[k];
  return a;
}

// Where a thread takes many entries (krylov_large) the loops are compiled for each count of 1 to 8
// vectors, so that all loads of an entry are in flight together: with loops of a run-time count the
// state solve of 2000x1000 (16 M unknowns) was 1.5 % slower than with these.  Where it takes one
// or two, the jump costs more than it gives (fluid at 40x40 8.5 ms against 8.1).
#define TOPO_KRYLOV_COUNT(count, CALL) \
  switch (count) {                     \
    case 1: CALL(1); break;            \
    case 2: CALL(2); break;            \
    case 3: CALL(3); break;            \
    case 4: CALL(4); break;            \
    case 5: CALL(5); break;            \
    case 6: CALL(6); break;            \
    case 7: CALL(7); break;            \
    case 8: CALL(8); break;            \
    default: break;                    \
  }
static_assert(kDotGroup == 8, "TOPO_KRYLOV_COUNT");

__device__ __forceinline__ double krylov_combine_all(double a, const double* v, size_t n, const double* c, int count) {
  int k = 0;
  for (; k + kDotGroup <= count; k += kDotGroup) a = krylov_combine<kDotGroup>(a, v + size_t(k) * n, n, c + k);
#define TOPO_COMBINE(C) a = krylov_combine<C>(a, v + size_t(k) * n, n, c + k)
  TOPO_KRYLOV_COUNT(count - k, TOPO_COMBINE)
#undef TOPO_COMBINE
  return a;
}

// A pass's products hp_i = v_i . w, i <= j, and |w|^2: blockIdx.y takes eight basis vectors,
// blockIdx.x a share of the entries.  w is wfix, or v_(j+1) where that is null.  The first pass
// also moves zc, the fluid's centred pressure, into z_j (the operator's launch could not: its
// other blocks read the uncentred one).
template <bool LARGE>
static __global__ void __launch_bounds__(kVecThreads)
    k_krylov_dot(const double* V, const double* wfix, double* Z, size_t n, size_t nv, const double* zc, int pass,
                 double* partials, unsigned* counters, KrylovDev* K) {
  TOPO_PDL_ENTRY();
  const int j = K->j, i0 = blockIdx.y * kDotGroup;
  if (pass == 1 && !K->second) return;
  if (pass == 0 && zc && blockIdx.y == 0) {
    double* z = Z + size_t(j) * n + (n - nv);
    TOPO_GRID_STRIDE(k, nv) z[k] = zc[k];
  }
  if (i0 > j) return;
  const double* w = wfix ? wfix : V + size_t(j + 1) * n;
  const double* v = V + size_t(i0) * n;
  const int count = min(kDotGroup, j + 1 - i0);
  double s[kDotGroup + 1];
#pragma unroll
  for (int k = 0; k <= kDotGroup; ++k) s[k] = 0.0;
  if constexpr (LARGE) {
#define TOPO_PRODUCTS(C) krylov_products<C>(v, w, n, i0 == 0, s)
    TOPO_KRYLOV_COUNT(count, TOPO_PRODUCTS)
#undef TOPO_PRODUCTS
  } else if (count == kDotGroup) {
    TOPO_GRID_STRIDE(i, n) {
      const double wi = w[i];
#pragma unroll
      for (int k = 0; k < kDotGroup; ++k) s[k] += v[size_t(k) * n + i] * wi;
      if (i0 == 0) s[kDotGroup] += wi * wi;
    }
  } else {
    TOPO_GRID_STRIDE(i, n) {
      const double wi = w[i];
#pragma unroll
      for (int k = 0; k < kDotGroup; ++k)
        if (k < count) s[k] += v[size_t(k) * n + i] * wi;
      if (i0 == 0) s[kDotGroup] += wi * wi;
    }
  }
  double tot[kDotGroup + 1];
  if (finish_reduction<kDotGroup + 1>(s, partials + size_t(blockIdx.y) * (kDotGroup + 1) * gridDim.x,
                                      counters + blockIdx.y, tot, blockIdx.x, gridDim.x)) {
    for (int k = 0; k < count; ++k) K->hp[i0 + k] = tot[k];
    if (i0 == 0) K->ww = tot[kDotGroup];
  }
}

// w -= sum hp_i v_i.  The first pass (classical Gram-Schmidt) decides on the second: it is needed
// where the products took most of |w|^2 (kReorthogonalise; Kahan's "twice is enough"); the
// second sums |w|^2.
template <bool LARGE>
static __global__ void __launch_bounds__(kVecThreads)
    k_krylov_sub(double* V, double* wfix, size_t n, int pass, double* partials, unsigned* counter, KrylovDev* K) {
  TOPO_PDL_ENTRY();
  __shared__ double h[kKrylovMax + 1];
  const int j = K->j;
  if (pass == 1 && !K->second) return;
  for (int i = threadIdx.x; i <= j; i += blockDim.x) h[i] = -K->hp[i];
  __syncthreads();
  double* w = wfix ? wfix : V + size_t(j + 1) * n;
  double s[1] = {0.0};
  TOPO_GRID_STRIDE(i, n) {
    double a = w[i];
    if constexpr (LARGE) {
      a = krylov_combine_all(a, V + i, n, h, j + 1);
    } else {
      int k = 0;
      for (; k + 8 <= j + 1; k += 8) {
#pragma unroll
        for (int q = 0; q < 8; ++q) a += h[k + q] * V[size_t(k + q) * n + i];
      }
      for (; k <= j; ++k) a += h[k] * V[size_t(k) * n + i];
    }
    w[i] = a;
    s[0] += a * a;
  }
  if (pass == 0) {
    // (a kernel after this one reads `second`; none of this grid does)
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      double hh = 0.0;
      for (int i = 0; i <= j; ++i) {
        K->h[i] = -h[i];
        hh += h[i] * h[i];
      }
      const double ww = K->ww, est = ww - hh;
      K->second = !(est >= kReorthogonalise * ww);
      K->hn = sqrt(est);
    }
    return;
  }
  double tot[1];
  if (finish_reduction<1>(s, partials, counter, tot)) {
    for (int i = 0; i <= j; ++i) K->h[i] -= h[i];
    K->hn = sqrt(tot[0]);
  }
}

// v_(j+1) = w / |w| and the sum of its pressure, in all blocks but the first, whose first warp
// rotates the column into the triangular factor, updates the residual norm and decides
// whether the cycle goes on.  The rotations' recurrence up' = -s_i up + c_i h_(i+1) is affine in
// up: a warp scan of two maps a lane (a thread's loop took ~10 us at 30 columns).
static __global__ void __launch_bounds__(kVecThreads)
    k_krylov_next(double* V, const double* wfix, size_t n, size_t nv, int m, double* partials, unsigned* counter,
                  KrylovDev* K, cudaGraphConditionalHandle cond, int use_cond) {
  TOPO_PDL_ENTRY();
  const int j = K->j;
  const double hn = K->hn, f = hn > 0 ? 1.0 / hn : 1.0;
  double s[1] = {0.0};
  if (blockIdx.x > 0) {
    double* vn = V + size_t(j + 1) * n;
    const double* w = wfix ? wfix : vn;
    for (size_t i = size_t(blockIdx.x - 1) * blockDim.x + threadIdx.x; i < n; i += size_t(gridDim.x - 1) * blockDim.x) {
      const double v = w[i] * f;
      vn[i] = v;
      if (i >= n - nv) s[0] += v;
    }
  } else if (threadIdx.x < 32) {
    const int e = 2 * int(threadIdx.x);
    double c[2], t[2], h[2], a[2], b[2];
    for (int q = 0; q < 2; ++q) {
      const bool on = e + q < j;
      c[q] = on ? K->cs[e + q] : 1.0;
      t[q] = on ? K->sn[e + q] : 0.0;
      h[q] = on ? K->h[e + q + 1] : 0.0;
      a[q] = on ? -t[q] : 1.0;
      b[q] = c[q] * h[q];
    }
    const double h0 = K->h[0];
    double A = a[1] * a[0], B = a[1] * b[0] + b[1];
    for (int o = 1; o < 32; o <<= 1) {
      const double pa = __shfl_up_sync(0xffffffffu, A, o), pb = __shfl_up_sync(0xffffffffu, B, o);
      if (int(threadIdx.x) >= o) {
        B = A * pb + B;
        A = A * pa;
      }
    }
    double Ea = __shfl_up_sync(0xffffffffu, A, 1), Eb = __shfl_up_sync(0xffffffffu, B, 1);
    if (threadIdx.x == 0) {
      Ea = 1.0;
      Eb = 0.0;
    }
    double up = Ea * h0 + Eb;
    for (int q = 0; q < 2; ++q) {
      if (e + q < j) K->H[(e + q) * kKrylovMax + j] = c[q] * up + t[q] * h[q];
      up = a[q] * up + b[q];
    }
    up = __shfl_sync(0xffffffffu, up, 31);
    if (threadIdx.x == 0) {
      const double den = hypot(up, hn);
      const double cj = den > 0 ? up / den : 1.0, tj = den > 0 ? hn / den : 0.0;
      K->cs[j] = cj;
      K->sn[j] = tj;
      K->H[j * kKrylovMax + j] = den;
      const double g = K->gv[j];
      K->gv[j + 1] = -tj * g;
      K->gv[j] = cj * g;
      const int it = K->it + 1;
      K->it = it;
      int st = 1;
      K->res = fabs(tj * g);
      if (K->bad) st = K->bad;
      else if (!isfinite(hn)) st = 4;
      else if (fabs(tj * g) <= K->target || hn == 0.0 || j + 1 >= m || it >= K->maxit) st = 0;
      K->status = st;
      if (use_cond) cudaGraphSetConditional(cond, st == 1 ? 1u : 0u);
    }
  }
  double tot[1];
  if (finish_reduction<1>(s, partials, counter, tot)) {
    K->psum = tot[0];
    K->j = j + 1;  // every block has read it
  }
}

static __global__ void k_krylov_start(KrylovDev* K, double beta, double target, int it, int maxit, double inner_tol,
                                      double inner_floor, int inner_maxit) {
  K->j = 0;
  K->it = it;
  K->maxit = maxit;
  K->status = 1;
  K->target = target;
  K->inner = K->bad = 0;
  K->inner_tol = inner_tol;
  K->inner_floor = inner_floor;
  K->inner_maxit = inner_maxit;
  K->res = beta;
  K->gv[0] = beta;
}

// y = R^-1 g by one warp: column by column, the lanes hold the remaining right-hand side
static __global__ void __launch_bounds__(32) k_krylov_backsolve(KrylovDev* K) {
  constexpr int P = (kKrylovMax + 31) / 32;
  const int k = K->j, lane = threadIdx.x;
  double g[P];
  for (int q = 0; q < P; ++q) g[q] = lane + 32 * q < k ? K->gv[lane + 32 * q] : 0.0;
  for (int i = k - 1; i >= 0; --i) {
    const double d = K->H[i * kKrylovMax + i];
    const double y = __shfl_sync(0xffffffffu, i < 32 ? g[0] : g[P - 1], i & 31) / d;
    const double yi = d != 0.0 ? y : 0.0;
    if (lane == 0) K->y[i] = yi;
    for (int q = 0; q < P; ++q)
      if (lane + 32 * q < i) g[q] -= K->H[(lane + 32 * q) * kKrylovMax + i] * yi;
  }
}
static_assert(kKrylovMax <= 64, "two values per lane, here and in k_krylov_next");

// x += sum_i y_i z_i over the cycle's directions
static __global__ void k_krylov_update(double* x, const double* Z, size_t n, const KrylovDev* K) {
  __shared__ double y[kKrylovMax];
  const int k = K->j;
  for (int i = threadIdx.x; i < k; i += blockDim.x) y[i] = K->y[i];
  __syncthreads();
  TOPO_GRID_STRIDE(i, n) x[i] = krylov_combine_all(x[i], Z + i, n, y, k);
}

// partial sums of the products with at most `blocks` blocks a group
inline size_t krylov_dots(int blocks) { return size_t(blocks) * (kDotGroup + 1) * kDotGroups; }

// Vectors and scratch of a cycle.  w: where the operator leaves A z_j (null: v_(j+1) itself).
struct KrylovSpace {
  double *V, *w, *Z;
  const double* zc;
  size_t n, nv;
  int m;
  double* dots;
  unsigned* counters;
  double* partials;
  unsigned* counter;
  KrylovDev* K;
};

constexpr size_t kKrylovLarge = 8;  // entries per thread of the dot products
inline bool krylov_large(size_t n, int gd) { return n > kKrylovLarge * kVecThreads * size_t(gd); }

template <bool LARGE>
inline void krylov_pass(const KrylovSpace& S, int pass, int gd, int gv, cudaStream_t s) {
  launch_pdl(k_krylov_dot<LARGE>, dim3(gd, unsigned((S.m + kDotGroup - 1) / kDotGroup)), kVecThreads, 0, s,
             static_cast<const double*>(S.V), static_cast<const double*>(S.w), S.Z, S.n, S.nv, S.zc, pass, S.dots,
             S.counters, S.K);
  launch_pdl(k_krylov_sub<LARGE>, gv, kVecThreads, 0, s, S.V, S.w, S.n, pass, S.partials, S.counter, S.K);
}

// From A z_j to v_(j+1) and the cycle's next test: orthogonalisation, column, normalisation.
inline void krylov_column(const KrylovSpace& S, int gd, int gv, cudaGraphConditionalHandle cond, int use_cond,
                          cudaStream_t s) {
  for (int pass = 0; pass < 2; ++pass) {
    if (krylov_large(S.n, gd)) krylov_pass<true>(S, pass, gd, gv, s);
    else krylov_pass<false>(S, pass, gd, gv, s);
  }
  launch_pdl(k_krylov_next, gd + 1, kVecThreads, 0, s, S.V, static_cast<const double*>(S.w), S.n, S.nv, S.m, S.partials,
             S.counter, S.K, cond, use_cond);
}

}  // namespace topo
