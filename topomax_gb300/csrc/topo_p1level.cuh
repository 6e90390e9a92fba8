// The V-cycle's two sweeps of a P1 level with an assembled stencil, one launch each:
//   down:  x = D Chebyshev steps from zero, r = b - A x, b_c = P^T r
//   up:    x += P x_c, D Chebyshev steps
// A block owns cx x cy coarse nodes and the 2cx x 2cy fine nodes over them and
// recomputes the ring its own results need (D + 1 nodes wide down, D up), so that the
// steps between the loads and the stores go through shared memory.
// Such a level is bound by latency: as separate launches (smoothing steps, residual,
// restriction, prolongation) each takes 4 to 6 us for vectors that stay in L2, while
// a further step inside a sweep is a barrier and seven products.  A thread keeps its
// node's stencil row, inverse diagonal, residual and iterate in registers; only the
// direction, which the neighbours read, goes through shared memory.  The rows and
// diagonals, which no solve changes, are loaded before the kernel waits for its
// predecessor.
#pragma once

#include "topo_p1.cuh"

namespace topo {

template <class T, int NC>
struct LevelSweep {
  int NX, NY, NXc, NYc;  // nodes of the level and of the next coarser one
  int cx, cy;            // coarse nodes per block
  const T* st;           // stencil rows (P1Stencil::s)
  const T* inner;        // one row for all interior nodes, or null
  const T* dinv;
  const T* cheb;
  Dir dirf, dirc;
};

// the threads' region, one node each: a block's nodes with a ring of D down (1 for the
// residual the restriction reads, D - 1 for the steps before it), of D - 1 up
template <int D, class L>
TOPO_HD int down_w(const L& P) { return 2 * P.cx + 2 * D - 1; }
template <int D, class L>
TOPO_HD int down_h(const L& P) { return 2 * P.cy + 2 * D - 1; }
template <int D, class L>
TOPO_HD int up_w(const L& P) { return 2 * P.cx + 2 * D - 2; }
template <int D, class L>
TOPO_HD int up_h(const L& P) { return 2 * P.cy + 2 * D - 2; }

// Two shared vectors over the region and a ring around it; the direction alternates
// between them.  Positions outside the part that a step still needs hold stale or no
// values; they are read (in bounds) and never reach a result.
TOPO_HD int sweep_shared(int w, int h, int NC) { return 2 * NC * (w + 2) * (h + 2); }

// 16-byte loads of N values (source and N * sizeof(T) multiples of 16 bytes)
template <class T, int N>
TOPO_HD void load_row(const T* src, T (&dst)[N]) {
#if defined(__CUDA_ARCH__)
  constexpr int V = 16 / int(sizeof(T));
  static_assert(N % V == 0, "whole 16-byte groups");
#pragma unroll
  for (int i = 0; i < N / V; ++i) {
    if constexpr (sizeof(T) == 4) {
      const float4 f = __ldg(reinterpret_cast<const float4*>(src) + i);
      dst[4 * i] = f.x;
      dst[4 * i + 1] = f.y;
      dst[4 * i + 2] = f.z;
      dst[4 * i + 3] = f.w;
    } else {
      const double2 f = __ldg(reinterpret_cast<const double2*>(src) + i);
      dst[2 * i] = f.x;
      dst[2 * i + 1] = f.y;
    }
  }
#else
  for (int i = 0; i < N; ++i) dst[i] = src[i];
#endif
}

// the same copy within shared memory's address space (generic loads and stores)
template <class T, int N>
TOPO_HD void copy_row(const T* src, T* dst) {
#if defined(__CUDA_ARCH__)
#pragma unroll
  for (int i = 0; i < N * int(sizeof(T)) / 16; ++i)
    reinterpret_cast<float4*>(dst)[i] = reinterpret_cast<const float4*>(src)[i];
#else
  for (int i = 0; i < N; ++i) dst[i] = src[i];
#endif
}

// Explicit fused operations: the sweeps and the one-block tail below give the same bits.
TOPO_HD float fma_t(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
  return __fmaf_rn(a, b, c);
#else
  return std::fma(a, b, c);
#endif
}
TOPO_HD double fma_t(double a, double b, double c) {
#if defined(__CUDA_ARCH__)
  return __fma_rn(a, b, c);
#else
  return std::fma(a, b, c);
#endif
}

// FP64 needs no difference form, and its pipe is the bound: block 0 becomes the node's own
// coupling (the row sum less the neighbours'), 7 products instead of 13 operations per value.
template <class T, int NC>
TOPO_HD void level_row(T (&st)[StencilLayout<NC>::stride]) {
  if constexpr (sizeof(T) == 8) {
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int k = 1; k < 7; ++k)
      for (int i = 0; i < NC * NC; ++i) st[i] -= st[k * NC * NC + i];
  }
}

// (A u) at the node of row st (level_row), u in a row-major region of width w, the node at
// position p.  Couplings to nodes outside the lattice and to clamped nodes are zero, and the
// row of a clamped node is the identity (p1_stencil_node): no test is needed, only values
// there.
template <class T, int NC>
TOPO_HD void level_apply(const T (&st)[StencilLayout<NC>::stride], const T* u, int w, int p, T (&acc)[NC]) {
  T un[NC];
  for (int c = 0; c < NC; ++c) un[c] = u[NC * p + c];
  for (int c = 0; c < NC; ++c) {
    acc[c] = st[c * NC] * un[0];
    for (int d = 1; d < NC; ++d) acc[c] = fma_t(st[c * NC + d], un[d], acc[c]);
  }
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
  for (int k = 1; k < 7; ++k) {
    const int q = p + st_db(k) * w + st_da(k);
    T ul[NC];
    for (int c = 0; c < NC; ++c) ul[c] = sizeof(T) == 8 ? u[NC * q + c] : u[NC * q + c] - un[c];
    for (int c = 0; c < NC; ++c)
      for (int d = 0; d < NC; ++d) acc[c] = fma_t(st[k * NC * NC + c * NC + d], ul[d], acc[c]);
  }
}

// the next Chebyshev direction c1 d + c2 Dinv r
template <class T>
TOPO_HD T level_direction(T c1, T d, T c2, T di, T r) {
  return fma_t(c2 * di, r, c1 * d);
}

// the iterate after the last direction: x + c1 d + c2 Dinv r
template <class T>
TOPO_HD T level_last(T x, T c1, T d, T c2, T di, T r) {
  return fma_t(c2 * di, r, fma_t(c1, d, x));
}

// (P^T r) from the residual at the coarse node's fine position and its six neighbours
template <class T, int NC>
TOPO_HD T level_restrict(const T* r, int w) {
  T h = r[-NC];
  h += r[NC];
  h += r[-NC * w];
  h += r[NC * w];
  h += r[NC * (w + 1)];
  h += r[-NC * (w + 1)];
  return fma_t(T(0.5), h, r[0]);
}

// A thread's node: what the two operator applications share.
template <class T, int NC>
struct LevelNode {
  int a, b;  // lattice position (may lie outside)
  bool in;
  T st[StencilLayout<NC>::stride];
  T di[NC], bv[NC];

  // row and inverse diagonal (zero outside the lattice)
  TOPO_HD void load(const LevelSweep<T, NC>& L, int a_, int b_) {
    a = a_;
    b = b_;
    in = a >= 0 && a < L.NX && b >= 0 && b < L.NY;
    const size_t n = in ? size_t(b) * L.NX + a : 0;
    const bool interior = L.inner && a > 0 && b > 0 && a < L.NX - 1 && b < L.NY - 1;
    load_row(interior ? L.inner : L.st + n * StencilLayout<NC>::stride, st);
    for (int c = 0; c < NC; ++c) di[c] = L.dinv[NC * n + c];
    if (!in) {
      for (int i = 0; i < StencilLayout<NC>::stride; ++i) st[i] = T(0);
      for (int c = 0; c < NC; ++c) di[c] = T(0);
    }
    level_row<T, NC>(st);
  }
  TOPO_HD size_t index(const LevelSweep<T, NC>& L) const { return size_t(b) * L.NX + a; }
  TOPO_HD void load_b(const LevelSweep<T, NC>& L, const T* bg) {
    for (int c = 0; c < NC; ++c) bv[c] = in ? bg[NC * index(L) + c] : T(0);
  }
};

// Phases of a sweep, a barrier between one and the next.  tid, nt: the thread and the block's
// threads (at least as many as the region has nodes); w: the region's width.
template <class T, int NC>
struct LevelPhases {
  using L = LevelSweep<T, NC>;
  struct Node : LevelNode<T, NC> {
    int p;              // position in the shared vectors
    T r[NC], x[NC], d[NC];
  };
  // the thread's node of a region of w x h nodes from lattice position (a0, b0)
  TOPO_HD static bool start(const L& P, int a0, int b0, int w, int h, int tid, Node& N) {
    if (tid >= w * h) return false;
    N.load(P, a0 + tid % w, b0 + tid / w);
    N.p = (tid / w + 1) * (w + 2) + tid % w + 1;
    return true;
  }
  // down: d0 = c0 Dinv b on the region and a ring around it
  TOPO_HD static void down_first(const L& P, int a0, int b0, int w, int h, int tid, int nt, const T* b, T* s) {
    const T c0 = P.cheb[0];
    for (int i = tid; i < (w + 2) * (h + 2); i += nt) {
      const int a = a0 - 1 + i % (w + 2), c = b0 - 1 + i / (w + 2);
      const bool in = a >= 0 && a < P.NX && c >= 0 && c < P.NY;
      const size_t g = in ? size_t(c) * P.NX + a : 0;
      for (int k = 0; k < NC; ++k) s[NC * i + k] = in ? (c0 * P.dinv[NC * g + k]) * b[NC * g + k] : T(0);
    }
  }
  // r = b, x = d = d0 of the thread's node, after the barrier
  TOPO_HD static void down_own(const T* s, Node& N) {
    for (int c = 0; c < NC; ++c) {
      N.r[c] = N.bv[c];
      N.x[c] = N.d[c] = s[NC * N.p + c];
    }
  }
  // up: x + P x_c on the region and a ring around it (zero outside the lattice)
  TOPO_HD static void up_first(const L& P, int a0, int b0, int w, int h, int tid, int nt, const T* x, const T* xc,
                               T* s) {
    for (int i = tid; i < (w + 2) * (h + 2); i += nt) {
      const int a = a0 - 1 + i % (w + 2), b = b0 - 1 + i / (w + 2);
      const bool in = a >= 0 && a < P.NX && b >= 0 && b < P.NY;
      if (!in) {
        for (int c = 0; c < NC; ++c) s[NC * i + c] = T(0);
        continue;
      }
      // the node's two coarse neighbours, or twice the coarse node it is
      const size_t m0 = size_t(b >> 1) * P.NXc + (a >> 1), m1 = size_t((b + 1) >> 1) * P.NXc + ((a + 1) >> 1);
      const bool free = !is_clamped(P.dirf, a, b);
      const size_t g = size_t(b) * P.NX + a;
      for (int c = 0; c < NC; ++c) {
        const T v = m0 == m1 ? xc[NC * m0 + c] : T(0.5) * (xc[NC * m0 + c] + xc[NC * m1 + c]);
        s[NC * i + c] = free ? x[NC * g + c] + v : x[NC * g + c];
      }
    }
  }
  // up: r = b - A x, d0 = c0 Dinv r, x += d0
  TOPO_HD static void up_residual(const L& P, int w, const T* sx, T* sd, Node& N) {
    T t[NC];
    level_apply<T, NC>(N.st, sx, w + 2, N.p, t);
    const T c0 = P.cheb[0];
    for (int c = 0; c < NC; ++c) {
      N.r[c] = N.bv[c] - t[c];
      N.d[c] = (c0 * N.di[c]) * N.r[c];
      N.x[c] = sx[NC * N.p + c] + N.d[c];
      sd[NC * N.p + c] = N.d[c];
    }
  }
  // step k >= 1: r -= A d, d = c1 d + c2 Dinv r, x += d; the direction from s to sn
  TOPO_HD static void step(const L& P, int k, int w, const T* s, T* sn, Node& N) {
    T t[NC];
    level_apply<T, NC>(N.st, s, w + 2, N.p, t);
    const T c1 = P.cheb[2 * k - 1], c2 = P.cheb[2 * k];
    for (int c = 0; c < NC; ++c) {
      N.r[c] -= t[c];
      N.d[c] = level_direction(c1, N.d[c], c2, N.di[c], N.r[c]);
      N.x[c] += N.d[c];
      sn[NC * N.p + c] = N.d[c];
    }
  }
  // the last step: x alone, to sn (the residual b - A x reads it)
  TOPO_HD static void last(const L& P, int k, int w, const T* s, T* sn, Node& N) {
    T t[NC];
    level_apply<T, NC>(N.st, s, w + 2, N.p, t);
    const T c1 = P.cheb[2 * k - 1], c2 = P.cheb[2 * k];
    for (int c = 0; c < NC; ++c) {
      N.x[c] = level_last(N.x[c], c1, N.d[c], c2, N.di[c], N.r[c] - t[c]);
      if (sn) sn[NC * N.p + c] = N.x[c];
    }
  }
  // down, at the end: r = b - A x (zero outside the lattice), to shared memory for the restriction
  TOPO_HD static void down_residual(int w, const T* s, T* sr, const Node& N) {
    T t[NC];
    level_apply<T, NC>(N.st, s, w + 2, N.p, t);
    for (int c = 0; c < NC; ++c) sr[NC * N.p + c] = N.bv[c] - t[c];
  }
  // stores the block's own nodes (ring: how far they lie inside the region)
  TOPO_HD static void store(const L& P, int w, int ring, int tid, const Node& N, T* x) {
    const int i = tid % w - ring, j = tid / w - ring;
    if (!N.in || i < 0 || i >= 2 * P.cx || j < 0 || j >= 2 * P.cy) return;
    for (int c = 0; c < NC; ++c) x[NC * N.index(P) + c] = N.x[c];
  }
  // ring: the position of the block's first coarse node inside the region
  TOPO_HD static void restrict_to(const L& P, int I0, int J0, int w, int ring, int tid, int nt, const T* sr, T* bc) {
    for (int i = tid; i < P.cx * P.cy; i += nt) {
      const int ic = i % P.cx, jc = i / P.cx, I = I0 + ic, J = J0 + jc;
      if (I >= P.NXc || J >= P.NYc) continue;
      const int p = (2 * jc + ring + 1) * (w + 2) + 2 * ic + ring + 1;
      const bool zero = is_clamped(P.dirc, I, J);
      for (int c = 0; c < NC; ++c)
        bc[NC * (size_t(J) * P.NXc + I) + c] = zero ? T(0) : level_restrict<T, NC>(sr + NC * p + c, w + 2);
    }
  }
};

// ---------------------------------------------------------------------------
// The V-cycle's last levels in one block: level 0 is the first of them, every level's
// vectors (with a ring of zeros) and the rows of levels >= 1 in shared memory, the rows
// of level 0 in the threads' registers, one node per thread.  A launch of its own costs a
// level ~2.5 us twice; here its phases are barriers and a few hundred cycles each.
// ---------------------------------------------------------------------------
constexpr int kTailMaxLevels = 6;                  // smoothed levels
constexpr size_t kTailShared = 48 * 1024;          // (no opt-in attribute needed)
// nodes of the first level, one per thread (1000x500: 33x17; a limit of 300 or 160 nodes
// measured the same or up to 2 % slower).  FP32 only: an FP64 product of a warp holds the
// block's SM for 16 cycles, and a tail of even 60 nodes was slower than the launches it
// replaced (FP64 loop at 160x80: 63.1 ms against 60.2).
constexpr int kTailNodes = 576;

template <class T, int NC>
struct TailSweep {
  struct Lev {
    int NX, NY;
    const T *st, *dinv, *cheb;
    Dir dir;
    int x, d;      // shared offsets of two vectors, rows of NX + 2 with a ring of zeros
    int b, row, di;  // right-hand side, rows and inverse diagonal (levels >= 1)
  };
  int nlev;        // smoothed levels; lv[nlev] is the coarsest, solved by cinv
  int vectors;     // shared values [0, vectors) start at zero
  int inv;         // shared offset of the inverse
  int shared;      // shared values in all
  const T* cinv;
  Lev lv[kTailMaxLevels + 1];

  // lays the shared memory out
  void plan() {
    auto align = [](int o) { return (o + 3) / 4 * 4; };
    int o = 0;
    for (int l = 0; l <= nlev; ++l) {
      // one more row and node of zeros: a padded coarse node sits one past the lattice, its
      // neighbours two (a column two past it is the next row's left ring)
      const int v = ((lv[l].NX + 2) * (lv[l].NY + 3) + 1) * NC, n = lv[l].NX * lv[l].NY;
      lv[l].x = o;
      lv[l].d = o + v;
      lv[l].b = o + 2 * v;
      o = align(o + 2 * v + n * NC);
    }
    vectors = o;
    for (int l = 1; l < nlev; ++l) {
      const int n = lv[l].NX * lv[l].NY;
      lv[l].row = o;
      o = align(o + n * StencilLayout<NC>::stride);
      lv[l].di = o;
      o = align(o + n * NC);
    }
    inv = o;
    const int m = lv[nlev].NX * lv[nlev].NY * NC;
    shared = o + m * m;
  }
};

}  // namespace topo
