// The V-cycle's two sweeps of a P1 level with an assembled stencil, one launch each:
//   down:  x = two Chebyshev steps from zero, r = b - A x, b_c = P^T r
//   up:    x += P x_c, two Chebyshev steps
// A block owns cx x cy coarse nodes and the 2cx x 2cy fine nodes over them and
// recomputes the ring its own results need (three nodes wide down, two up), so
// that the steps between the loads and the stores go through shared memory.
// Such a level is bound by latency: six launches (two smoothing, a residual, a
// restriction, a prolongation and a smoothing step more) of 4 to 6 us each, for
// vectors that stay in L2.  A thread keeps its node's stencil row, inverse
// diagonal and right-hand side in registers through both operator applications;
// the rows and diagonals, which no solve changes, are loaded before the kernel
// waits for its predecessor.
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

  TOPO_HD int down_w() const { return 2 * cx + 3; }  // region of x
  TOPO_HD int down_h() const { return 2 * cy + 3; }
  TOPO_HD int up_w() const { return 2 * cx + 2; }  // region of d0
  TOPO_HD int up_h() const { return 2 * cy + 2; }
  // shared values: the region's vector and the next wider one's
  TOPO_HD int down_shared() const { return NC * (down_w() * down_h() + (down_w() + 2) * (down_h() + 2)); }
  TOPO_HD int up_shared() const { return NC * (up_w() * up_h() + (up_w() + 2) * (up_h() + 2)); }
};

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

// u + c1 u + c2 Dinv r : the second Chebyshev step's result from the first's (pre-smoothing),
// and x2 + c1 d + c2 Dinv r (post-smoothing)
template <class T>
TOPO_HD T level_step(T x, T c1, T d, T c2, T di, T r) {
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

// Phases of the down sweep; a barrier between one and the next.  tid, nt: the thread and the
// block's threads (at least down_w x down_h of them).
template <class T, int NC>
struct LevelDown {
  using L = LevelSweep<T, NC>;
  using Node = LevelNode<T, NC>;
  // the thread's node of the x region
  TOPO_HD static bool start(const L& P, int I0, int J0, int tid, Node& N) {
    if (tid >= P.down_w() * P.down_h()) return false;
    N.load(P, 2 * I0 - 2 + tid % P.down_w(), 2 * J0 - 2 + tid / P.down_w());
    return true;
  }
  // d0 = c0 Dinv b on the x region and a ring around it
  TOPO_HD static void first(const L& P, int I0, int J0, int tid, int nt, const T* b, T* sd) {
    const int w = P.down_w() + 2, n = w * (P.down_h() + 2);
    const T c0 = P.cheb[0];
    for (int i = tid; i < n; i += nt) {
      const int a = 2 * I0 - 3 + i % w, r = 2 * J0 - 3 + i / w;
      const bool in = a >= 0 && a < P.NX && r >= 0 && r < P.NY;
      const size_t g = in ? size_t(r) * P.NX + a : 0;
      for (int c = 0; c < NC; ++c) sd[NC * i + c] = in ? (c0 * P.dinv[NC * g + c]) * b[NC * g + c] : T(0);
    }
  }
  // x = d0 + d1, d1 = c1 d0 + c2 Dinv (b - A d0)
  TOPO_HD static void smooth(const L& P, int tid, const Node& N, const T* sd, T* sx, T* x) {
    const int w = P.down_w(), i = tid % w, j = tid / w;
    const T c1 = P.cheb[1], c2 = P.cheb[2];
    const int p = (j + 1) * (w + 2) + i + 1;
    T t[NC];
    level_apply<T, NC>(N.st, sd, w + 2, p, t);
    const bool own = N.in && i >= 2 && i < 2 + 2 * P.cx && j >= 2 && j < 2 + 2 * P.cy;
    for (int c = 0; c < NC; ++c) {
      const T u = sd[NC * p + c], r1 = N.bv[c] - t[c];
      const T v = level_step(u, c1, u, c2, N.di[c], r1);
      sx[NC * tid + c] = v;
      if (own) x[NC * N.index(P) + c] = v;
    }
  }
  // r = b - A x on the x region less its outer ring (zero outside the lattice); sr in the
  // layout of the x region
  TOPO_HD static void residual(const L& P, int tid, const Node& N, const T* sx, T* sr) {
    const int w = P.down_w(), i = tid % w, j = tid / w;
    if (i < 1 || i > w - 2 || j < 1 || j > P.down_h() - 2) return;
    T t[NC];
    level_apply<T, NC>(N.st, sx, w, tid, t);
    for (int c = 0; c < NC; ++c) sr[NC * tid + c] = N.bv[c] - t[c];
  }
  TOPO_HD static void restrict_to(const L& P, int I0, int J0, int tid, int nt, const T* sr, T* bc) {
    const int w = P.down_w();
    for (int i = tid; i < P.cx * P.cy; i += nt) {
      const int ic = i % P.cx, jc = i / P.cx, I = I0 + ic, J = J0 + jc;
      if (I >= P.NXc || J >= P.NYc) continue;
      const int p = (2 * jc + 2) * w + 2 * ic + 2;
      const bool zero = is_clamped(P.dirc, I, J);
      for (int c = 0; c < NC; ++c)
        bc[NC * (size_t(J) * P.NXc + I) + c] = zero ? T(0) : level_restrict<T, NC>(sr + NC * p + c, w);
    }
  }
};

// Phases of the up sweep.
template <class T, int NC>
struct LevelUp {
  using L = LevelSweep<T, NC>;
  struct Node : LevelNode<T, NC> {
    T r0[NC], d0[NC], x2[NC];
  };
  TOPO_HD static bool start(const L& P, int I0, int J0, int tid, Node& N) {
    if (tid >= P.up_w() * P.up_h()) return false;
    N.load(P, 2 * I0 - 1 + tid % P.up_w(), 2 * J0 - 1 + tid / P.up_w());
    return true;
  }
  // x + P x_c on the d0 region and a ring around it (zero outside the lattice)
  TOPO_HD static void correct(const L& P, int I0, int J0, int tid, int nt, const T* x, const T* xc, T* sx) {
    const int w = P.up_w() + 2, n = w * (P.up_h() + 2);
    for (int i = tid; i < n; i += nt) {
      const int a = 2 * I0 - 2 + i % w, b = 2 * J0 - 2 + i / w;
      const bool in = a >= 0 && a < P.NX && b >= 0 && b < P.NY;
      if (!in) {
        for (int c = 0; c < NC; ++c) sx[NC * i + c] = T(0);
        continue;
      }
      // the node's two coarse neighbours, or twice the coarse node it is
      const size_t m0 = size_t(b >> 1) * P.NXc + (a >> 1), m1 = size_t((b + 1) >> 1) * P.NXc + ((a + 1) >> 1);
      const bool free = !is_clamped(P.dirf, a, b);
      const size_t g = size_t(b) * P.NX + a;
      for (int c = 0; c < NC; ++c) {
        const T v = m0 == m1 ? xc[NC * m0 + c] : T(0.5) * (xc[NC * m0 + c] + xc[NC * m1 + c]);
        sx[NC * i + c] = free ? x[NC * g + c] + v : x[NC * g + c];
      }
    }
  }
  // r0 = b - A x, d0 = c0 Dinv r0, x2 = x + d0
  TOPO_HD static void first(const L& P, int tid, Node& N, const T* sx, T* sd) {
    const int w = P.up_w(), p = (tid / w + 1) * (w + 2) + tid % w + 1;
    const T c0 = P.cheb[0];
    T t[NC];
    level_apply<T, NC>(N.st, sx, w + 2, p, t);
    for (int c = 0; c < NC; ++c) {
      N.r0[c] = N.bv[c] - t[c];
      N.d0[c] = (c0 * N.di[c]) * N.r0[c];
      N.x2[c] = sx[NC * p + c] + N.d0[c];
      sd[NC * tid + c] = N.d0[c];
    }
  }
  // whether the thread's node is one the block writes
  TOPO_HD static bool owned(const L& P, int tid, const Node& N) {
    const int w = P.up_w(), i = tid % w, j = tid / w;
    return N.in && i >= 1 && i <= 2 * P.cx && j >= 1 && j <= 2 * P.cy;
  }
  // x = x2 + c1 d0 + c2 Dinv (r0 - A d0)
  TOPO_HD static void second(const L& P, int tid, const Node& N, const T* sd, T* x) {
    const T c1 = P.cheb[1], c2 = P.cheb[2];
    T t[NC];
    level_apply<T, NC>(N.st, sd, P.up_w(), tid, t);
    for (int c = 0; c < NC; ++c) {
      const T r1 = N.r0[c] - t[c];
      x[NC * N.index(P) + c] = level_step(N.x2[c], c1, N.d0[c], c2, N.di[c], r1);
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
