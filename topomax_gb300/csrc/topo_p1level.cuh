// The V-cycle's two sweeps of a P1 level, one launch each:
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
// predecessor.  A level too large for an assembled stencil builds its rows from the
// triangles' coefficients instead (level_row_free).
#pragma once

#include "topo_p1.cuh"
#include "topo_p2.cuh"

namespace topo {

// Chebyshev steps of a sweep: two, or kCoarseDegree where a hierarchy asks for it (FP32 elasticity).
// Other counts have no kernels, and the coefficients of one polynomial are no prefix of another's.
constexpr int kCoarseDegree = 4;
template <class T>
constexpr int sweep_degree(int NC, int wanted) {
  return sizeof(T) == 4 && NC == 2 && wanted == kCoarseDegree ? kCoarseDegree : 2;
}

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

// one node's values (NC = 2: both at once, an address of twice their size)
template <class T, int NC>
TOPO_HD void load_node(const T* p, T (&v)[NC]) {
  if constexpr (NC == 2) ld2(p, v);
  else v[0] = p[0];
}
template <class T, int NC>
TOPO_HD void store_node(T* p, const T (&v)[NC]) {
  if constexpr (NC == 2) st2(p, v[0], v[1]);
  else p[0] = v[0];
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
// Results with either form are as far from 64-bit references to four digits (FP64 designs of
// 47x20 to 240x120: 5.533e-11, loops up to 160x80: 3.106e-12, geometric means).
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
  load_node<T, NC>(u + NC * p, un);
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
    load_node<T, NC>(u + NC * q, ul);
    if constexpr (sizeof(T) == 4)
      for (int c = 0; c < NC; ++c) ul[c] -= un[c];
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

// The row (not yet level_row) of node (a, b) from the coefficients of the level's triangles: what
// p1_stencil_node stores, in the level's precision.  A triangle's stiffness rows sum to zero, so
// the row sum of block 0 is the mass's, less the couplings that a clamped neighbour takes out.
// 48 products and 48 bytes of coefficients (shared with the neighbours) take the place of a load of
// 112 bytes: the rows of a level too large for L2.
template <class T, int NC>
TOPO_HD void level_row_free(const P1Params<T, NC>& Q, int a, int b, T (&st)[StencilLayout<NC>::stride]) {
  constexpr int SB = NC * NC;
  for (int i = 0; i < StencilLayout<NC>::stride; ++i) st[i] = T(0);
  // both triangles of the four cells around the node, zero outside the mesh
  T kk4[4][2], km4[4][2];
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
  for (int q = 0; q < 4; ++q) {
    const int ci = a - 1 + (q & 1), cj = b - 1 + (q >> 1);
    kk4[q][0] = kk4[q][1] = km4[q][0] = km4[q][1] = T(0);
    if (ci < 0 || ci >= Q.nx || cj < 0 || cj >= Q.ny) continue;
    const unsigned t = 2u * (unsigned(cj) * unsigned(Q.nx) + unsigned(ci));
    if (Q.kK) ld2(Q.kK + t, kk4[q]);
    else kk4[q][0] = kk4[q][1] = Q.kK_c;
    if constexpr (NC == 1) {
      if (Q.kM) ld2(Q.kM + t, km4[q]);
      else km4[q][0] = km4[q][1] = Q.kM_c;
    }
  }
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
  for (int e = 0; e < 6; ++e) {
    int dci, dcj, o, loc;
    p1_incidence(e, dci, dcj, o, loc);
    const T kk = kk4[dci + 1 + 2 * (dcj + 1)][o], km = km4[dci + 1 + 2 * (dcj + 1)][o];
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int L = 0; L < 3; ++L) {
      if constexpr (NC == 1) st[0] = fma_t(km, Q.Mm[o][loc][L], st[0]);
      if (L == loc) continue;
      T* bk = st + st_block(dci + p1_off_a(o, L), dcj + p1_off_b(o, L)) * SB;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
      for (int i = 0; i < SB; ++i) {
        bk[i] = fma_t(kk, Q.K[o][loc * NC + i / NC][L * NC + i % NC], bk[i]);
        if constexpr (NC == 1) bk[i] = fma_t(km, Q.Mm[o][loc][L], bk[i]);
      }
    }
  }
  if (!P1Kern<T, NC>::near_clamped(Q.dir, a, b)) return;
  const bool self = is_clamped(Q.dir, a, b);
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
  for (int k = 1; k < 7; ++k) {
    if (!self && !is_clamped(Q.dir, a + st_da(k), b + st_db(k))) continue;
    for (int i = 0; i < SB; ++i) {
      st[i] -= st[k * SB + i];
      st[k * SB + i] = T(0);
    }
  }
  if (self)
    for (int i = 0; i < SB; ++i) st[i] = i / NC == i % NC ? T(1) : T(0);
}

// A thread's node: what the two operator applications share.
template <class T, int NC>
struct LevelNode {
  int a, b;  // lattice position (may lie outside)
  bool in;
  T st[StencilLayout<NC>::stride];
  T di[NC], bv[NC];

  TOPO_HD void place(const LevelSweep<T, NC>& L, int a_, int b_) {
    a = a_;
    b = b_;
    in = a >= 0 && a < L.NX && b >= 0 && b < L.NY;
  }
  // row and inverse diagonal (zero outside the lattice); Q: the row from its coefficients
  TOPO_HD void load(const LevelSweep<T, NC>& L, const P1Params<T, NC>* Q = nullptr) {
    const unsigned n = in ? unsigned(b) * unsigned(L.NX) + unsigned(a) : 0u;
    load_node<T, NC>(L.dinv + NC * size_t(n), di);
    if (Q) {
      level_row_free<T, NC>(*Q, a, b, st);
    } else {
      const bool interior = L.inner && a > 0 && b > 0 && a < L.NX - 1 && b < L.NY - 1;
      load_row(interior ? L.inner : L.st + size_t(n) * StencilLayout<NC>::stride, st);
    }
    if (!in) {
      for (int i = 0; i < StencilLayout<NC>::stride; ++i) st[i] = T(0);
      for (int c = 0; c < NC; ++c) di[c] = T(0);
    }
    level_row<T, NC>(st);
  }
  TOPO_HD size_t index(const LevelSweep<T, NC>& L) const { return unsigned(b) * unsigned(L.NX) + unsigned(a); }
  TOPO_HD void load_b(const LevelSweep<T, NC>& L, const T* bg) {
    for (int c = 0; c < NC; ++c) bv[c] = T(0);
    if (in) load_node<T, NC>(bg + NC * index(L), bv);
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
    T cf[7];            // smoothing coefficients
  };
  // the thread's node of a region of w x h nodes from lattice position (a0, b0), and the
  // coefficients of D steps (its row and vectors come with load, load_b and up_own)
  template <int D>
  TOPO_HD static bool start(const L& P, int a0, int b0, int w, int h, int tid, Node& N) {
    for (int k = 0; k < 2 * D - 1; ++k) N.cf[k] = P.cheb[k];
    if (tid >= w * h) return false;
    const int i = int(unsigned(tid) % unsigned(w)), j = int(unsigned(tid) / unsigned(w));
    N.place(P, a0 + i, b0 + j);
    N.p = (j + 1) * (w + 2) + i + 1;
    return true;
  }
  // position i of the ring around the region, 0 <= i < ring_size: (column, row) of the shared vectors
  TOPO_HD static int ring_size(int w, int h) { return 2 * (w + 2) + 2 * h; }
  TOPO_HD static void ring_position(int i, int w, int h, int& u, int& v) {
    if (i < 2 * (w + 2)) {
      u = i < w + 2 ? i : i - (w + 2);
      v = i < w + 2 ? 0 : h + 1;
    } else {
      u = (i & 1) ? w + 1 : 0;
      v = ((i - 2 * (w + 2)) >> 1) + 1;
    }
  }
  // down: d0 = c0 Dinv b, at the thread's node (on) and in the ring around the region
  TOPO_HD static void down_first(const L& P, int a0, int b0, int w, int h, int tid, int nt, const T* b, T* s, bool on,
                                 Node& N) {
    const T c0 = N.cf[0];
    if (on) {
      for (int c = 0; c < NC; ++c) {
        N.r[c] = N.bv[c];
        N.x[c] = N.d[c] = (c0 * N.di[c]) * N.bv[c];
      }
      store_node<T, NC>(s + NC * N.p, N.d);
    }
    for (int i = tid; i < ring_size(w, h); i += nt) {
      int u, v;
      ring_position(i, w, h, u, v);
      const int a = a0 - 1 + u, c = b0 - 1 + v;
      T d[NC], bv[NC];
      for (int k = 0; k < NC; ++k) d[k] = T(0);
      if (a >= 0 && a < P.NX && c >= 0 && c < P.NY) {
        const size_t g = unsigned(c) * unsigned(P.NX) + unsigned(a);
        load_node<T, NC>(P.dinv + NC * g, d);
        load_node<T, NC>(b + NC * g, bv);
        for (int k = 0; k < NC; ++k) d[k] = (c0 * d[k]) * bv[k];
      }
      store_node<T, NC>(s + NC * (v * (w + 2) + u), d);
    }
  }
  // (x + P x_c) at node (a, b), zero outside the lattice
  TOPO_HD static void up_value(const L& P, int a, int b, const T* x, const T* xc, T (&v)[NC]) {
    for (int c = 0; c < NC; ++c) v[c] = T(0);
    if (a < 0 || a >= P.NX || b < 0 || b >= P.NY) return;
    // the node's two coarse neighbours, or twice the coarse node it is
    const unsigned m0 = unsigned(b >> 1) * unsigned(P.NXc) + unsigned(a >> 1),
                   m1 = unsigned((b + 1) >> 1) * unsigned(P.NXc) + unsigned((a + 1) >> 1);
    T y0[NC], y1[NC];
    load_node<T, NC>(x + NC * size_t(unsigned(b) * unsigned(P.NX) + unsigned(a)), v);
    load_node<T, NC>(xc + NC * size_t(m0), y0);
    load_node<T, NC>(xc + NC * size_t(m1), y1);
    const bool free = surely_free(P.dirf, a, b) || !is_clamped(P.dirf, a, b);
    for (int c = 0; c < NC; ++c) {
      const T y = m0 == m1 ? y0[c] : T(0.5) * (y0[c] + y1[c]);
      v[c] = free ? v[c] + y : v[c];
    }
  }
  // up: x + P x_c at the thread's node
  TOPO_HD static void up_own(const L& P, const T* x, const T* xc, Node& N) { up_value(P, N.a, N.b, x, xc, N.x); }
  // ... and in the ring around the region, to shared memory
  TOPO_HD static void up_first(const L& P, int a0, int b0, int w, int h, int tid, int nt, const T* x, const T* xc, T* s,
                               bool on, const Node& N) {
    if (on) store_node<T, NC>(s + NC * N.p, N.x);
    for (int i = tid; i < ring_size(w, h); i += nt) {
      int u, v;
      ring_position(i, w, h, u, v);
      T y[NC];
      up_value(P, a0 - 1 + u, b0 - 1 + v, x, xc, y);
      store_node<T, NC>(s + NC * (v * (w + 2) + u), y);
    }
  }
  // up: r = b - A x, d0 = c0 Dinv r, x += d0
  TOPO_HD static void up_residual(const L&, int w, const T* sx, T* sd, Node& N) {
    T t[NC];
    level_apply<T, NC>(N.st, sx, w + 2, N.p, t);
    const T c0 = N.cf[0];
    for (int c = 0; c < NC; ++c) {
      N.r[c] = N.bv[c] - t[c];
      N.d[c] = (c0 * N.di[c]) * N.r[c];
      N.x[c] += N.d[c];
    }
    store_node<T, NC>(sd + NC * N.p, N.d);
  }
  // step k >= 1: r -= A d, d = c1 d + c2 Dinv r, x += d; the direction from s to sn
  TOPO_HD static void step(const L&, int k, int w, const T* s, T* sn, Node& N) {
    T t[NC];
    level_apply<T, NC>(N.st, s, w + 2, N.p, t);
    const T c1 = N.cf[2 * k - 1], c2 = N.cf[2 * k];
    for (int c = 0; c < NC; ++c) {
      N.r[c] -= t[c];
      N.d[c] = level_direction(c1, N.d[c], c2, N.di[c], N.r[c]);
      N.x[c] += N.d[c];
    }
    store_node<T, NC>(sn + NC * N.p, N.d);
  }
  // the last step: x alone, to sn (the residual b - A x reads it)
  TOPO_HD static void last(const L&, int k, int w, const T* s, T* sn, Node& N) {
    T t[NC];
    level_apply<T, NC>(N.st, s, w + 2, N.p, t);
    const T c1 = N.cf[2 * k - 1], c2 = N.cf[2 * k];
    for (int c = 0; c < NC; ++c) N.x[c] = level_last(N.x[c], c1, N.d[c], c2, N.di[c], N.r[c] - t[c]);
    if (sn) store_node<T, NC>(sn + NC * N.p, N.x);
  }
  // down, at the end: r = b - A x (zero outside the lattice), to shared memory for the restriction
  TOPO_HD static void down_residual(int w, const T* s, T* sr, const Node& N) {
    T t[NC];
    level_apply<T, NC>(N.st, s, w + 2, N.p, t);
    for (int c = 0; c < NC; ++c) t[c] = N.bv[c] - t[c];
    store_node<T, NC>(sr + NC * N.p, t);
  }
  // stores the block's own nodes, of a region that starts `ring` nodes before them at (a0, b0)
  TOPO_HD static void store(const L& P, int a0, int b0, int ring, const Node& N, T* x) {
    const int i = N.a - a0 - ring, j = N.b - b0 - ring;
    if (!N.in || i < 0 || i >= 2 * P.cx || j < 0 || j >= 2 * P.cy) return;
    store_node<T, NC>(x + NC * N.index(P), N.x);
  }
  // ring: the position of the block's first coarse node inside the region
  TOPO_HD static void restrict_to(const L& P, int cx, int cy, int I0, int J0, int w, int ring, int tid, int nt,
                                  const T* sr, T* bc) {
    for (int i = tid; i < cx * cy; i += nt) {
      const int ic = int(unsigned(i) % unsigned(cx)), jc = int(unsigned(i) / unsigned(cx)), I = I0 + ic, J = J0 + jc;
      if (I >= P.NXc || J >= P.NYc) continue;
      const int p = (2 * jc + ring + 1) * (w + 2) + 2 * ic + ring + 1;
      const bool zero = is_clamped(P.dirc, I, J);
      T y[NC];
      for (int c = 0; c < NC; ++c) y[c] = zero ? T(0) : level_restrict<T, NC>(sr + NC * p + c, w + 2);
      store_node<T, NC>(bc + NC * size_t(unsigned(J) * unsigned(P.NXc) + unsigned(I)), y);
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
constexpr int kTailPhases = 2 * kTailMaxLevels + 2;  // down and up of each, the coarsest solve, the launches
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
  long long* trace;  // cycles of the phases (null: off)
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
