// Reference formulas, test only: the smoothing modes of a P1 level written node by node in the
// product's node operator (what the march kernels' phases are compared with), and the incidence
// of the P2 nodes by their parity.
#pragma once

#include "topo_p1.cuh"

namespace topo {

// PRE input: first step from x = 0, d0 = c0 Dinv b, computed per node
template <class T, int NC>
struct FetchPre {
  const T* b;
  const T* dinv;
  T c0;
  TOPO_HD void operator()(size_t m, int, int, T (&v)[NC]) const {
    for (int d = 0; d < NC; ++d) v[d] = c0 * dinv[NC * m + d] * b[NC * m + d];
  }
};

template <class T, int NC>
struct P1Smooth {
  // PRE: x = d0 + d1 with d0 = c0 Dinv b, r1 = b - A d0, d1 = c1 d0 + c2 Dinv r1
  template <class PP>
  TOPO_HD static void pre(int a, int b, const PP& P, const SmoothBufs<T>& B) {
    const int NX = P.nx + 1;
    const size_t n = size_t(b) * NX + a;
    const T c0 = B.cheb[0], c1 = B.cheb[1], c2 = B.cheb[2];
    const FetchPre<T, NC> f{B.b, B.dinv, c0};
    T t[NC], u[NC];
    f(n, a, b, u);
    if (!p1_node_eval<T, NC>(a, b, P, f, t))
      for (int c = 0; c < NC; ++c) t[c] = u[c];
    for (int c = 0; c < NC; ++c) {
      const size_t i = NC * n + c;
      const T r1 = B.b[i] - t[c];
      B.x[i] = u[c] + c1 * u[c] + c2 * B.dinv[i] * r1;
    }
  }
  // RES: r = b - A x
  template <class PP>
  TOPO_HD static void res(int a, int b, const PP& P, const SmoothBufs<T>& B) {
    const int NX = P.nx + 1;
    const size_t n = size_t(b) * NX + a;
    T t[NC];
    if (!p1_node_eval<T, NC>(a, b, P, FetchArray<T, NC>{B.x}, t))
      for (int c = 0; c < NC; ++c) t[c] = B.x[NC * n + c];
    for (int c = 0; c < NC; ++c) B.r[NC * n + c] = B.b[NC * n + c] - t[c];
  }
  // FIRST (after the coarse correction was added to x):
  // r0 = b - A x ; d0 = c0 Dinv r0 ; x2 = x + d0 (writes r, d, x2)
  template <class PP>
  TOPO_HD static void first(int a, int b, const PP& P, const SmoothBufs<T>& B) {
    const int NX = P.nx + 1;
    const size_t n = size_t(b) * NX + a;
    const T c0 = B.cheb[0];
    T t[NC];
    if (!p1_node_eval<T, NC>(a, b, P, FetchArray<T, NC>{B.x}, t))
      for (int c = 0; c < NC; ++c) t[c] = B.x[NC * n + c];
    for (int c = 0; c < NC; ++c) {
      const size_t i = NC * n + c;
      const T r0 = B.b[i] - t[c];
      const T d0 = c0 * B.dinv[i] * r0;
      B.r[i] = r0;
      B.d[i] = d0;
      B.x2[i] = B.x[i] + d0;
    }
  }
  // POST2: r1 = r0 - A d0 ; d1 = c1 d0 + c2 Dinv r1 ; x = x2 + d1
  template <class PP>
  TOPO_HD static void post2(int a, int b, const PP& P, const SmoothBufs<T>& B) {
    const int NX = P.nx + 1;
    const size_t n = size_t(b) * NX + a;
    const T c1 = B.cheb[1], c2 = B.cheb[2];
    const FetchArray<T, NC> f{B.d};
    T t[NC];
    if (!p1_node_eval<T, NC>(a, b, P, f, t))
      for (int c = 0; c < NC; ++c) t[c] = B.d[NC * n + c];
    for (int c = 0; c < NC; ++c) {
      const size_t i = NC * n + c;
      const T r1 = B.r[i] - t[c];
      B.x[i] = B.x2[i] + c1 * B.d[i] + c2 * B.dinv[i] * r1;
    }
  }
};

// Triangles incident to P2 node (a, b) of the (2nx+1) x (2ny+1) lattice, with
// the node's local index in each; a fixed order (cell row, cell column,
// orientation).  Returns the count (at most 6).
TOPO_HD int p2_node_incidence(int a, int b, int nx, int ny, size_t (&tri)[6], int (&loc)[6]) {
  int n = 0;
  for (int j = b / 2 - 1; j <= b / 2; ++j) {
    if (j < 0 || j >= ny || b - 2 * j > 2) continue;
    for (int i = a / 2 - 1; i <= a / 2; ++i) {
      if (i < 0 || i >= nx || a - 2 * i > 2) continue;
      for (int o = 0; o < 2; ++o)
        for (int k = 0; k < 6; ++k)
          if (p2_off_a(o, k) == a - 2 * i && p2_off_b(o, k) == b - 2 * j) {
            tri[n] = (size_t(j) * nx + i) * 2 + o;
            loc[n] = k;
            ++n;
          }
    }
  }
  return n;
}

}  // namespace topo
