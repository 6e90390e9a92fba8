// The density filter's weights by table (DEM_src/filter.py:8-31).
//
// A weight is radius - sqrt(dx*dx + dy*dy) with dx, dy the differences of two
// rounded np.linspace points, so |dx| takes a handful of values per column offset
// (1 to 15 that differ in the last bits: 404 values over the 53 offsets of 600
// points at radius 0.1732) and |dy| likewise: all weights fit a table of
// (values of dy) x (values of dx) entries, 1 MB at 600 x 300, and the square
// root leaves the neighbour loop.  The normalisation weight / row sum is the
// correctly rounded FP64 quotient, formed on the integer pipe from a 64-bit
// reciprocal of the row sum (GB300 issues FP64 at 1/64 of its FP32 rate), so
// that a neighbour costs two FP64 operations, the product and the ordered sum.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "topo_common.cuh"

namespace topo {

constexpr int kDensNone = 0xffff;                  // class of a neighbour outside the mesh
constexpr size_t kDensTableMax = size_t(1) << 23;  // weights in the table (64 MB)
constexpr size_t kDensIndexMax = size_t(1) << 23;  // classes per axis array

// floor((2^127 - 1) / m), m the significand of s shifted to 64 bits (s normal, > 0)
TOPO_HD uint64_t dens_reciprocal(double s) {
  uint64_t b;
  memcpy(&b, &s, 8);
  const uint64_t m = (b << 11) | (uint64_t(1) << 63);
  const unsigned __int128 num = ~(unsigned __int128)0 >> 1;
  return uint64_t(num / m);
}

TOPO_HD uint64_t dens_mulhi(uint64_t a, uint64_t b) {
#if defined(__CUDA_ARCH__)
  return __umul64hi(a, b);
#else
  return uint64_t(((unsigned __int128)a * b) >> 64);
#endif
}

// w / s rounded to nearest, r = dens_reciprocal(s); w >= 0, w and the quotient zero
// or normal.  With A and m the 64-bit significands, P = mulhi(A, r) lies in
// (P* - 2.01, P*] for the exact P* = 2^63 A / m in (2^62, 2^64): the rounded significand
// follows from P unless its discarded bits are within 3 below one half (a quotient of two
// 53-bit numbers is never exactly halfway), where the division itself decides.
TOPO_HD double dens_quotient(double w, double s, uint64_t r) {
  uint64_t wb, sb;
  memcpy(&wb, &w, 8);
  memcpy(&sb, &s, 8);
  if (wb == 0) return w;
  const uint64_t P = dens_mulhi((wb << 11) | (uint64_t(1) << 63), r);
  const unsigned top = unsigned(P >> 63), sh = 10 + top;
  const uint64_t half = uint64_t(512) << top;
  const uint64_t low = P & (2 * half - 1);
  if (low < half && low >= half - 3) return w / s;
  const uint64_t q = (P + half) >> sh;  // in [2^52, 2^53]; the carry of 2^53 raises the exponent
  const uint64_t e = (wb >> 52) - (sb >> 52) + (1021 + top);  // biased exponent - 1
  const uint64_t ob = (e << 52) + q;
  double out;
  memcpy(&out, &ob, 8);
  return out;
}

// One axis of the filter: for every offset o in [-reach, reach] and point k the class of
// |x[k + o] - x[k]| (offset-major, kDensNone outside), and the classes' values.
struct DensAxis {
  int reach = 0;
  std::vector<uint16_t> cls;   // (2 reach + 1) x n
  std::vector<double> value;   // distinct |differences|, grouped by |offset|
  std::vector<double> least;   // smallest of each |offset| (reach + 1)
};

// np.linspace(0, L, n)[k]: k * step, the end point exact
TOPO_HD double dens_point(int k, int n, double L, double step) {
  if (n <= 1) return 0.0;
#if defined(__CUDA_ARCH__)
  return k == n - 1 ? L : __dmul_rn(double(k), step);
#else
  return k == n - 1 ? L : double(k) * step;
#endif
}

// false: too many classes or entries for the table
inline bool dens_axis(int n, double L, double step, int reach, DensAxis& A) {
  reach = reach < n - 1 ? reach : n - 1;
  A.reach = reach;
  if (size_t(2 * reach + 1) * size_t(n) > kDensIndexMax) return false;
  A.cls.assign(size_t(2 * reach + 1) * n, uint16_t(kDensNone));
  std::vector<double> x(n);
  for (int k = 0; k < n; ++k) x[k] = dens_point(k, n, L, step);
  for (int o = 0; o <= reach; ++o) {
    const size_t first = A.value.size();
    for (int k = 0; k + o < n; ++k) {
      const double d = std::fabs(x[k + o] - x[k]);
      size_t c = first;
      while (c < A.value.size() && A.value[c] != d) ++c;
      if (c == A.value.size()) A.value.push_back(d);
      if (c >= size_t(kDensNone)) return false;
      A.cls[size_t(reach + o) * n + k] = uint16_t(c);
      A.cls[size_t(reach - o) * n + k + o] = uint16_t(c);
    }
    double lo = A.value[first];
    for (size_t c = first; c < A.value.size(); ++c) lo = A.value[c] < lo ? A.value[c] : lo;
    A.least.push_back(lo);
  }
  return true;
}

// widest column offset with a neighbour within the radius, per |row offset| (-1: none)
inline std::vector<int> dens_half_widths(const DensAxis& X, const DensAxis& Y, double radius) {
  std::vector<int> h(Y.reach + 1, -1);
  for (int oy = 0; oy <= Y.reach; ++oy) {
    const double dy2 = Y.least[oy] * Y.least[oy];
    for (int ox = 0; ox <= X.reach; ++ox)
      if (std::sqrt(X.least[ox] * X.least[ox] + dy2) <= radius) h[oy] = ox;
  }
  return h;
}

struct alignas(16) DensRow {  // a row's sum and its reciprocal, one 16-byte load
  uint64_t r;
  double s;
};

struct DensTable {
  int Nx, Ny, rx, ry, ncx;
  const uint16_t* cx;  // [2 rx + 1][Nx]
  const uint16_t* cy;  // [2 ry + 1][Ny]
  const int* half;     // [ry + 1]
  const double* w;     // [classes of y][classes of x]: weight, or -1 outside the radius
};

// f(column j, weight) for the neighbours of element i in ascending j (the sign of an
// excluded entry is read as an integer: a comparison would occupy the FP64 pipe)
template <class F>
TOPO_HD void dens_table_row(const DensTable& T, int i, F&& f) {
  const int iy = i / T.Nx, ix = i - iy * T.Nx;
  for (int oy = -T.ry; oy <= T.ry; ++oy) {
    const int cy = T.cy[size_t(oy + T.ry) * T.Ny + iy];
    if (cy == kDensNone) continue;
    const int h = T.half[oy < 0 ? -oy : oy];
    const double* wr = T.w + size_t(cy) * T.ncx;
    const uint16_t* cx = T.cx + size_t(T.rx - h) * T.Nx + ix;
    const int j0 = i + oy * T.Nx - h;
#if defined(__CUDA_ARCH__)
#pragma unroll 4
#endif
    for (int k = 0; k <= 2 * h; ++k) {
      const int c = cx[size_t(k) * T.Nx];
      if (c == kDensNone) continue;
      const double w = wr[c];
      int64_t wb;
      memcpy(&wb, &w, 8);
      if (wb >= 0) f(j0 + k, w);
    }
  }
}

}  // namespace topo
