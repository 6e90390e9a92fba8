// Stokes-Brinkman state on the P2-P1 (Taylor-Hood) lattice: element tables,
// node incidence, the operator by output node and the per-triangle phases of the
// objective and the gradient's right-hand side.
//
// Follows FEM_src/fluid_problem.py:48-155 and src/penalizers.py:49-67:
//   a((u,p),(v,q)) = (alpha(rho) u, v) + (grad u, grad v) + (grad p, v) + (div u, q),
//   alpha(rho) = a_max + (a_min - a_max) rho (1 + q) / (rho + q),
//   objective 1/2 int alpha(rho) |u|^2 + mu |grad u|^2 dx,
//   gradient  = L2 projection onto CG1 of 1/2 alpha'(rho) |u|^2.
// The form compiler integrates the state form and the objective with a degree-6
// rule (Strang-Fix, 12 points) and the projection's right-hand side with the
// collapsed Gauss-Jacobi 4 x 4 rule (degree 7); the same rules are used here.
//
// Everything here compiles for host and device: the test emulator runs the
// operator's rows and the triangle phases on the CPU against the oracle.
#pragma once

#include <cmath>
#include <cstddef>

#include "topo_common.cuh"

namespace topo {

constexpr int kFluidQ6 = 12;
constexpr int kFluidQ7 = 16;
constexpr int kFluidMass = 21;   // upper triangle of the 6 x 6 alpha-weighted P2 mass matrix

// alpha(rho) and alpha'(rho) in the reference's operation order
struct FluidPenal {
  double q = 0.0, amin = 0.0, amax = 0.0;
  TOPO_HD double a(double rho) const { return amax + (amin - amax) * rho * (1 + q) / (rho + q); }
  TOPO_HD double da(double rho) const {
    const double s = rho + q;
    return (amin - amax) * q * (1 + q) / (s * s);
  }
};

// Element tables shared by every triangle of the lattice (both orientations
// have the same area; gradients differ).  Built once per context on the host.
struct FluidTables {
  double area;
  double lam6[kFluidQ6][3], w6[kFluidQ6];
  double lam7[kFluidQ7][3], w7[kFluidQ7];
  double N6[kFluidQ6][6], N7[kFluidQ7][6];
  double dN6[2][kFluidQ6][6][2];  // physical basis gradients at the degree-6 points
  double lap[2][6][6];            // int grad N_i . grad N_j
  double grad[2][6][2][3];        // int N_i d_c lambda_k    (velocity row (i,c), pressure vertex k)
  double div[2][3][6][2];         // int lambda_k d_c N_j    (pressure row k, velocity column (j,c))
};

TOPO_HD int fluid_mass_index(int i, int j) {  // i <= j
  return i * 6 - (i * (i - 1)) / 2 + (j - i);
}

// P2 basis [A, B, C, mid(BC), mid(AC), mid(AB)] at barycentric point l
TOPO_HD void p2_values(const double (&l)[3], double (&N)[6]) {
  N[0] = l[0] * (2 * l[0] - 1);
  N[1] = l[1] * (2 * l[1] - 1);
  N[2] = l[2] * (2 * l[2] - 1);
  N[3] = 4 * l[1] * l[2];
  N[4] = 4 * l[0] * l[2];
  N[5] = 4 * l[0] * l[1];
}

TOPO_HD bool fluid_boundary_node(int a, int b, int NX, int NY) {
  return a == 0 || b == 0 || a == NX - 1 || b == NY - 1;
}

// rho at the three vertices of triangle t (cell-major, orientation t & 1)
TOPO_HD void fluid_tri_rho(const double* rho, int nx, size_t t, double (&r)[3]) {
  const int o = int(t & 1);
  const size_t cell = t >> 1;
  const int i = int(cell % nx), j = int(cell / nx);
  for (int k = 0; k < 3; ++k) r[k] = rho[size_t(j + p1_off_b(o, k)) * (nx + 1) + i + p1_off_a(o, k)];
}

TOPO_HD void fluid_tri_nodes(int nx, size_t t, size_t (&n)[6]) {
  const int o = int(t & 1);
  const size_t cell = t >> 1;
  const int i = int(cell % nx), j = int(cell / nx);
  const int NX = 2 * nx + 1;
  for (int k = 0; k < 6; ++k) n[k] = size_t(2 * j + p2_off_b(o, k)) * NX + 2 * i + p2_off_a(o, k);
}

// The alpha-weighted P2 mass matrix of triangle t (upper triangle, kFluidMass values):
// area * sum_q w_q alpha(rho_q) N_i(q) N_j(q), rho_q interpolated from the vertices.
TOPO_HD void fluid_tri_mass(const FluidTables& E, const FluidPenal& pen, const double (&r)[3], double* m) {
  double aw[kFluidQ6];
  for (int q = 0; q < kFluidQ6; ++q) {
    const double rq = r[0] * E.lam6[q][0] + r[1] * E.lam6[q][1] + r[2] * E.lam6[q][2];
    aw[q] = pen.a(rq) * E.w6[q];
  }
  for (int i = 0; i < 6; ++i)
    for (int j = i; j < 6; ++j) {
      double s = 0.0;
      for (int q = 0; q < kFluidQ6; ++q) s += aw[q] * E.N6[q][i] * E.N6[q][j];
      m[fluid_mass_index(i, j)] = E.area * s;
    }
}

// Objective integrand of triangle t: area * sum_q w_q (alpha |u|^2 + mu |grad u|^2)
TOPO_HD double fluid_tri_objective(const FluidTables& E, const FluidPenal& pen, double mu, int o,
                                   const double (&r)[3], const double (&ue)[6][2]) {
  double s = 0.0;
  for (int q = 0; q < kFluidQ6; ++q) {
    const double rq = r[0] * E.lam6[q][0] + r[1] * E.lam6[q][1] + r[2] * E.lam6[q][2];
    double u0 = 0.0, u1 = 0.0, g00 = 0.0, g01 = 0.0, g10 = 0.0, g11 = 0.0;
    for (int k = 0; k < 6; ++k) {
      u0 += E.N6[q][k] * ue[k][0];
      u1 += E.N6[q][k] * ue[k][1];
      g00 += E.dN6[o][q][k][0] * ue[k][0];
      g01 += E.dN6[o][q][k][1] * ue[k][0];
      g10 += E.dN6[o][q][k][0] * ue[k][1];
      g11 += E.dN6[o][q][k][1] * ue[k][1];
    }
    const double f = pen.a(rq) * (u0 * u0 + u1 * u1) + mu * (g00 * g00 + g01 * g01 + g10 * g10 + g11 * g11);
    s += f * E.w6[q];
  }
  return E.area * s;
}

// Gradient right-hand side of triangle t: out[k] = int 1/2 alpha'(rho) |u|^2 lambda_k
// with the degree-7 rule.
TOPO_HD void fluid_tri_gradient(const FluidTables& E, const FluidPenal& pen, const double (&r)[3],
                                const double (&ue)[6][2], double (&out)[3]) {
  out[0] = out[1] = out[2] = 0.0;
  for (int q = 0; q < kFluidQ7; ++q) {
    const double rq = r[0] * E.lam7[q][0] + r[1] * E.lam7[q][1] + r[2] * E.lam7[q][2];
    double u0 = 0.0, u1 = 0.0;
    for (int k = 0; k < 6; ++k) {
      u0 += E.N7[q][k] * ue[k][0];
      u1 += E.N7[q][k] * ue[k][1];
    }
    const double f = 0.5 * pen.da(rq) * (u0 * u0 + u1 * u1) * E.w7[q] * E.area;
    for (int k = 0; k < 3; ++k) out[k] += f * E.lam7[q][k];
  }
}

// ---------------------------------------------------------------------------
// the operator by output node
// ---------------------------------------------------------------------------
// P2 nodes by class: 0 vertices, midpoints of 1 horizontal, 2 vertical and 3 diagonal edges, so
// that the threads of a block do the same work.  The continuity rows are negated, which makes the
// operator symmetric on velocities that vanish on the boundary; (i, j): column and row of the vertex, or of
// the edge's lower left vertex.  (Class 4 in the kernels: the pressure vertices.)

// Incident triangles of a class's nodes, a byte each: column offset + 1 | (row offset + 1) << 1 |
// orientation << 2 | local index << 3 (six of a vertex, two of an edge)
TOPO_HD constexpr unsigned long long fluid_incidence(int cls) {
  return cls == 0 ? 0x07030a0d1410ull : cls == 1 ? 0x2b1dull : cls == 2 ? 0x2f1aull : 0x2723ull;
}
TOPO_HD constexpr int fluid_incidences(int cls) { return cls == 0 ? 6 : 2; }

// Offsets (in lattice steps) of the P2 nodes a class's node couples to: 19 of a vertex, 9 of an
// edge, and of the CG1 vertices (in cells, from (i, j)) its gradient row reads: 7 and 4.
constexpr int kFluidNodes = 19, kFluidEdgeNodes = 9, kFluidVerts = 7, kFluidEdgeVerts = 4;
TOPO_HD constexpr int fluid_nodes(int cls) { return cls == 0 ? kFluidNodes : kFluidEdgeNodes; }
TOPO_HD constexpr int fluid_verts(int cls) { return cls == 0 ? kFluidVerts : kFluidEdgeVerts; }
struct FluidOffset {
  signed char a, b;
};
template <int CLS>
TOPO_HD constexpr FluidOffset fluid_node_offset(int k) {
  if (CLS == 0) {  // both cells on the diagonal, then the two corners the other triangles add
    const FluidOffset t[kFluidNodes] = {{0, 0},   {1, 0},   {2, 0},   {0, 1},   {1, 1},  {2, 1},  {0, 2},
                                        {1, 2},   {2, 2},   {-1, 0},  {-2, 0},  {0, -1}, {-1, -1}, {-2, -1},
                                        {0, -2},  {-1, -2}, {-2, -2}, {1, -1},  {-1, 1}};
    return t[k];
  }
  if (CLS == 1) {  // triangle above (0: from the left vertex) and below the edge
    const FluidOffset t[kFluidEdgeNodes] = {{0, 0}, {-1, 0}, {1, 0}, {1, 1}, {0, 1}, {1, 2}, {-1, -1}, {-1, -2}, {0, -1}};
    return t[k];
  }
  if (CLS == 2) {
    const FluidOffset t[kFluidEdgeNodes] = {{0, 0}, {0, -1}, {0, 1}, {1, 1}, {1, 0}, {2, 1}, {-1, -1}, {-2, -1}, {-1, 0}};
    return t[k];
  }
  const FluidOffset t[kFluidEdgeNodes] = {{0, 0}, {-1, -1}, {1, 1}, {1, -1}, {0, -1}, {1, 0}, {-1, 1}, {-1, 0}, {0, 1}};
  return t[k];
}
template <int CLS>
TOPO_HD constexpr FluidOffset fluid_vert_offset(int k) {
  if (CLS == 0) {
    const FluidOffset t[kFluidVerts] = {{0, 0}, {1, 0}, {0, 1}, {1, 1}, {-1, 0}, {0, -1}, {-1, -1}};
    return t[k];
  }
  if (CLS == 1) {
    const FluidOffset t[kFluidEdgeVerts] = {{0, 0}, {1, 0}, {1, 1}, {0, -1}};
    return t[k];
  }
  if (CLS == 2) {
    const FluidOffset t[kFluidEdgeVerts] = {{0, 0}, {0, 1}, {1, 1}, {-1, 0}};
    return t[k];
  }
  const FluidOffset t[kFluidEdgeVerts] = {{0, 0}, {1, 0}, {0, 1}, {1, 1}};
  return t[k];
}

// The velocity rows' matrix entries live in memory class by class, entry k of all the class's
// nodes together: offset of the class's entries, and the number of all.
struct FluidRows {
  size_t count[4];   // nodes of a class
  size_t first[4];   // its entries
  size_t size;
  TOPO_HD FluidRows(int nx, int ny) : count{size_t(nx + 1) * (ny + 1), size_t(nx) * (ny + 1), size_t(nx + 1) * ny, size_t(nx) * ny} {
    size = 0;
    for (int c = 0; c < 4; ++c) {
      first[c] = size;
      size += count[c] * fluid_nodes(c);
    }
  }
};

// The gradient's and the divergence's coefficients depend only on which sides the node lies on:
// type 0, 1, 2 for the first, an inner, the last column (and row).  Built by fluid_stencils.
struct FluidStencils {
  double gv[9][kFluidVerts][2];      // vertex velocity rows, type = column type + 3 row type
  double ge[3][3][kFluidEdgeVerts][2];  // edges: [class - 1][type across the edge]
  double dv[9][kFluidNodes][2];      // pressure vertices, over the vertex node offsets
};

// Row of velocity node (class CLS, position (i, j)) from the triangles' matrices M + K.
template <int CLS>
TOPO_HD void fluid_build_row(const double* mk, int nx, int ny, int i, int j, double (&row)[kFluidNodes]) {
  for (int k = 0; k < fluid_nodes(CLS); ++k) row[k] = 0.0;
  // the node's own position inside its cell-based frame: (a, b) = (2 i + da, 2 j + db)
  const int da = CLS & 1, db = CLS >> 1;
  for (int e = 0; e < fluid_incidences(CLS); ++e) {
    const unsigned f = unsigned(fluid_incidence(CLS) >> (8 * e)) & 255u;
    const int ci = int(f & 1u) - 1, cj = int((f >> 1) & 1u) - 1, o = int((f >> 2) & 1u), r = int(f >> 3);
    if (i + ci < 0 || i + ci >= nx || j + cj < 0 || j + cj >= ny) continue;
    const double* m = mk + ((size_t(j + cj) * nx + i + ci) * 2 + o) * kFluidMass;
    for (int q = 0; q < 6; ++q) {
      const int oa = 2 * ci + p2_off_a(o, q) - da, ob = 2 * cj + p2_off_b(o, q) - db;
      for (int k = 0; k < fluid_nodes(CLS); ++k) {
        const FluidOffset t = fluid_node_offset<CLS>(k);
        if (t.a == oa && t.b == ob) row[k] += r <= q ? m[fluid_mass_index(r, q)] : m[fluid_mass_index(q, r)];
      }
    }
  }
}

TOPO_HD int fluid_side(int k, int n) { return k == 0 ? 0 : k == n ? 2 : 1; }

// Velocity rows of node (i, j) of class CLS, entry k of its matrix row at row[k * stride]: y.
// pm: a constant taken off the pressure.
template <int CLS>
TOPO_HD void fluid_velocity(const FluidStencils& S, const double* row, size_t stride, int nx, int ny, int i, int j,
                            const double* u, const double* p, double pm, double (&y)[2]) {
  const int NX = 2 * nx + 1, NY = 2 * ny + 1, a = 2 * i + (CLS & 1), b = 2 * j + (CLS >> 1);
  y[0] = y[1] = 0.0;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
  for (int k = 0; k < fluid_nodes(CLS); ++k) {
    const FluidOffset t = fluid_node_offset<CLS>(k);
    const int aa = a + t.a, bb = b + t.b;
    if (aa < 0 || aa >= NX || bb < 0 || bb >= NY) continue;
    const size_t nd = size_t(bb) * NX + aa;
    const double m = row[size_t(k) * stride];
    y[0] += m * u[2 * nd];
    y[1] += m * u[2 * nd + 1];
  }
  const int type = CLS == 0 ? fluid_side(i, nx) + 3 * fluid_side(j, ny) : CLS == 1 ? fluid_side(j, ny)
                   : CLS == 2 ? fluid_side(i, nx) : 1;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
  for (int k = 0; k < fluid_verts(CLS); ++k) {
    const FluidOffset t = fluid_vert_offset<CLS>(k);
    const int ii = i + t.a, jj = j + t.b;
    if (ii < 0 || ii > nx || jj < 0 || jj > ny) continue;
    const double q = p[size_t(jj) * (nx + 1) + ii] - pm;
    const double* g = CLS == 0 ? S.gv[type][k] : S.ge[CLS == 0 ? 0 : CLS - 1][CLS == 0 ? 0 : type][CLS == 0 ? 0 : k];
    y[0] += g[0] * q;
    y[1] += g[1] * q;
  }
}

// y at the k-th velocity node of class CLS, from the assembled rows (FluidRows).  clamp: boundary
// rows are the identity.
template <int CLS>
TOPO_HD void fluid_apply_class(int nx, int ny, const FluidStencils& S, const double* rows,
                                                  const FluidRows& R, size_t k, const double* x, double pm, bool clamp,
                                                  double* y) {
  const int NX = 2 * nx + 1, NY = 2 * ny + 1, w = CLS & 1 ? nx : nx + 1;
  const int i = int(k % w), j = int(k / w), a = 2 * i + (CLS & 1), b = 2 * j + (CLS >> 1);
  const size_t node = size_t(b) * NX + a;
  double v[2];
  if (clamp && fluid_boundary_node(a, b, NX, NY)) {
    v[0] = x[2 * node];
    v[1] = x[2 * node + 1];
  } else {
    fluid_velocity<CLS>(S, rows + R.first[CLS] + k, R.count[CLS], nx, ny, i, j, x, x + 2 * size_t(NX) * NY, pm, v);
  }
  y[2 * node] = v[0];
  y[2 * node + 1] = v[1];
}

// Continuity row of vertex (i, j)
TOPO_HD double fluid_continuity(const FluidStencils& S, int nx, int ny, int i, int j, const double* u) {
  const int NX = 2 * nx + 1, NY = 2 * ny + 1, type = fluid_side(i, nx) + 3 * fluid_side(j, ny);
  double s0 = 0.0, s1 = 0.0;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
  for (int k = 0; k < kFluidNodes; ++k) {
    const FluidOffset t = fluid_node_offset<0>(k);
    const int aa = 2 * i + t.a, bb = 2 * j + t.b;
    if (aa < 0 || aa >= NX || bb < 0 || bb >= NY) continue;
    const size_t nd = size_t(bb) * NX + aa;
    s0 += S.dv[type][k][0] * u[2 * nd];
    s1 += S.dv[type][k][1] * u[2 * nd + 1];
  }
  return -(s0 + s1);
}

}  // namespace topo
