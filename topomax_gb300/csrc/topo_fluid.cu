// C ABI of the Stokes-Brinkman fluid problem (FEM_src/fluid_problem.py:48-155):
// Taylor-Hood state solve, objective and CG1-projected gradient, FP64.
//
// State solve: the Dirichlet velocity rows (every side carries data: the flow
// profiles of BoundaryFlows or no slip) are eliminated, which leaves the
// symmetric saddle point [A B^T; B 0] (A = alpha-weighted P2 mass + vector
// Laplacian, B = -(div u, q)).  Its pressure is fixed up to a constant and the
// interpolated boundary data carry a small mass defect, so the continuity
// right-hand side is projected to zero sum and the pressure kept at zero sum
// (the reduced system's least-squares closure).  Flexible GMRES, right
// preconditioned with the block-diagonal
//   diag( P1-iso-P2 V-cycles of K + alpha M on the (2nx)x(2ny) lattice, one per component,
//         lumped-mass inverse + V-cycle of the 1/alpha-weighted P1 Laplacian )
// (a variable-coefficient Cahouet-Chabard Schur-complement approximation).  Everything is FP64;
// the V-cycles take both velocity components in one batch, the pressure's run beside them.
// (V-cycles in FP32 gave the same iterations and errors at 0.65 to 0.75 of the time, but the entry
// points promise FP64 and have no precision for the caller to choose.)  One restart cycle is one
// CUDA graph whose WHILE body is an iteration; the Givens rotations and the stopping test
// run on the device.
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "topomax_gb300.h"
#include "topo_fluid.cuh"
#include "topo_mg_impl.cuh"
#include "topo_fluid_setup.h"
#include "topo_krylov.cuh"
#include "topo_sens.cuh"
#include "topo_setup.h"

namespace topo {
extern template class MG<double>;
}  // namespace topo

using namespace topo;

namespace {

static_assert(kFluidRestartLong <= kKrylovMax, "the cycle's scalars");
constexpr double kLaplaceShift = 1e-3;  // mass shift of the pressure Laplacian (its constant mode)

// ---------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------
__global__ void k_fluid_mass(int nx, int ny, const FluidTables* __restrict__ E, FluidPenal pen,
                             const double* __restrict__ rho, double* __restrict__ mass) {
  const size_t nt = size_t(2) * nx * ny;
  TOPO_GRID_STRIDE(t, nt) {
    double r[3];
    fluid_tri_rho(rho, nx, t, r);
    double* m = mass + t * kFluidMass;
    fluid_tri_mass(*E, pen, r, m);
    for (int i = 0; i < 6; ++i)
      for (int j = i; j < 6; ++j) m[fluid_mass_index(i, j)] += E->lap[t & 1][i][j];
  }
}

// Blocks of the operator's kernels by class (topo_fluid.cuh): class c has blocks [start[c], start[c + 1])
constexpr int kFluidThreads = 64;
struct FluidGrid {
  unsigned start[6];
  FluidGrid(int nx, int ny) {
    const FluidRows R(nx, ny);
    start[0] = 0;
    for (int c = 0; c < 5; ++c)
      start[c + 1] = start[c] + unsigned((R.count[c < 4 ? c : 0] + kFluidThreads - 1) / kFluidThreads);
  }
};

// the thread's class and index among the class's nodes; false past the last one
__device__ __forceinline__ bool fluid_thread(const FluidGrid& G, const FluidRows& R, int& cls, size_t& k) {
  cls = 0;
  while (cls < 4 && blockIdx.x >= G.start[cls + 1]) ++cls;
  k = size_t(blockIdx.x - G.start[cls]) * kFluidThreads + threadIdx.x;
  return k < R.count[cls < 4 ? cls : 0];
}

// the velocity rows of the design, from the triangles' matrices (once per solve)
__global__ void __launch_bounds__(kFluidThreads)
    k_fluid_rows(int nx, int ny, FluidGrid G, const double* __restrict__ mk, double* __restrict__ rows) {
  const FluidRows R(nx, ny);
  int cls;
  size_t k;
  if (!fluid_thread(G, R, cls, k)) return;
  const int w = cls & 1 ? nx : nx + 1, i = int(k % w), j = int(k / w);
  double row[kFluidNodes];
  switch (cls) {
    case 0: fluid_build_row<0>(mk, nx, ny, i, j, row); break;
    case 1: fluid_build_row<1>(mk, nx, ny, i, j, row); break;
    case 2: fluid_build_row<2>(mk, nx, ny, i, j, row); break;
    default: fluid_build_row<3>(mk, nx, ny, i, j, row); break;
  }
  for (int e = 0; e < fluid_nodes(cls); ++e) rows[R.first[cls] + size_t(e) * R.count[cls] + k] = row[e];
}

// y = A x, x = [u (2 n2, interleaved) | p (nv)], by output node: assembled velocity rows, and
// gradient and divergence coefficients by node type.  KRYLOV: x = z_j with its pressure's mean
// taken off, y = v_(j+1).  clamp: boundary velocity rows are the identity.
// Bound: FP64, 42 products per P2 node on average (the triangles' matrices applied where they are
// needed take 72), all loads of a row in flight at once: 10.6 us at 128x128, 6.2 at 40x40; by
// triangle rows 19.6 and 17.4, through a per-triangle buffer and a gather 22 and 20.
template <bool KRYLOV>
__global__ void __launch_bounds__(kFluidThreads)
    k_fluid_apply(int nx, int ny, FluidGrid G, const FluidStencils* __restrict__ S, const double* __restrict__ rows,
                  const double* xin, double* yout, int clamp, const KrylovDev* K, size_t n, double* zc) {
  TOPO_PDL_ENTRY();
  const FluidRows R(nx, ny);
  const size_t n2 = size_t(2 * nx + 1) * (2 * ny + 1), nv = R.count[0];
  int cls;
  size_t k;
  if (!fluid_thread(G, R, cls, k)) return;
  const double* x = KRYLOV ? xin + size_t(K->j) * n : xin;
  double* y = KRYLOV ? yout + size_t(K->j + 1) * n : yout;
  const double pm = KRYLOV ? K->zsum / double(nv) : 0.0;
  switch (cls) {
    case 0: fluid_apply_class<0>(nx, ny, *S, rows, R, k, x, pm, clamp != 0, y); break;
    case 1: fluid_apply_class<1>(nx, ny, *S, rows, R, k, x, pm, clamp != 0, y); break;
    case 2: fluid_apply_class<2>(nx, ny, *S, rows, R, k, x, pm, clamp != 0, y); break;
    case 3: fluid_apply_class<3>(nx, ny, *S, rows, R, k, x, pm, clamp != 0, y); break;
    default:
      y[2 * n2 + k] = fluid_continuity(*S, nx, ny, int(k % (nx + 1)), int(k / (nx + 1)), x);
      if (KRYLOV) zc[k] = x[2 * n2 + k] - pm;  // the centred pressure, moved into z_j by k_krylov_dot
  }
}

__global__ void k_fluid_objective(int nx, int ny, const FluidTables* __restrict__ E, FluidPenal pen, double mu,
                                  const double* __restrict__ rho, const double* __restrict__ u, double* partials,
                                  unsigned* counter, double* out) {
  const size_t nt = size_t(2) * nx * ny;
  double v[1] = {0.0};
  TOPO_GRID_STRIDE(t, nt) {
    size_t nd[6];
    fluid_tri_nodes(nx, t, nd);
    double ue[6][2], r[3];
    for (int k = 0; k < 6; ++k) {
      ue[k][0] = u[2 * nd[k]];
      ue[k][1] = u[2 * nd[k] + 1];
    }
    fluid_tri_rho(rho, nx, t, r);
    v[0] += fluid_tri_objective(*E, pen, mu, int(t & 1), r, ue);
  }
  double tot[1];
  if (finish_reduction<1>(v, partials, counter, tot)) out[0] = 0.5 * tot[0];
}

__global__ void k_fluid_grad_tri(int nx, int ny, const FluidTables* __restrict__ E, FluidPenal pen,
                                 const double* __restrict__ rho, const double* __restrict__ u,
                                 double* __restrict__ tri3) {
  const size_t nt = size_t(2) * nx * ny;
  TOPO_GRID_STRIDE(t, nt) {
    size_t nd[6];
    fluid_tri_nodes(nx, t, nd);
    double ue[6][2], r[3], o3[3];
    for (int k = 0; k < 6; ++k) {
      ue[k][0] = u[2 * nd[k]];
      ue[k][1] = u[2 * nd[k] + 1];
    }
    fluid_tri_rho(rho, nx, t, r);
    fluid_tri_gradient(*E, pen, r, ue, o3);
    tri3[3 * t] = o3[0];
    tri3[3 * t + 1] = o3[1];
    tri3[3 * t + 2] = o3[2];
  }
}

// rho at P2 node (a, b): the CG1 field interpolated linearly (vertex, edge midpoint
// or the cell's diagonal midpoint)
__device__ double fluid_rho_node(const double* rho, int nx, int a, int b) {
  const int VX = nx + 1;
  const int i0 = a >> 1, j0 = b >> 1;
  const int i1 = i0 + (a & 1), j1 = j0 + (b & 1);
  return 0.5 * (rho[size_t(j0) * VX + i0] + rho[size_t(j1) * VX + i1]);
}

// velocity preconditioner coefficients on the refined lattice: kM = alpha(rho) at each
// triangle's centroid (kK = 1)
__global__ void k_fluid_refined_alpha(int nx, int ny, FluidPenal pen, const double* __restrict__ rho,
                                      double* __restrict__ kM) {
  const int NXc = 2 * nx;  // cells of the refined lattice per row
  const size_t nt = size_t(2) * NXc * (2 * ny);
  TOPO_GRID_STRIDE(t, nt) {
    const int o = int(t & 1);
    const size_t cell = t >> 1;
    const int I = int(cell % NXc), J = int(cell / NXc);
    double s = 0.0;
    for (int k = 0; k < 3; ++k) s += fluid_rho_node(rho, nx, I + p1_off_a(o, k), J + p1_off_b(o, k));
    kM[t] = pen.a(s / 3.0);
  }
}

// pressure Laplacian coefficient kK = 1 / alpha(rho) at each base triangle's centroid
__global__ void k_fluid_inv_alpha(int nx, int ny, FluidPenal pen, const double* __restrict__ rho,
                                  double* __restrict__ kK) {
  const size_t nt = size_t(2) * nx * ny;
  TOPO_GRID_STRIDE(t, nt) {
    double r[3];
    fluid_tri_rho(rho, nx, t, r);
    kK[t] = 1.0 / pen.a((r[0] + r[1] + r[2]) / 3.0);
  }
}

__global__ void k_fluid_coarsen(const double* __restrict__ kf, int nxf, int nyf, double* __restrict__ kc, int nxc,
                                int nyc) {
  const size_t nt = size_t(2) * nxc * nyc;
  TOPO_GRID_STRIDE(t, nt) {
    const size_t cell = t >> 1;
    kc[t] = coarsen_kappa(kf, nxf, nyf, int(cell % nxc), int(cell / nxc), int(t & 1));
  }
}

// y = x - sum(x)/n with the sum a device scalar (one reduction before); y may be x
__global__ void k_fluid_center(const double* x, double* y, size_t n, const double* __restrict__ sum) {
  const double m = *sum / double(n);
  TOPO_GRID_STRIDE(i, n) y[i] = x[i] - m;
}

// ---------------------------------------------------------------------------
// one flexible-GMRES iteration
// ---------------------------------------------------------------------------
// Right-hand sides of the preconditioner: the planar velocity components of v_j (zero on
// the boundary) and its pressure less the mean
__global__ void k_fluid_split(int NX, int NY, const double* V, size_t n, size_t nv, const KrylovDev* K,
                              double* c, double* pt) {
  TOPO_PDL_ENTRY();
  const size_t n2 = size_t(NX) * NY;
  const double* v = V + size_t(K->j) * n;
  const double pm = K->psum / double(nv);
  TOPO_GRID_STRIDE(i, n2 + nv) {
    if (i < n2) {
      const bool bd = fluid_boundary_node(int(i % NX), int(i / NX), NX, NY);
      c[i] = bd ? 0.0 : v[2 * i];
      c[n2 + i] = bd ? 0.0 : v[2 * i + 1];
    } else {
      pt[i - n2] = v[n2 + i] - pm;  // (pressure entry k at 2 n2 + k = n2 + i)
    }
  }
}

// z_j = the V-cycles' velocity, and pressure r / m_lumped + the V-cycle's; sums the pressure
__global__ void k_fluid_merge(int NX, int NY, const double* V, double* Z, size_t n, size_t nv, const double* c,
                              const double* pz, const double* ml, double* partials, unsigned* counter, KrylovDev* K) {
  TOPO_PDL_ENTRY();
  const size_t n2 = size_t(NX) * NY;
  const double* v = V + size_t(K->j) * n + 2 * n2;
  double* z = Z + size_t(K->j) * n;
  double s[1] = {0.0};
  TOPO_GRID_STRIDE(i, n2 + nv) {
    if (i < n2) {
      const bool bd = fluid_boundary_node(int(i % NX), int(i / NX), NX, NY);
      z[2 * i] = bd ? 0.0 : c[i];
      z[2 * i + 1] = bd ? 0.0 : c[n2 + i];
    } else {
      const size_t k = i - n2;
      const double p = v[k] / ml[k] + pz[k];
      z[2 * n2 + k] = p;
      s[0] += p;
    }
  }
  double tot[1];
  if (finish_reduction<1>(s, partials, counter, tot)) K->zsum = tot[0];
}

// zero the boundary velocity rows: b[2i+c] = 0 at boundary nodes
__global__ void k_fluid_zero_boundary(int NX, int NY, double* __restrict__ v) {
  const size_t n = size_t(NX) * NY;
  TOPO_GRID_STRIDE(i, n) {
    if (fluid_boundary_node(int(i % NX), int(i / NX), NX, NY)) {
      v[2 * i] = 0.0;
      v[2 * i + 1] = 0.0;
    }
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// context
// ---------------------------------------------------------------------------
struct topo_fluid_ctx {
  int nx = 0, ny = 0, sms = 148;
  double W = 0, H = 0, hx = 0, hy = 0, viscosity = 1.0;
  size_t n2 = 0, nv = 0, n = 0;  // P2 nodes, CG1 vertices, unknowns (2 n2 + nv)
  FluidPenal pen{};
  bool penal_set = false;
  long long launches = 0;
  std::string err;
  Arena arena;
  Reducer red;
  FluidTables host_tab{};
  FluidTables* tab = nullptr;  // device copy
  double* ub = nullptr;        // boundary data (interleaved, zero inside)
  double* mass = nullptr;      // [tri][21], the Laplacian added
  FluidStencils* sten = nullptr;  // device copy
  double* rows = nullptr;      // velocity rows (FluidRows)
  double* tri3 = nullptr;      // [tri][3]
  double* ml = nullptr;        // lumped CG1 mass (vertex weights)
  double* ones = nullptr;      // nv ones (sums by a dot)
  double* rhs = nullptr;       // n
  double* x = nullptr;         // n (interior velocity | pressure)
  int m = kFluidRestart;       // restart length
  double* V = nullptr;         // (m + 1) n
  double* Z = nullptr;         // m n
  KrylovDev* kry = nullptr;
  double* dots = nullptr;      // partial sums and counters of the Gram-Schmidt products
  unsigned* dot_counters = nullptr;
  int* hstat = nullptr;        // pinned: j, it, maxit, status of the cycle
  double* zc = nullptr;        // nv: z_j's centred pressure
  double* t = nullptr;         // n
  double* c = nullptr;          // preconditioner: planar velocity components (2 n2) in
  double* z = nullptr;          // and out,
  double* pt = nullptr;         // pressure (nv) in
  double* pz = nullptr;         // and out
  double* gb = nullptr;        // gradient right-hand side (nv)
  // preconditioner hierarchies
  std::vector<LevelSpec> uspec, pspec;
  std::vector<ElemRefs> urefs, prefs;
  std::vector<double*> uK, uM, pK, pM;
  MG<double> mgu, mgp;
  // graph of one restart cycle, its recording stream, and the pressure's V-cycle beside the
  // velocity's
  cudaGraphExec_t graph = nullptr;
  bool use_graph = true;
  int graph_levels[2] = {-1, -1};  // the coarse solves' levels it was recorded with
  long long body_nodes = 0;  // kernels of one recorded iteration
  cudaStream_t cap = nullptr, side = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  topo_ctx* proj = nullptr;  // the CG1 projection (mass-matrix solve: a filter of radius 0)

  ~topo_fluid_ctx() {
    if (graph) cudaGraphExecDestroy(graph);
    for (cudaStream_t c : {cap, side})
      if (c) cudaStreamDestroy(c);
    for (cudaEvent_t e : {fork, join})
      if (e) cudaEventDestroy(e);
    if (proj) topo_destroy(proj);
    if (red.host) cudaFreeHost(red.host);
    if (hstat) cudaFreeHost(hstat);
  }
  int fail(int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    err = buf;
    return code;
  }
  int cuda_check(const char* where) {
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(TOPO_ERR_CUDA, "%s: %s", where, cudaGetErrorString(e));
    return TOPO_OK;
  }
  int grid(size_t m) const { return vec_grid(m, sms); }
  int NX() const { return 2 * nx + 1; }
  int NY() const { return 2 * ny + 1; }
  double* pp(double* v) const { return v + 2 * n2; }

  double dot(const double* a, const double* b, size_t m, cudaStream_t s) {
    k_dot<double, double><<<red.blocks_for(m), kVecThreads, 0, s>>>(a, b, m, red.partials, red.counter, red.out);
    ++launches;
    cudaMemcpyAsync(red.host, red.out, sizeof(double), cudaMemcpyDeviceToHost, s);
    cudaStreamSynchronize(s);
    return red.host[0];
  }
  // y = x - mean(x) on the pressure block (device-side mean)
  void center(const double* xp, double* yp, cudaStream_t s) {
    k_dot<double, double><<<red.blocks_for(nv), kVecThreads, 0, s>>>(xp, ones, nv, red.partials, red.counter, red.out);
    k_fluid_center<<<grid(nv), kVecThreads, 0, s>>>(xp, yp, nv, red.out);
    launches += 2;
  }
  // y = A x (the rows are the last design's)
  void apply(const double* xin, double* y, bool clamp, cudaStream_t s) {
    const FluidGrid G(nx, ny);
    k_fluid_apply<false><<<G.start[5], kFluidThreads, 0, s>>>(nx, ny, G, sten, rows, xin, y, clamp ? 1 : 0, nullptr, n,
                                                              nullptr);
    ++launches;
  }
  // the operator of design rho
  void set_design(const double* rho, cudaStream_t s) {
    const size_t nt = size_t(2) * nx * ny;
    const FluidGrid G(nx, ny);
    k_fluid_mass<<<grid(nt), kVecThreads, 0, s>>>(nx, ny, tab, pen, rho, mass);
    k_fluid_rows<<<G.start[4], kFluidThreads, 0, s>>>(nx, ny, G, mass, rows);
    launches += 2;
  }
  // one iteration of the cycle in kry, on s
  void iteration(cudaStream_t s, cudaGraphConditionalHandle cond, int use_cond) {
    const FluidGrid G(nx, ny);
    const unsigned gn = unsigned(grid(n2 + nv)), gv = unsigned(grid(n));
    const unsigned gd = unsigned(red.spread(n)), gm = unsigned(red.spread(n2 + nv));
    const double *Vc = V, *mlc = ml, *zcc = zc, *rc = rows;
    const FluidStencils* sc = sten;
    const KrylovDev* kc = kry;
    launch_pdl(k_fluid_split, gn, kVecThreads, 0, s, NX(), NY(), Vc, n, nv, kc, c, pt);
    cudaEventRecord(fork, s);
    cudaStreamWaitEvent(side, fork, 0);
    mgp.vcycle(pt, pz, side);
    cudaEventRecord(join, side);
    mgu.vcycle(c, z, s);
    cudaStreamWaitEvent(s, join, 0);
    k_fluid_merge<<<gm, kVecThreads, 0, s>>>(NX(), NY(), Vc, Z, n, nv, z, pz, mlc, red.partials,
                                                                 red.counter, kry);
    const double* Zc = Z;
    launch_pdl(k_fluid_apply<true>, G.start[5], kFluidThreads, 0, s, nx, ny, G, sc, rc, Zc, V, 1, kc, n, zc);
    krylov_column(KrylovSpace{V, nullptr, Z, zcc, n, nv, m, dots, dot_counters, red.partials, red.counter, kry},
                  int(gd), int(gv), cond, use_cond, s);
    launches += 8;
  }
  int record();
  int cycle(cudaStream_t s);
};

// Records one restart cycle: a WHILE node whose body is an iteration (k_krylov_next decides
// on the device whether it runs again).  Nothing is launched unless every step succeeded.
int topo_fluid_ctx::record() {
  std::lock_guard<std::recursive_mutex> lock(device_lock());
  cudaGetLastError();
  const long long l0 = launches + mgu.launches + mgp.launches;
  cudaGraph_t graph_ = nullptr, body = nullptr;
  if (cudaGraphCreate(&graph_, 0) != cudaSuccess) return -5;
  cudaGraphConditionalHandle h = 0;
  bool ok = cudaGraphConditionalHandleCreate(&h, graph_, 1, cudaGraphCondAssignDefault) == cudaSuccess;
  cudaGraphNode_t node = nullptr;
  cudaGraphNodeParams cp = {};
  if (ok) {
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    ok = cudaGraphAddNode(&node, graph_, nullptr, nullptr, 0, &cp) == cudaSuccess &&
         cp.conditional.phGraph_out != nullptr;
  }
  if (ok) {
    body = cp.conditional.phGraph_out[0];
    ok = cudaStreamBeginCaptureToGraph(cap, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed) == cudaSuccess;
  }
  if (ok) {
    iteration(cap, h, 1);
    ok = cudaStreamEndCapture(cap, &body) == cudaSuccess;
  }
  if (ok) ok = cudaGraphInstantiate(&graph, graph_, 0) == cudaSuccess;
  cudaGraphDestroy(graph_);
  ok = cudaGetLastError() == cudaSuccess && ok;
  body_nodes = launches + mgu.launches + mgp.launches - l0;
  launches -= body_nodes;  // recording is not execution
  if (!ok && graph) {
    cudaGraphExecDestroy(graph);
    graph = nullptr;
  }
  return ok ? 0 : -5;
}

// Runs the cycle set up in kry to its end and reads its counters back (hstat).  Without a graph
// (TOPO_GRAPHS=0, or a recording that another thread's device-wide work spoiled) the host
// launches the same kernels, one round trip per iteration.
int topo_fluid_ctx::cycle(cudaStream_t s) {
  const int levels[2] = {mgu.coarse_cheb_level(), mgp.coarse_cheb_level()};
  if (graph && std::memcmp(levels, graph_levels, sizeof(levels))) {
    cudaGraphExecDestroy(graph);
    graph = nullptr;
  }
  if (use_graph && !graph) {
    std::memcpy(graph_levels, levels, sizeof(levels));
    if (cudaStreamSynchronize(s) != cudaSuccess) return -5;  // the recording must not see queued work
    if (record() != 0) cudaGetLastError();
  }
  const int before = hstat[1];
  if (use_graph && graph) {
    if (cudaGraphLaunch(graph, s) != cudaSuccess) return -5;
  } else {
    do {
      iteration(s, 0, 0);
      cudaMemcpyAsync(hstat, kry, 4 * sizeof(int), cudaMemcpyDeviceToHost, s);
      if (cudaStreamSynchronize(s) != cudaSuccess) return -5;
    } while (hstat[3] == 1);
    return cudaGetLastError() == cudaSuccess ? 0 : -5;
  }
  cudaMemcpyAsync(hstat, kry, 4 * sizeof(int), cudaMemcpyDeviceToHost, s);
  if (cudaStreamSynchronize(s) != cudaSuccess) return -5;
  launches += body_nodes * std::max(0, hstat[1] - before);
  return 0;
}

namespace {

int fluid_setup(topo_fluid_ctx* C, const double* rho, cudaStream_t s) {
  const size_t nt = size_t(2) * C->nx * C->ny;
  C->set_design(rho, s);
  k_fluid_refined_alpha<<<C->grid(C->uspec[0].ntri()), kVecThreads, 0, s>>>(C->nx, C->ny, C->pen, rho, C->uM[0]);
  k_fluid_inv_alpha<<<C->grid(nt), kVecThreads, 0, s>>>(C->nx, C->ny, C->pen, rho, C->pK[0]);
  C->launches += 2;
  for (size_t l = 1; l < C->uspec.size(); ++l) {
    const LevelSpec &F = C->uspec[l - 1], &Cc = C->uspec[l];
    k_fluid_coarsen<<<C->grid(Cc.ntri()), kVecThreads, 0, s>>>(C->uM[l - 1], F.nx, F.ny, C->uM[l], Cc.nx, Cc.ny);
    ++C->launches;
  }
  for (size_t l = 1; l < C->pspec.size(); ++l) {
    const LevelSpec &F = C->pspec[l - 1], &Cc = C->pspec[l];
    k_fluid_coarsen<<<C->grid(Cc.ntri()), kVecThreads, 0, s>>>(C->pK[l - 1], F.nx, F.ny, C->pK[l], Cc.nx, Cc.ny);
    ++C->launches;
  }
  // both hierarchies' coefficients follow the design: choose their truncation and
  // uniform-row shortcuts again
  C->mgu.coefficients_changed();
  C->mgp.coefficients_changed();
  int st = C->mgu.setup(s);
  if (!st) st = C->mgp.setup(s);
  if (st == -5) return C->fail(TOPO_ERR_CUDA, "fluid preconditioner set-up: CUDA error");
  if (st) return C->fail(TOPO_ERR_NOT_CONVERGED, "fluid preconditioner set-up: coarse operator not positive definite");
  return C->cuda_check("fluid set-up");
}

// Flexible GMRES(m), right preconditioned, on the clamped operator from x = 0;
// stops on the true residual |b - A x| <= rtol |b|.
int fluid_fgmres(topo_fluid_ctx* C, const double* b, double* x, double rtol, int maxit, int& iters, double& relres,
                 cudaStream_t s) {
  const size_t n = C->n;
  const int g = C->grid(n);
  iters = 0;
  relres = 0.0;
  k_fill<double><<<g, kVecThreads, 0, s>>>(x, 0.0, n);
  ++C->launches;
  const double bn = std::sqrt(C->dot(b, b, n, s));
  if (!std::isfinite(bn)) return C->fail(TOPO_ERR_NAN, "non-finite right-hand side");
  if (bn == 0.0) return TOPO_OK;
  for (int cycle = 0;; ++cycle) {
    double* r = C->V;
    if (cycle == 0) {
      cudaMemcpyAsync(r, b, n * sizeof(double), cudaMemcpyDeviceToDevice, s);
    } else {
      C->apply(x, C->t, true, s);
      k_sub<double><<<g, kVecThreads, 0, s>>>(r, b, C->t, n);
      ++C->launches;
    }
    const double beta = std::sqrt(C->dot(r, r, n, s));
    relres = beta / bn;
    if (!std::isfinite(beta)) return C->fail(TOPO_ERR_NAN, "non-finite residual in the fluid solve");
    if (beta <= rtol * bn) return TOPO_OK;
    if (iters >= maxit)
      return C->fail(TOPO_ERR_NOT_CONVERGED, "fluid state solve did not converge (relres %.3g after %d iterations)",
                     relres, iters);
    k_scale<double><<<g, kVecThreads, 0, s>>>(r, 1.0 / beta, n);
    k_dot<double, double><<<C->red.blocks_for(C->nv), kVecThreads, 0, s>>>(C->pp(r), C->ones, C->nv, C->red.partials,
                                                                         C->red.counter, &C->kry->psum);
    k_krylov_start<<<1, 1, 0, s>>>(C->kry, beta, 0.5 * rtol * bn, iters, maxit, 0.0, 0.0, 0);
    C->hstat[1] = iters;
    const int rc = C->cycle(s);
    if (rc) return C->fail(TOPO_ERR_CUDA, "fluid solve: CUDA error");
    k_krylov_backsolve<<<1, 32, 0, s>>>(C->kry);
    k_krylov_update<<<g, kVecThreads, 0, s>>>(x, C->Z, n, C->kry);
    C->launches += 5;
    iters = C->hstat[1];
    if (C->hstat[3] == 4) return C->fail(TOPO_ERR_NAN, "non-finite Krylov vector in the fluid solve");
  }
}

template <class F>
int fguard(topo_fluid_ctx* C, F&& f) {
  if (!C) return TOPO_ERR_ARG;
  try {
    C->err.clear();
    return f();
  } catch (const std::exception& e) {
    return C->fail(TOPO_ERR_CUDA, "exception: %s", e.what());
  } catch (...) {
    return C->fail(TOPO_ERR_CUDA, "unknown exception");
  }
}

int fluid_init(topo_fluid_ctx* C, const topo_grid_desc* g, double viscosity, const topo_flow* flows, int nf) {
  if (!g || g->nx < 1 || g->ny < 1 || !(g->width > 0) || !(g->height > 0))
    return C->fail(TOPO_ERR_ARG, "invalid grid description");
  if (size_t(2 * g->nx + 1) * size_t(2 * g->ny + 1) > (size_t(1) << 28)) return C->fail(TOPO_ERR_ARG, "grid too large");
  if (!std::isfinite(viscosity)) return C->fail(TOPO_ERR_ARG, "invalid viscosity");
  if (nf < 0 || (nf > 0 && !flows)) return C->fail(TOPO_ERR_ARG, "invalid flow list");
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return C->fail(TOPO_ERR_CUDA, "no CUDA device");
  cudaDeviceGetAttribute(&C->sms, cudaDevAttrMultiProcessorCount, dev);
  C->nx = g->nx;
  C->ny = g->ny;
  C->W = g->width;
  C->H = g->height;
  C->hx = g->width / g->nx;
  C->hy = g->height / g->ny;
  C->viscosity = viscosity;
  C->n2 = size_t(C->NX()) * C->NY();
  C->nv = size_t(C->nx + 1) * (C->ny + 1);
  C->n = 2 * C->n2 + C->nv;
  C->pen.amin = 2.5 / (100.0 * 100.0);  // src/penalizers.py:53-54
  C->pen.amax = 2.5 / (0.01 * 0.01);
  std::string msg;
  std::vector<double> ub;
  if (fluid_boundary_values(C->nx, C->ny, C->W, C->H, flows, nf, ub, msg)) return C->fail(TOPO_ERR_ARG, "%s", msg.c_str());
  fluid_tables(C->hx, C->hy, C->host_tab);
  C->red.init(C->arena, C->sms);
  const size_t nt = size_t(2) * C->nx * C->ny;
  C->tab = C->arena.alloc_n<FluidTables>(1);
  C->ub = C->arena.alloc_n<double>(2 * C->n2);
  C->mass = C->arena.alloc_n<double>(nt * kFluidMass);
  C->sten = C->arena.alloc_n<FluidStencils>(1);
  C->rows = C->arena.alloc_n<double>(FluidRows(C->nx, C->ny).size);
  C->tri3 = C->arena.alloc_n<double>(3 * nt);
  C->ml = C->arena.alloc_n<double>(C->nv);
  C->ones = C->arena.alloc_n<double>(C->nv);
  C->rhs = C->arena.alloc_n<double>(C->n);
  C->x = C->arena.alloc_n<double>(C->n);
  size_t free_bytes = 0, total_bytes = 0;
  if (cudaMemGetInfo(&free_bytes, &total_bytes) != cudaSuccess) return C->cuda_check("device memory");
  C->m = fluid_restart(C->n, free_bytes);
  C->V = C->arena.alloc_n<double>(size_t(C->m + 1) * C->n);
  C->Z = C->arena.alloc_n<double>(size_t(C->m) * C->n);
  C->t = C->arena.alloc_n<double>(C->n);
  C->kry = C->arena.alloc_n<KrylovDev>(1);
  C->dots = C->arena.alloc_n<double>(krylov_dots(C->red.spread(C->n)));
  C->dot_counters = C->arena.alloc_n<unsigned>(kDotGroups);
  C->zc = C->arena.alloc_n<double>(C->nv);
  C->c = C->arena.alloc_n<double>(2 * C->n2);
  C->z = C->arena.alloc_n<double>(2 * C->n2);
  C->pt = C->arena.alloc_n<double>(C->nv);
  C->pz = C->arena.alloc_n<double>(C->nv);
  if (cudaMallocHost(&C->hstat, 4 * sizeof(int)) != cudaSuccess) return C->fail(TOPO_ERR_CUDA, "out of host memory");
  std::memset(C->hstat, 0, 4 * sizeof(int));
  for (cudaStream_t* c : {&C->cap, &C->side})
    if (cudaStreamCreateWithFlags(c, cudaStreamNonBlocking) != cudaSuccess) return C->cuda_check("fluid streams");
  for (cudaEvent_t* e : {&C->fork, &C->join})
    if (cudaEventCreateWithFlags(e, cudaEventDisableTiming) != cudaSuccess) return C->cuda_check("fluid events");
  if (const char* e = std::getenv("TOPO_GRAPHS")) C->use_graph = e[0] != '0';
  C->gb = C->arena.alloc_n<double>(C->nv);
  if (C->arena.failed()) return C->fail(TOPO_ERR_CUDA, "out of device memory");
  const std::vector<double> w = vertex_weights(C->nx, C->ny, C->hx, C->hy);
  FluidStencils st{};
  fluid_stencils(C->host_tab, st);
  if (cudaMemcpy(C->sten, &st, sizeof(st), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(C->tab, &C->host_tab, sizeof(FluidTables), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(C->ub, ub.data(), ub.size() * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(C->ml, w.data(), w.size() * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess)
    return C->cuda_check("fluid set-up copies");
  cudaStream_t s = 0;
  k_fill<double><<<C->grid(C->nv), kVecThreads, 0, s>>>(C->ones, 1.0, C->nv);
  // velocity hierarchy: P1 on the refined lattice, every side clamped
  Dir du = no_dir(C->NX(), C->NY());
  du.x_lo = 1;
  du.y_lo = 1;
  du.x_hi_from = C->NX() - 1;
  du.y_hi_from = C->NY() - 1;
  C->uspec = build_levels(false, 2 * C->nx, 2 * C->ny, 0.5 * C->hx, 0.5 * C->hy, du, 1);
  C->pspec = build_levels(false, C->nx, C->ny, C->hx, C->hy, no_dir(C->nx + 1, C->ny + 1), 1);
  auto hierarchy = [&](std::vector<LevelSpec>& spec, std::vector<ElemRefs>& refs, std::vector<double*>& kK,
                       std::vector<double*>& kM) {
    const int L = int(spec.size());
    refs.resize(L);
    kK.assign(L, nullptr);
    kM.assign(L, nullptr);
    for (int l = 0; l < L; ++l) {
      refs[l] = make_elem_refs(spec[l].hx, spec[l].hy, 0.0, 0.0);
      kK[l] = C->arena.alloc_n<double>(spec[l].ntri());
      kM[l] = C->arena.alloc_n<double>(spec[l].ntri());
    }
  };
  hierarchy(C->uspec, C->urefs, C->uK, C->uM);
  hierarchy(C->pspec, C->prefs, C->pK, C->pM);
  if (C->arena.failed()) return C->fail(TOPO_ERR_CUDA, "out of device memory");
  // the design-independent coefficients: kK = 1 (velocity), kM = shift (pressure)
  for (size_t l = 0; l < C->uspec.size(); ++l)
    k_fill<double><<<C->grid(C->uspec[l].ntri()), kVecThreads, 0, s>>>(C->uK[l], 1.0, C->uspec[l].ntri());
  for (size_t l = 0; l < C->pspec.size(); ++l)
    k_fill<double><<<C->grid(C->pspec[l].ntri()), kVecThreads, 0, s>>>(C->pM[l], kLaplaceShift, C->pspec[l].ntri());
  for (auto* mg : {&C->mgu, &C->mgp}) {
    mg->use_graphs = false;  // only V-cycles are used
    mg->profile_levels = false;
    mg->element_bounds = true;
  }
  C->mgu.batch = 2;
  C->mgu.init(C->uspec, C->urefs.data(), 0.0, 0.0, C->arena, &C->red);
  C->mgu.set_coefficients(std::vector<const double*>(C->uK.begin(), C->uK.end()),
                          std::vector<const double*>(C->uM.begin(), C->uM.end()));
  C->mgp.init(C->pspec, C->prefs.data(), 0.0, 0.0, C->arena, &C->red);
  C->mgp.set_coefficients(std::vector<const double*>(C->pK.begin(), C->pK.end()),
                          std::vector<const double*>(C->pM.begin(), C->pM.end()));
  if (C->arena.failed()) return C->fail(TOPO_ERR_CUDA, "out of device memory");
  int rc = 0;
  C->proj = topo_create_filter(g, 0.0, TOPO_PREC_FP64, &rc);
  if (!C->proj) return C->fail(rc ? rc : TOPO_ERR_CUDA, "CG1 projection set-up failed");
  return C->cuda_check("fluid set-up");
}

}  // namespace

extern "C" {

topo_fluid_ctx* topo_fluid_create(const topo_grid_desc* grid, double viscosity, const topo_flow* flows, int n_flows,
                                  int* status) {
  std::lock_guard<std::recursive_mutex> lock(device_lock());
  topo_fluid_ctx* C = nullptr;
  int rc = TOPO_OK;
  try {
    C = new topo_fluid_ctx();
    rc = fluid_init(C, grid, viscosity, flows, n_flows);
    if (!rc) {
      const cudaError_t e = settle_setup_stream();
      if (e != cudaSuccess) rc = C->fail(TOPO_ERR_CUDA, "set-up: %s", cudaGetErrorString(e));
    }
  } catch (...) {
    rc = TOPO_ERR_CUDA;
  }
  if (status) *status = rc;
  if (rc) {
    if (C) std::fprintf(stderr, "topo_fluid_create: %s\n", C->err.c_str());
    delete C;
    return nullptr;
  }
  return C;
}

void topo_fluid_destroy(topo_fluid_ctx* ctx) {
  std::lock_guard<std::recursive_mutex> lock(device_lock());
  delete ctx;
}

const char* topo_fluid_last_error(const topo_fluid_ctx* ctx) { return ctx ? ctx->err.c_str() : "null context"; }

int topo_fluid_sizes(const topo_fluid_ctx* ctx, int64_t* n_vertices, int64_t* n_velocity) {
  if (!ctx) return TOPO_ERR_ARG;
  if (n_vertices) *n_vertices = int64_t(ctx->nv);
  if (n_velocity) *n_velocity = int64_t(2 * ctx->n2);
  return TOPO_OK;
}

int topo_fluid_set_penalization(topo_fluid_ctx* ctx, double q) {
  return fguard(ctx, [&]() {
    if (!std::isfinite(q) || !(q > 0)) return ctx->fail(TOPO_ERR_ARG, "invalid penalization");
    ctx->pen.q = q;
    ctx->penal_set = true;
    return TOPO_OK;
  });
}

int topo_fluid_boundary_values(topo_fluid_ctx* ctx, double* u, topo_stream_t stream) {
  return fguard(ctx, [&]() {
    if (!u) return ctx->fail(TOPO_ERR_ARG, "null output");
    cudaMemcpyAsync(u, ctx->ub, 2 * ctx->n2 * sizeof(double), cudaMemcpyDeviceToDevice,
                    reinterpret_cast<cudaStream_t>(stream));
    return ctx->cuda_check("boundary values");
  });
}

int topo_fluid_apply(topo_fluid_ctx* ctx, const double* rho, const double* x, double* y, int clamp,
                     topo_stream_t stream) {
  return fguard(ctx, [&]() {
    if (!ctx->penal_set) return ctx->fail(TOPO_ERR_STATE, "You must set penalization before calling penalizer");
    if (!rho || !x || !y || x == y) return ctx->fail(TOPO_ERR_ARG, "invalid apply arguments");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    ctx->set_design(rho, s);
    ctx->apply(x, y, clamp != 0, s);
    return ctx->cuda_check("fluid apply");
  });
}

int topo_fluid_state_solve(topo_fluid_ctx* ctx, const double* rho, double* u, double* p, double rtol, int* iters,
                           topo_stream_t stream) {
  return fguard(ctx, [&]() {
    if (!ctx->penal_set) return ctx->fail(TOPO_ERR_STATE, "You must set penalization before calling penalizer");
    if (!rho || !u || !(rtol > 0)) return ctx->fail(TOPO_ERR_ARG, "invalid state-solve arguments");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    int rc = fluid_setup(ctx, rho, s);
    if (rc) return rc;
    // right-hand side: minus the unclamped operator on the boundary data, boundary rows
    // zero, continuity part projected to zero sum
    double* lift = ctx->t;
    cudaMemsetAsync(lift, 0, ctx->n * sizeof(double), s);
    cudaMemcpyAsync(lift, ctx->ub, 2 * ctx->n2 * sizeof(double), cudaMemcpyDeviceToDevice, s);
    ctx->apply(lift, ctx->rhs, false, s);
    k_scale<double><<<ctx->grid(ctx->n), kVecThreads, 0, s>>>(ctx->rhs, -1.0, ctx->n);
    k_fluid_zero_boundary<<<ctx->grid(ctx->n2), kVecThreads, 0, s>>>(ctx->NX(), ctx->NY(), ctx->rhs);
    ctx->launches += 2;
    ctx->center(ctx->pp(ctx->rhs), ctx->pp(ctx->rhs), s);
    int it = 0;
    double rel = 0.0;
    rc = fluid_fgmres(ctx, ctx->rhs, ctx->x, rtol, 2000, it, rel, s);
    if (iters) *iters = it;
    if (rc) return rc;
    // u = interior solution + boundary data; p = the zero-sum pressure
    k_add_multi<double, double, 1><<<ctx->grid(2 * ctx->n2), kVecThreads, 0, s>>>(
        ctx->x, ctx->ub, 2 * ctx->n2, MultiCoef{{1.0}}, 2 * ctx->n2);
    cudaMemcpyAsync(u, ctx->x, 2 * ctx->n2 * sizeof(double), cudaMemcpyDeviceToDevice, s);
    if (p) cudaMemcpyAsync(p, ctx->pp(ctx->x), ctx->nv * sizeof(double), cudaMemcpyDeviceToDevice, s);
    ++ctx->launches;
    return ctx->cuda_check("fluid state solve");
  });
}

int topo_fluid_objective(topo_fluid_ctx* ctx, const double* rho, const double* u, double* objective,
                         topo_stream_t stream) {
  return fguard(ctx, [&]() {
    if (!ctx->penal_set) return ctx->fail(TOPO_ERR_STATE, "You must set penalization before calling penalizer");
    if (!rho || !u || !objective) return ctx->fail(TOPO_ERR_ARG, "invalid objective arguments");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    k_fluid_objective<<<ctx->red.blocks_for(size_t(8) * ctx->nx * ctx->ny), kVecThreads, 0, s>>>(ctx->nx, ctx->ny, ctx->tab, ctx->pen, ctx->viscosity,
                                                              rho, u, ctx->red.partials, ctx->red.counter, objective);
    ++ctx->launches;
    return ctx->cuda_check("fluid objective");
  });
}

int topo_fluid_gradient_rhs(topo_fluid_ctx* ctx, const double* rho, const double* u, double* b,
                            topo_stream_t stream) {
  return fguard(ctx, [&]() {
    if (!ctx->penal_set) return ctx->fail(TOPO_ERR_STATE, "You must set penalization before calling penalizer");
    if (!rho || !u || !b) return ctx->fail(TOPO_ERR_ARG, "invalid gradient arguments");
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const size_t nt = size_t(2) * ctx->nx * ctx->ny;
    k_fluid_grad_tri<<<ctx->grid(nt), kVecThreads, 0, s>>>(ctx->nx, ctx->ny, ctx->tab, ctx->pen, rho, u, ctx->tri3);
    k_vertex_gather3<double><<<ctx->grid(ctx->nv), kVecThreads, 0, s>>>(ctx->nx, ctx->ny, ctx->tri3, b);
    ctx->launches += 2;
    return ctx->cuda_check("fluid gradient");
  });
}

int topo_fluid_gradient(topo_fluid_ctx* ctx, const double* rho, const double* u, double* g, double rtol, int* iters,
                        topo_stream_t stream) {
  int rc = topo_fluid_gradient_rhs(ctx, rho, u, ctx ? ctx->gb : nullptr, stream);
  if (rc) return rc;
  return fguard(ctx, [&]() {
    if (!g || !(rtol > 0)) return ctx->fail(TOPO_ERR_ARG, "invalid gradient arguments");
    const int r = topo_filter_solve(ctx->proj, ctx->gb, g, rtol, iters, stream);
    if (r) return ctx->fail(r, "CG1 projection: %s", topo_last_error(ctx->proj));
    return TOPO_OK;
  });
}

int topo_fluid_launch_count(const topo_fluid_ctx* ctx, int64_t* launches) {
  if (!ctx || !launches) return TOPO_ERR_ARG;
  int64_t pl = 0;
  if (ctx->proj) topo_launch_count(ctx->proj, &pl);
  *launches = ctx->launches + ctx->mgu.launches + ctx->mgp.launches + pl;
  return TOPO_OK;
}

}  // extern "C"
