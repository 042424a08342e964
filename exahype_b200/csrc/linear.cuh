// Linear ADER-DG kernels for PDEs given by a non-conservative product
// (PDE::kLinear, e.g. ElasticPDE):
//   ck_predictor_kernel    spaceTimePredictorLinear (2d/spaceTimePredictorLinear.cpph:35-409,
//                          3d/spaceTimePredictorLinear.cpph:34-446) + volumeIntegralLinear
//                          (3d/volumeIntegralLinear.cpph:20-52); for a PDE with a point
//                          source also pointSource (3d/pointSource.cpph:28-143)
//   riemann_linear_kernel  riemannSolverLinear (3d/riemannSolverLinear.cpph:20-136)
//   boundary_linear_kernel boundaryConditions + riemannSolverLinear on boundary faces
//   volume_linear_kernel   volumeIntegralLinear on its own (kernel-level entry point)
// The surface integral is the corrector's linear form (aderdg.cuh).
//
// The predictor is the Cauchy-Kovalevski procedure: time derivative i+1 of
// the solution is -sum_d B_d(Q_i) grad_d Q_i, evaluated b-1 times; the time
// averages over [0, dt] weight derivative i by dt^i / (i+1)!. A linear PDE's
// coefficients depend on the cell's parameters only, so the time-averaged
// fluxes need no sums of their own: sum_i w_i B_d grad_d Q_i is B_d applied to
// the gradient of the time-averaged state, one more gradient pass at the end
// in the place of 2 d nV running sums per node. No iteration and no
// convergence test.
//
// The cell's state and gradients sit in shared memory as planes, one variable
// or gradient component of all nodes each, so that the per-node phase reads
// consecutive doubles. The gradients are 1-D line contractions with dudx (one
// thread per component and line, the components the product reads), the
// product and the averages are per node in registers.
//
// Bound: the shared-memory pipe (63 accesses per node and level; without the
// running sums three blocks share an SM). 27^3 N=5 elastic: 1.283 -> 0.757 ms.
#pragma once
#include "aderdg.cuh"
#include "line_tables.cuh"

namespace exa {

// the (direction, variable) gradient components the PDE's ncp reads, direction
// by direction; those of direction e are first[e] .. first[e + 1] - 1
template <class PDE, int DIM>
struct GradPairs {
  int d[DIM * PDE::nVar], v[DIM * PDE::nVar], first[DIM + 1], n;
  constexpr GradPairs() : d(), v(), first(), n(0) {
    for (int dd = 0; dd < DIM; dd++) {
      for (int vv = 0; vv < PDE::nVar; vv++)
        if (PDE::ncp_uses(dd, vv)) {
          d[n] = dd;
          v[n] = vv;
          n++;
        }
      first[dd + 1] = n;
    }
  }
  constexpr bool even() const {  // as many in every direction
    for (int dd = 0; dd < DIM; dd++)
      if ((first[dd + 1] - first[dd]) * DIM != n) return false;
    return true;
  }
};

// Where the planes of a cell lie in shared memory: the nD of the state, then
// the gradient components'. PL apart, except for six nodes in 3D with nine
// variables: there a line's threads meet in few banks only if each plane's
// position modulo the 16 banks of 64 bits is chosen by what is read and written
// together. The residues come from a search over a count of the wavefronts of
// the three directions' loads (state) and stores (components) with the item
// orders of the kernel (gen_planes.py); 966 a level against 1188 with all planes
// PL apart (882 if nothing met). The shared-memory pipe bounds the kernel (96 % busy
// before): 27^3 N=5 757 -> 720 us.
template <int PLANES, int PL, int CELL, bool PLACED>
struct CKPlanes {
  int at[PLANES + 1] = {};  // [PLANES]: the end
  constexpr CKPlanes() {
    constexpr int residue[30] = {0, 15, 1, 9, 5, 2, 11, 4, 13, 5, 14, 7,  // state (the last three are parameters)
                                 0, 1, 2, 3, 4, 5,                       // components of x
                                 0, 6, 12, 2, 8, 14,                     // y
                                 0, 4, 8, 12, 0, 4};                     // z
    for (int k = 1; k <= PLANES; k++) {
      at[k] = at[k - 1] + (PLACED ? CELL : PL);
      if (PLACED && k < PLANES) at[k] += (residue[k < 30 ? k : 0] - at[k] % 16 + 16) % 16;
    }
  }
};

template <int DIM, int N, class PDE>
struct CKCfg : Shape<DIM, N, PDE> {
  using S = Shape<DIM, N, PDE>;
  // what fits 128 threads, or one cell: a barrier joins fewer warps than in
  // blocks of up to 256 threads (9,975 cells 3D N=4 232 -> 206 us, 19,683 cells
  // N=3 218 -> 207, 6,561 cells 2D N=5 48 -> 44)
  static constexpr int CPB = S::P <= 128 ? 128 / S::P : 1;
  static constexpr int THREADS = CPB * S::P;
  static constexpr int LINES = S::F;                                             // lines per direction
  static constexpr int NPAIRS = GradPairs<PDE, DIM>().n;  // gradient components
  static constexpr bool kEven = GradPairs<PDE, DIM>().even();
  static constexpr int NU = kEven ? NPAIRS / DIM : 1;  // per direction, where as many in each (b > 1)
  // planes: row pitch (4 nodes: 5, or the x lines' threads would meet in four
  // banks), plane pitch (odd: the variables of one node lie in different banks)
  static constexpr int YP = S::b == 4 ? 5 : S::b, ZP = S::b * YP;
  static constexpr int PL = (ZP * (DIM == 3 ? S::b : 1)) | 1;
  static constexpr bool kPlaced = kEven && DIM == 3 && S::b == 6 && S::nV == 9 && S::nD == 12 && NPAIRS == 18;
  using Planes = CKPlanes<S::nD + NPAIRS, PL, S::b * ZP, kPlaced>;
  static constexpr int SC = Planes().at[S::nD + NPAIRS];  // doubles per cell
  static constexpr size_t SMEM = sizeof(double) * (size_t)CPB * SC;
  // gradient items per thread; with NU == b one direction per round
  static constexpr int ROUNDS = (NPAIRS + S::b - 1) / S::b;
  static constexpr bool kDirRounds = NU == S::b;
  // Blocks per SM of the register budget: three where a block is one cell of
  // N = 5 in 3D (27^3, planes PL apart: 0.753 ms, with two 0.793, four 0.775), else 512 threads
  // (N=4 with five blocks of 125 threads 208 us, with four 206). The point source's
  // code needs more: two blocks at 3D N=5, three at 3D N=3 (30^3 324 us, with four, which spill, 337).
  static constexpr int BLOCKS = S::P <= 128 ? (PDE::kPointSource && DIM == 3 ? 3 : 4) : PDE::kPointSource ? 2 : 3;
  static constexpr int NREG = regs_for_blocks<THREADS, BLOCKS>();
  // the second direction's fluxes lie behind the first's where the planes up to
  // its gradient components hold both (few components or no parameters: in the
  // first's place, after one more barrier)
  static constexpr bool kBehind = Planes().at[S::nD + GradPairs<PDE, DIM>().first[1]] >= 2 * S::nV * PL;
  static_assert(Planes().at[S::nD] >= S::nV * PL, "the first direction's fluxes take the place of the state");
  static __host__ __device__ constexpr int pos(int x, int y, int z) { return z * ZP + y * YP + x; }
  static __host__ __device__ constexpr int step(int d) { return d == 0 ? 1 : d == 1 ? YP : ZP; }
  // first node of line L along d (L enumerates the other coordinates in
  // (z, y, x) order, the face-node order of the reference)
  static __device__ __forceinline__ int line0(int d, int L) {
    const int a = L / S::b, c = L % S::b;
    if (DIM == 2) return d == 0 ? L * YP : L;
    return d == 0 ? a * ZP + c * YP : d == 1 ? a * ZP + c : a * YP + c;
  }
};

// Lagrange basis polynomial i of the Gauss-Legendre nodes of order N at xi
// (the reference's basisFunctions[N][i], kernels/DGBasisFunctions.h:53), as
// the product over the other nodes
template <int N>
__device__ double lagrange_at(int i, double xi) {
  const OrderTables& T = c_tab[N];
  double r = 1.0;
#pragma unroll
  for (int m = 0; m < N + 1; m++)
    if (m != i) r = __dmul_rn(r, __ddiv_rn(__dsub_rn(xi, T.x[m]), __dsub_rn(T.x[i], T.x[m])));
  return r;
}

// Whether the point source of PDE::sourcePosition lies in the closed cell of
// centre c and widths h, tested on the reference coordinates as pointSource
// tests them
template <int DIM, class PDE>
__device__ bool point_source_in_cell(const Geometry& geo, const double* c, const double* h) {
  double x0[3];
  PDE::sourcePosition(geo.ps, x0);
  bool in = true;
#pragma unroll
  for (int e = 0; e < DIM; e++) {
    const double xr = __ddiv_rn(__dsub_rn(x0[e], __dsub_rn(c[e], __ddiv_rn(h[e], 2.0))), h[e]);
    in = in && xr >= 0.0 && xr <= 1.0;
  }
  return in;
}

// pointSource (2d/pointSource.cpph:30-127, 3d/pointSource.cpph:28-143) at one
// node of the cell of centre c and widths h: the PDE's source at the node's
// position, projected onto the node's basis function at the source's reference
// coordinates (phi) and divided by the node's quadrature weight and the cell's
// widths (den); zero where the source lies outside the closed cell. The
// reference's operations in its order, rounded one by one; phi and den, which
// do not depend on the time, once per node (a small mesh waits for the cell with
// the source: 3^3 cells of 3D N=5 75 -> 32 us, 9^2 of 2D N=5 52 -> 20).
template <int DIM, int N, class PDE>
struct NodePointSource {
  double x[3], phi, den;
  bool in;
  const Geometry& geo;
  __device__ NodePointSource(const Geometry& g, const double* c, const double* h, int p) : geo(g) {
    constexpr int b = N + 1;
    const OrderTables& T = c_tab[N];
    const int ix = p % b, iy = (p / b) % b, iz = DIM == 3 ? p / (b * b) : 0;
    x[0] = __dadd_rn(c[0], __dmul_rn(h[0], __dsub_rn(T.x[ix], 0.5)));
    x[1] = __dadd_rn(c[1], __dmul_rn(h[1], __dsub_rn(T.x[iy], 0.5)));
    x[2] = DIM == 3 ? __dadd_rn(c[2], __dmul_rn(h[2], __dsub_rn(T.x[iz], 0.5))) : 0.0;
    double x0[3], xr[3] = {0.0, 0.0, 0.0};
    PDE::sourcePosition(geo.ps, x0);
    in = true;
#pragma unroll
    for (int e = 0; e < DIM; e++) {
      xr[e] = __ddiv_rn(__dsub_rn(x0[e], __dsub_rn(c[e], __ddiv_rn(h[e], 2.0))), h[e]);
      in = in && xr[e] >= 0.0 && xr[e] <= 1.0;
    }
    if (DIM == 3) {
      phi = __dmul_rn(__dmul_rn(lagrange_at<N>(iz, xr[2]), lagrange_at<N>(iy, xr[1])), lagrange_at<N>(ix, xr[0]));
      den = __dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(T.w[iz], h[2]), T.w[iy]), h[1]), T.w[ix]), h[0]);
    } else {
      phi = __dmul_rn(lagrange_at<N>(iy, xr[1]), lagrange_at<N>(ix, xr[0]));
      den = __dmul_rn(__dmul_rn(__dmul_rn(T.w[iy], h[1]), T.w[ix]), h[0]);
    }
  }
  // at time slot n (0: t; n >= 1: Gauss-Legendre time node n - 1 of [t, t + dt])
  __device__ void at(double t, double dt, int n, double* out) const {
    double x0[3];
    PDE::pointSource(x, n == 0 ? t : __dadd_rn(__dmul_rn(dt, c_tab[N].x[n - 1]), t), dt, out, x0, geo.ps);
#pragma unroll
    for (int v = 0; v < PDE::nVar; v++) out[v] = in ? __ddiv_rn(__dmul_rn(phi, out[v]), den) : 0.0;
  }
  // sum over the time slots n = 1..b of w[n-1] * pointSource (the time integral
  // the predictor adds, 3d/spaceTimePredictorLinear.cpph:77-90 and :294-308)
  __device__ void sum(double t, double dt, double* s) const {
#pragma unroll
    for (int v = 0; v < PDE::nVar; v++) s[v] = 0.0;
#pragma unroll 1
    for (int n = 1; n < N + 2; n++) {
      double val[PDE::nVar];
      at(t, dt, n, val);
#pragma unroll
      for (int v = 0; v < PDE::nVar; v++) s[v] = __dadd_rn(s[v], __dmul_rn(c_tab[N].w[n - 1], val[v]));
    }
  }
};

template <int DIM, int N, class PDE, int NREG = CKCfg<DIM, N, PDE>::NREG>
__global__ void __launch_bounds__(CKCfg<DIM, N, PDE>::THREADS) __maxnreg__(NREG)
    ck_predictor_kernel(const double* __restrict__ luh, double* __restrict__ lQhbnd, double* __restrict__ lFhbnd,
                        double* __restrict__ lduh, const double* __restrict__ dt_ptr, Geometry geo, int ncells,
                        const int* __restrict__ cell_list, const int* __restrict__ count,
                        double* __restrict__ lQhi_out, double* __restrict__ lFhi_out) {
  using C = CKCfg<DIM, N, PDE>;
  constexpr int b = C::b, P = C::P, nV = C::nV, nD = C::nD, LINES = C::LINES, PL = C::PL, F = C::F, NU = C::NU;
  extern __shared__ double smem[];
  const OrderTables& T = c_tab[N];
  const LineTables<N>& K = line_tab<N>();
  const int lc = threadIdx.x / P;
  const int p = threadIdx.x - lc * P;
  const int slot = blockIdx.x * C::CPB + lc;
  const int nact = count ? min(*count, ncells) : ncells;
  if ((int)blockIdx.x * C::CPB >= nact) return;  // whole block, before its first barrier
  const bool active = slot < nact;
  const int cell = active ? (cell_list ? cell_list[slot] : slot) : 0;
  double* sC = smem + lc * C::SC;
  const int x = p % b, y = (p / b) % b, z = DIM == 3 ? p / (b * b) : 0;
  double* own = sC + C::pos(x, y, z);
  constexpr typename C::Planes PT;
  __shared__ int s_plane[nD];  // the state's planes, for a variable known at run time
  if constexpr (C::kPlaced) {
#pragma unroll
    for (int v = 0; v < nD; v++)
      if (threadIdx.x == v) s_plane[v] = PT.at[v];
    __syncthreads();
  }
  auto plane = [&](int v) { return C::kPlaced ? s_plane[v] : v * PL; };
  const int inst = cell_instance(geo, cell);
  const double dt = dt_ptr[inst];
  double idx[DIM];
#pragma unroll
  for (int d = 0; d < DIM; d++) idx[d] = 1.0 / cell_width(geo, inst, d);
  // point sources: this cell's centre, widths and time stamp, and whether
  // the source lies in it (the same for all threads of the cell)
  constexpr bool PS = PDE::kPointSource;
  double pc[3] = {0.0, 0.0, 0.0}, ph[3] = {1.0, 1.0, 1.0}, pt = 0.0;
  bool here = false;
  if constexpr (PS) {
    if (active && geo.centre) {
#pragma unroll
      for (int d = 0; d < DIM; d++) {
        pc[d] = geo.centre[3 * (size_t)cell + d];
        ph[d] = cell_width(geo, inst, d);
      }
      pt = *geo.time;
      here = point_source_in_cell<DIM, PDE>(geo, pc, ph);
    }
  }
  // level 0: the solution (parameters included), read by consecutive threads;
  // inactive slots get unit parameters so that their arithmetic stays finite
  {
    const double* src = luh + (size_t)cell * P * nD;
#pragma unroll
    for (int k = 0; k < nD; k++) {
      const int e = p + k * P, n = e / nD, v = e - n * nD;
      const int nx = n % b, ny = (n / b) % b, nz = DIM == 3 ? n / (b * b) : 0;
      sC[plane(v) + C::pos(nx, ny, nz)] = active ? __ldg(src + e) : (v < nV ? 0.0 : 1.0);
    }
  }
  // gradient items of this thread: component j of the pairs, line L.
  // Consecutive threads take consecutive lines of one component; along x
  // (with one direction per round) consecutive components of one line, whose
  // lines start an even number of doubles apart; along y, where the planes are
  // placed for it, the lines of one z plane component by component.
  int g_src[C::ROUNDS], g_dst[C::ROUNDS];
#pragma unroll
  for (int r = 0; r < C::ROUNDS; r++) {
    int L, j;
    if (C::kDirRounds && r == 0) {
      L = p / NU;
      j = p % NU;
    } else if (C::kPlaced && r == 1) {
      L = p / (b * NU) * b + p % b;
      j = p / b % NU + NU;
    } else {
      L = p % LINES;
      j = p / LINES + b * r;
    }
    g_src[r] = -1;
    g_dst[r] = 0;
    if (j < C::NPAIRS) {
      constexpr GradPairs<PDE, DIM> GP;
      const int l0 = C::line0(j < GP.first[1] ? 0 : DIM == 2 || j < GP.first[2] ? 1 : 2, L);
      if constexpr (C::kPlaced) {
#pragma unroll
        for (int i = 0; i < C::NPAIRS; i++)
          if (i == j) {
            g_src[r] = PT.at[GP.v[i]] + l0;
            g_dst[r] = PT.at[nD + i] + l0;
          }
      } else {
        int v = 0;
#pragma unroll
        for (int i = 0; i < C::NPAIRS; i++)
          if (i == j) v = GP.v[i];
        g_src[r] = v * PL + l0;
        g_dst[r] = (nD + j) * PL + l0;
      }
    }
  }
  auto gradients = [&]() {
#pragma unroll
    for (int r = 0; r < C::ROUNDS; r++) {
      if (g_src[r] < 0) continue;
      int st;
      if (C::kDirRounds) st = C::step(r);
      else {
        constexpr GradPairs<PDE, DIM> GP;
        const int j = g_dst[r] / PL - nD;
        st = j < GP.first[1] ? C::step(0) : DIM == 2 || j < GP.first[2] ? C::step(1) : C::step(2);
      }
      const double* s = sC + g_src[r];
      double* g = sC + g_dst[r];
      double f[b];
#pragma unroll
      for (int n = 0; n < b; n++) f[n] = s[n * st];
      line_contract<b>(f, K.DP, K.DQ, [&](int l, double a) { g[l * st] = a; });
    }
  };
  auto product = [&](const double* Qp, int d, double* B) {
    double G[nV];
#pragma unroll
    for (int v = 0; v < nV; v++) G[v] = 0.0;
    int i = 0;
#pragma unroll
    for (int v = 0; v < nV; v++)
      if (PDE::ncp_uses(d, v)) G[v] = idx[d] * own[PT.at[nD + GradPairs<PDE, DIM>().first[d] + i++]];
    PDE::ncp_dir(Qp, d, G, B);
  };
  __syncthreads();
  double Qp[nD], qh[nV];  // the node's parameters, the time-averaged state
#pragma unroll
  for (int v = 0; v < nV; v++) qh[v] = own[PT.at[v]], Qp[v] = 0.0;
#pragma unroll
  for (int v = nV; v < nD; v++) Qp[v] = own[PT.at[v]];
  if constexpr (PS) {
    // a point source adds dt times its time integral to level 0
    // (3d/spaceTimePredictorLinear.cpph:77-90)
    if (here) {
      double psw[nV];
      NodePointSource<DIM, N, PDE>(geo, pc, ph, p).sum(pt, dt, psw);
#pragma unroll
      for (int v = 0; v < nV; v++) own[PT.at[v]] = qh[v] = __dadd_rn(qh[v], __dmul_rn(dt, psw[v]));
    }
    __syncthreads();
  }
  double fac = 0.5 * dt;  // weight of level i + 1 in the time averages
#pragma unroll 1
  for (int i = 0; i + 1 < b; i++) {
    if (i > 0) __syncthreads();  // level i complete
    gradients();
    __syncthreads();
    double qn[nV];
#pragma unroll
    for (int v = 0; v < nV; v++) qn[v] = 0.0;
    if constexpr (PS)  // level 1 starts from the point source's value at t (:93-101)
      if (here && i == 0) NodePointSource<DIM, N, PDE>(geo, pc, ph, p).at(pt, dt, 0, qn);
#pragma unroll
    for (int d = 0; d < DIM; d++) {
      double B[nV];
      product(Qp, d, B);
#pragma unroll
      for (int v = 0; v < nV; v++) qn[v] -= B[v];
    }
    const bool last = i + 2 == b;  // then the averages take the level's place
#pragma unroll
    for (int v = 0; v < nV; v++) {
      qh[v] = fma(fac, qn[v], qh[v]);
      own[PT.at[v]] = last ? qh[v] : qn[v];
    }
    fac = fac * (dt / (i + 3));
  }
  __syncthreads();
  gradients();  // of the time-averaged state, for the fluxes
  if (lQhi_out && active)
#pragma unroll
    for (int v = 0; v < nD; v++) lQhi_out[((size_t)cell * P + p) * nD + v] = v < nV ? qh[v < nV ? v : 0] : Qp[v];
  // extrapolated states (parameters included), written by consecutive threads
  double* Qb = lQhbnd + (size_t)cell * 2 * DIM * F * nD;
  double* Fb = lFhbnd + (size_t)cell * 2 * DIM * F * nV;
  if (active) {
#pragma unroll
    for (int d = 0; d < DIM; d++)
      for (int it = p; it < LINES * nD; it += P) {
        const int L = it / nD, v = it - L * nD;
        const double* q = sC + plane(v) + C::line0(d, L);
        double sl = 0.0, sr = 0.0;
#pragma unroll
        for (int l = 0; l < b; l++) {
          const double a = q[l * C::step(d)];
          sl += a * T.FL[l];
          sr += a * T.FR[l];
        }
        Qb[2 * d * F * nD + it] = sl;
        Qb[(2 * d + 1) * F * nD + it] = sr;
      }
  }
  __syncthreads();
  // time-averaged fluxes one direction at a time: the node's values to shared
  // memory (where nothing is read any more: the state planes, then, where they fit,
  // the planes behind the first direction's fluxes, then the first's again), their
  // extrapolation from there; volumeIntegralLinear is pointwise
  double du[nV];
  double psw[nV];
  if constexpr (PS)
    if (here) NodePointSource<DIM, N, PDE>(geo, pc, ph, p).sum(pt, dt, psw);
#pragma unroll
  for (int v = 0; v < nV; v++) du[v] = 0.0;
  const double w = (DIM == 3 ? T.w[z] * T.w[y] : T.w[y]) * T.w[x];
#pragma unroll
  for (int d = 0; d < DIM; d++) {
    double B[nV];
    product(Qp, d, B);
    if constexpr (PS) {  // the time integral of the source, split over the directions (:294-308)
      if (here)
#pragma unroll
        for (int v = 0; v < nV; v++) B[v] = __dadd_rn(B[v], __ddiv_rn(psw[v], (double)DIM));
    }
    constexpr int BEHIND = C::kBehind ? nV * PL : 0;
    if (!C::kBehind && d > 0) __syncthreads();
    double* st = sC + (d == 1 ? BEHIND : 0);
#pragma unroll
    for (int v = 0; v < nV; v++) {
      du[v] -= w * B[v];
      (own + (d == 1 ? BEHIND : 0))[v * PL] = B[v];
    }
    if (lFhi_out && active)
#pragma unroll
      for (int v = 0; v < nV; v++) lFhi_out[(((size_t)cell * DIM + d) * P + p) * nV + v] = B[v];
    __syncthreads();
    if (active)
      for (int it = p; it < LINES * nV; it += P) {
        const int L = it / nV, v = it - L * nV;
        const double* q = st + v * PL + C::line0(d, L);
        double sl = 0.0, sr = 0.0;
#pragma unroll
        for (int l = 0; l < b; l++) {
          const double a = q[l * C::step(d)];
          sl += a * T.FL[l];
          sr += a * T.FR[l];
        }
        Fb[2 * d * F * nV + it] = sl;
        Fb[(2 * d + 1) * F * nV + it] = sr;
      }
  }
  if (!lduh) return;
  __syncthreads();
  // staged node by node and written by consecutive threads
#pragma unroll
  for (int v = 0; v < nV; v++) sC[p * nV + v] = du[v];
  __syncthreads();
  if (active)
#pragma unroll
    for (int k = 0; k < nV; k++) lduh[(size_t)cell * P * nV + k * P + p] = sC[k * P + p];
}

// The linear Riemann solve of one face by one warp: face averages of both
// sides (parameters included), smax from both averages' eigenvalues, Bn the
// PDE's coefficient matrix in their mean, then per face node
// FL = (Bn - smax I)^T dQ and FR = (Bn + smax I)^T dQ with dQ = (QR - QL) / 2.
// Bn^T dQ is the PDE's product of the normal direction applied to dQ
// (ncp_dir: what it reads is all the matrix holds). sL, sR: both sides' states
// in shared memory (FaceStage); the node's results take its state's place
// there and are written by consecutive lanes. FL or FR may be NULL (not written).
// (Row by row from the stored matrix every value took 2 nV shared loads; 9,975
// cells of 3D N=4 with wall faces and update: 195 -> 173 us.)
template <int DIM, int N, class PDE>
__device__ __forceinline__ void linear_face_flux(double* sL, double* sR, double* FL, double* FR, int dir, int lane) {
  using S = FaceStage<DIM, N, PDE>;
  constexpr int F = S::F, nV = S::nV, nD = S::nD, QP = S::PITCH;
  double av[nD];
  face_averages<DIM, N, PDE>(sL, sR, lane, av);
  const double smax = warp_face_smax<DIM, PDE>(av, dir, lane);
#pragma unroll
  for (int k = 0; k < nD; k++) av[k] = 0.5 * (av[k] + __shfl_xor_sync(0xffffffffu, av[k], 16));
  for (int fn = lane; fn < F; fn += 32) {
    double dq[nV], B[nV];
#pragma unroll
    for (int k = 0; k < nV; k++) dq[k] = 0.5 * (sR[fn * QP + k] - sL[fn * QP + k]);
    if (dir == 0)
      PDE::ncp_dir(av, 0, dq, B);
    else if (dir == 1)
      PDE::ncp_dir(av, 1, dq, B);
    else
      PDE::ncp_dir(av, 2, dq, B);
#pragma unroll
    for (int k = 0; k < nV; k++) {
      sL[fn * QP + k] = fma(-smax, dq[k], B[k]);
      sR[fn * QP + k] = fma(smax, dq[k], B[k]);
    }
  }
  __syncwarp();
  for (int e = lane; e < F * nV; e += 32) {
    const int fn = e / nV, k = e - fn * nV;
    if (FL) FL[e] = sL[fn * QP + k];
    if (FR) FR[e] = sR[fn * QP + k];
  }
}

// riemannSolverLinear on interior faces, one warp per face. FL goes to the
// left cell's face 2 dir + 1, FR to the right cell's face 2 dir; the
// extrapolated fluxes there are not read.
template <int DIM, int N, class PDE>
__global__ void __launch_bounds__(128) riemann_linear_kernel(const double* __restrict__ lQhbnd,
                                                             double* __restrict__ lFhbnd,
                                                             const int* __restrict__ face_left,
                                                             const int* __restrict__ face_right,
                                                             const int* __restrict__ face_dir, int nfaces,
                                                             const int* __restrict__ gate = nullptr) {
  using S = FaceStage<DIM, N, PDE>;
  constexpr int F = S::F, nV = S::nV, nD = S::nD;
  constexpr int E = F * nD, EPL = (E + 31) / 32;
  __shared__ double sQ[4][2][S::SIZE];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int f = blockIdx.x * (blockDim.x >> 5) + w;
  if (gate && !*gate) return;
  if (f >= nfaces) return;
  const int cl = face_left[f], cr = face_right[f], dir = face_dir[f];
  const double* QL = lQhbnd + ((size_t)cl * 2 * DIM + 2 * dir + 1) * E;
  const double* QR = lQhbnd + ((size_t)cr * 2 * DIM + 2 * dir) * E;
  double* FL = lFhbnd + ((size_t)cl * 2 * DIM + 2 * dir + 1) * F * nV;
  double* FR = lFhbnd + ((size_t)cr * 2 * DIM + 2 * dir) * F * nV;
  // all of the face's loads in flight before the first shared store
  double ql[EPL], qr[EPL];
#pragma unroll
  for (int i = 0; i < EPL; i++) {
    const int e = lane + 32 * i;
    ql[i] = e < E ? QL[e] : 0.0;
    qr[i] = e < E ? QR[e] : 0.0;
  }
#pragma unroll
  for (int i = 0; i < EPL; i++) {
    const int e = lane + 32 * i;
    if (e < E) {
      sQ[w][0][S::at(e)] = ql[i];
      sQ[w][1][S::at(e)] = qr[i];
    }
  }
  __syncwarp();
  linear_face_flux<DIM, N, PDE>(sQ[w][0], sQ[w][1], FL, FR, dir, lane);
}

// Boundary faces of a linear solver: ADERDGSolver::applyBoundaryConditions
// (exahype/solvers/ADERDGSolver.cpp:2893-2962) -- the PDE's boundaryValues
// at every face node (boundaryConditions, 3d/boundaryConditions.cpph:24-85),
// staged in shared memory beside the inside state, then riemannSolverLinear
// with the outside state on the outer side (QOut, QIn for an even face, QIn,
// QOut for an odd one); only the cell's own fluctuation is written. One warp
// per boundary face.
template <int DIM, int N, class PDE>
__global__ void __launch_bounds__(128) boundary_linear_kernel(const double* __restrict__ lQhbnd,
                                                              double* __restrict__ lFhbnd,
                                                              const int* __restrict__ bcell,
                                                              const int* __restrict__ bface, int nb, int kind,
                                                              const int* __restrict__ gate = nullptr) {
  using S = FaceStage<DIM, N, PDE>;
  constexpr int F = S::F, nV = S::nV, nD = S::nD, QP = S::PITCH;
  constexpr int E = F * nD;
  __shared__ double sQ[4][2][S::SIZE];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int f = blockIdx.x * (blockDim.x >> 5) + w;
  if (f >= nb || (gate && !*gate)) return;
  const int c = bcell[f], face = bface[f], dir = face >> 1;
  const double* QIn = lQhbnd + ((size_t)c * 2 * DIM + face) * E;
  double* FIn = lFhbnd + ((size_t)c * 2 * DIM + face) * F * nV;
  const bool even = (face & 1) == 0;
  double* sIn = sQ[w][even ? 1 : 0];
  double* sOut = sQ[w][even ? 0 : 1];
  for (int e = lane; e < E; e += 32) sIn[S::at(e)] = QIn[e];
  __syncwarp();
  for (int fn = lane; fn < F; fn += 32) {
    double fo[nV];
    PDE::template boundaryValues<DIM>(kind, dir, FIn + fn * nV, sIn + fn * QP, fo, sOut + fn * QP);
  }
  __syncwarp();
  linear_face_flux<DIM, N, PDE>(sQ[w][0], sQ[w][1], even ? nullptr : FIn, even ? FIn : nullptr, dir, lane);
}

// volumeIntegralLinear alone: lduh = -w_node sum_d lFhi[d], lFhi per cell [d][b^d][nV]
template <int DIM, int N, class PDE>
__global__ void volume_linear_kernel(double* __restrict__ lduh, const double* __restrict__ lFhi, int ncells) {
  using S = Shape<DIM, N, PDE>;
  constexpr int b = S::b, P = S::P, nV = S::nV;
  const OrderTables& T = c_tab[N];
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= (long long)ncells * P) return;
  const int cell = (int)(i / P), p = (int)(i - (long long)cell * P);
  const int x = p % b, y = (p / b) % b, z = DIM == 3 ? p / (b * b) : 0;
  const double w = (DIM == 3 ? T.w[z] * T.w[y] : T.w[y]) * T.w[x];
#pragma unroll
  for (int v = 0; v < nV; v++) {
    double du = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; d++) du -= w * lFhi[(((size_t)cell * DIM + d) * P + p) * nV + v];
    lduh[((size_t)cell * P + p) * nV + v] = du;
  }
}

}  // namespace exa
