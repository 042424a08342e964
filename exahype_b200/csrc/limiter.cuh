// A-posteriori subcell limiter on the GPU: DG <-> FV projections, DMP and
// admissibility, MUSCL-Hancock FV update of limited cells, FV halo exchange
// and the limiter status machine, for the Euler PDE (nV = 5, no parameters).
//
// Reference semantics (cited per kernel): kernels/limiter/generic/c/Limiter.cpp,
// kernels/finitevolumes/musclhancock/c/{2d,3d}/musclhancock.cpph,
// kernels/finitevolumes/commons/c/commons.cpph and the sequencing of
// exahype/solvers/LimitingADERDGSolver.cpp.
//
// FV patches: lim[cell][(z)][y][x][nV], E = 2N+1+2g cells per axis, g = 2 ghost
// layers; the ghost corners stay zero (never written by the halo exchange).
// Per-cell status data: s (limiter status), s_prev, cure counter, facewise
// statuses fs[2d], has_lim (patch allocated), DMP blocks minB/maxB[2d][nV].
#pragma once
#include <type_traits>

#include "aderdg.cuh"

namespace exa {

constexpr int kGW = 2;  // ghost layer width (GenericFiniteVolumesMUSCLHancockInC.java:12)

template <int DIM, int N>
struct LimShape {
  static constexpr int b = N + 1;
  static constexpr int B = 2 * N + 1;
  static constexpr int E = B + 2 * kGW;
  static constexpr int P = ipow(b, DIM);
  static constexpr int PB = ipow(B, DIM);   // subcells
  static constexpr int PE = ipow(E, DIM);   // patch cells incl. ghosts
  static constexpr int nV = 5;
  static constexpr int LS = PE * nV;        // doubles per patch
};

struct LimParams {
  int A, T, cure_steps;  // activeFV = h+1, troubled = 2h+1, steps-till-cured
  double relax, scale;   // DMP delta0 and epsilon
};

// patch index of interior subcell (z,y,x) (0-based in [0,B))
template <int DIM, int N>
__device__ __forceinline__ int lim_index(int z, int y, int x) {
  using L = LimShape<DIM, N>;
  return DIM == 3 ? (((z + kGW) * L::E + y + kGW) * L::E + x + kGW) : ((y + kGW) * L::E + x + kGW);
}

// ---------------------------------------------------------------------------
// The threads that process one cell: a whole block, or one warp of a block
// that holds several cells (small 2D cells, where block-wide barriers would
// dominate the little work per cell).
struct BlockGroup {
  __device__ static int tid() { return threadIdx.x; }
  __device__ static int size() { return blockDim.x; }
  __device__ static int index() { return 0; }
  __device__ static void sync() { __syncthreads(); }
};
struct WarpGroup {
  __device__ static int tid() { return threadIdx.x & 31; }
  __device__ static int size() { return 32; }
  __device__ static int index() { return threadIdx.x >> 5; }
  __device__ static void sync() { __syncwarp(); }
};

// Copies src[0..n) to dst[0..n), eight loads per thread in flight before the
// stores (dst may be shared memory).
template <class G>
__device__ __forceinline__ void copy_group(double* __restrict__ dst, const double* __restrict__ src, int n) {
  constexpr int K = 8;
  for (int i0 = G::tid(); i0 < n; i0 += K * G::size()) {
    double x[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      const int i = i0 + k * G::size();
      if (i < n) x[k] = src[i];
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
      const int i = i0 + k * G::size();
      if (i < n) dst[i] = x[k];
    }
  }
}

// Exchanges the contents of a[0..n) and b[0..n) (the reference swaps a
// patch's solution and previous-solution pointers; here both live in dense
// per-cell arrays). Each thread issues the loads of eight elements of both
// arrays before any store, so that a group of one warp waits on a few
// memory round trips, not one per 32 elements.
template <class G>
__device__ __forceinline__ void swap_group(double* __restrict__ a, double* __restrict__ b, int n) {
  constexpr int K = 8;
  for (int i0 = G::tid(); i0 < n; i0 += K * G::size()) {
    double x[K], y[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      const int i = i0 + k * G::size();
      if (i < n) {
        x[k] = a[i];
        y[k] = b[i];
      }
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
      const int i = i0 + k * G::size();
      if (i < n) {
        a[i] = y[k];
        b[i] = x[k];
      }
    }
  }
}

// The 1-D projections of one order in constant memory: DG basis k -> subcell i
// [k][i], subcell i -> DG basis j [i][j], DG basis j at Lobatto node i [j][i].
template <int N>
struct ProjTables {
  static constexpr int b = N + 1, B = 2 * N + 1;
  double uh2lim[b * B], lim2uh[B * b], uh2lob[b * b];
};
struct ProjTablesAll {
  ProjTables<3> n3;
  ProjTables<4> n4;
  ProjTables<5> n5;
  ProjTables<7> n7;
};
__constant__ ProjTablesAll c_proj;
template <int N>
__device__ __forceinline__ const ProjTables<N>& proj_tab() {
  static_assert(N == 3 || N == 4 || N == 5 || N == 7, "no projection tables of this order");
  if constexpr (N == 3) return c_proj.n3;
  else if constexpr (N == 4) return c_proj.n4;
  else if constexpr (N == 5) return c_proj.n5;
  else return c_proj.n7;
}
enum class Proj { kToFV, kToDG, kToLobatto };
template <int N, Proj P>
__device__ __forceinline__ const double* proj_matrix() {
  return P == Proj::kToFV ? proj_tab<N>().uh2lim : P == Proj::kToDG ? proj_tab<N>().lim2uh : proj_tab<N>().uh2lob;
}

// Threads of a group that work on the lines of a tensor map: a multiple of the
// five variables, so that a thread keeps one variable (tid % 5) throughout.
template <class G>
__device__ __forceinline__ int line_threads() { return G::size() / 5 * 5; }

// out[o] = sum_i in[i] M[i][o] of one line, the matrix entries compile-time
// constant-memory operands
template <int IN, int OUT, class Out>
__device__ __forceinline__ void map_line(const double (&in)[IN], const double* M, Out out) {
#pragma unroll
  for (int o = 0; o < OUT; o++) {
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < IN; i++) s += in[i] * M[i * OUT + o];
    out(o, s);
  }
}

// Separable tensor-product maps for one cell, executed by one thread group.
// out[o1..][v] = sum_in src[in..][v] prod_d M[in_d][o_d], M row-major [IN][OUT].
// Summation is per axis (x, then y, then z) rather than the reference's single
// triple loop; the difference is at round-off level. A thread takes whole
// lines: it loads a line's IN values once and forms all OUT of its outputs (per
// output value each would load IN values and IN matrix entries, which made the
// projections shared-memory bound: 729 patches 3D N=5 to subcells 38 -> 13 us,
// a limiting step of 81^2 N=5 209 -> 195 us). Each loop over the lines stays a
// loop: its body is already OUT chains wide. dst is called with the thread's own
// variable, tid % 5.
template <int DIM, int IN, int OUT, class G = BlockGroup, class Src, class Dst>
__device__ void tensor_map(Src src, Dst dst, const double* M, double* tmp) {
  constexpr int nV = 5;
  const int A = line_threads<G>(), tid = G::tid(), v = tid % nV;
  if constexpr (DIM == 2) {
    if (tid < A) {
#pragma unroll 1
      for (int l = tid; l < IN * nV; l += A) {  // t[y][xo][v], line (y, v)
        const int y = l / nV;
        double in[IN];
#pragma unroll
        for (int x = 0; x < IN; x++) in[x] = src(0, y, x, v);
        map_line<IN, OUT>(in, M, [&](int xo, double s) { tmp[(y * OUT + xo) * nV + v] = s; });
      }
    }
    G::sync();
    if (tid < A) {
#pragma unroll 1
      for (int l = tid; l < OUT * nV; l += A) {  // line (xo, v)
        const int xo = l / nV;
        double in[IN];
#pragma unroll
        for (int y = 0; y < IN; y++) in[y] = tmp[y * OUT * nV + l];
        map_line<IN, OUT>(in, M, [&](int yo, double s) { dst(0, yo, xo, v, s); });
      }
    }
  } else {
    double* t1 = tmp;                      // [z][y][xo][v]
    double* t2 = tmp + IN * IN * OUT * nV;  // [z][yo][xo][v]
    if (tid < A) {
#pragma unroll 1
      for (int l = tid; l < IN * IN * nV; l += A) {  // line (z, y, v)
        const int zy = l / nV, z = zy / IN, y = zy - z * IN;
        double in[IN];
#pragma unroll
        for (int x = 0; x < IN; x++) in[x] = src(z, y, x, v);
        map_line<IN, OUT>(in, M, [&](int xo, double s) { t1[(zy * OUT + xo) * nV + v] = s; });
      }
    }
    G::sync();
    if (tid < A) {
#pragma unroll 1
      for (int l = tid; l < IN * OUT * nV; l += A) {  // line (z, xo, v)
        const int z = l / (OUT * nV), r = l - z * (OUT * nV);
        double in[IN];
#pragma unroll
        for (int y = 0; y < IN; y++) in[y] = t1[(z * IN + y) * OUT * nV + r];
        map_line<IN, OUT>(in, M, [&](int yo, double s) { t2[(z * OUT + yo) * OUT * nV + r] = s; });
      }
    }
    G::sync();
    if (tid < A) {
#pragma unroll 1
      for (int l = tid; l < OUT * OUT * nV; l += A) {  // line (yo, xo, v)
        const int yx = l / nV, yo = yx / OUT, xo = yx - yo * OUT;
        double in[IN];
#pragma unroll
        for (int z = 0; z < IN; z++) in[z] = t2[z * OUT * OUT * nV + l];
        map_line<IN, OUT>(in, M, [&](int zo, double s) { dst(zo, yo, xo, v, s); });
      }
    }
  }
  G::sync();
}

template <int DIM, int IN, int OUT>
constexpr int tensor_tmp() {
  return DIM == 2 ? IN * OUT * 5 : (IN * IN * OUT + IN * OUT * OUT) * 5;
}

// projectOnFVLimiterSpace (Limiter.cpp:23-66): DG nodes -> interior subcells
template <int DIM, int N, class G = BlockGroup>
__device__ void project_fv_block(const double* luh, double* lim, double* tmp) {
  using L = LimShape<DIM, N>;
  tensor_map<DIM, L::b, L::B, G>(
      [&](int z, int y, int x, int v) { return luh[(((DIM == 3 ? z * L::b : 0) + y) * L::b + x) * L::nV + v]; },
      [&](int z, int y, int x, int v, double s) { lim[lim_index<DIM, N>(z, y, x) * L::nV + v] = s; },
      proj_matrix<N, Proj::kToFV>(), tmp);
}
// projectOnDGSpace (Limiter.cpp:69-112): interior subcells -> DG nodes
template <int DIM, int N, class G = BlockGroup>
__device__ void project_dg_block(const double* lim, double* luh, double* tmp) {
  using L = LimShape<DIM, N>;
  tensor_map<DIM, L::B, L::b, G>(
      [&](int z, int y, int x, int v) { return lim[lim_index<DIM, N>(z, y, x) * L::nV + v]; },
      [&](int z, int y, int x, int v, double s) { luh[(((DIM == 3 ? z * L::b : 0) + y) * L::b + x) * L::nV + v] = s; },
      proj_matrix<N, Proj::kToDG>(), tmp);
}

// running minimum and maximum (a NaN never replaces them)
struct MinMax {
  double mn, mx;
  __device__ __forceinline__ MinMax() : mn(1.7976931348623157e308), mx(-1.7976931348623157e308) {}  // DBL_MAX
  __device__ __forceinline__ void fold(double lo, double hi) {
    mn = (lo < mn) ? lo : mn;
    mx = (mx < hi) ? hi : mx;
  }
};

// min/max per variable over a group whose thread tid < line_threads holds
// those of variable tid % 5. One warp: lane v < 5 ends with variable v's
// (lanes 5 apart hold the same variable: three exchanges).
__device__ __forceinline__ MinMax warp_minmax_lines(MinMax m) {
  if ((threadIdx.x & 31) >= 30) m = MinMax();
#pragma unroll
  for (int o : {15, 10, 5}) {
    // (other lanes fold values of their own variable, or neutral ones)
    const double lo = __shfl_down_sync(0xffffffffu, m.mn, o), hi = __shfl_down_sync(0xffffffffu, m.mx, o);
    m.fold(lo, hi);
  }
  return m;
}
// The same over a whole block, through shared memory (red: 2 blockDim.x + 10
// doubles): every thread ends with all five.
__device__ __forceinline__ void block_minmax_lines(MinMax m, double* mn, double* mx, double* red) {
  const int n = blockDim.x, A = line_threads<BlockGroup>();
  red[threadIdx.x] = m.mn;
  red[n + threadIdx.x] = m.mx;
  __syncthreads();
  if (threadIdx.x < 32) {
    MinMax r;
    if (threadIdx.x < 30)
      for (int i = threadIdx.x; i < A; i += 30) r.fold(red[i], red[n + i]);
    r = warp_minmax_lines(r);
    if (threadIdx.x < 5) {
      red[2 * n + threadIdx.x] = r.mn;
      red[2 * n + 5 + threadIdx.x] = r.mx;
    }
  }
  __syncthreads();
#pragma unroll
  for (int v = 0; v < 5; v++) {
    mn[v] = red[2 * n + v];
    mx[v] = red[2 * n + 5 + v];
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------
// Face merge (mergeSolutionMinMaxOnFace :1654-1690, mergeNeighboursLimiterStatus
// ADERDGSolver.cpp:2544-2595): one thread per interior face.
__host__ __device__ __forceinline__ int merged_face_status(int s1, int s2, int T) {
  const int a = s1 < T ? s1 : T, b = s2 < T ? s2 : T, m = (a < b ? b : a) - 1;
  return m > 0 ? m : 0;
}
template <int DIM>
__global__ void lim_merge_faces_kernel(const int* __restrict__ fl, const int* __restrict__ fr,
                                       const int* __restrict__ fd, int nfaces, const int* __restrict__ s,
                                       double* __restrict__ minB, double* __restrict__ maxB, int* __restrict__ fs,
                                       int T, const int* __restrict__ gate) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= nfaces || (gate && !*gate)) return;
  constexpr int D2 = 2 * DIM;
  const int c1 = fl[f], c2 = fr[f], d = fd[f];
  const int f1 = 2 * d + 1, f2 = 2 * d;
  const int v = merged_face_status(s[c1], s[c2], T);
  fs[c1 * D2 + f1] = v;
  fs[c2 * D2 + f2] = v;
  double* mn1 = minB + ((size_t)c1 * D2 + f1) * 5;
  double* mn2 = minB + ((size_t)c2 * D2 + f2) * 5;
  double* mx1 = maxB + ((size_t)c1 * D2 + f1) * 5;
  double* mx2 = maxB + ((size_t)c2 * D2 + f2) * 5;
  // all twenty loads before the first store (the four blocks lie in one
  // array each, so the compiler could not move a load above a store)
  double a1[5], a2[5], b1[5], b2[5];
#pragma unroll
  for (int i = 0; i < 5; i++) {
    a1[i] = mn1[i];
    a2[i] = mn2[i];
    b1[i] = mx1[i];
    b2[i] = mx2[i];
  }
#pragma unroll
  for (int i = 0; i < 5; i++) {
    const double mn = (a2[i] < a1[i]) ? a2[i] : a1[i];
    const double mx = (b1[i] < b2[i]) ? b2[i] : b1[i];
    mn1[i] = mn2[i] = mn;
    mx1[i] = mx2[i] = mx;
  }
}

// FV halo exchange (ghostLayerFilling, commons.cpph:336-401 / :873-981) on
// interior faces where either side is FV-active, and the outflow FV boundary
// (boundaryLayerExtraction + boundaryConditions + ghostLayerFillingAtBoundary,
// commons.cpph:98-334) on boundary faces of FV-active cells. One warp per face.
template <int DIM, int N>
__global__ void __launch_bounds__(128) lim_fv_halo_kernel(const int* __restrict__ fl, const int* __restrict__ fr,
                                                          const int* __restrict__ fd, int nfaces,
                                                          const int* __restrict__ bcell, const int* __restrict__ bface,
                                                          int nb, int nb_out, const int* __restrict__ s,
                                                          const int* __restrict__ has_lim, double* __restrict__ lim,
                                                          int A, const int* __restrict__ gate) {
  using L = LimShape<DIM, N>;
  constexpr int E = L::E, B = L::B, nV = L::nV;
  const int lane = threadIdx.x & 31;
  const int f = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (f >= nfaces + nb || (gate && !*gate)) return;
  constexpr int TR = DIM == 3 ? B * B : B;  // transverse subcells of a face
  constexpr int WORK = TR * kGW * nV;
  auto cell_at = [&](int d, int a, int c, int k) {  // (a, c) transverse, k along d
    int z, y, x;
    if (d == 0) { z = a; y = c; x = k; }
    else if (d == 1) { z = a; y = k; x = c; }
    else { z = k; y = a; x = c; }
    return DIM == 3 ? (z * E + y) * E + x : y * E + x;
  };
  const int zr = DIM == 3 ? kGW : 0;
  if (f < nfaces) {
    const int c1 = fl[f], c2 = fr[f], d = fd[f];
    if (!(s[c1] >= A || s[c2] >= A) || !has_lim[c1] || !has_lim[c2]) return;
    double* l1 = lim + (size_t)c1 * L::LS;
    double* l2 = lim + (size_t)c2 * L::LS;
    for (int i = lane; i < WORK; i += 32) {
      const int v = i % nV, k = (i / nV) % kGW, t = i / (nV * kGW);
      const int a = DIM == 3 ? t / B + kGW : (d == 2 ? 0 : zr), c = (DIM == 3 ? t % B : t) + kGW;
      const int aa = DIM == 3 ? a : 0;
      // c1's +d ghosts from c2's first layers; c2's -d ghosts from c1's last layers
      l1[cell_at(d, aa, c, B + kGW + k) * nV + v] = l2[cell_at(d, aa, c, kGW + k) * nV + v];
      l2[cell_at(d, aa, c, k) * nV + v] = l1[cell_at(d, aa, c, B + k) * nV + v];
    }
  } else {
    // boundary faces: the first nb_out outflow, the others rigid walls
    const int bf = f - nfaces, c = bcell[bf], face = bface[bf], d = face >> 1, side = face & 1;
    const bool wall = bf >= nb_out;
    if (!(s[c] >= A) || !has_lim[c]) return;
    double* l = lim + (size_t)c * L::LS;
    for (int i = lane; i < WORK; i += 32) {
      const int v = i % nV, k = (i / nV) % kGW, t = i / (nV * kGW);
      const int a = DIM == 3 ? t / B + kGW : 0, cc = (DIM == 3 ? t % B : t) + kGW;
      // the mirrored layer is the inside state; at 3D y- and z-left faces the
      // reference's boundaryLayerExtraction (commons.cpph:551-562, :581-592)
      // takes the first interior layer for both ghost layers
      const int K = kGW - k - 1;
      const int gi = side ? B + kGW + k : k;
      const int si = side ? B + K : kGW + ((DIM == 3 && d >= 1) ? 0 : K);
      // PDE::fvBoundaryValues: outflow copies it, the wall negates the normal momentum
      const double q = l[cell_at(d, a, cc, si) * nV + v];
      l[cell_at(d, a, cc, gi) * nV + v] = (wall && v == 1 + d) ? -q : q;
    }
  }
}

// ---------------------------------------------------------------------------
// MUSCL-Hancock (2d/musclhancock.cpph:50-276, 3d/musclhancock.cpph) on the
// cells of `list` (length *count when count is given, else nlist; list NULL:
// cells 0..n-1), then projectOnDGSpace of the result into luh (unless NULL). Before the
// update lim_prev <- lim (FiniteVolumesSolver::updateSolution,
// FiniteVolumesSolver.cpp:662-715). In 2D (lim_muscl_kernel) the evolved
// boundary states and the edge fluxes of the whole patch live in shared
// memory beside the patch itself; in 3D (lim_muscl3_kernel) those of one plane.
template <int N>
struct MusclCfg {
  using L = LimShape<2, N>;
  static constexpr int R = L::B + 2;  // interior + first ghost ring per axis
  static constexpr int NR = R * R;
  static constexpr int W = NR * 2 * 2 * L::nV;     // evolved wL/wR
  static constexpr int NE = (L::B + 1) * L::B;     // edges per direction
  static constexpr int FX = 2 * NE * L::nV;        // edge fluxes
  static constexpr int U = L::LS;                  // the patch
  // a thread per edge of both directions (and per subcell of the ring, which
  // are fewer): each phase is one round. A patch is a chain of three short
  // phases, so what counts is how many are in flight: three blocks an SM up to
  // N = 5 (81^2 N=5, about a tenth of the cells: 20.5 us with 256 threads and
  // the neighbours read from global memory, 16.2 with two blocks, 13.5 with
  // three). At N = 7 shared memory holds two blocks; for their registers the 480
  // edges take two rounds of 320 threads (one block of 480 threads is as fast up to
  // 148 patches, 11 us; 300: 25 -> 21, 1,000: 58 -> 42, 4,000: 241 -> 158).
  static constexpr int THREADS = N == 7 ? 320 : (2 * NE + 31) / 32 * 32;
  static constexpr int MINB = N == 7 ? 2 : 3;
  static constexpr size_t SMEM = sizeof(double) * (U + W + FX);
  static_assert(NR <= THREADS, "one subcell of the ring per thread");
  static_assert(tensor_tmp<2, L::B, L::b>() <= W, "the projection's scratch takes the states' place");
};

__device__ __forceinline__ double minmod_dev(double a, double b) {  // musclhancock.cpph:29-38
  if (a * b < 0.0) return 0.0;
  if (fabs(a) < fabs(b)) return a;
  return b;
}

template <int DIM, class PDE>
__device__ __forceinline__ void dir_flux(const double* q, int d, double* f) {
  double F[DIM][5];
  PDE::template flux<DIM>(q, F);
#pragma unroll
  for (int v = 0; v < 5; v++) f[v] = F[d][v];
}

// Rusanov flux on the subcell edge of direction d between the states ql and qr (rusanov.cpph)
template <int DIM, class PDE>
__device__ __forceinline__ void edge_flux(const double* ql, const double* qr, int d, double* f) {
  double lL[5], lR[5];
  Hooks<PDE, DIM>::eigenvalues(ql, d, lL);
  Hooks<PDE, DIM>::eigenvalues(qr, d, lR);
  double smax = -1.0;
#pragma unroll
  for (int v = 0; v < 5; v++) smax = (fabs(lL[v]) < smax) ? smax : fabs(lL[v]);
#pragma unroll
  for (int v = 0; v < 5; v++) smax = (fabs(lR[v]) < smax) ? smax : fabs(lR[v]);
  double fl[5], fr[5];
  dir_flux<DIM, PDE>(ql, d, fl);
  dir_flux<DIM, PDE>(qr, d, fr);
#pragma unroll
  for (int v = 0; v < 5; v++) {
    double fn = 0.5 * smax * (ql[v] - qr[v]);
    fn += 0.5 * (fl[v] + fr[v]);
    f[v] = fn;
  }
}

template <int N, class PDE>
__global__ void __launch_bounds__(MusclCfg<N>::THREADS, MusclCfg<N>::MINB)
    lim_muscl_kernel(const int* __restrict__ list, const int* __restrict__ count, int nlist, double* __restrict__ lim,
                     double* __restrict__ lim_prev, double* __restrict__ luh, Geometry geo,
                     const double* __restrict__ dt_ptr, const int* __restrict__ gate) {
  constexpr int DIM = 2;
  using L = LimShape<2, N>;
  using C = MusclCfg<N>;
  constexpr int E = L::E, B = L::B, nV = L::nV, R = C::R;
  if (gate && !*gate) return;
  extern __shared__ double smem[];
  double* sU = smem;  // the patch: read once from global memory
  double* W = sU + C::U;
  double* FX = W + C::W;
  const double dt = *dt_ptr;
  double cs[DIM], ics[DIM], icsdt[DIM];
  for (int d = 0; d < DIM; d++) {
    cs[d] = geo.dx[d] / B;
    ics[d] = 1. / cs[d];
    icsdt[d] = dt * ics[d];
  }
  const int n = count ? *count : nlist;
  for (int li = blockIdx.x; li < n; li += gridDim.x) {
    const int cell = list ? list[li] : li;
    double* l = lim + (size_t)cell * L::LS;
    double* lp = lim_prev + (size_t)cell * L::LS;
    for (int i = threadIdx.x; i < L::LS; i += C::THREADS) lp[i] = sU[i] = l[i];
    __syncthreads();
    auto U = [&](int y, int x, int v) { return sU[(y * E + x) * nV + v]; };
    // slopes, extrapolation and half-step evolution on interior + first ghost ring
    if (threadIdx.x < C::NR) {
      const int q = threadIdx.x;
      const int x = q % R + kGW - 1, y = q / R + kGW - 1;
      double wl[DIM][5], wr[DIM][5];
#pragma unroll
      for (int v = 0; v < nV; v++) {
        const double u = U(y, x, v);
        const double sx = minmod_dev(U(y, x + 1, v) - u, u - U(y, x - 1, v)) * ics[0];
        wl[0][v] = u - 0.5 * cs[0] * sx;
        wr[0][v] = u + 0.5 * cs[0] * sx;
        const double sy = minmod_dev(U(y + 1, x, v) - u, u - U(y - 1, x, v)) * ics[1];
        wl[1][v] = u - 0.5 * cs[1] * sy;
        wr[1][v] = u + 0.5 * cs[1] * sy;
      }
      double Qt[5] = {0, 0, 0, 0, 0};
#pragma unroll
      for (int d = 0; d < DIM; d++) {
        double f[5];
        dir_flux<DIM, PDE>(wl[d], d, f);
#pragma unroll
        for (int v = 0; v < nV; v++) Qt[v] += f[v] * ics[d];
        dir_flux<DIM, PDE>(wr[d], d, f);
#pragma unroll
        for (int v = 0; v < nV; v++) Qt[v] -= f[v] * ics[d];
      }
#pragma unroll
      for (int d = 0; d < DIM; d++)
#pragma unroll
        for (int v = 0; v < nV; v++) {  // [d][left, right][v][subcell]: consecutive threads, consecutive banks
          W[((d * 2 + 0) * nV + v) * C::NR + q] = wl[d][v] + 0.5 * dt * Qt[v];
          W[((d * 2 + 1) * nV + v) * C::NR + q] = wr[d][v] + 0.5 * dt * Qt[v];
        }
    }
    __syncthreads();
    // Rusanov flux on every subcell edge: edge e of direction d
    // joins positions k and k+1 along d, k in [-1, B) relative to the interior
#pragma unroll 1
    for (int i = threadIdx.x; i < DIM * C::NE; i += C::THREADS) {
      const int d = i / C::NE, e = i % C::NE;
      const int kk = e % (B + 1), t = e / (B + 1);  // position k + 1 along d, transverse interior coordinate
      const int qL = d == 0 ? (t + 1) * R + kk : kk * R + t + 1;  // ring index 0 = first ghost layer
      const int qR = qL + (d == 0 ? 1 : R);
      double ql[5], qr[5], f[5];  // wR of the left subcell, wL of the right subcell
#pragma unroll
      for (int v = 0; v < nV; v++) {
        ql[v] = W[((d * 2 + 1) * nV + v) * C::NR + qL];
        qr[v] = W[((d * 2 + 0) * nV + v) * C::NR + qR];
      }
      edge_flux<DIM, PDE>(ql, qr, d, f);
#pragma unroll
      for (int v = 0; v < nV; v++) FX[i * nV + v] = f[v];
    }
    __syncthreads();
    // update of the interior subcells in the reference's accumulation order:
    // +left x edge, -right x edge, then y
    for (int i = threadIdx.x; i < L::PB * nV; i += C::THREADS) {
      const int v = i % nV, sc = i / nV;
      const int x = sc % B, y = sc / B;
      const int at = lim_index<2, N>(0, y, x) * nV + v;
      double u = sU[at];
      // edge index within direction d: (transverse t, k) with k = position + 1 for the left edge
      u += icsdt[0] * FX[(y * (B + 1) + x) * nV + v];
      u -= icsdt[0] * FX[(y * (B + 1) + x + 1) * nV + v];
      u += icsdt[1] * FX[(C::NE + x * (B + 1) + y) * nV + v];
      u -= icsdt[1] * FX[(C::NE + x * (B + 1) + y + 1) * nV + v];
      sU[at] = l[at] = u;
    }
    // the reference's edge loops also touch the first ghost layer on every
    // face (one edge each); the ghost corners stay untouched
    for (int i = threadIdx.x; i < DIM * 2 * B * nV; i += C::THREADS) {
      const int v = i % nV, t = (i / nV) % B, side = (i / (nV * B)) % 2, d = i / (nV * B * 2);
      const int c = t + kGW, k = side ? B + kGW : kGW - 1;
      const int at = (d == 0 ? c * E + k : k * E + c) * nV + v;
      const double f = FX[((d * C::NE) + t * (B + 1) + (side ? B : 0)) * nV + v];
      l[at] = side ? sU[at] + icsdt[d] * f : sU[at] - icsdt[d] * f;
    }
    __syncthreads();
    if (luh) project_dg_block<2, N>(sU, luh + (size_t)cell * L::P * nV, W);  // (ends with a barrier)
  }
}

// 3D: the patch is walked plane by plane along z, everything on chip. A thread
// owns the column (x, y) of the interior and the first ghost ring. Per plane it
// forms the column's evolved states from three patch planes in shared memory
// (each read once from global memory, one plane ahead, and copied to lim_prev
// on the way); the x and y states go to shared memory for the plane's edge
// fluxes, the z states stay in the thread: the flux between two planes needs
// the column's own states only. The update of a plane is finished, in the
// reference's order of terms, when its upper z flux is known, one plane
// later; planes not read any more are overwritten in place.
//
// FP64-bound: some 400 operations per subcell of the ring and 250 per edge
// (slopes, six and two flux evaluations with their divisions, two square
// roots), 2 M per patch at N = 5.
template <int N>
struct Muscl3Cfg {
  using L = LimShape<3, N>;
  static constexpr int E = L::E, B = L::B, R = B + 2, RR = R * R;
  static constexpr int THREADS = (RR + 31) / 32 * 32;
  static constexpr int PLANE = E * E * L::nV;
  static constexpr int KP = (PLANE + THREADS - 1) / THREADS;  // a plane's values per thread
  static constexpr int W = 20 * RR;                           // evolved x and y states of one plane [value][cell]
  static constexpr int NE = (B + 1) * B;                      // edges of one direction in a plane
  static constexpr int FX = 2 * NE * L::nV;
  static constexpr int TMP = tensor_tmp<3, L::B, L::b>();
  static constexpr int DATA = 3 * PLANE + W + FX > TMP ? 3 * PLANE + W + FX : TMP;
  static constexpr size_t SMEM = sizeof(double) * (size_t)DATA;
  static constexpr int MINB = N == 7 ? 1 : 2;
};

template <int N, class PDE>
__global__ void __launch_bounds__(Muscl3Cfg<N>::THREADS, Muscl3Cfg<N>::MINB)
    lim_muscl3_kernel(const int* __restrict__ list, const int* __restrict__ count, int nlist,
                      double* __restrict__ lim, double* __restrict__ lim_prev, double* __restrict__ luh, Geometry geo,
                      const double* __restrict__ dt_ptr, const int* __restrict__ gate) {
  using L = LimShape<3, N>;
  using C = Muscl3Cfg<N>;
  constexpr int E = C::E, B = C::B, R = C::R, RR = C::RR, PLANE = C::PLANE, KP = C::KP, NE = C::NE, nV = 5;
  if (gate && !*gate) return;
  extern __shared__ double smem[];
  double* sU = smem;                  // three planes of the patch, plane z in slot z % 3
  double* sW = smem + 3 * PLANE;      // [direction x, y][left, right][v][cell of the ring plane]
  double* sX = sW + C::W;             // [direction][v][edge]
  const double dt = *dt_ptr;
  double cs[3], ics[3], icsdt[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    cs[d] = geo.dx[d] / B;
    ics[d] = 1. / cs[d];
    icsdt[d] = dt * ics[d];
  }
  const int t = threadIdx.x;
  const bool ring = t < RR;
  const int x = t % R + 1, y = t / R + 1;  // patch coordinates of this thread's column
  const bool inX = x >= kGW && x < kGW + B, inY = y >= kGW && y < kGW + B;
  const int n = count ? *count : nlist;
  for (int li = blockIdx.x; li < n; li += gridDim.x) {
    const int cell = list ? list[li] : li;
    double* l = lim + (size_t)cell * L::LS;
    double* lp = lim_prev + (size_t)cell * L::LS;
    for (int i = t; i < 3 * PLANE; i += C::THREADS) {
      const double q = l[i];
      sU[i] = q;
      lp[i] = q;
    }
    __syncthreads();
    double up[nV], wz[nV], fz[nV];  // plane z-1 up to its upper z edge, its right z state, the z edge below plane z
#pragma unroll
    for (int v = 0; v < nV; v++) up[v] = wz[v] = fz[v] = 0.0;
#pragma unroll 1
    for (int zr = 0; zr < R; zr++) {
      const int z = zr + 1;
      double pf[KP];
      const bool more = z + 2 < E;
      if (more)
#pragma unroll
        for (int k = 0; k < KP; k++) {
          const int i = t + k * C::THREADS;
          pf[k] = i < PLANE ? l[(z + 2) * PLANE + i] : 0.0;
        }
      const double* U0 = sU + (z % 3) * PLANE + (y * E + x) * nV;
      if (ring) {
        const double* Um = sU + ((z + 2) % 3) * PLANE + (y * E + x) * nV;
        const double* Up = sU + ((z + 1) % 3) * PLANE + (y * E + x) * nV;
        double wl[3][nV], wr[3][nV];
#pragma unroll
        for (int v = 0; v < nV; v++) {
          const double u = U0[v];
          const double sx = minmod_dev(U0[nV + v] - u, u - U0[v - nV]) * ics[0];
          wl[0][v] = u - 0.5 * cs[0] * sx;
          wr[0][v] = u + 0.5 * cs[0] * sx;
          const double sy = minmod_dev(U0[E * nV + v] - u, u - U0[v - E * nV]) * ics[1];
          wl[1][v] = u - 0.5 * cs[1] * sy;
          wr[1][v] = u + 0.5 * cs[1] * sy;
          const double sz = minmod_dev(Up[v] - u, u - Um[v]) * ics[2];
          wl[2][v] = u - 0.5 * cs[2] * sz;
          wr[2][v] = u + 0.5 * cs[2] * sz;
        }
        double Qt[nV] = {0, 0, 0, 0, 0};
#pragma unroll
        for (int d = 0; d < 3; d++) {
          double f[nV];
          dir_flux<3, PDE>(wl[d], d, f);
#pragma unroll
          for (int v = 0; v < nV; v++) Qt[v] += f[v] * ics[d];
          dir_flux<3, PDE>(wr[d], d, f);
#pragma unroll
          for (int v = 0; v < nV; v++) Qt[v] -= f[v] * ics[d];
        }
#pragma unroll
        for (int d = 0; d < 2; d++)
#pragma unroll
          for (int v = 0; v < nV; v++) {
            sW[((d * 2 + 0) * nV + v) * RR + t] = wl[d][v] + 0.5 * dt * Qt[v];
            sW[((d * 2 + 1) * nV + v) * RR + t] = wr[d][v] + 0.5 * dt * Qt[v];
          }
#pragma unroll
        for (int v = 0; v < nV; v++) wl[2][v] = wl[2][v] + 0.5 * dt * Qt[v];
        if (zr > 0 && inX && inY) edge_flux<3, PDE>(wz, wl[2], 2, fz);
#pragma unroll
        for (int v = 0; v < nV; v++) wz[v] = wr[2][v] + 0.5 * dt * Qt[v];
      }
      __syncthreads();
      if (more) {  // plane z-1 is not read any more
        double* to = sU + ((z + 2) % 3) * PLANE;
#pragma unroll
        for (int k = 0; k < KP; k++) {
          const int i = t + k * C::THREADS;
          if (i < PLANE) {
            to[i] = pf[k];
            lp[(z + 2) * PLANE + i] = pf[k];
          }
        }
      }
      const bool inZ = zr >= 1 && zr <= B;
      if (inZ) {
        for (int e = t; e < 2 * NE; e += C::THREADS) {
          const int d = e >= NE, j = e - d * NE;
          // x edges: (y, k) with k fastest; y edges: (k, x) with x fastest
          const int q = d == 0 ? (j / (B + 1) + 1) * R + j % (B + 1) : (j / B) * R + j % B + 1;
          const int o = d == 0 ? q + 1 : q + R;
          double ql[nV], qr[nV], f[nV];
#pragma unroll
          for (int v = 0; v < nV; v++) {
            ql[v] = sW[((d * 2 + 1) * nV + v) * RR + q];
            qr[v] = sW[((d * 2 + 0) * nV + v) * RR + o];
          }
          if (d == 0)
            edge_flux<3, PDE>(ql, qr, 0, f);
          else
            edge_flux<3, PDE>(ql, qr, 1, f);
#pragma unroll
          for (int v = 0; v < nV; v++) sX[(d * nV + v) * NE + j] = f[v];
        }
      }
      __syncthreads();
      if (ring) {
        double* out = l + (size_t)(z * E * E + y * E + x) * nV;
        if (inX && inY) {
          if (zr > 0) {
            double* below = out - (size_t)E * E * nV;
            if (zr == 1) {  // the ghost plane below: its upper edge only
#pragma unroll
              for (int v = 0; v < nV; v++) below[v] -= icsdt[2] * fz[v];
            } else {
#pragma unroll
              for (int v = 0; v < nV; v++) below[v] = up[v] - icsdt[2] * fz[v];
            }
          }
          if (inZ) {
            const int ex = (y - kGW) * (B + 1) + x - kGW, ey = (y - kGW) * B + x - kGW;
#pragma unroll
            for (int v = 0; v < nV; v++) {
              double u = U0[v];
              u += icsdt[0] * sX[v * NE + ex];
              u -= icsdt[0] * sX[v * NE + ex + 1];
              u += icsdt[1] * sX[(nV + v) * NE + ey];
              u -= icsdt[1] * sX[(nV + v) * NE + ey + B];
              up[v] = u + icsdt[2] * fz[v];
            }
          } else if (zr == R - 1) {  // the ghost plane above: its lower edge only
#pragma unroll
            for (int v = 0; v < nV; v++) out[v] = U0[v] + icsdt[2] * fz[v];
          }
        } else if (inZ && (inX || inY)) {  // first ghost layer in x or y: one edge each
          const int d = inY ? 0 : 1, hi = inY ? x > kGW : y > kGW;
          const int e = d == 0 ? (y - kGW) * (B + 1) + (hi ? B : 0) : (hi ? B : 0) * B + x - kGW;
          const double c = hi ? icsdt[d] : -icsdt[d];
#pragma unroll
          for (int v = 0; v < nV; v++) out[v] = U0[v] + c * sX[(d * nV + v) * NE + e];
        }
      }
    }
    __syncthreads();
    if (luh) project_dg_block<3, N>(l, luh + (size_t)cell * L::P * nV, smem);
  }
}

// ---------------------------------------------------------------------------
// Status bookkeeping kernels, one block per cell.

template <int DIM, int N>
struct PostCfg {
  using L = LimShape<DIM, N>;
  static constexpr int TMP = tensor_tmp<DIM, L::b, L::B>() > tensor_tmp<DIM, L::b, L::b>()
                                 ? tensor_tmp<DIM, L::b, L::B>() : tensor_tmp<DIM, L::b, L::b>();
  static constexpr int THREADS = 128;
  static constexpr size_t SMEM = sizeof(double) * (TMP + 2 * THREADS + 10);
  // the post-update kernel of 2D meshes runs one warp per cell, 4 per block
  static constexpr bool kWarp = DIM == 2;
  using Group = typename std::conditional<kWarp, WarpGroup, BlockGroup>::type;
  static constexpr int CELLS = kWarp ? THREADS / 32 : 1;
  // per SM, of the post-update kernel's registers. 3D states none: 128 to 135
  // registers a thread, lines instead of an output per thread (a limiting step of
  // 12^3 N=3 with its other kernels 503 -> 271 us, 9^3 N=5 864 -> 337, 7^3 N=7 2031 -> 539)
  static constexpr int BLOCKS = !kWarp ? 1 : N == 7 ? 5 : 8;
  // per cell: tensor-map scratch, reduction slots (a whole block's), the
  // staged DG solution
  static constexpr int RED = kWarp ? 0 : 2 * THREADS + 10;
  static constexpr int PER = TMP + RED + L::P * L::nV;
  static constexpr size_t POST_SMEM = sizeof(double) * CELLS * PER;
};

// Min/max of the observables (the conserved variables) over the
// Gauss-Legendre nodes, the Gauss-Lobatto nodes and the subcell centres of one
// cell (findCellLocalMinAndMax + compareWithADERDGSolutionAtGaussLobattoNodes +
// compareWithADERDGSolutionAtFVSubcellCenters, Limiter.cpp:210-368). By the whole
// group; a thread below line_threads ends with the part it saw of variable
// tid % 5, for block_minmax_lines or warp_minmax_lines to put together.
template <int DIM, int N, class G = BlockGroup>
__device__ MinMax local_minmax_lines(const double* u, double* tmp) {
  using L = LimShape<DIM, N>;
  constexpr int nV = L::nV;
  MinMax m;  // of this thread's variable
  const int A = line_threads<G>();
  if (G::tid() < A)
    for (int e = G::tid(); e < L::P * nV; e += A) m.fold(u[e], u[e]);
  // the projected values are folded in as they are produced
  auto fold = [&](int, int, int, int, double val) { m.fold(val, val); };
  auto src = [&](int z, int y, int x, int v) { return u[(((DIM == 3 ? z * L::b : 0) + y) * L::b + x) * nV + v]; };
  tensor_map<DIM, L::b, L::b, G>(src, fold, proj_matrix<N, Proj::kToLobatto>(), tmp);
  tensor_map<DIM, L::b, L::B, G>(src, fold, proj_matrix<N, Proj::kToFV>(), tmp);
  return m;
}

// Initial limiter status (updateLimiterStatusAndMinAndMaxAfterSetInitialConditions,
// LimitingADERDGSolver.cpp:1069-1083, determineSolverMinAndMax :1101-1130): the
// local min/max of the initial DG solution into every face block; a cell whose
// values are not physically admissible starts troubled. One block per cell.
template <int DIM, int N, class PDE>
__global__ void __launch_bounds__(128) lim_init_kernel(int ncells, const double* __restrict__ luh, int* __restrict__ s,
                                                       int* __restrict__ s_prev, int* __restrict__ cure,
                                                       int* __restrict__ fs, int* __restrict__ has_lim,
                                                       double* __restrict__ minB, double* __restrict__ maxB,
                                                       LimParams prm) {
  using L = LimShape<DIM, N>;
  using C = PostCfg<DIM, N>;
  constexpr int D2 = 2 * DIM;
  extern __shared__ double smem[];
  const int cell = blockIdx.x;
  if (cell >= ncells) return;
  double mn[5], mx[5];
  block_minmax_lines(local_minmax_lines<DIM, N>(luh + (size_t)cell * L::P * L::nV, smem), mn, mx, smem + C::TMP);
  if (threadIdx.x == 0) {
    double* mnB = minB + (size_t)cell * D2 * 5;
    double* mxB = maxB + (size_t)cell * D2 * 5;
    for (int i = 0; i < D2; i++)
      for (int v = 0; v < 5; v++) {
        mnB[i * 5 + v] = mn[v];
        mxB[i * 5 + v] = mx[v];
      }
    const bool ok = PDE::isPhysicallyAdmissible(mnB, mxB);
    s[cell] = ok ? 0 : prm.T;
    s_prev[cell] = 0;
    cure[cell] = ok ? 0 : prm.cure_steps + 1;
    has_lim[cell] = 0;
    for (int i = 0; i < D2; i++) fs[cell * D2 + i] = 0;
  }
}

// Limiter patches of the cells with s > 0 after the initial status spreading
// start from the FV solver's own initial condition at the subcell centres
// (fv_ic[cell][B^d][nV], LimitingADERDGSolver::setInitialConditions :745-770),
// or, without one, from the projection of the DG solution. One block per cell.
template <int DIM, int N>
__global__ void __launch_bounds__(128) lim_seed_kernel(int ncells, const int* __restrict__ s,
                                                       const double* __restrict__ luh, const double* __restrict__ fv_ic,
                                                       double* __restrict__ lim) {
  using L = LimShape<DIM, N>;
  extern __shared__ double tmp[];
  const int cell = blockIdx.x;
  if (cell >= ncells || s[cell] <= 0) return;
  double* l = lim + (size_t)cell * L::LS;
  if (fv_ic) {
    const double* src = fv_ic + (size_t)cell * L::PB * L::nV;
    for (int i = threadIdx.x; i < L::PB * L::nV; i += blockDim.x) {
      const int v = i % L::nV, q = i / L::nV;
      const int x = q % L::B, y = (q / L::B) % L::B, z = DIM == 3 ? q / (L::B * L::B) : 0;
      l[lim_index<DIM, N>(z, y, x) * L::nV + v] = src[i];
    }
  } else {
    project_fv_block<DIM, N>(luh + (size_t)cell * L::P * L::nV, l, tmp);
  }
}

// After the cell updates of a step (LimitingADERDGSolver::updateSolution
// :843-908 for 0 < s < A, updateLimiterStatusAndMinAndMaxAfterSolutionUpdate
// :910-937, determineLimiterStatusAfterSolutionUpdate :956-994,
// allocateLimiterPatchAfterSolutionUpdate :939-954): per cell
//   - 0 < s < A: FV copy swapped with its previous and refreshed by projection;
//     s == 0: patch released
//   - admissible step (exact arithmetic) -> *dt_min
//   - DMP over GL, Gauss-Lobatto and subcell values, admissibility, the
//     FV-subcell min/max for FV-active cells, the status machine
//   - an irregular change (a cell with s <= A became troubled) sets *irregular.
// run (optional): the kernel does nothing when it holds 0.
// G: one block per cell (BlockGroup) or one warp per cell, 4 cells per block
// (WarpGroup; 2D). A warp is a chain of some ten dependent phases, so its
// register budget is that of eight blocks an SM (81^2 N=5: all but 1.4 waves
// of warps in flight; 48 limiting steps 7.15 ms, with six 7.23, five 7.24);
// five at N = 7 (61^2, 40 steps: 6.93, with eight 6.99).
template <int DIM, int N, class PDE, class G = BlockGroup>
__global__ void __launch_bounds__(128, PostCfg<DIM, N>::BLOCKS) lim_post_update_kernel(
    int ncells, double* __restrict__ luh, int* __restrict__ s, int* __restrict__ s_prev, int* __restrict__ cure,
    int* __restrict__ fs, int* __restrict__ has_lim, double* __restrict__ minB, double* __restrict__ maxB,
    double* __restrict__ lim, double* __restrict__ lim_prev, Geometry geo, LimParams prm,
    double* __restrict__ dt_min, int* __restrict__ irregular, const int* __restrict__ run = nullptr) {
  using L = LimShape<DIM, N>;
  using C = PostCfg<DIM, N>;
  if (run && !*run) return;
  constexpr int nV = L::nV, D2 = 2 * DIM;
  extern __shared__ double smem[];
  double* tmp = smem + G::index() * C::PER;
  double* red = tmp + C::TMP;
  double* su = red + C::RED;  // the cell's DG solution after the update
  __shared__ int s_flags_all[4][4];
  int* s_flags = s_flags_all[G::index()];
  const int cell = blockIdx.x * (blockDim.x / G::size()) + G::index();
  if (cell >= ncells) return;
  const int st = s[cell];  // status before the update
  double* u = luh + (size_t)cell * L::P * nV;
  double* l = lim + (size_t)cell * L::LS;
  double* lp = lim_prev + (size_t)cell * L::LS;
  if (G::tid() == 0) {
    s_prev[cell] = st;
    s_flags[0] = has_lim[cell];
  }
  // one warp per cell: the cell's face min/max blocks, facewise statuses and
  // cure counter are loaded now, one value per lane, so that the status
  // machine at the end waits on no global load
  constexpr bool kWarp = std::is_same<G, WarpGroup>::value;
  double pmn = 0.0, pmx = 0.0;
  int pfs = 0, pcure = 0;
  if constexpr (kWarp) {
    const int j = G::tid();
    if (j < D2 * 5) {
      pmn = minB[(size_t)cell * D2 * 5 + j];
      pmx = maxB[(size_t)cell * D2 * 5 + j];
    }
    if (j < D2) pfs = fs[cell * D2 + j];
    if (j == 0) pcure = cure[cell];
  }
  G::sync();
  if (st > 0 && st < prm.A) {
    if (!s_flags[0])
      for (int i = G::tid(); i < L::LS; i += G::size()) l[i] = lp[i] = 0.0;
    G::sync();
    swap_group<G>(l, lp, L::LS);
    G::sync();
    project_fv_block<DIM, N, G>(u, l, tmp);
    if (G::tid() == 0) has_lim[cell] = 1;
  }
  if (st == 0 && G::tid() == 0) has_lim[cell] = 0;  // ensureNoUnrequiredLimiterPatchIsAllocatedOnComputeCell
  // admissible step of the new solution
  const double invDx0 = __ddiv_rn(1.0, geo.dx[0]), invDx1 = __ddiv_rn(1.0, geo.dx[1]);
  const double invDx2 = DIM == 3 ? __ddiv_rn(1.0, geo.dx[2]) : 0.0;
  // stage the (final) DG solution
  copy_group<G>(su, u, L::P * nV);
  G::sync();
  double dtm = __longlong_as_double(0x7fefffffffffffffll);
  for (int p = G::tid(); p < L::P; p += G::size()) {
    const double* q = su + p * nV;
    double den = 0.0;
    den = __dadd_rn(den, __dmul_rn(Hooks<PDE, DIM>::max_abs_eig_exact(q, 0), invDx0));
    den = __dadd_rn(den, __dmul_rn(Hooks<PDE, DIM>::max_abs_eig_exact(q, 1), invDx1));
    if (DIM == 3) den = __dadd_rn(den, __dmul_rn(Hooks<PDE, DIM>::max_abs_eig_exact(q, 2), invDx2));
    const double d = __ddiv_rn(__dmul_rn(0.9, pnpm(N)), den);
    dtm = (d < dtm) ? d : dtm;
  }
  {  // block min of the step
    double m = dtm;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double x = __shfl_xor_sync(0xffffffffu, m, o);
      m = (x < m) ? x : m;
    }
    if ((threadIdx.x & 31) == 0) atomic_min_pos_double(dt_min, m);
  }
  const MinMax dgm = local_minmax_lines<DIM, N, G>(su, tmp);
  // FV-subcell min/max of FV-active cells (findCellLocalLimiterMinAndMax, :167-205)
  MinMax fvm;  // of this thread's variable (a row holds B nV consecutive values)
  if (st >= prm.A) {
    const int A = line_threads<G>();
    if (G::tid() < A)
#pragma unroll 4
      for (int i = G::tid(); i < L::PB * nV; i += A) {
        const int row = i / (L::B * nV), o = i - row * (L::B * nV);
        const double q = l[lim_index<DIM, N>(row / L::B, row % L::B, 0) * nV + o];
        fvm.fold(q, q);
      }
  }
  if constexpr (kWarp) {
    // the same as the block form below, lane v < 5 taking variable v
    const int lane = G::tid(), v = lane % 5;
    const MinMax dr = warp_minmax_lines(dgm), fr = warp_minmax_lines(fvm);
    const double mnv = __shfl_sync(0xffffffffu, dr.mn, v), mxv = __shfl_sync(0xffffffffu, dr.mx, v);
    const double fmnv = __shfl_sync(0xffffffffu, fr.mn, v), fmxv = __shfl_sync(0xffffffffu, fr.mx, v);
    // discreteMaximumPrincipleAndMinAndMaxSearch (Limiter.cpp:114-165)
    double bmin = __shfl_sync(0xffffffffu, pmn, v), bmax = __shfl_sync(0xffffffffu, pmx, v);
#pragma unroll
    for (int i = 1; i < D2; i++) {
      const double a = __shfl_sync(0xffffffffu, pmn, i * 5 + v), c = __shfl_sync(0xffffffffu, pmx, i * 5 + v);
      bmin = (a < bmin) ? a : bmin;
      bmax = (bmax < c) ? c : bmax;
    }
    double sd = (bmax - bmin) * prm.scale;
    sd = (sd < prm.relax) ? prm.relax : sd;
    const bool okv = !((mnv < (bmin - sd)) || (mxv > (bmax + sd)));
    bool ok = __all_sync(0xffffffffu, lane >= 5 || okv);
    {
      double mn[5], mx[5];
#pragma unroll
      for (int w = 0; w < 5; w++) {
        mn[w] = __shfl_sync(0xffffffffu, mnv, w);
        mx[w] = __shfl_sync(0xffffffffu, mxv, w);
      }
      if (ok) ok = PDE::isPhysicallyAdmissible(mn, mx);  // on the new local min/max
    }
    double* mnB = minB + (size_t)cell * D2 * 5;
    double* mxB = maxB + (size_t)cell * D2 * 5;
    if (st >= prm.A) {
      if (lane < D2 * 5) {
        mnB[lane] = fmnv;
        mxB[lane] = fmxv;
      }
    } else if (lane < 5) {
      mnB[v] = mnv;
      mxB[v] = mxv;
      mnB[v + 5] = bmin;
      mxB[v + 5] = bmax;
    }
    int fm = 0;
#pragma unroll
    for (int i = 0; i < D2; i++) fm = max(fm, __shfl_sync(0xffffffffu, pfs, i));
    if (lane < D2) fs[cell * D2 + lane] = 0;
    if (lane == 0) {
      int ns;
      if (!ok) {
        cure[cell] = prm.cure_steps + 1;
        if (!(st > prm.A)) atomicOr(irregular, 1);
        ns = prm.T;
      } else if (st >= prm.T) {
        ns = prm.T;
        int c = pcure - 1;
        if (c == 0) {
          ns = prm.T - 1;
          c = prm.cure_steps + 1;
        }
        cure[cell] = c;
      } else {
        ns = fm;
      }
      s[cell] = ns;
      const int had = (st == 0) ? 0 : (st < prm.A ? 1 : s_flags[0]);
      s_flags[1] = ns;
      s_flags[2] = (ns > 0 && !had);
      if (s_flags[2]) has_lim[cell] = 1;
    }
  } else {
    double mn[5], mx[5], fmn[5], fmx[5];
    block_minmax_lines(dgm, mn, mx, red);
    if (st >= prm.A) block_minmax_lines(fvm, fmn, fmx, red);
    if (G::tid() == 0) {
      double* mnB = minB + (size_t)cell * D2 * 5;
      double* mxB = maxB + (size_t)cell * D2 * 5;
      // discreteMaximumPrincipleAndMinAndMaxSearch (Limiter.cpp:114-165)
      bool ok = true;
      for (int v = 0; v < 5; v++) {
        double bmin = mnB[v], bmax = mxB[v];
        for (int i = 1; i < D2; i++) bmin = (mnB[i * 5 + v] < bmin) ? mnB[i * 5 + v] : bmin;
        for (int i = 1; i < D2; i++) bmax = (bmax < mxB[i * 5 + v]) ? mxB[i * 5 + v] : bmax;
        double sd = (bmax - bmin) * prm.scale;
        sd = (sd < prm.relax) ? prm.relax : sd;
        if ((mn[v] < (bmin - sd)) || (mx[v] > (bmax + sd))) ok = false;
        mnB[v] = mn[v];
        mxB[v] = mx[v];
        mnB[v + 5] = bmin;
        mxB[v + 5] = bmax;
      }
      if (ok) ok = PDE::isPhysicallyAdmissible(mnB, mxB);  // on the new local min/max
      if (st >= prm.A)
        for (int i = 0; i < D2; i++)
          for (int v = 0; v < 5; v++) {
            mnB[i * 5 + v] = fmn[v];
            mxB[i * 5 + v] = fmx[v];
          }
      int ns;
      if (!ok) {
        cure[cell] = prm.cure_steps + 1;
        if (!(st > prm.A)) atomicOr(irregular, 1);
        ns = prm.T;
      } else if (st >= prm.T) {
        ns = prm.T;
        cure[cell] -= 1;
        if (cure[cell] == 0) {
          ns = prm.T - 1;
          cure[cell] = prm.cure_steps + 1;
        }
      } else {
        ns = 0;
        for (int i = 0; i < D2; i++) ns = max(ns, fs[cell * D2 + i]);
      }
      s[cell] = ns;
      for (int i = 0; i < D2; i++) fs[cell * D2 + i] = 0;
      const int had = (st == 0) ? 0 : (st < prm.A ? 1 : has_lim[cell]);
      s_flags[1] = ns;
      s_flags[2] = (ns > 0 && !had);
      if (s_flags[2]) has_lim[cell] = 1;
    }
  }
  G::sync();
  if (s_flags[2]) {  // newly allocated patch: zeroed; projection for helper cells
    for (int i = G::tid(); i < L::LS; i += G::size()) l[i] = lp[i] = 0.0;
    G::sync();
    if (s_flags[1] < prm.A) project_fv_block<DIM, N, G>(su, l, tmp);
  }
}

// the uniform mesh's cells, x fastest
template <int DIM>
struct CellGrid {
  int n[DIM];
  bool periodic[DIM];
  // the cell across face `face` of cell c, -1: none (a domain boundary)
  __device__ __forceinline__ int across(int c, int face) const {
    int at = c, stride = 1;
    const int d = face >> 1;
#pragma unroll
    for (int e = 0; e < DIM; e++)
      if (e < d) {
        at /= n[e];
        stride *= n[e];
      }
    int nd = n[0];
#pragma unroll
    for (int e = 1; e < DIM; e++) nd = e == d ? n[e] : nd;
    bool per = periodic[0];
#pragma unroll
    for (int e = 1; e < DIM; e++) per = e == d ? periodic[e] : per;
    const int i = at % nd;
    if (face & 1) return i + 1 < nd ? c + stride : per ? c - (nd - 1) * stride : -1;
    return i > 0 ? c - stride : per ? c + (nd - 1) * stride : -1;
  }
};

// the status of cell c after one spreading sweep: a cell below T takes the
// largest merged status of its interior faces
// (updateLimiterStatusDuringLimiterStatusSpreading, :392-405, after the merge
// of every face)
template <int DIM>
__device__ __forceinline__ int spread_once(const int* __restrict__ s, const CellGrid<DIM>& grid, int c, int T) {
  const int sc = s[c];
  if (sc >= T) return T;
  int ns = 0;
#pragma unroll
  for (int f = 0; f < 2 * DIM; f++) {
    const int o = grid.across(c, f);
    if (o >= 0) ns = max(ns, merged_face_status(sc, s[o], T));
  }
  return ns;
}

// SWEEPS (1 or 2) limiter status spreading sweeps from s_in to s_out: the
// merged face statuses of a sweep follow from the statuses on both sides, so
// a cell's status after two sweeps follows from those of its neighbours'
// neighbours, without a launch for the faces or between the two. One warp per
// cell: lanes 0 .. 2 DIM hold the cell and its neighbours; a newly required
// patch is zeroed by the whole warp.
template <int DIM, int N, int SWEEPS>
__global__ void __launch_bounds__(128) lim_spread_kernel(int ncells, const int* __restrict__ s_in,
                                                         int* __restrict__ s_out, int* __restrict__ cure,
                                                         int* __restrict__ has_lim, double* __restrict__ lim,
                                                         double* __restrict__ lim_prev, CellGrid<DIM> grid,
                                                         LimParams prm, const int* __restrict__ gate) {
  using L = LimShape<DIM, N>;
  const int c = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (c >= ncells || (gate && !*gate)) return;
  // lane f + 1: the cell across face f, after the first sweep
  const int mine = lane == 0 ? c : lane <= 2 * DIM ? grid.across(c, lane - 1) : -1;
  int st = -1;
  if (mine >= 0 && (SWEEPS == 2 || lane == 0)) st = spread_once<DIM>(s_in, grid, mine, prm.T);
  const int first = __shfl_sync(0xffffffffu, st, 0);
  int ns = first;
  if constexpr (SWEEPS == 2) {
    if (first < prm.T) {
      ns = lane >= 1 && mine >= 0 ? merged_face_status(first, st, prm.T) : 0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ns = max(ns, __shfl_xor_sync(0xffffffffu, ns, o));
    }
  }
  int alloc = 0;
  if (lane == 0) {
    if (s_in[c] >= prm.T) cure[c] = prm.cure_steps + 1;
    s_out[c] = ns;
    alloc = (first > 0 || ns > 0) && !has_lim[c];
    if (alloc) has_lim[c] = 1;
  }
  if (__shfl_sync(0xffffffffu, alloc, 0)) {
    double* l = lim + (size_t)c * L::LS;
    double* lp = lim_prev + (size_t)c * L::LS;
    for (int i = lane; i < L::LS; i += 32) l[i] = lp[i] = 0.0;
  }
}

// scratch of one cell's projections (either direction)
template <int DIM, int N>
constexpr int proj_tmp() {
  using L = LimShape<DIM, N>;
  return tensor_tmp<DIM, L::b, L::B>() > tensor_tmp<DIM, L::B, L::b>() ? tensor_tmp<DIM, L::b, L::B>()
                                                                         : tensor_tmp<DIM, L::B, L::b>();
}

// reinitialiseSolversLocally (:1329-1360). G: one block per cell, or one
// warp per cell with blockDim.x / 32 cells per block (2D).
template <int DIM, int N, class G = BlockGroup>
__global__ void __launch_bounds__(128) lim_reinit_kernel(int ncells, double* __restrict__ luh,
                                                         double* __restrict__ luh_prev, const int* __restrict__ s,
                                                         const int* __restrict__ s_prev, int* __restrict__ cure,
                                                         int* __restrict__ has_lim, double* __restrict__ lim,
                                                         double* __restrict__ lim_prev, LimParams prm,
                                                         const int* __restrict__ gate) {
  using L = LimShape<DIM, N>;
  extern __shared__ double smem[];
  double* tmp = smem + G::index() * proj_tmp<DIM, N>();
  const int c = blockIdx.x * (blockDim.x / G::size()) + G::index();
  if (c >= ncells || !*gate) return;
  const int st = s[c];
  if (st <= 0) {
    if (G::tid() == 0) has_lim[c] = 0;
    return;
  }
  double* u = luh + (size_t)c * L::P * L::nV;
  double* up = luh_prev + (size_t)c * L::P * L::nV;
  double* l = lim + (size_t)c * L::LS;
  double* lp = lim_prev + (size_t)c * L::LS;
  if (s_prev[c] >= prm.A) {
    swap_group<G>(l, lp, L::LS);
    G::sync();
    project_dg_block<DIM, N, G>(l, u, tmp);
  } else {
    swap_group<G>(u, up, L::P * L::nV);
    G::sync();
    project_fv_block<DIM, N, G>(u, l, tmp);
  }
  if (G::tid() == 0 && st >= prm.T) cure[c] = prm.cure_steps + 1;
}

// recomputeSolutionLocally (:1396-1436) for cells with 0 < s < A, then the
// admissible step of every cell (the FV-active cells were re-updated by
// lim_muscl_kernel just before). G as for lim_reinit_kernel.
template <int DIM, int N, class PDE, class G = BlockGroup>
__global__ void __launch_bounds__(128) lim_recompute_kernel(int ncells, double* __restrict__ luh,
                                                            double* __restrict__ luh_prev, const int* __restrict__ s,
                                                            const int* __restrict__ s_prev, double* __restrict__ lim,
                                                            double* __restrict__ lim_prev, Geometry geo, LimParams prm,
                                                            double* __restrict__ dt_min, const int* __restrict__ gate) {
  using L = LimShape<DIM, N>;
  extern __shared__ double smem[];
  double* tmp = smem + G::index() * proj_tmp<DIM, N>();
  const int c = blockIdx.x * (blockDim.x / G::size()) + G::index();
  if (c >= ncells || !*gate) return;
  const int st = s[c];
  double* u = luh + (size_t)c * L::P * L::nV;
  if (st > 0 && st < prm.A) {
    double* l = lim + (size_t)c * L::LS;
    if (s_prev[c] < prm.A) {
      double* up = luh_prev + (size_t)c * L::P * L::nV;
      swap_group<G>(u, up, L::P * L::nV);
      G::sync();
      project_fv_block<DIM, N, G>(u, l, tmp);
    } else {
      double* lp = lim_prev + (size_t)c * L::LS;
      swap_group<G>(l, lp, L::LS);
      G::sync();
      project_dg_block<DIM, N, G>(l, u, tmp);
    }
  }
  G::sync();
  const double invDx0 = __ddiv_rn(1.0, geo.dx[0]), invDx1 = __ddiv_rn(1.0, geo.dx[1]);
  const double invDx2 = DIM == 3 ? __ddiv_rn(1.0, geo.dx[2]) : 0.0;
  double dtm = __longlong_as_double(0x7fefffffffffffffll);
  for (int p = G::tid(); p < L::P; p += G::size()) {
    const double* q = u + p * L::nV;
    double den = 0.0;
    den = __dadd_rn(den, __dmul_rn(Hooks<PDE, DIM>::max_abs_eig_exact(q, 0), invDx0));
    den = __dadd_rn(den, __dmul_rn(Hooks<PDE, DIM>::max_abs_eig_exact(q, 1), invDx1));
    if (DIM == 3) den = __dadd_rn(den, __dmul_rn(Hooks<PDE, DIM>::max_abs_eig_exact(q, 2), invDx2));
    const double d = __ddiv_rn(__dmul_rn(0.9, pnpm(N)), den);
    dtm = (d < dtm) ? d : dtm;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double x = __shfl_xor_sync(0xffffffffu, dtm, o);
    dtm = (x < dtm) ? x : dtm;
  }
  // warps without a node hold DBL_MAX: no atomic
  if ((threadIdx.x & 31) == 0 && (threadIdx.x & ~31) % G::size() < L::P) atomic_min_pos_double(dt_min, dtm);
}

// Batched projections for the kernel-level entry points: one block per listed
// cell (list NULL: cells 0..n-1). TO_FV: luh -> interior subcells of lim, else
// interior subcells of lim -> luh. One kernel per direction, each with its own
// register budget (blocks per SM, 0: none stated): with both in one kernel the
// compiler held matrix entries of the way to the DG basis in registers (124 at
// order 7; 20,000 patches 2D N=7 191 us, with eight blocks 70, none stated 89;
// 3,000 patches 3D N=7 606, with one stated 400; N=5 66, 58, none stated 72). To
// the subcells any stated number costs (3,000 cells 3D N=7 212 us, with one 257,
// four 232).
template <int DIM, bool TO_FV>
constexpr int project_blocks() { return TO_FV ? 0 : DIM == 2 ? 8 : 1; }
template <int DIM, int N, bool TO_FV>
__global__ void __launch_bounds__(128, project_blocks<DIM, TO_FV>())
    lim_project_kernel(const int* __restrict__ list, int n, double* __restrict__ luh, double* __restrict__ lim) {
  using L = LimShape<DIM, N>;
  extern __shared__ double tmp[];
  if ((int)blockIdx.x >= n) return;
  const int c = list ? list[blockIdx.x] : (int)blockIdx.x;
  double* u = luh + (size_t)c * L::P * L::nV;
  double* l = lim + (size_t)c * L::LS;
  if constexpr (TO_FV)
    project_fv_block<DIM, N>(u, l, tmp);
  else
    project_dg_block<DIM, N>(l, u, tmp);
}

// Compacts the cells whose status satisfies lo1 <= s < hi1 into list1/count1
// and those with lo2 <= s < hi2 into list2/count2 (order is irrelevant: every
// cell is computed independently).
__global__ void lim_select2_kernel(int ncells, const int* __restrict__ s, int lo1, int hi1, int* __restrict__ list1,
                                   int* __restrict__ count1, int lo2, int hi2, int* __restrict__ list2,
                                   int* __restrict__ count2, const int* __restrict__ gate) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (gate && !*gate) return;
  if (c >= ncells) return;
  const int sc = s[c];
  if (sc >= lo1 && sc < hi1) list1[atomicAdd(count1, 1)] = c;
  if (sc >= lo2 && sc < hi2) list2[atomicAdd(count2, 1)] = c;
}

}  // namespace exa
