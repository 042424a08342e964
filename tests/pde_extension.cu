// PDEs of other shapes than the library's own, on the library's kernels: what
// a user's PDE may look like (built by test_pde_extension.py).
#include "aderdg.cuh"
#include "amr.cuh"
#include "linear.cuh"

using namespace exa;

// linear acoustics: pressure and velocity, no parameters (K = 2, rho = 0.5, c = 2)
struct AcousticPDE {
  static constexpr int nVar = 4, nPar = 0;
  static constexpr bool kLinear = true, kSource = false, kNCP = false, kPointSource = false;
  __device__ static void ncp_dir(const double*, int d, const double* G, double* B) {
    for (int v = 0; v < nVar; v++) B[v] = 0.0;
    B[0] = 2.0 * G[1 + d];
    B[1 + d] = 2.0 * G[0];
  }
  __host__ __device__ static constexpr bool ncp_uses(int d, int v) { return v == 0 || v == 1 + d; }
  __device__ static void eigenvalues(const double*, int, double* l) {
    l[0] = -2.0;
    l[1] = l[2] = 0.0;
    l[3] = 2.0;
  }
};

// elastic waves that name more gradient components than they need, and not as
// many in every direction
struct UnevenElasticPDE : ElasticPDE {
  __host__ __device__ static constexpr bool ncp_uses(int d, int v) { return d == 0 || ElasticPDE::ncp_uses(d, v); }
};

// more than 16 values per node; only the Riemann solver is used
struct WidePDE {
  static constexpr int nVar = 18, nPar = 1;
  static constexpr bool kLinear = false, kSource = false, kNCP = false, kPointSource = false;
  __device__ static void eigenvalues(const double* Q, int d, double* l) {
    for (int v = 0; v < nVar; v++) l[v] = (v - 9) * 0.1 * Q[v] * Q[18] * (1 + d);
  }
};

template <int N>
static void order_tables(OrderTables& t) {
  constexpr int b = N + 1;
  for (int i = 0; i < b; i++) {
    t.w[i] = exa_tab_weights[exa_tab_weights_off[N] + i];
    t.x[i] = exa_tab_nodes[exa_tab_nodes_off[N] + i];
    t.FL[i] = exa_tab_FLCoeff[exa_tab_FLCoeff_off[N] + i];
    t.FR[i] = exa_tab_FRCoeff[exa_tab_FRCoeff_off[N] + i];
  }
  for (int i = 0; i < b * b; i++) {
    t.Kxi[i] = exa_tab_Kxi[exa_tab_Kxi_off[N] + i];
    t.iK1[i] = exa_tab_iK1[exa_tab_iK1_off[N] + i];
    t.dudx[i] = exa_tab_dudx[exa_tab_dudx_off[N] + i];
  }
}

template <int DIM, int N, class PDE>
static int predictor(const double* luh, double* qb, double* fb, double* du, const double* dt, const double* dx, int n) {
  using C = CKCfg<DIM, N, PDE>;
  Geometry g{};
  for (int d = 0; d < DIM; d++) g.dx[d] = dx[d];
  auto k = ck_predictor_kernel<DIM, N, PDE>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
  if (e != cudaSuccess) return (int)e;
  k<<<(n + C::CPB - 1) / C::CPB, C::THREADS, C::SMEM>>>(luh, qb, fb, du, dt, g, n, nullptr, nullptr, nullptr, nullptr);
  return (int)cudaGetLastError();
}

extern "C" {
int ext_tables() {
  static OrderTables h[kMaxOrder + 1];
  static LineTablesAll lt;
  order_tables<3>(h[3]);
  order_tables<5>(h[5]);
  fill_line_tables(h[3], lt.n3);
  fill_line_tables(h[5], lt.n5);
  cudaError_t e = cudaMemcpyToSymbol(c_tab, h, sizeof(h));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_line, &lt, sizeof(lt));
  return (int)e;
}
int ext_predictor(int which, const double* luh, double* qb, double* fb, double* du, const double* dt, const double* dx,
                  int n) {
  switch (which) {
    case 0: return predictor<2, 3, AcousticPDE>(luh, qb, fb, du, dt, dx, n);
    case 1: return predictor<3, 3, AcousticPDE>(luh, qb, fb, du, dt, dx, n);
    case 2: return predictor<2, 5, UnevenElasticPDE>(luh, qb, fb, du, dt, dx, n);
    case 3: return predictor<3, 3, UnevenElasticPDE>(luh, qb, fb, du, dt, dx, n);
    case 4: return predictor<3, 5, UnevenElasticPDE>(luh, qb, fb, du, dt, dx, n);
    case 5: return predictor<3, 5, AcousticPDE>(luh, qb, fb, du, dt, dx, n);
  }
  return -1;
}
int ext_riemann_linear(const double* qb, double* fb, const int* l, const int* r, const int* d, int n) {
  riemann_linear_kernel<3, 3, AcousticPDE><<<(n + 3) / 4, 128>>>(qb, fb, l, r, d, n);
  return (int)cudaGetLastError();
}
int ext_riemann_wide(const double* qb, double* fb, const int* l, const int* r, const int* d, int n) {
  riemann_kernel<3, 3, WidePDE><<<(n + 3) / 4, 128>>>(qb, fb, l, r, d, n);
  return (int)cudaGetLastError();
}
}
