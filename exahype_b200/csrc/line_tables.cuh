// 1-D operators in the form the line kernels apply them, and the contraction
// of one line with one of them.
//
// For the symmetric Gauss-Legendre nodes the derivative matrix is
// centro-antisymmetric: M[b-1-n][b-1-l] = -M[n][l]. For even b a contraction
// out_l = sum_n f_n M[n][l] therefore splits into the even and odd parts of
// the line: with h = b/2, fp_n = f_n + f_(b-1-n), fm_n = f_n - f_(b-1-n)
// (n < h), A_l = sum_n fp_n P[n][l], B_l = sum_n fm_n Q[n][l] (l < h):
// out_l = B_l + A_l, out_(b-1-l) = B_l - A_l, where
// P[n][l] = (M[n][l] + M[b-1-n][l]) / 2 and Q the difference / 2: 30 instead
// of 36 operations at b = 6. For odd b P holds the whole matrix.
#pragma once
#include "common.cuh"

namespace exa {

// aligned to a line of the constant cache: what one order's kernel reads lies
// together (unaligned or spread over the constant bank the same operands cost
// the predictor up to a fifth of its time)
template <int N>
struct alignas(256) LineTables {
  static constexpr int b = N + 1, h = b / 2, M = b % 2 == 0 ? h * h : b * b;
  double KP[M], KQ[M];  // M[n][l] = Kxi[n][l] / w[l]: Picard contraction
  double VP[M], VQ[M];  // M[m][k] = Kxi[k][m] / w[k]: volume integral
  double niK1w[b * b];  // [t][l]: -iK1[l][t] w[t]
  // sum_t iK1[l][t] FL[t] and -sum_t iK1[l][t] w[t]: the first Picard sweep
  double alpha[b], beta[b];
  double w[b], FL[b], FR[b];
  double DP[M], DQ[M];  // M[n][l] = dudx[l][n]: derivative at node l
};
// The orders the line kernels are instantiated for, in constant memory.
struct LineTablesAll {
  LineTables<3> n3;
  LineTables<4> n4;
  LineTables<5> n5;
  LineTables<7> n7;
};
__constant__ LineTablesAll c_line;
template <int N>
__device__ __forceinline__ const LineTables<N>& line_tab() {
  static_assert(N == 3 || N == 4 || N == 5 || N == 7, "no line tables of this order");
  if constexpr (N == 3) return c_line.n3;
  else if constexpr (N == 4) return c_line.n4;
  else if constexpr (N == 5) return c_line.n5;
  else return c_line.n7;
}

// host side: fills one order's tables from the order's operators
template <int N>
void fill_line_tables(const OrderTables& T, LineTables<N>& L) {
  constexpr int b = N + 1, h = b / 2;
  auto split = [&](auto m, double* p, double* q) {
    if (b % 2 == 0) {
      for (int n = 0; n < h; n++)
        for (int l = 0; l < h; l++) {
          p[n * h + l] = 0.5 * (m(n, l) + m(b - 1 - n, l));
          q[n * h + l] = 0.5 * (m(n, l) - m(b - 1 - n, l));
        }
    } else {
      for (int n = 0; n < b; n++)
        for (int l = 0; l < b; l++) p[n * b + l] = q[n * b + l] = m(n, l);
    }
  };
  split([&](int n, int l) { return T.Kxi[n * b + l] / T.w[l]; }, L.KP, L.KQ);
  split([&](int m, int k) { return T.Kxi[k * b + m] / T.w[k]; }, L.VP, L.VQ);
  split([&](int n, int l) { return T.dudx[l * b + n]; }, L.DP, L.DQ);
  for (int l = 0; l < b; l++) {
    L.w[l] = T.w[l];
    L.FL[l] = T.FL[l];
    L.FR[l] = T.FR[l];
    L.alpha[l] = L.beta[l] = 0.0;
    for (int t = 0; t < b; t++) {
      L.niK1w[t * b + l] = -T.iK1[l * b + t] * T.w[t];
      L.alpha[l] += T.iK1[l * b + t] * T.FL[t];
      L.beta[l] -= T.iK1[l * b + t] * T.w[t];
    }
  }
}

// out(l, sum_n f_n M[n][l]) for every l, M given by its P and Q
template <int b, class Out>
__device__ __forceinline__ void line_contract(const double (&f)[b], const double* MP, const double* MQ, Out out) {
  if constexpr (b % 2 == 0) {
    constexpr int h = b / 2;
    double fp[h], fm[h];
#pragma unroll
    for (int n = 0; n < h; n++) {
      fp[n] = f[n] + f[b - 1 - n];
      fm[n] = f[n] - f[b - 1 - n];
    }
#pragma unroll
    for (int l = 0; l < h; l++) {
      double A = fp[0] * MP[l], B = fm[0] * MQ[l];
#pragma unroll
      for (int n = 1; n < h; n++) {
        A = fma(fp[n], MP[n * h + l], A);
        B = fma(fm[n], MQ[n * h + l], B);
      }
      out(l, B + A);
      out(b - 1 - l, B - A);
    }
  } else {
#pragma unroll
    for (int l = 0; l < b; l++) {
      double s = f[0] * MP[l];
#pragma unroll
      for (int n = 1; n < b; n++) s = fma(f[n], MP[n * b + l], s);
      out(l, s);
    }
  }
}

}  // namespace exa
