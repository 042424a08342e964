// AMR transfer operators and the plotters' vertex projection on the GPU.
//
//   amr_volume_kernel  volumeUnknownsProlongation / volumeUnknownsRestriction
//                      (kernels/aderdg/generic/c/{2d,3d}/amrRoutines.cpph)
//   amr_face_kernel    faceUnknownsProlongation / faceUnknownsRestriction
//   plot_vertex_kernel the (N+1)^d equidistant vertex values that
//                      ADERDG2CartesianVTK::plotVertexData writes
//                      (exahype/plotters/VTK/ADERDG2CartesianVTK.cpp)
//
// One block per transfer (a fine cell or face and its coarse ancestor,
// levelDelta levels apart, the subcell index holding one base-3 digit per
// level). Per level the tensor-product operator is applied one axis at a
// time in shared memory (the reference sums the full product per output; the
// sums differ in rounding order only): prolongation with
// P[third][n][m] = phi_n((third + x_m)/3) from the coarse level down,
// restriction with w_n P[third][m][n] / (3 w_m) per axis from the fine level
// up. Restrictions add into the coarse data with atomicAdd, so any number of
// descendants can be restricted into one ancestor in one launch (the sum order
// is not fixed).
//
// Bound: HBM (the fine data once; the coarse cells stay in L2), reached to a
// part only: a block's index loads, source loads, passes and stores are one
// chain, so the rate follows from how many small blocks an SM holds. Reading
// the first axis from and writing the last one to global memory halves the
// shared-memory traffic of the copy-in, three ping-pong passes, copy-out form,
// takes one buffer instead of two and two barriers instead of five:
// prolongation, restriction and vertex projection of 9^3 <-> 27^3 cells at
// N = 5 together 266 -> 197 us.
#pragma once
#include "aderdg.cuh"

namespace exa {

// Operator tables in constant memory, packed over the orders that have kernels
// (3, 4, 5 and 7; the offset of order N is the sum over the lower ones of
// (N'+1)^2, times 3 for the thirds):
// fineGridProjector1d [third][n][m], the restriction factors
// w_n P[third][m][n] / (3 w_m) as [third][m][n], equidistantGridProjector1d
// [n][i]. A block reads one matrix with block-uniform addresses, so the
// coefficients come from the constant cache by broadcast.
constexpr bool amr_has(int N) { return N == 3 || N == 4 || N == 5 || N == 7; }
// (an order added to the solvers is added here, to LineTablesAll and
// ProjTablesAll, and to upload_tables)
constexpr int amr_off(int N) { return N <= 3 ? 0 : amr_off(N - 1) + (amr_has(N - 1) ? N * N : 0); }
constexpr int kAmrSq = amr_off(8);  // sum of (N+1)^2 over the orders
__constant__ double c_amr_fine[3 * kAmrSq];
__constant__ double c_amr_restr[3 * kAmrSq];
__constant__ double c_amr_equi[kAmrSq];

// A block works on one tensor of NAX axes with b nodes each and NV values per
// node: one thread per line of the axis in turn, in ROUNDS rounds where that is
// more than 256 threads (order 7: 320). In a loop over rounds the compiler holds
// matrix entries of the transfers in registers across them and spills. So the 320
// lines of 3D order 7 take one round (96 registers and up to 884 bytes before, now
// 50 and none; 5,832 transfers: prolongation 77 -> 54 us, restriction 76 -> 56,
// vertex projection 71 -> 68), and the two rounds of the elastic state at order 5
// (432 lines) are unrolled, but for sums into global memory and in the vertex
// projection (20,000 cells 128 us in a loop, 160 unrolled). The lines of an axis
// are disjoint, so every pass works in place in one shared buffer; the first pass
// reads its lines from global memory and the last one writes its results there.
// Consecutive threads take consecutive values of the x rows, so the last
// axis (of two or three) is written coalesced; the first (x) pass reads each row
// whole, through L1. In the buffer the x rows (b NV values) have a pitch of
// NV modulo 16, which makes the x pass, whose threads stand NV values apart
// per row, free of bank conflicts too (half-warps, 64-bit accesses).
template <int b, int NAX, int NV>
struct TensorCfg {
  static_assert(amr_has(b - 1), "no transfer tables of this order");
  static constexpr int LINES = NV * ipow(b, NAX - 1), SIZE = LINES * b;
  static constexpr int ROUNDS = b >= 8 ? (LINES + 319) / 320 : (LINES + 255) / 256;
  static constexpr int THREADS = ((LINES + ROUNDS - 1) / ROUNDS + 31) / 32 * 32;
  static constexpr int ROW = b * NV, ROWS = ipow(b, NAX - 1);
  static constexpr int PITCH = ROW + ((NV - ROW) % 16 + 16) % 16;
  static constexpr int BUF = ROWS * PITCH;
  // blocks per SM the register budget leaves room for
  static constexpr int BLOCKS = b >= 8 ? 768 / THREADS : 1536 / THREADS < 32 ? 1536 / THREADS : 32;
  // first element and element stride of line `it` of axis AX, rows `pitch` apart
  template <int AX>
  static __device__ __forceinline__ int first(int it, int pitch) {
    if (AX == 0) return it / NV * pitch + it % NV;
    return it / ROW * (AX == 1 ? b * pitch : pitch) + it % ROW;
  }
  template <int AX>
  static constexpr __device__ int stride(int pitch) { return AX == 0 ? NV : AX == 1 ? pitch : b * pitch; }
};

// where a pass takes its lines from and where it puts them
enum class Place { kBuffer, kGlobal, kGlobalAdd };

// out[.., m, ..] = sum_n M[m][n] in[.., n, ..] along axis AX, M given as a
// constant-memory pointer and row / column strides (compile-time indices: the
// coefficients are constant-bank operands). `tid` of `THREADS` threads.
template <class C, int b, int AX, int RS, int CS, Place FROM, Place TO, bool UNROLL = false>
__device__ __forceinline__ void apply_axis(const double* src, double* dst, double* buf, const double* M, int tid) {
  constexpr int ROW = C::ROW;
#pragma unroll(UNROLL && TO != Place::kGlobalAdd ? C::ROUNDS : 1)
  for (int r = 0; r < C::ROUNDS; r++) {
    const int it = tid + r * C::THREADS;
    if (it >= C::LINES) break;
    const double* in = FROM == Place::kBuffer ? buf + C::template first<AX>(it, C::PITCH)
                                              : src + C::template first<AX>(it, ROW);
    double* out = TO == Place::kBuffer ? buf + C::template first<AX>(it, C::PITCH)
                                       : dst + C::template first<AX>(it, ROW);
    constexpr int is = C::template stride<AX>(FROM == Place::kBuffer ? C::PITCH : ROW);
    constexpr int os = C::template stride<AX>(TO == Place::kBuffer ? C::PITCH : ROW);
    double x[b];
#pragma unroll
    for (int n = 0; n < b; n++) x[n] = FROM == Place::kBuffer ? in[n * is] : __ldg(in + n * is);
#pragma unroll
    for (int m = 0; m < b; m++) {
      double s = 0.0;
#pragma unroll
      for (int n = 0; n < b; n++) s = fma(M[m * RS + n * CS], x[n], s);
      if (TO == Place::kGlobalAdd)
        atomicAdd(out + m * os, s);
      else
        out[m * os] = s;
    }
  }
}

// one axis of one level: the digit picks the third; each case
// has a compile-time table address, so that the coefficients are constant-bank
// operands (prolongation P[n][m], restriction R[m][n])
template <class C, int N, int AX, bool R, Place FROM, Place TO>
__device__ __forceinline__ void transfer_axis(const double* src, double* dst, double* buf, int digit, int tid) {
  constexpr int b = N + 1, base = 3 * amr_off(N), RS = R ? b : 1, CS = R ? 1 : b;
  const double* tab = R ? c_amr_restr : c_amr_fine;
  if (digit == 0) {
    apply_axis<C, b, AX, RS, CS, FROM, TO, true>(src, dst, buf, tab + base, tid);
  } else if (digit == 1) {
    apply_axis<C, b, AX, RS, CS, FROM, TO, true>(src, dst, buf, tab + base + b * b, tid);
  } else {
    apply_axis<C, b, AX, RS, CS, FROM, TO, true>(src, dst, buf, tab + base + 2 * b * b, tid);
  }
}

// barrier of the threads that share one buffer: the block, or a part of it
// (whole warps) under a hardware barrier of its own
template <int ID, int THREADS>
__device__ __forceinline__ void part_sync() {
  if constexpr (ID == 0)
    __syncthreads();
  else
    asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(THREADS) : "memory");
}

// the axes of one level in turn
template <int N, int NAX, int NV, bool R, Place FROM, Place TO, int ID>
__device__ __forceinline__ void transfer_level(const double* src, double* dst, double* buf, const int* digit, int tid) {
  using C = TensorCfg<N + 1, NAX, NV>;
  transfer_axis<C, N, 0, R, FROM, NAX == 1 ? TO : Place::kBuffer>(src, dst, buf, digit[0], tid);
  if constexpr (NAX > 1) {
    part_sync<ID, C::THREADS>();
    transfer_axis<C, N, 1, R, Place::kBuffer, NAX == 2 ? TO : Place::kBuffer>(src, dst, buf, digit[1], tid);
  }
  if constexpr (NAX > 2) {
    part_sync<ID, C::THREADS>();
    transfer_axis<C, N, 2, R, Place::kBuffer, TO>(src, dst, buf, digit[2], tid);
  }
}

// The same as a function of its own, for the loop over several levels: inlined
// there, the compiler loads the matrices of all thirds into registers before
// the loop (spills of up to 2 KB); with one rolled form for the three thirds
// every coefficient is a load of its own (19,683 transfers of 3D N=5 over two
// levels 203 us, so 101). buf: shared-memory address.
template <int N, int NAX, int NV, bool R, Place FROM, Place TO, int ID>
__device__ __noinline__ void transfer_level_call(const double* src, double* dst, uint32_t buf, int d0, int d1, int d2,
                                                 int tid) {
  const int digit[3] = {d0, d1, d2};
  transfer_level<N, NAX, NV, R, FROM, TO, ID>(src, dst, (double*)__cvta_shared_to_generic(buf), digit, tid);
}

// levelDelta in 1..kMaxLevelDelta and every index digit-string in
// [0, 3^levelDelta): transfers that break this are skipped (no table read
// outside the three thirds)
constexpr int kMaxLevelDelta = 12;
__device__ __forceinline__ bool valid_index(int ld, const int* index, int nax) {
  if (ld < 1 || ld > kMaxLevelDelta) return false;
  int lim = 1;
  for (int l = 0; l < ld; l++) lim *= 3;
  for (int k = 0; k < nax; k++)
    if (index[k] < 0 || index[k] >= lim) return false;
  return true;
}

// one transfer of NAX-dimensional nodal data (NV values per node) between
// levels: R false prolongates src (coarse) into dst (fine), R true restricts
// src (fine) and adds it to dst (coarse)
template <int N, int NAX, int NV, bool R, int ID = 0>
__device__ __forceinline__ void amr_transfer(const double* __restrict__ src, double* __restrict__ dst, int levelDelta,
                                             const int* index, double* buf, int tid) {
  constexpr Place TO = R ? Place::kGlobalAdd : Place::kGlobal;
  if (levelDelta == 1) {  // (block-uniform) the digits are the index
    transfer_level<N, NAX, NV, R, Place::kGlobal, TO, ID>(src, dst, buf, index, tid);
    return;
  }
  const uint32_t sbuf = (uint32_t)__cvta_generic_to_shared(buf);
  int rest[3] = {index[0], index[1], index[2]};
  int sig = 1;
  for (int l = 1; l < levelDelta; l++) sig *= 3;
#pragma unroll 1
  for (int l = 0; l < levelDelta; l++) {
    int digit[3] = {0, 0, 0};
#pragma unroll
    for (int k = 0; k < NAX; k++) {
      if (!R) {  // most significant digit first
        digit[k] = rest[k] / sig;
        rest[k] = rest[k] % sig;
      } else {  // least significant digit first
        digit[k] = rest[k] % 3;
        rest[k] = rest[k] / 3;
      }
    }
    sig = sig > 1 ? sig / 3 : 1;
    if (l > 0) part_sync<ID, TensorCfg<N + 1, NAX, NV>::THREADS>();
    const int d0 = digit[0], d1 = digit[1], d2 = digit[2];
    if (l == 0)
      transfer_level_call<N, NAX, NV, R, Place::kGlobal, Place::kBuffer, ID>(src, dst, sbuf, d0, d1, d2, tid);
    else if (l + 1 < levelDelta)
      transfer_level_call<N, NAX, NV, R, Place::kBuffer, Place::kBuffer, ID>(src, dst, sbuf, d0, d1, d2, tid);
    else
      transfer_level_call<N, NAX, NV, R, Place::kBuffer, TO, ID>(src, dst, sbuf, d0, d1, d2, tid);
  }
}

// R false: prolongation, true: restriction. item k: fine cell fine[k], coarse cell
// coarse[k], levelDelta[k], subcell index idx[3k .. 3k+2]
template <int DIM, int N, int ND, bool R>
__global__ void __launch_bounds__(TensorCfg<N + 1, DIM, ND>::THREADS, TensorCfg<N + 1, DIM, ND>::BLOCKS)
    amr_volume_kernel(double* __restrict__ luh_a, const double* __restrict__ luh_b, int n,
                      const int* __restrict__ fine, const int* __restrict__ coarse,
                      const int* __restrict__ level_delta, const int* __restrict__ idx) {
  using C = TensorCfg<N + 1, DIM, ND>;
  __shared__ double buf[C::BUF];
  const int k = blockIdx.x;
  if (k >= n) return;
  const int ld = level_delta[k];
  const int index[3] = {idx[3 * k], idx[3 * k + 1], DIM == 3 ? idx[3 * k + 2] : 0};
  const size_t f = (size_t)fine[k] * C::SIZE, c = (size_t)coarse[k] * C::SIZE;
  if (!valid_index(ld, index, DIM)) return;
  // luh_a: fine (written) and luh_b: coarse, or luh_a: coarse (added to) and luh_b: fine
  amr_transfer<N, DIM, ND, R>(luh_b + (R ? f : c), luh_a + (R ? c : f), ld, index, buf, threadIdx.x);
}

// faces: item k moves face slot fine[k] <-> coarse[k] (slot = cell * 2 DIM +
// face) of the state array (ND per node) and the flux array (NV per node),
// the first warps of the block working on the state, the others on the flux
template <int DIM, int N, int ND, int NV>
struct FaceCfg {
  using Q = TensorCfg<N + 1, DIM - 1, ND>;
  using F = TensorCfg<N + 1, DIM - 1, NV>;
  static constexpr int THREADS = Q::THREADS + F::THREADS;
};
template <int DIM, int N, int ND, int NV, bool R>
__global__ void __launch_bounds__(FaceCfg<DIM, N, ND, NV>::THREADS)
    amr_face_kernel(double* __restrict__ q_a, double* __restrict__ f_a, const double* __restrict__ q_b,
                    const double* __restrict__ f_b, int n, const int* __restrict__ fine,
                    const int* __restrict__ coarse, const int* __restrict__ level_delta,
                    const int* __restrict__ idx) {
  using C = FaceCfg<DIM, N, ND, NV>;
  __shared__ double bufQ[C::Q::BUF], bufF[C::F::BUF];
  const int k = blockIdx.x;
  if (k >= n) return;
  const int ld = level_delta[k];
  const int index[3] = {idx[2 * k], DIM == 3 ? idx[2 * k + 1] : 0, 0};
  const size_t fs = fine[k], cs = coarse[k];
  if (!valid_index(ld, index, DIM - 1)) return;
  const size_t from = R ? fs : cs, to = R ? cs : fs;
  const int tq = threadIdx.x, tf = tq - C::Q::THREADS;
  if (tf < 0)
    amr_transfer<N, DIM - 1, ND, R, 1>(q_b + from * C::Q::SIZE, q_a + to * C::Q::SIZE, ld, index, bufQ, tq);
  else
    amr_transfer<N, DIM - 1, NV, R, 2>(f_b + from * C::F::SIZE, f_a + to * C::F::SIZE, ld, index, bufF, tf);
}

// the solution of every cell at its (N+1)^d equidistant vertices (x fastest),
// one block per cell
template <int DIM, int N, int ND>
__global__ void __launch_bounds__(TensorCfg<N + 1, DIM, ND>::THREADS, TensorCfg<N + 1, DIM, ND>::BLOCKS)
    plot_vertex_kernel(const double* __restrict__ luh, double* __restrict__ out, int ncells) {
  constexpr int b = N + 1;
  using C = TensorCfg<b, DIM, ND>;
  __shared__ double buf[C::BUF];
  const int c = blockIdx.x;
  if (c >= ncells) return;
  const double* src = luh + (size_t)c * C::SIZE;
  double* dst = out + (size_t)c * C::SIZE;
  const double* E = c_amr_equi + amr_off(N);  // E[n][i]: out[i] = sum_n E[n][i] in[n]
  apply_axis<C, b, 0, 1, b, Place::kGlobal, Place::kBuffer>(src, dst, buf, E, threadIdx.x);
  __syncthreads();
  if constexpr (DIM == 2) {
    apply_axis<C, b, 1, 1, b, Place::kBuffer, Place::kGlobal>(src, dst, buf, E, threadIdx.x);
  } else {
    apply_axis<C, b, 1, 1, b, Place::kBuffer, Place::kBuffer>(src, dst, buf, E, threadIdx.x);
    __syncthreads();
    apply_axis<C, b, 2, 1, b, Place::kBuffer, Place::kGlobal>(src, dst, buf, E, threadIdx.x);
  }
}

}  // namespace exa
