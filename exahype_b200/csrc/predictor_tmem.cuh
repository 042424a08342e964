// Space-time predictor with the Picard iterate in tensor memory (five state
// variables, no parameters; orders 3, 4, 5 and 7).
//
// Same algorithm and outputs as predictor_kernel (aderdg.cuh): the Picard
// iteration of aderPicardLoopNonlinear (3d/spaceTimePredictorNonlinear.cpph:
// 42-329), time averaging (:337-409), extrapolation (:411-528) and
// volumeIntegralNonlinear (3d/volumeIntegralNonlinear.cpph:135-225).
//
// A thread owns one node of one cell. Its space-time iterate lives in tensor
// memory (tmem.cuh: one lane, 10 columns per time slice), its Picard
// accumulators in registers. A sweep passes through the time slices in pairs,
// each in three phases:
//   A  the node's fluxes go line-major to shared memory, sF[d][n][line][v];
//   B  a thread per (line, v) contracts the line with the stiffness matrix, in
//      place; where a cell has a thread for each, the same thread serves its
//      line index in every direction, so that one register and compile-time
//      constants make up every address;
//   C  the node's thread takes the directions' results, scales them by
//      dt / dx_d and folds them into its accumulators.
// C of one pair and A of the next read and rewrite the same slots by the same
// thread, so two barriers per pair suffice.
//
// The quadrature factors w_a w_c of a line and 1 / w_node of the Picard update
// cancel up to 1 / w_l along the line, which the tables hold (LineTables): no
// scaling in phase B, none by w_node in C. The guess lQi(:,t) = luh has the
// same fluxes in every slice, so the first sweep is one slice's A and B, and
// its fold over the slices is two table sums per slice.
//
// Bound: latency of the FP64 chains and the barriers between the phases at 14
// warps per SM (two blocks by registers; the accumulators alone are 60 at
// N = 5), next the shared-memory pipe (69 %) and the FP64 pipe (45 %). Measured
// without gain: overlapping the phases of consecutive pairs in two buffers
// (fewer barriers, the same chains: 0.96 ms against 0.88 on 27^3 N=5), two
// threads per node with half of the slices each (twice the warps at 72
// registers: 1.08 ms), running flux averages in tensor memory instead of
// re-evaluating the last sweep's fluxes (0.88 ms), the lines of phase B loaded
// one ahead (spills). Against the form with a factor per line, items over all
// directions and three barriers per pair: 27^3 N=5 1.052 -> 0.870 ms, 17x13x11
// N=7 1.144 -> 0.436, 37x33x29 N=3 list 0.408 -> 0.331, 2D 81^2 N=5 65 -> 52 us
// (1.8 to 2.1 sweeps per cell).
//
// Tensor-memory instructions are warp-collective, so the block is whole warps
// and each of them is issued by all threads under warp-uniform control; per-cell
// work is selected by the data (a warp can hold nodes of several cells).
#pragma once
#include "line_tables.cuh"
#include "predictor_lines.cuh"
#include "tmem.cuh"

namespace exa {

// Cells per block: what fits 128 threads (one warp for each quadrant of the
// tensor memory's lanes), or one cell. A block waits at its barriers for all of
// its cells and sweeps as often as the slowest, so smaller is better, as long as
// the register file (512 threads of 128 registers) stays full: against blocks of
// up to 256 threads 3D N=4 17,714 cells 474 -> 369 us, 3D N=3 31,868 cells
// 361 -> 317, 2D N=7 13,176 cells 230 -> 191, 2D N=3 53,144 cells 124 -> 110,
// 2D N=5 29,160 cells 197 -> 193 (the last warp of 128 is a third empty there).
// FEW: so few cells that the chip is not full anyway (kFewCells). One cell per
// block (two where they share a warp) spreads them over the SMs, and with no
// budget for other blocks nothing spills: 81 cells 2D N=3 9.9 -> 9.6 us, N=4
// 12.2 -> 10.4, N=7 17.6 -> 13.5, 216 cells 3D N=5 33.4 -> 31.5; at 729 cells
// 2D N=4 takes 13.4 instead of 12.5 us.
template <int DIM, int N, class PDE, bool FEW = false>
struct TmemCfg : Shape<DIM, N, PDE> {
  using S = Shape<DIM, N, PDE>;
  static constexpr int CPB = FEW ? (S::P == 16 ? 2 : 1) : S::P <= 128 ? 128 / S::P : 1;
  static constexpr int THREADS = (CPB * S::P + 31) / 32 * 32;
  static constexpr int MINB = FEW ? 1 : 512 / THREADS;  // blocks per SM of the register budget
  // cells up to which FEW is taken: two per SM
  static constexpr int kFewCells = S::P < 512 ? 2 * 148 : 0;  // (3D N=7: the same block)
  static constexpr int LINES = S::F, LI = LINES * S::nV;
  static constexpr bool kByDir = LI <= S::P;
  static constexpr int ROUNDS = kByDir ? DIM : (DIM * LI + S::P - 1) / S::P;
  // slab strides and line orders per direction (predictor_lines.cuh)
  static constexpr __host__ __device__ int sstride(int d) {
    return line_slab_dir(S::b, DIM, S::nV, d, line_slab(S::b, DIM, LINES * S::nV));
  }
  static constexpr __host__ __device__ int sbase(int d) {
    return S::b * ((d > 0 ? sstride(0) : 0) + (d > 1 ? sstride(1) : 0));
  }
  static constexpr __host__ __device__ bool sswap(int d) { return line_swap_dir(S::b, DIM, S::nV, d); }
  static constexpr int SFJ = sbase(DIM - 1) + S::b * sstride(DIM - 1);  // one slice of one cell
  static constexpr int TS = 2;                                          // slices per pair
  static constexpr int SF = TS * SFJ, PAIRS = (S::b + TS - 1) / TS;
  static constexpr bool kOne = CPB == 1;
  // residual sums: per warp where whole warps belong to a cell
  static constexpr int SR = kOne ? THREADS / 32 : S::P % 32 == 0 || S::P == 16 ? S::P / 16 : S::P + 1;
  static constexpr size_t SMEM = sizeof(double) * (size_t)(CPB * (SF + SR));
  // 32-bit columns per thread and per CTA (the warps of a lane quadrant take
  // consecutive ranges)
  static constexpr int COLS = 2 * S::b * S::nV;
  static constexpr int TCOLS = pow2ceil(COLS * ((THREADS / 32 + 3) / 4));
  static constexpr bool kFits = S::nD == 5 && S::nV == 5 && THREADS <= 512 && MINB * TCOLS <= 512 &&
                                MINB * (SMEM + 2048) <= 228 * 1024;
  static_assert(S::P * S::nV <= SFJ, "the time-averaged state is staged in the second slice buffer");
  static_assert(kByDir || sstride(0) == sstride(DIM - 1), "items over all directions: one stride");
  // items over all directions go by p + r P: a thread past the last node would take
  // another's item and contract its line a second time, in place
  static_assert(kByDir || THREADS == CPB * S::P, "items over all directions: a node for every thread");
};

template <int DIM, int N, class PDE, bool FEW>
__global__ void __launch_bounds__(TmemCfg<DIM, N, PDE, FEW>::THREADS, TmemCfg<DIM, N, PDE, FEW>::MINB)
    predictor_tmem_kernel(const double* __restrict__ luh, double* __restrict__ lQhbnd, double* __restrict__ lFhbnd,
                          double* __restrict__ lduh, int* __restrict__ iters, unsigned long long* __restrict__ sweeps,
                          const double* __restrict__ dt_ptr, Geometry geo, int ncells,
                          const int* __restrict__ cell_list, const int* __restrict__ count) {
  using C = TmemCfg<DIM, N, PDE, FEW>;
  constexpr int b = C::b, P = C::P, nV = C::nV, LI = C::LI, CPB = C::CPB, TS = C::TS;
  constexpr unsigned kAll = 0xffffffffu;
  extern __shared__ double smem[];
  const LineTables<N>& K = line_tab<N>();

  const int nact = count ? min(*count, ncells) : ncells;  // count: optional device-side list length
  if ((int)blockIdx.x * CPB >= nact) return;              // whole block, before its first barrier
  const int lc = min((int)threadIdx.x / P, CPB - 1);
  const int p = threadIdx.x - lc * P;
  const int slot = blockIdx.x * CPB + lc;
  const bool active = slot < nact;
  const bool node = active && p < P;  // the threads past the last node hold none
  const int cell = active ? (cell_list ? cell_list[slot] : slot) : 0;
  const int warp = threadIdx.x >> 5;

  __shared__ uint32_t s_tbase;
  __shared__ int s_sweeps;
  if (warp == 0) tmem::alloc(&s_tbase, C::TCOLS);
  if (threadIdx.x == 0) s_sweeps = 0;

  double* sF = smem + lc * C::SF;
  double* sQh = sF + C::SFJ;  // time-averaged state [P][nV] of a finished cell
  double* sR = smem + CPB * C::SF + lc * C::SR;
  const int pn = p < P ? p : 0;  // (a thread past the last node: indices in range, nothing stored)
  const int x = pn % b, y = (pn / b) % b, z = DIM == 3 ? pn / (b * b) : 0;
  int sa[DIM];  // this node's slot in each direction's part of a slice (+ v)
#pragma unroll
  for (int d = 0; d < DIM; d++) {
    int n, L;
    node_line<DIM, b>(d, z, y, x, n, L);
    sa[d] = C::sbase(d) + n * C::sstride(d) + line_swapped<b>(C::sswap(d), L) * nV;
  }
  // phase-B items of this thread: first element in a slice, -1: none
  int item[C::kByDir ? 1 : C::ROUNDS];
  if constexpr (C::kByDir) {
    item[0] = active && p < LI ? p : -1;
  } else {
#pragma unroll
    for (int r = 0; r < C::ROUNDS; r++) {
      const int it = p + r * P;
      item[r] = active && it < DIM * LI ? C::sbase(1) * (it / LI) + it % LI : -1;
    }
  }
  const int inst = cell_instance(geo, cell);
  const double dt = dt_ptr[inst];
  double cd[DIM];  // dt / dx_d
#pragma unroll
  for (int d = 0; d < DIM; d++) cd[d] = dt * (1.0 / cell_width(geo, inst, d));

  auto put_flux = [&](const double (&Fl)[DIM][nV], double* buf) {
#pragma unroll
    for (int d = 0; d < DIM; d++)
#pragma unroll
      for (int v = 0; v < nV; v++) buf[sa[d] + v] = Fl[d][v];
  };
  // phase B on one slice
  auto contract = [&](double* buf) {
#pragma unroll
    for (int r = 0; r < C::ROUNDS; r++) {
      const int it = item[C::kByDir ? 0 : r];
      const int is = C::kByDir ? C::sstride(r) : C::sstride(0);
      if (it < 0) continue;
      double* base = buf + it + (C::kByDir ? C::sbase(r) : 0);
      double f[b];
#pragma unroll
      for (int n = 0; n < b; n++) f[n] = base[n * is];
      line_contract<b>(f, K.KP, K.KQ, [&](int l, double s) { base[l * is] = s; });
    }
  };
  // phase C on one slice: sum_d dt/dx_d S_d at this node
  auto gather = [&](const double* buf, double (&s)[nV]) {
#pragma unroll
    for (int v = 0; v < nV; v++) {
      s[v] = cd[0] * buf[sa[0] + v];
#pragma unroll
      for (int d = 1; d < DIM; d++) s[v] = fma(cd[d], buf[sa[d] + v], s[v]);
    }
  };
  // the cell's sum of one value per thread, in a fixed order
  auto cell_sum = [&](double part) -> double {
    if (!node) part = 0.0;
    if constexpr (P == 16) {
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) part += __shfl_xor_sync(kAll, part, o);
      return part;
    } else if constexpr (C::kOne || P % 32 == 0) {
      constexpr int NW = C::kOne ? C::THREADS / 32 : P / 32;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(kAll, part, o);
      double* red = smem + CPB * C::SF;
      if ((threadIdx.x & 31) == 0) red[warp] = part;
      __syncthreads();
      double s = 0.0;
#pragma unroll
      for (int w = 0; w < NW; w++) s += red[lc * NW + w];
      return s;
    } else {
      if (p < P) sR[p] = part;
      __syncthreads();
      const int lane = threadIdx.x & 31;
      for (int c = warp; c < CPB; c += C::THREADS / 32) {
        double* rr = smem + CPB * C::SF + c * C::SR;
        double acc = 0.0;
        for (int i = lane; i < P; i += 32) acc += rr[i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(kAll, acc, o);
        if (lane == 0) rr[P] = acc;
      }
      __syncthreads();
      return sR[P];
    }
  };

  double q[nV];
  const double* src = luh + ((size_t)cell * P + pn) * nV;
#pragma unroll
  for (int v = 0; v < nV; v++) q[v] = node ? __ldg(src + v) : 0.0;

  // first sweep: one slice's phases for all (see above)
  if (node) {
    double Fl[DIM][nV];
    PDE::template flux<DIM>(q, Fl);
    put_flux(Fl, sF);
  }
  tmem::fence_before_sync();
  __syncthreads();  // (also the allocation's address)
  tmem::fence_after_sync();
  const uint32_t taddr = s_tbase + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(C::COLS * (warp >> 2));
  contract(sF);
  __syncthreads();
  bool done = !active;
  int it_done = 1;
  {
    double s[nV];
    gather(sF, s);
    double part = 0.0;
#pragma unroll
    for (int l = 0; l < b; l++) {
      double qn[nV];
#pragma unroll
      for (int v = 0; v < nV; v++) {
        qn[v] = fma(K.beta[l], s[v], K.alpha[l] * q[v]);
        const double dq = qn[v] - q[v];
        part = fma(dq, dq, part);
      }
      uint32_t r[10];
      tmem::pack5(qn, r);
      tmem::st10(taddr + 10u * l, r);
    }
    const double sq = cell_sum(part);
    tmem::wait_st();
    if (!done && (sq < 1e-7 * 1e-7 || C::maxIter == 1)) {
      done = true;
      if (node) {  // the time averages of the guess's fluxes and of the new iterate
        double W = 0.0;
#pragma unroll
        for (int t = 0; t < b; t++) W += K.w[t];
        double Fl[DIM][nV];
        PDE::template flux<DIM>(q, Fl);
#pragma unroll
        for (int d = 0; d < DIM; d++)
#pragma unroll
          for (int v = 0; v < nV; v++) sF[sa[d] + v] = Fl[d][v] * W;
#pragma unroll
        for (int v = 0; v < nV; v++) {
          double a = 0.0;
#pragma unroll
          for (int l = 0; l < b; l++) a += fma(K.beta[l], s[v], K.alpha[l] * q[v]) * K.w[l];
          sQh[p * nV + v] = a;
        }
      }
    }
  }

  for (int iter = 1; iter < C::maxIter; iter++) {
    if constexpr (C::kOne) {  // one cell: every thread read the same sum
      if (done) break;
    } else if (!__syncthreads_or(!done)) {
      break;
    }
    const bool live = node && !done;
    double qn[b][nV];
#pragma unroll
    for (int v = 0; v < nV; v++) {
      const double lu = node ? __ldg(src + v) : 0.0;
#pragma unroll
      for (int l = 0; l < b; l++) qn[l][v] = K.alpha[l] * lu;
    }
#pragma unroll 1
    for (int k = 0; k <= C::PAIRS; k++) {
#pragma unroll
      for (int j = 0; j < TS; j++) {
        const int tc = (k - 1) * TS + j, t = k * TS + j;
        if (k > 0 && live && (b % TS == 0 || tc < b)) {  // C of the pair before
          double s[nV];
          gather(sF + j * C::SFJ, s);
#pragma unroll
          for (int l = 0; l < b; l++) {
            const double c = K.niK1w[tc * b + l];
#pragma unroll
            for (int v = 0; v < nV; v++) qn[l][v] = fma(s[v], c, qn[l][v]);
          }
        }
        if (k < C::PAIRS && (b % TS == 0 || t < b)) {  // A
          __syncwarp();
          uint32_t r[10];
          double Q[nV], Fl[DIM][nV];
          tmem::ld10(taddr + 10u * t, r);
          tmem::wait_ld(r);
          tmem::unpack5(r, Q);
          PDE::template flux<DIM>(Q, Fl);
          if (live) put_flux(Fl, sF + j * C::SFJ);
        }
      }
      if (k == C::PAIRS) break;
      __syncthreads();
      if (!done)
#pragma unroll
        for (int j = 0; j < TS; j++)
          if (b % TS == 0 || k * TS + j < b) contract(sF + j * C::SFJ);
      __syncthreads();
    }
    // residual against the old iterate
    __syncwarp();
    double part = 0.0;
#pragma unroll
    for (int l = 0; l < b; l++) {
      uint32_t r[10];
      double qo[nV];
      tmem::ld10(taddr + 10u * l, r);
      tmem::wait_ld(r);
      tmem::unpack5(r, qo);
#pragma unroll
      for (int v = 0; v < nV; v++) {
        const double dq = qn[l][v] - qo[v];
        part = fma(dq, dq, part);
      }
    }
    const double sq = cell_sum(part);
    const bool conv = !done && (sq < 1e-7 * 1e-7 || iter + 1 == C::maxIter);
    if (!done) it_done = iter + 1;
    if (C::kOne ? conv : __any_sync(kAll, conv)) {
      // lFhi is the time average of the fluxes this sweep evaluated, of the
      // iterate before the update. Each slice of the new iterate replaces the
      // old one as soon as the old one's flux is taken, so that accumulators,
      // fluxes and averages are never live together (they would spill).
      double fh[DIM][nV], qa[nV];
#pragma unroll
      for (int v = 0; v < nV; v++) {
        qa[v] = 0.0;
#pragma unroll
        for (int d = 0; d < DIM; d++) fh[d][v] = 0.0;
      }
#pragma unroll
      for (int t = 0; t < b; t++) {
        uint32_t r[10];
        double Q[nV];
        tmem::ld10(taddr + 10u * t, r);
        tmem::wait_ld(r);
        tmem::unpack5(r, Q);
        if constexpr (!C::kOne) {  // (other cells of the warp go on)
          tmem::pack5(qn[t], r);
          tmem::st10(taddr + 10u * t, r);
        }
#pragma unroll
        for (int v = 0; v < nV; v++) qa[v] = fma(qn[t][v], K.w[t], qa[v]);
        double Fl[DIM][nV];
        PDE::template flux<DIM>(Q, Fl);
#pragma unroll
        for (int d = 0; d < DIM; d++)
#pragma unroll
          for (int v = 0; v < nV; v++) fh[d][v] = fma(Fl[d][v], K.w[t], fh[d][v]);
      }
      if (conv && node)
#pragma unroll
        for (int v = 0; v < nV; v++) {
          sQh[p * nV + v] = qa[v];
#pragma unroll
          for (int d = 0; d < DIM; d++) sF[sa[d] + v] = fh[d][v];
        }
      __syncwarp();
    } else {
#pragma unroll
      for (int l = 0; l < b; l++) {
        uint32_t r[10];
        tmem::pack5(qn[l], r);
        tmem::st10(taddr + 10u * l, r);
      }
    }
    if (conv) done = true;
    tmem::wait_st();
  }
  if (active && p == 0) {
    if (iters) iters[cell] = it_done;
    if (sweeps) atomicAdd(&s_sweeps, it_done);
  }
  tmem::fence_before_sync();
  __syncthreads();  // every cell's averages are in shared memory, every tensor-memory load has landed
  tmem::fence_after_sync();
  if (warp == 0) tmem::dealloc(s_tbase, C::TCOLS);
  if (sweeps && threadIdx.x == 0) atomicAdd(sweeps, (unsigned long long)s_sweeps);

  // extrapolated states and fluxes and the volume-integral contractions, one
  // thread per (line, v) and direction
  double* Qb = lQhbnd + (size_t)cell * 2 * DIM * LI;
  double* Fb = lFhbnd + (size_t)cell * 2 * DIM * LI;
#pragma unroll
  for (int r = 0; r < C::ROUNDS; r++) {
    const int it = C::kByDir ? p : p + r * P;
    if (!active || it >= (C::kByDir ? LI : DIM * LI)) continue;
    const int d = C::kByDir ? r : it / LI, e = C::kByDir ? it : it - d * LI;
    const int v = e % nV, Ls = e / nV;                // slab order
    const int L = line_swapped<b>(C::sswap(d), Ls);  // face-node order
    const int is = C::sstride(d);
    double* base = sF + C::sbase(d) + e;
    const int a0 = L / b, a1 = L % b;
    const int n0 = DIM == 2 ? (d == 0 ? L * b : L) : d == 0 ? (a0 * b + a1) * b : d == 1 ? a0 * b * b + a1 : a0 * b + a1;
    const int step = d == 0 ? 1 : d == 1 ? b : b * b;
    double f[b], sl = 0.0, sr = 0.0, ql = 0.0, qr = 0.0;
#pragma unroll
    for (int n = 0; n < b; n++) f[n] = base[n * is];
#pragma unroll
    for (int n = 0; n < b; n++) {
      sl += f[n] * K.FL[n];
      sr += f[n] * K.FR[n];
      const double qv = sQh[(n0 + n * step) * nV + v];
      ql += qv * K.FL[n];
      qr += qv * K.FR[n];
    }
    const int o = 2 * d * LI + L * nV + v;
    Fb[o] = sl;
    Fb[o + LI] = sr;
    Qb[o] = ql;
    Qb[o + LI] = qr;
    line_contract<b>(f, K.VP, K.VQ, [&](int l, double s) { base[l * is] = s; });
  }
  if (!lduh) return;
  __syncthreads();
  // the volume integral at this node, staged and written by consecutive
  // threads to consecutive addresses: a node's own nV doubles per thread
  // would make every store instruction a partial write of 32 sectors
  if (node) {
    const double wpt = (DIM == 3 ? K.w[z] : 1.0) * K.w[y] * K.w[x];
    double g[DIM];
#pragma unroll
    for (int d = 0; d < DIM; d++) g[d] = wpt / cell_width(geo, inst, d);
#pragma unroll
    for (int v = 0; v < nV; v++) {
      double du = g[0] * sF[sa[0] + v];
#pragma unroll
      for (int d = 1; d < DIM; d++) du = fma(g[d], sF[sa[d] + v], du);
      sQh[p * nV + v] = du;
    }
  }
  __syncthreads();
  if (active && p < P)
#pragma unroll
    for (int j = 0; j < nV; j++) lduh[(size_t)cell * P * nV + j * P + p] = sQh[j * P + p];
}

}  // namespace exa
