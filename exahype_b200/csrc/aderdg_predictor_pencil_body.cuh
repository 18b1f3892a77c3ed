// FP64 predictor + volume integral, one thread per space-time pencil.
//
// Same operator, stopping rule and precision as predictor_block (the
// reference's aderPicardLoopNonlinear / aderPredictorNonlinear /
// aderExtrapolatorNonlinear / volumeIntegralNonlinear); what changes is who
// holds what.  A cell of B^DIM nodes has B^DIM threads; thread (n, [z,] y)
// owns the x pencil ([z,] y) of time slice n and keeps its B x V iterate in
// registers.  All B slices of a Picard iteration advance together:
//   A  the owner evaluates the flux of its B nodes, takes the x derivative of
//      its pencil in registers and stores G_x, F_y and (3D) F_z;
//   Y  (3D) line tasks (n, z, x, variable) read a y line of F_y and add its
//      derivative to G;
//   T  line tasks ([y,] x, variable) of the last direction read their line of
//      F and G for every slice, finish G, contract it in time and store the
//      new iterate of all slices over G;
// and the owner reads its new pencil back and adds up the squared increment.
// The line-owner kernels this replaces moved 4 DIM doubles per node, variable
// and slice through shared memory and took one barrier per slice; here it is
// 10 (3D) or 6 (2D) doubles and three or two barriers per iteration, every
// thread has B independent fluxes (their divisions overlap), and cells are
// packed without padding to a power of two or to whole warps (2D order 5:
// five cells of 36 threads in 192 instead of three; order 2: 14 in 128 instead
// of 8).
//
// The arrays [n][z][y][x][variable] are padded so that every access above is
// free of bank conflicts or nearly so (16 banks of 8 bytes per half-warp).
//
// What bounds it (3D order 4, 39,304 cells): the shared-memory pipe, 77 % of
// its wavefront peak (427 M wavefronts, 4 % of them conflicts), with the FP64
// pipe at 57 %; 1.95 ms against 2.35 ms for the progressive line-owner kernel
// (67 % and 47 %).  2D order 4: 77 % and 48 %.  Registers decide: with 92 to 220
// bytes of spills the same code lost its whole gain, since three CTAs of 73 KB
// leave no L1 for them.
#pragma once
#include "exa_device.cuh"
#include "aderdg_predictor_mixed_body.cuh"

namespace exa {

// cells per CTA of the stand-alone kernel: what 128 threads hold (2D order 5:
// five cells in 192, 94 % of the lanes instead of 84 %), one in 3D
template <int DIM, int N>
constexpr int pencil_cells() {
  return DIM == 3 ? 1 : (N == 2 ? 14 : (N == 3 ? 8 : 5));
}

template <int DIM, int N, int CPB_ = pencil_cells<DIM, N>()>
struct PencilShape {
  using M = MixShape<DIM, N>;
  static constexpr int B = N + 1;
  static constexpr int V = kV;
  static constexpr int NPC = ipow(B, DIM);
  static constexpr int TPC = NPC;          // threads per cell: B slices x B^(DIM-1) pencils
  static constexpr int LINES = NPC / B;    // pencils of a slice
  static constexpr int CPB = CPB_;
  static constexpr int NT = round_up(CPB * TPC, 32);
  // strides in doubles and the padding that keeps the half-warps' addresses
  // in distinct banks (found by enumerating the access patterns)
  static constexpr int ROW = B * V + (DIM == 2 && N == 2 ? 2 : (N == 5 ? 1 : 0));
  static constexpr int PLANE = B * ROW + (DIM == 3 && N == 3 ? 1 : 0);
  static constexpr int SLICE = (DIM == 3 ? B * PLANE : B * ROW) + (DIM == 2 && N == 3 ? 1 : 0);
  static constexpr int ARRAY = B * SLICE;
  static constexpr int PAD_CELL = DIM == 2 ? (N == 2 || N == 4 ? 7 : (N == 5 ? 4 : 0)) : 0;
  static constexpr int CELL_D = (DIM * ARRAY > M::STAGE_D ? DIM * ARRAY : M::STAGE_D) + PAD_CELL;
  // residual partials: per warp (one cell), or per cell and warp piece, two
  // sets used alternately
  static constexpr int RED = CPB > 1 ? CPB * 3 : NT / 32;
  static constexpr int SM_DOUBLES = CPB * CELL_D + 2 * RED;
  static constexpr int T_TASKS = LINES * V;
  static constexpr int T_ROUNDS = (T_TASKS + TPC - 1) / TPC;
};

// y-line task order of a slice in 3D order 4: 125 tasks z * 25 + (x, variable)
// arranged so that each half-warp touches 16 distinct banks (in plain order
// half of the half-warps cross a plane and collide)
__device__ const unsigned char kPencilY34[125] = {
    0,   1,   2,   3,   4,   5,   6,   7,   8,   9,   10,  11,  12,  13,  14,  15,  16,  17,  18,  19,  20,
    21,  22,  23,  24,  37,  38,  39,  40,  25,  26,  27,  28,  29,  30,  31,  32,  33,  34,  35,  36,  65,
    50,  51,  52,  41,  42,  43,  44,  45,  46,  47,  48,  49,  62,  63,  64,  77,  66,  67,  68,  53,  54,
    55,  56,  57,  58,  59,  60,  61,  90,  75,  76,  93,  78,  79,  80,  69,  70,  71,  72,  73,  74,  87,
    88,  89,  102, 91,  92,  105, 94,  95,  96,  81,  82,  83,  84,  85,  86,  115, 100, 101, 118, 103, 104,
    121, 106, 107, 108, 97,  98,  99,  112, 113, 114, 116, 117, 119, 120, 122, 123, 124, 109, 110, 111};

// Sum of v over the threads of each cell (every thread of the CTA calls it;
// threads outside a cell pass cell -1).  The order depends on where the cell
// lies in the CTA; the parts are multiples of 2^-98 (kPicardBase), so the sum
// does not where it matters.  One barrier; the partials go to one
// of two sets chosen by the iteration's parity, so the next call's stores
// never meet this call's loads.
template <typename S>
__device__ __forceinline__ double pencil_sum(double v, int lc, int s, double* sred, int parity) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* slot = sred + (parity & 1) * S::RED;
  if constexpr (S::CPB == 1) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) slot[warp] = v;
    __syncthreads();
    double r = 0.0;
#pragma unroll
    for (int k = 0; k < S::NT / 32; k++) r += slot[k];
    return r;
  } else {
    // lane l adds the later lanes of its cell: the cell's first lane of the
    // warp ends with the warp's part of the cell
    const int left = S::TPC - s;  // lanes of this cell from this one on
#pragma unroll
    for (int o = 1; o < 32 && o < S::TPC; o <<= 1) {
      const double w = __shfl_down_sync(0xffffffffu, v, o);
      if (o < left && lane + o < 32) v += w;
    }
    const int first_warp = (lc * S::TPC) >> 5;
    if (lc < S::CPB && (s == 0 || lane == 0)) slot[lc * 3 + warp - first_warp] = v;
    __syncthreads();
    if (lc >= S::CPB) return 0.0;
    const int last_warp = (lc * S::TPC + S::TPC - 1) >> 5;
    double r = slot[lc * 3];
    if (last_warp > first_warp) r += slot[lc * 3 + 1];
    if (last_warp > first_warp + 1) r += slot[lc * 3 + 2];
    return r;
  }
}

template <int DIM, int N, bool PLANAR, int CPB_ = pencil_cells<DIM, N>()>
__device__ __forceinline__ void predictor_pencil_block(const PredArgs& a, long block, double* smem) {
  using S = PencilShape<DIM, N, CPB_>;
  constexpr int B = S::B, V = S::V, NPC = S::NPC, TPC = S::TPC, LINES = S::LINES;
  constexpr int ROW = S::ROW, PLANE = S::PLANE, SLICE = S::SLICE, ARRAY = S::ARRAY;
  constexpr int R5 = B * V;  // unpadded row: x, variable
  constexpr int MAXIT = 2 * (N + 1);
  constexpr bool kMulti = S::CPB > 1;
  // the new pencil stays in registers across the residual's barrier where
  // they allow it (one cell per CTA), else it is read again
  constexpr bool kHold = !kMulti;
  // slices unrolled in T: all where the registers allow it
  constexpr int kUnrollT = N <= 3 ? B : 1;
  const DGConst& T = c_dg[N];

  const int lc = threadIdx.x / TPC;
  const int s = threadIdx.x - lc * TPC;
  const long cell = block * S::CPB + lc;
  const bool valid = lc < S::CPB && cell < a.ncells;
  double* sG = smem + (lc < S::CPB ? lc : 0) * S::CELL_D;  // G, then the new iterate
  double* sF1 = sG + ARRAY;                                 // F_y
  double* sF2 = sG + 2 * ARRAY;                             // F_z (3D)
  double* sFT = sG + (DIM - 1) * ARRAY;                     // flux of T's direction
  double* sred = smem + S::CPB * S::CELL_D;
  const double* luh = a.luh + (valid ? cell : 0) * (long)NPC * V;
  const double dt = a.dt_dev ? *a.dt_dev : a.dt;

  // owner role: slice sn, pencil sl = (z, y)
  const int sn = s / LINES, sl = s - sn * LINES;
  const int pz = DIM == 3 ? sl / B : 0, py = DIM == 3 ? sl - pz * B : sl;
  const int own = sn * SLICE + pz * PLANE + py * ROW;
  // first T task: in 2D order 5 turned by four from cell to cell, which keeps
  // the half-warps that straddle two cells free of conflicts
  const int st = DIM == 2 && N == 5 ? (s + 4 * lc) % TPC : s;
  // node role: node s = (nz, ny, nx)
  const int nx = s % B, ny = (s / B) % B, nz = DIM == 3 ? s / (B * B) : 0;
  const int node = nz * PLANE + ny * ROW + nx * V;

  // ---- first iteration: the iterate is luh in every slice, so one slice is
  // evaluated and every other takes its values
  if (valid) {
    double u[V], F[DIM][V];
#pragma unroll
    for (int m = 0; m < V; m++) u[m] = luh[s * V + m];
    euler_flux<DIM, PLANAR>(u, F);
#pragma unroll
    for (int m = 0; m < V; m++) {
      sG[node + m] = F[0][m];
      sF1[node + m] = F[1][m];
      if (DIM == 3) sF2[node + m] = F[DIM - 1][m];
    }
  }
  __syncthreads();
  if (valid)
#pragma unroll
    for (int r = 0; r < S::T_ROUNDS; r++) {
      const int k = s + r * TPC;
      if (k < S::T_TASKS) {
        const int l = k / V, m = k - l * V;
        double* g = sG + (DIM == 3 ? (l / B) * PLANE + (l % B) * ROW : l * ROW) + m;
        double f[B];
#pragma unroll
        for (int p = 0; p < B; p++) f[p] = g[p * V];
#pragma unroll
        for (int i = 0; i < B; i++) {
          double d = 0.0;
#pragma unroll
          for (int p = 0; p < B; p++) d += T.deriv[i][p] * f[p];
          g[i * V] = a.idx[0] * d;
        }
      }
    }
  __syncthreads();
  if constexpr (DIM == 3) {
    if (valid)
#pragma unroll
      for (int r = 0; r < S::T_ROUNDS; r++) {
        const int k = s + r * TPC;
        if (k < S::T_TASKS) {
          const int o = (k / R5) * PLANE + k % R5;
          double f[B];
#pragma unroll
          for (int p = 0; p < B; p++) f[p] = sF1[o + p * ROW];
#pragma unroll
          for (int i = 0; i < B; i++) {
            double d = 0.0;
#pragma unroll
            for (int p = 0; p < B; p++) d += T.deriv[i][p] * f[p];
            sG[o + i * ROW] += a.idx[1] * d;
          }
        }
      }
    __syncthreads();
  }
  constexpr int TS = DIM == 3 ? PLANE : ROW;         // stride of T's direction in shared memory
  constexpr int TG = DIM == 3 ? B * B * V : B * V;   // and in luh
  if (valid)
#pragma unroll
    for (int r = 0; r < S::T_ROUNDS; r++) {
      const int k = s + r * TPC;
      if (k < S::T_TASKS) {
        const int o = DIM == 3 ? (k / R5) * ROW + k % R5 : k;
        double f[B], g[B];
#pragma unroll
        for (int p = 0; p < B; p++) {
          f[p] = sFT[o + p * TS];
          g[p] = sG[o + p * TS];
        }
#pragma unroll
        for (int i = 0; i < B; i++) {
          double d = 0.0;
#pragma unroll
          for (int p = 0; p < B; p++) d += T.deriv[i][p] * f[p];
          g[i] = fma(a.idx[DIM - 1], d, g[i]);
        }
#pragma unroll
        for (int i = 0; i < B; i++) {
          const double u = luh[i * TG + k];
#pragma unroll
          for (int t = 0; t < B; t++) sG[o + t * SLICE + i * TS] = picard_new(T.c0[t], u, dt, T.tAsum[t] * g[i]);
        }
      }
    }
  double q[B][V];  // the owner's iterate
#pragma unroll
  for (int x = 0; x < B; x++)
#pragma unroll
    for (int m = 0; m < V; m++) q[x][m] = valid ? luh[sl * R5 + x * V + m] : 0.0;
  __syncthreads();

  int it = 0;
  // done: this thread's cell has its outputs' values (uniform over the CTA
  // with one cell; threads without a cell are done after one iteration)
  bool conv = false, done = false;
  // lost: the last residual was NaN.  A cell of nothing but NaN (a run that has
  // blown up) would iterate to the limit, 2(N+1) times, and stay NaN, each value
  // being a sum over the others.  A thread whose pencil holds only NaN would
  // make the residual NaN again; it adds kVote in its stead, and a sum of TPC
  // votes (exact, and out of reach for fewer: the others add no less than 0) ends
  // the cell.  Any other sum with a vote in it is not below the tolerance.
  constexpr double kVote = -0x1p1000;
  bool lost = false;
  for (int iter = 0;; iter++) {
    // the new pencil and its squared increment
    double qn[B][V], r2 = 0.0;
    if (valid && !done) {
      r2 = kPicardBase;
#pragma unroll
      for (int x = 0; x < B; x++)
#pragma unroll
        for (int m = 0; m < V; m++) {
          const double v = sG[own + x * V + m];
          const double d = q[x][m] - v;
          r2 = fma(d, d, r2);
          if (kHold) qn[x][m] = v;
        }
      r2 -= kPicardBase;
    }
    if (lost && valid && !done) {
      bool all = true;
#pragma unroll
      for (int x = 0; x < B; x++)
#pragma unroll
        for (int m = 0; m < V; m++) all = all && isnan(q[x][m]);
      if (all) r2 = kVote;
    }
    const double res = pencil_sum<S>(r2, lc, s, sred, iter);
    if (!done) {
      it = res == TPC * kVote ? MAXIT : iter + 1;
      conv = res >= 0.0 && res < kPicardTol2;
      lost = !(res >= 0.0);
      done = conv || it == MAXIT;
      // the outputs need the last iteration's input (for its flux), put in
      // F_y's place, and its result, over G
      if (done && valid)
#pragma unroll
        for (int x = 0; x < B; x++)
#pragma unroll
          for (int m = 0; m < V; m++) sF1[own + x * V + m] = q[x][m];
      if (kHold) {
#pragma unroll
        for (int x = 0; x < B; x++)
#pragma unroll
          for (int m = 0; m < V; m++) q[x][m] = qn[x][m];
      } else if (valid && !done) {
#pragma unroll
        for (int x = 0; x < B; x++)
#pragma unroll
          for (int m = 0; m < V; m++) q[x][m] = sG[own + x * V + m];
      }
    }
    if constexpr (kMulti) {
      if (__syncthreads_and(done)) break;
    } else {
      if (done) break;
    }

    // A: fluxes of the pencil, x derivative
    if (valid && !done) {
      double g[B][V];
#pragma unroll
      for (int i = 0; i < B; i++)
#pragma unroll
        for (int m = 0; m < V; m++) g[i][m] = 0.0;
#pragma unroll
      for (int x = 0; x < B; x++) {
        double F[DIM][V];
        euler_flux<DIM, PLANAR>(q[x], F);
#pragma unroll
        for (int m = 0; m < V; m++) {
          sF1[own + x * V + m] = F[1][m];
          if (DIM == 3) sF2[own + x * V + m] = F[DIM - 1][m];
#pragma unroll
          for (int i = 0; i < B; i++) g[i][m] += T.deriv[i][x] * F[0][m];
        }
      }
#pragma unroll
      for (int x = 0; x < B; x++)
#pragma unroll
        for (int m = 0; m < V; m++) sG[own + x * V + m] = a.idx[0] * g[x][m];
    }
    __syncthreads();
    // Y: y lines of every slice (5 per thread)
    if constexpr (DIM == 3) {
      if (valid && !done) {
#pragma unroll
        for (int r = 0; r < V; r++) {
          int o;
          if constexpr (N == 4) {
            const int k = kPencilY34[s];
            o = r * SLICE + (k / R5) * PLANE + k % R5;
          } else if constexpr (N == 3) {
            // lines (n, z, 0..15) by half-warps, then the four left of each:
            // 16 distinct banks every time
            const int h = s >> 4, i = s & 15;
            o = r < 4 ? r * SLICE + h * PLANE + i : (i >> 2) * SLICE + h * PLANE + 16 + (i & 3);
          } else {
            const int k = s + r * TPC;
            const int n = k / (B * R5), j = k - n * (B * R5);
            o = n * SLICE + (j / R5) * PLANE + j % R5;
          }
          double f[B];
#pragma unroll
          for (int p = 0; p < B; p++) f[p] = sF1[o + p * ROW];
#pragma unroll
          for (int i = 0; i < B; i++) {
            double d = 0.0;
#pragma unroll
            for (int p = 0; p < B; p++) d += T.deriv[i][p] * f[p];
            sG[o + i * ROW] += a.idx[1] * d;
          }
        }
      }
      __syncthreads();
    }
    // T: lines of the last direction, time contraction, new iterate
    if (valid && !done)
#pragma unroll 1
      for (int k = st; k < S::T_TASKS; k += TPC) {
        const int o = DIM == 3 ? (k / R5) * ROW + k % R5 : k;
        double acc[B][B];  // [slice][line point]
#pragma unroll
        for (int t = 0; t < B; t++)
#pragma unroll
          for (int i = 0; i < B; i++) acc[t][i] = 0.0;
#pragma unroll kUnrollT
        for (int n = 0; n < B; n++) {
          double f[B];
#pragma unroll
          for (int p = 0; p < B; p++) f[p] = sFT[o + n * SLICE + p * TS];
#pragma unroll
          for (int i = 0; i < B; i++) {
            double d = 0.0;
#pragma unroll
            for (int p = 0; p < B; p++) d += T.deriv[i][p] * f[p];
            const double g = fma(a.idx[DIM - 1], d, sG[o + n * SLICE + i * TS]);
#pragma unroll
            for (int t = 0; t < B; t++) acc[t][i] = fma(T.tA[t][n], g, acc[t][i]);
          }
        }
#pragma unroll
        for (int i = 0; i < B; i++) {
          const double u = __ldg(luh + i * TG + k);
#pragma unroll
          for (int t = 0; t < B; t++) sG[o + t * SLICE + i * TS] = picard_new(T.c0[t], u, dt, acc[t][i]);
        }
      }
    __syncthreads();
  }

  // time averages of the fluxes (of the last input iterate) and the state at
  // node s, into the staging area of the outputs
  __syncthreads();
  double fa[DIM][V], qh[V];
#pragma unroll
  for (int m = 0; m < V; m++) {
    qh[m] = 0.0;
#pragma unroll
    for (int d = 0; d < DIM; d++) fa[d][m] = 0.0;
  }
  if (valid)
#pragma unroll
    for (int n = 0; n < B; n++) {
      double u[V], F[DIM][V];
#pragma unroll
      for (int m = 0; m < V; m++) u[m] = sF1[n * SLICE + node + m];
      euler_flux<DIM, PLANAR>(u, F);
#pragma unroll
      for (int m = 0; m < V; m++) {
        qh[m] += sG[n * SLICE + node + m] * T.w[n];
#pragma unroll
        for (int d = 0; d < DIM; d++) fa[d][m] += T.w[n] * F[d][m];
      }
    }
  __syncthreads();
  if (valid) {
#pragma unroll
    for (int m = 0; m < V; m++) {
      sG[s * V + m] = qh[m];
#pragma unroll
      for (int d = 0; d < DIM; d++) sG[((d + 1) * NPC + s) * V + m] = fa[d][m];
    }
  }
  dg_line_outputs<DIM, N, TPC>(a, cell, s, valid, valid, sG, it, conv);
}

}  // namespace exa
