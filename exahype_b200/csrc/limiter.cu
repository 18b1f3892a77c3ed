// A-posteriori subcell limiter kernels for batches of cells resident on the
// GPU: the reference's kernels/limiter/generic/c/Limiter.cpp
//   projectOnFVLimiterSpace      (:23-64)   DG nodes -> subcell means
//   projectOnDGSpace             (:67-110)  subcell means -> DG nodes
//   findCellLocalMinAndMax       (:212-251) with the Gauss-Lobatto (:258-306)
//                                           and subcell (:312-368) checks
//   findCellLocalLimiterMinAndMax (:170-207)
//   discreteMaximumPrincipleAndMinAndMaxSearch (:113-167)
// plus the copy of the new extrema to every face block that
// LimitingADERDGSolver::determineSolverMinAndMax / determineLimiterMinAndMax
// (exahype/solvers/LimitingADERDGSolver.cpp:1080-1150) do after the search.
//
// The reference evaluates every projection as a direct B^dim-term sum per
// output point.  The operators are tensor products of one 1D table, so here
// they are applied as dim one-dimensional sums.  With many columns a thread
// keeps all of them for one output column (x, variable) in registers: its x sums
// from the cell's staged values (loads that the lanes of one variable share, one
// wavefront each), then y, then z.  No intermediate arrays and no pass over
// them; consecutive lanes hold consecutive (x, variable), so stores run over
// whole rows.  Few columns take one pass per direction through shared memory
// (DG -> FV and the extrema), where more threads share a cell.
//
// Layouts (the reference's, KernelUtils.h idx4): luh [z][y][x][nvar] with B
// points per direction; lim [z][y][x][nvar] with S + 2g points per
// direction (S = 2N+1 subcells, g ghost layers); only the interior of lim is
// read or written.  Min/max blocks are [2 dim][nobs] per cell.  The
// observables are the first nobs variables (the generated solvers' default
// mapDiscreteMaximumPrincipleObservables,
// AbstractGenericADERDGSolverHeader.template:159-163).
#include <cfloat>

#include "exa_device.cuh"

#define EXA_TABLE_QUAL static const
#include "dg_tables.h"

namespace exa {

constexpr int kLimMaxOrder = 6;  // B <= 7, S <= 13
constexpr int kLimNT = 256;
constexpr int kLimColNT = 128;  // threads of the projections
constexpr int kLimMmNT = 128;   // and of the extrema
constexpr int kLimMaxSmem = (int)kMaxDynSmem;

struct LimConst {
  double uh2lim[7][13];  // [k][i]: mean of phi_k over subcell i
  double uh2lob[7][7];   // [k][i]: phi_k at Gauss-Lobatto node i
  double lim2uh[13][7];  // [i][k]: conservative least-squares inverse
};
static __constant__ LimConst c_lim[kLimMaxOrder + 1];

enum { kTabUh2Lim = 0, kTabUh2Lob = 1, kTabLim2Uh = 2 };

template <int TAB, int B>
__device__ __forceinline__ double lim_coef(int p, int m) {
  if (TAB == kTabUh2Lim) return c_lim[B - 1].uh2lim[p][m];
  if (TAB == kTabUh2Lob) return c_lim[B - 1].uh2lob[p][m];
  return c_lim[B - 1].lim2uh[p][m];
}

// std::min / std::max semantics: (b < a) ? b : a and (a < b) ? b : a
__device__ __forceinline__ double lim_min(double a, double b) { return b < a ? b : a; }
__device__ __forceinline__ double lim_max(double a, double b) { return a < b ? b : a; }

// CTAs per SM that the projections' registers are bounded for: the most that
// compile (nearly) without spills.  In DG -> FV a reload waits behind the row's
// stores: 40 bytes of them cost a third of the kernel.
template <int DIM, int B, bool TO_FV>
struct LimMinB {
  static constexpr int fv[8] = {0, 0, 8, 8, 5, 4, 2, 2}, dg[8] = {0, 0, 8, 8, 6, 5, 3, 2};  // by B
  static constexpr int value = DIM == 2 ? 8 : (TO_FV ? fv[B] : dg[B]);
};
// and those of the extrema
template <int DIM, int B, bool WALK>
struct LimMmMinB {
  static constexpr int walk[8] = {0, 0, 8, 8, 7, 3, 3, 3}, col[8] = {0, 0, 8, 8, 6, 5, 3, 2};
  static constexpr int value = WALK ? walk[B] : (DIM == 2 ? 8 : col[B]);
};

// Optional cell selection: the kernels run on cells list[0 .. *count) (at
// most ncells) instead of cells 0 .. ncells; a device-resident count lets a
// fixed launch sequence serve a selection that changes from step to step.
struct LimSel {
  const int* list = nullptr;
  const int* count = nullptr;
  __device__ __forceinline__ long cells(long ncells) const {
    return count ? min(ncells, (long)*count) : ncells;
  }
  __device__ __forceinline__ long cell(long k) const { return list ? (long)list[k] : k; }
};

// starts copying the selected cells' luh (n doubles each) to shared memory,
// every copy in flight at once (a load-store loop waited for each few); the
// caller waits (cp_async_commit_wait_all) and has a barrier
__device__ __forceinline__ void lim_stage_cells(double* dst, const double* __restrict__ src, int n, long c0, int nc,
                                                const LimSel& sel, int nt) {
  if (!sel.list) {
    for (int i = threadIdx.x; i < nc * n; i += nt) cp_async8(dst + i, src + c0 * n + i);
  } else {
    for (int i = threadIdx.x; i < nc * n; i += nt) {
      const int c = i / n;
      cp_async8(dst + i, src + sel.cell(c0 + c) * n + (i - c * n));
    }
  }
}

// ------------------------------------------------ few columns: passes
// The same operators as one pass per direction through shared memory: a
// column's sums are spread over threads that each own one line, so a cell's
// chain is short, at the price of a barrier and an intermediate array per pass.
// Faster than the register columns below while the columns are few (LimPassMax);
// the sums are the same in the same order, so a cell's values are the same bits.

template <int B>
struct LimOcc {
  // resident CTAs per SM the pass kernels are compiled for (register budget of
  // 64 / 85 / 255 per thread: the least that compiles without spills)
  static constexpr int value = B <= 4 ? 4 : (B == 5 ? 3 : 1);
};

// One 1D pass: applies table TAB (NI inputs -> NO outputs, T[p][m]) along
// direction D of a point array of extents EX x EY x EZ (x fastest), for
// `ncell` cells and variables v < nv.  Input point p of cell c starts at
// in + c * cs_in + p * ps_in.  Each thread takes (cell, line, variable)
// items, the variable fastest, starting with item (threadIdx.x - t0) mod NT
// (t0 lets a pass continue where the previous pass of the same phase left
// the threads); it hands the inputs and the NO outputs of its line to
// out.line<D>(c, x, y, z, v, inputs, outputs, item) with the D coordinate
// of (x, y, z) 0.  Strides and counts are plain ints: with the variable
// count a compile-time constant in the caller they fold into immediate
// offsets.
template <int TAB, int B, int EX, int EY, int EZ, int D, int NO, class Out>
__device__ __forceinline__ void lim_pass(const double* in, int ps_in, int cs_in, int ncell, int nv, Out& out,
                                         int t0 = 0) {
  constexpr int NI = D == 0 ? EX : (D == 1 ? EY : EZ);
  constexpr int LINES = EX * EY * EZ / NI;
  constexpr int SD = D == 0 ? 1 : (D == 1 ? EX : EX * EY);
  const int items = ncell * LINES * nv;
  for (int it = (threadIdx.x + kLimNT - t0 % kLimNT) % kLimNT; it < items; it += kLimNT) {
    const int v = it % nv;
    const int line = (it / nv) % LINES;
    const int c = it / (nv * LINES);
    int x = 0, y = 0, z = 0;
    if (D == 0) {
      y = line % EY;
      z = line / EY;
    } else if (D == 1) {
      x = line % EX;
      z = line / EX;
    } else {
      x = line % EX;
      y = line / EX;
    }
    const double* src = in + c * cs_in + ((z * EY + y) * EX + x) * ps_in + v;
    double a[NI];
#pragma unroll
    for (int p = 0; p < NI; p++) a[p] = src[p * SD * ps_in];
    double o[NO];
#pragma unroll
    for (int m = 0; m < NO; m++) {
      double acc = 0.0;
#pragma unroll
      for (int p = 0; p < NI; p++) acc = fma(lim_coef<TAB, B>(p, m), a[p], acc);
      o[m] = acc;
    }
    out.template line<D, NI, NO>(c, x, y, z, v, a, o, it);
  }
}

// writes a pass's outputs to a shared-memory array of extents ox x oy x .
struct SmemOut {
  double* base;
  int ps, cs, ox, oy;
  template <int D, int NI, int NO>
  __device__ __forceinline__ void line(int c, int x, int y, int z, int v, const double (&)[NI],
                                       const double (&o)[NO], int) {
    double* p = base + c * cs + ((z * oy + y) * ox + x) * ps + v;
    const int st = D == 0 ? ps : (D == 1 ? ox * ps : ox * oy * ps);
#pragma unroll
    for (int m = 0; m < NO; m++) p[m * st] = o[m];
  }
};

// writes to the interior of ghosted patches
template <int DIM>
struct PatchOut {
  double* base;  // cell 0 of the array
  long cs;       // doubles per cell
  int nvar, ext, ghost;
  long c0;       // first cell of the CTA
  template <int D, int NI, int NO>
  __device__ __forceinline__ void line(int c, int x, int y, int z, int v, const double (&)[NI],
                                       const double (&o)[NO], int) {
    const long pt = DIM == 3 ? ((long)(z + ghost) * ext + (y + ghost)) * ext + (x + ghost)
                             : (long)(y + ghost) * ext + (x + ghost);
    double* p = base + (c0 + c) * cs + pt * nvar + v;
    const long st = (D == 0 ? 1L : (D == 1 ? (long)ext : (long)ext * ext)) * nvar;
#pragma unroll
    for (int m = 0; m < NO; m++) p[m * st] = o[m];
  }
};

// extrema of the outputs of a line, stored per item
struct MinMaxOut {
  double* pmn;
  double* pmx;
  template <int D, int NI, int NO>
  __device__ __forceinline__ void line(int, int, int, int, int, const double (&)[NI], const double (&o)[NO],
                                       int it) {
    double mn = DBL_MAX, mx = -DBL_MAX;
#pragma unroll
    for (int m = 0; m < NO; m++) {
      mn = lim_min(mn, o[m]);
      mx = lim_max(mx, o[m]);
    }
    pmn[it] = mn;
    pmx[it] = mx;
  }
};

// a shared-memory store plus the extrema of the pass's INPUT line (the
// nodes themselves, seen by the first pass over luh)
struct SmemOutInputMinMax {
  SmemOut s;
  double* pmn;
  double* pmx;
  template <int D, int NI, int NO>
  __device__ __forceinline__ void line(int c, int x, int y, int z, int v, const double (&a)[NI],
                                       const double (&o)[NO], int it) {
    s.line<D, NI, NO>(c, x, y, z, v, a, o, it);
    double mn = DBL_MAX, mx = -DBL_MAX;
#pragma unroll
    for (int p = 0; p < NI; p++) {
      mn = lim_min(mn, a[p]);
      mx = lim_max(mx, a[p]);
    }
    pmn[it] = mn;
    pmx[it] = mx;
  }
};

// shared memory of a cell in k_lim_to_fv_pass (doubles per variable): luh,
// pass-x and pass-y results (3D)
template <int DIM, int B>
__host__ __device__ constexpr int lim_to_fv_pass_doubles() {
  return DIM == 3 ? B * B * B + B * B * (2 * B - 1) + B * (2 * B - 1) * (2 * B - 1) : B * B + B * (2 * B - 1);
}

// NVT: the variable count when known at compile time (0 = runtime nvar)
template <int DIM, int B, int NVT>
__global__ void __launch_bounds__(kLimNT, LimOcc<B>::value)
    k_lim_to_fv_pass(int nvar_rt, int ghost, long ncells, int cpb, const double* __restrict__ luh, double* lim) {
  constexpr int S = 2 * B - 1;
  constexpr int NPC = DIM == 3 ? B * B * B : B * B;
  const int nvar = NVT ? NVT : nvar_rt;
  extern __shared__ double sm[];
  const long c0 = (long)blockIdx.x * cpb;
  const int nc = (int)min((long)cpb, ncells - c0);
  const int SG = S + 2 * ghost;
  double* A = sm;
  double* T1 = A + cpb * NPC * nvar;
  lim_stage_cells(A, luh, NPC * nvar, c0, nc, LimSel(), kLimNT);
  cp_async_commit_wait_all();
  __syncthreads();
  PatchOut<DIM> go{lim, (long)nvar * (DIM == 3 ? SG * SG * SG : SG * SG), nvar, SG, ghost, c0};
  if (DIM == 2) {
    SmemOut o1{T1, nvar, S * B * nvar, S, B};
    lim_pass<kTabUh2Lim, B, B, B, 1, 0, S>(A, nvar, NPC * nvar, nc, nvar, o1);
    __syncthreads();
    lim_pass<kTabUh2Lim, B, S, B, 1, 1, S>(T1, nvar, S * B * nvar, nc, nvar, go);
  } else {
    double* T2 = T1 + cpb * B * B * S * nvar;
    SmemOut o1{T1, nvar, B * B * S * nvar, S, B};
    lim_pass<kTabUh2Lim, B, B, B, B, 0, S>(A, nvar, NPC * nvar, nc, nvar, o1);
    __syncthreads();
    SmemOut o2{T2, nvar, B * S * S * nvar, S, S};
    lim_pass<kTabUh2Lim, B, S, B, B, 1, S>(T1, nvar, B * B * S * nvar, nc, nvar, o2);
    __syncthreads();
    lim_pass<kTabUh2Lim, B, S, S, B, 2, S>(T2, nvar, B * S * S * nvar, nc, nvar, go);
  }
}

// Extrema and the DMP by passes.  The Gauss-Lobatto (B -> B) and subcell (B -> S) evaluations run side by
// side, pass by pass; the first pass also takes the extrema of the nodes
// (its input lines).  Per cell and observable, shared memory holds: the
// pass-x results of both (B^3 + B^2 S), the pass-y result of the subcells
// (B S^2) and of the Lobatto points (B^3, in the luh staging area, dead after
// pass x), and the per-line extrema of nodes, Lobatto points and subcells.
template <int DIM, int B>
struct LimMM {
  static constexpr int S = 2 * B - 1;
  static constexpr int NPC = DIM == 3 ? B * B * B : B * B;
  static constexpr int XL = DIM == 3 ? B * B * B : B * B;  // Lobatto pass-x result
  static constexpr int XS = DIM == 3 ? B * B * S : B * S;  // subcell pass-x result
  static constexpr int YS = DIM == 3 ? B * S * S : 0;      // subcell pass-y result
  static constexpr int NODE_LINES = DIM == 3 ? B * B : B;  // pass-x lines
  static constexpr int LOB_LINES = DIM == 3 ? B * B : B;   // final Lobatto lines
  static constexpr int SUB_LINES = DIM == 3 ? S * S : S;   // final subcell lines
  static constexpr int LINES = NODE_LINES + LOB_LINES + SUB_LINES;
  // doubles per cell
  __host__ __device__ static constexpr int doubles(int nvar, int nobs) {
    return NPC * nvar + (XL + XS + YS + 2 * LINES) * nobs;
  }
};

// (mode and arguments: k_lim_min_max)
template <int DIM, int B, int NVT>
__global__ void __launch_bounds__(kLimNT, LimOcc<B>::value)
    k_lim_min_max_pass(int mode, int nvar_rt, int nobs_rt, long ncells, int cpb, const double* __restrict__ luh, double relaxation,
                  double scaling, double* obs_min, double* obs_max, int* dmp_ok) {
  using M = LimMM<DIM, B>;
  constexpr int S = M::S, NPC = M::NPC, NF = 2 * DIM;
  const int nvar = NVT ? NVT : nvar_rt;
  const int nobs = NVT ? NVT : nobs_rt;
  extern __shared__ double sm[];
  const long c0 = (long)blockIdx.x * cpb;
  const int nc = (int)min((long)cpb, ncells - c0);
  double* A = sm;                         // luh, later the Lobatto pass-y result
  double* XL = A + cpb * NPC * nvar;      // [c][z][y][x][obs]
  double* XS = XL + cpb * M::XL * nobs;
  double* YS = XS + cpb * M::XS * nobs;
  double* pmn = YS + cpb * M::YS * nobs;  // [node | lob | sub lines]
  double* pmx = pmn + cpb * M::LINES * nobs;
  double* pn_mn = pmn;                    // node lines   [c][line][obs]
  double* pl_mn = pmn + cpb * M::NODE_LINES * nobs;
  double* ps_mn = pl_mn + cpb * M::LOB_LINES * nobs;
  double* pn_mx = pmx;
  double* pl_mx = pmx + cpb * M::NODE_LINES * nobs;
  double* ps_mx = pl_mx + cpb * M::LOB_LINES * nobs;
  if (mode == 1)
    for (int c = threadIdx.x; c < nc; c += kLimNT) dmp_ok[c0 + c] = 1;
  lim_stage_cells(A, luh, NPC * nvar, c0, nc, LimSel(), kLimNT);
  cp_async_commit_wait_all();
  __syncthreads();
  const int ix = nc * M::NODE_LINES * nobs;  // items of one pass-x
  if (DIM == 2) {
    SmemOutInputMinMax ol{{XL, nobs, B * B * nobs, B, B}, pn_mn, pn_mx};
    lim_pass<kTabUh2Lob, B, B, B, 1, 0, B>(A, nvar, NPC * nvar, nc, nobs, ol);
    SmemOut os{XS, nobs, S * B * nobs, S, B};
    lim_pass<kTabUh2Lim, B, B, B, 1, 0, S>(A, nvar, NPC * nvar, nc, nobs, os, ix);
    __syncthreads();
    MinMaxOut ml{pl_mn, pl_mx}, ms{ps_mn, ps_mx};
    lim_pass<kTabUh2Lob, B, B, B, 1, 1, B>(XL, nobs, B * B * nobs, nc, nobs, ml);
    lim_pass<kTabUh2Lim, B, S, B, 1, 1, S>(XS, nobs, S * B * nobs, nc, nobs, ms, nc * B * nobs);
  } else {
    SmemOutInputMinMax ol{{XL, nobs, B * B * B * nobs, B, B}, pn_mn, pn_mx};
    lim_pass<kTabUh2Lob, B, B, B, B, 0, B>(A, nvar, NPC * nvar, nc, nobs, ol);
    SmemOut os{XS, nobs, B * B * S * nobs, S, B};
    lim_pass<kTabUh2Lim, B, B, B, B, 0, S>(A, nvar, NPC * nvar, nc, nobs, os, ix);
    __syncthreads();
    double* YL = A;  // luh is dead after pass x
    SmemOut yl{YL, nobs, B * B * B * nobs, B, B};
    lim_pass<kTabUh2Lob, B, B, B, B, 1, B>(XL, nobs, B * B * B * nobs, nc, nobs, yl);
    SmemOut ys{YS, nobs, B * S * S * nobs, S, S};
    lim_pass<kTabUh2Lim, B, S, B, B, 1, S>(XS, nobs, B * B * S * nobs, nc, nobs, ys, nc * B * B * nobs);
    __syncthreads();
    MinMaxOut ml{pl_mn, pl_mx}, ms{ps_mn, ps_mx};
    lim_pass<kTabUh2Lob, B, B, B, B, 2, B>(YL, nobs, B * B * B * nobs, nc, nobs, ml);
    lim_pass<kTabUh2Lim, B, S, S, B, 2, S>(YS, nobs, B * S * S * nobs, nc, nobs, ms, nc * B * B * nobs);
  }
  __syncthreads();
  // per (cell, observable): the new extrema -> face blocks, and the DMP
  auto finish = [&](int pair, double mn, double mx) {
    const int c = pair / nobs, v = pair % nobs;
    double* bmn = obs_min + (c0 + c) * NF * nobs;
    double* bmx = obs_max + (c0 + c) * NF * nobs;
    if (mode == 0) {
      for (int f = 0; f < NF; f++) {
        bmn[f * nobs + v] = mn;
        bmx[f * nobs + v] = mx;
      }
    } else {
      double lo = bmn[v], hi = bmx[v];
      for (int f = 1; f < NF; f++) {
        lo = lim_min(lo, bmn[f * nobs + v]);
        hi = lim_max(hi, bmx[f * nobs + v]);
      }
      const double sd = lim_max((hi - lo) * scaling, relaxation);
      if (mn < lo - sd || mx > hi + sd) atomicAnd(dmp_ok + c0 + c, 0);
      bmn[v] = mn;
      bmx[v] = mx;
      bmn[v + nobs] = lo;
      bmx[v + nobs] = hi;
    }
  };
  auto line_index = [&](int c, int v, int l) {
    if (l < M::NODE_LINES) return (c * M::NODE_LINES + l) * nobs + v;
    if (l < M::NODE_LINES + M::LOB_LINES)
      return cpb * M::NODE_LINES * nobs + (c * M::LOB_LINES + l - M::NODE_LINES) * nobs + v;
    return cpb * (M::NODE_LINES + M::LOB_LINES) * nobs + (c * M::SUB_LINES + l - M::NODE_LINES - M::LOB_LINES) * nobs +
           v;
  };
  // reduction over the line extrema: a thread per pair when the pairs have
  // few lines (2D), a warp per pair otherwise
  if (M::LINES <= 32) {
    for (int pair = threadIdx.x; pair < nc * nobs; pair += kLimNT) {
      const int c = pair / nobs, v = pair % nobs;
      double mn = DBL_MAX, mx = -DBL_MAX;
#pragma unroll
      for (int l = 0; l < M::LINES; l++) {
        const int k = line_index(c, v, l);
        mn = lim_min(mn, pmn[k]);
        mx = lim_max(mx, pmx[k]);
      }
      finish(pair, mn, mx);
    }
  } else {
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    for (int pair = warp; pair < nc * nobs; pair += kLimNT / 32) {
      const int c = pair / nobs, v = pair % nobs;
      double mn = DBL_MAX, mx = -DBL_MAX;
      for (int l = lane; l < M::LINES; l += 32) {
        const int k = line_index(c, v, l);
        mn = lim_min(mn, pmn[k]);
        mx = lim_max(mx, pmx[k]);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        mn = lim_min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = lim_max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      }
      if (lane == 0) finish(pair, mn, mx);
    }
  }
}

// ------------------------------------------------------------ DG -> FV
// One thread per (cell, subcell column x, variable): the x sums of its
// column for every (z, y) in registers (B^2 doubles), then for every row of
// subcells the y sums and the z sums, stored as they are formed.  A CTA
// stages and serves cpb cells.  Bound by the stores (rows of S * nvar doubles
// that start and end inside a sector): ghosted patches (2 layers) leave at 2.3
// to 3 TB/s.  Per call, the passes through shared memory of before -> now:
// 24,000 3D cells of order 4 326 -> 313 us, 13,888 of order 5 555 -> 296, 8,746
// of order 6 551 -> 322, 166,666 2D cells of order 5 675 -> 334, 240,000 of
// order 4 405 -> 342; 3D orders 1 to 3 level (317 -> 320 at order 3).
template <int DIM, int B, int NVT>
__global__ void __launch_bounds__(kLimColNT, LimMinB<DIM, B, true>::value)
    k_lim_to_fv(int nvar_rt, int ghost, long ncells, int cpb, const double* __restrict__ luh, double* lim,
                LimSel sel) {
  constexpr int S = 2 * B - 1, BZ = DIM == 3 ? B : 1, SZ = DIM == 3 ? S : 1, NPC = BZ * B * B;
  const int nvar = NVT ? NVT : nvar_rt;
  const int SG = S + 2 * ghost;
  const long row = (long)SG * nvar, plane = row * SG;
  extern __shared__ double sm[];
  __shared__ double sT[S * B];  // means table, [subcell][node]
  for (int i = threadIdx.x; i < S * B; i += blockDim.x) sT[i] = c_lim[B - 1].uh2lim[i % B][i / B];
  const long nce = sel.cells(ncells);
  for (long c0 = (long)blockIdx.x * cpb; c0 < nce; c0 += (long)gridDim.x * cpb) {
    const int nc = (int)min((long)cpb, nce - c0);
    lim_stage_cells(sm, luh, NPC * nvar, c0, nc, sel, blockDim.x);
    cp_async_commit_wait_all();
    __syncthreads();
    for (int it = threadIdx.x; it < nc * S * nvar; it += blockDim.x) {
      const int v = it % nvar, x = (it / nvar) % S, c = it / (nvar * S);
      const double* src = sm + c * NPC * nvar + v;
      double cx[B];
#pragma unroll
      for (int p = 0; p < B; p++) cx[p] = sT[x * B + p];
      double a[BZ][B];
#pragma unroll
      for (int z = 0; z < BZ; z++)
#pragma unroll
        for (int y = 0; y < B; y++) {
          double acc = 0.0;
#pragma unroll
          for (int p = 0; p < B; p++) acc = fma(cx[p], src[((z * B + y) * B + p) * nvar], acc);
          a[z][y] = acc;
        }
      double* dst = lim + sel.cell(c0 + c) * (DIM == 3 ? plane * SG : plane) + (DIM == 3 ? ghost * plane : 0) +
                    ghost * row + (long)(ghost + x) * nvar + v;
      // (a loop, its coefficients in shared memory: unrolled, the y sums of
      // several rows live at once and spill)
#pragma unroll 1
      for (int y = 0; y < S; y++) {
        double b[BZ];
#pragma unroll
        for (int z = 0; z < BZ; z++) {
          double acc = 0.0;
#pragma unroll
          for (int p = 0; p < B; p++) acc = fma(sT[y * B + p], a[z][p], acc);
          b[z] = acc;
        }
        double* d = dst + y * row;
        if (DIM == 2) {
          d[0] = b[0];
        } else {
#pragma unroll
          for (int z = 0; z < SZ; z++) {
            double acc = 0.0;
#pragma unroll
            for (int p = 0; p < BZ; p++) acc = fma(c_lim[B - 1].uh2lim[p][z], b[p], acc);
            d[z * plane] = acc;
          }
        }
      }
    }
    __syncthreads();
  }
}

// interior subcells of nc ghosted patches -> shared [c][z][y][x][nvar]
// (rows of S * nvar contiguous doubles); each thread keeps four loads in
// flight before it stores them
template <int DIM, int S>
__device__ __forceinline__ void lim_stage_interior(double* A, const double* __restrict__ lim, long lim_cell, int nvar,
                                                   int ghost, long c0, int nc, const LimSel& sel) {
  const int SG = S + 2 * ghost;
  const int rowlen = S * nvar;
  constexpr int rows = DIM == 3 ? S * S : S;
  constexpr int U = 4;
  const int total = nc * rows * rowlen;
  for (int i0 = threadIdx.x; i0 < total; i0 += U * kLimNT) {
    double r[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int i = i0 + u * kLimNT;
      if (i < total) {
        const int k = i % rowlen;
        const int q = i / rowlen;
        const int row = q % rows;
        const int c = q / rows;
        const int yy = row % S, zz = row / S;
        const long p = DIM == 3 ? ((long)(zz + ghost) * SG + (yy + ghost)) * SG + ghost : (long)(yy + ghost) * SG + ghost;
        r[u] = __ldg(lim + sel.cell(c0 + c) * lim_cell + p * nvar + k);
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++)
      if (i0 + u * kLimNT < total) A[i0 + u * kLimNT] = r[u];
  }
}

// ------------------------------------------------------------ FV -> DG
// One thread per (cell, node column x, variable): plane by plane and row by
// row of the subcells, the row's x sum, added to the plane's y sums, and those
// to the column's B^2 results.  A CTA serves cpb cells; the planes of their
// subcells (the whole patch in 2D) pass through two shared buffers, the next
// plane's asynchronous copies in flight while this one is summed.  A plane is
// copied as it lies, from its first interior value to its last: the ghost
// values between the rows cost less than finding the rows -- except at order 1,
// where two ghost layers are more than half of it (375,000 3D cells: 328 us with
// them, 171 without).  Bound by the latency of the planes' loads at 12 to 20
// warps per SM.  Per call before -> now: 3D order 4 (24,000 cells) 344 -> 272 us,
// order 5 (13,888) 817 -> 283, 2D order 3 (375,000) 304 -> 260, order 5
// (166,666) 798 -> 347.
// FLAT: a plane has fewer values than the CTA has threads, which then share the
// planes of all cells (40,000 3D cells of order 3 with one variable 62 us, cell
// by cell 90).
template <int DIM, int B, int NVT, bool FLAT>
__global__ void __launch_bounds__(kLimColNT, LimMinB<DIM, B, false>::value)
    k_lim_to_dg(int nvar_rt, int ghost, long ncells, int cpb, const double* __restrict__ lim, double* luh,
                LimSel sel) {
  constexpr int S = 2 * B - 1, BZ = DIM == 3 ? B : 1, SZ = DIM == 3 ? S : 1;
  constexpr bool kRows = B <= 2;  // rows without the ghost values between them
  const int nvar = NVT ? NVT : nvar_rt;
  const int SG = S + 2 * ghost;
  const long row = (long)SG * nvar, plane = row * SG;
  const int irow = (kRows ? S : SG) * nvar, len = (S - 1) * irow + S * nvar, buf = cpb * len;  // a staged plane
  extern __shared__ double sm[];
  const long nce = sel.cells(ncells);
  for (long c0 = (long)blockIdx.x * cpb; c0 < nce; c0 += (long)gridDim.x * cpb) {
    const int nc = (int)min((long)cpb, nce - c0);
    auto stage = [&](int z) {
      double* d = sm + (z & 1) * buf;
      auto cell_plane = [&](int c) {
        return lim + sel.cell(c0 + c) * (DIM == 3 ? plane * SG : plane) + (DIM == 3 ? (z + ghost) * plane : 0) +
               ghost * row + (long)ghost * nvar;
      };
      if (FLAT) {
        for (int i = threadIdx.x; i < nc * len; i += kLimColNT) {
          const int c = i / len, k = i - c * len;
          cp_async8(d + i, cell_plane(c) + (kRows ? k + k / (S * nvar) * 2 * ghost * nvar : k));
        }
      } else {
        for (int c = 0; c < nc; c++) {
          const double* src = cell_plane(c);
          if (kRows) {
            for (int k = threadIdx.x; k < len; k += kLimColNT)
              cp_async8(d + c * len + k, src + k + k / (S * nvar) * 2 * ghost * nvar);
          } else {
            for (int k = threadIdx.x; k < len; k += kLimColNT) cp_async8(d + c * len + k, src + k);
          }
        }
      }
      cp_async_commit();
    };
    // this thread's first column; the rare further ones (more columns than
    // threads) run after it over the same planes
    for (int it0 = 0; it0 < nc * B * nvar; it0 += kLimColNT) {
      const int it = it0 + threadIdx.x;
      const bool on = it < nc * B * nvar;
      const int v = on ? it % nvar : 0, x = on ? (it / nvar) % B : 0, c = on ? it / (nvar * B) : 0;
      double cx[S];
#pragma unroll
      for (int p = 0; p < S; p++) cx[p] = c_lim[B - 1].lim2uh[p][x];
      double o[BZ][B];
#pragma unroll
      for (int z = 0; z < BZ; z++)
#pragma unroll
        for (int y = 0; y < B; y++) o[z][y] = 0.0;
      stage(0);
#pragma unroll 1
      for (int z = 0; z < SZ; z++) {
        if (z + 1 < SZ) {
          stage(z + 1);
          cp_async_wait<1>();
        } else {
          cp_async_wait<0>();
        }
        __syncthreads();
        const double* src = sm + (z & 1) * buf + c * len + v;
        double b[B];
#pragma unroll
        for (int y = 0; y < B; y++) b[y] = 0.0;
#pragma unroll
        for (int y = 0; y < S; y++) {
          double acc = 0.0;
#pragma unroll
          for (int p = 0; p < S; p++) acc = fma(cx[p], src[y * irow + p * nvar], acc);
#pragma unroll
          for (int m = 0; m < B; m++) b[m] = fma(c_lim[B - 1].lim2uh[y][m], acc, b[m]);
        }
        if (DIM == 2) {
#pragma unroll
          for (int m = 0; m < B; m++) o[0][m] = b[m];
        } else {
#pragma unroll
          for (int n = 0; n < BZ; n++)
#pragma unroll
            for (int m = 0; m < B; m++) o[n][m] = fma(c_lim[B - 1].lim2uh[z][n], b[m], o[n][m]);
        }
        __syncthreads();  // the buffer is free for plane z + 2
      }
      if (on) {
        double* dst = luh + sel.cell(c0 + c) * (long)(BZ * B * B * nvar) + (long)x * nvar + v;
#pragma unroll
        for (int z = 0; z < BZ; z++)
#pragma unroll
          for (int y = 0; y < B; y++) dst[(z * B + y) * B * nvar] = o[z][y];
      }
    }
  }
}

// The same for few 3D cells, one per CTA: plane after plane, a cell's column
// waits for memory S times and its sums are one thread's.  Here the whole patch
// is copied at once, one thread per (plane, node column, variable) forms the
// plane's sums and one per (node row, node column, variable) the z sums, each
// in the order above.  Order 4: 300 cells 24.6 us in the form above, 13.3 here
// (14.3 before both), 4,000 cells 73 and 57 (67).
template <int B, int NVT>
__global__ void __launch_bounds__(kLimNT) k_lim_to_dg_few(int nvar_rt, int ghost, long ncells,
                                                          const double* __restrict__ lim, double* luh) {
  constexpr int S = 2 * B - 1;
  const int nvar = NVT ? NVT : nvar_rt;
  const int SG = S + 2 * ghost, irow = SG * nvar, len = (S - 1) * irow + S * nvar;
  const long plane = (long)SG * irow;
  extern __shared__ double sm[];
  double* sb = sm + S * len;  // plane sums [z][y][x][nvar]
  const long c = blockIdx.x;
  for (int z = 0; z < S; z++) {
    const double* src = lim + c * plane * SG + (z + ghost) * plane + ghost * (irow + nvar);
    for (int k = threadIdx.x; k < len; k += kLimNT) cp_async8(sm + z * len + k, src + k);
  }
  cp_async_commit_wait_all();
  __syncthreads();
  for (int it = threadIdx.x; it < S * B * nvar; it += kLimNT) {
    const int v = it % nvar, x = (it / nvar) % B, z = it / (nvar * B);
    const double* src = sm + z * len + v;
    double b[B];
#pragma unroll
    for (int m = 0; m < B; m++) b[m] = 0.0;
#pragma unroll
    for (int y = 0; y < S; y++) {
      double acc = 0.0;
#pragma unroll
      for (int p = 0; p < S; p++) acc = fma(c_lim[B - 1].lim2uh[p][x], src[y * irow + p * nvar], acc);
#pragma unroll
      for (int m = 0; m < B; m++) b[m] = fma(c_lim[B - 1].lim2uh[y][m], acc, b[m]);
    }
#pragma unroll
    for (int m = 0; m < B; m++) sb[((z * B + m) * B + x) * nvar + v] = b[m];
  }
  __syncthreads();
  for (int it = threadIdx.x; it < B * B * nvar; it += kLimNT) {
    double o[B];
#pragma unroll
    for (int n = 0; n < B; n++) o[n] = 0.0;
#pragma unroll
    for (int z = 0; z < S; z++)
#pragma unroll
      for (int n = 0; n < B; n++) o[n] = fma(c_lim[B - 1].lim2uh[z][n], sb[z * B * B * nvar + it], o[n]);
#pragma unroll
    for (int n = 0; n < B; n++) luh[(c * B + n) * B * B * nvar + it] = o[n];
  }
}

// ------------------------------------------------ min/max and the DMP
// One thread per (cell, column, observable): S columns of subcells and B
// columns of Gauss-Lobatto points (which also take the node column of the
// same x), each evaluated as in k_lim_to_fv but only its extrema kept; then
// one thread per (cell, observable) reduces the S + B columns and finishes.
// WALK (2D): a column is too little work for its place in the reduction; one
// thread per (cell, observable) keeps the cell's B^2 values in registers and
// walks the columns.  A CTA holds cpb cells, for WALK staged at a pitch that
// puts the lanes' (cell, observable) values in consecutive banks.
// Bound by FP64 issue and, in 2D, by memory.  Per DMP call, passes through
// shared memory before -> now: 3D order 4 (24,000 cells) 263 -> 135 us, order 3
// (46,875) 256 -> 110, order 2 (111,111) 339 -> 99; 2D order 3 (375,000) 224 ->
// 120, order 1 (1,500,000) 374 -> 163.
//
// extrema over all points of a 2D cell evaluated with table TAB (NO per direction)
template <int B, int TAB, int NO>
__device__ __forceinline__ void lim_cell_extrema(const double (&q)[B][B], double& mn, double& mx) {
#pragma unroll 1
  for (int x = 0; x < NO; x++) {
    double a[B];
#pragma unroll
    for (int y = 0; y < B; y++) {
      double acc = 0.0;
#pragma unroll
      for (int p = 0; p < B; p++) acc = fma(lim_coef<TAB, B>(p, x), q[y][p], acc);
      a[y] = acc;
    }
#pragma unroll
    for (int y = 0; y < NO; y++) {
      double acc = 0.0;
#pragma unroll
      for (int p = 0; p < B; p++) acc = fma(lim_coef<TAB, B>(p, y), a[p], acc);
      mn = lim_min(mn, acc);
      mx = lim_max(mx, acc);
    }
  }
}

// extrema of a column evaluated with table TAB (NO points per direction)
template <int DIM, int B, int TAB, int NO>
__device__ __forceinline__ void lim_column_extrema(const double* src, int nvar, int x, double& mn, double& mx) {
  constexpr int BZ = DIM == 3 ? B : 1;
  double cx[B];
#pragma unroll
  for (int p = 0; p < B; p++) cx[p] = lim_coef<TAB, B>(p, x);
  double a[BZ][B];
#pragma unroll
  for (int z = 0; z < BZ; z++)
#pragma unroll
    for (int y = 0; y < B; y++) {
      double acc = 0.0;
#pragma unroll
      for (int p = 0; p < B; p++) acc = fma(cx[p], src[((z * B + y) * B + p) * nvar], acc);
      a[z][y] = acc;
    }
#pragma unroll 1
  for (int y = 0; y < NO; y++) {
    double b[BZ];
#pragma unroll
    for (int z = 0; z < BZ; z++) {
      double acc = 0.0;
#pragma unroll
      for (int p = 0; p < B; p++) acc = fma(lim_coef<TAB, B>(p, y), a[z][p], acc);
      b[z] = acc;
    }
    if (DIM == 2) {
      mn = lim_min(mn, b[0]);
      mx = lim_max(mx, b[0]);
    } else {
#pragma unroll
      for (int z = 0; z < NO; z++) {
        double acc = 0.0;
#pragma unroll
        for (int p = 0; p < BZ; p++) acc = fma(lim_coef<TAB, B>(p, z), b[p], acc);
        mn = lim_min(mn, acc);
        mx = lim_max(mx, acc);
      }
    }
  }
}

// doubles from one staged cell of k_lim_min_max to the next
template <int DIM, int B, bool WALK>
__host__ __device__ __forceinline__ int lim_pitch(int nvar) {
  const int n = (DIM == 3 ? B * B * B : B * B) * nvar;
  return !WALK ? n : n + ((nvar - n) % 16 + 16) % 16;
}

// mode 0: findCellLocalMinAndMax, result copied to all faces;
// mode 1: discreteMaximumPrincipleAndMinAndMaxSearch (obs_min/max in/out,
//         dmp_ok[cell] = 1 if the DMP holds).
template <int DIM, int B, int NVT, bool WALK>
__global__ void __launch_bounds__(kLimMmNT, LimMmMinB<DIM, B, WALK>::value)
    k_lim_min_max(int mode, int nvar_rt, int nobs_rt, long ncells, int cpb, const double* __restrict__ luh,
                  double relaxation, double scaling, double* obs_min, double* obs_max, int* dmp_ok) {
  constexpr int S = 2 * B - 1, NPC = DIM == 3 ? B * B * B : B * B, NF = 2 * DIM, COLS = S + B;
  const int nvar = NVT ? NVT : nvar_rt;
  const int nobs = NVT ? NVT : nobs_rt;
  extern __shared__ double sm[];
  const long c0 = (long)blockIdx.x * cpb;
  const int nc = (int)min((long)cpb, ncells - c0);
  const int pitch = lim_pitch<DIM, B, WALK>(nvar);
  double* sluh = sm;                // [cell][node][nvar]
  double* pmn = sm + cpb * pitch;   // !WALK: [cell][obs][column]
  double* pmx = pmn + cpb * nobs * COLS;
  if (mode == 1)
    for (int c = threadIdx.x; c < nc; c += kLimMmNT) dmp_ok[c0 + c] = 1;
  if (WALK) {
    const int n = NPC * nvar;
    for (int i = threadIdx.x; i < nc * n; i += kLimMmNT) cp_async8(sluh + i + i / n * (pitch - n), luh + c0 * n + i);
  } else {
    lim_stage_cells(sluh, luh, NPC * nvar, c0, nc, LimSel(), kLimMmNT);
  }
  // the bounds of this thread's (cell, observable), needed at the end
  double lo0 = 0.0, hi0 = 0.0;
  if (mode == 1 && threadIdx.x < nc * nobs) {
    const int c = threadIdx.x / nobs, v = threadIdx.x % nobs;
    const double* bmn = obs_min + (c0 + c) * NF * nobs + v;
    const double* bmx = obs_max + (c0 + c) * NF * nobs + v;
    lo0 = bmn[0];
    hi0 = bmx[0];
#pragma unroll
    for (int f = 1; f < NF; f++) {
      lo0 = lim_min(lo0, bmn[f * nobs]);
      hi0 = lim_max(hi0, bmx[f * nobs]);
    }
  }
  cp_async_commit_wait_all();
  __syncthreads();
  // the subcell columns of every cell first, then the Lobatto columns: few
  // warps hold both kinds
  const int nsub = nc * S * nobs, total = WALK ? 0 : nc * COLS * nobs;
  for (int it = threadIdx.x; it < total; it += kLimMmNT) {
    const bool sub = it < nsub;
    const int n = sub ? S : B, i = sub ? it : it - nsub;
    const int v = i % nobs, x = (i / nobs) % n, c = i / (nobs * n);
    const double* src = sluh + c * NPC * nvar + v;
    double mn = DBL_MAX, mx = -DBL_MAX;
    if (sub) {
      lim_column_extrema<DIM, B, kTabUh2Lim, S>(src, nvar, x, mn, mx);
    } else {
#pragma unroll
      for (int k = 0; k < NPC / B; k++) {
        const double q = src[(k * B + x) * nvar];
        mn = lim_min(mn, q);
        mx = lim_max(mx, q);
      }
      lim_column_extrema<DIM, B, kTabUh2Lob, B>(src, nvar, x, mn, mx);
    }
    const int slot = (c * nobs + v) * COLS + (sub ? x : S + x);
    pmn[slot] = mn;
    pmx[slot] = mx;
  }
  if (!WALK) __syncthreads();
  for (int pair = threadIdx.x; pair < nc * nobs; pair += kLimMmNT) {
    const int c = pair / nobs, v = pair % nobs;
    double mn = DBL_MAX, mx = -DBL_MAX;
    if constexpr (!WALK) {
#pragma unroll
      for (int l = 0; l < COLS; l++) {
        mn = lim_min(mn, pmn[pair * COLS + l]);
        mx = lim_max(mx, pmx[pair * COLS + l]);
      }
    } else {
      double q[B][B];
#pragma unroll
      for (int y = 0; y < B; y++)
#pragma unroll
        for (int x = 0; x < B; x++) {
          q[y][x] = sluh[c * pitch + (y * B + x) * nvar + v];
          mn = lim_min(mn, q[y][x]);
          mx = lim_max(mx, q[y][x]);
        }
      lim_cell_extrema<B, kTabUh2Lob, B>(q, mn, mx);
      lim_cell_extrema<B, kTabUh2Lim, S>(q, mn, mx);
    }
    // the new extrema -> face blocks, and the DMP
    double* bmn = obs_min + (c0 + c) * NF * nobs;
    double* bmx = obs_max + (c0 + c) * NF * nobs;
    if (mode == 0) {
      for (int f = 0; f < NF; f++) {
        bmn[f * nobs + v] = mn;
        bmx[f * nobs + v] = mx;
      }
    } else {
      double lo = lo0, hi = hi0;
      if (pair != threadIdx.x) {
        lo = bmn[v];
        hi = bmx[v];
        for (int f = 1; f < NF; f++) {
          lo = lim_min(lo, bmn[f * nobs + v]);
          hi = lim_max(hi, bmx[f * nobs + v]);
        }
      }
      const double sd = lim_max((hi - lo) * scaling, relaxation);
      if (mn < lo - sd || mx > hi + sd) atomicAnd(dmp_ok + c0 + c, 0);
      bmn[v] = mn;
      bmx[v] = mx;
      bmn[v + nobs] = lo;
      bmx[v + nobs] = hi;
    }
  }
}

// findCellLocalLimiterMinAndMax: extrema over the staged interior subcells,
// one warp per (cell, observable), written to every face block
template <int DIM, int B>
__global__ void __launch_bounds__(kLimNT) k_lim_fv_min_max(int nvar, int nobs, int ghost, long ncells, int cpb,
                                                           const double* lim, double* obs_min, double* obs_max,
                                                           LimSel sel) {
  constexpr int S = 2 * B - 1;
  constexpr int NS = DIM == 3 ? S * S * S : S * S;
  extern __shared__ double sm[];
  const long nce = sel.cells(ncells);
  // one cell block per iteration (a single one unless a selection launched
  // fewer CTAs than blocks)
  for (long c0 = (long)blockIdx.x * cpb; c0 < nce; c0 += (long)gridDim.x * cpb) {
    const int nc = (int)min((long)cpb, nce - c0);
    const int SG = S + 2 * ghost;
    const long lim_cell = (long)nvar * (DIM == 3 ? SG * SG * SG : SG * SG);
    lim_stage_interior<DIM, S>(sm, lim, lim_cell, nvar, ghost, c0, nc, sel);
    __syncthreads();
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    for (int pair = warp; pair < nc * nobs; pair += kLimNT / 32) {
      const int c = pair / nobs, v = pair % nobs;
      double mn = DBL_MAX, mx = -DBL_MAX;
      for (int p = lane; p < NS; p += 32) {
        const double q = sm[((long)c * NS + p) * nvar + v];
        mn = lim_min(mn, q);
        mx = lim_max(mx, q);
      }
  #pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        mn = lim_min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = lim_max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      }
      if (lane == 0)
        for (int f = 0; f < 2 * DIM; f++) {
          obs_min[(sel.cell(c0 + c) * 2 * DIM + f) * nobs + v] = mn;
          obs_max[(sel.cell(c0 + c) * 2 * DIM + f) * nobs + v] = mx;
        }
    }
    __syncthreads();
  }
}

// Columns (subcell columns x variables; for the extrema subcell and Lobatto
// columns x observables) of a call up to which it takes the passes, by B: the
// largest calls that measured faster there.  With five variables / observables
// and with any other number.  us per call, passes and columns: one 3D cell of
// order 4, DG -> FV 3.8 / 4.7, DMP 4.8 / 6.2, of order 6 7.8 / 9.4 and 8.4 / 11.3,
// one 2D cell of order 3 2.4 / 3.3 and 3.1 / 4.3; 100 3D cells of order 5, DMP
// 6.3 / 8.8; 5,000 2D cells of order 4, DMP 7.1 / 9.0; 300 3D cells of order 6
// with one variable, DG -> FV 7.9 / 19, extrema 8.9 / 23.
template <int DIM, bool FIVE>
struct LimPassMax {
  static constexpr long fv2[2][8] = {{0, 0, 90, 135, 1008000, 180, 198, 156}, {0, 0, 150, 250, 700000, 135, 165, 65}};
  static constexpr long fv3[2][8] = {{0, 0, 0, 30, 63, 360000, 44, 11700}, {0, 0, 45, 25, 28000, 45, 5500, 6500}};
  static constexpr long mm2[2][8] = {{0, 0, 0, 216, 13200, 280, 306, 240}, {0, 0, 0, 400, 110000, 840000, 255, 300}};
  static constexpr long mm3[2][8] = {{0, 0, 0, 0, 66, 11200, 13600, 320000}, {0, 0, 0, 40, 55, 84000, 102000, 30000}};
  static constexpr long fv(int B) { return DIM == 2 ? fv2[FIVE][B] : fv3[FIVE][B]; }
  static constexpr long mm(int B) { return DIM == 2 ? mm2[FIVE][B] : mm3[FIVE][B]; }
};

// cells per CTA of the passes: enough items for two rounds of the final pass,
// within a shared-memory budget that leaves room for `occ` resident CTAs per SM
static int lim_pass_cpb(long items_per_cell, long smem_per_cell, long ncells, int occ) {
  long cpb = (2 * kLimNT + items_per_cell - 1) / items_per_cell;
  const long cap = (220L * 1024 / occ) / smem_per_cell;
  cpb = min(cpb, min(64L, min(cap, ncells)));
  return (int)(cpb < 1 ? 1 : cpb);
}

// cells per CTA: the count whose items fill their rounds of nt threads best,
// within a shared-memory budget and up to 16 or one round's cells; no more than
// leave every SM four CTAs, but at least what lets all CTAs be resident at once
// (`occ` per SM) where that takes a few cells and no further round or, for the
// extrema, saves a wave that would be nearly empty: 1,200 3D cells of order 6, one
// observable, 17.5 us with six cells per CTA, 36 with one; 1,200 2D cells of
// order 5 5.5 and 7.0.  `latency`: share of a round that a CTA waits before its
// first one; more rounds share it (extrema of 12,000 2D cells of order 6, three
// observables: 23 us with eight cells, 28 with two).
static int lim_cpb(long items_per_cell, long smem_per_cell, long ncells, int nt, long budget, int sms, int occ,
                   bool extrema, double latency) {
  int best = 1;
  double fill = 0.0;
  const long round = nt / items_per_cell, most = round > 16 ? round : 16, spread = ncells / (4 * sms);
  for (int c = 1; c <= most && (c == 1 || (c * smem_per_cell <= budget && c <= spread)); c++) {
    const long items = c * items_per_cell, rounds = (items + nt - 1) / nt;
    const double f = (double)items / (double)(rounds * nt) * (1.0 - latency / (double)rounds);
    if (f > fill + 0.02) best = c, fill = f;
  }
  const long slots = (long)occ * sms, once = (ncells + slots - 1) / slots;
  if (once > best && once <= 8 && once * smem_per_cell * occ <= 220L * 1024) {
    const long rounds = (once * items_per_cell + nt - 1) / nt, rounds1 = (items_per_cell + nt - 1) / nt;
    if (rounds <= rounds1 || (extrema && rounds <= once * rounds1 && 2 * once * slots > 3 * ncells))
      best = (int)once;
  }
  return best;
}

template <int DIM, int B, int NVT>
static exa_status_t lim_run(int op, int nvar, int nobs, int ghost, long ncells, const double* in, double* out,
                            double* mn, double* mx, int* ok, double relax, double scaling, cudaStream_t st,
                            LimSel sel) {
  constexpr int S = 2 * B - 1, COLS = S + B;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // The entry points take cells whose 1D passes' arrays fit one CTA's shared
  // memory (doubles per variable or observable below).
  constexpr long P = DIM == 3 ? B * B * B : B * B, Q = DIM == 3 ? S * S * S : S * S;
  constexpr long fv_pass = DIM == 3 ? P + B * B * S + B * S * S : P + B * S;
  constexpr long dg_pass = DIM == 3 ? Q + S * S * B : Q + S * B;
  constexpr long mm_lines = DIM == 3 ? 2 * B * B + S * S : 2 * B + S;
  constexpr long mm_pass = DIM == 3 ? P + B * B * S + B * S * S + 2 * mm_lines : P + B * S + 2 * mm_lines;
  const long limit = op == kLimToFv ? fv_pass * nvar
                                    : (op == kLimToDg ? dg_pass * nvar
                                                      : (op == kLimFvMinMax ? Q * nvar : P * nvar + mm_pass * nobs));
  if (limit * (long)sizeof(double) > kLimMaxSmem)
    return set_error(EXA_EINVAL, "limiter: cell too large for shared memory");
  constexpr long NPC = P, D8 = (long)sizeof(double);
  const int cpb_set = tune_get(kTuneLimiterCellsPerCta, 0);
  const bool mm = op == kLimMinMax || op == kLimDmp;
  // (3D calls whose columns just fill one wave, one cell per CTA, are level with
  // the passes and ahead of them when their cells are not in L2)
  const long wave = (long)LimMmMinB<DIM, B, false>::value * sms;
  const bool full_wave = DIM == 3 && ncells <= wave && 20 * ncells > 17 * wave;
  if ((op == kLimToFv && !sel.list && ncells * S * nvar <= LimPassMax<DIM, NVT == 5>::fv(B)) ||
      (mm && !full_wave && ncells * COLS * nobs <= LimPassMax<DIM, NVT == 5>::mm(B))) {
    const long lines = DIM == 3 ? S * S : S;  // of the final pass
    const long per_cell = D8 * (mm ? LimMM<DIM, B>::doubles(nvar, nobs) : lim_to_fv_pass_doubles<DIM, B>() * nvar);
    int cpb = lim_pass_cpb(lines * (mm ? nobs : nvar), per_cell, ncells, LimOcc<B>::value);
    if (cpb_set > 0 && (long)cpb_set * per_cell <= kLimMaxSmem) cpb = cpb_set;
    const unsigned nblk = (unsigned)((ncells + cpb - 1) / cpb);
    cudaError_t e = mm ? allow_max_smem(k_lim_min_max_pass<DIM, B, NVT>) : allow_max_smem(k_lim_to_fv_pass<DIM, B, NVT>);
    if (e != cudaSuccess) return cuda_status(e, "limiter: shared-memory attribute");
    if (mm)
      k_lim_min_max_pass<DIM, B, NVT><<<nblk, kLimNT, (size_t)cpb * per_cell, st>>>(
          op == kLimDmp ? 1 : 0, nvar, nobs, ncells, cpb, in, relax, scaling, mn, mx, ok);
    else
      k_lim_to_fv_pass<DIM, B, NVT><<<nblk, kLimNT, (size_t)cpb * per_cell, st>>>(nvar, ghost, ncells, cpb, in, out);
    count_launch();
    return cuda_status(cudaGetLastError(), "limiter pass kernel");
  }
  if (op == kLimToFv || op == kLimToDg) {
    const bool fv = op == kLimToFv;
    // one column per thread of the last cell's end at most: FV -> DG walks its
    // planes once per round of columns
    const long plane = (long)(S - 1) * (S + 2 * ghost) + S;  // values of a variable in a staged plane
    const long per_cell = D8 * (fv ? NPC * nvar : (DIM == 3 ? 2 : 1) * plane * nvar);
    const long items = (long)(fv ? S : B) * nvar;
    int cpb;
    int nt = kLimColNT;
    if (fv) {
      cpb = lim_cpb(items, per_cell, ncells, kLimColNT, 44 * 1024, sms, LimMinB<DIM, B, true>::value, false, 0.0);
      if (DIM == 3) {
        // one round of columns if they fill whole warps well (order 4, 24,000
        // cells: 313 us, three rounds 348; order 6, a third of its lanes idle:
        // 394, several rounds 322; in 2D rounds are as good or better)
        const long spread = ncells / (4 * sms);
        double fill = 0.8;
        for (int c = 1; c * items <= kLimColNT && (c == 1 || c <= spread); c++) {
          const int t = (int)((c * items + 31) / 32 * 32);
          const double f = (double)(c * items) / (double)t;
          if (f >= fill) cpb = c, fill = f, nt = t;
        }
      }
    } else {
      // a round of columns, but two CTAs for every SM in 3D, four in 2D where
      // they then hold four cells (with four and single cells, few cells of few
      // variables waited longer for memory: 3,000 3D cells of order 4, one
      // variable, 24 us, 38 before; 1,000 2D cells of order 3 3.8 and 4.2)
      const long two = (ncells + 2 * sms - 1) / (2 * sms);
      const long spread = DIM == 3 ? two : max(ncells / (4 * sms), min(two, 4L));
      cpb = (int)(kLimColNT / items > 0 ? kLimColNT / items : 1);
      if (cpb > spread) cpb = (int)spread;
      while (cpb > 1 && cpb * per_cell > 72 * 1024) cpb--;
      if constexpr (DIM == 3) {
        const long few = D8 * (S * plane + (long)S * B * B) * nvar;
        // all planes of a cell at once up to ten patches' worth of the chip's
        // shared memory (five variables, order 4: 6,000 cells; beyond, the
        // streamed planes are level or better), and fewer where a cell's (plane,
        // column, variable) items leave three quarters of the CTA idle (order 1,
        // five variables, 40,000 cells: 45 us, streamed 19; order 2, one variable:
        // 88 and 28) and at the highest orders (order 6, one variable, 3,000
        // cells: 95 and 46; order 5, five variables: 81 and 74)
        const long work = (long)S * B * nvar;
        long most = 10L * kLimMaxSmem / few;  // cells per SM
        if (work < 64) most = min(most, max(8L, 7 * work / 10));
        if (B >= 6) most = min(most, B == 6 ? 12L : 6L);
        if (!cpb_set && !sel.list && few <= kLimMaxSmem && ncells <= most * sms) {
          cudaError_t e = allow_max_smem(k_lim_to_dg_few<B, NVT>);
          if (e != cudaSuccess) return cuda_status(e, "limiter: shared-memory attribute");
          k_lim_to_dg_few<B, NVT><<<(unsigned)ncells, kLimNT, (size_t)few, st>>>(nvar, ghost, ncells, in, out);
          count_launch();
          return cuda_status(cudaGetLastError(), "limiter projection");
        }
      }
    }
    if (per_cell > kLimMaxSmem) return set_error(EXA_EINVAL, "limiter: cell too large for shared memory");
    if (cpb_set > 0 && (long)cpb_set * per_cell <= kLimMaxSmem) cpb = cpb_set;
    const size_t smem = (size_t)cpb * per_cell;
    long nblk = (ncells + cpb - 1) / cpb;
    if (sel.count) nblk = nblk < 8L * sms ? nblk : 8L * sms;  // a selection usually holds a few cells: CTAs loop
    if (nblk > 0x7fffffffL) return set_error(EXA_EINVAL, "limiter: too many cells");
    const bool flat = (B <= 2 ? (long)S * S : plane) * nvar < kLimColNT;
    auto to_dg = flat ? k_lim_to_dg<DIM, B, NVT, true> : k_lim_to_dg<DIM, B, NVT, false>;
    cudaError_t e = fv ? allow_max_smem(k_lim_to_fv<DIM, B, NVT>) : allow_max_smem(to_dg);
    if (e != cudaSuccess) return cuda_status(e, "limiter: shared-memory attribute");
    if (fv)
      k_lim_to_fv<DIM, B, NVT><<<(unsigned)nblk, nt, smem, st>>>(nvar, ghost, ncells, cpb, in, out, sel);
    else
      to_dg<<<(unsigned)nblk, kLimColNT, smem, st>>>(nvar, ghost, ncells, cpb, in, out, sel);
    count_launch();
    return cuda_status(cudaGetLastError(), "limiter projection");
  }
  long per_cell;
  int cpb;
  // Extrema of a whole 2D cell in one thread: while its work is short (order 3,
  // 375,000 cells: 120 us, by columns 240), or from four warps of such threads
  // per scheduler on (order 4, 240,000 cells: 160, 231 by columns; but 1,000
  // cells: 17, 10 by columns).  Order 6 is faster by columns throughout (264, 294).
  const bool walk = DIM == 2 && (B <= 4 || (B <= 6 && ncells * nobs >= 512L * sms));
  if (op == kLimFvMinMax) {
    per_cell = (long)(DIM == 3 ? S * S * S : S * S) * nvar * (long)sizeof(double);
    // a warp per (cell, observable), two rounds of them, three CTAs per SM (four
    // up to order 3: 100 3D cells with five of twelve variables 8 us, 13 with three)
    const long want = (16 + nobs - 1) / nobs, cap = (B <= 4 ? 55L : 73L) * 1024 / per_cell;
    cpb = (int)(want < cap ? want : (cap < 1 ? 1 : cap));
    if (cpb > ncells) cpb = (int)ncells;
  } else {
    per_cell = D8 * (walk ? lim_pitch<DIM, B, true>(nvar) : NPC * nvar + 2L * COLS * nobs);
    cpb = lim_cpb((walk ? 1L : (long)COLS) * nobs, per_cell, ncells, kLimMmNT, 36 * 1024, sms,
                  walk ? LimMmMinB<DIM, B, true>::value : LimMmMinB<DIM, B, false>::value, true, NVT ? 0.0 : 0.25);
  }
  if (cpb_set > 0 && (long)cpb_set * per_cell <= kLimMaxSmem) cpb = cpb_set;
  const size_t smem = (size_t)cpb * per_cell;
  long nblk = (ncells + cpb - 1) / cpb;
  if (sel.count) nblk = nblk < 4L * sms ? nblk : 4L * sms;
  if (nblk > 0x7fffffffL) return set_error(EXA_EINVAL, "limiter: too many cells");
  cudaError_t e = cudaSuccess;
  if (op == kLimFvMinMax) {
    e = allow_max_smem(k_lim_fv_min_max<DIM, B>);
    if (e == cudaSuccess)
      k_lim_fv_min_max<DIM, B><<<(unsigned)nblk, kLimNT, smem, st>>>(nvar, nobs, ghost, ncells, cpb, in, mn, mx,
                                                                       sel);
  } else {
    auto kern = k_lim_min_max<DIM, B, NVT, false>;
    if constexpr (DIM == 2 && B <= 6)
      if (walk) kern = k_lim_min_max<DIM, B, NVT, true>;
    e = allow_max_smem(kern);
    if (e == cudaSuccess)
      kern<<<(unsigned)nblk, kLimMmNT, smem, st>>>(op == kLimDmp ? 1 : 0, nvar, nobs, ncells, cpb, in, relax, scaling, mn,
                                                  mx, ok);
  }
  if (e != cudaSuccess) return cuda_status(e, "limiter: shared-memory attribute");
  count_launch();
  return cuda_status(cudaGetLastError(), "limiter kernel");
}

// the Euler case (5 variables, 5 observables) runs kernels specialised for
// it; any other count the generic ones
template <int DIM, int B>
static exa_status_t lim_run_nv(int op, int nvar, int nobs, int ghost, long ncells, const double* in, double* out,
                               double* mn, double* mx, int* ok, double relax, double scaling, cudaStream_t st,
                               LimSel sel) {
  const bool five = nvar == 5 && (op < kLimMinMax || op == kLimFvMinMax || nobs == 5);
  if (five) return lim_run<DIM, B, 5>(op, nvar, nobs, ghost, ncells, in, out, mn, mx, ok, relax, scaling, st, sel);
  return lim_run<DIM, B, 0>(op, nvar, nobs, ghost, ncells, in, out, mn, mx, ok, relax, scaling, st, sel);
}

template <int DIM>
static exa_status_t lim_dispatch(int op, int order, int nvar, int nobs, int ghost, long ncells, const double* in,
                                 double* out, double* mn, double* mx, int* ok, double relax, double scaling,
                                 cudaStream_t st, LimSel sel) {
  switch (order) {
    case 1: return lim_run_nv<DIM, 2>(op, nvar, nobs, ghost, ncells, in, out, mn, mx, ok, relax, scaling, st, sel);
    case 2: return lim_run_nv<DIM, 3>(op, nvar, nobs, ghost, ncells, in, out, mn, mx, ok, relax, scaling, st, sel);
    case 3: return lim_run_nv<DIM, 4>(op, nvar, nobs, ghost, ncells, in, out, mn, mx, ok, relax, scaling, st, sel);
    case 4: return lim_run_nv<DIM, 5>(op, nvar, nobs, ghost, ncells, in, out, mn, mx, ok, relax, scaling, st, sel);
    case 5: return lim_run_nv<DIM, 6>(op, nvar, nobs, ghost, ncells, in, out, mn, mx, ok, relax, scaling, st, sel);
    case 6: return lim_run_nv<DIM, 7>(op, nvar, nobs, ghost, ncells, in, out, mn, mx, ok, relax, scaling, st, sel);
  }
  return set_error(EXA_EINVAL, "limiter: order must be in 1..6");
}

static exa_status_t lim_entry(int op, int dim, int order, int nvar, int nobs, int ghost, long ncells,
                              const double* in, double* out, double* mn, double* mx, int* ok, double relax,
                              double scaling, void* stream, LimSel sel = LimSel()) {
  if (exa_status_t s = ensure_tables()) return s;
  if (dim != 2 && dim != 3) return set_error(EXA_EINVAL, "limiter: dim must be 2 or 3");
  if (nvar < 1 || nvar > 64) return set_error(EXA_EINVAL, "limiter: nvar must be in 1..64");
  if (ghost < 0 || ghost > 8) return set_error(EXA_EINVAL, "limiter: ghost layer width must be in 0..8");
  if (ncells < 0) return set_error(EXA_EINVAL, "limiter: negative cell count");
  if (op >= kLimMinMax) {
    if (nobs < 0 || nobs > nvar) return set_error(EXA_EINVAL, "limiter: nobs must be in 0..nvar");
    if (!in || (nobs > 0 && (!mn || !mx)) || (op == kLimDmp && !ok))
      return set_error(EXA_EINVAL, "limiter: NULL pointer");
    // without observables the solver layer skips the search altogether
    // (LimitingADERDGSolver.cpp:993-1026); the DMP entry needs one
    if (nobs == 0) return op == kLimDmp ? set_error(EXA_EINVAL, "limiter: DMP needs nobs >= 1") : EXA_OK;
  } else if (!in || !out) {
    return set_error(EXA_EINVAL, "limiter: NULL pointer");
  }
  if (ncells == 0) return EXA_OK;
  cudaStream_t st = as_stream(stream);
  return dim == 2 ? lim_dispatch<2>(op, order, nvar, nobs, ghost, ncells, in, out, mn, mx, ok, relax, scaling, st, sel)
                  : lim_dispatch<3>(op, order, nvar, nobs, ghost, ncells, in, out, mn, mx, ok, relax, scaling, st, sel);
}

exa_status_t limiter_launch(int op, int dim, int order, int nvar, int nobs, int ghost, long ncells, const double* in,
                            double* out, double* mn, double* mx, int* ok, double relax, double scaling,
                            cudaStream_t st, const int* list, const int* count) {
  LimSel sel;
  sel.list = list;
  sel.count = count;
  return lim_entry(op, dim, order, nvar, nobs, ghost, ncells, in, out, mn, mx, ok, relax, scaling,
                   reinterpret_cast<void*>(st), sel);
}

exa_status_t upload_tables_limiter() {
  static LimConst h[kLimMaxOrder + 1];
  for (int n = 0; n <= kLimMaxOrder; n++) {
    const int B = n + 1, S = 2 * n + 1;
    for (int k = 0; k < 7; k++) {
      for (int i = 0; i < 13; i++) h[n].uh2lim[k][i] = (k < B && i < S) ? exa_uh2lim[n][k][i] : 0.0;
      for (int i = 0; i < 7; i++) h[n].uh2lob[k][i] = (k < B && i < B) ? exa_uh2lob[n][k][i] : 0.0;
    }
    for (int i = 0; i < 13; i++)
      for (int k = 0; k < 7; k++) h[n].lim2uh[i][k] = (i < S && k < B) ? exa_lim2uh[n][i][k] : 0.0;
  }
  return cuda_status(cudaMemcpyToSymbol(c_lim, h, sizeof(h)), "upload tables (limiter)");
}

}  // namespace exa

using namespace exa;

extern "C" {

exa_status_t exa_limiter_project_on_fv(int dim, int order, int nvar, int ghost_layer_width, long ncells,
                                       const double* luh, double* lim, void* stream) {
  return lim_entry(kLimToFv, dim, order, nvar, 0, ghost_layer_width, ncells, luh, lim, nullptr, nullptr, nullptr,
                   0.0, 0.0, stream);
}

exa_status_t exa_limiter_project_on_dg(int dim, int order, int nvar, int ghost_layer_width, long ncells,
                                       const double* lim, double* luh, void* stream) {
  return lim_entry(kLimToDg, dim, order, nvar, 0, ghost_layer_width, ncells, lim, luh, nullptr, nullptr, nullptr,
                   0.0, 0.0, stream);
}

exa_status_t exa_limiter_local_min_max(int dim, int order, int nvar, int nobs, long ncells, const double* luh,
                                       double* obs_min, double* obs_max, void* stream) {
  return lim_entry(kLimMinMax, dim, order, nvar, nobs, 0, ncells, luh, nullptr, obs_min, obs_max, nullptr, 0.0, 0.0,
                   stream);
}

exa_status_t exa_limiter_fv_min_max(int dim, int order, int nvar, int nobs, int ghost_layer_width, long ncells,
                                    const double* lim, double* obs_min, double* obs_max, void* stream) {
  return lim_entry(kLimFvMinMax, dim, order, nvar, nobs, ghost_layer_width, ncells, lim, nullptr, obs_min, obs_max,
                   nullptr, 0.0, 0.0, stream);
}

exa_status_t exa_limiter_dmp(int dim, int order, int nvar, int nobs, long ncells, const double* luh,
                             double relaxation, double difference_scaling, double* obs_min, double* obs_max,
                             int* dmp_ok, void* stream) {
  return lim_entry(kLimDmp, dim, order, nvar, nobs, 0, ncells, luh, nullptr, obs_min, obs_max, dmp_ok, relaxation,
                   difference_scaling, stream);
}

}  // extern "C"
