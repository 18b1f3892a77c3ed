// Cell-status and bookkeeping kernels of the limiting ADER-DG grid (the
// a-posteriori subcell limiter of exahype/solvers/LimitingADERDGSolver.cpp on
// a uniform 2D or 3D grid, periodic or with outflow / reflecting walls).  Per step, after the unlimited DG candidate:
//   k_lim_admissible   physical admissibility of the candidate (positive
//                      density and pressure at every node), folded into the
//                      DMP verdict (LimitingADERDGSolver.cpp:839-876,
//                      1028-1048)
//   k_lim_base_status  Troubled for cells that fail; cells that were
//                      Troubled stay so for steps-till-cured more steps, then
//                      become NeighbourOfTroubled1 (determineLimiterStatus-
//                      AfterSolutionUpdate, :933-991)
//   k_lim_spread       two face-neighbour hops of status spreading: with each
//                      hop a cell takes max(own, neighbour - 1) (ADERDGSolver.cpp
//                      mergeWithLimiterStatus :2482-2500); the second launch
//                      also lists the cells that need a subcell patch (status
//                      >= NeighbourOfTroubled3) and the cells the FV solver
//                      updates (status >= NeighbourOfTroubled2)
//   k_lim_local /      the new cell-local extrema and their merge with the
//   k_lim_merge        face neighbours' (mergeSolutionMinMaxOnFace,
//                      LimitingADERDGSolver.cpp:1792-1853)
// Status values follow ADERDGCellDescription::LimiterStatus: Ok 0,
// NeighbourOfTroubled4 1, ..3 2, ..2 3, ..1 4, Troubled 5.
#include <float.h>

#include "exa_device.cuh"

namespace exa {

constexpr int kLimTroubled = 5, kLimNT1 = 4, kLimNT2 = 3, kLimNT3 = 2;

__global__ void k_lim_admissible(int npc, long ncells, int planar, const double* luh, int* ok) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;  // node
  if (i >= ncells * npc) return;
  const double* q = luh + i * kV;
  const double rho = q[0];
  const double j2 = planar ? q[1] * q[1] + q[2] * q[2] : q[1] * q[1] + q[2] * q[2] + q[3] * q[3];
  const double p = (kGamma - 1.0) * (q[4] - 0.5 * j2 / rho);
  if (!(rho > 0.0 && p > 0.0 && isfinite(p))) ok[i / npc] = 0;
}

// also clears the counters that the listing adds to
__global__ void k_lim_base_status(long ncells, const int* ok, int* status, int* cure, int steps_till_cured,
                                  int* counts) {
  const long c = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c < 3) counts[c] = 0;
  if (c >= ncells) return;
  int base = 0;
  if (!ok[c]) {
    cure[c] = steps_till_cured + 1;
    base = kLimTroubled;
  } else if (status[c] == kLimTroubled) {
    const int left = cure[c] - 1;
    if (left <= 0) {
      base = kLimNT1;
      cure[c] = steps_till_cured;
    } else {
      base = kLimTroubled;
      cure[c] = left;
    }
  }
  status[c] = base;
}

// grid of n.x x n.y x n.z cells (n.z = 1 in 2D), x fastest; bc[d] = 0
// periodic, else the domain ends in direction d
struct LimGrid {
  int nx, ny, nz, dim;
  int bc[3];
  __host__ __device__ __forceinline__ long cells() const { return (long)nx * ny * nz; }
  // (32-bit divisions: the cells are far below 2^31)
  __device__ __forceinline__ void coords(long c, int& x, int& y, int& z) const {
    const unsigned row = (unsigned)c / (unsigned)nx;
    x = (int)((unsigned)c - row * (unsigned)nx);
    z = (int)(row / (unsigned)ny);
    y = (int)row - z * ny;
  }
  // the neighbour across face f = 2 d + (0 lower, 1 upper), -1 outside
  __device__ __forceinline__ long nb(long c, int f) const {
    int x, y, z;
    coords(c, x, y, z);
    const int d = f >> 1;
    const bool up = f & 1;
    int* p = d == 0 ? &x : (d == 1 ? &y : &z);
    const int n = d == 0 ? nx : (d == 1 ? ny : nz);
    if (up ? *p + 1 == n : *p == 0) {
      if (bc[d] != 0) return -1;
      *p = up ? 0 : n - 1;
    } else {
      *p += up ? 1 : -1;
    }
    return ((long)z * ny + y) * nx + x;
  }
};

// Two hops at once: the largest in[cell'] - k over the cells at face distance
// k <= 2 (in a box, walls or not, k is |dx| + |dy| + |dz|).  One hop per launch
// took four launches of 5 us for 59,049 cells and a memset and a launch for the
// lists; the launches, not their work, were the cost.
// LISTS: counts[0]: cells with a subcell patch, counts[1]: FV-updated cells,
// counts[2]: Troubled cells
template <bool LISTS>
__global__ void k_lim_spread(LimGrid G, const int* in, int* out, int* list_patch, int* list_fv, int* counts) {
  const long c = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= G.cells()) return;
  int x, y, z;
  G.coords(c, x, y, z);
  auto fold = [](int i, int n, int rule) {  // -1: outside the domain
    if (i >= 0 && i < n) return i;
    return rule != 0 ? -1 : (i % n + n) % n;
  };
  const int rz = G.dim == 3 ? 2 : 0;
  int s = 0;
  for (int dz = -rz; dz <= rz; dz++) {
    const int zz = fold(z + dz, G.nz, G.bc[2]);
    if (zz < 0) continue;
    const int ry = 2 - abs(dz);
    for (int dy = -ry; dy <= ry; dy++) {
      const int yy = fold(y + dy, G.ny, G.bc[1]);
      if (yy < 0) continue;
      const int rx = ry - abs(dy);
      for (int dx = -rx; dx <= rx; dx++) {
        const int xx = fold(x + dx, G.nx, G.bc[0]);
        if (xx >= 0) s = max(s, in[((long)zz * G.ny + yy) * G.nx + xx] - (abs(dx) + abs(dy) + abs(dz)));
      }
    }
  }
  out[c] = s;
  if (LISTS) {
    if (s >= kLimNT3) list_patch[atomicAdd(counts + 0, 1)] = (int)c;
    if (s >= kLimNT2) list_fv[atomicAdd(counts + 1, 1)] = (int)c;
    if (s == kLimTroubled) atomicAdd(counts + 2, 1);
  }
}

// face block 0 of the per-cell extrema -> loc [cell][min | max][nobs]
__global__ void k_lim_local(long ncells, int nf, int nobs, const double* bmin, const double* bmax, double* loc) {
  const long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= ncells * nobs) return;
  const long c = k / nobs;
  const int v = (int)(k % nobs);
  loc[(c * 2 + 0) * nobs + v] = bmin[c * nf * nobs + v];
  loc[(c * 2 + 1) * nobs + v] = bmax[c * nf * nobs + v];
}

// face f of a cell: extrema of the cell and of its neighbour across f; one
// thread per (cell, observable)
__global__ void k_lim_merge(LimGrid G, int nobs, const double* loc, double* bmin, double* bmax) {
  const long k = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= G.cells() * nobs) return;
  const int v = (int)(k % nobs);
  const long c = k / nobs;
  const int nf = 2 * G.dim;
  const double mo = loc[(c * 2) * nobs + v], xo = loc[(c * 2 + 1) * nobs + v];
  for (int f = 0; f < nf; f++) {
    const long nb0 = G.nb(c, f);
    const long nb = nb0 >= 0 ? nb0 : c;  // a domain-boundary face keeps the cell's own extrema
    const double mn = loc[(nb * 2) * nobs + v], xn = loc[(nb * 2 + 1) * nobs + v];
    bmin[(c * nf + f) * nobs + v] = mn < mo ? mn : mo;
    bmax[(c * nf + f) * nobs + v] = xo < xn ? xn : xo;
  }
}

// NaN / Inf in the final state of the FV-updated cells
__global__ void k_lim_finite(int npc, const double* luh, const int* list, const int* count, int* nan_flag) {
  const long total = (long)*count * npc * kV;
  for (long k = (long)blockIdx.x * blockDim.x + threadIdx.x; k < total; k += (long)gridDim.x * blockDim.x) {
    const long cell = list[k / (npc * kV)];
    if (!isfinite(luh[cell * npc * kV + k % (npc * kV)])) atomicOr(nan_flag, 1);
  }
}

static unsigned blocks(long n, int nt) { return (unsigned)((n + nt - 1) / nt); }

static LimGrid lim_grid(int dim, const int* n, const int* bc) {
  LimGrid G;
  G.nx = n[0];
  G.ny = n[1];
  G.nz = dim == 3 ? n[2] : 1;
  G.dim = dim;
  for (int d = 0; d < 3; d++) G.bc[d] = bc && d < dim ? bc[d] : 0;
  return G;
}

exa_status_t limiting_status(int dim, const int* ncell, const int* bc, int npc, int planar, int admissibility,
                             int steps_till_cured, const double* luh, int* ok, int* status, int* status_tmp,
                             int* cure, int* list_patch, int* list_fv, int* counts, cudaStream_t st) {
  const LimGrid G = lim_grid(dim, ncell, bc);
  const long n = (long)G.nx * G.ny * G.nz;
  if (admissibility) k_lim_admissible<<<blocks(n * npc, 256), 256, 0, st>>>(npc, n, planar, luh, ok);
  // (a grid of one or two cells still has the threads that clear the counters)
  k_lim_base_status<<<blocks(n, 256), 256, 0, st>>>(n, ok, status, cure, steps_till_cured, counts);
  // four hops: Troubled (5) reaches NeighbourOfTroubled4 (1)
  k_lim_spread<false><<<blocks(n, 256), 256, 0, st>>>(G, status, status_tmp, nullptr, nullptr, nullptr);
  k_lim_spread<true><<<blocks(n, 256), 256, 0, st>>>(G, status_tmp, status, list_patch, list_fv, counts);
  count_launch(3 + (admissibility ? 1 : 0));
  return cuda_status(cudaGetLastError(), "limiter status kernels");
}

exa_status_t limiting_merge_bounds(int dim, const int* ncell, const int* bc, int nobs, double* bmin, double* bmax,
                                   double* loc, cudaStream_t st) {
  const LimGrid G = lim_grid(dim, ncell, bc);
  const long n = (long)G.nx * G.ny * G.nz;
  k_lim_local<<<blocks(n * nobs, 256), 256, 0, st>>>(n, 2 * dim, nobs, bmin, bmax, loc);
  k_lim_merge<<<blocks(n * nobs, 256), 256, 0, st>>>(G, nobs, loc, bmin, bmax);
  count_launch(2);
  return cuda_status(cudaGetLastError(), "limiter bound merge");
}

exa_status_t limiting_check_finite(int npc, const double* luh, const int* list, const int* count, int* nan_flag,
                                   cudaStream_t st) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  k_lim_finite<<<(unsigned)(2 * sms), 256, 0, st>>>(npc, luh, list, count, nan_flag);
  count_launch();
  return cuda_status(cudaGetLastError(), "k_lim_finite");
}

}  // namespace exa
