// fg_ad.cu -- the momentum equation's line SOR on device fields:
// set_solve_ad's diffusion coefficients (CORE_SET_SOLVERS.F90:591-677),
// one pass of itsolv_ad (CORE_SOLVE_AD.F90:131-776: x, then y, then z line
// sweeps with the implicit convection terms) and calc_residual_ad
// (:780-964), the outer velocity boundaries (CORE_SET_OUTER_BC.F90
// set_outer_velocity_bc, set_outer_ghost_velocity) and the solve_ad
// iteration around them (CORE_SOLVE_AD.F90:11-127).  Fields are device
// arrays in the reference layout (0:nx+1, 0:ny+1, 0:nz+1), node counts.
//
// The reference sweeps the lines of each direction in lexicographic order,
// Gauss-Seidel style: an x line (j,k) reads the new values of lines (j-1,k)
// and (j,k-1) and the old values of (j+1,k) and (j,k+1).  A sweep is
// therefore a chain of lines, and a line a chain of rows; everything that
// is not on those chains is taken off them.  The pivots of the Thomas
// recursion depend on the coefficients alone: k_ad_factor forms them for
// all lines at once.  k_ad_sweeps then runs the lines as a wavefront, one
// block per column of lines (all k of one j, say), each block waiting for
// its neighbour's line through a progress counter in global memory, so the
// blocks work on one anti-diagonal without a launch between diagonals.
// Every operation of a row is the reference's, in its order, and this file
// is compiled without FMA contraction: the result is bit-identical to the
// sequential sweep.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "fg_case.h"
#include "fg_internal.h"

namespace fg {
namespace ad {

// 1-D arrays of each axis (reference indexing 0..n+1): the share of cell i
// in the value at its lower node (CORE_GRID.F90:194-202), 1/width, and
// set_solve_ad's couplings
struct MetAxis {
  const double *f, *di, *am, *ap;
};
struct Met {
  MetAxis a[3];
};

struct Dims {
  int nx, ny, nz;
  long long NX, NY;
  __device__ __forceinline__ long long id(int i, int j, int k) const { return i + NX * (j + NY * (long long)k); }
};

// the coupling to the lower and upper neighbour along one axis and the
// axis's share of the diagonal (CORE_SOLVE_AD.F90:215-330): diffusion, then
// the implicit convection of the faces f0 and f1 of cell s, central for
// 25 <= i <= 375 (the reference's switch is on i for all three directions),
// first-order upwind elsewhere
struct AxisCoef {
  double lo, hi, ac;
};
__device__ __forceinline__ AxisCoef axis_coef(const MetAxis &m, int s, double f0, double f1, double half_dt,
                                              bool central) {
  AxisCoef q;
  const double am = m.am[s], ap = m.ap[s], di = m.di[s];
  q.ac = -(am + ap);
  if (central) {
    const double t0 = m.f[s], t1 = m.f[s + 1];
    q.lo = am - half_dt * f0 * (1.0 - t0) * di;
    q.hi = ap + half_dt * f1 * t1 * di;
    q.ac = q.ac + half_dt * (f1 * (1.0 - t1) - f0 * t0) * di;
  } else {
    const double s0 = copysign(1.0, f0), s1 = copysign(1.0, f1);
    q.lo = am - half_dt * (0.5 * (1.0 + s0)) * f0 * di;
    q.hi = ap + half_dt * (0.5 * (1.0 - s1)) * f1 * di;
    q.ac = q.ac + half_dt * (f1 * (0.5 * (1.0 + s1)) - f0 * (0.5 * (1.0 - s0))) * di;
  }
  return q;
}

struct Faces {
  const double *f[3];  // face_u, face_v, face_w
};
template <int NC>
struct Comps {
  double *v[NC];
  const double *r[NC];
};

__device__ __forceinline__ bool central_at(int i) { return i >= 25 && i <= 375; }

// 1 on fluid non-ghost cells, 0 elsewhere
__device__ __forceinline__ double fluid(const int8_t *ib, const int8_t *gh, long long id) {
  return (1.0 - (double)ib[id]) * (1.0 - (double)abs((int)gh[id]));
}

// 1 / pivot of every row of every line (CORE_TDMA.F90:22-27), rows 1..n,
// blockIdx.y = axis.  A block takes 32 lines in tiles of FT_ROWS rows: warps
// 1..8 form a tile's coefficients in shared memory (loads along i whatever
// the axis) and store the pivots of the tile before last, while lane l of
// warp 0 runs line l's recurrence, whose division is the bound, over the
// tile between.  One thread per line did the loads, the coefficients and
// the recurrence in turn: 310 + 123 + 114 us at 192x96x96 cells, 100 us as
// one launch of this kernel.
constexpr int FT_ROWS = 16, FT_LINES = 32, FT_WORK = 256;
struct FactorTile {
  double lo[FT_ROWS][FT_LINES + 1], hi[FT_ROWS][FT_LINES + 1], ac[FT_ROWS][FT_LINES + 1];
};
template <int AXIS>
__device__ __forceinline__ void factor_lines(const Dims &d, const Met &m, const int8_t *__restrict__ ib,
                                             const int8_t *__restrict__ gh, const Faces &F, double half_dt,
                                             double *__restrict__ binv, FactorTile *tile) {
  constexpr int P = AXIS == 0 ? 1 : 0, Q = AXIS == 2 ? 1 : 2;
  const int np = AXIS == 0 ? d.ny - 1 : d.nx - 1, nq = AXIS == 2 ? d.ny - 1 : d.nz - 1;
  const int n = AXIS == 0 ? d.nx : AXIS == 1 ? d.ny : d.nz;
  const int groups = (np + FT_LINES - 1) / FT_LINES;  // line groups of one q
  if (blockIdx.x >= (unsigned)(groups * nq)) return;
  const int p0 = 1 + FT_LINES * (int)(blockIdx.x % groups), q = 1 + blockIdx.x / groups;
  const long long st[3] = {1, d.NX, d.NX * d.NY};
  const long long base = st[P] * p0 + st[Q] * q, step = st[AXIS];
  const int tid = threadIdx.x;
  const int ntile = (n - 1 + FT_ROWS - 1) / FT_ROWS;
  double bi = 1.0, c_prev = 0.0;
  for (int k = 0; k < ntile + 2; ++k) {
    if (tid < 32) {
      if (k >= 1 && k <= ntile) {
        FactorTile &t = tile[(k - 1) & 1];
        const int rows = min(FT_ROWS, n - 1 - (k - 1) * FT_ROWS);
        for (int r = 0; r < rows; ++r) {
          bi = 1.0 / (t.ac[r][tid] - t.lo[r][tid] * (c_prev * bi));
          c_prev = t.hi[r][tid];
          t.ac[r][tid] = bi;
        }
      }
    } else {
      FactorTile &t = tile[k & 1];
#pragma unroll
      for (int u = 0; u < FT_ROWS * FT_LINES / FT_WORK; ++u) {
        const int e = tid - 32 + FT_WORK * u;
        // neighbouring threads take neighbouring i: rows along x, lines else
        const int r = AXIS == 0 ? e % FT_ROWS : e / FT_LINES, l = AXIS == 0 ? e / FT_ROWS : e % FT_LINES;
        const int p = p0 + l;
        if (p > np) continue;
        const int sd = (k - 2) * FT_ROWS + r + 1, s = k * FT_ROWS + r + 1;
        if (k >= 2 && sd < n) binv[base + st[P] * l + step * sd] = t.ac[r][l];
        if (k < ntile && s < n) {
          const long long id = base + st[P] * l + step * s;
          const bool ce = central_at(AXIS == 0 ? s : p);
          const double *fo = F.f[AXIS], *fp = F.f[P], *fq = F.f[Q];
          const AxisCoef o = axis_coef(m.a[AXIS], s, fo[id], fo[id + step], half_dt, ce);
          const AxisCoef a = axis_coef(m.a[P], p, fp[id], fp[id + st[P]], half_dt, ce);
          const AxisCoef b = axis_coef(m.a[Q], q, fq[id], fq[id + st[Q]], half_dt, ce);
          const double rib = fluid(ib, gh, id);
          // acx + acy + acz
          const double sum = AXIS == 0 ? o.ac + a.ac + b.ac : AXIS == 1 ? a.ac + o.ac + b.ac : a.ac + b.ac + o.ac;
          t.lo[r][l] = o.lo * rib;
          t.hi[r][l] = o.hi * rib;
          t.ac[r][l] = 1.0 + sum * rib;
        }
      }
    }
    __syncthreads();
  }
  if (tid < 32 && p0 + tid <= np) binv[base + st[P] * tid + step * n] = 1.0 / (1.0 - 0.0 * (c_prev * bi));
}

// binv: one array of `nref` values per axis
__global__ void __launch_bounds__(32 + FT_WORK)
k_ad_factor(Dims d, Met m, const int8_t *__restrict__ ib, const int8_t *__restrict__ gh, Faces F, double half_dt,
            double *__restrict__ binv, long long nref) {
  extern __shared__ __align__(16) double ft_smem[];
  FactorTile *tile = reinterpret_cast<FactorTile *>(ft_smem);
  if (blockIdx.y == 0) factor_lines<0>(d, m, ib, gh, F, half_dt, binv, tile);
  else if (blockIdx.y == 1) factor_lines<1>(d, m, ib, gh, F, half_dt, binv + nref, tile);
  else factor_lines<2>(d, m, ib, gh, F, half_dt, binv + 2 * nref, tile);
}

__device__ __forceinline__ int ld_acquire(const int *p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int *p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void bar_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// The x, y and z sweeps of NC velocity components at once (the components
// share the coefficients and do not read one another).  A block takes a
// column of lines (x and y lines: all of one k; z lines: all of one j) and
// solves them in increasing order of the other index (x: j; y and z: i).
// Line l of a column reads the new line l of the column before, announced in
// that column's progress counter, and the new line l - 1 of its own.
//
// The sweeps overlap.  The y column k may start once the x column k + 1 is
// done (no x line still reads or writes plane k, and the plane it reads
// above is swept); z line l may start once every y column has passed line
// l + 1, which the last y column's counter tells (a column never passes the
// one before it).  Columns are drawn from a ticket in the order x, y, z, so
// whatever a block waits for has started: the waits end.  Each is bounded
// all the same; one that runs out sets *err and the blocks return.
//
// Warps: 0 runs the recurrence (lane c = component c) through shared
// memory; 1 waits for the neighbour column and fetches its line; 2 announces
// the column's progress, so that nobody else waits for the stores to become
// visible; the others hold R rows per thread, form the next line's
// coefficients while the recurrence runs, then its right-hand sides, and
// relax.  The recurrence, 3 dependent operations per row down and 2 up, is
// what bounds the pass: it takes about 35 ns per row (65 cycles for the 5
// operations), and (ny + nz) x lines, nx y lines and ny z lines follow one
// another, with some 7 us more for each step from a column to the next.
// Measured at 192x96x96 cells: 2.80 ms; one launch per direction, the
// announcement made by warp 0: 4.30 ms; one launch per anti-diagonal with
// the coefficients and pivots inside the line: 200 ms.
constexpr int SW_POLLS = 1 << 23;
constexpr int SW_ROLES = 96;       // threads of the three warps that hold no rows
constexpr int SW_ROW_THREADS = 512;
struct SweepSync {
  int *err, *ticket, *done[3];  // done[axis][column]
};

// false when the wait was given up
__device__ __forceinline__ bool wait_for(const int *p, int v, int *err, int &seen) {
  for (int polls = 1; (seen = ld_acquire(p)) < v; ++polls) {
    if (polls > SW_POLLS || ((polls & 1023) == 0 && ld_acquire(err))) {
      atomicExch(err, 1);
      return false;
    }
    __nanosleep(20);
  }
  return true;
}

template <int AXIS, int R, int NC>
__device__ __forceinline__ void sweep_column(const Dims &d, const Met &m, const int8_t *__restrict__ ib,
                                             const int8_t *__restrict__ gh, const Comps<NC> &C, const Faces &F,
                                             double half_dt, double omega, const double *__restrict__ binv,
                                             const SweepSync &sync, int c, int &s_bad, double *smem) {
  constexpr int P = AXIS == 0 ? 1 : 0, Q = AXIS == 2 ? 1 : 2;  // axes of the line index and of the column index
  const int nn[3] = {d.nx, d.ny, d.nz};
  const int n = nn[AXIS], nl = nn[P] - 1;
  const long long st[3] = {1, d.NX, d.NX * d.NY};
  const long long step = st[AXIS], sa = st[Q], sb = st[P], col = sa * c;
  double2 *s_ab = reinterpret_cast<double2 *>(smem);  // (lower coupling, 1/pivot) of row s
  double *s_g = smem + 2 * (n + 1);                   // gamma of row s + 1
  double *s_u = s_g + (n + 1);                        // right-hand sides, then the solution
  double *s_nb = s_u + NC * (n + 1);                  // the neighbour column's line
  const int tid = threadIdx.x, nt = blockDim.x, warp = tid >> 5, lane = tid & 31;
  const int np = nt - SW_ROLES;  // row threads
  int *done = sync.done[AXIS];
  // named barriers; those with two ids alternate by line, so that the
  // announcing warp may be a line behind
  enum { B_RHS = 1, B_SOL = 2, B_LINE = 3, B_STORED = 5 };
  // the sweep before this one: x columns are all there is for x
  const int *gate = AXIS == 0 ? nullptr : sync.done[AXIS - 1] + (AXIS == 1 ? min(c + 1, d.nz - 1) : d.nz - 1);
  if (AXIS != 0) {
    if (tid == 0) {
      int seen;
      if (!wait_for(gate, AXIS == 1 ? d.ny - 1 : min(2, d.nx - 1), sync.err, seen)) s_bad = 1;
    }
    __syncthreads();
    if (s_bad) return;
  }

  if (warp == 0) {
    for (int l = 1; l <= nl; ++l) {
      bar_sync(B_LINE + (l & 1), nt);
      if (s_bad) return;
      bar_sync(B_RHS, nt - 32);
      if (lane < NC) {
        double *u = s_u + lane * (n + 1);
        constexpr int U = 8;
        double x = u[0];
        int s = 1;
        double2 ab[U];
        double rr[U];
        if (n >= U) {
#pragma unroll
          for (int e = 0; e < U; ++e) { ab[e] = s_ab[s + e]; rr[e] = u[s + e]; }
          for (; s + 2 * U - 1 <= n; s += U) {
            double2 ab1[U];
            double rr1[U];
#pragma unroll
            for (int e = 0; e < U; ++e) { ab1[e] = s_ab[s + U + e]; rr1[e] = u[s + U + e]; }
#pragma unroll
            for (int e = 0; e < U; ++e) { x = (rr[e] - ab[e].x * x) * ab[e].y; u[s + e] = x; }
#pragma unroll
            for (int e = 0; e < U; ++e) { ab[e] = ab1[e]; rr[e] = rr1[e]; }
          }
#pragma unroll
          for (int e = 0; e < U; ++e) { x = (rr[e] - ab[e].x * x) * ab[e].y; u[s + e] = x; }
          s += U;
        }
        for (; s <= n; ++s) {
          const double2 w = s_ab[s];
          x = (u[s] - w.x * x) * w.y;
          u[s] = x;
        }
        s = n - 1;
        if (n - 1 >= U) {
          double gg[U];
#pragma unroll
          for (int e = 0; e < U; ++e) { gg[e] = s_g[s - e]; rr[e] = u[s - e]; }
          for (; s - 2 * U + 1 >= 1; s -= U) {
            double gg1[U], rr1[U];
#pragma unroll
            for (int e = 0; e < U; ++e) { gg1[e] = s_g[s - U - e]; rr1[e] = u[s - U - e]; }
#pragma unroll
            for (int e = 0; e < U; ++e) { x = rr[e] - gg[e] * x; u[s - e] = x; }
#pragma unroll
            for (int e = 0; e < U; ++e) { gg[e] = gg1[e]; rr[e] = rr1[e]; }
          }
#pragma unroll
          for (int e = 0; e < U; ++e) { x = rr[e] - gg[e] * x; u[s - e] = x; }
          s -= U;
        }
        for (; s >= 1; --s) {
          x = u[s] - s_g[s] * x;
          u[s] = x;
        }
      }
      __syncwarp();
      bar_sync(B_SOL, np + 32);
    }
    return;
  }

  if (warp == 1) {
    int seen = 0, gseen = 0;
    for (int l = 1; l <= nl; ++l) {
      bool ok = true;
      if (lane == 0) {
        if (c > 1 && seen < l) ok = wait_for(done + c - 1, l, sync.err, seen);
        // the row threads fetch line l + 1 (and the values of l + 2) next
        const int need = min(l + 2, d.nx - 1);
        if (AXIS == 2 && ok && gseen < need) ok = wait_for(gate, need, sync.err, gseen);
        if (!ok) s_bad = 1;
      }
      __syncwarp();
      const long long nb = col - sa + sb * l;
      for (int s = 1 + lane; s < n; s += 32) {
#pragma unroll
        for (int e = 0; e < NC; ++e) s_nb[e * (n + 1) + s] = __ldcg(C.v[e] + nb + step * s);
      }
      bar_sync(B_LINE + (l & 1), nt);
      if (s_bad) return;
      bar_sync(B_RHS, nt - 32);
    }
    return;
  }

  if (warp == 2) {
    bar_arrive(B_LINE + 1, nt);  // lines 1 and 2 wait for no announcement
    if (nl > 1) bar_arrive(B_LINE, nt);
    for (int l = 1; l <= nl; ++l) {
      bar_sync(B_STORED + (l & 1), np + 32);
      if (s_bad) return;
      if (lane == 0) st_release(done + c, l);
      __syncwarp();
      if (l + 2 <= nl) bar_arrive(B_LINE + (l & 1), nt);
    }
    return;
  }

  const int t = tid - SW_ROLES;
  double own[R][NC], prev[R][NC], hiA[R][NC], hiB[R][NC], rr[R][NC];
  double cp0[R], cp1[R], cq0[R], cq1[R], am[R], g[R], bi[R], rib[R];
  double end0[NC], end1[NC], endb = 1.0;  // rows 0 and n of the line (row thread 0)
  // everything of line l that no line in flight changes; the line's own old
  // values go to `own` later (relax still needs line l - 1's)
  auto fetch = [&](int l, double (&o)[R][NC]) {
    const long long b0 = col + sb * l;
#pragma unroll
    for (int w = 0; w < R; ++w) {
      const int s = 1 + t + np * w;
      if (s < n) {
        const long long id = b0 + step * s;
        const bool ce = central_at(AXIS == 0 ? s : l);
        const double *fo = F.f[AXIS], *fp = F.f[P], *fq = F.f[Q];
        const double o0 = __ldg(fo + id), o1 = __ldg(fo + id + step);
        const double p0 = __ldg(fp + id), p1 = __ldg(fp + id + st[P]);
        const double q0 = __ldg(fq + id), q1 = __ldg(fq + id + st[Q]);
        bi[w] = binv[id];
        rib[w] = fluid(ib, gh, id);
#pragma unroll
        for (int e = 0; e < NC; ++e) {
          rr[w][e] = C.r[e][id];
          o[w][e] = __ldcg(C.v[e] + id);
          hiA[w][e] = __ldcg(C.v[e] + id + sa);
          hiB[w][e] = __ldcg(C.v[e] + id + sb);
        }
        const AxisCoef xo = axis_coef(m.a[AXIS], s, o0, o1, half_dt, ce);
        const AxisCoef xp = axis_coef(m.a[P], l, p0, p1, half_dt, ce);
        const AxisCoef xq = axis_coef(m.a[Q], c, q0, q1, half_dt, ce);
        am[w] = xo.lo * rib[w];
        g[w] = xo.hi * rib[w] * bi[w];
        cp0[w] = xp.lo; cp1[w] = xp.hi;
        cq0[w] = xq.lo; cq1[w] = xq.hi;
      }
    }
    if (t == 0) {
#pragma unroll
      for (int e = 0; e < NC; ++e) {
        end0[e] = __ldcg(C.v[e] + b0);
        end1[e] = __ldcg(C.v[e] + b0 + step * n);
      }
      endb = binv[b0 + step * n];
    }
  };
  fetch(1, own);
#pragma unroll
  for (int w = 0; w < R; ++w) {
    const int s = 1 + t + np * w;
#pragma unroll
    for (int e = 0; e < NC; ++e) prev[w][e] = s < n ? __ldcg(C.v[e] + col + step * s) : 0.0;
  }
  for (int l = 1; l <= nl; ++l) {
    bar_sync(B_LINE + (l & 1), nt);
    if (s_bad) {
      bar_arrive(B_STORED + (l & 1), np + 32);
      return;
    }
#pragma unroll
    for (int w = 0; w < R; ++w) {
      const int s = 1 + t + np * w;
      if (s < n) {
#pragma unroll
        for (int e = 0; e < NC; ++e) {
          const double rh = rr[w][e] - (prev[w][e] * cp0[w] + hiB[w][e] * cp1[w] +
                                        s_nb[e * (n + 1) + s] * cq0[w] + hiA[w][e] * cq1[w]);
          s_u[e * (n + 1) + s] = rh * rib[w] + own[w][e] * (1.0 - rib[w]);
        }
        s_ab[s] = make_double2(am[w], bi[w]);
        s_g[s] = g[w];
      }
    }
    if (t == 0) {
#pragma unroll
      for (int e = 0; e < NC; ++e) {
        s_u[e * (n + 1)] = end0[e];
        s_u[e * (n + 1) + n] = end1[e];
      }
      s_ab[n] = make_double2(0.0, endb);
    }
    bar_sync(B_RHS, nt - 32);
    double nxt[R][NC];
    if (l < nl) fetch(l + 1, nxt);
    bar_sync(B_SOL, np + 32);
    const long long b0 = col + sb * l;
#pragma unroll
    for (int w = 0; w < R; ++w) {
      const int s = 1 + t + np * w;
      if (s < n) {
#pragma unroll
        for (int e = 0; e < NC; ++e) {
          const double v = own[w][e] + omega * (s_u[e * (n + 1) + s] - own[w][e]);
          __stcg(C.v[e] + b0 + step * s, v);
          prev[w][e] = v;
          own[w][e] = nxt[w][e];
        }
      }
    }
    bar_arrive(B_STORED + (l & 1), np + 32);
  }
}

template <int R, int NC>
__global__ void __launch_bounds__(SW_ROLES + SW_ROW_THREADS)
k_ad_sweeps(Dims d, Met m, const int8_t *__restrict__ ib, const int8_t *__restrict__ gh, Comps<NC> C, Faces F,
            double half_dt, double omega, const double *__restrict__ binv, long long nref, SweepSync sync) {
  extern __shared__ __align__(16) double sw_smem[];
  __shared__ int s_ticket, s_bad;
  if (threadIdx.x == 0) {
    s_ticket = atomicAdd(sync.ticket, 1);
    s_bad = 0;
  }
  __syncthreads();
  const int t = s_ticket, nk = d.nz - 1;
  if (t < nk)
    sweep_column<0, R, NC>(d, m, ib, gh, C, F, half_dt, omega, binv, sync, 1 + t, s_bad, sw_smem);
  else if (t < 2 * nk)
    sweep_column<1, R, NC>(d, m, ib, gh, C, F, half_dt, omega, binv + nref, sync, 1 + t - nk, s_bad, sw_smem);
  else
    sweep_column<2, R, NC>(d, m, ib, gh, C, F, half_dt, omega, binv + 2 * nref, sync, 1 + t - 2 * nk, s_bad, sw_smem);
}

// the lines of anti-diagonal `diag` along AXIS (0: x lines (j,k), j + k =
// diag; 1: y lines (i,k); 2: z lines (i,j)), one thread per line, gam and
// the forward values in the thread's slot of `scr` (2 (n+1) doubles), the
// pivots formed along the line: for lines longer than k_ad_sweeps' rows per
// thread hold, and where there is no memory for the pivots of all lines
template <int AXIS>
__global__ void k_ad_diag(Dims d, Met m, const int8_t *__restrict__ ib, const int8_t *__restrict__ gh, double *var,
                          const double *__restrict__ r, Faces F, double half_dt, double omega, int diag,
                          double *__restrict__ scr) {
  constexpr int P = AXIS == 0 ? 1 : 0, Q = AXIS == 2 ? 1 : 2;
  const int amax = AXIS == 0 ? d.ny - 1 : d.nx - 1;
  const int bmax = AXIS == 2 ? d.ny - 1 : d.nz - 1;
  const int a0 = max(1, diag - bmax), a1 = min(amax, diag - 1);
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int a = a0 + t;
  if (a > a1) return;
  const int b = diag - a;
  const int n = AXIS == 0 ? d.nx : AXIS == 1 ? d.ny : d.nz;  // rows 0..n, unknowns 1..n-1
  const long long st[3] = {1, d.NX, d.NX * d.NY};
  const long long base = st[P] * a + st[Q] * b, step = st[AXIS];
  double *g = scr + (size_t)t * 2 * (n + 1), *u = g + (n + 1);
  u[0] = var[base];  // row 0: the trivial equation u = var
  double c_prev = 0.0, bi = 1.0;
  for (int s = 1; s <= n; ++s) {
    double am = 0.0, ac = 1.0, ap = 0.0, rh;
    const long long id = base + step * s;
    if (s == n) {
      rh = var[id];
    } else {
      const bool ce = central_at(AXIS == 0 ? s : a);
      const double *fo = F.f[AXIS], *fp = F.f[P], *fq = F.f[Q];
      // every field's value before the coefficients' branches: a thread walks
      // its line at the latency of a row's loads, and together they cost one
      // (2100 x 64 x 64 cells: 1413 ms with the loads between the branches,
      // 1204 ms so)
      const double o0 = fo[id], o1 = fo[id + step], p0 = fp[id], p1 = fp[id + st[P]], q0 = fq[id], q1 = fq[id + st[Q]];
      const double vp0 = var[id - st[P]], vp1 = var[id + st[P]], vq0 = var[id - st[Q]], vq1 = var[id + st[Q]];
      const double rr = r[id], own = var[id], rib = fluid(ib, gh, id);
      const AxisCoef o = axis_coef(m.a[AXIS], s, o0, o1, half_dt, ce);
      const AxisCoef x = axis_coef(m.a[P], a, p0, p1, half_dt, ce);
      const AxisCoef y = axis_coef(m.a[Q], b, q0, q1, half_dt, ce);
      rh = rr - (vp0 * x.lo + vp1 * x.hi + vq0 * y.lo + vq1 * y.hi);
      // acx + acy + acz
      const double sum = AXIS == 0 ? o.ac + x.ac + y.ac : AXIS == 1 ? x.ac + o.ac + y.ac : x.ac + y.ac + o.ac;
      am = o.lo * rib;
      ap = o.hi * rib;
      ac = 1.0 + sum * rib;
      rh = rh * rib + own * (1.0 - rib);
    }
    // CORE_TDMA.F90:22-27
    g[s] = c_prev * bi;
    bi = 1.0 / (ac - am * g[s]);
    u[s] = (rh - am * u[s - 1]) * bi;
    c_prev = ap;
  }
  for (int s = n - 1; s >= 1; --s) u[s] = u[s] - g[s + 1] * u[s + 1];
  for (int s = 1; s <= n - 1; ++s) {
    const long long id = base + step * s;
    var[id] = var[id] + omega * (u[s] - var[id]);
  }
}

// calc_residual_ad of NC components: per block the largest |res| and the
// first cell (in the reference's k, j, i loop order) that has it.  One pass
// forms the coefficients of a cell once for all components.
template <int NC>
__global__ void __launch_bounds__(256)
k_ad_resid(Dims d, Met m, const int8_t *__restrict__ ib, const int8_t *__restrict__ gh, Comps<NC> C, Faces F,
           double half_dt, double *pval, long long *pidx) {
  const int ni = d.nx - 1, nj = d.ny - 1;
  const long long nt = (long long)ni * nj * (d.nz - 1);
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double v[NC];
  long long at[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) { v[c] = -1.0; at[c] = e; }
  if (e < nt) {
    const long long row = e / ni;
    const int i = 1 + (int)(e - row * ni), k = 1 + (int)(row / nj), j = 1 + (int)(row - (long long)(k - 1) * nj);
    const long long sy = d.NX, sz = d.NX * d.NY, id = d.id(i, j, k);
    const bool ce = central_at(i);
    const AxisCoef x = axis_coef(m.a[0], i, F.f[0][id], F.f[0][id + 1], half_dt, ce);
    const AxisCoef y = axis_coef(m.a[1], j, F.f[1][id], F.f[1][id + sy], half_dt, ce);
    const AxisCoef z = axis_coef(m.a[2], k, F.f[2][id], F.f[2][id + sz], half_dt, ce);
    const double fi = 1.0 - (double)ib[id], fg = 1.0 - (double)gh[id];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const double *var = C.v[c];
      double res = C.r[c][id] - var[id] * (1.0 + x.ac + y.ac + z.ac) - var[id - 1] * x.lo - var[id + 1] * x.hi -
                   var[id - sy] * y.lo - var[id + sy] * y.hi - var[id - sz] * z.lo - var[id + sz] * z.hi;
      res = res * fi * fg;
      v[c] = fabs(res);
    }
  }
  __shared__ double sv[NC][8];
  __shared__ long long sa[NC][8];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    // larger value wins; equal values: the earlier cell
    for (int o = 16; o > 0; o >>= 1) {
      const double ov = __shfl_down_sync(0xffffffffu, v[c], o);
      const long long oa = __shfl_down_sync(0xffffffffu, at[c], o);
      if (ov > v[c] || (ov == v[c] && oa < at[c])) { v[c] = ov; at[c] = oa; }
    }
    if ((threadIdx.x & 31) == 0) { sv[c][threadIdx.x >> 5] = v[c]; sa[c][threadIdx.x >> 5] = at[c]; }
  }
  __syncthreads();
  if (threadIdx.x < NC) {
    const int c = threadIdx.x;
    double bv = sv[c][0];
    long long ba = sa[c][0];
    for (int w = 1; w < 8; ++w)
      if (sv[c][w] > bv || (sv[c][w] == bv && sa[c][w] < ba)) { bv = sv[c][w]; ba = sa[c][w]; }
    pval[(size_t)c * gridDim.x + blockIdx.x] = bv;
    pidx[(size_t)c * gridDim.x + blockIdx.x] = ba;
  }
}

// the largest of the nb block results of component blockIdx.x, into
// out[2 c], out[2 c + 1] (the cell as an exact double).  The reference
// starts from resm = 0 and keeps the first cell whose |res| exceeds the
// running maximum.
__global__ void __launch_bounds__(1024) k_ad_resid_max(const double *pval, const long long *pidx, int nb, double *out) {
  const double *pv = pval + (size_t)blockIdx.x * nb;
  const long long *pi = pidx + (size_t)blockIdx.x * nb;
  double v = 0.0;
  long long at = 0;
  auto take = [&](double ov, long long oa) {
    if (ov > v || (ov == v && ov > 0.0 && oa < at)) { v = ov; at = oa; }
  };
  for (int b = threadIdx.x; b < nb; b += 1024) take(pv[b], pi[b]);
  __shared__ double sv[32];
  __shared__ long long sa[32];
  for (int o = 16; o > 0; o >>= 1) {
    const double ov = __shfl_down_sync(0xffffffffu, v, o);
    const long long oa = __shfl_down_sync(0xffffffffu, at, o);
    take(ov, oa);
  }
  if ((threadIdx.x & 31) == 0) { sv[threadIdx.x >> 5] = v; sa[threadIdx.x >> 5] = at; }
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int w = 1; w < 32; ++w) take(sv[w], sa[w]);
  out[2 * blockIdx.x] = v;
  out[2 * blockIdx.x + 1] = (double)at;
}

// ---- outer velocity boundaries (CORE_SET_OUTER_BC.F90:18-509, :739-823)
// Face order f: x1, x2, y1, y2, z1, z2.  puls holds the pulsatile values
// val * sin(2 pi freq t) (x1's u: val t / 30), formed on the host with the
// host's libm as the reference.
struct VelBC {
  int type[6];
  double val[6][3], puls[6][3];
  double yOrigin, yout, zOrigin, zout;
};
struct BCArr {
  double *a[9];  // bcxu, bcxv, bcxw, bcyu, bcyv, bcyw, bczu, bczv, bczw
};
struct Vel {
  const double *f[3];
};

// the user-specified channel profile val 6 (s - lo)(hi - s) / (hi - lo)^2
__device__ __forceinline__ double channel(double val, double s, double lo, double hi) {
  const double e = hi - lo;
  return val * 6.0 * (s - lo) * (hi - s) / (e * e);
}

// x faces: one thread per (side, j, k), j = 0..ny+1, k = 0..nz+1
__global__ void k_outer_bc_x(Dims d, VelBC p, const double *y, Vel U, BCArr B) {
  const long long n = d.NY * (long long)(d.nz + 2), e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= 2 * n) return;
  const int side = (int)(e / n), j = (int)((e % n) % d.NY), k = (int)((e % n) / d.NY);
  const int i = side ? d.nx - 1 : 1, io = side ? 1 : d.nx - 1;
  const long long b = side + 2 * (j + d.NY * (long long)k), id = d.id(i, j, k), ido = d.id(io, j, k);
  const double *val = p.val[side];
  switch (p.type[side]) {
    case 1: for (int a = 0; a < 3; ++a) B.a[a][b] = val[a]; break;
    case 2: for (int a = 0; a < 3; ++a) B.a[a][b] = U.f[a][id]; break;
    case 3: for (int a = 0; a < 3; ++a) B.a[a][b] = p.puls[side][a]; break;
    case 4: B.a[0][b] = 0.0; B.a[1][b] = U.f[1][id]; B.a[2][b] = U.f[2][id]; break;
    case 5: for (int a = 0; a < 3; ++a) B.a[a][b] = 0.5 * (U.f[a][id] + U.f[a][ido]); break;
    case 6:
      B.a[0][b] = channel(val[0], y[j], p.yOrigin, p.yout);
      if (side) { B.a[1][b] = val[1]; B.a[2][b] = val[2]; }
      break;
  }
}

// y faces: one thread per (side, i, k), i = 0..nx, k = 0..nz+1; the
// user-specified profile goes into the x2 arrays at (1, j, k), written by
// the i = 0 thread alone (the reference writes the same value for each i)
__global__ void k_outer_bc_y(Dims d, VelBC p, const double *z, Vel U, BCArr B) {
  const long long ni = d.nx + 1, n = ni * (d.nz + 2), e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= 2 * n) return;
  const int side = (int)(e / n), i = (int)((e % n) % ni), k = (int)((e % n) / ni), f = 2 + side;
  const int j = side ? d.ny - 1 : 1, jo = side ? 1 : d.ny - 1;
  const long long b = i + d.NX * (side + 2 * (long long)k), id = d.id(i, j, k), ido = d.id(i, jo, k);
  const double *val = p.val[f];
  switch (p.type[f]) {
    case 1: for (int a = 0; a < 3; ++a) B.a[3 + a][b] = val[a]; break;
    case 2: for (int a = 0; a < 3; ++a) B.a[3 + a][b] = U.f[a][id]; break;
    case 3: for (int a = 0; a < 3; ++a) B.a[3 + a][b] = p.puls[f][a]; break;
    case 4: B.a[3][b] = U.f[0][id]; B.a[4][b] = 0.0; B.a[5][b] = U.f[2][id]; break;
    case 5: for (int a = 0; a < 3; ++a) B.a[3 + a][b] = 0.5 * (U.f[a][id] + U.f[a][ido]); break;
    case 6:
      if (i == 0) {
        const long long bx = 1 + 2 * (j + d.NY * (long long)k);
        B.a[0][bx] = val[0];
        B.a[1][bx] = channel(val[1], z[k], p.zOrigin, p.zout);
        B.a[2][bx] = val[2];
      }
      break;
  }
}

// z faces: one thread per (side, i, j), i = 0..nx, j = 0..ny+1
__global__ void k_outer_bc_z(Dims d, VelBC p, const double *y, Vel U, BCArr B) {
  const long long ni = d.nx + 1, n = ni * d.NY, e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= 2 * n) return;
  const int side = (int)(e / n), i = (int)((e % n) % ni), j = (int)((e % n) / ni), f = 4 + side;
  const int k = side ? d.nz - 1 : 1, ko = side ? 1 : d.nz - 1;
  const long long b = i + d.NX * (j + d.NY * (long long)side), id = d.id(i, j, k), ido = d.id(i, j, ko);
  const double *val = p.val[f];
  switch (p.type[f]) {
    case 1: for (int a = 0; a < 3; ++a) B.a[6 + a][b] = val[a]; break;
    case 2: for (int a = 0; a < 3; ++a) B.a[6 + a][b] = U.f[a][id]; break;
    case 3: for (int a = 0; a < 3; ++a) B.a[6 + a][b] = p.puls[f][a]; break;
    case 4: B.a[6][b] = U.f[0][id]; B.a[7][b] = U.f[1][id]; B.a[8][b] = 0.0; break;
    case 5: for (int a = 0; a < 3; ++a) B.a[6 + a][b] = 0.5 * (U.f[a][id] + U.f[a][ido]); break;
    case 6:
      if (i == 0) {
        const long long bx = 1 + 2 * (j + d.NY * (long long)k);
        B.a[0][bx] = val[0];
        B.a[1][bx] = val[1];
        B.a[2][bx] = channel(val[2], y[j], p.yOrigin, p.yout);
      }
      break;
  }
}

// the outer ghost layer of one axis: u(ghost) = 2 bc - u(first interior);
// x over (j, k) of 0..ny+1 x 0..nz+1, y over (i, k) of 0..nx x 0..nz+1,
// z over (i, j) of 0..nx x 0..ny+1
template <int AXIS>
__global__ void k_outer_ghost(Dims d, double *u, double *v, double *w, BCArr B) {
  const long long n1 = AXIS == 0 ? d.NY : d.nx + 1, n2 = AXIS == 2 ? d.NY : d.nz + 2;
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n1 * n2) return;
  const int p = (int)(e % n1), q = (int)(e / n1);
  double *F[3] = {u, v, w};
  long long g0, g1, i0, i1, b0, b1;
  if (AXIS == 0) {
    g0 = d.id(0, p, q); i0 = d.id(1, p, q); g1 = d.id(d.nx, p, q); i1 = d.id(d.nx - 1, p, q);
    b0 = 2 * (p + d.NY * (long long)q); b1 = b0 + 1;
  } else if (AXIS == 1) {
    g0 = d.id(p, 0, q); i0 = d.id(p, 1, q); g1 = d.id(p, d.ny, q); i1 = d.id(p, d.ny - 1, q);
    b0 = p + d.NX * (2 * (long long)q); b1 = b0 + d.NX;
  } else {
    g0 = d.id(p, q, 0); i0 = d.id(p, q, 1); g1 = d.id(p, q, d.nz); i1 = d.id(p, q, d.nz - 1);
    b0 = p + d.NX * (long long)q; b1 = b0 + d.NX * d.NY;
  }
  for (int a = 0; a < 3; ++a) {
    const double *bc = B.a[3 * AXIS + a];
    F[a][g0] = 2.0 * bc[b0] - F[a][i0];
    F[a][g1] = 2.0 * bc[b1] - F[a][i1];
  }
}

}  // namespace ad
}  // namespace fg

using namespace fg;

namespace {

// set_solve_ad on the host (CORE_SET_SOLVERS.F90:650-675) and the metric
// arrays, uploaded into the case's buffer when the time step or the
// viscosity changed
fg_status ad_setup(fg_case *c, const fg_ad_params *prm, ad::Met &m, ad::Dims &d) {
  if (!c->prepared) {
    fg_status st = fg_mg_prepare(c);
    if (st != FG_OK) return st;
  }
  const HLevel &L = c->lev[0];
  const int n[3] = {c->nx, c->ny, c->nz};
  const size_t all = 4 * ((size_t)n[0] + n[1] + n[2] + 6);
  if (!c->d_admet || c->admet_dt != prm->dt || c->admet_nu != prm->reinv) {
    const double nu = prm->reinv, dt = prm->dt;
    const std::vector<double> *x[3] = {&L.x, &L.y, &L.z}, *xc[3] = {&L.xc, &L.yc, &L.zc};
    const std::vector<double> *di[3] = {&L.dxinv, &L.dyinv, &L.dzinv}, *dci[3] = {&L.dxcinv, &L.dycinv, &L.dzcinv};
    std::vector<double> v;
    v.reserve(all);
    for (int a = 0; a < 3; ++a) {
      const size_t N = (size_t)n[a] + 2;
      std::vector<double> f(N, 0.0), am(N, 0.0), ap(N, 0.0);
      for (int i = 1; i <= n[a]; ++i) f[i] = ((*x[a])[i] - (*xc[a])[i - 1]) / ((*xc[a])[i] - (*xc[a])[i - 1]);
      for (int i = 1; i <= n[a] - 1; ++i) {
        am[i] = (*dci[a])[i] * (*di[a])[i];
        ap[i] = (*dci[a])[i + 1] * (*di[a])[i];
        am[i] = -(0.50 * dt * nu) * am[i];
        ap[i] = -(0.50 * dt * nu) * ap[i];
      }
      for (const std::vector<double> *p : {(const std::vector<double> *)&f, di[a], (const std::vector<double> *)&am,
                                           (const std::vector<double> *)&ap})
        v.insert(v.end(), p->begin(), p->begin() + N);
    }
    if (!c->d_admet) FG_CUDA(fg::dev_alloc(&c->d_admet, all * sizeof(double)));
    FG_CUDA(cudaMemcpyAsync(c->d_admet, v.data(), all * sizeof(double), cudaMemcpyHostToDevice, c->stream));
    FG_CUDA(cudaStreamSynchronize(c->stream));  // v is pageable and goes out of scope
    c->admet_dt = dt;
    c->admet_nu = nu;
  }
  const double *p = c->d_admet;
  for (int a = 0; a < 3; ++a) {
    const size_t N = (size_t)n[a] + 2;
    m.a[a] = {p, p + N, p + 2 * N, p + 3 * N};
    p += 4 * N;
  }
  d.nx = n[0]; d.ny = n[1]; d.nz = n[2];
  d.NX = (long long)n[0] + 2; d.NY = (long long)n[1] + 2;
  return FG_OK;
}

bool ad_params_ok(const fg_ad_params *p) {
  return p && p->dt > 0.0 && std::isfinite(p->reinv) && std::isfinite(p->omega_ad);
}

bool bc_arrays_ok(const fg_velocity_bc_arrays *b) {
  return b && b->bcxu && b->bcxv && b->bcxw && b->bcyu && b->bcyv && b->bcyw && b->bczu && b->bczv && b->bczw;
}

ad::BCArr bc_arr(const fg_velocity_bc_arrays *b) {
  ad::BCArr B;
  double *const src[9] = {b->bcxu, b->bcxv, b->bcxw, b->bcyu, b->bcyv, b->bcyw, b->bczu, b->bczv, b->bczw};
  for (int q = 0; q < 9; ++q) B.a[q] = src[q];
  return B;
}

// the grid dimensions alone (the boundary kernels need no coefficients)
fg_status dims_setup(fg_case *c, ad::Dims &d) {
  if (!c->prepared) {
    fg_status st = fg_mg_prepare(c);
    if (st != FG_OK) return st;
  }
  d.nx = c->nx; d.ny = c->ny; d.nz = c->nz;
  d.NX = (long long)c->nx + 2; d.NY = (long long)c->ny + 2;
  return FG_OK;
}

unsigned blocks_of(long long n) { return (unsigned)((n + 255) / 256); }

// set_outer_velocity_bc's face data; the pulsatile values with the host's
// sin, pi = 4 atan(1) (CORE_SET_OUTER_BC.F90:40-42)
bool vel_bc(const fg_velocity_bc *vb, ad::VelBC &p) {
  const double pi = 4.0 * std::atan(1.0), t = vb->time;
  for (int f = 0; f < 6; ++f) {
    if (vb->type[f] < 1 || vb->type[f] > 6) return false;
    p.type[f] = vb->type[f];
    for (int a = 0; a < 3; ++a) {
      p.val[f][a] = vb->val[f][a];
      p.puls[f][a] = vb->val[f][a] * std::sin(2.0 * pi * vb->freq[f][a] * t);
    }
  }
  p.puls[0][0] = vb->val[0][0] * t / 30.0;
  p.yOrigin = vb->yOrigin; p.yout = vb->yout; p.zOrigin = vb->zOrigin; p.zout = vb->zout;
  return true;
}

// the three face kernels of set_outer_velocity_bc, in the reference's order
fg_status enqueue_outer_bc(fg_case *c, const ad::Dims &d, const double *u, const double *v, const double *w,
                           const fg_velocity_bc_arrays *bc, const fg_velocity_bc *vb) {
  ad::VelBC p;
  if (!vel_bc(vb, p)) return FG_BAD_INPUT;
  const HLevel &L = c->lev[0];
  if (!c->d_vbcmet) {
    std::vector<double> yz(L.y);
    yz.insert(yz.end(), L.z.begin(), L.z.end());
    FG_CUDA(fg::dev_alloc(&c->d_vbcmet, yz.size() * sizeof(double)));
    FG_CUDA(cudaMemcpy(c->d_vbcmet, yz.data(), yz.size() * sizeof(double), cudaMemcpyHostToDevice));
  }
  const double *y = c->d_vbcmet, *z = c->d_vbcmet + d.NY;
  const ad::Vel U = {{u, v, w}};
  const ad::BCArr B = bc_arr(bc);
  cudaStream_t s = c->stream;
  ad::k_outer_bc_x<<<blocks_of(2 * d.NY * (d.nz + 2)), 256, 0, s>>>(d, p, y, U, B);
  ad::k_outer_bc_y<<<blocks_of(2 * (long long)(d.nx + 1) * (d.nz + 2)), 256, 0, s>>>(d, p, z, U, B);
  ad::k_outer_bc_z<<<blocks_of(2 * (long long)(d.nx + 1) * d.NY), 256, 0, s>>>(d, p, y, U, B);
  note_launches(3);
  FG_CUDA(cudaGetLastError());
  return FG_OK;
}

fg_status enqueue_outer_ghost(fg_case *c, const ad::Dims &d, double *u, double *v, double *w,
                              const fg_velocity_bc_arrays *bc) {
  const ad::BCArr B = bc_arr(bc);
  cudaStream_t s = c->stream;
  ad::k_outer_ghost<0><<<blocks_of(d.NY * (d.nz + 2)), 256, 0, s>>>(d, u, v, w, B);
  ad::k_outer_ghost<1><<<blocks_of((long long)(d.nx + 1) * (d.nz + 2)), 256, 0, s>>>(d, u, v, w, B);
  ad::k_outer_ghost<2><<<blocks_of((long long)(d.nx + 1) * d.NY), 256, 0, s>>>(d, u, v, w, B);
  note_launches(3);
  FG_CUDA(cudaGetLastError());
  return FG_OK;
}

}  // namespace

namespace {

// rows one thread of k_ad_sweeps holds for lines of up to n cells, 0 when a
// line is too long for it
int sweep_rows(int n) { return n <= ad::SW_ROW_THREADS ? 1 : n <= 1024 ? 2 : n <= 2048 ? 4 : 0; }

template <int R, int NC>
cudaError_t launch_sweeps(const ad::Dims &d, const ad::Met &m, const int8_t *ib, const int8_t *gh,
                          const ad::Comps<NC> &C, const ad::Faces &F, double half_dt, double omega,
                          const double *binv, long long nref, const ad::SweepSync &sync, cudaStream_t s) {
  const int n = std::max(d.nx, std::max(d.ny, d.nz));
  const int rows = ((n - 1 + R - 1) / R + 31) / 32 * 32;
  const size_t sm = (size_t)(n + 1) * (3 + 2 * NC) * sizeof(double);
  auto kern = ad::k_ad_sweeps<R, NC>;
  if (sm > 48 * 1024) {
    const cudaError_t e = allow_smem(kern);
    if (e != cudaSuccess) return e;
  }
  kern<<<2 * (d.nz - 1) + d.ny - 1, ad::SW_ROLES + rows, sm, s>>>(d, m, ib, gh, C, F, half_dt, omega, binv, nref, sync);
  return cudaGetLastError();
}

// a sweep along AXIS one anti-diagonal at a time
template <int AXIS, int NC>
void diag_sweep(const ad::Dims &d, const ad::Met &m, const int8_t *ib, const int8_t *gh, const ad::Comps<NC> &C,
                const ad::Faces &F, double half_dt, double omega, double *scr, cudaStream_t s, long long &launches) {
  const int np = AXIS == 0 ? d.ny - 1 : d.nx - 1, nq = AXIS == 2 ? d.ny - 1 : d.nz - 1;
  for (int e = 0; e < NC; ++e)
    for (int diag = 2; diag <= np + nq; ++diag) {
      const int nl = std::min(np, diag - 1) - std::max(1, diag - nq) + 1;
      ad::k_ad_diag<AXIS><<<(unsigned)((nl + 63) / 64), 64, 0, s>>>(d, m, ib, gh, C.v[e], C.r[e], F, half_dt, omega,
                                                                    diag, scr);
      ++launches;
    }
}

// one itsolv_ad pass of NC components: x, then y, then z sweeps
template <int NC>
fg_status ad_sweeps(fg_case *c, const ad::Comps<NC> &C, const ad::Faces &F, const fg_ad_params *prm) {
  cudaSetDevice(c->device);
  ad::Met m;
  ad::Dims d;
  fg_status st = ad_setup(c, prm, m, d);
  if (st != FG_OK) return st;
  const size_t nref = (size_t)(c->nx + 2) * (c->ny + 2) * (c->nz + 2);
  const int8_t *ib = c->d_refmask, *gh = c->d_refmask + nref;
  const double half_dt = prm->crank_nicolson ? 0.5 * prm->dt : 0.0, om = prm->omega_ad;
  const int nmax = std::max(c->nx, std::max(c->ny, c->nz));
  int rows = sweep_rows(nmax);
  // scratch: the pivots of the three directions, an error flag, a ticket and
  // the columns' progress; for lines too long for k_ad_sweeps, and where
  // the three fields of pivots cannot be had, one line per thread of a
  // diagonal
  double *ws = nullptr;
  cudaError_t e = cudaErrorMemoryAllocation;
  const size_t nsync = 2 + 3 * (size_t)nmax;
  if (rows) {
    e = fg::dev_alloc(&ws, 3 * nref * sizeof(double) + nsync * sizeof(int));
    if (e == cudaErrorMemoryAllocation) {
      (void)cudaGetLastError();
      rows = 0;
    }
  }
  if (!rows) {
    const int lmax = std::max(std::min(c->ny, c->nz), std::max(std::min(c->nx, c->nz), std::min(c->nx, c->ny)));
    e = fg::dev_alloc(&ws, (size_t)lmax * 2 * (nmax + 1) * sizeof(double));
  }
  FG_CUDA(e);
  cudaStream_t s = c->stream;
  long long launches = 0;
  int *sync = reinterpret_cast<int *>(ws + 3 * nref);
  if (rows) {
    const double *binv = ws;
    const ad::SweepSync sy = {sync, sync + 1, {sync + 2, sync + 2 + nmax, sync + 2 + 2 * nmax}};
    e = cudaMemsetAsync(sync, 0, nsync * sizeof(int), s);
    const size_t ft = 2 * sizeof(ad::FactorTile);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(ad::k_ad_factor, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ft);
    if (e == cudaSuccess) {
      auto groups = [](int np, int nq) { return (np + ad::FT_LINES - 1) / ad::FT_LINES * nq; };
      const int nb =
          std::max(groups(d.ny - 1, d.nz - 1), std::max(groups(d.nx - 1, d.nz - 1), groups(d.nx - 1, d.ny - 1)));
      ad::k_ad_factor<<<dim3(nb, 3), 32 + ad::FT_WORK, ft, s>>>(d, m, ib, gh, F, half_dt, ws, (long long)nref);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
      launches = 2;
      const long long nr = (long long)nref;
      e = rows == 1   ? launch_sweeps<1, NC>(d, m, ib, gh, C, F, half_dt, om, binv, nr, sy, s)
          : rows == 2 ? launch_sweeps<2, NC>(d, m, ib, gh, C, F, half_dt, om, binv, nr, sy, s)
                      : launch_sweeps<4, NC>(d, m, ib, gh, C, F, half_dt, om, binv, nr, sy, s);
    }
  } else {
    diag_sweep<0, NC>(d, m, ib, gh, C, F, half_dt, om, ws, s, launches);
    diag_sweep<1, NC>(d, m, ib, gh, C, F, half_dt, om, ws, s, launches);
    diag_sweep<2, NC>(d, m, ib, gh, C, F, half_dt, om, ws, s, launches);
    e = cudaGetLastError();
  }
  note_launches(launches);
  int gave_up = 0;
  if (e == cudaSuccess && rows) e = cudaMemcpyAsync(&gave_up, sync, sizeof(int), cudaMemcpyDeviceToHost, s);
  const cudaError_t es = cudaStreamSynchronize(s);
  if (e == cudaSuccess) e = es;
  {
    fg::IdleFree drained;  // the stream that used the scratch is idle
    fg::dev_free(ws);
  }
  if (e != cudaSuccess) {
    set_last_error(cudaGetErrorString(e), __FILE__, __LINE__);
    return FG_CUDA_ERROR;
  }
  return gave_up ? FG_TIMEOUT : FG_OK;
}

// calc_residual_ad of NC components: resm[c] and loc[3 c ..]
template <int NC>
fg_status ad_residuals(fg_case *c, const ad::Comps<NC> &C, const ad::Faces &F, const fg_ad_params *prm,
                       double *resm, int *loc) {
  cudaSetDevice(c->device);
  ad::Met m;
  ad::Dims d;
  fg_status st = ad_setup(c, prm, m, d);
  if (st != FG_OK) return st;
  const size_t nref = (size_t)(c->nx + 2) * (c->ny + 2) * (c->nz + 2);
  const int8_t *ib = c->d_refmask, *gh = c->d_refmask + nref;
  const double half_dt = prm->crank_nicolson ? 0.5 * prm->dt : 0.0;
  const long long nt = (long long)(c->nx - 1) * (c->ny - 1) * (c->nz - 1);
  const unsigned nb = (unsigned)((nt + 255) / 256);
  double *pv = nullptr;
  FG_CUDA(fg::dev_alloc(&pv, (2 * NC * (size_t)nb + 2 * NC) * sizeof(double)));
  long long *pi = reinterpret_cast<long long *>(pv + NC * (size_t)nb);
  double *out = pv + 2 * NC * (size_t)nb;
  ad::k_ad_resid<NC><<<nb, 256, 0, c->stream>>>(d, m, ib, gh, C, F, half_dt, pv, pi);
  ad::k_ad_resid_max<<<NC, 1024, 0, c->stream>>>(pv, pi, (int)nb, out);
  note_launches(2);
  cudaError_t e = cudaGetLastError();
  double h[2 * NC] = {};
  if (e == cudaSuccess) e = cudaMemcpyAsync(h, out, sizeof(h), cudaMemcpyDeviceToHost, c->stream);
  const cudaError_t es = cudaStreamSynchronize(c->stream);
  if (e == cudaSuccess) e = es;
  {
    fg::IdleFree drained;  // the stream that used the scratch is idle
    fg::dev_free(pv);
  }
  if (e != cudaSuccess) {
    set_last_error(cudaGetErrorString(e), __FILE__, __LINE__);
    return FG_CUDA_ERROR;
  }
  const long long ni = c->nx - 1, nj = c->ny - 1;
  for (int a = 0; a < NC; ++a) {
    const double v = h[2 * a];
    const long long at = (long long)h[2 * a + 1];
    resm[a] = v;
    if (!loc) continue;
    loc[3 * a] = v > 0.0 ? 1 + (int)(at % ni) : 1;
    loc[3 * a + 1] = v > 0.0 ? 1 + (int)((at / ni) % nj) : 1;
    loc[3 * a + 2] = v > 0.0 ? 1 + (int)(at / (ni * nj)) : 1;
  }
  return FG_OK;
}

}  // namespace

extern "C" {

fg_status fg_itsolv_ad_device(fg_case *c, double *var, const double *r, const double *face_u, const double *face_v,
                              const double *face_w, const fg_ad_params *prm) {
  if (!c || !var || !r || !face_u || !face_v || !face_w || !ad_params_ok(prm)) return FG_BAD_INPUT;
  return ad_sweeps<1>(c, {{var}, {r}}, {{face_u, face_v, face_w}}, prm);
}

fg_status fg_calc_residual_ad_device(fg_case *c, const double *var, const double *r, const double *face_u,
                                     const double *face_v, const double *face_w, const fg_ad_params *prm,
                                     double *resm, int *loc) {
  if (!c || !var || !r || !face_u || !face_v || !face_w || !ad_params_ok(prm) || !resm) return FG_BAD_INPUT;
  return ad_residuals<1>(c, {{const_cast<double *>(var)}, {r}}, {{face_u, face_v, face_w}}, prm, resm, loc);
}

fg_status fg_set_outer_velocity_bc_device(fg_case *c, const double *u, const double *v, const double *w,
                                          const fg_velocity_bc_arrays *bc, const fg_velocity_bc *vb) {
  if (!c || !u || !v || !w || !bc_arrays_ok(bc) || !vb) return FG_BAD_INPUT;
  cudaSetDevice(c->device);
  ad::Dims d;
  fg_status st = dims_setup(c, d);
  if (st == FG_OK) st = enqueue_outer_bc(c, d, u, v, w, bc, vb);
  if (st != FG_OK) return st;
  FG_CUDA(cudaStreamSynchronize(c->stream));
  return FG_OK;
}

fg_status fg_set_outer_ghost_velocity_device(fg_case *c, double *u, double *v, double *w,
                                             const fg_velocity_bc_arrays *bc) {
  if (!c || !u || !v || !w || !bc_arrays_ok(bc)) return FG_BAD_INPUT;
  cudaSetDevice(c->device);
  ad::Dims d;
  fg_status st = dims_setup(c, d);
  if (st == FG_OK) st = enqueue_outer_ghost(c, d, u, v, w, bc);
  if (st != FG_OK) return st;
  FG_CUDA(cudaStreamSynchronize(c->stream));
  return FG_OK;
}

fg_status fg_solve_ad_device(fg_case *c, double *u, double *v, double *w, const double *nlu, const double *nlv,
                             const double *nlw, double *face_u, double *face_v, double *face_w,
                             const fg_velocity_bc_arrays *bc, const double *ubi_ghost, const double *ubi_dead,
                             const fg_ad_params *prm, const fg_velocity_bc *vb, int itermax_gc, double restol_gcv,
                             int itermax_ad, double restol_ad, fg_solve_ad_stats *stats) {
  if (!c || !u || !v || !w || !nlu || !nlv || !nlw || !face_u || !face_v || !face_w || !bc_arrays_ok(bc) ||
      !ad_params_ok(prm) || !vb || itermax_ad < 0)
    return FG_BAD_INPUT;
  ad::VelBC chk;
  if (!vel_bc(vb, chk)) return FG_BAD_INPUT;
  int vzg[6];
  for (int f = 0; f < 6; ++f) vzg[f] = vb->type[f] == 2;
  // u, v, w sweep together: a pass reads its own component and the faces
  const ad::Comps<3> C = {{u, v, w}, {nlu, nlv, nlw}};
  const ad::Faces F = {{face_u, face_v, face_w}};
  int iter = 0, loc[3] = {1, 1, 1};
  double res2 = 1.0e10;
  fg_status st = FG_OK;
  while (st == FG_OK && iter < itermax_ad && res2 > restol_ad) {
    st = ad_sweeps<3>(c, C, F, prm);
    if (st == FG_OK) st = fg_ghostcell_velocity_device(c, u, v, w, ubi_ghost, ubi_dead, itermax_gc, restol_gcv, nullptr);
    if (st == FG_OK) st = fg_face_vel_device(c, u, v, w, bc->bcxu, bc->bcyv, bc->bczw, face_u, face_v, face_w);
    if (st == FG_OK)
      st = fg_enforce_global_mass_consv_device(c, face_u, face_v, face_w, bc->bcxu, bc->bcyv, bc->bczw, vzg);
    if (st == FG_OK) st = fg_set_outer_velocity_bc_device(c, u, v, w, bc, vb);
    if (st == FG_OK) st = fg_set_outer_ghost_velocity_device(c, u, v, w, bc);
    double r[3] = {0.0, 0.0, 0.0};
    int l[3][3];
    if (st == FG_OK) st = ad_residuals<3>(c, C, F, prm, r, &l[0][0]);
    if (st != FG_OK) break;
    int best = 0;
    res2 = std::fabs(r[0]);
    for (int a = 1; a < 3; ++a)
      if (std::fabs(r[a]) > res2) { res2 = std::fabs(r[a]); best = a; }
    std::memcpy(loc, l[best], sizeof(loc));
    ++iter;
  }
  if (stats) {
    stats->iterations = iter;
    stats->residual = res2;
    std::memcpy(stats->loc, loc, sizeof(loc));
  }
  return st;
}

}  // extern "C"
