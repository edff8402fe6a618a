// fg_proj.cu -- the steps either side of the pressure solve on the device:
// face velocities (CORE_FRAC_STEP_ROUTINES.F90 face_vel), global mass
// conservation on zero-gradient outflow faces and the Poisson right-hand
// side (CORE_SET_OUTER_BC.F90 enforce_global_mass_consv, CORE_POISSON.F90
// rhs_poisson), and the velocity correction with the pressure gradient
// (CORE_FRAC_STEP_ROUTINES.F90 correct_vel, calc_pres_grad).  Fields are
// device arrays in the reference layout (0:nx+1, 0:ny+1, 0:nz+1), node
// counts; the face-velocity boundary arrays are the reference's bcxu(0:1,
// 0:ny+1, 0:nz+1), bcyv(0:nx+1, 0:1, 0:nz+1), bczw(0:nx+1, 0:ny+1, 0:1).
// With these, a time step's div and pPrime stay on the device from the
// face velocities to the corrected velocity.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "fg_case.h"
#include "fg_internal.h"

namespace fg {
namespace proj {

// the reference's 1-D grid arrays of the finest level, reference indexing
// (n+2 entries each): widths, their inverses, and the share of cell i in the
// value at its lower node (CORE_GRID.F90:194-202)
struct Met {
  const double *dx, *dy, *dz, *dxi, *dyi, *dzi, *fx, *fy, *fz;
};

struct Dims {
  int nx, ny, nz;  // node counts
  long long NX, NY;
  __device__ __forceinline__ long long id(int i, int j, int k) const { return i + NX * (j + NY * (long long)k); }
};

// The field kernels are bound by DRAM.  A block takes PJ_I x PJ_J columns of
// cells and a thread walks `kspan` planes of its column, so that the plane
// below or above it has just read stays in registers, the row next to it in
// L1, and nothing divides by a runtime extent.  On 512x256x256 cells (each
// thread one cell found by 64-bit divisions, the interpolation factors
// divided out per cell, before): face velocities 587 -> 319 us, divergence
// with the flux 251 + 362 -> 258 us, correction 739 -> 337 us; a plain
// copy's rate would take 254, 180 and 300 us.
constexpr int PJ_I = 64, PJ_J = 4, PJ_K = 8;
struct Col {
  int i, j, k0, k1;  // cells k0 <= k < k1
  bool ok;
};
__device__ __forceinline__ Col column(const Dims &d, int kspan) {
  Col c;
  c.i = 1 + blockIdx.x * PJ_I + threadIdx.x;
  c.j = 1 + blockIdx.y * PJ_J + threadIdx.y;
  c.k0 = 1 + blockIdx.z * kspan;
  c.k1 = min(c.k0 + kspan, d.nz);
  c.ok = c.i < d.nx && c.j < d.ny;
  return c;
}

// face_vel: face_u(i) for i = 2..nx-1 from the cell velocities, i = 1 and
// nx from bcxu (faces v, w alike); one thread per interior cell, which
// writes its own faces and, on the last cell of a line, the far boundary
__global__ void __launch_bounds__(PJ_I * PJ_J)
k_face_vel(Dims d, Met m, int kspan, const double *__restrict__ u, const double *__restrict__ v,
           const double *__restrict__ w, const double *__restrict__ bcxu, const double *__restrict__ bcyv,
           const double *__restrict__ bczw, double *__restrict__ fu, double *__restrict__ fv,
           double *__restrict__ fw) {
  const Col c = column(d, kspan);
  if (!c.ok) return;
  const int i = c.i, j = c.j;
  const double fi = m.fx[i], fj = m.fy[j];
  double wm = w[d.id(i, j, c.k0 - 1)];
#pragma unroll 4
  for (int k = c.k0; k < c.k1; ++k) {
    const long long id = d.id(i, j, k);
    const double wc = w[id];
    fu[id] = i >= 2 ? fi * u[id] + (1.0 - fi) * u[id - 1] : bcxu[2 * (j + d.NY * (long long)k)];
    fv[id] = j >= 2 ? fj * v[id] + (1.0 - fj) * v[id - d.NX] : bcyv[i + d.NX * (2 * (long long)k)];
    const double fk = m.fz[k];
    fw[id] = k >= 2 ? fk * wc + (1.0 - fk) * wm : bczw[i + d.NX * (long long)j];
    if (i == d.nx - 1) fu[id + 1] = bcxu[1 + 2 * (j + d.NY * (long long)k)];
    if (j == d.ny - 1) fv[id + d.NX] = bcyv[i + d.NX * (1 + 2 * (long long)k)];
    if (k == d.nz - 1) fw[id + d.NX * d.NY] = bczw[i + d.NX * (j + d.NY)];
    wm = wc;
  }
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
  return v;
}
// block sums of a and maximum of b (NW warps) in thread 0
template <int NW>
__device__ __forceinline__ void block_sum_max(double &a, double &b) {
  __shared__ double ra[NW], rb[NW];
  const int t = threadIdx.x + blockDim.x * threadIdx.y;
  a = warp_sum(a);
  b = warp_max(b);
  if ((t & 31) == 0) { ra[t >> 5] = a; rb[t >> 5] = b; }
  __syncthreads();
  if (t == 0) {
    double s = 0.0, x = 0.0;
    for (int q = 0; q < NW; ++q) { s += ra[q]; x = fmax(x, rb[q]); }
    a = s;
    b = x;
  }
  __syncthreads();
}

// the first of the flagged faces (bit f of vzg: x1, x2, y1, y2, z1, z2) whose
// cell layer holds (i, j, k); 6: none
__device__ __forceinline__ int layer_of(const Dims &d, int vzg, int i, int j, int k) {
  const unsigned at = (i == 1 ? 1u : 0u) | (i == d.nx - 1 ? 2u : 0u) | (j == 1 ? 4u : 0u) | (j == d.ny - 1 ? 8u : 0u) |
                      (k == 1 ? 16u : 0u) | (k == d.nz - 1 ? 32u : 0u);
  const unsigned hit = at & (unsigned)vzg;
  return hit ? __ffs(hit) - 1 : 6;
}

// rhs_poisson and the net mass flux in one pass: div on the fluid non-ghost
// cells (0 elsewhere), with block partials of the mass flux out of them, of
// sum div dV and of max |div|.  DIV = false: the flux alone.  The cells
// next to a zero-gradient face are left out of the last two: the flux
// correction changes their faces, and k_div_layer forms them again
// afterwards.  The blocks past the columns' nz clear div's boundary layers
// (indices 0, n and n + 1 of each axis) and the first block the counters of
// the reductions that follow: small grids are bound by the number of
// launches (24x16x16 cells, the call without and with an outflow correction:
// 35 and 49 us; with a launch each for these and for the sums 47 and 65).
template <bool DIV>
__global__ void __launch_bounds__(PJ_I * PJ_J)
k_div(Dims d, Met m, int kspan, int vzg, const int8_t *__restrict__ ib, const int8_t *__restrict__ gh,
      const double *__restrict__ fu, const double *__restrict__ fv, const double *__restrict__ fw, double dtinv,
      double *__restrict__ div, double *pflux, double *psum, double *pmax, int *count, int nz) {
  const bool first = threadIdx.x == 0 && threadIdx.y == 0;
  const int b = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
  if (first && b == 0) count[0] = count[1] = 0;
  if (DIV && blockIdx.z >= (unsigned)nz) {
    const int n0 = gridDim.x * gridDim.y * nz;
    const long long t = (long long)(b - n0) * (PJ_I * PJ_J) + threadIdx.x + PJ_I * threadIdx.y;
    const long long nt = (long long)(gridDim.x * gridDim.y * gridDim.z - n0) * (PJ_I * PJ_J);
    for (int a = 0; a < 3; ++a) {
      const int n = a == 0 ? d.nx : a == 1 ? d.ny : d.nz;
      const long long n1 = a == 0 ? d.NY : d.NX, n2 = a == 2 ? d.NY : d.nz + 2;
      for (long long e = t; e < n1 * n2; e += nt) {
        const int q = (int)(e / n1), p = (int)(e - n1 * q);
        for (const int l : {0, n, n + 1}) div[a == 0 ? d.id(l, p, q) : a == 1 ? d.id(p, l, q) : d.id(p, q, l)] = 0.0;
      }
    }
    return;
  }
  const Col c = column(d, kspan);
  double flux = 0.0, s = 0.0, mx = 0.0;
  if (c.ok) {
    const int i = c.i, j = c.j;
    const double dx = m.dx[i], dy = m.dy[j], dxi = m.dxi[i], dyi = m.dyi[j];
    const long long sz = d.NX * d.NY;
    double f0 = fw[d.id(i, j, c.k0)];
#pragma unroll 4
    for (int k = c.k0; k < c.k1; ++k) {
      const long long id = d.id(i, j, k);
      const double flag = (1.0 - (double)ib[id]) * (1.0 - (double)gh[id]);
      const double f1 = fw[id + sz], du = fu[id + 1] - fu[id], dv = fv[id + d.NX] - fv[id], dw = f1 - f0;
      const double dz = m.dz[k];
      if (vzg) flux += flag * (du * dy * dz + dv * dx * dz + dw * dx * dy);
      if (DIV) {
        const double v = dtinv * (du * dxi + dv * dyi + dw * m.dzi[k]) * flag;
        div[id] = v;
        if (layer_of(d, vzg, i, j, k) == 6) {
          s += v * dx * dy * dz;
          mx = fmax(mx, fabs(v));
        }
      }
      f0 = f1;
    }
  }
  if (vzg) {
    double none = 0.0;
    block_sum_max<PJ_I * PJ_J / 32>(flux, none);
    if (first) pflux[b] = flux;
  }
  if (DIV) {
    block_sum_max<PJ_I * PJ_J / 32>(s, mx);
    if (first) { psum[b] = s; pmax[b] = mx; }
  }
}

// div and its partials on the cells next to the zero-gradient faces, from
// the corrected faces; blockIdx.y = face, a cell of two layers belongs to the
// first
__global__ void __launch_bounds__(256)
k_div_layer(Dims d, Met m, int vzg, const int8_t *__restrict__ ib, const int8_t *__restrict__ gh,
            const double *__restrict__ fu, const double *__restrict__ fv, const double *__restrict__ fw, double dtinv,
            double *__restrict__ div, double *psum, double *pmax) {
  const int f = blockIdx.y, a = f >> 1, up = f & 1;
  double s = 0.0, mx = 0.0;
  if ((vzg >> f) & 1) {
    const int n1 = a == 0 ? d.ny - 1 : d.nx - 1, n2 = a == 2 ? d.ny - 1 : d.nz - 1;
    const int l = !up ? 1 : a == 0 ? d.nx - 1 : a == 1 ? d.ny - 1 : d.nz - 1;
    const long long e = (long long)blockIdx.x * 256 + threadIdx.x;
    if (e < (long long)n1 * n2) {
      const int p = 1 + (int)(e % n1), q = 1 + (int)(e / n1);
      const int i = a == 0 ? l : p, j = a == 0 ? p : a == 1 ? l : q, k = a == 2 ? l : q;
      if (layer_of(d, vzg, i, j, k) == f) {
        const long long id = d.id(i, j, k);
        const double flag = (1.0 - (double)ib[id]) * (1.0 - (double)gh[id]);
        const double v = dtinv * ((fu[id + 1] - fu[id]) * m.dxi[i] + (fv[id + d.NX] - fv[id]) * m.dyi[j] +
                                  (fw[id + d.NX * d.NY] - fw[id]) * m.dzi[k]) * flag;
        div[id] = v;
        s = v * m.dx[i] * m.dy[j] * m.dz[k];
        mx = fabs(v);
      }
    }
  }
  block_sum_max<8>(s, mx);
  if (threadIdx.x == 0) {
    const int b = blockIdx.x + gridDim.x * blockIdx.y;
    psum[b] = s;
    pmax[b] = mx;
  }
}

// Sums over the partials and what depends on them, up to RB blocks; the last
// one to finish adds the blocks' results in order.  AREA: out[0] = -flux / (fluid
// area of the flagged faces), the outflow correction; else out[0] = sum of
// psum, out[1] = maximum of pmax.
constexpr int RB = 64;
template <bool AREA>
__global__ void __launch_bounds__(256)
k_reduce(Dims d, Met m, const int8_t *__restrict__ ib, int vzg, const double *psum, const double *pmax, int n,
         double *blk, int *count, double *out) {
  double s = 0.0, x = 0.0;
  const int t0 = blockIdx.x * 256 + threadIdx.x, nt = gridDim.x * 256, nblk = gridDim.x;
  for (int b = t0; b < n; b += nt) {
    s += psum[b];
    if (!AREA) x = fmax(x, pmax[b]);
  }
  if (AREA) {
    for (int f = 0; f < 6; ++f) {
      if (!((vzg >> f) & 1)) continue;
      const int a = f >> 1, up = f & 1;
      const int nu = a == 0 ? d.ny - 1 : d.nx - 1, nv = a == 2 ? d.ny - 1 : d.nz - 1;
      const int layer = a == 0 ? (up ? d.nx - 1 : 1) : a == 1 ? (up ? d.ny - 1 : 1) : (up ? d.nz - 1 : 1);
      for (int e = t0; e < nu * nv; e += nt) {
        const int p = 1 + e % nu, q = 1 + e / nu;
        long long id;
        double w;
        if (a == 0) { id = d.id(layer, p, q); w = m.dy[p] * m.dz[q]; }
        else if (a == 1) { id = d.id(p, layer, q); w = m.dx[p] * m.dz[q]; }
        else { id = d.id(p, q, layer); w = m.dx[p] * m.dy[q]; }
        x += w * (1.0 - (double)ib[id]);
      }
    }
  }
  __shared__ double rs[8], rx[8];
  __shared__ bool last;
  s = warp_sum(s);
  x = AREA ? warp_sum(x) : warp_max(x);
  if ((threadIdx.x & 31) == 0) { rs[threadIdx.x >> 5] = s; rx[threadIdx.x >> 5] = x; }
  __syncthreads();
  auto store = [&](double a, double b) {
    if (AREA) out[0] = -a / b;
    else { out[0] = a; out[1] = b; }
  };
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
    for (int q = 0; q < 8; ++q) { a += rs[q]; b = AREA ? b + rx[q] : fmax(b, rx[q]); }
    last = false;
    if (nblk == 1) {
      store(a, b);
    } else {
      blk[2 * blockIdx.x] = a;
      blk[2 * blockIdx.x + 1] = b;
      __threadfence();
      last = atomicAdd(count, 1) == nblk - 1;
    }
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  __shared__ double fs[RB], fx[RB];  // read at once: one after another they cost a small grid 5 us
  if (threadIdx.x < nblk) {
    fs[threadIdx.x] = __ldcg(blk + 2 * threadIdx.x);
    fx[threadIdx.x] = __ldcg(blk + 2 * threadIdx.x + 1);
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  double a = 0.0, b = 0.0;
  for (int q = 0; q < nblk; ++q) {
    a += fs[q];
    b = AREA ? b + fx[q] : fmax(b, fx[q]);
  }
  store(a, b);
}

// the correction on the zero-gradient faces: the boundary arrays over
// every entry 0..n, the boundary face velocities over the interior
// (lower faces -, upper faces +); blockIdx.y = face
__global__ void k_massflux_apply(Dims d, int vzg, const double *cv, double *bcxu, double *bcyv, double *bczw,
                                 double *fu, double *fv, double *fw) {
  const int f = blockIdx.y;
  if (!((vzg >> f) & 1)) return;
  const int a = f >> 1, up = f & 1;
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int u1 = a == 0 ? d.ny : d.nx, v1 = a == 2 ? d.ny : d.nz;  // boundary array indices 0..u1, 0..v1
  if (e >= (long long)(u1 + 1) * (v1 + 1)) return;
  const int u = (int)(e % (u1 + 1)), v = (int)(e / (u1 + 1));
  const double c = up ? *cv : -*cv;
  if (a == 0) bcxu[up + 2 * (u + d.NY * (long long)v)] += c;
  else if (a == 1) bcyv[u + d.NX * (up + 2 * (long long)v)] += c;
  else bczw[u + d.NX * (v + d.NY * (long long)up)] += c;
  const bool in = u >= 1 && v >= 1 && u <= u1 - 1 && v <= v1 - 1;
  if (!in) return;
  if (a == 0) fu[d.id(up ? d.nx : 1, u, v)] += c;
  else if (a == 1) fv[d.id(u, up ? d.ny : 1, v)] += c;
  else fw[d.id(u, v, up ? d.nz : 1)] += c;
}

// correct_vel / calc_pres_grad: the face-interpolated gradient of p' on
// the non-iblank cells; u -= dt grad p' and/or the gradient stored.  The
// loads of CR_K planes come before their stores: a store to u may not be
// passed by the next plane's load of u, which left one plane's loads in
// flight per thread (512x256x256: 489 us plane by plane, 337 us so).
constexpr int CR_K = 4;
__global__ void __launch_bounds__(PJ_I * PJ_J)
k_correct(Dims d, Met m, int kspan, const int8_t *__restrict__ ib, const double *__restrict__ pp, double dt,
          double *__restrict__ u, double *__restrict__ v, double *__restrict__ w, double *__restrict__ gx,
          double *__restrict__ gy, double *__restrict__ gz) {
  const Col c = column(d, kspan);
  if (!c.ok) return;
  const int i = c.i, j = c.j;
  const long long sy = d.NX, sz = d.NX * d.NY;
  const double fx1 = m.fx[i + 1], fx0 = m.fx[i], fy1 = m.fy[j + 1], fy0 = m.fy[j], dxi = m.dxi[i], dyi = m.dyi[j];
  double pm = pp[d.id(i, j, c.k0 - 1)], pc = pp[d.id(i, j, c.k0)];
  for (int kb = c.k0; kb < c.k1; kb += CR_K) {
    double pk[CR_K], px1[CR_K], px0[CR_K], py1[CR_K], py0[CR_K], vel[CR_K][3];
    int8_t solid[CR_K];
#pragma unroll
    for (int q = 0; q < CR_K; ++q) {
      if (kb + q >= c.k1) break;
      const long long id = d.id(i, j, kb + q);
      pk[q] = pp[id + sz];
      px1[q] = pp[id + 1], px0[q] = pp[id - 1];
      py1[q] = pp[id + sy], py0[q] = pp[id - sy];
      solid[q] = ib[id];
      if (u) vel[q][0] = u[id], vel[q][1] = v[id], vel[q][2] = w[id];
    }
#pragma unroll
    for (int q = 0; q < CR_K; ++q) {
      const int k = kb + q;
      if (k >= c.k1) break;
      const long long id = d.id(i, j, k);
      const double fz1 = m.fz[k + 1], fz0 = m.fz[k];
      const double pe = fx1 * px1[q] + (1.0 - fx1) * pc, pw = fx0 * pc + (1.0 - fx0) * px0[q];
      const double pn = fy1 * py1[q] + (1.0 - fy1) * pc, ps = fy0 * pc + (1.0 - fy0) * py0[q];
      const double pf = fz1 * pk[q] + (1.0 - fz1) * pc, pb = fz0 * pc + (1.0 - fz0) * pm;
      const double pgx = (pe - pw) * dxi, pgy = (pn - ps) * dyi, pgz = (pf - pb) * m.dzi[k];
      const double flag = 1.0 - (double)solid[q];
      if (u) {
        u[id] = vel[q][0] - dt * pgx * flag;
        v[id] = vel[q][1] - dt * pgy * flag;
        w[id] = vel[q][2] - dt * pgz * flag;
      }
      if (gx) {
        gx[id] = pgx * flag;
        gy[id] = pgy * flag;
        gz[id] = pgz * flag;
      }
      pm = pc;
      pc = pk[q];
    }
  }
}

// update_pressure for one rank: p' = 0 on the solid cells not dead-marked -1
// (i = 0..nx, j = 0..ny+1, k = 0..nz+1) and on the domain's edge lines: i =
// 0..nx on j in {0, ny} and j = 0..ny+1 on i in {0, nx}, each in the planes
// 0, nz, nz+1, and the four k lines at (i, j) in {0, nx} x {0, ny}; then p =
// p' when p is not null.  One pass; a block takes PU_I x PU_J entries of
// planes z, z + gridDim.z, ..., the loads of PU_K of them before their
// stores (as above; 512x256x256: 164 us plane by plane, 110 us so).
constexpr int PU_I = 128, PU_J = 2, PU_K = 4;
__global__ void __launch_bounds__(PU_I * PU_J)
k_update(Dims d, const int8_t *__restrict__ ib, const int8_t *__restrict__ dead, double *__restrict__ pp,
         double *__restrict__ p) {
  const int i = blockIdx.x * PU_I + threadIdx.x, j = blockIdx.y * PU_J + threadIdx.y;
  if (i >= d.NX || j >= d.NY) return;
  const bool ci = i == 0 || i == d.nx, cj = j == 0 || j == d.ny;
  for (int kb = blockIdx.z; kb < d.nz + 2; kb += PU_K * gridDim.z) {
    double v[PU_K];
    int8_t in[PU_K], dd[PU_K];
#pragma unroll
    for (int q = 0; q < PU_K; ++q) {
      const int k = kb + q * gridDim.z;
      if (k >= d.nz + 2) break;
      const long long id = d.id(i, j, k);
      v[q] = p ? pp[id] : 0.0;
      in[q] = ib[id];
      dd[q] = dead[id];
    }
#pragma unroll
    for (int q = 0; q < PU_K; ++q) {
      const int k = kb + q * gridDim.z;
      if (k >= d.nz + 2) break;
      const long long id = d.id(i, j, k);
      const bool solid = i <= d.nx && in[q] != 0 && dd[q] != -1;
      const bool plane = k == 0 || k >= d.nz;
      const bool edge = (plane && ((cj && i <= d.nx) || ci)) || (ci && cj);
      const bool zero = solid || edge;
      if (zero) pp[id] = 0.0;
      if (p) p[id] = zero ? 0.0 : v[q];
    }
  }
}

}  // namespace proj
}  // namespace fg

using namespace fg;

namespace {

// the case's projection metrics (uploaded on first use) and its masks
fg_status proj_setup(fg_case *c, proj::Met &m, proj::Dims &d) {
  if (!c->prepared) {
    fg_status st = fg_mg_prepare(c);
    if (st != FG_OK) return st;
  }
  if (!c->d_pmet) {
    const HLevel &L = c->lev[0];
    std::vector<double> v;
    for (const std::vector<double> *a : {&L.x, &L.y, &L.z}) {
      const size_t n = a->size();
      for (size_t i = 0; i < n; ++i) v.push_back(i + 1 < n ? (*a)[i + 1] - (*a)[i] : 0.0);
    }
    for (const std::vector<double> *a : {&L.dxinv, &L.dyinv, &L.dzinv}) v.insert(v.end(), a->begin(), a->end());
    const std::vector<double> *x[3] = {&L.x, &L.y, &L.z}, *xc[3] = {&L.xc, &L.yc, &L.zc};
    for (int a = 0; a < 3; ++a)
      for (size_t i = 0; i < x[a]->size(); ++i)
        v.push_back(i > 0 ? ((*x[a])[i] - (*xc[a])[i - 1]) / ((*xc[a])[i] - (*xc[a])[i - 1]) : 0.0);
    FG_CUDA(fg::dev_alloc(&c->d_pmet, v.size() * sizeof(double)));
    FG_CUDA(cudaMemcpy(c->d_pmet, v.data(), v.size() * sizeof(double), cudaMemcpyHostToDevice));
  }
  const size_t NX = (size_t)c->nx + 2, NY = (size_t)c->ny + 2, NZ = (size_t)c->nz + 2;
  m.dx = c->d_pmet; m.dy = m.dx + NX; m.dz = m.dy + NY;
  m.dxi = m.dz + NZ; m.dyi = m.dxi + NX; m.dzi = m.dyi + NY;
  m.fx = m.dzi + NZ; m.fy = m.fx + NX; m.fz = m.fy + NY;
  d.nx = c->nx; d.ny = c->ny; d.nz = c->nz;
  d.NX = (long long)NX; d.NY = (long long)NY;
  return FG_OK;
}

// the columns of a field kernel: planes per thread as long as the blocks
// fill the GPU a few times over
struct Cols {
  dim3 grid, block;
  int kspan;
  int blocks() const { return (int)(grid.x * grid.y * grid.z); }
};
Cols columns(const fg_case *c) {
  Cols q;
  q.block = dim3(proj::PJ_I, proj::PJ_J);
  q.grid.x = (c->nx - 1 + proj::PJ_I - 1) / proj::PJ_I;
  q.grid.y = (c->ny - 1 + proj::PJ_J - 1) / proj::PJ_J;
  q.kspan = proj::PJ_K;
  while (q.kspan > 1 && (long long)q.grid.x * q.grid.y * ((c->nz - 1 + q.kspan - 1) / q.kspan) < 4 * 148) q.kspan /= 2;
  q.grid.z = (c->nz - 1 + q.kspan - 1) / q.kspan;
  return q;
}
// slices of blocks that clear a field's boundary layers beside such columns:
// about four index pairs of an axis's planes per thread
unsigned boundary_slices(const fg_case *c, const Cols &q) {
  const long long x = c->nx + 2, y = c->ny + 2, z = c->nz + 2;
  const long long slice = 4ll * proj::PJ_I * proj::PJ_J * q.grid.x * q.grid.y;
  return (unsigned)((x * y + y * z + x * z + slice - 1) / slice);
}
long long face_cells(const fg_case *c, int extra) {
  const long long x = c->nx + extra, y = c->ny + extra, z = c->nz + extra;
  return std::max(x * y, std::max(y * z, x * z));
}
unsigned face_blocks(const fg_case *c, int extra) { return (unsigned)((face_cells(c, extra) + 255) / 256); }
// blocks of a reduction over n values, four per thread
unsigned reduce_blocks(long long n) { return (unsigned)std::min<long long>(proj::RB, std::max(1ll, (n + 1023) / 1024)); }

// device scratch of one call, given back when its stream has been waited for
struct Scratch {
  double *p = nullptr;
  ~Scratch() {
    fg::IdleFree drained;
    fg::dev_free(p);
  }
};

int zero_gradient_faces(const int *vel_zero_gradient) {
  int vzg = 0;
  if (vel_zero_gradient)
    for (int f = 0; f < 6; ++f)
      if (vel_zero_gradient[f]) vzg |= 1 << f;
  return vzg;
}

// the outflow correction from the flux partials (cols blocks) into *cv, then
// onto the faces and boundary arrays
void enqueue_correction(fg_case *c, const proj::Met &m, const proj::Dims &d, int vzg, int nb, double *fu, double *fv,
                        double *fw, double *bcxu, double *bcyv, double *bczw, const double *part, double *blk,
                        int *count, double *cv) {
  cudaStream_t s = c->stream;
  proj::k_reduce<true><<<reduce_blocks(std::max<long long>(nb, face_cells(c, 0))), 256, 0, s>>>(
      d, m, c->d_refmask, vzg, part, nullptr, nb, blk, count, cv);
  proj::k_massflux_apply<<<dim3(face_blocks(c, 1), 6), 256, 0, s>>>(d, vzg, cv, bcxu, bcyv, bczw, fu, fv, fw);
}

}  // namespace

extern "C" {

fg_status fg_face_vel_device(fg_case *c, const double *u, const double *v, const double *w, const double *bcxu,
                             const double *bcyv, const double *bczw, double *face_u, double *face_v,
                             double *face_w) {
  if (!c || !u || !v || !w || !bcxu || !bcyv || !bczw || !face_u || !face_v || !face_w) return FG_BAD_INPUT;
  cudaSetDevice(c->device);
  proj::Met m;
  proj::Dims d;
  fg_status st = proj_setup(c, m, d);
  if (st != FG_OK) return st;
  const Cols q = columns(c);
  proj::k_face_vel<<<q.grid, q.block, 0, c->stream>>>(d, m, q.kspan, u, v, w, bcxu, bcyv, bczw, face_u, face_v, face_w);
  note_launches(1);
  FG_CUDA(cudaGetLastError());
  FG_CUDA(cudaStreamSynchronize(c->stream));
  return FG_OK;
}

fg_status fg_rhs_poisson_device(fg_case *c, double *face_u, double *face_v, double *face_w, double *bcxu,
                                double *bcyv, double *bczw, const int *vel_zero_gradient, double dt, double *div,
                                double *sumd, double *resdiv) {
  if (!c || !face_u || !face_v || !face_w || !div || !(dt > 0.0)) return FG_BAD_INPUT;
  const int vzg = zero_gradient_faces(vel_zero_gradient);
  if (vzg && (!bcxu || !bcyv || !bczw)) return FG_BAD_INPUT;
  cudaSetDevice(c->device);
  proj::Met m;
  proj::Dims d;
  fg_status st = proj_setup(c, m, d);
  if (st != FG_OK) return st;
  const size_t nref = (size_t)(c->nx + 2) * (c->ny + 2) * (c->nz + 2);
  const int8_t *ib = c->d_refmask, *gh = c->d_refmask + nref;
  const Cols q = columns(c);
  const int nb = q.blocks();
  const unsigned lb = vzg ? face_blocks(c, 0) : 0;  // blocks per face of the layers next to the outflow
  const int nl = 6 * (int)lb;
  // flux, sum and maximum partials (the layers' after the blocks'), block
  // results, the correction, the two results; two counters
  Scratch w;
  const size_t np = (size_t)nb + 2 * (size_t)(nb + nl);
  FG_CUDA(fg::dev_alloc(&w.p, (np + 4 * proj::RB + 3 + 1) * sizeof(double)));
  double *flux = w.p, *psum = flux + nb, *pmax = psum + nb + nl, *blk = pmax + nb + nl, *res = blk + 4 * proj::RB;
  int *count = reinterpret_cast<int *>(res + 3);
  cudaStream_t s = c->stream;
  const double dtinv = 1.0 / dt;
  dim3 grid = q.grid;
  grid.z += boundary_slices(c, q);
  proj::k_div<true><<<grid, q.block, 0, s>>>(d, m, q.kspan, vzg, ib, gh, face_u, face_v, face_w, dtinv, div, flux, psum,
                                             pmax, count, (int)q.grid.z);
  if (vzg) {
    enqueue_correction(c, m, d, vzg, nb, face_u, face_v, face_w, bcxu, bcyv, bczw, flux, blk, count, res + 2);
    proj::k_div_layer<<<dim3(lb, 6), 256, 0, s>>>(d, m, vzg, ib, gh, face_u, face_v, face_w, dtinv, div, psum + nb,
                                                  pmax + nb);
  }
  // a small grid's partials are fewer bytes than a launch is worth: summed
  // here (24x16x16 cells, 60 partials, the call 35 us so and 42 with the
  // reduction's launch; 64^3 cells, 1008 partials, 45 and 50 us)
  const int npart = nb + nl;
  const bool here = npart <= 1024;
  if (!here)
    proj::k_reduce<false><<<reduce_blocks(npart), 256, 0, s>>>(d, m, ib, 0, psum, pmax, npart, blk + 2 * proj::RB,
                                                               count + 1, res);
  note_launches((vzg ? 4 : 1) + (here ? 0 : 1));
  cudaError_t e = cudaGetLastError();
  double h[2] = {0.0, 0.0}, part[2 * 1024];
  if (e == cudaSuccess)
    e = here ? cudaMemcpyAsync(part, psum, 2 * npart * sizeof(double), cudaMemcpyDeviceToHost, s)
             : cudaMemcpyAsync(h, res, sizeof(h), cudaMemcpyDeviceToHost, s);
  const cudaError_t es = cudaStreamSynchronize(s);
  if (e == cudaSuccess) e = es;
  for (int q = 0; here && e == cudaSuccess && q < npart; ++q) {
    h[0] += part[q];
    h[1] = std::max(h[1], part[npart + q]);
  }
  if (e != cudaSuccess) {
    set_last_error(cudaGetErrorString(e), __FILE__, __LINE__);
    return FG_CUDA_ERROR;
  }
  if (sumd) *sumd = h[0] / (1.0 / dt);  // the mass flux, dt removed
  if (resdiv) *resdiv = h[1] / dtinv;  // division by a constant keeps the order
  return FG_OK;
}

fg_status fg_enforce_global_mass_consv_device(fg_case *c, double *face_u, double *face_v, double *face_w,
                                              double *bcxu, double *bcyv, double *bczw,
                                              const int *vel_zero_gradient) {
  if (!c || !face_u || !face_v || !face_w) return FG_BAD_INPUT;
  const int vzg = zero_gradient_faces(vel_zero_gradient);
  if (!vzg) return FG_OK;
  if (!bcxu || !bcyv || !bczw) return FG_BAD_INPUT;
  cudaSetDevice(c->device);
  proj::Met m;
  proj::Dims d;
  fg_status st = proj_setup(c, m, d);
  if (st != FG_OK) return st;
  const size_t nref = (size_t)(c->nx + 2) * (c->ny + 2) * (c->nz + 2);
  const int8_t *ib = c->d_refmask, *gh = c->d_refmask + nref;
  const Cols q = columns(c);
  const int nb = q.blocks();
  Scratch w;
  FG_CUDA(fg::dev_alloc(&w.p, ((size_t)nb + 2 * proj::RB + 1 + 1) * sizeof(double)));
  double *blk = w.p + nb, *cv = blk + 2 * proj::RB;
  int *count = reinterpret_cast<int *>(cv + 1);
  cudaStream_t s = c->stream;
  proj::k_div<false><<<q.grid, q.block, 0, s>>>(d, m, q.kspan, vzg, ib, gh, face_u, face_v, face_w, 0.0, nullptr, w.p,
                                                nullptr, nullptr, count, (int)q.grid.z);
  enqueue_correction(c, m, d, vzg, nb, face_u, face_v, face_w, bcxu, bcyv, bczw, w.p, blk, count, cv);
  note_launches(3);
  cudaError_t e = cudaGetLastError();
  const cudaError_t es = cudaStreamSynchronize(s);
  if (e == cudaSuccess) e = es;
  if (e != cudaSuccess) {
    set_last_error(cudaGetErrorString(e), __FILE__, __LINE__);
    return FG_CUDA_ERROR;
  }
  return FG_OK;
}

fg_status fg_correct_vel_device(fg_case *c, const double *pPrime, double dt, double *u, double *v, double *w,
                                double *dpdx, double *dpdy, double *dpdz) {
  if (!c || !pPrime) return FG_BAD_INPUT;
  if ((u || v || w) && !(u && v && w)) return FG_BAD_INPUT;
  if ((dpdx || dpdy || dpdz) && !(dpdx && dpdy && dpdz)) return FG_BAD_INPUT;
  cudaSetDevice(c->device);
  proj::Met m;
  proj::Dims d;
  fg_status st = proj_setup(c, m, d);
  if (st != FG_OK) return st;
  const Cols q = columns(c);
  proj::k_correct<<<q.grid, q.block, 0, c->stream>>>(d, m, q.kspan, c->d_refmask, pPrime, dt, u, v, w, dpdx, dpdy, dpdz);
  note_launches(1);
  FG_CUDA(cudaGetLastError());
  FG_CUDA(cudaStreamSynchronize(c->stream));
  return FG_OK;
}

fg_status fg_update_pressure_device(fg_case *c, double *pPrime, double *p) {
  if (!c || !pPrime) return FG_BAD_INPUT;
  cudaSetDevice(c->device);
  proj::Met m;
  proj::Dims d;
  fg_status st = proj_setup(c, m, d);
  if (st != FG_OK) return st;
  const size_t nref = (size_t)(c->nx + 2) * (c->ny + 2) * (c->nz + 2);
  const int8_t *ib = c->d_refmask, *dead = c->d_refmask + 2 * nref;
  cudaStream_t s = c->stream;
  const dim3 grid((c->nx + 2 + proj::PU_I - 1) / proj::PU_I, (c->ny + 2 + proj::PU_J - 1) / proj::PU_J,
                  std::max(1, (c->nz + 2 + 7) / 8));
  proj::k_update<<<grid, dim3(proj::PU_I, proj::PU_J), 0, s>>>(d, ib, dead, pPrime, p == pPrime ? nullptr : p);
  note_launches(1);
  FG_CUDA(cudaGetLastError());
  FG_CUDA(cudaStreamSynchronize(s));
  return FG_OK;
}

}  // extern "C"
