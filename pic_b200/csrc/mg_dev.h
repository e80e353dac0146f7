// mg_dev.h -- geometric multigrid V-cycle of the flexible-CG preconditioner:
// the per-node operations, shared by the persistent solver kernel
// (picgpu.cu) and the one-launch-per-operation path (precond.cu), so both
// compute the same numbers.
//
// Level 0 is the solver's own grid and operator.  Level l >= 1 is the uniform
// grid of every second node of level l-1 (nx_l = (nx_{l-1} - 1)/2 + 1), with
// the Galerkin operator A_l = P^T A_{l-1} P of bilinear interpolation P,
// assembled on the host; it is a 9-point stencil, stored per node as FP32
// coefficients st[3a+c][n] coupling node (I,J) with (I+a-1, J+c-1).  A level
// node whose support holds no unknown of the finer level is inactive:
// dinv = 0 there, and every vector stays 0 on it.  The coarsest level is
// solved with the dense FP16 inverse of its operator.
//
// One V-cycle, with damped Jacobi (weight w) as smoother, one sweep down and
// one up at every level:
//   down, l = 1..L-1:  r_l = P^T t_{l-1}, z_l = w D_l^-1 r_l (one pass)
//                      t_l = r_l - A_l z_l                          (l < L-1)
//                      z_{L-1} = A_{L-1}^-1 r_{L-1}                 (coarsest)
//   up,   l = L-2..1:  y = z_l + P e_{l+1},  e_l = y + w D_l^-1 (r_l - A_l y)
//   level 0:           zA += P e_1, then the solver's own post-smoothing.
// e_l is stored in t_l (no longer needed once r_{l+1} exists); the
// coarsest level's e is its z.
#ifndef PIC_MG_DEV_H
#define PIC_MG_DEV_H

#include <stdint.h>

namespace pic {

#define PIC_MG_MAX_LEVELS 8

struct MgLevel {
  int nx, ny;          // grid nodes
  const float *st;     // [9][nx*ny]
  const float *dinv;   // [nx*ny], 0 on inactive nodes
  double *r, *z, *t;   // [nx*ny]
};

struct MgK {
  int L;  // levels including the solver's grid (0: no multigrid)
  MgLevel lv[PIC_MG_MAX_LEVELS];
};

// Loads below are never behind a test: positions outside the grid read the
// nearest node inside and carry the weight or coefficient 0 (which leaves a
// sum as it is), and interpolation has one form for all parities.  A stencil
// is then one round of loads in flight; with a branch a position it was nine
// rounds, one after the other (up- and down-sweeps of the 129^2 level 5 us
// each, of which 1.4 the barrier).

__device__ __forceinline__ int mg_clamp(int v, int n) { return v < 0 ? 0 : (v >= n ? n - 1 : v); }

// r_l[I,J] = sum over the 3x3 finer nodes around (2I, 2J) of w_x w_y t[f],
// w = 1 at the centre and 1/2 beside it (P^T of bilinear interpolation);
// fixed order, rows then columns.
template <class T>
__device__ __forceinline__ double mg_restrict(const T *__restrict__ tf, int nxf, int nyf, int I, int J) {
  const int i0 = 2 * I, j0 = 2 * J;
  double t[9];
#pragma unroll
  for (int q = 0; q < 9; ++q)
    t[q] = (double)tf[(int64_t)mg_clamp(i0 + q / 3 - 1, nxf) * nyf + mg_clamp(j0 + q % 3 - 1, nyf)];
  double s = 0.0;
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    const int a = q / 3 - 1, c = q % 3 - 1, i = i0 + a, j = j0 + c;
    const double w = (a == 0 ? 1.0 : 0.5) * (c == 0 ? 1.0 : 0.5);
    s = fma(i >= 0 && i < nxf && j >= 0 && j < nyf ? w : 0.0, t[q], s);
  }
  return s;
}

// (P e)[i,j] on the finer grid from the coarser level's e (nyc nodes a
// column): bilinear, the mean of the coarse nodes i/2 (even i, twice) or
// (i-1)/2 and (i+1)/2 (odd i), and the same in j.  Sums of equal values and
// factors of 1/4 are exact, so every parity gets the bits of its own formula.
__device__ __forceinline__ double mg_prolong(const double *__restrict__ e, int nyc, int i, int j) {
  const int I = i >> 1, J = j >> 1;
  const double *p = e + (int64_t)I * nyc + J, *p1 = p + (i & 1) * (int64_t)nyc;
  const int oy = j & 1;
  return 0.25 * ((p[0] + p1[0]) + (p[oy] + p1[oy]));
}

// A_l applied at node n = (I,J) to the values v(a, c, m) of the 9 nodes m
// around (a, c: row and column of the stencil position; coefficients toward
// nodes outside the grid, or inactive ones, are 0)
template <class Fv>
__device__ __forceinline__ double mg_apply(const MgLevel &L, int I, int J, Fv v) {
  const int64_t nl = (int64_t)L.nx * L.ny, n = (int64_t)I * L.ny + J;
  float st[9];
  double x[9];
#pragma unroll
  for (int q = 0; q < 9; ++q) st[q] = L.st[q * nl + n];
#pragma unroll
  for (int q = 0; q < 9; ++q)
    x[q] = v(q / 3, q % 3, (int64_t)mg_clamp(I + q / 3 - 1, L.nx) * L.ny + mg_clamp(J + q % 3 - 1, L.ny));
  double acc = 0.0;
#pragma unroll
  for (int q = 0; q < 9; ++q) acc = fma((double)st[q], x[q], acc);
  return acc;
}

// restriction at node n of a level that is smoothed next: r = P^T t_f and
// z = w D^-1 r (0 on inactive nodes), so the down-sweep reads z at the
// neighbours instead of forming it from their r and D^-1
__device__ __forceinline__ void mg_restrict_put(const MgLevel &L, double r, double w, bool smoothed, int64_t n) {
  L.r[n] = r;
  if (smoothed) L.z[n] = (w * r) * (double)L.dinv[n];
}

template <class T>
__device__ __forceinline__ void mg_restrict_node(const MgLevel &L, const T *__restrict__ tf, int nxf, int nyf,
                                                 double w, bool smoothed, int64_t n) {
  const int I = (int)n / L.ny, J = (int)n - I * L.ny;  // level grids hold < 2^31 nodes
  mg_restrict_put(L, mg_restrict(tf, nxf, nyf, I, J), w, smoothed, n);
}

// The down- and up-sweep values at node n.  Every load is issued whatever
// the node's kind and the result selected at the end (0 on inactive nodes),
// so no load waits on D^-1: the same numbers as testing D^-1 first.
// down-sweep: t = r - A z with z = w D^-1 r stored by the restriction
__device__ __forceinline__ double mg_smooth_val(const MgLevel &L, int64_t n) {
  const double dn = (double)L.dinv[n];
  const int I = (int)n / L.ny, J = (int)n - I * L.ny;
  const double r = L.r[n];
  const double t = r - mg_apply(L, I, J, [&](int, int, int64_t m) { return L.z[m]; });
  return dn == 0.0 ? 0.0 : t;
}

// up-sweep: y = z + P e_c, e = y + w D^-1 (r - A y).  The 3x3 nodes interpolate
// from 3x3 coarse ones at most (two rows and columns suffice at odd I, J),
// loaded once.  (y is not 0 on inactive nodes, whose coefficients are.)
__device__ __forceinline__ double mg_post_val(const MgLevel &L, const double *__restrict__ ec, int nyc, double w,
                                              int64_t n) {
  const double dn = (double)L.dinv[n], r = L.r[n];
  const int I = (int)n / L.ny, J = (int)n - I * L.ny;
  const bool eI = (I & 1) == 0, eJ = (J & 1) == 0;
  const int nxc = (L.nx - 1) / 2 + 1, Ib = eI ? I / 2 - 1 : I / 2, Jb = eJ ? J / 2 - 1 : J / 2;
  double P[3][3], pe[3][3];
#pragma unroll
  for (int q = 0; q < 9; ++q)
    P[q / 3][q % 3] = ec[(int64_t)mg_clamp(Ib + q / 3, nxc) * nyc + mg_clamp(Jb + q % 3, nyc)];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    // coarse rows of neighbour row a: even I (0,1) (1,1) (1,2); odd I (0,0) (0,1) (1,1)
    double C[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double mid = eI ? P[1][c] : P[0][c];
      C[c] = a == 0 ? P[0][c] + mid : a == 1 ? mid + P[1][c] : P[1][c] + (eI ? P[2][c] : P[1][c]);
    }
    const double mid = eJ ? C[1] : C[0];
    pe[a][0] = 0.25 * (C[0] + mid);
    pe[a][1] = 0.25 * (mid + C[1]);
    pe[a][2] = 0.25 * (C[1] + (eJ ? C[2] : C[1]));
  }
  double yn = 0.0;
  const double Ay = mg_apply(L, I, J, [&](int a, int c, int64_t m) {
    const double y = L.z[m] + pe[a][c];
    if (a == 1 && c == 1) yn = y;
    return y;
  });
  const double e = fma(w * dn, r - Ay, yn);
  return dn == 0.0 ? 0.0 : e;
}

__device__ __forceinline__ void mg_smooth_node(const MgLevel &L, int64_t n) { L.t[n] = mg_smooth_val(L, n); }

__device__ __forceinline__ void mg_post_node(const MgLevel &L, const double *__restrict__ ec, int nyc, double w,
                                             int64_t n) {
  L.t[n] = mg_post_val(L, ec, nyc, w, n);
}

// e of level l (the coarsest level's z, else its t)
__host__ __device__ __forceinline__ const double *mg_e(const MgK &M, int l) { return l == M.L - 1 ? M.lv[l].z : M.lv[l].t; }

}  // namespace pic

#endif
