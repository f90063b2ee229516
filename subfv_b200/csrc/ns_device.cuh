// Device functions of the explicit Euler residual shared by its kernels (ns.cu and
// ns_node_tile.cu): state conversions, boundary states, reconstruction, the subface
// fluxes and the nodal 3x3 solves.
//
// Reference: src/ns/ns_euler_rs_module.F90, src/ns/ns_euler_recon_module.F90,
// src/ns/ns_euler_primitives_module.F90 (lines at each function).
#pragma once
#include "ns.cuh"

namespace subfv {
namespace {

constexpr double G = 1.4;  // ns_global_data_module.F90:9

__device__ inline double fmax2(double a, double b) { return b > a ? b : a; }
__device__ inline double fmin2(double a, double b) { return b < a ? b : a; }
template <class T>
__device__ inline T tmax2(T a, T b) { return b > a ? b : a; }
template <class T>
__device__ inline T tmin2(T a, T b) { return b < a ? b : a; }

template <class T>
__device__ inline void p2c(const T* w, T* u) {
  u[0] = w[0];
  for (int k = 1; k < 4; ++k) u[k] = w[k] * w[0];
  u[4] = w[4] / (T)(G - 1) + (T)0.5 * w[0] * (w[1] * w[1] + w[2] * w[2] + w[3] * w[3]);
}
template <class T>
__device__ inline void c2p(const T* u, T* w) {
  w[0] = u[0];
  for (int k = 1; k < 4; ++k) w[k] = qdiv(u[k], u[0]);
  w[4] = (T)(G - 1) * (u[4] - (T)0.5 * w[0] * (w[1] * w[1] + w[2] * w[2] + w[3] * w[3]));
}
template <class T>
__device__ inline T dotT(const T* a, const T* b) {
  T s = 0;
  s = s + a[0] * b[0];
  s = s + a[1] * b[1];
  s = s + a[2] * b[2];
  return s;
}
__device__ inline double sound_speed_w(const double* w) { return sqrt(G * w[4] / w[0]); }

__device__ inline void ld5(const double* U, int c, double* u) {
  const double* r = U + kRec * (size_t)c;
  for (int k = 0; k < 5; ++k) u[k] = r[k];
}

// ns_euler_primitives_module.F90:92-111
__device__ double max_omega_for_positivity(const double* U, const double* dU) {
  double omega = 1.0, US[5], WS[5];
  for (int k = 0; k < 5; ++k) US[k] = U[k] + omega * dU[k];
  c2p(US, WS);
  bool pos = WS[0] > 1e-17 && WS[4] > 1e-17;
  while (!pos && omega > 1e-6) {  // at most ~131 halvings by 0.9 before omega <= 1e-6
    omega = omega * 0.9;
    for (int k = 0; k < 5; ++k) US[k] = U[k] + omega * dU[k];
    c2p(US, WS);
    pos = WS[0] > 1e-17 && WS[4] > 1e-17;
  }
  return omega;
}

// When every singular value passes the cut, the pseudo-inverse is the inverse. The cut
// (3e-12 * sigma_max) is certainly passed when |det A| > 3e-12 ||A||_F^3, because
// sigma_min >= |det A| / sigma_max^2 and sigma_max <= ||A||_F. Then A^-1 = adj(A) / det,
// refined by one Newton step X <- X + X (I - A X); otherwise the Jacobi SVD below runs.
__device__ bool inv3_if_regular(double A[3][3]) {
  double f2 = 0.0;
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) f2 = f2 + A[i][j] * A[i][j];
  double C[3][3];  // cofactors
  C[0][0] = A[1][1] * A[2][2] - A[1][2] * A[2][1];
  C[0][1] = A[1][2] * A[2][0] - A[1][0] * A[2][2];
  C[0][2] = A[1][0] * A[2][1] - A[1][1] * A[2][0];
  C[1][0] = A[0][2] * A[2][1] - A[0][1] * A[2][2];
  C[1][1] = A[0][0] * A[2][2] - A[0][2] * A[2][0];
  C[1][2] = A[0][1] * A[2][0] - A[0][0] * A[2][1];
  C[2][0] = A[0][1] * A[1][2] - A[0][2] * A[1][1];
  C[2][1] = A[0][2] * A[1][0] - A[0][0] * A[1][2];
  C[2][2] = A[0][0] * A[1][1] - A[0][1] * A[1][0];
  const double det = A[0][0] * C[0][0] + A[0][1] * C[0][1] + A[0][2] * C[0][2];
  if (!(det * det > 9e-24 * (f2 * f2 * f2))) return false;
  const double r = 1.0 / det;
  double X[3][3], R[3][3];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) X[i][j] = C[j][i] * r;
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      double s = i == j ? 1.0 : 0.0;
      for (int k = 0; k < 3; ++k) s = s - A[i][k] * X[k][j];
      R[i][j] = s;
    }
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      double s = 0.0;
      for (int k = 0; k < 3; ++k) s = s + X[i][k] * R[k][j];
      A[i][j] = X[i][j] + s;
    }
  return true;
}

// Pseudo-inverse of a 3x3 matrix (A[r][c] = mat(r+1, c+1)); singular values below
// 3e-12 * max discarded (the cut of pseudo_inverse_inplace_lapack,
// linear_solver_module.F90:683-715): the inverse when the cut cannot bite, else a
// one-sided Jacobi SVD of six sweeps.
__device__ __noinline__ void pinv3_jacobi(double A[3][3]);
// the Jacobi case works on a copy: an array whose address reaches an out-of-line call
// lives in local memory on every path, so the caller's matrix keeps no escaping address
__device__ inline void pinv3(double A[3][3]) {
  if (!inv3_if_regular(A)) {
    double B[3][3];
    for (int d = 0; d < 3; ++d)
      for (int e = 0; e < 3; ++e) B[d][e] = A[d][e];
    pinv3_jacobi(B);
    for (int d = 0; d < 3; ++d)
      for (int e = 0; e < 3; ++e) A[d][e] = B[d][e];
  }
}
// the rank-deficient case, out of line (rare; keeps the callers' registers low)
__device__ __noinline__ void pinv3_jacobi(double A[3][3]) {
  double U[3][3], V[3][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}};
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) U[i][j] = A[i][j];
  const int pr[3][2] = {{0, 1}, {0, 2}, {1, 2}};
  for (int sweep = 0; sweep < 6; ++sweep)
    for (int r = 0; r < 3; ++r) {
      const int p = pr[r][0], q = pr[r][1];
      double al = 0.0, be = 0.0, ga = 0.0;
      for (int i = 0; i < 3; ++i) {
        al = al + U[i][p] * U[i][p];
        be = be + U[i][q] * U[i][q];
        ga = ga + U[i][p] * U[i][q];
      }
      if (!(fabs(ga) > 1e-15 * sqrt(al * be))) continue;
      double zeta = (be - al) / (2.0 * ga);
      double t = 1.0 / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
      if (zeta < 0.0) t = -t;
      double c = 1.0 / sqrt(1.0 + t * t), s = c * t;
      for (int i = 0; i < 3; ++i) {
        double up = U[i][p], uq = U[i][q];
        U[i][p] = c * up - s * uq;
        U[i][q] = s * up + c * uq;
        double vp = V[i][p], vq = V[i][q];
        V[i][p] = c * vp - s * vq;
        V[i][q] = s * vp + c * vq;
      }
    }
  double sig[3], smax = 0.0;
  for (int k = 0; k < 3; ++k) {
    double s = 0.0;
    for (int i = 0; i < 3; ++i) s = s + U[i][k] * U[i][k];
    sig[k] = sqrt(s);
    smax = fmax2(smax, sig[k]);
  }
  const double tol = 3 * 1e-12 * smax;
  double SUt[3][3];
  for (int k = 0; k < 3; ++k)
    for (int j = 0; j < 3; ++j) SUt[k][j] = sig[k] > tol ? (1.0 / sig[k]) * (U[j][k] / sig[k]) : 0.0;
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      double s = 0.0;
      for (int k = 0; k < 3; ++k) s = s + V[i][k] * SUt[k][j];
      A[i][j] = s;
    }
}

// LU with partial pivoting and the triangular solves, in the operation order of
// LAPACK dgetrf2/dgetrs with reference BLAS (lu_solve_inplace_lapack, :643-657). The row
// exchanges are selects between fixed rows, so that the matrix stays in registers (a row
// index would put it in local memory); the right-hand side follows them at once, as its
// elimination starts after the last. A column's reciprocal serves the multipliers and,
// through div_by, the back substitution.
__device__ inline void swap_if(bool s, double& a, double& b) {
  const double t = a;
  a = s ? b : a;
  b = s ? t : b;
}
__device__ inline void lu_solve3(double A[3][3], double* x, const double* b) {
  const double sfmin = 2.2250738585072014e-308;
  double y[3] = {b[0], b[1], b[2]}, rec[2] = {0.0, 0.0};
  bool has_rec[2] = {false, false};
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    int p = j;
    double amax = fabs(A[j][j]), ap = A[j][j];
#pragma unroll
    for (int i = j + 1; i < 3; ++i)
      if (fabs(A[i][j]) > amax) {
        amax = fabs(A[i][j]);
        ap = A[i][j];
        p = i;
      }
    const bool nz = ap != 0.0;
#pragma unroll
    for (int i = j + 1; i < 3; ++i) {
      swap_if(p == i, y[j], y[i]);
#pragma unroll
      for (int k = 0; k < 3; ++k) swap_if(nz && p == i, A[j][k], A[i][k]);
    }
    if (j < 2 && nz) {
      if (fabs(A[j][j]) >= sfmin) {
        const double r = 1.0 / A[j][j];
        rec[j] = r;
        has_rec[j] = true;
#pragma unroll
        for (int i = j + 1; i < 3; ++i) A[i][j] = r * A[i][j];
      } else {
#pragma unroll
        for (int i = j + 1; i < 3; ++i) A[i][j] = A[i][j] / A[j][j];
      }
    }
#pragma unroll
    for (int i = j + 1; i < 3; ++i)
#pragma unroll
      for (int k = j + 1; k < 3; ++k) A[i][k] = A[i][k] - A[j][k] * A[i][j];
  }
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (y[k] != 0.0)
#pragma unroll
      for (int i = k + 1; i < 3; ++i) y[i] = y[i] - y[k] * A[i][k];
#pragma unroll
  for (int k = 2; k >= 0; --k)
    if (y[k] != 0.0) {
      y[k] = k < 2 && has_rec[k] ? div_by(y[k], A[k][k], rec[k]) : y[k] / A[k][k];
#pragma unroll
      for (int i = 0; i < k; ++i) y[i] = y[i] - y[k] * A[i][k];
    }
  for (int k = 0; k < 3; ++k) x[k] = y[k];
}

// Boundary semantics on the device: flr.y >= 0 is the right cell; otherwise the face's
// reference right_neigh is flr.y + 1 (0 = default wall, -tag = boundary condition tag).
__device__ inline bool is_wall(const NsParams& P, int y) {
  if (y >= 0) return false;
  if (y == -1) return true;
  return P.bc_type[-(y + 1) - 1] == 1;
}

// OI (ns_euler_recon_module.F90:322-329): gfortran's scaled NORM2 of a 3-vector, in T
template <class T>
__device__ inline T oi3(T a0, T a1, T a2) {
  const T a[3] = {a0, a1, a2};
  T scale = 1, res = 0;
  for (int i = 0; i < 3; ++i)
    if (a[i] != (T)0) {
      T ax = fabs(a[i]);
      if (ax > scale) {
        T q = scale / ax;
        res = (T)1 + res * q * q;
        scale = ax;
      } else {
        T q = ax / scale;
        res += q * q;
      }
    }
  return scale * qsqrt(res);
}

// sol_potential_flow_2d / _3d (ns_euler_exact_sol_module.F90:105-170) at x, primitive.
// The 2-D routine's Mach number is a default-kind (single precision) literal, so its
// value is the float nearest 1e-4; the 3-D one is 1e-4 in double.
template <class T>
__device__ __noinline__ void potential_flow(const double4 x4, bool three_d, T* w) {
  const T x[3] = {(T)x4.x, (T)x4.y, (T)x4.z};
  const T r0 = (T)0.5, r1 = (T)5.5, rhoinf = (T)1.4, pinf = (T)1.0;
  const T mach = three_d ? (T)1e-4 : (T)1e-4f;
  const T vinf = mach * sqrt((T)G * pinf / rhoinf);
  T ux, uy, uz;
  if (!three_d) {
    const T r = sqrt(x[0] * x[0] + x[1] * x[1]);
    const T th = atan2(x[1], x[0]);
    const T c = r1 * r1 / (r1 * r1 - r0 * r0), q = (r0 / r) * (r0 / r);
    const T vr = c * ((T)1 - q) * cos(th);
    const T vt = -c * ((T)1 + q) * sin(th);
    ux = vinf * (cos(th) * vr - sin(th) * vt);
    uy = vinf * (sin(th) * vr + cos(th) * vt);
    uz = (T)0;
  } else {
    const T r = sqrt(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]);
    const T f = r0 * r0 * r0 / ((T)2 * (r * r * r * r * r));
    ux = vinf * ((T)1 + f * (r * r - (T)3 * (x[0] * x[0])));
    uy = (T)-3 * vinf * f * x[0] * x[1];
    uz = (T)-3 * vinf * f * x[0] * x[2];
  }
  const T vmag2 = ux * ux + uy * uy + uz * uz;
  w[0] = rhoinf;
  w[1] = ux;
  w[2] = uy;
  w[3] = uz;
  w[4] = pinf + (T)0.5 * rhoinf * (vinf * vinf - vmag2);
}

// compute_right_state (:331-409): the ghost state by boundary kind (1 wall, 2 adherence
// wall, 3 freestream, 4 supersonic outflow, 5 pondered inflow, 6 double-Mach inflow /
// outflow, 7 double-Mach bottom, 8 and 9 the potential flows in 2-D and 3-D); sol_l /
// sol_r conservative, n the subface normal. The kinds that read the face centroid fx or
// the time t (of the step being evaluated) are out of line. Their arguments are values
// only: a reference to the kernel's mesh or parameter block would make every thread of
// the calling kernel copy that block into local memory.
struct BcVals {
  double v[5];
};
template <class T>
__device__ __noinline__ void right_state_ext(int kind, const BcVals bv, const double4 fx, const double t, const T* n,
                                             const T* sol_l, T* sol_r) {
  if (kind == 2) {
    for (int k = 0; k < 5; ++k) sol_r[k] = sol_l[k];
    for (int k = 1; k < 4; ++k) sol_r[k] = (T)2.0 * sol_l[0] * (T)bv.v[k] - sol_l[k];
    const T nl = oi3<T>(qdiv(sol_l[1], sol_l[0]), qdiv(sol_l[2], sol_l[0]), qdiv(sol_l[3], sol_l[0]));
    const T nr = oi3<T>(qdiv(sol_r[1], sol_r[0]), qdiv(sol_r[2], sol_r[0]), qdiv(sol_r[3], sol_r[0]));
    sol_r[4] = sol_l[4] - (T)0.5 * sol_l[0] * (nl * nl) + (T)0.5 * sol_l[0] * (nr * nr);
    return;
  }
  if (kind == 5) {
    T w[5];
    for (int k = 0; k < 5; ++k) w[k] = (T)bv.v[k];
    p2c(w, sol_r);
    if (dotT(sol_r + 1, n) > (T)0)
      for (int k = 0; k < 5; ++k) sol_r[k] = sol_l[k];
    return;
  }
  if (kind == 8 || kind == 9) {
    T w[5];
    potential_flow<T>(fx, kind == 9, w);
    p2c(w, sol_r);
    return;
  }
  const T post[5] = {(T)8.0, (T)7.145, (T)-4.125, (T)0.0, (T)116.5}, pre[5] = {(T)1.4, 0, 0, 0, (T)1.0};
  if (kind == 6) {
    p2c((T)fx.y > (T)1.732 * ((T)fx.x - (T)0.1667 - (T)10.0 * (T)t) ? post : pre, sol_r);
  } else if ((T)fx.x < (T)0.1667) {  // kind 7
    p2c(post, sol_r);
  } else {
    for (int k = 0; k < 5; ++k) sol_r[k] = sol_l[k];
    T d = dotT(sol_r + 1, n);
    for (int k = 1; k < 4; ++k) sol_r[k] = sol_r[k] - (T)2.0 * d * n[k - 1];
  }
}

template <class T>
__device__ void right_state(const DevMesh& m, const NsParams& P, int y, int sf, const T* n, const T* sol_l, T* sol_r,
                            const NsScalars* sc) {
  int kind = y == -1 ? 1 : P.bc_type[-(y + 1) - 1];
  if (kind == 1) {
    for (int k = 0; k < 5; ++k) sol_r[k] = sol_l[k];
    T d = dotT(sol_r + 1, n);
    for (int k = 1; k < 4; ++k) sol_r[k] = sol_r[k] - (T)2.0 * d * n[k - 1];
  } else if (kind == 3) {
    T w[5];
    for (int k = 0; k < 5; ++k) w[k] = (T)P.bc_val[-(y + 1) - 1][k];
    p2c(w, sol_r);
  } else if (kind == 4) {
    for (int k = 0; k < 5; ++k) sol_r[k] = sol_l[k];
  } else {
    BcVals bv;
    for (int k = 0; k < 5; ++k) bv.v[k] = P.bc_val[-(y + 1) - 1][k];
    const double4 fx = kind >= 6 ? m.fc[m.sf_face[sf]] : make_double4(0.0, 0.0, 0.0, 0.0);
    const double t = (kind == 6 && sc) ? sc->t : 0.0;
    // on copies: an array whose address reaches the out-of-line routine lives in local
    // memory on every path
    T nc[3], l[5], r[5];
    for (int d = 0; d < 3; ++d) nc[d] = n[d];
    for (int k = 0; k < 5; ++k) l[k] = sol_l[k];
    right_state_ext<T>(kind, bv, fx, t, nc, l, r);
    for (int k = 0; k < 5; ++k) sol_r[k] = r[k];
  }
}

// reconstruct_lr_w (:427-451); grad records [15] with g[5*d + var] = grad(d+1, var+1)
template <class T>
__device__ void reconstruct(const DevMesh& m, const NsParams& P, const double* U, const double* grad, int v, int sf,
                            int le, int y, bool so, double* wl_out, double* wr_out, const NsScalars* sc) {
  T ul[5], wl[5], wr[5];
  double u64[5];
  ld5(U, le, u64);
  for (int k = 0; k < 5; ++k) ul[k] = (T)u64[k];
  c2p(ul, wl);
  const double4 xv = m.x[v];
  if (so) {
    const double4 cc = m.cc[le];
    const T dx[3] = {(T)(xv.x - cc.x), (T)(xv.y - cc.y), (T)(xv.z - cc.z)};
    const double* g = grad + 15 * (size_t)le;
    for (int k = 0; k < 5; ++k) {
      T s = 0;
      for (int d = 0; d < 3; ++d) s = s + (T)g[5 * d + k] * dx[d];
      wl[k] = wl[k] + s;
    }
  }
  if (y >= 0) {
    T ur[5];
    ld5(U, y, u64);
    for (int k = 0; k < 5; ++k) ur[k] = (T)u64[k];
    c2p(ur, wr);
    if (so) {
      const double4 cc = m.cc[y];
      const T dx[3] = {(T)(xv.x - cc.x), (T)(xv.y - cc.y), (T)(xv.z - cc.z)};
      const double* g = grad + 15 * (size_t)y;
      for (int k = 0; k < 5; ++k) {
        T s = 0;
        for (int d = 0; d < 3; ++d) s = s + (T)g[5 * d + k] * dx[d];
        wr[k] = wr[k] + s;
      }
    }
  } else {
    const double4 sn = m.sfn[sf];
    const T n[3] = {(T)sn.x, (T)sn.y, (T)sn.z};
    T uc[5], gh[5];
    p2c(wl, uc);
    right_state(m, P, y, sf, n, uc, gh, sc);
    c2p(gh, wr);
  }
  for (int k = 0; k < 5; ++k) {
    wl_out[k] = (double)wl[k];
    wr_out[k] = (double)wr[k];
  }
}

// two_wave (ns_euler_rs_module.F90:154-198)
template <class T>
__device__ void two_wave(const double* wl64, const double* wr64, const double* n64, double lr[2][5], double* sl_o,
                         double* sr_o) {
  T wl[5], wr[5], n[3];
  for (int k = 0; k < 5; ++k) {
    wl[k] = (T)wl64[k];
    wr[k] = (T)wr64[k];
  }
  for (int d = 0; d < 3; ++d) n[d] = (T)n64[d];
  T rhol = wl[0], vnl = dotT(wl + 1, n), pl = wl[4], al = sqrt((T)G * wl[4] / wl[0]), ul[5];
  p2c(wl, ul);
  T rhor = wr[0], vnr = dotT(wr + 1, n), pr = wr[4], ar = sqrt((T)G * wr[4] / wr[0]), ur[5];
  p2c(wr, ur);
  T fl[5], fr[5];
  fl[0] = vnl * ul[0];
  for (int k = 1; k < 4; ++k) fl[k] = vnl * ul[k] + pl * n[k - 1];
  fl[4] = (ul[4] + pl) * vnl;
  fr[0] = vnr * ur[0];
  for (int k = 1; k < 4; ++k) fr[k] = vnr * ur[k] + pr * n[k - 1];
  fr[4] = (ur[4] + pr) * vnr;
  T lam_l = tmax2(tmax2(al * rhol, qsqrt(rhol * tmax2((T)0, pr - pl))), -rhol * (vnr - vnl));
  T lam_r = tmax2(tmax2(ar * rhor, qsqrt(rhor * tmax2((T)0, pl - pr))), -rhor * (vnr - vnl));
  T sl = vnl - lam_l / rhol;
  T sr = vnr + lam_r / rhor;
  for (int k = 0; k < 5; ++k) {
    T et = qdiv(sr * ur[k] - sl * ul[k] - (fr[k] - fl[k]), sr - sl);
    T f = (T)0.5 * (fl[k] + fr[k]) - (T)0.5 * (fabs(sl) * (et - ul[k]) + fabs(sr) * (ur[k] - et));
    lr[0][k] = (double)f;
    lr[1][k] = (double)(-f);
  }
  *sl_o = (double)sl;
  *sr_o = (double)sr;
}

// three_wave (ns_euler_rs_module.F90:9-75) and modified_three_wave (:77-152): two-wave
// bounds, v* = v_bar, HLLC-type star states (the modified form averages the tangential
// velocity and carries its jump energy); arithmetic in T, results stored as double. The
// fluxes of the schemes beyond multi_point and two_wave are out of line, so the node
// kernel's register allocation for those two does not grow with them.
template <class T>
__device__ __noinline__ void three_wave(const double* wl64, const double* wr64, const double* n64, double lr[2][5],
                           double* sl_o, double* sr_o, bool modified) {
  T wl[5], wr[5], n[3];
  for (int k = 0; k < 5; ++k) {
    wl[k] = (T)wl64[k];
    wr[k] = (T)wr64[k];
  }
  for (int d = 0; d < 3; ++d) n[d] = (T)n64[d];
  const T c0 = (T)0, c1 = (T)1, ch = (T)0.5;
  T rhol = wl[0], vnl = dotT(wl + 1, n), pl = wl[4], ul[5];
  p2c(wl, ul);
  T el = ul[4] / rhol, al = sqrt((T)G * wl[4] / wl[0]);
  T rhor = wr[0], vnr = dotT(wr + 1, n), pr = wr[4], ur[5];
  p2c(wr, ur);
  T er = ur[4] / rhor, ar = sqrt((T)G * wr[4] / wr[0]);
  T fl[5], fr[5];
  fl[0] = vnl * ul[0];
  for (int k = 1; k < 4; ++k) fl[k] = vnl * ul[k] + pl * n[k - 1];
  fl[4] = (ul[4] + pl) * vnl;
  fr[0] = vnr * ur[0];
  for (int k = 1; k < 4; ++k) fr[k] = vnr * ur[k] + pr * n[k - 1];
  fr[4] = (ur[4] + pr) * vnr;
  T lam_l = tmax2(tmax2(al * rhol, qsqrt(rhol * tmax2(c0, pr - pl))), -rhol * (vnr - vnl));
  T lam_r = tmax2(tmax2(ar * rhor, qsqrt(rhor * tmax2(c0, pl - pr))), -rhor * (vnr - vnl));
  T v_et = qdiv(lam_l * vnl + lam_r * vnr - (pr - pl), lam_r + lam_l);
  T vt_et[3] = {c0, c0, c0}, tang_energy = c0;
  if (modified) {
    T vt_l[3], vt_r[3], dvt[3];
    for (int d = 0; d < 3; ++d) {
      vt_l[d] = wl[1 + d] - vnl * n[d];
      vt_r[d] = wr[1 + d] - vnr * n[d];
    }
    for (int d = 0; d < 3; ++d) vt_et[d] = qdiv(lam_l * vt_l[d] + lam_r * vt_r[d], lam_l + lam_r);
    for (int d = 0; d < 3; ++d) dvt[d] = vt_r[d] - vt_l[d];
    const T tang_coeff = -(lam_l * lam_r / (lam_l + lam_r));
    tang_energy = tang_coeff * dotT(dvt, vt_et);
  }
  T rhol_et = c1 / (c1 / rhol + qdiv(v_et - vnl, lam_l));
  T pl_bar = pl - lam_l * (v_et - vnl);
  T rhor_et = c1 / (c1 / rhor + qdiv(vnr - v_et, lam_r));
  T pr_bar = pr + lam_r * (v_et - vnr);
  T sle[5], sre[5];
  sle[0] = rhol_et;
  sre[0] = rhor_et;
  if (modified) {
    for (int k = 1; k < 4; ++k) sle[k] = rhol_et * (v_et * n[k - 1] + vt_et[k - 1]);
    sle[4] = rhol_et * (el + qdiv(pl * vnl - pl_bar * v_et - tang_energy, lam_l));
    for (int k = 1; k < 4; ++k) sre[k] = rhor_et * (v_et * n[k - 1] + vt_et[k - 1]);
    sre[4] = rhor_et * (er + qdiv(pr_bar * v_et - pr * vnr + tang_energy, lam_r));
  } else {
    for (int k = 1; k < 4; ++k) sle[k] = rhol_et * (wl[k] + (v_et - vnl) * n[k - 1]);
    sle[4] = rhol_et * (el + qdiv(pl * vnl - pl_bar * v_et, lam_l));
    for (int k = 1; k < 4; ++k) sre[k] = rhor_et * (wr[k] + (v_et - vnr) * n[k - 1]);
    sre[4] = rhor_et * (er + qdiv(pr_bar * v_et - pr * vnr, lam_r));
  }
  const T sl = vnl - lam_l / rhol, sr = vnr + lam_r / rhor;
  for (int k = 0; k < 5; ++k) {
    const T f = ch * (fl[k] + fr[k]) -
                ch * (fabs(sl) * (sle[k] - ul[k]) + fabs(v_et) * (sre[k] - sle[k]) + fabs(sr) * (ur[k] - sre[k]));
    lr[0][k] = (double)f;
    lr[1][k] = (double)(-f);
  }
  *sl_o = (double)sl;
  *sr_o = (double)sr;
}

// multi_point_pressure (ns_euler_rs_module.F90:555-616) and multi_point_pressure_ph
// (:618-679): star states from the nodal pressure and the nodal pressure solver's bounds.
template <class T>
__device__ __noinline__ void multi_point_pressure(const double* wl64, const double* wr64, const double* n64, double lr[2][5],
                                     double p_nodal64, double lam_l64, double lam_r64, double* sl_o, double* sr_o,
                                     bool ph) {
  T wl[5], wr[5], n[3];
  for (int k = 0; k < 5; ++k) {
    wl[k] = (T)wl64[k];
    wr[k] = (T)wr64[k];
  }
  for (int d = 0; d < 3; ++d) n[d] = (T)n64[d];
  const T lam_l = (T)lam_l64, lam_r = (T)lam_r64, p_nodal = (T)p_nodal64, c1 = (T)1, ch = (T)0.5;
  T rhol = wl[0], vnl = dotT(wl + 1, n), pl = wl[4], ul[5], vt_l[3];
  for (int d = 0; d < 3; ++d) vt_l[d] = wl[1 + d] - vnl * n[d];
  p2c(wl, ul);
  T el = ul[4] / rhol;
  T rhor = wr[0], vnr = dotT(wr + 1, n), pr = wr[4], ur[5], vt_r[3];
  for (int d = 0; d < 3; ++d) vt_r[d] = wr[1 + d] - vnr * n[d];
  p2c(wr, ur);
  T er = ur[4] / rhor;
  T fl[5], fr[5];
  fl[0] = vnl * ul[0];
  for (int k = 1; k < 4; ++k) fl[k] = vnl * ul[k] + pl * n[k - 1];
  fl[4] = (ul[4] + pl) * vnl;
  fr[0] = vnr * ur[0];
  for (int k = 1; k < 4; ++k) fr[k] = vnr * ur[k] + pr * n[k - 1];
  fr[4] = (ur[4] + pr) * vnr;
  T vn_bar = qdiv(lam_l * vnl + lam_r * vnr - (pr - pl), lam_r + lam_l);
  T vn_l_et = vnl - qdiv(p_nodal - pl, lam_l);
  T rhol_et = c1 / (c1 / rhol + qdiv(vn_bar - vnl, lam_l));
  T sle[5], sre[5];
  sle[0] = rhol_et;
  for (int k = 1; k < 4; ++k) sle[k] = rhol_et * (vt_l[k - 1] + vn_l_et * n[k - 1]);
  sle[4] = rhol_et * (el + qdiv(pl * vnl - p_nodal * (ph ? vn_l_et : vn_bar), lam_l));
  T vn_r_et = vnr + qdiv(p_nodal - pr, lam_r);
  T rhor_et = c1 / (c1 / rhor + qdiv(vnr - vn_bar, lam_r));
  sre[0] = rhor_et;
  for (int k = 1; k < 4; ++k) sre[k] = rhor_et * (vt_r[k - 1] + vn_r_et * n[k - 1]);
  sre[4] = rhor_et * (er + qdiv(p_nodal * (ph ? vn_r_et : vn_bar) - pr * vnr, lam_r));
  const T sl = vnl - lam_l / rhol, sr = vnr + lam_r / rhor;
  for (int k = 0; k < 5; ++k) {
    const T f = ch * (fl[k] + fr[k]) -
                ch * (fabs(sl) * (sle[k] - ul[k]) + fabs(vn_bar) * (sre[k] - sle[k]) + fabs(sr) * (ur[k] - sre[k]));
    lr[0][k] = (double)f;
    lr[1][k] = (double)(-f);
  }
  *sl_o = (double)sl;
  *sr_o = (double)sr;
}

// One subface's share of iteration `iter` of compute_lambdas_and_solve_nodal_pressure
// (ns_euler_rs_module.F90:681-758), FP64: the bounds lam_l, lam_r (updated in place),
// and the terms t1, t2 of s1 and s2 (p_node = s1 / s2). The previous iteration's p_bar
// (read at bc_style 1 walls) is recomputed from the bounds it ended with.
__device__ inline void nodal_pressure_terms(int iter, bool wall1, const double* wl, const double* wr,
                                            const double* n, double area, double p_node, double& lam_l,
                                            double& lam_r, double& t1, double& t2) {
  const double rhol = wl[0], vnl = dotT(wl + 1, n), pl = wl[4], al = sqrt(G * wl[4] / wl[0]);
  const double rhor = wr[0], vnr = dotT(wr + 1, n), pr = wr[4], ar = sqrt(G * wr[4] / wr[0]);
  auto pbar_of = [&](double ll, double lr) { return (lr * pl + ll * pr - lr * ll * (vnr - vnl)) / (lr + ll); };
  if (iter == 1) {
    lam_l = fmax2(fmax2(fmax2(lam_l, al * rhol), qsqrt(rhol * fmax2(0.0, pr - pl))), -rhol * (vnr - vnl));
    lam_r = fmax2(fmax2(fmax2(lam_r, ar * rhor), qsqrt(rhor * fmax2(0.0, pl - pr))), -rhor * (vnr - vnl));
    const double pb = pbar_of(lam_l, lam_r);
    lam_l = fmax2(lam_l, al * rhol + 1.5 * qsqrt(fmax2(0.0, (pb - pl) * rhol)));
    lam_r = fmax2(lam_r, ar * rhor + 1.5 * qsqrt(fmax2(0.0, (pb - pr) * rhor)));
  } else {
    const double pq = wall1 ? pbar_of(lam_l, lam_r) : p_node;
    lam_l = fmax2(lam_l, al * rhol + 1.5 * qsqrt(fmax2(0.0, (pq - pl) * rhol)));
    lam_r = fmax2(lam_r, ar * rhor + 1.5 * qsqrt(fmax2(0.0, (pq - pr) * rhor)));
  }
  const double pb = pbar_of(lam_l, lam_r);
  if (wall1) {
    t1 = (1.0 / lam_r + 1.0 / lam_l) * area * (lam_r * pl + lam_r * lam_l * vnl) / (lam_r + lam_l);
    t2 = (1.0 / lam_l) * area;
  } else {
    t1 = (1.0 / lam_r + 1.0 / lam_l) * area * pb;
    t2 = (1.0 / lam_r + 1.0 / lam_l) * area;
  }
}

// multi_point_iso's flux (ns_euler_module.F90:464-483): the multi-point (or, at an
// excluded boundary vertex, two-wave) flux blended with three_wave by
// warea = min area / area; the wave speeds sl, sr are three_wave's.
template <class T>
__device__ __noinline__ void blend_three_wave(const double* w10, const double* n, double amin, double lr[2][5], double* sl,
                                 double* sr) {
  double lr3[2][5];
  three_wave<T>(w10, w10 + 5, n, lr3, sl, sr, false);
  const double wa = amin / n[3];
  for (int q = 0; q < 2; ++q)
    for (int k = 0; k < 5; ++k) lr[q][k] = wa * lr[q][k] + (1.0 - wa) * lr3[q][k];
}

// The out-of-line fluxes called on private copies of the node kernels' arrays (the
// subface's states, its normal and area, the flux pair and wave speeds), so that those
// arrays keep no escaping address and stay in registers on the multi_point and two_wave
// paths; the called routines see the same values.
struct FluxCopy {
  double w[10], n[4], lr[2][5], sl, sr;
  __device__ void load(const double* w10, const double* n4) {
    for (int k = 0; k < 10; ++k) w[k] = w10[k];
    for (int d = 0; d < 4; ++d) n[d] = n4[d];
  }
  __device__ void store(double o[2][5], double* sl_o, double* sr_o) const {
    for (int q = 0; q < 2; ++q)
      for (int k = 0; k < 5; ++k) o[q][k] = lr[q][k];
    *sl_o = sl;
    *sr_o = sr;
  }
};
template <class T>
__device__ inline void three_wave_c(const double* w10, const double* n4, double lr[2][5], double* sl, double* sr,
                                    bool modified) {
  FluxCopy c;
  c.load(w10, n4);
  three_wave<T>(c.w, c.w + 5, c.n, c.lr, &c.sl, &c.sr, modified);
  c.store(lr, sl, sr);
}
template <class T>
__device__ inline void multi_point_pressure_c(const double* w10, const double* n4, double lr[2][5], double p_nodal,
                                              double lam_l, double lam_r, double* sl, double* sr, bool ph) {
  FluxCopy c;
  c.load(w10, n4);
  multi_point_pressure<T>(c.w, c.w + 5, c.n, c.lr, p_nodal, lam_l, lam_r, &c.sl, &c.sr, ph);
  c.store(lr, sl, sr);
}
template <class T>
__device__ inline void blend_three_wave_c(const double* w10, const double* n4, double amin, double lr[2][5],
                                          double* sl, double* sr) {
  FluxCopy c;
  c.load(w10, n4);
  for (int q = 0; q < 2; ++q)
    for (int k = 0; k < 5; ++k) c.lr[q][k] = lr[q][k];
  c.sl = *sl;
  c.sr = *sr;
  blend_three_wave<T>(c.w, c.n, amin, c.lr, &c.sl, &c.sr);
  c.store(lr, sl, sr);
}

// multi_point (ns_euler_rs_module.F90:200-286); false on a negative star density
template <class T>
__device__ bool multi_point(const double* wl64, const double* wr64, const double* n64, double lr[2][5],
                            double vn_nodal, double lam_l64, double lam_r64, double* sl_o, double* sr_o) {
  T wl[5], wr[5], n[3];
  for (int k = 0; k < 5; ++k) {
    wl[k] = (T)wl64[k];
    wr[k] = (T)wr64[k];
  }
  for (int d = 0; d < 3; ++d) n[d] = (T)n64[d];
  const T lam_l = (T)lam_l64, lam_r = (T)lam_r64;
  T rhol = wl[0], vnl = dotT(wl + 1, n), pl = wl[4], ul[5];
  p2c(wl, ul);
  T el = ul[4] / rhol;
  T rhor = wr[0], vnr = dotT(wr + 1, n), pr = wr[4], ur[5];
  p2c(wr, ur);
  T er = ur[4] / rhor;
  T fl[5], fr[5];
  fl[0] = vnl * ul[0];
  for (int k = 1; k < 4; ++k) fl[k] = vnl * ul[k] + pl * n[k - 1];
  fl[4] = (ul[4] + pl) * vnl;
  fr[0] = vnr * ur[0];
  for (int k = 1; k < 4; ++k) fr[k] = vnr * ur[k] + pr * n[k - 1];
  fr[4] = (ur[4] + pr) * vnr;
  T v_et = (T)vn_nodal;
  T rhol_et = (T)1.0 / ((T)1.0 / rhol + qdiv(v_et - vnl, lam_l));
  T pl_bar = pl - lam_l * (v_et - vnl);
  T sle[5], sre[5];
  sle[0] = rhol_et;
  for (int k = 1; k < 4; ++k) sle[k] = rhol_et * (wl[k] + (v_et - vnl) * n[k - 1]);
  sle[4] = rhol_et * (el + qdiv(pl * vnl - pl_bar * v_et, lam_l));
  T rhor_et = (T)1.0 / ((T)1.0 / rhor + qdiv(vnr - v_et, lam_r));
  T pr_bar = pr + lam_r * (v_et - vnr);
  sre[0] = rhor_et;
  for (int k = 1; k < 4; ++k) sre[k] = rhor_et * (wr[k] + (v_et - vnr) * n[k - 1]);
  sre[4] = rhor_et * (er + qdiv(pr_bar * v_et - pr * vnr, lam_r));
  bool ok = !(rhol_et < (T)0 || rhor_et < (T)0);
  T sl = vnl - lam_l / rhol;
  T sr = vnr + lam_r / rhor;
  // The pressure-jump term 0.5 (p*_r - p*_l) (0, n, v*) in FP64 whatever T is:
  // p*_r - p*_l = (lambda_l + lambda_r)(v* - vbar), so its sum over the node's subfaces
  // is M v* - R, which the FP64 nodal solve closes; with the same normal velocities and
  // pressures as vbar (the T-precision ones) the node's momentum and energy balance
  // then holds to FP64 rounding and the totals stay conserved. For T = double these
  // are the reference's expressions (:264-285) unchanged.
  const double vet64 = vn_nodal;
  const double plb64 = (double)pl - lam_l64 * (vet64 - (double)vnl);
  const double prb64 = (double)pr + lam_r64 * (vet64 - (double)vnr);
  const double e64[5] = {0.0, n64[0], n64[1], n64[2], vet64};
  for (int k = 0; k < 5; ++k) {
    T base = (T)0.5 * (fl[k] + fr[k]) -
             (T)0.5 * (fabs(sl) * (sle[k] - ul[k]) + fabs(v_et) * (sre[k] - sle[k]) + fabs(sr) * (ur[k] - sre[k]));
    const double jump = 0.5 * (prb64 - plb64) * e64[k];
    lr[0][k] = (double)base - jump;
    lr[1][k] = -((double)base + jump);
  }
  *sl_o = (double)sl;
  *sr_o = (double)sr;
  return ok;
}

// The 3x3 solve that ends each iteration of compute_lambdas_and_solve_nodal_velocity
// (ns_euler_rs_module.F90:404-421): bc_style 2 with a wall at the node imposes the wall
// pressure through B_p (pseudo-inverse of M); otherwise M v = R by LU (bc_style 2) or
// the pseudo-inverse (bc_style 0, 1). FP64. mat is overwritten.
__device__ void nodal_solve(const int bc_style, double mat[3][3], const double* Rp, const double* Bp, double* vnode) {
  if (bc_style == 2) {
    double bmax = fmax2(fmax2(fabs(Bp[0]), fabs(Bp[1])), fabs(Bp[2]));
    if (bmax > 1e-8) {
      pinv3(mat);
      double mr[3], mb[3], r2[3];
      for (int d = 0; d < 3; ++d) {
        double s = 0.0, t = 0.0;
        for (int e = 0; e < 3; ++e) {
          s = s + mat[d][e] * Rp[e];
          t = t + mat[d][e] * Bp[e];
        }
        mr[d] = s;
        mb[d] = t;
      }
      double p_bound = qdiv(dotT(mr, Bp), dotT(mb, Bp));
      for (int d = 0; d < 3; ++d) r2[d] = Rp[d] - p_bound * Bp[d];
      for (int d = 0; d < 3; ++d) {
        double s = 0.0;
        for (int e = 0; e < 3; ++e) s = s + mat[d][e] * r2[e];
        vnode[d] = s;
      }
      double f = qdiv(dotT(vnode, Bp), dotT(Bp, Bp));
      for (int d = 0; d < 3; ++d) vnode[d] = vnode[d] - f * Bp[d];
    } else {
      lu_solve3(mat, vnode, Rp);
    }
  } else {
    pinv3(mat);
    for (int d = 0; d < 3; ++d) {
      double s = 0.0;
      for (int e = 0; e < 3; ++e) s = s + mat[d][e] * Rp[e];
      vnode[d] = s;
    }
  }
}

// vbar = (lambda_l v_l + lambda_r v_r - (p_r - p_l)) / (lambda_r + lambda_l) (:309,316),
// always in FP64 from the normal velocities and pressures the flux itself uses: with
// FP32 wave speeds the node's momentum balance sum A (p*_r - p*_l) n =
// sum A (lambda_l + lambda_r)(v* - vbar) n, which the FP64 solve of M v* = R closes,
// then holds to FP64 rounding (with an FP64 flux), so the totals stay conserved.
__device__ inline double vbar_of(double lam_l, double lam_r, double vnl, double vnr, double pl, double pr) {
  return qdiv(lam_l * vnl + lam_r * vnr - (pr - pl), lam_r + lam_l);
}

}  // namespace
}  // namespace subfv
