// The node kernel of the multi_point and two_wave schemes in tiles of vertices
// (compute_rhs_around_vert, src/ns/ns_euler_module.F90:341-519): reconstruction, nodal
// velocity solver, subface fluxes and corner sums of a vertex.
//
// A block holds one tile: 256 threads, one per (vertex, position in the vertex's lists),
// vertex fastest, and a solving warp. Its phases, with block barriers between them, each run at the
// parallelism their data have:
//   corners   position k: the state of the vertex's k-th cell at the vertex
//             (reconstruction), with its sound speed, energy and reciprocals, once per
//             corner instead of once per subface side; kept in shared memory
//   subfaces  position j: subface j's wave-speed bounds and terms of M and R
//   sums      a thread per (vertex, component): the terms added in subface order
//   solve     a thread per vertex in the solving warp, which does nothing else: its
//             matrices and the other threads' subface states share the registers instead
//             of adding up
//   fluxes    position j: subface j's flux pair; then the corners' sums in subface order
// The expressions and the order of every sum are those of ns_node_vertex (ns.cu), so the
// results are the same bits. What bounds it: the FP64 divisions and square roots of these
// expressions (instruction issue 40%, FP64 pipe 25% on 39k triangles) and the barriers
// between phases. A thread per vertex kept 1.5 KB of per-subface arrays in local memory and
// recomputed a corner's state for each of its subface sides (201 us a launch there, 80 us
// here); a lane group per vertex repeated the 3x3 solve in every lane (64x64
// quadrilaterals 31 -> 19 us, 29k triangles two-wave 89 -> 40 us).
//
// A tile is 32 vertices of up to 8 subfaces (quadrilateral slabs), 16 of up to 16
// (triangle slabs, boxes) or 8 of up to 32: the vertices are sorted by subface count
// (vorder), so a tile's threads are nearly all used and the block always has as many.
#include <algorithm>

#include "ns.cuh"
#include "ns_device.cuh"

namespace subfv {

namespace {

template <class T>
__device__ inline T recip(T b) {
  return (T)1.0 / b;
}

constexpr int kTileThreads = 256, kTileBlock = kTileThreads + 32;
// Blocks per SM: three at 72 registers beat two at 96 (39k triangles, 24 second-order
// iterations: 14.9 against 16.3 ms; 64 tubes: 133 against 145 ms); shared memory, 59 KB a
// block, allows three as well.
constexpr int kTileBlocksPerSm = 3;
// A vertex of a one-layer slab or a hexahedral box has at most half as many corners as
// positions. Inside layers of prisms or tetrahedra it has two thirds as many corners as
// subfaces and may have more than its tile holds; the other kernels serve such a mesh.
constexpr int kTileCorners = kTileThreads / 2;
// log2 of a tile's vertices by class: the vertices with up to 8, 16 and 32 subfaces
__host__ __device__ constexpr int tile_log2(int cls) { return 5 - cls; }

// corner records: rho, u, v, w, p, E, E / rho, 1 / rho, sound speed and its reciprocal,
// field f of record k and vertex x at rec[f * kRecs + (k << log2) + x]: the corners (at most
// half as many as positions), then each subface's ghost state
constexpr int kRecs = 384;
enum { kRho, kU, kV, kW, kP, kE, kEl, kIr, kA, kIa, kRecFields };

template <class T>
struct TileSmem {
  double term[12][kTileThreads];  // component c of the thread's subface
  double sum[12][32];
  double vn[3][32];
  int nsf[32];
  T rec[kRecFields * kRecs];
};

// the record of the primitive state w (its density's reciprocal ir given); AL: the
// precision the scheme takes the sound speed in
template <class T, class AL>
__device__ inline void put_record(T* r, const T* w, const T ir) {
  const T E = div_by(w[4], (T)(G - 1), (T)(1.0 / (G - 1))) + (T)0.5 * w[0] * (w[1] * w[1] + w[2] * w[2] + w[3] * w[3]);
  for (int k = 0; k < 5; ++k) r[kRecs * k] = w[k];
  r[kRecs * kE] = E;
  r[kRecs * kEl] = div_by(E, w[0], ir);
  r[kRecs * kIr] = ir;
  AL a;
  if constexpr (sizeof(AL) == sizeof(T)) a = sqrt(div_by((AL)G * w[4], w[0], ir));
  else a = sqrt((AL)G * (AL)w[4] / (AL)w[0]);
  r[kRecs * kA] = (T)a;
  if (sizeof(AL) == 8) r[kRecs * kIa] = recip((T)a);
}

// c2p with the density's reciprocal returned
template <class T>
__device__ inline T c2p_ir(const T* u, T* w) {
  const T ir = recip(u[0]);
  w[0] = u[0];
  for (int k = 1; k < 4; ++k) w[k] = div_by(u[k], u[0], ir);
  w[4] = (T)(G - 1) * (u[4] - (T)0.5 * w[0] * (w[1] * w[1] + w[2] * w[2] + w[3] * w[3]));
  return ir;
}

// The solving warp's part of a tile: the 3x3 systems of the nodal solver's iterations, and
// the block's barriers.
__device__ inline void tile_solver(const DevMesh& m, const int bc_style, const int t0, const int nvt, const double* sums,
                                   double* vn) {
  const int x = threadIdx.x & 31;
  const bool live = x < nvt;
  double vv[3] = {0.0, 0.0, 0.0};
  for (int iter = 1; iter <= 4; ++iter) {
    if (!__syncthreads_or(0)) break;
    __syncthreads();
    if (live) {
      const double* a = sums + x;
      double mat[3][3] = {{a[0], a[32], a[64]}, {a[32], a[96], a[128]}, {a[64], a[128], a[160]}};
      const double Rp[3] = {a[192], a[224], a[256]}, Bp[3] = {a[288], a[320], a[352]};
      nodal_solve(bc_style, mat, Rp, Bp, vv);
      for (int d = 0; d < 3; ++d) vn[32 * d + x] = vv[d];
    }
    __syncthreads();
  }
  if (live) m.vp[m.vorder[t0 + x]] = make_double4(vv[0], vv[1], vv[2], 0.0);
}

// One tile: the vertices vorder[t0 .. t0 + nvt - 1], nvt <= 2^log2; every thread of the
// block calls.
template <class T, class L, int SCH>
__device__ void ns_node_tile(const DevMesh& m, const NsParams& P, const double* __restrict__ U,
                             const double* __restrict__ grad, double* __restrict__ fs, const int so, const int tile,
                             const int t0, const int nvt, const int log2, const NsScalars* sc, TileSmem<T>& sm) {
  using AL = typename std::conditional<SCH == 4, T, L>::type;
  if (threadIdx.x >= kTileThreads) {
    __syncthreads();  // corner records
    if (SCH == 1) tile_solver(m, P.bc_style, t0, nvt, &sm.sum[0][0], &sm.vn[0][0]);
    __syncthreads();  // flux terms
    return;
  }
  const int tv = 1 << log2;                                          // vertices, and threads between positions
  const int x = threadIdx.x & (tv - 1), w = threadIdx.x >> log2;     // this thread's vertex and position
  const int S = kTileThreads >> log2;                                // positions
  // this thread's subface, loaded beside the corners' states
  const int2 vs = m.vslot[(size_t)kTileThreads * tile + threadIdx.x];
  const bool mine = vs.x >= 0;
  const int nsfn = mine ? (vs.y >> 26) + 1 : 0;
  double n[4] = {0.0, 0.0, 0.0, 0.0};
  if (mine) {
    const double4 sn = m.sfn[vs.x];
    n[0] = sn.x;
    n[1] = sn.y;
    n[2] = sn.z;
    n[3] = sn.w;
  }
  const int c = threadIdx.x < kTileCorners ? m.vcorner[(size_t)kTileCorners * tile + threadIdx.x].y : -1;
  if (c >= 0) {
    double u64[5];
    ld5(U, c, u64);
    T u[5], ws[5];
    for (int i = 0; i < 5; ++i) u[i] = (T)u64[i];
    T ir = c2p_ir(u, ws);
    if (so) {
      const double4 cc = m.cc[c], xv = m.x[m.vorder[t0 + x]];
      const T dx[3] = {(T)(xv.x - cc.x), (T)(xv.y - cc.y), (T)(xv.z - cc.z)};
      const double* g = grad + 15 * (size_t)c;
      for (int i = 0; i < 5; ++i) {
        T s = 0;
        for (int d = 0; d < 3; ++d) s = s + (T)g[5 * d + i] * dx[d];
        ws[i] = ws[i] + s;
      }
      ir = recip(ws[0]);
    }
    put_record<T, AL>(sm.rec + (w << log2) + x, ws, ir);
  }
  if (w == 0) sm.nsf[x] = nsfn;
  __syncthreads();
  const int kl = mine ? vs.y & 31 : 0;
  int kr = mine ? (vs.y >> 5) & 31 : 0;
  bool wall = false;
  if (mine && kr == 31) {  // a boundary subface: its ghost state in a record of its own
    const int y = -1 - ((vs.y >> 10) & 0xffff);
    wall = is_wall(P, y);
    const T* r = sm.rec + (kl << log2) + x;
    const T nt[3] = {(T)n[0], (T)n[1], (T)n[2]};
    T uc[5], gh[5], wr[5];
    uc[0] = r[kRecs * kRho];
    for (int k = 1; k < 4; ++k) uc[k] = r[kRecs * k] * uc[0];
    uc[4] = r[kRecs * kE];
    right_state(m, P, y, vs.x, nt, uc, gh, sc);
    const T ir = c2p_ir(gh, wr);
    kr = (S >> 1) + w;  // the ghost records follow the corners'
    put_record<T, AL>(sm.rec + (kr << log2) + x, wr, ir);
  }
  const T *rl = sm.rec + (kl << log2) + x, *rr = sm.rec + (mine ? (kr << log2) + x : 0);
  double* term = &sm.term[0][threadIdx.x];  // component c of this subface: term[tc * c]
  constexpr int tc = kTileThreads;
  L lam_l = (L)0, lam_r = (L)0;
  double vn3[3] = {0.0, 0.0, 0.0};
  if (SCH == 1) {  // compute_lambdas_and_solve_nodal_velocity (ns_euler_rs_module.F90:288-422)
    const L c1 = (L)1, c15 = (L)1.5, c0 = (L)0;
    L vnl = 0, vnr = 0, al = 0, ar = 0, ial = 0, iar = 0, arl = 0, arr = 0;
    double vnl_f = 0.0, vnr_f = 0.0, pl_f = 0.0, pr_f = 0.0;
    // which sums the subface enters: M; R through q; R through the wall pressure
    const bool in_m = mine && (!wall || P.bc_style == 0 || P.bc_style == 2);
    const bool in_q = mine && (!wall || P.bc_style == 0);
    const bool in_p = mine && !in_q && P.bc_style == 2 && (!P.b2d || fabs(n[2]) < 1e-8);
    if (mine) {
      const L nl[3] = {(L)n[0], (L)n[1], (L)n[2]};
      const L vl[3] = {(L)rl[kRecs * kU], (L)rl[kRecs * kV], (L)rl[kRecs * kW]};
      const L vr[3] = {(L)rr[kRecs * kU], (L)rr[kRecs * kV], (L)rr[kRecs * kW]};
      vnl = dotT(vl, nl);
      vnr = dotT(vr, nl);
      al = (L)rl[kRecs * kA];
      ar = (L)rr[kRecs * kA];
      if (sizeof(L) == 8) {
        ial = (L)rl[kRecs * kIa];
        iar = (L)rr[kRecs * kIa];
      }
      // the flux's own normal velocities and pressures (precision T), for vbar
      if constexpr (sizeof(L) == sizeof(T)) {
        vnl_f = (double)vnl;
        vnr_f = (double)vnr;
      } else {
        const T nt[3] = {(T)n[0], (T)n[1], (T)n[2]};
        const T tvl[3] = {rl[kRecs * kU], rl[kRecs * kV], rl[kRecs * kW]}, tvr[3] = {rr[kRecs * kU], rr[kRecs * kV], rr[kRecs * kW]};
        vnl_f = (double)dotT(tvl, nt);
        vnr_f = (double)dotT(tvr, nt);
      }
      pl_f = (double)rl[kRecs * kP];
      pr_f = (double)rr[kRecs * kP];
      const L rhol = (L)rl[kRecs * kRho], rhor = (L)rr[kRecs * kRho], pl = (L)rl[kRecs * kP], pr = (L)rr[kRecs * kP];
      arl = al * rhol;
      arr = ar * rhor;
      // one of the two pressure jumps is positive at most: one square root serves both
      const bool up = pr > pl;
      const L sq = qsqrt(up ? rhol * tmax2(c0, pr - pl) : rhor * tmax2(c0, pl - pr));
      lam_l = tmax2(tmax2(tmax2(lam_l, arl), up ? sq : rhol * tmax2(c0, pr - pl)), -rhol * (vnr - vnl));
      lam_r = tmax2(tmax2(tmax2(lam_r, arr), up ? rhor * tmax2(c0, pl - pr) : sq), -rhor * (vnr - vnl));
      const double vb = vbar_of((double)lam_l, (double)lam_r, vnl_f, vnr_f, pl_f, pr_f);
      lam_l = tmax2(lam_l, arl * (c1 + c15 * tmax2(c0, div_by(-((L)vb - vnl), al, ial))));
      lam_r = tmax2(lam_r, arr * (c1 + c15 * tmax2(c0, div_by((L)vb - vnr, ar, iar))));
    }
    // wall_normal (ns_euler_primitives_module.F90:162-190): components 9-11 of the sums
    {
      const bool b = wall && !(P.b2d && fabs(n[2]) > 1e-12);
      for (int d = 0; d < 3; ++d) term[tc * (9 + d)] = b ? n[3] * n[d] : 0.0;
      for (int d = 0; d < 9; ++d) term[tc * d] = 0.0;  // a sum is never -0: adding +0 leaves it
    }
    const int nsfx = sm.nsf[x];  // subfaces of this thread's vertex
    for (int iter = 1; iter <= 4; ++iter) {
      bool changed = iter == 1;
      if (mine && iter > 1) {
        L xl, xr;
        if (wall && P.bc_style == 1) {  // the previous iteration's vbar, from the bounds it ended with
          const L vb = (L)vbar_of((double)lam_l, (double)lam_r, vnl_f, vnr_f, pl_f, pr_f);
          xl = -(vb - vnl);
          xr = vb - vnr;
        } else {
          const L v_et = (L)dotT(vn3, n);
          xl = -(v_et - vnl);
          xr = v_et - vnr;
        }
        const L nl = tmax2(lam_l, arl * (c1 + c15 * tmax2(c0, div_by(xl, al, ial))));
        const L nr = tmax2(lam_r, arr * (c1 + c15 * tmax2(c0, div_by(xr, ar, iar))));
        changed = !(nl == lam_l && nr == lam_r);
        lam_l = nl;
        lam_r = nr;
      }
      // A subface whose bounds stayed keeps its terms; when every bound of the tile stayed,
      // M, R and the velocity are the previous iteration's and so are all later ones.
      if (mine && changed) {
        const double lsum = (double)lam_r + (double)lam_l;
        if (in_m) {  // M += (lam_r + lam_l) A n n^T
          const double wgt = lsum * n[3];
          term[tc * 0] = wgt * (n[0] * n[0]);
          term[tc * 1] = wgt * (n[0] * n[1]);
          term[tc * 2] = wgt * (n[0] * n[2]);
          term[tc * 3] = wgt * (n[1] * n[1]);
          term[tc * 4] = wgt * (n[1] * n[2]);
          term[tc * 5] = wgt * (n[2] * n[2]);
        }
        if (in_q || in_p) {
          const double q = in_q ? n[3] * lsum * vbar_of((double)lam_l, (double)lam_r, vnl_f, vnr_f, pl_f, pr_f)
                                : n[3] * (double)(L)pl_f;
          for (int d = 0; d < 3; ++d) term[tc * (6 + d)] = q * n[d];
        }
      }
      if (!__syncthreads_or(changed)) break;
      for (int i = threadIdx.x; i < ((iter == 1 ? 12 : 9) << log2); i += kTileThreads) {
        const int c = i >> log2;  // (i - threadIdx.x is a multiple of the tile's vertices: i is vertex x)
        const double* tr = &sm.term[c][x];
        double s = 0.0;
        for (int j = 0; j < nsfx; ++j) s = s + tr[j << log2];
        sm.sum[c][x] = s;
      }
      __syncthreads();
      // (the solving warp's 3x3 systems)
      __syncthreads();
      for (int d = 0; d < 3; ++d) vn3[d] = sm.vn[d][x];
    }
    // the sums' readers are past their barrier: the terms may be overwritten
  }
  if (mine) {
    // The flux pair one component at a time, its states read from the records as they are
    // needed: u_k = w_k rho (the energy from the record), f_k = v_n u_k + p n_k.
    const T nt[3] = {(T)n[0], (T)n[1], (T)n[2]};
    const T vl[3] = {rl[kRecs * kU], rl[kRecs * kV], rl[kRecs * kW]}, vnl = dotT(vl, nt);
    const T vr[3] = {rr[kRecs * kU], rr[kRecs * kV], rr[kRecs * kW]}, vnr = dotT(vr, nt);
    const T rhol = rl[kRecs * kRho], pl = rl[kRecs * kP], irl = rl[kRecs * kIr];
    const T rhor = rr[kRecs * kRho], pr = rr[kRecs * kP], irr = rr[kRecs * kIr];
    const double area = n[3];
    T sl, sr;
    auto cons = [&](const T* r, T rho, int k) { return k == 0 ? rho : k == 4 ? r[kRecs * kE] : r[kRecs * k] * rho; };
    auto flux = [&](T vn, T u, T p, int k) { return k == 0 ? vn * u : k == 4 ? (u + p) * vn : vn * u + p * nt[k - 1]; };
    if (SCH == 1) {  // multi_point (ns_euler_rs_module.F90:200-286), as multi_point() of ns_device.cuh
      const double vet64 = wall ? 0.0 : dotT(vn3, n);
      const double lam_l64 = (double)lam_l, lam_r64 = (double)lam_r;
      const T tl_l = (T)lam_l64, tl_r = (T)lam_r64, v_et = (T)vet64;
      const T ill = recip(tl_l), ilr = recip(tl_r);
      const T rhol_et = (T)1.0 / (irl + div_by(v_et - vnl, tl_l, ill));
      const T rhor_et = (T)1.0 / (irr + div_by(vnr - v_et, tl_r, ilr));
      const T pl_bar = pl - tl_l * (v_et - vnl);
      const T pr_bar = pr + tl_r * (v_et - vnr);
      const T el_et = rhol_et * (rl[kRecs * kEl] + div_by(pl * vnl - pl_bar * v_et, tl_l, ill));
      const T er_et = rhor_et * (rr[kRecs * kEl] + div_by(pr_bar * v_et - pr * vnr, tl_r, ilr));
      if (rhol_et < (T)0 || rhor_et < (T)0) atomicOr(m.status, kErrNegDensity);
      sl = vnl - div_by(tl_l, rhol, irl);
      sr = vnr + div_by(tl_r, rhor, irr);
      const double plb64 = (double)pl - lam_l64 * (vet64 - (double)vnl);
      const double prb64 = (double)pr + lam_r64 * (vet64 - (double)vnr);
      const double hj = 0.5 * (prb64 - plb64);
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const T ulk = cons(rl, rhol, k), urk = cons(rr, rhor, k);
        const T flk = flux(vnl, ulk, pl, k), frk = flux(vnr, urk, pr, k);
        const T slek = k == 0 ? rhol_et
                              : k == 4 ? el_et : rhol_et * (rl[kRecs * k] + (v_et - vnl) * nt[k == 4 ? 0 : k - 1]);
        const T srek = k == 0 ? rhor_et
                              : k == 4 ? er_et : rhor_et * (rr[kRecs * k] + (v_et - vnr) * nt[k == 4 ? 0 : k - 1]);
        const T base = (T)0.5 * (flk + frk) -
                       (T)0.5 * (fabs(sl) * (slek - ulk) + fabs(v_et) * (srek - slek) + fabs(sr) * (urk - srek));
        const double jump = hj * (k == 0 ? 0.0 : k == 4 ? vet64 : n[k - 1]);
        term[tc * k] = area * ((double)base - jump);
        term[tc * (6 + k)] = area * (-((double)base + jump));
      }
    } else {  // two_wave (ns_euler_rs_module.F90:154-198)
      const T al = rl[kRecs * kA], ar = rr[kRecs * kA], c0 = (T)0;
      const bool up = pr > pl;
      const T sq = qsqrt(up ? rhol * tmax2(c0, pr - pl) : rhor * tmax2(c0, pl - pr));
      const T ll = tmax2(tmax2(al * rhol, up ? sq : rhol * tmax2(c0, pr - pl)), -rhol * (vnr - vnl));
      const T lr = tmax2(tmax2(ar * rhor, up ? rhor * tmax2(c0, pl - pr) : sq), -rhor * (vnr - vnl));
      sl = vnl - div_by(ll, rhol, irl);
      sr = vnr + div_by(lr, rhor, irr);
      const T den = sr - sl, iden = recip(den);
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const T ulk = cons(rl, rhol, k), urk = cons(rr, rhor, k);
        const T flk = flux(vnl, ulk, pl, k), frk = flux(vnr, urk, pr, k);
        const T et = div_by(sr * urk - sl * ulk - (frk - flk), den, iden);
        const T f = (T)0.5 * (flk + frk) - (T)0.5 * (fabs(sl) * (et - ulk) + fabs(sr) * (urk - et));
        term[tc * k] = area * (double)f;
        term[tc * (6 + k)] = area * (double)(-f);
      }
    }
    term[tc * 5] = area * fmax2(0.0, (double)-sl);
    term[tc * 11] = area * fmax2(0.0, (double)sr);
  }
  __syncthreads();
  // corner sums: a task per corner and half of the six components, in subface order
  {
    const int half = threadIdx.x / kTileCorners, c0 = 3 * half;
    const int4 cs = m.vcorner[(size_t)kTileCorners * tile + threadIdx.x - half * kTileCorners];
    if (cs.x < 0) return;  // no corner, or another vertex's subcell
    double s[3] = {0.0, 0.0, 0.0};
    for (unsigned b = (unsigned)cs.z | (unsigned)cs.w; b; b &= b - 1) {
      const int j = __ffs(b) - 1;
      const double* tr = &sm.term[c0][(j << log2) + x];
      if ((cs.z >> j) & 1)
        for (int i = 0; i < 3; ++i) s[i] = s[i] + tr[tc * i];
      if ((cs.w >> j) & 1)
        for (int i = 0; i < 3; ++i) s[i] = s[i] + tr[tc * (6 + i)];
    }
    double* out = fs + kNsFs * (size_t)cs.x + c0;
    for (int i = 0; i < 3; ++i) out[i] = s[i];
  }
}

// The tile with index t of a mesh: its class, first vertex position and vertex count.
__device__ inline void tile_at(const DevMesh& m, int t, int* log2, int* t0, int* nvt) {
  int begin = 0;
  for (int c = 0; c < 3; ++c) {
    const int l = tile_log2(c), end = m.tile_end[c], tiles = (end - begin + (1 << l) - 1) >> l;
    if (t < tiles || c == 2) {
      *log2 = l;
      *t0 = begin + (t << l);
      *nvt = min(1 << l, end - *t0);
      return;
    }
    t -= tiles;
    begin = end;
  }
}

extern __shared__ __align__(16) char g_tile_smem[];

template <class T, class L, int SCH>
__global__ void __launch_bounds__(kTileBlock, kTileBlocksPerSm) k_ns_node_tile(DevMesh m, NsParams P, const double* __restrict__ U,
                                                                  const double* __restrict__ grad,
                                                                  double* __restrict__ fs, int so,
                                                                  const NsScalars* sc) {
  if (sc && sc->done) return;
  int log2, t0, nvt;
  tile_at(m, blockIdx.x, &log2, &t0, &nvt);
  ns_node_tile<T, L, SCH>(m, P, U, grad, fs, so, blockIdx.x, t0, nvt, log2, sc, *reinterpret_cast<TileSmem<T>*>(g_tile_smem));
}

// the batched form: the tiles of every problem of the table (wt: their prefix) are shared
// out one by one; which: the state the phase reads (0: U0, 1: U1)
template <class T, class L, int SCH>
__global__ void __launch_bounds__(kTileBlock, kTileBlocksPerSm) kb_ns_node_tile(const NsItem* __restrict__ it,
                                                                   const int* __restrict__ wt,
                                                                   const int* __restrict__ hdr, NsParams P, int which,
                                                                   int so) {
  const int n = hdr[0], tiles = wt[n];
  for (int u = blockIdx.x; u < tiles; u += gridDim.x) {
    int lo = 0, hi = n;  // the problem of tile u
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (wt[mid] <= u) lo = mid;
      else hi = mid;
    }
    const NsItem& I = it[lo];
    if (I.sc->done) continue;
    int log2, t0, nvt;
    tile_at(I.m, u - wt[lo], &log2, &t0, &nvt);
    ns_node_tile<T, L, SCH>(I.m, P, which ? I.U1 : I.U0, I.grad, I.fs, so, u - wt[lo], t0, nvt, log2, I.sc,
                            *reinterpret_cast<TileSmem<T>*>(g_tile_smem));
    __syncthreads();  // the corner sums' reads before the next tile's terms
  }
}

// The codes of a tile, laid out as its threads read them. vslot[256 tile + thread]: the
// subface (-1: none), then from bit 0 its left cell's corner (5 bits), its right cell's (5
// bits, 31: boundary), the boundary's tag (16 bits) and the vertex's subface count less one
// (5 bits). vcorner[128 tile + thread]: the subcell that a corner's sums go to (-1: none),
// its cell (-1: no corner) and the positions whose left / right flux enters its sums. A
// vertex's corners are its own subcells, then the other cells of its subfaces (a periodic
// vertex's list holds its images' subfaces). Both arrays start as -1. fail: a vertex has
// more corners than the tile's class, or a tag beyond its bits; with CHECK that is all the
// kernel finds out.
template <bool CHECK>
__global__ void k_build_node_codes(DevMesh m, int2* __restrict__ vslot, int4* __restrict__ vcorner, unsigned* fail) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m.nv) return;
  const int cls = i < m.tile_end[0] ? 0 : i < m.tile_end[1] ? 1 : 2, log2 = tile_log2(cls);
  int tile = 0, begin = 0;
  for (int c = 0; c < cls; begin = m.tile_end[c++])
    tile += (m.tile_end[c] - begin + (1 << tile_log2(c)) - 1) >> tile_log2(c);
  tile += (i - begin) >> log2;
  const int x = (i - begin) & ((1 << log2) - 1);
  int2* slot = vslot + (size_t)kTileThreads * tile + x;
  int4* corner = vcorner + (size_t)kTileCorners * tile + x;
  const int v = m.vorder[i], p0 = m.vsf_off[v], ns = m.vsf_off[v + 1] - p0;
  const int q0 = m.vse_off[v], nq = m.vse_off[v + 1] - q0, cap = 4 << cls;
  int sub[16], cell[16], nc = 0;
  unsigned lm[16], rm[16];
  bool ok = true;
  for (int q = 0; q < nq; ++q) {
    const int s = m.vse[q0 + q];
    if (m.se_vert[s] != v) continue;
    if (nc == cap) {
      ok = false;
      break;
    }
    sub[nc] = s;
    cell[nc] = m.se_elem[s];
    lm[nc] = rm[nc] = 0u;
    ++nc;
  }
  auto corner_of = [&](int c) {
    for (int k = 0; k < nc; ++k)
      if (cell[k] == c) return k;
    if (nc == cap) {
      ok = false;
      return 0;
    }
    sub[nc] = -1;
    cell[nc] = c;
    lm[nc] = rm[nc] = 0u;
    return nc++;
  };
  for (int j = 0; ok && j < ns; ++j) {
    const int sf = m.vsf[p0 + j];
    const int2 lr = m.flr[m.sf_face[sf]];
    const int kl = corner_of(lr.x), kr = lr.y < 0 ? 31 : corner_of(lr.y);
    const unsigned tag = lr.y < 0 ? (unsigned)(-1 - lr.y) : 0u;
    if (tag > 0xffffu) ok = false;
    if (!CHECK) slot[j << log2] = make_int2(sf, (int)((unsigned)kl | ((unsigned)kr << 5) | (tag << 10) | ((unsigned)(ns - 1) << 26)));
    if (CHECK) continue;
    // the flux enters the sums of this vertex's subcells, by their positions in its list
    const int2 se = m.sf_se[sf];
    if (m.se_vert[se.x] == v && m.se_loc[se.x] < nq) {
      for (int k = 0; k < nc; ++k)
        if (sub[k] >= 0 && sub[k] == m.vse[q0 + m.se_loc[se.x]]) lm[k] |= 1u << j;
      if (se.y >= 0 && m.se_vert[se.y] == v && m.se_loc[se.y] < nq)
        for (int k = 0; k < nc; ++k)
          if (sub[k] >= 0 && sub[k] == m.vse[q0 + m.se_loc[se.y]]) rm[k] |= 1u << j;
    }
  }
  if (CHECK) {
    if (!ok) *fail = 1;
  } else {
    for (int k = 0; k < nc; ++k) corner[k << log2] = make_int4(sub[k], cell[k], (int)lm[k], (int)rm[k]);
  }
}

template <class T, class L, int SCH>
void launch_tile_t(const DevMesh& m, const NsParams& P, const double* U, const double* grad, double* fs, int so,
                   const NsScalars* sc) {
  constexpr int smem = (int)sizeof(TileSmem<T>);
  cudaFuncSetAttribute(k_ns_node_tile<T, L, SCH>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  k_ns_node_tile<T, L, SCH><<<node_tiles(m), kTileBlock, smem, m.stream>>>(m, P, U, grad, fs, so, sc);
}
template <class T, class L, int SCH>
void launch_kb_tile_t(const NsTable& t, const NsParams& P, cudaStream_t s, int which, int so) {
  constexpr int smem = (int)sizeof(TileSmem<T>);
  cudaFuncSetAttribute(kb_ns_node_tile<T, L, SCH>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  kb_ns_node_tile<T, L, SCH><<<t.grid_v, kTileBlock, smem, s>>>(t.items, t.wt, t.hdr, P, which, so);
}

}  // namespace

// multi_point with excluded boundary vertices mixes two fluxes: the other kernels take it
bool node_tile_scheme(const NsParams& P) { return P.scheme == 4 || (P.scheme == 1 && !P.excl); }

int node_tiles(const DevMesh& m) {
  int t = 0;
  for (int c = 0, begin = 0; c < 3; begin = m.tile_end[c++])
    t += (m.tile_end[c] - begin + (1 << tile_log2(c)) - 1) >> tile_log2(c);
  return t;
}
bool node_tile_serves(const DevMesh& m, const NsParams& P) { return m.node_codes && node_tile_scheme(P); }
bool node_tile_serves(const NsTable& t, const NsParams& P) { return t.tiles && node_tile_scheme(P); }

int64_t node_codes_bytes(const DevMesh& m) {
  return (int64_t)node_tiles(m) * (int64_t)(kTileThreads * sizeof(int2) + kTileCorners * sizeof(int4));
}

void launch_check_node_codes(const DevMesh& m, unsigned* fail) {
  if (node_tiles(m)) k_build_node_codes<true><<<grid_for(m.nv, 128), 128, 0, m.stream>>>(m, nullptr, nullptr, fail);
}

int ensure_node_codes(DevMesh* m, const NsParams& P) {
  if (m->node_codes || !node_tile_scheme(P) || !node_tiles(*m)) return 0;
  const size_t nt = node_tiles(*m), sb = nt * kTileThreads * sizeof(int2), cb = nt * kTileCorners * sizeof(int4);
  int2* slots = nullptr;
  int4* corners = nullptr;
  if (cudaMallocAsync((void**)&slots, sb, m->stream) != cudaSuccess ||
      cudaMallocAsync((void**)&corners, cb, m->stream) != cudaSuccess) {
    cudaGetLastError();
    if (slots) cudaFreeAsync(slots, m->stream);
    return 0;
  }
  m->vslot = slots;
  m->vcorner = corners;
  m->node_codes = 1;
  SUBFV_CUDA(cudaMemsetAsync(m->vslot, 0xff, sb, m->stream));
  SUBFV_CUDA(cudaMemsetAsync(m->vcorner, 0xff, cb, m->stream));
  k_build_node_codes<false><<<grid_for(m->nv, 128), 128, 0, m->stream>>>(*m, m->vslot, m->vcorner, nullptr);
  SUBFV_CUDA(cudaGetLastError());
  return 0;
}

void launch_node_tile(const DevMesh& m, const NsParams& P, const double* U, const double* grad, double* fs, int so,
                      const NsScalars* sc) {
  if (P.scheme == 4) {
    if (P.precision == 2) launch_tile_t<float, float, 4>(m, P, U, grad, fs, so, sc);
    else launch_tile_t<double, double, 4>(m, P, U, grad, fs, so, sc);
    return;
  }
  if (P.precision == 2) launch_tile_t<float, float, 1>(m, P, U, grad, fs, so, sc);
  else if (P.precision == 1) launch_tile_t<double, float, 1>(m, P, U, grad, fs, so, sc);
  else launch_tile_t<double, double, 1>(m, P, U, grad, fs, so, sc);
}

void launch_kb_node_tile(const NsTable& t, const NsParams& P, cudaStream_t s, int which, int so) {
  if (P.scheme == 4) {
    if (P.precision == 2) launch_kb_tile_t<float, float, 4>(t, P, s, which, so);
    else launch_kb_tile_t<double, double, 4>(t, P, s, which, so);
    return;
  }
  if (P.precision == 2) launch_kb_tile_t<float, float, 1>(t, P, s, which, so);
  else if (P.precision == 1) launch_kb_tile_t<double, float, 1>(t, P, s, which, so);
  else launch_kb_tile_t<double, double, 1>(t, P, s, which, so);
}

}  // namespace subfv
