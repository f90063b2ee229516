// Geometry of compute_geometry_mesh (src/mesh/mesh_geometry_module.F90) as per-entity
// device functions, shared by the solo kernels (mesh_dev.cu) and the batched Lagrangian
// kernels (lagrange.cu).
#pragma once
#include "common.cuh"
#include "mesh_dev.cuh"

namespace subfv {
namespace geo {

struct V3 {
  double x, y, z;
};
__device__ inline V3 ld3(const double4* a, int i) {
  double4 v = a[i];
  return {v.x, v.y, v.z};
}
__device__ inline V3 sub(V3 a, V3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ inline V3 cross(V3 a, V3 b) {
  return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ inline double dot(V3 a, V3 b) { return dot3(a.x, a.y, a.z, b.x, b.y, b.z); }
__device__ inline V3 half_sum(V3 a, V3 b) { return {0.5 * (a.x + b.x), 0.5 * (a.y + b.y), 0.5 * (a.z + b.z)}; }

__device__ inline V3 pick4(const V3 (&P)[4], int i) { return i == 0 ? P[0] : i == 1 ? P[1] : i == 2 ? P[2] : P[3]; }

// s / nvc, the vertex average of compute_elem_centroid: exact shortcuts for the usual
// vertex counts (a power of two scales exactly; div6 is exact), the division otherwise
__device__ inline V3 vertex_mean(V3 s, int nvc) {
  if (nvc == 8) return {s.x * 0.125, s.y * 0.125, s.z * 0.125};
  if (nvc == 4) return {s.x * 0.25, s.y * 0.25, s.z * 0.25};
  if (nvc == 6) return {div6(s.x), div6(s.y), div6(s.z)};
  return {qdiv(s.x, nvc), qdiv(s.y, nvc), qdiv(s.z, nvc)};
}

// compute_face_centroid + compute_subface_norm + compute_face_norm (:177-271), one thread
// per face. Also fS[f] = sum over the face's subfaces (in face%sub_face order) of
// area * unit normal, which the Lagrangian step's cell kernel uses for check_mesh's
// subface closure. FULL = 0 (the Lagrangian step) skips the subface unit normals, which
// the step does not read.
template <int FULL>
__device__ inline void face_geom_body(const DevMesh& m, const int f) {
  if (f >= m.nf) return;
  const int4 fv = m.fvert[f];
  const int vid[4] = {fv.x, fv.y, fv.z, fv.w};
  const int n = fv.w < 0 ? 3 : 4;
  V3 P[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) P[k] = k < n ? ld3(m.x, vid[k]) : V3{0.0, 0.0, 0.0};
  V3 cg = {0.0, 0.0, 0.0};
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (k < n) cg = {cg.x + P[k].x, cg.y + P[k].y, cg.z + P[k].z};
  cg = n == 4 ? V3{cg.x * 0.25, cg.y * 0.25, cg.z * 0.25} : V3{div3(cg.x), div3(cg.y), div3(cg.z)};
  V3 c = {0.0, 0.0, 0.0};
  double sum_area = 0.0;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (j < n) {
      const V3 pj = P[j], pp = pick4(P, j + 1 == n ? 0 : j + 1);
      const V3 x = cross(sub(pj, cg), sub(pp, cg));
      const double area = 0.5 * fnorm2_3(x.x, x.y, x.z);
      c.x = c.x + div3(area * (pj.x + pp.x + cg.x));
      c.y = c.y + div3(area * (pj.y + pp.y + cg.y));
      c.z = c.z + div3(area * (pj.z + pp.z + cg.z));
      sum_area = sum_area + area;
    }
  c = {qdiv(c.x, sum_area), qdiv(c.y, sum_area), qdiv(c.z, sum_area)};
  m.fc[f] = make_double4(c.x, c.y, c.z, 0.0);
  const int4 fs = m.fsf[f];
  const int sfi[4] = {fs.x, fs.y, fs.z, fs.w};
  const unsigned fp = m.fpos[f];
  V3 fnrm = {0.0, 0.0, 0.0}, S = {0.0, 0.0, 0.0};
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (k < n) {
      const int sf = sfi[k];
      const int j = (fp >> (2 * k)) & 3;  // the subface's vertex slot in the face
      const V3 cp = pick4(P, j);
      const V3 cpm = half_sum(pick4(P, j == 0 ? n - 1 : j - 1), cp), cpp = half_sum(pick4(P, j + 1 == n ? 0 : j + 1), cp);
      const V3 a = cross(sub(cpm, c), sub(cp, c));
      const V3 b = cross(sub(cp, c), sub(cpp, c));
      const V3 nr = {0.5 * (a.x + b.x), 0.5 * (a.y + b.y), 0.5 * (a.z + b.z)};
      const double area = fnorm2_3(nr.x, nr.y, nr.z);
      if (FULL) {
        const V3 un = {qdiv(nr.x, area), qdiv(nr.y, area), qdiv(nr.z, area)};
        m.sfn[sf] = make_double4(un.x, un.y, un.z, area);
        S = {S.x + area * un.x, S.y + area * un.y, S.z + area * un.z};
      } else {
        // the step keeps no unit normals: the closure sum takes the area vector itself
        // (A n of the check, up to rounding), which only feeds check_mesh's threshold
        S = {S.x + nr.x, S.y + nr.y, S.z + nr.z};
      }
      m.sfa[sf] = area;
      fnrm = {fnrm.x + nr.x, fnrm.y + nr.y, fnrm.z + nr.z};
    }
  const double fa = fnorm2_3(fnrm.x, fnrm.y, fnrm.z);
  m.fn[f] = make_double4(qdiv(fnrm.x, fa), qdiv(fnrm.y, fa), qdiv(fnrm.z, fa), fa);
  if (m.fS) m.fS[f] = make_double4(S.x, S.y, S.z, 0.0);
}

// The cell part of compute_geometry_mesh for the Lagrangian step, after k_face_geom<0>:
// compute_elem_centroid (:59-110), compute_subelem_volume (:112-160), compute_elem_volume
// (:162-175) and check_mesh (:374-411), then sol += dt * rhs (lagrange_main.F90:110). The
// local topology comes from static codes (built once by build_geom_codes below): no id is
// searched and no face or subface index array but the cell's own is read per step.
// check_mesh_subface_closed adds each face's subface sum S as a whole: the same total as
// the subface-by-subface sum up to rounding, and the test is a 1e-14 threshold on its norm.
// Every face vertex must be a vertex of the cell (no periodic faces); otherwise the cell
// reports SUBFV_ERR_INDEX.
constexpr int kGeoMaxV = 8, kGeoMaxF = 8;
// faces of a cell the step kernel stages (hexahedra have 6, prisms and pyramids 5,
// tetrahedra 4), and the (face, vertex of the face) pairs those can have
constexpr int kGeoCellFaces = 6, kGeoPairs = 24;

// cinfo: bits 0-3 the cell's vertices, 4-7 its faces, 8-12 its pairs, bit 13 valid (at most
// kGeoMaxV vertices and kGeoCellFaces faces, every face vertex found among the cell's
// vertices), bits 16-23 the faces it is the left neighbour of.
// gpair, pair q: bits 0-9 of the q-th (face, vertex k) pair in face order the local indices
// of the face's k-th and next vertex and the face slot (ef8 order), 3 bits each, then
// whether the cell is the face's left neighbour; bits 16-28 of the q-th (vertex, subface)
// pair in vertex order the local indices of the vertex and of the vertices before and after
// it in the face, the face slot, 3 bits each, the left bit and whether it is the vertex's
// last pair. gsub, per subcell: its first
// pair of the second kind, and from bit 8 how many.
constexpr unsigned kCiValid = 1u << 13;
__host__ __device__ inline size_t tile_entry(int c, int per, int q) {
  return ((size_t)(c >> 5) * per + q) * 32 + (c & 31);
}

// check_mesh's closure tests (mesh_geometry_module.F90:374-411) compare a norm2 with
// 1e-14. With every component at most 1 in magnitude gfortran's NORM2 is the correctly
// rounded sqrt(a*a + b*b + c*c), and rounding sqrt to nearest is monotone, so the test
// holds exactly when the sum is below the smallest double whose rounded square root
// reaches 1e-14; a component above 1 (or a NaN) fails both forms. The step's cell kernel
// takes this form and skips the two square roots.
constexpr double kClosedSumSq = 0x1.fb0f6be506018p-94;  // 9.999999999999999e-29
__device__ inline bool norm2_below_1em14(double a0, double a1, double a2) {
  return fabs(a0) <= 1.0 && fabs(a1) <= 1.0 && fabs(a2) <= 1.0 && (a0 * a0 + a1 * a1 + a2 * a2) < kClosedSumSq;
}

// The codes of cell c: a face vertex's local index is its first match among the cell's
// vertices; a subface's face slot is the first slot holding its face (else the last slot)
// and its vertex position the first match in that face (else the last position).
__device__ inline void build_geom_codes(const DevMesh& m, const int c) {
  if (c >= m.ne) return;
  const int vb = m.ev_off[c], nvc = m.ev_off[c + 1] - vb;
  int fid[kGeoMaxF], nfc = 0;
  for (int k = 0; k < kGeoMaxF; ++k) {
    const int f = m.ef8[8 * (size_t)c + k];
    if (f < 0) break;
    fid[nfc++] = f;
  }
  m.cinfo[c] = 0u;
  if (nvc > kGeoMaxV || nfc > kGeoCellFaces) return;
  int vid[kGeoMaxV], loc[kGeoCellFaces][4], fn[kGeoCellFaces];
  for (int k = 0; k < nvc; ++k) vid[k] = m.ev[vb + k];
  bool ok = true;
  unsigned left = 0u;
  int pairs = 0;
  for (int j = 0; j < nfc; ++j) {
    const int4 fv = m.fvert[fid[j]];
    const int gid[4] = {fv.x, fv.y, fv.z, fv.w};
    fn[j] = fv.w < 0 ? 3 : 4;
    for (int k = 0; k < fn[j]; ++k) {
      int q = 0;
      while (q < nvc - 1 && vid[q] != gid[k]) ++q;
      if (vid[q] != gid[k]) ok = false;
      loc[j][k] = q;
    }
    if (m.flr[fid[j]].x == c) left |= 1u << j;
    for (int k = 0; k < fn[j]; ++k, ++pairs)
      m.gpair[tile_entry(c, m.max_pairs, pairs)] =
          (unsigned)(loc[j][k] | (loc[j][k + 1 == fn[j] ? 0 : k + 1] << 3) | (j << 6)) | (((left >> j) & 1u) << 9);
  }
  int at = 0;
  for (int k = 0; k < nvc; ++k) {
    const int4 q4 = m.se_sf[vb + k];
    const int q[4] = {q4.x, q4.y, q4.z, q4.w};
    const int first = at;
    for (int jj = 0; jj < 4; ++jj) {
      if (q[jj] < 0) break;
      const int f = m.sf_face[q[jj]], vert = m.sf_vert[q[jj]];
      int j = 0;
      while (j < nfc - 1 && fid[j] != f) ++j;
      const int n = fn[j];
      int kk = 0;
      while (kk < n - 1 && vid[loc[j][kk]] != vert) ++kk;
      if (at == pairs) {
        ok = false;
        break;
      }
      const unsigned code = (unsigned)(loc[j][kk] | (loc[j][kk == 0 ? n - 1 : kk - 1] << 3) |
                                       (loc[j][kk + 1 == n ? 0 : kk + 1] << 6) | (j << 9)) |
                            (((left >> j) & 1u) << 12);
      m.gpair[tile_entry(c, m.max_pairs, at)] |= code << 16;
      ++at;
    }
    if (at > first) m.gpair[tile_entry(c, m.max_pairs, at - 1)] |= 1u << 29;
    else ok = false;
    m.gsub[vb + k] = (unsigned)first | ((unsigned)(at - first) << 8);
  }
  m.cinfo[c] = (unsigned)nvc | ((unsigned)nfc << 4) | ((unsigned)pairs << 8) | (ok ? kCiValid : 0u) | (left << 16);
}

// lagrange_main.F90:110: new_sol = sol + dt*rhs, and the cell's pressure record
__device__ inline void state_update(const DevMesh& m, double* sol6, const double* rhs6, const double dt,
                                    const int c) {
  double* u = sol6 + kRec * (size_t)c;
  const double* r = rhs6 + kRhs * (size_t)c;
  bool fin = true;
  for (int k = 0; k < 5; ++k) {
    u[k] = u[k] + dt * r[k];
    fin = fin && isfinite(u[k]);
  }
  u[6] = lag_pressure(u[0], u[1], u[2], u[3], u[4]);
  if (!fin) atomicOr(m.status, kErrNonFinite);
  if (!(u[0] > 0.0)) atomicOr(m.status, kErrNegDensity);
}

// A tile of 32 cells per block, lane = cell, the cells' vertices, faces and (face, vertex)
// pairs spread over the warps, with the sums between them in the reference's order:
//   vertices and faces to shared memory, the faces' check_mesh terms; the vertex mean;
//   the centroid's tetrahedra, one per pair, summed by a warp per component;
//   the subcells' tetrahedra, two per (vertex, subface) pair, summed per subcell;
//   the cell's volume and tests, and the state's update.
// What bounds it: latency, of the loads (43% of a warp's cycles at 3,034 prisms) and of the
// barriers between the phases (21%); issue is at 11%, the FP64 pipe at 7%. One thread per cell
// ran the 5,500 instructions of a prism as one chain (3,000 prisms 20 us, here 12.5).
// Above kTileCells cells (of a mesh, or of a batch's table) one thread per cell is as fast
// or faster (both cell kernels together: tiles 38.7 us at 16,200 prisms, 43.4 at 21,632,
// 45.3 at 27,848; a thread per cell 44.6 at 28,322, 46.6 at 33,800, and its time hardly
// falls on smaller meshes).
constexpr int kTileCells = 28000;
constexpr int kGeoWarps = 12, kGeoThreads = 32 * kGeoWarps;
// two pairs a warp; at least the warps that share the vertices and the summed components
__host__ __device__ inline int geo_warps(int pairs) { return pairs <= 12 ? 6 : pairs <= 18 ? 9 : kGeoWarps; }

struct GeoTile {
  double X[kGeoMaxV][3][32];        // vertex coordinates
  double CF[kGeoCellFaces][3][32];  // face centroids
  double chk[kGeoCellFaces][7][32];  // cf.an, an, S signed, per face
  double term[4][kGeoPairs][32];
  double ce[3][32], cen[3][32];     // vertex mean, centroid
  double vol[kGeoMaxV][32];         // subcell volumes
};

__device__ inline V3 ldX(const double (&a)[3][32], int lane) { return {a[0][lane], a[1][lane], a[2][lane]}; }

// every thread of the block calls; dt: the step's time step for the update (with sol6)
__device__ inline void geom_step_tile(const DevMesh& m, double* sol6, const double* rhs6, const double dt,
                                      const int tile, GeoTile& s) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, W = blockDim.x >> 5;
  const int c = 32 * tile + lane;
  const unsigned info = c < m.ne ? m.cinfo[c] : 0u;
  const bool valid = (info & kCiValid) != 0u;
  const int nvc = valid ? info & 15 : 0, nfc = valid ? (info >> 4) & 15 : 0, np = valid ? (info >> 8) & 31 : 0;
  const int vb = valid ? m.ev_off[c] : 0;
  if (w == 0 && c < m.ne && !valid) atomicOr(m.status, kErrIndex);
  for (int t = w; t < kGeoMaxV + kGeoCellFaces; t += W) {
    if (t < kGeoMaxV) {
      if (t < nvc) {
        const V3 x = ld3(m.x, m.ev[vb + t]);
        s.X[t][0][lane] = x.x;
        s.X[t][1][lane] = x.y;
        s.X[t][2][lane] = x.z;
      }
    } else if (t - kGeoMaxV < nfc) {
      const int j = t - kGeoMaxV, f = m.ef8[8 * (size_t)c + j];
      const V3 cf = ld3(m.fc, f);
      const double4 fn = m.fn[f], S = m.fS[f];
      s.CF[j][0][lane] = cf.x;
      s.CF[j][1][lane] = cf.y;
      s.CF[j][2][lane] = cf.z;
      // check_mesh_elem_volume / _closed / _subface_closed terms of this face (the subface
      // closure sums the face's own subface sum S, formed in face%sub_face order)
      const double sg = (info >> (16 + j)) & 1u ? 1.0 : -1.0;
      const V3 nn = {sg * fn.x, sg * fn.y, sg * fn.z};
      const V3 an = {fn.w * nn.x, fn.w * nn.y, fn.w * nn.z};
      s.chk[j][0][lane] = dot(cf, an);
      s.chk[j][1][lane] = an.x;
      s.chk[j][2][lane] = an.y;
      s.chk[j][3][lane] = an.z;
      s.chk[j][4][lane] = sg * S.x;
      s.chk[j][5][lane] = sg * S.y;
      s.chk[j][6][lane] = sg * S.z;
    }
  }
  __syncthreads();
  if (w < 3) {
    double e = 0.0;
    for (int k = 0; k < nvc; ++k) e = e + s.X[k][w][lane];
    s.ce[w][lane] = vertex_mean({e, e, e}, nvc).x;
  }
  __syncthreads();
  // compute_elem_centroid: tetrahedra (edge, face centroid, vertex mean)
  unsigned code[(kGeoPairs + 5) / 6];  // this thread's pairs, for both passes
  int n = 0;
  {
    const V3 ce = ldX(s.ce, lane);
#pragma unroll
    for (int i = 0; i < (kGeoPairs + 5) / 6; ++i) {
      const int q = w + i * W;
      if (q >= np) break;
      code[i] = m.gpair[tile_entry(c, m.max_pairs, q)];
      n = i + 1;
      const unsigned g = code[i];
      const V3 cp = ldX(s.X[g & 7], lane), cpp = ldX(s.X[(g >> 3) & 7], lane), cf = ldX(s.CF[(g >> 6) & 7], lane);
      const bool left = (g >> 9) & 1u;
      const V3 fe = sub(cf, ce), a = sub(cp, cf), b = sub(cpp, cf);
      const V3 x = cross(left ? a : b, left ? b : a);
      const double vol = div6(dot(x, fe));
      s.term[0][q][lane] = vol * (cp.x + cpp.x + cf.x + ce.x) * 0.25;
      s.term[1][q][lane] = vol * (cp.y + cpp.y + cf.y + ce.y) * 0.25;
      s.term[2][q][lane] = vol * (cp.z + cpp.z + cf.z + ce.z) * 0.25;
      s.term[3][q][lane] = vol;
    }
  }
  __syncthreads();
  if (w < 3 && valid) {
    double e = 0.0, v = 0.0;
    for (int q = 0; q < np; ++q) {
      e = e + s.term[w][q][lane];
      v = v + s.term[3][q][lane];
    }
    s.cen[w][lane] = qdiv(e, v);
  }
  __syncthreads();
  // compute_subelem_volume: subcell k is (cell, vertex k); its subfaces in sub_elem order
  {
    const V3 cen = ldX(s.cen, lane);
#pragma unroll
    for (int i = 0; i < (kGeoPairs + 5) / 6; ++i) {
      if (i >= n) break;
      const unsigned g = code[i] >> 16;
      const V3 cp = ldX(s.X[g & 7], lane), cf = ldX(s.CF[(g >> 9) & 7], lane);
      const V3 cpm = half_sum(ldX(s.X[(g >> 3) & 7], lane), cp), cpp = half_sum(ldX(s.X[(g >> 6) & 7], lane), cp);
      const bool left = (g >> 12) & 1u;
      const V3 fe = sub(cf, cen), a = sub(cpm, cf), b = sub(cp, cf), d = sub(cpp, cf);
      const V3 x1 = cross(left ? a : d, b), x2 = cross(b, left ? d : a);
      s.term[0][w + i * W][lane] = div6(dot(x1, fe));
      s.term[1][w + i * W][lane] = div6(dot(x2, fe));
    }
  }
  __syncthreads();
  for (int k = w; k < kGeoMaxV; k += W)
    if (k < nvc) {
      const unsigned g = m.gsub[vb + k];
      const int first = g & 255, end = first + (int)(g >> 8);
      double vol = 0.0;
      for (int q = first; q < end; ++q) vol = vol + s.term[0][q][lane] + s.term[1][q][lane];
      m.vol_se[vb + k] = vol;
      s.vol[k][lane] = vol;
    }
  __syncthreads();
  if (!valid) return;
  if (w == 0) {
    bool ok = true;
    double vcell = 0.0;
    for (int k = 0; k < nvc; ++k) {
      const double v = s.vol[k][lane];
      ok = ok && (v > 0.0);
      vcell = vcell + v;
    }
    m.vol[c] = vcell;
    double t[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (int j = 0; j < nfc; ++j)
      for (int i = 0; i < 7; ++i) t[i] = t[i] + s.chk[j][i][lane];
    ok = ok && (fabs(vcell - div3(t[0])) < 1e-14);
    ok = ok && norm2_below_1em14(t[1], t[2], t[3]);
    ok = ok && norm2_below_1em14(t[4], t[5], t[6]);
    if (!ok) atomicOr(m.status, kErrMeshCheck);
  } else if (w == 1 && sol6) {
    state_update(m, sol6, rhs6, dt, c);
  }
}

// The same, one cell per thread, for meshes that fill the GPU this way: the cell's vertex
// coordinates and face centroids in shared memory (one column per thread), its sums in
// registers. Every thread of a warp may call on its own.
constexpr int kGeoBlock = 64;
__device__ inline void geom_step_body(const DevMesh& m, double* sol6, const double* rhs6, const double dt,
                                      const int c) {
  __shared__ double sX[kGeoMaxV][3][kGeoBlock];
  __shared__ double sCF[kGeoCellFaces][3][kGeoBlock];
  const int t = threadIdx.x;
  if (c >= m.ne) return;
  const unsigned info = m.cinfo[c];
  if (!(info & kCiValid)) {
    atomicOr(m.status, kErrIndex);
    return;
  }
  const int nvc = info & 15, nfc = (info >> 4) & 15, np = (info >> 8) & 31;
  const int vb = m.ev_off[c];
  const uint32_t* pair = m.gpair + tile_entry(c, m.max_pairs, 0);  // pair q at pair[32 q]
  const int4 e0 = reinterpret_cast<const int4*>(m.ef8)[2 * (size_t)c];
  const int4 e1 = reinterpret_cast<const int4*>(m.ef8)[2 * (size_t)c + 1];
  const int fid[kGeoCellFaces] = {e0.x, e0.y, e0.z, e0.w, e1.x, e1.y};
  V3 ce = {0.0, 0.0, 0.0};
  for (int k = 0; k < nvc; ++k) {
    const V3 x = ld3(m.x, m.ev[vb + k]);
    sX[k][0][t] = x.x;
    sX[k][1][t] = x.y;
    sX[k][2][t] = x.z;
    ce = {ce.x + x.x, ce.y + x.y, ce.z + x.z};
  }
  double vdiv = 0.0;
  V3 nt = {0.0, 0.0, 0.0}, ns = {0.0, 0.0, 0.0};
#pragma unroll
  for (int j = 0; j < kGeoCellFaces; ++j)
    if (j < nfc) {
      const int f = fid[j];
      const V3 cf = ld3(m.fc, f);
      const double4 fn = m.fn[f];
      const double4 S = m.fS[f];
      sCF[j][0][t] = cf.x;
      sCF[j][1][t] = cf.y;
      sCF[j][2][t] = cf.z;
      const double sg = (info >> (16 + j)) & 1u ? 1.0 : -1.0;  // check_mesh's terms, as in the tile
      const V3 nn = {sg * fn.x, sg * fn.y, sg * fn.z};
      const V3 an = {fn.w * nn.x, fn.w * nn.y, fn.w * nn.z};
      vdiv = vdiv + dot(cf, an);
      nt = {nt.x + an.x, nt.y + an.y, nt.z + an.z};
      ns = {ns.x + sg * S.x, ns.y + sg * S.y, ns.z + sg * S.z};
    }
  ce = vertex_mean(ce, nvc);
  auto X = [&](unsigned q) { return V3{sX[q & 7][0][t], sX[q & 7][1][t], sX[q & 7][2][t]}; };
  auto CF = [&](unsigned j) { return V3{sCF[j & 7][0][t], sCF[j & 7][1][t], sCF[j & 7][2][t]}; };
  // compute_elem_centroid: tetrahedra (edge, face centroid, vertex mean)
  // the pairs' codes six at a time, the next six in flight
  constexpr int kAhead = 6;
  unsigned g6[kAhead], n6[kAhead];
  auto load = [&](unsigned (&g)[kAhead], int q0) {
#pragma unroll
    for (int i = 0; i < kAhead; ++i)
      if (q0 + i < np) g[i] = pair[32 * (q0 + i)];
  };
  V3 cen = {0.0, 0.0, 0.0};
  double sum_vol = 0.0;
  load(g6, 0);
  for (int q0 = 0; q0 < np; q0 += kAhead) {
    load(n6, q0 + kAhead < np ? q0 + kAhead : 0);  // after the last six the second pass's first
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      if (q0 + i >= np) break;
      const unsigned g = g6[i];
      const V3 cp = X(g), cpp = X(g >> 3), cf = CF(g >> 6);
      const bool left = (g >> 9) & 1u;
      const V3 fe = sub(cf, ce), a = sub(cp, cf), b = sub(cpp, cf);
      const V3 x = cross(left ? a : b, left ? b : a);
      const double vol = div6(dot(x, fe));
      cen.x = cen.x + vol * (cp.x + cpp.x + cf.x + ce.x) * 0.25;
      cen.y = cen.y + vol * (cp.y + cpp.y + cf.y + ce.y) * 0.25;
      cen.z = cen.z + vol * (cp.z + cpp.z + cf.z + ce.z) * 0.25;
      sum_vol = sum_vol + vol;
    }
#pragma unroll
    for (int i = 0; i < kAhead; ++i) g6[i] = n6[i];
  }
  cen = {qdiv(cen.x, sum_vol), qdiv(cen.y, sum_vol), qdiv(cen.z, sum_vol)};
  // compute_subelem_volume: subcell k is (cell, vertex k); its subfaces in sub_elem order
  bool ok = true;
  double vcell = 0.0, vol = 0.0;
  int k = 0;
  for (int q0 = 0; q0 < np; q0 += kAhead) {
    load(n6, q0 + kAhead);
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      if (q0 + i >= np) break;
      const unsigned g = g6[i] >> 16;
      const V3 cp = X(g), cf = CF(g >> 9);
      const V3 cpm = half_sum(X(g >> 3), cp), cpp = half_sum(X(g >> 6), cp);
      const bool left = (g >> 12) & 1u;
      const V3 fe = sub(cf, cen), a = sub(cpm, cf), b = sub(cp, cf), d = sub(cpp, cf);
      const V3 x1 = cross(left ? a : d, b), x2 = cross(b, left ? d : a);
      vol = vol + div6(dot(x1, fe)) + div6(dot(x2, fe));
      if ((g >> 13) & 1u) {  // the subcell's last pair
        m.vol_se[vb + k] = vol;
        ok = ok && (vol > 0.0);
        vcell = vcell + vol;
        vol = 0.0;
        ++k;
      }
    }
#pragma unroll
    for (int i = 0; i < kAhead; ++i) g6[i] = n6[i];
  }
  m.vol[c] = vcell;
  ok = ok && (fabs(vcell - div3(vdiv)) < 1e-14);
  ok = ok && norm2_below_1em14(nt.x, nt.y, nt.z);
  ok = ok && norm2_below_1em14(ns.x, ns.y, ns.z);
  if (!ok) atomicOr(m.status, kErrMeshCheck);
  if (sol6) state_update(m, sol6, rhs6, dt, c);
}

}  // namespace geo
}  // namespace subfv
