// mc_cell.cuh -- the per-cell marching-cubes construction (cut cells), shared by the update
// kernels and the learned-correction kernels.
//
// cut_cell_moments for a cut cell (src/marching_cubes/moments.jl:275-346): the six face clips
// (cut_cell_faces / _cut_cell_face, :150-257, with the walk of
// src/marching_squares/marching_squares.jl:240-251), the Lewiner dispatch over a tiling table
// (src/marching_cubes/marching_cubes.jl:538-651, deciders :401-504), the edge crossings
// (:306-330) and the divergence-theorem sums.
#pragma once
#include <cstdint>
#include <type_traits>
#include "cc_device.cuh"
#include "cc_internal.h"

namespace ccmc {

using namespace ccd;
using cci::DevTable;

// MC_NODE_BITS (src/marching_cubes/marching_cubes.jl:106-107), bit of corner c along axis a.
__host__ __device__ constexpr int cbit(int c, int a) {
  return a == 0 ? ((c ^ (c >> 1)) & 1) : (a == 1 ? ((c >> 1) & 1) : ((c >> 2) & 1));
}
// MC_FACE_NODES (:169-180), 0-based directions and corners.
__host__ __device__ constexpr int face_node(int dir, int k) {
  constexpr int t[6][4] = {{0, 3, 7, 4}, {1, 2, 6, 5}, {0, 1, 5, 4}, {3, 2, 6, 7}, {0, 1, 2, 3}, {4, 5, 6, 7}};
  return t[dir][k];
}
// MC_FACE_TEST_CODE (:385-388)
__host__ __device__ constexpr int face_test_code(int dir) {
  constexpr int t[6] = {4, 2, 1, 3, 5, 6};
  return t[dir];
}
// MC_EDGE_NODES (:135-137), 0-based corners.
__host__ __device__ constexpr int edge_node(int e, int s) {
  constexpr int t[12][2] = {{0, 1}, {1, 2}, {3, 2}, {0, 3}, {4, 5}, {5, 6}, {7, 6}, {4, 7}, {0, 4}, {1, 5}, {2, 6}, {3, 7}};
  return t[e][s];
}

// MC_TEST_FACE_QUADS (:372-373) and the twelve reference-edge branches of _test_interior
// (:450-486), 0-based corners, for indices only known at run time.
static __constant__ uint8_t c_quads[6][4] = {{0, 4, 5, 1}, {1, 5, 6, 2}, {2, 6, 7, 3}, {3, 7, 4, 0}, {0, 3, 2, 1}, {4, 7, 6, 5}};
static __constant__ uint8_t c_iedge[12][8] = {
    {0, 1, 3, 2, 7, 6, 4, 5}, {1, 2, 0, 3, 4, 7, 5, 6}, {2, 3, 1, 0, 5, 4, 6, 7}, {3, 0, 2, 1, 6, 5, 7, 4},
    {4, 5, 7, 6, 3, 2, 0, 1}, {5, 6, 4, 7, 0, 3, 1, 2}, {6, 7, 5, 4, 1, 0, 2, 3}, {7, 4, 6, 5, 2, 1, 3, 0},
    {0, 4, 3, 7, 2, 6, 1, 5}, {1, 5, 0, 4, 3, 7, 2, 6}, {2, 6, 1, 5, 0, 4, 3, 7}, {3, 7, 2, 6, 1, 5, 0, 4}};

template <class T>
__device__ __forceinline__ T nudge(T v) {
  const T e = Eps<T>::v();
  return fabs(v) < e ? e : v;
}

// _test_face, src/marching_cubes/marching_cubes.jl:401-406. With MX the determinant and the
// final product are evaluated in FP64 (R) from the FP32 corner values; the threshold stays eps(T).
template <class T, bool MX = false>
__device__ __forceinline__ bool test_face(const T* cb, int face) {
  using R = typename std::conditional<MX, double, T>::type;
  const int f = (face < 0 ? -face : face) - 1;
  const R A = cb[c_quads[f][0]], B = cb[c_quads[f][1]], C = cb[c_quads[f][2]], D = cb[c_quads[f][3]];
  const R det = A * C - B * D;
  if (fabs(det) < R(Eps<T>::v())) return face >= 0;
  return (R(face) * A) * det >= R(0);
}
// _test_interior, :427-504. With MX every step runs in FP64 (R) from the FP32 corner values; the
// thresholds stay eps(T).
template <class T, bool MX = false>
__device__ bool test_interior(int itype, int edge, const T* cbt, int s) {
  using R = typename std::conditional<MX, double, T>::type;
  R cb[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) cb[k] = cbt[k];
  R At = R(0), Bt = R(0), Ct = R(0), Dt = R(0);
  if (itype == CC_MC_INTERIOR_CASE4_10) {
    const R a = (cb[4] - cb[0]) * (cb[6] - cb[2]) - (cb[7] - cb[3]) * (cb[5] - cb[1]);
    const R b = ((cb[2] * (cb[4] - cb[0]) + cb[0] * (cb[6] - cb[2])) - cb[1] * (cb[7] - cb[3])) - cb[3] * (cb[5] - cb[1]);
    const R t = -b / (R(2) * a);
    if (t < R(0) || t > R(1)) return s > 0;
    At = cb[0] + (cb[4] - cb[0]) * t;
    Bt = cb[3] + (cb[7] - cb[3]) * t;
    Ct = cb[2] + (cb[6] - cb[2]) * t;
    Dt = cb[1] + (cb[5] - cb[1]) * t;
  } else {
    const uint8_t* e = c_iedge[edge];
    const R t = cb[e[0]] / (cb[e[0]] - cb[e[1]]);
    Bt = cb[e[2]] + (cb[e[3]] - cb[e[2]]) * t;
    Ct = cb[e[4]] + (cb[e[5]] - cb[e[4]]) * t;
    Dt = cb[e[6]] + (cb[e[7]] - cb[e[6]]) * t;
  }
  int test = 0;
  if (At >= R(0)) test += 1;
  if (Bt >= R(0)) test += 2;
  if (Ct >= R(0)) test += 4;
  if (Dt >= R(0)) test += 8;
  const R eps = R(Eps<T>::v());
  if (test == 6 || test == 8 || test == 9 || test == 12 || (test >= 0 && test <= 4)) return s > 0;
  if (test == 5) return (At * Ct - Bt * Dt < eps) ? s > 0 : s < 0;
  if (test == 10) return (At * Ct - Bt * Dt >= eps) ? s > 0 : s < 0;
  return s < 0;
}

// The cube edge (MC_EDGE_NODES) between two corners.
__host__ __device__ constexpr int edge_between(int a, int b) {
  for (int e = 0; e < 12; ++e)
    if ((edge_node(e, 0) == a && edge_node(e, 1) == b) || (edge_node(e, 0) == b && edge_node(e, 1) == a)) return e;
  return -1;
}
__host__ __device__ constexpr int edge_axis(int e) { return e >= 8 ? 2 : (e & 1); }
// Of a face's corner mask (bit k: corner k open), the first edge leaving the open part (corner k open,
// k + 1 not) and the one entering it (k not, k + 1 open), two bits per mask.
__host__ __device__ constexpr unsigned face_edges(bool leaving) {
  unsigned t = 0;
  for (unsigned m = 0; m < 16; ++m)
    for (int k = 3; k >= 0; --k) {
      const bool o = (m >> k) & 1, n = (m >> ((k + 1) & 3)) & 1;
      if (leaving ? (o && !n) : (!o && n)) t = (t & ~(3u << (2 * m))) | (unsigned(k) << (2 * m));
    }
  return t;
}

// The open part of a cut cube face in its own (p, q) frame, corners (0,0), (lp,0), (lp,lq), (0,lq) and
// corner mask m (bits open): cell_boundary_walk (src/marching_squares/marching_squares.jl:240-251) then
// _face_polygon (src/marching_cubes/moments.jl:111-139) with _chord_target (:91-98), from the cube edges'
// crossings x[k] (the coordinate that varies along edge k). Twice its area and three times its first
// moments, in the reference's order: the boundary segments of edges 0..3 (those of edges 0 and 3 lie
// on the axes through the frame's origin and add exact zeros), then a chord per crossing out of the open
// part. `connect`: the decider of a face with opposite corners open.
template <class T, class Connect>
__device__ __forceinline__ void face_polygon(unsigned m, T lp, T lq, const T x[4], Connect&& connect, T& area2, T& m0,
                                             T& m1) {
  const bool o1 = m & 2, o2 = m & 4, o3 = m & 8;
  area2 = T(0); m0 = T(0); m1 = T(0);
  if (o1 || o2) {
    const T a = o1 ? T(0) : x[1], b = o2 ? lq : x[1];
    const T cr = lp * b - a * lp;
    area2 = area2 + cr;
    m0 = m0 + (lp + lp) * cr;
    m1 = m1 + (a + b) * cr;
  }
  if (o2 || o3) {
    const T a = o2 ? lp : x[2], b = o3 ? T(0) : x[2];
    const T cr = a * lq - lq * b;
    area2 = area2 + cr;
    m0 = m0 + (a + b) * cr;
    m1 = m1 + (lq + lq) * cr;
  }
  auto chord = [&](unsigned k, unsigned j) {
    const T k0 = (k & 1) ? ((k & 2) ? T(0) : lp) : ((k & 2) ? x[2] : x[0]);
    const T k1 = (k & 1) ? ((k & 2) ? x[3] : x[1]) : ((k & 2) ? lq : T(0));
    const T j0 = (j & 1) ? ((j & 2) ? T(0) : lp) : ((j & 2) ? x[2] : x[0]);
    const T j1 = (j & 1) ? ((j & 2) ? x[3] : x[1]) : ((j & 2) ? lq : T(0));
    const T cr = k0 * j1 - k1 * j0;
    area2 = area2 + cr;
    m0 = m0 + (k0 + j0) * cr;
    m1 = m1 + (k1 + j1) * cr;
  };
  constexpr unsigned LEAVING = face_edges(true), ENTERING = face_edges(false);
  const unsigned k = (LEAVING >> (2 * m)) & 3u;
  if (m == 5u || m == 10u) {
    const unsigned j = connect() ? k + 1 : (k + 3) & 3u;
    chord(k, j);
    chord(k + 2, j ^ 2u);
  } else {
    chord(k, (ENTERING >> (2 * m)) & 3u);
  }
}

// x / 3 and x / 6 for x >= 0, correctly rounded without a division: q = x RN(1/D), then one step q + (x -
// D q) RN(1/D) whose residual is exact in an FMA. x / D lies at least ulp / 12 from any rounding boundary
// (a boundary times D has more significant bits than x), far beyond the step's error of 2^-48 (2^-106)
// relative. Below 2^-96 (2^-900) the residual could underflow, and x divides.
template <class T, int D>
__device__ __forceinline__ T div_const(T x) {
  constexpr T R = T(1) / T(D);
  if (!(x > (sizeof(T) == 4 ? T(0x1p-96) : T(0x1p-900)) || x == T(0))) return x / T(D);
  const T q = x * R;
  if constexpr (sizeof(T) == 4) return __fmaf_rn(__fmaf_rn(-float(D), q, x), R, q);
  else return __fma_rn(__fma_rn(-double(D), q, x), R, q);
}

// Shared-memory staging of one tile's output columns.
template <class T>
struct Stage {
  int8_t* kind;
  uint8_t* amb;
  T* vf;
  T* c;
  T* ff;
  T* fcl;
  T* ic;
};

template <class T>
__device__ __forceinline__ void put_vec(T* dst, const T* v, int n);

template <>
__device__ __forceinline__ void put_vec<float>(float* dst, const float* v, int n) {
  // n is 6 or 12 with dst 8- or 16-byte aligned respectively
  if (n == 12) {
    float4* d4 = reinterpret_cast<float4*>(dst);
    d4[0] = make_float4(v[0], v[1], v[2], v[3]);
    d4[1] = make_float4(v[4], v[5], v[6], v[7]);
    d4[2] = make_float4(v[8], v[9], v[10], v[11]);
  } else {
    float2* d2 = reinterpret_cast<float2*>(dst);
    d2[0] = make_float2(v[0], v[1]);
    d2[1] = make_float2(v[2], v[3]);
    d2[2] = make_float2(v[4], v[5]);
  }
}
template <>
__device__ __forceinline__ void put_vec<double>(double* dst, const double* v, int n) {
  double2* d2 = reinterpret_cast<double2*>(dst);
  for (int i = 0; i < n / 2; ++i) d2[i] = make_double2(v[2 * i], v[2 * i + 1]);
}

template <class T>
__device__ __forceinline__ void put_cell(const Stage<T>& st, long long lc, int kind, int amb, T vf, const T c[3],
                                         const T ff[6], const T fcl[12], const T ic[3]) {
  st.kind[lc] = int8_t(kind);
  st.amb[lc] = uint8_t(amb);
  st.vf[lc] = vf;
  st.c[3 * lc] = c[0]; st.c[3 * lc + 1] = c[1]; st.c[3 * lc + 2] = c[2];
  // wide stores where the columns allow them; a caller's need only their element's alignment
  if (((reinterpret_cast<uintptr_t>(st.ff) & (2 * sizeof(T) - 1)) | (reinterpret_cast<uintptr_t>(st.fcl) & 15u)) == 0) {
    put_vec<T>(st.ff + 6 * lc, ff, 6);
    put_vec<T>(st.fcl + 12 * lc, fcl, 12);
  } else {
#pragma unroll
    for (int i = 0; i < 6; ++i) st.ff[6 * lc + i] = ff[i];
#pragma unroll
    for (int i = 0; i < 12; ++i) st.fcl[12 * lc + i] = fcl[i];
  }
  st.ic[3 * lc] = ic[0]; st.ic[3 * lc + 1] = ic[1]; st.ic[3 * lc + 2] = ic[2];
}

// cell_triangles over the table (src/marching_cubes/marching_cubes.jl:538-651): the tile of a cube
// with nudged corner values `phi` (MC_NODE_BITS order).
template <class T, bool MX = false>
__device__ __forceinline__ int mc_tile(const T phi[8], const DevTable& tb) {
  int lut = 0;
#pragma unroll
  for (int p = 0; p < 8; ++p) lut |= (phi[p] >= T(0) ? 1 : 0) << p;
  const cc_mc_lut ent = tb.luts[lut];
  int o = 0;
  for (int i = 0; i < ent.ntests; ++i) o |= (test_face<T, MX>(phi, ent.face[i]) ? 1 : 0) << i;
  const cc_mc_outcome oc = tb.outs[ent.outcome_base + o];
  int tile = oc.tile_true;
  if (oc.itype != CC_MC_INTERIOR_NONE && !test_interior<T, MX>(oc.itype, oc.edge, phi, oc.s)) tile = oc.tile_false;
  return tile;
}

// cut_cell_moments (3D) for a cut cell, src/marching_cubes/moments.jl:275-346. `phr` are the
// raw corner values in MC_NODE_BITS order, `l` the cell's lattice edge lengths
// (x_{i+1} - x_i per axis: every corner's cell-local coordinate is 0 or l exactly), `org` the
// lower corner and `cs` the grid's cell size.
//
// A crossing belongs to two faces and to the triangles: it is formed once, one division per cut
// edge, and the faces take their segments and chords from the coordinate that varies along it.
// (Each face formed its own crossings and searched its chords over all four edges: 5300 warp instructions
// for 32 cells. Bound by latency and issue. The cut kernel at 512^3 Float32 137 -> 80 us, at 64^3 23 -> 10,
// at 256^3 Float64 75 -> 40; a wave field at 192 x 160 x 129, Float64, 244 -> 136.)
template <class T, bool MX = false>
__device__ __forceinline__ void mc_cut_cell(const T phr[8], const T l[3], const T org[3], const T cs[3],
                                            const DevTable& tb, const Stage<T>& st, long long lc) {
  T phi[8];
  unsigned lut = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    phi[k] = nudge(phr[k]);
    lut |= phi[k] >= T(0) ? 1u << k : 0u;
  }
  T centre[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) centre[a] = org[a] + T(0.5) * cs[a];
  const T vol_cell = (cs[0] * cs[1]) * cs[2];

  const cc_mc_tile tl = tb.tiles[mc_tile<T, MX>(phi, tb)];

  // edge_crossings (marching_cubes.jl:306-330)
  T pts[13][3], xc[12];
#pragma unroll
  for (int e = 0; e < 12; ++e) {
    const int a = edge_node(e, 0), b = edge_node(e, 1), ax = edge_axis(e);
    xc[e] = T(0);
    pts[e][0] = T(0); pts[e][1] = T(0); pts[e][2] = T(0);
    if (((lut >> a) ^ (lut >> b)) & 1u) {
      const T s = open_fraction<T, MX>(phi[a], phi[b]);
      // a is the edge's end at 0, b the one at l
      xc[e] = (lut >> a) & 1u ? T(0) + s * l[ax] : l[ax] + s * (T(0) - l[ax]);
      const T z = s * T(0);  // the other two coordinates: the corner's plus this (a NaN value spreads)
#pragma unroll
      for (int x = 0; x < 3; ++x) pts[e][x] = x == ax ? xc[e] : (cbit(a, x) ? l[x] : T(0)) + z;
    }
  }

  // the six face clips (cut_cell_faces / _cut_cell_face, moments.jl:150-257)
  T ff[6], fcl[12];
  bool amb_face = false;
#pragma unroll
  for (int dir = 0; dir < 6; ++dir) {
    const int ax = dir >> 1;
    const int p = ax == 0 ? 1 : 0;
    const int q = ax == 2 ? 1 : 2;
    unsigned m = 0;
    T x[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      m |= ((lut >> face_node(dir, k)) & 1u) << k;
      x[k] = xc[edge_between(face_node(dir, k), face_node(dir, (k + 1) & 3))];
    }
    amb_face = amb_face || m == 5u || m == 10u;
    const T avg0 = T(0.25) * (l[p] + l[p]);
    const T avg1 = T(0.25) * (l[q] + l[q]);
    T frac, c0, c1;
    if (m == 15u || m == 0u) {
      frac = m == 15u ? T(1) : T(0);
      c0 = avg0; c1 = avg1;
    } else {
      T area2, m0, m1;
      face_polygon<T>(m, l[p], l[q], x, [&]() { return test_face<T, MX>(phi, face_test_code(dir)); }, area2, m0, m1);
      const T full = (T(1) * cs[p]) * cs[q];
      frac = (T(0.5) * area2) / full;
      if (area2 != T(0)) { const T den = T(3) * area2; c0 = m0 / den; c1 = m1 / den; }
      else { c0 = avg0; c1 = avg1; }
    }
    ff[dir] = frac;
    fcl[2 * dir] = c0;
    fcl[2 * dir + 1] = c1;
  }

  // divergence theorem over the closed polyhedron (moments.jl:304-336)
  T vol3 = T(0);
  T cm0 = T(0), cm1 = T(0), cm2 = T(0);
#pragma unroll
  for (int dir = 0; dir < 6; ++dir) {
    const int ax = dir >> 1;
    const int p = ax == 0 ? 1 : 0;
    const int q = ax == 2 ? 1 : 2;
    const T s = (dir & 1) ? T(1) : T(-1);
    const T x_ax = (dir & 1) ? l[ax] : T(0);
    const T a_open = ff[dir] * ((T(1) * cs[p]) * cs[q]);
    vol3 = vol3 + (s * x_ax) * a_open;
    const T m = ((s * x_ax) * x_ax) * a_open;
    cm0 = cm0 + (ax == 0 ? m : T(0));
    cm1 = cm1 + (ax == 1 ? m : T(0));
    cm2 = cm2 + (ax == 2 ? m : T(0));
  }
  T iarea = T(0), ic0 = T(0), ic1 = T(0), ic2 = T(0);
  const uint8_t* codes = tb.codes + tl.code_off;
  bool have_centre = false;
  for (int t = 0; t < tl.ntris; ++t) {
    const int ca = codes[3 * t] - 1, cb = codes[3 * t + 1] - 1, cd = codes[3 * t + 2] - 1;
    if (!have_centre && (ca == 12 || cb == 12 || cd == 12)) {  // the crossings' mean, where a tile uses it
      T acc0 = T(0), acc1 = T(0), acc2 = T(0);
      int ncr = 0;
#pragma unroll
      for (int e = 0; e < 12; ++e)
        if (((lut >> edge_node(e, 0)) ^ (lut >> edge_node(e, 1))) & 1u) {
          acc0 = acc0 + pts[e][0]; acc1 = acc1 + pts[e][1]; acc2 = acc2 + pts[e][2];
          ++ncr;
        }
      pts[12][0] = ncr > 0 ? acc0 / T(ncr) : T(0);
      pts[12][1] = ncr > 0 ? acc1 / T(ncr) : T(0);
      pts[12][2] = ncr > 0 ? acc2 / T(ncr) : T(0);
      have_centre = true;
    }
    const T A0 = pts[ca][0], A1 = pts[ca][1], A2 = pts[ca][2];
    const T B0 = pts[cb][0], B1 = pts[cb][1], B2 = pts[cb][2];
    const T D0 = pts[cd][0], D1 = pts[cd][1], D2 = pts[cd][2];
    const T u0 = B0 - A0, u1 = B1 - A1, u2 = B2 - A2;
    const T v0 = D0 - A0, v1 = D1 - A1, v2 = D2 - A2;
    const T w0 = T(0.5) * (u1 * v2 - u2 * v1);
    const T w1 = T(0.5) * (u2 * v0 - u0 * v2);
    const T w2 = T(0.5) * (u0 * v1 - u1 * v0);
    const T x0 = div_const<T, 3>((A0 + B0) + D0);
    const T x1 = div_const<T, 3>((A1 + B1) + D1);
    const T x2 = div_const<T, 3>((A2 + B2) + D2);
    vol3 = vol3 - ((w0 * x0 + w1 * x1) + w2 * x2);
    const T q0 = div_const<T, 6>(((((A0 * A0 + B0 * B0) + D0 * D0) + A0 * B0) + B0 * D0) + D0 * A0);
    const T q1 = div_const<T, 6>(((((A1 * A1 + B1 * B1) + D1 * D1) + A1 * B1) + B1 * D1) + D1 * A1);
    const T q2 = div_const<T, 6>(((((A2 * A2 + B2 * B2) + D2 * D2) + A2 * B2) + B2 * D2) + D2 * A2);
    cm0 = cm0 - w0 * q0;
    cm1 = cm1 - w1 * q1;
    cm2 = cm2 - w2 * q2;
    const T len = sqrt((w0 * w0 + w1 * w1) + w2 * w2);
    iarea = iarea + len;
    ic0 = ic0 + len * x0;
    ic1 = ic1 + len * x1;
    ic2 = ic2 + len * x2;
  }
  const T volume = vol3 / T(3);
  T c[3], ic[3];
  if (volume > T(0)) {
    const T den = T(2) * volume;
    c[0] = org[0] + cm0 / den; c[1] = org[1] + cm1 / den; c[2] = org[2] + cm2 / den;
  } else {
    c[0] = centre[0]; c[1] = centre[1]; c[2] = centre[2];
  }
  if (iarea > T(0)) {
    ic[0] = org[0] + ic0 / iarea; ic[1] = org[1] + ic1 / iarea; ic[2] = org[2] + ic2 / iarea;
  } else {
    ic[0] = centre[0]; ic[1] = centre[1]; ic[2] = centre[2];
  }
  const int lc_case = tb.luts[lut].lcase;
  const bool amb_case = lc_case == 5 || lc_case == 7 || lc_case == 8 || lc_case == 11 || lc_case == 13 || lc_case == 14;
  put_cell<T>(st, lc, 2, (amb_face || amb_case) ? 1 : 0, volume / vol_cell, c, ff, fcl, ic);
}

}  // namespace ccmc
