// plic.cu -- PLICCutCell update_cache!, calc_volume and cut_cell_report on sm_100a.
//
// Fit pass (_plic_fit_kernel!, src/plic/cache.jl:96-113): per cell one evaluation of the op-tape's
// value and gradient at the centroid gives (dist, normal) -- get_sdf -- and cell_plane
// (src/plic/plic.jl:72-88) turns it into the stored plane. Faces (_plic_face_fraction_kernel!,
// src/plic/cache.jl:118-162): per cell, per face, the mean of the two one-sided candidates of the two
// cells' planes by the same _face_area (src/plic/apertures.jl:112-125), so both cells of a face hold
// identical bits. In 3D the fit writes the one-sided fractions and a second pass resolves the faces
// whose two cells differ; in 2D a face pass computes both sides from the stored planes.
#include <cmath>
#include <cstdint>
#include <limits>
#include <type_traits>
#include "cc_device.cuh"
#include "cc_internal.h"

namespace {

using namespace ccd;
using cci::Cols;
using cci::DevGrid;
using cci::DevTape;
using cci::TapeBounds;

constexpr int NT = 256;
constexpr int VOL_BLOCKS = 148 * 8;

template <class T, int D>
struct PlaneFit {
  T n[D];
  T a;
  T fraction;
  bool valid;
};

// cell_plane, src/plic/plic.jl:72-88, in 2D (with MX the line-square clip runs in FP64)
template <class T, bool MX>
__device__ __forceinline__ PlaneFit<T, 2> cell_plane(const STape<T>& t, const DevGrid<T>& g, const long long idx[2]) {
  Dual<T, 2> x[2];
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    x[a].v = centroid_coord(g.x0[a], g.d[a], idx[a]);
#pragma unroll
    for (int b = 0; b < 2; ++b) x[a].g[b] = a == b ? T(1) : T(0);
  }
  const Dual<T, 2> r = tape_eval<T, 2, Dual<T, 2>>(t, x);
  const T a = T(0.5) * (r.g[0] + r.g[1]) - r.v / g.d[0];
  PlaneFit<T, 2> pl;
  pl.valid = !(isnan(a) || (r.g[0] == T(0) && r.g[1] == T(0)));
#pragma unroll
  for (int q = 0; q < 2; ++q) pl.n[q] = pl.valid ? r.g[q] : T(0);
  pl.a = pl.valid ? a : T(0);
  if (pl.valid) pl.fraction = gvf2m<T, MX>(r.g[0], r.g[1], a);
  else pl.fraction = r.v <= T(0) ? T(1) : T(0);
  return pl;
}

// The 2D kernels' tile: NT cells, 32 along x (coalesced stores); the tape is pruned to the box of a
// tile's centroids when the body is a union of spheres.
constexpr int PX = 32, PY = 8;
static_assert(PX * PY == NT, "one cell per thread");
static_assert(NT >= CC_TAPE_MAX_OPS, "prune_union: an op per thread");

// Tile t's first cell, tiles numbered x fastest, from 32-bit quotients (a grid has far fewer
// than 2^32 tiles: that would be 2^40 cells).
__device__ __forceinline__ void tile_origin(unsigned t, unsigned tx, long long i0[2]) {
  const unsigned a = t / tx;
  i0[0] = (long long)(t - a * tx) * PX;
  i0[1] = (long long)a * PY;
}

// Shared-memory layout of a centroid kernel: the tape, then the pruned ops and the bounds.
struct CentroidSmem {
  int ops_off, ls_off, us_off, bytes;
  __host__ __device__ static CentroidSmem of(const DevTape& tape) {
    CentroidSmem c;
    c.ops_off = ((tape.bytes_len + 15) / 16) * 16;
    c.ls_off = c.ops_off + ((tape.n_ops * int(sizeof(cc_op)) + 15) / 16) * 16;
    c.us_off = c.ls_off + tape.n_ops * 8;
    c.bytes = c.us_off + tape.n_ops * 8;
    return c;
  }
};

// The tape a tile's cells (first cell i0, clipped to the grid) are evaluated with: pruned to the box of
// their centroids if it can be.
template <class T>
__device__ __forceinline__ STape<T> tile_tape(const STape<T>& t, const DevTape& tape, const DevGrid<T>& g,
                                              const long long i0[2], unsigned char* smem, int* count) {
  if (!tape.prunable) return t;
  const CentroidSmem L = CentroidSmem::of(tape);
  const int ext[2] = {PX, PY};
  double lo[2], hi[2];
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    const long long last = i0[a] + ext[a] - 1 < g.n[a] - 1 ? i0[a] + ext[a] - 1 : g.n[a] - 1;
    lo[a] = double(g.x0[a]) + (double(i0[a]) + 0.5) * double(g.d[a]);
    hi[a] = double(g.x0[a]) + (double(last) + 0.5) * double(g.d[a]);
  }
  cc_op* ops = reinterpret_cast<cc_op*>(smem + L.ops_off);
  const int m = prune_union<T>(t, tape.prunable, lo, hi, reinterpret_cast<double*>(smem + L.ls_off),
                                  reinterpret_cast<double*>(smem + L.us_off), ops, count);
  STape<T> u = t;
  u.ops = ops;
  u.n_ops = m;
  return u;
}

template <class T, bool MX>
__global__ void __launch_bounds__(NT) plic_fit_kernel(const DevGrid<T> g, const DevTape tape, const Cols cols,
                                                      T* normals, T* intercepts, uint8_t* valid) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_count;
  const STape<T> t = load_tape<T>(tape.bytes, tape.n_ops, tape.n_params, smem);
  __syncthreads();
  const long long n0 = g.n[0], n1 = g.n[1];
  const long long tx = (n0 + PX - 1) / PX, ty = (n1 + PY - 1) / PY;
  T* vf = static_cast<T*>(cols.vf);
  const unsigned ntiles = unsigned(tx * ty);
  for (unsigned tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    long long i0[2];
    tile_origin(tile, unsigned(tx), i0);
    const STape<T> u = tile_tape<T>(t, tape, g, i0, smem, &s_count);
    const long long idx[2] = {i0[0] + threadIdx.x % PX, i0[1] + threadIdx.x / PX};
    if (idx[0] < n0 && idx[1] < n1) {
      const long long ci = idx[0] + n0 * idx[1];
      const PlaneFit<T, 2> pl = cell_plane<T, MX>(u, g, idx);
      const T frac = T(1) - pl.fraction;
      normals[2 * ci] = pl.n[0];
      normals[2 * ci + 1] = pl.n[1];
      intercepts[ci] = pl.a;
      valid[ci] = pl.valid ? 1 : 0;
      vf[ci] = frac;
      cols.kind[ci] = frac == T(0) ? 0 : (frac == T(1) ? 1 : 2);
    }
    __syncthreads();  // the next tile's pruning overwrites the ops this one read
  }
}

// _cell_wet + _face_area, src/plic/apertures.jl:73-125, in 2D (k is the 0-based direction)
template <class T, bool MX>
__device__ __forceinline__ T face_area(const T* n, T a, T frac, bool valid, const T* cs, int k) {
  const T s = (k & 1) ? T(1) : T(0);
  const int c = k >> 1, p = 1 - c;
  const T len = cs[p];
  if (!valid) return frac < T(0.5) ? T(0) : len;
  const T base = n[c] * s - a;
  return open_fraction<T, MX>(base, base + n[p]) * len;
}

// Whether a valid 3D plane misses its cell by more than rounding, and on which side: -1 when
// every face's _face_area is 0, +1 when it is the face's full area U V, 0 when it must be computed.
// Over the unit cube n . xi spans [lo, hi] = [sum min(n_i, 0), sum max(n_i, 0)]. If a - hi exceeds
// 64 u (|n|_1 + |a|) (u the unit roundoff of T), every face has n_p x + n_q y < a - n_c s with that
// margin, so gvf2 (whose rounding error is a few u of the same scale, in T or, mixed, in FP64
// from T's base) reaches its alpha >= s return, 1, and the area is (U V) (1 - 1) = 0; if lo - a
// exceeds it, gvf2 returns 0 and the area is U V. A NaN or infinite plane fails both tests.
template <class T>
__device__ __forceinline__ int plane_side(const T n[3], T a) {
  const T zero = T(0);
  const T lo = (fmin(n[0], zero) + fmin(n[1], zero)) + fmin(n[2], zero);
  const T hi = (fmax(n[0], zero) + fmax(n[1], zero)) + fmax(n[2], zero);
  const T tol = (sizeof(T) == 4 ? T(0x1p-18) : T(0x1p-47)) * (((fabs(n[0]) + fabs(n[1])) + fabs(n[2])) + fabs(a));
  return a - hi > tol ? -1 : (lo - a > tol ? 1 : 0);
}

// m / full for a face area m of a face of area full > 0, bit for bit: an area of exactly 0 or
// exactly full (every face the plane misses) gives m itself (0 / full keeps m's sign) or 1
// without the division. The resolved value's halving, (a + b) / 2, is taken as (a + b) * 0.5:
// both round the same real number.
template <class T>
__device__ __forceinline__ T frac_of(T m, T full) { return m == T(0) ? m : (m == full ? T(1) : m / full); }

// The resolved faces (src/plic/cache.jl:118-162) in 2D, tile by tile: every cell's one-sided lengths
// (_face_area, apertures.jl:73-125) computed once into shared memory, with the faces the
// neighbouring cells outside the tile show it; each shared face is then resolved from its two
// one-sided lengths, (left / full + right / full) / 2, the same expression in the same order from
// either side, so the face is single-valued bit for bit. Boundary faces are one-sided.
template <class T, bool MX>
__global__ void __launch_bounds__(NT, 6) plic_face_kernel(const DevGrid<T> g, const Cols cols, const T* __restrict__ normals,
                                                       const T* __restrict__ intercepts, const uint8_t* __restrict__ valid) {
  constexpr int NF = 4;
  constexpr int NH = 2 * (PX + PY);         // the halo: 2 PY faces along x, then 2 PX along y
  __shared__ T own[NF][NT];                 // one-sided lengths, face-major (no bank conflicts)
  __shared__ T halo[NH];
  __shared__ __align__(16) T res[NT * NF];  // resolved fractions, cell-major as in the column
  const long long n[2] = {g.n[0], g.n[1]};
  const T* vf = static_cast<const T*>(cols.vf);
  T* ff = static_cast<T*>(cols.ff);
  const T cs[2] = {g.d[0], g.d[1]};
  const long long tx = (n[0] + PX - 1) / PX, ty = (n[1] + PY - 1) / PY;
  const unsigned ntiles = unsigned(tx * ty);
  const int q = threadIdx.x, lq[2] = {q % PX, q / PX};
  for (unsigned tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    long long i0[2];
    tile_origin(tile, unsigned(tx), i0);
    const long long idx[2] = {i0[0] + lq[0], i0[1] + lq[1]};
    const bool in = idx[0] < n[0] && idx[1] < n[1];
    if (in) {  // this cell's plane, read once, on all its faces
      const long long ci = idx[0] + n[0] * idx[1];
      const T nrm[2] = {normals[2 * ci], normals[2 * ci + 1]};
      const T a = intercepts[ci], frac = vf[ci];
      const bool ok = valid[ci] != 0;
#pragma unroll
      for (int k = 0; k < NF; ++k) own[k][q] = face_area<T, MX>(nrm, a, frac, ok, cs, k);
    }
    // the halo: for each axis and side, the cell beyond the tile shows its face toward the tile
    if (q < NH) {
      const int ax = q >= 2 * PY, h = ax ? q - 2 * PY : q, len = ax ? PX : PY;
      const int side = h / len, pos = h % len;
      long long nb[2];
      nb[ax] = side == 0 ? i0[ax] - 1 : i0[ax] + (ax ? PY : PX);
      nb[1 - ax] = i0[1 - ax] + pos;
      if (nb[ax] >= 0 && nb[ax] < n[ax] && nb[1 - ax] < n[1 - ax]) {
        const long long cj = nb[0] + n[0] * nb[1];
        halo[q] = face_area<T, MX>(normals + 2 * cj, intercepts[cj], vf[cj], valid[cj] != 0, cs,
                                   side == 0 ? 2 * ax + 1 : 2 * ax);
      }
    }
    __syncthreads();
    if (in) {
#pragma unroll
      for (int k = 0; k < NF; ++k) {
        const int c = k >> 1, stride = c == 0 ? 1 : PX, ext = c == 0 ? PX : PY;
        const T full = cs[1 - c];
        const T* shown = halo + (c == 0 ? 0 : 2 * PY) + lq[1 - c];  // by the cells beyond the lower side
        const T mine = own[k][q];
        T r;
        if ((k & 1) == 0) {
          const T below = lq[c] > 0 ? own[k + 1][q - stride] : shown[0];
          r = idx[c] >= 1 ? (frac_of(below, full) + frac_of(mine, full)) * T(0.5) : frac_of(mine, full);
        } else {
          const T above = lq[c] < ext - 1 ? own[k - 1][q + stride] : shown[c == 0 ? PY : PX];
          r = idx[c] <= n[c] - 2 ? (frac_of(mine, full) + frac_of(above, full)) * T(0.5) : frac_of(mine, full);
        }
        res[q * NF + k] = r;
      }
    }
    __syncthreads();
    // the tile's rows leave whole: a row is PX cells x NF values, contiguous in the column
    const int rowcells = (int)(n[0] - i0[0] < PX ? n[0] - i0[0] : PX);
    constexpr int RV = PX * NF * int(sizeof(T)) / 16;  // 16-byte vectors per full row
    for (int w = q; w < PY * RV; w += NT) {
      const int row = w / RV, v = w - row * RV;
      const long long j = i0[1] + row;
      if (j >= n[1]) continue;
      const long long c0 = i0[0] + n[0] * j;
      if (rowcells == PX && (reinterpret_cast<uintptr_t>(ff + NF * c0) & 15u) == 0) {
        reinterpret_cast<uint4*>(ff + NF * c0)[v] = reinterpret_cast<const uint4*>(res + row * PX * NF)[v];
      } else {
        constexpr int PER = 16 / int(sizeof(T));
        for (int e = v * PER; e < (v + 1) * PER; ++e)
          if (e < rowcells * NF) ff[NF * c0 + e] = res[row * PX * NF + e];
      }
    }
    __syncthreads();  // the next tile reuses own, halo and res
  }
}

// The 3D passes' row of cells (a warp), rows per CTA, and most layers per warp.
constexpr int FZ_X = 32, FZ_Y = 8, FZ_KZ = 32;

// What the 3D centroid passes know of a tape: a union (SPHERES) or smooth union (SMOOTH) of spheres,
// pruned per warp; a tape of hard combinators (SELECT), whose gradient is one primitive's; any other
// (DUAL), evaluated on duals throughout.
enum PlaneMode { DUAL = 0, SPHERES = 1, SMOOTH = 2, SELECT = 3 };

// The box of one warp's centroids: a row of ni cells, nk layers.
template <class T>
struct RowBox {
  float lo[3], hi[3], mag;
  __device__ __forceinline__ RowBox(const DevGrid<T>& g, double scale, long long i0, int ni, long long j, long long k0, int nk) {
    const long long first[3] = {i0, j, k0}, last[3] = {i0 + ni - 1, j, k0 + nk - 1};
    mag = 0.0f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      lo[a] = bound_f32<T, true>(g.x0[a] + (T(first[a]) + T(0.5)) * g.d[a], scale);
      hi[a] = bound_f32<T, true>(g.x0[a] + (T(last[a]) + T(0.5)) * g.d[a], scale);
      mag += fabsf(bound_f32<T, true>(g.x0[a], scale)) + float(g.n[a]) * bound_f32<T, true>(g.d[a], scale);
    }
  }
};

// The body's value and gradient at the points of a row's march in z, by the tape's mode; `list`: the
// warp's m kept spheres. A row that keeps one sphere holds it, with the x and y part of its distance,
// in registers (ONE).
template <class T, int MODE>
struct RowBody {
  const STape<T>& t;
  const unsigned* list;
  int m;
  T x[3];

  // the value alone
  __device__ __forceinline__ T value(T z) {
    x[2] = z;
    if constexpr (MODE == SPHERES || MODE == SMOOTH) {
      SphereAt<T> h;
      T v = sphere_at<T>(t.p + (list[0] & 0xffffu), x, h);
      for (int i = 1; i < m; ++i) {
        const T u = sphere_at<T>(t.p + (list[i] & 0xffffu), x, h);
        v = tape_combine<T, T>(MODE == SPHERES ? CC_COMB_MIN : CC_COMB_SMIN, v, u, MODE == SPHERES ? T(0) : t.p[list[i] >> 16]);
      }
      return v;
    } else {
      return tape_eval<T, 3, T>(t, x);
    }
  }
  __device__ __forceinline__ Dual<T, 3> at(T z) {
    x[2] = z;
    Dual<T, 3> r;
    if constexpr (MODE == SPHERES) {
      SphereAt<T> h;
      r.v = sphere_at<T>(t.p + (list[0] & 0xffffu), x, h);
      for (int i = 1; i < m; ++i) {
        SphereAt<T> w;
        T v;
        if (sphere_below<T>(t.p + (list[i] & 0xffffu), x, r.v, w, v)) { r.v = v; h = w; }
      }
      sphere_grad<T>(h, r.g);
    } else if constexpr (MODE == SMOOTH) {
      // the smooth step returns the smaller value unchanged where the two are k or more apart: then
      // no gradient is needed yet (`raw`: r is the sphere h, its gradient not formed)
      SphereAt<T> h;
      r.v = sphere_at<T>(t.p + (list[0] & 0xffffu), x, h);
      r.g[0] = r.g[1] = r.g[2] = T(0);
      bool raw = true;
      for (int i = 1; i < m; ++i) {
        const unsigned e = list[i];
        SphereAt<T> w;
        Dual<T, 3> v;
        v.v = sphere_at<T>(t.p + (e & 0xffffu), x, w);
        const T k = t.p[e >> 16];
        if (k - dabs(r.v - v.v) > T(0)) {
          if (raw) sphere_grad<T>(h, r.g);
          raw = false;
          sphere_grad<T>(w, v.g);
          r = tape_combine<T, Dual<T, 3>>(CC_COMB_SMIN, r, v, k);
        } else if (v.v < r.v) {
          r.v = v.v;
          h = w;
          raw = true;
        }
      }
      if (raw) sphere_grad<T>(h, r.g);
    } else if constexpr (MODE == SELECT) {
      r = tape_eval_select<T>(t, x);
    } else {
      Dual<T, 3> xd[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        xd[a].v = x[a];
#pragma unroll
        for (int b = 0; b < 3; ++b) xd[a].g[b] = a == b ? T(1) : T(0);
      }
      r = tape_eval<T, 3, Dual<T, 3>>(t, xd);
    }
    return r;
  }
};
template <class T>
struct OneSphere {  // sphere_at's arithmetic, the part that z does not change formed once
  SphereAt<T> h;
  T cz, rad, u01;
  __device__ __forceinline__ OneSphere(const T* p, T x, T y) {
    T c[4];
    ldq(p, c);
    h.d[0] = x - c[0];
    h.d[1] = y - c[1];
    u01 = h.d[0] * h.d[0];
    u01 = u01 + h.d[1] * h.d[1];
    cz = c[2];
    rad = c[3];
  }
  __device__ __forceinline__ Dual<T, 3> at(T z) {
    Dual<T, 3> r;
    h.d[2] = z - cz;
    h.s = dsqrt(u01 + h.d[2] * h.d[2]);
    r.v = h.s - rad;
    sphere_grad<T>(h, r.g);
    return r;
  }
};

// cell_plane (src/plic/plic.jl:72-88) from the body's dual at the centroid, with the cell's side: plane_side's
// of a valid plane, else closed (-1) or open (1) by the value's sign. Where plane_side says that a valid plane misses the cell, gvf3 returns 1 or 0: its
// alpha is then beyond s or below 0 by far more than the few roundings of its sums.
template <class T, bool MX>
__device__ __forceinline__ PlaneFit<T, 3> plane_of(const Dual<T, 3>& r, T h, int& side) {
  T s = r.g[0];
  s = s + r.g[1];
  s = s + r.g[2];
  const T a = T(0.5) * s - r.v / h;
  PlaneFit<T, 3> pl;
  pl.valid = !(isnan(a) || (r.g[0] == T(0) && r.g[1] == T(0) && r.g[2] == T(0)));
  if (!pl.valid) {
    pl.n[0] = pl.n[1] = pl.n[2] = pl.a = T(0);
    pl.fraction = r.v <= T(0) ? T(1) : T(0);
    side = T(1) - pl.fraction < T(0.5) ? -1 : 1;
    return pl;
  }
  pl.n[0] = r.g[0];
  pl.n[1] = r.g[1];
  pl.n[2] = r.g[2];
  pl.a = a;
  side = plane_side<T>(pl.n, a);
  if (side != 0) pl.fraction = side < 0 ? T(1) : T(0);
  else pl.fraction = gvf3m<T, MX>(r.g[0], r.g[1], r.g[2], a);
  return pl;
}

__device__ __forceinline__ void put_pair(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }
__device__ __forceinline__ void put_pair(double* p, double a, double b) { *reinterpret_cast<double2*>(p) = make_double2(a, b); }

// A cell that its plane crosses, kept until the warp clips its faces; `at`: its first face fraction
// from the warp's first.
template <class T>
struct CrossedCell {
  T n[3], a;
  long long at;
};
constexpr int CROSSED_MAX = 64;

// The one-sided fractions (_face_area over the full face, frac_of) of n crossed cells, one face per lane.
template <class T, bool MX>
__device__ __forceinline__ void clip_crossed(const CrossedCell<T>* cells, int n, const DevGrid<T>& g, T* ff) {
  const T full = (T(1) * g.d[0]) * g.d[0];  // PLIC grids are isotropic
  for (int e = threadIdx.x & 31; e < 6 * n; e += 32) {
    const int q = e / 6, f = e - 6 * q;
    const CrossedCell<T>& c = cells[q];
    const T np = c.n[f < 2 ? 1 : 0], nq = c.n[f < 4 ? 2 : 1];
    const T base = c.n[f >> 1] * ((f & 1) ? T(1) : T(0)) - c.a;
    T area;
    if (np == T(0) && nq == T(0)) area = base >= T(0) ? full : T(0);
    else area = full * (T(1) - gvf2m<T, MX>(np, nq, -base));
    ff[c.at + f] = frac_of(area, full);
  }
  __syncwarp();  // the list is filled again
}

// The fit pass in 3D: a warp owns a row of FZ_X cells and `depth` layers of it, prunes a union of
// spheres to that box by itself (no CTA barrier after the tape is loaded) and marches up the layers.
// Only the selected sphere's gradient is formed. Normals leave through the warp's own staging row so
// that each store covers whole sectors. A cell's faces are written here too, one-sided: of a cell that
// its plane misses, all open or all closed; a crossed cell's are clipped from a list, full warps at a
// time. plic_resolve_kernel then joins the two sides. (A face pass that read every cell's side and
// resolved all six faces through shared memory took as long as the fit.) Near both its bounds: 5.6 TB/s
// of stores (512^3 Float32, 64 spheres: 6.26 GB in 1.11 ms) and 84% of the issue slots (256^3). Boxes of 8 x 4
// and 16 x 2 columns keep fewer spheres (1.3 and 1.6 instead of 2.0 at 512^3), but their stores cost 8% and 6% more.
// CTAs per SM, updates at 512^3: at Float32 4 (3: 2% slower; mixed, whose SPHERES and SMOOTH forms spill a
// little there, 4 against 3: spheres 1385 and 1413 us, CSG body 2507 and 2538, smooth blob 2558 and 2531), at Float64 2
// with spheres (3: 3% slower), else 3 (2: 10% slower, CSG body at 150 x 97 x 131).
// Updates, before (a fit on duals pruned per CTA, a pass over every face) and now: 512^3, 64 spheres, Float32 3.27 ->
// 1.22 ms, Float64 5.10 -> 2.38, mixed 3.61 -> 1.39; a smooth blob at 256^3 Float32 now 427 us.
template <class T, bool MX, int MODE>
__global__ void __launch_bounds__(NT, sizeof(T) == 4 ? 4 : (MODE == SPHERES || MODE == SMOOTH ? 2 : 3))
    plic_fit_z_kernel(const DevGrid<T> g, const DevTape tape, const Cols cols, T* __restrict__ normals,
                      T* __restrict__ intercepts, uint8_t* __restrict__ valid, int8_t* __restrict__ sides, int depth) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ T s_nrm[NT / 32][3 * FZ_X];
  __shared__ CrossedCell<T> s_crossed[NT / 32][CROSSED_MAX];
  static_assert(sizeof(s_nrm) + sizeof(s_crossed) <= 27 * 1024, "see allow_dynamic_smem");
  const STape<T> t = load_tape<T>(tape.bytes, tape.n_ops, tape.n_params, smem);
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long n0 = g.n[0], n1 = g.n[1], n2 = g.n[2];
  const unsigned ntx = unsigned((n0 + FZ_X - 1) / FZ_X), nty = unsigned((n1 + FZ_Y - 1) / FZ_Y);
  unsigned b = blockIdx.x;
  const long long i0 = (long long)(b % ntx) * FZ_X;
  b /= ntx;
  const long long j = (long long)(b % nty) * FZ_Y + w, k0 = (long long)(b / nty) * depth;
  if (j >= n1) return;
  const int nk = n2 - k0 < depth ? int(n2 - k0) : depth, ni = n0 - i0 < FZ_X ? int(n0 - i0) : FZ_X;
  unsigned* list = reinterpret_cast<unsigned*>(smem + ((tape.bytes_len + 15) / 16) * 16) + w * tape.n_ops;
  int m = 0;
  if constexpr (MODE == SPHERES || MODE == SMOOTH) {
    const RowBox<T> box(g, tape.scale, i0, ni, j, k0, nk);
    m = prune_warp<T>(t, MODE, tape.scale, box.lo, box.hi, box.mag, list);
  }
  const bool in = lane < ni;
  const T x = centroid_coord(g.x0[0], g.d[0], i0 + lane), y = centroid_coord(g.x0[1], g.d[1], j);
  const T kf = T(k0), z0 = g.x0[2], dz = g.d[2];
  // T(k) + T(0.5) is T(double(k) + 0.5) while k + 0.5 fits T's mantissa
  const bool exact_z = sizeof(T) == 8 || k0 < (1 << 22) - FZ_KZ;
  T* const nrm = s_nrm[w];
  CrossedCell<T>* const crossed = s_crossed[w];
  int ncrossed = 0;
  const int cell_of[3] = {lane / 3, (lane + 32) / 3, (lane + 64) / 3};  // the cells of this lane's face pairs
  const long long nxy = n0 * n1, row = i0 + n0 * j + nxy * k0;
  // this lane's place in each column, moved up a layer at a time
  T* np = normals + 3 * row + lane;
  T* ap = intercepts + row + lane;
  T* vp = static_cast<T*>(cols.vf) + row + lane;
  T* fp = static_cast<T*>(cols.ff) + 6 * row;
  int8_t* kp = cols.kind + row + lane;
  int8_t* sp = sides + row + lane;
  uint8_t* okp = valid + row + lane;
  T* const ff0 = fp;
  const bool pairs = (reinterpret_cast<uintptr_t>(cols.ff) & (2 * sizeof(T) - 1)) == 0;
  // FULL: a whole row, whose stores need no bounds, in a column that takes pairs (the seven bounds tests a
  // layer were a tenth of the issue slots: update at 512^3 Float32 1.43 -> 1.29 ms)
  auto march = [&](auto&& body, auto full) {
    constexpr bool FULL = decltype(full)::value;
    for (int kk = 0; kk < nk; ++kk) {
      const T z = FULL || exact_z ? z0 + ((kf + T(kk)) + T(0.5)) * dz : centroid_coord(z0, dz, k0 + kk);
      int side;
      const PlaneFit<T, 3> pl = plane_of<T, MX>(body.at(z), g.d[0], side);
      const T frac = T(1) - pl.fraction;
      nrm[3 * lane] = pl.n[0];
      nrm[3 * lane + 1] = pl.n[1];
      nrm[3 * lane + 2] = pl.n[2];
      __syncwarp();
#pragma unroll
      for (int e = 0; e < 3; ++e)
        if (FULL || lane + 32 * e < 3 * ni) np[32 * e] = nrm[lane + 32 * e];
      __syncwarp();  // read before the next layer's normals are staged
      if (FULL || in) {
        *ap = pl.a;
        *vp = frac;
        *okp = pl.valid ? 1 : 0;
        *kp = frac == T(0) ? 0 : (frac == T(1) ? 1 : 2);
        *sp = int8_t(side);
      }
      // every face of a cell that its plane misses is open (1) or closed (0), all of it
      const unsigned open = __ballot_sync(0xffffffffu, side > 0);
      if (FULL || pairs) {
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          const T v = (open >> cell_of[e]) & 1u ? T(1) : T(0);
          if (FULL || cell_of[e] < ni) put_pair(fp + 2 * (lane + 32 * e), v, v);
        }
      } else {
        for (int e = lane; e < 6 * ni; e += 32) fp[e] = (open >> (e / 6)) & 1u ? T(1) : T(0);
      }
      // crossed cells wait until there are enough to clip their faces on full warps
      const unsigned cross = __ballot_sync(0xffffffffu, (FULL || in) && side == 0);
      if (cross) {
        if ((FULL || in) && side == 0) {
          CrossedCell<T>& c = crossed[ncrossed + __popc(cross & ((1u << lane) - 1u))];
          c.n[0] = pl.n[0];
          c.n[1] = pl.n[1];
          c.n[2] = pl.n[2];
          c.a = pl.a;
          c.at = 6 * (lane + nxy * kk);
        }
        ncrossed += __popc(cross);
        __syncwarp();  // also orders the layer's open / closed faces before the clipped ones
        if (ncrossed > CROSSED_MAX - 32) {
          clip_crossed<T, MX>(crossed, ncrossed, g, ff0);
          ncrossed = 0;
        }
      }
      np += 3 * nxy;
      ap += nxy;
      vp += nxy;
      fp += 6 * nxy;
      kp += nxy;
      sp += nxy;
      okp += nxy;
    }
    clip_crossed<T, MX>(crossed, ncrossed, g, ff0);
  };
  auto run = [&](auto full) {
    if (MODE == SPHERES && m == 1) march(OneSphere<T>(t.p + (list[0] & 0xffffu), x, y), full);
    else march(RowBody<T, MODE>{t, list, m, {x, y, T(0)}}, full);
  };
  if (ni == FZ_X && pairs && exact_z) run(std::true_type());
  else run(std::false_type());
}

// 0x80 in each byte of x that is zero, nothing elsewhere (no carry crosses a byte: (b & 0x7f) +
// 0x7f <= 0xfe).
__device__ __forceinline__ unsigned zero_bytes(unsigned x) {
  return ~(((x & 0x7f7f7f7fu) + 0x7f7f7f7fu) | x | 0x7f7f7f7fu);
}

// The resolved faces in 3D (src/plic/cache.jl:118-162). The fit has written every cell's one-sided
// fractions into its faces; a face between two cells takes their mean, (lower + upper) / 2, which only
// changes it where one of the two is crossed by its plane (side 0) or their sides differ, about the
// interface's area. A warp reads 512 side bytes and their +x, +y, +z neighbours' sixteen a lane, lists
// the cells that own such a face (the upper faces of a cell are its own) in shared memory, and forms
// the means, one cell per lane, written to both cells. Each face is resolved by its lower cell alone,
// with the expression and order of the reference, so it is single-valued bit for bit. Bytes compared
// across a row's or a layer's end, or past the grid (the array is padded by a layer), only list a
// cell that then turns out to own nothing.
template <class T>
__global__ void __launch_bounds__(NT) plic_resolve_kernel(const DevGrid<T> g, T* __restrict__ ff,
                                                          const int8_t* __restrict__ sides, long long total) {
  __shared__ uint16_t s_list[NT / 32][512];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long n0 = g.n[0], n1 = g.n[1], nxy = n0 * n1;
  const long long step[3] = {1, n0, nxy};
  for (long long base = 512 * ((long long)blockIdx.x * (NT / 32) + w); base < total; base += 512LL * gridDim.x * (NT / 32)) {
    const long long c = base + 16 * lane;
    unsigned act[4] = {0, 0, 0, 0};
    int mine = 0;
    if (c < total) {
      auto sixteen = [&](long long at, unsigned v[5]) {  // the word-aligned bytes from `at` (a multiple of 16) on
        const uint4 a = *reinterpret_cast<const uint4*>(sides + at);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
      };
      unsigned o[5], yz[2][4];
      sixteen(c, o);
      o[4] = *reinterpret_cast<const unsigned*>(sides + c + 16);
#pragma unroll
      for (int d = 0; d < 2; ++d) {
        const long long at = c + step[d + 1];
        const int r = int(at & 15);  // the same for every lane
        // no cell beyond: the padding's bytes would list them all (400 x 400 x 1 without a body: 41 -> 36 us a call)
        if (c >= total - step[d + 1]) {
#pragma unroll
          for (int q = 0; q < 4; ++q) yz[d][q] = o[q];
        } else if (r == 0) {
          sixteen(at, yz[d]);
        } else {
          unsigned u[8];
          sixteen(at - r, u);
          sixteen(at - r + 16, u + 4);
          const int q0 = r >> 2, sh = (r & 3) * 8;
          unsigned v[5];
#pragma unroll
          for (int q = 0; q < 5; ++q)
            v[q] = q0 == 0 ? u[q] : q0 == 1 ? u[q + 1] : q0 == 2 ? u[q + 2 < 8 ? q + 2 : 7] : u[q + 3 < 8 ? q + 3 : 7];
#pragma unroll
          for (int q = 0; q < 4; ++q) yz[d][q] = __funnelshift_r(v[q], v[q + 1], sh);
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const unsigned x = __funnelshift_r(o[q], o[q + 1], 8);
        const unsigned differ = (o[q] ^ x) | (o[q] ^ yz[0][q]) | (o[q] ^ yz[1][q]);
        act[q] = (zero_bytes(differ) ^ 0x80808080u) | zero_bytes(o[q]);
        mine += __popc(act[q]);
      }
    }
    if (__ballot_sync(0xffffffffu, mine != 0) == 0) continue;
    int at = mine;  // inclusive sum over the lanes, then this lane's first entry
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, at, s);
      if (lane >= s) at += v;
    }
    const int count = __shfl_sync(0xffffffffu, at, 31);
    at -= mine;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      for (unsigned m = act[q]; m; m &= m - 1) s_list[w][at++] = uint16_t(16 * lane + 4 * q + ((__ffs(m) - 1) >> 3));
    __syncwarp();
    for (int e = lane; e < count; e += 32) {
      const long long ci = base + s_list[w][e];
      if (ci >= total) continue;
      long long idx[3];
      if (total < (1LL << 32)) {
        const unsigned u = unsigned(ci), a = u / unsigned(n0);
        idx[0] = u - a * unsigned(n0);
        const unsigned k = a / unsigned(n1);
        idx[1] = a - k * unsigned(n1);
        idx[2] = k;
      } else {
        idx[0] = ci % n0;
        idx[1] = (ci / n0) % n1;
        idx[2] = ci / nxy;
      }
      const int sc = sides[ci];
      bool own[3];
      T lower[3], upper[3];
#pragma unroll
      for (int ax = 0; ax < 3; ++ax) {
        own[ax] = idx[ax] + 1 < g.n[ax];
        if (own[ax]) own[ax] = sc == 0 || sides[ci + step[ax]] != sc;
        lower[ax] = upper[ax] = T(0);
        if (own[ax]) {
          lower[ax] = ff[6 * ci + 2 * ax + 1];
          upper[ax] = ff[6 * (ci + step[ax]) + 2 * ax];
        }
      }
#pragma unroll
      for (int ax = 0; ax < 3; ++ax)
        if (own[ax]) {
          const T r = (lower[ax] + upper[ax]) * T(0.5);
          ff[6 * ci + 2 * ax + 1] = r;
          ff[6 * (ci + step[ax]) + 2 * ax] = r;
        }
    }
    __syncwarp();  // the next 512 cells reuse the list
  }
}

// Neumaier-compensated accumulation in Float64.
struct KSum {
  double s, c;
  __device__ __forceinline__ void add(double x) {
    const double t = s + x;
    if (fabs(s) >= fabs(x)) c += (s - t) + x;
    else c += (x - t) + s;
    s = t;
  }
};

// The CTA's sums into out[0..1] (sum, compensation): a butterfly per warp, then the warps in order.
__device__ __forceinline__ void block_ksum(KSum a, double* out) {
  __shared__ double s_part[NT / 32][2];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double s = __shfl_down_sync(0xffffffffu, a.s, o), c = __shfl_down_sync(0xffffffffu, a.c, o);
    a.add(s);
    a.c += c;
  }
  if ((threadIdx.x & 31) == 0) {
    s_part[threadIdx.x >> 5][0] = a.s;
    s_part[threadIdx.x >> 5][1] = a.c;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int w = 1; w < NT / 32; ++w) {
    a.add(s_part[w][0]);
    a.c += s_part[w][1];
  }
  out[0] = a.s;
  out[1] = a.c;
}

// calc_volume, src/volume.jl:29-40: every cell's cell_plane solid fraction, summed (2D).
template <class T, bool MX>
__global__ void __launch_bounds__(NT) calc_volume_kernel(const DevGrid<T> g, const DevTape tape, double* partial) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_count;
  const STape<T> t = load_tape<T>(tape.bytes, tape.n_ops, tape.n_params, smem);
  __syncthreads();
  const long long n0 = g.n[0], n1 = g.n[1];
  const long long tx = (n0 + PX - 1) / PX, ty = (n1 + PY - 1) / PY;
  KSum acc{0.0, 0.0};
  const unsigned ntiles = unsigned(tx * ty);
  for (unsigned tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    long long i0[2];
    tile_origin(tile, unsigned(tx), i0);
    const STape<T> u = tile_tape<T>(t, tape, g, i0, smem, &s_count);
    const long long idx[2] = {i0[0] + threadIdx.x % PX, i0[1] + threadIdx.x / PX};
    if (idx[0] < n0 && idx[1] < n1) acc.add(double(cell_plane<T, MX>(u, g, idx).fraction));
    __syncthreads();
  }
  block_ksum(acc, partial + 2 * blockIdx.x);
}

// calc_volume in 3D. Only cells near the interface have a fraction other than 0 or 1: with |grad|_1 <=
// L1 (the tape's bound), a plane whose value exceeds thr = h L1 / 2 (and 0.1% for rounding) misses its
// cell, and gvf3 returns 0 or 1; a cell without a valid plane takes its fraction from the value's sign,
// the same 0 or 1. So the grid is taken in boxes of VX x VY x VZ cells: a warp first evaluates the body at
// the centres of `group` boxes, a lane each, and settles every box whose value is beyond thr plus what
// the body can change over the box (its Lipschitz constant, and `margin` for the rounding of values and
// coordinates); the boxes left are evaluated cell by cell, and the gradient and the clip are formed only
// where |value| <= thr. Whole cells are counted, partial ones summed compensated in Float64. A tape
// without a Lipschitz bound settles nothing and every cell takes its plane.
// Before: every cell's plane on duals, 32 layers of a column one after another (the time of a 64^3
// grid was that of 256^3), and one thread adding up the CTAs' partials (80 us). 64 spheres, kernels:
// 256^3 Float64 687 -> 103 us, 64^3 Float64 667 -> 27 us, 512^3 Float32 1906 -> 150 us. Centres in Float32
// on all lanes, and listing the near cells, took the 256^3 time from 244 to 103 us.
constexpr int VX = 8, VY = 4, VZ = 8;

// SCALED: lengths are brought into Float32's range first (in_bounds_range); its own instantiation, since the
// multiplications made 512^3 Float64 3% slower.
template <class T, bool MX, int MODE, bool SCALED>
__global__ void __launch_bounds__(NT) calc_volume_z_kernel(const DevGrid<T> g, const DevTape tape, double* partial,
                                                           T thr, T beyond, int group) {
  extern __shared__ __align__(16) unsigned char smem[];
  const STape<T> t = load_tape<T>(tape.bytes, tape.n_ops, tape.n_params, smem);
  __syncthreads();
  __shared__ uint8_t s_near[NT / 32][VX * VY * VZ];
  static_assert(VX * VY == 32 && VX * VY * VZ <= 256, "a box's cells are numbered in a byte");
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned* list = reinterpret_cast<unsigned*>(smem + ((tape.bytes_len + 15) / 16) * 16) + w * tape.n_ops;
  const long long nx = (g.n[0] + VX - 1) / VX, ny = (g.n[1] + VY - 1) / VY, nz = (g.n[2] + VZ - 1) / VZ;
  const long long boxes = nx * ny * nz;
  const T h = g.d[0];
  KSum acc{0.0, 0.0};
  long long whole = 0;
  for (long long first = ((long long)blockIdx.x * (NT / 32) + w) * group; first < boxes;
       first += (long long)gridDim.x * (NT / 32) * group) {
    // the lane's box: its first cell, and its extents in the grid. Of a union of spheres, all 32 lanes
    // take part whatever the group, `share` of them on the spheres of one box, in Float32 (the margin
    // covers that); the first of them answers for the box
    const int share = MODE == SPHERES ? 32 / group : 1, mine = lane / share;
    long long i0[3] = {0, 0, 0};
    int ext[3] = {0, 0, 0};
    bool open = false;
    T v = T(0);
    const bool any = mine < group && first + mine < boxes;
    if (any) {
      const long long bx = first + mine, r = bx / nx;
      i0[0] = (bx - r * nx) * VX;
      i0[2] = r / ny;
      i0[1] = (r - i0[2] * ny) * VY;
      i0[2] *= VZ;
      const int full[3] = {VX, VY, VZ};
      T x[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        ext[a] = g.n[a] - i0[a] < full[a] ? int(g.n[a] - i0[a]) : full[a];
        x[a] = g.x0[a] + (T(i0[a]) + T(0.5) * T(full[a])) * g.d[a];
      }
      if constexpr (MODE == SPHERES) {
        float least = __int_as_float(0x7f800000);
        float probe = 0.0f;  // not a number once any distance is infinite or not one
        const float b[3] = {bound_f32<T, SCALED>(x[0], tape.scale), bound_f32<T, SCALED>(x[1], tape.scale), bound_f32<T, SCALED>(x[2], tape.scale)};
        for (int i = lane % share; i < t.n_ops; i += share) {
          float c[4];
          bound_sphere<T, SCALED>(t.p + t.ops[i].poff, tape.scale, c);
          const float d0 = b[0] - c[0], d1 = b[1] - c[1], d2 = b[2] - c[2];
          const float u = sqrt_approx(d0 * d0 + d1 * d1 + d2 * d2) - c[3];
          probe = __fmaf_rn(u, 0.0f, probe);
          least = fminf(least, u);
        }
        v = probe == 0.0f ? T(least) : qnan<T>();  // times the scale, as `beyond` is
      } else {
        v = tape_eval<T, 3, T>(t, x);
      }
    }
    if constexpr (MODE == SPHERES) {
      for (int o = share / 2; o > 0; o >>= 1) {
        const T u = __shfl_xor_sync(0xffffffffu, v, o);
        v = u < v || !(u == u) ? u : v;  // the least, or NaN
      }
    }
    if (any && lane % share == 0) {
      const bool inside = v < -beyond && v - v == T(0);  // an infinite value says nothing of the box: it overflowed
      if (inside) whole += ext[0] * ext[1] * ext[2];
      open = !inside && !(v > beyond && v - v == T(0));
    }
    for (unsigned left = __ballot_sync(0xffffffffu, open); left; left &= left - 1) {
      const int src = __ffs(left) - 1;
      long long c0[3];
      int ce[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        c0[a] = __shfl_sync(0xffffffffu, i0[a], src);
        ce[a] = __shfl_sync(0xffffffffu, ext[a], src);
      }
      int m = 0;
      if constexpr (MODE == SPHERES || MODE == SMOOTH) {
        float lo[3], hi[3], mag = 0.0f;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          lo[a] = bound_f32<T, SCALED>(g.x0[a] + (T(c0[a]) + T(0.5)) * g.d[a], tape.scale);
          hi[a] = bound_f32<T, SCALED>(g.x0[a] + (T(c0[a] + ce[a] - 1) + T(0.5)) * g.d[a], tape.scale);
          mag += fabsf(bound_f32<T, SCALED>(g.x0[a], tape.scale)) + float(g.n[a]) * bound_f32<T, SCALED>(g.d[a], tape.scale);
        }
        m = prune_warp<T, false, SCALED>(t, MODE, tape.scale, lo, hi, mag, list);
      }
      // cells near enough to need their plane are listed, then taken on full warps
      const bool in = lane % VX < ce[0] && lane / VX < ce[1];
      RowBody<T, MODE> body{t, list, m,
                            {centroid_coord(g.x0[0], g.d[0], c0[0] + lane % VX),
                             centroid_coord(g.x0[1], g.d[1], c0[1] + lane / VX), T(0)}};
      int count = 0;
      for (int k = 0; k < ce[2]; ++k) {
        const T vc = body.value(centroid_coord(g.x0[2], g.d[2], c0[2] + k));
        const bool near = in && !(vc > thr) && !(vc < -thr);
        whole += in && vc < -thr ? 1 : 0;
        const unsigned b = __ballot_sync(0xffffffffu, near);
        if (near) s_near[w][count + __popc(b & ((1u << lane) - 1u))] = uint8_t(k * 32 + lane);
        count += __popc(b);
      }
      __syncwarp();
      for (int e = lane; e < count; e += 32) {
        const int q = s_near[w][e] & 31, k = s_near[w][e] >> 5;
        body.x[0] = centroid_coord(g.x0[0], g.d[0], c0[0] + q % VX);
        body.x[1] = centroid_coord(g.x0[1], g.d[1], c0[1] + q / VX);
        int side;
        acc.add(double(plane_of<T, MX>(body.at(centroid_coord(g.x0[2], g.d[2], c0[2] + k)), h, side).fraction));
      }
      __syncwarp();  // the next box reuses the lists
    }
  }
  acc.add(double(whole));
  block_ksum(acc, partial + 2 * blockIdx.x);
}

__global__ void __launch_bounds__(NT) calc_volume_final(const double* partial, int nb, double* out) {
  KSum a{0.0, 0.0};
  for (int i = threadIdx.x; i < nb; i += NT) {
    a.add(partial[2 * i]);
    a.c += partial[2 * i + 1];
  }
  __shared__ double s_sum[2];
  block_ksum(a, s_sum);
  if (threadIdx.x == 0) out[0] = s_sum[0] + s_sum[1];
}

// cut_cell_report, src/cut_cell.jl:302-319: counts by kind, ambiguous, smallest cut fraction.
// Each thread takes 16 cells at a time with 16-byte loads of the kind and ambiguous columns (the
// caller guarantees 16-byte aligned columns for the vector part; the tail is scalar).
template <class T>
__device__ __forceinline__ void report_cell(int k, int a, T v, unsigned long long& cut, unsigned long long& ins,
                                            unsigned long long& out, unsigned long long& am, T& vmin) {
  cut += k == 2;
  ins += k == 0;
  out += k == 1;
  am += a != 0;
  if (k == 2 && v > T(0) && v < vmin) vmin = v;
}

template <class T>
__global__ void __launch_bounds__(NT) report_kernel(long long ncell, const int8_t* __restrict__ kind,
                                                    const uint8_t* __restrict__ amb, const T* __restrict__ vf,
                                                    unsigned long long* counts, unsigned long long* vmin_bits,
                                                    int vec_ok) {
  unsigned long long cut = 0, ins = 0, out = 0, am = 0;
  T vmin = T(1);
  const long long nvec = vec_ok ? ncell / 16 : 0;
  const uint4* kind4 = reinterpret_cast<const uint4*>(kind);
  const uint4* amb4 = reinterpret_cast<const uint4*>(amb);
  // sixteen cells: the bytes of each word equal to 2 (cut), 0 (inside), 1 (outside), and the
  // nonzero ambiguous bytes, counted exactly whatever the byte values; the fraction is only read
  // for cut cells, which are few
  auto sixteen = [&](const uint4 kk, const uint4 aa, long long g) {
    const unsigned kw[4] = {kk.x, kk.y, kk.z, kk.w};
    const unsigned aw[4] = {aa.x, aa.y, aa.z, aa.w};
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const unsigned cutm = zero_bytes(kw[w] ^ 0x02020202u);
      cut += __popc(cutm);
      ins += __popc(zero_bytes(kw[w]));
      out += __popc(zero_bytes(kw[w] ^ 0x01010101u));
      am += 4 - __popc(zero_bytes(aw[w]));
      for (unsigned m = cutm; m; m &= m - 1) {
        const T v = vf[16 * g + 4 * w + ((__ffs(m) - 1) >> 3)];
        if (v > T(0) && v < vmin) vmin = v;
      }
    }
  };
  const long long stride = (long long)gridDim.x * NT;
  long long g = blockIdx.x * (long long)NT + threadIdx.x;
  for (; g + 3 * stride < nvec; g += 4 * stride) {  // four strides' loads in flight before any test
    uint4 kk[4], aa[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      kk[u] = kind4[g + u * stride];
      aa[u] = amb4[g + u * stride];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) sixteen(kk[u], aa[u], g + u * stride);
  }
  for (; g < nvec; g += stride) sixteen(kind4[g], amb4[g], g);
  for (long long i = 16 * nvec + blockIdx.x * (long long)NT + threadIdx.x; i < ncell; i += (long long)gridDim.x * NT)
    report_cell<T>(kind[i], amb[i], kind[i] == 2 ? vf[i] : T(1), cut, ins, out, am, vmin);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    cut += __shfl_down_sync(0xffffffffu, cut, o);
    ins += __shfl_down_sync(0xffffffffu, ins, o);
    out += __shfl_down_sync(0xffffffffu, out, o);
    am += __shfl_down_sync(0xffffffffu, am, o);
    const T w = __shfl_down_sync(0xffffffffu, vmin, o);
    vmin = w < vmin ? w : vmin;
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(counts + 0, cut);
    atomicAdd(counts + 1, ins);
    atomicAdd(counts + 2, out);
    atomicAdd(counts + 3, am);
    // non-negative floats order as their bit patterns; the slot keeps the complement's maximum, so
    // it starts from 0 like the counters and the host zeroes all five with one memset
    const double dv = double(vmin);
    atomicMax(vmin_bits, ~(unsigned long long)__double_as_longlong(dv));
  }
}

int blocks_for(long long work, int per_sm) {
  long long b = (work + NT - 1) / NT;
  const long long cap = 148LL * per_sm;
  return int(b < 1 ? 1 : (b > cap ? cap : b));
}

// Monte Carlo volume of {phi < 0} in the box lo..hi: point p's coordinates are three
// successive splitmix64 outputs of (seed, 3p + a), 53 random bits each, mapped to [lo, hi);
// the body is evaluated in Float64. Counts accumulate per thread, then per CTA, then into
// out[0] with one atomic add per CTA.
__device__ __forceinline__ unsigned long long splitmix64(unsigned long long z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__global__ void __launch_bounds__(NT) monte_carlo_kernel(const DevTape tape, double lo0, double lo1, double lo2,
                                                         double hi0, double hi1, double hi2, long long npts,
                                                         unsigned long long seed, unsigned long long* out) {
  extern __shared__ __align__(16) unsigned char smem[];
  const STape<double> t = load_tape<double>(tape.bytes, tape.n_ops, tape.n_params, smem);
  __syncthreads();
  const double lo[3] = {lo0, lo1, lo2}, span[3] = {hi0 - lo0, hi1 - lo1, hi2 - lo2};
  unsigned long long inside = 0;
  for (long long p = blockIdx.x * (long long)NT + threadIdx.x; p < npts; p += (long long)gridDim.x * NT) {
    double x[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const unsigned long long r = splitmix64(seed ^ (unsigned long long)(3 * p + a));
      x[a] = lo[a] + double(r >> 11) * 0x1.0p-53 * span[a];
    }
    inside += tape_eval<double, 3, double>(t, x) < 0.0 ? 1 : 0;
  }
  __shared__ unsigned long long part[NT / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) inside += __shfl_xor_sync(0xffffffffu, inside, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x / 32] = inside;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long s = 0;
    for (int w = 0; w < NT / 32; ++w) s += part[w];
    atomicAdd(out, s);
  }
}

}  // namespace

namespace cci {

cudaError_t launch_monte_carlo(const DevTape& tape, const double lo[3], const double hi[3], long long npts,
                               unsigned long long seed, unsigned long long* out, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(out, 0, sizeof(unsigned long long), s);
  if (e != cudaSuccess || npts <= 0) return e;
  const int sm = ((tape.bytes_len + 15) / 16) * 16;
  monte_carlo_kernel<<<blocks_for(npts, 16), NT, sm, s>>>(tape, lo[0], lo[1], lo[2], hi[0], hi[1], hi[2], npts, seed,
                                                          out);
  return cudaGetLastError();
}

namespace {

// Layers per warp of the 3D fit: the pruning slab of a union of spheres, else 16; halved while the
// launch would leave SMs without their eight CTAs, so that a small grid is not a few long columns. Without
// pruning a box costs less to start and 16 CTAs are better (CSG body at 150 x 97 x 131, Float64: fit 134, 105
// and 94 us at 4, 8 and 16; with, 64 spheres at 128^3: 43, 43 and 49).
template <class T>
int fit_depth(const DevGrid<T>& g, const DevTape& tape) {
  int depth = tape.prunable && tape.slab > 0 && tape.slab <= FZ_KZ ? tape.slab : 16;
  const long long tiles = ((g.n[0] + FZ_X - 1) / FZ_X) * ((g.n[1] + FZ_Y - 1) / FZ_Y);
  const long long enough = 148 * (tape.prunable ? 8 : 16);
  while (depth > 2 && tiles * ((g.n[2] + depth - 1) / depth) < enough) depth /= 2;
  return depth;
}

template <class T, int MODE>
cudaError_t launch_fit_z(const DevGrid<T>& g, const DevTape& tape, const Cols& cols, T* normals, T* intercepts,
                         uint8_t* valid, int8_t* sides, bool mx, cudaStream_t s) {
  const int depth = fit_depth(g, tape);
  const long long blocks = ((g.n[0] + FZ_X - 1) / FZ_X) * ((g.n[1] + FZ_Y - 1) / FZ_Y) * ((g.n[2] + depth - 1) / depth);
  if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  // the tape, then each warp's list of kept spheres
  const int lists = MODE == SPHERES || MODE == SMOOTH ? (NT / 32) * tape.n_ops * int(sizeof(unsigned)) : 0;
  const int sm = ((tape.bytes_len + 15) / 16) * 16 + lists;
  auto run = [&](auto kernel) {
    const cudaError_t e = allow_dynamic_smem(kernel, sm);
    if (e != cudaSuccess) return e;
    kernel<<<unsigned(blocks), NT, sm, s>>>(g, tape, cols, normals, intercepts, valid, sides, depth);
    return cudaGetLastError();  // the resolve pass must not follow a fit that did not run
  };
  if constexpr (sizeof(T) == 4) {
    if (mx) return run(plic_fit_z_kernel<T, true, MODE>);
  }
  return run(plic_fit_z_kernel<T, false, MODE>);
}

}  // namespace

template <class T, int D>
cudaError_t launch_plic(const DevGrid<T>& g, const DevTape& body, const Cols& cols, T* normals, T* intercepts,
                        uint8_t* valid, int8_t* sides, cudaStream_t s, bool mixed) {
  const long long total = g.n[0] * g.n[1] * (D == 3 ? g.n[2] : 1);
  const DevTape tape = D == 3 ? in_bounds_range(body, g) : body;
  if constexpr (D == 3) {
    if (!sides) return cudaErrorInvalidValue;
    const bool mx = mixed && sizeof(T) == 4;
    cudaError_t e;
    if (tape.prunable == 1) e = launch_fit_z<T, SPHERES>(g, tape, cols, normals, intercepts, valid, sides, mx, s);
    else if (tape.prunable == 2) e = launch_fit_z<T, SMOOTH>(g, tape, cols, normals, intercepts, valid, sides, mx, s);
    else if (tape.select) e = launch_fit_z<T, SELECT>(g, tape, cols, normals, intercepts, valid, sides, mx, s);
    else e = launch_fit_z<T, DUAL>(g, tape, cols, normals, intercepts, valid, sides, mx, s);
    if (e != cudaSuccess) return e;
    const long long rows = (total + 512 * (NT / 32) - 1) / (512 * (NT / 32));
    const unsigned rb = unsigned(rows < 148 * 8 ? rows : 148 * 8);
    plic_resolve_kernel<T><<<rb, NT, 0, s>>>(g, static_cast<T*>(cols.ff), sides, total);
  } else {  // 2D works in tiles
    const int sm = CentroidSmem::of(tape).bytes;
    cudaError_t e = allow_dynamic_smem(plic_fit_kernel<T, true>, sm);
    if (e == cudaSuccess) e = allow_dynamic_smem(plic_fit_kernel<T, false>, sm);
    if (e != cudaSuccess) return e;
    if (mixed && sizeof(T) == 4) {
      plic_fit_kernel<T, true><<<blocks_for(total, 16), NT, sm, s>>>(g, tape, cols, normals, intercepts, valid);
      plic_face_kernel<T, true><<<blocks_for(total, 16), NT, 0, s>>>(g, cols, normals, intercepts, valid);
    } else {
      plic_fit_kernel<T, false><<<blocks_for(total, 16), NT, sm, s>>>(g, tape, cols, normals, intercepts, valid);
      plic_face_kernel<T, false><<<blocks_for(total, 16), NT, 0, s>>>(g, cols, normals, intercepts, valid);
    }
  }
  return cudaGetLastError();
}

int calc_volume_blocks() { return VOL_BLOCKS; }

namespace {

template <class T, int MODE>
cudaError_t launch_volume_z(const DevGrid<T>& g, const DevTape& tape, const TapeBounds& tb, double* partial, int* nb,
                            bool mx, cudaStream_t s) {
  const double h = double(g.d[0]);
  double mag = tb.mag;
  for (int a = 0; a < 3; ++a) mag += std::fabs(double(g.x0[a])) + double(g.n[a]) * double(g.d[a]);
  double thr = 0.5 * tb.grad1 * h * 1.001;
  const double half = 0.5 * h * std::sqrt(double(VX * VX + VY * VY + VZ * VZ));
  const double margin = (sizeof(T) == 4 || MODE == SPHERES ? 0x1p-16 : 0x1p-40) * (1.0 + tb.lipschitz) * mag;
  double beyond = (thr + tb.lipschitz * half) * 1.001 + margin;
  // where T's squares are not normal (as in in_bounds_range) values err by more than the margin: nothing is settled
  const double inf = std::numeric_limits<double>::infinity();
  if (!(mag >= (sizeof(T) == 8 ? 0x1p-480 : 0x1p-48) && mag <= (sizeof(T) == 8 ? 0x1p480 : 0x1p60))) thr = beyond = inf;
  if (MODE == SPHERES) beyond *= tape.scale;
  const long long boxes = ((g.n[0] + VX - 1) / VX) * ((g.n[1] + VY - 1) / VY) * ((g.n[2] + VZ - 1) / VZ);
  // boxes per warp at a time: few enough that every resident warp has some
  int group = 32;
  while (group > 1 && boxes < (long long)group * VOL_BLOCKS * (NT / 32)) group /= 2;
  const long long ctas = (boxes + group * (NT / 32) - 1) / (group * (NT / 32));
  *nb = int(ctas < VOL_BLOCKS ? ctas : VOL_BLOCKS);
  const int lists = MODE == SPHERES || MODE == SMOOTH ? (NT / 32) * tape.n_ops * int(sizeof(unsigned)) : 0;
  const int sm = ((tape.bytes_len + 15) / 16) * 16 + lists;
  auto run = [&](auto kernel) {
    const cudaError_t e = allow_dynamic_smem(kernel, sm);
    if (e != cudaSuccess) return e;
    kernel<<<*nb, NT, sm, s>>>(g, tape, partial, T(thr), T(beyond), group);
    return cudaGetLastError();
  };
  if constexpr (sizeof(T) == 4) {
    if (mx) return run(calc_volume_z_kernel<T, true, MODE, false>);
  } else if constexpr (MODE == SPHERES || MODE == SMOOTH) {
    if (tape.scale != 1.0) return run(calc_volume_z_kernel<T, false, MODE, true>);
  }
  return run(calc_volume_z_kernel<T, false, MODE, false>);
}

}  // namespace

template <class T, int D>
cudaError_t launch_calc_volume(const DevGrid<T>& g, const DevTape& body, const TapeBounds& tb, double* partial,
                               double* out, cudaStream_t s, bool mixed) {
  int nb = VOL_BLOCKS;
  const DevTape tape = D == 3 ? in_bounds_range(body, g) : body;
  cudaError_t e;
  if constexpr (D == 3) {
    const bool mx = mixed && sizeof(T) == 4;
    if (tape.prunable == 1) e = launch_volume_z<T, SPHERES>(g, tape, tb, partial, &nb, mx, s);
    else if (tape.prunable == 2) e = launch_volume_z<T, SMOOTH>(g, tape, tb, partial, &nb, mx, s);
    else if (tape.select) e = launch_volume_z<T, SELECT>(g, tape, tb, partial, &nb, mx, s);
    else e = launch_volume_z<T, DUAL>(g, tape, tb, partial, &nb, mx, s);
    if (e != cudaSuccess) return e;
  } else {
    const int sm = CentroidSmem::of(tape).bytes;
    e = allow_dynamic_smem(calc_volume_kernel<T, true>, sm);
    if (e == cudaSuccess) e = allow_dynamic_smem(calc_volume_kernel<T, false>, sm);
    if (e != cudaSuccess) return e;
    if (mixed && sizeof(T) == 4) calc_volume_kernel<T, true><<<nb, NT, sm, s>>>(g, tape, partial);
    else calc_volume_kernel<T, false><<<nb, NT, sm, s>>>(g, tape, partial);
  }
  calc_volume_final<<<1, NT, 0, s>>>(partial, nb, out);
  return cudaGetLastError();
}

cudaError_t launch_report(long long ncell, const int8_t* kind, const uint8_t* amb, const void* vf, int is_f64,
                          unsigned long long* counts, double* vmin, cudaStream_t s) {
  // four CTAs of 256 per SM (the unrolled loop's registers), each thread with eight 16-byte
  // loads in flight: 128 KB per SM
  const int nb = blocks_for((ncell + 15) / 16, 4);
  unsigned long long* vb = reinterpret_cast<unsigned long long*>(vmin);
  const int vec_ok = ((reinterpret_cast<uintptr_t>(kind) | reinterpret_cast<uintptr_t>(amb)) & 15u) == 0;
  if (is_f64)
    report_kernel<double><<<nb, NT, 0, s>>>(ncell, kind, amb, static_cast<const double*>(vf), counts, vb, vec_ok);
  else
    report_kernel<float><<<nb, NT, 0, s>>>(ncell, kind, amb, static_cast<const float*>(vf), counts, vb, vec_ok);
  return cudaGetLastError();
}

#define INST(T, D)                                                                                      \
  template cudaError_t launch_plic<T, D>(const DevGrid<T>&, const DevTape&, const Cols&, T*, T*, uint8_t*, int8_t*, \
                                         cudaStream_t, bool);                                           \
  template cudaError_t launch_calc_volume<T, D>(const DevGrid<T>&, const DevTape&, const TapeBounds&, double*, double*, \
                                                cudaStream_t, bool);
INST(float, 2)
INST(float, 3)
INST(double, 2)
INST(double, 3)
#undef INST

}  // namespace cci
