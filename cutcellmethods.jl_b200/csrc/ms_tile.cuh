// ms_tile.cuh -- marching squares over a strip of 32 cells by ty rows, one warp: its nodes sampled (or
// read) once into the warp's own shared memory, then its cells row by row, a lane per column. Shared by
// the single-grid update (ms.cu) and the batch (batch.cu). Nothing here waits for another warp.
//
// What one thread per cell paid again for every cell is per strip or per row here: a column's x
// coordinates and face centroids, the lower row's corner signs (the upper row's of the row before), the
// linear index, and the op dispatch (several nodes per lane and pass). An uncut cell is a dozen instructions
// and its stores. Cut cells are listed and take ms_cell, the same construction as everywhere, on full warps
// after the rows. Bound by its stores. A warp's row leaves as whole sectors (store_cell2's vectors).
#pragma once
#include <cstdint>
#include "cc_device.cuh"
#include "cc_internal.h"
#include "ms_cell.cuh"

namespace ccms {

constexpr int STRIP = 32;           // cells per row of a strip: a warp
constexpr int STRIP_X = STRIP + 1;  // its nodes per row
// a warp's shared memory: the strip's nodes, then the list of its cut cells (row * 32 + column)
template <class T> __host__ __device__ constexpr int strip_list(int ty) { return (STRIP_X * (ty + 1) * int(sizeof(T)) + 15) / 16 * 16; }
template <class T> __host__ __device__ constexpr int strip_bytes(int ty) { return (strip_list<T>(ty) + 2 * STRIP * ty + 15) / 16 * 16; }

// get_node's coordinate x0 + T(i) d from an index of either width: T(i) is the same value.
template <class T, class I>
__device__ __forceinline__ T node_coord_i(T x0, T d, I i) { return x0 + T(i) * d; }

template <class T>
__device__ __forceinline__ bool cols_vectors(const Cols& c) {  // store_cell2's condition
  return ((reinterpret_cast<uintptr_t>(c.c) | reinterpret_cast<uintptr_t>(c.ff) | reinterpret_cast<uintptr_t>(c.fcl) |
           reinterpret_cast<uintptr_t>(c.ic)) & 15u) == 0;
}
__device__ __forceinline__ void put2(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }
__device__ __forceinline__ void put2(double* p, double a, double b) { *reinterpret_cast<double2*>(p) = make_double2(a, b); }
__device__ __forceinline__ void put4(float* p, float a, float b, float c, float d) {
  *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}
__device__ __forceinline__ void put4(double* p, double a, double b, double c, double d) {
  reinterpret_cast<double2*>(p)[0] = make_double2(a, b);
  reinterpret_cast<double2*>(p)[1] = make_double2(c, d);
}

// The strip of cells i0.. , j0.. (ty rows) of an n0 x n1 grid. SAMPLE: nodes from the tape, those the strip
// owns written to phi; else read from phi. `own`: the warp's strip_bytes(ty).
template <class T, bool MX, bool SAMPLE, class I>
__device__ __forceinline__ void ms_strip(const STape<T>& tp, T gx0, T gy0, T dx, T dy, I n0, I n1, I i0, I j0, int ty,
                                         unsigned char* own, T* phi, const Cols& cols) {
  constexpr int NB = sizeof(T) == 4 ? 5 : 3;  // nodes per lane and pass (registers)
  T* const node = reinterpret_cast<T*>(own);
  uint16_t* const list = reinterpret_cast<uint16_t*>(own + strip_list<T>(ty));
  const int lane = threadIdx.x & 31;
  const int nj = n1 - j0 < ty ? int(n1 - j0) : ty, count = STRIP_X * (nj + 1);
  const long long nx = (long long)n0 + 1;
  T* const pnode = phi + (long long)i0 + nx * j0;
  for (int v0 = lane; v0 < count; v0 += 32 * NB) {
    T x[NB][2], val[NB];
    int a[NB], b[NB];
#pragma unroll
    for (int q = 0; q < NB; ++q) {
      const int v = v0 + 32 * q;
      b[q] = v / STRIP_X;
      a[q] = v - b[q] * STRIP_X;
      if (SAMPLE) {
        x[q][0] = node_coord_i(gx0, dx, I(i0 + a[q]));
        x[q][1] = node_coord_i(gy0, dy, I(j0 + b[q]));
      }
    }
    if (SAMPLE) tape_eval_multi<T, 2, NB>(tp, x, val);
#pragma unroll
    for (int q = 0; q < NB; ++q) {
      const int v = v0 + 32 * q;
      if (v < count && i0 + a[q] <= n0) {
        if (SAMPLE) {
          if ((a[q] < STRIP || i0 + a[q] == n0) && (b[q] < ty || j0 + b[q] == n1)) pnode[a[q] + nx * b[q]] = val[q];
        } else {
          val[q] = pnode[a[q] + nx * b[q]];
        }
        node[v] = val[q];
      }
    }
  }
  __syncwarp();
  const bool in = i0 + lane < n0;
  int ncut = 0;
  {
    const T xa = node_coord_i(gx0, dx, I(i0 + lane)), xb = node_coord_i(gx0, dx, I(i0 + lane + 1));
    const T ce0 = xa + T(0.5) * dx, fx = T(0.5) * (xa + xb) - xa;
    const bool vec = cols_vectors<T>(cols);
    long long ci = (long long)i0 + lane + (long long)n0 * j0;
    int below = (node[lane] >= T(0)) + (node[lane + 1] >= T(0));
    T ya = node_coord_i(gy0, dy, j0);
    for (int b = 0; b < nj; ++b) {
      const int above = (node[STRIP_X * (b + 1) + lane] >= T(0)) + (node[STRIP_X * (b + 1) + lane + 1] >= T(0));
      const int nout = below + above;
      const T yb = node_coord_i(gy0, dy, I(j0 + b + 1));
      const bool uncut = vec && (nout == 0 || nout == 4);
      if (in && uncut) {
        const T ce1 = ya + T(0.5) * dy, fy = T(0.5) * (ya + yb) - ya;
        const T one = nout == 4 ? T(1) : T(0);
        cols.kind[ci] = nout == 4 ? 1 : 0;
        cols.amb[ci] = 0;
        static_cast<T*>(cols.vf)[ci] = one;
        put2(static_cast<T*>(cols.c) + 2 * ci, ce0, ce1);
        put4(static_cast<T*>(cols.ff) + 4 * ci, one, one, one, one);
        put4(static_cast<T*>(cols.fcl) + 4 * ci, fy, fy, fx, fx);
        put2(static_cast<T*>(cols.ic) + 2 * ci, ce0, ce1);
      }
      const unsigned cut = __ballot_sync(0xffffffffu, in && !uncut);
      if (cut) {
        if (in && !uncut) list[ncut + __popc(cut & ((1u << lane) - 1u))] = uint16_t(STRIP * b + lane);
        ncut += __popc(cut);
      }
      below = above;
      ya = yb;
      ci += n0;
    }
  }
  __syncwarp();
  for (int e = lane; e < ncut; e += 32) {
    const int a = list[e] % STRIP, b = list[e] / STRIP;
    const T xa = node_coord_i(gx0, dx, I(i0 + a)), xb = node_coord_i(gx0, dx, I(i0 + a + 1));
    const T ya = node_coord_i(gy0, dy, I(j0 + b)), yb = node_coord_i(gy0, dy, I(j0 + b + 1));
    const T nd[4][2] = {{xa, ya}, {xb, ya}, {xb, yb}, {xa, yb}};
    const T* p = node + STRIP_X * b + a;
    const T ph[4] = {p[0], p[1], p[STRIP_X + 1], p[STRIP_X]};
    const T cs[2] = {dx, dy};
    ms_cell<T, MX>(nd, ph, cs, cols, (long long)i0 + a + (long long)n0 * (j0 + b));
  }
  __syncwarp();  // the next strip reuses the nodes and the list
}

// One leaf of a quadtree: its four corners sampled, its cell built (_leaf_cells_kernel!).
template <class T, bool MX>
__device__ __forceinline__ void ms_leaf(const STape<T>& tp, T x00, T x01, T bd0, T bd1, int lv, long long cx, long long cy,
                                        T* phi4, const Cols& cols, long long l) {
  const T scale = T(ldexp(1.0, -lv));
  const T h[2] = {bd0 * scale, bd1 * scale};
  const T xa = x00 + T(cx) * h[0], xb = x00 + T(cx + 1) * h[0];
  const T ya = x01 + T(cy) * h[1], yb = x01 + T(cy + 1) * h[1];
  const T nd[4][2] = {{xa, ya}, {xb, ya}, {xb, yb}, {xa, yb}};
  T ph[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    ph[q] = tape_eval<T, 2, T>(tp, nd[q]);
    phi4[4 * l + q] = ph[q];
  }
  ms_cell<T, MX>(nd, ph, h, cols, l);
}

}  // namespace ccms
