// ms.cu -- MarchingSquaresCutCell update_cache! on sm_100a: a grid (nodal phi block) and the
// leaves of an AdaptiveMesh{2} quadtree.
//
// Grid: a warp per strip of 32 cells by a few rows samples its nodes from the op-tape and builds its cells
// from them (the reference's _sample_nodes_kernel!, src/marching_squares/cache.jl:67-70, and
// _nodal_cells_kernel!, :75-78, in one pass), or, where that does not pay (strips_pay), two passes. Tree: one thread per leaf samples its four lattice corners
// and builds its moments from exactly those (_leaf_cells_kernel!, :129-137).
#include <cstdint>
#include <type_traits>
#include "cc_device.cuh"
#include "cc_internal.h"
#include "ms_cell.cuh"
#include "ms_tile.cuh"

namespace {

using namespace ccd;
using namespace ccms;
using cci::Cols;
using cci::DevGrid;
using cci::DevTape;

constexpr int NT = 256;

constexpr int GRID_NT = 128;  // four warps, each with its own strips

// SAMPLE: phi is written from the tape; else it holds the nodal values. I: the grid's index type. A strip per
// warp, strips numbered x fastest. Against the two passes (strips_pay): 2000 x 1500 Float32, one circle, 43 -> 32 us;
// 200 x 200 Float64, bound by one cut cell's latency, 6.3 -> 6.5 us with one launch less.
template <class T, bool MX, bool SAMPLE, class I>
__global__ void __launch_bounds__(GRID_NT, sizeof(T) == 4 ? 8 : 4) ms_grid_kernel(const DevGrid<T> g, const DevTape tape, T* phi, const Cols cols,
                                                          int ty) {
  extern __shared__ __align__(16) unsigned char smem[];
  STape<T> t{nullptr, nullptr, 0};
  if (SAMPLE) {
    t = load_tape<T>(tape.bytes, tape.n_ops, tape.n_params, smem);
    __syncthreads();
  }
  const int w = threadIdx.x >> 5;
  unsigned char* own = smem + (SAMPLE ? ((tape.bytes_len + 15) / 16) * 16 : 0) + w * strip_bytes<T>(ty);
  const I n0 = I(g.n[0]), n1 = I(g.n[1]);
  const unsigned long long nsx = ((unsigned long long)n0 + STRIP - 1) / STRIP, nsy = ((unsigned long long)n1 + ty - 1) / ty;
  for (unsigned long long s = blockIdx.x * (unsigned long long)(GRID_NT / 32) + w; s < nsx * nsy;
       s += gridDim.x * (unsigned long long)(GRID_NT / 32)) {
    const unsigned long long sy = nsx * nsy < (1ull << 32) ? unsigned(s) / unsigned(nsx) : s / nsx;
    ms_strip<T, MX, SAMPLE, I>(t, g.x0[0], g.x0[1], g.d[0], g.d[1], n0, n1, I((s - sy * nsx) * STRIP), I(sy * ty), ty,
                               own, phi, cols);
  }
}

// (i, j) of item v of an n0-wide box: a 32-bit quotient where the box has fewer than 2^32 items
// (every grid that fits a device), else 64-bit.
__device__ __forceinline__ void split2(long long v, long long n0, bool small, long long& i, long long& j) {
  if (small) {
    const unsigned q = unsigned(v) / unsigned(n0);
    j = q;
    i = (long long)(unsigned(v) - q * unsigned(n0));
  } else {
    j = v / n0;
    i = v - j * n0;
  }
}

// The two passes by nodes and by cells, a thread each, where strips do not pay (strips_pay).
template <class T>
__global__ void __launch_bounds__(NT) ms_sample_kernel(const DevGrid<T> g, const DevTape tape, T* phi) {
  extern __shared__ __align__(16) unsigned char smem[];
  const STape<T> t = load_tape<T>(tape.bytes, tape.n_ops, tape.n_params, smem);
  __syncthreads();
  const long long nx = g.n[0] + 1, ny = g.n[1] + 1, total = nx * ny;
  const bool small = total + (long long)gridDim.x * NT < (1LL << 32);
  for (long long v = blockIdx.x * (long long)NT + threadIdx.x; v < total; v += (long long)gridDim.x * NT) {
    long long i, j;
    split2(v, nx, small, i, j);
    const T x[2] = {node_coord(g.x0[0], g.d[0], i), node_coord(g.x0[1], g.d[1], j)};
    phi[v] = tape_eval<T, 2, T>(t, x);
  }
}

template <class T, bool MX>
__global__ void __launch_bounds__(NT) ms_cells_kernel(const DevGrid<T> g, const T* __restrict__ phi, const Cols cols) {
  const long long n0 = g.n[0], n1 = g.n[1], nx = n0 + 1, total = n0 * n1;
  const T cs[2] = {g.d[0], g.d[1]};
  const bool small = total + (long long)gridDim.x * NT < (1LL << 32);
  for (long long ci = blockIdx.x * (long long)NT + threadIdx.x; ci < total; ci += (long long)gridDim.x * NT) {
    long long i, j;
    split2(ci, n0, small, i, j);
    const T xa = node_coord(g.x0[0], g.d[0], i), xb = node_coord(g.x0[0], g.d[0], i + 1);
    const T ya = node_coord(g.x0[1], g.d[1], j), yb = node_coord(g.x0[1], g.d[1], j + 1);
    const T nd[4][2] = {{xa, ya}, {xb, ya}, {xb, yb}, {xa, yb}};
    const long long b = i + nx * j;
    const T ph[4] = {phi[b], phi[b + 1], phi[b + nx + 1], phi[b + nx]};
    ms_cell<T, MX>(nd, ph, cs, cols, ci);
  }
}

template <class T, bool MX>
__global__ void __launch_bounds__(NT) ms_tree_kernel(const T x00, const T x01, const double bd0, const double bd1,
                                                     long long nl, const int32_t* __restrict__ level,
                                                     const int32_t* __restrict__ coord, const DevTape tape, T* phi4,
                                                     const Cols cols) {
  extern __shared__ __align__(16) unsigned char smem[];
  const STape<T> t = load_tape<T>(tape.bytes, tape.n_ops, tape.n_params, smem);
  __syncthreads();
  for (long long i = blockIdx.x * (long long)NT + threadIdx.x; i < nl; i += (long long)gridDim.x * NT) {
    ms_leaf<T, MX>(t, x00, x01, T(bd0), T(bd1), level[i], coord[2 * i], coord[2 * i + 1], phi4, cols, i);
  }
}

int grid_blocks(long long work) {
  long long b = (work + NT - 1) / NT;
  const long long cap = 148LL * 16;
  return int(b < 1 ? 1 : (b > cap ? cap : b));
}

}  // namespace

namespace cci {

namespace {
template <class T>
bool strips_pay(const DevGrid<T>& g, const DevTape& tape, bool sample) {
  // Strips fuse the two passes and store whole sectors, but sample an extra node row and column each, evaluate
  // nodes in groups per lane, and idle the lanes beyond a narrow grid's end. Two passes / strips, us:
  //   one circle: Float32 500^2 21 / 18, 1000^2 22 / 19, 4096^2 231 / 152; Float64 21 / 18, 37 / 33, 422 / 297; 1 x 40000
  //     (whole calls) Float32 35 / 41, Float64 37 / 49, 33 x 20000 4% and 8% slower, 40 x 20000 level
  //   union of 8: Float32 1000^2 34 / 26, 4096^2 412 / 269, 100 x 20000 57 / 50; Float64 55 / 55, 674 / 546, 91 / 97
  //   of 20: Float32 500^2 25 / 31, 1000^2 56 / 48, 4096^2 724 / 540; Float64 1400^2 145 / 159, 3000^2 602 / 600
  //   of 100: Float32 500^2 62 / 123, 1000^2 185 / 184, 2047 x 1500 530 / 479; Float64 4096^2 3909 / 4762
  //   a star curve, 1400^2: Float32 48 / 50, Float64 91 / 106
  //   given values (whole calls), 1000^2, 2047 x 1500, 4096^2: Float32 41 / 42, 63 / 67, 224 / 219, Float64 57 / 59, 107 / 109, 436 / 391
  const long long cells = g.n[0] * g.n[1], lanes = (g.n[0] + STRIP - 1) / STRIP * STRIP;
  const bool full = 10 * g.n[0] >= 9 * lanes;
  if (!sample) return full && cells >= 6000000;
  if (tape.cost <= 2) return cells <= 16384 || 10 * g.n[0] >= 6 * lanes;
  if (tape.cost >= COSTLY || cells < 1000000) return false;
  if (sizeof(T) == 4) return tape.cost <= 8 ? 4 * g.n[0] >= 3 * lanes : full && (tape.cost <= 20 || cells >= 3000000);
  return full && (tape.cost <= 8 || (tape.cost <= 20 && cells >= 9000000));
}
}  // namespace

template <class T>
cudaError_t launch_ms(const DevGrid<T>& g, const DevTape& tape, const T* phi_in, T* phi_out,
                      const Cols& cols, cudaStream_t s, bool mixed) {
  if (!strips_pay<T>(g, tape, phi_in == nullptr)) {
    const T* phi = phi_in;
    if (!phi_in) {
      const int sm = ((tape.bytes_len + 15) / 16) * 16;
      const cudaError_t e = allow_dynamic_smem(ms_sample_kernel<T>, sm);
      if (e != cudaSuccess) return e;
      ms_sample_kernel<T><<<grid_blocks((g.n[0] + 1) * (g.n[1] + 1)), NT, sm, s>>>(g, tape, phi_out);
      phi = phi_out;
    }
    if (mixed && sizeof(T) == 4) ms_cells_kernel<T, true><<<grid_blocks(g.n[0] * g.n[1]), NT, 0, s>>>(g, phi, cols);
    else ms_cells_kernel<T, false><<<grid_blocks(g.n[0] * g.n[1]), NT, 0, s>>>(g, phi, cols);
    return cudaGetLastError();
  }
  // eight rows per strip, fewer while that leaves SMs without warps (the strip's one extra node row
  // then costs more, latency less)
  int ty = 8;
  const long long nsx = (g.n[0] + STRIP - 1) / STRIP;
  while (ty > 1 && nsx * ((g.n[1] + ty - 1) / ty) < 148 * 8) ty /= 2;
  const long long strips = nsx * ((g.n[1] + ty - 1) / ty), ctas = (strips + GRID_NT / 32 - 1) / (GRID_NT / 32);
  const unsigned blocks = unsigned(ctas < 148LL * 64 ? ctas : 148LL * 64);
  const int sm = (phi_in ? 0 : ((tape.bytes_len + 15) / 16) * 16) + (GRID_NT / 32) * strip_bytes<T>(ty);
  T* phi = phi_in ? const_cast<T*>(phi_in) : phi_out;  // read only without SAMPLE
  const bool wide = g.n[0] >= 0x7fffff00LL || g.n[1] >= 0x7fffff00LL;
  auto run = [&](auto kernel) {
    const cudaError_t e = allow_dynamic_smem(kernel, sm);
    if (e != cudaSuccess) return e;
    kernel<<<blocks, GRID_NT, sm, s>>>(g, tape, phi, cols, ty);
    return cudaGetLastError();
  };
  auto pick = [&](auto mx) {
    constexpr bool MX = decltype(mx)::value;
    if (phi_in) return wide ? run(ms_grid_kernel<T, MX, false, long long>) : run(ms_grid_kernel<T, MX, false, int>);
    return wide ? run(ms_grid_kernel<T, MX, true, long long>) : run(ms_grid_kernel<T, MX, true, int>);
  };
  if constexpr (sizeof(T) == 4) {
    if (mixed) return pick(std::true_type());
  }
  return pick(std::false_type());
}

template <class T>
cudaError_t launch_ms_tree(const T x0[2], const double base_d[2], long long nleaves, const int32_t* level,
                           const int32_t* coord, const DevTape& tape, T* phi4, const Cols& cols, cudaStream_t s,
                           bool mixed) {
  if (nleaves <= 0) return cudaSuccess;
  const int sm = ((tape.bytes_len + 15) / 16) * 16;
  if (mixed && sizeof(T) == 4)
    ms_tree_kernel<T, true><<<grid_blocks(nleaves), NT, sm, s>>>(x0[0], x0[1], base_d[0], base_d[1], nleaves, level,
                                                                 coord, tape, phi4, cols);
  else
    ms_tree_kernel<T, false><<<grid_blocks(nleaves), NT, sm, s>>>(x0[0], x0[1], base_d[0], base_d[1], nleaves, level,
                                                                  coord, tape, phi4, cols);
  return cudaGetLastError();
}

template cudaError_t launch_ms<float>(const DevGrid<float>&, const DevTape&, const float*, float*, const Cols&, cudaStream_t,
                                      bool);
template cudaError_t launch_ms<double>(const DevGrid<double>&, const DevTape&, const double*, double*, const Cols&,
                                       cudaStream_t, bool);
template cudaError_t launch_ms_tree<float>(const float*, const double*, long long, const int32_t*, const int32_t*,
                                           const DevTape&, float*, const Cols&, cudaStream_t, bool);
template cudaError_t launch_ms_tree<double>(const double*, const double*, long long, const int32_t*, const int32_t*,
                                            const DevTape&, double*, const Cols&, cudaStream_t, bool);

}  // namespace cci
