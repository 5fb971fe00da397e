// mc.cu -- MarchingCubesCutCell update_cache! on sm_100a.
//
// Two kernels replace the reference's two KernelAbstractions launches
// (_sample_nodes_kernel! and _nodal_cells_kernel!, src/marching_squares/cache.jl:55-78):
//
//   * mc_fill_kernel: a CTA owns a pencil of TX x TY cells in (x, y) and marches up to KZ slices
//     along z. Node slabs of (TX+1) x (TY+1) values are sampled from the op-tape NS at a time into
//     a shared-memory ring, so a node is evaluated once per CTA and written to phi once, by the
//     CTA that owns it. Every thread classifies one cell from its eight corners. Uncut cells (all
//     corners of one sign) get their fields directly -- their face centroids are half the lattice
//     edge lengths, a cheap affine fill -- into a double-buffered shared-memory staging tile that
//     leaves as one TMA tensor store per StructArray column (cp.async.bulk.tensor, shared ->
//     global), so the SM's threads never issue the column stores. Cut cells are compacted with a
//     warp ballot into a global work list.
//   * mc_cut_kernel: one lane per listed cut cell runs the full construction of
//     src/marching_cubes/moments.jl:275-346 densely and writes that cell's fields.
#include <atomic>
#include <cstdint>
#include <cstring>
#include <cuda.h>
#include "cc_device.cuh"
#include "cc_internal.h"
#include "mc_cell.cuh"

namespace {

using namespace ccd;
using namespace ccmc;
using cci::Cols;
using cci::DevGrid;
using cci::DevTable;
using cci::DevTape;

// Fill-kernel tile: TX cells along x (32 at Float32, 16 at Float64, so a staging buffer is about
// 26 KB either way) by TY = 8 rows, one thread per cell, marching up to KZ slices along z. A slab of
// (TX+1) x (TY+1) nodes serves TX x TY cells: 1.16 node evaluations per cell at Float32.
template <class T> struct Tile {
  static constexpr int TX = sizeof(T) == 4 ? 32 : 16;
  static constexpr int TY = 8;
  static constexpr int NT = TX * TY;
  static constexpr int NSX = TX + 1;
  static constexpr int NSLAB = (TX + 1) * (TY + 1);
  static constexpr int MINB = sizeof(T) == 4 ? 3 : 3;  // Float64 at 4 spills
};
constexpr int NS = 4;   // node slabs sampled per round (one op-major tape pass per thread)
constexpr int KZ = 31;  // most z slices marched per CTA: KZ + 1 = 32 node slabs, 8 sampling rounds (deepest_pencil)
// The cut kernel: 128 threads, bounded to 5 CTAs per SM at Float32 and 3 at Float64 (its registers: 111
// and 239 unbounded). Kernel time in us of 128 (5, 3), 256 (3, 2) and 64 (8, 4): 512^3 Float32 80, 87, 81;
// 256^3 Float64 40, 49, 46; a wave field at 192 x 160 x 129, Float64, 136, 138, 164.
constexpr int CUT_NT = 128;

template <class T>
struct McArgs {
  DevGrid<T> g;
  DevTape tape;
  const T* phi_in;
  T* phi_out;
  Cols cols;
  DevTable tb;
  unsigned* cut_list;
  unsigned* cut_count;
  int n_itiles, n_jtiles;
  int kz;  // z slices per pencil (pencil_slices)
  int tma_mask;  // bit c: column c leaves through TMA tensor stores (its map below is valid)
  int byte_words;  // kind/ambiguous rows start on 4-byte boundaries
  int thread_cols;  // bit c: column c is copied element by element by the threads (no TMA, no words)
};

// One TMA tensor map per output column: kind, ambiguous, volume_fraction (n0 x n1 x n2), centroid
// and interface_centroid (3 n0 x n1 x n2), face_fraction (6 n0 x n1 x n2), face_centroid_local
// (12 x n0 x n1 x n2). A staged tile is exactly one box of each.
struct ColumnMaps {
  CUtensorMap m[7];
};

// TMA bulk-group bookkeeping (the tensor stores below commit into bulk groups).
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;\n" ::"n"(N) : "memory"); }
template <int N>
__device__ __forceinline__ void bulk_wait() { asm volatile("cp.async.bulk.wait_group %0;\n" ::"n"(N) : "memory"); }
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ void tma_store3(const CUtensorMap* m, const void* ssrc, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];\n" ::"l"(m),
               "r"((unsigned)__cvta_generic_to_shared(ssrc)), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}
__device__ __forceinline__ void tma_store4(const CUtensorMap* m, const void* ssrc, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];\n" ::"l"(m),
               "r"((unsigned)__cvta_generic_to_shared(ssrc)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}

// Shared-memory byte layout of one fill CTA: two staging buffers, two node slabs, the tape.
template <class T>
struct Layout {
  using TL = Tile<T>;
  static constexpr int NC = TL::NT;  // cells per staging buffer
  static constexpr int kind = 0;
  static constexpr int amb = kind + NC;
  static constexpr int vf = amb + NC;
  static constexpr int c = vf + NC * int(sizeof(T));
  static constexpr int ff = c + 3 * NC * int(sizeof(T));
  static constexpr int fcl = ff + 6 * NC * int(sizeof(T));
  // an uncut cell's interface centroid is its centroid, and a cut cell's staged values are
  // overwritten by the cut kernel: the interface_centroid box is sent from the centroid column
  static constexpr int ic = c;
  static constexpr int stage_bytes = ((fcl + 12 * NC * int(sizeof(T)) + 127) / 128) * 128;
  static constexpr int slab_bytes = ((TL::NSLAB * int(sizeof(T)) + 15) / 16) * 16;
  static constexpr int slab0 = 2 * stage_bytes;
  static constexpr int tape = slab0 + (NS + 1) * slab_bytes;
  // TMA tensor stores read each staged column from a 128-byte aligned base
  static_assert(amb % 128 == 0 && vf % 128 == 0 && c % 128 == 0 && ff % 128 == 0 && fcl % 128 == 0 &&
                    ic % 128 == 0 && stage_bytes % 128 == 0,
                "staged columns must start on 128-byte boundaries");
};

// bytes per staged row of output column `col` (kind, amb, vf, c, ff, fcl, ic) and its offset
template <class T>
__device__ __forceinline__ constexpr int col_bytes(int col) {
  return col < 2 ? Tile<T>::TX
                 : (col == 2 ? 1 : col == 3 ? 3 : col == 4 ? 6 : col == 5 ? 12 : 3) * Tile<T>::TX * int(sizeof(T));
}
template <class T>
__device__ __forceinline__ constexpr int col_offset(int col) {
  return col == 0 ? Layout<T>::kind : col == 1 ? Layout<T>::amb : col == 2 ? Layout<T>::vf : col == 3 ? Layout<T>::c
       : col == 4 ? Layout<T>::ff : col == 5 ? Layout<T>::fcl : Layout<T>::ic;
}
template <class T>
__device__ __forceinline__ Stage<T> stage_at(unsigned char* base) {
  using L = Layout<T>;
  Stage<T> st;
  st.kind = reinterpret_cast<int8_t*>(base + L::kind);
  st.amb = base + L::amb;
  st.vf = reinterpret_cast<T*>(base + L::vf);
  st.c = reinterpret_cast<T*>(base + L::c);
  st.ff = reinterpret_cast<T*>(base + L::ff);
  st.fcl = reinterpret_cast<T*>(base + L::fcl);
  st.ic = reinterpret_cast<T*>(base + L::ic);
  return st;
}

// An uncut cell whose staging slot held an uncut cell of the same kind at the slot's previous use
// (two slices earlier, in the same column): kind, flag, fraction, face fractions and the x, y
// parts are the same values, so only what depends on the slice is written -- the centroid's and
// interface centroid's z and the face centroids' half-height entries (slots 1, 3, 5, 7, written
// with their neighbours as two 16-byte vectors). The slot then holds exactly what put_cell leaves.
// 512^3 CSG body: Float32 update 2.78 -> 2.74 ms.
__device__ __forceinline__ void put_uncut_z(const Stage<float>& st, int lc, float cz, float hx, float hy, float hz) {
  st.c[3 * lc + 2] = cz;
  float4* d4 = reinterpret_cast<float4*>(st.fcl + 12 * lc);
  d4[0] = make_float4(hy, hz, hy, hz);
  d4[1] = make_float4(hx, hz, hx, hz);
}

// A warp copies n <= MOST contiguous elements.
template <class E, int MOST>
__device__ __forceinline__ void copy_row(E* __restrict__ dst, const E* __restrict__ src, int n, int lane) {
  if (n == MOST && MOST % 32 == 0) {  // a whole row, without bounds
#pragma unroll
    for (int v = 0; v < MOST; v += 32) dst[v + lane] = src[v + lane];
    return;
  }
#pragma unroll
  for (int v = 0; v < MOST; v += 32)
    if (v + lane < n) dst[v + lane] = src[v + lane];
}

// ALL_TMA: every column leaves by TMA (the common case, x extents that are multiples of 16); the
// instantiation then carries none of the thread copies (update at 512^3 Float32 2.70 -> 2.65 ms, at
// 256^3 Float64 with the report 775 -> 749 us).
template <class T, bool SAMPLE, bool PRUNED, bool ALL_TMA>
__global__ void __launch_bounds__(Tile<T>::NT, Tile<T>::MINB) mc_fill_kernel(const McArgs<T> A,
                                                                            const __grid_constant__ ColumnMaps maps) {
  using TL = Tile<T>;
  using L = Layout<T>;
  constexpr int TX = TL::TX, TY = TL::TY, NT = TL::NT, NSX = TL::NSX, NSLAB = TL::NSLAB;
  extern __shared__ __align__(128) unsigned char smem[];
  const int tid = threadIdx.x;
  const long long n0 = A.g.n[0], n1 = A.g.n[1], n2 = A.g.n[2];
  const long long nx = n0 + 1, ny = n1 + 1;

  int b = blockIdx.x;
  const int it = b % A.n_itiles; b /= A.n_itiles;
  const int jt = b % A.n_jtiles; b /= A.n_jtiles;
  const long long i0 = (long long)it * TX, j0 = (long long)jt * TY;
  const long long k0 = (long long)b * A.kz;
  const long long k1 = (k0 + A.kz < n2) ? k0 + A.kz : n2;

  STape<T> tape;
  if (SAMPLE) {
    tape = load_tape<T>(A.tape.bytes, A.tape.n_ops, A.tape.n_params, smem + L::tape);
    if (PRUNED) {
      // a union of spheres: one warp prunes it to the box of the pencil's nodes, the kept ops follow the
      // tape. (A launch of its own used to write every pencil's ops to memory. At 256^3 Float32: 64 spheres
      // 470 -> 454 us an update, a smooth blob 581 -> 571. Unions of any primitives, bounded by their value at
      // the box's centre and a Lipschitz constant, were no faster: the CSG body at 512^3 2.57 -> 2.56 ms, at
      // 256^3 Float64 642 -> 662 us.)
      __shared__ int s_kept;
      const int n = A.tape.n_ops;
      cc_op* kept = reinterpret_cast<cc_op*>(smem + L::tape + ((A.tape.bytes_len + 15) / 16) * 16);
      __syncthreads();
      if (tid < 32) {
        const long long first[3] = {i0, j0, k0}, last[3] = {i0 + TX < n0 ? i0 + TX : n0, j0 + TY < n1 ? j0 + TY : n1, k1};
        float lo[3], hi[3], mag = 0.0f;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          lo[a] = bound_f32<T, true>(node_coord(A.g.x0[a], A.g.d[a], first[a]), A.tape.scale);
          hi[a] = bound_f32<T, true>(node_coord(A.g.x0[a], A.g.d[a], last[a]), A.tape.scale);
          mag += fabsf(bound_f32<T, true>(A.g.x0[a], A.tape.scale)) + float(A.g.n[a]) * bound_f32<T, true>(A.g.d[a], A.tape.scale);
        }
        unsigned* list = reinterpret_cast<unsigned*>(kept + n);
        const int m = prune_warp<T, true>(tape, A.tape.prunable, A.tape.scale, lo, hi, mag, list);
        for (int q = tid; q < m; q += 32) {
          cc_op op = tape.ops[list[q]];
          if (q == 0) op.combine = CC_COMB_PUSH;
          kept[q] = op;
        }
        if (tid == 0) s_kept = m;
      }
      __syncthreads();
      tape.ops = kept;
      tape.n_ops = s_kept;
    }
  }
  T* const ring = reinterpret_cast<T*>(smem + L::slab0);
  constexpr int RS = L::slab_bytes / int(sizeof(T));  // ring slot stride, elements
  if (SAMPLE) __syncthreads();

  const T x0 = A.g.x0[0], y0 = A.g.x0[1], z0 = A.g.x0[2];
  const T dx = A.g.d[0], dy = A.g.d[1], dz = A.g.d[2];
  const long long nxy = nx * ny;

  // Slabs are counted from the pencil's first, in 32 bits: nk + 1 of them, of which this CTA writes nown.
  // (64-bit slab numbers and node indices, a modulo per access and all eight corners compared on every slice
  // cost: the CSG body at 512^3 Float32 2.49 -> 2.41 ms a fill, 301 x 187 x 130 mixed 226 -> 195 us, 64 spheres
  // at 256^3 402 -> 382; 512^3 then writes 5.9 TB/s, the output pipeline alone 6.1-6.2. With pencils of 31
  // slices the quicker march was slower on the largest other grids, 512^3 Float64 4.64 -> 4.74 ms; see deepest_pencil.)
  const int nk = int(k1 - k0), kfirst = int(k0), nown = k1 == n2 ? nk + 1 : nk;

  // This thread's node slots for one sampling round of NS slabs, fixed for the whole march:
  // which of the round's slabs, the slab index, coordinates, its place in phi (moved up NS slabs a round),
  // and whether this CTA owns (writes) the node.
  constexpr int NSL = (NS * NSLAB + NT - 1) / NT;
  int sl_s[NSL], sl_v[NSL];
  T sl_x[NSL], sl_y[NSL];
  T* sl_p[NSL];
  bool sl_ok[NSL], sl_own[NSL];
#pragma unroll
  for (int q = 0; q < NSL; ++q) {
    const int flat = tid + q * NT;
    const int s = flat / NSLAB, v = flat - s * NSLAB;
    const int tx = v % NSX, ty = v / NSX;
    const long long i = i0 + tx, j = j0 + ty;
    sl_s[q] = s;
    sl_v[q] = v;
    sl_ok[q] = s < NS && i <= n0 && j <= n1;
    sl_own[q] = (tx < TX || i == n0) && (ty < TY || j == n1);
    sl_x[q] = node_coord(x0, dx, i);
    sl_y[q] = node_coord(y0, dy, j);
    sl_p[q] = (SAMPLE ? A.phi_out : const_cast<T*>(A.phi_in)) + (i + nx * j + nxy * (k0 + s));
  }

  // The next round: slabs zr, zr + 1, .. (slot s samples slab zr + s, for slabs <= nk), into ring slot
  // slab % (NS + 1); phi written for owned nodes of owned slabs.
  int zr = 0, ring_zr = 0;  // the round's first slab, and that modulo NS + 1
  auto sample_round = [&]() {
    T pts[NSL][3];
    T val[NSL];
    bool use[NSL];
#pragma unroll
    for (int q = 0; q < NSL; ++q) {
      const int z = zr + sl_s[q];
      use[q] = sl_ok[q] && z <= nk;
      pts[q][0] = sl_x[q];
      pts[q][1] = sl_y[q];
      pts[q][2] = z0 + T(kfirst + z) * dz;  // node_coord
    }
    if (SAMPLE) {
      tape_eval_multi<T, 3, NSL>(tape, pts, val);
    }
#pragma unroll
    for (int q = 0; q < NSL; ++q) {
      if (use[q]) {
        T v;
        if (SAMPLE) {
          v = val[q];
          if (zr + sl_s[q] < nown && sl_own[q]) *sl_p[q] = v;
        } else {
          v = *sl_p[q];
        }
        const int r = ring_zr + sl_s[q];
        ring[(r > NS ? r - (NS + 1) : r) * RS + sl_v[q]] = v;
      }
      sl_p[q] += NS * nxy;
    }
    zr += NS;
    ring_zr = ring_zr == 0 ? NS : ring_zr - 1;  // + NS modulo NS + 1
  };

  const int tx = tid % TX, ty = tid / TX;
  const long long ci = i0 + tx, cj = j0 + ty;
  const bool valid = ci < n0 && cj < n1;
  const T xa = node_coord(x0, dx, ci), xb = node_coord(x0, dx, ci + 1);
  const T ya = node_coord(y0, dy, cj), yb = node_coord(y0, dy, cj + 1);
  const T hx = T(0.5) * (xb - xa), hy = T(0.5) * (yb - ya);
  const T cx = xa + T(0.5) * dx, cy = ya + T(0.5) * dy;
  const int lc = ty * TX + tx;
  const int s00 = ty * NSX + tx;
  const bool fast = ALL_TMA || A.tma_mask != 0;
  const int rows = (int)((n1 - j0) < TY ? (n1 - j0) : TY);
  const int cnt = (int)((n0 - i0) < TX ? (n0 - i0) : TX);
  unsigned char* gcol[7] = {reinterpret_cast<unsigned char*>(A.cols.kind), A.cols.amb,
                            reinterpret_cast<unsigned char*>(A.cols.vf), reinterpret_cast<unsigned char*>(A.cols.c),
                            reinterpret_cast<unsigned char*>(A.cols.ff), reinterpret_cast<unsigned char*>(A.cols.fcl),
                            reinterpret_cast<unsigned char*>(A.cols.ic)};

  // nudge_zeros(v) >= 0  <=>  v > -eps  (and false for NaN, as there)
  const T neps = -Eps<T>::v();
  auto outside4 = [&](const T* slab) {  // of the cell's four corners on one slab
    return (slab[s00] > neps) + (slab[s00 + 1] > neps) + (slab[s00 + NSX + 1] > neps) + (slab[s00 + NSX] > neps);
  };
  // What this thread's slot of each staging buffer holds: 0 not known (first use, or a cut cell,
  // whose slot the fill leaves alone), 1 an uncut cell outside, 2 inside (2 bits per buffer).
  int slots = 0;
  int below = 0, rk = 0;  // corners outside on the lower slab, and its ring slot
  T za = z0 + T(kfirst) * dz;
  long long k = k0;
  for (int kk = 0; kk < nk; ++kk, ++k) {
    const int sb = kk & 1;
    unsigned char* sbase = smem + sb * L::stage_bytes;
    // round r samples slabs NS r .. NS r + NS - 1 before the slice that first needs its first slab; the slabs
    // it overwrites were last read before the previous slice's barriers
    if (kk == 0 || kk % NS == NS - 1) sample_round();
    if (fast && tid == 0) bulk_wait_read<1>();  // staging buffer sb: its copy two slices ago has been read
    __syncthreads();  // slabs kk and kk + 1 ready; staging sb free

    if (kk == 0) below = outside4(ring);
    rk = rk == NS ? 0 : rk + 1;
    const int above = outside4(ring + rk * RS), nout = below + above;
    below = above;
    const T zb = z0 + T(kfirst + kk + 1) * dz, zl = za;
    za = zb;
    bool is_cut = false;
    if (valid) {
      const int state = nout == 8 ? 2 : (nout == 0 ? 1 : 0);
      if (state != 0) {
        const T hz = T(0.5) * (zb - zl);
        const T one = nout == 8 ? T(1) : T(0);
        const T cen[3] = {cx, cy, zl + T(0.5) * dz};
        // (Float32 only: at Float64 the split cost more than the stores it saved, 4.91 vs 4.76 ms)
        if (sizeof(T) == 4 && ((slots >> (2 * sb)) & 3) == state) {
          if constexpr (sizeof(T) == 4) put_uncut_z(stage_at<T>(sbase), lc, cen[2], hx, hy, hz);
        } else {
          const T ff[6] = {one, one, one, one, one, one};
          const T fcl[12] = {hy, hz, hy, hz, hx, hz, hx, hz, hx, hy, hx, hy};
          const Stage<T> st = stage_at<T>(sbase);
          st.kind[lc] = int8_t(nout == 8 ? 1 : 0);
          st.amb[lc] = 0;
          st.vf[lc] = one;
          st.c[3 * lc] = cen[0]; st.c[3 * lc + 1] = cen[1]; st.c[3 * lc + 2] = cen[2];
          put_vec<T>(st.ff + 6 * lc, ff, 6);
          put_vec<T>(st.fcl + 12 * lc, fcl, 12);
        }
      } else {
        is_cut = true;
      }
      slots = (slots & ~(3 << (2 * sb))) | (state << (2 * sb));
    }
    // Warp-ballot compaction of the cut band into the global work list. A cut cell's staged slot
    // is left as it is: the span is copied out whole and the cut kernel, which runs after this
    // one in stream order, overwrites the cell.
    const unsigned m = __ballot_sync(0xffffffffu, is_cut);
    if (m) {
      const int lane = tid & 31;
      unsigned base = 0;
      if (lane == 0) base = atomicAdd(A.cut_count, (unsigned)__popc(m));
      base = __shfl_sync(0xffffffffu, base, 0);
      if (is_cut) A.cut_list[base + __popc(m & ((1u << lane) - 1))] = (unsigned)(ci + n0 * (cj + n1 * k));
    }
    if (fast) fence_proxy_async_smem();  // staged writes visible to the bulk-copy engine
    __syncthreads();  // staging sb complete

    const long long row0 = i0 + n0 * (j0 + n1 * k);
    if (fast && tid == 0) {
      // one thread stores the TMA-addressable columns: one box each (clipped at the grid's edge)
      const int ci0 = (int)i0, cj0 = (int)j0, ck = (int)k;
      if (ALL_TMA || (A.tma_mask & 1)) tma_store3(&maps.m[0], sbase + col_offset<T>(0), ci0, cj0, ck);
      if (ALL_TMA || (A.tma_mask & 2)) tma_store3(&maps.m[1], sbase + col_offset<T>(1), ci0, cj0, ck);
      if (ALL_TMA || (A.tma_mask & 4)) tma_store3(&maps.m[2], sbase + col_offset<T>(2), ci0, cj0, ck);
      if (ALL_TMA || (A.tma_mask & 8)) tma_store3(&maps.m[3], sbase + col_offset<T>(3), 3 * ci0, cj0, ck);
      if (ALL_TMA || (A.tma_mask & 16)) tma_store3(&maps.m[4], sbase + col_offset<T>(4), 6 * ci0, cj0, ck);
      if (ALL_TMA || (A.tma_mask & 32)) tma_store4(&maps.m[5], sbase + col_offset<T>(5), 0, ci0, cj0, ck);
      if (ALL_TMA || (A.tma_mask & 64)) tma_store3(&maps.m[6], sbase + col_offset<T>(6), 3 * ci0, cj0, ck);
      bulk_commit();
    }
    if constexpr (!ALL_TMA) {
      // the columns TMA cannot address, copied by every thread: kind / ambiguous as one 32-bit word
      // per thread where every row starts on a 4-byte boundary (rows x 2 columns x TX/4 words fit
      // in the CTA), else bytes; T columns by element
      static_assert(2 * TY * (TX / 4) <= NT, "one word of kind / ambiguous per thread");
      if (A.byte_words) {
        const int wpr = (cnt + 3) / 4;  // words per row (cnt is a multiple of 4 here)
        const int w = tid % wpr, rest = tid / wpr, r = rest % TY, col = rest / TY;
        if (col < 2 && r < rows && !(A.tma_mask & (1 << col))) {
          const long long rowc = row0 + (long long)r * n0;
          reinterpret_cast<uint32_t*>(gcol[col] + rowc)[w] =
              reinterpret_cast<const uint32_t*>(sbase + col_offset<T>(col) + r * col_bytes<T>(col))[w];
        }
      }
      // the rest row by row, a warp per row (at Float64 other warps staged it: the barrier above stands
      // between). A column's part of a row is contiguous, so lane-strided elements are full-width stores
      // whatever the row's alignment. (All threads stepping through every row and column were mostly idle:
      // 301 x 187 x 130 mixed: fill 581 -> 226 us; 203^3 Float64: 1126 -> 434 us.) Most grids have none.
      if (A.thread_cols) {
        const int lane = tid & 31;
        for (int r = tid >> 5; r < rows; r += NT / 32) {
          const long long rowc = row0 + (long long)r * n0;
          const int sr = r * TX;
          if (A.thread_cols & 1) copy_row<int8_t, TX>(A.cols.kind + rowc, reinterpret_cast<const int8_t*>(sbase + L::kind) + sr, cnt, lane);
          if (A.thread_cols & 2) copy_row<uint8_t, TX>(A.cols.amb + rowc, sbase + L::amb + sr, cnt, lane);
          if (A.thread_cols & 4) copy_row<T, TX>(static_cast<T*>(A.cols.vf) + rowc, reinterpret_cast<const T*>(sbase + L::vf) + sr, cnt, lane);
          if (A.thread_cols & 8) copy_row<T, 3 * TX>(static_cast<T*>(A.cols.c) + 3 * rowc, reinterpret_cast<const T*>(sbase + L::c) + 3 * sr, 3 * cnt, lane);
          if (A.thread_cols & 16) copy_row<T, 6 * TX>(static_cast<T*>(A.cols.ff) + 6 * rowc, reinterpret_cast<const T*>(sbase + L::ff) + 6 * sr, 6 * cnt, lane);
          if (A.thread_cols & 32) copy_row<T, 12 * TX>(static_cast<T*>(A.cols.fcl) + 12 * rowc, reinterpret_cast<const T*>(sbase + L::fcl) + 12 * sr, 12 * cnt, lane);
          if (A.thread_cols & 64) copy_row<T, 3 * TX>(static_cast<T*>(A.cols.ic) + 3 * rowc, reinterpret_cast<const T*>(sbase + L::ic) + 3 * sr, 3 * cnt, lane);
        }
      }
    }
  }
  if (fast && tid == 0) bulk_wait<0>();  // all tensor stores complete before the CTA retires
}

template <class T, bool SAMPLE, bool MX>
__global__ void __launch_bounds__(CUT_NT, sizeof(T) == 4 ? 5 : 3) mc_cut_kernel(const McArgs<T> A) {
  const long long n0 = A.g.n[0], n1 = A.g.n[1];
  const long long nx = n0 + 1, ny = n1 + 1;
  const T* phi = SAMPLE ? A.phi_out : A.phi_in;
  Stage<T> st;
  st.kind = A.cols.kind;
  st.amb = A.cols.amb;
  st.vf = static_cast<T*>(A.cols.vf);
  st.c = static_cast<T*>(A.cols.c);
  st.ff = static_cast<T*>(A.cols.ff);
  st.fcl = static_cast<T*>(A.cols.fcl);
  st.ic = static_cast<T*>(A.cols.ic);
  const T cs[3] = {A.g.d[0], A.g.d[1], A.g.d[2]};
  const unsigned total = *A.cut_count;
  for (unsigned q = blockIdx.x * CUT_NT + threadIdx.x; q < total; q += gridDim.x * CUT_NT) {
    const unsigned ci = A.cut_list[q];  // a cache has fewer than 2^32 cells: 32-bit quotients
    const unsigned row = ci / unsigned(n0), k = row / unsigned(n1);
    const unsigned i = ci - row * unsigned(n0), j = row - k * unsigned(n1);
    const long long b0 = i + nx * (j + ny * k);
    const long long bz = nx * ny;
    const T ph[8] = {phi[b0], phi[b0 + 1], phi[b0 + nx + 1], phi[b0 + nx],
                     phi[b0 + bz], phi[b0 + bz + 1], phi[b0 + bz + nx + 1], phi[b0 + bz + nx]};
    const T org[3] = {node_coord(A.g.x0[0], A.g.d[0], i), node_coord(A.g.x0[1], A.g.d[1], j),
                      node_coord(A.g.x0[2], A.g.d[2], k)};
    const T l[3] = {node_coord(A.g.x0[0], A.g.d[0], i + 1) - org[0], node_coord(A.g.x0[1], A.g.d[1], j + 1) - org[1],
                    node_coord(A.g.x0[2], A.g.d[2], k + 1) - org[2]};
    mc_cut_cell<T, MX>(ph, l, org, cs, A.tb, st, ci);
  }
}

template <class T>
constexpr int smem_bytes(int tape_bytes) {
  return Layout<T>::tape + ((tape_bytes + 15) / 16) * 16;
}

}  // namespace

namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// The column maps of a marching-cubes cache: bit c of the result is set when column c (kind,
// ambiguous, volume_fraction, centroid, face_fraction, face_centroid_local, interface_centroid) can
// be written by TMA tensor stores -- its base 16-byte aligned, its row pitch (x extent x bytes per
// cell) a multiple of 16 bytes, every dimension below 2^31. The CTA's threads copy the others.
template <class T>
int make_column_maps(const DevGrid<T>& g, const Cols& cols, ColumnMaps* maps) {
  using TL = Tile<T>;
  const long long n0 = g.n[0], n1 = g.n[1], n2 = g.n[2];
  if (12 * n0 >= 0x7fffffffLL || n1 >= 0x7fffffffLL || n2 >= 0x7fffffffLL) return 0;
  EncodeTiledFn enc = encode_fn();
  if (!enc) return 0;
  void* base[7] = {cols.kind, cols.amb, cols.vf, cols.c, cols.ff, cols.fcl, cols.ic};
  const CUtensorMapDataType tt = sizeof(T) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64;
  const cuuint64_t es = sizeof(T);
  const int width[7] = {1, 1, 1, 3, 6, 12, 3};
  int mask = 0;
  for (int c = 0; c < 7; ++c) {
    const CUtensorMapDataType dt = c < 2 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : tt;
    const cuuint64_t e = c < 2 ? 1 : es;
    const cuuint64_t w = width[c];
    if ((reinterpret_cast<uintptr_t>(base[c]) & 15u) || ((w * e * (cuuint64_t)n0) & 15u)) continue;
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r;
    if (c == 5) {
      const cuuint64_t dims[4] = {12, (cuuint64_t)n0, (cuuint64_t)n1, (cuuint64_t)n2};
      const cuuint64_t strides[3] = {12 * e, 12 * e * n0, 12 * e * n0 * n1};
      const cuuint32_t box[4] = {12, (cuuint32_t)TL::TX, (cuuint32_t)TL::TY, 1};
      r = enc(&maps->m[c], dt, 4, base[c], dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    } else {
      const cuuint64_t dims[3] = {w * n0, (cuuint64_t)n1, (cuuint64_t)n2};
      const cuuint64_t strides[2] = {w * e * n0, w * e * n0 * n1};
      const cuuint32_t box[3] = {(cuuint32_t)(w * TL::TX), (cuuint32_t)TL::TY, 1};
      r = enc(&maps->m[c], dt, 3, base[c], dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    }
    if (r == CUDA_SUCCESS) mask |= 1 << c;
  }
  return mask;
}

}  // namespace

namespace cci {

namespace {
constexpr long long DEFAULT_WAIT_LIMIT = 1ll << 22;  // mbarrier polls of the learned kernels' waits
long long g_wait_limit = DEFAULT_WAIT_LIMIT;
}  // namespace
long long set_wait_limit(long long polls) {
  const long long old = g_wait_limit;
  g_wait_limit = polls < 0 ? DEFAULT_WAIT_LIMIT : polls;
  return old;
}
long long wait_limit() { return g_wait_limit; }

namespace {
// SMs of the current device (read once per device).
long long device_sms() {
  static std::atomic<int> cache[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 148;
  std::atomic<int>* c = dev >= 0 && dev < 64 ? &cache[dev] : nullptr;
  int v = c ? c->load(std::memory_order_relaxed) : 0;
  if (v <= 0) {
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
    if (c) c->store(v, std::memory_order_relaxed);
  }
  return v;
}
}  // namespace

// Slices per fill pencil for an n0 x n1 x n2 grid. The CTAs are launched x-tile fastest and
// z-layer slowest, so every layer of pencils but the last is kz slices deep and the last is the
// remainder. Each candidate depth (kz + 1 a whole number of NS-slab sampling rounds) is scored by
// list-scheduling the launch on the resident CTAs (each pencil to the earliest free one, in launch
// order), a pencil taking its slices plus PENCIL_OVERHEAD slice-times (its tape load, first
// sampling round and last drain). Few waves of deep pencils leave SMs idle in the last wave: at
// 256^3, 31-slice pencils make 5.2 waves of the 444 resident CTAs; 27-slice pencils fill 5.8.
//
// The deepest candidate: CTAs drift apart in z by up to a pencil, and the further they do the more places each
// column is written in at once, which memory takes more slowly; a shallow pencil pays its first sampling
// round more often. Fill in us at most 31, 19, 15, 11 and 7 slices (CSG body; the field is given values):
//   Float32, all columns by TMA      512^3 2414 2423 2428 2451 2490    256^3 335 324 328 326 334    -> 19
//   Float32, some by the threads     500^3 2867 2593 2537 2548 2632    301 x 187 x 130 197 195 192 198 204    -> 15
//   Float64, all by TMA              512^3 4744 4397 4238 4090 4225    256^3 579 555 540 531 558
//                                    192 x 160 x 129 field 164 152 154 150 148    -> 11
//   Float64, some by the threads     404^3 2347 2379 2408 2463 2585    -> 31
//     (updates at most 31, 19 and 11: 301^3 1285 1296 1323, 203^3 437 441 442, 330 x 250 x 90 324 333 334)
int deepest_pencil(bool f64, bool all_tma) { return f64 ? (all_tma ? 11 : KZ) : (all_tma ? 19 : 15); }

int pencil_slices(long long n0, long long n1, long long n2, bool f64, int deepest) {
  const long long tx = f64 ? Tile<double>::TX : Tile<float>::TX, ty = Tile<float>::TY;
  const long long tiles = ((n0 + tx - 1) / tx) * ((n1 + ty - 1) / ty);
  const long long slots = device_sms() * (f64 ? Tile<double>::MINB : Tile<float>::MINB);
  constexpr double PENCIL_OVERHEAD = 2.0;
  int best = deepest;
  double best_t = 0;
  for (int kz = deepest; kz >= NS - 1; kz -= NS) {
    const long long layers = (n2 + kz - 1) / kz;
    const long long rem = n2 - (layers - 1) * kz;
    // groups of resident CTAs that become free at the same time: (time, count), times increasing
    double gt[8];
    long long gc[8];
    int ng = 1;
    gt[0] = 0;
    gc[0] = slots;
    double end = 0;
    const long long batch[2] = {tiles * (layers - 1), tiles};
    const double dur[2] = {kz + PENCIL_OVERHEAD, rem + PENCIL_OVERHEAD};
    for (int bi = 0; bi < 2; ++bi) {
      long long m = batch[bi];
      while (m > 0) {
        // the earliest group takes as many pencils as it has CTAs; they free up dur later
        const long long k = gc[0] < m ? gc[0] : m;
        const double t = gt[0] + dur[bi];
        end = t > end ? t : end;
        m -= k;
        if (k == gc[0]) {
          for (int q = 1; q < ng; ++q) { gt[q - 1] = gt[q]; gc[q - 1] = gc[q]; }
          --ng;
        } else {
          gc[0] -= k;
        }
        int q = 0;
        while (q < ng && gt[q] < t) ++q;
        if (q < ng && gt[q] == t) {
          gc[q] += k;
        } else if (ng < 8) {
          for (int r = ng; r > q; --r) { gt[r] = gt[r - 1]; gc[r] = gc[r - 1]; }
          gt[q] = t;
          gc[q] = k;
          ++ng;
        } else {
          gc[ng - 1] += k;  // out of groups: merge into the latest (a later free time, never earlier)
          gt[ng - 1] = t > gt[ng - 1] ? t : gt[ng - 1];
        }
      }
    }
    if (kz == deepest || end < best_t * 0.995) {  // a shallower pencil only for a clear gain
      best = kz;
      best_t = end;
    }
  }
  return best;
}

namespace {
// One fill launch. (4 CTAs per SM at Float32 was measured too: faster only while grids whose x
// extent is not a multiple of 16 still walked a per-row copy loop; without it 3 is faster at
// every size: 500^3 2.85 against 3.18 ms, 260^3 0.468 against 0.496.)
template <class T, bool SAMPLE, bool PRUNED>
cudaError_t launch_fill(const McArgs<T>& a, const ColumnMaps& maps, unsigned blocks, int sm, cudaStream_t s) {
  auto run = [&](auto kernel) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (e != cudaSuccess) return e;
    kernel<<<blocks, Tile<T>::NT, sm, s>>>(a, maps);
    return cudaSuccess;
  };
  if (a.tma_mask == 0x7f) return run(mc_fill_kernel<T, SAMPLE, PRUNED, true>);
  return run(mc_fill_kernel<T, SAMPLE, PRUNED, false>);
}
}  // namespace

template <class T>
cudaError_t launch_mc(const DevGrid<T>& g, const DevTape& tape, const T* phi_in, T* phi_out,
                      const Cols& cols, const DevTable& tb, unsigned* cut_list, unsigned* cut_count,
                      cudaStream_t s, bool mixed, bool count_zeroed) {
  using TL = Tile<T>;
  McArgs<T> a;
  a.g = g;
  a.tape = in_bounds_range(tape, g);
  a.phi_in = phi_in;
  a.phi_out = phi_out;
  a.cols = cols;
  a.tb = tb;
  a.cut_list = cut_list;
  a.cut_count = cut_count;
  ColumnMaps maps;
  std::memset(&maps, 0, sizeof maps);
  a.tma_mask = make_column_maps<T>(g, cols, &maps);
  a.byte_words = (g.n[0] % 4 == 0 && (reinterpret_cast<uintptr_t>(cols.kind) & 3u) == 0 &&
                  (reinterpret_cast<uintptr_t>(cols.amb) & 3u) == 0) ? 1 : 0;
  a.thread_cols = ~a.tma_mask & 0x7f & ~(a.byte_words ? 3 : 0);
  a.n_itiles = int((g.n[0] + TL::TX - 1) / TL::TX);
  a.n_jtiles = int((g.n[1] + TL::TY - 1) / TL::TY);
  a.kz = pencil_slices(g.n[0], g.n[1], g.n[2], sizeof(T) == 8, deepest_pencil(sizeof(T) == 8, a.tma_mask == 0x7f));
  const long long nk = (g.n[2] + a.kz - 1) / a.kz;
  const long long blocks = (long long)a.n_itiles * a.n_jtiles * nk;
  if (blocks <= 0 || blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  cudaError_t e = count_zeroed ? cudaSuccess : cudaMemsetAsync(cut_count, 0, sizeof(unsigned), s);
  if (e != cudaSuccess) return e;
  const bool sample = phi_in == nullptr;
  const bool pruned = sample && a.tape.prunable;
  int sm = smem_bytes<T>(sample ? tape.bytes_len : 0);
  if (pruned) sm += tape.n_ops * int(sizeof(cc_op) + sizeof(unsigned));
  const int cut_blocks = 148 * 16;
  // the FP64 islands of mixed precision exist for Float32 caches only
  const bool mx = mixed && sizeof(T) == 4;
  if (pruned) {
    e = launch_fill<T, true, true>(a, maps, unsigned(blocks), sm, s);
    if (e != cudaSuccess) return e;
    if (mx) mc_cut_kernel<T, true, true><<<cut_blocks, CUT_NT, 0, s>>>(a);
    else mc_cut_kernel<T, true, false><<<cut_blocks, CUT_NT, 0, s>>>(a);
  } else if (sample) {
    e = launch_fill<T, true, false>(a, maps, unsigned(blocks), sm, s);
    if (e != cudaSuccess) return e;
    if (mx) mc_cut_kernel<T, true, true><<<cut_blocks, CUT_NT, 0, s>>>(a);
    else mc_cut_kernel<T, true, false><<<cut_blocks, CUT_NT, 0, s>>>(a);
  } else {
    e = launch_fill<T, false, false>(a, maps, unsigned(blocks), sm, s);
    if (e != cudaSuccess) return e;
    if (mx) mc_cut_kernel<T, false, true><<<cut_blocks, CUT_NT, 0, s>>>(a);
    else mc_cut_kernel<T, false, false><<<cut_blocks, CUT_NT, 0, s>>>(a);
  }
  return cudaGetLastError();
}

template cudaError_t launch_mc<float>(const DevGrid<float>&, const DevTape&, const float*, float*,
                                      const Cols&, const DevTable&, unsigned*, unsigned*, cudaStream_t, bool, bool);
template cudaError_t launch_mc<double>(const DevGrid<double>&, const DevTape&, const double*, double*,
                                       const Cols&, const DevTable&, unsigned*, unsigned*, cudaStream_t, bool, bool);

}  // namespace cci
