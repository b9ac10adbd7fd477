// The slabs of the FP64 steps in passes: their boxes, the arrays of their
// workspace and the offsets in them.  Plain C++ with CUDA qualifiers where a
// CUDA compiler reads it, so the host tests can check the arithmetic at sizes
// no test runs.
#pragma once

#ifdef __CUDACC__
#define EK_SLAB_HD __host__ __device__ __forceinline__
#else
#define EK_SLAB_HD inline
#endif

namespace ekc
{

// One hydro slab: the interior cells [j0, j0 + ny) in 2D, [k0, k0 + nz) in 3D, and
// its part of the workspace.  Arrays are [..][variable][cells of the box], x
// fastest; a box is the slab's cells with 2 (q), 1 (s) or 0 (f, one more on the
// high side) layers around.
template <int NV>
struct HydroSlab
{
  static constexpr int DIM = NV == 4 ? 2 : 3;
  int       nx, ny, nz, j0, k0;
  int       last; // the step's last slab
  double *  q;    // primitives
  double *  s;    // face states [axis][low, high]
  double *  f;    // fluxes through the low faces [axis]
  EK_SLAB_HD long long
  box(int w) const // cells of a box with w more cells per axis
  {
    return (long long)(nx + w) * (ny + w) * (DIM == 3 ? nz + w : 1);
  }
  EK_SLAB_HD long long
  bytes() const
  {
    return (long long)sizeof(double) * NV * (box(4) + 2 * DIM * box(2) + DIM * box(1));
  }
};

// Field f of arrays with one field after another; the stride's type is that of
// the product: int for a tile's planes in shared memory, 64 bits for a slab's
// (47 fields of a plane of 4000 x 4000 pass 2^31).
template <class I>
EK_SLAB_HD I
field_offset(int f, I stride)
{
  return (I)f * stride;
}

// The MHD arrays of the whole grid, indexed as the state is ([variable][k][j][i]
// with ghosts), and one slab: interior cells [j0, j0 + ny) in 2D, [k0, k0 + nz) in 3D.
template <int DIM>
struct MhdSlab
{
  static constexpr int NE = DIM == 3 ? 3 : 1;   // edge fields (2D: z only, the last)
  static constexpr int NT = DIM == 3 ? 47 : 30; // trace fields
  static constexpr int NF = DIM == 3 ? 5 : 6;   // flux components
  int       nx, ny, nz, j0, k0;
  int       last;
  double *  q;  // [8] primitives
  double *  b;  // [3] face fields
  double *  e;  // [NE] edge fields
  double *  t;  // [NT] trace of the box with one more cell on every side
  double *  f;  // [DIM][NF] fluxes through the low faces, box with one more on the high side
  double *  em; // [NE] emfs of the low edges, the same box
  EK_SLAB_HD long long
  box(int w) const
  {
    return (long long)(nx + w) * (ny + w) * (DIM == 3 ? nz + w : 1);
  }
  EK_SLAB_HD long long
  trace_stride() const
  {
    return box(2);
  }
  EK_SLAB_HD long long
  slab_bytes() const
  {
    return (long long)sizeof(double) * (NT * box(2) + (DIM * NF + NE) * box(1));
  }
  // of the slab's boxes: trace cell and low face / edge of cell (i, j, k)
  EK_SLAB_HD long long
  tcell(int i, int j, int k) const
  {
    return ((DIM == 3 ? k + 1 : 0) * (long long)(ny + 2) + (j + 1)) * (nx + 2) + (i + 1);
  }
  EK_SLAB_HD long long
  face(int i, int j, int k) const
  {
    return ((DIM == 3 ? k : 0) * (long long)(ny + 1) + j) * (nx + 1) + i;
  }
};

// Cells of the last axis, N in all, per slab: the fewest slabs whose workspace,
// bytes(cells), is at most `limit` (one cell's may be more), about equal
template <class Bytes>
inline int
slab_cells(int N, long long limit, Bytes bytes)
{
  int n = N;
  for (int slabs = 2; n > 1 && bytes(n) > limit; ++slabs)
    n = (int)(((long long)N + slabs - 1) / slabs);
  return n;
}

// A workspace for slabs of n cells or, when it cannot be had, fewer: try_alloc is
// called with the bytes and tells whether it was.  The cells it holds, 0 for none.
template <class Bytes, class Try>
inline int
place_slab(int n, Bytes bytes, Try try_alloc)
{
  for (; n > 0; n = n > 1 ? (n + 1) / 2 : 0)
    if (try_alloc(bytes(n)))
      return n;
  return 0;
}

} // namespace ekc
