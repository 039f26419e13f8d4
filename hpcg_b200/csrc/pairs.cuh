// pairs.cuh -- index arithmetic of the row-pair kernels (SpMV and the sweeps),
// for the device and for a host program that checks it.
//
// A thread has the two rows (2i, 2i+1) of an x-line.  On each of the 9 stencil
// lines (dy, dz) both rows read x[2i-1 .. 2i+2] between them, so a pair gathers
// 9 x 4 entries with 27 loads (two entries in one vector load) instead of 54,
// from 9 line addresses instead of 54.
#pragma once
#include "common.cuh"

namespace hpcgx {

struct PairId {
  int64_t row;      // natural index of the even row
  int64_t ke, ko;   // storage rows
  int ix, iy, iz;   // of the even row
  int pos;          // pair inside its line
  bool left, odd, right;   // x-neighbours of the even row at -1, +1, +2 exist
  bool ym, yp, zm, zp;     // the lines below / above exist
};

// Pair t of the lines [j0, ...) of a class.
template <class VT>
__host__ __device__ __forceinline__ PairId pair_at(const LevelMat<VT> &A, const ClassInfo &C,
                                                   int j0, int t) {
  PairId id;
  const int Le = C.len[0];
  const int jl = (int)fdiv((uint32_t)t, C.dlen);
  id.pos = t - jl * Le;
  const int j = j0 + jl;
  const int jz = (int)fdiv((uint32_t)j, C.dnyq);
  id.iy = C.py + 2 * (j - jz * C.nyq);
  id.iz = C.pz + 2 * jz;
  id.ix = 2 * id.pos;
  id.row = ((int64_t)id.iz * A.ny + id.iy) * A.nx + id.ix;
  id.ke = C.start[0] + (int64_t)j * Le + id.pos;
  id.ko = C.start[1] + (int64_t)j * C.len[1] + id.pos;
  id.left = id.pos > 0;
  id.odd = id.pos < C.len[1];
  id.right = id.pos + 1 < Le;
  id.ym = id.iy > 0;
  id.yp = id.iy + 1 < A.ny;
  id.zm = id.iz > 0 || A.zlo;
  id.zp = id.iz + 1 < A.nz || A.zhi;
  if (!id.odd) id.ko = id.ke;
  return id;
}

// Stencil line l = (dz+1)*3 + (dy+1): does it exist for the pair's rows?
__host__ __device__ __forceinline__ bool has_line(const PairId &id, int l) {
  const int dy = l % 3 - 1, dz = l / 3 - 1;
  return (dy < 0 ? id.ym : dy > 0 ? id.yp : true) && (dz < 0 ? id.zm : dz > 0 ? id.zp : true);
}

// ---- the index-checked build

// The vector rows and storage rows of the pair lie in their arrays, the
// x-neighbours on its own line too (the sweeps read those without load_line).
template <class VT>
__host__ __device__ __forceinline__ bool pair_inside(const LevelMat<VT> &A, const PairId &id) {
  const int64_t first = id.row - (id.left ? 1 : 0), last = id.row + (id.right ? 2 : id.odd ? 1 : 0);
  return first >= 0 && last < A.n && id.ke >= 0 && id.ke < A.srows && id.ko >= 0 && id.ko < A.srows;
}

// What a pair outside them is replaced by: row 0 without neighbours on its line.
// It keeps the evenness that a vector access wants; such an access reads and
// writes row 1 as well, which exists wherever lines of even length allow it.
__host__ __device__ __forceinline__ void redirect(PairId &id) {
  id.row = id.ke = id.ko = 0;
  id.left = id.odd = id.right = false;
}

// Every entry that the pair's load of line l reads lies in the vector, its halo
// planes included.
template <class VT>
__host__ __device__ __forceinline__ bool line_inside(const LevelMat<VT> &A, const PairId &id,
                                                     bool vec, int l) {
  const int64_t at = id.row + A.off[3 * l + 1];
  const int64_t first = at - (id.left ? 1 : 0), last = at + (id.right ? 2 : id.odd || vec ? 1 : 0);
  return first >= A.lo && last < (int64_t)A.lo + A.span && !(vec && (at & 1));
}

}  // namespace hpcgx
