// kernels.cu -- the sm_100a kernels of libhpcgx.
//
// All kernels are HBM-bandwidth bound (no step of HPCG's PCG iteration is a
// dense contraction, so nothing here uses tensor cores).  The design points:
//   * stencil rows are walked by x-line classes (fixed iy&1, iz&1), two rows
//     (2i, 2i+1) per thread from one set of loads;
//   * a Gauss-Seidel half sweep is ONE launch per class: the two colours of a
//     class only depend on each other along x inside a line, so a CTA that owns
//     whole lines takes both with a __syncthreads between them; the last class's
//     forward and backward half sweeps are one launch too, so a symmetric sweep
//     is 7 launches instead of 16;
//   * launches depend on one another programmatically: a kernel starts under the
//     end of the one before it and waits before it reads a vector;
//   * restriction (src/ComputeRestriction_ref.cpp:51) is fused into the last
//     colour of the pre-smoother's backward sweep and prolongation
//     (src/ComputeProlongation_ref.cpp:49) into the first colour of the
//     post-smoother's forward sweep: the injected points are exactly colour 0;
//   * the first forward sweep of ComputeMG starts from x = 0
//     (src/ComputeMG_ref.cpp:42) and skips every term that multiplies a zero;
//   * reductions are deterministic: fixed per-block partials, then the last
//     block to finish sums them in index order and applies the CG scalar
//     update, so alpha/beta never leave the device.
#include "kernels.cuh"
#include "pairs.cuh"

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <type_traits>

namespace hpcgx {

namespace {

constexpr int kThreads = 256;

// ---------------------------------------------------------------- reductions

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

template <bool MAX>
__device__ __forceinline__ double warp_red(double v) {
  return MAX ? warp_max(v) : warp_sum(v);
}

// Sums (or maxes) `count` partials p[0], p[stride], ... over the block in a
// fixed order (strided per thread, warp tree, warps in order); the result is
// valid in every thread.
template <int NV, bool MAX>
__device__ void block_sum_partials(const double *p, int64_t count, int64_t stride,
                                   double (&out)[NV], double (&sh)[NV][32]) {
  __shared__ double res[NV];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    double t = 0.0;
    for (int64_t b = threadIdx.x; b < count; b += blockDim.x) {
      const double q = __ldcg(p + (int64_t)i * stride + b);
      t = MAX ? fmax(t, q) : t + q;
    }
    t = warp_red<MAX>(t);
    __syncthreads();
    if (lane == 0) sh[i][wid] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
      double s = 0.0;
      for (int w = 0; w < nw; ++w) s = MAX ? fmax(s, sh[i][w]) : s + sh[i][w];
      res[i] = s;
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < NV; ++i) out[i] = res[i];
}

// Reduces NV values over the block and publishes one partial per block; the
// last block to arrive returns true with the totals in tot (valid in every
// thread of that block).  Up to kReduceGroup blocks the last block sums the
// partials in block order.  Larger grids (the SpMV's one block per line
// group) reduce in two levels so that no counter takes more than
// kReduceGroup atomics and no block reads more than that many partials: the
// last block of each group of kReduceGroup sums its group's partials in block
// order, and the last group sums the group totals in group order.
// Deterministic for a fixed grid size either way.
constexpr int kReduceGroup = 1024;
template <int NV, bool MAX = false>
__device__ bool grid_reduce(double (&v)[NV], const Reduce &red, double (&tot)[NV]) {
  __shared__ double sh[NV][32];
  __shared__ int amlast;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  const int64_t G = gridDim.x;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    double t = warp_red<MAX>(v[i]);
    if (lane == 0) sh[i][wid] = t;
  }
  __syncthreads();
  const int64_t ngroups = (G + kReduceGroup - 1) / kReduceGroup;
  const int64_t group = blockIdx.x / kReduceGroup;
  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      double t = 0.0;
      for (int w = 0; w < nw; ++w) t = MAX ? fmax(t, sh[i][w]) : t + sh[i][w];
      red.partials[(int64_t)i * G + blockIdx.x] = t;
    }
    __threadfence();
    const int64_t gsize = ngroups == 1 ? G : min((int64_t)kReduceGroup, G - group * kReduceGroup);
    unsigned int *ctr = ngroups == 1 ? red.counter : red.counter + 1 + group;
    const unsigned int prev = atomicAdd(ctr, 1u);
    amlast = (prev == gsize - 1);
  }
  __syncthreads();
  if (!amlast) return false;
  __threadfence();
  if (ngroups == 1) {
    block_sum_partials<NV, MAX>(red.partials, G, G, tot, sh);
    if (threadIdx.x == 0) *red.counter = 0u;
    return true;
  }
  // last block of its group: the group's total, then the group-level count
  const int64_t base = group * kReduceGroup;
  const int64_t gsize = min((int64_t)kReduceGroup, G - base);
  double gt[NV];
  block_sum_partials<NV, MAX>(red.partials + base, gsize, G, gt, sh);
  double *gp = red.partials + (int64_t)NV * G;   // group totals
  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) gp[(int64_t)i * ngroups + group] = gt[i];
    red.counter[1 + group] = 0u;
    __threadfence();
    const unsigned int prev = atomicAdd(red.counter, 1u);
    amlast = (prev == ngroups - 1);
  }
  __syncthreads();
  if (!amlast) return false;
  __threadfence();
  block_sum_partials<NV, MAX>(gp, ngroups, ngroups, tot, sh);
  if (threadIdx.x == 0) *red.counter = 0u;
  return true;
}

// The scalar step that follows a reduction (done by one thread of the last
// block).  The formulas are CG's (src/CG.cpp:93-124).
template <int NV>
__device__ void finish(int fin, void *target, const double (&tot)[NV]) {
  if (fin == FIN_STORE || fin == FIN_MAX) {
    double *o = static_cast<double *>(target);
    for (int i = 0; i < NV; ++i) o[i] = tot[i];
    return;
  }
  CgState *st = static_cast<CgState *>(target);
  switch (fin) {
    case FIN_CG_INIT:
      st->normr = sqrt(tot[0]);
      st->normr0 = st->normr;
      st->k = 1;
      st->niters = 0;
      st->nonfinite = !isfinite(st->normr);
      st->done = !(st->normr / st->normr0 > st->tol) || st->max_iter < 1 || st->nonfinite;
      // a solve that is done here has no iteration that would leave its state
      if (st->mirror) st->mirror[0] = st->mirror[1] = *st;
      break;
    case FIN_CG_RZ:
      if (st->k == 1) {
        st->rtz = tot[0];
      } else {
        st->oldrtz = st->rtz;
        st->rtz = tot[0];
        if (st->flexible) {
          st->zAp = tot[NV > 1 ? 1 : 0];
          st->beta = -st->zAp / st->pAp;
        } else {
          st->beta = st->rtz / st->oldrtz;
        }
      }
      break;
    case FIN_CG_PAP:
      st->pAp = tot[0];
      st->alpha = st->rtz / st->pAp;
      break;
    case FIN_CG_RR:
      st->normr = sqrt(tot[0]);
      st->niters = st->k;
      st->k += 1;
      st->nonfinite = !isfinite(st->normr);
      st->done = !(st->normr / st->normr0 > st->tol) || st->k > st->max_iter || st->nonfinite;
      if (st->mirror) st->mirror[st->niters & 1] = *st;
      break;
    default:
      break;
  }
}

// Applies the scalar step, or (sharded solve) stores this rank's totals for
// the sum over the ranks that precedes it.
template <int NV>
__device__ void finish_or_defer(const Reduce &red, int fin, void *target, const double (&tot)[NV]) {
  if (red.defer) {
    for (int i = 0; i < NV; ++i) red.defer[i] = tot[i];
    return;
  }
  finish<NV>(fin, target, tot);
}

template <int NV>
__global__ void k_finish(int fin, const double *__restrict__ tot, CgState *st) {
  double t[NV];
  for (int i = 0; i < NV; ++i) t[i] = tot[i];
  finish<NV>(fin, st, t);
}

// Sum over the ranks of an in-process group, in rank order, written back to
// every rank's buffer.
__global__ void k_rank_sum(int nranks, double *const *bufs, int count) {
  for (int i = threadIdx.x; i < count; i += blockDim.x) {
    double s = 0.0;
    for (int r = 0; r < nranks; ++r) s += bufs[r][i];
    for (int r = 0; r < nranks; ++r) bufs[r][i] = s;
  }
}

// ---------------------------------------------------------------- index checks

// Built with -DHPCGX_CHECKED (libhpcgx_checked.so), the row kernels verify
// every storage row, vector row and gathered column before using it.  The first
// bad one is recorded (as site << 56 | index).  A bad row is replaced by index 0,
// which is always inside the buffers and on every vector access's boundary, and
// a stencil line with a bad column is not read, so nothing outside the buffers
// is touched.
// hpcgx_check_status() reports and clears the record.  The stand-in for a
// memory checker; without the macro the checks compile to nothing.
#ifdef HPCGX_CHECKED
__device__ unsigned long long g_check_record = 0ull;
__device__ __noinline__ void check_fail(int site, int64_t index) {
  atomicCAS(&g_check_record, 0ull,
            ((unsigned long long)site << 56) | ((unsigned long long)index & ((1ull << 56) - 1)));
}
#endif

struct RowId;
template <class VT>
__device__ __forceinline__ void check_row(const LevelMat<VT> &A, RowId &id, int site);
template <class VT, class NEED>
__device__ __forceinline__ void check_cols(const LevelMat<VT> &A, int32_t *col, NEED need,
                                           int site);
__device__ __forceinline__ int64_t check_index(int64_t i, int64_t n, int site) {
#ifdef HPCGX_CHECKED
  if (i < 0 || i >= n) {
    check_fail(site, i);
    return 0;
  }
#endif
  return i;
}

// ---------------------------------------------------------------- geometry

struct ClassSet {
  ClassInfo c[4];
  int nblk[4];     // blocks of each class
  int turns;       // groups of 256 pairs a block takes
  int common;      // min over the classes of nblk
  int total;       // sum of nblk: the grid
};

// Block g of a launch over all four classes -> (class, block inside the
// class).  The classes are interleaved round-robin (block b of class q is
// launch block 4 b + q) so that the four classes walk up the z-planes
// together and a plane of x is still in L2 when the next class reads it;
// blocks beyond the smallest class's count follow class by class.
__device__ __forceinline__ void class_block(const ClassSet &cs, int g, int &q, int &b) {
  if (g < 4 * cs.common) {
    q = g & 3;
    b = g >> 2;
    return;
  }
  g -= 4 * cs.common;
  q = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int extra = cs.nblk[q] - cs.common;
    if (g < extra) break;
    g -= extra;
    ++q;
  }
  b = cs.common + g;
}

// Row handled by thread-slot t of half px in a block that owns lines [j0, ...).
struct RowId {
  int64_t row;   // natural index
  int64_t k;     // storage row
  int ix, iy, iz;
};

template <class VT>
__device__ __forceinline__ void check_row(const LevelMat<VT> &A, RowId &id, int site) {
#ifdef HPCGX_CHECKED
  if (id.row < 0 || id.row >= A.n) {
    check_fail(site, id.row);
    id.row = 0;
  }
  if (id.k < 0 || id.k >= A.srows) {
    check_fail(site, id.k);
    id.k = 0;
  }
#endif
}

template <class VT, class NEED>
__device__ __forceinline__ void check_cols(const LevelMat<VT> &A, int32_t *col, NEED need,
                                           int site) {
#ifdef HPCGX_CHECKED
#pragma unroll
  for (int s = 0; s < HPCGX_STENCIL; ++s)
    if (need(s) && (uint32_t)(col[s] - A.lo) >= (uint32_t)A.span) {
      check_fail(site, col[s]);
      col[s] = 0;
    }
#endif
}

// ---------------------------------------------------------------- row loads

// Vector loads of one stencil z-plane (9 slots) of storage row k; a group is
// loaded only if need(s) holds for one of its slots (need folds to a
// constant in every kernel, so skipped groups cost nothing).
template <class NEED>
__device__ __forceinline__ void load_plane(const double *__restrict__ vals, int64_t k, int p,
                                           NEED need, double *v) {
  const double *q = vals + (k >> 5) * kSliceElems + p * kPlaneElems;
  const int lane = (int)(k & 31);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (need(9 * p + 2 * j) || need(9 * p + 2 * j + 1)) {
      const double2 t = __ldg(reinterpret_cast<const double2 *>(q + j * 64 + lane * 2));
      v[2 * j] = t.x;
      v[2 * j + 1] = t.y;
    }
  }
  if (need(9 * p + 8)) v[8] = __ldg(q + 256 + lane);
}

// BF16 values of one z-plane straight to FP32 (a BF16 pattern is the high
// half of the FP32 pattern of the same number).
template <class NEED>
__device__ __forceinline__ void load_plane_f32(const uint16_t *__restrict__ vals, int64_t k, int p,
                                               NEED need, float *v) {
  const uint16_t *q = vals + (k >> 5) * kSliceElems + p * kPlaneElems;
  const int lane = (int)(k & 31);
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    if (need(9 * p + 4 * j) || need(9 * p + 4 * j + 1) || need(9 * p + 4 * j + 2) ||
        need(9 * p + 4 * j + 3)) {
      const uint2 t = __ldg(reinterpret_cast<const uint2 *>(q + j * 128 + lane * 4));
      v[4 * j] = __uint_as_float(t.x << 16);
      v[4 * j + 1] = __uint_as_float(t.x & 0xffff0000u);
      v[4 * j + 2] = __uint_as_float(t.y << 16);
      v[4 * j + 3] = __uint_as_float(t.y & 0xffff0000u);
    }
  }
  if (need(9 * p + 8)) v[8] = __uint_as_float((uint32_t)__ldg(q + 256 + lane) << 16);
}
template <class NEED>
__device__ __forceinline__ void load_vals(const double *__restrict__ vals, int64_t k, int p,
                                          NEED need, double *v) {
  load_plane(vals, k, p, need, v);
}
template <class NEED>
__device__ __forceinline__ void load_vals(const uint16_t *__restrict__ vals, int64_t k, int p,
                                          NEED need, float *v) {
  load_plane_f32(vals, k, p, need, v);
}

// The values of one row in registers: FP64 as they are; BF16 packed as loaded
// (15 registers a row instead of 27) and widened where they are used.
template <class VT>
struct RowVals;
template <>
struct RowVals<double> {
  double v[HPCGX_STENCIL];
  template <class NEED>
  __device__ __forceinline__ void load(const double *vals, int64_t k, int p, NEED need) {
    load_plane(vals, k, p, need, v + 9 * p);
  }
  __device__ __forceinline__ double get(int s) const { return v[s]; }
};
template <>
struct RowVals<uint16_t> {
  uint2 q[6];
  uint32_t one[3];
  template <class NEED>
  __device__ __forceinline__ void load(const uint16_t *vals, int64_t k, int p, NEED need) {
    const uint16_t *w = vals + (k >> 5) * kSliceElems + p * kPlaneElems;
    const int lane = (int)(k & 31);
#pragma unroll
    for (int j = 0; j < 2; ++j)
      if (need(9 * p + 4 * j) || need(9 * p + 4 * j + 1) || need(9 * p + 4 * j + 2) ||
          need(9 * p + 4 * j + 3))
        q[2 * p + j] = __ldg(reinterpret_cast<const uint2 *>(w + j * 128 + lane * 4));
    if (need(9 * p + 8)) one[p] = __ldg(w + 256 + lane);
  }
  // a BF16 pattern is the high half of the FP32 pattern of the same number
  __device__ __forceinline__ float get(int s) const {
    const int p = s / 9, i = s % 9;
    if (i == 8) return __uint_as_float(one[p] << 16);
    const uint2 t = q[2 * p + i / 4];
    const uint32_t w = (i % 4) < 2 ? t.x : t.y;
    return (i & 1) ? __uint_as_float(w & 0xffff0000u) : __uint_as_float(w << 16);
  }
};

struct NeedAll {
  __device__ constexpr bool operator()(int) const { return true; }
};

// ---------------------------------------------------------------- columns

// Columns of storage row id: row + off[s] where that neighbour exists (in
// 32-bit arithmetic: vectors hold fewer than 2^31 rows), the row itself
// elsewhere and for a left-out entry, so that the product with the slot's 0
// reads nothing the row does not read anyway.
template <class VT>
__device__ __forceinline__ void stencil_cols(const LevelMat<VT> &A, const RowId &id, int32_t *col) {
  const int r32 = (int)id.row;
  const uint32_t out = A.left_out ? A.left_out[id.k] : 0u;
  const bool xm = id.ix > 0, xp = id.ix + 1 < A.nx, ym = id.iy > 0, yp = id.iy + 1 < A.ny,
             zm = id.iz > 0 || A.zlo, zp = id.iz + 1 < A.nz || A.zhi;
#pragma unroll
  for (int s = 0; s < HPCGX_STENCIL; ++s) {
    const int dx = s % 3 - 1, dy = (s / 3) % 3 - 1, dz = s / 9 - 1;
    const bool nb = (dx < 0 ? xm : dx > 0 ? xp : true) && (dy < 0 ? ym : dy > 0 ? yp : true) &&
                    (dz < 0 ? zm : dz > 0 ? zp : true) && !(out >> s & 1u);
    col[s] = nb ? r32 + A.off[s] : r32;
  }
}

// ---------------------------------------------------------------- row pairs

template <class VT>
__device__ __forceinline__ PairId pair_of(const LevelMat<VT> &A, const ClassInfo &C, int j0, int t,
                                          int site) {
  PairId id = pair_at(A, C, j0, t);
#ifdef HPCGX_CHECKED
  if (!pair_inside(A, id)) {
    check_fail(site, id.row);
    redirect(id);
  }
#endif
  return id;
}

__device__ __forceinline__ void load2(const double *p, double &u, double &v) {
  const double2 t = *reinterpret_cast<const double2 *>(p);
  u = t.x;
  v = t.y;
}
__device__ __forceinline__ void load2(const float *p, float &u, float &v) {
  const float2 t = *reinterpret_cast<const float2 *>(p);
  u = t.x;
  v = t.y;
}
__device__ __forceinline__ void store2(double *p, double u, double v) {
  *reinterpret_cast<double2 *>(p) = make_double2(u, v);
}
__device__ __forceinline__ void store2(float *p, float u, float v) {
  *reinterpret_cast<float2 *>(p) = make_float2(u, v);
}

// x[2i-1 .. 2i+2] on line l into v[0..3]; what does not exist reads as 0, the value its slots hold, so that the product drops out whatever
// x holds elsewhere.  vec: the two middle entries with one load (x and nx allow it).
template <class VT, class T>
__device__ __forceinline__ void load_line(const LevelMat<VT> &A, const PairId &id, const T *xr,
                                          int l, bool vec, T *v, int site) {
  bool ok = has_line(id, l);
  const T *q = xr + A.off[3 * l + 1];
#ifdef HPCGX_CHECKED
  if (ok && !line_inside(A, id, vec, l)) {
    check_fail(site, id.row + A.off[3 * l + 1]);
    ok = false;
  }
#endif
  v[0] = v[1] = v[2] = v[3] = T(0);
  if (ok && id.left) v[0] = q[-1];
  if (vec) {
    if (ok) load2(q, v[1], v[2]);
  } else {
    if (ok) v[1] = q[0];
    if (ok && id.odd) v[2] = q[1];
  }
  if (ok && id.right) v[3] = q[2];
}

// Slot s of a row sum.  out: the row's left-out entries (LevelMat::left_out),
// which add nothing whatever their neighbour holds; a stored zero multiplies it.
template <class T>
__device__ __forceinline__ T term_add(uint32_t out, int s, T sum, T v, T x) {
  return out >> s & 1u ? sum : mac_add(sum, v, x);
}
template <class T>
__device__ __forceinline__ T term_sub(uint32_t out, int s, T sum, T v, T x) {
  return out >> s & 1u ? sum : mac_sub(sum, v, x);
}

// ---------------------------------------------------------------- SpMV

// y = A x, rows summed left to right over the slots as ComputeSPMV_ref does
// (src/ComputeSPMV_ref.cpp:64-70).  With DOT, also reduces sum_i x_i y_i (the
// p.Ap of CG, src/CG.cpp:119) and runs the finishing scalar step (DOT_FUSED) or
// leaves a partial sum per block for k_sum_partials (DOT_PARTS, see
// kDotLaunchRows).  A block takes 256 consecutive pairs of one class (DOT_PARTS:
// cs.turns times as many), whatever lines they lie on (rows have no order to
// keep), so no thread idles on ragged lines; the classes are interleaved block by
// block (class_block).  HBM bounds it: 8 B per nonzero and 16 B per row at 256^3
// is 3.86 GB, 568 us = 6.8 TB/s, 1.04 of the measured copy rate (one row per
// thread and stored int32 columns: 824 us, and with derived columns, as the mixed
// solver had it: 596; 104^3: 59 against 78 us).  FP64 holds a z-plane's 18 values
// and 12 entries per step (128 registers, two blocks per SM); one and three blocks
// measured the same.
// The forms of the row-pair kernels.  FORM_WIDE: every vector starts on a
// two-element boundary and lines are even, so that two entries go with one
// access.  FORM_SCALAR: neither is sure.  FORM_HOLES: a matrix with left-out
// entries (LevelMat::left_out), vectors of either kind.
enum Form { FORM_WIDE = 0, FORM_SCALAR = 1, FORM_HOLES = 2 };
template <int FORM>
__device__ __forceinline__ bool is_wide(int vec) {
  return FORM == FORM_WIDE || (FORM == FORM_HOLES && vec);
}

enum SpmvDot { DOT_NONE = 0, DOT_FUSED = 1, DOT_PARTS = 2 };
template <class VT, class T, int DOT, int FORM>
__global__ void __launch_bounds__(kThreads, std::is_same<VT, double>::value ? 2 : 4)
k_spmv(const __grid_constant__ LevelMat<VT> A, const __grid_constant__ ClassSet cs, const T *x,
       T *y, int wide, Reduce red, int fin, void *fin_target, const int *done) {
  dependents_launch();
  const bool vec = is_wide<FORM>(wide);
  int q, b;
  class_block(cs, (int)blockIdx.x, q, b);
  const ClassInfo &C = cs.c[q];
  double acc = 0.0;
  const int turns = DOT == DOT_PARTS ? cs.turns : 1;
#pragma unroll 1
  for (int turn = 0; turn < turns; ++turn) {
    const int t = (b * turns + turn) * kThreads + (int)threadIdx.x;
    const bool act = t < C.lines * C.len[0];
    PairId id;
    T ve[9], vo[9];
    uint32_t oe = 0u, oo = 0u;   // left-out entries of the two rows
    if (act) {
      id = pair_of(A, C, 0, t, 1);
      if (FORM == FORM_HOLES && A.left_out) {
        oe = A.left_out[id.ke];
        oo = A.left_out[id.ko];
      }
      load_vals(A.vals, id.ke, 0, NeedAll(), ve);
      load_vals(A.vals, id.ko, 0, NeedAll(), vo);
    }
    if (turn == 0) {
      dependency_wait();
      if (done && *done) return;
    }
    if (act) {
      const T *xr = x + id.row;
      T se = T(0), so = T(0), xe = T(0), xo = T(0);
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        T v[3][4];
        if (p > 0) {
          load_vals(A.vals, id.ke, p, NeedAll(), ve);
          load_vals(A.vals, id.ko, p, NeedAll(), vo);
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) load_line(A, id, xr, 3 * p + i, vec, v[i], 2);
#pragma unroll
        for (int s = 0; s < 9; ++s) {
          se = term_add(oe, 9 * p + s, se, ve[s], v[s / 3][s % 3]);
          so = term_add(oo, 9 * p + s, so, vo[s], v[s / 3][s % 3 + 1]);
        }
        if (p == 1) {
          xe = v[1][1];
          xo = v[1][2];
        }
      }
      if (vec && id.odd) {
        store2(y + id.row, se, so);
      } else {
        y[id.row] = se;
        if (id.odd) y[id.row + 1] = so;
      }
      if (DOT) {
        acc += (double)xe * (double)se;
        if (id.odd) acc += (double)xo * (double)so;
      }
    }
  }
  if (DOT == DOT_FUSED) {
    double v[1] = {acc}, tot[1];
    if (grid_reduce<1>(v, red, tot) && threadIdx.x == 0)
      finish_or_defer<1>(red, fin, fin_target, tot);
  }
  if (DOT == DOT_PARTS) {
    __shared__ double sh[kThreads / 32];
    const double w = warp_red<false>(acc);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = w;
    __syncthreads();
    if (threadIdx.x == 0) {
      double sum = 0.0;
      for (int i = 0; i < kThreads / 32; ++i) sum += sh[i];
      red.partials[blockIdx.x] = sum;
    }
  }
}

// The sum of the n partials p of a launch with DOT_PARTS, kReduceGroup of them a
// block, and its scalar step.
__global__ void __launch_bounds__(kThreads)
k_sum_partials(const double *p, int64_t n, Reduce red, int fin, void *target, const int *done) {
  dependents_launch();
  dependency_wait();
  if (done && *done) return;
  double acc = 0.0;
#pragma unroll
  for (int j = 0; j < kReduceGroup / kThreads; ++j) {
    const int64_t i = blockIdx.x * (int64_t)kReduceGroup + j * kThreads + threadIdx.x;
    if (i < n) acc += p[i];
  }
  double v[1] = {acc}, tot[1];
  if (grid_reduce<1>(v, red, tot) && threadIdx.x == 0) finish_or_defer<1>(red, fin, target, tot);
}

// ---------------------------------------------------------------- Gauss-Seidel

// One Gauss-Seidel row update, src/ComputeSYMGS_ref.cpp:72-80:
//   sum = r_i - sum_j a_ij x_j (diagonal included, slot order); sum += x_i a_ii;
//   x_i = sum / a_ii.
// The terms are taken in two parts: the slots of the stencil lines 0 .. 3
// (slots 0 .. 11), and those of line 4, the row's own, and lines 5 .. 8.  Only
// the own line changes while a class is swept, so the first part is summed as
// soon as it is loaded -- once for a row that is updated twice (class 3) and
// for the residual that GS_RESTRICT forms -- and only the second part stays in
// registers over the exchange between the two rows of a pair.
// PX: the row's place in the pair (0 even, 1 odd); c: its colour; out: its
// left-out entries.
// ZERO: x is zero for every colour above c and for the row itself (first
//       forward sweep after ZeroVector); those terms are skipped.  Skipping a
//       product with a zero changes nothing but possibly the sign of an exact
//       zero.
constexpr int kHead = 12;   // slots of the first part

template <int PX, bool ZERO, class V, class T>
__device__ __forceinline__ T gs_head(uint32_t out, int c, const V &val, const T (&xl)[4][4], T sum) {
#pragma unroll
  for (int s = 0; s < kHead; ++s)
    if (!(ZERO && (c ^ slot_mask(s)) > c))
      sum = term_sub(out, s, sum, (T)val.get(s), xl[s / 3][s % 3 + PX]);
  return sum;
}

// xl[l - 4][0..3] = x[2i-1 .. 2i+2] of line l; xi: the row's own entry before
// the update.
template <int PX, bool ZERO, class V, class T>
__device__ __forceinline__ T gs_tail(uint32_t out, int c, const V &val, const T (&xl)[5][4], T sum,
                                     T xi) {
  const T d = val.get(HPCGX_DIAG_SLOT);
#pragma unroll
  for (int s = kHead; s < HPCGX_STENCIL; ++s) {
    if (s == HPCGX_DIAG_SLOT) {
      if (!ZERO) sum = mac_sub(sum, d, xi);
    } else if (!(ZERO && (c ^ slot_mask(s)) > c)) {
      sum = term_sub(out, s, sum, (T)val.get(s), xl[s / 3 - 4][s % 3 + PX]);
    }
  }
  if (!ZERO) sum = mac_add(sum, xi, d);
  return rn_div(sum, d);
}

// A half sweep of one class over its lines [j0, j1), by one block: colours ce
// then ce + 1 (DIR = 0) or ce + 1 then ce (DIR = 1), ce = 2 C.q.  A thread
// updates both rows of a pair; the colours of a class only depend on each
// other along x inside a line, and the block owns whole lines, so the entry
// that the second row needs from the next pair (the next even one forward, the
// previous odd one backward) comes through shared memory, and every load of
// the pair was issued before the first update.
// ZERO: x is zero for the colours above and for the row itself (first forward
//       sweep after ZeroVector); their terms are skipped at compile time.
// pro:  colour 0 first receives the prolongated coarse correction -- except in
//       the first plane of a slab with a halo below, whose correction is added
//       before the halo exchange (the slab below reads that plane).
// res:  after its update, the fine residual at the injected points (colour 0)
//       is formed and restricted: rc = r_i - (A x)_i with (A x)_i summed as in
//       SpMV (a slab with a halo below forms its first plane's again once the
//       halo holds the slab below's smoothed values).
// SYM3: forward and backward half sweep of the last class (DIR = 0): colour 6
//       forward, colour 7 forward and backward, colour 6 backward.
// AHEAD: the matrix values are loaded before the kernel ahead is waited for
// (launch_dependent); done: nothing to do once it is set.
// Lines longer than a block are taken in chunks of blockDim pairs, from right
// to left forward and from left to right backward: a chunk then finds the
// neighbours that its first row must see unchanged unchanged, and those that
// its second row must see updated updated.
template <int DIR, bool ZERO, bool SYM3, bool AHEAD, int FORM, class VT, class T, class RT>
__device__ __forceinline__ void gs_pairs(const LevelMat<VT> &A, const ClassInfo &C, int ce, int j0,
                                         int j1, bool pro, bool res, bool vec,
                                         const uint32_t *left_out, const RT *r, T *x, const T *xc,
                                         T *rc, T *sh, const int *done) {
  const int cnt = (j1 - j0) * C.len[0];
  const int nb = blockDim.x, tid = threadIdx.x;
  const int chunks = (cnt + nb - 1) / nb;
  const int co = ce + 1;
  // a value is read if its slot is: all, or (ZERO) those of the lower colours
  auto need_e = [=](int s) { return !ZERO || SYM3 || s == HPCGX_DIAG_SLOT || (ce ^ slot_mask(s)) < ce; };
  auto need_o = [=](int s) { return !ZERO || s == HPCGX_DIAG_SLOT || (co ^ slot_mask(s)) < co; };
  for (int ch = 0; ch < chunks; ++ch) {
    if (ch) __syncthreads();   // the chunk before has stored its rows and read sh
    const int t = (DIR == 0 ? chunks - 1 - ch : ch) * nb + tid;
    const bool act = t < cnt;
    PairId id;
    RowVals<VT> ve, vo;
    if (FORM != FORM_WIDE) vo = RowVals<VT>{};   // (the wide form loads it always)
    uint32_t oe = 0u, oo = 0u;
    T xl[5][4];
    T se = T(0), so = T(0), ax = T(0), xe = T(0), xo = T(0), re = T(0);
    int64_t crow = 0;
    if (!AHEAD && ch == 0) {
      dependency_wait();
      if (done && *done) return;
    }
    if (act) {
      id = pair_of(A, C, j0, t, 3);
      if (left_out) {
        oe = left_out[id.ke];
        oo = left_out[id.ko];
      }
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        ve.load(A.vals, id.ke, p, need_e);
        if (FORM == FORM_WIDE || id.odd) vo.load(A.vals, id.ko, p, need_o);
      }
    }
    if (AHEAD && ch == 0) {
      dependency_wait();
      if (done && *done) return;
    }
    if (act) {
      const T *xr = x + id.row;
      T ro = T(0);
      if (vec) {
        RT u, v;
        load2(r + id.row, u, v);
        re = vec_to(u, T());
        ro = vec_to(v, T());
      } else {
        re = vec_to(r[id.row], T());
        if (id.odd) ro = vec_to(r[id.row + 1], T());
      }
      {
        T xh[4][4];
#pragma unroll
        for (int l = 0; l < 9; ++l) {
          T *to = l < 4 ? xh[l < 4 ? l : 0] : xl[l < 4 ? 0 : l - 4];
          // in the zero-guess sweep the pair's own line and those of the higher
          // classes are not written yet
          const bool there = l != 4 && (ce ^ (slot_mask(3 * l + 1))) < ce;
          if (ZERO && !there)
            to[0] = to[1] = to[2] = to[3] = T(0);
          else
            load_line(A, id, xr, l, vec, to, 4);
        }
        se = gs_head<0, ZERO>(oe, ce, ve, xh, re);
        so = gs_head<1, ZERO>(oo, co, vo, xh, ro);
        if (res) {
#pragma unroll
          for (int s = 0; s < kHead; ++s) ax = term_add(oe, s, ax, (T)ve.get(s), xh[s / 3][s % 3]);
        }
      }
      if (pro || res) {
        const int nxc = A.nx >> 1, nyc = A.ny >> 1;
        crow = ((int64_t)(id.iz >> 1) * nyc + (id.iy >> 1)) * nxc + id.pos;
        crow = check_index(crow, (int64_t)nxc * nyc * (A.nz >> 1), 5);
      }
      xe = xl[0][1];
      xo = xl[0][2];
      if (pro && !(A.zlo && id.iz == 0)) xe = rn_add(xe, xc[crow]);
      if (DIR == 0) {
        xe = gs_tail<0, ZERO>(oe, ce, ve, xl, se, xe);
        sh[tid] = xe;
      } else if (id.odd) {
        xo = gs_tail<1, false>(oo, co, vo, xl, so, xo);
        sh[tid + 1] = xo;
      }
    }
    __syncthreads();
    if (act) {
      if (DIR == 0) {
        xl[0][1] = xe;
        if (id.right) xl[0][3] = tid + 1 < nb ? sh[tid + 1] : x[id.row + 2];
        if (id.odd) {
          xo = gs_tail<1, ZERO>(oo, co, vo, xl, so, xo);
          // forward then backward: between the two only the row's own entry
          // changes
          if (SYM3) xo = gs_tail<1, false>(oo, co, vo, xl, so, xo);
        }
      } else {
        xl[0][2] = xo;
        if (id.left) xl[0][0] = tid > 0 ? sh[tid] : x[id.row - 1];
        xe = gs_tail<0, false>(oe, ce, ve, xl, se, xe);
      }
      if (res) {
#pragma unroll
        for (int s = kHead; s < HPCGX_STENCIL; ++s)
          ax = term_add(oe, s, ax, (T)ve.get(s),
                        s == HPCGX_DIAG_SLOT ? xe : xl[s / 3 - 4][s % 3]);
        rc[crow] = rn_sub(re, ax);
      }
    }
    if (SYM3 && chunks == 1) {
      __syncthreads();
      if (act) sh[tid + 1] = xo;
      __syncthreads();
      if (act) {
        xl[0][2] = xo;
        if (id.left) xl[0][0] = sh[tid];
        xe = gs_tail<0, false>(oe, ce, ve, xl, se, xe);
      }
    }
    if (act) {
      if (vec) {
        store2(x + id.row, xe, xo);
      } else {
        x[id.row] = xe;
        if (id.odd) x[id.row + 1] = xo;
      }
    }
  }
  if (SYM3 && chunks > 1) {
    // colour 6 backward of a line in chunks, once every colour 7 row is final
    __syncthreads();
    for (int t = tid; t < cnt; t += nb) {
      const PairId id = pair_of(A, C, j0, t, 3);
      RowVals<VT> ve;
      T xh[4][4], xl[5][4];
#pragma unroll
      for (int p = 0; p < 3; ++p) ve.load(A.vals, id.ke, p, NeedAll());
#pragma unroll
      for (int l = 0; l < 9; ++l)
        load_line(A, id, (const T *)x + id.row, l, vec,
                  l < 4 ? xh[l < 4 ? l : 0] : xl[l < 4 ? 0 : l - 4], 4);
      const uint32_t oe = left_out ? left_out[id.ke] : 0u;
      const T sum = gs_head<0, false>(oe, ce, ve, xh, vec_to(r[id.row], T()));
      x[id.row] = gs_tail<0, false>(oe, ce, ve, xl, sum, xl[0][1]);
    }
  }
}

// Brings the values of the lines [j0, j1) of a class into L2: whole slices, one
// bulk prefetch per colour.  The large BF16 classes (three blocks per SM) wait
// for the latency of their loads more than for HBM; with the values of the block
// kAhead launches on under way they wait for L2's instead: mixed V-cycle at 384^3
// 2953 -> 2827 us, at 256^3 941 -> 923 (twice and four times the distance: 2829
// and 2854; ten times: 2947).  The FP64 sweeps, which HBM bounds, only lose by it
// (256^3: 2317 -> 2628), and so would a zero-guess sweep that skips most slots.
constexpr int kAhead = 222;
template <class VT>
__device__ __forceinline__ void prefetch_lines(const LevelMat<VT> &A, const ClassInfo &C, int j0,
                                               int j1) {
#pragma unroll
  for (int px = 0; px < 2; ++px) {
    const int64_t ka = C.start[px] + (int64_t)j0 * C.len[px];
    const int64_t kb = C.start[px] + (int64_t)j1 * C.len[px];
    if (kb <= ka) continue;
    const VT *from = A.vals + (ka >> 5) * kSliceElems;
    const uint32_t bytes = (uint32_t)((((kb - 1) >> 5) - (ka >> 5) + 1) * kSliceElems * sizeof(VT));
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(from), "r"(bytes) : "memory");
  }
}

// A half sweep over the lines [jbeg, jend) of a class, lpb lines per block (a
// sharded sweep splits its first launch into the lines that read no halo plane
// and the rest).  Q >= 0 fixes the class at compile time, which lets the
// zero-guess sweep drop the loads of the skipped slots.
// FORM: see Form.  Each form holds its own tests only, and the last pair of an odd
// line no values of a second row: one form for everything but FORM_WIDE, with a
// test for left-out entries at every term, took 1475 us for the symmetric FP64
// sweep at 255^3 (1190 so; with one row per thread 1601) and 640 for the BF16 one
// (460; 512); from vectors off the boundary FP64 1586 at 258 x 200 x 200 (1172;
// 1053), BF16 2556 at 384^3 (1430; 1590).
// Against one row per thread with a second load phase for the second colour
// (before) the pair issues all its loads once: FP64, HBM-bound, the symmetric
// sweep at 256^3 takes 1186 us = 6.1 TB/s of 8 B per nonzero and pass (before,
// with stored columns: 1596 us), the V-cycle at 104^3, latency-bound on its
// coarse levels, 399 us (545).  BF16: 2 B per nonzero leaves the loads' latency
// and x, which every class launch gathers again, as the bound: V-cycle at
// 256^3 1137 us (1205), at 64^3 218 us (269).
// Launched dependent on the launch before (launch_dependent): the launch, the
// index arithmetic and the values' loads go under the end of that one, 49
// times in a V-cycle: FP64 at 104^3 279 us (399), at 256^3 2341 us (2513);
// BF16 at 64^3 136 us (218), at 256^3 937 us (1137), at 384^3 2934 us (3293).
// The BF16 kernels with three blocks per SM wait first (AHEAD off): values held
// over the wait cost them spills (384^3: 3353 us).
template <int MODE, int DIR, int Q, int MINB, int FORM, class VT, class T, class RT>
__global__ void __launch_bounds__(kThreads, MINB)
k_gs_class(const __grid_constant__ LevelMat<VT> A, const __grid_constant__ ClassInfo C, int lpb,
           int jbeg, int jend, int vec, const RT *r, T *x, const T *xc, T *rc, const int *done) {
  constexpr bool ZERO = (MODE & GS_ZERO_GUESS) != 0;
  static_assert(!ZERO || Q >= 0, "the zero-guess sweep knows its class");
  __shared__ T sh[kThreads + 2];
  dependents_launch();
  const int j0 = jbeg + blockIdx.x * lpb;
  if (MINB == 3 && (!ZERO || (MODE & GS_SYM3)) && threadIdx.x == 0) {
    if (blockIdx.x < kAhead) prefetch_lines(A, C, j0, min(j0 + lpb, jend));
    const int jn = j0 + kAhead * lpb;
    if (jn < jend) prefetch_lines(A, C, jn, min(jn + lpb, jend));
  }
  gs_pairs<DIR, ZERO, (MODE & GS_SYM3) != 0, MINB != 3, FORM>(
      A, C, 2 * (Q >= 0 ? Q : C.q), j0, min(j0 + lpb, jend), (MODE & GS_PROLONG) != 0,
      (MODE & GS_RESTRICT) != 0, is_wide<FORM>(vec), FORM == FORM_HOLES ? A.left_out : nullptr, r, x,
      xc, rc, sh, done);
}

// Residual restricted at the injected points (colour 0: even ix, iy, iz):
// rc = rf - (A x) there, (A x)_i summed over the slots from 0 in order as
// ComputeSPMV_ref does (src/ComputeSPMV_ref.cpp:64-70), then
// src/ComputeRestriction_ref.cpp:51.  The standalone form of GS_RESTRICT, for
// the sharded V-cycle, where the halo of x is exchanged between the sweep and
// the residual (src/ComputeMG_ref.cpp:49-51): launched over the first coarse
// plane only (nc = nxc * nyc), the one injected plane that reads the halo.
template <class VT, class T, class RT>
__global__ void __launch_bounds__(kThreads)
k_restrict_residual(LevelMat<VT> A, ClassInfo C0, int64_t nc, const RT *__restrict__ rf,
                    const T *__restrict__ x, T *__restrict__ rc, const int *__restrict__ done) {
  if (done && *done) return;
  const int nxc = A.nx >> 1, nyc = A.ny >> 1;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nc;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int ixc = (int)(i % nxc), iyc = (int)((i / nxc) % nyc);
    const int izc = (int)(i / ((int64_t)nxc * nyc));
    RowId id;
    id.ix = 2 * ixc;
    id.iy = 2 * iyc;
    id.iz = 2 * izc;
    id.row = ((int64_t)id.iz * A.ny + id.iy) * A.nx + id.ix;
    id.k = C0.start[0] + ((int64_t)izc * C0.nyq + iyc) * C0.len[0] + ixc;  // colour 0
    check_row(A, id, 6);
    int32_t col[HPCGX_STENCIL];
    T val[HPCGX_STENCIL];
#pragma unroll
    for (int p = 0; p < 3; ++p) load_vals(A.vals, id.k, p, NeedAll(), val + 9 * p);
    stencil_cols(A, id, col);
    check_cols(A, col, NeedAll(), 7);
    T ax = T(0);
#pragma unroll
    for (int s = 0; s < HPCGX_STENCIL; ++s) ax = mac_add(ax, val[s], x[col[s]]);
    rc[i] = rn_sub(vec_to(__ldg(rf + id.row), T()), ax);
  }
}

// xf += xc at the injected points (src/ComputeProlongation_ref.cpp:49), in the
// vector type of the V-cycle.  The sharded V-cycle launches it over the first
// coarse plane only, before the halo exchange; GS_PROLONG adds the rest.
template <class T>
__global__ void __launch_bounds__(kThreads)
k_prolong(int64_t nc, int nxf, int nyf, const T *__restrict__ xc, T *xf,
          const int *__restrict__ done) {
  if (done && *done) return;
  const int nxc = nxf >> 1, nyc = nyf >> 1;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nc;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t ixc = i % nxc, iyc = (i / nxc) % nyc, izc = i / ((int64_t)nxc * nyc);
    const int64_t f = ((2 * izc) * nyf + 2 * iyc) * nxf + 2 * ixc;
    xf[f] = rn_add(xf[f], xc[i]);
  }
}

// ---------------------------------------------------------------- vectors

// The vector kernels are bound by HBM (or by L2, where the vectors fit it).  A
// block takes tiles of kTile elements; a thread handles four of a tile, two
// neighbouring ones and the two half a tile on, with one vector load each, so
// that a warp's load is one segment and a thread has two loads per vector under
// way.  One element per thread and step before: k_cg_xr at 384^3 331 us -> 270
// (5.9 TB/s), a mixed iteration 5.79 -> 5.71 ms; at 64^3 127 -> 123 us.
// WIDE: every vector of the launch starts on a two-element boundary; without it a
// thread takes the same elements one by one, so that a sum's order, and with it
// its last bits, depend on the length alone and not on where a view starts.
constexpr int kVec = 4;
constexpr int kTile = kVec * kThreads;
template <int N, bool WIDE>
struct Width {
  static constexpr int value = N;
};
// Runs body(i, width) over [0, n): width 4 for a thread's elements i, i + 1 and
// i + kTile / 2, i + kTile / 2 + 1 of a tile, width 1 for element i alone.
template <bool WIDE, class F>
__device__ __forceinline__ void sweep(int64_t n, F body) {
  const int64_t tiles = n / kTile;
  for (int64_t b = blockIdx.x; b < tiles; b += gridDim.x)
    body(b * kTile + 2 * (int)threadIdx.x, Width<kVec, WIDE>());
  for (int64_t i = tiles * kTile + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    body(i, Width<1, WIDE>());
}
template <int N, bool WIDE, class T>
__device__ __forceinline__ void get(Width<N, WIDE>, const T *p, int64_t i, T *v) {
  if (N == 1) {
    v[0] = p[i];
  } else if (WIDE) {
    load2(p + i, v[0], v[1]);
    load2(p + i + kTile / 2, v[2], v[3]);
  } else {
#pragma unroll
    for (int j = 0; j < kVec; ++j) v[j] = p[i + (j & 1) + (j >> 1) * (kTile / 2)];
  }
}
template <int N, bool WIDE, class T>
__device__ __forceinline__ void put(Width<N, WIDE>, T *p, int64_t i, const T *v) {
  if (N == 1) {
    p[i] = v[0];
  } else if (WIDE) {
    store2(p + i, v[0], v[1]);
    store2(p + i + kTile / 2, v[2], v[3]);
  } else {
#pragma unroll
    for (int j = 0; j < kVec; ++j) p[i + (j & 1) + (j >> 1) * (kTile / 2)] = v[j];
  }
}

template <bool WIDE>
__global__ void __launch_bounds__(kThreads)
k_waxpby(int64_t n, double alpha, const double *x, double beta, const double *y, double *w,
         const int *done) {
  if (done && *done) return;
  // The three branches of src/ComputeWAXPBY_ref.cpp:52-67 round differently.
  const int branch = alpha == 1.0 ? 0 : beta == 1.0 ? 1 : 2;
  sweep<WIDE>(n, [=](int64_t i, auto k) {
    double a[kVec], b[kVec];
    get(k, x, i, a);
    get(k, y, i, b);
#pragma unroll
    for (int j = 0; j < k.value; ++j)
      a[j] = rn_add(branch == 0 ? a[j] : rn_mul(alpha, a[j]), branch == 1 ? b[j] : rn_mul(beta, b[j]));
    put(k, w, i, a);
  });
}

// x.y; the last block stores the total (FIN_STORE into target) or runs a CG
// scalar step on it (target: the CgState).
template <bool WIDE>
__global__ void __launch_bounds__(kThreads)
k_dot(int64_t n, const double *x, const double *y, Reduce red, int fin, void *target,
      const int *done) {
  if (done && *done) return;
  double acc = 0.0;
  sweep<WIDE>(n, [&](int64_t i, auto k) {
    double a[kVec], b[kVec];
    get(k, x, i, a);
    get(k, y, i, b);
#pragma unroll
    for (int j = 0; j < k.value; ++j) acc += a[j] * b[j];
  });
  double v[1] = {acc}, tot[1];
  if (grid_reduce<1>(v, red, tot) && threadIdx.x == 0) finish_or_defer<1>(red, fin, target, tot);
}

__global__ void __launch_bounds__(kThreads)
k_absmax_diff(int64_t n, const double *__restrict__ a, const double *__restrict__ b, Reduce red,
              double *out) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  double m = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += stride)
    m = fmax(m, fabs(a[i] - b[i]));
  double v[1] = {m}, tot[1];
  if (grid_reduce<1, true>(v, red, tot) && threadIdx.x == 0) out[0] = tot[0];
}

__device__ __forceinline__ int64_t fine_of_coarse(int64_t ic, int nxf, int nyf) {
  const int nxc = nxf >> 1, nyc = nyf >> 1;
  const int64_t ixc = ic % nxc, iyc = (ic / nxc) % nyc, izc = ic / ((int64_t)nxc * nyc);
  return (2 * izc) * (int64_t)nxf * nyf + (2 * iyc) * (int64_t)nxf + 2 * ixc;
}

// src/ComputeRestriction_ref.cpp:51 with f2c of src/GenerateCoarseProblem.cpp:71-82.
__global__ void k_restriction(int64_t nc, int nxf, int nyf, const double *__restrict__ rf,
                              const double *__restrict__ Axf, double *rc) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nc;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t f = fine_of_coarse(i, nxf, nyf);
    rc[i] = rn_sub(rf[f], Axf[f]);
  }
}

// src/ComputeProlongation_ref.cpp:49.
__global__ void k_prolongation(int64_t nc, int nxf, int nyf, const double *__restrict__ xc,
                               double *xf) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nc;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t f = fine_of_coarse(i, nxf, nyf);
    xf[f] = rn_add(xf[f], xc[i]);
  }
}

__global__ void k_copy(int64_t n, const double *__restrict__ x, double *y,
                       const int *__restrict__ done) {
  if (done && *done) return;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    y[i] = x[i];
}

__global__ void k_fill_uniform(int64_t n, uint64_t seed, uint64_t offset, double lo, double hi,
                               double *v) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    v[i] = rn_add(lo, rn_mul(rn_sub(hi, lo), uniform01(seed, offset + (uint64_t)i)));
}

__device__ __forceinline__ double normal01(uint64_t seed, uint64_t i) {
  const double u1 = 1.0 - uniform01(seed, 2 * i);
  const double u2 = uniform01(seed, 2 * i + 1);
  return sqrt(-2.0 * log(u1)) * cos(6.283185307179586 * u2);
}

__global__ void k_fill_normal(int64_t n, uint64_t seed, uint64_t offset, double *v) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    v[i] = normal01(seed, offset + (uint64_t)i);
}

// ---------------------------------------------------------------- CG pieces

// r = b - Ap (WAXPBY(1, b, -1, Ap), src/CG.cpp:88) and |r|^2 -> normr0.
__global__ void __launch_bounds__(kThreads)
k_cg_init(int64_t n, const double *__restrict__ b, const double *__restrict__ Ap, double *r,
          float *r32, Reduce red, CgState *st) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  double acc = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += stride) {
    const double ri = rn_add(b[i], rn_mul(-1.0, Ap[i]));
    r[i] = ri;
    if (r32) r32[i] = (float)ri;
    acc += ri * ri;
  }
  double v[1] = {acc}, tot[1];
  if (grid_reduce<1>(v, red, tot) && threadIdx.x == 0)
    finish_or_defer<1>(red, FIN_CG_INIT, st, tot);
}

// rtz = r.z (src/CG.cpp:109/112); for the flexible solver also z.Ap_{k-1}.
template <bool WIDE, class ZT, bool FLEX>
__global__ void __launch_bounds__(kThreads)
k_cg_rz(int64_t n, const double *r, const ZT *z, const double *Ap, Reduce red, CgState *st) {
  dependents_launch();
  dependency_wait();
  if (st->done) return;
  const bool two = FLEX && st->k > 1;
  double a0 = 0.0, a1 = 0.0;
  sweep<WIDE>(n, [&](int64_t i, auto k) {
    double a[kVec], b[kVec];
    ZT c[kVec];
    get(k, r, i, a);
    get(k, z, i, c);
    if (two) get(k, Ap, i, b);
#pragma unroll
    for (int j = 0; j < k.value; ++j) {
      a0 += a[j] * (double)c[j];
      if (two) a1 += (double)c[j] * b[j];
    }
  });
  if (FLEX) {
    double v[2] = {a0, a1}, tot[2];
    if (grid_reduce<2>(v, red, tot) && threadIdx.x == 0)
      finish_or_defer<2>(red, FIN_CG_RZ, st, tot);
  } else {
    double v[1] = {a0}, tot[1];
    if (grid_reduce<1>(v, red, tot) && threadIdx.x == 0)
      finish_or_defer<1>(red, FIN_CG_RZ, st, tot);
  }
}

// p = z (k == 1) or p = z + beta p (WAXPBY(1, z, beta, p), src/CG.cpp:115).
// With x given, the previous iteration's x += alpha p (src/CG.cpp:121) is
// applied here, while p_{k-1} is read anyway, instead of in k_cg_xr: the same
// operation on the same operands, one read of p fewer per iteration.
// k_cg_xflush applies the last iteration's update after the loop.
template <bool WIDE, class ZT>
__global__ void __launch_bounds__(kThreads)
k_cg_p(int64_t n, const ZT *z, double *p, const CgState *st, double *x) {
  dependents_launch();
  dependency_wait();
  if (st->done) return;
  const bool first = st->k == 1;
  const double beta = st->beta, alpha = st->alpha;
  sweep<WIDE>(n, [=](int64_t i, auto k) {
    double a[kVec], b[kVec];
    ZT c[kVec];
    get(k, z, i, c);
    if (!first) {
      get(k, (const double *)p, i, a);
      if (x) {
        get(k, (const double *)x, i, b);
#pragma unroll
        for (int j = 0; j < k.value; ++j) b[j] = rn_add(b[j], rn_mul(alpha, a[j]));
        put(k, x, i, b);
      }
    }
#pragma unroll
    for (int j = 0; j < k.value; ++j)
      a[j] = first ? (double)c[j] : rn_add((double)c[j], rn_mul(beta, a[j]));
    put(k, p, i, a);
  });
}

// The deferred x += alpha p of the last iteration that ran.
__global__ void __launch_bounds__(kThreads)
k_cg_xflush(int64_t n, const double *__restrict__ p, double *x, const CgState *__restrict__ st) {
  if (st->niters < 1) return;
  const double alpha = st->alpha;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    x[i] = rn_add(x[i], rn_mul(alpha, p[i]));
}

// x += alpha p (unless deferred: x null); r -= alpha Ap; |r|^2
// (src/CG.cpp:121-124).  r32 (mixed solver): the FP32 copy of r that the
// V-cycle's finest level reads -- the value it would round r to itself.
template <bool WIDE>
__global__ void __launch_bounds__(kThreads)
k_cg_xr(int64_t n, const double *p, const double *Ap, double *x, double *r, float *r32,
        Reduce red, CgState *st) {
  dependents_launch();
  dependency_wait();
  if (st->done) return;
  const double alpha = st->alpha, malpha = -st->alpha;
  double acc = 0.0;
  sweep<WIDE>(n, [&](int64_t i, auto k) {
    double a[kVec], b[kVec];
    get(k, (const double *)r, i, a);
    get(k, Ap, i, b);
    if (x) {
      double c[kVec], e[kVec];
      get(k, (const double *)x, i, c);
      get(k, p, i, e);
#pragma unroll
      for (int j = 0; j < k.value; ++j) c[j] = rn_add(c[j], rn_mul(alpha, e[j]));
      put(k, x, i, c);
    }
    float f[kVec];
#pragma unroll
    for (int j = 0; j < k.value; ++j) {
      a[j] = rn_add(a[j], rn_mul(malpha, b[j]));
      f[j] = (float)a[j];
      acc += a[j] * a[j];
    }
    put(k, r, i, a);
    if (r32) put(k, r32, i, f);
  });
  double v[1] = {acc}, tot[1];
  if (grid_reduce<1>(v, red, tot) && threadIdx.x == 0)
    finish_or_defer<1>(red, FIN_CG_RR, st, tot);
}

__global__ void k_copy_z(int64_t n, const double *__restrict__ r, double *z,
                         const CgState *__restrict__ st) {
  if (st->done) return;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    z[i] = r[i];
}

// ---------------------------------------------------------------- set-up

struct Geo {
  int nx, ny, nz;
  int zlo, zhi;   // z-slab: the planes below / above belong to a neighbouring rank
  const uint32_t *left_out;   // LevelMat::left_out
  int64_t cstart[8], ccount[8];
  int len[2];
  int nyq[4];
};

__device__ __forceinline__ bool storage_to_natural(const Geo &g, int64_t k, int64_t &row, int &ix,
                                                   int &iy, int &iz) {
  int c = 0;
#pragma unroll
  for (int i = 1; i < 8; ++i)
    if (k >= g.cstart[i]) c = i;
  const int64_t rem = k - g.cstart[c];
  if (rem >= g.ccount[c]) return false;
  const int px = c & 1, q = c >> 1, py = q & 1, pz = q >> 1;
  const int Lp = g.len[px];
  const int64_t j = rem / Lp;
  const int pos = (int)(rem - j * Lp);
  iy = py + 2 * (int)(j % g.nyq[q]);
  iz = pz + 2 * (int)(j / g.nyq[q]);
  ix = px + 2 * pos;
  row = ((int64_t)iz * g.ny + iy) * g.nx + ix;
  return true;
}

__device__ __forceinline__ int64_t natural_to_storage(const Geo &g, int64_t row) {
  const int ix = (int)(row % g.nx);
  const int iy = (int)((row / g.nx) % g.ny);
  const int iz = (int)(row / ((int64_t)g.nx * g.ny));
  const int px = ix & 1, q = (iy & 1) + 2 * (iz & 1);
  const int c = px + 2 * q;
  const int64_t j = (int64_t)(iz >> 1) * g.nyq[q] + (iy >> 1);
  return g.cstart[c] + j * g.len[px] + (ix >> 1);
}

__device__ __forceinline__ bool neighbour(const Geo &g, int ix, int iy, int iz, int s,
                                          int64_t row, int64_t &col) {
  const int dx = s % 3 - 1, dy = (s / 3) % 3 - 1, dz = s / 9 - 1;
  const int jx = ix + dx, jy = iy + dy, jz = iz + dz;
  if (jx < 0 || jx >= g.nx || jy < 0 || jy >= g.ny) return false;
  if ((jz < 0 && !g.zlo) || (jz >= g.nz && !g.zhi)) return false;
  col = row + (int64_t)dz * g.nx * g.ny + (int64_t)dy * g.nx + dx;
  return true;
}

// The reference problem (src/GenerateProblem_ref.cpp:152-172) written
// straight into the device layout: 26 on the diagonal, -1 elsewhere.
__global__ void k_generate_hpcg(Geo g, int64_t storage_rows, double *vals) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < storage_rows;
       k += (int64_t)gridDim.x * blockDim.x) {
    int64_t row;
    int ix, iy, iz;
    const bool real = storage_to_natural(g, k, row, ix, iy, iz);
    for (int s = 0; s < HPCGX_STENCIL; ++s) {
      int64_t col;
      double v = 0.0;
      if (real && neighbour(g, ix, iy, iz, s, row, col))
        v = (s == HPCGX_DIAG_SLOT) ? 26.0 : -1.0;
      vals[vidx(k, s)] = v;
    }
  }
}

// Variable-coefficient SPD matrix (the oracle's or_generate_varcoef): each
// undirected edge {lo, hi} draws z ~ N(0,1) keyed by the finest-level index of
// lo and the direction, a = -exp(sigma z); diagonal = sum |a| + 2.
__global__ void k_generate_varcoef(Geo g, int64_t storage_rows, int level, int nx0, int ny0,
                                   uint64_t seed, double sigma, double *vals) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < storage_rows;
       k += (int64_t)gridDim.x * blockDim.x) {
    int64_t row;
    int ix, iy, iz;
    const bool real = storage_to_natural(g, k, row, ix, iy, iz);
    double dsum = 0.0;
    for (int s = 0; s < HPCGX_STENCIL; ++s) {
      int64_t col;
      double v = 0.0;
      if (real && s != HPCGX_DIAG_SLOT && neighbour(g, ix, iy, iz, s, row, col)) {
        int lx = ix, ly = iy, lz = iz, h = s - 14;
        if (s < HPCGX_DIAG_SLOT) {
          lx = ix + (s % 3 - 1);
          ly = iy + ((s / 3) % 3 - 1);
          lz = iz + (s / 9 - 1);
          h = 12 - s;
        }
        const int64_t lo = ((int64_t)(lz << level) * ny0 + (ly << level)) * nx0 + (lx << level);
        v = -exp(sigma * normal01(seed, (uint64_t)lo * 13u + (uint64_t)h));
        dsum += fabs(v);
      }
      vals[vidx(k, s)] = v;
    }
    if (real) vals[vidx(k, HPCGX_DIAG_SLOT)] = dsum + 2.0;
  }
}

// Coarse variable-coefficient operator from the fine one: the coarse edge
// {lo, lo+d} takes the fine value of the edge leaving the injected point of lo
// in direction d; the diagonal is again sum |a| + 2.
__global__ void k_coarsen_varcoef(Geo gf, Geo gc, int64_t storage_rows_c,
                                  const double *__restrict__ fvals, double *cvals) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < storage_rows_c;
       k += (int64_t)gridDim.x * blockDim.x) {
    int64_t row;
    int ix, iy, iz;
    if (!storage_to_natural(gc, k, row, ix, iy, iz)) continue;
    double dsum = 0.0;
    for (int s = 0; s < HPCGX_STENCIL; ++s) {
      if (s == HPCGX_DIAG_SLOT) continue;
      int64_t col;
      if (!neighbour(gc, ix, iy, iz, s, row, col)) {
        cvals[vidx(k, s)] = 0.0;
        continue;
      }
      int lx = ix, ly = iy, lz = iz, sl = s;
      if (s < HPCGX_DIAG_SLOT) {
        lx = ix + (s % 3 - 1);
        ly = iy + ((s / 3) % 3 - 1);
        lz = iz + (s / 9 - 1);
        sl = 26 - s;
      }
      const int64_t frow = ((int64_t)(2 * lz) * gf.ny + 2 * ly) * gf.nx + 2 * lx;
      const int64_t fk = natural_to_storage(gf, frow);
      const double v = fvals[vidx(fk, sl)];
      cvals[vidx(k, s)] = v;
      dsum += fabs(v);
    }
    cvals[vidx(k, HPCGX_DIAG_SLOT)] = dsum + 2.0;
  }
}

// BF16 copy of the FP64 values (the two arrays group slots differently): a
// thread converts one z-plane of one storage row, so that a warp reads and
// writes whole segments of a slice.  Bound by HBM (8 B read, 2 B written per
// slot); all levels of 192 x 160 x 96: 395 us with a thread per slot, 151 so.
__global__ void __launch_bounds__(kThreads)
k_to_bf16(int64_t rows, const double *__restrict__ v, uint16_t *__restrict__ h) {
  const int64_t m = rows * 3;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m;
       i += (int64_t)gridDim.x * blockDim.x) {
    // 32 rows of a slice side by side, plane by plane
    const int64_t k = i / 96 * 32 + (i & 31);
    const int p = (int)(i / 32 % 3);
    double a[9];
    load_plane(v, k, p, NeedAll(), a);
    uint32_t c[9];
#pragma unroll
    for (int j = 0; j < 9; ++j) c[j] = bf16_from_double(a[j]);
    uint16_t *w = h + (k >> 5) * kSliceElems + p * kPlaneElems;
    const int lane = (int)(k & 31);
#pragma unroll
    for (int j = 0; j < 2; ++j)
      *reinterpret_cast<uint2 *>(w + j * 128 + lane * 4) =
          make_uint2(c[4 * j] | c[4 * j + 1] << 16, c[4 * j + 2] | c[4 * j + 3] << 16);
    w[256 + lane] = (uint16_t)c[8];
  }
}

// The row-major arrays of 27 slots per natural row (set_values, get_values,
// adjoint_grad) are read and written by blocks of kTileRows consecutive rows,
// one segment of kTileRows x 216 B each: a thread per row touched them 216 B
// apart (set_values at 128^3: 300 us, 229 so).  What a block needs to know of its
// rows:
constexpr int kTileRows = 64;
struct TileRows {
  int64_t k[kTileRows];      // storage row
  uint32_t nb[kTileRows];    // bit s: the neighbour of slot s exists
};
__device__ __forceinline__ void tile_rows(const Geo &g, int64_t row0, int m, TileRows &t) {
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    const uint32_t row = (uint32_t)row0 + i, nx = g.nx, ny = g.ny;   // fewer than 2^31 rows
    const uint32_t line = row / nx, ix = row - line * nx, iz = line / ny, iy = line - iz * ny;
    t.nb[i] = stencil_bits(ix > 0, ix + 1 < nx, iy > 0, iy + 1 < ny, iz > 0 || g.zlo,
                           (int)iz + 1 < g.nz || g.zhi);
    const int px = ix & 1, q = (iy & 1) + 2 * (iz & 1);
    t.k[i] = g.cstart[px + 2 * q] + ((int64_t)(iz >> 1) * g.nyq[q] + (iy >> 1)) * g.len[px] + (ix >> 1);
  }
}
// Row r of a tile: does the matrix leave out its entry in slot s?
__device__ __forceinline__ bool left_out(const Geo &g, const TileRows &t, int r, int s) {
  return g.left_out && (g.left_out[t.k[r]] >> s & 1u);
}
// Row i of a tile for the i-th of kTileRows neighbouring threads: the even rows,
// then the odd ones, each a run of storage rows where nx is even.
__device__ __forceinline__ int tile_row(int i) {
  return i < kTileRows / 2 ? 2 * i : 2 * (i - kTileRows / 2) + 1;
}
__device__ __forceinline__ int64_t slot_column(const Geo &g, int64_t row, int s) {
  return row + (int64_t)(s / 9 - 1) * g.nx * g.ny + (int64_t)((s / 3) % 3 - 1) * g.nx + (s % 3 - 1);
}

// Values in natural row order, 27 stencil slots per row -> device layout.
// Slots without a neighbour stay 0 whatever the input holds.
__global__ void __launch_bounds__(kThreads)
k_set_values(Geo g, int64_t n, const double *__restrict__ in, double *__restrict__ vals) {
  __shared__ TileRows t;
  __shared__ double sh[kTileRows * HPCGX_STENCIL];
  const int64_t row0 = (int64_t)blockIdx.x * kTileRows;
  const int m = (int)min((int64_t)kTileRows, n - row0);
  tile_rows(g, row0, m, t);
  for (int i = threadIdx.x; i < m * HPCGX_STENCIL; i += blockDim.x)
    sh[i] = in[row0 * HPCGX_STENCIL + i];
  __syncthreads();
  // a plane's slots go out in pairs and one single (vidx): 5 groups a plane
  for (int i = threadIdx.x; i < 15 * kTileRows; i += blockDim.x) {
    const int r = tile_row(i % kTileRows), group = i / kTileRows;
    if (r >= m) continue;
    const int s = group / 5 * 9 + group % 5 * 2;
    const uint32_t nb = t.nb[r] >> s;
    const double *v = sh + r * HPCGX_STENCIL + s;
    double *to = vals + vidx(t.k[r], s);
    const double v0 = nb & 1u ? v[0] : 0.0;
    if (group % 5 < 4)
      store2(to, v0, nb & 2u ? v[1] : 0.0);
    else
      *to = v0;
  }
}

// The same with a thread per row, for grids with a side of one row: it reads the
// 3 or 9 slots that such a row has at most, which outweighs its strided accesses
// (512 x 512 x 1 60 us a call with the tiles, 46 so, 1,000,000 x 1 x 1 140 and 93;
// where all sides are longer the tiles win, 128^3 254 against 324).
__global__ void __launch_bounds__(kThreads)
k_set_values_flat(Geo g, int64_t n, const double *__restrict__ in, double *__restrict__ vals) {
  for (int64_t row = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; row < n;
       row += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = natural_to_storage(g, row);
    const int ix = (int)(row % g.nx), iy = (int)((row / g.nx) % g.ny),
              iz = (int)(row / ((int64_t)g.nx * g.ny));
    const uint32_t nb = stencil_bits(ix > 0, ix + 1 < g.nx, iy > 0, iy + 1 < g.ny, iz > 0 || g.zlo,
                                     iz + 1 < g.nz || g.zhi);
    for (int s = 0; s < HPCGX_STENCIL; ++s)
      vals[vidx(k, s)] = nb >> s & 1u ? in[row * HPCGX_STENCIL + s] : 0.0;
  }
}

// Device layout -> natural row order; the column of a slot is its neighbour, or
// the row itself where it has none or the matrix leaves the entry out.
__global__ void __launch_bounds__(kThreads)
k_get_values(Geo g, int64_t n, const double *__restrict__ vals, double *__restrict__ out,
             int32_t *__restrict__ cout) {
  __shared__ TileRows t;
  __shared__ double sh[kTileRows * HPCGX_STENCIL];
  const int64_t row0 = (int64_t)blockIdx.x * kTileRows;
  const int m = (int)min((int64_t)kTileRows, n - row0);
  tile_rows(g, row0, m, t);
  __syncthreads();
  for (int i = threadIdx.x; i < 15 * kTileRows; i += blockDim.x) {
    const int r = tile_row(i % kTileRows), group = i / kTileRows;
    if (r >= m) continue;
    const int s = group / 5 * 9 + group % 5 * 2;
    double *v = sh + r * HPCGX_STENCIL + s;
    const double *from = vals + vidx(t.k[r], s);
    if (group % 5 < 4)
      load2(from, v[0], v[1]);
    else
      v[0] = *from;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < m * HPCGX_STENCIL; i += blockDim.x) {
    const int r = i / HPCGX_STENCIL, s = i - r * HPCGX_STENCIL;
    const int64_t row = row0 + r;
    const bool has = (t.nb[r] >> s & 1u) && !left_out(g, t, r, s);
    if (out) out[row0 * HPCGX_STENCIL + i] = sh[i];
    if (cout) cout[row0 * HPCGX_STENCIL + i] = (int32_t)(has ? slot_column(g, row, s) : row);
  }
}

__global__ void k_set_diagonal(Geo g, int64_t n, const double *__restrict__ d, double *vals) {
  for (int64_t row = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; row < n;
       row += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = natural_to_storage(g, row);
    vals[vidx(k, HPCGX_DIAG_SLOT)] = d[row];
  }
}

__global__ void k_get_diagonal(Geo g, int64_t n, const double *__restrict__ vals, double *d) {
  for (int64_t row = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; row < n;
       row += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = natural_to_storage(g, row);
    d[row] = vals[vidx(k, HPCGX_DIAG_SLOT)];
  }
}

// dL/da_ij = -lambda_i x_j for every stored slot, natural row order, 27 slots
// per row (zero where the stencil has no neighbour).  A thread per slot: the
// 216 B written per row are the bound (128^3: 646 us with a thread per row, 152
// so).
__global__ void __launch_bounds__(kThreads)
k_adjoint_grad(Geo g, int64_t n, const double *__restrict__ lambda,
               const double *__restrict__ x, double *__restrict__ grad) {
  __shared__ TileRows t;
  const int64_t row0 = (int64_t)blockIdx.x * kTileRows;
  const int m = (int)min((int64_t)kTileRows, n - row0);
  tile_rows(g, row0, m, t);
  __syncthreads();
  for (int i = threadIdx.x; i < m * HPCGX_STENCIL; i += blockDim.x) {
    const int r = i / HPCGX_STENCIL, s = i - r * HPCGX_STENCIL;
    const int64_t row = row0 + r;
    double v = 0.0;
    if (t.nb[r] >> s & 1u) {
      // a left-out entry's column is the row itself
      v = -(lambda[row] * x[left_out(g, t, r, s) ? row : slot_column(g, row, s)]);
    }
    grad[row0 * HPCGX_STENCIL + i] = v;
  }
}

Geo geo_of(const LevelDev &L) {
  Geo g;
  g.nx = L.nx;
  g.ny = L.ny;
  g.nz = L.nz;
  g.zlo = L.zlo;
  g.zhi = L.zhi;
  g.left_out = L.holes ? L.left_out : nullptr;
  for (int c = 0; c < 8; ++c) {
    g.cstart[c] = L.cstart[c];
    g.ccount[c] = L.ccount[c];
  }
  g.len[0] = L.cls[0].len[0];
  g.len[1] = L.cls[0].len[1];
  for (int q = 0; q < 4; ++q) g.nyq[q] = L.cls[q].nyq;
  return g;
}

int tiles_for(int64_t n) { return (int)((n + kTileRows - 1) / kTileRows); }

int grid_for(int64_t n, int threads = kThreads) {
  int64_t b = (n + threads - 1) / threads;
  return (int)std::max<int64_t>(1, std::min<int64_t>(b, 148 * 16));
}

template <class VT>
LevelMat<VT> mat_of(const LevelDev &L, const VT *vals) {
  LevelMat<VT> A;
  A.vals = vals;
  for (int s = 0; s < HPCGX_STENCIL; ++s)
    A.off[s] = (s / 9 - 1) * L.nx * L.ny + ((s / 3) % 3 - 1) * L.nx + (s % 3 - 1);
  A.nx = L.nx;
  A.ny = L.ny;
  A.nz = L.nz;
  A.n = L.n;
  A.zlo = L.zlo;
  A.zhi = L.zhi;
  A.lo = L.zlo ? -L.nx * L.ny : 0;
  A.span = (int)L.n - A.lo + (L.zhi ? L.nx * L.ny : 0);
  A.srows = L.storage_rows;
  // left-out entries are a matter of the FP64 operators; the BF16 copy
  // multiplies the neighbour by 0
  A.left_out = L.holes && std::is_same<VT, double>::value ? L.left_out : nullptr;
  return A;
}

// Vector loads of x, y and the right-hand side: every line starts on an even
// row and the vectors on a two-element boundary (a halo plane of an odd size
// or a view at an odd offset does not).
template <class T>
bool aligned2(const T *v) {
  return reinterpret_cast<uintptr_t>(v) % (2 * sizeof(T)) == 0;
}

// The SpMV's blocks: `turns` groups of 256 consecutive pairs of a class each.
ClassSet classes_of(const LevelDev &L, int turns = 1) {
  ClassSet cs;
  cs.turns = turns;
  cs.common = INT_MAX;
  cs.total = 0;
  for (int q = 0; q < 4; ++q) {
    const ClassInfo &C = L.cls[q];
    const int64_t pairs = (int64_t)C.lines * C.len[0];
    cs.c[q] = C;
    cs.nblk[q] = (int)((pairs + turns * kThreads - 1) / (turns * kThreads));
    cs.common = std::min(cs.common, cs.nblk[q]);
    cs.total += cs.nblk[q];
  }
  return cs;
}

}  // namespace

// ======================================================================== host
// Every launch_* returns the number of kernels it launched (0 or 1).

cudaError_t CgMonitor::init() {
  if (slots) return cudaSuccess;
  for (cudaEvent_t &e : ev) {
    const cudaError_t rc = e ? cudaSuccess : cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
    if (rc != cudaSuccess) return rc;
  }
  const cudaError_t rc = cudaHostAlloc((void **)&slots, 2 * sizeof(CgState), cudaHostAllocMapped);
  if (rc != cudaSuccess) slots = nullptr;
  return rc;
}
CgMonitor::~CgMonitor() {
  for (cudaEvent_t e : ev)
    if (e) cudaEventDestroy(e);
  if (slots) cudaFreeHost(slots);
}

// Blocks of a tiled vector kernel, a tile each at least.  Up to eight per SM to stream
// from HBM (25 mixed iterations at 384^3: 5.71 ms each, with four 5.77), four
// where the vectors stay in L2 and the reduction over the blocks counts (104^3:
// 237.5 us against 233.7, 128^3: 322 against 317).
static int vector_blocks(int64_t n) {
  const int64_t b = (n + kTile - 1) / kTile;
  return (int)std::max<int64_t>(1, std::min<int64_t>(b, 148 * (n > (1 << 23) ? 8 : 4)));
}

// Blocks of k_dot, which writes nothing: five per SM where the vectors stream from
// HBM, at 512^3 335 us a call (eight: 357; one element per thread, before the tiles:
// 338), at 384^3 172 (184; 171), at 256^3 84 (85; 85).
static int dot_blocks(int64_t n) {
  return n > (1 << 23) ? std::min(vector_blocks(n), 148 * 5) : vector_blocks(n);
}

// Blocks of the kernels that take one element per thread and step (k_copy,
// k_copy_z, k_cg_xflush; with a reduction k_absmax_diff, k_cg_init), four elements
// a thread at least.  They have a quarter of a tiled kernel's loads under way and
// want more blocks: eight per SM, k_cg_xflush at 200^3 27.1 us (four: 36.6, twelve:
// 29.8), k_copy_z 17.3 (18.5, 18.1); at 384^3 198 us (twelve: 215).  A reduction
// takes as many as still sum in one level (grid_reduce): k_cg_init at 104^3 11.3 us
// (592 blocks: 12.4, 1099: 13.6), at 200^3 32.0 (38.3, 1184: 34.7), at 384^3 204
// (1184: 212); k_absmax_diff 9.1 (10.0, 11.5), 25.0 (27.1, 26.8), 132 (132).
static int element_blocks(int64_t n, bool reduces = false) {
  const int64_t b = (n + 4 * kThreads - 1) / (4 * kThreads);
  return (int)std::max<int64_t>(1, std::min<int64_t>(b, reduces ? kReduceGroup : 148 * 8));
}

int reduce_blocks(int64_t n) { return std::max(vector_blocks(n), element_blocks(n, true)); }

void plan_level(LevelDev &L, int nx, int ny, int nz) {
  L.nx = nx;
  L.ny = ny;
  L.nz = nz;
  L.n = (int64_t)nx * ny * nz;
  int64_t start = 0;
  for (int c = 0; c < 8; ++c) {
    const int px = c & 1, py = (c >> 1) & 1, pz = (c >> 2) & 1;
    const int64_t cx = (nx - px + 1) / 2, cy = (ny - py + 1) / 2, cz = (nz - pz + 1) / 2;
    L.ccount[c] = cx * cy * cz;
    L.cstart[c] = start;
    start += (L.ccount[c] + 31) / 32 * 32;
  }
  L.storage_rows = start;
  L.spmv_blocks = 0;
  for (int q = 0; q < 4; ++q) {
    ClassInfo &C = L.cls[q];
    C.q = q;
    C.py = q & 1;
    C.pz = q >> 1;
    C.nyq = (ny - C.py + 1) / 2;
    const int nzq = (nz - C.pz + 1) / 2;
    C.lines = C.nyq * nzq;
    C.len[0] = (nx + 1) / 2;
    C.len[1] = nx / 2;
    C.start[0] = L.cstart[2 * q];
    C.start[1] = L.cstart[2 * q + 1];
    C.dlen = make_fastdiv((uint32_t)C.len[0]);
    C.dnyq = make_fastdiv((uint32_t)C.nyq);
    L.spmv_blocks += (int)(((int64_t)C.lines * C.len[0] + kThreads - 1) / kThreads);
  }
}

int64_t storage_row_host(const LevelDev &L, int64_t row) {
  const int ix = (int)(row % L.nx), iy = (int)((row / L.nx) % L.ny),
            iz = (int)(row / ((int64_t)L.nx * L.ny));
  const int px = ix & 1, q = (iy & 1) + 2 * (iz & 1), c = px + 2 * q;
  const int64_t j = (int64_t)(iz >> 1) * L.cls[q].nyq + (iy >> 1);
  return L.cstart[c] + j * L.cls[q].len[px] + (ix >> 1);
}

int launch_generate_hpcg(const LevelDev &L, cudaStream_t s) {
  k_generate_hpcg<<<grid_for(L.storage_rows), kThreads, 0, s>>>(geo_of(L), L.storage_rows, L.vals);
  return 1;
}

int launch_generate_varcoef(const LevelDev &L, int level, int nx0, int ny0, uint64_t seed,
                            double sigma, cudaStream_t s) {
  k_generate_varcoef<<<grid_for(L.storage_rows), kThreads, 0, s>>>(
      geo_of(L), L.storage_rows, level, nx0, ny0, seed, sigma, L.vals);
  return 1;
}

int launch_coarsen_varcoef(const LevelDev &F, const LevelDev &Cc, cudaStream_t s) {
  k_coarsen_varcoef<<<grid_for(Cc.storage_rows), kThreads, 0, s>>>(geo_of(F), geo_of(Cc),
                                                                    Cc.storage_rows, F.vals, Cc.vals);
  return 1;
}

int launch_to_bf16(const LevelDev &L, cudaStream_t s) {
  k_to_bf16<<<grid_for(L.storage_rows * 3), kThreads, 0, s>>>(L.storage_rows, L.vals, L.vals16);
  return 1;
}

int launch_set_values(const LevelDev &L, const double *vals27, cudaStream_t s) {
  if (L.nx == 1 || L.ny == 1 || L.nz == 1)
    k_set_values_flat<<<grid_for(L.n), kThreads, 0, s>>>(geo_of(L), L.n, vals27, L.vals);
  else
    k_set_values<<<tiles_for(L.n), kThreads, 0, s>>>(geo_of(L), L.n, vals27, L.vals);
  return 1;
}

int launch_get_values(const LevelDev &L, double *vals27, int32_t *cols27, cudaStream_t s) {
  k_get_values<<<tiles_for(L.n), kThreads, 0, s>>>(geo_of(L), L.n, L.vals, vals27, cols27);
  return 1;
}

int launch_set_diagonal(const LevelDev &L, const double *diag, cudaStream_t s) {
  k_set_diagonal<<<grid_for(L.n), kThreads, 0, s>>>(geo_of(L), L.n, diag, L.vals);
  return 1;
}

int launch_get_diagonal(const LevelDev &L, double *diag, cudaStream_t s) {
  k_get_diagonal<<<grid_for(L.n), kThreads, 0, s>>>(geo_of(L), L.n, L.vals, diag);
  return 1;
}

// Rows from which the SpMV's dot product is summed by a launch of its own, after
// blocks of two turns.  With it fused each block ends in a fence and a counter,
// 0.3 us that keep its place on the SM: at 512^3, with 262,144 blocks of 5 us,
// p.Ap takes 4894 us fused and 4695 so (one row per thread and half the blocks,
// before the pairs: 4735), at 448^3 3216 and 3120, at 384^3 1979 and 1942, at 352^3
// 1509 and 1499; at 256^3 585 both, and below that the launch costs what it saves.
// (512^3 and 384^3 on another device, fused 4815 and 1944: so 4600 and 1920; one turn
// and a launch 4689 and 1939; two or four turns, fused, 4763 and 1988, 4652 and 1962.)
constexpr int64_t kDotLaunchRows = 1 << 25;

int launch_spmv(const LevelDev &L, const double *x, double *y, const Reduce *dot, int fin,
                void *fin_target, const int *done, cudaStream_t s) {
  if (L.spmv_blocks == 0) return 0;
  const int vec = L.nx % 2 == 0 && aligned2(x) && aligned2(y);
  const LevelMat<double> A = mat_of(L, L.vals);
  const Reduce red = dot ? *dot : Reduce();
  const bool parts = dot && L.n >= kDotLaunchRows;
  const ClassSet cs = classes_of(L, parts ? 2 : 1);
  auto go = [&](auto kernel) {
    launch_dependent(kernel, dim3(cs.total), dim3(kThreads), s, A, cs, x, y, vec, red, fin,
                     fin_target, done);
    return 1;
  };
  auto form = [&](auto dot_kind) {
    constexpr int D = decltype(dot_kind)::value;
    return L.holes ? go(k_spmv<double, double, D, FORM_HOLES>)
           : vec   ? go(k_spmv<double, double, D, FORM_WIDE>)
                   : go(k_spmv<double, double, D, FORM_SCALAR>);
  };
  if (!dot) return form(std::integral_constant<int, DOT_NONE>());
  if (!parts) return form(std::integral_constant<int, DOT_FUSED>());
  form(std::integral_constant<int, DOT_PARTS>());
  Reduce sums = red;   // the partials' own scratch follows them (reduce_scratch)
  sums.partials = red.partials + cs.total;
  launch_dependent(k_sum_partials, dim3((cs.total + kReduceGroup - 1) / kReduceGroup), dim3(kThreads),
                   s, (const double *)red.partials, (int64_t)cs.total, sums, fin, fin_target, done);
  return 2;
}

int launch_spmv32(const LevelDev &L, const float *x, float *y, cudaStream_t s) {
  if (L.spmv_blocks == 0) return 0;
  const ClassSet cs = classes_of(L);
  const int vec = L.nx % 2 == 0 && aligned2(x) && aligned2(y);
  auto go = [&](auto kernel) {
    launch_dependent(kernel, dim3(cs.total), dim3(kThreads), s, mat_of(L, L.vals16), cs, x, y, vec,
                     Reduce(), 0, (void *)nullptr, (const int *)nullptr);
    return 1;
  };
  return vec ? go(k_spmv<uint16_t, float, DOT_NONE, FORM_WIDE>)
             : go(k_spmv<uint16_t, float, DOT_NONE, FORM_SCALAR>);
}

template <class T>
struct ValsOf;
template <>
struct ValsOf<double> {
  using VT = double;
  static const double *get(const LevelDev &L) { return L.vals; }
};
template <>
struct ValsOf<float> {
  using VT = uint16_t;
  static const uint16_t *get(const LevelDev &L) { return L.vals16; }
};

// Pairs of a class from which the BF16 sweeps give up registers (105 -> 80, a
// few spilled) for a third block per SM: with several waves of blocks another
// block hides a block's latency (V-cycle at 384^3 3292 us against 3814), with
// about one wave it does not come to run (64^3: 218 against 228 us).
constexpr int64_t kManyPairs = 100000;

// The block of a class launch: whole lines.  FP64: a pair needs some 220
// registers, so two blocks of 128 threads share an SM and one loads while the
// other computes (V-cycle at 256^3: 2490 us against 2623 with blocks of 256; 128
// registers for two blocks of 256 spill: 4061).  BF16: blocks of up to 256; of
// 128 in a large class whose lines fill them (mixed iteration at 256^3 1728 us
// against 1757, at 128^3 310 against 315), not where threads would idle or a
// block would be shorter (lines of 192, 96 and 48 pairs, 384^3: 5630 against
// 5611).  A class of few lines takes fewer lines per block so that there is a
// block for each SM twice over (a launch is then bound by one block's latency).
// Lines longer than that (FP64: of more than 128 pairs) go a block each, in chunks.
// Their sweep takes one round of chunks after another, as many as waves of blocks
// times chunks of a line, whatever the block's size, for the registers keep the
// warps of an SM to the same number (FP64 8, BF16 with three blocks of 256 per SM
// 24).  FP64 takes 128 threads, or the one of 256 and 64 that saves a twentieth of
// the rounds and more; BF16 256, or 160 or 192 for a fifth.  Symmetric FP64 sweep,
// us, with 64 / 128 / 256 threads (one row per thread, before the pairs): 258 x 200
// x 200 876 / 1071 / 1159 (1054), 514 x 128 x 128 697 / 753 / 958 (905), 700 x 100 x
// 100 612 / 574 / 680 (789), 2048 x 64 x 64 702 / 702 / 666 (1012), 700 x 32 x 32 123
// / 95 / 106 (130); 384^3 3857 with 64, 4480 with 192 (5359); from a view at an odd
// element 514 x 128 x 128 709 / 763 / 1009 (902), 384^3 3955 with 64 (5380).  BF16,
// 256 / 192 / 160: 514 x 128 x 128 327 / 289 / 283 (339), at an odd element 367 / 324
// / 317 (340), 1026 x 64 x 64 181 / 159 / 174 (194), 3000 x 50 x 50 316 / 320 / 345
// (340).
struct GsBlock {
  int lines, threads;
};
int64_t gs_rounds(const ClassInfo &C, int threads, int per_sm) {
  const int64_t waves = (C.lines + 148 * per_sm - 1) / (148 * per_sm);
  return waves * ((C.len[0] + threads - 1) / threads);
}
template <class T>
int chunk_threads(const ClassInfo &C) {
  constexpr bool fp64 = std::is_same<T, double>::value;
  struct { int threads, per_sm; } const size[2][3] = {{{256, 3}, {160, 5}, {192, 4}},
                                                      {{128, 2}, {256, 1}, {64, 4}}};
  const auto &s = size[fp64];
  int best = 0;
  int64_t most = 0;   // rounds that a size may take to be chosen
  for (int i = 0; i < 3; ++i) {
    const int64_t r = gs_rounds(C, s[i].threads, s[i].per_sm);
    if (i > 0 && r > most) continue;
    best = i;
    most = i > 0 ? r - 1 : fp64 ? r * 19 / 20 : r * 4 / 5;
  }
  return s[best].threads;
}
template <class T>
GsBlock gs_block(const ClassInfo &C) {
  const int len = C.len[0];
  constexpr bool fp64 = std::is_same<T, double>::value;
  if (fp64 ? len > 128 : len > kThreads && (int64_t)C.lines * len > kManyPairs)
    return {1, std::min(chunk_threads<T>(C), (len + 31) / 32 * 32)};
  const bool fills = (int64_t)C.lines * len > kManyPairs && 128 / len * len >= 120;
  const int target = fp64 || fills ? 128 : kThreads;
  const int lines = std::min(std::max(1, target / len), std::max(1, C.lines / (2 * 148)));
  return {lines, std::min(kThreads, (lines * len + 31) / 32 * 32)};
}

// The class kernels, by blocks per SM and form (k_gs_class).
template <int MINB, int FORM, class T, class RT>
int launch_gs_rows(const LevelDev &L, int q, int backward, int mode, const RT *r, T *x,
                   const T *xc, T *rc, const int *done, cudaStream_t s, int jbeg, int jend,
                   GsBlock gb, int vec) {
  using VT = typename ValsOf<T>::VT;
  const LevelMat<VT> A = mat_of(L, ValsOf<T>::get(L));
  const dim3 g((unsigned)((jend - jbeg + gb.lines - 1) / gb.lines)), b(gb.threads);
  const ClassInfo &C = L.cls[q];
  auto go = [&](auto kernel) {
    launch_dependent(kernel, g, b, s, A, C, gb.lines, jbeg, jend, vec, r, x, xc, rc, done);
    return 1;
  };
  if (mode == GS_SYM3 && q == 3) return go(k_gs_class<GS_SYM3, 0, 3, MINB, FORM, VT, T, RT>);
  if (mode == (GS_SYM3 | GS_ZERO_GUESS) && q == 3)
    return go(k_gs_class<GS_SYM3 | GS_ZERO_GUESS, 0, 3, MINB, FORM, VT, T, RT>);
  if (mode == GS_ZERO_GUESS && !backward) {
    switch (q) {
      case 0: return go(k_gs_class<GS_ZERO_GUESS, 0, 0, MINB, FORM, VT, T, RT>);
      case 1: return go(k_gs_class<GS_ZERO_GUESS, 0, 1, MINB, FORM, VT, T, RT>);
      case 2: return go(k_gs_class<GS_ZERO_GUESS, 0, 2, MINB, FORM, VT, T, RT>);
      default: return go(k_gs_class<GS_ZERO_GUESS, 0, 3, MINB, FORM, VT, T, RT>);
    }
  }
  if (mode == GS_RESTRICT && backward && q == 0)
    return go(k_gs_class<GS_RESTRICT, 1, 0, MINB, FORM, VT, T, RT>);
  if (mode == GS_PROLONG && !backward && q == 0)
    return go(k_gs_class<GS_PROLONG, 0, 0, MINB, FORM, VT, T, RT>);
  if (mode != GS_PLAIN) return 0;
  return backward ? go(k_gs_class<GS_PLAIN, 1, -1, MINB, FORM, VT, T, RT>)
                  : go(k_gs_class<GS_PLAIN, 0, -1, MINB, FORM, VT, T, RT>);
}

template <class T, class RT>
int launch_gs_class(const LevelDev &L, int q, int backward, int mode, const RT *r, T *x,
                    const T *xc, T *rc, const int *done, cudaStream_t s, int jbeg, int jend) {
  if (jend < 0) jend = L.cls[q].lines;
  if (jend <= jbeg) return 0;
  if ((mode & GS_SYM3) && (jbeg != 0 || jend != L.cls[q].lines)) return 0;   // whole class only
  const GsBlock gb = gs_block<T>(L.cls[q]);
  const int vec = L.nx % 2 == 0 && aligned2(x) && aligned2(r);
  constexpr bool fp64 = std::is_same<T, double>::value;
  const bool many = (int64_t)L.cls[q].lines * L.cls[q].len[0] > kManyPairs;
  auto rows = [&](auto minb, auto form) {
    return launch_gs_rows<decltype(minb)::value, decltype(form)::value>(L, q, backward, mode, r, x, xc, rc,
                                                                        done, s, jbeg, jend, gb, vec);
  };
  using std::integral_constant;
  constexpr integral_constant<int, FORM_WIDE> wide{};
  constexpr integral_constant<int, FORM_SCALAR> scalar{};
  if constexpr (fp64) {
    constexpr integral_constant<int, 1> one{};
    return L.holes ? rows(one, integral_constant<int, FORM_HOLES>()) : vec ? rows(one, wide) : rows(one, scalar);
  } else {
    constexpr integral_constant<int, 2> two{};
    constexpr integral_constant<int, 3> three{};
    return many ? (vec ? rows(three, wide) : rows(three, scalar))
                : (vec ? rows(two, wide) : rows(two, scalar));
  }
}

template <class T, class RT>
int launch_restrict_residual(const LevelDev &F, int64_t nc, const RT *rf, const T *xf, T *rc,
                             const int *done, cudaStream_t s) {
  if (nc <= 0) return 0;
  nc = std::min(nc, (int64_t)(F.nx / 2) * (F.ny / 2) * (F.nz / 2));
  k_restrict_residual<<<grid_for(nc), kThreads, 0, s>>>(mat_of(F, ValsOf<T>::get(F)), F.cls[0],
                                                        nc, rf, xf, rc, done);
  return 1;
}
template int launch_restrict_residual<double, double>(const LevelDev &, int64_t, const double *,
                                                      const double *, double *, const int *,
                                                      cudaStream_t);
template int launch_restrict_residual<float, double>(const LevelDev &, int64_t, const double *,
                                                     const float *, float *, const int *,
                                                     cudaStream_t);
template int launch_restrict_residual<float, float>(const LevelDev &, int64_t, const float *,
                                                    const float *, float *, const int *,
                                                    cudaStream_t);

template <class T>
int launch_prolong(const LevelDev &F, int64_t nc, const T *xc, T *xf, const int *done,
                   cudaStream_t s) {
  if (nc <= 0) return 0;
  nc = std::min(nc, (int64_t)(F.nx / 2) * (F.ny / 2) * (F.nz / 2));
  k_prolong<T><<<grid_for(nc), kThreads, 0, s>>>(nc, F.nx, F.ny, xc, xf, done);
  return 1;
}
template int launch_prolong<double>(const LevelDev &, int64_t, const double *, double *,
                                    const int *, cudaStream_t);
template int launch_prolong<float>(const LevelDev &, int64_t, const float *, float *, const int *,
                                   cudaStream_t);

int read_check_record(unsigned long long *record) {
  *record = 0ull;
#ifdef HPCGX_CHECKED
  cudaError_t e = cudaMemcpyFromSymbol(record, g_check_record, sizeof(*record));
  if (e != cudaSuccess) return (int)e;
  const unsigned long long zero = 0ull;
  e = cudaMemcpyToSymbol(g_check_record, &zero, sizeof(zero));
  if (e != cudaSuccess) return (int)e;
#endif
  return 0;
}

int launch_finish(int fin, int nv, const double *tot, CgState *st, cudaStream_t s) {
  if (nv == 2)
    k_finish<2><<<1, 1, 0, s>>>(fin, tot, st);
  else
    k_finish<1><<<1, 1, 0, s>>>(fin, tot, st);
  return 1;
}

int launch_rank_sum(int nranks, double *const *bufs, int count, cudaStream_t s) {
  k_rank_sum<<<1, 32, 0, s>>>(nranks, bufs, count);
  return 1;
}

template int launch_gs_class<double, double>(const LevelDev &, int, int, int, const double *,
                                             double *, const double *, double *, const int *,
                                             cudaStream_t, int, int);
template int launch_gs_class<float, double>(const LevelDev &, int, int, int, const double *,
                                            float *, const float *, float *, const int *,
                                            cudaStream_t, int, int);
template int launch_gs_class<float, float>(const LevelDev &, int, int, int, const float *,
                                           float *, const float *, float *, const int *,
                                           cudaStream_t, int, int);

// Calls go(std::true_type()) if every vector of the launch (null: not used)
// allows two-element accesses, else go(std::false_type()).
template <class F, class... T>
void by_width(F go, const T *...v) {
  if ((aligned2(v) && ...))
    go(std::true_type());
  else
    go(std::false_type());
}

int launch_waxpby(int64_t n, double alpha, const double *x, double beta, const double *y,
                  double *w, const int *done, cudaStream_t s) {
  by_width([&](auto wide) {
    k_waxpby<wide.value><<<vector_blocks(n), kThreads, 0, s>>>(n, alpha, x, beta, y, w, done);
  }, x, y, w);
  return 1;
}

int launch_dot(int64_t n, const double *x, const double *y, const Reduce &red, double *out,
               cudaStream_t s) {
  by_width([&](auto wide) {
    k_dot<wide.value><<<dot_blocks(n), kThreads, 0, s>>>(n, x, y, red, FIN_STORE, out, nullptr);
  }, x, y);
  return 1;
}

int launch_dot_finish(int64_t n, const double *x, const double *y, const Reduce &red, int fin,
                      CgState *st, cudaStream_t s) {
  by_width([&](auto wide) {
    k_dot<wide.value><<<dot_blocks(n), kThreads, 0, s>>>(n, x, y, red, fin, st, &st->done);
  }, x, y);
  return 1;
}

int launch_absmax_diff(int64_t n, const double *a, const double *b, const Reduce &red,
                       double *out, cudaStream_t s) {
  k_absmax_diff<<<element_blocks(n, true), kThreads, 0, s>>>(n, a, b, red, out);
  return 1;
}

int launch_restriction(int64_t nc, const LevelDev &F, const double *rf, const double *Axf,
                       double *rc, cudaStream_t s) {
  k_restriction<<<grid_for(nc), kThreads, 0, s>>>(nc, F.nx, F.ny, rf, Axf, rc);
  return 1;
}

int launch_prolongation(int64_t nc, const LevelDev &F, const double *xc, double *xf,
                        cudaStream_t s) {
  k_prolongation<<<grid_for(nc), kThreads, 0, s>>>(nc, F.nx, F.ny, xc, xf);
  return 1;
}

int launch_copy(int64_t n, const double *x, double *y, const int *done, cudaStream_t s) {
  k_copy<<<element_blocks(n), kThreads, 0, s>>>(n, x, y, done);
  return 1;
}

int launch_fill_uniform(int64_t n, uint64_t seed, uint64_t offset, double lo, double hi, double *v,
                        cudaStream_t s) {
  k_fill_uniform<<<grid_for(n), kThreads, 0, s>>>(n, seed, offset, lo, hi, v);
  return 1;
}

int launch_fill_normal(int64_t n, uint64_t seed, uint64_t offset, double *v, cudaStream_t s) {
  k_fill_normal<<<grid_for(n), kThreads, 0, s>>>(n, seed, offset, v);
  return 1;
}

int launch_cg_init(int64_t n, const double *b, const double *Ap, double *r, float *r32,
                   const Reduce &red, CgState *st, cudaStream_t s) {
  k_cg_init<<<element_blocks(n, true), kThreads, 0, s>>>(n, b, Ap, r, r32, red, st);
  return 1;
}

template <class ZT>
int launch_cg_rz(int64_t n, const double *r, const ZT *z, const double *Ap, const Reduce &red,
                 CgState *st, cudaStream_t s) {
  by_width([&](auto wide) {
    launch_dependent(Ap ? k_cg_rz<wide.value, ZT, true> : k_cg_rz<wide.value, ZT, false>,
                     dim3(vector_blocks(n)), dim3(kThreads), s, n, r, z, Ap, red, st);
  }, r, z, Ap);
  return 1;
}
template int launch_cg_rz<double>(int64_t, const double *, const double *, const double *,
                                  const Reduce &, CgState *, cudaStream_t);
template int launch_cg_rz<float>(int64_t, const double *, const float *, const double *,
                                 const Reduce &, CgState *, cudaStream_t);

template <class ZT>
int launch_cg_p(int64_t n, const ZT *z, double *p, CgState *st, cudaStream_t s, double *x) {
  by_width([&](auto wide) {
    launch_dependent(k_cg_p<wide.value, ZT>, dim3(vector_blocks(n)), dim3(kThreads), s, n, z, p,
                     (const CgState *)st, x);
  }, z, p, x);
  return 1;
}
template int launch_cg_p<double>(int64_t, const double *, double *, CgState *, cudaStream_t,
                                 double *);
template int launch_cg_p<float>(int64_t, const float *, double *, CgState *, cudaStream_t,
                                double *);

int launch_cg_xflush(int64_t n, const double *p, double *x, const CgState *st, cudaStream_t s) {
  k_cg_xflush<<<element_blocks(n), kThreads, 0, s>>>(n, p, x, st);
  return 1;
}

int launch_cg_xr(int64_t n, const double *p, const double *Ap, double *x, double *r, float *r32,
                 const Reduce &red, CgState *st, cudaStream_t s) {
  by_width([&](auto wide) {
    launch_dependent(k_cg_xr<wide.value>, dim3(vector_blocks(n)), dim3(kThreads), s, n, p, Ap, x, r,
                     r32, red, st);
  }, p, Ap, x, r, r32);
  return 1;
}

int launch_copy_z(int64_t n, const double *r, double *z, const CgState *st, cudaStream_t s) {
  k_copy_z<<<element_blocks(n), kThreads, 0, s>>>(n, r, z, st);
  return 1;
}

int launch_adjoint_grad(const LevelDev &L, const double *lambda, const double *x, double *grad,
                        cudaStream_t s) {
  k_adjoint_grad<<<tiles_for(L.n), kThreads, 0, s>>>(geo_of(L), L.n, lambda, x, grad);
  return 1;
}

}  // namespace hpcgx
