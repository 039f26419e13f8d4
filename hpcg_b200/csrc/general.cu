// general.cu -- the reference operators on a general sparse matrix (any
// pattern); see general.cuh for the layout and what each operator restates.
#include "general.cuh"

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstring>
#include <memory>
#include <string>
#include <thread>
#include <vector>

#include "../../include/hpcgx.h"
#include "kernels.cuh"

namespace hpcgx {

int set_error(int code, const char *msg);

namespace {

constexpr int kT = 256;
// Rows up to which a level is one block's (k_gen_small).  Solves of the renumbered
// HPCG hierarchy, ms, without / up to 300 / 2000 / 4096 rows: 48^3 27.4 / 27.0 /
// 24.9 / 24.6, 32^3 15.4 / 14.8 / 13.2 / 14.1, 16^3 6.5 / 5.9 / 5.1 / 5.5 (where a
// level has 4096); up to 14000 rows, 48^3 takes 39.
constexpr int64_t kSmallRows = 2048;

// ------------------------------------------------------------------ kernels

// Entry j of storage row k: slice k / 32, lane k % 32, entries of a slice
// interleaved across its 32 rows (a warp's loads of entry j are contiguous).
__device__ __forceinline__ int64_t gen_entry(const int64_t *__restrict__ slice_off, int64_t k,
                                             int j) {
  return slice_off[k >> 5] + (int64_t)j * 32 + (k & 31);
}

// What a kernel needs of one level.
struct GenMat {
  int64_t n;
  const int64_t *slice_off;
  const uint8_t *nnz;
  const int32_t *perm, *cols;
  const double *vals, *diag;
};

// The entries of a storage row, kChunk at a time: their columns and values are
// loaded together and then their x entries together, so that a row waits for
// memory twice per chunk and not twice per entry (the sums keep the row's own
// order).  The padding up to the slice's width (value 0, column 0) is not read.
// Rows of up to 27 entries are one chunk.
constexpr int kChunk = 27;
struct GenRow {
  int m = 0;          // entries; 0: no row
  int32_t i = 0;      // natural index
  int64_t base = 0;
  int32_t c[kChunk];
  double v[kChunk];
};
__device__ __forceinline__ void gen_load(const GenMat &A, GenRow &w, int j0) {
#pragma unroll
  for (int j = 0; j < kChunk; ++j) {
    w.c[j] = 0;
    w.v[j] = 0.0;
    if (j0 + j < w.m) {
      w.c[j] = __ldg(A.cols + w.base + (int64_t)(j0 + j) * 32);
      w.v[j] = __ldg(A.vals + w.base + (int64_t)(j0 + j) * 32);
    }
  }
}
// The row's index and its first chunk: nothing that another kernel writes, so
// it may go before dependency_wait.
__device__ __forceinline__ void gen_begin(const GenMat &A, int64_t k, GenRow &w) {
  w.m = __ldg(A.nnz + k);
  w.i = __ldg(A.perm + k);
  w.base = __ldg(A.slice_off + (k >> 5)) + (k & 31);
  gen_load(A, w, 0);
}
template <class F>
__device__ __forceinline__ void gen_sum(const GenMat &A, GenRow &w, const double *x, F add) {
  for (int j0 = 0;;) {
    double xv[kChunk];
#pragma unroll
    for (int j = 0; j < kChunk; ++j) xv[j] = j0 + j < w.m ? x[w.c[j]] : 0.0;
#pragma unroll
    for (int j = 0; j < kChunk; ++j)
      if (j0 + j < w.m) add(w.v[j], xv[j]);
    j0 += kChunk;
    if (j0 >= w.m) break;
    gen_load(A, w, j0);
  }
}

// y_i = (A x)_i of storage row k (src/ComputeSPMV_ref.cpp:58-71: a sum from 0
// over the row's entries in order, each product and sum rounded on its own).
__device__ __forceinline__ double gen_product(const GenMat &A, GenRow &w, const double *x) {
  double sum = 0.0;
  gen_sum(A, w, x, [&](double v, double xj) { sum = __dadd_rn(sum, __dmul_rn(v, xj)); });
  return sum;
}

__global__ void __launch_bounds__(kT)
k_gen_spmv(GenMat A, const double *x, double *y, const int *done) {
  dependents_launch();
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  GenRow w;
  if (k < A.n) gen_begin(A, k, w);
  dependency_wait();
  if (done && *done) return;
  if (k < A.n) y[w.i] = gen_product(A, w, x);
}

// The Gauss-Seidel update of the storage rows [k0, k1) of one colour
// (src/ComputeSYMGS_ref.cpp:72-80): sum = r_i - sum_j a_ij x_j over the row's
// entries (diagonal included), sum += x_i a_ii, x_i = sum / a_ii.  Rows of one
// colour share no entry, so they update in parallel.  Bound by latency (a
// colour of the 48^3 hierarchy has at most some 7000 rows, and a V-cycle 230
// colour launches): a thread that walked its row entry by entry, each x entry
// behind its column, took 8.5 us a launch; with the row's entries loaded
// together, its matrix data under the end of the launch before (dependent
// launch), the V-cycle went from 2443 to 741 us, a solve to 1e-10 from 80 to
// 27 ms.  One cluster walking through a level's colours with a barrier between
// them instead of a launch per colour measured 2.7 us a colour, the launches
// without the overlap 4.2.
__global__ void __launch_bounds__(kT)
k_gen_gs(GenMat A, int64_t k0, int64_t k1, const double *r, double *x, const int *done) {
  dependents_launch();
  const int64_t k = k0 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  GenRow w;
  double d = 1.0;
  if (k < k1) {
    gen_begin(A, k, w);
    d = __ldg(A.diag + k);
  }
  dependency_wait();
  if (done && *done) return;
  if (k >= k1) return;
  const double xi = x[w.i];
  double sum = r[w.i];
  gen_sum(A, w, x, [&](double v, double xj) { sum = __dsub_rn(sum, __dmul_rn(v, xj)); });
  sum = __dadd_rn(sum, __dmul_rn(xi, d));
  x[w.i] = __ddiv_rn(sum, d);
}

// src/ComputeRestriction_ref.cpp:51 and src/ComputeProlongation_ref.cpp:49
// through a given injection f2c.  The residual is formed at the injected rows
// alone (pos: their storage rows): the others are never read.
__global__ void __launch_bounds__(kT)
k_gen_restrict(GenMat A, int64_t nc, const int32_t *__restrict__ pos, const double *rf, const double *xf, double *rc,
               const int *done) {
  dependents_launch();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  GenRow w;
  if (i < nc) gen_begin(A, pos[i], w);
  dependency_wait();
  if (done && *done) return;
  if (i < nc) rc[i] = __dsub_rn(rf[w.i], gen_product(A, w, xf));
}

__global__ void k_gen_prolong(int64_t nc, const int32_t *__restrict__ f2c, const double *xc,
                              double *xf, const int *done) {
  dependents_launch();
  dependency_wait();
  if (done && *done) return;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nc;
       i += (int64_t)gridDim.x * blockDim.x)
    xf[f2c[i]] = __dadd_rn(xf[f2c[i]], xc[i]);
}

__global__ void k_gen_zero(int64_t n, double *x, const int *done) {
  dependents_launch();
  dependency_wait();
  if (done && *done) return;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    x[i] = 0.0;
}

// ---- the small levels of a V-cycle in one block and one launch
//
// Below a few thousand rows a colour launch is bound by its latency, some 3 us
// whatever it updates, and a level has a launch per colour and direction.  One
// block walks through the colours with a block barrier between them; a thread
// has the entries of its row of the next colour in registers before it waits.
struct GenSmallLevel {
  GenMat A;
  int ncolors;
  const int64_t *cstart;
  const double *r;
  double *x;
  int64_t nc;
  const int32_t *f2c, *f2k;
};
struct GenSmallArgs {
  int n;
  GenSmallLevel l[kMaxLevels];
};

__device__ __forceinline__ void gen_update(const GenMat &A, GenRow &w, double d, double r,
                                           double *x) {
  const double xi = x[w.i];
  double sum = r;
  gen_sum(A, w, x, [&](double v, double xj) { sum = __dsub_rn(sum, __dmul_rn(v, xj)); });
  sum = __dadd_rn(sum, __dmul_rn(xi, d));
  x[w.i] = __ddiv_rn(sum, d);
}

__global__ void __launch_bounds__(kT, 1)
k_gen_small(const __grid_constant__ GenSmallArgs a, const int *done) {
  __shared__ int cs[kT + 1];   // colour starts of the level (a row has at most 255 entries)
  dependents_launch();
  dependency_wait();
  if (done && *done) return;
  const int t = threadIdx.x, last = a.n - 1;
#pragma unroll 1
  for (int s = 0; s <= 2 * last; ++s) {
    const bool down = s <= last;
    const GenSmallLevel &L = a.l[down ? s : 2 * last - s];
    const int n = (int)L.A.n, nc = (int)L.nc, C = L.ncolors;
    for (int c = t; c <= C; c += kT) cs[c] = (int)L.cstart[c];
    if (down) {
      for (int i = t; i < n; i += kT) L.x[i] = 0.0;
    } else {
      const double *xc = (&L)[1].x;
      for (int i = t; i < nc; i += kT) L.x[L.f2c[i]] = __dadd_rn(L.x[L.f2c[i]], xc[i]);
    }
    __syncthreads();
    GenRow w;
    double d = 1.0, r = 0.0;
    auto fetch = [&](int c) {
      const int k = cs[c] + t;
      w.m = 0;
      if (k >= cs[c + 1]) return;
      gen_begin(L.A, k, w);
      d = __ldg(L.A.diag + k);
      r = L.r[w.i];
    };
    fetch(0);
    // colours 0 .. C-1, then C-1 .. 0
#pragma unroll 1
    for (int e = 0; e < 2 * C; ++e) {
      const int c = e < C ? e : 2 * C - 1 - e;
      if (w.m > 0) gen_update(L.A, w, d, r, L.x);
      for (int k = cs[c] + t + kT; k < cs[c + 1]; k += kT) {
        GenRow o;
        gen_begin(L.A, k, o);
        gen_update(L.A, o, L.A.diag[k], L.r[o.i], L.x);
      }
      if (e + 1 == 2 * C) break;
      // the last colour forward and the first one backward are the same rows,
      // which this thread updates both times (from their first chunk on)
      if (e + 1 != C) fetch(e + 1 < C ? e + 1 : 2 * C - 2 - e);
      else if (w.m > kChunk) gen_load(L.A, w, 0);
      if (e + 1 != C) __syncthreads();
    }
    __syncthreads();
    if (down && s < last) {
      double *rc = const_cast<double *>((&L)[1].r);
      for (int i = t; i < nc; i += kT) {
        GenRow o;
        gen_begin(L.A, L.f2k[i], o);
        rc[i] = __dsub_rn(L.r[o.i], gen_product(L.A, o, L.x));
      }
      __syncthreads();
    }
  }
}

// Writes (set) or reads the diagonal of every row, natural order.
__global__ void k_gen_diag(int64_t n, const int64_t *__restrict__ slice_off,
                           const int32_t *__restrict__ perm, const uint8_t *__restrict__ dpos,
                           double *vals, double *diag, double *nat, int set) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
       k += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e = gen_entry(slice_off, k, dpos[k]);
    if (set) {
      vals[e] = nat[perm[k]];
      diag[k] = nat[perm[k]];
    } else {
      nat[perm[k]] = diag[k];
    }
  }
}

int grid(int64_t n) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((n + kT - 1) / kT, 148 * 16));
}
// One thread per row: blocks small enough that a colour of a few thousand rows
// spreads over the SMs.
int row_threads(int64_t n) { return n >= 148 * 2 * kT ? kT : 64; }
dim3 row_grid(int64_t n) { return dim3((unsigned)((n + row_threads(n) - 1) / row_threads(n))); }

template <class F>
void host_parallel(int64_t n, F f) {
  const unsigned hw = std::thread::hardware_concurrency();
  const int64_t nt = std::max<int64_t>(1, std::min<int64_t>(hw ? hw : 1, 64));
  if (n < 65536 || nt == 1) {
    f(0, n);
    return;
  }
  std::vector<std::thread> ts;
  const int64_t chunk = (n + nt - 1) / nt;
  for (int64_t t = 0; t < nt; ++t) {
    const int64_t a = t * chunk, b = std::min(n, a + chunk);
    if (a < b) ts.emplace_back(f, a, b);
  }
  for (auto &th : ts) th.join();
}

}  // namespace

// ------------------------------------------------------------------ host side

struct GLevel {
  int64_t n = 0, nc = 0, entries = 0;
  int ncolors = 0;
  std::vector<int64_t> cstart;     // storage row of the first row of each colour (+ end)
  int64_t *dcstart = nullptr;      // the same on the device
  int64_t *slice_off = nullptr;
  uint8_t *nnz = nullptr, *dpos = nullptr;
  int32_t *perm = nullptr, *cols = nullptr, *f2c = nullptr;
  int32_t *f2k = nullptr;          // storage row of f2c[i]
  double *vals = nullptr, *diag = nullptr;
  double *r = nullptr, *x = nullptr, *Axf = nullptr;   // V-cycle work vectors
  bool loaded = false;
  GenMat mat() const { return GenMat{n, slice_off, nnz, perm, cols, vals, diag}; }
};

struct GeneralProblem {
  int nlev = 0;
  cudaStream_t stream = nullptr;
  GLevel L[kMaxLevels];
  std::vector<void *> allocs;
  double bytes = 0.0;
  int64_t launches = 0;
  // CG
  double *r = nullptr, *z = nullptr, *p = nullptr, *Ap = nullptr;
  double *x = nullptr;             // the solution vector of the graphs
  CgState *st = nullptr;
  Reduce red;
  // one iteration without and with preconditioner, without [0] and with [1] the
  // events that time its phases
  cudaGraphExec_t graph[2][2] = {};
  cudaEvent_t phase[2][5] = {};
  bool timed = false;              // capturing with events
  CgMonitor monitor;

  int alloc(void **ptr, size_t n) {
    cudaError_t e = cudaMalloc(ptr, std::max<size_t>(n, 8));
    if (e != cudaSuccess) {
      *ptr = nullptr;
      cudaGetLastError();
      return set_error(HPCGX_ENOMEM, ("cudaMalloc of " + std::to_string(n) + " bytes failed").c_str());
    }
    allocs.push_back(*ptr);
    bytes += (double)n;
    return HPCGX_OK;
  }
  ~GeneralProblem() {
    for (int k = 0; k < 2; ++k) {
      for (cudaGraphExec_t exec : graph[k])
        if (exec) cudaGraphExecDestroy(exec);
      for (cudaEvent_t &ev : phase[k])
        if (ev) cudaEventDestroy(ev);
    }
    for (void *ptr : allocs) cudaFree(ptr);
  }
  void note(int k) { launches += k; }

  // ---- operators (launches only; the caller synchronises)
  void spmv(int l, const double *x, double *y, const int *done) {
    const GLevel &A = L[l];
    launch_dependent(k_gen_spmv, row_grid(A.n), dim3(row_threads(A.n)), stream, A.mat(), x, y, done);
    note(1);
  }
  void symgs(int l, const double *r, double *x, const int *done) {
    const GLevel &A = L[l];
    auto colour = [&](int c) {
      const int64_t k0 = A.cstart[c], k1 = A.cstart[c + 1];
      if (k1 > k0) {
        launch_dependent(k_gen_gs, row_grid(k1 - k0), dim3(row_threads(k1 - k0)), stream, A.mat(),
                         k0, k1, r, x, done);
        note(1);
      }
    };
    for (int c = 0; c < A.ncolors; ++c) colour(c);
    for (int c = A.ncolors - 1; c >= 0; --c) colour(c);
  }
  // The first of the small levels, and their part of the V-cycle.
  int small_from() const {
    int l = nlev;
    while (l > 0 && L[l - 1].n <= kSmallRows && L[l - 1].ncolors <= kT) --l;
    return l;
  }
  void small(int l, const double *r, double *x, const int *done) {
    GenSmallArgs a;
    a.n = nlev - l;
    for (int i = 0; i < a.n; ++i) {
      const GLevel &A = L[l + i];
      a.l[i] = GenSmallLevel{A.mat(), A.ncolors, A.dcstart, i ? A.r : r, i ? A.x : x,
                             A.nc, A.f2c, A.f2k};
    }
    launch_dependent(k_gen_small, dim3(1), dim3(kT), stream, a, done);
    note(1);
  }
  // src/ComputeMG_ref.cpp:39-63, one pre- and one post-smoothing sweep
  // (src/MGData.hpp:51-52).
  void mg(int l, const double *r, double *x, const int *done) {
    if (l >= small_from()) {
      small(l, r, x, done);
      return;
    }
    const GLevel &A = L[l];
    launch_dependent(k_gen_zero, dim3(grid(A.n)), dim3(kT), stream, A.n, x, done);
    note(1);
    symgs(l, r, x, done);
    if (l + 1 < nlev) {
      GLevel &C = L[l + 1];
      launch_dependent(k_gen_restrict, row_grid(A.nc), dim3(row_threads(A.nc)), stream, A.mat(),
                       A.nc, A.f2k, r, x, C.r, done);
      mg(l + 1, C.r, C.x, done);
      launch_dependent(k_gen_prolong, dim3(grid(A.nc)), dim3(kT), stream, A.nc, A.f2c, C.x, x, done);
      note(2);
      symgs(l, r, x, done);
    }
  }
  // One CG iteration (src/CG.cpp:100-130) on the device scalars of st.
  void iteration(int precond, double *x) {
    const int64_t n = L[0].n;
    const int *done = &st->done;
    if (timed) cudaEventRecordWithFlags(phase[precond][0], stream, cudaEventRecordExternal);
    if (precond)
      mg(0, r, z, done);
    else
      note(launch_copy_z(n, r, z, st, stream));
    if (timed) cudaEventRecordWithFlags(phase[precond][1], stream, cudaEventRecordExternal);
    note(launch_cg_rz<double>(n, r, z, nullptr, red, st, stream));
    note(launch_cg_p<double>(n, z, p, st, stream));
    if (timed) cudaEventRecordWithFlags(phase[precond][2], stream, cudaEventRecordExternal);
    spmv(0, p, Ap, done);
    note(launch_dot_finish(n, p, Ap, red, FIN_CG_PAP, st, stream));
    if (timed) cudaEventRecordWithFlags(phase[precond][3], stream, cudaEventRecordExternal);
    note(launch_cg_xr(n, p, Ap, x, r, nullptr, red, st, stream));
    if (timed) cudaEventRecordWithFlags(phase[precond][4], stream, cudaEventRecordExternal);
  }
};

#define GTRY(x)                     \
  do {                              \
    const int rc_ = (x);            \
    if (rc_ != HPCGX_OK) return rc_; \
  } while (0)
#define GCK(x)                                                           \
  do {                                                                   \
    const cudaError_t e_ = (x);                                          \
    if (e_ != cudaSuccess) {                                             \
      cudaGetLastError();                                                \
      return set_error(HPCGX_ECUDA, cudaGetErrorString(e_));             \
    }                                                                    \
  } while (0)

GeneralProblem *general_create(int nlev, cudaStream_t s) {
  GeneralProblem *g = new GeneralProblem;
  g->nlev = nlev;
  g->stream = s;
  return g;
}

void general_destroy(GeneralProblem *g) { delete g; }
void general_set_stream(GeneralProblem *g, cudaStream_t s) {
  g->stream = s;
  for (auto &kind : g->graph)
    for (cudaGraphExec_t &exec : kind)
      if (exec) {
        cudaGraphExecDestroy(exec);
        exec = nullptr;
      }
}

int64_t general_rows(const GeneralProblem *g, int level) {
  return (level >= 0 && level < g->nlev) ? g->L[level].n : -1;
}
int general_colours(const GeneralProblem *g, int level) {
  return (level >= 0 && level < g->nlev) ? g->L[level].ncolors : -1;
}
bool general_ready(const GeneralProblem *g) {
  for (int l = 0; l < g->nlev; ++l)
    if (!g->L[l].loaded) return false;
  return true;
}
double general_bytes(const GeneralProblem *g) { return g->bytes; }
int64_t general_launches(const GeneralProblem *g) { return g->launches; }

int general_load_level(GeneralProblem *g, int level, int64_t n, const char *nnz,
                       const int32_t *const *cols, const double *const *vals, const int32_t *f2c,
                       int64_t nc, const char **msg) {
  static thread_local std::string why;
  auto reject = [&](const std::string &m) {
    why = m;
    *msg = why.c_str();
    return HPCGX_ELAYOUT;
  };
  *msg = nullptr;
  if (level < 0 || level >= g->nlev) return set_error(HPCGX_EINVAL, "level out of range");
  if (g->L[level].loaded) return set_error(HPCGX_ESTATE, "level already loaded");
  if (n < 1 || n >= ((int64_t)1 << 31)) return set_error(HPCGX_EINVAL, "row count out of range");
  if (level > 0 && n != g->L[level - 1].nc)
    return set_error(HPCGX_EINVAL, "rows differ from the finer level's coarse row count");
  const bool coarse = level + 1 < g->nlev;
  if (coarse && (!f2c || nc < 1 || nc > n))
    return set_error(HPCGX_EINVAL, "every level but the last needs its injection f2c");
  GLevel &A = g->L[level];
  // ---- checks: entries in range, one diagonal entry per row (on the host's
  // cores; the failing row with the lowest index is reported)
  std::vector<uint8_t> dposn(n);
  auto check_row = [&](int64_t i, const char **why_row) {
    const int m = (unsigned char)nnz[i];
    if (m < 1) {
      *why_row = "no entries";
      return false;
    }
    int d = -1;
    for (int j = 0; j < m; ++j) {
      const int32_t c = cols[i][j];
      if (c < 0 || c >= n) {
        *why_row = "column out of range";
        return false;
      }
      if (c == i && d < 0) d = j;
    }
    if (d < 0) {
      *why_row = "no diagonal entry";
      return false;
    }
    dposn[i] = (uint8_t)d;
    return true;
  };
  std::atomic<int64_t> bad{n};
  host_parallel(n, [&](int64_t a, int64_t b) {
    const char *why_row = nullptr;
    for (int64_t i = a; i < b; ++i)
      if (!check_row(i, &why_row)) {
        int64_t seen = bad.load();
        while (i < seen && !bad.compare_exchange_weak(seen, i)) {
        }
        return;
      }
  });
  if (bad.load() < n) {
    const char *why_row = "";
    check_row(bad.load(), &why_row);
    return reject("row " + std::to_string(bad.load()) + ": " + why_row);
  }
  if (coarse)
    for (int64_t i = 0; i < nc; ++i)
      if (f2c[i] < 0 || f2c[i] >= n) return reject("f2c entry out of range");
  // ---- greedy multicolouring in natural row order, the algorithm of
  // src/OptimizeProblem.cpp:50-79: row i takes the lowest colour that no
  // already coloured neighbour (column < i) has.
  std::vector<int32_t> colour(n, -1);
  int total = 1;
  colour[0] = 0;
  std::vector<char> used;
  for (int64_t i = 1; i < n; ++i) {
    used.assign(total + 1, 0);
    const int m = (unsigned char)nnz[i];
    for (int j = 0; j < m; ++j) {
      const int32_t c = cols[i][j];
      if (c < i) used[colour[c]] = 1;
    }
    int pick = 0;
    while (pick < total && used[pick]) ++pick;
    if (pick == total) ++total;
    colour[i] = pick;
  }
  A.ncolors = total;
  // ---- storage order: colour-major, natural order inside a colour
  A.cstart.assign(total + 1, 0);
  for (int64_t i = 0; i < n; ++i) A.cstart[colour[i] + 1]++;
  for (int c = 0; c < total; ++c) A.cstart[c + 1] += A.cstart[c];
  std::vector<int32_t> perm(n);
  {
    std::vector<int64_t> next(A.cstart.begin(), A.cstart.end() - 1);
    for (int64_t i = 0; i < n; ++i) perm[next[colour[i]]++] = (int32_t)i;
  }
  // ---- sliced ELL: slice s (storage rows 32s .. 32s+31) is as wide as its
  // longest row; padding entries hold value 0 and column 0 and are never read
  const int64_t slices = (n + 31) / 32;
  std::vector<int64_t> off(slices + 1, 0);
  for (int64_t s = 0; s < slices; ++s) {
    int w = 0;
    for (int64_t k = 32 * s; k < std::min(n, 32 * s + 32); ++k)
      w = std::max(w, (int)(unsigned char)nnz[perm[k]]);
    off[s + 1] = off[s] + 32 * (int64_t)w;
  }
  const int64_t entries = off[slices];
  // staging written by the host's threads in one pass, padding included
  // (no serial zero-fill of the 12 B per entry first)
  std::unique_ptr<int32_t[]> hcp(new int32_t[entries]);
  std::unique_ptr<double[]> hvp(new double[entries]);
  int32_t *hc = hcp.get();
  double *hv = hvp.get();
  std::vector<uint8_t> hn(n), hd(n);
  std::vector<double> hdiag(n);
  host_parallel(n, [&](int64_t a, int64_t b) {
    for (int64_t k = a; k < b; ++k) {
      const int32_t i = perm[k];
      const int m = (unsigned char)nnz[i];
      hn[k] = (uint8_t)m;
      hd[k] = dposn[i];
      hdiag[k] = vals[i][dposn[i]];
      const int64_t sl = k >> 5, base = off[sl] + (k & 31);
      const int w = (int)((off[sl + 1] - off[sl]) / 32);
      for (int j = 0; j < m; ++j) {
        hc[base + 32 * j] = cols[i][j];
        hv[base + 32 * j] = vals[i][j];
      }
      for (int j = m; j < w; ++j) {
        hc[base + 32 * j] = 0;
        hv[base + 32 * j] = 0.0;
      }
    }
  });
  // lanes of the last slice past the last row
  for (int64_t k = n; k < 32 * slices; ++k) {
    const int64_t sl = k >> 5, base = off[sl] + (k & 31);
    for (int64_t j = 0; j < (off[sl + 1] - off[sl]) / 32; ++j) {
      hc[base + 32 * j] = 0;
      hv[base + 32 * j] = 0.0;
    }
  }
  // ---- device copies
  A.n = n;
  A.nc = coarse ? nc : 0;
  A.entries = entries;
  GTRY(g->alloc((void **)&A.slice_off, (slices + 1) * sizeof(int64_t)));
  GTRY(g->alloc((void **)&A.nnz, n));
  GTRY(g->alloc((void **)&A.dpos, n));
  GTRY(g->alloc((void **)&A.perm, n * sizeof(int32_t)));
  GTRY(g->alloc((void **)&A.dcstart, A.cstart.size() * sizeof(int64_t)));
  GTRY(g->alloc((void **)&A.cols, entries * sizeof(int32_t)));
  GTRY(g->alloc((void **)&A.vals, entries * sizeof(double)));
  GTRY(g->alloc((void **)&A.diag, n * sizeof(double)));
  GTRY(g->alloc((void **)&A.Axf, n * sizeof(double)));
  if (level > 0) {
    GTRY(g->alloc((void **)&A.r, n * sizeof(double)));
    GTRY(g->alloc((void **)&A.x, n * sizeof(double)));
  }
  std::vector<int32_t> f2k;
  if (coarse) {
    GTRY(g->alloc((void **)&A.f2c, nc * sizeof(int32_t)));
    GTRY(g->alloc((void **)&A.f2k, nc * sizeof(int32_t)));
    std::vector<int32_t> at(n);
    for (int64_t k = 0; k < n; ++k) at[perm[k]] = (int32_t)k;
    f2k.resize(nc);
    for (int64_t i = 0; i < nc; ++i) f2k[i] = at[f2c[i]];
  }
  cudaStream_t s = g->stream;
  GCK(cudaMemcpyAsync(A.slice_off, off.data(), (slices + 1) * sizeof(int64_t),
                      cudaMemcpyHostToDevice, s));
  GCK(cudaMemcpyAsync(A.nnz, hn.data(), n, cudaMemcpyHostToDevice, s));
  GCK(cudaMemcpyAsync(A.dcstart, A.cstart.data(), A.cstart.size() * sizeof(int64_t),
                      cudaMemcpyHostToDevice, s));
  GCK(cudaMemcpyAsync(A.dpos, hd.data(), n, cudaMemcpyHostToDevice, s));
  GCK(cudaMemcpyAsync(A.perm, perm.data(), n * sizeof(int32_t), cudaMemcpyHostToDevice, s));
  GCK(cudaMemcpyAsync(A.cols, hc, entries * sizeof(int32_t), cudaMemcpyHostToDevice, s));
  GCK(cudaMemcpyAsync(A.vals, hv, entries * sizeof(double), cudaMemcpyHostToDevice, s));
  GCK(cudaMemcpyAsync(A.diag, hdiag.data(), n * sizeof(double), cudaMemcpyHostToDevice, s));
  if (coarse) {
    GCK(cudaMemcpyAsync(A.f2c, f2c, nc * sizeof(int32_t), cudaMemcpyHostToDevice, s));
    GCK(cudaMemcpyAsync(A.f2k, f2k.data(), nc * sizeof(int32_t), cudaMemcpyHostToDevice, s));
  }
  if (level == 0) {
    for (double **v : {&g->r, &g->z, &g->p, &g->Ap, &g->x}) GTRY(g->alloc((void **)v, n * sizeof(double)));
    GTRY(g->alloc((void **)&g->st, sizeof(CgState)));
    const int64_t blocks = reduce_blocks(n);
    const int64_t cap = 2 * blocks + 2 * ((blocks + 1023) / 1024);
    GTRY(g->alloc((void **)&g->red.partials, cap * sizeof(double)));
    const int64_t counters = 1 + (cap + 1023) / 1024;
    GTRY(g->alloc((void **)&g->red.counter, counters * sizeof(unsigned int)));
    g->red.capacity = cap;
    GCK(cudaMemsetAsync(g->red.counter, 0, counters * sizeof(unsigned int), s));
  }
  GCK(cudaStreamSynchronize(s));
  A.loaded = true;
  return HPCGX_OK;
}

int general_spmv(GeneralProblem *g, int level, const double *x, double *y) {
  g->spmv(level, x, y, nullptr);
  GCK(cudaStreamSynchronize(g->stream));
  GCK(cudaGetLastError());
  return HPCGX_OK;
}

int general_symgs(GeneralProblem *g, int level, const double *r, double *x) {
  g->symgs(level, r, x, nullptr);
  GCK(cudaStreamSynchronize(g->stream));
  GCK(cudaGetLastError());
  return HPCGX_OK;
}

int general_mg(GeneralProblem *g, const double *r, double *x) {
  g->mg(0, r, x, nullptr);
  GCK(cudaStreamSynchronize(g->stream));
  GCK(cudaGetLastError());
  return HPCGX_OK;
}

int general_cg(GeneralProblem *g, const double *b, double *x, int max_iter, double tol,
               int precond, int *niters, double *normr, double *normr0, double *times) {
  if (max_iter < 0) return set_error(HPCGX_EINVAL, "max_iter < 0");
  const auto t0 = std::chrono::steady_clock::now();
  const int64_t n = g->L[0].n;
  const int kind = precond ? 1 : 0;
  cudaStream_t s = g->stream;
  CgState h;
  std::memset(&h, 0, sizeof(h));
  h.tol = tol;
  h.max_iter = max_iter;
  GCK(g->monitor.init());
  h.mirror = g->monitor.slots;
  GCK(cudaMemcpyAsync(g->st, &h, sizeof(h), cudaMemcpyHostToDevice, s));
  // p = x, Ap = A p, r = b - Ap, normr0 (src/CG.cpp:86-96)
  GCK(cudaMemcpyAsync(g->x, x, n * sizeof(double), cudaMemcpyDeviceToDevice, s));
  GCK(cudaMemcpyAsync(g->p, x, n * sizeof(double), cudaMemcpyDeviceToDevice, s));
  g->spmv(0, g->p, g->Ap, nullptr);
  g->note(launch_cg_init(n, b, g->Ap, g->r, nullptr, g->red, g->st, s));
  // one CUDA graph per iteration, captured on first use
  const bool timed = times != nullptr;
  cudaGraphExec_t &exec = g->graph[kind][timed];
  if (!exec) {
    if (timed)
      for (cudaEvent_t &ev : g->phase[kind])
        if (!ev) GCK(cudaEventCreate(&ev));
    cudaGraph_t gr = nullptr;
    GCK(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    g->timed = timed;
    const int64_t before = g->launches;
    g->iteration(kind, g->x);
    g->timed = false;
    g->launches = before;
    GCK(cudaStreamEndCapture(s, &gr));
    const cudaError_t e = cudaGraphInstantiate(&exec, gr, 0);
    cudaGraphDestroy(gr);
    GCK(e);
  }
  double t_mg = 0, t_vec = 0, t_spmv = 0;
  int launched = 0;
  if (!timed) {
    GCK(g->monitor.run(s, max_iter, &h, [&]() {
      ++launched;
      return cudaGraphLaunch(exec, s);
    }));
  }
  while (timed && launched < max_iter) {
    GCK(cudaGraphLaunch(exec, s));
    ++launched;
    GCK(cudaMemcpyAsync(&h, g->st, sizeof(h), cudaMemcpyDeviceToHost, s));
    GCK(cudaStreamSynchronize(s));
    if (h.niters == launched) {
      float a = 0, b2 = 0, c = 0, d = 0;
      GCK(cudaEventElapsedTime(&a, g->phase[kind][0], g->phase[kind][1]));
      GCK(cudaEventElapsedTime(&b2, g->phase[kind][1], g->phase[kind][2]));
      GCK(cudaEventElapsedTime(&c, g->phase[kind][2], g->phase[kind][3]));
      GCK(cudaEventElapsedTime(&d, g->phase[kind][3], g->phase[kind][4]));
      t_mg += a * 1e-3;
      t_vec += (b2 + d) * 1e-3;
      t_spmv += c * 1e-3;
    }
    if (h.done) break;
  }
  if (launched == 0)
    GCK(cudaMemcpyAsync(&h, g->st, sizeof(h), cudaMemcpyDeviceToHost, s));
  GCK(cudaMemcpyAsync(x, g->x, n * sizeof(double), cudaMemcpyDeviceToDevice, s));
  GCK(cudaStreamSynchronize(s));
  if (niters) *niters = h.niters;
  if (normr) *normr = h.normr;
  if (normr0) *normr0 = h.normr0;
  if (times) {
    times[0] += std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    times[2] += t_vec;
    times[3] += t_spmv;
    times[5] += t_mg;
  }
  if (h.nonfinite) return set_error(HPCGX_ENONFINITE, "CG: residual norm is not finite");
  return HPCGX_OK;
}

// The level's Axf work vector stages the natural-order diagonal.
int general_set_diagonal(GeneralProblem *g, int level, const double *diag) {
  GLevel &A = g->L[level];
  GCK(cudaMemcpyAsync(A.Axf, diag, A.n * sizeof(double), cudaMemcpyHostToDevice, g->stream));
  k_gen_diag<<<grid(A.n), kT, 0, g->stream>>>(A.n, A.slice_off, A.perm, A.dpos, A.vals, A.diag,
                                              A.Axf, 1);
  GCK(cudaGetLastError());
  GCK(cudaStreamSynchronize(g->stream));
  return HPCGX_OK;
}

int general_get_diagonal(GeneralProblem *g, int level, double *diag) {
  GLevel &A = g->L[level];
  k_gen_diag<<<grid(A.n), kT, 0, g->stream>>>(A.n, A.slice_off, A.perm, A.dpos, A.vals, A.diag,
                                              A.Axf, 0);
  GCK(cudaGetLastError());
  GCK(cudaMemcpyAsync(diag, A.Axf, A.n * sizeof(double), cudaMemcpyDeviceToHost, g->stream));
  GCK(cudaStreamSynchronize(g->stream));
  return HPCGX_OK;
}

}  // namespace hpcgx
