// Level-scheduled sparse sweeps of the reference's lusolver on the GPU.
//
//   scalar  SparseSolverNUM (lusolver/SparseSolverNUM.cpp): setELE/addELE
//           :115-140, solveILUSGS :144-212, solveGS :214-252
//   block   SparseSolver<Matrix4d, Vector4d> (lusolver/SparseSolver.cpp):
//           setD/setL/setU :35-48, solveILU :53-104
//
// The reference walks column lists (insertion order, duplicates kept):
// columns ascending for the products and the forward sweep, descending for
// the backward sweep.  Row-oriented, the same contributions reach each row
// in the same order when a row's entries are sorted by (column ascending,
// insertion order) -- or (column descending, insertion order) for the
// backward sweep.  Rows whose dependencies are all in earlier levels are
// independent, so each level is one parallel launch -- or, for scalar
// systems, a phase of one launch -- and every row adds
// its terms sequentially in that order: the results are bit-identical to the
// reference's (compiled with --fmad=false; 4x4 blocks use the adjugate
// inverse and left-to-right products of the oracle's Eigen shim).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "cluster_vec.cuh"
#include "ctx.hpp"
#include "smem_limit.hpp"

namespace cg = cooperative_groups;

namespace {

constexpr int kLuInterval = 5;  // LU_INTERVAL (include/CONST.h:57)

// ---- 4x4 block arithmetic, row-major, the shim's order ------------------
__device__ __forceinline__ double det3(double a, double b, double c, double d, double e,
                                       double f, double g, double h, double i) {
  return a * (e * i - f * h) - b * (d * i - f * g) + c * (d * h - e * g);
}
__device__ void inv4(const double* m, double* inv) {
  double cof[16];
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < 4; ++j) {
      const int r0 = (i == 0) ? 1 : 0, r1 = (i <= 1) ? 2 : 1, r2 = (i <= 2) ? 3 : 2;
      const int c0 = (j == 0) ? 1 : 0, c1 = (j <= 1) ? 2 : 1, c2 = (j <= 2) ? 3 : 2;
      const double v = det3(m[4 * r0 + c0], m[4 * r0 + c1], m[4 * r0 + c2], m[4 * r1 + c0],
                            m[4 * r1 + c1], m[4 * r1 + c2], m[4 * r2 + c0], m[4 * r2 + c1],
                            m[4 * r2 + c2]);
      cof[4 * i + j] = ((i + j) & 1) ? -v : v;
    }
  double det = m[0] * cof[0];
  det += m[1] * cof[1];
  det += m[2] * cof[2];
  det += m[3] * cof[3];
  const double id = 1.0 / det;
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < 4; ++j) inv[4 * i + j] = cof[4 * j + i] * id;
}
__device__ __forceinline__ void mv4(const double* a, const double* x, double* y) {
  for (int i = 0; i < 4; ++i) {
    double s = a[4 * i] * x[0];
    s += a[4 * i + 1] * x[1];
    s += a[4 * i + 2] * x[2];
    s += a[4 * i + 3] * x[3];
    y[i] = s;
  }
}
__device__ __forceinline__ void mm4(const double* a, const double* b, double* c) {
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < 4; ++j) {
      double s = a[4 * i] * b[j];
      s += a[4 * i + 1] * b[4 + j];
      s += a[4 * i + 2] * b[8 + j];
      s += a[4 * i + 3] * b[12 + j];
      c[4 * i + j] = s;
    }
}

// ---- kernels: B = 1 (scalar) or 4 (blocks) ---------------------------------
// Phase A: RHSUx[r] = sum_U U * X (then D^-1) ; GS: RHS = b - sum_U U * X
template <int B>
__global__ void k_upper_product(int dim, const int* __restrict__ ptr, const int* __restrict__ col,
                                const double* __restrict__ val, const double* __restrict__ x,
                                const double* __restrict__ D, const double* __restrict__ Di,
                                const double* __restrict__ b, double* __restrict__ out, int gs) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= dim) return;
  if (B == 1) {
    double s = 0.;
    for (int k = ptr[r]; k < ptr[r + 1]; ++k) s += val[k] * x[col[k]];
    out[r] = gs ? b[r] - s : s / D[r];
  } else {
    double s[4] = {0., 0., 0., 0.}, t[4];
    for (int k = ptr[r]; k < ptr[r + 1]; ++k) {
      mv4(val + 16 * (size_t)k, x + 4 * (size_t)col[k], t);
      for (int j = 0; j < 4; ++j) s[j] += t[j];
    }
    mv4(Di + 16 * (size_t)r, s, t);
    for (int j = 0; j < 4; ++j) out[4 * (size_t)r + j] = t[j];
  }
}

// Phase B: RHS[r] = b[r] + sum_L L * RHSUx
template <int B>
__global__ void k_lower_product(int dim, const int* __restrict__ ptr, const int* __restrict__ col,
                                const double* __restrict__ val, const double* __restrict__ y,
                                const double* __restrict__ b, double* __restrict__ rhs) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= dim) return;
  double s[B], t[4];
  for (int j = 0; j < B; ++j) s[j] = 0.;
  for (int k = ptr[r]; k < ptr[r + 1]; ++k) {
    if (B == 1) {
      s[0] += val[k] * y[col[k]];
    } else {
      mv4(val + 16 * (size_t)k, y + 4 * (size_t)col[k], t);
      for (int j = 0; j < B; ++j) s[j] += t[j];
    }
  }
  for (int j = 0; j < B; ++j) rhs[B * (size_t)r + j] = b[B * (size_t)r + j] + s[j];
}

// One level of a sweep: v[r] -= (M * D^-1[k]) * v[k] over the row's entries
// in order (forward: L, columns ascending; backward: U, columns descending)
template <int B>
__global__ void k_sweep_level(int n, const int* __restrict__ rows, const int* __restrict__ ptr,
                              const int* __restrict__ col, const double* __restrict__ val,
                              const double* __restrict__ D, const double* __restrict__ Di,
                              double* __restrict__ v) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int r = rows[i];
  if (B == 1) {
    double acc = v[r];
    for (int k = ptr[r]; k < ptr[r + 1]; ++k) {
      const int c = col[k];
      acc -= (val[k]) * (1. / D[c]) * v[c];
    }
    v[r] = acc;
  } else {
    double acc[4], M[16], t[4];
    for (int j = 0; j < 4; ++j) acc[j] = v[4 * (size_t)r + j];
    for (int k = ptr[r]; k < ptr[r + 1]; ++k) {
      const int c = col[k];
      mm4(val + 16 * (size_t)k, Di + 16 * (size_t)c, M);
      mv4(M, v + 4 * (size_t)c, t);
      for (int j = 0; j < 4; ++j) acc[j] -= t[j];
    }
    for (int j = 0; j < 4; ++j) v[4 * (size_t)r + j] = acc[j];
  }
}

// X1 = D^-1 RHS ; RHS1 = D X1
template <int B>
__global__ void k_middle(int dim, const double* __restrict__ D, const double* __restrict__ Di,
                         const double* __restrict__ rhs, double* __restrict__ rhs1) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= dim) return;
  if (B == 1) {
    const double x1 = (1. / D[r]) * rhs[r];
    rhs1[r] = D[r] * x1;
  } else {
    double x1[4], t[4];
    mv4(Di + 16 * (size_t)r, rhs + 4 * (size_t)r, x1);
    mv4(D + 16 * (size_t)r, x1, t);
    for (int j = 0; j < 4; ++j) rhs1[4 * (size_t)r + j] = t[j];
  }
}

// X = D^-1 v and, for the scalar solver, the largest |X - X'| / X (signed
// division and NaN behaviour of SparseSolverNUM.cpp:194-203) per block
template <int B>
__global__ void k_final(int dim, const double* __restrict__ D, const double* __restrict__ Di,
                        const double* __restrict__ v, double* __restrict__ x,
                        double* __restrict__ part) {
  __shared__ double red[8];
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  double res = 0.;
  if (r < dim) {
    if (B == 1) {
      const double xn = (1. / D[r]) * v[r];
      const double q = fabs(x[r] - xn) / x[r];
      res = (res < q) ? q : res;
      x[r] = xn;
    } else {
      double t[4];
      mv4(Di + 16 * (size_t)r, v + 4 * (size_t)r, t);
      for (int j = 0; j < 4; ++j) x[4 * (size_t)r + j] = t[j];
    }
  }
  if (B == 1) {
    for (int o = 16; o > 0; o >>= 1) {
      const double w = __shfl_xor_sync(0xffffffffu, res, o);
      res = (res < w) ? w : res;
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = res;
    __syncthreads();
    if (threadIdx.x == 0) {
      double m = red[0];
      for (int i = 1; i < (int)(blockDim.x >> 5); ++i) m = (m < red[i]) ? red[i] : m;
      part[blockIdx.x] = m;
    }
  }
}

template <int B>
__global__ void k_invert_blocks(int dim, const double* __restrict__ D, double* __restrict__ Di) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < dim) inv4(D + 16 * (size_t)r, Di + 16 * (size_t)r);
}

// ---- scalar systems: the whole solve in one launch ----------------------------
// The levels of a sweep are small (800 rows of an 18k-row mesh system) and
// depend on each other, so a launch per level pays launch and memory latency
// 230 times a solve.  Here one thread-block cluster runs all iterations and the
// exit test.  The swept vector lies in the CTAs' shared memory, 32 rows in turn
// to each CTA; a row's dependent values are read from the owner (distributed
// shared memory: two thirds of the latency of the same vector in L2), and a
// level ends with the hardware cluster barrier.  A row's columns and weights
// are fetched a level ahead, 32 rows a warp.  The FP64 pipe takes 64 cycles a
// warp instruction on each SM sub-partition, so the cluster is the largest the
// device places.  ILUSGS, 5 iterations, call included: 200 / 18,240 / 228,488
// rows 195 / 449 / 1,919 us (a launch per level 869 / 1,580 / 2,228; clusters of
// 1 / 4 / 8 at 18,240 rows 1,549 / 722 / 534).
constexpr int kLuThreads = 512;
constexpr int kLuMaxCta = 16;

// Rows of a sweep in level order, or of a product in row order.  The first four
// entries stand at fixed places, so that all of a row's loads can be issued at
// once; rows with more find the rest in the matrix itself, from meta.z.  A
// sweep's weight is L (1 / D[column]): the quotient and product the reference
// forms at every use.
struct LuRows {
  const int* lev;
  const int4* meta;  // row, entries, the fifth's place in col / val, -
  const int4* col4;
  const double4_32a* w4;
  const int* col;
  const double *val, *rD;  // rD = 1 / D, or null: a product
  int n_levels;
};
// lays them out (rows: the order, or null)
__global__ void k_lu_rows(int dim, const int* __restrict__ rows, const int* __restrict__ ptr,
                          const int* __restrict__ col, const double* __restrict__ val,
                          const double* __restrict__ rD, int4* __restrict__ meta,
                          int4* __restrict__ col4, double4_32a* __restrict__ w4) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= dim) return;
  const int r = rows ? rows[i] : i, k0 = ptr[r], n = ptr[r + 1] - k0;
  int c[4];
  double w[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    c[k] = k < n ? col[k0 + k] : 0;
    w[k] = k < n ? (rD ? val[k0 + k] * rD[c[k]] : val[k0 + k]) : 0.;
  }
  meta[i] = make_int4(r, n, k0 + 4, 0);
  col4[i] = make_int4(c[0], c[1], c[2], c[3]);
  w4[i] = double4_32a{w[0], w[1], w[2], w[3]};
}
__global__ void k_lu_reciprocal(int dim, const double* __restrict__ D, double* __restrict__ rD) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < dim) rD[r] = 1. / D[r];
}

struct LuSolve {
  int dim, gs, shift, rows;  // 2^shift CTAs, rows of the vector in each
  LuRows up, lo, fwd, bwd;
  const double *D, *rD, *b;  // rD = 1 / D
  double* x;
  unsigned* part;  // [kLuMaxCta]
  int* its;
};

struct LuVec : mst::ClusterVec<1> {
  __device__ __forceinline__ double operator[](int r) const { return *(volatile double*)at(r); }
};

struct LuRow {
  int4 meta, c;
  double4_32a w;
};
__device__ __forceinline__ void lu_fetch(LuRow& r, const LuRows& s, int i, int end) {
  r.meta.x = -1;
  if (i >= end) return;
  r.meta = s.meta[i];
  r.c = s.col4[i];
  r.w = s.w4[i];
}
// acc - sum w v (or + : the products), entries in order; lu_values: the first
// four entries' v
template <class V>
__device__ __forceinline__ double4_32a lu_values(const LuRow& r, const V& v) {
  const int n = r.meta.y;
  return double4_32a{n > 0 ? v[r.c.x] : 0., n > 1 ? v[r.c.y] : 0., n > 2 ? v[r.c.z] : 0.,
                     n > 3 ? v[r.c.w] : 0.};
}
template <bool SUB, class V>
__device__ __forceinline__ double lu_row(const LuRow& r, const double4_32a& x, const LuRows& s,
                                         const V& v, double acc) {
  const int n = r.meta.y;
  auto add = [&](double p) { acc = SUB ? acc - p : acc + p; };
  if (n > 0) add(r.w.x * x.x);
  if (n > 1) add(r.w.y * x.y);
  if (n > 2) add(r.w.z * x.z);
  if (n > 3) add(r.w.w * x.w);
  for (int k = r.meta.z; k < r.meta.z + n - 4; ++k) {
    const int c = s.col[k];
    add((s.rD ? s.val[k] * s.rD[c] : s.val[k]) * v[c]);
  }
  return acc;
}

struct LuGlobal {  // written by other CTAs of the cluster: read from L2
  const double* p;
  __device__ __forceinline__ double operator[](int r) const { return __ldcg(p + r); }
};

__device__ void lu_sweep(const LuRows& s, const LuVec& v, int first, int stride) {
  cg::cluster_group cl = cg::this_cluster();
  const int n = s.n_levels;
  if (n < 2) return;
  // rows [b, e) of this level, [e, e1) of the next, [e1, e2) after it; the
  // rows of level 0 have no entries
  int b = s.lev[1], e = s.lev[2], e1 = s.lev[min(3, n)], e2 = s.lev[min(4, n)];
  LuRow cur, nxt;
  lu_fetch(cur, s, b + first, e);
  for (int l = 1; l < n; ++l) {
    int e3 = 0;
    for (int i = b + first;;) {
      // the earlier rows' values first, the next level's row behind them
      double4_32a x{};
      double own = 0.;
      if (cur.meta.x >= 0) {
        x = lu_values(cur, v);
        own = v[cur.meta.x];
      }
      if (i == b + first) {
        lu_fetch(nxt, s, e + first, e1);
        e3 = s.lev[min(l + 4, n)];
      }
      if (cur.meta.x >= 0) *v.at(cur.meta.x) = lu_row<true>(cur, x, s, v, own);
      i += stride;
      if (i >= e) break;
      lu_fetch(cur, s, i, e);
    }
    cl.sync();
    cur = nxt;
    b = e;
    e = e1;
    e1 = e2;
    e2 = e3;
  }
}

__global__ void __launch_bounds__(kLuThreads, 1) k_lu_solve(const LuSolve S) {
  extern __shared__ double sm[];
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), n_cta = (int)cl.num_blocks();
  const LuVec y{{sm, S.shift}}, v{{sm + S.rows, S.shift}};
  // this thread's rows r0, r0 + stride, .. of the vectors (in its own CTA's shared
  // memory, at threadIdx.x, + kLuThreads, ..) and of a level: the warps' groups
  // of 32 go to the CTAs in turn
  const int stride = kLuThreads * n_cta;
  const int r0 = ((int)(threadIdx.x / 32) * n_cta + rank) * 32 + (int)(threadIdx.x % 32);
  cl.sync();  // every CTA runs before its shared memory is used
  int it = 0;
  for (it = 0; it < kLuInterval; ++it) {
    LuRow cur, nxt;
    // ILUSGS: y = D^-1 sum_U U X; GS: v = b - sum_U U X
    const LuGlobal x{S.x};
    lu_fetch(cur, S.up, r0, S.dim);
    for (int r = r0, j = threadIdx.x; r < S.dim; r += stride, j += kLuThreads) {
      lu_fetch(nxt, S.up, r + stride, S.dim);
      const double s = lu_row<false>(cur, lu_values(cur, x), S.up, x, 0.);
      if (S.gs) v.base[j] = S.b[r] - s;
      else y.base[j] = s / S.D[r];
      cur = nxt;
    }
    if (!S.gs) {
      // v = b + sum_L L y
      lu_fetch(cur, S.lo, r0, S.dim);
      cl.sync();
      for (int r = r0, j = threadIdx.x; r < S.dim; r += stride, j += kLuThreads) {
        lu_fetch(nxt, S.lo, r + stride, S.dim);
        v.base[j] = S.b[r] + lu_row<false>(cur, lu_values(cur, y), S.lo, y, 0.);
        cur = nxt;
      }
    }
    cl.sync();
    lu_sweep(S.fwd, v, r0, stride);
    if (!S.gs) {
      for (int r = r0, j = threadIdx.x; r < S.dim; r += stride, j += kLuThreads) {
        const double x1 = S.rD[r] * v.base[j];
        v.base[j] = S.D[r] * x1;
      }
      cl.sync();
      lu_sweep(S.bwd, v, r0, stride);
    }
    // X = D^-1 v
    unsigned ch = 0;
    for (int r = r0, j = threadIdx.x; r < S.dim; r += stride, j += kLuThreads) {
      const double xn = S.rD[r] * v.base[j];
      ch |= mst::gs_change(__ldcg(S.x + r), xn);
      S.x[r] = xn;
    }
    const unsigned big = __syncthreads_or(ch & 1u), any = __syncthreads_or(ch & 2u);
    if (threadIdx.x == 0) S.part[rank] = (big ? 1u : 0u) | (any ? 2u : 0u);
    cl.sync();
    ch = 0;
    for (int q = 0; q < n_cta; ++q) ch |= __ldcg(S.part + q);
    // the reference's exit test (:205, :245); the same value in every thread
    if (ch == 2u) {
      ++it;
      break;
    }
  }
  if (rank == 0 && threadIdx.x == 0) *S.its = it;
  // (every access to another CTA's shared memory is followed by a cluster
  // barrier above, so no CTA leaves too early)
}

// ---- host-side structure -----------------------------------------------------
struct Csr {
  std::vector<int> ptr, col;
  std::vector<double> val;
};

}  // namespace

struct mst_lu {
  int block = 1, dim = 0;
  int n_fwd_levels = 0, n_bwd_levels = 0;
  std::vector<int> fwd_ptr, bwd_ptr;  // level ranges into the row lists (host)
  // device
  cudaStream_t stream = nullptr;
  double *D = nullptr, *Di = nullptr;
  int *l_ptr = nullptr, *l_col = nullptr, *ua_ptr = nullptr, *ua_col = nullptr,
      *ud_ptr = nullptr, *ud_col = nullptr, *fwd_rows = nullptr, *bwd_rows = nullptr;
  double *l_val = nullptr, *ua_val = nullptr, *ud_val = nullptr;
  double *b = nullptr, *x = nullptr, *t1 = nullptr, *rhs = nullptr, *rhs1 = nullptr,
         *part = nullptr;
  std::vector<void*> allocs;
  // the one-launch solve of scalar systems (cluster = 0: not used)
  int cluster = 0;
  int *fwd_lev = nullptr, *bwd_lev = nullptr;
  LuRows r_up{}, r_lo{}, r_fwd{}, r_bwd{};
  double* rD = nullptr;
  unsigned* change = nullptr;
  int* its = nullptr;
};

namespace {

mst_status lu_fail(mst_status s, const std::string& m) { return mst_internal_fail(s, m); }

#define LU_CU(call)                                                                  \
  do {                                                                               \
    cudaError_t e_ = (call);                                                         \
    if (e_ != cudaSuccess)                                                           \
      return lu_fail(MST_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

// rows' entries below (lower) or above the diagonal, sorted by column
// (ascending or descending) and then insertion order
Csr build_rows(int dim, int n, const int* rows, const int* cols, const double* vals, int B,
               bool lower, bool desc) {
  Csr c;
  c.ptr.assign(dim + 1, 0);
  auto mine = [&](int i) { return lower ? rows[i] > cols[i] : rows[i] < cols[i]; };
  for (int i = 0; i < n; ++i)
    if (mine(i)) c.ptr[rows[i] + 1]++;
  for (int r = 0; r < dim; ++r) c.ptr[r + 1] += c.ptr[r];
  // entries into their rows in insertion order, then a stable sort within the row
  std::vector<int> idx(c.ptr[dim]), fill(c.ptr.begin(), c.ptr.end() - 1);
  for (int i = 0; i < n; ++i)
    if (mine(i)) idx[fill[rows[i]]++] = i;
  auto before = [&](int x, int y) { return desc ? cols[x] > cols[y] : cols[x] < cols[y]; };
  for (int r = 0; r < dim; ++r) {
    const int a = c.ptr[r], e = c.ptr[r + 1];
    if (e - a > 16) {
      std::stable_sort(idx.begin() + a, idx.begin() + e, before);
      continue;
    }
    for (int k = a + 1; k < e; ++k)
      for (int q = k; q > a && before(idx[q], idx[q - 1]); --q) std::swap(idx[q - 1], idx[q]);
  }
  c.col.reserve(idx.size());
  c.val.reserve(idx.size() * B * B);
  for (int i : idx) {
    c.col.push_back(cols[i]);
    for (int k = 0; k < B * B; ++k) c.val.push_back(vals[(size_t)B * B * i + k]);
  }
  return c;
}

// rows grouped by level; level(r) = 1 + max level of the rows it reads
void levels(const Csr& c, int dim, bool forward, std::vector<int>* rows_by_level,
            std::vector<int>* ptr, int* n_levels) {
  std::vector<int> lev(dim, 0);
  int maxl = -1;
  for (int t = 0; t < dim; ++t) {
    const int r = forward ? t : dim - 1 - t;
    int l = 0;
    for (int k = c.ptr[r]; k < c.ptr[r + 1]; ++k) l = std::max(l, lev[c.col[k]] + 1);
    lev[r] = l;
    maxl = std::max(maxl, l);
  }
  *n_levels = maxl + 1;
  ptr->assign(maxl + 2, 0);
  for (int r = 0; r < dim; ++r) (*ptr)[lev[r] + 1]++;
  for (int l = 0; l <= maxl; ++l) (*ptr)[l + 1] += (*ptr)[l];
  rows_by_level->assign(dim, 0);
  std::vector<int> fill(ptr->begin(), ptr->end() - 1);
  for (int r = 0; r < dim; ++r) (*rows_by_level)[fill[lev[r]]++] = r;
}

template <class T>
cudaError_t up(mst_lu* s, T** dst, const std::vector<T>& v) {
  const size_t bytes = std::max<size_t>(v.size(), 1) * sizeof(T);
  cudaError_t e = cudaMalloc((void**)dst, bytes);
  if (e != cudaSuccess) return e;
  s->allocs.push_back(*dst);
  // (returns once v has been read; mst_lu_create waits for the arrival)
  if (!v.empty()) e = cudaMemcpy(*dst, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
  return e;
}

// the tables of the one-launch solve, in one allocation
cudaError_t lu_tables(mst_lu* s) {
  const int dim = s->dim, nb = (dim + 127) / 128;
  size_t at = 0;
  auto place = [&](size_t bytes) {
    const size_t p = at;
    at += (bytes + 255) / 256 * 256;
    return p;
  };
  struct Rows {
    LuRows* out;
    const int *rows, *ptr, *col;
    const double* val;
    bool sweep;
    const int* lev;
    int n_levels;
    size_t meta, col4, w4;
  } t[4] = {{&s->r_up, nullptr, s->ua_ptr, s->ua_col, s->ua_val, false, nullptr, 1},
            {&s->r_lo, nullptr, s->l_ptr, s->l_col, s->l_val, false, nullptr, 1},
            {&s->r_fwd, s->fwd_rows, s->l_ptr, s->l_col, s->l_val, true, s->fwd_lev,
             s->n_fwd_levels},
            {&s->r_bwd, s->bwd_rows, s->ud_ptr, s->ud_col, s->ud_val, true, s->bwd_lev,
             s->n_bwd_levels}};
  for (Rows& q : t) {
    q.meta = place(sizeof(int4) * (size_t)dim);
    q.col4 = place(sizeof(int4) * (size_t)dim);
    q.w4 = place(sizeof(double4_32a) * (size_t)dim);
  }
  const size_t rD = place(sizeof(double) * (size_t)dim),
               change = place(sizeof(unsigned) * kLuMaxCta), its = place(sizeof(int));
  char* d = nullptr;
  cudaError_t e = cudaMalloc((void**)&d, at);
  if (e != cudaSuccess) return e;
  s->allocs.push_back(d);
  s->rD = (double*)(d + rD);
  s->change = (unsigned*)(d + change);
  s->its = (int*)(d + its);
  k_lu_reciprocal<<<nb, 128, 0, s->stream>>>(dim, s->D, s->rD);
  for (Rows& q : t) {
    *q.out = LuRows{q.lev, (int4*)(d + q.meta), (int4*)(d + q.col4), (double4_32a*)(d + q.w4),
                    q.col, q.val, q.sweep ? s->rD : nullptr, q.n_levels};
    k_lu_rows<<<nb, 128, 0, s->stream>>>(dim, q.rows, q.ptr, q.col, q.val, q.out->rD,
                                         (int4*)(d + q.meta), (int4*)(d + q.col4),
                                         (double4_32a*)(d + q.w4));
  }
  return cudaGetLastError();
}

int lu_cta_rows(int cluster, int dim) {
  const int span = cluster * kLuThreads;
  return (dim + span - 1) / span * kLuThreads;
}

void lu_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at, int cluster, int dim,
               cudaStream_t stream) {
  *cfg = cudaLaunchConfig_t{};
  cfg->gridDim = dim3(cluster);
  cfg->blockDim = dim3(kLuThreads);
  cfg->dynamicSmemBytes = 2 * sizeof(double) * (size_t)lu_cta_rows(cluster, dim);
  cfg->stream = stream;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = cluster;
  at->val.clusterDim.y = 1;
  at->val.clusterDim.z = 1;
  cfg->attrs = at;
  cfg->numAttrs = 1;
}

// The cluster of the one-launch solve: the largest the device places.  0, a
// launch per level on the whole device, where the vectors do not fit the
// cluster's shared memory (229,376 rows on 16 CTAs: still the faster there)
int lu_pick_cluster(int dim) {
  constexpr size_t kMaxSmem = 224 * 1024;
  static std::atomic<uint64_t> attr_done{0};
  if (mst::ensure_smem_limit(k_lu_solve, (int)kMaxSmem, attr_done) != cudaSuccess ||
      cudaFuncSetAttribute(k_lu_solve, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
          cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  for (int nb = kLuMaxCta; nb >= 1; nb /= 2) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at;
    lu_config(&cfg, &at, nb, dim, nullptr);
    if (cfg.dynamicSmemBytes > kMaxSmem) break;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_lu_solve, &cfg) == cudaSuccess && n > 0) return nb;
    cudaGetLastError();
  }
  return 0;
}

mst_status lu_solve_cluster(mst_lu* s, int gs, int* iterations) {
  LuSolve a{};
  a.dim = s->dim;
  a.gs = gs;
  while ((1 << a.shift) < s->cluster) ++a.shift;
  a.rows = lu_cta_rows(s->cluster, s->dim);
  a.up = s->r_up;
  a.lo = s->r_lo;
  a.fwd = s->r_fwd;
  a.bwd = s->r_bwd;
  a.D = s->D;
  a.rD = s->rD;
  a.b = s->b;
  a.x = s->x;
  a.part = s->change;
  a.its = s->its;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at;
  lu_config(&cfg, &at, s->cluster, s->dim, s->stream);
  LU_CU(cudaLaunchKernelEx(&cfg, k_lu_solve, a));
  int it = 0;
  LU_CU(cudaMemcpyAsync(&it, s->its, sizeof it, cudaMemcpyDeviceToHost, s->stream));
  LU_CU(cudaStreamSynchronize(s->stream));
  if (iterations) *iterations = it;
  return MST_OK;
}

template <int B>
mst_status lu_iterate(mst_lu* s, int gs, int* iterations) {
  const int dim = s->dim, nb = (dim + 127) / 128;
  int it = 0;
  std::vector<double> part(nb);
  for (it = 0; it < kLuInterval; ++it) {
    if (!gs) {
      k_upper_product<B><<<nb, 128, 0, s->stream>>>(dim, s->ua_ptr, s->ua_col, s->ua_val, s->x,
                                                    s->D, s->Di, s->b, s->t1, 0);
      k_lower_product<B><<<nb, 128, 0, s->stream>>>(dim, s->l_ptr, s->l_col, s->l_val, s->t1,
                                                    s->b, s->rhs);
    } else {
      k_upper_product<B><<<nb, 128, 0, s->stream>>>(dim, s->ua_ptr, s->ua_col, s->ua_val, s->x,
                                                    s->D, s->Di, s->b, s->rhs, 1);
    }
    for (int l = 0; l < s->n_fwd_levels; ++l) {
      const int a = s->fwd_ptr[l], n = s->fwd_ptr[l + 1] - a;
      k_sweep_level<B><<<(n + 127) / 128, 128, 0, s->stream>>>(
          n, s->fwd_rows + a, s->l_ptr, s->l_col, s->l_val, s->D, s->Di, s->rhs);
    }
    const double* last = s->rhs;
    if (!gs) {
      k_middle<B><<<nb, 128, 0, s->stream>>>(dim, s->D, s->Di, s->rhs, s->rhs1);
      for (int l = 0; l < s->n_bwd_levels; ++l) {
        const int a = s->bwd_ptr[l], n = s->bwd_ptr[l + 1] - a;
        k_sweep_level<B><<<(n + 127) / 128, 128, 0, s->stream>>>(
            n, s->bwd_rows + a, s->ud_ptr, s->ud_col, s->ud_val, s->D, s->Di, s->rhs1);
      }
      last = s->rhs1;
    }
    k_final<B><<<nb, 128, 0, s->stream>>>(dim, s->D, s->Di, last, s->x, s->part);
    LU_CU(cudaGetLastError());
    if (B == 1) {
      // the reference's exit test (SparseSolverNUM.cpp:205, :245)
      LU_CU(cudaMemcpyAsync(part.data(), s->part, nb * sizeof(double), cudaMemcpyDeviceToHost,
                            s->stream));
      LU_CU(cudaStreamSynchronize(s->stream));
      double res = 0.;
      for (double p : part) res = (res < p) ? p : res;
      if (res > 1e-10 * 1e-10 && res < 1e-7) {
        ++it;
        break;
      }
    }
  }
  LU_CU(cudaStreamSynchronize(s->stream));
  if (iterations) *iterations = it;
  return MST_OK;
}

}  // namespace

extern "C" {

mst_status mst_lu_create(int block, int dim, int n, const int* rows, const int* cols,
                         const int* ops, const double* vals, mst_lu** out) {
  if (!out || dim <= 0 || n < 0 || (n > 0 && (!rows || !cols || !vals)))
    return lu_fail(MST_EINVAL, "bad arguments");
  if (block != 1 && block != 4) return lu_fail(MST_EINVAL, "block must be 1 or 4");
  *out = nullptr;
  for (int i = 0; i < n; ++i)
    if (rows[i] < 0 || rows[i] >= dim || cols[i] < 0 || cols[i] >= dim)
      return lu_fail(MST_EINVAL, "entry outside the matrix");
  auto s = new (std::nothrow) mst_lu;
  if (!s) return lu_fail(MST_ENOMEM, "host allocation failed");
  s->block = block;
  s->dim = dim;
  const int BB = block * block;
  // diagonal: setELE sets, addELE adds (scalar); setD sets (blocks)
  std::vector<double> D((size_t)dim * BB, 0.0);
  for (int i = 0; i < n; ++i)
    if (rows[i] == cols[i]) {
      double* d = D.data() + (size_t)BB * rows[i];
      const double* v = vals + (size_t)BB * i;
      if (block == 1 && ops && ops[i] == 1) d[0] += v[0];
      else std::memcpy(d, v, BB * sizeof(double));
    }
  Csr L = build_rows(dim, n, rows, cols, vals, block, true, false);
  Csr Ua = build_rows(dim, n, rows, cols, vals, block, false, false);
  Csr Ud = build_rows(dim, n, rows, cols, vals, block, false, true);
  std::vector<int> fr, br;
  levels(L, dim, true, &fr, &s->fwd_ptr, &s->n_fwd_levels);
  levels(Ud, dim, false, &br, &s->bwd_ptr, &s->n_bwd_levels);
  cudaError_t e = cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = up(s, &s->D, D);
  const std::vector<double> zero((size_t)dim * block, 0.0);
  for (double** p : {&s->b, &s->x})
    if (e == cudaSuccess) e = up(s, p, zero);
  if (e == cudaSuccess) e = up(s, &s->l_ptr, L.ptr);
  if (e == cudaSuccess) e = up(s, &s->l_col, L.col);
  if (e == cudaSuccess) e = up(s, &s->l_val, L.val);
  if (e == cudaSuccess) e = up(s, &s->ua_ptr, Ua.ptr);
  if (e == cudaSuccess) e = up(s, &s->ua_col, Ua.col);
  if (e == cudaSuccess) e = up(s, &s->ua_val, Ua.val);
  if (e == cudaSuccess) e = up(s, &s->ud_ptr, Ud.ptr);
  if (e == cudaSuccess) e = up(s, &s->ud_col, Ud.col);
  if (e == cudaSuccess) e = up(s, &s->ud_val, Ud.val);
  if (e == cudaSuccess) e = up(s, &s->fwd_rows, fr);
  if (e == cudaSuccess) e = up(s, &s->bwd_rows, br);
  if (block == 1) s->cluster = lu_pick_cluster(dim);
  if (e == cudaSuccess && s->cluster > 0) {
    e = up(s, &s->fwd_lev, s->fwd_ptr);
    if (e == cudaSuccess) e = up(s, &s->bwd_lev, s->bwd_ptr);
  } else {
    for (double** p : {&s->t1, &s->rhs, &s->rhs1})
      if (e == cudaSuccess) e = up(s, p, zero);
    if (e == cudaSuccess) e = up(s, &s->part, std::vector<double>((dim + 127) / 128 + 1, 0.0));
  }
  if (e == cudaSuccess && block == 4)
    e = up(s, &s->Di, std::vector<double>((size_t)dim * 16, 0.0));
  if (e == cudaSuccess) e = mst::uploads_done();
  if (e == cudaSuccess && s->cluster > 0) e = lu_tables(s);
  if (e == cudaSuccess && block == 4) {
    // D^-1 once: the reference re-inverts D[i] at every use, always to the
    // same result
    k_invert_blocks<4><<<(dim + 127) / 128, 128, 0, s->stream>>>(dim, s->D, s->Di);
    e = cudaGetLastError();
  }
  // the set-up's failure is this call's
  if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
  if (e != cudaSuccess) {
    mst_lu_destroy(s);
    return lu_fail(MST_ECUDA, std::string("mst_lu_create: ") + cudaGetErrorString(e));
  }
  *out = s;
  return MST_OK;
}

mst_status mst_lu_solve(mst_lu* s, int method, const double* b, double* x, int* iterations) {
  if (!s || !b || !x) return lu_fail(MST_EINVAL, "NULL argument");
  if (method != MST_LU_ILUSGS && method != MST_LU_GS)
    return lu_fail(MST_EINVAL, "unknown method");
  if (s->block == 4 && method == MST_LU_GS)
    return lu_fail(MST_EUNSUPPORTED, "the block solver's GS is empty in the reference");
  const size_t bytes = (size_t)s->dim * s->block * sizeof(double);
  LU_CU(cudaMemcpyAsync(s->b, b, bytes, cudaMemcpyHostToDevice, s->stream));
  LU_CU(cudaMemcpyAsync(s->x, x, bytes, cudaMemcpyHostToDevice, s->stream));
  mst_status st = s->cluster      ? lu_solve_cluster(s, method == MST_LU_GS, iterations)
                  : s->block == 1 ? lu_iterate<1>(s, method == MST_LU_GS, iterations)
                                  : lu_iterate<4>(s, 0, iterations);
  if (st) return st;
  LU_CU(cudaMemcpyAsync(x, s->x, bytes, cudaMemcpyDeviceToHost, s->stream));
  LU_CU(cudaStreamSynchronize(s->stream));
  return MST_OK;
}

mst_status mst_lu_levels(const mst_lu* s, int* forward, int* backward) {
  if (!s) return lu_fail(MST_EINVAL, "NULL argument");
  if (forward) *forward = s->n_fwd_levels;
  if (backward) *backward = s->n_bwd_levels;
  return MST_OK;
}

mst_status mst_lu_destroy(mst_lu* s) {
  if (!s) return MST_OK;
  if (s->stream) cudaStreamSynchronize(s->stream);
  for (void* p : s->allocs) cudaFree(p);
  if (s->stream) cudaStreamDestroy(s->stream);
  delete s;
  return MST_OK;
}

}  // extern "C"
